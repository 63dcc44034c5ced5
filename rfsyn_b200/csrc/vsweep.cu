// vsweep.cu -- kernels of the vector sweep (see vsweep.cuh).
#include <cuda_runtime.h>

#include "vsweep.cuh"

namespace rfb {

// ---- vectors of cells ---------------------------------------------------------
template <typename T>
struct Vec;
template <>
struct Vec<float> {
    static constexpr int N = 4;
    unsigned long long p[2];
};
template <>
struct Vec<double> {
    static constexpr int N = 2;
    double p[2];
};

#define RFB_V_OP(NAME, PTX, FN)                                                                          \
    __device__ __forceinline__ Vec<float> NAME(const Vec<float> &a, const Vec<float> &b) {               \
        Vec<float> r;                                                                                    \
        asm(PTX ".rn.f32x2 %0, %1, %2;" : "=l"(r.p[0]) : "l"(a.p[0]), "l"(b.p[0]));                      \
        asm(PTX ".rn.f32x2 %0, %1, %2;" : "=l"(r.p[1]) : "l"(a.p[1]), "l"(b.p[1]));                      \
        return r;                                                                                        \
    }                                                                                                    \
    __device__ __forceinline__ Vec<double> NAME(const Vec<double> &a, const Vec<double> &b) {            \
        Vec<double> r;                                                                                   \
        r.p[0] = FN(a.p[0], b.p[0]);                                                                     \
        r.p[1] = FN(a.p[1], b.p[1]);                                                                     \
        return r;                                                                                        \
    }
RFB_V_OP(va, "add", __dadd_rn)
RFB_V_OP(vs, "sub", __dsub_rn)
#undef RFB_V_OP
// The rounded product.  The assembler contracts mul.rn.f32x2 feeding an
// add.rn.f32x2 into one rounding (-fmad=false does not stop it; the scalar
// mul.rn.f32 it leaves alone), which would round differently from every other
// sweep.  So the product is a b + z with z = -0 in both halves, exact for any
// a b, and z comes from the launch (VShape::nz), where the assembler cannot
// see its value: there is nothing left to contract.
__device__ __forceinline__ Vec<float> vm(const Vec<float> &a, const Vec<float> &b, unsigned long long z) {
    Vec<float> r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.p[0]) : "l"(a.p[0]), "l"(b.p[0]), "l"(z));
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.p[1]) : "l"(a.p[1]), "l"(b.p[1]), "l"(z));
    return r;
}
__device__ __forceinline__ Vec<double> vm(const Vec<double> &a, const Vec<double> &b, unsigned long long) {
    Vec<double> r;
    r.p[0] = __dmul_rn(a.p[0], b.p[0]);
    r.p[1] = __dmul_rn(a.p[1], b.p[1]);
    return r;
}

__device__ __forceinline__ unsigned long long v_pack(float x, float y) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ void v_unpack(unsigned long long v, float &x, float &y) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v));
}
__device__ __forceinline__ void v_get(const Vec<float> &v, float (&x)[4]) {
    v_unpack(v.p[0], x[0], x[1]);
    v_unpack(v.p[1], x[2], x[3]);
}
__device__ __forceinline__ void v_get(const Vec<double> &v, double (&x)[2]) {
    x[0] = v.p[0];
    x[1] = v.p[1];
}
__device__ __forceinline__ Vec<float> v_set(const float (&x)[4]) {
    Vec<float> r;
    r.p[0] = v_pack(x[0], x[1]);
    r.p[1] = v_pack(x[2], x[3]);
    return r;
}
__device__ __forceinline__ Vec<double> v_set(const double (&x)[2]) {
    Vec<double> r;
    r.p[0] = x[0];
    r.p[1] = x[1];
    return r;
}
__device__ __forceinline__ Vec<float> v_splat(float x) {
    Vec<float> r;
    r.p[0] = r.p[1] = v_pack(x, x);
    return r;
}
__device__ __forceinline__ Vec<double> v_splat(double x) {
    Vec<double> r;
    r.p[0] = r.p[1] = x;
    return r;
}
// differences along k: (v1 - v0, .., next - v_{N-1}) and (v0 - prev, ..,
// v_{N-1} - v_{N-2}); scalar, as the packed form would first have to move
// the shifted cells into register pairs
__device__ __forceinline__ Vec<float> v_diff_up(const Vec<float> &v, float next) {
    float x[4];
    v_get(v, x);
    const float y[4] = {__fsub_rn(x[1], x[0]), __fsub_rn(x[2], x[1]), __fsub_rn(x[3], x[2]), __fsub_rn(next, x[3])};
    return v_set(y);
}
__device__ __forceinline__ Vec<double> v_diff_up(const Vec<double> &v, double next) {
    const double y[2] = {__dsub_rn(v.p[1], v.p[0]), __dsub_rn(next, v.p[1])};
    return v_set(y);
}
__device__ __forceinline__ Vec<float> v_diff_down(float prev, const Vec<float> &v) {
    float x[4];
    v_get(v, x);
    const float y[4] = {__fsub_rn(x[0], prev), __fsub_rn(x[1], x[0]), __fsub_rn(x[2], x[1]), __fsub_rn(x[3], x[2])};
    return v_set(y);
}
__device__ __forceinline__ Vec<double> v_diff_down(double prev, const Vec<double> &v) {
    const double y[2] = {__dsub_rn(v.p[0], prev), __dsub_rn(v.p[1], v.p[0])};
    return v_set(y);
}
__device__ __forceinline__ float v_last(const Vec<float> &v) {
    float x, y;
    v_unpack(v.p[1], x, y);
    return y;
}
__device__ __forceinline__ double v_last(const Vec<double> &v) { return v.p[1]; }
// element e of the result: bit e of m ? x : y
template <typename T>
__device__ __forceinline__ Vec<T> v_sel(unsigned m, const Vec<T> &x, const Vec<T> &y) {
    T a[Vec<T>::N], b[Vec<T>::N];
    v_get(x, a);
    v_get(y, b);
#pragma unroll
    for (int e = 0; e < Vec<T>::N; e++) a[e] = (m >> e) & 1u ? a[e] : b[e];
    return v_set(a);
}
template <typename T>
__device__ __forceinline__ Vec<T> v_load(const void *p) {
    Vec<T> r;
    if constexpr (sizeof(T) == 4) {
        const ulonglong2 q = *reinterpret_cast<const ulonglong2 *>(p);
        r.p[0] = q.x;
        r.p[1] = q.y;
    } else {
        const double2 q = *reinterpret_cast<const double2 *>(p);
        r.p[0] = q.x;
        r.p[1] = q.y;
    }
    return r;
}
template <typename T>
__device__ __forceinline__ void v_store(void *p, const Vec<T> &v) {
    if constexpr (sizeof(T) == 4) *reinterpret_cast<ulonglong2 *>(p) = make_ulonglong2(v.p[0], v.p[1]);
    else *reinterpret_cast<double2 *>(p) = make_double2(v.p[0], v.p[1]);
}

// a vector at a byte offset of a global array
template <typename T>
__device__ __forceinline__ Vec<T> v_gload(const void *base, unsigned off) {
    return v_load<T>(static_cast<const char *>(base) + off);
}
template <typename T>
__device__ __forceinline__ void v_gstore(void *base, unsigned off, const Vec<T> &v) {
    v_store<T>(static_cast<char *>(base) + off, v);
}
// shared memory by 32-bit address
template <typename T>
__device__ __forceinline__ Vec<T> v_slds(unsigned p) {
    Vec<T> r;
    if constexpr (sizeof(T) == 4)
        asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(r.p[0]), "=l"(r.p[1]) : "r"(p) : "memory");
    else asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(r.p[0]), "=d"(r.p[1]) : "r"(p) : "memory");
    return r;
}
template <typename T>
__device__ __forceinline__ void v_ssts(unsigned p, const Vec<T> &v) {
    if constexpr (sizeof(T) == 4)
        asm volatile("st.shared.v2.b64 [%0], {%1, %2};" ::"r"(p), "l"(v.p[0]), "l"(v.p[1]) : "memory");
    else asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(p), "d"(v.p[0]), "d"(v.p[1]) : "memory");
}
__device__ __forceinline__ void s_lds(unsigned p, float &x) {
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(x) : "r"(p) : "memory");
}
__device__ __forceinline__ void s_lds(unsigned p, double &x) {
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(x) : "r"(p) : "memory");
}
__device__ __forceinline__ void s_sts(unsigned p, float x) {
    asm volatile("st.shared.f32 [%0], %1;" ::"r"(p), "f"(x) : "memory");
}
__device__ __forceinline__ void s_sts(unsigned p, double x) {
    asm volatile("st.shared.f64 [%0], %1;" ::"r"(p), "d"(x) : "memory");
}
// asynchronous copy of one vector into the thread's own shared slot
__device__ __forceinline__ void v_async(unsigned smem, const void *base, unsigned off) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem), "l"(static_cast<const char *>(base) + off)
                 : "memory");
}

// H - cbh d and Ca E + Cb t, every product and sum rounded on its own
template <typename T>
__device__ __forceinline__ Vec<T> v_upd_h(const Vec<T> &h, const Vec<T> &cbh, const Vec<T> &d,
                                          unsigned long long z) {
    return vs(h, vm(cbh, d, z));
}
template <typename T>
__device__ __forceinline__ Vec<T> v_upd_e(const Vec<T> &ca, const Vec<T> &e, const Vec<T> &cb, const Vec<T> &t,
                                          unsigned long long z) {
    return va(vm(ca, e, z), vm(cb, t, z));
}
// rfsyn's cpml_term on a vector: psi <- b psi + a d, returns d kinv + dx psi
template <typename T>
__device__ __forceinline__ Vec<T> v_stretch(const Vec<T> &d, const Vec<T> &kinv, const Vec<T> &b, const Vec<T> &ac,
                                            const Vec<T> &dx, Vec<T> &psi, unsigned long long z) {
    psi = va(vm(b, psi, z), vm(ac, d, z));
    return va(vm(d, kinv, z), vm(dx, psi, z));
}

// The march of one item.  KIND: which slabs its cells and halos touch (V_Z,
// V_Y, V_X bits; V_X items may touch any), 0 for tiles outside every slab and
// boundary.  Returns false when a copy did not complete in time.
template <typename T, int KIND>
__device__ __forceinline__ bool v_item(const Args<T> &a, const VShape &sh, const VMaps &maps, const VItem &it,
                                       unsigned char *smem) {
    using V = Vec<T>;
    constexpr int N = V::N;
    constexpr bool SLAB = KIND != 0, XS = (KIND & V_X) != 0, YS = (KIND & V_Y) != 0, ZS = (KIND & V_Z) != 0;
    constexpr unsigned FULL = (1u << N) - 1u, FULL3 = (1u << (3 * N)) - 1u;
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem);
    const int tid = threadIdx.x;
    const int nv1 = sh.nv + 1, nv2 = sh.nv + 2;
    const bool px = a.per & 1u, py = a.per & 2u;
    const int j0 = it.j0, k0 = it.k0, ib = it.ib, steps = it.ie - it.ib;
    const bool wlo = sh.wrap && j0 == 0, whi = sh.wrap && j0 + sh.tr >= a.ny;
    const int nx = a.nx;

    // iteration n works on plane ib - 1 + n (wrapped on a periodic x axis);
    // n = 0 only prepares the previous plane's H
    auto plane_of = [&](int n) {
        int p = ib - 1 + n;
        if (px) p = p < 0 ? p + nx : p >= nx ? p - nx : p;
        return p;
    };
    // one load takes the box of all three components
    auto load_e = [&](int slot, int p, uint64_t *bar) {
        unsigned char *d = smem + v_e_stage(sh, slot);
        tma_load_4d(d, &maps.e, k0 - N, j0 - 1, p, 0, bar);
        if (wlo) tma_load_4d(d + sh.erow, &maps.e1, k0 - N, a.ny - 1, p, 0, bar);
        if (whi) tma_load_4d(d + sh.erow + sh.ewrap, &maps.e1, k0 - N, 0, p, 0, bar);
    };
    auto load_h = [&](int slot, int p, uint64_t *bar) {
        unsigned char *d = smem + v_h_stage(sh, slot);
        tma_load_4d(d, &maps.h, k0 - N, j0 - 1, p, 0, bar);
        if (wlo) tma_load_4d(d + sh.hrow, &maps.h1, k0 - N, a.ny - 1, p, 0, bar);
    };
    // group n: E of iteration n + 1 and H of iteration n (group 0 also E of 0)
    auto issue = [&](int n, int eslot, int hslot) {
        uint64_t *bar = &bars[hslot];
        const unsigned e_tx = 48u * nv2 * (sh.tr + 2 + (wlo ? 1 : 0) + (whi ? 1 : 0));
        const unsigned h_tx = 48u * nv1 * (sh.tr + 1 + (wlo ? 1 : 0));
        mbar_expect_tx(bar, (n == 0 ? 2u : 1u) * e_tx + h_tx);
        if (n == 0) load_e(0, plane_of(0), bar);
        load_e(eslot, plane_of(n + 1), bar);
        load_h(hslot, plane_of(n), bar);
    };

    // ---- the thread's vector ----
    const int rr = tid / nv1, vv = tid - rr * nv1;
    const int j = j0 - 1 + rr, k = k0 - N + vv * N;
    const int jw = (py && j < 0) ? a.ny - 1 : j;
    const bool in_tile = rr <= sh.tr;
    const bool valid = in_tile && jw >= 0 && k >= 0 && jw < sh.cj && k < sh.ck;
    const bool own = valid && rr > 0 && vv > 0;
    // shared offsets of the vector in an E stage, of the vector one row up,
    // and in an H stage, and the component strides there
    int oe = 0, ou = 0, oh = 0, ce = sh.ebox, cu = sh.ebox, ch = sh.hbox;
    if (in_tile) {
        oe = (rr * nv2 + vv) * 16;
        ou = oe + nv2 * 16;
        oh = tid * 16;
        if (sh.wrap) {
            if (j == a.ny - 1) {
                ou = sh.erow + sh.ewrap + vv * 16;
                cu = nv2 * 16;
            }
            if (j < 0) {
                oe = sh.erow + vv * 16;
                oh = sh.hrow + vv * 16;
                ce = nv2 * 16;
                ch = nv1 * 16;
            }
        }
    }
    // update ranges at (j, k), plane apart: bits c * N + e of H and of E
    unsigned hm = 0, em = 0;
    if (SLAB && valid) {
        const int jmin = py ? 0 : 1, kmin = (a.per & 4u) ? 0 : 1;
        const int jhi = a.ny + (py ? 0 : 1), khi = a.nz + ((a.per & 4u) ? 0 : 1);
#pragma unroll
        for (int e = 0; e < N; e++) {
            const int q = k + e;
            const bool ij = jw < a.ny, ik = q < a.nz;
            if (ij && ik) hm |= 1u << e;
            if (jw < jhi && ik) hm |= 1u << (N + e);
            if (ij && q < khi) hm |= 1u << (2 * N + e);
            if (ij && ik) {
                if (jw >= jmin && q >= kmin) em |= 1u << e;
                if (q >= kmin) em |= 1u << (N + e);
                if (jw >= jmin) em |= 1u << (2 * N + e);
            }
        }
    }
    // slabs of the thread's row and vector: element offsets of its psi
    // vectors in a plane (-1: outside), masks of the vector's cells in the z
    // slab on the H and the E grid
    constexpr int ES = (int)sizeof(T);
    const int cjk = jw * (int)a.pitch + k, plane = (int)a.plane;
    // psi offsets by bytes: of the vector in a plane of the array, and the
    // array's plane stride
    bool yh = false, ym = false;
    unsigned pyh = 0, pym = 0, pzh = 0, pzm = 0;
    unsigned zhm = 0, zem = 0;
    if (SLAB && a.cpml_on && valid) {
        if constexpr (YS) {
            const int sh_ = jw < a.ny ? slab_of(jw, a.lo_h[1], a.hi_h[1], a.off_h[1]) : -1;
            const int sm_ = own ? slab_of(jw, a.lo_m[1], a.hi_m[1], a.off_m[1]) : -1;
            yh = sh_ >= 0;
            ym = sm_ >= 0;
            pyh = (unsigned)(sh_ * (int)a.pitch + k) * ES;
            pym = (unsigned)(sm_ * (int)a.pitch + k) * ES;
        }
        if constexpr (ZS) {
#pragma unroll
            for (int e = 0; e < N; e++) {
                const int q = k + e;
                if (q < a.lo_h[2] || (q >= a.hi_h[2] && q < a.nz)) zhm |= 1u << e;
                if (q < a.lo_m[2] || (q >= a.hi_m[2] && q <= a.nz)) zem |= 1u << e;
            }
            if (!own) zem = 0;
            pzh = (unsigned)(jw * a.ns_h[2] + (k < a.lo_h[2] ? k : k + a.off_h[2])) * ES;
            pzm = (unsigned)(jw * a.ns_m[2] + (k < a.lo_m[2] ? k : k + a.off_m[2])) * ES;
        }
    }
    const unsigned yph = (unsigned)(a.ns_h[1] * (int)a.pitch) * ES, ypm = (unsigned)(a.ns_m[1] * (int)a.pitch) * ES;
    const unsigned zph = (unsigned)(a.ns_h[2] * (a.ny + 1)) * ES, zpm = (unsigned)(a.ns_m[2] * (a.ny + 1)) * ES;
    const bool with_codes = a.codes != nullptr;
    // a code-less scene's list cells in this thread's column
    bool skips = false;
    if (SLAB && !with_codes && own)
        for (int s = 0; s < a.n_skip; s++) {
            const int r = (int)(a.skip[s] % a.plane) - cjk;
            skips |= r >= 0 && r < N;
        }
    const unsigned long long z = sh.nz;
    const V cbh = v_splat(a.cbh), dx = v_splat(a.dx), ca0 = v_splat(__ldg(a.tca)), cb0 = v_splat(__ldg(a.tcb));
    // tables of the item in shared memory: (Ca, Cb) per code, y profiles of
    // the tile's rows, z profiles of its vectors (kinv b a on the H grid,
    // then on the E grid)
    T *tab = reinterpret_cast<T *>(smem + sh.o_tab), *py6 = reinterpret_cast<T *>(smem + sh.o_py);
    unsigned char *pz6 = smem + sh.o_pz;
    if (with_codes)
        for (int t = tid; t < 256; t += blockDim.x) {
            tab[2 * t] = __ldg(a.tca + t);
            tab[2 * t + 1] = __ldg(a.tcb + t);
        }
    if (SLAB && a.cpml_on && in_tile) {
        if (YS && vv == 0) {
            const bool h = jw >= 0 && jw < a.ny, m = jw >= 0 && jw <= a.ny;
#pragma unroll
            for (int q = 0; q < 3; q++) {
                const T *ph = q == 0 ? a.kinv_h[1] : q == 1 ? a.b_h[1] : a.a_h[1];
                const T *pm = q == 0 ? a.kinv_m[1] : q == 1 ? a.b_m[1] : a.a_m[1];
                py6[6 * rr + q] = h ? ph[jw] : T(0);
                py6[6 * rr + 3 + q] = m ? pm[jw] : T(0);
            }
        }
        if (ZS && rr == 0) {
            const bool h = k >= 0 && k < a.nz, m = k >= 0 && k <= a.nz;
#pragma unroll
            for (int q = 0; q < 3; q++) {
                const T *ph = q == 0 ? a.kinv_h[2] : q == 1 ? a.b_h[2] : a.a_h[2];
                const T *pm = q == 0 ? a.kinv_m[2] : q == 1 ? a.b_m[2] : a.a_m[2];
                v_store<T>(pz6 + 16 * (6 * vv + q), h ? v_load<T>(ph + k) : v_splat(T(0)));
                v_store<T>(pz6 + 16 * (6 * vv + 3 + q), m ? v_load<T>(pm + k) : v_splat(T(0)));
            }
        }
    }
    const bool coded = with_codes && own;
    unsigned oc = (unsigned)ib * (unsigned)plane + (unsigned)cjk;  // byte offset of the next plane's codes
    auto code_word = [&]() -> unsigned {
        const uint8_t *c = a.codes + oc;
        if constexpr (N == 4) return __ldg(reinterpret_cast<const unsigned *>(c));
        else return __ldg(reinterpret_cast<const unsigned short *>(c));
    };
    unsigned cw = coded ? code_word() : 0u;

    const unsigned sb = smem_addr(smem);
    int es = 0, hs = 0;     // slots of the plane's E and H
    unsigned parity = 0;    // of the H slot's barrier
    const unsigned rows = sb + sh.o_rows + tid * 16, last = sb + sh.o_last + tid * ES;
    const unsigned rows_comp = 16 * sh.nt, last_comp = ES * sh.nt, tabs = sb + sh.o_tab;
    const unsigned pys = sb + sh.o_py + 6 * ES * rr, pzs = sb + sh.o_pz + 96 * vv;
    bool failed = false;

    // psi vectors y (0, 5), z (1, 2), x (3, 4) of H and, EQ slots on, of E: a
    // thread copies its own into its own shared slots one plane ahead, as
    // soon as the plane's are used (no other thread reads them)
    const unsigned slot = sb + sh.o_psi + tid * 16, slot_n = 16 * sh.nt;
    constexpr int ZQ = YS ? 2 : 0, XQ = ZQ + (ZS ? 2 : 0), EQ = XQ + (XS ? 2 : 0);
    auto slab_x = [&](int i, bool h) {
        if (!a.cpml_on || i < 0) return -1;
        return h ? (i < nx ? slab_of(i, a.lo_h[0], a.hi_h[0], a.off_h[0]) : -1)
                 : slab_of(i, a.lo_m[0], a.hi_m[0], a.off_m[0]);
    };
    auto load_qh = [&](int i) {
        if (i >= 0) {
            if constexpr (YS)
                if (yh) {
                    const unsigned o = i * yph + pyh;
                    v_async(slot, a.psi_hi[0], o);
                    v_async(slot + slot_n, a.psi_hi[5], o);
                }
            if constexpr (ZS)
                if (zhm) {
                    const unsigned o = i * zph + pzh;
                    v_async(slot + ZQ * slot_n, a.psi_hi[1], o);
                    v_async(slot + (ZQ + 1) * slot_n, a.psi_hi[2], o);
                }
            if constexpr (XS) {
                const int sx = slab_x(i, true);
                if (sx >= 0 && valid) {
                    const unsigned o = ((unsigned)sx * (unsigned)plane + (unsigned)cjk) * ES;
                    v_async(slot + XQ * slot_n, a.psi_hi[3], o);
                    v_async(slot + (XQ + 1) * slot_n, a.psi_hi[4], o);
                }
            }
        }
        cp_async_commit();
    };
    auto load_qe = [&](int i) {
        if constexpr (YS)
            if (ym) {
                const unsigned o = i * ypm + pym;
                v_async(slot + EQ * slot_n, a.psi_e[0], o);
                v_async(slot + (EQ + 1) * slot_n, a.psi_e[5], o);
            }
        if constexpr (ZS)
            if (zem) {
                const unsigned o = i * zpm + pzm;
                v_async(slot + (EQ + ZQ) * slot_n, a.psi_e[1], o);
                v_async(slot + (EQ + ZQ + 1) * slot_n, a.psi_e[2], o);
            }
        if constexpr (XS) {
            const int sx = slab_x(i, false);
            if (sx >= 0 && own) {
                const unsigned o = ((unsigned)sx * (unsigned)plane + (unsigned)cjk) * ES;
                v_async(slot + (EQ + XQ) * slot_n, a.psi_e[3], o);
                v_async(slot + (EQ + XQ + 1) * slot_n, a.psi_e[4], o);
            }
        }
        cp_async_commit();
    };
    // everything so far reads only what no step writes; from here on the
    // fields and psi of the launches before this one
    grid_wait();
    int issued = 0;
    if (tid == 0)
        for (; issued < V_NH && issued <= steps; issued++) issue(issued, issued + 1, issued);
    int i = plane_of(0);
    // groups of a thread's copies alternate H psi, E psi: each wait below
    // leaves the newest one in flight
    if constexpr (SLAB) {
        load_qh(i);
        cp_async_commit();
    }
    // the item's output planes, and the vector's byte offset from the first
    T *const ho0 = a.Ho[0] + (long long)ib * plane, *const ho1 = a.Ho[1] + (long long)ib * plane,
             *const ho2 = a.Ho[2] + (long long)ib * plane;
    T *const eo0 = a.Eo[0] + (long long)ib * plane, *const eo1 = a.Eo[1] + (long long)ib * plane,
             *const eo2 = a.Eo[2] + (long long)ib * plane;
    unsigned of = (unsigned)cjk * ES;
    __syncthreads();  // the tables

    if (!mbar_wait(&bars[0], 0)) failed = true;
    V cey = v_slds<T>(sb + v_e_stage(sh, 0) + oe + ce), cez = v_slds<T>(sb + v_e_stage(sh, 0) + oe + 2 * ce);
    V phy{}, phz{};
    for (int n = 0; n <= steps; n++) {
        const int inext = px && i + 1 == nx ? 0 : i + 1;
        // the plane's x profiles (kinv b a on the H grid, then on the E grid)
        int sxh = -1, sxm = -1;  // and its slots in the x psi arrays
        T xp[6];
        if constexpr (XS) {
            sxh = valid ? slab_x(i, true) : -1;
            sxm = own && n > 0 ? slab_x(i, false) : -1;
            if (sxh >= 0) {
                xp[0] = __ldg(a.kinv_h[0] + i);
                xp[1] = __ldg(a.b_h[0] + i);
                xp[2] = __ldg(a.a_h[0] + i);
            }
            if (sxm >= 0) {
                xp[3] = __ldg(a.kinv_m[0] + i);
                xp[4] = __ldg(a.b_m[0] + i);
                xp[5] = __ldg(a.a_m[0] + i);
            }
        }
        // a timed-out wait marks the thread failed; its later waits only look
        if (!mbar_wait_for(&bars[hs], parity, failed ? 0 : 2000000000LL)) failed = true;
        // ---- H of the plane ----
        const int en_s = es == V_NE - 1 ? 0 : es + 1;
        const unsigned e0s = sb + v_e_stage(sh, es), ec = e0s + oe, en = sb + v_e_stage(sh, en_s) + oe,
                       eu = e0s + ou, hc = sb + v_h_stage(sh, hs) + oh;
        const V cex = v_slds<T>(ec);
        T nx_, ny_;
        s_lds(ec + 16, nx_);
        s_lds(ec + ce + 16, ny_);
        const V uez = v_slds<T>(eu + 2 * cu), uex = v_slds<T>(eu);
        const V ney = v_slds<T>(en + ce), nez = v_slds<T>(en + 2 * ce);
        const V h0 = v_slds<T>(hc), h1 = v_slds<T>(hc + ch), h2 = v_slds<T>(hc + 2 * ch);
        V dxA = vs(uez, cez), dxB = v_diff_up(cey, ny_);  // Hx: d_y Ez, d_z Ey
        V dyA = v_diff_up(cex, nx_), dyB = vs(nez, cez);  // Hy: d_z Ex, d_x Ez
        V dzA = vs(ney, cey), dzB = vs(uex, cex);         // Hz: d_x Ey, d_y Ex
        const bool st = n > 0 && own;
        if constexpr (SLAB) cp_async_wait<1>();  // this plane's H psi (its E psi may be in flight)
        if constexpr (YS) {
            if (yh && i >= 0) {
                T p0, p1, p2;
                s_lds(pys, p0);
                s_lds(pys + ES, p1);
                s_lds(pys + 2 * ES, p2);
                const V ki = v_splat(p0), b = v_splat(p1), ac = v_splat(p2);
                V q0 = v_slds<T>(slot), q5 = v_slds<T>(slot + slot_n);
                dxA = v_stretch(dxA, ki, b, ac, dx, q0, z);
                dzB = v_stretch(dzB, ki, b, ac, dx, q5, z);
                if (st) {
                    const unsigned o = i * yph + pyh;
                    v_gstore<T>(a.psi_ho[0], o, q0);
                    v_gstore<T>(a.psi_ho[5], o, q5);
                }
            }
        }
        if constexpr (ZS) {
            if (zhm && i >= 0) {
                const V ki = v_slds<T>(pzs), b = v_slds<T>(pzs + 16), ac = v_slds<T>(pzs + 32);
                const V o1 = v_slds<T>(slot + ZQ * slot_n), o2 = v_slds<T>(slot + (ZQ + 1) * slot_n);
                V q1 = o1, q2 = o2;
                V r1 = v_stretch(dxB, ki, b, ac, dx, q1, z), r2 = v_stretch(dyA, ki, b, ac, dx, q2, z);
                if (zhm != FULL) {
                    r1 = v_sel<T>(zhm, r1, dxB);
                    r2 = v_sel<T>(zhm, r2, dyA);
                    q1 = v_sel<T>(zhm, q1, o1);
                    q2 = v_sel<T>(zhm, q2, o2);
                }
                dxB = r1;
                dyA = r2;
                if (st) {
                    const unsigned o = i * zph + pzh;
                    v_gstore<T>(a.psi_ho[1], o, q1);
                    v_gstore<T>(a.psi_ho[2], o, q2);
                }
            }
        }
        if constexpr (XS) {
            if (sxh >= 0) {
                const V ki = v_splat(xp[0]), b = v_splat(xp[1]), ac = v_splat(xp[2]);
                V q3 = v_slds<T>(slot + XQ * slot_n), q4 = v_slds<T>(slot + (XQ + 1) * slot_n);
                dyB = v_stretch(dyB, ki, b, ac, dx, q3, z);
                dzA = v_stretch(dzA, ki, b, ac, dx, q4, z);
                if (st) {
                    const unsigned o = ((unsigned)sxh * (unsigned)plane + (unsigned)cjk) * ES;
                    v_gstore<T>(a.psi_ho[3], o, q3);
                    v_gstore<T>(a.psi_ho[4], o, q4);
                }
            }
        }
        if constexpr (SLAB) {
            if (n < steps) load_qh(inext);
            else cp_async_commit();
        }
        V hx = v_upd_h(h0, cbh, vs(dxA, dxB), z), hy = v_upd_h(h1, cbh, vs(dyA, dyB), z),
          hz = v_upd_h(h2, cbh, vs(dzA, dzB), z);
        if constexpr (SLAB) {
            // cells outside a component's update range keep their H
            unsigned m = hm;
            if (i < 0 || i >= nx) m &= (i == nx && !px) ? FULL : 0u;
            if (m != FULL3) {
                hx = v_sel<T>(m, hx, h0);
                hy = v_sel<T>(m >> N, hy, h1);
                hz = v_sel<T>(m >> (2 * N), hz, h2);
            }
        }
        const unsigned rw = rows + (n & 1 ? 2 * rows_comp : 0u), ls = last + (n & 1 ? 2 * last_comp : 0u);
        v_ssts<T>(rw, hx);
        v_ssts<T>(rw + rows_comp, hz);
        s_sts(ls, v_last(hx));
        s_sts(ls + last_comp, v_last(hy));
        __syncthreads();
        // every read of E of iteration n and of H of iteration n is behind
        // the barrier: their slots take E of n + V_NE and H of n + V_NH
        if (tid == 0 && n + V_NH <= steps && !failed) {
            issue(n + V_NH, es, hs);
            issued++;
        }
        if (st) {
            // ---- E of the plane ----
            const V hxj = v_slds<T>(rw - nv1 * 16), hzj = v_slds<T>(rw + rows_comp - nv1 * 16);
            T hxk, hyk;
            s_lds(ls - ES, hxk);
            s_lds(ls + last_comp - ES, hyk);
            v_gstore<T>(ho0, of, hx);
            v_gstore<T>(ho1, of, hy);
            v_gstore<T>(ho2, of, hz);
            const unsigned w = cw;
            if (coded && n < steps) {
                oc += plane;
                cw = code_word();
            }
            V ca = ca0, cb = cb0;
            unsigned lm = 0;  // list cells of the vector
            if (w != 0u) {
                T x[N], y[N];
#pragma unroll
                for (int e = 0; e < N; e++) {
                    const unsigned cd = (w >> (8 * e)) & 0xffu;
                    s_lds(tabs + 2 * ES * cd, x[e]);
                    s_lds(tabs + 2 * ES * cd + ES, y[e]);
                    if (SLAB && cd == (unsigned)LIST_CODE) lm |= 1u << e;
                }
                ca = v_set(x);
                cb = v_set(y);
            }
            if constexpr (SLAB) {
                if (skips)
                    for (int s = 0; s < a.n_skip; s++) {
                        const long long r = a.skip[s] - ((long long)i * plane + cjk);
                        if (r >= 0 && r < N) lm |= 1u << (int)r;
                    }
            }
            V txA = vs(hz, hzj), txB = v_diff_down(hyk, hy);  // Ex: d_y Hz, d_z Hy
            V tyA = v_diff_down(hxk, hx), tyB = vs(hz, phz);  // Ey: d_z Hx, d_x Hz
            V tzA = vs(hy, phy), tzB = vs(hx, hxj);           // Ez: d_x Hy, d_y Hx
            const unsigned keep = FULL & ~lm;  // cells whose psi the sweep advances
            if constexpr (SLAB) cp_async_wait<1>();  // this plane's E psi
            if constexpr (YS) {
                if (ym) {
                    T p0, p1, p2;
                    s_lds(pys + 3 * ES, p0);
                    s_lds(pys + 4 * ES, p1);
                    s_lds(pys + 5 * ES, p2);
                    const V ki = v_splat(p0), b = v_splat(p1), ac = v_splat(p2);
                    const V o0 = v_slds<T>(slot + EQ * slot_n), o5 = v_slds<T>(slot + (EQ + 1) * slot_n);
                    V q0 = o0, q5 = o5;
                    txA = v_stretch(txA, ki, b, ac, dx, q0, z);
                    tzB = v_stretch(tzB, ki, b, ac, dx, q5, z);
                    if (lm) {
                        q0 = v_sel<T>(keep, q0, o0);
                        q5 = v_sel<T>(keep, q5, o5);
                    }
                    const unsigned o = i * ypm + pym;
                    v_gstore<T>(a.psi_e[0], o, q0);
                    v_gstore<T>(a.psi_e[5], o, q5);
                }
            }
            if constexpr (ZS) {
                if (zem) {
                    const V ki = v_slds<T>(pzs + 48), b = v_slds<T>(pzs + 64), ac = v_slds<T>(pzs + 80);
                    const V o1 = v_slds<T>(slot + (EQ + ZQ) * slot_n), o2 = v_slds<T>(slot + (EQ + ZQ + 1) * slot_n);
                    V q1 = o1, q2 = o2;
                    V r1 = v_stretch(txB, ki, b, ac, dx, q1, z), r2 = v_stretch(tyA, ki, b, ac, dx, q2, z);
                    const unsigned m = zem & keep;
                    if (m != FULL) {
                        r1 = v_sel<T>(zem, r1, txB);
                        r2 = v_sel<T>(zem, r2, tyA);
                        q1 = v_sel<T>(m, q1, o1);
                        q2 = v_sel<T>(m, q2, o2);
                    }
                    txB = r1;
                    tyA = r2;
                    const unsigned o = i * zpm + pzm;
                    v_gstore<T>(a.psi_e[1], o, q1);
                    v_gstore<T>(a.psi_e[2], o, q2);
                }
            }
            if constexpr (XS) {
                if (sxm >= 0) {
                    const V ki = v_splat(xp[3]), b = v_splat(xp[4]), ac = v_splat(xp[5]);
                    const V o3 = v_slds<T>(slot + (EQ + XQ) * slot_n), o4 = v_slds<T>(slot + (EQ + XQ + 1) * slot_n);
                    V q3 = o3, q4 = o4;
                    tyB = v_stretch(tyB, ki, b, ac, dx, q3, z);
                    tzA = v_stretch(tzA, ki, b, ac, dx, q4, z);
                    if (lm) {
                        q3 = v_sel<T>(keep, q3, o3);
                        q4 = v_sel<T>(keep, q4, o4);
                    }
                    const unsigned o = ((unsigned)sxm * (unsigned)plane + (unsigned)cjk) * ES;
                    v_gstore<T>(a.psi_e[3], o, q3);
                    v_gstore<T>(a.psi_e[4], o, q4);
                }
            }
            if constexpr (SLAB) {
                if (n < steps) load_qe(inext);
                else cp_async_commit();
            }
            V ex = v_upd_e(ca, cex, cb, vs(txA, txB), z), ey = v_upd_e(ca, cey, cb, vs(tyA, tyB), z),
              ez = v_upd_e(ca, cez, cb, vs(tzA, tzB), z);
            if constexpr (SLAB) {
                unsigned m = em;
                if (i >= nx) m = 0u;
                else if (i < 1 && !px) m &= FULL;
                if (m != FULL3) {
                    ex = v_sel<T>(m, ex, cex);
                    ey = v_sel<T>(m >> N, ey, cey);
                    ez = v_sel<T>(m >> (2 * N), ez, cez);
                }
            }
            v_gstore<T>(eo0, of, ex);
            v_gstore<T>(eo1, of, ey);
            v_gstore<T>(eo2, of, ez);
            of += (unsigned)plane * ES;
        } else if constexpr (SLAB) {
            if (n < steps) load_qe(inext);  // iteration 0; a halo thread loads nothing
            else cp_async_commit();
        }
        phy = hy;
        phz = hz;
        cey = ney;
        cez = nez;
        es = en_s;
        i = inext;
        if (++hs == V_NH) {
            hs = 0;
            parity ^= 1u;
        }
    }
    if (!__syncthreads_or(failed)) return true;
    // Copies still in flight land (bounded) before the shared memory is
    // released: the newest V_NH groups at most, each the newest of its barrier.
    // The parity of an older group says nothing once its barrier has moved on,
    // and waiting for it would run out.  (Starting at the groups thread 0 had
    // waited for as well costs a count through the march, and 24.6 for 23.8 us
    // a step on 38 x 164 x 129 FP32.)
    static_assert(V_NH <= 2, "an item's planes, one at least, and the one before make V_NH groups");
    if (tid == 0)
        for (int g = issued - V_NH; g < issued; g++) mbar_wait(&bars[g % V_NH], (unsigned)(g / V_NH) & 1u);
    __syncthreads();
    return false;
}

// The body of an item's kind.
template <typename T>
__device__ __forceinline__ bool v_run(const Args<T> &a, const VShape &sh, const VMaps &maps, const VItem &it,
                                      unsigned char *smem) {
    switch (it.kind) {
        case 0: return v_item<T, 0>(a, sh, maps, it, smem);
        case V_Z: return v_item<T, V_Z>(a, sh, maps, it, smem);
        case V_Y: return v_item<T, V_Y>(a, sh, maps, it, smem);
        case V_Y | V_Z: return v_item<T, V_Y | V_Z>(a, sh, maps, it, smem);
        default: return v_item<T, V_X | V_Y | V_Z>(a, sh, maps, it, smem);
    }
}

// Start of a CTA: shared memory aligned for the copies, barriers ready.
__device__ __forceinline__ bool v_begin(unsigned char *smem, int *err) {
    if (__cvta_generic_to_shared(smem) & 127u) {
        if (threadIdx.x == 0) atomicExch(err, 2);
        grid_wait();
        return false;
    }
    if (threadIdx.x == 0) {
        uint64_t *bars = reinterpret_cast<uint64_t *>(smem);
        for (int q = 0; q < V_NH; q++) mbar_init(&bars[q], 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    __syncthreads();
    return true;
}

template <typename T>
__global__ void __launch_bounds__(V_NT, V_MB)
    k_vsweep(const __grid_constant__ Args<T> a, const __grid_constant__ VShape sh, const VItem *items,
             const __grid_constant__ VMaps maps, int *err) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    grid_launch_next();
    if (!v_begin(smem_raw, err)) return;
    const VItem it = items[blockIdx.x];
    if (!v_run<T>(a, sh, maps, it, smem_raw) && threadIdx.x == 0) atomicExch(err, 1);
}

// Items of many scenes: the CTA copies its scene's parameters into shared
// memory behind the tile's (at args_off) and acquires the scene's tensor
// maps, which lie in global memory, through the tensormap proxy in the thread
// that issues the copies.
template <typename T>
__global__ void __launch_bounds__(V_NT, V_MB)
    k_vsweep_b(const Args<T> *args, const VShape *shapes, const VMaps *maps, const VItem *items, int args_off,
               int *err) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    grid_launch_next();
    const VItem it = items[blockIdx.x];
    Args<T> &sa = *reinterpret_cast<Args<T> *>(smem_raw + args_off);
    VShape &sh = *reinterpret_cast<VShape *>(smem_raw + args_off + (sizeof(Args<T>) + 15) / 16 * 16);
    {
        const unsigned *g = reinterpret_cast<const unsigned *>(args + it.scene);
        unsigned *d = reinterpret_cast<unsigned *>(&sa);
        for (int t = threadIdx.x; t < (int)(sizeof(Args<T>) / 4); t += blockDim.x) d[t] = g[t];
        const unsigned *gs = reinterpret_cast<const unsigned *>(shapes + it.scene);
        unsigned *ds = reinterpret_cast<unsigned *>(&sh);
        for (int t = threadIdx.x; t < (int)(sizeof(VShape) / 4); t += blockDim.x) ds[t] = gs[t];
    }
    const VMaps &m = maps[it.scene];
    if (threadIdx.x == 0) {
        const CUtensorMap *q[4] = {&m.e, &m.h, &m.e1, &m.h1};
#pragma unroll
        for (int t = 0; t < 4; t++)
            asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;\n" ::"l"(q[t]) : "memory");
    }
    if (!v_begin(smem_raw, err)) return;
    if (!v_run<T>(sa, sh, m, it, smem_raw) && threadIdx.x == 0) atomicExch(err, 1);
}

template <typename T>
int v_prepare() {
    return cudaFuncSetAttribute(k_vsweep<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, V_SMEM) == cudaSuccess &&
                   cudaFuncSetAttribute(k_vsweep_b<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, V_SMEM) ==
                       cudaSuccess
               ? 0
               : -1;
}

template <typename T>
void v_launch(const Args<T> &a, const VShape &sh, const VItem *items, int n, const VMaps &maps, int *err,
              cudaStream_t st, bool overlap) {
    if (n > 0) launch_step(k_vsweep<T>, dim3(n), dim3(sh.nt), sh.smem, st, overlap, a, sh, items, maps, err);
}

template <typename T>
void v_launch_b(const Args<T> *args, const VShape *shapes, const VMaps *maps, const VItem *items, int n, int nt,
                int smem, int *err, cudaStream_t st, bool overlap) {
    if (n > 0)
        launch_step(k_vsweep_b<T>, dim3(n), dim3(nt), smem + v_args_bytes<T>(), st, overlap, args, shapes, maps, items,
                    smem, err);
}

template int v_prepare<float>();
template int v_prepare<double>();
template void v_launch<float>(const Args<float> &, const VShape &, const VItem *, int, const VMaps &, int *,
                              cudaStream_t, bool);
template void v_launch<double>(const Args<double> &, const VShape &, const VItem *, int, const VMaps &, int *,
                               cudaStream_t, bool);
template void v_launch_b<float>(const Args<float> *, const VShape *, const VMaps *, const VItem *, int, int, int,
                                int *, cudaStream_t, bool);
template void v_launch_b<double>(const Args<double> *, const VShape *, const VMaps *, const VItem *, int, int, int,
                                 int *, cudaStream_t, bool);

}  // namespace rfb
