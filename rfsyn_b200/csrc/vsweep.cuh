// vsweep.cuh -- H+E sweep of vector cells (sweep mode 5): what grids without a
// periodic z axis run on, up to its 32-bit limits (v_fits).
//
// One launch per time step takes the whole grid.  A CTA marches one item --
// a tile of TR rows x NV vectors in (j, k), a range of planes -- along i; a
// thread owns one 16-byte vector of cells (4 FP32 or 2 FP64) of a row.
//
// What it is bound by, and why it looks like this.  The scalar sweeps
// (k_sweep_q: one or two cells a thread) were bound by instruction issue:
// ~155 warp instructions per 32 interior cells and ~650 in slab tiles, at
// 0.56 of the copy bandwidth on 256^3 FP32 and far below it on small grids,
// most of whose tiles are slab tiles.  Here a shared-memory access, a global
// access and an address serve four cells, and the FP32 arithmetic runs two
// cells to an instruction (add / sub / mul .rn.f32x2, each lane rounded on
// its own, so the results are the scalar sweeps' bit for bit).
//
// Tile threads: (TR + 1) x (NV + 1), linear, one vector each.  Row 0 and
// vector 0 are the tile's low-j / low-k halo: their threads recompute the
// neighbours' H (never stored) with the same code as everyone else, so no
// warp has an extra job.  NV and TR are run-time numbers chosen by the host
// for the grid (v_rule), so odd extents leave few idle lanes.
//
// Per plane: one thread issues one tiled TMA load for E (TR + 2 rows x NV + 2
// vectors x 3 components: the components of a buffer are one tensor) and one
// for H (TR + 1 x NV + 1 x 3) into rings of three E and two H stages; E of
// plane n + 1 and H of plane n complete on one mbarrier and are issued two
// planes ahead, right after the block barrier that frees their slots (rings
// of three and four planes measured the same).  H of the plane follows from shared E; its rows and its vectors'
// last cells go to shared memory (double-buffered by plane, so one barrier
// per plane suffices), and E follows from those and the previous plane's H
// kept in registers.
//
// CPML: a thread whose row, vector or plane lies in a slab copies its psi
// vectors into shared slots of its own one plane ahead (cp.async) and applies
// the recursion to whole vectors.  Held in registers instead, the next
// plane's psi cost up to 48 registers a thread, and spills of a few hundred
// bytes a thread thrash the L1 that the stages leave (256^3 FP32 at 96
// registers: 0.46 ms a sweep).  For the same reason the profiles and the
// material table sit in shared memory: a table read that misses L1 stalls
// every plane for the L2's latency.  z-slab psi rows are stored in
// vector-aligned slots (SlabExt); cells of a straddling vector outside the slab keep their plain difference.
//
// List cells: the sweep may write any E there (the list kernel overwrites
// it) but leaves their psi_e alone.  Cells a component's update range leaves
// out keep their input value.
//
// Measured (sweep alone, before = the scalar sweeps): 256^3 FP32 238 us
// (0.97 GB: 4.1 TB/s) for 265, 128 x 128 x 512 104 for 123; whole steps of
// 47 x 53 x 61 FP32 13 us for 50, of 64^3 FP64 20 for 54.  What bounds it now:
// on 256^3 FP32 it moves 714 MB in and 441 MB out in 227 us cold, 5.1 TB/s or
// 0.79 of the copy rate, where one pass would read 494 MB -- the rest are halo
// lines fetched again (a box is (TR + 2)(NV + 2) vectors and starts one vector
// before a line).  On 192^3 FP32 DRAM runs at 4.5 TB/s cold, issue slots are 29 %
// busy with 2.8 warps a scheduler, waits for loads and copies ahead of
// instruction fetch: the dependent chain of a plane with few warps to hide it,
// which registers and stages bound.  Tried: a warp that only issues copies (a plane 1.05 -> 0.87
// us alone, but its registers cost a resident CTA: 256^3 290 us and more); H
// and E of the plane before reread from shared memory instead of carried (262
// for 303 instructions a warp-plane, same time); unrolling by two planes
// (slower, instruction fetch); 256 threads at 128 registers (290 us).
//
// Periodic x wraps the plane index; periodic y reads the wrapped row through
// one-row boxes behind the tile's.  Every wait is bounded (mbar_wait).
#pragma once
#include "tma.cuh"

namespace rfb {

constexpr int V_NT = 192, V_MB = 2;   // threads a CTA may have, CTAs an SM holds
constexpr int V_NH = 2, V_NE = V_NH + 1;  // H and E stages
template <typename T>
constexpr int V_CELLS = 16 / (int)sizeof(T);  // cells of a vector
constexpr int V_SMEM = 220 * 1024;  // shared memory a CTA may have

// Tensor maps of one buffer parity: (k, j, i, component) with boxes of a
// tile's plane of all three components and, for periodic y, of one row of it.
struct VMaps {
    CUtensorMap e, h, e1, h1;
};

// Shared memory of a CTA from its 128-byte-aligned start: barriers (V_BARS
// bytes), E stages, H stages, then at the offsets of VShape the H rows of the
// plane (x, z; two parities), the vectors' last cells (Hx, Hy; two
// parities), the psi slots and the tables.
constexpr int V_BARS = 128;
__host__ __device__ __forceinline__ int v_e_stage(const VShape &s, int q) { return V_BARS + q * s.estage; }
__host__ __device__ __forceinline__ int v_h_stage(const VShape &s, int q) {
    return V_BARS + V_NE * s.estage + q * s.hstage;
}

// Host entry points (vsweep.cu): shared memory limits of the kernels; one
// launch of the sweep over n items (overlap: see launch_step).
template <typename T>
int v_prepare();
template <typename T>
void v_launch(const Args<T> &a, const VShape &sh, const VItem *items, int n, const VMaps &maps, int *err,
              cudaStream_t st, bool overlap);
// ... over n items of many scenes: CTAs of nt threads, smem bytes for the
// tile and v_args_bytes behind them for the scene's parameters (smem a
// multiple of 16).
template <typename T>
constexpr int v_args_bytes() {
    return (int)((sizeof(Args<T>) + 15) / 16 * 16 + sizeof(VShape));
}
template <typename T>
void v_launch_b(const Args<T> *args, const VShape *shapes, const VMaps *maps, const VItem *items, int n, int nt,
                int smem, int *err, cudaStream_t st, bool overlap);

}  // namespace rfb
