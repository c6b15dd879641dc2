// mpcf_stage.cuh -- the fused LSRK3 stage kernel.
//
// One launch advances every cell of every domain through one low-storage
// RK stage: ghost synthesis from the boundary conditions, WENO5/HLLC face
// fluxes in x, y and z, the non-conservative G/P extra terms, the flux
// divergence with the register update, and the state update.  It replaces
// the reference chain
//   _apply_bc (host) -> _xflux/_xextraterm_hllc -> _yflux/_yextraterm_hllc
//   -> _zflux/_zextraterm_hllc -> _divergence -> _update
// (BoundaryConditions.h:60-109, GPUkernels.cu:35-1179) and its per-stage
// PCIe streaming (GPUlab.cpp:202-372,703-793); all state stays in HBM.
//
// Work decomposition.  A tile is 32 x TY columns in x-y and a z-chunk of
// depth dz.  Warp w owns row w, one thread per column (in the reference forms
// at heights 3, 7 and 15 one more warp takes the tile's rim).  The CTA marches up
// the chunk one slab at a time, two phases and two barriers per slab k:
//   I  the x/y flux differences of cell k-1 (its own faces in registers, the
//      faces right of and above it from the neighbours); z: both edges of
//      cell k, the face k-1/2 from them and the carried upper edge of cell
//      k-1, and with it cell k-1 is finalised:
//      rhs = a*R - dtinvh*div(F) (with the G/P extra terms), R <- rhs,
//      U_next <- b*rhs + U;  then the y and x edges of cell k, and a share of
//      the ghost edges around the tile (rows -1 and TY, columns -1 and 32);
//   II the y face below and the x face left of cell k, two warps the faces
//      above and right of the tile; the next slab's primitives (the cell's
//      own column three slabs up, the tile's halo one slab up) are converted
//      into shared memory.
// Reconstruction is per cell: the three WENO smoothness indicators of a cell
// serve both its edge values (the minus side of the face right of it and the
// plus side of the face left of it), in every direction.  A face's edge
// values and fluxes stay in the registers of the cell above / right of it;
// what the neighbour needs goes through one shuffle in x (the right edge up,
// the flux down) and through one slot of shared memory in y, which holds the
// upper edge of the row below until the face is evaluated and its flux after.
// The G/P sums of the extra terms need only the cell's own six edges.
// Each cell is converted to primitives once per stage (the reference
// converts the six stencil cells again at every face).  The state is
// ping-ponged (read U[parity], write U[parity^1]) so neighbouring tiles
// always see the old state.
//
// Loads.  With TMA (domains whose rows are multiples of 16 bytes; a launch
// covers domains of one kind), three staging buffers in shared memory are filled while a phase is
// worked on, by four bulk tensor copies per slab that one elected thread
// issues: in phase I the halo of the next slab (a 40 x (TY+6) box, whose
// out-of-domain cells are mapped to their mirror / clamp source inside the
// box) and the interior of the slab three ahead, which phase II converts; in
// phase II the register and the state of the plane that the next phase I
// finalises.  Waits on the copies are bounded: a copy that does not complete
// sets an error bit, the CTA stops waiting for copies and carries on (its
// data are then stale, never out of bounds), so a failed copy cannot stall
// the launch.  Otherwise (any domain shape) every thread loads its cells with
// ordinary loads (per-thread cp.async into the staging buffers was 10-19 %
// slower on rows that are no multiples of 16 bytes, prefetching the slabs
// ahead into L1 2 %).  An instance has one of the two: with both, each was
// 2-4 % slower.
//
// DRAM traffic per cell-stage: read U (7 T) + read R (7 T) + write R and
// U_next (14 T) = 112 B in FP32.  Halo and ring re-reads hit L2.
//
// What bounds it: the latency of dependent FP32 operations, with shared
// memory's, at 16 warps per SM (the mixed form, 256^3: 1615 thread-
// instructions per cell-stage in 60 % of the issue slots, FMA pipe 49 %,
// special-function unit 49 % and DRAM 19 % busy; fewer uniform-pipe
// instructions or reciprocals did not help, fewer bank conflicts did).  512^3,
// 32 x 8 tiles, mixed: 27.8 ms a step against 35.0 for one slab pass with
// face slots of 28 planes, three barriers and two-sided fluxes; the parts: two
// phases, faces in registers, quantities in packed pairs, upwind fluxes 32.8;
// halo addresses once per tile 30.6; the row uniform to the compiler 30.0; y
// and x faces as a pair and the register and state by bulk copy 28.9; ghost
// edges in half records 27.8.
#pragma once

#include "mpcf_math.cuh"
#include "mpcf_types.h"

namespace mpcf {

constexpr int kTX = 32;

__host__ __device__ constexpr size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

// 16 bytes of T: the unit of the primitives' shared-memory planes.
template <class T> struct Vec16;
template <> struct Vec16<float>  { typedef float4 V; };
template <> struct Vec16<double> { typedef double2 V; };

__device__ __forceinline__ void unpack(const float4 v, float* q)   { q[0] = v.x; q[1] = v.y; q[2] = v.z; q[3] = v.w; }
__device__ __forceinline__ void unpack(const double2 v, double* q) { q[0] = v.x; q[1] = v.y; }
__device__ __forceinline__ float4  pack(const float* q)  { return make_float4(q[0], q[1], q[2], q[3]); }
__device__ __forceinline__ double2 pack(const double* q) { return make_double2(q[0], q[1]); }

// Shared-memory layout of one CTA.  A record of 8 values (the primitives rho,
// u, v, w, p, G, P and a spare, or a face's 7 fluxes and its velocity) is
// kVecs 16-byte vectors, vector v of every record in plane v, so that a warp
// reads and writes whole records without bank conflicts in kVecs
// instructions.  Inside a plane, in vectors:
//   ring [5 slots][TY][32]   z-ring of the tile's own columns, slabs k-2..k+2
//   cur  [TY+6][38]          slab k with 3-cell x/y halos
//   y    [TY+1][32]          face below row j: the upper edge of the row below
//                            (slot 0: of ghost row -1), then the face's flux
//   top  [32]                lower edge of ghost row TY
//   xg   [TY]                right edge of ghost column -1
//   xr   [TY]                right edge of column 31, then the flux right of it
//   xl   [TY]                left edge of ghost column 32
// then, in bytes: the FP64 reduction scratch [TY][5], the tile broadcast,
// three mbarriers and, with TMA, the staging buffers (128-byte aligned):
//   A     [7][TY+6][40]                   halo box, x from x0-4, y from y0-3
//   B     [7][TY][32]                     interior of a slab
//   C     [2][7][TY][32]                  register and state of the plane
//                                         that is finalised next
template <class T, int TY, bool TMA>
struct StageLayout
{
    static constexpr int kVecs   = 8 * (int)sizeof(T) / 16;
    static constexpr int kPer    = 16 / (int)sizeof(T);    // values per vector
    static constexpr int kCurW   = kTX + 6;                // cur row width
    static constexpr int kRing   = TY * kTX;               // one ring slot
    static constexpr int kCurOff = 5 * kRing;
    static constexpr int kYOff   = kCurOff + (TY + 6) * kCurW;
    static constexpr int kTopOff = kYOff + (TY + 1) * kTX;
    static constexpr int kXgOff  = kTopOff + kTX;
    static constexpr int kXrOff  = kXgOff + TY;
    static constexpr int kXlOff  = kXrOff + TY;
    static constexpr int kPP     = (kXlOff + TY + 7) / 8 * 8;   // plane pitch
    static constexpr int kAW     = kTX + 8;                // staged halo box width
    static constexpr int kAH     = TY + 6;                 // staged halo box height
    static constexpr size_t kRedBytes  = (size_t)kVecs * kPP * 16;
    static constexpr size_t kTileBytes = kRedBytes + sizeof(double) * TY * 5;
    static constexpr size_t kMbarBytes = align_up(kTileBytes + 16, 16);
    static constexpr size_t kABytes    = sizeof(T) * 7 * kAH * kAW;
    static constexpr size_t kBBytes    = sizeof(T) * 7 * TY * kTX;
    static constexpr size_t kStageA    = align_up(kMbarBytes + 32, 128);
    static constexpr size_t kStageB    = align_up(kStageA + kABytes, 128);
    static constexpr size_t kStageC    = align_up(kStageB + kBBytes, 128);
    // + 128: the kernel rounds the dynamic shared-memory base up to 128 B
    static constexpr size_t kBytes     = (TMA ? kStageC + 2 * kBBytes : kMbarBytes + 32) + 128;
};

// Boundary-condition map of one coordinate: absorbing clamps to the edge
// cell, reflecting mirrors (-1-i on the left, 2n-1-i on the right) and
// flips the sign of the normal momentum (BoundaryConditions.h:60-109).
// Halo faces never reach it: the stage sees a slab with its stored ghost
// planes as one extended domain.
__device__ __forceinline__ int bc_map(int i, const int n, const int lo, const int hi, bool& flip)
{
    if (i < 0)       { flip = (lo == BC_REFLECTING); i = flip ? -1 - i : 0; }
    else if (i >= n) { flip = (hi == BC_REFLECTING); i = flip ? 2 * n - 1 - i : n - 1; }
    else             { flip = false; }
    return min(max(i, 0), n - 1);
}

struct DomRegs
{
    int nx, ny, nz;
    int bc0, bc1, bc2, bc3, bc4, bc5;
    long long fs;
};

// Bounds-checking build (MPCF_CHECK_BOUNDS, libmpcf_b200_check.so): every
// computed shared-memory and global index of the stage kernel is checked
// against its region; one outside sets ERRBIT_BOUNDS and is clamped into the
// region, so no access leaves its buffer (the results are then void).
// Without the flag the checks compile to nothing.
#ifdef MPCF_CHECK_BOUNDS
template <class I> __device__ __forceinline__ I in_bounds(const I i, const I lo, const I hi, bool& oob)
{
    if (i < lo || i >= hi) { oob = true; return lo; }
    return i;
}
#define MPCF_IN(i, lo, hi) in_bounds<decltype(i)>((i), (decltype(i))(lo), (decltype(i))(hi), oob)
#else
#define MPCF_IN(i, lo, hi) (i)
#endif

// Load the conserved state of (ix,iy,iz) (any integers: out-of-domain cells
// are synthesised from the boundary conditions) and convert to primitives.
template <class Pol>
__device__ __forceinline__ void load_prim(const DomRegs& D, const typename Pol::T* __restrict__ U,
                                          int ix, int iy, int iz, typename Pol::T q[7], bool& oob)
{
    (void)oob;
    typedef typename Pol::T T;
    bool fx, fy, fz;
    ix = bc_map(ix, D.nx, D.bc0, D.bc1, fx);
    iy = bc_map(iy, D.ny, D.bc2, D.bc3, fy);
    iz = bc_map(iz, D.nz, D.bc4, D.bc5, fz);
    const long long idx = MPCF_IN((long long)ix + (long long)D.nx * ((long long)iy + (long long)D.ny * iz),
                                  0, (long long)D.nx * D.ny * D.nz);
    T c[7];
#pragma unroll
    for (int k = 0; k < 7; ++k) c[k] = __ldg(U + k * D.fs + idx);
    if (fx) c[1] = -c[1];
    if (fy) c[2] = -c[2];
    if (fz) c[3] = -c[3];
    to_primitive<Pol>(c, q);
}

template <class T>
__device__ __forceinline__ bool physical(const T r, const T e, const T G, const T P)
{
    // also false for NaN.  P is only required to be finite: it is 0 in pure
    // gas, and the update leaves round-off there (about -1e-17 in every
    // precision on a bubble cloud).  A state without a real sound speed
    // (p + pc <= 0) is flagged by the sound speed (ERRBIT_SOS).
    return (r > (T)0) && (e > (T)0) && (G > (T)0) && (e < (T)INFINITY) && (r < (T)INFINITY) &&
           (P < (T)INFINITY) && (P > -(T)INFINITY);
}

// ---------------------------------------------------------------------------
// Bulk tensor copies (TMA) and mbarriers, hand-written PTX for sm_100a.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_init_fence()
{
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(bar), "r"(bytes) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}

// Bounded wait for the phase with parity `parity`; false after the limit:
// 2^18 polls, about 1.3 s on the B200 (a copy completes in microseconds).
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity)
{
#pragma unroll 1
    for (int i = 0; i < (1 << 18); ++i)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}

// Prefetch the 128-byte line holding `p` into L1 (no register written).
__device__ __forceinline__ void prefetch_l1(const void* p)
{
    asm volatile("prefetch.global.L1 [%0];" :: "l"(p));
}

// Generic-proxy accesses of this thread before async-proxy (bulk copy)
// accesses that follow: orders shared-memory reuse of a staging buffer.
__device__ __forceinline__ void fence_proxy_async()
{
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// 4-D tile copy global -> shared, completion counted on `bar` (no multicast).
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const void* tmap, int c0, int c1, int c2, int c3, uint32_t bar)
{
    asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
                 " [%0], [%1, {%2, %3, %4, %5}], [%6];"
                 :: "r"(dst), "l"(tmap), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(bar) : "memory");
}

// Warps of one CTA: one per row and, in the reference-rounding forms at
// heights 2^n - 1, a helper warp that owns no column: it reconstructs the ghost
// edges around the tile and evaluates the faces above and right of it.
// Without it 3 rows take 7 ghost edges per warp beside the 21 of its own
// cells, 7 rows 3 and 15 rows 2, and with it the CTA has 2^n warps.  Without
// and with it, us a stage: 3 rows, 240x9x377 FP64 623 and 469, FP32 359 and
// 330; 7 rows, 112x62x128 FP32 304 and 292; 15 rows, 128^3 546 and 512.  (The
// fast forms' reconstruction is too short a share to pay for a warp.)
template <class Pol, int TY> __host__ __device__ constexpr bool stage_helper() { return !Pol::kFastWeno && ((TY + 1) & TY) == 0; }
template <class Pol, int TY> __host__ __device__ constexpr int stage_warps() { return TY + (stage_helper<Pol, TY>() ? 1 : 0); }
template <class Pol, int TY> __host__ __device__ constexpr int stage_threads() { return kTX * stage_warps<Pol, TY>(); }

// Register budget: at least kMinWarpsPerSM resident warps per SM (128
// registers per thread).  The slab's 21 reconstructions are independent, so
// the compiler would otherwise trade occupancy for unbounded
// instruction-level parallelism (239 registers).
// FP64 values take two registers, so its budget is half the warps.
#ifndef MPCF_MIN_WARPS_PER_SM
#define MPCF_MIN_WARPS_PER_SM 16
#endif
template <class Pol, int TY> struct MinBlocks
{
    static constexpr int w = sizeof(typename Pol::T) == 8 ? MPCF_MIN_WARPS_PER_SM / 2 : MPCF_MIN_WARPS_PER_SM;
    static constexpr int v = (w / stage_warps<Pol, TY>()) > 0 ? (w / stage_warps<Pol, TY>()) : 1;
};

// Record `i` (index of its vector in a plane) of 8 values, read / written.
template <class T, int PP>
__device__ __forceinline__ void ld8(const typename Vec16<T>::V* sm, const int i, T q[8])
{
#pragma unroll
    for (int v = 0; v < 8 * (int)sizeof(T) / 16; ++v) unpack(sm[i + v * PP], q + v * (16 / (int)sizeof(T)));
}
template <class T, int PP>
__device__ __forceinline__ void st8(typename Vec16<T>::V* sm, const int i, const T q[8])
{
#pragma unroll
    for (int v = 0; v < 8 * (int)sizeof(T) / 16; ++v) sm[i + v * PP] = pack(q + v * (16 / (int)sizeof(T)));
}

// Both edges of the cell whose stencil records are ad[0..4], all 7
// quantities.  The fast FP32 forms take (rho, u), (v, w) and (p, G) as packed
// pairs and P alone.
template <class Pol, int PP>
__device__ __forceinline__ void weno_record(const typename Vec16<typename Pol::T>::V* sm, const int ad[5],
                                            typename Pol::T R[8], typename Pol::T L[8])
{
    typedef typename Pol::T T;
    constexpr int kPer = 16 / (int)sizeof(T);
    // The FP64 forms take their reciprocals without branches (reference
    // rounding, 256^3: 20.5 against 23.3 ms a step).  In FP32, with half the registers
    // per value, the longer live ranges spill as much as the branches cost
    // (12.34 ms either way, 13.3 without the fences), so it keeps the
    // compiler's division.
    constexpr bool kBranchFree = sizeof(T) == 8 && !Pol::kWeno3;
    bool ok = true;         // every quantity's weights are in that form's range
#pragma unroll
    for (int w = 0; w < 8 / kPer; ++w)
    {
        const int v = Pol::kFastWeno && kPer == 4 ? 1 - w : w;     // (the half record first: fewer spills)
        T y[5][kPer];
#pragma unroll
        for (int j = 0; j < 5; ++j) unpack(sm[ad[j] + v * PP], y[j]);
#pragma unroll
        for (int i = 0; i < kPer; i += (Pol::kFastWeno && kPer == 4) ? 2 : 1)
        {
            const int q = v * kPer + i;
            if (q >= 7) continue;
            if constexpr (Pol::kFastWeno && kPer == 4)
            {
                if (q < 6)
                {
                    float2 r, l;
                    weno_edges<true, false>(make_float2(y[0][i], y[0][i + 1]), make_float2(y[1][i], y[1][i + 1]),
                                     make_float2(y[2][i], y[2][i + 1]), make_float2(y[3][i], y[3][i + 1]),
                                     make_float2(y[4][i], y[4][i + 1]), r, l);
                    R[q] = r.x; R[q + 1] = r.y; L[q] = l.x; L[q + 1] = l.y;
                    continue;
                }
            }
            if constexpr (kBranchFree)
            {
                if constexpr (Pol::kFastWeno) ok &= weno_edges<true, true>(y[0][i], y[1][i], y[2][i], y[3][i], y[4][i], R[q], L[q]);
                else                          ok &= weno_cell_ref<Pol, true>(y[0][i], y[1][i], y[2][i], y[3][i], y[4][i], R[q], L[q]);
                // two quantities at a time: more overlap than this spills
                // (fast form, 256^3: 11.5 ms a step, 13.1 without the fences)
                if (q % 2 == 0) __syncwarp();
            }
            else
                weno_cell<Pol>(y[0][i], y[1][i], y[2][i], y[3][i], y[4][i], R[q], L[q]);
        }
    }
    if constexpr (kBranchFree)
    {
        if (!ok)
        {
            const T* smT = reinterpret_cast<const T*>(sm);
#pragma unroll
            for (int q = 0; q < 7; ++q)
            {
                const int off = q % kPer + q / kPer * (PP * kPer);
                const Edges<T> e = weno_cell_call<Pol>(smT[ad[0] * kPer + off], smT[ad[1] * kPer + off], smT[ad[2] * kPer + off],
                                                       smT[ad[3] * kPer + off], smT[ad[4] * kPer + off]);
                R[q] = e.R;
                L[q] = e.L;
            }
        }
    }
    R[7] = L[7] = (T)0;
}

// Ghost edges of a tile, job g: 0 the right (upper) edges of row -1, 1 the
// left (lower) edges of row TY, 2 the right edges of column -1 (lanes
// 0..TY-1) and the left edges of column 32 (lanes 16..15+TY).  base: the
// stencil's centre record, step: to the next record towards the wanted edge
// (a left edge is the right edge of the mirrored stencil), dst: the record
// that takes the edge; false for the idle lanes.
template <class L, int TY>
__device__ __forceinline__ bool ghost_job(const int g, const int tx, int& base, int& step, int& dst)
{
    if (g == 0)      { base = L::kCurOff + 2 * L::kCurW + tx + 3;        step = L::kCurW;  dst = L::kYOff + tx; }
    else if (g == 1) { base = L::kCurOff + (TY + 3) * L::kCurW + tx + 3; step = -L::kCurW; dst = L::kTopOff + tx; }
    else if (tx < TY)                  { base = L::kCurOff + (tx + 3) * L::kCurW + 2;        step = 1;  dst = L::kXgOff + tx; }
    else if (tx >= 16 && tx < 16 + TY) { base = L::kCurOff + (tx - 13) * L::kCurW + kTX + 3; step = -1; dst = L::kXlOff + tx - 16; }
    else return false;
    return true;
}

template <class Pol, int TY, bool PERSIST, bool SUMS, bool TMA>
__global__ void __launch_bounds__(stage_threads<Pol, TY>(), MinBlocks<Pol, TY>::v)
stage_kernel(const StageArgs A)
{
    typedef typename Pol::T T;
    typedef StageLayout<T, TY, TMA> L;
    // the reference-rounding forms, short of registers, keep the lower y edge
    // from phase I to phase II in the ring slot of slab k-2, free by then
    constexpr bool kStashLy = !Pol::kFastWeno;
    constexpr bool kPairFaces = Pol::kFastWeno && sizeof(T) == 4;   // the y and x faces as one packed pair
    constexpr bool kHelp = stage_helper<Pol, TY>();
    typedef typename Vec16<T>::V V;
    extern __shared__ __align__(16) unsigned char smem_dyn[];
    // 128-byte aligned base (bulk tensor copies need it for their targets)
    unsigned char* smem_raw = smem_dyn + ((128u - (smem_u32(smem_dyn) & 127u)) & 127u);
    V* sm = reinterpret_cast<V*>(smem_raw);
    double* red = reinterpret_cast<double*>(smem_raw + L::kRedBytes);
    int* tile_bc = reinterpret_cast<int*>(smem_raw + L::kTileBytes);
    const uint32_t barA = smem_u32(smem_raw + L::kMbarBytes);
    const uint32_t barB = barA + 8, barC = barA + 16;
    T* stA = reinterpret_cast<T*>(smem_raw + L::kStageA);
    T* stB = reinterpret_cast<T*>(smem_raw + L::kStageB);
    T* stC = reinterpret_cast<T*>(smem_raw + L::kStageC);

    const int tx = threadIdx.x & (kTX - 1);
    // (the shuffle tells the compiler that the row is uniform over the warp)
    const int ty = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    const bool column = !kHelp || ty < TY;     // the warp owns a row of columns
    const T a = (T)A.a;
    const T b = (T)A.b;
    const T factor6 = (T)1.0f / (T)6.0f;   // GPUkernels.cu:1103
    bool ok = true;
    bool oob = false;                      // bounds-checking build: an index left its buffer
    uint32_t phA = 0, phB = 0, phC = 0;    // mbarrier phase parities
    __shared__ T sos_w[TY];                // per-warp maxima of the fused sound speed
    // A thread whose bounded wait runs out sets tma_late and waits for no
    // further copy.  Thread 0 issues every copy; once it has given up it
    // issues none, and before the CTA takes another tile or exits it waits
    // (bounded again) for its copies that no wait of its own has seen
    // complete: pendA/pendB, with the parity of that copy's phase.
    bool tma_late = false;
    bool pendA = false, pendB = false, pendC = false;
    uint32_t parA = 0, parB = 0, parC = 0;
    bool tma_inflight = false;             // a drain wait ran out as well
    // thread 0: one bulk copy of a slab into buffer A or B, with its phase
    // recorded as pending (and counted in failure-detection tests)
    auto issue = [&](const char* tmap, const bool isA, const int c0, const int c1, const int c2)
    {
        if (isA) { mbar_expect_tx(barA, (uint32_t)L::kABytes); tma_load_4d(smem_u32(stA), tmap, c0, c1, c2, 0, barA); pendA = true; parA = phA; }
        else     { mbar_expect_tx(barB, (uint32_t)L::kBBytes); tma_load_4d(smem_u32(stB), tmap + 128, c0, c1, c2, 0, barB); pendB = true; parB = phB; }
        if (A.test_flags) atomicAdd(A.copy_count, 1u);
    };
    // bounded wait of this thread for the copy into buffer A, B or C (0, 1,
    // 2); thread 0 clears the copy's pending mark when it sees it complete
    auto wait_copy = [&](const int which)
    {
        if (tma_late) return;
        const uint32_t bar = which == 0 ? barA : (which == 1 ? barB : barC);
        if (!mbar_wait(bar, which == 0 ? phA : (which == 1 ? phB : phC))) { tma_late = true; return; }
        if (threadIdx.x == 0) { if (which == 0) pendA = false; else if (which == 1) pendB = false; else pendC = false; }
    };

    if (TMA)
    {
        if (threadIdx.x == 0) { mbar_init(barA, 1); mbar_init(barB, 1); mbar_init(barC, 1); mbar_init_fence(); }
        __syncthreads();
    }

    // tiles tile0 .. ntiles-1: from the work counter, or one per CTA
    int t;
    if (PERSIST)
    {
        if (threadIdx.x == 0) *tile_bc = A.tile0 + (int)atomicAdd(A.counter, 1u);
        __syncthreads();
        t = __shfl_sync(0xffffffffu, *tile_bc, 0);
    }
    else t = A.tile0 + blockIdx.x;

    while (t < A.ntiles)
    {
        // ---- decode tile -> domain, tile coordinates
        int d = 0;
        while (d + 1 < A.ndom && (unsigned)(t - A.doms[d].tile_begin) >= (unsigned)A.doms[d].ntiles) ++d;
        const DomDev& DD = A.doms[d];
        // A slab with halo faces is seen as its extended domain, stored
        // ghost planes included (planes -zlo .. nz-1+zhi become 0 ..
        // nz+zlo+zhi-1); only its own planes zlo .. zlo+nz-1 are advanced, so
        // no stencil ever reaches past the stored planes on a halo side.
        DomRegs D;
        D.nx = DD.nx; D.ny = DD.ny; D.nz = DD.nzx;
        D.bc0 = DD.bc[0]; D.bc1 = DD.bc[1]; D.bc2 = DD.bc[2];
        D.bc3 = DD.bc[3]; D.bc4 = DD.bc[4]; D.bc5 = DD.bc[5];
        D.fs = DD.fs;
        const T* __restrict__ U    = (const T*)DD.Ux[A.parity];
        T* __restrict__       Un   = (T*)DD.Ux[A.parity ^ 1];
        T* __restrict__       R    = (T*)DD.Rx;
        const T dtinvh = ((const T*)A.dtinvh)[d];
        constexpr bool use_tma = TMA;
        // tensor maps of the buffer read in this stage (halo box, interior
        // box) and of the register (interior box, own planes only)
        const char* tm = (const char*)A.tmaps + ((size_t)d * 5 + (size_t)A.parity * 2) * 128;
        const char* tmR = (const char*)A.tmaps + ((size_t)d * 5 + 4) * 128;

        const int lt = t - DD.tile_begin;
        const int bx = lt % DD.tiles_x;
        const int by = (lt / DD.tiles_x) % DD.tiles_y;
        const int bz = lt / (DD.tiles_x * DD.tiles_y);
        const int x0 = bx * kTX, y0 = by * TY;
        const int z0 = DD.zlo + bz * A.dz;
        const int z1 = min(z0 + A.dz, DD.zlo + DD.nz);
        const int gx = x0 + tx, gy = y0 + ty;
        const bool valid = column && (gx < D.nx) && (gy < D.ny);
        const int own = ty * kTX + tx;     // own column inside a ring slot
        // the tile's columns are all inside the domain: its ring holds the
        // exact primitives of every cur interior cell
        const bool full = (x0 + kTX <= D.nx) && (y0 + TY <= D.ny);
        // the staged halo box needs no boundary mapping in x and y
        const bool inner = (x0 >= 4) && (x0 + kTX + 4 <= D.nx) && (y0 >= 3) && (y0 + TY + 3 <= D.ny);
        // the own column's record in ring slot r; slab k-2+j is in slot
        // r2 + j modulo 5 with r2 the slot of slab k-2
        auto ring = [&](int r) { r = r < 5 ? r : r - 5; return MPCF_IN(r * L::kRing + own, 0, L::kCurOff); };
        // thread 0: the copies that phase II of slab k converts: the interior
        // of slab k+3 and the halo box of slab k+1
        auto issue_for = [&](const int k)
        {
            bool fz;
            fence_proxy_async();
            // the failure-detection tests arm the barrier of a copy without
            // issuing it: the chunk's last copy, or its first copy after the
            // first slab's (then later waits find the CTA given up, and no
            // further copy is issued)
            const bool drop = !PERSIST && (((A.test_flags & TEST_DROP_LAST_COPY) && k + 1 == z1) ||
                                           ((A.test_flags & TEST_DROP_MID_COPY) && k == z0));
            if (drop) mbar_expect_tx(barB, (uint32_t)L::kBBytes);
            else      issue(tm, false, x0, y0, bc_map(k + 3, D.nz, D.bc4, D.bc5, fz));
            if (k + 1 < z1) issue(tm, true, x0 - 4, y0 - 3, bc_map(k + 1, D.nz, D.bc4, D.bc5, fz));
        };
        // halo cell i (0 .. 6*32 + 6*TY - 1: the cells the x/y stencils read;
        // the corners are never read) at (lx, ly) relative to the tile
        auto halo_place = [&](const int i, int& lx, int& ly)
        {
            if (i < 6 * kTX) { const int r = i >> 5; lx = i & (kTX - 1); ly = r < 3 ? r - 3 : TY + r - 3; }
            else             { const int j = i - 6 * kTX, c = j % 6; ly = j / 6; lx = c < 3 ? c - 3 : kTX + c - 3; }
        };
        // its cell of the staged box (a bulk copy's box holds the domain's own
        // cells), its record in cur and the momenta its boundary condition
        // flips, packed: box | cur << 12 | fx << 30 | fy << 31
        auto halo_cell = [&](const int lx, const int ly, const bool map)
        {
            bool fx = false, fy = false;
            int mx = lx + 4, my = ly + 3;
            if (map)
            {
                const int sx = bc_map(x0 + lx, D.nx, D.bc0, D.bc1, fx), sy = bc_map(y0 + ly, D.ny, D.bc2, D.bc3, fy);
                if (use_tma)
                {
                    mx = min(max(sx - x0 + 4, 0), L::kAW - 1);
                    my = min(max(sy - y0 + 3, 0), L::kAH - 1);
                }
            }
            return (unsigned)(my * L::kAW + mx) | (unsigned)(L::kCurOff + (ly + 3) * L::kCurW + lx + 3) << 12 |
                   (fx ? 1u << 30 : 0u) | (fy ? 1u << 31 : 0u);
        };
        auto convert_halo = [&](const unsigned hc, const int i, const int k)
        {
            T q[8];
            if (use_tma)
            {
                T c[7];
                const int ai = MPCF_IN((int)(hc & 0xfffu), 0, L::kAH * L::kAW);
#pragma unroll
                for (int m = 0; m < 7; ++m) c[m] = stA[m * L::kAH * L::kAW + ai];
                if (hc >> 30 & 1u) c[1] = -c[1];
                if (hc >> 31)      c[2] = -c[2];
                to_primitive<Pol>(c, q);
            }
            else
            {
                int lx, ly;
                halo_place(i, lx, ly);
                load_prim<Pol>(D, U, x0 + lx, y0 + ly, k, q, oob);
            }
            q[7] = (T)0;
            st8<T, L::kPP>(sm, MPCF_IN((int)(hc >> 12 & 0x3ffffu), L::kCurOff, L::kYOff), q);
        };
        // the threads that convert halo cells, and the first two cells of
        // each; in FP64 with bulk copies not the last two warps, which evaluate
        // the faces around the tile in the same phase (fast form, 256^3: 10.8
        // ms a step against 11.1; in FP32 29.6 against 29.1 at 512^3, and
        // slower with ordinary loads)
        constexpr int kHalo = 6 * kTX + 6 * TY, kHaloThreads = kHelp ? stage_threads<Pol, TY>() : (TMA && sizeof(T) == 8 && TY >= 7 ? TY - 2 : TY) * kTX;
        int hlx, hly;
        halo_place(threadIdx.x, hlx, hly);
        const unsigned hc0 = halo_cell(hlx, hly, !inner);
        halo_place(threadIdx.x + kHaloThreads, hlx, hly);
        const unsigned hc1 = halo_cell(hlx, hly, !inner);
        // the own column's cell of a staged interior and the momenta its
        // boundary condition flips
        bool own_fx, own_fy;
        const int own_sx = bc_map(gx, D.nx, D.bc0, D.bc1, own_fx), own_sy = bc_map(gy, D.ny, D.bc2, D.bc3, own_fy);
        const int own_b = use_tma && !full ? min(max(own_sy - y0, 0), TY - 1) * kTX + min(max(own_sx - x0, 0), kTX - 1) : own;
        // without bulk copies: lane l < 28 prefetches a row piece for the
        // finalisation: field l % 7 of R / U, first / second line
        const T* pf = U;
        if (!use_tma)
        {
            const int f = tx % 7, w = tx / 7;
            pf = ((w & 1) ? U : (const T*)R) + f * D.fs - (long long)D.nx * D.ny + (long long)D.nx * min(gy, D.ny - 1) + min(x0 + ((w & 2) ? 31 : 0), D.nx - 1);
        }
        if (use_tma && threadIdx.x == 0 && !tma_late) issue_for(z0 - 1);

        // ---- prologue: slabs z0-3 .. z0+1 of the own column into the ring
        if (column)
        {
#pragma unroll
            for (int j = 0; j < 5; ++j)
            {
                T q[8];
                load_prim<Pol>(D, U, gx, gy, z0 - 3 + j, q, oob);
                q[7] = (T)0;
                st8<T, L::kPP>(sm, ring(j), q);
            }
        }

        // carried from slab to slab: the z face below, the upper z edge and
        // the x/y faces left of / below the cell, the G/P sums of its edges
        T zfp[8], Rz[8], Fx[8], Fy[8];
        T sG = 0, sP = 0;
#pragma unroll
        for (int m = 0; m < 8; ++m) { zfp[m] = 0; Rz[m] = 0; Fx[m] = 0; Fy[m] = 0; }
        double cs[5] = {0, 0, 0, 0, 0};
        T smax = 0;              // fused sound speed of the new state (last stage)
        bool sbad = false;

        // slab z0-1 gives its upper z edge only
        int r2 = 0;
#pragma unroll 1
        for (int k = z0 - 1; ; ++k)
        {
            const bool xy = k >= z0 && k < z1;     // slab k has x and y faces
            // the staging buffers are free again (phase II of slab k-1 is
            // behind the barrier): copy while this slab is worked on
            if (use_tma) { if (threadIdx.x == 0 && !tma_late && xy) issue_for(k); }
            else if (column && k > z0 && tx < 28) prefetch_l1(pf + (long long)D.nx * D.ny * k);

            // ---- phase I
            const bool fin = (k > z0) && valid;
#ifdef MPCF_CHECK_BOUNDS
            // cell k-1 of the own column: inside the domain's own planes
            const long long idx = fin ? MPCF_IN((long long)gx + (long long)D.nx * ((long long)gy + (long long)D.ny * (k - 1)),
                                                (long long)DD.zlo * DD.nx * DD.ny, (long long)(DD.zlo + DD.nz) * DD.nx * DD.ny)
                                      : 0;
#else
            const long long idx = (long long)gx + (long long)D.nx * ((long long)gy + (long long)D.ny * (k - 1));
#endif
            // x/y part of cell k-1: its own faces, the face right of it from
            // the next lane (or the tile's extra face) and the face above it
            // from its slot
            T S[7], dU = 0;
#pragma unroll
            for (int m = 0; m < 7; ++m) S[m] = 0;
            if (column && k > z0)
            {
                T Fr[8], Fa[8];
#pragma unroll
                for (int m = 0; m < 8; ++m) Fr[m] = __shfl_down_sync(0xffffffffu, Fx[m], 1);
                if (tx == kTX - 1) ld8<T, L::kPP>(sm, L::kXrOff + ty, Fr);
                ld8<T, L::kPP>(sm, L::kYOff + own + kTX, Fa);
#pragma unroll
                for (int m = 0; m < 7; ++m)
                {
                    if constexpr (Pol::kFastWeno) S[m] = (Fr[m] - Fx[m]) + (Fa[m] - Fy[m]);
                    else                          S[m] = ((Fr[m] - Fx[m]) + Fa[m]) - Fy[m];
                }
                dU = (Fr[7] - Fx[7]) + (Fa[7] - Fy[7]);
            }
            // z: both edges of cell k, the face k-1/2, and cell k-1's
            // finalisation: rhs = a*R - dtinvh*div(F) (with the G/P extra
            // terms), R <- rhs, U_next <- b*rhs + U
            T Rv[8], Lv[8];
            if (column)
            {
                int ad[5];
#pragma unroll
                for (int j = 0; j < 5; ++j) ad[j] = ring(r2 + j);
                weno_record<Pol, L::kPP>(sm, ad, Rv, Lv);
            }
            if (column && k >= z0)
            {
                T zf[8];
                face_hllc<Pol>(Rz, Lv, 2, zf);
                if (use_tma && k > z0)
                {
                    wait_copy(2);
                    phC ^= 1;
                }
                if (fin)
                {
                    T Rold[7], Uold[7];
#pragma unroll
                    for (int m = 0; m < 7; ++m)
                    {
                        Rold[m] = use_tma ? stC[m * L::kRing + own] : R[m * D.fs + idx];
                        Uold[m] = use_tma ? stC[(7 + m) * L::kRing + own] : __ldg(U + m * D.fs + idx);
                    }
                    const T divU = dU + (zf[7] - zfp[7]);
                    T un[7];
#pragma unroll
                    for (int m = 0; m < 7; ++m)
                    {
                        T br;
                        if constexpr (Pol::kFastWeno) br = S[m] + (zf[m] - zfp[m]);
                        else                          br = (S[m] + zf[m]) - zfp[m];
                        if (m == 5) br = br - divU * sG * factor6;
                        if (m == 6) br = br - divU * sP * factor6;
                        const T rhs_m = dtinvh * br;
                        const T rhs = a * Rold[m] - rhs_m;
                        R[m * D.fs + idx] = rhs;
                        un[m] = b * rhs + Uold[m];
                        Un[m * D.fs + idx] = un[m];
                    }
                    ok = ok && physical<T>(un[0], un[4], un[5], un[6]);
                    if (A.sos_bits)
                    {
                        const T v = cell_sos_rn<Pol>(un[0], un[1], un[2], un[3], un[4], un[5], un[6]);
                        sbad = sbad || !(v >= (T)0);   // NaN (the maximum would drop it) or negative
                        smax = dmax(smax, v);
                    }
                    if (SUMS)
                    {
#pragma unroll
                        for (int m = 0; m < 5; ++m) cs[m] += (double)un[m];
                    }
                }
#pragma unroll
                for (int m = 0; m < 8; ++m) zfp[m] = zf[m];
            }
            if (k == z1) break;
            if (column)
            {
#pragma unroll
                for (int m = 0; m < 8; ++m) Rz[m] = Rv[m];
            }

            T Ly[8], Rx[8], Lx[8];
#pragma unroll
            for (int m = 0; m < 8; ++m) { Ly[m] = 0; Rx[m] = 0; Lx[m] = 0; }
            if (xy)
            {
                // y, then x edges of the own cell.  The fast forms unroll the
                // two; the reference-rounding forms, whose reconstruction is
                // five times the code, keep one copy.
                // (The helper warp's three ghost jobs go through that copy.)
                T szG = 0, szP = 0, syG = 0, syP = 0;
                if (column) { szG = Lv[5] + Rv[5]; szP = Lv[6] + Rv[6]; }
                constexpr int kXYUnroll = Pol::kFastWeno ? 2 : 1;
                const int nj = column ? 2 : 3;
#pragma unroll kXYUnroll
                for (int j = 0; j < nj; ++j)
                {
                    int step = j ? 1 : L::kCurW;
                    int base = L::kCurOff + (ty + 3) * L::kCurW + tx + 3;
                    int dst = -1;
                    bool lower = false;         // (a ghost job's) wanted edge: the left or lower one
                    if (kHelp && !column)
                    {
                        base = L::kCurOff + 2 * L::kCurW + tx + 3;      // (the idle lanes')
                        if (ghost_job<L, TY>(j, tx, base, step, dst)) { lower = step < 0; step = lower ? -step : step; }
                    }
                    int ad[5];
#pragma unroll
                    for (int i = 0; i < 5; ++i) ad[i] = MPCF_IN(base + (i - 2) * step, L::kCurOff, L::kYOff);
                    weno_record<Pol, L::kPP>(sm, ad, Rv, Lv);
                    if (kHelp && !column)
                    {
#pragma unroll
                        for (int m = 0; m < 7; ++m) Rv[m] = lower ? Lv[m] : Rv[m];
                        if (dst >= 0) st8<T, L::kPP>(sm, MPCF_IN(dst, L::kYOff, L::kPP), Rv);
                    }
                    else if (j == 0)
                    {
                        st8<T, L::kPP>(sm, L::kYOff + own + kTX, Rv);
                        if constexpr (kStashLy) st8<T, L::kPP>(sm, ring(r2), Lv);
#pragma unroll
                        for (int m = 0; m < 7; ++m) Ly[m] = Lv[m];
                        syG = Lv[5] + Rv[5];
                        syP = Lv[6] + Rv[6];
                    }
                    else
                    {
                        if (tx == kTX - 1) st8<T, L::kPP>(sm, L::kXrOff + ty, Rv);
#pragma unroll
                        for (int m = 0; m < 7; ++m) { Rx[m] = Rv[m]; Lx[m] = Lv[m]; }
                        sG = ((Lv[5] + Rv[5]) + syG) + szG;
                        sP = ((Lv[6] + Rv[6]) + syP) + szP;
                    }
                }
                // ghost edges around the tile, shared evenly by the warps
                const T* smT = reinterpret_cast<const T*>(sm);
                T* smTw = reinterpret_cast<T*>(sm);
                if constexpr (Pol::kFastWeno && sizeof(T) == 4)
                {
                    // 12 jobs: the pairs (rho, u), (v, w), (p, G) and P alone
                    // of each of the 3 of ghost_job (the stencil's pairs are
                    // half a record: half the loads and bank conflicts of one
                    // quantity on two sides)
#pragma unroll 1
                    for (int e = ty; e < 12; e += TY)
                    {
                        int base, step, dst;
                        if (!ghost_job<L, TY>(e >> 2, tx, base, step, dst)) continue;
                        const int q = 2 * (e & 3), off = (q & 3) + (q >> 2) * (L::kPP * 4);
                        int ad[5];
#pragma unroll
                        for (int i = 0; i < 5; ++i) ad[i] = MPCF_IN(base + (i - 2) * step, L::kCurOff, L::kYOff) * 4 + off;
                        const int at = MPCF_IN(dst, L::kYOff, L::kPP) * 4 + off;
                        if (q < 6)
                        {
                            float2 y[5], r, l;
#pragma unroll
                            for (int i = 0; i < 5; ++i) y[i] = *reinterpret_cast<const float2*>(smT + ad[i]);
                            weno_edges<false, false>(y[0], y[1], y[2], y[3], y[4], r, l);
                            *reinterpret_cast<float2*>(smTw + at) = r;
                        }
                        else
                        {
                            float r, l;
                            weno_edges<false, false>(smT[ad[0]], smT[ad[1]], smT[ad[2]], smT[ad[3]], smT[ad[4]], r, l);
                            smTw[at] = r;
                        }
                    }
                }
                else if constexpr (!kHelp)
                {
                    // 21 jobs (3 of ghost_job x 7 quantities) in contiguous
                    // ranges over the warps
                    constexpr int kPer = 21 / TY, kRem = 21 % TY;
                    int gi = ty * kPer + (ty < kRem ? ty : kRem);
                    const int ge = gi + kPer + (ty < kRem ? 1 : 0);
#pragma unroll 1
                    for (; gi < ge; ++gi)
                    {
                        const int g = gi >= 14 ? 2 : (gi >= 7 ? 1 : 0);
                        const int q = gi - 7 * g;
                        int base, step, dst;
                        if (!ghost_job<L, TY>(g, tx, base, step, dst)) continue;
                        const int off = q % L::kPer + q / L::kPer * (L::kPP * L::kPer);
                        // the reference's two edges are not mirror images bit
                        // for bit: those forms take the cells left to right
                        const int st = Pol::kFastWeno ? step : (step < 0 ? -step : step);
                        T y[5], rv, lv;
#pragma unroll
                        for (int i = 0; i < 5; ++i) y[i] = smT[MPCF_IN(base + (i - 2) * st, L::kCurOff, L::kYOff) * L::kPer + off];
                        if constexpr (Pol::kFastWeno)
                        {
                            // (a mirrored stencil's left edge is its right edge)
                            if (!weno_edges<false, true>(y[0], y[1], y[2], y[3], y[4], rv, lv))
                                rv = weno_cell_call<Pol>(y[0], y[1], y[2], y[3], y[4]).R;
                            lv = rv;
                        }
                        else                          weno_cell<Pol>(y[0], y[1], y[2], y[3], y[4], rv, lv);
                        smTw[MPCF_IN(dst, L::kYOff, L::kPP) * L::kPer + off] = step > 0 ? rv : lv;
                    }
                }
                __syncthreads();

                // the register and state of plane k, for phase I of slab k+1
                // (plane k-1's were last read before the barrier)
                if (use_tma && threadIdx.x == 0 && !tma_late)
                {
                    fence_proxy_async();
                    mbar_expect_tx(barC, 2 * (uint32_t)L::kBBytes);
                    if (PERSIST || !((A.test_flags & TEST_DROP_PLANE_COPY) && k == z0))
                    {
                        tma_load_4d(smem_u32(stC), tmR, x0, y0, k - DD.zlo, 0, barC);
                        tma_load_4d(smem_u32(stC + 7 * L::kRing), tm + 128, x0, y0, k, 0, barC);
                        pendC = true;
                        parC = phC;
                    }
                }
                // ---- phase II: the y face below and the x face left of the
                // own cell; the last two warps (the helper warp, where there
                // is one) the y faces above the tile and the x faces right of it
                if constexpr (kPairFaces)
                {
                    T my[8], mx[8];
                    ld8<T, L::kPP>(sm, L::kYOff + own, my);
#pragma unroll
                    for (int q = 0; q < 7; ++q) mx[q] = __shfl_up_sync(0xffffffffu, Rx[q], 1);
                    mx[7] = (T)0;
                    if (tx == 0) ld8<T, L::kPP>(sm, L::kXgOff + ty, mx);
                    face_hllc_yx(my, Ly, mx, Lx, Fy, Fx);
                    if (ty > 0) st8<T, L::kPP>(sm, L::kYOff + own, Fy);
                }
                constexpr int kFaceUnroll = Pol::kFastWeno ? 3 : 1;
#pragma unroll kFaceUnroll
                for (int j = kPairFaces || !column ? 2 : 0; j < (kHelp ? (column ? 2 : 4) : 3); ++j)
                {
                    if (!kHelp && j == 2 && ty < TY - 2) break;
                    T m[8], p[8], f[8];
                    int dir, dst = -1;
                    if (j == 0)
                    {
                        ld8<T, L::kPP>(sm, L::kYOff + own, m);
                        if constexpr (kStashLy) ld8<T, L::kPP>(sm, ring(r2), p);
                        else
                        {
#pragma unroll
                            for (int q = 0; q < 8; ++q) p[q] = Ly[q];
                        }
                        dir = 1;
                        if (ty > 0) dst = L::kYOff + own;
                    }
                    else if (j == 1)
                    {
#pragma unroll
                        for (int q = 0; q < 7; ++q) { m[q] = __shfl_up_sync(0xffffffffu, Rx[q], 1); p[q] = Lx[q]; }
                        m[7] = p[7] = (T)0;
                        if (tx == 0) ld8<T, L::kPP>(sm, L::kXgOff + ty, m);
                        dir = 0;
                    }
                    else if (kHelp ? j == 2 : ty == TY - 1)
                    {
                        dst = L::kYOff + TY * kTX + tx;
                        ld8<T, L::kPP>(sm, dst, m);
                        ld8<T, L::kPP>(sm, L::kTopOff + tx, p);
                        dir = 1;
                    }
                    else
                    {
                        if (tx >= TY) continue;
                        dst = L::kXrOff + tx;
                        ld8<T, L::kPP>(sm, dst, m);
                        ld8<T, L::kPP>(sm, L::kXlOff + tx, p);
                        dir = 0;
                    }
                    face_hllc<Pol>(m, p, dir, f);
                    if (j == 0)
                    {
#pragma unroll
                        for (int q = 0; q < 8; ++q) Fy[q] = f[q];
                    }
                    if (j == 1)
                    {
#pragma unroll
                        for (int q = 0; q < 8; ++q) Fx[q] = f[q];
                    }
                    if (dst >= 0) st8<T, L::kPP>(sm, MPCF_IN(dst, L::kYOff, L::kPP), f);
                }
            }

            // slab k+3 of the own column
            if (column)
            {
                if (use_tma) { wait_copy(1); phB ^= 1; }
                T q[8];
                if (use_tma)
                {
                    bool fz;
                    bc_map(k + 3, D.nz, D.bc4, D.bc5, fz);
                    T c[7];
                    const int bi = MPCF_IN(own_b, 0, L::kRing);
#pragma unroll
                    for (int m = 0; m < 7; ++m) c[m] = stB[m * L::kRing + bi];
                    if (own_fx) c[1] = -c[1];
                    if (own_fy) c[2] = -c[2];
                    if (fz) c[3] = -c[3];
                    to_primitive<Pol>(c, q);
                }
                else load_prim<Pol>(D, U, gx, gy, k + 3, q, oob);
                q[7] = (T)0;
                st8<T, L::kPP>(sm, ring(r2), q);   // in place of slab k-2
            }
            // slab k+1 with halos into cur (k+1 < z1: no z mapping)
            if (k + 1 < z1)
            {
                const bool box = use_tma && !full;
                if (!box && column)
                {
                    // interior from the ring
                    T q[8];
                    ld8<T, L::kPP>(sm, ring(r2 + 3), q);
                    st8<T, L::kPP>(sm, MPCF_IN(L::kCurOff + (ty + 3) * L::kCurW + tx + 3, L::kCurOff, L::kYOff), q);
                }
                if (use_tma)
                {
                    wait_copy(0);
                    phA ^= 1;
                }
                // the 6*32 + 6*TY halo cells the x/y stencils read (the
                // corners are never read); a tile reaching past the domain
                // converts the whole staged box, its out-of-domain cells
                // mapped to their sources
                if (box)
                {
                    for (int i = threadIdx.x; i < (TY + 6) * L::kCurW; i += stage_threads<Pol, TY>())
                    {
                        const int ly = i / L::kCurW - 3, lx = i % L::kCurW - 3;
                        convert_halo(halo_cell(lx, ly, true), 0, k + 1);
                    }
                }
                else if (threadIdx.x < (kHaloThreads < kHalo ? kHaloThreads : kHalo))
                {
                    convert_halo(hc0, threadIdx.x, k + 1);
                    if (threadIdx.x + kHaloThreads < kHalo) convert_halo(hc1, threadIdx.x + kHaloThreads, k + 1);
                    for (int i = threadIdx.x + 2 * kHaloThreads; i < kHalo; i += kHaloThreads)
                    {
                        int lx, ly;
                        halo_place(i, lx, ly);
                        convert_halo(halo_cell(lx, ly, !inner), i, k + 1);
                    }
                }
            }
            r2 = r2 < 4 ? r2 + 1 : 0;
            __syncthreads();
        }

        // ---- fused sound-speed maximum of the tile into its domain's
        // accumulator (the stand-alone reduction's order of the bits)
        if (A.sos_bits)
        {
            const bool bad = __syncthreads_or(sbad);
            const T m = shfl_max(smax);
            if (tx == 0 && column) sos_w[ty] = m;
            __syncthreads();
            if (threadIdx.x < 32)
            {
                T mm = threadIdx.x < TY ? sos_w[threadIdx.x] : (T)0;
                mm = shfl_max(mm);
                if (threadIdx.x == 0) atomic_max_bits((char*)A.sos_bits + (size_t)d * sizeof(T), bad ? (T)NAN : mm);
            }
        }

        // ---- per-tile FP64 conservation sums (deterministic: fixed order)
        if (SUMS)
        {
#pragma unroll
            for (int m = 0; m < 5; ++m)
            {
                double v = cs[m];
#pragma unroll
                for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
                if (tx == 0 && column) red[ty * 5 + m] = v;
            }
            __syncthreads();
            if (threadIdx.x < 5)
            {
                double v = 0;
                for (int w = 0; w < TY; ++w) v += red[w * 5 + threadIdx.x];
                A.tile_sums[(long long)t * 5 + threadIdx.x] = v;
            }
        }

        // copies this CTA issued and no wait of thread 0 saw complete (only
        // after a wait ran out): wait for them, bounded, so that none lands
        // in shared memory the CTA no longer owns; a CTA that gave up takes
        // no further tile
        if (TMA && threadIdx.x == 0 && (pendA || pendB || pendC))
        {
            if (pendA && !mbar_wait(barA, parA)) tma_inflight = true;
            if (pendB && !mbar_wait(barB, parB)) tma_inflight = true;
            if (pendC && !mbar_wait(barC, parC)) tma_inflight = true;
            pendA = pendB = pendC = false;
        }
        if (!PERSIST) break;
        __syncthreads();
        if (threadIdx.x == 0) *tile_bc = tma_late ? A.ntiles : A.tile0 + (int)atomicAdd(A.counter, 1u);
        __syncthreads();
        t = __shfl_sync(0xffffffffu, *tile_bc, 0);
    }

    if (!__all_sync(0xffffffffu, ok) && tx == 0) atomicOr(A.err, (unsigned)ERRBIT_NONPHYSICAL);
    if (TMA && tma_late) atomicOr(A.err, (unsigned)ERRBIT_TMA_TIMEOUT);
    if (TMA && tma_inflight) atomicOr(A.err, (unsigned)ERRBIT_TMA_INFLIGHT);
#ifdef MPCF_CHECK_BOUNDS
    if (__any_sync(0xffffffffu, oob) && tx == 0) atomicOr(A.err, (unsigned)ERRBIT_BOUNDS);
#endif
}

template <class Pol, int TY, bool TMA>
constexpr size_t stage_smem_bytes() { return StageLayout<typename Pol::T, TY, TMA>::kBytes; }

} // namespace mpcf
