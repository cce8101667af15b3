// Structured-grid triangular sweeps (k_sweep_grid).
//
// Used when a factor's pattern is exactly a 5- or 7-point grid stencil in
// natural order (TriFactor's grid layout, detected at preconditioner
// set-up); other factors keep the chunked and flat sweeps.  The arithmetic
// of a row is k_sweep's, entry for entry: rr = v[r]; rr -= a * w for the
// row's off-diagonal entries in the reference's storage order; w[r] = rr *
// dia (boost/numeric/mtl/operation/lower_trisolve.hpp:174-209,
// upper_trisolve.hpp:161-176).  Only the schedule differs:
//  - a lane owns one x-line and runs its rows in x order; a warp holds 8 x 4
//    lines of neighbouring y and z (7-point) or 32 of neighbouring y
//    (5-point), lane (a, b) running row i at step i + a + b: the x neighbour
//    is the lane's own previous result (a register), the y and z neighbours
//    are other lanes' results of the previous step (two warp shuffles);
//  - a CTA runs the warps of one tile (2 x NW/2 warps, or NW along y).  A
//    compute warp does nothing but the steps: it leaves its results in a
//    shared ring, row by row of 32 lanes, and publishes its step count every
//    kGridH steps; the warps at its upper y and z sides read their missing
//    neighbours from that ring;
//  - a helper warp per compute warp moves everything else: factor values by
//    bulk copies (TMA), right-hand sides by cp.async and results from the
//    ring to the output vector, both 8 consecutive rows of a line at a time
//    (a lane per line would touch 32 sectors per instruction);
//  - results on a tile's upper y and z sides also go, step by step, to a
//    hand-off buffer in global memory (TriFactor::ghalo, all sentinel between
//    sweeps), where the next tile's receiver warps poll them, fill a ring of
//    the same form and put the sentinel back.
// What bounds it: the dependency chain (nx + ny + nz steps and the hand-offs
// between warps and tiles), not bytes; a step costs one shuffle, a row's
// arithmetic and the shared-memory accesses that feed it.  Measured (one
// B200, apply = L + U sweep, queued): FP32 ILU(0) 128^3 439 -> 225 us, 2048^2
// 1,990 -> 692 us, FP64 128^3 773 -> 304 us against the previous kernel (one
// warp per 32 lines and plane, every lane moving its own line's right-hand
// sides, results and resets: 32 sectors per instruction, ~300 ns a step).
// Tiles are taken through one ticket in an order in which every tile a tile
// reads comes earlier, and a tile runs to its end on a running CTA.  Inside a
// tile a warp waits on lower warps by at most two blocks of steps and on
// upper ones only when a ring of four blocks is full, so the waits end; every
// wait is still bounded (the context's spin_limit polls), after which the
// kernel records a timeout and drains.
// The same kernel computes the FP64 pivots of an ILU(0) or IC(0)
// factorization of a grid-stencil pattern (OPK kGridILU0 / kGridIC0): a
// row's pivot needs its earlier neighbours' pivots exactly as an L sweep's
// row needs their results (boost/numeric/itl/pc/ilu_0.hpp:45-82,
// ic_0.hpp:124-186, with k_ilu0_factor's and k_ic0_factor's roundings).
#pragma once
#include "sweep.cuh"

#include <climits>

namespace mtlg {

constexpr int kGridG = 8;                    // steps per staged block
constexpr int kGridNB = 4;                   // staged blocks per warp (factor values and right-hand sides)
constexpr int kGridRing = kGridG * kGridNB;  // rows of a ring (right-hand sides, results)
constexpr int kGridH = 4;                    // steps between hand-offs inside a CTA
constexpr int kGridTell = 5;                 // lanes that publish a step count (own, two readers, two writers)
constexpr int kGridRecvWarps = 2;            // receiver warps: z sides, y sides
constexpr int kGridDiagRows = 8192;          // rows per tile of a factor without entries
static_assert(kGridStepPad % kGridG == 0, "layout padding must hold whole staged blocks");
static_assert(kGridG % kGridH == 0, "hand-offs split a block evenly");

// Row operations of the grid kernel: a triangular sweep, or the FP64 pivots
// of an ILU(0) or IC(0) factorization (the same dependencies: a row's pivot
// needs its three earlier neighbours' pivots).
constexpr int kGridSweep = 0, kGridILU0 = 1, kGridIC0 = 2;
// Slots per step (capacity): a sweep's entries and multiplier fit four; an
// ILU(0) pivot reads its L entries, the neighbours' entries in its column and
// its diagonal (up to seven).
__host__ __device__ constexpr int grid_cap(int opk) { return opk == kGridILU0 ? 7 : 4; }

// Elements between ring rows: 32 lanes and a pad that spreads the helper's
// accesses (8 rows x 4 or 2 lines at once) over all banks.
template <typename T>
__host__ __device__ constexpr int grid_pitch() { return sizeof(T) == 4 ? 36 : 34; }

// Warp and tile shapes of a stencil with NS off-diagonal entries per row.
template <int NW, int NS>
struct GridShapeOf {
    static constexpr int LY = NS == 3 ? kGridLY3 : 32, LZ = NS == 3 ? 32 / kGridLY3 : 1;   // lines per warp
    static constexpr int WY = NS == 3 ? 2 : NW, WZ = NS == 3 ? NW / 2 : 1;                 // warps per tile
    static constexpr int TY = LY * WY, TZ = LZ * WZ;                                       // lines per tile
    static constexpr int SKEW = LY + LZ - 2;                                               // of a warp's last lane
    static constexpr int ZCOLS = NS == 3 ? TY : 0;   // receiver ring columns of the z lines (first), then the y lines
};

// Dynamic shared memory of a k_sweep_grid CTA of nw compute warps: factor
// blocks, right-hand-side ring and result ring per warp, the receiver's ring.
template <typename T, typename S, int OPK = kGridSweep>
__host__ __device__ constexpr int grid_smem_bytes(int nw)
{
    const int ring = kGridRing * grid_pitch<T>() * int(sizeof(T));
    return nw * (kGridRing * grid_cap(OPK) * 32 * int(sizeof(S)) + (OPK == kGridSweep ? 2 : 1) * ring) + ring;
}

// Slot orders the kernel runs (TriFactor::gperm): the farthest neighbour's
// entry first (z, y, x / y, x: rows stored by ascending column from below),
// or the nearest first (x, y, z / x, y).
constexpr int kGridFar3 = 2 | (1 << 2) | (0 << 4);
constexpr int kGridNear3 = 0 | (1 << 2) | (2 << 4);
constexpr int kGridFar2 = 1 | (0 << 2);
constexpr int kGridNear2 = 0 | (1 << 2);

// Values of one 16-byte group of a step's slots: sweeps of 7-point factors
// keep a lane's four values together (one or two 16-byte shared loads a
// step), the other layouts slot by slot.
__host__ __device__ constexpr int grid_pack(int slots, int ssz) { return slots == 4 ? 16 / ssz : 1; }
// Offset of a lane's slot q inside a step.
__host__ __device__ inline int grid_slot(int pk, int q, int lane) { return (q / pk) * (32 * pk) + lane * pk + q % pk; }

// Hand-off rows between tiles: what a warp at a tile's upper z side leaves
// at each step in its LY upper lines, [tile along z][unit along y][step][LY],
// then at the upper y side, [tile along y][unit along z][step][LZ].
inline size_t grid_halo_elems(int steps, int njb, int nkb, int ny, int nz, int ty, int tz, bool three)
{
    const int ly = three ? kGridLY3 : 32, lz = 32 / ly;
    return ((three ? size_t((nz + tz - 1) / tz) * njb * ly : 0) + size_t((ny + ty - 1) / ty) * nkb * lz) * size_t(steps);
}

// VN consecutive elements (16 bytes, or one) of a hand-off row, each checked on its own.
template <int VN>
__device__ __forceinline__ void ld_row(const float* p, float (&v)[VN])
{
    if constexpr (VN == 4) ld_relaxed_gpu4(p, v);
    else v[0] = ld_relaxed_gpu(p);
}
template <int VN>
__device__ __forceinline__ void ld_row(const double* p, double (&v)[VN])
{
    if constexpr (VN == 2)
        asm volatile("ld.relaxed.gpu.global.v2.f64 {%0, %1}, [%2];" : "=d"(v[0]), "=d"(v[1]) : "l"(p));
    else v[0] = ld_relaxed_gpu(p);
}
__device__ __forceinline__ void st_sentinel_vec(void* p)
{
    asm volatile("st.global.v4.u32 [%0], {%1, %1, %1, %1};" ::"l"(p), "r"(0xFFFFFFFFu) : "memory");
}

// Shared memory by 32-bit address (the roles pick their rings at run time;
// generic pointers would cost two registers and a generic access each).
__device__ __forceinline__ void lds(unsigned a, float& v) { asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a)); }
__device__ __forceinline__ void lds(unsigned a, double& v) { asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a)); }
__device__ __forceinline__ void sts(unsigned a, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v)); }
__device__ __forceinline__ void sts(unsigned a, double v) { asm volatile("st.shared.f64 [%0], %1;" ::"r"(a), "d"(v)); }
__device__ __forceinline__ void bulk_g2s_to(unsigned dst, const void* src, unsigned bytes, unsigned long long* bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void lds_vec(unsigned a, float* v)
{
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "r"(a));
}
__device__ __forceinline__ void lds_vec(unsigned a, double* v)
{
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v[0]), "=d"(v[1]) : "r"(a));
}
template <int VN>
__device__ __forceinline__ void sts_row(unsigned a, const float (&v)[VN])
{
    if constexpr (VN == 4)
        asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]));
    else sts(a, v[0]);
}
template <int VN>
__device__ __forceinline__ void sts_row(unsigned a, const double (&v)[VN])
{
    if constexpr (VN == 2) asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(a), "d"(v[0]), "d"(v[1]));
    else sts(a, v[0]);
}
// Copies BYTES, or fills them with zeros (nothing is read then).
template <int BYTES>
__device__ __forceinline__ void cp_async_to(unsigned a, const void* gmem, bool copy)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(a), "l"(gmem), "n"(BYTES), "r"(copy ? BYTES : 0)
                 : "memory");
}

// Step counts published inside the CTA: everything the publishing warp
// stored before is visible to a warp that has read the count.
__device__ __forceinline__ void grid_count(unsigned p, int v)
{
    asm volatile("st.release.cta.shared.u32 [%0], %1;" ::"r"(p), "r"(v) : "memory");
}
__device__ __forceinline__ int grid_read(unsigned p)
{
    int v;
    asm volatile("ld.relaxed.cta.shared.u32 %0, [%1];" : "=r"(v) : "r"(p) : "memory");
    return v;
}
// After reading a count: what its writer stored before is visible from here on.
__device__ __forceinline__ void grid_acquire() { asm volatile("fence.acq_rel.cta;" ::: "memory"); }
// Whether a warp's bounded wait ends without its value: after lim polls
// (recorded as a timeout), or when another wait has expired.  Decided by all
// lanes together, every lane having counted the same polls: the waits below
// and what follows them use warp-wide votes.  A wait of more than kGridQuick
// polls (some 3 ms in shared memory, longer than the chain of a wave of tiles
// takes to come by) naps between them: it leaves the issue slots to the others,
// and the default limit stays about half a second whatever a poll costs (2^20
// polls of shared memory alone: some 40 ms).  Napping from 4,096 polls on found
// a waiting tile's rows late (FP64, lines of 2 rows, 782 tiles in a chain:
// applies of 16.8 ms instead of 16.1).
constexpr long long kGridQuick = 1 << 16;
__device__ __forceinline__ bool grid_give_up(long long& spins, int* err, long long lim)
{
    const bool over = ++spins > (lim > 0 ? lim : kSpinLimit);
    if (!over && (spins & 255) != 0) {
        if (spins > kGridQuick) __nanosleep(500);
        return false;
    }
    if (over) atomicExch(err, 1);
    return __any_sync(0xffffffffu, over || *(volatile int*)err);
}
// Waits until the count reaches `need` (on expiry the warp goes on with
// whatever the rings hold).
__device__ __forceinline__ void grid_wait(unsigned p, int need, int* err, long long lim)
{
    long long spins = 0;
    while (__any_sync(0xffffffffu, grid_read(p) < need))
        if (grid_give_up(spins, err, lim)) break;
    __syncwarp();
    grid_acquire();
}
// A compute warp's four counts, kept in one 16-byte slot that the other warps
// write into: steps done by the writers of its y and z neighbours' rows and by
// the readers of its own.
struct GridCounts {
    int y, z, yfree, zfree;
};
__device__ __forceinline__ GridCounts grid_counts(unsigned p)
{
    GridCounts c;
    asm volatile("ld.volatile.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(c.y), "=r"(c.z), "=r"(c.yfree), "=r"(c.zfree) : "r"(p) : "memory");
    return c;
}
// A staged block's barrier (own copies: a fixed bound, given up early once a
// wait has expired; the helper waits for every copy before the tile ends).
__device__ __forceinline__ void grid_bar_wait(unsigned long long* bar, unsigned parity, int* err)
{
    int spins = 0;
    while (!mbar_try_wait(bar, parity)) {
        if ((++spins & 255) == 0 && *(volatile int*)err) return;
        if (spins > 2 * int(kSpinLimit)) {
            atomicExch(err, 1);
            return;
        }
    }
}
// Whether the barrier's phase is over, without waiting.
__device__ __forceinline__ bool mbar_test(unsigned long long* bar, unsigned parity)
{
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// The thread's earlier cp.async copies arrive on the barrier when they land.
__device__ __forceinline__ void cp_async_arrive(unsigned long long* bar)
{
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// Shared-memory addresses of a tile's parts.
struct GridSmem {
    unsigned stage, rings;            // factor blocks, rings (per warp: results, right-hand sides; then the receiver's)
    unsigned prog;                    // step counts of the compute warps (and a cell nobody reads)
    unsigned slots;                   // GridCounts of the compute warps
    unsigned long long* full;         // the staged blocks' barriers, kGridNB per warp
    unsigned* blks;                   // staged blocks each warp has gone through before this tile
};

// What a compute warp works with (addresses of the lane's column where per lane).
template <typename T>
struct GridWarp {
    unsigned stage, rhs, ring;        // staged factor blocks, right-hand-side ring, result ring
    unsigned yin, zin;                // the y and z neighbours' columns (lanes at the warp's lower sides; no neighbour: a column of +0)
    unsigned slot;                    // own GridCounts
    int cy, cz, cyf, czf;             // what they have to exceed the next half's first step by (INT_MIN: nobody to wait for)
    unsigned tell;                    // lanes below kGridTell: where the own step count goes
    unsigned long long* full;
    T* yhalo;                         // the lane's place in the hand-off row of step 0
    T* zhalo;
    unsigned blk;
    int nx, nblk, lane;
    bool lane_on;
    bool yface, zface;                // the lane writes hand-off rows
    int* err;
    long long spin;
};

// Operands of kGridH steps of a lane: right-hand sides, neighbours' values
// (lanes at the warp's lower sides), factor values.
template <typename T, typename S, int SL>
struct GridHalf {
    T rr[kGridH], yv[kGridH], zv[kGridH];
    S a[kGridH][SL];
};

// The steps of one compute warp's unit.  NS entries per row, FAR: the
// farthest neighbour's entry first (z, y, x; else x, y, z).  While kGridH
// steps run, the next ones' operands are loaded, a few per step (a burst of
// shared loads would delay the shuffles behind it): factor values and
// right-hand sides always, the neighbours' values when their writers' counts,
// read at the start, already cover them; else they are waited for at the end.
// A warp that has to wait falls behind until it no longer does, so the pace
// is the chain of a step: shuffle, select, multiply, subtractions, multiply.
// A sweep needs no validity tests: outside a lane's line factor values,
// right-hand sides and so results are +0 (an absent neighbour).
template <typename T, typename S, int NW, int NS, bool FAR, int OPK>
__device__ __forceinline__ void grid_compute(const GridWarp<T>& g)
{
    typedef GridShapeOf<NW, NS> Sh;
    typedef typename std::conditional<(sizeof(S) > sizeof(T)), S, T>::type W;   // promoted type
    constexpr int G = kGridG, H = kGridH;
    static_assert(G == 2 * H, "a block is two halves");
    constexpr unsigned P = grid_pitch<T>() * sizeof(T);                         // bytes between ring rows
    constexpr int SL = OPK == kGridILU0 ? 2 * NS + 1 : NS + 1;                  // slots per step
    constexpr int PK = grid_pack(SL, int(sizeof(S)));
    constexpr unsigned SB = 32 * SL * sizeof(S);                                // bytes per step
    const int ly = g.lane % Sh::LY, lz = g.lane / Sh::LY;
    const int total = g.nblk * G;
    const bool ey = ly == 0, ez = lz == 0;
    GridHalf<T, S, SL> A, B;
    auto own = [&](GridHalf<T, S, SL>& d, int u, unsigned row, unsigned e) {   // step u's own operands
        d.rr[u] = T(0);
        if (OPK == kGridSweep) lds(g.rhs + row + u * P, d.rr[u]);
        if constexpr (PK > 1) {
#pragma unroll
            for (int k = 0; k < SL; k += PK) lds_vec(e + u * SB + k * (32 * unsigned(sizeof(S))), &d.a[u][k]);
        } else {
#pragma unroll
            for (int k = 0; k < SL; ++k) lds(e + u * SB + k * (32 * unsigned(sizeof(S))), d.a[u][k]);
        }
    };
    // step u's neighbours' values in the half at step 8 m + h: ring row of that
    // step + LY - 1 (LZ - 1), in block m, m + 1 or (LY 32) m + 3, m + 4
    auto near = [&](GridHalf<T, S, SL>& d, int u, int h, unsigned r0, unsigned r1, unsigned r3, unsigned r4) {
        constexpr int DY = (Sh::LY - 1) % G, BY = (Sh::LY - 1) / G, DZ = Sh::LZ - 1;
        static_assert((BY == 0 || BY == 3) && DZ < G, "8 or 32 lines along y");
        const int y = h + u + DY, z = h + u + DZ;
        lds(g.yin + (y < G ? (BY ? r3 : r0) : (BY ? r4 : r1)) + (y % G) * P, d.yv[u]);
        d.zv[u] = T(0);
        if (NS == 3) lds(g.zin + (z < G ? r0 : r1) + (z % G) * P, d.zv[u]);
    };
    auto ready = [&](const GridCounts& c, int s) { return c.y - s >= g.cy && c.z - s >= g.cz; };   // for the half at step s
    auto room = [&](const GridCounts& c, int s) { return c.yfree - s >= g.cyf && c.zfree - s >= g.czf; };   // for its results
    auto wait_for = [&](auto test, int s) {
        long long spins = 0;
        while (__any_sync(0xffffffffu, !test(grid_counts(g.slot), s)))
            if (grid_give_up(spins, g.err, g.spin)) break;
        __syncwarp();
        grid_acquire();
    };
    auto ringrow = [&](int m) { return unsigned((m * G) & (kGridRing - 1)) * P; };
    // result of the last step, and the y and z lower lanes' (+0 before a lane's first row)
    T out = T(0), sy = T(0), sz = T(0);
    T* yh = g.yhalo;
    T* zh = g.zhalo;
    // half h (0 or H) of block m from c's operands; the next half's into n
    auto half = [&](GridHalf<T, S, SL>& c, GridHalf<T, S, SL>& n, int m, auto hc, unsigned enext, bool more) {
        constexpr int h = decltype(hc)::value, hn = H - h;
        const int s0 = m * G + h, s1 = s0 + H, mn = h == 0 ? m : m + 1;
        const unsigned row = ringrow(m) + h * P, rown = ringrow(mn) + hn * P;
        const unsigned r0 = ringrow(mn), r1 = ringrow(mn + 1), r3 = NS == 3 ? 0u : ringrow(mn + 3), r4 = r0;   // ring of four blocks
        const GridCounts cnt = grid_counts(g.slot);
        T o[H];
#pragma unroll
        for (int u = 0; u < H; ++u) {
            const T wx = out, wy = ey ? c.yv[u] : sy, wz = ez ? c.zv[u] : sz;
            const S* e = c.a[u];
            T acc = OPK == kGridSweep ? c.rr[u] : T(e[SL - 1]);   // a pivot starts from a_ii
            if constexpr (OPK == kGridILU0) {
                // k_ilu0_factor on a grid stencil: per earlier neighbour k
                // (ascending column) l = a_ik / u_kk (rounded), u_ii -= l a_ki
                // (fused); L's entries and the other U entries do not change
                if (NS == 3) acc = __fma_rn(-__dmul_rn(e[0], wz), e[NS], acc);
                acc = __fma_rn(-__dmul_rn(e[NS - 2], wy), e[2 * NS - 2], acc);
                acc = __fma_rn(-__dmul_rn(e[NS - 1], wx), e[2 * NS - 1], acc);
            } else if constexpr (OPK == kGridIC0) {
                // k_ic0_factor: d = a_ki / sqrt(u_kk) (rounded), u_ii -= d d
                // (rounded product), per earlier neighbour k ascending
                T d;
                if (NS == 3) {
                    d = __dmul_rn(e[0], wz);
                    acc = __dsub_rn(acc, __dmul_rn(d, d));
                }
                d = __dmul_rn(e[NS - 2], wy);
                acc = __dsub_rn(acc, __dmul_rn(d, d));
                d = __dmul_rn(e[NS - 1], wx);
                acc = __dsub_rn(acc, __dmul_rn(d, d));
            } else if constexpr (FAR) {
                if (NS == 3) acc = sweep_step<T, S>(acc, e[0], wz);
                acc = sweep_step<T, S>(acc, e[NS - 2], wy);
                acc = sweep_step<T, S>(acc, e[NS - 1], wx);
            } else {
                acc = sweep_step<T, S>(acc, e[0], wx);
                acc = sweep_step<T, S>(acc, e[1], wy);
                if (NS == 3) acc = sweep_step<T, S>(acc, e[2], wz);
            }
            if constexpr (OPK == kGridSweep) {
                out = T(W(acc) * W(e[NS]));
            } else {
                // outside its line a lane's pivot is +0, as an absent neighbour's
                const bool valid = g.lane_on && unsigned(s0 + u - ly - lz) < unsigned(g.nx);
                if constexpr (OPK == kGridILU0) out = T(__ddiv_rn(1.0, double(acc)));
                else out = T(__ddiv_rn(1.0, __dsqrt_rn(double(acc))));
                out = valid ? out : T(0);
            }
            o[u] = out;
            sy = __shfl_up_sync(0xffffffffu, out, 1);
            if (NS == 3) sz = __shfl_up_sync(0xffffffffu, out, Sh::LY);
            // (after the last block: stale shared memory, never used)
            own(n, u, rown, enext);
            if (u == 0) grid_acquire();
            if (u > 0) near(n, u - 1, hn, r0, r1, r3, r4);
            if (u == H - 1) near(n, u, hn, r0, r1, r3, r4);
        }
        // (voted: lanes may have read the counts at different times)
        const bool ok = __all_sync(0xffffffffu, ready(cnt, s1) && room(cnt, s1));
        // the rows these results go to held those of a whole ring of steps ago
        if (!ok) wait_for(room, s1);
#pragma unroll
        for (int u = 0; u < H; ++u) sts(g.ring + row + u * P, o[u]);
        __syncwarp();
        if (g.lane < kGridTell) grid_count(g.tell, s1 < total ? s1 : INT_MAX);
        if (g.yface) {
#pragma unroll
            for (int u = 0; u < H; ++u) st_relaxed_gpu(yh + u * Sh::LZ, unsentinel(o[u]));
        }
        yh += H * Sh::LZ;
        if (NS == 3) {
            if (g.zface) {
#pragma unroll
                for (int u = 0; u < H; ++u) st_relaxed_gpu(zh + u * Sh::LY, unsentinel(o[u]));
            }
            zh += H * Sh::LY;
        }
        if (more && !ok) {
            wait_for(ready, s1);
#pragma unroll
            for (int u = 0; u < H; ++u) near(n, u, hn, r0, r1, r3, r4);
        }
    };
    auto block = [&](int m) { return g.stage + ((g.blk + unsigned(m)) % kGridNB) * (G * SB); };
    auto bar = [&](int m) {
        const unsigned q = g.blk + unsigned(m);
        grid_bar_wait(&g.full[q % kGridNB], (q / kGridNB) & 1u, g.err);
    };
    bar(0);
#pragma unroll
    for (int u = 0; u < H; ++u) own(A, u, 0u, block(0));
    wait_for(ready, 0);
#pragma unroll
    for (int u = 0; u < H; ++u) near(A, u, 0, ringrow(0), ringrow(1), NS == 3 ? 0u : ringrow(3), ringrow(0));
#pragma unroll 1
    for (int m = 0; m < g.nblk; ++m) {
        const unsigned q = g.blk + unsigned(m) + 1;
        const bool more = m + 1 < g.nblk, landed = mbar_test(&g.full[q % kGridNB], (q / kGridNB) & 1u);
        half(A, B, m, std::integral_constant<int, 0>(), block(m) + H * SB, true);
        if (more && !landed) bar(m + 1);
        half(B, A, m, std::integral_constant<int, H>(), block(m + 1), more);
    }
}

// A helper warp: thread t moves element t % 8 of lines t / 8 + 4 q, block by
// block of a compute warp's steps (line l of block m: the rows of its steps
// 8 m .. 8 m + 7, consecutive in x).
template <typename T, typename S, int NW, int NS, bool REV, int OPK>
__device__ __forceinline__ void grid_help(const S* src, unsigned stage, const T* vin, T* vout, unsigned rhs, unsigned ring,
                                          unsigned prog, unsigned long long* full, unsigned blk, int n, int nx,
                                          int ny, int nz, int j0, int k0, int nblk, int lane, int* err, long long spin)
{
    typedef GridShapeOf<NW, NS> Sh;
    constexpr int G = kGridG;
    constexpr unsigned P = grid_pitch<T>() * sizeof(T);
    constexpr int SL = OPK == kGridILU0 ? 2 * NS + 1 : NS + 1;
    constexpr int BE = G * SL * 32;   // elements per staged block
    const int xo = lane & 7, l0 = lane >> 3;
    // the thread's element of line l0 + 4 q in block m: x = x0[q] + 8 m,
    // vector index at[q] + (8 m or -8 m); kept in registers, since this
    // warp's instructions bound the pace of its compute warp
    int x0[8], at[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int a = (l0 + 4 * q) % Sh::LY, c = (l0 + 4 * q) / Sh::LY;
        const int r = nx * (j0 + a + ny * (k0 + c)) + xo - a - c;
        x0[q] = j0 + a < ny && k0 + c < nz ? xo - a - c : INT_MIN / 2;   // no such line: never inside
        at[q] = REV ? n - 1 - r : r;
    }
    auto fetch = [&](int m) {
        const unsigned c = blk + unsigned(m), b = c % kGridNB;
        if (lane == 0) {
            mbar_expect_tx(&full[b], unsigned(BE * int(sizeof(S))));
            bulk_g2s_to(stage + b * unsigned(BE * sizeof(S)), src + size_t(m) * BE, unsigned(BE * int(sizeof(S))), &full[b]);
        }
        if (OPK == kGridSweep) {
            const unsigned cell = rhs + (((m * G) & (kGridRing - 1)) + xo) * P + l0 * unsigned(sizeof(T));
            const int x = m * G, o = REV ? -x : x;
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const bool in = unsigned(x0[q] + x) < unsigned(nx);
                cp_async_to<sizeof(T)>(cell + 4 * q * unsigned(sizeof(T)), vin + (in ? at[q] + o : 0), in);
            }
        }
        cp_async_arrive(&full[b]);
    };
    for (int m = 0; m < kGridNB && m < nblk; ++m) fetch(m);
#pragma unroll 1
    for (int m = 0; m < nblk; ++m) {
        grid_wait(prog, (m + 1) * G, err, spin);
        const unsigned cell = ring + (((m * G) & (kGridRing - 1)) + xo) * P + l0 * unsigned(sizeof(T));
        T v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) lds(cell + 4 * q * unsigned(sizeof(T)), v[q]);
        __syncwarp();   // every lane has its results before the ring rows are released with the block
        if (m + kGridNB < nblk) {
            // block m's copies have landed (the compute warp has used them; an
            // expired wait may have come here early)
            const unsigned c = blk + unsigned(m);
            mbar_wait(&full[c % kGridNB], (c / kGridNB) & 1u, err);
            fetch(m + kGridNB);
        }
        const int x = m * G, o = REV ? -x : x;
#pragma unroll
        for (int q = 0; q < 8; ++q)
            if (unsigned(x0[q] + x) < unsigned(nx)) vout[at[q] + o] = OPK == kGridSweep ? v[q] : unsentinel(v[q]);
    }
    // every copy of the tile has landed (also after an expired wait)
    for (int m = max(0, nblk - kGridNB); m < nblk; ++m) {
        const unsigned c = blk + unsigned(m);
        mbar_wait(&full[c % kGridNB], (c / kGridNB) & 1u, err);
    }
}

// A receiver warp: polls the hand-off rows of up to NG warps of earlier
// tiles (`src`: rows of WD elements, one per step), puts each complete prefix
// of rows into its ring (columns col + WD g) with the sentinel back in its
// place, and publishes the count of rows there (group g is read by compute
// warp g * step: its count at `reader`, its slot's at `count`).  A thread holds VN elements
// (16 bytes) of a row, so a group's poll is one coalesced load or a few; sleep_ns
// (the context's "sweep_sleep_ns") passes between polls that brought nothing.
template <typename T, int WD, int NG>
__device__ __forceinline__ void grid_receive(T* const (&src)[NG], int total, unsigned ring, int col, unsigned count,
                                             unsigned reader, int step, int slack, int lane, int* err, long long spin,
                                             int sleep_ns)
{
    constexpr int VN = WD * int(sizeof(T)) >= 16 ? 16 / int(sizeof(T)) : 1;   // elements per thread
    constexpr int TR = WD / VN;                                              // threads per row
    constexpr int RL = 32 / TR;                                              // rows per load
    constexpr int NL = RL >= 16 ? 1 : 16 / RL;                               // loads per poll (at least 16 rows)
    static_assert(VN == 1 ? WD == 1 : WD % VN == 0, "a row is whole vectors");
    constexpr unsigned P = grid_pitch<T>() * sizeof(T);
    const int tr = lane / TR, tc = (lane % TR) * VN;
    int c[NG];   // rows delivered per group (warp-uniform)
    unsigned left = 0;
#pragma unroll
    for (int g = 0; g < NG; ++g) {
        c[g] = src[g] ? 0 : total;
        if (src[g]) left |= 1u << g;
    }
    long long spins = 0;
#pragma unroll 1
    while (left) {
        T v[NG][NL][VN];
#pragma unroll
        for (int g = 0; g < NG; ++g)
#pragma unroll
            for (int l = 0; l < NL; ++l) {
                const int r = c[g] + l * RL + tr;
                if (((left >> g) & 1u) && r < total) ld_row<VN>(src[g] + size_t(r) * WD + tc, v[g][l]);
            }
        bool moved = false;
#pragma unroll
        for (int g = 0; g < NG; ++g) {
            if (!((left >> g) & 1u)) continue;
            const int room = grid_read(reader + 4 * step * g) + slack + kGridRing;   // rows below this are free
            grid_acquire();
            int rows = 0;
            bool go = true;
#pragma unroll
            for (int l = 0; l < NL; ++l) {
                const int r = c[g] + l * RL + tr;
                bool ok = r < total && r < room;
#pragma unroll
                for (int e = 0; e < VN; ++e) ok = ok && !is_sentinel(v[g][l][e]);
                // complete rows before the first that is not
                const unsigned bad = ~__ballot_sync(0xffffffffu, ok);
                const int got = !go ? 0 : bad ? (__ffs(bad) - 1) / TR : RL;
                if (tr < got) {
                    T* p = src[g] + size_t(r) * WD + tc;
                    sts_row<VN>(ring + unsigned(r & (kGridRing - 1)) * P + unsigned(col + WD * g + tc) * unsigned(sizeof(T)), v[g][l]);
                    if constexpr (VN > 1) st_sentinel_vec(p);
                    else *p = sentinel_value<T>();
                }
                rows += got;
                go = got == RL;
            }
            if (rows > 0) {
                moved = true;
                c[g] += rows;
                __syncwarp();
                if (lane == 0) grid_count(count + 16 * step * g, c[g] < total ? c[g] : INT_MAX);
                if (c[g] >= total) left &= ~(1u << g);
            }
        }
        if (moved) {
            spins = 0;   // the limit is one wait's, not the tile's
            continue;
        }
        if (grid_give_up(spins, err, spin)) break;
        if (sleep_ns > 0) __nanosleep(sleep_ns);
    }
    __syncwarp();
    // after an expired wait nobody waits on these rows any more
    if (left && lane == 0)
        for (int g = 0; g < NG; ++g) grid_count(count + 16 * step * g, INT_MAX);
}

// The roles of one tile's warps (NS and FAR from the factor).  Not inlined:
// with the four variants in one body the compiler keeps values of all of
// them alive (96 registers and 370 bytes of spills instead of 80 and none).
template <typename T, typename S, int NW, int NS, bool FAR, bool REV, int OPK>
__device__ __noinline__ void grid_tile(const TriFactor& F, int n, const T* vin, T* vout, int ty, int tz,
                                          const GridSmem& sm, int warp, int lane, int* err, long long spin, int sleep_ns)
{
    typedef GridShapeOf<NW, NS> Sh;
    constexpr unsigned P = grid_pitch<T>() * sizeof(T), TS = sizeof(T);
    constexpr int SL = OPK == kGridILU0 ? 2 * NS + 1 : NS + 1;
    constexpr unsigned RB = kGridRing * P;                              // bytes of a ring
    constexpr unsigned RW = (OPK == kGridSweep ? 2 : 1) * RB;           // rings of one warp: results, right-hand sides
    constexpr unsigned SE = kGridRing * grid_cap(OPK) * 32 * sizeof(S); // staged bytes of one warp
    const int nx = F.gnx, ny = F.gny, nz = F.gnz, njb = F.gnjb, nkb = (nz + Sh::LZ - 1) / Sh::LZ;
    const int nblk = F.gnsp / kGridG, total = F.gnsp;
    const int ntz = NS == 3 ? (nz + Sh::TZ - 1) / Sh::TZ : 0;
    T* zh = static_cast<T*>(F.ghalo);                                    // [tile along z][unit along y][step][LY]
    T* yh = zh + size_t(ntz) * njb * total * Sh::LY;                     // [tile along y][unit along z][step][LZ]
    const unsigned rring = sm.rings + NW * RW;   // the receivers' (z columns, then y columns)
    if (warp == 2 * NW) {
        if constexpr (NS == 3) {
            T* src[Sh::WY];
#pragma unroll
            for (int a = 0; a < Sh::WY; ++a) {
                const int ju = ty * Sh::WY + a;
                src[a] = tz > 0 && ju < njb ? zh + (size_t(tz - 1) * njb + ju) * total * Sh::LY : nullptr;
            }
            grid_receive<T, Sh::LY, Sh::WY>(src, total, rring, 0, sm.slots + 4, sm.prog, 1, Sh::LZ - 1, lane, err, spin,
                                               sleep_ns);
        }
        return;
    }
    if (warp > 2 * NW) {
        T* src[Sh::WZ];
#pragma unroll
        for (int a = 0; a < Sh::WZ; ++a) {
            const int ku = tz * Sh::WZ + a;
            src[a] = ty > 0 && ku < nkb ? yh + (size_t(ty - 1) * nkb + ku) * total * Sh::LZ : nullptr;
        }
        grid_receive<T, Sh::LZ, Sh::WZ>(src, total, rring, Sh::ZCOLS, sm.slots, sm.prog, Sh::WY, Sh::LY - 1, lane, err, spin,
                                           sleep_ns);
        return;
    }
    const int w = warp % NW, wy = w % Sh::WY, wz = w / Sh::WY;
    const int ju = ty * Sh::WY + wy, ku = tz * Sh::WZ + wz;
    if (ju >= njb || ku >= nkb) return;
    const int j0 = ju * Sh::LY, k0 = ku * Sh::LZ;
    const unsigned blk = sm.blks[w], ring = sm.rings + w * RW;
    if (warp >= NW) {
        const S* src = static_cast<const S*>(F.gdata) + (size_t(ku) * njb + ju) * size_t(F.gnsp) * size_t(SL) * 32;
        grid_help<T, S, NW, NS, REV, OPK>(src, sm.stage + w * SE, vin, vout, ring + RB, ring, sm.prog + 4 * w,
                                          sm.full + w * kGridNB, blk, n, nx, ny, nz, j0, k0, nblk, lane, err, spin);
        return;
    }
    const int ly = lane % Sh::LY, lz = lane / Sh::LY, j = j0 + ly, k = k0 + lz;
    GridWarp<T> g;
    constexpr int PK = grid_pack(SL, int(sizeof(S)));
    g.stage = sm.stage + w * SE + lane * unsigned(PK * sizeof(S));
    g.rhs = ring + RB + lane * TS;
    g.ring = ring + lane * TS;
    const bool has_y = ju > 0, has_z = NS == 3 && ku > 0;
    const unsigned zero = rring + 32 * TS;   // the receivers' ring keeps its first pad column +0
    g.yin = !has_y ? zero : wy > 0 ? ring - RW + (Sh::LY - 1 + Sh::LY * lz) * TS : rring + (Sh::ZCOLS + wz * Sh::LZ + lz) * TS;
    g.zin = !has_z ? zero : wz > 0 ? ring - Sh::WY * RW + (Sh::LY * (Sh::LZ - 1) + ly) * TS : rring + (wy * Sh::LY + ly) * TS;
    // the half at step s reads its neighbours' rows of steps below s + kGridH
    // + LY - 1 (LZ - 1); results of steps below s replace rows that readers
    // have left once they are past s - kGridRing - (LY - 1)
    const bool yr = wy + 1 < Sh::WY && ju + 1 < njb, zr = wz + 1 < Sh::WZ && ku + 1 < nkb;
    g.slot = sm.slots + 16 * w;
    g.cy = has_y ? kGridH + Sh::LY - 1 : INT_MIN;
    g.cz = has_z ? kGridH + Sh::LZ - 1 : INT_MIN;
    g.cyf = yr ? -kGridRing - (Sh::LY - 1) : INT_MIN;
    g.czf = zr ? -kGridRing - (Sh::LZ - 1) : INT_MIN;
    g.tell = lane == 0 ? sm.prog + 4 * w
             : lane == 1 && yr ? sm.slots + 16 * (w + 1)
             : lane == 2 && zr ? sm.slots + 16 * (w + Sh::WY) + 4
             : lane == 3 && wy > 0 ? sm.slots + 16 * (w - 1) + 8
             : lane == 4 && wz > 0 ? sm.slots + 16 * (w - Sh::WY) + 12
                                   : sm.prog + 4 * NW;
    g.full = sm.full + w * kGridNB;
    g.lane_on = j < ny && k < nz;
    g.yface = wy == Sh::WY - 1 && ju + 1 < njb && ly == Sh::LY - 1;
    g.zface = NS == 3 && wz == Sh::WZ - 1 && ku + 1 < nkb && lz == Sh::LZ - 1;
    g.yhalo = yh + (size_t(ty) * nkb + ku) * total * Sh::LZ + lz;
    g.zhalo = zh + (size_t(tz) * njb + ju) * total * Sh::LY + ly;
    g.blk = blk;
    g.nx = nx;
    g.nblk = nblk;
    g.lane = lane;
    g.err = err;
    g.spin = spin;
    grid_compute<T, S, NW, NS, FAR, OPK>(g);
}

// One sweep over the grid tiles of a set of systems.  op.tasks: GroupTask
// {sys, tile along y, tile along z}; of a factor without entries (NS 0, its
// multipliers in row order) {sys, first of kGridDiagRows rows / kGridDiagRows}.
template <typename T, typename S, int NW, bool REV, int OPK = kGridSweep>
__global__ void __launch_bounds__(32 * (2 * NW + kGridRecvWarps), 1) k_sweep_grid(SetView sv, ChunkSweepOp op)
{
    constexpr int NTH = 32 * (2 * NW + kGridRecvWarps);
    typedef typename std::conditional<(sizeof(S) > sizeof(T)), S, T>::type W;   // promoted type
    if (blockDim.x != unsigned(NTH) || op.which != int(REV)) {   // launch shape mismatch: report, never wait
        if (threadIdx.x == 0) atomicExch(sv.err, 1);
        return;
    }
    extern __shared__ __align__(128) unsigned char grid_smem[];
    __shared__ __align__(8) unsigned long long full[NW * kGridNB];
    __shared__ int s_task, s_go;
    __shared__ int prog[NW + 1];
    __shared__ __align__(16) int slots[4 * NW];
    __shared__ unsigned blks[NW];
    constexpr int SE = kGridRing * grid_cap(OPK) * 32;
    GridSmem sm;
    sm.stage = smem_u32(grid_smem);
    sm.rings = sm.stage + unsigned(NW * SE * int(sizeof(S)));
    sm.prog = smem_u32(prog);
    sm.slots = smem_u32(slots);
    sm.full = full;
    sm.blks = blks;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        // 32 cp.async arrivals of the helper's threads and its bulk copy
        for (int b = 0; b < NW * kGridNB; ++b) mbar_init(&full[b], 33);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (tid < NW) blks[tid] = 0;
    if (tid < kGridRing) {
        // the pad column that stands for absent neighbours
        const unsigned rw = (OPK == kGridSweep ? 2u : 1u) * unsigned(kGridRing * grid_pitch<T>() * int(sizeof(T)));
        sts(sm.rings + NW * rw + unsigned(tid * grid_pitch<T>() + 32) * unsigned(sizeof(T)), T(0));
    }
    __syncthreads();
    for (;;) {
        if (tid == 0) {
            const int t = atomicAdd(op.ticket, 1);
            if (t == op.ntasks + int(gridDim.x) - 1) atomicExch(op.ticket, 0);
            s_task = t;
            s_go = t < op.ntasks && !skip_system(sv.st[op.tasks[t].sys], op.skip) && !*(volatile int*)sv.err;
        }
        if (tid >= 32 && tid < 32 + 4 * NW) slots[tid - 32] = 0;
        if (tid >= 64 && tid < 64 + NW) prog[tid - 64] = 0;
        __syncthreads();
        const int t = s_task;
        if (t >= op.ntasks) break;
        if (s_go) {
            const GroupTask gt = op.tasks[t];
            const SysDesc& d = sv.desc[gt.sys];
            const TriFactor& F = op.which == 0 ? d.L : d.U;
            const int n = d.n, ns = F.gns, ty = gt.pos0, tz = gt.count;
            const T* vin = OPK == kGridSweep ? vptr<T>(d, op.in) : nullptr;
            T* vout = vptr<T>(d, op.out);
            if (OPK == kGridSweep && ns == 0) {
                const S* dia = static_cast<const S*>(F.gdata);
                const int e = min(n, (ty + 1) * kGridDiagRows);
                for (int r = ty * kGridDiagRows + tid; r < e; r += NTH) vout[r] = unsentinel(T(W(vin[r]) * W(dia[r])));
            } else if (ns == 3) {
                if (OPK != kGridSweep || F.gperm == kGridFar3)
                    grid_tile<T, S, NW, 3, true, REV, OPK>(F, n, vin, vout, ty, tz, sm, warp, lane, sv.err, sv.spin, op.sleep_ns);
                else
                    grid_tile<T, S, NW, 3, false, REV, OPK>(F, n, vin, vout, ty, tz, sm, warp, lane, sv.err, sv.spin, op.sleep_ns);
            } else {
                if (OPK != kGridSweep || F.gperm == kGridFar2)
                    grid_tile<T, S, NW, 2, true, REV, OPK>(F, n, vin, vout, ty, tz, sm, warp, lane, sv.err, sv.spin, op.sleep_ns);
                else
                    grid_tile<T, S, NW, 2, false, REV, OPK>(F, n, vin, vout, ty, tz, sm, warp, lane, sv.err, sv.spin, op.sleep_ns);
            }
            __syncthreads();   // every warp has read its block count
            if (tid < NW && ns > 0) {
                // the blocks its warp went through keep the barriers' parity
                const int wyn = ns == 3 ? 2 : NW;
                const int lz = ns == 3 ? 32 / kGridLY3 : 1, wzn = ns == 3 ? NW / 2 : 1;
                const int ju = ty * wyn + tid % wyn, ku = tz * wzn + tid / wyn;
                if (ju < F.gnjb && ku < (F.gnz + lz - 1) / lz) blks[tid] += unsigned(F.gnsp / kGridG);
            }
        }
        __syncthreads();
    }
}

// Grid layout values straight from the matrix's CSR (no per-element index
// arrays): element (unit, step, slot, lane) is row r's entry of the slot's
// direction, found in A's row, with the sources and pivot rows of the
// preconditioner's factor row lists -- ILU(0): the entry (r, c) of the
// factorized values, no pivot; IC(0): L's (r, c) is a_cr times the inverse
// pivot of c, U's (r, c) is a_rc times the inverse pivot of r -- and the
// multiplier slot the inverse pivot of r (1 for a unit diagonal); padding +0.
// The same values and roundings as k_fill_grid and the chunked layout's fill.
// lmul: ILU(0) factorized on the grid (A's values in `src`): L's entries are
// a_rc times the inverse pivot of c, as k_ilu0_factor forms them.
struct GridFillGeom {
    int n, nx, ny, nz, ns, perm, nsp, njb;
    int pk;   // grid_pack of the layout's slots
};
// Element e of a grid layout with `slots` slots per step: its slot, its row
// r' (counted from the sweep's start) and the row's grid coordinates; false
// for padding.  (A factor without entries holds its multipliers in row order.)
struct GridElem {
    int q, i, j, k;
    long long r;
};
__host__ __device__ inline bool grid_elem(const GridFillGeom& g, int slots, long long e, GridElem& o)
{
    const int ly = g.ns == 3 ? kGridLY3 : 32;
    const int w = int(e % (32 * slots)), in = w % (32 * g.pk);   // place in the step, in its group of pk slots
    const int lane = in / g.pk;
    o.q = w / (32 * g.pk) * g.pk + in % g.pk;
    const long long rest = e / (32 * slots);
    const int s = int(rest % g.nsp);
    const long long u = rest / g.nsp;
    const int a = lane % ly, b = lane / ly;
    o.i = s - a - b;
    o.j = int(u % g.njb) * ly + a;
    o.k = int(u / g.njb) * (32 / ly) + b;
    o.r = o.i + (long long)g.nx * (o.j + (long long)g.ny * o.k);
    return o.i >= 0 && o.i < g.nx && o.j < g.ny && o.k < g.nz;
}
// The layout element of row r' and slot q.
__host__ __device__ inline long long grid_elem_of(const GridFillGeom& g, int slots, long long r, int q)
{
    const int ly = g.ns == 3 ? kGridLY3 : 32, lz = 32 / ly;
    const int i = int(r % g.nx), j = int((r / g.nx) % g.ny), k = int(r / ((long long)g.nx * g.ny));
    const long long u = (long long)(k / lz) * g.njb + j / ly;
    const int a = j % ly, b = k % lz;
    return (u * g.nsp + i + a + b) * slots * 32 + grid_slot(g.pk, q, a + ly * b);
}
constexpr int kGridFillILU = 0, kGridFillIC = 1;
__global__ void k_fill_grid_csr(long long nent, GridFillGeom g, int lower, int kind, int unit, int lmul,
                                const int* __restrict__ rp, const int* __restrict__ ci, const double* __restrict__ src,
                                const double* __restrict__ inv_dia, void* val, int f32)
{
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < nent;
         e += (long long)gridDim.x * blockDim.x) {
        GridElem o;
        bool in;
        if (g.ns == 0) {
            o.q = 0;
            o.r = lower ? e : g.n - 1 - e;
            in = e < g.n;
        } else {
            in = grid_elem(g, g.ns + 1, e, o);
        }
        const int q = o.q;
        double v = 0.0;
        if (in) {
            const int r = lower ? int(o.r) : int(g.n - 1 - o.r);
            if (q == g.ns) {
                v = unit ? 1.0 : inv_dia[r];
            } else {
                const int d = (g.perm >> (2 * q)) & 3;
                const bool present = d == 0 ? o.i > 0 : d == 1 ? o.j > 0 : o.k > 0;
                if (present) {
                    const long long off = d == 0 ? 1 : d == 1 ? g.nx : (long long)g.nx * g.ny;
                    const int c = int(lower ? r - off : r + off);
                    const bool tr = kind == kGridFillIC && lower;   // IC(0)'s L holds the transposed upper entries
                    const int row = tr ? c : r, col = tr ? r : c;
                    int pos = -1;
                    for (int f = rp[row]; f < rp[row + 1]; ++f)
                        if (ci[f] == col) pos = f;
                    if (pos >= 0) {
                        v = src[pos];
                        if (kind == kGridFillIC) v = v * inv_dia[lower ? c : r];
                        else if (lmul && lower) v = v * inv_dia[c];   // ILU(0)'s l_rc = a_rc / u_cc, as the factorization rounds it
                    }
                }
            }
        }
        if (f32) static_cast<float*>(val)[e] = float(v);
        else static_cast<double*>(val)[e] = v;
    }
}

// Layout of a grid factorization (L's geometry, farthest neighbour first):
// per step and lane the row's entries toward its earlier neighbours a_ik
// (ILU(0) only), those neighbours' entries in the row's column a_ki, then
// a_ii; +0 where the row has no such neighbour.  FP64 values of A.
__global__ void k_fill_grid_factor(long long nent, GridFillGeom g, int kind, const int* __restrict__ rp,
                                   const int* __restrict__ ci, const double* __restrict__ a, double* __restrict__ out)
{
    const int slots = kind == kGridILU0 ? 2 * g.ns + 1 : g.ns + 1;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < nent;
         e += (long long)gridDim.x * blockDim.x) {
        GridElem o;
        const bool in = grid_elem(g, slots, e, o);
        const int q = o.q;
        double v = 0.0;
        if (in) {
            const long long r = o.r;
            int row = int(r), col = int(r);   // q == slots - 1: the diagonal
            bool present = true;
            if (q < slots - 1) {
                const int qd = q < g.ns ? q : q - g.ns;
                const int d = (g.perm >> (2 * qd)) & 3;
                present = d == 0 ? o.i > 0 : d == 1 ? o.j > 0 : o.k > 0;
                const long long off = d == 0 ? 1 : d == 1 ? g.nx : (long long)g.nx * g.ny;
                const int nb = int(r - off);
                const bool toward = kind == kGridILU0 && q < g.ns;   // a_ik (row r, column nb); else a_ki
                row = toward ? int(r) : nb;
                col = toward ? nb : int(r);
            }
            if (present)
                for (int f = rp[row]; f < rp[row + 1]; ++f)
                    if (ci[f] == col) v = a[f];
        }
        out[e] = v;
    }
}

// Flat-layout values copied from the grid layout (a factor built with the
// grid layout only, when a flat sweep, a factor download or the ILU(0)
// adjoint needs its flat layout): flat position p is row row_of[p], its
// entry k (column ci[k]) the grid element of that row and direction.
__global__ void k_flat_from_grid(int npos, const int* __restrict__ row_of, const int* __restrict__ rp,
                                 const int* __restrict__ ci, GridFillGeom g, int lower,
                                 const unsigned char* __restrict__ gval, unsigned char* __restrict__ val, int ssz)
{
    int rank[3] = {-1, -1, -1};
    for (int q = 0; q < g.ns; ++q) rank[(g.perm >> (2 * q)) & 3] = q;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < npos; p += gridDim.x * blockDim.x) {
        const int r = row_of[p];
        if (r < 0) continue;
        const long long rpr = lower ? r : (long long)g.n - 1 - r;
        for (int e = rp[p]; e < rp[p + 1]; ++e) {
            const long long off = lower ? (long long)r - ci[e] : (long long)ci[e] - r;
            const int d = off == 1 ? 0 : off == g.nx ? 1 : 2;
            const long long src = grid_elem_of(g, g.ns + 1, rpr, rank[d]);
            if (ssz == 8) reinterpret_cast<double*>(val)[e] = reinterpret_cast<const double*>(gval)[src];
            else reinterpret_cast<float*>(val)[e] = reinterpret_cast<const float*>(gval)[src];
        }
    }
}

// Grid layout values: per element a value source (>= 0, times the inverse
// pivot named by gmul when >= 0), -2 for a row's multiplier (the inverse
// pivot of row gmul, 1 for a unit diagonal), -1 for padding (+0).
__global__ void k_fill_grid(long long nent, const int* __restrict__ gsrc, const int* __restrict__ gmul,
                            const double* __restrict__ src, const double* __restrict__ inv_dia, int unit, void* val,
                            int f32)
{
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < nent;
         e += (long long)gridDim.x * blockDim.x) {
        const int c = gsrc[e], m = gmul[e];
        double v = 0.0;
        if (c >= 0) {
            v = src[c];
            if (m >= 0) v = v * inv_dia[m];
        } else if (c == -2) {
            v = (unit || m < 0) ? 1.0 : inv_dia[m];
        }
        if (f32) static_cast<float*>(val)[e] = float(v);
        else static_cast<double*>(val)[e] = v;
    }
}

}  // namespace mtlg
