// CSR SpMV and fused vector passes with device-side Krylov scalar updates.
//
// SpMV follows the reference's row-major CSR product
// (boost/numeric/mtl/operation/mat_vec_mult.hpp:614-683): every row is an
// accumulator started at zero and updated entry by entry in storage order,
// tmp += A.data[j] * v[A.ref_minor()[j]], then assigned/added/subtracted
// into w (Assign::first_update).  The reference build (g++ -O3 with FMA
// available) evaluates that loop in groups of four entries whose products
// are rounded before the addition, and the row's last (L mod 4) entries as
// fused multiply-adds; in FP32 every product is rounded first.  row_step
// reproduces this, so rows of up to kShortRow entries, which keep the exact
// order (one thread per row), are bitwise the reference's in FP64 and FP32.
// Longer rows are split over a warp (or the whole CTA) and summed as a fixed
// tree.
#pragma once
#include "common.cuh"

namespace mtlg {

// ---------------------------------------------------------------- operands
// Vector operand codes: >= 0 workspace slot, negatives name descriptor
// vectors; OPND_* are per-row values available in epilogues.
enum Slot : int { SLOT_X = -1, SLOT_B = -2, SLOT_X64 = -3, SLOT_B64 = -4, SLOT_R64 = -5, SLOT_NONE = -100 };
enum Opnd : int { OPND_ONE = -1000, OPND_Y = -1001, OPND_XP = -1002, OPND_D = -1003 };

template <typename T>
__device__ __forceinline__ T* vptr(const SysDesc& d, int slot)
{
    if (slot >= 0) return wsvec<T>(d, slot);
    switch (slot) {
    case SLOT_X: return static_cast<T*>(d.x);
    case SLOT_B: return const_cast<T*>(static_cast<const T*>(d.b));
    default: return nullptr;
    }
}

// ---------------------------------------------------------------- finalize
enum Fin : int {
    FIN_NONE = 0,
    FIN_STORE,          // st.dots[j] = sum_j
    FIN_CG_INIT,        // rr -> finished?  (identity: rho = rr)
    FIN_CG_INIT_JAC,    // rr, r.Dr -> finished?  rho = r.z
    FIN_CG_ALPHA,       // p.q -> alpha = rho / p.q, ++iter
    FIN_CG_UPDATE,      // rr -> finished?  identity: beta = rr / rho
    FIN_CG_UPDATE_JAC,  // rr, r.z -> finished?  beta = r.z / rho
    FIN_CG_UPDATE_PC,   // rr -> finished?  (z follows from the sweeps)
    FIN_CG_RHO,         // r.z after the sweeps -> beta
    FIN_BI_TOP,         // rt.r, r.r at the loop top (init and after r update)
    FIN_BI_GAMMA,       // rt.v -> alpha
    FIN_BI_S,           // s.s -> finished(s)?
    FIN_BI_OMEGA,       // t.s, t.t -> omega
    FIN_REF_OUTER,      // FP64 r.r -> refinement stop test, scale
    FIN_NORM_R0,        // norm_r0 = sqrt(b.b)  (basic_iteration from b)
    FIN_REF_NB,         // refinement: nb = ||b||_FP64
    FIN_REF_CG_INIT,    // inner CG init on the scaled residual (norm_r0 = ||r||)
    FIN_REF_CG_INIT_JAC,
    FIN_REF_BI_INIT,    // inner BiCGSTAB init (norm_r0 = ||r||)
    FIN_PHASE_OUTER,    // served refinement: back to the outer residual
};

// Status flags
enum : int { FLAG_FINISHING = 1 };

__device__ __forceinline__ void bicg_top(const SetView& sv, SysState& s, double rtr, double rr, bool first_pass)
{
    if (!first_pass) s.rho_1 = s.rho;  // rho_2 = rho_1 (bicgstab.hpp:75)
    if (check_finished(sv, s, sqrt(fabs(rr)))) return;
    s.iter += 1;
    s.rho = rtr;  // rho_1 = dot(rtilde, r)
    if (s.rho == 0.0) { retire(sv, s, MTLG_ST_BREAKDOWN, 1); return; }
    if (s.iter > 1) {
        if (s.omega == 0.0) { retire(sv, s, MTLG_ST_BREAKDOWN, 1); return; }
        s.beta = (s.rho / s.rho_1) * (s.alpha / s.omega);
    }
}

__device__ void finalize(const SetView& sv, int fin, int sys, const double* dots)
{
    SysState& s = sv.st[sys];
    switch (fin) {
    case FIN_STORE:
        for (int j = 0; j < kMaxDots; ++j) s.dots[j] = dots[j];
        break;
    case FIN_NORM_R0:
        s.norm_r0 = sqrt(fabs(dots[0]));
        break;
    case FIN_REF_NB:
        s.nb = sqrt(fabs(dots[0]));
        break;
    case FIN_REF_CG_INIT:
        s.phase = PH_INNER;
        s.norm_r0 = sqrt(fabs(dots[0]));
        s.rr = dots[0];
        s.rho = dots[0];
        check_finished(sv, s, sqrt(fabs(dots[0])));
        break;
    case FIN_REF_CG_INIT_JAC:
        s.phase = PH_INNER;
        s.norm_r0 = sqrt(fabs(dots[0]));
        s.rr = dots[0];
        s.rho = dots[1];
        check_finished(sv, s, sqrt(fabs(dots[0])));
        break;
    case FIN_REF_BI_INIT:
        s.phase = PH_INNER;
        s.norm_r0 = sqrt(fabs(dots[1]));
        bicg_top(sv, s, dots[0], dots[1], true);
        break;
    case FIN_CG_INIT:
        s.phase = PH_INNER;
        s.rr = dots[0];
        s.rho = dots[0];
        s.iter = 0;
        check_finished(sv, s, sqrt(fabs(dots[0])));
        break;
    case FIN_CG_INIT_JAC:
        s.phase = PH_INNER;
        s.rr = dots[0];
        s.rho = dots[1];
        s.iter = 0;
        check_finished(sv, s, sqrt(fabs(dots[0])));
        break;
    case FIN_CG_ALPHA:
        s.dots[0] = dots[0];
        s.alpha = s.rho / dots[0];
        s.iter += 1;
        break;
    case FIN_CG_UPDATE:
        s.rr = dots[0];
        if (!check_finished(sv, s, sqrt(fabs(dots[0])))) {
            s.rho_1 = s.rho;
            s.rho = dots[0];
            s.beta = s.rho / s.rho_1;
        }
        break;
    case FIN_CG_UPDATE_JAC:
        s.rr = dots[0];
        if (!check_finished(sv, s, sqrt(fabs(dots[0])))) {
            s.rho_1 = s.rho;
            s.rho = dots[1];
            s.beta = s.rho / s.rho_1;
        }
        break;
    case FIN_CG_UPDATE_PC:
        s.rr = dots[0];
        check_finished(sv, s, sqrt(fabs(dots[0])));
        break;
    case FIN_CG_RHO:
        s.rho_1 = s.rho;
        s.rho = dots[0];
        s.beta = s.rho / s.rho_1;
        break;
    case FIN_BI_TOP:
        if (s.iter == 0) s.phase = PH_INNER;
        bicg_top(sv, s, dots[0], dots[1], s.iter == 0);
        break;
    case FIN_PHASE_OUTER:
        s.phase = PH_OUTER;
        break;
    case FIN_BI_GAMMA:
        s.gamma = dots[0];
        if (s.gamma == 0.0) { retire(sv, s, MTLG_ST_BREAKDOWN, 1); break; }
        s.alpha = s.rho / s.gamma;
        // a non-finite step would spoil the iterate: stop before the update
        if (!isfinite(s.alpha)) retire(sv, s, MTLG_ST_BREAKDOWN, 1);
        break;
    case FIN_BI_S: {
        // iter.finished(s) (bicgstab.hpp:64): on true, x += alpha*phat is
        // still due; the x/r pass does it and then retires the system.
        const double res = sqrt(fabs(dots[0]));
        log_check(s, res);
        s.resid = res;
        bool conv = (s.norm_r0 == 0.0) ? (res <= s.atol) : (res <= s.rtol * s.norm_r0 || res <= s.atol);
        if (conv) { s.flags |= FLAG_FINISHING; s.error = 0; s.dots[3] = MTLG_ST_CONVERGED; }
        else if (isnan(res) || isinf(res)) { retire(sv, s, MTLG_ST_BREAKDOWN, 1); }
        else if (s.iter >= s.max_iter) { s.flags |= FLAG_FINISHING; s.error = 1; s.dots[3] = MTLG_ST_MAXIT; }
        break;
    }
    case FIN_BI_OMEGA:
        s.omega = dots[0] / dots[1];
        // t.t == 0 or an overflow: stop before x and r take a non-finite step
        if (!isfinite(s.omega)) retire(sv, s, MTLG_ST_BREAKDOWN, 1);
        break;
    case FIN_REF_OUTER: {
        // Refinement stop test on the FP64 residual: ||b - A x|| <= rtol*||b||.
        const double rn = sqrt(fabs(dots[0]));
        const double prev = s.scale;   // the previous outer residual (outer >= 1)
        s.inner_total += s.iter;
        s.iter = 0;
        s.scale = rn;
        s.resid = rn;
        s.flags = 0;
        if (rn <= s.outer_rtol * s.nb) {
            s.ostatus = MTLG_ST_CONVERGED; s.status = MTLG_ST_CONVERGED; s.error = 0; s.phase = PH_DONE;
        } else if (isnan(rn) || isinf(rn)) {
            s.ostatus = MTLG_ST_BREAKDOWN; s.status = MTLG_ST_BREAKDOWN; s.error = 1; s.phase = PH_DONE;
        } else if (s.outer >= 1 && !(rn <= kRefMinGain * prev)) {
            // the FP32 inner solves no longer reduce the FP64 residual (the
            // operator is too ill-conditioned for FP32): stop; the host
            // finishes the system in FP64
            s.ostatus = MTLG_ST_STALLED; s.status = MTLG_ST_STALLED; s.error = 1; s.phase = PH_DONE;
        } else if (s.outer >= s.max_outer) {
            s.ostatus = MTLG_ST_MAXIT; s.status = MTLG_ST_MAXIT; s.error = 1; s.phase = PH_DONE;
        } else {
            s.outer += 1;
            s.status = MTLG_ST_RUNNING;
            s.phase = PH_CAST;
            atomicAdd(sv.running, 1);
        }
        break;
    }
    default:
        break;
    }
}

// ---------------------------------------------------------------- SpMV
enum XForm : int { XF_PLAIN = 0, XF_CG_P = 1, XF_CG_P_JAC = 2, XF_JAC = 3 };
enum Assign : int { ASG_SET = 0, ASG_ADD = 1, ASG_SUB = 2, ASG_WMINUS = 3 };
enum Skip : int { SKIP_NONE = 0, SKIP_INNER = 1, SKIP_OUTER = 2, SKIP_RUNNING = 3, SKIP_PH_BASE = 16 };
// SKIP_PH_BASE + p: act only on systems in phase p (served solves)

struct SpmvOp {
    int x, y, w;        // input slot, output slot, W for y = W - A x
    int y2;             // optional second output (copy of y)
    int p, z, pnew;     // XF_CG_*: old p, z (or r), new p
    int ndot;
    int da[kMaxDots], db[kMaxDots], dc[kMaxDots];
    int rk[kMaxDots];   // reference summation order of each dot (RK_*, refdot.cuh)
    int fin;
    int skip;
    int count_body;     // increments the body counter (first kernel of a loop body)
};

__device__ __forceinline__ bool skip_system(const SysState& s, int mode)
{
    if (mode == SKIP_INNER) return s.status != MTLG_ST_RUNNING || (s.flags & FLAG_FINISHING);
    if (mode == SKIP_OUTER) return s.ostatus != MTLG_ST_RUNNING;
    if (mode == SKIP_RUNNING) return s.status != MTLG_ST_RUNNING;
    if (mode >= SKIP_PH_BASE) return s.phase != mode - SKIP_PH_BASE;
    return false;
}

// acc + a*x with the product rounded first (no contraction)
__device__ __forceinline__ double mac(double acc, double a, double x) { return __dadd_rn(acc, __dmul_rn(a, x)); }
__device__ __forceinline__ float mac(float acc, float a, float x) { return __fadd_rn(acc, __fmul_rn(a, x)); }
// One step of a sequential row sum: entries before the row's last (L mod 4)
// add the rounded product, the last ones are fused (FP64 only), as in the
// reference build's row loop.  `fused` = the entry lies in that tail.
__device__ __forceinline__ double row_step(double acc, double a, double x, bool fused)
{
    return fused ? __fma_rn(a, x, acc) : mac(acc, a, x);
}
__device__ __forceinline__ float row_step(float acc, float a, float x, bool) { return mac(acc, a, x); }
// first entry of a row's fused tail: a + 4 * floor((e - a) / 4)
__device__ __forceinline__ int fused_tail(int a, int e) { return a + ((e - a) & ~3); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }

template <typename T, int XF>
struct XIn {
    const T* x;
    const T* p;
    const T* z;
    const T* dinv;
    T beta;
    bool first;
    __device__ __forceinline__ T operator()(int j) const
    {
        if (XF == XF_PLAIN) return x[j];
        if (XF == XF_JAC) return dinv[j] * x[j];
        T zj = (XF == XF_CG_P_JAC) ? dinv[j] * z[j] : z[j];
        return first ? zj : fma(beta, p[j], zj);
    }
};

// Slot codes that name a vector (workspace slot or descriptor vector).
__device__ __forceinline__ bool names_vector(int code) { return code >= SLOT_B; }

template <typename T, int ASG>
__device__ __forceinline__ T assign_out(T old_or_w, T acc)
{
    if (ASG == ASG_SET) return acc;
    if (ASG == ASG_ADD) return old_or_w + acc;
    return old_or_w - acc;  // ASG_SUB and ASG_WMINUS
}

// Per-row epilogue operand (a dot factor): a vector, or y / x' / D of the row.
template <typename T>
struct Opnd1 {
    int code;
    const T* v;
    __device__ __forceinline__ T get(int i, T y, T xp, const T* dinv) const
    {
        switch (code) {
        case OPND_ONE: return T(1);
        case OPND_Y: return y;
        case OPND_XP: return xp;
        case OPND_D: return dinv[i];
        default: return v[i];
        }
    }
};

template <typename T, int ASG, int XF>
struct RowEpilogue {
    T* y;
    T* y2;
    const T* w;
    T* pnew;
    int ndot;
    Opnd1<T> a0, b0, c0, a1, b1, c1;
    __device__ __forceinline__ void operator()(int i, T acc, T xp, const T* dinv, double& d0, double& d1) const
    {
        const T base = (ASG == ASG_SET) ? T(0) : ((ASG == ASG_WMINUS) ? w[i] : y[i]);
        const T out = assign_out<T, ASG>(base, acc);
        y[i] = out;
        if (y2) y2[i] = out;
        if (XF != XF_PLAIN) pnew[i] = xp;
        if (ndot > 0) d0 += double(a0.get(i, out, xp, dinv) * b0.get(i, out, xp, dinv) * c0.get(i, out, xp, dinv));
        if (ndot > 1) d1 += double(a1.get(i, out, xp, dinv) * b1.get(i, out, xp, dinv) * c1.get(i, out, xp, dinv));
    }
};

template <typename T, int ASG, int XF>
__device__ __forceinline__ RowEpilogue<T, ASG, XF> row_epilogue(const SysDesc& d, const SpmvOp& op)
{
    RowEpilogue<T, ASG, XF> epi;
    epi.y = vptr<T>(d, op.y);
    epi.y2 = op.y2 != SLOT_NONE ? vptr<T>(d, op.y2) : nullptr;
    epi.w = op.w != SLOT_NONE ? vptr<T>(d, op.w) : nullptr;
    epi.pnew = op.pnew != SLOT_NONE ? vptr<T>(d, op.pnew) : nullptr;
    epi.ndot = op.ndot;
    epi.a0 = {op.da[0], names_vector(op.da[0]) ? vptr<T>(d, op.da[0]) : nullptr};
    epi.b0 = {op.db[0], names_vector(op.db[0]) ? vptr<T>(d, op.db[0]) : nullptr};
    epi.c0 = {op.dc[0], names_vector(op.dc[0]) ? vptr<T>(d, op.dc[0]) : nullptr};
    epi.a1 = {op.da[1], names_vector(op.da[1]) ? vptr<T>(d, op.da[1]) : nullptr};
    epi.b1 = {op.db[1], names_vector(op.db[1]) ? vptr<T>(d, op.db[1]) : nullptr};
    epi.c1 = {op.dc[1], names_vector(op.dc[1]) ? vptr<T>(d, op.dc[1]) : nullptr};
    return epi;
}
template <typename T, int XF>
__device__ __forceinline__ XIn<T, XF> row_input(const SysDesc& d, const SysState& s, const SpmvOp& op)
{
    XIn<T, XF> xin;
    xin.x = vptr<T>(d, op.x);
    xin.p = op.p != SLOT_NONE ? vptr<T>(d, op.p) : nullptr;
    xin.z = op.z != SLOT_NONE ? vptr<T>(d, op.z) : nullptr;
    xin.dinv = static_cast<const T*>(d.inv_diag);
    xin.beta = T(s.beta);
    xin.first = (s.iter == 0);
    return xin;
}

// ---- shared-memory staging of a stream tile (16-byte cp.async copies)
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem)
{
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_1() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_0() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// Buffer layout: values (kTileNnz + one chunk), columns (kTileNnz + one
// chunk), row pointers (kTileRows + 1 + one chunk).  Every copy is widened to
// 16-byte boundaries; the device arrays carry 16 bytes of tail padding, so
// the widened range stays inside the allocation.
template <typename T>
struct StageLayout {
    static constexpr int VE = 16 / sizeof(T);
    static constexpr int VBYTES = (kTileNnz + 2 * VE) * sizeof(T);
    static constexpr int CBYTES = (kTileNnz + 8) * 4;
    static constexpr int RBYTES = ((kTileRows + 1 + 8) * 4 + 15) / 16 * 16;
    static constexpr int BYTES = VBYTES + CBYTES + RBYTES;
    static_assert(VBYTES % 16 == 0 && CBYTES % 16 == 0 && BYTES % 16 == 0, "16-byte aligned sections");
};

template <typename T>
__device__ __forceinline__ void stage_tile(const Tile& t, const int* rp, const int* ci, const T* va, unsigned char* buf)
{
    typedef StageLayout<T> SL;
    const int ka = t.nnz_begin & ~(SL::VE - 1);
    const int kb = (t.nnz_end + SL::VE - 1) & ~(SL::VE - 1);
    for (int c = threadIdx.x; c < (kb - ka) / SL::VE; c += blockDim.x)
        cp_async16(buf + c * 16, va + ka + c * SL::VE);
    const int ca = t.nnz_begin & ~3, cb = (t.nnz_end + 3) & ~3;
    for (int c = threadIdx.x; c < (cb - ca) / 4; c += blockDim.x)
        cp_async16(buf + SL::VBYTES + c * 16, ci + ca + c * 4);
    const int ra = t.row_begin & ~3, rb = (t.row_end + 1 + 3) & ~3;
    for (int c = threadIdx.x; c < (rb - ra) / 4; c += blockDim.x)
        cp_async16(buf + SL::VBYTES + SL::CBYTES + c * 16, rp + ra + c * 4);
}

// Persistent CTAs walk the tiles with a stride of the grid.  A stream tile's
// values, columns and row pointers are copied into one of two shared-memory
// buffers while the previous tile is summed from the other.  Every thread
// then sums one row sequentially; rows longer than kShortRow are summed by a
// warp from shared memory.  A long tile (one row with more than kTileNnz
// entries) is summed by the whole CTA straight from global memory.
// Publishes a CTA's tally of a system's finished SpMV tiles; the CTA that
// completes the system gathers its partials and finalizes.
// ALL: all kMaxDots partials are there and are gathered, whatever op.ndot is.
// (k_spmv: choosing among the three gathers costs its 80 registers 110 bytes
// of spills in FP32 and 100 more in FP64, on 14 random entries a row 114 us
// instead of 85 and 140 instead of 115.)
template <bool ALL, typename OpT>
__device__ __forceinline__ void spmv_publish(const SetView& sv, const OpT& op, TileTally& tally, double* s_red)
{
    if (publish_tally(sv, tally)) {
        double tot[kMaxDots];
        if (ALL) gather_dots<kMaxDots>(sv, sv.sys_tile_begin[tally.sys], sv.sys_tile_begin[tally.sys + 1], tot, s_red);
        else gather_partials(sv, tally.sys, op.ndot, tot, s_red);
        if (threadIdx.x == 0) finalize(sv, op.fin, tally.sys, tot);
    }
}

template <typename T, int XF, int ASG>
__global__ void __launch_bounds__(kBlock, 3) k_spmv(SetView sv, SpmvOp op)
{
    typedef StageLayout<T> SL;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int s_med[kTileRows];
    __shared__ int s_nmed;
    __shared__ double s_red[kMaxDots * 32];
    __shared__ T s_acc[32];

    if (op.count_body && blockIdx.x == 0 && threadIdx.x == 0) {
        // loop-body counter: bounds a graph while-loop independently of the
        // solver's own termination test
        int runs = atomicAdd(&sv.err[1], 1) + 1;
        if (runs > sv.err[2] || *(volatile int*)sv.running <= 0) set_cond(sv, 0u);
    }
    const int G = gridDim.x;
    int t = blockIdx.x;
    if (t >= sv.n_tiles) return;
    TileTally tally;   // finished tiles of the current system, published per system run

    Tile cur = sv.tiles[t];
    {
        const SysDesc& d0 = sv.desc[cur.sys];
        if (cur.kind == TILE_STREAM && !skip_system(sv.st[cur.sys], op.skip))
            stage_tile<T>(cur, d0.rp, d0.ci, static_cast<const T*>(d0.val), smem_raw);
        cp_async_commit();
    }
    Tile nxt = (t + G < sv.n_tiles) ? sv.tiles[t + G] : cur;

    for (int it = 0; t < sv.n_tiles; t += G, ++it) {
        const int tn = t + G;
        Tile nn = (tn + G < sv.n_tiles) ? sv.tiles[tn + G] : nxt;   // metadata one tile ahead
        unsigned char* buf = smem_raw + (it & 1) * SL::BYTES;
        if (tn < sv.n_tiles) {
            const SysDesc& dn = sv.desc[nxt.sys];
            if (nxt.kind == TILE_STREAM && !skip_system(sv.st[nxt.sys], op.skip))
                stage_tile<T>(nxt, dn.rp, dn.ci, static_cast<const T*>(dn.val), smem_raw + ((it + 1) & 1) * SL::BYTES);
        }
        cp_async_commit();
        cp_async_wait_1();
        __syncthreads();

        const Tile tile = cur;
        const int sys = tile.sys;
        if (op.fin != FIN_NONE && sys != tally.sys) {
            spmv_publish<true>(sv, op, tally, s_red);
            tally.sys = sys;
        }
        const SysDesc& d = sv.desc[sys];
        const SysState& s = sv.st[sys];
        if (!skip_system(s, op.skip)) {
            const XIn<T, XF> xin = row_input<T, XF>(d, s, op);
            const T* dinv = xin.dinv;

            const RowEpilogue<T, ASG, XF> epi = row_epilogue<T, ASG, XF>(d, op);
            double d0 = 0.0, d1 = 0.0;

            if (tile.kind == TILE_STREAM) {
                const T* s_val = reinterpret_cast<const T*>(buf);
                const int* s_col = reinterpret_cast<const int*>(buf + SL::VBYTES);
                const int* s_rp = reinterpret_cast<const int*>(buf + SL::VBYTES + SL::CBYTES);
                const int ka = tile.nnz_begin & ~(SL::VE - 1), ca = tile.nnz_begin & ~3, ra = tile.row_begin & ~3;
                if (threadIdx.x == 0) s_nmed = 0;
                __syncthreads();
                const int i = tile.row_begin + threadIdx.x;
                if (i < tile.row_end) {
                    const int a = s_rp[i - ra], e = s_rp[i + 1 - ra];
                    if (e - a <= kShortRow) {
                        // gathers issued 8 at a time, summed in storage order
                        T acc = T(0);
                        const int q = fused_tail(a, e);
                        int k = a;
                        for (; k + 8 <= e; k += 8) {
                            T xv[8];
#pragma unroll
                            for (int u = 0; u < 8; ++u) xv[u] = xin(s_col[k + u - ca]);
#pragma unroll
                            for (int u = 0; u < 8; ++u) acc = row_step(acc, s_val[k + u - ka], xv[u], k + u >= q);
                        }
                        T xv[8];
#pragma unroll
                        for (int u = 0; u < 8; ++u) if (k + u < e) xv[u] = xin(s_col[k + u - ca]);
#pragma unroll
                        for (int u = 0; u < 8; ++u)
                            if (k + u < e) acc = row_step(acc, s_val[k + u - ka], xv[u], k + u >= q);
                        epi(i, acc, xin(i), dinv, d0, d1);
                    } else {
                        s_med[atomicAdd(&s_nmed, 1)] = i;
                    }
                }
                __syncthreads();
                const int nmed = s_nmed;
                const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
                for (int m = warp; m < nmed; m += nw) {
                    const int r = s_med[m];
                    const int a = s_rp[r - ra], e = s_rp[r + 1 - ra];
                    T acc = T(0);
                    int k = a + lane;
                    for (; k + 3 * 32 < e; k += 4 * 32) {
                        const T x0 = xin(s_col[k - ca]), x1 = xin(s_col[k + 32 - ca]);
                        const T x2 = xin(s_col[k + 64 - ca]), x3 = xin(s_col[k + 96 - ca]);
                        acc = mac(acc, s_val[k - ka], x0);
                        acc = mac(acc, s_val[k + 32 - ka], x1);
                        acc = mac(acc, s_val[k + 64 - ka], x2);
                        acc = mac(acc, s_val[k + 96 - ka], x3);
                    }
                    for (; k < e; k += 32) acc = mac(acc, s_val[k - ka], xin(s_col[k - ca]));
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
                    if (lane == 0) epi(r, acc, xin(r), dinv, d0, d1);
                }
            } else {
                const int r = tile.row_begin;
                const int* __restrict__ ci = d.ci;
                const T* __restrict__ va = static_cast<const T*>(d.val);
                T acc = T(0);
                int k = tile.nnz_begin + threadIdx.x;
                const int B = blockDim.x;
                for (; k + 3 * B < tile.nnz_end; k += 4 * B) {
                    const int c0 = ci[k], c1 = ci[k + B], c2 = ci[k + 2 * B], c3 = ci[k + 3 * B];
                    const T v0 = va[k], v1 = va[k + B], v2 = va[k + 2 * B], v3 = va[k + 3 * B];
                    const T x0 = xin(c0), x1 = xin(c1), x2 = xin(c2), x3 = xin(c3);
                    acc = mac(acc, v0, x0);
                    acc = mac(acc, v1, x1);
                    acc = mac(acc, v2, x2);
                    acc = mac(acc, v3, x3);
                }
                for (; k < tile.nnz_end; k += B) acc = mac(acc, va[k], xin(ci[k]));
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
                const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
                if (lane == 0) s_acc[warp] = acc;
                __syncthreads();
                if (warp == 0) {
                    acc = lane < (int)(blockDim.x >> 5) ? s_acc[lane] : T(0);
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
                    if (lane == 0) epi(r, acc, xin(r), dinv, d0, d1);
                }
            }
            if (op.fin != FIN_NONE) {
                double dd[kMaxDots] = {d0, d1, 0.0, 0.0};
                block_reduce<kMaxDots>(dd, s_red);
                store_partials<kMaxDots>(sv, t, dd);
                ++tally.n;
            }
        }
        __syncthreads();   // the buffer is refilled two tiles later
        cur = nxt;
        nxt = nn;
    }
    cp_async_wait_0();
    if (op.fin != FIN_NONE) spmv_publish<true>(sv, op, tally, s_red);
}

// ---------------------------------------------------------------- SpMV, thread per row
// The in-solve product of sets whose rows are all short and regular
// (SetView::short_rows): a thread takes one row of each tile straight from
// global memory, entries 8 at a time in storage order (k_spmv's arithmetic to
// the bit).  Bound by HBM: adjacent rows of a warp use the sectors the first
// of them brought in, and there is no staging and no barrier per tile (FP64
// BiCGSTAB product with two dots on 128^3, cold caches: k_spmv 106 us, this
// kernel 80 us; floor 39 us at 6.55 TB/s).  Each CTA walks a contiguous run of
// tiles.
template <typename T, int XF, int ASG, int ND>
__global__ void __launch_bounds__(kBlock, 2) k_spmv_short(SetView sv, SpmvOp op)
{
    __shared__ double s_red[kMaxDots * 32];
    __shared__ double s_part[kPartTiles * (kBlock / 32) * (ND > 0 ? ND : 1)];
    if (op.count_body && blockIdx.x == 0 && threadIdx.x == 0) {
        int runs = atomicAdd(&sv.err[1], 1) + 1;   // bounds a graph while-loop (see k_spmv)
        if (runs > sv.err[2] || *(volatile int*)sv.running <= 0) set_cond(sv, 0u);
    }
    const int t_begin = int((long long)sv.n_tiles * blockIdx.x / gridDim.x);
    const int t_end = int((long long)sv.n_tiles * (blockIdx.x + 1) / gridDim.x);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    TileTally tally;
    int t = t_begin;
    while (t < t_end) {
        const int sys = sv.n_sys == 1 ? 0 : sv.tiles[t].sys;
        const int te = sv.n_sys == 1 ? t_end : min(t_end, sv.sys_tile_begin[sys + 1]);   // this system's tiles in the CTA's run
        if (op.fin != FIN_NONE && sys != tally.sys) {
            spmv_publish<false>(sv, op, tally, s_red);
            tally.sys = sys;
        }
        const SysState& s = sv.st[sys];
        if (skip_system(s, op.skip)) {
            t = te;
            continue;
        }
        const SysDesc& d = sv.desc[sys];
        const int* __restrict__ rp = d.rp;
        const int* __restrict__ ci = d.ci;
        const T* __restrict__ va = static_cast<const T*>(d.val);
        const XIn<T, XF> xin = row_input<T, XF>(d, s, op);
        const RowEpilogue<T, ASG, XF> epi = row_epilogue<T, ASG, XF>(d, op);
        // Row bounds two tiles ahead, the first 8 columns one tile ahead: a
        // tile then costs one round of loads (values and gathers), not the
        // chain row pointers -> columns -> gathers.
        auto tile_row = [&](int k) {   // this thread's row of tile k, or -1
            const int r = sv.tiles[k].row_begin + int(threadIdx.x);
            return k < te && r < sv.tiles[k].row_end ? r : -1;
        };
        auto bounds = [&](int r) { return r >= 0 ? make_int2(rp[r], rp[r + 1]) : make_int2(0, 0); };
        int i = tile_row(t), in = t + 1 < te ? tile_row(t + 1) : -1;
        int2 ae = bounds(i), aen = bounds(in);
        int c[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) c[u] = ae.x + u < ae.y ? ci[ae.x + u] : 0;
        int held = 0;
        for (; t < te; ++t) {
            const int a = ae.x, e = ae.y, q = fused_tail(a, e);
            T xv[8], av[8], acc = T(0);
#pragma unroll
            for (int u = 0; u < 8; ++u) if (a + u < e) { av[u] = va[a + u]; xv[u] = xin(c[u]); }
            const int inn = t + 2 < te ? tile_row(t + 2) : -1;
            const int2 aenn = bounds(inn);
            int cn[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) cn[u] = aen.x + u < aen.y ? ci[aen.x + u] : 0;
            double d0 = 0.0, d1 = 0.0;
#pragma unroll
            for (int u = 0; u < 8; ++u) if (a + u < e) acc = row_step(acc, av[u], xv[u], a + u >= q);
            for (int k = a + 8; k < e; k += 8) {
#pragma unroll
                for (int u = 0; u < 8; ++u) if (k + u < e) { av[u] = va[k + u]; xv[u] = xin(ci[k + u]); }
#pragma unroll
                for (int u = 0; u < 8; ++u) if (k + u < e) acc = row_step(acc, av[u], xv[u], k + u >= q);
            }
            if (i >= 0) epi(i, acc, xin(i), xin.dinv, d0, d1);
            i = in;
            in = inn;
            ae = aen;
            aen = aenn;
#pragma unroll
            for (int u = 0; u < 8; ++u) c[u] = cn[u];
            if constexpr (ND > 0) {
                double dd[ND];
                dd[0] = d0;
                if (ND > 1) dd[ND - 1] = d1;
                const double sum = warp_sums<ND>(dd);
                if (lane % (32 / ND) == 0) s_part[(held * (kBlock / 32) + warp) * ND + warp_sum_index<ND>(lane)] = sum;
                if (++held == kPartTiles) {
                    flush_parts<ND>(sv, t + 1 - held, held, s_part);
                    tally.n += unsigned(held);
                    held = 0;
                }
            }
        }
        if constexpr (ND > 0) {
            if (held) flush_parts<ND>(sv, t - held, held, s_part);
            tally.n += unsigned(held);
        }
    }
    if (op.fin != FIN_NONE) spmv_publish<false>(sv, op, tally, s_red);
}

// ---------------------------------------------------------------- SpMV, warp tasks
// Row-aligned warp tasks for matrices with irregular row lengths.  A task is
// either a run of consecutive rows with at most kWarpNnz entries in total
// (and at most kWarpNnz rows), or one row with more entries.
constexpr int kWarpNnz = 256;
constexpr int kSeqRow = 32;   // rows of a run task summed by one lane in storage order

struct WarpTask {
    int row_begin, row_end, nnz_begin, nnz_end;
};

// Element copies global -> shared without register staging (cp.async of 4
// or 8 bytes, cached in L1 as the only size-generic form allows).
template <int BYTES>
__device__ __forceinline__ void cp_async_elem(void* smem, const void* gmem)
{
    const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(s), "l"(gmem), "n"(BYTES) : "memory");
}
__device__ __forceinline__ void cp_async_drain_warp()
{
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
    __syncwarp();
}

// Run tasks: each lane loads 8 column indices (coalesced) and issues, without
// register staging, the copies of the matching values and the 8 gathers of x
// into the warp's shared buffers (cp.async), plus the task's row pointers;
// every lane then sums whole rows of up to kSeqRow entries from there,
// sequentially in storage order with row_step (so such a row's result is
// bitwise the reference's row sum); longer rows are summed by the whole warp.
// Long-row tasks: the warp strides over the row 256 entries at a time
// through the same buffers and reduces with a fixed tree.
// Scheduling: warps take tasks from a counter (one atomic per task) in the
// order of the task list -- long-row tasks first, most entries first, then
// the runs in row order -- so no warp is left holding several long rows at
// the end; the next task's descriptor is loaded while the current one runs.
// The last warp to finish resets the counter for the next launch.  No CTA
// barrier: warps proceed independently.
template <typename T, int ASG>
__global__ void __launch_bounds__(kBlock, 3)
k_spmv_rows(const WarpTask* __restrict__ tasks, int ntasks, int* __restrict__ ctr, const int* __restrict__ rp,
            const int* __restrict__ ci, const T* __restrict__ va, const T* __restrict__ x, T* __restrict__ y)
{
    __shared__ T s_a[kBlock / 32][kWarpNnz];
    __shared__ T s_x[kBlock / 32][kWarpNnz];
    __shared__ int s_rp[kBlock / 32][kWarpNnz + 1];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    T* sa = s_a[wib];
    T* sx = s_x[wib];
    int* srp = s_rp[wib];
    auto grab = [&]() {
        int v = 0;
        if (lane == 0) v = atomicAdd(ctr, 1);
        return __shfl_sync(0xffffffffu, v, 0);
    };
    int t = grab();
    WarpTask nxt;
    if (t < ntasks) nxt = tasks[t];
    while (t < ntasks) {
        const WarpTask task = nxt;
        t = grab();
        if (t < ntasks) nxt = tasks[t];
        const int k0 = task.nnz_begin, k1 = task.nnz_end;
        if (task.row_end - task.row_begin == 1 && k1 - k0 > kWarpNnz) {
            T acc = T(0);
            for (int kb = k0; kb < k1; kb += 32 * 8) {
                int cc[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const int k = kb + lane + 32 * u;
                    if (k < k1) {
                        cc[u] = __ldg(ci + k);
                        cp_async_elem<sizeof(T)>(sa + lane + 32 * u, va + k);
                    }
                }
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    if (kb + lane + 32 * u < k1) cp_async_elem<sizeof(T)>(sx + lane + 32 * u, x + cc[u]);
                cp_async_drain_warp();
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    if (kb + lane + 32 * u < k1) acc = mac(acc, sa[lane + 32 * u], sx[lane + 32 * u]);
                __syncwarp();   // the buffers are refilled by the next 256 entries
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
            if (lane == 0) {
                const int r = task.row_begin;
                const T base = (ASG == ASG_SET) ? T(0) : y[r];
                y[r] = assign_out<T, ASG>(base, acc);
            }
            continue;
        }
        const int nr = task.row_end - task.row_begin;
        int cc[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int k = k0 + lane + 32 * u;
            if (k < k1) {
                cc[u] = __ldg(ci + k);
                cp_async_elem<sizeof(T)>(sa + lane + 32 * u, va + k);
            }
        }
#pragma unroll
        for (int u = 0; u < 9; ++u) {
            const int r = lane + 32 * u;
            if (r <= nr) cp_async_elem<4>(srp + r, rp + task.row_begin + r);
        }
#pragma unroll
        for (int u = 0; u < 8; ++u)
            if (k0 + lane + 32 * u < k1) cp_async_elem<sizeof(T)>(sx + lane + 32 * u, x + cc[u]);
        cp_async_drain_warp();
        // rows of up to kSeqRow entries: one lane each, summed sequentially
        // (bitwise the sequential row sum); longer rows: the whole warp,
        // lane-strided partial sums and a fixed shuffle tree, so no lane
        // walks a long row alone while the others wait
        for (int base = 0; base < nr; base += 32) {
            const int r = base + lane;
            int a = 0, e = 0;
            if (r < nr) {
                a = srp[r] - k0;
                e = srp[r + 1] - k0;
            }
            const bool seq = r < nr && e - a <= kSeqRow;
            if (seq) {
                T acc = T(0);
                const int q = fused_tail(a, e);
                for (int j = a; j < e; ++j) acc = row_step(acc, sa[j], sx[j], j >= q);
                const int row = task.row_begin + r;
                const T yb = (ASG == ASG_SET) ? T(0) : y[row];
                y[row] = assign_out<T, ASG>(yb, acc);
            }
            unsigned lng = __ballot_sync(0xffffffffu, r < nr && !seq);
            while (lng) {
                const int rr = base + __ffs(lng) - 1;
                lng &= lng - 1;
                T acc = T(0);
                const int ra = srp[rr] - k0, re = srp[rr + 1] - k0;
                for (int j = ra + lane; j < re; j += 32) acc = mac(acc, sa[j], sx[j]);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
                if (lane == 0) {
                    const int row = task.row_begin + rr;
                    const T yb = (ASG == ASG_SET) ? T(0) : y[row];
                    y[row] = assign_out<T, ASG>(yb, acc);
                }
            }
        }
        __syncwarp();
    }
    // self-reset: the last warp out zeroes the task counter and itself
    if (lane == 0) {
        const int nw = gridDim.x * (blockDim.x >> 5);
        if (atomicAdd(ctr + 1, 1) == nw - 1) {
            ctr[0] = 0;
            ctr[1] = 0;
            __threadfence();
        }
    }
}

// Gather floor of y = A x (a measurement kernel): every entry's value and
// column are streamed and x[col] gathered, 8 entries in flight per thread,
// with no row structure; one partial sum per thread.
__global__ void __launch_bounds__(kBlock) k_gather_floor(long long nnz, const int* __restrict__ ci,
                                                         const double* __restrict__ va, const double* __restrict__ x,
                                                         double* __restrict__ out)
{
    double acc = 0.0;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long k0 = blockIdx.x * (long long)blockDim.x + threadIdx.x; k0 < nnz; k0 += 8 * stride) {
        int c[8];
        double v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const long long k = k0 + u * stride;
            c[u] = k < nnz ? __ldg(ci + k) : 0;
            v[u] = k < nnz ? __ldg(va + k) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) acc = fma(v[u], __ldg(x + c[u]), acc);
    }
    out[blockIdx.x * (long long)blockDim.x + threadIdx.x] = acc;
}

// Thread per row straight from global memory (rows of consecutive threads are
// adjacent, so a warp's value and column loads stay in the sectors L1 just
// fetched); gathers issued 8 at a time, summed in storage order.
template <typename T, int ASG>
__global__ void __launch_bounds__(kBlock)
k_spmv_scalar(int n, const int* __restrict__ rp, const int* __restrict__ ci, const T* __restrict__ va,
              const T* __restrict__ x, T* __restrict__ y)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int a = rp[i], e = rp[i + 1], q = fused_tail(a, e);
        T acc = T(0);
        int k = a;
        for (; k + 8 <= e; k += 8) {
            T xv[8], av[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) { av[u] = va[k + u]; xv[u] = x[ci[k + u]]; }
#pragma unroll
            for (int u = 0; u < 8; ++u) acc = row_step(acc, av[u], xv[u], k + u >= q);
        }
        T xv[8], av[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) if (k + u < e) { av[u] = va[k + u]; xv[u] = x[ci[k + u]]; }
#pragma unroll
        for (int u = 0; u < 8; ++u) if (k + u < e) acc = row_step(acc, av[u], xv[u], k + u >= q);
        const T base = (ASG == ASG_SET) ? T(0) : y[i];
        y[i] = assign_out<T, ASG>(base, acc);
    }
}

// ---------------------------------------------------------------- vector passes
enum VOp : int {
    VOP_DOT = 0,        // dots only
    VOP_AXPY,           // y += a x             (a = op.scalar)
    VOP_CG_UPDATE,      // x += alpha p ; r -= alpha q
    VOP_BI_P,           // p = r + beta (p - omega v)   (first: p = r)
    VOP_BI_S,           // s = r - alpha v
    VOP_BI_XR,          // x += omega shat + alpha phat ; r = s - omega t  (finishing: x += alpha phat)
    VOP_REF_CAST,       // r32 = float(r64 / scale); d = 0; z/r inner init
    VOP_REF_UPDATE,     // x64 += scale * double(d)
    VOP_FILL,           // v = scalar
    VOP_COPY,           // y = x
    VOP_SCALE_COPY,     // y = a x
};

struct VecOp {
    int op;
    int a, b, c, e, f, g;   // slots (meaning per op)
    int ndot;
    int da[kMaxDots], db[kMaxDots], dc[kMaxDots];
    int rk[kMaxDots];   // reference summation order of each dot (RK_*, refdot.cuh)
    int fin;
    int skip;
    int count_body;
    double scalar;
};

// The vectors a pass writes, as dot factors see them: op.a (what is computed
// first), and a second result (CG's and BiCGSTAB's r; the copies of the inner
// right-hand side).
template <int OP>
__device__ __forceinline__ int vec_out1(const VecOp& op)
{
    return OP == VOP_AXPY || OP == VOP_CG_UPDATE || OP == VOP_BI_P || OP == VOP_BI_S || OP == VOP_BI_XR ? op.a : SLOT_NONE;
}
template <int OP>
__device__ __forceinline__ bool vec_is_out2(const VecOp& op, int code)
{
    if (OP == VOP_CG_UPDATE) return code == op.c;
    if (OP == VOP_BI_XR) return code == op.g;
    if (OP == VOP_REF_CAST) return code == op.a || code == op.c || code == op.e;
    return false;
}

// Publishes a CTA's tally of a system's finished vector-pass tiles; the CTA
// that completes the system gathers its partials and finalizes (or retires a
// finishing BiCGSTAB system).
template <int OP>
__device__ __forceinline__ void vec_publish(const SetView& sv, const VecOp& op, TileTally& tally, double* s_red)
{
    const int count = int(tally.need);
    if (publish_tally(sv, tally)) {
        double tot[kMaxDots];
        gather_partials(sv, tally.sys, op.ndot, tot, s_red, count);
        if (threadIdx.x == 0) {
            SysState& s = sv.st[tally.sys];
            if (OP == VOP_BI_XR && (s.flags & FLAG_FINISHING)) {
                s.flags &= ~FLAG_FINISHING;
                retire(sv, s, (int)s.dots[3], s.error);
            } else {
                finalize(sv, op.fin, tally.sys, tot);
            }
        }
    }
}

constexpr int kVecGroup = 4;   // tiles a vector-pass CTA works on at once (one row of each per thread)

// A vector pass splits each system into row tiles of kTileRows (tile v:
// rows v kTileRows .. + kTileRows), as many as fit in the system's share of
// the SpMV tile indices (at least that many: SpMV tiles hold at most
// kTileRows rows), whose partial slots it uses.  One CTA per run of
// consecutive tile indices (the launch sizes the grid to the SMs),
// kVecGroup tiles of one system at a time (thread k takes row k of each, so
// its loads of the group's rows are in flight together, with no tile
// metadata to read); the system's vectors and scalars are read once per run.
// Each tile's partial dots are summed on their own in a fixed order, so the
// sums do not depend on the grid, the grouping or the batch.  ND (0, 1 or 2):
// the pass's dots; a group's are reduced together (warp_sums), and the warps'
// sums meet in shared memory only every kPartTiles tiles, so the streams of
// loads run on (FP64 BiCGSTAB x / r pass on 128^3: 84 us with a block
// reduction of 16 values per group, 57 us so; floor 20 us at 6.55 TB/s).
template <typename T, int OP, int ND>
__global__ void __launch_bounds__(kBlock, 2) k_vec(SetView sv, VecOp op)
{
    static_assert(kBlock == kTileRows, "a vector-pass thread takes one row of each tile");
    static_assert(kPartTiles % kVecGroup == 0, "whole groups of tiles wait in shared memory");
    constexpr int NV = ND > 0 ? ND : 1, NR = kVecGroup * NV;
    __shared__ double s_red[kMaxDots * 32];
    __shared__ double s_part[kPartTiles * (kBlock / 32) * NV];
    if (op.count_body && blockIdx.x == 0 && threadIdx.x == 0) {
        int runs = atomicAdd(&sv.err[1], 1) + 1;
        if (runs > sv.err[2] || *(volatile int*)sv.running <= 0) set_cond(sv, 0u);
    }
    const int t_begin = int((long long)sv.n_tiles * blockIdx.x / gridDim.x);
    const int t_end = int((long long)sv.n_tiles * (blockIdx.x + 1) / gridDim.x);
    TileTally tally;
    int t = t_begin;
    while (t < t_end) {
        // (a set of one system needs no look at the tiles)
        const bool one = sv.n_sys == 1;
        const int sys = one ? 0 : sv.tiles[t].sys;
        const int tb = one ? 0 : sv.sys_tile_begin[sys];
        const int te = one ? t_end : min(t_end, sv.sys_tile_begin[sys + 1]);   // this system's tile indices in the CTA's range
        const SysDesc& d = sv.desc[sys];
        const int n = d.n;   // its rows
        const int nvt = (n + kTileRows - 1) / kTileRows;                   // its row tiles
        if (sys != tally.sys) {
            vec_publish<OP>(sv, op, tally, s_red);
            tally.sys = sys;
            tally.need = unsigned(nvt);
        }
        SysState& s = sv.st[sys];
        if (skip_system(s, op.skip)) {
            t = te;
            continue;
        }
        const T* dinv = static_cast<const T*>(d.inv_diag);
        // Dot factors: a vector in memory, or a result of this pass (taken
        // from the register it was just computed in: 1 what A gets, 2 the
        // second result).
        const T* dm[2 * NV];
        int from[2 * NV];
        bool by_d[NV];
#pragma unroll
        for (int j = 0; j < ND; ++j) {
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const int code = k == 0 ? op.da[j] : op.db[j];
                from[2 * j + k] = code == vec_out1<OP>(op) ? 1 : vec_is_out2<OP>(op, code) ? 2 : 0;
                dm[2 * j + k] = from[2 * j + k] == 0 && names_vector(code) ? vptr<T>(d, code) : nullptr;
            }
            by_d[j] = op.dc[j] == OPND_D;
        }
        T* A = op.a != SLOT_NONE ? vptr<T>(d, op.a) : nullptr;
        T* B = op.b != SLOT_NONE ? vptr<T>(d, op.b) : nullptr;
        T* C = op.c != SLOT_NONE ? vptr<T>(d, op.c) : nullptr;
        T* E = op.e != SLOT_NONE ? vptr<T>(d, op.e) : nullptr;
        T* F = op.f != SLOT_NONE ? vptr<T>(d, op.f) : nullptr;
        T* G = op.g != SLOT_NONE ? vptr<T>(d, op.g) : nullptr;
        const bool finishing = (s.flags & FLAG_FINISHING) != 0;
        const T alpha = T(s.alpha), beta = T(s.beta), omega = T(s.omega);
        const bool first = (s.iter <= 1);
        const double scale = s.scale;
        const bool reduce = op.fin != FIN_NONE || (OP == VOP_BI_XR && finishing);
        int held = 0;   // tiles whose warp sums wait in shared memory
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        for (; t < te; t += kVecGroup) {
            const int v0 = t - tb;
            const int ng = max(0, min(min(kVecGroup, te - t), nvt - v0));   // row tiles among these indices
            double dot[NR];
#pragma unroll
            for (int k = 0; k < NR; ++k) dot[k] = 0.0;
            // all rows' loads, then their arithmetic and stores (a store
            // between them would hold the next row's loads back)
            T a[kVecGroup], b[kVecGroup], c[kVecGroup], e[kVecGroup], f[kVecGroup], dd[kVecGroup], m[kVecGroup][2 * NV];
            double w[kVecGroup];
            const int i0 = v0 * kTileRows + int(threadIdx.x);
#pragma unroll
            for (int q = 0; q < kVecGroup; ++q) {
                const int i = i0 + q * kTileRows;
                if (q >= ng || i >= n) continue;
                if (OP == VOP_AXPY || OP == VOP_CG_UPDATE || OP == VOP_BI_XR || (OP == VOP_BI_P && !first) || OP == VOP_REF_UPDATE) a[q] = A[i];
                if (OP == VOP_AXPY || OP == VOP_CG_UPDATE || OP == VOP_BI_P || OP == VOP_BI_S || OP == VOP_BI_XR || OP == VOP_COPY || OP == VOP_SCALE_COPY) b[q] = B[i];
                if (OP == VOP_CG_UPDATE || (OP == VOP_BI_P && !first) || OP == VOP_BI_S || (OP == VOP_BI_XR && !finishing)) c[q] = C[i];
                if (OP == VOP_CG_UPDATE || (OP == VOP_BI_XR && !finishing)) e[q] = E[i];
                if (OP == VOP_BI_XR && !finishing) f[q] = F[i];
                if (OP == VOP_REF_CAST) w[q] = d.r64[i];
                if (OP == VOP_REF_UPDATE) w[q] = d.x64[i];
#pragma unroll
                for (int j = 0; j < 2 * ND; ++j) if (from[j] == 0) m[q][j] = dm[j] ? dm[j][i] : T(1);
#pragma unroll
                for (int j = 0; j < ND; ++j) if (by_d[j]) dd[q] = dinv[i];
            }
#pragma unroll
            for (int q = 0; q < kVecGroup; ++q) {
                const int i = i0 + q * kTileRows;
                if (q >= ng || i >= n) continue;
                T o1 = T(0), o2 = T(0);
                if (OP == VOP_AXPY) {
                    o1 = fma(T(op.scalar), b[q], a[q]);                     // A += s B
                    A[i] = o1;
                } else if (OP == VOP_CG_UPDATE) {
                    o1 = fma(alpha, b[q], a[q]);                            // x += alpha p
                    o2 = fma(-alpha, e[q], c[q]);                           // r -= alpha q
                    A[i] = o1;
                    C[i] = o2;
                } else if (OP == VOP_BI_P) {
                    // p = r + beta * (p - omega * v)     (bicgstab.hpp:49-53)
                    o1 = first ? b[q] : fma(beta, fma(-omega, c[q], a[q]), b[q]);
                    A[i] = o1;
                } else if (OP == VOP_BI_S) {
                    o1 = fma(-alpha, c[q], b[q]);                           // s = r - alpha v
                    A[i] = o1;
                } else if (OP == VOP_BI_XR) {
                    // A x, B phat, C shat, E s, F t, G r
                    if (finishing) {
                        A[i] = fma(alpha, b[q], a[q]);                      // x += alpha phat
                    } else {
                        // x += omega shat + alpha phat, evaluated as the reference
                        // build does: x + fma(alpha, phat, omega shat)
                        o1 = a[q] + fma(alpha, b[q], omega * c[q]);
                        o2 = fma(-omega, f[q], e[q]);                       // r = s - omega t
                        A[i] = o1;
                        G[i] = o2;
                    }
                } else if (OP == VOP_REF_CAST) {
                    // inner right-hand side float(r64 / ||r64||); inner x = 0, r = b
                    o2 = T(w[q] / scale);
                    A[i] = o2;
                    if (B) B[i] = T(0);
                    if (C) C[i] = o2;
                    if (E) E[i] = o2;
                } else if (OP == VOP_REF_UPDATE) {
                    d.x64[i] = fma(scale, double(a[q]), w[q]);              // x += ||r|| * d
                } else if (OP == VOP_FILL) {
                    A[i] = T(op.scalar);
                } else if (OP == VOP_COPY) {
                    A[i] = b[q];
                } else if (OP == VOP_SCALE_COPY) {
                    A[i] = T(op.scalar) * b[q];
                }
#pragma unroll
                for (int j = 0; j < ND; ++j) {
                    const T x = from[2 * j] == 1 ? o1 : from[2 * j] == 2 ? o2 : m[q][2 * j];
                    const T y = from[2 * j + 1] == 1 ? o1 : from[2 * j + 1] == 2 ? o2 : m[q][2 * j + 1];
                    dot[q * NV + j] += double(x * y * (by_d[j] ? dd[q] : T(1)));
                }
            }
            if (!reduce || ng == 0) continue;
            if constexpr (ND > 0) {
                const double sum = warp_sums<NR>(dot);
                const int k = warp_sum_index<NR>(lane), q = k / NV;
                if (lane % (32 / NR) == 0 && q < ng) s_part[((held + q) * (kBlock / 32) + warp) * NV + k % NV] = sum;
                held += ng;
                if (held > kPartTiles - kVecGroup) {
                    flush_parts<NV>(sv, t + ng - held, held, s_part);
                    held = 0;
                }
            }
            tally.n += unsigned(ng);
        }
        if (ND > 0 && held) flush_parts<NV>(sv, tb + min(te - tb, nvt) - held, held, s_part);
        t = te;
    }
    vec_publish<OP>(sv, op, tally, s_red);
}

}  // namespace mtlg
