// Conjugate gradients on one small system in one launch (k_cg_small).
//
// The reference body (boost/numeric/itl/krylov/cg.hpp:40-111) without a
// preconditioner or with the diagonal one, for a system whose rows fit the
// running threads, R to a thread.  The same passes as k_spmv_short (XF_CG_P*)
// and k_vec<VOP_CG_UPDATE>, with the same sums to the bit, but the CTAs stay
// and meet twice per iteration.  What bounds such a solve is latency: two
// kernels an iteration cost 20 us at 65,536 rows (launch, tile metadata,
// partials, a last CTA that gathers them), while its bytes take 1 us.
// Measured (one B200, 256 x 256, FP64, diagonal): 20.9 -> 10.4 us an iteration;
// other sizes at the rule that chooses it (cg_small_rows).
//
// A meeting: every CTA puts its tiles' partial dots into cells of a buffer
// that is all sentinel before; CTA 0 polls the cells, adds them in
// gather_dots' order, runs the scalar update and leaves its outcome in a
// record (several copies, all sentinel before) that the others poll.  (With
// every CTA adding up all cells a meeting is one hop shorter, but the cells
// are then polled by all: 65,536 rows 14.2 us an iteration.)  Cells and
// records are used in a rotation of four: at meeting e the sentinel goes back
// into those of e + 2, last read at e - 2, and everybody has been through
// e - 1 since.  The residual update's meetings also order the vectors
// (release / acquire on both hops): what a CTA reads of its neighbours' r and
// p was stored before a meeting both have passed, and is read through L2.
// All CTAs run at once (cooperative launch); the polls are bounded (spin
// limit), after which the kernel records a timeout and returns.
#pragma once
#include "kernels.cuh"

namespace mtlg {

__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

constexpr int kCgCopies = 8;   // copies of a meeting's record, one 32-byte sector each

__host__ __device__ constexpr long long cg_cells(int nt) { return 8LL * nt + 4 * kCgCopies * 4; }

// Polls a cell until it holds a value (bounded: then +0, a timeout and stop).
__device__ __forceinline__ double cg_poll(const double* p, int* err, long long lim, int* s_stop)
{
    double v = ld_volatile(p);
    long long spins = 0;
    while (is_sentinel(v)) {
        if (++spins > lim || ((spins & 255) == 0 && *(volatile int*)err)) {
            atomicExch(err, 1);
            *(volatile int*)s_stop = 1;
            return 0.0;
        }
        v = ld_volatile(p);
    }
    return v;
}

// One meeting: the CTA's per-warp sums (s_part: [row group][warp][dot]) of
// its tiles out, the outcome in: out[0] the new alpha (ALPHA) or beta, out[1]
// the status.  lv: CTA 0's view of its copy of the state.
template <int R, int ND, bool ORDER>
__device__ __forceinline__ void cg_meet(const SetView& sv, const SetView& lv, int fin, double* cells, int e, int nt,
                                        const double* s_part, double* s_red, int* s_stop, double* s_out)
{
    constexpr int NWP = kBlock / 32;
    double* buf = cells + (long long)(e & 3) * 2 * nt;
    double* old = cells + (long long)((e + 2) & 3) * 2 * nt;
    double* rec = cells + 8LL * nt + (e & 3) * kCgCopies * 4;
    double* orec = cells + 8LL * nt + ((e + 2) & 3) * kCgCopies * 4;
    const long long lim = sv.spin > 0 ? sv.spin : kSpinLimit;
    __syncthreads();
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x, r = lane / ND, j = lane % ND, tile = int(blockIdx.x) + r * int(gridDim.x);
        const bool mine = lane < R * ND && tile < nt;
        double part = 0.0;
        if (mine) {
            const double* w = s_part + r * NWP * ND + j;
            double t[NWP];
#pragma unroll
            for (int q = 0; q < NWP; ++q) t[q] = w[q * ND] + 0.0;   // as flush_parts
            part = unsentinel(((t[0] + t[4]) + (t[2] + t[6])) + ((t[1] + t[5]) + (t[3] + t[7])));
            st_volatile(old + (long long)j * nt + tile, sentinel_value<double>());
        }
        __syncwarp();
        if (ORDER) fence_gpu();
        if (mine) st_volatile(buf + (long long)j * nt + tile, part);
    }
    if (blockIdx.x == 0) {
        double sum[ND];
#pragma unroll
        for (int j = 0; j < ND; ++j) {
            sum[j] = 0.0;
            for (int t = threadIdx.x; t < nt; t += kBlock) sum[j] += cg_poll(buf + (long long)j * nt + t, sv.err, lim, s_stop);
        }
        if (ORDER) fence_gpu();
        block_reduce<ND>(sum, s_red);
        if (threadIdx.x == 0) {
            double tot[kMaxDots] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
            for (int j = 0; j < ND; ++j) tot[j] = sum[j];
            finalize(lv, fin, 0, tot);
            s_out[0] = unsentinel(fin == FIN_CG_ALPHA ? lv.st[0].alpha : lv.st[0].beta);
            s_out[1] = double(lv.st[0].status);
        }
        __syncthreads();
        if (threadIdx.x < 32) {
            const int k = threadIdx.x;
            if (k < kCgCopies * 2) st_volatile(orec + (k / 2) * 4 + k % 2, sentinel_value<double>());
            __syncwarp();
            if (ORDER) fence_gpu();
            if (k < kCgCopies * 2) st_volatile(rec + (k / 2) * 4 + k % 2, s_out[k % 2]);
        }
    } else {
        if (threadIdx.x < 2) s_out[threadIdx.x] = cg_poll(rec + (blockIdx.x % kCgCopies) * 4 + threadIdx.x, sv.err, lim, s_stop);
        if (ORDER && threadIdx.x < 32) fence_gpu();
        __syncthreads();
    }
}

// JAC: diagonal preconditioner.  cells: cg_cells(n_tiles) doubles, all sentinel.
template <typename T, bool JAC, int R>
__global__ void __launch_bounds__(kBlock, 1) k_cg_small(SetView sv, double* cells)
{
    constexpr int NWP = kBlock / 32, ND = JAC ? 2 : 1;
    __shared__ SysState s;
    __shared__ int s_running, s_stop;
    __shared__ double s_red[kMaxDots * 32];
    __shared__ double s_part[R * NWP * 2], s_out[2];
    static_assert(sizeof(SysState) % 4 == 0, "copied as words");
    for (int k = threadIdx.x; k < int(sizeof(SysState) / 4); k += kBlock)
        reinterpret_cast<unsigned*>(&s)[k] = reinterpret_cast<const unsigned*>(sv.st)[k];
    if (threadIdx.x == 0) {
        s_running = *sv.running;
        s_stop = 0;
    }
    __syncthreads();
    if (s.status != MTLG_ST_RUNNING) return;
    SetView lv = sv;   // the scalar updates on CTA 0's copy of the state
    lv.st = &s;
    lv.running = &s_running;
    lv.use_cond = 0;

    const SysDesc& d = sv.desc[0];
    const int n = d.n, nt = sv.n_tiles, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int* __restrict__ rp = d.rp;
    const int* __restrict__ ci = d.ci;
    const T* __restrict__ va = static_cast<const T*>(d.val);
    const T* __restrict__ dinv = static_cast<const T*>(d.inv_diag);
    T* X = vptr<T>(d, SLOT_X);
    T* RV = vptr<T>(d, V_R);
    T* P = vptr<T>(d, V_P0);
    T* PN = vptr<T>(d, V_P1);
    int row[R];
    int2 ae[R];
    T x[R], rv[R], di[R], p[R], q[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const long long i = (long long)(int(blockIdx.x) + r * int(gridDim.x)) * kTileRows + threadIdx.x;
        row[r] = i < n ? int(i) : -1;
        ae[r] = make_int2(0, 0);
        x[r] = rv[r] = di[r] = p[r] = q[r] = T(0);
        if (row[r] >= 0) {
            ae[r] = make_int2(rp[i], rp[i + 1]);
            x[r] = X[i];
            rv[r] = RV[i];
            if (JAC) di[r] = dinv[i];
        }
    }
    // the first 8 entries of a row stay in registers where they fit: the
    // meetings' fences leave nothing in L1
    constexpr bool KEEP = R <= 2;
    constexpr int RK = KEEP ? R : 1;
    int cc[RK][8];
    T aa[RK][8], dj[RK][8];
    if (KEEP) {
#pragma unroll
        for (int r = 0; r < RK; ++r)
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const bool in = ae[r].x + u < ae[r].y;
                cc[r][u] = in ? ci[ae[r].x + u] : 0;
                aa[r][u] = in ? va[ae[r].x + u] : T(0);
                dj[r][u] = JAC && in ? dinv[cc[r][u]] : T(0);
            }
    }
    bool first = s.iter == 0;
    T beta = T(s.beta);
    for (int e = 0;; e += 2) {
        // p = z + beta p; q = A p; p.q  (z = r or D r; first: p = z)
        auto dir = [&](T zr, T dj, T pj) {
            const T z = JAC ? dj * zr : zr;
            return first ? z : fma(beta, pj, z);
        };
#pragma unroll
        for (int r = 0; r < R; ++r) {
            double d0 = 0.0;
            if (row[r] >= 0) {
                const int a = ae[r].x, en = ae[r].y, tail = fused_tail(a, en);
                T acc = T(0);
                if (KEEP) {
                    T xv[8];
#pragma unroll
                    for (int u = 0; u < 8; ++u)
                        if (a + u < en)
                            xv[u] = dir(__ldcg(RV + cc[r % RK][u]), dj[r % RK][u], first ? T(0) : __ldcg(P + cc[r % RK][u]));
#pragma unroll
                    for (int u = 0; u < 8; ++u) if (a + u < en) acc = row_step(acc, aa[r % RK][u], xv[u], a + u >= tail);
                }
                for (int k = KEEP ? a + 8 : a; k < en; k += 8) {
                    T xv[8], av[8];
#pragma unroll
                    for (int u = 0; u < 8; ++u)
                        if (k + u < en) {
                            const int c = ci[k + u];
                            av[u] = va[k + u];
                            xv[u] = dir(__ldcg(RV + c), JAC ? dinv[c] : T(0), first ? T(0) : __ldcg(P + c));
                        }
#pragma unroll
                    for (int u = 0; u < 8; ++u) if (k + u < en) acc = row_step(acc, av[u], xv[u], k + u >= tail);
                }
                p[r] = dir(rv[r], di[r], p[r]);
                q[r] = acc;
                __stcg(PN + row[r], p[r]);
                d0 += double(p[r] * acc * T(1));
            }
            double dd[1] = {d0};
            const double sum = warp_sums<1>(dd);
            if (lane == 0) s_part[r * NWP + warp] = sum;
        }
        cg_meet<R, 1, false>(sv, lv, FIN_CG_ALPHA, cells, e, nt, s_part, s_red, &s_stop, s_out);
        if (*(volatile int*)&s_stop) return;
        // x += alpha p; r -= alpha q; r.r (and r.D r)
        const T alpha = T(s_out[0]);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            double dd[ND];
#pragma unroll
            for (int j = 0; j < ND; ++j) dd[j] = 0.0;
            if (row[r] >= 0) {
                x[r] = fma(alpha, p[r], x[r]);
                rv[r] = fma(-alpha, q[r], rv[r]);
                __stcg(RV + row[r], rv[r]);
                dd[0] += double(rv[r] * rv[r] * T(1));
                if (JAC) dd[ND - 1] += double(rv[r] * rv[r] * di[r]);
            }
            const double sum = warp_sums<ND>(dd);
            if (lane % (32 / ND) == 0) s_part[(r * NWP + warp) * ND + warp_sum_index<ND>(lane)] = sum;
        }
        cg_meet<R, ND, true>(sv, lv, JAC ? FIN_CG_UPDATE_JAC : FIN_CG_UPDATE, cells, e + 1, nt, s_part, s_red, &s_stop, s_out);
        if (*(volatile int*)&s_stop) return;
        if (int(s_out[1]) != MTLG_ST_RUNNING) break;
        beta = T(s_out[0]);
        first = false;
        T* const t = P;
        P = PN;
        PN = t;
    }
#pragma unroll
    for (int r = 0; r < R; ++r)
        if (row[r] >= 0) X[row[r]] = x[r];
    if (blockIdx.x == 0) {
        for (int k = threadIdx.x; k < int(sizeof(SysState) / 4); k += kBlock)
            reinterpret_cast<unsigned*>(sv.st)[k] = reinterpret_cast<const unsigned*>(&s)[k];
        if (threadIdx.x == 0) *sv.running = s_running;
    }
}

}  // namespace mtlg
