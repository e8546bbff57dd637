// Partial-pivot LU of a dense complex FP64 matrix and its triangular solves
// (solve.rs:166-171 -> nalgebra lu() / solve_mut): pivots by the first row of
// the largest |re| + |im| (icamax), results at FP64 accuracy.
//
// GB300 runs FP64 arithmetic at two multiply-adds per clock and SM (1.2
// TFLOP/s for the whole chip), so the O(n^3) part leaves the FP64 pipe: the
// trailing update is an exact fixed-point product on the tensor cores
// (Ozaki's error-free splitting: Ozaki, Ogita, Oishi and Rump 2012; on FP16
// tensor cores Mukunoki et al. 2020).  The matrix advances in blocks of 32
// columns, per block:
//
//   panel  a thread-block cluster holds the block's columns in its shared
//          memory and factors them column by column; one exchange of stores
//          counted on barriers per column.  A tall block is cut into narrower panels that
//          fit, and the rest of the block's columns take a panel's update over
//          the whole GPU (lu64_mid_kernel).
//   rows   the columns right of the block take the block's row exchanges,
//          become U12 = L11^-1 A12 (FP64) and are split into digits; L21 is
//          split by the same launch.
//   gemm   A22 -= L21 U12 from the digits (tcgen05, FP16 operands, FP32
//          accumulation that is exact), one FP64 subtraction per entry; the
//          first tile of columns ahead of the others, which run beside the next
//          block's panel.
//
// Device time of one factorization and solve, against one launch per column,
// FP64 tiles for the trailing update and one thread per triangular block before:
// n = 324 10.2 -> 1.5 ms, n = 2001 99 -> 11.0 ms, n = 6144 776 -> 63.7 ms.
//
// Beside the factors the row order and the inverses of the diagonal blocks are
// kept; the substitutions run over the whole GPU (lu64_solve_kernel).
//
// Digits.  An entry x of L21 (row i) is stored relative to the largest entry
// of its row as I 2^-56 with |I| <= 2^55, I cut into seven digits of eight bits
// in [-128, 128]; U12 likewise relative to the largest of its column.  Digit
// products are integers <= 2^14, a sum over K = 64 (32 complex entries) of at
// most seven of them stays below 2^23, so FP32 accumulation has no rounding at
// all.  Of the 49 digit products the 34 of weight 256^-2 ... 256^-9 are formed,
// in eight groups of equal weight; the groups are added in 64-bit integers and
// rounded once to FP64.  What the splitting, the rounding and the products left
// out lose is about 2^-54 of (largest of the row) x (largest of the column): a
// chain of 32 FP64 multiply-adds rounds 64 times at 2^-54 of its partial sums.
// (Without the group of weight 256^-9 the products left out were the largest
// error, and x had half again to twice the error of FP64 elimination; the group
// costs 9 % at n = 6144.  With it, geometric mean of the error of x over random
// matrices, against FP64 tiles: n = 324 5.3e-14 / 9.4e-14, 1300 3.8e-13 / 7.0e-13,
// 2001 1.4e-12 / 1.9e-12.)
//
// The columns of L21 and the rows of U12 are scaled against each other by the
// exponent of the column's largest entry once the block's exchanges are done, so
// that a matrix whose rows or columns differ by orders of magnitude keeps that
// bound for each of them.  It is a bound by the largest of a row and of a column:
// an entry below an eighth of it has fewer than FP64's 53 bits.  What that means
// for rows scaled over 18 decades, where hardly a pivot is chosen for its size and
// the largest entry says less of the others (400 to 600 matrices up to n = 100, 16
// of n = 1100, against FP64 elimination): the largest |b - A x|_i / (|A| |x|)_i is
// 0.88 of FP64's at n = 40, 0.62 at 100, 0.17 at 1100; the error of x 1.22, 1.16 and
// 0.93 of FP64's.  Without such scales both are smaller at every size: 0.78, 0.56,
// 0.17 and 0.92, 0.85, 0.63.
#include <cooperative_groups.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <functional>

#include "cluster.cuh"
#include "common.cuh"
#include "complex.cuh"
#include "umma.cuh"

namespace cg = cooperative_groups;

namespace bem {

int* device_err(Context& ctx);
void check_device_err(Context& ctx);

namespace {

constexpr int NB = 32;        // columns per block
constexpr int SLICES = 7;     // digits per entry
constexpr int GROUPS = SLICES + 1;  // groups of digit products of equal weight
constexpr int TM = 128;       // tile rows (real): 64 complex rows
constexpr int TN = 64;        // tile columns
constexpr uint32_t A_SLICE = TM * 128, B_SLICE = TN * 128;  // 64 halves = 128 bytes per row
constexpr uint32_t A_IMG = SLICES * A_SLICE, B_IMG = SLICES * B_SLICE;
constexpr int EXP_NONE = -(1 << 20);  // exponent of zero; the sum of any two exponents
// with an EXP_BAD among them is far outside the range of numbers
constexpr int EXP_BAD = 1 << 22;      // row or column with an infinity or a NaN

// ---------------------------------------------------------------------------
// Row exchanges of one block (or of one panel): position top0 + t (t < 32)
// receives the row that was at top[t], position opos[q] the row that was at
// osrc[q] (q < count); both relative to the first column of the block.
struct RowMoves {
    int top[NB], opos[NB], osrc[NB];
    int count, pad[31];
};

// Exchanges (position j < lim with position p) collected in a RowMoves held in
// the 32 lanes of a warp.
struct LaneMoves {
    int top, opos, osrc, count, lim;  // positions below lim are the top rows
    __device__ __forceinline__ void start(int lane, int limit) {
        top = lane;
        opos = -1;
        osrc = -1;
        count = 0;
        lim = limit;
    }
    __device__ __forceinline__ void exchange(int j, int p, int lane) {
        if (j == p) return;
        const unsigned all = 0xffffffffu;
        const int cj = __shfl_sync(all, top, j);
        int cp;
        if (p < lim) {
            cp = __shfl_sync(all, top, p);
            if (lane == p) top = cj;
        } else {
            const unsigned hit = __ballot_sync(all, opos == p);
            if (hit) {
                const int l = __ffs(hit) - 1;
                cp = __shfl_sync(all, osrc, l);
                if (lane == l) osrc = cj;
            } else {
                cp = p;
                if (lane == count) {
                    opos = p;
                    osrc = cj;
                }
                ++count;
            }
        }
        if (lane == j) top = cp;
    }
    __device__ __forceinline__ void store(RowMoves* m, int lane) const {
        m->top[lane] = top;
        m->opos[lane] = opos;
        m->osrc[lane] = osrc;
        if (lane == 0) m->count = count;
    }
    __device__ __forceinline__ void load(const RowMoves* m, int lane) {
        top = m->top[lane];
        opos = m->opos[lane];
        osrc = m->osrc[lane];
        count = m->count;
    }
};

// acc -= b c (negations as operand modifiers: a negated value on its own costs
// an FP64 instruction).
__device__ __forceinline__ void cfms(z2& acc, z2 b, z2 c) {
    acc.x = fma(-b.x, c.x, fma(b.y, c.y, acc.x));
    acc.y = fma(-b.x, c.y, fma(-b.y, c.x, acc.y));
}

// Smallest e with |v| < 2^e (subnormals count as 2^-1022).
__device__ __forceinline__ int exp_above(double v) {
    const int e = (int)((__double_as_longlong(v) >> 52) & 0x7ff);
    if (e == 0x7ff) return EXP_BAD;
    if (v == 0.0) return EXP_NONE;
    return max(e, 1) - 1022;
}

// ---------------------------------------------------------------------------
// Panel: columns [c0, c0 + w) of the rows c0 .. n - 1, rpc rows (a multiple of
// 32) per CTA of the cluster, resident in shared memory.  Per column every CTA
// sends its largest entry's row to all others (asynchronous stores counted on
// an mbarrier in the receiver: a step can run ahead of the slowest CTA by one,
// so two sets of buffers do); then every CTA picks the winner, while a second
// warp inverts all candidates, one per lane.  The rank-1 update of the other
// columns runs one step behind, while the rows travel; only the next column is
// updated at once.
//
// What bounds it: an FP64 instruction of a warp occupies the FP64 pipe of its
// SM quarter for 65 clocks, however many lanes are active, so the chain of a
// column is its 16 dependent FP64 instructions, the rows' way and three
// reductions, and a tall panel is limited by (rows / 32) x (columns) x 4 such
// instructions on the cluster's 64 quarters.  (With a cluster barrier per
// column and remote reads behind it a column took 2.7 us: the barrier's release
// waits for every outstanding store, 1100 clocks.)
constexpr int PANEL_WORKERS = 256, PANEL_THREADS = PANEL_WORKERS + 32, PANEL_WARPS = PANEL_WORKERS / 32;
constexpr size_t PANEL_SMEM = 200 * 1024;  // beside 20 KB of static shared memory
constexpr unsigned NO_ROW = 0x7fffffffu;

struct Cand {
    unsigned hi, lo, row;
};

__device__ __forceinline__ Cand warp_best(unsigned hi, unsigned lo, unsigned row) {
    const unsigned all = 0xffffffffu;
    Cand c;
    c.hi = __reduce_max_sync(all, hi);
    c.lo = __reduce_max_sync(all, hi == c.hi ? lo : 0u);
    c.row = __reduce_min_sync(all, hi == c.hi && lo == c.lo ? row : NO_ROW);
    return c;
}

// The larger of the candidate and (|v.x| + |v.y|, row); rows ascend.
__device__ __forceinline__ void consider(Cand& best, double2 v, unsigned row) {
    const double a = fabs(v.x) + fabs(v.y);
    const unsigned hi = (unsigned)__double2hiint(a), lo = (unsigned)__double2loint(a);
    if (hi > 0x7ff00000u || (hi == 0x7ff00000u && lo != 0u)) return;  // a NaN is no pivot
    if (best.row == NO_ROW || hi > best.hi || (hi == best.hi && lo > best.lo)) best = Cand{hi, lo, row};
}

// 1 / d (0 for d = 0): |d|^-2 from the FP32 reciprocal and one third-order
// correction, three FP64 instructions where a division takes ten.
__device__ __forceinline__ double2 recip(double2 d) {
    const double den = fma(d.x, d.x, d.y * d.y);
    double r;
    const int e = (__double2hiint(den) >> 20) & 0x7ff;
    if (e > 1023 - 120 && e < 1023 + 120) {
        r = (double)__frcp_rn((float)den);
        const double c = fma(-den, r, 1.0);
        r = fma(r, fma(c, c, c), r);
    } else {
        // |d|^2 near or past the ends of the range: scaled by a power of two
        const int k = max(exp_above(d.x), exp_above(d.y));
        if (k <= EXP_NONE || k >= EXP_BAD) {
            r = k <= EXP_NONE ? 0.0 : 1.0 / den;
        } else {
            const double x = scalbn(d.x, -k), y = scalbn(d.y, -k);
            r = 1.0 / fma(x, x, y * y);
            return make_double2(scalbn(x * r, -k), scalbn(-y * r, -k));
        }
    }
    return make_double2(d.x * r, -d.y * r);
}

// Bounded wait for data written by other CTAs of the cluster.
__device__ __forceinline__ void wait_peers(uint64_t* bar, uint32_t phase, int* err) {
    if (!peers_arrived(bar, phase)) atomicOr(err, DEVERR_MBAR_TIMEOUT);
}

__global__ void __launch_bounds__(PANEL_THREADS, 1)
    lu64_panel_kernel(int64_t n, double2* __restrict__ A, int64_t lda, int64_t c0, int w, int64_t b0, int nb, int rpc,
                      RowMoves* __restrict__ moves, int* __restrict__ cexp, double2* __restrict__ pinv,
                      int* __restrict__ info, int* __restrict__ err) {
    extern __shared__ double2 P[];  // w x rpc, column-major
    // what the CTAs send one another, by parity of the step: key and row of
    // every CTA's candidate, and row j
    __shared__ uint4 ckey[2][MAX_CLUSTER];
    __shared__ double2 crow[2][MAX_CLUSTER][NB], drow[2][NB];
    __shared__ uint64_t mb[2];
    __shared__ double2 cinv[MAX_CLUSTER], prow[2][NB], sinv[NB];
    __shared__ Cand wred[PANEL_WARPS];
    __shared__ int piv[2], prank;
    __shared__ RowMoves own;
    cg::cluster_group cl = cg::this_cluster();
    const int cs = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const bool worker = warp < PANEL_WARPS;
    const int64_t R = n - c0;
    const int row0 = rank * rpc;
    const int nr = (int)max((int64_t)0, min((int64_t)rpc, R - row0)), chunks = (nr + 31) / 32;
    const uint32_t step_bytes = 16u * (uint32_t)(cs * (1 + w) + w);
    double2* Ag = A + c0 * lda + c0 + row0;
    if (tid == 0) {
        mbar_init(&mb[0], 1);
        mbar_init(&mb[1], 1);
        fence_mbar_init();
    }
    Cand best{0u, 0u, NO_ROW};
    if (worker) {
        for (int q = warp; q < w; q += PANEL_WARPS)
            for (int lr = lane; lr < nr; lr += 32) P[q * rpc + lr] = Ag[(int64_t)q * lda + lr];
    }
    LaneMoves mown, mblk;  // the extra warp of rank 0 follows the exchanges
    mown.start(lane, w);
    mblk.start(lane, NB);
    if (!worker && rank == 0 && c0 > b0) mblk.load(moves, lane);
    cl.sync();  // barriers ready everywhere, the panel loaded
    if (worker)
        for (int lr = tid; lr < nr; lr += PANEL_WORKERS) consider(best, P[lr], (unsigned)(row0 + lr));
    for (int j = 0; j < w; ++j) {
        const int par = j & 1;
        const uint32_t bar = smem_u32(&mb[par]);
        if (worker) {
            const Cand c = warp_best(best.hi, best.lo, best.row);
            if (lane == 0) wred[warp] = c;
        }
        if (tid == 0) mbar_arrive_expect_tx(&mb[par], step_bytes);
        __syncthreads();
        if (worker) {
            // this CTA's candidate row, as it stands: its columns right of j
            // still lack step j - 1, which the receivers add.  Every warp sends
            // to its share of the CTAs; row j lives in CTA 0 (rpc >= w > j).
            Cand c = lane < PANEL_WARPS ? wred[lane] : Cand{0u, 0u, NO_ROW};
            c = warp_best(c.hi, c.lo, c.row);
            const uint4 v = lane < w && c.row != NO_ROW ? as_uint4(P[lane * rpc + (int)c.row - row0])
                                                         : make_uint4(0u, 0u, 0u, 0u);
            for (int d = warp; d < cs; d += PANEL_WARPS) {
                const uint32_t to = peer_addr(bar, d);
                if (lane < w) st_async16(peer_addr(smem_u32(&crow[par][rank][lane]), d), to, v);
                if (lane == 0)
                    st_async16(peer_addr(smem_u32(&ckey[par][rank]), d), to, make_uint4(c.hi, c.lo, c.row, 0u));
                if (rank == 0 && lane < w)
                    st_async16(peer_addr(smem_u32(&drow[par][lane]), d), to, as_uint4(P[lane * rpc + j]));
            }
        }
        __syncthreads();  // the rows are read before the update below touches them
        if (worker && j > 0) {
            const double2* lc = P + (j - 1) * rpc;
            const int first = max(0, j - row0), tasks = (w - 1 - j) * chunks;
            for (int t = warp; t < tasks; t += PANEL_WARPS) {
                const int q = j + 1 + t / chunks, lr = (t % chunks) * 32 + lane;
                if (lr < first || lr >= nr) continue;
                cfms(P[q * rpc + lr], lc[lr], prow[par ^ 1][q]);
            }
        }
        __syncthreads();  // the swap below follows the update above
        if (warp == 0) {
            wait_peers(&mb[par], (uint32_t)((j >> 1) & 1), err);
            const uint4 e = lane < cs ? ckey[par][lane] : make_uint4(0u, 0u, NO_ROW, 0u);
            const Cand c = warp_best(e.x, e.y, e.z);
            const bool any = c.row != NO_ROW;
            const int p = any ? (int)c.row : j;
            const int po = any ? __ffs(__ballot_sync(0xffffffffu, e.z == c.row)) - 1 : 0;  // its CTA
            if (lane == 0) {
                piv[par] = p;
                prank = any ? po : -1;
                if (rank == 0 && any && c.hi == 0u && c.lo == 0u && *info == 0) *info = (int)(c0 + j + 1);
            }
            if (lane < w) {
                const double2* row = any ? crow[par][po] : drow[par];
                const bool late = j > 0 && lane > j;
                double2 pv = row[lane];
                if (late) cfms(pv, row[j - 1], prow[par ^ 1][lane]);
                prow[par][lane] = pv;
                if (p != j) {
                    if (rank == po) {
                        double2 dv = drow[par][lane];
                        if (late) cfms(dv, drow[par][j - 1], prow[par ^ 1][lane]);
                        P[lane * rpc + p - row0] = dv;
                    }
                    if (rank == 0) P[lane * rpc + j] = pv;
                }
            }
        } else if (warp == 1) {
            wait_peers(&mb[par], (uint32_t)((j >> 1) & 1), err);
            if (lane < cs && ckey[par][lane].z != NO_ROW) cinv[lane] = recip(crow[par][lane][j]);
        }
        __syncthreads();
        if (worker) {
            const double nan = __longlong_as_double(0x7ff8000000000000ll);
            const double2 inv = prank >= 0 ? cinv[prank] : make_double2(nan, nan);
            const double2 u = prow[par][min(j + 1, NB - 1)];
            double2* lc = P + j * rpc;
            best = Cand{0u, 0u, NO_ROW};
            for (int lr = tid; lr < nr; lr += PANEL_WORKERS) {
                if (row0 + lr <= j) continue;
                const double2 l = cmul(lc[lr], inv);
                lc[lr] = l;
                if (j + 1 < w) {
                    double2 v = lc[rpc + lr];
                    cfms(v, l, u);
                    lc[rpc + lr] = v;
                    consider(best, v, (unsigned)(row0 + lr));
                }
            }
            if (tid == 0) sinv[j] = inv;
        } else if (rank == 0) {
            const int p = piv[par], sh = (int)(c0 - b0);
            mown.exchange(j, p, lane);
            mblk.exchange(sh + j, sh + p, lane);
        }
    }
    if (!worker && rank == 0) {
        mown.store(&own, lane);
        mblk.store(moves, lane);
    }
    cl.sync();
    // (behind the barrier: the last column's reciprocal is thread 0's)
    if (warp == 0 && rank == 0 && lane < w) pinv[c0 - b0 + lane] = sinv[lane];
    // The block's last panel takes the largest entry of each column of L21: before
    // its exchanges the rows below the block are not final.
    const bool last = c0 + w == b0 + nb;
    if (worker) {
        // the factored panel
        const int below = last ? (int)(b0 + nb - c0) - row0 : nr;
        for (int q = warp; q < w; q += PANEL_WARPS) {
            int e = EXP_NONE;
            for (int lr = lane; lr < nr; lr += 32) {
                const double2 v = P[q * rpc + lr];
                Ag[(int64_t)q * lda + lr] = v;
                if (lr >= below) e = max(e, max(exp_above(v.x), exp_above(v.y)));
            }
            e = __reduce_max_sync(0xffffffffu, e);
            if (lane == 0 && e != EXP_NONE) atomicMax(cexp + (c0 - b0) + q, e);
        }
    }
    if (w < nb) {
        // the block's other columns: this panel's exchanges, and for those on
        // the right the panel's rows of U (one warp per column)
        const double2* P0 = cl.map_shared_rank(P, 0);
        const RowMoves* mv = cl.map_shared_rank(&own, 0);
        double2(*top)[NB] = reinterpret_cast<double2(*)[NB]>(crow);  // the panel's unit lower block
        static_assert(sizeof(crow) >= sizeof(double2) * NB * NB, "");
        for (int t = tid; t < w * w; t += PANEL_THREADS) top[t / w][t % w] = P0[(t / w) * rpc + t % w];
        __syncthreads();
        const int left = (int)(c0 - b0);
        for (int i = rank + cs * warp; i < nb - w; i += cs * (PANEL_THREADS / 32)) {
            const int64_t c = b0 + (i < left ? i : i + w);
            double2* col = A + c * lda + c0;
            const int cnt = mv->count;
            double2 x = make_double2(0, 0), y = x;
            if (lane < w) x = col[mv->top[lane]];
            if (lane < cnt) y = col[mv->osrc[lane]];
            __syncwarp();
            if (lane < cnt) col[mv->opos[lane]] = y;
            if (i >= left) {
                for (int q = 0; q < w; ++q) {
                    double2 xq;
                    xq.x = __shfl_sync(0xffffffffu, x.x, q);
                    xq.y = __shfl_sync(0xffffffffu, x.y, q);
                    if (lane > q && lane < w) cfms(x, top[q][lane], xq);
                }
            }
            if (lane < w) col[lane] = x;
        }
        // The columns of the block's earlier panels (all of them on the left), each
        // by the CTA that has just exchanged its rows.  Maxima kept from the earlier
        // panels would still count rows that a later one moved up into the block:
        // 24 rows a billion times the others, n = 1100, cost the others seven
        // digits.  The pass takes 0.7 us per block (n = 6144: 63.51 -> 63.63 ms).
        if (last) {
            __shared__ int most;
            for (int i = rank; i < left; i += cs) {
                if (tid == 0) most = EXP_NONE;
                __syncthreads();
                const double2* col = A + (b0 + i) * lda;
                int e = EXP_NONE;
#pragma unroll 4
                for (int64_t r = b0 + nb + tid; r < n; r += PANEL_THREADS)
                    e = max(e, max(exp_above(col[r].x), exp_above(col[r].y)));
                e = __reduce_max_sync(0xffffffffu, e);
                if (lane == 0) atomicMax(&most, e);
                __syncthreads();
                if (tid == 0) cexp[i] = most;
            }
        }
    }
    cl.sync();  // shared memory stays up while other CTAs read it
}

// The rest of a block's columns [c1, c1 + nc) after the panel [c0, c0 + w),
// c1 = c0 + w: rows below c1 take A -= L U in FP64.  One warp per 32 rows and 2
// columns: short chains on as many FP64 pipes as there are (a warp with 8
// columns took 21 us at any size).
constexpr int MID_COLS = 2;
__global__ void __launch_bounds__(32) lu64_mid_kernel(int64_t n, double2* __restrict__ A, int64_t lda, int64_t c0,
                                                      int w, int nc) {
    const int64_t c1 = c0 + w, cc = c1 + (int64_t)blockIdx.y * MID_COLS;
    const int ncol = min(MID_COLS, nc - (int)blockIdx.y * MID_COLS), lane = threadIdx.x;
    double2 u[MID_COLS];  // lane q holds U's row q
#pragma unroll
    for (int c = 0; c < MID_COLS; ++c)
        u[c] = lane < w && c < ncol ? A[(cc + c) * lda + c0 + lane] : make_double2(0, 0);
    const int64_t r = c1 + (int64_t)blockIdx.x * 32 + lane, rr = r < n ? r : n - 1;
    double2 acc[MID_COLS];
#pragma unroll
    for (int c = 0; c < MID_COLS; ++c) acc[c] = A[(c < ncol ? cc + c : cc) * lda + rr];
    for (int q0 = 0; q0 < w; q0 += 8) {
        double2 l[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) l[q] = q0 + q < w ? A[(c0 + q0 + q) * lda + rr] : make_double2(0, 0);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            if (q0 + q >= w) break;
#pragma unroll
            for (int c = 0; c < MID_COLS; ++c) {
                double2 v;
                v.x = __shfl_sync(0xffffffffu, u[c].x, q0 + q);
                v.y = __shfl_sync(0xffffffffu, u[c].y, q0 + q);
                cfms(acc[c], l[q], v);
            }
        }
    }
    if (r >= n) return;
#pragma unroll
    for (int c = 0; c < MID_COLS; ++c)
        if (c < ncol) A[(cc + c) * lda + r] = acc[c];
}

// ---------------------------------------------------------------------------
// Digits.  v = I 2^(e - 55) rounded, |v| < 2^e, biased so that every digit is a
// byte: digit s (s = 0 highest) of v is field(u, s) - 128.
__device__ __forceinline__ uint64_t digits_of(double v, int e) {
    const uint64_t b = (uint64_t)__double_as_longlong(v);
    const int ex = (int)((b >> 52) & 0x7ff);
    const uint64_t m = (b & 0xfffffffffffffull) | (ex ? 0x10000000000000ull : 0ull);
    const int sh = max(ex, 1) - 1075 + 55 - e;  // <= 2
    uint64_t I;
    if (sh >= 0) I = m << sh;
    else if (sh > -55) I = (m + (1ull << (-sh - 1))) >> -sh;
    else I = 0;
    const int64_t s = (b >> 63) ? -(int64_t)I : (int64_t)I;
    return (uint64_t)(s + 0x80808080808080ll);
}
// The digits s of a real and an imaginary part as a pair of halves.
__device__ __forceinline__ uint32_t digit_pair(uint64_t re, uint64_t im, int s) {
    const int sh = 8 * (SLICES - 1 - s);
    const uint32_t a = s == 0 ? (uint32_t)(re >> sh) : (uint32_t)(re >> sh) & 0xffu;
    const uint32_t b = s == 0 ? (uint32_t)(im >> sh) : (uint32_t)(im >> sh) & 0xffu;
    const uint32_t bits = (0x6400u + a) | ((0x6400u + b) << 16);  // 1024 + field, exactly
    const __half2 h = __hsub2(*reinterpret_cast<const __half2*>(&bits), __floats2half2_rn(1152.f, 1152.f));
    return *reinterpret_cast<const uint32_t*>(&h);
}
// Images: 64 halves = 128 bytes per row of K.  Those of L21 go to tensor memory
// row by row and are plain; those of U12 are shared-memory operands, the
// 16-byte chunks of a row exchanged by the 128-byte swizzle of tcgen05: offset
// of chunk c of a row.
__device__ __forceinline__ uint32_t img_off(int row, int chunk) {
    return (uint32_t)row * 128u + (uint32_t)((chunk ^ (row & 7)) << 4);
}

// Rows launch, after a block is factored.  CTAs of 64 threads, in this order:
//   right  columns right of the block: its row exchanges, U12 = L11^-1 A12,
//          digits; a warp takes CPW columns, 32 / CPW lanes per column, rows
//          i (32 / CPW) + g in lane group g, so that every step of the
//          elimination leaves all lanes the same number of rows
//   left   columns left of the block: exchanges only
//   unit   the columns of L11^-1 and U11^-1, which the substitutions use
//   low    digits of 64 rows of L21
//   order  the exchanges followed by one vector of row numbers
// A warp's chain is 32 steps of up to CPW complex multiply-adds of 4 x 65
// clocks: two columns per warp while there are pipes to spare (12 thousand
// clocks), up to eight where the columns outnumber them (less idle lanes).
constexpr int ROWS_THREADS = 64;
struct RowsParts {
    int right, left, unit, low;  // CTAs
};

template <int CPW>
__global__ void __launch_bounds__(ROWS_THREADS) lu64_rows_kernel(
    int64_t n, double2* __restrict__ A, int64_t lda, int64_t b0, int nb, RowsParts parts,
    const RowMoves* __restrict__ moves, const int* __restrict__ cexp, const double2* __restrict__ pinv,
    unsigned char* __restrict__ Aimg, unsigned char* __restrict__ Bimg, int* __restrict__ er, int* __restrict__ ec,
    double2* __restrict__ Dinv, int* __restrict__ order) {
    constexpr int LPC = 32 / CPW, RPL = CPW;
    __shared__ double2 L[NB][NB + 1];  // L[q][r]: column q
    __shared__ double2 ys[ROWS_THREADS / 32][NB][CPW];
    __shared__ RowMoves mv;
    __shared__ int ce[NB];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int64_t t0 = b0 + nb, m = n - t0;
    int part = (int)blockIdx.x;
    if (tid < NB) {
        const int e = cexp[tid];
        ce[tid] = e <= EXP_NONE || e >= EXP_BAD ? 0 : -e;
    }
    for (int t = tid; t < (int)(sizeof(RowMoves) / sizeof(int)); t += ROWS_THREADS)
        reinterpret_cast<int*>(&mv)[t] = reinterpret_cast<const int*>(moves)[t];
    if (part < parts.right + parts.left + parts.unit) {
        const bool right = part < parts.right, left = !right && part < parts.right + parts.left;
        const bool unit = !right && !left;
        if (!left)
            for (int t = tid; t < NB * NB; t += ROWS_THREADS) {
                const int q = t / NB, r = t % NB;
                L[q][r] = q < nb && r < nb ? A[(b0 + q) * lda + b0 + r] : make_double2(0, 0);
            }
        __syncthreads();
        const int g = lane % LPC, cl = lane / LPC;
        int64_t j = (int64_t)part * (2 * CPW) + warp * CPW + cl;  // column of this part
        int64_t count = m;
        if (left) {
            j -= (int64_t)parts.right * (2 * CPW);
            count = b0;
        } else if (unit) {
            j -= (int64_t)(parts.right + parts.left) * (2 * CPW);
            count = 2 * NB;
        }
        const bool ok = j < count;
        double2 x[RPL];
        if (unit) {
            // column j of L11^-1 (j < 32) or column j - 32 of U11^-1
            const int c = (int)(j & (NB - 1));
#pragma unroll
            for (int i = 0; i < RPL; ++i) x[i] = make_double2(LPC * i + g == c ? 1.0 : 0.0, 0.0);
            if (__any_sync(0xffffffffu, j >= NB)) {
#pragma unroll
                for (int q = NB - 1; q >= 0; --q) {
                    if (q >= nb) continue;
                    if (g == q % LPC) x[q / LPC] = cmul(x[q / LPC], pinv[q]);
                    double2 xq;
                    xq.x = __shfl_sync(0xffffffffu, x[q / LPC].x, cl * LPC + q % LPC);
                    xq.y = __shfl_sync(0xffffffffu, x[q / LPC].y, cl * LPC + q % LPC);
#pragma unroll
                    for (int i = 0; i <= q / LPC; ++i)
                        if (i < q / LPC || g < q % LPC) cfms(x[i], L[q][LPC * i + g], xq);
                }
                double2* D = Dinv + (b0 / NB * 2 + 1) * (NB * NB) + c * NB;
#pragma unroll
                for (int i = 0; i < RPL; ++i) D[LPC * i + g] = x[i];
                return;
            }
        } else {
            double2* col = A + (ok ? (left ? j : t0 + j) : t0 - 1) * lda + b0;
            const int cnt = mv.count;
#pragma unroll
            for (int i = 0; i < RPL; ++i) {
                const int r = LPC * i + g;
                x[i] = ok && r < nb ? col[mv.top[r]] : make_double2(0, 0);
            }
            if (ok)
                for (int q = g; q < cnt; q += LPC) ys[warp][q][cl] = col[mv.osrc[q]];
            __syncwarp();
            if (ok) {
                for (int q = g; q < cnt; q += LPC) col[mv.opos[q]] = ys[warp][q][cl];
                if (left) {
#pragma unroll
                    for (int i = 0; i < RPL; ++i)
                        if (LPC * i + g < nb) col[LPC * i + g] = x[i];
                }
            }
            if (left) return;
        }
#pragma unroll
        for (int q = 0; q < NB - 1; ++q) {
            double2 xq;
            xq.x = __shfl_sync(0xffffffffu, x[q / LPC].x, cl * LPC + q % LPC);
            xq.y = __shfl_sync(0xffffffffu, x[q / LPC].y, cl * LPC + q % LPC);
#pragma unroll
            for (int i = q / LPC; i < RPL; ++i)
                if (i > q / LPC || g > q % LPC) cfms(x[i], L[q][LPC * i + g], xq);
        }
        if (unit) {
            double2* D = Dinv + (b0 / NB * 2) * (NB * NB) + j * NB;
#pragma unroll
            for (int i = 0; i < RPL; ++i) D[LPC * i + g] = x[i];
            return;
        }
        // (nb = 32 here: there are columns on the right)
        double2* col = A + (t0 + (ok ? j : 0)) * lda + b0;
        int e = EXP_NONE;
#pragma unroll
        for (int i = 0; i < RPL; ++i) {
            if (ok) col[LPC * i + g] = x[i];
            const int v = max(exp_above(x[i].x), exp_above(x[i].y));
            e = max(e, v == EXP_NONE || v == EXP_BAD ? v : v - ce[LPC * i + g]);
        }
#pragma unroll
        for (int o = 1; o < LPC; o *= 2) e = max(e, __shfl_xor_sync(0xffffffffu, e, o));
        if (!ok) return;
        if (g == 0) ec[j] = e;
        const int ee = e == EXP_BAD || e == EXP_NONE ? 0 : e;
        unsigned char* img = Bimg + (j / TN) * (size_t)B_IMG;
        const int row = (int)(j % TN);
#pragma unroll
        for (int i = 0; i < RPL; ++i) {
            const int p = LPC * i + g, et = ee + ce[p];
            const uint64_t re = digits_of(x[i].x, et), im = digits_of(x[i].y, et);
#pragma unroll
            for (int s = 0; s < SLICES; ++s)
                *reinterpret_cast<uint32_t*>(img + s * B_SLICE + img_off(row, p >> 2) + 4 * (p & 3)) =
                    digit_pair(re, im, s);
        }
        return;
    }
    __syncthreads();
    part -= parts.right + parts.left + parts.unit;
    if (part >= parts.low) {
        // order[i]: the row of the original matrix now at row i
        if (b0 == 0)
            for (int64_t i = tid; i < n; i += ROWS_THREADS) order[i] = (int)i;
        __syncthreads();
        int x = 0, y = 0;
        if (tid < nb) x = order[b0 + mv.top[tid]];
        if (tid < mv.count) y = order[b0 + mv.osrc[tid]];
        __syncthreads();
        if (tid < nb) order[b0 + tid] = x;
        if (tid < mv.count) order[b0 + mv.opos[tid]] = y;
        return;
    }
    const int64_t ir = (int64_t)part * 64 + tid;  // complex row of L21
    if (ir >= m) return;
    const double2* row = A + b0 * lda + t0 + ir;
    double2 x[NB];
#pragma unroll
    for (int p = 0; p < NB; ++p) x[p] = row[p * lda];
    int e = EXP_NONE;
#pragma unroll
    for (int p = 0; p < NB; ++p) {
        const int v = max(exp_above(x[p].x), exp_above(x[p].y));
        e = max(e, v == EXP_NONE || v == EXP_BAD ? v : v + ce[p]);
    }
    er[ir] = e;
    const int ee = e == EXP_BAD || e == EXP_NONE ? 0 : e;
    unsigned char* img = Aimg + part * (size_t)A_IMG;
#pragma unroll
    for (int c = 0; c < NB / 4; ++c) {
        uint64_t re[4], im[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            re[u] = digits_of(x[4 * c + u].x, ee - ce[4 * c + u]);
            im[u] = digits_of(x[4 * c + u].y, ee - ce[4 * c + u]);
        }
#pragma unroll
        for (int s = 0; s < SLICES; ++s) {
            // real rows of the embedding: [re, -im] and [im, re]
            uint32_t d[4], f[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const uint32_t h = digit_pair(re[u], im[u], s);
                d[u] = h ^ 0x80000000u;
                f[u] = __byte_perm(h, h, 0x1032);
            }
            uint4* row2 = reinterpret_cast<uint4*>(img + s * A_SLICE + 256 * tid + 16 * c);
            row2[0] = make_uint4(d[0], d[1], d[2], d[3]);
            row2[8] = make_uint4(f[0], f[1], f[2], f[3]);
        }
    }
}

// ---------------------------------------------------------------------------
// Trailing update A22 -= L21 U12 from the digit images: tiles of 128 real rows
// (64 complex) x 64 columns, K = 64.  A persistent CTA walks a contiguous run
// of tiles, row block slowest.  The seven slices of a row block live in tensor
// memory (7 x 32 columns) as the MMAs' A operand; those of the column tiles
// stream through two stages of 56 KB of shared memory.  Warp 0 copies, warp 1
// issues the MMAs weight by weight into a ring of four accumulators of 64
// tensor-memory columns, sixteen warps drain them into 32-bit partial sums and
// finish with one FP64 subtraction per entry while the next tile's MMAs run.
//
// Why: with both operands in shared memory an MMA of 128 x 64 took 91 clocks
// and one of 128 x 128 took 165 (operand reads), a tile's MMAs more than its
// epilogue; and with all of shared memory taken by operands the epilogue's
// register spills went to L2.  The epilogue's floor is the FP64 pipe: 8192
// subtractions a tile at two per clock.
constexpr int GEMM_THREADS = 576, GEMM_EPI = GEMM_THREADS - 64, EPI_COLS = 16;
constexpr int RING = 4;
constexpr uint32_t GEMM_SMEM = 2 * B_IMG + 256;
constexpr uint32_t GEMM_TMEM = 512, TMEM_A = RING * TN, TMEM_A_SLICE = 32;

// Shared-memory descriptor of a K-major operand in the 128-byte swizzle
// layout: rows of 128 bytes, 8-row atoms of 1024 bytes.
__device__ __forceinline__ uint64_t desc_sw128(uint32_t saddr) {
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | (uint64_t)1 << 16 | (uint64_t)(1024 >> 4) << 32 | (uint64_t)1 << 46 |
           (uint64_t)2 << 61;
}

// D[tmem] (+)= A[tmem] B[smem]^T: FP16 A and B (K-major), FP32 D, M = 128, N = 64, K = 16.
__device__ __forceinline__ void mma_f16(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t accumulate) {
    constexpr uint32_t idesc = (1u << 4) | ((uint32_t)(TN >> 3) << 17) | ((uint32_t)(TM >> 4) << 24);
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(tmem_d),
        "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// One row per lane of 32 consecutive 32-bit columns into tensor memory.
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
        "%14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31};" ::"r"(r[0]),
        "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
        "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]),
        "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]),
        "r"(r[29]), "r"(r[30]), "r"(r[31]), "r"(taddr)
        : "memory");
}

// 8 consecutive FP32 columns of this warp's 32 tensor-memory lanes.
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float (&v)[8]) {
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}

// An integer-valued float with |v| <= 2^22 as an integer: two full-rate
// instructions where the conversion instruction runs at an eighth of the rate.
__device__ __forceinline__ int small_int(float v) { return __float_as_int(v + 12582912.0f) - 0x4B400000; }

// c - T 2^q rounded to FP64 (T an integer, |T| < 2^62) with one FP64
// instruction; `bad` is set, and the result meaningless, where the product
// leaves the range of normal numbers.
__device__ __forceinline__ double sub_scaled(double c, int64_t T, int q, bool& bad) {
    const uint64_t u0 = T < 0 ? (uint64_t)(-T) : (uint64_t)T;
    const int lz = __clzll((long long)(u0 | 1ull));
    const uint64_t u = u0 << lz;
    const uint64_t mant = (u >> 11) + ((u >> 10) & 1ull);
    const int e = 63 - lz + q + 1022;  // exponent field - 1: the leading bit of mant adds one
    bad = (unsigned)e > 2044u;
    const uint64_t bits = ((uint64_t)T & 0x8000000000000000ull) | (((uint64_t)(unsigned)e << 52) + mant);
    return c - (T == 0 ? 0.0 : __longlong_as_double((long long)bits));
}
// A load that stays where it is written.
__device__ __forceinline__ double ld_now(const double* p) {
    double v;
    asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
    return v;
}
// The same for any exponent, and for rows and columns with an infinity or NaN.
__device__ __forceinline__ double sub_scaled_any(double c, int64_t T, int rexp, int cexp) {
    if (rexp == EXP_BAD || cexp == EXP_BAD) return __longlong_as_double(0x7ff8000000000000ll);
    if (T == 0) return c;
    // two exact steps (the first cannot leave the normal range), one rounding
    const int q = max(-2000, min(2000, rexp + cexp - 54)), q1 = q / 2;
    return c - ((double)T * __hiloint2double((q1 + 1023) << 20, 0)) * __hiloint2double((q - q1 + 1023) << 20, 0);
}

__global__ void __launch_bounds__(GEMM_THREADS, 1)
    lu64_gemm_kernel(double* __restrict__ F, int64_t lda2, int m, int cols, int row_blocks, int col_tiles,
                     const unsigned char* __restrict__ Aimg, const unsigned char* __restrict__ Bimg,
                     const int* __restrict__ er, const int* __restrict__ ec, int* __restrict__ err) {
    extern __shared__ __align__(1024) unsigned char smem[];
    uint64_t* bfull = reinterpret_cast<uint64_t*>(smem + 2 * B_IMG);
    uint64_t *bempty = bfull + 2, *tfull = bempty + 2, *tempty = tfull + RING, *aready = tempty + RING,
             *drain = aready + 1;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (warp == 0) tmem_alloc(tmem_slot, GEMM_TMEM);
    if (tid == 0) {
        for (int s = 0; s < 2; ++s) {
            mbar_init(&bfull[s], 1);
            mbar_init(&bempty[s], 1);
        }
        for (int s = 0; s < RING; ++s) {
            mbar_init(&tfull[s], 1);
            mbar_init(&tempty[s], GEMM_EPI / 32);
        }
        mbar_init(aready, GEMM_EPI / 32);
        mbar_init(drain, 1);
        *abort_flag = 0;
        fence_mbar_init();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot, base = smem_u32(smem);
    const int64_t tiles = (int64_t)row_blocks * col_tiles;
    const int first = (int)(tiles * blockIdx.x / gridDim.x), last = (int)(tiles * (blockIdx.x + 1) / gridDim.x);
    auto fail = [&]() {
        *abort_flag = 1;
        atomicOr(err, DEVERR_MBAR_TIMEOUT);
    };
    if (warp == 0) {
        if (lane == 0) {
            int it = 0;
            for (int t = first; t < last && !*abort_flag; ++t, ++it) {
                const int st = it & 1;
                if (it >= 2 && !mbar_wait_bounded(&bempty[st], (uint32_t)(((it >> 1) - 1) & 1))) {
                    fail();
                    break;
                }
                mbar_arrive_expect_tx(&bfull[st], B_IMG);
                bulk_g2s(smem + st * B_IMG, Bimg + (t % col_tiles) * (size_t)B_IMG, B_IMG, &bfull[st]);
            }
            // copies may still be landing: wait for them
            if (*abort_flag)
                for (int j = it > 2 ? it - 2 : 0; j < it; ++j) mbar_wait_bounded(&bfull[j & 1], (uint32_t)((j >> 1) & 1));
        }
        __syncwarp();
    } else if (warp == 1) {
        if (lane == 0) {
            int rb_now = -1, it = 0, idx = 0, nload = 0;
            bool ok = true;
            for (int t = first; t < last && ok && !*abort_flag; ++t, ++it) {
                const int rb = t / col_tiles, st = it & 1;
                if (rb != rb_now) {
                    ok = mbar_wait_bounded(aready, (uint32_t)(nload & 1));
                    rb_now = rb;
                    ++nload;
                }
                ok = ok && mbar_wait_bounded(&bfull[st], (uint32_t)((it >> 1) & 1));
                for (int g = GROUPS; g >= 1 && ok; --g, ++idx) {
                    const int i0 = max(0, g - SLICES), i1 = min(g, SLICES);  // digits of A in this group
                    const int blk = idx % RING, use = idx / RING;
                    ok = use == 0 || mbar_wait_bounded(&tempty[blk], (uint32_t)((use - 1) & 1));
                    if (!ok) break;
                    tc_fence_after();
                    for (int i = i0; i < i1; ++i) {
                        const uint32_t as = tmem + TMEM_A + i * TMEM_A_SLICE, bd = base + st * B_IMG + (g - 1 - i) * B_SLICE;
#pragma unroll
                        for (int kk = 0; kk < 4; ++kk)
                            mma_f16(tmem + (uint32_t)(blk * TN), as + 8 * kk, desc_sw128(bd + kk * 32),
                                    i > i0 || kk ? 1u : 0u);
                    }
                    umma_commit(&tfull[blk]);
                }
                if (ok) umma_commit(&bempty[st]);
            }
            if (!ok) fail();
        }
        __syncwarp();
    } else {
        const int quarter = warp & 3, part = (warp - 2) >> 2;
        const uint32_t mine = tmem + ((uint32_t)(32 * quarter) << 16);
        int idx = 0, rb_now = -1;
        bool ok = true;
        // waits for ring block k and returns its address
        auto arrived = [&](int k) {
            if (ok && !mbar_wait_bounded(&tfull[k % RING], (uint32_t)((k / RING) & 1))) ok = false;
            tc_fence_after();
            return mine + (uint32_t)(EPI_COLS * part + (k % RING) * TN);
        };
        auto release = [&](int k) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&tempty[k % RING]);
        };
        for (int t = first; t < last && !*abort_flag; ++t, idx += GROUPS) {
            const int rb = t / col_tiles, ct = t - rb * col_tiles;
            if (rb != rb_now) {
                // this row block's slices into tensor memory (its MMAs have all
                // finished: the last tile's accumulators have been drained)
                rb_now = rb;
                for (int s = part; s < SLICES; s += 4) {
                    const uint4* src = reinterpret_cast<const uint4*>(Aimg + rb * (size_t)A_IMG + s * A_SLICE +
                                                                      (32 * quarter + lane) * 128);
                    uint32_t w[32];
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const uint4 x = src[i];
                        w[4 * i] = x.x;
                        w[4 * i + 1] = x.y;
                        w[4 * i + 2] = x.z;
                        w[4 * i + 3] = x.w;
                    }
                    tmem_st32(mine + TMEM_A + s * TMEM_A_SLICE, w);
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(aready);
            }
            const int r = rb * TM + 32 * quarter + lane, j0 = ct * TN + EPI_COLS * part;
            const bool rok = r < 2 * m;
            const int nq = max(0, min(EPI_COLS, cols - j0));
            const int rexp = rok ? er[r >> 1] : 0;  // (outside the matrix: any exponent in range)
            const int cexps = lane < nq ? ec[j0 + lane] : 0;
            double* p = F + (int64_t)j0 * lda2 + r;
            // (the entries are loaded four at a time when the sums are complete:
            // more of them do not fit the registers, and spills go to L2 here)
            if ((lane & 15) == 0 && rok)
                for (int q = 0; q < nq; ++q) asm volatile("prefetch.global.L2 [%0];" ::"l"(p + q * lda2));
            // T = lo + 2^16 mid + 2^32 top
            int lo[EPI_COLS], mid[EPI_COLS];
            float v[8];
#pragma unroll
            for (int g = 0; g < 6; ++g) {
                const uint32_t a = arrived(idx + g);
#pragma unroll
                for (int h = 0; h < EPI_COLS / 8; ++h) {
                    tmem_ld8(a + 8 * h, v);
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        const int k = 8 * h + q;
                        if (g == 0) lo[k] = __float2int_rn(v[q]) + 32768;
                        else if (g == 1) lo[k] = (lo[k] + __float2int_rn(v[q]) * 256) >> 16;
                        else if (g == 2) lo[k] += __float2int_rn(v[q]);
                        else if (g == 3) lo[k] += __float2int_rn(v[q]) * 256;
                        else if (g == 4) mid[k] = small_int(v[q]);
                        else mid[k] += small_int(v[q]) * 256;
                    }
                }
                release(idx + g);
            }
            const uint32_t a2 = arrived(idx + 6), a1 = arrived(idx + 7);
            if (!ok) {
                fail();
                break;
            }
#pragma unroll
            for (int h = 0; h < EPI_COLS / 8; ++h) {
                int top[8];
                tmem_ld8(a2 + 8 * h, v);
#pragma unroll
                for (int q = 0; q < 8; ++q) top[q] = small_int(v[q]);
                tmem_ld8(a1 + 8 * h, v);
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const int k = 8 * h + q;
                    const int64_t T = (int64_t)lo[k] + (int64_t)mid[k] * 65536 +
                                      ((int64_t)(top[q] + small_int(v[q]) * 256) << 32);
                    lo[k] = (int)T;  // the two halves of T from here on
                    mid[k] = (int)(T >> 32);
                }
            }
            release(idx + 6);
            release(idx + 7);
#pragma unroll
            for (int h = 0; h < EPI_COLS / 4; ++h) {
                double c[4], d[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) c[q] = rok && 4 * h + q < nq ? ld_now(p + (4 * h + q) * lda2) : 0.0;
                bool any = false;
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int k = 4 * h + q;
                    bool bad;
                    d[q] = sub_scaled(c[q], ((int64_t)mid[k] << 32) | (unsigned)lo[k],
                                      rexp + __shfl_sync(0xffffffffu, cexps, k) - 54, bad);
                    any = any || bad;
                }
                if (__any_sync(0xffffffffu, any)) {
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int k = 4 * h + q;
                        d[q] = sub_scaled_any(c[q], ((int64_t)mid[k] << 32) | (unsigned)lo[k], rexp,
                                              __shfl_sync(0xffffffffu, cexps, k));
                    }
                }
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (rok && 4 * h + q < nq) p[(4 * h + q) * lda2] = d[q];
            }
        }
    }
    __syncthreads();
    if (*abort_flag) {
        // every MMA this CTA issued is tracked by one more commit
        if (tid == 32) umma_commit(drain);
        if (tid == 32) mbar_wait_bounded(drain, 0);
        __syncthreads();
    }
    tc_fence_after();
    if (warp == 0) tmem_dealloc(tmem, GEMM_TMEM);
}

// ---------------------------------------------------------------------------
// Both substitutions in one launch.  A ticket is one block of 32 rows in one
// direction:
//   forward  row block b:  z_b = L_bb^-1 (b_b - sum_{k<b} L_bk z_k)
//   backward row block b:  x_b = U_bb^-1 (z_b - sum_{k>b} U_bk x_k)
// CTAs take tickets from a counter in an order where every block a ticket
// needs has a smaller ticket, so a CTA waits only on blocks that running CTAs
// hold.  The solution blocks are their own flags: the buffers start as all
// ones bits and a reader polls the values it needs (one trip through L2 per
// block instead of two).  Waits are bounded (error word, then the ticket
// carries on).  Four warps take 8 columns of a 32 x 32 block each; a block's
// product is 8 complex multiply-adds of 4 x 65 clocks per warp, which with the
// trip through L2 and the diagonal's three products is the chain per block
// (one cluster of 16 SMs walking the blocks took 14 to 24 us per block).
//
// The inverse of a triangular block loses digits where the block is
// ill-conditioned (twice the error of a substitution for random matrices), so its
// product is corrected once by the residual against the block itself.  And the
// sums over the blocks cancel against the right-hand side, so the blocks' products
// are added without rounding error: as one running sum they made up most of the
// error of x (n = 320: 1.7e-13 against 0.4e-13).
constexpr int SOLVE_THREADS = 128;
constexpr unsigned long long UNSET = ~0ull;

__device__ __forceinline__ bool is_unset(double2 v) {
    return (unsigned long long)__double_as_longlong(v.x) == UNSET ||
           (unsigned long long)__double_as_longlong(v.y) == UNSET;
}
// acc + low += v, the rounding error of acc + v kept in low (Knuth's two-sum).
__device__ __forceinline__ void add_exactly(double& acc, double& low, double v) {
    const double s = acc + v, t = s - acc;
    low += (acc - (s - t)) + (v - t);
    acc = s;
}
__device__ __forceinline__ bool finite_bits(double v) { return (__double2hiint(v) & 0x7ff00000) != 0x7ff00000; }
__device__ __forceinline__ double settled(double v) {
    return (unsigned long long)__double_as_longlong(v) == UNSET ? __longlong_as_double(0x7ff8000000000000ll) : v;
}
__device__ __forceinline__ double2 ld_relaxed(const double2* p) {
    double2 v;
    asm volatile("ld.relaxed.gpu.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed(double2* p, double2 v) {
    asm volatile("st.relaxed.gpu.global.v2.f64 [%0], {%1, %2};" ::"l"(p), "d"(v.x), "d"(v.y) : "memory");
}

// acc += (this warp's 8 columns of a block, a[i] = column 8 warp + i of the
// lane's row) times the values xv of lanes 0 .. 7.
__device__ __forceinline__ void block_product(double2& acc, const double2 (&a)[8], double2 xv) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        double2 x;
        x.x = __shfl_sync(0xffffffffu, xv.x, i);
        x.y = __shfl_sync(0xffffffffu, xv.y, i);
        cfma(acc, a[i], x);
    }
}

__global__ void __launch_bounds__(SOLVE_THREADS) lu64_solve_kernel(int64_t n, const double2* __restrict__ A,
                                                                   int64_t lda, const double2* __restrict__ Dinv,
                                                                   const int* __restrict__ order, double2* b, double2* z,
                                                                   double2* xr, int* __restrict__ counter,
                                                                   int* __restrict__ info, int* __restrict__ err) {
    __shared__ double2 red[3][4][NB], ysum[NB];
    __shared__ int tk;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    auto sum = [&](int set, int row) {
        return cadd(cadd(red[set][0][row], red[set][1][row]), cadd(red[set][2][row], red[set][3][row]));
    };
    const int nblk = (int)((n + NB - 1) / NB);
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) tk = atomicAdd(counter, 1);
        __syncthreads();
        const int t = tk;
        if (t >= 2 * nblk) return;
        const bool fwd = t < nblk;
        const int rb = fwd ? t : 2 * nblk - 1 - t;
        const int64_t r = (int64_t)rb * NB + lane;
        const bool rok = r < n;
        const double2* y = fwd ? z : xr;
        const int steps = fwd ? rb : nblk - 1 - rb;
        double2 acc = make_double2(0, 0), low = acc;
        // the diagonal block, its inverse and the right-hand side, ahead of the waits
        double2 d[8], e[8], rhs = make_double2(0, 0);
        const double2* D = Dinv + ((int64_t)rb * 2 + (fwd ? 0 : 1)) * (NB * NB) + (8 * warp) * NB + lane;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int col = 8 * warp + i;
            const int64_t c = (int64_t)rb * NB + col;
            d[i] = D[i * NB];
            e[i] = rok && c < n && (fwd ? col < lane : col >= lane) ? A[c * lda + r]
                                                                    : make_double2(fwd && col == lane ? 1.0 : 0.0, 0);
        }
        if (warp == 0 && fwd && rok) rhs = b[order[r]];
        for (int i = 0; i < steps; ++i) {
            const int k = fwd ? i : nblk - 1 - i;
            const int64_t c0 = (int64_t)k * NB + 8 * warp;
            double2 a[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) a[q] = rok && c0 + q < n ? A[(c0 + q) * lda + r] : make_double2(0, 0);
            double2 xv = make_double2(0, 0);
            if (lane < 8 && c0 + lane < n) {
                xv = ld_relaxed(y + c0 + lane);
                for (unsigned it = 0; is_unset(xv); ++it) {
                    if (it > (1u << 22)) {
                        atomicOr(err, DEVERR_BARRIER_TIMEOUT);
                        break;
                    }
                    xv = ld_relaxed(y + c0 + lane);
                }
            }
            __syncwarp();
            double2 part = make_double2(0, 0);
            block_product(part, a, xv);
            add_exactly(acc.x, low.x, part.x);
            add_exactly(acc.y, low.y, part.y);
        }
        if (finite_bits(low.x)) acc.x += low.x;
        if (finite_bits(low.y)) acc.y += low.y;
        red[0][warp][lane] = acc;
        if (!fwd && warp == 0 && rok) {
            rhs = ld_relaxed(z + r);
            for (unsigned it = 0; is_unset(rhs); ++it) {
                if (it > (1u << 22)) {
                    atomicOr(err, DEVERR_BARRIER_TIMEOUT);
                    break;
                }
                rhs = ld_relaxed(z + r);
            }
            const double2 u = A[r * lda + r];
            if (u.x == 0.0 && u.y == 0.0) atomicCAS(info, 0, (int)(r + 1));
        }
        __syncthreads();
        if (warp == 0) ysum[lane] = csub(rhs, sum(0, lane));
        __syncthreads();
        // y = D^-1 (right-hand side), then once more with what D y leaves of it
        const int c8 = 8 * warp + (lane & 7);
        acc = make_double2(0, 0);
        block_product(acc, d, ysum[c8]);
        red[1][warp][lane] = acc;
        __syncthreads();
        acc = make_double2(0, 0);
        block_product(acc, e, sum(1, c8));
        red[2][warp][lane] = acc;
        __syncthreads();
        acc = make_double2(0, 0);
        block_product(acc, d, csub(ysum[c8], sum(2, c8)));
        red[0][warp][lane] = acc;
        __syncthreads();
        if (warp == 0 && rok) {
            double2 v = sum(1, lane);
            const double2 f = sum(0, lane);
            if (finite_bits(f.x) && finite_bits(f.y)) v = cadd(v, f);
            v = make_double2(settled(v.x), settled(v.y));
            st_relaxed((fwd ? z : xr) + r, v);
            if (!fwd) b[r] = v;  // every forward block has been read by now
        }
    }
}

// ---------------------------------------------------------------------------
}  // namespace

// What a factorization leaves beside the factors: the row order and the
// inverses of the diagonal blocks.
static size_t aux_order_bytes(int64_t n) { return (sizeof(int) * (size_t)n + 255) / 256 * 256; }
size_t lu_aux_bytes(int64_t n) {
    return aux_order_bytes(n) + sizeof(double2) * 2 * NB * NB * (size_t)((n + NB - 1) / NB);
}

void lu_factor_fp64(Context& ctx, int64_t n, double2* A, int64_t lda, void* aux, int* d_info) {
    BEM_CUDA(cudaMemsetAsync(d_info, 0, sizeof(int), ctx.stream));
    int* err = device_err(ctx);
    BEM_CUDA(cudaMemsetAsync(err, 0, sizeof(int), ctx.stream));
    int* order = static_cast<int*>(aux);
    double2* Dinv = reinterpret_cast<double2*>(static_cast<char*>(aux) + aux_order_bytes(n));
    const void* panel = (const void*)lu64_panel_kernel;
    BEM_CUDA(cudaFuncSetAttribute(panel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PANEL_SMEM));
    BEM_CUDA(cudaFuncSetAttribute(panel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    BEM_CUDA(cudaFuncSetAttribute(lu64_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GEMM_SMEM));
    if (!ctx.lu64_cluster) ctx.lu64_cluster = max_cluster(panel, PANEL_THREADS, PANEL_SMEM);
    int nsm = 0;
    BEM_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, ctx.device));
    // digit images of the first (largest) trailing update, the exponents of its
    // rows and columns and those of every column of L21, the current block's
    // exchanges and pivot reciprocals
    const int64_t m0 = std::max<int64_t>(n - NB, 1), tiles0 = (m0 + 63) / 64, nblk = (n + NB - 1) / NB;
    auto up = [](size_t b) { return (b + 255) / 256 * 256; };
    const size_t a_bytes = (size_t)tiles0 * A_IMG, b_bytes = (size_t)tiles0 * B_IMG, e_bytes = up(sizeof(int) * (size_t)m0);
    const size_t c_bytes = up(sizeof(int) * NB * (size_t)nblk), v_bytes = up(sizeof(RowMoves));
    ctx.w_lu64.ensure(a_bytes + b_bytes + 2 * e_bytes + c_bytes + v_bytes + sizeof(double2) * NB);
    unsigned char* Aimg = ctx.w_lu64.as<unsigned char>();
    unsigned char* Bimg = Aimg + a_bytes;
    int* er = reinterpret_cast<int*>(Bimg + b_bytes);
    int* ec = er + e_bytes / sizeof(int);
    int* cexp = ec + e_bytes / sizeof(int);
    RowMoves* mv = reinterpret_cast<RowMoves*>(reinterpret_cast<char*>(cexp) + c_bytes);
    double2* pinv = reinterpret_cast<double2*>(reinterpret_cast<char*>(mv) + v_bytes);
    BEM_CUDA(cudaMemsetAsync(cexp, 0x80, c_bytes, ctx.stream));  // below every exponent
    ctx.need_side();
    std::function<void()> beside;  // the part of the last update that runs beside this block's panels
    for (int64_t b0 = 0; b0 < n; b0 += NB) {
        const int nb = (int)std::min<int64_t>(NB, n - b0);
        const int64_t R = n - b0;
        bool ahead = false;
        int cs = 1;  // CTAs of the panels' cluster: 32 rows each where the cluster reaches
        while (cs < ctx.lu64_cluster && (int64_t)cs * 32 < R) cs *= 2;
        auto rows_of = [&](int64_t rows) { return ((rows + cs - 1) / cs + 31) / 32 * 32; };
        // panel width: the whole block up to 1024 rows, then narrower ones:
        // the FP64 work of a panel runs on the cluster's SMs alone
        int w = R > 1024 ? 16 : NB;
        while (w > 1 && (size_t)rows_of(R) * w * sizeof(double2) > PANEL_SMEM) w /= 2;
        require((size_t)rows_of(R) * w * sizeof(double2) <= PANEL_SMEM, "LU: matrix too large", BEM_ERR_OOM);
        for (int64_t c0 = b0; c0 < b0 + nb; c0 += w) {
            const int pw = (int)std::min<int64_t>(w, b0 + nb - c0), rpc = (int)rows_of(n - c0);
            launch_cluster(ctx, lu64_panel_kernel, cs, cs, PANEL_THREADS, sizeof(double2) * (size_t)rpc * pw, n, A, lda, c0,
                           pw, b0, nb, rpc, mv, cexp + b0, pinv, d_info, err);
            if (beside) {  // (behind the panel in the order of submission)
                beside();
                beside = nullptr;
                ahead = true;
            }
            const int nc = (int)(b0 + nb - c0 - pw);
            if (nc > 0) {
                lu64_mid_kernel<<<dim3((unsigned)((n - c0 - pw + 31) / 32), (unsigned)((nc + MID_COLS - 1) / MID_COLS)),
                                  32, 0, ctx.stream>>>(n, A, lda, c0, pw, nc);
                BEM_CHECK_LAUNCH(&ctx);
            }
        }
        if (ahead) ctx.join();
        const int64_t m = n - b0 - nb, rb = (m + 63) / 64, ct = (m + TN - 1) / TN;
        // columns per warp: a warp for every two columns while the SM quarters
        // (four per SM) outnumber the warps
        const int cpw = m <= 8 * nsm ? 2 : m <= 16 * nsm ? 4 : 8;
        auto groups = [&](int64_t cols) { return (int)((cols + 2 * cpw - 1) / (2 * cpw)); };
        RowsParts parts{groups(m), groups(b0), 2 * NB / (2 * cpw), (int)rb};
        const unsigned ctas = (unsigned)(parts.right + parts.left + parts.unit + parts.low + 1);
        auto rows = cpw == 2 ? lu64_rows_kernel<2> : cpw == 4 ? lu64_rows_kernel<4> : lu64_rows_kernel<8>;
        rows<<<ctas, ROWS_THREADS, 0, ctx.stream>>>(n, A, lda, b0, nb, parts, mv, cexp + b0, pinv, Aimg, Bimg, er, ec,
                                                    Dinv, order);
        BEM_CHECK_LAUNCH(&ctx);
        if (m <= 0) continue;
        const int64_t t0 = b0 + nb;
        // column tiles first .. last of the update
        auto update = [=, &ctx](int64_t first, int64_t last, int64_t sms, cudaStream_t stream) {
            const int64_t cols = m - first * TN;
            lu64_gemm_kernel<<<(unsigned)std::min<int64_t>(rb * (last - first), sms), GEMM_THREADS, GEMM_SMEM, stream>>>(
                reinterpret_cast<double*>(A + (t0 + first * TN) * lda + t0), 2 * lda, (int)m, (int)cols, (int)rb,
                (int)(last - first), Aimg, Bimg + first * (size_t)B_IMG, er, ec + first * TN, err);
            BEM_CHECK_LAUNCH(&ctx);
        };
        if (ct < 2) {
            update(0, ct, nsm, ctx.stream);
            continue;
        }
        // The next panel needs the first tile of columns only: the others are
        // updated beside it, on the SMs that its cluster leaves.  The panel comes
        // first on the SMs because its stream goes straight on.  (One after the
        // other, update and solve included: n = 1000 5.05 ms, 2001 11.9, 4000 35.2,
        // 6144 79.9; this way 4.98, 10.9, 28.7, 63.7.)
        update(0, 1, nsm, ctx.stream);
        ctx.fork();
        beside = [=, &ctx] {
            update(1, ct, nsm - cs, ctx.side);
        };
    }
}

int lu_status(Context& ctx) {
    int h[2] = {0, 0};
    BEM_CUDA(cudaMemcpyAsync(h, ctx.w_flags.p, sizeof(h), cudaMemcpyDeviceToHost, ctx.stream));
    ctx.sync();
    if (h[0]) check_device_err(ctx);
    return h[1];
}

void lu_solve_fp64(Context& ctx, int64_t n, const double2* A, int64_t lda, const void* aux, double2* b) {
    int* flags = ctx.w_flags.as<int>();
    const int* order = static_cast<const int*>(aux);
    const double2* Dinv = reinterpret_cast<const double2*>(static_cast<const char*>(aux) + aux_order_bytes(n));
    const size_t v_bytes = sizeof(double2) * (size_t)n;
    ctx.w_lu64.ensure(2 * v_bytes + sizeof(int));
    double2* z = ctx.w_lu64.as<double2>();
    int* counter = reinterpret_cast<int*>(z + 2 * n);
    BEM_CUDA(cudaMemsetAsync(z, 0xff, 2 * v_bytes, ctx.stream));
    BEM_CUDA(cudaMemsetAsync(counter, 0, sizeof(int), ctx.stream));
    int nsm = 0;
    BEM_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, ctx.device));
    const int64_t tickets = 2 * ((n + NB - 1) / NB);
    lu64_solve_kernel<<<(unsigned)std::min<int64_t>(tickets, nsm), SOLVE_THREADS, 0, ctx.stream>>>(
        n, A, lda, Dinv, order, b, z, z + n, counter, flags + 1, flags);
    BEM_CHECK_LAUNCH(&ctx);
}

}  // namespace bem
