// Restarted GMRES (gmres.rs:35-202) as a device-side state machine over a
// batch of independent systems: of equal size n (uniform layout), or of
// different sizes (ragged layout, per-system offsets in GmSys).
//
// One iteration is the fixed launch sequence
//   [precondition] -> apply(Q) -> Gram-Schmidt and rotations -> apply(CHECK) -> check
// after one start (with an apply(START) before it in the reference form), where
// every kernel reads the per-system state and returns immediately when it has
// nothing to do.  The host therefore launches ahead of the device, which tells it
// when every system is done.
//
// Operator: FP64 matrix (plain form, bit-for-bit the reference arithmetic up
// to summation order) or FP32 matrix with FP64 vectors and compensated
// products/sums (mixed form).  Arnoldi, Givens rotations, the small
// triangular solve and the stopping test are FP64: the reference form keeps
// modified Gram-Schmidt, on one thread-block cluster per system, the mixed and
// refined forms orthogonalise across the whole GPU (classical Gram-Schmidt twice).
#include <mutex>

#include "cluster.cuh"
#include "common.cuh"
#include "complex.cuh"
#include "gmres.cuh"

namespace bem {

constexpr int MV_ROWS_PER_THREAD = 2;
constexpr int MV_THREADS = 256;
constexpr int MV_ROWS = MV_ROWS_PER_THREAD * MV_THREADS;  // 512
constexpr int MV_COLS = 512;
// row block of the small-batch product, and the tickets that a row block of
// MV_ROWS holds for it
constexpr int SMALL_ROWS = 64;
constexpr int TICKETS = MV_ROWS / SMALL_ROWS;
constexpr int AR_THREADS = 1024;
// dynamic shared memory of the Arnoldi kernels
constexpr size_t AR_SMEM_CAP = 200 * 1024;

__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
    s = a + b;
    float bb = s - a;
    e = (a - (s - bb)) + (b - bb);
}

// acc (hi, lo) += a * b with a*b = p + e exactly (FMA) and a small extra term.
__device__ __forceinline__ void ff_acc(float& hi, float& lo, float a, float b) {
    float p = a * b;
    float e = fmaf(a, b, -p);
    float s, err;
    two_sum(hi, p, s, err);
    hi = s;
    lo += err + e;
}

// Batched operator application W_s = A_s v_s, v_s = x_s (START/CHECK) or
// Q_s[:, k] (Q).  Grid (row blocks, column chunks, systems); partial sums of
// the column chunks are reduced in a fixed order by the last CTA of each row
// block (ticket counter, no waiting).  Each thread owns two consecutive rows
// and streams its columns with 16-byte loads, eight columns in flight.
//
// FP32 operators, two accumulation schemes:
//  EXACT (true residuals, START/CHECK): x split into hi + lo floats, every
//        product split exactly with an FMA and summed in float-float;
//  FAST  (Krylov vectors, Q): FP32 sums of 8 columns folded into a float-float
//        accumulator; ~1e-7 relative, which only perturbs the Krylov basis:
//        the exact residual at each check and restart keeps the answer exact.
// Split FP64 operators (EXACT == 2, every mode): the EXACT scheme over the
// FP32 matrix plus the products of its remainder plane with x's hi part, so
// the mat-vec carries the FP64 operator to ~2^-44 on the FP32 pipe (GB300's
// FP64 rate is 1/64 of it) while streaming the same 16 B per entry.
constexpr int MV_UNROLL = 8;

// NV == 2 (FAST only): two systems with the same operator (several right-hand
// sides) in one pass over it, where both are active; memory bounds the product,
// so the second one is nearly free (two operators of n = 40960 with two waves: the
// whole solve 522 -> 499 ms).  Each system's sums are the same bits.
template <typename T, int EXACT, int U = MV_UNROLL, int NV = 1>
__global__ void __launch_bounds__(MV_THREADS) gm_apply_kernel(GmBatch bt, int mode) {
    static_assert(MV_COLS % U == 0, "the column chunk is a whole number of unrolled groups");
    static_assert(NV == 1 || (sizeof(T) == sizeof(float2) && EXACT == 0), "two vectors: the FAST scheme only");
    int s, bx, by;
    if (bt.sys) {
        // ragged batch: one flattened grid over every system's (row block,
        // column chunk) tiles; the system is found by bisection on tile0
        const int64_t t = blockIdx.x;
        int lo = 0, hi = bt.nsys - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (bt.sys[mid].tile0 <= t) lo = mid;
            else hi = mid - 1;
        }
        s = lo;
        const int64_t local = t - bt.sys[s].tile0;
        const int rbs = bt.sys[s].rb;
        bx = (int)(local % rbs);
        by = (int)(local / rbs);
    } else {
        s = blockIdx.z;
        bx = blockIdx.x;
        by = blockIdx.y;
    }
    GmState& st = bt.st[s];
    if (!gm_apply_active(st, mode)) return;
    int s2 = -1;
    if (NV == 2) {
        const int mate = bt.sys[s].mate;
        if (mate >= 0 && gm_apply_active(bt.st[mate], mode)) {
            if (mate < s) return;  // the mate's CTA does both
            s2 = mate;
        }
    }
    const GmView g = gm_view(bt, s);
    const int64_t n = g.n;
    const double2* kv = bt.Z ? bt.Z : bt.Q;  // right preconditioning applies A to M q_k
    const double2* v = (mode == MV_Q) ? kv + g.q + (size_t)st.k * n : bt.X + g.v;
    const GmView g2 = NV == 2 && s2 >= 0 ? gm_view(bt, s2) : g;
    const double2* v2 = NV == 2 && s2 >= 0 ? kv + g2.q + (size_t)bt.st[s2].k * n : v;
    __shared__ float2 xh[MV_COLS], xl[NV == 2 ? 1 : MV_COLS], yh[NV == 2 ? MV_COLS : 1];
    __shared__ double2 xd[MV_COLS];
    __shared__ int last;
    const int64_t j0 = (int64_t)by * MV_COLS;
    const int jn = (int)min((int64_t)MV_COLS, n - j0);
    for (int t = threadIdx.x; t < MV_COLS; t += MV_THREADS) {
        double2 x = t < jn ? v[j0 + t] : make_double2(0, 0);
        if (sizeof(T) == sizeof(float2)) {
            float hx = (float)x.x, hy = (float)x.y;
            xh[t] = make_float2(hx, hy);
            if (NV == 2) {
                const double2 y = t < jn ? v2[j0 + t] : make_double2(0, 0);
                yh[t] = make_float2((float)y.x, (float)y.y);
            } else {
                xl[t] = make_float2((float)(x.x - (double)hx), (float)(x.y - (double)hy));
            }
        } else {
            xd[t] = x;
        }
    }
    __syncthreads();
    const int64_t i0 = (int64_t)bx * MV_ROWS + MV_ROWS_PER_THREAD * threadIdx.x;
    const int64_t lda = g.lda;
    double2 r0 = make_double2(0, 0), r1 = make_double2(0, 0);
    if (i0 < n) {
        const bool pair = (i0 + 1 < n);
        if (sizeof(T) == sizeof(float2)) {
            const float2* A = reinterpret_cast<const float2*>(bt.A) + g.a + i0;
            // float-float accumulators for (re0, im0, re1, im1)
            float h0 = 0, l0 = 0, h1 = 0, l1 = 0, h2 = 0, l2 = 0, h3 = 0, l3 = 0;
            float yhi[4] = {0, 0, 0, 0}, ylo[4] = {0, 0, 0, 0};
            for (int q0 = 0; q0 < jn; q0 += U) {
                float4 a[U], z[EXACT == 2 ? U : 1];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int q = q0 + u;
                    if (q < jn) {
                        const float2* col = A + (j0 + q) * lda;
                        if (pair) a[u] = __ldcs(reinterpret_cast<const float4*>(col));
                        else { float2 t = col[0]; a[u] = make_float4(t.x, t.y, 0.f, 0.f); }
                        if (EXACT == 2) {
                            const float2* cl = col + bt.split_lo;
                            if (pair) z[u] = __ldcs(reinterpret_cast<const float4*>(cl));
                            else { float2 t = cl[0]; z[u] = make_float4(t.x, t.y, 0.f, 0.f); }
                        }
                    } else {
                        a[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (EXACT == 2) z[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                    }
                }
                if (EXACT) {
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const float2 H = xh[q0 + u], L = xl[q0 + u];
                        const float4 w = a[u];
                        ff_acc(h0, l0, w.x, H.x); ff_acc(h0, l0, -w.y, H.y);
                        ff_acc(h1, l1, w.x, H.y); ff_acc(h1, l1, w.y, H.x);
                        ff_acc(h2, l2, w.z, H.x); ff_acc(h2, l2, -w.w, H.y);
                        ff_acc(h3, l3, w.z, H.y); ff_acc(h3, l3, w.w, H.x);
                        l0 = fmaf(w.x, L.x, fmaf(-w.y, L.y, l0));
                        l1 = fmaf(w.x, L.y, fmaf(w.y, L.x, l1));
                        l2 = fmaf(w.z, L.x, fmaf(-w.w, L.y, l2));
                        l3 = fmaf(w.z, L.y, fmaf(w.w, L.x, l3));
                        if (EXACT == 2) {
                            const float4 y = z[EXACT == 2 ? u : 0];
                            l0 = fmaf(y.x, H.x, fmaf(-y.y, H.y, l0));
                            l1 = fmaf(y.x, H.y, fmaf(y.y, H.x, l1));
                            l2 = fmaf(y.z, H.x, fmaf(-y.w, H.y, l2));
                            l3 = fmaf(y.z, H.y, fmaf(y.w, H.x, l3));
                        }
                    }
                } else {
                    float b0 = 0, b1 = 0, b2 = 0, b3 = 0;
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const float2 H = xh[q0 + u];
                        const float4 w = a[u];
                        b0 = fmaf(w.x, H.x, fmaf(-w.y, H.y, b0));
                        b1 = fmaf(w.x, H.y, fmaf(w.y, H.x, b1));
                        b2 = fmaf(w.z, H.x, fmaf(-w.w, H.y, b2));
                        b3 = fmaf(w.z, H.y, fmaf(w.w, H.x, b3));
                    }
                    float e, t;
                    two_sum(h0, b0, t, e); h0 = t; l0 += e;
                    two_sum(h1, b1, t, e); h1 = t; l1 += e;
                    two_sum(h2, b2, t, e); h2 = t; l2 += e;
                    two_sum(h3, b3, t, e); h3 = t; l3 += e;
                    if (NV == 2) {
                        float c[4] = {0, 0, 0, 0};
#pragma unroll
                        for (int u = 0; u < U; ++u) {
                            const float2 H = yh[q0 + u];
                            const float4 w = a[u];
                            c[0] = fmaf(w.x, H.x, fmaf(-w.y, H.y, c[0]));
                            c[1] = fmaf(w.x, H.y, fmaf(w.y, H.x, c[1]));
                            c[2] = fmaf(w.z, H.x, fmaf(-w.w, H.y, c[2]));
                            c[3] = fmaf(w.z, H.y, fmaf(w.w, H.x, c[3]));
                        }
#pragma unroll
                        for (int p = 0; p < 4; ++p) {
                            two_sum(yhi[p], c[p], t, e);
                            yhi[p] = t;
                            ylo[p] += e;
                        }
                    }
                }
            }
            if (NV == 2 && s2 >= 0) {
                double2* part2 = bt.part + g2.p + (size_t)by * g2.n_pad;
                part2[i0] = make_double2((double)yhi[0] + (double)ylo[0], (double)yhi[1] + (double)ylo[1]);
                if (pair) part2[i0 + 1] = make_double2((double)yhi[2] + (double)ylo[2], (double)yhi[3] + (double)ylo[3]);
            }
            r0 = make_double2((double)h0 + (double)l0, (double)h1 + (double)l1);
            r1 = make_double2((double)h2 + (double)l2, (double)h3 + (double)l3);
        } else {
            const double2* A = reinterpret_cast<const double2*>(bt.A) + g.a + i0;
            for (int q0 = 0; q0 < jn; q0 += U) {
                double2 a0[U], a1[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int q = q0 + u;
                    const double2* col = A + (j0 + (q < jn ? q : 0)) * lda;
                    a0[u] = q < jn ? col[0] : make_double2(0, 0);
                    a1[u] = (q < jn && pair) ? col[1] : make_double2(0, 0);
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const double2 xv = xd[q0 + u];
                    cfma(r0, a0[u], xv);
                    cfma(r1, a1[u], xv);
                }
            }
        }
        double2* part = bt.part + g.p + (size_t)by * g.n_pad;
        part[i0] = r0;
        if (pair) part[i0 + 1] = r1;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        int* tk = bt.tickets + g.t + bx;
        last = (atomicAdd(tk, 1) == g.cb - 1);
        if (last) *tk = 0;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double2* W = bt.W + g.v;
    for (int rr = 0; rr < MV_ROWS_PER_THREAD; ++rr) {
        int64_t i = i0 + rr;
        if (i >= n) break;
        double2 acc = make_double2(0, 0);
        const double2* part = bt.part + g.p;
        for (int c = 0; c < g.cb; ++c) acc = cadd(acc, part[(size_t)c * g.n_pad + i]);
        W[i] = acc;
        if (NV == 2 && s2 >= 0) {
            acc = make_double2(0, 0);
            for (int c = 0; c < g2.cb; ++c) acc = cadd(acc, bt.part[g2.p + (size_t)c * g2.n_pad + i]);
            bt.W[g2.v + i] = acc;
        }
    }
}

// The same product cut finer, for batches whose MV_ROWS x MV_COLS tiles are too
// few to fill the SMs: a CTA of eight warps takes SMALL_ROWS rows of a column
// chunk, the warps share its columns.  Latency bounds such a batch, so what
// counts is loads in flight on every SM (four systems of n = 1280: 36 wide tiles
// 37 us, 240 of these 11 us).
//
// The sums keep their order.  In the FAST scheme the warps take the groups of U
// columns in turn and leave each group's FP32 sum in shared memory; a thread
// per row and component folds them in column order, so that the result is the
// same bits as the wide tile's.  In the others a warp accumulates its own
// columns and the eight sums are added in FP64.
constexpr int SMALL_WARPS = 8;
template <typename T, int EXACT, int U>
constexpr size_t small_smem() {
    return sizeof(T) == sizeof(float2) && !EXACT ? sizeof(float2) * (MV_COLS / U) * SMALL_ROWS
                                                 : sizeof(double2) * SMALL_WARPS * SMALL_ROWS;
}

template <typename T, int EXACT, int U>
__global__ void __launch_bounds__(32 * SMALL_WARPS) gm_apply_small_kernel(GmBatch bt, int mode) {
    static_assert(MV_COLS % (U * SMALL_WARPS) == 0, "every warp takes the same number of column groups");
    constexpr bool F32 = sizeof(T) == sizeof(float2);
    int s, bx, by;
    if (bt.sys) {
        const int64_t t = blockIdx.x;
        int lo = 0, hi = bt.nsys - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (bt.sys[mid].tile64 <= t) lo = mid;
            else hi = mid - 1;
        }
        s = lo;
        const int64_t local = t - bt.sys[s].tile64;
        const int64_t rbs = (bt.sys[s].n + SMALL_ROWS - 1) / SMALL_ROWS;
        bx = (int)(local % rbs);
        by = (int)(local / rbs);
    } else {
        s = blockIdx.z;
        bx = blockIdx.x;
        by = blockIdx.y;
    }
    if (!gm_apply_active(bt.st[s], mode)) return;
    const GmView g = gm_view(bt, s);
    const int64_t n = g.n, lda = g.lda;
    const double2* kv = bt.Z ? bt.Z : bt.Q;
    const double2* v = (mode == MV_Q) ? kv + g.q + (size_t)bt.st[s].k * n : bt.X + g.v;
    __shared__ float2 xh[F32 ? MV_COLS : 1], xl[F32 && EXACT ? MV_COLS : 1];
    __shared__ double2 xd[F32 ? 1 : MV_COLS];
    __shared__ int last;
    extern __shared__ double2 sums[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int64_t j0 = (int64_t)by * MV_COLS;
    const int jn = (int)min((int64_t)MV_COLS, n - j0);
    for (int t = tid; t < MV_COLS; t += 32 * SMALL_WARPS) {
        const double2 x = t < jn ? v[j0 + t] : make_double2(0, 0);
        if (F32) {
            const float hx = (float)x.x, hy = (float)x.y;
            xh[t] = make_float2(hx, hy);
            if (EXACT) xl[t] = make_float2((float)(x.x - (double)hx), (float)(x.y - (double)hy));
        } else {
            xd[t] = x;
        }
    }
    __syncthreads();
    const int64_t b0 = (int64_t)bx * SMALL_ROWS;
    double2* part = bt.part + g.p + (size_t)by * g.n_pad;
    if (F32 && !EXACT) {
        float2* gs = reinterpret_cast<float2*>(sums);  // [group][row]
        const int64_t i0 = b0 + 2 * lane;
        if (i0 < n) {
            const bool pair = i0 + 1 < n;
            const float2* A = reinterpret_cast<const float2*>(bt.A) + g.a + i0;
            for (int q0 = warp * U; q0 < jn; q0 += SMALL_WARPS * U) {
                float4 a[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int q = q0 + u;
                    if (q < jn) {
                        const float2* col = A + (j0 + q) * lda;
                        if (pair) a[u] = __ldcs(reinterpret_cast<const float4*>(col));
                        else { float2 t = col[0]; a[u] = make_float4(t.x, t.y, 0.f, 0.f); }
                    } else {
                        a[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                    }
                }
                float b0_ = 0, b1 = 0, b2 = 0, b3 = 0;
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const float2 H = xh[q0 + u];
                    const float4 w = a[u];
                    b0_ = fmaf(w.x, H.x, fmaf(-w.y, H.y, b0_));
                    b1 = fmaf(w.x, H.y, fmaf(w.y, H.x, b1));
                    b2 = fmaf(w.z, H.x, fmaf(-w.w, H.y, b2));
                    b3 = fmaf(w.z, H.y, fmaf(w.w, H.x, b3));
                }
                reinterpret_cast<float4*>(gs)[(q0 / U) * (SMALL_ROWS / 2) + lane] = make_float4(b0_, b1, b2, b3);
            }
        }
        __syncthreads();
        if (tid < 2 * SMALL_ROWS && b0 + (tid >> 1) < n) {
            const float* f = reinterpret_cast<const float*>(gs) + tid;
            const int groups = (jn + U - 1) / U;
            float h = 0, l = 0, e, t;
#pragma unroll 4
            for (int q = 0; q < groups; ++q) {
                two_sum(h, f[(size_t)q * 2 * SMALL_ROWS], t, e);
                h = t;
                l += e;
            }
            reinterpret_cast<double*>(part + b0)[tid] = (double)h + (double)l;
        }
    } else {
        double2 r0 = make_double2(0, 0), r1 = make_double2(0, 0);
        if (F32) {
            const int64_t i0 = b0 + 2 * lane;
            if (i0 < n) {
                const bool pair = i0 + 1 < n;
                const float2* A = reinterpret_cast<const float2*>(bt.A) + g.a + i0;
                float h0 = 0, l0 = 0, h1 = 0, l1 = 0, h2 = 0, l2 = 0, h3 = 0, l3 = 0;
                for (int q0 = warp * U; q0 < jn; q0 += SMALL_WARPS * U) {
                    float4 a[U], z[EXACT == 2 ? U : 1];
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const int q = q0 + u;
                        const float2* col = A + (j0 + (q < jn ? q : 0)) * lda;
                        if (q >= jn) a[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                        else if (pair) a[u] = __ldcs(reinterpret_cast<const float4*>(col));
                        else { float2 t = col[0]; a[u] = make_float4(t.x, t.y, 0.f, 0.f); }
                        if (EXACT == 2) {
                            const float2* cl = col + bt.split_lo;
                            if (q >= jn) z[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                            else if (pair) z[u] = __ldcs(reinterpret_cast<const float4*>(cl));
                            else { float2 t = cl[0]; z[u] = make_float4(t.x, t.y, 0.f, 0.f); }
                        }
                    }
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const float2 H = xh[q0 + u], L = xl[q0 + u];
                        const float4 w = a[u];
                        ff_acc(h0, l0, w.x, H.x); ff_acc(h0, l0, -w.y, H.y);
                        ff_acc(h1, l1, w.x, H.y); ff_acc(h1, l1, w.y, H.x);
                        ff_acc(h2, l2, w.z, H.x); ff_acc(h2, l2, -w.w, H.y);
                        ff_acc(h3, l3, w.z, H.y); ff_acc(h3, l3, w.w, H.x);
                        l0 = fmaf(w.x, L.x, fmaf(-w.y, L.y, l0));
                        l1 = fmaf(w.x, L.y, fmaf(w.y, L.x, l1));
                        l2 = fmaf(w.z, L.x, fmaf(-w.w, L.y, l2));
                        l3 = fmaf(w.z, L.y, fmaf(w.w, L.x, l3));
                        if (EXACT == 2) {
                            const float4 y = z[EXACT == 2 ? u : 0];
                            l0 = fmaf(y.x, H.x, fmaf(-y.y, H.y, l0));
                            l1 = fmaf(y.x, H.y, fmaf(y.y, H.x, l1));
                            l2 = fmaf(y.z, H.x, fmaf(-y.w, H.y, l2));
                            l3 = fmaf(y.z, H.y, fmaf(y.w, H.x, l3));
                        }
                    }
                }
                r0 = make_double2((double)h0 + (double)l0, (double)h1 + (double)l1);
                r1 = make_double2((double)h2 + (double)l2, (double)h3 + (double)l3);
            }
            sums[warp * SMALL_ROWS + 2 * lane] = r0;
            sums[warp * SMALL_ROWS + 2 * lane + 1] = r1;
        } else {
            // (rows lane and lane + 32: each load of a warp is 512 bytes in one piece)
            const int64_t i0 = b0 + lane;
            const bool in0 = i0 < n, in1 = i0 + 32 < n;
            const double2* A = reinterpret_cast<const double2*>(bt.A) + g.a + i0;
            for (int q0 = warp * U; q0 < jn; q0 += SMALL_WARPS * U) {
                double2 a0[U], a1[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int q = q0 + u;
                    const double2* col = A + (j0 + (q < jn ? q : 0)) * lda;
                    a0[u] = (q < jn && in0) ? __ldcs(col) : make_double2(0, 0);
                    a1[u] = (q < jn && in1) ? __ldcs(col + 32) : make_double2(0, 0);
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const double2 xv = xd[q0 + u];
                    cfma(r0, a0[u], xv);
                    cfma(r1, a1[u], xv);
                }
            }
            sums[warp * SMALL_ROWS + lane] = r0;
            sums[warp * SMALL_ROWS + lane + 32] = r1;
        }
        __syncthreads();
        if (tid < 2 * SMALL_ROWS && b0 + (tid >> 1) < n) {
            const double* f = reinterpret_cast<const double*>(sums) + tid;
            double t = f[0];
#pragma unroll
            for (int w = 1; w < SMALL_WARPS; ++w) t += f[w * 2 * SMALL_ROWS];
            reinterpret_cast<double*>(part + b0)[tid] = t;
        }
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) {
        int* tk = bt.tickets + g.t + bx;
        last = (atomicAdd(tk, 1) == g.cb - 1);
        if (last) *tk = 0;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    if (tid < 2 * SMALL_ROWS && b0 + (tid >> 1) < n) {
        const double* p = reinterpret_cast<const double*>(bt.part + g.p + b0) + tid;
        double acc = 0;
        for (int c = 0; c < g.cb; ++c) acc += p[(size_t)c * 2 * g.n_pad];
        reinterpret_cast<double*>(bt.W + g.v + b0)[tid] = acc;
    }
}

// ---------------------------------------------------------------------------
// Block-wide FP64 reductions (1024 threads).
__device__ __forceinline__ double block_sum(double v, double* sh) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) sh[w] = v;
    __syncthreads();
    if (w == 0) {
        v = l < (int)(blockDim.x >> 5) ? sh[l] : 0.0;
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (l == 0) sh[32] = v;
    }
    __syncthreads();
    return sh[32];
}

__device__ double vec_norm(const double2* v, int64_t n, double* sh) {
    double s = 0;
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) s += v[i].x * v[i].x + v[i].y * v[i].y;
    return sqrt(block_sum(s, sh));
}

// Krylov state of a cycle that starts with residual norm rn (one thread).
__device__ __forceinline__ void gm_cycle_state(const GmBatch& bt, int s, double rn) {
    GmSmall sm = gm_small(bt, s);
    for (int i = 0; i <= bt.m; ++i) sm.beta[i] = make_double2(0, 0);
    for (int i = 0; i < bt.m; ++i) { sm.cs[i] = make_double2(0, 0); sm.sn[i] = make_double2(0, 0); }
    sm.beta[0] = make_double2(rn, 0.0);
    bt.st[s].k = 0;
}

// Start of the first cycle (gmres.rs:84-106; gm_check_kernel starts the others): r = b - A x, q_0 = r / ||r||, beta_0 = ||r||.
__global__ void __launch_bounds__(AR_THREADS) gm_start_kernel(GmBatch bt) {
    const int s = blockIdx.x;
    GmState& st = bt.st[s];
    if (st.done || !st.need_start) return;
    __shared__ double sh[80];
    const GmView g = gm_view(bt, s);
    const int64_t n = g.n;
    const double2* b = bt.B + g.v;
    const double2* W = bt.W + g.v;
    double2* Q = bt.Q + g.q;
    const bool zero_x = !bt.ref_dotc;  // x = 0, and the reference's A x is not formed
    double acc = 0;
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
        double2 r = zero_x ? b[i] : csub(b[i], W[i]);
        Q[i] = r;
        acc += r.x * r.x + r.y * r.y;
    }
    double rn = sqrt(block_sum(acc, sh));
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
        double2 r = Q[i];
        Q[i] = make_double2(r.x / rn, r.y / rn);
    }
    double xn = vec_norm(bt.X + g.v, n, sh);
    if (threadIdx.x == 0) {
        st.xnorm = xn;
        st.error = rn / (st.anorm * xn + st.bnorm);
        gm_cycle_state(bt, s, rn);
        st.need_start = 0;
        st.check = 0;
        st.num_mv += zero_x ? 0 : 1;
    }
}

// ---------------------------------------------------------------------------
// Gram-Schmidt of the mixed and refined forms across the whole GPU: classical
// Gram-Schmidt applied twice (the second pass re-orthogonalises; as accurate
// as the modified form), in FP64.  Every CTA owns a chunk of rows of one
// system: the dots kernel forms its chunk's contribution to q_i^H w for every
// i <= k, the update kernel adds the chunks' contributions in a fixed order and
// subtracts Q h from its rows (and, after the second pass, leaves the squared
// norm of its rows).  Systems pending a
// Krylov step only (the Arnoldi kernel's predicate).
//
// FP64 instructions bound both (65 clocks per warp instruction and SM quarter),
// so a small batch is cut into chunks of down to 64 rows until the CTAs cover
// the SMs, and a basis vector takes eight lanes: a reduction over 32 lanes
// would cost as much as the products of 64 rows.  (Four systems of n = 1280, 12
// chunks of 512 rows and a warp per vector: 10.5 us per kernel; 80 chunks of 64:
// 3.7 and 5.3 us.)
constexpr int GS_ROWS = 512, GS_THREADS = 256;

__device__ __forceinline__ bool gm_arnoldi_active(const GmState& st) {
    return !(st.done || st.need_start || st.check);
}

// Sum over the eight lanes of a group; every lane gets it.
__device__ __forceinline__ double2 sum8(double2 v) {
    const double s = sum8_parts(v);
    const int base = threadIdx.x & 24;
    return make_double2(__shfl_sync(0xffffffffu, s, base), __shfl_sync(0xffffffffu, s, base + 1));
}

__global__ void __launch_bounds__(GS_THREADS) gm_gs_dots_kernel(GmBatch bt) {
    const int s = blockIdx.y, c = blockIdx.x;
    const GmState& st = bt.st[s];
    if (!gm_arnoldi_active(st)) return;
    const GmView g = gm_view(bt, s);
    const int64_t r0 = (int64_t)c * bt.gs_rows;
    if (r0 >= g.n) return;
    const int rows = (int)min((int64_t)bt.gs_rows, g.n - r0);
    __shared__ double2 ws[GS_ROWS];
    const double2* W = bt.W + g.v + r0;
    for (int l = threadIdx.x; l < rows; l += GS_THREADS) ws[l] = W[l];
    __syncthreads();
    const int grp = threadIdx.x >> 3, lane = threadIdx.x & 7;
    const double2* Q = bt.Q + g.q + r0;
    double2* part = bt.gs_part + ((size_t)s * bt.gs_chunks + c) * (bt.m + 1);
    // few vectors: several groups share the rows of one (16 systems of n = 6144,
    // k below 8: 13.7 us per kernel with a group each, 7.2 this way)
    int split = 1;
    while (2 * split * (st.k + 1) <= GS_THREADS / 8) split *= 2;
    if (split > 1) {
        __shared__ double2 psum[GS_THREADS / 8];
        const int i = grp / split;
        double2 acc = make_double2(0, 0);
        if (i <= st.k) {
            const double2* qi = Q + (size_t)i * g.n;
            for (int l = 8 * (grp % split) + lane; l < rows; l += 8 * split) cfma(acc, cconj(qi[l]), ws[l]);
        }
        acc = sum8(acc);
        if (lane == 0) psum[grp] = acc;
        __syncthreads();
        if (threadIdx.x <= st.k) {
            acc = psum[threadIdx.x * split];
            for (int q = 1; q < split; ++q) acc = cadd(acc, psum[threadIdx.x * split + q]);
            part[threadIdx.x] = acc;
        }
        return;
    }
    for (int i0 = 0; i0 <= st.k; i0 += GS_THREADS / 8) {
        const int i = i0 + grp;
        if (i0 + (grp & ~3) > st.k) break;  // (a whole warp)
        const double2* qi = Q + (size_t)min(i, st.k) * g.n;
        double2 acc = make_double2(0, 0);
        for (int l = lane; l < rows; l += 8) cfma(acc, cconj(qi[l]), ws[l]);
        acc = sum8(acc);
        if (lane == 0 && i <= st.k) part[i] = acc;
    }
}

// pass 0: hk1[i] = h_i; pass 1: hk1[i] += h_i and the chunk's squared norm.
__global__ void __launch_bounds__(GS_THREADS) gm_gs_update_kernel(GmBatch bt, int pass) {
    const int s = blockIdx.y, c = blockIdx.x;
    const GmState& st = bt.st[s];
    if (!gm_arnoldi_active(st)) return;
    const GmView g = gm_view(bt, s);
    const int64_t r0 = (int64_t)c * bt.gs_rows;
    if (r0 >= g.n) return;
    const int rows = (int)min((int64_t)bt.gs_rows, g.n - r0);
    const int k = st.k;
    const int nch = (int)((g.n + bt.gs_rows - 1) / bt.gs_rows);
    extern __shared__ double2 hsum[];  // k + 1 coefficients
    __shared__ double2 partial[GS_THREADS];
    __shared__ double red[GS_THREADS / 32];
    const double2* part = bt.gs_part + (size_t)s * bt.gs_chunks * (bt.m + 1);
    const int grp = threadIdx.x >> 3, lane = threadIdx.x & 7;
    for (int i0 = 0; i0 <= k; i0 += GS_THREADS / 8) {
        const int i = i0 + grp;
        if (i0 + (grp & ~3) > k) break;
        double2 h = make_double2(0, 0);
        for (int cc = lane; cc < nch; cc += 8) h = cadd(h, part[(size_t)cc * (bt.m + 1) + min(i, k)]);
        h = sum8(h);
        if (lane == 0 && i <= k) hsum[i] = h;
    }
    __syncthreads();
    if (c == 0) {
        GmSmall sm = gm_small(bt, s);
        for (int i = threadIdx.x; i <= k; i += GS_THREADS) sm.hk1[i] = pass == 0 ? hsum[i] : cadd(sm.hk1[i], hsum[i]);
    }
    double2* W = bt.W + g.v + r0;
    const double2* Q = bt.Q + g.q + r0;
    double nn = 0;
    // rows x groups of coefficients: with fewer than 256 rows the threads share
    // a row's coefficients
    const int wide = min(bt.gs_rows, GS_THREADS), groups = GS_THREADS / wide;
    const int lr = threadIdx.x % wide, kg = threadIdx.x / wide;
    for (int l0 = 0; l0 < rows; l0 += wide) {
        const int l = l0 + lr;
        double2 a = make_double2(0, 0);
        if (l < rows) {
            if (kg == 0) a = W[l];
            for (int i = kg; i <= k; i += groups) cfma(a, cneg(hsum[i]), Q[(size_t)i * g.n + l]);
        }
        if (groups > 1) {
            partial[threadIdx.x] = a;
            __syncthreads();
            if (kg == 0)
                for (int q = 1; q < groups; ++q) a = cadd(a, partial[q * wide + lr]);
        }
        if (l < rows && kg == 0) {
            W[l] = a;
            nn = fma(a.x, a.x, fma(a.y, a.y, nn));
        }
    }
    if (pass == 1) {
        for (int o = 16; o > 0; o >>= 1) nn += __shfl_down_sync(0xffffffffu, nn, o);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = nn;
        __syncthreads();
        if (threadIdx.x == 0) {
            double t = 0;
            for (int w = 0; w < wide / 32; ++w) t += red[w];
            bt.gs_norm[(size_t)s * bt.gs_chunks + c] = t;
        }
    }
}

// The small part of an Arnoldi step, in shared memory: the new column h of H
// turned by the earlier rotations, the new one, the residual estimate and, where
// the step is checked, y (gmres.rs:146-157, 178-202).
struct GmStep {
    double2 *h, *a, *cs, *sn;  // k + 1 entries each
    double2 *dinv, *y;         // of the triangular solve, in the place of a and cs
    double2 *cs_k, *sn_k, *beta_k, *beta_k1;
    double *scale, *error;
    int* chk;
};
constexpr size_t gm_step_smem(int m) { return sizeof(double2) * 4 * (size_t)(m + 1); }
#define GM_STEP_SHARED(name, smem)                                                                         \
    __shared__ double2 name##_z[4];                                                                        \
    __shared__ double name##_d[2];                                                                         \
    __shared__ int name##_i;                                                                               \
    GmStep name;                                                                                           \
    name.h = smem; name.a = name.h + (bt.m + 1); name.cs = name.a + (bt.m + 1);                            \
    name.sn = name.cs + (bt.m + 1); name.dinv = name.a; name.y = name.cs;                                  \
    name.cs_k = name##_z; name.sn_k = name##_z + 1; name.beta_k = name##_z + 2; name.beta_k1 = name##_z + 3; \
    name.scale = name##_d; name.error = name##_d + 1; name.chk = &name##_i

// One warp; nn = |w|^2.
__device__ __forceinline__ void gm_rotate(const GmStep& t, const GmState& st, const GmSmall& sm, double nn) {
    const int k = st.k, lane = threadIdx.x & 31;
    // a_i = the entry rotation i meets: a_0 = h_0, a_{i+1} = -conj(sn_i) a_i + cs_i h_{i+1}
    // (lane 0 the real, lane 1 the imaginary part; cs_i h_{i+1} is laid down beforehand)
    for (int i = lane; i < k; i += 32)
        t.a[i + 1] = make_double2(t.cs[i].x * t.h[i + 1].x, t.cs[i].x * t.h[i + 1].y);
    __syncwarp();
    double2 cur = t.h[0];
    for (int i = 0; i < k; ++i) {
        const double2 ss = t.sn[i], b = t.a[i + 1];
        if (lane == 0) t.a[i] = cur;
        const double p = lane ? cur.y : cur.x, q = lane ? -cur.x : cur.y;
        const double v = fma(-ss.y, q, fma(-ss.x, p, lane ? b.y : b.x));
        cur.x = __shfl_sync(0xffffffffu, v, 0);
        cur.y = __shfl_sync(0xffffffffu, v, 1);
    }
    __syncwarp();
    // the rotated entries, off the chain
    for (int i = lane; i < k; i += 32)
        t.a[i] = cadd(make_double2(t.cs[i].x * t.a[i].x, t.cs[i].x * t.a[i].y), cmul(t.sn[i], t.h[i + 1]));
    __syncwarp();
    for (int i = lane; i < k; i += 32) t.h[i] = t.a[i];
    // new rotation (LAWN 148): v1 = cur, v2 = |w| real.  The roots and the
    // quotients are taken side by side, a lane each: one costs 600 clocks.
    const double c2 = cnorm2(cur);
    double rt = sqrt(lane == 0 ? nn : lane == 1 ? c2 : c2 + nn);
    if (lane == 1 && !(c2 > 1e-280)) rt = cabs_(cur);
    const double hn = __shfl_sync(0xffffffffu, rt, 0), a1 = __shfl_sync(0xffffffffu, rt, 1),
                 r = __shfl_sync(0xffffffffu, rt, 2);
    const double qt = (lane == 0 ? cur.x : lane == 1 ? cur.y : lane == 2 ? a1 : lane == 3 ? hn : 1.0) /
                      (lane < 2 ? a1 : lane < 4 ? r : hn);
    double2 signf = make_double2(__shfl_sync(0xffffffffu, qt, 0), __shfl_sync(0xffffffffu, qt, 1));
    const double c0 = __shfl_sync(0xffffffffu, qt, 2), t0 = __shfl_sync(0xffffffffu, qt, 3),
                 sc = __shfl_sync(0xffffffffu, qt, 4);
    if (cur.x == 0.0 && cur.y == 0.0) signf = make_double2(1.0, 0.0);
    const double2 s0 = make_double2(signf.x * t0, signf.y * t0);
    const double2 bk = sm.beta[k];
    const double2 b1 = cmul(cneg(cconj(s0)), bk), b0 = make_double2(bk.x * c0, bk.y * c0);
    if (lane == 0) {
        t.h[k] = cadd(make_double2(c0 * cur.x, c0 * cur.y), make_double2(s0.x * hn, s0.y * hn));
        *t.scale = sc;
        *t.cs_k = make_double2(c0, 0.0);
        *t.sn_k = s0;
        *t.beta_k = b0;
        *t.beta_k1 = b1;
        *t.error = cabs_(b1) / (st.anorm * st.xnorm + st.bnorm);
        *t.chk = (*t.error < st.tol) || (k == st.m - 1);
    }
}

// The whole CTA: y = H_k^{-1} beta_k, column by column from the last (H_k is
// upper triangular after the rotations).
__device__ __forceinline__ void gm_solve_y(const GmStep& t, const GmSmall& sm, int k, int m) {
    for (int i = threadIdx.x; i <= k; i += blockDim.x)
        t.dinv[i] = cdiv(make_double2(1.0, 0.0), i == k ? t.h[k] : sm.H[(size_t)i * (m + 1) + i]);
    for (int i = threadIdx.x; i <= k; i += blockDim.x) t.y[i] = i == k ? *t.beta_k : sm.beta[i];
    __syncthreads();
    if (threadIdx.x < 32)
        for (int i = k; i >= 0; --i) {
            const double2 yi = cmul(t.y[i], t.dinv[i]);
            __syncwarp();
            if (threadIdx.x == 0) t.y[i] = yi;
            for (int r = threadIdx.x; r < i; r += 32) {
                const double2 e = i == k ? t.h[r] : sm.H[(size_t)i * (m + 1) + r];
                t.y[r] = csub(t.y[r], cmul(e, yi));
            }
            __syncwarp();
        }
    __syncthreads();
}

// x += Q_k y, or Z_k y with flexible right preconditioning, rows l0 .. l1.
__device__ __forceinline__ void gm_add_correction(const GmBatch& bt, const GmView& g, const double2* y, int k,
                                                  int64_t l0, int64_t l1) {
    double2* x = bt.X + g.v;
    const double2* Zs = (bt.Z ? bt.Z : bt.Q) + g.q;
    for (int64_t l = l0 + threadIdx.x; l < l1; l += blockDim.x) {
        double2 v = x[l];
        for (int j = 0; j <= k; ++j) cfma(v, Zs[(size_t)j * g.n + l], y[j]);
        x[l] = v;
    }
}

// One CTA, when every other one is done with the state.
__device__ __forceinline__ void gm_record(const GmStep& t, GmState& st, const GmSmall& sm, int m) {
    const int k = st.k;
    for (int i = threadIdx.x; i <= k; i += blockDim.x) {
        sm.H[(size_t)k * (m + 1) + i] = t.h[i];
        if (*t.chk) sm.y[i] = t.y[i];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        sm.H[(size_t)k * (m + 1) + k + 1] = make_double2(0, 0);
        sm.cs[k] = *t.cs_k;
        sm.sn[k] = *t.sn_k;
        sm.beta[k] = *t.beta_k;
        sm.beta[k + 1] = *t.beta_k1;
        st.error = *t.error;
        st.num_mv += 1;
        st.iterations += 1;
        st.check = *t.chk;
        if (!*t.chk) st.k = k + 1;
    }
}

// The rest of an Arnoldi step after the Gram-Schmidt kernels: Givens rotations
// (gmres.rs:178-202), residual estimate and, when the estimate passes or the
// cycle ends, y = H_k^{-1} beta_k (gmres.rs:146-157); q_{k+1} = w / |w| and
// x += Z_k y by chunks of rows.  Every CTA of a system does the small part for
// itself (so that nothing but the chunks' results has to travel); the last one
// of a system to finish records it.
//
// The chain bounds it: two dependent FP64 multiply-adds (130 clocks) and a
// shuffle per earlier rotation, the other products of a rotation off the chain,
// one lane per unknown in the triangular solve.  (One thread doing all of it
// took 36 us per step at n = 1280, k up to 30, and x += Z y another 40 us on
// one SM; now 12.5 us on average with the update.)
constexpr int GV_STEP_THREADS = 256;
__global__ void __launch_bounds__(GV_STEP_THREADS) gm_givens_kernel(GmBatch bt, int chunks) {
    const int s = blockIdx.y;
    GmState& st = bt.st[s];
    if (!gm_arnoldi_active(st)) return;
    extern __shared__ double2 sh2[];
    __shared__ int last;
    GM_STEP_SHARED(t, sh2);
    const GmView g = gm_view(bt, s);
    const int64_t n = g.n;
    const int k = st.k, m = bt.m, tid = threadIdx.x;
    const GmSmall sm = gm_small(bt, s);
    for (int i = tid; i <= k; i += GV_STEP_THREADS) t.h[i] = sm.hk1[i];
    for (int i = tid; i < k; i += GV_STEP_THREADS) {
        t.cs[i] = sm.cs[i];
        t.sn[i] = sm.sn[i];
    }
    __syncthreads();
    if (tid < 32) {
        double nn = 0;
        const int nch = (int)((n + bt.gs_rows - 1) / bt.gs_rows);  // this system's chunks (ragged batches)
        for (int c = tid; c < nch; c += 32) nn += bt.gs_norm[(size_t)s * bt.gs_chunks + c];
        for (int o = 16; o > 0; o >>= 1) nn += __shfl_xor_sync(0xffffffffu, nn, o);
        gm_rotate(t, st, sm, nn);
    }
    __syncthreads();
    if (*t.chk) gm_solve_y(t, sm, k, m);
    // this CTA's rows
    const int64_t per = (n + chunks - 1) / chunks, l0 = (int64_t)blockIdx.x * per, l1 = min(n, l0 + per);
    const double sc = *t.scale;
    const double2* Wg = bt.W + g.v;
    double2* qk1 = bt.Q + g.q + (size_t)(k + 1) * n;
    for (int64_t l = l0 + tid; l < l1; l += GV_STEP_THREADS) {
        const double2 w = Wg[l];
        qk1[l] = make_double2(w.x * sc, w.y * sc);
    }
    if (*t.chk) gm_add_correction(bt, g, t.y, k, l0, l1);
    __threadfence();
    __syncthreads();
    if (tid == 0) {
        int* tk = bt.tickets + g.t;  // (between the products' launches: zero)
        last = atomicAdd(tk, 1) == chunks - 1;
        if (last) *tk = 0;
    }
    __syncthreads();
    if (last) gm_record(t, st, sm, m);
}

// Arnoldi step k of the reference's form: modified Gram-Schmidt (gmres.rs:158-176)
// with its product conj(w)^T q, and the small part as above.  One cluster per
// system; a CTA holds its share of w in shared memory where it fits
// (`w_in_smem`), and every coefficient is one exchange: each warp sends its part
// of the sum to all CTAs, which add the parts in one order.  Two slots by parity
// are enough, since nobody sends for step i + 1 before it has read step i.
//
// FP64 instructions bound it: subtracting h_i q_i and the next product are one
// pass over the rows, with q_{i+1} loaded before the wait.  (One CTA with two
// block-wide reductions per coefficient: 23 us each at n = 6144; now 3.5 us, 16
// steps 3.15 -> 0.50 ms.)
constexpr int MG_THREADS = 128, MG_WARPS = MG_THREADS / 32, MG_UNROLL = 4;

__global__ void __launch_bounds__(MG_THREADS) gm_arnoldi_kernel(GmBatch bt, int w_in_smem, int cluster) {
    const int s = blockIdx.x / cluster, rank = blockIdx.x % cluster;
    GmState& st = bt.st[s];
    if (!gm_arnoldi_active(st)) return;
    extern __shared__ double2 sh2[];
    __shared__ double2 slot[2][MAX_CLUSTER * MG_WARPS];
    __shared__ uint64_t mb[2];
    GM_STEP_SHARED(t, sh2);
    const GmView g = gm_view(bt, s);
    const int64_t n = g.n;
    const int k = st.k, m = bt.m, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const GmSmall sm = gm_small(bt, s);
    const int64_t per = (n + cluster - 1) / cluster, l0 = min(n, (int64_t)rank * per), l1 = min(n, l0 + per);
    const int rows = (int)(l1 - l0);
    const double2* Q = bt.Q + g.q + l0;
    double2* Wg = bt.W + g.v + l0;
    double2* w = w_in_smem ? sh2 + 4 * (m + 1) : Wg;
    const uint32_t bytes = (uint32_t)(cluster * MG_WARPS * sizeof(double2));
    const uint32_t bar = (uint32_t)__cvta_generic_to_shared(mb), box = (uint32_t)__cvta_generic_to_shared(slot);
    auto arm = [&](int p) {
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar + 8 * p), "r"(bytes) : "memory");
    };
    if (tid == 0) {
        for (int p = 0; p < 2; ++p)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar + 8 * p) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        arm(0);
        arm(1);
    }
    for (int i = tid; i < k; i += MG_THREADS) {
        t.cs[i] = sm.cs[i];
        t.sn[i] = sm.sn[i];
    }
    if (w_in_smem)
        for (int l = tid; l < rows; l += MG_THREADS) w[l] = Wg[l];
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    // (a thread's rows are its own from here on)
    bool ok = true;
    // this warp's part of step e's sum, to every CTA
    auto send = [&](int e, double2 acc) {
        const bool odd = lane & 1;
        double v = odd ? acc.y : acc.x;
        v += __shfl_xor_sync(0xffffffffu, odd ? acc.x : acc.y, 1);
        for (int o = 2; o < 32; o *= 2) v += __shfl_xor_sync(0xffffffffu, v, o);
        acc = make_double2(__shfl_sync(0xffffffffu, v, 0), __shfl_sync(0xffffffffu, v, 1));
        const int p = e & 1;
        if (lane < cluster)
            st_async16(peer_addr(box + (uint32_t)sizeof(double2) * (p * MAX_CLUSTER * MG_WARPS + rank * MG_WARPS + warp),
                                 lane),
                       peer_addr(bar + 8 * p, lane), as_uint4(acc));
    };
    // the sum of step e, the same in every thread
    auto collect = [&](int e) {
        const int p = e & 1;
        ok = ok && peers_arrived(&mb[p], (uint32_t)(e >> 1) & 1);
        ok = __all_sync(0xffffffffu, ok);
        const double* f = reinterpret_cast<const double*>(slot[p]);
        double v = 0;
        for (int q = lane; q < 2 * MG_WARPS * cluster; q += 32) v += f[q];
        for (int o = 2; o < 32; o *= 2) v += __shfl_xor_sync(0xffffffffu, v, o);
        const double2 h = make_double2(__shfl_sync(0xffffffffu, v, 0), __shfl_sync(0xffffffffu, v, 1));
        // for step e + 2, whose parts come after everyone has step e + 1's
        if (tid == 0) arm(p);
        return h;
    };
    double2 acc = make_double2(0, 0);
    for (int l = tid; l < rows; l += MG_THREADS) cfma(acc, cconj(w[l]), Q[l]);
    for (int i = 0; i <= k && ok; ++i) {
        send(i, acc);
        const double2 *qi = Q + (size_t)i * n, *qn = Q + (size_t)(i + 1) * n;
        const bool more = i < k;
        double2 a[MG_UNROLL], b[MG_UNROLL];
        auto load = [&](int base) {
#pragma unroll
            for (int u = 0; u < MG_UNROLL; ++u) {
                const int l = base + u * MG_THREADS;
                a[u] = l < rows ? qi[l] : make_double2(0, 0);
                b[u] = l < rows && more ? qn[l] : make_double2(0, 0);
            }
        };
        load(tid);
        const double2 h = collect(i);
        if (tid == 0) t.h[i] = h;
        acc = make_double2(0, 0);
        for (int base = tid; base < rows; base += MG_UNROLL * MG_THREADS) {
            double2 qa[MG_UNROLL], qb[MG_UNROLL];
#pragma unroll
            for (int u = 0; u < MG_UNROLL; ++u) {
                qa[u] = a[u];
                qb[u] = b[u];
            }
            load(base + MG_UNROLL * MG_THREADS);
#pragma unroll
            for (int u = 0; u < MG_UNROLL; ++u) {
                const int l = base + u * MG_THREADS;
                if (l < rows) {
                    double2 v = w[l];
                    cfma(v, cneg(h), qa[u]);
                    w[l] = v;
                    if (more) cfma(acc, cconj(v), qb[u]);
                    else acc.x = fma(v.x, v.x, fma(v.y, v.y, acc.x));
                }
            }
        }
    }
    double nn = 0;
    if (ok) {
        send(k + 1, acc);
        nn = collect(k + 1).x;
    }
    ok = __syncthreads_and(ok);
    if (ok) {
        if (tid < 32) gm_rotate(t, st, sm, nn);
        __syncthreads();
        if (*t.chk) gm_solve_y(t, sm, k, m);
        const double sc = *t.scale;
        double2* qk1 = bt.Q + g.q + (size_t)(k + 1) * n + l0;
        for (int l = tid; l < rows; l += MG_THREADS) qk1[l] = make_double2(w[l].x * sc, w[l].y * sc);
        if (*t.chk) gm_add_correction(bt, g, t.y, k, l0, l1);
    }
    if (!ok && tid == 0) {  // a wait ran out: the system ends here, gm_require_waits reports it
        st.gave_up = 1;
        st.done = 1;
        __threadfence();
    }
    // nobody leaves while its shared memory may still be written, and the state
    // changes when everyone has read it
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (ok && rank == 0) gm_record(t, st, sm, m);
}

// True residual check (gmres.rs:122-138), and the start of the next cycle
// (gmres.rs:84-106) where the check ends one: x has not changed since, so its
// residual is the one at hand.
__global__ void __launch_bounds__(AR_THREADS) gm_check_kernel(GmBatch bt) {
    const int s = blockIdx.x;
    GmState& st = bt.st[s];
    if (st.done || !st.check) return;
    __shared__ double sh[80];
    __shared__ int restart;
    const GmView g = gm_view(bt, s);
    const int64_t n = g.n;
    const double2* b = bt.B + g.v;
    const double2* W = bt.W + g.v;
    double acc = 0;
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
        double2 r = csub(b[i], W[i]);
        acc += r.x * r.x + r.y * r.y;
    }
    double rn = sqrt(block_sum(acc, sh));
    double xn = vec_norm(bt.X + g.v, n, sh);
    if (threadIdx.x == 0) {
        st.num_mv += 1;
        st.xnorm = xn;
        st.error = rn / (st.anorm * xn + st.bnorm);
        st.check = 0;
        restart = 0;
        if (st.error < st.tol) {
            st.done = 1;
            st.converged = 1;
        } else if (st.k == st.m - 1 || !bt.ref_dotc) {
            // End of the cycle.  Outside the reference-faithful mode a failed
            // check also restarts from the updated x (an iterative-refinement
            // step), instead of continuing the Arnoldi process and adding the
            // Krylov correction to x a second time at the next check.
            st.restarts += 1;
            if (st.restarts >= st.max_restarts) st.done = 1;
            else restart = 1;
        } else {
            st.k += 1;
        }
    }
    __syncthreads();
    if (!restart) return;
    // the next cycle starts from the residual that was just formed
    double2* Q = bt.Q + g.q;
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
        const double2 r = csub(b[i], W[i]);
        Q[i] = make_double2(r.x / rn, r.y / rn);
    }
    if (threadIdx.x == 0) {
        gm_cycle_state(bt, s, rn);
        st.num_mv += 1;  // (A x counts for the check and for the start)
    }
}

// Zero initial guess and the per-system constants.
__global__ void gm_init_kernel(GmBatch bt, const double* anorm, double tol, int64_t max_restarts,
                               const double* __restrict__ tols, const int64_t* __restrict__ maxrs,
                               const int* __restrict__ ms) {
    const int s = blockIdx.x;
    __shared__ double sh[80];
    const GmView g = gm_view(bt, s);
    const int64_t n = g.n;
    double2* x = bt.X + g.v;
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) x[i] = make_double2(0, 0);
    double bn = vec_norm(bt.B + g.v, n, sh);
    if (threadIdx.x == 0) {
        GmState& st = bt.st[s];
        st.anorm = anorm[s];
        st.bnorm = bn;
        st.tol = tols ? tols[s] : tol;
        st.m = ms ? ms[s] : bt.m;
        st.xnorm = 0;
        st.error = 1.0;
        st.k = 0;
        st.need_start = 1;
        st.check = 0;
        st.done = 0;
        st.converged = 0;
        st.gave_up = 0;
        st.num_mv = 0;
        st.iterations = 0;
        st.restarts = 0;
        st.max_restarts = maxrs ? maxrs[s] : max_restarts;
        if (bn == 0.0) {  // zero right-hand side: x = 0 is exact
            st.done = 1;
            st.converged = 1;
            st.error = 0;
        }
    }
}

// Frobenius norms of a batch of matrices (FP64 or FP32 entries): CTAs stride
// over columns, threads over rows (coalesced, no index division).
template <typename T>
__global__ void batch_frob_kernel(const void* A, int64_t n, int64_t lda, size_t mat_stride, double* part, int nb) {
    __shared__ double sh[80];
    int s = blockIdx.y;
    const T* M = reinterpret_cast<const T*>(A) + (size_t)s * mat_stride;
    double acc = 0;
    for (int64_t j = blockIdx.x; j < n; j += gridDim.x) {
        const T* col = M + j * lda;
        for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
            T v = col[i];
            acc += (double)v.x * (double)v.x + (double)v.y * (double)v.y;
        }
    }
    double r = block_sum(acc, sh);
    if (threadIdx.x == 0) part[(size_t)s * nb + blockIdx.x] = r;
}

__global__ void finish_norms_kernel(const double* part, int nb, int nsys, double* out) {
    int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nsys) return;
    double acc = 0;
    for (int b = 0; b < nb; ++b) acc += part[(size_t)s * nb + b];
    out[s] = sqrt(acc);
}

// ---------------------------------------------------------------------------
// Kernel attributes are process-wide, so the limits of dynamic shared memory are
// raised once per device to their caps and never lowered: a smaller solve on
// another thread cannot shrink one under a larger one's launch or graph.
namespace {
constexpr int AR_MAX_DEVICES = 64;
std::once_flag g_ar_smem_once[AR_MAX_DEVICES];
}  // namespace

static void gm_kernel_attributes(Context& ctx) {
    const int device = ctx.device;
    require(device >= 0 && device < AR_MAX_DEVICES, "device index out of range");
    // a failed set throws out of call_once, which leaves the flag unset so the
    // next call tries again
    std::call_once(g_ar_smem_once[device], [] {
        auto allow = [](const void* kernel, size_t bytes, const char* name) {
            cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
            if (err != cudaSuccess)
                throw Error(BEM_ERR_CUDA, std::string("cudaFuncSetAttribute(") + name + "): " + cudaGetErrorString(err));
        };
        allow((const void*)gm_arnoldi_kernel, AR_SMEM_CAP, "gm_arnoldi_kernel");
        BEM_CUDA(cudaFuncSetAttribute(gm_arnoldi_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        allow((const void*)gm_givens_kernel, AR_SMEM_CAP, "gm_givens_kernel");
        allow((const void*)gm_gs_update_kernel, AR_SMEM_CAP, "gm_gs_update_kernel");
        allow((const void*)gm_apply_small_kernel<float2, 0, 4>, small_smem<float2, 0, 4>(), "gm_apply_small_kernel");
    });
    if (!ctx.gm_cluster) ctx.gm_cluster = max_cluster((const void*)gm_arnoldi_kernel, MG_THREADS, AR_SMEM_CAP);
}

// Rows per Gram-Schmidt chunk: halved from 512 until the chunks cover the SMs.
static int gs_rows_for(const GmWorkspace& ws, int nsys, int64_t n) {
    int rows = GS_ROWS;
    while (rows > 64 && (n + rows - 1) / rows * nsys < ws.sms) rows /= 2;
    return rows;
}

void gm_prepare(Context& ctx, GmWorkspace& ws, int nsys, int64_t n, int m, const void* A, int64_t lda,
                size_t mat_stride, bool fp32, bool ref_dotc) {
    BEM_CUDA(cudaDeviceGetAttribute(&ws.sms, cudaDevAttrMultiProcessorCount, ctx.device));
    GmBatch& bt = ws.bt;
    bt.nsys = nsys;
    bt.n = n;
    bt.n_pad = (n + MV_ROWS - 1) / MV_ROWS * MV_ROWS;
    bt.m = m;
    bt.A = A;
    bt.lda = lda;
    bt.mat_stride = mat_stride;
    bt.ref_dotc = ref_dotc ? 1 : 0;
    bt.qstride = (size_t)n * (m + 1);
    ws.fp32 = fp32;
    int rb = (int)((n + MV_ROWS - 1) / MV_ROWS), cb = (int)((n + MV_COLS - 1) / MV_COLS);
    ws.rb = rb;
    ws.cb = cb;
    bt.rb = rb;
    bt.cb = cb;
    bt.tpr = TICKETS;
    bt.sys = nullptr;
    bt.mates = 0;
    bt.ntiles = 0;
    ws.sys_host.clear();
    size_t small = gm_small_size(m);
    size_t bytes = 0;
    auto carve = [&](size_t b) { size_t o = bytes; bytes += (b + 255) / 256 * 256; return o; };
    size_t oX = carve(sizeof(double2) * nsys * n), oB = carve(sizeof(double2) * nsys * n);
    size_t oQ = carve(sizeof(double2) * nsys * bt.qstride), oW = carve(sizeof(double2) * nsys * n);
    size_t oP = carve(sizeof(double2) * nsys * cb * bt.n_pad), oT = carve(sizeof(int) * nsys * rb * TICKETS);
    size_t oS = carve(sizeof(double2) * nsys * small), oSt = carve(sizeof(GmState) * nsys);
    size_t oN = carve(sizeof(double) * nsys * 1024 + sizeof(double) * nsys);
    // partial sums of the whole-GPU Gram-Schmidt (forms other than the reference's)
    bt.gs_rows = gs_rows_for(ws, nsys, n);
    const int gsc = ref_dotc ? 0 : (int)((n + bt.gs_rows - 1) / bt.gs_rows);
    size_t oG = gsc ? carve(sizeof(double2) * nsys * gsc * (m + 1)) : 0;
    size_t oGn = gsc ? carve(sizeof(double) * nsys * gsc) : 0;
    ws.memb().ensure(bytes);
    char* base = ws.memb().as<char>();
    bt.X = reinterpret_cast<double2*>(base + oX);
    bt.B = reinterpret_cast<double2*>(base + oB);
    bt.Q = reinterpret_cast<double2*>(base + oQ);
    bt.gs_chunks = gsc;
    bt.gs_part = gsc ? reinterpret_cast<double2*>(base + oG) : nullptr;
    bt.gs_norm = gsc ? reinterpret_cast<double*>(base + oGn) : nullptr;
    bt.W = reinterpret_cast<double2*>(base + oW);
    bt.part = reinterpret_cast<double2*>(base + oP);
    bt.tickets = reinterpret_cast<int*>(base + oT);
    bt.small = reinterpret_cast<double2*>(base + oS);
    bt.small_stride = small;
    bt.st = reinterpret_cast<GmState*>(base + oSt);
    ws.norm_part = reinterpret_cast<double*>(base + oN);
    ws.anorm = ws.norm_part + (size_t)nsys * 1024;
    BEM_CUDA(cudaMemsetAsync(bt.tickets, 0, sizeof(int) * nsys * rb * TICKETS, ctx.stream));
    gm_kernel_attributes(ctx);
}

// Same layout as gm_prepare, carved from caller-provided device memory instead
// of an allocation.  Returns the bytes the layout needs; when that exceeds
// `capacity` nothing is written and the workspace is left unset.
size_t gm_prepare_external(Context& ctx, GmWorkspace& ws, int nsys, int64_t n, int m, const void* A, int64_t lda,
                           size_t mat_stride, bool fp32, bool ref_dotc, void* mem, size_t capacity) {
    const int64_t n_pad = (n + MV_ROWS - 1) / MV_ROWS * MV_ROWS;
    const size_t qstride = (size_t)n * (m + 1);
    const int rb = (int)((n + MV_ROWS - 1) / MV_ROWS), cb = (int)((n + MV_COLS - 1) / MV_COLS);
    const size_t small = gm_small_size(m);
    size_t bytes = 0;
    auto carve = [&](size_t b) { size_t o = bytes; bytes += (b + 255) / 256 * 256; return o; };
    size_t oX = carve(sizeof(double2) * nsys * n), oB = carve(sizeof(double2) * nsys * n);
    size_t oQ = carve(sizeof(double2) * nsys * qstride), oW = carve(sizeof(double2) * nsys * n);
    size_t oP = carve(sizeof(double2) * nsys * cb * n_pad), oT = carve(sizeof(int) * nsys * rb);
    size_t oS = carve(sizeof(double2) * nsys * small), oSt = carve(sizeof(GmState) * nsys);
    size_t oN = carve(sizeof(double) * nsys * 1024 + sizeof(double) * nsys);
    if (bytes > capacity) return bytes;
    BEM_CUDA(cudaDeviceGetAttribute(&ws.sms, cudaDevAttrMultiProcessorCount, ctx.device));
    GmBatch& bt = ws.bt;
    bt.nsys = nsys;
    bt.n = n;
    bt.n_pad = n_pad;
    bt.m = m;
    bt.A = A;
    bt.lda = lda;
    bt.mat_stride = mat_stride;
    bt.ref_dotc = ref_dotc ? 1 : 0;
    bt.qstride = qstride;
    ws.fp32 = fp32;
    ws.rb = rb;
    ws.cb = cb;
    bt.rb = rb;
    bt.cb = cb;
    bt.tpr = 1;  // caller memory: no finer tiling
    bt.sys = nullptr;
    bt.mates = 0;
    bt.ntiles = 0;
    ws.sys_host.clear();
    char* base = static_cast<char*>(mem);
    bt.X = reinterpret_cast<double2*>(base + oX);
    bt.B = reinterpret_cast<double2*>(base + oB);
    bt.Q = reinterpret_cast<double2*>(base + oQ);
    bt.gs_part = nullptr;  // (the reference form only)
    bt.gs_norm = nullptr;
    bt.gs_chunks = 0;
    bt.W = reinterpret_cast<double2*>(base + oW);
    bt.part = reinterpret_cast<double2*>(base + oP);
    bt.tickets = reinterpret_cast<int*>(base + oT);
    bt.small = reinterpret_cast<double2*>(base + oS);
    bt.small_stride = small;
    bt.st = reinterpret_cast<GmState*>(base + oSt);
    ws.norm_part = reinterpret_cast<double*>(base + oN);
    ws.anorm = ws.norm_part + (size_t)nsys * 1024;
    // the last-CTA tickets must start at zero; every other region is written
    // before it is read
    BEM_CUDA(cudaMemsetAsync(bt.tickets, 0, sizeof(int) * nsys * rb, ctx.stream));
    gm_kernel_attributes(ctx);
    return bytes;
}

void gm_prepare_ragged(Context& ctx, GmWorkspace& ws, const std::vector<int64_t>& ns,
                       const std::vector<int64_t>& ldas, const std::vector<size_t>& a_offs, int m, const void* A,
                       bool fp32) {
    const int nsys = (int)ns.size();
    require(nsys >= 1 && ldas.size() == ns.size() && a_offs.size() == ns.size(), "ragged batch: bad layout");
    std::vector<GmSys>& sys = ws.sys_host;
    sys.assign(nsys, GmSys{});
    size_t v = 0, q = 0, p = 0, t = 0;
    int64_t tiles = 0, tiles64 = 0, nmax = 0, npmax = 0;
    for (int s = 0; s < nsys; ++s) {
        GmSys& d = sys[s];
        d.n = ns[s];
        require(d.n >= 1 && ldas[s] >= d.n, "ragged batch: bad system size");
        d.lda = ldas[s];
        d.rb = (int)((d.n + MV_ROWS - 1) / MV_ROWS);
        d.cb = (int)((d.n + MV_COLS - 1) / MV_COLS);
        d.n_pad = (int64_t)d.rb * MV_ROWS;
        d.a_off = a_offs[s];
        d.v_off = v;
        d.q_off = q;
        d.p_off = p;
        d.t_off = t;
        d.tile0 = tiles;
        v += (size_t)d.n;
        q += (size_t)d.n * (m + 1);
        p += (size_t)d.cb * d.n_pad;
        t += (size_t)d.rb * TICKETS;
        d.tile64 = tiles64;
        tiles64 += (d.n + SMALL_ROWS - 1) / SMALL_ROWS * d.cb;
        tiles += (int64_t)d.rb * d.cb;
        nmax = std::max(nmax, d.n);
        npmax = std::max(npmax, d.n_pad);
    }
    BEM_CUDA(cudaDeviceGetAttribute(&ws.sms, cudaDevAttrMultiProcessorCount, ctx.device));
    const int mates = gm_pair_systems(sys);
    GmBatch& bt = ws.bt;
    bt.mates = mates;
    bt.nsys = nsys;
    bt.n = nmax;
    bt.n_pad = npmax;
    bt.m = m;
    bt.A = A;
    bt.lda = 0;
    bt.mat_stride = 0;
    bt.ref_dotc = 0;
    bt.qstride = 0;
    bt.rb = bt.cb = 0;
    bt.ntiles = tiles;
    bt.ntiles64 = tiles64;
    bt.tpr = TICKETS;
    ws.fp32 = fp32;
    ws.rb = ws.cb = 0;
    const size_t small = gm_small_size(m);
    size_t bytes = 0;
    auto carve = [&](size_t b) { size_t o = bytes; bytes += (b + 255) / 256 * 256; return o; };
    size_t oX = carve(sizeof(double2) * v), oB = carve(sizeof(double2) * v);
    size_t oQ = carve(sizeof(double2) * q), oW = carve(sizeof(double2) * v);
    size_t oP = carve(sizeof(double2) * p), oT = carve(sizeof(int) * t);
    size_t oS = carve(sizeof(double2) * nsys * small), oSt = carve(sizeof(GmState) * nsys);
    size_t oN = carve(sizeof(double) * nsys * 1024 + sizeof(double) * nsys);
    size_t oD = carve(sizeof(GmSys) * nsys);
    // partial sums of the whole-GPU Gram-Schmidt
    bt.gs_rows = gs_rows_for(ws, nsys, nmax);
    const int gsc = (int)((nmax + bt.gs_rows - 1) / bt.gs_rows);
    size_t oG = carve(sizeof(double2) * nsys * gsc * (m + 1));
    size_t oGn = carve(sizeof(double) * nsys * gsc);
    ws.memb().ensure(bytes);
    char* base = ws.memb().as<char>();
    bt.X = reinterpret_cast<double2*>(base + oX);
    bt.B = reinterpret_cast<double2*>(base + oB);
    bt.Q = reinterpret_cast<double2*>(base + oQ);
    bt.gs_chunks = gsc;
    bt.gs_part = reinterpret_cast<double2*>(base + oG);
    bt.gs_norm = reinterpret_cast<double*>(base + oGn);
    bt.W = reinterpret_cast<double2*>(base + oW);
    bt.part = reinterpret_cast<double2*>(base + oP);
    bt.tickets = reinterpret_cast<int*>(base + oT);
    bt.small = reinterpret_cast<double2*>(base + oS);
    bt.small_stride = small;
    bt.st = reinterpret_cast<GmState*>(base + oSt);
    ws.norm_part = reinterpret_cast<double*>(base + oN);
    ws.anorm = ws.norm_part + (size_t)nsys * 1024;
    GmSys* dsys = reinterpret_cast<GmSys*>(base + oD);
    BEM_CUDA(cudaMemcpyAsync(dsys, sys.data(), sizeof(GmSys) * nsys, cudaMemcpyHostToDevice, ctx.stream));
    bt.sys = dsys;
    BEM_CUDA(cudaMemsetAsync(bt.tickets, 0, sizeof(int) * t, ctx.stream));
    gm_kernel_attributes(ctx);
}

size_t gm_q_total(const GmWorkspace& ws) {
    if (ws.sys_host.empty()) return (size_t)ws.bt.nsys * ws.bt.qstride;
    const GmSys& d = ws.sys_host.back();
    return d.q_off + (size_t)d.n * (ws.bt.m + 1);
}

void gm_matrix_norms(Context& ctx, GmWorkspace& ws) {
    const int nb = 512;
    if (!ws.sys_host.empty()) {
        for (int s = 0; s < ws.bt.nsys; ++s) {
            const GmSys& d = ws.sys_host[s];
            dim3 g1(nb, 1);
            if (ws.fp32)
                batch_frob_kernel<float2><<<g1, 256, 0, ctx.stream>>>(
                    static_cast<const float2*>(ws.bt.A) + d.a_off, d.n, d.lda, 0, ws.norm_part + (size_t)s * nb, nb);
            else
                batch_frob_kernel<double2><<<g1, 256, 0, ctx.stream>>>(
                    static_cast<const double2*>(ws.bt.A) + d.a_off, d.n, d.lda, 0, ws.norm_part + (size_t)s * nb,
                    nb);
            BEM_CHECK_LAUNCH(&ctx);
        }
        finish_norms_kernel<<<(ws.bt.nsys + 127) / 128, 128, 0, ctx.stream>>>(ws.norm_part, nb, ws.bt.nsys,
                                                                               ws.anorm);
        BEM_CHECK_LAUNCH(&ctx);
        return;
    }
    dim3 grid(nb, ws.bt.nsys);
    if (ws.fp32)
        batch_frob_kernel<float2><<<grid, 256, 0, ctx.stream>>>(ws.bt.A, ws.bt.n, ws.bt.lda, ws.bt.mat_stride,
                                                                ws.norm_part, nb);
    else
        batch_frob_kernel<double2><<<grid, 256, 0, ctx.stream>>>(ws.bt.A, ws.bt.n, ws.bt.lda, ws.bt.mat_stride,
                                                                 ws.norm_part, nb);
    BEM_CHECK_LAUNCH(&ctx);
    finish_norms_kernel<<<(ws.bt.nsys + 127) / 128, 128, 0, ctx.stream>>>(ws.norm_part, nb, ws.bt.nsys, ws.anorm);
    BEM_CHECK_LAUNCH(&ctx);
}

void gm_init(Context& ctx, GmWorkspace& ws, double tol, int64_t max_restarts) {
    gm_init_kernel<<<ws.bt.nsys, AR_THREADS, 0, ctx.stream>>>(ws.bt, ws.anorm, tol, max_restarts, nullptr, nullptr,
                                                              nullptr);
    BEM_CHECK_LAUNCH(&ctx);
}

void gm_init_each(Context& ctx, GmWorkspace& ws, const std::vector<double>& tol,
                  const std::vector<int64_t>& max_restarts, const std::vector<int>& m) {
    const size_t ns = (size_t)ws.bt.nsys;
    require(tol.size() == ns && max_restarts.size() == ns && m.size() == ns, "gmres: per-system settings");
    for (int x : m) require(x >= 1 && x <= ws.bt.m, "gmres: restart length above the batch's");
    ws.init_args.ensure(ns * (sizeof(double) + sizeof(int64_t) + sizeof(int)));
    char* base = ws.init_args.as<char>();
    BEM_CUDA(cudaMemcpyAsync(base, tol.data(), ns * sizeof(double), cudaMemcpyHostToDevice, ctx.stream));
    BEM_CUDA(cudaMemcpyAsync(base + ns * 8, max_restarts.data(), ns * sizeof(int64_t), cudaMemcpyHostToDevice,
                             ctx.stream));
    BEM_CUDA(cudaMemcpyAsync(base + ns * 16, m.data(), ns * sizeof(int), cudaMemcpyHostToDevice, ctx.stream));
    gm_init_kernel<<<ws.bt.nsys, AR_THREADS, 0, ctx.stream>>>(
        ws.bt, ws.anorm, 0.0, 0, reinterpret_cast<const double*>(base), reinterpret_cast<const int64_t*>(base + ns * 8),
        reinterpret_cast<const int*>(base + ns * 16));
    BEM_CHECK_LAUNCH(&ctx);
    ctx.sync();  // the host arrays are pageable and owned by the caller
}

static void launch_apply(Context& ctx, GmWorkspace& ws, int mode) {
    if (ws.hook) {
        ws.hook(ctx, ws, mode, ws.hook_user);
        return;
    }
    const GmBatch& bt = ws.bt;
    // Finer tiles where they were the faster ones.  FP64: at every size (us per
    // product, wide -> finer: n = 2048 263 -> 39, 6144 312 -> 269, 16384 1820 ->
    // 1749; the wide tiles remain for caller-provided memory, which has no room for
    // the tickets).  FP32: below 1.5 wide tiles per SM (Krylov products, us of eight,
    // wide -> finer: 36 tiles 295 -> 92, 144 384 -> 373, 196 751 -> 568, 288 822 ->
    // 870, 1152 2447 -> 3069; beyond, memory bounds them and the longer columns of
    // the wide tiles read it better).  One choice for all products of a solve, so
    // that they sum in one order.
    const int64_t tiles = bt.sys ? bt.ntiles : (int64_t)ws.rb * ws.cb * bt.nsys;
    const bool small = bt.tpr == TICKETS && (!ws.fp32 || 2 * tiles < 3 * ws.sms);
    const dim3 grid = bt.sys ? dim3((unsigned)(small ? bt.ntiles64 : bt.ntiles))
                             : dim3((unsigned)(small ? (bt.n + SMALL_ROWS - 1) / SMALL_ROWS : ws.rb),
                                    (unsigned)ws.cb, (unsigned)bt.nsys);
#define BEM_APPLY(T, E, U)                                                                              \
    do {                                                                                                \
        if (small)                                                                                      \
            gm_apply_small_kernel<T, E, U>                                                              \
                <<<grid, 32 * SMALL_WARPS, small_smem<T, E, U>(), ctx.stream>>>(bt, mode);              \
        else                                                                                            \
            gm_apply_kernel<T, E, U><<<grid, MV_THREADS, 0, ctx.stream>>>(bt, mode);                    \
    } while (0)
    if (bt.split_lo) {
        BEM_APPLY(float2, 2, 4);
    } else if (ws.fp32) {
        if (mode == MV_Q) {
            // columns per load batch (loads in flight per thread), tuned per size
            const int u = ctx.tuning.pick("gm_apply_fp32", "unroll", bt.n, bt.nsys, MV_UNROLL);
            if (bt.mates && !small) {
                if (u == 4) gm_apply_kernel<float2, 0, 4, 2><<<grid, MV_THREADS, 0, ctx.stream>>>(bt, mode);
                else if (u == 16) gm_apply_kernel<float2, 0, 16, 2><<<grid, MV_THREADS, 0, ctx.stream>>>(bt, mode);
                else gm_apply_kernel<float2, 0, 8, 2><<<grid, MV_THREADS, 0, ctx.stream>>>(bt, mode);
                BEM_CHECK_LAUNCH(&ctx);
                return;
            }
            if (u == 4) BEM_APPLY(float2, 0, 4);
            else if (u == 16) BEM_APPLY(float2, 0, 16);
            else BEM_APPLY(float2, 0, 8);
        } else {
            BEM_APPLY(float2, 1, MV_UNROLL);
        }
    } else {
        BEM_APPLY(double2, 1, MV_UNROLL);
    }
#undef BEM_APPLY
    BEM_CHECK_LAUNCH(&ctx);
}

void gm_launch_start(Context& ctx, GmWorkspace& ws) {
    // outside the reference-faithful mode the residual of x = 0 is b itself
    if (ws.bt.ref_dotc) launch_apply(ctx, ws, MV_START);
    gm_start_kernel<<<ws.bt.nsys, AR_THREADS, 0, ctx.stream>>>(ws.bt);
    BEM_CHECK_LAUNCH(&ctx);
}

void gm_launch_iteration(Context& ctx, GmWorkspace& ws, cudaEvent_t ev_q0, cudaEvent_t ev_q1) {
    const int nsys = ws.bt.nsys;
    if (ws.precond) {
        if (ws.ev_p0) BEM_CUDA(cudaEventRecord(ws.ev_p0, ctx.stream));
        ws.precond(ctx, ws, MV_Q, ws.precond_user);
        if (ws.ev_p1) BEM_CUDA(cudaEventRecord(ws.ev_p1, ctx.stream));
    }
    if (ev_q0) BEM_CUDA(cudaEventRecord(ev_q0, ctx.stream));
    launch_apply(ctx, ws, MV_Q);
    if (ev_q1) BEM_CUDA(cudaEventRecord(ev_q1, ctx.stream));
    if (ws.bt.gs_part && !ws.bt.ref_dotc) {
        const dim3 grid((unsigned)ws.bt.gs_chunks, (unsigned)nsys);
        const size_t hsm = sizeof(double2) * (size_t)(ws.bt.m + 1);
        for (int pass = 0; pass < 2; ++pass) {
            gm_gs_dots_kernel<<<grid, GS_THREADS, 0, ctx.stream>>>(ws.bt);
            BEM_CHECK_LAUNCH(&ctx);
            gm_gs_update_kernel<<<grid, GS_THREADS, hsm, ctx.stream>>>(ws.bt, pass);
            BEM_CHECK_LAUNCH(&ctx);
        }
        const int chunks = (int)std::max<int64_t>(
            1, std::min<int64_t>((ws.bt.n + GV_STEP_THREADS - 1) / GV_STEP_THREADS, 2 * ws.sms / nsys));
        gm_givens_kernel<<<dim3((unsigned)chunks, (unsigned)nsys), GV_STEP_THREADS, gm_step_smem(ws.bt.m),
                           ctx.stream>>>(ws.bt, chunks);
    } else {
        // 128 rows per CTA while the cluster reaches
        int cs = 1;
        while (cs < ctx.gm_cluster && (int64_t)cs * MG_THREADS < ws.bt.n) cs *= 2;
        const size_t step = gm_step_smem(ws.bt.m), slice = sizeof(double2) * (size_t)((ws.bt.n + cs - 1) / cs);
        const bool in_smem = step + slice <= AR_SMEM_CAP;
        launch_cluster(ctx, gm_arnoldi_kernel, nsys * cs, cs, MG_THREADS, step + (in_smem ? slice : 0), ws.bt,
                       in_smem ? 1 : 0, cs);
    }
    BEM_CHECK_LAUNCH(&ctx);
    launch_apply(ctx, ws, MV_CHECK);
    gm_check_kernel<<<nsys, AR_THREADS, 0, ctx.stream>>>(ws.bt);
    BEM_CHECK_LAUNCH(&ctx);
}

void gm_read_states(Context& ctx, GmWorkspace& ws, std::vector<GmState>& out) {
    out.resize(ws.bt.nsys);
    BEM_CUDA(cudaMemcpyAsync(out.data(), ws.bt.st, sizeof(GmState) * ws.bt.nsys, cudaMemcpyDeviceToHost, ctx.stream));
    ctx.sync();
    gm_require_waits(out.data(), out.size());
}

// One iteration at a time; the Krylov mat-vec of every iteration is timed with
// events on the launching stream.
static void gm_run_profiled(Context& ctx, GmWorkspace& ws, int64_t max_total_iterations) {
    std::vector<GmState> st, prev;
    int64_t issued = 0;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    BEM_CUDA(cudaEventCreate(&e0));
    BEM_CUDA(cudaEventCreate(&e1));
    if (ws.precond) {
        BEM_CUDA(cudaEventCreate(&ws.ev_p0));
        BEM_CUDA(cudaEventCreate(&ws.ev_p1));
    }
    gm_read_states(ctx, ws, prev);
    gm_launch_start(ctx, ws);
    for (;;) {
        gm_launch_iteration(ctx, ws, e0, e1);
        ++issued;
        gm_read_states(ctx, ws, st);
        float ms = 0;
        BEM_CUDA(cudaEventElapsedTime(&ms, e0, e1));
        double entries = 0, mvs = 0;
        for (size_t s = 0; s < st.size(); ++s) {
            const double ns = ws.sys_host.empty() ? (double)ws.bt.n : (double)ws.sys_host[s].n;
            entries += (double)(st[s].iterations - prev[s].iterations) * ns * ns;
            mvs += (double)(st[s].iterations - prev[s].iterations);
        }
        if (entries > 0)
            ctx.stage_add(ws.mv_stage ? ws.mv_stage : (ws.fp32 ? "gmres_matvec_fp32" : "gmres_matvec_fp64"), ms,
                          1, ws.mv_bytes > 0 ? ws.mv_bytes * mvs : entries * (ws.fp32 ? 8.0 : 16.0));
        if (ws.ev_p0 && entries > 0) {
            float pms = 0;
            BEM_CUDA(cudaEventElapsedTime(&pms, ws.ev_p0, ws.ev_p1));
            ctx.stage_add("precond_apply", pms, 1, 0);
        }
        prev = st;
        bool all = true;
        for (auto& s : st) all = all && s.done;
        if (all || issued >= max_total_iterations) break;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (ws.ev_p0) cudaEventDestroy(ws.ev_p0);
    if (ws.ev_p1) cudaEventDestroy(ws.ev_p1);
    ws.ev_p0 = ws.ev_p1 = nullptr;
}

// After a round of iterations: its number and whether a system is still open, in
// one word of mapped host memory.
__global__ void gm_progress_kernel(const GmState* __restrict__ st, int nsys, int* __restrict__ round,
                                   volatile int* out) {
    int open = 0;
    for (int s = threadIdx.x; s < nsys; s += blockDim.x) open |= !st[s].done;
    open = __syncthreads_or(open);
    if (threadIdx.x == 0) {
        *out = 2 * ++*round + (open ? 1 : 0);
        __threadfence_system();
    }
}

// Run to completion, in rounds of `chunk` iterations that are launched one round
// ahead of the device; it reports every finished round to the host, and the round
// that follows the last one finds nothing to do.  (A state read after every
// iteration left the device idle for 16 us each: n = 6144 in FP64, 16 iterations,
// 9.6 ms, this way 9.3.)  Rounds of several iterations are one graph: the kernels
// of a small batch are shorter than their launches (whole call with four systems
// of n = 1280: 3.8 ms, launched one by one 4.5).  With profiling every iteration
// is followed by a state read.
void gm_run(Context& ctx, GmWorkspace& ws, int chunk, int64_t max_total_iterations) {
    if (ctx.profiling) {
        gm_run_profiled(ctx, ws, max_total_iterations);
        return;
    }
    constexpr int AHEAD = 2;  // rounds in flight
    if (!ctx.progress) {
        void* p = nullptr;
        BEM_CUDA(cudaHostAlloc(&p, sizeof(int), cudaHostAllocMapped));
        ctx.progress = static_cast<int*>(p);
    }
    int* dev = nullptr;
    BEM_CUDA(cudaHostGetDevicePointer(reinterpret_cast<void**>(&dev), ctx.progress, 0));
    volatile int* seen = ctx.progress;
    *seen = 1;  // round 0, open (nothing of an earlier run is in flight)
    ctx.w_rounds.ensure(sizeof(int));
    BEM_CUDA(cudaMemsetAsync(ctx.w_rounds.p, 0, sizeof(int), ctx.stream));
    gm_launch_start(ctx, ws);
    auto launch_round = [&] {
        for (int c = 0; c < chunk; ++c) gm_launch_iteration(ctx, ws, nullptr, nullptr);
        gm_progress_kernel<<<1, 128, 0, ctx.stream>>>(ws.bt.st, ws.bt.nsys, ctx.w_rounds.as<int>(), dev);
        BEM_CHECK_LAUNCH(&ctx);
    };
    struct Graph {
        cudaGraph_t g = nullptr;
        cudaGraphExec_t exec = nullptr;
        ~Graph() {
            if (exec) cudaGraphExecDestroy(exec);
            if (g) cudaGraphDestroy(g);
        }
    } graph;
    int64_t launches = 0;
    if (chunk > 1) {
        const int64_t before = ctx.launches;
        BEM_CUDA(cudaStreamBeginCapture(ctx.stream, cudaStreamCaptureModeThreadLocal));
        try {
            launch_round();
        } catch (...) {
            cudaStreamEndCapture(ctx.stream, &graph.g);  // leave the stream out of capture mode
            ctx.launches = before;
            throw;
        }
        BEM_CUDA(cudaStreamEndCapture(ctx.stream, &graph.g));
        launches = ctx.launches - before;
        ctx.launches = before;
        BEM_CUDA(cudaGraphInstantiate(&graph.exec, graph.g, 0));
    }
    int64_t issued = 0;
    for (int round = 1;; ++round) {
        if (graph.exec) {
            BEM_CUDA(cudaGraphLaunch(graph.exec, ctx.stream));
            ctx.launches += launches;
        } else {
            launch_round();
        }
        issued += chunk;
        int now = *seen;
        for (unsigned spin = 0; (now & 1) && round - (now >> 1) >= AHEAD; now = *seen)
            if ((++spin & 1023) == 0) {
                const cudaError_t e = cudaStreamQuery(ctx.stream);
                if (e == cudaErrorNotReady) cudaGetLastError();  // (not an error)
                else if (e == cudaSuccess) break;
                else BEM_CUDA(e);
            }
        now = *seen;
        if (!(now & 1) || issued >= max_total_iterations) break;
    }
    ctx.sync();
}

// gmres.rs:35-59 GMRES::solve over one dense FP64 matrix on the device.
GmresResult gmres_dense_fp64(Context& ctx, int64_t n, const double2* A, int64_t lda, int64_t max_it, double tol,
                             double2* x) {
    if (max_it <= 0) max_it = 1000;
    if (max_it > n) max_it = n;
    if (tol <= 0.0) tol = 1e-5;
    int m = (int)std::ceil(std::sqrt((double)max_it));
    int64_t restarts = max_it / m;
    GmWorkspace ws;
    ws.mem_pool = &ctx.w_gm;
    gm_prepare(ctx, ws, 1, n, m, A, lda, 0, false, true);
    BEM_CUDA(cudaMemcpyAsync(ws.bt.B, x, sizeof(double2) * n, cudaMemcpyDeviceToDevice, ctx.stream));
    gm_matrix_norms(ctx, ws);
    gm_init(ctx, ws, tol, restarts);
    gm_run(ctx, ws, 1, restarts * (int64_t)m + 1);
    std::vector<GmState> st;
    gm_read_states(ctx, ws, st);
    BEM_CUDA(cudaMemcpyAsync(x, ws.bt.X, sizeof(double2) * n, cudaMemcpyDeviceToDevice, ctx.stream));
    ctx.sync();
    GmresResult r;
    r.num_mv = st[0].num_mv;
    r.restarts = st[0].restarts + (st[0].converged ? 1 : 0);
    r.iterations = st[0].iterations;
    r.error = st[0].error;
    r.flag = st[0].converged ? 1 : 2;
    return r;
}

}  // namespace bem
