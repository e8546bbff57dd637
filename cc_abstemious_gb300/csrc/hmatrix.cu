// Hierarchical matrices (h_matrix.rs, aca.rs, cluster.rs, block.rs).
//
// Device: the geometric cluster tree and the block tree with its flattened
// leaf list (tree.cu), then every leaf block is filled in one batched pass -- inadmissible
// leaves as dense FP64 blocks, admissible leaves by adaptive cross
// approximation (one CTA per leaf running the reference's partially pivoted
// ACA with the rand 0.9 StdRng pivot stream restated below), followed by the
// QR + SVD recompression, also one CTA per leaf.  The mat-vec multiplies every
// leaf in parallel into a per-leaf output slice, then reduces each global row
// over its leaves in a fixed order (deterministic).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <functional>
#include <memory>

#include "common.cuh"
#include "complex.cuh"
#include "gmres.cuh"
#include "hmatrix.cuh"
#include "kernels.cuh"
#include "mixed.cuh"
#include "tree.cuh"

struct bem_hmatrix {
    bem::HMatrixDev* h;
    bem_ctx* ctx;
};

namespace bem {

// Leaf descriptor shared with the kernels.
struct HLeaf {
    int64_t row_off, m;   // into rows[]
    int64_t col_off, n;   // into cols[]
    int64_t store_off;    // dense: m*n entries; admissible: U (m*kmax) then V (n*kmax)
    int64_t scratch_off;  // ACA scratch: 2(m+n) complex + flags
    int64_t y_off;        // mat-vec output slice (m entries)
    int32_t adm, kmax;
    int32_t rank, pad;
    double norm;
};

struct HMatrixDev {
    int64_t n = 0;
    double norm = 0;
    std::vector<HLeaf> leaves;
    std::vector<int64_t> rows, cols;
    DevBuf d_leaves, d_rows, d_cols, d_store, d_scratch, d_y, d_rowptr, d_rowent, d_vec;
    DevBuf d_order;  // leaves by the work of their product, largest first
    int64_t nadm = 0, ninadm = 0, stored = 0, rank_sum = 0;
};

// ---------------------------------------------------------------------------
// Entry (i, j) of alpha H + beta G (influence_matrix.rs:170-230 restated per
// entry; column lists hold distinct indices so the diagonal appears once).
struct GenParams {
    KParams kp;
    z2 alpha, beta;
    int64_t npad;
    const double* geo;
};

__device__ __forceinline__ z2 gen_entry(const GenParams& g, int64_t i, int64_t j) {
    const double* geo = g.geo;
    const int64_t np = g.npad;
    z2 gg, hh;
    if (i == j) {
        self_term64(geo[GAREA * np + j], geo[GWT * np + j], g.kp.bm, g.kp.beta_im, g.kp.hdiag, g.kp.gdiag_im, gg, hh);
    } else {
        pair64_at(g.kp, np, geo, i, j, gg, hh);
    }
    z2 a = cmul(g.beta, gg);
    cfma(a, g.alpha, hh);
    return a;
}

// ---------------------------------------------------------------------------
// rand 0.9 StdRng (ChaCha12, rand_core seed_from_u64 via PCG32) and
// UniformUsize sampling of ranges below 2^32 -- the ACA pivot stream of
// aca.rs:64-68, evaluated by one thread.
struct DevRng {
    uint32_t key[8];
    uint64_t counter;
    uint32_t buf[16];
    int idx;
};

__device__ __forceinline__ uint32_t rotl32d(uint32_t v, int c) { return (v << c) | (v >> (32 - c)); }

__device__ void chacha12_block_dev(const uint32_t* key, uint64_t ctr, uint32_t* out) {
    uint32_t st[16] = {0x61707865u, 0x3320646eu, 0x79622d32u, 0x6b206574u, key[0], key[1], key[2], key[3],
                       key[4], key[5], key[6], key[7], (uint32_t)ctr, (uint32_t)(ctr >> 32), 0u, 0u};
    uint32_t s[16];
    for (int i = 0; i < 16; ++i) s[i] = st[i];
#define DQR(a, b, c, d)                                   \
    s[a] += s[b]; s[d] = rotl32d(s[d] ^ s[a], 16);        \
    s[c] += s[d]; s[b] = rotl32d(s[b] ^ s[c], 12);        \
    s[a] += s[b]; s[d] = rotl32d(s[d] ^ s[a], 8);         \
    s[c] += s[d]; s[b] = rotl32d(s[b] ^ s[c], 7);
    for (int r = 0; r < 6; ++r) {
        DQR(0, 4, 8, 12) DQR(1, 5, 9, 13) DQR(2, 6, 10, 14) DQR(3, 7, 11, 15)
        DQR(0, 5, 10, 15) DQR(1, 6, 11, 12) DQR(2, 7, 8, 13) DQR(3, 4, 9, 14)
    }
#undef DQR
    for (int i = 0; i < 16; ++i) out[i] = s[i] + st[i];
}

// Words are consumed in block order; the reference buffers four blocks at a
// time, which yields the same stream.
__device__ void rng_seed(DevRng& r, uint64_t state) {
    for (int i = 0; i < 8; ++i) {
        state = state * 6364136223846793005ull + 11634580027462260723ull;
        uint32_t xs = (uint32_t)(((state >> 18) ^ state) >> 27);
        uint32_t rot = (uint32_t)(state >> 59);
        r.key[i] = (xs >> rot) | (xs << ((32 - rot) & 31));
    }
    r.counter = 0;
    r.idx = 16;
}

__device__ uint32_t rng_u32(DevRng& r) {
    if (r.idx >= 16) {
        chacha12_block_dev(r.key, r.counter, r.buf);
        r.counter += 1;
        r.idx = 0;
    }
    return r.buf[r.idx++];
}

__device__ int64_t rng_uniform_incl(DevRng& r, uint32_t hi) {
    uint32_t range = hi + 1u;
    if (range == 0) return (int64_t)rng_u32(r);
    uint32_t thresh = (0u - range) % range;
    for (int guard = 0; guard < 1 << 20; ++guard) {
        uint64_t m = (uint64_t)rng_u32(r) * range;
        if ((uint32_t)m >= thresh) return (int64_t)(m >> 32);
    }
    return 0;
}

// ---------------------------------------------------------------------------
// Block-level reductions for the leaf kernels (blockDim multiple of 32, <= 1024).
__device__ __forceinline__ double bsum(double v, double* sh) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) sh[w] = v;
    __syncthreads();
    if (w == 0) {
        v = l < (int)(blockDim.x >> 5) ? sh[l] : 0.0;
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (l == 0) sh[40] = v;
    }
    __syncthreads();
    return sh[40];
}

// Sum of a complex value over the 32 lanes of a warp (every lane gets it).
// The parts part ways in the first step: five FP64 additions, not ten (each
// occupies the FP64 pipe of the SM quarter for 65 clocks).
__device__ __forceinline__ z2 wsum2(z2 v) {
    const bool odd = threadIdx.x & 1;
    double s = odd ? v.y : v.x;
    s += __shfl_xor_sync(0xffffffffu, odd ? v.x : v.y, 1);
    for (int o = 2; o <= 16; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return make_double2(__shfl_sync(0xffffffffu, s, 0), __shfl_sync(0xffffffffu, s, 1));
}
// Two complex values at once: six additions.
__device__ __forceinline__ void wsum4(z2& a, z2& b) {
    const bool odd = threadIdx.x & 1, up = threadIdx.x & 2;
    double x = odd ? a.y : a.x, y = odd ? b.y : b.x;
    x += __shfl_xor_sync(0xffffffffu, odd ? a.x : a.y, 1);
    y += __shfl_xor_sync(0xffffffffu, odd ? b.x : b.y, 1);
    double s = up ? y : x;
    s += __shfl_xor_sync(0xffffffffu, up ? x : y, 2);
    for (int o = 4; o <= 16; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    a = make_double2(__shfl_sync(0xffffffffu, s, 0), __shfl_sync(0xffffffffu, s, 1));
    b = make_double2(__shfl_sync(0xffffffffu, s, 2), __shfl_sync(0xffffffffu, s, 3));
}

__device__ __forceinline__ double wsum(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// argmax of |v[t]| over t not excluded; first index wins ties (aca.rs:256-268).
// Moduli (hypot, about 25 FP64 instructions) only of the entries whose square
// is within a few rounding errors of the largest square, which decides the
// others.  The winner's is returned beside its index.  Where every entry that is
// not excluded is a NaN, the first of them (modulus -1): the index addresses the
// leaf's rows and columns and is always one of them.
__device__ int64_t bargmax_excl(const double2* v, const int8_t* excl, int64_t len, double* sh, int64_t* shi,
                                double& modulus) {
    const long long inf = 0x7ff0000000000000ll;
    auto square = [&](int64_t t) {  // as the bits of a non-negative double; -1: NaN, -2: excluded
        if (excl[t]) return -2ll;
        const long long k = __double_as_longlong(cnorm2(v[t])) & 0x7fffffffffffffffll;
        return k > inf ? -1ll : k;
    };
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
    long long top = -2;
    for (int64_t t = threadIdx.x; t < len; t += blockDim.x) top = max(top, square(t));
    for (int o = 16; o > 0; o >>= 1) top = max(top, __shfl_xor_sync(0xffffffffu, top, o));
    __syncthreads();
    if (l == 0) shi[w] = top;
    __syncthreads();
    top = l < nw ? (long long)shi[l] : -2ll;
    for (int o = 16; o > 0; o >>= 1) top = max(top, __shfl_xor_sync(0xffffffffu, top, o));
    // 2^-47 below the largest (zero where squares underflow: every entry)
    const long long floor_ = top < 0 ? -1 : top < (64ll << 52) ? 0 : top == inf ? inf : top - 64;
    double best = -1.0;
    int64_t bi = len;
    for (int64_t t = threadIdx.x; t < len; t += blockDim.x) {
        const long long k = square(t);
        if (k < floor_) continue;
        const double a = k < 0 ? -1.0 : hypot(v[t].x, v[t].y);
        if (best < a || bi == len) { best = a; bi = t; }
    }
    for (int o = 16; o > 0; o >>= 1) {
        double ob = __shfl_down_sync(0xffffffffu, best, o);
        int64_t oi = __shfl_down_sync(0xffffffffu, bi, o);
        if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
    }
    __syncthreads();
    if (l == 0) { sh[w] = best; shi[w] = bi; }
    __syncthreads();
    if (w == 0) {
        best = l < nw ? sh[l] : -1.0;
        bi = l < nw ? shi[l] : len;
        for (int o = 16; o > 0; o >>= 1) {
            double ob = __shfl_down_sync(0xffffffffu, best, o);
            int64_t oi = __shfl_down_sync(0xffffffffu, bi, o);
            if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
        }
        if (l == 0) {
            shi[32] = bi;
            sh[41] = best;
        }
    }
    __syncthreads();
    modulus = sh[41];
    return shi[32];
}

constexpr int LEAF_THREADS = 256;
constexpr int ACA_RMAX = 256;  // largest rank of a compressed leaf
constexpr int JACOBI_SMEM = 32;  // ranks up to this run the Jacobi sweeps in shared memory

// Dense (inadmissible) leaves: one CTA per leaf, entries column-major m x n.
__global__ void __launch_bounds__(LEAF_THREADS) hm_dense_fill_kernel(const HLeaf* __restrict__ leaves,
                                                                     const int32_t* __restrict__ list,
                                                                     const int64_t* __restrict__ rows,
                                                                     const int64_t* __restrict__ cols, GenParams g,
                                                                     double2* __restrict__ store) {
    const HLeaf L = leaves[list[blockIdx.x]];
    double2* D = store + L.store_off;
    for (int64_t t = threadIdx.x; t < L.m * L.n; t += blockDim.x) {
        int64_t jj = t / L.m, ii = t - jj * L.m;
        D[t] = gen_entry(g, rows[L.row_off + ii], cols[L.col_off + jj]);
    }
}

// Residual row i (local) of the current approximation: A[i, :] - sum_k u_k[i] v_k.
__device__ void aca_res_row(const GenParams& g, const HLeaf& L, const int64_t* rows, const int64_t* cols,
                            const double2* U, const double2* V, int rank, int64_t i, double2* out) {
    const int64_t gi = rows[L.row_off + i];
    for (int64_t j = threadIdx.x; j < L.n; j += blockDim.x) {
        z2 a = gen_entry(g, gi, cols[L.col_off + j]);
        for (int k = 0; k < rank; ++k) cfma(a, cneg(U[(size_t)k * L.m + i]), V[(size_t)k * L.n + j]);
        out[j] = a;
    }
    __syncthreads();
}

__device__ void aca_res_col(const GenParams& g, const HLeaf& L, const int64_t* rows, const int64_t* cols,
                            const double2* U, const double2* V, int rank, int64_t j, double2* out) {
    const int64_t gj = cols[L.col_off + j];
    for (int64_t i = threadIdx.x; i < L.m; i += blockDim.x) {
        z2 a = gen_entry(g, rows[L.row_off + i], gj);
        for (int k = 0; k < rank; ++k) cfma(a, cneg(V[(size_t)k * L.n + j]), U[(size_t)k * L.m + i]);
        out[i] = a;
    }
    __syncthreads();
}

__device__ __forceinline__ double bnsq(const double2* a, int64_t len, double* sh) {
    double acc = 0;
    for (int64_t t = threadIdx.x; t < len; t += blockDim.x) acc += a[t].x * a[t].x + a[t].y * a[t].y;
    return bsum(acc, sh);
}

// The warp that does a leaf's single-warp work: a different one from CTA to CTA,
// since a warp's number decides the SM quarter whose FP64 pipe it uses.
__device__ __forceinline__ int lead_warp(int warps) {
    return (int)((blockIdx.x * 0x9E3779B1u) >> 20) & (warps - 1);
}

// Partially pivoted ACA (aca.rs:57-136) of every admissible leaf.
//
// FP64 instructions bound it, and in a small leaf those that are not entries:
// moduli, quotients and roots cost 600 to 1600 clocks of an SM quarter per warp
// however few lanes want them.  So they are gathered: the moduli of the norm
// estimate one lane per earlier rank, the pivot's quotient and the roots once per
// leaf, by one warp that differs from leaf to leaf.  (1534 leaves of n = 2560: 3.7
// ms with every warp doing them, 2.8 this way.)
constexpr int ACA_THREADS = 128;
__global__ void __launch_bounds__(ACA_THREADS, 4) hm_aca_kernel(HLeaf* __restrict__ leaves,
                                                              const int32_t* __restrict__ list,
                                                              const int64_t* __restrict__ rows,
                                                              const int64_t* __restrict__ cols, GenParams g,
                                                              double2* __restrict__ store, double2* __restrict__ scr,
                                                              double tol, int* __restrict__ err) {
    __shared__ double sh[48];
    __shared__ int64_t shi[33];
    __shared__ DevRng rng;
    __shared__ int64_t s_iref, s_jref;
    __shared__ double s_total;
    __shared__ int s_stop;
    __shared__ double2 s_f, s_du[ACA_RMAX], s_dv[ACA_RMAX];  // one per rank (kmax <= ACA_RMAX)
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = ACA_THREADS / 32, lead = lead_warp(nw);
    const double limit = tol / 50.0;
    HLeaf& L = leaves[list[blockIdx.x]];
    const int64_t m = L.m, n = L.n;
    const int64_t nr = m < n ? m : n;
    double2* U = store + L.store_off;
    double2* V = U + (size_t)m * L.kmax;
    double2* riref = scr + L.scratch_off;
    double2* rjref = riref + n;
    double2* ristar = rjref + m;
    double2* rjstar = ristar + n;
    int8_t* iex = reinterpret_cast<int8_t*>(rjstar + m);
    int8_t* jex = iex + m;
    for (int64_t t = threadIdx.x; t < m; t += blockDim.x) iex[t] = 0;
    for (int64_t t = threadIdx.x; t < n; t += blockDim.x) jex[t] = 0;
    if (threadIdx.x == 0) {
        rng_seed(rng, 10);
        s_iref = rng_uniform_incl(rng, (uint32_t)(nr - 1));
        s_jref = rng_uniform_incl(rng, (uint32_t)(nr - 1));
        s_total = 0;
        s_stop = 0;
    }
    __syncthreads();
    aca_res_row(g, L, rows, cols, U, V, 0, s_iref, riref);
    aca_res_col(g, L, rows, cols, U, V, 0, s_jref, rjref);
    int rank = 0;
    for (int64_t k = 0; k < nr; ++k) {
        if (k >= L.kmax) {  // rank cap of the storage reached before the stopping test
            if (threadIdx.x == 0) atomicOr(err, 8);
            break;
        }
        // (read here, barriers ahead of the updates below: a warp that read them
        // there could find thread 0's new ones, take the other branch and part
        // ways with the rest of the CTA)
        const int64_t iref = s_iref, jref = s_jref;
        double jval, ival, unused;
        int64_t jstar = bargmax_excl(riref, jex, n, sh, shi, jval);
        int64_t istar = bargmax_excl(rjref, iex, m, sh, shi, ival);
        if (ival > jval) {
            aca_res_row(g, L, rows, cols, U, V, rank, istar, ristar);
            jstar = bargmax_excl(ristar, jex, n, sh, shi, unused);
            aca_res_col(g, L, rows, cols, U, V, rank, jstar, rjstar);
        } else {
            aca_res_col(g, L, rows, cols, U, V, rank, jstar, rjstar);
            istar = bargmax_excl(rjstar, iex, m, sh, shi, unused);
            aca_res_row(g, L, rows, cols, U, V, rank, istar, ristar);
        }
        if (warp == lead) {  // 1 / pivot, a part per lane
            const z2 piv = ristar[jstar];
            const double den = piv.x * piv.x + piv.y * piv.y, part = (lane ? -piv.y : piv.x) / den;
            if (lane < 2) reinterpret_cast<double*>(&s_f)[lane] = part;
            if (lane == 0) {
                iex[istar] = 1;
                jex[jstar] = 1;
            }
        }
        __syncthreads();
        const z2 f = s_f;
        double2* uk = U + (size_t)k * m;
        double2* vk = V + (size_t)k * n;
        for (int64_t t = threadIdx.x; t < n; t += blockDim.x) vk[t] = cmul(ristar[t], f);
        for (int64_t t = threadIdx.x; t < m; t += blockDim.x) uk[t] = rjstar[t];
        __syncthreads();
        rank = (int)k + 1;
        // update_norm_estimate (aca.rs:224-241): the products with every
        // earlier rank and the new rank's norms one warp each, the moduli one lane
        // each, summed in rank order
        for (int t = warp; t <= k; t += nw) {
            const double2* ut = U + (size_t)t * m;
            const double2* vt = V + (size_t)t * n;
            z2 du = make_double2(0, 0), dv = make_double2(0, 0);
            if (t < k) {
                for (int64_t i = lane; i < m; i += 32) cfma(du, ut[i], uk[i]);
                for (int64_t j = lane; j < n; j += 32) cfma(dv, vt[j], vk[j]);
            } else {
                for (int64_t i = lane; i < m; i += 32) du.x = fma(uk[i].x, uk[i].x, fma(uk[i].y, uk[i].y, du.x));
                for (int64_t j = lane; j < n; j += 32) dv.x = fma(vk[j].x, vk[j].x, fma(vk[j].y, vk[j].y, dv.x));
            }
            wsum4(du, dv);
            if (lane == 0) {
                s_du[t] = du;
                s_dv[t] = dv;
            }
        }
        __syncthreads();
        if (warp == lead) {
            for (int t = lane; t < k; t += 32)
                s_du[t].x = 2.0 * hypot(s_du[t].x, s_du[t].y) * hypot(s_dv[t].x, s_dv[t].y);
            __syncwarp();
            const double nk = s_du[k].x * s_dv[k].x;
            double add = 0;
            for (int t = 0; t < k; ++t) add += s_du[t].x;
            const double total = s_total + nk + add;
            __syncwarp();
            const double root = sqrt(lane ? total : nk);
            const double step = __shfl_sync(0xffffffffu, root, 0) / __shfl_sync(0xffffffffu, root, 1);
            if (lane == 0) {
                s_total = total;
                s_stop = step < limit;
                }
        }
        __syncthreads();
        if (s_stop) break;
        // reference row / column updates
        if (iref == istar) {
            if (threadIdx.x == 0) {
                int64_t v = iref;
                if (iex[v]) {
                    v = rng_uniform_incl(rng, (uint32_t)(nr - 1));
                    for (int64_t t = 0; t < nr - 1; ++t) {
                        v = (v + 1) % nr;
                        if (!iex[v]) break;
                    }
                }
                s_iref = v;
            }
            __syncthreads();
            aca_res_row(g, L, rows, cols, U, V, rank, s_iref, riref);
        } else {
            const z2 c = uk[iref];
            for (int64_t t = threadIdx.x; t < n; t += blockDim.x) cfma(riref[t], cneg(c), vk[t]);
            __syncthreads();
        }
        if (jref == jstar) {
            if (threadIdx.x == 0) {
                int64_t v = jref;
                if (jex[v]) {
                    v = rng_uniform_incl(rng, (uint32_t)(nr - 1));
                    for (int64_t t = 0; t < nr - 1; ++t) {
                        v = (v + 1) % nr;
                        if (!jex[v]) break;
                    }
                }
                s_jref = v;
            }
            __syncthreads();
            aca_res_col(g, L, rows, cols, U, V, rank, s_jref, rjref);
        } else {
            const z2 c = vk[jref];
            for (int64_t t = threadIdx.x; t < m; t += blockDim.x) cfma(rjref[t], cneg(c), uk[t]);
            __syncthreads();
        }
    }
    if (threadIdx.x == 0) {
        L.rank = rank;
        L.norm = sqrt(s_total);
    }
}

// ---------------------------------------------------------------------------
// QR + SVD recompression (aca.rs:137-179) and the ab-initio norm estimate
// (aca.rs:212-222).  Householder QR of U (m x r) and V (n x r) in place (the
// reflectors overwrite the factor, R goes to scratch), SVD of R_u R_v^T by
// one-sided Jacobi, truncation at s < tol * cumulative sum (+1, at least 1),
// then U <- Q_u W Sigma and V <- Q_v Z with Z = (V^H)^T (plain transpose, the
// factors pair as u v^T).
//
// A leaf's CTA has four warps, one per SM quarter; both factors are reduced in the
// same loop, so that the serial part of a reflector (a root and a quotient, lanes
// side by side) is paid once for the two.
constexpr int RC_THREADS = 128, RC_WARPS = RC_THREADS / 32;

// x -= tau v (v^H x) for two columns at once (q may be missing), rows k .. m of a
// warp: one pass over v, and the two sums share their additions.
__device__ __forceinline__ void reflect_two(const double2* __restrict__ v, double2* __restrict__ p,
                                            double2* __restrict__ q, int64_t k, int64_t m, double tau, int lane) {
    z2 d = make_double2(0, 0), e = d;
    if (q) {
#pragma unroll 2
        for (int64_t i = k + lane; i < m; i += 32) {
            const z2 a = cconj(v[i]);
            cfma(d, a, p[i]);
            cfma(e, a, q[i]);
        }
        wsum4(d, e);
        d = cscale(d, -tau);
        e = cscale(e, -tau);
#pragma unroll 2
        for (int64_t i = k + lane; i < m; i += 32) {
            const z2 a = v[i];
            z2 x = p[i], y = q[i];
            cfma(x, a, d);
            cfma(y, a, e);
            p[i] = x;
            q[i] = y;
        }
    } else {
        for (int64_t i = k + lane; i < m; i += 32) cfma(d, cconj(v[i]), p[i]);
        d = cscale(wsum2(d), -tau);
        for (int64_t i = k + lane; i < m; i += 32) cfma(p[i], v[i], d);
    }
}

__device__ void house_qr_dev(double2* A0, int64_t m0, double2* R0, double2* tau0, double2* A1, int64_t m1, double2* R1,
                             double2* tau1, int r, int lead) {
    // A: m x r column-major; on exit the reflectors v_k = x - alpha e_k are
    // kept in A below and on the diagonal.  One warp per factor forms column k's
    // reflector (|v_k|^2 = 2 |x| (|x| + |x_0|), no second reduction), every warp
    // applies them to its share of the later columns: two barriers per k.
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, mine = (warp - lead) & (RC_WARPS - 1);
    __shared__ double s_tau[2];
    for (int k = 0; k < r; ++k) {
        if (mine < 2) {
            double2* a = (mine ? A1 : A0) + (size_t)k * (mine ? m1 : m0);
            const int64_t m = mine ? m1 : m0;
            const z2 x0 = a[k];
            double nx2 = 0;
            for (int64_t i = k + lane; i < m; i += 32) nx2 = fma(a[i].x, a[i].x, fma(a[i].y, a[i].y, nx2));
            nx2 = wsum(nx2);
            const double root = sqrt(lane ? cnorm2(x0) : nx2);
            const double nx = __shfl_sync(0xffffffffu, root, 0), ax0 = __shfl_sync(0xffffffffu, root, 1);
            const double half = nx * (nx + ax0);
            const double part = (lane == 0 ? x0.x : lane == 1 ? x0.y : 1.0) / (lane < 2 ? ax0 : half);
            z2 ph = make_double2(__shfl_sync(0xffffffffu, part, 0), __shfl_sync(0xffffffffu, part, 1));
            double tk = __shfl_sync(0xffffffffu, part, 2);
            if (ax0 == 0) ph = make_double2(1.0, 0.0);
            if (half == 0) tk = 0.0;
            const z2 alpha = make_double2(-ph.x * nx, -ph.y * nx);
            __syncwarp();
            if (lane == 0) {
                a[k] = csub(x0, alpha);
                (mine ? R1 : R0)[(size_t)k * r + k] = alpha;
                (mine ? tau1 : tau0)[k] = make_double2(tk, 0.0);
                s_tau[mine] = tk;
            }
        }
        __syncthreads();
        const int later = r - k - 1, pairs = (later + 1) / 2;
        for (int t = warp; t < 2 * pairs; t += RC_WARPS) {
            const bool second = t >= pairs;
            const int64_t m = second ? m1 : m0;
            const int j = k + 1 + 2 * (second ? t - pairs : t);
            double2* A = second ? A1 : A0;
            reflect_two(A + (size_t)k * m, A + (size_t)j * m, j + 1 < r ? A + (size_t)(j + 1) * m : nullptr, k, m,
                        s_tau[second], lane);
        }
        __syncthreads();
    }
    // R above the diagonal lives in rows < k of columns k
    for (int t = threadIdx.x; t < r * r; t += RC_THREADS) {
        const int i = t % r, j = t / r;
        if (i == j) continue;
        R0[t] = i < j ? A0[(size_t)j * m0 + i] : make_double2(0, 0);
        R1[t] = i < j ? A1[(size_t)j * m1 + i] : make_double2(0, 0);
    }
    __syncthreads();
}

// out (m x c) = Q [B; 0] where Q = H_0 ... H_{r-1} (reflectors in A), B r x c,
// for both factors.  A warp carries its columns through all reflectors; the
// columns do not meet.
__device__ void house_apply_dev(const double2* A0, int64_t m0, const double2* tau0, const double2* B0, double2* out0,
                                const double2* A1, int64_t m1, const double2* tau1, const double2* B1, double2* out1,
                                int r, int c) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, pairs = (c + 1) / 2;
    for (int t = warp; t < 2 * pairs; t += RC_WARPS) {
        const bool second = t >= pairs;
        const int j = 2 * (second ? t - pairs : t);
        const int64_t m = second ? m1 : m0;
        const double2 *A = second ? A1 : A0, *tau = second ? tau1 : tau0, *b = (second ? B1 : B0) + (size_t)j * r;
        double2 *o = (second ? out1 : out0) + (size_t)j * m, *p = j + 1 < c ? o + m : nullptr;
        for (int64_t i = lane; i < m; i += 32) {
            o[i] = i < r ? b[i] : make_double2(0, 0);
            if (p) p[i] = i < r ? b[r + i] : make_double2(0, 0);
        }
        __syncwarp();
        for (int k = r - 1; k >= 0; --k) {
            const double tk = tau[k].x;
            if (tk == 0.0) continue;
            reflect_two(A + (size_t)k * m, o, p, k, m, tk, lane);
            __syncwarp();
        }
    }
    __syncthreads();
}

// One-sided Jacobi on the columns of the r x r matrix M (overwritten by W Sigma):
// each sweep visits every column pair once in the round-robin order, r' - 1
// steps (r' = r rounded up to even) of r' / 2 disjoint pairs, until a sweep
// finds no pair further than 1e-15 from orthogonal.
//
// Bound by FP64 issue (65 clocks per warp instruction however few lanes are
// active), so a pair takes only as many lanes as fill the warps (18 columns:
// one warp, three lanes per pair; more warps only for the largest ranks, which
// would be the last to finish) and the rotation's angle comes from FP32: it
// only has to be near, the next sweep corrects it; what is kept to FP64 is that
// the rotation is unitary (its cosine and the phase, each one FP32 seed and a
// third-order correction).  The columns' norms follow the rotations and are
// summed anew in every sweep.  The right factor is not accumulated; the caller
// forms it from W Sigma and the original matrix.  2560 triangles, leaf 32, eta 4,
// 1534 leaves with ranks up to 38: the whole recompression 24.7 -> 3.8 ms.
// 1 / sqrt(v) for 0 < v (normal numbers).
__device__ __forceinline__ double near_rsqrt(double v) {
    const int e = (((__double2hiint(v) >> 20) & 0x7ff) - 1023) & ~1;  // even
    const double s = wide(rsqrtf(near_float(v, e))) * __hiloint2double((1023 - e / 2) << 20, 0);
    const double c = fma(-(v * s), s, 1.0);
    return fma(s * c, fma(0.375, c, 0.5), s);
}

__device__ void jacobi_dev(double2* M, int r, double* S, int* perm, int lead) {
    const int lane = threadIdx.x & 31, nw = RC_WARPS, warp = ((threadIdx.x >> 5) - lead) & (nw - 1);
    const int rr = r + (r & 1), pairs = rr / 2;  // players of the round robin (index r: a bye when r is odd)
    const int warps = r <= 24 ? 1 : r <= 32 ? 2 : 4;
    int lpp = 32;  // lanes per pair, any number: groups do not reach over warps
    while (lpp > 1 && 32 / lpp * warps < pairs) --lpp;
    __shared__ int s_turned;
    __shared__ double s_n[ACA_RMAX];  // squared norms of the columns
    if (warp < warps) {
        auto together = [&]() {
            // (a warp whose pairs have not all turned comes here in parts; the
            // barrier wants it whole)
            __syncwarp();
            if (warps > 1) asm volatile("bar.sync 1, %0;" ::"r"(32 * warps) : "memory");
        };
        const int per = 32 / lpp, groups = per * warps, first = lane / lpp * lpp;
        const int grp = lane < per * lpp ? warp * per + lane / lpp : 1 << 20, g = lane - first;
        // sum over a group's lanes, in one order in all of them
        auto group_sum = [&](double v) {
            double t = __shfl_sync(0xffffffffu, v, first);
            for (int o = 1; o < lpp; ++o) t += __shfl_sync(0xffffffffu, v, (first + o) & 31);
            return t;
        };
        for (int sweep = 0; sweep < 60 && r > 1; ++sweep) {
            together();
            if (warp == 0 && lane == 0) s_turned = 0;
            for (int c0 = 0; c0 < r; c0 += groups) {
                const int c = c0 + grp;
                double a = 0;
                if (c < r)
                    for (int i = g; i < r; i += lpp) {
                        const z2 x = M[(size_t)c * r + i];
                        a = fma(x.x, x.x, fma(x.y, x.y, a));
                    }
                a = group_sum(a);
                if (c < r && g == 0) s_n[c] = a;
            }
            together();
            for (int step = 0; step < rr - 1; ++step) {
                for (int p0 = 0; p0 < pairs; p0 += groups) {
                    // circle method: player 0 fixed, the others rotate by `step`
                    const int pi = p0 + grp;
                    const int a0 = pi == 0 ? 0 : 1 + (pi - 1 + step) % (rr - 1);
                    const int b0 = 1 + (rr - 2 - pi + step) % (rr - 1);
                    const int p = min(a0, b0), q = max(a0, b0);
                    const bool on = pi < pairs && q < r;  // (q = r: the bye)
                    double2* up = M + (size_t)p * r;
                    double2* uq = M + (size_t)q * r;
                    const double a = on ? s_n[p] : 0.0, b = on ? s_n[q] : 0.0;
                    z2 cc = make_double2(0, 0);
                    if (on)
                        for (int i = g; i < r; i += lpp) cfma(cc, cconj(up[i]), uq[i]);
                    cc = make_double2(group_sum(cc.x), group_sum(cc.y));
                    const double n2 = cnorm2(cc);
                    const bool turn = on && n2 > 1e-290 && n2 > 1e-30 * (a * b);
                    if (!__any_sync(0xffffffffu, turn)) continue;
                    if (lane == 0) s_turned = 1;
                    if (!turn) continue;
                    // tan of the angle from FP32, everything relative to max(a, b)
                    const int e = ((__double2hiint(fmax(a, b)) >> 20) & 0x7ff) - 1023;
                    const double ri = near_rsqrt(n2), mod = n2 * ri;
                    const float d = near_float(b, e) - near_float(a, e), f = 2.0f * near_float(mod, e);
                    const double t = (double)copysignf(__fdividef(f, fmaxf(fabsf(d) + sqrtf(fmaf(d, d, f * f)), 1e-37f)), d);
                    const double cs = near_rsqrt(fma(t, t, 1.0)), sn = cs * t;
                    const z2 se = cscale(cc, ri * sn);
                    if (g == 0) {  // the norms after this rotation, whatever its angle
                        const double t2 = t * t, c2 = cs * cs, tm = 2.0 * t * mod;
                        s_n[p] = fmax(fma(t2, b, a - tm) * c2, 0.0);
                        s_n[q] = fmax(fma(t2, a, b + tm) * c2, 0.0);
                    }
                    for (int i = g; i < r; i += lpp) {
                        const z2 x = up[i], y = uq[i];
                        up[i] = make_double2(fma(cs, x.x, -fma(se.x, y.x, se.y * y.y)),
                                             fma(cs, x.y, -fma(se.x, y.y, -se.y * y.x)));
                        uq[i] = make_double2(fma(cs, y.x, fma(se.x, x.x, -se.y * x.y)),
                                             fma(cs, y.y, fma(se.x, x.y, se.y * x.x)));
                    }
                }
                together();
            }
            if (*(volatile int*)&s_turned == 0) break;
        }
    }
    __syncthreads();
    // singular values and their descending order
    for (int j = warp; j < r; j += nw) {
        double v = 0;
        for (int i = lane; i < r; i += 32) v += cnorm2(M[(size_t)j * r + i]);
        v = wsum(v);
        if (lane == 0) S[j] = sqrt(v);
    }
    __syncthreads();
    for (int j = threadIdx.x; j < r; j += blockDim.x) perm[descending_rank(S, r, j)] = j;
    __syncthreads();
}

__global__ void __launch_bounds__(RC_THREADS, 5) hm_recompress_kernel(HLeaf* __restrict__ leaves,
                                                                     const int32_t* __restrict__ list,
                                                                     double2* __restrict__ store,
                                                                     double2* __restrict__ scr,
                                                                     const int64_t* __restrict__ scr2_off,
                                                                     double tol) {
    __shared__ double2 sM[JACOBI_SMEM * JACOBI_SMEM];
    HLeaf& L = leaves[list[blockIdx.x]];
    const int r = L.rank;
    const int64_t m = L.m, n = L.n;
    double2* U = store + L.store_off;
    double2* V = U + (size_t)m * L.kmax;
    double2* w = scr + scr2_off[blockIdx.x];
    double2* Ru = w;
    double2* Rv = Ru + (size_t)r * r;
    double2* RR = Rv + (size_t)r * r;
    double2* M = RR + (size_t)r * r;
    double2* B = M + (size_t)r * r;
    if (r <= JACOBI_SMEM) M = sM;
    double2* tauu = B + (size_t)r * r;
    double2* tauv = tauu + r;
    double2* outU = tauv + r;             // m x r
    double2* outV = outU + (size_t)m * r; // n x r
    double* S = reinterpret_cast<double*>(outV + (size_t)n * r);
    int* perm = reinterpret_cast<int*>(S + r);
    const int lead = lead_warp(RC_WARPS);
    house_qr_dev(U, m, Ru, tauu, V, n, Rv, tauv, r, lead);
    // RR = R_u R_v^T
    for (int t = threadIdx.x; t < r * r; t += blockDim.x) {
        int i = t % r, j = t / r;
        z2 acc = make_double2(0, 0);
        for (int l = 0; l < r; ++l) cfma(acc, Ru[(size_t)l * r + i], Rv[(size_t)l * r + j]);
        RR[(size_t)j * r + i] = acc;
        M[(size_t)j * r + i] = acc;
    }
    __syncthreads();
    jacobi_dev(M, r, S, perm, lead);
    // truncation (aca.rs:162-171)
    __shared__ int s_keep;
    if (threadIdx.x == 0) {
        int index = 0;
        double sum = 0;
        for (int t = 0; t < r; ++t) {
            double sv = S[perm[t]];
            sum += sv;
            if (sv < tol * sum) break;
            index++;
        }
        index = index + 1 < r ? index + 1 : r;
        if (index < 1) index = 1;
        s_keep = index;
    }
    __syncthreads();
    const int keep = s_keep;
    // U_new = Q_u (W Sigma)
    for (int t = 0; t < keep; ++t)
        for (int i = threadIdx.x; i < r; i += blockDim.x) B[(size_t)t * r + i] = M[(size_t)perm[t] * r + i];
    // V_new = Q_v Z with Z the transpose of Sigma^-1 W^H (R_u R_v^T) =
    // Sigma^-2 (W Sigma)^H (R_u R_v^T)
    for (int t = threadIdx.x; t < keep * r; t += blockDim.x) {
        const int c = t / r, i = t % r;
        const double2* wt = M + (size_t)perm[c] * r;
        const double sv = S[perm[c]], s2 = sv > 0 ? 1.0 / (sv * sv) : 0.0;
        z2 acc = make_double2(0, 0);
        for (int l = 0; l < r; ++l) cfma(acc, cconj(wt[l]), RR[(size_t)i * r + l]);
        Rv[t] = cscale(acc, s2);  // (R_v is done with)
    }
    __syncthreads();
    house_apply_dev(U, m, tauu, B, outU, V, n, tauv, Rv, outV, r, keep);
    for (int t = 0; t < keep; ++t) {
        for (int64_t i = threadIdx.x; i < m; i += blockDim.x) U[(size_t)t * m + i] = outU[(size_t)t * m + i];
        for (int64_t i = threadIdx.x; i < n; i += blockDim.x) V[(size_t)t * n + i] = outV[(size_t)t * n + i];
    }
    __syncthreads();
    // calculate_norm_estimate (aca.rs:212-222): |u_a|^2 |v_a|^2 and twice the
    // products of every pair of ranks, one warp per pair
    __shared__ double s_tot[RC_WARPS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    double sum = 0;
    for (int t = warp; t < keep * (keep + 1) / 2; t += nw) {
        int a = (int)((sqrtf(8.0f * (float)t + 1.0f) - 1.0f) * 0.5f);
        while (a * (a + 1) / 2 > t) --a;
        while ((a + 1) * (a + 2) / 2 <= t) ++a;
        const int b = t - a * (a + 1) / 2;
        z2 du = make_double2(0, 0), dv = make_double2(0, 0);
        if (a == b) {
            for (int64_t i = lane; i < m; i += 32) du.x += cnorm2(U[(size_t)a * m + i]);
            for (int64_t j = lane; j < n; j += 32) dv.x += cnorm2(V[(size_t)a * n + j]);
        } else {
            for (int64_t i = lane; i < m; i += 32) cfma(du, U[(size_t)a * m + i], U[(size_t)b * m + i]);
            for (int64_t j = lane; j < n; j += 32) cfma(dv, V[(size_t)a * n + j], V[(size_t)b * n + j]);
        }
        wsum4(du, dv);
        sum += a == b ? du.x * dv.x : 2.0 * sqrt(cnorm2(du) * cnorm2(dv));
    }
    if (lane == 0) s_tot[warp] = sum;
    __syncthreads();
    double tot = 0;
    if (threadIdx.x == 0)
        for (int i = 0; i < nw; ++i) tot += s_tot[i];
    if (threadIdx.x == 0) {
        L.rank = keep;
        L.norm = sqrt(tot);
    }
}

// Frobenius norm of dense leaves.
__global__ void hm_dense_norm_kernel(HLeaf* __restrict__ leaves, const int32_t* __restrict__ list,
                                     const double2* __restrict__ store) {
    __shared__ double sh[48];
    HLeaf& L = leaves[list[blockIdx.x]];
    double v = bnsq(store + L.store_off, L.m * L.n, sh);
    if (threadIdx.x == 0) L.norm = sqrt(v);
}

// ---------------------------------------------------------------------------
// Mat-vec: every leaf multiplies its gathered slice of x (alpha applied), the
// row reduction adds the slices of each global row in leaf order.
//
// FP64 instructions bound it (65 clocks per warp and SM quarter), so the four
// warps of a leaf's CTA, one per quarter, get equal shares: of the column range
// in V^T x (eight lanes per rank, so that a sum costs four additions for four
// ranks), of the rows or, in a leaf of few rows, of the columns in U t and D x.
// The leaves are taken heaviest first.  (A block-wide reduction per rank and
// threads without a row: 735 us at n = 10240 with 27 M stored entries, whose
// products alone take 173 us; now 276 us.)
constexpr int HMV_THREADS = 128, HMV_WARPS = HMV_THREADS / 32, HMV_CHUNK = 512;

// out[i] (+)= sum over k < nc of M[k m + i] c[k], M column-major in device
// memory, c and `part` (HMV_THREADS entries) in shared memory; the whole CTA.
__device__ __forceinline__ void leaf_columns(const double2* __restrict__ M, int64_t m, int nc, const double2* c,
                                             double2* part, bool add, z2 alpha, double2* __restrict__ out) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int groups = m <= 32 ? HMV_WARPS : m <= 64 ? HMV_WARPS / 2 : 1;  // warps sharing a row
    const int tiles = HMV_WARPS / groups, kg = warp / tiles;
    const int per = (nc + groups - 1) / groups, ka = min(nc, kg * per), kb = min(nc, ka + per);
    for (int64_t i0 = 0; i0 < m; i0 += 32 * tiles) {
        const int64_t i = i0 + 32 * (warp % tiles) + lane;
        z2 acc = make_double2(0, 0);
        if (i < m) {
            const double2* col = M + i;
            int k = ka;
            for (; k + 8 <= kb; k += 8) {
                double2 v[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) v[u] = __ldcs(col + (size_t)(k + u) * m);
#pragma unroll
                for (int u = 0; u < 8; ++u) cfma(acc, v[u], c[k + u]);
            }
            for (; k < kb; ++k) cfma(acc, __ldcs(col + (size_t)k * m), c[k]);
        }
        if (groups > 1) {
            part[threadIdx.x] = acc;
            __syncthreads();
            if (kg == 0)
                for (int q = 1; q < groups; ++q) acc = cadd(acc, part[threadIdx.x + 32 * tiles * q]);
        }
        if (i < m && kg == 0) {
            acc = cmul(alpha, acc);
            out[i] = add ? cadd(out[i], acc) : acc;
        }
    }
}

__global__ void __launch_bounds__(HMV_THREADS) hm_leaf_mv_kernel(const HLeaf* __restrict__ leaves,
                                                                 const int32_t* __restrict__ order,
                                                                 const int64_t* __restrict__ cols,
                                                                 const double2* __restrict__ store, GmBatch bt,
                                                                 int mode, const double2* __restrict__ xin, z2 alpha,
                                                                 double2* __restrict__ y) {
    __shared__ double2 xs[HMV_CHUNK], part[HMV_THREADS];
    __shared__ double2 tw[HMV_WARPS][64], tk[64];
    const double2* x = xin;
    if (bt.st) {
        const GmState& st = bt.st[0];
        if (!gm_apply_active(st, mode)) return;
        x = (mode == MV_Q) ? bt.Q + (size_t)st.k * bt.n : bt.X;
    }
    const HLeaf L = leaves[order[blockIdx.x]];
    const double2* D = store + L.store_off;
    double2* yo = y + L.y_off;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const z2 one = make_double2(1, 0);
    if (!L.adm) {
        for (int64_t j0 = 0; j0 < L.n; j0 += HMV_CHUNK) {
            const int jn = (int)min((int64_t)HMV_CHUNK, L.n - j0);
            if (j0) __syncthreads();
            for (int j = tid; j < jn; j += HMV_THREADS) xs[j] = x[cols[L.col_off + j0 + j]];
            __syncthreads();
            leaf_columns(D + (size_t)j0 * L.m, L.m, jn, xs, part, j0 > 0, alpha, yo);
        }
        return;
    }
    const double2* U = D;
    const double2* V = U + (size_t)L.m * L.kmax;
    if (L.rank == 0)
        for (int64_t i = tid; i < L.m; i += HMV_THREADS) yo[i] = make_double2(0, 0);
    const int l8 = lane & 7;
    for (int k0 = 0; k0 < L.rank; k0 += 64) {
        const int kc = min(64, L.rank - k0);
        for (int k = tid; k < HMV_WARPS * 64; k += HMV_THREADS) (&tw[0][0])[k] = make_double2(0, 0);
        for (int64_t j0 = 0; j0 < L.n; j0 += HMV_CHUNK) {
            const int jn = (int)min((int64_t)HMV_CHUNK, L.n - j0);
            __syncthreads();
            for (int j = tid; j < jn; j += HMV_THREADS) xs[j] = x[cols[L.col_off + j0 + j]];
            __syncthreads();
            // this warp's columns, a multiple of eight
            const int per = ((jn + 8 * HMV_WARPS - 1) / (8 * HMV_WARPS)) * 8;
            const int ja = min(jn, warp * per), jb = min(jn, ja + per);
            for (int k = 0; k < kc; k += 4) {
                const int kk = k + (lane >> 3);
                const double2* vk = V + (size_t)(k0 + min(kk, kc - 1)) * L.n + j0;
                z2 acc = make_double2(0, 0);
                int j = ja + l8;
                for (; j + 24 < jb; j += 32) {
                    double2 v[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) v[u] = __ldcs(vk + j + 8 * u);
#pragma unroll
                    for (int u = 0; u < 4; ++u) cfma(acc, v[u], xs[j + 8 * u]);
                }
                for (; j < jb; j += 8) cfma(acc, __ldcs(vk + j), xs[j]);
                const double sum = sum8_parts(acc);
                if (l8 < 2 && kk < kc) reinterpret_cast<double*>(&tw[warp][kk])[l8] += sum;
            }
        }
        __syncthreads();
        for (int k = tid; k < kc; k += HMV_THREADS)  // alpha * (v_k . x), aca.rs:187-193
            tk[k] = cmul(alpha, cadd(cadd(tw[0][k], tw[1][k]), cadd(tw[2][k], tw[3][k])));
        __syncthreads();
        leaf_columns(U + (size_t)k0 * L.m, L.m, kc, tk, part, k0 > 0, one, yo);
        __syncthreads();
    }
}

// out[i] = beta * out[i] + sum over the leaves covering row i (fixed order): a
// row's entries are gathered from all over y, so eight lanes share them (one
// thread per row waits for one after another: 43 us at n = 10240, now 10).
constexpr int ROW_LANES = 8, ROW_THREADS = 128;
__global__ void __launch_bounds__(ROW_THREADS) hm_row_reduce_kernel(int64_t n, const int64_t* __restrict__ rowptr,
                                                                    const int64_t* __restrict__ ent,
                                                                    const double2* __restrict__ y, GmBatch bt,
                                                                    int mode, z2 beta, double2* __restrict__ out) {
    if (bt.st) {
        const GmState& st = bt.st[0];
        if (!gm_apply_active(st, mode)) return;
    }
    const int64_t i = (blockIdx.x * (int64_t)ROW_THREADS + threadIdx.x) / ROW_LANES;
    const int l8 = threadIdx.x & (ROW_LANES - 1);
    z2 acc = make_double2(0, 0), b = acc;
    if (i < n) {
        if (beta.x != 0.0 || beta.y != 0.0) b = cmul(beta, out[i]);
        for (int64_t t = rowptr[i] + l8; t < rowptr[i + 1]; t += ROW_LANES) acc = cadd(acc, y[ent[t]]);
    }
    const double s = sum8_parts(acc);  // (every lane has read out[i])
    __syncwarp();
    if (i < n && l8 < 2) reinterpret_cast<double*>(out + i)[l8] = (l8 ? b.y : b.x) + s;
}

static unsigned row_grid(int64_t n) { return (unsigned)((n * ROW_LANES + ROW_THREADS - 1) / ROW_THREADS); }

// ---------------------------------------------------------------------------
static GenParams gen_params(const Problem& p, int side) {
    GenParams g;
    g.kp = kparams(p);
    cd a, b;
    if (side) lhs_factors(p, a, b); else rhs_factors(p, a, b);
    g.alpha = make_double2(a.re, a.im);
    g.beta = make_double2(b.re, b.im);
    g.npad = p.geo.npad;
    g.geo = p.geo.arr(0);
    return g;
}

// The cluster tree and block leaves of a problem's collocation points (they
// depend on the geometry, the leaf size and eta only, not on the frequency),
// built on the device.
struct HTrees {
    std::shared_ptr<Forest> F;
    std::vector<BlockLeaf> bl;
};

static std::shared_ptr<HTrees> build_trees(Context& c, const Problem& p) {
    auto T = std::make_shared<HTrees>();
    T->F = build_forest(c, std::vector<const Problem*>{&p}, p.in.hm_leaf);
    T->bl = forest_block_leaves(c, *T->F, p.in.hm_eta);
    return T;
}

// A leaf whose recompression is more than this share of an SM's is launched first
// and keeps most others off its SM by the shared memory that it asks for, since the
// largest leaf is the last to finish (1534 leaves: 5.7 ms without; shares of 0.1,
// 0.2 and 0.35 all 3.9 ms, 0.9 4.9; with 60 KB 5.1, with 150 and 200 KB, which
// leave it less L1 cache, 4.4 and 5.4).
constexpr double RC_ALONE = 0.2;
constexpr int RC_ALONE_SMEM = 100 * 1024;

template <class Work>
static std::vector<int32_t> heaviest_first(size_t count, Work work) {
    std::vector<std::pair<int64_t, int32_t>> key(count);
    for (size_t b = 0; b < count; ++b) key[b] = {-(int64_t)work(b), (int32_t)b};
    std::sort(key.begin(), key.end());
    std::vector<int32_t> order(count);
    for (size_t b = 0; b < count; ++b) order[b] = key[b].second;
    return order;
}

// trees: the problem's trees from an earlier build (several frequencies of
// one body), or null to build them here.
std::unique_ptr<HMatrixDev> hmatrix_build(Context& c, const Problem& p, int side,
                                          std::shared_ptr<HTrees> trees = nullptr) {
    auto H = std::make_unique<HMatrixDev>();
    const int64_t n = p.n;
    H->n = n;
    if (!trees) trees = build_trees(c, p);
    const Forest& F = *trees->F;
    // every cluster is a range of the cluster-order permutation, so the row
    // and column lists of all leaves are that one array
    H->rows = F.perm;
    H->cols = F.perm;
    int64_t store = 0, scratch = 0, yoff = 0;
    for (const BlockLeaf& t : trees->bl) {
        const TreeNode& r = F.nodes[(size_t)t.r];
        const TreeNode& cc = F.nodes[(size_t)t.c];
        HLeaf L{};
        L.row_off = r.begin;
        L.m = r.end - r.begin;
        L.col_off = cc.begin;
        L.n = cc.end - cc.begin;
        L.adm = t.adm;
        L.store_off = store;
        L.y_off = yoff;
        yoff += L.m;
        if (L.adm) {
            L.kmax = (int32_t)std::min<int64_t>(std::min(L.m, L.n), ACA_RMAX);
            store += (L.m + L.n) * L.kmax;
            L.scratch_off = scratch;
            scratch += 2 * (L.m + L.n) + (L.m + L.n + 15) / 16 + 2;
        } else {
            L.kmax = 0;
            store += L.m * L.n;
        }
        H->leaves.push_back(L);
    }
    // device copies
    const size_t nl = H->leaves.size();
    H->d_leaves.ensure(sizeof(HLeaf) * nl);
    H->d_rows.ensure(sizeof(int64_t) * std::max<size_t>(H->rows.size(), 1));
    H->d_cols.ensure(sizeof(int64_t) * std::max<size_t>(H->cols.size(), 1));
    H->d_store.ensure(sizeof(double2) * (size_t)std::max<int64_t>(store, 1));
    H->d_scratch.ensure(sizeof(double2) * (size_t)std::max<int64_t>(scratch, 1));
    H->d_y.ensure(sizeof(double2) * (size_t)std::max<int64_t>(yoff, 1));
    BEM_CUDA(cudaMemcpyAsync(H->d_leaves.p, H->leaves.data(), sizeof(HLeaf) * nl, cudaMemcpyHostToDevice, c.stream));
    BEM_CUDA(cudaMemcpyAsync(H->d_rows.p, F.d_perm.p, sizeof(int64_t) * H->rows.size(), cudaMemcpyDeviceToDevice,
                             c.stream));
    BEM_CUDA(cudaMemcpyAsync(H->d_cols.p, F.d_perm.p, sizeof(int64_t) * H->cols.size(), cudaMemcpyDeviceToDevice,
                             c.stream));
    // the compressed leaves by size, then by the work their rank makes: a large
    // one begun last would run alone
    std::vector<int32_t> adm_list, dense_list;
    for (int32_t b : heaviest_first(nl, [&](size_t b) { return H->leaves[b].m + H->leaves[b].n; }))
        if (H->leaves[(size_t)b].adm) adm_list.push_back(b);
    for (size_t b = 0; b < nl; ++b)
        if (!H->leaves[b].adm) dense_list.push_back((int32_t)b);
    DevBuf &d_adm = c.w_tree[16], &d_dense = c.w_tree[17];
    d_adm.ensure(sizeof(int32_t) * std::max<size_t>(adm_list.size(), 1));
    d_dense.ensure(sizeof(int32_t) * std::max<size_t>(dense_list.size(), 1));
    BEM_CUDA(cudaMemcpyAsync(d_adm.p, adm_list.data(), sizeof(int32_t) * adm_list.size(), cudaMemcpyHostToDevice,
                             c.stream));
    BEM_CUDA(cudaMemcpyAsync(d_dense.p, dense_list.data(), sizeof(int32_t) * dense_list.size(),
                             cudaMemcpyHostToDevice, c.stream));
    GenParams g = gen_params(p, side);
    HLeaf* dl = H->d_leaves.as<HLeaf>();
    if (!dense_list.empty()) {
        hm_dense_fill_kernel<<<(unsigned)dense_list.size(), LEAF_THREADS, 0, c.stream>>>(
            dl, d_dense.as<int32_t>(), H->d_rows.as<int64_t>(), H->d_cols.as<int64_t>(), g, H->d_store.as<double2>());
        BEM_CHECK_LAUNCH(&c);
        hm_dense_norm_kernel<<<(unsigned)dense_list.size(), LEAF_THREADS, 0, c.stream>>>(dl, d_dense.as<int32_t>(),
                                                                                         H->d_store.as<double2>());
        BEM_CHECK_LAUNCH(&c);
    }
    if (!adm_list.empty()) {
        int* err = device_err(c);
        BEM_CUDA(cudaMemsetAsync(err, 0, sizeof(int), c.stream));
        hm_aca_kernel<<<(unsigned)adm_list.size(), ACA_THREADS, 0, c.stream>>>(
            dl, d_adm.as<int32_t>(), H->d_rows.as<int64_t>(), H->d_cols.as<int64_t>(), g, H->d_store.as<double2>(),
            H->d_scratch.as<double2>(), p.in.hm_aca_tol, err);
        BEM_CHECK_LAUNCH(&c);
        int herr = 0;
        BEM_CUDA(cudaMemcpyAsync(&herr, err, sizeof(int), cudaMemcpyDeviceToHost, c.stream));
        BEM_CUDA(cudaMemcpyAsync(H->leaves.data(), dl, sizeof(HLeaf) * nl, cudaMemcpyDeviceToHost, c.stream));
        c.sync();
        require(herr == 0, "ACA rank exceeded the storage cap of " + std::to_string(ACA_RMAX),
                BEM_ERR_NOT_CONVERGED);
        // FP64 clocks of a leaf's recompression, about
        auto work = [&](int32_t l) {
            const HLeaf& L = H->leaves[(size_t)l];
            return (double)L.rank * L.rank * (8.0 * (double)(L.m + L.n) + 64.0 * L.rank);
        };
        std::stable_sort(adm_list.begin(), adm_list.end(), [&](int32_t a, int32_t b) { return work(a) > work(b); });
        BEM_CUDA(cudaMemcpyAsync(d_adm.p, adm_list.data(), sizeof(int32_t) * adm_list.size(), cudaMemcpyHostToDevice,
                                 c.stream));
        // recompression scratch sized by the ranks just found
        std::vector<int64_t> off(adm_list.size());
        int64_t tot = 0;
        for (size_t a = 0; a < adm_list.size(); ++a) {
            const HLeaf& L = H->leaves[(size_t)adm_list[a]];
            int64_t r = L.rank;
            off[a] = tot;
            tot += 5 * r * r + 2 * r + (L.m + L.n) * r + r + r / 2 + 2;
        }
        DevBuf d_off, d_scr2;
        d_off.ensure(sizeof(int64_t) * off.size());
        d_scr2.ensure(sizeof(double2) * (size_t)std::max<int64_t>(tot, 1));
        BEM_CUDA(cudaMemcpyAsync(d_off.p, off.data(), sizeof(int64_t) * off.size(), cudaMemcpyHostToDevice, c.stream));
        // the largest leaves apart (RC_ALONE)
        int sms = 0;
        BEM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c.device));
        double total = 0;
        for (int32_t l : adm_list) total += work(l);
        size_t alone = 0;
        while (alone < adm_list.size() && alone < (size_t)sms / 2 && work(adm_list[alone]) > RC_ALONE * total / sms) ++alone;
        auto recompress = [&](size_t first, size_t last, size_t smem, cudaStream_t stream) {
            if (first == last) return;
            hm_recompress_kernel<<<(unsigned)(last - first), RC_THREADS, smem, stream>>>(
                dl, d_adm.as<int32_t>() + first, H->d_store.as<double2>(), d_scr2.as<double2>(),
                d_off.as<int64_t>() + first, p.in.hm_aca_tol);
            BEM_CHECK_LAUNCH(&c);
        };
        if (alone) {
            BEM_CUDA(cudaFuncSetAttribute(hm_recompress_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, RC_ALONE_SMEM));
            c.fork();
            recompress(0, alone, RC_ALONE_SMEM, c.stream);  // (goes straight on: ahead of the others)
            recompress(alone, adm_list.size(), 0, c.side);
            c.join();
        } else {
            recompress(0, adm_list.size(), 0, c.stream);
        }
        c.sync();
    }
    BEM_CUDA(cudaMemcpyAsync(H->leaves.data(), dl, sizeof(HLeaf) * nl, cudaMemcpyDeviceToHost, c.stream));
    c.sync();
    // update_norm (h_matrix.rs:189-196): dense leaves first, then low-rank
    double nrm = 0;
    for (auto& L : H->leaves)
        if (!L.adm) nrm += L.norm;
    for (auto& L : H->leaves)
        if (L.adm) nrm += L.norm;
    H->norm = nrm;
    for (auto& L : H->leaves) {
        if (L.adm) {
            H->nadm++;
            H->stored += L.rank * (L.m + L.n);
            H->rank_sum += L.rank;
        } else {
            H->ninadm++;
            H->stored += L.m * L.n;
        }
    }
    const std::vector<int32_t> order = heaviest_first(nl, [&](size_t b) {
        const HLeaf& L = H->leaves[b];
        return L.adm ? L.rank * (L.m + L.n) : L.m * L.n;
    });
    H->d_order.ensure(sizeof(int32_t) * std::max<size_t>(nl, 1));
    BEM_CUDA(cudaMemcpyAsync(H->d_order.p, order.data(), sizeof(int32_t) * nl, cudaMemcpyHostToDevice, c.stream));
    // row CSR over the leaves' output slices (leaf order)
    std::vector<int64_t> cnt((size_t)n + 1, 0);
    for (auto& L : H->leaves)
        for (int64_t i = 0; i < L.m; ++i) cnt[(size_t)H->rows[(size_t)(L.row_off + i)] + 1]++;
    for (int64_t i = 0; i < n; ++i) cnt[(size_t)i + 1] += cnt[(size_t)i];
    std::vector<int64_t> ent((size_t)cnt[(size_t)n]), pos(cnt.begin(), cnt.end() - 1);
    for (auto& L : H->leaves)
        for (int64_t i = 0; i < L.m; ++i) ent[(size_t)pos[(size_t)H->rows[(size_t)(L.row_off + i)]]++] = L.y_off + i;
    H->d_rowptr.ensure(sizeof(int64_t) * cnt.size());
    H->d_rowent.ensure(sizeof(int64_t) * std::max<size_t>(ent.size(), 1));
    BEM_CUDA(cudaMemcpyAsync(H->d_rowptr.p, cnt.data(), sizeof(int64_t) * cnt.size(), cudaMemcpyHostToDevice,
                             c.stream));
    BEM_CUDA(cudaMemcpyAsync(H->d_rowent.p, ent.data(), sizeof(int64_t) * ent.size(), cudaMemcpyHostToDevice,
                             c.stream));
    BEM_CUDA(cudaMemcpyAsync(H->d_leaves.p, H->leaves.data(), sizeof(HLeaf) * nl, cudaMemcpyHostToDevice, c.stream));
    c.sync();
    return H;
}

void hmatrix_gemv(Context& c, const HMatrixDev& H, cd alpha, const double2* x, cd beta, double2* b);

// The built leaves for the mixed form's repacking (hmixed.cu): index lists,
// ranks, norms and the device data of the FP64 build, kept alive by `keep`.
HBuilt hmatrix_build_view(Context& c, const Problem& p, int side, std::shared_ptr<void>* tree_cache) {
    std::shared_ptr<HTrees> trees;
    if (tree_cache && *tree_cache) trees = std::static_pointer_cast<HTrees>(*tree_cache);
    if (!trees) {
        trees = build_trees(c, p);
        if (tree_cache) *tree_cache = trees;
    }
    std::shared_ptr<HMatrixDev> H(hmatrix_build(c, p, side, trees).release());
    HBuilt v;
    v.n = H->n;
    v.norm = H->norm;
    v.leaves.reserve(H->leaves.size());
    for (const HLeaf& L : H->leaves)
        v.leaves.push_back(HLeafView{L.row_off, L.m, L.col_off, L.n, L.store_off, L.adm, L.kmax, L.rank, L.norm});
    v.rows = H->rows;
    v.cols = H->cols;
    v.d_rows = H->d_rows.as<int64_t>();
    v.d_cols = H->d_cols.as<int64_t>();
    v.d_store = H->d_store.as<double2>();
    v.keep = H;
    return v;
}

std::shared_ptr<const Forest> hmatrix_forest(Context& c, const Problem& p, std::shared_ptr<void>* tree_cache) {
    std::shared_ptr<HTrees> trees;
    if (tree_cache && *tree_cache) trees = std::static_pointer_cast<HTrees>(*tree_cache);
    if (!trees) {
        trees = build_trees(c, p);
        if (tree_cache) *tree_cache = trees;
    }
    return trees->F;
}

// out = (alpha H + beta G) 1 with the FP64 H-matrix of `side`
// (h_matrix.rs:218-234 applied to the constant vector), device memory.
void hmatrix_row_sums(Context& c, const Problem& p, int side, double2* out) {
    auto H = hmatrix_build(c, p, side);
    DevBuf ones;
    ones.ensure(sizeof(double2) * (size_t)p.n);
    std::vector<double2> h((size_t)p.n, make_double2(1.0, 0.0));
    BEM_CUDA(cudaMemcpyAsync(ones.p, h.data(), sizeof(double2) * (size_t)p.n, cudaMemcpyHostToDevice, c.stream));
    hmatrix_gemv(c, *H, {1.0, 0.0}, ones.as<double2>(), {0.0, 0.0}, out);
    c.sync();
}

// b = alpha H x + beta b on device vectors (h_matrix.rs:218-234).
void hmatrix_gemv(Context& c, const HMatrixDev& H, cd alpha, const double2* x, cd beta, double2* b) {
    GmBatch none{};
    if (!H.leaves.empty()) {
        hm_leaf_mv_kernel<<<(unsigned)H.leaves.size(), HMV_THREADS, 0, c.stream>>>(
            H.d_leaves.as<HLeaf>(), H.d_order.as<int32_t>(), H.d_cols.as<int64_t>(), H.d_store.as<double2>(), none, 0,
            x, make_double2(alpha.re, alpha.im), const_cast<double2*>(H.d_y.as<double2>()));
        BEM_CHECK_LAUNCH(&c);
    }
    hm_row_reduce_kernel<<<row_grid(H.n), ROW_THREADS, 0, c.stream>>>(
        H.n, H.d_rowptr.as<int64_t>(), H.d_rowent.as<int64_t>(), H.d_y.as<double2>(), none, 0,
        make_double2(beta.re, beta.im), b);
    BEM_CHECK_LAUNCH(&c);
}

// GMRES operator hook: W = H v, predicated on the (single) system's state.
static void hm_apply_hook(Context& c, GmWorkspace& ws, int mode, void* user) {
    const HMatrixDev& H = *static_cast<const HMatrixDev*>(user);
    hm_leaf_mv_kernel<<<(unsigned)H.leaves.size(), HMV_THREADS, 0, c.stream>>>(
        H.d_leaves.as<HLeaf>(), H.d_order.as<int32_t>(), H.d_cols.as<int64_t>(), H.d_store.as<double2>(), ws.bt, mode,
        nullptr, make_double2(1.0, 0.0), const_cast<double2*>(H.d_y.as<double2>()));
    BEM_CHECK_LAUNCH(&c);
    hm_row_reduce_kernel<<<row_grid(H.n), ROW_THREADS, 0, c.stream>>>(
        H.n, H.d_rowptr.as<int64_t>(), H.d_rowent.as<int64_t>(), H.d_y.as<double2>(), ws.bt, mode,
        make_double2(0.0, 0.0), ws.bt.W);
    BEM_CHECK_LAUNCH(&c);
}

GmresResult gmres_hmatrix(Context& c, const HMatrixDev& H, int64_t max_it, double tol, double2* x) {
    const int64_t n = H.n;
    if (max_it <= 0) max_it = 1000;
    if (max_it > n) max_it = n;
    if (tol <= 0.0) tol = 1e-5;
    int m = (int)std::ceil(std::sqrt((double)max_it));
    int64_t restarts = max_it / m;
    GmWorkspace ws;
    ws.mem_pool = &c.w_gm;
    gm_prepare(c, ws, 1, n, m, nullptr, n, 0, false, true);
    ws.hook = hm_apply_hook;
    ws.hook_user = const_cast<HMatrixDev*>(&H);
    BEM_CUDA(cudaMemcpyAsync(ws.bt.B, x, sizeof(double2) * n, cudaMemcpyDeviceToDevice, c.stream));
    BEM_CUDA(cudaMemcpyAsync(ws.anorm, &H.norm, sizeof(double), cudaMemcpyHostToDevice, c.stream));
    gm_init(c, ws, tol, restarts);
    gm_run(c, ws, 1, restarts * (int64_t)m + 1);
    std::vector<GmState> st;
    gm_read_states(c, ws, st);
    BEM_CUDA(cudaMemcpyAsync(x, ws.bt.X, sizeof(double2) * n, cudaMemcpyDeviceToDevice, c.stream));
    c.sync();
    GmresResult r;
    r.num_mv = st[0].num_mv;
    r.restarts = st[0].restarts + (st[0].converged ? 1 : 0);
    r.iterations = st[0].iterations;
    r.error = st[0].error;
    r.flag = st[0].converged ? 1 : 2;
    return r;
}

// solve.rs:74-150 get_surface_hmatrix.
void solve_surface_hmatrix(Context& c, const Problem& p, const double2* d_rhs_inc, double2* d_phi, double2* d_vn,
                           bem_solve_report* rep) {
    const int64_t n = p.n;
    DevBuf vb;
    vb.ensure(sizeof(double2) * 2 * n);
    double2* rhs = vb.as<double2>();
    double2* fillv = rhs + n;
    BEM_CUDA(cudaMemcpyAsync(rhs, d_rhs_inc, sizeof(double2) * n, cudaMemcpyDeviceToDevice, c.stream));
    const bool zero_bc = p.in.bc_value[0] == 0.0 && p.in.bc_value[1] == 0.0;
    cd bcv = {p.in.bc_value[0], p.in.bc_value[1]};
    if (p.in.bc_type == 2) {
        // rhs = 0 * rhs_inc + (-1) rhs
        launch_rhs_combine(c, n, -1.0, d_rhs_inc, {0, 0}, nullptr, rhs);
    } else {
        cd beta = p.in.bc_type == 0 ? cd{1.0, 0.0} : cd{-1.0, 0.0};
        if (!zero_bc) {
            auto Hr = hmatrix_build(c, p, 0);
            std::vector<double2> hv((size_t)n, make_double2(bcv.re, bcv.im));
            BEM_CUDA(cudaMemcpyAsync(fillv, hv.data(), sizeof(double2) * n, cudaMemcpyHostToDevice, c.stream));
            hmatrix_gemv(c, *Hr, {1.0, 0.0}, fillv, beta, rhs);
            c.sync();
        } else if (beta.re != 1.0) {
            launch_rhs_combine(c, n, -1.0, d_rhs_inc, {0, 0}, nullptr, rhs);
        }
    }
    auto Hl = hmatrix_build(c, p, 1);
    GmresResult r = gmres_hmatrix(c, *Hl, p.in.max_iterations, p.in.tolerance, rhs);
    if (rep) {
        rep->num_mv = r.num_mv;
        rep->restarts = r.restarts;
        rep->iterations = r.iterations;
        rep->backward_error = r.error;
        rep->flag = r.flag;
    }
    unpack_solution(c, p, rhs, d_phi, d_vn);
    c.sync();
}

}  // namespace bem

using namespace bem;

extern "C" {

BEM_API bem_status bem_hmatrix_build(bem_ctx* ctx, const bem_problem* pp, bem_side side, bem_hmatrix** out) {
    if (!ctx || !pp || !out) return BEM_ERR_BAD_INPUT;
    *out = nullptr;
    try {
        Context& c = ctx->c;
        BEM_CUDA(cudaSetDevice(c.device));
        auto H = hmatrix_build(c, pp->p, side == BEM_SIDE_LHS ? 1 : 0);
        *out = new bem_hmatrix{H.release(), ctx};
        return BEM_OK;
    } catch (const Error& e) {
        ctx->c.last_error = e.what();
        return e.status;
    } catch (const std::exception& e) {
        ctx->c.last_error = e.what();
        return BEM_ERR_CUDA;
    }
}

BEM_API void bem_hmatrix_destroy(bem_hmatrix* h) {
    if (!h) return;
    delete h->h;
    delete h;
}

BEM_API bem_status bem_hmatrix_gemv(bem_ctx* ctx, const bem_hmatrix* h, bem_cplx alpha, const bem_cplx* x,
                                    bem_cplx beta, bem_cplx* b) {
    if (!ctx || !h || !x || !b) return BEM_ERR_BAD_INPUT;
    try {
        Context& c = ctx->c;
        BEM_CUDA(cudaSetDevice(c.device));
        const int64_t n = h->h->n;
        DevBuf d;
        d.ensure(sizeof(double2) * 2 * n);
        double2* dx = d.as<double2>();
        double2* db = dx + n;
        BEM_CUDA(cudaMemcpyAsync(dx, x, sizeof(double2) * n, cudaMemcpyHostToDevice, c.stream));
        BEM_CUDA(cudaMemcpyAsync(db, b, sizeof(double2) * n, cudaMemcpyHostToDevice, c.stream));
        hmatrix_gemv(c, *h->h, {alpha.re, alpha.im}, dx, {beta.re, beta.im}, db);
        BEM_CUDA(cudaMemcpyAsync(b, db, sizeof(double2) * n, cudaMemcpyDeviceToHost, c.stream));
        c.sync();
        return BEM_OK;
    } catch (const Error& e) {
        ctx->c.last_error = e.what();
        return e.status;
    }
}

BEM_API double bem_hmatrix_norm(const bem_hmatrix* h) { return h ? h->h->norm : 0.0; }

BEM_API bem_status bem_hmatrix_stats(const bem_hmatrix* h, int64_t* s) {
    if (!h || !s) return BEM_ERR_BAD_INPUT;
    s[0] = h->h->nadm;
    s[1] = h->h->ninadm;
    s[2] = h->h->stored;
    s[3] = h->h->rank_sum;
    return BEM_OK;
}

BEM_API bem_status bem_hmatrix_to_full(bem_ctx* ctx, const bem_hmatrix* h, bem_cplx* A, int64_t lda) {
    if (!ctx || !h || !A || lda < h->h->n) return BEM_ERR_BAD_INPUT;
    // columns of the identity through the mat-vec kernels (h_matrix.rs:236-246)
    const int64_t n = h->h->n;
    std::vector<double2> e((size_t)n), col((size_t)n);
    try {
        Context& c = ctx->c;
        BEM_CUDA(cudaSetDevice(c.device));
        DevBuf d;
        d.ensure(sizeof(double2) * 2 * n);
        double2* dx = d.as<double2>();
        double2* db = dx + n;
        BEM_CUDA(cudaMemsetAsync(dx, 0, sizeof(double2) * n, c.stream));
        const double2 one = make_double2(1, 0), zero = make_double2(0, 0);
        for (int64_t j = 0; j < n; ++j) {
            if (j > 0) BEM_CUDA(cudaMemcpyAsync(dx + j - 1, &zero, sizeof(double2), cudaMemcpyHostToDevice, c.stream));
            BEM_CUDA(cudaMemcpyAsync(dx + j, &one, sizeof(double2), cudaMemcpyHostToDevice, c.stream));
            hmatrix_gemv(c, *h->h, {1.0, 0.0}, dx, {0.0, 0.0}, db);
            BEM_CUDA(cudaMemcpyAsync(A + j * lda, db, sizeof(double2) * n, cudaMemcpyDeviceToHost, c.stream));
            c.sync();
        }
        return BEM_OK;
    } catch (const Error& e) {
        ctx->c.last_error = e.what();
        return e.status;
    }
}

}  // extern "C"
