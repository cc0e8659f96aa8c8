// Fit of the HLQ parameters of one group of weights (q plane scales and one offset) by
// alternating between the assignment of every weight to the nearest of the 2^q values
// sum_j s_j b_j + c and a least-squares solve for (s, c) under that assignment.
//
// Replaces the reference quantizer's
//   find_optimal_params_alternating        GPTQ/quant.py:118-153
//   optimize_s_batch_with_constant         GPTQ/quant.py:104-116   (batched (q+1) x (q+1) normal equations, pinv)
//   generate_augmented_bit_combinations    GPTQ/quant.py:95-102    (value i has bit j = (i >> j) & 1, then the constant)
// Two kernels.  fit_lanes_kernel keeps a group of 32, 64 or 128 weights in the registers of 4 or 8
// lanes for all iterations and can go on to the assignment and the reconstruction
// (hlq_pseudo_quantize_device), so that a weight is read once and each result written once.
// fit_alternating_kernel (any group up to 1024 weights, any alignment): one warp per group, the
// weights in shared memory.
//
// The (q+1) x (q+1) matrix of the normal equations is the Gram matrix of 0/1 vectors, so its
// determinant is a whole number: it is either singular or at least 1, and in the second case (the
// inverse of a 0/1 matrix of order <= 5 has entries of at most 3) its smallest eigenvalue is at least
// 1/225, above the cut-off max(q+1) * eps_f32 * largest of torch.linalg.pinv for float32 up to 1024
// weights.  So the pseudo-inverse is the inverse unless a pivot of the elimination vanishes, and
// the systems are solved by elimination in double precision; only where a pivot vanishes (a plane
// that no weight uses, a constant group) the eigen-decomposition (Jacobi) does it, as before.
#include <cuda_runtime.h>
#include <math.h>

#include "hlq_internal.h"

namespace hlq {
namespace {

constexpr int kFitWarps = 4;
constexpr int kFitMaxG = 1024;

// pinv(A) * r for a symmetric positive semi-definite A of order n <= 5, in place: x = result
template <int N>
__device__ void solve_pinv(double (&A)[N][N], const double (&r)[N], double (&x)[N], double rtol) {
    double V[N][N];
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
        for (int j = 0; j < N; ++j) V[i][j] = i == j ? 1.0 : 0.0;
    for (int sweep = 0; sweep < 12; ++sweep) {
        double off = 0.0;
#pragma unroll
        for (int p = 0; p < N; ++p)
#pragma unroll
            for (int q = p + 1; q < N; ++q) off += A[p][q] * A[p][q];
        if (off < 1e-26) break;
#pragma unroll
        for (int p = 0; p < N; ++p) {
#pragma unroll
            for (int q = p + 1; q < N; ++q) {
                const double apq = A[p][q];
                if (fabs(apq) < 1e-300) continue;
                const double theta = (A[q][q] - A[p][p]) / (2.0 * apq);
                const double t = (theta >= 0 ? 1.0 : -1.0) / (fabs(theta) + sqrt(theta * theta + 1.0));
                const double c = 1.0 / sqrt(t * t + 1.0), s = t * c;
#pragma unroll
                for (int k = 0; k < N; ++k) {          // A <- A J
                    const double akp = A[k][p], akq = A[k][q];
                    A[k][p] = c * akp - s * akq;
                    A[k][q] = s * akp + c * akq;
                }
#pragma unroll
                for (int k = 0; k < N; ++k) {          // A <- J^T A
                    const double apk = A[p][k], aqk = A[q][k];
                    A[p][k] = c * apk - s * aqk;
                    A[q][k] = s * apk + c * aqk;
                }
#pragma unroll
                for (int k = 0; k < N; ++k) {
                    const double vkp = V[k][p], vkq = V[k][q];
                    V[k][p] = c * vkp - s * vkq;
                    V[k][q] = s * vkp + c * vkq;
                }
            }
        }
    }
    double lmax = 0.0;
#pragma unroll
    for (int i = 0; i < N; ++i) lmax = fmax(lmax, fabs(A[i][i]));
#pragma unroll
    for (int i = 0; i < N; ++i) x[i] = 0.0;
#pragma unroll
    for (int e = 0; e < N; ++e) {
        const double lam = A[e][e];
        if (fabs(lam) <= rtol * lmax) continue;
        double proj = 0.0;
#pragma unroll
        for (int k = 0; k < N; ++k) proj += V[k][e] * r[k];
        proj /= lam;
#pragma unroll
        for (int k = 0; k < N; ++k) x[k] += V[k][e] * proj;
    }
}

// The solution of A x = r by elimination (A symmetric positive definite, integer entries); false
// when a pivot vanishes, i.e. A is singular.  A pivot of a nonsingular A is at least its smallest
// eigenvalue, 1/225; rounding leaves 1e-12 in place of a zero.
template <int N>
__device__ __forceinline__ bool solve_pd(const double (&Ain)[N][N], const double (&rin)[N], double (&x)[N]) {
    double A[N][N], r[N], inv[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
        r[i] = rin[i];
#pragma unroll
        for (int j = i; j < N; ++j) A[i][j] = Ain[i][j];
    }
    bool ok = true;
#pragma unroll
    for (int p = 0; p < N; ++p) {
        ok = ok && A[p][p] > 1e-4;
        inv[p] = 1.0 / A[p][p];
#pragma unroll
        for (int i = p + 1; i < N; ++i) {
            const double f = A[p][i] * inv[p];
#pragma unroll
            for (int j = i; j < N; ++j) A[i][j] -= f * A[p][j];
            r[i] -= f * r[p];
        }
    }
#pragma unroll
    for (int p = N - 1; p >= 0; --p) {
        double t = r[p];
#pragma unroll
        for (int j = p + 1; j < N; ++j) t -= A[p][j] * x[j];
        x[p] = t * inv[p];
    }
    return ok;
}
// The same where A is singular.
template <int N>
__device__ __noinline__ void solve_singular(const double *Ain, const double *rin, double *xout) {
    double A[N][N], r[N], x[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
        r[i] = rin[i];
#pragma unroll
        for (int j = 0; j < N; ++j) A[i][j] = Ain[i * N + j];
    }
    solve_pinv<N>(A, r, x, (double)N * 1.1920928955078125e-7);
#pragma unroll
    for (int i = 0; i < N; ++i) xout[i] = x[i];
}
template <int N>
__device__ __forceinline__ void solve_normal(const double (&A)[N][N], const double (&r)[N], float (&s)[N]) {
    double x[N];
    if (!solve_pd<N>(A, r, x)) {
        double At[N * N], rt[N];
#pragma unroll
        for (int i = 0; i < N; ++i) {
            rt[i] = r[i];
#pragma unroll
            for (int j = 0; j < N; ++j) At[i * N + j] = A[i][j];
        }
        solve_singular<N>(At, rt, x);
    }
#pragma unroll
    for (int i = 0; i < N; ++i) s[i] = (float)x[i];
}

template <int Q>
__global__ void __launch_bounds__(kFitWarps * 32) fit_alternating_kernel(const float *__restrict__ w,
                                                                         float *__restrict__ scales,
                                                                         float *__restrict__ zeros, int64_t blocks,
                                                                         int g, int iters) {
    __shared__ float ys[kFitWarps][kFitMaxG];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t b = (int64_t)blockIdx.x * kFitWarps + warp;
    if (b >= blocks) return;
    float *y = ys[warp];
    float lo = INFINITY, hi = -INFINITY;
    for (int e = lane; e < g; e += 32) {
        const float v = w[b * g + e];
        y[e] = v;
        lo = fminf(lo, v);
        hi = fmaxf(hi, v);
    }
#pragma unroll
    for (int d = 16; d; d >>= 1) {
        lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, d));
        hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, d));
    }
    __syncwarp();
    // start: plane j gets range / (2^q - 1) * 2^j, the constant the minimum (quant.py:128-134)
    float s[Q + 1];
    const float step = (hi - lo) / (float)((1 << Q) - 1);
#pragma unroll
    for (int j = 0; j < Q; ++j) s[j] = step * (float)(1 << j);
    s[Q] = lo;
    for (int it = 0; it < iters; ++it) {
        float comb[1 << Q];
#pragma unroll
        for (int v = 0; v < (1 << Q); ++v) {
            float t = 0.f;
#pragma unroll
            for (int j = 0; j < Q; ++j)
                if ((v >> j) & 1) t += s[j];
            comb[v] = t + s[Q];
        }
        // sums of the normal equations over this lane's weights
        constexpr int NP = Q * (Q + 1) / 2;      // pairs i <= j < Q
        float cnt[NP], sy[Q + 1];
#pragma unroll
        for (int i = 0; i < NP; ++i) cnt[i] = 0.f;
#pragma unroll
        for (int i = 0; i <= Q; ++i) sy[i] = 0.f;
        for (int e = lane; e < g; e += 32) {
            const float v = y[e];
            float best = INFINITY;
            int arg = 0;
#pragma unroll
            for (int c = 0; c < (1 << Q); ++c) {
                const float dist = fabsf(v - comb[c]);
                if (dist < best) {               // first minimum, as torch.argmin
                    best = dist;
                    arg = c;
                }
            }
            int idx = 0;
#pragma unroll
            for (int i = 0; i < Q; ++i) {
#pragma unroll
                for (int j = i; j < Q; ++j) {
                    if (((arg >> i) & 1) && ((arg >> j) & 1)) cnt[idx] += 1.f;
                    ++idx;
                }
                if ((arg >> i) & 1) sy[i] += v;
            }
            sy[Q] += v;
        }
#pragma unroll
        for (int d = 16; d; d >>= 1) {
#pragma unroll
            for (int i = 0; i < NP; ++i) cnt[i] += __shfl_xor_sync(0xffffffffu, cnt[i], d);
#pragma unroll
            for (int i = 0; i <= Q; ++i) sy[i] += __shfl_xor_sync(0xffffffffu, sy[i], d);
        }
        double A[Q + 1][Q + 1], r[Q + 1];
        int idx = 0;
#pragma unroll
        for (int i = 0; i < Q; ++i) {
#pragma unroll
            for (int j = i; j < Q; ++j) {
                A[i][j] = A[j][i] = (double)cnt[idx];
                ++idx;
            }
        }
        idx = 0;
#pragma unroll
        for (int i = 0; i < Q; ++i) {
            A[i][Q] = A[Q][i] = (double)cnt[idx];      // sum of b_i = count of (i, i)
            idx += Q - i;
            r[i] = (double)sy[i];
        }
        A[Q][Q] = (double)g;
        r[Q] = (double)sy[Q];
        solve_normal<Q + 1>(A, r, s);
    }
    if (lane == 0) {
#pragma unroll
        for (int j = 0; j < Q; ++j) scales[b * Q + j] = s[j];
        zeros[b] = s[Q];
    }
}

// L = 4 or 8 lanes own a group of L * E weights, E of them in each lane's registers: lane l has the runs
// of four elements l, l + L, l + 2 L, ...
//
// Bound by issue slots.  Per weight and iteration: the distances to the 2^q values and a tournament among
// them (the lower code wins a tie, which is the first minimum), whose winners' bits are predicates of the
// additions to the planes' sums and packed pair counts.  The system is solved once per group by each
// of its lanes: the fewer lanes, the less that costs per group (32/L groups a warp).
// The sums are taken in the order of fit_alternating_kernel (elements e, e + 32, ... one after the
// other, then the 32 sums pairwise, those 16 apart first), so both kernels give the same bits.
// Measured (B200, 4096 x 4096, g = 128, 10 iterations, with assignment and reconstruction): 2 bits
// 158 us, against 3409 us for a warp per group with the eigen-decomposition in every iteration and the
// assignment and the reconstruction as passes of their own.
template <int Q, int L, int E>
__global__ void __launch_bounds__(128) fit_lanes_kernel(const float *__restrict__ w, float *__restrict__ scales,
                                                        float *__restrict__ zeros, float *__restrict__ recon,
                                                        uint8_t *__restrict__ quant, int64_t blocks, int iters) {
    static_assert(L == 4 || L == 8, "the summation order wants runs of 32 elements inside one lane group");
    constexpr int NV = 1 << Q, G = L * E;
    constexpr int H = 8 / L;                         // 1: a run of 32 is one round of the lanes; 2: two
    constexpr int NP = Q * (Q + 1) / 2, NW = (NP + 3) / 4;
    static_assert(E % (4 * H) == 0 && G <= 255, "whole runs of 32; byte counts");
    const int l = threadIdx.x % L;
    const int64_t own = (int64_t)blockIdx.x * (128 / L) + threadIdx.x / L;
    const bool live = own < blocks;
    const int64_t b = live ? own : blocks - 1;      // lanes without a group follow the last one and store nothing
    float v[E];
    float lo = INFINITY, hi = -INFINITY;
#pragma unroll
    for (int i = 0; i < E / 4; ++i) {
        const float4 f = __ldg((const float4 *)(w + b * G) + i * L + l);
        v[4 * i] = f.x; v[4 * i + 1] = f.y; v[4 * i + 2] = f.z; v[4 * i + 3] = f.w;
    }
#pragma unroll
    for (int e = 0; e < E; ++e) {
        lo = fminf(lo, v[e]);
        hi = fmaxf(hi, v[e]);
    }
#pragma unroll
    for (int d = L / 2; d; d >>= 1) {
        lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, d));
        hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, d));
    }
    // part[h][c]: this lane's elements with index (4 (l + L h) + c) mod 32, added up; all lanes get the total
    auto reduce = [&](float (&part)[H][4]) {
        float t[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            t[c] = H == 2 ? part[0][c] + part[H - 1][c] : part[0][c];
#pragma unroll
            for (int d = L / 2; d; d >>= 1) t[c] += __shfl_xor_sync(0xffffffffu, t[c], d);
        }
        return (t[0] + t[2]) + (t[1] + t[3]);
    };
    float total;
    {
        float part[H][4] = {};
#pragma unroll
        for (int e = 0; e < E; ++e) part[(e >> 2) % H][e & 3] += v[e];
        total = reduce(part);
    }
    // start: plane j gets range / (2^q - 1) * 2^j, the constant the minimum (quant.py:128-134)
    float s[Q + 1];
    const float step = (hi - lo) / (float)(NV - 1);
#pragma unroll
    for (int j = 0; j < Q; ++j) s[j] = step * (float)(1 << j);
    s[Q] = lo;
#pragma unroll 1
    for (int it = 0; it < iters; ++it) {
        float comb[NV];
#pragma unroll
        for (int c = 0; c < NV; ++c) {
            float t = 0.f;
#pragma unroll
            for (int j = 0; j < Q; ++j)
                if ((c >> j) & 1) t += s[j];
            comb[c] = t + s[Q];
        }
        float part[Q][H][4] = {};
        uint32_t cnt[NW] = {};               // pairs i <= j < Q, a byte each
#pragma unroll
        for (int e = 0; e < E; ++e) {
            float best[NV];
            bool bit[Q][NV / 2];
#pragma unroll
            for (int c = 0; c < NV; ++c) best[c] = fabsf(v[e] - comb[c]);
#pragma unroll
            for (int lv = 0; lv < Q; ++lv)
#pragma unroll
                for (int i = 0; i < (NV >> (lv + 1)); ++i) {
                    const bool up = best[2 * i + 1] < best[2 * i];
#pragma unroll
                    for (int j = 0; j < lv; ++j) bit[j][i] = up ? bit[j][(2 * i + 1) % (NV / 2)] : bit[j][(2 * i) % (NV / 2)];
                    bit[lv][i] = up;
                    best[i] = fminf(best[2 * i], best[2 * i + 1]);
                }
            int idx = 0;
#pragma unroll
            for (int i = 0; i < Q; ++i) {
                if (bit[i][0]) part[i][(e >> 2) % H][e & 3] += v[e];
#pragma unroll
                for (int j = i; j < Q; ++j, ++idx)
                    if (bit[i][0] && bit[j][0]) cnt[idx >> 2] += 1u << (8 * (idx & 3));
            }
        }
#pragma unroll
        for (int k = 0; k < NW; ++k)
#pragma unroll
            for (int d = L / 2; d; d >>= 1) cnt[k] += __shfl_xor_sync(0xffffffffu, cnt[k], d);
        double A[Q + 1][Q + 1], r[Q + 1];
        int idx = 0;
#pragma unroll
        for (int i = 0; i < Q; ++i) {
            r[i] = (double)reduce(part[i]);
#pragma unroll
            for (int j = i; j < Q; ++j, ++idx) A[i][j] = A[j][i] = (double)((cnt[idx >> 2] >> (8 * (idx & 3))) & 0xffu);
            A[i][Q] = A[Q][i] = A[i][i];
        }
        A[Q][Q] = (double)G;
        r[Q] = (double)total;
        solve_normal<Q + 1>(A, r, s);
    }
    if (live && l == 0) {
#pragma unroll
        for (int j = 0; j < Q; ++j) scales[b * Q + j] = s[j];
        zeros[b] = s[Q];
    }
    if (!quant || !live) return;
    // The assignment of the finished fit, in the arithmetic of quantize_with_scales (GPTQ/quant.py:154-174):
    // first minimum over the codes with plane 0 in the highest bit, distances to w - zero.
    float cand[NV];
#pragma unroll
    for (int c = 0; c < NV; ++c) {
        float t = 0.f;
#pragma unroll
        for (int j = 0; j < Q; ++j)
            if ((c >> (Q - 1 - j)) & 1) t = __fadd_rn(t, s[j]);
        cand[c] = t;
    }
#pragma unroll
    for (int i = 0; i < E / 4; ++i) {
        float rec[4];
        uint32_t bytes[Q] = {};
#pragma unroll
        for (int c4 = 0; c4 < 4; ++c4) {
            const float t = __fsub_rn(v[4 * i + c4], s[Q]);
            float best = INFINITY, bv = 0.f;
            int arg = 0;
#pragma unroll
            for (int c = 0; c < NV; ++c) {
                const float dist = fabsf(__fsub_rn(cand[c], t));
                if (dist < best) {
                    best = dist;
                    arg = c;
                    bv = cand[c];
                }
            }
            rec[c4] = __fadd_rn(bv, s[Q]);
#pragma unroll
            for (int j = 0; j < Q; ++j) {
                const int at = c4 * Q + j;
                bytes[at >> 2] |= (uint32_t)((arg >> (Q - 1 - j)) & 1) << (8 * (at & 3));
            }
        }
        const int64_t e4 = b * (G / 4) + i * L + l;          // index of this run of four weights
        ((float4 *)recon)[e4] = make_float4(rec[0], rec[1], rec[2], rec[3]);
        uint32_t *qo = (uint32_t *)quant + e4 * Q;
        if constexpr (Q == 4) *(uint4 *)qo = make_uint4(bytes[0], bytes[1 % Q], bytes[2 % Q], bytes[3 % Q]);
        else if constexpr (Q == 2) *(uint2 *)qo = make_uint2(bytes[0], bytes[1 % Q]);
        else {
#pragma unroll
            for (int j = 0; j < Q; ++j) qo[j] = bytes[j];
        }
    }
}

template <int Q, int L, int E>
int launch_lanes(const float *w, float *scales, float *zeros, float *recon, uint8_t *quant, int64_t blocks, int iters,
                 cudaStream_t st) {
    const int64_t per = 128 / L;
    fit_lanes_kernel<Q, L, E><<<(unsigned)((blocks + per - 1) / per), 128, 0, st>>>(w, scales, zeros, recon, quant, blocks, iters);
    count_launch();
    return note_cuda(cudaGetLastError());
}

// Whether fit_lanes_kernel takes the group size.
bool lanes_group(int g) { return g == 32 || g == 64 || g == 128; }

// Four lanes per group, or eight where eight fill the GPU less than twice over (148 SMs x 2048
// threads): a group's ten iterations are one serial chain, which more lanes shorten.
template <int Q>
int launch_lanes_q(int g, const float *w, float *scales, float *zeros, float *recon, uint8_t *quant, int64_t blocks,
                   int iters, cudaStream_t st) {
    const bool few = blocks * 8 < 2 * 148 * 2048;
    if (g == 32) return few ? launch_lanes<Q, 8, 4>(w, scales, zeros, recon, quant, blocks, iters, st)
                            : launch_lanes<Q, 4, 8>(w, scales, zeros, recon, quant, blocks, iters, st);
    if (g == 64) return few ? launch_lanes<Q, 8, 8>(w, scales, zeros, recon, quant, blocks, iters, st)
                            : launch_lanes<Q, 4, 16>(w, scales, zeros, recon, quant, blocks, iters, st);
    return few ? launch_lanes<Q, 8, 16>(w, scales, zeros, recon, quant, blocks, iters, st)
               : launch_lanes<Q, 4, 32>(w, scales, zeros, recon, quant, blocks, iters, st);
}
int launch_lanes_fit(int q, int g, const float *w, float *scales, float *zeros, float *recon, uint8_t *quant,
                     int64_t blocks, int iters, cudaStream_t st) {
    switch (q) {
        case 1: return launch_lanes_q<1>(g, w, scales, zeros, recon, quant, blocks, iters, st);
        case 2: return launch_lanes_q<2>(g, w, scales, zeros, recon, quant, blocks, iters, st);
        case 3: return launch_lanes_q<3>(g, w, scales, zeros, recon, quant, blocks, iters, st);
        default: return launch_lanes_q<4>(g, w, scales, zeros, recon, quant, blocks, iters, st);
    }
}

// y = sum of the planes' scales whose bit is set + zero, for quantized bytes made by another kernel
template <int Q>
__global__ void reconstruct_kernel(const uint8_t *__restrict__ quant, const float *__restrict__ scales,
                                   const float *__restrict__ zeros, float *__restrict__ recon, int64_t total, int g) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
        const int64_t b = i / g;
        float t = 0.f;
#pragma unroll
        for (int j = 0; j < Q; ++j)
            if (quant[i * Q + j]) t += scales[b * Q + j];
        recon[i] = t + zeros[b];
    }
}

}  // namespace
}  // namespace hlq

using namespace hlq;

extern "C" int hlq_fit_alternating_device(const float *d_w, float *d_scales, float *d_zeros, int64_t blocks, int g,
                                          int q, int iters, void *stream) {
    if (blocks < 0 || g <= 0 || iters < 0) return HLQ_ERR_INVALID_ARGUMENT;
    if (q < 1 || q > 4) return HLQ_ERR_SHAPE;
    if (g > kFitMaxG) return HLQ_ERR_UNSUPPORTED;
    if (blocks == 0) return HLQ_OK;
    if (!d_w || !d_scales || !d_zeros) return HLQ_ERR_INVALID_ARGUMENT;
    if (lanes_group(g) && !((uintptr_t)d_w & 15))
        return launch_lanes_fit(q, g, d_w, d_scales, d_zeros, nullptr, nullptr, blocks, iters, (cudaStream_t)stream);
    const unsigned grid = (unsigned)((blocks + kFitWarps - 1) / kFitWarps);
    cudaStream_t st = (cudaStream_t)stream;
    switch (q) {
        case 1: fit_alternating_kernel<1><<<grid, kFitWarps * 32, 0, st>>>(d_w, d_scales, d_zeros, blocks, g, iters); break;
        case 2: fit_alternating_kernel<2><<<grid, kFitWarps * 32, 0, st>>>(d_w, d_scales, d_zeros, blocks, g, iters); break;
        case 3: fit_alternating_kernel<3><<<grid, kFitWarps * 32, 0, st>>>(d_w, d_scales, d_zeros, blocks, g, iters); break;
        default: fit_alternating_kernel<4><<<grid, kFitWarps * 32, 0, st>>>(d_w, d_scales, d_zeros, blocks, g, iters); break;
    }
    count_launch();
    return note_cuda(cudaGetLastError());
}

extern "C" int hlq_pseudo_quantize_device(const float *d_w, float *d_recon, uint8_t *d_quant, float *d_scales,
                                          float *d_zeros, int64_t blocks, int g, int q, int iters, void *stream) {
    if (blocks < 0 || g <= 0 || iters < 0) return HLQ_ERR_INVALID_ARGUMENT;
    if (q < 1 || q > 4) return HLQ_ERR_SHAPE;
    if (g > kFitMaxG) return HLQ_ERR_UNSUPPORTED;
    if (blocks == 0) return HLQ_OK;
    if (!d_w || !d_recon || !d_quant || !d_scales || !d_zeros) return HLQ_ERR_INVALID_ARGUMENT;
    cudaStream_t st = (cudaStream_t)stream;
    if (lanes_group(g) && !(((uintptr_t)d_w | (uintptr_t)d_recon | (uintptr_t)d_quant) & 15))
        return launch_lanes_fit(q, g, d_w, d_scales, d_zeros, d_recon, d_quant, blocks, iters, st);
    int rc = hlq_fit_alternating_device(d_w, d_scales, d_zeros, blocks, g, q, iters, stream);
    if (!rc) rc = hlq_quantize_with_scales_device(d_w, d_scales, d_zeros, d_quant, blocks, g, q, stream);
    if (rc) return rc;
    const int64_t total = blocks * g, want = (total + 255) / 256;
    const unsigned grid = (unsigned)(want < 148 * 16 ? want : 148 * 16);
    switch (q) {
        case 1: reconstruct_kernel<1><<<grid, 256, 0, st>>>(d_quant, d_scales, d_zeros, d_recon, total, g); break;
        case 2: reconstruct_kernel<2><<<grid, 256, 0, st>>>(d_quant, d_scales, d_zeros, d_recon, total, g); break;
        case 3: reconstruct_kernel<3><<<grid, 256, 0, st>>>(d_quant, d_scales, d_zeros, d_recon, total, g); break;
        default: reconstruct_kernel<4><<<grid, 256, 0, st>>>(d_quant, d_scales, d_zeros, d_recon, total, g); break;
    }
    count_launch();
    return note_cuda(cudaGetLastError());
}
