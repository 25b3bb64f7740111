// fd2_surrogate.cu -- the learned surrogate: MLP training and inference.
//
// Network (hidden width H, 256 by default):
//   x0 [B][32]  normalised features (8 used, zero padded to the GEMM's K)
//   h1 = relu(x0 W1^T + b1), h2 = relu(h1 W2^T + b2), h3 = relu(h2 W3^T + b3)
//   out = h3 W4^T + b4       [B][64] (25 used)
// All products run on fd2_sg_gemm.cuh (BF16 operands, FP32 accumulation);
// FP32 master parameters, BF16 copies for the GEMMs, Adam in FP32.  One
// training step (batch gather, forward, loss, backward, Adam) is a CUDA
// graph replayed `steps` times; the step counter lives on the device.
//
// Loss per point with N photons, d detected and radial label counts h_j
// (j < R: quadratic bins inside radial_max_um, j = R beyond):
//   L = BCE(sigmoid(out0), d / N)
//     + lambda * sum_j y_j (-log q_j),   y_j = h_j / sum h
// with q_j the probability of bin j under the mixture of Gaussian rings
//   PRF(r) = sum_k w_k N(r; mu_k, s_k) / S_k per unit area (fd2_sg_mix.cuh),
//   w = softmax(out[1..8]), mu = 50 um * softplus(out[9..16]),
//   s = 10 um * exp(clamp(out[17..24], -6, 4)).
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#include "fd2.h"
#include "fd2_sg_gemm.cuh"
#include "fd2_sg_tc.cuh"
#include "fd2_sg_internal.h"
#include "fd2_sg_mix.cuh"
#include "fd2_surrogate.h"

using fd2::sg::GemmArgs;

namespace fd2 {
namespace sg {

// ------------------------------------------------------------ device math

__device__ __forceinline__ uint4 philox10(uint4 c, uint32_t k0, uint32_t k1)
{
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        const uint32_t lo0 = 0xD2511F53u * c.x, hi0 = __umulhi(0xD2511F53u, c.x);
        const uint32_t lo1 = 0xCD9E8D57u * c.z, hi1 = __umulhi(0xCD9E8D57u, c.z);
        c = make_uint4(hi1 ^ c.y ^ k0, lo1, hi0 ^ c.w ^ k1, lo0);
        k0 += 0x9E3779B9u;
        k1 += 0xBB67AE85u;
    }
    return c;
}

// One point's loss and the gradients of its outputs, in a warp: lanes 0..7
// hold the gradients of component lane's weight, radius and width outputs.
struct PointLoss {
    float det, rad, total;
    float gz, ga, gom, gls;
};

constexpr int kLossWarps = 4;
constexpr int kSums = 3 * kComponents + 1;  // sums over the categories: A1, Amu, Asd of the components, and the loss

// What the warp of a row shares.
struct LossShared {
    float v[kSums][33];         // per category of a pass: M, dM/dmu, dM/dsd of the components, log q
    float c[32], ny[32];        // y / q and -y of the pass's categories
    float4 mix[kComponents];    // w, mu, sd, S
    float cross[kComponents];   // lower tail at the first edge past the ring's radius
    float4 edge[kComponents];   // the last edge of the pass before: t, tail, pdf
};

// Loss of one point and its gradients, computed by the 32 lanes of a warp
// together.  o: the network's outputs; y: normalised radial label over bins + 1
// categories, used when has_rad (else the point has no radial term).  The
// radial term is the cross-entropy -sum_j y_j log q_j of the ring mixture's
// category probabilities q_j = sum_k w_k M_k(e_j, e_j+1) / S_k
// (fd2_sg_mix.cuh).  A lane holds one upper edge of the categories, 32 a pass
// (96 bins: three passes), and goes through the components in order; the first
// edge and the category beyond r_max, one each, are a lane per component.  The
// sums over the categories run in category order, a lane per sum, from shared
// memory.
__device__ __forceinline__ PointLoss point_loss(const float *o, float t, const float *y, bool has_rad, int bins,
                                                float r_max, float lambda, LossShared &h)
{
    const int lane = threadIdx.x & 31, k = lane % kComponents;
    PointLoss p;
    // detection
    const float z = o[0];
    const float pd = 1.0f / (1.0f + expf(-z));
    // log p = -softplus(-z), log(1 - p) = -softplus(z)
    const float sp_neg = fmaxf(-z, 0.0f) + log1pf(expf(-fabsf(z)));
    const float sp_pos = fmaxf(z, 0.0f) + log1pf(expf(-fabsf(z)));
    const float ld = t * sp_neg + (1.0f - t) * sp_pos;
    p.gz = pd - t;
    p.det = p.total = ld;
    p.rad = p.ga = p.gom = p.gls = 0.0f;
    if (!has_rad) return p;
    // component k, the same in lanes k, 8 + k, ...
    const float om = o[1 + kComponents + k], ls = o[1 + 2 * kComponents + k];
    const float w = lane_weight(o[1 + k]);
    const Ring ring = decode_ring(om, ls);
    const float mu = ring.mu, sd = ring.sd, S = ring.S;
    const float dmu = kMuScale / (1.0f + expf(-om));  // d mu / d output
    const bool clamped = ls < kLogSdMin || ls > kLogSdMax;
    __syncwarp();  // every lane is done with the row before
    if (lane < kComponents) {
        // of an edge's two tails only the one away from the ring is kept, and
        // at the first edge past the ring's radius the other one as well: the
        // interval that holds the radius reads it (ring_mass)
        int j = min(max((int)((float)bins * sqrtf(mu / r_max)) - 1, 1), bins);
        while (j <= bins && radial_edge(j, bins, r_max) < mu) ++j;
        h.cross[lane] = normcdff((radial_edge(j, bins, r_max) - mu) / sd);
        const float te = (0.0f - mu) / sd;
        h.edge[lane] = make_float4(te, normcdff(te >= 0.0f ? -te : te), norm_pdf(te), 0.0f);
        h.mix[lane] = make_float4(w, mu, sd, S);
    }
    __syncwarp();
    // lane c of the first kSums: A1 = sum_j c_j M_j, Amu = sum_j c_j dM_j/dmu,
    // Asd = sum_j c_j dM_j/dsd of component c % 8, and the last the loss
    float sum = 0.0f;
    for (int j0 = 1; j0 <= bins; j0 += 32) {
        const int j = j0 + lane, n = min(32, bins + 1 - j0);  // of the pass's categories j - 1 and edges j
        Edge lo, hi;
        lo.inf = hi.inf = false;
        lo.e = radial_edge(j - 1, bins, r_max);
        hi.e = radial_edge(j, bins, r_max);
        float q = 0.0f;
#pragma unroll 2
        for (int c = 0; c < kComponents; ++c) {
            const float4 mix = h.mix[c];
            const float wc = mix.x, mc = mix.y, sc = mix.z, Sc = mix.w;
            hi.t = (hi.e - mc) / sc;
            const bool past = hi.t >= 0.0f;
            const float tail = normcdff(past ? -hi.t : hi.t);
            hi.pdf = norm_pdf(hi.t);
            lo.t = __shfl_up_sync(0xffffffffu, hi.t, 1);
            lo.cdf = lo.ccdf = __shfl_up_sync(0xffffffffu, tail, 1);
            lo.pdf = __shfl_up_sync(0xffffffffu, hi.pdf, 1);
            if (lane == 0) {
                const float4 e = h.edge[c];
                lo.t = e.x;
                lo.cdf = lo.ccdf = e.y;
                lo.pdf = e.z;
            }
            hi.ccdf = tail;
            hi.cdf = past ? h.cross[c] : tail;
            float dM_mu, dM_sd;
            const float M = ring_mass(lo, hi, mc, sc, &dM_mu, &dM_sd);
            q += wc * M / Sc;
            h.v[c][lane] = M;
            h.v[kComponents + c][lane] = dM_mu;
            h.v[2 * kComponents + c][lane] = dM_sd;
            __syncwarp();  // lane 0 has read the edge
            if (lane == n - 1) h.edge[c] = make_float4(hi.t, tail, hi.pdf, 0.0f);
        }
        const float yj = lane < n ? y[j - 1] : 0.0f;
        const float qe = q + 1e-12f;
        h.v[kSums - 1][lane] = yj > 0.0f ? logf(qe) : 0.0f;
        h.c[lane] = yj > 0.0f ? yj / qe : 0.0f;
        h.ny[lane] = -yj;
        __syncwarp();
        if (lane < kSums) {
            const float *f = lane == kSums - 1 ? h.ny : h.c, *x = h.v[lane];
#pragma unroll 4
            for (int i = 0; i < n; ++i) sum = fmaf(f[i], x[i], sum);
        }
        __syncwarp();
    }
    // the category beyond r_max, component k in lane k
    {
        const float4 e = h.edge[k];
        Edge lo, hi;
        lo.t = e.x;
        lo.cdf = lo.ccdf = e.y;
        lo.pdf = e.z;
        lo.e = radial_edge(bins, bins, r_max);
        lo.inf = false;
        hi.t = 0.0f;
        hi.cdf = 1.0f;
        hi.ccdf = 0.0f;
        hi.pdf = 0.0f;
        hi.e = 0.0f;
        hi.inf = true;
        float dM_mu, dM_sd;
        const float M = ring_mass(lo, hi, mu, sd, &dM_mu, &dM_sd);
        const float part = w * M / S;
        float q = 0.0f;
#pragma unroll
        for (int c = 0; c < kComponents; ++c) q += __shfl_sync(0xffffffffu, part, c);
        const float yj = y[bins], qe = q + 1e-12f;
        const float cj = yj > 0.0f ? yj / qe : 0.0f;
        const float x = lane < kComponents ? M : lane < 2 * kComponents ? dM_mu : dM_sd;
        if (lane < kSums - 1) sum = fmaf(cj, x, sum);
        else if (lane == kSums - 1) sum = fmaf(-yj, yj > 0.0f ? logf(qe) : 0.0f, sum);
    }
    const float A1 = __shfl_sync(0xffffffffu, sum, k), Amu = __shfl_sync(0xffffffffu, sum, kComponents + k);
    const float Asd = __shfl_sync(0xffffffffu, sum, 2 * kComponents + k);
    p.rad = __shfl_sync(0xffffffffu, sum, kSums - 1);
    p.total = ld + lambda * p.rad;
    const float gw = -A1 / S;
    float wg = 0.0f;
#pragma unroll
    for (int c = 0; c < kComponents; ++c)
        wg += __shfl_sync(0xffffffffu, w, c) * __shfl_sync(0xffffffffu, gw, c);
    const float f = w / S;
    const float gmu = -f * (Amu - A1 * ring.c0 / S);
    const float gsd = -f * (Asd - A1 * ring.p0 / S);
    p.ga = lambda * w * (gw - wg);
    p.gom = lambda * dmu * gmu;
    p.gls = clamped ? 0.0f : lambda * sd * gsd;
    return p;
}

// ------------------------------------------------------------ kernels

// Normalised, zero-padded BF16 network input of one feature row.
__device__ __forceinline__ void write_input(const float *f, const float *lo, const float *inv, __nv_bfloat16 *x)
{
#pragma unroll
    for (int i = 0; i < kFeatures; ++i) x[i] = __float2bfloat16(2.0f * (f[i] - lo[i]) * inv[i] - 1.0f);
#pragma unroll
    for (int i = kFeatures; i < kInPad; ++i) x[i] = __float2bfloat16(0.0f);
}

// Training batch: rows drawn with Philox(seed, step, row) from [0, n_train),
// or the rows [first, first + b) in order when `sequential`.  One warp per
// row, its lanes across the radial categories: a thread per row walked 97
// uncoalesced counts twice (8,192 rows 34 -> 9 us).
__global__ void gather_kernel(const float *__restrict__ feat, const int32_t *__restrict__ photons,
                              const int32_t *__restrict__ detected, const uint32_t *__restrict__ radial, int bins,
                              int64_t n_train, int64_t first, int b, bool sequential, uint64_t seed,
                              const unsigned long long *step, const __grid_constant__ NormParams norm, __nv_bfloat16 *__restrict__ x0,
                              float *__restrict__ target, float *__restrict__ ylab, float *__restrict__ has_rad)
{
    const int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (r >= b) return;
    int64_t i;
    if (sequential) {
        i = first + r;
    } else {
        const uint4 h = philox10(make_uint4((uint32_t)r, (uint32_t)*step, (uint32_t)(*step >> 32), 0x5347u),
                                 (uint32_t)seed, (uint32_t)(seed >> 32));
        const unsigned long long v = ((unsigned long long)h.x << 32) | h.y;
        i = (int64_t)(v % (unsigned long long)n_train);
    }
    const uint32_t *h = radial + i * (int64_t)(bins + 1);
    // whole numbers: exact in any order
    unsigned long long n = 0;
    for (int j = lane; j <= bins; j += 32) n += h[j];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
    const double tot = (double)n;
    const float inv = tot > 0.0 ? (float)(1.0 / tot) : 0.0f;
    for (int j = lane; j <= bins; j += 32) ylab[(int64_t)r * (bins + 1) + j] = (float)h[j] * inv;
    static_assert(kInPad == 32, "one input column per lane");
    x0[(int64_t)r * kInPad + lane] = __float2bfloat16(
        lane < kFeatures ? 2.0f * (feat[i * kFeatures + lane] - norm.lo[lane & 7]) * norm.inv[lane & 7] - 1.0f : 0.0f);
    if (lane == 0) {
        const int32_t N = photons[i];
        target[r] = N > 0 ? (float)detected[i] / (float)N : 0.0f;
        has_rad[r] = tot > 0.0 ? 1.0f : 0.0f;
    }
}

// Loss (summed into acc[0..2] = total, detection, radial) and, when dout is
// set, dL/dout / b as BF16 [b][64].  A warp per row (point_loss); instruction
// issue bounds it (normal tails, exponentials and divisions of 96 x 8 bin
// masses, issue slots 78 % busy).  8,192 rows: a thread per row left 64 threads
// per SM that waited for their dependent instructions, 588 us; eight lanes per
// row 136; a warp per row with 31 categories a pass (four passes for 97) and
// both tails of each crossed edge in the pass 105 us and 88.5 M instructions,
// this 76 us and 59.4 M.
__global__ void __launch_bounds__(32 * kLossWarps) loss_kernel(const float *__restrict__ out, int ldo,
                                                               const float *__restrict__ target,
                                                               const float *__restrict__ ylab,
                                                               const float *__restrict__ has_rad, int bins,
                                                               float r_max, float lambda, int b, float scale,
                                                               __nv_bfloat16 *__restrict__ dout, double *acc)
{
    __shared__ LossShared h[kLossWarps];
    __shared__ float s[3][kLossWarps];
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31, r = blockIdx.x * kLossWarps + wid;
    PointLoss p{};
    if (r < b) {
        p = point_loss(out + (int64_t)r * ldo, target[r], ylab + (int64_t)r * (bins + 1), has_rad[r] > 0.0f, bins,
                       r_max, lambda, h[wid]);
        if (dout) {
            __nv_bfloat16 *d = dout + (int64_t)r * kOutPad;
            if (lane < kComponents) {
                if (lane == 0) d[0] = __float2bfloat16(p.gz * scale);
                d[1 + lane] = __float2bfloat16(p.ga * scale);
                d[1 + kComponents + lane] = __float2bfloat16(p.gom * scale);
                d[1 + 2 * kComponents + lane] = __float2bfloat16(p.gls * scale);
            }
            for (int i = kOutputs + lane; i < kOutPad; i += 32) d[i] = __float2bfloat16(0.0f);
        }
    }
    if (lane == 0) {
        s[0][wid] = p.total;
        s[1][wid] = p.det;
        s[2][wid] = p.rad;
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        double t = 0.0;
        for (int i = 0; i < kLossWarps; ++i) t += s[threadIdx.x][i];
        atomicAdd(&acc[threadIdx.x], t);
    }
}

// db[n] = sum_r dy[r][n] (BF16 rows), FP32 result; one block per 32 columns.
__global__ void colsum_kernel(const __nv_bfloat16 *__restrict__ dy, int ld, int rows, int cols, float *__restrict__ db)
{
    const int n = blockIdx.x * 32 + (threadIdx.x & 31);
    const int part = threadIdx.x >> 5, parts = blockDim.x >> 5;
    float s = 0.0f;
    if (n < cols)
        for (int r = part; r < rows; r += parts) s += __bfloat162float(dy[(int64_t)r * ld + n]);
    __shared__ float sh[32][33];
    sh[part][threadIdx.x & 31] = s;
    __syncthreads();
    if (part == 0 && n < cols) {
        float t = 0.0f;
        for (int p = 0; p < parts; ++p) t += sh[p][threadIdx.x & 31];
        db[n] = t;
    }
}

// Sum of split-K partials: out[i] = sum_z ws[z][i].
__global__ void split_sum_kernel(const float *__restrict__ ws, int splits, int64_t n, float *__restrict__ out)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        float s = 0.0f;
        for (int z = 0; z < splits; ++z) s += ws[(int64_t)z * n + i];
        out[i] = s;
    }
}

// The two reductions of a tcgen05 weight gradient in one launch.  Blocks
// [0, sum_blocks): out[i] = sum_z ws[z][i] (split_sum_kernel); the others:
// db[n] = sum_r dyT[n][r], a warp per column on the transposed gradient
// (rows_pad contiguous rows, zeros past the last), in the order of
// colsum_kernel: lane l the rows l, l + 32, ..., then the lanes' sums in order.
// (8,192 rows: the column sums of the untransposed gradient took 41 us on 2 or
// 8 blocks beside 6 us for the split sum; both now 12.)
__global__ void __launch_bounds__(256) finish_grad_kernel(const float *__restrict__ ws, int splits, int64_t n,
                                                          float *__restrict__ out, int sum_blocks,
                                                          const __nv_bfloat16 *__restrict__ dyT, int rows_pad,
                                                          int cols, float *__restrict__ db)
{
    if ((int)blockIdx.x < sum_blocks) {
        for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)sum_blocks * blockDim.x) {
            float s = 0.0f;
#pragma unroll 8
            for (int z = 0; z < splits; ++z) s += ws[(int64_t)z * n + i];
            out[i] = s;
        }
        return;
    }
    const int c = ((int)blockIdx.x - sum_blocks) * (int)(blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (c >= cols) return;
    const __nv_bfloat16 *p = dyT + (int64_t)c * rows_pad + lane;
    float s = 0.0f;
#pragma unroll 16
    for (int r = 0; r < rows_pad; r += 32) s += __bfloat162float(p[r]);
    float t = 0.0f;
#pragma unroll
    for (int k = 0; k < 32; ++k) t += __shfl_sync(0xffffffffu, s, k);
    if (lane == 0) db[c] = t;
}

// Adam on the FP32 masters, then the BF16 copies.  `mask` zeroes the update
// of padding entries (their gradients are zero anyway).
__global__ void adam_kernel(float *__restrict__ p, const float *__restrict__ g, float *__restrict__ m,
                            float *__restrict__ v, __nv_bfloat16 *__restrict__ pb, int64_t n, const float *lr_ptr, float b1,
                            float b2, float eps, unsigned long long *step, const uint8_t *__restrict__ live)
{
    const unsigned long long t = *step + 1;
    const float lr = *lr_ptr;
    const float c1 = 1.0f - powf(b1, (float)t), c2 = 1.0f - powf(b2, (float)t);
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        if (!live[i]) continue;
        const float gi = g[i];
        const float mi = b1 * m[i] + (1.0f - b1) * gi;
        const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        const float w = p[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
        p[i] = w;
        pb[i] = __float2bfloat16(w);
    }
}

__global__ void step_kernel(unsigned long long *step) { *step += 1; }

__global__ void to_bf16_kernel(const float *__restrict__ p, __nv_bfloat16 *__restrict__ pb, int64_t n)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        pb[i] = __float2bfloat16(p[i]);
}

// out[c][r] = in[r][c] for r < rows, 0 for rows <= r < rows_pad (BF16; in is
// [rows][ld_in], out [cols][rows_pad]), for up to three matrices (blockIdx.z).
// Feeds the tcgen05 backward products, whose operands must be contiguous along
// the contraction.  64 x 64 tiles through shared memory, 16 bytes a thread on
// both sides: ld_in, cols and rows_pad are multiples of 8 and the matrices
// 16-byte aligned.  An element at a time took 14 us for a layer's two operands
// at 8,192 rows, this 4.9.
struct TransposeArgs {
    const __nv_bfloat16 *in[3];
    __nv_bfloat16 *out[3];
    int ld_in[3], rows[3], cols[3], rows_pad[3];
};

__global__ void __launch_bounds__(256) transpose_bf16_kernel(const __grid_constant__ TransposeArgs a)
{
    // 66 elements a row: a column's reads fall on different banks
    __shared__ __nv_bfloat16 t[64][66];
    const int m = blockIdx.z, r0 = blockIdx.x * 64, c0 = blockIdx.y * 64;
    const int rows = a.rows[m], cols = a.cols[m], rows_pad = a.rows_pad[m], ld_in = a.ld_in[m];
    if (r0 >= rows_pad || c0 >= cols) return;
    const __nv_bfloat16 *in = a.in[m];
    __nv_bfloat16 *out = a.out[m];
    const int piece = (threadIdx.x & 7) * 8, line = threadIdx.x >> 3;
#pragma unroll
    for (int p = 0; p < 64; p += 32) {
        const int r = r0 + line + p, c = c0 + piece;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (r < rows && c < cols) v = *reinterpret_cast<const uint4 *>(in + (int64_t)r * ld_in + c);
        uint32_t *d = reinterpret_cast<uint32_t *>(&t[line + p][piece]);
        d[0] = v.x;
        d[1] = v.y;
        d[2] = v.z;
        d[3] = v.w;
    }
    __syncthreads();
#pragma unroll
    for (int p = 0; p < 64; p += 32) {
        const int c = c0 + line + p, r = r0 + piece;
        if (c >= cols || r >= rows_pad) continue;
        __nv_bfloat16 e[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) e[i] = t[piece + i][line + p];
        uint4 v;
        v.x = (uint32_t)__bfloat16_as_ushort(e[0]) | (uint32_t)__bfloat16_as_ushort(e[1]) << 16;
        v.y = (uint32_t)__bfloat16_as_ushort(e[2]) | (uint32_t)__bfloat16_as_ushort(e[3]) << 16;
        v.z = (uint32_t)__bfloat16_as_ushort(e[4]) | (uint32_t)__bfloat16_as_ushort(e[5]) << 16;
        v.w = (uint32_t)__bfloat16_as_ushort(e[6]) | (uint32_t)__bfloat16_as_ushort(e[7]) << 16;
        *reinterpret_cast<uint4 *>(out + (int64_t)c * rows_pad + r) = v;
    }
}

// Normalised inputs of host-given feature rows.
__global__ void input_kernel(const float *__restrict__ feat, int64_t n, const __grid_constant__ NormParams norm, __nv_bfloat16 *__restrict__ x0)
{
    for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < n; r += (int64_t)gridDim.x * blockDim.x)
        write_input(feat + r * kFeatures, norm.lo, norm.inv, x0 + r * kInPad);
}

// The network's outputs without the padding of their rows: out[r][k] =
// in[r][k], k < kOutputs, in [rows][kOutPad].
__global__ void pack_outputs_kernel(const float *__restrict__ in, int64_t n, float *__restrict__ out)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n * kOutputs; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = in[i / kOutputs * kOutPad + i % kOutputs];
}

}  // namespace sg
}  // namespace fd2

// ================================================================ host

using namespace fd2::sg;

namespace {

unsigned grid_for(int64_t n, int block, int cap = 4096)
{
    return (unsigned)std::max<int64_t>(1, std::min<int64_t>((n + block - 1) / block, cap));
}

}  // namespace

// Blocks of 256 threads with a warp per row.
static unsigned warps_for(int64_t rows) { return (unsigned)((rows + 7) / 8); }
static unsigned loss_blocks(int64_t rows) { return (unsigned)((rows + kLossWarps - 1) / kLossWarps); }

fd2_status sg_fail(fd2_sg *s, fd2_status st, const std::string &msg)
{
    if (s) s->last_error = msg;
    return st;
}

fd2_status sg_cuda(fd2_sg *s, cudaError_t e, const char *what)
{
    if (e == cudaSuccess) return FD2_OK;
    return sg_fail(s, e == cudaErrorMemoryAllocation ? FD2_ERR_OUT_OF_MEMORY : FD2_ERR_CUDA,
                   std::string(what) + ": " + cudaGetErrorString(e));
}

#define SG_CUDA(s, call)                                      \
    do {                                                      \
        cudaError_t e_ = (call);                              \
        if (e_ != cudaSuccess) return sg_cuda(s, e_, #call);  \
    } while (0)

cudaError_t sg_gemm(cudaStream_t st, bool a_kc, bool b_kc, const GemmArgs &g, int splits)
{
    dim3 grid((unsigned)((g.N + kBN - 1) / kBN), (unsigned)((g.M + kBM - 1) / kBM), (unsigned)splits);
    if (a_kc && b_kc) gemm_kernel<true, true><<<grid, kGemmThreads, 0, st>>>(g);
    else if (a_kc && !b_kc) gemm_kernel<true, false><<<grid, kGemmThreads, 0, st>>>(g);
    else if (!a_kc && !b_kc) gemm_kernel<false, false><<<grid, kGemmThreads, 0, st>>>(g);
    else return cudaErrorInvalidValue;
    return cudaGetLastError();
}

namespace {

GemmArgs gemm_args(const __nv_bfloat16 *A, int lda, const __nv_bfloat16 *B, int ldb, int M, int N, int K, int epi,
                   void *C, int ldc)
{
    GemmArgs g;
    std::memset(&g, 0, sizeof g);
    g.A = A;
    g.B = B;
    g.lda = lda;
    g.ldb = ldb;
    g.M = M;
    g.N = N;
    g.K = K;
    g.k_per_split = K;
    g.epi = epi;
    g.C = C;
    g.ldc = ldc;
    return g;
}

}  // namespace

namespace {
cudaError_t launch_tc(fd2_sg *s, cudaStream_t st, const TcArgs &t0, unsigned grid_x, unsigned grid_y);
}  // namespace

// One forward product (K-contiguous operands, bias epilogue): tcgen05 when
// the shapes fit one pass of fd2_sg_tc.cuh, else the mma.sync kernel.
static cudaError_t sg_dense(fd2_sg *s, cudaStream_t st, const GemmArgs &g)
{
    const bool tc = s->use_tc && g.K % 16 == 0 && g.K <= kTcMaxK && g.N % 16 == 0 && g.N >= 16 && g.N <= kTcMaxN &&
                    g.lda % 8 == 0 && g.ldb % 8 == 0 && g.ldc % 16 == 0 && g.M > 0;
    if (!tc) {
        if ((int64_t)g.M > (int64_t)65535 * kBM) return cudaErrorInvalidValue;  // one grid row per 64 rows
        return sg_gemm(st, true, true, g, 1);
    }
    TcArgs t{};
    t.A = g.A;
    t.B = g.B;
    t.lda = g.lda;
    t.ldb = g.ldb;
    t.M = g.M;
    t.N = g.N;
    t.K = g.K;
    t.m_limit = g.m_limit;
    t.epi = g.epi;
    t.bias = g.bias;
    t.C = g.C;
    t.ldc = g.ldc;
    t.fault = s->d_tc_fault;
    const unsigned grid = (unsigned)std::min((g.M + kTcRows - 1) / kTcRows, s->sm_count);
    return launch_tc(s, st, t, grid, 1);
}

fd2_status sg_tc_check(fd2_sg *s)
{
    if (!s || !s->d_tc_fault) return FD2_OK;
    unsigned f = 0;
    SG_CUDA(s, cudaMemcpy(&f, s->d_tc_fault, sizeof f, cudaMemcpyDeviceToHost));
    if (!f) return FD2_OK;
    SG_CUDA(s, cudaMemsetAsync(s->d_tc_fault, 0, sizeof f, s->stream));
    return sg_fail(s, FD2_ERR_DEVICE_ABORT, "a tensor-core GEMM tile gave up waiting for its MMAs");
}

// Forward pass over `rows` input rows in sg->x0 (row capacity >= rows):
// activations h1..h3 (BF16) and out (FP32 [rows][64]).
cudaError_t sg_forward(fd2_sg *s, cudaStream_t st, const __nv_bfloat16 *x0, int rows, const int *m_limit,
                       __nv_bfloat16 *h1, __nv_bfloat16 *h2, __nv_bfloat16 *h3, float *out)
{
    const int H = s->hidden;
    cudaError_t e;
    GemmArgs g = gemm_args(x0, kInPad, s->pb + s->off[kW1], kInPad, rows, H, kInPad, kEpiBiasReluBf16, h1, H);
    g.bias = s->p + s->off[kB1];
    g.m_limit = m_limit;
    if ((e = sg_dense(s, st, g)) != cudaSuccess) return e;
    g = gemm_args(h1, H, s->pb + s->off[kW2], H, rows, H, H, kEpiBiasReluBf16, h2, H);
    g.bias = s->p + s->off[kB2];
    g.m_limit = m_limit;
    if ((e = sg_dense(s, st, g)) != cudaSuccess) return e;
    g = gemm_args(h2, H, s->pb + s->off[kW3], H, rows, H, H, kEpiBiasReluBf16, h3, H);
    g.bias = s->p + s->off[kB3];
    g.m_limit = m_limit;
    if ((e = sg_dense(s, st, g)) != cudaSuccess) return e;
    g = gemm_args(h3, H, s->pb + s->off[kW4], H, rows, kOutPad, H, kEpiBiasF32, out, kOutPad);
    g.bias = s->p + s->off[kB4];
    g.m_limit = m_limit;
    return sg_dense(s, st, g);
}

namespace {

// Weight gradient dW [M][K] = dy^T x over `rows` batch rows, split-K.
cudaError_t weight_grad(fd2_sg *s, cudaStream_t st, const __nv_bfloat16 *dy, int ldy, int M, const __nv_bfloat16 *x,
                        int ldx, int K, int rows, float *dw)
{
    const int splits = std::max(1, std::min(kMaxSplits, rows / 512));
    const int per = ((rows + splits - 1) / splits + kBK - 1) / kBK * kBK;
    GemmArgs g = gemm_args(dy, ldy, x, ldx, M, K, rows, kEpiPartialF32, s->ws, K);
    g.k_per_split = per;
    g.split_stride = (long long)M * K;
    const int z = (rows + per - 1) / per;
    cudaError_t e = sg_gemm(st, false, false, g, z);
    if (e != cudaSuccess) return e;
    split_sum_kernel<<<grid_for((int64_t)M * K, 256), 256, 0, st>>>(s->ws, z, (int64_t)M * K, dw);
    return cudaGetLastError();
}

constexpr int kTcSlice = 256;  // batch rows per weight-gradient slice (the contraction of one tcgen05 pass)

int rows_pad(int rows) { return (rows + kTcSlice - 1) / kTcSlice * kTcSlice; }

// The transposes of n <= 3 matrices: {in, ld_in, rows, cols, rows_pad, out}.
struct Transpose {
    const __nv_bfloat16 *in;
    int ld_in, rows, cols, rows_pad;
    __nv_bfloat16 *out;
};

cudaError_t launch_transpose(cudaStream_t st, const Transpose *t, int n)
{
    TransposeArgs a{};
    int x = 1, y = 1;
    for (int i = 0; i < n; ++i) {
        a.in[i] = t[i].in;
        a.out[i] = t[i].out;
        a.ld_in[i] = t[i].ld_in;
        a.rows[i] = t[i].rows;
        a.cols[i] = t[i].cols;
        a.rows_pad[i] = t[i].rows_pad;
        x = std::max(x, (t[i].rows_pad + 63) / 64);
        y = std::max(y, (t[i].cols + 63) / 64);
    }
    transpose_bf16_kernel<<<dim3((unsigned)x, (unsigned)y, (unsigned)n), 256, 0, st>>>(a);
    return cudaGetLastError();
}

// The driver's cuTensorMapEncodeTiled, through the runtime (no libcuda link).
static PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder()
{
    static PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q{};
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            p = nullptr;
        return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    }();
    return fn;
}

// A 2D map of a row-major BF16 matrix (rows x cols, row stride ld elements)
// whose boxes are box_rows rows by 8 columns (16 bytes: one K column of the
// canonical no-swizzle layout) or, with sw128, by 64 columns (128 bytes,
// written with the 128-byte swizzle); rows past the matrix read as zeros.
static bool encode_map(CUtensorMap *m, const __nv_bfloat16 *base, int rows, int cols, int ld, int box_rows, bool sw128)
{
    PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
    const int box_cols = sw128 ? 64 : 8;
    if (!enc || reinterpret_cast<uintptr_t>(base) % 16 != 0 || (ld * 2) % 16 != 0 || rows < 1 || cols < box_cols ||
        box_rows < 1 || box_rows > 256)
        return false;
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    const cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
    const cuuint32_t estr[2] = {1, 1};
    return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<__nv_bfloat16 *>(base), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, sw128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

cudaError_t launch_tc(fd2_sg *s, cudaStream_t st, const TcArgs &t0, unsigned grid_x, unsigned grid_y)
{
    const dim3 grid(grid_x, grid_y);
    if (s->tc_pipe && t0.K % 16 == 0 && (t0.K <= kPipeChunkK || t0.K % kPipeChunkK == 0)) {
        // operands by TMA where the product has no batch slices and the maps
        // can be made (16-byte aligned bases and row strides), in 128-byte
        // swizzled rows where K is a multiple of 64 (the ring's chunks are
        // then 64 wide), else cp.async
        TcArgs t = t0;
        const bool sw = s->tc_sw128 && t.K % 64 == 0;
        t.tma = s->tc_tma && t.a_split == 0 && t.b_split == 0 &&
                encode_map(&t.tmap_a, t.A, t.M, t.K, t.lda, kTcRows, sw) &&
                encode_map(&t.tmap_b, t.B, t.N, t.K, t.ldb, t.N, sw);
        if (t.tma && sw) t.tma = 2;
        // the staged BF16 epilogues store whole 32-row blocks by TMA
        t.tma_store = s->tc_tma_store && (t.epi == kEpiBiasReluBf16 || t.epi == kEpiMaskBf16) && t.N % 64 == 0 &&
                      t.c_split == 0 && encode_map(&t.tmap_c, static_cast<const __nv_bfloat16 *>(t.C), t.M, t.N,
                                                   t.ldc, 32, true);
        const size_t smem = tc_pipe_smem_bytes(t.N, t.K);
        if (t.epi == kEpiBiasReluBf16) gemm_tc_pipe_kernel<kEpiBiasReluBf16><<<grid, kPipeThreads, smem, st>>>(t);
        else if (t.epi == kEpiBiasF32) gemm_tc_pipe_kernel<kEpiBiasF32><<<grid, kPipeThreads, smem, st>>>(t);
        else if (t.epi == kEpiMaskBf16) gemm_tc_pipe_kernel<kEpiMaskBf16><<<grid, kPipeThreads, smem, st>>>(t);
        else if (t.epi == kEpiPartialF32) gemm_tc_pipe_kernel<kEpiPartialF32><<<grid, kPipeThreads, smem, st>>>(t);
        else return cudaErrorInvalidValue;
        return cudaGetLastError();
    }
    const TcArgs &t = t0;
    const size_t smem = tc_smem_bytes(t.N, t.K);
    if (t.epi == kEpiBiasReluBf16) gemm_tc_kernel<kEpiBiasReluBf16><<<grid, kTcThreads, smem, st>>>(t);
    else if (t.epi == kEpiBiasF32) gemm_tc_kernel<kEpiBiasF32><<<grid, kTcThreads, smem, st>>>(t);
    else if (t.epi == kEpiMaskBf16) gemm_tc_kernel<kEpiMaskBf16><<<grid, kTcThreads, smem, st>>>(t);
    else if (t.epi == kEpiPartialF32) gemm_tc_kernel<kEpiPartialF32><<<grid, kTcThreads, smem, st>>>(t);
    else return cudaErrorInvalidValue;
    return cudaGetLastError();
}

// The backward products fit one tcgen05 pass per tile when every
// contraction (64 outputs, H hidden, 256-row batch slices) is <= 256 and
// every width a multiple of 16.
bool tc_backward(const fd2_sg *s) { return s->use_tc && s->hidden % 16 == 0 && s->hidden >= 32 && s->hidden <= kTcMaxN; }

bool tc_backward_ok(const fd2_sg *s, int rows)
{
    return tc_backward(s) && s->tA && rows > 0 && rows <= s->cap_rows;
}

// Weight gradient on tcgen05: dW [M][K] = sum over 256-row slices z of
// dy_z^T x_z, with dy^T ([M][rows_pad]) and x^T ([K][rows_pad]) staged
// contiguous along the batch; one CTA per (128-row tile of dW, slice), FP32
// partial planes summed in slice order (deterministic).
// The bias gradient (column sums of dy) comes with it.
// On the layer's own stream and buffers, after what `st` holds: nothing of the
// backward pass waits for it before its end, so the layers' weight gradients
// run beside the chain of input gradients (8,192 rows: 64 CTAs a launch on 148
// SMs).
cudaError_t weight_grad_tc(fd2_sg *s, cudaStream_t main, int layer, const __nv_bfloat16 *dy, int ldy, int M,
                           const __nv_bfloat16 *x, int ldx, int K, int rows, float *dw, float *db)
{
    cudaError_t e;
    cudaStream_t st = s->side[layer];
    __nv_bfloat16 *tA = s->tA + layer * s->t_stride, *tB = s->tB + layer * s->t_stride;
    float *ws = s->ws + layer * s->ws_floats;
    const int rp = rows_pad(rows), z = rp / kTcSlice;
    if ((int64_t)z * M * K > s->ws_floats || (int64_t)std::max(M, K) * rp > s->t_stride) return cudaErrorInvalidValue;
    if ((e = cudaEventRecord(s->ev_main[layer], main)) != cudaSuccess) return e;
    if ((e = cudaStreamWaitEvent(st, s->ev_main[layer], 0)) != cudaSuccess) return e;
    const Transpose t2[2] = {{dy, ldy, rows, M, rp, tA}, {x, ldx, rows, K, rp, tB}};
    if ((e = launch_transpose(st, t2, 2)) != cudaSuccess) return e;
    TcArgs t{};
    t.A = tA;
    t.B = tB;
    t.lda = rp;
    t.ldb = rp;
    t.M = M;
    t.N = K;
    t.K = kTcSlice;
    t.epi = kEpiPartialF32;
    t.C = ws;
    t.ldc = K;
    t.a_split = kTcSlice;
    t.b_split = kTcSlice;
    t.c_split = (long long)M * K;
    t.fault = s->d_tc_fault;
    if ((e = launch_tc(s, st, t, (unsigned)((M + kTcRows - 1) / kTcRows), (unsigned)z)) != cudaSuccess) return e;
    const unsigned sums = grid_for((int64_t)M * K, 256);
    finish_grad_kernel<<<sums + (unsigned)((M + 7) / 8), 256, 0, st>>>(ws, z, (int64_t)M * K, dw, (int)sums, tA,
                                                                       rp, M, db);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    return cudaEventRecord(s->ev_side[layer], st);
}

// Input gradient on tcgen05: d [rows][H] = (dy [rows][Nout] W [Nout][H]) *
// (h > 0), with W^T ([H][Nout]) as the K-contiguous second operand.
cudaError_t input_grad_tc(fd2_sg *s, cudaStream_t st, const __nv_bfloat16 *dy, int Nout, const __nv_bfloat16 *wT,
                          const __nv_bfloat16 *h, int rows, __nv_bfloat16 *d)
{
    const int H = s->hidden;
    TcArgs t{};
    t.A = dy;
    t.B = wT;
    t.lda = Nout;
    t.ldb = Nout;
    t.M = rows;
    t.N = H;
    t.K = Nout;
    t.epi = kEpiMaskBf16;
    t.mask = h;
    t.ldm = H;
    t.C = d;
    t.ldc = H;
    t.fault = s->d_tc_fault;
    return launch_tc(s, st, t, (unsigned)std::min((rows + kTcRows - 1) / kTcRows, s->sm_count), 1);
}

// Backward pass from dout (BF16 [rows][64], already scaled by 1/rows).
cudaError_t backward(fd2_sg *s, cudaStream_t st, int rows)
{
    const int H = s->hidden;
    cudaError_t e;
    float *G = s->g;
    if (tc_backward_ok(s, rows)) {
        // the weights' transposes (BF16 copies of this step's parameters)
        __nv_bfloat16 *w2T = s->pbT, *w3T = s->pbT + (size_t)H * H, *w4T = s->pbT + 2 * (size_t)H * H;
        const Transpose tw[3] = {{s->pb + s->off[kW4], H, kOutPad, H, kOutPad, w4T},
                                 {s->pb + s->off[kW3], H, H, H, H, w3T},
                                 {s->pb + s->off[kW2], H, H, H, H, w2T}};
        if ((e = launch_transpose(st, tw, 3)) != cudaSuccess) return e;
        // layer 4
        if ((e = weight_grad_tc(s, st, 3, s->dout, kOutPad, kOutPad, s->h3, H, H, rows, G + s->off[kW4],
                                G + s->off[kB4])) != cudaSuccess)
            return e;
        if ((e = input_grad_tc(s, st, s->dout, kOutPad, w4T, s->h3, rows, s->d3)) != cudaSuccess) return e;
        // layer 3
        if ((e = weight_grad_tc(s, st, 2, s->d3, H, H, s->h2, H, H, rows, G + s->off[kW3], G + s->off[kB3])) != cudaSuccess)
            return e;
        if ((e = input_grad_tc(s, st, s->d3, H, w3T, s->h2, rows, s->d2)) != cudaSuccess) return e;
        // layer 2
        if ((e = weight_grad_tc(s, st, 1, s->d2, H, H, s->h1, H, H, rows, G + s->off[kW2], G + s->off[kB2])) != cudaSuccess)
            return e;
        if ((e = input_grad_tc(s, st, s->d2, H, w2T, s->h1, rows, s->d1)) != cudaSuccess) return e;
        // layer 1
        if ((e = weight_grad_tc(s, st, 0, s->d1, H, H, s->x0, kInPad, kInPad, rows, G + s->off[kW1],
                                G + s->off[kB1])) != cudaSuccess)
            return e;
        for (cudaEvent_t ev : s->ev_side)
            if ((e = cudaStreamWaitEvent(st, ev, 0)) != cudaSuccess) return e;
        return cudaSuccess;
    }
    // layer 4
    if ((e = weight_grad(s, st, s->dout, kOutPad, kOutPad, s->h3, H, H, rows, G + s->off[kW4])) != cudaSuccess)
        return e;
    colsum_kernel<<<(kOutPad + 31) / 32, 1024, 0, st>>>(s->dout, kOutPad, rows, kOutPad, G + s->off[kB4]);
    GemmArgs g = gemm_args(s->dout, kOutPad, s->pb + s->off[kW4], H, rows, H, kOutPad, kEpiMaskBf16, s->d3, H);
    g.mask = s->h3;
    g.ldm = H;
    if ((e = sg_gemm(st, true, false, g, 1)) != cudaSuccess) return e;
    // layer 3
    if ((e = weight_grad(s, st, s->d3, H, H, s->h2, H, H, rows, G + s->off[kW3])) != cudaSuccess) return e;
    colsum_kernel<<<(H + 31) / 32, 1024, 0, st>>>(s->d3, H, rows, H, G + s->off[kB3]);
    g = gemm_args(s->d3, H, s->pb + s->off[kW3], H, rows, H, H, kEpiMaskBf16, s->d2, H);
    g.mask = s->h2;
    g.ldm = H;
    if ((e = sg_gemm(st, true, false, g, 1)) != cudaSuccess) return e;
    // layer 2
    if ((e = weight_grad(s, st, s->d2, H, H, s->h1, H, H, rows, G + s->off[kW2])) != cudaSuccess) return e;
    colsum_kernel<<<(H + 31) / 32, 1024, 0, st>>>(s->d2, H, rows, H, G + s->off[kB2]);
    g = gemm_args(s->d2, H, s->pb + s->off[kW2], H, rows, H, H, kEpiMaskBf16, s->d1, H);
    g.mask = s->h1;
    g.ldm = H;
    if ((e = sg_gemm(st, true, false, g, 1)) != cudaSuccess) return e;
    // layer 1
    if ((e = weight_grad(s, st, s->d1, H, H, s->x0, kInPad, kInPad, rows, G + s->off[kW1])) != cudaSuccess) return e;
    colsum_kernel<<<(H + 31) / 32, 1024, 0, st>>>(s->d1, H, rows, H, G + s->off[kB1]);
    return cudaGetLastError();
}

// One training step on s->batch rows (everything on the device).
cudaError_t train_step(fd2_sg *s, cudaStream_t st)
{
    const int B = s->batch, bins = s->bins;
    cudaError_t e;
    gather_kernel<<<warps_for(B), 256, 0, st>>>(s->d_feat, s->d_photons, s->d_detected, s->d_radial, bins,
                                                    s->n_train, 0, B, false, s->seed, s->d_step, s->norm, s->x0,
                                                    s->target, s->ylab, s->has_rad);
    if ((e = sg_forward(s, st, s->x0, B, nullptr, s->h1, s->h2, s->h3, s->out)) != cudaSuccess) return e;
    loss_kernel<<<loss_blocks(B), 32 * kLossWarps, 0, st>>>(s->out, kOutPad, s->target, s->ylab, s->has_rad, bins,
                                                  (float)s->radial_max, s->lambda, B, 1.0f / (float)B,
                                                  s->dout, s->d_acc);
    if ((e = backward(s, st, B)) != cudaSuccess) return e;
    adam_kernel<<<grid_for(s->n_params, 256), 256, 0, st>>>(s->p, s->g, s->m, s->v, s->pb, s->n_params, s->d_lr,
                                                            s->beta1, s->beta2, s->eps, s->d_step, s->d_live);
    step_kernel<<<1, 1, 0, st>>>(s->d_step);
    return cudaGetLastError();
}

void layout(fd2_sg *s)
{
    const int64_t H = s->hidden;
    int64_t o = 0;
    auto put = [&](int idx, int64_t n) {
        s->off[idx] = o;
        o += (n + 63) / 64 * 64;  // keep every block 128-byte aligned in BF16
    };
    put(kW1, H * kInPad);
    put(kB1, H);
    put(kW2, H * H);
    put(kB2, H);
    put(kW3, H * H);
    put(kB3, H);
    put(kW4, (int64_t)kOutPad * H);
    put(kB4, kOutPad);
    s->n_params = o;
}

// Which master entries are real parameters (not padding).
std::vector<uint8_t> live_mask(const fd2_sg *s)
{
    const int64_t H = s->hidden;
    std::vector<uint8_t> live((size_t)s->n_params, 0);
    for (int64_t r = 0; r < H; ++r)
        for (int c = 0; c < kFeatures; ++c) live[(size_t)(s->off[kW1] + r * kInPad + c)] = 1;
    for (int64_t i = 0; i < H; ++i) {
        live[(size_t)(s->off[kB1] + i)] = 1;
        live[(size_t)(s->off[kB2] + i)] = 1;
        live[(size_t)(s->off[kB3] + i)] = 1;
    }
    for (int64_t i = 0; i < H * H; ++i) {
        live[(size_t)(s->off[kW2] + i)] = 1;
        live[(size_t)(s->off[kW3] + i)] = 1;
    }
    for (int r = 0; r < kOutputs; ++r) {
        for (int64_t c = 0; c < H; ++c) live[(size_t)(s->off[kW4] + r * H + c)] = 1;
        live[(size_t)(s->off[kB4] + r)] = 1;
    }
    return live;
}

// Public parameter order (no padding) <-> master layout.
template <class F>
void for_each_public(const fd2_sg *s, F f)
{
    const int64_t H = s->hidden;
    int64_t k = 0;
    for (int64_t r = 0; r < H; ++r)
        for (int c = 0; c < kFeatures; ++c) f(k++, s->off[kW1] + r * kInPad + c);
    for (int64_t i = 0; i < H; ++i) f(k++, s->off[kB1] + i);
    for (int64_t i = 0; i < H * H; ++i) f(k++, s->off[kW2] + i);
    for (int64_t i = 0; i < H; ++i) f(k++, s->off[kB2] + i);
    for (int64_t i = 0; i < H * H; ++i) f(k++, s->off[kW3] + i);
    for (int64_t i = 0; i < H; ++i) f(k++, s->off[kB3] + i);
    for (int r = 0; r < kOutputs; ++r)
        for (int64_t c = 0; c < H; ++c) f(k++, s->off[kW4] + r * H + c);
    for (int r = 0; r < kOutputs; ++r) f(k++, s->off[kB4] + r);
}

int64_t public_count(const fd2_sg *s)
{
    const int64_t H = s->hidden;
    return H * kFeatures + H + 2 * (H * H + H) + kOutputs * H + kOutputs;
}

void set_norm(fd2_sg *s)
{
    for (int i = 0; i < kFeatures; ++i) {
        s->norm.lo[i] = s->norm_box.lo[i];
        const float span = s->norm_box.hi[i] - s->norm_box.lo[i];
        s->norm.inv[i] = span > 0.0f ? 1.0f / span : 0.5f;  // constant feature -> 0 after 2(f-lo)*inv - 1 + 1
    }
}

// Uploads go through the surrogate's stream.  It does not wait for the default
// stream, on which a copy from pageable memory may still be under way when
// cudaMemcpy returns: a kernel of the stream could read what was there before.
cudaError_t upload(fd2_sg *s, void *dst, const void *src, size_t bytes)
{
    return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s->stream);
}

template <class T>
cudaError_t alloc(T **p, size_t n)
{
    if (*p) cudaFree(*p);
    *p = nullptr;
    return cudaMalloc((void **)p, sizeof(T) * std::max<size_t>(n, 1));
}

fd2_status upload_params(fd2_sg *s, const std::vector<float> &master)
{
    SG_CUDA(s, cudaSetDevice(s->device));
    SG_CUDA(s, upload(s, s->p, master.data(), sizeof(float) * master.size()));
    to_bf16_kernel<<<grid_for(s->n_params, 256), 256, 0, s->stream>>>(s->p, s->pb, s->n_params);
    SG_CUDA(s, cudaGetLastError());
    SG_CUDA(s, cudaMemsetAsync(s->m, 0, sizeof(float) * s->n_params, s->stream));
    SG_CUDA(s, cudaMemsetAsync(s->v, 0, sizeof(float) * s->n_params, s->stream));
    SG_CUDA(s, cudaMemsetAsync(s->d_step, 0, sizeof(unsigned long long), s->stream));
    SG_CUDA(s, cudaStreamSynchronize(s->stream));
    return FD2_OK;
}

// Activation buffers for `rows` rows.
fd2_status ensure_rows(fd2_sg *s, int rows)
{
    if (rows <= s->cap_rows) return FD2_OK;
    const size_t H = (size_t)s->hidden, R = (size_t)rows;
    const size_t plane = std::max<size_t>(H * H, (size_t)kOutPad * H);
    if (tc_backward(s)) {
        // transposed operands over the rows padded to 256, and one FP32 partial
        // plane per 256-row slice, for each layer: the four weight gradients run
        // side by side (at most 256 hidden units; 8,192 rows: 34 + 34 MB)
        const size_t RP = (size_t)rows_pad(rows), ts = std::max<size_t>(H, kOutPad) * RP;
        SG_CUDA(s, alloc(&s->tA, 4 * ts));
        SG_CUDA(s, alloc(&s->tB, 4 * ts));
        s->t_stride = (int64_t)ts;
        s->ws_floats = (int64_t)(std::max<size_t>((size_t)kMaxSplits, RP / kTcSlice) * plane);
        SG_CUDA(s, alloc(&s->ws, 4 * (size_t)s->ws_floats));
    } else {
        // the layers one after another, at most kMaxSplits partial planes
        s->ws_floats = (int64_t)(kMaxSplits * plane);
        SG_CUDA(s, alloc(&s->ws, (size_t)s->ws_floats));
    }
    SG_CUDA(s, alloc(&s->x0, R * kInPad));
    SG_CUDA(s, alloc(&s->h1, R * H));
    SG_CUDA(s, alloc(&s->h2, R * H));
    SG_CUDA(s, alloc(&s->h3, R * H));
    SG_CUDA(s, alloc(&s->d1, R * H));
    SG_CUDA(s, alloc(&s->d2, R * H));
    SG_CUDA(s, alloc(&s->d3, R * H));
    SG_CUDA(s, alloc(&s->out, R * kOutPad));
    SG_CUDA(s, alloc(&s->dout, R * kOutPad));
    SG_CUDA(s, alloc(&s->target, R));
    SG_CUDA(s, alloc(&s->has_rad, R));
    SG_CUDA(s, alloc(&s->ylab, R * (size_t)(s->bins + 1)));
    s->cap_rows = rows;
    if (s->graph) cudaGraphExecDestroy(s->graph);
    s->graph = nullptr;
    return FD2_OK;
}

}  // namespace

extern "C" {

void fd2_sg_default_config(fd2_sg_config *c)
{
    if (!c) return;
    std::memset(c, 0, sizeof *c);
    c->device = 0;
    c->hidden = 256;
    c->radial_bins = 96;
    c->radial_max_um = 400.0;
    c->batch = 8192;
    c->lr = 1e-3f;
    c->beta1 = 0.9f;
    c->beta2 = 0.999f;
    c->adam_eps = 1e-8f;
    c->radial_weight = 1.0f;
    c->lateral_um = 50.0f;
    c->seed = 0x5347fd2ull;
    c->depth_margin_um = 1.0f;
}

const char *fd2_sg_last_error(const fd2_sg *s) { return s ? s->last_error.c_str() : "no surrogate"; }

fd2_status fd2_sg_create(const fd2_sg_config *cfg, fd2_sg **out)
{
    if (!out) return FD2_ERR_INVALID_ARGUMENT;
    *out = nullptr;
    fd2_sg_config c;
    if (cfg) c = *cfg;
    else fd2_sg_default_config(&c);
    if (c.hidden < 64 || c.hidden % 64 || c.hidden > 1024 || c.radial_bins < 1 || c.radial_bins > 1024 ||
        !(c.radial_max_um > 0) || c.batch < 64 || c.batch % 64 || c.batch > (1 << 20) || !(c.lr > 0) ||
        !(c.lateral_um >= 0) || !(c.depth_margin_um >= 0))
        return FD2_ERR_INVALID_ARGUMENT;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev <= 0) return FD2_ERR_NO_DEVICE;
    if (c.device < 0 || c.device >= ndev) return FD2_ERR_INVALID_ARGUMENT;
    fd2_sg *s = new fd2_sg();
    s->device = c.device;
    s->hidden = c.hidden;
    s->bins = c.radial_bins;
    s->radial_max = c.radial_max_um;
    s->batch = c.batch;
    s->lr = c.lr;
    s->beta1 = c.beta1;
    s->beta2 = c.beta2;
    s->eps = c.adam_eps;
    s->lambda = c.radial_weight;
    s->lateral_um = c.lateral_um;
    s->depth_margin_um = c.depth_margin_um;
    s->seed = c.seed;
    for (int i = 0; i < kFeatures; ++i) {
        s->hull.lo[i] = 0.0f;
        s->hull.hi[i] = 1.0f;
        s->norm_box.lo[i] = 0.0f;
        s->norm_box.hi[i] = 1.0f;
    }
    set_norm(s);
    auto bail = [&](fd2_status st) {
        fd2_sg_destroy(s);
        return st;
    };
    if (cudaSetDevice(s->device) != cudaSuccess) return bail(FD2_ERR_CUDA);
    if (cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking) != cudaSuccess) return bail(FD2_ERR_CUDA);
    for (int l = 0; l < 4; ++l)
        if (cudaStreamCreateWithFlags(&s->side[l], cudaStreamNonBlocking) != cudaSuccess ||
            cudaEventCreateWithFlags(&s->ev_main[l], cudaEventDisableTiming) != cudaSuccess ||
            cudaEventCreateWithFlags(&s->ev_side[l], cudaEventDisableTiming) != cudaSuccess)
            return bail(FD2_ERR_CUDA);
    layout(s);
    const size_t P = (size_t)s->n_params;
    if (alloc(&s->p, P) || alloc(&s->g, P) || alloc(&s->m, P) || alloc(&s->v, P) || alloc(&s->pb, P) ||
        alloc(&s->d_live, P) || alloc(&s->d_step, 1) || alloc(&s->d_acc, 4) || alloc(&s->d_lr, 1) ||
        alloc(&s->pbT, 2 * (size_t)s->hidden * s->hidden + (size_t)s->hidden * kOutPad))
        return bail(FD2_ERR_OUT_OF_MEMORY);
    if (upload(s, s->d_lr, &s->lr, sizeof(float)) != cudaSuccess) return bail(FD2_ERR_CUDA);
    if (alloc(&s->d_tc_fault, 1) || cudaMemsetAsync(s->d_tc_fault, 0, sizeof(unsigned), s->stream) != cudaSuccess)
        return bail(FD2_ERR_OUT_OF_MEMORY);
    {
        int sms = 0;
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, s->device) == cudaSuccess && sms > 0)
            s->sm_count = sms;
        const char *env = std::getenv("FD2_SG_GEMM");
        s->use_tc = !(env && std::strcmp(env, "mma") == 0);
        s->tc_pipe = !(env && std::strcmp(env, "tc1") == 0);
        s->tc_tma = !(env && std::strcmp(env, "cpasync") == 0);
        s->tc_sw128 = !(env && std::strcmp(env, "noswizzle") == 0);
        s->tc_tma_store = !(env && std::strcmp(env, "nostore") == 0);
        // the tcgen05 kernels' shared memory (outside any stream capture)
        const int bytes = (int)tc_smem_bytes(kTcMaxN, kTcMaxK);
        if (cudaFuncSetAttribute(gemm_tc_kernel<kEpiBiasReluBf16>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) !=
                cudaSuccess ||
            cudaFuncSetAttribute(gemm_tc_kernel<kEpiBiasF32>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) !=
                cudaSuccess ||
            cudaFuncSetAttribute(gemm_tc_kernel<kEpiMaskBf16>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) !=
                cudaSuccess ||
            cudaFuncSetAttribute(gemm_tc_kernel<kEpiPartialF32>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) !=
                cudaSuccess)
            return bail(FD2_ERR_CUDA);
        const int pbytes = (int)tc_pipe_smem_bytes(kTcMaxN, kTcMaxK);
        if (cudaFuncSetAttribute(gemm_tc_pipe_kernel<kEpiBiasReluBf16>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 pbytes) != cudaSuccess ||
            cudaFuncSetAttribute(gemm_tc_pipe_kernel<kEpiBiasF32>, cudaFuncAttributeMaxDynamicSharedMemorySize, pbytes) !=
                cudaSuccess ||
            cudaFuncSetAttribute(gemm_tc_pipe_kernel<kEpiMaskBf16>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 pbytes) != cudaSuccess ||
            cudaFuncSetAttribute(gemm_tc_pipe_kernel<kEpiPartialF32>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 pbytes) != cudaSuccess)
            return bail(FD2_ERR_CUDA);
    }
    const std::vector<uint8_t> live = live_mask(s);
    if (upload(s, s->d_live, live.data(), P) != cudaSuccess) return bail(FD2_ERR_CUDA);
    if (cudaMemsetAsync(s->g, 0, sizeof(float) * P, s->stream) != cudaSuccess) return bail(FD2_ERR_CUDA);
    // He-normal weights (Box-Muller on a splitmix64 stream), small last
    // layer, zero biases; mixture biases spread the components in radius
    // and width.
    std::vector<float> master(P, 0.0f);
    uint64_t st = c.seed ^ 0x9E3779B97F4A7C15ull;
    auto next = [&]() {
        st += 0x9E3779B97F4A7C15ull;
        uint64_t z = st;
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        z ^= z >> 31;
        return ((z >> 11) + 0.5) * (1.0 / 9007199254740992.0);
    };
    auto gauss = [&]() { return std::sqrt(-2.0 * std::log(next())) * std::cos(6.283185307179586 * next()); };
    const int64_t H = s->hidden;
    for (int64_t r = 0; r < H; ++r)
        for (int cc = 0; cc < kFeatures; ++cc)
            master[(size_t)(s->off[kW1] + r * kInPad + cc)] = (float)(gauss() * std::sqrt(2.0 / kFeatures));
    for (int64_t i = 0; i < H * H; ++i) {
        master[(size_t)(s->off[kW2] + i)] = (float)(gauss() * std::sqrt(2.0 / H));
        master[(size_t)(s->off[kW3] + i)] = (float)(gauss() * std::sqrt(2.0 / H));
    }
    for (int r = 0; r < kOutputs; ++r)
        for (int64_t cc = 0; cc < H; ++cc) master[(size_t)(s->off[kW4] + r * H + cc)] = (float)(gauss() * 0.01);
    for (int k = 0; k < kComponents; ++k) {
        const double mu0 = (2.5 + 7.5 * k) / kMuScale;                                          // 2.5 .. 55 um
        master[(size_t)(s->off[kB4] + 1 + kComponents + k)] = (float)std::log(std::expm1(mu0));  // softplus^-1
        master[(size_t)(s->off[kB4] + 1 + 2 * kComponents + k)] = std::log(0.2f + 0.4f * k);  // sd: 2 .. 30 um
    }
    fd2_status r = upload_params(s, master);
    if (r != FD2_OK) return bail(r);
    *out = s;
    return FD2_OK;
}

void fd2_sg_destroy(fd2_sg *s)
{
    if (!s) return;
    cudaSetDevice(s->device);
    if (s->stream) cudaStreamSynchronize(s->stream);
    for (int l = 0; l < 4; ++l) {
        if (s->side[l]) cudaStreamSynchronize(s->side[l]);
        if (s->side[l]) cudaStreamDestroy(s->side[l]);
        if (s->ev_main[l]) cudaEventDestroy(s->ev_main[l]);
        if (s->ev_side[l]) cudaEventDestroy(s->ev_side[l]);
    }
    if (s->graph) cudaGraphExecDestroy(s->graph);
    for (void *p : {(void *)s->p, (void *)s->g, (void *)s->m, (void *)s->v, (void *)s->pb, (void *)s->d_live,
                    (void *)s->d_step, (void *)s->d_acc, (void *)s->d_lr, (void *)s->ws, (void *)s->x0, (void *)s->h1, (void *)s->h2,
                    (void *)s->h3, (void *)s->d1, (void *)s->d2, (void *)s->d3, (void *)s->out, (void *)s->dout,
                    (void *)s->target, (void *)s->has_rad, (void *)s->ylab, (void *)s->d_feat, (void *)s->d_photons,
                    (void *)s->d_detected, (void *)s->d_radial, (void *)s->d_tc_fault, (void *)s->pbT, (void *)s->pout, (void *)s->tA,
                    (void *)s->tB})
        if (p) cudaFree(p);
    sg_free_run_buffers(s);
    if (s->stream) cudaStreamDestroy(s->stream);
    delete s;
}

int64_t fd2_sg_num_params(const fd2_sg *s) { return s ? public_count(s) : 0; }

fd2_status fd2_sg_set_lr(fd2_sg *s, float lr)
{
    if (!s || !(lr > 0.0f) || !std::isfinite(lr)) return FD2_ERR_INVALID_ARGUMENT;
    SG_CUDA(s, cudaSetDevice(s->device));
    SG_CUDA(s, cudaStreamSynchronize(s->stream));
    s->lr = lr;
    SG_CUDA(s, upload(s, s->d_lr, &s->lr, sizeof(float)));
    SG_CUDA(s, cudaStreamSynchronize(s->stream));
    return FD2_OK;
}

fd2_status fd2_sg_get_params(fd2_sg *s, float *params, int64_t n)
{
    if (!s || !params || n < public_count(s)) return FD2_ERR_INVALID_ARGUMENT;
    std::vector<float> master((size_t)s->n_params);
    SG_CUDA(s, cudaSetDevice(s->device));
    SG_CUDA(s, cudaStreamSynchronize(s->stream));
    SG_CUDA(s, cudaMemcpy(master.data(), s->p, sizeof(float) * master.size(), cudaMemcpyDeviceToHost));
    for_each_public(s, [&](int64_t k, int64_t i) { params[k] = master[(size_t)i]; });
    return FD2_OK;
}

fd2_status fd2_sg_set_params(fd2_sg *s, const float *params, int64_t n)
{
    if (!s || !params || n < public_count(s)) return FD2_ERR_INVALID_ARGUMENT;
    std::vector<float> master((size_t)s->n_params, 0.0f);
    for_each_public(s, [&](int64_t k, int64_t i) { master[(size_t)i] = params[k]; });
    return upload_params(s, master);
}

fd2_status fd2_sg_get_hull(fd2_sg *s, fd2_sg_hull *h)
{
    if (!s || !h) return FD2_ERR_INVALID_ARGUMENT;
    *h = s->hull;
    return FD2_OK;
}

fd2_status fd2_sg_set_edge(fd2_sg *s, float amplitude, float length_um)
{
    if (!s || !(amplitude >= 0.0f && amplitude < 1.0f) || !(length_um > 0.0f) || !std::isfinite(length_um))
        return FD2_ERR_INVALID_ARGUMENT;
    s->edge_amp = amplitude;
    s->edge_len_um = length_um;
    return FD2_OK;
}

fd2_status fd2_sg_get_edge(const fd2_sg *s, float *amplitude, float *length_um)
{
    if (!s || !amplitude || !length_um) return FD2_ERR_INVALID_ARGUMENT;
    *amplitude = s->edge_amp;
    *length_um = s->edge_len_um;
    return FD2_OK;
}

fd2_status fd2_sg_set_hull(fd2_sg *s, const fd2_sg_hull *h)
{
    if (!s || !h) return FD2_ERR_INVALID_ARGUMENT;
    for (int i = 0; i < kFeatures; ++i)
        if (!(std::isfinite(h->lo[i]) && std::isfinite(h->hi[i]) && h->hi[i] >= h->lo[i]))
            return FD2_ERR_INVALID_ARGUMENT;
    s->hull = *h;
    if (!s->norm_fixed) {
        // the network's input normalisation comes from its first hull and
        // stays with the network (later hulls only change the routing)
        s->norm_box = *h;
        s->norm_fixed = true;
        set_norm(s);
    }
    if (s->graph) cudaGraphExecDestroy(s->graph);
    s->graph = nullptr;
    return FD2_OK;
}

fd2_status fd2_sg_set_data(fd2_sg *s, const float *features, const int32_t *photons, const int32_t *detected,
                           const uint32_t *radial, int64_t n, int64_t n_val)
{
    if (!s || !features || !photons || !detected || !radial || n <= 0 || n_val < 0 || n_val >= n)
        return FD2_ERR_INVALID_ARGUMENT;
    for (int64_t i = 0; i < n; ++i) {
        if (photons[i] < 0 || detected[i] < 0 || detected[i] > photons[i])
            return sg_fail(s, FD2_ERR_INVALID_ARGUMENT, "label counts out of range");
        for (int f = 0; f < kFeatures; ++f)
            if (!std::isfinite(features[i * kFeatures + f]))
                return sg_fail(s, FD2_ERR_INVALID_ARGUMENT, "non-finite feature");
    }
    // hull = box of the training points
    fd2_sg_hull h;
    for (int f = 0; f < kFeatures; ++f) {
        h.lo[f] = features[f];
        h.hi[f] = features[f];
    }
    const int64_t n_train = n - n_val;
    for (int64_t i = 0; i < n_train; ++i)
        for (int f = 0; f < kFeatures; ++f) {
            h.lo[f] = std::min(h.lo[f], features[i * kFeatures + f]);
            h.hi[f] = std::max(h.hi[f], features[i * kFeatures + f]);
        }
    fd2_status st = fd2_sg_set_hull(s, &h);
    if (st != FD2_OK) return st;
    const size_t N = (size_t)n, nb = (size_t)(s->bins + 1);
    SG_CUDA(s, cudaSetDevice(s->device));
    SG_CUDA(s, alloc(&s->d_feat, N * kFeatures));
    SG_CUDA(s, alloc(&s->d_photons, N));
    SG_CUDA(s, alloc(&s->d_detected, N));
    SG_CUDA(s, alloc(&s->d_radial, N * nb));
    SG_CUDA(s, upload(s, s->d_feat, features, sizeof(float) * N * kFeatures));
    SG_CUDA(s, upload(s, s->d_photons, photons, sizeof(int32_t) * N));
    SG_CUDA(s, upload(s, s->d_detected, detected, sizeof(int32_t) * N));
    SG_CUDA(s, upload(s, s->d_radial, radial, sizeof(uint32_t) * N * nb));
    SG_CUDA(s, cudaStreamSynchronize(s->stream));  // the arrays are the caller's
    s->n_points = n;
    s->n_train = n_train;
    s->n_val = n_val;
    return ensure_rows(s, s->batch);
}

fd2_status fd2_sg_eval(fd2_sg *s, float *loss, float *det_loss, float *radial_loss)
{
    if (!s || s->n_points <= 0) return FD2_ERR_STATE;
    SG_CUDA(s, cudaSetDevice(s->device));
    const int64_t first = s->n_val > 0 ? s->n_train : 0;
    const int64_t count = s->n_val > 0 ? s->n_val : s->n_points;
    fd2_status st = ensure_rows(s, s->batch);
    if (st != FD2_OK) return st;
    SG_CUDA(s, cudaMemsetAsync(s->d_acc, 0, sizeof(double) * 4, s->stream));
    for (int64_t at = 0; at < count; at += s->batch) {
        const int b = (int)std::min<int64_t>(s->batch, count - at);
        gather_kernel<<<warps_for(b), 256, 0, s->stream>>>(s->d_feat, s->d_photons, s->d_detected, s->d_radial,
                                                               s->bins, s->n_train, first + at, b, true, s->seed,
                                                               s->d_step, s->norm, s->x0, s->target, s->ylab,
                                                               s->has_rad);
        SG_CUDA(s, sg_forward(s, s->stream, s->x0, b, nullptr, s->h1, s->h2, s->h3, s->out));
        loss_kernel<<<loss_blocks(b), 32 * kLossWarps, 0, s->stream>>>(s->out, kOutPad, s->target, s->ylab, s->has_rad,
                                                             s->bins, (float)s->radial_max, s->lambda, b,
                                                             1.0f, nullptr, s->d_acc);
        SG_CUDA(s, cudaGetLastError());
    }
    double acc[4];
    SG_CUDA(s, cudaMemcpyAsync(acc, s->d_acc, sizeof acc, cudaMemcpyDeviceToHost, s->stream));
    SG_CUDA(s, cudaStreamSynchronize(s->stream));
    if ((st = sg_tc_check(s)) != FD2_OK) return st;
    if (loss) *loss = (float)(acc[0] / (double)count);
    if (det_loss) *det_loss = (float)(acc[1] / (double)count);
    if (radial_loss) *radial_loss = (float)(acc[2] / (double)count);
    return FD2_OK;
}

fd2_status fd2_sg_train(fd2_sg *s, int32_t steps, float *train_loss, float *val_loss)
{
    if (!s || steps < 0) return FD2_ERR_INVALID_ARGUMENT;
    if (s->n_train <= 0) return sg_fail(s, FD2_ERR_STATE, "no training data");
    SG_CUDA(s, cudaSetDevice(s->device));
    fd2_status st = ensure_rows(s, s->batch);
    if (st != FD2_OK) return st;
    if (!s->graph) {
        cudaGraph_t gr = nullptr;
        SG_CUDA(s, cudaStreamBeginCapture(s->stream, cudaStreamCaptureModeThreadLocal));
        cudaError_t e = train_step(s, s->stream);
        cudaError_t e2 = cudaStreamEndCapture(s->stream, &gr);
        if (e != cudaSuccess || e2 != cudaSuccess) {
            if (gr) cudaGraphDestroy(gr);
            return sg_cuda(s, e != cudaSuccess ? e : e2, "capture training step");
        }
        e = cudaGraphInstantiate(&s->graph, gr, 0);
        cudaGraphDestroy(gr);
        SG_CUDA(s, e);
    }
    // the mean loss of the last min(steps, 50) steps
    const int tail = std::min(steps, 50);
    for (int i = 0; i < steps; ++i) {
        if (i == steps - tail) SG_CUDA(s, cudaMemsetAsync(s->d_acc, 0, sizeof(double) * 4, s->stream));
        SG_CUDA(s, cudaGraphLaunch(s->graph, s->stream));
    }
    double acc[4] = {0, 0, 0, 0};
    SG_CUDA(s, cudaMemcpyAsync(acc, s->d_acc, sizeof acc, cudaMemcpyDeviceToHost, s->stream));
    SG_CUDA(s, cudaStreamSynchronize(s->stream));
    if ((st = sg_tc_check(s)) != FD2_OK) return st;
    if (train_loss) *train_loss = tail > 0 ? (float)(acc[0] / ((double)tail * s->batch)) : 0.0f;
    if (val_loss) {
        st = fd2_sg_eval(s, val_loss, nullptr, nullptr);
        if (st != FD2_OK) return st;
    }
    return FD2_OK;
}

fd2_status fd2_sg_loss_grad(fd2_sg *s, const float *features, const int32_t *photons, const int32_t *detected,
                            const uint32_t *radial, int32_t b, float *loss, float *grad)
{
    if (!s || !features || !photons || !detected || !radial || b <= 0 || b > s->batch)
        return FD2_ERR_INVALID_ARGUMENT;
    SG_CUDA(s, cudaSetDevice(s->device));
    fd2_status st = ensure_rows(s, s->batch);
    if (st != FD2_OK) return st;
    const size_t nb = (size_t)(s->bins + 1);
    float *df = nullptr;
    int32_t *dp = nullptr, *dd = nullptr;
    uint32_t *dr = nullptr;
    cudaError_t e = cudaMalloc(&df, sizeof(float) * b * kFeatures);
    if (e == cudaSuccess) e = cudaMalloc(&dp, sizeof(int32_t) * b);
    if (e == cudaSuccess) e = cudaMalloc(&dd, sizeof(int32_t) * b);
    if (e == cudaSuccess) e = cudaMalloc(&dr, sizeof(uint32_t) * b * nb);
    if (e == cudaSuccess) e = upload(s, df, features, sizeof(float) * b * kFeatures);
    if (e == cudaSuccess) e = upload(s, dp, photons, sizeof(int32_t) * b);
    if (e == cudaSuccess) e = upload(s, dd, detected, sizeof(int32_t) * b);
    if (e == cudaSuccess) e = upload(s, dr, radial, sizeof(uint32_t) * b * nb);
    if (e == cudaSuccess) e = cudaMemsetAsync(s->d_acc, 0, sizeof(double) * 4, s->stream);
    if (e == cudaSuccess) {
        gather_kernel<<<warps_for(b), 256, 0, s->stream>>>(df, dp, dd, dr, s->bins, b, 0, b, true, s->seed,
                                                               s->d_step, s->norm, s->x0, s->target, s->ylab,
                                                               s->has_rad);
        e = sg_forward(s, s->stream, s->x0, b, nullptr, s->h1, s->h2, s->h3, s->out);
    }
    if (e == cudaSuccess) {
        loss_kernel<<<loss_blocks(b), 32 * kLossWarps, 0, s->stream>>>(s->out, kOutPad, s->target, s->ylab, s->has_rad,
                                                             s->bins, (float)s->radial_max, s->lambda, b,
                                                             1.0f / (float)b, s->dout, s->d_acc);
        e = backward(s, s->stream, b);
    }
    double acc[4] = {0, 0, 0, 0};
    std::vector<float> g((size_t)s->n_params);
    if (e == cudaSuccess) e = cudaMemcpyAsync(acc, s->d_acc, sizeof acc, cudaMemcpyDeviceToHost, s->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(g.data(), s->g, sizeof(float) * g.size(), cudaMemcpyDeviceToHost, s->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s->stream);
    cudaFree(df);
    cudaFree(dp);
    cudaFree(dd);
    cudaFree(dr);
    SG_CUDA(s, e);
    if (fd2_status t = sg_tc_check(s)) return t;
    if (loss) *loss = (float)(acc[0] / b);
    if (grad) for_each_public(s, [&](int64_t k, int64_t i) { grad[k] = g[(size_t)i]; });
    return FD2_OK;
}

fd2_status fd2_sg_predict(fd2_sg *s, const float *features, int64_t n, float *out)
{
    if (!s || !features || !out || n < 0) return FD2_ERR_INVALID_ARGUMENT;
    if (n == 0) return FD2_OK;
    SG_CUDA(s, cudaSetDevice(s->device));
    // two tiles of 128 rows for every SM a pass (fewer with wider layers), where
    // the training batch's 8,192 rows are 64 tiles in all.  The outputs leave the
    // device packed, straight into the caller's array (50,001 rows: seven batches
    // of padded rows, each waited for and unpadded on the host, 2.5 ms; two passes
    // 0.9)
    const int64_t rows = 2 * 128 * (int64_t)s->sm_count, most = std::min(rows, rows * 256 / s->hidden);
    const int64_t cap = std::min(n, most);
    if (cap > s->predict_cap) {
        // one allocation: outputs, packed outputs and features in FP32, then
        // the network's input and two layers in BF16, each 256-byte aligned
        const size_t C = ((size_t)cap + 63) / 64 * 64, H = (size_t)s->hidden;
        s->predict_cap = 0;
        SG_CUDA(s, alloc(&s->pout, C * (kOutPad + kOutputs + kFeatures) + C * (kInPad + 2 * H) / 2));
        s->ppack = s->pout + C * kOutPad;
        s->pf = s->ppack + C * kOutputs;
        s->px = reinterpret_cast<__nv_bfloat16 *>(s->pf + C * kFeatures);
        s->pha = s->px + C * kInPad;
        s->phb = s->pha + C * H;
        s->predict_cap = cap;
    }
    cudaError_t e = cudaSuccess;
    for (int64_t at = 0; at < n && e == cudaSuccess; at += most) {
        const int b = (int)std::min<int64_t>(most, n - at);
        e = cudaMemcpyAsync(s->pf, features + at * kFeatures, sizeof(float) * b * kFeatures, cudaMemcpyHostToDevice,
                            s->stream);
        if (e != cudaSuccess) break;
        input_kernel<<<grid_for(b, 256), 256, 0, s->stream>>>(s->pf, b, s->norm, s->px);
        e = sg_forward(s, s->stream, s->px, b, nullptr, s->pha, s->phb, s->pha, s->pout);
        if (e != cudaSuccess) break;
        pack_outputs_kernel<<<grid_for((int64_t)b * kOutputs, 256), 256, 0, s->stream>>>(s->pout, b, s->ppack);
        e = cudaGetLastError();
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(out + at * kOutputs, s->ppack, sizeof(float) * b * kOutputs, cudaMemcpyDeviceToHost,
                                s->stream);
    }
    const cudaError_t e2 = cudaStreamSynchronize(s->stream);
    SG_CUDA(s, e);
    SG_CUDA(s, e2);
    return sg_tc_check(s);
}

// File: "FD2SG002", hidden, bins, radial_max, normalisation box, routing
// hull, public parameters; then, optionally, "EDGE" and the edge survival's
// amplitude and length (float each; a file without them loads amplitude 0).
fd2_status fd2_sg_save(fd2_sg *s, const char *path)
{
    if (!s || !path) return FD2_ERR_INVALID_ARGUMENT;
    std::vector<float> p((size_t)public_count(s));
    fd2_status st = fd2_sg_get_params(s, p.data(), (int64_t)p.size());
    if (st != FD2_OK) return st;
    FILE *f = std::fopen(path, "wb");
    if (!f) return sg_fail(s, FD2_ERR_IO, std::string("cannot write ") + path);
    const int32_t hdr[2] = {s->hidden, s->bins};
    bool ok = std::fwrite("FD2SG002", 1, 8, f) == 8 && std::fwrite(hdr, sizeof hdr, 1, f) == 1 &&
              std::fwrite(&s->radial_max, sizeof(double), 1, f) == 1 &&
              std::fwrite(&s->norm_box, sizeof s->norm_box, 1, f) == 1 &&
              std::fwrite(&s->hull, sizeof s->hull, 1, f) == 1 &&
              std::fwrite(p.data(), sizeof(float), p.size(), f) == p.size();
    if (s->edge_amp > 0.0f) {
        const float edge[2] = {s->edge_amp, s->edge_len_um};
        ok = ok && std::fwrite("EDGE", 1, 4, f) == 4 && std::fwrite(edge, sizeof edge, 1, f) == 1;
    }
    ok = (std::fclose(f) == 0) && ok;
    return ok ? FD2_OK : sg_fail(s, FD2_ERR_IO, std::string("write failed: ") + path);
}

fd2_status fd2_sg_load(fd2_sg *s, const char *path)
{
    if (!s || !path) return FD2_ERR_INVALID_ARGUMENT;
    FILE *f = std::fopen(path, "rb");
    if (!f) return sg_fail(s, FD2_ERR_IO, std::string("cannot read ") + path);
    char magic[8];
    int32_t hdr[2];
    double rmax = 0;
    fd2_sg_hull nb, h;
    std::vector<float> p((size_t)public_count(s));
    bool ok = std::fread(magic, 1, 8, f) == 8 && std::memcmp(magic, "FD2SG002", 8) == 0 &&
              std::fread(hdr, sizeof hdr, 1, f) == 1 && std::fread(&rmax, sizeof rmax, 1, f) == 1 &&
              std::fread(&nb, sizeof nb, 1, f) == 1 && std::fread(&h, sizeof h, 1, f) == 1;
    ok = ok && hdr[0] == s->hidden && hdr[1] == s->bins && rmax == s->radial_max &&
         std::fread(p.data(), sizeof(float), p.size(), f) == p.size();
    float edge[2] = {0.0f, 1.0f};
    char tag[4];
    if (ok && std::fread(tag, 1, 4, f) == 4) {
        ok = std::memcmp(tag, "EDGE", 4) == 0 && std::fread(edge, sizeof edge, 1, f) == 1 && edge[0] >= 0.0f &&
             edge[0] < 1.0f && edge[1] > 0.0f;
    }
    std::fclose(f);
    if (!ok) return sg_fail(s, FD2_ERR_IO, std::string("not a matching surrogate file: ") + path);
    s->edge_amp = edge[0];
    s->edge_len_um = edge[1];
    fd2_status st = fd2_sg_set_params(s, p.data(), (int64_t)p.size());
    if (st != FD2_OK) return st;
    s->norm_box = nb;
    s->norm_fixed = true;
    set_norm(s);
    return fd2_sg_set_hull(s, &h);
}

}  // extern "C"
