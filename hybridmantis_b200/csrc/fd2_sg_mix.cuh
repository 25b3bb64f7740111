// fd2_sg_mix.cuh -- the surrogate's radial model: a mixture of Gaussian rings.
//
// The detected photons' 2D density around their deposition is modelled as
//   PRF(r) = sum_k w_k N(r; mu_k, sd_k) / S_k        (per unit area, r >= 0)
// i.e. each component is a ring of radius mu_k >= 0 and width sd_k (mu = 0:
// an isotropic 2D Gaussian), so the radial density of component k is
//   f_k(r) = r N(r; mu, sd) / S_k,
//   S_k = int_0^inf r N(r; mu, sd) dr = mu Phi_c(t0) + sd phi(t0),  t0 = -mu / sd.
// Its mass on [a, b) has the closed form
//   M(a, b) = mu [Phi(t_b) - Phi(t_a)] + sd [phi(t_a) - phi(t_b)],  t = (r - mu) / sd,
// with derivatives
//   dM/dmu = [Phi(t_b) - Phi(t_a)] + (a phi(t_a) - b phi(t_b)) / sd
//   dM/dsd = [phi(t_a) - phi(t_b)] + (t_a a phi(t_a) - t_b b phi(t_b)) / sd.
// CDF differences use lower tails left of the mean and upper tails right of
// it, so far-tail bins keep their relative accuracy in FP32.
#pragma once

#include <cuda_runtime.h>

#include "fd2_sg_internal.h"

namespace fd2 {
namespace sg {

struct Mix {
    float w[kComponents], mu[kComponents], sd[kComponents], S[kComponents];
};

__device__ __forceinline__ float norm_pdf(float a) { return 0.3989422804014327f * expf(-0.5f * a * a); }

// Values of one bin edge for one component; `inf` marks the edge at +inf.
struct Edge {
    float t, cdf, ccdf, pdf, e;
    bool inf;
};

__device__ __forceinline__ Edge edge_at(float e, bool inf, float mu, float sd)
{
    Edge x;
    x.e = e;
    x.inf = inf;
    if (inf) {
        x.t = 0.0f;
        x.cdf = 1.0f;
        x.ccdf = 0.0f;
        x.pdf = 0.0f;
    } else {
        x.t = (e - mu) / sd;
        x.cdf = normcdff(x.t);
        x.ccdf = normcdff(-x.t);
        x.pdf = norm_pdf(x.t);
    }
    return x;
}

// Mass of a ring component between two edges, and its derivatives.
__device__ __forceinline__ float ring_mass(const Edge &lo, const Edge &hi, float mu, float sd, float *dmu, float *dsd)
{
    const float dphi = fmaxf(lo.t >= 0.0f && !lo.inf ? lo.ccdf - hi.ccdf : hi.cdf - lo.cdf, 0.0f);
    const float m = fmaxf(mu * dphi + sd * (lo.pdf - hi.pdf), 0.0f);
    if (dmu) {
        const float ehi = hi.inf ? 0.0f : hi.e * hi.pdf;
        const float thi = hi.inf ? 0.0f : hi.t * hi.e * hi.pdf;
        *dmu = dphi + (lo.e * lo.pdf - ehi) / sd;
        *dsd = (lo.pdf - hi.pdf) + (lo.t * lo.e * lo.pdf - thi) / sd;
    }
    return m;
}

// A ring from its radius and width outputs, with its normaliser S and the
// derivatives dS/dmu = c0 and dS/dsd = p0.
struct Ring {
    float mu, sd, c0, p0, S;
};

__device__ __forceinline__ Ring decode_ring(float om, float ls)
{
    Ring r;
    r.mu = kMuScale * (fmaxf(om, 0.0f) + log1pf(expf(-fabsf(om))));  // softplus
    r.sd = kSdScale * expf(fminf(fmaxf(ls, kLogSdMin), kLogSdMax));
    const float t0 = -r.mu / r.sd;
    r.c0 = normcdff(-t0);
    r.p0 = norm_pdf(t0);
    r.S = fmaxf(r.mu * r.c0 + r.sd * r.p0, 1e-30f);
    return r;
}

// The softmax weight of the lane's component: `a` is the weight output of
// component lane % kComponents, the same in all lanes of a component.
__device__ __forceinline__ float lane_weight(float a)
{
    float amax = a;
#pragma unroll
    for (int d = kComponents / 2; d > 0; d >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, d));
    const float e = expf(a - amax);
    float s = 0.0f;
#pragma unroll
    for (int c = 0; c < kComponents; ++c) s += __shfl_sync(0xffffffffu, e, c);
    return e / s;
}

// Decode the network's mixture outputs (o[1..24]) in every lane.
__device__ __forceinline__ void decode_mix(const float *o, Mix &m)
{
    float amax = o[1];
#pragma unroll
    for (int k = 1; k < kComponents; ++k) amax = fmaxf(amax, o[1 + k]);
    float s = 0.0f;
#pragma unroll
    for (int k = 0; k < kComponents; ++k) {
        m.w[k] = expf(o[1 + k] - amax);
        s += m.w[k];
    }
#pragma unroll
    for (int k = 0; k < kComponents; ++k) {
        m.w[k] /= s;
        const Ring r = decode_ring(o[1 + kComponents + k], o[1 + 2 * kComponents + k]);
        m.mu[k] = r.mu;
        m.sd[k] = r.sd;
        m.S[k] = r.S;
    }
}

}  // namespace sg
}  // namespace fd2
