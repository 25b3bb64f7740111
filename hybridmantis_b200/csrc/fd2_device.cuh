// fd2_device.cuh -- device-side core of the production transport.
//
// Philox-4x32-10 uniforms and the FP32 photon walker.  The walker follows
// the reference's per-photon random walk (main/kernel_cuda_c_ver1_0.cu, C
// path: algo :553, isotropic :702, dist_to_surface :966, detection :3372,
// boundary_analysis :1582, transmit :2421, refl_bottom :2985,
// trans_dir_cos :3169, RoughSurface :3261) decision for decision, with
// changes that keep the distribution and suit sm_100a:
//   * each photon draws from its own xoshiro128+ stream (Blackman & Vigna,
//     "Scrambled linear pseudorandom number generators", ACM TOMS 47(4),
//     2021) whose 128-bit state is one Philox-4x32-10 block (Salmon et al.,
//     "Parallel random numbers: as easy as 1, 2, 3", SC'11) keyed by the run
//     seed at counter (0, photon-in-event, event, run): a photon's walk does
//     not depend on which lane runs it or when, and a draw costs a handful
//     of integer operations in registers instead of a Philox block per four
//     uniforms;
//   * angle tests are made on cosines (acos(c) > 1.57 <=> c < cos 1.57) and
//     the Fresnel coefficients use the cosine forms, so the walk needs no
//     acos/asin/tan/pow; the refraction keeps the reference's formula
//     d' = -cos(t_t) n - (sin t_t / sin t_i)(d + cos(t_i) n);
//   * the wall quadratic uses the cancellation-free root, with the
//     discriminant recomputed in FP64 when it nearly cancels;
//   * the whole walk is inlined around one photon held in registers, and its
//     rarer, longer parts can run later, from the photon's state alone.
// Tallies are not touched here: a step returns the photon's fate and the
// kernel tallies ended photons together.
#pragma once

#include <cstdint>

#include "fd2_types.h"

namespace fd2 {

// ---------------------------------------------------------------- Philox

__device__ __forceinline__ uint4 philox4x32_10(uint4 c, uint32_t k0, uint32_t k1)
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

// Philox-4x32-10 with the key schedule precomputed: rk[2r], rk[2r+1] are
// the two key words of round r (the run's keys, identical for every lane).
__device__ __forceinline__ uint4 philox4x32_10_rk(uint4 c, const uint32_t *rk)
{
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        const uint32_t lo0 = 0xD2511F53u * c.x, hi0 = __umulhi(0xD2511F53u, c.x);
        const uint32_t lo1 = 0xCD9E8D57u * c.z, hi1 = __umulhi(0xCD9E8D57u, c.z);
        c = make_uint4(hi1 ^ c.y ^ rk[2 * r], lo1, hi0 ^ c.w ^ rk[2 * r + 1], lo0);
    }
    return c;
}

// Uniform k 2^-23 + 2^-24 in [2^-24, 1 - 2^-24] from the top 23 bits k:
// (1 + k 2^-23) - (1 - 2^-24), exact in float.
__device__ __forceinline__ float u01(uint32_t r)
{
    // 0x3F800000 + (r >> 9) as one multiply-add, which runs beside the integer
    // pipe that the generator fills (a funnel shift of 0x7F and r: 1 % slower
    // with several geometries, the same with one)
    uint32_t b;
    asm("mad.hi.u32 %0, %1, 0x800000, 0x3f800000;" : "=r"(b) : "r"(r));
    return __uint_as_float(b) - 0.99999994039535522461f;
}

// What a part of the walk returns, and the state of the lane that holds the
// photon (a lane without one: 0): a fate (1 to 7), or one of these.  Bit 3:
// the photon is in flight; bit 1: it waits for a part that runs later.
enum Flight : int {
    kFlies = 8,       // goes on with its next step
    kRetryNormal = 9, // its crosstalk normal was rejected: tried again in the next step
    kWaits = 10,      // at a column wall or the top reflector: surface_wait
    kHops = 11,       // has left its column: surface_wait from the hop on
    kNeedsNormal = 16 // crosses into the adjacent column: crosstalk_normal next
};

// Warp-uniform part of a photon's seed: the Philox round keys of the run
// seed (the kernel keeps them in shared memory) and the run counter.
struct RngKey {
    const uint32_t *rk;
    uint32_t run;
};


// ---------------------------------------------------------------- walker

// a b + c d with c d rounded and a b fused, and a b + c d + e f with c d
// rounded and the others fused.  Written out because which product of a sum
// the compiler fuses depends on the code around it: the transport's kernel
// variants must round a walk alike (a column billiard turns a last-bit
// difference into another history), so that label runs, geometry scans and
// single-geometry runs of the same photons keep giving the same tallies.  Not
// written out is the neighbour test of the hexagonal lattice (fx, fy, disc in
// grid_flight), whose fusing no explicit form tried reproduces: its kernels are
// those that the compiler rounds alike, and a compiler that fuses it otherwise
// changes their histories.
__device__ __forceinline__ float sum2(float a, float b, float c, float d) { return __fmaf_rn(a, b, __fmul_rn(c, d)); }
__device__ __forceinline__ float sum3(float a, float b, float c, float d, float e, float f)
{
    return __fmaf_rn(e, f, sum2(a, b, c, d));
}

__device__ __forceinline__ void renorm(float &x, float &y, float &z)
{
    const float nrm = sqrtf(sum3(x, x, y, y, z, z));
    if (nrm < 1.0f - kEps || nrm > 1.0f + kEps) {
        const float inv = 1.0f / nrm;
        x *= inv; y *= inv; z *= inv;
    }
}

// Fresnel reflectance (unpolarised) for cos(incidence) c, cos(refraction)
// ct and relative index eta = n_incident / n_transmitted.
__device__ __forceinline__ float fresnel(float c, float ct, float eta)
{
    const float a = eta * c, b = eta * ct;
    const float rs = __fdividef(a - ct, a + ct);
    const float rp = __fdividef(c - b, c + b);
    return 0.5f * sum2(rs, rs, rp, rp);
}

// Larger root of a t^2 + b t + c = 0 (the far wall of the column), without
// cancellation; 999 where the reference's formula yields NaN.
__device__ __forceinline__ float wall_root(float qa, float qb, float qc)
{
    float disc = sum2(-(4.0f * qa), qc, qb, qb);
    if (fabsf(disc) < 2.44140625e-4f * (qb * qb)) {
        // near-cancelling discriminant: products of floats are exact in FP64
        disc = (float)((double)qb * (double)qb - 4.0 * (double)qa * (double)qc);
    }
    // one division for both signs of qb, chosen by selects: the lanes of a
    // warp have both
    const float s = sqrtf(disc);
    const bool far = qb >= 0.0f;
    const float den = far ? qb + s : 2.0f * qa;
    float t = (far ? -2.0f * qc : s - qb) / den;
    t = far && den == 0.0f ? 0.0f : t;
    return !(qa > 0.0f) || !(disc >= 0.0f) ? 999.0f : t;
}

// The PRF pixel of a photon detected at (x, y); -1 outside the PRF's bounds.
template <class G>
__device__ __forceinline__ void detection_pixel(const G &g, float x, float y, int &ii, int &jj)
{
    ii = -1;
    jj = -1;
    if (x <= g.ub_x && y <= g.ub_y && x >= g.lb_x && y >= g.lb_y) {
        ii = (int)floorf(__fdiv_rn(x - g.lb_x, g.pixel));
        jj = (int)floorf(__fdiv_rn(y - g.lb_y, g.pixel));
    }
}

struct Walker {
    // photon
    float px, py, pz;   // position
    float dx, dy, dz;   // direction
    float nx, ny, nz;   // current surface normal
    float xc, yc;       // centre of the current column
    float dist;         // path length of the lane's photons since it was last summed
    float budget;       // absorption lengths left before bulk absorption
    uint32_t rebound;   // boundary interactions
    // The photon's random stream: xoshiro128+ state (never all zero; a
    // Philox block is all zero with probability 2^-128, and start() then
    // sets one bit).  The float uses the top 23 bits of each output, the
    // bits the generator's authors recommend for floating point.
    uint32_t s0, s1, s2, s3;

    __device__ __forceinline__ float u()
    {
        const uint32_t r = s0 + s3;
        const uint32_t t = s1 << 9;
        s2 ^= s0;
        s3 ^= s1;
        s1 ^= s2;
        s0 ^= s3;
        s2 ^= t;
        s3 = __funnelshift_l(s3, s3, 11);
        return u01(r);
    }

    // Start photon `photon_in_event` of event `event_index` at the event's
    // position (ex, ey, ez), in the column centred on it.  The event record
    // itself stays outside the walker (the kernel keeps it in shared memory),
    // so it holds no registers through the walk.
    __device__ __forceinline__ void start(float ex, float ey, float ez, uint32_t photon_in_event,
                                          uint32_t event_index, bool first, const RngKey &key)
    {
        const uint4 k = philox4x32_10_rk(make_uint4(0u, photon_in_event, event_index, key.run), key.rk);
        s0 = k.x;
        s1 = k.y;
        s2 = k.z;
        s3 = k.w | ((k.x | k.y | k.z | k.w) == 0u ? 1u : 0u);
        px = ex; py = ey; pz = ez;
        xc = ex; yc = ey;
        nx = 0.0f; ny = 0.0f; nz = 0.0f;
        rebound = 0;
        emit(first);
        budget = -__logf(u());  // Exp(1)
    }

    // Isotropic emission; the first photon of an event rejects |cos| <= 0.01
    // (the reference's CPU driver, hybridMANTIS_c_ver1_0.c:257-262).
    __device__ __forceinline__ void emit(bool first)
    {
        float c = 2.0f * u() - 1.0f;
        if (first) {
            for (int t = 0; t < 64 && fabsf(c) <= 0.01f; ++t) c = 2.0f * u() - 1.0f;
        }
        const float rr = sqrtf(fmaxf(0.0f, 1.0f - c * c));
        float s, co;
        __sincosf(kPi * (2.0f * u() - 1.0f), &s, &co);
        dx = rr * co;
        dy = rr * s;
        dz = c;
        renorm(dx, dy, dz);
    }

    // n <- normalize(n + beta * q), q the reference's perturbation vector:
    // z = 2u1 - 1, transverse radius sqrt(1 - u1^2), uniform azimuth, then
    // normalised (RoughSurface).
    __device__ __forceinline__ void roughen(float beta)
    {
        const float u1 = u();
        const float qz = 2.0f * u1 - 1.0f;
        const float rr = sqrtf(1.0f - u1 * u1);  // u1 < 1, also rounded
        float s, c;
        __sincosf(kPi * (2.0f * u() - 1.0f), &s, &c);
        const float qx = rr * c, qy = rr * s;
        // |q|^2 = (1 - u1^2) + (2 u1 - 1)^2 = 3 u1^2 - 4 u1 + 2 for u1 in (0, 1)
        const float bq = beta * rsqrtf(fmaf(u1, fmaf(3.0f, u1, -4.0f), 2.0f));
        const float rx = fmaf(bq, qx, nx), ry = fmaf(bq, qy, ny), rz = fmaf(bq, qz, nz);
        const float ir = rsqrtf(sum3(rx, rx, ry, ry, rz, rz));
        nx = rx * ir; ny = ry * ir; nz = rz * ir;
    }

    // A new column's orientation before its own roughening: (ix, iy, iz)
    // roughened with beta = 1 and flattened to the x-y plane (the
    // reference's RoughSurface(1) followed by nz = 0 and a 2D
    // normalisation).  The 3D normalisation between the two is a positive
    // scale the 2D one removes, so the flattened direction of i + q/|q| is
    // taken directly; the draws are roughen's.
    __device__ __forceinline__ void flat_rough(float ix, float iy, float iz)
    {
        const float u1 = u();
        const float qz = 2.0f * u1 - 1.0f;
        const float rr = sqrtf(1.0f - u1 * u1);  // u1 < 1, also rounded
        float s, c;
        __sincosf(kPi * (2.0f * u() - 1.0f), &s, &c);
        const float qx = rr * c, qy = rr * s;
        const float iq = rsqrtf(fmaf(u1, fmaf(3.0f, u1, -4.0f), 2.0f));  // 1 / |q|, as in roughen
        const float vx = fmaf(iq, qx, ix), vy = fmaf(iq, qy, iy);
        const float inv = rsqrtf(sum2(vx, vx, vy, vy));
        nx = vx * inv;
        ny = vy * inv;
        nz = 0.0f;
        (void)iz;
    }

    // A photon that bulk absorption cannot end keeps a positive budget (the
    // draw's logarithm may round to zero).
    template <class G>
    __device__ __forceinline__ void fill_budget(const G &g)
    {
        budget = g.neg_inv_mu != 0.0f ? budget : 1.0f;
    }
    template <class G>
    __device__ __forceinline__ bool outside_xy(const G &g) const
    {
        return px < kEps || px > g.xdet || py < kEps || py > g.ydet;
    }
    template <class G>
    __device__ __forceinline__ bool outside_detector(const G &g) const
    {
        return outside_xy(g) || pz < -g.half || pz > g.half;
    }
    template <class G>
    __device__ __forceinline__ bool at_top(const G &g) const
    {
        return fabsf(pz - g.half) < kEps && dz > 0.0f;
    }

    // Wall or z plane ahead, then the reference's pull-back into the column
    // (dist_to_surface), then bulk absorption (isotropic).  Selects instead of
    // early exits and of branches that most lanes take (a branch is three
    // instructions for the warp): the pull-back's first step and the absorption
    // run for all lanes (20,000 config-1 x-rays 41.4 ms, by branches 42.9).
    // `ended`: the photon's walk is over, with the fate that is returned.
    template <class G>
    __device__ __forceinline__ int flight(const G &g, bool &ended)
    {
        const float ddx = px - xc, ddy = py - yc;
        const float qa = sum2(dy, dy, dx, dx);
        const float qb = 2.0f * sum2(ddy, dy, ddx, dx);
        const float qc = __fmaf_rn(-g.R, g.R, sum2(ddy, ddy, ddx, ddx));
        const float dcyl = wall_root(qa, qb, qc);
        const float zp = copysignf(g.half, dz);
        const bool straight = fabsf(dx) < kEps && fabsf(dy) < kEps && fabsf(fabsf(dz) - 1.0f) < kEps;
        const float dplane = (zp - pz) / dz;
        const bool plane = dz != 0.0f && (straight || !(dplane >= dcyl));
        const float d = plane ? dplane : dcyl;
        pz = plane ? zp : fmaf(d, dz, pz);
        px = fmaf(d, dx, px);
        py = fmaf(d, dy, py);
        const bool lost = outside_detector(g);
        const float thr = g.R - 1e-5f;
        float r = sqrtf(sum2(px - xc, px - xc, py - yc, py - yc));
        r = lost ? 0.0f : r;
        // the first half-micron back, all that most photons need
        const bool at_wall = r > thr;
        float sx = px, sy = py;
        px = fmaf(-0.5f, dx, sx);
        py = fmaf(-0.5f, dy, sy);
        float rn = sqrtf(sum2(px - xc, px - xc, py - yc, py - yc));
        bool back = rn > r;
        px = back || !at_wall ? sx : px;
        py = back || !at_wall ? sy : py;
        r = back || !at_wall ? r : rn;
        // the others at a wall (grazing: a chord below the step): at most ten
        // steps moved (bits 0-3, from 6 on) and ten halved (bits 8-11)
        float step = back ? 0.25f : 0.5f;
        uint32_t n = back ? 0x0706u : 0x0607u;
        while (r > thr && !(n & 0x1010u)) {
            sx = px, sy = py;
            px = fmaf(-step, dx, px);
            py = fmaf(-step, dy, py);
            rn = sqrtf(sum2(px - xc, px - xc, py - yc, py - yc));
            back = rn > r;
            px = back ? sx : px;
            py = back ? sy : py;
            r = back ? r : rn;
            step = back ? 0.5f * step : step;
            n += back ? 0x100u : 1u;
        }
        // (pz has not moved since `lost`)
        const bool whole = !lost && !(r > thr) && !outside_xy(g);
        dist += whole ? d : 0.0f;
        // bulk absorption: one Exp(1) budget of absorption lengths per photon,
        // spent flight by flight; by the exponential's lack of memory the same
        // law as the reference's fresh draw per flight (absorbed when
        // d >= -ln(u) / mu); without absorption nothing is spent of it
        const float da = d * g.mu;
        ended = !whole || (da >= budget && d >= 0.0f);
        budget -= da;
        return whole ? kAbsBulk : lost || !(r > thr) ? kLost : kOutOfCol;
    }

    // Orientation of the next column: a random normal within 1.57 rad of
    // the reversed direction, flattened to the x-y plane, roughened.
    template <class G>
    __device__ __forceinline__ int new_column_normal(const G &g, float ix, float iy, float iz, int &tries,
                                                     bool always_rough)
    {
        for (;;) {
            flat_rough(ix, iy, iz);
            if (always_rough || g.beta > 0.0f) roughen(g.beta);
            if (!(sum3(iy, ny, ix, nx, iz, nz) < kCos157)) return kFlies;
            if (tries < 100) {
                ++tries;
                continue;
            }
            return kTheta1;
        }
    }

    // Leave the current column after a transmission through its wall
    // (transmit without crosstalk; crosstalk is crosstalk_normal): hop
    // U(d_min, d_max) with the top reflector and the sensor on the way, then
    // orient the next column.  Hops after a top reflection repeat the loop.
    // A photon reflected by the sensor between columns hops again
    // (refl_bottom): up to the top, or into a new column whose normal is
    // drawn around its own reversed direction, always roughened; after a
    // sensor met at the hop's end it stays where that hop left it unless it
    // reached the top.
    // Written as a state machine so that the kernel holds one copy of each
    // part (hop, sensor, hop after the sensor, next normal, top reflector):
    // the walk's instruction fetch grows with the kernel's code size.
    // The parts stand in the order photons pass them, so that one round of the
    // loop takes most photons through and the lanes meet at the next normal (a
    // part per round 1 % slower).
    template <class G>
    __device__ __forceinline__ int leave_column(const G &g)
    {
        enum { kHop, kSensor, kSensorHop, kNormal, kAfterSensor, kEnd };
        float ix = -dx, iy = -dy, iz = -dz;  // the next normal is drawn around these
        // One register for the rest: retries of the side hop's and the top
        // hops' normals (bits 0-7 and 8-15, each at most 100), top
        // reflections (bits 16-28, at most kMaxTopLoops), and three flags.
        constexpr uint32_t kSideHop = 1u << 29;     // the hop leaves a column wall (not the top)
        constexpr uint32_t kFromEnd = 1u << 30;     // the sensor was met at a hop's end, not during it
        constexpr uint32_t kAfterHop = 1u << 31;    // the pending normal follows a sensor hop
        constexpr uint32_t kTopOne = 1u << 16, kTopMask = 0x1fffu << 16;
        uint32_t counts = kSideHop;
        int st = kHop;
        for (;;) {
            if (st == kHop) {
                const float sx = px, sy = py, sz = pz;
                const float d = fmaf(u(), g.d_span, g.d_min);
                px = fmaf(dx, d, sx);
                py = fmaf(dy, d, sy);
                pz = fmaf(dz, d, sz);
                if (outside_xy(g)) return kLost;
                counts &= ~kAfterHop;
                st = kNormal;
                if (pz < -g.half || pz > g.half) {
                    const float dtop = (g.half - sz) / dz;
                    const float dbot = (-g.half - sz) / dz;
                    if (dtop < d && dtop > kEps) {
                        px = fmaf(dx, dtop, sx);
                        py = fmaf(dy, dtop, sy);
                        pz = g.half;
                        dist += dtop;
                    } else if (dbot < d && dbot > kEps) {
                        px = fmaf(dx, dbot, sx);
                        py = fmaf(dy, dbot, sy);
                        pz = -g.half;
                        dist += dbot;
                        counts &= ~kFromEnd;
                        st = kSensor;
                    } else {
                        return kLost;
                    }
                } else {
                    dist += d;
                }
            }
            if (st == kSensor) {
                // sensor between columns: reflect with sensorRefl, else detect
                if (!(g.sensor_refl > 0.0f && u() < g.sensor_refl)) {
                    return kDetect;
                }
                dz = -dz;
                renorm(dx, dy, dz);
                st = kSensorHop;
            }
            if (st == kSensorHop) {
                const float sx = px, sy = py, sz = pz;
                const float hop = fmaf(u(), g.d_span, g.d_min);
                px = fmaf(dx, hop, sx);
                py = fmaf(dy, hop, sy);
                pz = fmaf(dz, hop, sz);
                if (outside_xy(g)) return kLost;
                if (pz > g.half) {
                    const float dtop = (g.half - sz) / dz;
                    if (!(dtop < hop && dtop > kEps)) return kLost;
                    px = fmaf(dx, dtop, sx);
                    py = fmaf(dy, dtop, sy);
                    pz = g.half;
                    dist += dtop;
                    st = kAfterSensor;
                } else {
                    dist += hop;
                    counts |= kAfterHop;
                    st = kNormal;
                }
            }
            if (st == kNormal) {
                const bool after_sensor = (counts & kAfterHop) != 0u, side_hop = (counts & kSideHop) != 0u;
                int t = after_sensor ? 0 : (int)((side_hop ? counts : counts >> 8) & 0xffu);
                // after a sensor hop: around the hop's own reversed direction
                const float ax = after_sensor ? -dx : ix, ay = after_sensor ? -dy : iy, az = after_sensor ? -dz : iz;
                const int f = new_column_normal(g, ax, ay, az, t, after_sensor);
                if (f != kFlies) return f;
                if (after_sensor) {
                    st = kAfterSensor;
                } else {
                    counts = side_hop ? (counts & ~0xffu) | (uint32_t)t : (counts & ~0xff00u) | ((uint32_t)t << 8);
                    if (side_hop && (fabsf(px) < kEps || fabsf(px - g.xdet) < kEps || fabsf(py) < kEps ||
                                     fabsf(py - g.ydet) < kEps))
                        return kLost;
                    st = kEnd;
                }
            }
            if (st == kAfterSensor) {
                counts &= ~kAfterHop;
                if (!(counts & kFromEnd)) {
                    // a sensor met during the hop: the next normal follows
                    // unless the sensor hop reached the top
                    if (at_top(g)) {
                        st = kEnd;
                    } else {
                        st = kNormal;
                    }
                } else {
                    // a sensor hop that reached the top ends at the top
                    // reflector (the hop's end check finds the top at once)
                    if (!at_top(g)) return kFlies;
                    st = kEnd;
                }
            }
            if (st == kEnd) {
                // top reflector / sensor at the end of the hop
                if (at_top(g)) {
                    if (g.top_absfrac > 0.0f && u() < g.top_absfrac) return kAbsTop;
                    dz = -fabsf(2.0f * u() - 1.0f);
                    const float rr = sqrtf(fmaxf(0.0f, 1.0f - dz * dz));
                    float s, c;
                    __sincosf(kPi * (2.0f * u() - 1.0f), &s, &c);
                    dx = rr * c;
                    dy = rr * s;
                    ix = -dx; iy = -dy; iz = -dz;
                    counts = (counts & ~kSideHop) + kTopOne;
                    if ((counts & kTopMask) == ((uint32_t)kMaxTopLoops << 16)) return kCapped;
                    st = kHop;
                } else {
                    if (fabsf(pz + g.half) >= kEps) return kFlies;
                    counts |= kFromEnd;
                    st = kSensor;
                }
            }
        }
    }

    // Top reflector above the columns: absorb, or diffuse reflection down.
    template <class G>
    __device__ __forceinline__ int top_reflector(const G &g)
    {
        if (g.top_absfrac > 0.0f && u() < g.top_absfrac) return kAbsTop;
        dz = -fabsf(2.0f * u() - 1.0f);
        const float rr = sqrtf(fmaxf(0.0f, 1.0f - dz * dz));
        float s, c;
        __sincosf(kPi * (2.0f * u() - 1.0f), &s, &c);
        dx = rr * c;
        dy = rr * s;
        return kFlies;
    }

    // Interaction with a column wall (boundary_analysis), first part: whether
    // the photon crosses into the adjacent column (kNeedsNormal) or meets the
    // wall (kWaits); the rest (crosstalk_normal, surface_wait) can run
    // later, from the photon state alone.
    template <class G>
    __device__ __forceinline__ int surface_entry(const G &g)
    {
        // columnar crosstalk: certain in the top 20 %, linear to 0.5 at mid
        // depth, back to 1 at the sensor
        const float above = fmaf(pz, g.cct_k_hi, 0.5f), below = fmaf(pz + g.half, g.cct_k_lo, 1.0f);
        // (a step that ends outside the layer does not get here)
        float cct = pz < 0.0f ? below : above;
        cct = pz >= g.cct_band_lo ? 1.0f : cct;
        return u() < cct ? kNeedsNormal : kWaits;
    }

    // Crosstalk into the adjacent column (transmit with crosstalk): one
    // attempt at the new column's normal, a random normal within 1.57 rad of
    // the reversed direction, flattened and roughened.  Returns kFlies (the
    // photon is in the new column), kTheta1 (no normal after 100 retries) or
    // kRetryNormal (rejected: the kernel retries in its next round, beside
    // the other lanes' first attempts, instead of looping here with the few
    // rejected lanes of the warp).
    template <class G>
    __device__ __forceinline__ int crosstalk_normal(const G &g, int &tries)
    {
        const float ix = -dx, iy = -dy, iz = -dz;
        flat_rough(ix, iy, iz);
        if (g.beta > 0.0f) roughen(g.beta);
        if (!(sum3(iy, ny, ix, nx, iz, nz) < kCos157)) {
            xc = fmaf(-g.R, nx, px);
            yc = fmaf(-g.R, ny, py);
            return kFlies;
        }
        if (tries < 100) {
            ++tries;
            return kRetryNormal;
        }
        return kTheta1;
    }

    // The photon's tag: its geometry in bits 0-7, bit 8 just reflected by the
    // sensor, above it the retry counts of a wall interaction while it waits:
    // tries at an incidence angle and at a next normal (at most 100 each),
    // perturbations (3) and smooth attempts (25).
    static constexpr uint32_t kGeomBits = 0xffu, kReflected = 1u << 8;
    static constexpr int kTheta = 9, kPerturb = 16, kSmooth = 18, kNormalTry = 23;
    static constexpr uint32_t kCounts = (0x7fu << kTheta) | (3u << kPerturb) | (0x1fu << kSmooth) | (0x7fu << kNormalTry);

    // What a waiting photon waits for: the top reflector, or Fresnel reflection
    // / refraction on the rough wall (boundary_analysis, second part).  A
    // photon that refracts out of its column waits again, for its hop
    // (kHops); with `hop` it continues there, until it is back inside a
    // column or meets the next column's wall from outside and hops again.  Hops
    // count as boundary interactions, which bounds them.  One
    // in five wall interactions leaves the column: run to their end beside the
    // others, the hops took half of the pass at 2 to 3 lanes.  `counts` keeps
    // the retry counts between the two.
    template <class G>
    __device__ __forceinline__ int surface_wait(const G &g, bool hop, uint32_t &counts)
    {
        if (!hop && at_top(g)) return top_reflector(g);
        if (hop && ++rebound > kMaxBoundaryCalls) return kCapped;
        bool outside = hop;
        int tries_theta = (counts >> kTheta) & 0x7f, tries_normal = (counts >> kNormalTry) & 0x7f;
        int reperturbs = (counts >> kPerturb) & 3, smooth = (counts >> kSmooth) & 0x1f;
        counts &= ~kCounts;
        float pr = __int_as_float(0x7fc00000);  // 0/0 until a rule sets it
        float st = 0.0f, ct = 1.0f;            // sin, cos of the last refraction angle
        float kx = 0, ky = 0, kz = 0, kdx = 0, kdy = 0, kdz = 0;
        enum { kLeave, kNewSurface, kRestore, kIncidence } stage = hop ? kLeave : kNewSurface;
        int fate = kFlies;
        for (int loop = 0; loop < kMaxSurfaceLoops; ++loop) {
            if (stage == kNewSurface) {
                if (!outside) {
                    const float ax = xc - px, ay = yc - py;
                    const float im = rsqrtf(sum2(ay, ay, ax, ax));
                    nx = ax * im; ny = ay * im; nz = 0.0f;
                    if (g.beta > 0.0f) roughen(g.beta);
                } else {
                    xc = fmaf(-g.R, nx, px);
                    yc = fmaf(-g.R, ny, py);
                }
                kx = nx; ky = ny; kz = nz;
                kdx = dx; kdy = dy; kdz = dz;
                stage = kRestore;
            }
            if (stage == kRestore) {
                nx = kx; ny = ky; nz = kz;
                dx = kdx; dy = kdy; dz = kdz;
                if (reperturbs != 0) {
                    if (g.beta > 0.0f) roughen(g.beta);
                    if (outside) {
                        xc = fmaf(-g.R, nx, px);
                        yc = fmaf(-g.R, ny, py);
                    }
                }
                stage = kIncidence;
            }
            if (stage == kIncidence) {
                const float c1 = -sum3(dy, ny, dx, nx, dz, nz);
                if (c1 > 1.0f || c1 < 0.0f) {
                    if (outside) {
                        const int f = new_column_normal(g, -dx, -dy, -dz, tries_normal, false);
                        if (f != kFlies) {
                            fate = f;
                            break;
                        }
                    }
                    if (tries_theta < 100) {
                        ++tries_theta;
                        if (!outside) {
                            // from within the column nothing else is carried
                            // over: tried again in the next pass
                            counts |= (uint32_t)tries_theta << kTheta | (uint32_t)reperturbs << kPerturb |
                                      (uint32_t)smooth << kSmooth;
                            return kWaits;
                        }
                        stage = kNewSurface;
                        continue;
                    }
                    fate = kTheta1;
                    break;
                }
                const float si = sqrtf(fmaxf(0.0f, 1.0f - c1 * c1));
                // selects: total reflection and the rest, inside and out, in
                // one piece of code (by branches 0.5 % slower)
                const bool stale = outside && g.stale_out;
                const float eta = outside ? g.eta_out : g.eta_in;
                const float nst = eta * si, nct = sqrtf(fmaxf(0.0f, 1.0f - nst * nst)), npr = fresnel(c1, nct, eta);
                const bool total = outside ? stale && c1 < g.cos_tir_out : c1 < g.cos_tir_in;
                const bool keep = stale || total;
                st = keep ? st : nst;
                ct = keep ? ct : nct;
                pr = total ? 1.0f : stale ? pr : npr;
                if (u() < pr) {
                    // specular reflection
                    dx = fmaf(2.0f * c1, nx, dx);
                    dy = fmaf(2.0f * c1, ny, dy);
                    dz = fmaf(2.0f * c1, nz, dz);
                    renorm(dx, dy, dz);
                    if (sum3(ky, dy, kx, dx, kz, dz) < kCos157) {
                        if (++reperturbs < 4) {
                            stage = kRestore;
                            continue;
                        }
                        nx = kx; ny = ky; nz = kz;
                        dx = kdx; dy = kdy; dz = kdz;
                        reperturbs = 0;
                        if (smooth < 25) {
                            ++smooth;
                            continue;  // stage stays kIncidence
                        }
                        fate = kTheta1;
                        break;
                    }
                    if (!outside) break;  // reflected inside the column: done
                    stage = kLeave;
                } else {
                    // refraction with the reference's formula
                    const float ratio = si > 0.0f ? __fdividef(st, si) : 0.0f;
                    const float tx = fmaf(c1, nx, dx), ty = fmaf(c1, ny, dy), tz = fmaf(c1, nz, dz);
                    dx = sum2(-ct, nx, -ratio, tx);
                    dy = sum2(-ct, ny, -ratio, ty);
                    dz = sum2(-ct, nz, -ratio, tz);
                    renorm(dx, dy, dz);
                    // a direction that is no number (columns of a nanometre) has
                    // the sign that flight takes for downwards, as a comparison
                    // with 0 would (two more instructions in every step)
                    if (!(dz == dz)) dz = __int_as_float(-1);
                    if (outside) break;  // entered the next column: done
                    stage = kLeave;
                }
                // the low-contrast rule looks back at the last refraction:
                // such photons go on at once
                if (!g.stale_out) {
                    counts |= (uint32_t)tries_theta << kTheta | (uint32_t)tries_normal << kNormalTry |
                              (uint32_t)reperturbs << kPerturb | (uint32_t)smooth << kSmooth;
                    return kHops;
                }
            }
            // kLeave: hop between columns
            const int f = leave_column(g);
            if (f != kFlies) {
                fate = f;
                break;
            }
            outside = true;
            stage = kNewSurface;
            if (loop + 1 == kMaxSurfaceLoops) fate = kCapped;
        }
        return fate;
    }

    // ---- explicit column lattice (options.column_grid = 1 or 2; no
    // counterpart in the reference, whose next column is drawn at random
    // after every crossing).  Columns are the cylinders of radius R around
    // the square lattice points ((i + 1/2) p, (j + 1/2) p), or around the
    // hexagonal lattice points ((i + 1/2) p + o_j, (j + 1/2) h), h = p sqrt(3)/2,
    // o_j = p/2 on odd rows; the photon is either inside the column centred at
    // (xc, yc) or in the gap medium between them.
    // Walls refract and reflect with the unpolarised Fresnel coefficients on
    // the roughened geometric normal (vector Snell law); in the gap the
    // photon flies straight until it meets a column (traced cell by cell),
    // the top reflector, the sensor or the detector's side.  Bulk absorption
    // acts inside the columns only.
    // The column nearest to a new photon; whether it starts in the gap.
    template <bool kSquare, class G>
    __device__ __forceinline__ bool grid_place(const G &g)
    {
        if (!kSquare && g.grid == 2) {
            // the nearest of the brick's own column and its four diagonal
            // neighbours in the rows above and below
            const float h = g.pitch * 0.8660254037844386f;
            const int j = (int)floorf(py / h);
            const float o = (j & 1) ? 0.5f * g.pitch : 0.0f;
            const int i = (int)floorf((px - o) / g.pitch);
            float bx = 0.0f, by = 0.0f, bd = 3.0e38f;
#pragma unroll
            for (int q = 0; q < 5; ++q) {
                float cx, cy;
                hex_candidate(g, i, j, q, cx, cy);
                const float d2 = sum2(px - cx, px - cx, py - cy, py - cy);
                if (d2 < bd) { bd = d2; bx = cx; by = cy; }
            }
            xc = bx;
            yc = by;
            return bd >= g.R * g.R;
        }
        xc = (floorf(px / g.pitch) + 0.5f) * g.pitch;
        yc = (floorf(py / g.pitch) + 0.5f) * g.pitch;
        const float rx = px - xc, ry = py - yc;
        return sum2(rx, rx, ry, ry) >= g.R * g.R;
    }

    // Hexagonal lattice: the rows are strips of height h; in row j the
    // bricks [i p + o_j, (i + 1) p + o_j) each hold one column at their
    // centre.  A column reaches at most R < p/2 sideways but may reach past
    // its strip (R > h/2 when the gap is small), so the columns that
    // overlap brick (i, j) are its own (q = 0) and the four centred on its
    // corners' columns in rows j - 1 and j + 1 (q = 1..4).
    template <class G>
    __device__ __forceinline__ static void hex_candidate(const G &g, int i, int j, int q, float &cx, float &cy)
    {
        const float p = g.pitch, h = p * 0.8660254037844386f;
        const float o = (j & 1) ? 0.5f * p : 0.0f;
        cx = ((float)i + 0.5f) * p + o;
        cy = ((float)j + 0.5f) * h;
        if (q > 0) {
            cy += q <= 2 ? h : -h;
            cx += (q & 1) ? -0.5f * p : 0.5f * p;
        }
    }

    // Top reflector (absorb or diffuse reflection downwards, the reference's
    // top rule) or sensor (detect, or specular reflection with sensor_refl).
    template <class G>
    __device__ __forceinline__ int grid_plane(const G &g, bool top)
    {
        if (top) return top_reflector(g);
        if (!(g.sensor_refl > 0.0f && u() < g.sensor_refl)) {
            return kDetect;
        }
        dz = -dz;
        return kFlies;
    }

    // A wall of the column centred at (cx, cy), met at (px, py); kInside: from
    // within the column.  The normal toward the incident side is roughened
    // (redrawn while the photon would not meet it); reflect with the Fresnel
    // probability (total reflection included), else refract.  Returns kFlies
    // inside a column, kWaits in the gap.
    template <bool kInside, class G>
    __device__ __forceinline__ int grid_wall(const G &g, float cx, float cy)
    {
        float ox = px - cx, oy = py - cy;
        const float inv = rsqrtf(sum2(oy, oy, ox, ox));
        ox *= inv;
        oy *= inv;
        const float sgn = kInside ? -1.0f : 1.0f;  // normal toward the incident medium
        float c1 = 0.0f;
        for (int t = 0; t < 8; ++t) {
            nx = sgn * ox; ny = sgn * oy; nz = 0.0f;
            if (g.beta > 0.0f) roughen(g.beta);
            c1 = -sum3(dy, ny, dx, nx, dz, nz);
            if (c1 > 0.0f) break;
        }
        if (!(c1 > 0.0f)) {
            nx = sgn * ox; ny = sgn * oy; nz = 0.0f;
            c1 = fmaxf(-sum2(dx, nx, dy, ny), 0.0f);
        }
        const float eta = kInside ? g.eta_in : g.eta_out;  // n_incident / n_transmitted
        const float st2 = eta * eta * fmaxf(0.0f, 1.0f - c1 * c1);
        float pr = 1.0f, ct = 0.0f;
        if (st2 < 1.0f) {
            ct = sqrtf(1.0f - st2);
            pr = fresnel(c1, ct, eta);
        }
        const bool refl = u() < pr;
        const float k = eta * c1 - ct;
        dx = refl ? fmaf(2.0f * c1, nx, dx) : fmaf(eta, dx, k * nx);
        dy = refl ? fmaf(2.0f * c1, ny, dy) : fmaf(eta, dy, k * ny);
        dz = refl ? fmaf(2.0f * c1, nz, dz) : fmaf(eta, dz, k * nz);
        renorm(dx, dy, dz);
        if (!kInside && !refl) {
            xc = cx;
            yc = cy;
        }
        return kInside == refl ? kFlies : kWaits;
    }

    // The flight of a lattice segment, inside a column or through the gap: to
    // a plane (kToPlane), to the wall of the column at (wx, wy) (kToWall), or
    // a fate.
    static constexpr int kToPlane = 200, kToWall = 201;
    template <bool kSquare, bool kInside, class G>
    __device__ __forceinline__ int grid_flight(const G &g, float &wx, float &wy)
    {
        const float zp = dz > 0.0f ? g.half : -g.half;
        const float dplane = dz != 0.0f ? (zp - pz) / dz : 3.0e38f;
        if (kInside) {
            const float ddx = px - xc, ddy = py - yc;
            const float qa = sum2(dy, dy, dx, dx);
            const float qb = 2.0f * sum2(ddy, dy, ddx, dx);
            // a photon on the wall (rounded just outside it) is on the wall:
            // the far root then always exists
            const float qc = fminf(__fmaf_rn(-g.R, g.R, sum2(ddy, ddy, ddx, ddx)), 0.0f);
            const float dw = wall_root(qa, qb, qc);
            const bool plane = dplane <= dw;
            const float d = fmaxf(plane ? dplane : dw, 0.0f);
            px = fmaf(d, dx, px);
            py = fmaf(d, dy, py);
            pz = plane ? zp : fmaf(d, dz, pz);
            dist += d;
            if (g.neg_inv_mu != 0.0f) {
                const float da = d * g.mu;
                if (da >= budget) return kAbsBulk;
                budget -= da;
            }
            if (outside_xy(g)) return kLost;
            if (plane) return kToPlane;
            wx = xc;
            wy = yc;
            return kToWall;
        }
        // in the gap: the first column along the ray, cell by cell (a column
        // lies inside its own cell, so the first hit is in the first cell
        // that holds one)
        const float p = g.pitch;
        const float tx = dx != 0.0f ? (dx > 0.0f ? g.xdet - px : -px) / dx : 3.0e38f;
        const float ty = dy != 0.0f ? (dy > 0.0f ? g.ydet - py : -py) / dy : 3.0e38f;
        const float tside = fminf(tx, ty);
        const float tend = fminf(dplane, tside);
        if (!kSquare && g.grid == 2) {
            // brick by brick; a hit counts in the brick where it lies
            const float h = p * 0.8660254037844386f;
            int j = (int)floorf(py / h);
            int i = (int)floorf((px - ((j & 1) ? 0.5f * p : 0.0f)) / p);
            const float qa = sum2(dy, dy, dx, dx);
            float tin = 0.0f;
            for (int k = 0; k < kMaxGridCells; ++k) {
                const float o = (j & 1) ? 0.5f * p : 0.0f;
                const float xl = (float)i * p + o;
                const float tX = dx != 0.0f ? (dx > 0.0f ? xl + p - px : xl - px) / dx : 3.0e38f;
                const float tY = dy != 0.0f ? ((float)(dy > 0.0f ? j + 1 : j) * h - py) / dy : 3.0e38f;
                const float tout = fminf(tX, tY);
                float tb = 3.0e38f, bx = 0.0f, by = 0.0f;
#pragma unroll
                for (int q = 0; q < 5; ++q) {
                    float cx, cy;
                    hex_candidate(g, i, j, q, cx, cy);
                    const float fx = px - cx, fy = py - cy;
                    const float qb = 2.0f * (fx * dx + fy * dy);
                    const float qc = fx * fx + fy * fy - g.R * g.R;
                    if (qa > 0.0f && qb < 0.0f) {
                        const float disc = sum2(qb, qb, -(4.0f * qa), qc);
                        if (disc >= 0.0f) {
                            const float t1 = (2.0f * qc) / (-qb + sqrtf(disc));
                            if (t1 > 1e-4f && t1 >= tin - 1e-4f && t1 <= tout + 1e-4f && t1 < tb) {
                                tb = t1;
                                bx = cx;
                                by = cy;
                            }
                        }
                    }
                }
                if (tb < tend) {
                    px = fmaf(tb, dx, px);
                    py = fmaf(tb, dy, py);
                    pz = fmaf(tb, dz, pz);
                    dist += tb;
                    wx = bx;
                    wy = by;
                    return kToWall;
                }
                if (tout >= tend) break;
                if (tX < tY) {
                    i += dx > 0.0f ? 1 : -1;
                } else {
                    // the next row: the brick under the crossing point
                    j += dy > 0.0f ? 1 : -1;
                    const float xo = fmaf(tout, dx, px) - ((j & 1) ? 0.5f * p : 0.0f);
                    i = (int)floorf(xo / p);
                }
                tin = tout;
                if (k + 1 == kMaxGridCells) return kCapped;
            }
            if (dplane <= tside) {
                px = fmaf(dplane, dx, px);
                py = fmaf(dplane, dy, py);
                pz = zp;
                dist += dplane;
                return kToPlane;
            }
            return kLost;
        }
        int i = (int)floorf(px / p), j = (int)floorf(py / p);
        const int si = dx > 0.0f ? 1 : -1, sj = dy > 0.0f ? 1 : -1;
        float tmx = dx != 0.0f ? (((float)(dx > 0.0f ? i + 1 : i)) * p - px) / dx : 3.0e38f;
        float tmy = dy != 0.0f ? (((float)(dy > 0.0f ? j + 1 : j)) * p - py) / dy : 3.0e38f;
        const float tdx = dx != 0.0f ? p / fabsf(dx) : 3.0e38f;
        const float tdy = dy != 0.0f ? p / fabsf(dy) : 3.0e38f;
        const float qa = sum2(dy, dy, dx, dx);
        for (int k = 0; k < kMaxGridCells; ++k) {
            const float cx = ((float)i + 0.5f) * p, cy = ((float)j + 0.5f) * p;
            const float fx = px - cx, fy = py - cy;
            const float qb = 2.0f * sum2(fx, dx, fy, dy);
            const float qc = __fadd_rn(sum2(fx, fx, fy, fy), -__fmul_rn(g.R, g.R));
            if (qa > 0.0f && qb < 0.0f) {
                const float disc = sum2(qb, qb, -(4.0f * qa), qc);
                if (disc >= 0.0f) {
                    const float t1 = (2.0f * qc) / (-qb + sqrtf(disc));  // the entry root
                    if (t1 > 1e-4f && t1 < tend) {
                        px = fmaf(t1, dx, px);
                        py = fmaf(t1, dy, py);
                        pz = fmaf(t1, dz, pz);
                        dist += t1;
                        wx = cx;
                        wy = cy;
                        return kToWall;
                    }
                }
            }
            const float tn = fminf(tmx, tmy);
            if (tn >= tend) break;
            if (tmx < tmy) {
                i += si;
                tmx += tdx;
            } else {
                j += sj;
                tmy += tdy;
            }
            if (k + 1 == kMaxGridCells) return kCapped;
        }
        if (dplane <= tside) {
            px = fmaf(dplane, dx, px);
            py = fmaf(dplane, dy, py);
            pz = zp;
            dist += dplane;
            return kToPlane;
        }
        return kLost;
    }

    // One segment of the lattice walk: a flight to the next surface and what
    // happens there.  Photons inside a column (kInside) run it in the warp's
    // steps, those in the gap in its passes for waiting photons: one routine
    // for both, asking each lane which, took 10,001 x-rays 68.5 ms (hexagonal
    // lattice 91.8), this 61.7 (83.0).
    template <bool kSquare, bool kInside, class G>
    __device__ __forceinline__ int grid_segment(const G &g)
    {
        if (++rebound > kMaxBoundaryCalls) return kCapped;
        float wx = 0.0f, wy = 0.0f;
        int f = grid_flight<kSquare, kInside>(g, wx, wy);
        if (f == kToWall) return grid_wall<kInside>(g, wx, wy);
        if (f == kToPlane) f = grid_plane(g, pz > 0.0f);
        return !kInside && f == kFlies ? kWaits : f;
    }

    // One transport step (the body of the reference's step function algo):
    // flight, sensor, trapped-photon restart (from `*event`, the x, y, z of
    // the photon's event), or a surface interaction up to the part that waits.
    // Returns the photon's fate, kFlies while it is in flight, kNeedsNormal
    // (run crosstalk_normal next) or kWaits (surface_wait next).  A
    // photon reflected by the sensor inside a column flies on in its next step,
    // beside the warp's others; a bit of its tag then keeps it from meeting the
    // sensor again where it stands.
    template <class G>
    __device__ __forceinline__ int step(const G &g, const float4 *event, uint32_t &tag)
    {
        bool ended;
        const int f = flight(g, ended);
        // one branch for all that few lanes do, at a plane, ended or trapped (four
        // in turn 1 % slower)
        const bool trapped = fabsf(dz) < kEps;
        if (ended || fabsf(fabsf(pz) - g.half) < kEps || trapped || rebound >= (uint32_t)kMaxBoundaryCalls) {
            if (ended) return f;
            const bool sensor = !(tag & kReflected) && fabsf(pz + g.half) < kEps;
            tag &= ~kReflected;
            if (sensor) {
                // sensor plane inside a column (detection)
                if (!(g.sensor_refl > 0.0f && u() < g.sensor_refl)) return kDetect;
                dz = dz == dz ? -dz : dz;  // specular reflection on the flat sensor
                renorm(dx, dy, dz);
                tag |= kReflected;
                return kFlies;
            }
            if (trapped) {
                // trapped travelling horizontally: restart from the event position,
                // keeping the current column (the reference does not reset it)
                const float4 e = *event;
                px = e.x; py = e.y; pz = e.z;
                emit(false);
                return kFlies;
            }
            if (rebound >= (uint32_t)kMaxBoundaryCalls) return kCapped;
            if (at_top(g)) {
                ++rebound;
                return kWaits;
            }
        }
        tag &= ~kReflected;
        ++rebound;
        return surface_entry(g);
    }
};

}  // namespace fd2
