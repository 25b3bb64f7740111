// fd2_kernels.cu -- event preparation, photon-count sampling, work-queue
// construction, the persistent transport kernel and the PHS/Swank pass.
//
// Pipeline of one run (all on the context's stream, graph-capturable):
//   prep      events -> float4 (x, y, z um; history index) + energy     (at submit)
//   count     N ~ Poisson(E * yield) | Gaussian | given; chunks per event
//   scan      exclusive scan of chunks per event
//   fill      chunk descriptors (event, first photon)
//   transport persistent kernel: warps pull chunks, lanes regenerate photons
//   phs       per-primary counts -> PHS histogram + FP64 moments (Swank)
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "fd2_device.cuh"
#include "fd2_internal.h"

namespace fd2 {

namespace {

constexpr unsigned kFull = 0xFFFFFFFFu;

__device__ __forceinline__ unsigned lanemask_lt()
{
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// ------------------------------------------------------------------ prep

__device__ __forceinline__ bool finite_f(double v) { return isfinite(v); }

__global__ void prep_cm_kernel(int64_t n, const double *__restrict__ x, const double *__restrict__ y,
                               const double *__restrict__ z, const double *__restrict__ de,
                               const int32_t *__restrict__ hist, int32_t n_prim, float4 *__restrict__ ev_pos,
                               double *__restrict__ ev_e, double *__restrict__ ev_xyz, int *status)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        // cm -> um exactly as the reference's host driver (double * 10000.0f),
        // then the float the transport carries
        const double xu = x[i] * (double)10000.0f, yu = y[i] * (double)10000.0f, zu = z[i] * (double)10000.0f;
        const int32_t h = hist[i];
        const double e = de[i];
        if (!(finite_f(xu) && finite_f(yu) && finite_f(zu) && finite_f(e)) || e < 0.0 || h < 1 || h > n_prim)
            atomicOr(status, kStatusBadEvent);
        ev_pos[i] = make_float4((float)xu, (float)yu, (float)zu, __int_as_float(h - 1));
        ev_e[i] = e;
        ev_xyz[3 * i] = xu;
        ev_xyz[3 * i + 1] = yu;
        ev_xyz[3 * i + 2] = zu;
    }
}

__global__ void prep_um_kernel(int64_t n, const float *__restrict__ x, const float *__restrict__ y,
                               const float *__restrict__ z, const float *__restrict__ e,
                               const int32_t *__restrict__ hist, int32_t n_prim, float4 *__restrict__ ev_pos,
                               double *__restrict__ ev_e, double *__restrict__ ev_xyz, int *status)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t h = hist[i];
        const double ee = e ? (double)e[i] : 0.0;
        if (!(isfinite(x[i]) && isfinite(y[i]) && isfinite(z[i]) && isfinite(ee)) || ee < 0.0 || h < 1 || h > n_prim)
            atomicOr(status, kStatusBadEvent);
        ev_pos[i] = make_float4(x[i], y[i], z[i], __int_as_float(h - 1));
        ev_e[i] = ee;
        ev_xyz[3 * i] = (double)x[i];
        ev_xyz[3 * i + 1] = (double)y[i];
        ev_xyz[3 * i + 2] = (double)z[i];
    }
}

// ---------------------------------------------------------------- counts

// Uniform double in (0, 1) from two 32-bit words.
__device__ __forceinline__ double u01d(uint32_t a, uint32_t b)
{
    const uint64_t m = ((uint64_t)a << 21) ^ (uint64_t)(b >> 11);  // 53 bits
    return ((double)(m & ((1ull << 53) - 1)) + 0.5) * (1.0 / 9007199254740992.0);
}

struct CountRng {
    uint32_t k0, k1, event, tag, block;
    uint4 buf;
    int avail;
    __device__ double u()
    {
        if (avail == 0) {
            buf = philox4x32_10(make_uint4(block++, kCountStream, event, tag), k0, k1);
            avail = 2;
        }
        const double r = avail == 2 ? u01d(buf.x, buf.y) : u01d(buf.z, buf.w);
        --avail;
        return r;
    }
};

// Poisson(mu): inversion by multiplication for mu < 10; above, the
// transformed rejection with squeeze PTRS of W. Hormann, "The transformed
// rejection method for generating Poisson random variables", Insurance:
// Mathematics and Economics 12 (1993) 39-45.
__device__ int64_t poisson(CountRng &rng, double mu)
{
    if (!(mu > 0.0)) return 0;
    if (mu < 10.0) {
        const double limit = exp(-mu);
        double prod = rng.u();
        int64_t k = 0;
        while (prod > limit && k < 1000) {
            prod *= rng.u();
            ++k;
        }
        return k;
    }
    const double smu = sqrt(mu), logmu = log(mu);
    const double b = 0.931 + 2.53 * smu;
    const double a = -0.059 + 0.02483 * b;
    const double inv_alpha = 1.1239 + 1.1328 / (b - 3.4);
    const double vr = 0.9277 - 3.6224 / (b - 2.0);
    for (int it = 0; it < 10000; ++it) {
        const double U = rng.u() - 0.5;
        const double V = rng.u();
        const double us = 0.5 - fabs(U);
        const double k = floor((2.0 * a / us + b) * U + mu + 0.43);
        if (us >= 0.07 && V <= vr) return (int64_t)k;
        if (k < 0.0 || (us < 0.013 && V > us)) continue;
        if (log(V) + log(inv_alpha) - log(a / (us * us) + b) <= -mu + k * logmu - lgamma(k + 1.0))
            return (int64_t)k;
    }
    return (int64_t)floor(mu + 0.5);  // unreachable in practice
}

__global__ void count_kernel(int64_t n, int64_t event_base, int mode, double yield, int64_t max_per_event, uint64_t seed,
                             const uint32_t *__restrict__ run_tag_ptr, int chunk, const double *__restrict__ ev_e,
                             const int32_t *__restrict__ given_n, const uint16_t *__restrict__ ev_geom,
                             const float4 *__restrict__ ev_pos, int32_t *__restrict__ ev_n,
                             uint32_t *__restrict__ ev_nchunks, unsigned long long *photons_per_geom,
                             unsigned long long *photons_total, int32_t *__restrict__ prim_geom, int32_t n_prim,
                             int *status)
{
    const uint32_t run_tag = *run_tag_ptr;
    const int lane = threadIdx.x & 31;
    // the warp's lanes take events base + lane together, so that with one
    // geometry the warp adds its photon total with one atomic per counter
    // (every event adding its own count to the same two addresses
    // serialised the kernel at millions of events)
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;  // a multiple of 32
    for (int64_t base = blockIdx.x * (int64_t)blockDim.x + (threadIdx.x & ~31); base < n; base += stride) {
        const int64_t i = base + lane;
        const bool live = i < n;
        int64_t k = 0;
        int g = 0;
        if (live) {
            if (mode == kCountGiven) {
                k = given_n[i];
            } else {
                CountRng rng{(uint32_t)seed, (uint32_t)(seed >> 32), (uint32_t)(event_base + i), run_tag, 0u,
                             make_uint4(0, 0, 0, 0), 0};
                const double mu = ev_e[i] * yield;
                if (mode == kCountGaussian) {
                    const double u1 = rng.u(), u2 = rng.u();
                    const double zn = sqrt(-2.0 * log(u1)) * cospi(2.0 * u2);
                    k = (int64_t)llrint(mu + sqrt(fmax(mu, 0.0)) * zn);
                } else {
                    k = poisson(rng, mu);
                }
            }
            if (k < 0) k = 0;
            if (k > max_per_event) {
                atomicOr(status, kStatusTooManyPhotons);
                k = 0;
            }
            // an event the preparation flagged (non-finite, negative energy,
            // history outside 1..num_hist) gets no photons: a streamed ingest
            // queues its transport before the host sees the flag
            const float4 p = ev_pos[i];
            const int32_t prim = __float_as_int(p.w);
            const double e = ev_e ? ev_e[i] : 0.0;  // no energies with given counts (fd2_transport_noalloc)
            if (!(isfinite(p.x) && isfinite(p.y) && isfinite(p.z) && isfinite(e)) || e < 0.0 || prim < 0 || prim >= n_prim)
                k = 0;
            ev_n[i] = (int32_t)k;
            ev_nchunks[i] = (uint32_t)((k + chunk - 1) / chunk);
            g = ev_geom ? ev_geom[i] : 0;
            if (ev_geom && k) {
                atomicAdd(&photons_per_geom[g], (unsigned long long)k);
                if (photons_total) atomicAdd(&photons_total[g], (unsigned long long)k);
            }
            if (prim_geom && prim >= 0 && prim < n_prim) prim_geom[prim] = g;
        }
        if (!ev_geom) {
            unsigned long long t = (unsigned long long)k;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(kFull, t, o);
            if (lane == 0 && t) {
                atomicAdd(&photons_per_geom[0], t);
                if (photons_total) atomicAdd(&photons_total[0], t);
            }
        }
    }
}

// ------------------------------------------------------------------ scan

constexpr int kScanBlock = 1024;
constexpr int kScanItems = 4;
constexpr int kScanTile = kScanBlock * kScanItems;

template <typename T>
__device__ unsigned long long block_exclusive_scan(unsigned long long v, unsigned long long *warp_sums,
                                                   unsigned long long *total)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    unsigned long long x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(kFull, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[wid] = x;
    __syncthreads();
    if (wid == 0) {
        unsigned long long s = lane < (int)(blockDim.x >> 5) ? warp_sums[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long y = __shfl_up_sync(kFull, s, o);
            if (lane >= o) s += y;
        }
        warp_sums[lane] = s;
    }
    __syncthreads();
    const unsigned long long before = wid ? warp_sums[wid - 1] : 0;
    *total = warp_sums[(blockDim.x >> 5) - 1];
    return before + x - v;
}

// Pass 1: per-tile exclusive scan into offsets, tile totals into block_sums.
template <typename In>
__global__ void scan_tiles(int64_t n, const In *__restrict__ in, unsigned long long *__restrict__ out,
                           unsigned long long *__restrict__ block_sums)
{
    __shared__ unsigned long long warp_sums[32];
    const int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems;
    unsigned long long v[kScanItems], sum = 0;
#pragma unroll
    for (int j = 0; j < kScanItems; ++j) {
        v[j] = (base + j < n) ? (unsigned long long)in[base + j] : 0ull;
        sum += v[j];
    }
    unsigned long long total;
    unsigned long long run = block_exclusive_scan<unsigned long long>(sum, warp_sums, &total);
#pragma unroll
    for (int j = 0; j < kScanItems; ++j) {
        if (base + j < n) out[base + j] = run;
        run += v[j];
    }
    if (threadIdx.x == 0) block_sums[blockIdx.x] = total;
}

// Pass 2: exclusive scan of the tile totals (one CTA, looping).
__global__ void scan_sums(int64_t tiles, unsigned long long *block_sums, unsigned long long *total)
{
    __shared__ unsigned long long warp_sums[32];
    unsigned long long carry = 0;
    for (int64_t b = 0; b < tiles; b += blockDim.x) {
        const int64_t i = b + threadIdx.x;
        const unsigned long long v = i < tiles ? block_sums[i] : 0ull;
        unsigned long long t;
        const unsigned long long ex = block_exclusive_scan<unsigned long long>(v, warp_sums, &t);
        if (i < tiles) block_sums[i] = carry + ex;
        carry += t;
        __syncthreads();
    }
    if (threadIdx.x == 0) *total = carry;
}

// Pass 3: add tile offsets.
__global__ void scan_add(int64_t n, unsigned long long *__restrict__ out, const unsigned long long *__restrict__ block_sums)
{
    const int64_t base = (int64_t)blockIdx.x * kScanTile;
    const unsigned long long add = block_sums[blockIdx.x];
    for (int j = threadIdx.x; j < kScanTile; j += blockDim.x)
        if (base + j < n) out[base + j] += add;
}

template <typename In>
cudaError_t scan_impl(cudaStream_t s, int64_t n, const In *in, unsigned long long *offsets,
                      unsigned long long *block_sums, unsigned long long *total)
{
    const int64_t tiles = (n + kScanTile - 1) / kScanTile;
    if (n > 0) {
        scan_tiles<In><<<(unsigned)tiles, kScanBlock, 0, s>>>(n, in, offsets, block_sums);
    }
    scan_sums<<<1, kScanBlock, 0, s>>>(tiles, block_sums, total);
    if (n > 0) scan_add<<<(unsigned)tiles, 256, 0, s>>>(n, offsets, block_sums);
    return cudaGetLastError();
}

__global__ void fill_chunks_kernel(int64_t n, int chunk, const int32_t *__restrict__ ev_n,
                                   const unsigned long long *__restrict__ offsets, uint2 *__restrict__ chunks,
                                   int64_t capacity, int *status)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t k = ev_n[i];
        const unsigned long long off = offsets[i];
        const int32_t nc = (k + chunk - 1) / chunk;
        if ((int64_t)(off + nc) > capacity) {
            atomicOr(status, kStatusChunkOverflow);
            continue;
        }
        for (int32_t c = 0; c < nc; ++c) chunks[off + c] = make_uint2((uint32_t)i, (uint32_t)(c * chunk));
    }
}

// ------------------------------------------------------------- transport

struct Slot {
    float4 pos;      // event x, y, z and history index bits
    uint32_t event;  // event index
    uint32_t first;  // first photon of the chunk
    uint32_t count;  // photons in the chunk
    uint32_t geom;
};
constexpr int kRing = 32;
// Photons a warp holds beside its lanes' (in shared memory), of each kind, and
// the 16-byte words of one: position, direction, column centre, absorption
// budget, boundary count, tag, event, random state.
constexpr int kPark = 32;
constexpr int kParkWords = 4;
constexpr int kParkKind = kPark * kParkWords;  // words from one kind's photons to the other's
// Ended photons a warp holds: fewer than 32 wait, and up to 32 end in a pass.
constexpr int kEnded = 64;

// A warp's shared memory: its parked photons (those that wait at a wall, and
// those that wait for a hop), its ended photons and its ring of chunks.
struct WarpMem {
    float4 park[2 * kParkKind];
    float park_dist[2 * kPark];  // path lengths, where they are summed by geometry
    float4 ended[kEnded];
    Slot ring[kRing];
    int slot, len;   // the ring's current slot and its filled slots
    uint32_t used;   // photons of the current slot handed out
    uint32_t pad;
};

// Shared-memory layout of the transport kernel (dynamic): the warps' blocks,
// at constant offsets of the warp's base so that one register addresses them.
struct SmemLayout {
    size_t geom, cnt, dist, win, total;
    __host__ __device__ SmemLayout(int block, int n_geom, int window)
    {
        size_t o = sizeof(WarpMem) * (size_t)(block / 32);
        geom = o;
        o += n_geom > 1 ? sizeof(DevGeom) * (size_t)n_geom : 0;
        cnt = o;
        o += n_geom > 1 ? 0 : sizeof(unsigned) * kCounterStride;  // kAgg: one geometry
        dist = o;
        o += sizeof(float) * (size_t)n_geom;
        o = (o + 15) & ~(size_t)15;
        win = o;
        o += sizeof(unsigned) * (size_t)window * window;
        total = o;
    }
};

// Tallies of ended photons, one per lane of `lanes` (e: the place; event index;
// fate and geometry): fate and
// per-history counts with one reduction per distinct address of the warp, the
// PRF pixel with one of its lane.
template <bool kMulti, bool kRadial, bool kAgg>
__device__ __forceinline__ void tally_ended(const TransportArgs &a, const DevGeom *s_geom, unsigned *s_cnt,
                                            unsigned *s_win, const float4 &e, unsigned lanes)
{
    const int lane = threadIdx.x & 31;
    const int code = __float_as_int(e.w), fate = code & 0xff, geom = kMulti ? code >> 8 : 0;
    const float4 ev = a.ev_pos[__float_as_uint(e.z)];
    const int prim = __float_as_int(ev.w);
    const DevGeom &g = kMulti ? s_geom[geom] : a.g0;
    const unsigned key = (unsigned)(geom * kCounterStride + fate);
    unsigned peers = __match_any_sync(lanes, key);
    if (lane == __ffs(peers) - 1) {
        if (kAgg) atomicAdd(&s_cnt[key], (unsigned)__popc(peers));
        else atomicAdd(&a.counters[key], (unsigned long long)__popc(peers));
    }
    const unsigned det = __ballot_sync(lanes, fate == kDetect);
    if (fate != kDetect) return;
    const bool counted = (unsigned)prim < (unsigned)a.n_prim;
    peers = __match_any_sync(det, prim);
    if (lane == __ffs(peers) - 1 && counted) atomicAdd(&a.per_primary[prim], __popc(peers));
    if (kRadial) {
        // quadratic edges: bin = floor(bins sqrt(r / r_max))
        const float rx = e.x - ev.x, ry = e.y - ev.y;
        const float rr = sqrtf(rx * rx + ry * ry) * a.radial_inv_max;
        const int b = rr < 1.0f ? min((int)(sqrtf(rr) * (float)a.radial_bins), a.radial_bins - 1) : a.radial_bins;
        if (counted && b >= 0) atomicAdd(&a.radial[(long long)prim * (a.radial_bins + 1) + b], 1u);
        return;
    }
    int ii, jj;
    detection_pixel(g, e.x, e.y, ii, jj);
    const bool in = ii >= 0 && jj >= 0 && ii < g.xdim && jj < g.ydim;
    const unsigned seen = __ballot_sync(det, in);
    if (!in) return;
    // geometry by geometry where the warp's photons have several
    peers = kMulti ? __match_any_sync(seen, geom) : seen;
    if (lane == __ffs(peers) - 1) {
        if (kAgg) atomicAdd(&s_cnt[kNumFates], (unsigned)__popc(peers));
        else atomicAdd(&a.counters[geom * kCounterStride + kNumFates], (unsigned long long)__popc(peers));
    }
    const int win = a.window, wx = ii - a.win_x0, wy = jj - a.win_y0;
    if (kAgg && win > 0 && (unsigned)wx < (unsigned)win && (unsigned)wy < (unsigned)win)
        atomicAdd(&s_win[wx * win + wy], 1u);
    else
        atomicAdd(&a.prf[g.prf_offset + (long long)ii * g.ydim + jj], 1ull);
}

// Persistent transport.  Each warp keeps a ring of up to 32 chunk slots in
// shared memory, filled with one coalesced load per lane; each lane runs one
// photon at a time and takes another as soon as (or, with refill > 1, once
// enough lanes of the warp are) idle, so lanes never wait for the longest walk
// in the warp.  What bounds the kernel is instruction issue, so what counts is
// how many lanes of a warp share each instruction.  Photons that wait for the
// rarer, longer parts of the walk (the Fresnel part at a wall, the hop between
// columns after it; with a column lattice the flight through the gap) leave
// their lane for the warp's shared memory (up to 32 of either kind, 64 bytes
// each) and the lane goes on with another photon; once `fresnel_batch` wait,
// they are exchanged into the lanes and that part runs for all of them, the
// photons they displaced waiting as ready ones.  Run in the lane they wait in,
// beside 8 others, those parts had 9 lanes (the hops 2 to 3) and a third of the
// warps' time: 20,000 config-1 x-rays 59.1 ms that way, 38.7 this way; 10,001
// x-rays in the square / hexagonal lattice 102.5 / 142.9 and 60.9 / 83.0.  Per
// photon 843 warp instructions at 23.8 of 32 lanes, issue slots 88 % busy; in
// the square / hexagonal lattice 2,731 at 19.6, 91 % / 3,442 at 18.0, 84 %.
// Tallies:
// ended photons are tallied 32 at a time (tally_ended) with L2 reductions;
// with kAgg (tally_mode 1) the fates and the PRF core of geometry 0 are
// tallied in shared memory first (identical tallies).  kMulti: the
// geometry of each photon comes from the table in shared memory; otherwise
// the single geometry is read from the kernel parameters.  kRadial (label
// mode): a detected photon is binned by its distance from its event into
// the history's radial histogram instead of the PRF image.
template <bool kMulti, int kMaxThreads, int kMinBlocks, bool kRadial = false, bool kGrid = false, bool kAgg = false>
__global__ void __launch_bounds__(kMaxThreads, kMinBlocks) transport_kernel(const __grid_constant__ TransportArgs a)
{
    // of the column lattices, four CTAs per SM walk the square one only
    constexpr bool kSquare = kGrid && kMinBlocks == 4;
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int win = a.window;
    const SmemLayout L(blockDim.x, a.n_geom, win);
    DevGeom *s_geom = reinterpret_cast<DevGeom *>(smem + L.geom);
    unsigned int *s_cnt = reinterpret_cast<unsigned int *>(smem + L.cnt);
    float *s_dist = reinterpret_cast<float *>(smem + L.dist);
    unsigned int *s_win = reinterpret_cast<unsigned int *>(smem + L.win);

    if (kMulti)
        for (int i = threadIdx.x; i < a.n_geom; i += blockDim.x) s_geom[i] = a.geoms[i];
    if (kAgg)
        for (int i = threadIdx.x; i < kCounterStride; i += blockDim.x) s_cnt[i] = 0;
    for (int i = threadIdx.x; i < a.n_geom; i += blockDim.x) s_dist[i] = 0.0f;
    for (int i = threadIdx.x; i < win * win; i += blockDim.x) s_win[i] = 0;
    __syncthreads();

    WarpMem &m = reinterpret_cast<WarpMem *>(smem)[wid];
    if (lane == 0) {
        m.slot = m.len = 0;
        m.used = 0;
    }
    bool exhausted = false;
    int state = 0;  // of the lane: no photon, a fate not yet recorded, or Flight
    int xtries = 0; // tries at the crosstalk normal of a kRetryNormal photon
    // Philox round keys and run counter, shared by the CTA
    __shared__ uint32_t s_rk[20];
    __shared__ uint32_t s_run;
    if (threadIdx.x < 20) s_rk[threadIdx.x] = a.round_keys[threadIdx.x];
    if (threadIdx.x == 0) s_run = *a.run_tag;

    Walker w;
    constexpr uint32_t kGeomBits = Walker::kGeomBits;
    uint32_t tag = 0, event = 0;  // the photon's tag (Walker::kGeomBits ...) and event
    w.dist = 0.0f;
    // the lane's path-length sum
    __shared__ float s_ldist[kMaxThreads];
    s_ldist[threadIdx.x] = 0.0f;
    // Of either kind of parked photons, [0, n_wait) wait and
    // [n_wait, n_wait + n_ready) are ready (never more than kPark - 1
    // together: a photon is added only while fewer than `batch` wait and none
    // is ready).
    int n_wait = 0, n_ready = 0, n_hop = 0, n_hready = 0;
    int n_ended = 0;  // ended photons not yet tallied
    __syncthreads();
    const RngKey key{s_rk, s_run};

    for (;;) {
        // ---- photons that ended: kept in shared memory (place, history,
        // fate and geometry) until a warp's worth is tallied together.  One to
        // two photons end in a step, and their pixel's two divisions and their
        // reductions cost the warp as many instructions as 32 photons' do.
        const unsigned live = __ballot_sync(kFull, state >= kFlies);
        const unsigned some = __ballot_sync(kFull, state != 0);
        const unsigned odd = __ballot_sync(kFull, (state & 1) != 0);
        const unsigned late = __ballot_sync(kFull, (state & 2) != 0) & live;
        unsigned run = live & ~late;
        const unsigned held = kGrid ? late : late & ~odd, hops = kGrid ? 0u : late & odd;
        if (some != live) {
            const unsigned over = some & ~live;
            if (state != 0 && state < kFlies) {
                m.ended[n_ended + __popc(over & lanemask_lt())] =
                    make_float4(w.px, w.py, __uint_as_float(event), __int_as_float((int)(tag & kGeomBits) << 8 | state));
                if (kMulti) {
                    atomicAdd(&s_dist[tag & kGeomBits], w.dist);
                } else {
                    s_ldist[threadIdx.x] += w.dist;  // lane-private: no atomic
                    w.dist = 0.0f;
                }
                state = 0;
            }
            n_ended += __popc(over);
        }
        // ---- which pass: steps of the lanes' photons, or the waiting ones
        const int n_held = __popc(held), n_hops = __popc(hops);
        const int waiting = n_wait + n_held, hopping = n_hop + n_hops;
        bool supply = n_ready + n_hready > 0 || !exhausted;
        const bool finished = !run && !supply && waiting + hopping == 0;
        while (n_ended >= 32 || (finished && n_ended > 0)) {
            const int n = min(n_ended, 32);
            n_ended -= n;
            __syncwarp();
            if (lane < n)
                tally_ended<kMulti, kRadial, kAgg>(a, s_geom, s_cnt, s_win, m.ended[n_ended + lane],
                                                   kFull >> (32 - n));
            __syncwarp();
        }
        if (finished) break;
        int at = -1;     // the parked photon this lane exchanges its own with
        int moved = 0;   // lanes that do
        bool flush = false, hop = false, deal = false;
        // Once the queue and the ready photons are used up every waiting photon
        // starts a pass: more would only hold up the last photons, whose serial
        // walks are what a small run takes (25 / 400 / 2,311 x-rays with passes
        // from 1 photon 0.35 / 0.74 / 5.60 ms, from 2 0.37 / 0.74 / 5.61, from
        // 8 0.49 / 0.85 / 5.84).
        const int batch = supply ? a.fresnel_batch : 1;
        if (waiting >= batch || hopping >= batch) {
            // waiting photons into the lanes that hold none of their kind:
            // first the empty lanes (when no photon is ready among them), then
            // lanes whose photon can wait as a ready one.  Without a lane that
            // can run one, the others step first.
            const unsigned none = ~live, other = run & ~odd;
            const int n_none = __popc(none), n_other = __popc(other);
            hop = !kGrid && hopping >= batch && (n_hops > 0 || n_other > 0 || (n_hready == 0 && n_none > 0));
            flush = hop || (waiting >= batch && (n_held > 0 || n_other > 0 || (n_ready == 0 && n_none > 0)));
            if (flush) {
                const int nw = hop ? n_hop : n_wait, nr = hop ? n_hready : n_ready;
                const unsigned take = nr == 0 ? none : 0u;
                const int n_take = __popc(take);
                moved = min(nw, n_take + n_other);
                const bool empty = (take >> lane) & 1u;
                const int rank = empty ? __popc(take & lanemask_lt()) : n_take + __popc(other & lanemask_lt());
                if ((((take | other) >> lane) & 1u) && rank < moved) at = (hop ? kParkKind : 0) + nw - 1 - rank;
                const int ready = nr + moved - min(moved, n_take);
                (hop ? n_hop : n_wait) = nw - moved;
                (hop ? n_hready : n_ready) = ready;
            }
        }
        if (!flush && supply && (32 - __popc(run) >= (exhausted ? 1 : a.refill) || !run)) {
            // lanes with a waiting photon park it, for a ready one of its kind
            // if there is one; empty lanes take ready ones; the rest get new
            // photons
            const int n_none = 32 - __popc(live);
            const int left = max(n_ready - n_held, 0), hleft = max(n_hready - n_hops, 0);
            const int taken = min(left, n_none), htaken = min(hleft, n_none - taken);
            const bool flying = (run >> lane) & 1u;
            const bool at_wall = state == kWaits, hopper = !kGrid && state == kHops;
            const unsigned same = at_wall ? held : hopper ? hops : ~live;
            const int rank = __popc(same & lanemask_lt());
            const bool got = rank < (at_wall ? n_ready : hopper ? n_hready : taken + htaken);
            const int own = (at_wall ? n_wait : kParkKind + n_hop) + rank;
            const int next = (rank < taken ? n_wait + n_ready : kParkKind + n_hop + n_hready + taken) - 1 - rank;
            at = at_wall || hopper ? own : got ? next : -1;
            at = flying ? -1 : at;
            state = flying ? state : got ? kFlies : 0;
            moved = n_held + n_hops + taken + htaken;
            n_wait += n_held;
            n_hop += n_hops;
            n_ready = left - taken;
            n_hready = hleft - htaken;
            deal = !exhausted;
        }
        if (moved) {
            __syncwarp();
            if (at >= 0) {
                float4 *q = m.park + at, t = q[0];
                q[0] = make_float4(w.px, w.py, w.pz, w.dx);
                w.px = t.x, w.py = t.y, w.pz = t.z, w.dx = t.w;
                t = q[kPark];
                q[kPark] = make_float4(w.dy, w.dz, w.xc, w.yc);
                w.dy = t.x, w.dz = t.y, w.xc = t.z, w.yc = t.w;
                t = q[2 * kPark];
                q[2 * kPark] = make_float4(w.budget, __uint_as_float(w.rebound), __uint_as_float(tag),
                                           __uint_as_float(event));
                if (kMulti) {
                    float &pd = m.park_dist[at < kParkKind ? at : at - kParkKind + kPark];
                    const float d = pd;
                    pd = w.dist;
                    w.dist = d;
                }
                w.budget = t.x, w.rebound = __float_as_uint(t.y), tag = __float_as_uint(t.z);
                event = __float_as_uint(t.w);
                t = q[3 * kPark];
                q[3 * kPark] = make_float4(__uint_as_float(w.s0), __uint_as_float(w.s1), __uint_as_float(w.s2),
                                           __uint_as_float(w.s3));
                w.s0 = __float_as_uint(t.x), w.s1 = __float_as_uint(t.y);
                w.s2 = __float_as_uint(t.z), w.s3 = __float_as_uint(t.w);
                if (flush) state = !kGrid && hop ? kHops : kWaits;
            }
            __syncwarp();
        }
        if (flush) {
            // ---- the waiting photons' pass
            if (state == (!kGrid && hop ? kHops : kWaits)) {
                if constexpr (kGrid) {
                    state = w.grid_segment<kSquare, false>(a.g0);
                } else {
                    state = kMulti ? w.surface_wait(s_geom[tag & kGeomBits], hop, tag) : w.surface_wait(a.g0, hop, tag);
                }
            }
            continue;
        }
        // ---- hand out photons to idle lanes
        unsigned needy = __ballot_sync(kFull, state == 0);
        if (deal && needy && (__popc(needy) >= a.refill || needy == kFull)) {
            // (which photon first; they start together below, also where the
            // lanes' photons come from several chunks)
            int slot = m.slot, len = m.len;
            bool fresh = false;
            uint32_t first = 0;  // the photon's number in its event
            uint32_t used = m.used;
            while (needy) {
                if (slot >= len) {
                    // A refill takes a share of what is left: 32 chunks while
                    // every warp can still take that many twice, then fewer,
                    // down to one, so that a small run spreads over the warps
                    // (always taking 32 chunks gave a 25-x-ray run to 66 of
                    // 4,736 warps) and a large one ends evenly.
                    // The abort flag lies in host memory: one warp of the
                    // grid polls it and the others see the device's status
                    // word.  Every warp reading it at its first refill queued
                    // 4,736 reads on PCIe, 4.2 ms of every launch.
                    unsigned long long base = 0;
                    int take = 0;
                    if (lane == 0) {
                        if (a.abort_flag && blockIdx.x == 0 && wid == 0 && *a.abort_flag)
                            atomicOr(a.status, kStatusAborted);
                        const unsigned long long head = *(const volatile unsigned long long *)a.queue_head;
                        if (!(*(const volatile int *)a.status & kStatusAborted)) {
                            const unsigned long long total = min(*a.n_chunks, (unsigned long long)a.chunk_capacity);
                            const unsigned long long left = total > head ? total - head : 0ull;
                            take = (int)min(max(left >> a.pull_shift, 1ull), (unsigned long long)kRing);
                            base = atomicAdd(a.queue_head, (unsigned long long)take);
                            // never read past the chunk buffer, whatever the scan produced
                            if (base + take > total) take = base < total ? (int)(total - base) : 0;
                        }
                    }
                    take = __shfl_sync(kFull, take, 0);
                    base = __shfl_sync(kFull, base, 0);
                    if (take == 0) {
                        exhausted = true;
                        break;
                    }
                    const unsigned long long idx = base + lane;
                    const bool ok = lane < take;
                    __syncwarp();  // every lane is done reading the old ring
                    if (ok) {
                        const uint2 c = a.chunks[idx];
                        Slot s;
                        s.pos = a.ev_pos[c.x];
                        s.event = c.x;
                        s.first = c.y;
                        const int32_t n = a.ev_n[c.x];
                        s.count = (uint32_t)min(a.chunk, n - (int32_t)c.y);
                        s.geom = (kMulti && a.ev_geom) ? a.ev_geom[c.x] : 0;
                        m.ring[lane] = s;
                    }
                    len = take;
                    __syncwarp();
                    slot = 0;
                    used = 0;
                }
                const uint32_t count = m.ring[slot].count;
                if (used >= count) {
                    ++slot;
                    used = 0;
                    continue;
                }
                const unsigned take = min((unsigned)(count - used), (unsigned)__popc(needy));
                const unsigned rank = __popc(needy & lanemask_lt());
                const bool mine = ((needy >> lane) & 1u) && rank < take;
                if (mine) {
                    const Slot &s = m.ring[slot];
                    first = s.first + used + rank;
                    tag = s.geom;
                    event = s.event;
                    w.px = s.pos.x;
                    w.py = s.pos.y;
                    w.pz = s.pos.z;
                    fresh = true;
                }
                needy &= ~__ballot_sync(kFull, mine);
                used += take;
            }
            if (lane == 0) {
                m.slot = slot;
                m.len = len;
                m.used = used;
            }
            if (fresh) {
                if (kMulti) w.dist = 0.0f;
                w.start(w.px, w.py, w.pz, first, (uint32_t)(a.event_base + event), first == 0, key);
                state = kFlies;
                if constexpr (kGrid) {
                    if (w.grid_place<kSquare>(a.g0)) state = kWaits;
                } else if constexpr (kMulti) {
                    w.fill_budget(s_geom[tag & kGeomBits]);
                } else {
                    w.fill_budget(a.g0);
                }
            }
            __syncwarp();
            supply = n_ready > 0 || !exhausted;
        }
        // ---- steps of the lanes' photons until enough lanes are idle to make
        // the exchange worth its instructions; with nothing to fill them, until
        // one more is
        // (in flight and not waiting: kFlies or kRetryNormal)
        run = __ballot_sync(kFull, (state & 10) == 8);
        if (!run) continue;
        const int stay = supply ? 33 - a.refill : __popc(run);
        do {
            if ((state & 10) == 8) {
                if constexpr (kGrid) {
                    // explicit column lattice: one segment, of a photon in a column
                    state = w.grid_segment<kSquare, true>(a.g0);
                } else {
                    int f = kNeedsNormal;
                    if (state == kFlies) {
                        xtries = 0;
                        f = kMulti ? w.step(s_geom[tag & kGeomBits], a.ev_pos + event, tag)
                                   : w.step(a.g0, a.ev_pos + event, tag);
                    }
                    // crosstalk: one attempt at the next column's normal per
                    // step, so a rejected attempt is retried beside the other
                    // lanes' first ones
                    if (f == kNeedsNormal)
                        f = kMulti ? w.crosstalk_normal(s_geom[tag & kGeomBits], xtries)
                                   : w.crosstalk_normal(a.g0, xtries);
                    state = f;
                }
            }
            run = __ballot_sync(kFull, (state & 10) == 8);
        } while (__popc(run) >= stay);
    }

    // ---- flush the CTA's private tallies
    __syncthreads();
    if (kAgg)
        for (int i = threadIdx.x; i < kCounterStride; i += blockDim.x)
            if (s_cnt[i]) atomicAdd(&a.counters[i], (unsigned long long)s_cnt[i]);
    if (!kMulti) {
        // the lanes' path-length sums: summed per warp in double, then added to the CTA's
        double d = (double)s_ldist[threadIdx.x] + (double)w.dist;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(kFull, d, o);
        if (lane == 0 && d != 0.0) atomicAdd(&a.distance[0], d);
    }
    for (int i = threadIdx.x; i < a.n_geom; i += blockDim.x)
        if (s_dist[i] != 0.0f) atomicAdd(&a.distance[i], (double)s_dist[i]);
    if (win > 0) {
        const long long off = kMulti ? s_geom[0].prf_offset : a.g0.prf_offset;
        const int ydim = kMulti ? s_geom[0].ydim : a.g0.ydim;
        for (int i = threadIdx.x; i < win * win; i += blockDim.x) {
            const unsigned v = s_win[i];
            if (v) {
                const int ii = a.win_x0 + i / win, jj = a.win_y0 + i % win;
                atomicAdd(&a.prf[off + (long long)ii * ydim + jj], (unsigned long long)v);
            }
        }
    }
}

// -------------------------------------------------------------------- PHS

// PHS binning of the reference (hybridMANTIS_cuda_ver1_0.cu:376-399) per
// geometry, plus FP64 moments over histories with >= 1 detected photon.
__global__ void phs_kernel(int32_t n_prim, const int32_t *__restrict__ per_primary,
                           const int32_t *__restrict__ prim_geom, int n_geom, int32_t min_photons,
                           int32_t max_photons, int32_t num_bins, int32_t width, int32_t shift,
                           int32_t *__restrict__ phs, double *__restrict__ moments,
                           unsigned long long *dropped)
{
    const int lane = threadIdx.x & 31;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t base = (int64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31); base < n_prim; base += stride) {
        const int64_t i = base + lane;
        const int32_t c = i < n_prim ? per_primary[i] : 0;
        const int g = (i < n_prim && prim_geom) ? prim_geom[i] : 0;
        const bool has = c > 0 && g >= 0 && g < n_geom;
        if (has) {
            int32_t bin;
            if (c <= min_photons) bin = 0;
            else if (c >= max_photons) bin = num_bins - 1;
            else bin = c / width - shift;
            if (bin >= 0 && bin < num_bins) atomicAdd(&phs[(int64_t)g * num_bins + bin], 1);
            else atomicAdd(&dropped[g], 1ull);
        }
        // FP64 moments, summed over the lanes of the warp with the same geometry
        const unsigned m = __ballot_sync(kFull, has);
        if (has) {
            const unsigned peers = __match_any_sync(m, g);
            const double v1 = (double)c, v2 = (double)c * (double)c;
            double a1 = 0.0, a2 = 0.0;
            for (unsigned q = peers; q; q &= q - 1) {
                const int src = __ffs(q) - 1;
                a1 += __shfl_sync(peers, v1, src);
                a2 += __shfl_sync(peers, v2, src);
            }
            if (lane == __ffs(peers) - 1) {
                atomicAdd(&moments[g * 3 + 0], (double)__popc(peers));
                atomicAdd(&moments[g * 3 + 1], a1);
                atomicAdd(&moments[g * 3 + 2], a2);
            }
        }
    }
}

__global__ void bump_kernel(uint32_t *run_tag) { *run_tag += 1u; }

// The walk's wall root (the far intersection with the column) for given
// quadratic coefficients, compiled with the transport's flags.
__global__ void wall_root_kernel(int n, const float *__restrict__ qa, const float *__restrict__ qb,
                                 const float *__restrict__ qc, float *__restrict__ out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = wall_root(qa[i], qb[i], qc[i]);
}

}  // namespace

// ------------------------------------------------------------- launchers

cudaError_t launch_bump_run_tag(cudaStream_t s, uint32_t *run_tag)
{
    bump_kernel<<<1, 1, 0, s>>>(run_tag);
    return cudaGetLastError();
}

static unsigned grid_for(int64_t n, int block, int cap = 148 * 32)
{
    int64_t g = (n + block - 1) / block;
    if (g < 1) g = 1;
    if (g > cap) g = cap;
    return (unsigned)g;
}

cudaError_t launch_prep_cm(cudaStream_t s, int64_t n, const double *x_cm, const double *y_cm, const double *z_cm,
                           const double *de, const int32_t *hist, int32_t n_prim, float4 *ev_pos, double *ev_e,
                           double *ev_xyz, int *status)
{
    if (n <= 0) return cudaSuccess;
    prep_cm_kernel<<<grid_for(n, 256), 256, 0, s>>>(n, x_cm, y_cm, z_cm, de, hist, n_prim, ev_pos, ev_e, ev_xyz,
                                                    status);
    return cudaGetLastError();
}

cudaError_t launch_prep_um(cudaStream_t s, int64_t n, const float *x, const float *y, const float *z, const float *e,
                           const int32_t *hist, int32_t n_prim, float4 *ev_pos, double *ev_e, double *ev_xyz,
                           int *status)
{
    if (n <= 0) return cudaSuccess;
    prep_um_kernel<<<grid_for(n, 256), 256, 0, s>>>(n, x, y, z, e, hist, n_prim, ev_pos, ev_e, ev_xyz, status);
    return cudaGetLastError();
}

cudaError_t launch_count(cudaStream_t s, int64_t n, int64_t event_base, int mode, double yield, int64_t max_per_event, uint64_t seed,
                         const uint32_t *run_tag, int chunk, const double *ev_e, const int32_t *given_n,
                         const uint16_t *ev_geom, const float4 *ev_pos, int32_t *ev_n, uint32_t *ev_nchunks,
                         unsigned long long *photons_per_geom, unsigned long long *photons_total,
                         int32_t *prim_geom, int32_t n_prim, int *status)
{
    if (n <= 0) return cudaSuccess;
    count_kernel<<<grid_for(n, 128), 128, 0, s>>>(n, event_base, mode, yield, max_per_event, seed, run_tag, chunk, ev_e, given_n,
                                                  ev_geom, ev_pos, ev_n, ev_nchunks, photons_per_geom, photons_total,
                                                  prim_geom, n_prim, status);
    return cudaGetLastError();
}

size_t scan_block_sums_needed(int64_t n) { return (size_t)((n + kScanTile - 1) / kScanTile) + 1; }

cudaError_t launch_scan(cudaStream_t s, int64_t n, const uint32_t *in, unsigned long long *offsets,
                        unsigned long long *block_sums, unsigned long long *total)
{
    return scan_impl<uint32_t>(s, n, in, offsets, block_sums, total);
}

cudaError_t launch_photon_offsets(cudaStream_t s, int64_t n, const int32_t *ev_n, unsigned long long *first,
                                  unsigned long long *block_sums, unsigned long long *total)
{
    return scan_impl<int32_t>(s, n, ev_n, first, block_sums, total);
}

cudaError_t launch_fill_chunks(cudaStream_t s, int64_t n, int chunk, const int32_t *ev_n,
                               const unsigned long long *offsets, uint2 *chunks, int64_t capacity, int *status)
{
    if (n <= 0) return cudaSuccess;
    fill_chunks_kernel<<<grid_for(n, 256), 256, 0, s>>>(n, chunk, ev_n, offsets, chunks, capacity, status);
    return cudaGetLastError();
}

// Register budgets: blocks of up to 256 threads are compiled for 2, 3 or 4
// resident CTAs per SM (128, 85, 64 registers), blocks of 320 threads for
// two (102 registers: 20 warps per SM; the walk fits without spills, 352
// threads would spill), other larger blocks for one.
#define FD2_TRANSPORT_VARIANTS(X)                                                          \
    X(false, 512, 1, false, false, false) X(false, 256, 2, false, false, false)            \
    X(false, 320, 2, false, false, false) X(true, 320, 2, false, false, false)             \
    X(false, 256, 2, false, true, false) X(false, 320, 2, false, true, false)              \
    X(false, 256, 3, false, false, false) X(false, 256, 4, false, false, false)            \
    X(true, 512, 1, false, false, false) X(true, 256, 2, false, false, false)              \
    X(true, 256, 3, false, false, false) X(true, 256, 3, true, false, false)               \
    X(true, 256, 4, false, false, false) X(false, 256, 3, false, true, false)              \
    X(false, 256, 4, false, true, false)                                                   \
    X(false, 512, 1, false, false, true) X(false, 256, 2, false, false, true)              \
    X(false, 320, 2, false, false, true) X(false, 256, 3, false, false, true)              \
    X(false, 256, 4, false, false, true) X(false, 256, 4, true, false, false)

cudaError_t prepare_transport(const TransportConfig &cfg, int n_geom)
{
    // The attribute is global to each kernel, shared by every context of the
    // process, so it is set to the device's opt-in maximum (a launch only
    // reserves what it asks for): contexts with different shared-memory
    // needs cannot undo each other's setting.
    int dev = 0, max_optin = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&max_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e != cudaSuccess) return e;
    const size_t need = transport_smem_bytes(cfg, n_geom);
    // dynamic limit = opt-in maximum - the kernel's static shared memory
#define FD2_SET_ATTR(M, T, B, R, L, A)                                                                       \
    if (e == cudaSuccess) {                                                                               \
        cudaFuncAttributes fa;                                                                            \
        e = cudaFuncGetAttributes(&fa, transport_kernel<M, T, B, R, L, A>);                                  \
        const int lim = max_optin - (int)fa.sharedSizeBytes;                                              \
        if (e == cudaSuccess && need > (size_t)lim) e = cudaErrorInvalidValue;                            \
        if (e == cudaSuccess)                                                                             \
            e = cudaFuncSetAttribute(transport_kernel<M, T, B, R, L, A>, cudaFuncAttributeMaxDynamicSharedMemorySize, lim); \
    }
    FD2_TRANSPORT_VARIANTS(FD2_SET_ATTR)
#undef FD2_SET_ATTR
    return e;
}

size_t transport_smem_bytes(const TransportConfig &cfg, int n_geom)
{
    return SmemLayout(cfg.block, n_geom, cfg.window).total;
}

// The CTAs per SM of a launch.  Label mode has one kernel for one geometry (the
// surrogate's audit), with the production run's four CTAs per SM whatever
// ctas_per_sm says, and one for several (training labels) with three (80
// registers without a spill; 25,600 points x 4,000 photons in 64 geometries: 66.8
// ms, 82 with two).  From 182 geometries on the table beside the parked photons
// leaves room for two CTAs on an SM, and the third of each runs when the queue is
// empty (182 / 256 geometries: 82.8 / 83.4 ms).  A single geometry never goes to a kMulti kernel:
// SmemLayout keeps its geometry table for several geometries only.
int transport_ctas(const TransportConfig &cfg, int n_geom, bool label)
{
    if (cfg.grid_ctas) return cfg.grid_ctas;
    if (label) return n_geom > 1 ? 3 : 4;
    return cfg.ctas_per_sm;
}

cudaError_t launch_transport(cudaStream_t s, const TransportConfig &cfg, int sm_count, const TransportArgs &args)
{
    TransportArgs a = args;
    const size_t smem = transport_smem_bytes(cfg, a.n_geom);
    const bool multi = a.n_geom > 1;
    const unsigned grid = (unsigned)(sm_count * transport_ctas(cfg, a.n_geom, a.radial != nullptr));
    a.refill = std::min(std::max(a.refill, 1), 32);
    a.fresnel_batch = std::min(std::max(a.fresnel_batch, 1), kPark);
    // a refill takes 1 / 2^pull_shift of the chunks left: at most half of a
    // warp's even share
    for (a.pull_shift = 1; (1ll << a.pull_shift) < 2ll * grid * (cfg.block / 32); ++a.pull_shift) {
    }
    const int per_sm = cfg.block > 256 ? 1 : std::min(std::max(cfg.ctas_per_sm, 2), 4);
    if (a.g0.grid) {
        // explicit column lattice: single geometry, 256 or 320 threads
        if (multi || a.radial) return cudaErrorInvalidConfiguration;
        // four CTAs per SM for the square lattice only (10,001 x-rays 60.9 ms,
        // 64.5 with three): compiled for 64 registers, the test of a hexagonal
        // lattice's neighbour columns is contracted differently, and 9,092 of
        // 10,001 x-rays would count other photons
        if (cfg.block == 320) transport_kernel<false, 320, 2, false, true><<<grid, cfg.block, smem, s>>>(a);
        else if (cfg.block <= 256 && per_sm == 4 && a.g0.grid == 1)
            transport_kernel<false, 256, 4, false, true><<<grid, cfg.block, smem, s>>>(a);
        else if (cfg.block <= 256 && per_sm >= 3) transport_kernel<false, 256, 3, false, true><<<grid, cfg.block, smem, s>>>(a);
        else if (cfg.block <= 256) transport_kernel<false, 256, 2, false, true><<<grid, cfg.block, smem, s>>>(a);
        else return cudaErrorInvalidConfiguration;
    } else if (a.radial) {
        if (cfg.block > 256) return cudaErrorInvalidConfiguration;
        if (!multi) transport_kernel<false, 256, 4, true><<<grid, cfg.block, smem, s>>>(a);
        else transport_kernel<true, 256, 3, true><<<grid, cfg.block, smem, s>>>(a);
    } else if (!multi && cfg.aggregate) {
        // warp-aggregated, shared-memory privatised tallies (tally_mode 1)
        if (cfg.block == 320) transport_kernel<false, 320, 2, false, false, true><<<grid, cfg.block, smem, s>>>(a);
        else if (per_sm == 1) transport_kernel<false, 512, 1, false, false, true><<<grid, cfg.block, smem, s>>>(a);
        else if (per_sm == 2) transport_kernel<false, 256, 2, false, false, true><<<grid, cfg.block, smem, s>>>(a);
        else if (per_sm == 3) transport_kernel<false, 256, 3, false, false, true><<<grid, cfg.block, smem, s>>>(a);
        else transport_kernel<false, 256, 4, false, false, true><<<grid, cfg.block, smem, s>>>(a);
    } else if (!multi) {
        if (cfg.block == 320) transport_kernel<false, 320, 2><<<grid, cfg.block, smem, s>>>(a);
        else if (per_sm == 1) transport_kernel<false, 512, 1><<<grid, cfg.block, smem, s>>>(a);
        else if (per_sm == 2) transport_kernel<false, 256, 2><<<grid, cfg.block, smem, s>>>(a);
        else if (per_sm == 3) transport_kernel<false, 256, 3><<<grid, cfg.block, smem, s>>>(a);
        else transport_kernel<false, 256, 4><<<grid, cfg.block, smem, s>>>(a);
    } else {
        if (cfg.block == 320) transport_kernel<true, 320, 2><<<grid, cfg.block, smem, s>>>(a);
        else if (per_sm == 1) transport_kernel<true, 512, 1><<<grid, cfg.block, smem, s>>>(a);
        else if (per_sm == 2) transport_kernel<true, 256, 2><<<grid, cfg.block, smem, s>>>(a);
        else if (per_sm == 3) transport_kernel<true, 256, 3><<<grid, cfg.block, smem, s>>>(a);
        else transport_kernel<true, 256, 4><<<grid, cfg.block, smem, s>>>(a);
    }
    return cudaGetLastError();
}

cudaError_t launch_phs(cudaStream_t s, int32_t n_prim, const int32_t *per_primary, const int32_t *prim_geom,
                       int n_geom, int32_t min_photons, int32_t max_photons, int32_t num_bins, int32_t *phs,
                       double *moments, unsigned long long *dropped)
{
    if (n_prim <= 0) return cudaSuccess;
    const int32_t width = num_bins > 0 ? (max_photons - min_photons) / num_bins : 0;
    if (width <= 0) return cudaErrorInvalidValue;
    const int32_t shift = min_photons / width;
    phs_kernel<<<grid_for(n_prim, 256, 1024), 256, 0, s>>>(n_prim, per_primary, prim_geom, n_geom, min_photons,
                                                           max_photons, num_bins, width, shift, phs, moments,
                                                           dropped);
    return cudaGetLastError();
}

}  // namespace fd2

// Diagnostic entry point (tests): evaluates the transport's wall-root routine
// on the current device for n quadratics a t^2 + b t + c = 0 given in host
// arrays, so a test can drive its FP64 fallback for a nearly cancelling
// discriminant.  Synchronous.
extern "C" __attribute__((visibility("default"))) int fd2_debug_wall_root(int32_t n, const float *qa, const float *qb,
                                                                          const float *qc, float *out)
{
    if (n < 0 || (n > 0 && (!qa || !qb || !qc || !out))) return 1;
    if (n == 0) return 0;
    float *d = nullptr;
    const size_t b = sizeof(float) * (size_t)n;
    cudaError_t e = cudaMalloc(&d, 4 * b);
    if (e != cudaSuccess) return 5;
    if (e == cudaSuccess) e = cudaMemcpy(d, qa, b, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(d + n, qb, b, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(d + 2 * (size_t)n, qc, b, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        fd2::wall_root_kernel<<<(unsigned)((n + 255) / 256), 256>>>(n, d, d + n, d + 2 * (size_t)n, d + 3 * (size_t)n);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, d + 3 * (size_t)n, b, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e == cudaSuccess ? 0 : 4;
}

