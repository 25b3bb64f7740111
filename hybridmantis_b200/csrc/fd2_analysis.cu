// fd2_analysis.cu -- MTF and NNPS of the transport's images (include/fd2_analysis.h).
//
// Both are discrete Fourier transforms of modest images (hundreds of pixels
// a side), taken as two passes of direct sums in FP64 with exact integer phase
// reduction: pass 1 transforms every row at the wanted column frequencies,
// pass 2 every resulting column at the wanted row frequencies.  The images are
// real, so only column frequencies >= 0 are computed; the others are their
// conjugates.  The passes are matrix products with twiddle factors
// exp(-2 pi i m / N) from a table, bound by FP64 multiply-adds and
// shared-memory reads: a thread keeps four complex sums in registers, the
// twiddles of a warp are the same for its lanes (broadcast reads), and the
// next chunk of a tile is loaded while one is summed.  One thread per output
// with a table read of its own per multiply-add took 164 us and 323 us for a
// 501 x 501 image at all frequencies; the passes below take 46 and 45 us.  The
// axes alone (MTF without mtf_r) come from the two line spread functions.  All
// regions of all images of a noise spectrum go through them together (144
// regions of 128 x 128 pixels: 89 and 121 us; region by region 288 launches).
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <vector>

#include "fd2.h"
#include "fd2_analysis.h"

namespace {

constexpr int kThreads = 128;
constexpr int kFreqs = 16;      // frequencies of a block: 4 warps x 4
constexpr int kRowTile = 32;    // pass 1: rows of a block, 1 a lane
constexpr int kColTile = 32;    // pass 2: column frequencies of a block, 1 a lane
constexpr int kDepth = 32;      // terms staged in shared memory at a time

// tw[m] = exp(-2 pi i m / N), m < N
__global__ void twiddle_kernel(int n, double2 *tw)
{
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= n) return;
    double s, c;
    sincospi(2.0 * (double)m / (double)n, &s, &c);
    tw[m] = make_double2(c, -s);
}

// The regions to transform: rows x cols of every image at the origins of a
// grid of regions, minus the mean image, or with a single image minus each
// region's mean (sum / (rows cols)).
struct Regions {
    const double *img;
    int64_t ld, image;          // row and image strides
    int x0, y0, rows, cols, across, per_image;  // grid of regions: `across` along y
    const double *mean;         // mean image, or null
    const double *sums;         // region sums of a single image, or null
};

// out[z][r][k] = sum_c (in_z[r][c] - mean) tw[(k c) mod n] for k < nk of the
// region z = first + blockIdx.z.  grid (row tiles, frequency tiles, regions).
__global__ void __launch_bounds__(kThreads) dft_rows_kernel(const __grid_constant__ Regions g, int first, int nk,
                                                            const double2 *__restrict__ tw, int n,
                                                            double2 *__restrict__ out)
{
    __shared__ double tile[kDepth][kRowTile + 1];
    __shared__ double2 wt[kDepth][kFreqs];
    const int z = first + blockIdx.z, image = z / g.per_image, q = z % g.per_image;
    const int ox = g.x0 + q / g.across * g.rows, oy = g.y0 + q % g.across * g.cols;
    const int64_t origin = (int64_t)ox * g.ld + oy;
    const double *src = g.img + image * g.image + origin;
    const double *mean = g.mean ? g.mean + origin : nullptr;
    const double sub = g.sums ? g.sums[q] / ((double)g.rows * g.cols) : 0.0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int r0 = blockIdx.x * kRowTile, k0 = blockIdx.y * kFreqs;
    double re[4] = {}, im[4] = {};
    // the next chunk is loaded while this one is summed: a warp takes rows
    // warp, warp + 4, ... of the tile, its lanes the chunk's columns
    constexpr int kLoads = kRowTile / 4, kTw = kDepth * kFreqs / kThreads;
    double next[kLoads];
    double2 next_w[kTw];
    auto load = [&](int c0) {
        const bool in = c0 + lane < g.cols;
#pragma unroll
        for (int i = 0; i < kLoads; ++i) {
            const int r = r0 + warp + 4 * i;
            const int64_t at = (int64_t)r * g.ld + c0 + lane;
            double v = 0.0;
            if (in && r < g.rows) {
                v = src[at];
                if (mean) v -= mean[at];
                else if (g.sums) v -= sub;
            }
            next[i] = v;
        }
#pragma unroll
        for (int i = 0; i < kTw; ++i) {
            const int t = threadIdx.x + i * kThreads;
            // below 2^32: sides are at most 16,384
            next_w[i] = tw[(uint32_t)(k0 + t % kFreqs) * (uint32_t)(c0 + t / kFreqs) % (uint32_t)n];
        }
    };
    load(0);
    for (int c0 = 0; c0 < g.cols; c0 += kDepth) {
        const int nc = min(kDepth, g.cols - c0);
#pragma unroll
        for (int i = 0; i < kLoads; ++i) tile[lane][warp + 4 * i] = next[i];
#pragma unroll
        for (int i = 0; i < kTw; ++i) {
            const int t = threadIdx.x + i * kThreads;
            wt[t / kFreqs][t % kFreqs] = next_w[i];
        }
        __syncthreads();
        if (c0 + kDepth < g.cols) load(c0 + kDepth);
#pragma unroll 4
        for (int c = 0; c < nc; ++c) {
            const double a = tile[c][lane];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const double2 w = wt[c][warp * 4 + j];
                re[j] = fma(a, w.x, re[j]);
                im[j] = fma(a, w.y, im[j]);
            }
        }
        __syncthreads();
    }
    double2 *o = out + (int64_t)blockIdx.z * g.rows * nk;
    const int r = r0 + lane;
    if (r >= g.rows) return;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int k = k0 + warp * 4 + j;
        if (k < nk) o[(int64_t)r * nk + k] = make_double2(re[j], im[j]);
    }
}

// Pass 2 at the row frequencies s_u = u + shift, u < nu, of every column k of
// (nrows x nk) matrices: h = sum_r a[r][k] tw[(s_u r) mod n].  power == 0:
// map[u][k] = |h| of the single matrix.  power == 1: plane blockIdx.z of map
// [u][k] += |h|^2 over the matrices blockIdx.z, + gridDim.z, ... (one block
// per element of a plane, so sums run in a fixed order).
// grid (column tiles, frequency tiles, planes).
__global__ void __launch_bounds__(kThreads) dft_cols_kernel(const double2 *__restrict__ a, int matrices, int nrows,
                                                            int nk, int nu, int shift,
                                                            const double2 *__restrict__ tw, int n, int power,
                                                            double *__restrict__ map)
{
    __shared__ double2 tile[kDepth][kColTile];
    __shared__ double2 wt[kDepth][kFreqs];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int k0 = blockIdx.x * kColTile, u0 = blockIdx.y * kFreqs, k = k0 + lane;
    double sum[4] = {};
    for (int m = blockIdx.z; m < matrices; m += gridDim.z) {
        const double2 *src = a + (int64_t)m * nrows * nk;
        double re[4] = {}, im[4] = {};
        constexpr int kLoads = kDepth / 4, kTw = kDepth * kFreqs / kThreads;
        double2 next[kLoads], next_w[kTw];
        auto load = [&](int r0) {
#pragma unroll
            for (int i = 0; i < kLoads; ++i) {
                const int r = r0 + warp + 4 * i;
                next[i] = r < nrows && k < nk ? src[(int64_t)r * nk + k] : make_double2(0.0, 0.0);
            }
#pragma unroll
            for (int i = 0; i < kTw; ++i) {
                const int t = threadIdx.x + i * kThreads;
                const uint32_t f = (uint32_t)((u0 + t % kFreqs + shift) % n + n);  // the signed frequency mod n, plus n
                next_w[i] = tw[f * (uint32_t)(r0 + t / kFreqs) % (uint32_t)n];
            }
        };
        load(0);
        for (int r0 = 0; r0 < nrows; r0 += kDepth) {
            const int nr = min(kDepth, nrows - r0);
#pragma unroll
            for (int i = 0; i < kLoads; ++i) tile[warp + 4 * i][lane] = next[i];
#pragma unroll
            for (int i = 0; i < kTw; ++i) {
                const int t = threadIdx.x + i * kThreads;
                wt[t / kFreqs][t % kFreqs] = next_w[i];
            }
            __syncthreads();
            if (r0 + kDepth < nrows) load(r0 + kDepth);
#pragma unroll 4
            for (int r = 0; r < nr; ++r) {
                const double2 x = tile[r][lane];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const double2 w = wt[r][warp * 4 + j];
                    re[j] = fma(x.x, w.x, fma(-x.y, w.y, re[j]));
                    im[j] = fma(x.x, w.y, fma(x.y, w.x, im[j]));
                }
            }
            __syncthreads();
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) sum[j] += power ? re[j] * re[j] + im[j] * im[j] : sqrt(re[j] * re[j] + im[j] * im[j]);
    }
    if (k >= nk) return;
    double *o = map + (int64_t)blockIdx.z * nu * nk;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int u = u0 + warp * 4 + j;
        if (u >= nu) continue;
        if (power) o[(int64_t)u * nk + k] += sum[j];
        else o[(int64_t)u * nk + k] = sum[j];
    }
}

// Radial average of a map [nu][nk] of a real image's transform: signed row
// frequency u + shift (folded to (-wrap / 2, wrap / 2] with wrap > 0), column
// frequency k >= 0, whose mirror (-u, -k) the map leaves out and counts as a
// second value (`single`: the column frequency besides 0 that is its own
// mirror, or -1).  Block b averages the values whose radius rounds to b.
__global__ void __launch_bounds__(kThreads) radial_kernel(const double *__restrict__ map, int nu, int nk, int shift,
                                                          int wrap, int single, double *__restrict__ out)
{
    __shared__ double part[kThreads];
    __shared__ int count[kThreads];
    const int b = blockIdx.x;
    const double lo = b - 0.5, hi = b + 0.5;
    double s = 0.0;
    int n = 0;
    for (int u = threadIdx.x; u < nu; u += kThreads) {
        int su = u + shift;
        if (wrap > 0 && su > wrap / 2) su -= wrap;
        const double u2 = (double)su * su;
        // the columns whose radius can round to b, one more on both sides
        const int k_lo = max((int)sqrt(fmax(lo * lo - u2, 0.0)) - 1, 0);
        const int k_hi = min((int)sqrt(fmax(hi * hi - u2, 0.0)) + 1, nk - 1);
        for (int k = k_lo; k <= k_hi; ++k) {
            if ((int)llrint(sqrt(u2 + (double)k * k)) != b) continue;
            const int weight = k == 0 || k == single ? 1 : 2;
            s += weight * map[(int64_t)u * nk + k];
            n += weight;
        }
    }
    part[threadIdx.x] = s;
    count[threadIdx.x] = n;
    __syncthreads();
    for (int w = kThreads / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) {
            part[threadIdx.x] += part[threadIdx.x + w];
            count[threadIdx.x] += count[threadIdx.x + w];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) out[b] = count[0] > 0 ? part[0] / count[0] : 0.0;
}

// The line spread functions of an image: lines[i] = sum_j img[i][j] for i <
// xdim, and per band b of kBandRows rows part[b][j] = sum of img[i][j] over the
// band (line_dft_kernel adds the bands).  Bound by reading the image once.  A
// block takes a band's kThreads columns, and its warps the band's rows in turn
// for the row sums.  grid (column tiles, bands).
constexpr int kBandRows = 64;
__global__ void __launch_bounds__(kThreads) line_sums_kernel(const double *__restrict__ img, int xdim, int ydim,
                                                             double *__restrict__ lines, double *__restrict__ part)
{
    const int r0 = blockIdx.y * kBandRows, r1 = min(r0 + kBandRows, xdim);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int j = blockIdx.x * kThreads + threadIdx.x;
    if (j < ydim) {
        double s = 0.0;
#pragma unroll 8
        for (int i = r0; i < r1; ++i) s += img[(int64_t)i * ydim + j];
        part[(int64_t)blockIdx.y * ydim + j] = s;
    }
    // the band's rows shared out over the blocks of its column tiles
    for (int i = r0 + blockIdx.x * 4 + warp; i < r1; i += gridDim.x * 4) {
        double s = 0.0;
#pragma unroll 4
        for (int c = lane; c < ydim; c += 32) s += img[(int64_t)i * ydim + c];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (lane == 0) lines[i] = s;
    }
}

// lines[xdim + j] = the column sums from their bands.
__global__ void line_bands_kernel(const double *__restrict__ part, int bands, int xdim, int ydim,
                                  double *__restrict__ lines)
{
    const int j = blockIdx.x * kThreads + threadIdx.x;
    if (j >= ydim) return;
    double s = 0.0;
    for (int b = 0; b < bands; ++b) s += part[(int64_t)b * ydim + j];
    lines[xdim + j] = s;
}

// out[axis nk + k] = |sum_i l[i] tw[(k i) mod n]|, l the line spread function of
// axis blockIdx.y (0: x, 1: y), and out[2 nk] = the sum of the rows' (k = 0 of
// axis 0, before the magnitude).  A warp per frequency.
__global__ void __launch_bounds__(kThreads) line_dft_kernel(const double *__restrict__ lines, int xdim, int ydim,
                                                            int nk, const double2 *__restrict__ tw, int n,
                                                            double *__restrict__ out)
{
    const int k = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31, axis = blockIdx.y;
    if (k >= nk) return;
    const double *l = lines + (axis ? xdim : 0);
    const int len = axis ? ydim : xdim;
    double re = 0.0, im = 0.0;
    // k below 2^13, terms below 2^14
    uint32_t m = (uint32_t)(k * lane) % (uint32_t)n;
    const uint32_t step = (uint32_t)(k * 32) % (uint32_t)n;
    for (int i = lane; i < len; i += 32) {
        const double2 w = tw[m];
        re = fma(l[i], w.x, re);
        im = fma(l[i], w.y, im);
        m += step;
        if (m >= (uint32_t)n) m -= (uint32_t)n;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        re += __shfl_down_sync(0xffffffffu, re, o);
        im += __shfl_down_sync(0xffffffffu, im, o);
    }
    if (lane != 0) return;
    out[axis * nk + k] = sqrt(re * re + im * im);
    if (axis == 0 && k == 0) out[2 * nk] = re;
}

// out[k] = |h(k, 0)|, out[n + k] = |h(0, k)| from the map of |h| (row frequency
// 0 at row `zero`): the transforms of the two line spread functions (row and
// column sums); out[2 n]: the image's sum.
__global__ void axes_kernel(const double *__restrict__ map, int nk, int zero, const double2 *__restrict__ a, int nrows,
                            double *__restrict__ out)
{
    __shared__ double part[kThreads];
    double s = 0.0;
    for (int r = threadIdx.x; r < nrows; r += kThreads) s += a[(int64_t)r * nk].x;  // the rows' sums
    part[threadIdx.x] = s;
    __syncthreads();
    for (int w = kThreads / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) part[threadIdx.x] += part[threadIdx.x + w];
        __syncthreads();
    }
    for (int k = threadIdx.x; k < nk; k += kThreads) {
        out[k] = map[(int64_t)(zero + k) * nk];
        out[nk + k] = map[(int64_t)zero * nk + k];
    }
    if (threadIdx.x == 0) out[2 * nk] = part[0];
}

// Per-pixel mean over n images (x n stacked images of `count` values).
__global__ void mean_images_kernel(const double *__restrict__ imgs, int n, int64_t count, double *__restrict__ mean)
{
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < count; p += (int64_t)gridDim.x * blockDim.x) {
        double s = 0.0;
        for (int r = 0; r < n; ++r) s += imgs[(int64_t)r * count + p];
        mean[p] = s / (double)n;
    }
}

// Sums of the regions of an image, a block per region.  Pixel t goes to partial
// sum t mod 128, pixels in order, then the partial sums are added in a tree: the
// order decides the sign of a mean signal near zero, and with it whether nnps
// refuses the images, so it stays.  Bound by those chains of additions; the
// whole block loads, through shared memory, the next tile while one is added
// (a 128 x 128 / 4,096 x 4,096 region: 10 us / 6.7 ms, 128 threads that load for
// themselves 23 us / 13 ms).
constexpr int kSumThreads = 1024, kSumTile = 4 * kSumThreads;
__global__ void __launch_bounds__(kSumThreads) region_sum_kernel(const __grid_constant__ Regions g,
                                                              double *__restrict__ out)
{
    __shared__ double tile[kSumTile];
    double *const part = tile;
    const int q = blockIdx.x, n = g.rows * g.cols;
    const double *img = g.img + (int64_t)(g.x0 + q / g.across * g.rows) * g.ld + g.y0 + q % g.across * g.cols;
    double next[4], s = 0.0;
    auto load = [&](int t0) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int t = t0 + threadIdx.x + i * kSumThreads;
            next[i] = t < n ? img[(int64_t)(t / g.cols) * g.ld + t % g.cols] : 0.0;
        }
    };
    load(0);
    for (int t0 = 0; t0 < n; t0 += kSumTile) {
#pragma unroll
        for (int i = 0; i < 4; ++i) tile[threadIdx.x + i * kSumThreads] = next[i];
        __syncthreads();
        if (t0 + kSumTile < n) load(t0 + kSumTile);
        if (threadIdx.x < kThreads) {
#pragma unroll
            for (int i = 0; i < kSumTile; i += kThreads) s += tile[i + threadIdx.x];
        }
        __syncthreads();
    }
    if (threadIdx.x < kThreads) part[threadIdx.x] = s;
    __syncthreads();
    for (int w = kThreads / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) part[threadIdx.x] += part[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[q] = part[0];
}

// The scaled power map of an n x n transform from its planes [n][nk] over
// column frequencies 0..n/2: half[u][k] = scale sum_z planes[z][u][k], and the
// full map in unsigned DFT order.  scale = factor / m^2 with the mean signal m
// of the `regions` region sums, kept in *mean_signal.
__global__ void power_map_kernel(const double *__restrict__ planes, int nplanes, int n, int nk,
                                 const double *__restrict__ sums, int regions, double factor,
                                 double *__restrict__ half, double *__restrict__ out2d,
                                 double *__restrict__ mean_signal)
{
    double m = 0.0;
    for (int q = 0; q < regions; ++q) m += sums[q];
    m /= (double)regions * n * n;
    const double scale = factor / (m * m);
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t == 0) *mean_signal = m;
    if (t >= (int64_t)n * nk) return;
    double s = 0.0;
    for (int z = 0; z < nplanes; ++z) s += planes[(int64_t)z * n * nk + t];
    const double val = s * scale;
    half[t] = val;
    if (!out2d) return;
    const int u = (int)(t / nk), k = (int)(t % nk);
    out2d[(int64_t)u * n + k] = val;
    if (k > 0 && 2 * k != n) out2d[(int64_t)((n - u) % n) * n + n - k] = val;
}

// Offsets of a call's arrays in one device allocation.
struct Layout {
    size_t bytes = 0;
    template <typename T>
    size_t add(size_t n)
    {
        const size_t at = bytes;
        bytes += (sizeof(T) * std::max<size_t>(n, 1) + 255) & ~(size_t)255;
        return at;
    }
};

// The identity of the current CUDA context, never used twice in a process; false
// where the driver cannot say.
bool context_id(unsigned long long *id)
{
    struct Entry {
        PFN_cuCtxGetCurrent_v4000 current = nullptr;
        PFN_cuCtxGetId_v12000 id = nullptr;
        Entry()
        {
            void *a = nullptr, *b = nullptr;
            cudaDriverEntryPointQueryResult q{};
            if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &a, cudaEnableDefault, &q) != cudaSuccess ||
                q != cudaDriverEntryPointSuccess ||
                cudaGetDriverEntryPoint("cuCtxGetId", &b, cudaEnableDefault, &q) != cudaSuccess ||
                q != cudaDriverEntryPointSuccess)
                return;
            current = reinterpret_cast<PFN_cuCtxGetCurrent_v4000>(a);
            id = reinterpret_cast<PFN_cuCtxGetId_v12000>(b);
        }
    };
    static const Entry entry;
    CUcontext c = nullptr;
    return entry.id && entry.current(&c) == CUDA_SUCCESS && c && entry.id(c, id) == CUDA_SUCCESS;
}

// A call's device memory and stream.  One of each is kept per device between
// calls (allocating and freeing them took 1 to 5 ms of a 501 x 501 MTF, its
// kernels 0.12 ms): up to kKept bytes, for one call at a time, until
// fd2_analysis_release.  A call that needs more, or that runs beside another on
// the device, has its own.  A device reset takes the kept ones away with their
// context, so they belong to a context's identity and are forgotten, untouched,
// when the device's context is another one.  Nothing is freed at the process's
// end, when the runtime may be gone.
class Workspace {
  public:
    static constexpr size_t kKept = (size_t)128 << 20;

    // with `device` current
    cudaError_t open(int device, size_t bytes)
    {
        unsigned long long id = 0;
        if (device < kDevices && bytes <= kKept && context_id(&id) && kept(device).lock.try_lock()) {
            Kept &k = kept(device);
            held_ = &k;
            k.belong_to(id);
            cudaError_t e = k.stream ? cudaSuccess : cudaStreamCreateWithFlags(&k.stream, cudaStreamNonBlocking);
            if (e == cudaSuccess && k.bytes < bytes) {
                if (k.base) cudaFree(k.base);
                k.base = nullptr;
                k.bytes = 0;
                e = cudaMalloc((void **)&k.base, bytes);
                if (e == cudaSuccess) k.bytes = bytes;
            }
            base = k.base;
            stream = k.stream;
            return e;
        }
        cudaError_t e = cudaMalloc((void **)&base, bytes);
        if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking);
        return e;
    }
    template <typename T>
    T *at(size_t offset) const
    {
        return reinterpret_cast<T *>(base + offset);
    }
    ~Workspace()
    {
        if (held_) {
            if (stream) cudaStreamSynchronize(stream);  // after an error too: the next call finds it idle
            held_->lock.unlock();
            return;
        }
        if (stream) cudaStreamDestroy(stream);
        if (base) cudaFree(base);
    }
    // Gives the device's kept memory and stream back, after the call that uses
    // them; with `device` current.
    static cudaError_t release(int device)
    {
        unsigned long long id = 0;
        if (device >= kDevices || !context_id(&id)) return cudaSuccess;  // nothing is kept
        Kept &k = kept(device);
        std::lock_guard<std::mutex> lock(k.lock);
        k.belong_to(id);
        cudaError_t e = k.base ? cudaFree(k.base) : cudaSuccess;
        if (k.stream) {
            const cudaError_t e2 = cudaStreamDestroy(k.stream);
            if (e == cudaSuccess) e = e2;
        }
        k.forget();
        return e;
    }
    cudaStream_t stream = nullptr;

  private:
    static constexpr int kDevices = 16;
    struct Kept {
        std::mutex lock;
        unsigned long long context = 0;  // whose they are
        char *base = nullptr;
        size_t bytes = 0;
        cudaStream_t stream = nullptr;
        void forget()
        {
            base = nullptr;
            bytes = 0;
            stream = nullptr;
        }
        void belong_to(unsigned long long id)
        {
            if (context != id) forget();
            context = id;
        }
    };
    static Kept &kept(int device)
    {
        static Kept k[kDevices];
        return k[device];
    }
    char *base = nullptr;
    Kept *held_ = nullptr;
};

fd2_status to_status(cudaError_t e)
{
    if (e == cudaSuccess) return FD2_OK;
    return e == cudaErrorMemoryAllocation ? FD2_ERR_OUT_OF_MEMORY
           : (e == cudaErrorNoDevice || e == cudaErrorInvalidDevice) ? FD2_ERR_NO_DEVICE
                                                                      : FD2_ERR_CUDA;
}

// The image's sum, pixel by pixel: an image has signal when it is positive and finite.
double image_sum(const double *image, int64_t n)
{
    double total = 0.0;
    for (int64_t p = 0; p < n; ++p) total += image[p];
    return total;
}

bool any_sign_bit(const double *image, int64_t n)
{
    uint64_t any = 0;
    for (int64_t p = 0; p < n; ++p) {
        uint64_t b;
        std::memcpy(&b, image + p, sizeof b);
        any |= b;
    }
    return any >> 63;
}

unsigned tiles(int64_t n, int tile) { return (unsigned)((n + tile - 1) / tile); }

unsigned blocks_for(int64_t n) { return (unsigned)std::max<int64_t>(1, std::min<int64_t>((n + kThreads - 1) / kThreads, 1 << 20)); }

}  // namespace

extern "C" {

fd2_status fd2_mtf(int32_t device, const double *image, int32_t xdim, int32_t ydim, double pixel_um, int32_t n_freq,
                   double *freq_per_mm, double *mtf_x, double *mtf_y, double *mtf_r)
{
    if (!image || xdim < 1 || ydim < 1 || xdim > 16384 || ydim > 16384 || !(pixel_um > 0.0) || n_freq < 1)
        return FD2_ERR_INVALID_ARGUMENT;
    const int N = std::max(xdim, ydim);
    if (n_freq > N / 2 + 1) return FD2_ERR_INVALID_ARGUMENT;
    const int64_t npx = (int64_t)xdim * ydim;
    cudaError_t e = cudaSetDevice(device);
    if (e != cudaSuccess) {
        // an image without signal is refused whatever the device
        const double total = image_sum(image, npx);
        return !(total > 0.0) || !std::isfinite(total) ? FD2_ERR_INVALID_ARGUMENT : to_status(e);
    }
    const int K = n_freq, V = 2 * K - 1, bands = (int)tiles(xdim, kBandRows);
    // Without mtf_r the two axes are transforms of line spread functions (2 N K
    // multiply-adds) and need no transform of the image (N^2 K and N K V).  With
    // it they are two lines of its map.  (Both axes at every frequency, copy of
    // the image included: 501 x 501 208 us this way and 255 by the map, 2,048 x
    // 2,048 2.8 ms and 5.6, 6,144 x 6,144 51 ms and 137.)
    const bool map2d = mtf_r != nullptr;
    Layout l;
    Workspace d;
    const size_t o_img = l.add<double>((size_t)npx), o_tw = l.add<double2>((size_t)N);
    // out: mtf_x, mtf_y, the image's sum, mtf_r, all but the division by the sum
    const size_t o_out = l.add<double>(3 * (size_t)K + 1);
    const size_t o_a = map2d ? l.add<double2>((size_t)xdim * K) : l.add<double>((size_t)bands * ydim);
    const size_t o_map = map2d ? l.add<double>((size_t)V * K) : l.add<double>((size_t)xdim + ydim);
    if ((e = d.open(device, l.bytes)) != cudaSuccess) return to_status(e);
    const cudaStream_t s = d.stream;
    double *img = d.at<double>(o_img), *out = d.at<double>(o_out);
    double2 *tw = d.at<double2>(o_tw);
    e = cudaMemcpyAsync(img, image, sizeof(double) * npx, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) {
        twiddle_kernel<<<blocks_for(N), kThreads, 0, s>>>(N, tw);
        if (map2d) {
            const Regions g{img, ydim, npx, 0, 0, xdim, ydim, 1, 1, nullptr, nullptr};
            double2 *a = d.at<double2>(o_a);
            double *map = d.at<double>(o_map);
            dft_rows_kernel<<<dim3(tiles(xdim, kRowTile), tiles(K, kFreqs)), kThreads, 0, s>>>(g, 0, K, tw, N, a);
            dft_cols_kernel<<<dim3(tiles(K, kColTile), tiles(V, kFreqs)), kThreads, 0, s>>>(a, 1, xdim, K, V, 1 - K,
                                                                                          tw, N, 0, map);
            axes_kernel<<<1, kThreads, 0, s>>>(map, K, K - 1, a, xdim, out);
            radial_kernel<<<(unsigned)K, kThreads, 0, s>>>(map, V, K, 1 - K, 0, -1, out + 2 * K + 1);
        } else {
            double *part = d.at<double>(o_a), *lines = d.at<double>(o_map);
            line_sums_kernel<<<dim3(tiles(ydim, kThreads), (unsigned)bands), kThreads, 0, s>>>(img, xdim, ydim, lines,
                                                                                              part);
            line_bands_kernel<<<tiles(ydim, kThreads), kThreads, 0, s>>>(part, bands, xdim, ydim, lines);
            line_dft_kernel<<<dim3(tiles(K, 4), 2), kThreads, 0, s>>>(lines, xdim, ydim, K, tw, N, out);
        }
        e = cudaGetLastError();
    }
    const bool sign = any_sign_bit(image, npx);  // while the kernels run
    std::vector<double> r(3 * (size_t)K + 1);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(r.data(), out, sizeof(double) * (mtf_r ? r.size() : 2 * (size_t)K + 1),
                            cudaMemcpyDeviceToHost, s);
    const cudaError_t e2 = cudaStreamSynchronize(s);
    if (e == cudaSuccess) e = e2;
    if (e != cudaSuccess) return to_status(e);
    // The device's sum, in rows, is the image's where nothing cancels.  With
    // negative values (or no number) the order decides a sum near zero, and with
    // it whether the image has signal: then pixel by pixel (0.25 ms of host time
    // at 501 x 501, which is why it is not always taken).
    double total = r[2 * (size_t)K];
    if (sign || !(total > 0.0) || !std::isfinite(total)) total = image_sum(image, npx);
    if (!(total > 0.0) || !std::isfinite(total)) return FD2_ERR_INVALID_ARGUMENT;
    for (int k = 0; k < K; ++k) {
        if (freq_per_mm) freq_per_mm[k] = 1000.0 * k / (N * pixel_um);
        if (mtf_x) mtf_x[k] = r[(size_t)k] / total;
        if (mtf_y) mtf_y[k] = r[(size_t)K + k] / total;
        if (mtf_r) mtf_r[k] = r[2 * (size_t)K + 1 + k] / total;
    }
    return FD2_OK;
}

fd2_status fd2_nnps(int32_t device, const double *images, int32_t n_images, int32_t xdim, int32_t ydim,
                    double pixel_um, int32_t roi, int32_t x0, int32_t y0, int32_t rois_x, int32_t rois_y,
                    int32_t n_freq, double *freq_per_mm, double *nnps_r, double *nnps_2d, double *mean_signal)
{
    if (!images || n_images < 1 || xdim < 1 || ydim < 1 || !(pixel_um > 0.0) || roi < 2 || roi > 4096 ||
        rois_x < 1 || rois_y < 1 || x0 < 0 || y0 < 0 || n_freq < 1 || n_freq > roi / 2 + 1 ||
        (int64_t)x0 + (int64_t)rois_x * roi > xdim || (int64_t)y0 + (int64_t)rois_y * roi > ydim)
        return FD2_ERR_INVALID_ARGUMENT;
    if (freq_per_mm)
        for (int k = 0; k < n_freq; ++k) freq_per_mm[k] = 1000.0 * k / (roi * pixel_um);
    cudaError_t e = cudaSetDevice(device);
    if (e != cudaSuccess) return to_status(e);
    const int R = roi, K = n_freq, n = n_images, H = R / 2 + 1, nroi = rois_x * rois_y;
    // regions of all images are transformed together, as many at a time as fit
    // 128 MiB; pass 2 sums their power in `planes` planes, so that blocks share
    // the regions of small maps
    const int64_t all = (int64_t)n * nroi, per_region = (int64_t)R * H;
    const int batch = (int)std::max<int64_t>(1, std::min<int64_t>({all, 65535, (128ll << 20) / (16 * per_region)}));
    const unsigned tiles2 = tiles(H, kColTile) * tiles(R, kFreqs);
    int sms = 0;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device)) != cudaSuccess) return to_status(e);
    const int planes = (int)std::max<int64_t>(1, std::min<int64_t>(batch, 8 * (unsigned)sms / tiles2));
    Layout l;
    Workspace d;
    // only the regions' pixels are copied
    const int wx = rois_x * R, wy = rois_y * R;
    const int64_t npx = (int64_t)wx * wy;
    const size_t o_imgs = l.add<double>((size_t)(npx * n)), o_mean = l.add<double>((size_t)npx);
    const size_t o_tw = l.add<double2>((size_t)R), o_a = l.add<double2>((size_t)(per_region * batch));
    const size_t o_planes = l.add<double>((size_t)(per_region * planes)), o_half = l.add<double>((size_t)per_region);
    const size_t o_sums = l.add<double>((size_t)nroi), o_out = l.add<double>((size_t)K + 1);
    const size_t o_2d = nnps_2d ? l.add<double>((size_t)R * R) : 0;
    if ((e = d.open(device, l.bytes)) != cudaSuccess) return to_status(e);
    const cudaStream_t s = d.stream;
    double *imgs = d.at<double>(o_imgs), *mean = d.at<double>(o_mean), *sums = d.at<double>(o_sums);
    double *acc = d.at<double>(o_planes), *half = d.at<double>(o_half), *out = d.at<double>(o_out);
    double *out2d = nnps_2d ? d.at<double>(o_2d) : nullptr;
    double2 *tw = d.at<double2>(o_tw), *a = d.at<double2>(o_a);
    for (int i = 0; e == cudaSuccess && i < n; ++i)
        e = cudaMemcpy2DAsync(imgs + i * npx, sizeof(double) * wy, images + ((int64_t)i * xdim + x0) * ydim + y0,
                              sizeof(double) * ydim, sizeof(double) * wy, (size_t)wx, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(acc, 0, sizeof(double) * per_region * planes, s);
    if (e == cudaSuccess) {
        Regions g{imgs, wy, npx, 0, 0, R, R, rois_y, nroi, nullptr, nullptr}, gm = g;
        twiddle_kernel<<<blocks_for(R), kThreads, 0, s>>>(R, tw);
        if (n > 1) {
            mean_images_kernel<<<blocks_for(npx), kThreads, 0, s>>>(imgs, n, npx, mean);
            gm.img = g.mean = mean;
        } else {
            g.sums = sums;  // one image: each region's own mean is subtracted
        }
        // region sums of the mean image (the signal)
        region_sum_kernel<<<(unsigned)nroi, kSumThreads, 0, s>>>(gm, sums);
        for (int64_t first = 0; first < all; first += batch) {
            const int m = (int)std::min<int64_t>(batch, all - first);
            dft_rows_kernel<<<dim3(tiles(R, kRowTile), tiles(H, kFreqs), (unsigned)m), kThreads, 0, s>>>(
                g, (int)first, H, tw, R, a);
            dft_cols_kernel<<<dim3(tiles(H, kColTile), tiles(R, kFreqs), (unsigned)planes), kThreads, 0, s>>>(
                a, m, R, H, R, 0, tw, R, 1, acc);
        }
        // NNPS = pixel^2 (mm^2) / roi^2 * <|F|^2> * n/(n-1) / m^2
        const double px_mm = pixel_um / 1000.0;
        const double corr = n > 1 ? (double)n / (double)(n - 1) : 1.0;
        const double factor = px_mm * px_mm / ((double)R * R) * corr / ((double)n * nroi);
        power_map_kernel<<<blocks_for(per_region), kThreads, 0, s>>>(acc, planes, R, H, sums, nroi, factor, half,
                                                                     out2d, out + K);
        radial_kernel<<<(unsigned)K, kThreads, 0, s>>>(half, R, H, 0, R, R % 2 == 0 ? R / 2 : -1, out);
        e = cudaGetLastError();
    }
    std::vector<double> r((size_t)K + 1);
    if (e == cudaSuccess) e = cudaMemcpyAsync(r.data(), out, sizeof(double) * r.size(), cudaMemcpyDeviceToHost, s);
    cudaError_t e2 = cudaStreamSynchronize(s);
    const double m = r[(size_t)K];
    const bool signal = e == cudaSuccess && e2 == cudaSuccess && m > 0.0;
    if (signal && nnps_2d) {
        e = cudaMemcpyAsync(nnps_2d, out2d, sizeof(double) * R * R, cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    }
    if (e == cudaSuccess) e = e2;
    if (e != cudaSuccess) return to_status(e);
    if (!signal) return FD2_ERR_INVALID_ARGUMENT;
    if (nnps_r) std::copy(r.begin(), r.begin() + K, nnps_r);
    if (mean_signal) *mean_signal = m;
    return FD2_OK;
}

fd2_status fd2_analysis_release(int32_t device)
{
    const cudaError_t e = cudaSetDevice(device);
    return to_status(e == cudaSuccess ? Workspace::release(device) : e);
}

}  // extern "C"
