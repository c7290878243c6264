// MorphSpotClean (replace mode) on the GPU.
//
// Reference: core/algorithms/ImagingAlgorithms/src/MorphSpotClean.cpp:41-175,264-351 with the
// grey-scale reconstructions of core/kipl/kipl/include/morphology/morphgeo.h:151-371 and the
// markers of morphextrema.h:265-328.
//
// Per image: optional inf/NaN replacement and clamping; padding by 5 (zero columns, the
// first/last 5 rows mirrored) and an in-place sliding median along the first and last
// padded rows (sequential, one thread per edge row, as the reference's loop); the
// reconstructions; threshold replacement or sigmoid blend; unpadding.
//
// Reconstructions. FillHole (erosion) and the dual FillPeaks of the 'both' mode are
// textbook reconstructions, unique fixpoints of min/max operations, so any order of
// monotone updates reaches exactly the reference's result. FillPeaks (peaks mode) runs
// RecByDilation, whose forward raster scan compares the running image but assigns the
// marker value (morphgeo.h:213-214); after that scan the reference computes the exact
// reconstruction of the scanned marker. The scanned marker differs from the initial one
// only on the border and on pixels with a border pixel among their backward neighbours
// (every other value stays the marker's interior minimum), so the scan
// is replayed over that band (k_peaks_band_smem), and the exact reconstruction follows.
//
// Few images are reconstructed by merging basins over the whole GPU (k_descend and following), many
// (few_units) by sweeps and a worklist, one CTA per image:
//
// Each reconstruction runs in two kernels, one CTA per image in both. The sweep kernel
// alternates downward and upward row sweeps for a few rounds (it stops early when a round
// changes nothing). A sweep combines each row with the neighbouring row just finished
// (vertical and, for 8-connectivity, diagonal neighbours), then propagates along the row in
// both directions with a CTA-wide scan: the row update v[c] = min(g[c], max(v[c], v[c-1]))
// (dilation) or max(g[c], min(v[c], v[c-1])) (erosion) is a clamp x -> min(hi, max(lo, x)),
// and clamps compose into clamps, so the sequential recurrence is a parallel prefix. On noisy
// projections the sweeps alone need 20-30 rounds (every change of vertical direction along a
// propagation path costs a round), while after a few rounds only a thin set of pixels still
// changes; the completion kernel finishes from there with a worklist (k_complete).
#include "mr_common.cuh"

#include <algorithm>
#include <cfloat>
#include <climits>
#include <cmath>
#include <type_traits>

namespace mr {

// Error word of this file's bounded loops (device globals are per translation unit without
// relocatable device code); mr_device_status reads and clears it with the other kernels' words.
__device__ int g_msc_error = 0;

MR_BOUNDS_TAKE(bounds_take_spot)

int msc_device_status_take()
{
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_msc_error, sizeof(int)) != cudaSuccess) return -1;
    if (cudaMemcpyToSymbol(g_msc_error, &zero, sizeof(int)) != cudaSuccess) return -1;
    return v;
}

namespace msc {

constexpr int kMargin = 5;
constexpr int kSweepRounds = 3; // dense sweep rounds before the worklist completion (2-6 measured: 3 is fastest)
constexpr int kMaxEdge = 63;
// Few reconstructions merge basins, many take sweeps. Basins cost 90 ps per pixel over the whole GPU.
// Sweeps have one CTA per image: up to 148 of them take as long as one (rows times a step that grows
// slowly with the row: 10 ns per pixel on rows of 1000, 17 on 500, 34 on 200), and 34 ps per pixel beyond
// that. So the line falls with the row length. Images whose paths wind take up to three times as long in
// the worklist, with 8 neighbours above all. Basins against sweeps in ms, smooth images to projections of
// a phantom with counting noise and stuck pixels:
//   holes, 8 neighbours:  110 of 700 x 1000  6.8-8.0 against 7.4-19    200  12-14 against 8.6-24
//                         200 of 300 x 500   2.7-3.3 against 2.8-7.9   400  5.1-6.1 against 3.3-6.6
//   peaks, 4 neighbours:  110 of 700 x 1000  6.6-7.7 against 6.9-12    200  12-14 against 8.2-15
//                         148 of 300 x 500   2.0-2.4 against 2.5-3.9   295  3.6-4.4 against 2.8-4.0
// Over 40 to 590 reconstructions of eight sizes (16 x 2048 to 500 x 300) the choice is within 2 % of the
// faster one on average and 1.7 at worst; basins for all of them: 14 to 20 % and 2.6. With 590 the sweeps
// are faster but on rows below 100 pixels and on winding paths in rows of 300; 592, four CTAs per SM, is
// the most that was measured.
inline bool few_units(size_t units, size_t pw, bool conn8)
{
    return units < std::min<size_t>(592, 40 + (conn8 ? 190000 : 100000) / pw);
}
constexpr size_t kBandSmem = 200 * 1024; // shared memory of k_peaks_band_smem

// ---- preparation

__global__ void k_finite_max(const float *__restrict__ img, size_t per, float *__restrict__ out)
{
    const float *p = img + blockIdx.x * per;
    float m = -FLT_MAX;
    for (size_t i = threadIdx.x; i < per; i += blockDim.x)
        if (isfinite(p[i]) && m < p[i]) m = p[i];
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    __shared__ float s[32];
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x < 32) {
        m = threadIdx.x < (blockDim.x + 31) / 32 ? s[threadIdx.x] : -FLT_MAX;
        for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        if (threadIdx.x == 0) out[blockIdx.x] = m;
    }
}

// Order-preserving integer keys of floats (atomics compare them as ints).
__device__ __forceinline__ int fkey(float f)
{
    const int i = __float_as_int(f);
    return i >= 0 ? i : i ^ 0x7FFFFFFF;
}

__device__ __forceinline__ float funkey(int k) { return __int_as_float(k >= 0 ? k : k ^ 0x7FFFFFFF); }

// Starting values of the per-image minimum and maximum keys.
__global__ void k_range_init(int n, int *__restrict__ mn, int *__restrict__ mx)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    mn[i] = fkey(FLT_MAX);
    mx[i] = fkey(-FLT_MAX);
}

// Padded image (MorphSpotClean::PadEdges :264-281) after replaceInfNaN (:514-536) and
// LimitDynamics (core/kipl/kipl/include/segmentation/thresholds.h:60-85), and the image's range as
// keys (NaN ignored). The edge medians that follow change rows 0 and ph - 1 only, within the range of
// those rows' samples, which rows 9 and ph - 10 hold too, so the range is theirs as well.
__global__ void __launch_bounds__(256) k_pad(const float *__restrict__ img, int w, int h, const float *__restrict__ finite_max, int clamp,
                      float lo, float hi, float *__restrict__ pad, int *__restrict__ mn, int *__restrict__ mx)
{
    float a = FLT_MAX, z = -FLT_MAX;
    const int pw = w + 2 * kMargin, ph = h + 2 * kMargin;
    const size_t n = static_cast<size_t>(pw) * ph;
    const int b = blockIdx.y;
    const float *src = img + static_cast<size_t>(b) * w * h;
    float *dst = pad + b * n;
    for (int y = blockIdx.x; y < ph; y += gridDim.x) {
        int sy = y - kMargin;
        if (sy < 0) sy = -1 - sy;              // padded row m-1-i <- image row i
        else if (sy >= h) sy = 2 * h - 1 - sy; // padded row ph-m+i <- image row h-1-i
        const float *srow = src + static_cast<size_t>(sy) * w;
        float *drow = dst + static_cast<size_t>(y) * pw;
        for (int xp = threadIdx.x; xp < pw; xp += blockDim.x) {
            const int x = xp - kMargin;
            float v = 0.0f;
            if (x >= 0 && x < w) {
                v = srow[x];
                if (finite_max && !isfinite(v)) v = finite_max[b];
                if (clamp) v = v < lo ? lo : (v > hi ? hi : v);
            }
            drow[xp] = v;
            a = fminf(a, v);
            z = fmaxf(z, v);
        }
    }
    __shared__ int ra[8], rz[8];
    const int ka = __reduce_min_sync(0xffffffffu, fkey(a)), kz = __reduce_max_sync(0xffffffffu, fkey(z));
    if ((threadIdx.x & 31) == 0) {
        ra[threadIdx.x >> 5] = ka;
        rz[threadIdx.x >> 5] = kz;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int lowest = ra[0], highest = rz[0];
        for (int k = 1; k < 8; ++k) {
            lowest = min(lowest, ra[k]);
            highest = max(highest, rz[k]);
        }
        atomicMin(mn + b, lowest);
        atomicMax(mx + b, highest);
    }
}

// Sliding in-place median of E samples in registers: the window holds the E samples of the
// current position, the median just written enters it at its place, the next sample at its
// end. The samples are ordered by an odd-even transposition sort, which swaps only adjacent
// samples in strictly decreasing order and so ends in the same (stable) order as the
// reference's insertion sort for any input without NaN.
template <int E>
__device__ void edge_median_reg(float *srow, int pw)
{
    constexpr int l2 = E / 2;
    float win[E];
#pragma unroll
    for (int q = 0; q < E; ++q) win[q] = q < pw ? srow[q] : 0.0f;
    for (int i = l2; i < pw - l2; ++i) {
        float b[E];
#pragma unroll
        for (int q = 0; q < E; ++q) b[q] = win[q];
#pragma unroll
        for (int pass = 0; pass < E; ++pass) {
#pragma unroll
            for (int k = pass & 1; k + 1 < E; k += 2) {
                const float a = b[k], c = b[k + 1];
                const bool sw = a > c;
                b[k] = sw ? c : a;
                b[k + 1] = sw ? a : c;
            }
        }
        const float m = (E & 1) ? b[E / 2] : static_cast<float>(0.5 * (static_cast<double>(b[E / 2 - 1]) + b[E / 2]));
        srow[i] = m;
#pragma unroll
        for (int q = 0; q + 1 < E; ++q) win[q] = win[q + 1];
        win[l2 - 1 >= 0 ? l2 - 1 : 0] = l2 >= 1 ? m : win[0];
        win[E - 1] = i + 1 + l2 < pw ? srow[i + 1 + l2] : 0.0f;
    }
}

// In-place sliding median of `edge` samples along padded rows 0 and ph-1 (:283-299). One warp
// per edge row: the row is staged in shared memory, lane 0 runs the sequential in-place loop
// there (each median sees the medians already written to its left, as in the reference), and
// the warp writes the row back. Edges 3, 5, 7 and 9 of a row without NaN run in registers.
__global__ void k_edge_median(float *__restrict__ pad, int pw, int ph, int edge)
{
    extern __shared__ float srow[];
    const int lane = threadIdx.x;
    float *row = pad + static_cast<size_t>(blockIdx.x >> 1) * pw * ph + ((blockIdx.x & 1) ? static_cast<size_t>(ph - 1) * pw : 0);
    bool nan = false;
    for (int i = lane; i < pw; i += 32) {
        srow[i] = row[i];
        nan |= isnan(srow[i]);
    }
    nan = __any_sync(0xffffffffu, nan);
    __syncwarp();
    if (lane == 0 && !nan && (edge == 3 || edge == 5 || edge == 7 || edge == 9)) {
        if (edge == 3) edge_median_reg<3>(srow, pw);
        else if (edge == 5) edge_median_reg<5>(srow, pw);
        else if (edge == 7) edge_median_reg<7>(srow, pw);
        else edge_median_reg<9>(srow, pw);
    } else if (lane == 0) {
        const int l2 = edge / 2;
        float buf[kMaxEdge];
        for (int i = l2; i < pw - l2; ++i) {
            for (int q = 0; q < edge; ++q) buf[q] = srow[i - l2 + q];
            for (int a = 1; a < edge; ++a) { // insertion sort
                float key = buf[a];
                int c = a - 1;
                while (c >= 0 && buf[c] > key) {
                    buf[c + 1] = buf[c];
                    --c;
                }
                buf[c + 1] = key;
            }
            srow[i] = (edge & 1) ? buf[edge / 2]
                                 : static_cast<float>(0.5 * (static_cast<double>(buf[edge / 2 - 1]) + buf[edge / 2]));
        }
    }
    __syncwarp();
    for (int i = lane; i < pw; i += 32) row[i] = srow[i];
}

// Marker of FillHole (interior = image maximum) or FillPeaks (interior = minimum), the image
// on its border (morphextrema.h:268-283, 299-314). sign -1 builds the marker of the negated
// image (FillHole of -padded in the 'both' mode).
__global__ void k_marker(const float *__restrict__ pad, int pw, int ph, const int *__restrict__ interior,
                         float sign, float *__restrict__ v)
{
    const size_t n = static_cast<size_t>(pw) * ph;
    const int b = blockIdx.y;
    const float in = sign * funkey(interior[b]); // max(-P) = -min(P) for the negated image
    for (int y = blockIdx.x; y < ph; y += gridDim.x) {
        const size_t ro = b * n + static_cast<size_t>(y) * pw;
        for (int x = threadIdx.x; x < pw; x += blockDim.x) {
            const bool border = y == 0 || y == ph - 1 || x == 0 || x == pw - 1;
            v[ro + x] = border ? sign * pad[ro + x] : in;
        }
    }
}

// Offset of a pixel in the band of a marker (rows 0, 1, ph - 1 of pw values, then columns 0, 1, pw - 2,
// pw - 1 of ph values); -1 outside it.
__device__ __forceinline__ int band_at(int x, int y, int pw, int ph)
{
    if (y <= 1) return y * pw + x;
    if (y == ph - 1) return 2 * pw + x;
    if (x <= 1) return 3 * pw + x * ph + y;
    if (x >= pw - 2) return 3 * pw + (x - pw + 4) * ph + y;
    return -1;
}

__host__ __device__ inline size_t band_size(int pw, int ph) { return 3 * static_cast<size_t>(pw) + 4 * static_cast<size_t>(ph); }

__device__ __forceinline__ bool is_border(int x, int y, int pw, int ph)
{
    return y == 0 || y == ph - 1 || x == 0 || x == pw - 1;
}

// Replay of RecByDilation's forward scan (morphgeo.h:207-215) over the pixels that can
// change: the border and every pixel with a border pixel among its backward neighbours.
// One thread per image, raster order. v holds the marker on entry.
__global__ void k_peaks_forward_band(const float *__restrict__ pad, int pw, int ph, int nimg, int conn8,
                                     const int *__restrict__ minval, float *__restrict__ v)
{
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= nimg) return;
    const size_t n = static_cast<size_t>(pw) * ph;
    const float *g = pad + b * n;
    float *t = v + b * n;
    const float mnv = funkey(minval[b]);
    const int bx[4] = {-1, 0, -1, 1}, by[4] = {0, -1, -1, -1};
    const int nb = conn8 ? 4 : 2;
    auto visit = [&](int x, int y) {
        const size_t pos = static_cast<size_t>(y) * pw + x;
        float mx = t[pos];
        for (int i = 0; i < nb; ++i) {
            const int qx = x + bx[i], qy = y + by[i];
            if (qx < 0 || qx >= pw || qy < 0) continue;
            const size_t q = static_cast<size_t>(qy) * pw + qx;
            if (t[q] > mx) mx = is_border(qx, qy, pw, ph) ? g[q] : mnv; // assigns the marker value
        }
        t[pos] = mx < g[pos] ? mx : g[pos];
    };
    for (int y = 0; y < ph; ++y) {
        if (y <= 1 || y == ph - 1) {
            for (int x = 0; x < pw; ++x) visit(x, y);
        } else {
            visit(0, y);
            visit(1, y);
            if (conn8 && pw - 2 > 1) visit(pw - 2, y);
            if (pw - 1 > 1) visit(pw - 1, y);
        }
    }
}

// The same replay for images whose border columns fit in shared memory, one CTA per image. Only the
// columns and the last row are chains: row 0 keeps the image (its backward neighbours are border pixels,
// whose marker is the image, and v <= g everywhere); a pixel of row 1 past x = 1 takes marker values of
// row 0 only (its left neighbour's marker is the minimum it starts from), except the last, which also
// compares its left neighbour. The two column chains run on two lanes from shared copies, then the last
// row on one. 64 images of 1010 x 710: 3.14 ms (one thread per image on global memory) -> 0.2 ms.
__global__ void __launch_bounds__(128) k_peaks_band_smem(const float *__restrict__ pad, int pw, int ph, int conn8,
                                                         const int *__restrict__ minval, float *__restrict__ out)
{
    extern __shared__ float band[];
    // image columns 0, 1, pw - 2, pw - 1 and their running values; image and running last row
    float *gc = band, *tc = gc + 4 * ph, *gl = tc + 4 * ph, *tl = gl + pw;
    const size_t n = static_cast<size_t>(pw) * ph;
    const float *g = pad + blockIdx.x * n;
    float *t = out + blockIdx.x * band_size(pw, ph); // rows 0 and 1 first (band_at)
    const float mnv = funkey(minval[blockIdx.x]);
    const int tid = threadIdx.x;
    for (int i = tid; i < 4 * ph; i += 128) {
        const int y = i >> 2, c = i & 3;
        const float gv = g[static_cast<size_t>(y) * pw + (c < 2 ? c : pw - 4 + c)];
        gc[c * ph + y] = gv;
        tc[c * ph + y] = (c == 0 || c == 3 || y == 0 || y == ph - 1) ? gv : mnv; // the marker
    }
    for (int x = tid; x < pw; x += 128) {
        gl[x] = g[static_cast<size_t>(ph - 1) * pw + x];
        t[x] = g[x];
    }
    // row 1: pixels 2 .. pw - 2 (and pixel 1 of row 1 below, which has a border pixel to its left)
    for (int x = 2 + tid; x <= pw - 2; x += 128) {
        const float gv = g[pw + x];
        float mx = mnv;
        const float up = g[x], ul = g[x - 1], ur = g[x + 1];
        if (up > mx) mx = up;
        if (conn8) {
            if (ul > mx) mx = ul;
            if (ur > mx) mx = ur;
        }
        const float r = mx < gv ? mx : gv;
        t[pw + x] = r;
        if (x == pw - 2) tc[2 * ph + 1] = r;
    }
    __syncthreads();
    // raised by a neighbour with running value tq and marker value mq
    auto see = [](float &mx, float tq, float mq) {
        if (tq > mx) mx = mq;
    };
    if (tid == 0) {
        // row 1 of columns 0 and 1, then the rows below: column 2 holds row 1's values at y = 1 and the
        // marker's minimum below
        const float t12 = t[pw + 2];
        for (int y = 1; y < ph - 1; ++y) {
            const float g0 = gc[y], g0u = gc[y - 1], t0u = tc[y - 1], t1u = tc[ph + y - 1];
            float mx = g0;
            see(mx, t0u, g0u);
            if (conn8) see(mx, t1u, y == 1 ? gc[ph] : mnv);
            const float r0 = mx < g0 ? mx : g0;
            tc[y] = r0;
            const float g1 = gc[ph + y];
            mx = mnv;
            see(mx, r0, g0);
            see(mx, t1u, y == 1 ? gc[ph] : mnv);
            if (conn8) {
                see(mx, t0u, g0u);
                if (y == 1) see(mx, g[2], g[2]);
                else if (y == 2) see(mx, t12, mnv);
            }
            tc[ph + y] = mx < g1 ? mx : g1;
        }
    } else if (tid == 32) {
        const float t1l = t[pw + pw - 3];
        for (int y = 1; y < ph - 1; ++y) {
            const float g2u = gc[2 * ph], t2u = tc[2 * ph + y - 1], g3u = gc[3 * ph + y - 1], t3u = tc[3 * ph + y - 1];
            if (y > 1 && conn8) {
                const float g2 = gc[2 * ph + y];
                float mx = mnv; // its left neighbours hold the minimum, except row 1's at y = 2
                see(mx, t2u, mnv);
                if (y == 2) see(mx, t1l, mnv);
                see(mx, t3u, g3u);
                tc[2 * ph + y] = mx < g2 ? mx : g2;
            }
            const float g3 = gc[3 * ph + y];
            float mx = g3;
            see(mx, tc[2 * ph + y], mnv);
            see(mx, t3u, g3u);
            if (conn8) see(mx, t2u, y == 1 ? g2u : mnv);
            tc[3 * ph + y] = mx < g3 ? mx : g3;
        }
    }
    __syncthreads();
    // the last row: above it the columns' values and the minimum elsewhere (row 1's when ph is 3: not
    // reached, the padding alone is 10 rows)
    if (tid == 0) {
        const int y = ph - 2;
        auto above = [&](int x) { return x <= 1 ? tc[x * ph + y] : x >= pw - 2 ? tc[(x - pw + 4) * ph + y] : mnv; };
        auto mark = [&](int x) { return x == 0 ? gc[y] : x == pw - 1 ? gc[3 * ph + y] : mnv; };
        float left = 0.0f;
        for (int x = 0; x < pw; ++x) {
            const float gv = gl[x];
            float mx = gv;
            if (x > 0) see(mx, left, gl[x - 1]);
            see(mx, above(x), mark(x));
            if (conn8) {
                if (x > 0) see(mx, above(x - 1), mark(x - 1));
                if (x < pw - 1) see(mx, above(x + 1), mark(x + 1));
            }
            left = mx < gv ? mx : gv;
            tl[x] = left;
        }
    }
    __syncthreads();
    for (int i = tid; i < 4 * (ph - 2); i += 128) {
        const int y = 1 + (i >> 2), c = i & 3;
        t[band_at(c < 2 ? c : pw - 4 + c, y, pw, ph)] = tc[c * ph + y];
    }
    for (int x = tid; x < pw; x += 128) t[2 * pw + x] = tl[x];
}

// The band out of a whole marker image (k_peaks_forward_band's).
__global__ void k_band_of(const float *__restrict__ v, int pw, int ph, float *__restrict__ out)
{
    const float *t = v + blockIdx.x * (static_cast<size_t>(pw) * ph);
    float *o = out + blockIdx.x * band_size(pw, ph);
    for (int x = threadIdx.x; x < pw; x += blockDim.x) {
        o[x] = t[x];
        o[pw + x] = t[pw + x];
        o[2 * pw + x] = t[static_cast<size_t>(ph - 1) * pw + x];
    }
    for (int i = threadIdx.x; i < 4 * (ph - 3); i += blockDim.x) {
        const int y = 2 + (i >> 2), c = i & 3, x = c < 2 ? c : pw - 4 + c;
        o[band_at(x, y, pw, ph)] = t[static_cast<size_t>(y) * pw + x];
    }
}

// The band into a whole marker image.
__global__ void k_band_into(const float *__restrict__ band, int pw, int ph, float *__restrict__ v)
{
    float *t = v + blockIdx.x * (static_cast<size_t>(pw) * ph);
    const float *b = band + blockIdx.x * band_size(pw, ph);
    for (int x = threadIdx.x; x < pw; x += blockDim.x) {
        t[pw + x] = b[pw + x];
        t[static_cast<size_t>(ph - 1) * pw + x] = b[2 * pw + x];
    }
    for (int i = threadIdx.x; i < 4 * (ph - 3); i += blockDim.x) {
        const int y = 2 + (i >> 2), c = i & 3, x = c < 2 ? c : pw - 4 + c;
        t[static_cast<size_t>(y) * pw + x] = b[band_at(x, y, pw, ph)];
    }
}

// ---- reconstruction by merging basins
//
// The erosion-reconstruction of g from a marker m >= g is a minimax path problem: H(p) is the smallest,
// over the pixels q and the paths from q to p, of the largest of m(q) and g along the path. FillHole's
// marker is g on the border and the maximum inside, so only the border's m counts: an "ocean" next to
// every border pixel, entered at height m. FillPeaks (the dilation) is the same on -g, with the marker
// of the replayed band. With keys (order-preserving integers) for the heights:
//
//  1. every pixel points to the smallest of its neighbourhood by (height, index); the chains end in
//     local minima, which name the basins (k_descend, k_basins). A path from p may first descend to its
//     basin's bottom, so H(p) = max(g(p), level of the basin), its minimax height to the ocean;
//  2. Boruvka rounds on the basins: every component of basins not yet joined to the ocean finds its
//     lowest edge to another component, of height max(g, g) of two neighbouring pixels, or to the ocean
//     (k_edges), and is merged over it (k_hook, k_join). Any path out of a component crosses an edge at
//     least that high, so its basins' levels rise to that height; and a component's inner edges were the
//     lowest out of some part of it, so that the maximum over the rounds is the level exactly. Edges are
//     ordered by (height, edge index), a strict order, so the only cycles are pairs that chose the same
//     edge. Every round at least halves the components that are left; basins of noise shrink to a
//     third.
//
// Every value is a maximum or minimum of pixel values: the result is the unique reconstruction, the
// reference's bit for bit. Its comparisons are false for a NaN, which leaves such a pixel as it is and
// lets no path through: its height is kWall, above every other. A region whose level is not below that
// is shut in by such pixels; there the marker stays, the image's maximum (k_replace). There are no chains of dependent
// relaxations along paths: the work is full passes of 8 bytes per pixel while components are smaller
// than a tile, then only over tiles that still hold a boundary.
//
// Measured against row sweeps finished by a worklist, which are bound by the latency of their relaxation
// chains: see few_units.

constexpr int kOcean = -1, kNone = -2;
constexpr int kStripThreads = 256;
constexpr uint32_t kOceanEdge = 0xFFFFFFFFu;
constexpr int kRounds = 12;      // rounds as launches over the whole GPU
constexpr int kMostRounds = 40;  // 2^31 pixels need 31

typedef unsigned long long u64;

// One or two reconstructions of the same images (holes of the image, and of its negation): unit u <
// nimg is image u with sign[0], unit nimg + i image i with sign[1].
struct Flood {
    const int *pad;       // keys (k_to_keys)
    int flip0, flip1;     // 0, or -1 for the negated image
    int *lab0, *lab1;     // per pixel: while basins are found, the pixel pointed to or ~basin; then ~basin
    const float *band;    // peaks: the marker's border band per image (see band_at), else null
    int *comp, *lev, *par; // per unit and basin: component (a basin, or kOcean), level key, hook target
    u64 *best0, *best1;   // per unit and basin: a component's lowest edge, in even and odd rounds
    int *nbasin;          // per unit
    int *active;          // [round][unit]: components are left
    unsigned char *uniform; // per unit and strip: nothing to find here any more
    int nimg, units, pw, ph, cap;
    // (chosen by selects: an array indexed by the job would be copied to local memory by every thread)
    __device__ __forceinline__ int flip(int job) const { return job ? flip1 : flip0; }
    __device__ __forceinline__ int *lab(int job, int img) const
    {
        return (job ? lab1 : lab0) + img * (static_cast<size_t>(pw) * ph);
    }
    __device__ __forceinline__ u64 *best(int round) const { return round & 1 ? best1 : best0; }
};

constexpr int kWall = 0x7F800001; // height of a NaN (key INT_MIN, see k_to_keys), above +inf's

// Height of a pixel: its key, or its negation's (the complement, flip -1).
__device__ __forceinline__ int height(int key, int flip) { return key == INT_MIN ? kWall : key ^ flip; }

// Height at which the ocean enters pixel (x, y) of height gp; INT_MAX: not here. (Not below kWall at a
// NaN, whose band value is a NaN too.)
__device__ __forceinline__ int ocean_height(const Flood &F, int job, int img, int x, int y, int gp)
{
    if (!F.band) return x == 0 || y == 0 || x == F.pw - 1 || y == F.ph - 1 ? gp : INT_MAX;
    const int at = band_at(x, y, F.pw, F.ph);
    return at < 0 ? INT_MAX : max(gp, fkey(F.band[img * band_size(F.pw, F.ph) + at]) ^ F.flip(job));
}

// The passes over pixels give each warp a strip of kStripX columns by kStripY rows: lanes 1 .. 30 are its
// columns, lanes 0 and 31 the columns beside it, and the warp walks the rows with the last three in
// registers, neighbours of a row by shuffles. Bound by instruction issue, so that a value is loaded and
// turned into its height once per strip and there is no tile in shared memory.
constexpr int kStripX = 30, kStripY = 32, kStripBatch = 4;

struct Strip {
    int u, job, img, x, y0, y1, lane;
    bool in, mine; // a column of the image; of this strip
    size_t flag;   // of Flood::uniform
};

// The strip of this warp; false past the last one.
__device__ __forceinline__ bool strip_of(const Flood &F, int u, int task, Strip &S)
{
    const int across = (F.pw + kStripX - 1) / kStripX, down = (F.ph + kStripY - 1) / kStripY;
    if (task >= across * down) return false;
    const int sy = task / across, sx = task - sy * across;
    S.u = u;
    S.job = u >= F.nimg;
    S.img = u - S.job * F.nimg;
    S.lane = threadIdx.x & 31;
    S.x = sx * kStripX + S.lane - 1;
    S.y0 = sy * kStripY;
    S.y1 = min(S.y0 + kStripY, F.ph);
    S.in = S.x >= 0 && S.x < F.pw;
    S.mine = S.in && S.lane >= 1 && S.lane <= kStripX;
    S.flag = static_cast<size_t>(u) * (across * down) + task;
    return true;
}

// The padded images as keys, in place; a NaN of any bits as INT_MIN (whose float is a NaN again).
__global__ void __launch_bounds__(256) k_to_keys(float *__restrict__ pad, size_t n)
{
    int *key = reinterpret_cast<int *>(pad);
    for (size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
         i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const float v = pad[i];
        key[i] = v != v ? INT_MIN : fkey(v);
    }
}

// Each pixel's lowest neighbour by (height, index), or a basin of its own.
template <bool CONN8>
__global__ void __launch_bounds__(kStripThreads) k_descend(const Flood F)
{
    Strip S;
    if (!strip_of(F, blockIdx.y, blockIdx.x * (kStripThreads / 32) + (threadIdx.x >> 5), S)) return;
    const size_t n = static_cast<size_t>(F.pw) * F.ph;
    const int *pad = F.pad + S.img * n + (S.in ? S.x : 0);
    int *lab = F.lab(S.job, S.img);
    const int flip = F.flip(S.job);
    // heights of a row, and (8 neighbours) the lowest of three by index
    struct Row {
        int c, l, r, low, dx;
    };
    auto fetch = [&](int y) { return S.in && y >= 0 && y < F.ph ? height(__ldg(pad + static_cast<size_t>(y) * F.pw), flip) : INT_MAX; };
    auto row = [&](int h) {
        Row R;
        R.c = h;
        R.l = __shfl_up_sync(0xffffffffu, h, 1);
        R.r = __shfl_down_sync(0xffffffffu, h, 1);
        R.low = R.l;
        R.dx = -1;
        if (R.c < R.low) R.low = R.c, R.dx = 0;
        if (R.r < R.low) R.low = R.r, R.dx = 1;
        return R;
    };
    Row up = row(fetch(S.y0 - 1)), at = row(fetch(S.y0));
    unsigned rows = 0; // lane k: the bottoms of row k
    for (int yb = S.y0; yb < S.y1; yb += kStripBatch) {
        int ahead[kStripBatch];
#pragma unroll
        for (int k = 0; k < kStripBatch; ++k) ahead[k] = fetch(yb + 1 + k);
#pragma unroll
        for (int k = 0; k < kStripBatch; ++k) {
            const int y = yb + k;
            if (y >= S.y1) break; // uniform
            const Row down = row(ahead[k]);
            int low, dx = 0, dy = -1;
            if (CONN8) {
                low = up.low, dx = up.dx;
                if (at.low < low) low = at.low, dx = at.dx, dy = 0;
                if (down.low < low) low = down.low, dx = down.dx, dy = 1;
            } else {
                low = up.c;
                if (at.low < low) low = at.low, dx = at.dx, dy = 0;
                if (down.c < low) low = down.c, dx = 0, dy = 1;
            }
            const bool bottom = S.mine && dx == 0 && dy == 0;
            const unsigned bottoms = __ballot_sync(0xffffffffu, bottom);
            if (S.lane == y - S.y0) rows = bottoms;
            const int p = y * F.pw + S.x;
            if (S.mine && !bottom) lab[p] = p + dy * F.pw + dx;
            up = at;
            at = down;
        }
    }
    // the strip's bottoms numbered by one atomic: lane k holds row k's
    static_assert(kStripY <= 32, "a lane per row");
    int upto = __popc(rows);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, upto, o);
        if (S.lane >= o) upto += v;
    }
    int first = 0;
    if (S.lane == 31 && upto) first = atomicAdd(F.nbasin + S.u, upto);
    first = __shfl_sync(0xffffffffu, first, 31) + upto - __popc(rows);
    for (int k = 0; k < S.y1 - S.y0; ++k) {
        const unsigned bottoms = __shfl_sync(0xffffffffu, rows, k);
        const int id = __shfl_sync(0xffffffffu, first, k) + __popc(bottoms & ((1u << S.lane) - 1));
        if (!(bottoms >> S.lane & 1) || !MR_IN_BOUNDS(id, F.cap, kSiteSpotNbr)) continue;
        const size_t b = static_cast<size_t>(S.u) * F.cap + id;
        F.comp[b] = id;
        F.lev[b] = INT_MIN;
        F.best0[b] = ~0ull;
        lab[(S.y0 + k) * F.pw + S.x] = ~id;
    }
}

// Every pixel's basin: the chain to its end. Pixels written meanwhile end other chains early.
__global__ void __launch_bounds__(256) k_basins(const Flood F)
{
    const int u = blockIdx.y, job = u >= F.nimg, img = u - job * F.nimg;
    const int n = F.pw * F.ph;
    volatile int *lab = F.lab(job, img);
    constexpr int U = 4; // chains in flight per thread
    for (int p0 = blockIdx.x * 256 * U + threadIdx.x; p0 < n; p0 += gridDim.x * 256 * U) {
        int x[U];
        bool point[U], more = false;
#pragma unroll
        for (int k = 0; k < U; ++k) {
            const int p = p0 + k * 256;
            x[k] = p < n ? lab[p] : -1;
            point[k] = x[k] >= 0;
            more |= point[k];
        }
        while (more) {
            more = false;
#pragma unroll
            for (int k = 0; k < U; ++k) {
                if (x[k] >= 0) x[k] = lab[x[k]];
                more |= x[k] >= 0;
            }
        }
#pragma unroll
        for (int k = 0; k < U; ++k)
            if (point[k]) lab[p0 + k * 256] = x[k];
    }
}

// Lowest edges of the components in one strip. The lowest height of a pixel's edges is max(g, least g
// of the neighbours in other components). A pixel that does not beat its component's edge so far ends
// there. Edges of one height are ordered by their index, 4 * (smaller pixel) + direction (0 right, 1
// down, 2 down right, 3 down left): up left, up, up right, left, right, down, down right, down left, and
// the pixel's is the first of these not above its height. A run of kStripBatch rows in which no pixel
// has an edge is skipped from then on (a bit of `uniform`).
template <bool CONN8>
__device__ __forceinline__ void edges_of_strip(const Flood &F, const Strip &S, int round)
{
    static_assert(kStripY / kStripBatch <= 8, "a bit per run of rows");
    unsigned skip = F.uniform[S.flag];
    if (skip == 0xFF) return; // warp-uniform
    const size_t n = static_cast<size_t>(F.pw) * F.ph;
    const int *pad = F.pad + S.img * n + (S.in ? S.x : 0);
    const int *lab = F.lab(S.job, S.img) + (S.in ? S.x : 0);
    const int *comp = F.comp + static_cast<size_t>(S.u) * F.cap;
    u64 *best = F.best(round) + static_cast<size_t>(S.u) * F.cap;
    const int flip = F.flip(S.job), pw = F.pw, ph = F.ph;
    const bool shore = S.mine && (F.band ? S.x <= 1 || S.x >= pw - 2 : S.x == 0 || S.x == pw - 1); // a column the ocean touches
    struct Row {
        int c, cl, cr, g, gl, gr;
    };
    auto row = [&](int c, int g) {
        Row R;
        R.c = c;
        R.g = g;
        R.cl = __shfl_up_sync(0xffffffffu, c, 1);
        R.cr = __shfl_down_sync(0xffffffffu, c, 1);
        R.gl = __shfl_up_sync(0xffffffffu, g, 1);
        R.gr = __shfl_down_sync(0xffffffffu, g, 1);
        return R;
    };
    // pixels outside the image are higher than any: never the lowest neighbour
    auto label = [&](int y) { return S.in && y >= 0 && y < ph ? ~lab[static_cast<size_t>(y) * pw] : -1; };
    auto value = [&](int y) { return S.in && y >= 0 && y < ph ? height(pad[static_cast<size_t>(y) * pw], flip) : INT_MAX; };
    auto component = [&](int l) { return l >= 0 ? comp[l] : kNone; };
    Row up{}, at{};
    bool have = false;
    for (int yb = S.y0, run = 0; yb < S.y1; yb += kStripBatch, ++run) {
        if (skip >> run & 1) { // uniform
            have = false;
            continue;
        }
        int l[kStripBatch], c[kStripBatch], g[kStripBatch];
        uint32_t limit[kStripBatch]; // height of the component's edge so far, as ordered unsigned
#pragma unroll
        for (int k = 0; k < kStripBatch; ++k) {
            l[k] = label(yb + 1 + k);
            g[k] = value(yb + 1 + k);
        }
        if (!have) {
            const int lu = label(yb - 1), la = label(yb);
            const int gu = value(yb - 1), ga = value(yb);
            up = row(component(lu), gu);
            at = row(component(la), ga);
            have = true;
        }
#pragma unroll
        for (int k = 0; k < kStripBatch; ++k) c[k] = component(l[k]);
#pragma unroll
        for (int k = 0; k < kStripBatch; ++k) {
            const int own = k == 0 ? at.c : c[k - 1];
            limit[k] = S.mine && own >= 0 ? reinterpret_cast<const uint32_t *>(best + own)[1] : 0;
        }
        bool differ = false;
#pragma unroll
        for (int k = 0; k < kStripBatch; ++k) {
            const int y = yb + k;
            if (y >= S.y1) break; // uniform
            const Row down = row(c[k], g[k]);
            int least = INT_MAX;
            auto see = [&](int cq, int gq) { least = min(least, cq != at.c ? gq : INT_MAX); };
            see(up.c, up.g), see(at.cl, at.gl), see(at.cr, at.gr), see(down.c, down.g);
            if (CONN8) see(up.cl, up.gl), see(up.cr, up.gr), see(down.cl, down.gl), see(down.cr, down.gr);
            int sea = INT_MAX;
            if ((shore || (F.band ? y <= 1 : y == 0) || y == ph - 1) && S.mine && at.c != kOcean)
                sea = ocean_height(F, S.job, S.img, S.x, y, at.g);
            const int low = min(max(at.g, least), sea);
            const bool any = S.mine && min(least, sea) != INT_MAX;
            differ |= any;
            if (any && (static_cast<uint32_t>(low) ^ 0x80000000u) <= limit[k]) {
                const uint32_t p4 = 4u * (static_cast<uint32_t>(y) * pw + S.x), w4 = 4u * pw;
                uint32_t edge = kOceanEdge;
                if (max(at.g, least) <= low) {
                    auto first = [&](int cq, int gq, uint32_t e) { edge = cq != at.c && gq <= low ? e : edge; };
                    if (CONN8) first(down.cl, down.gl, p4 + 3), first(down.cr, down.gr, p4 + 2);
                    first(down.c, down.g, p4 + 1), first(at.cr, at.gr, p4), first(at.cl, at.gl, p4 - 4);
                    if (CONN8) first(up.cr, up.gr, p4 - w4 + 4 + 3);
                    first(up.c, up.g, p4 - w4 + 1);
                    if (CONN8) first(up.cl, up.gl, p4 - w4 - 4 + 2);
                }
                const u64 e = static_cast<u64>(static_cast<uint32_t>(low) ^ 0x80000000u) << 32 | edge;
                if (e < __ldcg(best + at.c)) atomicMin(best + at.c, e);
            }
            up = at;
            at = down;
        }
        if (!__any_sync(0xffffffffu, differ)) skip |= 1u << run;
    }
    if (S.y1 - S.y0 < kStripY) skip |= 0xFFu << (S.y1 - S.y0 + kStripBatch - 1) / kStripBatch; // rows past the image
    if (S.lane == 0) F.uniform[S.flag] = static_cast<unsigned char>(skip);
}

template <bool CONN8>
__global__ void __launch_bounds__(kStripThreads) k_edges(const Flood F, int round)
{
    if (round > 0 && !F.active[static_cast<size_t>(round) * F.units + blockIdx.y]) return;
    Strip S;
    if (strip_of(F, blockIdx.y, blockIdx.x * (kStripThreads / 32) + (threadIdx.x >> 5), S)) edges_of_strip<CONN8>(F, S, round);
}

// A component's hook: the component at the other end of its lowest edge; of a pair that chose the same
// edge the smaller stays.
__device__ __forceinline__ void hook(const Flood &F, int u, int r, int round)
{
    const size_t base = static_cast<size_t>(u) * F.cap;
    if (F.comp[base + r] != r) return;
    F.best(round + 1)[base + r] = ~0ull; // the components left are among these
    const int job = u >= F.nimg, img = u - job * F.nimg;
    const int *lab = F.lab(job, img);
    const u64 e = F.best(round)[base + r];
    const uint32_t edge = static_cast<uint32_t>(e);
    int to = kOcean;
    if (edge != kOceanEdge) {
        const uint32_t p = edge >> 2, dir = edge & 3;
        const uint32_t q = p + (dir == 0 ? 1 : dir == 1 ? F.pw : dir == 2 ? F.pw + 1 : F.pw - 1);
        const int cp = F.comp[base + ~lab[p]], cq = F.comp[base + ~lab[q]];
        to = cp == r ? cq : cp;
        if (to >= 0 && r < to && F.best(round)[base + to] == e) to = r;
    }
    F.par[base + r] = to;
}

// A basin's new component and level. True when it is a component that is left.
__device__ __forceinline__ bool join(const Flood &F, int u, int b, int round)
{
    const size_t base = static_cast<size_t>(u) * F.cap;
    const int c = F.comp[base + b];
    if (c == kOcean) return false;
    const int h = static_cast<int>(static_cast<uint32_t>(F.best(round)[base + c] >> 32) ^ 0x80000000u);
    F.lev[base + b] = max(F.lev[base + b], h);
    int x = F.par[base + c];
    while (x >= 0) {
        const int y = F.par[base + x];
        if (y == x) break;
        x = y;
    }
    F.comp[base + b] = x;
    return x == b;
}

__global__ void __launch_bounds__(256) k_hook(const Flood F, int round)
{
    const int u = blockIdx.y;
    if (round > 0 && !F.active[static_cast<size_t>(round) * F.units + u]) return;
    const int nb = F.nbasin[u];
    for (int b = blockIdx.x * 256 + threadIdx.x; b < nb; b += gridDim.x * 256) hook(F, u, b, round);
}

// comp is written here while other threads follow par only.
__global__ void __launch_bounds__(256) k_join(const Flood F, int round)
{
    const int u = blockIdx.y;
    if (round > 0 && !F.active[static_cast<size_t>(round) * F.units + u]) return;
    const int nb = F.nbasin[u];
    bool left = false;
    for (int b = blockIdx.x * 256 + threadIdx.x; b < nb; b += gridDim.x * 256) left |= join(F, u, b, round);
    if (__any_sync(0xffffffffu, left) && (threadIdx.x & 31) == 0) F.active[static_cast<size_t>(round + 1) * F.units + u] = 1;
}

// The rounds that are left (usually none), one CTA per unit.
template <bool CONN8>
__global__ void __launch_bounds__(kStripThreads) k_finish(const Flood F, int round)
{
    const int u = blockIdx.x, nb = F.nbasin[u];
    bool left = F.active[static_cast<size_t>(round) * F.units + u] != 0;
    for (; left && round < kMostRounds; ++round) { // uniform
        Strip S;
        for (int task = threadIdx.x >> 5; strip_of(F, u, task, S); task += kStripThreads / 32) edges_of_strip<CONN8>(F, S, round);
        __syncthreads();
        for (int b = threadIdx.x; b < nb; b += kStripThreads) hook(F, u, b, round);
        __syncthreads();
        bool more = false;
        for (int b = threadIdx.x; b < nb; b += kStripThreads) more |= join(F, u, b, round);
        left = __syncthreads_or(more);
    }
    if (left && threadIdx.x == 0) atomicExch(&g_msc_error, 2);
}

// Basins of an image: local minima are not neighbours, so with 8 neighbours at most one pixel of each
// 2 x 2 block, with 4 every second one.
inline size_t most_basins(int pw, int ph, int conn8)
{
    const size_t hw = (pw + 1) / 2, hh = (ph + 1) / 2;
    return conn8 ? hw * hh : (static_cast<size_t>(pw) * ph + 1) / 2;
}

inline size_t strips_of(int pw, int ph) { return div_up(pw, kStripX) * static_cast<size_t>(div_up(ph, kStripY)); }

// Basin levels of the units (lab and lev on return; see Flood).
template <bool CONN8>
static mr_status launch_flood(const Flood &F, cudaStream_t s)
{
    const size_t n = static_cast<size_t>(F.pw) * F.ph;
    MR_CUDA_TRY(cudaMemsetAsync(F.nbasin, 0, F.units * sizeof(int), s));
    MR_CUDA_TRY(cudaMemsetAsync(F.active, 0, (kMostRounds + 1) * static_cast<size_t>(F.units) * sizeof(int), s));
    MR_CUDA_TRY(cudaMemsetAsync(F.uniform, 0, F.units * strips_of(F.pw, F.ph), s));
    const dim3 strips(div_up(strips_of(F.pw, F.ph), kStripThreads / 32), F.units);
    const unsigned per = std::max(1u, 148 * 8 / static_cast<unsigned>(F.units));
    const dim3 flat(std::min<unsigned>(div_up(n, 1024), std::max(per, 16u)), F.units);
    const dim3 basins(std::min<unsigned>(div_up(static_cast<size_t>(F.cap), 256), std::max(per, 4u)), F.units);
    k_descend<CONN8><<<strips, kStripThreads, 0, s>>>(F);
    k_basins<<<flat, 256, 0, s>>>(F);
    for (int r = 0; r < kRounds; ++r) {
        k_edges<CONN8><<<strips, kStripThreads, 0, s>>>(F, r);
        k_hook<<<basins, 256, 0, s>>>(F, r);
        k_join<<<basins, 256, 0, s>>>(F, r);
    }
    k_finish<CONN8><<<F.units, kStripThreads, 0, s>>>(F, kRounds);
    return check_launch("morphspotclean reconstruction");
}

// ---- reconstruction by row sweeps and a worklist (many images; see few_units)

// One or two reconstructions of the same images in one launch (FillHole of the image and of its
// negation in the 'both' mode): CTA b < nimg works on image b with sign[0] into vol[0], CTA
// nimg + b on image b with sign[1] into vol[1]. Independent images share the SMs, so the long
// completions of either set overlap.
struct RecJobs {
    float sign[2];
    float *vol[2];
    int nimg;
    const int *interior[2]; // per-image interior value (key) of the marker, formed by the sweeps; null:
                              // the marker is in vol already
};

// Exact reconstruction by alternating row sweeps (see the file comment), one warp per image.
// DILATE: v = min(g, max over neighbourhood); else v = max(g, min over neighbourhood); g is
// `sign * pad`. Rows are staged in shared memory (coalesced global traffic); lane l owns the
// contiguous chunk [l*C, l*C + C) of a row, C odd so that the 32 lanes' chunk positions fall
// in 32 different banks. Positions beyond the row hold the neutral value (-inf for
// dilation, +inf for erosion), which neither propagates into the row nor changes.

//
// A NaN of the mask takes and passes on nothing, as in the reference, whose comparisons it fails: the
// outer operation keeps it, the inner one takes the other operand.
template <bool DILATE>
__device__ __forceinline__ float rec_op(float g, float v, float x)
{
    const float inner = DILATE ? fmaxf(v, x) : fminf(v, x);
    float r;
    if (DILATE) asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(g), "f"(inner));
    else asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(g), "f"(inner));
    return r;
}

// Key of a mask or marker value; of a NaN the one that improves no neighbour and that nothing improves.
// (The NaN that arithmetic makes, as in sign * g and rec_op, is 0x7FFFFFFF: its fkey is INT_MAX.)
template <bool DILATE>
__device__ __forceinline__ int rec_key(float v)
{
    return DILATE && v != v ? INT_MIN : fkey(v);
}

__device__ __forceinline__ void cp_async4(float *dst, const float *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
                 "l"(src)
                 : "memory");
}

__device__ __forceinline__ void cp_async_wait_all()
{
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}

// Barrier of the RW warps of one image (named barrier 1 + image slot; the block holds one image).
template <int RW>
__device__ __forceinline__ void image_sync()
{
    if constexpr (RW == 1) __syncwarp();
    else asm volatile("bar.sync 1, %0;" ::"n"(RW * 32) : "memory");
}

// Clamp pair of a run of elements: for dilation F(x) = min(hi, max(lo, x)) with lo = F(-inf),
// hi = F(+inf); for erosion the same with min/max exchanged (lo = F(+inf), hi = F(-inf)).
// (a then b): apply a first.
template <bool DILATE>
__device__ __forceinline__ void clamp_then(float al, float ah, float &bl, float &bh)
{
    const float nl = rec_op<DILATE>(bh, bl, al), nh = rec_op<DILATE>(bh, bl, ah);
    bl = nl;
    bh = nh;
}

// One image per block of RW warps; lane t of the image owns the row chunk [t*C, t*C + C), held
// in registers across the vertical step and both scans. C odd: the lanes' chunk positions in
// the shared row buffers fall in distinct banks.
//
// The marker leaves this kernel as keys (fkey): the upward sweep of the last round stores them,
// and an image that converged earlier is converted by one more pass. That sweep also lists the
// pixels it changed (at most cap, then only counted) as the completion's first worklist: after
// it every pixel has been relaxed from its neighbours' current values except from those in the
// row above it that changed later in the sweep, and exactly those are listed. An image whose
// round changed nothing is finished and lists nothing.
template <bool DILATE, int RW, int C>
__global__ void __launch_bounds__(32 * RW) k_reconstruct(const float *__restrict__ pad, RecJobs jobs, int pw, int ph,
                                                         int conn8, int rounds, int *__restrict__ lists, int cap,
                                                         int *__restrict__ counts)
{
    static_assert(C <= 64, "per-pixel change mask");
    const int job = blockIdx.x >= jobs.nimg, img = blockIdx.x - job * jobs.nimg;
    const float sign = jobs.sign[job];
    constexpr int T = 32 * RW, L = T * C + 2 + 1; // row buffer: a neutral element before and after
    extern __shared__ float rows_sm[];
    float(*Gb)[L] = reinterpret_cast<float(*)[L]>(rows_sm);         // [2][L] mask rows
    float(*Rb)[L] = reinterpret_cast<float(*)[L]>(rows_sm + 2 * L); // [3][L] marker rows
    __shared__ float wagg[2][RW][2];
    __shared__ int any_changed[2];
    __shared__ int listed;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const size_t n = static_cast<size_t>(pw) * ph;
    const float *g = pad + img * n;
    float *v = jobs.vol[job] + img * n;
    int *list = lists + blockIdx.x * 2 * static_cast<size_t>(cap);
    const float neutral = DILATE ? -FLT_MAX : FLT_MAX;
    for (int c = t; c < L; c += T) {
        Gb[0][c] = Gb[1][c] = neutral * sign; // sign * stored = neutral
        Rb[0][c] = Rb[1][c] = Rb[2][c] = neutral;
    }
    if (t < 2) any_changed[t] = 0;
    if (t == 0) listed = 0;
    __syncthreads();
    const int c0 = 1 + t * C; // buffer index of the chunk's first element (index 0 is the lead)
    // row y of the mask into G and of the marker into V; from_marker: the initial marker row,
    // formed here (the image on the border, the interior value inside; morphextrema.h:268-283)
    const int *inter = jobs.interior[job];
    const float in_val = inter ? sign * funkey(inter[img]) : 0.0f;
    auto fetch = [&](int y, float *G, float *V, bool from_marker) {
        const size_t ro = static_cast<size_t>(y) * pw;
        const bool brow = y == 0 || y == ph - 1;
        for (int c = t; c < pw; c += T) {
            cp_async4(G + 1 + c, g + ro + c);
            if (!from_marker) cp_async4(V + 1 + c, v + ro + c);
            else V[1 + c] = brow || c == 0 || c == pw - 1 ? sign * g[ro + c] : in_val;
        }
    };
    // exclusive scan over the image's lanes of clamp pairs; returns the carry into this lane
    auto carry_in = [&](float xl, float xh, bool fwd, int slot) -> float {
        for (int o = 1; o < 32; o <<= 1) {
            const float pl = fwd ? __shfl_up_sync(0xffffffffu, xl, o) : __shfl_down_sync(0xffffffffu, xl, o);
            const float pu = fwd ? __shfl_up_sync(0xffffffffu, xh, o) : __shfl_down_sync(0xffffffffu, xh, o);
            if (fwd ? lane >= o : lane + o < 32) clamp_then<DILATE>(pl, pu, xl, xh);
        }
        // (xl, xh): inclusive prefix within the warp
        float before_l = neutral, before_h = -neutral; // identity
        if constexpr (RW > 1) {
            if (fwd ? lane == 31 : lane == 0) {
                wagg[slot][warp][0] = xl;
                wagg[slot][warp][1] = xh;
            }
            image_sync<RW>();
            // warps earlier in the scan direction, in order (copies: wagg is shared)
            for (int k = 0; k < RW; ++k) {
                const int w = fwd ? k : RW - 1 - k;
                if (fwd ? w >= warp : w <= warp) break;
                float bl = wagg[slot][w][0], bh = wagg[slot][w][1];
                clamp_then<DILATE>(before_l, before_h, bl, bh);
                before_l = bl;
                before_h = bh;
            }
        }
        // lanes before this one within the warp
        float il = fwd ? __shfl_up_sync(0xffffffffu, xl, 1) : __shfl_down_sync(0xffffffffu, xl, 1);
        float ih = fwd ? __shfl_up_sync(0xffffffffu, xh, 1) : __shfl_down_sync(0xffffffffu, xh, 1);
        if (fwd ? lane > 0 : lane < 31) {
            clamp_then<DILATE>(before_l, before_h, il, ih);
            before_l = il;
        }
        return before_l; // the prefix applied to the neutral input
    };

    // one sweep (pass 0 downward, 1 upward); LAST: the upward sweep of the last round, which lists
    // the pixels it changes and stores keys. Returns whether this thread's chunks changed.
    auto sweep = [&](int pass, bool from_marker, auto last_tag) -> bool {
        constexpr bool LAST = decltype(last_tag)::value;
        bool changed = false;
        int gi = 0, vi = 0;
        fetch(pass == 0 ? 0 : ph - 1, Gb[0], Rb[0], from_marker);
        cp_async_wait_all();
        image_sync<RW>();
        for (int step = 0; step < ph; ++step) {
            const int y = pass == 0 ? step : ph - 1 - step;
            const float *G = Gb[gi];
            float *V = Rb[vi];
            const float *Pv = Rb[(vi + 2) % 3];
            if (step + 1 < ph) fetch(pass == 0 ? y + 1 : y - 1, Gb[gi ^ 1], Rb[(vi + 1) % 3], from_marker);
            float gv[C], cv[C];
            unsigned long long chg = 0; // LAST: bit j = element j of the chunk changed in this step
            auto note = [&](int j, bool moved) {
                if constexpr (LAST) chg |= static_cast<unsigned long long>(moved) << j;
                else changed |= moved;
            };
#pragma unroll
            for (int j = 0; j < C; ++j) {
                gv[j] = sign * G[c0 + j];
                cv[j] = V[c0 + j];
            }
            if (step > 0) {
#pragma unroll
                for (int j = 0; j < C; ++j) {
                    float nb = Pv[c0 + j];
                    if (conn8)
                        nb = DILATE ? fmaxf(nb, fmaxf(Pv[c0 + j - 1], Pv[c0 + j + 1]))
                                    : fminf(nb, fminf(Pv[c0 + j - 1], Pv[c0 + j + 1]));
                    const float nvl = rec_op<DILATE>(gv[j], cv[j], nb);
                    note(j, nvl != cv[j]);
                    cv[j] = nvl;
                }
            }
            // forward along the row
            {
                float lo = neutral, hi = -neutral;
#pragma unroll
                for (int j = 0; j < C; ++j) {
                    lo = rec_op<DILATE>(gv[j], cv[j], lo);
                    hi = rec_op<DILATE>(gv[j], cv[j], hi);
                }
                float run = carry_in(lo, hi, true, 0);
#pragma unroll
                for (int j = 0; j < C; ++j) {
                    run = rec_op<DILATE>(gv[j], cv[j], run);
                    note(j, run != cv[j]);
                    cv[j] = run;
                }
            }
            // backward
            {
                float lo = neutral, hi = -neutral;
#pragma unroll
                for (int j = C - 1; j >= 0; --j) {
                    lo = rec_op<DILATE>(gv[j], cv[j], lo);
                    hi = rec_op<DILATE>(gv[j], cv[j], hi);
                }
                float run = carry_in(lo, hi, false, 1);
#pragma unroll
                for (int j = C - 1; j >= 0; --j) {
                    run = rec_op<DILATE>(gv[j], cv[j], run);
                    note(j, run != cv[j]);
                    cv[j] = run;
                }
            }
            if constexpr (LAST) {
                changed |= chg != 0;
                // positions past the row never change (neutral), so every bit is a pixel
                if (chg) {
#pragma unroll
                    for (int j = 0; j < C; ++j) {
                        if (!((chg >> j) & 1)) continue;
                        const int pos = atomicAdd(&listed, 1);
                        if (pos < cap) list[pos] = y * pw + c0 + j - 1;
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < C; ++j) V[c0 + j] = cv[j];
            image_sync<RW>();
            const size_t ro = static_cast<size_t>(y) * pw;
            if constexpr (LAST) {
                int *vk = reinterpret_cast<int *>(v);
                for (int c = t; c < pw; c += T) vk[ro + c] = rec_key<DILATE>(V[1 + c]);
            } else {
                for (int c = t; c < pw; c += T) v[ro + c] = V[1 + c];
            }
            cp_async_wait_all(); // the next row has landed
            image_sync<RW>();
            gi ^= 1;
            vi = (vi + 1) % 3;
        }
        return changed;
    };

    bool keys = false; // the marker in global memory is stored as keys
    for (int round = 0; round < rounds; ++round) {
        bool changed = sweep(0, round == 0 && inter, std::false_type{});
        if (round == rounds - 1) {
            changed |= sweep(1, false, std::true_type{});
            keys = true;
        } else {
            changed |= sweep(1, false, std::false_type{});
        }
        // image-wide vote (alternating flags: the one read now is cleared for the round after)
        if (changed) any_changed[round & 1] = 1;
        image_sync<RW>();
        const int any = any_changed[round & 1];
        if (t == 0) any_changed[(round + 1) & 1] = 0;
        image_sync<RW>();
        if (!any) break;
    }
    if (!keys) {
        // converged before the last round: nothing to list; store the marker as keys
        int *vk = reinterpret_cast<int *>(v);
        for (size_t i = t; i < n; i += T) vk[i] = rec_key<DILATE>(__int_as_float(vk[i]));
    }
    if (t == 0) counts[blockIdx.x] = listed; // the pushes precede the barriers of the last vote
}

template <bool DILATE, int RW, int C>
static mr_status launch_rec(const RecJobs &jobs, int njobs, const float *pad, int pw, int ph, int conn8, int *lists,
                            int cap, int *counts, cudaStream_t s)
{
    const size_t smem = 5 * static_cast<size_t>(32 * RW * C + 3) * sizeof(float);
    MR_CUDA_TRY(cudaFuncSetAttribute(k_reconstruct<DILATE, RW, C>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     static_cast<int>(smem)));
    k_reconstruct<DILATE, RW, C><<<jobs.nimg * njobs, 32 * RW, smem, s>>>(pad, jobs, pw, ph, conn8, kSweepRounds,
                                                                          lists, cap, counts);
    return check_launch("k_reconstruct");
}

// ---- completion: worklist relaxation
//
// After the sweeps the remaining changes are sparse (thin, winding paths through the noise),
// so each image's CTA finishes the reconstruction with a worklist. Values are order-preserving
// integer keys (the sweeps leave them so) so that the relaxation is one atomicMin (erosion:
// v[q] = min(v[q], max(g[q], v[p]))) or atomicMax (dilation: v[q] = max(v[q], min(g[q], v[p])))
// per neighbour. The first list is the sweeps' (the pixels their last sweep changed); an image
// whose sweeps converged lists nothing and is done. A relaxation is issued, without waiting for
// its result, when its candidate improves the neighbour's value as loaded, and the neighbour is
// then listed for the next iteration (or followed, below): every change of a value is made by
// such an update, whose pixel is listed with the value written, so the last value of every
// pixel is propagated; a listing whose update lost to a better concurrent one only repeats
// work. It then relaxes its neighbours with its current value. When a list overflows, the next
// iteration relaxes every pixel from its neighbours instead. The reconstruction ends when an
// iteration lists nothing: every pixel then satisfies the fixpoint equations with all its
// neighbours, and the fixpoint is unique, so the result equals the reference's whatever the
// order of the updates. Values are read through L2 (ld.cg), where the atomics resolve. Latency
// shapes the code: an entry issues all its neighbour loads, then all its updates, and the dense
// passes handle kUnroll pixels per thread at a time.

constexpr int kFrontThreads = 512;
constexpr int kMaxIterations = 1 << 22;
constexpr int kUnroll = 4;
constexpr int kChase = 32; // pixels one thread follows within an iteration

template <bool DILATE>
__device__ __forceinline__ void relax(int *addr, int c)
{
    if (DILATE) atomicMax(addr, c);
    else atomicMin(addr, c);
}

template <bool DILATE, bool CONN8>
__global__ void __launch_bounds__(kFrontThreads) k_complete(const float *__restrict__ pad, RecJobs jobs, int pw,
                                                            int ph, int *__restrict__ lists, int cap,
                                                            const int *__restrict__ counts)
{
    const int first = counts[blockIdx.x]; // the sweeps' list (uniform over the CTA)
    if (first == 0) return;
    const int t = threadIdx.x;
    const int n = pw * ph;
    const int job = blockIdx.x >= jobs.nimg, img = blockIdx.x - job * jobs.nimg;
    const float sign = jobs.sign[job];
    const float *g = pad + img * static_cast<size_t>(n);
    int *v = reinterpret_cast<int *>(jobs.vol[job] + img * static_cast<size_t>(n));
    int *cur = lists + blockIdx.x * 2 * static_cast<size_t>(cap), *next = cur + cap;
    __shared__ int count[3];
    if (t < 3) count[t] = 0;
    __syncthreads();

    const int nx[8] = {-1, 1, 0, 0, -1, 1, -1, 1}, ny[8] = {0, 0, -1, 1, -1, -1, 1, 1};
    constexpr int NN = CONN8 ? 8 : 4;
    auto improves = [](int c, int old) { return DILATE ? c > old : c < old; };
    auto push = [&](int q, int it) {
        const int pos = atomicAdd(&count[it % 3], 1);
        if (pos < cap) next[pos] = q;
    };

    bool dense = first > cap;
    int nf = min(first, cap), it = 0;
    for (; it < kMaxIterations; ++it) {
        if (dense) {
            // every pixel from the extreme of its neighbours, kUnroll pixels at a time
            for (int i0 = t; i0 < n; i0 += kUnroll * kFrontThreads) {
                int c[kUnroll], kv[kUnroll];
#pragma unroll
                for (int u = 0; u < kUnroll; ++u) {
                    const int i = i0 + u * kFrontThreads;
                    const int y = i / pw, x = i % pw;
                    int kn = DILATE ? INT_MIN : INT_MAX;
#pragma unroll
                    for (int k = 0; k < NN; ++k) {
                        const int qx = x + nx[k], qy = y + ny[k];
                        if (i >= n || qx < 0 || qx >= pw || qy < 0 || qy >= ph) continue;
                        const int kq = __ldcg(v + qy * pw + qx);
                        kn = DILATE ? max(kn, kq) : min(kn, kq);
                    }
                    const int kg = i < n ? rec_key<DILATE>(sign * __ldg(g + i)) : 0;
                    c[u] = DILATE ? min(kg, kn) : max(kg, kn);
                    kv[u] = i < n ? __ldcg(v + i) : c[u];
                }
#pragma unroll
                for (int u = 0; u < kUnroll; ++u) {
                    if (!improves(c[u], kv[u])) continue;
                    relax<DILATE>(v + i0 + u * kFrontThreads, c[u]);
                    push(i0 + u * kFrontThreads, it);
                }
            }
        } else {
            for (int e = t; e < nf; e += kFrontThreads) {
                // relax the neighbours of p; the thread then follows the first neighbour it moved
                // (chasing) for up to kChase steps and lists the others it moved, so a change
                // travels along a path without waiting for a barrier per pixel. Every moved
                // pixel is relaxed afterwards, by this thread's chase or from the next list.
                int p = cur[e];
                // value of p: read for a listed pixel; for a chased one, the value this thread
                // just gave it (a lower value someone else gave it meanwhile is propagated by that
                // thread, and a candidate from a higher one is still an upper bound of the
                // result), which saves a round trip to L2 per step
                int kp = __ldcg(v + p);
                for (int step = 0; p >= 0; ++step) {
                    const int y = p / pw, x = p % pw;
                    int c[NN], kv[NN];
                    unsigned ok = 0;
#pragma unroll
                    for (int k = 0; k < NN; ++k) {
                        const int qx = x + nx[k], qy = y + ny[k];
                        const bool in = qx >= 0 && qx < pw && qy >= 0 && qy < ph;
                        const int q = qy * pw + qx;
                        const int kg = in ? rec_key<DILATE>(sign * __ldg(g + q)) : 0;
                        kv[k] = in ? __ldcg(v + q) : 0;
                        c[k] = DILATE ? min(kg, kp) : max(kg, kp);
                        if (in && improves(c[k], kv[k])) ok |= 1u << k;
                    }
                    int follow = -1, kf = 0;
#pragma unroll
                    for (int k = 0; k < NN; ++k) {
                        if (!((ok >> k) & 1)) continue;
                        const int q = p + ny[k] * pw + nx[k];
                        if (!MR_IN_BOUNDS(q, n, kSiteSpotNbr)) continue;
                        relax<DILATE>(v + q, c[k]);
                        if (follow < 0 && step + 1 < kChase) {
                            follow = q;
                            kf = c[k];
                        } else {
                            push(q, it);
                        }
                    }
                    p = follow;
                    kp = kf;
                }
            }
        }
        __syncthreads();
        // count[it % 3] is final; count[(it + 2) % 3] was read by everyone before this barrier
        // and is next written in iteration it + 2
        const int pushed = count[it % 3];
        if (t == 0) count[(it + 2) % 3] = 0;
        int *tmp = cur;
        cur = next;
        next = tmp;
        if (pushed == 0) break;
        dense = pushed > cap;
        nf = min(pushed, cap);
    }
    if (it == kMaxIterations && t == 0) atomicExch(&g_msc_error, 2);
}

// Worklist capacity per image (entries); a larger frontier falls back to a dense iteration.
inline int complete_cap(size_t n) { return static_cast<int>(std::min<size_t>(n, std::max<size_t>(256, n / 16))); }

// Sweeps, then the completion, of jobs.nimg x njobs reconstructions (one CTA each). lists: two
// worklists of complete_cap entries per CTA; counts: one word per CTA (the sweeps' list length).
template <bool DILATE>
static mr_status launch_reconstruct(const RecJobs &jobs, int njobs, const float *pad, int pw, int ph, int conn8,
                                    int *lists, int *counts, cudaStream_t s)
{
    constexpr int RW = 4;
    const int per = (pw + 32 * RW - 1) / (32 * RW);
    const int cap = complete_cap(static_cast<size_t>(pw) * ph);
    mr_status st;
    if (per <= 3) st = launch_rec<DILATE, RW, 3>(jobs, njobs, pad, pw, ph, conn8, lists, cap, counts, s);
    else if (per <= 5) st = launch_rec<DILATE, RW, 5>(jobs, njobs, pad, pw, ph, conn8, lists, cap, counts, s);
    else if (per <= 9) st = launch_rec<DILATE, RW, 9>(jobs, njobs, pad, pw, ph, conn8, lists, cap, counts, s);
    else if (per <= 17) st = launch_rec<DILATE, RW, 17>(jobs, njobs, pad, pw, ph, conn8, lists, cap, counts, s);
    else if (per <= 33) st = launch_rec<DILATE, RW, 33>(jobs, njobs, pad, pw, ph, conn8, lists, cap, counts, s);
    else return fail(MR_ERR_UNSUPPORTED, "mr_morphspotclean: rows longer than %d pixels", 32 * RW * 33 - 2 * kMargin);
    if (st != MR_OK) return st;
    const int nb = jobs.nimg * njobs;
    if (conn8) k_complete<DILATE, true><<<nb, kFrontThreads, 0, s>>>(pad, jobs, pw, ph, lists, cap, counts);
    else k_complete<DILATE, false><<<nb, kFrontThreads, 0, s>>>(pad, jobs, pw, ph, lists, cap, counts);
    return check_launch("k_complete");
}

// Replacement / blend and unpadding (MorphSpotClean::ProcessReplace :108-175,
// kipl::math::SigmoidWeights mathfunctions.hpp:92-99).
template <bool LEVELS>
__global__ void k_replace(const void *__restrict__ pad, const int *__restrict__ hole_lab, const int *__restrict__ hole_lev,
                          const int *__restrict__ peak_lab, const int *__restrict__ peak_lev, size_t cap,
                          const int *__restrict__ mn, const int *__restrict__ mx, int w, int h, int detect, float th0,
                          float th1, float s0, float s1, float *__restrict__ img)
{
    const int pw = w + 2 * kMargin, ph = h + 2 * kMargin;
    const size_t n = static_cast<size_t>(pw) * ph;
    const int b = blockIdx.y;
    const size_t per = static_cast<size_t>(w) * h;
    for (int y = blockIdx.x; y < h; y += gridDim.x)
    for (int x = threadIdx.x; x < w; x += blockDim.x) {
        const size_t idx = static_cast<size_t>(y) * w + x;
        const size_t pi = b * n + static_cast<size_t>(y + kMargin) * pw + x + kMargin;
        // LEVELS: the image as keys, a reconstruction the larger of the pixel and its basin's level (peaks:
        // of the negated image), or the marker where no path leads; else reconstructions stored as keys
        // (peaks alone: of the image itself)
        float val, hv = 0.0f, pv = 0.0f;
        bool stays = false;
        if (LEVELS) {
            const int key = static_cast<const int *>(pad)[pi];
            stays = key == INT_MIN; // a NaN, with its bits (no branch: the loads below need not wait for the key)
            val = funkey(key);
            if (hole_lab) {
                const int rec = max(key, hole_lev[b * cap + ~hole_lab[pi]]);
                hv = funkey(rec);
                if (rec >= kWall) hv = funkey(mx[b]);
            }
            if (peak_lab) {
                const int rec = max(~key, peak_lev[b * cap + ~peak_lab[pi]]);
                pv = -funkey(rec);
                if (rec >= kWall) pv = funkey(mn[b]);
            }
        } else {
            val = static_cast<const float *>(pad)[pi];
            if (hole_lab) hv = funkey(hole_lab[pi]);
            if (peak_lab) pv = detect == 2 ? -funkey(peak_lab[pi]) : funkey(peak_lab[pi]);
        }
        float out = val;
        if (s0 == 0.0f && s1 == 0.0f) {
            if (detect != 1 && th0 < fabsf(__fsub_rn(val, hv))) out = hv;
            if (detect != 0 && th1 < fabsf(__fsub_rn(pv, val))) out = pv;
        } else {
            auto sw = [](float x, float a, float bb, float level, float width) {
                const float wgt = __fdiv_rn(1.0f, __fadd_rn(1.0f, expf(__fdiv_rn(__fsub_rn(level, x), width))));
                return __fadd_rn(a, __fmul_rn(__fsub_rn(bb, a), wgt));
            };
            if (detect == 0) out = sw(__fsub_rn(hv, val), val, hv, th0, s0);
            else if (detect == 1) out = sw(__fsub_rn(val, pv), val, pv, th1, s1);
            else {
                const float dp = __fsub_rn(val, pv), dh = __fsub_rn(hv, val);
                out = fabsf(dh) < fabsf(dp) ? sw(dp, val, pv, th0, s0) : sw(dh, val, hv, th1, s1);
            }
        }
        if (!stays) img[static_cast<size_t>(b) * per + idx] = out;
    }
}

} // namespace msc
} // namespace mr

using namespace mr;
using namespace mr::msc;

extern "C" {

mr_status mr_morphspotclean(float *proj_d, size_t nu, size_t nv, size_t nproj, int detect, int conn8,
                            const float *th_h, const float *sigma_h, int edge, int clamp, float minlevel,
                            float maxlevel, int removeinfnan, void *stream)
{
    MR_TRACE();
    if (!proj_d || !th_h || !sigma_h) return fail(MR_ERR_ARGUMENT, "mr_morphspotclean: null pointer");
    if (detect < 0 || detect > 2) return fail(MR_ERR_ARGUMENT, "Unkown detection method selected");
    if (nv < 5) return fail(MR_ERR_ARGUMENT, "mr_morphspotclean: images need at least 5 rows (the edge padding mirrors 5 rows)");
    if (edge < 1 || edge > kMaxEdge) return fail(MR_ERR_ARGUMENT, "mr_morphspotclean: edge smoothing length must be 1..%d", kMaxEdge);
    if (nu == 0 || nproj == 0) return MR_OK;
    const int w = static_cast<int>(nu), h = static_cast<int>(nv);
    const int pw = w + 2 * kMargin, ph = h + 2 * kMargin;
    if (pw > 128 * 33) return fail(MR_ERR_UNSUPPORTED, "mr_morphspotclean: rows longer than %d pixels", 128 * 33 - 2 * kMargin);
    const size_t n = static_cast<size_t>(pw) * ph;
    cudaStream_t s = as_stream(stream);
    // images per batch: the padded image and, per reconstruction, a result or the labels with the basins'
    // component, level, hook and two edges, or two worklists; up to a quarter of the free device memory.
    // An image whose basins (26 to 40 bytes a pixel with both modes) do not fit that takes the sweeps (13).
    const int jobs = detect == 2 ? 2 : 1;
    const size_t band = detect == 1 ? band_size(pw, ph) : 0;
    const size_t most = std::min<size_t>(nproj, size_t(65535) / jobs);
    bool flood = few_units(nproj * jobs, pw, conn8) && n < size_t(1) << 30;
    size_t cap, per_img, budget;
    for (;;) {
        cap = flood ? most_basins(pw, ph, conn8) : static_cast<size_t>(complete_cap(n));
        const size_t per_unit = n * 4 + (flood ? cap * (3 * 4 + 2 * 8) + strips_of(pw, ph) + (kMostRounds + 2) * 4 : 2 * cap * 4 + 4);
        per_img = (n + band + 3) * 4 + jobs * per_unit + 64;
        budget = scratch_budget(most * per_img);
        if (!flood || per_img <= budget) break;
        flood = false;
    }
    const size_t batch = std::max<size_t>(1, std::min<size_t>(most, budget / per_img));
    char *scratch = nullptr;
    MR_TRY(device_alloc(&scratch, batch * per_img, s, "mr_morphspotclean: scratch"));
    const size_t units = batch * jobs;
    Flood F{};
    F.best0 = reinterpret_cast<u64 *>(scratch); // (flood) 8-byte words first
    F.best1 = F.best0 + (flood ? units * cap : 0);
    float *P = reinterpret_cast<float *>(F.best1 + (flood ? units * cap : 0));
    int *lab = reinterpret_cast<int *>(P + batch * n); // labels, or results as keys
    F.comp = lab + units * n;
    F.lev = F.comp + (flood ? units * cap : 0);
    F.par = F.lev + (flood ? units * cap : 0);
    float *bands = reinterpret_cast<float *>(F.par + (flood ? units * cap : 0)), *fmax = bands + batch * band;
    int *mn = reinterpret_cast<int *>(fmax + batch), *mx = mn + batch; // keys
    F.nbasin = mx + batch;
    F.active = F.nbasin + units;
    F.uniform = reinterpret_cast<unsigned char *>(F.active + (kMostRounds + 1) * units);
    int *counts = mx + batch, *lists = counts + units; // the sweeps' list lengths and worklists
    F.pad = reinterpret_cast<const int *>(P);
    F.band = detect == 1 ? bands : nullptr;
    F.pw = pw;
    F.ph = ph;
    F.cap = static_cast<int>(cap);
    // peaks are holes of the negated image
    F.flip0 = detect == 1 ? -1 : 0;
    F.flip1 = -1;
    mr_status st = MR_OK;
    for (size_t b0 = 0; b0 < nproj && st == MR_OK; b0 += batch) {
        const int nb = static_cast<int>(std::min(batch, nproj - b0));
        float *img = proj_d + b0 * nu * nv;
        const unsigned gx = std::min<unsigned>(div_up(n, 256), 128u);
        F.nimg = nb;
        F.units = nb * jobs;
        F.lab0 = lab;
        F.lab1 = lab + nb * n;
        int *peak_lab = jobs == 2 ? F.lab1 : F.lab0;
        float *H = reinterpret_cast<float *>(F.lab0), *K = reinterpret_cast<float *>(peak_lab);
        if (removeinfnan) k_finite_max<<<nb, 256, 0, s>>>(img, nu * nv, fmax);
        k_range_init<<<div_up(nb, 256), 256, 0, s>>>(nb, mn, mx);
        k_pad<<<dim3(gx, nb), 256, 0, s>>>(img, w, h, removeinfnan ? fmax : nullptr, clamp, minlevel, maxlevel, P, mn, mx);
        k_edge_median<<<2 * nb, 32, pw * sizeof(float), s>>>(P, pw, ph, edge);
        if (detect == 1) { // the forward scan's border band; the rest of the marker is the minimum
            const size_t smem = (8 * static_cast<size_t>(ph) + 2 * static_cast<size_t>(pw)) * sizeof(float);
            const bool fits = smem <= kBandSmem;
            if (!fits || !flood) k_marker<<<dim3(gx, nb), 256, 0, s>>>(P, pw, ph, mn, 1.0f, K);
            if (fits) {
                const cudaError_t e = cudaFuncSetAttribute(k_peaks_band_smem, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                           static_cast<int>(kBandSmem));
                if (e != cudaSuccess) {
                    st = fail(MR_ERR_CUDA, "k_peaks_band_smem: %s", cudaGetErrorString(e));
                    break;
                }
                k_peaks_band_smem<<<nb, 128, smem, s>>>(P, pw, ph, conn8, mn, bands);
                if (!flood) k_band_into<<<nb, 256, 0, s>>>(bands, pw, ph, K);
            } else { // columns beyond a CTA's shared memory: replayed on the whole marker image
                k_peaks_forward_band<<<div_up(nb, 32), 32, 0, s>>>(P, pw, ph, nb, conn8, mn, K);
                if (flood) k_band_of<<<nb, 256, 0, s>>>(K, pw, ph, bands);
            }
        }
        if (flood) {
            k_to_keys<<<std::min<unsigned>(div_up(nb * n, 1024), 148 * 16), 256, 0, s>>>(P, nb * n);
            st = conn8 ? launch_flood<true>(F, s) : launch_flood<false>(F, s);
        } else if (detect == 1) {
            const RecJobs rec{{1.0f, 1.0f}, {K, K}, nb, {nullptr, nullptr}};
            st = launch_reconstruct<true>(rec, 1, P, pw, ph, conn8, lists, counts, s);
        } else {
            // FillHole: erosion from a max marker (formed by the first sweep); of the negated image too
            // for 'both' (marker max(-P) = -min(P)), in the same launches
            const RecJobs rec{{1.0f, -1.0f}, {H, K}, nb, {mx, mn}};
            st = launch_reconstruct<false>(rec, jobs, P, pw, ph, conn8, lists, counts, s);
        }
        if (st != MR_OK) break;
        const int *hole_lab = detect != 1 ? F.lab0 : nullptr, *peaks = detect != 0 ? peak_lab : nullptr;
        if (flood) // (a block per row of few images: with 128 blocks one of 2000 x 2000 took 77 us, 20 now)
            k_replace<true><<<dim3(std::min<unsigned>(h, std::max(gx, 148u * 8 / nb)), nb), 256, 0, s>>>(
                P, hole_lab, F.lev, peaks, F.lev + (jobs - 1) * nb * cap, cap, mn, mx, w, h, detect, th_h[0], th_h[1],
                sigma_h[0], sigma_h[1], img);
        else
            k_replace<false><<<dim3(gx, nb), 256, 0, s>>>(P, hole_lab, nullptr, peaks, nullptr, 0, mn, mx, w, h, detect,
                                                          th_h[0], th_h[1], sigma_h[0], sigma_h[1], img);
        st = check_launch("k_replace");
    }
    cudaFreeAsync(scratch, s);
    return st;
}

} // extern "C"
