// Differentiation form matched to the parallel-beam backprojector: a forward projector that is
// the exact transpose of MultiProjectionBPparallel's linear-interpolation backprojection
// (MultiProjBPparallel.cpp:39-170), and that backprojection with a per-slice detector centre.
//
// Backprojection (the adjoint), voxel (x, y, z) with 1-based x, y inside the circle mask, every
// projection i (no buffer-drop rule, weight 1):
//     u = (startu[i][z] + cos_i * y) - sin_i * x,   n = (int)u in [0, nu - 2],
//     wb = |u - n|, wa = 1 - wb,   vol[y-1][x-1][z] += P_i[z][n] * wa + P_i[z][n+1] * wb
// with the reference's float operations in its order; startu[i][z] = (nu/2)(sin_i - cos_i) + c_z
// and c_z = centre + tan(tilt) (z - pivot) (the detector centre of slice z). With tilt 0 this is
// the production backprojector bit for bit (mr_bp_parallel with no weights).
//
// Forward projection (the exact transpose): detector bin m of slice z and projection i collects
// wa * vol from every voxel whose n is m and wb * vol from every voxel whose n is m - 1, with the
// same u, n, wa and wb evaluated by the same expressions, so <A x, p> = <x, A^T p> holds to float
// summation. Two kernels, both driven by the voxels: k_mbp_forward_smem holds a projection's bins for 32
// slices in shared memory, k_mbp_forward_strip (wider detectors) gives each warp a few bins of its own.
// The derivative d proj / d c_z (-vol for the wa term, +vol for the wb term: d wa / du = -1,
// d wb / du = +1, du / dc_z = 1) comes out of the same walks.
#include "mr_common.cuh"
#include "mr_tma.cuh"

#include <cooperative_groups.h>
#include <cuda.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <type_traits>
#include <vector>

namespace mr {

static const float kFPi = 3.1415926535897932384626f;

MR_BOUNDS_TAKE(bounds_take_matched)

// The adjoint with its projection rows staged in shared memory by TMA, as the production backprojector
// (mr_bp_tma.cu): a CTA owns 32 (x) x 8 or 4 (y) voxel columns x 32 slices, a thread one column's 32 slices in
// registers over all projections. Each slice has its own position (the detector centre moves with it):
// u is affine in x, y and, through the slice centre, z, so its floor is extreme at the tile's corners;
// a projection's box of 48 columns x 32 slices starts at most four columns before the smallest (the TMA
// unit's 16-byte steps and a column of margin for the float rounding) and must hold two past the largest,
// else that projection is read from global memory for this tile. Every voxel adds its projections in
// order with the same float operations as the plain kernel: the result is the same bit for bit.
//
// Bound by instruction issue: position, floor and weights of each slice, two loads, two products and
// sums. Slices go in pairs through the paired FP32 pipe (products as fmas with a -0 addend the compiler
// cannot see, so that they are not contracted with their sum), the floor from the bits of u + 1.5 * 2^23
// added rounding down, and boxes come by one instruction of one thread instead of 48 cp.async per thread
// and batch: 256^2 x 64 slices from 180 projections 1061 -> 605 us, 564 in shorter tiles (launch_adjoint).
constexpr int kAdjTX = 32, kAdjTZ = 32, kAdjBW = 48;
constexpr int kAdjBox = kAdjBW * kAdjTZ;     // floats
constexpr int kAdjGeo = kAdjTZ + 4;          // slice start positions, sin, cos, pad
constexpr float kAdjMagic = 12582912.0f;     // 1.5 * 2^23
constexpr int kAdjMagicBits = 0x4B400000;
// how a tile reads a projection: footprint beyond the box, nothing, staged, staged and on the detector
enum { kAdjUnfit, kAdjNothing, kAdjStaged, kAdjClean };

__host__ __device__ constexpr size_t adj_smem_bytes(int nb)
{
    return sizeof(float) * (2ull * nb * kAdjBox + 3ull * nb * kAdjGeo) + sizeof(int2) * 2 * nb + 2 * sizeof(uint64_t);
}

struct AdjParams {
    const float *proj; // rows of `pitch` floats
    const float2 *sc;
    const float *startu;
    const uint32_t *mask;
    float *vol;
    int nproj, n, nz, pitch, accumulate, wait_limit;
    int staged; // 0: rows that TMA cannot address, every sample by guarded global loads
    float neg_zero;
};

__device__ int g_mbp_error = 0;

int mbp_device_status_take()
{
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_mbp_error, sizeof(int)) != cudaSuccess) return -1;
    if (cudaMemcpyToSymbol(g_mbp_error, &zero, sizeof(int)) != cudaSuccess) return -1;
    return v;
}

// Tiles of 32 x TY columns, batches of NB projections.
template <int TY, int NB, int CTAS>
__global__ void __launch_bounds__(kAdjTX * TY, CTAS) k_mbp_adjoint_staged(const __grid_constant__ CUtensorMap tmap,
                                                                              const AdjParams P)
{
    extern __shared__ __align__(1024) float adj_smem[];
    float *box = adj_smem;                                          // [2][NB][TZ][BW]
    float *geo = box + 2 * NB * kAdjBox;                        // [3][NB][kAdjGeo]
    int2 *meta = reinterpret_cast<int2 *>(geo + 3 * NB * kAdjGeo); // [2][NB]: first staged column, mode
    uint64_t *bars = reinterpret_cast<uint64_t *>(meta + 2 * NB);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n = P.n, nz = P.nz;
    const int x0 = blockIdx.x * kAdjTX, y0 = blockIdx.y * TY, z0 = blockIdx.z * kAdjTZ;
    const int x1 = x0 + lane + 1, y1 = y0 + warp + 1; // 1-based voxel
    const bool valid = x1 <= n && y1 <= n;
    const bool inside = valid && static_cast<uint32_t>(x1) > P.mask[2 * (y1 - 1)] &&
                        static_cast<uint32_t>(x1) <= P.mask[2 * (y1 - 1) + 1];
    const int zmax = min(kAdjTZ, nz - z0);
    float *col = P.vol + (static_cast<size_t>(valid ? y1 - 1 : 0) * n + (valid ? x1 - 1 : 0)) * nz + z0;
    float2 acc[kAdjTZ / 2];
#pragma unroll
    for (int c = 0; c < kAdjTZ; ++c) {
        const float v = (P.accumulate && inside && c < zmax) ? col[c] : 0.0f;
        if (c & 1) acc[c >> 1].y = v; else acc[c >> 1].x = v;
    }
    const int nbatch = (P.nproj + NB - 1) / NB;
    const int xa = x0 + 1, xb = min(x0 + kAdjTX, n), ya = y0 + 1, yb = min(y0 + TY, n);
    const bool any = __syncthreads_or(inside);
    if (threadIdx.x == 0) {
        tma::mbar_init(&bars[0], 1);
        tma::mbar_init(&bars[1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    // geometry of batch s into buffer gb; slices past the volume repeat the last one, projections past
    // the list the first
    auto stage_geometry = [&](int s, int gb) {
        for (int e = threadIdx.x; e < NB * (kAdjTZ + 2); e += kAdjTX * TY) {
            const int b = e / (kAdjTZ + 2), c = e - b * (kAdjTZ + 2), i = s * NB + b < P.nproj ? s * NB + b : 0;
            const float *src = c < kAdjTZ ? P.startu + static_cast<size_t>(i) * nz + min(z0 + c, nz - 1)
                                          : reinterpret_cast<const float *>(P.sc + i) + (c - kAdjTZ);
            tma::copy4_zfill(geo + (gb * NB + b) * kAdjGeo + c, src, true);
        }
    };
    // batch s (geometry in buffer gb) into stage st: windows from 8 corner lanes per projection
    auto issue = [&](int s, int st, int gb) {
        if (warp != 0) return;
#pragma unroll 1
        for (int r = 0; r < NB; r += 4) {
            const int b = r + (lane >> 3), corner = lane & 7, i = s * NB + b;
            const float *g = geo + (gb * NB + b) * kAdjGeo;
            const float fx = static_cast<float>((corner & 1) ? xb : xa), fy = static_cast<float>((corner & 2) ? yb : ya);
            const float u = __fsub_rn(__fadd_rn(g[(corner & 4) ? zmax - 1 : 0], __fmul_rn(g[kAdjTZ + 1], fy)),
                                      __fmul_rn(g[kAdjTZ], fx));
            bool ok = fabsf(u) < 1.0e6f;
            int lo = ok ? __float2int_rd(u) : 0, hi = lo;
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) {
                lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
                hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
                ok = __shfl_xor_sync(0xffffffffu, static_cast<int>(ok), o) && ok;
            }
            int mode = kAdjNothing;
            const int w0 = (lo - 1) & ~3;
            if (i < P.nproj) {
                if (!ok || !P.staged || hi + 2 >= w0 + kAdjBW) mode = kAdjUnfit;
                else if (hi >= -1 && lo <= n) mode = lo >= 1 && hi <= n - 3 ? kAdjClean : kAdjStaged;
            }
            const bool head = corner == 0, load = head && mode >= kAdjStaged;
            const uint32_t bytes = __popc(__ballot_sync(0xffffffffu, load)) * kAdjBox * sizeof(float);
            if (lane == 0) { // the phase completes on the last round's arrival
                if (r + 4 < NB) tma::mbar_add_tx(&bars[st], bytes);
                else tma::mbar_expect_tx(&bars[st], bytes);
            }
            __syncwarp();
            if (head) meta[st * NB + b] = make_int2(w0, mode);
            if (load) {
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                tma::load_3d(box + (st * NB + b) * kAdjBox, &tmap, w0, z0, i, &bars[st]);
            }
        }
    };
    uint32_t phase0 = 0, phase1 = 0;
    bool failed = false, stopped = false; // a wait of this warp expired; of any warp
    int s = 0;
    if (any) {
        for (int k = 0; k < 3 && k < nbatch; ++k) stage_geometry(k, k);
        tma::copy_wait_all();
        __syncthreads();
        for (int k = 0; k < 2 && k < nbatch; ++k) issue(k, k, k);
        __syncthreads();
    }
    // threads past the volume follow its last column or row: their positions stay inside the corners'
    const float fx = static_cast<float>(min(x1, n)), fy = static_cast<float>(min(y1, n));
    const float2 nz2 = make_float2(P.neg_zero, P.neg_zero), one = make_float2(1.0f, 1.0f), minus = make_float2(-1.0f, -1.0f);
    const float2 magic = make_float2(kAdjMagic, kAdjMagic), unmagic = make_float2(-kAdjMagic, -kAdjMagic);
    for (int gb = 0; any && s < nbatch; ++s, gb = gb == 2 ? 0 : gb + 1) {
        const int st = s & 1;
        const bool got = __all_sync(0xffffffffu, tma::mbar_wait(&bars[st], st ? phase1 : phase0, P.wait_limit));
        if (got) {
            if (st) phase1 ^= 1; else phase0 ^= 1;
        } else {
            failed = true;
            if (lane == 0) atomicExch(&g_mbp_error, 1);
        }
        // WHOLE: all 32 slices exist; else the loops end after the last group of four that holds some. (Their
        // tests would cost whole tiles 4 %: 256^2 x 64 slices from 180 projections 567 -> 592 us. Without them
        // 256^2 x 4 slices from 60 took 102 us, as much as 32, with them 41.)
        auto project = [&](auto whole) {
            constexpr bool WHOLE = decltype(whole)::value;
#pragma unroll 1
            for (int b = 0; b < NB && s * NB + b < P.nproj; ++b) {
                const int2 m = meta[st * NB + b];
                if (m.y == kAdjNothing) continue;
                const float *g = geo + (gb * NB + b) * kAdjGeo;
                const float cy = __fmul_rn(g[kAdjTZ + 1], fy), sx = __fmul_rn(g[kAdjTZ], fx);
                const float *bx = box + (st * NB + b) * kAdjBox;
                if (m.y == kAdjClean) {
                    const float2 cy2 = make_float2(cy, cy), sx2 = make_float2(-sx, -sx);
                    const int base = -kAdjMagicBits - m.x;
#pragma unroll
                    for (int q = 0; q < kAdjTZ / 4; ++q) {
                        if (!WHOLE && 4 * q >= zmax) break; // uniform
                        const float4 su = reinterpret_cast<const float4 *>(g)[q];
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const int c = 4 * q + 2 * h;
                            const float2 u = __fadd2_rn(__fadd2_rn(h ? make_float2(su.z, su.w) : make_float2(su.x, su.y), cy2), sx2);
                            const float2 k = __fadd2_rd(u, magic);
                            const float2 wb = __ffma2_rn(__fadd2_rn(k, unmagic), minus, u); // u - floor(u), u >= 0
                            const float2 wa = __ffma2_rn(wb, minus, one);
                            const int m0 = __float_as_int(k.x) + base, m1 = __float_as_int(k.y) + base;
                            if (!MR_IN_BOUNDS(m0 + 1, kAdjBW, kSiteMbpAdjoint) || !MR_IN_BOUNDS(m1 + 1, kAdjBW, kSiteMbpAdjoint))
                                continue;
                            const float *r0 = bx + c * kAdjBW + m0, *r1 = bx + (c + 1) * kAdjBW + m1;
                            const float2 t = __fadd2_rn(__ffma2_rn(make_float2(r0[0], r1[0]), wa, nz2),
                                                        __ffma2_rn(make_float2(r0[1], r1[1]), wb, nz2));
                            acc[c / 2] = __fadd2_rn(acc[c / 2], t);
                        }
                    }
                    continue;
                }
                // edges of the detector, or a footprint beyond the box: slice by slice
                const float *img = P.proj + (static_cast<size_t>(s * NB + b) * nz + z0) * P.pitch;
#pragma unroll
                for (int c = 0; c < kAdjTZ; ++c) {
                    if (!WHOLE && c % 4 == 0 && c >= zmax) break; // uniform
                    const float u = __fsub_rn(__fadd_rn(g[c], cy), sx);
                    const int k = __float2int_rz(u);
                    if (!WHOLE && c >= zmax) continue;
                    if (k < 0 || k > n - 2) continue;
                    const float wb = fabsf(__fsub_rn(u, static_cast<float>(k))), wa = __fsub_rn(1.0f, wb);
                    float pa, pb;
                    if (m.y == kAdjStaged) {
                        if (!MR_IN_BOUNDS(k - m.x + 1, kAdjBW, kSiteMbpAdjoint)) continue;
                        pa = bx[c * kAdjBW + k - m.x];
                        pb = bx[c * kAdjBW + k - m.x + 1];
                    } else {
                        pa = __ldg(img + static_cast<size_t>(c) * P.pitch + k);
                        pb = __ldg(img + static_cast<size_t>(c) * P.pitch + k + 1);
                    }
                    float &a = (c & 1) ? acc[c >> 1].y : acc[c >> 1].x;
                    a = __fadd_rn(a, __fadd_rn(__fmul_rn(pa, wa), __fmul_rn(pb, wb)));
                }
            }
        };
        if (got && inside) {
            if (zmax == kAdjTZ) project(std::true_type{});
            else project(std::false_type{});
        }
        // batch s + 2's geometry is published; stage st and geometry buffer gb are free
        tma::copy_wait_all();
        stopped = __syncthreads_or(failed);
        if (stopped) break;
        if (s + 2 < nbatch) issue(s + 2, st, gb == 0 ? 2 : gb - 1);
        if (s + 3 < nbatch) stage_geometry(s + 3, gb);
    }
    if (failed) {
        // copies still in flight: batch s (its wait expired) and s + 1 when it was issued
        const int st = s & 1;
        tma::mbar_wait(&bars[st], st ? phase1 : phase0);
        if (s + 1 < nbatch) tma::mbar_wait(&bars[st ^ 1], st ? phase0 : phase1);
    }
    if (valid && (inside || !P.accumulate)) {
        // sums that a stopped tile has not finished pass for values in a gradient that nobody checks: NaN
        const bool lost = stopped && inside;
#pragma unroll
        for (int c = 0; c < kAdjTZ; ++c)
            if (c < zmax) col[c] = lost ? __int_as_float(0x7FC00000) : (c & 1) ? acc[c >> 1].y : acc[c >> 1].x;
    }
}

// Projection rows copied to `pitch` floats, zeros past the n bins (what the TMA unit needs: a pitch and
// base of 16 bytes, a box no wider than the row).
__global__ void __launch_bounds__(256) k_pad_rows(const float *__restrict__ src, size_t rows, int n, int pitch,
                                                  float *__restrict__ dst)
{
    const size_t total = rows * pitch;
    for (size_t e = static_cast<size_t>(blockIdx.x) * 256 + threadIdx.x; e < total; e += static_cast<size_t>(gridDim.x) * 256) {
        const size_t r = e / pitch;
        const int c = static_cast<int>(e - r * pitch);
        dst[e] = c < n ? src[r * n + c] : 0.0f;
    }
}

static mr_status launch_adjoint(AdjParams P, int width, cudaStream_t s)
{
    CUtensorMap map = {};
    if (P.staged) {
        PFN_cuTensorMapEncodeTiled enc = tma::encode_fn();
        if (!enc) return fail(MR_ERR_CUDA, "cuTensorMapEncodeTiled unavailable");
        cuuint64_t dims[3] = {static_cast<cuuint64_t>(width), static_cast<cuuint64_t>(P.nz), static_cast<cuuint64_t>(P.nproj)};
        cuuint64_t strides[2] = {static_cast<cuuint64_t>(P.pitch) * 4, static_cast<cuuint64_t>(P.pitch) * P.nz * 4};
        cuuint32_t box[3] = {kAdjBW, kAdjTZ, 1}, estr[3] = {1, 1, 1};
        const CUresult cr = enc(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float *>(P.proj), dims, strides, box, estr,
                                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (cr != CUDA_SUCCESS) return fail(MR_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", static_cast<int>(cr));
    }
    // 32 x 8 columns, two CTAs per SM, while these fill the last wave; else 32 x 4, whose shorter CTAs even it
    // out for up to 3 % more work: 256^2 x 64 slices from 180 projections (512 CTAs on 296 places) 605 -> 561
    // us, 64^2 x 8 from 60 79 -> 73, but 192^2 x 64 from 360 (288 CTAs) 795 -> 817
    const size_t across = div_up(static_cast<size_t>(P.n), kAdjTX), deep = div_up(static_cast<size_t>(P.nz), kAdjTZ);
    const size_t tiles = across * div_up(static_cast<size_t>(P.n), 8) * deep, places = 2 * 148;
    auto launch = [&](auto kernel, int ty, int nb) -> mr_status {
        MR_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(adj_smem_bytes(nb))));
        const dim3 grid(static_cast<unsigned>(across), div_up(static_cast<size_t>(P.n), ty), static_cast<unsigned>(deep));
        kernel<<<grid, kAdjTX * ty, adj_smem_bytes(nb), s>>>(map, P);
        return check_launch("k_mbp_adjoint_staged");
    };
    if (20 * tiles < 19 * places * div_up(tiles, places)) return launch(k_mbp_adjoint_staged<4, 4, 4>, 4, 4);
    return launch(k_mbp_adjoint_staged<8, 8, 2>, 8, 8);
}

// Forward projection. Both kernels walk lines of voxels along the axis on which u changes least (x when
// |sin| <= |cos|, else y; |du| <= 1/sqrt(2) per step, so a lane's bin moves by at most one between steps), one
// slice per lane, with the adjoint's u, n, wa and wb. A lane keeps the sums of its current pair of bins
// (n, n + 1) in registers and hands a bin on (Put) when its walk leaves it. On a line whose positions all lie on
// the detector the floor comes from the bits of u + 1.5 * 2^23 added rounding down, without conversions.
constexpr int kFwdPad = 33; // words between bins: 32 lanes' slices hit 32 banks, the write-out's bins do too
constexpr int kFwdU = 4;    // voxels loaded ahead

// Sums of a walk whose u grows (UP) or falls: bins cur and cur + 1 (as kAdjMagic bits, 0: none yet), the
// values a0, a1, and for the derivative the sum s of v over the current run (-v for the lower bin, +v for
// the upper) with what the run before left in the bin that the walk leaves next (carry).
template <bool DERIV, bool UP, class Put>
struct BinRun {
    int cur = 0;
    float a0 = 0.0f, a1 = 0.0f, s = 0.0f, carry = 0.0f;
    Put put;
    __device__ __forceinline__ explicit BinRun(const Put &p) : put(p) {}
    __device__ __forceinline__ void done()
    {
        if (cur == 0) return;
        put(cur, a0, UP ? carry - s : -s);
        put(cur + 1, a1, UP ? s : carry + s);
        cur = 0;
        a0 = a1 = s = carry = 0.0f;
    }
    // one voxel of value v: bin m (bits), weights 1 - wb and wb
    __device__ __forceinline__ void add(int m, float wb, float v)
    {
        if (m != cur) {
            if (m == cur + (UP ? 1 : -1)) {
                put(UP ? cur : cur + 1, UP ? a0 : a1, UP ? carry - s : carry + s);
                if (UP) a0 = a1, a1 = 0.0f;
                else a1 = a0, a0 = 0.0f;
                carry = UP ? s : -s;
                s = 0.0f;
            } else done();
            cur = m;
        }
        a0 = fmaf(v, __fsub_rn(1.0f, wb), a0);
        a1 = fmaf(v, wb, a1);
        if (DERIV) s = __fadd_rn(s, v);
    }
};

// Wide detectors: a warp owns kStripBins consecutive bins of a projection for 32 slices and collects them
// alone, so nothing is added atomically and a result does not depend on timing. It walks, on each line, the
// voxels that can reach one of its bins: the interval of the affine u for its 32 slices, widened by a bound
// of u's float evaluation; each voxel's contribution is decided by its own n. Bins beyond the warp's own are
// dropped when the walk leaves them (their own warp has the voxel too).
//
// Bound by instruction issue (80 %). With the derivative, 512^2 x 20 slices x 120 projections 2010 -> 1411 us
// (by all of a projection's bins in shared memory before), 1024^2 x 32 x 60 11520 -> 3010 (by one warp per bin
// before). 4 bins per warp: 1744 and 3720, the ends of a strip being visited twice; 16: 1480 and 3511.
constexpr int kStripBins = 8;
constexpr int kStripWarps = 4; // projections per CTA (neighbours walk almost the same voxels)

struct FwdParams {
    const float *vol;
    const float2 *sc;
    const float *startu;
    int nproj, n, nz;
    const uint32_t *mask;
    float *proj, *dproj;
};

// adds to the lane's column in shared memory, for the warp's own bins; the derivative's column follows
template <bool DERIV>
struct StripPut {
    float *bins;
    int base; // bits of the first bin
    __device__ __forceinline__ void operator()(int bin, float v, float d) const
    {
        const unsigned k = static_cast<unsigned>(bin - base);
        if (k >= kStripBins) return;
        bins[k * kFwdPad] = __fadd_rn(bins[k * kFwdPad], v);
        if (DERIV) bins[(k + kStripBins) * kFwdPad] = __fadd_rn(bins[(k + kStripBins) * kFwdPad], d);
    }
};

// The integers from lo to hi within [first, last] that t0 .. t1 (in either order) spans; a NaN end is open.
__device__ __forceinline__ void fwd_span(float t0, float t1, int first, int last, int &lo, int &hi)
{
    const float a = fminf(t0, t1), b = fmaxf(t0, t1);
    lo = static_cast<int>(fminf(fmaxf(floorf(a), static_cast<float>(first)), static_cast<float>(last) + 1.0f));
    hi = static_cast<int>(fmaxf(fminf(ceilf(b), static_cast<float>(last)), static_cast<float>(first) - 1.0f));
}

// ROWS: lines are rows y, walked along x; else columns x, walked along y.
template <bool DERIV, bool ROWS, bool UP>
__device__ __forceinline__ void strip_walk(const FwdParams &P, float2 s, float suz, int z, int first, float *bins)
{
    const int lane = threadIdx.x & 31;
    BinRun<DERIV, UP, StripPut<DERIV>> run({bins, first + kAdjMagicBits});
    // u = su + h line + g f, with the warp's range of su
    const float g = ROWS ? -s.x : s.y, h = ROWS ? s.y : -s.x, fn = static_cast<float>(P.n);
    float sul = suz, suh = suz;
    for (int o = 16; o > 0; o >>= 1) {
        sul = fminf(sul, __shfl_xor_sync(0xffffffffu, sul, o));
        suh = fmaxf(suh, __shfl_xor_sync(0xffffffffu, suh, o));
    }
    if (__any_sync(0xffffffffu, !(fabsf(suz) <= FLT_MAX))) sul = -INFINITY, suh = INFINITY;
    // u (and the bounds below) are a few roundings of terms of at most 2 n + |su|
    const float eps = (fn + fmaxf(fabsf(sul), fabsf(suh))) * 0x1p-18f;
    const float u0 = static_cast<float>(first) - 1.0f - eps - suh, u1 = static_cast<float>(first + kStripBins) + eps - sul;
    const float inv = 1.0f / g;
    int l0, l1;
    {
        const float ih = 1.0f / h;
        fwd_span((u0 - fmaxf(g, g * fn)) * ih, (u1 - fminf(g, g * fn)) * ih, 1, P.n, l0, l1);
    }
    const uint32_t stride = ROWS ? static_cast<uint32_t>(P.nz) : static_cast<uint32_t>(P.n) * static_cast<uint32_t>(P.nz);
    for (int l = l0; l <= l1; ++l) {
        const float fl = static_cast<float>(l), at = h * fl;
        int lo = 0, hi = 0; // 1-based
        if (ROWS) {
            const uint32_t ma = P.mask[2 * (l - 1)], mb = P.mask[2 * (l - 1) + 1];
            fwd_span((u0 - at) * inv, (u1 - at) * inv, static_cast<int>(min(ma, static_cast<uint32_t>(P.n))) + 1,
                     static_cast<int>(min(mb, static_cast<uint32_t>(P.n))), lo, hi);
        } else
            fwd_span((u0 - at) * inv, (u1 - at) * inv, 1, P.n, lo, hi);
        const float fixed = ROWS ? __fadd_rn(suz, __fmul_rn(s.y, fl)) : __fmul_rn(s.x, fl);
        auto position = [&](float f) {
            return ROWS ? __fsub_rn(fixed, __fmul_rn(s.x, f)) : __fsub_rn(__fadd_rn(suz, __fmul_rn(s.y, f)), fixed);
        };
        for (int f = lo; f <= hi; f += 32) {
            // the voxels of the mask among the next 32
            int cnt = min(32, hi - f + 1), skip = 0;
            uint32_t word = 0xffffffffu >> (32 - cnt);
            if (!ROWS) {
                bool in = lane < cnt;
                if (in) {
                    const uint32_t ma = P.mask[2 * (f + lane - 1)], mb = P.mask[2 * (f + lane - 1) + 1];
                    in = static_cast<uint32_t>(l) > ma && static_cast<uint32_t>(l) <= mb;
                }
                word = __ballot_sync(0xffffffffu, in);
                if (word == 0) continue;
                skip = __ffs(word) - 1;
                word >>= skip;
                cnt = 32 - __clz(word);
            }
            const int f0 = f + skip;
            float ff = static_cast<float>(f0);
            const float *p = P.vol + (ROWS ? (static_cast<size_t>(l - 1) * P.n + (f0 - 1)) * P.nz
                                           : (static_cast<size_t>(f0 - 1) * P.n + (l - 1)) * P.nz) + z;
            // (position is monotone: the ends bound it)
            const float ua = position(ff), ub = position(static_cast<float>(f0 + cnt - 1));
            const bool clean = __all_sync(0xffffffffu, fminf(ua, ub) >= 0.0f && fmaxf(ua, ub) < fn - 1.0f);
            for (int q = 0; q < cnt; q += kFwdU, word >>= kFwdU - 1, word >>= 1) {
                constexpr uint32_t ALL = (1u << kFwdU) - 1;
                float v[kFwdU];
                if (clean && (word & ALL) == ALL) {
#pragma unroll
                    for (int j = 0; j < kFwdU; ++j) v[j] = __ldg(p + static_cast<size_t>(stride) * j);
#pragma unroll
                    for (int j = 0; j < kFwdU; ++j) {
                        const float u = position(ff + static_cast<float>(j));
                        const float k = __fadd_rd(u, kAdjMagic);
                        run.add(__float_as_int(k), __fsub_rn(u, __fsub_rn(k, kAdjMagic)), v[j]);
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < kFwdU; ++j) v[j] = (word >> j & 1) ? __ldg(p + static_cast<size_t>(stride) * j) : 0.0f;
#pragma unroll 1
                    for (int j = 0; j < kFwdU; ++j) {
                        if (!(word >> j & 1)) continue;
                        const float u = position(ff + static_cast<float>(j));
                        const int m = __float2int_rz(u);
                        float vj = v[0];
#pragma unroll
                        for (int i = 1; i < kFwdU; ++i) vj = j == i ? v[i] : vj;
                        if (m >= 0 && m <= P.n - 2) run.add(m + kAdjMagicBits, fabsf(__fsub_rn(u, static_cast<float>(m))), vj);
                    }
                }
                ff += static_cast<float>(kFwdU);
                p += static_cast<size_t>(stride) * kFwdU;
            }
        }
        run.done();
    }
}

template <bool DERIV>
__global__ void __launch_bounds__(kStripWarps * 32, 10) k_mbp_forward_strip(const __grid_constant__ FwdParams P)
{
    constexpr int WORDS = kStripBins * kFwdPad * (DERIV ? 2 : 1);
    __shared__ float sums[kStripWarps][WORDS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int i = blockIdx.x * kStripWarps + warp;
    if (i >= P.nproj) return;
    // chunks of bins from the middle outwards: those that cross most of the mask start first
    const int c = blockIdx.y, first = (static_cast<int>(gridDim.y) / 2 + (c & 1 ? -((c + 1) / 2) : c / 2)) * kStripBins;
    const int z0 = blockIdx.z * 32, z = min(z0 + lane, P.nz - 1); // (lanes beyond the last slice repeat it)
    float *mine = sums[warp];
    for (int e = lane; e < WORDS; e += 32) mine[e] = 0.0f;
    __syncwarp();
    const float2 s = P.sc[i];
    const float suz = P.startu[static_cast<size_t>(i) * P.nz + z];
    // u falls along x by sin and grows along y by cos
    if (fabsf(s.x) <= fabsf(s.y)) {
        if (s.x <= 0.0f) strip_walk<DERIV, true, true>(P, s, suz, z, first, mine + lane);
        else strip_walk<DERIV, true, false>(P, s, suz, z, first, mine + lane);
    } else if (s.y >= 0.0f) strip_walk<DERIV, false, true>(P, s, suz, z, first, mine + lane);
    else strip_walk<DERIV, false, false>(P, s, suz, z, first, mine + lane);
    __syncwarp();
    for (int e = lane; e < 32 * kStripBins; e += 32) {
        const int zz = e / kStripBins, k = e % kStripBins;
        if (z0 + zz >= P.nz || first + k >= P.n) continue;
        const size_t o = (static_cast<size_t>(i) * P.nz + z0 + zz) * P.n + first + k;
        if (!MR_IN_BOUNDS(o, static_cast<size_t>(P.nproj) * P.nz * P.n, kSiteMbpBins)) continue;
        P.proj[o] = mine[k * kFwdPad + zz];
        if (DERIV) P.dproj[o] = mine[(k + kStripBins) * kFwdPad + zz];
    }
}

// Narrow detectors: a cluster of one or two CTAs per (projection i, 32 slices) holds that projection's bins of
// its slices in shared memory; its warps share the lines of voxels and add a bin atomically when a walk leaves
// it, so most voxels cost no shared-memory access. Two CTAs' bins are summed on the way out. The order of
// the additions into a bin depends on the warps' timing: results agree with the strips' to float summation,
// not bit for bit.
//
// Bound by instruction issue. 256^2 x 64 slices, 180 projections, with the derivative: 1231 -> 965 us (two CTAs
// where they shorten the last wave: 991 with one), 192^2 x 16 x 60 307 -> 125 (one: 216), 64^2 x 8 x 60 42 -> 22.
// Clusters of four and eight find too few places for CTAs that fill an SM (192^2 x 64 x 360: 994 -> 3661 with
// eight). A CTA of 1024 threads at 64 registers has its SM alone. Narrow detectors beat the strips: 384^2 x 20 x
// 120 815 against 887 us, 64^2 x 8 x 60 22 against 86; at 512^2 1455 against 1401, and 1387 against 888 with 8
// slices and 60 projections. kFwdSmemBins lies between; where exactly they cross was not measured.
constexpr int kFwdThreads = 1024;
constexpr size_t kFwdSmemBins = 400;

__host__ __device__ inline size_t fwd_smem_bytes(int n, bool deriv)
{
    return static_cast<size_t>(n) * kFwdPad * sizeof(float) * (deriv ? 2 : 1) + static_cast<size_t>(n) * sizeof(uint2) * 2;
}

template <bool DERIV>
struct AtomicPut {
    float *bins, *dbins; // of this lane, bin 0
    __device__ __forceinline__ void operator()(int bin, float v, float d) const
    {
        atomicAdd(bins + (bin - kAdjMagicBits) * kFwdPad, v);
        if (DERIV) atomicAdd(dbins + (bin - kAdjMagicBits) * kFwdPad, d);
    }
};

// (warp: of nwarps in the cluster)
template <bool DERIV, bool UP>
__device__ __forceinline__ void forward_walk(const float *__restrict__ vol, float2 s, float suz, int n, int nz, int z, bool by_rows,
                                             int warp, int nwarps,
                                             const uint2 *rowmask, const uint2 *colspan, float *bins, float *dbins)
{
    BinRun<DERIV, UP, AtomicPut<DERIV>> run({bins, dbins});
    constexpr int U = kFwdU;
    // positions of a line: u(f) for the line coordinate f
    auto visit = [&](float u, float v, bool clean) {
        if (clean) {
            const float k = __fadd_rd(u, kAdjMagic);
            if (!MR_IN_BOUNDS(__float_as_int(k) - kAdjMagicBits + 1, n, kSiteMbpBins)) return;
            run.add(__float_as_int(k), __fsub_rn(u, __fsub_rn(k, kAdjMagic)), v);
        } else {
            const int m = __float2int_rz(u);
            if (m < 0 || m > n - 2 || !MR_IN_BOUNDS(m + 1, n, kSiteMbpBins)) return;
            run.add(m + kAdjMagicBits, fabsf(__fsub_rn(u, static_cast<float>(m))), v);
        }
    };
    auto line = [&](int from, int to, const float *p, size_t stride, auto position, auto inside) {
        // (position is monotone: its ends bound it)
        const float ua = position(static_cast<float>(from + 1)), ub = position(static_cast<float>(to));
        const bool clean = __all_sync(__activemask(), fminf(ua, ub) >= 0.0f && fmaxf(ua, ub) < static_cast<float>(n - 1));
        float f = static_cast<float>(from + 1);
        for (int q = from; q < to; q += U, p += U * stride) {
            float v[U];
            bool in[U];
#pragma unroll
            for (int j = 0; j < U; ++j) {
                in[j] = q + j < to && inside(q + j);
                v[j] = in[j] ? __ldg(p + j * stride) : 0.0f;
            }
#pragma unroll
            for (int j = 0; j < U; ++j, f = __fadd_rn(f, 1.0f))
                if (in[j]) visit(position(f), v[j], clean);
        }
    };
    if (by_rows) {
        // line y: voxels x in (first, second], u = (su + cos y) - sin x
        for (int y = warp; y < n; y += nwarps) {
            const uint2 r = rowmask[y];
            const int xa = static_cast<int>(r.x), xe = min(static_cast<int>(r.y), n);
            if (xe <= xa) continue;
            const float a = __fadd_rn(suz, __fmul_rn(s.y, static_cast<float>(y + 1)));
            line(xa, xe, vol + (static_cast<size_t>(y) * n + xa) * nz + z, nz,
                 [&](float f) { return __fsub_rn(a, __fmul_rn(s.x, f)); }, [](int) { return true; });
        }
    } else {
        // line x: voxels y in the column's span that the row masks hold (bit 31 of its end: all of them)
        for (int x = warp; x < n; x += nwarps) {
            const uint2 span = colspan[x];
            const uint32_t x1 = static_cast<uint32_t>(x) + 1;
            const int ya = static_cast<int>(span.x), ye = static_cast<int>(span.y & 0x7FFFFFFFu);
            if (ye <= ya) continue;
            const float sx = __fmul_rn(s.x, static_cast<float>(x1));
            const float *p = vol + (static_cast<size_t>(ya) * n + x) * nz + z;
            const size_t stride = static_cast<size_t>(n) * nz;
            auto position = [&](float f) { return __fsub_rn(__fadd_rn(suz, __fmul_rn(s.y, f)), sx); };
            if (span.y >> 31) line(ya, ye, p, stride, position, [](int) { return true; });
            else line(ya, ye, p, stride, position, [&](int y) { return x1 > rowmask[y].x && x1 <= rowmask[y].y; });
        }
    }
    run.done();
}

template <bool DERIV>
__global__ void __launch_bounds__(kFwdThreads, 1) k_mbp_forward_smem(const float *__restrict__ vol, const float2 *__restrict__ sc,
                                                                  const float *__restrict__ startu, int nproj, int n,
                                                                  int nz, const uint32_t *__restrict__ mask,
                                                                  float *__restrict__ proj, float *__restrict__ dproj)
{
    extern __shared__ uint2 rowmask[]; // the masks, then bins [n][kFwdPad] (+ [n][kFwdPad] for the derivative)
    float *bins = reinterpret_cast<float *>(rowmask + 2 * n), *dbins = bins + static_cast<size_t>(n) * kFwdPad;
    uint2 *colspan = rowmask + n; // per column x: the rows [lo, hi) that hold voxels of it; bit 31: all of them do
    const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    const int rank = cluster.block_rank(), ctas = cluster.num_blocks();
    const int i = blockIdx.x / ctas, z0 = blockIdx.y * 32;
    const int lane = threadIdx.x & 31;
    const int z = z0 + lane;
    const bool zok = z < nz;
    for (int e = threadIdx.x; e < n * kFwdPad * (DERIV ? 2 : 1); e += blockDim.x) bins[e] = 0.0f;
    for (int y = threadIdx.x; y < n; y += blockDim.x) rowmask[y] = make_uint2(mask[2 * y], mask[2 * y + 1]);
    const float2 s = sc[i];
    const bool by_rows = fabsf(s.x) <= fabsf(s.y);
    __syncthreads();
    if (!by_rows)
        for (int x = threadIdx.x; x < n; x += blockDim.x) {
            const uint32_t x1 = static_cast<uint32_t>(x) + 1;
            int lo = 0, hi = -1, count = 0;
            for (int y = 0; y < n; ++y)
                if (x1 > rowmask[y].x && x1 <= rowmask[y].y) {
                    if (count++ == 0) lo = y;
                    hi = y;
                }
            const uint32_t all = count == hi + 1 - lo ? 0x80000000u : 0u;
            colspan[x] = make_uint2(static_cast<uint32_t>(lo), static_cast<uint32_t>(hi + 1) | all);
        }
    __syncthreads();
    if (zok) {
        const float suz = startu[static_cast<size_t>(i) * nz + z];
        const int per = static_cast<int>(blockDim.x >> 5), warp = rank * per + static_cast<int>(threadIdx.x >> 5), nwarps = ctas * per;
        // u falls along x by sin and grows along y by cos
        if (by_rows ? s.x <= 0.0f : s.y >= 0.0f)
            forward_walk<DERIV, true>(vol, s, suz, n, nz, z, by_rows, warp, nwarps, rowmask, colspan, bins + lane, dbins + lane);
        else
            forward_walk<DERIV, false>(vol, s, suz, n, nz, z, by_rows, warp, nwarps, rowmask, colspan, bins + lane, dbins + lane);
    }
    cluster.sync();
    // write-out: consecutive threads take consecutive bins of one slice (coalesced stores), summed over the CTAs
    const int zs = min(32, nz - z0);
    for (int e = rank * blockDim.x + threadIdx.x; e < zs * n; e += ctas * blockDim.x) {
        const int zz = e / n, m = e - zz * n;
        const size_t o = (static_cast<size_t>(i) * nz + z0 + zz) * n + m;
        float a = 0.0f, d = 0.0f;
        for (int r = 0; r < ctas; ++r) {
            const float *there = cluster.map_shared_rank(bins, r);
            a = __fadd_rn(a, there[m * kFwdPad + zz]);
            if (DERIV) d = __fadd_rn(d, there[(n + m) * kFwdPad + zz]);
        }
        proj[o] = a;
        if (DERIV) dproj[o] = d;
    }
    cluster.sync(); // (the others may still read these bins)
}

} // namespace mr

using namespace mr;

extern "C" {

mr_status mr_mbp_geometry(const float *angles_h, size_t nproj, size_t n, size_t nz, float centre, float tan_tilt,
                          float pivot, int direction, float *sincos_h, float *startu_h)
{
    MR_TRACE();
    if (nproj && (!angles_h || !sincos_h || !startu_h)) return fail(MR_ERR_ARGUMENT, "mr_mbp_geometry: null pointer");
    if (n < 2) return fail(MR_ERR_ARGUMENT, "mr_mbp_geometry: n must be at least 2");
    // StdBackProjectorBase::Process 2D (StdBackProjectorBase.cpp:72-79) with the centre of slice z
    const float dirweight = 2.0f * (static_cast<float>(direction) - 0.5f);
    const size_t mcx = n / 2;
    for (size_t k = 0; k < nproj; ++k) {
        const float s = std::sin(dirweight * angles_h[k] * kFPi / 180.0f);
        const float c = std::cos(dirweight * angles_h[k] * kFPi / 180.0f);
        sincos_h[2 * k] = s;
        sincos_h[2 * k + 1] = c;
        for (size_t z = 0; z < nz; ++z) {
            const float cz = centre + tan_tilt * (static_cast<float>(z) - pivot);
            startu_h[k * nz + z] = mcx * (s - c) + cz;
        }
    }
    return MR_OK;
}

mr_status mr_mbp_adjoint(const float *proj_d, size_t n, size_t nz, const float *sincos_d, const float *startu_d,
                         size_t nproj, const uint32_t *mask_d, int accumulate, float *vol_d, void *stream)
{
    MR_TRACE();
    if (!proj_d || !sincos_d || !startu_d || !mask_d || !vol_d) return fail(MR_ERR_ARGUMENT, "mr_mbp_adjoint: null pointer");
    if (n < 2 || n > 65536 || nz == 0 || nz > 65536 || nproj > 0x7fffffff)
        return fail(MR_ERR_ARGUMENT, "mr_mbp_adjoint: unsupported size");
    AdjParams P;
    P.sc = reinterpret_cast<const float2 *>(sincos_d);
    P.startu = startu_d;
    P.mask = mask_d;
    P.vol = vol_d;
    P.n = static_cast<int>(n);
    P.nz = static_cast<int>(nz);
    P.accumulate = accumulate;
    P.wait_limit = tma::g_batch_wait_limit.load();
    P.neg_zero = -0.0f;
    P.staged = 1;
    cudaStream_t s = as_stream(stream);
    const bool direct = n % 4 == 0 && n >= kAdjBW && reinterpret_cast<uintptr_t>(proj_d) % 16 == 0;
    if (nproj == 0) { // an empty sum
        if (!accumulate) MR_CUDA_TRY(cudaMemsetAsync(vol_d, 0, n * n * nz * sizeof(float), s));
        return MR_OK;
    }
    if (direct) {
        P.proj = proj_d;
        P.pitch = P.n;
        P.nproj = static_cast<int>(nproj);
        return launch_adjoint(P, P.n, s);
    }
    // padded copies, a run of projections (64 MiB of scratch) at a time; the volume carries the sums
    const size_t pitch = std::max<size_t>(kAdjBW, (n + 3) / 4 * 4), per = nz * pitch;
    const size_t run = std::min(nproj, std::max<size_t>(8, (size_t(64) << 20) / (per * 4)));
    float *scratch = nullptr;
    if (device_alloc(&scratch, run * per * sizeof(float), s, "mr_mbp_adjoint: padded projections") != MR_OK) {
        P.proj = proj_d; // no room for copies
        P.pitch = P.n;
        P.nproj = static_cast<int>(nproj);
        P.staged = 0;
        return launch_adjoint(P, P.n, s);
    }
    mr_status st = MR_OK;
    for (size_t i = 0; i < nproj && st == MR_OK; i += run) {
        const size_t m = std::min(run, nproj - i);
        k_pad_rows<<<std::min<unsigned>(div_up(m * per, 1024), 148 * 16), 256, 0, s>>>(proj_d + i * nz * n, m * nz, P.n,
                                                                                     static_cast<int>(pitch), scratch);
        P.proj = scratch;
        P.pitch = static_cast<int>(pitch);
        P.nproj = static_cast<int>(m);
        P.sc = reinterpret_cast<const float2 *>(sincos_d) + i;
        P.startu = startu_d + i * nz;
        P.accumulate = accumulate || i > 0;
        if ((st = check_launch("k_pad_rows")) == MR_OK) st = launch_adjoint(P, P.pitch, s);
    }
    cudaFreeAsync(scratch, s);
    return st;
}

mr_status mr_mbp_forward(const float *vol_d, size_t n, size_t nz, const float *sincos_d, const float *startu_d,
                         size_t nproj, const uint32_t *mask_d, float *proj_d, float *dproj_d, void *stream)
{
    MR_TRACE();
    if (!vol_d || !sincos_d || !startu_d || !mask_d || !proj_d) return fail(MR_ERR_ARGUMENT, "mr_mbp_forward: null pointer");
    if (n < 2 || n > 65536 || nz == 0 || nz > 65536 || nproj == 0 || nproj > 65535)
        return fail(MR_ERR_ARGUMENT, "mr_mbp_forward: unsupported size");
    const float2 *sc = reinterpret_cast<const float2 *>(sincos_d);
    if (n <= kFwdSmemBins) {
        // Two CTAs per (projection, 32 slices) where that shortens the last wave. Zeroing, masks and the cluster's
        // barriers are paid once per wave, so the shorter the lines the fewer waves may be: 192^2 x 32 slices,
        // 180 projections (2 waves) 325 us with two against 351, but 96^2 113 against 101, and 128^2 with 310
        // projections (3 waves) 271 against 220. Detectors so narrow that the lines leave warps idle take half
        // as many threads from two waves on, two CTAs to an SM: 48^2 x 128 x 360 152 us against 181.
        const size_t units = nproj * div_up(nz, 32), waves = div_up(units, 148);
        const unsigned ctas = div_up(2 * units, 148) < 2 * waves && (waves == 1 || n >= 64 * waves) ? 2 : 1;
        const unsigned threads = waves > 1 && n <= 48 ? kFwdThreads / 2 : kFwdThreads;
        const size_t smem = fwd_smem_bytes(static_cast<int>(n), dproj_d != nullptr);
        auto launch = [&](auto kernel) -> mr_status {
            MR_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
            cudaLaunchAttribute attr;
            attr.id = cudaLaunchAttributeClusterDimension;
            attr.val.clusterDim = {ctas, 1, 1};
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(static_cast<unsigned>(nproj) * ctas, div_up(nz, 32));
            cfg.blockDim = dim3(threads);
            cfg.dynamicSmemBytes = smem;
            cfg.stream = as_stream(stream);
            cfg.attrs = &attr;
            cfg.numAttrs = 1;
            MR_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, vol_d, sc, startu_d, static_cast<int>(nproj), static_cast<int>(n),
                                           static_cast<int>(nz), mask_d, proj_d, dproj_d));
            return check_launch("k_mbp_forward_smem");
        };
        return dproj_d ? launch(k_mbp_forward_smem<true>) : launch(k_mbp_forward_smem<false>);
    }
    FwdParams P;
    P.vol = vol_d;
    P.sc = reinterpret_cast<const float2 *>(sincos_d);
    P.startu = startu_d;
    P.nproj = static_cast<int>(nproj);
    P.n = static_cast<int>(n);
    P.nz = static_cast<int>(nz);
    P.mask = mask_d;
    P.proj = proj_d;
    P.dproj = dproj_d;
    const dim3 grid(div_up(nproj, kStripWarps), div_up(n, kStripBins), div_up(nz, 32));
    if (dproj_d) k_mbp_forward_strip<true><<<grid, kStripWarps * 32, 0, as_stream(stream)>>>(P);
    else k_mbp_forward_strip<false><<<grid, kStripWarps * 32, 0, as_stream(stream)>>>(P);
    return check_launch("k_mbp_forward_strip");
}

} // extern "C"
