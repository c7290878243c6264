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
// summation. Two kernels: a voxel-driven one (k_mbp_forward_smem, below) while a projection's
// bins for 32 slices fit in shared memory, else a ray-driven one: a warp owns one (i, m) and 32 consecutive slices (lanes), walks the
// volume rows when |sin_i| >= |cos_i| (else the columns) and, in each, only the candidate
// voxels whose u can fall in [m - 1, m + 1): the interval of the affine u, widened by one voxel
// on each side for the float evaluation (u is exact to ~1e-4 pixel, the walk's step is at least
// 1/sqrt(2) pixel). Each candidate's contribution is decided by its own n, as in the adjoint.
// The derivative d proj / d c_z (-vol for the wa term, +vol for the wb term: d wa / du = -1,
// d wb / du = +1, du / dc_z = 1) comes out of the same walk.
#include "mr_common.cuh"
#include "mr_tma.cuh"

#include <cuda.h>

#include <algorithm>
#include <cmath>
#include <vector>

namespace mr {

static const float kFPi = 3.1415926535897932384626f;

MR_BOUNDS_TAKE(bounds_take_matched)

// The adjoint with its projection rows staged in shared memory by TMA, as the production backprojector
// (mr_bp_tma.cu): a CTA owns 32 (x) x 8 (y) voxel columns x 32 slices, a thread one column's 32 slices in
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
// and batch: 256^2 x 64 slices from 180 projections 1061 -> 602 us.
constexpr int kAdjTX = 32, kAdjTY = 8, kAdjTZ = 32, kAdjNB = 8, kAdjBW = 48;
constexpr int kAdjThreads = kAdjTX * kAdjTY, kAdjCtas = 2;
constexpr int kAdjBox = kAdjBW * kAdjTZ;     // floats
constexpr int kAdjGeo = kAdjTZ + 4;          // slice start positions, sin, cos, pad
constexpr float kAdjMagic = 12582912.0f;     // 1.5 * 2^23
constexpr int kAdjMagicBits = 0x4B400000;
// how a tile reads a projection: footprint beyond the box, nothing, staged, staged and on the detector
enum { kAdjUnfit, kAdjNothing, kAdjStaged, kAdjClean };

__host__ __device__ constexpr size_t adj_smem_bytes()
{
    return sizeof(float) * (2ull * kAdjNB * kAdjBox + 3ull * kAdjNB * kAdjGeo) + sizeof(int2) * 2 * kAdjNB + 2 * sizeof(uint64_t);
}

struct AdjParams {
    const float *proj; // rows of `pitch` floats
    const float2 *sc;
    const float *startu;
    const uint32_t *mask;
    float *vol;
    int nproj, n, nz, pitch, accumulate, wait_limit;
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

__global__ void __launch_bounds__(kAdjThreads, kAdjCtas) k_mbp_adjoint_staged(const __grid_constant__ CUtensorMap tmap,
                                                                              const AdjParams P)
{
    extern __shared__ __align__(1024) float adj_smem[];
    float *box = adj_smem;                                          // [2][NB][TZ][BW]
    float *geo = box + 2 * kAdjNB * kAdjBox;                        // [3][NB][kAdjGeo]
    int2 *meta = reinterpret_cast<int2 *>(geo + 3 * kAdjNB * kAdjGeo); // [2][NB]: first staged column, mode
    uint64_t *bars = reinterpret_cast<uint64_t *>(meta + 2 * kAdjNB);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n = P.n, nz = P.nz;
    const int x0 = blockIdx.x * kAdjTX, y0 = blockIdx.y * kAdjTY, z0 = blockIdx.z * kAdjTZ;
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
    const int nbatch = (P.nproj + kAdjNB - 1) / kAdjNB;
    const int xa = x0 + 1, xb = min(x0 + kAdjTX, n), ya = y0 + 1, yb = min(y0 + kAdjTY, n);
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
        for (int e = threadIdx.x; e < kAdjNB * (kAdjTZ + 2); e += kAdjThreads) {
            const int b = e / (kAdjTZ + 2), c = e - b * (kAdjTZ + 2), i = s * kAdjNB + b < P.nproj ? s * kAdjNB + b : 0;
            const float *src = c < kAdjTZ ? P.startu + static_cast<size_t>(i) * nz + min(z0 + c, nz - 1)
                                          : reinterpret_cast<const float *>(P.sc + i) + (c - kAdjTZ);
            tma::copy4_zfill(geo + (gb * kAdjNB + b) * kAdjGeo + c, src, true);
        }
    };
    // batch s (geometry in buffer gb) into stage st: windows from 8 corner lanes per projection
    auto issue = [&](int s, int st, int gb) {
        if (warp != 0) return;
#pragma unroll 1
        for (int r = 0; r < kAdjNB; r += 4) {
            const int b = r + (lane >> 3), corner = lane & 7, i = s * kAdjNB + b;
            const float *g = geo + (gb * kAdjNB + b) * kAdjGeo;
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
                if (!ok || hi + 2 >= w0 + kAdjBW) mode = kAdjUnfit;
                else if (hi >= -1 && lo <= n) mode = lo >= 1 && hi <= n - 3 ? kAdjClean : kAdjStaged;
            }
            const bool head = corner == 0, load = head && mode >= kAdjStaged;
            const uint32_t bytes = __popc(__ballot_sync(0xffffffffu, load)) * kAdjBox * sizeof(float);
            if (lane == 0) { // the phase completes on the last round's arrival
                if (r + 4 < kAdjNB) tma::mbar_add_tx(&bars[st], bytes);
                else tma::mbar_expect_tx(&bars[st], bytes);
            }
            __syncwarp();
            if (head) meta[st * kAdjNB + b] = make_int2(w0, mode);
            if (load) {
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                tma::load_3d(box + (st * kAdjNB + b) * kAdjBox, &tmap, w0, z0, i, &bars[st]);
            }
        }
    };
    uint32_t phase0 = 0, phase1 = 0;
    bool failed = false;
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
        if (got && inside) {
#pragma unroll 1
            for (int b = 0; b < kAdjNB && s * kAdjNB + b < P.nproj; ++b) {
                const int2 m = meta[st * kAdjNB + b];
                if (m.y == kAdjNothing) continue;
                const float *g = geo + (gb * kAdjNB + b) * kAdjGeo;
                const float cy = __fmul_rn(g[kAdjTZ + 1], fy), sx = __fmul_rn(g[kAdjTZ], fx);
                const float *bx = box + (st * kAdjNB + b) * kAdjBox;
                if (m.y == kAdjClean) {
                    const float2 cy2 = make_float2(cy, cy), sx2 = make_float2(-sx, -sx);
                    const int base = -kAdjMagicBits - m.x;
#pragma unroll
                    for (int q = 0; q < kAdjTZ / 4; ++q) {
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
                const float *img = P.proj + (static_cast<size_t>(s * kAdjNB + b) * nz + z0) * P.pitch;
#pragma unroll
                for (int c = 0; c < kAdjTZ; ++c) {
                    const float u = __fsub_rn(__fadd_rn(g[c], cy), sx);
                    const int k = __float2int_rz(u);
                    if (c >= zmax || k < 0 || k > n - 2) continue;
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
        }
        // batch s + 2's geometry is published; stage st and geometry buffer gb are free
        tma::copy_wait_all();
        if (__syncthreads_or(failed)) break;
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
#pragma unroll
        for (int c = 0; c < kAdjTZ; ++c)
            if (c < zmax) col[c] = (c & 1) ? acc[c >> 1].y : acc[c >> 1].x;
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
    PFN_cuTensorMapEncodeTiled enc = tma::encode_fn();
    if (!enc) return fail(MR_ERR_CUDA, "cuTensorMapEncodeTiled unavailable");
    CUtensorMap map;
    cuuint64_t dims[3] = {static_cast<cuuint64_t>(width), static_cast<cuuint64_t>(P.nz), static_cast<cuuint64_t>(P.nproj)};
    cuuint64_t strides[2] = {static_cast<cuuint64_t>(P.pitch) * 4, static_cast<cuuint64_t>(P.pitch) * P.nz * 4};
    cuuint32_t box[3] = {kAdjBW, kAdjTZ, 1}, estr[3] = {1, 1, 1};
    const CUresult cr = enc(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float *>(P.proj), dims, strides, box, estr,
                            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (cr != CUDA_SUCCESS) return fail(MR_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", static_cast<int>(cr));
    MR_CUDA_TRY(cudaFuncSetAttribute(k_mbp_adjoint_staged, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     static_cast<int>(adj_smem_bytes())));
    const dim3 grid(div_up(static_cast<size_t>(P.n), kAdjTX), div_up(static_cast<size_t>(P.n), kAdjTY),
                    div_up(static_cast<size_t>(P.nz), kAdjTZ));
    k_mbp_adjoint_staged<<<grid, kAdjThreads, adj_smem_bytes(), s>>>(map, P);
    return check_launch("k_mbp_adjoint_staged");
}

// One warp per (projection i, bin m), lanes = 32 consecutive slices from z0.
template <bool DERIV>
__global__ void __launch_bounds__(128) k_mbp_forward(const float *__restrict__ vol, const float2 *__restrict__ sc,
                                                     const float *__restrict__ startu, int nproj, int n, int nz,
                                                     const uint32_t *__restrict__ mask, float *__restrict__ proj,
                                                     float *__restrict__ dproj)
{
    const int lane = threadIdx.x & 31;
    const int m = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int i = blockIdx.y;
    const int z0 = blockIdx.z * 32, z = z0 + lane;
    if (m >= n) return;
    const bool zok = z < nz;
    const float2 s = sc[i];
    const float *su = startu + static_cast<size_t>(i) * nz;
    const float suz = zok ? su[z] : 0.0f;
    // the warp's extreme start positions (startu is affine in z), for the candidate interval
    const int zl = min(z0 + 31, nz - 1);
    const float sua = fminf(su[z0], su[zl]), sub = fmaxf(su[z0], su[zl]);
    const float fm = static_cast<float>(m);
    float acc = 0.0f, dacc = 0.0f;
    auto visit = [&](int x1, int y1) {
        const float u = __fsub_rn(__fadd_rn(suz, __fmul_rn(s.y, static_cast<float>(y1))), __fmul_rn(s.x, static_cast<float>(x1)));
        const int k = __float2int_rz(u);
        if (k < 0 || k > n - 2 || (k != m && k != m - 1)) return;
        const float wb = fabsf(__fsub_rn(u, static_cast<float>(k)));
        const float v = __ldg(vol + (static_cast<size_t>(y1 - 1) * n + (x1 - 1)) * nz + z);
        if (k == m) {
            acc = __fadd_rn(acc, __fmul_rn(v, __fsub_rn(1.0f, wb)));
            if (DERIV) dacc = __fsub_rn(dacc, v);
        } else {
            acc = __fadd_rn(acc, __fmul_rn(v, wb));
            if (DERIV) dacc = __fadd_rn(dacc, v);
        }
    };
    if (fabsf(s.x) >= fabsf(s.y)) {
        // walk the rows y; in row y, u = (su + cos y) - sin x lies in [m - 1, m + 1) for x in
        // ((su + cos y - m - 1) / sin, (su + cos y - m + 1) / sin] (sin > 0; reversed for sin < 0)
        const float inv = 1.0f / s.x;
        for (int y1 = 1; y1 <= n; ++y1) {
            const uint32_t first = mask[2 * (y1 - 1)], second = mask[2 * (y1 - 1) + 1];
            if (second <= first) continue;
            const float cy = s.y * static_cast<float>(y1);
            const float e0 = (sua + cy - fm - 1.0f) * inv, e1 = (sub + cy - fm + 1.0f) * inv;
            int xa = static_cast<int>(floorf(fminf(e0, e1))) - 1, xb = static_cast<int>(ceilf(fmaxf(e0, e1))) + 1;
            xa = max(xa, static_cast<int>(first) + 1);
            xb = min(xb, static_cast<int>(second));
            if (zok)
                for (int x1 = xa; x1 <= xb; ++x1) visit(x1, y1);
        }
    } else {
        // walk the columns x; u lies in [m - 1, m + 1) for y in
        // ((m - 1 - su + sin x) / cos, (m + 1 - su + sin x) / cos] (cos > 0; reversed otherwise)
        const float inv = 1.0f / s.y;
        for (int x1 = 1; x1 <= n; ++x1) {
            const float sx = s.x * static_cast<float>(x1);
            const float e0 = (fm - 1.0f - sub + sx) * inv, e1 = (fm + 1.0f - sua + sx) * inv;
            int ya = max(static_cast<int>(floorf(fminf(e0, e1))) - 1, 1);
            int yb = min(static_cast<int>(ceilf(fmaxf(e0, e1))) + 1, n);
            if (zok)
                for (int y1 = ya; y1 <= yb; ++y1) {
                    const uint32_t first = mask[2 * (y1 - 1)], second = mask[2 * (y1 - 1) + 1];
                    if (static_cast<uint32_t>(x1) > first && static_cast<uint32_t>(x1) <= second) visit(x1, y1);
                }
        }
    }
    if (zok) {
        const size_t o = (static_cast<size_t>(i) * nz + z) * n + m;
        proj[o] = acc;
        if (DERIV) dproj[o] = dacc;
    }
}

// The same forward projection, voxel-driven (used while the bins fit in shared memory): one CTA
// per (projection i, 32 slices) holds that projection's bins of its slices in shared memory
// (bin-major rows padded to 33 words, so the 32 lanes - one slice each - of a warp hit 32 banks
// and the write-out reads 32 consecutive bins without conflicts). Its warps walk the masked
// voxels line by line, along the axis on which u changes least (x when |sin| <= |cos|, else y;
// |du| <= 1/sqrt(2) per step, so a lane's bin moves by at most one between steps), each voxel
// once, with the adjoint's u, n, wa and wb. A lane keeps the running sums of its current pair of
// bins (n, n + 1) in registers and adds a bin to shared memory (atomically) when its walk leaves
// it, so most voxels cost no shared-memory access. The order of the additions into a bin depends
// on the warps' timing: results agree with the ray-driven kernel to float summation, not bit for
// bit.
constexpr int kFwdPad = 33;
constexpr int kFwdThreads = 1024;

__host__ __device__ inline size_t fwd_smem_bytes(int n, bool deriv)
{
    return static_cast<size_t>(n) * kFwdPad * sizeof(float) * (deriv ? 2 : 1) + static_cast<size_t>(n) * sizeof(uint2) * 2;
}

template <bool DERIV>
struct BinRun {
    int mc = -2; // current bin (-2: none yet)
    float a0 = 0.0f, a1 = 0.0f, d0 = 0.0f, d1 = 0.0f;
    // one voxel: bin m (0 <= m <= n - 2), weights wa, wb, value v
    __device__ __forceinline__ void add(float *bins, float *dbins, int lane, int m, float wa, float wb, float v)
    {
        (void)dbins; // (the derivative bins follow the value bins)
        const float pa = __fmul_rn(v, wa), pb = __fmul_rn(v, wb);
        const int diff = m - mc;
        if (diff == 0) {
            a0 = __fadd_rn(a0, pa);
            a1 = __fadd_rn(a1, pb);
            if (DERIV) {
                d0 = __fsub_rn(d0, v);
                d1 = __fadd_rn(d1, v);
            }
        } else if (diff == -1) { // bin mc + 1 is left behind
            atomicAdd(bins + (mc + 1) * kFwdPad + lane, a1);
            a1 = __fadd_rn(a0, pb);
            a0 = pa;
            if (DERIV) {
                atomicAdd(dbins + (mc + 1) * kFwdPad + lane, d1);
                d1 = __fadd_rn(d0, v);
                d0 = -v;
            }
            mc = m;
        } else if (diff == 1) { // bin mc is left behind
            atomicAdd(bins + mc * kFwdPad + lane, a0);
            a0 = __fadd_rn(a1, pa);
            a1 = pb;
            if (DERIV) {
                atomicAdd(dbins + mc * kFwdPad + lane, d0);
                d0 = __fsub_rn(d1, v);
                d1 = v;
            }
            mc = m;
        } else {
            done(bins, dbins, lane);
            a0 = pa;
            a1 = pb;
            if (DERIV) {
                d0 = -v;
                d1 = v;
            }
            mc = m;
        }
    }
    __device__ __forceinline__ void done(float *bins, float *dbins, int lane) const
    {
        if (mc < 0) return;
        atomicAdd(bins + mc * kFwdPad + lane, a0);
        atomicAdd(bins + (mc + 1) * kFwdPad + lane, a1);
        if (DERIV) {
            atomicAdd(dbins + mc * kFwdPad + lane, d0);
            atomicAdd(dbins + (mc + 1) * kFwdPad + lane, d1);
        }
    }
};

template <bool DERIV>
__global__ void __launch_bounds__(kFwdThreads, 1) k_mbp_forward_smem(const float *__restrict__ vol, const float2 *__restrict__ sc,
                                                                  const float *__restrict__ startu, int nproj, int n,
                                                                  int nz, const uint32_t *__restrict__ mask,
                                                                  float *__restrict__ proj, float *__restrict__ dproj)
{
    extern __shared__ float bins[]; // [n][kFwdPad] (+ [n][kFwdPad] for the derivative), then the masks
    float *dbins = bins + static_cast<size_t>(n) * kFwdPad;
    uint2 *rowmask = reinterpret_cast<uint2 *>(bins + static_cast<size_t>(n) * kFwdPad * (DERIV ? 2 : 1));
    uint2 *colspan = rowmask + n; // per column x: the rows [lo, hi] that hold voxels of it
    const int i = blockIdx.x, z0 = blockIdx.y * 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
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
            int lo = 0, hi = -1;
            for (int y = 0; y < n; ++y)
                if (x1 > rowmask[y].x && x1 <= rowmask[y].y) {
                    lo = y;
                    break;
                }
            for (int y = n - 1; y >= lo; --y)
                if (x1 > rowmask[y].x && x1 <= rowmask[y].y) {
                    hi = y;
                    break;
                }
            colspan[x] = make_uint2(static_cast<uint32_t>(lo), static_cast<uint32_t>(hi + 1));
        }
    __syncthreads();
    BinRun<DERIV> run;
    const float suz = zok ? startu[static_cast<size_t>(i) * nz + z] : 0.0f;
    if (zok) {
        if (by_rows) {
            // line y: voxels x in (first, second], u = (su + cos y) - sin x
            for (int y = warp; y < n; y += nwarps) {
                const uint2 r = rowmask[y];
                const float a = __fadd_rn(suz, __fmul_rn(s.y, static_cast<float>(y + 1)));
                const float *p = vol + (static_cast<size_t>(y) * n + r.x) * nz + z;
                constexpr int U = 4;
                int x = static_cast<int>(r.x);
                const int xe = min(static_cast<int>(r.y), n);
                for (; x < xe; x += U) {
                    float v[U];
#pragma unroll
                    for (int j = 0; j < U; ++j) v[j] = (x + j < xe) ? __ldg(p + static_cast<size_t>(j) * nz) : 0.0f;
#pragma unroll
                    for (int j = 0; j < U; ++j) {
                        if (x + j >= xe) continue;
                        const float u = __fsub_rn(a, __fmul_rn(s.x, static_cast<float>(x + j + 1)));
                        const int m = __float2int_rz(u);
                        if (m < 0 || m > n - 2) continue;
                        const float wb = fabsf(__fsub_rn(u, static_cast<float>(m)));
                        if (!MR_IN_BOUNDS(m + 1, n, kSiteMbpBins)) continue;
                        run.add(bins, dbins, lane, m, __fsub_rn(1.0f, wb), wb, v[j]);
                    }
                    p += static_cast<size_t>(U) * nz;
                }
            }
        } else {
            // line x: voxels y in the column's span that the row masks hold
            for (int x = warp; x < n; x += nwarps) {
                const uint2 span = colspan[x];
                const uint32_t x1 = static_cast<uint32_t>(x) + 1;
                const float sx = __fmul_rn(s.x, static_cast<float>(x1));
                const size_t ystride = static_cast<size_t>(n) * nz;
                const float *p = vol + (static_cast<size_t>(span.x) * n + x) * nz + z;
                constexpr int U = 4;
                int y = static_cast<int>(span.x);
                const int ye = static_cast<int>(span.y);
                for (; y < ye; y += U) {
                    float v[U];
                    bool in[U];
#pragma unroll
                    for (int j = 0; j < U; ++j) {
                        in[j] = y + j < ye && x1 > rowmask[y + j].x && x1 <= rowmask[y + j].y;
                        v[j] = in[j] ? __ldg(p + static_cast<size_t>(j) * ystride) : 0.0f;
                    }
#pragma unroll
                    for (int j = 0; j < U; ++j) {
                        if (!in[j]) continue;
                        const float u = __fsub_rn(__fadd_rn(suz, __fmul_rn(s.y, static_cast<float>(y + j + 1))), sx);
                        const int m = __float2int_rz(u);
                        if (m < 0 || m > n - 2) continue;
                        const float wb = fabsf(__fsub_rn(u, static_cast<float>(m)));
                        if (!MR_IN_BOUNDS(m + 1, n, kSiteMbpBins)) continue;
                        run.add(bins, dbins, lane, m, __fsub_rn(1.0f, wb), wb, v[j]);
                    }
                    p += static_cast<size_t>(U) * ystride;
                }
            }
        }
        run.done(bins, dbins, lane);
    }
    __syncthreads();
    // write-out: consecutive threads take consecutive bins of one slice (coalesced stores)
    const int zs = min(32, nz - z0);
    for (int e = threadIdx.x; e < zs * n; e += blockDim.x) {
        const int zz = e / n, m = e - zz * n;
        const size_t o = (static_cast<size_t>(i) * nz + z0 + zz) * n + m;
        proj[o] = bins[m * kFwdPad + zz];
        if (DERIV) dproj[o] = dbins[m * kFwdPad + zz];
    }
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
    const size_t run = std::min(nproj, std::max<size_t>(kAdjNB, (size_t(64) << 20) / (per * 4)));
    float *scratch = nullptr;
    MR_TRY(device_alloc(&scratch, run * per * sizeof(float), s, "mr_mbp_adjoint: padded projections"));
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
    int dev = 0, optin = 0;
    MR_CUDA_TRY(cudaGetDevice(&dev));
    MR_CUDA_TRY(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    const size_t smem = fwd_smem_bytes(static_cast<int>(n), dproj_d != nullptr);
    if (smem <= static_cast<size_t>(optin)) {
        dim3 sgrid(static_cast<unsigned>(nproj), div_up(nz, 32));
        auto launch = [&](auto kernel, float *d) -> mr_status {
            MR_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
            kernel<<<sgrid, kFwdThreads, smem, as_stream(stream)>>>(vol_d, sc, startu_d, static_cast<int>(nproj),
                                                                   static_cast<int>(n), static_cast<int>(nz), mask_d,
                                                                   proj_d, d);
            return check_launch("k_mbp_forward_smem");
        };
        return dproj_d ? launch(k_mbp_forward_smem<true>, dproj_d) : launch(k_mbp_forward_smem<false>, nullptr);
    }
    // bins beyond shared memory: the ray-driven kernel
    dim3 grid(div_up(n, 4), static_cast<unsigned>(nproj), div_up(nz, 32));
    if (dproj_d)
        k_mbp_forward<true><<<grid, 128, 0, as_stream(stream)>>>(vol_d, reinterpret_cast<const float2 *>(sincos_d),
                                                               startu_d, static_cast<int>(nproj), static_cast<int>(n),
                                                               static_cast<int>(nz), mask_d, proj_d, dproj_d);
    else
        k_mbp_forward<false><<<grid, 128, 0, as_stream(stream)>>>(vol_d, reinterpret_cast<const float2 *>(sincos_d),
                                                                startu_d, static_cast<int>(nproj), static_cast<int>(n),
                                                                static_cast<int>(nz), mask_d, proj_d, nullptr);
    return check_launch("k_mbp_forward");
}

} // extern "C"
