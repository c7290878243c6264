// Parallel-beam backprojection with TMA-staged projection rows (sm_100a).
//
// Arithmetic of MultiProjectionBPparallel::BackProject (MultiProjBPparallel.cpp:39-170), with and
// without tilt correction, and of the factory's serial and nearest-neighbour backprojectors, every
// float operation in the reference's order and rounded on its own, so the volume is bit-identical
// to the plain kernel and to the reference; without tilt
//   u = (startu_i + cos_i y) - sin_i x,  n = (int)u in [0, nu-2],  f = |u - n|,
//   vol[y-1][x-1][z] += (P[z][n] (1 - f) + P[z][n+1] f)          (P pre-multiplied by weight_i)
//
// Tiling: a CTA owns 32 (x) x 2 NW (y) voxel columns x TZ slices; a thread keeps the TZ slices of
// two neighbouring rows' columns in registers over all projections. In this geometry the detector
// column of a voxel does not depend on its slice, so one projection's footprint on the tile is at
// most ~37 columns by the tile's TZ detector rows: a producer warp projects the 4 tile corners with
// the voxel formula (affine in x and y, and float rounding is monotone, so the corners bound every
// voxel exactly; the per-projection sin/cos/startu are copied into shared memory with cp.async three
// batches ahead and the corners use those copies, as the voxels do), and one TMA tile load
// (cp.async.bulk.tensor.3d, no multicast) brings a 48 x TZ box per projection into shared memory,
// batches of NB projections on two stages with bounded mbarrier waits. Rows beyond the detector are
// zero-filled by the TMA unit (slices from 4*(nv/4) on are computed and never stored). A footprint
// that does not fit the box falls back to guarded global loads for that tile and projection (same
// arithmetic). The volume (z fastest) is read and written as float4 runs.
//
// Bound: shared-memory load wavefronts (78 % of the LSU's peak) and instruction issue (64 %). One
// row per thread needs two samples per update, 2.2 wavefronts and 6.9 warp instructions with the
// set-up; two rows share three samples, and slices go in pairs through the paired FP32 pipe: 1.7
// wavefronts and 5.6 instructions. 2048^2 x 64 slices from 1125 projections: 60.8 -> 47.4 ms;
// 1001^2 x 60 with tilt from 625 projections: 30.1 (direct-load kernel) -> 7.8 ms.
#include "mr_common.cuh"
#include "mr_tma.cuh"

#include <algorithm>
#include <cmath>

namespace mr {

// Error word of this file's bounded waits (device globals are per translation unit);
// mr_device_status reads and clears it with the FDK kernels' word.
__device__ int g_bp_error = 0;

MR_BOUNDS_TAKE(bounds_take_bp)

int bp_device_status_take()
{
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_bp_error, sizeof(int)) != cudaSuccess) return -1;
    if (cudaMemcpyToSymbol(g_bp_error, &zero, sizeof(int)) != cudaSuccess) return -1;
    return v;
}

namespace bp2 {

constexpr int TX = 32, G = 4, BW = 48;
constexpr float kMagic = 12582912.0f; // 1.5 * 2^23
constexpr int kMagicBits = 0x4B400000;
constexpr int GEO = 4; // sin, cos, startu, slab (as int bits)

// What a voxel adds per projection (MultiProjBPparallel.cpp:39-170 and the factory's other two):
//   kLinear      acc += pa (1 - f) + pb f, f = |u - n|
//   kNearest     acc += pa (NNMultiProjBP.cpp:84-90)
//   kTilt        u shifted by the centre offset before the x term; f of slice group g is
//                |(u - n) - g inc - g inc|, the first shift a running subtraction (:86-105)
//   kTiltSerial  u shifted after the x term, f = |(u - n) - g inc| (MultiProjBP.cpp:61-84)
//   kTiltNearest u shifted after the x term, the sample at n (NNMultiProjBP.cpp:61-90)
enum Mode { kLinear, kNearest, kTilt, kTiltSerial, kTiltNearest };

// How a tile reads one projection: its footprint does not fit the box (guarded global loads), no
// voxel of the tile lies on the detector, staged, staged with every voxel of the tile on the detector
// and n of neighbouring rows the same or one apart (rows_share).
enum Footprint { kUnfit, kNothing, kStaged, kClean };

struct Params {
    const float *proj;
    const int32_t *index;
    const float *sinv, *cosv, *startu;
    const uint32_t *mask;
    float *vol;
    int nproj, nu, nv, nz4;
    int wait_limit; // tries of each per-batch wait
    int ybegin, yend; // volume rows y1 - 1 in [ybegin, yend)
    int pitch;        // floats between detector rows
    float toff, tinc; // tilt: centre offset and its step per group of 4 slices
    float neg_zero;   // -0 (see blend_add)
};

template <int TZ, int NB>
struct Smem {
    static constexpr int BOXBYTES = BW * TZ * 4;
    float *box;      // [2][NB][TZ][BW]
    float *geo;      // [3][NB][GEO]
    int4 *meta;      // [2][NB]: x0, mode
    uint64_t *bars;  // [2]
    __device__ explicit Smem(unsigned char *base)
    {
        box = reinterpret_cast<float *>(base);
        geo = reinterpret_cast<float *>(base + 2 * NB * BOXBYTES);
        meta = reinterpret_cast<int4 *>(geo + 3 * NB * GEO);
        bars = reinterpret_cast<uint64_t *>(meta + 2 * NB);
    }
    static constexpr size_t bytes()
    {
        return 2 * NB * static_cast<size_t>(BOXBYTES) + 3 * NB * GEO * sizeof(float) + 2 * NB * sizeof(int4) +
               2 * sizeof(uint64_t);
    }
};

// Detector position of voxel (x1, y1) (1-based) for list entry i, reference order.
template <int MODE>
__device__ __forceinline__ float posu(float sn, float cs, float su, float fx, float fy, float toff)
{
    float local = __fadd_rn(su, __fmul_rn(cs, fy));
    if constexpr (MODE == kTilt) local = __fsub_rn(local, toff);
    const float u = __fsub_rn(local, __fmul_rn(sn, fx));
    if constexpr (MODE == kTiltSerial || MODE == kTiltNearest) return __fsub_rn(u, toff);
    return u;
}

// Are n(x, y) and n(x, y + 1) at most one apart? u changes by cos between the two, plus the rounding of
// cos y, of the sum and of the differences that follow, half a step of each value per row (sin x is the
// same value in both). The values' sum is convex in x and y, so that of the tile's corners bounds it. At
// 2048 columns |cos| may reach 0.999, at 65536 columns 0.97.
template <int MODE>
__device__ __forceinline__ bool rows_share(float cs, float su, float fy, float toff, float u)
{
    const float cy = cs * fy;
    float values = fabsf(cy) + fabsf(su + cy) + fabsf(u);
    if constexpr (MODE == kTilt || MODE == kTiltSerial || MODE == kTiltNearest)
        values += fabsf(su + cy) + fabsf(u) + 2.0f * fabsf(toff);
    return fabsf(cs) + 1.25f * 0x1p-23f * values < 1.0f;
}

// Two slices of acc += pa * wa + pb * wb in the reference's order, every product and sum rounded on
// its own. ptxas contracts a paired multiply that feeds a paired add even when both carry .rn, so the
// products are paired fmas with an addend of -0 that it cannot see (`nz`, a kernel argument): p + -0 is
// p bit for bit, signed zeros included, and the sum that follows stays an add.
__device__ __forceinline__ void blend_add(float2 &acc, float2 pa, float2 pb, float2 wa, float2 wb, float2 nz)
{
    acc = __fadd2_rn(acc, __fadd2_rn(__ffma2_rn(pa, wa, nz), __ffma2_rn(pb, wb, nz)));
}

__device__ __forceinline__ float2 both(float v) { return make_float2(v, v); }

// Interpolation weight of slice group g (float) of a voxel whose u - n is d; kTilt also steps d.
template <int MODE>
__device__ __forceinline__ float group_weight(float &d, float g, float tinc)
{
    if constexpr (MODE != kTilt && MODE != kTiltSerial) return fabsf(d);
    const float f = fabsf(__fsub_rn(d, __fmul_rn(g, tinc)));
    if constexpr (MODE == kTilt) d = __fsub_rn(d, tinc);
    return f;
}

// One voxel column's slices for one staged projection: p points at the sample pair of slice 0 (row
// pitch BW), d is u - n.
template <int MODE, int TZ>
__device__ __forceinline__ void staged_column(float2 (&acc)[TZ / 2], const float *p, float d, float g0, float tinc, float2 nz)
{
#pragma unroll
    for (int q4 = 0; q4 < TZ; q4 += 4) {
        const float wb = group_weight<MODE>(d, g0 + static_cast<float>(q4 / 4), tinc), wa = __fsub_rn(1.0f, wb);
#pragma unroll
        for (int q = q4; q < q4 + 4; q += 2) {
            const float2 pa = make_float2(p[q * BW], p[(q + 1) * BW]);
            if constexpr (MODE == kNearest || MODE == kTiltNearest) acc[q / 2] = __fadd2_rn(acc[q / 2], pa);
            else blend_add(acc[q / 2], pa, make_float2(p[q * BW + 1], p[(q + 1) * BW + 1]), both(wa), both(wb), nz);
        }
    }
}

// Two voxel columns at once, each only where it reaches the detector (on0, on1): footprints that lie partly
// outside it, on tiles of few slices. One column after the other, behind a branch each, their latency held up
// the tiles at the volume's corners: 128^2 x 8 slices from 180 projections 59 -> 53 us. (32-slice tiles have
// the warps to hide it: 256^2 x 64 from 360 takes 388 us that way, 399 this way.)
template <int MODE, int TZ>
__device__ __forceinline__ void staged_columns(float2 (&acc0)[TZ / 2], float2 (&acc1)[TZ / 2], const float *p0, const float *p1,
                                               float d0, float d1, bool on0, bool on1, float g0, float tinc, float2 nz)
{
#pragma unroll
    for (int q4 = 0; q4 < TZ; q4 += 4) {
        const float g = g0 + static_cast<float>(q4 / 4);
        const float wb0 = group_weight<MODE>(d0, g, tinc), wa0 = __fsub_rn(1.0f, wb0);
        const float wb1 = group_weight<MODE>(d1, g, tinc), wa1 = __fsub_rn(1.0f, wb1);
#pragma unroll
        for (int q = q4; q < q4 + 4; q += 2) {
            float2 s0 = acc0[q / 2], s1 = acc1[q / 2];
            const float2 a0 = make_float2(p0[q * BW], p0[(q + 1) * BW]), a1 = make_float2(p1[q * BW], p1[(q + 1) * BW]);
            if constexpr (MODE == kNearest || MODE == kTiltNearest) {
                s0 = __fadd2_rn(s0, a0);
                s1 = __fadd2_rn(s1, a1);
            } else {
                blend_add(s0, a0, make_float2(p0[q * BW + 1], p0[(q + 1) * BW + 1]), both(wa0), both(wb0), nz);
                blend_add(s1, a1, make_float2(p1[q * BW + 1], p1[(q + 1) * BW + 1]), both(wa1), both(wb1), nz);
            }
            acc0[q / 2] = make_float2(on0 ? s0.x : acc0[q / 2].x, on0 ? s0.y : acc0[q / 2].y);
            acc1[q / 2] = make_float2(on1 ? s1.x : acc1[q / 2].x, on1 ? s1.y : acc1[q / 2].y);
        }
    }
}

// The slices of two voxels of neighbouring rows for one staged projection. u changes by cos between
// them, so the second voxel's pair of samples is the first one's (step false) or the next (step
// true): three samples serve both, where each alone loads two. lo is the voxel with the smaller n.
template <int MODE, int TZ>
__device__ __forceinline__ void staged_pair(float2 (&lo)[TZ / 2], float2 (&hi)[TZ / 2], const float *p, bool step, float dlo,
                                            float dhi, float g0, float tinc, float2 nz)
{
#pragma unroll
    for (int q4 = 0; q4 < TZ; q4 += 4) {
        const float g = g0 + static_cast<float>(q4 / 4);
        const float wbl = group_weight<MODE>(dlo, g, tinc), wal = __fsub_rn(1.0f, wbl);
        const float wbh = group_weight<MODE>(dhi, g, tinc), wah = __fsub_rn(1.0f, wbh);
#pragma unroll
        for (int q = q4; q < q4 + 4; q += 2) {
            const float2 s0 = make_float2(p[q * BW], p[(q + 1) * BW]);
            const float2 s1 = make_float2(p[q * BW + 1], p[(q + 1) * BW + 1]);
            const float2 s2 = make_float2(p[q * BW + 2], p[(q + 1) * BW + 2]);
            blend_add(lo[q / 2], s0, s1, both(wal), both(wbl), nz);
            blend_add(hi[q / 2], make_float2(step ? s1.x : s0.x, step ? s1.y : s0.y),
                      make_float2(step ? s2.x : s1.x, step ? s2.y : s1.y), both(wah), both(wbh), nz);
        }
    }
}

// A CTA of NW warps owns 32 (x) x 2 NW (y) voxel columns x TZ slices; a thread keeps the TZ slices
// of two neighbouring rows' columns in registers over all projections.
template <int MODE, int TZ, int NW, int NB, int CTAS>
__global__ void __launch_bounds__(32 * NW, CTAS) k_bp_par_staged(const __grid_constant__ CUtensorMap tmap, const Params P)
{
    constexpr int THREADS = 32 * NW, TY = 2 * NW;
    constexpr bool kOneSample = MODE == kNearest || MODE == kTiltNearest;
    constexpr int BOXBYTES = Smem<TZ, NB>::BOXBYTES;
    extern __shared__ __align__(1024) unsigned char smem[];
    Smem<TZ, NB> S(smem);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int i0 = blockIdx.x * TX, j0 = P.ybegin + blockIdx.y * TY, z0 = blockIdx.z * TZ;
    const int x1 = i0 + lane + 1, y1 = j0 + 2 * warp + 1; // rows y1 and y1 + 1
    const int zmax = min(TZ, P.nz4 - z0);
    bool inside[2];
    float *col[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const bool valid = x1 <= P.nu && y1 + r <= P.yend;
        inside[r] = valid && static_cast<uint32_t>(x1) > P.mask[2 * (y1 + r - 1)] &&
                    static_cast<uint32_t>(x1) <= P.mask[2 * (y1 + r - 1) + 1];
        col[r] = P.vol + (static_cast<size_t>(valid ? y1 + r - 1 : 0) * P.nu + (valid ? x1 - 1 : 0)) * P.nv + z0;
    }
    const bool vec = (P.nv & 3) == 0 && zmax == TZ;

    float2 acc0[TZ / 2], acc1[TZ / 2];
    auto load = [&](float2 (&acc)[TZ / 2], const float *c, bool in) {
#pragma unroll
        for (int q = 0; q < TZ; q += 4) {
            float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (in && vec) {
                v = *reinterpret_cast<const float4 *>(c + q);
            } else if (in && q < zmax) {
                v = make_float4(c[q], c[q + 1], c[q + 2], c[q + 3]);
            }
            acc[q / 2] = make_float2(v.x, v.y);
            acc[q / 2 + 1] = make_float2(v.z, v.w);
        }
    };
    load(acc0, col[0], inside[0]);
    load(acc1, col[1], inside[1]);
    const bool any_inside = inside[0] || inside[1];
    if (!__syncthreads_or(any_inside)) return;

    if (threadIdx.x == 0) {
        tma::mbar_init(&S.bars[0], 1);
        tma::mbar_init(&S.bars[1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();

    const int xa = i0 + 1, xb = min(i0 + TX, P.nu), ya = j0 + 1, yb = min(j0 + TY, P.yend);
    const int nbatch = (P.nproj + NB - 1) / NB;

    // Geometry of batch s into geometry buffer gb (cp.async by all threads, three batches
    // ahead; the slab only with an index list).
    auto stage_geometry = [&](int s, int gb) {
        for (int idx = threadIdx.x; idx < NB * GEO; idx += THREADS) {
            const int b = idx / GEO, e = idx % GEO, i = s * NB + b;
            const float *src = e == 0 ? P.sinv : e == 1 ? P.cosv : e == 2 ? P.startu : reinterpret_cast<const float *>(P.index);
            const bool ok = i < P.nproj && (e < 3 || P.index);
            tma::copy4_zfill(S.geo + gb * NB * GEO + idx, ok ? src + i : P.sinv, ok);
        }
    };
    // Batch s (geometry in buffer gb) into stage st: warp 0 forms the footprints from the
    // staged geometry (4 corner lanes per projection) and issues the TMA copies.
    auto issue_batch = [&](int s, int st, int gb) {
        if (warp != 0) return;
#pragma unroll 1
        for (int r = 0; r < NB; r += 8) {
            const int b = r + (lane >> 2), corner = lane & 3;
            const int i = s * NB + b;
            const float *g = S.geo + (gb * NB + (b < NB ? b : 0)) * GEO;
            int nmin = 0, nmax = 0;
            bool ok = b < NB && i < P.nproj, pairs = true;
            if (ok) {
                const float fy = static_cast<float>((corner & 2) ? yb : ya);
                const float u = posu<MODE>(g[0], g[1], g[2], static_cast<float>((corner & 1) ? xb : xa), fy, P.toff);
                ok = fabsf(u) < 1.0e9f;
                nmin = nmax = ok ? __float2int_rz(u) : 0;
                pairs = u >= 0.0f && rows_share<MODE>(g[1], g[2], fy, P.toff, u);
            }
#pragma unroll
            for (int o = 1; o < 4; o <<= 1) {
                nmin = min(nmin, __shfl_xor_sync(0xffffffffu, nmin, o));
                nmax = max(nmax, __shfl_xor_sync(0xffffffffu, nmax, o));
                ok = __shfl_xor_sync(0xffffffffu, static_cast<int>(ok), o) && ok;
                pairs = __shfl_xor_sync(0xffffffffu, static_cast<int>(pairs), o) && pairs;
            }
            int mode = kUnfit, x0 = 0;
            if (ok) {
                if (nmax < 0 || nmin > P.nu - 2) {
                    mode = kNothing;
                } else {
                    x0 = nmin >= 0 ? (nmin & ~3) : -(((-nmin) + 3) & ~3);
                    if (nmax + 1 < x0 + BW) mode = pairs && nmax <= P.nu - 2 ? kClean : kStaged;
                }
            }
            const unsigned staged = __ballot_sync(0xffffffffu, corner == 0 && mode >= kStaged);
            if (lane == 0) {
                // the phase completes on the last round's arrival; earlier rounds only add their bytes
                const uint32_t bytes = static_cast<uint32_t>(__popc(staged)) * BOXBYTES;
                if (r + 8 < NB) tma::mbar_add_tx(&S.bars[st], bytes);
                else tma::mbar_expect_tx(&S.bars[st], bytes);
            }
            __syncwarp();
            if (corner == 0 && b < NB && i < P.nproj) {
                S.meta[st * NB + b] = make_int4(x0, mode, 0, 0);
                if (mode >= kStaged) {
                    const int slab = P.index ? __float_as_int(g[3]) : i;
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    tma::load_3d(S.box + (st * NB + b) * (BW * TZ), &tmap, x0, z0, slab, &S.bars[st]);
                }
            }
        }
    };

    for (int s = 0; s < 3 && s < nbatch; ++s) stage_geometry(s, s);
    tma::copy_wait_all();
    __syncthreads();
    for (int s = 0; s < 2 && s < nbatch; ++s) issue_batch(s, s, s);
    __syncthreads();

    uint32_t phase0 = 0, phase1 = 0;
    bool failed = false;
    // a thread past the volume follows the last column or row (its sums are never stored), so every
    // position of the tile lies between the corners'
    const float fx = static_cast<float>(min(x1, P.nu)), fy0 = static_cast<float>(min(y1, P.yend)),
                fy1 = static_cast<float>(min(y1 + 1, P.yend));
    const int um2 = P.nu - 2;
    const int group0 = z0 / 4;
    const float g0 = static_cast<float>(group0);
    const float2 nz = both(P.neg_zero);
    int s = 0;
    for (int gb = 0; s < nbatch; ++s, gb = gb == 2 ? 0 : gb + 1) {
        const int st = s & 1; // stage buffer; geometry buffer gb = s % 3
        // a wait that timed out skips the batch in its whole warp; the block then leaves the
        // loop together at the barrier below
        const bool got = __all_sync(0xffffffffu, tma::mbar_wait(&S.bars[st], st ? phase1 : phase0, P.wait_limit));
        if (got) {
            if (st) phase1 ^= 1; else phase0 ^= 1;
        } else {
            failed = true;
            if (lane == 0) atomicExch(&g_bp_error, 1);
        }
        if (got && any_inside) {
            // kTilt: the running shift of the slice groups below this tile
            auto skip_groups = [&](float &d) {
                if constexpr (MODE == kTilt)
                    for (int g = 0; g < group0; ++g) d = __fsub_rn(d, P.tinc);
            };
            // One row's column from any footprint (fallback, and edges of 32-slice tiles: positions formed here).
            auto row = [&](float2 (&acc)[TZ / 2], int b, float4 g, int4 m, float fy) {
                const float u = posu<MODE>(g.x, g.y, g.z, fx, fy, P.toff);
                const int n = __float2int_rz(u);
                if (n < 0 || n > um2) return;
                float d = __fsub_rn(u, static_cast<float>(n));
                skip_groups(d);
                if (TZ >= 32 && m.y != kUnfit) {
                    // the box holds all TZ rows (zeros beyond the detector); slices from zmax on are not stored
                    const uint32_t off = static_cast<uint32_t>((st * NB + b) * (BW * TZ) + (n - m.x));
                    if (MR_IN_BOUNDS(off + (TZ - 1) * BW + 1, 2 * NB * BW * TZ, kSiteBpStaged))
                        staged_column<MODE, TZ>(acc, S.box + off, d, g0, P.tinc, nz);
                    return;
                }
                const int slab = P.index ? __float_as_int(g.w) : s * NB + b;
                const float *img = P.proj + (static_cast<size_t>(slab) * P.nv + z0) * P.pitch + n;
#pragma unroll
                for (int q4 = 0; q4 < TZ; q4 += 4) {
                    if (q4 >= zmax) break;
                    const float wb = group_weight<MODE>(d, g0 + static_cast<float>(q4 / 4), P.tinc);
                    const float wa = __fsub_rn(1.0f, wb);
#pragma unroll
                    for (int q = q4; q < q4 + 4; q += 2) {
                        const float *r0 = img + static_cast<size_t>(q) * P.pitch, *r1 = r0 + P.pitch;
                        const float2 pa = make_float2(__ldg(r0), __ldg(r1));
                        if constexpr (kOneSample) acc[q / 2] = __fadd2_rn(acc[q / 2], pa);
                        else blend_add(acc[q / 2], pa, make_float2(__ldg(r0 + 1), __ldg(r1 + 1)), both(wa), both(wb), nz);
                    }
                }
            };
#pragma unroll 1
            for (int b0 = 0; b0 < NB && s * NB + b0 < P.nproj; b0 += G) {
                // the set-up of a group's clean footprints is formed first so its latency overlaps,
                // then the group's slice loops run in projection order (the reference's summation
                // order), one copy of them in the instruction cache: the set-up moves down a register
                // per projection. n is the floor of u >= 0, from the bits of u + 1.5 * 2^23 added
                // rounding down. The smaller n's offset, twice, plus the step to the other row's.
                uint32_t q_at[G];
                float q_d0[G], q_d1[G];
#pragma unroll
                for (int e = 0; e < G; ++e) {
                    const float4 g = reinterpret_cast<const float4 *>(S.geo)[gb * NB + b0 + e];
                    const float u0 = posu<MODE>(g.x, g.y, g.z, fx, fy0, P.toff), u1 = posu<MODE>(g.x, g.y, g.z, fx, fy1, P.toff);
                    const float k0 = __fadd_rd(u0, kMagic), k1 = __fadd_rd(u1, kMagic);
                    q_d0[e] = __fsub_rn(u0, __fsub_rn(k0, kMagic));
                    q_d1[e] = __fsub_rn(u1, __fsub_rn(k1, kMagic));
                    const int n0 = __float_as_int(k0), n1 = __float_as_int(k1); // biased by kMagicBits
                    const int lo = g.y >= 0.0f ? n0 : n1;
                    q_at[e] = static_cast<uint32_t>(2 * (lo + ((st * NB + b0 + e) * (BW * TZ) - kMagicBits - S.meta[st * NB + b0 + e].x)) +
                                                    (n0 != n1));
                }
                if constexpr (MODE == kTilt) {
                    for (int g = 0; g < group0; ++g) {
#pragma unroll
                        for (int e = 0; e < G; ++e) {
                            q_d0[e] = __fsub_rn(q_d0[e], P.tinc);
                            q_d1[e] = __fsub_rn(q_d1[e], P.tinc);
                        }
                    }
                }
#pragma unroll 1
                for (int e = 0; e < G && s * NB + b0 + e < P.nproj; ++e) {
                    const int b = b0 + e;
                    const int4 m = S.meta[st * NB + b];
                    const float4 g = reinterpret_cast<const float4 *>(S.geo)[gb * NB + b];
                    if (m.y == kClean) {
                        const bool step = q_at[0] & 1;
                        const uint32_t at = q_at[0] >> 1;
                        if (!MR_IN_BOUNDS(at + (TZ - 1) * BW + 1 + step, 2 * NB * BW * TZ, kSiteBpStaged)) {
                        } else if constexpr (kOneSample) {
                            const uint32_t a0 = at + (step && g.y < 0.0f), a1 = at + (step && g.y >= 0.0f);
                            staged_column<MODE, TZ>(acc0, S.box + a0, q_d0[0], g0, P.tinc, nz);
                            staged_column<MODE, TZ>(acc1, S.box + a1, q_d1[0], g0, P.tinc, nz);
                        } else if (g.y >= 0.0f) { // uniform
                            staged_pair<MODE, TZ>(acc0, acc1, S.box + at, step, q_d0[0], q_d1[0], g0, P.tinc, nz);
                        } else {
                            staged_pair<MODE, TZ>(acc1, acc0, S.box + at, step, q_d1[0], q_d0[0], g0, P.tinc, nz);
                        }
                    } else if (m.y == kStaged && TZ < 32) {
                        // positions formed here, truncated as the reference does. The box holds all TZ rows
                        // (zeros beyond the detector); slices from zmax on are not stored
                        const float u0 = posu<MODE>(g.x, g.y, g.z, fx, fy0, P.toff), u1 = posu<MODE>(g.x, g.y, g.z, fx, fy1, P.toff);
                        const int n0 = __float2int_rz(u0), n1 = __float2int_rz(u1);
                        bool on0 = inside[0] && n0 >= 0 && n0 <= um2, on1 = inside[1] && n1 >= 0 && n1 <= um2;
                        float d0 = __fsub_rn(u0, static_cast<float>(n0)), d1 = __fsub_rn(u1, static_cast<float>(n1));
                        skip_groups(d0);
                        skip_groups(d1);
                        const uint32_t at = static_cast<uint32_t>((st * NB + b) * (BW * TZ));
                        const uint32_t a0 = at + (on0 ? n0 - m.x : 0), a1 = at + (on1 ? n1 - m.x : 0);
                        if (!MR_IN_BOUNDS(a0 + (TZ - 1) * BW + 1, 2 * NB * BW * TZ, kSiteBpStaged)) on0 = false;
                        if (!MR_IN_BOUNDS(a1 + (TZ - 1) * BW + 1, 2 * NB * BW * TZ, kSiteBpStaged)) on1 = false;
                        staged_columns<MODE, TZ>(acc0, acc1, S.box + (on0 ? a0 : at), S.box + (on1 ? a1 : at), d0, d1, on0, on1, g0, P.tinc, nz);
                    } else if (m.y != kNothing) {
                        if (inside[0]) row(acc0, b, g, m, fy0);
                        if (inside[1]) row(acc1, b, g, m, fy1);
                    }
#pragma unroll
                    for (int k = 0; k + 1 < G; ++k) {
                        q_at[k] = q_at[k + 1];
                        q_d0[k] = q_d0[k + 1];
                        q_d1[k] = q_d1[k + 1];
                    }
                }
            }
        }
        // batch s+2's geometry complete and published; stage st and geometry buffer gb free
        tma::copy_wait_all();
        if (__syncthreads_or(failed)) break;
        if (s + 2 < nbatch) issue_batch(s + 2, st, gb == 0 ? 2 : gb - 1);
        if (s + 3 < nbatch) stage_geometry(s + 3, gb);
    }
    if (failed) {
        // copies still in flight: batch s (its wait expired) and batch s+1 when it was issued;
        // wait for them (bounded) before the block's shared memory is released
        const int st = s & 1;
        tma::mbar_wait(&S.bars[st], st ? phase1 : phase0);
        if (s + 1 < nbatch) tma::mbar_wait(&S.bars[st ^ 1], st ? phase0 : phase1);
    }
    auto store = [&](const float2 (&acc)[TZ / 2], float *c, bool in) {
        if (!in) return;
#pragma unroll
        for (int q = 0; q < TZ; q += 4) {
            if (vec) {
                *reinterpret_cast<float4 *>(c + q) = make_float4(acc[q / 2].x, acc[q / 2].y, acc[q / 2 + 1].x, acc[q / 2 + 1].y);
            } else if (q < zmax) {
                c[q] = acc[q / 2].x;
                c[q + 1] = acc[q / 2].y;
                c[q + 2] = acc[q / 2 + 1].x;
                c[q + 3] = acc[q / 2 + 1].y;
            }
        }
    };
    store(acc0, col[0], inside[0]);
    store(acc1, col[1], inside[1]);
}

// Projections of a list (all, or through an index) copied to rows of `pitch` floats, multiplied by
// their weights: what the TMA unit needs (16-byte row pitch and base) when the caller's rows are not.
__global__ void __launch_bounds__(256) k_repitch(const float *__restrict__ proj, const int32_t *__restrict__ index,
                                                 const float *__restrict__ weight, int nu, int nv, int pitch,
                                                 float *__restrict__ out)
{
    const int b = blockIdx.y;
    const size_t slab = index ? index[b] : b;
    const float *src = proj + slab * nv * static_cast<size_t>(nu);
    float *dst = out + static_cast<size_t>(b) * nv * pitch;
    for (int y = blockIdx.x; y < nv; y += gridDim.x)
        for (int x = threadIdx.x; x < nu; x += blockDim.x) {
            const float v = __ldg(src + static_cast<size_t>(y) * nu + x);
            dst[static_cast<size_t>(y) * pitch + x] = weight ? __fmul_rn(v, weight[b]) : v;
        }
}

template <int MODE, int TZ, int NW, int NB, int CTAS>
static mr_status launch_tile(PFN_cuTensorMapEncodeTiled enc, const Params &P, size_t nslabs, cudaStream_t s)
{
    CUtensorMap map;
    cuuint64_t dims[3] = {static_cast<cuuint64_t>(P.nu), static_cast<cuuint64_t>(P.nv), nslabs};
    cuuint64_t strides[2] = {static_cast<cuuint64_t>(P.pitch) * 4, static_cast<cuuint64_t>(P.pitch) * P.nv * 4};
    cuuint32_t box[3] = {static_cast<cuuint32_t>(BW), static_cast<cuuint32_t>(TZ), 1};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult cr = enc(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float *>(P.proj), dims, strides, box, estr,
                      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (cr != CUDA_SUCCESS) return fail(MR_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", static_cast<int>(cr));
    const size_t smem = Smem<TZ, NB>::bytes();
    dim3 grid(div_up(static_cast<size_t>(P.nu), TX), div_up(static_cast<size_t>(P.yend - P.ybegin), 2 * NW),
              div_up(static_cast<size_t>(P.nz4), TZ));
    const auto kernel = k_bp_par_staged<MODE, TZ, NW, NB, CTAS>;
    MR_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
    kernel<<<grid, 32 * NW, smem, s>>>(map, P);
    return check_launch("k_bp_par_staged");
}

// The tile by size. A thread's set-up per projection is shared by its TZ slices, so a slice costs
// 1 : 1.2 : 1.5 on 32-, 16- and 8-slice tiles (47.4, 56.9, 73.1 ms on 2048^2 x 64 slices from 1125
// projections), and the slices a tile holds beyond the volume's cost the same: 40 slices at 500^2
// from 500 projections take 1.49, 1.33 and 1.46 ms, 12 slices at 700^2 from 400 1.18, 0.69 and 0.92.
// A volume with fewer 16-slice tiles than SMs is bound by the latency of one tile's projection loop:
// 96^2 x 16 from 200 projections takes 136, 81 and 66 us (59 since two columns go at once). With fewer than
// half as many, 4-slice tiles are shorter still and batches of 32 projections put half the barriers in them:
// 49 us, and 128^2 x 8 from 180 53 -> 45 (16 projections per batch: 54 -> 52 before).
template <int MODE>
static mr_status launch_mode(PFN_cuTensorMapEncodeTiled enc, const Params &P, size_t nslabs, cudaStream_t s)
{
    const auto padded = [&](int tz) { return (P.nz4 + tz - 1) / tz * tz; };
    const int cost32 = 10 * padded(32), cost16 = 12 * padded(16), cost8 = 15 * padded(8);
    const size_t tiles16 = static_cast<size_t>(div_up(static_cast<size_t>(P.nu), TX)) *
                           div_up(static_cast<size_t>(P.yend - P.ybegin), 8) * div_up(static_cast<size_t>(P.nz4), 16);
    if (2 * tiles16 < 148) return launch_tile<MODE, 4, 4, 32, 4>(enc, P, nslabs, s);
    if (tiles16 < 148 || (cost8 < cost16 && cost8 < cost32)) return launch_tile<MODE, 8, 4, 16, 4>(enc, P, nslabs, s);
    if (cost16 < cost32) return launch_tile<MODE, 16, 4, 8, 4>(enc, P, nslabs, s);
    return launch_tile<MODE, 32, 8, 8, 2>(enc, P, nslabs, s);
}

static mr_status launch(int mode, const Params &P, size_t nslabs, cudaStream_t s)
{
    PFN_cuTensorMapEncodeTiled enc = tma::encode_fn();
    if (!enc) return MR_ERR_UNSUPPORTED;
    switch (mode) {
    case kLinear: return launch_mode<kLinear>(enc, P, nslabs, s);
    case kNearest: return launch_mode<kNearest>(enc, P, nslabs, s);
    case kTilt: return launch_mode<kTilt>(enc, P, nslabs, s);
    case kTiltSerial: return launch_mode<kTiltSerial>(enc, P, nslabs, s);
    default: return launch_mode<kTiltNearest>(enc, P, nslabs, s);
    }
}

} // namespace bp2

// Scratch of the re-pitched projections: projections go through in runs of about this many bytes.
constexpr size_t kRepitchBytes = size_t(1) << 30;

// Returns MR_ERR_UNSUPPORTED when staging does not apply (the caller uses the plain kernel).
mr_status bp_parallel_staged_launch(int variant, const float *proj_d, size_t nslabs, const float *weight_d,
                                    const int32_t *index_d, const float *sin_d, const float *cos_d,
                                    const float *startu_d, size_t nproj, size_t nu, size_t nv, const uint32_t *mask_d,
                                    int tilt, float toff, float tinc, size_t y_begin, size_t y_end, float *vol_d,
                                    cudaStream_t s)
{
    using namespace bp2;
    if (nv < 4 || nslabs == 0 || nu < static_cast<size_t>(BW)) return MR_ERR_UNSUPPORTED;
    const int mode = variant == MR_BP_NEAREST           ? (tilt ? kTiltNearest : kNearest)
                     : !tilt                            ? kLinear
                     : variant == MR_BP_MULTIPROJ_SERIAL ? kTiltSerial
                                                         : kTilt;
    Params P;
    P.mask = mask_d;
    P.vol = vol_d;
    P.nu = static_cast<int>(nu);
    P.nv = static_cast<int>(nv);
    P.nz4 = static_cast<int>((nv / 4) * 4);
    P.wait_limit = tma::g_batch_wait_limit.load();
    P.ybegin = static_cast<int>(y_begin);
    P.yend = static_cast<int>(y_end);
    P.toff = toff;
    P.tinc = tinc;
    P.neg_zero = -0.0f;
    if (!weight_d && nu % 4 == 0 && reinterpret_cast<uintptr_t>(proj_d) % 16 == 0) {
        P.proj = proj_d;
        P.index = index_d;
        P.sinv = sin_d;
        P.cosv = cos_d;
        P.startu = startu_d;
        P.nproj = static_cast<int>(nproj);
        P.pitch = P.nu;
        return launch(mode, P, nslabs, s);
    }
    // rows the TMA unit cannot address: re-pitched (and weighted) copies, a run of projections at a
    // time; the volume carries the sums from one run to the next, in projection order
    const size_t pitch = (nu + 3) / 4 * 4, per = pitch * nv * sizeof(float);
    const size_t run = std::min(nproj, std::max<size_t>(32, kRepitchBytes / per / 32 * 32));
    float *scratch = nullptr;
    if (run > 65535 || device_alloc(&scratch, run * per, s, "mr_bp_parallel: re-pitched projections") != MR_OK)
        return MR_ERR_UNSUPPORTED; // no room: the direct-load kernel needs none
    mr_status st = MR_OK;
    for (size_t a = 0; a < nproj && st == MR_OK; a += run) {
        const size_t n = std::min(run, nproj - a);
        k_repitch<<<dim3(static_cast<unsigned>(std::min<size_t>(nv, 64)), static_cast<unsigned>(n)), 256, 0, s>>>(
            index_d ? proj_d : proj_d + a * nu * nv, index_d ? index_d + a : nullptr, weight_d ? weight_d + a : nullptr,
            P.nu, P.nv, static_cast<int>(pitch), scratch);
        st = check_launch("k_repitch");
        P.proj = scratch;
        P.index = nullptr;
        P.sinv = sin_d + a;
        P.cosv = cos_d + a;
        P.startu = startu_d + a;
        P.nproj = static_cast<int>(n);
        P.pitch = static_cast<int>(pitch);
        if (st == MR_OK) st = launch(mode, P, n, s);
    }
    cudaFreeAsync(scratch, s);
    return st;
}

// mr_backproject.cu: the direct-load kernel for a range of volume rows
mr_status bp_parallel_rows(const void *proj_d, int dtype, const float *scale_d, const float *weight_d,
                           const int32_t *index_d, const float *sin_d, const float *cos_d, const float *startu_d,
                           size_t nproj, size_t nu, size_t nv, const uint32_t *mask_d, int correcttilt,
                           float tiltoffset, float tiltinc, size_t y_begin, size_t y_end, int variant, float *vol_d,
                           void *stream);

} // namespace mr

using namespace mr;

extern "C" mr_status mr_bp_parallel_variant(int variant, const void *proj_d, size_t nslabs, int dtype,
                                            const float *scale_d, const float *weight_d, const int32_t *index_d,
                                            const float *sin_d, const float *cos_d, const float *startu_d, size_t nproj,
                                            size_t nu, size_t nv, const uint32_t *mask_d, int correcttilt,
                                            float tiltoffset, float tiltinc, size_t y_begin, size_t y_end, float *vol_d,
                                            void *stream)
{
    MR_TRACE();
    if (!proj_d || !sin_d || !cos_d || !startu_d || !mask_d || !vol_d)
        return fail(MR_ERR_ARGUMENT, "mr_bp_parallel_variant: null pointer");
    if (variant < MR_BP_MULTIPROJ_PARALLEL || variant > MR_BP_NEAREST)
        return fail(MR_ERR_ARGUMENT, "mr_bp_parallel_variant: unknown backprojector variant %d", variant);
    if (y_begin > y_end || y_end > nu) return fail(MR_ERR_ARGUMENT, "mr_bp_parallel_variant: row range outside [0, nu]");
    // the serial MultiProjectionBP computes exactly what MultiProjectionBPparallel computes
    // unless the tilt is corrected or the slice count is not a multiple of 4 (its second
    // interpolation sample is then read from another place of its projection buffer)
    if (variant == MR_BP_MULTIPROJ_SERIAL && !correcttilt && (nv & 3) == 0) variant = MR_BP_MULTIPROJ_PARALLEL;
    const bool other_column = variant == MR_BP_MULTIPROJ_SERIAL && (nv & 3) != 0;
    if (!other_column && dtype == MR_F32 && nproj > 0 && nproj <= 0x7fffffff && nu >= 2 && nu <= 65536 &&
        nv <= 65536 && y_begin < y_end) {
        if (!index_d && nslabs < nproj) {
            // with tilt correction a caller need not count the slabs: they are the list's
            if (!correcttilt) return fail(MR_ERR_ARGUMENT, "mr_bp_parallel_variant: nslabs below nproj");
            nslabs = nproj;
        }
        mr_status st = bp_parallel_staged_launch(variant, static_cast<const float *>(proj_d), nslabs, weight_d, index_d,
                                                 sin_d, cos_d, startu_d, nproj, nu, nv, mask_d, correcttilt, tiltoffset,
                                                 tiltinc, y_begin, y_end, vol_d, as_stream(stream));
        if (st != MR_ERR_UNSUPPORTED) return st;
    }
    return bp_parallel_rows(proj_d, dtype, scale_d, weight_d, index_d, sin_d, cos_d, startu_d, nproj, nu, nv, mask_d,
                            correcttilt, tiltoffset, tiltinc, y_begin, y_end, variant, vol_d, stream);
}

extern "C" mr_status mr_bp_parallel_rows(const void *proj_d, size_t nslabs, int dtype, const float *scale_d,
                                         const float *weight_d, const int32_t *index_d, const float *sin_d,
                                         const float *cos_d, const float *startu_d, size_t nproj, size_t nu, size_t nv,
                                         const uint32_t *mask_d, int correcttilt, float tiltoffset, float tiltinc,
                                         size_t y_begin, size_t y_end, float *vol_d, void *stream)
{
    MR_TRACE();
    return mr_bp_parallel_variant(MR_BP_MULTIPROJ_PARALLEL, proj_d, nslabs, dtype, scale_d, weight_d, index_d, sin_d,
                                  cos_d, startu_d, nproj, nu, nv, mask_d, correcttilt, tiltoffset, tiltinc, y_begin,
                                  y_end, vol_d, stream);
}

extern "C" mr_status mr_bp_parallel_staged(const void *proj_d, size_t nslabs, int dtype, const float *scale_d,
                                           const float *weight_d, const int32_t *index_d, const float *sin_d,
                                           const float *cos_d, const float *startu_d, size_t nproj, size_t nu, size_t nv,
                                           const uint32_t *mask_d, int correcttilt, float tiltoffset, float tiltinc,
                                           float *vol_d, void *stream)
{
    MR_TRACE();
    return mr_bp_parallel_rows(proj_d, nslabs, dtype, scale_d, weight_d, index_d, sin_d, cos_d, startu_d, nproj, nu, nv,
                               mask_d, correcttilt, tiltoffset, tiltinc, 0, nu, vol_d, stream);
}
