// Direct-sum gravity of few particles (sm_100a): the whole j-range of a group of i-particles in one
// block, no split partials and no finish launch.
//
// direct.cu's kernels give a block 256 to 512 i-particles and one or more j-tiles of 256, so N =
// 2,048 makes 32 blocks for 148 SMs and every evaluation a second launch that adds the splits.
// Here a block holds IG = 4 .. 32 i-particles and all j: its 16 warps take 32 j each of every 512,
// and the 32 / IG lanes that share an i-particle take every (32 / IG)-th of those. Each warp stages
// its own 32 j in shared memory (prefetched, no block barrier), then the lanes' sums meet by
// shuffles, the warps' in shared memory, in a fixed order, FP64; the leapfrog epilogue follows in
// the same launch. IG is the largest that still gives two thirds of the SMs a block. It is taken
// while blocks of 32 fit one per SM (4,736 particles on 148): with a second wave the ordered
// kernels are faster (N = 6,000 FP32 27 us against 21, FP64 74 against 58).
//
// FP32 pairs are those of direct_f32jp_kernel (one i against two j per paired instruction),
// MIXED those of direct_f32_kernel (a chunk's sum in FP32, the chunks' in FP64), FP64 those of
// direct_f64_kernel.
//
// Bound: latency up to N = 2,048, above the FP32 pipe (66% busy at 4,096) or the FP64 pipe. Per step
// on B200, split kernels and finish -> here, us: FP32 N = 512 18.3 -> 3.0, 1,024 19.5 -> 3.5, 2,048
// 20.0 -> 5.3, 4,096 15.1 -> 12.0; MIXED 2,048 14.0 -> 7.3, 4,096 22.1 -> 19.0; FP64 1,024 71.7 ->
// 4.7, 4,096 49.5 -> 27.1.
#include "direct_epi.cuh"
#include "kernels.cuh"

namespace rrg {
namespace {

constexpr int kWarps = 16;
constexpr int kThreads = 32 * kWarps;

template <typename R>
struct SmallParams {
    const V4<R>* posm;
    const V4<float>* poslo;  // MIXED
    const R* hsoft;
    R uniform_h, uniform_m;
    int n;
    EpiDev<R> epi;
};

// Sums of a lane over the j-subsets that share its i-particle (lanes IG apart), fixed order.
template <int IG>
__device__ __forceinline__ double over_lanes(double v) {
#pragma unroll
    for (int o = 16; o >= IG; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

template <int PREC, int IG, bool USOFT, bool POT, bool UMASS, typename R>
__global__ void __launch_bounds__(kThreads) direct_small_kernel(const SmallParams<R> p) {
    constexpr bool MIXED = PREC == RRG_PREC_MIXED, F64 = PREC == RRG_PREC_FP64;
    // a warp's 32 j: FP32 (x0, x1, y0, y1) and (z0, z1, m0, m1) per pair; else (x, y, z, m) per j
    __shared__ V4<R> s_a[kWarps][32];
    __shared__ V4<float> s_lo[MIXED ? kWarps : 1][32];
    __shared__ R s_h[USOFT ? 1 : kWarps][32];
    __shared__ double s_sum[kWarps][32][POT ? 4 : 3];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int subs = 32 / IG;
    const int sub = lane / IG;
    const int i = blockIdx.x * IG + (lane & (IG - 1));
    const R pad = F64 ? R(1e150) : R(kDirectPad);
    V4<R> pi = v4<R>(R(0), R(0), R(0), R(0));
    V4<float> li = v4<float>(0.f, 0.f, 0.f, 0.f);
    R hi = p.uniform_h;
    if (i < p.n) {
        pi = p.posm[i];
        if constexpr (!USOFT) hi = pair_soft(p.hsoft[i]);
        if constexpr (MIXED) li = p.poslo[i];
    }
    const R hh = USOFT ? hi + hi : hi;
    V4<R> nxt;
    V4<float> nxl = v4<float>(0.f, 0.f, 0.f, 0.f);
    R nxh;
    auto fetch = [&](int j) {
        nxt = v4<R>(pad, pad, pad, R(0));
        nxl = v4<float>(0.f, 0.f, 0.f, 0.f);
        nxh = R(1);
        if (j < p.n) {
            nxt = p.posm[j];
            if constexpr (!USOFT) nxh = p.hsoft[j];
            if constexpr (MIXED) nxl = p.poslo[j];
        }
    };
    double sx = 0, sy = 0, sz = 0, sp = 0;           // MIXED and FP64 sums
    float2 ax = make_float2(0.f, 0.f), ay = ax, az = ax, ap = ax;  // FP32: even and odd j
    fetch(tid);
    for (int j0 = 0; j0 < p.n; j0 += kThreads) {
        __syncwarp();
        if constexpr (!F64 && !MIXED) {
            float* const f = reinterpret_cast<float*>(s_a[warp]) + 8 * (lane >> 1) + (lane & 1);
            f[0] = nxt.x;
            f[2] = nxt.y;
            f[4] = nxt.z;
            f[6] = nxt.w;
        } else {
            s_a[warp][lane] = nxt;
        }
        if constexpr (MIXED) s_lo[warp][lane] = nxl;
        if constexpr (!USOFT) s_h[warp][lane] = nxh;
        __syncwarp();
        if (j0 + kThreads < p.n) fetch(j0 + kThreads + tid);
        if (j0 + 32 * warp >= p.n) continue;  // (no j of this chunk for the warp)
        if constexpr (!F64 && !MIXED) {
            const float2 nx = make_float2(-pi.x, -pi.x), ny = make_float2(-pi.y, -pi.y),
                         nz = make_float2(-pi.z, -pi.z), h2 = make_float2(hh, hh);
            // U pairs of j at a time, stage by stage: their chains overlap
            constexpr int U = 16 / subs < 4 ? 16 / subs : 4;
#pragma unroll
            for (int t = 0; t < 16 / subs; t += U) {
                float2 dx[U], dy[U], dz[U], m[U], r2[U];
#pragma unroll
                for (int k = 0; k < U; ++k) {
                    const int q = (t + k) * subs + sub;
                    const V4<R> xy = s_a[warp][2 * q], zm = s_a[warp][2 * q + 1];
                    dx[k] = __fadd2_rn(make_float2(xy.x, xy.y), nx);
                    dy[k] = __fadd2_rn(make_float2(xy.z, xy.w), ny);
                    dz[k] = __fadd2_rn(make_float2(zm.x, zm.y), nz);
                    m[k] = make_float2(zm.z, zm.w);
                    r2[k] = h2;
                    if constexpr (!USOFT)
                        r2[k] = __fadd2_rn(h2, *reinterpret_cast<const float2*>(&s_h[warp][2 * q]));
                }
#pragma unroll
                for (int k = 0; k < U; ++k) r2[k] = __ffma2_rn(dx[k], dx[k], r2[k]);
#pragma unroll
                for (int k = 0; k < U; ++k) r2[k] = __ffma2_rn(dy[k], dy[k], r2[k]);
#pragma unroll
                for (int k = 0; k < U; ++k) r2[k] = __ffma2_rn(dz[k], dz[k], r2[k]);
#pragma unroll
                for (int k = 0; k < U; ++k) {
                    const float2 inv = make_float2(rsqrt_sfu(r2[k].x), rsqrt_sfu(r2[k].y));
                    const float2 minv = UMASS ? inv : __fmul2_rn(m[k], inv);
                    const float2 kk = __fmul2_rn(minv, __fmul2_rn(inv, inv));
                    ax = __ffma2_rn(dx[k], kk, ax);
                    ay = __ffma2_rn(dy[k], kk, ay);
                    az = __ffma2_rn(dz[k], kk, az);
                    if constexpr (POT) ap = __fadd2_rn(ap, minv);
                }
            }
        } else if constexpr (MIXED) {
            float tx = 0.f, ty = 0.f, tz = 0.f, tp = 0.f;
#pragma unroll 8
            for (int t = 0; t < 32 / subs; ++t) {
                const int q = t * subs + sub;
                const V4<R> pj = s_a[warp][q];
                const V4<float> lj = s_lo[warp][q];
                const float dx = (pj.x - pi.x) + (lj.x - li.x), dy = (pj.y - pi.y) + (lj.y - li.y),
                            dz = (pj.z - pi.z) + (lj.z - li.z);
                const float s = USOFT ? hh : hh + s_h[warp][q];
                const float inv = rsqrt_sfu(fmaf(dz, dz, fmaf(dy, dy, fmaf(dx, dx, s))));
                const float minv = pj.w * inv;
                const float kk = minv * (inv * inv);
                tx = fmaf(dx, kk, tx);
                ty = fmaf(dy, kk, ty);
                tz = fmaf(dz, kk, tz);
                if constexpr (POT) tp += minv;
            }
            sx += tx;
            sy += ty;
            sz += tz;
            sp += tp;
        } else {
#pragma unroll 4
            for (int t = 0; t < 32 / subs; ++t) {
                const int q = t * subs + sub;
                const V4<R> pj = s_a[warp][q];
                const double dx = pj.x - pi.x, dy = pj.y - pi.y, dz = pj.z - pi.z;
                const double s = USOFT ? hh : hh + s_h[warp][q];
                const double inv = rsqrt_pair(dx * dx + dy * dy + dz * dz + s);
                const double kk = pj.w * (inv * inv * inv);
                sx += dx * kk;
                sy += dy * kk;
                sz += dz * kk;
                if constexpr (POT) sp += pj.w * inv;
            }
        }
    }
    if constexpr (!F64 && !MIXED) {
        sx = static_cast<double>(ax.x) + ax.y;
        sy = static_cast<double>(ay.x) + ay.y;
        sz = static_cast<double>(az.x) + az.y;
        sp = static_cast<double>(ap.x) + ap.y;
    }
    sx = over_lanes<IG>(sx);
    sy = over_lanes<IG>(sy);
    sz = over_lanes<IG>(sz);
    if constexpr (POT) sp = over_lanes<IG>(sp);
    if (lane < IG) {
        s_sum[warp][lane][0] = sx;
        s_sum[warp][lane][1] = sy;
        s_sum[warp][lane][2] = sz;
        if constexpr (POT) s_sum[warp][lane][3] = sp;
    }
    __syncthreads();
    if (tid >= IG || i >= p.n) return;
    double t[4] = {0, 0, 0, 0};
#pragma unroll
    for (int w = 0; w < kWarps; ++w)
#pragma unroll
        for (int c = 0; c < (POT ? 4 : 3); ++c) t[c] += s_sum[w][lane][c];
    const double um = UMASS ? static_cast<double>(p.uniform_m) : 1.0;
    apply_epi<R, MIXED>(p.epi, i, static_cast<R>(um * t[0]), static_cast<R>(um * t[1]),
                        static_cast<R>(um * t[2]), static_cast<R>(-um * t[3]), POT, p.posm,
                        p.poslo);
}

template <int PREC, int IG, bool UMASS, typename R>
void dispatch_ig(bool usoft, bool pot, const SmallParams<R>& p, cudaStream_t s) {
    auto go = [&](auto* k) {
        k<<<div_up(p.n, IG), kThreads, 0, s>>>(p);
        RRG_LAUNCHED();
    };
    if (usoft) {
        if (pot) go(direct_small_kernel<PREC, IG, true, true, UMASS, R>);
        else go(direct_small_kernel<PREC, IG, true, false, UMASS, R>);
    } else {
        if (pot) go(direct_small_kernel<PREC, IG, false, true, UMASS, R>);
        else go(direct_small_kernel<PREC, IG, false, false, UMASS, R>);
    }
}

template <int PREC, bool UMASS, typename R>
void dispatch(int ig, bool usoft, bool pot, const SmallParams<R>& p, cudaStream_t s) {
    if (ig == 32) dispatch_ig<PREC, 32, UMASS>(usoft, pot, p, s);
    else if (ig == 16) dispatch_ig<PREC, 16, UMASS>(usoft, pot, p, s);
    else if (ig == 8) dispatch_ig<PREC, 8, UMASS>(usoft, pot, p, s);
    else dispatch_ig<PREC, 4, UMASS>(usoft, pot, p, s);
}

}  // namespace

bool direct_small_applies(int64_t n, int sms) { return n <= 32ll * sms; }

void launch_direct_small(const DirectLaunch& L, int sms) {
    int ig = 32;
    while (ig > 4 && 3ll * div_up(L.n, ig) < 2ll * sms) ig /= 2;
    auto fill = [&](auto& p) {
        using R = std::remove_const_t<std::remove_reference_t<decltype(p.uniform_h)>>;
        p.posm = static_cast<const V4<R>*>(L.posm);
        p.poslo = static_cast<const V4<float>*>(L.poslo);
        p.hsoft = static_cast<const R*>(L.hsoft);
        p.uniform_h = pair_soft(static_cast<R>(L.uniform_hsoft));
        p.uniform_m = static_cast<R>(L.uniform_mass);
        p.n = static_cast<int>(L.n);
        p.epi = make_epi<R>(L.epi);
    };
    const bool usoft = L.hsoft == nullptr;
    if (L.prec == RRG_PREC_FP64) {
        SmallParams<double> p{};
        fill(p);
        dispatch<RRG_PREC_FP64, false>(ig, usoft, L.want_pot, p, L.stream);
        return;
    }
    SmallParams<float> p{};
    fill(p);
    if (L.prec == RRG_PREC_MIXED) {
        RRG_REQUIRE(L.poslo != nullptr, RRG_ERR_INVALID,
                    "direct sum: MIXED precision needs the low position parts");
        dispatch<RRG_PREC_MIXED, false>(ig, usoft, L.want_pot, p, L.stream);
    } else if (L.uniform_mass >= 0.0) {
        dispatch<RRG_PREC_FP32, true>(ig, usoft, L.want_pot, p, L.stream);
    } else {
        dispatch<RRG_PREC_FP32, false>(ig, usoft, L.want_pot, p, L.stream);
    }
}

}  // namespace rrg
