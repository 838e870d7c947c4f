// Direct-sum gravity with every unordered pair evaluated once (sm_100a).
//
// direct.cu's kernels evaluate each ordered pair (nbody.cu:19-114): 11 FMA-pipe operations per
// interaction, and the pipe is the bound (81% busy). d_ij, its length and the reciprocal cube are
// the same for (i, j) and (j, i) up to the sign of d_ij, so one evaluation serves both particles:
// 3 differences, 3 multiply-adds for |d|^2, the reciprocal square root and its cube (2), then 3
// multiply-adds for i and 3 for j: 14 operations for two interactions instead of 22 (equal
// masses). The FP64 reciprocal square root alone is most of a pair in that precision.
//
// Work: the particles fall into i-tiles of A = 256 G (G per thread, in registers) and j-tiles of
// 256. A unit is (i-tile a, j-tile t), t at or above a's own: its own tiles (t in a) are
// evaluated for i alone over ordered pairs (self pair included, as the reference), the tiles
// above for both sides. The units, listed a by a, are eight rounds of 32 j per warp each, and the
// rounds are cut into one equal run per resident block (they cost about the same: 11 operations
// per ordered pair against 14 for an unordered one).
//
// j sums: in step s of a chunk of 32 j a lane takes j = (lane + s) mod 32 and adds its G
// particles' terms to the sums that travel along the warp with that j (one shuffle per sum and
// step, over G pairs); after 32 steps lane l holds the warp's sums of j = l. The eight warps of a
// block start at different chunks of the tile and move on together (a barrier per chunk), so each
// chunk's shared accumulator is added to by one warp at a time in a fixed order: no atomics, the
// same bits every run. A unit writes its j sums to slot js[a][j] (a run that starts inside a unit
// writes its part of that unit to js2[block]); a block writes its i sums when it leaves an i-tile,
// to slot is[block - first block of the tile][i]. direct_sym_finish adds a particle's slots in
// order in FP64 and applies the leapfrog epilogue.
//
// Sums: G terms x 32 steps per travelling sum, 256 terms per i-tile sum, both then added into
// shared memory (FP32; FP64 in MIXED and FP64), the slots in FP64: shorter FP32 chains than the
// tile sums of direct.cu.
#include <algorithm>

#include "direct_epi.cuh"
#include "kernels.cuh"
#include "pair_plan.cuh"
#include "wave_cells.cuh"

namespace rrg {
namespace {

constexpr int kBS = kDirectThreads;
constexpr int kWarps = kPairWarps;

template <typename R, typename S>
struct SymParams {
    SymPlan plan;
    const V4<R>* posm;
    const V4<float>* poslo;  // MIXED
    const R* hsoft;
    R uniform_h;
    R uniform_m;
    V4<S>* js;   // [tiles - 1][n]
    V4<S>* is;   // [islots][n]
    V4<S>* js2;  // [blocks][kBS]
};

// ----------------------------------------------------------------------------------------------
// FP32 and MIXED: G2 packed pairs of i-particles per thread on the paired FP32 instructions
// (i = tile + (2 g + e) 256 + tid in half e of pair g). The pair arithmetic is direct_f32x2_kernel's
// (MIXED: direct_f32_kernel's, both halves of the double-float positions in the differences).
// UMASS: every mass is uniform_m, applied to the finished sums. The travelling sums enter the
// first pair's multiply-add, so a step costs one FP32 addition per sum beside the pairs.
//
// Bound: the FP32 pipe (74% of the issue peak at N = 65,536; shared memory 19%). Per evaluation
// with its finish on B200, before (direct.cu) -> here, us: FP32 equal masses N = 16,384 109 -> 88,
// 65,536 1572 -> 1147 (3.75e12 pairs/s); unequal 65,536 1805 -> 1468; MIXED 30,011 666 -> 454.
// With a first form that added the travelling sums after the step: 1222 at 65,536.
// ----------------------------------------------------------------------------------------------
template <int G2, bool USOFT, bool POT, bool UMASS, bool MIXED>
struct Sym32 {
    using S = typename std::conditional<MIXED, double, float>::type;  // shared and slot sums
    static constexpr int NV = POT ? 4 : 3;
    static constexpr size_t smem = sizeof(S) * NV * 2 * G2 * kBS     // i sums
                                   + sizeof(V4<S>) * kBS             // j sums
                                   + sizeof(float4) * kBS            // x, y, z, m
                                   + (MIXED ? sizeof(float4) * kBS : 0)
                                   + (USOFT ? 0 : sizeof(float) * kBS);
};

template <int G2, bool USOFT, bool POT, bool UMASS, bool MIXED>
__global__ void __launch_bounds__(kBS, 2)
    direct_sym32_kernel(const SymParams<float, typename Sym32<G2, USOFT, POT, UMASS, MIXED>::S> p) {
    using K = Sym32<G2, USOFT, POT, UMASS, MIXED>;
    using S = typename K::S;
    constexpr int NV = K::NV;
    extern __shared__ __align__(32) unsigned char sm_raw[];
    V4<S>* const s_j = reinterpret_cast<V4<S>*>(sm_raw);          // [kBS]
    float4* const s_p = reinterpret_cast<float4*>(s_j + kBS);     // [kBS]
    float4* const s_lo = s_p + kBS;                               // [kBS] (MIXED)
    S* const s_i = reinterpret_cast<S*>(s_lo + (MIXED ? kBS : 0));  // [2 G2][NV][kBS]
    float* const s_h = reinterpret_cast<float*>(s_i + 2 * G2 * NV * kBS);  // [kBS]

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const SymPlan& pl = p.plan;
    const int64_t q0 = pl.run_start(blockIdx.x), q1 = pl.run_start(blockIdx.x + 1);  // rounds
    const int64_t u0 = q0 / kWarps, u1 = (q1 + kWarps - 1) / kWarps;                  // units
    int a = 0;
    while (a + 1 < pl.tiles && pl.first_unit(a + 1) <= u0) ++a;

    float2 nx[G2], ny[G2], nz[G2], hs[G2], mi[G2];
    float2 lx[G2], ly[G2], lz[G2];
    auto load_i = [&]() {
#pragma unroll
        for (int g = 0; g < G2; ++g) {
            float v[2][5], l[2][3];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int64_t i = static_cast<int64_t>(a) * (kBS * 2 * G2) + (2 * g + e) * kBS + tid;
                V4<float> pi = v4<float>(kDirectPad, kDirectPad, kDirectPad, 0.f);
                V4<float> li = v4<float>(0.f, 0.f, 0.f, 0.f);
                v[e][4] = USOFT ? 0.f : 1.f;
                if (i < pl.n) {
                    pi = p.posm[i];
                    if constexpr (!USOFT) v[e][4] = p.hsoft[i];
                    if constexpr (MIXED) li = p.poslo[i];
                }
                v[e][0] = pi.x;
                v[e][1] = pi.y;
                v[e][2] = pi.z;
                v[e][3] = pi.w;
                l[e][0] = li.x;
                l[e][1] = li.y;
                l[e][2] = li.z;
            }
            nx[g] = make_float2(-v[0][0], -v[1][0]);
            ny[g] = make_float2(-v[0][1], -v[1][1]);
            nz[g] = make_float2(-v[0][2], -v[1][2]);
            mi[g] = make_float2(v[0][3], v[1][3]);
            hs[g] = USOFT ? dup2(p.uniform_h + p.uniform_h) : make_float2(v[0][4], v[1][4]);
            if constexpr (MIXED) {
                lx[g] = make_float2(-l[0][0], -l[1][0]);
                ly[g] = make_float2(-l[0][1], -l[1][1]);
                lz[g] = make_float2(-l[0][2], -l[1][2]);
            }
#pragma unroll
            for (int e = 0; e < 2; ++e)
#pragma unroll
                for (int c = 0; c < NV; ++c) s_i[((2 * g + e) * NV + c) * kBS + tid] = S(0);
        }
    };
    auto flush_i = [&]() {
        const int slot = static_cast<int>(blockIdx.x) - pl.first_block(a);
        const S um = UMASS ? static_cast<S>(p.uniform_m) : S(1);
#pragma unroll
        for (int q = 0; q < 2 * G2; ++q) {
            const int64_t i = static_cast<int64_t>(a) * (kBS * 2 * G2) + q * kBS + tid;
            if (i >= pl.n) continue;
            const S* const v = s_i + q * NV * kBS + tid;
            p.is[static_cast<int64_t>(slot) * pl.n + i] =
                v4<S>(um * v[0], um * v[kBS], um * v[2 * kBS], POT ? um * v[(NV - 1) * kBS] : S(0));
        }
    };

    V4<float> nxt, nxl;
    float nxh;
    auto fetch = [&](int64_t t) {
        const int64_t j = t * kBS + tid;
        nxt = v4<float>(kDirectPad, kDirectPad, kDirectPad, 0.f);
        nxl = v4<float>(0.f, 0.f, 0.f, 0.f);
        nxh = 1.f;
        if (j < pl.n) {
            nxt = p.posm[j];
            if constexpr (!USOFT) nxh = p.hsoft[j];
            if constexpr (MIXED) nxl = p.poslo[j];
        }
    };

    float2 tx[G2], ty[G2], tz[G2], tp[G2];
    // the pair of two i (pair g) and one j: d, 1 / |d| (softened)
    auto geometry = [&](int g, const float4& pj, const float4& lj, float hj, float2& dx,
                        float2& dy, float2& dz) -> float2 {
        dx = __fadd2_rn(dup2(pj.x), nx[g]);
        dy = __fadd2_rn(dup2(pj.y), ny[g]);
        dz = __fadd2_rn(dup2(pj.z), nz[g]);
        if constexpr (MIXED) {
            dx = __fadd2_rn(dx, __fadd2_rn(dup2(lj.x), lx[g]));
            dy = __fadd2_rn(dy, __fadd2_rn(dup2(lj.y), ly[g]));
            dz = __fadd2_rn(dz, __fadd2_rn(dup2(lj.z), lz[g]));
        }
        const float2 s = USOFT ? hs[g] : __fadd2_rn(hs[g], dup2(hj));
        const float2 r2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __ffma2_rn(dx, dx, s)));
        return make_float2(rsqrt_sfu(r2.x), rsqrt_sfu(r2.y));
    };

    pdl_next();  // (the finish may start and wait)
    load_i();
    int64_t base = pl.first_unit(a);
    fetch(static_cast<int64_t>(a) * pl.g + (u0 - base));
    for (int64_t u = u0; u < u1; ++u) {
        if (u >= base + (pl.nt - static_cast<int64_t>(a) * pl.g)) {
            flush_i();
            ++a;
            base = pl.first_unit(a);
            load_i();
        }
        const int64_t t = static_cast<int64_t>(a) * pl.g + (u - base);
        const int r0 = u == u0 ? static_cast<int>(q0 - u0 * kWarps) : 0;
        const int r1 = u + 1 == u1 ? static_cast<int>(q1 - u * kWarps) : kWarps;
        __syncthreads();  // the tile before is done with (its j sums are stored)
        s_p[tid] = make_float4(nxt.x, nxt.y, nxt.z, nxt.w);
        if constexpr (MIXED) s_lo[tid] = make_float4(nxl.x, nxl.y, nxl.z, 0.f);
        if constexpr (!USOFT) s_h[tid] = nxh;
        s_j[tid] = v4<S>(S(0), S(0), S(0), S(0));
        __syncthreads();
        if (u + 1 < u1) {
            const bool same = u + 1 < base + (pl.nt - static_cast<int64_t>(a) * pl.g);
            fetch(same ? t + 1 : static_cast<int64_t>(a + 1) * pl.g);
        }
#pragma unroll
        for (int g = 0; g < G2; ++g) tx[g] = ty[g] = tz[g] = tp[g] = make_float2(0.f, 0.f);
        const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
        if (t < static_cast<int64_t>(a + 1) * pl.g) {
            // a's own tiles: i alone, every ordered pair
#pragma unroll 4
            for (int k = 32 * r0; k < 32 * r1; ++k) {
                const float4 pj = s_p[k];
                const float4 lj = MIXED ? s_lo[k] : zero4;
                const float hj = USOFT ? 0.f : s_h[k];
#pragma unroll
                for (int g = 0; g < G2; ++g) {
                    float2 dx, dy, dz;
                    const float2 inv = geometry(g, pj, lj, hj, dx, dy, dz);
                    const float2 minv = UMASS ? inv : __fmul2_rn(dup2(pj.w), inv);
                    const float2 kk = __fmul2_rn(minv, __fmul2_rn(inv, inv));
                    tx[g] = __ffma2_rn(dx, kk, tx[g]);
                    ty[g] = __ffma2_rn(dy, kk, ty[g]);
                    tz[g] = __ffma2_rn(dz, kk, tz[g]);
                    if constexpr (POT) tp[g] = __fadd2_rn(tp[g], minv);
                }
            }
        } else {
            for (int r = r0; r < r1; ++r) {
                const int c = ((warp + r) & (kWarps - 1)) * 32;
                float cx = 0.f, cy = 0.f, cz = 0.f, cp = 0.f;
                const int from = (lane + 1) & 31;
#pragma unroll 4
                for (int s = 0; s < 32; ++s) {
                    const int k = c + ((lane + s) & 31);
                    const float4 pj = s_p[k];
                    const float4 lj = MIXED ? s_lo[k] : zero4;
                    const float hj = USOFT ? 0.f : s_h[k];
                    float2 jx = make_float2(cx, 0.f), jy = make_float2(cy, 0.f);
                    float2 jz = make_float2(cz, 0.f), jp = make_float2(cp, 0.f);
#pragma unroll
                    for (int g = 0; g < G2; ++g) {
                        float2 dx, dy, dz;
                        const float2 inv = geometry(g, pj, lj, hj, dx, dy, dz);
                        const float2 inv2 = __fmul2_rn(inv, inv);
                        float2 ki, kj, pi = inv, pjv = inv;
                        if constexpr (UMASS) {
                            ki = kj = __fmul2_rn(inv, inv2);
                        } else {
                            pi = __fmul2_rn(dup2(pj.w), inv);
                            pjv = __fmul2_rn(mi[g], inv);
                            ki = __fmul2_rn(pi, inv2);
                            kj = __fmul2_rn(pjv, inv2);
                        }
                        tx[g] = __ffma2_rn(dx, ki, tx[g]);
                        ty[g] = __ffma2_rn(dy, ki, ty[g]);
                        tz[g] = __ffma2_rn(dz, ki, tz[g]);
                        if constexpr (POT) tp[g] = __fadd2_rn(tp[g], pi);
                        jx = __ffma2_rn(dx, kj, jx);
                        jy = __ffma2_rn(dy, kj, jy);
                        jz = __ffma2_rn(dz, kj, jz);
                        if constexpr (POT) jp = __fadd2_rn(jp, pjv);
                    }
                    cx = __shfl_sync(0xffffffffu, half_sum(jx), from);
                    cy = __shfl_sync(0xffffffffu, half_sum(jy), from);
                    cz = __shfl_sync(0xffffffffu, half_sum(jz), from);
                    if constexpr (POT) cp = __shfl_sync(0xffffffffu, half_sum(jp), from);
                }
                V4<S> v = s_j[c + lane];
                v.x += static_cast<S>(cx);
                v.y += static_cast<S>(cy);
                v.z += static_cast<S>(cz);
                if constexpr (POT) v.w += static_cast<S>(cp);
                s_j[c + lane] = v;
                __syncthreads();  // the next warp to add to this chunk comes after
            }
            const int64_t j = t * kBS + tid;
            if (j < pl.n) {
                const S um = UMASS ? static_cast<S>(p.uniform_m) : S(1);
                const V4<S> v = s_j[tid];
                // (d points from i to j: j is pulled along -d)
                V4<S>* const to = r0 == 0 ? p.js + static_cast<int64_t>(a) * pl.n + j
                                          : p.js2 + static_cast<int64_t>(blockIdx.x) * kBS + tid;
                *to =
                    v4<S>(-um * v.x, -um * v.y, -um * v.z, POT ? um * v.w : S(0));
            }
        }
#pragma unroll
        for (int g = 0; g < G2; ++g) {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                S* const v = s_i + (2 * g + e) * NV * kBS + tid;
                v[0] += static_cast<S>(e ? tx[g].y : tx[g].x);
                v[kBS] += static_cast<S>(e ? ty[g].y : ty[g].x);
                v[2 * kBS] += static_cast<S>(e ? tz[g].y : tz[g].x);
                if constexpr (POT) v[(NV - 1) * kBS] += static_cast<S>(e ? tp[g].y : tp[g].x);
            }
        }
    }
    flush_i();
}

// ----------------------------------------------------------------------------------------------
// FP64: G i-particles per thread. The reciprocal square root is rsqrt_pair instead of 1 / sqrt,
// whose square root and division each cost a Newton sequence on the FP64 pipe, the bound of this
// kernel; without a branch the pairs of a thread overlap. Per evaluation on B200, ordered pairs with
// 1 / sqrt -> each pair once with CUDA's rsqrt -> with rsqrt_pair, us: N = 8,192 177 -> 89 -> 84;
// 20,011 869 -> 400 -> 381; 32,768 2211 -> 982 -> 940 (relative error of the forces against 64-bit
// sums at 20,011 4.0e-16 -> 3.5e-16).
// ----------------------------------------------------------------------------------------------
template <int G, bool USOFT, bool POT>
struct Sym64 {
    static constexpr int NV = POT ? 4 : 3;
    static constexpr size_t smem = sizeof(double) * NV * G * kBS + 2 * sizeof(V4<double>) * kBS +
                                   (USOFT ? 0 : sizeof(double) * kBS);
};

template <int G, bool USOFT, bool POT>
__global__ void __launch_bounds__(kBS, 2) direct_sym64_kernel(const SymParams<double, double> p) {
    constexpr int NV = Sym64<G, USOFT, POT>::NV;
    extern __shared__ __align__(32) unsigned char sm_raw[];
    V4<double>* const s_j = reinterpret_cast<V4<double>*>(sm_raw);    // [kBS]
    V4<double>* const s_p = s_j + kBS;                                // [kBS]
    double* const s_i = reinterpret_cast<double*>(s_p + kBS);         // [G][NV][kBS]
    double* const s_h = s_i + G * NV * kBS;                           // [kBS]

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const SymPlan& pl = p.plan;
    const int64_t q0 = pl.run_start(blockIdx.x), q1 = pl.run_start(blockIdx.x + 1);  // rounds
    const int64_t u0 = q0 / kWarps, u1 = (q1 + kWarps - 1) / kWarps;                  // units
    int a = 0;
    while (a + 1 < pl.tiles && pl.first_unit(a + 1) <= u0) ++a;

    double xi[G], yi[G], zi[G], hi[G], mi[G];
    auto load_i = [&]() {
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const int64_t i = static_cast<int64_t>(a) * (kBS * G) + g * kBS + tid;
            V4<double> pi = v4<double>(1e150, 1e150, 1e150, 0.0);
            hi[g] = USOFT ? p.uniform_h + p.uniform_h : 1.0;
            if (i < pl.n) {
                pi = p.posm[i];
                if constexpr (!USOFT) hi[g] = pair_soft(p.hsoft[i]);
            }
            xi[g] = pi.x;
            yi[g] = pi.y;
            zi[g] = pi.z;
            mi[g] = pi.w;
#pragma unroll
            for (int c = 0; c < NV; ++c) s_i[(g * NV + c) * kBS + tid] = 0.0;
        }
    };
    auto flush_i = [&]() {
        const int slot = static_cast<int>(blockIdx.x) - pl.first_block(a);
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const int64_t i = static_cast<int64_t>(a) * (kBS * G) + g * kBS + tid;
            if (i >= pl.n) continue;
            const double* const v = s_i + g * NV * kBS + tid;
            p.is[static_cast<int64_t>(slot) * pl.n + i] =
                v4<double>(v[0], v[kBS], v[2 * kBS], POT ? v[(NV - 1) * kBS] : 0.0);
        }
    };
    V4<double> nxt;
    double nxh;
    auto fetch = [&](int64_t t) {
        const int64_t j = t * kBS + tid;
        nxt = v4<double>(1e150, 1e150, 1e150, 0.0);
        nxh = 1.0;
        if (j < pl.n) {
            nxt = p.posm[j];
            if constexpr (!USOFT) nxh = p.hsoft[j];
        }
    };
    double tx[G], ty[G], tz[G], tp[G];
    auto geometry = [&](int g, const V4<double>& pj, double hj, double& dx, double& dy,
                        double& dz) -> double {
        dx = pj.x - xi[g];
        dy = pj.y - yi[g];
        dz = pj.z - zi[g];
        const double s = USOFT ? hi[g] : hi[g] + hj;
        return rsqrt_pair(dx * dx + dy * dy + dz * dz + s);
    };

    pdl_next();  // (the finish may start and wait)
    load_i();
    int64_t base = pl.first_unit(a);
    fetch(static_cast<int64_t>(a) * pl.g + (u0 - base));
    for (int64_t u = u0; u < u1; ++u) {
        if (u >= base + (pl.nt - static_cast<int64_t>(a) * pl.g)) {
            flush_i();
            ++a;
            base = pl.first_unit(a);
            load_i();
        }
        const int64_t t = static_cast<int64_t>(a) * pl.g + (u - base);
        const int r0 = u == u0 ? static_cast<int>(q0 - u0 * kWarps) : 0;
        const int r1 = u + 1 == u1 ? static_cast<int>(q1 - u * kWarps) : kWarps;
        __syncthreads();  // the tile before is done with (its j sums are stored)
        s_p[tid] = nxt;
        if constexpr (!USOFT) s_h[tid] = nxh;
        s_j[tid] = v4<double>(0.0, 0.0, 0.0, 0.0);
        __syncthreads();
        if (u + 1 < u1) {
            const bool same = u + 1 < base + (pl.nt - static_cast<int64_t>(a) * pl.g);
            fetch(same ? t + 1 : static_cast<int64_t>(a + 1) * pl.g);
        }
#pragma unroll
        for (int g = 0; g < G; ++g) tx[g] = ty[g] = tz[g] = tp[g] = 0.0;
        if (t < static_cast<int64_t>(a + 1) * pl.g) {
#pragma unroll 2
            for (int k = 32 * r0; k < 32 * r1; ++k) {
                const V4<double> pj = s_p[k];
                const double hj = USOFT ? 0.0 : s_h[k];
#pragma unroll
                for (int g = 0; g < G; ++g) {
                    double dx, dy, dz;
                    const double inv = geometry(g, pj, hj, dx, dy, dz);
                    const double kk = pj.w * (inv * inv * inv);
                    tx[g] += dx * kk;
                    ty[g] += dy * kk;
                    tz[g] += dz * kk;
                    if constexpr (POT) tp[g] += pj.w * inv;
                }
            }
        } else {
            for (int r = r0; r < r1; ++r) {
                const int c = ((warp + r) & (kWarps - 1)) * 32;
                double cx = 0.0, cy = 0.0, cz = 0.0, cp = 0.0;
                const int from = (lane + 1) & 31;
#pragma unroll 2
                for (int s = 0; s < 32; ++s) {
                    const int k = c + ((lane + s) & 31);
                    const V4<double> pj = s_p[k];
                    const double hj = USOFT ? 0.0 : s_h[k];
#pragma unroll
                    for (int g = 0; g < G; ++g) {
                        double dx, dy, dz;
                        const double inv = geometry(g, pj, hj, dx, dy, dz);
                        const double k3 = inv * inv * inv;
                        const double ki = pj.w * k3, kj = mi[g] * k3;
                        tx[g] += dx * ki;
                        ty[g] += dy * ki;
                        tz[g] += dz * ki;
                        cx -= dx * kj;
                        cy -= dy * kj;
                        cz -= dz * kj;
                        if constexpr (POT) {
                            tp[g] += pj.w * inv;
                            cp += mi[g] * inv;
                        }
                    }
                    cx = __shfl_sync(0xffffffffu, cx, from);
                    cy = __shfl_sync(0xffffffffu, cy, from);
                    cz = __shfl_sync(0xffffffffu, cz, from);
                    if constexpr (POT) cp = __shfl_sync(0xffffffffu, cp, from);
                }
                V4<double> v = s_j[c + lane];
                v.x += cx;
                v.y += cy;
                v.z += cz;
                if constexpr (POT) v.w += cp;
                s_j[c + lane] = v;
                __syncthreads();  // the next warp to add to this chunk comes after
            }
            const int64_t j = t * kBS + tid;
            if (j < pl.n) {
                V4<double>* const to = r0 == 0
                                           ? p.js + static_cast<int64_t>(a) * pl.n + j
                                           : p.js2 + static_cast<int64_t>(blockIdx.x) * kBS + tid;
                *to = s_j[tid];
            }
        }
#pragma unroll
        for (int g = 0; g < G; ++g) {
            double* const v = s_i + g * NV * kBS + tid;
            v[0] += tx[g];
            v[kBS] += ty[g];
            v[2 * kBS] += tz[g];
            if constexpr (POT) v[(NV - 1) * kBS] += tp[g];
        }
    }
    flush_i();
}

// A particle's slots in order (j slots of the i-tiles below its own, then its own tile's i
// slots), FP64, and the epilogue.
template <typename R, typename S, bool MIXED>
__global__ void __launch_bounds__(128) direct_sym_finish(const SymParams<R, S> p,
                                                         const EpiDev<R> epi, bool want_pot) {
    const SymPlan& pl = p.plan;
    const int64_t k = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    pdl_next();
    pdl_wait();
    if (k >= pl.n) return;
    const int a = static_cast<int>(k / (kBS * pl.g));
    const int cnt = pl.last_block(a) - pl.first_block(a) + 1;
    const int64_t t = k / kBS;
    double sx = 0, sy = 0, sz = 0, sp = 0;
#pragma unroll 4
    for (int s = 0; s < a; ++s) {
        const V4<S> v = p.js[static_cast<int64_t>(s) * pl.n + k];
        sx += v.x; sy += v.y; sz += v.z; sp += v.w;
        // the second part of a unit that two runs share
        const int64_t q = 8 * (pl.first_unit(s) + t - static_cast<int64_t>(s) * pl.g);
        const int b = pl.block_of(q + 7);
        if (pl.run_start(b) > q) {
            const V4<S> w = p.js2[static_cast<int64_t>(b) * kBS + (k & (kBS - 1))];
            sx += w.x; sy += w.y; sz += w.z; sp += w.w;
        }
    }
#pragma unroll 8
    for (int s = 0; s < cnt; ++s) {
        const V4<S> v = p.is[static_cast<int64_t>(s) * pl.n + k];
        sx += v.x; sy += v.y; sz += v.z; sp += v.w;
    }
    apply_epi<R, MIXED>(epi, k, static_cast<R>(sx), static_cast<R>(sy), static_cast<R>(sz),
                        static_cast<R>(-sp), want_pot, p.posm, p.poslo);
}

template <int G2, bool USOFT, bool POT, bool UMASS, bool MIXED>
void launch32(const SymParams<float, typename Sym32<G2, USOFT, POT, UMASS, MIXED>::S>& p,
              cudaStream_t s) {
    constexpr size_t smem = Sym32<G2, USOFT, POT, UMASS, MIXED>::smem;
    auto* k = direct_sym32_kernel<G2, USOFT, POT, UMASS, MIXED>;
    if (smem > 48 * 1024)
        RRG_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      static_cast<int>(smem)));
    k<<<p.plan.blocks, kBS, smem, s>>>(p);
}

template <int G2, bool MIXED>
void dispatch32(bool usoft, bool pot, bool umass,
                const SymParams<float, typename std::conditional<MIXED, double, float>::type>& p,
                cudaStream_t s) {
#define RRG_SYM(US, PO, UM) launch32<G2, US, PO, UM, MIXED>(p, s)
    if constexpr (!MIXED) {
        if (umass) {
            if (usoft) { if (pot) RRG_SYM(true, true, true); else RRG_SYM(true, false, true); }
            else { if (pot) RRG_SYM(false, true, true); else RRG_SYM(false, false, true); }
            return;
        }
    }
    if (usoft) { if (pot) RRG_SYM(true, true, false); else RRG_SYM(true, false, false); }
    else { if (pot) RRG_SYM(false, true, false); else RRG_SYM(false, false, false); }
#undef RRG_SYM
}

template <int G>
void dispatch64(bool usoft, bool pot, const SymParams<double, double>& p, cudaStream_t s) {
#define RRG_SYM(US, PO)                                                                       \
    do {                                                                                      \
        constexpr size_t smem = Sym64<G, US, PO>::smem;                                       \
        auto* k = direct_sym64_kernel<G, US, PO>;                                             \
        if (smem > 48 * 1024)                                                                 \
            RRG_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,     \
                                          static_cast<int>(smem)));                           \
        k<<<p.plan.blocks, kBS, smem, s>>>(p);                                                \
    } while (0)
    if (usoft) { if (pot) RRG_SYM(true, true); else RRG_SYM(true, false); }
    else { if (pot) RRG_SYM(false, true); else RRG_SYM(false, false); }
#undef RRG_SYM
}

// Blocks per SM of the kernels of (prec, g) (the force kernel without potential; the one with it
// has as many or leaves the runs a little longer).
int resident_blocks(int prec, int g) {
    if (prec == RRG_PREC_FP64) {
        if (g == 2) return pair_blocks_per_sm(direct_sym64_kernel<2, true, false>, Sym64<2, true, false>::smem);
        return pair_blocks_per_sm(direct_sym64_kernel<4, true, false>, Sym64<4, true, false>::smem);
    }
    if (prec == RRG_PREC_MIXED) {
        if (g == 2) return pair_blocks_per_sm(direct_sym32_kernel<1, true, false, false, true>, Sym32<1, true, false, false, true>::smem);
        return pair_blocks_per_sm(direct_sym32_kernel<2, true, false, false, true>, Sym32<2, true, false, false, true>::smem);
    }
    if (g == 2) return pair_blocks_per_sm(direct_sym32_kernel<1, true, false, true, false>, Sym32<1, true, false, true, false>::smem);
    if (g == 4) return pair_blocks_per_sm(direct_sym32_kernel<2, true, false, true, false>, Sym32<2, true, false, true, false>::smem);
    return pair_blocks_per_sm(direct_sym32_kernel<4, true, false, true, false>, Sym32<4, true, false, true, false>::smem);
}

// i-particles per thread: the more, the fewer shuffles and tile reads a pair costs, but the fewer
// units there are to spread. With enough units for a run of at least one per resident block, the
// time is units x cost / blocks, with fewer it is one unit on each SM's two blocks, or one alone
// (about 1.1 of half the time of two together). Relative pair rates measured on B200 at
// N = 131,072 (FP64: 32,768), Gpairs/s of ordered pairs.
double pair_rate(int prec, int g, bool umass) {
    if (prec == RRG_PREC_FP64) return g == 2 ? 970 : 1020;
    if (prec == RRG_PREC_MIXED) return g == 2 ? 1960 : 2200;
    if (umass) return g == 2 ? 2810 : g == 4 ? 3390 : 3750;
    return g == 2 ? 2400 : g == 4 ? 2840 : 3050;
}

SymPlan plan_for(int prec, int64_t n, bool umass, int sms) {
    SymPlan best{};
    double t_best = 0.0;
    for (int g = 2; g <= (prec == RRG_PREC_FP32 ? 8 : 4); g *= 2) {
        const int per_sm = resident_blocks(prec, g);
        const SymPlan p = make_pair_plan(n, g, sms * per_sm);
        const double unit = g / pair_rate(prec, g, umass);  // per block of a full SM, x per_sm
        const double units = static_cast<double>(p.rounds) / 8;
        double t = per_sm * unit * std::max(1.0, units / (static_cast<double>(sms) * per_sm));
        if (units <= sms) t = 1.1 * unit;
        if (best.blocks == 0 || t <= t_best) {
            best = p;
            t_best = t;
        }
    }
    return best;
}

// js, is and js2 of a plan
size_t slot_bytes(int prec, const SymPlan& pl) {
    return (prec == RRG_PREC_FP32 ? sizeof(V4<float>) : sizeof(V4<double>)) *
           (static_cast<size_t>(pl.n) * static_cast<size_t>(pl.tiles - 1 + pl.islots) +
            static_cast<size_t>(pl.blocks) * kBS);
}

}  // namespace

// From 32 j-tiles on: at N = 8,192 FP32 takes 34 us (ordered pairs 38), MIXED 47 (65), FP64 84
// (109); at 6,000 33 (25) and FP64 77 (64), the units being too few to fill the SMs. Up to
// 131,072 particles the slots stay below 600 MB.
size_t direct_sym_scratch_bytes(int prec, int64_t n, bool umass, int sms) {
    if (!pair_plan_range(n)) return 0;
    return slot_bytes(prec, plan_for(prec, n, umass, sms));
}

void launch_direct_sym(const DirectLaunch& L, int sms) {
    RRG_REQUIRE(pair_plan_range(L.n), RRG_ERR_INVALID,
                "direct sum: too few or too many particles for pair slots");
    const bool umass = L.uniform_mass >= 0.0;
    const SymPlan pl = plan_for(L.prec, L.n, umass, sms);
    const size_t rows = static_cast<size_t>(pl.tiles - 1);
    RRG_REQUIRE(L.sym_scratch_bytes >= slot_bytes(L.prec, pl), RRG_ERR_INVALID,
                "direct sum: pair slots smaller than the schedule needs");
    RRG_REQUIRE(L.sym_scratch != nullptr && (reinterpret_cast<uintptr_t>(L.sym_scratch) & 31u) == 0,
                RRG_ERR_INVALID, "direct sum: pair slots must start on a 32-byte boundary");
    const bool usoft = L.hsoft == nullptr;
    const int bl = div_up(L.n, 128);
    if (L.prec == RRG_PREC_FP64) {
        SymParams<double, double> p{};
        p.plan = pl;
        p.posm = static_cast<const V4<double>*>(L.posm);
        p.hsoft = static_cast<const double*>(L.hsoft);
        p.uniform_h = pair_soft(L.uniform_hsoft);
        p.js = static_cast<V4<double>*>(L.sym_scratch);
        p.is = p.js + rows * L.n;
        p.js2 = p.is + static_cast<size_t>(pl.islots) * L.n;
        if (pl.g == 2) dispatch64<2>(usoft, L.want_pot, p, L.stream);
        else dispatch64<4>(usoft, L.want_pot, p, L.stream);
        RRG_LAUNCHED();
        launch_pdl(direct_sym_finish<double, double, false>, bl, 128, 0, L.stream, p,
                   make_epi<double>(L.epi), L.want_pot);
        RRG_LAUNCHED();
        return;
    }
    auto fill = [&](auto& p) {
        p.plan = pl;
        p.posm = static_cast<const V4<float>*>(L.posm);
        p.poslo = static_cast<const V4<float>*>(L.poslo);
        p.hsoft = static_cast<const float*>(L.hsoft);
        p.uniform_h = static_cast<float>(L.uniform_hsoft);
        p.uniform_m = umass ? static_cast<float>(L.uniform_mass) : 0.f;
        p.js = static_cast<decltype(p.js)>(L.sym_scratch);
        p.is = p.js + rows * L.n;
        p.js2 = p.is + static_cast<size_t>(pl.islots) * L.n;
    };
    if (L.prec == RRG_PREC_MIXED) {
        RRG_REQUIRE(L.poslo != nullptr, RRG_ERR_INVALID,
                    "direct sum: MIXED precision needs the low position parts");
        SymParams<float, double> p{};
        fill(p);
        if (pl.g == 2) dispatch32<1, true>(usoft, L.want_pot, umass, p, L.stream);
        else dispatch32<2, true>(usoft, L.want_pot, umass, p, L.stream);
        RRG_LAUNCHED();
        launch_pdl(direct_sym_finish<float, double, true>, bl, 128, 0, L.stream, p,
                   make_epi<float>(L.epi), L.want_pot);
    } else {
        SymParams<float, float> p{};
        fill(p);
        if (pl.g == 2) dispatch32<1, false>(usoft, L.want_pot, umass, p, L.stream);
        else if (pl.g == 4) dispatch32<2, false>(usoft, L.want_pot, umass, p, L.stream);
        else dispatch32<4, false>(usoft, L.want_pot, umass, p, L.stream);
        RRG_LAUNCHED();
        launch_pdl(direct_sym_finish<float, float, false>, bl, 128, 0, L.stream, p,
                   make_epi<float>(L.epi), L.want_pot);
    }
    RRG_LAUNCHED();
}

}  // namespace rrg
