// Hand-written adjoint of the direct-sum leapfrog on sm_100a.
//
// Forward (nbody.cu:19-65): a_i = sum_j m_j d_ij f_ij, d_ij = x_j - x_i,
//   f_ij = (|d_ij|^2 + h_i + h_j)^(-3/2).
// With g_ij = -3 (|d_ij|^2 + h_i + h_j)^(-5/2) the Jacobian blocks are
//   da_i/dx_j = m_j (f_ij I + g_ij d_ij d_ij^T)   (j != i),   da_i/dx_i = -sum_j (same),
//   da_i/dm_j = d_ij f_ij.
// For a cotangent lam on a (vector-Jacobian product):
//   xbar_k = sum_j (f_kj u_kj + g_kj d_kj (d_kj . u_kj)),  u_kj = m_k lam_j - m_j lam_k
//   mbar_k = -sum_j f_kj (lam_j . d_kj)
// The self pair contributes exactly zero (d = 0, u = 0), so the loop runs over all j like the
// forward kernel: j-tiles of 256 through shared memory, split-j partials summed in FP64 in a
// fixed order.
//
// Leapfrog (predict_step_ / correct_step_, nbody.cu:122-181), one step n -> n+1:
//   x' = x + dt v + dt^2/2 a(x),   v' = v + dt/2 (a(x) + a(x')).
// Backward with cotangents (X, V) of (x_{n+1}, v_{n+1}), X already holding the path through
// a(x_{n+1}) into v_{n+1}:
//   V_n = dt X + V
//   c_n = dt^2/2 X + dt/2 V + dt/2 V_n      (the last term: v_n's own dependence on a(x_n),
//                                             absent for n = 0 where v_0 is an input)
//   X_n = X + J(x_n)^T c_n,   mbar += (da(x_n)/dm)^T c_n
// so each step costs one vector-Jacobian product at x_n. The forward keeps (x, v, a(x)) every
// K steps. Between checkpoints the states come back two ways:
//   FP64: recomputed forward from the checkpoint below (K - 2 force evaluations per K steps),
//         so the gradient is the exact adjoint of the forward trajectory;
//   FP32: the leapfrog run backwards from the checkpoint above (reverse_init_kernel,
//         vjp_reverse_finish), the force a(x_m) summed in the same pass over the pairs as the
//         VJP at x_m (3 more operations per pair instead of a separate force evaluation).
//         Each reversed step rounds once more than the forward did; every segment restarts
//         from an exact checkpoint.
#include <algorithm>
#include <cstring>
#include <string>
#include <vector>

#include "host_io.h"
#include "kernels.cuh"
#include "pair_plan.cuh"

namespace rrg {
namespace {

constexpr int kBS = 256;

template <typename R>
struct VjpParams {
    const V4<R>* posm;
    const R* hsoft;
    R uniform_h;
    int64_t n;
    int64_t jchunk;
    const V4<R>* lam;
    V4<R>* out;
    V4<R>* part;
    int accumulate;  // out += result instead of out = result
    V4<R>* part_a;   // force partials (kernels with FORCE)
};

// Backward elementwise update of one step (applied to X after the VJP of the step before):
//   V_n = dt X + V;  c = dt^2/2 X + dt/2 V + [n > 0] dt/2 V_n.  V == nullptr: none.
template <typename R>
struct AdjUpd {
    V4<R>* V = nullptr;
    V4<R>* c = nullptr;
    R dt = 0;
    int with_vn = 0;
};

template <typename R>
__device__ __forceinline__ void adjoint_update_at(int64_t i, R xx, R xy, R xz,
                                                  const AdjUpd<R>& u) {
    const V4<R> v = u.V[i];
    const R dt = u.dt, h = dt * R(0.5), h2 = dt * dt * R(0.5);
    const R vx = dt * xx + v.x, vy = dt * xy + v.y, vz = dt * xz + v.z;
    R cx = h2 * xx + h * v.x, cy = h2 * xy + h * v.y, cz = h2 * xz + h * v.z;
    if (u.with_vn) {
        cx += h * vx;
        cy += h * vy;
        cz += h * vz;
    }
    u.V[i] = v4<R>(vx, vy, vz, R(0));
    u.c[i] = v4<R>(cx, cy, cz, R(0));
}

// FP64: rsqrt_pair, as the forward; the VJP's pair loop is FP64-pipe bound
template <typename R>
__device__ __forceinline__ R inv_sqrt(R x) {
    if constexpr (sizeof(R) == 4) return rsqrt_sfu(x);
    else return rsqrt_pair(x);
}

// ----------------------------------------------------------------------------------------------
// FP32 VJP on Blackwell's paired FP32 instructions (add/mul/fma .f32x2): each thread owns two
// k-particles, k0 = base + tid and k1 = base + 256 + tid, as the two halves of float2 registers;
// the j-tile is staged pre-duplicated, (x, x, y, y) (z, z, m, m) (lx, lx, ly, ly) (lz, lz, h, h),
// so each shared-memory broadcast lands in the register pairs the paired instructions read.
// Per pair: d = x_j - x_k, r2 = |d|^2 + h_k + h_j, f = r2^-3/2, g3 = r2^-5/2,
//   u = m_k lam_j - m_j lam_k  (UMASS: lam_j - lam_k, the common mass applied once at the end),
//   A += f u,  B += g3 (d . u) d,  M += f (d . lam_j);
// then x-bar_k = A - 3 B (x m for UMASS), m-bar_k = -M. 26 FMA-pipe operations per pair with
// uniform mass and softening (29 in general) and one SFU reciprocal square root; the FMA pipe
// is the bound.
// Sums run tile-blocked (256 j) like the forward kernels; j-split partials are summed in FP64
// in a fixed order by vjp_finish. Padding j sits 1e18 away with zero mass and cotangent: its
// f and g3 flush to zero, so it adds exactly nothing.
constexpr float kVjpPad = 1e18f;

// MGRAD = false: the mass gradient is not wanted (w of the result is 0), 4 operations less.
// FORCE: the same pass also sums the force a_k = sum_j m_j f d (3 operations more, 4 with
// unequal masses) into p.part_a, and every result goes to the split partials (a finish pass
// always follows).
template <bool USOFT, bool UMASS, bool MGRAD, bool FORCE>
__global__ void __launch_bounds__(kBS, 2) vjp_f32x2_kernel(const VjpParams<float> p, float um) {
    __shared__ float4 s_xy[kBS];
    __shared__ float4 s_zm[kBS];
    __shared__ float4 s_lxy[kBS];
    __shared__ float4 s_lzh[kBS];
    const int tid = threadIdx.x;
    const int64_t n = p.n;
    const int64_t kbase = static_cast<int64_t>(blockIdx.x) * (2 * kBS);

    float2 nx, ny, nz, hs, mk, lkx, lky, lkz;
    {
        float v[2][4], l[2][3], h[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int64_t k = kbase + e * kBS + tid;
            V4<float> pk = v4<float>(0.f, 0.f, 0.f, 0.f), lk = pk;
            h[e] = p.uniform_h;
            if (k < n) {
                pk = p.posm[k];
                lk = p.lam[k];
                if constexpr (!USOFT) h[e] = p.hsoft[k];
            }
            v[e][0] = pk.x;
            v[e][1] = pk.y;
            v[e][2] = pk.z;
            v[e][3] = pk.w;
            l[e][0] = lk.x;
            l[e][1] = lk.y;
            l[e][2] = lk.z;
        }
        nx = make_float2(-v[0][0], -v[1][0]);
        ny = make_float2(-v[0][1], -v[1][1]);
        nz = make_float2(-v[0][2], -v[1][2]);
        mk = make_float2(v[0][3], v[1][3]);
        // lam_k enters u with a minus sign: keep it negated
        lkx = make_float2(-l[0][0], -l[1][0]);
        lky = make_float2(-l[0][1], -l[1][1]);
        lkz = make_float2(-l[0][2], -l[1][2]);
        hs = USOFT ? make_float2(2.f * p.uniform_h, 2.f * p.uniform_h) : make_float2(h[0], h[1]);
    }
    const float2 z2 = make_float2(0.f, 0.f);
    float2 Ax = z2, Ay = z2, Az = z2, Bx = z2, By = z2, Bz = z2, Mm = z2;
    float2 Fx = z2, Fy = z2, Fz = z2;

    const int64_t jb = static_cast<int64_t>(blockIdx.y) * p.jchunk;
    const int64_t je = min(n, jb + p.jchunk);
    V4<float> nxt = v4<float>(kVjpPad, kVjpPad, kVjpPad, 0.f), nxl = v4<float>(0.f, 0.f, 0.f, 0.f);
    float nxt_h = 1.f;
    {
        const int64_t j = jb + tid;
        if (j < je) {
            nxt = p.posm[j];
            nxl = p.lam[j];
            if constexpr (!USOFT) nxt_h = p.hsoft[j];
        }
    }
    for (int64_t j0 = jb; j0 < je; j0 += kBS) {
        __syncthreads();
        s_xy[tid] = make_float4(nxt.x, nxt.x, nxt.y, nxt.y);
        s_zm[tid] = make_float4(nxt.z, nxt.z, nxt.w, nxt.w);
        s_lxy[tid] = make_float4(nxl.x, nxl.x, nxl.y, nxl.y);
        s_lzh[tid] = make_float4(nxl.z, nxl.z, nxt_h, nxt_h);
        __syncthreads();
        {
            const int64_t j = j0 + kBS + tid;
            nxt = v4<float>(kVjpPad, kVjpPad, kVjpPad, 0.f);
            nxl = v4<float>(0.f, 0.f, 0.f, 0.f);
            nxt_h = 1.f;
            if (j < je) {
                nxt = p.posm[j];
                nxl = p.lam[j];
                if constexpr (!USOFT) nxt_h = p.hsoft[j];
            }
        }
        float2 tAx = z2, tAy = z2, tAz = z2, tBx = z2, tBy = z2, tBz = z2, tM = z2;
        float2 tFx = z2, tFy = z2, tFz = z2;
        // (a chunk may be shorter than a tile; what is staged past its end adds nothing)
        const int cnt = static_cast<int>(min(static_cast<int64_t>(kBS), (je - j0 + 3) & ~int64_t(3)));
#pragma unroll 4
        for (int q = 0; q < cnt; ++q) {
            const float4 xy = s_xy[q], zm = s_zm[q], lxy = s_lxy[q], lzh = s_lzh[q];
            const float2 px = make_float2(xy.x, xy.y), py = make_float2(xy.z, xy.w);
            const float2 pz = make_float2(zm.x, zm.y);
            const float2 ljx = make_float2(lxy.x, lxy.y), ljy = make_float2(lxy.z, lxy.w);
            const float2 ljz = make_float2(lzh.x, lzh.y);
            const float2 dx = __fadd2_rn(px, nx);
            const float2 dy = __fadd2_rn(py, ny);
            const float2 dz = __fadd2_rn(pz, nz);
            const float2 s = USOFT ? hs : __fadd2_rn(hs, make_float2(lzh.z, lzh.w));
            const float2 r2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __ffma2_rn(dx, dx, s)));
            // one SFU op per pair: a second (rcp for r2^-1) would make the SFU pipe the bound
            const float2 inv = make_float2(rsqrt_sfu(r2.x), rsqrt_sfu(r2.y));
            const float2 inv2 = __fmul2_rn(inv, inv);
            const float2 f = __fmul2_rn(inv, inv2);
            const float2 g3 = __fmul2_rn(f, inv2);
            float2 ux, uy, uz;
            if constexpr (UMASS) {
                ux = __fadd2_rn(ljx, lkx);
                uy = __fadd2_rn(ljy, lky);
                uz = __fadd2_rn(ljz, lkz);
            } else {
                const float2 mj = make_float2(zm.z, zm.w);
                ux = __ffma2_rn(mk, ljx, __fmul2_rn(mj, lkx));
                uy = __ffma2_rn(mk, ljy, __fmul2_rn(mj, lky));
                uz = __ffma2_rn(mk, ljz, __fmul2_rn(mj, lkz));
            }
            const float2 dot = __ffma2_rn(dz, uz, __ffma2_rn(dy, uy, __fmul2_rn(dx, ux)));
            const float2 t = __fmul2_rn(g3, dot);
            tAx = __ffma2_rn(f, ux, tAx);
            tAy = __ffma2_rn(f, uy, tAy);
            tAz = __ffma2_rn(f, uz, tAz);
            tBx = __ffma2_rn(t, dx, tBx);
            tBy = __ffma2_rn(t, dy, tBy);
            tBz = __ffma2_rn(t, dz, tBz);
            if constexpr (MGRAD) {
                const float2 dl = __ffma2_rn(dz, ljz, __ffma2_rn(dy, ljy, __fmul2_rn(dx, ljx)));
                tM = __ffma2_rn(f, dl, tM);
            }
            if constexpr (FORCE) {
                const float2 fm = UMASS ? f : __fmul2_rn(make_float2(zm.z, zm.w), f);
                tFx = __ffma2_rn(fm, dx, tFx);
                tFy = __ffma2_rn(fm, dy, tFy);
                tFz = __ffma2_rn(fm, dz, tFz);
            }
        }
        Ax = __fadd2_rn(Ax, tAx);
        Ay = __fadd2_rn(Ay, tAy);
        Az = __fadd2_rn(Az, tAz);
        Bx = __fadd2_rn(Bx, tBx);
        By = __fadd2_rn(By, tBy);
        Bz = __fadd2_rn(Bz, tBz);
        Mm = __fadd2_rn(Mm, tM);
        if constexpr (FORCE) {
            Fx = __fadd2_rn(Fx, tFx);
            Fy = __fadd2_rn(Fy, tFy);
            Fz = __fadd2_rn(Fz, tFz);
        }
    }
    const float sc = UMASS ? um : 1.f;
    const float gx[2] = {sc * (Ax.x - 3.f * Bx.x), sc * (Ax.y - 3.f * Bx.y)};
    const float gy[2] = {sc * (Ay.x - 3.f * By.x), sc * (Ay.y - 3.f * By.y)};
    const float gz[2] = {sc * (Az.x - 3.f * Bz.x), sc * (Az.y - 3.f * Bz.y)};
    const float gm[2] = {MGRAD ? -Mm.x : 0.f, MGRAD ? -Mm.y : 0.f};
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const int64_t k = kbase + e * kBS + tid;
        if (k >= n) continue;
        if (FORCE || gridDim.y > 1) {
            const int64_t o = static_cast<int64_t>(blockIdx.y) * n + k;
            p.part[o] = v4<float>(gx[e], gy[e], gz[e], gm[e]);
            if constexpr (FORCE) {
                p.part_a[o] = e ? v4<float>(sc * Fx.y, sc * Fy.y, sc * Fz.y, 0.f)
                                : v4<float>(sc * Fx.x, sc * Fy.x, sc * Fz.x, 0.f);
            }
        } else if (p.accumulate) {
            const V4<float> o = p.out[k];
            p.out[k] = v4<float>(o.x + gx[e], o.y + gy[e], o.z + gz[e], o.w + gm[e]);
        } else {
            p.out[k] = v4<float>(gx[e], gy[e], gz[e], gm[e]);
        }
    }
}

// ----------------------------------------------------------------------------------------------
// FP32 VJP (and force) with each unordered pair evaluated once, on direct_sym.cu's schedule: the
// pair's geometry, f, g and the vector T = f u - 3 g (d . u) d serve both particles (T changes
// sign), so a pair with the mass gradient and the force costs 41 FMA-pipe operations (equal
// masses) instead of twice 29. The j sums (T, m-bar and the force) travel along the warp. G2 packed
// pairs of i-particles per thread. NV sums per particle: T (3), m-bar, FORCE: the force (3).
// Slots as in direct_sym.cu, one array of (T, m-bar) and, FORCE, one of the force behind it.
// Bound: the FP32 pipe (77% of the active cycles; the runs end unevenly). N = 16,384, equal masses, with the finish, us, ordered
// pairs (vjp_f32x2_kernel) -> here: with the force and the mass gradient 284 -> 246, without the
// force 252 -> 205.
// ----------------------------------------------------------------------------------------------
struct VjpPairParams {
    SymPlan plan;
    const V4<float>* posm;
    const float* hsoft;
    float uniform_h, um;  // um: the common mass (UMASS)
    const V4<float>* lam;
    V4<float>* js;    // [tiles - 1][n]
    V4<float>* is;    // [islots][n]
    V4<float>* js2;   // [blocks][kBS]
    int64_t force;    // offset of the force's three arrays from these
};

template <int G2, bool FORCE>
constexpr size_t vjp_pair_smem() {
    return sizeof(float) * (FORCE ? 7 : 4) * 2 * G2 * kBS + sizeof(float4) * (FORCE ? 4 : 3) * kBS;
}

template <int G2, bool USOFT, bool UMASS, bool MGRAD, bool FORCE>
__global__ void __launch_bounds__(kBS, 2) vjp_pair_kernel(const VjpPairParams p) {
    constexpr int NV = FORCE ? 7 : 4;
    extern __shared__ __align__(16) unsigned char sm_raw[];
    float4* const s_p = reinterpret_cast<float4*>(sm_raw);  // x, y, z, m
    float4* const s_l = s_p + kBS;                          // lam, h
    V4<float>* const s_j = reinterpret_cast<V4<float>*>(s_l + kBS);
    V4<float>* const s_jf = s_j + (FORCE ? kBS : 0);
    float* const s_i = reinterpret_cast<float*>(s_jf + kBS);  // [2 G2][NV][kBS]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const SymPlan& pl = p.plan;
    const int64_t q0 = pl.run_start(blockIdx.x), q1 = pl.run_start(blockIdx.x + 1);  // rounds
    const int64_t u0 = q0 / kPairWarps, u1 = (q1 + kPairWarps - 1) / kPairWarps;      // units
    int a = 0;
    while (a + 1 < pl.tiles && pl.first_unit(a + 1) <= u0) ++a;

    float2 nx[G2], ny[G2], nz[G2], hs[G2], mi[G2], lx[G2], ly[G2], lz[G2];  // (lam negated)
    auto load_i = [&]() {
#pragma unroll
        for (int g = 0; g < G2; ++g) {
            V4<float> pi[2], li[2];
            float h[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int64_t i = static_cast<int64_t>(a) * (kBS * 2 * G2) + (2 * g + e) * kBS + tid;
                pi[e] = v4<float>(kVjpPad, kVjpPad, kVjpPad, 0.f);
                li[e] = v4<float>(0.f, 0.f, 0.f, 0.f);
                h[e] = 1.f;
                if (i < pl.n) {
                    pi[e] = p.posm[i];
                    li[e] = p.lam[i];
                    if constexpr (!USOFT) h[e] = p.hsoft[i];
                }
            }
            nx[g] = make_float2(-pi[0].x, -pi[1].x);
            ny[g] = make_float2(-pi[0].y, -pi[1].y);
            nz[g] = make_float2(-pi[0].z, -pi[1].z);
            mi[g] = make_float2(pi[0].w, pi[1].w);
            lx[g] = make_float2(-li[0].x, -li[1].x);
            ly[g] = make_float2(-li[0].y, -li[1].y);
            lz[g] = make_float2(-li[0].z, -li[1].z);
            hs[g] = USOFT ? dup2(p.uniform_h + p.uniform_h) : make_float2(h[0], h[1]);
        }
#pragma unroll
        for (int k = 0; k < 2 * G2 * NV; ++k) s_i[k * kBS + tid] = 0.f;
    };
    const float um = UMASS ? p.um : 1.f;
    auto flush_i = [&]() {
        const int slot = static_cast<int>(blockIdx.x) - pl.first_block(a);
#pragma unroll
        for (int q = 0; q < 2 * G2; ++q) {
            const int64_t i = static_cast<int64_t>(a) * (kBS * 2 * G2) + q * kBS + tid;
            if (i >= pl.n) continue;
            const float* const v = s_i + q * NV * kBS + tid;
            V4<float>* const to = p.is + static_cast<int64_t>(slot) * pl.n + i;
            *to = v4<float>(um * v[0], um * v[kBS], um * v[2 * kBS], -v[3 * kBS]);
            if constexpr (FORCE)
                to[p.force] = v4<float>(um * v[4 * kBS], um * v[5 * kBS], um * v[6 * kBS], 0.f);
        }
    };
    V4<float> nxt, nxl;
    auto fetch = [&](int64_t t) {
        const int64_t j = t * kBS + tid;
        nxt = v4<float>(kVjpPad, kVjpPad, kVjpPad, 0.f);
        nxl = v4<float>(0.f, 0.f, 0.f, 1.f);
        if (j < pl.n) {
            nxt = p.posm[j];
            nxl = p.lam[j];
            if constexpr (!USOFT) nxl.w = p.hsoft[j];
        }
    };
    float2 tT[3][G2], tM[G2], tF[3][G2];

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
        const int r0 = u == u0 ? static_cast<int>(q0 - u0 * kPairWarps) : 0;
        const int r1 = u + 1 == u1 ? static_cast<int>(q1 - u * kPairWarps) : kPairWarps;
        const bool own = t < static_cast<int64_t>(a + 1) * pl.g;  // a's own tiles: i alone
        __syncthreads();  // the tile before is done with (its j sums are stored)
        s_p[tid] = make_float4(nxt.x, nxt.y, nxt.z, nxt.w);
        s_l[tid] = make_float4(nxl.x, nxl.y, nxl.z, nxl.w);
        s_j[tid] = v4<float>(0.f, 0.f, 0.f, 0.f);
        if constexpr (FORCE) s_jf[tid] = v4<float>(0.f, 0.f, 0.f, 0.f);
        __syncthreads();
        if (u + 1 < u1) {
            const bool same = u + 1 < base + (pl.nt - static_cast<int64_t>(a) * pl.g);
            fetch(same ? t + 1 : static_cast<int64_t>(a + 1) * pl.g);
        }
#pragma unroll
        for (int g = 0; g < G2; ++g) {
            tM[g] = make_float2(0.f, 0.f);
#pragma unroll
            for (int k = 0; k < 3; ++k) tT[k][g] = tF[k][g] = make_float2(0.f, 0.f);
        }
        // one j against the thread's i: the i sums, and (BOTH) the j sums jT, jM, jF
        float2 jT[3], jM, jF[3];
        auto pairs = [&](auto both, const float4& pj, const float4& lj) {
            constexpr bool BOTH = decltype(both)::value;
#pragma unroll
            for (int g = 0; g < G2; ++g) {
                const float2 dx = __fadd2_rn(dup2(pj.x), nx[g]);
                const float2 dy = __fadd2_rn(dup2(pj.y), ny[g]);
                const float2 dz = __fadd2_rn(dup2(pj.z), nz[g]);
                const float2 s = USOFT ? hs[g] : __fadd2_rn(hs[g], dup2(lj.w));
                const float2 r2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __ffma2_rn(dx, dx, s)));
                const float2 inv = make_float2(rsqrt_sfu(r2.x), rsqrt_sfu(r2.y));
                const float2 inv2 = __fmul2_rn(inv, inv);
                const float2 f = __fmul2_rn(inv, inv2);
                const float2 g3 = __fmul2_rn(__fmul2_rn(f, inv2), dup2(-3.f));
                const float2 mj = dup2(pj.w);
                float2 ux, uy, uz, dot, dli, dlj;
                if constexpr (UMASS) {
                    ux = __fadd2_rn(dup2(lj.x), lx[g]);
                    uy = __fadd2_rn(dup2(lj.y), ly[g]);
                    uz = __fadd2_rn(dup2(lj.z), lz[g]);
                } else {
                    ux = __ffma2_rn(mi[g], dup2(lj.x), __fmul2_rn(mj, lx[g]));
                    uy = __ffma2_rn(mi[g], dup2(lj.y), __fmul2_rn(mj, ly[g]));
                    uz = __ffma2_rn(mi[g], dup2(lj.z), __fmul2_rn(mj, lz[g]));
                }
                dot = __ffma2_rn(dz, uz, __ffma2_rn(dy, uy, __fmul2_rn(dx, ux)));
                if constexpr (MGRAD) {
                    dlj = __ffma2_rn(dz, dup2(lj.z),
                                     __ffma2_rn(dy, dup2(lj.y), __fmul2_rn(dx, dup2(lj.x))));
                    tM[g] = __ffma2_rn(f, dlj, tM[g]);
                    if constexpr (BOTH) {  // (lam_i is held negated)
                        dli = __ffma2_rn(dz, lz[g], __ffma2_rn(dy, ly[g], __fmul2_rn(dx, lx[g])));
                        jM = __ffma2_rn(f, dli, jM);
                    }
                }
                const float2 tt = __fmul2_rn(g3, dot);
                const float2 Tx = __ffma2_rn(tt, dx, __fmul2_rn(f, ux));
                const float2 Ty = __ffma2_rn(tt, dy, __fmul2_rn(f, uy));
                const float2 Tz = __ffma2_rn(tt, dz, __fmul2_rn(f, uz));
                tT[0][g] = __fadd2_rn(tT[0][g], Tx);
                tT[1][g] = __fadd2_rn(tT[1][g], Ty);
                tT[2][g] = __fadd2_rn(tT[2][g], Tz);
                if constexpr (BOTH) {
                    jT[0] = __fadd2_rn(jT[0], Tx);
                    jT[1] = __fadd2_rn(jT[1], Ty);
                    jT[2] = __fadd2_rn(jT[2], Tz);
                }
                if constexpr (FORCE) {
                    const float2 fi = UMASS ? f : __fmul2_rn(mj, f);
                    tF[0][g] = __ffma2_rn(fi, dx, tF[0][g]);
                    tF[1][g] = __ffma2_rn(fi, dy, tF[1][g]);
                    tF[2][g] = __ffma2_rn(fi, dz, tF[2][g]);
                    if constexpr (BOTH) {
                        const float2 fj = UMASS ? f : __fmul2_rn(mi[g], f);
                        jF[0] = __ffma2_rn(fj, dx, jF[0]);
                        jF[1] = __ffma2_rn(fj, dy, jF[1]);
                        jF[2] = __ffma2_rn(fj, dz, jF[2]);
                    }
                }
            }
        };
        if (own) {
#pragma unroll 2
            for (int k = 32 * r0; k < 32 * r1; ++k) pairs(std::false_type{}, s_p[k], s_l[k]);
        } else {
            for (int r = r0; r < r1; ++r) {
                const int c = ((warp + r) & (kPairWarps - 1)) * 32;
                const int from = (lane + 1) & 31;
                float cT[3] = {0.f, 0.f, 0.f}, cM = 0.f, cF[3] = {0.f, 0.f, 0.f};
#pragma unroll 2
                for (int s = 0; s < 32; ++s) {
                    const int k = c + ((lane + s) & 31);
                    jM = make_float2(cM, 0.f);
#pragma unroll
                    for (int e = 0; e < 3; ++e) {
                        jT[e] = make_float2(cT[e], 0.f);
                        jF[e] = make_float2(cF[e], 0.f);
                    }
                    pairs(std::true_type{}, s_p[k], s_l[k]);
#pragma unroll
                    for (int e = 0; e < 3; ++e) {
                        cT[e] = __shfl_sync(0xffffffffu, half_sum(jT[e]), from);
                        if constexpr (FORCE) cF[e] = __shfl_sync(0xffffffffu, half_sum(jF[e]), from);
                    }
                    if constexpr (MGRAD) cM = __shfl_sync(0xffffffffu, half_sum(jM), from);
                }
                V4<float> v = s_j[c + lane];
                s_j[c + lane] = v4<float>(v.x + cT[0], v.y + cT[1], v.z + cT[2], v.w + cM);
                if constexpr (FORCE) {
                    v = s_jf[c + lane];
                    s_jf[c + lane] = v4<float>(v.x + cF[0], v.y + cF[1], v.z + cF[2], 0.f);
                }
                __syncthreads();  // the next warp to add to this chunk comes after
            }
            const int64_t j = t * kBS + tid;
            if (j < pl.n) {
                V4<float>* const to = r0 == 0 ? p.js + static_cast<int64_t>(a) * pl.n + j
                                              : p.js2 + static_cast<int64_t>(blockIdx.x) * kBS + tid;
                // T and the force change sign for j; jM holds f (-lam_i . d) = -(m-bar_j's term)
                V4<float> v = s_j[tid];
                *to = v4<float>(-um * v.x, -um * v.y, -um * v.z, -v.w);
                if constexpr (FORCE) {
                    v = s_jf[tid];
                    to[p.force] = v4<float>(-um * v.x, -um * v.y, -um * v.z, 0.f);
                }
            }
        }
#pragma unroll
        for (int g = 0; g < G2; ++g) {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                float* const v = s_i + (2 * g + e) * NV * kBS + tid;
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    v[k * kBS] += e ? tT[k][g].y : tT[k][g].x;
                    if constexpr (FORCE) v[(4 + k) * kBS] += e ? tF[k][g].y : tF[k][g].x;
                }
                if constexpr (MGRAD) v[3 * kBS] += e ? tM[g].y : tM[g].x;
            }
        }
    }
    flush_i();
}

// ----------------------------------------------------------------------------------------------
// Symmetric VJP: the pair term is antisymmetric (T_jk = -T_kj for x-bar), so each unordered
// pair of particles is evaluated once. Blocks run over tile pairs (a, b), a <= b, of 256
// particles: threads own k in tile a (two each), tile b sits in shared memory. For a < b the j-side sums
// (x-bar_j -= T, m-bar_j += f (lam_k . d)) travel along the warp with the j they belong to (one
// shuffle per sum and step, see the kernel) and each warp adds its sums for a chunk of 32 j into
// a shared accumulator; block (a, b) then writes its tile-a sums to slot [a][b] and its
// tile-b sums to slot [b][a]. A finish pass adds the T slots of each particle in order. (The four
// warps add to the shared accumulator in no fixed order: the last bits of an FP64 gradient may differ
// from run to run.) Diagonal tiles evaluate only the k-side, as a non-symmetric pass would.
template <typename R>
struct VjpSymParams {
    const V4<R>* posm;
    const R* hsoft;
    R uniform_h;
    int64_t n;
    int tiles;
    int parts;     // of a tile pair: 256 / parts j each, 1 to 8
    const V4<R>* lam;
    V4<R>* slots;  // [tiles][tiles][parts][256]
};


// Two k per thread (tile a = k0 + 128 e): each j read from shared memory and each travelling sum
// serves two pairs (one k per thread was bound by shared memory as much as by the FP64 pipe).
constexpr int kSymThreads = kBS / 2;
template <typename R, bool USOFT>
__global__ void __launch_bounds__(kSymThreads) vjp_sym_kernel(const VjpSymParams<R> p) {
    __shared__ V4<R> s_pos[kBS];
    __shared__ V4<R> s_lam[kBS];
    __shared__ R s_h[USOFT ? 1 : kBS];
    __shared__ R s_acc[kBS][4];
    const int tid = threadIdx.x, lane = tid & 31;
    // upper-triangular (with diagonal) row-major tile-pair index -> (a, b)
    const int T = p.tiles;
    const int64_t t = blockIdx.x / p.parts;
    const int part = static_cast<int>(blockIdx.x) - static_cast<int>(t) * p.parts;
    const int len = kBS / p.parts, q0 = part * len;  // this block's j in the tile
    auto S = [T](int64_t a) { return a * T - a * (a - 1) / 2; };
    const double B2 = 2.0 * T + 1.0;
    int64_t a = static_cast<int64_t>(floor((B2 - sqrt(B2 * B2 - 8.0 * static_cast<double>(t))) * 0.5));
    if (a < 0) a = 0;
    while (a + 1 < T && S(a + 1) <= t) ++a;
    while (a > 0 && S(a) > t) --a;
    const int64_t b = t - S(a) + a;

    V4<R> pk[2], lk[2];
    R hk[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const int l = tid + e * kSymThreads;
        pk[e] = v4<R>(R(1e18), R(1e18), R(1e18), R(0));
        lk[e] = v4<R>(0, 0, 0, 0);
        hk[e] = p.uniform_h;
        const int64_t k = a * kBS + l;
        if (k < p.n) {
            pk[e] = p.posm[k];
            lk[e] = p.lam[k];
            if constexpr (!USOFT) hk[e] = pair_soft(p.hsoft[k]);
        }
        const int64_t j = b * kBS + l;
        const bool in = j < p.n;
        s_pos[l] = in ? p.posm[j] : v4<R>(R(1e18), R(1e18), R(1e18), R(0));
        s_lam[l] = in ? p.lam[j] : v4<R>(0, 0, 0, 0);
        if constexpr (!USOFT) s_h[l] = in ? p.hsoft[j] : R(1);
        s_acc[l][0] = s_acc[l][1] = s_acc[l][2] = s_acc[l][3] = R(0);
    }
    __syncthreads();
    const bool sym = (a != b);
    R gx[2] = {}, gy[2] = {}, gz[2] = {}, gm[2] = {};
    // one j against both k: the k-side terms into (gx, gy, gz, gm), the j-side ones added to v
    auto pairs = [&](int q, R v[4]) {
        const V4<R> pj = s_pos[q];
        const V4<R> lj = s_lam[q];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const R dx = pj.x - pk[e].x, dy = pj.y - pk[e].y, dz = pj.z - pk[e].z;
            const R s = USOFT ? (hk[e] + hk[e]) : (hk[e] + s_h[q]);
            const R r2 = dx * dx + dy * dy + dz * dz + s;
            const R inv = inv_sqrt(r2);
            const R inv2 = inv * inv;
            const R f = inv * inv2;
            const R g = R(-3) * f * inv2;
            const R ux = pk[e].w * lj.x - pj.w * lk[e].x;
            const R uy = pk[e].w * lj.y - pj.w * lk[e].y;
            const R uz = pk[e].w * lj.z - pj.w * lk[e].z;
            const R tt = g * (dx * ux + dy * uy + dz * uz);
            const R Tx = f * ux + tt * dx, Ty = f * uy + tt * dy, Tz = f * uz + tt * dz;
            gx[e] += Tx;
            gy[e] += Ty;
            gz[e] += Tz;
            gm[e] -= f * (dx * lj.x + dy * lj.y + dz * lj.z);
            v[0] -= Tx;
            v[1] -= Ty;
            v[2] -= Tz;
            v[3] += f * (dx * lk[e].x + dy * lk[e].y + dz * lk[e].z);
        }
    };
    if (!sym) {
#pragma unroll 2
        for (int q = q0; q < q0 + len; ++q) {
            R v[4] = {};
            pairs(q, v);
        }
    } else {
        // the j-side terms ride along the warp: in step t of a chunk of 32 j, lane l takes
        // j = 32 c + (l + t) mod 32 and adds to the sums that lane l + 1 held for it, so after
        // 32 steps lane l holds its warp's sums for j = 32 c + l (one shuffle per sum and step,
        // and one shared add per chunk, instead of a warp reduction per j)
        for (int c = q0 / 32; c < (q0 + len) / 32; ++c) {
            R v[4] = {};
#pragma unroll 2
            for (int t = 0; t < 32; ++t) {
                pairs(c * 32 + ((lane + t) & 31), v);
                const int from = (lane + 1) & 31;
#pragma unroll
                for (int k = 0; k < 4; ++k) v[k] = __shfl_sync(0xffffffffu, v[k], from);
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) atomicAdd(&s_acc[c * 32 + lane][k], v[k]);
        }
    }
    V4<R>* const ks = p.slots + ((a * T + b) * p.parts + part) * kBS;
#pragma unroll
    for (int e = 0; e < 2; ++e)
        ks[tid + e * kSymThreads] = v4<R>(gx[e], gy[e], gz[e], gm[e]);
    if (sym) {
        __syncthreads();
        for (int l = q0 + tid; l < q0 + len; l += kSymThreads)  // (every j of the tile is in one part)
            p.slots[(b * T + a) * p.parts * kBS + l] =
                v4<R>(s_acc[l][0], s_acc[l][1], s_acc[l][2], s_acc[l][3]);
    }
}

// A block of (32, 8) threads takes 32 particles of one tile, warp w every eighth of their sums;
// warp 0 adds the eight in order.
constexpr int kFinWarps = 8;
template <typename R>
__global__ void __launch_bounds__(32 * kFinWarps)
vjp_sym_finish(int64_t n, int T, int parts, const V4<R>* __restrict__ slots, V4<R>* __restrict__ out,
               int accumulate, const AdjUpd<R> upd) {
    __shared__ double sh[kFinWarps][4][32];
    const int lane = threadIdx.x, w = threadIdx.y;
    const int64_t k = static_cast<int64_t>(blockIdx.x) * 32 + lane;
    const int64_t a = k / kBS, l = k % kBS;
    double v[4] = {};
    if (k < n) {
        // the tiles before (one sum each, in their first part), then the parts of the others
        const V4<R>* const from = slots + a * T * parts * kBS + l;
        const int count = static_cast<int>(a + (T - a) * parts);
#pragma unroll 4
        for (int i = w; i < count; i += kFinWarps) {
            const V4<R> q = from[(i < a ? i * parts : a * parts + (i - a)) * kBS];
            v[0] += q.x;
            v[1] += q.y;
            v[2] += q.z;
            v[3] += q.w;
        }
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) sh[w][c][lane] = v[c];
    __syncthreads();
    if (w != 0 || k >= n) return;
#pragma unroll
    for (int c = 0; c < 4; ++c)
        for (int i = 1; i < kFinWarps; ++i) v[c] += sh[i][c][lane];
    if (accumulate) {
        const V4<R> o = out[k];
        v[0] += o.x;
        v[1] += o.y;
        v[2] += o.z;
        v[3] += o.w;
    }
    const V4<R> r = v4<R>(static_cast<R>(v[0]), static_cast<R>(v[1]), static_cast<R>(v[2]),
                          static_cast<R>(v[3]));
    out[k] = r;
    if (upd.V) adjoint_update_at(k, r.x, r.y, r.z, upd);
}

// Parts of a tile pair: 1, 2, 4 or 8, the most that keep the blocks within eight per SM. Whole pairs
// leave SMs idle below ~8,000 particles (N = 2,000: 36 blocks) and fill the last ones badly above.
// Product and finish, us, whole pairs and one k per thread -> parts -> two k per thread: N = 1,000
// 56.6 -> 11.9 -> 13.2, 2,000 57.3 -> 18.7 -> 16.7, 3,000 - -> 42.1 -> 29.7, 5,000 100 -> 76.6 -> 59.6,
// 6,500 - -> 146 -> 94.5, 8,000 195 -> 192 -> 138 (four blocks per SM: 5,000 61.2, 8,000 147).
int vjp_sym_parts(int64_t n, int sms) {
    const int64_t T = (n + kBS - 1) / kBS, blocks = T * (T + 1) / 2;
    int parts = 1;
    while (parts < 8 && 2 * parts * blocks <= 8 * static_cast<int64_t>(sms)) parts *= 2;
    return parts;
}

template <typename R>
size_t vjp_sym_slot_bytes(int64_t n, int sms) {
    const int64_t T = (n + kBS - 1) / kBS;
    return sizeof(V4<R>) * static_cast<size_t>(T * T * vjp_sym_parts(n, sms) * kBS);
}

template <typename R>
void vjp_sym_launch(const void* posm, const void* hsoft, double uniform_h, int64_t n,
                    const void* lam, void* out, bool accumulate, void* slots,
                    int sms, cudaStream_t stream, const AdjUpd<R>& upd = AdjUpd<R>()) {
    const int T = static_cast<int>((n + kBS - 1) / kBS);
    VjpSymParams<R> p;
    p.posm = static_cast<const V4<R>*>(posm);
    p.hsoft = static_cast<const R*>(hsoft);
    p.uniform_h = pair_soft(static_cast<R>(uniform_h));
    p.n = n;
    p.tiles = T;
    p.parts = vjp_sym_parts(n, sms);
    p.lam = static_cast<const V4<R>*>(lam);
    p.slots = static_cast<V4<R>*>(slots);
    const unsigned blocks = static_cast<unsigned>(static_cast<int64_t>(T) * (T + 1) / 2 * p.parts);
    if (hsoft) vjp_sym_kernel<R, false><<<blocks, kSymThreads, 0, stream>>>(p);
    else vjp_sym_kernel<R, true><<<blocks, kSymThreads, 0, stream>>>(p);
    RRG_LAUNCHED();
    vjp_sym_finish<R><<<div_up(n, 32), dim3(32, kFinWarps), 0, stream>>>(
        n, T, p.parts, p.slots, static_cast<V4<R>*>(out), accumulate ? 1 : 0, upd);
    RRG_LAUNCHED();
}

// Sums of a particle's split partials in FP64 and a fixed order: a block of (32, 8) threads takes
// 32 particles, warp w the splits w, w + 8, ..., and warp 0 adds the eight sums in order. f: the
// force partials', with FORCE. True for the threads (of warp 0) that hold a particle's sums.
template <bool FORCE>
__device__ __forceinline__ bool vjp_part_sum(const VjpParams<float>& p, int splits, int64_t k,
                                             double s[4], double f[3]) {
    constexpr int NV = FORCE ? 7 : 4;
    __shared__ double sh[kFinWarps][NV][32];
    const int lane = threadIdx.x, w = threadIdx.y;
    double v[NV] = {};
    if (k < p.n) {
#pragma unroll 4
        for (int i = w; i < splits; i += kFinWarps) {
            const int64_t o = static_cast<int64_t>(i) * p.n + k;
            const V4<float> q = p.part[o];
            v[0] += q.x;
            v[1] += q.y;
            v[2] += q.z;
            v[3] += q.w;
            if constexpr (FORCE) {
                const V4<float> a = p.part_a[o];
                v[4] += a.x;
                v[5] += a.y;
                v[6] += a.z;
            }
        }
    }
#pragma unroll
    for (int c = 0; c < NV; ++c) sh[w][c][lane] = v[c];
    __syncthreads();
    if (w != 0 || k >= p.n) return false;
#pragma unroll
    for (int c = 0; c < NV; ++c)
        for (int i = 1; i < kFinWarps; ++i) v[c] += sh[i][c][lane];
#pragma unroll
    for (int c = 0; c < 4; ++c) s[c] = v[c];
    if constexpr (FORCE) {
#pragma unroll
        for (int c = 0; c < 3; ++c) f[c] = v[4 + c];
    }
    return true;
}

__global__ void __launch_bounds__(32 * kFinWarps) vjp_finish(const VjpParams<float> p, int splits,
                                                             const AdjUpd<float> upd) {
    const int64_t k = static_cast<int64_t>(blockIdx.x) * 32 + threadIdx.x;
    double s[4];
    if (!vjp_part_sum<false>(p, splits, k, s, nullptr)) return;
    if (p.accumulate) {
        const V4<float> o = p.out[k];
        s[0] += o.x;
        s[1] += o.y;
        s[2] += o.z;
        s[3] += o.w;
    }
    const V4<float> r = v4<float>(static_cast<float>(s[0]), static_cast<float>(s[1]),
                                  static_cast<float>(s[2]), static_cast<float>(s[3]));
    p.out[k] = r;
    if (upd.V) adjoint_update_at(k, r.x, r.y, r.z, upd);
}

// j-chunks of the ordered FP32 VJP. Where 256-particle chunks fill less than one wave of resident
// blocks (up to ~6,000 particles): the shortest multiple of 32 that stays within a wave. Beyond:
// whole tiles, the fewest chunks whose blocks fill whole waves to within 2% of the best achievable
// (the rule of the forward kernels). Product with force and its finish, us, whole tiles and one thread
// per particle in the finish -> here: N = 600 62.4 -> 7.8, 1,000 43.4 -> 8.1, 2,000 44.3 -> 12.0,
// 3,000 27.6 -> 16.5, 4,000 29.2 -> 25.6, 6,000 51.9 -> 44.8.
struct VjpChunks {
    int64_t chunk;
    int splits;
};
VjpChunks vjp_f32x2_chunks(int64_t n, int sms) {
    const int resident = resident_blocks_per_sm(
        reinterpret_cast<const void*>(&vjp_f32x2_kernel<true, true, true, false>), kBS, 0);
    const int64_t kblocks = (n + 2 * kBS - 1) / (2 * kBS);
    const int64_t tiles = (n + kBS - 1) / kBS;
    const int64_t slots = static_cast<int64_t>(sms) * resident;
    for (int64_t c = 32; c <= kBS; c += 32)
        if (kblocks * ((n + c - 1) / c) <= slots)
            return {c, static_cast<int>((n + c - 1) / c)};
    double best = 0, eff[65] = {};
    const int64_t top = std::min<int64_t>(tiles, 64);
    for (int64_t sp = 1; sp <= top; ++sp) {
        const int64_t total = kblocks * sp;
        const int64_t waves = (total + slots - 1) / slots;
        eff[sp] = static_cast<double>(total) / static_cast<double>(waves * slots);
        best = std::max(best, eff[sp]);
    }
    int64_t sp = 1;
    while (eff[sp] < best - 0.02) ++sp;
    const int64_t per = (tiles + sp - 1) / sp;
    return {per * kBS, static_cast<int>((tiles + per - 1) / per)};
}

size_t vjp_f32x2_part_bytes(int64_t n, int splits) {
    return splits > 1 ? sizeof(V4<float>) * static_cast<size_t>(n) * splits : 0;
}

// uniform_m >= 0: every particle has this mass (the caller has checked).
void adjoint_update_launch(int64_t n, const void* X, const AdjUpd<float>& upd, cudaStream_t s);

// upd.V != nullptr: also applies the next step's adjoint update to out (= X) afterwards.
// mgrad = false: no mass gradient (the w slot gets 0, or keeps its value when accumulating).
void vjp_f32x2_launch(const void* posm, const void* hsoft, double uniform_h, double uniform_m,
                      int64_t n, const void* lam, void* out, bool accumulate, void* part,
                      const VjpChunks& chunks, cudaStream_t stream,
                      const AdjUpd<float>& upd = AdjUpd<float>(), bool mgrad = true) {
    const int real = chunks.splits;
    VjpParams<float> p;
    p.posm = static_cast<const V4<float>*>(posm);
    p.hsoft = static_cast<const float*>(hsoft);
    p.uniform_h = static_cast<float>(uniform_h);
    p.n = n;
    p.jchunk = chunks.chunk;
    p.lam = static_cast<const V4<float>*>(lam);
    p.out = static_cast<V4<float>*>(out);
    p.part = static_cast<V4<float>*>(part);
    p.accumulate = accumulate ? 1 : 0;
    p.part_a = nullptr;
    RRG_REQUIRE(real == 1 || part != nullptr, RRG_ERR_STATE, "vjp: missing split partials");
    dim3 grid(static_cast<unsigned>((n + 2 * kBS - 1) / (2 * kBS)), real);
    const float um = uniform_m >= 0 ? static_cast<float>(uniform_m) : 1.f;
#define RRG_VJP2(US, UM, MG) vjp_f32x2_kernel<US, UM, MG, false><<<grid, kBS, 0, stream>>>(p, um)
#define RRG_VJP2_M(US, UM) \
    do {                   \
        if (mgrad)         \
            RRG_VJP2(US, UM, true); \
        else               \
            RRG_VJP2(US, UM, false); \
    } while (0)
    if (uniform_m >= 0) {
        if (hsoft) RRG_VJP2_M(false, true);
        else RRG_VJP2_M(true, true);
    } else {
        if (hsoft) RRG_VJP2_M(false, false);
        else RRG_VJP2_M(true, false);
    }
#undef RRG_VJP2_M
#undef RRG_VJP2
    RRG_LAUNCHED();
    if (real > 1) {
        vjp_finish<<<div_up(n, 32), dim3(32, kFinWarps), 0, stream>>>(p, real, upd);
        RRG_LAUNCHED();
    } else if (upd.V) {
        adjoint_update_launch(n, out, upd, stream);
    }
}

// ----------------------------------------------------------------------------------------------
// Reverse leapfrog between checkpoints (FP32 backward). The step x' = x + dt v + dt^2/2 a(x),
// v' = v + dt/2 (a(x) + a(x')) inverts exactly in real arithmetic:
//   w = v' - dt/2 a(x'),  x = x' - dt w,  v = w - dt/2 a(x),
// so the backward sweep rebuilds x_m from the state at m + 1, the force a(x_m) coming out of
// the same pass over the pairs as the VJP at x_m. In FP32 each reversed step rounds once more
// than the forward did, and every segment starts again from an exact checkpoint.
struct RevStep {
    const V4<float>* x;  // x_m (positions and masses)
    V4<float>* x_next;   // x_{m-1} out, or nullptr
    V4<float>* w;        // half-step velocity, updated in place: w -= dt a(x_m)
    float dt;
};

// w -= dt a(x_m), x_{m-1} = x_m - dt w for particle k
__device__ __forceinline__ void reverse_step_at(int64_t k, double ax, double ay, double az,
                                                const RevStep& r) {
    V4<float> w = r.w[k];
    w.x -= r.dt * static_cast<float>(ax);
    w.y -= r.dt * static_cast<float>(ay);
    w.z -= r.dt * static_cast<float>(az);
    r.w[k] = w;
    if (r.x_next) {
        const V4<float> x = r.x[k];
        r.x_next[k] = v4<float>(x.x - r.dt * w.x, x.y - r.dt * w.y, x.z - r.dt * w.z, x.w);
    }
}

// Top of a segment: w = v - dt/2 a, x_out = x - dt w (mass carried).
__global__ void reverse_init_kernel(int64_t n, const V4<float>* __restrict__ x,
                                    const V4<float>* __restrict__ v,
                                    const V4<float>* __restrict__ a, V4<float>* __restrict__ w,
                                    V4<float>* __restrict__ x_out, float dt) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float h = 0.5f * dt;
    const V4<float> vi = v[i], ai = a[i], xi = x[i];
    const V4<float> wi = v4<float>(vi.x - h * ai.x, vi.y - h * ai.y, vi.z - h * ai.z, 0.f);
    w[i] = wi;
    x_out[i] = v4<float>(xi.x - dt * wi.x, xi.y - dt * wi.y, xi.z - dt * wi.z, xi.w);
}

// Finish of a FORCE pass at x_m: X += sum of the VJP partials (fixed order, FP64), a(x_m) from
// the force partials, w -= dt a, x_{m-1} = x_m - dt w, then the adjoint update of step m - 1.
__global__ void __launch_bounds__(32 * kFinWarps) vjp_reverse_finish(const VjpParams<float> p,
                                                                     int splits,
                                                                     const AdjUpd<float> upd,
                                                                     const RevStep r) {
    const int64_t k = static_cast<int64_t>(blockIdx.x) * 32 + threadIdx.x;
    double s[4], f[3];
    if (!vjp_part_sum<true>(p, splits, k, s, f)) return;
    const V4<float> o = p.out[k];
    const V4<float> X = v4<float>(static_cast<float>(s[0] + o.x), static_cast<float>(s[1] + o.y),
                                  static_cast<float>(s[2] + o.z), static_cast<float>(s[3] + o.w));
    p.out[k] = X;
    reverse_step_at(k, f[0], f[1], f[2], r);
    if (upd.V) adjoint_update_at(k, X.x, X.y, X.z, upd);
}

// One reverse step at x_m = r.x: VJP with cotangent lam accumulated into out (= X), a(x_m),
// the reverse update of (w, positions) and the adjoint update upd. part / part_a hold
// [splits][n] V4 each.
void vjp_reverse_launch(const void* hsoft, double uniform_h, double uniform_m, int64_t n,
                        const void* lam, void* out, void* part, void* part_a,
                        const VjpChunks& chunks, cudaStream_t stream, const AdjUpd<float>& upd, const RevStep& r,
                        bool mgrad) {
    const int real = chunks.splits;
    RRG_REQUIRE(part && part_a, RRG_ERR_STATE, "vjp: missing partials");
    VjpParams<float> p;
    p.posm = r.x;
    p.hsoft = static_cast<const float*>(hsoft);
    p.uniform_h = static_cast<float>(uniform_h);
    p.n = n;
    p.jchunk = chunks.chunk;
    p.lam = static_cast<const V4<float>*>(lam);
    p.out = static_cast<V4<float>*>(out);
    p.part = static_cast<V4<float>*>(part);
    p.accumulate = 1;
    p.part_a = static_cast<V4<float>*>(part_a);
    dim3 grid(static_cast<unsigned>((n + 2 * kBS - 1) / (2 * kBS)), real);
    const float um = uniform_m >= 0 ? static_cast<float>(uniform_m) : 1.f;
#define RRG_VJPF(US, UM, MG) vjp_f32x2_kernel<US, UM, MG, true><<<grid, kBS, 0, stream>>>(p, um)
#define RRG_VJPF_M(US, UM)          \
    do {                            \
        if (mgrad)                  \
            RRG_VJPF(US, UM, true); \
        else                        \
            RRG_VJPF(US, UM, false); \
    } while (0)
    if (uniform_m >= 0) {
        if (hsoft) RRG_VJPF_M(false, true);
        else RRG_VJPF_M(true, true);
    } else {
        if (hsoft) RRG_VJPF_M(false, false);
        else RRG_VJPF_M(true, false);
    }
#undef RRG_VJPF_M
#undef RRG_VJPF
    RRG_LAUNCHED();
    vjp_reverse_finish<<<div_up(n, 32), dim3(32, kFinWarps), 0, stream>>>(p, real, upd, r);
    RRG_LAUNCHED();
}

// A particle's slots in order, FP64 (direct_sym_finish): (T, m-bar) sums, and with FORCE the force.
template <bool FORCE>
__device__ __forceinline__ void vjp_pair_sum(const VjpPairParams& p, int64_t k, double s[4],
                                             double f[3]) {
    const SymPlan& pl = p.plan;
    const int a = static_cast<int>(k / (kBS * pl.g));
    const int cnt = pl.last_block(a) - pl.first_block(a) + 1;
    const int64_t t = k / kBS;
    auto add = [&](const V4<float>* q) {
        const V4<float> v = *q;
        s[0] += v.x;
        s[1] += v.y;
        s[2] += v.z;
        s[3] += v.w;
        if constexpr (FORCE) {
            const V4<float> w = q[p.force];
            f[0] += w.x;
            f[1] += w.y;
            f[2] += w.z;
        }
    };
#pragma unroll 4
    for (int i = 0; i < a; ++i) {
        add(p.js + static_cast<int64_t>(i) * pl.n + k);
        // the second part of a unit that two runs share
        const int64_t q = 8 * (pl.first_unit(i) + t - static_cast<int64_t>(i) * pl.g);
        const int b = pl.block_of(q + 7);
        if (pl.run_start(b) > q) add(p.js2 + static_cast<int64_t>(b) * kBS + (k & (kBS - 1)));
    }
#pragma unroll 4
    for (int i = 0; i < cnt; ++i) add(p.is + static_cast<int64_t>(i) * pl.n + k);
}

// vjp_finish and vjp_reverse_finish (FORCE) on those sums.
template <bool FORCE>
__global__ void __launch_bounds__(128) vjp_pair_finish(const VjpPairParams p, V4<float>* out,
                                                       int accumulate, const AdjUpd<float> upd,
                                                       const RevStep r) {
    const int64_t k = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (k >= p.plan.n) return;
    double s[4] = {0, 0, 0, 0}, f[3] = {0, 0, 0};
    vjp_pair_sum<FORCE>(p, k, s, f);
    if (accumulate) {
        const V4<float> o = out[k];
        s[0] += o.x;
        s[1] += o.y;
        s[2] += o.z;
        s[3] += o.w;
    }
    const V4<float> X = v4<float>(static_cast<float>(s[0]), static_cast<float>(s[1]),
                                  static_cast<float>(s[2]), static_cast<float>(s[3]));
    out[k] = X;
    if constexpr (FORCE) reverse_step_at(k, f[0], f[1], f[2], r);
    if (upd.V) adjoint_update_at(k, X.x, X.y, X.z, upd);
}

int vjp_pair_blocks(int sms, bool umass) {
    // the kernel of the reversed steps, with equal masses or not
    const size_t smem = vjp_pair_smem<2, true>();
    return sms * (umass ? pair_blocks_per_sm(vjp_pair_kernel<2, true, true, true, true>, smem)
                        : pair_blocks_per_sm(vjp_pair_kernel<2, true, false, true, true>, smem));
}

SymPlan vjp_pair_plan(int64_t n, int sms, bool umass) {
    return make_pair_plan(n, 4, vjp_pair_blocks(sms, umass));
}

// V4 records of one slot array (js, is and js2 together)
int64_t vjp_pair_records(const SymPlan& pl) {
    return static_cast<int64_t>(pl.tiles - 1 + pl.islots) * pl.n +
           static_cast<int64_t>(pl.blocks) * kBS;
}

// bytes of the slots ((T, m-bar) and force), 0 where the ordered kernel is the faster one
size_t vjp_pair_bytes(int64_t n, int sms) {
    if (!pair_plan_range(n)) return 0;
    return 2 * sizeof(V4<float>) *
           static_cast<size_t>(std::max(vjp_pair_records(vjp_pair_plan(n, sms, true)),
                                        vjp_pair_records(vjp_pair_plan(n, sms, false))));
}

template <bool USOFT, bool UMASS>
void vjp_pair_dispatch(const VjpPairParams& p, bool mgrad, bool force, cudaStream_t s) {
    auto go = [&](auto* k, size_t smem) {
        if (smem > 48 * 1024)
            RRG_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          static_cast<int>(smem)));
        k<<<p.plan.blocks, kBS, smem, s>>>(p);
    };
    if (force) {
        if (mgrad) go(vjp_pair_kernel<2, USOFT, UMASS, true, true>, vjp_pair_smem<2, true>());
        else go(vjp_pair_kernel<2, USOFT, UMASS, false, true>, vjp_pair_smem<2, true>());
    } else {
        if (mgrad) go(vjp_pair_kernel<2, USOFT, UMASS, true, false>, vjp_pair_smem<2, false>());
        else go(vjp_pair_kernel<2, USOFT, UMASS, false, false>, vjp_pair_smem<2, false>());
    }
    RRG_LAUNCHED();
}

// X (out) += VJP at posm with cotangent lam; r != nullptr: also the force there and the reverse
// step; then the adjoint update upd.
void vjp_pair_launch(const void* posm, const void* hsoft, double uniform_h, double uniform_m,
                     int64_t n, const void* lam, void* out, bool accumulate, void* slots,
                     size_t slot_bytes, int sms, cudaStream_t s, const AdjUpd<float>& upd, const RevStep* r,
                     bool mgrad) {
    const bool umass = uniform_m >= 0;
    RRG_REQUIRE(pair_plan_range(n), RRG_ERR_INVALID,
                "vjp: too few or too many particles for pair slots");
    VjpPairParams p{};
    p.plan = vjp_pair_plan(n, sms, umass);
    RRG_REQUIRE(slot_bytes >= 2 * sizeof(V4<float>) * static_cast<size_t>(vjp_pair_records(p.plan)),
                RRG_ERR_INVALID, "vjp: pair slots smaller than the schedule needs");
    p.posm = static_cast<const V4<float>*>(posm);
    p.hsoft = static_cast<const float*>(hsoft);
    p.uniform_h = static_cast<float>(uniform_h);
    p.um = umass ? static_cast<float>(uniform_m) : 1.f;
    p.lam = static_cast<const V4<float>*>(lam);
    p.js = static_cast<V4<float>*>(slots);
    p.is = p.js + static_cast<int64_t>(p.plan.tiles - 1) * n;
    p.js2 = p.is + static_cast<int64_t>(p.plan.islots) * n;
    p.force = vjp_pair_records(p.plan);
    const bool force = r != nullptr;
    if (hsoft) {
        if (umass) vjp_pair_dispatch<false, true>(p, mgrad, force, s);
        else vjp_pair_dispatch<false, false>(p, mgrad, force, s);
    } else {
        if (umass) vjp_pair_dispatch<true, true>(p, mgrad, force, s);
        else vjp_pair_dispatch<true, false>(p, mgrad, force, s);
    }
    auto* o = static_cast<V4<float>*>(out);
    if (force) vjp_pair_finish<true><<<div_up(n, 128), 128, 0, s>>>(p, o, accumulate ? 1 : 0, upd, *r);
    else vjp_pair_finish<false><<<div_up(n, 128), 128, 0, s>>>(p, o, accumulate ? 1 : 0, upd, RevStep{});
    RRG_LAUNCHED();
}

// Does every particle's mass equal posm[0].w?  flags[0] (zeroed by the caller) becomes 1 on a
// mismatch; flags[1] receives posm[0].w as double bits.
template <typename R>
__global__ void uniform_mass_kernel(int64_t n, const V4<R>* __restrict__ posm,
                                    unsigned long long* __restrict__ flags) {
    const R m0 = posm[0].w;
    bool same = true;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x)
        same &= posm[i].w == m0;
    if (!__all_sync(0xffffffffu, same) && (threadIdx.x & 31) == 0) flags[0] = 1ull;
    if (blockIdx.x == 0 && threadIdx.x == 0)
        flags[1] = static_cast<unsigned long long>(__double_as_longlong(static_cast<double>(m0)));
}

// ----------------------------------------------------------------------------------------------
// The adjoint update on its own (first step of the backward sweep, or no split finish to
// carry it)
template <typename R>
__global__ void adjoint_update_kernel(int64_t n, const V4<R>* __restrict__ X, const AdjUpd<R> upd) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const V4<R> x = X[i];
    adjoint_update_at(i, x.x, x.y, x.z, upd);
}

void adjoint_update_launch(int64_t n, const void* X, const AdjUpd<float>& upd, cudaStream_t s) {
    adjoint_update_kernel<float><<<div_up(n, 256), 256, 0, s>>>(
        n, static_cast<const V4<float>*>(X), upd);
    RRG_LAUNCHED();
}

// c = s V (x, y, z; w = 0)
template <typename R>
__global__ void scale_xyz_kernel(int64_t n, const V4<R>* __restrict__ V, V4<R>* __restrict__ c,
                                 R s) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const V4<R> v = V[i];
    c[i] = v4<R>(s * v.x, s * v.y, s * v.z, R(0));
}

struct ABuf {
    void* p = nullptr;
    size_t bytes = 0;
    ~ABuf() {
        if (p) cudaFree(p);
    }
    void alloc(size_t b) {
        if (p) cudaFree(p);
        p = nullptr;
        bytes = 0;
        if (!b) return;
        cudaError_t e = cudaMalloc(&p, b);
        if (e != cudaSuccess) {
            p = nullptr;
            (void)cudaGetLastError();
            throw Error(RRG_ERR_NOMEM, std::string("adjoint: cudaMalloc failed: ") +
                                           cudaGetErrorString(e));
        }
        bytes = b;
    }
    char* c() const { return static_cast<char*>(p); }
};

}  // namespace

void launch_direct_vjp_f32(const void* posm, const void* hsoft, float uniform_hsoft, int64_t n,
                           const void* lam, void* out, cudaStream_t stream) {
    int dev = 0;
    RRG_CUDA(cudaGetDevice(&dev));
    const VjpChunks chunks = vjp_f32x2_chunks(n, num_sms(dev));
    void* part = nullptr;
    const size_t pb = vjp_f32x2_part_bytes(n, chunks.splits);
    if (pb) RRG_CUDA(cudaMallocAsync(&part, pb, stream));
    try {
        vjp_f32x2_launch(posm, hsoft, uniform_hsoft, -1.0, n, lam, out, false, part, chunks,
                         stream);
    } catch (...) {
        if (part) cudaFreeAsync(part, stream);
        throw;
    }
    if (part) RRG_CUDA(cudaFreeAsync(part, stream));
}

}  // namespace rrg

using namespace rrg;

// ================================================================================================
// Leapfrog adjoint object
// ================================================================================================
struct rrg_adjoint {
    int device = 0;
    int prec = RRG_PREC_FP32;
    size_t rsz = 4;
    int64_t n = 0;
    double dt = 0.0;
    int nsteps = 0;
    int every = 20;
    double uniform_h = 0.0;
    ABuf hsoft;
    ABuf ckpt_x, ckpt_v, ckpt_a;  // (nsteps / every + 1) x n x V4: state and a(x) there
    ABuf seg_x;            // (every + 1) x n x V4
    ABuf x, x2, v, a, u, X, V, c, g, xN, scratch, sym_slots;
    ABuf vjp_part;          // FP32: pair slots (vjp_pairs) or j-split partials of the VJP
    bool vjp_pairs = false;
    int sms = 148;
    ABuf vjp_part_a;        // FP32: force partials of the reverse steps
    ABuf w;                 // FP32: half-step velocity of the reverse steps
    ABuf mflags;            // uniform-mass check: mismatch flag, mass bits
    int splits = 1;
    bool force_sym = false;  // scratch holds the pair slots of the symmetric direct sum
    VjpChunks vjp_chunks{};
    double uniform_m = -1;  // >= 0 while every particle of the last forward has this mass
    bool mass_grad = true;  // compute dL/dm (the w slot of the position gradient)
    bool forward_done = false;
    std::string err;
};

namespace {

size_t vb(const rrg_adjoint* A) { return 4 * A->rsz * static_cast<size_t>(A->n); }

void forces(rrg_adjoint* A, const void* x, void* acc, cudaStream_t s) {
    DirectLaunch L;
    L.prec = A->prec;
    L.posm = x;
    L.hsoft = A->hsoft.p;
    L.uniform_hsoft = A->uniform_h;
    L.n = A->n;
    L.uniform_mass = A->uniform_m;
    L.epi.mode = EPI_STORE;
    L.epi.acc = acc;
    L.splits = A->splits;
    L.scratch = A->scratch.p;
    L.scratch_bytes = A->scratch.bytes;
    L.sym_scratch = A->force_sym ? A->scratch.p : nullptr;
    L.sym_scratch_bytes = A->force_sym ? A->scratch.bytes : 0;
    L.stream = s;
    launch_direct(L);
}

// Force evaluation at the positions `in` with the leapfrog epilogue. out != nullptr: correct,
// then the next step's predict (u, positions into out), storing the corrected v and a where
// vel / acc are given; out == nullptr: correct only, into vel and acc (both required).
void direct_step(rrg_adjoint* A, const void* in, void* out, void* vel, void* acc,
                 cudaStream_t s) {
    DirectLaunch L;
    L.prec = A->prec;
    L.posm = in;
    L.hsoft = A->hsoft.p;
    L.uniform_hsoft = A->uniform_h;
    L.uniform_mass = A->uniform_m;
    L.n = A->n;
    L.epi.mode = out ? EPI_CORRECT_PREDICT : EPI_CORRECT;
    L.epi.dt = A->dt;
    L.epi.u = A->u.p;
    L.epi.pos_out = out;
    L.epi.vel = vel;
    L.epi.acc = acc;
    L.splits = A->splits;
    L.scratch = A->scratch.p;
    L.scratch_bytes = A->scratch.bytes;
    L.sym_scratch = A->force_sym ? A->scratch.p : nullptr;
    L.sym_scratch_bytes = A->force_sym ? A->scratch.bytes : 0;
    L.stream = s;
    launch_direct(L);
}

// Where the forward keeps x_n: in its checkpoint slot on checkpoint steps, else in one of two
// work buffers (consecutive steps never share one).
char* forward_pos(rrg_adjoint* A, int n) {
    if (n % A->every == 0) return A->ckpt_x.c() + vb(A) * (n / A->every);
    return (n & 1) ? A->x.c() : A->x2.c();
}

// The adjoint update of step m (m < 0: none).
template <typename R>
AdjUpd<R> step_update(rrg_adjoint* A, int m) {
    AdjUpd<R> u;
    if (m < 0) return u;
    u.V = static_cast<V4<R>*>(A->V.p);
    u.c = static_cast<V4<R>*>(A->c.p);
    u.dt = static_cast<R>(A->dt);
    u.with_vn = m > 0 ? 1 : 0;
    return u;
}

// X += J(x)^T c, w slot += dm: the paired kernel in FP32, the symmetric one in FP64; then
// the update of step m (m >= 0) from the new X, in the same finish pass.
void vjp(rrg_adjoint* A, const void* x, int m, cudaStream_t s) {
    if (A->prec == RRG_PREC_FP64)
        vjp_sym_launch<double>(x, A->hsoft.p, A->uniform_h, A->n, A->c.p, A->X.p, true,
                               A->sym_slots.p, A->sms, s, step_update<double>(A, m));
    else if (A->vjp_pairs)
        vjp_pair_launch(x, A->hsoft.p, A->uniform_h, A->uniform_m, A->n, A->c.p, A->X.p, true,
                        A->vjp_part.p, A->vjp_part.bytes, A->sms, s, step_update<float>(A, m),
                        nullptr, A->mass_grad);
    else
        vjp_f32x2_launch(x, A->hsoft.p, A->uniform_h, A->uniform_m, A->n, A->c.p, A->X.p, true,
                         A->vjp_part.p, A->vjp_chunks, s, step_update<float>(A, m),
                         A->mass_grad);
}

// Sets A->uniform_m from the masses in x (one small kernel and a 16-byte read-back).
void detect_uniform_mass(rrg_adjoint* A, const void* x, cudaStream_t s) {
    RRG_CUDA(cudaMemsetAsync(A->mflags.p, 0, 16, s));
    const int blocks = static_cast<int>(std::min<int64_t>(div_up(A->n, 256), 1184));
    if (A->prec == RRG_PREC_FP64)
        uniform_mass_kernel<double><<<blocks, 256, 0, s>>>(A->n, static_cast<const V4<double>*>(x),
                                                           static_cast<unsigned long long*>(A->mflags.p));
    else
        uniform_mass_kernel<float><<<blocks, 256, 0, s>>>(A->n, static_cast<const V4<float>*>(x),
                                                          static_cast<unsigned long long*>(A->mflags.p));
    RRG_LAUNCHED();
    unsigned long long f[2] = {1, 0};
    RRG_CUDA(cudaMemcpyAsync(f, A->mflags.p, 16, cudaMemcpyDeviceToHost, s));
    RRG_CUDA(cudaStreamSynchronize(s));
    double m = 0;
    std::memcpy(&m, &f[1], 8);
    A->uniform_m = (f[0] == 0 && m >= 0) ? m : -1.0;
}

#define ADJ_ENTRY(A, ...)                                                                    \
    try {                                                                                    \
        RRG_REQUIRE((A) != nullptr, RRG_ERR_INVALID, "null adjoint");                        \
        RRG_CUDA(cudaSetDevice((A)->device));                                               \
        __VA_ARGS__;                                                                         \
        return RRG_OK;                                                                       \
    } catch (const Error& x_) {                                                              \
        if (A) (A)->err = x_.what();                                                         \
        set_thread_error(x_.what());                                                         \
        return x_.code;                                                                      \
    }

}  // namespace

extern "C" {

RRG_API rrg_status rrg_dev_direct_vjp(const void* posm, const void* hsoft, double uniform_hsoft,
                                      int64_t n, const void* lam, void* out, int precision,
                                      void* stream) {
    try {
        RRG_REQUIRE(posm && lam && out && n > 0, RRG_ERR_INVALID, "rrg_dev_direct_vjp: bad args");
        RRG_REQUIRE(precision == RRG_PREC_FP32 || precision == RRG_PREC_FP64, RRG_ERR_INVALID,
                    "rrg_dev_direct_vjp: precision must be FP32 or FP64");
        int dev = 0;
        RRG_CUDA(cudaGetDevice(&dev));
        cudaStream_t s = static_cast<cudaStream_t>(stream);
        if (precision == RRG_PREC_FP32) {
            launch_direct_vjp_f32(posm, hsoft, static_cast<float>(uniform_hsoft), n, lam, out, s);
            return RRG_OK;
        }
        void* slots = nullptr;
        const int sms = num_sms(dev);
        RRG_CUDA(cudaMallocAsync(&slots, vjp_sym_slot_bytes<double>(n, sms), s));
        try {
            vjp_sym_launch<double>(posm, hsoft, uniform_hsoft, n, lam, out, false, slots, sms, s);
        } catch (...) {
            cudaFreeAsync(slots, s);
            throw;
        }
        RRG_CUDA(cudaFreeAsync(slots, s));
        return RRG_OK;
    } catch (const Error& e) {
        set_thread_error(e.what());
        return e.code;
    }
}

RRG_API rrg_status rrg_adjoint_create(int device, int precision, int64_t n, double dt,
                                      int nsteps, int checkpoint_every, const double* soft2,
                                      rrg_adjoint** out) {
    rrg_adjoint* A = nullptr;
    try {
        RRG_REQUIRE(out && soft2, RRG_ERR_INVALID, "rrg_adjoint_create: NULL argument");
        RRG_REQUIRE(precision == RRG_PREC_FP32 || precision == RRG_PREC_FP64, RRG_ERR_INVALID,
                    "rrg_adjoint_create: precision must be FP32 or FP64");
        RRG_REQUIRE(n >= 1 && n < (int64_t(1) << 31) && nsteps >= 1 && dt > 0,
                    RRG_ERR_INVALID, "rrg_adjoint_create: bad sizes or dt");
        RRG_CUDA(cudaSetDevice(device));
        A = new rrg_adjoint();
        A->device = device;
        A->prec = precision;
        A->rsz = precision == RRG_PREC_FP64 ? 8 : 4;
        A->n = n;
        A->dt = dt;
        A->nsteps = nsteps;
        A->every = checkpoint_every <= 0 ? nsteps : std::min(checkpoint_every, nsteps);
        bool uniform = true;
        for (int64_t i = 1; i < n && uniform; ++i) uniform = soft2[i] == soft2[0];
        A->uniform_h = 0.5 * soft2[0];
        if (!uniform) {
            A->hsoft.alloc(A->rsz * n);
            std::vector<double> h(n);
            for (int64_t i = 0; i < n; ++i) h[i] = 0.5 * soft2[i];
            if (A->rsz == 8) {
                RRG_CUDA(cudaMemcpy(A->hsoft.p, h.data(), 8 * n, cudaMemcpyHostToDevice));
            } else {
                std::vector<float> hf(h.begin(), h.end());
                RRG_CUDA(cudaMemcpy(A->hsoft.p, hf.data(), 4 * n, cudaMemcpyHostToDevice));
            }
        }
        const int nck = (nsteps + A->every - 1) / A->every + 1;
        A->ckpt_x.alloc(vb(A) * nck);
        A->ckpt_v.alloc(vb(A) * nck);
        A->ckpt_a.alloc(vb(A) * nck);
        if (precision == RRG_PREC_FP64) A->seg_x.alloc(vb(A) * (A->every + 1));
        for (ABuf* b : {&A->x, &A->x2, &A->v, &A->a, &A->u, &A->X, &A->V, &A->c, &A->g, &A->xN})
            b->alloc(vb(A));
        const int sms = num_sms(device);
        A->sms = sms;
        A->splits = direct_choose_splits(precision, n, sms);
        const size_t sb = direct_scratch_bytes(precision, n, A->splits);
        // (whether the masses are equal is known only in the forward pass)
        const size_t fs = std::max(direct_sym_scratch_bytes(precision, n, true, sms),
                                   direct_sym_scratch_bytes(precision, n, false, sms));
        if (fs) {
            try {
                A->scratch.alloc(fs);
                A->force_sym = true;
            } catch (const Error&) {
                // no room for the slots: the ordered kernels
            }
        }
        if (!A->force_sym && sb) A->scratch.alloc(sb);
        if (precision == RRG_PREC_FP64) {
            A->sym_slots.alloc(vjp_sym_slot_bytes<double>(n, sms));
        } else {
            if (const size_t pairs = vjp_pair_bytes(n, sms)) {
                try {
                    A->vjp_part.alloc(pairs);
                    A->vjp_pairs = true;
                } catch (const Error&) {
                    // no room for the slots: the ordered kernel
                }
            }
            if (!A->vjp_pairs) {
                A->vjp_chunks = vjp_f32x2_chunks(n, sms);
                // the reverse steps write partials even with one split
                const size_t pb = sizeof(V4<float>) * static_cast<size_t>(n) *
                                  static_cast<size_t>(A->vjp_chunks.splits);
                A->vjp_part.alloc(pb);
                A->vjp_part_a.alloc(pb);
            }
            A->w.alloc(vb(A));
        }
        A->mflags.alloc(16);
        *out = A;
        return RRG_OK;
    } catch (const Error& e) {
        set_thread_error(e.what());
        delete A;
        return e.code;
    }
}

RRG_API rrg_status rrg_adjoint_destroy(rrg_adjoint* A) {
    if (!A) return RRG_OK;
    cudaSetDevice(A->device);
    cudaDeviceSynchronize();
    delete A;
    return RRG_OK;
}

// Forward: nsteps leapfrog steps from (x0 = (x, y, z, m) per particle, v0), on caller device
// memory (V4 of the object's precision). Saves checkpoints; writes the final state.
RRG_API rrg_status rrg_adjoint_forward(rrg_adjoint* A, const void* x0, const void* v0,
                                       void* x_out, void* v_out, void* stream) {
    ADJ_ENTRY(A, {
        RRG_REQUIRE(x0 && v0, RRG_ERR_INVALID, "rrg_adjoint_forward: NULL input");
        cudaStream_t s = static_cast<cudaStream_t>(stream);
        const size_t b = vb(A);
        char* x_0 = A->ckpt_x.c();
        RRG_CUDA(cudaMemcpyAsync(x_0, x0, b, cudaMemcpyDeviceToDevice, s));
        RRG_CUDA(cudaMemcpyAsync(A->ckpt_v.p, v0, b, cudaMemcpyDeviceToDevice, s));
        detect_uniform_mass(A, x_0, s);
        forces(A, x_0, A->ckpt_a.p, s);
        // x_1 from (x_0, v_0, a_0); then one fused launch per step (correct + next predict),
        // checkpoints written by the epilogue itself
        char* x_1 = forward_pos(A, 1);
        RRG_CUDA(cudaMemcpyAsync(x_1, x_0, b, cudaMemcpyDeviceToDevice, s));
        launch_predict(A->prec, A->n, x_1, nullptr, A->ckpt_v.p, A->ckpt_a.p, A->u.p, A->dt, s);
        for (int n = 1; n < A->nsteps; ++n) {
            const bool ck = n % A->every == 0;
            const size_t k = static_cast<size_t>(n / A->every);
            direct_step(A, forward_pos(A, n), forward_pos(A, n + 1),
                        ck ? A->ckpt_v.c() + b * k : nullptr, ck ? A->ckpt_a.c() + b * k : nullptr,
                        s);
        }
        char* x_N = forward_pos(A, A->nsteps);
        direct_step(A, x_N, nullptr, A->v.p, A->a.p, s);
        RRG_CUDA(cudaMemcpyAsync(A->xN.p, x_N, b, cudaMemcpyDeviceToDevice, s));
        if (x_out) RRG_CUDA(cudaMemcpyAsync(x_out, x_N, b, cudaMemcpyDeviceToDevice, s));
        if (v_out) RRG_CUDA(cudaMemcpyAsync(v_out, A->v.p, b, cudaMemcpyDeviceToDevice, s));
        A->forward_done = true;
    })
}

// Backward: cotangents of the final (x, v) in, gradients of the initial (x, v, m) out.
// gx_out[i] = (dL/dx, dL/dy, dL/dz, dL/dm), gv_out[i] = (dL/dvx, dL/dvy, dL/dvz, 0).
RRG_API rrg_status rrg_adjoint_backward(rrg_adjoint* A, const void* gx_final,
                                        const void* gv_final, void* gx_out, void* gv_out,
                                        void* stream) {
    ADJ_ENTRY(A, {
        RRG_REQUIRE(A->forward_done, RRG_ERR_STATE, "rrg_adjoint_backward before forward");
        RRG_REQUIRE(gx_out && gv_out, RRG_ERR_INVALID, "rrg_adjoint_backward: NULL output");
        cudaStream_t s = static_cast<cudaStream_t>(stream);
        const size_t b = vb(A);
        // X (cotangent of x, w = accumulated mass gradient), V
        if (gx_final) RRG_CUDA(cudaMemcpyAsync(A->X.p, gx_final, b, cudaMemcpyDeviceToDevice, s));
        else RRG_CUDA(cudaMemsetAsync(A->X.p, 0, b, s));
        if (gv_final) RRG_CUDA(cudaMemcpyAsync(A->V.p, gv_final, b, cudaMemcpyDeviceToDevice, s));
        else RRG_CUDA(cudaMemsetAsync(A->V.p, 0, b, s));
        // the w slot of X accumulates dL/dm: start it at zero
        RRG_CUDA(cudaMemset2DAsync(A->X.c() + 3 * A->rsz, 4 * A->rsz, 0, A->rsz, A->n, s));
        if (gv_final) {
            // v_N = v_{N-1} + dt/2 (a_{N-1} + a(x_N)): the final velocity's own dependence on
            // a(x_N) reaches x_N (and m) through one product with cotangent dt/2 V_N
            const int bl = div_up(A->n, 256);
            if (A->prec == RRG_PREC_FP64)
                scale_xyz_kernel<double><<<bl, 256, 0, s>>>(A->n, static_cast<const V4<double>*>(A->V.p),
                                                            static_cast<V4<double>*>(A->c.p), 0.5 * A->dt);
            else
                scale_xyz_kernel<float><<<bl, 256, 0, s>>>(A->n, static_cast<const V4<float>*>(A->V.p),
                                                           static_cast<V4<float>*>(A->c.p),
                                                           static_cast<float>(0.5 * A->dt));
            RRG_LAUNCHED();
            vjp(A, A->xN.p, A->nsteps - 1, s);
        } else {
            const int bl = div_up(A->n, 256);
            const int m = A->nsteps - 1;
            if (A->prec == RRG_PREC_FP64)
                adjoint_update_kernel<double><<<bl, 256, 0, s>>>(
                    A->n, static_cast<const V4<double>*>(A->X.p), step_update<double>(A, m));
            else
                adjoint_update_kernel<float><<<bl, 256, 0, s>>>(
                    A->n, static_cast<const V4<float>*>(A->X.p), step_update<float>(A, m));
            RRG_LAUNCHED();
        }
        const int nseg = (A->nsteps + A->every - 1) / A->every;
        for (int seg = nseg - 1; seg >= 0 && A->prec == RRG_PREC_FP32; --seg) {
            // FP32: reverse steps from the state at the segment's top (the next checkpoint, or
            // the final state) down to n0 + 1, each one pass of the fused VJP + force kernel;
            // x_n0 is the checkpoint itself
            const int n0 = seg * A->every;
            const int n1 = std::min(A->nsteps, n0 + A->every);
            char* xc = A->ckpt_x.c() + b * seg;
            if (n1 - n0 > 1) {
                const bool last = seg == nseg - 1;
                const size_t top = static_cast<size_t>(seg + 1);
                const void* xt = last ? A->xN.p : A->ckpt_x.c() + b * top;
                const void* vt = last ? A->v.p : A->ckpt_v.c() + b * top;
                const void* at = last ? A->a.p : A->ckpt_a.c() + b * top;
                char* xbuf[2] = {A->x.c(), A->x2.c()};
                reverse_init_kernel<<<div_up(A->n, 256), 256, 0, s>>>(
                    A->n, static_cast<const V4<float>*>(xt), static_cast<const V4<float>*>(vt),
                    static_cast<const V4<float>*>(at), static_cast<V4<float>*>(A->w.p),
                    reinterpret_cast<V4<float>*>(xbuf[(n1 - 1) & 1]), static_cast<float>(A->dt));
                RRG_LAUNCHED();
                for (int m = n1 - 1; m > n0; --m) {
                    RevStep r;
                    r.x = reinterpret_cast<const V4<float>*>(xbuf[m & 1]);
                    r.x_next = m - 1 > n0 ? reinterpret_cast<V4<float>*>(xbuf[(m - 1) & 1]) : nullptr;
                    r.w = static_cast<V4<float>*>(A->w.p);
                    r.dt = static_cast<float>(A->dt);
                    if (A->vjp_pairs)
                        vjp_pair_launch(r.x, A->hsoft.p, A->uniform_h, A->uniform_m, A->n, A->c.p,
                                        A->X.p, true, A->vjp_part.p, A->vjp_part.bytes, A->sms, s,
                                        step_update<float>(A, m - 1), &r, A->mass_grad);
                    else
                        vjp_reverse_launch(A->hsoft.p, A->uniform_h, A->uniform_m, A->n, A->c.p,
                                           A->X.p, A->vjp_part.p, A->vjp_part_a.p, A->vjp_chunks,
                                           s, step_update<float>(A, m - 1), r, A->mass_grad);
                }
            }
            vjp(A, xc, n0 - 1, s);
        }
        for (int seg = nseg - 1; seg >= 0 && A->prec == RRG_PREC_FP64; --seg) {
            const int n0 = seg * A->every;
            const int n1 = std::min(A->nsteps, n0 + A->every);
            // FP64: recompute the segment from its checkpoint: x_n0 is the checkpoint itself, x_n for
            // n0 < n < n1 go to seg_x[n - n0] (a predict, then fused steps)
            char* xc = A->ckpt_x.c() + b * seg;
            if (n1 - n0 > 1) {
                char* x1 = A->seg_x.c() + b;
                RRG_CUDA(cudaMemcpyAsync(x1, xc, b, cudaMemcpyDeviceToDevice, s));
                launch_predict(A->prec, A->n, x1, nullptr, A->ckpt_v.c() + b * seg,
                               A->ckpt_a.c() + b * seg, A->u.p, A->dt, s);
                for (int jn = 1; jn + 1 < n1 - n0; ++jn)
                    direct_step(A, A->seg_x.c() + b * jn, A->seg_x.c() + b * (jn + 1), nullptr,
                                nullptr, s);
            }
            for (int n = n1 - 1; n >= n0; --n) {
                // X += J(x_n)^T c_n (and its w slot += dm), then step n - 1's update
                vjp(A, n == n0 ? xc : A->seg_x.c() + b * (n - n0), n - 1, s);
            }
        }
        if (!A->mass_grad)
            RRG_CUDA(cudaMemset2DAsync(A->X.c() + 3 * A->rsz, 4 * A->rsz, 0, A->rsz, A->n, s));
        RRG_CUDA(cudaMemcpyAsync(gx_out, A->X.p, b, cudaMemcpyDeviceToDevice, s));
        RRG_CUDA(cudaMemcpyAsync(gv_out, A->V.p, b, cudaMemcpyDeviceToDevice, s));
    })
}

RRG_API rrg_status rrg_adjoint_set_mass_gradient(rrg_adjoint* A, int enabled) {
    ADJ_ENTRY(A, { A->mass_grad = enabled != 0; })
}

}  // extern "C"
