// Hand-written adjoint of the particle-mesh leapfrog (periodic wave potential) on sm_100a.
//
// Forward step (RectWaveIntegrationSolver::calc_step, rrgsim_integration_rect.cuh:99-112):
//   u  = 2 v + dt a;  x' = x + dt/2 u                       (predict_step_, nbody.cu:122-152)
//   M  = CIC(x', m)                                         (rm_p2mesh.cu:176-236)
//   f  = 4 pi (M / dx^3 - rho_mean)                         (wave.cu:150-153)
//   S substeps  phi_new = K_M L6(phi) + K_A phi + K_O phi_old + K_F f   (wave.cu:163-192)
//   g  = -D phi                                             (rm_p2mesh.cu:238-290)
//   a' = T(x') g                                            (rm_mesh2p.cu:48-114)
//   v' = (u + dt a') / 2                                    (correct_step_, nbody.cu:159-181)
// Every map but the two particle/grid couplings is linear, so the backward pass is:
//   - correct:  U = V'/2, A'' = A' + dt/2 V'
//   - interp:   gbar = T(x')^T A'' (a CIC-style scatter); x' gets sum_c dw_c/dx' (g_c . A'')
//   - gradient: Phi_cur += -D^T gbar
//   - substeps in reverse: (P, C) -> (K_O C, K_M L6 C + K_A C + P), F += K_F C (L6 is
//     symmetric on the periodic box, so the adjoint substep is the same stencil)
//   - source:   Mbar = 4 pi F / dx^3
//   - deposit:  m gets sum_c w_c Mbar_c (a trilinear gather, the CIC adjoint); x' gets
//               m sum_c dw_c/dx' Mbar_c (zero where the reference clamps)
//   - predict:  U += dt/2 X, V = 2 U, A = dt U, X passes through.
// The initial potential is a fixed input (the relaxation before the first step is not
// differentiated); a_0 = T(x_0) g_0 is, through x_0. The fixed-point rounding of the deposit
// is treated as the identity (its relative size is 2^-27).
#include <algorithm>
#include <cmath>
#include <string>
#include <vector>

#include "host_io.h"
#include "kernels.cuh"

namespace rrg {
namespace {

constexpr double kPi = 3.14159265358979;

__device__ __forceinline__ void interp_axis_w(double x, double dmin, double dx, int nx, int& i0,
                                              int& i1, double& w) {
    const double f = (x - dmin) / dx - 0.5;
    const int a = static_cast<int>(floorf(static_cast<float>(f)));
    w = f - a;
    i0 = max(0, min(a, nx - 1));
    i1 = max(0, min(a + 1, nx - 1));
}

// interp adjoint with the correct adjoint before it: with A' = A + h V (the correction
// v' = (u + dt a) / 2; V null: A alone), gbar += T(x)^T A' (atomics, when gbar != nullptr; gbar
// holds 4 values per cell, the fourth unused); X = sum dW/dx (g . A')
template <typename R>
__global__ void __launch_bounds__(256) interp_adjoint_kernel(int64_t n, const V4<R>* __restrict__ posm,
                                                             GridDev g, const V4<R>* __restrict__ acc4,
                                                             const V4<R>* __restrict__ A,
                                                             const V4<R>* __restrict__ V, R h,
                                                             R* __restrict__ gbar,
                                                             V4<R>* __restrict__ X) {
    const int64_t p = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const bool active = p < n;
    V4<R> q = v4<R>(0, 0, 0, 0), a = v4<R>(0, 0, 0, 0);
    if (active) {
        q = posm[p];
        a = A[p];
        if (V) {
            const V4<R> v = V[p];
            a.x += h * v.x;
            a.y += h * v.y;
            a.z += h * v.z;
        }
    }
    int ii[2], jj[2], kk[2];
    double wx, wy, wz;
    interp_axis_w(q.x, g.domain_min, g.dx, g.nx, ii[0], ii[1], wx);
    interp_axis_w(q.y, g.domain_min, g.dx, g.nx, jj[0], jj[1], wy);
    interp_axis_w(q.z, g.domain_min, g.dx, g.nx, kk[0], kk[1], wz);
    R wxs[2] = {R(1) - R(wx), R(wx)}, wys[2] = {R(1) - R(wy), R(wy)},
      wzs[2] = {R(1) - R(wz), R(wz)};
    const R inv = R(1.0 / g.dx);
    const R dws[2] = {-inv, inv};
    const int64_t nx = g.nx;
    R gx = 0, gy = 0, gz = 0;
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int64_t c = kk[k] * nx * nx + jj[j] * nx + ii[i];
                const V4<R> f = acc4[c];
                const R s = f.x * a.x + f.y * a.y + f.z * a.z;
                gx += dws[i] * wys[j] * wzs[k] * s;
                gy += wxs[i] * dws[j] * wzs[k] * s;
                gz += wxs[i] * wys[j] * dws[k] * s;
            }
    if (active) X[p] = v4<R>(gx, gy, gz, R(0));
    if (!gbar) return;
    // Lanes of the same eight corners that sit next to each other (particles sorted by cell) are
    // summed by a segmented scan and their last lane adds the sums: the atomics of a dense cell
    // otherwise queue on its corners (262,144 sorted disk particles on 64^3: 67 us with one set
    // of atomics per particle, 41 unsorted). As the particles drift from the order of the first
    // step, runs fragment: a warp of more than four first sorts its (cell, lane) pairs (bitonic, as
    // the deposit does). A warp of many runs adds lane by lane. Over 200 steps on average, with no
    // sort and always five scan steps -> here: FP32 32.1 -> 18.5 us, FP64 96.7 -> 47.8.
    auto side = [&](const int e[2]) {
        return e[0] != e[1] ? e[0] + 1 : (e[0] == 0 ? 0 : g.nx);
    };
    const int n1 = g.nx + 1;  // (n1^3 < 2^31)
    int key = active ? side(ii) + n1 * (side(jj) + n1 * side(kk)) : -1;
    const int lane = threadIdx.x & 31;
    constexpr int sparse = 24;
    {
        const int below = __shfl_up_sync(0xffffffffu, key, 1);
        const int runs = __popc(__ballot_sync(0xffffffffu, lane == 0 || below != key));
        if (runs > 4 && runs < sparse && g.nx <= 405) {  // (warp-uniform; n1^3 < 2^26)
            int kv = ((key + 1) << 5) | lane;
#pragma unroll
            for (int k = 2; k <= 32; k <<= 1) {
#pragma unroll
                for (int j = k >> 1; j > 0; j >>= 1) {
                    const int pk = __shfl_xor_sync(0xffffffffu, kv, j);
                    const bool ascending = (lane & k) == 0, lower = (lane & j) == 0;
                    if (lower == ascending ? pk < kv : pk > kv) kv = pk;
                }
            }
            key = (kv >> 5) - 1;
            const int src = kv & 31;
            a.x = __shfl_sync(0xffffffffu, a.x, src);
            a.y = __shfl_sync(0xffffffffu, a.y, src);
            a.z = __shfl_sync(0xffffffffu, a.z, src);
            const R mx = __shfl_sync(0xffffffffu, wxs[1], src);
            const R my = __shfl_sync(0xffffffffu, wys[1], src);
            const R mz = __shfl_sync(0xffffffffu, wzs[1], src);
            wxs[0] = R(1) - mx;
            wxs[1] = mx;
            wys[0] = R(1) - my;
            wys[1] = my;
            wzs[0] = R(1) - mz;
            wzs[1] = mz;
            // side back to the two indices
            auto indices = [&](int s, int e[2]) {
                e[0] = max(s - 1, 0);
                e[1] = min(s, g.nx - 1);
            };
            const int c = max(key, 0), yz = c / n1;
            indices(c - yz * n1, ii);
            indices(yz % n1, jj);
            indices(yz / n1, kk);
        }
    }
    const int below = __shfl_up_sync(0xffffffffu, key, 1);
    const int above = __shfl_down_sync(0xffffffffu, key, 1);
    const unsigned heads = __ballot_sync(0xffffffffu, lane == 0 || below != key);
    const bool scan = __popc(heads) < sparse;  // warp-uniform
    const bool tail = !scan || lane == 31 || above != key;
    const int first = 31 - __clz(heads & (0xffffffffu >> (31 - lane)));  // the run's first lane
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const R w = wxs[i] * wys[j] * wzs[k];
                R vx = w * a.x, vy = w * a.y, vz = w * a.z;
                if (scan) {
                    // distance d only while some run has more than d lanes
                    unsigned longer = ~heads;
                    for (int d = 1; longer != 0u; d <<= 1) {
                        const R tx = __shfl_up_sync(0xffffffffu, vx, d);
                        const R ty = __shfl_up_sync(0xffffffffu, vy, d);
                        const R tz = __shfl_up_sync(0xffffffffu, vz, d);
                        if (lane - d >= first) {
                            vx += tx;
                            vy += ty;
                            vz += tz;
                        }
                        longer &= longer >> d;
                    }
                }
                if (!tail || key < 0) continue;
                const int64_t c = kk[k] * nx * nx + jj[j] * nx + ii[i];
                if constexpr (sizeof(R) == 4) {
                    // one 16-byte vector atomic per corner instead of three scalar ones
                    atomicAdd(reinterpret_cast<float4*>(gbar) + c, make_float4(vx, vy, vz, 0.f));
                } else {
                    atomicAdd(gbar + 4 * c, vx);
                    atomicAdd(gbar + 4 * c + 1, vy);
                    atomicAdd(gbar + 4 * c + 2, vz);
                }
            }
}

// gradient adjoint: phi += -1/dx D^T gbar (D: central inside, one-sided on the faces)
template <typename R>
__device__ __forceinline__ R dT_axis(const R* gb, int comp, int64_t c, int j, int n, int64_t st) {
    R s = 0;
    if (j - 1 >= 0) s += (j - 1 == 0 ? R(1) : R(0.5)) * gb[4 * (c - st) + comp];
    if (j + 1 <= n - 1) s -= (j + 1 == n - 1 ? R(1) : R(0.5)) * gb[4 * (c + st) + comp];
    if (j == 0) s -= gb[4 * c + comp];
    if (j == n - 1) s += gb[4 * c + comp];
    return s;
}

template <typename R>
__global__ void __launch_bounds__(256) gradient_adjoint_kernel(int nx, R coef, const R* __restrict__ gbar,
                                                               R* __restrict__ phi_bar) {
    const int64_t c = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const int64_t nc = static_cast<int64_t>(nx) * nx * nx;
    if (c >= nc) return;
    const int x = static_cast<int>(c % nx), y = static_cast<int>((c / nx) % nx),
              z = static_cast<int>(c / (static_cast<int64_t>(nx) * nx));
    const R s = dT_axis(gbar, 0, c, x, nx, 1) + dT_axis(gbar, 1, c, y, nx, nx) +
                dT_axis(gbar, 2, c, z, nx, static_cast<int64_t>(nx) * nx);
    phi_bar[c] += coef * s;
}

// deposit adjoint at x: m_bar += sum_c W_c Mbar_c; Xd = m sum_c dW_c/dx Mbar_c
// (CIC weights of rm_p2mesh.cu:191-216; derivative zero where u is clamped)
__device__ __forceinline__ void cic_axis_d(double x, double dmin, double inv_dx, int nx, int& i0,
                                           int& i1, double& w0, double& w1, double& du) {
    double u = (x - dmin) * inv_dx - 0.5;
    const double hi = static_cast<double>(nx - 1) - 1e-6;
    du = inv_dx;
    if (!(u >= 0.0)) {
        u = 0.0;
        du = 0.0;
    }
    if (u > hi) {
        u = hi;
        du = 0.0;
    }
    i0 = static_cast<int>(floor(u));
    i1 = min(i0 + 1, nx - 1);
    const double f = u - i0;
    w0 = 1.0 - f;
    w1 = f;
}

// and the predict adjoint after it, with U = V / 2: Xt = X + Xi + Xd (w: m_bar accumulates);
// U += dt/2 Xt; V = 2 U; A = dt U; X = Xt
template <typename R>
__global__ void __launch_bounds__(256) deposit_predict_adjoint_kernel(
    int64_t n, const V4<R>* __restrict__ posm, GridDev g, const R* __restrict__ F, R mscale,
    V4<R>* __restrict__ X, const V4<R>* __restrict__ Xi, V4<R>* __restrict__ V,
    V4<R>* __restrict__ A, R dt) {
    const int64_t p = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (p >= n) return;
    const V4<R> q = posm[p];
    int ii[2], jj[2], kk[2];
    double wx[2], wy[2], wz[2], dux, duy, duz;
    cic_axis_d(q.x, g.domain_min, g.inv_dx, g.nx, ii[0], ii[1], wx[0], wx[1], dux);
    cic_axis_d(q.y, g.domain_min, g.inv_dx, g.nx, jj[0], jj[1], wy[0], wy[1], duy);
    cic_axis_d(q.z, g.domain_min, g.inv_dx, g.nx, kk[0], kk[1], wz[0], wz[1], duz);
    const double sgn[2] = {-1.0, 1.0};
    const int64_t nx = g.nx;
    double mb = 0, gx = 0, gy = 0, gz = 0;
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const double Mb = static_cast<double>(mscale) *
                                  static_cast<double>(F[kk[k] * nx * nx + jj[j] * nx + ii[i]]);
                mb += wx[i] * wy[j] * wz[k] * Mb;
                gx += sgn[i] * dux * wy[j] * wz[k] * Mb;
                gy += wx[i] * sgn[j] * duy * wz[k] * Mb;
                gz += wx[i] * wy[j] * sgn[k] * duz * Mb;
            }
    const double m = q.w;
    const V4<R> x = X[p], xi = Xi[p], v = V[p];
    const R tx = x.x + xi.x + static_cast<R>(m * gx), ty = x.y + xi.y + static_cast<R>(m * gy),
            tz = x.z + xi.z + static_cast<R>(m * gz);
    const R h = dt * R(0.5);
    const R ux = R(0.5) * v.x + h * tx, uy = R(0.5) * v.y + h * ty, uz = R(0.5) * v.z + h * tz;
    X[p] = v4<R>(tx, ty, tz, x.w + static_cast<R>(mb));
    V[p] = v4<R>(R(2) * ux, R(2) * uy, R(2) * uz, R(0));
    A[p] = v4<R>(dt * ux, dt * uy, dt * uz, R(0));
}

// The positions' cotangent without its fourth component, the accelerations' zero
template <typename R>
__global__ void cotangent_start_kernel(int64_t n, V4<R>* X, V4<R>* A) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    X[i].w = R(0);
    A[i] = v4<R>(R(0), R(0), R(0), R(0));
}

template <typename R>
__global__ void add_xyz_kernel(int64_t n, V4<R>* __restrict__ X, const V4<R>* __restrict__ Y) {
    const int64_t p = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (p >= n) return;
    V4<R> x = X[p];
    const V4<R> y = Y[p];
    x.x += y.x;
    x.y += y.y;
    x.z += y.z;
    X[p] = x;
}

// out[i] = in[dest[i]]: particles back into the caller's order
template <typename R>
__global__ void __launch_bounds__(256) gather_kernel(int64_t n, const uint32_t* __restrict__ dest,
                                                     const V4<R>* __restrict__ in,
                                                     V4<R>* __restrict__ out) {
    const int64_t p = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (p < n) out[p] = in[dest[p]];
}

struct PBuf {
    void* p = nullptr;
    size_t bytes = 0;
    ~PBuf() {
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
            throw Error(RRG_ERR_NOMEM, std::string("pm adjoint: cudaMalloc failed: ") +
                                           cudaGetErrorString(e));
        }
        bytes = b;
    }
    char* c() const { return static_cast<char*>(p); }
};

}  // namespace
}  // namespace rrg

using namespace rrg;

struct rrg_pm_adjoint {
    int device = 0;
    int prec = RRG_PREC_FP32;
    size_t rsz = 4;
    int64_t n = 0;
    double dt = 0.0;
    int nsteps = 0, every = 20, substeps = 20;
    rrg_grid_info grid{};
    GridDev gdev{};
    WaveCoef wc{};
    double rho_mean = 0.0;
    int64_t nc = 0;
    int shift_s = 0;
    PBuf x, v, a, u, mg, src, phi[2], acc4;
    PBuf ck_x, ck_v, ck_a, ck_phi;     // per checkpoint: x, v, a, phi_prev, phi_cur
    PBuf seg_x, seg_phi;               // per step of a segment: x_{n+1}, phi_cur_{n+1}
    PBuf X, V, A, Xi, gbar, Cb, Pb, F;
    // The particles' order inside the object: sorted by the CIC cell of x0 (dest: a particle's
    // slot), so that deposits, gathers and the field cotangent's scatter of a warp meet in few
    // cells. Made by each forward pass, undone where states and gradients leave the object.
    bool sort = false;
    PBuf keys, dest, counts, offsets, cursor, temp;
    size_t temp_bytes = 0;
    bool forward_done = false;
    // Recorded on the first step of a pass and replayed (own buffers only): [0] a forward step, [1]
    // a step's reversed substeps, each for both orders of the two levels that the substeps swap.
    cudaGraphExec_t graphs[2][2] = {};
    cudaStream_t recording = nullptr;
    const void *phi_a = nullptr, *cot_a = nullptr;  // phi[0] and Cb as allocated
    std::string err;
    ~rrg_pm_adjoint() {
        for (auto& kind : graphs)
            for (cudaGraphExec_t g : kind)
                if (g) cudaGraphExecDestroy(g);
        if (recording) cudaStreamDestroy(recording);
    }
};

namespace {

size_t pvb(const rrg_pm_adjoint* P) { return 4 * P->rsz * static_cast<size_t>(P->n); }
size_t gvb(const rrg_pm_adjoint* P) { return P->rsz * static_cast<size_t>(P->nc); }

// Runs enqueue(stream), which launches `kernels` kernels on the object's buffers: recorded as a graph
// once and replayed on s. From 4 steps a pass on, where the launches saved pay for the recording
// (~150 us; a launch costs the host 2.3 us, a graph of a step 7: 262,144 particles on 64^3, 10 steps
// forward and backward, 2.69 -> 2.16 ms). While s itself is being captured, plain launches.
template <typename F>
void replay(rrg_pm_adjoint* P, cudaGraphExec_t& exec, int kernels, cudaStream_t s, F&& enqueue) {
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    const bool known = cudaStreamIsCapturing(s, &status) == cudaSuccess;
    if (!known) (void)cudaGetLastError();
    if (P->nsteps < 4 || !known || status != cudaStreamCaptureStatusNone) {
        enqueue(s);
        return;
    }
    if (!exec) {
        if (!P->recording)
            RRG_CUDA(cudaStreamCreateWithFlags(&P->recording, cudaStreamNonBlocking));
        cudaGraph_t g = nullptr;
        RRG_CUDA(cudaStreamBeginCapture(P->recording, cudaStreamCaptureModeThreadLocal));
        set_capturing(true);
        try {
            enqueue(P->recording);
        } catch (...) {
            set_capturing(false);
            cudaStreamEndCapture(P->recording, &g);
            if (g) cudaGraphDestroy(g);
            throw;
        }
        set_capturing(false);
        RRG_CUDA(cudaStreamEndCapture(P->recording, &g));
        const cudaError_t e = cudaGraphInstantiate(&exec, g, 0);
        cudaGraphDestroy(g);
        if (e != cudaSuccess) exec = nullptr;
        RRG_CUDA(e);
    }
    RRG_CUDA(cudaGraphLaunch(exec, s));
    count_launches(kernels);
}

// one PM step in place on (x, v, a, phi[0] = prev, phi[1] = cur); mg is zero before and after
void pm_step(rrg_pm_adjoint* P, cudaStream_t s) {
    PmParticleArgs a{};
    a.prec = P->prec;
    a.n = P->n;
    a.posm = P->x.p;
    a.vel = P->v.p;
    a.acc = P->a.p;
    a.u = P->u.p;
    a.acc4 = P->acc4.p;
    a.g = P->gdev;
    a.shift_s = P->shift_s;
    a.mgrid = static_cast<unsigned long long*>(P->mg.p);
    a.dt = P->dt;
    auto* mg = static_cast<unsigned long long*>(P->mg.p);
    replay(P, P->graphs[0][P->phi[0].p == P->phi_a], P->substeps + 4, s, [&](cudaStream_t t) {
        launch_pm_particles(a, PM_PREDICT_DEPOSIT, t);
        launch_wave_source(P->prec, P->grid.nx, mg, P->shift_s, P->grid.dx, P->rho_mean, 1.0,
                           P->src.p, mg, t);
        // phi[1] current, phi[0] previous: the new level overwrites phi[0], then roles swap
        void *cur = P->phi[1].p, *old = P->phi[0].p;
        for (int k = 0; k < P->substeps; ++k) {
            launch_wave_step(P->prec, P->grid.nx, cur, old, P->src.p, P->wc, nullptr, t);
            std::swap(cur, old);
        }
        launch_gradient(P->prec, P->grid.nx, P->grid.dx, cur, P->acc4.p, t);
        launch_pm_particles(a, PM_INTERP_CORRECT | PM_WRITE_SYNC, t);
    });
    if (P->substeps % 2 == 1) std::swap(P->phi[0].p, P->phi[1].p);
}

// caller's particle array (n x 4) into the object's order, and back
void take_in(rrg_pm_adjoint* P, const void* in, void* to, cudaStream_t s) {
    if (P->sort)
        launch_permute(P->n, 4 * P->rsz, static_cast<const uint32_t*>(P->dest.p), in, to, s);
    else
        RRG_CUDA(cudaMemcpyAsync(to, in, pvb(P), cudaMemcpyDeviceToDevice, s));
}

void give_back(rrg_pm_adjoint* P, const void* from, void* out, cudaStream_t s) {
    if (!P->sort) {
        RRG_CUDA(cudaMemcpyAsync(out, from, pvb(P), cudaMemcpyDeviceToDevice, s));
        return;
    }
    const int b = div_up(P->n, 256);
    const auto* d = static_cast<const uint32_t*>(P->dest.p);
    if (P->prec == RRG_PREC_FP64)
        gather_kernel<double><<<b, 256, 0, s>>>(P->n, d, static_cast<const V4<double>*>(from),
                                               static_cast<V4<double>*>(out));
    else
        gather_kernel<float><<<b, 256, 0, s>>>(P->n, d, static_cast<const V4<float>*>(from),
                                              static_cast<V4<float>*>(out));
    RRG_LAUNCHED();
}

template <typename R>
void backward_step(rrg_pm_adjoint* P, const void* xn1, const void* phin1, cudaStream_t s) {
    const int64_t n = P->n, nc = P->nc;
    const int bp = div_up(n, 256), bg = div_up(nc, 256);
    auto* X = static_cast<V4<R>*>(P->X.p);
    auto* V = static_cast<V4<R>*>(P->V.p);
    auto* A = static_cast<V4<R>*>(P->A.p);
    auto* Xi = static_cast<V4<R>*>(P->Xi.p);
    const R dt = static_cast<R>(P->dt);
    launch_gradient(P->prec, P->grid.nx, P->grid.dx, phin1, P->acc4.p, s);
    RRG_CUDA(cudaMemsetAsync(P->gbar.p, 0, P->gbar.bytes, s));
    interp_adjoint_kernel<R><<<bp, 256, 0, s>>>(n, static_cast<const V4<R>*>(xn1), P->gdev,
                                                static_cast<const V4<R>*>(P->acc4.p), A, V,
                                                dt * R(0.5), static_cast<R*>(P->gbar.p), Xi);
    RRG_LAUNCHED();
    // Cb holds the cotangent of the current level, Pb that of the one before over K_O (each
    // reversed substep leaves C in its place, whose share of the level before is K_O C)
    gradient_adjoint_kernel<R><<<bg, 256, 0, s>>>(P->grid.nx, static_cast<R>(-1.0 / P->grid.dx),
                                                  static_cast<const R*>(P->gbar.p),
                                                  static_cast<R*>(P->Cb.p));
    RRG_LAUNCHED();
    replay(P, P->graphs[1][P->Cb.p == P->cot_a], P->substeps, s, [&](cudaStream_t t) {
        RRG_CUDA(cudaMemsetAsync(P->F.p, 0, P->F.bytes, t));
        void *cur = P->Cb.p, *old = P->Pb.p;
        for (int k = 0; k < P->substeps; ++k) {
            launch_wave_adjoint_step(P->prec, P->grid.nx, cur, old, P->F.p, P->wc.K_MAIN,
                                     P->wc.K_ACTUAL, P->wc.K_OLD, P->wc.K_F, t);
            std::swap(cur, old);
        }
    });
    if (P->substeps % 2 == 1) std::swap(P->Cb.p, P->Pb.p);
    deposit_predict_adjoint_kernel<R><<<bp, 256, 0, s>>>(
        n, static_cast<const V4<R>*>(xn1), P->gdev, static_cast<const R*>(P->F.p),
        static_cast<R>(4.0 * kPi / (P->grid.dx * P->grid.dx * P->grid.dx)), X, Xi, V, A, dt);
    RRG_LAUNCHED();
}

#define PMA_ENTRY(P, ...)                                                                    \
    try {                                                                                    \
        RRG_REQUIRE((P) != nullptr, RRG_ERR_INVALID, "null pm adjoint");                     \
        RRG_CUDA(cudaSetDevice((P)->device));                                                \
        __VA_ARGS__;                                                                         \
        return RRG_OK;                                                                       \
    } catch (const Error& x_) {                                                              \
        if (P) (P)->err = x_.what();                                                         \
        set_thread_error(x_.what());                                                         \
        return x_.code;                                                                      \
    }

}  // namespace

extern "C" {

RRG_API rrg_status rrg_pm_adjoint_create(int device, int precision, int64_t n, double m_max,
                                         const rrg_grid_info* grid, const rrg_wave_params* wave,
                                         double total_mass_for_rho, double dt, int nsteps,
                                         int checkpoint_every, rrg_pm_adjoint** out) {
    rrg_pm_adjoint* P = nullptr;
    try {
        RRG_REQUIRE(out && grid && wave, RRG_ERR_INVALID, "rrg_pm_adjoint_create: NULL argument");
        RRG_REQUIRE(precision == RRG_PREC_FP32 || precision == RRG_PREC_FP64, RRG_ERR_INVALID,
                    "rrg_pm_adjoint_create: precision must be FP32 or FP64");
        RRG_REQUIRE(n >= 1 && nsteps >= 1 && dt > 0 && grid->nx >= 2 && grid->nx <= 1024,
                    RRG_ERR_INVALID, "rrg_pm_adjoint_create: bad sizes");
        RRG_CUDA(cudaSetDevice(device));
        P = new rrg_pm_adjoint();
        P->device = device;
        P->prec = precision;
        P->rsz = precision == RRG_PREC_FP64 ? 8 : 4;
        P->n = n;
        P->dt = dt;
        P->nsteps = nsteps;
        P->every = checkpoint_every <= 0 ? nsteps : std::min(checkpoint_every, nsteps);
        P->substeps = wave->iterations;
        P->grid = *grid;
        P->gdev.nx = grid->nx;
        P->gdev.dx = grid->dx;
        P->gdev.domain_min = grid->domain_min;
        P->gdev.inv_dx = 1.0 / grid->dx;
        P->gdev.sim_l = grid->sim_l;
        P->nc = static_cast<int64_t>(grid->nx) * grid->nx * grid->nx;
        const double L = grid->nx * grid->dx;
        P->rho_mean = total_mass_for_rho / (L * L * L);
        {
            int e = 0;
            std::frexp(m_max > 0 ? m_max : 1.0, &e);
            P->shift_s = 26 - e;
        }
        const double C = wave->wave_speed, DT = wave->dt, DX = grid->dx;
        const double Q = wave->diss_base * C * DT * 0.5, W = 1 + Q,
                     K = C * C * DT * DT / (DX * DX);
        P->wc.K_MAIN = K / W;
        P->wc.K_F = -C * C * DT * DT / W;
        P->wc.K_ACTUAL = 2 * (1 - 3 * K) / W;
        P->wc.K_OLD = (Q - 1) / W;
        P->wc.bc_type = RRG_BC_PERIODIC;
        P->wc.keep_layer = 0;
        P->wc.C = C;
        P->wc.DT = DT;
        P->wc.DX = DX;
        P->wc.domain_min = grid->domain_min;
        const size_t pb = pvb(P), gb = gvb(P);
        for (PBuf* b : {&P->x, &P->v, &P->a, &P->u, &P->X, &P->V, &P->A, &P->Xi})
            b->alloc(pb);
        P->mg.alloc(8 * P->nc);
        for (PBuf* b : {&P->src, &P->phi[0], &P->phi[1], &P->Cb, &P->Pb, &P->F}) b->alloc(gb);
        P->phi_a = P->phi[0].p;
        P->cot_a = P->Cb.p;
        P->acc4.alloc(4 * gb);
        P->gbar.alloc(4 * gb);
        // sorting costs ~50 us a forward pass and saves ~0.2 ns per particle and deposit (262,144
        // disk particles on 64^3: predict and deposit 66 -> 9 us, the field cotangent's scatter
        // 41 -> 13 us), two deposits and a scatter a step
        P->sort = n * nsteps >= (int64_t(1) << 18) && n < (int64_t(1) << 31);
        if (P->sort) {
            P->keys.alloc(4 * n);
            P->dest.alloc(4 * n);
            for (PBuf* b : {&P->counts, &P->offsets, &P->cursor}) b->alloc(4 * (P->nc + 1));
            P->temp_bytes = sort_scan_temp_bytes(P->nc);
            P->temp.alloc(std::max<size_t>(P->temp_bytes, 256));
        }
        const int nck = (nsteps + P->every - 1) / P->every;
        P->ck_x.alloc(pb * nck);
        P->ck_v.alloc(pb * nck);
        P->ck_a.alloc(pb * nck);
        P->ck_phi.alloc(2 * gb * nck);
        P->seg_x.alloc(pb * P->every);
        P->seg_phi.alloc(gb * P->every);
        *out = P;
        return RRG_OK;
    } catch (const Error& e) {
        set_thread_error(e.what());
        delete P;
        return e.code;
    }
}

RRG_API rrg_status rrg_pm_adjoint_destroy(rrg_pm_adjoint* P) {
    if (!P) return RRG_OK;
    cudaSetDevice(P->device);
    cudaDeviceSynchronize();
    delete P;
    return RRG_OK;
}

// Forward from x0[i] = (x, y, z, m), v0 (n x 4 of the precision) and the initial wave levels
// phi_prev0, phi_cur0 (nx^3): a_0 = T(x_0) g(phi_cur0), then nsteps PM steps. x_out / v_out /
// phi_out (may be NULL) receive the final positions, velocities and current level.
RRG_API rrg_status rrg_pm_adjoint_forward(rrg_pm_adjoint* P, const void* x0, const void* v0,
                                          const void* phi_prev0, const void* phi_cur0,
                                          void* x_out, void* v_out, void* phi_out,
                                          void* stream) {
    PMA_ENTRY(P, {
        cudaStream_t s = static_cast<cudaStream_t>(stream);
        const size_t pb = pvb(P), gb = gvb(P);
        if (P->sort) {
            RRG_CUDA(cudaMemsetAsync(P->counts.p, 0, P->counts.bytes, s));
            RRG_CUDA(cudaMemsetAsync(P->cursor.p, 0, P->cursor.bytes, s));
            launch_cell_keys(P->prec, P->n, x0, nullptr, P->gdev, static_cast<uint32_t*>(P->keys.p),
                             static_cast<uint32_t*>(P->counts.p), s);
            launch_scan_counts(static_cast<const uint32_t*>(P->counts.p),
                               static_cast<uint32_t*>(P->offsets.p), P->nc, P->temp.p,
                               P->temp_bytes, s);
            launch_sort_dest(P->n, static_cast<const uint32_t*>(P->keys.p),
                             static_cast<const uint32_t*>(P->offsets.p),
                             static_cast<uint32_t*>(P->cursor.p),
                             static_cast<uint32_t*>(P->dest.p), s);
        }
        RRG_CUDA(cudaMemsetAsync(P->mg.p, 0, P->mg.bytes, s));
        take_in(P, x0, P->x.p, s);
        take_in(P, v0, P->v.p, s);
        RRG_CUDA(cudaMemcpyAsync(P->phi[0].p, phi_prev0, gb, cudaMemcpyDeviceToDevice, s));
        RRG_CUDA(cudaMemcpyAsync(P->phi[1].p, phi_cur0, gb, cudaMemcpyDeviceToDevice, s));
        launch_gradient(P->prec, P->grid.nx, P->grid.dx, P->phi[1].p, P->acc4.p, s);
        launch_interp(P->prec, P->n, P->x.p, nullptr, P->gdev, P->acc4.p, P->a.p, s);
        for (int k = 0; k < P->nsteps; ++k) {
            if (k % P->every == 0) {
                const int c = k / P->every;
                RRG_CUDA(cudaMemcpyAsync(P->ck_x.c() + pb * c, P->x.p, pb, cudaMemcpyDeviceToDevice, s));
                RRG_CUDA(cudaMemcpyAsync(P->ck_v.c() + pb * c, P->v.p, pb, cudaMemcpyDeviceToDevice, s));
                RRG_CUDA(cudaMemcpyAsync(P->ck_a.c() + pb * c, P->a.p, pb, cudaMemcpyDeviceToDevice, s));
                RRG_CUDA(cudaMemcpyAsync(P->ck_phi.c() + 2 * gb * c, P->phi[0].p, gb, cudaMemcpyDeviceToDevice, s));
                RRG_CUDA(cudaMemcpyAsync(P->ck_phi.c() + 2 * gb * c + gb, P->phi[1].p, gb, cudaMemcpyDeviceToDevice, s));
            }
            pm_step(P, s);
        }
        if (x_out) give_back(P, P->x.p, x_out, s);
        if (v_out) give_back(P, P->v.p, v_out, s);
        if (phi_out) RRG_CUDA(cudaMemcpyAsync(phi_out, P->phi[1].p, gb, cudaMemcpyDeviceToDevice, s));
        P->forward_done = true;
    })
}

// Backward: cotangents of the final x (n x 4, w ignored) and v in (NULL = zero); out gx[i] =
// (dL/dx, dL/dy, dL/dz, dL/dm) and gv[i] of the initial state. The initial potential is held
// fixed.
RRG_API rrg_status rrg_pm_adjoint_backward(rrg_pm_adjoint* P, const void* gx_final,
                                           const void* gv_final, void* gx_out, void* gv_out,
                                           void* stream) {
    PMA_ENTRY(P, {
        RRG_REQUIRE(P->forward_done, RRG_ERR_STATE, "rrg_pm_adjoint_backward before forward");
        cudaStream_t s = static_cast<cudaStream_t>(stream);
        const size_t pb = pvb(P), gb = gvb(P);
        if (gx_final) take_in(P, gx_final, P->X.p, s);
        else RRG_CUDA(cudaMemsetAsync(P->X.p, 0, pb, s));
        if (gv_final) take_in(P, gv_final, P->V.p, s);
        else RRG_CUDA(cudaMemsetAsync(P->V.p, 0, pb, s));
        // (a strided memset takes 149 us at 262,144 particles, this kernel 3)
        if (P->prec == RRG_PREC_FP64)
            cotangent_start_kernel<double><<<div_up(P->n, 256), 256, 0, s>>>(
                P->n, static_cast<V4<double>*>(P->X.p), static_cast<V4<double>*>(P->A.p));
        else
            cotangent_start_kernel<float><<<div_up(P->n, 256), 256, 0, s>>>(
                P->n, static_cast<V4<float>*>(P->X.p), static_cast<V4<float>*>(P->A.p));
        RRG_LAUNCHED();
        RRG_CUDA(cudaMemsetAsync(P->Cb.p, 0, gb, s));
        RRG_CUDA(cudaMemsetAsync(P->Pb.p, 0, gb, s));
        const int nseg = (P->nsteps + P->every - 1) / P->every;
        for (int seg = nseg - 1; seg >= 0; --seg) {
            const int n0 = seg * P->every, n1 = std::min(P->nsteps, n0 + P->every);
            RRG_CUDA(cudaMemcpyAsync(P->x.p, P->ck_x.c() + pb * seg, pb, cudaMemcpyDeviceToDevice, s));
            RRG_CUDA(cudaMemcpyAsync(P->v.p, P->ck_v.c() + pb * seg, pb, cudaMemcpyDeviceToDevice, s));
            RRG_CUDA(cudaMemcpyAsync(P->a.p, P->ck_a.c() + pb * seg, pb, cudaMemcpyDeviceToDevice, s));
            RRG_CUDA(cudaMemcpyAsync(P->phi[0].p, P->ck_phi.c() + 2 * gb * seg, gb, cudaMemcpyDeviceToDevice, s));
            RRG_CUDA(cudaMemcpyAsync(P->phi[1].p, P->ck_phi.c() + 2 * gb * seg + gb, gb, cudaMemcpyDeviceToDevice, s));
            for (int k = n0; k < n1; ++k) {
                pm_step(P, s);
                RRG_CUDA(cudaMemcpyAsync(P->seg_x.c() + pb * (k - n0), P->x.p, pb, cudaMemcpyDeviceToDevice, s));
                RRG_CUDA(cudaMemcpyAsync(P->seg_phi.c() + gb * (k - n0), P->phi[1].p, gb, cudaMemcpyDeviceToDevice, s));
            }
            for (int k = n1 - 1; k >= n0; --k) {
                const void* xk1 = P->seg_x.c() + pb * (k - n0);
                const void* pk1 = P->seg_phi.c() + gb * (k - n0);
                if (P->prec == RRG_PREC_FP64) backward_step<double>(P, xk1, pk1, s);
                else backward_step<float>(P, xk1, pk1, s);
            }
        }
        // a_0 = T(x_0) g(phi_cur0): its cotangent A reaches x_0 (the grid is held fixed)
        RRG_CUDA(cudaMemcpyAsync(P->x.p, P->ck_x.p, pb, cudaMemcpyDeviceToDevice, s));
        launch_gradient(P->prec, P->grid.nx, P->grid.dx, P->ck_phi.c() + gb, P->acc4.p, s);
        const int bp = div_up(P->n, 256);
        if (P->prec == RRG_PREC_FP64) {
            interp_adjoint_kernel<double><<<bp, 256, 0, s>>>(
                P->n, static_cast<const V4<double>*>(P->x.p), P->gdev,
                static_cast<const V4<double>*>(P->acc4.p), static_cast<const V4<double>*>(P->A.p),
                nullptr, 0.0, nullptr, static_cast<V4<double>*>(P->Xi.p));
            RRG_LAUNCHED();
            add_xyz_kernel<double><<<bp, 256, 0, s>>>(P->n, static_cast<V4<double>*>(P->X.p),
                                                     static_cast<const V4<double>*>(P->Xi.p));
        } else {
            interp_adjoint_kernel<float><<<bp, 256, 0, s>>>(
                P->n, static_cast<const V4<float>*>(P->x.p), P->gdev,
                static_cast<const V4<float>*>(P->acc4.p), static_cast<const V4<float>*>(P->A.p),
                nullptr, 0.f, nullptr, static_cast<V4<float>*>(P->Xi.p));
            RRG_LAUNCHED();
            add_xyz_kernel<float><<<bp, 256, 0, s>>>(P->n, static_cast<V4<float>*>(P->X.p),
                                                    static_cast<const V4<float>*>(P->Xi.p));
        }
        RRG_LAUNCHED();
        give_back(P, P->X.p, gx_out, s);
        give_back(P, P->V.p, gv_out, s);
    })
}

}  // extern "C"
