// Particle-mesh kernels on sm_100a: CIC deposit into int64 fixed point, damped-wave potential
// relaxation, gradient, trilinear force interpolation, and the fused particle pass.
//
// Grid layout is the reference's AT(x, y, z) = x + y nx + z nx^2
// (solver/lib/rrgsim_common/include/co_device_utils.cuh:61), nx^3 cells, cell centres at
// domain_min + (i + 1/2) dx for CIC / interpolation and nodes at domain_min + i dx for the wave
// boundary terms (wave.cu:18-20), exactly as in the reference.
#include <cstdlib>

#include "kernels.cuh"
#include "sums.cuh"
#include "wave_cells.cuh"

namespace rrg {
namespace {

constexpr double kPi = 3.14159265358979;  // the reference's PI (co_info_structs.h:7)
static_assert(kPmSumValues == kConsTerms, "PM_SUMS records hold the 8 conservation terms");

__device__ __forceinline__ int wrap_mod(int i, int n) {
    i %= n;
    return i < 0 ? i + n : i;
}

__device__ __forceinline__ double load_x(const V4<float>* posm, const V4<float>* lo, int64_t i,
                                         double& y, double& z, float& m) {
    const V4<float> p = posm[i];
    double x = p.x;
    y = p.y;
    z = p.z;
    if (lo) {
        const V4<float> l = lo[i];
        x += l.x;
        y += l.y;
        z += l.z;
    }
    m = p.w;
    return x;
}

// ----------------------------------------------------------------------------------------------
// CIC weights exactly as deposit_cell_mass_CIC_ (rm_p2mesh.cu:184-226), in FP64 with every
// operation rounded separately (no FMA contraction) so that the host oracle, compiled with
// -ffp-contract=off, produces the same bits:
//   u = (x - domain_min) * inv_dx - 0.5 ; clamp to [0, nx - 1 - 1e-6]
//   i0 = floor(u) ; i1 = min(i0 + 1, nx - 1) ; f = u - i0 ; w0 = 1 - f ; w1 = f
// A NaN coordinate is treated as u = 0 (the reference would index out of bounds).
// ----------------------------------------------------------------------------------------------
__device__ __forceinline__ void cic_axis(double x, double dmin, double inv_dx, int nx, int& i0,
                                         int& i1, double& w0, double& w1) {
    double u = __dsub_rn(__dmul_rn(__dsub_rn(x, dmin), inv_dx), 0.5);
    const double hi = __dsub_rn(static_cast<double>(nx - 1), 1e-6);
    if (!(u >= 0.0)) u = 0.0;  // also catches NaN
    if (u > hi) u = hi;
    i0 = static_cast<int>(floor(u));
    i1 = min(i0 + 1, nx - 1);
    const double f = __dsub_rn(u, static_cast<double>(i0));
    w0 = __dsub_rn(1.0, f);
    w1 = f;
}

// Deposits one particle (all lanes of the warp call this together, converged).
// Lanes with the same base cell form a run once they sit next to each other: particles sorted by
// cell make long runs, but as they drift from the sorted order a warp's cells interleave. A warp
// holding more than four runs therefore first sorts its (cell, lane) pairs with a bitonic
// network of full-warp shuffles (15 compare-exchange steps) and takes each lane's values along.
// Each of the 8 corner values is then summed over its run by a segmented warp scan (a full-warp
// shuffle per doubling of the longest run), and the run's last lane adds the eight sums with 64-bit
// atomics at fixed offsets from the cell: one set of atomics per distinct cell in the warp. (Always
// five scan steps, and the corners taken from the cell's coordinates by divisions: 120.0 against
// 116.2 us per PM step with 1M particles on 128^3; the pass issues 70 % of its cycles.) Values fit in 27 bits (the scale S is chosen so that
// m_max 2^S <= 2^26), so a warp's sum fits 32 bits; integer sums are exact in any order, so the
// grid does not depend on how particles fall into runs. (Grouping lanes with __match_any_sync and
// summing each group with __reduce_add_sync cost more: every distinct group mask in a warp is a
// separate divergent pass. Without the warp sort the atomics multiply as runs fragment: at 2^20
// disk particles 0.3 cell off their sorted order, 51 us against 27. The hardware reduction with
// each lane's run mask taken from the run heads, for warps of up to 4, 8 or 32 runs instead of
// 2: 126.4, 131.6 and 144.9 against 124.7 us per PM step. Floors without conversion
// instructions (rounded-down additions of 2^52 and 1.5 2^23) in these weights and in the
// interpolation's: 124.6 against 124.6 us.)
__device__ __forceinline__ void cic_deposit_warp(bool active, double x, double y, double z,
                                                 double m, const GridDev& g, double scale,
                                                 unsigned long long* __restrict__ grid) {
    const int nx = g.nx;
    int i0 = 0, i1 = 0, j0 = 0, j1 = 0, k0 = 0, k1 = 0;
    double wx0 = 0, wx1 = 0, wy0 = 0, wy1 = 0, wz0 = 0, wz1 = 0;
    if (active) {
        cic_axis(x, g.domain_min, g.inv_dx, nx, i0, i1, wx0, wx1);
        cic_axis(y, g.domain_min, g.inv_dx, nx, j0, j1, wy0, wy1);
        cic_axis(z, g.domain_min, g.inv_dx, nx, k0, k1, wz0, wz1);
    }
    const int nx2 = nx * nx;  // nx^3 < 2^31 (nx <= 1024)
    const int lane = threadIdx.x & 31;
    const double ms = __dmul_rn(m, scale);
    // corner order and weight products as rm_p2mesh.cu:219-235
    const double wxs[2] = {wx0, wx1}, wys[2] = {wy0, wy1}, wzs[2] = {wz0, wz1};
    unsigned q[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        q[c] = 0;
        if (active) {
            const double w = __dmul_rn(__dmul_rn(wxs[c & 1], wys[(c >> 1) & 1]), wzs[c >> 2]);
            // round to the nearest integer, ties to even, as __double2ll_rn: adding 1.5 * 2^52
            // leaves the integer in the low mantissa bits (exact for 0 <= value < 2^31; values
            // here are below 2^27), an FP64 add instead of a conversion on the XU pipe
            q[c] = static_cast<unsigned>(
                __double2loint(__dadd_rn(__dmul_rn(ms, w), 6755399441055744.0)));
        }
    }
    // every lane takes part in every shuffle (none behind a short-circuit or a divergent branch)
    int key = active ? (i0 + j0 * nx + k0 * nx2) : -1;
    const int below0 = __shfl_up_sync(0xffffffffu, key, 1);
    const unsigned heads0 = __ballot_sync(0xffffffffu, lane == 0 || below0 != key);
    // a warp of 28 or more runs (sparse outskirts: nearly one cell per lane) skips the sort and
    // the scan, and every lane adds its own values (121.5 against 122.1 us per PM step; from 20
    // runs on the extra atomics cost more than the scan saves: 126.8; skipping the sort also for
    // warps whose lanes are already in cell order, one ballot: 121.6 against 121.8, not kept)
    constexpr int sparse = 28;
    if (__popc(heads0) > 4 && __popc(heads0) < sparse) {  // warp-uniform
        int src = lane;
        if (nx <= 406) {
            // (cell + 1, lane) packed into one int (nx^3 < 2^26): one shuffle per step
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
            src = kv & 31;
        } else {
#pragma unroll
            for (int k = 2; k <= 32; k <<= 1) {
#pragma unroll
                for (int j = k >> 1; j > 0; j >>= 1) {
                    const int pk = __shfl_xor_sync(0xffffffffu, key, j);
                    const int ps = __shfl_xor_sync(0xffffffffu, src, j);
                    const bool ascending = (lane & k) == 0, lower = (lane & j) == 0;
                    const bool less = pk < key || (pk == key && ps < src);
                    if (lower == ascending ? less : !less) {
                        key = pk;
                        src = ps;
                    }
                }
            }
        }
#pragma unroll
        for (int c = 0; c < 8; ++c) q[c] = __shfl_sync(0xffffffffu, q[c], src);
    }
    const int below = __shfl_up_sync(0xffffffffu, key, 1);
    const int above = __shfl_down_sync(0xffffffffu, key, 1);
    const bool head = lane == 0 || below != key;
    bool tail = lane == 31 || above != key;
    const unsigned heads = __ballot_sync(0xffffffffu, head);
    unsigned sum[8];
    if (__popc(heads) >= sparse) {
        // (nearly) every lane its own cell: each adds its own values
#pragma unroll
        for (int c = 0; c < 8; ++c) sum[c] = q[c];
        tail = true;
    } else if (__popc(heads) <= 2) {
        // one or two runs (warp-uniform; the common case in dense regions of sorted
        // particles): one hardware reduction per run and corner instead of the scan
        const unsigned second = heads & ~1u;  // the second run's head lane bit, or 0
        const unsigned mask = second == 0u ? 0xffffffffu
                              : ((lane < __ffs(second) - 1) ? second - 1u : ~(second - 1u));
#pragma unroll
        for (int c = 0; c < 8; ++c) sum[c] = __reduce_add_sync(mask, q[c]);
    } else {
        const int first = 31 - __clz(heads & (0xffffffffu >> (31 - lane)));  // the run's first lane
#pragma unroll
        for (int c = 0; c < 8; ++c) sum[c] = q[c];
        // distance d only while some run has more than d lanes (d lanes in a row that are no heads)
        unsigned longer = ~heads;
        for (int d = 1; longer != 0u; d <<= 1) {
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const unsigned t = __shfl_up_sync(0xffffffffu, sum[c], d);
                if (lane - d >= first) sum[c] += t;
            }
            longer &= longer >> d;
        }
        // (at the run's last lane: the run's total)
    }
    if (key >= 0 && tail) {
        // the run's cell and its corners (cic_axis keeps i0 <= nx - 2: no corner is clamped)
        unsigned long long* const at = grid + key;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            if (sum[c] != 0u)
                atomicAdd(at + ((c & 1) + (c & 2 ? nx : 0) + (c & 4 ? nx2 : 0)),
                          static_cast<unsigned long long>(sum[c]));
        }
    }
}

template <typename R>
__device__ __forceinline__ void load_pos(const void* posm, const V4<float>* lo, int64_t i,
                                         double& x, double& y, double& z, double& m) {
    if constexpr (sizeof(R) == 8) {
        const V4<double> p = static_cast<const V4<double>*>(posm)[i];
        x = p.x;
        y = p.y;
        z = p.z;
        m = p.w;
    } else {
        float mf;
        x = load_x(static_cast<const V4<float>*>(posm), lo, i, y, z, mf);
        m = mf;
    }
}

template <typename R>
__global__ void __launch_bounds__(256) cic_kernel(int64_t n, const void* __restrict__ posm,
                                                  const V4<float>* __restrict__ lo, GridDev g,
                                                  double scale,
                                                  unsigned long long* __restrict__ grid) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const bool active = i < n;
    double x = 0, y = 0, z = 0, m = 0;
    if (active) load_pos<R>(posm, lo, i, x, y, z, m);
    cic_deposit_warp(active, x, y, z, m, g, scale, grid);
}

// ----------------------------------------------------------------------------------------------
// Wave source: f = 4 pi G rho, rho = mass / dx^3 - rho_sub (wave.cu:150-153), mass from the
// fixed-point grid. Optionally clears the fixed-point grid for the next deposit.
// ----------------------------------------------------------------------------------------------
// FP64 divides by dx^3 as the reference does; FP32, whose source is rounded to float anyway,
// multiplies by the host's 1 / dx^3 (an FP64 division per cell made this pass instruction-bound).
template <typename R>
__global__ void wave_source_kernel(int64_t ncells, const unsigned long long* mgrid,
                                   double inv_scale, double dx3, double inv_dx3, double rho_sub,
                                   double mult, R* src, unsigned long long* zero_grid) {
    const int64_t c = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    pdl_wait();
    if (c >= ncells) return;
    const unsigned long long q = mgrid[c];
    if (zero_grid) zero_grid[c] = 0ull;  // (mgrid itself, or the next deposit's grid)
    if constexpr (sizeof(R) == 8) {
        const double mass = static_cast<double>(q) * inv_scale;
        const double rho = mass / dx3 - rho_sub;
        src[c] = static_cast<R>(mult * (4.0 * kPi * 1.0 * rho));
    } else {
        src[c] = static_cast<R>(__dmul_rn(mult, wave_source_value(q, inv_scale, inv_dx3, rho_sub)));
    }
}

// The incremental solve's preparation (wave_inc_source), V consecutive x-cells per thread.
// FIRST: also the first substep, which needs no neighbours (the increments start at zero):
// d_1 = K_OLD d_old + g, stored over d_old's place, with level 0 of the increments (zero) in d
// (null: not stored).
// Bound: HBM at 256^3 (32 to 36 B per cell); below, the FP64 arithmetic of g.
template <int V, bool FIRST>
__global__ void __launch_bounds__(256) wave_inc_prep_kernel(
    int nx, const unsigned long long* mg, unsigned long long* mg_zero,
    double inv_scale, double inv_dx3, double rho_sub, const float* phi0,
    const float* phi_prev, double kf, double km, double kao, float ko,
    float* g, float* d, float* d_old,
    float* src) {
    using C = Cells<float, V>;
    const int W = nx / V;
    // (at most 2^30 units: 32-bit divisions; PM step with 64-bit ones 256^3 845 against 837 us)
    const unsigned int u = blockIdx.x * 256u + threadIdx.x;
    const unsigned int units = static_cast<unsigned int>(W) * nx * nx;
    if (u >= units) {  // (every block waits)
        pdl_wait();
        return;
    }
    const unsigned int r0 = u / static_cast<unsigned int>(W);
    const int q = static_cast<int>(u - r0 * W);
    const int z = static_cast<int>(r0 / static_cast<unsigned int>(nx)),
              y = static_cast<int>(r0) - z * nx;
    const int64_t row = r0;
    const int64_t plane = static_cast<int64_t>(nx) * nx;
    const int64_t c = row * nx + q * V;
    pdl_wait();
    auto cells = [&](int64_t at) { return *reinterpret_cast<const C*>(phi0 + at); };
    const C p = cells(c), pp = *reinterpret_cast<const C*>(phi_prev + c);
    const float l = phi0[row * nx + (q == 0 ? nx : q * V) - 1];
    const float r = phi0[row * nx + (q == W - 1 ? 0 : q * V + V)];
    const C ym = cells(c + (y == 0 ? (nx - 1) * nx : -nx));
    const C yp = cells(c + (y == nx - 1 ? -(nx - 1) * nx : nx));
    const C zm = cells(c + (z == 0 ? (nx - 1) * plane : -plane));
    const C zp = cells(c + (z == nx - 1 ? -(nx - 1) * plane : plane));
    unsigned long long q8[V];
#pragma unroll
    for (int i = 0; i < V; i += (V > 1 ? 2 : 1)) {
        if constexpr (V > 1) {
            const ulonglong2 m = *reinterpret_cast<const ulonglong2*>(mg + c + i);
            q8[i] = m.x;
            q8[i + 1] = m.y;
            if (mg_zero) *reinterpret_cast<ulonglong2*>(mg_zero + c + i) = make_ulonglong2(0ull, 0ull);
        } else {
            q8[i] = mg[c];
            if (mg_zero) mg_zero[c] = 0ull;
        }
    }
    C og, od, oo, os;
#pragma unroll
    for (int i = 0; i < V; ++i) {
        const double sd = wave_source_value(q8[i], inv_scale, inv_dx3, rho_sub);
        og.v[i] = wave_inc_source(sd, i == 0 ? l : p.v[i > 0 ? i - 1 : 0],
                                  i == V - 1 ? r : p.v[i < V - 1 ? i + 1 : 0], ym.v[i], yp.v[i],
                                  zm.v[i], zp.v[i], p.v[i], kf, km, kao);
        const float before = __fsub_rn(pp.v[i], p.v[i]);
        od.v[i] = 0.f;
        oo.v[i] = FIRST ? __fmaf_rn(og.v[i], 1.f, __fmaf_rn(before, ko, 0.f)) : before;
        os.v[i] = static_cast<float>(sd);
    }
    *reinterpret_cast<C*>(g + c) = og;
    if (d) *reinterpret_cast<C*>(d + c) = od;
    *reinterpret_cast<C*>(d_old + c) = oo;
    if (src) *reinterpret_cast<C*>(src + c) = os;
}

__global__ void wave_inc_finish_kernel(int64_t nc, const float* phi0, const float* d_fin,
                                       const float* d_prv, float* fin, float* prv) {
    const int64_t c = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (c >= nc) return;
    const float p = phi0[c], a = d_fin[c], b = d_prv[c];
    fin[c] = __fadd_rn(p, a);
    prv[c] = __fadd_rn(p, b);
}

// ----------------------------------------------------------------------------------------------
// Damped wave substep (wave_diss_iteration, wave.cu:106-193).
//   phi_new = K_MAIN sum6 + K_ACTUAL phi + K_OLD phi_old + K_F f
// Every variant marches a thread through a chunk of z-planes with the z-neighbours in
// registers; phi_new overwrites phi_old in place (each cell's old value is read only by its own
// thread), so two grid buffers rotate instead of the reference's three.
// ----------------------------------------------------------------------------------------------
constexpr int kTX = 32, kTY = 8;
constexpr int kVecThreads = 128;

struct WaveDev {
    int nx;
    int zc;
    int bc;          // rrg_boundary_type
    int uniform;     // periodic without absorbing layer -> constant coefficients
    double K_MAIN, K_ACTUAL, K_OLD, K_F;
    double C, DT, DX, diss_base, diss_extra, sim_l, domain_min;
    double bc_mass, comx, comy, comz, r_min;
};

__device__ __forceinline__ double layer_diss(const WaveDev& w, double x) {
    const double x_in = 0.5 * w.sim_l;
    const double d = fabs(x) - x_in;
    return d > 0 ? w.diss_extra * d * d : 0.0;
}

__device__ __forceinline__ double monopole_phi(const WaveDev& w, double x, double y, double z) {
    const double rx = w.comx - x, ry = w.comy - y, rz = w.comz - z;
    const double dist = sqrt(rx * rx + ry * ry + rz * rz);
    const double r = fmax(dist, w.r_min);
    return -1.0 * w.bc_mass / r;
}

template <typename R>
__device__ __forceinline__ double psi_at(const WaveDev& w, const R* phi, int i, int j, int k) {
    const int64_t nx = w.nx;
    const double x = w.domain_min + i * w.DX, y = w.domain_min + j * w.DX,
                 z = w.domain_min + k * w.DX;
    return static_cast<double>(phi[i + j * nx + k * nx * nx]) - monopole_phi(w, x, y, z);
}

// Radiative boundary node (radiative_boundary / upwind_axis, wave.cu:51-104).
template <typename R>
__device__ double radiative_value(const WaveDev& w, const R* phi, int ix, int iy, int iz) {
    const double x = w.domain_min + ix * w.DX, y = w.domain_min + iy * w.DX,
                 z = w.domain_min + iz * w.DX;
    const double rx = x - w.comx, ry = y - w.comy, rz = z - w.comz;
    const double r = fmax(sqrt(rx * rx + ry * ry + rz * rz), w.r_min);
    const double n3[3] = {rx / r, ry / r, rz / r};
    const double psi0 = psi_at<R>(w, phi, ix, iy, iz);
    double dpsi_dr = 0.0;
    const int idx[3] = {ix, iy, iz};
    for (int axis = 0; axis < 3; ++axis) {
        const int i0 = idx[axis];
        int in = (n3[axis] > 0) ? i0 - 1 : i0 + 1;
        if (in < 0 || in >= w.nx) in = 2 * i0 - in;
        int jx = ix, jy = iy, jz = iz;
        if (axis == 0) jx = in;
        else if (axis == 1) jy = in;
        else jz = in;
        const double d = (psi0 - psi_at<R>(w, phi, jx, jy, jz)) / ((i0 - in) * w.DX);
        dpsi_dr += n3[axis] * d;
    }
    const double psi_new = psi0 - w.C * w.DT * (dpsi_dr + psi0 / r);
    return psi_new + monopole_phi(w, x, y, z);
}

__device__ __forceinline__ unsigned long long dbits(double v) {
    return static_cast<unsigned long long>(__double_as_longlong(v));
}

// Block-wide max of (dmax, amax) folded into maxbits[0..1] (non-negative doubles compare as
// their bit patterns).
__device__ __forceinline__ void block_max_to(double dmax, double amax, int tid,
                                             unsigned long long* maxbits) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        dmax = fmax(dmax, __shfl_down_sync(0xffffffffu, dmax, o));
        amax = fmax(amax, __shfl_down_sync(0xffffffffu, amax, o));
    }
    __shared__ double sd[kTX * kTY / 32], sa[kTX * kTY / 32];  // blocks of up to 256 threads
    const int lane = tid & 31, wid = tid >> 5;
    if (lane == 0) {
        sd[wid] = dmax;
        sa[wid] = amax;
    }
    __syncthreads();
    if (tid == 0) {
        double d = 0, a = 0;
        const int warps = static_cast<int>((blockDim.x * blockDim.y + 31) / 32);
        for (int k = 0; k < warps; ++k) {
            d = fmax(d, sd[k]);
            a = fmax(a, sa[k]);
        }
        atomicMax(maxbits, dbits(d));
        atomicMax(maxbits + 1, dbits(a));
    }
}

// Periodic box without an absorbing layer (the reference's wired path, wave.cu:177-181): constant
// coefficients, V consecutive x-cells per thread (16 bytes: four FP32 or two FP64, fewer where
// the row length does not divide). A warp takes 32 V consecutive cells of a plane, so the x
// neighbours are shuffles, with a scalar load where a row or the warp ends; rows y +- 1 are
// coalesced vector loads, the z neighbours a register pipeline over ZC planes whose ZC + 2 values
// are all requested before the first update (a latency-bound stencil). The arithmetic is
// wave_cell's, every rounding written out, in every V and precision.
// ADJ: the adjoint substep of the PM adjoint instead (phi the current cotangent C, phi_old the
// previous one P, no source): P <- K_MAIN L6(C) + K_ACTUAL C + K_OLD P and F += K_F C.
// Successive substeps are launched with programmatic dependence: a block's indices are ready when
// the substep before it ends (no load is ahead of the wait).
//
// Bound: launch and L2 latency up to ~100^3, L2 bandwidth to ~160^3, HBM beyond (256^3: 268 MB in
// 38.9 us, 1.05 of the copy peak, part of it L2 hits; the fused FP32 solves take three substeps per
// launch there, wave_march.cu). Per substep in a graph on B200, us: one-cell
// columns (FP64, and rows that do not tile a warp) or float4 rows, chunks of up to 8 planes, normal
// launches -> vectors everywhere and programmatic launches -> loads a plane ahead, 2 planes: FP32
// 33^3 2.61 -> 2.05 -> 1.5, 64^3 2.39 -> 2.13 -> 1.72, 96^3 4.68 -> 3.05 -> 2.64, 128^3 4.59 -> 4.35
// -> 4.5, 160^3 13.2 -> 8.5 -> 7.3, 256^3 48.1 -> 45.6 -> 38.9; FP64 64^3 2.99 -> 2.80 -> 2.13,
// 128^3 9.89 -> 8.19 -> 7.37.
// LAST: the last substep of an incremental solve (wave_inc_source; phi and phi_old the increments
// d and d_old, src their source g): instead of d_new, the levels in full, phi0 + d_new to fin and
// phi0 + d to prv (either may be phi0: a cell's phi0 is read by its own thread alone, a plane ahead
// like the rest: PM step on 256^3 848 -> 843 us, 96^3 67.8 -> 67.1).
enum VecMode { VEC_STEP, VEC_ADJ, VEC_LAST };
template <typename R, int V, int ZC, bool CHECK, VecMode MODE>
__global__ void __launch_bounds__(kVecThreads, 6) wave_periodic_vec_kernel(
    const R* phi, R* phi_old, const R* src, const WaveDev w,
    unsigned long long* __restrict__ maxbits, R* fadj, const R* phi0, R* fin, R* prv) {
    using C = Cells<R, V>;
    constexpr bool ADJ = MODE == VEC_ADJ;
    // the first plane's rows are requested with the column, the next plane's before a plane is
    // computed: one round trip to L2 instead of one per plane
    const int nx = w.nx;
    const int W = nx / V;        // V-cell units per row
    const int plane = nx * nx;
    const int tid = threadIdx.x, lane = tid & 31;
    const int g = blockIdx.x * kVecThreads + tid;  // unit within a plane
    const bool valid = g < W * nx;
    const int y = valid ? g / W : 0, q = valid ? g - y * W : 0;
    const int at = y * nx + q * V;
    // rows that tile a warp keep the x neighbours in it; else those across the row's ends
    // (periodic) or the warp's ends are loaded
    const bool tiles = W <= 32 && 32 % W == 0;
    const int lsrc = tiles && q == 0 ? lane + W - 1 : lane - 1;
    const int rsrc = tiles && q == W - 1 ? lane - (W - 1) : lane + 1;
    const bool lload = valid && !tiles && (lane == 0 || q == 0);
    const bool rload = valid && !tiles && (lane == 31 || q == W - 1);
    const int xl = (q == 0 ? nx : q * V) - 1 + y * nx, xr = (q == W - 1 ? 0 : q * V + V) + y * nx;
    const int aym = y > 0 ? at - nx : at + plane - nx, ayp = y < nx - 1 ? at + nx : at - plane + nx;
    const R km = static_cast<R>(w.K_MAIN), ka = static_cast<R>(w.K_ACTUAL),
            ko = static_cast<R>(w.K_OLD), kf = static_cast<R>(w.K_F);
    const int z0 = blockIdx.y * ZC;
    pdl_next();
    pdl_wait();
    C pv[ZC + 2];  // phi at z0 - 1 ... z0 + ZC (wrapped)
#pragma unroll
    for (int k = 0; k < ZC + 2; ++k) {
        int z = z0 - 1 + k;
        z = z < 0 ? z + nx : z;
        while (z >= nx) z -= nx;
        pv[k] = load_cells<R, V>(phi + (at + z * plane));
    }
    double dmax = 0.0, amax = 0.0;
    struct Plane {
        C ym, yp, po, other;  // other: the source, or F
        C p0;                 // VEC_LAST
        R l, r;
    };
    auto fetch = [&](int z) -> Plane {
        Plane p{};
        if (valid && z < nx) {
            const int zb = z * plane;
            if (lload) p.l = load_cells<R, 1>(phi + (xl + zb)).v[0];
            if (rload) p.r = load_cells<R, 1>(phi + (xr + zb)).v[0];
            p.ym = load_cells<R, V>(phi + (aym + zb));
            p.yp = load_cells<R, V>(phi + (ayp + zb));
            p.po = load_cells<R, V>(phi_old + (at + zb));
            if constexpr (ADJ) p.other = load_cells<R, V>(fadj + (at + zb));
            else p.other = load_cells<R, V>(src + (at + zb));
            if constexpr (MODE == VEC_LAST) p.p0 = load_cells<R, V>(phi0 + (at + zb));
        }
        return p;
    };
    Plane next = fetch(z0);
#pragma unroll
    for (int k = 0; k < ZC; ++k) {
        const int z = z0 + k;
        if (z >= nx) break;
        Plane p = next;
        if (k + 1 < ZC) next = fetch(z + 1);
        const C c = pv[k + 1];
        R lft = __shfl_sync(0xffffffffu, c.v[V - 1], lsrc & 31);
        R rgt = __shfl_sync(0xffffffffu, c.v[0], rsrc & 31);
        if (lload) lft = p.l;
        if (rload) rgt = p.r;
        if (valid) {
            const int zb = z * plane;
            C out;
#pragma unroll
            for (int i = 0; i < V; ++i) {
                const R l = i == 0 ? lft : c.v[i > 0 ? i - 1 : 0];
                const R r = i == V - 1 ? rgt : c.v[i < V - 1 ? i + 1 : 0];
                const R t = wave_cell_adj(l, r, p.ym.v[i], p.yp.v[i], pv[k].v[i], pv[k + 2].v[i],
                                          c.v[i], p.po.v[i], km, ka, ko);
                if constexpr (ADJ) {
                    out.v[i] = t;
                    p.other.v[i] = rfma(kf, c.v[i], p.other.v[i]);
                } else {
                    out.v[i] = rfma(p.other.v[i], kf, t);
                }
                if constexpr (CHECK) {
                    // differences in FP64
                    dmax = fmax(dmax, fabs(double(out.v[i]) - double(c.v[i])));
                    amax = fmax(amax, fabs(double(out.v[i])));
                }
            }
            if constexpr (MODE == VEC_LAST) {
                C full, before;
#pragma unroll
                for (int i = 0; i < V; ++i) {
                    full.v[i] = radd(p.p0.v[i], out.v[i]);
                    before.v[i] = radd(p.p0.v[i], c.v[i]);
                }
                *reinterpret_cast<C*>(fin + (at + zb)) = full;
                *reinterpret_cast<C*>(prv + (at + zb)) = before;
            } else {
                *reinterpret_cast<C*>(phi_old + (at + zb)) = out;
            }
            if constexpr (ADJ) *reinterpret_cast<C*>(fadj + (at + zb)) = p.other;
        }
    }
    if constexpr (CHECK) block_max_to(dmax, amax, tid, maxbits);
}

// Every other boundary, and the absorbing layer.
template <typename R, bool CHECK>
__global__ void __launch_bounds__(kTX* kTY, 2) wave_step_kernel(
    const R* __restrict__ phi, R* __restrict__ phi_old, const R* __restrict__ src,
    const WaveDev w, unsigned long long* __restrict__ maxbits) {
    // One thread per (x, y) column marches through zc planes: phi(z - 1), phi(z), phi(z + 1)
    // stay in registers, the four in-plane neighbours come through L1 (adjacent threads share
    // their cache lines). No shared memory, no barriers. int32 indexing: nx <= 1024.
    const int nx = w.nx;
    const int plane = nx * nx;
    const int tid = threadIdx.y * kTX + threadIdx.x;
    const int x = blockIdx.x * kTX + threadIdx.x;
    const int y = blockIdx.y * kTY + threadIdx.y;
    const bool valid = (x < nx) && (y < nx);
    const bool periodic = w.bc == RRG_BC_PERIODIC;
    double dmax = 0.0, amax = 0.0;
    if (valid) {
        // in-plane neighbour offsets: periodic wrap, or clamped (unused on the boundary nodes)
        const int oxm = x > 0 ? -1 : (periodic ? nx - 1 : 0);
        const int oxp = x < nx - 1 ? 1 : (periodic ? -(nx - 1) : 0);
        const int oym = y > 0 ? -nx : (periodic ? (nx - 1) * nx : 0);
        const int oyp = y < nx - 1 ? nx : (periodic ? -(nx - 1) * nx : 0);
        const bool xy_edge = x == 0 || x == nx - 1 || y == 0 || y == nx - 1;
        const int col = x + y * nx;
        const int z0 = blockIdx.z * w.zc;
        const int z1 = min(nx, z0 + w.zc);
        const int zm0 = z0 > 0 ? z0 - 1 : (periodic ? nx - 1 : 0);
        R pm = __ldg(phi + col + zm0 * plane);
        R pc = __ldg(phi + col + z0 * plane);
        for (int z = z0; z < z1; ++z) {
            const int zn = z < nx - 1 ? z + 1 : (periodic ? 0 : nx - 1);
            const R pn = __ldg(phi + col + zn * plane);
            const int c = col + z * plane;
            R out;
            if (!periodic && (xy_edge || z == 0 || z == nx - 1)) {
                double v = 0.0;
                if (w.bc == RRG_BC_MONOPOLE_DIRICHLET)
                    v = monopole_phi(w, w.domain_min + x * w.DX, w.domain_min + y * w.DX,
                                     w.domain_min + z * w.DX);
                else if (w.bc == RRG_BC_MONOPOLE_RADIATIVE)
                    v = radiative_value<R>(w, phi, x, y, z);
                out = static_cast<R>(v);
            } else {
                const R lap = __ldg(phi + c + oxm) + __ldg(phi + c + oxp) +
                              __ldg(phi + c + oym) + __ldg(phi + c + oyp) + pm + pn;
                double diss = w.diss_base;
                diss += layer_diss(w, w.domain_min + x * w.DX);
                diss += layer_diss(w, w.domain_min + y * w.DX);
                diss += layer_diss(w, w.domain_min + z * w.DX);
                const double Q = diss * w.C * w.DT * 0.5;
                const double W = 1 + Q;
                const double K = w.C * w.C * w.DT * w.DT / (w.DX * w.DX);
                const R kmain = static_cast<R>(K / W);
                const R kf = static_cast<R>(-w.C * w.C * w.DT * w.DT / W);
                const R kact = static_cast<R>(2 * (1 - 3 * K) / W);
                const R kold = static_cast<R>((Q - 1) / W);
                out = lap * kmain + pc * kact + phi_old[c] * kold + src[c] * kf;
            }
            phi_old[c] = out;
            if constexpr (CHECK) {
                dmax = fmax(dmax, fabs(static_cast<double>(out) - static_cast<double>(pc)));
                amax = fmax(amax, fabs(static_cast<double>(out)));
            }
            pm = pc;
            pc = pn;
        }
    }
    if constexpr (CHECK) {
        // warp max -> block max -> one atomicMax per block on the (non-negative) double bits
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            dmax = fmax(dmax, __shfl_down_sync(0xffffffffu, dmax, o));
            amax = fmax(amax, __shfl_down_sync(0xffffffffu, amax, o));
        }
        __shared__ double sd[kTX * kTY / 32], sa[kTX * kTY / 32];
        const int lane = tid & 31, wid = tid >> 5;
        if (lane == 0) {
            sd[wid] = dmax;
            sa[wid] = amax;
        }
        __syncthreads();
        if (tid == 0) {
            double d = 0, a = 0;
            for (int k = 0; k < kTX * kTY / 32; ++k) {
                d = fmax(d, sd[k]);
                a = fmax(a, sa[k]);
            }
            atomicMax(maxbits, dbits(d));
            atomicMax(maxbits + 1, dbits(a));
        }
    }
}

// ----------------------------------------------------------------------------------------------
// Gradient (calc_acceleration_field_, rm_p2mesh.cu:238-290): central differences inside,
// one-sided at the faces, a = -dphi / dx. Output cell (ax, ay, az, phi).
// ----------------------------------------------------------------------------------------------
// V consecutive x-cells per thread and ZC planes, as wave_periodic_vec_kernel: x +- 1 by warp
// shuffles (a scalar load where a warp ends inside a row), rows y +- 1 as coalesced vector loads a
// plane ahead, the z neighbours in registers. A warp's 32 V cells are consecutive in memory: they
// are staged in shared memory and stored 512 contiguous bytes per instruction (64-byte strides
// before: 256^3 78 -> 54 us, 0.95 of the copy peak).
// Bound: launch and L2 latency on small grids, HBM on large ones (FP32 20 B, FP64 40 B per cell).
//
// This kernel, the source, the increments' preparation and the particle pass are launched with
// programmatic dependence but do not let the kernel after them start early (no pdl_next): a chain
// in which every kernel does lets the waiting blocks of many substeps pile up on the SMs. PM steps,
// us, normal launches / programmatic / programmatic and early starts: FP32 48^3 38.3 / 38.1 / 45.5,
// 96^3 71.4 / 68.6 / 68.2, 160^3 227 / 216 / 218, 256^3 905 / 872 / 876; FP64 33^3 38.5 / 37.0 / 40.
constexpr int kGradThreads = 128;
template <typename R, int V, int ZC>
__global__ void __launch_bounds__(kGradThreads) gradient_vec_kernel(int nx, R coef, const R* phi,
                                                                    V4<R>* acc4) {
    using C = Cells<R, V>;
    constexpr int U = V * static_cast<int>(sizeof(V4<R>)) / 16;  // 16-byte units of a thread's cells
    constexpr int cellU = static_cast<int>(sizeof(V4<R>)) / 16;
    __shared__ float4 stage[kGradThreads / 32][32 * U];
    const int W = nx / V, plane = nx * nx, units = W * nx;
    const int tid = threadIdx.x, lane = tid & 31;
    const int g = blockIdx.x * kGradThreads + tid;  // unit within a plane
    const bool valid = g < units;
    const int y = valid ? g / W : 0, q = valid ? g - y * W : 0;
    const int at = y * nx + q * V;
    // (a neighbour across the row's end is not used: the faces are one-sided)
    const bool lload = valid && lane == 0 && q > 0, rload = valid && lane == 31 && q < W - 1;
    const int aym = y > 0 ? at - nx : at, ayp = y < nx - 1 ? at + nx : at;
    const int z0 = blockIdx.y * ZC;
    float4* const st = stage[tid >> 5];
    // the warp's cells of a plane: from cell first on, count 16-byte units
    const int first = (g - lane) * V, count = min(32, units - (g - lane)) * U;
    pdl_wait();
    C pv[ZC + 2];  // phi at z0 - 1 ... z0 + ZC (clamped to the box; faces are one-sided)
#pragma unroll
    for (int k = 0; k < ZC + 2; ++k)
        pv[k] = load_cells<R, V>(phi + (at + min(max(z0 - 1 + k, 0), nx - 1) * plane));
    struct Plane {
        C ym, yp;
        R l, r;
    };
    auto fetch = [&](int z) -> Plane {
        Plane p{};
        if (valid && z < nx) {
            const int zb = z * plane;
            if (lload) p.l = load_cells<R, 1>(phi + (at - 1 + zb)).v[0];
            if (rload) p.r = load_cells<R, 1>(phi + (at + V + zb)).v[0];
            p.ym = load_cells<R, V>(phi + (aym + zb));
            p.yp = load_cells<R, V>(phi + (ayp + zb));
        }
        return p;
    };
    // central inside, one-sided at the first and the last node
    auto diff = [&](int i, R m, R c, R p) {
        return i == 0 ? p - c : i == nx - 1 ? c - m : R(0.5) * (p - m);
    };
    Plane next = fetch(z0);
#pragma unroll
    for (int k = 0; k < ZC; ++k) {
        const int z = z0 + k;
        if (z >= nx) break;
        const Plane p = next;
        if (k + 1 < ZC) next = fetch(z + 1);
        const C c = pv[k + 1];
        R lft = __shfl_up_sync(0xffffffffu, c.v[V - 1], 1);
        R rgt = __shfl_down_sync(0xffffffffu, c.v[0], 1);
        if (lload) lft = p.l;
        if (rload) rgt = p.r;
        __syncwarp();  // (the plane before has been read from the stage)
#pragma unroll
        for (int i = 0; i < V; ++i) {
            const R l = i == 0 ? lft : c.v[i > 0 ? i - 1 : 0];
            const R r = i == V - 1 ? rgt : c.v[i < V - 1 ? i + 1 : 0];
            const V4<R> o = v4<R>(diff(q * V + i, l, c.v[i], r) * coef,
                                  diff(y, p.ym.v[i], c.v[i], p.yp.v[i]) * coef,
                                  diff(z, pv[k].v[i], c.v[i], pv[k + 2].v[i]) * coef, c.v[i]);
            const float4* const o4 = reinterpret_cast<const float4*>(&o);
#pragma unroll
            for (int j = 0; j < cellU; ++j) {
                const int slot = lane * U + i * cellU + j;
                st[slot ^ ((slot >> 3) & 7)] = o4[j];  // (no bank conflicts on either side)
            }
        }
        __syncwarp();
        float4* const to =
            reinterpret_cast<float4*>(acc4 + (static_cast<size_t>(z) * plane + first));
#pragma unroll
        for (int j = 0; j < U; ++j) {
            const int slot = j * 32 + lane;
            if (slot < count) to[slot] = st[slot ^ ((slot >> 3) & 7)];
        }
    }
}

// ----------------------------------------------------------------------------------------------
// Trilinear gather (interpolate_acceleration_to_particles_kernel, rm_mesh2p.cu:48-114).
// Index selection as the reference: f = (x - domain_min) / dx - 0.5 in FP64, i0 = floorf(f)
// (the reference passes its double to floorf, i.e. floors the float-rounded value), weights
// from the unclamped fraction, indices clamped to [0, nx - 1]; summation order z, y, x.
// ----------------------------------------------------------------------------------------------
// DIV: divide by dx as the reference (FP64 path); else multiply by 1 / dx (FP32 and MIXED,
// whose weights are rounded to float: an FP64 division per axis dominated the particle pass).
template <bool DIV>
__device__ __forceinline__ void interp_axis(double x, double dmin, double dx, double inv_dx,
                                            int nx, int& i0, int& i1, double& w) {
    const double f = (DIV ? (x - dmin) / dx : (x - dmin) * inv_dx) - 0.5;
    int a = static_cast<int>(floorf(static_cast<float>(f)));
    w = f - a;
    i0 = max(0, min(a, nx - 1));
    i1 = max(0, min(a + 1, nx - 1));
}

template <typename R>
__device__ __forceinline__ void trilinear(const V4<R>* __restrict__ acc4, const GridDev& g,
                                          double x, double y, double z, R& ax, R& ay, R& az) {
    int i0, i1, j0, j1, k0, k1;
    double wxd, wyd, wzd;
    constexpr bool DIV = sizeof(R) == 8;
    interp_axis<DIV>(x, g.domain_min, g.dx, g.inv_dx, g.nx, i0, i1, wxd);
    interp_axis<DIV>(y, g.domain_min, g.dx, g.inv_dx, g.nx, j0, j1, wyd);
    interp_axis<DIV>(z, g.domain_min, g.dx, g.inv_dx, g.nx, k0, k1, wzd);
    const R wx = static_cast<R>(wxd), wy = static_cast<R>(wyd), wz = static_cast<R>(wzd);
    const int nx = g.nx;  // nx^3 < 2^31 (nx <= 1024)
    ax = ay = az = R(0);
#pragma unroll
    for (int k = 0; k <= 1; ++k) {
        const int kk = k == 0 ? k0 : k1;
        const R wk = k == 0 ? (R(1) - wz) : wz;
#pragma unroll
        for (int j = 0; j <= 1; ++j) {
            const int jj = j == 0 ? j0 : j1;
            const R wj = j == 0 ? (R(1) - wy) : wy;
#pragma unroll
            for (int i = 0; i <= 1; ++i) {
                const int ii = i == 0 ? i0 : i1;
                const R wi = i == 0 ? (R(1) - wx) : wx;
                const R weight = wi * wj * wk;
                const V4<R> f = acc4[(kk * nx + jj) * nx + ii];
                ax += weight * f.x;
                ay += weight * f.y;
                az += weight * f.z;
            }
        }
    }
}

template <typename R>
__global__ void __launch_bounds__(256) interp_kernel(int64_t n, const void* __restrict__ posm,
                                                     const V4<float>* __restrict__ lo, GridDev g,
                                                     const V4<R>* __restrict__ acc4,
                                                     V4<R>* __restrict__ acc) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double x, y, z, m;
    load_pos<R>(posm, lo, i, x, y, z, m);
    R ax, ay, az;
    trilinear<R>(acc4, g, x, y, z, ax, ay, az);
    acc[i] = v4<R>(ax, ay, az, R(0));
}

// NGP cell as assign_particles_to_cells_ (rm_p2mesh.cu:37-49): truncation, clamp.
__device__ __forceinline__ int ngp_axis(double x, double dmin, double dx, int nx) {
    const double f = (x - dmin) / dx;
    int a = (f == f) ? static_cast<int>(f) : 0;
    return max(0, min(a, nx - 1));
}

template <typename R>
__global__ void __launch_bounds__(256) ngp_phi_kernel(int64_t n, const void* __restrict__ posm,
                                                      const V4<float>* __restrict__ lo,
                                                      GridDev g, const R* __restrict__ phi,
                                                      R* __restrict__ pot) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double x, y, z, m;
    load_pos<R>(posm, lo, i, x, y, z, m);
    const int64_t nx = g.nx;
    const int64_t c = ngp_axis(x, g.domain_min, g.dx, g.nx) +
                      ngp_axis(y, g.domain_min, g.dx, g.nx) * nx +
                      ngp_axis(z, g.domain_min, g.dx, g.nx) * nx * nx;
    pot[i] = phi[c];
}

// ----------------------------------------------------------------------------------------------
// NGP projections of particle values onto the grid (N-body strategy with a grid,
// rrgsim_integration_nbody.cuh:32-48): per-cell particle counts (assign_particles_to_cells_,
// rm_p2mesh.cu:25-66), then each particle adds value / count of its cell
// (deposit_cell_grav_NGP_ / deposit_cell_acc_NGP_, rm_p2mesh.cu:142-174).
template <typename R>
__device__ __forceinline__ int64_t ngp_cell(const void* posm, const V4<float>* lo, int64_t i,
                                            const GridDev& g) {
    double x, y, z, m;
    load_pos<R>(posm, lo, i, x, y, z, m);
    const int64_t nx = g.nx;
    return ngp_axis(x, g.domain_min, g.dx, g.nx) + ngp_axis(y, g.domain_min, g.dx, g.nx) * nx +
           ngp_axis(z, g.domain_min, g.dx, g.nx) * nx * nx;
}

template <typename R>
__global__ void __launch_bounds__(256) ngp_count_kernel(int64_t n, const void* __restrict__ posm,
                                                        const V4<float>* __restrict__ lo,
                                                        GridDev g, int* __restrict__ count) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    atomicAdd(count + ngp_cell<R>(posm, lo, i, g), 1);
}

template <typename R>
__global__ void __launch_bounds__(256) ngp_project_kernel(int64_t n, const void* __restrict__ posm,
                                                          const V4<float>* __restrict__ lo,
                                                          GridDev g, const int* __restrict__ count,
                                                          const R* __restrict__ pot,
                                                          const V4<R>* __restrict__ acc,
                                                          R* __restrict__ phi_grid,
                                                          R* __restrict__ acc_grid) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int64_t c = ngp_cell<R>(posm, lo, i, g);
    const R cnt = static_cast<R>(count[c]);
    if (phi_grid) atomicAdd(phi_grid + c, pot[i] / cnt);
    if (acc_grid) {
        const V4<R> a = acc[i];
        const R inv = R(1) / cnt;
        atomicAdd(acc_grid + 4 * c, a.x * inv);
        atomicAdd(acc_grid + 4 * c + 1, a.y * inv);
        atomicAdd(acc_grid + 4 * c + 2, a.z * inv);
    }
}

// ----------------------------------------------------------------------------------------------
// Fused particle pass of the wave strategy (one launch per step):
//   [INTERP_CORRECT]  a = trilinear(x); v = (u + dt a) / 2                  (correct_step_)
//   [PREDICT_DEPOSIT] v* = v + dt a; u = v + v*; x += dt/2 u; CIC(x)        (predict_step_ +
//                                                                             deposit)
// ----------------------------------------------------------------------------------------------
template <typename R, bool MIXED, int MODE>
__global__ void __launch_bounds__(kPmThreads, 6) pm_particle_kernel(PmParticleArgs a, double scale) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const bool active = i < a.n;
    // PM_SUMS: every particle's 8 conservation terms, kept in shared memory until the block's
    // record is formed at the end of the pass (16 KB per block, reused by the reduction)
    constexpr bool SUMS = (MODE & PM_SUMS) != 0;
    __shared__ double terms[SUMS ? kConsTerms : 1][SUMS ? kPmThreads : 1];
    V4<R>* posm = static_cast<V4<R>*>(a.posm);
    V4<float>* lo = static_cast<V4<float>*>(a.poslo);
    V4<R>* vel = static_cast<V4<R>*>(a.vel);
    V4<R>* accp = static_cast<V4<R>*>(a.acc);
    V4<R>* u = static_cast<V4<R>*>(a.u);
    const R dt = static_cast<R>(a.dt);
    pdl_wait();
    double x = 0, y = 0, z = 0, m = 0;
    if (active) load_pos<R>(a.posm, MIXED ? lo : nullptr, i, x, y, z, m);

    R vx = 0, vy = 0, vz = 0, ax = 0, ay = 0, az = 0;
    if (active) {
        if constexpr ((MODE & PM_INTERP_CORRECT) != 0) {
            trilinear<R>(static_cast<const V4<R>*>(a.acc4), a.g, x, y, z, ax, ay, az);
            const V4<R> uu = u[i];
            vx = R(0.5) * (uu.x + dt * ax);
            vy = R(0.5) * (uu.y + dt * ay);
            vz = R(0.5) * (uu.z + dt * az);
            if constexpr ((MODE & PM_WRITE_SYNC) != 0) {
                vel[i] = v4<R>(vx, vy, vz, R(0));
                accp[i] = v4<R>(ax, ay, az, R(0));
            }
        } else {
            const V4<R> v = vel[i];
            const V4<R> ac = accp[i];
            vx = v.x; vy = v.y; vz = v.z;
            ax = ac.x; ay = ac.y; az = ac.z;
        }
    }
    if constexpr (SUMS) {
        // the synced state's terms, formed as conservation_kernel forms them (x, v and phi
        // promoted to double); stored now, so the deposit below has the registers
        const double ph = active ? static_cast<double>(static_cast<const R*>(a.pot)[i]) : 0.0;
#pragma unroll
        for (int k = 0; k < kConsTerms; ++k)
            terms[k][threadIdx.x] =
                active ? cons_term(k, x, y, z, m, static_cast<double>(vx),
                                   static_cast<double>(vy), static_cast<double>(vz), ph)
                       : 0.0;
    }
    if constexpr ((MODE & PM_PREDICT_DEPOSIT) != 0) {
        if (active) {
            const R sx = vx + dt * ax, sy = vy + dt * ay, sz = vz + dt * az;
            const R ux = vx + sx, uy = vy + sy, uz = vz + sz;
            u[i] = v4<R>(ux, uy, uz, R(0));
            const R hdt = dt * R(0.5);
            V4<R> p = posm[i];
            if constexpr (MIXED) {
                V4<float> l = lo[i];
                df_add(p.x, l.x, hdt * ux);
                df_add(p.y, l.y, hdt * uy);
                df_add(p.z, l.z, hdt * uz);
                (a.lo_out ? static_cast<V4<float>*>(a.lo_out) : lo)[i] = l;
                x = static_cast<double>(p.x) + l.x;
                y = static_cast<double>(p.y) + l.y;
                z = static_cast<double>(p.z) + l.z;
            } else {
                p.x = p.x + hdt * ux;
                p.y = p.y + hdt * uy;
                p.z = p.z + hdt * uz;
                x = p.x;
                y = p.y;
                z = p.z;
            }
            (a.pos_out ? static_cast<V4<R>*>(a.pos_out) : posm)[i] = p;
        }
        cic_deposit_warp(active, x, y, z, m, a.g, scale, a.mgrid);
    }
    if constexpr (SUMS) {
        // the block's record, in three fixed-order stages (FP64 issue, not latency, is what
        // this costs, so every stage keeps its warps' lanes busy): warp k sums term k, each
        // lane 8 particles' terms (cascaded); two warps combine those 32 partials per term 4 at
        // a time; then one lane per term adds the last 8. Records are value-major,
        // partial[(k gridDim.x + block) 2 + {0, 1}], so the finishing kernel reads them
        // coalesced.
        static_assert(kPmThreads / 32 == kConsTerms, "one warp per term");
        static_assert(sizeof(DD) * kConsTerms * 40 <= sizeof(double) * kConsTerms * kPmThreads,
                      "the stages fit in the terms' shared memory");
        DD (*stage)[40] = reinterpret_cast<DD (*)[40]>(&terms[0][0]);
        __syncthreads();
        const int t = threadIdx.x;
        {
            const int k = t >> 5, lane = t & 31;
            Casc c{terms[k][lane], 0.0};
#pragma unroll
            for (int j = lane + 32; j < kPmThreads; j += 32) casc_add(c, terms[k][j]);
            __syncthreads();  // every term read before the stages overwrite them
            stage[k][lane] = dd_norm(c.s, c.c);
        }
        __syncthreads();
        if (t < 64) {
            const int k = t >> 3, q = t & 7;
            DD d = stage[k][4 * q];
#pragma unroll
            for (int j = 1; j < 4; ++j) d = dd_add(d, stage[k][4 * q + j]);
            stage[k][32 + q] = d;
        }
        __syncthreads();
        if (t < kConsTerms) {
            DD d = stage[t][32];
#pragma unroll
            for (int j = 1; j < 8; ++j) d = dd_add(d, stage[t][32 + j]);
            const int64_t o = (static_cast<int64_t>(t) * gridDim.x + blockIdx.x) * 2;
            a.partial[o] = d.hi;
            a.partial[o + 1] = d.lo;
        }
    }
}

template <typename R, bool MIXED>
void dispatch_pm(const PmParticleArgs& a, int mode, double scale, cudaStream_t s) {
    auto go = [&](auto* kernel) { launch_pdl(kernel, div_up(a.n, 256), 256, 0, s, a, scale); };
    switch (mode) {
        case PM_INTERP_CORRECT | PM_WRITE_SYNC:
            go(pm_particle_kernel<R, MIXED, PM_INTERP_CORRECT | PM_WRITE_SYNC>);
            break;
        case PM_PREDICT_DEPOSIT:
            go(pm_particle_kernel<R, MIXED, PM_PREDICT_DEPOSIT>);
            break;
        case PM_INTERP_CORRECT | PM_PREDICT_DEPOSIT:
            go(pm_particle_kernel<R, MIXED, PM_INTERP_CORRECT | PM_PREDICT_DEPOSIT>);
            break;
        case PM_INTERP_CORRECT | PM_PREDICT_DEPOSIT | PM_WRITE_SYNC:
            go(pm_particle_kernel<R, MIXED, PM_INTERP_CORRECT | PM_PREDICT_DEPOSIT | PM_WRITE_SYNC>);
            break;
        case PM_INTERP_CORRECT | PM_PREDICT_DEPOSIT | PM_WRITE_SYNC | PM_SUMS:
            go(pm_particle_kernel<R, MIXED,
                                  PM_INTERP_CORRECT | PM_PREDICT_DEPOSIT | PM_WRITE_SYNC | PM_SUMS>);
            break;
        default:
            throw Error(RRG_ERR_INVALID, "pm particle pass: unsupported mode");
    }
}

}  // namespace

// ----------------------------------------------------------------------------------------------
void launch_cic_deposit(int prec, int64_t n, const void* posm, const void* poslo,
                        const GridDev& g, int shift_s, unsigned long long* grid,
                        cudaStream_t s) {
    const double scale = ldexp(1.0, shift_s);
    const int b = div_up(n, 256);
    if (prec == RRG_PREC_FP64)
        cic_kernel<double><<<b, 256, 0, s>>>(n, posm, nullptr, g, scale, grid);
    else
        cic_kernel<float><<<b, 256, 0, s>>>(
            n, posm, prec == RRG_PREC_MIXED ? static_cast<const V4<float>*>(poslo) : nullptr, g,
            scale, grid);
    RRG_LAUNCHED();
}

void launch_wave_source(int prec, int nx, const unsigned long long* mgrid, int shift_s,
                        double dx, double rho_mean, double scale, void* src,
                        unsigned long long* zero_grid, cudaStream_t s) {
    const int64_t nc = static_cast<int64_t>(nx) * nx * nx;
    const double inv_scale = ldexp(1.0, -shift_s);
    const double dx3 = dx * dx * dx;
    if (prec == RRG_PREC_FP64)
        launch_pdl(wave_source_kernel<double>, div_up(nc, 256), 256, 0, s, nc, mgrid, inv_scale,
                   dx3, 1.0 / dx3, rho_mean, scale, static_cast<double*>(src), zero_grid);
    else
        launch_pdl(wave_source_kernel<float>, div_up(nc, 256), 256, 0, s, nc, mgrid, inv_scale,
                   dx3, 1.0 / dx3, rho_mean, scale, static_cast<float*>(src), zero_grid);
    RRG_LAUNCHED();
}

void launch_wave_inc_prep(int nx, bool first, const unsigned long long* mg,
                          unsigned long long* mg_zero, int shift_s, double dx, double rho_sub,
                          const float* phi0, const float* phi_prev, const WaveCoef& w, float* g,
                          float* d, float* d_old, float* src, cudaStream_t s) {
    const int V = nx % 4 == 0 ? 4 : nx % 2 == 0 ? 2 : 1;
    const int64_t units = static_cast<int64_t>(nx / V) * nx * nx;
    auto go = [&](auto* kernel) {
        launch_pdl(kernel, div_up(units, 256), 256, 0, s, nx, mg, mg_zero, ldexp(1.0, -shift_s),
                   1.0 / (dx * dx * dx), rho_sub, phi0, phi_prev, w.K_F, w.K_MAIN,
                   w.K_ACTUAL + w.K_OLD - 1.0, static_cast<float>(w.K_OLD), g, d, d_old, src);
        RRG_LAUNCHED();
    };
    if (first) {
        if (V == 4) go(wave_inc_prep_kernel<4, true>);
        else if (V == 2) go(wave_inc_prep_kernel<2, true>);
        else go(wave_inc_prep_kernel<1, true>);
    } else {
        if (V == 4) go(wave_inc_prep_kernel<4, false>);
        else if (V == 2) go(wave_inc_prep_kernel<2, false>);
        else go(wave_inc_prep_kernel<1, false>);
    }
}

void launch_wave_inc_finish(int nx, const float* phi0, const float* d_fin, const float* d_prv,
                            float* fin, float* prv, cudaStream_t s) {
    const int64_t nc = static_cast<int64_t>(nx) * nx * nx;
    wave_inc_finish_kernel<<<div_up(nc, 256), 256, 0, s>>>(nc, phi0, d_fin, d_prv, fin, prv);
    RRG_LAUNCHED();
}

namespace {

// V-cell units of a thread's 16 bytes (or fewer, for the row length)
int cells_per_thread(int nx, bool f64) {
    if (!f64 && nx % 4 == 0) return 4;
    return nx % 2 == 0 ? 2 : 1;
}

struct VecArgs {
    const void* phi;
    void* old;
    const void* src;
    void* f = nullptr;                      // VEC_ADJ
    unsigned long long* maxbits = nullptr;  // VEC_STEP
    const void* phi0 = nullptr;             // VEC_LAST
    void* fin = nullptr;
    void* prv = nullptr;
};

template <typename R, int V, int ZC, VecMode MODE>
void launch_vec(const WaveDev& w, const VecArgs& a, cudaStream_t s) {
    const dim3 grid(div_up(static_cast<int64_t>(w.nx / V) * w.nx, kVecThreads), div_up(w.nx, ZC));
    auto go = [&](auto* kernel) {
        launch_pdl(kernel, grid, kVecThreads, 0, s, static_cast<const R*>(a.phi),
                   static_cast<R*>(a.old), static_cast<const R*>(a.src), w, a.maxbits,
                   static_cast<R*>(a.f), static_cast<const R*>(a.phi0), static_cast<R*>(a.fin),
                   static_cast<R*>(a.prv));
        RRG_LAUNCHED();
    };
    if constexpr (MODE == VEC_STEP) {
        if (a.maxbits) {
            go(wave_periodic_vec_kernel<R, V, ZC, true, MODE>);
            return;
        }
    }
    go(wave_periodic_vec_kernel<R, V, ZC, false, MODE>);
}

// z-chunk: 2 planes (the most loads in flight, the shortest chain), or 4 where those blocks fill one
// wave of six per SM and those of 2 planes take a second. Measured with 2 / 4 / 8 planes, us per
// substep: FP32 64^3 1.72 / 2.28 / 4.59, 96^3 2.64 / 3.09 / 5.38, 112^3 (0.79 of a wave)
// 3.71 / 3.62 / 6.83, 256^3 38.9 / 40.4 / 46.3; FP64 96^3 (0.97) 4.16 / 3.72 / 8.27, 128^3
// 7.37 / 7.80 / 9.72.
template <typename R, int V, VecMode MODE>
void launch_vec_z(const WaveDev& w, const VecArgs& a, cudaStream_t s) {
    int dev = 0;
    RRG_CUDA(cudaGetDevice(&dev));
    const int64_t wave = 6ll * num_sms(dev);
    const int64_t rows = div_up(static_cast<int64_t>(w.nx / V) * w.nx, kVecThreads);
    const int64_t b2 = rows * div_up(w.nx, 2), b4 = rows * div_up(w.nx, 4);
    if (b2 > wave && b4 <= wave && 4 * b4 >= 3 * wave) launch_vec<R, V, 4, MODE>(w, a, s);
    else launch_vec<R, V, 2, MODE>(w, a, s);
}

template <VecMode MODE>
void launch_vec_any(int prec, const WaveDev& w, const VecArgs& a, cudaStream_t s) {
    const bool f64 = prec == RRG_PREC_FP64;
    const int V = cells_per_thread(w.nx, f64);
    if (f64) {
        if constexpr (MODE != VEC_LAST) {  // (the incremental solves are FP32)
            if (V == 2) launch_vec_z<double, 2, MODE>(w, a, s);
            else launch_vec_z<double, 1, MODE>(w, a, s);
        }
    } else {
        if (V == 4) launch_vec_z<float, 4, MODE>(w, a, s);
        else if (V == 2) launch_vec_z<float, 2, MODE>(w, a, s);
        else launch_vec_z<float, 1, MODE>(w, a, s);
    }
}

WaveDev periodic_dev(int nx, double km, double ka, double ko, double kf) {
    WaveDev w{};
    w.nx = nx;
    w.uniform = 1;
    w.bc = RRG_BC_PERIODIC;
    w.K_MAIN = km;
    w.K_ACTUAL = ka;
    w.K_OLD = ko;
    w.K_F = kf;
    return w;
}

}  // namespace

void launch_wave_inc_last(int nx, const float* d, const float* d_old, const float* g,
                          const float* phi0, float* fin, float* prv, const WaveCoef& w,
                          cudaStream_t s) {
    VecArgs a{d, const_cast<float*>(d_old), g};
    a.phi0 = phi0;
    a.fin = fin;
    a.prv = prv;
    launch_vec_any<VEC_LAST>(RRG_PREC_FP32,
                             periodic_dev(nx, w.K_MAIN, w.K_ACTUAL, w.K_OLD, 1.0), a, s);
}

void launch_wave_adjoint_step(int prec, int nx, const void* C, void* P, void* F, double km,
                              double ka, double beta, double kf, cudaStream_t s) {
    VecArgs a{C, P, nullptr};
    a.f = F;
    launch_vec_any<VEC_ADJ>(prec, periodic_dev(nx, km, ka, beta, kf), a, s);
}

void launch_wave_step(int prec, int nx, const void* phi, void* phi_old_inout, const void* src,
                      const WaveCoef& c, unsigned long long* maxbits, cudaStream_t s) {
    WaveDev w;
    w.nx = nx;
    w.bc = c.bc_type;
    w.uniform = (c.bc_type == RRG_BC_PERIODIC && !c.keep_layer) ? 1 : 0;
    w.K_MAIN = c.K_MAIN;
    w.K_ACTUAL = c.K_ACTUAL;
    w.K_OLD = c.K_OLD;
    w.K_F = c.K_F;
    w.C = c.C;
    w.DT = c.DT;
    w.DX = c.DX;
    w.diss_base = c.diss_base;
    w.diss_extra = c.diss_extra;
    w.sim_l = c.sim_l;
    w.domain_min = c.domain_min;
    w.bc_mass = c.bc_mass;
    w.comx = c.com[0];
    w.comy = c.com[1];
    w.comz = c.com[2];
    w.r_min = c.r_min;
    const bool check = maxbits != nullptr;
    if (w.uniform) {
        VecArgs a{phi, phi_old_inout, src};
        a.maxbits = maxbits;
        launch_vec_any<VEC_STEP>(prec, w, a, s);
        return;
    }
    const int gx = div_up(nx, kTX), gy = div_up(nx, kTY);
    // z-chunk: trade wave efficiency (blocks against 8 resident 256-thread blocks per SM)
    // against the one extra plane each column loads per chunk
    int dev = 0;
    RRG_CUDA(cudaGetDevice(&dev));
    const int sms = num_sms(dev);
    const int64_t slots = static_cast<int64_t>(sms) * 8;
    int zc = 32;
    double best = -1.0;
    for (int cand : {2, 4, 8, 16, 32, 64}) {
        if (cand > nx && cand != 2) break;
        const int64_t blocks = static_cast<int64_t>(gx) * gy * div_up(nx, cand);
        const int64_t waves = (blocks + slots - 1) / slots;
        const double eff = static_cast<double>(blocks) / static_cast<double>(waves * slots) *
                           cand / (cand + 1.0);
        if (eff > best + 1e-9) {
            best = eff;
            zc = cand;
        }
    }
    w.zc = zc;
    dim3 grid(gx, gy, div_up(nx, zc));
    dim3 block(kTX, kTY);
#define RRG_WAVE_LAUNCH(R)                                                                    \
    do {                                                                                      \
        const R* p = static_cast<const R*>(phi);                                              \
        R* po = static_cast<R*>(phi_old_inout);                                               \
        const R* sr = static_cast<const R*>(src);                                             \
        if (check) wave_step_kernel<R, true><<<grid, block, 0, s>>>(p, po, sr, w, maxbits);   \
        else wave_step_kernel<R, false><<<grid, block, 0, s>>>(p, po, sr, w, maxbits);        \
    } while (0)
    if (prec == RRG_PREC_FP64) RRG_WAVE_LAUNCH(double);
    else RRG_WAVE_LAUNCH(float);
#undef RRG_WAVE_LAUNCH
    RRG_LAUNCHED();
}

namespace {

template <typename R, int V>
void launch_gradient_vec(int nx, double coef, const void* phi, void* acc4, cudaStream_t s) {
    constexpr int ZC = 2;
    const dim3 grid(div_up(static_cast<int64_t>(nx / V) * nx, kGradThreads), div_up(nx, ZC));
    launch_pdl(gradient_vec_kernel<R, V, ZC>, grid, kGradThreads, 0, s, nx, static_cast<R>(coef),
               static_cast<const R*>(phi), static_cast<V4<R>*>(acc4));
    RRG_LAUNCHED();
}

}  // namespace

void launch_gradient(int prec, int nx, double dx, const void* phi, void* acc4, cudaStream_t s) {
    const double coef = -1.0 / dx;
    const bool f64 = prec == RRG_PREC_FP64;
    const int V = cells_per_thread(nx, f64);
    if (f64) {
        if (V == 2) launch_gradient_vec<double, 2>(nx, coef, phi, acc4, s);
        else launch_gradient_vec<double, 1>(nx, coef, phi, acc4, s);
    } else {
        if (V == 4) launch_gradient_vec<float, 4>(nx, coef, phi, acc4, s);
        else if (V == 2) launch_gradient_vec<float, 2>(nx, coef, phi, acc4, s);
        else launch_gradient_vec<float, 1>(nx, coef, phi, acc4, s);
    }
}

void launch_interp(int prec, int64_t n, const void* posm, const void* poslo, const GridDev& g,
                   const void* acc4, void* acc, cudaStream_t s) {
    const int b = div_up(n, 256);
    if (prec == RRG_PREC_FP64)
        interp_kernel<double><<<b, 256, 0, s>>>(n, posm, nullptr, g,
                                                static_cast<const V4<double>*>(acc4),
                                                static_cast<V4<double>*>(acc));
    else
        interp_kernel<float><<<b, 256, 0, s>>>(
            n, posm, prec == RRG_PREC_MIXED ? static_cast<const V4<float>*>(poslo) : nullptr, g,
            static_cast<const V4<float>*>(acc4), static_cast<V4<float>*>(acc));
    RRG_LAUNCHED();
}

void launch_ngp_phi(int prec, int64_t n, const void* posm, const void* poslo, const GridDev& g,
                    const void* phi, void* pot, cudaStream_t s) {
    const int b = div_up(n, 256);
    if (prec == RRG_PREC_FP64)
        ngp_phi_kernel<double><<<b, 256, 0, s>>>(n, posm, nullptr, g,
                                                 static_cast<const double*>(phi),
                                                 static_cast<double*>(pot));
    else
        ngp_phi_kernel<float><<<b, 256, 0, s>>>(
            n, posm, prec == RRG_PREC_MIXED ? static_cast<const V4<float>*>(poslo) : nullptr, g,
            static_cast<const float*>(phi), static_cast<float*>(pot));
    RRG_LAUNCHED();
}

void launch_ngp_project(int prec, int64_t n, const void* posm, const void* poslo,
                        const GridDev& g, int* count, const void* pot, const void* acc,
                        void* phi_grid, void* acc4_grid, cudaStream_t s) {
    const int b = div_up(n, 256);
    const V4<float>* lo = prec == RRG_PREC_MIXED ? static_cast<const V4<float>*>(poslo) : nullptr;
    if (prec == RRG_PREC_FP64) {
        ngp_count_kernel<double><<<b, 256, 0, s>>>(n, posm, nullptr, g, count);
        RRG_LAUNCHED();
        ngp_project_kernel<double><<<b, 256, 0, s>>>(
            n, posm, nullptr, g, count, static_cast<const double*>(pot),
            static_cast<const V4<double>*>(acc), static_cast<double*>(phi_grid),
            static_cast<double*>(acc4_grid));
    } else {
        ngp_count_kernel<float><<<b, 256, 0, s>>>(n, posm, lo, g, count);
        RRG_LAUNCHED();
        ngp_project_kernel<float><<<b, 256, 0, s>>>(
            n, posm, lo, g, count, static_cast<const float*>(pot),
            static_cast<const V4<float>*>(acc), static_cast<float*>(phi_grid),
            static_cast<float*>(acc4_grid));
    }
    RRG_LAUNCHED();
}

void launch_pm_particles(const PmParticleArgs& a, int mode, cudaStream_t s) {
    const double scale = ldexp(1.0, a.shift_s);
    if (a.prec == RRG_PREC_FP64) dispatch_pm<double, false>(a, mode, scale, s);
    else if (a.prec == RRG_PREC_MIXED) dispatch_pm<float, true>(a, mode, scale, s);
    else dispatch_pm<float, false>(a, mode, scale, s);
    RRG_LAUNCHED();
}

}  // namespace rrg
