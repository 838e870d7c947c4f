// Three damped-wave substeps per launch (wave_diss_iteration, wave.cu:106-193, FP32 periodic box
// without an absorbing layer) for grids whose levels do not stay in L2.
//
// One substep per launch reads two levels and the source and writes a level, 16 B per cell: at the
// HBM limit from ~200^3 on (256^3: 268 MB in 38.9 us). Here a block marches its tile of rows up z
// with T = 3 substeps in flight: when plane p of level 0 arrives, level k is computed on plane
// p - k (k = 1 .. 3), so two levels and the source are read once and two levels written once per
// three substeps, 20 B per cell instead of 48. The price is a halo of three cells around each tile,
// computed by several blocks from the same values by the same expression (wave_cell's roundings):
// the results are the bits of one substep per launch.
//
// A warp owns two adjacent rows of the tile, a lane two cells of each: the x neighbours are
// shuffles, the y neighbour between the two rows is in registers, those outside come from shared
// memory, where the step before left the centre plane of every level (one barrier per plane). The
// inputs come by asynchronous copies kAhead planes ahead into the same memory. Each thread keeps
// three planes of every level and of the source in registers; the plane loop is unrolled by three,
// so that every ring index is a constant and no value moves. New levels go to other buffers than
// the ones read: the neighbours' halos need the old ones.
//
// Bound: shared-memory and shuffle throughput (256^3, a steady launch: shared-memory wavefronts 69 %,
// DRAM 3.5 TB/s, issue 42 % of the active cycles, the longest waits on shared-memory results and their
// queue; the halos cost 1.9 times the arithmetic).
// Tried and slower at 256^3, us per substep: loads three planes ahead into registers instead of
// the copies 32.0, the sums over the steps before formed for all levels first 30.6, 40 rows per
// block 29.9, four cells per lane with 48 rows and one even share of all planes per block 33.8
// (its blocks drift apart, and the halos come from DRAM again).
#include <algorithm>

#include "kernels.cuh"
#include "wave_cells.cuh"

namespace rrg {
namespace {

constexpr int T = 3;                     // substeps per launch
constexpr int kHalo = 2;                 // halo lanes on each side of a tile (2 cells each, >= T)
constexpr int kLanes = 32 - 2 * kHalo;   // interior lanes
constexpr int kMaxRows = 32;
constexpr int kStages = 6;               // planes in shared memory, copied kAhead steps ahead: the
constexpr int kAhead = kStages - 2;      // one before is still read, the one overwritten is not

struct MarchArgs {
    const float* cur;   // level 0 and the one before it (null: zero)
    const float* old;
    const float* src;
    float* out;         // level 3 and level 2
    float* out_old;
    float km, ka, ko, kf;
    int nx, rb, zl;     // interior rows per tile, planes per block
};

__device__ __forceinline__ void copy8(uint32_t to, const float* from) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(to), "l"(from) : "memory");
}

__global__ void __launch_bounds__(16 * kMaxRows, 1) wave_march_kernel(const MarchArgs a) {
    // kStages x (level 0, the level before, source), then [level 1, 2][3 buffers], each of
    // kMaxRows x 32 cell pairs
    extern __shared__ __align__(16) float2 sm[];
    constexpr int buf = kMaxRows * 32, stage = 3 * buf;
    float2* const lv = sm + kStages * stage;
    const int lane = threadIdx.x, rows = 2 * blockDim.y, nx = a.nx, W = nx / 2;
    const int r0 = 2 * threadIdx.y;  // the warp's rows of the tile: r0, r0 + 1
    int q = static_cast<int>(blockIdx.x) * kLanes + lane - kHalo;
    const bool inside = lane >= kHalo && lane < 32 - kHalo && q < W;
    q %= W;
    if (q < 0) q += W;
    bool mine[2];
    int at[2];  // the rows' cells in a plane
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        int y = static_cast<int>(blockIdx.y) * a.rb + r0 + r - T;
        mine[r] = inside && r0 + r >= T && r0 + r < T + a.rb && y < nx;
        y %= nx;
        if (y < 0) y += nx;
        at[r] = y * nx + 2 * q;
    }
    const int plane = nx * nx;
    const int z0 = static_cast<int>(blockIdx.z) * a.zl, zl = min(a.zl, nx - z0);
    const int up = min(r0 + 2, rows - 1) * 32 + lane, dn = max(r0 - 1, 0) * 32 + lane;
    const int me = r0 * 32 + lane;
    const uint32_t sm0 = static_cast<uint32_t>(__cvta_generic_to_shared(sm + me));
    const float2 km = make_float2(a.km, a.km), ka = make_float2(a.ka, a.ka),
                 ko = make_float2(a.ko, a.ko), kf = make_float2(a.kf, a.kf);
    const float2 zero = make_float2(0.f, 0.f);
    const int steps = zl + 2 * T;

    pdl_next();
    pdl_wait();
    // the copies of step s: level 0 of plane z0 - T + s, the level before and the source of the
    // plane below it
    int zc = z0 - T, zo = z0 - T - 1;
    if (zc < 0) zc += nx;
    if (zo < 0) zo += nx;
    int sc = 0;  // stage of the next copies
    auto load = [&](bool go) {
        if (go) {
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const uint32_t to = sm0 + 8u * (sc + 32 * r);
                copy8(to, a.cur + (zc * plane + at[r]));
                if (a.old) copy8(to + 8u * buf, a.old + (zo * plane + at[r]));
                copy8(to + 16u * buf, a.src + (zo * plane + at[r]));
            }
            zo = zc;
            zc = zc + 1 == nx ? 0 : zc + 1;
            sc = sc + stage == kStages * stage ? 0 : sc + stage;
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll 1
    for (int f = 0; f < kAhead; ++f) load(f < steps);

    float2 v[T][3][2];  // level k, plane p - k in slot f, the planes below in f - 1, f - 2
    float2 g[3][2];     // source of plane p - 1 in slot f
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            g[i][r] = zero;
#pragma unroll
            for (int k = 0; k < T; ++k) v[k][i][r] = zero;
        }
    int so = 0, so_last = (kStages - 1) * stage;  // stages of this step and of the one before
#pragma unroll 1
    for (int s0 = 0; s0 < steps; s0 += 3) {
#pragma unroll
        for (int f = 0; f < 3; ++f) {
            const int s = s0 + f;
            if (s >= steps) break;
            constexpr int next[3] = {1, 2, 0}, last[3] = {2, 0, 1};
            load(s + kAhead < steps);
            asm volatile("cp.async.wait_group %0;" ::"n"(kAhead) : "memory");
            float2 old[2];
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                v[0][f][r] = sm[so + me + 32 * r];
                old[r] = a.old ? sm[so + buf + me + 32 * r] : zero;
                g[f][r] = sm[so + 2 * buf + me + 32 * r];
            }
            // level k on plane p - k, from level k - 1 on planes p - k - 1 .. p - k + 1
#pragma unroll
            for (int k = 1; k <= T; ++k) {
                if (s < 2 * k) break;  // (its planes start at z0 - T + k)
                const float2* const from =
                    k == 1 ? sm + so_last : lv + ((k - 2) * 3 + last[f]) * buf;
                const float2 below = from[dn], above = from[up];
                const float2 c0 = v[k - 1][last[f]][0], c1 = v[k - 1][last[f]][1];
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const float2 c = r ? c1 : c0;
                    const float lft = __shfl_up_sync(0xffffffffu, c.y, 1);
                    const float rgt = __shfl_down_sync(0xffffffffu, c.x, 1);
                    float2 nb = make_float2(__fadd_rn(lft, c.y), __fadd_rn(c.x, rgt));
                    nb = __fadd2_rn(__fadd2_rn(nb, r ? c0 : below), r ? above : c1);
                    nb = __fadd2_rn(__fadd2_rn(nb, v[k - 1][next[f]][r]), v[k - 1][f][r]);
                    const float2 before = k == 1 ? old[r] : v[k >= 2 ? k - 2 : 0][next[f]][r];
                    // the source of plane p - k: slot f - (k - 1)
                    const float2 gs = g[(f + 4 - k) % 3][r];
                    const float2 out = __ffma2_rn(
                        gs, kf, __ffma2_rn(before, ko, __ffma2_rn(c, ka, __fmul2_rn(nb, km))));
                    if (k < T) {
                        v[k < T ? k : 0][f][r] = out;
                        lv[((k - 1) * 3 + f) * buf + me + 32 * r] = out;
                    } else if (mine[r]) {
                        const int o = (z0 + s - 2 * T) * plane + at[r];
                        *reinterpret_cast<float2*>(a.out + o) = out;
                        *reinterpret_cast<float2*>(a.out_old + o) = c;
                    }
                }
            }
            so_last = so;
            so = so + stage == kStages * stage ? 0 : so + stage;
            __syncthreads();
        }
    }
}

// Rows per tile and planes per block: the fewest row-steps on the busiest SM (one block each).
void choose_tile(int nx, int sms, int& rb, int& zl) {
    const int tx = (nx / 2 + kLanes - 1) / kLanes;
    int64_t best = 0;
    for (int rows = 8; rows <= kMaxRows; rows += 2) {
        const int b = rows - 2 * T, ty = (nx + b - 1) / b;
        for (int cz = 1; cz <= nx / 8 + 1; ++cz) {
            const int z = (nx + cz - 1) / cz;
            const int64_t blocks = static_cast<int64_t>(tx) * ty * ((nx + z - 1) / z);
            const int64_t cost = (blocks + sms - 1) / sms * (z + 2 * T) * (rows + 2);
            if (best == 0 || cost < best) {
                best = cost;
                rb = b;
                zl = z;
            }
        }
    }
}

}  // namespace

// 20 B per cell and three substeps of HBM traffic pay once the levels and the source that one
// substep touches (12 B per cell) take more than two thirds of L2; below, the substeps run from
// L2. us per substep, one launch each / marched: 192^3 13.4 / 14.4, 200^3 17.7 / 16.2, 224^3
// 26.7 / 17.6, 256^3 38.9 / 29.6, 288^3 54.7 / 40.5, 320^3 74.4 / 54.7; rows of 2 mod 4 cells
// 198^3 20.8 / 16.0, 258^3 47.1 / 33.
bool wave_march_applies(int nx) {
    if (nx % 2 != 0) return false;
    int dev = 0, l2 = 0;
    RRG_CUDA(cudaGetDevice(&dev));
    RRG_CUDA(cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, dev));
    return 18.0 * nx * nx * nx > l2;
}

void launch_wave_march(int nx, const float* cur, const float* old, const float* src, float* out,
                       float* out_old, double km, double ka, double ko, double kf,
                       cudaStream_t s) {
    RRG_REQUIRE(nx % 2 == 0 && nx >= 8, RRG_ERR_INVALID, "wave march: rows of cell pairs");
    int dev = 0;
    RRG_CUDA(cudaGetDevice(&dev));
    MarchArgs a{cur, old, src, out, out_old, static_cast<float>(km), static_cast<float>(ka),
                static_cast<float>(ko), static_cast<float>(kf), nx, 0, 0};
    choose_tile(nx, num_sms(dev), a.rb, a.zl);
    const dim3 grid((nx / 2 + kLanes - 1) / kLanes, div_up(nx, a.rb), div_up(nx, a.zl));
    constexpr size_t smem = sizeof(float2) * (kStages + T - 1) * 3 * kMaxRows * 32;
    RRG_CUDA(cudaFuncSetAttribute(wave_march_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  static_cast<int>(smem)));
    launch_pdl(wave_march_kernel, grid, dim3(32, (a.rb + 2 * T) / 2), smem, s, a);
    RRG_LAUNCHED();
}

}  // namespace rrg
