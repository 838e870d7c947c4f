// Shared by the direct-sum kernels (direct.cu, direct_sym.cu): tile length, padding and the
// leapfrog epilogue of a particle's finished force.
#pragma once

#include "kernels.cuh"

namespace rrg {

constexpr int kDirectThreads = 256;   // threads per block = j-tile length
constexpr float kDirectPad = 1e18f;   // padding particles: far away and massless

template <typename R>
struct EpiDev {
    int mode;
    R dt;
    V4<R>* acc;
    R* pot;
    V4<R>* vel;
    V4<R>* u;
    V4<R>* pos_out;
    V4<float>* lo_out;
};

template <typename R>
EpiDev<R> make_epi(const DirectEpi& e) {
    EpiDev<R> d;
    d.mode = e.mode;
    d.dt = static_cast<R>(e.dt);
    d.acc = static_cast<V4<R>*>(e.acc);
    d.pot = static_cast<R*>(e.pot);
    d.vel = static_cast<V4<R>*>(e.vel);
    d.u = static_cast<V4<R>*>(e.u);
    d.pos_out = static_cast<V4<R>*>(e.pos_out);
    d.lo_out = static_cast<V4<float>*>(e.lo_out);
    return d;
}

// Per-particle epilogue. Arithmetic order follows predict_step_ / correct_step_
// (nbody.cu:139-151, 175-180): v = 0.5 (u + dt a) with u = v_old + v*, v* = v + dt a,
// x += (dt 0.5) (v + v*).
template <typename R, bool MIXED>
__device__ __forceinline__ void apply_epi(const EpiDev<R>& e, int64_t i, R ax, R ay, R az,
                                          R phi, bool want_pot, const V4<R>* posm,
                                          const V4<float>* poslo) {
    if (want_pot && e.pot) e.pot[i] = phi;
    if (e.mode == EPI_STORE) {
        e.acc[i] = v4<R>(ax, ay, az, R(0));
        return;
    }
    const V4<R> u = e.u[i];
    const R dt = e.dt;
    const R vx = R(0.5) * (u.x + dt * ax);
    const R vy = R(0.5) * (u.y + dt * ay);
    const R vz = R(0.5) * (u.z + dt * az);
    if (e.mode == EPI_CORRECT) {
        e.vel[i] = v4<R>(vx, vy, vz, R(0));
        e.acc[i] = v4<R>(ax, ay, az, R(0));
        return;
    }
    // EPI_CORRECT_PREDICT: next step's predict on the corrected velocity; the synced (v, a)
    // of this step are stored too where the caller asks (checkpoints)
    if (e.vel) e.vel[i] = v4<R>(vx, vy, vz, R(0));
    if (e.acc) e.acc[i] = v4<R>(ax, ay, az, R(0));
    const R sx = vx + dt * ax, sy = vy + dt * ay, sz = vz + dt * az;  // v*
    const R ux = vx + sx, uy = vy + sy, uz = vz + sz;
    e.u[i] = v4<R>(ux, uy, uz, R(0));
    const R hdt = dt * R(0.5);
    const V4<R> p = posm[i];
    if constexpr (MIXED) {
        const V4<float> lo = poslo[i];
        float hx = p.x, lx = lo.x, hy = p.y, ly = lo.y, hz = p.z, lz = lo.z;
        df_add(hx, lx, hdt * ux);
        df_add(hy, ly, hdt * uy);
        df_add(hz, lz, hdt * uz);
        e.pos_out[i] = v4<R>(hx, hy, hz, p.w);
        e.lo_out[i] = v4<float>(lx, ly, lz, 0.f);
    } else {
        e.pos_out[i] = v4<R>(p.x + hdt * ux, p.y + hdt * uy, p.z + hdt * uz, p.w);
    }
}

}  // namespace rrg
