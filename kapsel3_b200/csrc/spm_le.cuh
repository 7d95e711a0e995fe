// Lees-Edwards (sheared) step: kernels in oblique coordinates.
//
// The velocity field is held on the sheared grid with contravariant
// components; degree_oblique (gamma) grows by Shear_rate*dt per step
// (Time_evolution_hydro_OBL, sp_3d_ns.cxx:328-433).  gamma is tracked on the
// host and passed by value; Shear_rate_eff (which the reference corrects by a
// field average every step, sp_3d_ns.h:189-203) lives on the device.
#pragma once

#include "spm_common.cuh"
#include "spm_kernels.cuh"

namespace spm {

// Field slots the Lees-Edwards step needs beyond the common arena: the
// Cartesian velocity ucp (3) and one spare.
constexpr int LE_EXTRA_SLOTS = 4;

// Device-side scalars of the sheared run.
struct LEDev {
    double srate_eff;   // Shear_rate_eff
    double strain;      // Shear_strain_realized
    double correction;  // field-average part of Calc_shear_rate_eff
    double reynolds;    // Inertia_stress (Calc_Reynolds_shear_stress)
    double hydro_old;   // hydro_stress[1][0] from Hydro_force
    double hydro_new;   // hydro_stress[1][0] from Hydro_force_new
    double lj;          // dev_shear_stress_lj * Ivolume
    double time;
};

struct LEState {
    int     enabled        = 0;
    double  shear_rate     = 0.0;
    double  degree_oblique = 0.0;
    double  xy_aspect      = 1.0;
    LEDev  *dev            = nullptr;  // device scalars
    double *ppart          = nullptr;  // per-particle stress partials [Np][kLePart]
    double *partial        = nullptr;  // per-CTA partial sums of the field reductions
    double  stress_host[8] = {0, 0, 0, 0, 0, 0, 0, 0};
};

// ---------------------------------------------------------------------------
// k-space helpers (oblique metric)
// ---------------------------------------------------------------------------
__device__ __forceinline__ double ik2_obl(const KPoint &p, double gam) {
    const double a  = p.ky - p.kx * gam;
    const double k2 = p.kx * p.kx + a * a + p.kz * p.kz;  // Update_K2_OBL (fluid_solver.h:342-361)
    return k2 > 0.0 ? 1.0 / k2 : 0.0;
}
__device__ __forceinline__ double k2_obl(const KPoint &p, double gam) {
    const double a = p.ky - p.kx * gam;
    return p.kx * p.kx + a * a + p.kz * p.kz;
}

// reduced contravariant vorticity -> full (case split on KX, then KZ:
// Zeta_k2u_k_OBL / Zeta_k2omega_k_OBL, fft_wrapper.cxx:714-745, 806-845)
template <typename T>
__device__ __forceinline__ void zeta_to_omega_obl(const KPoint &p, cplx<T> z0, cplx<T> z1, cplx<T> om[3]) {
    if (p.KX != 0) {
        const T a  = -(T)(1.0 / p.kx);
        const T ky = (T)p.ky, kz = (T)p.kz;
        om[0]      = cplx<T>{a * (ky * z0.re + kz * z1.re), a * (ky * z0.im + kz * z1.im)};
        om[1]      = z0;
        om[2]      = z1;
    } else if (p.KZ != 0) {
        const T dmy = (T)(-(p.ky / p.kz));
        om[0]       = z1;
        om[1]       = z0;
        om[2]       = cplx<T>{dmy * z0.re, dmy * z0.im};
    } else {
        om[0] = z0;
        om[1] = cplx<T>{0, 0};
        om[2] = z1;
    }
}
// Omega_k2zeta_k_OBL (fft_wrapper.cxx:265-292)
template <typename T>
__device__ __forceinline__ void omega_to_zeta_obl(const KPoint &p, const cplx<T> om[3], cplx<T> &z0, cplx<T> &z1) {
    if (p.KX != 0) {
        z0 = om[1];
        z1 = om[2];
    } else if (p.KZ != 0) {
        z0 = om[1];
        z1 = om[0];
    } else {
        z0 = om[0];
        z1 = om[2];
    }
}
// contra2co_single (fft_wrapper.h:613-622)
template <typename T>
__device__ __forceinline__ void contra2co(cplx<T> v[3], T g) {
    const cplx<T> a = v[0], b = v[1];
    v[0]            = cplx<T>{a.re + g * b.re, a.im + g * b.im};
    v[1]            = cplx<T>{g * a.re + ((T)1 + g * g) * b.re, g * a.im + ((T)1 + g * g) * b.im};
}

// u_hat (contravariant) from zeta: Zeta_k2u_k_OBL (fft_wrapper.cxx:690-768)
template <typename T>
__device__ __forceinline__ void zeta_to_u_obl(const KPoint &p, cplx<T> z0, cplx<T> z1, double gam, cplx<T> u[3]) {
    cplx<T> om[3];
    zeta_to_omega_obl<T>(p, z0, z1, om);
    contra2co<T>(om, (T)gam);
    const T ik2 = (T)ik2_obl(p, gam);
    i_cross<T>((T)p.kx * ik2, (T)p.ky * ik2, (T)p.kz * ik2, om, u);
}

// ---------------------------------------------------------------------------
// zeta -> u_hat (contra) [+ omega_hat] of the oblique advection term
// (Zeta_k2u_cpuky + Zeta_k2omega_OBL, operate_omega.h:150-185).
// ---------------------------------------------------------------------------
// BOX: only the retained 2/3 box is visited (the step: the pruned inverse
// passes read everything outside it as zero); else every mode (getters).
template <typename T, int BOX>
__global__ void k_le_zeta_to_u(Grid g, const cplx<T> *__restrict__ z0p, const cplx<T> *__restrict__ z1p,
                               const double *__restrict__ uk_dc, double gam, cplx<T> *__restrict__ u0,
                               cplx<T> *__restrict__ u1, cplx<T> *__restrict__ u2, cplx<T> *__restrict__ w0,
                               cplx<T> *__restrict__ w1, cplx<T> *__restrict__ w2) {
    for_modes<BOX>(g, [&](size_t idx, const KPoint &p, bool valid) {
        cplx<T> u[3] = {{0, 0}, {0, 0}, {0, 0}}, om[3] = {{0, 0}, {0, 0}, {0, 0}};
        if (valid) {
            const cplx<T> z0 = z0p[idx], z1 = z1p[idx];
            zeta_to_u_obl<T>(p, z0, z1, gam, u);
            if (w0) zeta_to_omega_obl<T>(p, z0, z1, om);
        }
        if (idx == 0) {
            u[0].re = (T)uk_dc[0];
            u[1].re = (T)uk_dc[1];
            u[2].re = (T)uk_dc[2];
            om[0].re = om[1].re = om[2].re = (T)0;  // omega[d][0] = 0 (fft_wrapper.cxx:841-843)
        }
        u0[idx] = u[0];
        u1[idx] = u[1];
        u2[idx] = u[2];
        if (w0) {
            w0[idx] = om[0];
            w1[idx] = om[1];
            w2[idx] = om[2];
        }
    });
}

// a = u x omega (real space, operate_omega.cxx:113-136), in place over u.
template <typename T>
__global__ void r_le_cross(Grid g, T *__restrict__ u0, T *__restrict__ u1, T *__restrict__ u2,
                           const T *__restrict__ w0, const T *__restrict__ w1, const T *__restrict__ w2) {
    const size_t rowlen = 2 * (size_t)g.hnzp;
    const size_t n      = (size_t)g.nx * g.ny * rowlen;
    for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < n; idx += (size_t)gridDim.x * blockDim.x) {
        if ((int)(idx % rowlen) >= g.nz) continue;
        const T a = u0[idx], b = u1[idx], c = u2[idx];
        const T x = w0[idx], y = w1[idx], z = w2[idx];
        u0[idx] = b * z - c * y;
        u1[idx] = c * x - a * z;
        u2[idx] = a * y - b * x;
    }
}

// Oblique advection closure and slaved-Euler update
// (operate_omega.cxx:138-154, fluid_solver.cxx:411-437): a_hat -= 2 srate
// (1, gamma, 0) u_hat_y; f = reduced (i k x a_hat); zeta += (e^{-nu dt K2}-1)
// (zeta - IK2 f / nu) on the retained modes with the oblique K2.
// Over the retained box; modes outside it are not read again before
// k_le_project_to_zeta writes every mode.  The thread of mode 0 then applies
// FIX_CELLxyz to uk_dc (k_fix_cell).
template <typename T>
__global__ void k_le_ns_update(Grid g, cplx<T> *__restrict__ z0p, cplx<T> *__restrict__ z1p,
                               const cplx<T> *__restrict__ a0p, const cplx<T> *__restrict__ a1p,
                               const cplx<T> *__restrict__ a2p, RunWords *__restrict__ rw,
                               const LEDev *__restrict__ le, double gam, double nu, double dt) {
    const double srate = le->srate_eff;
    for_modes<2>(g, [&](size_t idx, const KPoint &p, bool) {
        const cplx<T> z0 = z0p[idx], z1 = z1p[idx];
        cplx<T>       u[3];
        zeta_to_u_obl<T>(p, z0, z1, gam, u);
        if (idx == 0) {
            u[1].re = (T)rw->uk_dc[1];
            for (int d = 0; d < 3; d++)
                if (rw->fix_mask & (1 << d)) rw->uk_dc[d] = 0.0;
        }
        cplx<T>  a[3] = {a0p[idx], a1p[idx], a2p[idx]};
        const T  c0   = (T)(2.0 * srate);
        const T  c1   = (T)(2.0 * srate * gam);
        a[0].re -= c0 * u[1].re;
        a[0].im -= c0 * u[1].im;
        a[1].re -= c1 * u[1].re;
        a[1].im -= c1 * u[1].im;
        cplx<T> rot[3];
        i_cross<T>((T)p.kx, (T)p.ky, (T)p.kz, a, rot);
        cplx<T> f0, f1;
        omega_to_zeta_obl<T>(p, rot, f0, f1);
        const double k2 = k2_obl(p, gam);
        T            dmy;
        if (sizeof(T) == 8)
            dmy = (T)(exp(-nu * dt * k2) - 1.0);
        else
            dmy = (T)expm1(-nu * dt * k2);
        const T c = (T)((1.0 / nu) * (k2 > 0.0 ? 1.0 / k2 : 0.0));
        cplx<T> n0 = z0, n1 = z1;
        n0.re += dmy * (z0.re - c * f0.re);
        n0.im += dmy * (z0.im - c * f0.im);
        n1.re += dmy * (z1.re - c * f1.re);
        n1.im += dmy * (z1.im - c * f1.im);
        z0p[idx] = n0;
        z1p[idx] = n1;
    });
}

// Solenoidal_uk_OBL + U_k2zeta_k_OBL (operate_omega.cxx:197-227,
// fft_wrapper.cxx:528-589).
template <typename T>
__global__ void k_le_project_to_zeta(Grid g, const cplx<T> *__restrict__ u0p, const cplx<T> *__restrict__ u1p,
                                     const cplx<T> *__restrict__ u2p, cplx<T> *__restrict__ z0p,
                                     cplx<T> *__restrict__ z1p, double *__restrict__ uk_dc, double gam) {
    const size_t n = g.field_elems_c();
    for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < n; idx += (size_t)gridDim.x * blockDim.x) {
        KPoint p;
        size_t row;
        if (!k_point(g, idx, p, row)) {
            z0p[idx] = z1p[idx] = cplx<T>{0, 0};
            continue;
        }
        cplx<T>  u[3] = {u0p[idx], u1p[idx], u2p[idx]};
        const T  kx = (T)p.kx, ky = (T)p.ky, kz = (T)p.kz;
        const T  ik2 = (T)ik2_obl(p, gam);
        const T  g1  = (T)gam;
        const T  kxc = ((T)1 + g1 * g1) * kx - g1 * ky;
        const T  kyc = -g1 * kx + ky;
        const T  dr  = ik2 * (u[0].re * kx + u[1].re * ky + u[2].re * kz);
        const T  di  = ik2 * (u[0].im * kx + u[1].im * ky + u[2].im * kz);
        u[0].re -= dr * kxc;
        u[0].im -= di * kxc;
        u[1].re -= dr * kyc;
        u[1].im -= di * kyc;
        u[2].re -= dr * kz;
        u[2].im -= di * kz;
        if (idx == 0) {
            uk_dc[0] = (double)u[0].re;
            uk_dc[1] = (double)u[1].re;
            uk_dc[2] = (double)u[2].re;
        }
        contra2co<T>(u, g1);
        cplx<T> om[3];
        i_cross<T>(kx, ky, kz, u, om);
        cplx<T> a, b;
        omega_to_zeta_obl<T>(p, om, a, b);
        z0p[idx] = a;
        z1p[idx] = b;
    }
}

// Block-wide sum of K doubles (blockDim.x a multiple of 32, <= 1024); the
// result is valid in thread 0.
template <int K>
__device__ __forceinline__ void block_sumK(double v[K]) {
    __shared__ double red[32][K];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < K; k++)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
    __syncthreads();
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < K; k++) red[wid][k] = v[k];
    __syncthreads();
    if (wid == 0) {
        const int nw = blockDim.x >> 5;
#pragma unroll
        for (int k = 0; k < K; k++) {
            double a = lane < nw ? red[lane][k] : 0.0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
            v[k] = a;
        }
    }
}

// ---------------------------------------------------------------------------
// Oblique <-> Cartesian grid transfers (linear interpolation along x).
// ---------------------------------------------------------------------------
struct ShiftRow {
    int    io;     // integer x shift of the row
    int    sign;   // +-1, 0 on the middle row
    double alpha;  // interpolation weight of the neighbour
};
// orth2obl (to_oblique) / obl2orth (fft_wrapper.h:315-340)
__device__ __forceinline__ ShiftRow shift_row(int j, int ny, double gam, bool to_oblique) {
    const int    dj  = j - ny / 2;
    const double sgn = dj == 0 ? 0.0 : (dj > 0) == (gam >= 0.0) ? 1.0 : -1.0;
    const double base = (double)(int)(sgn * gam * dj);
    ShiftRow     s;
    if (to_oblique) {
        const double io = base * sgn;
        s.io            = (int)io;
        s.alpha         = (gam * dj - io) * sgn;
    } else {
        const double io = base * sgn + sgn;
        s.io            = (int)io;
        s.alpha         = (io - gam * dj) * sgn;
    }
    s.sign = (int)sgn;
    return s;
}
__device__ __forceinline__ int wrap_x(double v, int nx) { return (int)fmod(v, (double)nx); }

// ucp = U_oblique2u(u) (fft_wrapper.h:515-546): Cartesian velocity on the
// Cartesian grid, mean shear flow srate*(j - NY/2) added.  Written as a
// gather over the output points.
// One cell per thread and round, its indices by shifts and masks (every axis is a
// power of two) and its row's shift without a division or fmod: with 64-bit
// divisions per cell this kernel took 29 us and the average gradient apart 19
// us at 128^3 FP32 on B200, 24 us for both here.  (A warp per row, one shift
// for its cells, takes as long here and 36 against 28 us in r_le_force_add.)
// The cells also add up
// Calc_shear_rate_eff's average gradient of the oblique x velocity (sp_3d_ns.h:
// 166-203): one FP64 partial per CTA, summed by k_le_shear_rate.
template <typename T>
__global__ void r_le_obl2cart(Grid g, const T *__restrict__ u0, const T *__restrict__ u1, const T *__restrict__ u2,
                              T *__restrict__ c0, T *__restrict__ c1, T *__restrict__ c2, double gam,
                              double srate, double *__restrict__ partial) {
    const unsigned rowlen = 2 * (unsigned)g.hnzp, n = (unsigned)g.nx * g.ny * g.nz;
    const int      lz = 31 - __clz(g.nz), ly = 31 - __clz(g.ny);
    double         acc[1] = {0.0};
    for (unsigned t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        const unsigned k = t & (g.nz - 1), row = t >> lz;
        const int      io = (int)(row >> ly), j = (int)(row & (g.ny - 1));  // output x index (i_oblique)
        const ShiftRow s  = shift_row(j, g.ny, gam, false);
        // i_oblique = fmod(i + io_shift + 4 NX, NX)  =>  i = (io - io_shift) mod NX
        const int    i = (io - s.io) & (g.nx - 1), ip = (i + s.sign) & (g.nx - 1);
        const double beta = 1.0 - s.alpha;
        const unsigned a = ((unsigned)i * g.ny + j) * rowlen + k, b = ((unsigned)ip * g.ny + j) * rowlen + k;
        const unsigned o = row * rowlen + k;
        const int xp = (io + 1) & (g.nx - 1), xm = (io - 1) & (g.nx - 1);
        const int yp = (j + 1) & (g.ny - 1), ym = (j - 1) & (g.ny - 1);
        auto      at = [&](int x, int y) { return (double)u0[((unsigned)x * g.ny + y) * rowlen + k]; };
        const T   vy = (T)(beta * (double)u1[a] + s.alpha * (double)u1[b]);
        T         vx = (T)(beta * (double)u0[a] + s.alpha * (double)u0[b]);
        vx += (T)gam * vy;
        vx += (T)(srate * (j - g.ny / 2.0));
        c0[o] = vx;
        c1[o] = vy;
        c2[o] = (T)(beta * (double)u2[a] + s.alpha * (double)u2[b]);
        const double p1 = 0.5 * ((1 - gam) * at(xp, yp) + (1 + gam) * at(xm, yp));
        const double m1 = 0.5 * ((1 - gam) * at(xm, ym) + (1 + gam) * at(xp, ym));
        acc[0] += (p1 - m1) * (1.0 / (2.0 * g.dx));
    }
    block_sumK<1>(acc);
    if (threadIdx.x == 0) partial[blockIdx.x] = acc[0];
}

// u += U2u_oblique(up - min(phi_sum, 1) ucp)  (Make_f_particle_dt_nonsole,
// Transform_obl_u cartesian2oblique, Add_f_particle; fft_wrapper.h:486-512).
// Cells as in r_le_obl2cart.  f is zero where neither of its two cells has a
// particle (phi_sum = 0, and then up = 0): those cells of u are left alone.  The
// cells also add up Calc_Reynolds_shear_stress of the Cartesian velocity
// (fluid_solver.h:165-183), each once: i0 runs over a row's cells as i does.
template <typename T>
__global__ void r_le_force_add(Grid g, const T *__restrict__ up0, const T *__restrict__ up1,
                               const T *__restrict__ up2, const T *__restrict__ phis, const T *__restrict__ c0,
                               const T *__restrict__ c1, const T *__restrict__ c2, T *__restrict__ u0,
                               T *__restrict__ u1, T *__restrict__ u2, double gam, const LEDev *__restrict__ le,
                               double *__restrict__ partial) {
    const unsigned rowlen = 2 * (unsigned)g.hnzp, n = (unsigned)g.nx * g.ny * g.nz;
    const int      lz = 31 - __clz(g.nz), ly = 31 - __clz(g.ny);
    const double   srate  = le->srate_eff;
    double         acc[1] = {0.0};
    for (unsigned t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        const unsigned k = t & (g.nz - 1), row = t >> lz;
        const int      i = (int)(row >> ly), j = (int)(row & (g.ny - 1));
        const ShiftRow s  = shift_row(j, g.ny, gam, true);
        const int      i0 = (i + s.io) & (g.nx - 1), i1 = (i0 + s.sign) & (g.nx - 1);
        const unsigned a = ((unsigned)i0 * g.ny + j) * rowlen + k, b = ((unsigned)i1 * g.ny + j) * rowlen + k;
        const unsigned o = row * rowlen + k;
        const T pa = phis[a], pb = phis[b];
        const T x = c0[a], y = c1[a], z = c2[a], xb = c0[b], yb = c1[b], zb = c2[b];
        acc[0] += ((double)x - srate * ((j - g.ny / 2) * g.dx)) * (double)y;
        if (pa == (T)0 && pb == (T)0) continue;
        const double beta = 1.0 - s.alpha;
        const T      qa = pa < (T)1 ? pa : (T)1, qb = pb < (T)1 ? pb : (T)1;
        const double fx = beta * (double)(up0[a] - qa * x) + s.alpha * (double)(up0[b] - qb * xb);
        const double fy = beta * (double)(up1[a] - qa * y) + s.alpha * (double)(up1[b] - qb * yb);
        const double fz = beta * (double)(up2[a] - qa * z) + s.alpha * (double)(up2[b] - qb * zb);
        const T      fyT = (T)fy;
        u0[o] += (T)fx - (T)gam * fyT;
        u1[o] += fyT;
        u2[o] += (T)fz;
    }
    block_sumK<1>(acc);
    if (threadIdx.x == 0) partial[blockIdx.x] = acc[0];
}

// Reset_U_OBL (fluid_solver.h:312-337): remap when |gamma| reaches XYaspect.
template <typename T>
__global__ void r_le_reset(Grid g, const T *__restrict__ u0, const T *__restrict__ u1, const T *__restrict__ u2,
                           T *__restrict__ o0, T *__restrict__ o1, T *__restrict__ o2, double delta) {
    const size_t rowlen = 2 * (size_t)g.hnzp;
    const size_t n      = (size_t)g.nx * g.ny * g.nz;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < n; t += (size_t)gridDim.x * blockDim.x) {
        const int k  = (int)(t % g.nz);
        const int j  = (int)((t / g.nz) % g.ny);
        const int i  = (int)(t / ((size_t)g.nz * g.ny));
        double    sg = (double)(j - g.ny / 2);
        if (sg != 0.0) sg = sg / fabs(sg);
        const double io  = (double)(int)(sg * (j - g.ny / 2)) * sg;
        const int    iob = (int)fmod(i + delta * io + 4.0 * g.nx, (double)g.nx);
        const size_t a   = ((size_t)i * g.ny + j) * rowlen + k;
        const size_t o   = ((size_t)iob * g.ny + j) * rowlen + k;
        o0[o]            = u0[a] + (T)delta * u1[a];
        o1[o]            = u1[a];
        o2[o]            = u2[a];
    }
}

// The sums over CTA partials and over particles are one block's: each thread
// adds every kLeFinishThreads-th term, a tree over the block follows, so the
// order is fixed.  One thread walking the list waits for every load in turn
// (2368 partials: 86 us a launch on B200, 128^3 and 64^3 alike; a block of
// 1024 takes 4 us).
constexpr int kLeFinishThreads = 1024;

// Shear_rate_eff = shear_rate + ivol * sum (set once per step)
__global__ void __launch_bounds__(kLeFinishThreads)
    k_le_shear_rate(LEDev *le, const double *__restrict__ partial, int nparts, double ivol, double shear_rate) {
    double s[1] = {0.0};
    for (int i = threadIdx.x; i < nparts; i += kLeFinishThreads) s[0] += partial[i];
    block_sumK<1>(s);
    if (threadIdx.x != 0) return;
    le->correction = s[0] * ivol;
    le->srate_eff  = shear_rate + le->correction;
}

// ---------------------------------------------------------------------------
// Stencil with the Lees-Edwards image (Relative_coord_check_stepover_Y,
// make_phi.h:229-265; Distance0_OBL, interaction.h:50-72).
// ---------------------------------------------------------------------------
struct StencilPointLE {
    size_t idx;
    double r[3];
    double dist;   // Distance_OBL(grid point, particle)
    double rnorm;  // |r| (used by Calc_f_hydro_correct_precision_OBL)
    int    sign;   // y stepover (+-1, 0)
    int    rm1;    // grid y index
};

__device__ __forceinline__ void stencil_point_le(const Grid &g, const Phys &ph, const double xp[3], int cell_packed,
                                                 double gam, StencilPointLE &s) {
    const int    c[3] = {(int)(int8_t)(cell_packed & 0xff), (int)(int8_t)((cell_packed >> 8) & 0xff),
                         (int)(int8_t)((cell_packed >> 16) & 0xff)};
    const double idx  = 1.0 / g.dx;
    int          xi[3];
    double       res[3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
        const double dmy = xp[d] * idx;
        xi[d]            = (int)dmy;
        res[d]           = (dmy - (double)xi[d]) * g.dx;
    }
    const int yy = xi[1] + c[1];
    const int r1 = (yy + g.ny) % g.ny;
    int       sg = yy - r1;
    if (sg != 0) sg = sg / abs(sg);
    const double fx = fmod((double)xi[0] - sg * gam * g.ny + res[0] / g.dx + c[0] + 4 * g.nx, (double)g.nx);
    const int    r0 = (int)fx;
    const double xr = fx - r0;
    const int    r2 = (xi[2] + c[2] + g.nz) % g.nz;
    s.r[0]          = c[0] * g.dx - xr * g.dx;
    s.r[1]          = c[1] * g.dx - res[1];
    s.r[2]          = c[2] * g.dx - res[2];
    s.rnorm         = sqrt(s.r[0] * s.r[0] + s.r[1] * s.r[1] + s.r[2] * s.r[2]);
    s.sign          = sg;
    s.rm1           = r1;
    // Distance0_OBL(x_mesh, x_p)
    const double xm[3] = {r0 * g.dx, r1 * g.dx, r2 * g.dx};
    double       y12   = xp[1] - xm[1];
    double       sy    = y12;
    y12 -= (double)nint_d(y12 / ph.L[1]) * ph.L[1];
    sy -= y12;
    int sd = (int)sy;
    if (sd != 0) sd = sd / abs(sd);
    double x12 = xp[0] - (xm[0] + (double)sd * gam * ph.L[1]);
    x12 -= (double)nint_d(x12 / ph.L[0]) * ph.L[0];
    double z12 = xp[2] - xm[2];
    z12 -= (double)nint_d(z12 / ph.L[2]) * ph.L[2];
    double d2 = 0.0;
    d2 += y12 * y12;
    d2 += x12 * x12;
    d2 += z12 * z12;
    s.dist = sqrt(d2);
    s.idx  = ((size_t)r0 * g.ny + r1) * (2 * (size_t)g.hnzp) + r2;
}

// Make_phi_particle_sum_OBL (make_phi.cxx:262-311)
template <typename T>
__global__ void s_le_phi_scatter(Grid g, Phys ph, const double *__restrict__ x, const int *__restrict__ cells,
                                 int ncells, double gam, T *__restrict__ phi_sum, unsigned int *err) {
    const int p = blockIdx.y;
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= ph.np || m >= ncells) return;
    const double xp[3] = {x[3 * p], x[3 * p + 1], x[3 * p + 2]};
    if (!particle_in_box(ph, xp)) {
        if (m == 0) atomicOr(err, (unsigned)SPM_DEVERR_PARTICLE_OUT_OF_BOX);
        return;
    }
    StencilPointLE s;
    stencil_point_le(g, ph, xp, cells[m], gam, s);
    const double v = phi_prof(s.dist, ph.radius, ph.hxi, g.dx);
    if (v != 0.0) atomicAdd(&phi_sum[s.idx], (T)v);
}

// Make_u_particle_sum_OBL (make_phi.cxx:356-402)
template <typename T>
__global__ void s_le_up_scatter(Grid g, Phys ph, const double *__restrict__ x, const double *__restrict__ v,
                                const double *__restrict__ w, const int *__restrict__ cells, int ncells, double gam,
                                const LEDev *__restrict__ le, const T *__restrict__ phi_sum, T *__restrict__ up0,
                                T *__restrict__ up1, T *__restrict__ up2) {
    const int p = blockIdx.y;
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= ph.np || m >= ncells) return;
    const double xp[3] = {x[3 * p], x[3 * p + 1], x[3 * p + 2]};
    if (!particle_in_box(ph, xp)) return;
    StencilPointLE s;
    stencil_point_le(g, ph, xp, cells[m], gam, s);
    double wgt = phi_prof(s.dist, ph.radius, ph.hxi, g.dx);
    if (wgt == 0.0) return;
    const double ps = (double)phi_sum[s.idx];
    wgt /= (ps > 1.0 ? ps : 1.0);
    double vs[3] = {v[3 * p] - s.sign * le->srate_eff * ph.L[1], v[3 * p + 1], v[3 * p + 2]};
    if (ph.rotation) {
        const double *o = w + 3 * p;
        vs[0] += o[1] * s.r[2] - o[2] * s.r[1];
        vs[1] += o[2] * s.r[0] - o[0] * s.r[2];
        vs[2] += o[0] * s.r[1] - o[1] * s.r[0];
    }
    atomicAdd(&up0[s.idx], (T)(vs[0] * wgt));
    atomicAdd(&up1[s.idx], (T)(vs[1] * wgt));
    atomicAdd(&up2[s.idx], (T)(vs[2] * wgt));
}

// Calc_f_hydro_correct_precision_OBL (md_force.cxx:508-745): force and torque
// of each particle, and per-particle partial sums of the Hydro_force and
// Hydro_force_new fields' totals (all that Mean_shear_stress reads of them).
// ppart[p] = {A, Y, force0, volume, new_p, mdf0/volume * Y, Yy, Yz} with
// Y = sum w dry, Yy = sum w dry r_y, Yz = sum w dry r_z over the particle's
// stencil (dry the cell's y with its image).  Rigid beads (rigid != 0) leave
// the spheres' extra term out of new_p: r_le_stress_new adds the bodies' one
// from Yy and Yz once their forces are summed.
constexpr int kLePart = 8;
struct LeRhoP {
    double v[4];  // RHO_particle of each species
};
template <typename T>
__global__ void s_le_hydro_force(Grid g, Phys ph, const double *__restrict__ x, const double *__restrict__ v,
                                 const double *__restrict__ w, const double *__restrict__ mdf,
                                 const int *__restrict__ cells, int ncells, double gam, const LEDev *__restrict__ le,
                                 LeRhoP rho_s, const T *__restrict__ phi_sum, const T *__restrict__ c0,
                                 const T *__restrict__ c1, const T *__restrict__ c2, double *__restrict__ f_hydro,
                                 double *__restrict__ torque_hydro, double *__restrict__ ppart, int rigid) {
    const int p = blockIdx.x;
    if (p >= ph.np) return;
    const double xp[3] = {x[3 * p], x[3 * p + 1], x[3 * p + 2]};
    const double vp[3] = {v[3 * p], v[3 * p + 1], v[3 * p + 2]};
    const double op[3] = {w[3 * p], w[3 * p + 1], w[3 * p + 2]};
    const double srate = le->srate_eff;
    const double rho_p = rho_s.v[spec_of(ph, p)];
    // force 3, torque 3, volume, itrace, A, then Y, Yy, Yz
    double acc[12] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
    for (int m = threadIdx.x; m < ncells; m += blockDim.x) {
        StencilPointLE s;
        stencil_point_le(g, ph, xp, cells[m], gam, s);
        double wgt = phi_prof(s.rnorm, ph.radius, ph.hxi, g.dx);
        if (wgt == 0.0) continue;
        const double ps = (double)phi_sum[s.idx];
        wgt /= (ps > 1.0 ? ps : 1.0);
        double vs[3] = {vp[0] - s.sign * srate * ph.L[1], vp[1], vp[2]};
        if (ph.rotation) {
            vs[0] += op[1] * s.r[2] - op[2] * s.r[1];
            vs[1] += op[2] * s.r[0] - op[0] * s.r[2];
            vs[2] += op[0] * s.r[1] - op[1] * s.r[0];
        }
        const double fp0 = (vs[0] - (double)c0[s.idx]) * wgt;
        const double fp1 = (vs[1] - (double)c1[s.idx]) * wgt;
        const double fp2 = (vs[2] - (double)c2[s.idx]) * wgt;
        const double dry = s.rm1 + s.sign * ph.L[1], yw = dry * wgt;
        acc[0] += fp0;
        acc[1] += fp1;
        acc[2] += fp2;
        acc[3] += s.r[1] * fp2 - s.r[2] * fp1;
        acc[4] += s.r[2] * fp0 - s.r[0] * fp2;
        acc[5] += s.r[0] * fp1 - s.r[1] * fp0;
        acc[6] += wgt;
        acc[7] += wgt * s.rnorm * s.rnorm;
        acc[8] += fp0 * dry * rho_p;
        acc[9] += yw;
        acc[10] += yw * s.r[1];
        acc[11] += yw * s.r[2];
    }
    block_sumK<12>(acc);
    if (threadIdx.x == 0) {
        const double volume = acc[6], itrace = acc[7] * (2.0 / 3.0);
        // sum over the cells of (sv + sw) dry w, sw = -rho (t_y r_z - t_z r_y) / itrace,
        // from the sums Y, Yy, Yz: no second pass over the stencil (60 -> 33 us
        // at 128^3 with 400 colloids on B200)
        const double sv    = -ph.rho * acc[0] / volume;
        const double extra = sv * acc[9] - ph.rho * (acc[4] * acc[11] - acc[5] * acc[10]) / itrace;
        const double dmy   = -ph.dx3 * ph.rho / ph.dt;
        for (int d = 0; d < 3; d++) f_hydro[3 * p + d] = dmy * acc[d];
        if (ph.rotation)
            for (int d = 0; d < 3; d++) torque_hydro[3 * p + d] = dmy * acc[3 + d];
        double *pp = ppart + (size_t)kLePart * p;
        pp[0]      = acc[8];
        pp[1]      = acc[9];
        pp[2]      = acc[0];
        pp[3]      = volume;
        pp[4]      = rigid ? acc[8] : acc[8] + extra;
        pp[5]      = mdf[3 * p] / volume * acc[9];
        pp[6]      = acc[10];
        pp[7]      = acc[11];
    }
}

// Totals of the hydrodynamic stress fields and the LJ stress
// (Calc_hydro_stress, fluid_solver.h:253-279; Force_OBL, particle_solver.h:113-128).
// Ends the step too: the Reynolds partials of r_le_force_add, the strain, the
// time and the step counter.
__global__ void __launch_bounds__(kLeFinishThreads)
    k_le_step_finish(LEDev *le, const double *__restrict__ ppart, const double *__restrict__ lj_stress, int np,
                     const double *__restrict__ partial, int nparts, double ivol, double ivolume_lj, double dt,
                     double rho, double time, RunWords *rw) {
    double t[8] = {0, 0, 0, 0, 0, 0, 0, 0};  // A, Y, force, volume, new, mdf, LJ, Reynolds
    for (int p = threadIdx.x; p < np; p += kLeFinishThreads) {
        const double *pp = ppart + (size_t)kLePart * p;
#pragma unroll
        for (int k = 0; k < 6; k++) t[k] += pp[k];
        t[6] += lj_stress[p];
    }
    for (int i = threadIdx.x; i < nparts; i += kLeFinishThreads) t[7] += partial[i];
    block_sumK<8>(t);
    if (threadIdx.x != 0) return;
    if (np > 0) {
        const double sum_volume = t[3] / rho;
        const double hf_old     = t[0] - t[5] - (t[2] / sum_volume) * t[1];
        le->hydro_old           = -hf_old * ivol / dt;
        le->hydro_new           = -t[4] * ivol / dt;
        le->lj                  = t[6] * ivolume_lj;
    }
    le->reynolds = -ivol * rho * t[7];
    le->strain += le->srate_eff * dt;
    le->time = time;
    rw->ts += 1;
}

// The position update with the PBC_OBL wrap (particle_solver.cxx:283-334,
// periodic_boundary.h:26-45): crossing the y boundary shifts x by the
// oblique image and v_x by -+ Shear_rate_eff * LY.  Obstacles stay where
// they are (the wrap sits inside the non-obstacle branch there).
__global__ void p_position_le(Phys ph, PState s, const int *__restrict__ ts_dev, double gam,
                              const LEDev *__restrict__ le) {
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= ph.np || ph.janus_prop == 3) return;
    position_one(ph, s, n, *ts_dev == 0, 0);
    const double dvx = pbc_obl(ph, s.x + 3 * n, gam, le->srate_eff);
    s.v[3 * n] += dvx;
    s.v_old[3 * n] += dvx;
}

// Show_parameter zeroes v_x and omega_z of a sheared run after the initial
// projection (init_particle.cxx:767-781).
__global__ void p_le_zero_vx(Phys ph, PState s) {
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= ph.np) return;
    s.v[3 * n] = s.v_old[3 * n] = 0.0;
    s.omega[3 * n + 2] = s.omega_old[3 * n + 2] = 0.0;
}

inline void le_init(LEState &le, const Grid &g, const Phys &, const spm_params &p) {
    le.enabled    = p.equation == SPM_EQ_LEES_EDWARDS;
    le.shear_rate = p.shear_rate;
    le.xy_aspect  = (double)g.nx / (double)g.ny;
}
inline void le_reset(LEState &le) {
    le.degree_oblique = 0.0;
    if (le.dev) cudaMemset(le.dev, 0, sizeof(LEDev));
}

}  // namespace spm
