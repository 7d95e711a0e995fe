// The X pass of the step's transforms fused with the k-space stage beside it.
//
// A z column tile (W kz values of one ky line, all N = NX points) is a whole
// set of x lines, so the thread that ends a forward X transform holds modes
// (kx, ky, kz) of every field of the tile, and the same modes are its input to
// an inverse X transform: the four-step split n = g + N1 m reads and leaves
// index set {g + N1 m}.  So the pointwise stages between a forward and an
// inverse X pass run in registers:
//   kXZeta  zeta -> u_hat -> inverse X of u            (Zeta_k2u_k)
//   kXNs    forward X of the 5 advection products -> slaved-Euler update of
//           zeta [-> u_hat of the new zeta -> inverse X of u]
//           (U2advection_k's k part, NS_solver_slavedEuler)
//   kXProj  forward X of the rigidity force f -> zeta += zeta(i k x P f)
//           (Solenoidal_u closed in k space)
//   kXSole  forward X of three fields -> 2/3 truncation and P -> inverse X
//           (Solenoidal_u) [, zeta and uk_dc of the result: U_k2zeta_k]
// The update is linear in the products, so a thread adds each product's share
// to two accumulators per retained mode as its transform ends, and never holds
// more than one of the five; the projection keeps the three components of f.
//
// What bounds it and why this form: the stages are HBM traffic.  Unfused, the
// update at 256^3 wrote and read back five product fields and three velocity
// fields of the retained box (FP32: 761 MB in four launches against 400 MB
// here).  W is 128 bytes of kz per line: two CTAs of 256 (FP32) or 128 (FP64)
// threads fit an SM with a three-tile TMA ring each.
#pragma once

#include "spm_fft_plan.cuh"
#include "spm_kernels.cuh"

namespace spm {

template <int I>
struct XInt {
    static constexpr int value = I;
};
enum XOp { kXZeta = 0, kXNs = 1, kXProj = 2, kXSole = 3 };

// Arguments of the fused passes.  Fields of run r start r * run_stride complex
// values after run 0's; slots (fields) of a run lie slot_stride apart.
template <typename T>
struct XArgs {
    Grid         g;
    cplx<T>     *z0, *z1;    // zeta
    cplx<T>     *zl0, *zl1;  // its compensation words, or null
    cplx<T>     *u;          // first slot of the transformed fields and of the velocity written
    RunWords    *rw;
    size_t       run_stride, slot_stride;
    int          ct_used, n_used, ntiles;  // set by x_fused
    int          ts_inc;                    // kXProj: added to the step counter
    double       nu, dt;
    const cplx<T> *tw;
};

template <int N>
struct XModes {
    static constexpr int N1 = Split<N>::N1, N2 = Split<N>::N2, R = N2 / N1;
    static constexpr int TRN = (N + 2) / 3;  // Grid::trn of an axis of N points
    // whether index n = g + N1 m can be a retained mode for some g < N1
    static constexpr bool maybe(int m) { return N1 * m < TRN || N1 * m + N1 - 1 > N - TRN; }
    // whether it is one for every g < N1
    static constexpr bool always(int m) { return N1 * m + N1 - 1 < TRN || N1 * m > N - TRN; }
    static __host__ __device__ __forceinline__ bool retained(int g, int m) {
        const int k = signed_mode(g + N1 * m, N);
        return always(m) || (k < TRN && -k < TRN);
    }
    // The index whose zeta the thread of n = g + N1 m loads, without a branch: n
    // itself, or where n is outside the box its own first mode (always inside: N1
    // <= TRN).  Nobody but this thread writes that word; one word for all such
    // threads would be read while the thread that owns it writes it.
    static __host__ __device__ __forceinline__ int zeta_index(int g, int m) { return retained(g, m) ? g + N1 * m : g; }
};
// Element offset of column kz of ky line o inside a field.  A tile reaches past
// the retained columns; those beyond the row share its last column, which is
// outside the box (hnz - 1 = NZ/2 >= trn), so that no thread writes it.
__host__ __device__ __forceinline__ unsigned x_line(const Grid &g, int o, int kz) {
    return (unsigned)o * g.hnzp + (kz < g.hnzp ? kz : g.hnzp - 1);
}

// Twiddled step 1 of the four-step transform on v[m] = x[g + N1 m], its
// results to rows g + N1 k1 of the exchange tile B.  stw[N1 k1 + g] =
// e^{-2 pi i g k1 / N}: constant offsets from a thread's own entry.
template <typename T, int N, int W, int DIR>
__device__ __forceinline__ void x_step1(cplx<T> (&v)[Split<N>::N2], int g, int c, cplx<T> *B, const cplx<T> *stw) {
    constexpr int N1 = Split<N>::N1, N2 = Split<N>::N2;
    dft_reg<T, N2, DIR>(v);
#pragma unroll
    for (int k1 = 1; k1 < N2; k1++) {
        cplx<T> w = stw[N1 * k1 + g];
        if (DIR > 0) w.im = -w.im;
        v[k1] = cmul(v[k1], w);
    }
#pragma unroll
    for (int k1 = 0; k1 < N2; k1++) B[(g + N1 * k1) * W + c] = v[k1];
}
// Step 2: v[i + R k2] = X[(g + N1 i) + N2 k2], i.e. v[m] = X[g + N1 m].
template <typename T, int N, int W, int DIR>
__device__ __forceinline__ void x_step2(cplx<T> (&v)[Split<N>::N2], int g, int c, const cplx<T> *B) {
    constexpr int N1 = Split<N>::N1, R = Split<N>::N2 / N1;
#pragma unroll
    for (int i = 0; i < R; i++) {
        cplx<T> u[N1];
#pragma unroll
        for (int n1 = 0; n1 < N1; n1++) u[n1] = B[(n1 + N1 * (g + N1 * i)) * W + c];
        dft_reg<T, N1, DIR>(u);
#pragma unroll
        for (int k2 = 0; k2 < N1; k2++) v[i + R * k2] = u[k2];
    }
}

// Field F's share of the reduced advection term, acc0 += a P and acc1 += b P
// (U2advection_k's curl of the products u2u3, u3u1, u1u2, u2^2-u3^2,
// u3^2-u1^2 and Omega_k2zeta_k's component choice).  K0: the mode may have
// KX = 0.
template <typename T, int F, bool K0>
__device__ __forceinline__ void x_ns_coef(T k1, T k2, T k3, bool kx0, bool ky0, T &a, T &b) {
    const T o1 = F == 0 ? -(k1 * k2) : F == 1 ? -((k1 - k3) * (k1 + k3)) : F == 2 ? k2 * k3 : F == 3 ? (T)0 : -(k3 * k1);
    const T o2 = F == 0 ? k3 * k1 : F == 1 ? -(k2 * k3) : F == 2 ? -((k2 - k1) * (k2 + k1)) : k1 * k2;
    a = o1;
    b = o2;
    if constexpr (K0) {
        const T o0 = F == 0 ? -((k3 - k2) * (k3 + k2)) : F == 1 ? k1 * k2 : F == 2 ? -(k3 * k1) : F == 3 ? -(k2 * k3) : (T)0;
        if (kx0) {
            a = ky0 ? o0 : o2;
            b = ky0 ? o1 : o0;
        }
    }
}
// The increment zeta(i k x P f) of one mode, P f = f - k (k . f) / k^2
// (Solenoidal_uk; i_cross and Omega_k2zeta_k's component choice).  k x P f =
// k x f, but the rounding of the product is then relative to f with its
// longitudinal part: measured over FP32 runs, 20% more error in the forces.
template <typename T, bool K0>
__device__ __forceinline__ void x_proj_increment(T kx, T ky, T kz, T ik2, bool kx0, bool ky0, cplx<T> f0, cplx<T> f1,
                                                 cplx<T> f2, cplx<T> &d0, cplx<T> &d1) {
    const T dr = ik2 * (f0.re * kx + f1.re * ky + f2.re * kz);
    const T di = ik2 * (f0.im * kx + f1.im * ky + f2.im * kz);
    cplx<T> f[3] = {{f0.re - dr * kx, f0.im - di * kx}, {f1.re - dr * ky, f1.im - di * ky}, {f2.re - dr * kz, f2.im - di * kz}};
    cplx<T> om[3];
    i_cross<T>(kx, ky, kz, f, om);
    d0 = om[1];
    d1 = om[2];
    if constexpr (K0) {
        if (kx0) {
            d0 = ky0 ? om[0] : om[2];
            d1 = ky0 ? om[1] : om[0];
        }
    }
}

// Component D of u_hat = i (k / k^2) x omega(zeta) (Zeta_k2u_k).  The factor
// 1/k^2 goes to the wave vector, as the separate kernel has it: dividing zeta
// instead rounds omega_x three times more, 11 to 15% more error in the forces
// of FP32 runs.
template <typename T, int D, bool K0>
__device__ __forceinline__ cplx<T> x_velocity(T kx, T ky, T kz, T ik2, T inv_kx, bool kx0, bool ky0, T kz_ky,
                                              const cplx<T> &z0, const cplx<T> &z1) {
    cplx<T> om[3];
    om[0] = cplx<T>{-inv_kx * (ky * z0.re + kz * z1.re), -inv_kx * (ky * z0.im + kz * z1.im)};
    om[1] = z0;
    om[2] = z1;
    if constexpr (K0) {
        if (kx0) {
            om[0] = ky0 ? z0 : z1;
            om[1] = ky0 ? z1 : cplx<T>{-kz_ky * z0.re, -kz_ky * z0.im};
            om[2] = ky0 ? cplx<T>{0, 0} : z0;
        }
    }
    kx *= ik2, ky *= ik2, kz *= ik2;
    if (D == 0) return cplx<T>{-(ky * om[2].im - kz * om[1].im), ky * om[2].re - kz * om[1].re};
    if (D == 1) return cplx<T>{-(kz * om[0].im - kx * om[2].im), kz * om[0].re - kx * om[2].re};
    return cplx<T>{-(kx * om[1].im - ky * om[0].im), kx * om[1].re - ky * om[0].re};
}

// 1 / k^2 (0 at k = 0) from the approximate FP32 reciprocal (1 ulp, x_fused
// checks that k^2 is in its range): a Newton step in FP64 leaves an error below
// 2^-44, enough for FP32; FP64 takes a second, whose last operation rounds once
// (the error before it is below 2^-88), as a division does.
template <typename T>
__device__ __forceinline__ double x_reciprocal(double k2) {
    float r;
    asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"((float)k2));
    double y = (double)r;
    y        = fma(y, fma(-k2, y, 1.0), y);
    if (sizeof(T) == 8) y = fma(y, fma(-k2, y, 1.0), y);
    return k2 > 0.0 ? y : 0.0;
}
__device__ __forceinline__ void prefetch_l2(const void *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

constexpr int kXChunk = 4;  // modes whose zeta a thread loads together
constexpr int kXRing = 3;  // tiles of the TMA ring; the last field's tile is the exchange tile of the inverse
template <typename T, int N, int W, int OP>
constexpr size_t x_fuse_smem() {
    return (size_t)(OP == kXZeta ? 1 : kXRing) * N * W * sizeof(cplx<T>) + N * (sizeof(cplx<T>) + 2 * sizeof(double) + 2 * sizeof(T));
}

template <typename T, int N, int W, int OP, bool INV>
__global__ void __launch_bounds__(W *Split<N>::N1, N >= 256 ? 2 : 1)
    x_fused_kernel(const __grid_constant__ CUtensorMap lmap, const __grid_constant__ XArgs<T> A, unsigned int *err,
                   unsigned long long wait_ns, int skip_loads) {
    using M                       = XModes<N>;
    constexpr int      N1 = M::N1, N2 = M::N2;
    constexpr bool     kThree     = OP == kXProj || OP == kXSole;  // three fields, all kept
    constexpr int      NF         = OP == kXNs ? 5 : kThree ? 3 : 0;
    constexpr int      ND         = NF > 0 ? NF : 1;  // divisor of the load sequence
    constexpr int      S          = OP == kXZeta ? 1 : kXRing;
    constexpr unsigned tile_bytes = (unsigned)(N * W * sizeof(cplx<T>));
    // two CTAs of 256 threads leave a thread 128 registers (FP32 at 256 points): the
    // values that the branch-free loads of zeta keep alive then spill (112 bytes in
    // kXNs, none with a predicate per mode; ten steps 10132 -> 10008 us).  With 255
    // registers the branch-free form is faster (512 points FP32: 7731 against 7597 us)
    constexpr bool kFewRegs = N >= 256 && W * N1 >= 256;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    cplx<T> *buf = reinterpret_cast<cplx<T> *>(smem_raw);
    double  *skx = reinterpret_cast<double *>(buf + (size_t)S * N * W);  // kx of index n
    double  *sex = skx + N;                                              // e^{-nu dt kx^2} - 1
    cplx<T> *stw = reinterpret_cast<cplx<T> *>(sex + N);                 // step-1 twiddles (x_step1)
    T       *skt = reinterpret_cast<T *>(stw + N);                       // kx in T
    T       *sik = skt + N;                                              // 1 / kx
    __shared__ __align__(8) uint64_t full[S];
    const Grid &gr  = A.g;
    const int   tid = threadIdx.x;
    const int   c   = tid % W;
    const int   g   = tid / W;
    for (int j = tid; j < N; j += W * N1) {
        stw[j]         = A.tw[((j % N1) * (j / N1)) & (N - 1)];
        const double k = gr.wave[0] * (double)signed_mode(j, N);
        skx[j]         = k;
        if (OP == kXNs) sex[j] = expm1(-A.nu * A.dt * (k * k));
        skt[j]         = (T)k;
        sik[j]         = j ? (T)(1.0 / k) : (T)0;
    }
    if (NF > 0 && tid == 0) {
        for (int b = 0; b < S; b++) mbar_init(&full[b], 1);
        fence_mbar_init();
    }
    __syncthreads();
    // loads in order: number q is field q % NF of this CTA's (q / NF)-th tile
    const int ntl    = (int)blockIdx.x < A.ntiles ? (A.ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    const int nloads = ntl * NF;
    auto      decode = [&](int t, int &ct, int &o, int &run) {
        ct             = t % A.ct_used;
        const int rest = t / A.ct_used;
        o              = outer_line(rest % A.n_used, gr.ny, gr.trn[1]);
        run            = rest / A.n_used;
    };
    int  issued = 0;  // thread 0
    auto load   = [&](int q) {
        if (skip_loads) return;
        issued = q + 1;
        int ct, o, run;
        decode((int)blockIdx.x + (q / ND) * (int)gridDim.x, ct, o, run);
        mbar_expect_tx(&full[q % S], tile_bytes);
        cplx<T> *dst = buf + (size_t)(q % S) * N * W;
        tma_load_5d(dst, &lmap, 2 * ct * W, o, 0, run, q % ND, &full[q % S]);
        if constexpr (N > 256)  // a box has at most 256 lines
            tma_load_5d(dst + (size_t)N / 2 * W, &lmap, 2 * ct * W, o, N / 2, run, q % ND, &full[q % S]);
    };
    if (NF > 0 && tid == 0)
        for (int q = 0; q < S - 1 && q < nloads; q++) load(q);
    bool stopped = false;
    int  q       = 0;  // next load to consume
    for (int t = blockIdx.x; t < A.ntiles; t += gridDim.x) {
        int ct, o, run;
        decode(t, ct, o, run);
        const int    kz   = ct * W + c;
        const bool   col  = kz < gr.trn[2];
        const size_t ro   = (size_t)run * A.run_stride;
        // element offsets inside a field fit 32 bits (x_fused checks it)
        const unsigned line = x_line(gr, o, kz);  // + n * nst for index n
        const unsigned nst  = (unsigned)gr.ny * gr.hnzp;
        cplx<T>  *pz0 = A.z0 + ro, *pz1 = A.z1 + ro;
        const bool comp = sizeof(T) == 4 && A.zl0 != nullptr;
        cplx<T>  *pl0 = comp ? A.zl0 + ro : nullptr, *pl1 = comp ? A.zl1 + ro : nullptr;
        const double dky  = gr.wave[1] * (double)signed_mode(o, gr.ny), dkz = gr.wave[2] * (double)kz;
        const T      kyt = (T)dky, kzt = (T)dkz;
        const bool   kx0 = g == 0, ky0 = o == 0;  // at m = 0 only
        const bool   dc  = kx0 && ky0 && kz == 0;
        auto         keep = [&](int m) { return col && M::retained(g, m); };
        // kXNs: the two accumulators; kXProj, kXSole: the three transformed
        // components; then zeta of the retained modes in a0, a1 (kXSole: P f)
        cplx<T> a0[N2], a1[N2], a2[kThree ? N2 : 1];
        if constexpr (NF > 0) {
            // zeta is needed once the fields are transformed: start it towards L2
#pragma unroll
            for (int m = 0; m < N2; m++) {
                a0[m] = a1[m] = cplx<T>{0, 0};
                if (OP == kXSole || !M::maybe(m) || !keep(m)) continue;
                const unsigned idx = (unsigned)(g + N1 * m) * nst + line;
                prefetch_l2(pz0 + idx);
                prefetch_l2(pz1 + idx);
                if (comp) {
                    prefetch_l2(pl0 + idx);
                    prefetch_l2(pl1 + idx);
                }
            }
            // transforms the tile of load q; false: its wait ran out
            cplx<T> v[N2];
            auto    field = [&]() -> bool {
                cplx<T>   *B = buf + (size_t)(q % S) * N * W;
                const bool w = mbar_wait(&full[q % S], (unsigned)((q / S) & 1), err, wait_ns);
#pragma unroll
                for (int m = 0; m < N2; m++) v[m] = B[(g + N1 * m) * W + c];
                x_step1<T, N, W, -1>(v, g, c, B, stw);
                // this thread's accesses to the previous tile's buffer come
                // before the load that refills it
                fence_proxy_async();
                if (!__syncthreads_and(w)) return false;
                if (tid == 0 && q + S - 1 < nloads) load(q + S - 1);
                x_step2<T, N, W, -1>(v, g, c, B);
                q++;
                return true;
            };
            if constexpr (OP == kXNs) {
#pragma unroll 1
                for (int f = 0; f < NF; f++) {
                    if (!field()) {
                        stopped = true;
                        break;
                    }
                    auto add = [&](auto F) {
#pragma unroll
                        for (int m = 0; m < N2; m++) {
                            if (!M::maybe(m)) continue;
                            const T kx = skt[g + N1 * m];
                            T       a, b;
                            if (m == 0)
                                x_ns_coef<T, F.value, true>(kx, kyt, kzt, kx0, ky0, a, b);
                            else
                                x_ns_coef<T, F.value, false>(kx, kyt, kzt, false, false, a, b);
                            a0[m].re += a * v[m].re;
                            a0[m].im += a * v[m].im;
                            a1[m].re += b * v[m].re;
                            a1[m].im += b * v[m].im;
                        }
                    };
                    switch (f) {
                        case 0: add(XInt<0>{}); break;
                        case 1: add(XInt<1>{}); break;
                        case 2: add(XInt<2>{}); break;
                        case 3: add(XInt<3>{}); break;
                        default: add(XInt<4>{}); break;
                    }
                }
            } else {
                auto take = [&](cplx<T>(&to)[N2], int f) {
                    if (stopped || !field()) {
                        stopped = true;
                        return;
                    }
                    // the k = 0 mode takes Re f_hat(0), not touched by the projection
                    if (OP == kXProj && dc) A.rw[run].uk_dc[f] += (double)v[0].re;
                    if (OP == kXSole && dc && A.z0) A.rw[run].uk_dc[f] = (double)v[0].re;
#pragma unroll
                    for (int m = 0; m < N2; m++) to[m] = v[m];
                };
                take(a0, 0);
                take(a1, 1);
                take(a2, 2);
            }
            if (stopped) break;
        }
        if constexpr (OP == kXSole) {
            const double dkyz2 = dky * dky + dkz * dkz;
#pragma unroll
            for (int m = 0; m < N2; m++) {
                if (!M::maybe(m)) continue;
                const double dkx = skx[g + N1 * m];
                const T      kx  = skt[g + N1 * m], ik2 = (T)x_reciprocal<T>(dkx * dkx + dkyz2);
                const T      dr = ik2 * (a0[m].re * kx + a1[m].re * kyt + a2[m].re * kzt);
                const T      di = ik2 * (a0[m].im * kx + a1[m].im * kyt + a2[m].im * kzt);
                const bool   k  = keep(m);
                a0[m] = k ? cplx<T>{a0[m].re - dr * kx, a0[m].im - di * kx} : cplx<T>{0, 0};
                a1[m] = k ? cplx<T>{a1[m].re - dr * kyt, a1[m].im - di * kyt} : cplx<T>{0, 0};
                a2[m] = k ? cplx<T>{a2[m].re - dr * kzt, a2[m].im - di * kzt} : cplx<T>{0, 0};
                if (!k || !A.z0) continue;
                const cplx<T> u[3] = {a0[m], a1[m], a2[m]};
                cplx<T>       om[3], z0, z1;
                i_cross<T>(kx, kyt, kzt, u, om);
                z0 = om[1], z1 = om[2];
                if (m == 0 && kx0) {
                    z0 = ky0 ? om[0] : om[2];
                    z1 = ky0 ? om[1] : om[0];
                }
                const unsigned idx = (unsigned)(g + N1 * m) * nst + line;
                pz0[idx] = z0;
                pz1[idx] = z1;
            }
        }
        // k-space stage: a0, a1 become zeta.  zeta of kXChunk modes at a time is
        // loaded without branches (XModes::zeta_index; kFewRegs: its own modes only),
        // so its loads are in flight together; what a mode outside the box loads is
        // dropped.
        // e^{x + y} - 1 = ex + ey + ex ey for x, y <= 0 has no cancellation, so a
        // mode costs no exponential of its own.
        const double dkyz2 = dky * dky + dkz * dkz;
        const double eyz   = OP == kXNs ? expm1(-A.nu * A.dt * dkyz2) : 0.0;
        const double inu   = 1.0 / A.nu;
#pragma unroll
        for (int mc = 0; OP != kXSole && mc < N2; mc += kXChunk) {
            cplx<T> z0[kXChunk], z1[kXChunk], l0[kXChunk], l1[kXChunk];
#pragma unroll
            for (int j = 0; j < kXChunk; j++) {
                const int m = mc + j;
                if (m >= N2 || !M::maybe(m)) continue;
                const unsigned idx = (unsigned)(kFewRegs ? g + N1 * m : M::zeta_index(g, m)) * nst + line;
                const bool     ld  = !kFewRegs || keep(m);
                if (kFewRegs) z0[j] = z1[j] = l0[j] = l1[j] = cplx<T>{0, 0};
                if (ld) z0[j] = pz0[idx], z1[j] = pz1[idx];
                if (OP != kXZeta && comp && ld) l0[j] = pl0[idx], l1[j] = pl1[idx];
            }
#pragma unroll
            for (int j = 0; j < kXChunk; j++) {
                const int m = mc + j;
                if (m >= N2 || !M::maybe(m)) continue;
                const double dkx   = skx[g + N1 * m];
                const double k2sum = dkx * dkx + dkyz2;
                const double ik2   = x_reciprocal<T>(k2sum);
                if constexpr (OP == kXNs || OP == kXProj) {
                    cplx<T> d0 = a0[m], d1 = a1[m];
                    if constexpr (OP == kXNs) {
                        // zeta += (e^{-nu dt k^2} - 1) (zeta - f / (nu k^2)); compensated: the
                        // increment is formed from (hi - c f) + lo and added by TwoSum
                        const double ex  = sex[g + N1 * m];
                        const T      dmy = (T)(ex + (eyz + ex * eyz));
                        const T      cc  = (T)(inu * ik2);
                        d0 = {z0[j].re - cc * d0.re, z0[j].im - cc * d0.im};
                        d1 = {z1[j].re - cc * d1.re, z1[j].im - cc * d1.im};
                        if (comp) d0 = cadd(d0, l0[j]), d1 = cadd(d1, l1[j]);
                        d0 = {dmy * d0.re, dmy * d0.im};
                        d1 = {dmy * d1.re, dmy * d1.im};
                    }
                    if constexpr (OP == kXProj) {
                        const T kx = skt[g + N1 * m];
                        if (m == 0)
                            x_proj_increment<T, true>(kx, kyt, kzt, (T)ik2, kx0, ky0, a0[m], a1[m], a2[m], d0, d1);
                        else
                            x_proj_increment<T, false>(kx, kyt, kzt, (T)ik2, false, false, a0[m], a1[m], a2[m], d0, d1);
                    }
                    if (comp) {
                        comp_add<T>(z0[j], l0[j], d0);
                        comp_add<T>(z1[j], l1[j], d1);
                    } else {
                        z0[j] = cadd(z0[j], d0);
                        z1[j] = cadd(z1[j], d1);
                    }
                    if (OP == kXProj && m == 0 && dc) {
                        z0[j] = z1[j] = l0[j] = l1[j] = cplx<T>{0, 0};
                        A.rw[run].ts += A.ts_inc;
                    }
                    if (keep(m)) {
                        const unsigned idx = (unsigned)(g + N1 * m) * nst + line;
                        pz0[idx] = z0[j];
                        pz1[idx] = z1[j];
                        if (comp) pl0[idx] = l0[j], pl1[idx] = l1[j];
                    }
                }
                if constexpr (INV) {
                    a0[m] = keep(m) ? z0[j] : cplx<T>{0, 0};
                    a1[m] = keep(m) ? z1[j] : cplx<T>{0, 0};
                }
            }
        }
        if constexpr (INV) {
            // exchange tile: the last field's buffer, which no load refills before
            // the next tile's first barrier
            cplx<T> *B = NF > 0 ? buf + (size_t)((q - 1) % S) * N * W : buf;
            if (OP == kXNs && dc) {  // FIX_CELLxyz, before Zeta_k2u_k reads uk_dc
                for (int d = 0; d < 3; d++)
                    if (A.rw[run].fix_mask & (1 << d)) A.rw[run].uk_dc[d] = 0.0;
            }
            const T kz_ky = ky0 ? (T)0 : (T)(dkz / dky);
#pragma unroll 1
            for (int d = 0; d < 3; d++) {
                cplx<T> v[N2];
                auto    vel = [&](auto D) {
#pragma unroll
                    for (int m = 0; m < N2; m++) {
                        v[m] = cplx<T>{0, 0};
                        if (!M::maybe(m)) continue;
                        if constexpr (OP == kXSole) {
                            v[m] = D.value == 0 ? a0[m] : D.value == 1 ? a1[m] : a2[kThree ? m : 0];
                            continue;
                        }
                        const T kx = skt[g + N1 * m], ikx = sik[g + N1 * m];
                        // formed again for each component: kept, its 12 values per thread spill
                        // (beyond the 64 to 80 bytes that FP64 spills as it is; ten steps at
                        // 256^3: FP64 15674 against 15280 us, FP32 10143 against 9929)
                        const T ik2 = (T)x_reciprocal<T>(skx[g + N1 * m] * skx[g + N1 * m] + dkyz2);
                        if (m == 0)
                            v[m] = x_velocity<T, D.value, true>(kx, kyt, kzt, ik2, ikx, kx0, ky0, kz_ky, a0[m], a1[m]);
                        else
                            v[m] = x_velocity<T, D.value, false>(kx, kyt, kzt, ik2, ikx, false, false, kz_ky, a0[m], a1[m]);
                    }
                };
                if (d == 0)
                    vel(XInt<0>{});
                else if (d == 1)
                    vel(XInt<1>{});
                else
                    vel(XInt<2>{});
                if (OP != kXSole && dc) v[0].re = (T)A.rw[run].uk_dc[d];
                __syncthreads();
                x_step1<T, N, W, +1>(v, g, c, B, stw);
                __syncthreads();
                x_step2<T, N, W, +1>(v, g, c, B);
                cplx<T> *out = A.u + (size_t)d * A.slot_stride + ro;
                if (col) {
#pragma unroll
                    for (int m = 0; m < N2; m++) out[(unsigned)(g + N1 * m) * nst + line] = v[m];
                }
            }
        }
    }
    if (NF > 0 && stopped && tid == 0)
        // loads issued and not consumed are still owed to this CTA's shared memory
        for (int j = q; j < issued; j++) mbar_wait(&full[j % S], (unsigned)((j / S) & 1), nullptr, wait_ns);
}

// ---------------------------------------------------------------------------
// Host side.
// ---------------------------------------------------------------------------
// Columns of a tile: 128 bytes of kz per line, 64 at N = 512 (FP32; a thread of
// an FP64 tile would need 22 modes of two accumulators, 176 registers, beside a
// 32-point transform: FP64 runs of 512 points take the separate passes).
template <typename T, int N>
constexpr int kXCols = (sizeof(T) == 8 ? 8 : 16) / (N > 256 ? 2 : 1);

// Index of an instance's occupancy in FFTPlan::x_occ.
constexpr int x_instance(int op, bool inv) { return op == kXNs && !inv ? 4 : op; }

// Raises the shared-memory limit of one instance on the current device and asks
// how many of its CTAs an SM holds there.  Both belong to the device, so they are
// taken at every plan creation and kept in the plan: asked once per process, a
// context on another device would launch without its limit.  0: not available
// (the caller takes the separate passes).
template <typename T, int N, int OP, bool INV>
int x_fused_occupancy() {
    constexpr int    W    = kXCols<T, N>;
    constexpr size_t smem = x_fuse_smem<T, N, W, OP>();
    auto             kern = x_fused_kernel<T, N, W, OP, INV>;
    int              n    = 0;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, W * Split<N>::N1, smem) != cudaSuccess) {
        cudaGetLastError();
        n = 0;
    }
    return n;
}
template <typename T, int N>
void x_fused_setup_n(FFTPlan<T> &P) {
    P.x_occ[x_instance(kXZeta, true)] = x_fused_occupancy<T, N, kXZeta, true>();
    P.x_occ[x_instance(kXNs, true)]   = x_fused_occupancy<T, N, kXNs, true>();
    P.x_occ[x_instance(kXNs, false)]  = x_fused_occupancy<T, N, kXNs, false>();
    P.x_occ[x_instance(kXProj, true)] = x_fused_occupancy<T, N, kXProj, false>();
    P.x_occ[x_instance(kXSole, true)] = x_fused_occupancy<T, N, kXSole, true>();
}
// The instances of the plan's axis, on the current device.
template <typename T>
void x_fused_setup(FFTPlan<T> &P) {
    switch (P.g.nx) {
#define SPM_XF(NN) case NN: x_fused_setup_n<T, NN>(P); break;
        SPM_XF(8) SPM_XF(16) SPM_XF(32) SPM_XF(64) SPM_XF(128) SPM_XF(256)
#undef SPM_XF
        case 512:
            if constexpr (sizeof(T) == 4) x_fused_setup_n<T, 512>(P);
            break;
        default: break;
    }
}

template <typename T, int N, int OP, bool INV>
cudaError_t x_fused_launch(const CUtensorMap &map, const XArgs<T> &A, int ctas, unsigned int *err,
                           unsigned long long wait_ns, int skip, cudaStream_t st) {
    constexpr int W = kXCols<T, N>;
    x_fused_kernel<T, N, W, OP, INV><<<std::min(A.ntiles, ctas), W * Split<N>::N1, x_fuse_smem<T, N, W, OP>(), st>>>(
        map, A, err, wait_ns, skip);
    return cudaGetLastError();
}

// One fused X pass.  Returns cudaErrorNotSupported where it cannot run (an
// FP64 axis of 512 points, no tensor-map entry point, no resident CTA); the
// caller then takes the separate passes.
template <typename T, int OP, bool INV>
cudaError_t x_fused(const FFTPlan<T> &P, XArgs<T> A, int runs, int nslots, cudaStream_t st) {
    const Grid &g = A.g;
    if (g.nx > (sizeof(T) == 8 ? 256 : 512) || g.field_elems_c() >> 32 || !encode_tiled_fn())
        return cudaErrorNotSupported;
    double kmin = 1e300, kmax = 0.0;  // x_reciprocal's range
    for (int d = 0; d < 3; d++) {
        const double n = d == 0 ? g.nx : d == 1 ? g.ny : g.nz;
        kmin           = std::min(kmin, g.wave[d] * g.wave[d]);
        kmax += 0.25 * n * n * g.wave[d] * g.wave[d];
    }
    if (!(kmin > 1e-30) || !(kmax < 1e30)) return cudaErrorNotSupported;
    const int W     = g.nx > 256 ? kXCols<T, 512> : kXCols<T, 256>;
    A.ct_used       = (g.trn[2] + W - 1) / W;
    A.n_used        = outer_count(g.ny, g.trn[1]);
    A.ntiles        = A.ct_used * A.n_used * runs;
    A.tw            = P.tw_x;
    const int ctas  = P.sm_count * P.x_occ[x_instance(OP, INV)];
    if (ctas < 1) return cudaErrorNotSupported;
    CUtensorMap map{};
    int         skip = 0;
    if (OP != kXZeta) {
        const uint64_t dims[5]    = {(uint64_t)2 * g.hnz, (uint64_t)g.ny, (uint64_t)g.nx, (uint64_t)runs,
                                     (uint64_t)nslots};
        const uint64_t strides[4] = {(uint64_t)2 * g.hnzp * sizeof(T), (uint64_t)g.ny * 2 * g.hnzp * sizeof(T),
                                     (uint64_t)A.run_stride * sizeof(cplx<T>),
                                     (uint64_t)A.slot_stride * sizeof(cplx<T>)};
        const uint32_t box[5]     = {(uint32_t)(2 * W), 1u, (uint32_t)std::min(g.nx, 256), 1u, 1u};
        if (!make_map<T>(&map, A.u, dims, strides, box)) return cudaErrorNotSupported;
        skip = P.skip_loads > 0 ? 1 : 0;
        if (skip) P.skip_loads--;
    }
    switch (g.nx) {
#define SPM_XF(NN)     case NN: return x_fused_launch<T, NN, OP, INV>(map, A, ctas, P.err, P.wait_ns, skip, st);
        SPM_XF(8) SPM_XF(16) SPM_XF(32) SPM_XF(64) SPM_XF(128) SPM_XF(256)
#undef SPM_XF
        case 512:
            if constexpr (sizeof(T) == 4)
                return x_fused_launch<T, 512, OP, INV>(map, A, ctas, P.err, P.wait_ns, skip, st);
            return cudaErrorNotSupported;
        default: return cudaErrorNotSupported;
    }
}

}  // namespace spm
