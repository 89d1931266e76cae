// solver_kernels.cuh -- the five fused passes of one pseudospectral step and the
// small kernels around them (B200 / sm_100a, bandwidth-bound, no tensor cores).
//
// Data layout in HBM (complex elements, kz contiguous everywhere):
//   S0 compact spectral state   [iy][ix][kz]   Ky x Kx x Kz   (retained modes only)
//   S1 after the x transform    [iy][x][kz]    Ky x Mx x Kp
//   S2 after the y transform    [y][x][kz]     My x Mx x Kp
// with Kp >= Kz the row pitch of the work buffers (row_pitch).
// Kx=2*hx+1 (kx=-hx..hx), Ky=2*hy+1, Kz=hz+1 (kz=0..hz) with h=N/2: the 3/2-rule
// box of the reference (src/HIT_LES.cpp:858-873, both +-N/2 kept for even N).
// Wavenumbers are k = s*m with s the length factor of the axis, so a non-cubic
// box of the reference (src/MAIN.cpp:216-260, src/HIT_LES.cpp:867-871) runs on
// its true grid (ActualM) instead of the expanded one.
//
// Pass plan of one step (DNS, advective form of the reference):
//   K1 inverse x : S0 u,v,w          -> S1 u,v,w, du/dx, dv/dx, dw/dx
//   K2 inverse y : S1 (6)            -> S2 + du/dy, dv/dy, dw/dy (9)
//   K3 z         : c2r of 12 fields (dz from u,v,w), conv = u_j d_j u_i (+ CFL
//                  maxima), r2c -> S2 conv_x, conv_y, conv_z
//   K4 forward y : S2 (3)            -> S1 (3)
//   K5 forward x : S1 (3)            -> S0 G (3)
//   K6 sweep     : G, u, R^{n-1} [, u^{n-1}] -> 1/M^3, R, Coriolis, forcing,
//                  AB2 or kappa-scheme predictor, projection -> u^{n+1}, R^n.
// The rotational form (the default of DNS) carries u and the vorticity instead: K1 writes
// six fields from five transforms, K2 six, K3 three over the first of them.  LES (Smagorinsky) adds the SGS stress, whose
// divergence is folded into the forward passes (i kz t_i3 in K3, i ky t_i2 in
// K4, i kx t_i1 in K5).
#pragma once
#include "fft_core.cuh"

namespace spns {

enum Mode { MODE_VEL = 0, MODE_ROT = 1, MODE_ADV = 2, MODE_LES = 3, MODE_INV = 4 };
// MODE_INV: velocity-gradient invariants (post-processing, not a step): the x/y
// passes form the gradients as in MODE_ADV, the z pass forms Q_G, Q_S, R_G, R_S, V^2
// on the grid and transforms them forward, the forward y/x passes carry 5 fields.

struct Geo {
    int Kx, Ky, Kz;   // retained mode counts (Ky: rows held, the slab's in a slab decomposition)
    int hx, hy, hz;   // half widths
    int Mx, My, Mz;   // true FFT grid (Mx: x planes held, the slab's in the y/z passes of a slab decomposition)
    int sx, sy, sz;   // wavenumber scale per axis (length factor)
    long long S0, S1, S2; // elements per field in each layout
    int y0, Kyg;      // first compact ky row held and the box's compact ky count (0 and Ky on one GPU)
    int Kp;           // row pitch of S1 and S2
};

// Row pitch of the work buffers: Kz is odd for the usual even N/2, so packed rows start at
// every offset within a line, and the passes' 128-byte row pieces straddle two lines each
// (N = 512 with Kz 257 against 256: y pass 7.0 against 6.3 ms per 1 % fewer modes in
// double, 4.15 against 3.43 in single precision).  Rows of 1 KB and more start on a
// 128-byte line, shorter ones (small boxes, held in L2) on a 32-byte sector.
__host__ __device__ inline int row_pitch(int Kz, int bytes) {
    const int a = (Kz * bytes >= 1024 ? 128 : 32) / bytes;
    return (Kz + a - 1) / a * a;
}

// m2 (ky/sy) of compact row iy held by this geometry
__host__ __device__ __forceinline__ int ky_mode(const Geo &g, int iy) {
    const int r = g.y0 + iy;
    return r <= g.hy ? r : r - g.Kyg;
}

// Solver scalars living in device memory (read by kernels, updated by the
// finisher), so that a captured step stays valid while they change.
struct DevScalars {
    double dt, time, nu, kappa, alpha;
    double maxvel, phi0;
    double ek_tot, ok_tot, relambda;
    double sumsq_phys;                   // sum of u^2+v^2+w^2 over the grid (energy check)
    unsigned long long max_bits[4];      // max|u|, max|v|, max|w|, max(|u|/Ax+|v|/Ay+|w|/Az)
    long long iter;
    int nonfinite, domain_err;
    int wait_timeout;                    // a bounded wait of a staged pass gave up (SPNS_ERR_TIMEOUT)
    double ef;                           // slab decomposition: this slab's energy of the forced shells
};

struct StepConsts {
    double inv_norm;      // 1/(Mx*My*Mz) of the true grid
    double omega_x, omega_y, omega_z;
    double Ax, Ay, Az, inv_Ax, inv_Ay, inv_Az;
    double C_At, Ah, t1;
    double kopt_k[2], phi[3], c[14];
    double les_ct;        // (C_Smag*delta)^2
    double fixed_dt;
    int eps_on, eps_kmin, eps_kmax;
    int rotating, self_adaptive;
};

__device__ __forceinline__ int ffreq(int a, int M) { return a <= M / 2 ? a : a - M; }

// Blocks per SM the x/y passes are compiled for (their register budget), per
// pass (1 inverse x, 2 inverse y, 4 forward y, 5 forward x).
#ifndef SPNS_AX_MINB
#define SPNS_AX_MINB 2
#endif
#ifndef SPNS_K2_MINB
#define SPNS_K2_MINB SPNS_AX_MINB
#endif
#ifndef SPNS_K1_MINB
#define SPNS_K1_MINB SPNS_AX_MINB
#endif
#ifndef SPNS_K5_MINB
#define SPNS_K5_MINB SPNS_AX_MINB
#endif
#ifndef SPNS_F32_AX_MINB
#define SPNS_F32_AX_MINB 2
#endif
// The LES forward passes hold two arrays of 12 values per thread: three blocks of 128 threads.
// Blocks of 256 threads (length 768), LES N=512, double / single: y two blocks 10.0 / 5.2 ms, one 11.0 /
// 5.5; x two 5.1 / 3.0, one 4.0 / 2.65.
template <typename T, int PASS, int MODE, int THREADS> struct AxisMinBlocks {
    static constexpr int N = MODE == 3 /* LES */ && PASS >= 4 ? (THREADS <= 128 ? 3 : THREADS <= 256 && PASS == 4 ? 2 : 1)
                             : sizeof(T) == 8 ? ((PASS == 2 || PASS == 4) ? SPNS_K2_MINB : PASS == 1 ? SPNS_K1_MINB : SPNS_K5_MINB)
                                            : SPNS_F32_AX_MINB;
};

// Field counts of the work buffers per mode.
template <int MODE> struct Fields {
    static constexpr int K1 = MODE == MODE_VEL ? 3 : 6;                          // S1 after the inverse x pass
    static constexpr int K2 = MODE == MODE_VEL ? 3 : MODE == MODE_ROT ? 6 : 9;  // S2 after the inverse y pass
    static constexpr int K4 = MODE == MODE_LES ? 6 : MODE == MODE_INV ? 5 : 3;  // S1 after the forward y pass
    static constexpr int NOUT = MODE == MODE_INV ? 5 : 3;                       // compact outputs of the forward x pass
};

// Start of a step: the maxima of the grid velocity and its squared sum begin at zero (they
// are gathered by the z pass; the first kernel of a step resets them, after the last step's
// end has used them and long before this step's z pass).
__device__ __forceinline__ void reset_maxima(DevScalars *ds) {
    if (ds && (blockIdx.x | blockIdx.y) == 0 && threadIdx.x == 0) {
        for (int i = 0; i < 4; i++) ds->max_bits[i] = 0ull;
        ds->sumsq_phys = 0.0;
    }
}

// ===========================================================================
// Elements of the x/y passes.  A thread transforms one kz column, or in single precision
// (T = f2) two adjacent ones, which are 16 bytes of a row: the same tiles, shared-memory
// layouts and launch shapes as in double precision.
// ===========================================================================
template <typename T> using SCx = cx<typename Arith<T>::S>;   // element of the arrays in memory
// Work buffers (S1, S2): rows start on 16 bytes and are padded, so both columns are always there.
__device__ __forceinline__ cx<double> ld_work(const cx<double> *p, cx<double> *) { return *p; }
__device__ __forceinline__ cx<float> ld_work(const cx<float> *p, cx<float> *) { return *p; }
__device__ __forceinline__ cx<f2> ld_work(const cx<float> *p, cx<f2> *) {
    const float4 a = *reinterpret_cast<const float4 *>(p);
    return mk<f2>(f2(a.x, a.z), f2(a.y, a.w));
}
__device__ __forceinline__ void st_work(cx<double> *p, cx<double> v) { *p = v; }
__device__ __forceinline__ void st_work(cx<float> *p, cx<float> v) { *p = v; }
__device__ __forceinline__ void st_work(cx<float> *p, cx<f2> v) {
    *reinterpret_cast<float4 *>(p) = make_float4(v.x.lo(), v.y.lo(), v.x.hi(), v.y.hi());
}
// Compact arrays (S0): rows of Kz elements, so a pair may straddle 16 bytes and the last row end (two: it is whole).
__device__ __forceinline__ cx<double> ld_compact(const cx<double> *p, bool, cx<double> *) { return *p; }
__device__ __forceinline__ cx<float> ld_compact(const cx<float> *p, bool, cx<float> *) { return *p; }
__device__ __forceinline__ void st_compact(cx<double> *p, cx<double> v, bool) { *p = v; }
__device__ __forceinline__ void st_compact(cx<float> *p, cx<float> v, bool) { *p = v; }
__device__ __forceinline__ void st_compact(cx<float> *p, cx<f2> v, bool two) {
    p[0] = mk<float>(v.x.lo(), v.y.lo());
    if (two) p[1] = mk<float>(v.x.hi(), v.y.hi());
}
// s kz of the thread's columns
__device__ __forceinline__ double col_k(int s, int kz, double *) { return (double)(s * kz); }
__device__ __forceinline__ float col_k(int s, int kz, float *) { return (float)(s * kz); }

// The x/y passes wait on the loads of a field with nothing else in flight, so while it is
// transformed the rows of the block's next field are asked for in L2.  addr(e): the tile's
// first element in the thread's row e (null: no row); the P threads of a row share its E lines.
// Without and with, in ms, rotational form, double / single:
//   N=256  K1 0.516 -> 0.450 / 0.276 -> 0.251     K2 0.915 -> 0.648 / 0.483 -> 0.389
//          K4 0.324 -> 0.301 / 0.190 -> 0.170     K5 0.223 -> 0.201 / 0.129 -> 0.137
//   N=512  K1 4.13 -> 4.00 / 2.27 -> 2.21         K2 5.75 -> 5.71 / 2.97 -> 3.01
//          K4 2.63 -> 2.70 / 1.27 -> 1.43         K5 1.80 -> 1.84 / 1.17 -> 1.22
// From length 768 on the current and the next tiles of all resident blocks (100 KB each, 58 MB
// together) with their output do not stay in the near half of L2 until they are used: there K2
// (input rows below the cut-off only) asks after the transform, before the stores (5.58 /
// 2.89), and K4 and K5 not at all (K4 so 2.72 / 1.36); nor K2 at 1536 (N=1024 single 48.6 -> 59.8).
// The LES passes write more per read and
// their forward ones have three blocks per SM to cover each other's loads: K2 0.952 -> 0.977 / 0.672 ->
// 0.576 (on in single precision), K4 1.04 -> 1.17 / 0.61 -> 0.63, K5 0.56 -> 0.65 / 0.34 -> 0.40.
template <int L> constexpr bool PREFETCH_LATE = L >= 768;
template <typename T, int L, int MODE> constexpr bool PREFETCH_2 = L <= 768 && (MODE != MODE_LES || Arith<T>::SINGLE);
template <int L, int MODE> constexpr bool PREFETCH_4 = L < 768 && MODE != MODE_LES;
template <typename T, int L, int MODE> constexpr bool PREFETCH_5 = L < 768 && MODE != MODE_LES && !Arith<T>::SINGLE;
template <int E, int P, class Addr> __device__ __forceinline__ void prefetch_rows(int p, Addr addr) {
#pragma unroll
    for (int i = 0; i < (E + P - 1) / P; i++) {
        const int e = i * P + p;
        if (E % P != 0 && e >= E) break;
        const void *a = addr(e);
        if (a) asm volatile("prefetch.global.L2 [%0];\n" ::"l"(a));
    }
}

// ===========================================================================
// K1: inverse transform along x.  Block = (kz chunk, iy).
//   VEL: u,v,w   ROT: u,v,w and the vorticity   ADV/LES: u,v,w, du/dx, dv/dx, dw/dx
// ky and kz are constant along a line, so of the vorticity w_x = i(ky w - kz v),
// w_y = i(kz u - kx w), w_z = i(kx v - ky u) only the parts with kx need transforms of
// their own: five transforms (v, w, u, kx w, kx v) and five reads of the state per point
// instead of six and nine.  The one transformed field a later output needs (v for w_x, u
// for w_y and w_z) waits in shared memory, each thread its own values (K1Smem).
// ===========================================================================
template <typename T, int L, int E, int P, int MODE> struct K1Smem {
    static constexpr size_t BYTES = (size_t)L * P * sizeof(cx<T>) * (MODE == MODE_ROT ? 2 : 1);
};
template <typename T, int L, int E, int P, int MODE>
__device__ __forceinline__ void k1_inv_x_body(Geo g, const SCx<T> *__restrict__ u, const SCx<T> *__restrict__ v,
                                              const SCx<T> *__restrict__ w, SCx<T> *__restrict__ out, const cx<T> *__restrict__ tw,
                                              int f0, int fs) {
    extern __shared__ __align__(16) unsigned char smraw[];
    constexpr int THREADS = P * (L / E);
    const int tid = threadIdx.x, p = tid % P, q = tid / P;
    const int iy = blockIdx.y, kz = (blockIdx.x * P + p) * Arith<T>::W;
    const bool ok = kz < g.Kz, two = kz + 1 < g.Kz;
    SmRowMajor<T, P> sm{reinterpret_cast<cx<T> *>(smraw), p};
    const long long rb = (long long)iy * g.Kx * g.Kz + kz, ob = (long long)iy * g.Mx * g.Kp + kz;
    // loads the field into the input rows, times kx where `deriv` (all loads before the first use)
    auto load = [&](cx<T>(&r)[E], const SCx<T> *src, bool deriv) {
#pragma unroll
        for (int e = 0; e < E; e++) {
            const int m1 = ffreq(in_row<L, E, true>(q, e), L);
            r[e] = (ok && m1 <= g.hx && m1 >= -g.hx) ? ld_compact(src + rb + (long long)(m1 >= 0 ? m1 : m1 + g.Kx) * g.Kz, two, (cx<T> *)nullptr)
                                                           : zero<T>();
        }
        if (deriv) {
#pragma unroll
            for (int e = 0; e < E; e++) r[e] = T(g.sx * ffreq(in_row<L, E, true>(q, e), L)) * r[e];
        }
    };
    // the first column of each row; a compact row's tile may end in the next line
    auto prefetch = [&](const SCx<T> *src) {
        const int last = (g.Kz - (kz - p * Arith<T>::W) < P * Arith<T>::W ? g.Kz - (kz - p * Arith<T>::W) : P * Arith<T>::W) - 1;
        prefetch_rows<E, P>(p, [&](int e) -> const void * {
            const int m1 = ffreq(in_row<L, E, true>(q, e), L);
            if (m1 > g.hx || m1 < -g.hx) return nullptr;
            const SCx<T> *a = src + (rb - p * Arith<T>::W) + (long long)(m1 >= 0 ? m1 : m1 + g.Kx) * g.Kz;
            asm volatile("prefetch.global.L2 [%0];\n" ::"l"(a + last));
            return a;
        });
    };
    auto put = [&](int f, auto value) {
        if (!ok) return;
        SCx<T> *o = out + (long long)f * g.S1 + ob;
#pragma unroll
        for (int e = 0; e < E; e++) st_work(o + (long long)out_row<L, E, true>(q, e) * g.Kp, value(e));
    };
    if constexpr (MODE == MODE_ROT) {
        const T kzf = col_k(g.sz, kz, (T *)nullptr), kyf = T(g.sy * ky_mode(g, iy));
        cx<T> *const slot = reinterpret_cast<cx<T> *>(smraw) + L * P + tid;
        if (fs > 1) {   // outputs split over blocks: each forms its own input
#pragma unroll 1
            for (int f = f0; f < 6; f += fs) {
                cx<T> r[E];
                load(r, f == 0 || f == 4 ? u : f == 1 || f == 5 ? v : w, f == 5);
                if (f >= 3) {
                    cx<T> b[E];
                    load(b, f == 5 ? u : f == 4 ? w : v, f == 4);
                    const T ka = f == 3 ? kyf : f == 4 ? kzf : T(1), kb = f == 3 ? kzf : f == 4 ? T(1) : kyf;
#pragma unroll
                    for (int e = 0; e < E; e++) r[e] = mul_i(ka * r[e] - kb * b[e]);
                }
                fft<T, L, E, true>(r, sm, q, tw);
                put(f, [&](int e) { return r[e]; });
            }
            return;
        }
#pragma unroll 1
        for (int s = 0; s < 5; s++) {
            cx<T> r[E];
            load(r, s == 2 ? u : (s == 0 || s == 4) ? v : w, s >= 3);
            if (s < 2) prefetch(s == 0 ? w : u);
            fft<T, L, E, true>(r, sm, q, tw);
            if (s < 3) put(s == 0 ? 1 : s == 1 ? 2 : 0, [&](int e) { return r[e]; });
            if (s == 1) put(3, [&](int e) { return mul_i(kyf * r[e] - kzf * slot[e * THREADS]); });
            if (s == 3) put(4, [&](int e) { return mul_i(kzf * slot[e * THREADS] - r[e]); });
            if (s == 4) put(5, [&](int e) { return mul_i(r[e] - kyf * slot[e * THREADS]); });
            if (s == 0 || s == 2) {
#pragma unroll
                for (int e = 0; e < E; e++) slot[e * THREADS] = r[e];
            }
        }
    } else {
#pragma unroll 1
        for (int f = f0; f < Fields<MODE>::K1; f += fs) {
            cx<T> r[E];
            load(r, f % 3 == 0 ? u : f % 3 == 1 ? v : w, f >= 3);
            if (f + fs < 3) prefetch(f + fs == 1 ? v : w);
            fft<T, L, E, true>(r, sm, q, tw);
            if (f < 3) put(f, [&](int e) { return r[e]; });
            else put(f, [&](int e) { return mul_i(r[e]); });
        }
    }
}

// ===========================================================================
// K2: inverse transform along y.  Block = (kz chunk, x).
//   ROT: u,v,w, w_x, w_y, w_z (formed by K1)
//   ADV/LES: u,v,w, du/dx,dv/dx,dw/dx, du/dy,dv/dy,dw/dy
// ===========================================================================
template <typename T, int L, int E, int P, int MODE>
__device__ __forceinline__ void k2_inv_y_body(Geo g, const SCx<T> *__restrict__ in, SCx<T> *__restrict__ out,
                                              const cx<T> *__restrict__ tw, int f0, int fs) {
    extern __shared__ __align__(16) unsigned char smraw[];
    const int tid = threadIdx.x, p = tid % P, q0 = tid / P;
    const int x = blockIdx.y, kz = (blockIdx.x * P + p) * Arith<T>::W;
    const bool ok = kz < g.Kz;
    SmRowMajor<T, P> sm{reinterpret_cast<cx<T> *>(smraw), p};
    // row offsets in 32 bits (a field has fewer than 2^31 elements at every compiled length):
    // one register and one multiply-add per address instead of a 64-bit chain
    const unsigned col = (unsigned)x * g.Kp + kz, rs = (unsigned)g.Mx * g.Kp;
    // Nine fields: d/dy of u, v, w follow right after their own transforms, whose input is
    // then still in L2 (u, d/dy u, v, ..., then the x derivatives).
    constexpr bool DERIV = Fields<MODE>::K2 == 9;
    auto field = [](int i) { return !DERIV ? i : i >= 6 ? i - 3 : i & 1 ? 6 + i / 2 : i / 2; };
    auto source = [](int f) { return f >= 6 ? f - 6 : f; };
#pragma unroll 1
    for (int i = f0; i < Fields<MODE>::K2; i += fs) {
        const int q = opaque(q0), f = field(i);
        cx<T> r[E];
        const bool deriv = f >= 6;
        const SCx<T> *F = in + (long long)source(f) * g.S1;
#pragma unroll
        for (int e = 0; e < E; e++) {
            const int m2 = ffreq(in_row<L, E, true>(q, e), L);
            r[e] = (ok && m2 <= g.hy && m2 >= -g.hy) ? ld_work(F + (col + (unsigned)(m2 >= 0 ? m2 : m2 + g.Ky) * rs), (cx<T> *)nullptr) : zero<T>();
        }
        auto prefetch = [&] {
            if (!PREFETCH_2<T, L, MODE> || i + fs >= Fields<MODE>::K2 || source(field(i + fs)) == source(f)) return;
            const SCx<T> *N = in + (long long)source(field(i + fs)) * g.S1;
            prefetch_rows<E, P>(p, [&](int e) -> const void * {
                const int m2 = ffreq(in_row<L, E, true>(q, e), L);
                return m2 <= g.hy && m2 >= -g.hy ? N + (col - p * Arith<T>::W + (unsigned)(m2 >= 0 ? m2 : m2 + g.Ky) * rs) : nullptr;
            });
        };
        if constexpr (!PREFETCH_LATE<L>) prefetch();
        if (deriv) {
#pragma unroll
            for (int e = 0; e < E; e++) r[e] = mul_i(T(g.sy * ffreq(in_row<L, E, true>(q, e), L)) * r[e]);
        }
        fft<T, L, E, true>(r, sm, q, tw);
        if constexpr (PREFETCH_LATE<L>) prefetch();
        if (ok) {
            SCx<T> *o = out + (long long)f * g.S2;
#pragma unroll
            for (int e = 0; e < E; e++) st_work(o + (col + (unsigned)out_row<L, E, true>(q, e) * rs), r[e]);
        }
    }
}

// ===========================================================================
// K3: along z.  c2r of two real fields per complex transform (a + i b with
// Hermitian extension; the kz=0 entries keep their real parts only, as a c2r of
// the reference does), pointwise products on the grid, r2c of the products
// (again two per transform) truncated to kz<=hz.  Block = P consecutive
// pencils; each thread keeps the values of its own grid rows in registers, so
// the inverse/forward hand-off needs no shared-memory round trip.
// ===========================================================================
// Element k of the pencil(s) a thread transforms: one pencil, or two (T = f2) that lie
// `step` elements apart.
__device__ __forceinline__ cx<double> ld_pencil(const cx<double> *p, int k, int, cx<double> *) { return p[k]; }
__device__ __forceinline__ cx<float> ld_pencil(const cx<float> *p, int k, int, cx<float> *) { return p[k]; }
__device__ __forceinline__ cx<f2> ld_pencil(const cx<float> *p, int k, int step, cx<f2> *) {
    const cx<float> a = p[k], b = p[k + step];
    return mk<f2>(f2(a.x, b.x), f2(a.y, b.y));
}
__device__ __forceinline__ void st_pencil(cx<double> *p, int k, int, cx<double> v) { p[k] = v; }
__device__ __forceinline__ void st_pencil(cx<float> *p, int k, int, cx<float> v) { p[k] = v; }
__device__ __forceinline__ void st_pencil(cx<float> *p, int k, int step, cx<f2> v) {
    p[k] = mk<float>(v.x.lo(), v.y.lo());
    p[k + step] = mk<float>(v.x.hi(), v.y.hi());
}
// Loads the 2-for-1 spectrum Z = Xa + i Xb at the thread's input rows.
// ma/mb: multiply the field by i*kz (z derivative) first.
template <typename T, int L, int E>
__device__ __forceinline__ void k3_load_pair(cx<T> (&r)[E], const SCx<T> *__restrict__ A, bool ma, const SCx<T> *__restrict__ B,
                                             bool mb, int Kz, T sz, int q, bool ok, int step = 0) {
#pragma unroll
    for (int e = 0; e < E; e++) {
        const int row = in_row<L, E, true>(q, e);
        cx<T> z = zero<T>();
        if (ok) {
            const bool lo = row < Kz, hi = row > L - Kz;
            if (lo || hi) {
                const int kk = lo ? row : L - row;
                cx<T> a = ld_pencil(A, kk, step, (cx<T> *)nullptr), b = B ? ld_pencil(B, kk, step, (cx<T> *)nullptr) : zero<T>();
                if (ma) a = mul_i(T(kk) * sz * a);
                if (mb) b = mul_i(T(kk) * sz * b);
                if (row == 0) z = mk<T>(a.x, b.x);
                else if (lo) z = mk<T>(a.x - b.y, a.y + b.x);
                else z = mk<T>(a.x + b.y, b.x - a.y);
            }
        }
        r[e] = z;
    }
}

template <typename T> __device__ __forceinline__ void block_max4(const double (&v)[4], DevScalars *ds) {
    __shared__ double red[4][32];
    double m[4] = {v[0], v[1], v[2], v[3]};
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int i = 0; i < 4; i++) m[i] = fmax(m[i], __shfl_xor_sync(0xffffffffu, m[i], o));
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    if (lane == 0)
#pragma unroll
        for (int i = 0; i < 4; i++) red[i][wid] = m[i];
    __syncthreads();
    if (wid == 0) {
#pragma unroll
        for (int i = 0; i < 4; i++) m[i] = lane < nw ? red[i][lane] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int i = 0; i < 4; i++) m[i] = fmax(m[i], __shfl_xor_sync(0xffffffffu, m[i], o));
        if (lane == 0)
#pragma unroll
            for (int i = 0; i < 4; i++) {
                double x = m[i];
                if (!(x <= 1.7976931348623157e308)) atomicExch(&ds->nonfinite, 1); // NaN or Inf
                else atomicMax(&ds->max_bits[i], (unsigned long long)__double_as_longlong(x));
            }
    }
    __syncthreads();
}

__device__ __forceinline__ void block_sum(double v, double *dst) {
    __shared__ double red[32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    if (lane == 0) red[wid] = v;
    __syncthreads();
    if (wid == 0) {
        v = lane < nw ? red[lane] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) atomicAdd(dst, v);
    }
    __syncthreads();
}

// Block maximum of a non-negative double, folded into *dst (its bits order as the values do).
__device__ __forceinline__ void block_max_bits(double v, unsigned long long *dst) {
    __shared__ double red[32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    if (lane == 0) red[wid] = v;
    __syncthreads();
    if (wid == 0) {
        v = lane < nw ? red[lane] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
        if (lane == 0) atomicMax(dst, (unsigned long long)__double_as_longlong(v));
    }
    __syncthreads();
}

// Forward transform of the register pair z = a + i b and extraction of both half spectra
// for kz < Kz:  Xa = (Z_k + conj Z_{L-k})/2, Xb = (Z_k - conj Z_{L-k})/(2i); with `single`
// one real field (b = 0), stored from the registers.  One copy of the transform code.
template <typename T, int L, int E>
__device__ __forceinline__ void k3_store_job(cx<T> (&r)[E], SmPencil<T, L, E> sm, int q, int Kz, cx<T> *A, cx<T> *B,
                                             bool single, bool ok, const cx<T> *__restrict__ tw) {
    constexpr int Q = L / E;
    fft<T, L, E, false, SmPencil<T, L, E>, (32 % (L / E) == 0)>(r, sm, q, tw);
    if (single) {
        if (ok) {
#pragma unroll
            for (int e = 0; e < E; e++) {
                const int row = out_row<L, E, false>(q, e);
                if (row < Kz) A[row] = r[e];
            }
        }
        return;
    }
    __syncthreads();
#pragma unroll
    for (int e = 0; e < E; e++) sm.at(out_row<L, E, false>(q, e)) = r[e];
    __syncthreads();
    if (ok) {
        const T h = T(0.5);
        for (int k = q; k < Kz; k += Q) {
            cx<T> zk = sm.at(k), zm = sm.at(k == 0 ? 0 : L - k);
            A[k] = mk<T>(h * (zk.x + zm.x), h * (zk.y - zm.y));
            B[k] = mk<T>(h * (zk.y + zm.y), h * (zm.x - zk.x));
        }
    }
    __syncthreads();
}

// Running CFL maxima; a NaN or Inf velocity turns the maxima into +Inf (fmax
// alone would drop NaN), which the block reduction reports as non-finite.
template <typename T>
__device__ __forceinline__ void cfl_update(double (&mx)[4], double uu, double vv, double ww, const StepConsts &c) {
    const double au = fabs(uu), av = fabs(vv), aw = fabs(ww);
    const double s = au * c.inv_Ax + av * c.inv_Ay + aw * c.inv_Az;
    if (!(s <= 1.7976931348623157e308)) { mx[0] = mx[1] = mx[2] = mx[3] = __longlong_as_double(0x7ff0000000000000LL); return; }
    mx[0] = fmax(mx[0], au); mx[1] = fmax(mx[1], av); mx[2] = fmax(mx[2], aw);
    mx[3] = fmax(mx[3], s);
}

__device__ __forceinline__ void cfl_rows(double (&mx)[4], double u, double v, double w, const StepConsts &c) { cfl_update<double>(mx, u, v, w, c); }
__device__ __forceinline__ void cfl_rows(double (&mx)[4], float u, float v, float w, const StepConsts &c) { cfl_update<float>(mx, u, v, w, c); }
__device__ __forceinline__ void cfl_rows(double (&mx)[4], f2 u, f2 v, f2 w, const StepConsts &c) {
    cfl_update<float>(mx, u.lo(), v.lo(), w.lo(), c);
    cfl_update<float>(mx, u.hi(), v.hi(), w.hi(), c);
}

// Asynchronous global->shared copy of one complex element (LDGSTS; 16 B for
// double, 8 B for float), completed per thread by commit/wait groups.
template <typename T> __device__ __forceinline__ void cp_async_elem(cx<T> *smem_dst, const cx<T> *gsrc) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem_dst);
    if constexpr (sizeof(cx<T>) == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gsrc) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

#ifndef SPNS_Z_STAGE_PAIRS
#define SPNS_Z_STAGE_PAIRS 3      // double rotational z pass: input pairs staged in shared memory
#endif
#ifndef SPNS_F32_Z_STAGE_PAIRS
#define SPNS_F32_Z_STAGE_PAIRS 3
#endif
template <typename T> struct K3StagePairs { static constexpr int N = sizeof(T) == 8 ? SPNS_Z_STAGE_PAIRS : SPNS_F32_Z_STAGE_PAIRS; };
// STAGE (rotational form): the six input fields of the block's pencils are
// copied into shared memory asynchronously at the start, in the order the
// three pairs use them, so the loads of the second and third pairs overlap the
// transforms of the first.  Dynamic shared memory then holds P*6*Kz extra
// complex values after the exchange buffers.
// Register budget of the z pass, as registers per thread (0: none), turned into the
// minimum resident blocks per SM of __launch_bounds__ for the block size at hand: single
// precision 128 (16 warps per SM), double precision none.
#ifndef SPNS_K3_REGS_ROT
#define SPNS_K3_REGS_ROT 0
#endif
#ifndef SPNS_F32_K3_REGS_ROT
#define SPNS_F32_K3_REGS_ROT 128
#endif
template <typename T, int THREADS> struct K3MinBlocks {
    static constexpr int REGS = sizeof(T) == 8 ? SPNS_K3_REGS_ROT : SPNS_F32_K3_REGS_ROT;
    static constexpr int B = REGS > 0 ? 65536 / (REGS * THREADS) : 1;
    static constexpr int N = B < 1 ? 1 : B;
};
template <typename T, int L, int E, int P, int MODE, bool STAGE>
__device__ __forceinline__ void k3_z_body(Geo g, cx<T> *__restrict__ buf, const StepConsts &c, DevScalars *ds,
                                          double *__restrict__ phys, const cx<T> *__restrict__ tw) {
    extern __shared__ __align__(16) unsigned char smraw[];
    constexpr int Q = L / E;
    const int tid = threadIdx.x, p = tid / Q, q = tid % Q;
    const long long npen = (long long)g.Mx * g.My;
    const long long pen = (long long)blockIdx.x * P + p;
    const bool ok = pen < npen;
    const long long base = (ok ? pen : 0) * g.Kp;
    cx<T> *smc = reinterpret_cast<cx<T> *>(smraw);
    constexpr int PITCH = SmPencil<T, L, E>::PITCH;
    SmPencil<T, L, E> sm{smc + p * PITCH};
    const T sz = T(g.sz);
    cx<T> *const B0 = buf + base;
#define F(i) (B0 + (long long)(i) * g.S2)
    double mx[4] = {0.0, 0.0, 0.0, 0.0};

    if constexpr (MODE == MODE_VEL) {
        cx<T> A[E], B[E];
        k3_load_pair<T, L, E>(A, F(0), false, F(1), false, g.Kz, sz, q, ok);
        fft<T, L, E, true, SmPencil<T, L, E>, (32 % (L / E) == 0)>(A, sm, q, tw);
        k3_load_pair<T, L, E>(B, F(2), false, nullptr, false, g.Kz, sz, q, ok);
        fft<T, L, E, true, SmPencil<T, L, E>, (32 % (L / E) == 0)>(B, sm, q, tw);
        double ss = 0.0;
#pragma unroll
        for (int e = 0; e < E; e++) {
            const double uu = A[e].x, vv = A[e].y, ww = B[e].x;
            cfl_update<T>(mx, uu, vv, ww, c);
            ss += uu * uu + vv * vv + ww * ww;
        }
        if (!ok) { mx[0] = mx[1] = mx[2] = mx[3] = 0.0; ss = 0.0; }
        if (phys && ok) {
            const int y = (int)(pen / g.Mx), x = (int)(pen % g.Mx);
            const long long n3 = (long long)g.Mx * g.My * g.Mz;
            double *o = phys + ((long long)x * g.My + y) * g.Mz;
#pragma unroll
            for (int e = 0; e < E; e++) {
                const int row = out_row<L, E, true>(q, e);
                o[row] = A[e].x; o[n3 + row] = A[e].y; o[2 * n3 + row] = B[e].x;
            }
        }
        block_max4<T>(mx, ds);
        block_sum(ss, &ds->sumsq_phys);
    } else {
        static_assert(MODE == MODE_ROT, "the other forms run in k3_field");
        // pairs (u, w_x), (v, w_y), (w, w_z);  c = w x u  (= u.grad u + gradient)
        // STAGE: the input fields of the last NSP pairs are copied into shared memory
        // asynchronously at the start, in the order the pairs use them, so their loads
        // overlap the transforms of the earlier pairs.
        constexpr int NSP = STAGE ? K3StagePairs<T>::N : 0;
        constexpr int FIRST = 3 - NSP;
        cx<T> A[E];
        const cx<T> *src[6] = {F(0), F(1), F(2), F(3), F(4), F(5)};
        if constexpr (STAGE) {
            cx<T> *st = smc + P * PITCH + (long long)p * 2 * NSP * g.Kz;
#pragma unroll
            for (int gp = FIRST; gp < 3; gp++) {
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int f = gp + 3 * h, slot = 2 * (gp - FIRST) + h;
                    if (ok)
                        for (int k = q; k < g.Kz; k += Q) cp_async_elem<T>(st + slot * g.Kz + k, src[f] + k);
                }
                cp_async_commit();
            }
#pragma unroll
            for (int gp = FIRST; gp < 3; gp++) {
                src[gp] = st + 2 * (gp - FIRST) * g.Kz;
                src[gp + 3] = st + (2 * (gp - FIRST) + 1) * g.Kz;
            }
        }
        // Physical values in register slots 0 u, 1 w_x, 2 v, 3 w_y, 4 c_z.  The pair
        // loop is unrolled (rolled, with slots written in one iteration and read in a
        // later one, it computed wrong products); the two forward jobs share one
        // transform body.  The slots are defined on entry all the same.
        T rs[5][E];
#pragma unroll
        for (int i = 0; i < 5; i++)
#pragma unroll
            for (int e = 0; e < E; e++) rs[i][e] = T(0);
#pragma unroll
        for (int pi = 0; pi < 3; pi++) {
            if constexpr (STAGE) {
                if (pi == FIRST) { cp_async_wait<NSP - 1>(); __syncthreads(); }
                else if (pi == FIRST + 1) { cp_async_wait<(NSP >= 2 ? NSP - 2 : 0)>(); __syncthreads(); }
                else if (pi == FIRST + 2) { cp_async_wait<0>(); __syncthreads(); }
            }
            k3_load_pair<T, L, E>(A, src[pi], false, src[pi + 3], false, g.Kz, sz, q, ok);
            fft<T, L, E, true, SmPencil<T, L, E>, (32 % (L / E) == 0)>(A, sm, q, tw);
            if (pi == 0) {
#pragma unroll
                for (int e = 0; e < E; e++) { rs[0][e] = A[e].x; rs[1][e] = A[e].y; }
            } else if (pi == 1) {
#pragma unroll
                for (int e = 0; e < E; e++) { rs[2][e] = A[e].x; rs[3][e] = A[e].y; rs[4][e] = rs[1][e] * A[e].x - A[e].y * rs[0][e]; }
            }
        }
#pragma unroll
        for (int e = 0; e < E; e++) {
            const T uu = rs[0][e], ox = rs[1][e], vv = rs[2][e], oy = rs[3][e], ww = A[e].x, oz = A[e].y;
            cfl_update<T>(mx, uu, vv, ww, c);
            A[e] = mk<T>(oy * ww - oz * vv, oz * uu - ox * ww);
        }
        if (!ok) { mx[0] = mx[1] = mx[2] = mx[3] = 0.0; }
        block_max4<T>(mx, ds);
#pragma unroll 1
        for (int j = 0; j < 2; j++) {
            if (j == 1) {
#pragma unroll
                for (int e = 0; e < E; e++) A[e] = mk<T>(rs[4][e], T(0));
            }
            // c_z goes over w_x (field 3, consumed by the first pair): the forward y pass
            // reads the rotational nonlinear term from fields 0, 1 and 3 (k4_in_field)
            k3_store_job<T, L, E>(A, sm, q, g.Kz, j == 0 ? F(0) : F(3), j == 0 ? F(1) : nullptr, j == 1, ok, tw);
        }
    }
#undef F
}

// S2 field holding component f of the nonlinear term after the z pass: the
// rotational form writes c_z over w_x (field 3), the others in order.
template <int MODE> __host__ __device__ constexpr int k4_in_field(int f) { return (MODE == MODE_ROT && f == 2) ? 3 : f; }

// ===========================================================================
// K4: forward transform along y with ky truncation.  Block = (kz chunk, x).
// LES: G_i += i ky t_i2 (SGS divergence, y part).
// ===========================================================================
template <typename T, int L, int E, int P, int MODE>
__device__ __forceinline__ void k4_fwd_y_body(Geo g, const SCx<T> *__restrict__ in, SCx<T> *__restrict__ out,
                                              const cx<T> *__restrict__ tw, int f0, int fs) {
    extern __shared__ __align__(16) unsigned char smraw[];
    const int tid = threadIdx.x, p = tid % P, q0 = tid / P;
    const int x = blockIdx.y, kz = (blockIdx.x * P + p) * Arith<T>::W;
    const bool ok = kz < g.Kz;
    SmRowMajor<T, P> sm{reinterpret_cast<cx<T> *>(smraw), p};
    const unsigned col = (unsigned)x * g.Kp + kz, rs = (unsigned)g.Mx * g.Kp;
    constexpr bool LES = MODE == MODE_LES;
    // LES.  in (S2): 0 G_x, 1 G_y, 2 G_z, 3 t11, 4 t12, 5 t13, 6 t22, 7 t23
    //       out (S1): 0 G_x + i ky t12, 1 G_y + i ky t22, 2 G_z + i ky t23, 3 t11, 4 t12, 5 t13
    // Groups: (t12, G_x), (t22, G_y), (t23, G_z), then t11 and t13 alone.
    constexpr int NG = LES ? 5 : Fields<MODE>::NOUT;
    // (next: the field read after this one, -1 for none)
    auto load_fft = [&](cx<T>(&r)[E], int f, int next) {
        const int q = opaque(q0);
        const SCx<T> *src = in + (long long)f * g.S2;
#pragma unroll
        for (int e = 0; e < E; e++) r[e] = ok ? ld_work(src + (col + (unsigned)in_row<L, E, false>(q, e) * rs), (cx<T> *)nullptr) : zero<T>();
        if (PREFETCH_4<L, MODE> && next >= 0) {
            const SCx<T> *N = in + (long long)next * g.S2;
            prefetch_rows<E, P>(p, [&](int e) -> const void * { return N + (col - p * Arith<T>::W + (unsigned)in_row<L, E, false>(q, e) * rs); });
        }
        fft<T, L, E, false>(r, sm, q, tw);
    };
    auto store = [&](int f, auto value) {
        if (!ok) return;
        const int q = opaque(q0);
        SCx<T> *o = out + (long long)f * g.S1;
#pragma unroll
        for (int e = 0; e < E; e++) {
            const int m2 = ffreq(out_row<L, E, false>(q, e), L);
            if (m2 <= g.hy && m2 >= -g.hy) st_work(o + (col + (unsigned)(m2 >= 0 ? m2 : m2 + g.Ky) * rs), value(e, m2));
        }
    };
    // first field of a group
    auto first = [&](int grp) { return grp >= NG ? -1 : !LES ? k4_in_field<MODE>(grp) : grp == 0 ? 4 : grp >= 3 ? 2 * grp - 3 : grp + 5; };
#pragma unroll 1
    for (int grp = f0; grp < NG; grp += fs) {
        cx<T> r[E];
        if (!LES || grp >= 3) {
            const int f = first(grp);
            load_fft(r, f, first(grp + fs));
            store(LES ? f : grp, [&](int e, int) { return r[e]; });
        } else {
            cx<T> t[E];
            load_fft(t, first(grp), grp);
            if (grp == 0) store(4, [&](int e, int) { return t[e]; });
            load_fft(r, grp, first(grp + fs));
            store(grp, [&](int e, int m2) { return r[e] + mul_i(T(g.sy * m2) * t[e]); });
        }
    }
}

// ===========================================================================
// K5: forward transform along x with kx truncation into the compact layout
// (S0).  Block = (kz chunk, iy).  LES: G_i += i kx t_i1 (SGS divergence, x part).
// ===========================================================================
template <typename T, int L, int E, int P, int MODE>
__device__ __forceinline__ void k5_fwd_x_body(Geo g, const SCx<T> *__restrict__ in, SCx<T> *__restrict__ G,
                                              const cx<T> *__restrict__ tw, int f0, int fs) {
    extern __shared__ __align__(16) unsigned char smraw[];
    const int tid = threadIdx.x, p = tid % P, q = tid / P;
    const int iy = blockIdx.y, kz = (blockIdx.x * P + p) * Arith<T>::W;
    const bool ok = kz < g.Kz, two = kz + 1 < g.Kz;
    SmRowMajor<T, P> sm{reinterpret_cast<cx<T> *>(smraw), p};
    const long long col = (long long)iy * g.Mx * g.Kp + kz;
    constexpr bool LES = MODE == MODE_LES;
    auto load_fft = [&](cx<T>(&r)[E], int f, int next) {
        const SCx<T> *src = in + (long long)f * g.S1 + col;
#pragma unroll
        for (int e = 0; e < E; e++) r[e] = ok ? ld_work(src + (long long)in_row<L, E, false>(q, e) * g.Kp, (cx<T> *)nullptr) : zero<T>();
        if (PREFETCH_5<T, L, MODE> && next >= 0) {
            const SCx<T> *N = in + (long long)next * g.S1 + (col - p * Arith<T>::W);
            prefetch_rows<E, P>(p, [&](int e) -> const void * { return N + (long long)in_row<L, E, false>(q, e) * g.Kp; });
        }
        fft<T, L, E, false>(r, sm, q, tw);
    };
#pragma unroll 1
    for (int f = f0; f < Fields<MODE>::NOUT; f += fs) {
        cx<T> r[E], t[LES ? E : 1];
        const int next = f + fs < Fields<MODE>::NOUT ? f + fs : -1;
        load_fft(r, f, LES ? 3 + f : next);
        if constexpr (LES) load_fft(t, 3 + f, next);   // t11, t12, t13
        if (!ok) continue;
        SCx<T> *o = G + (long long)f * g.S0 + (long long)iy * g.Kx * g.Kz + kz;
#pragma unroll
        for (int e = 0; e < E; e++) {
            const int m1 = ffreq(out_row<L, E, false>(q, e), L);
            if (m1 > g.hx || m1 < -g.hx) continue;
            cx<T> val = r[e];
            if constexpr (LES) val = val + mul_i(T(g.sx * m1) * t[e]);
            st_compact(o + (long long)(m1 >= 0 ? m1 : m1 + g.Kx) * g.Kz, val, two);
        }
    }
}

// ===========================================================================
// K6: the spectral sweep of the step over the compact state (streaming; every
// load of a mode is issued before any store):
//   src/HIT_LES.cpp:196-242  R = -conv (0 at k=0) - nu k^2 u [- div tau] [+ Coriolis]
//   src/HIT_LES.cpp:243-278  constant-power forcing (when enabled)
//   src/HIT_LES.cpp:295-339  predictor: AB2, or the kappa scheme
//   src/HIT_LES.cpp:346-359  projection  u -= k (k.u)/k^2
// G holds the un-normalised nonlinear term (x1/M^3 here).  Kappa scheme: the
// new state is written over the u^{n-1} buffer Un1 and the caller swaps U/Un1.
// Single precision (T = float) is the compensated form: the states u^n, u^{n-1}
// and u^{n+1} are pairs hi + lo of floats (about 48 significant bits) that this
// sweep combines and splits in double, so the small increments dt*R are not
// rounded away; G and R are plain floats.  In double precision the lo pointers
// are unused (null).
// ===========================================================================
template <typename T, bool SELF>
__device__ __forceinline__ void k6_sweep_body(Geo g, const cx<T> *__restrict__ G, const cx<T> *U, const cx<T> *Ulo, cx<T> *R,
                                              cx<T> *Uout, cx<T> *Uoutlo, const cx<T> *Un1, const cx<T> *Un1lo, const StepConsts &c,
                                              const DevScalars *__restrict__ ds) {
    constexpr bool HILO = sizeof(T) == 4;
    const int iy = blockIdx.y;
    const int n = g.Kx * g.Kz;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const int ix = t / g.Kz, kz = t - ix * g.Kz;
    const long long idx = (long long)iy * n + t;
    const long long S0 = g.S0;
    // loads first
    cx<T> gg[3], uu[3], r0[3], up[3], ul[3], upl[3];
#pragma unroll
    for (int i = 0; i < 3; i++) { gg[i] = G[i * S0 + idx]; uu[i] = U[i * S0 + idx]; r0[i] = R[i * S0 + idx]; }
    if constexpr (HILO) {
#pragma unroll
        for (int i = 0; i < 3; i++) ul[i] = Ulo[i * S0 + idx];
    }
    const double nu = ds->nu, dt = ds->dt, kap = ds->kappa, alpha = ds->alpha;
    const bool first = ds->iter == 0;
    if (SELF) {
#pragma unroll
        for (int i = 0; i < 3; i++) up[i] = first ? uu[i] : Un1[i * S0 + idx];
        if constexpr (HILO) {
#pragma unroll
            for (int i = 0; i < 3; i++) upl[i] = first ? ul[i] : Un1lo[i * S0 + idx];
        }
    }
    const int m1 = ix <= g.hx ? ix : ix - g.Kx, m2 = ky_mode(g, iy);
    const long long k1 = (long long)g.sx * m1, k2 = (long long)g.sy * m2, k3 = (long long)g.sz * kz;
    const double rad2 = (double)(k1 * k1 + k2 * k2 + k3 * k3);
    const bool mean = !(rad2 > 0.0);
    const double ct = nu * rad2;
    double ur[3], ui[3], rr[3], ri[3];
#pragma unroll
    for (int i = 0; i < 3; i++) {
        ur[i] = uu[i].x; ui[i] = uu[i].y;
        if constexpr (HILO) { ur[i] += (double)ul[i].x; ui[i] += (double)ul[i].y; }
        const double gr = mean ? 0.0 : (double)gg[i].x * c.inv_norm;
        const double gi = mean ? 0.0 : (double)gg[i].y * c.inv_norm;
        rr[i] = -gr - ct * ur[i];
        ri[i] = -gi - ct * ui[i];
    }
    if (c.rotating) {
        rr[0] += 2 * (c.omega_z * ur[1] - c.omega_y * ur[2]); ri[0] += 2 * (c.omega_z * ui[1] - c.omega_y * ui[2]);
        rr[1] += 2 * (c.omega_x * ur[2] - c.omega_z * ur[0]); ri[1] += 2 * (c.omega_x * ui[2] - c.omega_z * ui[0]);
        rr[2] += 2 * (c.omega_y * ur[0] - c.omega_x * ur[1]); ri[2] += 2 * (c.omega_y * ui[0] - c.omega_x * ui[1]);
    }
    if (c.eps_on) {
        const int K = (int)round(sqrt(rad2));
        if (c.eps_kmin <= K && K <= c.eps_kmax) {
#pragma unroll
            for (int i = 0; i < 3; i++) { rr[i] += alpha * ur[i]; ri[i] += alpha * ui[i]; }
        } else if (K == 0) {
#pragma unroll
            for (int i = 0; i < 3; i++) { rr[i] = 0.0; ri[i] = 0.0; }
        }
    }
    double sr[3], si[3];
    const double k05 = SELF ? 1.0 / (kap + 0.5) : 0.0;
#pragma unroll
    for (int i = 0; i < 3; i++) {
        if (SELF) {
            double pr = (double)up[i].x, pi = (double)up[i].y;
            if constexpr (HILO) { pr += (double)upl[i].x; pi += (double)upl[i].y; }
            sr[i] = k05 * (2.0 * kap * ur[i] + dt * ((1.0 + kap) * rr[i] - kap * (double)r0[i].x) - (kap - 0.5) * pr);
            si[i] = k05 * (2.0 * kap * ui[i] + dt * ((1.0 + kap) * ri[i] - kap * (double)r0[i].y) - (kap - 0.5) * pi);
        } else {
            sr[i] = ur[i] + dt * (1.5 * rr[i] - 0.5 * (double)r0[i].x);
            si[i] = ui[i] + dt * (1.5 * ri[i] - 0.5 * (double)r0[i].y);
        }
    }
    if (rad2 > 0.0) {
        const double kk[3] = {(double)k1, (double)k2, (double)k3};
        const double inv = 1.0 / rad2;
        const double ar = (kk[0] * sr[0] + kk[1] * sr[1] + kk[2] * sr[2]) * inv;
        const double ai = (kk[0] * si[0] + kk[1] * si[1] + kk[2] * si[2]) * inv;
#pragma unroll
        for (int i = 0; i < 3; i++) { sr[i] -= ar * kk[i]; si[i] -= ai * kk[i]; }
    }
#pragma unroll
    for (int i = 0; i < 3; i++) {
        R[i * S0 + idx] = mk<T>(T(rr[i]), T(ri[i]));
        const T hr = T(sr[i]), hi = T(si[i]);
        Uout[i * S0 + idx] = mk<T>(hr, hi);
        if constexpr (HILO) Uoutlo[i * S0 + idx] = mk<T>(T(sr[i] - (double)hr), T(si[i] - (double)hi));
    }
}

// ===========================================================================
// Small kernels
// ===========================================================================
__device__ __forceinline__ double Topt_d(const StepConsts &c, double phi0, int *err) {
    const double PI_ = 3.141592653589793238462643;
    auto FuL = [](double x, double x0, double x1, double f0, double f1) { return f0 + (x - x0) * (f1 - f0) / (x1 - x0); };
    auto FuG = [&](double x, double a, double b, double cc, double x0, double x1, double f0, double f1) {
        return (a * x * x + b * x + cc) * ((x - x0) * (x - x1)) + FuL(x, x0, x1, f0, f1);
    };
    if (phi0 >= 0.0 && phi0 < c.phi[0]) return FuG(phi0, 0.0, c.c[0], c.c[1], 0.0, c.phi[0], 4.0 / 3.0, c.t1);
    if (phi0 >= c.phi[0] && phi0 <= PI_ / 2.0) return FuG(phi0, c.c[2], c.c[3], c.c[4], c.phi[0], PI_ / 2.0, c.t1, 1.0);
    *err = 1;
    return 0.0;
}
__device__ __forceinline__ double Kopt_d(const StepConsts &c, double phi0, int *err) {
    const double PI_ = 3.141592653589793238462643;
    auto FuL = [](double x, double x0, double x1, double f0, double f1) { return f0 + (x - x0) * (f1 - f0) / (x1 - x0); };
    auto FuG = [&](double x, double a, double b, double cc, double x0, double x1, double f0, double f1) {
        return (a * x * x + b * x + cc) * ((x - x0) * (x - x1)) + FuL(x, x0, x1, f0, f1);
    };
    if (phi0 >= 0.0 && phi0 <= c.phi[0]) return 1.0;
    if (phi0 > c.phi[0] && phi0 <= c.phi[1]) return FuG(phi0, c.c[5], c.c[6], c.c[7], c.phi[0], c.phi[1], 1.0, c.kopt_k[0]);
    if (phi0 > c.phi[1] && phi0 <= c.phi[2]) return FuG(phi0, c.c[8], c.c[9], c.c[10], c.phi[1], c.phi[2], c.kopt_k[0], c.kopt_k[1]);
    if (phi0 > c.phi[2] && phi0 <= PI_ / 2.0) return FuG(phi0, c.c[11], c.c[12], c.c[13], c.phi[2], PI_ / 2.0, c.kopt_k[1], 0.0);
    *err = 1;
    return 0.0;
}

// src/HIT_LES.cpp:365-403, from the maxima gathered by the last inverse transform.
__device__ __forceinline__ void recalc_dt(const StepConsts &c, DevScalars *ds) {
    if (c.fixed_dt > 0.0) { ds->dt = c.fixed_dt; return; }
    const double nu = ds->nu;
    if (c.self_adaptive) {
        const double MaxVel = __longlong_as_double((long long)ds->max_bits[3]);
        ds->maxvel = MaxVel;
        const double Ah = c.Ah;
        const double phi0 = atan(MaxVel * Ah * Ah / (0.35 * nu * 12.0));
        ds->phi0 = phi0;
        int err = 0;
        double At = Topt_d(c, phi0, &err) / sqrt((MaxVel * MaxVel) / (0.35 * 0.35) + (144.0 * nu * nu / (Ah * Ah * Ah * Ah)));
        ds->kappa = Kopt_d(c, phi0, &err);
        if (err) ds->domain_err = 1;
        ds->dt = c.C_At * At;
    } else {
        const double mu = __longlong_as_double((long long)ds->max_bits[0]);
        const double mv = __longlong_as_double((long long)ds->max_bits[1]);
        const double mw = __longlong_as_double((long long)ds->max_bits[2]);
        const double MaxVel = fmax(mu / c.Ax, fmax(mv / c.Ay, mw / c.Az));
        ds->maxvel = MaxVel;
        const double C_visc = 0.2 * fmin(c.Ax * c.Ax, fmin(c.Ay * c.Ay, c.Az * c.Az)) / nu;
        const double C_conv = 0.35 / MaxVel;
        ds->dt = c.C_At * fmin(C_visc, C_conv);
    }
}

static __global__ void k_recalc_dt(StepConsts c, DevScalars *ds) { recalc_dt(c, ds); }

// End of New_Fractional_Step_Method (src/HIT_LES.cpp:19-24).
static __global__ void k_finish_step(StepConsts c, DevScalars *ds) {
    recalc_dt(c, ds);
    ds->time = ds->time + ds->dt;
    ds->iter += 1;
}

// Shell sums of the spectral state (src/HIT_LES.cpp:1137-1214 with the
// KineticEnergy and Enstrophy integrands of :991-1003).  Modes with kz>0 carry
// their conjugate (weight 2).  Ek[K], Om[K] for K=round(|k|) <= Kmax.
// State value hi (+ lo when the compensated single-precision form passes one) in double.
template <typename T> __device__ __forceinline__ cx<double> load_state(const cx<T> *hi, const cx<T> *lo, long long i) {
    const cx<T> a = hi[i];
    cx<double> r = mk<double>((double)a.x, (double)a.y);
    if (lo) { const cx<T> b = lo[i]; r.x += (double)b.x; r.y += (double)b.y; }
    return r;
}

// Adds each lane's e (and o, when hO is given) to the bins hE[K] (hO[K]) in shared
// memory, K < 0 adding nothing.  Called by all 32 lanes with K non-decreasing in the
// lane (consecutive kz of one row): the lanes of one shell are then contiguous,
// a segmented scan over the runs of equal K (five shuffle steps) leaves each run's
// sum in its last lane, and those lanes add to distinct bins in one atomic
// instruction.  (Consecutive kz fall in different shells about every other mode,
// so per-lane atomics would collide on few bins and a loop over the warp's shells
// would run about twenty rounds.)  Lanes out of order only cost extra atomics.
__device__ __forceinline__ void warp_shell_add(int K, double e, double o, double *hE, double *hO) {
    const int lane = threadIdx.x & 31;
    const int Kprev = __shfl_up_sync(0xffffffffu, K, 1);
    const unsigned heads = __ballot_sync(0xffffffffu, lane == 0 || Kprev != K);
    const int start = 31 - __clz(heads & (0xffffffffu >> (31 - lane)));   // first lane of this lane's run
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const double te = __shfl_up_sync(0xffffffffu, e, off);
        const double to = hO ? __shfl_up_sync(0xffffffffu, o, off) : 0.0;
        if (lane - off >= start) { e += te; o += to; }
    }
    const bool tail = lane == 31 || ((heads >> (lane + 1)) & 1u);
    if (tail && K >= 0) {
        atomicAdd(&hE[K], e);
        if (hO) atomicAdd(&hO[K], o);
    }
}

// Walks this warp's share of the compact modes 32 at a time: a contiguous run of whole
// rows (iy, ix), flattened, so that every round but the last is 32 consecutive modes
// (coalesced loads, no idle lanes at the end of a row of Kz modes).  Calls
// f(valid, idx, kz, r12) on all 32 lanes each round, r12 = (sx m1)^2 + (sy m2)^2 of
// the lane's row (recomputed only when the lane enters a new row).  Along a row K
// grows with kz, so a round's lanes form runs of equal K, as warp_shell_add wants.
template <typename F> __device__ __forceinline__ void warp_mode_rounds(const Geo &g, F &&f) {
    const int lane = threadIdx.x & 31;
    const int rows = g.Ky * g.Kx;
    const int nw = (gridDim.x * blockDim.x) >> 5, wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int per = (rows + nw - 1) / nw;
    const int r0 = (int)min((long long)wid * per, (long long)rows), r1 = min(rows, r0 + per);
    const long long end = (long long)r1 * g.Kz;
    int row = r0, kz = lane;
    while (kz >= g.Kz) { kz -= g.Kz; row++; }
    int crow = -1;
    long long r12 = 0;
    for (long long base = (long long)r0 * g.Kz; base < end; base += 32) {
        const long long idx = base + lane;
        const bool valid = idx < end;
        if (valid && row != crow) {
            crow = row;
            const int ix = row % g.Kx, iy = row / g.Kx;
            const long long k1 = (long long)g.sx * (ix <= g.hx ? ix : ix - g.Kx);
            const long long k2 = (long long)g.sy * ky_mode(g, iy);
            r12 = k1 * k1 + k2 * k2;
        }
        f(valid, idx, kz, r12);
        kz += 32;
        while (kz >= g.Kz) { kz -= g.Kz; row++; }
    }
}

// Shell-sum kernels: 256 threads, at most 42 registers, so six blocks fill an SM
// and a grid of SHELL_BLOCKS_PER_SM blocks per SM is one wave.
constexpr int SHELL_BLOCKS_PER_SM = 6;

template <typename T>
__global__ void __launch_bounds__(256, SHELL_BLOCKS_PER_SM) k_shell_sums(Geo g, const cx<T> *__restrict__ u, const cx<T> *__restrict__ v, const cx<T> *__restrict__ w,
                             const cx<T> *__restrict__ ulo, const cx<T> *__restrict__ vlo, const cx<T> *__restrict__ wlo,
                             int Kmax, double *__restrict__ Ek, double *__restrict__ Om) {
    extern __shared__ double hist[];
    double *hE = hist, *hO = hist + (Kmax + 1);
    for (int i = threadIdx.x; i < 2 * (Kmax + 1); i += blockDim.x) hist[i] = 0.0;
    __syncthreads();
    warp_mode_rounds(g, [&](bool valid, long long idx, int kz, long long r12) {
        int K = -1;
        double e = 0.0, o = 0.0;
        if (valid) {
            const long long k3 = (long long)g.sz * kz;
            const double rad2 = (double)(r12 + k3 * k3);
            K = (int)round(sqrt(rad2));
            if (K <= Kmax) {
                const cx<double> a = load_state(u, ulo, idx), b = load_state(v, vlo, idx), cc = load_state(w, wlo, idx);
                e = 0.5 * (a.x * a.x + a.y * a.y + b.x * b.x + b.y * b.y + cc.x * cc.x + cc.y * cc.y);
                if (kz != 0) e *= 2.0;
                o = 2.0 * rad2 * e;
            } else {
                K = -1;
            }
        }
        warp_shell_add(K, e, o, hE, hO);
    });
    __syncthreads();
    for (int i = threadIdx.x; i <= Kmax; i += blockDim.x) {
        if (hE[i] != 0.0) atomicAdd(&Ek[i], hE[i]);
        if (hO[i] != 0.0) atomicAdd(&Om[i], hO[i]);
    }
}

// Shell sums of |F|^2 (conjugate weight 2 for kz>0), scaled by `scale`: the
// spectrum of one scalar field (src/HIT_LES.cpp:1137-1214 with the integrands of
// the invariant spectra, :1006-1025).
template <typename T>
__global__ void __launch_bounds__(256, SHELL_BLOCKS_PER_SM) k_shell_sums_scalar(Geo g, const cx<T> *__restrict__ F, double scale, int Kmax, double *__restrict__ out) {
    extern __shared__ double hist[];
    for (int i = threadIdx.x; i <= Kmax; i += blockDim.x) hist[i] = 0.0;
    __syncthreads();
    warp_mode_rounds(g, [&](bool valid, long long idx, int kz, long long r12) {
        int K = -1;
        double e = 0.0;
        if (valid) {
            const long long k3 = (long long)g.sz * kz;
            K = (int)round(sqrt((double)(r12 + k3 * k3)));
            if (K <= Kmax) {
                const cx<T> a = F[idx];
                e = scale * ((double)a.x * a.x + (double)a.y * a.y);
                if (kz != 0) e *= 2.0;
            } else {
                K = -1;
            }
        }
        warp_shell_add(K, e, 0.0, hist, nullptr);
    });
    __syncthreads();
    for (int i = threadIdx.x; i <= Kmax; i += blockDim.x)
        if (hist[i] != 0.0) atomicAdd(&out[i], hist[i]);
}

// Totals of the shell sums: Ek_Tot over K=0..Kmax, Ok_Tot over K=1..Kmax.
// what: 0 energy only, 1 energy+enstrophy (+ReLambda), 2 Forcing_Reynolds_Lambda.
static __global__ void k_totals(const double *Ek, const double *Om, int Kmax, DevScalars *ds, int what, double relambda) {
    double e = 0.0, o = 0.0;
    for (int K = 0; K <= Kmax; K++) e += Ek[K];
    for (int K = 1; K <= Kmax; K++) o += Om[K];
    ds->ek_tot = e;
    if (what >= 1) ds->ok_tot = o;
    if (what == 1) ds->relambda = e / ds->nu * sqrt(20.0 / 3.0 / o);
    if (what == 2) ds->nu = e / relambda * sqrt(20.0 / 3.0 / o);
}

// Constant-power forcing coefficient alpha = eps/(2 E_f), E_f the energy of
// shells [kmin,kmax] of the current state (src/HIT_LES.cpp:250-256).
// Constant-power forcing amplitude (the disabled block of src/HIT_LES.cpp:243-278,
// with eps as a parameter): alpha = eps / (2 Ef), Ef the energy of the
// shells kmin..kmax of the state (the sum over those shells of the E(K) of k_shell_sums).
// Only modes with |s m| <= kmax + 1 on every axis can round into those shells,
// so one block visits that sub-box directly, in a fixed order with a fixed
// reduction tree: alpha does not depend on timing.  EPS_BAND_THREADS threads.
constexpr int EPS_BAND_THREADS = 256;
// partial (slab decomposition): only the rows this geometry holds are summed and the
// sum goes to ds->ef, for the caller to add up over the slabs and k_eps_alpha to use.
template <typename T>
__global__ void __launch_bounds__(EPS_BAND_THREADS) k_eps_band(Geo g, const cx<T> *__restrict__ u, const cx<T> *__restrict__ v,
                                                               const cx<T> *__restrict__ w, const cx<T> *__restrict__ ulo,
                                                               const cx<T> *__restrict__ vlo, const cx<T> *__restrict__ wlo,
                                                               int kmin, int kmax, double eps, DevScalars *ds, int partial = 0) {
    __shared__ double red[EPS_BAND_THREADS];
    const int mx = min(g.hx, (kmax + 1) / g.sx), my = min(g.hy, (kmax + 1) / g.sy), mz = min(g.hz, (kmax + 1) / g.sz);
    const int nx = 2 * mx + 1, ny = 2 * my + 1, nz = mz + 1;
    const int count = nx * ny * nz;
    double acc = 0.0;
    for (int c = threadIdx.x; c < count; c += EPS_BAND_THREADS) {
        const int kz = c % nz, t = c / nz;
        const int m1 = t % nx - mx, m2 = t / nx - my;
        const int ix = m1 >= 0 ? m1 : m1 + g.Kx, iy = (m2 >= 0 ? m2 : m2 + g.Kyg) - g.y0;
        if (iy < 0 || iy >= g.Ky) continue;   // row held by another slab
        const long long k1 = (long long)g.sx * m1, k2 = (long long)g.sy * m2, k3 = (long long)g.sz * kz;
        const int K = (int)round(sqrt((double)(k1 * k1 + k2 * k2 + k3 * k3)));
        if (K < kmin || K > kmax) continue;
        const long long idx = ((long long)iy * g.Kx + ix) * g.Kz + kz;
        const cx<double> a = load_state(u, ulo, idx), b = load_state(v, vlo, idx), cc = load_state(w, wlo, idx);
        double e = 0.5 * (a.x * a.x + a.y * a.y + b.x * b.x + b.y * b.y + cc.x * cc.x + cc.y * cc.y);
        if (kz != 0) e *= 2.0;
        acc += e;
    }
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int o = EPS_BAND_THREADS / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        const double Ef = red[0];
        if (partial) ds->ef = Ef;
        else ds->alpha = Ef > 1e-30 ? eps / (2.0 * Ef) : 0.0;
    }
}

// alpha from the forced shells' energy summed over the slabs (ds->ef)
static __global__ void k_eps_alpha(double eps, DevScalars *ds) {
    const double Ef = ds->ef;
    ds->alpha = Ef > 1e-30 ? eps / (2.0 * Ef) : 0.0;
}


// src/HIT_LES.cpp:417-419: FT[K] = sqrt(Forced_Ek[K]/Ek[K]).
static __global__ void k_forcing_factors(const double *Ek, const double *Forced, int last_eff, double *FT) {
    for (int K = threadIdx.x; K <= last_eff; K += blockDim.x) FT[K] = Ek[K] > 0.0 ? sqrt(Forced[K] / Ek[K]) : 0.0;
}

// src/HIT_LES.cpp:421-438: scale shells K<=last_eff, optionally zero the rest.
// With lo parts (compensated single precision) the product is formed in double
// and split again into hi + lo.
template <typename T>
__global__ void k_forcing_scale(Geo g, cx<T> *u, cx<T> *v, cx<T> *w, cx<T> *ulo, cx<T> *vlo, cx<T> *wlo, const double *FT,
                                int last_eff, int nullify) {
    const long long n = g.S0;
    for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < n; idx += (long long)gridDim.x * blockDim.x) {
        const int kz = (int)(idx % g.Kz);
        const long long t = idx / g.Kz;
        const int ix = (int)(t % g.Kx), iy = (int)(t / g.Kx);
        const long long k1 = (long long)g.sx * (ix <= g.hx ? ix : ix - g.Kx);
        const long long k2 = (long long)g.sy * ky_mode(g, iy);
        const long long k3 = (long long)g.sz * kz;
        const int K = (int)round(sqrt((double)(k1 * k1 + k2 * k2 + k3 * k3)));
        if (K <= last_eff) {
            if (ulo) {
                cx<T> *hs[3] = {u, v, w}, *ls[3] = {ulo, vlo, wlo};
                for (int i = 0; i < 3; i++) {
                    const cx<double> x = load_state<T>(hs[i], ls[i], idx);
                    const double xr = FT[K] * x.x, xi = FT[K] * x.y;
                    const T hr = T(xr), hi = T(xi);
                    hs[i][idx] = mk<T>(hr, hi);
                    ls[i][idx] = mk<T>(T(xr - (double)hr), T(xi - (double)hi));
                }
            } else {
                const T f = T(FT[K]);
                u[idx] = f * u[idx]; v[idx] = f * v[idx]; w[idx] = f * w[idx];
            }
        } else if (nullify) {
            u[idx] = zero<T>(); v[idx] = zero<T>(); w[idx] = zero<T>();
            if (ulo) { ulo[idx] = zero<T>(); vlo[idx] = zero<T>(); wlo[idx] = zero<T>(); }
        }
    }
}

// src/HIT_LES.cpp:446-476 on the kz=0 plane: u(k1<0 or k1=0,k2<0) = conj(u(-k)).
// The written and the read halves are disjoint, so no staging copy is needed.
template <typename T>
__global__ void k_conj_correction(Geo g, cx<T> *u, cx<T> *v, cx<T> *w, cx<T> *ulo, cx<T> *vlo, cx<T> *wlo) {
    const int n = g.Kx * g.Ky;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        const int ix = t % g.Kx, iy = t / g.Kx;
        const int m1 = ix <= g.hx ? ix : ix - g.Kx, m2 = iy <= g.hy ? iy : iy - g.Ky;
        if (m1 < 0 || (m1 == 0 && m2 < 0)) {
            const int jx = -m1, jy = -m2 >= 0 ? -m2 : -m2 + g.Ky;
            const long long dst = ((long long)iy * g.Kx + ix) * g.Kz, src = ((long long)jy * g.Kx + jx) * g.Kz;
            u[dst] = conj(u[src]); v[dst] = conj(v[src]); w[dst] = conj(w[src]);
            if (ulo) { ulo[dst] = conj(ulo[src]); vlo[dst] = conj(vlo[src]); wlo[dst] = conj(wlo[src]); }
        }
    }
}

// ===========================================================================
// Slab decomposition: reorder of a [nf][n1][n2][Kz] array into per-rank blocks
// [s][f][n1_s][n2_s][Kz] split along axis 1 (rows n1) or 2 (n2) by the ranks'
// block ranges (FFTW-MPI's default block: ceil(n/ranks) per rank), and back.
// Block s starts at off[s] of the staging array; a rank's outgoing blocks are
// contiguous there, in rank order, as an all-to-all sends them.
// ===========================================================================
#define SPNS_SLAB_MAX_RANKS 64
struct SlabRanges {
    int n, blk;                          // ranks, block size of the split axis
    int start[SPNS_SLAB_MAX_RANKS], count[SPNS_SLAB_MAX_RANKS];
    long long off[SPNS_SLAB_MAX_RANKS];  // element offset of rank s's block in the staging array
};
template <typename T>
__global__ void k_slab_pack(cx<T> *__restrict__ full, cx<T> *__restrict__ stage, int nf, int n1, int n2, int Kz, int Kp, SlabRanges r,
                            int axis, int unpack) {
    const long long n = (long long)nf * n1 * n2 * Kz;
    for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < n; idx += (long long)gridDim.x * blockDim.x) {
        const int kz = (int)(idx % Kz);
        long long t = idx / Kz;
        const int i2 = (int)(t % n2);
        t /= n2;
        const int i1 = (int)(t % n1), f = (int)(t / n1);
        const int a = axis == 1 ? i1 : i2;
        const int s = a / r.blk;
        const int loc = a - r.start[s];
        const int n1s = axis == 1 ? r.count[s] : n1, n2s = axis == 1 ? n2 : r.count[s];
        const long long st = r.off[s] + (((long long)f * n1s + (axis == 1 ? loc : i1)) * n2s + (axis == 1 ? i2 : loc)) * Kz + kz;
        const long long fi = idx / Kz * Kp + kz;   // the work buffers' rows have pitch Kp, the staging's are packed
        if (unpack) full[fi] = stage[st];
        else stage[st] = full[fi];
    }
}

// ===========================================================================
// Seeded initial field on the device (no reference counterpart: the reference
// starts from its K41 draw or a file).  Philox4x32-10 (Salmon, Moraes, Dror and
// Shaw, "Parallel random numbers: as easy as 1, 2, 3", SC'11), key = seed,
// counter = (compact mode index, draw number), so every mode draws its own
// numbers and the field does not depend on the launch shape.
// ===========================================================================
struct Philox4 { unsigned x, y, z, w; };
__host__ __device__ __forceinline__ Philox4 philox4x32_10(Philox4 c, unsigned k0, unsigned k1) {
#pragma unroll
    for (int r = 0; r < 10; r++) {
        const unsigned long long p0 = 0xD2511F53ull * c.x, p1 = 0xCD9E8D57ull * c.z;
        Philox4 n;
        n.x = (unsigned)(p1 >> 32) ^ c.y ^ k0;
        n.y = (unsigned)p1;
        n.z = (unsigned)(p0 >> 32) ^ c.w ^ k1;
        n.w = (unsigned)p0;
        c = n;
        k0 += 0x9E3779B9u;
        k1 += 0xBB67AE85u;
    }
    return c;
}

// Two standard normals from one Philox block: two 53-bit uniforms, Box-Muller.
__device__ __forceinline__ void philox_normal2(unsigned long long idx, unsigned draw, unsigned long long seed, double &z0, double &z1) {
    Philox4 c{(unsigned)idx, (unsigned)(idx >> 32), draw, 0u};
    const Philox4 r = philox4x32_10(c, (unsigned)seed, (unsigned)(seed >> 32));
    const double u0 = (double)(((unsigned long long)(r.x >> 5) << 26) | (r.y >> 6)) * 0x1.0p-53;
    const double u1 = (double)(((unsigned long long)(r.z >> 5) << 26) | (r.w >> 6)) * 0x1.0p-53;
    const double rad = sqrt(-2.0 * log(1.0 - u0));
    double sn, cs;
    sincospi(2.0 * u1, &sn, &cs);
    z0 = rad * cs;
    z1 = rad * sn;
}

// Complex Gaussian velocity of every retained mode, projected onto k-perp;
// zero outside |m_i| <= lim_i and at k=0; on kz=0 the half with m1<0 (or
// m1=0, m2<0) is the conjugate of its partner's draw.  Written as the state
// (hi + lo split when lo is given).
template <typename T>
__global__ void k_seed_draw(Geo g, unsigned long long seed, int lim_x, int lim_y, int lim_z, cx<T> *u, cx<T> *v, cx<T> *w,
                            cx<T> *ulo, cx<T> *vlo, cx<T> *wlo) {
    const long long n = g.S0;
    for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < n; idx += (long long)gridDim.x * blockDim.x) {
        const int kz = (int)(idx % g.Kz);
        const long long t = idx / g.Kz;
        const int ix = (int)(t % g.Kx), iy = (int)(t / g.Kx);
        int m1 = ix <= g.hx ? ix : ix - g.Kx, m2 = iy <= g.hy ? iy : iy - g.Ky;
        const double k1 = (double)g.sx * m1, k2 = (double)g.sy * m2, k3 = (double)g.sz * kz;
        const double k2s = k1 * k1 + k2 * k2 + k3 * k3;
        const bool keep = (m1 <= lim_x && -m1 <= lim_x && m2 <= lim_y && -m2 <= lim_y && kz <= lim_z && k2s > 0.0);
        double re[3] = {0.0, 0.0, 0.0}, im[3] = {0.0, 0.0, 0.0};
        if (keep) {
            const bool mirror = kz == 0 && (m1 < 0 || (m1 == 0 && m2 < 0));
            long long src = idx;
            if (mirror) {
                const int p1 = -m1, p2 = -m2;
                src = ((long long)(p2 >= 0 ? p2 : p2 + g.Ky) * g.Kx + (p1 >= 0 ? p1 : p1 + g.Kx)) * g.Kz;
            }
            for (int c = 0; c < 3; c++) philox_normal2((unsigned long long)src, (unsigned)c, seed, re[c], im[c]);
            const double kk[3] = {mirror ? -k1 : k1, mirror ? -k2 : k2, k3};
            const double dr = (kk[0] * re[0] + kk[1] * re[1] + kk[2] * re[2]) / k2s;
            const double di = (kk[0] * im[0] + kk[1] * im[1] + kk[2] * im[2]) / k2s;
            for (int c = 0; c < 3; c++) { re[c] -= dr * kk[c]; im[c] -= di * kk[c]; }
            if (mirror) for (int c = 0; c < 3; c++) im[c] = -im[c];
        }
        cx<T> *hs[3] = {u, v, w}, *ls[3] = {ulo, vlo, wlo};
        for (int c = 0; c < 3; c++) {
            const T hr = T(re[c]), hi = T(im[c]);
            hs[c][idx] = mk<T>(hr, hi);
            if (ulo) ls[c][idx] = mk<T>(T(re[c] - (double)hr), T(im[c] - (double)hi));
        }
    }
}

// Shell factors of the seeded field: target(K) = K^4 exp(-2 (K/kp)^2) on the
// non-empty shells K >= 1, normalised to total energy 3/2 urms^2;
// FT[K] = sqrt(target(K) / E(K)).  One block.
static __global__ void k_seed_factors(const double *Ek, int Kmax, double kp, double urms, double *FT) {
    __shared__ double tot;
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int K = 1; K <= Kmax; K++)
            if (Ek[K] > 0.0) { const double x = (double)K / kp; s += (double)K * K * K * K * exp(-2.0 * x * x); }
        tot = s;
    }
    __syncthreads();
    for (int K = threadIdx.x; K <= Kmax; K += blockDim.x) {
        double f = 0.0;
        if (K >= 1 && Ek[K] > 0.0 && tot > 0.0) {
            const double x = (double)K / kp;
            const double target = (double)K * K * K * K * exp(-2.0 * x * x) * (1.5 * urms * urms) / tot;
            f = sqrt(target / Ek[K]);
        }
        FT[K] = f;
    }
}

// Direct DFT along one axis (initial-field transform of the input file; init only).
// in: complex lines, out: complex lines; out[o][k] = sum_n in[o][n] * w^(k*n mod N).
// Line l of `nl` lines starts at (l / inner)*outer_stride + (l % inner), element stride `es`.
static __global__ void k_dft_axis(const double2 *__restrict__ in, double2 *__restrict__ out, int N, int nk, const int *__restrict__ kidx,
                           long long nl, long long inner, long long in_outer, long long out_outer, long long es_in,
                           long long es_out, const double2 *__restrict__ twN) {
    const long long tot = nl * nk;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < tot; t += (long long)gridDim.x * blockDim.x) {
        const int kk = (int)(t % nk);
        const long long l = t / nk;
        const long long ib = (l / inner) * in_outer + (l % inner), ob = (l / inner) * out_outer + (l % inner);
        const int k = kidx[kk];
        double sr = 0.0, si = 0.0;
        long long m = 0;
        for (int n = 0; n < N; n++) {
            const double2 a = in[ib + n * es_in], wv = twN[m];
            sr += a.x * wv.x - a.y * wv.y;
            si += a.x * wv.y + a.y * wv.x;
            m += k; if (m >= N) m -= N;
        }
        out[ob + (long long)kk * es_out] = make_double2(sr, si);
    }
}

// ===========================================================================
// Kernels of the passes, for one box and for a batch of boxes of the same
// geometry and launch shape.  A batch runs one launch per pass for all its
// members: blockIdx.z selects the member, whose buffers, scalars and constants
// come from a device table (BatchMember).  The arithmetic is the one-box kernel's.
// ===========================================================================
template <typename T, int L, int E, int P, int MODE>
__global__ void __launch_bounds__(P *(L / E), AxisMinBlocks<T, 1, MODE, P *(L / E)>::N) k1_inv_x(Geo g, const SCx<T> *__restrict__ u, const SCx<T> *__restrict__ v,
                                                                           const SCx<T> *__restrict__ w, SCx<T> *__restrict__ out,
                                                                           const cx<T> *__restrict__ tw, DevScalars *reset) {
    if (blockIdx.z == 0) reset_maxima(reset);
    k1_inv_x_body<T, L, E, P, MODE>(g, u, v, w, out, tw, blockIdx.z, gridDim.z);
}
template <typename T, int L, int E, int P, int MODE>
__global__ void __launch_bounds__(P *(L / E), AxisMinBlocks<T, 2, MODE, P *(L / E)>::N) k2_inv_y(Geo g, const SCx<T> *__restrict__ in, SCx<T> *__restrict__ out,
                                                                           const cx<T> *__restrict__ tw) {
    k2_inv_y_body<T, L, E, P, MODE>(g, in, out, tw, blockIdx.z, gridDim.z);
}
template <typename T, int L, int E, int P, int MODE, bool STAGE = false>
__global__ void __launch_bounds__(P *(L / E), K3MinBlocks<T, P *(L / E)>::N) k3_z(Geo g, cx<T> *__restrict__ buf, StepConsts c,
                                                                                        DevScalars *ds, double *__restrict__ phys,
                                                                                        const cx<T> *__restrict__ tw) {
    k3_z_body<T, L, E, P, MODE, STAGE>(g, buf, c, ds, phys, tw);
}
template <typename T, int L, int E, int P, int MODE>
__global__ void __launch_bounds__(P *(L / E), AxisMinBlocks<T, 4, MODE, P *(L / E)>::N) k4_fwd_y(Geo g, const SCx<T> *__restrict__ in, SCx<T> *__restrict__ out,
                                                                           const cx<T> *__restrict__ tw) {
    k4_fwd_y_body<T, L, E, P, MODE>(g, in, out, tw, blockIdx.z, gridDim.z);
}
template <typename T, int L, int E, int P, int MODE>
__global__ void __launch_bounds__(P *(L / E), AxisMinBlocks<T, 5, MODE, P *(L / E)>::N) k5_fwd_x(Geo g, const SCx<T> *__restrict__ in, SCx<T> *__restrict__ G,
                                                                           const cx<T> *__restrict__ tw) {
    k5_fwd_x_body<T, L, E, P, MODE>(g, in, G, tw, blockIdx.z, gridDim.z);
}
template <typename T, bool SELF>
__global__ void __launch_bounds__(256) k6_sweep(Geo g, const cx<T> *__restrict__ G, const cx<T> *U, const cx<T> *Ulo, cx<T> *R, cx<T> *Uout,
                                                cx<T> *Uoutlo, const cx<T> *Un1, const cx<T> *Un1lo, StepConsts c,
                                                const DevScalars *__restrict__ ds) {
    k6_sweep_body<T, SELF>(g, G, U, Ulo, R, Uout, Uoutlo, Un1, Un1lo, c, ds);
}

// One member of a batched launch.  The state is [3][S0] (hi parts; Ulo the
// compensated form's lo parts, else null), R the previous right-hand side, B1/B2
// the S1/S2 work buffers (B2 also holds the nonlinear term after the x pass).
struct BatchMember {
    void *U, *Ulo, *R, *B1, *B2;
    DevScalars *ds;
    StepConsts c;
};
template <typename T, int L, int E, int P, int MODE>
__global__ void __launch_bounds__(P *(L / E), AxisMinBlocks<T, 1, MODE, P *(L / E)>::N) k1_inv_x_batch(Geo g, const BatchMember *__restrict__ tab,
                                                                                 const cx<T> *__restrict__ tw) {
    const BatchMember &m = tab[blockIdx.z];
    reset_maxima(m.ds);
    const SCx<T> *U = static_cast<const SCx<T> *>(m.U);
    k1_inv_x_body<T, L, E, P, MODE>(g, U, U + g.S0, U + 2 * g.S0, static_cast<SCx<T> *>(m.B1), tw, 0, 1);
}
template <typename T, int L, int E, int P, int MODE>
__global__ void __launch_bounds__(P *(L / E), AxisMinBlocks<T, 2, MODE, P *(L / E)>::N) k2_inv_y_batch(Geo g, const BatchMember *__restrict__ tab,
                                                                                 const cx<T> *__restrict__ tw) {
    const BatchMember &m = tab[blockIdx.z];
    k2_inv_y_body<T, L, E, P, MODE>(g, static_cast<const SCx<T> *>(m.B1), static_cast<SCx<T> *>(m.B2), tw, 0, 1);
}
template <typename T, int L, int E, int P, int MODE>
__global__ void __launch_bounds__(P *(L / E), AxisMinBlocks<T, 4, MODE, P *(L / E)>::N) k4_fwd_y_batch(Geo g, const BatchMember *__restrict__ tab,
                                                                                 const cx<T> *__restrict__ tw) {
    const BatchMember &m = tab[blockIdx.z];
    k4_fwd_y_body<T, L, E, P, MODE>(g, static_cast<const SCx<T> *>(m.B2), static_cast<SCx<T> *>(m.B1), tw, 0, 1);
}
template <typename T, int L, int E, int P, int MODE>
__global__ void __launch_bounds__(P *(L / E), AxisMinBlocks<T, 5, MODE, P *(L / E)>::N) k5_fwd_x_batch(Geo g, const BatchMember *__restrict__ tab,
                                                                                 const cx<T> *__restrict__ tw) {
    const BatchMember &m = tab[blockIdx.z];
    k5_fwd_x_body<T, L, E, P, MODE>(g, static_cast<const SCx<T> *>(m.B1), static_cast<SCx<T> *>(m.B2), tw, 0, 1);
}
// Adams-Bashforth members only (the kappa scheme swaps state buffers every step).
template <typename T>
__global__ void __launch_bounds__(256) k6_sweep_batch(Geo g, const BatchMember *__restrict__ tab) {
    const BatchMember &m = tab[blockIdx.z];
    cx<T> *U = static_cast<cx<T> *>(m.U), *Ulo = static_cast<cx<T> *>(m.Ulo);
    k6_sweep_body<T, false>(g, static_cast<const cx<T> *>(m.B2), U, Ulo, static_cast<cx<T> *>(m.R), U, Ulo, nullptr, nullptr, m.c, m.ds);
}
static __global__ void k_finish_step_batch(const BatchMember *__restrict__ tab) {
    const BatchMember &m = tab[blockIdx.x];
    recalc_dt(m.c, m.ds);
    m.ds->time = m.ds->time + m.ds->dt;
    m.ds->iter += 1;
}

} // namespace spns
