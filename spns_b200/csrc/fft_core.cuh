// fft_core.cuh -- register/shared-memory Stockham FFT engine for sm_100a.
//
// One pencil of length L is processed by Q = L/E threads, each holding E
// complex values in registers.  A stage of radix R performs E/R butterflies
// per thread; between stages the values are exchanged through shared memory
// (one buffer, two barriers per stage: before the writes, so that the threads of
// a pencil may drift over a stage's arithmetic, and between writes and reads; the
// last reads of a transform are not followed by one; warp barriers when a pencil lives in
// one warp).  The first stage reads its inputs from registers filled by the
// caller at rows  j + r*(L/R_first)  and the last stage leaves its outputs in
// registers at rows  j + r*(L/R_last)  (j = q + Q*m), so callers load pencils
// straight from global memory and store results straight back (or keep them
// in registers for fused pointwise work).
//
// Stockham autosort, stage (R, Ns): butterfly j, k = j mod Ns,
//   inputs  x_r = in[j + r*L/R],  x_r *= w_L^{r*k*L/(Ns*R)},  y = DFT_R(x),
//   outputs out[(j/Ns)*Ns*R + k + r*Ns] = y_r.
// Radices 2, 3, 4, 6, 8, 12, and 16 in the uneven plan (has_uneven): those with a factor 3 use the
// prime-factor (Good-Thomas) split 2x3 / 4x3, which needs no inner twiddles.
// Twiddles: w^1 of a butterfly is read from a table w_L^m = exp(-2 pi i m/L)
// computed on the host in extended precision.  Stage (R, Ns) needs w_L^{r k L/(Ns R)}
// = w_n^{r k} with n = Ns R and k = j mod Ns; the table carries, after its L base
// entries, a copy w_n^m of the base values for every divisor n < L of L
// (tw_sub_offset), so the lanes of a warp (consecutive k) read consecutive
// entries instead of entries L/n apart: one or two L1 wavefronts per warp load
// instead of up to 32 lines.  The values are the same table entries, so results
// do not change.  In double precision its powers
// w^r are formed by repeated complex multiplication (one table read per
// butterfly instead of R-1: the table reads contend with the shared-memory
// exchange for the load/store pipe); in single precision, where a chain of up
// to 10 products would add ~1e-6 relative error, the powers of two are read
// from the table and every other power is one or two products of them
// (twiddle_powers).  The inverse uses the conjugates.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "fft_layouts.h"

namespace spns {

// Two single-precision values operated on by the packed instructions of sm_100a
// (add/sub/mul/fma.rn.f32x2): lane 0 belongs to one transform, lane 1 to another, so a
// thread runs two single-precision transforms with the instructions of one.  Each lane is
// rounded as the scalar instruction rounds it.  One packed instruction takes the issue
// slot of one scalar one and does the work of two (measured: 130 lanes per clock and SM
// packed, 115-123 scalar, at half the issue slots).
struct f2 {
    unsigned long long v;
    f2() = default;
    __device__ __forceinline__ f2(float a, float b) { asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b)); }
    __device__ __forceinline__ explicit f2(float a) : f2(a, a) {}
    __device__ __forceinline__ explicit f2(double a) : f2((float)a) {}
    __device__ __forceinline__ explicit f2(int a) : f2((float)a) {}
    __device__ __forceinline__ float lo() const { float a; asm("mov.b64 {%0, _}, %1;" : "=f"(a) : "l"(v)); return a; }
    __device__ __forceinline__ float hi() const { float b; asm("mov.b64 {_, %0}, %1;" : "=f"(b) : "l"(v)); return b; }
};
__device__ __forceinline__ f2 operator+(f2 a, f2 b) { f2 r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v)); return r; }
__device__ __forceinline__ f2 operator-(f2 a, f2 b) { f2 r; asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v)); return r; }
__device__ __forceinline__ f2 operator*(f2 a, f2 b) { f2 r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v)); return r; }
__device__ __forceinline__ f2 operator-(f2 a) { f2 r; r.v = a.v ^ 0x8000000080000000ull; return r; }
// a * b + c; the scalar forms leave the contraction to the compiler
__device__ __forceinline__ f2 mad(f2 a, f2 b, f2 c) { f2 r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v)); return r; }
__device__ __forceinline__ float mad(float a, float b, float c) { return a * b + c; }
__device__ __forceinline__ double mad(double a, double b, double c) { return a * b + c; }

// Precision and storage of an arithmetic type: the element type of the arrays in memory,
// and how many of them (columns or pencils) a thread transforms at once.
template <typename T> struct Arith { using S = T; static constexpr int W = 1; static constexpr bool SINGLE = sizeof(T) == 4; };
template <> struct Arith<f2> { using S = float; static constexpr int W = 2; static constexpr bool SINGLE = true; };

template <typename T> struct alignas(2 * sizeof(T)) cx { T x, y; };

template <typename T> __device__ __forceinline__ cx<T> mk(T a, T b) { cx<T> r; r.x = a; r.y = b; return r; }
template <typename T> __device__ __forceinline__ cx<T> operator+(cx<T> a, cx<T> b) { return mk<T>(a.x + b.x, a.y + b.y); }
template <typename T> __device__ __forceinline__ cx<T> operator-(cx<T> a, cx<T> b) { return mk<T>(a.x - b.x, a.y - b.y); }
template <typename T> __device__ __forceinline__ cx<T> operator*(T s, cx<T> a) { return mk<T>(s * a.x, s * a.y); }
// products of packed values: the same two roundings per part as the contracted scalar forms
__device__ __forceinline__ cx<f2> cmul(cx<f2> a, cx<f2> b) { cx<f2> r; r.x = mad(a.x, b.x, a.y * -b.y); r.y = mad(a.x, b.y, a.y * b.x); return r; }
__device__ __forceinline__ cx<f2> cmulc(cx<f2> a, cx<f2> b) { cx<f2> r; r.x = mad(a.x, b.x, a.y * b.y); r.y = mad(a.y, b.x, a.x * -b.y); return r; }
template <typename T> __device__ __forceinline__ cx<T> cmul(cx<T> a, cx<T> b) { return mk<T>(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
template <typename T> __device__ __forceinline__ cx<T> cmulc(cx<T> a, cx<T> b) { return mk<T>(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y); }
template <typename T> __device__ __forceinline__ cx<T> conj(cx<T> a) { return mk<T>(a.x, -a.y); }
// i*a
template <typename T> __device__ __forceinline__ cx<T> mul_i(cx<T> a) { return mk<T>(-a.y, a.x); }
template <typename T> __device__ __forceinline__ cx<T> zero() { return mk<T>(T(0), T(0)); }

// ---------------------------------------------------------------------------
// Radix plan: greedy factors of L from {12, 8, 6, 4, 3, 2}, each dividing E.
// Forward order = greedy order, inverse order = reversed, so the last radix of
// an inverse transform equals the first radix of a forward one (the register
// hand-off between them needs the same row mapping).
// ---------------------------------------------------------------------------
__host__ __device__ constexpr int pick_radix(int rem, int E) {
    return (rem % 12 == 0 && E % 12 == 0) ? 12
         : (rem % 8 == 0 && E % 8 == 0) ? 8
         : (rem % 6 == 0 && E % 6 == 0) ? 6
         : (rem % 4 == 0 && E % 4 == 0) ? 4
         : (rem % 3 == 0 && E % 3 == 0) ? 3
         : (rem % 2 == 0 && E % 2 == 0) ? 2 : 0;
}
__host__ __device__ constexpr int n_stages(int L, int E) {
    int n = 0, rem = L;
    while (rem > 1) { int r = pick_radix(rem, E); if (r == 0) return -1; rem /= r; n++; }
    return n;
}
__host__ __device__ constexpr int greedy_radix(int L, int E, int s) {
    int rem = L;
    for (int i = 0; i < s; i++) rem /= pick_radix(rem, E);
    return pick_radix(rem, E);
}
// Plan with a middle radix that does not divide the values per thread (UNEVEN): 768 = 12 x
// 16 x 4 at 12 values per thread, two exchanges where the greedy plan 12 x 4 x 4 x 4 takes
// three.  48 radix-16 butterflies over 64 threads per pencil leave a quarter of them idle in
// that stage.  For the x/y passes (whole warps idle: inverse x at N=512, double, 4.58 ->
// 4.14 ms); in the z pass, whose threads hold more beside the transform, the 16 values
// spilled (13.0 -> 14.0 ms), and with 384 = 12 x 8 x 4, half of each warp taking a second
// butterfly, it was slower too.  First and last radix, and so the rows of a thread's values,
// are those of the greedy plan.
__host__ __device__ constexpr bool has_uneven(int L, int E) { return L == 768 && E == 12; }
__host__ __device__ constexpr int uneven_radix(int s) { return s == 0 ? 12 : s == 1 ? 16 : 4; }
template <int L, int E, bool INV, bool UNEVEN = false> struct Plan {
    static constexpr int NST = UNEVEN ? 3 : n_stages(L, E);
    static_assert(NST > 0, "length not factorable with radices dividing E");
    static_assert(L % E == 0, "E must divide L");
    static constexpr int Q = L / E;
    __host__ __device__ static constexpr int radix(int s) { 
        const int f = INV ? NST - 1 - s : s;
        return UNEVEN ? uneven_radix(f) : greedy_radix(L, E, f);
    }
    __host__ __device__ static constexpr int ns(int s) { int p = 1; for (int i = 0; i < s; i++) p *= radix(i); return p; }
    // butterflies of stage s, and how many a thread takes at most (the last of them where j < NB)
    __host__ __device__ static constexpr int nb(int s) { return L / radix(s); }
    __host__ __device__ static constexpr int mb(int s) { return (nb(s) + Q - 1) / Q; }
    // values a thread holds at most
    __host__ __device__ static constexpr int width() {
        int v = E;
        for (int s = 0; s < NST; s++) v = mb(s) * radix(s) > v ? mb(s) * radix(s) : v;
        return v;
    }
    static_assert(nb(0) % Q == 0 && nb(NST - 1) % Q == 0, "the first and last stage are even");
    static constexpr int R_first = radix(0);
    static constexpr int R_last = radix(NST - 1);
};

// ---------------------------------------------------------------------------
// Small DFTs (in place); INV selects exp(+2*pi*i/R).
// ---------------------------------------------------------------------------
template <typename T, bool INV> __device__ __forceinline__ void dft2(cx<T> *x) {
    cx<T> a = x[0], b = x[1];
    x[0] = a + b; x[1] = a - b;
}
template <typename T, bool INV> __device__ __forceinline__ void dft3(cx<T> *x) {
    const T c3 = T(-0.5);
    const T s3 = INV ? T(0.86602540378443864676372317075294) : T(-0.86602540378443864676372317075294);
    const T n3 = INV ? T(-0.86602540378443864676372317075294) : T(0.86602540378443864676372317075294);
    cx<T> s = x[1] + x[2], d = x[1] - x[2];
    cx<T> y0 = x[0] + s;
    cx<T> m = mk<T>(mad(c3, s.x, x[0].x), mad(c3, s.y, x[0].y));
    x[0] = y0;
    x[1] = mk<T>(mad(n3, d.y, m.x), mad(s3, d.x, m.y));
    x[2] = mk<T>(mad(s3, d.y, m.x), mad(n3, d.x, m.y));
}
template <typename T, bool INV> __device__ __forceinline__ void dft4(cx<T> *x) {
    cx<T> t0 = x[0] + x[2], t1 = x[0] - x[2], t2 = x[1] + x[3], t3 = x[1] - x[3];
    // x1, x3 = t1 +- (+/-i) t3
    const cx<T> a = mk<T>(t1.x - t3.y, t1.y + t3.x), b = mk<T>(t1.x + t3.y, t1.y - t3.x);
    x[0] = t0 + t2; x[2] = t0 - t2; x[1] = INV ? a : b; x[3] = INV ? b : a;
}
template <typename T, bool INV> __device__ __forceinline__ void dft8(cx<T> *x) {
    const T h = T(0.70710678118654752440084436210485);
    cx<T> e[4] = {x[0], x[2], x[4], x[6]}, o[4] = {x[1], x[3], x[5], x[7]};
    dft4<T, INV>(e); dft4<T, INV>(o);
    // w8^k for k=1..3: forward exp(-i*pi*k/4)
    const T n = T(-0.70710678118654752440084436210485);
    cx<T> o1 = INV ? mk<T>(h * (o[1].x - o[1].y), h * (o[1].x + o[1].y)) : mk<T>(h * (o[1].x + o[1].y), h * (o[1].y - o[1].x));
    cx<T> o3 = INV ? mk<T>(n * (o[3].x + o[3].y), h * (o[3].x - o[3].y)) : mk<T>(h * (o[3].y - o[3].x), n * (o[3].x + o[3].y));
    // x2, x6 = e2 +- (+/-i) o2
    const cx<T> a = mk<T>(e[2].x - o[2].y, e[2].y + o[2].x), b = mk<T>(e[2].x + o[2].y, e[2].y - o[2].x);
    x[0] = e[0] + o[0]; x[4] = e[0] - o[0];
    x[1] = e[1] + o1;   x[5] = e[1] - o1;
    x[2] = INV ? a : b; x[6] = INV ? b : a;
    x[3] = e[3] + o3;   x[7] = e[3] - o3;
}
// Twiddles and 16-point DFT of one butterfly: x[r] times w^r, then 16 points as 4 x 4.  With
// r = 4 n1 + n2 the factor w^(4 n1) goes before the DFT4 of column n2 and w^(n2), joined with
// the inner twiddle w16^(n2 k1), after it: the multipliers of a column or a row are few and
// short-lived, where the fifteen powers of one pass over x spilled.  w1, w2, w4, w8: powers of
// the forward twiddle.
template <typename T, bool INV> __device__ __forceinline__ void dft16_tw(cx<T> *x, cx<T> w1, cx<T> w2, cx<T> w4, cx<T> w8) {
    const T c1 = T(0.92387953251128675612818318939679), s1 = T(0.38268343236508977172845998403040);   // cos, sin of pi/8
    const T n_s1 = T(-0.38268343236508977172845998403040), n_c1 = T(-0.92387953251128675612818318939679);
    const T h = T(0.70710678118654752440084436210485), n_h = T(-0.70710678118654752440084436210485);
    auto mul = [](cx<T> a, cx<T> w) { return INV ? cmulc(a, w) : cmul(a, w); };
    {
        const cx<T> w12 = cmul(w8, w4);
#pragma unroll
        for (int n2 = 0; n2 < 4; n2++) {
            cx<T> c[4] = {x[n2], mul(x[4 + n2], w4), mul(x[8 + n2], w8), mul(x[12 + n2], w12)};
            dft4<T, INV>(c);
#pragma unroll
            for (int k1 = 0; k1 < 4; k1++) x[4 * k1 + n2] = c[k1];
        }
    }
    const cx<T> w3 = cmul(w2, w1);
    // w times w16^m (forward) = (c - i s), given c, s, -s
    auto rot = [](cx<T> w, T c, T sn, T ns) { return mk<T>(mad(w.x, c, w.y * sn), mad(w.y, c, w.x * ns)); };
    cx<T> y[16];
#pragma unroll
    for (int k1 = 0; k1 < 4; k1++) {
        cx<T> m1 = w1, m2 = w2, m3 = w3;
        if (k1 == 1) { m1 = rot(w1, c1, s1, n_s1); m2 = rot(w2, h, h, n_h); m3 = rot(w3, s1, c1, n_c1); }
        else if (k1 == 2) { m1 = rot(w1, h, h, n_h); m2 = mk<T>(w2.y, -w2.x); m3 = rot(w3, n_h, h, n_h); }
        else if (k1 == 3) { m1 = rot(w1, s1, c1, n_c1); m2 = rot(w2, n_h, h, n_h); m3 = rot(w3, n_c1, n_s1, s1); }
        cx<T> c[4] = {x[4 * k1], mul(x[4 * k1 + 1], m1), mul(x[4 * k1 + 2], m2), mul(x[4 * k1 + 3], m3)};
        dft4<T, INV>(c);
#pragma unroll
        for (int k2 = 0; k2 < 4; k2++) y[k1 + 4 * k2] = c[k2];
    }
#pragma unroll
    for (int r = 0; r < 16; r++) x[r] = y[r];
}
// Good-Thomas split of R = A*B (gcd 1): input n = (B a + A b) mod R, output
// k with k = ka (mod A), k = kb (mod B); DFT_A over a, then DFT_B over b.
template <int A, int B> struct PFA {
    static constexpr int R = A * B;
    __host__ __device__ static constexpr int in(int a, int b) { return (B * a + A * b) % R; }
    __host__ __device__ static constexpr int out(int ka, int kb) {
        int invB = 1;
        while ((B * invB) % A != 1 % A) invB++;
        int invA = 1;
        while ((A * invA) % B != 1 % B) invA++;
        return (ka * B * invB + kb * A * invA) % R;
    }
};
template <typename T, bool INV, int A, int B> __device__ __forceinline__ void dft_pfa(cx<T> *x) {
    using P = PFA<A, B>;
    cx<T> t[A * B];
#pragma unroll
    for (int b = 0; b < B; b++) {
        cx<T> col[A];
#pragma unroll
        for (int a = 0; a < A; a++) col[a] = x[P::in(a, b)];
        if constexpr (A == 2) dft2<T, INV>(col);
        else if constexpr (A == 4) dft4<T, INV>(col);
        else dft8<T, INV>(col);
#pragma unroll
        for (int a = 0; a < A; a++) t[a * B + b] = col[a];
    }
#pragma unroll
    for (int ka = 0; ka < A; ka++) {
        cx<T> row[B];
#pragma unroll
        for (int b = 0; b < B; b++) row[b] = t[ka * B + b];
        dft3<T, INV>(row);
#pragma unroll
        for (int kb = 0; kb < B; kb++) x[P::out(ka, kb)] = row[kb];
    }
}
template <typename T, int R, bool INV> __device__ __forceinline__ void dft(cx<T> *x) {
    if constexpr (R == 2) dft2<T, INV>(x);
    else if constexpr (R == 3) dft3<T, INV>(x);
    else if constexpr (R == 4) dft4<T, INV>(x);
    else if constexpr (R == 6) dft_pfa<T, INV, 2, 3>(x);
    else if constexpr (R == 8) dft8<T, INV>(x);
    else if constexpr (R == 12) dft_pfa<T, INV, 4, 3>(x);
}

// ---------------------------------------------------------------------------
// Stage engine.  SM is a shared-memory accessor:  cx<T>& SM::at(int row).
// v[m*R + r] holds the input (before the stage) / output (after) of butterfly
// j = q + Q*m, leg r.  WARP: the threads of a pencil exchange within one warp.
// ---------------------------------------------------------------------------
template <class SM, class = void> struct SmPadded { static constexpr bool value = false; };
template <class SM> struct SmPadded<SM, decltype((void)SM::PADDED)> { static constexpr bool value = SM::PADDED; };
// layout of exchange S of a padded accessor (pad >= 0, or -1 for the XOR swizzle); 0 for the others
template <class SM, bool INV, int S> __host__ __device__ constexpr int ex_pad() {
    if constexpr (SmPadded<SM>::value) return SM::template Ex<INV, S>::PAD;
    else return 0;
}

// accessors whose transforms take the uneven plan where there is one
template <class SM, int L, int E> __host__ __device__ constexpr bool uneven_plan() { return has_uneven(L, E) && !SmPadded<SM>::value; }

// Offset of the sub-table w_n^m (m < n) in a twiddle table of length L: 0 for
// n = L (the base table), else L plus the sizes of the sub-tables of the divisors
// of L below n (spns_make_twiddles lays them out in increasing n).
__host__ __device__ constexpr int tw_sub_offset(int L, int n) {
    if (n >= L) return 0;
    int off = L;
    for (int d = 2; d < n; d++)
        if (L % d == 0) off += d;
    return off;
}
// Entries of a twiddle table of length L with all its sub-tables.
__host__ __device__ constexpr int tw_table_size(int L) {
    int s = L;
    for (int d = 2; d < L; d++)
        if (L % d == 0) s += d;
    return s;
}
// Single precision reads the powers of two of a butterfly's twiddle; w_n^{r k} for
// r = 2, 4, 8 sits in a power table of its own (n entries, k contiguous) so that those
// reads are contiguous across a warp too.  Three power tables follow the sub-tables,
// each holding every divisor n >= 2 of L (L included) in increasing n.
__host__ __device__ constexpr int tw_pow_offset(int L, int n, int r) {
    const int ri = r == 2 ? 0 : r == 4 ? 1 : 2;
    int off = tw_table_size(L) * (1 + ri);
    for (int d = 2; d < n; d++)
        if (L % d == 0) off += d;
    return off;
}
__host__ __device__ constexpr int tw_full_size(int L) { return 4 * tw_table_size(L); }

// Barrier of an exchange: the block's (WARP 0), the whole warp's (1), that of the warps of an
// aligned group of 64, 96 or 128 threads (GROUP + threads: named barrier 1 + group), or that of the
// lanes of the mask WARP, the only ones that run the transform.
constexpr unsigned GROUP = 0x40000000u;
template <unsigned WARP> __device__ __forceinline__ void stage_barrier() {
    if constexpr (WARP == 0) __syncthreads();
    else if constexpr (WARP == 1) __syncwarp();
    else if constexpr (WARP == GROUP + 64 || WARP == GROUP + 96 || WARP == GROUP + 128)
        asm volatile("bar.sync %0, %1;\n" ::"r"(1 + threadIdx.x / (WARP - GROUP)), "n"(WARP - GROUP) : "memory");
    else __syncwarp(WARP);
}

// Single precision: the powers w^r of a butterfly's twiddle.  With SPNS_F32_TW_POW the
// powers of two come from the table and the others are one or two products of
// them (w^3 = w^2 w, w^7 = w^4 w^3, ...; about 2e-7 relative error at most), which
// reads 4 instead of 11 table entries for a radix-12 butterfly; without it every
// power is read.  At N=512 the single-precision z pass took 10.31 ms against 11.89.
#ifndef SPNS_F32_TW_POW
#define SPNS_F32_TW_POW 1
#endif
template <typename T, int R>
__device__ __forceinline__ void twiddle_powers(cx<T> (&wp)[R], const cx<T> *__restrict__ tw, int step) {
#pragma unroll
    for (int r = 1; r < R; r++) {
        if (!SPNS_F32_TW_POW || (r & (r - 1)) == 0) {
            wp[r] = tw[r * step];
        } else {
            int hb = 1;
            while (hb * 2 <= r) hb *= 2;
            wp[r] = cmul(wp[hb], wp[r - hb]);
        }
    }
}

template <typename T, int L, int E, bool INV, unsigned WARP, int S, class SM>
__device__ __forceinline__ void fft_run(cx<T> (&v)[Plan<L, E, INV, uneven_plan<SM, L, E>()>::width()], SM sm, int q, const cx<T> *__restrict__ tw) {
    using PL = Plan<L, E, INV, uneven_plan<SM, L, E>()>;
    constexpr int R = PL::radix(S);
    constexpr int Ns = PL::ns(S);
    constexpr int Q = PL::Q;
    constexpr int NB = PL::nb(S), MB = PL::mb(S);
#pragma unroll
    for (int m = 0; m < MB; m++) {
        if (NB % Q != 0 && q + Q * m >= NB) continue;
        if constexpr (Ns > 1) {
            const int j = q + Q * m;
            const int k = j % Ns;                  // w^r = w_n^{r k}, n = Ns R, r k < n
            constexpr int TWO = tw_sub_offset(L, Ns * R);
            const cx<T> *__restrict__ twn = tw + TWO;
            if constexpr (R == 16) {
                constexpr int P2 = tw_pow_offset(L, Ns * R, 2), P4 = tw_pow_offset(L, Ns * R, 4), P8 = tw_pow_offset(L, Ns * R, 8);
                const cx<T> w1 = twn[k];
                if constexpr (Arith<T>::SINGLE) {
                    dft16_tw<T, INV>(&v[m * R], w1, tw[P2 + k], tw[P4 + k], tw[P8 + k]);
                } else {
                    const cx<T> w2 = cmul(w1, w1), w4 = cmul(w2, w2);
                    dft16_tw<T, INV>(&v[m * R], w1, w2, w4, cmul(w4, w4));
                }
                continue;
            } else if constexpr (Arith<T>::SINGLE) {
                cx<T> wp[R];
                if constexpr (SPNS_F32_TW_POW) {
                    constexpr int P2 = tw_pow_offset(L, Ns * R, 2), P4 = tw_pow_offset(L, Ns * R, 4),
                                  P8 = tw_pow_offset(L, Ns * R, 8);
                    wp[1] = twn[k];
#pragma unroll
                    for (int r = 2; r < R; r++) {
                        if (r == 2) wp[r] = tw[P2 + k];
                        else if (r == 4) wp[r] = tw[P4 + k];
                        else if (r == 8) wp[r] = tw[P8 + k];
                        else {
                            int hb = 1;
                            while (hb * 2 <= r) hb *= 2;
                            wp[r] = cmul(wp[hb], wp[r - hb]);
                        }
                    }
                } else {
                    twiddle_powers<T, R>(wp, twn, k);
                }
#pragma unroll
                for (int r = 1; r < R; r++) v[m * R + r] = INV ? cmulc(v[m * R + r], wp[r]) : cmul(v[m * R + r], wp[r]);
            } else {
                const cx<T> w1 = twn[k];
                cx<T> w = w1;
#pragma unroll
                for (int r = 1; r < R; r++) {
                    v[m * R + r] = INV ? cmulc(v[m * R + r], w) : cmul(v[m * R + r], w);
                    if (r + 1 < R) w = cmul(w, w1);
                }
            }
        }
        dft<T, R, INV>(&v[m * R]);
    }
    if constexpr (S + 1 < PL::NST) {
        constexpr int R2 = PL::radix(S + 1);
        constexpr int NB2 = PL::nb(S + 1), MB2 = PL::mb(S + 1);
        // every reader of the buffer's last contents is done (waited for here, after this
        // stage's arithmetic, rather than right after the reads)
        stage_barrier<WARP>();
        if constexpr (ex_pad<SM, INV, S>() < 0) {
            // XOR-swizzled layout (fewer bank conflicts for this exchange)
#pragma unroll
            for (int m = 0; m < MB; m++) {
                if (NB % Q != 0 && q + Q * m >= NB) continue;
                const int j = q + Q * m;
                const int base = (j / Ns) * Ns * R + (j % Ns);
#pragma unroll
                for (int r = 0; r < R; r++) sm.xr(base + r * Ns) = v[m * R + r];
            }
            stage_barrier<WARP>();
#pragma unroll
            for (int m = 0; m < MB2; m++) {
                if (NB2 % Q != 0 && q + Q * m >= NB2) continue;
                const int j = q + Q * m;
#pragma unroll
                for (int r = 0; r < R2; r++) v[m * R2 + r] = sm.xr(j + r * (L / R2));
            }
        } else if constexpr (SmPadded<SM>::value) {
            // padded layout: one base address per butterfly group, offsets in the instructions
            constexpr int X = Ns * R, PAD = SM::template Ex<INV, S>::PAD, XP = X + PAD;
            cx<T> *const b = sm.base;
#pragma unroll
            for (int m = 0; m < MB; m++) {
                if (NB % Q != 0 && q + Q * m >= NB) continue;
                cx<T> *w;
                if constexpr (Q % Ns == 0) {
                    w = b + (q / Ns) * XP + (q % Ns) + m * (Q / Ns) * XP;
                } else {
                    const int j = q + Q * m, hi = j / Ns;
                    w = b + hi * XP + (j - hi * Ns);
                }
#pragma unroll
                for (int r = 0; r < R; r++) w[r * Ns] = v[m * R + r];
            }
            stage_barrier<WARP>();
            constexpr int STEP = L / R2, PSTEP = STEP + (STEP / X) * PAD;
            static_assert(STEP % X == 0, "exchange read stride must be a multiple of the pad block");
#pragma unroll
            for (int m = 0; m < MB2; m++) {
                if (NB2 % Q != 0 && q + Q * m >= NB2) continue;
                const cx<T> *rd;
                if constexpr (Q % X == 0) {
                    rd = b + q + (q / X) * PAD + m * (Q + (Q / X) * PAD);
                } else {
                    const int row = q + Q * m;
                    rd = b + row + (row / X) * PAD;
                }
#pragma unroll
                for (int r = 0; r < R2; r++) v[m * R2 + r] = rd[r * PSTEP];
            }
        } else {
#pragma unroll
            for (int m = 0; m < MB; m++) {
                if (NB % Q != 0 && q + Q * m >= NB) continue;
                const int j = q + Q * m;
                const int base = (j / Ns) * Ns * R + (j % Ns);
#pragma unroll
                for (int r = 0; r < R; r++) sm.at(base + r * Ns) = v[m * R + r];
            }
            stage_barrier<WARP>();
#pragma unroll
            for (int m = 0; m < MB2; m++) {
                if (NB2 % Q != 0 && q + Q * m >= NB2) continue;
                const int j = q + Q * m;
#pragma unroll
                for (int r = 0; r < R2; r++) v[m * R2 + r] = sm.at(j + r * (L / R2));
            }
        }
        fft_run<T, L, E, INV, WARP, S + 1, SM>(v, sm, q, tw);
    }
}

// Row of register slot e before the first stage (inputs) / after the last stage (outputs).
template <int L, int E, bool INV> __device__ __forceinline__ int in_row(int q, int e) {
    using PL = Plan<L, E, INV>;
    constexpr int R = PL::R_first;
    return q + PL::Q * (e / R) + (e % R) * (L / R);
}
template <int L, int E, bool INV> __device__ __forceinline__ int out_row(int q, int e) {
    using PL = Plan<L, E, INV>;
    constexpr int R = PL::R_last;
    return q + PL::Q * (e / R) + (e % R) * (L / R);
}

// Opaque copy of an index: the row and address arithmetic that depends on it is
// recomputed where it is used instead of being hoisted out of a loop over fields or
// pencils and kept live in registers for every register slot.
__device__ __forceinline__ int opaque(int q) {
    int r;
    asm volatile("mov.b32 %0, %1;" : "=r"(r) : "r"(q));
    return r;
}

// The thread index goes through an opaque move so that the shared-memory
// addresses of the stages are recomputed per transform instead of being kept
// live across every transform of a kernel (which exhausts the register file).
// WARP=true only where each pencil's threads lie in one warp (Q divides 32 in a
// pencil-major thread layout).
template <typename T, int L, int E, bool INV, class SM, unsigned WARP = 0>
__device__ __forceinline__ void fft(cx<T> (&v)[E], SM sm, int q, const cx<T> *__restrict__ tw) {
    constexpr int V = Plan<L, E, INV, uneven_plan<SM, L, E>()>::width();
    if constexpr (V == E) {
        fft_run<T, L, E, INV, WARP, 0, SM>(v, sm, opaque(q), tw);
    } else {
        cx<T> x[V];
#pragma unroll
        for (int e = 0; e < E; e++) x[e] = v[e];
        fft_run<T, L, E, INV, WARP, 0, SM>(x, sm, opaque(q), tw);
#pragma unroll
        for (int e = 0; e < E; e++) v[e] = x[e];
    }
}

// Accessor: tile of P pencils stored row-major [row][P] (pencil index fastest).
template <typename T, int P> struct SmRowMajor {
    cx<T> *base; int p;
    __device__ __forceinline__ cx<T> &at(int row) const { return base[row * P + p]; }
};
// Accessor: pencil-major [p][PITCH], rows stored in order (post-processing
// reads rows k and L-k of consecutive k: conflict-free as is).  The Stockham
// exchanges of fft_run use their own padded layouts inside the same buffer
// (PencilLayout below), so `at` is only for accesses outside the transform.
template <typename T, int L, int E> struct SmPencil;

// ---------------------------------------------------------------------------
// Padded exchange layouts of the pencil-major buffer.
//
// Exchange S (written by stage S: radix R, span Ns; read by stage S+1: radix
// R2) stores row r at  r + (r / X) * PAD  with X = Ns*R.  A butterfly's R
// writes  (j/Ns)*X + j%Ns + r*Ns  all lie in one block of X rows, and the
// reads  q + Q*m + r2*(L/R2)  step by multiples of X (L/R2 = X * the radices
// after S+1), so every access of a thread is one base address plus
// compile-time offsets: no per-access index arithmetic.  PAD per exchange and
// the pencil pitch come from fft_layouts.h, generated by gen_layouts.py, which
// counts the shared-memory wavefronts of each exchange's writes and reads; where
// the XOR swizzle below has fewer, the table selects it (PAD = -1) and that
// exchange pays per-access index arithmetic instead.
// ---------------------------------------------------------------------------
template <typename T, int L, int E> struct SmPencil {
    cx<T> *base;
    static constexpr bool PADDED = true;
    static constexpr int WPL = (int)(sizeof(cx<T>) / 4);
    static constexpr int PITCH = exch::table_pitch(WPL, L, E);
    static_assert(PITCH >= L, "no exchange layout generated for this length and E (gen_layouts.py)");
    static constexpr int G = WPL == 4 ? 8 : 16;   // rows of one 128-byte bank line
    // layout of exchange S of the inverse (INV) or forward plan: pad >= 0, or -1 for the XOR swizzle
    template <bool INV, int S> struct Ex {
#ifdef SPNS_EXCH_XOR_ONLY
        static constexpr int PAD = -1;
#else
        static constexpr int PAD = exch::table_pad(WPL, L, E, INV, S);
#endif
        static_assert(PAD >= -1, "no exchange layout generated for this stage (gen_layouts.py)");
        static_assert((PAD < 0 ? (L + G - 1) / G * G : L + (L / (Plan<L, E, INV>::ns(S) * Plan<L, E, INV>::radix(S))) * PAD) <= PITCH,
                      "exchange layout exceeds the pencil pitch");
    };
    __device__ __forceinline__ cx<T> &at(int row) const { return base[row]; }
    // XOR swizzle of the low row bits by the bits two places up; maps each aligned block of G rows onto itself
    __device__ __forceinline__ cx<T> &xr(int row) const { return base[row ^ ((row >> 2) & (G - 1))]; }
};

} // namespace spns
