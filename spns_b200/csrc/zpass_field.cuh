// zpass_field.cuh -- the z pass with the fields of a pencil transformed side by side
// and the physical values of the pencil held in shared memory.
//
// Same arithmetic as the z pass of the reference's step (src/HIT_LES.cpp:74-171): c2r of
// the real fields two per complex transform (inverse pairs), pointwise products on the
// grid, r2c of the products two per transform (forward jobs), truncated to kz <= hz.
//
// A block owns PB pencils and has NT teams of Q = L/E threads.  Every inverse pair of a
// pencil has a complex exchange buffer of its own, so the teams transform different pairs
// at the same time and a pair's two real fields stay in its buffer, row by row, as the
// physical slots of the pencil.  Then all threads of the block form the products row by
// row (each row is read and written by one thread, so the jobs' inputs go over the pairs'
// values in place), and the teams transform the jobs out of the same buffers.  Between the
// three parts is one block barrier; inside a transform only the warp synchronises
// (Q <= 32; where Q does not divide 32 a warp has 32/Q teams and idle lanes).
//
// What bounds it: a thread holds one array of E values and no slots, so registers no
// longer limit the pass to 8 (double) or 12 (single precision) warps per SM as they did
// with up to 12 slots per grid row in the thread that owns the row; what is left is the
// shared-memory traffic of the exchanges, and E = 24 plans (one exchange less) fit.
//
// Blocks walk the groups of PB pencils (LenLaunch::walking_blocks), so the CFL maxima are
// reduced once per block.
#pragma once
#include "solver_kernels.cuh"

namespace spns {

// Inverse pairs and forward jobs per form.
template <int MODE> struct ZFieldForm {
    static_assert(MODE == MODE_ADV || MODE == MODE_LES || MODE == MODE_INV, "the rotational form runs in k3_rot_staged or k3_z");
    static constexpr int NPAIR = MODE == MODE_INV ? 5 : 6;
    static constexpr int NJOB = MODE == MODE_LES ? 5 : MODE == MODE_INV ? 3 : 2;
};

// S2 fields of inverse pair p and whether each enters as its z derivative (b < 0: none).
//   ADV, LES  (u, v), (w, du/dz), (du/dx, du/dy), (dv/dx, dv/dy), (dw/dx, dw/dy), (dv/dz, dw/dz)
//   INV  (du/dx, du/dy), (dv/dx, dv/dy), (dw/dx, dw/dy), (du/dz, dv/dz), (dw/dz, -)
struct ZPair { int a, b; bool da, db; };
template <int MODE> __device__ __forceinline__ ZPair zfield_pair(int p) {
    if constexpr (MODE == MODE_INV) return p < 3 ? ZPair{3 + p, 6 + p, false, false} : p == 3 ? ZPair{0, 1, true, true} : ZPair{2, -1, true, false};
    else return ZPair{p == 0 ? 0 : p == 1 ? 2 : p == 5 ? 1 : p + 1, p == 0 ? 1 : p == 1 ? 0 : p == 5 ? 2 : p + 4, p == 5, p == 1 || p == 5};
}

// Outputs of forward job j (S2 fields; b < 0: none).  fold: a += i kz b (SGS divergence);
// single: one real field, stored without the separation of a pair.
struct ZJob { int a, b; bool fold, single; };
template <int MODE> __device__ __forceinline__ ZJob zfield_job(int j) {
    if constexpr (MODE == MODE_ADV) return j == 0 ? ZJob{0, 1, false, false} : ZJob{2, -1, false, true};
    else if constexpr (MODE == MODE_INV) return j < 2 ? ZJob{2 * j, 2 * j + 1, false, false} : ZJob{4, -1, false, true};
    // 0 G_x = conv_x + i kz t13, 1 G_y, 2 G_z, 3 t11, 4 t12, 5 t13, 6 t22, 7 t23
    else return j == 0 ? ZJob{0, 5, true, false} : j == 1 ? ZJob{1, 7, true, false} : j == 2 ? ZJob{2, -1, true, false}
              : j == 3 ? ZJob{3, 4, false, false} : ZJob{6, -1, false, true};
}

// Products of one grid row: v[p] holds the two real fields of pair p on entry and the two
// real inputs of job p on return.
template <typename T, int MODE>
__device__ __forceinline__ void zfield_row(cx<T> (&v)[ZFieldForm<MODE>::NPAIR], const StepConsts &c, double (&mx)[4], double (&nut)[3]) {
    if constexpr (MODE == MODE_INV) {
        // Invariants of G_ij = d_j u_i (src/HIT_LES.cpp:1297-1319, definitions
        // src/tensor_algebra.cpp:165-306, 356-358) and the eddy-viscosity statistics, in double.
        double G[3][3], S[3][3], O[3][3];
        G[0][0] = v[0].x; G[0][1] = v[0].y; G[0][2] = v[3].x;
        G[1][0] = v[1].x; G[1][1] = v[1].y; G[1][2] = v[3].y;
        G[2][0] = v[2].x; G[2][1] = v[2].y; G[2][2] = v[4].x;
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int j = 0; j < 3; j++) { S[i][j] = 0.5 * G[i][j] + 0.5 * G[j][i]; O[i][j] = G[i][j] - S[i][j]; }
        const double trG = G[0][0] + G[1][1] + G[2][2], trS = S[0][0] + S[1][1] + S[2][2];
        double trGG = 0.0, trSS = 0.0, trS2O2 = 0.0;
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int j = 0; j < 3; j++) {
                trGG += G[i][j] * G[j][i];
                trSS += S[i][j] * S[j][i];
            }
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int k = 0; k < 3; k++) {
                double s2 = 0.0, o2 = 0.0;
#pragma unroll
                for (int l = 0; l < 3; l++) { s2 += S[i][l] * S[l][k]; o2 += O[k][l] * O[l][i]; }
                trS2O2 += s2 * o2;
            }
        auto det3 = [](const double (&t)[3][3]) {
            double d = 0.0;
            d += t[0][0] * t[1][1] * t[2][2];
            d += t[0][1] * t[1][2] * t[2][0];
            d += t[0][2] * t[1][0] * t[2][1];
            d -= t[0][2] * t[1][1] * t[2][0];
            d -= t[0][1] * t[1][0] * t[2][2];
            d -= t[0][0] * t[1][2] * t[2][1];
            return d;
        };
        const double QG = 0.5 * (trG * trG - trGG), QS = 0.5 * (trS * trS - trSS);
        // eddy viscosity of this grid point (src/HIT_LES.cpp:130-142, same expression order)
        double ne = 2.0 * G[0][0] * G[0][0];
        ne += 2.0 * G[1][1] * G[1][1];
        ne += 2.0 * G[2][2] * G[2][2];
        ne += (G[0][1] + G[1][0]) * (G[0][1] + G[1][0]);
        ne += (G[0][2] + G[2][0]) * (G[0][2] + G[2][0]);
        ne += (G[1][2] + G[2][1]) * (G[1][2] + G[2][1]);
        const double nt = c.les_ct * sqrt(ne);
        nut[0] += nt; nut[1] += nt * nt; nut[2] = fmax(nut[2], nt);
        v[0] = mk<T>(T(QG), T(QS));
        v[1] = mk<T>(T(det3(G)), T(det3(S)));
        v[2] = mk<T>(T(4.0 * (trS2O2 - 2.0 * QS * (QG - QS))), T(0));
    } else {
        // conv_i = u_j d_j u_i (src/HIT_LES.cpp:74-125)
        const T uu = v[0].x, vv = v[0].y, ww = v[1].x, uz = v[1].y, ux = v[2].x, uy = v[2].y, vx = v[3].x, vy = v[3].y, wx = v[4].x,
                wy = v[4].y, vz = v[5].x, wz = v[5].y;
        cfl_update<T>(mx, uu, vv, ww, c);
        const T cu = uu * ux + vv * uy + ww * uz;
        const T cv = uu * vx + vv * vy + ww * vz;
        const T cw = uu * wx + vv * wy + ww * wz;
        if constexpr (MODE == MODE_ADV) {
            v[0] = mk<T>(cu, cv);
            v[1] = mk<T>(cw, T(0));
        } else {
            // eddy viscosity and SGS stress (src/HIT_LES.cpp:130-154)
            const T a12 = uy + vx, a13 = uz + wx, a23 = wy + vz;
            T ne = T(2.0) * ux * ux;
            ne += T(2.0) * vy * vy;
            ne += T(2.0) * wz * wz;
            ne += a12 * a12;
            ne += a13 * a13;
            ne += a23 * a23;
            ne = T(c.les_ct) * sqrt(ne);
            v[0] = mk<T>(cu, T(-1.0) * ne * a13);
            v[1] = mk<T>(cv, T(-1.0) * ne * a23);
            v[2] = mk<T>(cw, T(-2.0) * ne * wz);
            v[3] = mk<T>(T(-2.0) * ne * ux, T(-1.0) * ne * a12);
            v[4] = mk<T>(T(-2.0) * ne * vy, T(0));
        }
    }
}

// The row of a thread: one pencil's, or one of each pencil of a pair.
template <int MODE, typename T>
__device__ __forceinline__ void zfield_rows(cx<T> (&v)[ZFieldForm<MODE>::NPAIR], const StepConsts &c, double (&mx)[4], double (&nut)[3]) {
    if constexpr (Arith<T>::W == 1) {
        zfield_row<T, MODE>(v, c, mx, nut);
    } else {
        constexpr int N = ZFieldForm<MODE>::NPAIR;
        cx<float> a[N], b[N];
#pragma unroll
        for (int p = 0; p < N; p++) { a[p] = mk<float>(v[p].x.lo(), v[p].y.lo()); b[p] = mk<float>(v[p].x.hi(), v[p].y.hi()); }
        zfield_row<float, MODE>(a, c, mx, nut);
        zfield_row<float, MODE>(b, c, mx, nut);
#pragma unroll
        for (int p = 0; p < ZFieldForm<MODE>::NJOB; p++) v[p] = mk<f2>(f2(a[p].x, b[p].x), f2(a[p].y, b[p].y));
    }
}

template <typename T, int L, int E, int PB, int NT, int MODE> struct ZFieldLayout {
    static constexpr int Q = L / E;
    // teams of a warp; where Q does not divide 32 the last lanes of a warp have no team
    static constexpr int TPW = Q < 32 ? 32 / Q : 1;
    static constexpr int THREADS = Q <= 32 ? NT / TPW * 32 : NT * Q;
    static constexpr unsigned WARP = Q > 32 ? 0u : 32 % Q == 0 ? 1u : (1u << (TPW * Q)) - 1u;
    static_assert(Q <= 32 ? NT % TPW == 0 : Q % 32 == 0, "whole warps");
    static constexpr int NPAIR = ZFieldForm<MODE>::NPAIR, NJOB = ZFieldForm<MODE>::NJOB;
    static constexpr int PITCH = SmPencil<T, L, E>::PITCH;
    static constexpr int RI = PB * NPAIR / NT;                  // rounds of the teams over the inverse pairs
    static constexpr int RF = (PB * NJOB + NT - 1) / NT;        // and over the forward jobs
    static_assert(PB * NPAIR % NT == 0, "whole rounds of inverse pairs");
    static_assert(RF * NT <= PB * NPAIR, "a team without a job needs a buffer that no job uses");
    static constexpr size_t SMEM = (size_t)PB * NPAIR * PITCH * sizeof(cx<T>);
};

template <typename T, int L, int E, int PB, int NT, int MODE>
__device__ __forceinline__ void k3_field_body(Geo g, SCx<T> *__restrict__ buf, const StepConsts &c, DevScalars *ds,
                                              double *__restrict__ nut_out, const cx<T> *__restrict__ tw) {
    using LY = ZFieldLayout<T, L, E, PB, NT, MODE>;
    constexpr int Q = LY::Q, NPAIR = LY::NPAIR, NJOB = LY::NJOB, PITCH = LY::PITCH;
    constexpr unsigned WARP = LY::WARP;
    extern __shared__ __align__(16) unsigned char smraw[];
    cx<T> *const smc = reinterpret_cast<cx<T> *>(smraw);
    const int tid = threadIdx.x, lane = tid & 31;
    const int team = Q <= 32 ? (tid >> 5) * LY::TPW + lane / Q : tid / Q, q = Q <= 32 ? lane % Q : tid % Q;
    const bool has_team = Q > 32 || lane < LY::TPW * Q;
    // pencils, or pairs of neighbouring pencils (npen is even: every compiled length is)
    constexpr int W = Arith<T>::W;
    const long long npen = (long long)g.Mx * g.My / W, ngrp = (npen + PB - 1) / PB;
    const T sz = T(g.sz);
    const int Kz = g.Kz;
    double mx[4] = {0.0, 0.0, 0.0, 0.0}, nut[3] = {0.0, 0.0, 0.0};

    for (long long grp = blockIdx.x; grp < ngrp; grp += gridDim.x) {
        const long long p0 = grp * PB;
        const int np = (int)(npen - p0 < PB ? npen - p0 : PB);
        cx<T> A[E];
        if (has_team)
#pragma unroll 1
        for (int r = 0; r < LY::RI; r++) {
            const int item = team + r * NT, pl = item / NPAIR;
            const ZPair pr = zfield_pair<MODE>(item - pl * NPAIR);
            const bool ok = pl < np;
            const SCx<T> *base = buf + (p0 + (ok ? pl : 0)) * W * g.Kp;
            SmPencil<T, L, E> sm{smc + item * PITCH};
            k3_load_pair<T, L, E>(A, base + pr.a * g.S2, pr.da, pr.b < 0 ? nullptr : base + pr.b * g.S2, pr.db, Kz, sz, q, ok, g.Kp);
            fft<T, L, E, true, SmPencil<T, L, E>, WARP>(A, sm, q, tw);
            stage_barrier<WARP>();
#pragma unroll
            for (int e = 0; e < E; e++) sm.at(out_row<L, E, true>(q, e)) = A[e];
        }
        __syncthreads();
#pragma unroll 1
        for (int i = tid; i < np * L; i += LY::THREADS) {
            const int pl = i / L;
            cx<T> *b = smc + pl * NPAIR * PITCH + (i - pl * L);
            cx<T> v[NPAIR];
#pragma unroll
            for (int p = 0; p < NPAIR; p++) v[p] = b[p * PITCH];
            zfield_rows<MODE>(v, c, mx, nut);
#pragma unroll
            for (int j = 0; j < NJOB; j++) b[j * PITCH] = v[j];
        }
        __syncthreads();
        if (has_team)
#pragma unroll 1
        for (int r = 0; r < LY::RF; r++) {
            const int item = team + r * NT, idle = item - PB * NJOB;
            const int pl = idle < 0 ? item / NJOB : idle / (NPAIR - NJOB);
            const int j = idle < 0 ? item - pl * NJOB : NJOB + idle - pl * (NPAIR - NJOB);
            const ZJob jb = zfield_job<MODE>(idle < 0 ? j : 0);
            const bool ok = idle < 0 && pl < np;
            SmPencil<T, L, E> sm{smc + (pl * NPAIR + j) * PITCH};
            SCx<T> *base = buf + (p0 + (ok ? pl : 0)) * W * g.Kp;
            SCx<T> *oa = base + jb.a * g.S2, *ob = jb.b < 0 ? nullptr : base + jb.b * g.S2;
#pragma unroll
            for (int e = 0; e < E; e++) A[e] = sm.at(in_row<L, E, false>(q, e));
            fft<T, L, E, false, SmPencil<T, L, E>, WARP>(A, sm, q, tw);
            stage_barrier<WARP>();
#pragma unroll
            for (int e = 0; e < E; e++) sm.at(out_row<L, E, false>(q, e)) = A[e];
            stage_barrier<WARP>();
            if (ok) {
                const T h = T(0.5);
                for (int k = q; k < Kz; k += Q) {
                    const cx<T> zk = sm.at(k), zm = sm.at(k == 0 ? 0 : L - k);
                    if (jb.single) {
                        st_pencil(oa, k, g.Kp, zk);
                    } else {
                        cx<T> xa = mk<T>(h * (zk.x + zm.x), h * (zk.y - zm.y));
                        const cx<T> xb = mk<T>(h * (zk.y + zm.y), h * (zm.x - zk.x));
                        if (jb.fold) xa = xa + mul_i(T(k) * sz * xb);
                        st_pencil(oa, k, g.Kp, xa);
                        if (ob) st_pencil(ob, k, g.Kp, xb);
                    }
                }
            }
        }
        __syncthreads();
    }
    if constexpr (MODE == MODE_INV) {
        if (nut_out) {
            block_sum(nut[0], nut_out);
            block_sum(nut[1], nut_out + 1);
            block_max_bits(nut[2], reinterpret_cast<unsigned long long *>(nut_out + 2));
        }
    } else {
        block_max4<T>(mx, ds);
    }
}

template <typename T, int L, int E, int PB, int NT, int MODE, int MINB>
__global__ void __launch_bounds__(ZFieldLayout<T, L, E, PB, NT, MODE>::THREADS, MINB) k3_field(Geo g, SCx<T> *__restrict__ buf, StepConsts c, DevScalars *ds,
                                                              double *__restrict__ nut_out, const cx<T> *__restrict__ tw) {
    k3_field_body<T, L, E, PB, NT, MODE>(g, buf, c, ds, nut_out, tw);
}
// Members of a batched class: blockIdx.y selects the member (solver_kernels.cuh, BatchMember).
template <typename T, int L, int E, int PB, int NT, int MODE, int MINB>
__global__ void __launch_bounds__(ZFieldLayout<T, L, E, PB, NT, MODE>::THREADS, MINB) k3_field_batch(Geo g, const BatchMember *__restrict__ tab, const cx<T> *__restrict__ tw) {
    const BatchMember &m = tab[blockIdx.y];
    k3_field_body<T, L, E, PB, NT, MODE>(g, static_cast<SCx<T> *>(m.B2), m.c, m.ds, nullptr, tw);
}

} // namespace spns
