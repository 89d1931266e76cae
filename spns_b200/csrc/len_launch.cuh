// len_launch.cuh -- launches of the pass kernels of one FFT length, templated on the
// arithmetic type T of the transforms (double: FP64 form; float: compensated FP32
// hi/lo form).  spns_len.cu instantiates one (precision, length) per object, so the
// lengths compile in parallel, and exports its LenTable; passes.cuh runs the step
// through those tables.
#pragma once
#include "handle.h"

#include <algorithm>

template <typename T> struct LenLaunch {
    using C = spns::cx<T>;

    static C *U(spns_handle *h, int f = 0) { return (C *)h->U + (long long)f * h->g.S0; }
    static const C *tw(spns_handle *h, int L) { return (const C *)h->tw[L]; }
    // arithmetic of the z passes: single precision runs two pencils per thread in packed pairs
    using A = typename std::conditional<sizeof(T) == 4, spns::f2, T>::type;
    // arithmetic of the x/y passes
    template <int PASS, int L> using AX = typename std::conditional<sizeof(T) == 4 && spns_pair_pass(PASS, L), spns::f2, T>::type;
    template <int PASS, int L> static const spns::cx<AX<PASS, L>> *twx(spns_handle *h) {
        return (const spns::cx<AX<PASS, L>> *)(sizeof(AX<PASS, L>) != sizeof(T) ? h->tw2[L] : h->tw[L]);
    }
    static const spns::cx<A> *twa(spns_handle *h, int L) { return (const spns::cx<A> *)(sizeof(T) == 4 ? h->tw2[L] : h->tw[L]); }

    // kz chunks of an x/y pass with P threads along kz
    template <typename X> static int axis_chunks(const spns_handle *h, int P) { const int w = P * spns::Arith<X>::W; return (h->g.Kz + w - 1) / w; }
    // Grid of an x/y pass: kz chunks x lines, and for small boxes the fields (or groups of
    // fields) of the pass spread over blocks.
    template <typename X> static dim3 axis_grid(const spns_handle *h, int P, int lines, int fields) {
        const int chunks = axis_chunks<X>(h, P);
        return dim3(chunks, lines, (long long)chunks * lines < (long long)SPNS_SPLIT_WAVES * h->sms ? fields : 1);
    }
    template <int L, int MODE, int ALT = 0> static cudaError_t launch_k1(spns_handle *h) {
        using S = ShapeK1A<AX<1, L>, L, ALT>;
        auto kern = spns::k1_inv_x<AX<1, L>, L, S::E, S::P, MODE>;
        constexpr size_t smem = spns::K1Smem<AX<1, L>, L, S::E, S::P, MODE>::BYTES;
        cudaError_t e = spns_set_smem(kern, smem);
        if (e != cudaSuccess) return e;
        const dim3 grid = axis_grid<AX<1, L>>(h, S::P, h->g.Ky, spns::Fields<MODE>::K1);
        kern<<<grid, S::THREADS, smem, h->st>>>(h->g, U(h, 0), U(h, 1), U(h, 2), (C *)h->B1, twx<1, L>(h),
             MODE == spns::MODE_INV ? nullptr : h->ds);
        return cudaGetLastError();
    }
    template <int L, int MODE, int ALT = 0> static cudaError_t launch_k2(spns_handle *h) {
        using S = ShapeK2A<AX<2, L>, L, ALT>;
        auto kern = spns::k2_inv_y<AX<2, L>, L, S::E, S::P, MODE>;
        cudaError_t e = spns_set_smem(kern, S::SMEM_ROW);
        if (e != cudaSuccess) return e;
        const dim3 grid = axis_grid<AX<2, L>>(h, S::P, h->g.Mx, spns::Fields<MODE>::K2);
        kern<<<grid, S::THREADS, S::SMEM_ROW, h->st>>>(h->g, (const C *)h->B1, (C *)h->B2, twx<2, L>(h));
        return cudaGetLastError();
    }
    // Blocks of a z pass over n items whose blocks walk the box, `wave` of them resident at once.
    // A block holds its place on an SM until it ends, so a run of higher priority on the same
    // device waits that long: one wave where a block has at most 16 items (14 to 29 us each),
    // else as many whole waves as leave it 8.  32^3 and 64^3 LES of higher priority beside two
    // 256^3 LES boxes, us a step, one wave against this: single 209 -> 160 and 443 -> 365, double
    // 269 -> 192 and 567 -> 430 (with a block for every few pencils 211, 390, 265, 519).  The pass
    // alone, ms: 256^3 LES single 2.28 -> 2.20, double 4.00 -> 3.82; 512^3 single 7.23 -> 6.80,
    // double 11.53 -> 11.47; 512 x 512 x 64 LES double 3.61 -> 3.77.  With four items for eight the
    // waits are 5 to 15 % shorter, 512^3 single 7.6 and 512 x 512 x 64 3.91.
    static unsigned walking_blocks(long long wave, long long n) {
        const long long rounds = (n + wave - 1) / wave;
        return (unsigned)std::min(n, rounds <= 16 ? wave : wave * ((rounds + 7) / 8));
    }
    // Rotational z pass staged pair by pair with bulk copies (zpass_staged.cuh),
    // one block per SM at a time.  Units of the box, and units the SMs hold in one round.
    template <int L> static long long staged_units(const spns_handle *h) {
        using LY = spns::ZStagedLayout<A, L, SPNS_ZS_E>;
        return (long long)h->g.Mx * h->g.My / (LY::PPU * LY::W);
    }
    template <int L> static long long staged_round(const spns_handle *h) {
        return (long long)spns::ZStagedLayout<A, L, SPNS_ZS_E>::max_units(h->g.Kz, h->g.Kp) * h->sms;
    }
    // A unit's pairs follow one another, so the pass needs rounds to overlap: against k3_z, whose
    // blocks copy all six fields at their start, it is faster from half a round in double
    // precision (0.24..0.49 rounds, 48 x 48 pencils of 96..192: 0.020..0.023 against 0.016..0.019 ms;
    // 0.55, 72 x 72 of 96: 0.023 against 0.029) and from three in single precision (3.5, 144 x 144 of
    // 288: 0.115 against 0.125; 3.9, 192^3: 0.111 against 0.125; 2.2, 144 x 144 of 192: 0.086 against 0.076).
    template <int L> static bool staged_pays(const spns_handle *h) {
        return sizeof(T) == 8 ? 2 * staged_units<L>(h) >= staged_round<L>(h) : staged_units<L>(h) >= 3 * staged_round<L>(h);
    }
    template <int L> static cudaError_t launch_k3_staged(spns_handle *h) {
        using LY = spns::ZStagedLayout<A, L, SPNS_ZS_E>;
        auto kern = spns::k3_rot_staged<A, L, SPNS_ZS_E>;
        const long long ngrp = staged_units<L>(h), per_round = staged_round<L>(h), rounds = (ngrp + per_round - 1) / per_round;
        // as many units as spread the pencils evenly over the rounds
        const int units = (int)((ngrp + rounds * h->sms - 1) / (rounds * h->sms));
        const size_t smem = LY::smem_bytes(units, h->g.Kz, h->g.Kp);
        cudaError_t e = spns_set_smem(kern, LY::SMEM_MAX);
        if (e != cudaSuccess) return e;
        const unsigned blocks = walking_blocks(h->sms, (ngrp + units - 1) / units);
        kern<<<blocks, units * LY::U, smem, h->st>>>(h->g, (C *)h->B2, h->c, h->ds, twa(h, L), h->stage_polls);
        return cudaGetLastError();
    }
    // Launch of k3_field: blocks that walk the pencils.
    template <int L, int MODE, int ALT> static cudaError_t launch_k3_field(spns_handle *h, double *nut) {
        using S = ZFieldShape<A, L, MODE, ALT>;
        auto kern = spns::k3_field<A, L, S::E, S::PB, S::NT, MODE, S::MINB>;
        unsigned blocks = 0;
        cudaError_t e = walking_grid(h, kern, S::THREADS, S::LY::SMEM, ((long long)h->g.Mx * h->g.My / spns::Arith<A>::W + S::PB - 1) / S::PB, &blocks);
        if (e != cudaSuccess) return e;
        kern<<<blocks, S::THREADS, S::LY::SMEM, h->st>>>(h->g, (C *)h->B2, h->c, h->ds, nut, twa(h, L));
        return cudaGetLastError();
    }
    // Shared-memory opt-in and grid of a kernel whose blocks walk n work items.
    template <class K> static cudaError_t walking_grid(spns_handle *h, K kern, int threads, size_t smem, long long n, unsigned *blocks) {
        cudaError_t e = spns_set_smem(kern, smem);
        if (e != cudaSuccess) return e;
        int per_sm = 0;
        if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem)) != cudaSuccess) return e;
        if (per_sm < 1) return cudaErrorInvalidConfiguration;
        *blocks = walking_blocks((long long)h->sms * per_sm, n);
        return cudaSuccess;
    }
    template <int L, int MODE, int ALT = 0> static cudaError_t launch_k3(spns_handle *h, double *phys) {
        if constexpr (MODE != spns::MODE_VEL && MODE != spns::MODE_ROT) {
            return launch_k3_field<L, MODE, ALT>(h, phys);
        } else {
        if constexpr (MODE == spns::MODE_ROT && ALT == 0 && spns_zstaged_length<T>(L))
            if (staged_pays<L>(h)) return launch_k3_staged<L>(h);
        using S3 = Shape3<T, L, ALT>;
        constexpr bool STAGE = MODE == spns::MODE_ROT && ShapeSel<T>::Z_STAGE;
        auto kern = spns::k3_z<T, L, S3::E, S3::P, MODE, STAGE>;
        constexpr size_t stage_fields = STAGE ? 2 * spns::K3StagePairs<T>::N : 0;
        // the staging is sized by Kz at run time: at most L/2+1 values per field and pencil
        constexpr size_t most = S3::SMEM + (size_t)S3::P * stage_fields * (L / 2 + 1) * sizeof(C);
        static_assert(most <= 225 * 1024, "z-pass shared memory (exchange and staging) exceeds 227 KB, less the reductions', for this shape");
        const size_t smem = S3::SMEM + (size_t)S3::P * stage_fields * h->g.Kz * sizeof(C);
        cudaError_t e = spns_set_smem(kern, most);
        if (e != cudaSuccess) return e;
        const long long npen = (long long)h->g.Mx * h->g.My;
        dim3 grid((unsigned)((npen + S3::P - 1) / S3::P));
        kern<<<grid, S3::THREADS, smem, h->st>>>(h->g, (C *)h->B2, h->c, h->ds, phys, tw(h, L));
        return cudaGetLastError();
        }
    }
    template <int L, int MODE, int ALT = 0> static cudaError_t launch_k4(spns_handle *h) {
        using S = ShapeK4A<AX<4, L>, L, MODE, ALT>;
        auto kern = spns::k4_fwd_y<AX<4, L>, L, S::E, S::P, MODE>;
        cudaError_t e = spns_set_smem(kern, S::SMEM_ROW);
        if (e != cudaSuccess) return e;
        const dim3 grid = axis_grid<AX<4, L>>(h, S::P, h->g.Mx, MODE == spns::MODE_LES ? 5 : spns::Fields<MODE>::NOUT);
        kern<<<grid, S::THREADS, S::SMEM_ROW, h->st>>>(h->g, (const C *)h->B2, (C *)h->B1, twx<4, L>(h));
        return cudaGetLastError();
    }
    template <int L, int MODE, int ALT = 0> static cudaError_t launch_k5(spns_handle *h) {
        using S = ShapeK5A<AX<5, L>, L, MODE, ALT>;
        auto kern = spns::k5_fwd_x<AX<5, L>, L, S::E, S::P, MODE>;
        cudaError_t e = spns_set_smem(kern, S::SMEM_ROW);
        if (e != cudaSuccess) return e;
        const dim3 grid = axis_grid<AX<5, L>>(h, S::P, h->g.Ky, spns::Fields<MODE>::NOUT);
        kern<<<grid, S::THREADS, S::SMEM_ROW, h->st>>>(h->g, (const C *)h->B1, (C *)h->B2, twx<5, L>(h));
        return cudaGetLastError();
    }
    // Launch of pass K1..K5 in the shape the handle selected (shape_alt).
#define SPNS_SELECT(name, idx, ...)                                                              \
    template <int L, int MODE> static cudaError_t sel_##name(spns_handle *h) {                    \
        if constexpr (shape_alt_ok<L, MODE>())                                                    \
            if (h->shape_alt[idx]) return launch_##name<L, MODE, 1>(h __VA_ARGS__);               \
        return launch_##name<L, MODE, 0>(h __VA_ARGS__);                                          \
    }
    SPNS_SELECT(k1, 1)
    SPNS_SELECT(k2, 2)
    SPNS_SELECT(k3, 3, , nullptr)
    SPNS_SELECT(k4, 4)
    SPNS_SELECT(k5, 5)
#undef SPNS_SELECT

    // Batched 1-D FFTs for the 2-D edge planes.
    template <int L, bool INV> static cudaError_t launch_lines(spns_handle *h, C *data, long long batch) {
        using S = Shape<T, L>;
        auto kern = spns::k_lines<T, L, S::E, S::P, INV>;
        cudaError_t e = spns_set_smem(kern, S::SMEM_PEN);
        if (e != cudaSuccess) return e;
        kern<<<(unsigned)((batch + S::P - 1) / S::P), S::THREADS, S::SMEM_PEN, h->st>>>(data, batch, tw(h, L));
        return cudaGetLastError();
    }
    template <int L, bool INV> static cudaError_t launch_cols(spns_handle *h, C *data, int ncols, int nbatch) {
        using S = Shape<T, L>;
        auto kern = spns::k_cols<T, L, S::E, S::P, INV>;
        cudaError_t e = spns_set_smem(kern, S::SMEM_ROW);
        if (e != cudaSuccess) return e;
        dim3 grid((ncols + S::P - 1) / S::P, nbatch);
        kern<<<grid, S::THREADS, S::SMEM_ROW, h->st>>>(data, ncols, tw(h, L));
        return cudaGetLastError();
    }
    // ---- batched launches: one per pass for the members of a table, all of h0's class ----
    template <int L, int MODE, int ALT> static cudaError_t launch_k1b(spns_handle *h, const spns::BatchMember *tab, int n, cudaStream_t st) {
        using S = ShapeK1A<AX<1, L>, L, ALT>;
        auto kern = spns::k1_inv_x_batch<AX<1, L>, L, S::E, S::P, MODE>;
        cudaError_t e = spns_set_smem(kern, S::SMEM_ROW);
        if (e != cudaSuccess) return e;
        kern<<<dim3(axis_chunks<AX<1, L>>(h, S::P), h->g.Ky, n), S::THREADS, S::SMEM_ROW, st>>>(h->g, tab, twx<1, L>(h));
        return cudaGetLastError();
    }
    template <int L, int MODE, int ALT> static cudaError_t launch_k2b(spns_handle *h, const spns::BatchMember *tab, int n, cudaStream_t st) {
        using S = ShapeK2A<AX<2, L>, L, ALT>;
        auto kern = spns::k2_inv_y_batch<AX<2, L>, L, S::E, S::P, MODE>;
        cudaError_t e = spns_set_smem(kern, S::SMEM_ROW);
        if (e != cudaSuccess) return e;
        kern<<<dim3(axis_chunks<AX<2, L>>(h, S::P), h->g.Mx, n), S::THREADS, S::SMEM_ROW, st>>>(h->g, tab, twx<2, L>(h));
        return cudaGetLastError();
    }
    template <int L, int MODE, int ALT> static cudaError_t launch_k3b(spns_handle *h, const spns::BatchMember *tab, int n, cudaStream_t st) {
        using S = ZFieldShape<A, L, MODE, ALT>;
        auto kern = spns::k3_field_batch<A, L, S::E, S::PB, S::NT, MODE, S::MINB>;
        unsigned blocks = 0;
        cudaError_t e = walking_grid(h, kern, S::THREADS, S::LY::SMEM, ((long long)h->g.Mx * h->g.My / spns::Arith<A>::W + S::PB - 1) / S::PB, &blocks);
        if (e != cudaSuccess) return e;
        kern<<<dim3(blocks, n), S::THREADS, S::LY::SMEM, st>>>(h->g, tab, twa(h, L));
        return cudaGetLastError();
    }
    template <int L, int MODE, int ALT> static cudaError_t launch_k4b(spns_handle *h, const spns::BatchMember *tab, int n, cudaStream_t st) {
        using S = ShapeK4A<AX<4, L>, L, MODE, ALT>;
        auto kern = spns::k4_fwd_y_batch<AX<4, L>, L, S::E, S::P, MODE>;
        cudaError_t e = spns_set_smem(kern, S::SMEM_ROW);
        if (e != cudaSuccess) return e;
        kern<<<dim3(axis_chunks<AX<4, L>>(h, S::P), h->g.Mx, n), S::THREADS, S::SMEM_ROW, st>>>(h->g, tab, twx<4, L>(h));
        return cudaGetLastError();
    }
    template <int L, int MODE, int ALT> static cudaError_t launch_k5b(spns_handle *h, const spns::BatchMember *tab, int n, cudaStream_t st) {
        using S = ShapeK5A<AX<5, L>, L, MODE, ALT>;
        auto kern = spns::k5_fwd_x_batch<AX<5, L>, L, S::E, S::P, MODE>;
        cudaError_t e = spns_set_smem(kern, S::SMEM_ROW);
        if (e != cudaSuccess) return e;
        kern<<<dim3(axis_chunks<AX<5, L>>(h, S::P), h->g.Ky, n), S::THREADS, S::SMEM_ROW, st>>>(h->g, tab, twx<5, L>(h));
        return cudaGetLastError();
    }
#define SPNS_SELECT_B(name, idx)                                                                                       \
    template <int L, int MODE> static cudaError_t sel_##name(spns_handle *h, const spns::BatchMember *tab, int n, cudaStream_t st) { \
        if constexpr (shape_alt_ok<L, MODE>())                                                                         \
            if (h->shape_alt[idx]) return launch_##name<L, MODE, 1>(h, tab, n, st);                                    \
        return launch_##name<L, MODE, 0>(h, tab, n, st);                                                               \
    }
    SPNS_SELECT_B(k1b, 1)
    SPNS_SELECT_B(k2b, 2)
    SPNS_SELECT_B(k3b, 3)
    SPNS_SELECT_B(k4b, 4)
    SPNS_SELECT_B(k5b, 5)
#undef SPNS_SELECT_B

    // ---- the table of one length ----
    // Pass k (1..5: K1..K5) of `mode`; `select`: in the shape the handle chose for it
    // (steps), else in the default shape.  `phys` goes to the z pass.
    template <int L, int MODE> static cudaError_t run_mode(spns_handle *h, int k, bool select, double *phys) {
        switch (k) {
        case 1: return select ? sel_k1<L, MODE>(h) : launch_k1<L, MODE>(h);
        case 2: return select ? sel_k2<L, MODE>(h) : launch_k2<L, MODE>(h);
        case 3: return select ? sel_k3<L, MODE>(h) : launch_k3<L, MODE>(h, phys);
        case 4: return select ? sel_k4<L, MODE>(h) : launch_k4<L, MODE>(h);
        default: return select ? sel_k5<L, MODE>(h) : launch_k5<L, MODE>(h);
        }
    }
    template <int L> static cudaError_t run_vel(spns_handle *h, int k, double *phys) {
        return k == 1 ? launch_k1<L, spns::MODE_VEL>(h) : k == 2 ? launch_k2<L, spns::MODE_VEL>(h) : launch_k3<L, spns::MODE_VEL>(h, phys);
    }
    template <int L> static cudaError_t pass(spns_handle *h, int k, int mode, bool select, double *phys) {
        switch (mode) {
        case spns::MODE_VEL: return run_vel<L>(h, k, phys);
        case spns::MODE_ROT: return run_mode<L, spns::MODE_ROT>(h, k, select, phys);
        case spns::MODE_ADV: return run_mode<L, spns::MODE_ADV>(h, k, select, phys);
        case spns::MODE_LES: return run_mode<L, spns::MODE_LES>(h, k, select, phys);
        default: return run_mode<L, spns::MODE_INV>(h, k, select, phys);
        }
    }
    template <int L, int MODE> static cudaError_t batch_mode(spns_handle *h, const spns::BatchMember *tab, int n, cudaStream_t st, int k) {
        switch (k) {
        case 1: return sel_k1b<L, MODE>(h, tab, n, st);
        case 2: return sel_k2b<L, MODE>(h, tab, n, st);
        case 3: return sel_k3b<L, MODE>(h, tab, n, st);
        case 4: return sel_k4b<L, MODE>(h, tab, n, st);
        default: return sel_k5b<L, MODE>(h, tab, n, st);
        }
    }
    template <int L> static cudaError_t batch(spns_handle *h, const spns::BatchMember *tab, int n, cudaStream_t st, int k, int mode) {
        if constexpr (spns_batch_length(L))
            return mode == spns::MODE_LES ? batch_mode<L, spns::MODE_LES>(h, tab, n, st, k) : batch_mode<L, spns::MODE_ADV>(h, tab, n, st, k);
        return cudaErrorNotSupported;
    }
    template <int L> static cudaError_t lines(spns_handle *h, void *data, long long batch, bool inv) {
        return inv ? launch_lines<L, true>(h, (C *)data, batch) : launch_lines<L, false>(h, (C *)data, batch);
    }
    template <int L> static cudaError_t cols(spns_handle *h, void *data, int ncols, int nbatch, bool inv) {
        return inv ? launch_cols<L, true>(h, (C *)data, ncols, nbatch) : launch_cols<L, false>(h, (C *)data, ncols, nbatch);
    }
    template <int L> static constexpr LenTable table() { return LenTable{&pass<L>, &batch<L>, &lines<L>, &cols<L>}; }
};
