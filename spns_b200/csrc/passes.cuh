// passes.cuh -- launch code of one step, templated on the arithmetic type T of
// the transforms (double: FP64 form; float: compensated FP32 hi/lo form).
// Included by exactly one translation unit per precision (spns_f64.cu,
// spns_f32.cu), which exports the PrecOps table of that precision.
#pragma once
#include "handle.h"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

template <typename T> struct Passes {
    using C = spns::cx<T>;
    static constexpr bool HILO = sizeof(T) == 4;

    static C *U(spns_handle *h, int f = 0) { return (C *)h->U + (long long)f * h->g.S0; }
    static C *Ulo(spns_handle *h, int f = 0) { return HILO ? (C *)h->Ulo + (long long)f * h->g.S0 : nullptr; }
    // FFT length of pass K1..K5: x, y, z, y, x
    static int pass_length(const spns_handle *h, int k) { return k == 3 ? h->g.Mz : (k == 2 || k == 4) ? h->g.My : h->g.Mx; }
    // Pass k of `mode` on the handle's stream (LenTable::pass).
    static cudaError_t pass(spns_handle *h, int k, int mode, bool select, double *phys = nullptr) {
        return spns_len_table<T>(pass_length(h, k))->pass(h, k, mode, select, phys);
    }


    // Spectral sweep; with the kappa scheme the new state goes into the u^{n-1}
    // buffers and the state buffers are swapped after the launch.
    static cudaError_t launch_k6(spns_handle *h) {
        const int n = h->g.Kx * h->g.Kz;
        dim3 grid((n + 255) / 256, h->g.Ky);
        const C *G = (const C *)h->B2;
        if (h->a.isSelfAdaptive) {
            spns::k6_sweep<T, true><<<grid, 256, 0, h->st>>>(h->g, G, U(h), Ulo(h), (C *)h->R, (C *)h->Up, (C *)h->Uplo,
                                                              (const C *)h->Up, (const C *)h->Uplo, h->c, h->ds);
            std::swap(h->U, h->Up);
            std::swap(h->Ulo, h->Uplo);
        } else {
            spns::k6_sweep<T, false><<<grid, 256, 0, h->st>>>(h->g, G, U(h), Ulo(h), (C *)h->R, U(h), Ulo(h), nullptr, nullptr,
                                                               h->c, h->ds);
        }
        return cudaGetLastError();
    }

    // Inverse transform of the velocity only (Recalculate_Velocity_Antitransform):
    // refreshes the CFL maxima and, if phys != NULL, writes u,v,w on the grid.
    static int run_velocity(spns_handle *h, double *phys) {
        for (int k = 1; k <= 3; k++) LAUNCH(pass(h, k, spns::MODE_VEL, false, phys));
        return SPNS_OK;
    }

    // E(K), Om(K) of the state into h->bins.
    static int shell_sums(spns_handle *h) {
        const int nb = h->last_rad_max + 1;
        CK(cudaMemsetAsync(h->bins, 0, sizeof(double) * 2 * nb, h->st));
        const long long n = h->g.S0;
        const int blocks = (int)std::min<long long>((n + 255) / 256, (long long)spns::SHELL_BLOCKS_PER_SM * h->sms);
        spns::k_shell_sums<T><<<blocks, 256, sizeof(double) * 2 * nb, h->st>>>(h->g, U(h, 0), U(h, 1), U(h, 2), Ulo(h, 0), Ulo(h, 1),
                                                                              Ulo(h, 2), h->last_rad_max, h->bins, h->bins + nb);
        CKL();
        return SPNS_OK;
    }

    static int forcing_scale(spns_handle *h, int last_eff, int nullify) {
        const long long n = h->g.S0;
        const int blocks = (int)std::min<long long>((n + 255) / 256, 16LL * h->sms);
        spns::k_forcing_scale<T><<<blocks, 256, 0, h->st>>>(h->g, U(h, 0), U(h, 1), U(h, 2), Ulo(h, 0), Ulo(h, 1), Ulo(h, 2), h->FT,
                                                           last_eff, nullify);
        CKL();
        return SPNS_OK;
    }

    static int conj_correction(spns_handle *h) {
        spns::k_conj_correction<T><<<64, 256, 0, h->st>>>(h->g, U(h, 0), U(h, 1), U(h, 2), Ulo(h, 0), Ulo(h, 1), Ulo(h, 2));
        CKL();
        return SPNS_OK;
    }

    static int seed_draw(spns_handle *h, unsigned long long seed, int lim_x, int lim_y, int lim_z) {
        const long long n = h->g.S0;
        const int blocks = (int)std::min<long long>((n + 255) / 256, 16LL * h->sms);
        spns::k_seed_draw<T><<<blocks, 256, 0, h->st>>>(h->g, seed, lim_x, lim_y, lim_z, U(h, 0), U(h, 1), U(h, 2), Ulo(h, 0),
                                                       Ulo(h, 1), Ulo(h, 2));
        CKL();
        return SPNS_OK;
    }

    // Spectra of the velocity-gradient invariants Q_G, Q_S, R_G, R_S, V^2 of the
    // current state (Recalculate_Invariants_Distribution, src/HIT_LES.cpp:1297-1319):
    // the five passes in MODE_INV on work buffers of the advective size (allocated
    // on first use and kept; the step's own buffers and graphs are not touched),
    // then shell sums of |F|^2 / (Mx My Mz)^2.  out[c*(last_rad_max+1) + K] on the host.
    static int invariant_spectra(spns_handle *h, double *out) {
        const spns::Geo &g = h->g;
        const int nb = h->last_rad_max + 1;
        if (!h->inv_B1) {
            CK(cudaMallocAsync(&h->inv_B1, sizeof(C) * 6 * (size_t)g.S1, h->st));
            CK(cudaMallocAsync(&h->inv_B2, sizeof(C) * 9 * (size_t)g.S2, h->st));
            CK(cudaMallocAsync((void **)&h->inv_bins, sizeof(double) * (5 * nb + 3), h->st));
        }
        double *nut = h->inv_bins + 5 * nb;               // nu_t sum, sum of squares, max bits
        CK(cudaMemsetAsync(nut, 0, sizeof(double) * 3, h->st));
        std::swap(h->B1, h->inv_B1);
        std::swap(h->B2, h->inv_B2);
        auto passes = [&]() -> int {
            for (int k = 1; k <= 5; k++) LAUNCH(pass(h, k, spns::MODE_INV, false, nut));
            return SPNS_OK;
        };
        const int r = passes();
        std::swap(h->B1, h->inv_B1);
        std::swap(h->B2, h->inv_B2);
        if (r) return r;
        CK(cudaMemsetAsync(h->inv_bins, 0, sizeof(double) * 5 * nb, h->st));
        const double scale = h->c.inv_norm * h->c.inv_norm;
        const int blocks = (int)std::min<long long>((g.S0 + 255) / 256, (long long)spns::SHELL_BLOCKS_PER_SM * h->sms);
        for (int c = 0; c < 5; c++) {
            spns::k_shell_sums_scalar<T><<<blocks, 256, sizeof(double) * nb, h->st>>>(
                g, (const C *)h->inv_B2 + (long long)c * g.S0, scale, h->last_rad_max, h->inv_bins + (long long)c * nb);
            CKL();
        }
        std::vector<double> host((size_t)5 * nb + 3);
        CK(cudaMemcpyAsync(host.data(), h->inv_bins, sizeof(double) * host.size(), cudaMemcpyDeviceToHost, h->st));
        CK(cudaStreamSynchronize(h->st));
        if (out) std::copy(host.begin(), host.begin() + 5 * nb, out);
        const double npts = (double)g.Mx * g.My * g.Mz;
        unsigned long long mb;
        std::memcpy(&mb, &host[5 * nb + 2], sizeof(mb));
        double mx;
        std::memcpy(&mx, &mb, sizeof(mx));
        h->nut_stats[0] = host[5 * nb] / npts;
        h->nut_stats[1] = std::sqrt(host[5 * nb + 1] / npts);
        h->nut_stats[2] = mx;
        return SPNS_OK;
    }

    // Exact aliasing correction of the rotational form on the +-N/2 planes
    // (edge_kernels.cuh), added to the compact nonlinear term G held in B2.  Its launches follow
    // the passes in the stream, though the planes need only the state: as a branch of the
    // step's graph they took 0.03 ms less of a 64^3 step and 0.26 ms of a 512^3 one, but
    // destroying a graph with branches waits for all work on the device (closing a box while
    // another steps: 600 ms against 1), and runs side by side held up each other's copies to the
    // host (served workload, median of eight: p50 3.1 s against 1.1).
    static int edge_correction(spns_handle *h) {
        const spns::Geo &g = h->g;
        // group the aliasing axes by the size of their 2-D transforms (one group for a cubic box)
        int RC[3][2] = {{g.My, g.Mz}, {g.Mx, g.Mz}, {g.Mx, g.My}};
        bool done[3] = {false, false, false};
        for (int a0 = 0; a0 < 3; a0++) {
            if (!h->edge_axis[a0] || done[a0]) continue;
            spns::EdgeSet es;
            es.naxes = 0;
            es.R = RC[a0][0];
            es.C = RC[a0][1];
            es.first[0] = 0;
            for (int a = a0; a < 3; a++) {
                if (!h->edge_axis[a] || done[a] || RC[a][0] != es.R || RC[a][1] != es.C) continue;
                done[a] = true;
                es.axis[es.naxes] = a;
                es.first[es.naxes + 1] = es.first[es.naxes] + (a == 2 ? 1 : 2);
                es.naxes++;
            }
            const int np = es.first[es.naxes];
            const long long n = (long long)es.R * es.C;
            C *V = (C *)h->edge, *Phi = V + 3 * (long long)np * n;
            const long long nb = n * 3 * np;
            const int blocks = (int)std::min<long long>((nb + 255) / 256, 16LL * h->sms);
            spns::k_edge_build<T><<<blocks, 256, 0, h->st>>>(g, U(h), es, V);
            CKL();
            LAUNCH(spns_len_table<T>(es.C)->lines(h, V, (long long)es.R * 3 * np, true));
            LAUNCH(spns_len_table<T>(es.R)->cols(h, V, es.C, 3 * np, true));
            spns::k_edge_square<T><<<blocks, 256, 0, h->st>>>(V, n, np, Phi);
            CKL();
            LAUNCH(spns_len_table<T>(es.C)->lines(h, Phi, (long long)es.R * np, false));
            LAUNCH(spns_len_table<T>(es.R)->cols(h, Phi, es.C, np, false));
            const int ablocks = (int)std::min<long long>((n * 2 + 255) / 256, 8LL * h->sms);
            spns::k_edge_apply<T><<<dim3(ablocks, es.naxes), 256, 0, h->st>>>(g, (C *)h->B2, es, Phi);
            CKL();
            h->edge_launches += 7;
        }
        return SPNS_OK;
    }

    // Records an event before the next kernel of a profiled step.
    static void prof_mark(spns_handle *h, int slot, const char *name) {
        if (h->prof_steps >= h->prof_cap_steps) return;
        if (slot >= 16) return;
        if (h->prof_steps == 0 && (int)h->prof_names.size() <= slot) h->prof_names.push_back(name ? name : "");
        cudaEventRecord(h->prof_ev[(size_t)h->prof_steps * 16 + slot], h->st);
    }

    // One New_Fractional_Step_Method (src/HIT_LES.cpp:9-25).
    static int step_once(spns_handle *h) {
        int nk = 0;
        h->edge_launches = 0;
        int slot = 0;
        const bool prof = h->prof_steps < h->prof_cap_steps;
#define MARK(name) do { if (prof) prof_mark(h, slot++, name); } while (0)
        if (h->a.eps_forcing > 0.0) {
            MARK("eps_band");
            spns::k_eps_band<T><<<1, spns::EPS_BAND_THREADS, 0, h->st>>>(h->g, U(h, 0), U(h, 1), U(h, 2), Ulo(h, 0), Ulo(h, 1), Ulo(h, 2),
                                                                      h->a.eps_kmin, h->a.eps_kmax, h->a.eps_forcing, h->ds);
            CKL();
            nk += 1;
        }
        const int mode = h->a.isLES ? spns::MODE_LES : h->a.nonlinear_form == 2 ? spns::MODE_ADV : spns::MODE_ROT;
        MARK("k1_inv_x");
        LAUNCH(pass(h, 1, mode, true));
        MARK("k2_inv_y");
        LAUNCH(pass(h, 2, mode, true));
        MARK("k3_z");
        LAUNCH(pass(h, 3, mode, true));
        MARK("k4_fwd_y");
        LAUNCH(pass(h, 4, mode, true));
        MARK("k5_fwd_x");
        LAUNCH(pass(h, 5, mode, true));
        if (mode == spns::MODE_ROT && h->edge) {
            MARK("edge_correction");
            int r_ = edge_correction(h);
            if (r_) return r_;
        }
        MARK("k6_sweep");
        LAUNCH(launch_k6(h));
        MARK("finish_step");
        spns::k_finish_step<<<1, 1, 0, h->st>>>(h->c, h->ds);
        CKL();
        MARK(nullptr);
        if (prof) { if (h->prof_steps == 0) h->prof_nk = slot - 1; h->prof_steps++; }
        if (mode == spns::MODE_ROT && h->edge) nk += h->edge_launches;             // build, 2+2 line FFTs, square, apply per group
        h->kernels_per_step = nk + 7;
        return SPNS_OK;
#undef MARK
    }

    // ---- slab decomposition (spns_slab_phase) ----
    // Reorder between a [nf][n1][n2][Kz] array and the all-to-all staging blocks.
    static cudaError_t slab_pack(spns_handle *h, void *full, void *stage, int nf, int n1, int n2, const spns::SlabRanges &r, int axis,
                                 int unpack) {
        const long long n = (long long)nf * n1 * n2 * h->g.Kz;
        const int blocks = (int)std::min<long long>((n + 255) / 256, 16LL * h->sms);
        spns::k_slab_pack<T><<<blocks, 256, 0, h->st>>>((C *)full, (C *)stage, nf, n1, n2, h->g.Kz, h->g.Kp, r, axis, unpack);
        return cudaGetLastError();
    }
    // Offsets of the staging blocks: block s holds nf * (axis 1: count_s * n2, axis 2: n1 * count_s) * Kz.
    static spns::SlabRanges slab_offsets(const spns::SlabRanges &r0, int nf, int n1, int n2, int Kz, int axis) {
        spns::SlabRanges r = r0;
        long long o = 0;
        for (int s = 0; s < r.n; s++) {
            r.off[s] = o;
            o += (long long)nf * (axis == 1 ? (long long)r.count[s] * n2 : (long long)n1 * r.count[s]) * Kz;
        }
        return r;
    }
    // The y and z passes run on this rank's x planes: swap the x-slab geometry and S1 buffer in.
    static void slab_swap(spns_handle *h) {
        std::swap(h->g, h->gx);
        std::swap(h->B1, h->B1x);
    }
    // Phases of one step (advective arithmetic or LES; the caller exchanges the
    // staging arrays and reduces the scalars between phases, see include/spns.h):
    //   VEL_A  inverse x pass of u, v, w on this rank's ky rows; pack for the exchange
    //   VEL_B  unpack; inverse y pass and z pass of u, v, w on this rank's x planes (CFL maxima)
    //   DT     time step from the maxima reduced over the ranks
    //   A      [forced shells' energy of this slab]; inverse x pass; pack
    //   B      unpack; [forcing amplitude]; inverse y, z and forward y passes; pack back
    //   C      unpack; forward x pass; spectral sweep; end of the step
    static int slab_phase(spns_handle *h, int phase) {
        const spns::Geo gy = h->g, gx = h->gx;
        const int ny = gy.Ky, Mx = gy.Mx, Ky = gx.Ky, nx = gx.Mx, Kz = gy.Kz;
        const bool les = h->a.isLES;
        const int mode = les ? spns::MODE_LES : spns::MODE_ADV;
        const int nf1 = spns::Fields<spns::MODE_ADV>::K1;                        // 6 (advective and LES)
        const int nf4 = les ? spns::Fields<spns::MODE_LES>::K4 : spns::Fields<spns::MODE_ADV>::K4;
        const spns::SlabRanges fwd_pack3 = slab_offsets(h->xr, 3, ny, Mx, Kz, 2), fwd_unpack3 = slab_offsets(h->yr, 3, Ky, nx, Kz, 1);
        const spns::SlabRanges fwd_pack = slab_offsets(h->xr, nf1, ny, Mx, Kz, 2), fwd_unpack = slab_offsets(h->yr, nf1, Ky, nx, Kz, 1);
        const spns::SlabRanges back_pack = slab_offsets(h->yr, nf4, Ky, nx, Kz, 1), back_unpack = slab_offsets(h->xr, nf4, ny, Mx, Kz, 2);
        int r = SPNS_OK;
        auto xpasses = [&](auto body) -> int {
            slab_swap(h);
            const int rr = body();
            slab_swap(h);
            return rr;
        };
        switch (phase) {
        case SPNS_SLAB_VEL_A:
            LAUNCH(pass(h, 1, spns::MODE_VEL, false));
            LAUNCH(slab_pack(h, h->B1, h->XS, 3, ny, Mx, fwd_pack3, 2, 0));
            return SPNS_OK;
        case SPNS_SLAB_VEL_B:
            LAUNCH(slab_pack(h, h->B1x, h->XR, 3, Ky, nx, fwd_unpack3, 1, 1));
            r = xpasses([&]() -> int {
                LAUNCH(pass(h, 2, spns::MODE_VEL, false));
                LAUNCH(pass(h, 3, spns::MODE_VEL, false));
                return SPNS_OK;
            });
            return r;
        case SPNS_SLAB_DT:
            spns::k_recalc_dt<<<1, 1, 0, h->st>>>(h->c, h->ds);
            CKL();
            return SPNS_OK;
        case SPNS_SLAB_A:
            if (h->a.eps_forcing > 0.0) {
                spns::k_eps_band<T><<<1, spns::EPS_BAND_THREADS, 0, h->st>>>(gy, U(h, 0), U(h, 1), U(h, 2), Ulo(h, 0), Ulo(h, 1), Ulo(h, 2),
                                                                          h->a.eps_kmin, h->a.eps_kmax, h->a.eps_forcing, h->ds, 1);
                CKL();
            }
            LAUNCH(pass(h, 1, mode, false));
            LAUNCH(slab_pack(h, h->B1, h->XS, nf1, ny, Mx, fwd_pack, 2, 0));
            return SPNS_OK;
        case SPNS_SLAB_B:
            LAUNCH(slab_pack(h, h->B1x, h->XR, nf1, Ky, nx, fwd_unpack, 1, 1));
            if (h->a.eps_forcing > 0.0) {
                spns::k_eps_alpha<<<1, 1, 0, h->st>>>(h->a.eps_forcing, h->ds);
                CKL();
            }
            r = xpasses([&]() -> int {
                LAUNCH(pass(h, 2, mode, false));
                LAUNCH(pass(h, 3, mode, false));
                LAUNCH(pass(h, 4, mode, false));
                return SPNS_OK;
            });
            if (r) return r;
            LAUNCH(slab_pack(h, h->B1x, h->XS, nf4, Ky, nx, back_pack, 1, 0));
            return SPNS_OK;
        case SPNS_SLAB_C:
            LAUNCH(slab_pack(h, h->B1, h->XR, nf4, ny, Mx, back_unpack, 2, 1));
            LAUNCH(pass(h, 5, mode, false));
            LAUNCH(launch_k6(h));
            spns::k_finish_step<<<1, 1, 0, h->st>>>(h->c, h->ds);
            CKL();
            return SPNS_OK;
        default:
            return spns_fail(h, SPNS_ERR_INVALID_ARGUMENT, "unknown slab phase %d", phase);
        }
    }

    // ---- batched step of same-class boxes (ensembles) ----
    // Every member of the table has h0's geometry, form, launch shapes and the
    // Adams-Bashforth scheme without constant-power forcing or edge correction.
    static int batch_step(spns_handle *h, const spns::BatchMember *tab, int n, cudaStream_t st) {
        const int mode = h->a.isLES ? spns::MODE_LES : spns::MODE_ADV;
        for (int k = 1; k <= 5; k++) LAUNCH(spns_len_table<T>(pass_length(h, k))->batch(h, tab, n, st, k, mode));
        {
            const int nk = h->g.Kx * h->g.Kz;
            spns::k6_sweep_batch<T><<<dim3((nk + 255) / 256, h->g.Ky, n), 256, 0, st>>>(h->g, tab);
            CKL();
        }
        spns::k_finish_step_batch<<<n, 1, 0, st>>>(tab);
        CKL();
        return SPNS_OK;
    }

    static constexpr PrecOps ops() {
        return PrecOps{&step_once, &run_velocity, &shell_sums, &forcing_scale, &conj_correction, &seed_draw, &invariant_spectra,
                       &slab_phase, &batch_step};
    }
};
