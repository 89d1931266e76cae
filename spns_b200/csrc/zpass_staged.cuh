// zpass_staged.cuh -- the rotational-form z pass, whose blocks walk the grid, with
// its input pairs staged by bulk asynchronous copies.
//
// Same arithmetic as k3_z<MODE_ROT> (solver_kernels.cuh): c2r of the six real
// fields u, v, w, w_x, w_y, w_z as three 2-for-1 complex transforms, the
// product c = w x u and the CFL maxima on the grid, r2c of c truncated to
// kz <= hz (src/HIT_LES.cpp:74-125 up to the gradient the projection removes).
// What differs is the schedule:
//   * One block per SM at a time, of independent units: one or several pencils (Q = L/E
//     threads each) that fill one to four warps.  Each unit walks the
//     pencils with the stride of the grid (LenLaunch::walking_blocks), with its own staging, mbarrier and exchange
//     barrier.  Only the two fields of the next input pair are staged in shared memory, by
//     cp.async.bulk (TMA bulk copies global -> shared, completion counted in bytes on an
//     mbarrier), while the current pair is transformed; the first pair of the next pencils
//     is fetched during the last transforms.
//     In single precision (T = f2) a thread transforms two neighbouring pencils with
//     packed arithmetic.
//   * The four physical slots (u, v, w_x, w_y) are thread-private and live in tensor
//     memory beside the running CFL maxima (104 columns a warp).  Two of them took 48 of
//     the 168 registers and two 12 KB of shared memory per pencil at length 768, which held the
//     pass to 12 warps per SM; now it is 16, and the slots' accesses leave the
//     shared-memory pipe, the busiest one (77 % of its cycles; the FP64 pipe 44 %).
//     Before and now: double 512^3 13.0 -> 11.5 ms, single 8.25 -> 7.2 (6.7 in waves).
//   * c_z is transformed as soon as it is known (after the second pair) and written
//     over the w_x field of the same pencil (S2 field 3, consumed at the first
//     pair), so the forward y pass reads the nonlinear term from fields 0, 1, 3.
//   * CFL maxima accumulate per thread over all pencils and are reduced once per
//     block at the end.
// Every mbarrier wait is bounded; a wait that gives up records wait_timeout in
// the solver scalars (reported as SPNS_ERR_TIMEOUT by the host) and the unit
// skips its remaining pencils.  The copies that it waited for may still be on
// their way then, into shared memory that the SM hands to its next block, so the
// unit waits for them once more, as long as a wait may take, before it leaves.
#pragma once
#include "solver_kernels.cuh"

namespace spns {

__device__ __forceinline__ unsigned smem_addr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(unsigned long long *bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
// makes the barrier initialisation visible to the asynchronous (TMA) proxy
__device__ __forceinline__ void fence_mbar_init() { asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory"); }
// orders earlier generic-proxy accesses of shared memory before later async-proxy ones
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }
__device__ __forceinline__ void mbar_arrive_expect_tx(unsigned long long *bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
// bulk copy of `bytes` (multiple of 16, both addresses 16-byte aligned) from global to shared memory
__device__ __forceinline__ void bulk_copy_g2s(void *dst, const void *src, unsigned bytes, unsigned long long *bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(smem_addr(dst)),
                 "l"(src), "r"(bytes), "r"(smem_addr(bar))
                 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long *bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Polls the barrier phase `parity` at most `limit` times (each poll may suspend the
// thread for a short, hardware-defined time); false if it did not complete.
__device__ __forceinline__ bool mbar_wait_bounded(unsigned long long *bar, unsigned parity, int limit) {
    for (int i = 0; i < limit; i++)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}

constexpr int ZS_WAIT_LIMIT = 1 << 22;   // polls of a wait

// ---------------------------------------------------------------------------
// Thread-private values in tensor memory.  A warp may store and load 32-bit columns of its
// own 32 lanes (shape 32x32b: lane i of the warp, its rank in the block modulo 4 selecting
// the lanes), so an allocation of C columns is C words of storage for each of 128 lanes
// beside registers and shared memory, with its own path to the SM.
// ---------------------------------------------------------------------------
// One whole warp; the address (columns' base) is written to shared memory.
template <int COLS> __device__ __forceinline__ void tmem_alloc(unsigned *dst) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_addr(dst)), "n"(COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
}
template <int COLS> __device__ __forceinline__ void tmem_free(unsigned addr) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(addr), "n"(COLS) : "memory");
}
// Tensor-memory accesses of different warps are ordered by a barrier only between these two:
// the one before it after a warp's own accesses, the other after it before what depends on them.
__device__ __forceinline__ void tmem_fence_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tmem_fence_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ unsigned long long bits64(double v) { return (unsigned long long)__double_as_longlong(v); }
__device__ __forceinline__ unsigned long long bits64(f2 v) { return v.v; }
__device__ __forceinline__ void from_bits64(unsigned long long b, double &v) { v = __longlong_as_double((long long)b); }
__device__ __forceinline__ void from_bits64(unsigned long long b, f2 &v) { v.v = b; }
// four 64-bit values of the thread to / from 8 columns; a load's values are defined after tmem_wait_ld
template <typename T> __device__ __forceinline__ void tmem_st4(unsigned addr, T a, T b, T c, T d) {
    const unsigned long long v[4] = {bits64(a), bits64(b), bits64(c), bits64(d)};
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n" ::"r"(addr), "r"((unsigned)v[0]),
                 "r"((unsigned)(v[0] >> 32)), "r"((unsigned)v[1]), "r"((unsigned)(v[1] >> 32)), "r"((unsigned)v[2]),
                 "r"((unsigned)(v[2] >> 32)), "r"((unsigned)v[3]), "r"((unsigned)(v[3] >> 32))
                 : "memory");
}
struct Tmem4 { unsigned r[8]; };
__device__ __forceinline__ void tmem_ld4(unsigned addr, Tmem4 &v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
                 : "=r"(v.r[0]), "=r"(v.r[1]), "=r"(v.r[2]), "=r"(v.r[3]), "=r"(v.r[4]), "=r"(v.r[5]), "=r"(v.r[6]), "=r"(v.r[7])
                 : "r"(addr)
                 : "memory");
}
// completes the loads; the values pass through it, so no use moves above
__device__ __forceinline__ void tmem_wait_ld(Tmem4 &v) {
    asm volatile("tcgen05.wait::ld.sync.aligned;\n"
                 : "+r"(v.r[0]), "+r"(v.r[1]), "+r"(v.r[2]), "+r"(v.r[3]), "+r"(v.r[4]), "+r"(v.r[5]), "+r"(v.r[6]), "+r"(v.r[7])::"memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }
template <typename T> __device__ __forceinline__ T tmem_value(const Tmem4 &v, int i) {
    T x;
    from_bits64((unsigned long long)v.r[2 * i] | ((unsigned long long)v.r[2 * i + 1] << 32), x);
    return x;
}

// One block per SM of up to ZSTAGED_THREADS threads (the runtime places one block with
// tensor memory per SM, so the SM's warps are one block).  A unit is a warp with 32/Q
// pencils (pairs of pencils, T = f2), the two warps of one (Q = 64) or three warps of four (Q = 24); each unit has the
// exchange buffers of its pencils, 2 staging fields (rows of the work buffers' pitch Kp, the
// last without its padding) and an mbarrier; one word for the block's tensor-memory address.
constexpr int ZSTAGED_THREADS = 512;
constexpr int whole_warps(int q) { return q % 32 == 0 ? q : 32 % q == 0 ? 32 : 96; }   // q = 24: four pencils in three warps
template <typename T, int L, int E> struct ZStagedLayout {
    static constexpr int Q = L / E, W = Arith<T>::W, U = whole_warps(Q), PPU = U / Q;
    using SM = SmPencil<T, L, E>;
    static_assert((U == 32 || U == 64 || U == 96 || U == 128) && U % Q == 0, "a unit's pencils fill one to four warps");
    static_assert(E == 12, "twelve values a thread: three tensor-memory accesses of four per slot");
    static constexpr unsigned BAR = U == 32 ? 1u : GROUP + U;
    static constexpr int COLS = 512;                 // all of the SM's; 128 (of 104 used) for each of the 4 warps of a lane quarter
    // every compiled length is a multiple of 8 (and so are the rows of a field, of a slab too): no unit is partly filled
    static_assert(8 % (PPU * W) == 0, "rows of a unit");
    // the unit's rows of one field, the last without its padding (whole 16-byte units, as Kp is)
    __host__ __device__ static constexpr size_t stage_bytes(int Kz, int Kp) {
        constexpr int A = 16 / (int)sizeof(SCx<T>);
        return (size_t)((PPU * W - 1) * Kp + (Kz + A - 1) / A * A) * sizeof(SCx<T>);
    }
    static constexpr size_t EXCH = (size_t)PPU * SM::PITCH * sizeof(cx<T>);
    __host__ __device__ static constexpr size_t unit_bytes(int Kz, int Kp) { return EXCH + 2 * stage_bytes(Kz, Kp) + sizeof(unsigned long long); }
    __host__ __device__ static constexpr size_t smem_bytes(int units, int Kz, int Kp) { return units * unit_bytes(Kz, Kp) + 16; }
    static constexpr size_t SMEM_MAX = 225 * 1024 + 16;   // of any box
    // most units of a block
    __host__ __device__ static constexpr int max_units(int Kz, int Kp) {
        const int s = (int)((SMEM_MAX - 16) / unit_bytes(Kz, Kp)), t = ZSTAGED_THREADS / U;
        return s < t ? s : t;
    }
};

// true on every thread of the unit if `ok` is on all of them (a barrier of the group)
template <int U> __device__ __forceinline__ bool unit_all(bool ok) {
    if constexpr (U == 32) {
        return __all_sync(0xffffffffu, ok) != 0;
    } else {
        unsigned r;
        asm volatile("{\n.reg .pred p, r;\nsetp.ne.u32 p, %1, 0;\nbar.red.and.pred r, %2, %3, p;\nselp.u32 %0, 1, 0, r;\n}\n"
                     : "=r"(r)
                     : "r"((unsigned)ok), "r"(1 + threadIdx.x / U), "n"(U)
                     : "memory");
        return r != 0;
    }
}

template <typename T, int L, int E>
__global__ void __launch_bounds__(ZSTAGED_THREADS, 1) k3_rot_staged(Geo g, SCx<T> *__restrict__ buf, StepConsts c, DevScalars *ds,
                                                        const cx<T> *__restrict__ tw, int polls) {
    using LY = ZStagedLayout<T, L, E>;
    constexpr int Q = LY::Q, W = LY::W, U = LY::U, PPU = LY::PPU;
    constexpr unsigned BAR = LY::BAR;
    extern __shared__ __align__(128) unsigned char smraw_zs[];
    const int tid = threadIdx.x, unit = tid / U, units = blockDim.x / U, sub = tid % U / Q, q0 = tid % Q;
    const int Kz = g.Kz, Kp = g.Kp;
    const size_t sb = LY::stage_bytes(Kz, Kp);
    unsigned char *const mine = smraw_zs + unit * (LY::EXCH + 2 * sb);
    typename LY::SM sm{reinterpret_cast<cx<T> *>(mine) + sub * LY::SM::PITCH};
    SCx<T> *const stA = reinterpret_cast<SCx<T> *>(mine + LY::EXCH);             // staging: field a of the pair
    SCx<T> *const stB = reinterpret_cast<SCx<T> *>(mine + LY::EXCH + sb);        // field b
    unsigned long long *const bars = reinterpret_cast<unsigned long long *>(smraw_zs + units * (LY::EXCH + 2 * sb)), *const bar = bars + unit;
    unsigned *const taddr = reinterpret_cast<unsigned *>(bars + units);
    if (tid < 32) tmem_alloc<LY::COLS>(taddr);
    if (tid % U == 0) {
        mbar_init(bar, 1);
        fence_mbar_init();
    }
    tmem_fence_before_sync();
    __syncthreads();
    tmem_fence_after_sync();
    // this warp's lanes and columns; slots of 24 columns: 0 u, 1 v, 2 w_x, 3 w_y
    const unsigned tbase = *taddr;
    const unsigned slots = tbase + ((unsigned)(tid >> 5 & 3) << 21) + (unsigned)(tid >> 7) * 128u;

    const long long ngrp = (long long)g.Mx * g.My / (PPU * W), step = (long long)gridDim.x * units;
    const T sz = T(g.sz);
    unsigned parity = 0;
    bool bad = false;
    // running CFL maxima of the thread: four doubles in columns 96..103
    tmem_st4<double>(slots + 96, 0.0, 0.0, 0.0, 0.0);
    tmem_wait_st();

    // stage fields fa, fb of the PPU pencils of group grp (their rows are contiguous in each field)
    auto issue = [&](long long grp, int fa, int fb) {
        if (tid % U != 0) return;
        const unsigned bytes = (unsigned)sb;
        const SCx<T> *p = buf + grp * (PPU * W) * Kp;
        fence_proxy_async_smem();
        mbar_arrive_expect_tx(bar, 2 * bytes);
        bulk_copy_g2s(stA, p + fa * g.S2, bytes, bar);
        bulk_copy_g2s(stB, p + fb * g.S2, bytes, bar);
    };
    // the staged pair is complete and visible to every thread of the unit
    auto wait_stage = [&]() -> bool {
        const bool ok = mbar_wait_bounded(bar, parity, polls);
        parity ^= 1u;
        return unit_all<U>(ok);
    };

    long long grp = (long long)blockIdx.x * units + unit;
    if (grp < ngrp) issue(grp, 0, 3);
    for (; grp < ngrp; grp += step) {
        const int q = opaque(q0);
        SCx<T> *const B0 = buf + (grp * PPU + sub) * W * Kp;
        const SCx<T> *const sa = stA + sub * W * Kp, *const sb_ = stB + sub * W * Kp;
        cx<T> A[E];
        // pair 0: u + i w_x
        if (!wait_stage()) { bad = true; break; }
        k3_load_pair<T, L, E>(A, sa, false, sb_, false, Kz, sz, q, true, Kp);
        stage_barrier<BAR>();
        issue(grp, 1, 4);
        fft<T, L, E, true, typename LY::SM, BAR>(A, sm, q, tw);
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 3; i++) {
            tmem_st4<T>(slots + 8 * i, A[4 * i].x, A[4 * i + 1].x, A[4 * i + 2].x, A[4 * i + 3].x);
            tmem_st4<T>(slots + 48 + 8 * i, A[4 * i].y, A[4 * i + 1].y, A[4 * i + 2].y, A[4 * i + 3].y);
        }
        tmem_wait_st();
        // pair 1: v + i w_y; then c_z = w_x v - w_y u, transformed and written over w_x (field 3)
        if (!wait_stage()) { bad = true; break; }
        k3_load_pair<T, L, E>(A, sa, false, sb_, false, Kz, sz, q, true, Kp);
        stage_barrier<BAR>();
        issue(grp, 2, 5);
        fft<T, L, E, true, typename LY::SM, BAR>(A, sm, q, tw);
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 3; i++) {
            Tmem4 tu, tx;
            tmem_ld4(slots + 8 * i, tu);
            tmem_ld4(slots + 48 + 8 * i, tx);
            tmem_st4<T>(slots + 24 + 8 * i, A[4 * i].x, A[4 * i + 1].x, A[4 * i + 2].x, A[4 * i + 3].x);
            tmem_st4<T>(slots + 72 + 8 * i, A[4 * i].y, A[4 * i + 1].y, A[4 * i + 2].y, A[4 * i + 3].y);
            tmem_wait_ld(tu);
            tmem_wait_ld(tx);
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int e = 4 * i + k;
                A[e] = mk<T>(tmem_value<T>(tx, k) * A[e].x - A[e].y * tmem_value<T>(tu, k), T(0));
            }
        }
        tmem_wait_st();
        fft<T, L, E, false, typename LY::SM, BAR>(A, sm, q, tw);
        {
            SCx<T> *o = B0 + 3 * g.S2;
#pragma unroll
            for (int e = 0; e < E; e++) {
                const int row = out_row<L, E, false>(q, e);
                if (row < Kz) st_pencil(o, row, Kp, A[e]);
            }
        }
        // pair 2: w + i w_z; then (c_x, c_y) and the CFL maxima
        if (!wait_stage()) { bad = true; break; }
        k3_load_pair<T, L, E>(A, sa, false, sb_, false, Kz, sz, q, true, Kp);
        stage_barrier<BAR>();
        if (grp + step < ngrp) issue(grp + step, 0, 3);
        fft<T, L, E, true, typename LY::SM, BAR>(A, sm, q, tw);
        __syncwarp();
        Tmem4 tm;
        tmem_ld4(slots + 96, tm);
        tmem_wait_ld(tm);
        double mx[4] = {tmem_value<double>(tm, 0), tmem_value<double>(tm, 1), tmem_value<double>(tm, 2), tmem_value<double>(tm, 3)};
#pragma unroll
        for (int i = 0; i < 3; i++) {
            Tmem4 tu, tv, tx, ty;
            tmem_ld4(slots + 8 * i, tu);
            tmem_ld4(slots + 24 + 8 * i, tv);
            tmem_ld4(slots + 48 + 8 * i, tx);
            tmem_ld4(slots + 72 + 8 * i, ty);
            tmem_wait_ld(tu);
            tmem_wait_ld(tv);
            tmem_wait_ld(tx);
            tmem_wait_ld(ty);
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int e = 4 * i + k;
                const T ww = A[e].x, oz = A[e].y, uu = tmem_value<T>(tu, k), vv = tmem_value<T>(tv, k);
                cfl_rows(mx, uu, vv, ww, c);
                A[e] = mk<T>(tmem_value<T>(ty, k) * ww - oz * vv, oz * uu - tmem_value<T>(tx, k) * ww);
            }
        }
        tmem_st4<double>(slots + 96, mx[0], mx[1], mx[2], mx[3]);
        tmem_wait_st();
        // forward transform of c_x + i c_y and extraction of both half spectra, kz < Kz
        fft<T, L, E, false, typename LY::SM, BAR>(A, sm, q, tw);
        stage_barrier<BAR>();
#pragma unroll
        for (int e = 0; e < E; e++) sm.at(out_row<L, E, false>(q, e)) = A[e];
        stage_barrier<BAR>();
        {
            const T h = T(0.5);
            SCx<T> *oa = B0, *ob = B0 + g.S2;
            for (int k = q; k < Kz; k += Q) {
                const cx<T> zk = sm.at(k), zm = sm.at(k == 0 ? 0 : L - k);
                st_pencil(oa, k, Kp, mk<T>(h * (zk.x + zm.x), h * (zk.y - zm.y)));
                st_pencil(ob, k, Kp, mk<T>(h * (zk.y + zm.y), h * (zm.x - zk.x)));
            }
        }
    }
    if (bad) {
        mbar_wait_bounded(bar, parity ^ 1u, ZS_WAIT_LIMIT);   // the phase that the failed wait was for
        if (tid % U == 0) atomicExch(&ds->wait_timeout, 1);
    }
    __syncwarp();
    Tmem4 tm;
    tmem_ld4(slots + 96, tm);
    tmem_wait_ld(tm);
    const double mx[4] = {tmem_value<double>(tm, 0), tmem_value<double>(tm, 1), tmem_value<double>(tm, 2), tmem_value<double>(tm, 3)};
    tmem_fence_before_sync();
    block_max4<T>(mx, ds);   // (a block barrier: every warp is done with the tensor memory)
    tmem_fence_after_sync();
    if (tid < 32) tmem_free<LY::COLS>(tbase);
}

} // namespace spns
