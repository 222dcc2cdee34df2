// Resident step kernel: whole solves of small meshes in one cooperative launch.
//
// On a mesh of up to ~130,000 cells (FP64; ~250,000 in FP32; the largest wedges of triangles that fit
// 148 SMs are 361x181 and 501x251 nodes) a step of the tiled kernels is two launches, each filling barriers, descriptors and copies before its few tiles per CTA and
// draining after them, far from its bytes or operations.  Here every SM holds one tile in shared
// memory (state, limited gradients, face records, fluxes, slots) for all steps of a call.
//
//   half 1: gradient, limiter, CFL of the tile's cells (Pass1Cell, as pass 1); the limited
//           gradients stay in shared memory
//   half 2: flux per face entry, then sum and update per cell, ghosts (FaceIn, cell_flux_sum,
//           cell_update, as pass 2)
//
// What crosses tiles goes through L2 as stamped words (see ll_store), with no grid barrier: the
// state and limited gradient of the cells in another tile's halo, and under a global CFL number
// each tile's largest iv lam.  A grid barrier (fence, counter, poll) measured 3,500-5,500 cycles
// and the loads behind it 900-1,400; a stamped word arrives in about 1,400, and the CFL words
// travel while the fluxes are computed.
//
// The arithmetic is that of the tiled kernels, function for function: a state depends on which of them
// stepped it by no more than the fused multiply-adds the compiler picks in each (1e-13 in FP64 and 1e-6 in
// FP32 over a few steps).
//
// Measured (one step of a long call, B200; the tiled kernels beside it): 161x81 nodes FP64 6.2 us
// against 11.7 (18.5 when each of its launches waited for the one before and its producer warp for
// its loads), FP32 4.9 against 8.0; 333x178 FP64 15.1 against 19.8; at the largest sizes that fit,
// 361x181 FP64 15.5 against 20.1 and 501x251 FP32 13.4 against 17.1.
//
// What bounds it: at 26,000 cells (184 a tile) a chain of latencies, of 12,000 cycles a step about
// 3,000 for gradient and limiter, 1,500 for a flux, 1,400 for the update (FP64 operations at some
// 20 cycles each, quotients and square roots among them) and 1,000-1,500 for each exchange; 27 % of
// issue slots are used.  At 800 cells a tile, issue (35-57 % within the phases).
//
// Tiles wait for one another, so the grid must be co-resident: the host launches it
// cooperatively, one CTA per tile, at most one per SM.  Every wait is bounded; one that gives
// up sets the error word, which every other wait polls, and all CTAs leave (the copies into a
// CTA's shared memory are waited for first).
#pragma once
#include "hcfd_tile.cuh"

namespace hcfd {

constexpr int kResidentThreads = 512;       // 128 registers a thread, what the two halves need in FP64

// Flags per cell.
constexpr unsigned char kCellExported = 1, kCellHasGhost = 2, kCellIsGhost = 4;

struct ResidentArgs {
    const unsigned char* __restrict__ flags;      // [ntiles * B]
    ulonglong2* llU;                              // exchanged states: 8 bytes a word pair, cell-major
    ulonglong2* llG;                              // exchanged limited gradients
    ulonglong2* llX;                              // [2][ntiles]: largest iv lam of a tile, by step parity
    unsigned int epoch;                           // stamp of this launch's first step (later launches' are larger)
    unsigned long long* dtmin;                    // local time stepping, profiling: +inf between whole steps
    double* partial_first;                        // [grid]: residual partials of the first step since initialise
    int nsteps;
    int phases;                                   // 3: whole steps; 1 or 2: one half of one step (profiling)
    int refetch;                                  // fluxes overwrite the r vectors, which are fetched again each step
};

// Shared memory of one tile (all offsets multiples of 128 bytes).  With `refetch` the fluxes have
// no room of their own (they take the r vectors' place, as in pass 2).
template <class T>
struct ResidentSmem {
    size_t u, g, geo, flux, meta, nbr, iv, dt, flags, halo, total;
    __host__ __device__ ResidentSmem(int B, int Hmax, int Fmax, int Wp, bool refetch) {
        size_t p = kHeader;
        u = p;        p += align128((size_t) (B + Hmax) * sizeof(Cell4<T>));
        g = p;        p += align128((size_t) (B + Hmax) * sizeof(Grad8<T>));
        geo = p;      p += align128((size_t) Fmax * sizeof(FaceGeo<T>));
        flux = p;     p += refetch ? 0 : align128((size_t) Fmax * sizeof(Cell4<T>));
        meta = p;     p += align128((size_t) Fmax * 4);
        nbr = p;      p += align128((size_t) B * Wp * sizeof(unsigned));
        iv = p;       p += align128((size_t) B * sizeof(T));
        dt = p;       p += align128((size_t) B * sizeof(T));          // local time steps
        flags = p;    p += align128((size_t) B);
        halo = p;     p += align128((size_t) Hmax * sizeof(int));
        total = p;
    }
};

// Stamped words (the method of NCCL's LL protocol, payload and flag in one atomic word, in code and stamps of
// this library's own): 8 bytes of payload travel as two 64-bit words, each 32 bits of payload under
// the step's stamp.  A 64-bit access is single-copy atomic, so a word that carries the stamp
// carries its payload: no fence, flag or barrier orders the exchange.  A slot is free for the next
// step when its reader has answered with data of its own that depends on it: neighbours exchange
// states and gradients in turn, and each needs the other's last answer to go on, so one buffer of
// each is enough; the CFL words of a step are read by every tile before any tile can publish those
// of the step after the next, so they take two.
__device__ __forceinline__ void ll_store(ulonglong2* p, unsigned long long x, unsigned stamp) {
    const unsigned long long st = (unsigned long long) stamp << 32;
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"((x & 0xFFFFFFFFULL) | st), "l"((x >> 32) | st)
                 : "memory");
}
__device__ __forceinline__ bool ll_load(const ulonglong2* p, unsigned stamp, unsigned long long& x, unsigned polls,
                                        unsigned* err) {
#pragma unroll 1
    for (unsigned i = 0; i < polls; i++) {
        unsigned long long a, b;
        asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
        if ((unsigned) (a >> 32) == stamp && (unsigned) (b >> 32) == stamp) {
            x = (a & 0xFFFFFFFFULL) | (b << 32);
            return true;
        }
        if ((i & 63u) == 63u && *(volatile unsigned*) err) return false;
    }
    atomicOr(err, 1u);
    return false;
}
__device__ __forceinline__ unsigned long long payload(double x) { return (unsigned long long) __double_as_longlong(x); }
__device__ __forceinline__ unsigned long long payload(float x, float y) {
    return (unsigned long long) __float_as_uint(x) | ((unsigned long long) __float_as_uint(y) << 32);
}
// n values (even) from word pair k0 of a cell's record at p.
template <int n>
__device__ __forceinline__ void ll_values(ulonglong2* p, int k0, const double* x, unsigned stamp) {
#pragma unroll
    for (int i = 0; i < n; i++) ll_store(p + k0 + i, payload(x[i]), stamp);
}
template <int n>
__device__ __forceinline__ void ll_values(ulonglong2* p, int k0, const float* x, unsigned stamp) {
#pragma unroll
    for (int i = 0; i < n / 2; i++) ll_store(p + k0 / 2 + i, payload(x[2 * i], x[2 * i + 1]), stamp);
}

// Halo records of a step into chunk planes of stride NL, from local cell B on, by threads t of n:
// 8 bytes a thread.  Ghosts in the halo (ids stored complemented) are refreshed by this tile itself.
template <class R>
__device__ __forceinline__ bool halo_receive(R* s, int NL, int B, const ulonglong2* ll, const int* sHalo, int nh, int t, int n,
                                             unsigned stamp, unsigned polls, unsigned* err) {
    constexpr int K = sizeof(R) / 8;
    unsigned long long* d = reinterpret_cast<unsigned long long*>(s);
    bool ok = true;
    for (int q = t; q < nh * K; q += n) {
        const int h = q / K, k = q % K, ci = sHalo[h];
        if (ci < 0) continue;
        unsigned long long x = 0;
        if (!ll_load(ll + (size_t) ci * K + k, stamp, x, polls, err)) { ok = false; break; }
        d[2 * ((k >> 1) * NL + B + h) + (k & 1)] = x;
    }
    return ok;
}

// Largest of a warp's values >= 0 (their bit patterns order them).
__device__ __forceinline__ float warp_max_pos(float x) {
    return __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(x)));
}
__device__ __forceinline__ double warp_max_pos(double x) {
    const unsigned long long b = (unsigned long long) __double_as_longlong(x);
    const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned) (b >> 32));
    const unsigned lo = __reduce_max_sync(0xffffffffu, (unsigned) (b >> 32) == hi ? (unsigned) b : 0u);
    return __longlong_as_double((long long) (((unsigned long long) hi << 32) | lo));
}

// Smallest of n stamped doubles >= 0, by one warp, up to five words a lane in flight at once.
__device__ __forceinline__ bool ll_least(const ulonglong2* p, int n, unsigned stamp, double& least_out, unsigned polls,
                                         unsigned* err) {
    constexpr int U = 5;
    const int lane = threadIdx.x & 31;
    double m = __longlong_as_double(0x7FF0000000000000LL);
    bool ok = true;
    for (int i0 = 0; i0 < n && ok; i0 += 32 * U) {
        unsigned i = 0;
        for (bool all = false; !all; i++) {
            unsigned long long a[U], b[U];
#pragma unroll
            for (int k = 0; k < U; k++) {
                const int at = i0 + 32 * k + lane;
                a[k] = b[k] = (unsigned long long) stamp << 32 | 0x7FF00000u;
                if (at < n)
                    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(a[k]), "=l"(b[k]) : "l"(p + at) : "memory");
                else
                    a[k] = (unsigned long long) stamp << 32;
            }
            all = true;
            double t = m;
#pragma unroll
            for (int k = 0; k < U; k++) {
                all = all && (unsigned) (a[k] >> 32) == stamp && (unsigned) (b[k] >> 32) == stamp;
                t = least(t, __longlong_as_double((long long) ((a[k] & 0xFFFFFFFFULL) | (b[k] << 32))));
            }
            all = __all_sync(0xffffffffu, all);
            if (all) m = t;
            else if (i >= polls || ((i & 63u) == 63u && __any_sync(0xffffffffu, *(volatile unsigned*) err))) { ok = false; break; }
        }
    }
    if (!ok) atomicOr(err, 1u);
    least_out = warp_min_pos(m);
    return ok;
}

// Block sum in a fixed order: per warp by shuffles, then the warps in order.  sm: 32 doubles.
__device__ __forceinline__ double block_sum(double x, double* sm) {
    x = warp_sum(x);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = x;
    __syncthreads();
    double t = 0.0;
    for (int w = 0; w < (int) (blockDim.x >> 5); w++) t += sm[w];
    return t;
}

// NVAR 2: two threads per cell, each with one pair of variables (gradient, limiter, flux sum and
// update are independent per variable), for tiles of at most 256 cells, whose steps are a chain
// of latencies with one or two warps per scheduler (161x81: FP64 6.2 us a step against 7.6 with a
// thread per cell, FP32 4.9 against 5.1); NVAR 4: a thread per cell.
// One CTA per SM: the tile takes most of an SM's shared memory at the upper end, and at the lower
// end more CTAs would only add halo.
template <class T, int W, int NVAR>
__global__ void __launch_bounds__(kResidentThreads, 1) resident_kernel(const TileArgs<T> a, const ResidentArgs r) {
    constexpr bool COMP = sizeof(T) == 4;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ double red[32], red3[32], s_dt;
    __shared__ int s_bad;
    __shared__ bool s_last;
    const bool refetch = r.refetch != 0;
    const ResidentSmem<T> L(a.B, a.Hmax, a.Fmax, a.Wp, refetch);
    const StepArgs<T>& s = a.s;
    const int NT = blockDim.x, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int NL = a.B + a.Hmax, Bp = (a.B + 31) & ~31;
    int base, nb, f0, nf, h0, nh, inst;
    tile_info<false>(a, (int) blockIdx.x, base, nb, f0, nf, h0, nh, inst);
    bool good = true;
    if constexpr (kChecked) {
        good = index_ok(nb >= 0 && nb <= a.B && base + nb <= a.ps && base + a.B <= a.ncap && f0 >= 0 && nf >= 0 &&
                        nf <= a.Fmax && f0 + nf <= a.nentries && h0 >= 0 && nh >= 0 && nh <= a.Hmax &&
                        h0 + nh <= a.nhalo, a.err);
        if (!good) nb = nf = nh = 0;
    }
    Cell4<T>* sU = reinterpret_cast<Cell4<T>*>(smem + L.u);
    Grad8<T>* sG = reinterpret_cast<Grad8<T>*>(smem + L.g);
    T* sGeo = reinterpret_cast<T*>(smem + L.geo);
    T* sF = refetch ? sGeo + 4 * nf : reinterpret_cast<T*>(smem + L.flux);
    unsigned* sMeta = reinterpret_cast<unsigned*>(smem + L.meta);
    unsigned* sNbr = reinterpret_cast<unsigned*>(smem + L.nbr);
    T* sIv = reinterpret_cast<T*>(smem + L.iv);
    T* sDt = reinterpret_cast<T*>(smem + L.dt);
    unsigned char* sFlag = smem + L.flags;
    int* sHalo = reinterpret_cast<int*>(smem + L.halo);
    Cell4<T>* gU = const_cast<Cell4<T>*>(s.U);
    unsigned long long* full = reinterpret_cast<unsigned long long*>(smem);
    constexpr int CU = sizeof(Cell4<T>) / 16, CG = sizeof(Grad8<T>) / 16;
    constexpr int KU = sizeof(Cell4<T>) / 8, KG = sizeof(Grad8<T>) / 8;

    // the tile: bulk copies of its contiguous blocks, halo ids and halo states by the threads
    if (tid == 0) {
        mbar_init(full, 1);
        *abort_word(smem) = 0;
        fence_mbar_init();
        s_bad = 0;
        if ((int) blockIdx.x != a.skip_tile) {       // failure injection for tests: nothing armed
            const unsigned bu = nb * 16u * CU, bg = r.phases == 2 ? nb * 16u * CG : 0u;
            const unsigned bf = nf * 8u * (unsigned) sizeof(T), bm = nf * 4u;
            const unsigned bs = good ? a.B * W * 4u : 0u, bi = good ? a.B * (unsigned) sizeof(T) : 0u;
            mbar_arrive_expect_tx(full, bu + bg + bf + bm + bs + bi);
            if (good) {
#pragma unroll
                for (int j = 0; j < CU; j++)
                    bulk_g2s(reinterpret_cast<uint4*>(sU) + j * NL, reinterpret_cast<const uint4*>(s.U) + ((size_t) j * a.ps + base),
                             nb * 16u, full);
                if (bg)
#pragma unroll
                    for (int j = 0; j < CG; j++)
                        bulk_g2s(reinterpret_cast<uint4*>(sG) + j * NL,
                                 reinterpret_cast<const uint4*>(s.phiG) + ((size_t) j * a.ps + base), nb * 16u, full);
                if (bf) {
                    bulk_g2s(sGeo, a.tgeo + (size_t) f0 * 8, bf, full);
                    bulk_g2s(sMeta, a.tmeta + f0, bm, full);
                }
                bulk_g2s(sNbr, a.nbr + (size_t) base * W, bs, full);
                bulk_g2s(sIv, s.iv + base, bi, full);
            }
        }
    }
    for (int c = tid; c < nb; c += NT) sFlag[c] = r.flags[base + c];
    for (int h = tid; h < nh; h += NT) {
        int ci = __ldg(a.halo + h0 + h);
        if (!index_ok(ci >= 0 && ci < a.ps, a.err)) ci = 0;
        sHalo[h] = (r.flags[ci] & kCellIsGhost) ? ~ci : ci;
        T u[4], g[8];
        ld_cell(s.U, a.ps, ci, u);
        st_cell(sU, NL, a.B + h, u);
        if (r.phases == 2) {
            ld_grad(s.phiG, a.ps, ci, g);
            st_grad(sG, NL, a.B + h, g);
        }
    }
    const long long steps0 = s.stats->steps;
    __syncthreads();
    // a wait that gives up is the whole CTA's; copies that were armed land (they read valid
    // memory) and are drained before leaving
    if (!__syncthreads_and(mbar_wait(full, 0, a.polls, a.err, abort_word(smem)))) {
        if (tid == 0 && (int) blockIdx.x != a.skip_tile) mbar_drain(full, 0, a.err);
        return;
    }
    if (r.phases == 2) {
        // no exchange of half 1 stands between these halo reads and the other CTAs' updates: wait for all tiles
        if (tid == 0) ll_store(r.llX + blockIdx.x, 0ULL, r.epoch);
        bool ok = true;
        unsigned long long x;
        for (int i = tid; i < (int) gridDim.x && ok; i += NT) ok = ll_load(r.llX + i, r.epoch, x, a.polls, a.err);
        if (!__syncthreads_and(ok)) return;
    }

    // The wave speeds of the coming step, from the state it starts with: local time steps, or the
    // tile's largest iv lam, left per warp in `red`.  Formed behind the update of the step before,
    // so that the tiles' words for a global CFL number travel during half 1 and the fluxes.
    auto wave_speeds = [&]() {
        if (s.time_mode == TM_FIXED) return;
        T xmx = T(0);
        for (int c = tid; c < nb; c += NT) {
            unsigned x[W];
            lds_nbr<W>(sNbr + c * W, x);
            if (x[0] == kNoFace) continue;
            T u[4];
            lds_cell(sU, NL, c, u);
            const T rate = sIv[c] * cell_wave_sum<T, W>(x, sGeo, nf, 8, u, s.gma, a.err);
            xmx = fmax(xmx, rate);
            if (s.time_mode == TM_LOCAL) sDt[c] = T(s.dt_or_cfl) * qrcp(rate);
        }
        xmx = warp_max_pos(xmx);
        if (lane == 0) red[wid] = (double) xmx;
    };
    wave_speeds();                                   // (warps without a cell leave 0)
    __syncthreads();

    double r2 = 0.0, dt_used = s.dt_or_cfl;
    int top = 0;
    for (int step = 0;; step++) {
        const bool last_step = step + 1 == r.nsteps;
        const unsigned stamp = r.epoch + (unsigned) step;
        bool ok = true;
        if (r.phases & 1) {
            const int lmode = limiter_mode(steps0 + step, s.freeze_after);
            for (int w = tid; w < (NVAR == 4 ? nb : Bp + nb); w += NT) {
                const int j = NVAR == 4 ? 0 : w >= Bp, c = w - j * Bp;
                if (NVAR != 4 && c >= nb) continue;
                unsigned x[W];
                lds_nbr<W>(sNbr + c * W, x);
                if (x[0] == kNoFace) continue;
                const T iv = sIv[c];
                Pass1Cell<T, NVAR> p;
                T ro[W][2];
                tile_faces<T, W, NVAR>(p, x, sU, sGeo, NL, nf, c, j, false, s.gma, iv, nb, a.B, nh, a.err, ro);
                T out[2 * NVAR], phis[NVAR];
                if (lmode == LIM_FROZEN) {
                    // perhaps written in this launch (by this thread): not through the read-only path
#pragma unroll
                    for (int h = 0; h < NVAR / 2; h++) {
                        const auto x = __ldcg(pair_at(s.phiF, a.ps, base + c, j + h));
                        phis[2 * h] = x.x; phis[2 * h + 1] = x.y;
                    }
                } else {
                    p.limiter_values(iv, s.limiter, s.venkat_K, phis);
                }
                p.limited(phis, out);
#pragma unroll
                for (int h = 0; h < NVAR / 2; h++) {
                    if (lmode == LIM_RECORD) {
                        auto* q = pair_at(s.phiF, a.ps, base + c, j + h);
                        q->x = phis[2 * h]; q->y = phis[2 * h + 1];
                    }
                    st_grad_pair(sG, NL, c, j + h, out + 4 * h);
                    if (r.phases == 1) st_grad_pair(s.phiG, a.ps, base + c, j + h, out + 4 * h);
                }
                if (r.phases == 3 && (sFlag[c] & kCellExported)) ll_values<2 * NVAR>(r.llG + (size_t) (base + c) * KG, 4 * j, out, stamp);
            }
            __syncthreads();
            // The last warp posts the tile's smallest step at CFL 1 (to every tile under a global CFL
            // number; folded into one minimum for the statistics under local time stepping) while
            // the others receive the halo's gradients.
            const bool fold = r.phases == 1 ? s.time_mode != TM_FIXED : s.time_mode == TM_LOCAL && last_step;
            if (wid == (NT >> 5) - 1 && (s.time_mode == TM_GLOBAL || fold)) {
                const double m = warp_max_pos(lane < (NT >> 5) ? red[lane] : 0.0);
                const double d = m > 0.0 ? dt_of_max(T(m)) : __longlong_as_double(0x7FF0000000000000LL);
                if (lane == 0) {
                    if (!fold) ll_store(r.llX + (size_t) (step & 1) * gridDim.x + blockIdx.x, payload(d), stamp);
                    else atomicMin(r.dtmin, payload(d));
                }
            }
            if (r.phases == 1) return;
            if (tid < NT - 32) ok = halo_receive(sG, NL, a.B, r.llG, sHalo, nh, tid, NT - 32, stamp, a.polls, a.err);
            if (!__syncthreads_and(ok)) return;
        }
#pragma unroll 1
        for (int e = tid; e < nf; e += NT) {
            if constexpr (kChecked)
                if (!entry_ok(sMeta[e], nb, a.B, nh, a.err)) continue;
            FaceIn<T> A;
            T FA[4];
            A.load(sU, sG, NL, sGeo, sMeta, nf, 8, e);
            A.flux(s.gma, FA);
            A.template store<COMP>(sF, nf, FA);
        }
        // the smallest of the tiles' CFL words, by the last warp (the one with the fewest fluxes)
        if (s.time_mode == TM_GLOBAL && r.phases == 3 && wid == (NT >> 5) - 1) {
            double d;
            ok = ll_least(r.llX + (size_t) (step & 1) * gridDim.x, (int) gridDim.x, stamp, d, a.polls, a.err);
            if (lane == 0) s_dt = s.dt_or_cfl * d;
        }
        if (!__syncthreads_and(ok)) return;
        if (r.phases == 2) {
            if (s.time_mode != TM_FIXED) dt_used = s.dt_or_cfl * __longlong_as_double((long long) __ldcg(r.dtmin));
        } else if (s.time_mode == TM_GLOBAL) {
            dt_used = s_dt;
        }
        const bool want_r2 = last_step || steps0 + step == 0;
        r2 = 0.0;
        for (int w = tid; w < (NVAR == 4 ? nb : Bp + nb); w += NT) {
            const int j = NVAR == 4 ? 0 : w >= Bp, c = w - j * Bp;
            if (NVAR != 4 && c >= nb) continue;
            unsigned x[W];
            lds_nbr<W>(sNbr + c * W, x);
            if (x[0] == kNoFace) continue;
            T u[NVAR], R[NVAR], un[NVAR];
            lds_vars<NVAR>(sU, NL, c, j, u);
            cell_flux_sum<T, W, COMP, NVAR>(x, sF, sGeo, nf, 8, j, R, a.err);
            const T dt = s.time_mode == TM_LOCAL ? sDt[c] : T(dt_used);
            const T Rr = cell_update<NVAR>(u, R, sIv[c], dt, un, top);
            if (j == 0) {
                if (sizeof(T) == 4) top = max(top, exponent_word(Rr));   // its square fits a double
                if (sizeof(T) == 8 || want_r2) {
                    const double q = (double) Rr * (double) Rr;
                    r2 += q;
                    if (sizeof(T) == 8) top = max(top, exponent_word(q));
                }
            }
            if (!last_step && (sFlag[c] & kCellExported)) ll_values<NVAR>(r.llU + (size_t) (base + c) * KU, 2 * j, un, stamp);
            st_vars<NVAR>(sU, NL, c, j, un);
            if (last_step) st_vars<NVAR>(gU, a.ps, base + c, j, un);
        }
        __syncthreads();
        // ghost refresh (Euler.cpp:96, :138-142): a cell is its ghosts' only neighbour
        for (int c = tid; c < nb; c += NT) {
            if (!(sFlag[c] & kCellHasGhost)) continue;
            T un[4];
            lds_cell(sU, NL, c, un);
#pragma unroll 1
            for (int k = 0; k < W; k++) {
                const unsigned x = sNbr[c * W + k];
                if (x == kNoFace || !(x & kBoundaryFace)) continue;
                const int e = nbr_entry(x), lb = nbr_local(x);
                if (!index_ok(e < nf && local_ok(lb, nb, a.B, nh), a.err)) continue;
                const int bc = meta_bc(sMeta[e]);
                if (!index_ok(bc >= 0 && bc < MAXBC, a.err)) continue;
                T gnx, gny, gA, ug[4];
                lds_geo3(sGeo, nf, e, 8, gnx, gny, gA);
                ghost_state(s.bc.type[bc], un, gnx, gny, s.gma, s.bc.UBC[bc], s.bc.QBC[bc], ug);
                st_cell(sU, NL, lb, ug);
                if (last_step) st_cell(gU, a.ps, lb < a.B ? base + lb : ~sHalo[lb - a.B], ug);
            }
        }
        if (want_r2) {
            const double t = block_sum(r2, red3);
            if (tid == 0) {
                if (steps0 + step == 0) r.partial_first[blockIdx.x] = t;
                if (last_step) s.partial[blockIdx.x] = t;
            }
        }
        if (last_step) break;
        if (refetch && tid == 0) {
            // the r vectors back over the fluxes, which every thread has read
            fence_proxy_async();
            mbar_arrive_expect_tx(full, nf * 4u * (unsigned) sizeof(T));
            if (nf) bulk_g2s(sF, a.tgeo + (size_t) f0 * 8 + 4 * (size_t) nf, nf * 4u * (unsigned) sizeof(T), full);
        }
        // the halo's states by the second half of the threads while the first forms the wave speeds
        // (two threads a cell), or by all behind it
        if (NVAR == 4 || tid < Bp) wave_speeds();
        if (NVAR == 4) ok = halo_receive(sU, NL, a.B, r.llU, sHalo, nh, tid, NT, stamp, a.polls, a.err);
        else if (tid >= Bp) ok = halo_receive(sU, NL, a.B, r.llU, sHalo, nh, tid - Bp, NT - Bp, stamp, a.polls, a.err);
        if (refetch && !mbar_wait(full, (unsigned) (step + 1) & 1u, a.polls, a.err, abort_word(smem))) ok = false;
        if (!__syncthreads_and(ok)) {
            if (refetch && tid == 0) mbar_drain(full, (unsigned) (step + 1) & 1u, a.err);
            return;
        }
    }

    // statistics: the last CTA to arrive sums the partials in CTA order
    if (not_finite<T>(top)) s_bad = 1;
    __syncthreads();
    if (tid == 0) {
        if (s_bad) atomicOr(&s.stats->nonfinite, 1);
        __threadfence();
        s_last = atomicAdd(s.counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    double x = 0.0, y = 0.0;
    for (int i = tid; i < (int) gridDim.x; i += NT) {
        x += __ldcg(s.partial + i);
        if (steps0 == 0) y += __ldcg(r.partial_first + i);
    }
    x = block_sum(x, red3);
    if (steps0 == 0) y = block_sum(y, red3);
    if (tid == 0) {
        if (s.time_mode == TM_LOCAL) dt_used = s.dt_or_cfl * __longlong_as_double((long long) __ldcg(r.dtmin));
        StepStats* st = s.stats;
        st->res2_last = x;
        if (steps0 == 0) st->res2_first = y;
        st->steps = steps0 + r.nsteps;
        st->dt_last = dt_used;
        if (!(x == x) || x > 1.7e308) st->nonfinite = 1;
        *s.counter = 0u;
        *r.dtmin = 0x7FF0000000000000ULL;
    }
}

}  // namespace hcfd
