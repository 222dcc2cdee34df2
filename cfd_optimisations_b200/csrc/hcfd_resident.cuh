// Resident step kernel: whole solves of small meshes in one cooperative launch.
//
// A step of a mesh of up to ~120,000 cells (FP64; ~230,000 in FP32) takes the tiled kernels
// far longer than its bytes or operations: two launches, each filling barriers, descriptors
// and copies before its one tile per CTA and draining after it.  Here every SM holds one tile
// in shared memory (state, limited gradients, face records, fluxes, slots) for all steps
// of a call.  What crosses tiles goes through global memory (L2): the state and the limited
// gradient of the cells that are in another tile's halo, and the CFL minimum; a grid barrier
// after each of the step's two halves orders it.
//
//   half 1: gradient, limiter, CFL of the tile's cells (Pass1Cell, as pass 1); the limited
//           gradients stay in shared memory, those of exported cells are written out too
//   barrier; halo gradients read
//   half 2: flux per face entry, sum and update per cell, ghosts (FaceIn, cell_flux_sum,
//           cell_update, as pass 2); exported cells written out
//   barrier; halo states read
//
// The arithmetic is that of the tiled kernels, function for function, so a state does not
// depend on which of them stepped it.
//
// The grid must be co-resident (the host launches it cooperatively, one CTA per tile, at most
// one per SM).  Every spin is bounded: a wait that gives up sets the error word, which every
// other waiting CTA polls, and all of them leave; copies into shared memory in flight are
// waited for first.
#pragma once
#include "hcfd_tile.cuh"

namespace hcfd {

constexpr int kResidentThreads = 512;       // 128 registers a thread, what the two halves need in FP64

struct ResidentArgs {
    const unsigned char* __restrict__ exported;   // [ntiles * B]: the cell is in another tile's halo
    unsigned int* bar;                            // arrivals at grid barriers, never reset while the handle works
    unsigned int bar_base;                        // its value before this launch
    unsigned long long* dtmin;                    // [2], both +inf between launches
    double* partial_first;                        // [grid]: residual partials of the first step since initialise
    int nsteps;
    int phases;                                   // 3: whole steps; 1 or 2: one half of one step (profiling)
};

// Shared memory of one tile (all offsets multiples of 128 bytes).
template <class T>
struct ResidentSmem {
    size_t u, g, geo, flux, meta, cslot, iv, exported, halo, total;
    __host__ __device__ ResidentSmem(int B, int Hmax, int Fmax, int Wp) {
        size_t p = kHeader;
        u = p;        p += align128((size_t) (B + Hmax) * sizeof(Cell4<T>));
        g = p;        p += align128((size_t) (B + Hmax) * sizeof(Grad8<T>));
        geo = p;      p += align128((size_t) Fmax * sizeof(FaceGeo<T>));
        flux = p;     p += align128((size_t) Fmax * sizeof(Cell4<T>));
        meta = p;     p += align128((size_t) Fmax * 4);
        cslot = p;    p += align128((size_t) B * Wp * sizeof(short));
        iv = p;       p += align128((size_t) B * sizeof(T));
        exported = p; p += align128((size_t) B);
        halo = p;     p += align128((size_t) Hmax * sizeof(int));
        total = p;
    }
};

// Loads of values that other CTAs wrote during this kernel: from L2, never through L1.
__device__ __forceinline__ uint4 ld_l2(const void* p) { return __ldcg(reinterpret_cast<const uint4*>(p)); }
template <class R>   // 16-byte chunks j of record i, chunk planes of stride ps -> planes of stride NL
__device__ __forceinline__ void halo_load(R* s, int NL, int l, const R* g, size_t ps, int i) {
    constexpr int C = sizeof(R) / 16;
    uint4 x[C];
#pragma unroll
    for (int j = 0; j < C; j++) x[j] = ld_l2(reinterpret_cast<const uint4*>(g) + j * ps + i);
#pragma unroll
    for (int j = 0; j < C; j++) reinterpret_cast<uint4*>(s)[j * NL + l] = x[j];
}

__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Arrival of thread 0 for its CTA and bounded wait for the whole grid (`target` arrivals since
// the counter was zeroed; the counter wraps).  False when the wait gave up or another CTA set
// the error word.  Call between two __syncthreads: the first orders the CTA's writes before the
// arrival (with the fence), the second the other CTAs' writes before the CTA's reads.
__device__ __forceinline__ bool grid_arrive_wait(unsigned* bar, unsigned target, unsigned polls, unsigned* err) {
    __threadfence();
    atomicAdd(bar, 1u);
    bool ok = false;
#pragma unroll 1
    for (unsigned i = 0; i < polls; i++) {
        if ((int) (ld_acquire(bar) - target) >= 0) { ok = true; break; }
        if ((i & 63u) == 63u && *(volatile unsigned*) err) break;
    }
    if (!ok) atomicOr(err, 1u);
    __threadfence();
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

// What bounds it: a chain of latencies, not bytes.  At 26,000 cells (176 a CTA) a step is two
// barriers, two halo exchanges and two arithmetic chains of ~1,000 cycles each.  One CTA per SM,
// since the tile takes most of an SM's shared memory at the upper end and the lower end is not
// short of warps but of latency.
template <class T, int W, bool COMP>
__global__ void __launch_bounds__(kResidentThreads, 1) resident_kernel(const TileArgs<T> a, const ResidentArgs r) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ double red[32];
    __shared__ int s_bad;
    __shared__ bool s_last;
    const ResidentSmem<T> L(a.B, a.Hmax, a.Fmax, a.Wp);
    const StepArgs<T>& s = a.s;
    const int NT = blockDim.x, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int NL = a.B + a.Hmax;
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
    T* sF = reinterpret_cast<T*>(smem + L.flux);
    unsigned* sMeta = reinterpret_cast<unsigned*>(smem + L.meta);
    short* sSlot = reinterpret_cast<short*>(smem + L.cslot);
    T* sIv = reinterpret_cast<T*>(smem + L.iv);
    unsigned char* sExp = smem + L.exported;
    int* sHalo = reinterpret_cast<int*>(smem + L.halo);
    Cell4<T>* gU = const_cast<Cell4<T>*>(s.U);
    unsigned long long* full = reinterpret_cast<unsigned long long*>(smem);
    constexpr int CU = sizeof(Cell4<T>) / 16, CG = sizeof(Grad8<T>) / 16;

    // the tile: bulk copies of its contiguous blocks, halo ids and halo states by the threads
    if (tid == 0) {
        mbar_init(full, 1);
        *abort_word(smem) = 0;
        fence_mbar_init();
        s_bad = 0;
        if ((int) blockIdx.x != a.skip_tile) {       // failure injection for tests: nothing armed
            const unsigned bu = nb * 16u * CU, bg = r.phases == 2 ? nb * 16u * CG : 0u;
            const unsigned bf = nf * 8u * (unsigned) sizeof(T), bm = nf * 4u;
            const unsigned bs = good ? a.B * a.Wp * (unsigned) sizeof(short) : 0u, bi = good ? a.B * (unsigned) sizeof(T) : 0u;
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
                bulk_g2s(sSlot, a.cslot + (size_t) base * a.Wp, bs, full);
                bulk_g2s(sIv, s.iv + base, bi, full);
            }
        }
    }
    for (int c = tid; c < nb; c += NT) sExp[c] = r.exported[base + c];
    for (int h = tid; h < nh; h += NT) {
        int ci = __ldg(a.halo + h0 + h);
        if (!index_ok(ci >= 0 && ci < a.ps, a.err)) ci = 0;
        sHalo[h] = ci;
        halo_load(sU, NL, a.B + h, s.U, a.ps, ci);
        if (r.phases == 2) halo_load(sG, NL, a.B + h, s.phiG, a.ps, ci);
    }
    const long long steps0 = s.stats->steps;
    __syncthreads();
    // a wait that gives up is the whole CTA's; copies that were armed land (they read valid
    // memory) and are drained before leaving
    if (!__syncthreads_and(mbar_wait(full, 0, a.polls, a.err, abort_word(smem)))) {
        if (tid == 0 && (int) blockIdx.x != a.skip_tile) mbar_drain(full, 0, a.err);
        return;
    }

    unsigned target = r.bar_base;
    if (r.phases == 2) {
        // no barrier of half 1 stands between these halo reads and the other CTAs' updates
        target += gridDim.x;
        if (!__syncthreads_and(tid != 0 || grid_arrive_wait(r.bar, target, a.polls, a.err))) return;
    }
    double r2 = 0.0, dt_used = s.dt_or_cfl;
    int bad = 0;
    for (int step = 0; step < r.nsteps; step++) {
        const bool last_step = step + 1 == r.nsteps;
        unsigned long long* dtmin = r.dtmin + (step & 1);
        if (r.phases & 1) {
            const int lmode = limiter_mode(steps0 + step, s.freeze_after);
            T xmx = T(0);
            for (int c = tid; c < nb; c += NT) {
                short cs[8];
                lds_slots(sSlot + c * a.Wp, a.Wp, cs);
                if (cs[0] < 0) continue;
                Pass1Cell<T, W> p;
                lds_cell(sU, NL, c, p.u);
                tile_faces<T, W>(p, a, sU, sGeo, sMeta, cs, NL, nf, nb, nh, c);
                T out[8], phis[4];
                if (lmode == LIM_FROZEN) {
                    // written by this thread's SM, perhaps in this launch: not through the read-only path
                    const uint4* q = reinterpret_cast<const uint4*>(s.phiF);
#pragma unroll
                    for (int j = 0; j < CU; j++) {
                        const uint4 x = ld_l2(q + (size_t) j * a.ps + base + c);
                        memcpy(reinterpret_cast<char*>(phis) + 16 * j, &x, 16);
                    }
                }
                const T iv = sIv[c];
                p.finish(iv, s.limiter, s.venkat_K, lmode, phis, out);
                if (lmode == LIM_RECORD) st_cell(s.phiF, a.ps, base + c, phis);
                st_grad(sG, NL, c, out);
                if (sExp[c] || r.phases == 1) st_grad(s.phiG, a.ps, base + c, out);
                if (s.time_mode != TM_FIXED) xmx = fmax(xmx, iv * p.lam);
            }
            if (s.time_mode != TM_FIXED) {
                const T m = warp_max(xmx);
                if (lane == 0) red[wid] = (double) m;
            }
            __syncthreads();
            if (s.time_mode != TM_FIXED && wid == 0) {
                const double m = warp_max(lane < (NT >> 5) ? red[lane] : 0.0);
                const double d = dt_of_max(T(m));
                if (lane == 0 && d < 1e300) atomicMin(dtmin, (unsigned long long) __double_as_longlong(d));
            }
            if (r.phases == 1) return;
            target += gridDim.x;
            if (!__syncthreads_and(tid != 0 || grid_arrive_wait(r.bar, target, a.polls, a.err))) return;
            // the other slot is no longer read: its readers arrived at this barrier after reading it
            if (blockIdx.x == 0 && tid == 0) r.dtmin[(step + 1) & 1] = 0x7FF0000000000000ULL;
            for (int h = tid; h < nh; h += NT) halo_load(sG, NL, a.B + h, s.phiG, a.ps, sHalo[h]);
        }
        if (s.time_mode != TM_FIXED) dt_used = s.dt_or_cfl * __longlong_as_double((long long) __ldcg(dtmin));
        __syncthreads();
        for (int e = tid; e < nf; e += 2 * NT) {
            const int eB = (e + NT < nf) ? e + NT : e;
            if constexpr (kChecked)
                if (!entry_ok(sMeta[e], nb, a.B, nh, a.err) || !entry_ok(sMeta[eB], nb, a.B, nh, a.err)) continue;
            FaceIn<T> A;
            T FA[4];
            A.load(sU, sG, NL, sGeo, sMeta, nf, 8, e);
            if (e - lane + NT < nf) {                // some thread of this warp has a second entry
                FaceIn<T> Bq;
                T FB[4];
                Bq.load(sU, sG, NL, sGeo, sMeta, nf, 8, eB);
                A.flux(s.gma, FA);
                Bq.flux(s.gma, FB);
                if (eB != e) Bq.template store<COMP>(sF, nf, FB);
            } else {
                A.flux(s.gma, FA);
            }
            A.template store<COMP>(sF, nf, FA);
        }
        __syncthreads();
        const bool want_r2 = last_step || steps0 + step == 0;
        r2 = 0.0;
        for (int c = tid; c < nb; c += NT) {
            short cs[8];
            lds_slots(sSlot + c * a.Wp, a.Wp, cs);
            if (cs[0] < 0) continue;
            T u[4], R[4], lam, un[4];
            lds_cell(sU, NL, c, u);
            const T iv = sIv[c];
            cell_flux_sum<T, W, COMP>(cs, sF, sGeo, nf, 8, s.time_mode, u, s.gma, R, lam, a.err);
            const T dt = s.time_mode == TM_LOCAL ? T(s.dt_or_cfl) * qrcp(iv * lam) : T(dt_used);
            const T Rr = cell_update(u, R, iv, dt, un, bad);
            const double q = (double) Rr * (double) Rr;
            r2 += q;
            bad |= !isfinite(q);
            st_cell(sU, NL, c, un);
            if (last_step || sExp[c]) st_cell(gU, a.ps, base + c, un);
            // ghost refresh (Euler.cpp:96, :138-142): this cell is its ghosts' only neighbour
#pragma unroll
            for (int k = 0; k < W; k++) {
                if (cs[k] < 0 || (cs[k] & 1)) continue;
                const int e = cs[k] >> 1;
                const unsigned w = sMeta[e];
                const int bc = meta_bc(w);
                if (bc < 0) continue;
                const int lb = meta_lb(w);
                if (!index_ok(local_ok(lb, nb, a.B, nh) && bc < MAXBC, a.err)) continue;
                T gnx, gny, gA, ug[4];
                lds_geo3(sGeo, nf, e, 8, gnx, gny, gA);
                ghost_state(s.bc.type[bc], un, gnx, gny, s.gma, s.bc.UBC[bc], s.bc.QBC[bc], ug);
                st_cell(sU, NL, lb, ug);
                // a ghost of another tile's range is re-read with the halo
                if (last_step || lb >= a.B) st_cell(gU, a.ps, lb < a.B ? base + lb : sHalo[lb - a.B], ug);
            }
        }
        if (want_r2) {
            const double t = block_sum(r2, red);
            if (tid == 0) {
                if (steps0 + step == 0) r.partial_first[blockIdx.x] = t;
                if (last_step) s.partial[blockIdx.x] = t;
            }
        }
        if (last_step) break;
        __syncthreads();
        target += gridDim.x;
        if (!__syncthreads_and(tid != 0 || grid_arrive_wait(r.bar, target, a.polls, a.err))) return;
        for (int h = tid; h < nh; h += NT) halo_load(sU, NL, a.B + h, s.U, a.ps, sHalo[h]);
        __syncthreads();
    }

    // statistics: the last CTA to arrive sums the partials in CTA order
    if (bad) s_bad = 1;
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
    x = block_sum(x, red);
    if (steps0 == 0) y = block_sum(y, red);
    if (tid == 0) {
        StepStats* st = s.stats;
        st->res2_last = x;
        if (steps0 == 0) st->res2_first = y;
        st->steps = steps0 + r.nsteps;
        st->dt_last = dt_used;
        if (!(x == x) || x > 1.7e308) st->nonfinite = 1;
        *s.counter = 0u;
        r.dtmin[0] = r.dtmin[1] = 0x7FF0000000000000ULL;
    }
}

}  // namespace hcfd
