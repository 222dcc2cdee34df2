// Tiled step kernels (meshes beyond the resident kernel's size, arenas, explicit tiles): persistent
// CTAs walk the tiles of the execution plan (hcfd_plan.cpp).
// Per tile, the contiguous blocks (the tile's own cells, its face records, face words and, in pass 2,
// face metadata) are staged into shared memory with TMA bulk copies (cp.async.bulk, completion
// on an mbarrier) and the halo cells with 16-byte cp.async gathers; all arithmetic then
// reads shared memory.
//
// pass 1 (thread per tile cell): Green-Gauss gradient, limiter, CFL dt -> phiG (global).
// pass 2: face phase (thread per face entry) computes each face flux once per tile and
//         writes F over the staged face record's two r pairs (the cell phase does not read
//         them); cell phase (thread per tile cell) sums A_f F of its faces in increasing face
//         order, updates the cell and refreshes its ghost cells.
// The arithmetic is that of the thread-per-cell kernels in hcfd_kernels.cuh, operation for
// operation; only where the operands come from differs.
//
// What bounds them at 2001x1001 in FP64: bytes and the latency of staging them.  The two passes move
// 1.85 GB a step, 283 us at the measured copy bandwidth, and take 343-359 us (175-183 and 193-203 us a
// pass on its own): 14 and 12 compute warps an SM, two CTAs of two stages each, which registers and
// shared memory allow no more of, wait 17 % and 6 % of their time for a stage.
#pragma once
#include "hcfd_internal.hpp"
#include "hcfd_kernels.cuh"

#include <vector>

namespace hcfd {

template <class T>
struct TileArgs {
    StepArgs<T> s;                         // state, stats, BC table, modes
    const T* __restrict__ tgeo;            // face records, per tile pair-major (see ldp), rec values each
    int rec;                               // values per face record: 8, or 7 in a pass-2 plan of its own
    const unsigned* __restrict__ tmeta;    // one word per entry (pack_meta): la, lb, bc
    const int* __restrict__ foff;          // [ntiles + 1], multiples of 4
    const int* __restrict__ hoff;          // [ntiles + 1]
    const int* __restrict__ halo;          // internal cell ids
    const unsigned* __restrict__ nbr;      // [ntiles * B * Wp]: a word per cell and face (pack_nbr_kernel); Wp = W
    const short* __restrict__ cslot;       // the same as the plan's 16-bit {entry, side}, staged in their place by the
                                           // kRareToo variants; null: the words are staged
    int ntiles, B, Wp, Hmax, Fmax;
    unsigned int* err;                     // bit 0: a bounded wait gave up; bit 1: copies did not drain;
                                           // bit 2: an index out of range (checked build)
    unsigned polls;                        // poll limit of every bounded wait (2^22 by default)
    int skip_tile;                         // failure injection for tests: the producer arms nothing
                                           // for this tile (-1: none)
    int ps;                                // plane stride of the cell planes (Nc, or the arena's capacity)
    // Arena mode (many meshes in one flat arena; see hcfd_arena.cu).  Tile i of the active
    // list is described by tiles[2i] = {first cell, first entry, entries, instance} and
    // tiles[2i+1] = {first halo id, halo count, instance's first tile, -}; every arena tile holds B cells.
    const int4* __restrict__ tiles;
    const double* __restrict__ inst_dt;    // per instance: dt (fixed mode) or CFL number
    unsigned long long* inst_dtmin;        // per instance, two parity slots (double bits)
    const BCTable* __restrict__ inst_bc;   // per instance
    StepStats* inst_stats;                 // per instance
    double* tile_r2;                       // per active tile and compute warp (t * B/32 + warp): sum of R_rho^2
    int* tile_bad;                         // same layout: a NaN/Inf appeared
    int par;                               // which dtmin slot this step uses
    // Tile queue: each CTA takes three tiles by position first (every gridDim.x-th from blockIdx.x),
    // then, with `claim` set, the tile 3 gridDim.x + atomicAdd(claim, 1) (CTAs that finish early take more
    // tiles), else every gridDim.x-th tile.  `claim_reset` (the other pass's queue) is zeroed by this kernel:
    // the other pass runs before and after it in stream order, never during it.
    int* claim;
    int* claim_reset;
    // Pass 2: whether this step's residual is wanted (the first of a solve, for res2_first, and
    // the last of a call, for whoever asks); steps without it skip the squares and their sums.
    int want_res;
    long long nentries, nhalo, ncap;       // lengths of tgeo/tmeta (entries), halo, and of the
                                           // per-cell arrays iv/nbr (cells): checked build
};

// Metadata of a face entry in one 32-bit word: the local index (tile cell 0..B-1, halo cell
// B..) of its left cell in bits 0-12, of its right cell in bits 13-25, and its boundary
// condition's index + 1 in bits 26-30 (0: an interior face).  The plan keeps B + halo below
// 8192 and at most 16 boundary conditions.
__host__ __device__ __forceinline__ unsigned pack_meta(int la, int lb, int bc) {
    return (unsigned) la | ((unsigned) lb << 13) | ((unsigned) (bc + 1) << 26);
}
inline std::vector<unsigned> packed_meta(const TilePlan& P) {
    std::vector<unsigned> w(P.meta.size() / 4);
    for (size_t i = 0; i < w.size(); i++) w[i] = pack_meta(P.meta[4 * i], P.meta[4 * i + 1], P.meta[4 * i + 2]);
    return w;
}
__device__ __forceinline__ int meta_la(unsigned w) { return (int) (w & 0x1FFFu); }
__device__ __forceinline__ int meta_lb(unsigned w) { return (int) ((w >> 13) & 0x1FFFu); }
__device__ __forceinline__ int meta_bc(unsigned w) { return (int) (w >> 26) - 1; }

// One face of a tile cell in one word: its entry (bits 0-13), the cell's side (bit 14: right), the
// local index of the cell across it (bits 15-27) and whether it is a boundary face (bit 28);
// kNoFace for a position the cell does not use.  With it a cell's loads of face record and neighbour
// state both hang on one word, not on the entry's metadata in between (pass 1 reads none).
constexpr unsigned kNoFace = 0xFFFFFFFFu, kBoundaryFace = 1u << 28;
// The word of the plan's {entry, side} (-1: none), m the packed metadata of the tile's entries.
__device__ __forceinline__ unsigned nbr_word(int s, const unsigned* m) {
    if (s < 0) return kNoFace;
    const unsigned e = (unsigned) s >> 1, side = s & 1, x = m[e];
    return e | (side << 14) | ((side ? x & 0x1FFFu : (x >> 13) & 0x1FFFu) << 15) | (x >> 26 ? kBoundaryFace : 0u);
}
// A block per tile: the words of its cells, from the plan's {entry, side} table (cslot, -1: none) and the
// packed metadata of the tile's entries.  Packed on the host, creating a solver of 1025x513 nodes took
// 1,171 ms (FP64) and 1,195 (FP32), packed here 1,123 and 1,165 (the quickest of 14).
static __global__ void pack_nbr_kernel(int per, const int* __restrict__ foff, const unsigned* __restrict__ meta,
                                const short* __restrict__ cslot, unsigned* __restrict__ nbr) {
    const size_t t0 = (size_t) blockIdx.x * per;
    const unsigned* m = meta + foff[blockIdx.x];
    for (int i = threadIdx.x; i < per; i += blockDim.x) nbr[t0 + i] = nbr_word(cslot[t0 + i], m);
}
__device__ __forceinline__ int nbr_entry(unsigned w) { return (int) (w & 0x3FFFu); }
__device__ __forceinline__ bool nbr_right(unsigned w) { return (w >> 14) & 1u; }
__device__ __forceinline__ int nbr_local(unsigned w) { return (int) ((w >> 15) & 0x1FFFu); }
template <int W>   // a cell's W words
__device__ __forceinline__ void lds_nbr(const unsigned* p, unsigned x[W]) {
    if constexpr (W == 3) {
        x[0] = p[0]; x[1] = p[1]; x[2] = p[2];
    } else {
#pragma unroll
        for (int k = 0; k < W; k += 4) {
            const uint4 v = *reinterpret_cast<const uint4*>(p + k);
            x[k] = v.x; x[k + 1] = v.y; x[k + 2] = v.z; x[k + 3] = v.w;
        }
    }
}

// Values of a kernel's template arguments beside those fixed at compile time: read from the arguments
// (W = 8, meshes no workload has); the same with what few handles need on top, 16-bit face words
// (GEN) and a limiter by_face.  On W = 8, whose other handles took the same variant at first, these cost
// 6-7 % (260,000 cells of three to eight faces, FP64 52.2 us a step without them and 55.7 with, FP32 31.9 and 33.8).
constexpr int kRunTime = -1, kRareToo = -2;

// GEN: the variant may have 16-bit words staged (sNbr then points at them), which are widened here.
template <int W, bool GEN>
__device__ __forceinline__ void cell_words(const unsigned* sNbr, bool short_words, const unsigned* sMeta, int c, unsigned x[W]) {
    if (GEN && short_words) {
        const short* q = reinterpret_cast<const short*>(sNbr) + c * W;
#pragma unroll
        for (int k = 0; k < W; k++) x[k] = nbr_word(q[k], sMeta);
    } else {
        lds_nbr<W>(sNbr + c * W, x);
    }
}

// A local cell index of a tile: one of its nb cells, or one of its nh halo cells (B..).
__device__ __forceinline__ bool local_ok(int l, int nb, int B, int nh) {
    return (l >= 0 && l < nb) || (l >= B && l < B + nh);
}
// A face entry's metadata: both cells local to the tile, the boundary condition in the table.
__device__ __forceinline__ bool entry_ok(unsigned w, int nb, int B, int nh, unsigned int* err) {
    return index_ok(local_ok(meta_la(w), nb, B, nh) && local_ok(meta_lb(w), nb, B, nh) && meta_bc(w) < MAXBC, err);
}

// Cells, face entries and halo of tile t (single mesh) or of active tile t (arena).
template <bool ARENA, class T>
__device__ __forceinline__ void tile_info(const TileArgs<T>& a, int t, int& base, int& nb, int& f0, int& nf,
                                          int& h0, int& nh, int& inst) {
    if constexpr (ARENA) {
        const int4 d0 = __ldg(a.tiles + 2 * t), d1 = __ldg(a.tiles + 2 * t + 1);
        base = d0.x; nb = a.B; f0 = d0.y; nf = d0.z; inst = d0.w; h0 = d1.x; nh = d1.y;
    } else {
        base = t * a.B; nb = min(a.B, a.s.Nc - base);
        f0 = __ldg(a.foff + t); nf = __ldg(a.foff + t + 1) - f0;
        h0 = __ldg(a.hoff + t); nh = __ldg(a.hoff + t + 1) - h0;
        inst = 0;
    }
}

struct TileDesc {
    int base, nb, f0, nf, h0, nh, inst, first;
};

// What the compute warps need of a tile besides its data, written by the producer into the
// stage header with the tile's copies (published by the same mbarrier), so that the compute
// warps start a tile without dependent global loads: its descriptor, and for its instance
// the step count (limiter freezing), the dt or CFL number and the dt minimum of this step.
struct StageInfo {
    int base, nb, f0, nf, h0, nh, inst, next_inst;   // next_inst (pass 1, arena): of this CTA's next tile, -1 at the end
    double dt_or_cfl;
    double dtmin;
    long long steps;
    int t;                                            // the tile, or -1: the CTA has no more tiles
    int first;                                        // (arena) the instance's first tile
};
static_assert(sizeof(StageInfo) == 64, "stage info is 64 bytes");
// Header of a CTA's shared memory: full[2] and empty[2] mbarriers (bytes 0-31), the abort
// words (32-39), then StageInfo per stage (two, from byte 64).
constexpr int kHeader = 256;
constexpr unsigned kDrainPolls = 1u << 24;

// ---------------------------------------------------------------------------------------
// PTX helpers (sm_90+ bulk copies and mbarriers; sm_80+ cp.async)

__device__ __forceinline__ unsigned smem_u32(const void* p) {
    return static_cast<unsigned>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned long long* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long* bar, unsigned bytes) {
    asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(unsigned long long* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
// 1-D bulk copy global -> shared (no tensor map, no multicast); dst, src 16-B aligned,
// bytes a multiple of 16.
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, unsigned bytes, unsigned long long* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}
// Orders this thread's (and, behind a barrier, its CTA's) ordinary accesses to shared memory before
// bulk copies it issues afterwards.
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ bool mbar_try_wait(unsigned long long* bar, unsigned parity) {
    unsigned ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n}"
                 : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return ok != 0;
}
// Bounded wait for an mbarrier phase.  Gives up after `polls` polls, or early once another
// thread of the CTA has given up (its abort word is set); on giving up it records the failure
// in the kernel's error word (the host reports HCFD_ETIMEOUT) and in the abort word, and
// returns false.  A thread whose wait failed never reads the stage it waited for: the
// producer then stops issuing copies, and the consumers leave their tile loop (see
// producer_loop and HCFD_TILE_LOOP_BEGIN).
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, unsigned parity, unsigned polls, unsigned int* err,
                                          volatile int* abort) {
#pragma unroll 1
    for (unsigned i = 0; i < polls; i++) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((i & 255u) == 255u && *abort) return false;
    }
    atomicOr(err, 1u);
    *abort = 1;
    return false;
}
// Bounded wait for copies already issued (they only read valid global memory, so they land);
// used before a CTA exits so that nothing is written into its shared memory afterwards.
__device__ __forceinline__ void mbar_drain(unsigned long long* bar, unsigned parity, unsigned int* err) {
#pragma unroll 1
    for (unsigned i = 0; i < kDrainPolls; i++)
        if (mbar_try_wait(bar, parity)) return;
    atomicOr(err, 2u);
}
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}
__device__ __forceinline__ volatile int* abort_word(unsigned char* smem) { return reinterpret_cast<volatile int*>(smem + 32); }
// Set by compute threads only, before the compute barrier that follows the stage wait
// (pass 2): read after that barrier, every compute warp sees the same value.
__device__ __forceinline__ volatile int* compute_abort_word(unsigned char* smem) {
    return reinterpret_cast<volatile int*>(smem + 36);
}

// Shared-memory loads (plain loads: the __ldg helpers of hcfd_kernels.cuh are global-only).
// (chunk-plane layout of hcfd_kernels.cuh, plane stride ps = staged cell count)
__device__ __forceinline__ void lds_cell(const Cell4<double>* p, int ps, int i, double u[4]) {
    const double2* q = reinterpret_cast<const double2*>(p);
    const double2 a = q[i], b = q[ps + i];
    u[0] = a.x; u[1] = a.y; u[2] = b.x; u[3] = b.y;
}
__device__ __forceinline__ void lds_cell(const Cell4<float>* p, int, int i, float u[4]) {
    const float4 a = reinterpret_cast<const float4*>(p)[i];
    u[0] = a.x; u[1] = a.y; u[2] = a.z; u[3] = a.w;
}
__device__ __forceinline__ void lds_grad(const Grad8<double>* p, int ps, int i, double g[8]) {
    const double2* q = reinterpret_cast<const double2*>(p);
#pragma unroll
    for (int k = 0; k < 4; k++) { const double2 a = q[k * ps + i]; g[2 * k] = a.x; g[2 * k + 1] = a.y; }
}
__device__ __forceinline__ void lds_grad(const Grad8<float>* p, int ps, int i, float g[8]) {
    const float4* q = reinterpret_cast<const float4*>(p);
    const float4 a = q[i], b = q[ps + i];
    g[0] = a.x; g[1] = a.y; g[2] = a.z; g[3] = a.w; g[4] = b.x; g[5] = b.y; g[6] = b.z; g[7] = b.w;
}
// Face records of a tile are stored pair-major: four planes of pairs, (nx, ny), (Af, If),
// (rLx, rLy), (rRx, rRy); pair j of entry e at index j nf + e of the pair array (16 bytes a pair
// in double, 8 in float).  One load brings a pair, and consecutive threads reading consecutive
// entries touch consecutive words (no bank conflicts).
template <class T> struct PairOf;
template <> struct PairOf<double> { using type = double2; };
template <> struct PairOf<float> { using type = float2; };
template <class T>
__device__ __forceinline__ typename PairOf<T>::type ldp(const T* p, int nf, int j, int e) {
    return reinterpret_cast<const typename PairOf<T>::type*>(p)[j * nf + e];
}
template <class T>
__device__ __forceinline__ void stp(T* p, int nf, int j, int e, T x, T y) {
    typename PairOf<T>::type v;
    v.x = x; v.y = y;
    reinterpret_cast<typename PairOf<T>::type*>(p)[j * nf + e] = v;
}
// Records of 8 values (pass 1, and pass 2 when it shares pass 1's plan, the arena's too):
// pairs (nx, ny), (Af, If), (rLx, rLy), (rRx, rRy).  Records of 7 values (pass 2 on a plan of
// its own, which never reads If): pairs (nx, ny), (rLx, rLy), (rRx, rRy), then Af alone in a
// plane of scalars.  rplane gives the pair plane of rL (rR follows it).
__device__ __forceinline__ int rplane(int rec) { return rec == 7 ? 1 : 2; }
template <class T>
__device__ __forceinline__ T lds_area(const T* p, int nf, int e, int rec) {
    return rec == 7 ? p[6 * nf + e] : p[2 * (nf + e)];
}

// Normal, length and interpolation weight (pass 1 reads the r vector of one side apart).
template <class T>
__device__ __forceinline__ void lds_geo4(const T* p, int nf, int e, FaceGeo<T>& g) {
    const auto a = ldp(p, nf, 0, e), b = ldp(p, nf, 1, e);
    g.nx = a.x; g.ny = a.y; g.Af = b.x; g.If = b.y;
}

// Normal and length only (the components pass 2's flux write leaves intact).
template <class T>
__device__ __forceinline__ void lds_geo3(const T* p, int nf, int e, int rec, T& nx, T& ny, T& Af) {
    const auto a = ldp(p, nf, 0, e);
    nx = a.x; ny = a.y; Af = lds_area(p, nf, e, rec);
}

__host__ __device__ constexpr size_t align128(size_t x) { return (x + 127) & ~size_t(127); }

// Shared-memory layout of one CTA: two mbarriers and two staging buffers (double buffering:
// tile i+1 is in flight while tile i is computed).  One staging buffer holds the tile's and
// its halo's cells (and limited gradients in pass 2), its face records and metadata
// (pass 2), its cells' face words and its iv.  Pass 2 keeps its fluxes in the staged face records, so a CTA
// needs no other scratch (three CTAs of 128 + 32 threads fit an SM at 128-cell tiles).
template <class T>
struct TileSmem {
    size_t u, g, geo, meta, nbr, iv, stage, total;   // byte offsets within a stage
    // short_words: the plan's 16-bit face words and the metadata they need, in place of the 32-bit words
    __host__ __device__ TileSmem(int B, int Hmax, int Fmax, int W, int Wp, bool pass2, bool short_words = false) {
        size_t p = 0;
        u = p;     p += align128((size_t) (B + Hmax) * sizeof(Cell4<T>));
        g = p;     if (pass2) p += align128((size_t) (B + Hmax) * sizeof(Grad8<T>));
        geo = p;   p += align128((size_t) Fmax * sizeof(FaceGeo<T>));
        meta = p;  if (pass2 || short_words) p += align128((size_t) Fmax * 4);
        nbr = p;   p += align128((size_t) B * Wp * (short_words ? sizeof(short) : sizeof(unsigned)));
        iv = p;    p += align128((size_t) B * sizeof(T));
        stage = p;
        total = kHeader + 2 * stage;
        (void) W;
    }
};

// Arrival on `bar` once all cp.async operations issued so far by this thread have landed;
// counts as one of the barrier's expected arrivals (.noinc).
__device__ __forceinline__ void cp_async_arrive_noinc(unsigned long long* bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// Barrier over the compute warps only (named barrier 1; the producer warp never joins it).
__device__ __forceinline__ void compute_sync(int nthreads) {
    asm volatile("bar.sync 1, %0;" ::"r"(nthreads) : "memory");
}

// Producer warp: for each of this CTA's tiles, waits until the compute warps have released
// the staging buffer, then lane 0 arms the buffer's `full` mbarrier with the byte counts of
// the bulk copies and issues them (those of the first tile that no kernel writes ahead of the rest), and
// every lane gathers its share of the halo cells with cp.async and signals their completion on the same mbarrier.  The `full` barrier therefore
// completes when all of the tile's data has landed: 1 expect-tx arrival + 32 cp.async
// arrivals + the transaction bytes.
// Once any wait of the CTA has given up, the producer issues nothing more; before it
// returns it waits for the copies it has issued (the last armed phase of each buffer; earlier
// ones completed before their buffer was re-armed), so no copy lands after the CTA exits.
template <class T>   // within the arrays and the staging capacity
__device__ __forceinline__ bool desc_ok(const TileArgs<T>& a, const TileDesc& d) {
    return d.base >= 0 && d.nb >= 0 && d.nb <= a.B && d.base + d.nb <= a.ps && d.base + a.B <= a.ncap && d.f0 >= 0 &&
           d.nf >= 0 && d.nf <= a.Fmax && d.f0 + d.nf <= a.nentries && d.h0 >= 0 && d.nh >= 0 && d.nh <= a.Hmax &&
           d.h0 + d.nh <= a.nhalo;
}

// The next tile of the queue, a predicated atomic: with a branch around it the warp would wait for
// the result where the branch ends, not where the tile is needed.
__device__ __forceinline__ void claim_tile(int* queue, bool on, int& tile) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %2, 0;\n\t@p atom.global.add.u32 %0, [%1], 1;\n\t}"
                 : "+r"(tile) : "l"(queue), "r"((int) on) : "memory");
}

// The producer's own latencies are pipelined over tiles: while tile t0 is staged, the halo ids and
// instance scalars of t1, the descriptor of t2 and the claim of the tile after it are on their way.
// Done one after the other for each tile they made the producer the slower side (5,200 cycles a
// tile in FP64 pass 1 and 4,700-5,500 in the FP32 passes, where computing one takes 3,500 and
// 1,700-2,000).  A deeper pipeline of claims (five tiles by position, results taken up an iteration
// later) cost FP64 2 % at 2001x1001: tiles claimed early are tiles the CTAs that end first cannot take.
template <class T, bool PASS2, bool ARENA, bool GEN>
__device__ __forceinline__ void producer_loop(const TileArgs<T>& a, unsigned char* smem, unsigned long long* full,
                                              unsigned long long* empty, const TileSmem<T>& L) {
    const int lane = threadIdx.x & 31;
    constexpr int CU = sizeof(Cell4<T>) / 16, CG = PASS2 ? sizeof(Grad8<T>) / 16 : 0;
    constexpr int KH = 4;          // halo ids a lane holds for the next tile (128 a tile; the rest are loaded late)
    const int NL = a.B + a.Hmax;   // plane stride of the staged cells
    volatile int* abort = abort_word(smem);
    int armed[2] = {-1, -1};       // last iteration whose copies were issued into each buffer
    // dt or CFL number, dt minimum (pass 2) and step count of the tile's instance; none of them changes
    // during the kernel in a way the kernel reads (dt minima and step counts come from earlier kernels)
    struct Scalars {
        double dt, dtmin;
        long long steps;
    };
    auto load_scalars = [&](int inst, Scalars& v) {      // (from L2: the kernel before may still run)
        v.dt = ARENA ? __ldg(a.inst_dt + inst) : a.s.dt_or_cfl;
        if constexpr (PASS2)
            v.dtmin = __longlong_as_double((long long) __ldcg(ARENA ? a.inst_dtmin + 2 * inst + a.par : a.s.dtmin));
        else
            v.steps = __ldcg(ARENA ? &a.inst_stats[inst].steps : &a.s.stats->steps);
    };
    // A descriptor as loaded (nothing computed from it until it is needed, a tile later).
    struct Raw {
        int x, y, z, w, u, v, first;
    };
    // (Not inside a branch, past the end the last tile's is read again: where a branch's sides meet,
    // the warp would wait for what one of them loaded.)
    const int last = a.ntiles - 1;
    auto load_raw = [&](int tile, Raw& q) {
        tile = min(tile, last);
        if constexpr (ARENA) {
            const int4 e0 = __ldg(a.tiles + 2 * tile);
            const int4 e1 = __ldg(a.tiles + 2 * tile + 1);
            q = Raw{e0.x, e0.y, e0.z, e0.w, e1.x, e1.y, e1.z};
        } else {
            q = Raw{__ldg(a.foff + tile), __ldg(a.foff + tile + 1), __ldg(a.hoff + tile), __ldg(a.hoff + tile + 1), 0, 0, 0};
        }
    };
    auto describe = [&](int tile, const Raw& q) {
        TileDesc d;
        tile = min(tile, last);
        if constexpr (ARENA) {
            d = TileDesc{q.x, a.B, q.y, q.z, q.u, q.v, q.w, q.first};
        } else {
            const int base = tile * a.B;
            d = TileDesc{base, min(a.B, a.s.Nc - base), q.x, q.y - q.x, q.z, q.w - q.z, 0, 0};
        }
        if constexpr (kChecked)
            if (!index_ok(desc_ok<T>(a, d), a.err)) d.nb = d.nf = d.nh = -1;   // staged empty
        return d;
    };
    auto load_ids = [&](int tile, const TileDesc& d, int id[KH]) {
        // Arena: never inside a branch either (an empty halo reads one past its place, where the list is
        // padded): its steps took 129 us with the branch, 116 without.  Single mesh, where descriptors
        // need no instance: only the ids there are (FP32 pass 2 40 us against 35).
        if (!ARENA && tile >= a.ntiles) return;
        const int top = max(d.nh - 1, 0);
#pragma unroll
        for (int k = 0; k < KH; k++)
            if (ARENA || lane + 32 * k < d.nh) id[k] = __ldg(a.halo + d.h0 + min(lane + 32 * k, top));
    };
    // the first three tiles are the CTA's by position; the queue hands out the rest
    int t0 = blockIdx.x, t1 = t0 + (int) gridDim.x, t2 = t1 + (int) gridDim.x;
    TileDesc d0, d1;
    Raw q0{}, q1{}, q2{};
    Scalars v0{}, v1{};
    int id0[KH], id1[KH];
    load_raw(t0, q0);
    load_raw(t1, q1);
    d0 = describe(t0, q0);
    load_ids(t0, d0, id0);
    d1 = describe(t1, q1);
    // Copies into stage `buf` what no kernel writes of a tile, its face records and metadata, face words
    // and 1 / areas, and adds their bytes to the stage's phase.
    auto stage_static = [&](const TileDesc& d, bool good, int buf) {
        if (lane != 0) return;
        const unsigned nf = good ? d.nf : 0;
        const bool short_words = GEN && a.cslot;
        const unsigned bf = nf * a.rec * (unsigned) sizeof(T), bm = PASS2 || short_words ? nf * 4u : 0u;
        const unsigned bs = good ? a.B * a.Wp * (short_words ? sizeof(short) : sizeof(unsigned)) : 0u;
        const unsigned bi = good ? a.B * sizeof(T) : 0u;
        unsigned char* st = smem + kHeader + buf * L.stage;
        mbar_expect_tx(full + buf, bf + bm + bs + bi);
        if (bf) {
            bulk_g2s(st + L.geo, a.tgeo + (size_t) d.f0 * a.rec, bf, full + buf);
            if (bm) bulk_g2s(st + L.meta, a.tmeta + d.f0, bm, full + buf);
        }
        if (bs) {
            bulk_g2s(st + L.nbr, short_words ? (const void*) (a.cslot + (size_t) d.base * a.Wp) : a.nbr + (size_t) d.base * a.Wp,
                     bs, full + buf);
            bulk_g2s(st + L.iv, a.s.iv + d.base, bi, full + buf);
        }
    };
    // the first tile's while the kernel before this one ends; everything else waits for it
    if (t0 < a.ntiles && t0 != a.skip_tile) stage_static(d0, !kChecked || d0.nb >= 0, 0);
    grid_wait_previous();
    load_scalars(d0.inst, v0);
    v1 = v0;
    for (unsigned iter = 0;; iter++) {
        const int buf = iter & 1;
        load_raw(t2, q2);
        load_ids(t1, d1, id1);
        int pending = 0;
        if (ARENA) load_scalars(d1.inst, v1);
        claim_tile(a.claim, a.claim && lane == 0 && t2 < a.ntiles, pending);
        if (__any_sync(0xffffffffu, *abort)) break;
        if (iter >= 2 && !__all_sync(0xffffffffu, mbar_wait(empty + buf, ((iter >> 1) - 1) & 1, a.polls, a.err, abort)))
            break;
        if (t0 >= a.ntiles) {
            // no more tiles: a stage with tile -1 and nothing copied ends the compute warps' loop
            grid_launch_next();      // this CTA's place falls free soon
            if (lane == 0) {
                reinterpret_cast<StageInfo*>(smem + 64)[buf].t = -1;
                mbar_arrive_expect_tx(full + buf, 0u);
            }
            cp_async_arrive_noinc(full + buf);
            armed[buf] = (int) iter;
            break;
        }
        if (t0 != a.skip_tile) {             // failure injection: nothing armed, nothing in flight
            const bool good = !kChecked || d0.nb >= 0;
            const int base = d0.base, nb = good ? d0.nb : 0, nf = good ? d0.nf : 0, nh = good ? d0.nh : 0;
            unsigned char* st = smem + kHeader + buf * L.stage;
            Cell4<T>* sU = reinterpret_cast<Cell4<T>*>(st + L.u);
            Grad8<T>* sG = reinterpret_cast<Grad8<T>*>(st + L.g);
            if (iter) stage_static(d0, good, buf);
            if (lane == 0) {
                // the tile's descriptor and instance scalars, published by the release of the arrive
                StageInfo* si = reinterpret_cast<StageInfo*>(smem + 64) + buf;
                si->base = base; si->nb = nb; si->f0 = d0.f0; si->nf = nf; si->h0 = d0.h0; si->nh = nh; si->inst = d0.inst;
                si->t = t0;
                si->first = d0.first;
                si->next_inst = (ARENA && !PASS2 && t1 < a.ntiles) ? d1.inst : -1;
                si->dt_or_cfl = v0.dt;
                si->dtmin = v0.dtmin;
                si->steps = v0.steps;
                mbar_arrive_expect_tx(full + buf, nb * (unsigned) (sizeof(Cell4<T>) + (PASS2 ? sizeof(Grad8<T>) : 0)));
                if (nb) {
                    // one bulk copy per 16-byte chunk plane of the tile's cell range
#pragma unroll
                    for (int j = 0; j < CU; j++)
                        bulk_g2s(reinterpret_cast<char*>(sU) + (size_t) 16 * j * NL,
                                 reinterpret_cast<const char*>(a.s.U) + 16 * ((size_t) j * a.ps + base), nb * 16u, full + buf);
#pragma unroll
                    for (int j = 0; j < CG; j++)
                        bulk_g2s(reinterpret_cast<char*>(sG) + (size_t) 16 * j * NL,
                                 reinterpret_cast<const char*>(a.s.phiG) + 16 * ((size_t) j * a.ps + base), nb * 16u,
                                 full + buf);
                }
            }
            auto gather = [&](int h, int ci) {
                if (!index_ok(ci >= 0 && ci < a.ps, a.err)) return;
#pragma unroll
                for (int j = 0; j < CU; j++)
                    cp_async16(reinterpret_cast<char*>(sU) + 16 * ((size_t) j * NL + a.B + h),
                               reinterpret_cast<const char*>(a.s.U) + 16 * ((size_t) j * a.ps + ci));
#pragma unroll
                for (int j = 0; j < CG; j++)
                    cp_async16(reinterpret_cast<char*>(sG) + 16 * ((size_t) j * NL + a.B + h),
                               reinterpret_cast<const char*>(a.s.phiG) + 16 * ((size_t) j * a.ps + ci));
            };
#pragma unroll
            for (int k = 0; k < KH; k++)
                if (lane + 32 * k < nh) gather(lane + 32 * k, id0[k]);
            for (int h = lane + 32 * KH; h < nh; h += 32) gather(h, __ldg(a.halo + d0.h0 + h));
            cp_async_arrive_noinc(full + buf);
            armed[buf] = (int) iter;
        }
        t0 = t1; d0 = d1; v0 = v1;
#pragma unroll
        for (int k = 0; k < KH; k++) id0[k] = id1[k];
        t1 = t2;
        d1 = describe(t2, q2);
        if (t2 < a.ntiles)
            t2 = a.claim ? 3 * (int) gridDim.x + __shfl_sync(0xffffffffu, pending, 0) : t2 + (int) gridDim.x;
    }
    cp_async_wait_all();
    if ((int) blockIdx.x < a.ntiles && (int) blockIdx.x != a.skip_tile && armed[0] < 0) {
        // The CTA gave up before the first tile's stage was armed in full, with its static copies in flight:
        // the stage is closed as at the end, with tile -1 and the arrivals it lacks, and completes when
        // they have landed.  (The test is formed anew: kept in a register through the loop, it cost the FP32
        // arena's step 0.2 %.)
        if (lane == 0) {
            reinterpret_cast<StageInfo*>(smem + 64)[0].t = -1;
            mbar_arrive(full);
        }
        cp_async_arrive_noinc(full);
        armed[0] = 0;
    }
    for (int b = 0; b < 2; b++)
        if (armed[b] >= 0) mbar_drain(full + b, ((unsigned) armed[b] >> 1) & 1, a.err);
}

// Residual / non-finite / dt bookkeeping shared by the last pass of a step.
template <class T>
__device__ __forceinline__ void finish_step(const StepArgs<T>& a, double r2, int bad, double dt_used) {
    __shared__ double sm[32];
    __shared__ int smbad[32];
    __shared__ bool last;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    double w = warp_sum(r2);
    int wb = __any_sync(0xffffffffu, bad);
    if (lane == 0) { sm[wid] = w; smbad[wid] = wb; }
    __syncthreads();
    if (wid == 0) {
        const int nw = (int) (blockDim.x >> 5);
        double x = lane < nw ? sm[lane] : 0.0;
        int xb = lane < nw ? smbad[lane] : 0;
        x = warp_sum(x);
        xb = __any_sync(0xffffffffu, xb);
        if (lane == 0) {
            a.partial[blockIdx.x] = x;
            if (xb) atomicOr(&a.stats->nonfinite, 1);
            __threadfence();
            const unsigned int done = atomicAdd(a.counter, 1u);
            last = (done == gridDim.x - 1);
        }
    }
    __syncthreads();
    if (last) {
        __threadfence();
        double x = 0.0;
        for (int i = threadIdx.x; i < (int) gridDim.x; i += blockDim.x) x += ((volatile double*) a.partial)[i];
        x = warp_sum(x);
        if (lane == 0) sm[wid] = x;
        __syncthreads();
        if (threadIdx.x == 0) {
            double tot = 0.0;
            for (int i = 0; i < (int) (blockDim.x >> 5); i++) tot += sm[i];
            StepStats* st = a.stats;
            st->res2_last = tot;
            if (st->steps == 0) st->res2_first = tot;
            st->steps += 1;
            st->dt_last = dt_used;
            if (!(tot == tot) || tot > 1.7e308) st->nonfinite = 1;
            *a.counter = 0u;
            // after a fixed step too: the next call may step under a CFL number, and the other slot
            // holds the minimum of the step before
            *a.dtmin_next = 0x7FF0000000000000ULL;
        }
    }
}

// ---------------------------------------------------------------------------------------

// One face entry of pass 2: operands gathered from shared memory and reduced at once to the
// MUSCL states on both sides (Flux.cpp:83-87), then the Rusanov flux in the face's own
// L -> R orientation.  Only the reconstructed states stay live between load and flux.
template <class T>
struct FaceIn {
    T uoL[4], uqR[4], nx, ny, Af;
    int e;
    __device__ __forceinline__ void load(const Cell4<T>* sU, const Grad8<T>* sG, int NL, const T* sGeo,
                                         const unsigned* sMeta, int nf, int rec, int e_) {
        e = e_;
        const unsigned w = sMeta[e];
        const int bc = meta_bc(w);
        const int mx = meta_la(w), my = meta_lb(w);
        const int rp = rplane(rec);
        // Ghost on the right: -grad and the same phi as the interior cell with r_R = -r_L
        // (BoundaryConditions/Base.cpp:29-53, Domain.cpp:84-88): the same increment, so both
        // sides read the left cell's gradient and r.
        const bool interior = bc < 0;
        const auto n2 = ldp(sGeo, nf, 0, e), rl = ldp(sGeo, nf, rp, e), rr = ldp(sGeo, nf, interior ? rp + 1 : rp, e);
        nx = n2.x; ny = n2.y; Af = lds_area(sGeo, nf, e, rec);
        T gL[8], gR[8];
        lds_cell(sU, NL, mx, uoL);
        lds_cell(sU, NL, my, uqR);
        lds_grad(sG, NL, mx, gL);
        lds_grad(sG, NL, interior ? my : mx, gR);
#pragma unroll
        for (int v = 0; v < 4; v++) {
            uoL[v] += gL[2 * v] * rl.x + gL[2 * v + 1] * rl.y;
            uqR[v] += gR[2 * v] * rr.x + gR[2 * v + 1] * rr.y;
        }
    }
    __device__ __forceinline__ void flux(T gma, T F[4]) const { rusanov(uoL, uqR, nx, ny, gma, F); }
    // F as two pairs at sF (plane stride nf).  With AF the product A_f F is stored instead (the
    // compensated FP32 sums round that product before adding it, so forming it once per face
    // gives the same bits as forming it in each of the two cells).
    template <bool AF>
    __device__ __forceinline__ void store(T* sF, int nf, const T F[4]) const {
        if (AF) {
            stp(sF, nf, 0, e, F[0] * Af, F[1] * Af);
            stp(sF, nf, 1, e, F[2] * Af, F[3] * Af);
        } else {
            stp(sF, nf, 0, e, F[0], F[1]);
            stp(sF, nf, 1, e, F[2], F[3]);
        }
    }
};

// Sum of A_f F over one cell's faces in increasing face order (Flux.cpp:39-42), F as stored by
// FaceIn::store at sF.  NVAR 2: the sums of variable pair j alone.  FP32 sums are compensated; the first term needs no two-sum,
// 0 + x being exact.
template <class T, int W, bool COMP, int NVAR>
__device__ __forceinline__ void cell_flux_sum(const unsigned x[W], const T* sF, const T* sGeo, int nf, int rec, int j, T* R,
                                              unsigned int* err) {
    T Rc[NVAR];
#pragma unroll
    for (int v = 0; v < NVAR; v++) { R[v] = T(0); Rc[v] = T(0); }
#pragma unroll
    for (int k = 0; k < W; k++) {
        if (W > 3 && x[k] == kNoFace) continue;
        // (W = 3) an unused position reads entry 0 with weight zero, in place of a branch per face
        const bool on = W > 3 || x[k] != kNoFace;
        int e = on ? nbr_entry(x[k]) : 0;
        if constexpr (kChecked) e = index_ok(e < nf, err) ? e : 0;
        T Fk[NVAR];
#pragma unroll
        for (int h = 0; h < NVAR / 2; h++) {
            const auto f = ldp(sF, nf, NVAR == 4 ? h : j, e);
            Fk[2 * h] = f.x; Fk[2 * h + 1] = f.y;
        }
        // one face's flux leaves its left cell and enters its right one; COMP: Fk holds A_f F
        T w = COMP ? T(1) : lds_area(sGeo, nf, e, rec);
        w = nbr_right(x[k]) ? w : -w;
        if (W == 3) w = on ? w : T(0);
#pragma unroll
        for (int v = 0; v < NVAR; v++) {
            if constexpr (COMP) {
                if (k == 0) R[v] = w * Fk[v];
                else two_sum(R[v], Rc[v], __fmul_rn(w, Fk[v]));
            } else {
                R[v] += w * Fk[v];
            }
        }
    }
    if constexpr (COMP)
#pragma unroll
        for (int v = 0; v < NVAR; v++) R[v] += Rc[v];
}

// The wave-speed sum of a cell with state u.
template <class T, int W>
__device__ __forceinline__ T cell_wave_sum(const unsigned x[W], const T* sGeo, int nf, int rec, const T u[4], T gma,
                                           unsigned int* err) {
    T cu, cv, ca, lam = T(0);
    cell_speed(u, gma, cu, cv, ca);
#pragma unroll
    for (int k = 0; k < W; k++) {
        if (W > 3 && x[k] == kNoFace) continue;
        const bool on = W > 3 || x[k] != kNoFace;
        int e = on ? nbr_entry(x[k]) : 0;
        if constexpr (kChecked) e = index_ok(e < nf, err) ? e : 0;
        T nx, ny, A;
        lds_geo3(sGeo, nf, e, rec, nx, ny, A);
        lam += wave(cu, cv, ca, nx, ny, on ? A : T(0));
    }
    return lam;
}

// U += dt R (Flux.cpp:45-49, Euler.cpp:107-113); returns the density residual R_rho.
// `top` keeps the largest exponent word seen, for not_finite.
__device__ __forceinline__ int exponent_word(double x) { return __double2hiint(x) & 0x7FFFFFFF; }
__device__ __forceinline__ int exponent_word(float x) { return __float_as_int(x) & 0x7FFFFFFF; }
template <class T>
__device__ __forceinline__ bool not_finite(int top) { return top >= (sizeof(T) == 8 ? 0x7FF00000 : 0x7F800000); }
template <int NVAR, class T>
__device__ __forceinline__ T cell_update(const T* u, const T* R, T iv, T dt, T* un, int& top) {
#pragma unroll
    for (int v = 0; v < NVAR; v++) {
        un[v] = u[v] + dt * (R[v] * iv);
        top = max(top, exponent_word(un[v]));
    }
    return R[0] * iv;
}

// Warp-specialised persistent tile loop.  The last warp of the CTA is the producer
// (producer_loop); the first NT = blockDim.x - 32 threads compute.  Compute iteration i
// reads staging buffer i & 1 once its `full` barrier completes and releases it on its
// `empty` barrier (one arrival per compute warp) when done.  The tile comes with the stage
// (StageInfo::t); after the CTA's last tile the producer stages tile -1 with nothing copied,
// and the compute warps leave the loop on it (in pass 2 after the face-phase barrier, which
// every compute warp meets once more).
// A compute warp whose stage wait gives up reads nothing of that stage.  In pass 1 (no
// barrier among the compute warps inside the loop) it leaves the loop at once.  In pass 2
// it marks the compute abort word and skips the face phase (`staged` false); every compute
// warp then meets at the compute barrier that ends the face phase and leaves the loop
// there if any of them gave up, so none is left waiting at that barrier.
#define HCFD_TILE_LOOP_BEGIN(PASS2, ARENA, GEN)                                                  \
    const int NT = blockDim.x - 32;                                                              \
    const int NL = a.B + a.Hmax;                                                                 \
    unsigned long long* full = reinterpret_cast<unsigned long long*>(smem);                      \
    unsigned long long* empty = full + 2;                                                        \
    if (threadIdx.x == 0) {                                                                      \
        mbar_init(full, 33); mbar_init(full + 1, 33);                                            \
        mbar_init(empty, NT / 32); mbar_init(empty + 1, NT / 32);                                \
        *abort_word(smem) = 0;                                                                   \
        *compute_abort_word(smem) = 0;                                                           \
        fence_mbar_init();                                                                       \
    }                                                                                            \
    __syncthreads();                                                                             \
    if ((int) threadIdx.x >= NT) {                                                               \
        producer_loop<T, PASS2, ARENA, GEN>(a, smem, full, empty, L);                            \
    } else {                                                                                     \
    grid_wait_previous();                                                                        \
    if (a.claim_reset && blockIdx.x == 0 && threadIdx.x == 0) *a.claim_reset = 0;               \
    for (unsigned iter = 0;; iter++) {                                                           \
        const int buf = iter & 1;                                                                \
        unsigned char* st = smem + kHeader + buf * L.stage;                                      \
        const bool staged = __all_sync(0xffffffffu,                                              \
                                       mbar_wait(full + buf, (iter >> 1) & 1, a.polls, a.err,    \
                                                 abort_word(smem)));                             \
        if (!PASS2 && !staged) break;                                                            \
        if (PASS2 && !staged && (threadIdx.x & 31) == 0) *compute_abort_word(smem) = 1;          \
        const StageInfo& si = reinterpret_cast<const StageInfo*>(smem + 64)[buf];                \
        const int t = staged ? si.t : 0;                                                         \
        const bool fin = staged && t < 0;     /* the producer has no more tiles */               \
        if (!PASS2 && fin) break;                                                                \
        const int base = si.base, nb = si.nb, inst = si.inst;                                   \
        const Cell4<T>* sU = reinterpret_cast<const Cell4<T>*>(st + L.u);                        \
        const T* sGeo = reinterpret_cast<const T*>(st + L.geo);                                  \
        const int nfl = si.nf;                                                                   \
        const unsigned* sNbr = reinterpret_cast<const unsigned*>(st + L.nbr);                    \
        const unsigned* sMeta = reinterpret_cast<const unsigned*>(st + L.meta);                  \
        const T* sIv = reinterpret_cast<const T*>(st + L.iv);

#define HCFD_TILE_LOOP_END                                                                       \
        __syncwarp();                                                                            \
        if ((threadIdx.x & 31) == 0) mbar_arrive(empty + buf);                                   \
    }                                                                                            \
    }

// Pair j of a cell's variables (0: rho, rho u; 1: rho v, E) in chunk planes.
__device__ __forceinline__ double2* pair_at(Cell4<double>* p, size_t ps, int i, int j) {
    return reinterpret_cast<double2*>(p) + j * ps + i;
}
__device__ __forceinline__ float2* pair_at(Cell4<float>* p, size_t, int i, int j) {
    return reinterpret_cast<float2*>(p) + 2 * (size_t) i + j;
}
// Limited gradients of pair j (four values) into chunk planes.
__device__ __forceinline__ void st_grad_pair(Grad8<double>* p, size_t ps, int i, int j, const double g[4]) {
    double2* q = reinterpret_cast<double2*>(p) + 2 * j * ps + i;
    q[0] = make_double2(g[0], g[1]);
    q[ps] = make_double2(g[2], g[3]);
}
__device__ __forceinline__ void st_grad_pair(Grad8<float>* p, size_t ps, int i, int j, const float g[4]) {
    reinterpret_cast<float4*>(p)[j * ps + i] = make_float4(g[0], g[1], g[2], g[3]);
}
template <int NVAR, class T>   // all four variables, or pair j
__device__ __forceinline__ void st_vars(Cell4<T>* p, size_t ps, int i, int j, const T* u) {
    if constexpr (NVAR == 4) {
        st_cell(p, ps, i, u);
    } else {
        auto* q = pair_at(p, ps, i, j);
        q->x = u[0]; q->y = u[1];
    }
}
template <int NVAR, class T>
__device__ __forceinline__ void lds_vars(const Cell4<T>* p, int ps, int i, int j, T* u) {
    if constexpr (NVAR == 4) {
        lds_cell(p, ps, i, u);
    } else {
        const auto x = *pair_at(const_cast<Cell4<T>*>(p), ps, i, j);
        u[0] = x.x; u[1] = x.y;
    }
}

// Pass 1 of tile cell c (pair j of its variables when NVAR is 2) up to the limiter's increments,
// operands from shared memory (its centre-to-face vectors stay in ro): its face words in x, nf entries,
// nb tile cells and nh halo cells of NL staged.  Unrolled: the face loads overlap.
template <class T, int W, int NVAR>
__device__ __forceinline__ void tile_faces(Pass1Cell<T, NVAR>& p, const unsigned x[W], const Cell4<T>* sU, const T* sGeo, int NL,
                                           int nf, int c, int j, bool with_lam, T gma, T iv, int nb, int B, int nh,
                                           unsigned int* err, T (&ro)[W][2]) {
    lds_vars<NVAR>(sU, NL, c, j, p.u);
    p.begin(with_lam, gma, p.u);
#pragma unroll
    for (int k = 0; k < W; k++) {
        ro[k][0] = T(0); ro[k][1] = T(0);
        if (W > 3 && x[k] == kNoFace) continue;
        // A position a cell does not use (W = 3: a cell of an open mesh with fewer faces) reads
        // entry 0 with zero length, the cell itself as its neighbour and r = 0, which adds
        // nothing, in place of a branch per face.
        const bool on = W > 3 || x[k] != kNoFace;
        int e = on ? nbr_entry(x[k]) : 0, nbl = on ? nbr_local(x[k]) : c;
        const bool isL = !nbr_right(x[k]);
        if constexpr (kChecked) {  // a bad index is replaced by entry 0 / tile cell 0 (no branch)
            e = index_ok(e < nf, err) ? e : 0;
            nbl = index_ok(!on || local_ok(nbl, nb, B, nh), err) ? nbl : 0;
        }
        FaceGeo<T> g;
        lds_geo4(sGeo, nf, e, g);
        T un[NVAR];
        lds_vars<NVAR>(sU, NL, nbl, j, un);
        p.face(un, isL, g.nx, g.ny, on ? g.Af : T(0), g.If, with_lam);
        // this cell's own centre-to-face vector: one pair, at its side's plane
        const auto rr = ldp(sGeo, nf, isL ? 2 : 3, e);
        ro[k][0] = on ? rr.x : T(0);
        ro[k][1] = on ? rr.y : T(0);
    }
    p.gradient(iv);
#pragma unroll
    for (int k = 0; k < W; k++) p.increment(ro[k][0], ro[k][1]);
}

// LIM and LAM: the limiter and whether the CFL sums are wanted, fixed at compile time (the branches
// on them, eight a cell, and the register moves where their sides meet were a tenth of the kernel's
// instructions), or kRunTime or kRareToo.
template <class T, int W, bool ARENA, int LIM, int LAM>
__global__ void __maxnreg__(sizeof(T) == 8 ? 128 : W == 3 ? 56 : 72) tile_pass1_kernel(const TileArgs<T> a) {
    extern __shared__ __align__(128) unsigned char smem[];
    constexpr bool GEN = LIM == kRareToo;
    const TileSmem<T> L(a.B, a.Hmax, a.Fmax, W, a.Wp, false, GEN && a.cslot);
    const StepArgs<T>& s = a.s;
    T xmx = T(0);                        // largest iv * lam (see dt_of_max)
    HCFD_TILE_LOOP_BEGIN(false, ARENA, GEN)
    const int lmode = limiter_mode(si.steps, s.freeze_after);
    const bool with_lam = LAM >= 0 ? LAM != 0 : s.time_mode != TM_FIXED;
    for (int c = threadIdx.x; c < nb; c += NT) {
        unsigned x[W];
        cell_words<W, GEN>(sNbr, a.cslot, sMeta, c, x);
        if (x[0] == kNoFace) continue;
        Pass1Cell<T> p;
        const T iv = sIv[c];
        T ro[W][2];
        tile_faces<T, W, 4>(p, x, sU, sGeo, NL, nfl, c, 0, with_lam, s.gma, iv, nb, a.B, si.nh, a.err, ro);
        T out[8], phis[4];
        if (lmode == LIM_FROZEN) ld_cell_l2(s.phiF, a.ps, base + c, phis);
        else if (LIM == kRareToo && by_face(s.limiter, s.venkat_K)) p.limiter_by_face(iv, s.venkat_K, ro, phis);
        else p.template limiter_values<LIM>(iv, s.limiter, s.venkat_K, phis);
        p.limited(phis, out);
        if (lmode == LIM_RECORD) st_cell(s.phiF, a.ps, base + c, phis);
        st_grad(s.phiG, a.ps, base + c, out);
        if (with_lam) xmx = fmax(xmx, iv * p.lam);
    }
    if constexpr (ARENA) {
        // per-instance minimum (exact and order-free): each warp carries its minimum across
        // this CTA's consecutive tiles of one instance and posts it with one atomic when the
        // next tile belongs to another instance, so a large instance sees a few atomics per
        // CTA rather than one per warp and tile on a single address
        if (with_lam) {
            if (si.next_inst != inst) {
                const double m = dt_of_max(warp_max(xmx));
                if ((threadIdx.x & 31) == 0 && m < 1e300)
                    atomicMin(a.inst_dtmin + 2 * inst + a.par, (unsigned long long) __double_as_longlong(m));
                xmx = T(0);
            }
        }
    }
    HCFD_TILE_LOOP_END
    if (!ARENA && (LAM >= 0 ? LAM != 0 : s.time_mode != TM_FIXED)) {
        __shared__ T sm[32];
        T m = warp_max(xmx);
        const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
        if (lane == 0) sm[wid] = m;
        __syncthreads();
        if (wid == 0) {
            m = lane < (int) (blockDim.x >> 5) ? sm[lane] : T(0);
            const double d = dt_of_max(warp_max(m));
            if (lane == 0 && d < 1e300) atomicMin(s.dtmin, (unsigned long long) __double_as_longlong(d));
        }
    }
}

// REC and LOCAL: the record length and local time stepping, fixed at compile time as in pass 1
// (or kRunTime or kRareToo).
template <class T, int W, bool ARENA, int REC, int LOCAL>
__global__ void __maxnreg__(128) tile_pass2_kernel(const TileArgs<T> a) {
    constexpr bool COMP = sizeof(T) == 4;
    extern __shared__ __align__(128) unsigned char smem[];
    constexpr bool GEN = REC == kRareToo;
    const TileSmem<T> L(a.B, a.Hmax, a.Fmax, W, a.Wp, true, GEN && a.cslot);
    const StepArgs<T>& s = a.s;
    double dt_used = 0.0;
    double r2 = 0.0;
    int top = 0;
    const int rec = REC >= 0 ? REC : a.rec;
    const bool local = LOCAL >= 0 ? LOCAL != 0 : s.time_mode == TM_LOCAL;
    HCFD_TILE_LOOP_BEGIN(true, ARENA, GEN)
    const T cfl_or_dt = T(si.dt_or_cfl);
    if (staged && !fin) dt_used = (s.time_mode == TM_FIXED) ? si.dt_or_cfl : si.dt_or_cfl * si.dtmin;
    const Grad8<T>* sG = reinterpret_cast<const Grad8<T>*>(st + L.g);
    // a stage whose wait gave up is not read, nor the closing stage (tile -1)
    const int nf = (staged && !fin) ? nfl : 0;
    // face phase: one Rusanov flux per face entry (Flux.cpp:19-38).  Each thread takes two
    // entries per round and computes both before storing either, so the two independent
    // FP64 dependency chains (divisions, square roots) interleave.
    // Threads below nf - NT (per round) have a second entry.  In FP64, whole warps take the
    // one-entry path when none of their threads has one (the warp that straddles the boundary
    // takes the two-entry path throughout, its threads without a second entry computing theirs
    // twice, so that no warp runs both paths one after the other); this saves FP64 work.  In
    // FP32 every warp takes the two-entry path: the flux is cheap there, and measured on the
    // B200 the split costs more than it saves.
    // The fluxes go over the r pairs of the staged records, which only the entry's own thread
    // reads in pass 2, and has read by then.
    T* sF = reinterpret_cast<T*>(st + L.geo) + 2 * rplane(rec) * nf;
    for (int e = threadIdx.x; e < nf; e += 2 * NT) {
        const int base2 = e - (int) threadIdx.x;                 // first entry of this round
        const int pairs = min(NT, max(0, nf - base2 - NT));      // threads with a second entry
        if (sizeof(T) == 4 || (int) (threadIdx.x & ~31u) < pairs) {
            const int eB = (e + NT < nf) ? e + NT : e;
            if constexpr (kChecked)
                if (!entry_ok(sMeta[e], nb, a.B, si.nh, a.err) || !entry_ok(sMeta[eB], nb, a.B, si.nh, a.err)) continue;
            FaceIn<T> A, Bq;
            A.load(sU, sG, NL, sGeo, sMeta, nf, rec, e);
            Bq.load(sU, sG, NL, sGeo, sMeta, nf, rec, eB);
            T FA[4], FB[4];
            A.flux(s.gma, FA);
            Bq.flux(s.gma, FB);
            A.template store<COMP>(sF, nf, FA);
            if (eB != e) Bq.template store<COMP>(sF, nf, FB);
        } else {
            if constexpr (kChecked)
                if (!entry_ok(sMeta[e], nb, a.B, si.nh, a.err)) continue;
            FaceIn<T> A;
            A.load(sU, sG, NL, sGeo, sMeta, nf, rec, e);
            T FA[4];
            A.flux(s.gma, FA);
            A.template store<COMP>(sF, nf, FA);
        }
    }
    compute_sync(NT);
    // some compute warp's stage wait gave up, or the closing stage (every compute warp that
    // read the stage sees its tile -1; one whose wait gave up sees the abort word)
    if (*compute_abort_word(smem) || fin) break;
    // cell phase: slots in increasing face order, update, ghost refresh
    for (int c = threadIdx.x; c < nb; c += NT) {
        unsigned x[W];
        cell_words<W, GEN>(sNbr, a.cslot, sMeta, c, x);
        if (x[0] == kNoFace) continue;
        T u[4];
        lds_cell(sU, NL, c, u);
        const T iv = sIv[c];
        T R[4], un_[4];
        cell_flux_sum<T, W, COMP, 4>(x, sF, sGeo, nf, rec, 0, R, a.err);
        T dt = T(dt_used);
        if (local) dt = cfl_or_dt * qrcp(iv * cell_wave_sum<T, W>(x, sGeo, nf, rec, u, s.gma, a.err));
        const T Rr = cell_update<4>(u, R, iv, dt, un_, top);
        if (a.want_res) r2 += (double) Rr * (double) Rr;
        st_cell(s.Unew, a.ps, base + c, un_);
        // ghost refresh (Euler.cpp:96, :138-142): this cell is its ghosts' only neighbour
        bool any = false;
#pragma unroll
        for (int k = 0; k < W; k++) any |= x[k] != kNoFace && (x[k] & kBoundaryFace);
        if (!any) continue;
#pragma unroll 1
        for (int k = 0; k < W; k++) {
            const unsigned xk = GEN && a.cslot ? nbr_word(reinterpret_cast<const short*>(sNbr)[c * W + k], sMeta) : sNbr[c * W + k];
            if (xk == kNoFace || !(xk & kBoundaryFace)) continue;
            const int e = nbr_entry(xk), lb = nbr_local(xk);
            if (!index_ok(e < nf && local_ok(lb, nb, a.B, si.nh), a.err)) continue;
            const int bc = meta_bc(sMeta[e]);
            if (!index_ok(bc >= 0 && bc < MAXBC, a.err)) continue;
            const int gi = lb < a.B ? base + lb : __ldg(a.halo + si.h0 + lb - a.B);
            if (!index_ok(gi >= 0 && gi < a.ps, a.err)) continue;
            T gnx, gny, gA;
            lds_geo3(sGeo, nf, e, rec, gnx, gny, gA);
            T ug[4];
            const BCTable* bt = ARENA ? a.inst_bc + inst : &s.bc;
            ghost_state(bt->type[bc], un_, gnx, gny, s.gma, bt->UBC[bc], bt->QBC[bc], ug);
            st_cell(s.Unew, a.ps, gi, ug);
        }
    }
    if constexpr (ARENA) {
        const int wb = __any_sync(0xffffffffu, not_finite<T>(top));
        if (a.want_res) {
            // per-tile residual: one partial per warp (fixed order, no barrier); the finalize
            // kernel sums an instance's partials in order and does the step's bookkeeping
            const double w = warp_sum(r2);
            if ((threadIdx.x & 31) == 0) {
                const int k = t * (NT >> 5) + (int) (threadIdx.x >> 5);
                a.tile_r2[k] = w;
                a.tile_bad[k] = wb;
            }
        } else {
            if (wb && (threadIdx.x & 31) == 0) atomicOr(&a.inst_stats[inst].nonfinite, 1);
            if (si.first && threadIdx.x == 0) {
                a.inst_stats[inst].steps += 1;
                a.inst_dtmin[2 * inst + (1 - a.par)] = 0x7FF0000000000000ULL;
            }
        }
        r2 = 0.0;
        top = 0;
    }
    HCFD_TILE_LOOP_END
    if constexpr (!ARENA) {
        if (a.want_res) {
            finish_step(s, r2, not_finite<T>(top), dt_used);
        } else {
            if (not_finite<T>(top)) atomicOr(&s.stats->nonfinite, 1);
            if (blockIdx.x == 0 && threadIdx.x == 0) {
                s.stats->steps += 1;
                *s.dtmin_next = 0x7FF0000000000000ULL;
            }
        }
    }
}

// The variants of a handle's shape.
template <class T>
using TileKernel = void (*)(const TileArgs<T>);
// Launches a tiled kernel so that it may start while the stream's kernel before it still runs: its
// CTAs take the places of those that have left, fetch what no kernel writes and wait for the rest
// in grid_wait_previous.
template <class T>
cudaError_t launch_dependent(TileKernel<T> kernel, int grid, int block, size_t smem, cudaStream_t stream, const TileArgs<T>& a) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, a);
}
template <class T, int W, bool ARENA>
TileKernel<T> pass1_variant(int limiter, double venkat_K, int time_mode, bool short_words = false) {
    if (by_face(limiter, T(venkat_K)) || short_words) return tile_pass1_kernel<T, W, ARENA, kRareToo, -1>;
    if constexpr (W == 8) {
        return tile_pass1_kernel<T, W, ARENA, kRunTime, -1>;
    } else {
        const bool lam = time_mode != TM_FIXED;
        if (limiter == LIM_BJ) return lam ? tile_pass1_kernel<T, W, ARENA, LIM_BJ, 1> : tile_pass1_kernel<T, W, ARENA, LIM_BJ, 0>;
        return lam ? tile_pass1_kernel<T, W, ARENA, LIM_VENKAT, 1> : tile_pass1_kernel<T, W, ARENA, LIM_VENKAT, 0>;
    }
}
template <class T, int W, bool ARENA>
TileKernel<T> pass2_variant(int rec, int time_mode, bool short_words = false) {
    if constexpr (!ARENA)
        if (short_words) return tile_pass2_kernel<T, W, ARENA, kRareToo, -1>;
    if constexpr (W == 8) {
        return tile_pass2_kernel<T, W, ARENA, kRunTime, -1>;
    } else {
        const bool local = time_mode == TM_LOCAL;
        if constexpr (!ARENA)
            if (rec == 7) return local ? tile_pass2_kernel<T, W, ARENA, 7, 1> : tile_pass2_kernel<T, W, ARENA, 7, 0>;
        return local ? tile_pass2_kernel<T, W, ARENA, 8, 1> : tile_pass2_kernel<T, W, ARENA, 8, 0>;
    }
}

// Face records in tile order, pair-major per tile, rec values each (8 or 7; see rplane):
// tile t with entries [f0, f0 + nf) starts at tgeo[rec f0] (zeros for padding).
template <class T>
__global__ void gather_geo_kernel(int ntiles, const int* __restrict__ foff, const int* __restrict__ efid,
                                  const FaceGeo<double>* __restrict__ geo, T* __restrict__ tgeo, int rec) {
    const int t = blockIdx.x;
    if (t >= ntiles) return;
    const int f0 = foff[t], nf = foff[t + 1] - f0;
    T* out = tgeo + (size_t) rec * f0;
    for (int e = threadIdx.x; e < nf; e += blockDim.x) {
        const int f = efid[f0 + e];
        double c[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        if (f >= 0) {
            const FaceGeo<double> g = geo[f];
            c[0] = g.nx; c[1] = g.ny; c[2] = g.Af; c[3] = g.If; c[4] = g.rLx; c[5] = g.rLy; c[6] = g.rRx; c[7] = g.rRy;
        }
        if (rec == 7) {
            stp(out, nf, 0, e, T(c[0]), T(c[1]));
            stp(out, nf, 1, e, T(c[4]), T(c[5]));
            stp(out, nf, 2, e, T(c[6]), T(c[7]));
            out[6 * nf + e] = T(c[2]);
        } else {
#pragma unroll
            for (int j = 0; j < 4; j++) stp(out, nf, j, e, T(c[2 * j]), T(c[2 * j + 1]));
        }
    }
}

}  // namespace hcfd
