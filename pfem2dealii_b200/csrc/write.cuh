// The write pass: count correction, the new sorted layout, projection partial
// sums and the step's counters, in one kernel.
//
// A block takes a tile of consecutive cells, whose old slots are one range of
// the arrays.  The range is bulk-copied into shared memory, the cells'
// arrivals are gathered behind it, and the block then works on these entries
// one per thread: part counts, survivors of over-full parts (by key), places
// in the new layout (stayers by a prefix of their survival bits, arrivals by
// their key), stores.  A particle that stays in its cell is read from global
// memory once, one that changed it twice (with its old cell's slots, and as an
// arrival), and a warp's lanes are all in use whatever a cell holds.  At last
// a warp per cell takes the partial sums from the staged entries in the new
// order.
//
// What bounds it, and why tiles.  A time step's memory traffic here is 69
// bytes a particle (FP32, 3D): 73 us for 7 M at the HBM rate.  One warp per
// cell with one register round per 32 particles (the layout before) lost its
// lanes to cells of 33 or 97 particles, could stage four cells only at
// seeding density, re-read the written particles for the partial sums of
// cells above 32, and sent cells above 96 to a path that counts positions
// through global scratch.  A run seeded with one particle a part and max 2
// fills towards 1.9 a part (54 a cell at 27 parts, 124 at 64) at a pace that
// depends on the flow: after 500 steps a 12^3 cube holds 1.83, a 64x16 channel
// 1.49 and a 32x8x8 duct 1.20 (1.47 after 1200), so full cells take those
// paths, and runs stay between the two densities for long (LIGHT).  Measured,
// before -> now: duct FP32 (7.0 M particles) 480 -> 199 us, FP64 940 -> 406;
// cube FP32 (32 M) 8414 -> 917, 37^3 cube FP64 (6.2 M) 3253 -> 373; Turek
// mesh FP32 (1.9 M) 291 -> 91, FP64 429 -> 140.  Now bound by instruction
// issue and the latencies a tile waits on one after the other (its copies,
// about a third of its time, five barriers): a tile's headers and first
// arrivals are therefore copied while the tile before it is worked on, and
// its new particles, whose parts are known from the move's occupancy, are
// computed while its copies are in flight (221 -> 199 us with both).
#pragma once

#include "cellwork.cuh"

namespace pfem2 {

template <int DIM, typename Real>
struct PData {
    uint32_t i, id;
    Real xi[DIM], v[DIM];
    Real x[std::is_same<Real, double>::value ? DIM : 1];
};

template <int DIM, typename Real>
__device__ __forceinline__ void load_global(const StepArgs& a, uint32_t i, PData<DIM, Real>& p)
{
    p.i = i;
    p.id = a.S0.id[i];
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
        p.xi[d] = ldr<Real>(a.T.xi[d], i);
        p.v[d] = ldr<Real>(a.T.v[d], i);
        if constexpr (std::is_same<Real, double>::value) p.x[d] = ldr<double>(a.T.x[d], i);
    }
}

template <int DIM, typename Real>
__device__ __forceinline__ void store_particle(const StepArgs& a, uint32_t dst, uint32_t c, const PData<DIM, Real>& p)
{
    a.S1.cell[dst] = c;
    a.S1.id[dst] = p.id;
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
        str<Real>(a.S1.xi[d], dst, p.xi[d]);
        str<Real>(a.S1.v[d], dst, p.v[d]);
        if constexpr (std::is_same<Real, double>::value) str<double>(a.S1.x[d], dst, p.x[d]);
    }
}

// Empty slots [from, to) of a cell's range (one warp).
__device__ __forceinline__ void write_holes(const StepArgs& a, uint32_t from, uint32_t to, int lane)
{
    for (uint32_t j = from + lane; j < to; j += 32)
        if (j < a.capacity) a.S1.cell[j] = HOLE;
}

// New particles of one cell (one warp): the k-th seeded part (in part order)
// goes to slot base + k and gets id id0 + sb + k + 1.  Returns the number of
// new particles and error bits.
template <int DIM, typename Real>
__device__ __forceinline__ uint2 write_seeds(const StepArgs& a, uint32_t c, const int* cnt, uint32_t n, uint32_t base,
                                             uint32_t id0, uint32_t sb, int lane)
{
    uint32_t done = 0, err = 0;
    for (int p0 = 0; p0 < a.pp.npe; p0 += 32) {
        const int p = p0 + lane;
        const bool sf = p < a.pp.npe && gets_seed(a, p, cnt[p < a.pp.npe ? p : 0], n);
        const unsigned m = __ballot_sync(0xffffffffu, sf);
        if (sf) {
            const uint32_t k = done + __popc(m & ((1u << lane) - 1u));
            const uint32_t dst = base + k;
            int idx[3] = {0, 0, 0};
            real_part<DIM>(p, a.pp, idx);
            if (dst < a.capacity) new_particle<DIM, Real>(a, a.S1, dst, c, idx, id0 + sb + k + 1);
            else err |= ERR_CAPACITY;
        }
        done += __popc(m);
    }
    return make_uint2(done, err);
}

// A cell's new range [off, off + ub), within the capacity, and the advect
// chunks' recorded slots (ADV_REC) in it.
__device__ __forceinline__ void new_range(const StepArgs& a, uint32_t c, uint32_t off, uint32_t ub)
{
    const uint32_t first = off < a.capacity ? off : a.capacity, end = ub < a.capacity - first ? first + ub : a.capacity;
    a.cs_new[c] = first;
    if (a.chunk_first)
        for (uint32_t k = (first + ADV_REC - 1) / ADV_REC; (uint64_t)k * ADV_REC < end; ++k) a.chunk_first[k] = c;
}

// FP32 partial sums of up to 32 particles, one per lane (lanes without a
// particle add zeros): a pairwise tree over the 32 rows, then one compensated
// add into acc (lane = entry).  The first level of the tree, rows
// u + (u + 16), is taken through one shuffle instead of shared memory: lane
// u < 16 keeps the entries of the vertices whose highest reference-coordinate
// bit is clear, lane u + 16 those with it set, and receives them from its
// partner, so each entry crosses the warp once and 16 rows of PW entries are
// staged; the tree's other levels follow.  Shape values and products are
// those of partial_row (N = (x0 factor * x1 factor) * x2 factor).  EXACT:
// every product is rounded before it is added, as partial_row's are.
template <int DIM, bool EXACT>
__device__ __forceinline__ void partial_pairs32(float (*tr)[TRW], bool active, const float* xi, const float* v,
                                                int lane, PartialAcc<float>& acc)
{
    constexpr int NV = 1 << DIM, H = NV / 2, PW = Dims<DIM>::PW;
    const bool hi = lane >= 16;
    float x[DIM], w[DIM];
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
        x[d] = active ? xi[d] : 0.0f;
        w[d] = active ? v[d] : 0.0f;
    }
    float lowN[H];  // products of the factors below the highest direction
#pragma unroll
    for (int k = 0; k < H; ++k) {
        float n = (k & 1) ? x[0] : 1.0f - x[0];
        if (DIM > 2) n *= ((k >> 1) & 1) ? x[1] : 1.0f - x[1];
        lowN[k] = n;
    }
    // a lane without a particle adds nothing (its shape values are zero too)
    const float top = x[DIM - 1], bot = 1.0f - x[DIM - 1];
    const float fk = active ? (hi ? top : bot) : 0.0f, fs = active ? (hi ? bot : top) : 0.0f;
    float keep[4 * H];
#pragma unroll
    for (int k = 0; k < H; ++k) {
        const float nk = EXACT ? __fmul_rn(lowN[k], fk) : lowN[k] * fk;
        const float ns = EXACT ? __fmul_rn(lowN[k], fs) : lowN[k] * fs;
        float e[4], f[4];
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
            e[d] = EXACT ? __fmul_rn(nk, w[d]) : nk * w[d];
            f[d] = EXACT ? __fmul_rn(ns, w[d]) : ns * w[d];
        }
        e[DIM] = nk;
        f[DIM] = ns;
        if (DIM == 2) e[3] = f[3] = 0.0f;
#pragma unroll
        for (int j = 0; j < 4; ++j) keep[4 * k + j] = e[j] + __shfl_xor_sync(0xffffffffu, f[j], 16);
    }
    const int row = lane & 15, col0 = hi ? 4 * H : 0;
#pragma unroll
    for (int k = 0; k < H; ++k)
        *reinterpret_cast<float4*>(&tr[row][col0 + 4 * k]) =
            make_float4(keep[4 * k], keep[4 * k + 1], keep[4 * k + 2], keep[4 * k + 3]);
    __syncwarp();
    if (lane < PW) {
        float t[16];
#pragma unroll
        for (int r = 0; r < 16; ++r) t[r] = tr[r][lane];
#pragma unroll
        for (int wd = 8; wd >= 1; wd >>= 1)
#pragma unroll
            for (int r = 0; r < wd; ++r) t[r] = t[r] + t[r + wd];
        const float y = t[0] - acc.c;
        const float sm = acc.s + y;
        acc.c = (sm - acc.s) - y;
        acc.s = sm;
    }
}

// FP64 partial sums of up to 32 particles, one per lane, added to acc in lane
// order, as the oracle adds them (lane = entry): 16 rows of PW entries at a
// time through shared memory.  5 instructions a particle; one lane per entry
// that recomputes or shuffles the shape values takes 15 (duct write pass,
// 7.0 M particles: 489 us against 406).
template <int DIM>
struct Rows64 {
    static constexpr int W = DIM == 3 ? 34 : 18;  // 16-byte stores of 8 lanes meet no bank twice
};
template <int DIM>
__device__ __forceinline__ void partial_rows64(double (*tr)[Rows64<DIM>::W], uint32_t rows, const double* xi,
                                               const double* v, int lane, double& acc)
{
    constexpr int NV = 1 << DIM, PW = Dims<DIM>::PW;
    double N[NV];
    shape64<DIM>(xi, N);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const uint32_t n = rows > 16u * h ? (rows - 16u * h < 16u ? rows - 16u * h : 16u) : 0u;
        if (n == 0) break;
        if ((lane >> 4) == h && (uint32_t)lane < rows) {
            double* t = tr[lane & 15];
#pragma unroll
            for (int iv = 0; iv < NV; ++iv) {
                *reinterpret_cast<double2*>(t + iv * 4) = make_double2(N[iv] * v[0], N[iv] * v[1]);
                *reinterpret_cast<double2*>(t + iv * 4 + 2) =
                    DIM == 3 ? make_double2(N[iv] * v[DIM - 1], N[iv]) : make_double2(N[iv], 0.0);
            }
        }
        __syncwarp();
        if (lane < PW) {
            if (n == 16) {
#pragma unroll
                for (int r = 0; r < 16; ++r) acc = acc + tr[r][lane];
            } else {
                for (uint32_t r = 0; r < n; ++r) acc = acc + tr[r][lane];
            }
        }
        __syncwarp();
    }
}

// Copies of a few bytes, global -> shared, that complete at async_wait.
template <int BYTES>
__device__ __forceinline__ void async_copy(void* dst, const void* src)
{
    if constexpr (BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_u32(dst)), "l"(src), "n"(BYTES) : "memory");
}
__device__ __forceinline__ void async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// ---------------------------------------------------------------------------
// Tiles.  TCAP entries (old slots, arrivals, new particles) fit one tile's
// shared memory.  The kernel takes as many cells per tile as bring it near
// TARGET particles at the layout's mean density, and then shares the cells
// out over the waves of blocks this takes; a tile that holds more than TCAP is
// worked through in runs of cells that fit, and a single cell beyond TCAP
// takes the general path.  Sizes measured (write pass, us; FP32 duct of 7.0 M
// particles / cube of 32 M): 512 entries, 7 blocks per SM 215 / 990; 640, 6
// blocks 199 / 917; 896, 5 blocks 202 / 868, which leaves smaller meshes too
// few tiles.  FP64 (duct / 37^3 cube): 384, 5 blocks 520 / 532; 512, 4 blocks
// 489 / 465.
//
// Where cells differ little, more waves of smaller tiles only add tiles: with
// 8 waves in place of 2 or 3 a 64x16x16 duct of 0.9 M particles takes 61 us
// for 39 in FP32 and 83 for 71 in FP64, a 30^3 cube of 1.4 M 76 for 53 and
// 109 for 103.  Where the largest cell has more than 8 times the smallest
// one's volume, the small ones' arrivals make some tiles much the larger, and
// smaller tiles even that out: Turek mesh, 1.9 M, FP32 4 waves 125 us, 6 89, 8
// 94; FP64 8 waves 145, 13 137; seeded cylinder channel of 25 k cells FP32 1
// wave 56, 5 44, 8 52.  So at least 6 waves there while a tile keeps 100
// entries, and never more than `most` entries a tile.  (The ratio is 98 and
// 72 on these meshes, 1.7 on the cube with its vertices moved by a tenth.)
// ---------------------------------------------------------------------------
constexpr int WT_CELLS = 24;  // cells per tile at most
constexpr int WT_CNT = 1024;  // part counters of a run of cells
constexpr int WT_ARR = 8;     // arrivals per cell copied with its header
constexpr int WT_OCC = 32;    // occupancy words of a tile: cells x ceil(npe / 64), where cells x npe <= WT_CNT

template <int DIM, typename Real>
struct WtCfg {
    static constexpr bool HX = std::is_same<Real, double>::value;
    static constexpr int TCAP = HX ? 512 : 640;
    static constexpr int TARGET = HX ? 470 : 600;
    static constexpr int WARPS = 4, THREADS = WARPS * 32, BLOCKS = HX ? 4 : 6;
};

// One cell of any particle count (the whole block), for the cells that fit no
// tile.  Per-element data goes to the cell's own slot range of the scratch
// array; survivors and positions are found by counting.  Order: stayers by
// slot, arrivals by key, new particles by part -- the same as the tiles'.
// Quadratic in the cell's particles, so all threads share the counting: with
// one warp of the block at it a 64x16x16 duct of 54 a cell with 800 in one of
// 50 took 6354 us in FP32 and 8679 in FP64 (a warp per cell before the tiles
// 4164 and 3779), now 1716 and 2262; 1536 cells of 700 3950 and 5408, now 1274
// and 1733.
template <int DIM, typename Real>
__device__ __noinline__ uint2 write_cell_general(const StepArgs& a, int* cnt, uint32_t* sc, Real (*tr)[TRW], uint32_t c,
                                                 uint32_t s0, uint32_t L, uint32_t na, uint32_t h, uint32_t off,
                                                 uint32_t ub, uint32_t nseed_expect, uint32_t sb, uint32_t id0)
{
    constexpr int WARPS = WtCfg<DIM, Real>::WARPS, THREADS = WtCfg<DIM, Real>::THREADS;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    uint32_t removed = 0, err = 0;
    uint4* G = a.gscr + off;  // element -> (particle index, part, key, flags: 1 stayer, 2 survivor)
    const int npe = a.pp.npe;
    for (int p = tid; p < npe; p += THREADS) cnt[p] = 0;
    if (tid == 0) sc[WARPS] = 0;  // survivors
    __syncthreads();
    // nothing is written for a cell that does not fit: its slots are empty, not what stood there two steps ago
    auto refuse = [&](uint32_t flag) {
        for (uint32_t j = off + tid; j < off + ub && j < a.capacity; j += THREADS) a.S1.cell[j] = HOLE;
        return make_uint2(0u, flag);
    };
    if (off + ub > a.capacity) return refuse(ERR_CAPACITY);
    // stayers: elements 0..ns-1 in slot order
    uint32_t ns = 0;
    for (uint32_t base = 0; base < L; base += THREADS) {
        const uint32_t j = base + tid;
        const bool stay = j < L && a.key[s0 + j] == c;
        const unsigned m = __ballot_sync(0xffffffffu, stay);
        if (lane == 0) sc[warp] = __popc(m);
        __syncthreads();
        uint32_t before = ns;
#pragma unroll
        for (int k = 0; k < WARPS; ++k) {
            before += k < warp ? sc[k] : 0u;
            ns += sc[k];
        }
        if (stay) {
            const uint32_t i = s0 + j, e = before + __popc(m & ((1u << lane) - 1u));
            Real xi[DIM];
#pragma unroll
            for (int d = 0; d < DIM; ++d) xi[d] = ldr<Real>(a.T.xi[d], i);
            const int pe = ext_part<DIM, Real>(xi, a.pp);
            if (e < ub) G[e] = make_uint4(i, (uint32_t)pe, key_of(a.S0.id[i], a.pp.seed), 1u);
            atomicAdd(cnt + pe, 1);
        }
        __syncthreads();
    }
    // arrivals: elements ns.. (slots in parallel; the overflow list walked by all threads)
    uint32_t t = 0, p = h;
    for (; t < na && t < a.capacity; ++t) {
        uint32_t i;
        if (t < (uint32_t)ARRCAP) {
            i = a.carrs[(size_t)c * ARRCAP + t];
        } else {
            if (p == LOST) break;
            i = p;
            p = a.next[p];
        }
        if (t % THREADS == (uint32_t)tid) {
            Real xi[DIM];
#pragma unroll
            for (int d = 0; d < DIM; ++d) xi[d] = ldr<Real>(a.T.xi[d], i);
            const int pe = ext_part<DIM, Real>(xi, a.pp);
            if (ns + t < ub) G[ns + t] = make_uint4(i, (uint32_t)pe, key_of(a.S0.id[i], a.pp.seed), 0u);
            atomicAdd(cnt + pe, 1);
        }
    }
    const uint32_t n = ns + t;
    __syncthreads();
    if (n > ub) return refuse(ERR_COUNT_UB);
    // survivors: rank by key (equal ones by particle) inside the part
    uint32_t nsurv = 0;
    for (uint32_t e = tid; e < n; e += THREADS) {
        const uint4 g = G[e];
        const int k = cnt[g.y];
        int rank = 0;
        if (a.apply_counts && k > a.pp.maxpp + 1) {
#pragma unroll 8
            for (uint32_t m = 0; m < n; ++m) {
                const uint4 o = G[m];
                rank += (o.y == g.y && (o.z < g.z || (o.z == g.z && o.x < g.x))) ? 1 : 0;
            }
        }
        if (rank < survivors(k, a.pp.maxpp, a.apply_counts)) {
            G[e].w = g.w | 2u;
            nsurv++;
        } else {
            removed++;
        }
    }
    nsurv = __reduce_add_sync(0xffffffffu, nsurv);
    if (lane == 0) atomicAdd(&sc[WARPS], nsurv);
    __syncthreads();
    nsurv = sc[WARPS];
    // positions: survivors before in (stayers by slot | arrivals by key) order
    for (uint32_t e = tid; e < n; e += THREADS) {
        const uint4 g = G[e];
        if (!(g.w & 2u)) continue;
        const bool gs = g.w & 1u;
        uint32_t pos = 0;
#pragma unroll 8
        for (uint32_t m = 0; m < n; ++m) {
            const uint4 o = G[m];
            const bool os = o.w & 1u;
            const bool less = os ? o.x < g.x : o.z < g.z || (o.z == g.z && o.x < g.x);
            pos += ((o.w & 2u) && ((os && !gs) || (os == gs && less))) ? 1u : 0u;
        }
        PData<DIM, Real> pd;
        load_global<DIM, Real>(a, g.x, pd);
        store_particle<DIM, Real>(a, off + pos, c, pd);
    }
    __syncthreads();
    if (warp == 0) {
        const uint2 sd = write_seeds<DIM, Real>(a, c, cnt, n, off + nsurv, id0, sb, lane);
        err |= sd.y;
        const uint32_t fin = nsurv + sd.x;
        if (sd.x != nseed_expect) err |= ERR_COUNT;
        if (fin > ub) err |= ERR_COUNT_UB;
        write_holes(a, off + fin, off + ub, lane);
        __syncwarp();
        __threadfence_block();
        partials_of_range<DIM, Real>(a, a.S1, c, off, fin < ub ? fin : ub, tr, lane);
    }
    return make_uint2(removed, err);
}

// What a tile needs to know of its cells, copied while the tile before it is
// worked on.
struct __align__(16) WtHead {
    uint32_t arr[WT_CELLS][WT_ARR];  // the first arrivals
    unsigned long long occ[WT_OCC];  // occupied parts, occw words per cell
    uint2 co[WT_CELLS + 1];          // x: new slot offset, y: new particles before
    uint32_t cs[WT_CELLS + 1];       // old slots
    uint32_t na[WT_CELLS];           // arrivals
    uint32_t aoff[WT_CELLS + 1];     // and their offsets in the tile
    uint32_t tile;                   // written while other warps may still read the header before it
};

template <int DIM, typename Real>
struct __align__(128) WtTile {
    static constexpr bool HX = WtCfg<DIM, Real>::HX;
    static constexpr int TCAP = WtCfg<DIM, Real>::TCAP;
    union {
        struct {
            uint32_t key[TCAP];  // old slots: the move's cell; arrivals: key_of(id), the dead ones' ~0
            uint32_t id[TCAP];
            int cnt[WT_CNT];
            uint16_t meta[TCAP];  // arrivals, new particles, over-full parts: local cell << 8 | extended part
        };
        // FP32 partial rows, 16 per warp (once placed)
        Real tr[HX ? 1 : WtCfg<DIM, Real>::WARPS][HX ? 1 : 16][TRW];
    };
    Real x[HX ? DIM : 1][HX ? TCAP : 4];  // FP64: the partial rows take the space up to its end
    Real xi[DIM][TCAP];
    Real v[DIM][TCAP];
    using Row64 = double[16][Rows64<DIM>::W];
    static_assert(!HX || 10 * TCAP + 4 * WT_CNT + DIM * TCAP * 8 >= (int)sizeof(Row64) * WtCfg<DIM, Real>::WARPS,
                  "the rows fit where keys, ids, counters and positions were");
    uint16_t perm[TCAP];       // over-full parts' entries, then the entry of each new slot
    uint32_t mask[TCAP / 32];  // survivors
    WtHead hdr[2];             // this tile's cells and the next one's
    uint64_t bar;
    uint32_t nover;
    int ties[2];  // below zero once equal keys share a rank: over-full parts, arrivals
};

// Equal keys (a caller's duplicate ids, or 32-bit ids that wrapped) go by the
// particles' indices, so that every entry has a rank and a place of its own:
// a place that two entries share would leave another without one, and the
// partial sums would take what stands there for an entry.  The ranks of k
// distinct keys add up to k (k - 1) / 2, those of equal ones to less: k_write
// sums the difference over a run (a compare in its inner loops instead costs
// 4 % of the FP32 pass) and calls these two, all threads together, where it
// is not zero.
template <int DIM, typename Real>
__device__ __forceinline__ uint32_t entry_particle(const StepArgs& a, const WtHead& h, uint32_t c0, uint32_t lc,
                                                   uint32_t SA, uint32_t nold, uint32_t a0, uint32_t e)
{
    if (e < nold) return SA + e;
    const uint32_t k = e - nold - (h.aoff[lc] - a0);
    if (k < (uint32_t)WT_ARR) return h.arr[lc][k];
    if (k < (uint32_t)ARRCAP) return a.carrs[(size_t)(c0 + lc) * ARRCAP + k];
    uint32_t p = a.head[c0 + lc];
    for (uint32_t t = ARRCAP; t < k && p < a.capacity; ++t) p = a.next[p];
    return p;
}

// Over-full entries (perm[0 .. nov)) that survive by their key but not by
// their index; returns how many this thread took out.
template <int DIM, typename Real>
__device__ __noinline__ uint32_t ties_in_parts(const StepArgs& a, WtTile<DIM, Real>& w, uint32_t hb, uint32_t c0,
                                               uint32_t cb, uint32_t ce, uint32_t nov)
{
    const WtHead& h = w.hdr[hb];
    const uint32_t SA = h.cs[cb] & ~3u, nold = h.cs[cb] < h.cs[ce] ? ((h.cs[ce] + 3u) & ~3u) - SA : 0u;
    uint32_t out = 0;
    for (uint32_t j = threadIdx.x; j < nov; j += WtCfg<DIM, Real>::THREADS) {
        const uint32_t e = w.perm[j], me = w.meta[e], lc = me >> 8, kk = key_of(w.id[e], a.pp.seed);
        const uint32_t i = entry_particle<DIM, Real>(a, h, c0, lc, SA, nold, h.aoff[cb], e);
        int rank = 0, before = 0;
        for (uint32_t o = 0; o < nov; ++o) {
            const uint32_t f = w.perm[o], kf = key_of(w.id[f], a.pp.seed);
            if (w.meta[f] != me) continue;
            rank += kf < kk ? 1 : 0;
            before += kf == kk && entry_particle<DIM, Real>(a, h, c0, lc, SA, nold, h.aoff[cb], f) < i ? 1 : 0;
        }
        if (rank < a.pp.maxpp + 1 && rank + before >= a.pp.maxpp + 1) {
            atomicAnd(w.mask + (e >> 5), ~(1u << (e & 31u)));
            w.key[e] = ~0u;
            out++;
        }
    }
    __syncthreads();  // every thread has seen the count and the list
    if (threadIdx.x == 0) w.ties[0] = 0;
    return out;
}

// Arrivals of one key: the places after the first, and the first once more
// (all of them were put there).
template <int DIM, typename Real>
__device__ __noinline__ void ties_in_cells(const StepArgs& a, WtTile<DIM, Real>& w, uint32_t hb, uint32_t c0,
                                           uint32_t cb, uint32_t ce)
{
    const WtHead& h = w.hdr[hb];
    const uint32_t SA = h.cs[cb] & ~3u, nold = h.cs[cb] < h.cs[ce] ? ((h.cs[ce] + 3u) & ~3u) - SA : 0u;
    const uint32_t a0 = h.aoff[cb], nE = nold + h.aoff[ce] - a0, ob = h.co[cb].x;
    auto live = [&](uint32_t e) { return (w.mask[e >> 5] >> (e & 31u)) & 1u; };
    for (uint32_t e = nold + threadIdx.x; e < nE; e += WtCfg<DIM, Real>::THREADS) {
        if (!live(e)) continue;
        const uint32_t lc = w.meta[e] >> 8, o1 = nold + h.aoff[lc + 1] - a0;
        const uint32_t i = entry_particle<DIM, Real>(a, h, c0, lc, SA, nold, a0, e);
        uint32_t pos = 0, same = 0;
        for (uint32_t o = nold + h.aoff[lc] - a0; o < o1; ++o) {
            if (!live(o)) continue;
            const bool eq = w.key[o] == w.key[e];
            same += eq ? 1u : 0u;
            pos += (w.key[o] < w.key[e] || (eq && entry_particle<DIM, Real>(a, h, c0, lc, SA, nold, a0, o) < i)) ? 1u : 0u;
        }
        if (same < 2) continue;
        if (nold)
            for (uint32_t o = h.cs[lc] - SA; o < h.cs[lc + 1] - SA; ++o) pos += live(o);
        const uint32_t dst = h.co[lc].x + pos;
        if (pos >= h.co[lc + 1].x - h.co[lc].x) continue;
        w.perm[dst - ob] = (uint16_t)e;
        if (dst >= a.capacity) continue;
        a.S1.cell[dst] = c0 + lc;
        a.S1.id[dst] = w.id[e];
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
            str<Real>(a.S1.xi[d], dst, w.xi[d][e]);
            str<Real>(a.S1.v[d], dst, w.v[d][e]);
            if constexpr (WtTile<DIM, Real>::HX) str<double>(a.S1.x[d], dst, w.x[d][e]);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) w.ties[1] = 0;
}

// LIGHT: an instance for layouts of few particles per part (note_density): a run
// in whose cells no part can be over-full, by their counts and their occupied
// parts, takes no part counts.  The two give the same results.
template <int DIM, typename Real, bool LIGHT>
__global__ void __launch_bounds__((WtCfg<DIM, Real>::THREADS), (WtCfg<DIM, Real>::BLOCKS))
    k_write(const __grid_constant__ StepArgs a)
{
    constexpr bool HX = WtCfg<DIM, Real>::HX;
    constexpr int TCAP = WtCfg<DIM, Real>::TCAP, TARGET = WtCfg<DIM, Real>::TARGET;
    constexpr int WARPS = WtCfg<DIM, Real>::WARPS, THREADS = WARPS * 32, ROUNDS = TCAP / THREADS;
    constexpr int HW = WARPS - 1;  // the warp that keeps the tickets and the headers
    constexpr uint32_t NONE = 0xffffu;
    static_assert(TCAP % THREADS == 0 && TCAP / 32 < 32, "whole rounds, one survivor word per lane");
    extern __shared__ __align__(128) unsigned char wr_raw[];
    auto& w = *reinterpret_cast<WtTile<DIM, Real>*>(wr_raw);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const unsigned ltm = (1u << lane) - 1u;
    if (tid == 0) {
        mbar_init(&w.bar, 1);
        mbar_fence_init();
        w.nover = 0;
        w.ties[0] = w.ties[1] = 0;
    }
    pdl_entry();
    const uint32_t nC = (uint32_t)a.mesh.nC, cap = a.capacity;
    const uint32_t id0 = a.stats->next_id;
    const int apply = a.apply_counts, maxpp = a.pp.maxpp, npe = a.pp.npe, occw = a.pp.occw;
    uint32_t NC;  // cells per tile
    {
        // near TARGET particles at the mean density, in as few waves of blocks as that takes, each wave full
        const uint32_t total = (uint32_t)a.coff[nC];
        const unsigned long long by_load = total ? (unsigned long long)TARGET * nC / total : WT_CELLS;
        const uint32_t by_cnt = WT_CNT / npe;
        NC = by_load < WT_CELLS ? (uint32_t)by_load : WT_CELLS;
        NC = max(min(NC, by_cnt), 1u);
        uint32_t waves = (nC + NC * gridDim.x - 1) / (NC * gridDim.x);
        if (a.mesh.uneven) {  // smaller cells are left by more of their particles: more and smaller tiles even that out
            const uint32_t block = total / gridDim.x, most = HX ? TCAP / 2 : TCAP * 3 / 5;
            waves = max(waves, max(min(6u, block / 100u), (block + most - 1) / most));
        }
        NC = min(NC, (nC + waves * gridDim.x - 1) / (waves * gridDim.x));
        NC = NC < 1 ? 1 : NC;
    }
    const uint32_t ntiles = (nC + NC - 1) / NC;
    auto cells_of = [&](uint32_t tile) { return tile >= ntiles ? 0u : nC - tile * NC < NC ? nC - tile * NC : NC; };
    unsigned long long removed = 0;
    uint32_t err = 0, phase = 0;
    bool stage_ok = true;  // cleared for good if a copy ever fails to land in time
    auto fetch_head = [&](WtHead& h, uint32_t tile) {
        const uint32_t c0 = tile * NC, ncell = cells_of(tile);
        if (ncell && (uint32_t)lane <= ncell) {
            async_copy<4>(&h.cs[lane], a.cs_old + c0 + lane);
            async_copy<8>(&h.co[lane], a.coff + c0 + lane);
        }
        if ((uint32_t)lane < ncell) {
            async_copy<4>(&h.na[lane], a.carr + c0 + lane);
#pragma unroll
            for (int k = 0; k < WT_ARR; k += 4)
                async_copy<16>(&h.arr[lane][k], a.carrs + (size_t)(c0 + lane) * ARRCAP + k);
        }
        if ((uint32_t)lane < ncell * occw) async_copy<8>(&h.occ[lane], a.cocc + (size_t)c0 * occw + lane);
    };
    auto land_head = [&](WtHead& h, uint32_t tile) {
        async_wait();
        __syncwarp();
        const uint32_t ncell = cells_of(tile);
        const uint32_t na = (uint32_t)lane < ncell ? h.na[lane] : 0u;
        uint32_t inc = na;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += y;
        }
        if ((uint32_t)lane <= ncell) h.aoff[lane] = inc - na;
        if (lane == 0) h.tile = tile;
    };
    uint32_t tk = 0;  // (the header warp) the next tile: the block's own first, then drawn ones
    if (warp == HW) {
        fetch_head(w.hdr[0], blockIdx.x);
        if (lane == 0) tk = gridDim.x + atomicAdd(&a.stats->write_next, 1u);
        land_head(w.hdr[0], blockIdx.x);
        tk = __shfl_sync(0xffffffffu, tk, 0);
    }
    for (uint32_t hb = 0;; hb ^= 1u) {
        __syncthreads();
        const WtHead& h = w.hdr[hb];
        const uint32_t tile = h.tile;
        if (tile >= ntiles) break;
        const uint32_t c0 = tile * NC, ncell = cells_of(tile);
        uint32_t tk2 = 0;
        if (warp == HW) {
            fetch_head(w.hdr[hb ^ 1u], tk);
            if (lane == 0) tk2 = gridDim.x + atomicAdd(&a.stats->write_next, 1u);
        }
        for (uint32_t cb = 0; cb < ncell;) {
            // the longest run of cells [cb, ce) that fits
            const uint32_t SA = h.cs[cb] & ~3u, a0 = h.aoff[cb], ob = h.co[cb].x, sb0 = h.co[cb].y;
            uint32_t ce;
            {
                const uint32_t j = cb + 1 + lane;
                bool fits = false;
                if (j <= ncell) {
                    const uint32_t ent = ((h.cs[j] + 3u) & ~3u) - SA + (h.aoff[j] - a0) + (h.co[j].y - sb0);
                    fits = ent <= (uint32_t)TCAP && h.co[j].x - ob <= (uint32_t)TCAP;
                }
                ce = cb + (uint32_t)__popc(__ballot_sync(0xffffffffu, fits));
            }
            if (ce == cb) {  // a single cell beyond a tile
                const uint32_t c = c0 + cb, ub = h.co[cb + 1].x - ob;
                auto* tr = reinterpret_cast<Real(*)[TRW]>(&w.xi[0][0]);  // rows where a tile's entries would be
                const uint2 gr = write_cell_general<DIM, Real>(a, w.cnt, w.mask, tr, c, h.cs[cb], h.cs[cb + 1] - h.cs[cb],
                                                               h.na[cb], a.head[c], ob, ub, h.co[cb + 1].y - sb0, sb0, id0);
                if (tid == 0) new_range(a, c, ob, ub);
                removed += gr.x;
                err |= gr.y;
                ce = cb + 1;
            } else {
                // Entries: the old slots [SA, EA), the arrivals, the new particles.
                const uint32_t E = h.cs[ce], EA = (E + 3u) & ~3u;
                const uint32_t nold = h.cs[cb] < E ? EA - SA : 0u, narr = h.aoff[ce] - a0;
                const uint32_t nE = nold + narr, nT = nE + (h.co[ce].y - sb0);
                // LIGHT, a cell per lane: can a part be over-full (the cell's count exceeds its occupied parts by
                // more than max)?  And the cells whose sums go by the old slots' rows (see there).
                bool count = true;
                uint32_t rows = 0;
                if constexpr (LIGHT) {
                    const uint32_t lc = cb + lane < ce ? cb + lane : cb;
                    const uint32_t nseed = h.co[lc + 1].y - h.co[lc].y, n = h.co[lc + 1].x - h.co[lc].x - nseed;
                    uint32_t occ = 0;
                    for (int q = 0; q < occw; ++q) occ += __popcll(h.occ[lc * occw + q]);
                    const bool over = apply && !(maxpp >= 0 && n <= occ + (uint32_t)maxpp);
                    rows = __ballot_sync(0xffffffffu, nseed == 0 && h.cs[lc + 1] - h.cs[lc] + h.na[lc] <= 32u && !over);
                    count = __any_sync(0xffffffffu, over);
                }
                if (nold) {
                    if (stage_ok) {
                        if (tid == 0) {
                            fence_proxy_async();  // the previous run's reads come first
                            constexpr uint32_t per = 8u + 2u * DIM * sizeof(Real) + (HX ? DIM * 8u : 0u);
                            mbar_expect_tx(&w.bar, nold * per);
                            bulk_g2s(w.key, a.key + SA, nold * 4u, &w.bar);
                            bulk_g2s(w.id, a.S0.id + SA, nold * 4u, &w.bar);
#pragma unroll
                            for (int d = 0; d < DIM; ++d) {
                                bulk_g2s(w.xi[d], reinterpret_cast<const Real*>(a.T.xi[d]) + SA,
                                         nold * (uint32_t)sizeof(Real), &w.bar);
                                bulk_g2s(w.v[d], reinterpret_cast<const Real*>(a.T.v[d]) + SA,
                                         nold * (uint32_t)sizeof(Real), &w.bar);
                                if constexpr (HX)
                                    bulk_g2s(w.x[d], reinterpret_cast<const double*>(a.T.x[d]) + SA, nold * 8u, &w.bar);
                            }
                        }
                    } else {
                        for (uint32_t j = tid; j < nold; j += THREADS) {
                            PData<DIM, Real> p;
                            load_global<DIM, Real>(a, SA + j, p);
                            w.key[j] = a.key[SA + j];
                            w.id[j] = p.id;
#pragma unroll
                            for (int d = 0; d < DIM; ++d) {
                                w.xi[d][j] = p.xi[d];
                                w.v[d][j] = p.v[d];
                                if constexpr (HX) w.x[d][j] = p.x[d];
                            }
                        }
                    }
                }
                // arrivals beyond their cell's slots: one thread walks each overflow list
                bool ovf = false;
                if (cb + lane < ce) ovf = h.na[cb + lane] > (uint32_t)ARRCAP;
                if (__any_sync(0xffffffffu, ovf)) {
                    if (warp == 0 && ovf) {
                        const uint32_t lc = cb + lane, na = h.na[lc];
                        uint32_t p = a.head[c0 + lc];
                        for (uint32_t k = ARRCAP; k < na; ++k) {
                            w.key[nold + (h.aoff[lc] - a0) + k] = p;
                            if (p < cap) p = a.next[p];
                        }
                    }
                    __syncthreads();
                }
                for (uint32_t t = tid; t < narr; t += THREADS) {
                    uint32_t lc = cb;
#pragma unroll
                    for (uint32_t st = 16; st; st >>= 1)
                        if (lc + st < ce && h.aoff[lc + st] - a0 <= t) lc += st;
                    const uint32_t k = t - (h.aoff[lc] - a0), e = nold + t;
                    const uint32_t i = k < (uint32_t)WT_ARR   ? h.arr[lc][k]
                                       : k < (uint32_t)ARRCAP ? a.carrs[(size_t)(c0 + lc) * ARRCAP + k]
                                                              : w.key[e];
                    if (i < cap) {
                        PData<DIM, Real> p;
                        load_global<DIM, Real>(a, i, p);
                        w.id[e] = p.id;
#pragma unroll
                        for (int d = 0; d < DIM; ++d) {
                            w.xi[d][e] = p.xi[d];
                            w.v[d][e] = p.v[d];
                            if constexpr (HX) w.x[d][e] = p.x[d];
                        }
                        w.meta[e] = (uint16_t)(lc << 8);
                    } else {
                        err |= ERR_ARRIVAL;
                        w.meta[e] = (uint16_t)NONE;
                    }
                }
                if (!LIGHT || count)
                    for (uint32_t t = tid; t < (ce - cb) * npe; t += THREADS) w.cnt[t] = 0;
                // new particles, while the copies are in flight: the real parts the move left empty
                {
                    uint32_t todo = __ballot_sync(0xffffffffu, cb + lane < ce && h.co[cb + lane + 1].y != h.co[cb + lane].y);
                    for (int k = 1; todo; ++k, todo &= todo - 1) {
                        if (k % WARPS != warp) continue;  // one cell per warp in turn, from the second warp on
                        const uint32_t lc = cb + __ffs(todo) - 1, sb = h.co[lc].y, n1 = h.co[lc + 1].y - sb;
                        uint32_t done = 0;
                        for (int p0 = 0; p0 < npe; p0 += 32) {
                            const int p = p0 + lane;
                            const bool sf = p < npe && ((a.pp.realmask[p >> 6] >> (p & 63)) & 1ull) &&
                                            (maxpp < 0 || !((h.occ[lc * occw + (p >> 6)] >> (p & 63)) & 1ull));
                            const unsigned b = __ballot_sync(0xffffffffu, sf);
                            const uint32_t j = done + __popc(b & ltm);
                            if (sf && j < n1) {
                                const uint32_t e = nE + (sb - sb0) + j;
                                int idx[3] = {0, 0, 0};
                                real_part<DIM>(p, a.pp, idx);
                                Real xi[DIM], v[DIM];
                                double x[DIM];
                                new_particle_at<DIM, Real>(a, c0 + lc, idx, xi, v, x);
#pragma unroll
                                for (int d = 0; d < DIM; ++d) {
                                    w.xi[d][e] = xi[d];
                                    w.v[d][e] = v[d];
                                    if constexpr (HX) w.x[d][e] = x[d];
                                }
                                w.id[e] = id0 + sb + j + 1;
                                w.meta[e] = (uint16_t)(lc << 8);
                            }
                            done += __popc(b);
                        }
                        if (done != n1) {  // every entry has a cell all the same
                            err |= ERR_COUNT;
                            for (uint32_t j = done + lane; j < n1; j += 32) w.meta[nE + (sb - sb0) + j] = (uint16_t)(lc << 8);
                        }
                    }
                }
                async_wait();
                if (nold && stage_ok) {
                    // one thread polls, the others rest at the barrier
                    if (__syncthreads_or(tid == 0 && !mbar_wait(&w.bar, phase))) {
                        // give the copy one more bounded wait, then stop staging; this run's particles are lost
                        err |= ERR_TIMEOUT;
                        if (tid == 0) mbar_wait(&w.bar, phase);
                        stage_ok = false;
                        __syncthreads();
                    }
                    phase ^= 1u;
                } else {
                    __syncthreads();
                }
                // cell and part of every entry; part counts.  Entry r * THREADS + tid stays in this thread's
                // registers; word r * WARPS + warp of the survivors is this warp's.
                uint32_t m[ROUNDS];
                auto place = [&](int r, uint32_t e) {
                    m[r] = NONE;
                    if (e < nold) {
                        const uint32_t lc = w.key[e] - c0, slot = SA + e;
                        if (lc >= cb && lc < ce && slot >= h.cs[lc] && slot < h.cs[lc + 1]) m[r] = lc << 8;
                    } else if (e < nT) {
                        m[r] = w.meta[e];
                        if (e < nE) w.key[e] = m[r] != NONE ? key_of(w.id[e], a.pp.seed) : ~0u;
                    }
                };
                if (!LIGHT || count) {
#pragma unroll
                    for (int r = 0; r < ROUNDS; ++r) {
                        const uint32_t e = r * THREADS + tid;
                        place(r, e);
                        if (e < nE && m[r] != NONE) {
                            Real xi[DIM];
#pragma unroll
                            for (int d = 0; d < DIM; ++d) xi[d] = w.xi[d][e];
                            const int pe = ext_part<DIM, Real>(xi, a.pp);
                            if (apply) atomicAdd(w.cnt + ((m[r] >> 8) - cb) * npe + pe, 1);
                            m[r] |= (uint32_t)pe;
                        }
                    }
                    __syncthreads();
                    // survivors: everyone outside the over-full parts, and there the smallest keys
                    bool over = false;
#pragma unroll
                    for (int r = 0; r < ROUNDS; ++r) {
                        const uint32_t e = r * THREADS + tid;
                        bool live = e < nE && m[r] != NONE;
                        if (live && apply && w.cnt[((m[r] >> 8) - cb) * npe + (m[r] & 255u)] > maxpp + 1) {
                            w.perm[atomicAdd(&w.nover, 1u)] = (uint16_t)e;
                            w.meta[e] = (uint16_t)m[r];
                            over = true;
                            live = false;
                        }
                        const unsigned b = __ballot_sync(0xffffffffu, live);
                        if (lane == 0) w.mask[r * WARPS + warp] = b;
                    }
                    if (__syncthreads_or(over)) {
                        const uint32_t nov = w.nover;
                        int tie = 0;
                        for (uint32_t j = tid; j < nov; j += THREADS) {
                            const uint32_t e = w.perm[j], me = w.meta[e], kk = key_of(w.id[e], a.pp.seed);
                            int rank = 0;
                            for (uint32_t o = 0; o < nov; ++o) {
                                const uint32_t f = w.perm[o], kf = key_of(w.id[f], a.pp.seed);
                                rank += (w.meta[f] == me && kf < kk) ? 1 : 0;
                            }
                            tie += 2 * rank - (w.cnt[((me >> 8) - cb) * npe + (me & 255u)] - 1);
                            if (rank < maxpp + 1) {
                                atomicOr(w.mask + (e >> 5), 1u << (e & 31u));
                            } else {
                                w.key[e] = ~0u;
                                removed++;
                            }
                        }
                        tie = __reduce_add_sync(0xffffffffu, tie);
                        if (lane == 0 && tie) atomicAdd(&w.ties[0], tie);
                        __syncthreads();
                        if (w.ties[0]) removed += ties_in_parts<DIM, Real>(a, w, hb, c0, cb, ce, nov);
                        if (tid == 0) w.nover = 0;
                    }
                } else {
#pragma unroll
                    for (int r = 0; r < ROUNDS; ++r) {
                        const uint32_t e = r * THREADS + tid;
                        place(r, e);
                        const unsigned b = __ballot_sync(0xffffffffu, e < nE && m[r] != NONE);
                        if (lane == 0) w.mask[r * WARPS + warp] = b;
                    }
                    __syncthreads();
                }
                // survivors before an entry: words by a scan over the lanes, bits by a count
                const uint32_t word = lane < TCAP / 32 ? w.mask[lane] : 0u;
                uint32_t wpre = __popc(word);
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t y = __shfl_up_sync(0xffffffffu, wpre, o);
                    if (lane >= o) wpre += y;
                }
                wpre -= __popc(word);
                auto before = [&](uint32_t e) {  // called by whole warps
                    const uint32_t p = __shfl_sync(0xffffffffu, wpre, (int)(e >> 5));
                    const uint32_t b = __shfl_sync(0xffffffffu, word, (int)(e >> 5));
                    return p + (uint32_t)__popc(b & ((1u << (e & 31u)) - 1u));
                };
                // the run's cells, one per lane: survivors before the cell's old slots, its stayers, all its survivors
                uint32_t c_pb, c_ns, c_nsurv;
                {
                    const uint32_t lc = cb + lane < ce ? cb + lane : cb;
                    c_pb = before(nold ? h.cs[lc] - SA : 0u);
                    c_ns = before(nold ? h.cs[lc + 1] - SA : 0u) - c_pb;
                    c_nsurv = c_ns + before(nold + h.aoff[lc + 1] - a0) - before(nold + h.aoff[lc] - a0);
                }
                // places and stores
                int ties = 0;
#pragma unroll
                for (int r = 0; r < ROUNDS; ++r) {
                    const uint32_t e = r * THREADS + tid;
                    const uint32_t wd = __shfl_sync(0xffffffffu, word, r * WARPS + warp);
                    const uint32_t ps = __shfl_sync(0xffffffffu, wpre, r * WARPS + warp) + __popc(wd & ltm);
                    const bool live = ((wd >> lane) & 1u) || (e >= nE && e < nT);
                    const uint32_t lc = live ? m[r] >> 8 : cb;
                    const uint32_t pb = __shfl_sync(0xffffffffu, c_pb, (int)(lc - cb));
                    const uint32_t nst = __shfl_sync(0xffffffffu, c_ns, (int)(lc - cb));
                    const uint32_t nsv = __shfl_sync(0xffffffffu, c_nsurv, (int)(lc - cb));
                    if (!live) continue;
                    const uint2 co = h.co[lc];
                    uint32_t pos;
                    if (e < nold) {
                        pos = ps - pb;
                    } else if (e < nE) {  // arrivals by key
                        pos = nst;
                        const uint32_t kk = w.key[e];
                        const uint32_t o1 = nold + h.aoff[lc + 1] - a0;
                        for (uint32_t o = nold + h.aoff[lc] - a0; o < o1; ++o)
                            pos += w.key[o] < kk ? 1u : 0u;
                        ties += 2 * (int)(pos - nst) - (int)(nsv - nst - 1u);
                    } else {
                        pos = nsv + (e - nE - (co.y - sb0));
                    }
                    const uint32_t dst = co.x + pos;
                    if (pos >= h.co[lc + 1].x - co.x) {
                        err |= ERR_COUNT_UB;
                        continue;
                    }
                    w.perm[dst - ob] = (uint16_t)e;
                    if (dst >= cap) {
                        err |= ERR_CAPACITY;
                        continue;
                    }
                    a.S1.cell[dst] = c0 + lc;
                    a.S1.id[dst] = w.id[e];
#pragma unroll
                    for (int d = 0; d < DIM; ++d) {
                        str<Real>(a.S1.xi[d], dst, w.xi[d][e]);
                        str<Real>(a.S1.v[d], dst, w.v[d][e]);
                        if constexpr (HX) str<double>(a.S1.x[d], dst, w.x[d][e]);
                    }
                }
                // empty slots and the new ranges, a cell per lane
                if (warp == HW && cb + lane < ce) {
                    const uint2 co = h.co[cb + lane], cn = h.co[cb + lane + 1];
                    for (uint32_t j = co.x + c_nsurv + (cn.y - co.y); j < cn.x; ++j)
                        if (j < cap) a.S1.cell[j] = HOLE;
                    new_range(a, c0 + cb + lane, co.x, cn.x - co.x);
                }
                ties = __reduce_add_sync(0xffffffffu, ties);
                if (lane == 0 && ties) atomicAdd(&w.ties[1], ties);
                __syncthreads();
                if (w.ties[1]) ties_in_cells<DIM, Real>(a, w, hb, c0, cb, ce);
                // partial sums, a warp per cell; every place below a cell's count has its entry in perm
                for (uint32_t lc = cb + warp; lc < ce; lc += WARPS) {
                    const uint32_t c = c0 + lc, ub = h.co[lc + 1].x - h.co[lc].x, nseed = h.co[lc + 1].y - h.co[lc].y;
                    const uint16_t* perm = w.perm + (h.co[lc].x - ob);
                    const uint32_t ns = __shfl_sync(0xffffffffu, c_ns, (int)(lc - cb));
                    uint32_t fin = __shfl_sync(0xffffffffu, c_nsurv, (int)(lc - cb)) + nseed;
                    fin = fin < ub ? fin : ub;
                    if constexpr (HX) {
                        auto* tr = reinterpret_cast<typename WtTile<DIM, Real>::Row64*>(&w)[warp];
                        double acc = 0.0;
                        for (uint32_t r0 = 0; r0 < fin; r0 += 32) {
                            const uint32_t e = perm[r0 + lane < fin ? r0 + lane : r0];
                            double xs[DIM], vs[DIM];
#pragma unroll
                            for (int d = 0; d < DIM; ++d) {
                                xs[d] = w.xi[d][e];
                                vs[d] = w.v[d][e];
                            }
                            partial_rows64<DIM>(tr, fin - r0 < 32u ? fin - r0 : 32u, xs, vs, lane, acc);
                        }
                        if (lane < Dims<DIM>::PW)
                            reinterpret_cast<double*>(a.partials)[(size_t)c * Dims<DIM>::PW + lane] = acc;
                    } else {
                        PartialAcc<Real> acc;
                        const uint32_t L = h.cs[lc + 1] - h.cs[lc], na = h.na[lc];
                        // no new particles, none removed by its counts alone (the cell's count exceeds its
                        // occupied parts by at most max) and one round: rows are the old slots, then the
                        // arrivals, with the leavers' rows empty
                        bool simple = LIGHT ? ((rows >> (lc - cb)) & 1u) != 0u : nseed == 0 && L + na <= 32u;
                        if (!LIGHT && simple && apply) {
                            uint32_t occ = 0;
                            for (int q = 0; q < occw; ++q) occ += __popcll(h.occ[lc * occw + q]);
                            simple = maxpp >= 0 && ub <= occ + (uint32_t)maxpp;
                        }
                        if (simple) {
                            uint32_t e = 0;
                            bool act = false;
                            if ((uint32_t)lane < L) {
                                e = h.cs[lc] - SA + lane;
                                act = (w.mask[e >> 5] >> (e & 31u)) & 1u;
                            } else if ((uint32_t)lane < L + na) {
                                act = ns + lane - L < fin;
                                e = act ? perm[ns + lane - L] : 0u;
                            }
                            Real xs[DIM], vs[DIM];
#pragma unroll
                            for (int d = 0; d < DIM; ++d) {
                                xs[d] = w.xi[d][e];
                                vs[d] = w.v[d][e];
                            }
                            partial_pairs32<DIM, false>(w.tr[warp], act, xs, vs, lane, acc);
                        } else {
                            for (uint32_t r0 = 0; r0 < fin; r0 += 32) {
                                const bool act = r0 + lane < fin;
                                const uint32_t e = perm[act ? r0 + lane : r0];
                                Real xs[DIM], vs[DIM];
#pragma unroll
                                for (int d = 0; d < DIM; ++d) {
                                    xs[d] = w.xi[d][e];
                                    vs[d] = w.v[d][e];
                                }
                                __syncwarp();
                                partial_pairs32<DIM, true>(w.tr[warp], act, xs, vs, lane, acc);
                            }
                        }
                        __syncwarp();
                        store_partial<DIM, Real>(a, c, acc, lane);
                    }
                }
            }
            cb = ce;
            if (cb < ncell) __syncthreads();
        }
        // the cells' counters, for the next move
        if (warp == 0 && (uint32_t)lane < ncell) {
            const uint32_t c = c0 + lane, na = h.na[lane];
            a.ccount[c] = 0;
            if (na) a.carr[c] = 0;
            if (na > (uint32_t)ARRCAP) a.head[c] = LOST;
            for (int q = 0; q < occw; ++q) a.cocc[(size_t)c * occw + q] = 0ull;
        }
        if (warp == HW) {
            land_head(w.hdr[hb ^ 1u], tk);
            tk = __shfl_sync(0xffffffffu, tk2, 0);
        }
    }
    warp_count(&a.stats->removed, removed);
    warp_count(&a.stats->step_holes, removed);
    err = __reduce_or_sync(0xffffffffu, err);
    if (lane == 0 && err) atomicOr(&a.stats->error_flags, err);
    // the last block to finish finalises the step (no waiting: the others
    // have published their counters before counting themselves done)
    __syncthreads();
    if (tid == 0) {
        __threadfence();
        if (atomicAdd(&a.stats->write_done, 1u) == gridDim.x - 1) {
            __threadfence();
            finalize_step(a);
            a.stats->write_done = 0;
            a.stats->write_next = 0;
        }
    }
}

}  // namespace pfem2
