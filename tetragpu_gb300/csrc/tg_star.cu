// tg_star.cu -- the per-vertex "star" pass of the relation pipeline and the
// per-edge and per-cell passes that follow it.
//
// The star of a vertex v is its VT row: the cells around v, ascending.  Every
// cell that holds an edge or a face at v is in it, so within the star
//   * the first position holding a neighbour u is the first occurrence of
//     edge (v,u) in the reference's cell-order scan, and
//   * the first position holding both x and y is the first occurrence of
//     face (v,x,y),
// which is what the reference CPU ids are ranks of (src/cpu_extraction.cpp:
// 28-62 edges, 122-174 faces).
//
// An edge and a face belong to their lowest vertex: only that vertex's star
// looks at them, so every edge and every face is found once.
//
//   k_star, k_star_wide
//                   a warp per vertex, a lane per star cell: the vertex's own
//                   edges (each with the mask of star positions holding it)
//                   and faces; first-occurrence bitmaps, a record per edge, a
//                   face's second cell at its first occurrence
//   k_cell_faces    a thread per cell: TF, FT and FV of the faces first met in
//                   it (the face ids are ranks in the bitmap)
//   k_edge_ids      a thread per edge record: its id, its entries in its ends'
//                   incident rows, its row lengths
//   k_edge_offsets  EV and the ET / EF / EE offsets: three sums over the
//                   lengths in id order (one pass with a look-back scan)
//   k_inc_sort      VV rows and incident-edge rows sorted
//   k_edge_rows     a lane per cell of an edge: TE, the ET and EF rows
#include <climits>
#include <type_traits>

#include "tg_internal.h"
#include "tg_rowsort.h"

namespace tg {
namespace {

constexpr unsigned kAll = 0xffffffffu;
constexpr int kNarrowStar = 31;   // the most cells a star may have for one lane a cell

__device__ __forceinline__ int get4(const int4 &w, int i)
{
    return i == 0 ? w.x : (i == 1 ? w.y : (i == 2 ? w.z : w.w));
}
__device__ __forceinline__ int pair_slot(int s, int t)  // s < t, reference TE order
{
    return s == 0 ? t - 1 : (s == 1 ? t + 1 : 5);
}
// id of occurrence p: the set bits of the first-occurrence bitmap below p
__device__ __forceinline__ int rank_of(const uint2 *__restrict__ rk, long long p)
{
    const uint2 w = __ldg(rk + (p >> 5));
    return (int)w.y + __popc(w.x & ((1u << (p & 31)) - 1u));
}
__device__ __forceinline__ int mctz(unsigned m) { return __ffs((int)m) - 1; }
__device__ __forceinline__ int mctz(unsigned long long m) { return __ffsll((long long)m) - 1; }

// ---------------------------------------------------------------------------
// k_star.  Lane l of a vertex's warp holds star cell l (and l + 32 in a star
// of 32 to 64 cells) and, of that cell's vertices, those above v: the
// candidates.  The warp takes its smallest candidate u (one warp reduction);
// a ballot of the lanes whose cell holds u is the edge's mask, and its lowest
// bit the lane of the first occurrence.  A cell's vertices are sorted, so a
// lane only ever compares its first remaining candidate, and one that has been
// taken leaves the front as the next ones move up.  A vertex costs one such
// round of a dozen instructions per edge it owns (seven on average in a grid)
// and nothing
// is shared between warps but the record buffer; the block-wide hash of
// (vertex, neighbour) pairs this replaces spent 600 warp instructions a vertex
// on table inserts, work lists and barriers, and a second pass over it 840
// more, doing every edge from both of its ends.
//
// The edges of a warp's vertices gather in its own part of shared memory, and
// go out with a lane each once the warp is through (or has no room for
// another vertex): first-occurrence flags, places in the high ends' incident
// rows, records.  No warp waits for another.
//
// Bound by the integer pipe (118 of its instructions a vertex; 166 with three
// candidates compared each round and each face's cells counted in full): 700 ->
// 668 us at 128^3 cubes (DRAM: 1.6 GB), 306 -> 252 at 96^3, 118 -> 95 on the
// 64^3 coned mesh.
constexpr int kStarThreads = TG_STAR_THREADS;
constexpr int kStarPer = TG_STAR_PER;     // most vertices per warp, in sequence
constexpr int kRecCap = TG_STAR_WIN;      // edges a warp keeps
constexpr int kStarWarps = kStarThreads / 32;
constexpr int64_t kStarFill = 152 * 48;   // warps that fill the GPU once
static_assert(kStarPer <= 32, "a warp fetches its vertices' rows a lane each");
static_assert(kRecCap >= 3 * kMaxStar, "any one vertex's edges must fit");

// H: cells per lane (2: stars of more than kNarrowStar cells)
template <int H>
struct RecBuf {
    uint2 e[kStarWarps][kRecCap];   // mask (low), high end
    uint32_t hi[H == 2 ? kStarWarps : 1][H == 2 ? kRecCap : 1];
};

__device__ __forceinline__ int4 load_cell(const int4 *__restrict__ tvs, int c)
{
    return c >= 0 ? __ldg(tvs + c) : make_int4(-1, -1, -1, -1);
}
// the slots of v < u in w, which holds both
__device__ __forceinline__ void slots_of(const int4 &w, int v, int u, int &s, int &t)
{
    s = (w.x < v) + (w.y < v);
    t = 1 + (w.y < u) + (w.z < u);
}

// the warp's n edges out; lane k holds its k-th vertex and where that vertex's
// edges start among them (ascending; a vertex that comes later: past them all)
template <int H>
__device__ __forceinline__ void put_edges(const StarPass &p, const RecBuf<H> &S, int n, int lv, int lrs,
                                          int start)
{
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    __syncwarp();
    unsigned base = 0u;
    if (lane == 0) base = atomicAdd(p.n_rec, (unsigned)n);
    base = __shfl_sync(kAll, base, 0);
    for (int i0 = 0; i0 < n; i0 += 32) {
        const int i = i0 + lane;
        int k = 0;   // the last vertex that starts at or before i
#pragma unroll
        for (int step = 16; step > 0; step >>= 1)
            k += __shfl_sync(kAll, start, k + step) <= i ? step : 0;
        const int v = __shfl_sync(kAll, lv, k), rs = __shfl_sync(kAll, lrs, k);
        const unsigned place = (unsigned)(i - __shfl_sync(kAll, start, k));
        if (i >= n) break;
        const uint2 e = S.e[wp][i];
        unsigned hi = 0u;
        if constexpr (H == 2) hi = S.hi[wp][i];
        const unsigned in = (unsigned)atomicAdd(p.deg_in + e.y, 1);
        // the first occurrence: the lowest position's cell
        const int pos = e.x ? __ffs((int)e.x) - 1 : 31 + __ffs((int)hi);
        const int c = __ldg(p.vt + rs + pos);
        int sv, su;
        slots_of(__ldg(p.tvs + c), v, (int)e.y, sv, su);
        const unsigned slot = (unsigned)(6 * c + pair_slot(sv, su));
        atomicOr(p.eflag + (slot >> 5), 1u << (slot & 31));
        // (records without room are written over the last: a branch here costs 15 %)
        const unsigned g = min(base + (unsigned)i, p.rec_last);
        p.rec[g] = make_uint2(slot, e.x);
        p.place[g] = make_uint2(place, in);
        if constexpr (H == 2) p.rec_hi[g] = hi;
    }
    __syncwarp();
}

// the highest set bit (-1: none; shuffles take their lane modulo 32)
__device__ __forceinline__ int last_bit(unsigned m)
{
    int b;
    asm("bfind.u32 %0, %1;" : "=r"(b) : "r"(m));
    return b;
}
__device__ __forceinline__ int last_bit(unsigned long long m)
{
    int b;
    asm("bfind.u64 %0, %1;" : "=r"(b) : "l"(m));
    return b;
}

// predicated accesses: as branches the compiler splits and rejoins the warp
// around each of them
__device__ __forceinline__ void store_if(bool yes, int *at, int x)
{
    asm volatile("{ .reg .pred q; setp.ne.s32 q, %0, 0; @q st.global.s32 [%1], %2; }" ::"r"((int)yes),
                 "l"(at), "r"(x)
                 : "memory");
}
__device__ __forceinline__ void or_if(bool yes, uint32_t *at, unsigned x)
{
    asm volatile("{ .reg .pred q; setp.ne.s32 q, %0, 0; @q red.global.or.b32 [%1], %2; }" ::"r"((int)yes),
                 "l"(at), "r"(x)
                 : "memory");
}
// the same words by the whole warp
__device__ __forceinline__ void store_shared(unsigned at, const uint2 &x)
{
    asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(at), "r"(x.x), "r"(x.y) : "memory");
}

// One vertex; H: cells per lane.  n: edges the warp holds, with room for any
// vertex of such a star.  F: the faces' second cells are wanted (fnext).
template <int H, bool F>
__device__ __forceinline__ void star_vertex(const StarPass &p, RecBuf<H> &S, int v,
                                            const int (&c)[H], const int4 (&w)[H], int &n)
{
    using M = typename std::conditional<H == 1, unsigned, unsigned long long>::type;
    // d: a cell's vertices above v, ascending (the slots after v's), looked at
    // from the first on; one that has been looked at leaves for the end as its
    // mask, marked by the top bit (a vertex is below 2^31, and so is a narrow
    // star's mask: at most kNarrowStar cells); with two cells a lane the marks
    // and the masks are apart.  In the end they stand for slots 1 to 3 (slot 0
    // is never above another vertex of its cell), empty where not above v
    constexpr unsigned kDone = 0x80000000u;
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    unsigned d[H][3];
    M m[H][3];
#pragma unroll
    for (int h = 0; h < H; h++) {
        const bool above1 = w[h].y > v, above2 = w[h].z > v, above3 = w[h].w > v;
        d[h][0] = above1 ? (unsigned)w[h].y : (above2 ? (unsigned)w[h].z : (above3 ? (unsigned)w[h].w : kDone));
        d[h][1] = above1 ? (unsigned)w[h].z : (above2 ? (unsigned)w[h].w : kDone);
        d[h][2] = above1 ? (unsigned)w[h].w : kDone;
        m[h][0] = m[h][1] = m[h][2] = 0;
    }
    const unsigned out0 = (unsigned)__cvta_generic_to_shared(S.e[wp] + n);
    unsigned out = out0;
    while (true) {
        unsigned cn = d[0][0];
        if constexpr (H == 2) cn = min(cn, d[1][0]);
        const unsigned u = __reduce_min_sync(kAll, cn);
        if (u >= kDone) break;
        M mu = 0;
        bool hit[H];
#pragma unroll
        for (int h = 0; h < H; h++) {
            hit[h] = d[h][0] == u;
            mu |= (M)__ballot_sync(kAll, hit[h]) << (32 * h);
        }
#pragma unroll
        for (int h = 0; h < H; h++) {
            d[h][0] = hit[h] ? d[h][1] : d[h][0];
            d[h][1] = hit[h] ? d[h][2] : d[h][1];
            d[h][2] = hit[h] ? (H == 1 ? (unsigned)mu | kDone : kDone) : d[h][2];
            if constexpr (H == 2) {
                m[h][0] = hit[h] ? m[h][1] : m[h][0];
                m[h][1] = hit[h] ? m[h][2] : m[h][1];
                m[h][2] = hit[h] ? mu : m[h][2];
            }
        }
        store_shared(out, make_uint2((unsigned)mu, u));
        if constexpr (H == 2) S.hi[wp][n + (int)((out - out0) / sizeof(uint2))] = (unsigned)(mu >> 32);
        out += sizeof(uint2);
    }
    const int own = (int)((out - out0) / sizeof(uint2));
    store_if(lane == 0, p.deg_own + v, own);
    n += own;

    // faces whose lowest vertex is v: two of the candidates, the third left
    // out (v in slot 0: slot 1, 2 or 3; v in slot 1: slot 0; the masks of
    // slots at or below v's are zero)
#pragma unroll
    for (int h = 0; h < H; h++) {
        if constexpr (H == 1) {
#pragma unroll
            for (int k = 0; k < 3; k++) m[0][k] = d[0][k] & ~kDone;
        }
        // this lane's position, and those up to it
        const M bit = (M)1 << (lane + 32 * h), upto = bit | (bit - 1);
        const int sh = 4 * (c[h] & 7);
        // the column of the face omitting slot o is 3 - o
        const int col0 = w[h].x == v ? 2 : 3;
        auto face = [&](int k) {
            return k == 0 ? m[h][1] & m[h][2] : (k == 1 ? m[h][0] & m[h][2] : m[h][0] & m[h][1]);
        };
        auto cells = [](M f) { return sizeof(M) == 8 ? __popcll((unsigned long long)f) : __popc((unsigned)f); };
        unsigned firsts = 0u;
        bool odd = false;   // a face of other than two cells is first met here
        int *next = F ? p.fnext + 4LL * c[h] : nullptr;
        int *next0 = F ? next + col0 : nullptr;
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const M f = face(k);
            const bool is_first = (f & upto) == bit;
            firsts |= is_first ? (k == 0 ? 1u << col0 : 1u << (2 - k)) : 0u;
            odd = odd || (is_first && cells(f) != 2);
            if constexpr (F) {
                const int s2 = last_bit(f);
                int c2 = __shfl_sync(kAll, c[0], s2);
                if constexpr (H == 2) {
                    const int c2b = __shfl_sync(kAll, c[1], s2);
                    c2 = s2 >= 32 ? c2b : c2;
                }
                store_if(is_first, k == 0 ? next0 : next + (2 - k), c2);
            }
        }
        or_if(firsts != 0u, p.fflag + (c[h] >> 3), firsts << sh);
        if (__any_sync(kAll, odd) && odd) {   // boundary faces, faces of too many cells
#pragma unroll
            for (int k = 0; k < 3; k++) {
                const M f = face(k);
                if ((f & upto) != bit) continue;
                if (cells(f) == 1) {
                    const int col = k == 0 ? col0 : 2 - k;
                    if (F) next[col] = -1;
                    atomicOr(p.fbnd + (c[h] >> 3), 1u << (sh + col));
                    p.vbnd[col == 3 ? w[h].y : w[h].x] = 1;
                    p.vbnd[col >= 2 ? w[h].z : w[h].y] = 1;
                    p.vbnd[col >= 1 ? w[h].w : w[h].z] = 1;
                } else if (cells(f) > 2) {   // reported by the face's first cell
                    atomicOr(&p.st->flags, ST_NONMANIFOLD_FACE);
                    note_lowest(&p.st->bad_cell, c[h]);
                }
            }
        }
    }
}

// Stars of one or two cells (D; 0: none), a lane each: every edge and face by
// itself, compared with the other cell.  All 32 lanes call it.
__device__ __forceinline__ bool holds(const int4 &w, int x)
{
    return w.x == x || w.y == x || w.z == x || w.w == x;
}
constexpr int kFewCells = 2;
constexpr int kFewLanes = 4;   // in a warp from which on this is less work than a round each
template <bool F>
__device__ __forceinline__ void few_cells(const StarPass &p, int v, int rs, int D)
{
    const int lane = threadIdx.x & 31;
    int c[2];
    int4 w[2];
#pragma unroll
    for (int q = 0; q < 2; q++) {
        c[q] = q < D ? __ldg(p.vt + rs + q) : -1;
        w[q] = load_cell(p.tvs, c[q]);
    }
    unsigned first = 0u;   // bit 4 q + t: the edge to slot t of cell q, first met there
#pragma unroll
    for (int q = 0; q < 2; q++)
#pragma unroll
        for (int t = 0; t < 4; t++) {
            const int u = get4(w[q], t);
            if (q < D && u > v && !(q == 1 && holds(w[0], u))) first |= 1u << (4 * q + t);
        }
    const int own = __popc(first);
    int end = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(kAll, end, o);
        if (lane >= o) end += y;
    }
    unsigned base = 0u;
    if (lane == 31) base = atomicAdd(p.n_rec, (unsigned)end);
    const unsigned g0 = __shfl_sync(kAll, base, 31) + (unsigned)(end - own);
    if (D == 0) return;
    p.deg_own[v] = own;
    unsigned place = 0u;
#pragma unroll
    for (int q = 0; q < 2; q++) {
        const int sv = (w[q].x < v) + (w[q].y < v) + (w[q].z < v);
#pragma unroll
        for (int t = 1; t < 4; t++) {   // (slot 0 is never above another vertex of its cell)
            if (!(first >> (4 * q + t) & 1u)) continue;
            const int u = get4(w[q], t);
            const unsigned in = (unsigned)atomicAdd(p.deg_in + u, 1);
            const unsigned slot = (unsigned)(6 * c[q] + pair_slot(sv, t));
            atomicOr(p.eflag + (slot >> 5), 1u << (slot & 31));
            const unsigned g = min(g0 + place, p.rec_last);
            p.rec[g] = make_uint2(slot, q == 1 ? 2u : (D == 2 && holds(w[1], u) ? 3u : 1u));
            p.place[g] = make_uint2(place, in);
            place++;
        }
        if (q >= D || sv > 1) continue;
        // faces whose lowest vertex is v: v in slot 0 (all but the one that omits
        // it) or in slot 1 (the one that omits slot 0)
        unsigned firsts = 0u, alone = 0u;
#pragma unroll
        for (int o = 0; o < 4; o++) {
            if ((sv == 0) == (o == 0)) continue;
            const int x = o == 0 || o == 1 ? w[q].z : w[q].y, y = o == 3 ? w[q].z : w[q].w;
            const bool both = D == 2 && holds(w[1 - q], x) && holds(w[1 - q], y);
            if (q == 1 && both) continue;   // first met in the other cell
            firsts |= 8u >> o;
            if (!both) alone |= 8u >> o;
            if (F) p.fnext[4LL * c[q] + 3 - o] = both ? c[1 - q] : -1;
            if (!both) {
                p.vbnd[v] = 1;
                p.vbnd[x] = 1;
                p.vbnd[y] = 1;
            }
        }
        const int sh = 4 * (c[q] & 7);
        atomicOr(p.fflag + (c[q] >> 3), firsts << sh);
        if (alone) atomicOr(p.fbnd + (c[q] >> 3), alone << sh);
    }
}

// The light vertices of at most kNarrowStar cells; the others go on a list
// (about in processing order) that k_star_wide takes.  Stars of one or two cells
// go lane by lane where a warp has several: on 1.5M cells that share nothing a
// warp's round for each takes 1,100 us, this 530.
template <bool F>
__global__ void __launch_bounds__(kStarThreads, TG_STAR_MINB) k_star(StarPass p, int per)
{
    griddep_wait();
    __shared__ RecBuf<1> S;
    const int lane = threadIdx.x & 31;
    const int64_t pos = ((int64_t)blockIdx.x * kStarWarps + (threadIdx.x >> 5)) * per;
    // lane k < per: the warp's k-th vertex, its row's start and length
    int lv = -1, lrs = 0, lD = 0;
    if (lane < per && pos + lane < p.n_light) {
        lv = p.vorder[pos + lane];
        lrs = (int)p.vt_off[lv];
        lD = (int)(p.vt_off[lv + 1] - lrs);
        if (lD > kNarrowStar) p.wide[atomicAdd(p.n_wide, 1u)] = lv;
    }
    const bool few = lD > 0 && lD <= kFewCells;
    if (__popc(__ballot_sync(kAll, few)) >= kFewLanes) {
        few_cells<F>(p, lv, lrs, few ? lD : 0);
        if (few) lD = 0;
        if (!__any_sync(kAll, lD > 0)) return;
    }
    auto load_entry = [&](int k) {   // this lane's cell of the k-th vertex (the first 32)
        const int rs = __shfl_sync(kAll, lrs, k & 31), D = __shfl_sync(kAll, lD, k & 31);
        return lane < D ? __ldg(p.vt + rs + lane) : -1;
    };
    // the next vertex's cells and the one after's row are in flight while a
    // vertex is worked on (past the warp's last vertex the rows are empty but
    // for a wrap to its first, which is not looked at)
    int c0 = load_entry(0), c1 = load_entry(1);
    int4 w0 = load_cell(p.tvs, c0);
    int n = 0, start = INT_MAX;
#pragma unroll 1
    for (int k = 0; k < per; k++) {
        const int v = __shfl_sync(kAll, lv, k);
        if (v < 0) break;
        const int4 w1 = load_cell(p.tvs, c1);
        const int c2 = load_entry(k + 2);
        const int D = __shfl_sync(kAll, lD, k);
        if (D > 0 && D <= kNarrowStar) {
            if (n > kRecCap - 3 * kNarrowStar) {   // out with the edges of the vertices before this
                put_edges<1>(p, S, n, lv, lrs, start);
                n = 0;
                if (lane < k) start = -1;
            }
            if (lane == k) start = n;
            const int c[1] = {c0};
            const int4 w[1] = {w0};
            star_vertex<1, F>(p, S, v, c, w, n);
        } else if (lane == k) {
            start = n;   // no edges here (a wide star, or done)
        }
        c0 = c1;
        w0 = w1;
        c1 = c2;
    }
    if (n) put_edges<1>(p, S, n, lv, lrs, start);
}

// a vertex of kNarrowStar + 1 to kMaxStar cells per warp
template <bool F>
__global__ void __launch_bounds__(kStarThreads) k_star_wide(StarPass p)
{
    griddep_wait();
    __shared__ RecBuf<2> S;
    const int lane = threadIdx.x & 31;
    const unsigned i = blockIdx.x * kStarWarps + (threadIdx.x >> 5);
    if (i >= *p.n_wide) return;
    const int v = p.wide[i];
    const int rs = (int)p.vt_off[v], D = (int)(p.vt_off[v + 1] - rs);
    const int c[2] = {lane < D ? __ldg(p.vt + rs + lane) : -1,
                      lane + 32 < D ? __ldg(p.vt + rs + lane + 32) : -1};
    const int4 w[2] = {load_cell(p.tvs, c[0]), load_cell(p.tvs, c[1])};
    int n = 0;
    star_vertex<2, F>(p, S, v, c, w, n);
    if (n) put_edges<2>(p, S, n, v, rs, lane == 0 ? 0 : INT_MAX);
}

// ---------------------------------------------------------------------------
// k_cell_faces.  The faces first met in cell c take the ids from c's rank on,
// in column order: TF here and in the face's second cell, FT, FV.  A block's
// faces have consecutive ids: their FT and FV rows pass through shared memory
// and go out as whole lines.
constexpr int kCellThreads = 256;
__global__ void __launch_bounds__(kCellThreads, 6)
k_cell_faces(int64_t T, const int4 *__restrict__ tvs, const uint2 *__restrict__ frank,
             const int4 *__restrict__ fnext, int *__restrict__ tf, int2 *__restrict__ ft,
             int *__restrict__ fv)
{
    griddep_wait();
    __shared__ int2 s_ft[4 * kCellThreads];
    __shared__ int s_fv[12 * kCellThreads];
    const int64_t c0 = (int64_t)blockIdx.x * kCellThreads;   // a multiple of 8: a word's first cell
    const int64_t c = c0 + threadIdx.x;
    const int64_t f0 = (int64_t)__ldg(frank + (c0 >> 3)).y;
    // the closing word counts every face: T is past the last word's first cell
    // or on its boundary
    const int64_t c1 = min(c0 + kCellThreads, T);
    const uint2 r1 = __ldg(frank + (c1 >> 3));
    const int nf = (int)((int64_t)r1.y + __popc(r1.x & ((1u << (4 * (int)(c1 & 7))) - 1u)) - f0);
    unsigned first = 0u;
    if (c < T) {
        const uint2 rk = __ldg(frank + (c >> 3));
        const int sh = 4 * (int)(c & 7);
        first = (rk.x >> sh) & 15u;
        if (first) {
            int fid = (int)rk.y + __popc(rk.x & ((1u << sh) - 1u));
            const int4 w = __ldg(tvs + c);
            const int4 nx = fnext ? __ldg(fnext + c) : make_int4(-1, -1, -1, -1);
            int4 w2[4];
            if (tf) {
#pragma unroll
                for (int col = 0; col < 4; col++) {
                    const int c2 = get4(nx, col);
                    if (((first >> col) & 1u) && c2 >= 0) w2[col] = __ldg(tvs + c2);
                }
            }
#pragma unroll
            for (int col = 0; col < 4; col++) {
                if (!((first >> col) & 1u)) continue;
                // the face's vertices: all but slot 3 - col
                const int a = col == 3 ? w.y : w.x, b = col >= 2 ? w.z : w.y;
                const int d = col >= 1 ? w.w : w.z;
                const int c2 = get4(nx, col);
                const int k = fid - (int)f0;
                if (ft) s_ft[k] = make_int2((int)c, c2);
                if (fv) {
                    s_fv[3 * k] = a;
                    s_fv[3 * k + 1] = b;
                    s_fv[3 * k + 2] = d;
                }
                if (tf) {
                    tf[4 * c + col] = fid;
                    if (c2 >= 0) {
                        // sorted rows: the first slot that differs from (a, b, d)
                        // is the one the face leaves out
                        const int4 x = w2[col];
                        const int o2 = x.x != a ? 0 : (x.y != b ? 1 : (x.z != d ? 2 : 3));
                        tf[4LL * c2 + 3 - o2] = fid;
                    }
                }
                fid++;
            }
        }
    }
    if (!ft && !fv) return;
    __syncthreads();
    if (ft)
        for (int i = threadIdx.x; i < nf; i += kCellThreads) ft[f0 + i] = s_ft[i];
    if (fv)
        for (int i = threadIdx.x; i < 3 * nf; i += kCellThreads) fv[3 * f0 + i] = s_fv[i];
}

// ---------------------------------------------------------------------------
struct EdgeEnds {
    int c, j, v, u;   // first cell, pair slot there, low and high end
};
__device__ __forceinline__ EdgeEnds edge_ends(const int4 *__restrict__ tvs, unsigned slot)
{
    EdgeEnds e;
    e.c = (int)(slot / 6u);
    e.j = (int)(slot - 6u * (unsigned)e.c);
    const int4 w = __ldg(tvs + e.c);
    e.v = e.j < 3 ? w.x : (e.j < 5 ? w.y : w.z);
    e.u = e.j == 0 ? w.y : (e.j == 1 || e.j == 3 ? w.z : w.w);
    return e;
}
// The cells of an edge record: the star positions of its owner v that its
// mask holds, ascending.  W: masks of stars of more than kNarrowStar cells
// have a high half in rec_hi; a star of more than 64 cells (tg_heavy.cu) keeps
// its (neighbour, position) pairs instead: the mask is the run's first pair
// and rec_hi its length.
//
// k_edge_ids, a thread per record: the edge's id (the rank of its first
// occurrence), its entries in its ends' incident rows (unsorted: a row fills
// from the front for the edges the vertex is the high end of, from the back
// for its own), its row lengths; the record moves to its id's place, so that
// the passes after this one write in id order.  Each cell of the edge holds
// two of its faces and each face lies in two of its cells but for the boundary
// faces, in one: faces = cells + boundary faces / 2.  A boundary face of the
// edge makes both ends boundary vertices; only such edges look at their cells
// (a boundary face is its only cell's first occurrence, so fbnd tells).
template <bool W>
__global__ void __launch_bounds__(256) k_edge_ids(EdgePass p)
{
    griddep_wait();
    const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= p.E) return;
    const uint2 rec = __ldg(p.rec + r);
    const uint2 place = __ldg(p.place + r);
    const EdgeEnds e = edge_ends(p.tvs, rec.x);
    const int64_t ru = __ldg(p.vv_off + e.u), rv1 = __ldg(p.vv_off + e.v + 1);
    int id = 0;
    if (p.erank) id = rank_of(p.erank, rec.x);
    if (p.inc) {
        p.inc[rv1 - 1 - place.x] = make_int2(e.u, id);
        p.inc[ru + place.y] = make_int2(e.v, id);
    } else {
        p.vv[rv1 - 1 - place.x] = e.u;
        p.vv[ru + place.y] = e.v;
    }
    if (!p.edge) return;
    const bool walk = p.count_ef && __ldg(p.vbnd + e.v) && __ldg(p.vbnd + e.u);
    const int64_t rs = W || walk ? __ldg(p.vt_off + e.v) : 0;
    const int D = W ? (int)(__ldg(p.vt_off + e.v + 1) - rs) : 0;
    const unsigned hi = W && D > kNarrowStar ? __ldg(p.rec_hi + r) : 0u;
    int nb = 0, n_et;
    auto look = [&](int pos) {
        const int c = __ldg(p.vt + rs + pos);
        int s, t;
        slots_of(__ldg(p.tvs + c), e.v, e.u, s, t);
        // its faces there leave out one of the other two slots
        const unsigned out = 0xfu & ~((8u >> s) | (8u >> t));
        nb += __popc((__ldg(p.fbnd + (c >> 3)) >> (4 * (c & 7))) & out);
    };
    if (W && D > kMaxStar) {
        n_et = (int)hi;
        if (walk)
            for (int k = 0; k < n_et; k++) look(p.pairs[(int64_t)rec.y + k].y);
    } else {
        unsigned long long m = rec.y;
        if (W) m |= (unsigned long long)hi << 32;
        n_et = W ? __popcll(m) : __popc(rec.y);
        if (walk)
            for (; m; m &= m - 1) look(mctz(m));
    }
    const unsigned ee = (unsigned)((rv1 - __ldg(p.vv_off + e.v)) +
                                   (__ldg(p.vv_off + e.u + 1) - ru) - 2);
    p.edge[id] = make_uint4(rec.x, rec.y, (unsigned)n_et | (unsigned)(n_et + nb / 2) << 16, ee);
    if (W && D > kNarrowStar) p.edge_hi[id] = hi;
}

// k_edge_rows: TE at each cell of an edge, ET and EF rows, and EV when nothing
// before it needs it (without ET, EF or EE k_edge_offsets has nothing else to
// do: 60 us at 96^3 cubes).  A warp takes 32 consecutive edges and spreads their
// cells over its lanes (a list in shared memory, two bytes a cell: 180 -> 168 us
// for TE and EV at 96^3 against a word and a byte), so that the cells gathered
// and the entries written by one instruction belong to a few neighbouring
// edges and share cache lines: what bounds the pass is the number of lines its
// instructions touch (about 0.8 a clock and SM get through to L2).  A thread per
// edge touched 20 lines an edge; records in the star pass's order 13, their ET
// and EF rows lying apart.
//
// EF: an edge's faces at a cell are the columns omitting one of the other two
// slots.  A face's cells all hold the edge, so a row is the faces at the cells
// where they are first met, ascending: ids are ranks of first occurrences (4 *
// cell + column), so one word pair of frank gives both which faces these are
// and their ids (78 us at 64^3 cubes; with TF read for the ids, 91).
constexpr int kRowsThreads = 128;
constexpr int kRowsTake = 16;                // cells an edge lists at a time
constexpr int kRowsCap = 32 * kRowsTake;
// EF: whether EF rows are wanted
template <bool W, bool EF>
__global__ void __launch_bounds__(kRowsThreads) k_edge_rows(EdgePass p)
{
    griddep_wait();
    // a cell of an edge: its position in the low end's star << 5 | the edge's lane
    __shared__ unsigned short s_list[kRowsThreads / 32][kRowsCap];
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const int64_t id = (int64_t)blockIdx.x * kRowsThreads + threadIdx.x;
    if ((id & ~(int64_t)31) >= p.E) return;   // warp-uniform
    int v = 0, u = 0, rs = 0, et = 0, ef = 0;
    // EF has up to 12T entries, past 2^31: the warp's rows from an int64 start,
    // a lane's within them (below 32 * 2^16)
    const int64_t ef0 = EF ? __ldg(p.ef_off + (id & ~(int64_t)31)) : 0;
    int *const ef_out = p.ef + ef0;
    unsigned long long m = 0ull;
    if (id < p.E) {
        const uint2 rec = __ldg(reinterpret_cast<const uint2 *>(p.edge + id));
        const EdgeEnds e = edge_ends(p.tvs, rec.x);
        v = e.v;
        u = e.u;
        if (p.ev) reinterpret_cast<int2 *>(p.ev)[id] = make_int2(v, u);
        rs = (int)__ldg(p.vt_off + v);
        if (p.et) et = (int)__ldg(p.et_off + id);
        if constexpr (EF) ef = (int)(__ldg(p.ef_off + id) - ef0);
        m = rec.y;
        if constexpr (W) {
            const int D = (int)(__ldg(p.vt_off + v + 1) - rs);
            if (D > kMaxStar) {   // alone, cell after cell
                const int n = (int)p.edge_hi[id];
                int k_ef = ef;
                for (int k = 0; k < n; k++) {
                    const int c = __ldg(p.vt + rs + p.pairs[(int64_t)rec.y + k].y);
                    int s, t;
                    slots_of(__ldg(p.tvs + c), v, u, s, t);
                    if (p.te) p.te[6LL * c + pair_slot(s, t)] = (int)id;
                    if (p.et) p.et[et + k] = c;
                    if constexpr (EF) {
                        const uint2 rk = __ldg(p.frank + (c >> 3));
                        const int sh = 4 * (c & 7);
                        const unsigned out = (rk.x >> sh) & 0xfu & ~((8u >> s) | (8u >> t));
                        for (unsigned o = out; o; o &= o - 1)
                            ef_out[k_ef++] = (int)rk.y + __popc(rk.x & ((1u << (sh + mctz(o))) - 1u));
                    }
                }
                m = 0ull;
            } else if (D > kNarrowStar) {
                m |= (unsigned long long)p.edge_hi[id] << 32;
            }
        }
    }
    unsigned short *list = s_list[wp];
    while (__any_sync(kAll, m != 0ull)) {
        // this lane's cells (at most kRowsTake now) in the list
        const int cnt = min(W ? __popcll(m) : __popc((unsigned)m), kRowsTake);
        int end = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(kAll, end, o);
            if (lane >= o) end += y;
        }
        const int off = end - cnt, total = __shfl_sync(kAll, end, 31);
        if constexpr (W) {
            for (int k = off; k < end; k++, m &= m - 1) list[k] = (unsigned short)(mctz(m) << 5 | lane);
        } else {
            unsigned mm = (unsigned)m;
            for (int k = off; k < end; k++, mm &= mm - 1) list[k] = (unsigned short)(mctz(mm) << 5 | lane);
            m = mm;
        }
        __syncwarp();
        const int etb = et - off;   // entry i of the list goes to etb + i
        for (int i0 = 0; i0 < total; i0 += 32) {
            const int i = i0 + lane;
            const bool act = i < total;
            const unsigned item = act ? list[i] : 0u;
            const int l = (int)(item & 31u);
            const int xs = __shfl_sync(kAll, rs, l);
            const int c = act ? __ldg(p.vt + xs + (item >> 5)) : 0;
            const int xv = __shfl_sync(kAll, v, l), xu = __shfl_sync(kAll, u, l);
            const int4 w = act ? __ldg(p.tvs + c) : make_int4(0, 0, 0, 0);
            int s, t;
            slots_of(w, xv, xu, s, t);
            if (p.te && act) p.te[6LL * c + pair_slot(s, t)] = (int)(id - lane) + l;
            if (p.et) {
                const int b = __shfl_sync(kAll, etb, l);
                if (act) p.et[b + i] = c;
            }
            if constexpr (EF) {
                const int t1 = s == 0 ? (t == 1 ? 2 : 1) : 0, t2 = 6 - s - t - t1;
                const uint2 rk = act ? __ldg(p.frank + (c >> 3)) : make_uint2(0u, 0u);
                // columns 3 - t2 < 3 - t1
                const int qa = 4 * (c & 7) + 3 - t2, qb = 4 * (c & 7) + 3 - t1;
                const bool first_a = (rk.x >> qa) & 1u, first_b = (rk.x >> qb) & 1u;
                const unsigned ba = __ballot_sync(kAll, first_a), bb = __ballot_sync(kAll, first_b);
                // the entries of this edge before this one in the list's window
                const int o = __shfl_sync(kAll, off, l) - i0;
                const unsigned below = ((1u << lane) - 1u) & (o > 0 ? ~0u << o : ~0u);
                int k = __shfl_sync(kAll, ef, l) + __popc(ba & below) + __popc(bb & below);
                if (first_a) ef_out[k++] = (int)rk.y + __popc(rk.x & ((1u << qa) - 1u));
                if (first_b) ef_out[k] = (int)rk.y + __popc(rk.x & ((1u << qb) - 1u));
                // this lane's own edge: past the entries written for it now
                const int lo = max(off - i0, 0), hi = min(end - i0, 32);
                if (lo < hi) {
                    const unsigned own = (hi == 32 ? ~0u : (1u << hi) - 1u) & (~0u << lo);
                    ef += __popc(ba & own) + __popc(bb & own);
                }
            }
        }
        et += cnt;
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------
// Star processing order (see k_vorder_place): vertex v with first cell c in
// slot k has key 4c + k; its bit in vflag marks it, its rank is v's position.
// A vertex whose star holds more than kMaxStar cells is heavy: it takes no
// key, but a bit among the heavy vertices (hflag), which follow every other
// vertex with cells in the processing order, by id, so that the star pass
// stops where they begin (tg_heavy.cu processes them).
__device__ __forceinline__ void mark_first(const int4 *__restrict__ tvs, uint32_t *vflag,
                                           int64_t *vkey, uint32_t *hflag, int v, int c, int D)
{
    if (D > kMaxStar) {
        vkey[v] = -1;
        atomicOr(hflag + (v >> 5), 1u << (v & 31));
        return;
    }
    const int4 w = __ldg(tvs + c);
    const long long key = 4LL * c + (w.x == v ? 0 : (w.y == v ? 1 : (w.z == v ? 2 : 3)));
    vkey[v] = key;
    atomicOr(vflag + (key >> 5), 1u << (key & 31));
}

// ---------------------------------------------------------------------------
// CSR rows sorted ascending, a row to a thread (tg_rowsort.h).  A block's
// kVtsThreads rows are contiguous: they pass through shared memory so that
// global memory sees whole rows; rows that do not fit are sorted in place.
// `first` is given each non-empty row's smallest entry.  Bound by its memory
// accesses; ranking every entry against its row by a loop over shared memory
// instead was issue-bound: VT 362 -> 137 us at 128^3 (12.6M cells), 70 -> 22
// us on the 64^3 coned mesh.
constexpr int kVtsThreads = TG_VTS_THREADS;
constexpr int kVtsCap = 32 * kVtsThreads;
struct RowStage {
    int4 word[kVtsCap / 4 + 1];
};
// total: entries of the whole array
template <typename Fn>
__device__ __forceinline__ void sort_block_rows(RowStage &S, const int64_t *__restrict__ off, int64_t rows,
                                                int64_t total, int *__restrict__ ent, Fn first)
{
    int *stage = reinterpret_cast<int *>(S.word);
    const int64_t v0 = (int64_t)blockIdx.x * kVtsThreads;
    const int64_t v1 = min(v0 + kVtsThreads, rows);
    const int64_t v = v0 + threadIdx.x;
    const int64_t base = off[v0];
    const int64_t n = off[v1] - base;
    const int64_t b = v < rows ? off[v] : 0;
    const int D = v < rows ? (int)(off[v + 1] - b) : 0;
    if (n > kVtsCap) {   // block-uniform
        sort_rows_warp(ent + b, D);
        if (D > 0) first((int)v, ent[b], D);
        return;
    }
    // whole 16-byte words from the one holding the first entry
    const int shift = (int)(base & 3);
    const int words = (int)((n + shift + 3) >> 2);
    for (int i = threadIdx.x; i < words; i += kVtsThreads) {
        const int64_t g = base - shift + 4LL * i;
        if (g + 4 <= total) {
            S.word[i] = *reinterpret_cast<const int4 *>(ent + g);
        } else {
            for (int k = 0; g + k < total; k++) stage[4 * i + k] = ent[g + k];
        }
    }
    __syncthreads();
    int *row = stage + shift + (int)(b - base);
    sort_rows_warp(row, D);
    if (D > 0) first((int)v, row[0], D);
    __syncthreads();
    for (int i = threadIdx.x; i < (int)n; i += kVtsThreads) ent[base + i] = stage[shift + i];
}

__global__ void __launch_bounds__(kVtsThreads)
k_vt_sort(const int64_t *__restrict__ vt_off, int64_t V, int64_t total, int *__restrict__ vt,
          const int4 *__restrict__ tvs, uint32_t *__restrict__ vflag, int64_t *__restrict__ vkey,
          uint32_t *__restrict__ hflag, int *__restrict__ heavy_cnt)
{
    griddep_wait();
    __shared__ RowStage S;
    int wide = 0;
    sort_block_rows(S, vt_off, V, total, vt, [&](int v, int c, int D) {
        wide = D > kNarrowStar && D <= kMaxStar;
        mark_first(tvs, vflag, vkey, hflag, v, c, D);
    });
    // heavy_cnt[2]: light stars of more than kNarrowStar cells
    wide = __syncthreads_count(wide);
    if (wide && threadIdx.x == 0) atomicAdd(heavy_cnt + 2, wide);
}

// VV rows in place
__global__ void __launch_bounds__(kVtsThreads)
k_vv_sort(const int64_t *__restrict__ off, int64_t V, int64_t total, int *__restrict__ vv)
{
    griddep_wait();
    __shared__ RowStage S;
    sort_block_rows(S, off, V, total, vv, [](int, int, int) {});
}

// VV and incident-edge rows from inc (the same rows, {neighbour, edge id}
// pairs), each sorted by itself; the incident-edge rows padded with ~0 to
// eid_words at eid_off.  Nine blocks to an SM spill 32 bytes a thread: 64 us at
// 96^3 cubes, 66 with eight and no spills.
constexpr int kIncCap = 20 * kVtsThreads;
__global__ void __launch_bounds__(kVtsThreads, 9)
k_inc_sort(const int64_t *__restrict__ off, int64_t V, const int2 *__restrict__ inc,
           int *__restrict__ vv, const int64_t *__restrict__ eid_off, int *__restrict__ eid)
{
    griddep_wait();
    __shared__ int s_row[2][kIncCap];
    __shared__ int s_at[kVtsThreads], s_len[kVtsThreads];
    __shared__ long long s_out[kVtsThreads];
    const int64_t v0 = (int64_t)blockIdx.x * kVtsThreads;
    const int64_t v = v0 + threadIdx.x;
    const int64_t base = off[v0];
    const int64_t n = off[min(v0 + kVtsThreads, V)] - base;
    const int64_t b = v < V ? off[v] : 0;
    const int d = v < V ? (int)(off[v + 1] - b) : 0;
    const int64_t out = v < V ? eid_off[v] : 0;
    if (n > kIncCap) {   // block-uniform: in place
        for (int k = 0; k < d; k++) {
            const int2 x = inc[b + k];
            vv[b + k] = x.x;
            eid[out + k] = x.y;
        }
        for (int k = d; k < (v < V ? eid_words(d) : 0); k++) eid[out + k] = -1;
#pragma unroll 1
        for (int q = 0; q < 2; q++) sort_rows_warp(q ? eid + out : vv + b, d);
        return;
    }
    s_at[threadIdx.x] = (int)(b - base);
    s_len[threadIdx.x] = d;
    s_out[threadIdx.x] = out;
    for (int i = threadIdx.x; i < (int)n; i += kVtsThreads) {
        const int2 x = __ldg(inc + base + i);
        s_row[0][i] = x.x;
        s_row[1][i] = x.y;
    }
    __syncthreads();
#pragma unroll 1
    for (int q = 0; q < 2; q++) sort_rows_warp(s_row[q] + (int)(b - base), d);
    __syncthreads();
    for (int i = threadIdx.x; i < (int)n; i += kVtsThreads) vv[base + i] = s_row[0][i];
    const int rows = (int)min((int64_t)kVtsThreads, V - v0);
    for (int r = threadIdx.x >> 4; r < rows; r += kVtsThreads / 16) {
        const int at = s_at[r], len = s_len[r], words = eid_words(len);
        int *row = eid + s_out[r];
        for (int k = threadIdx.x & 15; k < words; k += 16)
            row[k] = k < len ? s_row[1][at + k] : -1;
    }
}

// ---------------------------------------------------------------------------
// ET / EF / EE offsets: exclusive sums of the row lengths in edge-id order, in
// one pass (a block takes the next tile in start order, sums it, adds the
// tiles before it by look-back, and writes its offsets).  EV of the tile's
// edges beside it, while the look-back waits.  Two neighbouring edges to a lane
// (one 32-byte record load, 16-byte stores), rows of 64 to a warp, so that a
// request carries whole lines; ET and EF lengths are summed in the halves of
// one word.  172 us at 128^3 cubes (208 with eight consecutive edges to a
// thread, whose 128 bytes were lines of their own); its 0.9 GB take 135 at the
// copy rate.  Six blocks to an SM spill 36 bytes a thread and are still ahead:
// 190 us with four.
constexpr int kEdgeThreads = 256;
constexpr int kEdgeItems = TG_EDGE_ITEMS;             // edges per thread
constexpr int kEdgeTile = kEdgeItems * kEdgeThreads;  // edges per tile
static_assert(kEdgeItems % 2 == 0, "edges per thread: whole 16-byte words");

struct EdgeOffsets {
    const uint4 *edge;           // [E] as EdgePass
    const int4 *tvs;
    int64_t E, n_tiles;
    unsigned long long *tiles;   // 3 * n_tiles tile words (ET, EF, EE), then the ticket
    unsigned long long *next;    // the workspace buffer zeroed for the next user
    int64_t next_words;
    unsigned *err;
    int64_t *et_off, *ef_off, *ee_off;
    int2 *ev;
};

// two offsets, 16 bytes (k is even)
__device__ __forceinline__ void store_offsets(int64_t *out, int64_t k, int64_t E, long long first,
                                              unsigned len)
{
    if (!out) return;
    if (k + 1 < E) *reinterpret_cast<longlong2 *>(out + k) = make_longlong2(first, first + len);
    else if (k < E) out[k] = first;
}

__global__ void __launch_bounds__(kEdgeThreads, 6) k_edge_offsets(EdgeOffsets p)
{
    griddep_wait();
    {
        const int64_t nthreads = (int64_t)gridDim.x * blockDim.x;
        for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < p.next_words;
             i += nthreads)
            p.next[i] = 0ull;
    }
    __shared__ long long s_tile, s_pre[3];
    if (threadIdx.x == 0) s_tile = (long long)atomicAdd(p.tiles + 3 * p.n_tiles, 1ull);
    __syncthreads();
    const long long tile = s_tile;
    if (p.n_tiles == 0) {   // no edges: the totals alone
        if (tile == 0 && threadIdx.x == 0) {
            if (p.et_off) p.et_off[0] = 0;
            if (p.ef_off) p.ef_off[0] = 0;
            if (p.ee_off) p.ee_off[0] = 0;
        }
        return;
    }
    if (tile >= p.n_tiles) return;
    // rows of 64 edges a warp, two to a lane: records, offsets and EV move as
    // whole lines
    constexpr int kRows = kEdgeItems / 2, kWarps = kEdgeThreads / 32;
    __shared__ unsigned long long s_tef[kWarps];
    __shared__ long long s_ee[kWarps];
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const int64_t k0 = tile * kEdgeTile + wp * (32 * kEdgeItems) + 2 * lane;
    unsigned slot[kRows][2], x[kRows], ex[kRows];   // x, ex: lengths of the first of the two
    unsigned long long tef[kRows], run_tef = 0;   // sums of ET (low half) and EF lengths: below 2^27 each
    long long ee[kRows], run_ee = 0;
#pragma unroll
    for (int r = 0; r < kRows; r++) {
        const int64_t k = k0 + 64 * r;
        unsigned w[8] = {};
        if (k + 1 < p.E) {
            load8(reinterpret_cast<const unsigned *>(p.edge + k), w);
        } else if (k < p.E) {
            const uint4 q = __ldg(p.edge + k);
            w[0] = q.x;
            w[2] = q.z;
            w[3] = q.w;
        }
        slot[r][0] = w[0];
        slot[r][1] = w[4];
        x[r] = w[2];
        ex[r] = w[3];
        tef[r] = (unsigned long long)((w[2] & 0xffffu) + (w[6] & 0xffffu)) |
                 (unsigned long long)((w[2] >> 16) + (w[6] >> 16)) << 32;
        ee[r] = (long long)w[3] + w[7];
        const unsigned long long a0 = tef[r];
        const long long b0 = ee[r];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long a = __shfl_up_sync(0xffffffffu, tef[r], o);
            const long long b = __shfl_up_sync(0xffffffffu, ee[r], o);
            if (lane >= o) {
                tef[r] += a;
                ee[r] += b;
            }
        }
        const unsigned long long a = __shfl_sync(0xffffffffu, tef[r], 31);
        const long long b = __shfl_sync(0xffffffffu, ee[r], 31);
        tef[r] += run_tef - a0;
        ee[r] += run_ee - b0;
        run_tef += a;
        run_ee += b;
    }
    if (lane == 0) {
        s_tef[wp] = run_tef;
        s_ee[wp] = run_ee;
    }
    __syncthreads();
    unsigned long long pre_tef = 0, tot_tef = 0;
    long long pre_ee = 0, tot_ee = 0;
#pragma unroll
    for (int i = 0; i < kWarps; i++) {
        if (i == wp) {
            pre_tef = tot_tef;
            pre_ee = tot_ee;
        }
        tot_tef += s_tef[i];
        tot_ee += s_ee[i];
    }
    if (wp < 3) {   // one look-back per sum, warps 0-2 at once
        const long long t = wp == 0 ? (long long)(tot_tef & 0xffffffffu)
                                    : (wp == 1 ? (long long)(tot_tef >> 32) : tot_ee);
        const long long pre = look_back(p.tiles + wp * p.n_tiles, tile, t, p.err);
        if (lane == 0) s_pre[wp] = pre;
    }
    if (p.ev) {   // while they look
#pragma unroll
        for (int r = 0; r < kRows; r++) {
            const int64_t k = k0 + 64 * r;
            if (k >= p.E) continue;
            const EdgeEnds e = edge_ends(p.tvs, slot[r][0]);
            if (k + 1 < p.E) {
                const EdgeEnds f = edge_ends(p.tvs, slot[r][1]);
                *reinterpret_cast<int4 *>(p.ev + k) = make_int4(e.v, e.u, f.v, f.u);
            } else {
                p.ev[k] = make_int2(e.v, e.u);
            }
        }
    }
    __syncthreads();
    const long long et0 = s_pre[0] + (long long)(pre_tef & 0xffffffffu);
    const long long ef0 = s_pre[1] + (long long)(pre_tef >> 32), ee0 = s_pre[2] + pre_ee;
#pragma unroll
    for (int r = 0; r < kRows; r++) {
        const int64_t k = k0 + 64 * r;
        store_offsets(p.et_off, k, p.E, et0 + (long long)(tef[r] & 0xffffffffu), x[r] & 0xffffu);
        store_offsets(p.ef_off, k, p.E, ef0 + (long long)(tef[r] >> 32), x[r] >> 16);
        store_offsets(p.ee_off, k, p.E, ee0 + ee[r], ex[r]);
    }
    if (tile == p.n_tiles - 1 && threadIdx.x == 0) {
        if (p.et_off) p.et_off[p.E] = s_pre[0] + (long long)(tot_tef & 0xffffffffu);
        if (p.ef_off) p.ef_off[p.E] = s_pre[1] + (long long)(tot_tef >> 32);
        if (p.ee_off) p.ee_off[p.E] = s_pre[2] + tot_ee;
    }
}

// win[w] = first vertex whose row starts at or after entry win_size * w, for
// w in [0, n_win], with win[n_win] = V.  Vertex v owns the windows w with
// off[v-1] < win_size * w <= off[v]; the windows past the last entry (n_win may
// be sized for more) are all threads' work.
__global__ void __launch_bounds__(256)
k_window_starts(const int64_t *__restrict__ off, int64_t V, int64_t n_win, int win_size,
                int *__restrict__ win)
{
    griddep_wait();
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t past = off[V] / win_size + 1;
    for (int64_t w = past + v; w <= n_win; w += (int64_t)gridDim.x * blockDim.x) win[w] = (int)V;
    if (v > V) return;
    const long long lo = v == 0 ? -1 : off[v - 1], hi = off[v];
    for (long long w = lo < 0 ? 0 : lo / win_size + 1; w <= hi / win_size && w <= n_win; w++)
        win[w] = (int)v;
}

// ---------------------------------------------------------------------------
// Star processing order.  Vertex ids need not carry locality (meshes are
// often renumbered; the workloads here permute them) while cell order usually
// does (generators and partitioners emit cells in space-filling order).  The
// star pass therefore visits vertices by first cell, the head of the sorted
// VT row, ties by slot: consecutive vertices then share cells, so a block's
// cell gathers hit L2, and so do those of the per-edge passes, whose records
// come in that order; the output sectors of cell- and id-ordered relations
// they write are completed by blocks running at the same time.
// k_vt_sort marks each vertex's key 4 * first cell + slot in a bitmap over
// the 4T cell slots; the key's rank is the vertex's position.  Heavy vertices
// (vkey < 0) follow at n_light + their rank among the heavy ones; vertices
// without cells come last, in any order (no row of any relation names them).
__global__ void __launch_bounds__(256)
k_vorder_place(const int64_t *__restrict__ vt_off, int64_t V, const int64_t *__restrict__ vkey,
               const uint2 *__restrict__ vrank, int64_t nwk, const uint2 *__restrict__ hrank,
               int *__restrict__ heavy_cnt, int *__restrict__ heavy_off, int *__restrict__ vorder,
               int *__restrict__ vpos)
{
    griddep_wait();
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= V) return;
    const int64_t n_light = (int64_t)__ldg(&vrank[nwk].y), n_heavy = (int64_t)__ldg(&hrank[(V + 31) / 32].y);
    if (v == 0) heavy_cnt[0] = (int)n_heavy;
    int64_t pos;
    if (vt_off[v + 1] == vt_off[v]) {
        const unsigned together = __activemask();
        const int lane = threadIdx.x & 31, leader = __ffs((int)together) - 1;
        int at = 0;
        if (lane == leader) at = atomicAdd(heavy_cnt + 3, __popc(together));
        at = __shfl_sync(together, at, leader) + __popc(together & ((1u << lane) - 1u));
        pos = n_light + n_heavy + at;
    } else {
        const long long key = vkey[v];
        if (key < 0) {
            const int k = rank_of(hrank, v);
            pos = n_light + k;
            // its share of the heavy scratch
            heavy_off[k] = atomicAdd(heavy_cnt + 1, (int)(vt_off[v + 1] - vt_off[v]));
        } else {
            const uint2 r = __ldg(vrank + (key >> 5));
            pos = (int64_t)r.y + __popc(r.x & ((1u << (key & 31)) - 1u));
        }
    }
    vorder[pos] = (int)v;
    vpos[v] = (int)pos;
}

// How far apart neighbours lie by id and by position: the lines of 32 vertices
// (32 words of a field) that the cells of 32 consecutive vertices name, a warp
// per run of them and four cells a vertex; counted as the bits set in a bitmap
// that the lines hash to.
constexpr int kLinesWarps = 4;
__global__ void __launch_bounds__(32 * kLinesWarps)
k_order_lines(int64_t V, const int64_t *__restrict__ vt_off, const int *__restrict__ vt,
              const int4 *__restrict__ tvs, const int *__restrict__ vorder, const int *__restrict__ vpos,
              int *__restrict__ lines)
{
    griddep_wait();
    __shared__ unsigned s_bits[kLinesWarps][128];
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const int i = blockIdx.x * kLinesWarps + wp;
    const bool by_pos = i & 1;
    const int64_t at = 32 * (V / 32 * (i >> 1) / kOrderRuns) + lane;
#pragma unroll
    for (int k = 0; k < 4; k++) s_bits[wp][32 * k + lane] = 0u;
    __syncwarp();
    const int64_t v = by_pos ? vorder[at] : at;
    const int64_t b = vt_off[v];
    const int D = (int)(vt_off[v + 1] - b);
    if (D > 0) {
        int4 w[4];
#pragma unroll
        for (int k = 0; k < 4; k++) w[k] = __ldg(tvs + __ldg(vt + b + (int64_t)D * k / 4));
#pragma unroll
        for (int k = 0; k < 4; k++)
#pragma unroll
            for (int t = 0; t < 4; t++) {
                const int u = get4(w[k], t), x = by_pos ? __ldg(vpos + u) : u;
                const unsigned h = (unsigned)(x >> 5) * 0x9E3779B1u >> 20;
                atomicOr(&s_bits[wp][h >> 5], 1u << (h & 31));
            }
    }
    __syncwarp();
    int n = 0;
#pragma unroll
    for (int k = 0; k < 4; k++) n += __popc(s_bits[wp][32 * k + lane]);
    n = __reduce_add_sync(kAll, n);
    if (lane == 0) atomicAdd(lines + by_pos, n);
}

// First edge and face id of each segment of cells (a mesh of a batch):
// ids are ranks of first occurrences in cell order, so segment i's ids start
// at the rank of its first cell's first occurrence slot.
__global__ void __launch_bounds__(256)
k_seg_ranks(const int64_t *__restrict__ seg_c, int64_t n, const uint2 *__restrict__ erank,
            const uint2 *__restrict__ frank, int64_t *__restrict__ seg_ef)
{
    griddep_wait();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i > n) return;
    seg_ef[i] = rank_of(erank, 6LL * seg_c[i]);
    seg_ef[n + 1 + i] = rank_of(frank, 4LL * seg_c[i]);
}

}  // namespace

int64_t window_count(int64_t n_entries, int win_size) { return n_entries / win_size + 1; }

void launch_window_starts(const int64_t *off, int64_t V, int64_t n_entries, int win_size,
                          int32_t *win, cudaStream_t s)
{
    Launch L("k_window_starts", s);
    launch_pdl(k_window_starts, (unsigned)((V + 1 + 255) / 256), 256, 0, s,
        off, V, window_count(n_entries, win_size), win_size, win);
}

int64_t edge_offsets_words(int64_t max_edges)
{
    return 3 * ((max_edges + kEdgeTile - 1) / kEdgeTile) + 1;
}

void launch_edge_offsets(const EdgePass &e, int64_t *et_off, int64_t *ef_off, int64_t *ee_off,
                         int32_t *ev, ScanWorkspace &ws, DevStatus *st, cudaStream_t s)
{
    EdgeOffsets p{};
    p.edge = e.edge;
    p.tvs = e.tvs;
    p.E = e.E;
    p.n_tiles = (e.E + kEdgeTile - 1) / kEdgeTile;
    p.err = &st->flags;
    p.et_off = et_off;
    p.ef_off = ef_off;
    p.ee_off = ee_off;
    p.ev = reinterpret_cast<int2 *>(ev);
    scan_ws_begin(ws, s, &p.tiles, &p.next, &p.next_words);
    {
        Launch L("k_edge_offsets", s);
        launch_pdl(k_edge_offsets, (unsigned)std::max<int64_t>(p.n_tiles, 1), kEdgeThreads, 0, s, p);
    }
    scan_ws_end(ws, s);
}

void launch_star(const StarPass &p, cudaStream_t s)
{
    if (p.n_light == 0) return;
    Launch L("k_star", s);
    // vertices per warp: enough warps for every SM before long sequences
    const int per = (int)std::min<int64_t>(std::max<int64_t>(p.n_light / kStarFill, 1), kStarPer);
    const int64_t warps = (p.n_light + per - 1) / per;
    const unsigned grid = (unsigned)((warps + kStarWarps - 1) / kStarWarps);
    launch_pdl(p.fnext ? k_star<true> : k_star<false>, grid, kStarThreads, 0, s, p, per);
}

void launch_star_wide(const StarPass &p, int64_t n_wide, cudaStream_t s)
{
    if (n_wide == 0) return;
    Launch L("k_star_wide", s);
    launch_pdl(p.fnext ? k_star_wide<true> : k_star_wide<false>,
               (unsigned)((n_wide + kStarWarps - 1) / kStarWarps), kStarThreads, 0, s, p);
}

void launch_cell_faces(int64_t T, const int4 *tvs, const uint2 *frank, const int32_t *fnext,
                       int32_t *tf, int32_t *ft, int32_t *fv, cudaStream_t s)
{
    if (T == 0) return;
    Launch L("k_cell_faces", s);
    launch_pdl(k_cell_faces, (unsigned)((T + kCellThreads - 1) / kCellThreads), kCellThreads, 0, s, T, tvs, frank,
               reinterpret_cast<const int4 *>(fnext), tf, reinterpret_cast<int2 *>(ft), fv);
}

void launch_edge_ids(const EdgePass &p, cudaStream_t s)
{
    if (p.E == 0) return;
    Launch L("k_edge_ids", s);
    const unsigned grid = (unsigned)((p.E + 255) / 256);
    if (p.rec_hi)
        launch_pdl(k_edge_ids<true>, grid, 256, 0, s, p);
    else
        launch_pdl(k_edge_ids<false>, grid, 256, 0, s, p);
}

void launch_edge_rows(const EdgePass &p, cudaStream_t s)
{
    if (p.E == 0) return;
    Launch L("k_edge_rows", s);
    const unsigned grid = (unsigned)((p.E + kRowsThreads - 1) / kRowsThreads);
    if (p.rec_hi)
        launch_pdl(p.ef ? k_edge_rows<true, true> : k_edge_rows<true, false>, grid, kRowsThreads, 0, s, p);
    else
        launch_pdl(p.ef ? k_edge_rows<false, true> : k_edge_rows<false, false>, grid, kRowsThreads, 0, s, p);
}

void launch_vt_sort(const int64_t *vt_off, int32_t *vt, int64_t V, int64_t nvt, const int4 *tvs,
                    uint32_t *vflag, int64_t *vkey, uint32_t *hflag, int32_t *heavy_cnt, cudaStream_t s)
{
    if (V == 0) return;
    Launch L("k_vt_sort", s);
    launch_pdl(k_vt_sort, (unsigned)((V + kVtsThreads - 1) / kVtsThreads), kVtsThreads, 0, s, vt_off,
               V, nvt, vt, tvs, vflag, vkey, hflag, heavy_cnt);
}

void launch_vv_sort(const int64_t *vv_off, int64_t V, int64_t nvv, int32_t *vv, cudaStream_t s)
{
    if (V == 0 || nvv == 0) return;
    Launch L("k_vv_sort", s);
    launch_pdl(k_vv_sort, (unsigned)((V + kVtsThreads - 1) / kVtsThreads), kVtsThreads, 0, s, vv_off, V,
               nvv, vv);
}

void launch_inc_sort(const int64_t *vv_off, int64_t V, const int2 *inc, int32_t *vv,
                     const int64_t *eid_off, uint32_t *eid, cudaStream_t s)
{
    if (V == 0) return;
    Launch L("k_inc_sort", s);
    launch_pdl(k_inc_sort, (unsigned)((V + kVtsThreads - 1) / kVtsThreads), kVtsThreads, 0, s, vv_off, V,
               inc, vv, eid_off, reinterpret_cast<int *>(eid));
}

void launch_vorder_place(const int64_t *vt_off, int64_t V, const int64_t *vkey, const uint2 *vrank,
                         int64_t nwk, const uint2 *hrank, int32_t *heavy_cnt, int32_t *heavy_off,
                         int32_t *vorder, int32_t *vpos, cudaStream_t s)
{
    if (V == 0) return;
    Launch L("k_vorder_place", s);
    launch_pdl(k_vorder_place, (unsigned)((V + 255) / 256), 256, 0, s, vt_off, V, vkey, vrank, nwk,
               hrank, heavy_cnt, heavy_off, vorder, vpos);
}

void launch_order_lines(int64_t V, const int64_t *vt_off, const int32_t *vt, const int4 *tvs,
                        const int32_t *vorder, const int32_t *vpos, int32_t *lines, cudaStream_t s)
{
    if (V / 32 < kOrderRuns) return;
    Launch L("k_order_lines", s);
    static_assert(2 * kOrderRuns % kLinesWarps == 0, "whole blocks");
    launch_pdl(k_order_lines, 2 * kOrderRuns / kLinesWarps, 32 * kLinesWarps, 0, s, V, vt_off, vt, tvs, vorder,
               vpos, lines);
}

void launch_seg_ranks(const int64_t *seg_c, int64_t n, const uint2 *erank, const uint2 *frank,
                      int64_t *seg_ef, cudaStream_t s)
{
    Launch L("k_seg_ranks", s);
    launch_pdl(k_seg_ranks, (unsigned)((n + 1 + 255) / 256), 256, 0, s, seg_c, n, erank, frank, seg_ef);
}

}  // namespace tg
