// tg_crit.cu -- critical-point classification of a vertex scalar field.
//
// Semantics of the reference critPoints kernel (tlranda/TetraGPU,
// src/alg/critPoints.cu:49-331), restated on an exact VV:
//   * neighbour u of v is lower when f[u] < f[v], or f[u] == f[v] and u < v
//     (:136-140);
//   * two neighbours of the same kind are joined when the mesh has the edge
//     between them, i.e. w is in VV[u] (:172-202), not only edges in v's star;
//   * the lower-link and upper-link component counts go to classes[3v] and
//     classes[3v+1] (:275-284) and the code to classes[3v+2]: (>=1, 0) -> 2,
//     (0, >=1) -> 1, (1, 1) -> 3, anything else -> 4 (:303-330).
//
// The graph both kernels work on is VV renumbered into the star processing
// order (vertices by first cell): rows of neighbour positions, ascending, row
// after row in that order.  Vertex ids need not carry locality; positions
// mostly do, so the neighbours' rows and field values a block gathers lie
// together.  Where ids keep neighbours together as well as positions do,
// positions are ids.  (So they are for the no-allocation entry point, which
// works on VV as it is.)
//
//   k_rows_in_order  VV -> the renumbered rows
//   k_crit_adj       field-independent: for every entry (v, u), the bitmask
//                    of v's neighbours adjacent to u.  Thread per edge (both
//                    of its entries), v's row in a shared-memory hash table.
//   k_crit_classify  field-dependent: lower/upper split, then the components
//                    of each kind counted by a bitmask search over the
//                    adjacency masks of same-kind neighbours.
// A second field on the same mesh reuses the first two.
#include <algorithm>
#include <climits>

#include "tg_internal.h"
#include "tg_rowsort.h"

namespace tg {
namespace {

// ---------------------------------------------------------------------------
// Rows into processing order, each padded with -1 to whole 32-byte sectors (so
// that a thread loads eight entries at once): sixteen lanes copy a row, four rows'
// loads in flight; a thread sorts it (a word between the rows in shared memory:
// 16-word rows would all begin in two banks).  Nine blocks to an SM spill 32 bytes
// a thread, eight none: 79 and 76 us at 96^3 cubes, 37.6 and 38.9 on the 64^3
// coned mesh.
constexpr int kOrderThreads = 128;
constexpr int kOrderCap = 24 * kOrderThreads;
constexpr int kOrderRows = 4;
__global__ void __launch_bounds__(kOrderThreads, 9)
k_rows_in_order(const int64_t *__restrict__ vv_off, const int *__restrict__ vv,
                const int *__restrict__ order, const int *__restrict__ vpos, int64_t V,
                const int64_t *__restrict__ off, int *__restrict__ ent, int *__restrict__ ids,
                int *__restrict__ win, int64_t n_win)
{
    griddep_wait();
    __shared__ int row[kOrderCap + kOrderThreads];
    __shared__ long long s_src[kOrderThreads];
    __shared__ int s_at[kOrderThreads], s_len[kOrderThreads];
    const int64_t i0 = (int64_t)blockIdx.x * kOrderThreads;
    const int64_t i1 = min(i0 + kOrderThreads, V);
    const int64_t i = i0 + threadIdx.x;
    const int64_t base = off[i0];
    const int64_t n = off[i1] - base;
    const int64_t b = off[min(i, i1)];
    auto place = [&](int u) { return vpos ? __ldg(vpos + u) : u; };
    long long src = 0;
    int d = 0;
    if (i < V) {
        const int v = order ? __ldg(order + i) : (int)i;
        src = __ldg(vv_off + v);
        d = (int)(__ldg(vv_off + v + 1) - src);
    }
    if (win) {
        // as k_window_starts: the windows that start in or right after row i,
        // and those past the last entry
        for (int64_t w = off[V] / kAdjWin + 1 + i; w <= n_win; w += (int64_t)gridDim.x * kOrderThreads)
            win[w] = (int)V;
        if (i == 0) win[0] = 0;
        if (i < V)
            for (int64_t w = b / kAdjWin + 1; w <= off[i + 1] / kAdjWin && w <= n_win; w++)
                win[w] = (int)i + 1;
    }
    if (n > kOrderCap) {   // block-uniform: in place
        for (int k = 0; k < d; k++) ent[b + k] = place(__ldg(vv + src + k));
        for (int k = d; k < pad8(d); k++) ent[b + k] = -1;
        if (vpos) sort_rows_warp(ent + b, d);
        __syncwarp();   // a row may have been written by the whole warp
        if (ids)
            for (int k = 0; k < pad8(d); k++) ids[b + k] = ent[b + k] < 0 ? -1 : __ldg(order + ent[b + k]);
        return;
    }
    s_src[threadIdx.x] = src;
    s_at[threadIdx.x] = (int)(b - base);
    s_len[threadIdx.x] = d;
    __syncthreads();
    constexpr int kStep = kOrderThreads / 16;
    const int lane = threadIdx.x & 15;
    for (int r = threadIdx.x >> 4; r < kOrderThreads; r += kStep * kOrderRows) {
        int u[kOrderRows];
#pragma unroll
        for (int t = 0; t < kOrderRows; t++) {
            const int q = r + kStep * t;
            u[t] = lane < s_len[q] ? __ldg(vv + s_src[q] + lane) : -1;
        }
#pragma unroll
        for (int t = 0; t < kOrderRows; t++)
            if (u[t] >= 0) u[t] = place(u[t]);
#pragma unroll
        for (int t = 0; t < kOrderRows; t++) {
            const int q = r + kStep * t, at = s_at[q] + q, len = s_len[q], full = pad8(len);
            if (lane < full) row[at + lane] = u[t];
            for (int k = lane + 16; k < full; k += 16)
                row[at + k] = k < len ? place(__ldg(vv + s_src[q] + k)) : -1;
        }
    }
    __syncthreads();
    if (vpos) {   // (VV's rows are ascending)
        sort_rows_warp(row + (int)(b - base) + threadIdx.x, d);
        __syncthreads();
    }
    for (int q = threadIdx.x >> 4; q < kOrderThreads; q += kStep) {
        const int at = s_at[q], full = pad8(s_len[q]);
        for (int k = lane; k < full; k += 16) {
            const int x = row[at + q + k];
            ent[base + at + k] = x;
            if (ids) ids[base + at + k] = x < 0 ? -1 : __ldg(order + x);
        }
    }
}

// ---------------------------------------------------------------------------
// Link adjacency: for every entry (v, u), bit j of the mask is set when v's
// j-th neighbour is also a neighbour of u.  The common neighbours of v and u
// give both entries (v, u) and (u, v), so one thread takes each edge once, from
// its lower end v: it scans u's row from global memory, looks each w up in v's
// row, and sets bit j in (v, u)'s mask and bit i (w's place in u's row) in
// (u, v)'s, which sits at v's place in u's row.  A block takes the vertices
// whose rows start in a 256-entry window (win); the entries it owns (u > v)
// form a work list.
//
// The look-up is what the pass consists of (14 entries an edge), so a row gets
// a hash table in shared memory: 2^k buckets of two words (64 buckets for 14
// neighbours).  x = w * multiplier (odd) is a bijection of 32-bit words: its
// top k bits are the bucket, and a neighbour's word holds the other bits above
// its place in the row (k bits; a free word all ones, a place that no
// neighbour has), so one 8-byte load and one compare decide.  The row's first
// neighbour that finds its bucket full (one row of 12 has one) is kept apart,
// where every look-up compares with it; a row with a second one is hashed
// again with the next multiplier, and one that no multiplier was found for
// keeps its sorted entries padded with INT_MAX for a binary search.  Bound by
// the shared-memory pipe (86%) and issue (64%).  A binary search over VV in id
// order (four dependent loads and 35 instructions an entry, neighbours' rows
// scattered: 5.2 requests to L2 an edge against 2): 709 -> 488 us at 128^3,
// 127 -> 88 us on the 64^3 coned mesh, the renumbering included 890 -> 780 us.
constexpr int kAdjCap = kAdjWin + kMaxDeg;
constexpr int kAdjThreads = TG_ADJ_THREADS;
constexpr int kAdjWords = 8;       // table words per entry
constexpr int kHashTries = 8;

// buckets of a row of d entries, log2: two words each in the row's share
__device__ __forceinline__ int hash_bits(int d) { return min(30 - __clz(kAdjWords * d), 8); }

__device__ __forceinline__ unsigned multiplier(unsigned i)   // some odd word per i
{
    unsigned x = (i + 1u) * 0x9E3779B1u;
    x ^= x >> 15;
    x *= 0x85EBCA77u;
    x ^= x >> 13;
    return x | 1u;
}

// v's row as u's row is matched against it: a hash table (mul not 0) or the
// padded row
struct AdjRow {
    const unsigned *tab;
    unsigned mul;
    int apart, apart_at;   // the neighbour kept apart (-2: none) and its place
    int k, d, top;         // top: the power of two at or above d
};

// u's row (urow, un entries) against v's: each w found at place j of v's row
// sets bit j of bits_v and bit i of bits_u; pv = v's place in u's row.  PAD:
// rows are padded with -1 (which no row holds) to whole sectors.  HASH: v's
// row has a table; else a binary search of the steps top / 2, .. 1 (those
// above top / 2 skipped by a per-thread predicate, so the lanes of a warp stay
// together; every probe lies in the padded row).
template <typename M, bool PAD, bool HASH>
__device__ __forceinline__ void adj_scan(const AdjRow &R, const int *__restrict__ urow, int un, int v,
                                         M &bits_v, M &bits_u, int &pv)
{
    const int *row = reinterpret_cast<const int *>(R.tab);
    const int up = 32 - R.k;
    for (int i0 = 0; i0 < un; i0 += 8) {
        int q[8];
        if constexpr (PAD) {
            unsigned w8[8];
            load8(reinterpret_cast<const unsigned *>(urow + i0), w8);
#pragma unroll
            for (int t = 0; t < 8; t++) q[t] = (int)w8[t];
        } else {
#pragma unroll
            for (int t = 0; t < 8; t++) q[t] = i0 + t < un ? __ldg(urow + i0 + t) : -1;
        }
        // look-ups in lock step (independent shared-memory loads in flight
        // together)
        unsigned hits = 0u;
#pragma unroll
        for (int t0 = 0; t0 < 8; t0 += 4) {
            unsigned at[4];
            if constexpr (HASH) {
                uint2 w[4];
                unsigned x[4];
#pragma unroll
                for (int t = 0; t < 4; t++) {
                    x[t] = (unsigned)q[t0 + t] * R.mul;
                    w[t] = reinterpret_cast<const uint2 *>(R.tab)[x[t] >> up];
                }
                // the place, if below d (at most one of the two words is w's)
#pragma unroll
                for (int t = 0; t < 4; t++) {
                    at[t] = min(w[t].x ^ (x[t] << R.k), w[t].y ^ (x[t] << R.k));
                    at[t] = q[t0 + t] == R.apart ? (unsigned)R.apart_at : at[t];
                }
            } else {
                int lo[4] = {0, 0, 0, 0};
#pragma unroll
                for (int step = kMaxDeg / 2; step > 0; step >>= 1) {
                    if (2 * step > R.top) continue;
#pragma unroll
                    for (int t = 0; t < 4; t++)
                        lo[t] += row[lo[t] + step - 1] < q[t0 + t] ? step : 0;
                }
#pragma unroll
                for (int t = 0; t < 4; t++)
                    at[t] = row[lo[t]] == q[t0 + t] ? (unsigned)lo[t] : ~0u;
            }
#pragma unroll
            for (int t = 0; t < 4; t++) {
                pv = q[t0 + t] == v ? i0 + t0 + t : pv;
                const bool hit = at[t] < (unsigned)R.d;
                bits_v |= hit ? (M)1 << (at[t] & (8 * sizeof(M) - 1)) : (M)0;
                hits |= hit ? 1u << (t0 + t) : 0u;
            }
        }
        bits_u |= (M)hits << (i0 & (8 * (int)sizeof(M) - 1));
    }
}

// Rows longer than kMaxDeg (vertices whose classes tg_heavy.cu computes) are
// not staged and get no masks; with heavy = 1 an entry (v, u) of a light v
// whose neighbour u is such a vertex is computed from v's side whichever end
// is lower (u computes nothing); heavy = 2 reports them instead
// (ST_HEAVY_DEG) for callers without the heavy path.  Light rows start
// below kAdjWin in their window and end below kAdjCap, so they always fit.
// M: the masks (32-bit when no row holds more than 32 entries).  PAD: as in
// adj_scan (row lengths include the padding).
template <typename M, bool PAD>
__global__ void __launch_bounds__(kAdjThreads)
k_crit_adj(const int64_t *__restrict__ off, const int *__restrict__ ent, const int *__restrict__ win,
           M *__restrict__ adj, DevStatus *st, int heavy)
{
    griddep_wait();
    __shared__ __align__(16) int nb[kAdjCap];
    __shared__ __align__(16) unsigned tab[kAdjWords * kAdjCap];   // tables (or padded rows)
    // an entry's row by its first entry here; kNoRow: no light row there
    __shared__ __align__(16) unsigned short meta[kAdjCap];
    __shared__ unsigned short own[kAdjCap];
    // at a row's first entry: its vertex, its length, its multiplier (0 without
    // a table), the neighbour kept apart and its place
    __shared__ int vid[kAdjCap], apart[kAdjCap];
    __shared__ unsigned mul[kAdjCap];
    __shared__ unsigned char len[kAdjCap], apart_at[kAdjCap];
    __shared__ int n_own;
    constexpr unsigned kNoRow = 0xffffu;
    const int lane = threadIdx.x & 31;
    // every thread reads the window's bounds itself (the same words: one
    // transaction each), so the block needs no barrier before the rows
    // unless the heavy modes leave rows out
    const int s_vlo = win[blockIdx.x], s_vhi = win[blockIdx.x + 1];
    const long long base = off[s_vlo];
    const int s_n = (int)(off[s_vhi] - base);
    if (s_n == 0) return;
    const int n = min(s_n, kAdjCap);
    if (threadIdx.x == 0) n_own = 0;
    if (heavy) {
        for (int e = threadIdx.x; e < kAdjCap; e += kAdjThreads) meta[e] = kNoRow;
        __syncthreads();
    }
    if (heavy == 2 && s_n > kAdjCap) {  // a row longer than kMaxDeg lies in this window
        if (threadIdx.x == 0) {
            atomicOr(&st->flags, ST_HEAVY_DEG);
            note_lowest(&st->bad_vertex, s_vlo);
        }
        return;
    }
    if constexpr (PAD) {
        for (int e = 4 * threadIdx.x; e < n; e += 4 * kAdjThreads) cp_async<16>(&nb[e], ent + base + e);
    } else {
        for (int e = threadIdx.x; e < n; e += kAdjThreads) cp_async<4>(&nb[e], ent + base + e);
    }
    cp_async_commit();
    for (int j = threadIdx.x; j < kAdjWords * kAdjCap / 4; j += kAdjThreads)   // free words
        if (4 * j < kAdjWords * n)
            reinterpret_cast<uint4 *>(tab)[j] = make_uint4(~0u, ~0u, ~0u, ~0u);
    for (int i = s_vlo + threadIdx.x; i < s_vhi; i += kAdjThreads) {
        const int rs = (int)(off[i] - base);
        const int d = (int)(off[i + 1] - off[i]);
        if (d == 0) continue;
        if (d > kMaxDeg) {
            if (heavy == 2) {
                atomicOr(&st->flags, ST_HEAVY_DEG);
                note_lowest(&st->bad_vertex, i);
            }
            continue;
        }
        vid[rs] = i;
        len[rs] = (unsigned char)d;
        mul[rs] = multiplier(0u);
        apart[rs] = -2;
        if constexpr (PAD) {
            const unsigned two = (unsigned)rs * 0x10001u;
            for (int k = 0; k < d; k += 8)
                *reinterpret_cast<uint4 *>(meta + rs + k) = make_uint4(two, two, two, two);
        } else {
            for (int k = 0; k < d; k++) meta[rs + k] = (unsigned short)rs;
        }
    }
    cp_async_wait();
    __syncthreads();
    // the entries into their rows' tables; those of a row that did not fit
    // again under the next multiplier.  The owned entries on the first way.
    for (int trial = 0; trial < kHashTries; trial++) {
        const unsigned c = multiplier((unsigned)trial);
        bool failed = false;
        for (int e0 = threadIdx.x - lane; e0 < n; e0 += kAdjThreads) {
            const int e = e0 + lane;
            const unsigned rs = e < n ? meta[e] : kNoRow;
            const int u = rs != kNoRow ? nb[e] : -1;
            if (u >= 0 && mul[rs] == c) {
                const int k = hash_bits(len[rs]);
                const unsigned x = (unsigned)u * c;
                const unsigned word = x << k | (unsigned)(e - rs);
                unsigned *bucket = tab + kAdjWords * rs + 2 * (x >> (32 - k));
                if (atomicCAS(bucket, ~0u, word) != ~0u && atomicCAS(bucket + 1, ~0u, word) != ~0u) {
                    if (atomicCAS(&apart[rs], -2, u) == -2) {
                        apart_at[rs] = (unsigned char)(e - rs);
                    } else {
                        failed = true;
                        mul[rs] = 0u;   // this row again
                    }
                }
            }
            if (trial == 0) {
                bool mine = u >= 0 && u > vid[rs];
                if (heavy == 1 && u >= 0 && !mine)   // a heavy lower end computes nothing
                    mine = __ldg(off + u + 1) - __ldg(off + u) > kMaxDeg;
                const unsigned b = __ballot_sync(0xffffffffu, mine);
                int o = 0;
                if (lane == 0 && b) o = atomicAdd(&n_own, __popc(b));
                o = __shfl_sync(0xffffffffu, o, 0) + __popc(b & ((1u << lane) - 1u));
                if (mine) own[o] = (unsigned short)e;
            }
        }
        if (!__syncthreads_or(failed)) break;
        for (int e = threadIdx.x; e < n; e += kAdjThreads) {
            const unsigned rs = meta[e];
            if (rs == kNoRow || mul[rs]) continue;
            // this entry's part of the row's share of the tables: free words,
            // or out of multipliers the row itself
            unsigned *t = tab + kAdjWords * rs;
            if (trial + 1 < kHashTries) {
                for (int j = 0; j < kAdjWords; j++) t[kAdjWords * (e - rs) + j] = ~0u;
                if (e == rs) apart[rs] = -2;
            } else {
                t[e - rs] = nb[e] >= 0 ? (unsigned)nb[e] : (unsigned)INT_MAX;
                t[e - rs + len[rs]] = (unsigned)INT_MAX;
            }
        }
        __syncthreads();
        if (trial + 1 < kHashTries) {
            for (int e = threadIdx.x; e < n; e += kAdjThreads)
                if (meta[e] == e && !mul[e]) mul[e] = multiplier((unsigned)trial + 1u);
            __syncthreads();
        }
    }
    const int no = n_own;
    for (int k = threadIdx.x; k < no; k += kAdjThreads) {
        const int e = own[k], rs = meta[e], d = len[rs];
        const int v = vid[rs], u = nb[e];
        const int64_t ub = off[u];
        const int un = (int)(off[u + 1] - ub);
        if (un > kMaxDeg && heavy != 1) continue;  // reported by u's own block
        int pv = -1;
        M bv, bu;
        AdjRow R;
        R.tab = tab + kAdjWords * rs;
        R.mul = mul[rs];
        R.apart = apart[rs];
        R.apart_at = apart_at[rs];
        R.k = hash_bits(d);
        R.d = d;
        R.top = d <= 1 ? 1 : 1 << (32 - __clz(d - 1));
        if (sizeof(M) == 4 || (d <= 32 && un <= 32)) {   // both masks fit 32 bits
            unsigned bv32 = 0u, bu32 = 0u;
            if (R.mul) adj_scan<unsigned, PAD, true>(R, ent + ub, un, v, bv32, bu32, pv);
            else adj_scan<unsigned, PAD, false>(R, ent + ub, un, v, bv32, bu32, pv);
            bv = bv32;
            bu = bu32;
        } else {
            bv = bu = 0;
            if (R.mul) adj_scan<M, PAD, true>(R, ent + ub, un, v, bv, bu, pv);
            else adj_scan<M, PAD, false>(R, ent + ub, un, v, bv, bu, pv);
        }
        adj[base + e] = bv;
        // u's mask is u's to keep only when u's row is light (else it has none)
        if (pv >= 0 && un <= kMaxDeg) adj[ub + pv] = bu;
    }
}

// ---------------------------------------------------------------------------
constexpr int kClassifyThreads = 128;
// From kOrderField vertices on the field is put in processing order first (a
// launch and a buffer: 3 to 4 us), so that a block's field gathers lie together;
// below, they hit L1 and L2 anyway.  A call by id and in order, grids with ids
// permuted: 11.6 and 16.3 us at 4,913 vertices, 16.0 and 17.2 at 118k, 18.6 and
// 18.5 at 185k, 24.0 and 21.8 at 275k, 143 and 95 at 2.1M (float64 17.7 and 20.2,
// 19.9 and 22.5, 27.0 and 26.7, 152 and 119 from 118k on).
// The rows of smaller meshes are kept as vertices too, one gather of a chain
// of four fewer.
//
// A field's values by position: of every vertex (vpos null: a thread per
// position), or of the vertices from v0 on (a thread per vertex)
template <typename F>
__global__ void __launch_bounds__(256)
k_field_in_order(const F *__restrict__ field_v0, const int *__restrict__ order,
                 const int *__restrict__ vpos, int64_t v0, int64_t nv, F *__restrict__ out)
{
    griddep_wait();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nv) return;
    if (vpos) out[vpos[v0 + i]] = field_v0[i];
    else out[i] = __ldg(field_v0 + order[i]);
}

// u == v for many u.  Doubles by their bits: the FP64 pipe, which takes the other
// comparison, bounds the classification of float64 fields (128^3 cubes: 146 us a
// call with both there, 99 with one; none there is no faster).
template <typename F>
struct EqualTo {
    F v;
    unsigned long long care = ~0ull, bits = 0ull;
    __device__ __forceinline__ explicit EqualTo(F x) : v(x)
    {
        if constexpr (sizeof(F) == 8) {
            bits = (unsigned long long)__double_as_longlong(x);
            if (bits << 1 == 0ull) {   // both zeros
                care = ~0ull >> 1;
                bits = 0ull;
            } else if (bits << 1 > 0xffe0000000000000ull) {   // NaN: nothing
                care = 0ull;
            }
        }
    }
    __device__ __forceinline__ bool operator()(F u) const
    {
        if constexpr (sizeof(F) == 8) return ((unsigned long long)__double_as_longlong(u) & care) == bits;
        else return u == v;
    }
};

// Components of the lower and upper link subgraphs by bitmask search: a
// component grows from its lowest unreached member, each member reached
// once adding its same-kind neighbours (its adjacency mask) to the frontier,
// until none is left to reach: at most deg turns whatever the link's shape.  One
// loop over the members of all components: with a loop per component the lanes
// of a warp wait for each other at the end of each (86 -> 74 us at 128^3 cubes).
// The heavy stars' rows, a mesh's longest, are neighbours in star order: they
// take the last lane of a warp each, of the first warps (hn of them, from
// position h0 on), and the rows of those lanes the places of the heavy ones.
//
// A thread per vertex: positions v0 .. v0 + nv - 1 (vpos null: all of them, or
// positions are ids), or the positions of the vertices v0 .. v0 + nv - 1 (a
// vertex range that holds every neighbour of its vertices: a whole mesh of a
// batch).  order: the vertex at each position
// (null: positions are ids), for output; to_id: the vertex of an entry (null:
// entries are vertices), for ties and by id.  field: values by position, or
// (BY_ID) by vertex from v0.
template <typename F, typename M, bool PAD, bool BY_ID>
__global__ void __launch_bounds__(kClassifyThreads)
k_crit_classify(const int64_t *__restrict__ off, const int *__restrict__ ent,
                const M *__restrict__ adj, const F *__restrict__ field,
                const int *__restrict__ order, const int *__restrict__ to_id,
                const int *__restrict__ vpos, int64_t v0, int64_t nv, int64_t h0, int64_t hn,
                unsigned *__restrict__ classes3_v0)
{
    griddep_wait();
    int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nv) return;
    if ((t & 31) == 31 && (t >> 5) < hn) t = h0 + (t >> 5);
    else if (t >= h0 && t < h0 + hn) t = 32 * (t - h0) + 31;
    const int64_t i = vpos ? vpos[v0 + t] : v0 + t;
    const int64_t v = vpos || !order ? v0 + t : order[t];
    unsigned *classes3 = classes3_v0 - 3 * v0;
    const int64_t b = off[i];
    const int n = (int)(off[i + 1] - b);
    if (n > kMaxDeg) return;   // tg_heavy.cu classifies it
    auto first = [](M m) {
        return sizeof(M) == 8 ? __ffsll((long long)m) - 1 : __ffs((int)(unsigned)m) - 1;
    };
    unsigned lo = 0, up = 0;
    {
        if constexpr (BY_ID) field -= v0;
        const F fv = field[BY_ID ? v : i];
        const EqualTo<F> equal(fv);
        M lower = 0, all = 0, same = 0;   // same: ties, decided by id afterwards
        // eight entries at a time without a branch (four of rows that are not
        // padded), so that their values are on the way together; a missing entry
        // looks at the vertex itself
        constexpr int kRow = PAD ? 8 : 4;
        for (int k = 0; k < n; k += kRow) {
            unsigned u[kRow];
            if constexpr (PAD) {
                load8(reinterpret_cast<const unsigned *>(ent + b + k), u);
            } else {
#pragma unroll
                for (int q = 0; q < kRow; q++) u[q] = k + q < n ? (unsigned)__ldg(ent + b + k + q) : ~0u;
            }
            unsigned some = 0u, less = 0u, tie = 0u;
            // (doubles four by four: registers)
            constexpr int kStep = sizeof(F) == 8 ? 4 : kRow;
#pragma unroll
            for (int q0 = 0; q0 < kRow; q0 += kStep) {
                if (q0 > 0 && (int)u[q0] < 0) break;   // padding from there on
                F fu[kStep];
#pragma unroll
                for (int q = 0; q < kStep; q++) {
                    const int x = (int)u[q0 + q];
                    if constexpr (BY_ID) {
                        const int id = to_id && x >= 0 ? __ldg(to_id + x) : x;
                        fu[q] = __ldg(field + (x >= 0 ? id : (int)v));
                    } else {
                        fu[q] = __ldg(field + (x >= 0 ? x : (int)i));
                    }
                }
#pragma unroll
                for (int q = 0; q < kStep; q++) {
                    some |= (int)u[q0 + q] >= 0 ? 1u << (q0 + q) : 0u;
                    less |= fu[q] < fv ? 1u << (q0 + q) : 0u;
                    tie |= equal(fu[q]) ? 1u << (q0 + q) : 0u;
                }
            }
            all |= (M)some << k;
            lower |= (M)less << k;
            same |= (M)(tie & some) << k;
        }
        for (; same; same &= same - 1) {
            const int u = __ldg(ent + b + first(same));
            if ((to_id ? __ldg(to_id + u) : u) < (int)v) lower |= same & (0 - same);
        }
        M rem = all, frontier = 0, kind = 0;   // rem: not reached yet
        while (rem) {
            if (!frontier) {   // the next component
                frontier = rem & (0 - rem);
                rem ^= frontier;
                const bool is_lo = (lower & frontier) != 0;
                kind = is_lo ? lower : ~lower;
                if (is_lo) lo++; else up++;
            }
            const int j = first(frontier);
            frontier &= frontier - 1;
            const M nb = __ldg(adj + b + j) & kind & rem;
            rem ^= nb;
            frontier |= nb;
        }
    }
    unsigned code;
    if (lo >= 1 && up == 0) code = 2;
    else if (lo == 0 && up >= 1) code = 1;
    else if (lo == 1 && up == 1) code = 3;
    else code = 4;
    // two stores for three words (rows lie by vertex id, a request each):
    // 90 -> 86 us at 2.1M vertices, ids permuted
    unsigned *c = classes3 + 3 * v;
    const bool even = ((uintptr_t)c & 7) == 0;
    *reinterpret_cast<uint2 *>(even ? c : c + 1) = even ? make_uint2(lo, up) : make_uint2(up, code);
    c[even ? 2 : 0] = even ? code : lo;
}

}  // namespace

int crit_window() { return kAdjWin; }

void launch_rows_in_order(const int64_t *vv_off, const int32_t *vv, const int32_t *order,
                          const int32_t *vpos, int64_t V, const int64_t *off, int32_t *ent, int32_t *ids,
                          int32_t *win, int64_t n_win, cudaStream_t s)
{
    if (V == 0) return;
    Launch L("k_rows_in_order", s);
    launch_pdl(k_rows_in_order, (unsigned)((V + kOrderThreads - 1) / kOrderThreads), kOrderThreads, 0, s,
               vv_off, vv, order, vpos, V, off, ent, ids, win, n_win);
}

void launch_crit_adj(const LinkGraph &g, const int32_t *win, DevStatus *st, int heavy, cudaStream_t s)
{
    if (g.V == 0) return;
    Launch L("k_crit_adj", s);
    const unsigned grid = (unsigned)window_count(g.n_ent, kAdjWin);
    if (!g.padded)   // plain VV: 64-bit masks
        launch_pdl(k_crit_adj<unsigned long long, false>, grid, kAdjThreads, 0, s, g.off, g.ent, win,
                   (unsigned long long *)g.adj, st, heavy);
    else if (g.wide)
        launch_pdl(k_crit_adj<unsigned long long, true>, grid, kAdjThreads, 0, s, g.off, g.ent, win,
                   (unsigned long long *)g.adj, st, heavy);
    else
        launch_pdl(k_crit_adj<unsigned, true>, grid, kAdjThreads, 0, s, g.off, g.ent, win,
                   (unsigned *)g.adj, st, heavy);
}

namespace {
template <typename F, bool BY_ID>
void classify(const LinkGraph &g, const F *field, const int32_t *vpos, int64_t v0, int64_t nv,
              uint32_t *classes3, cudaStream_t s)
{
    const unsigned grid = (unsigned)((nv + kClassifyThreads - 1) / kClassifyThreads);
    Launch L("k_crit_classify", s);
    // by id, over the rows as vertices where there are such
    const int32_t *ent = BY_ID && g.ids ? g.ids : g.ent;
    const int32_t *to_id = BY_ID && g.ids ? nullptr : g.order;
    // (positions are ids, or a range by vertex: those rows lie anywhere)
    const int64_t h0 = g.heavy0, hn = g.order && !vpos ? std::min(g.n_heavy, g.heavy0 / 32) : 0;
    if (!g.padded)
        launch_pdl(k_crit_classify<F, unsigned long long, false, BY_ID>, grid, kClassifyThreads, 0, s,
                   g.off, ent, (const unsigned long long *)g.adj, field, g.order, to_id, vpos, v0, nv,
                   h0, hn, classes3);
    else if (g.wide)
        launch_pdl(k_crit_classify<F, unsigned long long, true, BY_ID>, grid, kClassifyThreads, 0, s,
                   g.off, ent, (const unsigned long long *)g.adj, field, g.order, to_id, vpos, v0, nv,
                   h0, hn, classes3);
    else
        launch_pdl(k_crit_classify<F, unsigned, true, BY_ID>, grid, kClassifyThreads, 0, s, g.off, ent,
                   (const unsigned *)g.adj, field, g.order, to_id, vpos, v0, nv, h0, hn,
                   classes3);
}

template <typename F>
void classify(const LinkGraph &g, const F *field, F *ordered, int64_t v0, int64_t nv,
              uint32_t *classes3, cudaStream_t s)
{
    const int32_t *vpos = nv < g.V ? g.vpos : nullptr;
    if (!ordered) {
        classify<F, true>(g, field, vpos, v0, nv, classes3, s);
        return;
    }
    {
        Launch L("k_field_in_order", s);
        launch_pdl(k_field_in_order<F>, (unsigned)((nv + 255) / 256), 256, 0, s, field, g.order, vpos, v0,
                   nv, ordered);
    }
    classify<F, false>(g, ordered, vpos, v0, nv, classes3, s);
}
}  // namespace

void launch_field_in_order(const float *field, const int32_t *order, int64_t V, float *out,
                           cudaStream_t s)
{
    if (V == 0) return;
    Launch L("k_field_in_order", s);
    launch_pdl(k_field_in_order<float>, (unsigned)((V + 255) / 256), 256, 0, s, field, order, nullptr,
               (int64_t)0, V, out);
}

bool classify_orders_field(int64_t nv) { return nv >= kOrderField; }

void launch_crit_classify(const LinkGraph &g, const void *field, int field_type, void *ordered,
                          int64_t v0, int64_t nv, uint32_t *classes3, cudaStream_t s)
{
    if (nv == 0) return;
    if (field_type == 1)
        classify(g, (const double *)field, (double *)ordered, v0, nv, classes3, s);
    else
        classify(g, (const float *)field, (float *)ordered, v0, nv, classes3, s);
}

}  // namespace tg
