// tg_kernels.cu -- the relation-extraction pipeline for sm_103a.
//
// Id rules reproduced (reference tlranda/TetraGPU, src/cpu_extraction.cpp):
//   edge id = rank of the edge's first occurrence p = 6*cell + j, pairs j in
//             order (0,1),(0,2),(0,3),(1,2),(1,3),(2,3)         (:28-62)
//   face id = rank of the face's first occurrence q = 4*cell + k, faces
//             visited with skip = 3,2,1,0 (:145) and k = TF column = 3 - skip,
//             skip being the omitted slot                        (:122-174)
// on row-sorted TV.  Instead of the reference's serial table scans, the
// first occurrences are found per vertex: the cells around a vertex v (its
// star, the sorted VT row) contain every cell holding any edge or face at v,
// so the lowest star position holding a neighbour u is the first occurrence
// of edge (v,u), and the lowest holding both x and y is the first occurrence
// of face (v,x,y).  First occurrences are marked in bitmaps over all
// occurrence slots; a popcount prefix turns any occurrence into its id.
//
// Kernels, in pipeline order (one thread per cell/face/edge unless noted):
//   k_canon        sort TV rows, validate ids, count cells per vertex
//   k_vt_fill      cells into VT rows, those of 32 cells vertex by vertex
//   k_vt_sort, k_star, k_cell_faces, k_edge_ids, k_edge_offsets, k_inc_sort,
//   k_vv_sort, k_edge_rows    the star pass and what follows it (tg_star.cu)
//   k_cell_tt      face-sharing TT
//   k_face_fill    FE (from TE of a face's first cell), FF
//   k_ee_fill      EE
//   k_tt_vertex, k_tt_vertex_far   vertex-sharing TT
#include <algorithm>
#include <climits>

#include "tg_internal.h"

namespace tg {
namespace {

constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ int get4(const int4 &w, int i)
{
    return i == 0 ? w.x : (i == 1 ? w.y : (i == 2 ? w.z : w.w));
}

// index of the vertex pair (s, t), s < t, in the reference TE order
__device__ __forceinline__ int pair_slot(int s, int t)
{
    return s == 0 ? t - 1 : (s == 1 ? t + 1 : 5);
}

#define TG_CSWAP(x, y) \
    if ((x) > (y)) { int _t = (x); (x) = (y); (y) = _t; }

// one comparator of a sorting network: (x, y) <- (min, max)
__device__ __forceinline__ void cswap(int &x, int &y)
{
    const int lo = min(x, y);
    y = max(x, y);
    x = lo;
}

// ---------------------------------------------------------------------------
// k_canon
// ---------------------------------------------------------------------------
// A warp's 128 (cell, slot) pairs name far fewer distinct vertices on meshes
// whose cells come in spatial order (a run of cubes shares its corners): some
// 26.  The pairs of a vertex agree on one of them (each writes its number where
// the vertex hashes to and reads back whose stayed; a vertex that finds another
// there tries again elsewhere), count themselves at it, and that one makes one
// global atomic, whose return value is the warp's base in the vertex's VT row.
// The warp leaves its pairs' order by vertex: a pair's place in it, a bit per
// place that begins a vertex, and each vertex with its base less that place, so
// that k_vt_fill writes a vertex's cells of the warp together.  210 us at 128^3 cubes,
// vertex ids permuted (318 with a table of the block's 1024 pairs and barriers:
// a compare-and-swap and an add a pair, of which lanes naming the same vertex
// wait for each other); bound by the shared-memory pipe (83 %).  Whole warps
// that agree by match instructions first took as long as the table.
constexpr int kCanonThreads = 256, kCanonWarps = kCanonThreads / 32;
constexpr int kCanonPairs = 128;   // of a warp
constexpr int kCanonTable = 512;
struct CanonStage {
    int key[kCanonPairs];                // pair 32 k + lane: slot k of the lane's cell
    int cnt[kCanonPairs];                // at the pair that stands for a vertex
    unsigned char table[kCanonTable];
    unsigned char pair[kCanonPairs];     // of each vertex, and its first place
    unsigned char start[kCanonPairs + 4];
};

__global__ void __launch_bounds__(kCanonThreads, 6)
k_canon(const int32_t *tv, int64_t T, int V, int4 *tvs, int *deg_t, VtOrder vo, DevStatus *st,
        int aligned)
{
    griddep_wait();
    __shared__ CanonStage s_stage[kCanonWarps];
    const int lane = threadIdx.x & 31;
    CanonStage &S = s_stage[threadIdx.x >> 5];
    const int64_t c = (int64_t)blockIdx.x * kCanonThreads + threadIdx.x;
    int q[4] = {-1, -1, -1, -1};
    bool ok = false;
    if (c < T) {
        int a, b, d, e;
        if (aligned) {
            int4 w = reinterpret_cast<const int4 *>(tv)[c];
            a = w.x; b = w.y; d = w.z; e = w.w;
        } else {
            a = tv[4 * c]; b = tv[4 * c + 1]; d = tv[4 * c + 2]; e = tv[4 * c + 3];
        }
        // A rejected cell is overwritten with -1s (the input may alias tvs)
        // and takes no part in the counts; every later kernel skips it, and
        // the host reports the error before anything reads the mesh again.
        if ((unsigned)a >= (unsigned)V || (unsigned)b >= (unsigned)V ||
            (unsigned)d >= (unsigned)V || (unsigned)e >= (unsigned)V) {
            atomicOr(&st->flags, ST_BAD_ID);
            note_lowest(&st->bad_cell, (int)c);
            tvs[c] = make_int4(-1, -1, -1, -1);
        } else {
            TG_CSWAP(a, b);
            TG_CSWAP(d, e);
            TG_CSWAP(a, d);
            TG_CSWAP(b, e);
            TG_CSWAP(b, d);
            if (a == b || b == d || d == e) {
                atomicOr(&st->flags, ST_DUP_VERTEX);
                note_lowest(&st->bad_cell, (int)c);
                tvs[c] = make_int4(-1, -1, -1, -1);
            } else {
                tvs[c] = make_int4(a, b, d, e);
                q[0] = a; q[1] = b; q[2] = d; q[3] = e;
                ok = true;
            }
        }
    }
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 4; k++) {
        S.key[32 * k + lane] = q[k];
        S.cnt[32 * k + lane] = 0;
    }
    // rep[k]: the pair that stands for the vertex (a rejected cell's -1s are one
    // more).  A vertex's pairs look in the same place each time, and one vertex
    // at each place looked at stays: at most kCanonPairs rounds
    int rep[4];
    bool todo[4] = {true, true, true, true};
    unsigned mul = 0x9E3779B1u;
    for (int round = 0; round < kCanonPairs; round++, mul += 0x85EBCA6Eu) {
        __syncwarp();
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (todo[k]) S.table[((unsigned)q[k] * mul) >> 23] = (unsigned char)(32 * k + lane);
        __syncwarp();
        int r[4];
#pragma unroll
        for (int k = 0; k < 4; k++) r[k] = S.table[((unsigned)q[k] * mul) >> 23] & (kCanonPairs - 1);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const bool found = S.key[r[k]] == q[k];
            rep[k] = todo[k] ? r[k] : rep[k];
            todo[k] = todo[k] && !found;
        }
        if (!__any_sync(kFull, todo[0] || todo[1] || todo[2] || todo[3])) break;
    }
    int rk[4];
#pragma unroll
    for (int k = 0; k < 4; k++) rk[k] = atomicAdd(&S.cnt[rep[k]], 1);
    __syncwarp();
    // the places of this lane's vertices: vertices and pairs of the lanes
    // before it, in the halves of a word
    int n[4];
    unsigned own = 0;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const int m = S.cnt[32 * k + lane];
        n[k] = ok && rep[k] == 32 * k + lane ? m : 0;
        own += n[k] ? (unsigned)n[k] << 16 | 1u : 0u;
    }
    unsigned at = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(kFull, at, o);
        if (lane >= o) at += y;
    }
    const unsigned all = __shfl_sync(kFull, at, 31);
    at -= own;
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 4; k++)
        if (n[k]) {
            S.pair[at & 0xffffu] = (unsigned char)(32 * k + lane);
            S.start[at & 0xffffu] = (unsigned char)(at >> 16);
            S.cnt[32 * k + lane] = (int)(at >> 16);
            at += (unsigned)n[k] << 16 | 1u;
        }
    const int verts = (int)(all & 0xffffu);
    if (lane == 0) S.start[verts] = (unsigned char)(all >> 16);
    __syncwarp();
    // the count so far of cells at a vertex is the warp's base in its VT row
    // (rows are sorted afterwards)
    const int64_t tile = c >> 5;
    unsigned head[4] = {0, 0, 0, 0};
    for (int i = lane; i < verts; i += 32) {
        const int v = S.key[S.pair[i]], place = S.start[i];
        vo.verts[tile * kCanonPairs + i] =
            make_int2(v, atomicAdd(deg_t + v, S.start[i + 1] - place) - place);
        const unsigned bit = 1u << (place & 31);
#pragma unroll
        for (int w = 0; w < 4; w++) head[w] |= place >> 5 == w ? bit : 0u;
    }
#pragma unroll
    for (int w = 0; w < 4; w++) head[w] = __reduce_or_sync(kFull, head[w]);
    if (c >= T) return;
    if (lane == 0) vo.head[tile] = make_uint4(head[0], head[1], head[2], head[3]);
    unsigned place = ~0u;   // rejected
    if (ok) {
        place = 0;
#pragma unroll
        for (int k = 0; k < 4; k++) place |= (unsigned)(S.cnt[rep[k]] + rk[k]) << (8 * k);
    }
    vo.place[c] = place;
}

// ---------------------------------------------------------------------------
// k_vt_fill
// ---------------------------------------------------------------------------
// The cells of a k_canon warp to their vertices' VT rows, in the warp's order
// by vertex: 32 words are some ten runs, not 32 words of their own.  229 us at 128^3 cubes,
// vertex ids permuted (275 with a store and an offset's gather a pair), bound by
// its gathers' and stores' latency; loading the vertices before their number is
// known, 264.
__global__ void __launch_bounds__(kCanonThreads)
k_vt_fill(int64_t T, const int64_t *__restrict__ vt_off, const VtOrder vo, int *__restrict__ vt)
{
    griddep_wait();
    __shared__ long long s_to[kCanonWarps][kCanonPairs];   // of a vertex: the warp's part of its
                                                           // row, less its place
    __shared__ unsigned char s_cell[kCanonWarps][kCanonPairs];
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const int64_t c = (int64_t)blockIdx.x * kCanonThreads + threadIdx.x, tile = c >> 5;
    if (32 * tile >= T) return;   // warp-uniform
    const unsigned place = c < T ? vo.place[c] : ~0u;
    const uint4 h = __ldg(vo.head + tile);
    const int2 *verts = vo.verts + tile * kCanonPairs;
    const int n = __popc(h.x) + __popc(h.y) + __popc(h.z) + __popc(h.w);
    for (int i = lane; i < n; i += 32) {
        const int2 v = __ldg(verts + i);
        s_to[wp][i] = vt_off[v.x] + v.y;
    }
    const bool ok = place != ~0u;
    if (ok) {
#pragma unroll
        for (int k = 0; k < 4; k++) s_cell[wp][place >> (8 * k) & 0xffu] = (unsigned char)lane;
    }
    const int pairs = 4 * __popc(__ballot_sync(kFull, ok));
    __syncwarp();
    int before = -1;
#pragma unroll
    for (int w = 0; w < 4; w++) {
        const unsigned bits = w == 0 ? h.x : (w == 1 ? h.y : (w == 2 ? h.z : h.w));
        const int at = 32 * w + lane;
        const int k = before + __popc(bits & (0xffffffffu >> (31 - lane)));
        if (at < pairs) vt[s_to[wp][k] + at] = (int)(32 * tile) + s_cell[wp][at];
        before += __popc(bits);
    }
}

// ---------------------------------------------------------------------------
// Cell, face and edge fills
// ---------------------------------------------------------------------------
__device__ __forceinline__ int rank_of(const uint2 *__restrict__ rk, long long p)
{
    const uint2 w = __ldg(rk + (p >> 5));
    return (int)w.y + __popc(w.x & ((1u << (p & 31)) - 1u));
}

// Face-sharing TT rows at offset 4c - (boundary faces in cells before c),
// since a cell's TT row holds one entry per interior face (the cell across
// each face from FT, sorted); the closing offsets of TT and FF.
__global__ void __launch_bounds__(256)
k_cell_tt(int64_t T, int64_t F, const int *__restrict__ tf, const int *__restrict__ ft,
          const uint2 *__restrict__ brank, int64_t *__restrict__ tt_off, int *__restrict__ tt,
          int64_t *__restrict__ ff_off)
{
    griddep_wait();
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= T) return;
    if (c == T - 1) {
        const int64_t nb = rank_of(brank, 4 * T);
        if (tt_off) tt_off[T] = 4 * T - nb;
        if (ff_off) ff_off[F] = 3 * (2 * F - nb);
    }
    if (!tt) return;
    const int4 f4 = reinterpret_cast<const int4 *>(tf)[c];
    int nbr[4];
    int n = 0;
#pragma unroll
    for (int col = 0; col < 4; col++) {
        const int2 cells = reinterpret_cast<const int2 *>(ft)[get4(f4, col)];
        const int o = (cells.x == (int)c) ? cells.y : cells.x;
        nbr[col] = o >= 0 ? o : INT_MAX;   // no cell across a boundary face
        n += o >= 0;
    }
    // a sorting network (no data-dependent loops); the missing neighbours
    // sort last
    cswap(nbr[0], nbr[1]);
    cswap(nbr[2], nbr[3]);
    cswap(nbr[0], nbr[2]);
    cswap(nbr[1], nbr[3]);
    cswap(nbr[1], nbr[2]);
    const int64_t off = 4 * c - rank_of(brank, 4 * c);
    tt_off[c] = off;
    int *row = tt + off;
#pragma unroll
    for (int i = 0; i < 4; i++)
        if (i < n) row[i] = nbr[i];
}

// Thread per face f (consecutive threads write consecutive rows): its first
// cell c (FT[f][0]) and its column in c's TF row give the face's occurrence
// slot q = 4c + column and its slots in c (all but 3 - column); FE from c's TE
// row, the FF offset 3 * (2f - boundary faces before f, counted over
// occurrence slots up to q) and the FF row (the faces of both cells, f itself
// (once in each row) and a missing second cell as INT_MAX, sorted by a
// 19-comparator network: the first 6 (interior) or 3 (boundary) are the row).
__global__ void __launch_bounds__(256)
k_face_fill(const int *__restrict__ ft, const int *__restrict__ tf, const int *__restrict__ te,
            const uint2 *__restrict__ brank, int64_t F, int *__restrict__ fe,
            int64_t *__restrict__ ff_off, int *__restrict__ ff)
{
    griddep_wait();
    const int64_t f = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= F) return;
    const int2 cells = reinterpret_cast<const int2 *>(ft)[f];
    const int4 w0 = reinterpret_cast<const int4 *>(tf)[cells.x];
    const int col = w0.x == (int)f ? 0 : (w0.y == (int)f ? 1 : (w0.z == (int)f ? 2 : 3));
    if (fe) {
        // the face's slots in its first cell: all but 3 - col
        const int omit = 3 - col;
        const int s0 = omit == 0 ? 1 : 0, s1 = omit <= 1 ? 2 : 1, s2 = omit <= 2 ? 3 : 2;
        const int *row = te + 6LL * cells.x;
        fe[3 * f] = row[pair_slot(s0, s1)];
        fe[3 * f + 1] = row[pair_slot(s0, s2)];
        fe[3 * f + 2] = row[pair_slot(s1, s2)];
    }
    if (!ff) return;
    const int64_t off = 3 * (2 * f - rank_of(brank, 4LL * cells.x + col));
    ff_off[f] = off;
    const int4 w1 = cells.y >= 0 ? reinterpret_cast<const int4 *>(tf)[cells.y]
                                 : make_int4((int)f, (int)f, (int)f, (int)f);
    int r[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
    for (int k = 0; k < 8; k++)
        if (r[k] == (int)f) r[k] = INT_MAX;
    cswap(r[0], r[2]); cswap(r[1], r[3]); cswap(r[4], r[6]); cswap(r[5], r[7]);
    cswap(r[0], r[4]); cswap(r[1], r[5]); cswap(r[2], r[6]); cswap(r[3], r[7]);
    cswap(r[0], r[1]); cswap(r[2], r[3]); cswap(r[4], r[5]); cswap(r[6], r[7]);
    cswap(r[2], r[4]); cswap(r[3], r[5]);
    cswap(r[1], r[4]); cswap(r[3], r[6]);
    cswap(r[1], r[2]); cswap(r[3], r[4]); cswap(r[5], r[6]);
    const int n = cells.y >= 0 ? 6 : 3;
    int *row = ff + off;
#pragma unroll
    for (int i = 0; i < 6; i++)
        if (i < n) row[i] = r[i];
}

// EE: an edge (a, b)'s row is the merge of the sorted incident-edge rows of a
// and b without the edge itself, which is in both (they share nothing else).
// A warp takes 32 consecutive edges, a lane each: both rows are loaded into
// registers eight entries at a time (padded to whole sectors with ~0), a's
// ascending and b's descending around ~0s form one bitonic sequence, and one
// bitonic merge in registers sorts it.  The warp's rows are contiguous in EE:
// they pass through shared memory and go out as whole lines.  Bound by the load / store pipe (80%; a lane's two rows are lines
// of their own, the entries reach shared memory a word at a time).  Four lanes
// to an edge instead, whose entries went out in 16-byte pieces, sent 11
// requests to L2 an edge (0.8 a clock and SM, what gets through; now 4) and 33
// warp instructions (19): 92 -> 64 us at 64^3, 135 -> 93 us beside other kernels
// on the 64^3 coned mesh, whose rows pass 16.  Without bank conflicts of rows of
// one length (rows below 16) and with eleven blocks of these to an SM (20 bytes of
// spills a thread): 545 -> 533 us at 128^3 beside other kernels.  A warp with
// longer ends: the short rows a lane each, stored as they are, the others by the
// whole warp (all of them so: 294 us instead of 152 on 200,000 Delaunay vertices).
constexpr int kEeThreads = 128;
constexpr int kEeWarps = kEeThreads / 32;
// words that a warp's rows come to, of ends of at most N edges
constexpr int ee_stage(int n) { return 32 * (2 * n - 2) + 4; }

template <int P>
__device__ __forceinline__ void bitonic_merge(unsigned (&x)[P])
{
#pragma unroll
    for (int stride = P / 2; stride >= 1; stride >>= 1) {
#pragma unroll
        for (int i = 0; i < P; i++) {
            if (i & stride) continue;
            const unsigned lo = min(x[i], x[i + stride]);
            x[i + stride] = max(x[i], x[i + stride]);
            x[i] = lo;
        }
    }
}

// One edge a lane, rows of at most N entries; a lane's n words of EE (from o;
// the lanes' rows follow one another) through `stage`, or (APART: some lanes have
// no part in it) each lane's own stored by itself.  P: the power of two at or
// above 2 N; a, b: the rows' first 16 words.
template <int N, int P, bool APART = false>
__device__ __forceinline__ void ee_merge_lanes(const unsigned (&a)[16], const unsigned (&b)[16],
                                               const unsigned *__restrict__ ra,
                                               const unsigned *__restrict__ rb, unsigned e, int64_t o,
                                               int n, unsigned *stage, int *__restrict__ ee)
{
    unsigned x[P];
#pragma unroll
    for (int i = N; i < P - N; i++) x[i] = ~0u;
#pragma unroll
    for (int i = 0; i < 16; i++) {
        x[i] = a[i];
        x[P - 1 - i] = b[i];
    }
#pragma unroll
    for (int k = 16; k < N; k += 8) {
        unsigned t[8], u[8];
#pragma unroll
        for (int i = 0; i < 8; i++) t[i] = u[i] = ~0u;
        if (a[15] != ~0u) load8(ra + k, t);
        if (b[15] != ~0u) load8(rb + k, u);
#pragma unroll
        for (int i = 0; i < 8; i++) {
            x[k + i] = t[i];
            x[P - 1 - (k + i)] = u[i];
        }
    }
    bitonic_merge<P>(x);
    if constexpr (APART) {
#pragma unroll
        for (int i = 0; i < 2 * N; i++)
            if (i < n + 2 && x[i] != e) ee[o + (x[i] > e ? i - 2 : i)] = (int)x[i];
        return;
    }
    const int lane = threadIdx.x & 31;
    const int64_t o0 = __shfl_sync(kFull, o, 0);
    const int shift = (int)(o0 & 3);   // word i of the stage is word i of the line o0 is in
    const int at = shift + (int)(o - o0);
    // sorted: an entry above e follows both copies of e
    if constexpr (N == 16) {
        // two by two, the upper half of the lanes the second one first: short
        // rows are often of one even length, which puts lanes l and l + 16 on
        // one bank (the longer ones' lengths vary: no gain there, 20 us lost on
        // the 64^3 coned mesh)
        const int late = lane >> 4;
        unsigned *row = stage + at + late;
#pragma unroll
        for (int i = 0; i < 2 * N - 2; i += 2) {
            const unsigned u = x[i] >= e ? x[i + 2] : x[i], w = x[i + 1] >= e ? x[i + 3] : x[i + 1];
            if (i + late < n) row[i] = late ? w : u;
            if (i + 1 - late < n) row[i + 1 - 2 * late] = late ? u : w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < 2 * N; i++)
            if (i < n + 2 && x[i] != e) stage[at + (x[i] > e ? i - 2 : i)] = x[i];
    }
    __syncwarp();
    const int end = __reduce_max_sync(kFull, n >= 0 ? at + n : 0);
    int *line = ee + (o0 - shift);
    for (int i = 4 * lane; i < end; i += 128) {
        const uint4 w = *reinterpret_cast<const uint4 *>(stage + i);
        if (i >= shift && i + 4 <= end) {
            *reinterpret_cast<uint4 *>(line + i) = w;
        } else {
            const unsigned q[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
            for (int t = 0; t < 4; t++)
                if (i + t >= shift && i + t < end) line[i + t] = (int)q[t];
        }
    }
}

// An edge by the whole warp: the same merge over 32 * R positions (lane l holds
// positions l + 32 r), for rows of at most 16 R entries; wa, wb: the rows' words,
// padding included, n: the entries written.
template <int R>
__device__ __forceinline__ void ee_merge_warp_r(const unsigned *__restrict__ ra, int wa,
                                                const unsigned *__restrict__ rb, int wb, int n, unsigned e,
                                                int *__restrict__ out, int lane)
{
    constexpr int P = 32 * R;
    unsigned x[R];
#pragma unroll
    for (int r = 0; r < R; r++) {
        const int p = lane + 32 * r;
        const int j = P - 1 - p;
        x[r] = p < P / 2 ? (p < wa ? __ldg(ra + p) : ~0u) : (j < wb ? __ldg(rb + j) : ~0u);
    }
    // strides >= 32: between registers
#pragma unroll
    for (int sr = R / 2; sr >= 1; sr >>= 1) {
#pragma unroll
        for (int r = 0; r < R; r++) {
            if (r & sr) continue;
            const unsigned lo = min(x[r], x[r + sr]), hi = max(x[r], x[r + sr]);
            x[r] = lo;
            x[r + sr] = hi;
        }
    }
    // strides 16 .. 1: between lanes
#pragma unroll
    for (int sl = 16; sl >= 1; sl >>= 1) {
        const bool upper = lane & sl;
#pragma unroll
        for (int r = 0; r < R; r++) {
            const unsigned y = __shfl_xor_sync(kFull, x[r], sl);
            x[r] = upper ? max(x[r], y) : min(x[r], y);
        }
    }
    // (the two copies of e are at adjacent positions)
#pragma unroll
    for (int r = 0; r < R; r++) {
        const int p = lane + 32 * r;
        if (p < n + 2 && x[r] != e) out[p - (x[r] > e ? 2 : 0)] = (int)x[r];
    }
}
// eid: each vertex's incident edges, ascending, from word eid_off[v] on, padded
// with ~0 to 16 words, or beyond those to a multiple of eight that leaves a
// ~0 at the end (so that a row's sixteenth word tells whether it goes on).
// ROWS: 16 or 24 when every row is shorter than that (fewer registers), else 0.
template <int ROWS>
__global__ void __launch_bounds__(kEeThreads, ROWS == 16 ? 11 : 5)
k_ee_fill(const int2 *__restrict__ ev, int64_t E, const int64_t *__restrict__ eid_off,
          const unsigned *__restrict__ eid, const int64_t *__restrict__ ee_off, int *__restrict__ ee)
{
    griddep_wait();
    __shared__ __align__(16) unsigned s_stage[kEeWarps][ee_stage(ROWS == 16 ? 16 : 24)];
    const int lane = threadIdx.x & 31;
    const int64_t e0 = ((int64_t)blockIdx.x * kEeWarps + (threadIdx.x >> 5)) * 32;
    if (e0 >= E) return;  // warp-uniform
    const int64_t e = e0 + lane;
    int64_t o = 0;
    const unsigned *ra = eid, *rb = eid;
    int n = -2;   // no edge
    unsigned a[16], b[16];
#pragma unroll
    for (int i = 0; i < 16; i++) a[i] = b[i] = ~0u;
    if (e < E) {
        const int2 ab = __ldg(ev + e);
        o = __ldg(ee_off + e);
        n = (int)(__ldg(ee_off + e + 1) - o);
        ra += __ldg(eid_off + ab.x);
        rb += __ldg(eid_off + ab.y);
        load8(ra, reinterpret_cast<unsigned(&)[8]>(a[0]));
        load8(ra + 8, reinterpret_cast<unsigned(&)[8]>(a[8]));
        load8(rb, reinterpret_cast<unsigned(&)[8]>(b[0]));
        load8(rb + 8, reinterpret_cast<unsigned(&)[8]>(b[8]));
    }
    unsigned *stage = s_stage[threadIdx.x >> 5];
    // a row of 16 or more
    const bool more = ROWS != 16 && (a[15] != ~0u || b[15] != ~0u);
    if (ROWS == 16 || !__any_sync(kFull, more)) {
        ee_merge_lanes<16, 32>(a, b, ra, rb, (unsigned)e, o, n, stage, ee);
        return;
    }
    if constexpr (ROWS == 16) return;
    bool longer = false;   // of 24 or more
    if (ROWS == 0 && a[15] != ~0u) longer |= __ldg(ra + 23) != ~0u;
    if (ROWS == 0 && b[15] != ~0u) longer |= __ldg(rb + 23) != ~0u;
    if (ROWS == 24 || !__any_sync(kFull, longer)) {
        ee_merge_lanes<24, 64>(a, b, ra, rb, (unsigned)e, o, n, stage, ee);
        return;
    }
    if constexpr (ROWS != 0) return;
    // the others a lane each all the same, those by the whole warp (but for rows
    // of more than kMaxDeg entries: k_ee_heavy's)
    ee_merge_lanes<24, 64, true>(a, b, ra, rb, (unsigned)e, o, longer ? -2 : n, nullptr, ee);
    int wa = 0, wb = 0;
    if (longer) {
        const int2 ab = __ldg(ev + e);
        wa = (int)(__ldg(eid_off + ab.x + 1) - (ra - eid));
        wb = (int)(__ldg(eid_off + ab.y + 1) - (rb - eid));
        // a row of kMaxDeg entries has the words of the few after it
        constexpr int kLast = (kMaxDeg + 8) & ~7;
        if (wa > kLast || wb > kLast || (wa == kLast && __ldg(ra + kMaxDeg) != ~0u) ||
            (wb == kLast && __ldg(rb + kMaxDeg) != ~0u))
            longer = false;
    }
    for (unsigned by_warp = __ballot_sync(kFull, longer); by_warp; by_warp &= by_warp - 1) {
        const int j = __ffs((int)by_warp) - 1;
        const unsigned *pa = (const unsigned *)__shfl_sync(kFull, (unsigned long long)ra, j);
        const unsigned *pb = (const unsigned *)__shfl_sync(kFull, (unsigned long long)rb, j);
        const int ja = __shfl_sync(kFull, wa, j), jb = __shfl_sync(kFull, wb, j), jn = __shfl_sync(kFull, n, j);
        int *out = ee + __shfl_sync(kFull, o, j);
        if (max(ja, jb) <= 32) ee_merge_warp_r<2>(pa, ja, pb, jb, jn, (unsigned)(e0 + j), out, lane);
        else ee_merge_warp_r<4>(pa, ja, pb, jb, jn, (unsigned)(e0 + j), out, lane);
    }
}

// Vertex-sharing TT: the union of the VT rows of the cell's four vertices,
// minus the cell itself, by a four-way merge of sorted rows, a cell to a lane.
// A merge reads a word or two per entry it writes; out of and into global
// memory each of them is a cache line of its own for every lane (8,000 of the
// load / store pipe's cycles a warp, which bounded the pass).  So a warp first
// copies its cells' rows into shared memory, a row once (a table of the
// vertices: 32 cells of a grid name some 28), an INT_MAX after each, and the
// filling pass collects the warp's rows of TT, which are contiguous, there and
// writes them out as whole lines; where those do not fit, each lane stores its
// own row as it merges.  Warps whose VT rows do not fit (cells in no order,
// vertices in very many cells) leave their cells to k_tt_vertex_far, which
// merges in global memory with a full SM of warps and the rows' heads in
// registers (64^3 cubes, cells scattered: 0.81 ms a pass; 5.6 here, with the
// twelve warps an SM that the stage leaves).  On 40^3 cubes, a tenth coned, ids
// permuted (0.42 M cells, 70 entries each): 145 us for the two passes (400
// merging in global memory throughout), bounded by the shared-memory merges
// (load / store pipe 67 % busy counting; filling, four blocks to an SM by what
// they collect).
constexpr int kTtWarps = 2;
constexpr int kTtLists = 1536;    // words of rows a warp keeps
constexpr int kTtTable = 256;     // twice the vertices 32 cells can name
constexpr int kTtOut = 2560;      // entries of TT it collects (70 a cell in a grid)
struct TtStage {
    int list[kTtLists];
    int key[kTtTable], off[kTtTable];
    unsigned char row[kTtTable / 2];   // the table's slots in use
    int n;
};
// the cell's merge in global memory
template <bool FILL>
__device__ __forceinline__ void tt_merge_far(const int4 w, int c, const int64_t *__restrict__ vt_off,
                                             const int *__restrict__ vt, int *cnt, int *out)
{
    int pos[4], stop[4], h[4];   // VT has 4T entries: below 2^31
#pragma unroll
    for (int k = 0; k < 4; k++) {
        pos[k] = (int)vt_off[get4(w, k)];
        stop[k] = (int)vt_off[get4(w, k) + 1];
        h[k] = pos[k] < stop[k] ? vt[pos[k]] : INT_MAX;
    }
    int n = 0;
    while (true) {
        const int m = min(min(h[0], h[1]), min(h[2], h[3]));
        if (m == INT_MAX) break;
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (h[k] == m) h[k] = ++pos[k] < stop[k] ? vt[pos[k]] : INT_MAX;
        if (m != c) {
            if (FILL) out[n] = m;
            n++;
        }
    }
    if (!FILL) *cnt = n;
}
template <bool FILL>
__device__ __noinline__ void tt_merge_global(const int4 w, int c, const int64_t *__restrict__ vt_off,
                                             const int *__restrict__ vt, int *cnt, int *out)
{
    tt_merge_far<FILL>(w, c, vt_off, vt, cnt, out);
}

// a warp per 32 cells that k_tt_vertex listed (far null: of all cells)
template <bool FILL>
__global__ void __launch_bounds__(256)
k_tt_vertex_far(const int4 *__restrict__ tvs, int64_t T, const int64_t *__restrict__ vt_off,
                const int *__restrict__ vt, const int *__restrict__ far, const int *__restrict__ n_far,
                int *__restrict__ cnt, const int64_t *__restrict__ tt_off, int *__restrict__ tt)
{
    griddep_wait();
    const int64_t n = far ? *n_far : (T + 31) / 32;
    for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n;
         i += (int64_t)gridDim.x * (blockDim.x >> 5)) {
        const int64_t c = 32 * (far ? far[i] : i) + (threadIdx.x & 31);
        if (c < T)
            tt_merge_far<FILL>(tvs[c], (int)c, vt_off, vt, FILL ? nullptr : cnt + c,
                               FILL ? tt + tt_off[c] : nullptr);
    }
}

// far, n_far: where the warps whose rows do not fit are listed; far null: they
// merge in global memory themselves (n_far null) or are left out
template <bool FILL>
__global__ void __launch_bounds__(32 * kTtWarps)
k_tt_vertex(const int4 *__restrict__ tvs, int64_t T, const int64_t *__restrict__ vt_off,
            const int *__restrict__ vt, int *__restrict__ far, int *__restrict__ n_far, int *__restrict__ cnt,
            const int64_t *__restrict__ tt_off, int *__restrict__ tt)
{
    griddep_wait();
    __shared__ TtStage s_stage[kTtWarps];
    __shared__ __align__(16) int s_out[FILL ? kTtWarps : 1][FILL ? kTtOut : 4];
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const int64_t c0 = ((int64_t)blockIdx.x * kTtWarps + wp) * 32;
    if (c0 >= T) return;   // warp-uniform
    TtStage &S = s_stage[wp];
    const int64_t c = c0 + lane;
    for (int i = lane; i < kTtTable; i += 32) S.key[i] = -1;
    if (lane == 0) S.n = 0;
    __syncwarp();
    int4 w = make_int4(0, 0, 0, 0);
    int slot[4] = {0, 0, 0, 0};
    if (c < T) {
        w = tvs[c];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int v = get4(w, k);
            unsigned h = ((unsigned)v * 0x9E3779B1u) >> 24;
            for (int probe = 0; probe < kTtTable; probe++) {   // never full
                const int old = atomicCAS(&S.key[h], -1, v);
                if (old == -1) S.row[atomicAdd(&S.n, 1)] = (unsigned char)h;
                if (old == -1 || old == v) break;
                h = (h + 1) & (kTtTable - 1);
            }
            slot[k] = (int)h;
        }
    }
    int64_t o0 = 0, o = 0;
    bool collect = false;   // the warp's rows of TT fit what it collects
    if (FILL) {
        o0 = tt_off[c0];
        o = tt_off[min(c, T)];
        collect = tt_off[min(c0 + 32, T)] - o0 + 4 <= kTtOut;
    }
    __syncwarp();
    const int rows = S.n;
    bool fits = true;
    if (rows > 32) {   // before any is copied
        int words = 0;
        for (int r = lane; r < rows; r += 32) {
            const int v = S.key[S.row[r]];
            words += 1 + (int)min(vt_off[v + 1] - vt_off[v], (int64_t)kTtLists);
        }
        fits = __reduce_add_sync(kFull, words) <= kTtLists;
    }
    // the rows, a lane each, then eight lanes to each of four to copy them
    int total = 0;
    for (int r0 = 0; r0 < rows && fits; r0 += 32) {
        int64_t src = 0;
        int len = 0;
        if (r0 + lane < rows) {
            const int v = S.key[S.row[r0 + lane]];
            src = vt_off[v];
            len = (int)min(vt_off[v + 1] - src, (int64_t)kTtLists);
        }
        const int words = r0 + lane < rows ? len + 1 : 0;
        int end = words;
#pragma unroll
        for (int q = 1; q < 32; q <<= 1) {
            const int y = __shfl_up_sync(kFull, end, q);
            if (lane >= q) end += y;
        }
        const int at = total + end - words;
        total += __shfl_sync(kFull, end, 31);
        fits = total <= kTtLists;   // warp-uniform
        if (!fits) break;
        if (words) {
            S.off[S.row[r0 + lane]] = at;
            S.list[at + len] = INT_MAX;
        }
        for (int j = 0; j < min(rows - r0, 32); j += 4) {
            const int q = j + (lane >> 3);
            const int64_t r = __shfl_sync(kFull, src, q);
            const int n = __shfl_sync(kFull, len, q), to = __shfl_sync(kFull, at, q);
            for (int i = lane & 7; i < n; i += 8) S.list[to + i] = __ldg(vt + r + i);
        }
    }
    if (!fits) {   // warp-uniform
        if (far) {
            if (lane == 0) far[atomicAdd(n_far, 1)] = (int)(c0 >> 5);
        } else if (!n_far && c < T) {
            tt_merge_global<FILL>(w, (int)c, vt_off, vt, FILL ? nullptr : cnt + c, FILL ? tt + o : nullptr);
        }
        return;
    }
    __syncwarp();
    int p[4], h[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        p[k] = c < T ? S.off[slot[k]] : 0;
        h[k] = c < T ? S.list[p[k]] : INT_MAX;
    }
    const int shift = (int)(o0 & 3);   // word i collected is word i of the line o0 is in
    int n = 0;
    auto merge = [&](int *out) {
        while (true) {
            const int m = min(min(h[0], h[1]), min(h[2], h[3]));
            if (m == INT_MAX) break;
#pragma unroll
            for (int k = 0; k < 4; k++)
                if (h[k] == m) h[k] = S.list[++p[k]];
            if (m != (int)c) {
                if (FILL) out[n] = m;
                n++;
            }
        }
    };
    if (!FILL) {
        merge(nullptr);
        if (c < T) cnt[c] = n;
        return;
    }
    if (!collect) {   // warp-uniform
        merge(tt + o);
        return;
    }
    merge(s_out[wp] + shift + (int)(o - o0));
    __syncwarp();
    const int stop = __reduce_max_sync(kFull, c < T ? shift + (int)(o - o0) + n : 0);
    int *line = tt + (o0 - shift);
    for (int i = 4 * lane; i < stop; i += 128) {
        const int4 q = *reinterpret_cast<const int4 *>(s_out[wp] + i);
        if (i >= shift && i + 4 <= stop) {
            *reinterpret_cast<int4 *>(line + i) = q;
        } else {
#pragma unroll
            for (int t = 0; t < 4; t++)
                if (i + t >= shift && i + t < stop) line[i + t] = get4(q, t);
        }
    }
}

// int32 -> int64 (the reference's vtkIdType) copy
__global__ void __launch_bounds__(256)
k_widen(const int *__restrict__ src, long long *__restrict__ dst, int64_t n)
{
    griddep_wait();
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        dst[i] = src[i];
}

// int64 -> int32 copy (CSR offsets of a relation below 2^31 entries)
__global__ void __launch_bounds__(256)
k_narrow(const int64_t *__restrict__ src, int *__restrict__ dst, int64_t n)
{
    griddep_wait();
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        dst[i] = (int)src[i];
}

__global__ void __launch_bounds__(256) k_narrow_multi(NarrowJobs j)
{
    griddep_wait();
    const int64_t total = j.start[j.n];
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (int64_t)gridDim.x * blockDim.x) {
        int k = 0;
        while (i >= j.start[k + 1]) k++;
        j.dst[i] = (int)j.src[k][i - j.start[k]];
    }
}

// CSR rows -> the reference's padded device_VV layout: row v at v * width,
// unused slots -1, plus the row lengths
__global__ void __launch_bounds__(256)
k_pad_rows(const int64_t *__restrict__ off, const int *__restrict__ ent, int64_t rows, int width,
           long long *__restrict__ out, unsigned *__restrict__ counts)
{
    griddep_wait();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= rows * width) return;
    const int64_t r = i / width;
    const int k = (int)(i - r * width);
    const int64_t b = off[r];
    const int n = (int)(off[r + 1] - b);
    out[i] = k < n ? (long long)ent[b + k] : -1ll;
    if (k == 0 && counts) counts[r] = (unsigned)n;
}

inline unsigned blocks_for(int64_t n, int threads)
{
    return (unsigned)((n + threads - 1) / threads);
}

}  // namespace

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
void launch_widen(const int32_t *src, int64_t *dst, int64_t n, cudaStream_t s)
{
    if (n == 0) return;
    Launch L("k_widen", s);
    const int64_t blocks = std::min<int64_t>((n + 255) / 256, 152 * 32);
    launch_pdl(k_widen, (unsigned)blocks, 256, 0, s, src, reinterpret_cast<long long *>(dst), n);
}

void launch_narrow(const int64_t *src, int32_t *dst, int64_t n, cudaStream_t s)
{
    if (n == 0) return;
    Launch L("k_narrow", s);
    const int64_t blocks = std::min<int64_t>((n + 255) / 256, 152 * 32);
    launch_pdl(k_narrow, (unsigned)blocks, 256, 0, s, src, dst, n);
}

void launch_narrow_multi(const NarrowJobs &j, cudaStream_t s)
{
    const int64_t n = j.start[j.n];
    if (n == 0) return;
    Launch L("k_narrow_multi", s);
    const int64_t blocks = std::min<int64_t>((n + 255) / 256, 152 * 32);
    launch_pdl(k_narrow_multi, (unsigned)blocks, 256, 0, s, j);
}

void launch_pad_rows(const int64_t *off, const int32_t *ent, int64_t rows, int width,
                     int64_t *out, uint32_t *counts, cudaStream_t s)
{
    if (rows == 0 || width == 0) return;
    Launch L("k_pad_rows", s);
    launch_pdl(k_pad_rows, blocks_for(rows * width, 256), 256, 0, s, off, ent, rows, width,
                                                            reinterpret_cast<long long *>(out), counts);
}

// copies the status and the sizes to mapped host memory, then resets the
// status for the next call on the mesh (the host has consumed it)
__global__ void k_publish(PublishArgs a)
{
    griddep_wait();
    if (threadIdx.x != 0) return;
    *a.h_st = *a.st;
    for (int i = 0; i < a.n; i++)
        a.h_sz[i] = a.wide[i] ? *(const int64_t *)a.src[i] : (int64_t) * (const int32_t *)a.src[i];
    __threadfence_system();
    a.st->flags = 0;
    a.st->bad_cell = 0;
    a.st->bad_vertex = 0;
    a.st->max_deg = 0;
}

void launch_publish(const PublishArgs &a, cudaStream_t s)
{
    Launch L("k_publish", s);
    launch_pdl(k_publish, 1, 32, 0, s, a);
}

int64_t canon_tiles(int64_t T) { return (T + 31) / 32; }
int64_t canon_pairs() { return kCanonPairs; }

void launch_canon(const int32_t *tv_in, int64_t T, int64_t V, int4 *tvs, int32_t *deg_t,
                  const VtOrder &vo, DevStatus *st, cudaStream_t s)
{
    if (T == 0) return;
    const int aligned = ((uintptr_t)tv_in & 15) == 0;
    {
        Launch L("k_canon", s);
        launch_pdl(k_canon, blocks_for(T, kCanonThreads), kCanonThreads, 0, s, tv_in, T, (int)V, tvs,
                   deg_t, vo, st, aligned);
    }
}

void launch_vt_fill(int64_t T, const int64_t *vt_off, const VtOrder &vo, int32_t *vt, cudaStream_t s)
{
    if (T == 0) return;
    {
        Launch L("k_vt_fill", s);
        launch_pdl(k_vt_fill, blocks_for(T, kCanonThreads), kCanonThreads, 0, s, T, vt_off, vo, vt);
    }
}

void launch_cell_tt(int64_t T, int64_t F, const int32_t *tf, const int32_t *ft, const uint2 *brank,
                    int64_t *tt_off, int32_t *tt, int64_t *ff_off, cudaStream_t s)
{
    if (T == 0) return;
    {
        Launch L("k_cell_tt", s);
        launch_pdl(k_cell_tt, blocks_for(T, 256), 256, 0, s, T, F, tf, ft, brank, tt_off, tt,
                   ff_off);
    }
}

void launch_face_fill(const int32_t *ft, const int32_t *tf, const int32_t *te, const uint2 *brank,
                      int64_t F, int32_t *fe, int64_t *ff_off, int32_t *ff, cudaStream_t s)
{
    if (F == 0) return;
    {
        Launch L("k_face_fill", s);
        launch_pdl(k_face_fill, blocks_for(F, 256), 256, 0, s, ft, tf, te, brank, F, fe, ff_off, ff);
    }
}

void launch_ee_fill(const int32_t *ev, int64_t E, const int64_t *eid_off, const uint32_t *eid,
                    const int64_t *ee_off, int32_t *ee, int max_deg, cudaStream_t s)
{
    if (E == 0) return;
    Launch L("k_ee_fill", s);
    launch_pdl(max_deg < 16 ? k_ee_fill<16> : (max_deg < 24 ? k_ee_fill<24> : k_ee_fill<0>),
               blocks_for(E, kEeThreads), kEeThreads, 0, s, reinterpret_cast<const int2 *>(ev), E, eid_off,
               eid, ee_off, ee);
}

// Below kTtFar cells every warp is on the GPU at once whichever kernel has it: no
// list.  With two vertices a cell or more (cells that share little) rows are a
// word or two, and staging them costs more than merging them: k_tt_vertex_far for
// all (1.5M cells that share nothing: 23 us a pass against 249).
constexpr int64_t kTtFar = 1 << 16;
static bool tt_short_rows(int64_t T, int64_t V) { return V >= 2 * T; }
int64_t tt_far_tiles(int64_t T, int64_t V) { return T >= kTtFar && !tt_short_rows(T, V) ? (T + 31) / 32 : 0; }

void launch_tt_vertex_count(const int4 *tvs, int64_t T, int64_t V, const int64_t *vt_off, const int32_t *vt,
                            int32_t *far, int32_t *n_far, int32_t *cnt, cudaStream_t s)
{
    if (T == 0) return;
    if (tt_short_rows(T, V)) {
        Launch L("k_tt_vertex_far", s);
        launch_pdl(k_tt_vertex_far<false>, blocks_for(T, 256), 256, 0, s, tvs, T, vt_off, vt, nullptr, nullptr,
                   cnt, nullptr, nullptr);
        return;
    }
    {
        Launch L("k_tt_vertex", s);
        launch_pdl(k_tt_vertex<false>, blocks_for(T, 32 * kTtWarps), 32 * kTtWarps, 0, s, tvs, T, vt_off, vt,
                   far, n_far, cnt, nullptr, nullptr);
    }
    if (far) {   // (how many there are is known on the device)
        Launch L("k_tt_vertex_far", s);
        launch_pdl(k_tt_vertex_far<false>, (unsigned)std::min<int64_t>((T + 255) / 256, 152 * 8), 256, 0, s,
                   tvs, T, vt_off, vt, (const int *)far, (const int *)n_far, cnt, nullptr, nullptr);
    }
}

void launch_tt_vertex_fill(const int4 *tvs, int64_t T, int64_t V, const int64_t *vt_off, const int32_t *vt,
                           const int32_t *far, int32_t *n_far, int64_t listed, const int64_t *tt_off,
                           int32_t *tt, cudaStream_t s)
{
    if (T == 0) return;
    if (tt_short_rows(T, V)) {
        Launch L("k_tt_vertex_far", s);
        launch_pdl(k_tt_vertex_far<true>, blocks_for(T, 256), 256, 0, s, tvs, T, vt_off, vt, nullptr, nullptr,
                   nullptr, tt_off, tt);
        return;
    }
    if (listed < (T + 31) / 32) {
        Launch L("k_tt_vertex", s);
        launch_pdl(k_tt_vertex<true>, blocks_for(T, 32 * kTtWarps), 32 * kTtWarps, 0, s, tvs, T, vt_off, vt,
                   nullptr, n_far, nullptr, tt_off, tt);
    }
    if (listed > 0) {
        Launch L("k_tt_vertex_far", s);
        launch_pdl(k_tt_vertex_far<true>, blocks_for(32 * listed, 256), 256, 0, s, tvs, T, vt_off, vt, far,
                   (const int *)n_far, nullptr, tt_off, tt);
    }
}

}  // namespace tg
