// tg_internal.h -- declarations shared by the host orchestration (tg_api.cu)
// and the kernel translation units.  Not part of the public ABI.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>
#include <utility>

#include "tetragpu.h"
#include "tg_tuning.h"

namespace tg {

// Device-side status word, written by kernels with atomics, read back by the
// host at the synchronisation points of tg_extract.  All zeros: clean.
struct DevStatus {
    unsigned int flags;
    int bad_cell;      // INT_MAX - the lowest offending cell (note_lowest), 0 if none
    int bad_vertex;    // the same of vertices
    int max_deg;       // largest number of neighbours of a vertex
    int pad[4];
};

enum StatusFlag : unsigned int {
    ST_BAD_ID = 1u,            // vertex id outside [0, n_verts)
    ST_DUP_VERTEX = 2u,        // a cell repeats a vertex
    ST_STAR_OVERFLOW = 8u,     // an edge lies in more cells than the row lengths hold
    ST_NONMANIFOLD_FACE = 16u, // a face lies in more than two cells
    ST_HEAVY_DEG = 64u,        // a vertex has more neighbours than the link masks hold (tg_noalloc.cu)
    ST_SCAN_STALLED = 128u     // a scan tile gave up waiting for the tiles before it
};

// Largest star (cells around one vertex) and neighbourhood handled on the
// fast path: star positions and neighbours are bits of a 64-bit mask.
constexpr int kMaxStar = 64;
constexpr int kMaxDeg = 64;
constexpr int kNarrowDeg = 32;   // the most neighbours of a 32-bit link mask

// VV entries per window of the link-adjacency kernel (tg_crit.cu): its
// window table has n_vv / kAdjWin + 2 entries
constexpr int kAdjWin = TG_ADJ_WIN;
static_assert(kAdjWin >= 64 && kAdjWin <= 4096, "link-adjacency window size");

// ---- scans (tg_scan.cu) ----
enum ScanKind : int {
    SCAN_COUNT_I32 = 0,  // in: int32 counts (+ in2's when given), out: int64 offsets [n + 1]
    SCAN_POPC_RANK = 1,  // in: uint32 bit words, out: uint2 {word, popcount prefix} [n + 1],
                         //     out[n] = {0, total}: rank of bit p = one 8-byte load
    SCAN_ROW_PAD8 = 3,   // in: int64 CSR offsets; SCAN_COUNT_I32 of the lengths of rows in2[i]
                         //     (null: i), rounded up to multiples of eight
    SCAN_EID_WORDS = 4,  // SCAN_COUNT_I32 of eid_words of the counts
    SCAN_DEG_SQUARE = 2  // in: int32 x (+ in2's), out: int64 prefix of x*x [n + 1]; the largest
                         //     x goes to the status word's max_deg
};
struct ScanJob {
    const void *in;
    void *out;
    int64_t n;
    int kind;
    const int32_t *in2;
};
constexpr int kMaxScanJobs = 8;
// Exclusive scans of up to kMaxScanJobs arrays in one launch, over a
// workspace of two buffers of kMaxScanJobs * job_words words (zeroed once when
// made): a scan uses one buffer and zeroes the other for the next scan, so no
// scan needs a memset.  A scan issued on another stream than the last one
// waits for the last one first (event `done`; null: used on one stream only).  A stalled scan sets
// ST_SCAN_STALLED in st.
struct ScanWorkspace {
    unsigned long long *buf = nullptr;   // 2 * kMaxScanJobs * job_words words
    int64_t job_words = 0;               // tile words + ticket of the longest array
    int cur = 0;
    cudaEvent_t done = nullptr;
    cudaStream_t last = nullptr;
    bool used = false;
};
int64_t scan_job_words(int64_t max_n);
void scan_batch(const ScanJob *jobs, int n_jobs, ScanWorkspace &ws, DevStatus *st, cudaStream_t s);
// For another single-pass kernel on the workspace: the buffer to use now
// (kMaxScanJobs * job_words words, zero), the one to zero for the next user;
// scan_ws_end after the launch.
void scan_ws_begin(ScanWorkspace &ws, cudaStream_t s, unsigned long long **cur,
                   unsigned long long **next, int64_t *next_words);
void scan_ws_end(ScanWorkspace &ws, cudaStream_t s);

#ifdef __CUDACC__
__device__ __forceinline__ void note_lowest(int *at, int i) { atomicMax(at, 0x7fffffff - i); }

// Single-pass scan step (decoupled look-back, Merrill and Garland), called by
// one whole warp: publish tile `tile`'s sum in w[tile] (sum << 2 | 1), add
// the published sums of the tiles before it, 32 at a time (lane i reads the
// i-th tile back), until one holds an inclusive prefix (sum << 2 | 2); then
// publish its own inclusive prefix.  Returns the sum of the tiles before it
// (in every lane).  Tiles are numbered in block start order, so the tiles
// waited for are running; after kLookbackPolls polls the wait gives up and
// sets ST_SCAN_STALLED.
constexpr unsigned kLookbackPolls = 1u << 16;
__device__ __forceinline__ long long look_back(unsigned long long *w, long long tile, long long sum,
                                               unsigned *err)
{
    const int lane = threadIdx.x & 31;
    if (tile == 0) {
        if (lane == 0) atomicExch(w, ((unsigned long long)sum << 2) | 2ull);
        return 0;
    }
    if (lane == 0) atomicExch(w + tile, ((unsigned long long)sum << 2) | 1ull);
    long long prefix = 0;
    long long k = tile - 1;   // the window: tiles k - 31 .. k
    unsigned polls = 0;
    while (true) {
        const long long t = k - lane;
        const unsigned long long x =
            t >= 0 ? *reinterpret_cast<volatile unsigned long long *>(w + t) : 0ull;
        const unsigned f = (unsigned)(x & 3ull);
        const unsigned pre = __ballot_sync(0xffffffffu, f == 2);
        const int first = pre ? __ffs(pre) - 1 : 31;   // nearest inclusive prefix, or all
        const unsigned need = first >= 31 ? 0xffffffffu : (2u << first) - 1u;
        if (__ballot_sync(0xffffffffu, f == 0) & need) {   // a tile has not published yet
            if (++polls > kLookbackPolls) {
                if (lane == 0) atomicOr(err, ST_SCAN_STALLED);
                break;
            }
            __nanosleep(32);
            continue;
        }
        long long v = lane <= first ? (long long)(x >> 2) : 0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        prefix += v;
        if (pre) break;
        k -= 32;
    }
    if (lane == 0) atomicExch(w + tile, ((unsigned long long)(prefix + sum) << 2) | 2ull);
    return prefix;
}
#endif

// ---- pipeline kernels (tg_kernels.cu) ----
// Status word and up to 8 sizes (int64, or int32 sign-extended) stored by a
// kernel into device-mapped pinned host memory (no copy engine involved)
struct PublishArgs {
    DevStatus *st;           // reset once copied
    const void *src[8];
    int wide[8];
    int n;
    DevStatus *h_st;
    int64_t *h_sz;
};
void launch_publish(const PublishArgs &a, cudaStream_t s);
void launch_widen(const int32_t *src, int64_t *dst, int64_t n, cudaStream_t s);
void launch_narrow(const int64_t *src, int32_t *dst, int64_t n, cudaStream_t s);
// up to 16 int64 arrays narrowed into one int32 array, back to back
struct NarrowJobs {
    const int64_t *src[16];
    int64_t start[17];   // start[k]: first output element of array k; start[n] = total
    int n;
    int32_t *dst;
};
void launch_narrow_multi(const NarrowJobs &j, cudaStream_t s);
void launch_pad_rows(const int64_t *off, const int32_t *ent, int64_t rows, int width,
                     int64_t *out, uint32_t *counts, cudaStream_t s);
// What k_canon leaves of the (cell, vertex) pairs of each 32 cells for
// k_vt_fill: their order by vertex
struct VtOrder {
    uint32_t *place;   // [T] the cell's four places in it, 8 bits each (all ones: rejected)
    uint4 *head;       // [tiles] a bit per place that begins a vertex
    int2 *verts;       // [tiles x canon_pairs] {vertex, place in its VT row less its place here}
};
int64_t canon_tiles(int64_t T);
int64_t canon_pairs();
// sort each TV row, validate ids, count cells per vertex
void launch_canon(const int32_t *tv_in, int64_t T, int64_t V, int4 *tvs, int32_t *deg_t,
                  const VtOrder &vo, DevStatus *st, cudaStream_t s);
void launch_vt_fill(int64_t T, const int64_t *vt_off, const VtOrder &vo, int32_t *vt, cudaStream_t s);
// Windows of win_size entries over a CSR: win[w] = first row starting at or
// after entry win_size * w (w = 0 .. window_count), win[window_count] = rows.
int64_t window_count(int64_t n_entries, int win_size);
void launch_window_starts(const int64_t *off, int64_t rows, int64_t n_entries, int win_size,
                          int32_t *win, cudaStream_t s);
// sort every VT row (tg_star.cu).  Also marks each vertex's star-order key
// 4 * (lowest cell) + (slot in it) in vflag (4T bits, zeroed by the caller)
// and stores it in vkey[v]; rows with no cells are left alone.  A vertex of
// more than kMaxStar cells takes no key: its bit is set in hflag (V bits,
// zeroed).  heavy_cnt[2] counts the wide light stars.
void launch_vt_sort(const int64_t *vt_off, int32_t *vt, int64_t V, int64_t nvt, const int4 *tvs,
                    uint32_t *vflag, int64_t *vkey, uint32_t *hflag, int32_t *heavy_cnt, cudaStream_t s);
// sort VV rows in place
void launch_vv_sort(const int64_t *vv_off, int64_t V, int64_t nvv, int32_t *vv, cudaStream_t s);
// VV rows and incident-edge rows from inc (EdgePass), sorted; the latter at
// eid_off (SCAN_EID_WORDS), padded with ~0 to eid_words
void launch_inc_sort(const int64_t *vv_off, int64_t V, const int2 *inc, int32_t *vv,
                     const int64_t *eid_off, uint32_t *eid, cudaStream_t s);
// Star processing order (vertices by first cell): vorder[pos] = vertex, pos =
// rank of its key; vpos the way back (heavy vertices after the light ones, by
// id, vertices without cells last).  vrank, hrank: ranks of vflag and hflag.
// heavy_off[i]: where the i-th heavy vertex's entries start among theirs.
// heavy_cnt[0], [1], [3]: heavy vertices, their entries, vertices without cells
// (zeroed by the caller).
void launch_vorder_place(const int64_t *vt_off, int64_t V, const int64_t *vkey, const uint2 *vrank,
                         int64_t nwk, const uint2 *hrank, int32_t *heavy_cnt, int32_t *heavy_off,
                         int32_t *vorder, int32_t *vpos, cudaStream_t s);
// Whether positions or ids keep neighbours together: the lines of 32 vertices
// that the cells of kOrderRuns runs of 32 vertices name, by id added to lines[0]
// and by position to lines[1] (fewer vertices: nothing).
constexpr int kOrderRuns = 128;
void launch_order_lines(int64_t V, const int64_t *vt_off, const int32_t *vt, const int4 *tvs,
                        const int32_t *vorder, const int32_t *vpos, int32_t *lines, cudaStream_t s);

// Star pass (tg_star.cu): the edges and faces of the light vertices.
struct StarPass {
    int64_t n_light;           // the light vertices: vorder[0 .. n_light)
    const int32_t *vorder;
    const int64_t *vt_off;
    const int32_t *vt;
    const int4 *tvs;
    uint32_t *eflag;           // bit per edge occurrence 6c+j (first occurrences)
    uint32_t *fflag;           // bit per face occurrence 4c+k (first occurrences)
    uint32_t *fbnd;            // bit per face occurrence: first and only (boundary face)
    uint8_t *vbnd;             // [V] whether a vertex lies on a boundary face (zeroed)
    int32_t *fnext;            // [4T] a face's second cell (-1: none) at its first
                               // occurrence, or null
    int32_t *deg_own;          // [V] edges a vertex is the low end of (zeroed by the caller)
    int32_t *deg_in;           // [V] edges it is the high end of (zeroed by the caller)
    // a record per edge, in no particular order; those past the room are counted
    // only (and written over the last)
    unsigned rec_last;         // the room less one
    uint2 *rec;                // {first occurrence slot, star positions of the low end's star
                               // holding the edge (the low 32)}
    uint2 *place;              // {place among the low end's own edges, among the high end's others}
    uint32_t *rec_hi;          // the high 32 positions, of edges of wide stars only; null when
                               // there are none
    uint32_t *n_rec;           // the number of records (zeroed by the caller)
    int32_t *wide;             // [V] light vertices of wide stars (more than 31 cells), or null
    uint32_t *n_wide;          // their number (zeroed by the caller)
    DevStatus *st;
};
// launch_star lists the wide stars for launch_star_wide (n_wide: at least
// their number)
void launch_star(const StarPass &p, cudaStream_t s);
void launch_star_wide(const StarPass &p, int64_t n_wide, cudaStream_t s);
// seg_ef[i] = first edge id and seg_ef[n + 1 + i] = first face id of the
// cells from seg_c[i] on (i = 0 .. n; seg_c[n] = T gives the totals)
void launch_seg_ranks(const int64_t *seg_c, int64_t n, const uint2 *erank, const uint2 *frank,
                      int64_t *seg_ef, cudaStream_t s);

// TF, FT and FV (each may be null) from the faces' first occurrences; fnext
// as StarPass leaves it (may be null when neither TF nor FT is wanted)
void launch_cell_faces(int64_t T, const int4 *tvs, const uint2 *frank, const int32_t *fnext,
                       int32_t *tf, int32_t *ft, int32_t *fv, cudaStream_t s);

// Per-edge passes over the star pass's records.
struct EdgePass {
    int64_t E;
    const uint2 *rec;
    const uint2 *place;
    const uint32_t *rec_hi;    // null: no star of more than 32 cells
    const int2 *pairs;         // the heavy stars' pairs (tg_heavy.cu), or null
    const int64_t *vt_off;
    const int32_t *vt;
    const int4 *tvs;
    const uint2 *erank;        // {bits, prefix} per 32 edge occurrences; null when no ids are
                               // wanted (neither inc nor edge)
    const uint2 *frank;        // {bits, prefix} per 32 face occurrences; read for ef
    const uint32_t *fbnd;
    const uint8_t *vbnd;
    const int64_t *vv_off;
    // ids
    int2 *inc;                 // [2E] each vertex's {neighbour, edge id}, unsorted, or null:
    int32_t *vv;               // [2E] VV rows, unsorted
    uint4 *edge;               // [E] by id: the record, {ET | EF << 16, EE} row lengths; or null
    uint32_t *edge_hi;         // [E] rec_hi by id (with rec_hi)
    int count_ef;              // whether the EF lengths are wanted
    // rows (each or null), of the edges by id
    int32_t *ev;               // [2E]
    int32_t *te;               // [6T]
    const int64_t *et_off, *ef_off;
    int32_t *et, *ef;
};
void launch_edge_ids(const EdgePass &p, cudaStream_t s);
void launch_edge_rows(const EdgePass &p, cudaStream_t s);
// ET / EF / EE offsets and EV (each may be null) from the edges by id;
// edge_offsets_words = the tile words it needs in the scan workspace
int64_t edge_offsets_words(int64_t max_edges);
void launch_edge_offsets(const EdgePass &e, int64_t *et_off, int64_t *ef_off, int64_t *ee_off,
                         int32_t *ev, ScanWorkspace &ws, DevStatus *st, cudaStream_t s);

// TT offsets (4c - boundary faces before cell c), TT rows (or null), and the
// closing TT and FF offsets.
void launch_cell_tt(int64_t T, int64_t F, const int32_t *tf, const int32_t *ft, const uint2 *brank,
                    int64_t *tt_off, int32_t *tt, int64_t *ff_off, cudaStream_t s);
// per face (each may be null): FE, FF offsets (but the closing one) and FF
// rows (ff_off and ff together)
void launch_face_fill(const int32_t *ft, const int32_t *tf, const int32_t *te, const uint2 *brank,
                      int64_t F, int32_t *fe, int64_t *ff_off, int32_t *ff, cudaStream_t s);
// EE rows; eid / eid_off: incident-edge rows as launch_inc_sort leaves them,
// max_deg the longest
void launch_ee_fill(const int32_t *ev, int64_t E, const int64_t *eid_off, const uint32_t *eid,
                    const int64_t *ee_off, int32_t *ee, int max_deg, cudaStream_t s);
// Vertex-sharing TT.  far (tt_far_tiles entries, null for none), n_far (zeroed
// by the caller, null with far): the runs of 32 cells listed by the count for the
// kernel that merges in global memory; listed: their number, for the fill.
int64_t tt_far_tiles(int64_t T, int64_t V);
void launch_tt_vertex_count(const int4 *tvs, int64_t T, int64_t V, const int64_t *vt_off, const int32_t *vt,
                            int32_t *far, int32_t *n_far, int32_t *cnt, cudaStream_t s);
void launch_tt_vertex_fill(const int4 *tvs, int64_t T, int64_t V, const int64_t *vt_off, const int32_t *vt,
                           const int32_t *far, int32_t *n_far, int64_t listed, const int64_t *tt_off,
                           int32_t *tt, cudaStream_t s);

// ---- heavy vertices (tg_heavy.cu) ----
// Stars of more than kMaxStar cells: they follow every other vertex with
// cells in the star processing order (positions n_light .. n_light +
// n_heavy - 1), and k_heavy does their share of the star pass.
struct HeavyStars {
    StarPass star;             // n_light, the mesh and the star pass's outputs (rec_hi not null)
    int64_t n_heavy;
    const int32_t *heavy_off;  // where each heavy star's entries start among the heavy entries
    int2 *pairs;               // 3 per heavy star entry: (neighbour, position), sorted here
};
void launch_heavy(const HeavyStars &h, cudaStream_t s);
// EE rows of edges with an endpoint of more than kMaxDeg neighbours
void launch_ee_heavy(const int32_t *ev, int64_t E, const int64_t *vv_off, const int64_t *eid_off,
                     const uint32_t *eid, const int64_t *ee_off, int32_t *ee, cudaStream_t s);
// classes of the vertices in [v0, v0 + nv) with more than kMaxDeg neighbours
// (at most max_listed of them): list (capacity max_listed) and n_list (one
// int, zeroed by the caller) are scratch, scratch holds one int per VV entry
void launch_crit_heavy(const int64_t *vv_off, const int32_t *vv, int64_t v0, int64_t nv,
                       int64_t max_listed, const void *field, int field_type, uint32_t *classes3,
                       int32_t *list, int32_t *n_list, int32_t *scratch, cudaStream_t s);

// critical points (tg_crit.cu)
// The graph of the link adjacency: VV's rows by position, each vertex named by
// its position in `order` (null: its id), entries ascending and padded with -1
// to a multiple of eight; or (not padded) VV itself
struct LinkGraph {
    int64_t V, n_ent;              // n_ent: at least the entries, padding included
    const int64_t *off;
    const int32_t *ent;
    const int32_t *order, *vpos;   // vertex at each position, and back; both null or neither
    void *adj;                     // a mask per entry: 64-bit when wide, else 32-bit
    bool wide;                     // a row holds more than 32 entries (always so if not padded)
    bool padded;
    const int32_t *ids;            // the rows as vertices (small meshes), or null
    int64_t heavy0, n_heavy;       // positions of the heavy stars (with an order)
};
// From this many vertices on a field is put in processing order for its
// classification; the rows of smaller meshes are there as vertices too
constexpr int64_t kOrderField = 1 << 17;
// VV's row lengths by position, and (off their prefix) its rows
// (order and vpos null: in the order of ids; ids, unless null: the rows as
// vertices; win, unless null: the rows' window starts, n_win + 1 of them)
void launch_rows_in_order(const int64_t *vv_off, const int32_t *vv, const int32_t *order,
                          const int32_t *vpos, int64_t V, const int64_t *off, int32_t *ent, int32_t *ids,
                          int32_t *win, int64_t n_win, cudaStream_t s);
// the masks; win: window table of off (launch_window_starts, crit_window())
int crit_window();
// heavy: 0 no row longer than kMaxDeg, 1 such rows get the heavy path
// (masks of their light neighbours computed from the light side), 2 report
// them with ST_HEAVY_DEG (positions are ids)
void launch_crit_adj(const LinkGraph &g, const int32_t *win, DevStatus *st, int heavy, cudaStream_t s);
// classify the vertices [v0, v0 + nv) (all of them, or a range that holds
// every neighbour of its vertices): field and classes3 hold nv values / rows
// from v0; ordered: scratch for V field values, worth having if
// classify_orders_field(nv) (never without an order), or null
bool classify_orders_field(int64_t nv);
void launch_crit_classify(const LinkGraph &g, const void *field, int field_type, void *ordered,
                          int64_t v0, int64_t nv, uint32_t *classes3, cudaStream_t s);

// the message tg_last_error_string returns on this thread
void set_last_error(const char *msg);
// the mesh's VV by position, made if it has none yet (off null when there is no
// memory for it or positions are ids), VV being extracted
tg_status link_rows(tg_mesh *m, cudaStream_t s, LinkGraph *out);
// the stream was given work that reads the mesh's VV or (rows) VV by position:
// what frees them waits for it, whatever the mesh's last stream
tg_status note_reader(tg_mesh *m, cudaStream_t s, bool rows);
// work on the stream is being recorded, not run
bool capturing(cudaStream_t s);
// field values of every vertex by position
void launch_field_in_order(const float *field, const int32_t *order, int64_t V, float *out,
                           cudaStream_t s);
// a temporary from the library's own pool (freed with cudaFreeAsync)
cudaError_t take_temp(size_t bytes, cudaStream_t s, void **out);
// Cell segments of a mesh (the meshes of a batch, tg_batch.cu): seg_c_host
// holds n + 1 cell starts; each extraction then fills n + 1 first edge ids
// followed by n + 1 first face ids (device, read by mesh_segment_ids).
tg_status mesh_set_segments(tg_mesh *m, const int64_t *seg_c_host, int64_t n, cudaStream_t s);
const int64_t *mesh_segment_ids(const tg_mesh *m);
// tg_critical_points restricted to the vertices [v0, v0 + nv), which must
// hold every neighbour of their vertices (a whole mesh of a batch): field
// holds their nv values, classes_out their nv rows
tg_status critical_points_rows(tg_mesh *m, int64_t v0, int64_t nv, const void *field,
                               int field_type, int field_on_device, uint32_t *classes_out,
                               int out_on_device, cudaStream_t s);

// launch accounting and optional CUDA-event timing of one named kernel
void count_launch(int n = 1);
void prof_begin(const char *name, cudaStream_t s);
void prof_end(const char *name, cudaStream_t s);

// RAII wrapper around every launch: counts it and, when the kernel is the
// one selected with tg_profile_kernel, brackets it with CUDA events.
#ifdef __CUDACC__
// Programmatic dependent launch.  Kernels go out with programmatic stream
// serialisation allowed, so a kernel's launch is processed while the kernel
// before it on the stream runs.  Every kernel starts with griddep_wait(),
// which returns once the grids it depends on have completed and their memory
// is visible (at once when it was not launched that way).  The kernels do not
// signal their dependents early: blocks of the next kernel waiting on SMs
// cost the running one more than the earlier start saves.
__device__ __forceinline__ void griddep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Asynchronous global -> shared copies (cp.async): no register holds the
// data in flight, so a kernel can put many dependent-load chains' loads in
// flight at once.  A thread sees its own copies after cp_async_wait(); other
// threads' after that and a barrier.
// eight words from a 32-byte boundary (a sector) in one load
__device__ __forceinline__ void load8(const unsigned *p, unsigned (&x)[8])
{
    asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(x[0]), "=r"(x[1]), "=r"(x[2]), "=r"(x[3]), "=r"(x[4]), "=r"(x[5]), "=r"(x[6]),
                   "=r"(x[7])
                 : "l"(p));
}
__device__ __forceinline__ int pad8(int d) { return (d + 7) & ~7; }
// words of an incident-edge row of d edges: 16, or with a free word at the end
// a multiple of eight
__device__ __forceinline__ int eid_words(int d) { return d < 16 ? 16 : pad8(d + 1); }

template <int B>
__device__ __forceinline__ void cp_async(void *smem, const void *gmem)
{
    static_assert(B == 4 || B == 8 || B == 16, "cp.async copies 4, 8 or 16 bytes");
    const unsigned d = (unsigned)__cvta_generic_to_shared(smem);
    if constexpr (B == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(gmem) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(d), "l"(gmem), "n"(B)
                     : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }
template <typename... KArgs, typename... Args>
inline void launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                       Args &&...args)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}
#endif

struct Launch {
    const char *name;
    cudaStream_t s;
    Launch(const char *n, cudaStream_t st) : name(n), s(st) { prof_begin(name, s); }
    ~Launch()
    {
        prof_end(name, s);
        count_launch();
    }
};

}  // namespace tg
