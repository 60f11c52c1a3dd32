// tg_api.cu -- host orchestration of the relation pipeline behind the C ABI
// declared in include/tetragpu.h.
//
// One tg_mesh owns its device buffers.  Memory comes from the device's
// stream-ordered pool (cudaMallocAsync) with an unlimited release threshold,
// so repeated extractions reuse blocks instead of returning them to the
// driver.  tg_extract synchronises the stream at two points, to learn the
// edge/face/neighbour counts and then the CSR totals that size the outputs;
// everything between those points is asynchronous on the caller's stream.
#include <algorithm>
#include <atomic>
#include <climits>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "tetragpu.h"
#include "tg_internal.h"

namespace tg {
static std::atomic<long long> g_launches{0};
void count_launch(int n) { g_launches.fetch_add(n, std::memory_order_relaxed); }

// Optional timing of one named kernel with CUDA events on its own stream
// (tg_profile_kernel / tg_profile_read).  Off unless a name is set.
namespace {
std::mutex g_prof_mu;
std::string g_prof_name;
std::atomic<bool> g_prof_on{false};
struct EvPair {
    cudaEvent_t a, b;
};
std::vector<EvPair> g_prof_events;
std::vector<cudaEvent_t> g_prof_pool;
cudaEvent_t g_prof_open = nullptr;

cudaEvent_t prof_event()
{
    if (!g_prof_pool.empty()) {
        cudaEvent_t e = g_prof_pool.back();
        g_prof_pool.pop_back();
        return e;
    }
    cudaEvent_t e = nullptr;
    cudaEventCreate(&e);
    return e;
}
}  // namespace

void prof_begin(const char *name, cudaStream_t s)
{
    if (!g_prof_on.load(std::memory_order_relaxed)) return;
    std::lock_guard<std::mutex> lk(g_prof_mu);
    if (g_prof_name != name) return;
    g_prof_open = prof_event();
    cudaEventRecord(g_prof_open, s);
}

void prof_end(const char *name, cudaStream_t s)
{
    if (!g_prof_on.load(std::memory_order_relaxed)) return;
    std::lock_guard<std::mutex> lk(g_prof_mu);
    if (g_prof_name != name || !g_prof_open) return;
    cudaEvent_t b = prof_event();
    cudaEventRecord(b, s);
    g_prof_events.push_back({g_prof_open, b});
    g_prof_open = nullptr;
}
}  // namespace tg

using namespace tg;

namespace {

thread_local std::string g_err;

tg_status fail(tg_status code, const char *fmt, ...)
{
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    g_err = buf;
    return code;
}

tg_status cuda_fail(cudaError_t e, const char *what, int line)
{
    (void)cudaGetLastError();
    return fail(e == cudaErrorMemoryAllocation ? TG_ERR_OUT_OF_MEMORY : TG_ERR_CUDA,
                "%s (%s) at tg_api.cu:%d: %s", cudaGetErrorName(e), cudaGetErrorString(e), line,
                what);
}

#define CK(call)                                                        \
    do {                                                                \
        cudaError_t _e = (call);                                        \
        if (_e != cudaSuccess) return cuda_fail(_e, #call, __LINE__);   \
    } while (0)

#define TRY(expr)                                   \
    do {                                            \
        tg_status _s = (expr);                      \
        if (_s != TG_OK) return _s;                 \
    } while (0)

constexpr int64_t kMaxCells = 357913941LL;  // 6 * cells must fit in 31 bits

std::mutex g_pool_mu;
bool g_pool_ready[64];

void setup_pool(int dev)
{
    std::lock_guard<std::mutex> lk(g_pool_mu);
    if (dev < 0 || dev >= 64 || g_pool_ready[dev]) return;
    cudaMemPool_t pool;
    if (cudaDeviceGetDefaultMemPool(&pool, dev) == cudaSuccess) {
        uint64_t thr = UINT64_MAX;
        cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &thr);
    }
    (void)cudaGetLastError();
    g_pool_ready[dev] = true;
}

// Pinned, device-mapped host slots for the status word and the sizes read
// back at the synchronisation points: a kernel stores them there directly,
// so a read-back never queues behind large copies in flight on the copy
// engines (a caller draining an earlier mesh's relations).  Pinned
// allocation is slow, so slots come from a process-wide pool of 4 KiB
// chunks and are recycled.
struct PinnedPool {
    std::mutex mu;
    std::vector<void *> free_slots;
    void *get()
    {
        std::lock_guard<std::mutex> lk(mu);
        if (free_slots.empty()) {
            char *chunk = nullptr;
            if (cudaHostAlloc((void **)&chunk, 4096, cudaHostAllocMapped) != cudaSuccess)
                return nullptr;
            for (int i = 0; i < 16; i++) free_slots.push_back(chunk + 256 * i);
        }
        void *p = free_slots.back();
        free_slots.pop_back();
        return p;
    }
    void put(void *p)
    {
        if (!p) return;
        std::lock_guard<std::mutex> lk(mu);
        free_slots.push_back(p);
    }
};
PinnedPool g_pinned;

// Side streams for kernels of one extraction that need nothing from each
// other (EF, TT, the per-face rows and the link adjacency beside EE):
// a stream and its fork / join events, kept per device and reused, so that a
// mesh built per request creates none.
struct SideLane {
    int device = 0;
    cudaStream_t s = nullptr;
    cudaEvent_t fork = nullptr, join = nullptr;
};
struct SidePool {
    std::mutex mu;
    std::vector<SideLane *> free_lanes;
    SideLane *get(int device)
    {
        {
            std::lock_guard<std::mutex> lk(mu);
            for (size_t i = 0; i < free_lanes.size(); i++)
                if (free_lanes[i]->device == device) {
                    SideLane *l = free_lanes[i];
                    free_lanes.erase(free_lanes.begin() + (std::ptrdiff_t)i);
                    return l;
                }
        }
        SideLane *l = new SideLane();
        l->device = device;
        if (cudaStreamCreateWithFlags(&l->s, cudaStreamNonBlocking) != cudaSuccess ||
            cudaEventCreateWithFlags(&l->fork, cudaEventDisableTiming) != cudaSuccess ||
            cudaEventCreateWithFlags(&l->join, cudaEventDisableTiming) != cudaSuccess) {
            (void)cudaGetLastError();
            if (l->s) cudaStreamDestroy(l->s);
            if (l->fork) cudaEventDestroy(l->fork);
            delete l;
            return nullptr;
        }
        return l;
    }
    void put(SideLane *l)
    {
        if (!l) return;
        std::lock_guard<std::mutex> lk(mu);
        free_lanes.push_back(l);
    }
};
SidePool g_side;

// One fork of an extraction's stream: the stream fork() returns runs what it
// is given after everything enqueued on the main stream before the call;
// join() makes the main stream wait for that work.  The destructor joins, so
// declared after the extraction's temporaries it orders their frees after
// the side work, on every return path.  Without a side stream (none could
// be made) fork() returns the main stream itself.
struct Fork {
    cudaStream_t main;
    int device;
    SideLane *lane = nullptr;
    bool open = false;
    Fork(cudaStream_t s, int dev) : main(s), device(dev) {}
    cudaStream_t fork()
    {
        join();
        if (!lane) lane = g_side.get(device);
        if (!lane) return main;
        if (cudaEventRecord(lane->fork, main) != cudaSuccess ||
            cudaStreamWaitEvent(lane->s, lane->fork, 0) != cudaSuccess) {
            (void)cudaGetLastError();
            return main;
        }
        open = true;
        return lane->s;
    }
    void join()
    {
        if (!open) return;
        open = false;
        if (cudaEventRecord(lane->join, lane->s) != cudaSuccess ||
            cudaStreamWaitEvent(main, lane->join, 0) != cudaSuccess) {
            // the main stream cannot be ordered after the side stream: wait
            // for it from the host instead
            (void)cudaGetLastError();
            cudaStreamSynchronize(lane->s);
        }
    }
    ~Fork()
    {
        join();
        g_side.put(lane);
    }
};

struct Rel {
    int64_t rows = 0, entries = 0;
    int width = 0;
    int64_t *off = nullptr;
    int32_t *ent = nullptr;
    bool ready = false;
    uint32_t opts = 0;
};

const int kWidth[14] = {0, 6, 2, 0, 4, 3, 3, 2, 0, 0, 0, 0, 0, 0};
const char *kName[14] = {"validate", "TE", "EV", "ET", "TF", "FV", "FE",
                         "FT",       "EF", "VT", "TT", "FF", "EE", "VV"};

// Scoped list of stream-ordered temporaries, freed when the stage ends.
struct Temps {
    cudaStream_t s;
    void *p[64];
    int n = 0;
    explicit Temps(cudaStream_t st) : s(st) {}
    ~Temps()
    {
        for (int i = 0; i < n; i++)
            if (p[i]) cudaFreeAsync(p[i], s);
    }
    template <class T>
    tg_status alloc(T **out, int64_t count, bool zero = false)
    {
        size_t b = (size_t)std::max<int64_t>(count, 1) * sizeof(T);
        if (n >= 64) return fail(TG_ERR_UNSUPPORTED, "too many temporaries in one stage");
        void *q = nullptr;
        cudaError_t e = cudaMallocAsync(&q, b, s);
        if (e != cudaSuccess) return cuda_fail(e, "cudaMallocAsync (temporary)", __LINE__);
        if (zero) {
            e = cudaMemsetAsync(q, 0, b, s);
            if (e != cudaSuccess) return cuda_fail(e, "cudaMemsetAsync", __LINE__);
        }
        p[n++] = q;
        *out = (T *)q;
        return TG_OK;
    }
    // free q with the others if the stage fails (list sized for every path)
    void track(void *q) { p[n++] = q; }
    // hand a temporary over to the caller (it is not freed here)
    void keep(void *q)
    {
        for (int i = 0; i < n; i++)
            if (p[i] == q) p[i] = nullptr;
    }
};

template <class T>
tg_status dalloc(T **out, int64_t count, cudaStream_t s)
{
    size_t b = (size_t)std::max<int64_t>(count, 1) * sizeof(T);
    void *q = nullptr;
    cudaError_t e = cudaMallocAsync(&q, b, s);
    if (e != cudaSuccess) return cuda_fail(e, "cudaMallocAsync", __LINE__);
    *out = (T *)q;
    return TG_OK;
}

// Offsets of several arrays in one allocation (each on a 256-byte boundary),
// so that arrays zeroed together cost one memset.
struct Carve {
    size_t bytes = 0;
    template <class T>
    size_t add(int64_t n)
    {
        const size_t off = bytes;
        bytes += ((size_t)std::max<int64_t>(n, 1) * sizeof(T) + 255) & ~size_t(255);
        return off;
    }
};

}  // namespace

void tg::set_last_error(const char *msg) { g_err = msg; }

struct tg_mesh {
    int device = 0;
    cudaStream_t last_stream = nullptr;  // stream of the last call, used to free asynchronously
    int64_t V = 0, T = 0, E = -1, F = -1;
    int4 *tvs = nullptr;
    // star processing order: vertices by first cell (see tg_star.cu)
    int32_t *vorder = nullptr;          // [V] vertex at each position (cell-less ones last)
    int32_t *vpos = nullptr;            // [V] position of each vertex
    int32_t *heavy_off = nullptr;       // where each heavy star's entries start among theirs
    ScanWorkspace scan;                 // every prefix scan of the mesh (tg_scan.cu)
    // segments of cells (the meshes of a batch): cell starts, and after each
    // extraction their first edge and face ids (device, n_seg + 1 each)
    int64_t n_seg = 0;
    int64_t *seg_c = nullptr;
    int64_t *seg_ef = nullptr;
    Rel rel[14];
    // stars of more than kMaxStar cells (tg_heavy.cu): processing positions
    // n_light .. n_light + n_heavy - 1, heavy_entries VT entries in all
    int64_t n_light = 0, n_heavy = 0, heavy_entries = 0;
    int64_t n_wide = 0;         // light stars of more than 31 cells (64-bit masks)
    int max_deg = 0;            // largest degree above kMaxDeg seen by the extraction, else 0
    bool wide_deg = false;      // a vertex has more than kNarrowDeg neighbours
    // the link adjacency of critical points (LinkGraph; adj null: not built)
    int64_t *lg_off = nullptr;
    int32_t *lg_ent = nullptr;
    void *lg_adj = nullptr;
    DevStatus *st = nullptr;    // device
    DevStatus *st_host = nullptr;
    int64_t *sz_host = nullptr; // pinned slots for sizes read back at sync points
};

namespace {

void free_rel(Rel &r, cudaStream_t s = nullptr, bool async = false)
{
    if (async) {
        if (r.off) cudaFreeAsync(r.off, s);
        if (r.ent) cudaFreeAsync(r.ent, s);
    } else {
        if (r.off) cudaFree(r.off);
        if (r.ent) cudaFree(r.ent);
    }
    r = Rel();
}

tg_status reset_status(tg_mesh *m, cudaStream_t s)
{
    launch_reset_status(m->st, s);
    return TG_OK;
}

// Read the status word plus up to 8 device scalars (int64 if `wide[i]`,
// else int32) into m->sz_host, synchronously.
tg_status sync_read(tg_mesh *m, cudaStream_t s, int n, const void *const *src, const bool *wide)
{
    PublishArgs a{};
    a.st = m->st;
    a.n = n;
    for (int i = 0; i < n; i++) {
        a.src[i] = src[i];
        a.wide[i] = wide[i] ? 1 : 0;
    }
    CK(cudaHostGetDevicePointer((void **)&a.h_st, m->st_host, 0));
    CK(cudaHostGetDevicePointer((void **)&a.h_sz, m->sz_host, 0));
    launch_publish(a, s);
    CK(cudaGetLastError());
    CK(cudaStreamSynchronize(s));
    return TG_OK;
}

tg_status check_flags(const tg_mesh *m, unsigned mask_ok = 0)
{
    const DevStatus &h = *m->st_host;
    const unsigned f = h.flags & ~mask_ok;
    if (!f) return TG_OK;
    if (f & ST_BAD_ID)
        return fail(TG_ERR_INVALID_MESH, "cell %d has a vertex id outside [0, %lld)", h.bad_cell,
                    (long long)m->V);
    if (f & ST_DUP_VERTEX)
        return fail(TG_ERR_INVALID_MESH, "cell %d repeats a vertex", h.bad_cell);
    if (f & ST_NONMANIFOLD_FACE)
        return fail(TG_ERR_INVALID_MESH, "a face of cell %d lies in more than two cells",
                    h.bad_cell);
    if (f & ST_HEAVY_STAR)
        return fail(TG_ERR_UNSUPPORTED,
                    "vertex %d lies in more than %d cells (largest star this build handles)",
                    h.bad_vertex, kMaxStar);
    if (f & ST_HEAVY_DEG)
        return fail(TG_ERR_UNSUPPORTED,
                    "a vertex has %d neighbours (more than %d, the largest this build handles)",
                    h.max_deg, kMaxDeg);
    if (f & ST_HASH_FULL)
        return fail(TG_ERR_UNSUPPORTED, "vertex %d: neighbour table overflow", h.bad_vertex);
    if (f & ST_STAR_OVERFLOW)
        return fail(TG_ERR_UNSUPPORTED, "vertex %d: neighbour summary overflow", h.bad_vertex);
    if (f & ST_SCAN_STALLED)
        return fail(TG_ERR_CUDA, "a prefix scan gave up waiting for a preceding tile");
    return fail(TG_ERR_CUDA, "unexpected device status 0x%x", f);
}

inline uint32_t bit(int r) { return 1u << r; }

tg_status set_fixed(tg_mesh *m, int r, int32_t *ent, int64_t rows)
{
    free_rel(m->rel[r]);
    Rel &x = m->rel[r];
    x.rows = rows;
    x.width = kWidth[r];
    x.entries = rows * kWidth[r];
    x.ent = ent;
    x.ready = true;
    return TG_OK;
}

void set_csr(tg_mesh *m, int r, int64_t *off, int32_t *ent, int64_t rows, int64_t entries,
             uint32_t opts = 0)
{
    free_rel(m->rel[r]);
    Rel &x = m->rel[r];
    x.rows = rows;
    x.entries = entries;
    x.width = 0;
    x.off = off;
    x.ent = ent;
    x.ready = true;
    x.opts = opts;
}

void free_link_graph(tg_mesh *m, cudaStream_t s)
{
    if (m->lg_off) cudaFreeAsync(m->lg_off, s);
    if (m->lg_ent) cudaFreeAsync(m->lg_ent, s);
    if (m->lg_adj) cudaFreeAsync(m->lg_adj, s);
    m->lg_off = nullptr;
    m->lg_ent = nullptr;
    m->lg_adj = nullptr;
}

// entries of the link graph, at most: its rows are padded to multiples of eight
int64_t link_entries(const tg_mesh *m, int64_t nvv) { return nvv + 7 * m->V; }

LinkGraph link_graph(const tg_mesh *m, int64_t nvv)
{
    return {m->V, link_entries(m, nvv), m->lg_off, m->lg_ent, m->vorder, m->vpos, m->lg_adj, m->wide_deg};
}

// The link adjacency of critical points: VV renumbered into the star
// processing order and its masks, kept on the mesh.  alloc makes every buffer,
// the temporaries too, on the extraction's own stream (before a fork, so that
// a side stream may use them); build launches.
struct LinkBuild {
    int32_t *len, *win;
    tg_status alloc(tg_mesh *m, int64_t nvv, Temps &tmp, cudaStream_t s)
    {
        TRY(tmp.alloc(&len, m->V));
        const int64_t n = link_entries(m, nvv);
        TRY(tmp.alloc(&win, window_count(n, crit_window()) + 1));
        int64_t *off;
        int32_t *ent;
        char *adj;
        TRY(dalloc(&off, m->V + 1, s));
        m->lg_off = off;
        TRY(dalloc(&ent, n, s));
        m->lg_ent = ent;
        TRY(dalloc(&adj, n * (m->wide_deg ? 8 : 4), s));
        m->lg_adj = adj;
        return TG_OK;
    }
    void build(tg_mesh *m, const int64_t *vv_off, const int32_t *vv, int64_t nvv, cudaStream_t s)
    {
        const LinkGraph g = link_graph(m, nvv);
        launch_vv_lengths_in_order(vv_off, m->vorder, m->V, len, s);
        ScanJob job{len, m->lg_off, m->V, SCAN_COUNT_PAD8, nullptr};
        scan_batch(&job, 1, m->scan, m->st, s);
        launch_window_starts(m->lg_off, m->V, g.n_ent, crit_window(), win, s);
        launch_rows_in_order(vv_off, vv, m->vorder, m->vpos, m->V, m->lg_off, m->lg_ent, s);
        launch_crit_adj(g, win, m->st, m->max_deg ? 1 : 0, s);
    }
};

tg_status run_extract(tg_mesh *m, uint32_t mask, uint32_t opts, cudaStream_t s)
{
    const int64_t V = m->V, T = m->T;
    const bool tt_vertex = (opts & TG_OPT_TT_VERTEX_SHARING) != 0;
    const bool want_tt_face = (mask & TG_TT) && !tt_vertex;
    const uint32_t star_rel = TG_TE | TG_EV | TG_ET | TG_TF | TG_FV | TG_FE | TG_FT | TG_EF |
                              TG_FF | TG_EE | TG_VV;
    const bool want_star = (mask & star_rel) || want_tt_face;
    const int64_t *vt_off = m->rel[TG_REL_VT].off;
    const int32_t *vt = m->rel[TG_REL_VT].ent;
    Temps tmp(s);
    Fork side(s, m->device);   // after tmp: joined before its frees

    if (want_star) {
        // the status is clean: the read-back that ended the last call reset it
        // ---- star pass: first occurrences, edge records, neighbour counts ----
        const int64_t nwe = (6 * T + 31) / 32, nwf = (4 * T + 31) / 32;
        uint32_t *eflag, *fflag, *fbnd;
        uint2 *erank, *frank, *brank;
        int64_t *vv_off;
        // FE is read off each face's first cell (k_face_fill), which the
        // face's FT row and the cell's TF row tell; EF off TF
        const bool need_tf = (mask & (TG_TF | TG_FE | TG_FF | TG_EF)) || want_tt_face;
        const bool need_ft = (mask & (TG_FT | TG_FE | TG_FF)) || want_tt_face;
        const bool need_te = mask & (TG_TE | TG_FE);
        const bool need_ev = mask & (TG_EV | TG_EE);
        // the edges by id: for everything per edge
        const bool need_edge = need_te || need_ev || (mask & (TG_ET | TG_EF));
        StarPass sp{};
        {
            // the bitmaps the star pass sets bits in, the neighbour counts
            // and the record counter: one zeroed allocation
            Carve c;
            const size_t o_e = c.add<uint32_t>(nwe), o_f = c.add<uint32_t>(nwf),
                         o_b = c.add<uint32_t>(nwf), o_d = c.add<int32_t>(V),
                         o_i = c.add<int32_t>(V),
                         o_v = c.add<uint8_t>(V), o_n = c.add<uint32_t>(2);
            char *z;
            TRY(tmp.alloc(&z, (int64_t)c.bytes, true));
            eflag = (uint32_t *)(z + o_e);
            fflag = (uint32_t *)(z + o_f);
            fbnd = (uint32_t *)(z + o_b);
            sp.deg_own = (int32_t *)(z + o_d);
            sp.deg_in = (int32_t *)(z + o_i);
            sp.vbnd = (uint8_t *)(z + o_v);
            sp.n_rec = (uint32_t *)(z + o_n);
            sp.n_wide = sp.n_rec + 1;
        }
        TRY(tmp.alloc(&erank, nwe + 1));
        TRY(tmp.alloc(&frank, nwf + 1));
        TRY(tmp.alloc(&brank, nwf + 1));
        TRY(dalloc(&vv_off, V + 1, s));
        tmp.track(vv_off);  // owned by the VV relation once it is ready
        int64_t *deg_sq;  // prefix of deg^2: its total sizes EE (sum deg^2 - 2E)
        TRY(tmp.alloc(&deg_sq, V + 1));
        // at most six edges a cell (their number is read back below)
        TRY(tmp.alloc(&sp.rec, 6 * T));
        TRY(tmp.alloc(&sp.place, 6 * T));
        if (m->n_wide > 0 || m->n_heavy > 0) TRY(tmp.alloc(&sp.rec_hi, 6 * T));
        if (m->n_wide > 0) TRY(tmp.alloc(&sp.wide, m->n_wide));
        if (need_tf || need_ft) TRY(tmp.alloc(&sp.fnext, 4 * T));
        sp.n_light = m->n_light;
        sp.vorder = m->vorder;
        sp.vt_off = vt_off;
        sp.vt = vt;
        sp.tvs = m->tvs;
        sp.eflag = eflag;
        sp.fflag = fflag;
        sp.fbnd = fbnd;
        sp.st = m->st;
        launch_star(sp, s);
        launch_star_wide(sp, m->n_wide, s);
        HeavyStars hv{};
        if (m->n_heavy > 0) {
            hv.star = sp;
            hv.n_heavy = m->n_heavy;
            hv.heavy_off = m->heavy_off;
            TRY(tmp.alloc(&hv.pairs, 3 * m->heavy_entries));
            launch_heavy(hv, s);
        }
        // (the incident-edge rows of EE are padded)
        const bool want_ee = mask & TG_EE;
        int64_t *eid_off = nullptr;
        if (want_ee) TRY(tmp.alloc(&eid_off, V + 1));
        ScanJob jobs[6] = {{sp.deg_own, vv_off, V, SCAN_COUNT_I32, sp.deg_in},
                           {eflag, erank, nwe, SCAN_POPC_RANK, nullptr},
                           {fflag, frank, nwf, SCAN_POPC_RANK, nullptr},
                           {fbnd, brank, nwf, SCAN_POPC_RANK, nullptr},
                           {sp.deg_own, deg_sq, V, SCAN_DEG_SQUARE, sp.deg_in},
                           {sp.deg_own, eid_off, V, SCAN_EID_WORDS, sp.deg_in}};
        scan_batch(jobs, want_ee ? 6 : 5, m->scan, m->st, s);

        // ---- the one synchronisation: edge, face, neighbour and boundary
        // counts size every output from here on ----
        {
            const void *src[5] = {vv_off + V, &erank[nwe].y, &frank[nwf].y, &brank[nwf].y,
                                  deg_sq + V};
            const bool w8[5] = {true, false, false, false, true};
            TRY(sync_read(m, s, 5, src, w8));
        }
        if (m->st_host->flags) return check_flags(m);
        m->max_deg = m->st_host->max_deg > kMaxDeg ? m->st_host->max_deg : 0;
        m->wide_deg = m->st_host->max_deg > kNarrowDeg;
        const int largest_deg = m->st_host->max_deg;
        const int64_t nvv = m->sz_host[0];
        const int64_t E = m->sz_host[1], F = m->sz_host[2];
        const int64_t n_bnd = m->sz_host[3];  // boundary faces
        const int64_t sum_deg_sq = m->sz_host[4];
        m->E = E;
        m->F = F;
        if (m->seg_c) launch_seg_ranks(m->seg_c, m->n_seg, erank, frank, m->seg_ef, s);

        // ---- ids: VV, EV, row lengths (per edge); TF, FT, FV (per cell).
        // Each kernel goes out once its own buffers exist; the later
        // allocations are made while it runs
        int32_t *vv;
        uint32_t *eid = nullptr;
        int32_t *ev = nullptr, *te = nullptr, *tf = nullptr, *fv = nullptr, *ft = nullptr;
        TRY(dalloc(&vv, nvv, s));
        tmp.track(vv);
        int2 *inc = nullptr;
        if (mask & TG_EE) {
            TRY(tmp.alloc(&eid, nvv + 16 * V));   // eid_words of each row at most
            TRY(tmp.alloc(&inc, nvv));
        }
        EdgePass ep{};
        if (need_edge) TRY(tmp.alloc(&ep.edge, E));
        if (need_edge && sp.rec_hi) TRY(tmp.alloc(&ep.edge_hi, E));
        ep.E = E;
        ep.rec = sp.rec; ep.place = sp.place; ep.rec_hi = sp.rec_hi; ep.pairs = hv.pairs;
        ep.vt_off = vt_off; ep.vt = vt; ep.tvs = m->tvs;
        ep.erank = need_edge ? erank : nullptr;
        ep.fflag = fflag; ep.fbnd = fbnd; ep.vbnd = sp.vbnd;
        ep.vv_off = vv_off; ep.inc = inc; ep.vv = vv;
        ep.count_ef = (mask & TG_EF) != 0;
        launch_edge_ids(ep, s);
        if (need_tf) TRY(tmp.alloc(&tf, 4 * T));
        if (need_ft) TRY(tmp.alloc(&ft, 2 * F));
        if (mask & TG_FV) TRY(tmp.alloc(&fv, 3 * F));
        if (tf || ft || fv) launch_cell_faces(T, m->tvs, frank, sp.fnext, tf, ft, fv, s);
        int64_t *et_off = nullptr, *ef_off = nullptr, *ee_off = nullptr, *ff_off = nullptr;
        if (mask & TG_ET) TRY(dalloc(&et_off, E + 1, s));
        if (et_off) tmp.track(et_off);
        if (mask & TG_EF) TRY(dalloc(&ef_off, E + 1, s));
        if (ef_off) tmp.track(ef_off);
        if (mask & TG_EE) TRY(dalloc(&ee_off, E + 1, s));
        if (ee_off) tmp.track(ee_off);
        if (need_ev) TRY(tmp.alloc(&ev, 2 * E));
        if (et_off || ef_off || ee_off || ev)
            launch_edge_offsets(ep, et_off, ef_off, ee_off, ev, m->scan, m->st, s);
        if (inc) launch_inc_sort(vv_off, V, inc, vv, eid_off, eid, s);
        else launch_vv_sort(vv_off, V, nvv, vv, s);
        // CSR totals: ET = 6T, EF = 3F always; TT and FF from the
        // boundary-face count
        int32_t *et = nullptr, *ef = nullptr, *ee = nullptr, *ff = nullptr, *tt = nullptr,
                *fe = nullptr;
        int64_t *tt_off = nullptr;
        const int64_t n_et = 6 * T, n_ef = 3 * F;
        const int64_t n_tt = 4 * T - n_bnd, n_ff = 3 * (2 * F - n_bnd);
        if (need_te) TRY(tmp.alloc(&te, 6 * T));
        if (et_off) TRY(dalloc(&et, n_et, s));
        if (ef_off) TRY(dalloc(&ef, n_ef, s));
        if (mask & TG_FE) TRY(dalloc(&fe, 3 * F, s));
        if (want_tt_face) {
            TRY(dalloc(&tt_off, T + 1, s));
            TRY(dalloc(&tt, n_tt, s));
            if (T == 0) CK(cudaMemsetAsync(tt_off, 0, 8, s));
        }
        if (mask & TG_FF) {
            TRY(tmp.alloc(&ff_off, F + 1));
            TRY(dalloc(&ff, n_ff, s));
            if (T == 0) CK(cudaMemsetAsync(ff_off, 0, 8, s));
        }
        tmp.keep(vv);
        tmp.keep(vv_off);
        set_csr(m, TG_REL_VV, vv_off, vv, V, nvv);
        free_link_graph(m, s);

        // ET and EF rows, the per-cell TT rows, the per-face FE / FF rows and on
        // request the link adjacency of critical points, on a side stream
        // beside EE (each reads only what the passes before it wrote)
        const int64_t n_ee = sum_deg_sq - 2 * E;   // deg(a) + deg(b) - 2 per edge (a,b)
        if (ee_off) TRY(dalloc(&ee, n_ee, s));
        const bool prep_adj = (opts & TG_OPT_LINK_ADJACENCY) && (mask & TG_VV);
        LinkBuild lb;
        if (prep_adj) TRY(lb.alloc(m, nvv, tmp, s));
        if (te || fe || tt || ff_off || ff || et || ef || prep_adj) {
            const cudaStream_t s2 = side.fork();
            ep.te = te; ep.et_off = et_off; ep.ef_off = ef_off; ep.et = et; ep.ef = ef; ep.tf = tf;
            if (te || et || ef) launch_edge_rows(ep, s2);
            if (tt || ff_off) launch_cell_tt(T, F, tf, ft, brank, tt_off, tt, ff_off, s2);
            if (fe || ff) launch_face_fill(ft, tf, te, brank, F, fe, ff_off, ff, s2);
            if (prep_adj) lb.build(m, vv_off, vv, nvv, s2);
        }
        if (ee_off) {
            launch_ee_fill(ev, E, eid_off, eid, ee_off, ee, largest_deg, s);
            if (m->max_deg) launch_ee_heavy(ev, E, vv_off, eid_off, eid, ee_off, ee, s);
        }
        side.join();
        CK(cudaGetLastError());

        auto give_fixed = [&](int r, int32_t *p, int64_t rows) {
            tmp.keep(p);
            set_fixed(m, r, p, rows);
        };
        if (mask & TG_EV) give_fixed(TG_REL_EV, ev, E);
        if (mask & TG_TE) give_fixed(TG_REL_TE, te, T);
        if (mask & TG_TF) give_fixed(TG_REL_TF, tf, T);
        if (mask & TG_FV) give_fixed(TG_REL_FV, fv, F);
        if (mask & TG_FT) give_fixed(TG_REL_FT, ft, F);
        if (fe) set_fixed(m, TG_REL_FE, fe, F);
        if (et) {
            tmp.keep(et_off);
            set_csr(m, TG_REL_ET, et_off, et, E, n_et);
        }
        if (ef) {
            tmp.keep(ef_off);
            set_csr(m, TG_REL_EF, ef_off, ef, E, n_ef);
        }
        if (ee) {
            tmp.keep(ee_off);
            set_csr(m, TG_REL_EE, ee_off, ee, E, n_ee);
        }
        if (ff) {
            tmp.keep(ff_off);
            set_csr(m, TG_REL_FF, ff_off, ff, F, n_ff);
        }
        if (tt) set_csr(m, TG_REL_TT, tt_off, tt, T, n_tt, 0);
    }

    if ((mask & TG_TT) && tt_vertex) {
        int32_t *cnt;
        int64_t *tt_off;
        TRY(tmp.alloc(&cnt, T));
        TRY(dalloc(&tt_off, T + 1, s));
        launch_tt_vertex_count(m->tvs, T, vt_off, vt, cnt, s);
        ScanJob job{cnt, tt_off, T, SCAN_COUNT_I32, nullptr};
        scan_batch(&job, 1, m->scan, m->st, s);
        const void *src[1] = {tt_off + T};
        const bool w8[1] = {true};
        TRY(sync_read(m, s, 1, src, w8));
        int32_t *tt;
        TRY(dalloc(&tt, m->sz_host[0], s));
        launch_tt_vertex_fill(m->tvs, T, vt_off, vt, tt_off, tt, s);
        set_csr(m, TG_REL_TT, tt_off, tt, T, m->sz_host[0], TG_OPT_TT_VERTEX_SHARING);
    }
    CK(cudaGetLastError());
    return TG_OK;
}

}  // namespace

tg_status tg::critical_points_rows(tg_mesh *m, int64_t v0, int64_t nv, const void *field,
                                   int field_type, int field_on_device, uint32_t *classes_out,
                                   int out_on_device, cudaStream_t s)
{
    if (!m || !field || !classes_out) return fail(TG_ERR_INVALID_ARGUMENT, "NULL argument");
    if (field_type != TG_FIELD_F32 && field_type != TG_FIELD_F64)
        return fail(TG_ERR_INVALID_ARGUMENT, "field_type must be TG_FIELD_F32 or TG_FIELD_F64");
    if (v0 < 0 || nv < 0 || v0 + nv > m->V) return fail(TG_ERR_INVALID_ARGUMENT, "bad vertex range");
    m->last_stream = s;
    if (!m->rel[TG_REL_VV].ready) TRY(tg_extract(m, TG_VV, 0, s));
    const Rel &vv = m->rel[TG_REL_VV];
    if (!m->lg_adj) {
        // VV rows longer than the adjacency masks take the heavy path of the
        // classification, so no status read-back here
        free_link_graph(m, s);
        Temps adj_tmp(s);
        LinkBuild lb;
        TRY(lb.alloc(m, vv.entries, adj_tmp, s));
        lb.build(m, vv.off, vv.ent, vv.entries, s);
    }
    Temps tmp(s);
    const size_t esz = field_type == TG_FIELD_F64 ? 8 : 4;
    const void *f = field;
    if (!field_on_device) {
        char *d;
        TRY(tmp.alloc(&d, (int64_t)(nv * esz)));
        CK(cudaMemcpyAsync(d, field, nv * esz, cudaMemcpyHostToDevice, s));
        f = d;
    }
    uint32_t *out = classes_out;
    if (!out_on_device) TRY(tmp.alloc(&out, 3 * nv));
    char *ordered = nullptr;
    if (classify_orders_field(nv)) TRY(tmp.alloc(&ordered, m->V * (int64_t)esz));
    launch_crit_classify(link_graph(m, vv.entries), f, field_type, ordered, v0, nv, out, s);
    if (m->max_deg) {
        // vertices of more than kMaxDeg neighbours: at most one per
        // kMaxDeg + 1 VV entries
        const int64_t max_listed = std::min<int64_t>(nv, vv.entries / (kMaxDeg + 1) + 1);
        int32_t *list, *n_list, *scratch;
        TRY(tmp.alloc(&list, max_listed));
        TRY(tmp.alloc(&n_list, 1, true));
        TRY(tmp.alloc(&scratch, vv.entries));
        launch_crit_heavy(vv.off, vv.ent, v0, nv, max_listed, f, field_type, out, list, n_list,
                          scratch, s);
    }
    CK(cudaGetLastError());
    if (!out_on_device) {
        CK(cudaMemcpyAsync(classes_out, out, (size_t)nv * 12, cudaMemcpyDeviceToHost, s));
        CK(cudaStreamSynchronize(s));
    }
    return TG_OK;
}

extern "C" {

const char *tg_version(void) { return "tetragpu-gb300 1.1 (sm_103a)"; }

const char *tg_tuning_info(void)
{
    static std::string info;
    static std::once_flag once;
    std::call_once(once, [] {
        char buf[512];
        snprintf(buf, sizeof buf,
                 "{\"TG_STAR_WIN\": %d, \"TG_STAR_THREADS\": %d, \"TG_STAR_PER\": %d, "
                 "\"TG_VTS_THREADS\": %d, \"TG_EDGE_ITEMS\": %d, "
                 "\"TG_ADJ_WIN\": %d, \"TG_ADJ_THREADS\": %d}",
                 TG_STAR_WIN, TG_STAR_THREADS, TG_STAR_PER, TG_VTS_THREADS, TG_EDGE_ITEMS,
                 TG_ADJ_WIN, TG_ADJ_THREADS);
        info = buf;
    });
    return info.c_str();
}

const char *tg_last_error_string(void) { return g_err.c_str(); }

int64_t tg_kernel_launch_count(void) { return tg::g_launches.load(); }

tg_status tg_mesh_destroy(tg_mesh *m)
{
    if (!m) return TG_OK;
    int cur = 0;
    cudaGetDevice(&cur);
    cudaSetDevice(m->device);
    // stream-ordered frees on the stream the mesh was last used on, then one
    // wait for that stream (no device-wide synchronisation)
    cudaStream_t s = m->last_stream;
    for (auto &r : m->rel) free_rel(r, s, true);
    if (m->tvs) cudaFreeAsync(m->tvs, s);
    if (m->vorder) cudaFreeAsync(m->vorder, s);
    if (m->heavy_off) cudaFreeAsync(m->heavy_off, s);
    if (m->seg_c) cudaFreeAsync(m->seg_c, s);
    if (m->seg_ef) cudaFreeAsync(m->seg_ef, s);
    if (m->vpos) cudaFreeAsync(m->vpos, s);
    free_link_graph(m, s);
    if (m->st) cudaFreeAsync(m->st, s);
    if (m->scan.buf) {
        // after the last scan, whichever stream it ran on
        if (m->scan.used && m->scan.last != s) cudaStreamWaitEvent(s, m->scan.done, 0);
        cudaFreeAsync(m->scan.buf, s);
    }
    cudaStreamSynchronize(s);  // no copy into the pinned slots is still in flight
    if (m->scan.done) cudaEventDestroy(m->scan.done);
    g_pinned.put(m->st_host);
    g_pinned.put(m->sz_host);
    cudaSetDevice(cur);
    (void)cudaGetLastError();
    delete m;
    return TG_OK;
}

static tg_status mesh_create_impl(const int32_t *tv, int64_t T, int64_t V, int on_device,
                                  cudaStream_t s, tg_mesh *m)
{
    CK(cudaGetDevice(&m->device));
    setup_pool(m->device);
    m->st_host = (DevStatus *)g_pinned.get();
    m->sz_host = (int64_t *)g_pinned.get();
    if (!m->st_host || !m->sz_host) return fail(TG_ERR_OUT_OF_MEMORY, "pinned host memory");
    TRY(dalloc(&m->st, 1, s));
    TRY(reset_status(m, s));
    TRY(dalloc(&m->tvs, T, s));
    const int32_t *src = tv;
    if (!on_device && T > 0) {
        CK(cudaMemcpyAsync(m->tvs, tv, (size_t)T * 16, cudaMemcpyHostToDevice, s));
        src = reinterpret_cast<const int32_t *>(m->tvs);
    }
    // the scan workspace of every later scan on the mesh, zeroed once
    m->scan.job_words = std::max(scan_job_words(std::max(std::max(V, T), (6 * T + 31) / 32)),
                                 (edge_offsets_words(6 * T) + kMaxScanJobs - 1) / kMaxScanJobs);
    const size_t ws_bytes = (size_t)2 * kMaxScanJobs * m->scan.job_words * 8;
    CK(cudaMallocAsync((void **)&m->scan.buf, ws_bytes, s));
    CK(cudaMemsetAsync(m->scan.buf, 0, ws_bytes, s));
    CK(cudaEventCreateWithFlags(&m->scan.done, cudaEventDisableTiming));
    Temps tmp(s);
    // the per-vertex cell counts and the first-cell bitmap: one zeroed
    // allocation
    const int64_t nwk = (4 * T + 31) / 32;
    int32_t *deg_t, *heavy_cnt;
    uint32_t *vflag;
    {
        Carve c;
        const size_t o_d = c.add<int32_t>(V), o_f = c.add<uint32_t>(nwk), o_h = c.add<int32_t>(4);
        char *z;
        TRY(tmp.alloc(&z, (int64_t)c.bytes, true));
        deg_t = (int32_t *)(z + o_d);
        vflag = (uint32_t *)(z + o_f);
        heavy_cnt = (int32_t *)(z + o_h);
    }
    int4 *occ;
    TRY(tmp.alloc(&occ, T));
    launch_canon(src, T, V, m->tvs, deg_t, occ, m->st, s);
    int64_t *vt_off;
    int32_t *vt;
    TRY(dalloc(&vt_off, V + 1, s));
    ScanJob job{deg_t, vt_off, V, SCAN_COUNT_I32, nullptr};
    scan_batch(&job, 1, m->scan, m->st, s);
    TRY(dalloc(&vt, 4 * T, s));
    launch_vt_fill(m->tvs, T, vt_off, occ, vt, s);
    // VT row sort, which also marks each vertex's star-order key; then the
    // star processing order
    uint2 *vrank;
    int64_t *vkey;
    TRY(tmp.alloc(&vrank, nwk + 1));
    TRY(tmp.alloc(&vkey, V));
    TRY(dalloc(&m->heavy_off, 4 * T / (kMaxStar + 1) + 1, s));
    launch_vt_sort(vt_off, vt, V, 4 * T, m->tvs, vflag, vkey, heavy_cnt, m->heavy_off, s);
    ScanJob jf{vflag, vrank, nwk, SCAN_POPC_RANK, nullptr};
    scan_batch(&jf, 1, m->scan, m->st, s);
    TRY(dalloc(&m->vorder, V, s));
    TRY(dalloc(&m->vpos, V, s));
    launch_vorder_place(vt_off, V, vkey, vrank, nwk, heavy_cnt, m->vorder, m->vpos, s);
    CK(cudaGetLastError());
    set_csr(m, TG_REL_VT, vt_off, vt, V, 4 * T);
    // vertices with light stars, heavy ones, the heavy stars' entries and
    // the light stars of more than 31 cells
    const void *rd[4] = {&vrank[nwk].y, heavy_cnt, heavy_cnt + 1, heavy_cnt + 2};
    const bool w8[4] = {false, false, false, false};
    TRY(sync_read(m, s, 4, rd, w8));
    m->n_light = T ? m->sz_host[0] : 0;
    m->n_heavy = T ? m->sz_host[1] : 0;
    m->heavy_entries = T ? m->sz_host[2] : 0;
    m->n_wide = T ? m->sz_host[3] : 0;
    return check_flags(m);
}

tg_status tg_mesh_create(const int32_t *tv, int64_t n_cells, int64_t n_verts, int tv_on_device,
                         void *stream, tg_mesh **out)
{
    if (!out) return fail(TG_ERR_INVALID_ARGUMENT, "out is NULL");
    *out = nullptr;
    if (n_cells < 0 || n_verts < 0 || (n_cells > 0 && !tv))
        return fail(TG_ERR_INVALID_ARGUMENT, "bad mesh sizes or NULL TV");
    if (n_cells > kMaxCells)
        return fail(TG_ERR_UNSUPPORTED, "more than %lld cells (occurrence ids use 31 bits)",
                    (long long)kMaxCells);
    if (n_verts > INT_MAX) return fail(TG_ERR_UNSUPPORTED, "more than 2^31-1 vertices");
    tg_mesh *m = new tg_mesh();
    m->V = n_verts;
    m->T = n_cells;
    m->last_stream = (cudaStream_t)stream;
    tg_status st = mesh_create_impl(tv, n_cells, n_verts, tv_on_device, (cudaStream_t)stream, m);
    if (st != TG_OK) {
        std::string keep = g_err;
        tg_mesh_destroy(m);
        g_err = keep;
        return st;
    }
    *out = m;
    return TG_OK;
}

tg_status tg_tv_narrow_i64(const int64_t *cells, int64_t n_cells, int64_t n_points, int32_t *out)
{
    if (n_cells < 0 || n_points < 0 || (n_cells > 0 && (!cells || !out)))
        return fail(TG_ERR_INVALID_ARGUMENT, "bad sizes or NULL pointer");
    if (n_points > INT_MAX)
        return fail(TG_ERR_UNSUPPORTED, "%lld points: ids must fit int32 (at most 2^31-1 points)",
                    (long long)n_points);
    for (int64_t i = 0; i < 4 * n_cells; i++) {
        const int64_t x = cells[i];
        if (x < 0 || x >= n_points)
            return fail(TG_ERR_INVALID_MESH, "cell %lld has vertex id %lld, outside [0, %lld)",
                        (long long)(i / 4), (long long)x, (long long)n_points);
        out[i] = (int32_t)x;
    }
    return TG_OK;
}

tg_status tg_mesh_create_i64(const int64_t *tv, int64_t n_cells, int64_t n_verts, void *stream,
                             tg_mesh **out)
{
    if (!out) return fail(TG_ERR_INVALID_ARGUMENT, "out is NULL");
    *out = nullptr;
    if (n_cells < 0 || n_cells > kMaxCells)
        return fail(n_cells < 0 ? TG_ERR_INVALID_ARGUMENT : TG_ERR_UNSUPPORTED,
                    "bad cell count %lld", (long long)n_cells);
    std::vector<int32_t> tv32((size_t)(4 * n_cells));
    TRY(tg_tv_narrow_i64(tv, n_cells, n_verts, tv32.data()));
    return tg_mesh_create(tv32.data(), n_cells, n_verts, 0, stream, out);
}

tg_status tg_extract(tg_mesh *m, uint32_t mask, uint32_t options, void *stream)
{
    if (!m) return fail(TG_ERR_INVALID_ARGUMENT, "mesh is NULL");
    mask &= TG_ALL_RELATIONS;
    bool all_ready = true;
    for (int r = 1; r < 14; r++)
        if ((mask & bit(r)) && !(m->rel[r].ready && (r != TG_REL_TT || m->rel[r].opts ==
                                                     (options & TG_OPT_TT_VERTEX_SHARING))))
            all_ready = false;
    if (all_ready) return TG_OK;
    int cur = 0;
    cudaGetDevice(&cur);
    if (cur != m->device) CK(cudaSetDevice(m->device));
    m->last_stream = (cudaStream_t)stream;
    tg_status st = run_extract(m, mask, options, (cudaStream_t)stream);
    if (cur != m->device) cudaSetDevice(cur);
    return st;
}

tg_status tg_mesh_counts(const tg_mesh *m, int64_t *nv, int64_t *ne, int64_t *nf, int64_t *nc)
{
    if (!m) return fail(TG_ERR_INVALID_ARGUMENT, "mesh is NULL");
    if (nv) *nv = m->V;
    if (ne) *ne = m->E;
    if (nf) *nf = m->F;
    if (nc) *nc = m->T;
    return TG_OK;
}

tg_status tg_get_relation(const tg_mesh *m, int r, const int64_t **off, const int32_t **ent,
                          int64_t *rows, int64_t *entries, int32_t *width)
{
    if (!m || r < 1 || r > 13) return fail(TG_ERR_INVALID_ARGUMENT, "bad mesh or relation index");
    const Rel &x = m->rel[r];
    if (!x.ready) return fail(TG_ERR_NOT_COMPUTED, "relation %s has not been extracted", kName[r]);
    if (off) *off = x.off;
    if (ent) *ent = x.ent;
    if (rows) *rows = x.rows;
    if (entries) *entries = x.entries;
    if (width) *width = x.width;
    return TG_OK;
}

tg_status tg_copy_relation(const tg_mesh *m, int r, int64_t *off_host, int32_t *ent_host,
                           void *stream)
{
    if (!m || r < 1 || r > 13) return fail(TG_ERR_INVALID_ARGUMENT, "bad mesh or relation index");
    const Rel &x = m->rel[r];
    if (!x.ready) return fail(TG_ERR_NOT_COMPUTED, "relation %s has not been extracted", kName[r]);
    cudaStream_t s = (cudaStream_t)stream;
    if (off_host && x.off)
        CK(cudaMemcpyAsync(off_host, x.off, (size_t)(x.rows + 1) * 8, cudaMemcpyDeviceToHost, s));
    if (ent_host && x.entries)
        CK(cudaMemcpyAsync(ent_host, x.ent, (size_t)x.entries * 4, cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    return TG_OK;
}

tg_status tg_copy_relation_async(tg_mesh *m, int r, int64_t *off_host, int32_t *ent_host,
                                 void *stream)
{
    if (!m || r < 1 || r > 13) return fail(TG_ERR_INVALID_ARGUMENT, "bad mesh or relation index");
    const Rel &x = m->rel[r];
    if (!x.ready) return fail(TG_ERR_NOT_COMPUTED, "relation %s has not been extracted", kName[r]);
    cudaStream_t s = (cudaStream_t)stream;
    m->last_stream = s;
    if (off_host && x.off)
        CK(cudaMemcpyAsync(off_host, x.off, (size_t)(x.rows + 1) * 8, cudaMemcpyDeviceToHost, s));
    if (ent_host && x.entries)
        CK(cudaMemcpyAsync(ent_host, x.ent, (size_t)x.entries * 4, cudaMemcpyDeviceToHost, s));
    return TG_OK;
}

tg_status tg_copy_relation_async_i32(tg_mesh *m, int r, int32_t *off_host, int32_t *ent_host,
                                     void *stream)
{
    if (!m || r < 1 || r > 13) return fail(TG_ERR_INVALID_ARGUMENT, "bad mesh or relation index");
    const Rel &x = m->rel[r];
    if (!x.ready) return fail(TG_ERR_NOT_COMPUTED, "relation %s has not been extracted", kName[r]);
    cudaStream_t s = (cudaStream_t)stream;
    m->last_stream = s;
    if (off_host && x.off) {
        if (x.entries > INT32_MAX)
            return fail(TG_ERR_UNSUPPORTED, "relation %s has %lld entries: its offsets need int64",
                        kName[r], (long long)x.entries);
        int32_t *d = nullptr;
        const size_t b = (size_t)(x.rows + 1) * 4;
        CK(cudaMallocAsync(&d, b, s));
        launch_narrow(x.off, d, x.rows + 1, s);
        const cudaError_t e = cudaMemcpyAsync(off_host, d, b, cudaMemcpyDeviceToHost, s);
        cudaFreeAsync(d, s);   // stream-ordered: after the copy
        if (e != cudaSuccess) return cuda_fail(e, "cudaMemcpyAsync (offsets)", __LINE__);
    }
    if (ent_host && x.entries)
        CK(cudaMemcpyAsync(ent_host, x.ent, (size_t)x.entries * 4, cudaMemcpyDeviceToHost, s));
    return TG_OK;
}

tg_status tg_copy_relations_async_i32(tg_mesh *m, uint32_t mask, int32_t *const *off_host,
                                      int32_t *const *ent_host, void *stream)
{
    if (!m || !off_host || !ent_host) return fail(TG_ERR_INVALID_ARGUMENT, "NULL argument");
    mask &= TG_ALL_RELATIONS;
    cudaStream_t s = (cudaStream_t)stream;
    m->last_stream = s;
    NarrowJobs j{};
    int64_t at[14] = {};
    for (int r = 1; r < 14; r++) {
        if (!(mask & bit(r))) continue;
        const Rel &x = m->rel[r];
        if (!x.ready)
            return fail(TG_ERR_NOT_COMPUTED, "relation %s has not been extracted", kName[r]);
        if (!off_host[r] || !x.off) continue;
        if (x.entries > INT32_MAX)
            return fail(TG_ERR_UNSUPPORTED, "relation %s has %lld entries: its offsets need int64",
                        kName[r], (long long)x.entries);
        at[r] = j.start[j.n];
        j.src[j.n] = x.off;
        j.start[j.n + 1] = j.start[j.n] + x.rows + 1;
        j.n++;
    }
    int32_t *d = nullptr;
    if (j.n > 0) {
        CK(cudaMallocAsync(&d, (size_t)j.start[j.n] * 4, s));
        j.dst = d;
        launch_narrow_multi(j, s);
    }
    cudaError_t e = cudaSuccess;
    for (int r = 1; r < 14 && e == cudaSuccess; r++) {
        if (!(mask & bit(r))) continue;
        const Rel &x = m->rel[r];
        if (off_host[r] && x.off)
            e = cudaMemcpyAsync(off_host[r], d + at[r], (size_t)(x.rows + 1) * 4,
                                cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess && ent_host[r] && x.entries)
            e = cudaMemcpyAsync(ent_host[r], x.ent, (size_t)x.entries * 4, cudaMemcpyDeviceToHost,
                                s);
    }
    if (d) cudaFreeAsync(d, s);   // stream-ordered: after the copies
    if (e != cudaSuccess) return cuda_fail(e, "cudaMemcpyAsync (relations)", __LINE__);
    return TG_OK;
}

tg_status tg_copy_relation_i32(tg_mesh *m, int r, int32_t *off_host, int32_t *ent_host,
                               void *stream)
{
    TRY(tg_copy_relation_async_i32(m, r, off_host, ent_host, stream));
    CK(cudaStreamSynchronize((cudaStream_t)stream));
    return TG_OK;
}

tg_status tg_export_relation_i64(const tg_mesh *m, int r, int64_t *entries_out,
                                 int64_t *offsets_out, int out_on_device, void *stream)
{
    if (!m || r < 1 || r > 13) return fail(TG_ERR_INVALID_ARGUMENT, "bad mesh or relation index");
    const Rel &x = m->rel[r];
    if (!x.ready) return fail(TG_ERR_NOT_COMPUTED, "relation %s has not been extracted", kName[r]);
    cudaStream_t s = (cudaStream_t)stream;
    if (entries_out && x.entries) {
        int64_t *dst = entries_out;
        Temps tmp(s);
        if (!out_on_device) TRY(tmp.alloc(&dst, x.entries));
        launch_widen(x.ent, dst, x.entries, s);
        if (!out_on_device)
            CK(cudaMemcpyAsync(entries_out, dst, (size_t)x.entries * 8, cudaMemcpyDeviceToHost, s));
        CK(cudaGetLastError());
    }
    if (offsets_out && x.off)
        CK(cudaMemcpyAsync(offsets_out, x.off, (size_t)(x.rows + 1) * 8,
                           out_on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost, s));
    if (!out_on_device) CK(cudaStreamSynchronize(s));
    return TG_OK;
}

tg_status tg_export_rows_padded(const tg_mesh *m, int r, int32_t width, int64_t *padded_out,
                                uint32_t *counts_out, void *stream)
{
    if (!m || r < 1 || r > 13 || width < 0 || !padded_out)
        return fail(TG_ERR_INVALID_ARGUMENT, "bad mesh, relation index, width or output");
    const Rel &x = m->rel[r];
    if (!x.ready) return fail(TG_ERR_NOT_COMPUTED, "relation %s has not been extracted", kName[r]);
    if (!x.off) return fail(TG_ERR_INVALID_ARGUMENT, "relation %s is fixed width", kName[r]);
    cudaStream_t s = (cudaStream_t)stream;
    launch_pad_rows(x.off, x.ent, x.rows, width, padded_out, counts_out, s);
    CK(cudaGetLastError());
    return TG_OK;
}

tg_status tg_get_tv(const tg_mesh *m, const int32_t **tv)
{
    if (!m || !tv) return fail(TG_ERR_INVALID_ARGUMENT, "NULL argument");
    *tv = reinterpret_cast<const int32_t *>(m->tvs);
    return TG_OK;
}

tg_status tg_critical_points(tg_mesh *m, const void *field, int field_type, int field_on_device,
                             uint32_t *classes_out, int out_on_device, void *stream)
{
    if (!m) return fail(TG_ERR_INVALID_ARGUMENT, "NULL argument");
    return critical_points_rows(m, 0, m->V, field, field_type, field_on_device, classes_out,
                                out_on_device, (cudaStream_t)stream);
}

tg_status tg_profile_kernel(const char *name)
{
    std::lock_guard<std::mutex> lk(tg::g_prof_mu);
    tg::g_prof_name = name ? name : "";
    tg::g_prof_on.store(!tg::g_prof_name.empty());
    return TG_OK;
}

tg_status tg_profile_read(double *total_ms, int64_t *launches, int reset)
{
    std::lock_guard<std::mutex> lk(tg::g_prof_mu);
    double ms = 0.0;
    for (auto &p : tg::g_prof_events) {
        CK(cudaEventSynchronize(p.b));
        float x = 0.f;
        CK(cudaEventElapsedTime(&x, p.a, p.b));
        ms += x;
    }
    if (total_ms) *total_ms = ms;
    if (launches) *launches = (int64_t)tg::g_prof_events.size();
    if (reset) {
        for (auto &p : tg::g_prof_events) {
            tg::g_prof_pool.push_back(p.a);
            tg::g_prof_pool.push_back(p.b);
        }
        tg::g_prof_events.clear();
    }
    return TG_OK;
}

int64_t tg_mesh_device_bytes(const tg_mesh *m)
{
    if (!m) return 0;
    int64_t b = m->T * 16;
    for (int r = 1; r < 14; r++) {
        const Rel &x = m->rel[r];
        if (!x.ready) continue;
        b += x.entries * 4;
        if (x.off) b += (x.rows + 1) * 8;
    }
    b += m->V * 8;
    if (m->lg_adj)
        b += link_entries(m, m->rel[TG_REL_VV].entries) * (m->wide_deg ? 12 : 8) + (m->V + 1) * 8;
    return b;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// internal: segments (tg_batch.cu)
tg_status tg::mesh_set_segments(tg_mesh *m, const int64_t *seg_c_host, int64_t n, cudaStream_t s)
{
    if (m->seg_c) cudaFreeAsync(m->seg_c, s);
    if (m->seg_ef) cudaFreeAsync(m->seg_ef, s);
    m->seg_c = m->seg_ef = nullptr;
    m->n_seg = n;
    TRY(dalloc(&m->seg_c, n + 1, s));
    TRY(dalloc(&m->seg_ef, 2 * (n + 1), s));
    CK(cudaMemcpyAsync(m->seg_c, seg_c_host, (size_t)(n + 1) * 8, cudaMemcpyHostToDevice, s));
    CK(cudaStreamSynchronize(s));  // the host array may go away
    return TG_OK;
}

const int64_t *tg::mesh_segment_ids(const tg_mesh *m) { return m->seg_ef; }
