// tg_api.cu -- host orchestration of the relation pipeline behind the C ABI
// declared in include/tetragpu.h.
//
// One tg_mesh owns its device buffers.  Memory comes from stream-ordered pools
// with an unlimited release threshold, so repeated extractions reuse blocks
// instead of returning them to the driver; a stage's arrays come out of one
// allocation each for what stays and what does not (some forty calls a step
// before: 357 -> 308 us at 24,576 cells, 24 requests to the server 5.6 -> 4.8
// ms).  tg_extract synchronises the stream at two points, to learn the
// edge/face/neighbour counts and then the CSR totals that size the outputs;
// everything between those points is asynchronous on the caller's stream.
#include <algorithm>
#include <atomic>
#include <climits>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <memory>
#include <mutex>
#include <new>
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
constexpr int64_t kFewRecords = 1 << 20;    // cells from which room for edge records is tight

// Where memory comes from: the device's default stream-ordered pool for what a
// mesh keeps, a pool of the library's own for temporaries.  Out of one pool, a
// stage's temporaries took the place of the relations of the mesh destroyed
// before, and relations of 5 GB found no room in one piece: the driver then
// remaps memory, 2.7 ms of a 128^3 step in a loop that keeps the previous mesh
// until the next is made.  Both pools keep what is freed for the next call (the
// temporaries' up to an eighth of the device's memory); when one cannot grow,
// the other gives back what it does not use.
struct Pools {
    cudaMemPool_t keep = nullptr, temp = nullptr;
    bool ready = false;
};
std::mutex g_pool_mu;
Pools g_pools[64];

const Pools *device_pools(int dev)
{
    if (dev < 0 || dev >= 64) return nullptr;
    std::lock_guard<std::mutex> lk(g_pool_mu);
    Pools &p = g_pools[dev];
    if (!p.ready) {
        uint64_t thr = UINT64_MAX;
        if (cudaDeviceGetDefaultMemPool(&p.keep, dev) != cudaSuccess) p.keep = nullptr;
        else cudaMemPoolSetAttribute(p.keep, cudaMemPoolAttrReleaseThreshold, &thr);
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        if (cudaMemPoolCreate(&p.temp, &props) != cudaSuccess) p.temp = nullptr;
        size_t free_b = 0, total_b = 0;
        if (cudaMemGetInfo(&free_b, &total_b) == cudaSuccess) thr = total_b / 8;
        if (p.temp) cudaMemPoolSetAttribute(p.temp, cudaMemPoolAttrReleaseThreshold, &thr);
        (void)cudaGetLastError();
        p.ready = true;
    }
    return p.keep && p.temp ? &p : nullptr;
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

// Device memory of a mesh: one allocation that several arrays share, given
// back (in the order of the mesh's last stream) when nothing refers to it.
struct Block {
    void *p = nullptr;
    const tg_mesh *m = nullptr;
    Block(void *q, const tg_mesh *mesh) : p(q), m(mesh) {}
    Block(const Block &) = delete;
    ~Block();
};
using BlockRef = std::shared_ptr<Block>;

struct Rel {
    int64_t rows = 0, entries = 0;
    int width = 0;
    int64_t *off = nullptr;
    int32_t *ent = nullptr;
    BlockRef hold_off, hold_ent;   // null for VT, which lies in the mesh's own block
    bool ready = false;
    uint32_t opts = 0;
};

const int kWidth[14] = {0, 6, 2, 0, 4, 3, 3, 2, 0, 0, 0, 0, 0, 0};
const char *kName[14] = {"validate", "TE", "EV", "ET", "TF", "FV", "FE",
                         "FT",       "EF", "VT", "TT", "FF", "EE", "VV"};

// Arrays that come out of one allocation, each on a 256-byte boundary: a call
// to the allocator costs a microsecond or more, and a stage has up to twenty
// arrays.  add() names the pointer to set.
struct Plan {
    void **at[32];
    size_t off[32];
    int n = 0;
    size_t bytes = 0;
    template <class T>
    void add(T **out, int64_t count)
    {
        at[n] = (void **)out;
        off[n++] = bytes;
        bytes += ((size_t)std::max<int64_t>(count, 1) * sizeof(T) + 255) & ~size_t(255);
    }
    void place(void *base) const
    {
        for (int i = 0; i < n; i++) *at[i] = (char *)base + off[i];
    }
};

// from the pool of kept memory (temp false) or of temporaries; need false: the
// caller can do without, so the call waits for nothing
cudaError_t take_cuda(size_t bytes, cudaStream_t s, void **out, bool temp, bool need)
{
    bytes = std::max<size_t>(bytes, 256);
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const Pools *p = device_pools(dev);
    e = p ? cudaMallocFromPoolAsync(out, bytes, temp ? p->temp : p->keep, s)
          : cudaMallocAsync(out, bytes, s);
    if (e == cudaErrorMemoryAllocation && p && need && !capturing(s)) {
        (void)cudaGetLastError();
        // what was freed on this stream counts once the stream is through; what
        // lies idle in either pool goes back to the device
        cudaStreamSynchronize(s);
        cudaMemPoolTrimTo(p->keep, 0);
        cudaMemPoolTrimTo(p->temp, 0);
        e = cudaMallocFromPoolAsync(out, bytes, temp ? p->temp : p->keep, s);
        if (e == cudaErrorMemoryAllocation) {
            // blocks freed on streams that are still running serve their pool only
            (void)cudaGetLastError();
            e = cudaMallocFromPoolAsync(out, bytes, temp ? p->keep : p->temp, s);
        }
    }
    return e;
}
tg_status take(size_t bytes, cudaStream_t s, void **out, bool temp = false, bool need = true)
{
    const cudaError_t e = take_cuda(bytes, s, out, temp, need);
    return e == cudaSuccess ? TG_OK : cuda_fail(e, "cudaMallocFromPoolAsync", __LINE__);
}

// a plan's arrays in a block
tg_status take_block(const Plan &plan, const tg_mesh *m, cudaStream_t s, BlockRef *out, bool need = true)
{
    if (plan.n == 0) return TG_OK;
    void *q = nullptr;
    TRY(take(plan.bytes, s, &q, false, need));
    try {
        *out = std::make_shared<Block>(q, m);
    } catch (const std::bad_alloc &) {
        cudaFreeAsync(q, s);
        return fail(TG_ERR_OUT_OF_MEMORY, "host memory");
    }
    plan.place(q);
    return TG_OK;
}

// Stream-ordered temporaries, freed when the stage ends.
struct Temps {
    cudaStream_t s;
    void *p[8];
    int n = 0;
    explicit Temps(cudaStream_t st) : s(st) {}
    ~Temps()
    {
        for (int i = 0; i < n; i++) cudaFreeAsync(p[i], s);
    }
    // the last plan's arrays go back
    void drop() { cudaFreeAsync(p[--n], s); }
    // a plan's arrays; the first zero_bytes zeroed
    tg_status add(const Plan &plan, size_t zero_bytes = 0, bool need = true)
    {
        if (plan.n == 0) return TG_OK;
        if (n >= 8) return fail(TG_ERR_UNSUPPORTED, "too many temporaries in one stage");
        void *q = nullptr;
        TRY(take(plan.bytes, s, &q, true, need));
        p[n++] = q;
        if (zero_bytes) {
            const cudaError_t e = cudaMemsetAsync(q, 0, zero_bytes, s);
            if (e != cudaSuccess) return cuda_fail(e, "cudaMemsetAsync", __LINE__);
        }
        plan.place(q);
        return TG_OK;
    }
};

}  // namespace

void tg::set_last_error(const char *msg) { g_err = msg; }

// VV by position (LinkGraph; off null: not there) and the link adjacency of
// critical points on it (adj null: not there)
struct LinkArrays {
    int64_t *off = nullptr;
    int32_t *ent = nullptr, *ids = nullptr;
    char *adj = nullptr;
};

struct tg_mesh {
    int device = 0;
    // stream of the last call, which frees are ordered on (classifications of
    // one mesh may come from several threads)
    std::atomic<cudaStream_t> last_stream{nullptr};
    // streams that smoothed over the mesh besides, with an event after that each
    // (lg_mu)
    std::vector<std::pair<cudaStream_t, cudaEvent_t>> readers;
    int64_t V = 0, T = 0, E = -1, F = -1;
    void *base = nullptr;       // one allocation: everything from here to VT, the scan workspace
                                // and the status word
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
    bool lg_plain = false;       // short rows: the link graph is VV as it is
    bool lg_by_id = false;       // ids keep neighbours as close as positions: positions are ids there
    LinkArrays lg;
    BlockRef lg_rows, lg_masks;
    std::mutex lg_mu;                // while a call looks for them or builds them
    cudaEvent_t lg_done = nullptr;   // after the build of either outside an extraction
    bool lg_pending = false;         // which has not been seen to be over
    DevStatus *st = nullptr;    // device
    DevStatus *st_host = nullptr;
    int64_t *sz_host = nullptr; // pinned slots for sizes read back at sync points
};

namespace {

Block::~Block()
{
    if (p) cudaFreeAsync(p, m->last_stream.load(std::memory_order_relaxed));
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

tg_status check_flags(const tg_mesh *m)
{
    const DevStatus &h = *m->st_host;
    const unsigned f = h.flags;
    if (!f) return TG_OK;
    auto lowest = [](int noted) { return INT_MAX - noted; };
    if (f & ST_BAD_ID)
        return fail(TG_ERR_INVALID_MESH, "cell %d has a vertex id outside [0, %lld)", lowest(h.bad_cell),
                    (long long)m->V);
    if (f & ST_DUP_VERTEX)
        return fail(TG_ERR_INVALID_MESH, "cell %d repeats a vertex", lowest(h.bad_cell));
    if (f & ST_NONMANIFOLD_FACE)
        return fail(TG_ERR_INVALID_MESH, "a face of cell %d lies in more than two cells",
                    lowest(h.bad_cell));
    if (f & ST_STAR_OVERFLOW)
        return fail(TG_ERR_UNSUPPORTED, "vertex %d: neighbour summary overflow", lowest(h.bad_vertex));
    if (f & ST_SCAN_STALLED)
        return fail(TG_ERR_CUDA, "a prefix scan gave up waiting for a preceding tile");
    return fail(TG_ERR_CUDA, "unexpected device status 0x%x", f);
}

inline uint32_t bit(int r) { return 1u << r; }

void set_fixed(tg_mesh *m, int r, int32_t *ent, int64_t rows, const BlockRef &hold)
{
    m->rel[r] = Rel();
    Rel &x = m->rel[r];
    x.rows = rows;
    x.width = kWidth[r];
    x.entries = rows * kWidth[r];
    x.ent = ent;
    x.hold_ent = hold;
    x.ready = true;
}

void set_csr(tg_mesh *m, int r, int64_t *off, int32_t *ent, int64_t rows, int64_t entries,
             const BlockRef &hold_off, const BlockRef &hold_ent, uint32_t opts = 0)
{
    m->rel[r] = Rel();
    Rel &x = m->rel[r];
    x.rows = rows;
    x.entries = entries;
    x.width = 0;
    x.off = off;
    x.ent = ent;
    x.hold_off = hold_off;
    x.hold_ent = hold_ent;
    x.ready = true;
    x.opts = opts;
}

// The link graph is built, and VV and it are smoothed over, on the caller's
// stream, which need not be the one the mesh's memory goes back on: what frees
// any of them waits for all of that first.
void await_readers(tg_mesh *m)
{
    const cudaStream_t s = m->last_stream.load(std::memory_order_relaxed);
    std::lock_guard<std::mutex> lk(m->lg_mu);
    if (m->lg_pending) cudaStreamWaitEvent(s, m->lg_done, 0);
    for (const auto &r : m->readers) cudaStreamWaitEvent(s, r.second, 0);
}

void free_link_graph(tg_mesh *m)
{
    m->lg_rows.reset();
    m->lg_masks.reset();
    m->lg = LinkArrays();
}

// entries of the link graph, at most: its rows are padded to multiples of eight
int64_t link_entries(const tg_mesh *m, int64_t nvv) { return m->lg_plain ? nvv : nvv + 7 * m->V; }

LinkGraph link_graph(const tg_mesh *m, const LinkArrays &a, int64_t nvv)
{
    const bool by_id = m->lg_by_id || m->lg_plain;
    return {m->V, link_entries(m, nvv), a.off, a.ent, by_id ? nullptr : m->vorder, by_id ? nullptr : m->vpos,
            a.adj, m->wide_deg || m->lg_plain, !m->lg_plain, a.ids, m->n_light, m->n_heavy};
}

// A call may use on one stream what an earlier call built on another.  (Under
// capture work outside of it cannot be waited for: the caller has then.)
tg_status link_built(tg_mesh *m, cudaStream_t s)
{
    if (!m->lg_done) CK(cudaEventCreateWithFlags(&m->lg_done, cudaEventDisableTiming));
    m->lg_pending = true;
    CK(cudaEventRecord(m->lg_done, s));
    return TG_OK;
}

tg_status link_wait(tg_mesh *m, cudaStream_t s)
{
    if (!m->lg_pending || capturing(s)) return TG_OK;
    if (cudaEventQuery(m->lg_done) == cudaSuccess) {
        m->lg_pending = false;
        return TG_OK;
    }
    (void)cudaGetLastError();   // not yet
    CK(cudaStreamWaitEvent(s, m->lg_done, 0));
    return TG_OK;
}

// The link adjacency of critical points: VV renumbered into the star
// processing order (what of it is missing) and its masks (unless only the rows
// are wanted), kept on the mesh.  alloc makes every buffer, the temporaries
// too, on the extraction's own stream (before a fork, so that a side stream may
// use them); build launches.
struct LinkBuild {
    LinkArrays a;
    int32_t *win = nullptr;
    bool rows = false, masks = false;
    ScanWorkspace own;   // recorded only
    // recorded: the calls are being recorded into a graph, which owns what it
    // allocates and may run later, often or never: nothing stays on the mesh,
    // and the scan has a workspace of its own (the mesh's alternates between two
    // buffers from call to call)
    tg_status alloc(tg_mesh *m, int64_t nvv, bool with_masks, Temps &tmp, cudaStream_t s,
                    bool recorded = false, bool need = true)
    {
        const int64_t n = link_entries(m, nvv);
        a = m->lg;
        if (m->lg_plain && !a.off) {
            a.off = m->rel[TG_REL_VV].off;
            a.ent = m->rel[TG_REL_VV].ent;
        }
        rows = !a.off;
        masks = with_masks && !a.adj;
        Plan t, keep_rows, keep_masks;
        Plan &r = recorded ? t : keep_rows, &k = recorded ? t : keep_masks;
        size_t zero = 0;
        if (recorded && rows) {
            own.job_words = scan_job_words(m->V);
            t.add(&own.buf, 2 * kMaxScanJobs * own.job_words);
            zero = t.bytes;
        }
        if (rows) {
            r.add(&a.off, m->V + 1);
            r.add(&a.ent, n);
            if (m->V < kOrderField && !m->lg_by_id) r.add(&a.ids, n);
        }
        if (masks) {
            t.add(&win, window_count(n, crit_window()) + 1);
            k.add(&a.adj, n * (m->wide_deg || m->lg_plain ? 8 : 4));
        }
        BlockRef held_rows, held_masks;
        TRY(tmp.add(t, zero, need));
        TRY(take_block(keep_masks, m, s, &held_masks, need));
        TRY(take_block(keep_rows, m, s, &held_rows, need));
        if (!recorded) {
            if (held_rows) m->lg_rows = held_rows;
            if (held_masks) m->lg_masks = held_masks;
            m->lg = a;
        }
        return TG_OK;
    }
    void build(tg_mesh *m, const int64_t *vv_off, const int32_t *vv, int64_t nvv, cudaStream_t s)
    {
        const LinkGraph g = link_graph(m, a, nvv);
        if (rows) {
            ScanJob job{vv_off, a.off, m->V, SCAN_ROW_PAD8, g.order};
            scan_batch(&job, 1, own.buf ? own : m->scan, m->st, s);
            launch_rows_in_order(vv_off, vv, g.order, g.vpos, m->V, a.off, a.ent, a.ids, win,
                                 masks ? window_count(g.n_ent, crit_window()) : 0, s);
        }
        if (masks) {
            if (!rows || m->V == 0)   // else beside the rows
                launch_window_starts(a.off, m->V, g.n_ent, crit_window(), win, s);
            launch_crit_adj(g, win, m->st, m->max_deg ? 1 : 0, s);
        }
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
        uint2 *erank, *frank, *brank;
        int64_t *vv_off;
        // FE is read off each face's first cell (k_face_fill), which the
        // face's FT row and the cell's TF row tell; EF off TF
        const bool need_tf = (mask & (TG_TF | TG_FE | TG_FF)) || want_tt_face;
        const bool need_ft = (mask & (TG_FT | TG_FE | TG_FF)) || want_tt_face;
        const bool need_te = mask & (TG_TE | TG_FE);
        const bool need_ev = mask & (TG_EV | TG_EE);
        // the edges by id: for everything per edge
        const bool need_edge = need_te || need_ev || (mask & (TG_ET | TG_EF));
        const bool want_ee = mask & TG_EE;
        StarPass sp{};
        HeavyStars hv{};
        int64_t *deg_sq, *eid_off = nullptr;
        BlockRef hold_vv_off, hold_vv, hold_tt, hold;
        {
            Plan o;
            o.add(&vv_off, V + 1);
            TRY(take_block(o, m, s, &hold_vv_off));
        }
        sp.n_light = m->n_light;
        sp.vorder = m->vorder;
        sp.vt_off = vt_off;
        sp.vt = vt;
        sp.tvs = m->tvs;
        sp.st = m->st;
        // room for records: a mesh has at most six edges a cell (cells that share
        // nothing).  Cells glued into manifolds have about T + 2V at most: E = V +
        // T + half the boundary faces less the Euler characteristic, and a closed
        // surface has two faces a vertex.  A large mesh that has more goes through
        // the pass again.  16 to 20 bytes each: all of six would be 0.9 GB more at
        // 128^3 cubes
        for (int64_t room = T >= kFewRecords ? std::min(6 * T, T + 2 * V) : 6 * T;; room = 6 * T) {
            sp.rec_last = (unsigned)std::max<int64_t>(room, 1) - 1;
            // the bitmaps the star pass sets bits in, the neighbour counts
            // and the record counter are zeroed
            Plan t;
            t.add(&sp.eflag, nwe);
            t.add(&sp.fflag, nwf);
            t.add(&sp.fbnd, nwf);
            t.add(&sp.deg_own, V);
            t.add(&sp.deg_in, V);
            t.add(&sp.vbnd, V);
            t.add(&sp.n_rec, 2);
            const size_t zero = t.bytes;
            t.add(&erank, nwe + 1);
            t.add(&frank, nwf + 1);
            t.add(&brank, nwf + 1);
            t.add(&deg_sq, V + 1);   // prefix of deg^2: its total sizes EE (sum deg^2 - 2E)
            if (want_ee) t.add(&eid_off, V + 1);   // EE's incident-edge rows are padded
            t.add(&sp.rec, room);
            t.add(&sp.place, room);
            if (m->n_wide > 0 || m->n_heavy > 0) t.add(&sp.rec_hi, room);
            if (m->n_wide > 0) t.add(&sp.wide, m->n_wide);
            if (m->n_heavy > 0) t.add(&hv.pairs, 3 * m->heavy_entries);
            if (need_tf || need_ft) t.add(&sp.fnext, 4 * T);
            TRY(tmp.add(t, zero));
            sp.n_wide = sp.n_rec + 1;
            launch_star(sp, s);
            launch_star_wide(sp, m->n_wide, s);
            if (m->n_heavy > 0) {
                hv.star = sp;
                hv.n_heavy = m->n_heavy;
                hv.heavy_off = m->heavy_off;
                launch_heavy(hv, s);
            }
            ScanJob jobs[6] = {{sp.deg_own, vv_off, V, SCAN_COUNT_I32, sp.deg_in},
                               {sp.eflag, erank, nwe, SCAN_POPC_RANK, nullptr},
                               {sp.fflag, frank, nwf, SCAN_POPC_RANK, nullptr},
                               {sp.fbnd, brank, nwf, SCAN_POPC_RANK, nullptr},
                               {sp.deg_own, deg_sq, V, SCAN_DEG_SQUARE, sp.deg_in},
                               {sp.deg_own, eid_off, V, SCAN_EID_WORDS, sp.deg_in}};
            scan_batch(jobs, want_ee ? 6 : 5, m->scan, m->st, s);

            // ---- the one synchronisation: edge, face, neighbour and boundary
            // counts size every output from here on ----
            const void *src[6] = {vv_off + V, &erank[nwe].y, &frank[nwf].y, &brank[nwf].y,
                                  deg_sq + V, eid_off + V};
            const bool w8[6] = {true, false, false, false, true, true};
            TRY(sync_read(m, s, want_ee ? 6 : 5, src, w8));
            if (m->st_host->flags) return check_flags(m);
            if (m->sz_host[1] <= room) break;
            tmp.drop();
        }
        m->max_deg = m->st_host->max_deg > kMaxDeg ? m->st_host->max_deg : 0;
        m->wide_deg = m->st_host->max_deg > kNarrowDeg;
        // rows of four entries or fewer on average would be half padding: 1.5M
        // cells that share nothing, VV and classification 1.90 ms padded, 1.39 as
        // it is
        m->lg_plain = m->sz_host[0] <= 4 * (m->n_light + m->n_heavy);
        const int largest_deg = m->st_host->max_deg;
        const int64_t nvv = m->sz_host[0];
        const int64_t E = m->sz_host[1], F = m->sz_host[2];
        const int64_t n_bnd = m->sz_host[3];  // boundary faces
        const int64_t sum_deg_sq = m->sz_host[4];
        m->E = E;
        m->F = F;
        if (m->seg_c) launch_seg_ranks(m->seg_c, m->n_seg, erank, frank, m->seg_ef, s);

        // ---- every other array: relations that were asked for in one block (TT,
        // which may be made again in its other form, and VV, which every
        // extraction makes, in their own), the rest temporary
        int32_t *vv, *ev = nullptr, *te = nullptr, *tf = nullptr, *fv = nullptr, *ft = nullptr;
        int32_t *et = nullptr, *ef = nullptr, *ee = nullptr, *ff = nullptr, *tt = nullptr, *fe = nullptr;
        int64_t *et_off = nullptr, *ef_off = nullptr, *ee_off = nullptr, *ff_off = nullptr;
        int64_t *tt_off = nullptr;
        uint32_t *eid = nullptr;
        int2 *inc = nullptr;
        EdgePass ep{};
        // CSR totals: ET = 6T, EF = 3F always; TT and FF from the
        // boundary-face count; EE deg(a) + deg(b) - 2 per edge (a,b)
        const int64_t n_et = 6 * T, n_ef = 3 * F, n_ee = sum_deg_sq - 2 * E;
        const int64_t n_tt = 4 * T - n_bnd, n_ff = 3 * (2 * F - n_bnd);
        {
            Plan t, o, ovv, ott;
            ovv.add(&vv, nvv);
            if (want_ee) {
                t.add(&eid, m->sz_host[5]);
                t.add(&inc, nvv);
            }
            if (need_edge) t.add(&ep.edge, E);
            if (need_edge && sp.rec_hi) t.add(&ep.edge_hi, E);
            if (need_ev) (mask & TG_EV ? o : t).add(&ev, 2 * E);
            if (need_te) (mask & TG_TE ? o : t).add(&te, 6 * T);
            if (need_tf) (mask & TG_TF ? o : t).add(&tf, 4 * T);
            if (need_ft) (mask & TG_FT ? o : t).add(&ft, 2 * F);
            if (mask & TG_FV) o.add(&fv, 3 * F);
            if (mask & TG_FE) o.add(&fe, 3 * F);
            if (mask & TG_ET) {
                o.add(&et_off, E + 1);
                o.add(&et, n_et);
            }
            if (mask & TG_EF) {
                o.add(&ef_off, E + 1);
                o.add(&ef, n_ef);
            }
            if (want_ee) {
                o.add(&ee_off, E + 1);
                o.add(&ee, n_ee);
            }
            if (mask & TG_FF) {
                o.add(&ff_off, F + 1);
                o.add(&ff, n_ff);
            }
            if (want_tt_face) {
                ott.add(&tt_off, T + 1);
                ott.add(&tt, n_tt);
            }
            TRY(take_block(ovv, m, s, &hold_vv));
            TRY(tmp.add(t));
            TRY(take_block(o, m, s, &hold));
            TRY(take_block(ott, m, s, &hold_tt));
        }
        if (T == 0 && tt_off) CK(cudaMemsetAsync(tt_off, 0, 8, s));
        if (T == 0 && ff_off) CK(cudaMemsetAsync(ff_off, 0, 8, s));

        // ---- ids: VV, EV, row lengths (per edge); TF, FT, FV (per cell)
        ep.E = E;
        ep.rec = sp.rec; ep.place = sp.place; ep.rec_hi = sp.rec_hi; ep.pairs = hv.pairs;
        ep.vt_off = vt_off; ep.vt = vt; ep.tvs = m->tvs;
        ep.erank = need_edge ? erank : nullptr;
        ep.frank = frank; ep.fbnd = sp.fbnd; ep.vbnd = sp.vbnd;
        ep.vv_off = vv_off; ep.inc = inc; ep.vv = vv;
        ep.count_ef = (mask & TG_EF) != 0;
        launch_edge_ids(ep, s);
        if (tf || ft || fv) launch_cell_faces(T, m->tvs, frank, sp.fnext, tf, ft, fv, s);
        // EV by the first pass over the edges by id; EE reads it
        const bool ev_with_rows = ev && !want_ee && (te || et || ef);
        if (et_off || ef_off || ee_off || (ev && !ev_with_rows))
            launch_edge_offsets(ep, et_off, ef_off, ee_off, ev_with_rows ? nullptr : ev, m->scan, m->st, s);
        if (inc) launch_inc_sort(vv_off, V, inc, vv, eid_off, eid, s);
        else launch_vv_sort(vv_off, V, nvv, vv, s);
        await_readers(m);
        set_csr(m, TG_REL_VV, vv_off, vv, V, nvv, hold_vv_off, hold_vv);
        free_link_graph(m);

        // ET and EF rows, the per-cell TT rows, the per-face FE / FF rows and on
        // request the link adjacency of critical points, on a side stream
        // beside EE (each reads only what the passes before it wrote)
        const bool prep_adj = (opts & TG_OPT_LINK_ADJACENCY) && (mask & TG_VV);
        LinkBuild lb;
        if (prep_adj) TRY(lb.alloc(m, nvv, true, tmp, s));
        if (te || fe || tt || ff_off || ff || et || ef || prep_adj) {
            const cudaStream_t s2 = side.fork();
            ep.ev = ev_with_rows ? ev : nullptr;
            ep.te = te; ep.et_off = et_off; ep.ef_off = ef_off; ep.et = et; ep.ef = ef;
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

        if (mask & TG_EV) set_fixed(m, TG_REL_EV, ev, E, hold);
        if (mask & TG_TE) set_fixed(m, TG_REL_TE, te, T, hold);
        if (mask & TG_TF) set_fixed(m, TG_REL_TF, tf, T, hold);
        if (mask & TG_FV) set_fixed(m, TG_REL_FV, fv, F, hold);
        if (mask & TG_FT) set_fixed(m, TG_REL_FT, ft, F, hold);
        if (fe) set_fixed(m, TG_REL_FE, fe, F, hold);
        if (et) set_csr(m, TG_REL_ET, et_off, et, E, n_et, hold, hold);
        if (ef) set_csr(m, TG_REL_EF, ef_off, ef, E, n_ef, hold, hold);
        if (ee) set_csr(m, TG_REL_EE, ee_off, ee, E, n_ee, hold, hold);
        if (ff) set_csr(m, TG_REL_FF, ff_off, ff, F, n_ff, hold, hold);
        if (tt) set_csr(m, TG_REL_TT, tt_off, tt, T, n_tt, hold_tt, hold_tt, 0);
    }

    if ((mask & TG_TT) && tt_vertex) {
        int32_t *cnt, *tt, *far = nullptr, *n_far = nullptr;
        int64_t *tt_off;
        BlockRef hold_off, hold_ent;
        Plan t, o;
        size_t zero = 0;
        if (const int64_t n = tt_far_tiles(T, V)) {
            t.add(&n_far, 1);
            zero = t.bytes;
            t.add(&far, n);
        }
        t.add(&cnt, T);
        o.add(&tt_off, T + 1);
        TRY(tmp.add(t, zero));
        TRY(take_block(o, m, s, &hold_off));
        launch_tt_vertex_count(m->tvs, T, V, vt_off, vt, far, n_far, cnt, s);
        ScanJob job{cnt, tt_off, T, SCAN_COUNT_I32, nullptr};
        scan_batch(&job, 1, m->scan, m->st, s);
        const void *src[2] = {tt_off + T, n_far};
        const bool w8[2] = {true, false};
        TRY(sync_read(m, s, far ? 2 : 1, src, w8));
        const int64_t listed = far ? m->sz_host[1] : 0;
        Plan e;
        e.add(&tt, m->sz_host[0]);
        TRY(take_block(e, m, s, &hold_ent));
        launch_tt_vertex_fill(m->tvs, T, V, vt_off, vt, far, n_far, listed, tt_off, tt, s);
        set_csr(m, TG_REL_TT, tt_off, tt, T, m->sz_host[0], hold_off, hold_ent,
                TG_OPT_TT_VERTEX_SHARING);
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
    Temps adj_tmp(s), tmp(s);
    std::unique_lock<std::mutex> lk(m->lg_mu);
    LinkArrays lg = m->lg;
    TRY(link_wait(m, s));
    if (!lg.adj) {
        // VV rows longer than the adjacency masks take the heavy path of the
        // classification, so no status read-back here
        const bool recorded = capturing(s);
        LinkBuild lb;
        TRY(lb.alloc(m, vv.entries, true, adj_tmp, s, recorded));
        lb.build(m, vv.off, vv.ent, vv.entries, s);
        if (!recorded) TRY(link_built(m, s));
        lg = lb.a;
    }
    lk.unlock();
    const LinkGraph g = link_graph(m, lg, vv.entries);
    const size_t esz = field_type == TG_FIELD_F64 ? 8 : 4;
    const void *f = field;
    uint32_t *out = classes_out;
    char *d_field, *ordered = nullptr;
    int32_t *list, *n_list, *scratch;
    // vertices of more than kMaxDeg neighbours: at most one per kMaxDeg + 1 VV
    // entries
    const int64_t max_listed = std::min<int64_t>(nv, vv.entries / (kMaxDeg + 1) + 1);
    {
        Plan t;
        size_t zero = 0;
        if (m->max_deg) {
            t.add(&n_list, 1);
            zero = t.bytes;
            t.add(&list, max_listed);
            t.add(&scratch, vv.entries);
        }
        if (!field_on_device) t.add(&d_field, nv * (int64_t)esz);
        if (!out_on_device) t.add(&out, 3 * nv);
        TRY(tmp.add(t, zero));
    }
    // the field in processing order is worth a buffer, not an error: without
    // the memory, or recorded (no allocations in the graph), by vertex
    Temps opt(s);
    if (classify_orders_field(nv) && g.order && !capturing(s)) {
        Plan o;
        o.add(&ordered, m->V * (int64_t)esz);
        const std::string before = g_err;
        if (opt.add(o, 0, false) != TG_OK) {
            ordered = nullptr;
            g_err = before;
        }
    }
    if (!field_on_device) {
        CK(cudaMemcpyAsync(d_field, field, nv * esz, cudaMemcpyHostToDevice, s));
        f = d_field;
    }
    launch_crit_classify(g, f, field_type, ordered, v0, nv, out, s);
    if (m->max_deg)
        launch_crit_heavy(vv.off, vv.ent, v0, nv, max_listed, f, field_type, out, list, n_list,
                          scratch, s);
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
    const cudaStream_t s = m->last_stream.load(std::memory_order_relaxed);
    await_readers(m);
    for (auto &r : m->rel) r = Rel();
    free_link_graph(m);
    if (m->seg_c) cudaFreeAsync(m->seg_c, s);
    if (m->seg_ef) cudaFreeAsync(m->seg_ef, s);
    if (m->base) {
        // after the last scan, whichever stream it ran on
        if (m->scan.used && m->scan.last != s) cudaStreamWaitEvent(s, m->scan.done, 0);
        cudaFreeAsync(m->base, s);
    }
    cudaStreamSynchronize(s);  // no copy into the pinned slots is still in flight
    if (m->scan.done) cudaEventDestroy(m->scan.done);
    if (m->lg_done) cudaEventDestroy(m->lg_done);
    for (const auto &r : m->readers) cudaEventDestroy(r.second);
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
    m->st_host = (DevStatus *)g_pinned.get();
    m->sz_host = (int64_t *)g_pinned.get();
    if (!m->st_host || !m->sz_host) return fail(TG_ERR_OUT_OF_MEMORY, "pinned host memory");
    // the scan workspace of every later scan on the mesh, zeroed once
    m->scan.job_words = std::max(scan_job_words(std::max(std::max(V, T), (6 * T + 31) / 32)),
                                 (edge_offsets_words(6 * T) + kMaxScanJobs - 1) / kMaxScanJobs);
    int64_t *vt_off;
    int32_t *vt;
    {
        Plan b;
        b.add(&m->st, 1);
        b.add(&m->scan.buf, 2 * kMaxScanJobs * m->scan.job_words);
        const size_t zero = b.bytes;
        b.add(&m->tvs, T);
        b.add(&vt_off, V + 1);
        b.add(&vt, 4 * T);
        b.add(&m->vorder, V);
        b.add(&m->vpos, V);
        b.add(&m->heavy_off, 4 * T / (kMaxStar + 1) + 1);
        TRY(take(b.bytes, s, &m->base));
        b.place(m->base);
        CK(cudaMemsetAsync(m->base, 0, zero, s));
    }
    const int32_t *src = tv;
    if (!on_device && T > 0) {
        CK(cudaMemcpyAsync(m->tvs, tv, (size_t)T * 16, cudaMemcpyHostToDevice, s));
        src = reinterpret_cast<const int32_t *>(m->tvs);
    }
    CK(cudaEventCreateWithFlags(&m->scan.done, cudaEventDisableTiming));
    Temps tmp(s);
    const int64_t nwk = (4 * T + 31) / 32, nwh = (V + 31) / 32;
    int32_t *deg_t, *heavy_cnt;
    uint32_t *vflag, *hflag;
    VtOrder vo{};
    uint2 *vrank, *hrank;
    int64_t *vkey;
    {
        // the per-vertex cell counts and the bitmaps of first cells and of
        // heavy vertices are zeroed
        Plan t;
        t.add(&deg_t, V);
        t.add(&vflag, nwk);
        t.add(&hflag, nwh);
        t.add(&heavy_cnt, 6);
        const size_t zero = t.bytes;
        t.add(&vo.place, T);
        t.add(&vo.head, canon_tiles(T));
        t.add(&vo.verts, canon_tiles(T) * canon_pairs());
        t.add(&vrank, nwk + 1);
        t.add(&hrank, nwh + 1);
        t.add(&vkey, V);
        TRY(tmp.add(t, zero));
    }
    launch_canon(src, T, V, m->tvs, deg_t, vo, m->st, s);
    ScanJob job{deg_t, vt_off, V, SCAN_COUNT_I32, nullptr};
    scan_batch(&job, 1, m->scan, m->st, s);
    launch_vt_fill(T, vt_off, vo, vt, s);
    // VT row sort, which also marks each vertex's star-order key; then the
    // star processing order
    launch_vt_sort(vt_off, vt, V, 4 * T, m->tvs, vflag, vkey, hflag, heavy_cnt, s);
    const ScanJob jf[2] = {{vflag, vrank, nwk, SCAN_POPC_RANK, nullptr},
                           {hflag, hrank, nwh, SCAN_POPC_RANK, nullptr}};
    scan_batch(jf, 2, m->scan, m->st, s);
    launch_vorder_place(vt_off, V, vkey, vrank, nwk, hrank, heavy_cnt, m->heavy_off, m->vorder, m->vpos, s);
    if (V >= kOrderField)
        launch_order_lines(V, vt_off, vt, m->tvs, m->vorder, m->vpos, heavy_cnt + 4, s);
    CK(cudaGetLastError());
    set_csr(m, TG_REL_VT, vt_off, vt, V, 4 * T, nullptr, nullptr);
    // vertices with light stars, heavy ones, the heavy stars' entries and
    // the light stars of more than 31 cells; what k_order_lines counted
    const void *rd[6] = {&vrank[nwk].y, heavy_cnt, heavy_cnt + 1, heavy_cnt + 2, heavy_cnt + 4, heavy_cnt + 5};
    const bool w8[6] = {};
    TRY(sync_read(m, s, 6, rd, w8));
    m->n_light = T ? m->sz_host[0] : 0;
    m->n_heavy = T ? m->sz_host[1] : 0;
    m->heavy_entries = T ? m->sz_host[2] : 0;
    m->n_wide = T ? m->sz_host[3] : 0;
    // VV in star order pays where that keeps a run of vertices' neighbours on well
    // fewer lines than ids do.  By id and by position on 64^3 cubes: 14 and 14
    // with both in order, 274 and 14 with ids permuted, 14 and 155 with cells
    // scattered, 274 and 155 with both; on a Delaunay mesh of random points 292
    // and 88.  A field on 64^3, cells scattered and ids in order: 18 us by id, 30
    // by position.  The count is a launch: 4 us of 100 to 200 at 64^3
    m->lg_by_id = 2 * m->sz_host[5] > m->sz_host[4];
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
        TRY(take(b, s, (void **)&d, true));
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
        TRY(take((size_t)j.start[j.n] * 4, s, (void **)&d, true));
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
        if (!out_on_device) {
            Plan t;
            t.add(&dst, x.entries);
            TRY(tmp.add(t));
        }
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
    const int64_t n = link_entries(m, m->rel[TG_REL_VV].entries);
    if (m->lg.off && !m->lg_plain) b += n * (m->lg.ids ? 8 : 4) + (m->V + 1) * 8;
    if (m->lg.adj) b += n * (m->wide_deg || m->lg_plain ? 8 : 4);
    return b;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// internal: VV by position (tg_consumers.cu)
bool tg::capturing(cudaStream_t s)
{
    cudaStreamCaptureStatus c;
    if (cudaStreamIsCapturing(s, &c) == cudaSuccess) return c != cudaStreamCaptureStatusNone;
    (void)cudaGetLastError();   // the legacy stream, while another is capturing
    return true;
}

tg_status tg::link_rows(tg_mesh *m, cudaStream_t s, LinkGraph *out)
{
    *out = LinkGraph{};
    if (m->lg_by_id || m->lg_plain) return TG_OK;
    const Rel &vv = m->rel[TG_REL_VV];
    std::lock_guard<std::mutex> lk(m->lg_mu);
    if (m->lg.off) {
        TRY(link_wait(m, s));
    } else {
        Temps tmp(s);
        LinkBuild lb;
        const std::string before = g_err;
        if (lb.alloc(m, vv.entries, false, tmp, s, false, false) != TG_OK) {
            g_err = before;
            return TG_OK;   // without the memory: none
        }
        lb.build(m, vv.off, vv.ent, vv.entries, s);
        TRY(link_built(m, s));
    }
    *out = link_graph(m, m->lg, vv.entries);
    return TG_OK;
}

tg_status tg::note_reader(tg_mesh *m, cudaStream_t s, bool rows)
{
    // on the mesh's own stream what frees VV comes later anyway (the rows may be
    // freed from another).  (Asking whether a stream is being recorded takes a
    // microsecond, a tenth of a short call.)
    if (!rows && (m->last_stream.load(std::memory_order_relaxed) == s || capturing(s))) return TG_OK;
    std::lock_guard<std::mutex> lk(m->lg_mu);
    cudaEvent_t done = nullptr;
    for (const auto &r : m->readers)
        if (r.first == s) done = r.second;
    if (!done) {
        CK(cudaEventCreateWithFlags(&done, cudaEventDisableTiming));
        try {
            m->readers.push_back({s, done});
        } catch (const std::bad_alloc &) {
            cudaEventDestroy(done);
            return fail(TG_ERR_OUT_OF_MEMORY, "host memory");
        }
    }
    CK(cudaEventRecord(done, s));
    return TG_OK;
}

// internal: temporaries and segments (tg_batch.cu)
cudaError_t tg::take_temp(size_t bytes, cudaStream_t s, void **out)
{
    return take_cuda(bytes, s, out, true, true);
}

tg_status tg::mesh_set_segments(tg_mesh *m, const int64_t *seg_c_host, int64_t n, cudaStream_t s)
{
    if (m->seg_c) cudaFreeAsync(m->seg_c, s);
    if (m->seg_ef) cudaFreeAsync(m->seg_ef, s);
    m->seg_c = m->seg_ef = nullptr;
    m->n_seg = n;
    TRY(take((size_t)(n + 1) * 8, s, (void **)&m->seg_c));
    TRY(take((size_t)(n + 1) * 16, s, (void **)&m->seg_ef));
    CK(cudaMemcpyAsync(m->seg_c, seg_c_host, (size_t)(n + 1) * 8, cudaMemcpyHostToDevice, s));
    CK(cudaStreamSynchronize(s));  // the host array may go away
    return TG_OK;
}

const int64_t *tg::mesh_segment_ids(const tg_mesh *m) { return m->seg_ef; }
