// tg_scan.cu -- batched exclusive scans in one pass (decoupled look-back).
//
// Every CSR offset array and every bit-rank prefix of the pipeline comes out
// of here.  Up to kMaxScanJobs independent arrays are scanned by one launch
// (blockIdx.y selects the array), reading each input once.  A block takes the
// next tile of its array in start order (a ticket), sums the tile, publishes
// the sum, and adds the published sums of the tiles before it until it meets
// one whose inclusive prefix is already known (Merrill and Garland's
// single-pass scan).  A block waits only on tiles whose blocks started before
// it, so every wait ends; it is bounded all the same: after kLookbackPolls
// polls the block records ST_SCAN_STALLED in the mesh status (reported at the
// next status read-back) and goes on.
//
// A warp takes rows of 64 elements, two neighbours to a lane, so that its loads
// and stores are whole lines: the four scans of an extraction of all relations
// at 128^3 cubes take 105 us (140 with eight consecutive elements to a thread,
// 128 with four elements a thread and six blocks to an SM; 114 without the bound
// of five blocks, which spills 4 bytes a thread); what is left is the look-back's
// latency.
#include "tg_internal.h"

namespace tg {
namespace {

constexpr int kThreads = 256;
constexpr int kItems = 8;
constexpr int kTile = kThreads * kItems;  // 2048 elements per tile

struct ScanParams {
    ScanJob job[kMaxScanJobs];
    // per array: one word per tile (sum << 2 | 1 once the tile's sum is
    // published, inclusive prefix << 2 | 2 once that is known, 0 before),
    // then the ticket counter; zeroed before the launch
    unsigned long long *tiles[kMaxScanJobs];
    unsigned long long *next;   // the other buffer, zeroed here for the next scan
    int64_t next_words;
    unsigned *err;
    int *max_deg;
    int n_jobs;
};

// the value of element i, whose words are x and (in2) y
__device__ __forceinline__ int64_t value(const ScanJob &j, unsigned word, unsigned word2, int &largest)
{
    if (j.kind == SCAN_POPC_RANK) return (int64_t)__popc(word);
    const int x = (int)(word + word2);
    if (j.kind == SCAN_COUNT_I32) return x;
    if (j.kind == SCAN_ROW_PAD8) return pad8(x);
    if (j.kind == SCAN_EID_WORDS) return eid_words(x);
    largest = max(largest, x);
    return (int64_t)x * x;
}

// elements i and i + 1 (i even), those past the end 0
__device__ __forceinline__ uint2 load_two(const void *in, int64_t i, int64_t n)
{
    if (i + 1 < n) return __ldg(reinterpret_cast<const uint2 *>((const unsigned *)in + i));
    return make_uint2(i < n ? __ldg((const unsigned *)in + i) : 0u, 0u);
}

// SCAN_ROW_PAD8: the lengths of rows in2[i] and in2[i + 1] of the CSR offsets (in2
// null: rows i and i + 1)
__device__ __forceinline__ uint2 load_rows(const ScanJob &j, int64_t i)
{
    const int64_t *off = (const int64_t *)j.in;
    const uint2 r = j.in2 ? load_two(j.in2, i, j.n) : make_uint2((unsigned)i, (unsigned)i + 1u);
    uint2 len = make_uint2(0u, 0u);
    if (i < j.n) len.x = (unsigned)(__ldg(off + r.x + 1) - __ldg(off + r.x));
    if (i + 1 < j.n) len.y = (unsigned)(__ldg(off + r.y + 1) - __ldg(off + r.y));
    return len;
}

// the sums before elements i and i + 1, as they are stored (i even; element n
// is the closing one, stored by itself)
__device__ __forceinline__ void store_two(const ScanJob &j, int64_t i, uint2 w, int64_t a, int64_t b)
{
    if (i >= j.n) return;
    longlong2 v = make_longlong2(a, b);
    if (j.kind == SCAN_POPC_RANK)   // {bits, prefix}
        v = make_longlong2((long long)((unsigned long long)a << 32 | w.x),
                           (long long)((unsigned long long)b << 32 | w.y));
    int64_t *out = (int64_t *)j.out + i;
    if (i + 1 < j.n) *reinterpret_cast<longlong2 *>(out) = v;
    else *out = v.x;
}

__global__ void __launch_bounds__(kThreads, 5) k_scan(ScanParams p)
{
    griddep_wait();
    const int jb = blockIdx.y;
    if (jb >= p.n_jobs) return;
    const ScanJob &j = p.job[jb];
    const int64_t ntiles = (j.n + kTile - 1) / kTile;
    unsigned long long *w = p.tiles[jb];
    {
        const int64_t nthreads = (int64_t)gridDim.x * gridDim.y * blockDim.x;
        const int64_t t0 = ((int64_t)blockIdx.y * gridDim.x + blockIdx.x) * blockDim.x + threadIdx.x;
        for (int64_t i = t0; i < p.next_words; i += nthreads) p.next[i] = 0ull;
    }
    __shared__ int64_t s_warp[kThreads / 32], s_tile, s_prefix;
    if (threadIdx.x == 0) s_tile = (int64_t)atomicAdd(w + ntiles, 1ull);   // the ticket
    __syncthreads();
    const int64_t tile = s_tile;
    if (ntiles == 0) {   // an empty array: its total alone
        if (tile == 0 && threadIdx.x == 0) *(int64_t *)j.out = 0;
        return;
    }
    if (tile >= ntiles) return;   // a surplus block of a shorter array
    // rows of 64 elements to a warp, two neighbours to a lane
    constexpr int kRows = kItems / 2;
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const int64_t k0 = tile * kTile + wp * (32 * kItems) + 2 * lane;
    uint2 word[kRows];
    int64_t before[kRows], first[kRows], run = 0;
    int largest = 0;
#pragma unroll
    for (int r = 0; r < kRows; r++)
        word[r] = j.kind == SCAN_ROW_PAD8 ? load_rows(j, k0 + 64 * r) : load_two(j.in, k0 + 64 * r, j.n);
#pragma unroll
    for (int r = 0; r < kRows; r++) {
        const uint2 more = j.in2 && j.kind != SCAN_ROW_PAD8 ? load_two(j.in2, k0 + 64 * r, j.n) : make_uint2(0u, 0u);
        const bool b0 = k0 + 64 * r < j.n, b1 = k0 + 64 * r + 1 < j.n;
        first[r] = b0 ? value(j, word[r].x, more.x, largest) : 0;
        const int64_t two = first[r] + (b1 ? value(j, word[r].y, more.y, largest) : 0);
        int64_t x = two;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int64_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        before[r] = run + x - two;
        run += __shfl_sync(0xffffffffu, x, 31);
    }
    if (j.kind == SCAN_DEG_SQUARE) {   // block-uniform
        largest = __reduce_max_sync(0xffffffffu, largest);
        if (lane == 0 && largest > *(volatile int *)p.max_deg) atomicMax(p.max_deg, largest);
    }
    if (lane == 0) s_warp[wp] = run;
    __syncthreads();
    int64_t total = 0, warps = 0;
#pragma unroll
    for (int i = 0; i < kThreads / 32; i++) {
        if (i == wp) warps = total;
        total += s_warp[i];
    }
    if (wp == 0) {
        const int64_t pre = look_back(w, tile, total, p.err);
        if (lane == 0) s_prefix = pre;
    }
    __syncthreads();
    const int64_t base = s_prefix + warps;
#pragma unroll
    for (int r = 0; r < kRows; r++)
        store_two(j, k0 + 64 * r, word[r], base + before[r], base + before[r] + first[r]);
    if (tile == ntiles - 1 && threadIdx.x == 0) {
        const int64_t all = s_prefix + total;
        ((int64_t *)j.out)[j.n] = j.kind == SCAN_POPC_RANK ? all << 32 : all;
    }
}

}  // namespace

int64_t scan_job_words(int64_t max_n)
{
    return (max_n + kTile - 1) / kTile + 1;
}

void scan_batch(const ScanJob *jobs, int n_jobs, ScanWorkspace &ws, DevStatus *st, cudaStream_t s)
{
    if (n_jobs <= 0) return;
    ScanParams p{};
    p.n_jobs = n_jobs;
    p.err = &st->flags;
    p.max_deg = &st->max_deg;
    int64_t max_tiles = 1;
    unsigned long long *cur;
    scan_ws_begin(ws, s, &cur, &p.next, &p.next_words);
    for (int i = 0; i < n_jobs; i++) {
        p.job[i] = jobs[i];
        p.tiles[i] = cur + (int64_t)i * ws.job_words;
        const int64_t t = (jobs[i].n + kTile - 1) / kTile;
        if (t > max_tiles) max_tiles = t;
    }
    dim3 grid((unsigned)max_tiles, n_jobs);
    {
        Launch L("k_scan", s);
        launch_pdl(k_scan, grid, kThreads, 0, s, p);
    }
    scan_ws_end(ws, s);
}

void scan_ws_begin(ScanWorkspace &ws, cudaStream_t s, unsigned long long **cur,
                   unsigned long long **next, int64_t *next_words)
{
    const int64_t words = (int64_t)kMaxScanJobs * ws.job_words;
    *cur = ws.buf + (int64_t)ws.cur * words;
    *next = ws.buf + (int64_t)(ws.cur ^ 1) * words;
    *next_words = words;
    if (ws.used && ws.last != s) cudaStreamWaitEvent(s, ws.done, 0);
}

void scan_ws_end(ScanWorkspace &ws, cudaStream_t s)
{
    if (ws.done) cudaEventRecord(ws.done, s);
    ws.last = s;
    ws.used = true;
    ws.cur ^= 1;
}

}  // namespace tg
