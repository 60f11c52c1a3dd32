// tg_rowsort.h -- ascending sorts of short CSR rows in registers.
//
// A row of at most 32 entries is one thread's work: its entries go through a
// sorting network held in registers (Batcher's odd-even merge sort, the
// comparators reaching past N dropped: the padding is the largest key and
// never moves), so sorting costs a fixed number of min / max pairs, no
// data-dependent loop and no lanes idling on the rows' different lengths.
#pragma once

#include <climits>
#include <utility>

#include <cuda_runtime.h>

namespace tg {

constexpr int net_size(int n, bool count_only, int want, bool second)
{
    int p2 = 1;
    while (p2 < n) p2 *= 2;
    int c = 0;
    for (int p = 1; p < p2; p *= 2)
        for (int k = p; k >= 1; k /= 2)
            for (int j = k % p; j + k < p2; j += 2 * k)
                for (int i = 0; i < k; i++) {
                    const int a = i + j, b = i + j + k;
                    if (b >= n || a / (2 * p) != b / (2 * p)) continue;
                    if (!count_only && c == want) return second ? b : a;
                    c++;
                }
    return c;
}

template <int N>
struct SortNet {
    static constexpr int kCount = net_size(N, true, 0, false);
    template <int A, int B>
    static __device__ __forceinline__ void step(int (&x)[N])
    {
        const int lo = min(x[A], x[B]);
        x[B] = max(x[A], x[B]);
        x[A] = lo;
    }
    template <int... I>
    static __device__ __forceinline__ void run(int (&x)[N], std::integer_sequence<int, I...>)
    {
        (step<net_size(N, false, I, false), net_size(N, false, I, true)>(x), ...);
    }
    static __device__ __forceinline__ void sort(int (&x)[N])
    {
        run(x, std::make_integer_sequence<int, kCount>());
    }
};

// row[0 .. n), n <= N, ascending (one thread)
template <int N>
__device__ __forceinline__ void sort_row_net(int *row, int n)
{
    int x[N];
#pragma unroll
    for (int k = 0; k < N; k++) x[k] = k < n ? row[k] : INT_MAX;
    SortNet<N>::sort(x);
#pragma unroll
    for (int k = 0; k < N; k++)
        if (k < n) row[k] = x[k];
}

// heapsort: O(n log n) whatever the input, no recursion, no extra memory
// (rows too long for the registers; rare)
template <typename T, typename Less>
__device__ void sift_down(T *a, int root, int n, Less less)
{
    while (true) {
        int child = 2 * root + 1;
        if (child >= n) return;
        if (child + 1 < n && less(a[child], a[child + 1])) child++;
        if (!less(a[root], a[child])) return;
        const T t = a[root];
        a[root] = a[child];
        a[child] = t;
        root = child;
    }
}
template <typename T, typename Less>
__device__ void heap_sort(T *a, int n, Less less)
{
    for (int start = n / 2 - 1; start >= 0; start--) sift_down(a, start, n, less);
    for (int end = n - 1; end > 0; end--) {
        const T t = a[0];
        a[0] = a[end];
        a[end] = t;
        sift_down(a, 0, end, less);
    }
}

// One row per lane, row[0 .. n) in shared or global memory (n = 0: none): the
// warp's longest row of at most 32 entries picks the network (the branch is
// warp-uniform), rows of 33 to 64 entries are ranked by the whole warp one
// after another, longer ones by their lane.  All 32 lanes call it.
__device__ __forceinline__ void sort_rows_warp(int *row, int n)
{
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int m = n <= 32 ? n : 0;
    if (__any_sync(kAll, m > 24))
        sort_row_net<32>(row, m);
    else if (__any_sync(kAll, m > 16))
        sort_row_net<24>(row, m);
    else if (__any_sync(kAll, m > 8))
        sort_row_net<16>(row, m);
    else if (__any_sync(kAll, m > 1))   // (rows of cells that share little)
        sort_row_net<8>(row, m);
    for (unsigned mid = __ballot_sync(kAll, n > 32 && n <= 64); mid; mid &= mid - 1) {
        const int src = __ffs(mid) - 1;
        int *r = (int *)__shfl_sync(kAll, (unsigned long long)row, src);
        const int len = __shfl_sync(kAll, n, src);
        const int x = r[lane], y = lane + 32 < len ? r[lane + 32] : INT_MAX;
        int rx = 0, ry = 0;
        for (int j = 0; j < len; j++) {
            const int z = __shfl_sync(kAll, j < 32 ? x : y, j & 31);
            // ties (none in VT or in incident edges) by position
            rx += z < x || (z == x && j < lane);
            ry += z < y || (z == y && j < lane + 32);
        }
        __syncwarp();
        r[rx] = x;
        if (lane + 32 < len) r[ry] = y;
        __syncwarp();
    }
    if (n > 64) heap_sort(row, n, [](int a, int b) { return a < b; });
}

}  // namespace tg
