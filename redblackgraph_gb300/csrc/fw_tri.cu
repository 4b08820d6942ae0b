// fw_tri.cu -- dense closure of acyclic matrices by the DAG closure.
//
// The reference's warshall (redblackgraph/core/src/redblackgraph/warshall.c.in:88-106) runs the
// sequential loop  for k, i, j: W(i, j) = W(i, j) (+) W(i, k) (x) W(k, j)  over the whole matrix.
// When every off-diagonal entry lies below the diagonal (an edge i -> k only for k < i, as in a
// pedigree whose vertices are numbered oldest first), a path from i to k passes only vertices
// numbered above k, none of which an earlier step has used: before step k, W(i, k) is still the
// input A(i, k), while row k is already final (every path from k descends through vertices
// below k).  Step k therefore adds A(i, k) (x) C(k, .) to the rows of k's children, and the
// closure is the DAG recurrence  C(i, .) = A(i, .) (+) sum over parents k of A(i, k) (x) C(k, .)
// that the closure by levels computes.  Above the diagonal (edges to higher numbers) it is the
// mirror image: before step k, W(i, k) = C(i, k) and W(k, j) = A(k, j).
//
// In the clean regime (off-diagonal values 0 or >= 2, diagonal in {-1, 0, 1}) products with the
// diagonal change nothing and a cell only decreases once it holds a value, so the largest value
// the loop ever writes -- the diameter's source -- is, per cell, its first value: A(i, j), else
// the product of the first step that reaches the cell.  Below the diagonal that is the smallest
// parent k of i with j in C(k); above it, the smallest k in C(i) with j a parent of k.  A
// product whose most significant bit may reach bit 31 sends the matrix to the blocked kernels
// (which report the reference's overflow or wrap for 32-bit storage, and carry 64-bit values
// exactly), as does anything outside the clean regime or the 32-bit value range, a row of more
// than TRI_CAP entries or n > 8192.  For 64-bit storage no product below bit 31 can overflow, so
// the values, the diameter and the absence of errors are the reference's as well.  A matrix the
// closure went through whose loop does compute a product reaching bit 31 is reported as such
// (TRI_TOP_BIT): its caller skips the 32-bit lanes, which could only report that risk.
//
// A matrix with entries on both sides of the diagonal (an acyclic graph in any numbering) has the
// same closure values, but which product reaches a cell first depends on the numbering: two searches
// from every vertex k through the vertices below k give step k's products, hence the exact product
// MSBs and first values.  A
// vertex the closure by levels never places (a cycle, or below one) sends its matrix on.
//
// Pipeline (one call, every decision on the device): scan the dense rows (clean-regime test,
// which side of the diagonal, up to TRI_CAP off-diagonal entries per row) -> CSR of the
// candidate matrices with batch-global row numbers -> closure by levels -> for matrices in any
// numbering, the searches from every vertex -> per-row statistics
// (largest product MSB, largest first-value MSB) -> the dense rows of the accepted matrices
// written from the closure rows -> one result record per matrix, read back once.  Scratch is
// carved from the caller's workspace; with RBG_MODE_GRAPH the sequence, level loop included (a
// while node the device ends), is one CUDA graph replayed for the same layout.
#include <cuda_runtime.h>
#include <cub/cub.cuh>
#include <string.h>
#include <algorithm>
#include <mutex>
#include <vector>
#include "rbg_internal.cuh"
#include "dag_rows.cuh"

namespace rbg {
namespace {

constexpr int TRI_ROWS = 8;                  // rows per CTA, one warp each
constexpr int TRI_THREADS = 32 * TRI_ROWS;
constexpr int TRI_CAP = 16;                  // off-diagonal entries per row the scan keeps
constexpr int64_t TRI_MAX_N = DAG_MAX_N;     // rows of a matrix on this path (bitmap size)
constexpr int TRI_BM_WORDS = (int)(TRI_MAX_N / 32);
constexpr unsigned TF_UNCLEAN = 1u, TF_BELOW = 2u, TF_ABOVE = 4u, TF_WIDE = 8u;
constexpr int KIND_NONE = DAG_KIND_NONE, KIND_BELOW = DAG_KIND_BELOW, KIND_ABOVE = DAG_KIND_ABOVE;
constexpr int KIND_GENERAL = DAG_KIND_GENERAL;
constexpr int KIND_PENDING = -1;             // short closures: any numbering, left to the levels
constexpr int TRI_TOP = DAG_TOP_MSB;         // products reaching bit 31 leave the path

struct TriComp {
    int64_t n, in_off, out_off, row_base;    // row_base: first batch-global row
};

constexpr int32_t TRI_PENDING = 3;           // closed by the levels in a second pass of the call

// Result of one matrix, written on the device and read back once per call.
struct TriOut {
    int32_t verdict, diameter;               // verdict: TRI_OPEN .. TRI_WIDE_ABOVE or TRI_PENDING
    unsigned long long executed;
};

__device__ __forceinline__ int tri_find(const int64_t *__restrict__ prefix, int count, int64_t cta) {
    int lo = 0, hi = count - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(prefix + mid) <= cta) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// A 16-byte vector of the storage type, unpacked.
template <typename T> struct TriVec {
    static constexpr int E = 16 / (int)sizeof(T);
    __device__ __forceinline__ static void split(const int4 &x, T (&v)[E]) {
        static_assert(sizeof(T) == 4 || sizeof(T) == 8, "int32 or int64 storage");
        if constexpr (sizeof(T) == 4) {
            v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
        } else {
            v[0] = (T)(((unsigned long long)(unsigned)x.y << 32) | (unsigned)x.x);
            v[1] = (T)(((unsigned long long)(unsigned)x.w << 32) | (unsigned)x.z);
        }
    }
};

// Off-diagonal entries of E consecutive columns j0 .. j0 + E - 1 held by each lane (m of them
// valid): clean-regime flags, and the nonzeros appended to the row's slots in column order.
// Column numbers fit 32 bits (n <= 8192 on this path); values outside [2, 2^31) are unclean.
template <typename T, int E>
__device__ __forceinline__ void tri_take(T (&v)[E], int j0, int m, int i, int lane, int64_t g,
                                         int32_t *__restrict__ slot_col, int32_t *__restrict__ slot_val,
                                         unsigned &flags, int &cnt) {
    int c4 = 0;
#pragma unroll
    for (int k = 0; k < E; ++k) {
        const int j = j0 + k;
        if (k >= m) {
            v[k] = 0;
        } else if (j == i) {
            if (!(v[k] == 0 || v[k] == 1 || v[k] == -1)) flags |= TF_UNCLEAN;
            v[k] = 0;                        // the diagonal is not an edge
        } else if (v[k] != 0) {
            if (v[k] == 1 || v[k] < 0 || (sizeof(T) == 8 && (long long)v[k] > (long long)INT32_MAX))
                flags |= TF_UNCLEAN;
            flags |= j < i ? TF_BELOW : TF_ABOVE;
            ++c4;
        }
    }
    if (!__any_sync(0xffffffffu, c4 != 0)) return;
    int x = c4;                              // inclusive prefix over the lanes
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    int pos = cnt + x - c4;
#pragma unroll
    for (int k = 0; k < E; ++k) {
        if (v[k] != 0) {
            if (pos < TRI_CAP) {
                slot_col[g * TRI_CAP + pos] = j0 + k;
                slot_val[g * TRI_CAP + pos] = (int32_t)v[k];
            }
            ++pos;
        }
    }
    cnt += __shfl_sync(0xffffffffu, x, 31);
}

// One warp per row: clean-regime test, side of the diagonal, the row's off-diagonal entries in
// column order into its TRI_CAP slots (the count may exceed TRI_CAP: then only flagged).  The
// row is read as 16-byte vectors from its first 16-byte boundary (scalar head and tail), four
// vectors per lane in flight; a vector of zeros (the common case) costs one vote.
template <typename T>
__global__ void __launch_bounds__(TRI_THREADS, 5)
tri_scan_kernel(const T *__restrict__ in, int64_t ld_in, const TriComp *__restrict__ comps,
                const int64_t *__restrict__ pre, int count, int32_t *__restrict__ slot_col,
                int32_t *__restrict__ slot_val, int32_t *__restrict__ row_cnt, int32_t *__restrict__ row_comp,
                unsigned *__restrict__ cflags, unsigned long long *__restrict__ state) {
    constexpr int E = TriVec<T>::E;
    const int ci = tri_find(pre, count, blockIdx.x);
    const TriComp c = comps[ci];
    const int i = (int)(((int64_t)blockIdx.x - pre[ci]) * TRI_ROWS) + (threadIdx.x >> 5);
    if (i >= c.n) return;                    // warp-uniform
    const int lane = threadIdx.x & 31;
    const int n = (int)c.n;
    const int64_t g = c.row_base + i;
    const T *row = in + c.in_off + (int64_t)i * (ld_in ? ld_in : c.n);
    const int lead = (int)(((16 - ((uintptr_t)row & 15)) & 15) / sizeof(T));   // to the first boundary
    const int head = lead < n ? lead : n;
    const int nv = (n - head) / E;           // 16-byte vectors after the head
    const int tail = n - head - E * nv;
    unsigned flags = 0;
    int cnt = 0;
    T v1[1];
    if (head) {                              // columns 0 .. head - 1, one per lane
        v1[0] = lane < head ? row[lane] : (T)0;
        tri_take<T, 1>(v1, lane, lane < head ? 1 : 0, i, lane, g, slot_col, slot_val, flags, cnt);
    }
    // vectors s0 + 32 u + lane (u = 0..3), taken in column order (u ascending)
    for (int s0 = 0; s0 < nv; s0 += 128) {
        int4 x[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int q = s0 + 32 * u + lane;
            x[u] = q < nv ? *reinterpret_cast<const int4 *>(row + head + E * q) : make_int4(0, 0, 0, 0);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int q = s0 + 32 * u + lane;
            const int j0 = head + E * q;
            // all-zero vectors (a zero diagonal included) leave nothing to take
            if (__any_sync(0xffffffffu, (x[u].x | x[u].y | x[u].z | x[u].w) != 0)) {
                T v[E];
                TriVec<T>::split(x[u], v);
                tri_take<T, E>(v, j0, q < nv ? E : 0, i, lane, g, slot_col, slot_val, flags, cnt);
            }
        }
    }
    if (tail) {
        const int j = head + E * nv + lane;
        v1[0] = lane < tail ? row[j] : (T)0;
        tri_take<T, 1>(v1, j, lane < tail ? 1 : 0, i, lane, g, slot_col, slot_val, flags, cnt);
    }
    if (cnt > TRI_CAP) flags |= TF_WIDE;
    flags = __reduce_or_sync(0xffffffffu, flags);
    if (lane == 0) {
        row_cnt[g] = cnt;
        row_comp[g] = ci;
        if (state) state[g] = 0;             // short closures: not closed yet
        if (flags) atomicOr(cflags + ci, flags);
    }
}

// Per matrix: candidate kind from the scan's flags, and the statistics' starting values.
__global__ void tri_kind_kernel(int count, const TriComp *__restrict__ comps, const unsigned *__restrict__ cflags,
                                int general, int32_t *__restrict__ ckind, int *__restrict__ cam, int *__restrict__ cfm,
                                unsigned long long *__restrict__ cprod, unsigned *__restrict__ cbad,
                                unsigned *__restrict__ any_gen) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
        const unsigned f = cflags[i];
        int k = KIND_NONE;
        if (comps[i].n > 0 && !(f & (TF_UNCLEAN | TF_WIDE)))
            k = ((f & TF_BELOW) && (f & TF_ABOVE)) ? (general ? KIND_GENERAL : KIND_NONE)
                                                  : (f & TF_ABOVE) ? KIND_ABOVE : KIND_BELOW;
        ckind[i] = k;
        cam[i] = -1;
        cfm[i] = -1;
        cprod[i] = 0;
        cbad[i] = 0;
        if (k == KIND_GENERAL) atomicOr(any_gen, 1u);
    }
}

// entries of each row in the CSR of the candidate matrices (rows of other matrices empty)
__global__ void tri_count_kernel(int64_t R, const int32_t *__restrict__ row_cnt, const int32_t *__restrict__ row_comp,
                                 const int32_t *__restrict__ ckind, int64_t *__restrict__ cnt64) {
    for (int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; g <= R; g += (int64_t)gridDim.x * blockDim.x)
        cnt64[g] = g < R && ckind[row_comp[g]] != KIND_NONE ? row_cnt[g] : 0;
}

__global__ void tri_csr_fill_kernel(int64_t R, const int32_t *__restrict__ row_comp, const int32_t *__restrict__ ckind,
                                    const TriComp *__restrict__ comps, const int64_t *__restrict__ indptr,
                                    const int32_t *__restrict__ slot_col, const int32_t *__restrict__ slot_val,
                                    int32_t *__restrict__ a_col, int32_t *__restrict__ a_val) {
    for (int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; g < R; g += (int64_t)gridDim.x * blockDim.x) {
        const int ci = row_comp[g];
        if (ckind[ci] == KIND_NONE) continue;
        const int32_t base = (int32_t)comps[ci].row_base;
        const int64_t o = indptr[g];
        const int m = (int)(indptr[g + 1] - o);
        for (int p = 0; p < m; ++p) {
            a_col[o + p] = base + slot_col[g * TRI_CAP + p];
            a_val[o + p] = slot_val[g * TRI_CAP + p];
        }
    }
}

// The closure by levels kept every row in the pool (no pool overflow); otherwise nothing of this
// call's DAG path is used.  A matrix with a row never placed (a cycle: only matrices with entries
// on both sides of the diagonal can hold one) is marked in cbad.
constexpr int TRI_DAG_BAD = 15;              // DagCounters::flags that reject the call's DAG path
constexpr int TRI_GAVE_UP = 8;               // a bounded wait of the short closure ran out
__device__ __forceinline__ bool tri_dag_ok(const DagCounters *dc) { return !(dc->flags & TRI_DAG_BAD); }

// A closure row entry outside its matrix (which a consistent closure never holds): the access is
// skipped and the call's DAG path rejected (flag 4), so the blocked kernels decide.
constexpr int TRI_BAD_ROW = 4;

// The row statistics of dag_rows.cuh, reduced per matrix (largest product MSB, largest
// first-value MSB, products): a group of DAG_STATS_G lanes per row, runs of `run` rows per
// group, one set of atomics per run and matrix.  Each group's bitmap takes 1 KB of shared
// memory, so TRI_STATS_CTAS CTAs of TRI_STATS_GROUPS groups fit on an SM.
constexpr int TRI_STATS_GROUPS = TRI_THREADS / DAG_STATS_G;
constexpr int TRI_STATS_CTAS = 5;
__global__ void __launch_bounds__(TRI_THREADS, TRI_STATS_CTAS)
tri_stats_kernel(int64_t R, const int32_t *__restrict__ row_comp, const int32_t *__restrict__ ckind,
                 const TriComp *__restrict__ comps, const int64_t *__restrict__ indptr,
                 const int32_t *__restrict__ a_col, const int32_t *__restrict__ a_val,
                 const int64_t *__restrict__ row_off, const int32_t *__restrict__ row_len,
                 const int32_t *__restrict__ p_col, const int32_t *__restrict__ p_val, const DagCounters *dc,
                 int *__restrict__ cam, int *__restrict__ cfm, unsigned long long *__restrict__ cprod, int run) {
    constexpr int G = DAG_STATS_G;
    __shared__ __align__(16) unsigned bm_all[TRI_STATS_GROUPS][TRI_BM_WORDS];
    if (!tri_dag_ok(dc)) return;             // block-uniform
    const int grp = threadIdx.x / G, lane = threadIdx.x & (G - 1);
    const unsigned gmask = dag_group_mask<G>();
    int cur = -1, am = -1, fm = -1;          // the matrix of the run's current rows, its statistics,
    int kind = KIND_NONE, base = 0, words = 0;   // its kind, first row and bitmap words
    unsigned long long prods = 0;
    auto flush = [&]() {                     // group-uniform
        const int am_r = __reduce_max_sync(gmask, am);
        const int fm_r = __reduce_max_sync(gmask, fm);
        if (lane == 0 && cur >= 0) {
            if (am_r >= 0) atomicMax(cam + cur, am_r);
            if (fm_r >= 0) atomicMax(cfm + cur, fm_r);
            if (prods) atomicAdd(cprod + cur, prods);
        }
    };
    auto crow = [&](int64_t r, int64_t &off, int &len) { off = row_off[r]; len = row_len[r]; };
    const int64_t stride = (int64_t)gridDim.x * TRI_STATS_GROUPS * run;
    for (int64_t r0 = ((int64_t)blockIdx.x * TRI_STATS_GROUPS + grp) * run; r0 < R; r0 += stride) {
        const int64_t r1 = min(R, r0 + run);
        for (int64_t g = r0; g < r1; ++g) {
            const int ci = row_comp[g];
            const int64_t a0 = indptr[g];
            const int alen = (int)(indptr[g + 1] - a0);
            if (ci != cur) {                     // group-uniform
                flush();
                cur = ci;
                am = fm = -1;
                prods = 0;
                kind = ckind[ci];
                base = (int32_t)comps[ci].row_base;
                words = (int)((comps[ci].n + 31) >> 5);
            }
            if (kind == KIND_NONE || kind == KIND_GENERAL) continue;   // group-uniform
            dag_row_stats<G>(bm_all[grp], words, kind, g, a0, alen, indptr, a_col, a_val, crow, p_col, p_val,
                             [&](int32_t col) { return col - base; }, lane, gmask, am, fm, prods);
        }
    }
    flush();
}


// ------------------------------------------------------------------------------------------
// Matrices in any numbering (entries on both sides of the diagonal)
// ------------------------------------------------------------------------------------------
// Before step k of the loop, W(i, j) holds the smallest value of the paths from i to j whose
// intermediate vertices are all below k.  In the clean regime msb(x (x) y) = msb(x) + msb(y) and
// the sum is a minimum, so the MSB of W(i, j) is the shortest such path, the MSB of an edge being
// its length.  Step k performs exactly the products (i, k, j) with i in In(k) and j in Out(k):
// the vertices that reach k, and those k reaches, through intermediates below k.  Hence
//   - the largest product MSB of step k is max over In(k) + max over Out(k) of those lengths;
//   - a cell without an entry of A gets its first value at the smallest k with i in In(k) and j in
//     Out(k), and that value's MSB is the two lengths' sum (the diameter's source);
//   - the number of products is the sum over k of |In(k)| |Out(k)|.
// Every k is searched on its own (no step waits for another), by the two searches from k along the
// edges and against them; In(k) and Out(k) are disjoint in a DAG, so they share a table.
//
// A warp per k.  The vertices reached live in a table of TRI_TAB words in shared memory, (local
// vertex << 8 | length), and in a list of table slots in the order of discovery, which is the
// search's queue.  A vertex shortened after it was taken from the queue sends the list through
// once more.  Searches that reach more vertices than the list holds go to a second launch (DENSE)
// whose table has a word per vertex of the largest matrix.  Latency bound (a search is a few
// dependent loads per length).  Replaying the loop in step order instead, one warp per matrix
// walking its chain of non-empty steps, took 665 us of the 1,226 us of a renumbered n = 3001
// pedigree's closure; with the searches the closure takes 541 us (n = 8191: 2,730 us to 656 us).
constexpr int TRI_TAB = 512;                 // table words of a warp's search
constexpr int TRI_LIST = 320;                // vertices it may reach before it goes to the dense one
constexpr int TRI_SEARCH_WARPS = 8;          // warps per CTA (table searches)
constexpr uint32_t TRI_EMPTY = 0xffffffffu;
constexpr int TRI_FAR = 126;                 // lengths are capped (a product of MSB 31 is already a risk)

// The candidates' graph for the searches, vertices batch-global: rows in CSR (columns batch-global)
// or, with row_cnt, in TRI_CAP slots each (columns local); children of a vertex in any order.
struct TriGraphView {
    const int64_t *indptr;
    const int32_t *row_cnt;
    const int32_t *a_col, *a_val;
    const int64_t *coff;
    const int32_t *kid_cnt;                  // null: coff[v + 1] ends vertex v's list
    const int32_t *children;
    __device__ __forceinline__ int64_t row(int64_t g, int &cnt) const {
        if (row_cnt) {
            cnt = row_cnt[g];
            return g * TRI_CAP;
        }
        const int64_t e = indptr[g];
        cnt = (int)(indptr[g + 1] - e);
        return e;
    }
    __device__ __forceinline__ int local(int64_t e, int64_t base) const {
        return row_cnt ? a_col[e] : a_col[e] - (int)base;
    }
    __device__ __forceinline__ int64_t kids(int64_t g, int &cnt) const {
        const int64_t e = coff[g];
        cnt = kid_cnt ? kid_cnt[g] : (int)(coff[g + 1] - e);
        return e;
    }
};

// position of column c in the sorted closure row [o, o + len), or -1
__device__ __forceinline__ int64_t tri_find_col(const int32_t *__restrict__ p_col, int64_t o, int len, int32_t c) {
    int lo = 0, hi = len - 1;
    while (lo <= hi) {
        const int mid = (lo + hi) >> 1;
        const int32_t v = p_col[o + mid];
        if (v == c) return o + mid;
        if (v < c) lo = mid + 1;
        else hi = mid - 1;
    }
    return -1;
}

// One warp per candidate row of a general matrix: a row never placed by the closure by levels (on
// or below a cycle) marks its matrix; the cells of A's entries start with key 0 (their first value
// is A's), the other cells empty.  Cell q of the row is cell[row_off + q].
__global__ void tri_gen_init_kernel(int64_t R, const int32_t *__restrict__ row_comp, const int32_t *__restrict__ ckind,
                                    const TriComp *__restrict__ comps, TriGraphView G,
                                    const int64_t *__restrict__ row_off,
                                    const int32_t *__restrict__ row_len, const int32_t *__restrict__ p_col,
                                    const DagCounters *dc, const unsigned *any_gen, unsigned *gflags,
                                    unsigned *__restrict__ cbad, uint32_t *__restrict__ cell) {
    if (!tri_dag_ok(dc) || !*any_gen) return;
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t g = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); g < R; g += warps) {
        const int ci = row_comp[g];
        if (ckind[ci] != KIND_GENERAL || cbad[ci]) continue;   // warp-uniform
        const int len = row_len[g];
        if (len < 0) {
            if (lane == 0) atomicOr(cbad + ci, 1u);
            continue;
        }
        const int64_t o = row_off[g];
        for (int q = lane; q < len; q += 32) cell[o + q] = TRI_EMPTY;
        __syncwarp();
        const int64_t base = comps[ci].row_base;
        int cnt;
        const int64_t e0 = G.row(g, cnt);
        for (int64_t e = e0 + lane; e < e0 + cnt; e += 32) {
            const int64_t q = tri_find_col(p_col, o, len, (int32_t)(base + G.local(e, base)));
            if (q < 0) atomicOr(gflags, 2u);
            else cell[q] = (uint32_t)msb_u32((uint32_t)G.a_val[e]);   // a clean value: 2 <= v < 2^31
        }
    }
}

// The table of a warp's search.  put() lowers vertex v's length to d and tells whether v is new
// (`at`: where) or was shortened; the list holds `at`s.
template <bool DENSE> struct TriTable {
    uint32_t *word;
    __device__ __forceinline__ int vertex(int at) const { return DENSE ? at : (int)(word[at] >> 8); }
    __device__ __forceinline__ int length(int at) const { return (int)(word[at] & 0xffu); }
    __device__ __forceinline__ int put(int v, int d, int &at) {   // 1: new, 2: shortened, 0: neither
        const uint32_t w = ((uint32_t)v << 8) | (uint32_t)d;
        if (DENSE) {
            at = v;
            const uint32_t old = atomicMin(&word[v], w);
            return old == TRI_EMPTY ? 1 : old > w ? 2 : 0;
        }
        int h = (int)(((uint32_t)v * 2654435761u) >> 16) & (TRI_TAB - 1);
        while (true) {                       // the list is shorter than the table: a slot is free
            uint32_t cur = *(volatile uint32_t *)&word[h];
            if (cur == TRI_EMPTY) {
                cur = atomicCAS(&word[h], TRI_EMPTY, w);
                if (cur == TRI_EMPTY) { at = h; return 1; }
            }
            if ((int)(cur >> 8) == v) {
                at = h;
                return atomicMin(&word[h], w) > w ? 2 : 0;
            }
            h = (h + 1) & (TRI_TAB - 1);
        }
    }
};

// One search from vertex k (local number) through intermediates below k, along the edges (FWD) or
// against them; the vertices reached are list[n0, n1).  Returns n1, or -1 when the list is full.
template <bool DENSE, bool FWD>
__device__ __forceinline__ int tri_search(const TriGraphView &G, TriTable<DENSE> &T, volatile uint16_t *list, int cap,
                                          int n0, int k, int64_t base, int lane) {
    int n1 = n0, h = n0 - 1;                 // position n0 - 1 stands for k itself
    bool again = false;
    while (true) {
        if (h >= n1) {                       // the end of the list: done, or once more from its start
            if (!again) return n1;
            again = false;
            h = n0;
        }
        // up to 32 vertices of the queue, their edges flattened over the warp
        const int left = h < n0 ? 1 : min(32, n1 - h);
        int x = -1, dx = 0, cnt = 0;
        int64_t e0 = 0;
        if (lane < left) {
            if (h < n0) {
                x = k;
            } else {
                const int at = list[h + lane];
                const int v = T.vertex(at);
                dx = T.length(at);
                x = v < k ? v : -1;          // a vertex above k is an end, never an intermediate
            }
            if (x >= 0) e0 = FWD ? G.row(base + x, cnt) : G.kids(base + x, cnt);
        }
        h += left;
        int incl = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        const int excl = incl - cnt;
        const int total = __shfl_sync(0xffffffffu, incl, 31);
        for (int b = 0; b < total; b += 32) {
            const int idx = b + lane;
            int lo = 0;
#pragma unroll
            for (int st = 16; st > 0; st >>= 1) {
                const int v = __shfl_sync(0xffffffffu, excl, lo + st);
                if (v <= idx) lo += st;
            }
            const int64_t eq = __shfl_sync(0xffffffffu, e0, lo) + (idx - __shfl_sync(0xffffffffu, excl, lo));
            const int xq = __shfl_sync(0xffffffffu, x, lo), dq = __shfl_sync(0xffffffffu, dx, lo);
            // a full list would leave no free slot in the table: stop before it can
            if (n1 + 32 > cap) return -1;    // warp-uniform
            int got = 0, at = 0;
            if (idx < total) {
                int y, len = 0;
                if (FWD) {
                    y = G.local(eq, base);
                    len = msb_u32((uint32_t)G.a_val[eq]);
                } else {
                    const int32_t c = G.children[eq];
                    y = c - (int)base;
                    int rc;                  // the edge's value, in the child's row
                    const int64_t r0 = G.row(c, rc);
                    for (int64_t e = r0; e < r0 + rc; ++e)
                        if (G.local(e, base) == xq) len = msb_u32((uint32_t)G.a_val[e]);
                }
                got = T.put(y, min(dq + len, TRI_FAR), at);
            }
            const unsigned fresh = __ballot_sync(0xffffffffu, got == 1);
            if (got == 1) list[n1 + __popc(fresh & ((1u << lane) - 1u))] = (uint16_t)at;
            n1 += __popc(fresh);
            again |= __any_sync(0xffffffffu, got == 2);
            __syncwarp();
        }
    }
}

// The searches of every vertex k of the general matrices, the statistics of step k, and the key
// (k + 1, product MSB) offered to each cell (i, j) of In(k) x Out(k): a cell keeps its smallest.
// The table searches walk all rows and leave the ones that outgrow the list to `ovf`, which the
// dense ones then walk (tables of `words` words and lists per warp in dynamic shared memory).
template <bool DENSE>
__global__ void __launch_bounds__(DENSE ? 32 : 32 * TRI_SEARCH_WARPS)
tri_gen_search_kernel(int64_t R, const int32_t *__restrict__ row_comp, const int32_t *__restrict__ ckind,
                      const unsigned *__restrict__ cbad, const TriComp *__restrict__ comps, TriGraphView G,
                      const int64_t *__restrict__ row_off, const int32_t *__restrict__ row_len,
                      const int32_t *__restrict__ p_col, const DagCounters *dc, const unsigned *any_gen,
                      unsigned *gflags, uint32_t *__restrict__ cell, int32_t *__restrict__ ovf, int words,
                      int *__restrict__ cam, unsigned long long *__restrict__ cprod) {
    if (!tri_dag_ok(dc) || !*any_gen || *gflags) return;
    extern __shared__ __align__(16) unsigned char tri_search_smem[];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int tab = DENSE ? words : TRI_TAB, cap = DENSE ? words + 32 : TRI_LIST;
    unsigned char *mine = tri_search_smem + (size_t)w * ((size_t)tab * 4 + (size_t)cap * 2);
    TriTable<DENSE> T{reinterpret_cast<uint32_t *>(mine)};
    volatile uint16_t *list = reinterpret_cast<uint16_t *>(mine + (size_t)tab * 4);
    for (int q = lane; q < tab; q += 32) T.word[q] = TRI_EMPTY;
    __syncwarp();
    const int64_t todo = DENSE ? (int64_t)ovf[0] : R;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t t = (int64_t)blockIdx.x * (blockDim.x >> 5) + w; t < todo; t += warps) {
        const int64_t g = DENSE ? (int64_t)ovf[1 + t] : t;
        const int ci = row_comp[g];
        if (ckind[ci] != KIND_GENERAL || cbad[ci]) continue;   // warp-uniform
        const int64_t base = comps[ci].row_base;
        const int k = (int)(g - base);
        // a vertex without parents or without children is on no product
        int parents, kids;
        G.row(g, parents);
        G.kids(g, kids);
        if (parents == 0 || kids == 0) continue;
        const int no = tri_search<DENSE, true>(G, T, list, cap, 0, k, base, lane);
        const int used = no < 0 ? no : tri_search<DENSE, false>(G, T, list, cap, no, k, base, lane);
        const int ni = used - no;
        if (used < 0) {                        // (a dense list holds every vertex)
            if (lane == 0) {
                if (DENSE) atomicOr(gflags, 2u);
                else ovf[1 + atomicAdd(ovf, 1)] = (int32_t)g;
            }
        } else {                             // both are non-empty
            int mo = 0, mi = 0;
            for (int q = lane; q < no; q += 32) mo = max(mo, T.length(list[q]));
            for (int q = lane; q < ni; q += 32) mi = max(mi, T.length(list[no + q]));
            mo = __reduce_max_sync(0xffffffffu, mo);
            mi = __reduce_max_sync(0xffffffffu, mi);
            const int64_t pairs = (int64_t)no * ni;
            if (lane == 0) {
                atomicMax(cam + ci, mo + mi);
                atomicAdd(cprod + ci, (unsigned long long)pairs);
            }
            for (int64_t q = lane; q < pairs; q += 32) {
                const int a = (int)(q / no), b = (int)(q - (int64_t)a * no);
                const int ai = list[no + a], bj = list[b];
                const int64_t i = base + T.vertex(ai);
                const int64_t at = tri_find_col(p_col, row_off[i], row_len[i], (int32_t)(base + T.vertex(bj)));
                if (at < 0) atomicOr(gflags, 2u);
                else atomicMin(cell + at, ((uint32_t)(k + 1) << 8) | (uint32_t)(T.length(ai) + T.length(bj)));
            }
        }
        __syncwarp();
        if (used < 0) {                      // the list lacks some of the slots in use
            for (int q = lane; q < tab; q += 32) T.word[q] = TRI_EMPTY;
        } else {
            for (int q = lane; q < used; q += 32) T.word[list[q]] = TRI_EMPTY;
        }
        __syncwarp();
    }
}

// The largest first value of each general matrix, over its cells.
__global__ void tri_gen_first_kernel(int64_t R, const int32_t *__restrict__ row_comp, const int32_t *__restrict__ ckind,
                                     const unsigned *__restrict__ cbad, const int64_t *__restrict__ row_off,
                                     const int32_t *__restrict__ row_len, const DagCounters *dc, const unsigned *any_gen,
                                     unsigned *gflags, const uint32_t *__restrict__ cell, int *__restrict__ cfm) {
    if (!tri_dag_ok(dc) || !*any_gen || *gflags) return;
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t g = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); g < R; g += warps) {
        const int ci = row_comp[g];
        if (ckind[ci] != KIND_GENERAL || cbad[ci]) continue;   // warp-uniform
        const int64_t o = row_off[g];
        const int len = row_len[g];
        int fm = -1;
        for (int q = lane; q < len; q += 32) {
            const uint32_t c = cell[o + q];
            if (c == TRI_EMPTY) atomicOr(gflags, 2u);          // a cell no step reaches: inconsistent
            else fm = max(fm, (int)(c & 0xffu));
        }
        fm = __reduce_max_sync(0xffffffffu, fm);
        if (lane == 0 && fm >= 0) atomicMax(cfm + ci, fm);
    }
}

// ------------------------------------------------------------------------------------------
// Short closures: matrices in a topological order, few rows in all
// ------------------------------------------------------------------------------------------
// With few rows the closure by levels is launches and their latency (three kernels a level, the
// children lists and row orders before them).  Here every row is one warp that waits for its
// parents itself: the warp takes the next row in the order of a ticket (a matrix with entries
// below the diagonal from its first row, one with entries above from its last), so a row's parents
// have smaller tickets, held by warps that run already, and every wait ends (it is bounded all the
// same).  A finished row is published as one 64-bit word, its pool position and length, stored
// after a fence and read with an acquire.
//
// The row itself: the columns of its entries and of its parents' rows are marked in a bitmap (a
// word per 32 columns), whose prefix counts give every column its place in the row; the values
// meet there by atomic minima.  The bitmap also tells a product that reaches a cell first, the
// statistics of dag_rows.cuh: below the diagonal while the parents are folded in (ascending, the
// loop's step order), above it in a second walk after the row is published.
//
// Latency bound: about 2 us per generation.  One n = 512 pedigree in 12 generations takes 81 us,
// 389 us by levels; n = 8192, int64: 313 us, 835 us by levels.
constexpr int TRI_PULL_WARPS = 8;            // warps (rows) per CTA
constexpr int TRI_PULL_CTAS = 4;             // CTAs per SM
constexpr int64_t TRI_PULL_ROWS = 16384;     // rows of a call on this path
constexpr int TRI_PULL_VALS = 512;           // columns of a row kept in shared memory
constexpr int TRI_PULL_TRIES = 1 << 22;      // polls of a parent before the call's DAG path is given up
constexpr int TRI_STATE_LEN_BITS = 24;

struct TriPullWarp {
    unsigned bm[TRI_BM_WORDS];
    unsigned short pre[TRI_BM_WORDS];        // columns before the word
    int col[TRI_PULL_VALS], val[TRI_PULL_VALS];
};

__device__ __forceinline__ unsigned long long tri_acquire(const unsigned long long *p) {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void tri_release(unsigned long long *p, unsigned long long v) {
    asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

__global__ void __launch_bounds__(32 * TRI_PULL_WARPS, TRI_PULL_CTAS)
tri_pull_kernel(int64_t R, const int32_t *__restrict__ row_comp, const TriComp *__restrict__ comps,
                const unsigned *__restrict__ cflags, const int32_t *__restrict__ slot_col,
                const int32_t *__restrict__ slot_val, const int32_t *__restrict__ row_cnt,
                unsigned long long *state, int64_t *__restrict__ row_off, int32_t *__restrict__ row_len,
                int32_t *p_col, int32_t *p_val, int64_t capacity, DagCounters *dc, int *ticket,
                int32_t *__restrict__ ckind, int *__restrict__ cam, int *__restrict__ cfm,
                unsigned long long *__restrict__ cprod, const int32_t *__restrict__ order,
                const unsigned *__restrict__ cbad) {
    __shared__ TriPullWarp warps[TRI_PULL_WARPS];
    TriPullWarp &S = warps[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    while (true) {
        int t = 0;
        if (lane == 0) t = atomicAdd(ticket, 1);
        t = __shfl_sync(0xffffffffu, t, 0);
        if (t >= R) return;
        const int ci = row_comp[t];
        const unsigned f = cflags[ci];
        const TriComp c = comps[ci];
        const int n = (int)c.n, words = (n + 31) >> 5;
        int kind;                            // warp-uniform
        int64_t g = t;
        if (order) {                         // the matrices in any numbering (tri_order_kernel)
            kind = cbad[ci] ? KIND_NONE : ckind[ci];
            if (kind <= KIND_NONE) continue;
            g = order[t];
        } else {
            kind = (f & (TF_UNCLEAN | TF_WIDE)) ? KIND_NONE
                   : ((f & TF_BELOW) && (f & TF_ABOVE)) ? KIND_PENDING
                   : (f & TF_ABOVE) ? KIND_ABOVE : KIND_BELOW;
            if (t == c.row_base && lane == 0) ckind[ci] = kind;
            if (kind <= KIND_NONE) continue;
            // a matrix with entries above the diagonal goes from its last row to its first
            if (kind == KIND_ABOVE) g = 2 * c.row_base + n - 1 - t;
        }
        const int cnt = row_cnt[g];          // at most TRI_CAP
        int w = -1, v = 0, len = 0;
        int64_t off = 0;
        if (lane < cnt) {
            w = slot_col[g * TRI_CAP + lane];
            v = slot_val[g * TRI_CAP + lane];
        }
        for (int q = lane; q < words; q += 32) S.bm[q] = 0;
        __syncwarp();
        if (lane < cnt) atomicOr(&S.bm[w >> 5], 1u << (w & 31));
        // the parents' rows, as soon as they are published
        bool late = false;
        if (lane < cnt) {
            unsigned long long st = 0;
            int tries = 0;
            while ((st = tri_acquire(state + c.row_base + w)) == 0 && ++tries < TRI_PULL_TRIES) {}
            late = st == 0;
            if (st) {
                off = (int64_t)(st >> TRI_STATE_LEN_BITS) - 1;
                len = (int)(st & ((1u << TRI_STATE_LEN_BITS) - 1u));
            }
        }
        __syncwarp();
        int incl = len;                      // the parents' entries, flattened over the warp
#pragma unroll
        for (int o = 1; o < TRI_CAP; o <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += x;
        }
        const int excl = incl - len;
        const int total = __shfl_sync(0xffffffffu, incl, TRI_CAP - 1);
        // pool room for the row's bound, asked for while the parents' rows are read
        unsigned long long at = 0;
        if (lane == 0) at = atomicAdd(&dc->reserved, (unsigned long long)(total + cnt));
        int am = -1, fm = lane < cnt ? dag_row_msb(v) : -1;
        // candidate idx of the flattened rows: its column and product (0 beyond the end)
        auto candidate = [&](int idx, int &col, int &pm) -> int {
            int lo = 0;
#pragma unroll
            for (int sft = TRI_CAP / 2; sft > 0; sft >>= 1) {
                const int x = __shfl_sync(0xffffffffu, excl, lo + sft);
                if (lo + sft < cnt && x <= idx) lo += sft;
            }
            const int vq = __shfl_sync(0xffffffffu, v, lo), xq = __shfl_sync(0xffffffffu, excl, lo);
            const int64_t oq = __shfl_sync(0xffffffffu, off, lo);
            col = -1 - lane;                 // no column, each lane its own
            pm = -1;
            if (idx >= total) return 0;
            col = __ldcg(p_col + oq + (idx - xq)) - (int)c.row_base;
            const int y = __ldcg(p_val + oq + (idx - xq));
            pm = dag_row_msb(vq) + dag_row_msb(y);
            return cy_product(vq, y);
        };
        // the first 128 candidates stay in registers
        int kc[4], kv[4];
        for (int b = 0; b < total; b += 128) {
            int km[4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (b + 32 * u < total) {
                    int cc, pp;
                    const int vv = candidate(b + 32 * u + lane, cc, pp);
                    km[u] = pp;
                    if (b == 0) { kc[u] = cc; kv[u] = vv; }
                    am = max(am, pp);
                    // the lowest lane of a column not yet marked performs the cell's first product
                    const unsigned same = __match_any_sync(0xffffffffu, cc);
                    if (cc >= 0 && !(same & below) && !((S.bm[cc >> 5] >> (cc & 31)) & 1u)) {
                        if (kind == KIND_BELOW) fm = max(fm, km[u]);
                        atomicOr(&S.bm[cc >> 5], 1u << (cc & 31));
                    }
                    __syncwarp();
                }
        }
        // places of the columns: words [lane * wl, lane * wl + wl) per lane
        const int wl = (words + 31) >> 5;
        int mine = 0;
        for (int q = lane * wl; q < min(words, (lane + 1) * wl); ++q) mine += __popc(S.bm[q]);
        int run = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, run, o);
            if (lane >= o) run += x;
        }
        const int nd = __shfl_sync(0xffffffffu, run, 31);
        run -= mine;
        for (int q = lane * wl; q < min(words, (lane + 1) * wl); ++q) {
            S.pre[q] = (unsigned short)run;
            run += __popc(S.bm[q]);
        }
        at = __shfl_sync(0xffffffffu, at, 0);
        const bool room = (int64_t)at + total + cnt <= capacity;
        const bool wide = nd > TRI_PULL_VALS;    // the values meet in the pool instead
        int32_t *oc = wide ? p_col + at : S.col, *ov = wide ? p_val + at : S.val;
        if (room) {
            for (int q = lane; q < nd; q += 32) ov[q] = INT_MAX;
            if (wide) __threadfence();
            __syncwarp();
            auto put = [&](int col, int val) {
                const int r = S.pre[col >> 5] + __popc(S.bm[col >> 5] & ((1u << (col & 31)) - 1u));
                oc[r] = (int)c.row_base + col;
                if (val != 0) atomicMin(ov + r, val);
            };
            if (lane < cnt) put(w, v);
            for (int b = 0; b < total; b += 128) {
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (b + 32 * u < total) {
                        int cc = kc[u], pp, vv = kv[u];
                        if (b > 0) vv = candidate(b + 32 * u + lane, cc, pp);
                        if (cc >= 0) put(cc, vv);
                    }
            }
            __syncwarp();
            if (!wide)
                for (int q = lane; q < nd; q += 32) {
                    p_col[at + q] = S.col[q];
                    p_val[at + q] = S.val[q];
                }
        }
        late = __any_sync(0xffffffffu, late);
        if (lane == 0) {
            if (!room) atomicOr(&dc->flags, 1);
            if (late) atomicOr(&dc->flags, TRI_GAVE_UP);
            row_off[g] = (int64_t)at;
            row_len[g] = room ? nd : 0;
            __threadfence();
            tri_release(state + g, ((at + 1) << TRI_STATE_LEN_BITS) | (unsigned long long)(room ? nd : 0));
        }
        __syncwarp();
        unsigned long long prods = (unsigned long long)total;
        if (kind == KIND_ABOVE) {
            // steps k over the row ascending, each adding C(i, k) (x) A(k, .), two steps at a time
            prods = 0;
            for (int q = lane; q < words; q += 32) S.bm[q] = 0;
            __syncwarp();
            if (lane < cnt) atomicOr(&S.bm[w >> 5], 1u << (w & 31));
            __syncwarp();
            const int e = lane & (TRI_CAP - 1), half = lane / TRI_CAP;
            for (int q = 0; room && q < nd; q += 32 / TRI_CAP) {
                int j = -1 - lane, pm = -1;
                if (q + half < nd) {
                    const int64_t k = wide ? (int64_t)__ldcg(p_col + at + q + half) : (int64_t)S.col[q + half];
                    const int kvv = wide ? __ldcg(p_val + at + q + half) : S.val[q + half];
                    if (e < row_cnt[k]) {
                        j = slot_col[k * TRI_CAP + e];
                        pm = dag_row_msb(kvv) + dag_row_msb(slot_val[k * TRI_CAP + e]);
                    }
                }
                am = max(am, pm);
                prods += __popc(__ballot_sync(0xffffffffu, j >= 0));
                const unsigned same = __match_any_sync(0xffffffffu, j);
                if (j >= 0 && !(same & below) && !((S.bm[j >> 5] >> (j & 31)) & 1u)) {
                    fm = max(fm, pm);
                    atomicOr(&S.bm[j >> 5], 1u << (j & 31));
                }
                __syncwarp();
            }
        }
        if (kind == KIND_GENERAL) continue;  // the searches take its statistics
        am = __reduce_max_sync(0xffffffffu, am);
        fm = __reduce_max_sync(0xffffffffu, fm);
        if (lane == 0) {
            if (am >= 0) atomicMax(cam + ci, am);
            if (fm >= 0) atomicMax(cfm + ci, fm);
            if (prods) atomicAdd(cprod + ci, prods);
        }
    }
}

// Second pass of a short closure, one CTA per matrix: a matrix in any numbering gets its children
// lists and its rows in a topological order (Kahn's algorithm by levels, the counters and the
// frontier in shared memory, so a level costs two barriers and one read of the frontier's children);
// one with a cycle is marked in cbad, every other matrix is taken off the path (its result is read
// already).
constexpr int TRI_ORDER_THREADS = 1024;
struct TriOrderSmem {
    int end[TRI_MAX_N];                      // children of v: [end[v - 1], end[v]) of the matrix's list
    int rem[TRI_MAX_N];                      // parents not placed yet
    unsigned short list[TRI_MAX_N];          // placed vertices
};

__global__ void __launch_bounds__(TRI_ORDER_THREADS)
tri_order_kernel(const TriComp *__restrict__ comps, int32_t *ckind, const int32_t *__restrict__ slot_col,
                 const int32_t *__restrict__ row_cnt, int32_t *__restrict__ order, int64_t *__restrict__ coff,
                 int32_t *__restrict__ kid_cnt, int32_t *__restrict__ children, unsigned *__restrict__ cbad,
                 int *ticket, unsigned *any_gen) {
    extern __shared__ __align__(16) unsigned char tri_order_smem[];
    TriOrderSmem &S = *reinterpret_cast<TriOrderSmem *>(tri_order_smem);
    __shared__ int s_sum[TRI_ORDER_THREADS / 32], s_tail;
    const int ci = blockIdx.x, tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    if (ci == 0 && tid == 0) *ticket = 0;
    const int kind = ckind[ci];
    __syncthreads();
    if (kind != KIND_PENDING) {
        if (tid == 0) ckind[ci] = KIND_NONE;
        return;
    }
    if (tid == 0) {
        ckind[ci] = KIND_GENERAL;
        atomicOr(any_gen, 1u);
        s_tail = 0;
    }
    const TriComp c = comps[ci];
    const int n = (int)c.n;
    const int64_t g0 = c.row_base;
    int32_t *kids = children + g0 * TRI_CAP;
    for (int v = tid; v < n; v += TRI_ORDER_THREADS) S.end[v] = 0;
    __syncthreads();
    for (int v = tid; v < n; v += TRI_ORDER_THREADS) {
        const int m = row_cnt[g0 + v];
        S.rem[v] = m;
        for (int e = 0; e < m; ++e) atomicAdd(&S.end[slot_col[(g0 + v) * TRI_CAP + e]], 1);
    }
    __syncthreads();
    // exclusive scan of the counts, a run of consecutive vertices per thread
    const int run = (n + TRI_ORDER_THREADS - 1) / TRI_ORDER_THREADS;
    int sum = 0;
    for (int v = tid * run; v < min(n, (tid + 1) * run); ++v) sum += S.end[v];
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += x;
    }
    if (lane == 31) s_sum[w] = incl;
    __syncthreads();
    int at = incl - sum;
    for (int q = 0; q < w; ++q) at += s_sum[q];
    for (int v = tid * run; v < min(n, (tid + 1) * run); ++v) {
        const int k = S.end[v];
        coff[g0 + v] = g0 * TRI_CAP + at;
        kid_cnt[g0 + v] = k;
        S.end[v] = at;                       // a cursor that ends at the list's end
        at += k;
    }
    __syncthreads();
    for (int v = tid; v < n; v += TRI_ORDER_THREADS) {
        const int m = S.rem[v];
        for (int e = 0; e < m; ++e)
            kids[atomicAdd(&S.end[slot_col[(g0 + v) * TRI_CAP + e]], 1)] = (int32_t)(g0 + v);
        if (m == 0) S.list[atomicAdd(&s_tail, 1)] = (unsigned short)v;
    }
    __syncthreads();                         // (the lists' writes are visible to the CTA)
    // levels: 8 lanes per frontier vertex
    int h = 0, tail = s_tail;
    __syncthreads();                         // everyone has the first level's end before it moves
    while (h < tail) {                       // block-uniform
        for (int q = h + (tid >> 3); q < tail; q += TRI_ORDER_THREADS / 8) {
            const int v = S.list[q];
            for (int e = (v ? S.end[v - 1] : 0) + (tid & 7); e < S.end[v]; e += 8) {
                const int k = kids[e] - (int)g0;
                if (atomicSub(&S.rem[k], 1) == 1) S.list[atomicAdd(&s_tail, 1)] = (unsigned short)k;
            }
        }
        __syncthreads();
        h = tail;
        tail = s_tail;
        __syncthreads();
    }
    for (int q = tid; q < tail; q += TRI_ORDER_THREADS) order[g0 + q] = (int32_t)(g0 + S.list[q]);
    if (tid == 0 && tail < n) cbad[ci] = 1u; // on a cycle, or below one
}

// shared memory of a dense search over matrices of up to n rows, and of a CTA of table searches
constexpr size_t tri_dense_smem(int n) { return (size_t)n * 4 + (size_t)(n + 32) * 2; }
constexpr size_t TRI_TAB_SMEM = (size_t)TRI_SEARCH_WARPS * (TRI_TAB * 4 + TRI_LIST * 2);

PerDeviceOnce g_tri_configured;
int tri_configure() {
    return g_tri_configured.run([] {
        RBG_CUDA_TRY(cudaFuncSetAttribute(tri_gen_search_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)tri_dense_smem((int)TRI_MAX_N)));
        RBG_CUDA_TRY(cudaFuncSetAttribute(tri_order_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)sizeof(TriOrderSmem)));
        return (int)RBG_OK;
    });
}

// Recorded graphs: the IF node around the searches opens only when the closure by levels went
// through and some matrix needs them; the decision is also kept for the launch count.
__global__ void tri_gen_gate_kernel(const DagCounters *dc, const unsigned *any_gen, unsigned *ran,
                                    cudaGraphConditionalHandle h) {
    if (threadIdx.x != 0) return;
    const unsigned go = (tri_dag_ok(dc) && *any_gen) ? 1u : 0u;
    *ran = go;
    cudaGraphSetConditional(h, go);
}

// Inside the capture on `s`: `gate(h)` launches on s the kernel that sets the condition, then an
// IF node whose body `body(stream)` records from a second stream captured into it.
template <typename Gate, typename Body>
int tri_captured_if(cudaStream_t s, Gate gate, Body body) {
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    cudaGraph_t g = nullptr;
    const cudaGraphNode_t *deps = nullptr;
    size_t ndeps = 0;
    RBG_CUDA_TRY(cudaStreamGetCaptureInfo(s, &st, nullptr, &g, &deps, nullptr, &ndeps));
    if (st != cudaStreamCaptureStatusActive || !g) return RBG_ERR_INVALID;
    cudaGraphConditionalHandle h;
    RBG_CUDA_TRY(cudaGraphConditionalHandleCreate(&h, g, 0, cudaGraphCondAssignDefault));
    gate(h);
    RBG_CUDA_TRY(cudaGetLastError());
    RBG_CUDA_TRY(cudaStreamGetCaptureInfo(s, &st, nullptr, &g, &deps, nullptr, &ndeps));
    cudaGraphNodeParams p = {};
    p.type = cudaGraphNodeTypeConditional;
    p.conditional.handle = h;
    p.conditional.type = cudaGraphCondTypeIf;
    p.conditional.size = 1;
    cudaGraphNode_t node;
    RBG_CUDA_TRY(cudaGraphAddNode(&node, g, deps, nullptr, ndeps, &p));
    static thread_local cudaStream_t side = nullptr;
    if (!side) RBG_CUDA_TRY(cudaStreamCreateWithFlags(&side, cudaStreamNonBlocking));
    RBG_CUDA_TRY(cudaStreamBeginCaptureToGraph(side, p.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                               cudaStreamCaptureModeThreadLocal));
    const int rc = body(side);
    cudaGraph_t got = nullptr;
    const cudaError_t ee = cudaStreamEndCapture(side, &got);
    if (rc) return rc;
    if (ee != cudaSuccess) return RBG_ERR_CUDA;
    RBG_CUDA_TRY(cudaStreamUpdateCaptureDependencies(s, &node, nullptr, 1, cudaStreamSetCaptureDependencies));
    return RBG_OK;
}

constexpr int TRI_GEN_LAUNCHES = 4;          // launches of the any-numbering block

__device__ __forceinline__ bool tri_accepted(int ci, const int32_t *ckind, const int *cam, const unsigned *cbad,
                                             const DagCounters *dc, const unsigned *gflags) {
    const int k = ckind[ci];
    return k > KIND_NONE && cam[ci] < TRI_TOP && !cbad[ci] && tri_dag_ok(dc) && !(k == KIND_GENERAL && *gflags);
}

// The statistics are complete and some product of the loop reaches bit 31 (the first such
// product is computed from exact operands, so the test is exact).
__device__ __forceinline__ bool tri_top_bit(int ci, const int32_t *ckind, const int *cam, const unsigned *cbad,
                                            const DagCounters *dc, const unsigned *gflags) {
    const int k = ckind[ci];
    return k > KIND_NONE && cam[ci] >= TRI_TOP && !cbad[ci] && tri_dag_ok(dc) && !(k == KIND_GENERAL && *gflags);
}

// One warp per row of an accepted matrix.  Out of place, the whole dense row is written in
// segments of SEG columns (2 KB) built in shared memory (zeros, the closure row's entries, the
// diagonal) and stored as full 16-byte vectors on the row's 16-byte grid, so no DRAM line is
// written partially; in place, only the closure's entries (the other cells already hold the
// result).  The row statistics are recorded when asked for (32-bit storage).  The first CTA of a
// matrix writes its result record.
template <typename T>
__global__ void __launch_bounds__(TRI_THREADS)
tri_write_kernel(const T *__restrict__ in, int64_t ld_in, T *__restrict__ out, int64_t ld_out,
                 const TriComp *__restrict__ comps, const int64_t *__restrict__ pre, int count,
                 const int32_t *__restrict__ ckind, const int *__restrict__ cam, const unsigned *__restrict__ cbad,
                 const DagCounters *dc, const unsigned *gflags,
                 const int64_t *__restrict__ row_off, const int32_t *__restrict__ row_len,
                 const int32_t *__restrict__ p_col, const int32_t *__restrict__ p_val, RowStats rs,
                 const int *__restrict__ cfm, const unsigned long long *__restrict__ cprod,
                 const unsigned *__restrict__ cflags, TriOut *__restrict__ res) {
    constexpr int SEG = 2048 / (int)sizeof(T);
    constexpr int E = TriVec<T>::E;
    __shared__ __align__(16) T seg_all[TRI_ROWS][SEG];
    const int ci = tri_find(pre, count, blockIdx.x);
    const bool accepted = tri_accepted(ci, ckind, cam, cbad, dc, gflags);   // block-uniform
    if ((int64_t)blockIdx.x == pre[ci] && threadIdx.x == 0) {
        TriOut o;
        o.verdict = accepted ? TRI_CLOSED : tri_top_bit(ci, ckind, cam, cbad, dc, gflags) ? TRI_TOP_BIT
                    : ckind[ci] == KIND_PENDING ? TRI_PENDING
                    : (cflags[ci] & ~(TF_BELOW | TF_ABOVE)) != TF_WIDE ? TRI_OPEN
                    : !(cflags[ci] & TF_ABOVE) ? TRI_WIDE_BELOW
                    : !(cflags[ci] & TF_BELOW) ? TRI_WIDE_ABOVE : TRI_OPEN;
        o.diameter = cfm[ci] > 0 ? cfm[ci] : 0;
        o.executed = cprod[ci];
        res[ci] = o;
    }
    if (!accepted) return;
    const TriComp c = comps[ci];
    const int i = (int)(((int64_t)blockIdx.x - pre[ci]) * TRI_ROWS) + (threadIdx.x >> 5);
    if (i >= c.n) return;                    // warp-uniform
    const int lane = threadIdx.x & 31;
    const int n = (int)c.n;
    const int64_t g = c.row_base + i;
    const T *rin = in + c.in_off + (int64_t)i * (ld_in ? ld_in : c.n);
    T *rout = out + c.out_off + (int64_t)i * (ld_out ? ld_out : c.n);
    const T diag = rin[i];
    const int64_t c0 = row_off[g];
    const int clen = row_len[g];
    const int32_t base = (int32_t)c.row_base;
    // chunk masks of the row (n <= 8192: at most four 64-bit words), held in registers
    unsigned long long w0 = 0, w1 = 0, w2 = 0, w3 = 0;
    auto mark = [&](int chunk) {
        const unsigned long long bit = 1ull << (chunk & 63);
        const int t = chunk >> 6;
        w0 |= t == 0 ? bit : 0ull;
        w1 |= t == 1 ? bit : 0ull;
        w2 |= t == 2 ? bit : 0ull;
        w3 |= t == 3 ? bit : 0ull;
    };
    int mx = 0;
    if (rin == rout) {
        for (int q = lane; q < clen; q += 32) {
            const int j = p_col[c0 + q] - base;
            const int32_t v = p_val[c0 + q];
            if ((unsigned)j >= (unsigned)n) {
                atomicOr(const_cast<int *>(&dc->flags), TRI_BAD_ROW);
                continue;
            }
            rout[j] = (T)v;
            mx = max(mx, v);
            mark(j >> 5);
        }
    } else {
        T *seg = seg_all[threadIdx.x >> 5];
        // column j sits at j' = j + shift on the 16-byte grid; segment s0 holds j' in [s0, s0 + SEG)
        const int shift = (int)(((uintptr_t)rout & 15) / sizeof(T));
        int e = 0;                           // first closure entry not yet placed (warp-uniform)
        for (int s0 = 0; s0 < n + shift; s0 += SEG) {
            for (int t = lane; t < SEG / E; t += 32) reinterpret_cast<int4 *>(seg)[t] = make_int4(0, 0, 0, 0);
            __syncwarp();
            const int lim = s0 + SEG - shift;            // entries with j < lim belong to this segment
            for (;;) {                                   // batches of 32 entries, ascending
                const int q = e + lane;
                int j = INT_MAX;
                int32_t v = 0;
                if (q < clen) {
                    j = p_col[c0 + q] - base;
                    v = p_val[c0 + q];
                }
                const bool here = j < lim;
                if (here) {
                    if (j < 0 || j >= n || j + shift < s0) {   // outside the matrix, or out of order
                        atomicOr(const_cast<int *>(&dc->flags), TRI_BAD_ROW);
                    } else {
                        seg[j + shift - s0] = (T)v;
                        mx = max(mx, v);
                        mark(j >> 5);
                    }
                }
                const unsigned bal = __ballot_sync(0xffffffffu, here);
                e += __popc(bal);
                if (bal != 0xffffffffu) break;
            }
            if (lane == 0 && i + shift >= s0 && i + shift < s0 + SEG) seg[i + shift - s0] = diag;
            __syncwarp();
            for (int t = lane; t < SEG / E; t += 32) {
                const int j0 = s0 + E * t - shift;
                if (j0 >= n) break;
                const int4 z = reinterpret_cast<const int4 *>(seg)[t];
                if (j0 >= 0 && j0 + E <= n) {
                    *reinterpret_cast<int4 *>(rout + j0) = z;
                } else {                                 // the row's ragged ends
                    T zz[E];
                    TriVec<T>::split(z, zz);
#pragma unroll
                    for (int k = 0; k < E; ++k)
                        if (j0 + k >= 0 && j0 + k < n) rout[j0 + k] = zz[k];
                }
            }
            __syncwarp();                                // before the next segment is zeroed
        }
    }
    if constexpr (sizeof(T) == 4) {
        if (rs.row_count) {
            if (lane == 0 && diag != 0) {
                mark(i >> 5);
                mx = max(mx, (int)diag);
            }
            auto orw = [](unsigned long long x) {
                const unsigned lo = __reduce_or_sync(0xffffffffu, (unsigned)x);
                const unsigned hi = __reduce_or_sync(0xffffffffu, (unsigned)(x >> 32));
                return ((unsigned long long)hi << 32) | lo;
            };
            const unsigned long long wd[4] = {orw(w0), orw(w1), orw(w2), orw(w3)};
            mx = __reduce_max_sync(0xffffffffu, mx);
            if (lane == 0) {
                const int64_t at = rs.row_base[ci] + i;
                rs.row_count[rs.row_id ? (int64_t)rs.row_id[at] : at] = clen + (diag != 0 ? 1 : 0);
                if (rs.chunk_mask) {
                    const int64_t words = (n + 2047) / 2048;
                    unsigned long long *mrow = rs.chunk_mask + (c.in_off + 2047) / 2048 + rs.row_base[ci] + ci +
                                               (int64_t)i * words;
#pragma unroll
                    for (int t = 0; t < 4; ++t)
                        if (t < words) mrow[t] = wd[t];
                }
                if (rs.comp_max && mx > 0) atomicMax(rs.comp_max + ci, mx);
            }
        }
    }
}

struct Carve {
    unsigned char *p;
    size_t off = 0;
    template <typename X> X *take(size_t n) {
        off = align_up(off, 256);
        X *r = p ? reinterpret_cast<X *>(p + off) : nullptr;
        off += n * sizeof(X);
        return r;
    }
};

// The scratch of one call, carved from the caller's workspace: the matrix table, per-matrix
// flags, statistics and results with the call's counters (`head`, uploaded whole at the start of a
// call in its starting state), the scan's row slots, then either the candidates' CSR, the closure's
// workspace and row index (levels) or the rows' states (short closures), and the row pool in
// whatever remains.
struct TriLayout {
    TriComp *dc;
    int64_t *dpre, *indptr, *row_off;
    unsigned *cflags, *cbad, *gflags;        // gflags[0]: the searches' scratch is inconsistent; [1]: any general;
                                             // [2]: the any-numbering block ran (its IF node's decision)
    int32_t *ckind, *row_cnt, *row_comp, *slot_col, *slot_val, *a_col, *a_val, *row_len, *p_col, *p_val;
    int32_t *ovf;                            // any numbering: count and rows of the searches the table is too small for
    uint32_t *cell;                          // any numbering: per pool entry, the key of the cell's first value
    int *cam, *cfm;
    unsigned long long *cprod;
    TriOut *res;
    DagCounters *counters;                   // short closures: the call's counters, beside the results
    int *ticket;
    unsigned long long *state;               // short closures: per row 0, or (pool position + 1) << 24 | length
    int32_t *order, *kid_cnt, *children;     // short closures in any numbering: rows in a topological order and
    int64_t *coff;                           // the children lists (tri_order_kernel)
    void *tmp, *dag_ws;
    size_t scan_tmp;
    int64_t pool;
    size_t head;                             // bytes uploaded at the start of a call
    size_t fixed;                            // bytes before the pool
};

// Scratch of a scan over NR + 1 words.
size_t tri_scan_tmp(size_t NR) {
    static thread_local LastSize last;
    return last.get((int64_t)NR, [NR] {
        size_t b = 0;
        cub::DeviceScan::ExclusiveSum(nullptr, b, (int64_t *)nullptr, (int64_t *)nullptr, (int)(NR + 1));
        return b;
    });
}

void tri_layout(unsigned char *base, size_t ws_bytes, size_t C, size_t NR, bool is_short, TriLayout &L) {
    Carve cv{base};
    L.dc = cv.take<TriComp>(C);
    L.dpre = cv.take<int64_t>(C + 1);
    L.cflags = cv.take<unsigned>(C);
    L.ckind = cv.take<int32_t>(C);
    L.cam = cv.take<int>(C);
    L.cfm = cv.take<int>(C);
    L.cprod = cv.take<unsigned long long>(C);
    L.cbad = cv.take<unsigned>(C);
    L.gflags = cv.take<unsigned>(3);
    L.ticket = cv.take<int>(1);
    L.counters = cv.take<DagCounters>(1);
    L.res = cv.take<TriOut>(C);
    L.head = cv.off;
    L.row_cnt = cv.take<int32_t>(NR);
    L.row_comp = cv.take<int32_t>(NR);
    L.slot_col = cv.take<int32_t>(NR * TRI_CAP);
    L.slot_val = cv.take<int32_t>(NR * TRI_CAP);
    L.row_off = cv.take<int64_t>(NR);
    L.row_len = cv.take<int32_t>(NR);
    L.ovf = cv.take<int32_t>(NR + 1);
    if (is_short) {
        L.state = cv.take<unsigned long long>(NR);
        L.order = cv.take<int32_t>(NR);
        L.coff = cv.take<int64_t>(NR);
        L.kid_cnt = cv.take<int32_t>(NR);
        L.children = cv.take<int32_t>(NR * TRI_CAP);
    } else {
        L.scan_tmp = tri_scan_tmp(NR);
        L.indptr = cv.take<int64_t>(NR + 1);
        L.tmp = cv.take<unsigned char>(L.scan_tmp);
        L.a_col = cv.take<int32_t>(NR * TRI_CAP);
        L.a_val = cv.take<int32_t>(NR * TRI_CAP);
        L.dag_ws = cv.take<unsigned char>(dag_workspace_for((int64_t)NR, (int64_t)(NR * TRI_CAP)));
    }
    L.fixed = align_up(cv.off, 256);
    // the rest: the row pool, 12 bytes an entry (column, value, first-value key)
    const size_t rest = ws_bytes > L.fixed + 1024 ? ws_bytes - L.fixed - 1024 : 0;
    L.pool = std::min<int64_t>((int64_t)(rest / 12 / 64 * 64), (int64_t)INT32_MAX / 64 * 64);
    Carve tail{base};
    tail.off = L.fixed;
    L.p_col = tail.take<int32_t>((size_t)L.pool);
    L.p_val = tail.take<int32_t>((size_t)L.pool);
    L.cell = tail.take<uint32_t>((size_t)L.pool);
}

struct TriShape {
    int64_t count, R, ctas;
    int64_t ld_in, ld_out;
    int max_n;                               // rows of the largest matrix on the path
};

// The any-numbering block: TRI_GEN_LAUNCHES launches.
void tri_searches(const TriShape &sh, const TriLayout &L, const TriGraphView &G, const DagCounters *dc, cudaStream_t s) {
    const int64_t R = sh.R;
    const int gw = grid_for(R * 32, 256);
    const unsigned *any = L.gflags + 1;
    tri_gen_init_kernel<<<gw, 256, 0, s>>>(R, L.row_comp, L.ckind, L.dc, G, L.row_off, L.row_len, L.p_col, dc, any,
                                           L.gflags, L.cbad, L.cell);
    tri_gen_search_kernel<false><<<grid_for(R * 32, 32 * TRI_SEARCH_WARPS), 32 * TRI_SEARCH_WARPS, TRI_TAB_SMEM, s>>>(
        R, L.row_comp, L.ckind, L.cbad, L.dc, G, L.row_off, L.row_len, L.p_col, dc, any, L.gflags, L.cell, L.ovf, TRI_TAB,
        L.cam, L.cprod);
    tri_gen_search_kernel<true><<<4 * sm_count(), 32, tri_dense_smem(sh.max_n), s>>>(
        R, L.row_comp, L.ckind, L.cbad, L.dc, G, L.row_off, L.row_len, L.p_col, dc, any, L.gflags, L.cell, L.ovf,
        sh.max_n, L.cam, L.cprod);
    tri_gen_first_kernel<<<gw, 256, 0, s>>>(R, L.row_comp, L.ckind, L.cbad, L.row_off, L.row_len, dc, any, L.gflags,
                                            L.cell, L.cfm);
}

// Every launch of the DAG path, in stream order, with no host synchronisation when `captured`
// (the level loop then is a while node).  Returns the number of kernel launches issued.
template <typename T>
int tri_enqueue(const TriShape &sh, const TriLayout &L, const T *in, T *out, cudaStream_t s, bool captured,
                const RowStats &rs, DagCounters **dcount, int64_t *launches) {
    const int64_t R = sh.R;
    const int count = (int)sh.count;
    // 1. scan
    {
        cudaEvent_t t = timer_begin(4, s);
        note_launches(1);
        tri_scan_kernel<T><<<(unsigned)sh.ctas, TRI_THREADS, 0, s>>>(in, sh.ld_in, L.dc, L.dpre, count, L.slot_col,
                                                                     L.slot_val, L.row_cnt, L.row_comp, L.cflags,
                                                                     nullptr);
        RBG_CUDA_TRY(cudaGetLastError());
        timer_end(4, t, s);
    }
    // 2. CSR of the candidates and their closure by levels
    cudaEvent_t tdag = timer_begin(5, s);
    note_launches(4);
    tri_kind_kernel<<<(unsigned)std::min<int64_t>((count + 255) / 256, 1024), 256, 0, s>>>(
        count, L.dc, L.cflags, 1, L.ckind, L.cam, L.cfm, L.cprod, L.cbad, L.gflags + 1);
    tri_count_kernel<<<grid_for(R + 1, 256), 256, 0, s>>>(R, L.row_cnt, L.row_comp, L.ckind, L.indptr);
    size_t tb = L.scan_tmp;
    RBG_CUDA_TRY(cub::DeviceScan::ExclusiveSum(L.tmp, tb, L.indptr, L.indptr, (int)(R + 1), s));
    tri_csr_fill_kernel<<<grid_for(R, 256), 256, 0, s>>>(R, L.row_comp, L.ckind, L.dc, L.indptr, L.slot_col,
                                                        L.slot_val, L.a_col, L.a_val);
    RBG_CUDA_TRY(cudaGetLastError());
    *launches += 5;
    rbg_csr_t A{R, R, L.indptr, L.a_col, L.a_val};
    DagChildren kids;
    int rc = dag_enqueue(&A, R * TRI_CAP, L.dag_ws, L.p_col, L.p_val, L.pool, L.row_off, L.row_len, s, captured,
                         dcount, &kids, launches);
    if (rc) return rc;
    timer_end(5, tdag, s);
    // 2b. matrices in any numbering: the searches from every vertex (every kernel returns at once
    // when the batch holds none; a recorded graph skips the block by an IF node)
    {
        cudaEvent_t tg = timer_begin(8, s);
        const DagCounters *dcn = *dcount;
        const unsigned *any = L.gflags + 1;
        RBG_CUDA_TRY(cudaMemsetAsync(L.ovf, 0, 4, s));
        auto body = [&](cudaStream_t b) -> int {
            const TriGraphView G{L.indptr, nullptr, L.a_col, L.a_val, kids.coff, nullptr, kids.children};
            tri_searches(sh, L, G, dcn, b);
            RBG_CUDA_TRY(cudaGetLastError());
            return (int)RBG_OK;
        };
        if (captured) {
            rc = tri_captured_if(
                s, [&](cudaGraphConditionalHandle h) { tri_gen_gate_kernel<<<1, 32, 0, s>>>(dcn, any, L.gflags + 2, h); },
                body);
            *launches += 1;                  // the gate; the block is counted when it runs
        } else {
            note_launches(TRI_GEN_LAUNCHES);
            rc = body(s);
            *launches += TRI_GEN_LAUNCHES;
        }
        if (rc) return rc;
        timer_end(8, tg, s);
    }
    // 3. statistics
    {
        cudaEvent_t t = timer_begin(6, s);
        note_launches(1);
        const int64_t ctas = (int64_t)sm_count() * TRI_STATS_CTAS;
        const int run = dag_stats_run(R, ctas * TRI_STATS_GROUPS);
        const int64_t need = (R + (int64_t)run * TRI_STATS_GROUPS - 1) / ((int64_t)run * TRI_STATS_GROUPS);
        tri_stats_kernel<<<(unsigned)std::max<int64_t>(1, std::min<int64_t>(need, ctas)), TRI_THREADS, 0, s>>>(
            R, L.row_comp, L.ckind, L.dc, L.indptr, L.a_col, L.a_val, L.row_off, L.row_len, L.p_col, L.p_val, *dcount,
            L.cam, L.cfm, L.cprod, run);
        RBG_CUDA_TRY(cudaGetLastError());
        timer_end(6, t, s);
    }
    // 4. dense rows of the accepted matrices (decided on the device from the statistics)
    {
        cudaEvent_t t = timer_begin(7, s);
        note_launches(1);
        tri_write_kernel<T><<<(unsigned)sh.ctas, TRI_THREADS, 0, s>>>(in, sh.ld_in, out, sh.ld_out, L.dc, L.dpre,
                                                                      count, L.ckind, L.cam, L.cbad, *dcount,
                                                                      L.gflags, L.row_off, L.row_len, L.p_col,
                                                                      L.p_val, rs, L.cfm, L.cprod, L.cflags, L.res);
        RBG_CUDA_TRY(cudaGetLastError());
        timer_end(7, t, s);
    }
    *launches += 2;
    return RBG_OK;
}

// ------------------------------------------------------------------------------------------
// RBG_MODE_GRAPH: the whole sequence recorded once per layout and replayed
// ------------------------------------------------------------------------------------------
struct TriGraphKey {
    int device, tbytes;
    const void *in;
    void *out;
    unsigned char *ws;
    size_t ws_bytes;
    int64_t ld_in, ld_out;
    std::vector<int64_t> sizes, in_off, out_off;
    RowStats rs;
    bool operator==(const TriGraphKey &o) const {
        return device == o.device && tbytes == o.tbytes && in == o.in && out == o.out && ws == o.ws &&
               ws_bytes == o.ws_bytes && ld_in == o.ld_in && ld_out == o.ld_out && sizes == o.sizes &&
               in_off == o.in_off && out_off == o.out_off && rs == o.rs;
    }
};
struct TriGraph {
    TriGraphKey key;
    cudaGraphExec_t exec;
    DagCounters *dcount;
    int64_t launches;                        // outside the level loop
    unsigned long long stamp;
};
std::mutex g_tri_graph_mu;
std::vector<TriGraph> g_tri_graphs;
unsigned long long g_tri_clock = 0;
constexpr size_t TRI_GRAPH_CACHE = 8;

// Record the sequence into a graph on a private stream (the caller's may be the legacy default
// stream, which cannot be captured); nothing runs while recording.
template <typename T>
int tri_record(const TriShape &sh, const TriLayout &L, const T *in, T *out, const RowStats &rs, TriGraph &g) {
    static thread_local cudaStream_t cap = nullptr;
    if (!cap) RBG_CUDA_TRY(cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking));
    RBG_CUDA_TRY(cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal));
    launch_recording(true);
    int64_t launches = 0;
    const int rc = tri_enqueue<T>(sh, L, in, out, cap, true, rs, &g.dcount, &launches);
    launch_recording(false);
    cudaGraph_t graph = nullptr;
    const cudaError_t ec = cudaStreamEndCapture(cap, &graph);
    if (rc || ec != cudaSuccess) {
        if (graph) cudaGraphDestroy(graph);
        return rc ? rc : RBG_ERR_CUDA;
    }
    const cudaError_t ei = cudaGraphInstantiate(&g.exec, graph, 0);
    cudaGraphDestroy(graph);
    if (ei != cudaSuccess) return RBG_ERR_CUDA;
    g.launches = launches;
    return RBG_OK;
}

}  // namespace

namespace {

// The host's part of one call over `count` matrices: the tables, the layout and the results.
template <typename T> struct TriCall {
    int64_t count;
    const int64_t *sizes, *in_off, *out_off;
    int64_t ld_in, ld_out;
    const T *in;
    T *out;
    unsigned char *ws;
    size_t ws_bytes;
    uint32_t mode;
    cudaStream_t s;
    const RowStats &rs;
    TriShape sh;
    TriLayout L;
    std::vector<unsigned char> head;         // the head of the layout in its starting state
    std::vector<TriOut> res;
    DagCounters hd;

    // rows and CTAs of the call; false: no matrix is within the path's sizes
    bool shape() {
        sh = TriShape{count, 0, 0, ld_in, ld_out, 0};
        for (int64_t i = 0; i < count; ++i) {
            const int64_t n = rows(i);
            sh.R += n;
            sh.ctas += (n + TRI_ROWS - 1) / TRI_ROWS;
            sh.max_n = std::max<int>(sh.max_n, (int)n);
        }
        return sh.R > 0 && sh.R * TRI_CAP <= INT32_MAX;
    }
    int64_t rows(int64_t i) const { return (sizes[i] > 0 && sizes[i] <= TRI_MAX_N) ? sizes[i] : 0; }
    // carve the workspace; false: no room for a closure (the other paths decide)
    bool layout(bool is_short) {
        tri_layout(nullptr, ws_bytes, (size_t)count, (size_t)sh.R, is_short, L);
        if (L.pool < 4 * sh.R) return false;
        TriLayout H;                         // the same offsets over the host's copy of the head
        head.assign(L.head, 0);
        tri_layout(head.data(), ws_bytes, (size_t)count, (size_t)sh.R, is_short, H);
        tri_layout(ws, ws_bytes, (size_t)count, (size_t)sh.R, is_short, L);
        int64_t row = 0, cta = 0;
        for (int64_t i = 0; i < count; ++i) {
            const int64_t n = rows(i);
            H.dc[i] = TriComp{n, in_off[i], out_off[i], row};
            H.dpre[i] = cta;
            H.cam[i] = H.cfm[i] = -1;
            row += n;
            cta += (n + TRI_ROWS - 1) / TRI_ROWS;
        }
        H.dpre[count] = cta;
        return true;
    }
    int upload() {
        HostStaging hs(s, head.size() + (size_t)count * sizeof(TriOut) + sizeof(DagCounters) + 512);
        return hs.up(ws, head.data(), head.size());
    }
    int read(const DagCounters *dcount, unsigned *gate_ran) {
        res.resize((size_t)count);
        HostStaging hs(s, (size_t)count * sizeof(TriOut) + sizeof(DagCounters) + 128);
        int rc = hs.down(res.data(), L.res, (size_t)count * sizeof(TriOut));
        if (!rc) rc = hs.down(&hd, dcount, sizeof(hd));
        if (!rc && gate_ran) rc = hs.down(gate_ran, L.gflags + 2, 4);
        if (!rc) rc = hs.finish();
        return rc;
    }
};

template <typename T> int tri_levels(TriCall<T> &c) {
    if (!c.layout(false)) return RBG_OK;
    int rc = c.upload();
    if (rc) return rc;
    DagCounters *dcount = nullptr;
    int64_t fixed_launches = -1;             // >= 0: a graph ran; its level loop is counted below
    if ((c.mode & RBG_MODE_GRAPH) && !timer_on()) {
        int dev = 0;
        RBG_CUDA_TRY(cudaGetDevice(&dev));
        const int64_t count = c.count;
        TriGraphKey key{dev, (int)sizeof(T), c.in, c.out, c.ws, c.ws_bytes, c.ld_in, c.ld_out,
                        std::vector<int64_t>(c.sizes, c.sizes + count),
                        std::vector<int64_t>(c.in_off, c.in_off + count),
                        std::vector<int64_t>(c.out_off, c.out_off + count), c.rs};
        std::lock_guard<std::mutex> lk(g_tri_graph_mu);
        TriGraph *hit = nullptr;
        for (auto &e : g_tri_graphs)
            if (e.key == key) hit = &e;
        if (!hit) {
            TriGraph g;
            g.key = std::move(key);
            rc = tri_record<T>(c.sh, c.L, c.in, c.out, c.rs, g);
            if (rc) return rc;
            if (g_tri_graphs.size() >= TRI_GRAPH_CACHE) {
                size_t old = 0;
                for (size_t k = 1; k < g_tri_graphs.size(); ++k)
                    if (g_tri_graphs[k].stamp < g_tri_graphs[old].stamp) old = k;
                RBG_CUDA_TRY(cudaDeviceSynchronize());   // the evicted graph may still run on another stream
                cudaGraphExecDestroy(g_tri_graphs[old].exec);
                g_tri_graphs.erase(g_tri_graphs.begin() + (long)old);
            }
            g_tri_graphs.push_back(std::move(g));
            hit = &g_tri_graphs.back();
        }
        hit->stamp = ++g_tri_clock;
        RBG_CUDA_TRY(cudaGraphLaunch(hit->exec, c.s));
        dcount = hit->dcount;
        fixed_launches = hit->launches;
    } else {
        int64_t launches = 0;
        rc = tri_enqueue<T>(c.sh, c.L, c.in, c.out, c.s, false, c.rs, &dcount, &launches);
        if (rc) return rc;
    }
    unsigned gate_ran = 0;
    rc = c.read(dcount, fixed_launches >= 0 ? &gate_ran : nullptr);
    if (rc) return rc;
    if (fixed_launches >= 0) {
        const int64_t iters = std::max<int64_t>(1, (c.hd.nlevels + DAG_GRAPH_CHUNK - 1) / DAG_GRAPH_CHUNK);
        note_launches(fixed_launches + iters * (3 * DAG_GRAPH_CHUNK + 1) + (gate_ran ? TRI_GEN_LAUNCHES : 0));
    }
    return RBG_OK;
}

// Short closures, first pass: scan, closure kernel, write.  Second pass, over the same scratch, for
// the matrices the first one left pending: their order, closure kernel, searches, write.
template <typename T> int tri_short(TriCall<T> &c, bool second) {
    if (!second) {
        if (!c.layout(true)) return RBG_OK;
        const int rc = c.upload();
        if (rc) return rc;
    }
    const TriLayout &L = c.L;
    const int count = (int)c.count;
    cudaStream_t s = c.s;
    note_launches(second ? 3 + TRI_GEN_LAUNCHES : 3);
    if (!second) {
        cudaEvent_t t = timer_begin(4, s);
        tri_scan_kernel<T><<<(unsigned)c.sh.ctas, TRI_THREADS, 0, s>>>(c.in, c.ld_in, L.dc, L.dpre, count, L.slot_col,
                                                                      L.slot_val, L.row_cnt, L.row_comp, L.cflags,
                                                                      L.state);
        timer_end(4, t, s);
    }
    {
        cudaEvent_t t = timer_begin(5, s);
        if (second)
            tri_order_kernel<<<(unsigned)count, TRI_ORDER_THREADS, sizeof(TriOrderSmem), s>>>(
                L.dc, L.ckind, L.slot_col, L.row_cnt, L.order, L.coff, L.kid_cnt, L.children, L.cbad, L.ticket,
                L.gflags + 1);
        const int64_t need = (c.sh.R + TRI_PULL_WARPS - 1) / TRI_PULL_WARPS, most = (int64_t)TRI_PULL_CTAS * sm_count();
        tri_pull_kernel<<<(unsigned)std::min<int64_t>(need, most), 32 * TRI_PULL_WARPS, 0, s>>>(
            c.sh.R, L.row_comp, L.dc, L.cflags, L.slot_col, L.slot_val, L.row_cnt, L.state, L.row_off, L.row_len, L.p_col,
            L.p_val, L.pool, L.counters, L.ticket, L.ckind, L.cam, L.cfm, L.cprod, second ? L.order : nullptr, L.cbad);
        timer_end(5, t, s);
    }
    if (second) {
        cudaEvent_t t = timer_begin(8, s);
        RBG_CUDA_TRY(cudaMemsetAsync(L.ovf, 0, 4, s));
        const TriGraphView G{nullptr, L.row_cnt, L.slot_col, L.slot_val, L.coff, L.kid_cnt, L.children};
        tri_searches(c.sh, L, G, L.counters, s);
        timer_end(8, t, s);
    }
    {
        cudaEvent_t t = timer_begin(7, s);
        tri_write_kernel<T><<<(unsigned)c.sh.ctas, TRI_THREADS, 0, s>>>(c.in, c.ld_in, c.out, c.ld_out, L.dc, L.dpre,
                                                                       count, L.ckind, L.cam, L.cbad, L.counters,
                                                                       L.gflags, L.row_off, L.row_len, L.p_col,
                                                                       L.p_val, c.rs, L.cfm, L.cprod, L.cflags, L.res);
        timer_end(7, t, s);
    }
    RBG_CUDA_TRY(cudaGetLastError());
    return c.read(L.counters, nullptr);
}

// The call's results; `pending`: only of matrices marked so.  Returns how many stay pending.
template <typename T>
int64_t tri_take_results(const TriCall<T> &c, bool pending, rbg_result_t *results, char *closed) {
    int64_t left = 0;
    for (int64_t i = 0; i < c.count; ++i) {
        if (pending && closed[i] != (char)TRI_PENDING) continue;
        closed[i] = TRI_OPEN;
        if (c.res.empty() || (c.hd.flags & TRI_DAG_BAD)) continue;   // nothing of the DAG path is used
        const TriOut &h = c.res[(size_t)i];
        closed[i] = (char)h.verdict;
        left += h.verdict == TRI_PENDING;
        if (h.verdict != TRI_CLOSED) continue;
        rbg_result_t &r = results[i];
        r.status = RBG_OK;
        r.flags = 0;
        r.diameter = h.diameter;
        r.k = r.i = r.j = -1;
        r.path = RBG_PATH_DAG;
        r.executed = (int64_t)h.executed;
    }
    return left;
}

}  // namespace

template <typename T>
int tri_batch(int64_t count, const int64_t *sizes, const int64_t *in_off, const int64_t *out_off, int64_t ld_in,
              int64_t ld_out, const T *in, T *out, rbg_result_t *results, char *closed, unsigned char *ws,
              size_t ws_bytes, uint32_t mode, cudaStream_t s, const RowStats &rs) {
    if (count <= 0 || count > INT32_MAX || !ws) return RBG_OK;
    {
        const int rc = tri_configure();     // before any capture: kernel attributes per device
        if (rc) return rc;
    }
    TriCall<T> c{count, sizes, in_off, out_off, ld_in, ld_out, in, out, ws, ws_bytes, mode, s, rs};
    if (!c.shape()) return RBG_OK;
    // up to TRI_PULL_ROWS rows the levels' launches cost more than the rows: warps that wait for
    // their parents.  Beyond, waiting warps would fill the GPU (rows of one family are neighbours)
    // and the levels, each as wide as the batch, are faster.
    const bool is_short = c.sh.R <= TRI_PULL_ROWS;
    int rc = is_short ? tri_short(c, false) : tri_levels(c);
    if (rc) return rc;
    if (tri_take_results(c, false, results, closed) == 0) return RBG_OK;
    rc = tri_short(c, true);
    if (!rc) tri_take_results(c, true, results, closed);
    return rc;
}

template int tri_batch<int32_t>(int64_t, const int64_t *, const int64_t *, const int64_t *, int64_t, int64_t,
                                const int32_t *, int32_t *, rbg_result_t *, char *, unsigned char *, size_t, uint32_t,
                                cudaStream_t, const RowStats &);
template int tri_batch<int64_t>(int64_t, const int64_t *, const int64_t *, const int64_t *, int64_t, int64_t,
                                const int64_t *, int64_t *, rbg_result_t *, char *, unsigned char *, size_t, uint32_t,
                                cudaStream_t, const RowStats &);

}  // namespace rbg

// Frees the DAG path's cached CUDA graphs (device memory is never held by this library outside
// rbg_fw_dense_noalloc's fixed array).
extern "C" int32_t rbg_release_scratch(void) {
    std::lock_guard<std::mutex> lk(rbg::g_tri_graph_mu);
    if (!rbg::g_tri_graphs.empty()) RBG_CUDA_TRY(cudaDeviceSynchronize());
    for (auto &g : rbg::g_tri_graphs) cudaGraphExecDestroy(g.exec);
    rbg::g_tri_graphs.clear();
    return RBG_OK;
}
