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
// computed here row by row.  Above the diagonal (edges to higher numbers) it is the
// mirror image: before step k, W(i, k) = C(i, k) and W(k, j) = A(k, j).
//
// In the clean regime (off-diagonal values 0 or >= 2, diagonal in {-1, 0, 1}) products with the
// diagonal change nothing and a cell only decreases once it holds a value, so the largest value
// the loop ever writes -- the diameter's source -- is, per cell, its first value: A(i, j) (or step 0's
// product where that is less, as the loop looks at a value after the step: tri_gen_init_kernel), else
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
// vertex that no topological order reaches (a cycle, or below one) sends its matrix on.
//
// Pipeline (one call): scan the dense rows (clean-regime test, which side of the diagonal, up to
// TRI_CAP off-diagonal entries per row) -> the closure kernel, a warp per row that waits for its
// parents, with the statistics (largest product MSB, largest first-value MSB) -> the dense rows of the
// accepted matrices written from the closure rows, one result record per matrix -> read back.  When
// that left matrices in any numbering, a second pass over the same scratch orders their rows, closes
// them with the same kernel, runs the searches and writes them.  Every accept / reject decision is
// made on the device; scratch is carved from the caller's workspace.
#include <cuda_runtime.h>
#include <cub/cub.cuh>
#include <string.h>
#include <algorithm>
#include <vector>
#include "rbg_internal.cuh"
#include "dag_rows.cuh"

namespace rbg {
namespace {

constexpr int TRI_ROWS = 8;                  // rows per CTA, one warp each
constexpr int TRI_THREADS = 32 * TRI_ROWS;
constexpr int TRI_CAP = 16;                  // off-diagonal entries per row the scan keeps
constexpr int64_t TRI_FAT_CTAS = 2048;       // CTAs of eight rows from which a call is `fat` (tri_cta_rows)
constexpr int64_t TRI_MAX_N = DAG_MAX_N;     // rows of a matrix on this path (bitmap size)
constexpr int TRI_BM_WORDS = (int)(TRI_MAX_N / 32);
constexpr unsigned TF_UNCLEAN = 1u, TF_BELOW = 2u, TF_ABOVE = 4u, TF_WIDE = 8u;
constexpr int KIND_NONE = DAG_KIND_NONE, KIND_BELOW = DAG_KIND_BELOW, KIND_ABOVE = DAG_KIND_ABOVE;
constexpr int KIND_GENERAL = DAG_KIND_GENERAL;
constexpr int KIND_PENDING = -1;             // any numbering: left to the second pass
constexpr int TRI_TOP = DAG_TOP_MSB;         // products reaching bit 31 leave the path

struct TriComp {
    int64_t n, in_off, out_off, row_base;    // row_base: first batch-global row
};

constexpr int32_t TRI_PENDING = 3;           // closed by a second pass of the call

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

// The row number q of place p: qstart[q] <= p < qstart[q + 1], q < nq.
__device__ __forceinline__ int tri_place_row(const int32_t *__restrict__ qstart, int nq, int p) {
    int q = 0;
    for (int hi = nq - 1; q < hi;) {
        const int mid = (q + hi + 1) >> 1;
        if (qstart[mid] <= p) q = mid;
        else hi = mid - 1;
    }
    return q;
}

// Rows of a matrix per CTA of the scan and the write.  A warp takes one; in calls of many CTAs (`fat`)
// several, more of the short ones, as what a CTA looks up before its first row otherwise takes longer than
// its rows.  16000 pedigrees of 16 to 1024 rows (8.2 GB): scan and write 2.87 + 2.89 ms with half the
// rows, 2.04 + 2.00 with these, 2.03 + 1.92 with twice the rows of the shortest; 512 pedigrees of 16 to 4096
// rows (3.5 GB): 606 + 603, 569 + 566 and 565 + 564 us.  A call of few CTAs leaves SMs idle that way.
__host__ __device__ __forceinline__ int tri_cta_rows(int64_t n, bool fat) {
    return !fat ? TRI_ROWS : n <= 256 ? 8 * TRI_ROWS : n <= 1024 ? 4 * TRI_ROWS : 2 * TRI_ROWS;
}

// For the calls of many CTAs: the matrix of every CTA of the scan and the write, and the places of the
// closure kernel's rows, each a search that is a chain of dependent loads where it is needed.
__global__ void tri_map_kernel(const int64_t *__restrict__ pre, int count, int64_t ctas, int32_t *__restrict__ cta_comp,
                               const int32_t *__restrict__ qstart, int nq, const int32_t *__restrict__ tmat,
                               int2 *__restrict__ place, int places) {
    const int64_t step = (int64_t)gridDim.x * blockDim.x, first = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (int64_t c = first; c < ctas; c += step) cta_comp[c] = tri_find(pre, count, c);
    for (int64_t p = first; p < places; p += step) {
        const int q = tri_place_row(qstart, nq, (int)p);
        place[p] = make_int2(tmat[(int)p - qstart[q]], q);
    }
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
            c4 = 1;
        }
    }
    if (!__any_sync(0xffffffffu, c4 != 0)) return;
    const unsigned below = (1u << lane) - 1u;
    int pos = cnt;                           // entries before the lane's
#pragma unroll
    for (int k = 0; k < E; ++k) {
        const unsigned m = __ballot_sync(0xffffffffu, v[k] != 0);
        pos += __popc(m & below);
        cnt += __popc(m);
    }
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
}

// A warp per row, or several rows one after another: clean-regime test, side of the diagonal, the row's
// off-diagonal entries in column order in its slots, and the row's starting state.  Bound by the read of
// the matrix: the vectors on the row's 16-byte grid are loaded 16 bytes per lane, four in flight per lane
// while the four before (of this row or the one before) are taken; a vector of zeros (the common case)
// costs one vote.
template <typename T>
__global__ void __launch_bounds__(TRI_THREADS, 4)
tri_scan_kernel(const T *__restrict__ in, int64_t ld_in, const TriComp *__restrict__ comps,
                const int64_t *__restrict__ pre, int count, bool fat, const int32_t *__restrict__ cta_comp,
                int32_t *__restrict__ slot_col, int32_t *__restrict__ slot_val, int32_t *__restrict__ row_cnt,
                int32_t *__restrict__ row_comp, unsigned *__restrict__ cflags, unsigned long long *__restrict__ state) {
    constexpr int E = TriVec<T>::E;
    const int ci = cta_comp ? cta_comp[blockIdx.x] : tri_find(pre, count, blockIdx.x);
    const TriComp c = comps[ci];
    const int n = (int)c.n, rows = tri_cta_rows(c.n, fat);
    const int first = (int)(((int64_t)blockIdx.x - pre[ci]) * rows), end = min(n, first + rows);
    const int lane = threadIdx.x & 31;
    int i = first + (threadIdx.x >> 5);
    if (i >= end) return;                    // warp-uniform
    const T *row;
    int head, nv, tail;                      // columns before the first 16-byte boundary, vectors, columns after
    auto start = [&](int r) {
        row = in + c.in_off + (int64_t)r * (ld_in ? ld_in : c.n);
        const int lead = (int)(((16 - ((uintptr_t)row & 15)) & 15) / sizeof(T));
        head = lead < n ? lead : n;
        nv = (n - head) / E;
        tail = n - head - E * nv;
    };
    T ends = 0;                              // lane k < E: head column k; lane E + k: tail column k
    int4 x[4];                               // vectors s0 + 32 u + lane
    auto load = [&](int s0) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int q = s0 + 32 * u + lane;
            x[u] = q < nv ? *reinterpret_cast<const int4 *>(row + head + E * q) : make_int4(0, 0, 0, 0);
        }
    };
    auto load_ends = [&]() {
        ends = 0;
        if (lane < head) ends = row[lane];
        else if (lane >= E && lane - E < tail) ends = row[n - tail + lane - E];
    };
    start(i);
    load_ends();
    load(0);
    unsigned all = 0;
    while (true) {
        const int64_t g = c.row_base + i;
        const int h = head, nvec = nv, tl = tail;
        unsigned flags = 0;
        int cnt = 0;
        T v1[1];
        const T ends_now = ends;
        if (h) {                             // columns 0 .. head - 1, one per lane
            v1[0] = lane < h ? ends_now : (T)0;
            tri_take<T, 1>(v1, lane, lane < h ? 1 : 0, i, lane, g, slot_col, slot_val, flags, cnt);
        }
        const bool more = i + TRI_ROWS < end;
        int s0 = 0;
        do {
            int4 y[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) y[u] = x[u];
            if (s0 + 128 < nvec) {
                load(s0 + 128);
            } else if (more) {
                start(i + TRI_ROWS);
                load_ends();
                load(0);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {    // in column order
                const int q = s0 + 32 * u + lane;
                // all-zero vectors (a zero diagonal included) leave nothing to take
                if (__any_sync(0xffffffffu, (y[u].x | y[u].y | y[u].z | y[u].w) != 0)) {
                    T v[E];
                    TriVec<T>::split(y[u], v);
                    tri_take<T, E>(v, h + E * q, q < nvec ? E : 0, i, lane, g, slot_col, slot_val, flags, cnt);
                }
            }
            s0 += 128;
        } while (s0 < nvec);
        if (tl) {
            v1[0] = __shfl_sync(0xffffffffu, ends_now, (lane + E) & 31);
            if (lane >= tl) v1[0] = 0;
            tri_take<T, 1>(v1, n - tl + lane, lane < tl ? 1 : 0, i, lane, g, slot_col, slot_val, flags, cnt);
        }
        if (cnt > TRI_CAP) flags |= TF_WIDE;
        all |= flags;
        if (lane == 0) {
            row_cnt[g] = cnt;
            row_comp[g] = ci;
            state[g] = 0;                    // not closed yet
        }
        if (!more) break;
        i += TRI_ROWS;
    }
    all = __reduce_or_sync(0xffffffffu, all);
    // only flags not seen yet: an atomic per row on one word holds up the reads of its L2 slice
    // (64 matrices of 3000 to 4096 rows, 3.2 GB: 685 us with it, 509 without)
    if (lane == 0 && (all & ~__ldcg(cflags + ci))) atomicOr(cflags + ci, all);
}

// Every row found room in the pool and every wait ended; otherwise nothing of this call's DAG path is
// used.  A matrix with a cycle (only one with entries on both sides of the diagonal can hold one) is
// marked in cbad.
constexpr int TRI_DAG_BAD = 15;              // DagCounters::flags that reject the call's DAG path
constexpr int TRI_GAVE_UP = 8;               // a bounded wait ran out
__device__ __forceinline__ bool tri_dag_ok(const DagCounters *dc) { return !(dc->flags & TRI_DAG_BAD); }

// A closure row entry outside its matrix (which a consistent closure never holds): the access is
// skipped and the call's DAG path rejected (flag 4), so the blocked kernels decide.
constexpr int TRI_BAD_ROW = 4;

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

// The candidates' graph, vertices batch-global: rows of TRI_CAP slots (columns local to the matrix);
// the children of a vertex in any order.
struct TriGraphView {
    const int32_t *row_cnt, *col, *val;
    const int64_t *coff;
    const int32_t *kid_cnt, *children;
    __device__ __forceinline__ int64_t row(int64_t g, int &cnt) const {
        cnt = row_cnt[g];
        return g * TRI_CAP;
    }
    __device__ __forceinline__ int64_t kids(int64_t g, int &cnt) const {
        cnt = kid_cnt[g];
        return coff[g];
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

// One warp per candidate row of a general matrix: the cells of A's entries start with key 0, the other
// cells empty.  The loop looks at a value only after it has folded the step's product in, so the first
// value of such a cell is A's, or the product of step 0 where that is less (A(i, 0) (x) A(0, j); only
// numberings in which vertex 0 has parents and children hold one).  Cell q of the row is
// cell[row_off + q].
__global__ void tri_gen_init_kernel(int64_t R, const int32_t *__restrict__ row_comp, const int32_t *__restrict__ ckind,
                                    const TriComp *__restrict__ comps, TriGraphView G,
                                    const int64_t *__restrict__ row_off,
                                    const int32_t *__restrict__ row_len, const int32_t *__restrict__ p_col,
                                    const DagCounters *dc, const unsigned *any_gen, unsigned *gflags,
                                    const unsigned *__restrict__ cbad, uint32_t *__restrict__ cell) {
    if (!tri_dag_ok(dc) || !*any_gen) return;
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t g = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); g < R; g += warps) {
        const int ci = row_comp[g];
        if (ckind[ci] != KIND_GENERAL || cbad[ci]) continue;   // warp-uniform
        const int len = row_len[g];
        const int64_t o = row_off[g];
        for (int q = lane; q < len; q += 32) cell[o + q] = TRI_EMPTY;
        __syncwarp();
        const int64_t base = comps[ci].row_base;
        int cnt, cnt0;
        const int64_t e0 = G.row(g, cnt), z0 = G.row(base, cnt0);
        const uint32_t x = g != base && cnt > 0 && G.col[e0] == 0 ? (uint32_t)G.val[e0] : 0u;   // A(i, 0)
        for (int64_t e = e0 + lane; e < e0 + cnt; e += 32) {
            const int32_t c = G.col[e];
            uint32_t v = (uint32_t)G.val[e];             // a clean value: 2 <= v < 2^31
            for (int64_t z = z0; x != 0 && z < z0 + cnt0; ++z) {
                const uint32_t y = (uint32_t)G.val[z];
                if (G.col[z] == c) v = (uint32_t)min((uint64_t)v, ((uint64_t)(x - 1) << msb_u32(y)) + y);
            }
            const int64_t q = tri_find_col(p_col, o, len, (int32_t)(base + c));
            if (q < 0) atomicOr(gflags, 2u);
            else cell[q] = (uint32_t)msb_u32(v);
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
                    y = G.col[eq];
                    len = msb_u32((uint32_t)G.val[eq]);
                } else {
                    const int32_t c = G.children[eq];
                    y = c - (int)base;
                    int rc;                  // the edge's value, in the child's row
                    const int64_t r0 = G.row(c, rc);
                    for (int64_t e = r0; e < r0 + rc; ++e)
                        if (G.col[e] == xq) len = msb_u32((uint32_t)G.val[e]);
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
// The closure kernel
// ------------------------------------------------------------------------------------------
// Closed level by level, a batch is launches and their latency (three kernels a level, the children
// lists and row orders before them).  Here every row is a warp's, which waits for the row's parents
// itself.  The rows are taken in one order over all matrices: the first row of every matrix (of one with
// entries above the diagonal the last, in any numbering the first of tri_order_kernel's order), the
// second row of every matrix that has one, and so on.  A ticket is a few places of that order.  A row's
// parents so lie in the same ticket before it or in an earlier one, held by a warp that runs already, and
// every wait ends (it is bounded all the same); and as the rows in flight come from as many matrices as
// there are, a parent is nearly always done.  A finished row is published as one 64-bit word, its pool
// position and length, stored after a fence and read with an acquire; a warp publishes the rows of its
// ticket with one fence, but always before it waits.
//
// The row itself: with its products at most 32 entries, a lane each; the lanes that hold the same column
// take the least of their values and the first one's place is the count of smaller columns.  Longer rows
// mark the columns of their entries and of their parents' rows in a bitmap (a word per 32 columns),
// whose prefix counts give every column its place; the values meet there by atomic minima.  Either way
// tells a product that reaches a cell first, the statistics of dag_rows.cuh: below the diagonal while the
// parents are folded in (ascending, the loop's step order), above it in a second walk.
//
// One matrix is bound by latency, about 2 us per generation: n = 512 in 12 generations takes 90 us, 390
// by levels; n = 8192, int64: 320 us, 835 by levels.  Large batches are bound by the issue of about 500
// instructions per row and by their waits for L2: 411 000 rows of 512 pedigrees take 0.36 ms (0.76 by
// levels with their statistics), 3.9 M rows of 16000 pedigrees 2.2 ms (3.3).
constexpr int TRI_PULL_WARPS = 8;            // warps (rows) per CTA
constexpr int TRI_PULL_CTAS = 4;             // CTAs per SM
constexpr int TRI_PULL_BATCH = 8;            // rows per ticket, at most
constexpr int TRI_PULL_PART = 24;            // the tickets in flight: about a 24th of the rows
constexpr int TRI_PULL_BLOCK = 1024;         // pool entries a warp asks for at a time
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

// Places [qstart[q], qstart[q + 1]): row q of the matrices tmat[0 ..] (most rows first); place[p]: {matrix,
// q} where it has been written out.  A ticket is `batch` places; `block`: pool entries a warp asks for at a
// time (0: a row's).
struct TriTickets {
    const int2 *place;
    const int32_t *qstart, *tmat;
    int nq, places, batch, block;
};

// A row to close: its matrix, the kind, vertices and first row of that, the row, its number of entries and
// (TriCsrRows) their first position.
struct TriPlace {
    int ci, kind, n, base, g, cnt, e0;
};

// The rows of a batch of dense matrices: the scan's slots.
struct TriSlotRows {
    static constexpr bool CSR = false;
    TriTickets tk;
    const TriComp *comps;
    const unsigned *cflags, *cbad;
    int32_t *ckind;
    const int32_t *order, *col, *val, *cnt;
    __device__ __forceinline__ TriPlace at(int p) const {
        int2 pl;
        if (tk.place) {
            pl = tk.place[p];
        } else {
            pl.y = tk.nq == tk.places ? p : tri_place_row(tk.qstart, tk.nq, p);   // one matrix: its rows
            pl.x = tk.tmat[p - tk.qstart[pl.y]];
        }
        TriPlace m{pl.x, KIND_NONE, (int)comps[pl.x].n, (int)comps[pl.x].row_base, 0, 0, 0};
        const unsigned f = cflags[m.ci];
        if (order) {                         // the matrices in any numbering (tri_order_kernel)
            m.kind = cbad[m.ci] ? KIND_NONE : ckind[m.ci];
        } else {
            m.kind = (f & (TF_UNCLEAN | TF_WIDE)) ? KIND_NONE
                     : ((f & TF_BELOW) && (f & TF_ABOVE)) ? KIND_PENDING
                     : (f & TF_ABOVE) ? KIND_ABOVE : KIND_BELOW;
            if (pl.y == 0) ckind[m.ci] = m.kind;
        }
        if (m.kind > KIND_NONE) {
            // a matrix with entries above the diagonal goes from its last row to its first
            m.g = order ? order[m.base + pl.y] : m.base + (m.kind == KIND_ABOVE ? m.n - 1 - pl.y : pl.y);
            m.cnt = cnt[m.g];                // at most TRI_CAP
        }
        return m;
    }
    __device__ __forceinline__ int64_t begin(int64_t g, int) const { return g * TRI_CAP; }
    __device__ __forceinline__ int64_t row(int64_t g, int &n) const {
        n = cnt[g];
        return g * TRI_CAP;
    }
    __device__ __forceinline__ int column(int64_t e, int) const { return col[e]; }
};

// The components of a graph (CSR, the off-diagonal entries): the vertices in the order `order`, by their
// place among their component's (from the last for entries above the diagonal); a component is the
// matrix of its lowest to its highest vertex.
struct TriCsrRows {
    static constexpr bool CSR = true;
    TriTickets tk;
    const int32_t *order, *label, *kind, *sorted_vertex;
    const int64_t *start, *ptr;
    const int32_t *col, *val;
    const int32_t *diag;
    int *cmax;                               // per component, the largest value of its rows
    __device__ __forceinline__ TriPlace at(int p) const {
        const int v = order[p], c = label[v];
        const int64_t e0 = ptr[v], s0 = start[c], s1 = start[c + 1];
        const int lo = sorted_vertex[s0];
        return TriPlace{c, kind[c], sorted_vertex[s1 - 1] - lo + 1, lo, v, (int)(ptr[v + 1] - e0), (int)e0};
    }
    __device__ __forceinline__ int64_t begin(int64_t, int e0) const { return e0; }
    __device__ __forceinline__ int64_t row(int64_t g, int &n) const {
        const int64_t e0 = ptr[g];
        n = (int)(ptr[g + 1] - e0);
        return e0;
    }
    __device__ __forceinline__ int column(int64_t e, int base) const { return col[e] - base; }
};

template <typename Rows>
__global__ void __launch_bounds__(32 * TRI_PULL_WARPS, TRI_PULL_CTAS)
tri_pull_kernel(Rows A, unsigned long long *state, int64_t *__restrict__ row_off, int32_t *__restrict__ row_len,
                int32_t *p_col, int32_t *p_val, int64_t capacity, DagCounters *dc, int *ticket,
                int *__restrict__ cam, int *__restrict__ cfm, int32_t *__restrict__ row_prods) {
    const TriTickets &tk = A.tk;
    if (Rows::CSR && (dc->flags & TRI_BAD_ROW)) return;   // set before the launch
    __shared__ TriPullWarp warps[TRI_PULL_WARPS];
    TriPullWarp &S = warps[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    unsigned long long blk_at = 0;           // lane 0: the warp's part of the pool
    int blk_left = 0;
    while (true) {
        int t = 0;
        if (lane == 0) t = atomicAdd(ticket, 1);
        t = __shfl_sync(0xffffffffu, t, 0);
        if ((int64_t)t * tk.batch >= tk.places) return;
        // lane u: the ticket's place u
        const int here = min(tk.batch, tk.places - t * tk.batch);
        TriPlace m{0, KIND_NONE, 0, 0, 0, 0, 0};
        if (lane < here) m = A.at(t * tk.batch + lane);
        int m_am = -1, m_fm = -1, m_prods = 0, m_mx = 0;   // lane u: the statistics of place u
        unsigned long long m_pub = 0;        // and its state, while it is not published yet
        // the closed rows' states, all with one fence (which a row otherwise waits for in every case)
        auto publish = [&]() {
            __syncwarp();
            if (m_pub) {
                tri_release(state + m.g, m_pub);
                row_off[m.g] = (int64_t)(m_pub >> TRI_STATE_LEN_BITS) - 1;
                row_len[m.g] = (int)(m_pub & ((1u << TRI_STATE_LEN_BITS) - 1u));
            }
            m_pub = 0;
            __syncwarp();
        };
        int w_next = -1, v_next = 0;         // the next row's slots and its parents' states
        unsigned long long st_next = 0;
        {
            const int64_t e0 = A.begin(__shfl_sync(0xffffffffu, m.g, 0), __shfl_sync(0xffffffffu, m.e0, 0));
            const int base0 = __shfl_sync(0xffffffffu, m.base, 0);
            if (lane < __shfl_sync(0xffffffffu, m.cnt, 0)) {
                w_next = A.column(e0 + lane, base0);
                v_next = A.val[e0 + lane];
            }
        }
        for (int u = 0; u < here; ++u) {
            const int kind = __shfl_sync(0xffffffffu, m.kind, u);   // warp-uniform
            const int g = __shfl_sync(0xffffffffu, m.g, u), cnt = __shfl_sync(0xffffffffu, m.cnt, u);
            const int n = __shfl_sync(0xffffffffu, m.n, u), base = __shfl_sync(0xffffffffu, m.base, u);
            const int words = (n + 31) >> 5;
            int w = w_next, v = v_next, len = 0;
            int64_t off = 0;
            unsigned long long st = st_next;
            // the next row's slots, while this row is closed
            {
                const int u1 = min(u + 1, here - 1);
                const int64_t e1 = A.begin(__shfl_sync(0xffffffffu, m.g, u1), __shfl_sync(0xffffffffu, m.e0, u1));
                const int cnt1 = __shfl_sync(0xffffffffu, m.cnt, u1), base1 = __shfl_sync(0xffffffffu, m.base, u1);
                st_next = 0;
                if (u1 > u && lane < cnt1) {
                    w_next = A.column(e1 + lane, base1);
                    v_next = A.val[e1 + lane];
                }
            }
            if (kind <= KIND_NONE) continue;
            int am = -1, fm = lane < cnt ? dag_row_msb(v) : -1, mx = 0;
            int prods = 0;
            auto mark = [&]() {                  // the bitmap, with the row's own columns
                for (int q = lane; q < words; q += 32) S.bm[q] = 0;
                __syncwarp();
                if (lane < cnt) atomicOr(&S.bm[w >> 5], 1u << (w & 31));
                __syncwarp();
            };
            if (tk.batch == 1) mark();           // while the parents are waited for
            // the parents' rows, as soon as they are published
            bool late = false;
            // a parent that is not there yet may be a row of this ticket, or wait for one
            if (__any_sync(0xffffffffu, lane < cnt && st == 0)) publish();
            if (lane < cnt) {
                for (int tries = 0; st == 0 && tries < TRI_PULL_TRIES; ++tries) st = tri_acquire(state + base + w);
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
            const int bound = total + cnt;
            if (lane == 0 && blk_left < bound) {
                blk_left = max(bound, tk.block);
                blk_at = atomicAdd(&dc->reserved, (unsigned long long)blk_left);
            }
            // candidate idx of the flattened rows: its column and product.  0 beyond the end, and for a product
            // past 31 bits, which would wrap: it is never a cell's minimum, as a matrix with such a minimum
            // leaves the path (in any numbering the recurrence forms products that the loop, which has a
            // shorter path by then, does not)
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
                if (idx < 0 || idx >= total) return 0;
                col = __ldcg(p_col + oq + (idx - xq)) - base;
                const int y = __ldcg(p_val + oq + (idx - xq));
                pm = dag_row_msb(vq) + dag_row_msb(y);
                return pm >= TRI_TOP ? 0 : cy_product(vq, y);
            };
            int nd = 0;                          // the row's entries
            unsigned long long at = 0;
            bool room = false, wide = false;
            auto take = [&]() {                  // their place in the pool; the rest is the warp's next rows'
                at = __shfl_sync(0xffffffffu, blk_at, 0);
                room = (int64_t)at + bound <= capacity;
                blk_at += nd;
                blk_left -= nd;
            };
            if (bound <= 32) {
                // a lane per entry and product: their places are the counts of smaller columns
                int cc, pm;
                int vv = candidate(lane - cnt, cc, pm);
                if (lane < cnt) cc = w, vv = v;
                am = max(am, pm);
                if (vv == 0) vv = INT_MAX;
                const unsigned same = __match_any_sync(0xffffffffu, cc);
                const bool lead = cc >= 0 && !(same & below);
                if (lead && kind == KIND_BELOW) fm = max(fm, pm);   // the cell's first product (pm < 0: A's entry)
                unsigned others = cc >= 0 ? same & ~(1u << lane) : 0u;
                while (__any_sync(0xffffffffu, others != 0)) {
                    const int x = __shfl_sync(0xffffffffu, vv, others ? __ffs(others) - 1 : lane);
                    others &= others - 1;
                    vv = min(vv, x);
                }
                unsigned leads = __ballot_sync(0xffffffffu, lead);
                nd = __popc(leads);
                int rank = 0;
                for (; leads; leads &= leads - 1) rank += __shfl_sync(0xffffffffu, cc, __ffs(leads) - 1) < cc;
                take();
                if (room && lead) {
                    p_col[at + rank] = base + cc;
                    p_val[at + rank] = vv;
                    if (Rows::CSR) mx = vv;
                    if (kind == KIND_ABOVE) S.col[rank] = base + cc, S.val[rank] = vv;
                }
                __syncwarp();
            } else {
                if (tk.batch > 1) mark();
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
                nd = __shfl_sync(0xffffffffu, run, 31);
                run -= mine;
                for (int q = lane * wl; q < min(words, (lane + 1) * wl); ++q) {
                    S.pre[q] = (unsigned short)run;
                    run += __popc(S.bm[q]);
                }
                take();
                wide = nd > TRI_PULL_VALS;    // the values meet in the pool instead
                int32_t *oc = wide ? p_col + at : S.col, *ov = wide ? p_val + at : S.val;
                if (room) {
                    for (int q = lane; q < nd; q += 32) ov[q] = INT_MAX;
                    if (wide) __threadfence();
                    __syncwarp();
                    auto put = [&](int col, int val) {
                        const int r = S.pre[col >> 5] + __popc(S.bm[col >> 5] & ((1u << (col & 31)) - 1u));
                        oc[r] = base + col;
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
                    if (Rows::CSR)
                        for (int q = lane; q < nd; q += 32) mx = max(mx, wide ? __ldcg(p_val + at + q) : S.val[q]);
                }
            }
            if (u + 1 < here) {              // the next row's parents, while this row is stored
                const int cnt1 = __shfl_sync(0xffffffffu, m.cnt, u + 1), base1 = __shfl_sync(0xffffffffu, m.base, u + 1);
                if (lane < cnt1) st_next = tri_acquire(state + base1 + w_next);
            }
            if (lane == 0 && !room) atomicOr(&dc->flags, 1);
            if (late) atomicOr(&dc->flags, TRI_GAVE_UP);
            if (lane == u) m_pub = ((at + 1) << TRI_STATE_LEN_BITS) | (unsigned long long)(room ? nd : 0);
            __syncwarp();
            if (kind == KIND_BELOW) prods = total;
            if (kind == KIND_ABOVE) {
                // steps k over the row ascending, each adding C(i, k) (x) A(k, .), two steps at a time
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
                        int kn;
                        const int64_t k0 = A.row(k, kn);
                        if (e < kn) {
                            j = A.column(k0 + e, base);
                            pm = dag_row_msb(kvv) + dag_row_msb(A.val[k0 + e]);
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
            am = __reduce_max_sync(0xffffffffu, am);
            fm = __reduce_max_sync(0xffffffffu, fm);
            if (lane == u) m_am = am, m_fm = fm, m_prods = prods;
            if (Rows::CSR) {
                mx = __reduce_max_sync(0xffffffffu, mx);
                if (lane == u) m_mx = mx;
            }
        }
        publish();
        // a matrix's maxima rarely grow: an atomic per row on one word would be the kernel's bound
        // (any numbering: the searches take the statistics)
        if (m.kind == KIND_BELOW || m.kind == KIND_ABOVE) {
            if constexpr (Rows::CSR) {
                m_mx = max(m_mx, A.diag[m.g]);
                if (m_mx > 0 && m_mx > __ldcg(A.cmax + m.ci)) atomicMax(A.cmax + m.ci, m_mx);
            } else {
                row_prods[m.g] = m_prods;
            }
            if (m_am > __ldcg(cam + m.ci)) atomicMax(cam + m.ci, m_am);
            if (m_fm > __ldcg(cfm + m.ci)) atomicMax(cfm + m.ci, m_fm);
        }
    }
}

// Second pass, one CTA per matrix: a matrix in any numbering gets its children
// lists and its rows in a topological order (Kahn's algorithm by levels, the counters and the
// frontier in shared memory, so a level costs two barriers and one read of the frontier's children);
// one with a cycle is marked in cbad, every other matrix is taken off the path (its result is read
// already).
constexpr int TRI_ORDER_THREADS = 1024;
// Shared memory of max_n vertices: int end[]: children of v: [end[v - 1], end[v]) of the matrix's list;
// int rem[]: parents not placed yet; unsigned short list[]: placed vertices.
inline size_t tri_order_smem_bytes(int max_n) { return (size_t)max_n * 10; }

__global__ void __launch_bounds__(TRI_ORDER_THREADS)
tri_order_kernel(const TriComp *__restrict__ comps, int32_t *ckind, const int32_t *__restrict__ slot_col,
                 const int32_t *__restrict__ row_cnt, int32_t *__restrict__ order, int64_t *__restrict__ coff,
                 int32_t *__restrict__ kid_cnt, int32_t *__restrict__ children, unsigned *__restrict__ cbad,
                 int *ticket, unsigned *any_gen, int max_n) {
    extern __shared__ __align__(16) unsigned char tri_order_smem[];
    int *s_end = reinterpret_cast<int *>(tri_order_smem), *s_rem = s_end + max_n;
    unsigned short *s_list = reinterpret_cast<unsigned short *>(s_rem + max_n);
    const int nthr = blockDim.x;
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
    for (int v = tid; v < n; v += nthr) s_end[v] = 0;
    __syncthreads();
    for (int v = tid; v < n; v += nthr) {
        const int m = row_cnt[g0 + v];
        s_rem[v] = m;
        for (int e = 0; e < m; ++e) atomicAdd(&s_end[slot_col[(g0 + v) * TRI_CAP + e]], 1);
    }
    __syncthreads();
    // exclusive scan of the counts, a run of consecutive vertices per thread
    const int run = (n + nthr - 1) / nthr;
    int sum = 0;
    for (int v = tid * run; v < min(n, (tid + 1) * run); ++v) sum += s_end[v];
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
        const int k = s_end[v];
        coff[g0 + v] = g0 * TRI_CAP + at;
        kid_cnt[g0 + v] = k;
        s_end[v] = at;                       // a cursor that ends at the list's end
        at += k;
    }
    __syncthreads();
    for (int v = tid; v < n; v += nthr) {
        const int m = s_rem[v];
        for (int e = 0; e < m; ++e)
            kids[atomicAdd(&s_end[slot_col[(g0 + v) * TRI_CAP + e]], 1)] = (int32_t)(g0 + v);
        if (m == 0) s_list[atomicAdd(&s_tail, 1)] = (unsigned short)v;
    }
    __syncthreads();                         // (the lists' writes are visible to the CTA)
    // levels: 8 lanes per frontier vertex
    int h = 0, tail = s_tail;
    __syncthreads();                         // everyone has the first level's end before it moves
    while (h < tail) {                       // block-uniform
        for (int q = h + (tid >> 3); q < tail; q += nthr >> 3) {
            const int v = s_list[q];
            for (int e = (v ? s_end[v - 1] : 0) + (tid & 7); e < s_end[v]; e += 8) {
                const int k = kids[e] - (int)g0;
                if (atomicSub(&s_rem[k], 1) == 1) s_list[atomicAdd(&s_tail, 1)] = (unsigned short)k;
            }
        }
        __syncthreads();
        h = tail;
        tail = s_tail;
        __syncthreads();
    }
    for (int q = tid; q < tail; q += nthr) order[g0 + q] = (int32_t)(g0 + s_list[q]);
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
                                          (int)tri_order_smem_bytes(TRI_MAX_N)));
        return (int)RBG_OK;
    });
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

// A warp per row of an accepted matrix, or several rows one after another.  Bound by the write of the
// matrix: the row is zeroed with full 16-byte vectors, while its entries are on their way, and the
// closure's entries and the diagonal are then stored over the zeros, which are still in L2 (built in
// shared memory first, the row costs two more passes over it there: 3.9 M rows of 16 to 1024 columns took
// 2.64 ms that way, 2.30 so).  The registers keep it at four CTAs per SM on purpose: with five, writes of
// more rows at a time, 512 pedigrees take 607 us for 591, with six 897.  In place, only the closure's
// entries are stored (the other cells already hold the result).  The row statistics are recorded when
// asked for (32-bit storage).  The first CTA of a matrix writes its result record.
template <typename T>
__global__ void __launch_bounds__(TRI_THREADS)
tri_write_kernel(const T *__restrict__ in, int64_t ld_in, T *__restrict__ out, int64_t ld_out,
                 const TriComp *__restrict__ comps, const int64_t *__restrict__ pre, int count, bool fat,
                 const int32_t *__restrict__ cta_comp, const int32_t *__restrict__ ckind, const int *__restrict__ cam,
                 const unsigned *__restrict__ cbad, const DagCounters *dc, const unsigned *gflags,
                 const int64_t *__restrict__ row_off, const int32_t *__restrict__ row_len,
                 const int32_t *__restrict__ p_col, const int32_t *__restrict__ p_val, RowStats rs,
                 const int *__restrict__ cfm, const unsigned long long *__restrict__ cprod,
                 const int32_t *__restrict__ row_prods, const unsigned *__restrict__ cflags, TriOut *__restrict__ res) {
    constexpr int E = TriVec<T>::E;
    const int ci = cta_comp ? cta_comp[blockIdx.x] : tri_find(pre, count, blockIdx.x);
    const bool accepted = tri_accepted(ci, ckind, cam, cbad, dc, gflags);   // block-uniform
    if ((int64_t)blockIdx.x == pre[ci] && threadIdx.x < 32) {
        unsigned long long prods = 0;        // the rows' products, summed here
        if (accepted && row_prods)
#pragma unroll 8
            for (int q = threadIdx.x; q < (int)comps[ci].n; q += 32) prods += (unsigned)row_prods[comps[ci].row_base + q];
        for (int o = 16; o; o >>= 1) prods += __shfl_xor_sync(0xffffffffu, prods, o);
        if (threadIdx.x == 0) {
            TriOut o;
            o.verdict = accepted ? TRI_CLOSED : tri_top_bit(ci, ckind, cam, cbad, dc, gflags) ? TRI_TOP_BIT
                        : ckind[ci] == KIND_PENDING ? TRI_PENDING
                        : (cflags[ci] & ~(TF_BELOW | TF_ABOVE)) != TF_WIDE ? TRI_OPEN
                        : !(cflags[ci] & TF_ABOVE) ? TRI_WIDE_BELOW
                        : !(cflags[ci] & TF_BELOW) ? TRI_WIDE_ABOVE : TRI_OPEN;
            o.diameter = cfm[ci] > 0 ? cfm[ci] : 0;
            o.executed = cprod[ci] + prods;
            res[ci] = o;
        }
    }
    if (!accepted) return;
    const TriComp c = comps[ci];
    const int n = (int)c.n, rows = tri_cta_rows(c.n, fat);
    const int first = (int)(((int64_t)blockIdx.x - pre[ci]) * rows), end = min(n, first + rows);
    const int lane = threadIdx.x & 31;
    const int32_t base = (int32_t)c.row_base;
    // the warp's rows i, i + 8, ..: what a row needs is read two rows ahead, its first 32 entries one
    struct Row {
        T diag;
        int at, len;
    };
    auto row_of = [&](int r) {
        Row x{0, 0, 0};
        if (r < end) {
            x.diag = in[c.in_off + (int64_t)r * (ld_in ? ld_in : c.n) + r];
            x.at = (int)row_off[c.row_base + r];
            x.len = row_len[c.row_base + r];
        }
        return x;
    };
    auto entry = [&](const Row &x, int q, int32_t &v) {   // column and value of entry q (INT_MAX past the end)
        if (q >= x.len) return INT_MAX;
        v = p_val[(int64_t)x.at + q];
        return p_col[(int64_t)x.at + q] - base;
    };
    const int i0 = first + (threadIdx.x >> 5);
    Row now = row_of(i0), next = row_of(i0 + TRI_ROWS);
    int32_t v_now = 0;
    int j_now = entry(now, lane, v_now);
    for (int i = i0; i < end; i += TRI_ROWS) {   // warp-uniform
        const Row later = row_of(i + 2 * TRI_ROWS);
        int32_t v_next = 0;
        const int j_next = entry(next, lane, v_next);
        const T *rin = in + c.in_off + (int64_t)i * (ld_in ? ld_in : c.n);
        T *rout = out + c.out_off + (int64_t)i * (ld_out ? ld_out : c.n);
        const T diag = now.diag;
        const int clen = now.len;
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
        if (rin != rout) {                   // in place the other cells hold the result already
            const int lead = (int)(((16 - ((uintptr_t)rout & 15)) & 15) / sizeof(T));
            const int head = lead < n ? lead : n, nv = (n - head) / E, tail = n - head - E * nv;
            for (int q = lane; q < nv; q += 32) reinterpret_cast<int4 *>(rout + head)[q] = make_int4(0, 0, 0, 0);
            if (lane < head) rout[lane] = 0;
            if (lane < tail) rout[n - tail + lane] = 0;
            __syncwarp();
            if (lane == 0) rout[i] = diag;
        }
        for (int q = lane; q < clen; q += 32) {
            int32_t v = v_now;
            const int j = q == lane ? j_now : entry(now, q, v);
            if ((unsigned)j >= (unsigned)n) {
                atomicOr(const_cast<int *>(&dc->flags), TRI_BAD_ROW);
                continue;
            }
            rout[j] = (T)v;
            mx = max(mx, v);
            mark(j >> 5);
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
                    if (rs.comp_max && mx > 0 && mx > __ldcg(rs.comp_max + ci)) atomicMax(rs.comp_max + ci, mx);
                }
            }
        }
        now = next;
        next = later;
        j_now = j_next;
        v_now = v_next;
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

struct TriShape {
    int64_t count, R, ctas;
    int64_t ld_in, ld_out;
    int max_n;                               // rows of the largest matrix on the path
    int nq;                                  // max_n, at least 1
    bool fat;                                // many CTAs: several short rows per warp, searches done once
};

// The scratch of one call, carved from the caller's workspace: the matrix table, the tickets,
// per-matrix flags, statistics and results with the call's counters (`head`, uploaded whole at the
// start of a call in its starting state), the scan's row slots, the rows' states, the second pass's
// order, children lists and searches, and the row pool in whatever remains.
struct TriLayout {
    TriComp *dc;
    int64_t *dpre, *row_off;
    int2 *place;                             // per row of the closure kernel's order
    int32_t *qstart, *tmat, *cta_comp;
    unsigned *cflags, *cbad, *gflags;        // gflags[0]: the searches' scratch is inconsistent; [1]: any general
    int32_t *ckind, *row_cnt, *row_comp, *slot_col, *slot_val, *row_len, *p_col, *p_val;
    int32_t *ovf;                            // any numbering: count and rows of the searches the table is too small for
    uint32_t *cell;                          // any numbering: per pool entry, the key of the cell's first value
    int *cam, *cfm;
    unsigned long long *cprod;
    TriOut *res;
    DagCounters *counters;
    int *ticket;
    unsigned long long *state;               // per row 0, or (pool position + 1) << 24 | length
    int32_t *row_prods;                      // products of a row (numbered in a topological order)
    int32_t *order, *kid_cnt, *children;     // any numbering: rows in a topological order and the children
    int64_t *coff;                           // lists (tri_order_kernel)
    int64_t pool;
    size_t head;                             // bytes uploaded at the start of a call
    size_t fixed;                            // bytes before the pool
};

void tri_layout(unsigned char *base, size_t ws_bytes, const TriShape &sh, TriLayout &L) {
    const size_t C = (size_t)sh.count, NR = (size_t)sh.R;
    Carve cv{base};
    L.dc = cv.take<TriComp>(C);
    L.dpre = cv.take<int64_t>(C + 1);
    L.qstart = cv.take<int32_t>((size_t)sh.nq + 1);
    L.tmat = cv.take<int32_t>(C);
    L.cflags = cv.take<unsigned>(C);
    L.ckind = cv.take<int32_t>(C);
    L.cam = cv.take<int>(C);
    L.cfm = cv.take<int>(C);
    L.cprod = cv.take<unsigned long long>(C);
    L.cbad = cv.take<unsigned>(C);
    L.gflags = cv.take<unsigned>(2);
    L.ticket = cv.take<int>(1);
    L.counters = cv.take<DagCounters>(1);
    L.res = cv.take<TriOut>(C);
    L.head = cv.off;
    L.cta_comp = cv.take<int32_t>(sh.fat ? (size_t)sh.ctas : 0);
    L.place = cv.take<int2>(sh.fat ? NR : 0);
    L.row_cnt = cv.take<int32_t>(NR);
    L.row_comp = cv.take<int32_t>(NR);
    L.slot_col = cv.take<int32_t>(NR * TRI_CAP);
    L.slot_val = cv.take<int32_t>(NR * TRI_CAP);
    L.row_off = cv.take<int64_t>(NR);
    L.row_len = cv.take<int32_t>(NR);
    L.state = cv.take<unsigned long long>(NR);
    L.row_prods = cv.take<int32_t>(NR);
    L.order = cv.take<int32_t>(NR);
    L.coff = cv.take<int64_t>(NR);
    L.kid_cnt = cv.take<int32_t>(NR);
    L.children = cv.take<int32_t>(NR * TRI_CAP);
    L.ovf = cv.take<int32_t>(NR + 1);
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

// The host's part of one call over `count` matrices: the tables, the layout and the results.
template <typename T> struct TriCall {
    int64_t count;
    const int64_t *sizes, *in_off, *out_off;
    int64_t ld_in, ld_out;
    const T *in;
    T *out;
    unsigned char *ws;
    size_t ws_bytes;
    cudaStream_t s;
    const RowStats &rs;
    TriShape sh;
    TriLayout L;
    std::vector<unsigned char> head;         // the head of the layout in its starting state
    std::vector<TriOut> res;
    DagCounters hd;

    // rows, CTAs and tickets of the call; false: no matrix is within the path's sizes
    bool shape() {
        sh = TriShape{count, 0, 0, ld_in, ld_out, 0, 0, false};
        for (int pass = 0; pass < 2; ++pass) {
            sh.R = sh.ctas = 0;
            for (int64_t i = 0; i < count; ++i) {
                const int64_t n = rows(i), k = tri_cta_rows(n, sh.fat);
                sh.R += n;
                sh.ctas += (n + k - 1) / k;
                sh.max_n = std::max<int>(sh.max_n, (int)n);
            }
            if (sh.fat || count == 1 || sh.ctas < TRI_FAT_CTAS) break;
            sh.fat = true;
        }
        sh.nq = std::max(sh.max_n, 1);
        return sh.R > 0 && sh.R * TRI_CAP <= INT32_MAX;
    }
    int64_t rows(int64_t i) const { return (sizes[i] > 0 && sizes[i] <= TRI_MAX_N) ? sizes[i] : 0; }
    // carve the workspace; false: no room for a closure (the other paths decide)
    bool layout() {
        tri_layout(nullptr, ws_bytes, sh, L);
        if (L.pool < 4 * sh.R) return false;
        TriLayout H;                         // the same offsets over the host's copy of the head
        head.assign(L.head, 0);
        tri_layout(head.data(), ws_bytes, sh, H);
        tri_layout(ws, ws_bytes, sh, L);
        int64_t row = 0, cta = 0;
        std::vector<int32_t> at((size_t)sh.nq + 2, 0);
        for (int64_t i = 0; i < count; ++i) {
            const int64_t n = rows(i);
            H.dc[i] = TriComp{n, in_off[i], out_off[i], row};
            H.dpre[i] = cta;
            H.cam[i] = H.cfm[i] = -1;
            row += n;
            cta += (n + tri_cta_rows(n, sh.fat) - 1) / tri_cta_rows(n, sh.fat);
            ++at[(size_t)n];
        }
        H.dpre[count] = cta;
        // at[n]: matrices of n rows or more, so row q belongs to at[q + 1] of them; then their places
        for (int n = sh.nq - 1; n >= 0; --n) at[(size_t)n] += at[(size_t)n + 1];
        for (int q = 0; q < sh.nq; ++q) H.qstart[q + 1] = H.qstart[q] + at[(size_t)q + 1];
        for (int64_t i = 0; i < count; ++i) H.tmat[at[(size_t)rows(i) + 1]++] = (int32_t)i;
        return true;
    }
    int upload() {
        HostStaging hs(s, head.size() + (size_t)count * sizeof(TriOut) + sizeof(DagCounters) + 512);
        return hs.up(ws, head.data(), head.size());
    }
    int read() {
        res.resize((size_t)count);
        HostStaging hs(s, (size_t)count * sizeof(TriOut) + sizeof(DagCounters) + 128);
        int rc = hs.down(res.data(), L.res, (size_t)count * sizeof(TriOut));
        if (!rc) rc = hs.down(&hd, L.counters, sizeof(hd));
        if (!rc) rc = hs.finish();
        return rc;
    }
};

// Rows far more than resident warps: several rows per ticket (fewer fences and atomics on one word) while
// the tickets in flight stay a small part of the rows, so that parents are seldom among them.  411 000
// rows: 454 us with one row, 349 with three, 382 with five, 540 with eight; 227 000 rows: 266 us with one,
// 212 with two, 247 with five.  And pool entries for some rows at once (the warps' rests together at most
// a 16th of the pool).
inline TriTickets tri_tickets(int64_t rows, int64_t pool, TriTickets t) {
    const int64_t warps = (int64_t)TRI_PULL_CTAS * sm_count() * TRI_PULL_WARPS, part = TRI_PULL_PART * warps;
    t.places = (int)rows;
    t.batch = (int)std::min<int64_t>(TRI_PULL_BATCH, std::max<int64_t>(1, (rows + part / 2) / part));
    t.block = rows >= 4 * warps ? (int)std::min<int64_t>(TRI_PULL_BLOCK, pool / (16 * warps)) : 0;
    return t;
}
inline unsigned tri_pull_grid(int64_t rows) {
    return (unsigned)std::min<int64_t>((rows + TRI_PULL_WARPS - 1) / TRI_PULL_WARPS, (int64_t)TRI_PULL_CTAS * sm_count());
}

// First pass: scan, closure kernel, write.  Second pass, over the same scratch, for the matrices the
// first one left pending: their order, closure kernel, searches, write.
template <typename T> int tri_pass(TriCall<T> &c, bool second) {
    if (!second) {
        if (!c.layout()) return RBG_OK;
        const int rc = c.upload();
        if (rc) return rc;
    }
    const TriLayout &L = c.L;
    const int count = (int)c.count;
    cudaStream_t s = c.s;
    const bool fat = c.sh.fat;
    note_launches(second ? 3 + TRI_GEN_LAUNCHES : fat ? 4 : 3);
    if (!second) {
        cudaEvent_t t = timer_begin(4, s);
        if (fat)
            tri_map_kernel<<<grid_for(c.sh.R, 256), 256, 0, s>>>(L.dpre, count, c.sh.ctas, L.cta_comp, L.qstart, c.sh.nq,
                                                                L.tmat, L.place, (int)c.sh.R);
        tri_scan_kernel<T><<<(unsigned)c.sh.ctas, TRI_THREADS, 0, s>>>(
            c.in, c.ld_in, L.dc, L.dpre, count, fat, fat ? L.cta_comp : nullptr, L.slot_col, L.slot_val, L.row_cnt,
            L.row_comp, L.cflags, L.state);
        timer_end(4, t, s);
    }
    {
        cudaEvent_t t = timer_begin(5, s);
        if (second)
            // many matrices: small CTAs, several per SM; few: more threads per level
            tri_order_kernel<<<(unsigned)count, fat ? 256 : TRI_ORDER_THREADS, tri_order_smem_bytes(c.sh.max_n), s>>>(
                L.dc, L.ckind, L.slot_col, L.row_cnt, L.order, L.coff, L.kid_cnt, L.children, L.cbad, L.ticket,
                L.gflags + 1, c.sh.max_n);
        const TriSlotRows rows{tri_tickets(c.sh.R, L.pool, TriTickets{fat ? L.place : nullptr, L.qstart, L.tmat, c.sh.nq}),
                               L.dc, L.cflags, L.cbad, L.ckind, second ? L.order : nullptr, L.slot_col, L.slot_val,
                               L.row_cnt};
        tri_pull_kernel<<<tri_pull_grid(c.sh.R), 32 * TRI_PULL_WARPS, 0, s>>>(
            rows, L.state, L.row_off, L.row_len, L.p_col, L.p_val, L.pool, L.counters, L.ticket, L.cam, L.cfm,
            L.row_prods);
        timer_end(5, t, s);
    }
    if (second) {
        cudaEvent_t t = timer_begin(8, s);
        RBG_CUDA_TRY(cudaMemsetAsync(L.ovf, 0, 4, s));
        const TriGraphView G{L.row_cnt, L.slot_col, L.slot_val, L.coff, L.kid_cnt, L.children};
        tri_searches(c.sh, L, G, L.counters, s);
        timer_end(8, t, s);
    }
    {
        cudaEvent_t t = timer_begin(7, s);
        tri_write_kernel<T><<<(unsigned)c.sh.ctas, TRI_THREADS, 0, s>>>(
            c.in, c.ld_in, c.out, c.ld_out, L.dc, L.dpre, count, fat, fat ? L.cta_comp : nullptr, L.ckind, L.cam, L.cbad,
            L.counters, L.gflags, L.row_off, L.row_len, L.p_col, L.p_val, c.rs, L.cfm, L.cprod,
            second ? nullptr : L.row_prods, L.cflags, L.res);
        timer_end(7, t, s);
    }
    RBG_CUDA_TRY(cudaGetLastError());
    return c.read();
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
              size_t ws_bytes, cudaStream_t s, const RowStats &rs) {
    if (count <= 0 || count > INT32_MAX || !ws) return RBG_OK;
    {
        const int rc = tri_configure();     // before any capture: kernel attributes per device
        if (rc) return rc;
    }
    TriCall<T> c{count, sizes, in_off, out_off, ld_in, ld_out, in, out, ws, ws_bytes, s, rs};
    if (!c.shape()) return RBG_OK;
    int rc = tri_pass(c, false);
    if (rc) return rc;
    if (tri_take_results(c, false, results, closed) == 0) return RBG_OK;
    rc = tri_pass(c, true);
    if (!rc) tri_take_results(c, true, results, closed);
    return rc;
}

template int tri_batch<int32_t>(int64_t, const int64_t *, const int64_t *, const int64_t *, int64_t, int64_t,
                                const int32_t *, int32_t *, rbg_result_t *, char *, unsigned char *, size_t,
                                cudaStream_t, const RowStats &);
template int tri_batch<int64_t>(int64_t, const int64_t *, const int64_t *, const int64_t *, int64_t, int64_t,
                                const int64_t *, int64_t *, rbg_result_t *, char *, unsigned char *, size_t,
                                cudaStream_t, const RowStats &);

}  // namespace rbg

// ------------------------------------------------------------------------------------------
// The components of a graph
// ------------------------------------------------------------------------------------------
namespace rbg {
namespace {

struct CcWork {
    int32_t *order, *vertex;                 // vertices by key; all vertices
    unsigned short *key, *key_out;
    unsigned long long *state;
    DagCounters *counters;
    int *ticket;
    unsigned char *tmp;
    size_t tmp_bytes, bytes;
};

void cc_work(unsigned char *base, int64_t n, CcWork &W) {
    static thread_local LastSize size;
    W.tmp_bytes = size.get(n, [&] {
        size_t t = 0;
        cub::DeviceRadixSort::SortPairs(nullptr, t, (unsigned short *)nullptr, (unsigned short *)nullptr,
                                        (int32_t *)nullptr, (int32_t *)nullptr, (int)n, 0, 13);
        return t;
    });
    const size_t N = (size_t)n;
    Carve cv{base};
    W.counters = cv.take<DagCounters>(1);
    W.ticket = cv.take<int>(1);
    W.state = cv.take<unsigned long long>(N);
    W.order = cv.take<int32_t>(N);
    W.vertex = cv.take<int32_t>(N);
    W.key = cv.take<unsigned short>(N);
    W.key_out = cv.take<unsigned short>(N);
    W.tmp = cv.take<unsigned char>(W.tmp_bytes);
    W.bytes = cv.off;
}

// A vertex's key is its place among its component's vertices, from the last where the entries lie above
// the diagonal.  A row of more than TRI_CAP entries, or a component that spans more numbers than a
// bitmap has bits, keeps the call off the path.
__global__ void cc_key_kernel(int64_t n, const int32_t *__restrict__ label, const int32_t *__restrict__ local,
                              const int64_t *__restrict__ start, const int32_t *__restrict__ sorted_vertex,
                              const int32_t *__restrict__ kind, const int64_t *__restrict__ ptr,
                              const int32_t *__restrict__ col, unsigned short *__restrict__ key, int32_t *__restrict__ vertex,
                              unsigned long long *__restrict__ state, DagCounters *dc) {
    bool off = false;
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
        const int c = label[v];
        const int64_t s0 = start[c], s1 = start[c + 1];
        const int k = local[v];
        const int64_t e0 = ptr[v], e1 = ptr[v + 1];
        bool bad = e1 - e0 > TRI_CAP || e1 > INT32_MAX || sorted_vertex[s1 - 1] - sorted_vertex[s0] >= TRI_MAX_N;
        for (int64_t e = e0; e < e1 && !bad; ++e) {
            const int w = col[e];
            bad = w < 0 || w >= n || label[w] != c || (kind[c] == KIND_ABOVE ? w <= v : w >= v);
        }
        off |= bad;
        key[v] = (unsigned short)(kind[c] == KIND_ABOVE ? (int)(s1 - s0) - 1 - k : k);
        vertex[v] = (int32_t)v;
        state[v] = 0;
    }
    if (off) atomicOr(&dc->flags, TRI_BAD_ROW);
}

}  // namespace
}  // namespace rbg

extern "C" int32_t rbg_cc_dag_close_workspace_bytes(int64_t n, int64_t *bytes) {
    if (n < 0 || n > INT32_MAX || !bytes) return RBG_ERR_INVALID;
    rbg::CcWork W;
    rbg::cc_work(nullptr, n, W);
    *bytes = (int64_t)W.bytes + 256;
    return RBG_OK;
}

extern "C" int32_t rbg_cc_dag_close(int64_t n, int64_t ncomp, const int32_t *label, const int32_t *local,
                                    const int64_t *start, const int32_t *sorted_vertex, const int32_t *comp_kind,
                                    const rbg_csr_t *edges, const int32_t *diag, void *workspace,
                                    int64_t workspace_bytes, int32_t *pool_cols, int32_t *pool_vals,
                                    int64_t pool_capacity, int64_t *row_off, int32_t *row_len, int32_t *top_msb,
                                    int32_t *first_msb, int32_t *comp_max, int32_t *closed, rbg_stream_t stream) {
    using namespace rbg;
    if (n < 0 || n > INT32_MAX || ncomp < 0 || ncomp > n || !edges || !closed) return RBG_ERR_INVALID;
    *closed = 1;
    if (n == 0) return RBG_OK;
    if (!label || !local || !start || !sorted_vertex || !comp_kind || !diag || !workspace || !row_off || !row_len ||
        !top_msb || !first_msb || !comp_max || !edges->indptr ||
        !edges->indices || !edges->data || !pool_cols || !pool_vals || edges->n_rows != n)
        return RBG_ERR_INVALID;
    CcWork W;
    cc_work(reinterpret_cast<unsigned char *>(workspace), n, W);
    if (workspace_bytes < (int64_t)W.bytes) return RBG_ERR_NOMEM;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    *closed = 0;
    if (n > (int64_t)1 << 27) return RBG_OK;
    RBG_CUDA_TRY(cudaMemsetAsync(W.counters, 0, (size_t)((unsigned char *)W.state - (unsigned char *)W.counters), s));
    RBG_CUDA_TRY(cudaMemsetAsync(top_msb, 0xff, (size_t)ncomp * 4, s));
    RBG_CUDA_TRY(cudaMemsetAsync(first_msb, 0xff, (size_t)ncomp * 4, s));
    RBG_CUDA_TRY(cudaMemsetAsync(comp_max, 0, (size_t)ncomp * 4, s));
    note_launches(2);
    cc_key_kernel<<<grid_for(n, 256), 256, 0, s>>>(n, label, local, start, sorted_vertex, comp_kind, edges->indptr,
                                                  edges->indices, W.key, W.vertex, W.state, W.counters);
    RBG_CUDA_TRY(cub::DeviceRadixSort::SortPairs(W.tmp, W.tmp_bytes, W.key, W.key_out, W.vertex, W.order, (int)n, 0, 13, s));
    const TriCsrRows rows{tri_tickets(n, pool_capacity, TriTickets{}), W.order, label, comp_kind, sorted_vertex, start,
                          edges->indptr, edges->indices, static_cast<const int32_t *>(edges->data), diag, comp_max};
    tri_pull_kernel<<<tri_pull_grid(n), 32 * TRI_PULL_WARPS, 0, s>>>(rows, W.state, row_off, row_len, pool_cols, pool_vals,
                                                                    pool_capacity, W.counters, W.ticket, top_msb,
                                                                    first_msb, nullptr);
    RBG_CUDA_TRY(cudaGetLastError());
    DagCounters hd;
    HostStaging hs(s, sizeof(hd) + 128);
    int rc = hs.down(&hd, W.counters, sizeof(hd));
    if (!rc) rc = hs.finish();
    if (rc) return rc;
    *closed = hd.flags == 0;
    return RBG_OK;
}

extern "C" int32_t rbg_cc_dag_close_reserved(const void *workspace, int64_t *entries, rbg_stream_t stream) {
    using namespace rbg;
    if (!workspace || !entries) return RBG_ERR_INVALID;
    DagCounters hd;                              // (the workspace starts with them)
    HostStaging hs(reinterpret_cast<cudaStream_t>(stream), sizeof(hd) + 128);
    int rc = hs.down(&hd, workspace, sizeof(hd));
    if (!rc) rc = hs.finish();
    if (rc) return rc;
    *entries = hd.flags == 1 ? (int64_t)hd.reserved : 0;
    return RBG_OK;
}

// The DAG path keeps nothing between calls.
extern "C" int32_t rbg_release_scratch(void) { return RBG_OK; }
