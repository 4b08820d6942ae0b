// avos_gemm.cu -- dense AVOS matrix product C = A (x) B for rb.array @ (sm_103a).
//
// Reference: the AVOS einsum 'ij,jk' (redblackgraph/core/src/redblackgraph/redblack.c.src:554-594,
// reached from redblackgraph/core/redblack.py:14-38):  C[i,k] = (+)_j A[i,j] (x) B[j,k] with the
// C core scalar semantics (rbg_math.c.in:30-121).  (+) is associative and commutative, so the
// accumulation order does not change C; an OverflowError is raised when any product signals one.
//
// One kernel, 128 x 128 outputs per CTA, the reduction staged through shared memory in chunks of
// 32 steps.  Operands in the clean regime run on 32-bit lanes (avos.cuh): a product is one
// multiply-add x * 2^msb(y) + (y - 2^msb(y)), a sum one unsigned min.  Two things are kept out of
// the inner loop:
//   - steps of a chunk whose column of A or row of B (within the tile) is all zero are skipped,
//     as are the steps at which a warp's rows of A are zero (closures are sparse);
//   - the identities.  A -1 on the left is staged as a lane value that yields the right operand;
//     1 and -1 on the right (parity filters) are staged as zeros and folded in by a pass of their
//     own over the chunk's steps that hold one.
// With dense operands the issue slots bound it (64 multiply-adds and mins per 5 vector loads from
// shared memory); with a closure times its pedigree most steps are skipped and a chunk's staging
// latency does: one CTA of 512 threads per SM (the accumulators and the next chunk's values, in
// flight during a chunk's products, take its registers), one barrier per chunk.  n = 2048, W (x) A
// of a pedigree: 7.32 ms with the full scalar semantics per product (64 x 64 tiles), 0.36 ms now.
// A tile in which some product may reach the storage type's top bit, or which holds a negative
// value other than -1, is redone by the same CTA with the full scalar semantics (wrap, overflow
// events).
#include <cuda_runtime.h>
#include <cooperative_groups.h>
#include <string.h>
#include <algorithm>
#include "rbg_internal.cuh"

namespace rbg {

namespace cg = cooperative_groups;

constexpr int MM_T = 128;        // output tile edge
constexpr int MM_K = 32;         // reduction steps per chunk (one per lane of a warp)
constexpr int MM_THREADS = 512;  // 32 x 16 threads, 4 x 8 outputs each
constexpr int MM_SPLIT = 8;      // CTAs of a cluster that share one tile's reduction, at most
constexpr uint32_t MM_NONE = 0xffffffffu;      // lane: zero operand / no product yet
constexpr uint32_t MM_RED_LEFT = 0x80000001u;  // lane: -1 as the left operand (times 2^s, s >= 1, is 2^s)

struct MmSmem {
    uint32_t as[2][MM_K][MM_T];   // A's chunk, transposed; 4-row groups swizzled by the step (mm_as)
    uint32_t bm[2][MM_K][MM_T];   // 2^msb of B's values (0: zero or an identity)
    uint32_t bl[2][MM_K][MM_T];   // value - 2^msb (MM_NONE with bm 0)
    uint32_t ident[2][2][MM_K][4];// columns 4 l + c whose value is 1 / -1: bit l of word c
    uint32_t or_b[2][MM_K];       // OR of the step's values in B (identities as 1)
    // written by atomics, so three slots in turn: one read, one being written, one cleared
    uint32_t or_a[3][MM_K];       // OR of the step's values in A
    uint32_t id_any[3];           // steps that hold an identity in B
};

// position of row i of step j in MmSmem::as: the transposing stores of a warp (8 steps apart by
// 4, 4 rows) hit 32 banks, and four consecutive rows stay one 16-byte vector
__device__ __forceinline__ int mm_as(int j, int i) { return ((((i >> 2) ^ ((j >> 2) & 7)) << 2) | (i & 3)); }

__device__ __forceinline__ void mm_flush_flags(unsigned *dflags, unsigned f) {
    for (int o = 16; o > 0; o >>= 1) f |= __shfl_xor_sync(0xffffffffu, f, o);
    if ((threadIdx.x & 31) == 0 && f) atomicOr(dflags, f);
}

// column of a thread's output c within the tile
__device__ __forceinline__ int mm_col(int tx, int c) { return (c < 4 ? 0 : 60) + 4 * tx + c; }

// the sum as a minimum: the red one first, "no path" last
template <typename U> __device__ __forceinline__ U mm_enc(U v) { return v == 0 ? (U)~(U)0 : v == (U)~(U)0 ? (U)0 : v; }

// Four consecutive values of a row from column c (`cols` valid columns); `vec`: the row starts
// and the leading dimension are aligned for vector loads.
template <typename T> struct alignas(sizeof(T) * 4 > 16 ? 16 : sizeof(T) * 4) MmVec { T v[4]; };
template <typename T>
__device__ __forceinline__ void mm_load4(const T *__restrict__ row, bool live, int64_t c, int64_t cols, bool vec,
                                         T (&x)[4]) {
    if (live && vec && c + 4 <= cols) {
        const MmVec<T> t = *reinterpret_cast<const MmVec<T> *>(row + c);
#pragma unroll
        for (int k = 0; k < 4; ++k) x[k] = t.v[k];
    } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) x[k] = (live && c + k < cols) ? row[c + k] : (T)0;
    }
}

// Full scalar semantics for one tile, steps [j0, j1): its outputs into `tile`, in the encoding of
// mm_enc.  Every thread of the CTA calls it.  The quarters of the tile come one after another (a quarter
// beyond the matrix not at all), 2 x 4 outputs per thread, so that small products spread over the CTA.
// Only steps with a negative value in the quarter take every case; the others ask for zeros and
// identities, and for the top bit where a thread's operands may reach it.  Bound by issue, 64-bit shifts and mins.  int64 operands
// with a third of their entries up to 2^40, 64 x 64 x 64: 328 us with every case on 32 outputs per thread,
// 115 so (193 us one 64 x 64 tile per CTA); 1500 x 1500 x 1500: 12.3, 6.3 (9.9) ms.
constexpr int MM_Q = MM_T / 2;               // quarter edge
template <typename T> struct MmExact {
    T as[MM_Q][MM_K + 1];
    T bs[MM_K][MM_Q + 4];
    unsigned negative;                       // steps of the chunk with a negative value other than -1
};
template <typename T>
__device__ __noinline__ void mm_exact_tile(int64_t m, int64_t p, int64_t i0, int64_t k0, int64_t j0, int64_t j1,
                                           const T *__restrict__ A, int64_t lda, const T *__restrict__ B, int64_t ldb,
                                           typename utype<T>::type *tile, MmExact<T> &S, unsigned *dflags) {
    typedef typename utype<T>::type U;
    constexpr int BITS = (int)sizeof(U) * 8;
    constexpr U NONE = (U)~(U)0, RED = (U)~(U)0;   // mm_enc of no path; the red one itself
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    unsigned ev = 0;
    __syncthreads();                         // the last chunk's reads of the staging buffers
    for (int q = 0; q < 4; ++q) {
        const int64_t iq = i0 + MM_Q * (q >> 1), kq = k0 + MM_Q * (q & 1);
        if (iq >= m || kq >= p) continue;    // block-uniform
        U acc[2][4];
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[r][c] = NONE;
        const bool mine = iq + 2 * ty < m && kq + 4 * tx < p;
        for (int64_t j = j0; j < j1; j += MM_K) {
            __syncthreads();
            if (tid == 0) S.negative = 0;
            __syncthreads();
            unsigned neg = 0;
            auto negative_value = [](T v) { return utype<T>::is_signed && v < 0 && v != (T)-1; };
            for (int e = tid; e < MM_Q * MM_K; e += MM_THREADS) {
                const int r = e / MM_K, c = e % MM_K, rr = e / MM_Q, cc = e % MM_Q;
                const T a = (iq + r < m && j + c < j1) ? A[(iq + r) * lda + j + c] : (T)0;
                const T b = (j + rr < j1 && kq + cc < p) ? B[(j + rr) * ldb + kq + cc] : (T)0;
                S.as[r][c] = a;
                S.bs[rr][cc] = b;
                neg |= (negative_value(a) ? 1u << c : 0u) | (negative_value(b) ? 1u << rr : 0u);
            }
            neg = __reduce_or_sync(0xffffffffu, neg);
            if ((tid & 31) == 0 && neg) atomicOr(&S.negative, neg);
            __syncthreads();
            const int steps = j1 - j < MM_K ? (int)(j1 - j) : MM_K;
            const unsigned negative = S.negative;
            for (int t = 0; mine && t < steps; ++t) {
                const U x[2] = {(U)S.as[2 * ty][t], (U)S.as[2 * ty + 1][t]};
                if (x[0] == 0 && x[1] == 0) continue;
                U y[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) y[c] = (U)S.bs[t][4 * tx + c];
                if ((negative >> t) & 1u) {          // block-uniform
#pragma unroll
                    for (int r = 0; r < 2; ++r)
#pragma unroll
                        for (int c = 0; c < 4; ++c)
                            acc[r][c] = min(acc[r][c], mm_enc<U>(avos_product<T>((T)x[r], (T)y[c], ev)));
                    continue;
                }
                U z[2], yo = 0;                      // the left operands, the red one as 1; plain right ones ORed
#pragma unroll
                for (int r = 0; r < 2; ++r) z[r] = x[r] == RED ? (U)1 : x[r];
#pragma unroll
                for (int c = 0; c < 4; ++c) yo |= (U)(y[c] + 1) <= 2 ? (U)0 : y[c];
                const int mx[2] = {msb_nz<U>((U)(z[0] | 1)), msb_nz<U>((U)(z[1] | 1))};
                // may a product of the thread's reach the top bit?
                const bool top = max(mx[0], mx[1]) + msb_nz<U>((U)(yo | 1)) >= BITS - 1;
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    if ((U)(y[c] + 1) <= 2) {        // 0 or an identity: 1 keeps an odd left value, -1 an even one
                        if (y[c] == 0) continue;
#pragma unroll
                        for (int r = 0; r < 2; ++r)
                            if (x[r] == RED ? y[c] == RED : x[r] != 0 && (x[r] & 1) == (U)(y[c] == 1))
                                acc[r][c] = min(acc[r][c], mm_enc<U>(x[r]));
                        continue;
                    }
                    const int s = msb_nz<U>(y[c]);
                    const U low = (U)(y[c] ^ ((U)1 << s));
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        if (z[r] == 0) continue;
                        const U v = (U)((U)(z[r] << s) | low);
                        if (top) {
                            if (mx[r] + s >= BITS) ev |= RBG_EV_OVF_SIZE;
                            if (v == RED) ev |= RBG_EV_OVF_ONES;
                        }
                        acc[r][c] = min(acc[r][c], top ? mm_enc<U>(v) : v);
                    }
                }
            }
        }
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int c = 0; c < 4; ++c)
                tile[(MM_Q * (q >> 1) + 2 * ty + r) * MM_T + MM_Q * (q & 1) + 4 * tx + c] = acc[r][c];
    }
    mm_flush_flags(dflags, ev);
}

// Shared memory of a CTA: the lanes' staging buffers, over them the tile when it is shared by a cluster
// or redone; the exact tile's staging buffers behind the tile.
template <typename T> constexpr size_t mm_smem_bytes() {
    return std::max(sizeof(MmSmem), sizeof(T) * MM_T * MM_T + sizeof(MmExact<T>));
}

// One 128 x 128 tile of C per cluster of `split` CTAs (1, 2, 4 or 8), each taking an equal part of
// the reduction's chunks; the parts meet through distributed shared memory.
template <typename T>
__global__ void __launch_bounds__(MM_THREADS, 1)
mm_kernel(int64_t m, int64_t q, int64_t p, const T *__restrict__ A, int64_t lda, const T *__restrict__ B, int64_t ldb,
          T *__restrict__ C, int64_t ldc, int split, bool vec_a, bool vec_b, bool vec_c, unsigned *dflags) {
    typedef typename utype<T>::type U;
    constexpr int LBITS = sizeof(T) >= 4 ? 32 : (int)sizeof(T) * 8;   // a clean product's MSB stays below LBITS - 1
    extern __shared__ __align__(16) unsigned char mm_smem[];
    MmSmem &S = *reinterpret_cast<MmSmem *>(mm_smem);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tx = tid & 15, ty = tid >> 4;
    const int part = (int)(blockIdx.x % split);
    const int64_t k0 = (int64_t)(blockIdx.x / split) * MM_T, i0 = (int64_t)blockIdx.y * MM_T;
    const int64_t chunks = (q + MM_K - 1) / MM_K;
    const int64_t c0 = chunks * part / split, c1 = chunks * (part + 1) / split;

    uint32_t acc[4][8];
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 8; ++c) acc[r][c] = MM_NONE;
    if (tid < 3 * MM_K) (&S.or_a[0][0])[tid] = 0;
    if (tid < 3) S.id_any[tid] = 0;

    // a thread's part of a chunk: 4 steps of rows ar and ar + 64 of A, 4 columns of steps warp and
    // warp + 16 of B
    const int ar = tid >> 3, aj = (tid & 7) * 4;
    T xa[2][4], xb[2][4];
    auto fetch = [&](int64_t ch) {
        const int64_t j = ch * MM_K;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int64_t i = i0 + ar + 64 * h;
            mm_load4<T>(A + i * lda, i < m, j + aj, q, vec_a, xa[h]);
            const int64_t jb = j + warp + 16 * h;
            mm_load4<T>(B + jb * ldb, jb < q, k0 + 4 * lane, p, vec_b, xb[h]);
        }
    };
    if (c0 < c1) fetch(c0);
    bool dirty = false;
    int s3 = 0;                              // or_a's slot: chunk number modulo 3
    __syncthreads();
    for (int64_t ch = c0; ch < c1; ++ch) {
        const int buf = (int)((ch - c0) & 1);
        bool bad = false;                    // a value the lanes cannot hold
        uint32_t oa[4] = {0, 0, 0, 0};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const T v = xa[h][k];
                const bool red = v == (T)-1;
                bad |= !red && ((U)v >> (LBITS - 1)) != 0;
                oa[k] |= red ? 1u : (uint32_t)(U)v;
                S.as[buf][aj + k][mm_as(aj + k, ar + 64 * h)] =
                    red ? MM_RED_LEFT : v == 0 ? MM_NONE : (uint32_t)(U)v;
            }
            const int jb = warp + 16 * h;
            uint32_t ob = 0, mv[4], lv[4];
            bool some_id = false;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const T v = xb[h][k];
                const bool id = v == (T)-1 || v == (T)1;
                some_id |= id;
                bad |= !id && ((U)v >> (LBITS - 1)) != 0;
                ob |= id ? 1u : (uint32_t)(U)v;
                const bool plain = !id && v != 0;
                mv[k] = plain ? 0x80000000u >> __clz((int)(uint32_t)(U)v) : 0u;
                lv[k] = plain ? (uint32_t)(U)v ^ mv[k] : MM_NONE;
            }
            *reinterpret_cast<uint4 *>(&S.bm[buf][jb][4 * lane]) = make_uint4(mv[0], mv[1], mv[2], mv[3]);
            *reinterpret_cast<uint4 *>(&S.bl[buf][jb][4 * lane]) = make_uint4(lv[0], lv[1], lv[2], lv[3]);
            ob = __reduce_or_sync(0xffffffffu, ob);
            if (lane == 0) S.or_b[buf][jb] = ob;
            if (__any_sync(0xffffffffu, some_id)) {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const unsigned one = __ballot_sync(0xffffffffu, xb[h][k] == (T)1);
                    const unsigned red = __ballot_sync(0xffffffffu, xb[h][k] == (T)-1);
                    if (lane == 0) {
                        S.ident[buf][0][jb][k] = one;
                        S.ident[buf][1][jb][k] = red;
                    }
                }
                if (lane == 0) atomicOr(&S.id_any[s3], 1u << jb);
            }
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {        // lanes l, l + 8, l + 16, l + 24 hold the same steps
            oa[k] |= __shfl_xor_sync(0xffffffffu, oa[k], 8);
            oa[k] |= __shfl_xor_sync(0xffffffffu, oa[k], 16);
            if (lane < 8 && oa[k]) atomicOr(&S.or_a[s3][aj + k], oa[k]);
        }
        if (__syncthreads_or(bad)) { dirty = true; break; }
        if (ch + 1 < c1) fetch(ch + 1);      // in flight during this chunk's products
        const uint32_t va = S.or_a[s3][lane], vb = S.or_b[buf][lane];
        const uint32_t idm = S.id_any[s3];
        // the previous chunk's slots: read before this chunk's barrier, written after the next one
        if (warp == 0) {
            const int old = s3 == 0 ? 2 : s3 - 1;
            S.or_a[old][lane] = 0;
            if (lane == 0) S.id_any[old] = 0;
        }
        const bool live = va != 0 && vb != 0;
        uint32_t act = __ballot_sync(0xffffffffu, live);
        const bool risk = live && (31 - __clz((int)va)) + (31 - __clz((int)vb)) >= LBITS - 1;
        if (__any_sync(0xffffffffu, risk)) { dirty = true; break; }   // the same vote in every warp
        uint32_t ids = idm & act;
        while (act) {
            const int j = __ffs((int)act) - 1;
            act &= act - 1;
            const uint4 x4 = *reinterpret_cast<const uint4 *>(&S.as[buf][j][mm_as(j, 4 * ty)]);
            const uint32_t x[4] = {x4.x, x4.y, x4.z, x4.w};
            if (!__any_sync(0xffffffffu, (x[0] & x[1] & x[2] & x[3]) != MM_NONE)) continue;
            const uint4 m0 = *reinterpret_cast<const uint4 *>(&S.bm[buf][j][4 * tx]);
            const uint4 m1 = *reinterpret_cast<const uint4 *>(&S.bm[buf][j][64 + 4 * tx]);
            const uint4 l0 = *reinterpret_cast<const uint4 *>(&S.bl[buf][j][4 * tx]);
            const uint4 l1 = *reinterpret_cast<const uint4 *>(&S.bl[buf][j][64 + 4 * tx]);
            const uint32_t mm[8] = {m0.x, m0.y, m0.z, m0.w, m1.x, m1.y, m1.z, m1.w};
            const uint32_t ll[8] = {l0.x, l0.y, l0.z, l0.w, l1.x, l1.y, l1.z, l1.w};
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int c = 0; c < 8; ++c) acc[r][c] = min(acc[r][c], x[r] * mm[c] + ll[c]);
        }
        // identities on the right: 1 keeps an odd left value (and 1), -1 an even one; -1 (x) -1 is
        // the red one (0 in the encoding, which absorbs)
        while (ids) {
            const int j = __ffs((int)ids) - 1;
            ids &= ids - 1;
            const uint4 x4 = *reinterpret_cast<const uint4 *>(&S.as[buf][j][mm_as(j, 4 * ty)]);
            const uint32_t x[4] = {x4.x, x4.y, x4.z, x4.w};
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const int bit = c < 4 ? tx : 16 + tx;
                const bool one = (S.ident[buf][0][j][c & 3] >> bit) & 1u, red = (S.ident[buf][1][j][c & 3] >> bit) & 1u;
                if (!(one || red)) continue;
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    uint32_t v = MM_NONE;
                    if (x[r] == MM_RED_LEFT) v = red ? 0u : MM_NONE;
                    else if (x[r] != MM_NONE && (x[r] & 1u) == (one ? 1u : 0u)) v = x[r];
                    acc[r][c] = min(acc[r][c], v);
                }
            }
        }
        s3 = s3 == 2 ? 0 : s3 + 1;
    }
    // outputs: straight from the registers, or through the tile in shared memory when it was redone
    // or is shared by a cluster
    U *tile = reinterpret_cast<U *>(mm_smem);
    auto dec = [](U e) -> T { return (T)mm_enc<U>(e); };   // the encoding is its own inverse
    auto lane_enc = [](uint32_t v) -> U { return (v >> 31) ? (U)~(U)0 : (U)v; };
    if (dirty) {
        mm_exact_tile<T>(m, p, i0, k0, c0 * MM_K, c1 * MM_K < q ? c1 * MM_K : q, A, lda, B, ldb, tile,
                         *reinterpret_cast<MmExact<T> *>(mm_smem + sizeof(T) * MM_T * MM_T), dflags);
    } else if (split > 1) {
        __syncthreads();                     // the last chunk's reads of the staging buffers
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int c = 0; c < 8; ++c) tile[(4 * ty + r) * MM_T + mm_col(tx, c)] = lane_enc(acc[r][c]);
    } else {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int64_t gi = i0 + 4 * ty + r;
            if (gi >= m) break;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int64_t gk = k0 + 64 * h + 4 * tx;
                MmVec<T> o;
#pragma unroll
                for (int c = 0; c < 4; ++c) o.v[c] = dec(lane_enc(acc[r][4 * h + c]));
                if (vec_c && gk + 4 <= p) {
                    *reinterpret_cast<MmVec<T> *>(C + gi * ldc + gk) = o;
                } else {
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        if (gk + c < p) C[gi * ldc + gk + c] = o.v[c];
                }
            }
        }
        return;
    }
    if (split > 1) cg::this_cluster().sync();
    else __syncthreads();
    const int rows = MM_T / split;
    for (int e = tid; e < rows * MM_T; e += MM_THREADS) {
        const int at = part * rows * MM_T + e;
        U v = (U)~(U)0;
        if (split > 1) {
            for (int s = 0; s < split; ++s) v = min(v, cg::this_cluster().map_shared_rank(tile, s)[at]);
        } else {
            v = tile[at];
        }
        const int64_t gi = i0 + at / MM_T, gk = k0 + at % MM_T;
        if (gi < m && gk < p) C[gi * ldc + gk] = dec(v);
    }
    if (split > 1) cg::this_cluster().sync();   // no CTA leaves while its tile is read
}

template <typename T>
static int matmul_t(int64_t m, int64_t q, int64_t p, const T *A, int64_t lda, const T *B,
                    int64_t ldb, T *C, int64_t ldc, unsigned *dflags, cudaStream_t s) {
    if (m == 0 || p == 0) return RBG_OK;
    if (q == 0) {
        RBG_CUDA_TRY(cudaMemset2DAsync(C, ldc * sizeof(T), 0, p * sizeof(T), m, s));
        return RBG_OK;
    }
    constexpr size_t smem = mm_smem_bytes<T>();
    static PerDeviceOnce once;               // per storage type, for every device
    const int configured = once.run([] {
        RBG_CUDA_TRY(cudaFuncSetAttribute(mm_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        return (int)RBG_OK;
    });
    if (configured) return configured;
    const int64_t tx = (p + MM_T - 1) / MM_T, ty = (m + MM_T - 1) / MM_T, chunks = (q + MM_K - 1) / MM_K;
    // too few tiles for the SMs: clusters share a tile's reduction, down to two chunks per CTA
    // (135 x 655 x 17: 564 us with one CTA per 64 x 64 tile, 68 us; 300 x 310 x 290: 307 us, 94 us)
    int split = 1;
    while (split < MM_SPLIT && tx * ty * split * 2 <= sm_count() && chunks >= 4 * split) split *= 2;
    auto vec = [](const void *ptr, int64_t ld) {
        return (uintptr_t)ptr % alignof(MmVec<T>) == 0 && (ld * (int64_t)sizeof(T)) % (int64_t)alignof(MmVec<T>) == 0;
    };
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(tx * split), (unsigned)ty);
    cfg.blockDim = dim3(MM_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)split;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    note_launches(1);
    RBG_CUDA_TRY(cudaLaunchKernelEx(&cfg, mm_kernel<T>, m, q, p, A, lda, B, ldb, C, ldc, split, vec(A, lda),
                                    vec(B, ldb), vec(C, ldc), dflags));
    return RBG_OK;
}

}  // namespace rbg

using namespace rbg;

extern "C" int32_t rbg_avos_matmul_workspace_bytes(int32_t dtype, int64_t m, int64_t q, int64_t p,
                                                   int64_t *bytes) {
    if (!bytes || dtype_bytes(dtype) == 0 || m < 0 || q < 0 || p < 0) return RBG_ERR_INVALID;
    *bytes = 256;
    return RBG_OK;
}

extern "C" int32_t rbg_avos_matmul(int32_t dtype, int64_t m, int64_t q, int64_t p, const void *A,
                                   int64_t lda, const void *B, int64_t ldb, void *C, int64_t ldc,
                                   void *workspace, int64_t workspace_bytes, uint32_t *flags,
                                   rbg_stream_t stream) {
    if (m < 0 || q < 0 || p < 0 || !flags || lda < q || ldb < p || ldc < p) return RBG_ERR_INVALID;
    if (dtype_bytes(dtype) == 0) return RBG_ERR_INVALID;
    if (workspace_bytes < 256 || !workspace) return RBG_ERR_NOMEM;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    unsigned *dflags = reinterpret_cast<unsigned *>(workspace);
    RBG_CUDA_TRY(cudaMemsetAsync(dflags, 0, sizeof(unsigned), s));
    int rc = RBG_ERR_INVALID;
    RBG_DISPATCH_DTYPE(dtype, T,
        rc = matmul_t<T>(m, q, p, reinterpret_cast<const T *>(A), lda,
                         reinterpret_cast<const T *>(B), ldb, reinterpret_cast<T *>(C), ldc, dflags, s));
    if (rc) return rc;
    unsigned hf = 0;
    RBG_CUDA_TRY(cudaMemcpyAsync(&hf, dflags, sizeof(unsigned), cudaMemcpyDeviceToHost, s));
    RBG_CUDA_TRY(cudaStreamSynchronize(s));
    *flags = hf;
    return (hf & (RBG_EV_OVF_SIZE | RBG_EV_OVF_ONES | RBG_EV_HANG)) ? RBG_ERR_OVERFLOW : RBG_OK;
}
