// fw_sided.cuh -- closure of one dense matrix numbered in a topological order, block row by block row.
// Included by fw_dense.cu (which defines FW_B, lane<>, flush_status, DevStatus) and for matrices the
// DAG path leaves because of rows of more than its slots (fw_tri.cu): clean values, every entry on
// one side of the diagonal.
//
// The sequential loop ends with the DAG recurrence there (fw_tri.cu), so nothing needs the snapshots
// and the 64-step rounds of the general blocked kernels.  With blocks of SD_B rows, block row I is
//     T(I, J) = A(I, J) (+) sum over the blocks K between I and J of A(I, K) (x) C(K, J)
//     C(I, J) = T(I, J) (+) D(I) (x) T(I, J)
// with D(I) the closure of the diagonal block (paths inside the block; products of paths are
// associative).  The D(I) are closed all at once; then step K (downwards below the diagonal, upwards
// above it) is one launch that adds A(I, K) (x) C(K, J) to every tile it reaches, a CTA per tile; the
// tiles of the next block row, complete with that, are multiplied by D in the same CTA.
//
// The loop's diameter is the largest first value of a cell (an entry of A, else the product of the
// first step that reaches the cell): below the diagonal A(i, k) (x) C(k, j) with the smallest k,
// above it C(i, k) (x) A(k, j) with the smallest k.  Row and column bit masks give that k per cell
// at the end.  A step whose largest operands reach the top bit together marks the matrix
// RBG_EV_RISK, and it goes to the general kernels.
//
// Bound by the chain of steps (a launch and two products of depth SD_B each) and, from a few
// thousand rows, by the multiply-adds and mins.  A layered DAG of n = 2048 with half of the links:
// 2.22 ms in the general kernels' 32 rounds of five launches, 0.67 ms here; n = 4096: 6.45 ms, 2.37
// ms.  (Block row by block row with the long reduction split over clusters took 1.10 ms and 4.66 ms:
// the tiles of a block row differ in depth by up to its length.)
#pragma once

constexpr int SD_B = 128;                    // block rows and columns
constexpr int SD_K = 32;                     // reduction steps per chunk
constexpr int SD_THREADS = 512;
constexpr uint32_t SD_NONE = 0xffffffffu;
constexpr int SD_TOP = 31;

template <int BN> struct SdSmem {
    uint32_t as[2][SD_K][SD_B];              // the left operand's chunk, transposed, 4-row groups swizzled (sd_as)
    uint32_t bm[2][SD_K][BN], bl[2][SD_K][BN];
    uint32_t tm[SD_B][BN], tl[SD_B][BN];     // the completed tile T, split, as the right operand of D (x) T
    uint32_t or_b[2][SD_K];                  // OR of the step's values
    uint32_t or_t[SD_B];
    uint32_t or_a[3][SD_K];                  // three slots in turn: read, written, cleared
};

__device__ __forceinline__ int sd_as(int j, int i) { return ((((i >> 2) ^ ((j >> 2) & 7)) << 2) | (i & 3)); }
__device__ __forceinline__ bool sd_valid(uint32_t v) { return (v >> 31) == 0; }
__device__ __forceinline__ void sd_split(uint32_t y, uint32_t &m, uint32_t &low) {
    const bool v = sd_valid(y);
    m = v ? 0x80000000u >> __clz((int)y) : 0u;
    low = v ? y ^ m : SD_NONE;
}
// an entry of A as a lane (0 and the diagonal: none)
template <typename T> __device__ __forceinline__ uint32_t sd_lane(T v, bool off_diagonal) {
    return off_diagonal && v != 0 ? (uint32_t)v : SD_NONE;
}

// D(I): the diagonal blocks of the lane matrix closed in place, one CTA per block.  Its two 64 x 64
// halves on the diagonal are closed first, 256 threads each (4 x 4 cells per thread in registers; step
// t's row and column are published before one barrier, the column with its zeros as all ones, whose
// products keep the top bit: a zero multiplied along a chain of steps would lose it); then the remaining
// quarter X is multiplied by the halves on both sides, X <- X (+) X (x) P, then X <- X (+) Q (x) X.
__global__ void __launch_bounds__(SD_THREADS)
sd_diag_kernel(uint32_t *__restrict__ work, int64_t np, int above, DevStatus *st) {
    constexpr int H = SD_B / 2;
    __shared__ __align__(16) uint32_t s_col[2][2][H], s_m[2][2][H], s_l[2][2][H];
    __shared__ __align__(16) uint32_t s_x[H][H + 4], s_bm[H][H], s_bl[H][H];
    __shared__ int s_cmax[2][H], s_rmax[2][H];
    const int tid = threadIdx.x, half = tid >> 8, tx = tid & 15, ty = (tid & 255) >> 4;
    uint32_t *blk = work + (int64_t)blockIdx.x * SD_B * (np + 1);
    uint32_t *own = blk + (int64_t)half * H * (np + 1);
    if (tid < 2 * H) (&s_cmax[0][0])[tid] = (&s_rmax[0][0])[tid] = -1000;
    uint32_t R[4][4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const uint4 v = *reinterpret_cast<const uint4 *>(own + (int64_t)(4 * ty + r) * np + 4 * tx);
        R[r][0] = v.x; R[r][1] = v.y; R[r][2] = v.z; R[r][3] = v.w;
    }
    __syncthreads();
    for (int t0 = 0; t0 < H; t0 += 4) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int t = t0 + u, b = u & 1;
            if (ty == t0 >> 2) {             // row t: register row u of these threads
                int top = -1;
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    uint32_t m, l;
                    sd_split(R[u][c], m, l);
                    s_m[half][b][4 * tx + c] = m;
                    s_l[half][b][4 * tx + c] = l;
                    if (m) top = max(top, 31 - __clz((int)m));
                }
                if (top >= 0) atomicMax(&s_rmax[half][t], top);
            }
            if (tx == t0 >> 2) {             // column t: register column u
                int top = -1;
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const bool on = sd_valid(R[r][u]);
                    s_col[half][b][4 * ty + r] = on ? R[r][u] : SD_NONE;
                    if (on) top = max(top, 31 - __clz((int)R[r][u]));
                }
                if (top >= 0) atomicMax(&s_cmax[half][t], top);
            }
            __syncthreads();
            const uint4 x4 = *reinterpret_cast<const uint4 *>(&s_col[half][b][4 * ty]);
            const uint32_t x[4] = {x4.x, x4.y, x4.z, x4.w};
            if (!__any_sync(0xffffffffu, sd_valid(x[0]) || sd_valid(x[1]) || sd_valid(x[2]) || sd_valid(x[3]))) continue;
            const uint4 m4 = *reinterpret_cast<const uint4 *>(&s_m[half][b][4 * tx]);
            const uint4 l4 = *reinterpret_cast<const uint4 *>(&s_l[half][b][4 * tx]);
            const uint32_t m[4] = {m4.x, m4.y, m4.z, m4.w}, l[4] = {l4.x, l4.y, l4.z, l4.w};
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int c = 0; c < 4; ++c) R[r][c] = min(R[r][c], x[r] * m[c] + l[c]);
        }
    }
    unsigned flags = 0;
    __syncthreads();
    if (tid < 2 * H && (&s_cmax[0][0])[tid] + (&s_rmax[0][0])[tid] >= SD_TOP) flags |= RBG_EV_RISK;
    // the quarter off the diagonal: rows of half `bot`, columns of the other one; P is the closed half
    // of its columns, Q that of its rows
    const int bot = above ? 0 : 1;
    uint32_t *quarter = blk + (int64_t)bot * H * np + (1 - bot) * H;
    auto clean = [&]() {
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int c = 0; c < 4; ++c)
                if (!sd_valid(R[r][c])) R[r][c] = SD_NONE;
    };
    clean();
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        if (ty == tx && R[r][r] != SD_NONE) flags |= RBG_EV_CYCLE;
        *reinterpret_cast<uint4 *>(own + (int64_t)(4 * ty + r) * np + 4 * tx) = make_uint4(R[r][0], R[r][1], R[r][2], R[r][3]);
    }
    // products of 64 steps: 32 x 16 threads, 2 rows and 4 columns each
    const int py = tid >> 4;
    uint32_t X[2][4];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const uint4 v = *reinterpret_cast<const uint4 *>(quarter + (int64_t)(2 * py + r) * np + 4 * tx);
        X[r][0] = v.x; X[r][1] = v.y; X[r][2] = v.z; X[r][3] = v.w;
    }
    for (int pass = 0; pass < 2; ++pass) {
        // left operand transposed in s_x, right one split: pass 0 X and P, pass 1 Q and X
        if (half == (pass == 0 ? 1 - bot : bot)) {
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    if (pass == 0) sd_split(R[r][c], s_bm[4 * ty + r][4 * tx + c], s_bl[4 * ty + r][4 * tx + c]);
                    else s_x[4 * tx + c][4 * ty + r] = R[r][c];
                }
        }
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                if (pass == 0) s_x[4 * tx + c][2 * py + r] = X[r][c];
                else sd_split(X[r][c], s_bm[2 * py + r][4 * tx + c], s_bl[2 * py + r][4 * tx + c]);
            }
        __syncthreads();
        int top = -1;
        for (int t = tid >> 5; t < H; t += SD_THREADS / 32) {   // a warp per step: its largest operands
            const int ln = tid & 31;
            int a = -1000, c = -1000;
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const uint32_t xv = s_x[t][ln + 32 * q], mv = s_bm[t][ln + 32 * q];
                if (sd_valid(xv)) a = max(a, 31 - __clz((int)xv));
                if (mv) c = max(c, 31 - __clz((int)mv));
            }
            a = __reduce_max_sync(0xffffffffu, a);
            c = __reduce_max_sync(0xffffffffu, c);
            top = max(top, a + c);
        }
        if (top >= SD_TOP) flags |= RBG_EV_RISK;
#pragma unroll 4
        for (int t = 0; t < H; ++t) {
            const uint2 x2 = *reinterpret_cast<const uint2 *>(&s_x[t][2 * py]);
            const uint4 m4 = *reinterpret_cast<const uint4 *>(&s_bm[t][4 * tx]);
            const uint4 l4 = *reinterpret_cast<const uint4 *>(&s_bl[t][4 * tx]);
            const uint32_t x[2] = {x2.x, x2.y}, m[4] = {m4.x, m4.y, m4.z, m4.w}, l[4] = {l4.x, l4.y, l4.z, l4.w};
#pragma unroll
            for (int r = 0; r < 2; ++r)
#pragma unroll
                for (int c = 0; c < 4; ++c) X[r][c] = min(X[r][c], x[r] * m[c] + l[c]);
        }
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int c = 0; c < 4; ++c)
                if (!sd_valid(X[r][c])) X[r][c] = SD_NONE;
        __syncthreads();                     // before the operands are staged again
    }
#pragma unroll
    for (int r = 0; r < 2; ++r)
        *reinterpret_cast<uint4 *>(quarter + (int64_t)(2 * py + r) * np + 4 * tx) = make_uint4(X[r][0], X[r][1], X[r][2], X[r][3]);
    flush_status(st, 0, flags);
}

// Step K.  The launch's tiles: block rows I below K (above: K - 1 upwards), the next one first, and
// for each the block columns J up to K (from K on), in BN columns.
template <typename T, int BN>
__global__ void __launch_bounds__(SD_THREADS, 1)
sd_step_kernel(const T *__restrict__ in, int64_t ld_in, uint32_t *work, int64_t np, int64_t n, int K, int above,
               bool vec, DevStatus *st) {
    constexpr int NC = BN / 16;              // columns per thread (32 x 16 threads, 4 rows each)
    typedef typename std::conditional<NC == 4, uint4, uint2>::type Vec;
    static_assert(NC == 2 || NC == 4, "32 or 64 columns");
    extern __shared__ __align__(16) unsigned char sd_smem[];
    SdSmem<BN> &S = *reinterpret_cast<SdSmem<BN> *>(sd_smem);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tx = tid & 15, ty = tid >> 4;
    const int nb = (int)(np / SD_B), cols = (int)((above ? nb - K : K + 1) * (SD_B / BN));
    const int r = (int)blockIdx.x / cols, q = (int)blockIdx.x % cols;
    const int I = above ? K - 1 - r : K + 1 + r;
    const bool next = r == 0;                // the block row this step completes
    const int64_t i0 = (int64_t)I * SD_B, k0 = (int64_t)K * SD_B;
    const int64_t j0 = (above ? k0 : 0) + (int64_t)q * BN;
    unsigned flags = 0;
    unsigned steps = 0;

    uint32_t acc[4][NC];
    auto load = [](const uint32_t *p, uint32_t (&v)[NC]) {
        const Vec t = *reinterpret_cast<const Vec *>(p);
        const uint32_t *w = reinterpret_cast<const uint32_t *>(&t);
#pragma unroll
        for (int c = 0; c < NC; ++c) v[c] = w[c];
    };
    auto store = [](uint32_t *p, const uint32_t (&v)[NC]) {
        Vec t;
        uint32_t *w = reinterpret_cast<uint32_t *>(&t);
#pragma unroll
        for (int c = 0; c < NC; ++c) w[c] = v[c];
        *reinterpret_cast<Vec *>(p) = t;
    };
#pragma unroll
    for (int e = 0; e < 4; ++e) load(work + (i0 + 4 * ty + e) * np + j0 + NC * tx, acc[e]);
    if (tid < 3 * SD_K) (&S.or_a[0][0])[tid] = 0;

    // chunk ch: 4 steps of rows ar and ar + 64 of the left operand (A(I, K), or D(I) for the second
    // product) and NC columns of step ty of the right one (C(K, J))
    const int ar = tid >> 3, aj = (tid & 7) * 4;
    uint32_t xa[2][4], xb[NC];
    auto fetch = [&](int ch, bool second) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int64_t i = i0 + ar + 64 * h;
            if (second) {
                const uint4 v = *reinterpret_cast<const uint4 *>(work + i * np + i0 + ch * SD_K + aj);
                xa[h][0] = v.x; xa[h][1] = v.y; xa[h][2] = v.z; xa[h][3] = v.w;
            } else {
                const int64_t k = k0 + ch * SD_K + aj;
                const T *row = in + i * ld_in + k;
                T a[4] = {0, 0, 0, 0};
                if (vec && i < n && k + 4 <= n) {    // 4-byte storage, aligned rows
                    *reinterpret_cast<uint4 *>(a) = *reinterpret_cast<const uint4 *>(row);
                } else {
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (i < n && k + e < n) a[e] = row[e];
                }
#pragma unroll
                for (int e = 0; e < 4; ++e) xa[h][e] = sd_lane<T>(a[e], true);
            }
        }
        if (!second) load(work + (k0 + ch * SD_K + ty) * np + j0 + NC * tx, xb);
    };
    // acc (+)= left (x) right over SD_B steps; the right operand is staged beside the left one, or is
    // the tile in tm / tl
    int s3 = 0;
    auto product = [&](bool second) {
        fetch(0, second);
        for (int ch = 0; ch < SD_B / SD_K; ++ch) {
            const int buf = ch & 1;
            uint32_t oa[4] = {0, 0, 0, 0};
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    S.as[buf][aj + e][sd_as(aj + e, ar + 64 * h)] = xa[h][e];
                    if (sd_valid(xa[h][e])) oa[e] |= xa[h][e];
                }
            if (!second) {
                uint32_t m[NC], l[NC], ob = 0;
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    sd_split(xb[c], m[c], l[c]);
                    if (m[c]) ob |= xb[c];
                }
                store(&S.bm[buf][ty][NC * tx], m);
                store(&S.bl[buf][ty][NC * tx], l);
#pragma unroll
                for (int o = 8; o > 0; o >>= 1) ob |= __shfl_xor_sync(0xffffffffu, ob, o);
                if (tx == 0) S.or_b[buf][ty] = ob;
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                oa[e] |= __shfl_xor_sync(0xffffffffu, oa[e], 8);
                oa[e] |= __shfl_xor_sync(0xffffffffu, oa[e], 16);
                if (lane < 8 && oa[e]) atomicOr(&S.or_a[s3][aj + e], oa[e]);
            }
            __syncthreads();
            if (ch + 1 < SD_B / SD_K) fetch(ch + 1, second);   // in flight during this chunk's products
            const uint32_t va = S.or_a[s3][lane], vb = second ? S.or_t[ch * SD_K + lane] : S.or_b[buf][lane];
            // the previous chunk's slot: read before this chunk's barrier, written after the next one
            if (warp == 0) S.or_a[s3 == 0 ? 2 : s3 - 1][lane] = 0;
            const bool live = va != 0 && vb != 0;
            uint32_t act = __ballot_sync(0xffffffffu, live);
            if (live && (31 - __clz((int)va)) + (31 - __clz((int)vb)) >= SD_TOP) flags |= RBG_EV_RISK;
            steps += __popc(act);
            while (act) {                    // two steps at a time (the last one twice when alone)
                int j[2];
                uint32_t x[2][4], m[2][NC], l[2][NC];
                j[0] = __ffs((int)act) - 1;
                act &= act - 1;
                j[1] = act ? __ffs((int)act) - 1 : j[0];
                act &= act - 1;
                uint32_t none = SD_NONE;
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const uint4 x4 = *reinterpret_cast<const uint4 *>(&S.as[buf][j[u]][sd_as(j[u], 4 * ty)]);
                    x[u][0] = x4.x; x[u][1] = x4.y; x[u][2] = x4.z; x[u][3] = x4.w;
                    none &= x4.x & x4.y & x4.z & x4.w;
                }
                if (!__any_sync(0xffffffffu, none != SD_NONE)) continue;
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    load(second ? &S.tm[ch * SD_K + j[u]][NC * tx] : &S.bm[buf][j[u]][NC * tx], m[u]);
                    load(second ? &S.tl[ch * SD_K + j[u]][NC * tx] : &S.bl[buf][j[u]][NC * tx], l[u]);
                }
#pragma unroll
                for (int u = 0; u < 2; ++u)
#pragma unroll
                    for (int e = 0; e < 4; ++e)
#pragma unroll
                        for (int c = 0; c < NC; ++c) acc[e][c] = min(acc[e][c], x[u][e] * m[u][c] + l[u][c]);
            }
            s3 = s3 == 2 ? 0 : s3 + 1;
        }
    };
    __syncthreads();
    product(false);
#pragma unroll
    for (int e = 0; e < 4; ++e)
#pragma unroll
        for (int c = 0; c < NC; ++c)
            if (!sd_valid(acc[e][c])) acc[e][c] = SD_NONE;
    if (next) {                              // block-uniform: C = T (+) D(I) (x) T
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            uint32_t m[NC], l[NC], o = 0;
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                sd_split(acc[e][c], m[c], l[c]);
                if (m[c]) o |= acc[e][c];
            }
            store(&S.tm[4 * ty + e][NC * tx], m);
            store(&S.tl[4 * ty + e][NC * tx], l);
#pragma unroll
            for (int b = 8; b > 0; b >>= 1) o |= __shfl_xor_sync(0xffffffffu, o, b);
            if (tx == 0) S.or_t[4 * ty + e] = o;
        }
        // (product() writes `as` slot 0 at once: last read two chunks and a barrier ago)
        product(true);
#pragma unroll
        for (int e = 0; e < 4; ++e)
#pragma unroll
            for (int c = 0; c < NC; ++c)
                if (!sd_valid(acc[e][c])) acc[e][c] = SD_NONE;
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) store(work + (i0 + 4 * ty + e) * np + j0 + NC * tx, acc[e]);
    if (tid == 0 && steps) atomicAdd(&st->executed, (unsigned long long)steps * SD_B * BN);
    flush_status(st, 0, flags);
}

// Bit masks of the left (z = 0: by rows, bit k of row[i][w] is (i, 32 w + k)) and the right operand
// matrix (z = 1: by columns, bit k of col[w][j] is (32 w + k, j)), with the largest MSB of each step's
// operands (lmax: columns of the left one, rmax: rows of the right one).  Below the diagonal the left
// one is A and the right one C, above it the other way round.  A thread per column of 32 rows.
template <typename T>
__device__ __forceinline__ uint32_t sd_cell(const T *in, int64_t ld_in, const uint32_t *work, int64_t np, int64_t n,
                                            bool of_in, int64_t i, int64_t j) {
    if (i >= n || j >= n) return SD_NONE;
    return of_in ? sd_lane<T>(in[i * ld_in + j], i != j) : work[i * np + j];
}
template <typename T>
__global__ void __launch_bounds__(256)
sd_mask_kernel(const T *__restrict__ in, int64_t ld_in, const uint32_t *__restrict__ work, int64_t np, int64_t n,
               int above, uint32_t *__restrict__ row, uint32_t *__restrict__ col, int *__restrict__ lmax,
               int *__restrict__ rmax) {
    const int lane = threadIdx.x & 31;
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, w = blockIdx.y;
    if (j >= np) return;                     // whole warps: np is a multiple of 32
    const bool left = blockIdx.z == 0;
    const bool of_in = left != (above != 0);
    uint32_t v[32];
#pragma unroll
    for (int k = 0; k < 32; ++k) v[k] = sd_cell<T>(in, ld_in, work, np, n, of_in, 32 * w + k, j);
    uint32_t bits = 0, any = 0;
#pragma unroll
    for (int k = 0; k < 32; ++k) {
        const bool on = sd_valid(v[k]);
        if (left) {
            const unsigned ballot = __ballot_sync(0xffffffffu, on);
            if (lane == k) bits = ballot;    // lane k: row 32 w + k, the warp's 32 columns
            if (on) any |= v[k];             // this column
        } else {
            bits |= (uint32_t)on << k;
            const unsigned o = __reduce_or_sync(0xffffffffu, on ? v[k] : 0u);
            if (lane == k) any = o;          // lane k: row 32 w + k
        }
    }
    if (left) row[(32 * w + lane) * (np / 32) + j / 32] = bits;
    else col[w * np + j] = bits;
    int *to = left ? lmax + j : rmax + 32 * w + lane;
    if (any) atomicMax(to, 31 - __clz((int)any));
}

// Each cell's first value: the smallest step k with bit k in both masks, a thread per column and
// rows in turn.  lmax and rmax: the largest MSB of step k's left and right operands, whose product
// may reach the top bit.
template <typename T>
__global__ void __launch_bounds__(256)
sd_first_kernel(const T *__restrict__ in, int64_t ld_in, const uint32_t *__restrict__ work, int64_t np, int64_t n,
                int above, const uint32_t *__restrict__ row, const uint32_t *__restrict__ col,
                const int *__restrict__ lmax, const int *__restrict__ rmax, DevStatus *st) {
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, nw = np / 32;
    int top = -1;
    unsigned flags = 0;
    if (j < n) {
        if (blockIdx.y == 0 && lmax[j] >= 0 && rmax[j] >= 0 && lmax[j] + rmax[j] >= SD_TOP) flags |= RBG_EV_RISK;
        for (int64_t i = blockIdx.y; i < n; i += gridDim.y) {
            if (!(above ? j > i : j < i) || !sd_valid(work[i * np + j]) || in[i * ld_in + j] != 0) continue;
            int64_t k = -1;
            for (int64_t w = (above ? i : j) / 32; w < nw; ++w) {
                const uint32_t both = row[i * nw + w] & col[w * np + j];
                if (both) {
                    k = 32 * w + __ffs((int)both) - 1;
                    break;
                }
            }
            if (k < 0) {
                flags |= RBG_EV_RISK;        // inconsistent: the general kernels decide
                continue;
            }
            const uint32_t x = sd_cell<T>(in, ld_in, work, np, n, !above, i, k);
            const uint32_t y = sd_cell<T>(in, ld_in, work, np, n, above, k, j);
            top = max(top, (31 - __clz((int)x)) + (31 - __clz((int)y)));
        }
    }
    flush_status(st, top > 0 && top < SD_TOP ? 1ull << top : 0ull, flags);
}

// The whole closure of a plan of one matrix (its tables uploaded): conversion, block rows, first
// values, finalization.  Nothing is written to `out` when a flag asks for another path.
template <typename T>
static int launch_sided(const FwPlan &P, const T *in, int64_t ld_in, T *out, unsigned char *ws, cudaStream_t s,
                        bool above) {
    static PerDeviceOnce once;               // per storage type, for every device
    const int configured = once.run([] {
        RBG_CUDA_TRY(cudaFuncSetAttribute(sd_step_kernel<T, 32>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)sizeof(SdSmem<32>)));
        RBG_CUDA_TRY(cudaFuncSetAttribute(sd_step_kernel<T, 64>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)sizeof(SdSmem<64>)));
        return (int)RBG_OK;
    });
    if (configured) return configured;
    const FwComp &c = P.comps[0];
    const int64_t n = c.n, np = c.np, nb = np / SD_B, nw = np / 32;
    DevStatus *st = reinterpret_cast<DevStatus *>(ws + P.off_status);
    const FwComp *comps = reinterpret_cast<const FwComp *>(ws + P.off_comps);
    const int64_t *pconv = reinterpret_cast<const int64_t *>(ws + P.off_pconv);
    uint32_t *work = reinterpret_cast<uint32_t *>(ws + P.off_lanes) + c.work_off;
    unsigned char *occ = ws + P.off_occ;
    uint32_t *row = reinterpret_cast<uint32_t *>(ws + P.off_sided), *col = row + np * nw;
    int *lmax = reinterpret_cast<int *>(col + np * nw), *rmax = lmax + np;
    note_launches(6 + nb - 1);
    RBG_CUDA_TRY(cudaMemsetAsync(occ, 1, std::max<size_t>(P.occ_bytes, 1), s));   // finalization reads every block
    RBG_CUDA_TRY(cudaMemsetAsync(lmax, 0xff, (size_t)np * 8, s));
    cudaEvent_t t = timer_begin(3, s);
    status_init_kernel<<<1, 128, 0, s>>>(st, 1);
    fw_convert_kernel<T, uint32_t><<<(unsigned)P.pre_conv[1], FW_THREADS, 0, s>>>(
        in, reinterpret_cast<uint32_t *>(ws + P.off_lanes), occ, comps, pconv, 1, 32, (int)sizeof(T) * 8, st);
    timer_end(3, t, s);
    t = timer_begin(2, s);
    sd_diag_kernel<<<(unsigned)nb, SD_THREADS, 0, s>>>(work, np, above ? 1 : 0, st);
    timer_end(2, t, s);
    t = timer_begin(0, s);
    const bool vec = sizeof(T) == 4 && (uintptr_t)in % 16 == 0 && ld_in % 4 == 0;
    for (int64_t q = 0; q + 1 < nb; ++q) {
        const int K = (int)(above ? nb - 1 - q : q);
        const int64_t tiles = (nb - 1 - q) * (q + 1);    // of SD_B x SD_B
        // 32 columns per CTA while that keeps to about two CTAs per SM in turn: the chain through the
        // next block row is half as long
        if (4 * tiles <= 2 * sm_count())
            sd_step_kernel<T, 32><<<(unsigned)(4 * tiles), SD_THREADS, sizeof(SdSmem<32>), s>>>(
                in, ld_in, work, np, n, K, above ? 1 : 0, vec, st);
        else
            sd_step_kernel<T, 64><<<(unsigned)(2 * tiles), SD_THREADS, sizeof(SdSmem<64>), s>>>(
                in, ld_in, work, np, n, K, above ? 1 : 0, vec, st);
    }
    timer_end(0, t, s);
    t = timer_begin(1, s);
    sd_mask_kernel<T><<<dim3((unsigned)((np + 255) / 256), (unsigned)nw, 2), 256, 0, s>>>(
        in, ld_in, work, np, n, above ? 1 : 0, row, col, lmax, rmax);
    sd_first_kernel<T><<<dim3((unsigned)((np + 255) / 256), (unsigned)std::min<int64_t>(n, 128)), 256, 0, s>>>(
        in, ld_in, work, np, n, above ? 1 : 0, row, col, lmax, rmax, st);
    timer_end(1, t, s);
    t = timer_begin(3, s);
    fw_finalize_kernel<T, uint32_t><<<(unsigned)P.pre_conv[1], FW_THREADS, 0, s>>>(
        in, reinterpret_cast<uint32_t *>(ws + P.off_lanes), out, comps, pconv, 1, st, occ, RowStats());
    timer_end(3, t, s);
    RBG_CUDA_TRY(cudaGetLastError());
    return RBG_OK;
}
