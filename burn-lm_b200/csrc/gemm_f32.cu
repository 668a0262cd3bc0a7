// y[N, M] = x[N, K] . W[M, K]^T in true fp32: FFMA on CUDA cores, no tensor-core mode of any kind.
// This is the matrix product of the 32-bit path.  The sum over K runs in one fixed order that depends on neither N nor M, so a
// token's result is the same whatever else is in the batch: K is cut into shares of 1,024, each is summed in order, and the
// shares' sums are added in order by a second kernel.
//
// What bounds it: fp32 multiply-adds from some 50 rows on (74 TFLOP/s on this chip at best), the weights' way in below.  Both
// operands lie along K and stay so in shared memory (rows padded by a 16-byte piece, so that eight rows start in eight different
// groups of banks): a slice comes by cp.async two slices ahead, nothing is transposed, and twelve 16-byte loads feed 128
// multiply-adds of a thread with 8 x 4 outputs.  The shares give a product of few columns as many blocks as one of many
// (317 x 2,048 x 8,192: 160 tiles, 1,280 blocks).  Two places of K an instruction (fma.rn.f32x2) ran at the same rate, 8 x 8
// outputs a thread too (four blocks a multiprocessor hide the loads, two do not).  With 16,384 x 2,048 / 2,048 x 8,192 weights,
// us: 1 row 189 / 381 -> 48 / 30, 16 rows 189 / 383 -> 49 / 31, 48 rows 192 / 437 -> 101 / 58, 317 rows 703 / 671 -> 497 / 254.
#include <algorithm>

#include "common.cuh"

BLM_API const char* blm_gemm_last_error() { return g_blm_error; }

constexpr int kShare = 1024;      // places of K of a share
constexpr int kBK = 32;           // places of K of a slice in shared memory
constexpr int kRow = kBK + 4;     // floats a row of a slice
constexpr int kSlices = 3;

__device__ __forceinline__ void cp16(float* dst, const float* src, int bytes) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp4(float* dst, const float* src, int bytes) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}

struct GemmArgs {
    const float *x, *w;
    float* y;                     // [N, ldy], or with several shares [share][batch][N][M]
    int N, M, K, shares, batch;
    long long ldx, ldw, ldy, bx, bw, by;
};

// A block: TN x TM threads of AN x AM outputs each; thread (tn, tm) owns the rows tn + TN i of x and tm + TM j of W.
template <int TN, int TM, int AN, int AM, bool VEC>
__global__ void __launch_bounds__(TN * TM) gemm_f32_kernel(const GemmArgs a) {
    constexpr int T = TN * TM, BN = TN * AN, BM = TM * AM, kStage = (BN + BM) * kRow;
    extern __shared__ __align__(16) float sm[];
    const int tid = threadIdx.x, tm = tid % TM, tn = tid / TM;
    const int b = blockIdx.z / a.shares, share = blockIdx.z % a.shares;
    const int n0 = blockIdx.y * BN, m0 = blockIdx.x * BM;
    const float* x = a.x + (size_t)b * a.bx;
    const float* w = a.w + (size_t)b * a.bw;
    const int k_lo = share * kShare, k_hi = min(a.K, k_lo + kShare);
    const int slices = (k_hi - k_lo + kBK - 1) / kBK;

    // the thread's pieces of a slice: places c .. of the rows r0 + i kStep, x's rows first.  A row of W beyond the
    // end is read as the last one (its outputs are not stored), one of x comes as zeros, from the last one's address.
    constexpr int P = VEC ? 4 : 1, kPer = kBK / P, kStep = T / kPer, kPieces = (BN + BM) / kStep;
    static_assert(T % kPer == 0 && BN % kStep == 0 && BM % kStep == 0, "a piece of every row falls to one thread");
    const int r0 = tid / kPer, c = tid % kPer * P;
    const float* xt = x + (size_t)n0 * a.ldx + k_lo + c;
    const float* wt = w + (size_t)m0 * a.ldw + k_lo + c;
    int off[VEC ? kPieces : 1];                // (VEC: a tile's rows lie within 2^31 places, which the caller makes sure of)
    auto offset = [&](int i) {
        const int r = r0 + i * kStep;
        return r < BN ? min(r, a.N - 1 - n0) * a.ldx : min(r - BN, a.M - 1 - m0) * a.ldw;
    };
    if (VEC) {
#pragma unroll
        for (int i = 0; i < kPieces; ++i) off[VEC ? i : 0] = (int)offset(i);
    }
    auto load = [&](int slice) {
        if (slice < slices) {
            float* st = sm + slice % kSlices * kStage + r0 * kRow + c;
            const int k0 = slice * kBK, bytes = k_lo + k0 + c < k_hi ? 4 * P : 0;
            const int at = bytes ? k0 : -c;    // (nothing is copied then, from an address inside the row)
#pragma unroll
            for (int i = 0; i < kPieces; ++i) {
                const float* src = (i * kStep < BN ? xt : wt) + (VEC ? off[VEC ? i : 0] : offset(i)) + at;
                const int copied = i * kStep < BN && n0 + r0 + i * kStep >= a.N ? 0 : bytes;      // (rows that are not there come as zeros)
                if (VEC) cp16(st + i * kStep * kRow, src, copied);
                else cp4(st + i * kStep * kRow, src, copied);
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };

    float acc[AN][AM];
#pragma unroll
    for (int i = 0; i < AN; ++i)
#pragma unroll
        for (int j = 0; j < AM; ++j) acc[i][j] = 0.f;
    for (int s = 0; s < kSlices - 1; ++s) load(s);
    for (int slice = 0; slice < slices; ++slice) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(kSlices - 2) : "memory");
        __syncthreads();                       // this slice is there, and the one before is done with
        load(slice + kSlices - 1);
        const float* st = sm + slice % kSlices * kStage;
        const float* xs = st + tn * kRow;
        const float* ws = st + (BN + tm) * kRow;
#pragma unroll
        for (int k = 0; k < kBK; k += 4) {
            float4 xv[AN], wv[AM];
#pragma unroll
            for (int i = 0; i < AN; ++i) xv[i] = *reinterpret_cast<const float4*>(xs + i * TN * kRow + k);
#pragma unroll
            for (int j = 0; j < AM; ++j) wv[j] = *reinterpret_cast<const float4*>(ws + j * TM * kRow + k);
#pragma unroll
            for (int e = 0; e < 4; ++e)
#pragma unroll
                for (int i = 0; i < AN; ++i)
#pragma unroll
                    for (int j = 0; j < AM; ++j)
                        acc[i][j] = fmaf((&xv[i].x)[e], (&wv[j].x)[e], acc[i][j]);
        }
    }
    float* y = a.shares > 1 ? a.y + ((size_t)share * a.batch + b) * a.N * a.M : a.y + (size_t)b * a.by;
    const long long ldy = a.shares > 1 ? a.M : a.ldy;
#pragma unroll
    for (int i = 0; i < AN; ++i)
#pragma unroll
        for (int j = 0; j < AM; ++j) {
            const int n = n0 + tn + TN * i, m = m0 + tm + TM * j;
            if (n < a.N && m < a.M) y[(size_t)n * ldy + m] = acc[i][j];
        }
}

// y[b][n][m] = the shares' sums added in order; a block a row (or a share of it), four columns a thread where they lie so
template <int V>
__global__ void add_shares_kernel(const float* __restrict__ part, float* __restrict__ y, int N, int M, int shares, int batch, long long ldy,
                                  long long by) {
    const size_t row = blockIdx.x, all = (size_t)batch * N * M;
    const float* from = part + row * M;
    float* to = y + row / N * by + row % N * ldy;
    for (int m = (blockIdx.y * blockDim.x + threadIdx.x) * V; m < M; m += gridDim.y * blockDim.x * V) {
        if (V == 4) {
            float4 s = *reinterpret_cast<const float4*>(from + m);
            for (int k = 1; k < shares; ++k) {
                const float4 t = *reinterpret_cast<const float4*>(from + k * all + m);
                s.x += t.x;
                s.y += t.y;
                s.z += t.z;
                s.w += t.w;
            }
            *reinterpret_cast<float4*>(to + m) = s;
        } else {
            float s = from[m];
            for (int k = 1; k < shares; ++k) s += from[k * all + m];
            to[m] = s;
        }
    }
}

template <int TN, int TM, int AN, int AM>
static int launch(const GemmArgs& a, bool vec, cudaStream_t stream) {
    constexpr int BN = TN * AN, BM = TM * AM;
    constexpr int smem = kSlices * (BN + BM) * kRow * 4;
    const dim3 grid((a.M + BM - 1) / BM, (a.N + BN - 1) / BN, a.batch * a.shares);
    auto k = vec ? gemm_f32_kernel<TN, TM, AN, AM, true> : gemm_f32_kernel<TN, TM, AN, AM, false>;
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return blm_fail(BLM_CUDA_ERROR, "gemm_f32: %s", cudaGetErrorString(e));
    }
    k<<<grid, TN * TM, smem, stream>>>(a);
    return blm_check_launch("gemm_f32");
}

static int shares_of(int K) { return (K + kShare - 1) / kShare; }

// What one pass of a product takes: products (the grid's third dimension holds their shares), rows, columns.  With several shares a
// pass is cut so that its planes of sums stay within kPlanes floats (256 MB), in even parts of whole tiles along the longer side
// (every pass reads the shorter side's operand again): a large product would otherwise hold K / 1,024 times its result (2,048 rows
// of logits over 128,256 columns and K 4,096: 4.2 GB).  Every pass ends in a round of blocks that
// is not full: 600 x 32,768 x 4,096 in two passes 3,731 -> 3,776 us, 2,048 x 4,096 x 14,336 5,198 -> 5,229 (in six and eight: 3,842, 5,492).
constexpr long long kPlanes = 64 << 20;
struct Pass {
    int products, rows, cols;
};
static Pass pass_of(int batch, int N, int M, int K) {
    const int shares = shares_of(K);
    Pass p = {std::max(1, std::min(batch, 65535 / std::max(1, shares))), std::max(1, N), std::max(1, M)};
    if (shares <= 1) return p;
    const long long one = (long long)shares * p.rows * p.cols;
    if (one <= kPlanes) {
        p.products = (int)std::min<long long>(p.products, kPlanes / one);
        return p;
    }
    p.products = 1;
    auto cut = [&](int& side, int other) {     // in even parts, as many as it takes, none below a tile
        const long long parts = ((long long)shares * side * other + kPlanes - 1) / kPlanes;
        side = (int)std::min<long long>(side, ((side + parts - 1) / parts + 63) / 64 * 64);
        while (side > 64 && (long long)shares * side * other > kPlanes) side = (side - 1) / 64 * 64;
    };
    int &longer = p.cols >= p.rows ? p.cols : p.rows, &other = p.cols >= p.rows ? p.rows : p.cols;
    cut(longer, other);
    if ((long long)shares * longer * other > kPlanes) cut(other, longer);
    return p;
}

// Floats of scratch a product needs: a plane of sums a share, none for a single share; and how many kernels it launches.
BLM_API long long blm_gemm_f32_scratch(int batch, int N, int M, int K) {
    if (batch <= 0 || N <= 0 || M <= 0 || K <= 0) return 0;
    const Pass p = pass_of(batch, N, M, K);
    return shares_of(K) > 1 ? (long long)shares_of(K) * p.products * p.rows * p.cols : 0;
}
BLM_API int blm_gemm_f32_launches(int batch, int N, int M, int K) {
    if (batch <= 0 || N <= 0 || M <= 0 || K <= 0) return 0;
    const Pass p = pass_of(batch, N, M, K);
    return ((batch - 1) / p.products + 1) * ((N - 1) / p.rows + 1) * ((M - 1) / p.cols + 1) * (shares_of(K) > 1 ? 2 : 1);
}

// `batch` products y[b] = x[b] . W[b]^T of one shape; the operands of product b lie b * (bx, bw, by) elements on.
BLM_API int blm_gemm_f32_batched(const float* x, const float* w, float* y, int batch, int N, int M, int K, long long ldx, long long ldw,
                                 long long ldy, long long bx, long long bw, long long by, float* scratch, cudaStream_t stream) {
    if (N == 0 || M == 0 || batch == 0) return BLM_OK;
    BLM_REQUIRE(N > 0 && M > 0 && K > 0 && batch > 0, "gemm_f32: bad sizes %d x %d %d %d", batch, N, M, K);
    const int shares = shares_of(K);
    BLM_REQUIRE(batch <= 65535 && shares <= 65535 && N <= 64 * 65535, "gemm_f32: too many rows or products (%d x %d)", batch, N);
    BLM_REQUIRE(shares == 1 || scratch != nullptr, "gemm_f32: a sum over %d places needs scratch", K);
    // 16-byte pieces where every row starts at a multiple of 16 bytes, and 64 rows lie within what an int can tell
    const bool vec = (((size_t)x | (size_t)w) & 15) == 0 && ldx < (1 << 25) && ldw < (1 << 25) && K % 4 == 0 && ldx % 4 == 0 && ldw % 4 == 0 && bx % 4 == 0 && bw % 4 == 0;
    const bool vec4 = (((size_t)y | (size_t)scratch) & 15) == 0 && M % 4 == 0 && ldy % 4 == 0 && by % 4 == 0;
    const Pass pass = pass_of(batch, N, M, K);
    for (int b0 = 0; b0 < batch; b0 += pass.products)
        for (int n0 = 0; n0 < N; n0 += pass.rows)
            for (int m0 = 0; m0 < M; m0 += pass.cols) {
                const int products = std::min(pass.products, batch - b0), rows = std::min(pass.rows, N - n0), cols = std::min(pass.cols, M - m0);
                float* to = y + (size_t)b0 * by + (size_t)n0 * ldy + m0;
                const GemmArgs a = {x + (size_t)b0 * bx + (size_t)n0 * ldx, w + (size_t)b0 * bw + (size_t)m0 * ldw, shares > 1 ? scratch : to,
                                    rows, cols, K, shares, products, ldx, ldw, ldy, bx, bw, by};
                // few rows: what takes the time is the weights' way in, which wants many small blocks (16 rows of 16,384 x 2,048 weights
                // 49 us, with tiles of 32 rows 73); then the smallest tile that holds the rows (48 rows: 101 us, in tiles of 64 rows 121)
                const int rc = rows <= 16   ? launch<4, 16, 4, 2>(a, vec, stream)
                               : rows <= 32 ? launch<8, 16, 4, 4>(a, vec, stream)
                               : rows <= 48 ? launch<8, 16, 6, 4>(a, vec, stream)
                                            : launch<8, 16, 8, 4>(a, vec, stream);
                if (rc != BLM_OK) return rc;
                if (shares == 1) continue;
                const int per = 256 * (vec4 ? 4 : 1);
                const dim3 grid(products * rows, (cols + per - 1) / per);
                if (vec4) add_shares_kernel<4><<<grid, 256, 0, stream>>>(scratch, to, rows, cols, shares, products, ldy, by);
                else add_shares_kernel<1><<<grid, 256, 0, stream>>>(scratch, to, rows, cols, shares, products, ldy, by);
                if (int added = blm_check_launch("gemm_f32 (shares)")) return added;
            }
    return BLM_OK;
}

BLM_API int blm_gemm_f32(const float* x, const float* w, float* y, int N, int M, int K,
                         long long ldx, long long ldw, long long ldy, float* scratch, cudaStream_t stream) {
    return blm_gemm_f32_batched(x, w, y, 1, N, M, K, ldx, ldw, ldy, 0, 0, 0, scratch, stream);
}
