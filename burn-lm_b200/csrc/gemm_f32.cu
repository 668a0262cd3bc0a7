// y[N, M] = x[N, K] . W[M, K]^T in 32 bits: all 24 bits of both operands, float32 sums.
// This is the matrix product of the 32-bit path.  The sum over K runs in one fixed order that depends on the weight alone, so a
// token's result is the same whatever else is in the batch: K is cut into shares, each is summed in order, and the shares' sums are
// added in order.  Two kernels: on the tensor cores (further down) where K and W's rows come in 16-byte pieces, and FFMA for
// small weights and everything else.
//
// FFMA: what bounds it is fp32 multiply-adds from some 50 rows on (74 TFLOP/s on this chip at best), the weights' way in below.  Both
// operands lie along K and stay so in shared memory (rows padded by a 16-byte piece, so that eight rows start in eight different
// groups of banks): a slice comes by cp.async two slices ahead, nothing is transposed, and twelve 16-byte loads feed 128
// multiply-adds of a thread with 8 x 4 outputs.  The shares of 1,024 give a product of few columns as many blocks as one of many
// (317 x 2,048 x 8,192: 160 tiles, 1,280 blocks); a second kernel adds their sums.  Two places of K an instruction (fma.rn.f32x2) ran at the
// same rate, 8 x 8 outputs a thread too (four blocks a multiprocessor hide the loads, two do not).  Rows in 16-byte pieces run here if the
// weight is small (kTcWeight has the times) or K is below kTcLeast; others by pieces of four bytes: with 16,384 x 2,050 / 2,048 x 8,190
// weights, us, 1 row 59 / 37, 16 rows 60 / 39, 64 rows 143 / 74, 317 rows 628 / 317 (in 16-byte pieces 50 / 36, 58 / 36, 128 / 77, 507 / 263).
#include <algorithm>

#include "tcgen05.cuh"

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

    // rows in 16-byte pieces: a slice is summed by itself and then added (one chain of 256 places: 2.9e-7 off, so 1.2e-7)
    float acc[AN][AM], sum[AN][AM];
#pragma unroll
    for (int i = 0; i < AN; ++i)
#pragma unroll
        for (int j = 0; j < AM; ++j) acc[i][j] = sum[i][j] = 0.f;
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
            if (VEC && k == kBK - 4) {
#pragma unroll
                for (int i = 0; i < AN; ++i)
#pragma unroll
                    for (int j = 0; j < AM; ++j) {
                        sum[i][j] += acc[i][j];
                        acc[i][j] = 0.f;
                    }
            }
        }
    }
    float* y = a.shares > 1 ? a.y + ((size_t)share * a.batch + b) * a.N * a.M : a.y + (size_t)b * a.by;
    const long long ldy = a.shares > 1 ? a.M : a.ldy;
#pragma unroll
    for (int i = 0; i < AN; ++i)
#pragma unroll
        for (int j = 0; j < AM; ++j) {
            const int n = n0 + tn + TN * i, m = m0 + tm + TM * j;
            if (n < a.N && m < a.M) y[(size_t)n * ldy + m] = VEC ? sum[i][j] : acc[i][j];
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

// ---------------------------------------------------------------------------------------------
// The product on the tensor cores, for K a multiple of 4 from kTcLeast on and rows of W at multiples of 16 bytes, unless the weight is
// small: a choice by the weight alone, so that a row's bits do not depend on what else is in the batch.
//
// Both operands as three bfloat16 numbers a float (tcgen05.cuh): 24 bits and six products, 282 TFLOP/s of the chip's 1,692 against
// 74 of FFMA.  x is split once by a launch of its own (it is read by every tile of W's rows); W, which is read once or a few times,
// comes as it lies and is split on its way, so no weight is kept twice.  A block: 128 rows of W x nt rows of x, K in steps of 64.
// One warp brings W by TMA, one x's parts; four warps split W's floats, a lane a row, into tensor memory, from where the tensor
// core takes its 128-row operand (through shared memory that operand's reads took its whole bandwidth: 317 rows below 142 us);
// two threads in turn issue the 24 tcgen05.mma of a step, the small products first; eight warps add the finished step to their sums.  The
// tensor core's additions cut bits off, so no more than a step is left to it (four additions of the large products); the sums over
// the steps are float32 additions in order, and so are those over shares of 1,024 places of K.  The shares of a tile are a
// block's, which adds them up in y, or where there are few tiles a block each and planes of sums: the same additions.
// x's parts are rounded, which leaves the products left out of either sign, W's cut off: their conversion is on the way of every step (rounded, too,
// 444 rows of 10,752 x 816 weights 43.3 us for 42.3).
// Infinities: an infinite x1 makes x2 not a number, and a zero x2 times an infinity is not one either, so an output that is not
// finite is formed again with fmaf from the floats themselves (so is one of an x whose x1 rounds to infinity).  Operands below 2^-109 lose their last bits (x3 would be below
// the smallest bfloat16 number).
// With 16,384 x 2,048 / 2,048 x 8,192 weights, us (FFMA above): 1 row 40 / 30, 16 rows 40 / 30, 64 rows 44 / 32, 160 rows 62 / 44, 317 rows
// 110 / 69, 2,000 rows 603 / 390 (FFMA in 16-byte pieces 3,000 / 1,513); launched back to back 28 / 17, 29 / 18, 33 / 20, 56 / 32, 104 / 59; the error against 64 bits 1.2e-7 (5.7e-7).  A step of 160 rows of x takes some 2,900 clocks
// of which the tensor core works 1,920: x's parts have room for two steps only.
// ---------------------------------------------------------------------------------------------
constexpr int kTcLeast = 64;
// Floats of W and K up to which FFMA is the faster one: a launch less, no tensor memory to take, tiles of 16 x 32.  us, FFMA and so, 17 / 317 / 2,000 rows:
// 64 x 64 2.4 / 2.4 / 3.0 and 6.3 / 6.4 / 6.8; 512 x 64 2.3 / 3.1 / 5.9 and 6.5 / 6.7 / 7.8; 128 x 256 4.9 / 4.9 / 8.1 and 7.9 / 8.0 / 8.4; 64 x 512
// 8.2 / 8.2 / 9.4 and 9.8 / 9.8 / 11.  Twice as many: 1,024 x 64 2.2 / 3.8 / 11 and 6.5 / 7.0 / 9.0; 256 x 256 4.7 / 5.3 / 11 and 7.9 / 8.0 / 9.0.
// (Large batches of such products are the exception: 64 of 128 x 256, 2,000 rows 207 and 136.)  From 1,024 places on FFMA gains nothing.
constexpr int kTcWeight = 1 << 15, kTcSmall = 512;
constexpr int kTcShare = 1024;    // places of K of a share at most
constexpr int kTcK = 32;          // of a slice; two slices are a step
constexpr int kTcRows = 128;      // rows of W of a tile
constexpr int kTcMost = 160;      // rows of x of a tile at most
constexpr int kTcFew = 64;        // up to so many rows of x a tile, W's way through the converting warps is what takes the time
constexpr int kTcW = 2 * kTcRows * kTcK * 4;          // bytes of a step of W's floats
constexpr int kTcCols = 512, kTcPart = kTcK / 2;      // columns of tensor memory: all, of a part of a slice of W
constexpr int kTcSmem = 227 * 1024 - 1024;
constexpr int kTcThreads = 16 * 32;

struct TcArgs {
    const float *x, *w;
    float* y;                     // as GemmArgs
    int N, M, K, shares, share_len, batch;
    long long ldx, ldw, ldy, bx, bw, by;
    int nt, n_tiles, m_tiles, w_stages, x_stages, w_batches;
    int planes;                   // every share by a block of its own, its sums a plane of y; else a block adds a tile's shares up in y
    int* status;
};

struct RingAt {                    // a place of a ring and the parity of its phase
    int at = 0;
    unsigned phase = 0;
    __device__ __forceinline__ void next(int n) {
        if (++at == n) {
            at = 0;
            phase ^= 1;
        }
    }
};

// one output that is not finite, formed again by the whole warp
__device__ __noinline__ float tc_again(const float* x, const float* w, int k) {
    const int lane = threadIdx.x & 31;
    float s = 0.f;
    for (int c0 = 0; c0 < k; c0 += 128) {
        const int c = c0 + 4 * lane;
        if (c < k) {
#pragma unroll
            for (int e = 0; e < 4; ++e) s = fmaf(x[c + e], w[c + e], s);
        }
        if (__any_sync(0xffffffffu, isnan(s))) break;      // (stays so)
    }
    return warp_sum(s);
}

template <bool FEW>
__global__ void __launch_bounds__(kTcThreads, 1) gemm_f32_tc_kernel(const TcArgs a, const __grid_constant__ CUtensorMap xmap,
                                                                    const __grid_constant__ CUtensorMap wmap) {
    using namespace tc5;
    constexpr int kConverters = FEW ? 8 : 4, kAdders = FEW ? 4 : 8, kMine = FEW ? kTcFew : kTcMost / 2;      // rows of x a warp adds
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const int x_part = a.nt * 2 * kTcK * 2, x_bytes = 3 * x_part;
    unsigned char* w_ring = smem;                              // [w_stages][2][128][32] floats
    unsigned char* x_ring = smem + a.w_stages * kTcW;          // [x_stages][3][nt][128 bytes]
    unsigned long long* w_full = reinterpret_cast<unsigned long long*>(x_ring + a.x_stages * x_bytes);
    unsigned long long* w_empty = w_full + a.w_stages;
    unsigned long long* x_full = w_empty + a.w_stages;
    unsigned long long* split = x_full + a.x_stages;           // W's parts are there
    unsigned long long* done = split + a.x_stages;             // a step's products are in tensor memory, x's and W's parts free
    unsigned long long* added = done + a.x_stages;             // [2] and have been added to the sums
    unsigned* tmem_slot = reinterpret_cast<unsigned*>(added + 2);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned parts0 = 2 * a.nt;          // tensor memory: two accumulators, then W's parts [x_stages][2][3][16 columns]
    if (threadIdx.x == 0) {
        for (int s = 0; s < a.w_stages; ++s) {
            mbar_init(w_full + s, 1);
            mbar_init(w_empty + s, kConverters);
        }
        for (int s = 0; s < a.x_stages; ++s) {
            mbar_init(x_full + s, 1);
            mbar_init(split + s, kConverters);
            mbar_init(done + s, 1);
        }
        for (int b = 0; b < 2; ++b) mbar_init(added + b, kAdders);
        mbar_init_fence();
    }
    if (warp == 1) tmem_alloc(tmem_slot, kTcCols);
    fence_before();
    __syncthreads();
    fence_after();
    const unsigned tmem_base = *tmem_slot;

    // unit t: a tile's share.  The rows of x beside one another (they share W's slices in L2), then W's rows, the planes, the
    // products; a block that adds a tile's shares up takes them one after the other
    const int at_once = a.planes ? 1 : a.shares;
    const long long units = (long long)a.n_tiles * a.m_tiles * (a.planes ? a.shares : 1) * a.batch * at_once;
    auto next_unit = [&](long long t) { return (t + 1) % at_once ? t + 1 : t + 1 + (long long)(gridDim.x - 1) * at_once; };
    const long long first_unit = (long long)blockIdx.x * at_once;
    struct Unit {
        int n0, m0, k0, steps, share, b;
    };
    auto unit_at = [&](long long t) {
        Unit r;
        r.share = (int)(t % at_once);
        t /= at_once;
        r.n0 = (int)(t % a.n_tiles) * a.nt;
        t /= a.n_tiles;
        r.m0 = (int)(t % a.m_tiles) * kTcRows;
        t /= a.m_tiles;
        if (a.planes) {
            r.share = (int)(t % a.shares);
            t /= a.shares;
        }
        r.b = (int)t;
        r.k0 = r.share * a.share_len;
        r.steps = (min(a.share_len, a.K - r.k0) + 2 * kTcK - 1) / (2 * kTcK);      // (places beyond K come as zeros)
        return r;
    };
    bool ok = true;
    auto wait = [&](unsigned long long* bar, unsigned phase) {
        if (ok && !mbar_wait(bar, phase)) {
            ok = false;
            if (lane == 0) atomicCAS(a.status, TC5_OK, TC5_TIMEOUT_PRODUCT);
        }
        return ok;
    };

    if (warp == 0 || warp == 15) {
        // ---------------- the loads: warp 0 W's floats, warp 15 x's parts as soon as the kernel before has written them ----------------
        const bool of_w = warp == 0;
        const int stages = of_w ? a.w_stages : a.x_stages;
        unsigned long long *full = of_w ? w_full : x_full, *empty = of_w ? w_empty : done;
        RingAt r;
        unsigned free = stages;                // stages that nothing was in yet
        if (!of_w) pdl_wait();
        for (long long t = first_unit; t < units && ok; t = next_unit(t)) {
            const Unit u = unit_at(t);
            for (int k = 0; k < u.steps; ++k) {
                if (free) --free;
                else if (!wait(empty + r.at, r.phase ^ 1)) break;
                if (elect()) {
                    const int c = u.k0 + k * 2 * kTcK;
                    if (of_w) {
                        unsigned char* to = w_ring + r.at * kTcW;
                        mbar_expect_tx(full + r.at, kTcW);
                        tma_load_3d(to, &wmap, c, u.m0, min(u.b, a.w_batches - 1), full + r.at);
                        tma_load_3d(to + kTcW / 2, &wmap, c + kTcK, u.m0, min(u.b, a.w_batches - 1), full + r.at);
                    } else {
                        mbar_expect_tx(full + r.at, x_bytes);
                        tma_load_3d(x_ring + r.at * x_bytes, &xmap, c, u.n0, u.b * 3, full + r.at);
                    }
                }
                __syncwarp();
                r.next(stages);
            }
        }
        // no copy is on its way when the block ends, not even where a wait ran out
        for (int s = 0; s < (free ? r.at : stages); ++s) mbar_wait(full + s, s < r.at ? r.phase : r.phase ^ 1);
    } else if (warp < 3) {
        // ---------------- the tensor core: a warp the even steps, one the odd ones (one warp for all: 64 rows of x 128 us instead of 114) ----------------
        const int b = warp - 1;
        const unsigned idesc = instruction(a.nt), d = tmem_base + (unsigned)(b * a.nt);
        const unsigned long long x_desc = operand(x_ring, 2, 1024);
        RingAt r, last;                        // (last: where the last products went, if any)
        last.at = -1;
        unsigned turn = 0;
        for (long long t = first_unit; t < units && ok; t = next_unit(t)) {
            const int steps = unit_at(t).steps;
            for (int k = 0; k < steps; ++k, ++turn, r.next(a.x_stages)) {
                if ((int)(turn & 1) != b) continue;
                if (turn >= 2) wait(added + b, ((turn >> 1) - 1) & 1);
                wait(x_full + r.at, r.phase);
                if (!wait(split + r.at, r.phase)) break;
                fence_after();
                if (elect()) {
                    // (part of W, part of x): the smallest products first
                    constexpr int of_w[6] = {2, 0, 1, 1, 0, 0}, of_x[6] = {0, 2, 1, 0, 1, 0};
                    const unsigned wd = tmem_base + parts0 + r.at * 6 * kTcPart;
                    const unsigned long long xd = x_desc + (unsigned)(r.at * (x_bytes >> 4));
#pragma unroll
                    for (int p = 0; p < 6; ++p)
#pragma unroll
                        for (int kk = 0; kk < 4; ++kk)
                            mma_ts(d, wd + (kk >> 1) * 3 * kTcPart + of_w[p] * kTcPart + 8 * (kk & 1),
                                   xd + (unsigned)(of_x[p] * (x_part >> 4) + 2 * kk), idesc, p > 0 || kk > 0);
                    commit(done + r.at);
                }
                __syncwarp();
                last = r;
            }
        }
        if (last.at >= 0) mbar_wait(done + last.at, last.phase);       // nor are products
    } else if (warp < 3 + kConverters) {
        // ---------------- W's floats into parts: a lane a row; four warps both slices of a step, or eight one each ----------------
        const int row = (warp & 3) * 32 + lane, only = (warp - 3) >> 2;
        const unsigned to = tmem_base + ((unsigned)((warp & 3) * 32) << 16) + parts0;
        RingAt r, o;                           // where W comes from, and where its parts go
        unsigned free = a.x_stages;
        for (long long t = first_unit; t < units && ok; t = next_unit(t)) {
            const int steps = unit_at(t).steps;
            for (int k = 0; k < steps; ++k) {
                if (free) --free;
                else wait(done + o.at, o.phase ^ 1);
                if (!wait(w_full + r.at, r.phase)) break;
                fence_after();
#pragma unroll 1
                for (int half = FEW ? only : 0; half < (FEW ? only + 1 : 2); ++half) {
                    const unsigned char* w = w_ring + r.at * kTcW + half * (kTcW / 2) + row * (kTcK * 4);
                    float4 v[kTcK / 4];
#pragma unroll
                    for (int c = 0; c < kTcK / 4; ++c) v[c] = *reinterpret_cast<const float4*>(w + ((c ^ (row & 7)) << 4));      // 128-byte swizzle
                    unsigned p[3][kTcPart];
#pragma unroll
                    for (int c = 0; c < kTcK / 4; ++c) {
                        split3_as<false, false>(v[c].x, v[c].y, p[0][2 * c], p[1][2 * c], p[2][2 * c]);
                        split3_as<false, false>(v[c].z, v[c].w, p[0][2 * c + 1], p[1][2 * c + 1], p[2][2 * c + 1]);
                    }
#pragma unroll
                    for (int i = 0; i < 3; ++i) tmem_st16(to + ((o.at * 2 + half) * 3 + i) * kTcPart, p[i]);
                }
                wait_st();
                fence_before();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(w_empty + r.at);
                    mbar_arrive(split + o.at);
                }
                r.next(a.w_stages);
                o.next(a.x_stages);
            }
        }
    } else {
        // ---------------- the sums: a lane a row of W, all or half of the tile's rows of x a warp ----------------
        const int quarter = warp & 3, half = FEW ? a.nt : a.nt >> 1, c0 = warp >= 3 + kConverters + 4 ? half : 0;
        RingAt r;
        unsigned turn = 0;
        for (long long t = first_unit; t < units && ok; t = next_unit(t)) {
            const Unit u = unit_at(t);
            float sum[kMine];
#pragma unroll
            for (int j = 0; j < kMine; ++j) sum[j] = 0.f;
            for (int k = 0; k < u.steps; ++k, ++turn, r.next(a.x_stages)) {
                const int b = turn & 1;
                if (!wait(done + r.at, r.phase)) break;
                fence_after();
                const unsigned at = tmem_base + ((unsigned)(quarter * 32) << 16) + (unsigned)(b * a.nt + c0);
#pragma unroll
                for (int j = 0; j < kMine; j += 16) {
                    if (j < half) {
                        float v[16];
                        tmem_ld16(at + j, v);
                        wait_ld();
#pragma unroll
                        for (int e = 0; e < 16; ++e) sum[j + e] += v[e];
                    }
                }
                fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(added + b);
            }
            if (!ok) break;
            const int m = u.m0 + quarter * 32 + lane, n0 = u.n0 + c0;
            float bad = 0.f;
#pragma unroll
            for (int j = 0; j < kMine; ++j) bad += j < half ? sum[j] * 0.f : 0.f;      // not zero if one is not finite
            if (__any_sync(0xffffffffu, bad != 0.f)) {
                const float* x = a.x + (size_t)u.b * a.bx + u.k0;
                const float* w = a.w + (size_t)u.b * a.bw + u.k0;
#pragma unroll
                for (int j = 0; j < kMine; ++j) {
                    const bool mine = j < half && n0 + j < a.N && m < a.M && !isfinite(sum[j]);
                    unsigned rows = __ballot_sync(0xffffffffu, mine);
                    while (rows) {
                        const int l = __ffs(rows) - 1;
                        rows &= rows - 1;
                        const float v = tc_again(x + (size_t)(n0 + j) * a.ldx, w + (size_t)(u.m0 + quarter * 32 + l) * a.ldw, min(a.share_len, a.K - u.k0));
                        if (lane == l) sum[j] = v;
                    }
                }
            }
            const long long ldy = a.planes ? a.M : a.ldy;
            float* y = (a.planes ? a.y + ((size_t)u.share * a.batch + u.b) * a.N * a.M : a.y + (size_t)u.b * a.by) + (size_t)n0 * ldy + m;
            const bool more = !a.planes && u.share > 0;        // (the same thread wrote the shares before)
#pragma unroll
            for (int j = 0; j < kMine; j += 8) {
                if (j >= half || m >= a.M) continue;
                if (more) {
                    float before[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e) before[e] = n0 + j + e < a.N ? y[(size_t)e * ldy] : 0.f;
#pragma unroll
                    for (int e = 0; e < 8; ++e) sum[j + e] += before[e];
                }
#pragma unroll
                for (int e = 0; e < 8; ++e)
                    if (n0 + j + e < a.N) y[(size_t)e * ldy] = sum[j + e];
                y += 8 * ldy;
            }
        }
    }
    fence_before();
    __syncthreads();
    if (warp == 1) {
        fence_after();
        tmem_free(tmem_base, kTcCols);
    }
}

// x's rows as three bfloat16 numbers a float: planes [batch][3][N][pitch].  A thread four places of K of a row; `rows` short rows a block, or
// (0) a block a row or a part of one (64 products of 2,000 rows of 64 places 168 us so, of which the products take 30; but the division
// shows in long rows, 104 us of a product for 103).
template <bool VEC>
__global__ void __launch_bounds__(256) split_rows_kernel(const float* __restrict__ x, __nv_bfloat16* __restrict__ out, int N, int K, int pitch,
                                                         long long ldx, long long bx, int rows) {
    pdl_launch_dependents();
    int n = blockIdx.x, first = blockIdx.y * blockDim.x + threadIdx.x, step = gridDim.y * blockDim.x;
    if (rows > 0) {
        const int own = threadIdx.x / (K / 4);
        if (own >= rows) return;
        n = n * rows + own;
        first = threadIdx.x - own * (K / 4);
        step = K;
    }
    if (n >= N) return;
    const int b = blockIdx.z;
    const float* row = x + (size_t)b * bx + (size_t)n * ldx;
    __nv_bfloat16* to = out + ((size_t)b * 3 * N + n) * pitch;
    const size_t plane = (size_t)N * pitch;
    for (int c = first * 4; c < K; c += step * 4) {
        const float4 v = VEC ? *reinterpret_cast<const float4*>(row + c) : make_float4(row[c], row[c + 1], row[c + 2], row[c + 3]);
        uint2 p1, p2, p3;
        tc5::split3_as<true, true>(v.x, v.y, p1.x, p2.x, p3.x);
        tc5::split3_as<true, true>(v.z, v.w, p1.y, p2.y, p3.y);
        *reinterpret_cast<uint2*>(to + c) = p1;
        *reinterpret_cast<uint2*>(to + plane + c) = p2;
        *reinterpret_cast<uint2*>(to + 2 * plane + c) = p3;
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

// Rows of x of a tile, and whether every share of K is a block's own: the ones with the least time by this count.  A slice of a tile
// takes what was measured for its rows of x (a block alone, 256 slices after one another: 87, 114, 132, 169, 202 us), the end of a
// share some 1.5 us; planes of sums are a launch more and are written and read.
struct Plan {
    int nt, planes;
};
static Plan tc_plan(int batch, int N, int M, int K, int sms) {
    constexpr double slice_us[kTcMost / 32] = {0.32, 0.405, 0.49, 0.63, 0.76};
    Plan best = {32, 0};
    double least = -1;
    const int shares = (K + kTcShare - 1) / kTcShare;
    for (int nt = 32; nt <= kTcMost; nt += 32)
        for (int planes = 0; planes <= (shares > 1 ? 1 : 0); ++planes) {
            const long long units = (long long)((N + nt - 1) / nt) * ((M + kTcRows - 1) / kTcRows) * batch * (planes ? shares : 1);
            const long long rounds = (units + sms - 1) / sms;
            const double share = (double)K / shares / kTcK * slice_us[nt / 32 - 1] + 1.5;
            const double cost = rounds * share * (planes ? 1 : shares) + (planes ? 3 + 1.6e-6 * batch * shares * N * M : 0);
            if (least < 0 || cost < least) {
                least = cost;
                best = {nt, planes};
            }
        }
    return best;
}

// The tensor cores take it: by W's size and how it lies, never by N.
static bool tc_size(int M, int K) { return K >= kTcLeast && K % 4 == 0 && (K > kTcSmall || (long long)M * K > kTcWeight); }
static bool tc_takes(const float* w, int M, int K, long long ldw, long long bw) {
    return tc_size(M, K) && ((size_t)w & 15) == 0 && ldw > 0 && ldw % 4 == 0 && ldw < (1ll << 37) && bw >= 0 && bw % 4 == 0 &&
           bw < (1ll << 37) && tc5::encode_tiled() != nullptr;
}

// x's parts go to `scratch`
static int launch_tc(const GemmArgs& g, const Plan& plan, float* scratch, int* status, cudaStream_t stream) {
    const int pitch = (g.K + 7) / 8 * 8;
    __nv_bfloat16* parts = reinterpret_cast<__nv_bfloat16*>(scratch);
    TcArgs a = {g.x, g.w, g.y, g.N, g.M, g.K, g.shares, ((g.K + g.shares - 1) / g.shares + 63) / 64 * 64, g.batch, g.ldx, g.ldw, g.ldy, g.bx, g.bw, g.by};
    a.m_tiles = (g.M + kTcRows - 1) / kTcRows;
    a.nt = plan.nt;
    a.planes = plan.planes;
    a.n_tiles = (g.N + a.nt - 1) / a.nt;
    a.w_batches = g.batch > 1 && g.bw > 0 ? g.batch : 1;
    a.status = status;
    constexpr int kBarriers = 256;
    const int x_step = 2 * a.nt * kTcK * 6;
    a.x_stages = std::min(4, (kTcCols - 2 * a.nt) / (6 * kTcPart));
    a.w_stages = std::min(6, (kTcSmem - kBarriers - a.x_stages * x_step) / kTcW);
    const int smem = a.w_stages * kTcW + a.x_stages * x_step + kBarriers + 1024;
    CUtensorMap xmap, wmap;
    if (!tc5::make_map_3d(&xmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, parts, {g.K, g.N, 3ll * g.batch}, {2ll * pitch, 2ll * pitch * g.N}, {2 * kTcK, a.nt, 3},
                          CU_TENSOR_MAP_SWIZZLE_128B) ||
        !tc5::make_map_3d(&wmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, g.w, {g.K, g.M, a.w_batches}, {4 * g.ldw, a.w_batches > 1 ? 4 * g.bw : 4 * g.ldw},
                          {kTcK, kTcRows, 1}, CU_TENSOR_MAP_SWIZZLE_128B))
        return blm_fail(BLM_CUDA_ERROR, "gemm_f32: cuTensorMapEncodeTiled refused %d x %d x %d", g.N, g.M, g.K);
    auto kernel = a.nt <= kTcFew ? gemm_f32_tc_kernel<true> : gemm_f32_tc_kernel<false>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kTcSmem + 1024);
    if (e != cudaSuccess) return blm_fail(BLM_CUDA_ERROR, "gemm_f32: %s", cudaGetErrorString(e));
    const bool vec = ((size_t)g.x & 15) == 0 && g.ldx % 4 == 0 && g.bx % 4 == 0;
    const int rows = g.K <= 512 ? 256 / (g.K / 4) : 0;
    const dim3 grid(rows ? (g.N + rows - 1) / rows : g.N, rows ? 1 : std::min(8, (g.K + 1023) / 1024), g.batch);
    if (vec) split_rows_kernel<true><<<grid, 256, 0, stream>>>(g.x, parts, g.N, g.K, pitch, g.ldx, g.bx, rows);
    else split_rows_kernel<false><<<grid, 256, 0, stream>>>(g.x, parts, g.N, g.K, pitch, g.ldx, g.bx, rows);
    if (int rc = blm_check_launch("gemm_f32 (parts)")) return rc;
    const long long tiles = (long long)a.n_tiles * a.m_tiles * (a.planes ? g.shares : 1) * g.batch;
    e = blm_launch_dependent(kernel, dim3((unsigned)std::min<long long>(tiles, blm_sm_count())), dim3(kTcThreads), smem, stream, a, xmap, wmap);
    if (e != cudaSuccess) return blm_fail(BLM_CUDA_ERROR, "gemm_f32: %s", cudaGetErrorString(e));
    return blm_check_launch("gemm_f32 (tensor cores)");
}

static int shares_of(bool tc, int K) { return tc ? (K + kTcShare - 1) / kTcShare : (K + kShare - 1) / kShare; }

// What one pass of a product takes: products (the grid's third dimension holds their shares), rows, columns.  With several shares a
// pass is cut so that its planes of sums stay within kPlanes floats (256 MB; on the tensor cores 192 MB, beside 24 MB for x's parts, which stay in L2), in
// even parts of whole tiles along the longer side (every pass reads the shorter side's operand again): a large product would
// otherwise hold K / 1,024 times its result (2,048 rows of logits over 128,256 columns and K 4,096: 4.2 GB).  Every pass ends in a
// round of blocks that is not full: FFMA with rows in 16-byte pieces, 600 x 32,768 x 4,096 in two passes 3,731 -> 3,776 us, 2,048 x 4,096 x
// 14,336 5,198 -> 5,229 (in six and eight: 3,842, 5,492); by pieces of four bytes, as they run here, 4,825 and 6,676.
constexpr long long kPlanes = 64 << 20, kTcPlanes = 48 << 20, kTcParts = 6 << 20;
struct Pass {
    int products, rows, cols;
};
static long long tc_parts(int products, int rows, int K) { return (long long)products * rows * ((K + 7) / 8 * 8) * 3 / 2; }      // floats
static Pass pass_of(bool tc, int batch, int N, int M, int K) {
    const int shares = shares_of(tc, K);
    const long long planes = tc ? kTcPlanes : kPlanes;
    Pass p = {std::max(1, std::min(batch, 65535 / std::max(1, shares))), std::max(1, N), std::max(1, M)};
    if (tc && tc_parts(1, p.rows, K) > kTcParts) {
        const long long parts = (tc_parts(1, p.rows, K) + kTcParts - 1) / kTcParts;
        p.rows = (int)std::min<long long>(p.rows, ((p.rows + parts - 1) / parts + 63) / 64 * 64);
        while (p.rows > 64 && tc_parts(1, p.rows, K) > kTcParts) p.rows = (p.rows - 1) / 64 * 64;
    }
    if (tc) p.products = (int)std::max(1ll, std::min<long long>(p.products, kTcParts / tc_parts(1, p.rows, K)));
    if (shares <= 1 || (tc && !tc_plan(p.products, p.rows, p.cols, K, blm_sm_count()).planes)) return p;
    const long long one = (long long)shares * p.rows * p.cols;
    if (one <= planes) {
        p.products = (int)std::min<long long>(p.products, planes / one);
        return p;
    }
    p.products = 1;
    auto cut = [&](int& side, int other) {     // in even parts, as many as it takes, none below a tile
        const long long parts = ((long long)shares * side * other + planes - 1) / planes;
        side = (int)std::min<long long>(side, ((side + parts - 1) / parts + 63) / 64 * 64);
        while (side > 64 && (long long)shares * side * other > planes) side = (side - 1) / 64 * 64;
    };
    int &longer = p.cols >= p.rows ? p.cols : p.rows, &other = p.cols >= p.rows ? p.rows : p.cols;
    cut(longer, other);
    if ((long long)shares * longer * other > planes) cut(other, longer);
    return p;
}
static bool planes_of(bool tc, const Pass& p, int K) {
    return shares_of(tc, K) > 1 && (!tc || tc_plan(p.products, p.rows, p.cols, K, blm_sm_count()).planes);
}
static long long scratch_of(bool tc, int batch, int N, int M, int K) {
    const Pass p = pass_of(tc, batch, N, M, K);
    return (planes_of(tc, p, K) ? (long long)shares_of(tc, K) * p.products * p.rows * p.cols : 0) + (tc ? tc_parts(p.products, p.rows, K) : 0);
}

// Whether the tensor cores form a product (`w`, its strides: what the product itself is given),
BLM_API int blm_gemm_f32_tensor(const float* w, int M, int K, long long ldw, long long bw) { return tc_takes(w, M, K, ldw, bw); }
// floats of scratch that it then needs (planes of sums, x's parts), or however W lies, and how many kernels it launches.
BLM_API long long blm_gemm_f32_scratch_as(int tensor, int batch, int N, int M, int K) {
    return batch <= 0 || N <= 0 || M <= 0 || K <= 0 ? 0 : scratch_of(tensor, batch, N, M, K);
}
BLM_API long long blm_gemm_f32_scratch(int batch, int N, int M, int K) {
    const long long ffma = blm_gemm_f32_scratch_as(0, batch, N, M, K);
    return tc_size(M, K) ? std::max(ffma, blm_gemm_f32_scratch_as(1, batch, N, M, K)) : ffma;
}
BLM_API int blm_gemm_f32_launches(int tensor, int batch, int N, int M, int K) {
    if (batch <= 0 || N <= 0 || M <= 0 || K <= 0) return 0;
    const Pass p = pass_of(tensor, batch, N, M, K);
    return ((batch - 1) / p.products + 1) * ((N - 1) / p.rows + 1) * ((M - 1) / p.cols + 1) * (1 + (tensor ? 1 : 0) + (planes_of(tensor, p, K) ? 1 : 0));
}

// `batch` products y[b] = x[b] . W[b]^T of one shape; the operands of product b lie b * (bx, bw, by) elements on.
BLM_API int blm_gemm_f32_batched(const float* x, const float* w, float* y, int batch, int N, int M, int K, long long ldx, long long ldw,
                                 long long ldy, long long bx, long long bw, long long by, float* scratch, int* status, cudaStream_t stream) {
    if (N == 0 || M == 0 || batch == 0) return BLM_OK;
    BLM_REQUIRE(N > 0 && M > 0 && K > 0 && batch > 0, "gemm_f32: bad sizes %d x %d %d %d", batch, N, M, K);
    const bool tc = tc_takes(w, M, K, ldw, batch > 1 ? bw : 0);
    const int shares = shares_of(tc, K);
    BLM_REQUIRE(batch <= 65535 && shares <= 65535 && N <= 64 * 65535, "gemm_f32: too many rows or products (%d x %d)", batch, N);
    BLM_REQUIRE((shares == 1 && !tc) || (scratch != nullptr && status != nullptr), "gemm_f32: a sum over %d places needs scratch and a status word", K);
    // 16-byte pieces where every row starts at a multiple of 16 bytes, and 64 rows lie within what an int can tell
    const bool vec = (((size_t)x | (size_t)w) & 15) == 0 && ldx < (1 << 25) && ldw < (1 << 25) && K % 4 == 0 && ldx % 4 == 0 && ldw % 4 == 0 && bx % 4 == 0 && bw % 4 == 0;
    const bool vec4 = (((size_t)y | (size_t)scratch) & 15) == 0 && M % 4 == 0 && ldy % 4 == 0 && by % 4 == 0;
    const Pass pass = pass_of(tc, batch, N, M, K);
    const bool planes = planes_of(tc, pass, K);      // (a last, smaller pass as the others)
    for (int b0 = 0; b0 < batch; b0 += pass.products)
        for (int n0 = 0; n0 < N; n0 += pass.rows)
            for (int m0 = 0; m0 < M; m0 += pass.cols) {
                const int products = std::min(pass.products, batch - b0), rows = std::min(pass.rows, N - n0), cols = std::min(pass.cols, M - m0);
                float* to = y + (size_t)b0 * by + (size_t)n0 * ldy + m0;
                float* sums = tc ? scratch + tc_parts(products, rows, K) : scratch;
                const GemmArgs a = {x + (size_t)b0 * bx + (size_t)n0 * ldx, w + (size_t)b0 * bw + (size_t)m0 * ldw, planes ? sums : to,
                                    rows, cols, K, shares, products, ldx, ldw, ldy, bx, bw, by};
                // few rows: what takes the time is the weights' way in, which wants many small blocks (16 rows of 16,384 x 2,048 weights
                // 49 us, with tiles of 32 rows 73); so do small weights, a block's slices following one another (317 rows of 256 x 256
                // 5.5 us, with tiles of 64 rows 10.5); then the smallest tile that holds the rows (48 rows: 101 us, in tiles of 64 rows 121)
                const bool few = rows <= 16 || (vec && (long long)((rows + 15) / 16) * ((cols + 31) / 32) * products * shares <= 4 * blm_sm_count());
                const int rc = tc           ? launch_tc(a, {tc_plan(products, rows, cols, K, blm_sm_count()).nt, planes}, scratch, status, stream)
                               : few        ? launch<4, 16, 4, 2>(a, vec, stream)
                               : rows <= 32 ? launch<8, 16, 4, 4>(a, vec, stream)
                               : rows <= 48 ? launch<8, 16, 6, 4>(a, vec, stream)
                                            : launch<8, 16, 8, 4>(a, vec, stream);
                if (rc != BLM_OK) return rc;
                if (!planes) continue;
                const int per = 256 * (vec4 ? 4 : 1);
                const dim3 grid(products * rows, (cols + per - 1) / per);
                if (vec4) add_shares_kernel<4><<<grid, 256, 0, stream>>>(sums, to, rows, cols, shares, products, ldy, by);
                else add_shares_kernel<1><<<grid, 256, 0, stream>>>(sums, to, rows, cols, shares, products, ldy, by);
                if (int added = blm_check_launch("gemm_f32 (shares)")) return added;
            }
    return BLM_OK;
}

BLM_API int blm_gemm_f32(const float* x, const float* w, float* y, int N, int M, int K,
                         long long ldx, long long ldw, long long ldy, float* scratch, int* status, cudaStream_t stream) {
    return blm_gemm_f32_batched(x, w, y, 1, N, M, K, ldx, ldw, ldy, 0, 0, 0, scratch, status, stream);
}
