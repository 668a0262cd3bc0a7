// Attention without a softmax whose heads' weights are mixed before they meet the values (attention_sigmoid.cu states the
// equations), bfloat16, up to four query heads a key/value head and up to eight key/value heads: scores, mix and values of a
// tile of keys in one warp's registers.
//
// What bounds the form with shared memory between the three (attention_sigmoid.cu): every weight is written, read once a mixed
// head and written again, and three barriers a chunk keep the tensor cores idle 95 % of the time.  Here the three products
// are laid so that each leaves its result where the next one wants its operand:
//   scores, transposed:  S^T = K Q^T.  A tile's sixteen rows are keys; its eight columns are (head of the key/value head, query),
//     column 2 h + x.  Lane l then holds head l % 4 of every key/value head at key l / 4 - which is the B operand of
//   the mix:  M = talk W, m16n8k16: k runs over (four key/value heads, l % 4), the columns are keys.  Weights and talk are each
//     the sum of three bfloat16 numbers, which hold all 24 bits of a float; of their nine products the six that reach 2^-24 of
//     a product are formed.  (Two tf32 numbers each hold 22 bits: 24-bit weights of heads that cancel came out wrong.)
//     Lane l gets head row l / 4 at keys 2 (l % 4), + 1 - which, packed to bfloat16, is the B operand of
//   the values, transposed:  O^T += V^T M^T: rows are value lanes, k runs over keys, columns are eight head rows, of which four
//     belong to the key/value head.  Two queries fill both halves: the second query's rows cross over by one shuffle.
// Weights, their mix and the outputs never leave registers; shared memory holds keys, values, the queries' and talk's fragments.
// 1,536 tokens of 32 heads of 64 on 8, the kernel alone: 695 us with shared memory between the three, 167 with blocks of four warps
// that met at a barrier a tile, 130 with tiles by TMA and no barrier (quad_rows_kernel); 64 single tokens over 1,088 keys: 220, 38
// and 33 us (4.3 TB/s).
#include <type_traits>

#include "tcgen05.cuh"

BLM_API const char* blm_attention_quads_last_error() { return g_blm_error; }

constexpr int kQuads = 8;          // key/value heads, four query heads (or fewer, the others' talk being zero) each

struct QuadArgs {
    const __nv_bfloat16* q;        // [N, H dk]
    const __nv_bfloat16* pool;     // pages: keys [G][page][dk] then values [G][page][dv]
    const int* block_table;
    int table_stride;
    const int *cu_seqlens, *slot_of_seq, *start_pos, *token_seq;
    const float* talk;             // [H, H] or null
    const float* head_bias;        // [H] or null
    __nv_bfloat16* out;            // [N, H dv] (one range)
    float* partial;                // [ranges][N][H dv] fp32 (several ranges)
    int n_tokens, n_seqs, q_tiles, H, G, dk, dv, page, ranges;
    float scale, softcap;
};

// Tiles of a range when a row's `tiles` are cut into `ranges` ranges of `least` tiles at least (fewer ranges then): 256 keys where
// a block shares them among its queries, 64 for a single token.
__host__ __device__ inline int tiles_of_range(int tiles, int ranges, int least) {
    const int even = (tiles + ranges - 1) / ranges;
    return even > least ? even : least;
}
constexpr int kLeastSingle = 64 / 16;

__device__ __forceinline__ unsigned smem_at(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void ldsm_x4(unsigned (&r)[4], unsigned addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_trans(unsigned (&r)[4], unsigned addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint4& a, unsigned b0, unsigned b1) {
    const unsigned v[4] = {a.x, a.y, a.z, a.w};
    mma_bf16(c, v, b0, b1);
}
__device__ __forceinline__ void cp16(unsigned dst, const void* src, bool on) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(on ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

__device__ __forceinline__ unsigned pack_bf16(float a, float b) {
    __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<unsigned*>(&v);
}

// Two floats as the sums of three bfloat16 numbers each: eight bits a number, so all 24 of a float.
struct Limbs {
    unsigned hi, mid, lo;          // pairs, the first float in the lower half
};
__device__ __forceinline__ Limbs split_bf16(float a, float b) {
    Limbs l;
    l.hi = pack_bf16(a, b);
    a -= __uint_as_float(l.hi << 16);
    b -= __uint_as_float(l.hi & 0xffff0000u);
    l.mid = pack_bf16(a, b);
    l.lo = pack_bf16(a - __uint_as_float(l.mid << 16), b - __uint_as_float(l.mid & 0xffff0000u));
    return l;
}

// talk's fragments for the mix in shared memory: [row tile][k tile][hi, mid, lo][lane] of 16 bytes.  Row r of row tile m is head
// r % 4 of key/value head 4 m + r / 4; k = 2 h + e + 8 half of k tile t is head h of key/value head 4 t + 2 half + e.  Heads that
// are not there: zero.
constexpr int kTalkBytes = 2 * 2 * 3 * 32 * 16;
__device__ __forceinline__ void stage_talk(uint4* to, const QuadArgs& a, int tid, int threads) {
    const int per = a.H / a.G;
    for (int e = tid; e < 2 * 2 * 32; e += threads) {
        const int lane = e % 32, t = e / 32 % 2, m = e / 64;
        unsigned hi[4], mid[4], lo[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = (lane >> 2) + (i & 1) * 8, gr = 4 * m + r / 4, hr = r % 4, hk = lane & 3;
            float v[2] = {0.f, 0.f};
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                const int gk = 4 * t + 2 * (i >> 1) + x;
                if (gr < a.G && hr < per && gk < a.G && hk < per)
                    v[x] = a.talk ? a.talk[(size_t)(gr * per + hr) * a.H + gk * per + hk] : (gr == gk && hr == hk ? 1.f : 0.f);
            }
            const Limbs l = split_bf16(v[0], v[1]);
            hi[i] = l.hi;
            mid[i] = l.mid;
            lo[i] = l.lo;
        }
        uint4* at = to + (m * 2 + t) * 3 * 32 + lane;
        at[0] = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        at[32] = make_uint4(mid[0], mid[1], mid[2], mid[3]);
        at[64] = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    }
}

// The queries' fragments of one pair of queries: [key/value head][32 lanes of a key][lane] of 16 bytes (two steps of sixteen; the
// second one zero beyond the last); column n is head n / 2, query n % 2 (rows row0, row0 + 1; a query beyond `rows` is zero).  Warps
// take every `by`-th piece from `from` on, and eight of a warp's pieces are on their way together: one after another they held a
// block some 5 us before its first product.
template <int KS, bool FULL>
__device__ __forceinline__ void stage_queries(uint4* to, const QuadArgs& a, size_t row0, int rows, int lane, int from, int by) {
    const int per = a.H / a.G, steps = FULL ? KS : a.dk / 16, pairs = (steps + 1) / 2, n = lane >> 2, h = n >> 1, x = n & 1;
    const int G = FULL ? kQuads : a.G;
    const bool live = h < per && x < rows;
    const __nv_bfloat16* q = a.q + (row0 + (live ? x : 0)) * a.H * a.dk + (lane & 3) * 2;
#pragma unroll 8
    for (int i = from; i < G * pairs; i += by) {
        const int g = i / pairs, s = i % pairs;
        uint4 v = make_uint4(0, 0, 0, 0);
        if (live) {
            const unsigned* p = reinterpret_cast<const unsigned*>(q + (g * per + h) * a.dk + s * 32);
            v.x = __ldg(p);
            v.y = __ldg(p + 4);
            if (2 * s + 1 < steps) {
                v.z = __ldg(p + 8);
                v.w = __ldg(p + 12);
            }
        }
        to[i * 32 + lane] = v;
    }
}

// Rows of keys and values in shared memory are 128 bytes (256 beyond 64 lanes); the 16-byte piece c of row r lies in place
// c ^ (r % 8), so that the eight rows an ldmatrix reads at one piece lie in eight different groups of banks.
//
// Scores of a tile of sixteen keys (keys at `k`, rows of `row` bytes, a key/value head every `head` bytes) for the staged queries:
// key/value heads u0 to u0 + 3, whose products are independent, so that one's latency hides behind the others'.
template <int KS, bool FULL>
__device__ __forceinline__ void score_tile(float (&c)[4][4], int u0, unsigned k, int row, int head, const uint4* qf, int G, int steps, int lane) {
    const unsigned at = k + ((lane & 7) + (lane >> 3 & 1) * 8) * row, turn = ((lane >> 4) ^ (lane & 7)) * 16;
    const int pairs = FULL ? KS / 2 : (steps + 1) / 2;
#pragma unroll
    for (int u = 0; u < 4; ++u) c[u][0] = c[u][1] = c[u][2] = c[u][3] = 0.f;
#pragma unroll
    for (int s = 0; s < KS / 2; ++s) {
        if (FULL || s < pairs) {
            unsigned f[4][4];
            uint4 b[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int v = FULL || u0 + u < G ? u0 + u : 0;
                ldsm_x4(f[u], at + v * head + (turn ^ (s * 64)));
                b[u] = qf[(v * pairs + s) * 32 + lane];
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) mma_bf16(c[u], f[u], b[u].x, b[u].y);
            if (FULL || 2 * s + 1 < steps) {
#pragma unroll
                for (int u = 0; u < 4; ++u) ldsm_x4(f[u], at + (FULL || u0 + u < G ? u0 + u : 0) * head + (turn ^ (s * 64 + 32)));
#pragma unroll
                for (int u = 0; u < 4; ++u) mma_bf16(c[u], f[u], b[u].z, b[u].w);
            }
        }
    }
}

__device__ __forceinline__ float exp2_fast(float v) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float rcp_fast(float v) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}

// The numbers a score meets on its way to a weight 1 / (1 + exp(-(s' + bias))), s' = scale s or cap tanh(scale s / cap):
// cap tanh(x) = cap - 2 cap / (1 + exp(2 x)), so that with a cap the exponent is one multiply-add of a reciprocal.
struct WeighConsts {
    float in, out;                 // exp2(s in); exponent: start + out / (1 + that), or start + s out without a cap
};
__device__ __forceinline__ WeighConsts weigh_consts(float scale, float cap) {
    constexpr float kLog2e = 1.4426950408889634f;
    WeighConsts w;
    w.in = cap > 0.f ? 2.0f * scale / cap * kLog2e : 0.f;
    w.out = cap > 0.f ? 2.0f * cap * kLog2e : -scale * kLog2e;
    return w;
}
__device__ __forceinline__ float weigh_start(float cap, float bias) { return -(cap > 0.f ? cap + bias : bias) * 1.4426950408889634f; }

// Scores to weights, in place; key of c[.][2 r + x]: j + 8 r (j: the lane's first), query x at position p0 + x.
template <int X, bool CAP, bool OPEN>
__device__ __forceinline__ void weigh(float (&c)[4][4], const float* start, int j, int p0, const WeighConsts& k) {
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int x = 0; x < X; ++x) {
                float& v = c[u][2 * r + x];
                const float t = CAP ? rcp_fast(1.0f + exp2_fast(v * k.in)) : v;
                v = rcp_fast(1.0f + exp2_fast(fmaf(k.out, t, start[u])));
                if (!OPEN && j + 8 * r > p0 + x) v = 0.f;
            }
}

// The mixed weights of X queries for a tile of sixteen keys, packed: p[query][row tile][row half][key half] is head row
// (lane / 4) + 8 half at keys 2 (lane % 4), + 1.  Four key/value heads at a time go from scores to their share of the mix, without a
// branch in between: one half's products can run under the other half's exponentials.  A k tile's talk serves every query and
// key half, and their products do not wait for one another.  Of the nine products of limbs the three below 2^-24 of a product
// are left out; the smallest are added first.
template <int KS, int X, bool FULL, bool CAP, bool OPEN, typename F>
__device__ __forceinline__ void mixed_tile_of(unsigned (&p)[X][2][2][2], unsigned k, int row, int head, const uint4* qf, const uint4* talk,
                                              const float (&start)[kQuads], int j, int p0, const WeighConsts& consts, int G, int steps,
                                              int lane, F done) {
    float c[X][2][2][4];
#pragma unroll
    for (int x = 0; x < X; ++x)
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int r = 0; r < 2; ++r) c[x][m][r][0] = c[x][m][r][1] = c[x][m][r][2] = c[x][m][r][3] = 0.f;
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        if (FULL || 4 * t < G) {
            float w[4][4];
            score_tile<KS, FULL>(w, 4 * t, k, row, head, qf, G, steps, lane);
            if (t == 1 || (!FULL && G <= 4)) done();
            weigh<X, CAP, OPEN>(w, start + 4 * t, j, p0, consts);
            Limbs b[X][2][2];
#pragma unroll
            for (int x = 0; x < X; ++x)
#pragma unroll
                for (int r = 0; r < 2; ++r)
#pragma unroll
                    for (int half = 0; half < 2; ++half) b[x][r][half] = split_bf16(w[2 * half][2 * r + x], w[2 * half + 1][2 * r + x]);
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                if (FULL || 4 * m < G) {
                    const uint4* at = talk + (m * 2 + t) * 3 * 32 + lane;
                    const uint4 hi = at[0], mid = at[32], lo = at[64];
#define BLM_MIX(A, B)                                                                            \
    _Pragma("unroll") for (int x = 0; x < X; ++x) _Pragma("unroll") for (int r = 0; r < 2; ++r) \
        mma_bf16(c[x][m][r], A, b[x][r][0].B, b[x][r][1].B)
                    BLM_MIX(lo, hi);
                    BLM_MIX(hi, lo);
                    BLM_MIX(mid, mid);
                    BLM_MIX(mid, hi);
                    BLM_MIX(hi, mid);
                    BLM_MIX(hi, hi);
#undef BLM_MIX
                }
            }
        }
    }
#pragma unroll
    for (int x = 0; x < X; ++x)
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int half = 0; half < 2; ++half)
#pragma unroll
                for (int r = 0; r < 2; ++r) p[x][m][half][r] = pack_bf16(c[x][m][r][2 * half], c[x][m][r][2 * half + 1]);
}
// (`open`: every query sees all sixteen keys; `done` is called when the keys have been read)
template <int KS, int X, bool FULL, bool CAP, typename F>
__device__ __forceinline__ void mixed_tile(unsigned (&p)[X][2][2][2], unsigned k, int row, int head, const uint4* qf, const uint4* talk,
                                           const float (&start)[kQuads], int j, int p0, bool open, const WeighConsts& consts, int G, int steps,
                                           int lane, F done) {
    if (open) mixed_tile_of<KS, X, FULL, CAP, true>(p, k, row, head, qf, talk, start, j, p0, consts, G, steps, lane, done);
    else mixed_tile_of<KS, X, FULL, CAP, false>(p, k, row, head, qf, talk, start, j, p0, consts, G, steps, lane, done);
}

// The mixed weights of two queries as operands of the value products: b[parity] is the even and the odd key/value heads' of every
// pair, both queries in one operand.
__device__ __forceinline__ void cross(unsigned (&b)[2][2][2][2], const unsigned (&p)[2][2][2][2], int lane) {
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int half = 0; half < 2; ++half)
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const unsigned other = __shfl_xor_sync(0xffffffffu, p[1][m][half][r], 16);
                b[0][m][half][r] = lane < 16 ? p[0][m][half][r] : other;
                b[1][m][half][r] = lane < 16 ? other : p[0][m][half][r];
            }
}

// Sixteen keys of values (64 lanes from the address on, rows of `row` bytes, a key/value head every `head` bytes) times the packed
// weights of both queries.
template <bool FULL>
__device__ __forceinline__ void value_tile(float (&o)[kQuads][4][4], unsigned v, int row, int head, const unsigned (&b)[2][2][2][2], int G,
                                           int lane) {
    const unsigned at = v + ((lane & 7) + (lane >> 4) * 8) * row, turn = ((lane >> 3 & 1) ^ (lane & 7)) * 16;
#pragma unroll
    for (int u = 0; u < kQuads; ++u) {
        if (FULL || u < G) {
            const unsigned b0 = b[u & 1][u >> 2][u >> 1 & 1][0], b1 = b[u & 1][u >> 2][u >> 1 & 1][1];
#pragma unroll
            for (int d = 0; d < 4; ++d) {
                unsigned f[4];
                ldsm_x4_trans(f, at + u * head + (turn ^ (d * 32)));
                mma_bf16(o[u][d], f, b0, b1);
            }
        }
    }
}

// Two queries' outputs (rows row0, row0 + 1, of which `rows` exist), value lanes lane0 and on, to the result or to the range's share.
// Column n of key/value head u: head n % 4; an even u's columns 0 .. 3 are query 0's, an odd one's query 1's.
__device__ __forceinline__ void store_rows(const QuadArgs& a, const float (&o)[kQuads][4][4], size_t row0, int rows, int lane0, int range, int G,
                                           int lane) {
    const int per_kv = a.H / a.G, HD = a.H * a.dv;
#pragma unroll
    for (int u = 0; u < kQuads; ++u)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int n = 2 * (lane & 3) + e, h = n & 3, x = (n >> 2) ^ (u & 1);
            if (u >= G || h >= per_kv || x >= rows) continue;
            const size_t at = (row0 + x) * HD + (u * per_kv + h) * a.dv;
#pragma unroll
            for (int d = 0; d < 4; ++d)
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const int lanev = lane0 + d * 16 + (lane >> 2) + 8 * r;
                    if (lanev < a.dv) {
                        if (a.ranges > 1) a.partial[(size_t)range * a.n_tokens * HD + at + lanev] = o[u][d][2 * r + e];
                        else a.out[at + lanev] = __float2bfloat16_rn(o[u][d][2 * r + e]);
                    }
                }
        }
}

__device__ __forceinline__ void head_starts(float (&begin)[kQuads], const QuadArgs& a, int G, int lane) {
    const int per_kv = a.H / a.G;
#pragma unroll
    for (int u = 0; u < kQuads; ++u)
        begin[u] = weigh_start(a.softcap, a.head_bias && u < G && (lane & 3) < per_kv ? a.head_bias[u * per_kv + (lane & 3)] : 0.f);
}

// A portion block's sequence, queries and range of keys: the longest blocks first (the last rows of the longest sequences see the
// most keys, a row's ranges are of one length).
struct PortionWork {
    int seq, first, n_new, i0, start, kv_hi, lo, hi, range;
};
__device__ __forceinline__ PortionWork portion_work(const QuadArgs& a, int bq, int keys) {
    PortionWork w;
    w.range = blockIdx.x % a.ranges;
    const int at = blockIdx.x / a.ranges;
    w.seq = at % a.n_seqs;
    w.i0 = (a.q_tiles - 1 - at / a.n_seqs) * bq;
    w.first = a.cu_seqlens[w.seq];
    w.n_new = a.cu_seqlens[w.seq + 1] - w.first;
    w.start = a.start_pos[w.seq];
    w.kv_hi = w.start + min(w.i0 + bq, w.n_new);
    const int tiles = (w.kv_hi + keys - 1) / keys, per = tiles_of_range(tiles, a.ranges, 256 / keys);
    w.lo = w.range * per;
    w.hi = w.i0 < w.n_new ? min(tiles, w.lo + per) : 0;
    return w;
}

// ---------------------------------------------------------------------------------------------
// portions, keys and values of up to 64 lanes: a block of eight warps owns sixteen queries of a sequence and a range of its keys; a
// warp owns two queries.  Tiles of 16 keys come by TMA (whose 128-byte swizzle is the order of the pieces above) into a ring of four,
// and a warp goes through them at its own pace: no barrier between the warps, so that one's scores and products run under
// another's exponentials.  The last warp to leave a tile asks for the one four further on into its place.
// What bounds it (1,536 tokens of 32 heads of 64 on 8, 130 us): no unit alone; a tile's 160 products, its 128 special functions, the
// 1,700 instructions around them and the 1,700 cycles of shared-memory reads (every two queries read all keys and values again)
// take 30 to 40 % of the time each, and two warps a scheduler, all that the outputs' registers leave room for, hide only part of
// one under another.  Left out one at a time, copies, scores, weights, mix and values each took 24 to 37 us off the form before.
// Measured on the way: copies by TMA and no barrier 167 -> 145 us; the queries' pieces fetched together 145 -> 135; scores, weights and
// mix by halves of the key/value heads 135 -> 130.  A late start for half of the warps: 137.  Limbs cut off instead of rounded: 129.
// ---------------------------------------------------------------------------------------------
constexpr int kRowWarps = 8, kRowStages = 4, kRowBytes = 128;

struct RowLayout {
    size_t talk, q, tiles, stage, sync, total;
};
__host__ __device__ inline RowLayout row_layout(int G, int dk) {
    RowLayout l;
    l.talk = 0;
    l.q = kTalkBytes;
    l.tiles = (l.q + (size_t)kRowWarps * G * ((dk + 16) / 32) * 32 * 16 + 1023) / 1024 * 1024;
    l.stage = (size_t)2 * G * 16 * kRowBytes;
    l.sync = l.tiles + kRowStages * l.stage;
    l.total = l.sync + kRowStages * 16;
    return l;
}

template <bool FULL, bool CAP>
__global__ void __launch_bounds__(kRowWarps * 32, 1)
    quad_rows_kernel(const QuadArgs a, const __grid_constant__ CUtensorMap keys, const __grid_constant__ CUtensorMap values, int* status) {
    extern __shared__ __align__(1024) unsigned char smem[];
    const int G = FULL ? kQuads : a.G;
    const RowLayout L = row_layout(G, a.dk);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const PortionWork w = portion_work(a, 2 * kRowWarps, 16);
    if (w.lo >= w.hi) return;
    const int* table = a.block_table + (size_t)a.slot_of_seq[w.seq] * a.table_stride;
    unsigned long long* full = reinterpret_cast<unsigned long long*>(smem + L.sync);
    unsigned* left = reinterpret_cast<unsigned*>(smem + L.sync + kRowStages * 8);        // warps that have left a place's tiles, in all
    const int half = G * 16 * kRowBytes;
    auto load = [&](int t, int place, int pg) {
        unsigned char* to = smem + L.tiles + place * L.stage;
        tc5::mbar_expect_tx(full + place, 2 * half);
        tc5::tma_load_4d(to, &keys, 0, t * 16 % a.page, 0, pg, full + place);
        tc5::tma_load_4d(to + half, &values, 0, t * 16 % a.page, 0, pg, full + place);
    };
    auto page_of = [&](int t) { return t < w.hi ? table[t * 16 / a.page] : 0; };
    if (tid == 0) {
        for (int p = 0; p < kRowStages; ++p) {
            tc5::mbar_init(full + p, 1);
            left[p] = 0;
        }
        tc5::mbar_init_fence();
        for (int p = 0; p < kRowStages && w.lo + p < w.hi; ++p) load(w.lo + p, p, page_of(w.lo + p));
    }
    const uint4* talk = reinterpret_cast<const uint4*>(smem + L.talk);
    const int steps = FULL ? 4 : a.dk / 16, iq = w.i0 + 2 * warp, p0 = w.start + iq;     // the warp's queries: rows iq, iq + 1 at p0, p0 + 1
    uint4* qf = reinterpret_cast<uint4*>(smem + L.q) + (size_t)warp * G * ((steps + 1) / 2) * 32;
    stage_talk(reinterpret_cast<uint4*>(smem + L.talk), a, tid, kRowWarps * 32);
    stage_queries<4, FULL>(qf, a, (size_t)w.first + min(iq, w.n_new - 1), max(0, min(2, w.n_new - iq)), lane, 0, 1);
    const WeighConsts consts = weigh_consts(a.scale, a.softcap);
    float begin[kQuads];
    head_starts(begin, a, G, lane);
    float o[kQuads][4][4];
#pragma unroll
    for (int u = 0; u < kQuads; ++u)
#pragma unroll
        for (int d = 0; d < 4; ++d) o[u][d][0] = o[u][d][1] = o[u][d][2] = o[u][d][3] = 0.f;
    __syncthreads();

    const unsigned ring = smem_at(smem + L.tiles);
    const int khead = 16 * kRowBytes;
    for (int t = w.lo; t < w.hi; ++t) {
        const int place = (t - w.lo) % kRowStages, ahead = page_of(t + kRowStages), j0 = t * 16;
        if (!tc5::mbar_wait(full + place, (t - w.lo) / kRowStages & 1)) {
            if (status) *status = tc5::TC5_TIMEOUT_QUADS;
            for (int u = t; u < min(w.hi, t + kRowStages); ++u)        // (no copy is on its way when the block ends)
                tc5::mbar_wait(full + (u - w.lo) % kRowStages, (u - w.lo) / kRowStages & 1);
            return;
        }
        if (j0 + 16 > w.kv_hi) {                               // the sequence's last tile (no other follows): values of rows that
            __syncthreads();                                   // no key has may be anything and count as zero
            unsigned char* v = smem + L.tiles + place * L.stage + half;
            const int from = (w.kv_hi - j0) * (kRowBytes / 16), pieces = 16 * (kRowBytes / 16);
            for (int e = tid; e < G * pieces; e += kRowWarps * 32)
                if (e % pieces >= from) reinterpret_cast<uint4*>(v)[e] = make_uint4(0, 0, 0, 0);
            __syncthreads();
        }
        if (j0 <= p0 + 1) {                                    // the warp's queries see some of the keys
            const unsigned at = ring + place * (unsigned)L.stage;
            unsigned p[2][2][2][2], b[2][2][2][2];
            mixed_tile<4, 2, FULL, CAP>(p, at, kRowBytes, khead, qf, talk, begin, j0 + (lane >> 2), p0, j0 + 15 <= p0, consts, G, steps, lane,
                                        [] {});
            cross(b, p, lane);
            value_tile<FULL>(o, at + half, kRowBytes, khead, b, G, lane);
        }
        __threadfence_block();
        __syncwarp();
        if (lane == 0 && t + kRowStages < w.hi && atomicAdd(left + place, 1u) % kRowWarps == kRowWarps - 1) {
            __threadfence_block();
            tc5::fence_async_smem();
            load(t + kRowStages, place, ahead);
        }
    }
    store_rows(a, o, (size_t)w.first + iq, w.n_new - iq, 0, w.range, G, lane);
}

// ---------------------------------------------------------------------------------------------
// portions, more than 64 lanes: a block of eight warps owns eight queries; a team of two warps owns two queries.  The two take 16 keys
// each up to the mix, hand the mixed weights to each other through shared memory, and take 64 value lanes each.  Tiles of 32 keys,
// keys and values in one buffer each, the next tile's keys on their way from the end of the scores, its values from the end of
// the value product.
// ---------------------------------------------------------------------------------------------
constexpr int kTeamWarps = 8, kTeamKeys = 32, kTeamRow = 256;

struct PortionLayout {
    size_t talk, q, swap, k, v, total;
};
__host__ __device__ inline PortionLayout portion_layout(int G, int dk) {
    PortionLayout l;
    l.talk = 0;
    l.q = kTalkBytes;
    l.swap = l.q + (size_t)(kTeamWarps / 2) * G * ((dk + 16) / 32) * 32 * 16;
    l.k = l.swap + (size_t)kTeamWarps * 16 * 32 * 4;
    l.v = l.k + (size_t)G * kTeamKeys * kTeamRow;
    l.total = l.v + (size_t)G * kTeamKeys * kTeamRow;
    return l;
}

template <int KS, bool FULL, bool CAP>
__global__ void __launch_bounds__(kTeamWarps * 32, 1) quad_portions_kernel(const QuadArgs a) {
    extern __shared__ __align__(1024) unsigned char smem[];
    const int G = FULL ? kQuads : a.G;
    const PortionLayout L = portion_layout(G, a.dk);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, team = warp / 2, part = warp % 2;
    const PortionWork w = portion_work(a, kTeamWarps, kTeamKeys);
    if (w.lo >= w.hi) return;
    const int kv_hi = w.kv_hi, hi = w.hi;
    const int* table = a.block_table + (size_t)a.slot_of_seq[w.seq] * a.table_stride;
    const uint4* talk = reinterpret_cast<const uint4*>(smem + L.talk);
    const int steps = FULL ? KS : a.dk / 16, kp = 2 * steps, vp = FULL ? 16 : a.dv / 8;
    uint4* qf = reinterpret_cast<uint4*>(smem + L.q) + (size_t)team * G * ((steps + 1) / 2) * 32;
    const unsigned ks = smem_at(smem + L.k), vs = smem_at(smem + L.v);
    const int khead = kTeamKeys * kTeamRow;
    const size_t page_elems = (size_t)G * a.page * (a.dk + a.dv);
    const int iq = w.i0 + 2 * team, p0 = w.start + iq;         // the team's queries: rows iq, iq + 1, positions p0, p0 + 1

    auto load_keys = [&](int t, int pg) {
        if (t < hi) {
            const int j0 = t * kTeamKeys, live = kv_hi - j0;
            const __nv_bfloat16* from = a.pool + (size_t)pg * page_elems + (size_t)(j0 % a.page) * a.dk;
            for (int e = tid; e < G * kTeamKeys * kp; e += kTeamWarps * 32) {
                const int c = e % kp, j = e / kp % kTeamKeys, g = e / (kp * kTeamKeys);
                cp16(ks + g * khead + j * kTeamRow + (c ^ (j & 7)) * 16, from + ((size_t)g * a.page + j) * a.dk + c * 8, j < live);
            }
        }
        cp_commit();
    };
    auto load_values = [&](int t, int pg) {
        if (t < hi) {
            const int j0 = t * kTeamKeys, live = kv_hi - j0;
            const __nv_bfloat16* from = a.pool + (size_t)pg * page_elems + (size_t)G * a.page * a.dk + (size_t)(j0 % a.page) * a.dv;
            for (int e = tid; e < G * kTeamKeys * vp; e += kTeamWarps * 32) {
                const int c = e % vp, j = e / vp % kTeamKeys, g = e / (vp * kTeamKeys);
                cp16(vs + g * khead + j * kTeamRow + (c ^ (j & 7)) * 16, from + ((size_t)g * a.page + j) * a.dv + c * 8, j < live);
            }
        }
        cp_commit();
    };
    auto page_of = [&](int t) { return t < hi ? table[t * kTeamKeys / a.page] : 0; };

    {
        const int pg = page_of(w.lo);
        load_keys(w.lo, pg);
        load_values(w.lo, pg);
    }
    int ahead = page_of(w.lo + 1);                             // the page of the next tile to be asked for
    stage_talk(reinterpret_cast<uint4*>(smem + L.talk), a, tid, kTeamWarps * 32);
    stage_queries<KS, FULL>(qf, a, (size_t)w.first + min(iq, w.n_new - 1), max(0, min(2, w.n_new - iq)), lane, part, 2);
    const WeighConsts consts = weigh_consts(a.scale, a.softcap);
    float begin[kQuads];
    head_starts(begin, a, G, lane);
    float o[kQuads][4][4];
#pragma unroll
    for (int u = 0; u < kQuads; ++u)
#pragma unroll
        for (int d = 0; d < 4; ++d) o[u][d][0] = o[u][d][1] = o[u][d][2] = o[u][d][3] = 0.f;

    for (int t = w.lo; t < hi; ++t) {
        cp_wait<1>();
        __syncthreads();                                       // this tile's keys are there
        const int j0 = t * kTeamKeys + part * 16;
        const bool some = j0 <= p0 + 1;                        // the warp's queries see some of its keys
        unsigned b[2][2][2][2];
        auto refill = [&] {                                    // (warps come here from two places: a barrier of its own)
            asm volatile("bar.sync 1, %0;\n" ::"n"(kTeamWarps * 32) : "memory");
            load_keys(t + 1, ahead);
        };
        if (some) {
            unsigned p[2][2][2][2];
            mixed_tile<KS, 2, FULL, CAP>(p, ks + part * 16 * kTeamRow, kTeamRow, khead, qf, talk, begin, j0 + (lane >> 2), p0, j0 + 15 <= p0, consts, G,
                                         steps, lane, refill);
            cross(b, p, lane);
        } else {
            refill();
#pragma unroll
            for (int e = 0; e < 16; ++e) b[e >> 3][e >> 2 & 1][e >> 1 & 1][e & 1] = 0u;
        }
        unsigned* mine = reinterpret_cast<unsigned*>(smem + L.swap) + (size_t)warp * 16 * 32 + lane;
        const unsigned* theirs = reinterpret_cast<unsigned*>(smem + L.swap) + (size_t)(warp ^ 1) * 16 * 32 + lane;
#pragma unroll
        for (int e = 0; e < 16; ++e) mine[e * 32] = b[e >> 3][e >> 2 & 1][e >> 1 & 1][e & 1];
        cp_wait<1>();                                          // the values; the next keys may be on their way
        __syncthreads();
        const unsigned v = vs + part * 128;                    // (a piece's place keeps its upper bit: 64 lanes are 8 pieces)
        const bool own = FULL || part * 64 < a.dv;             // the warp has value lanes
        if (own) value_tile<FULL>(o, v + part * 16 * kTeamRow, kTeamRow, khead, b, G, lane);
#pragma unroll
        for (int e = 0; e < 16; ++e) b[e >> 3][e >> 2 & 1][e >> 1 & 1][e & 1] = theirs[e * 32];
        if (own) value_tile<FULL>(o, v + (part ^ 1) * 16 * kTeamRow, kTeamRow, khead, b, G, lane);
        __syncthreads();                                       // the values and the weights are done with
        load_values(t + 1, ahead);
        ahead = page_of(t + 2);
    }
    store_rows(a, o, (size_t)w.first + iq, w.n_new - iq, part * 64, w.range, G, lane);
}

// ---------------------------------------------------------------------------------------------
// single tokens: a block owns (sequence, range of keys); every warp walks tiles of sixteen keys of its own, with one buffer of
// keys and one of values that are refilled as soon as their product is done, and no barrier between warps before the end.
// The key/value heads 2 p and 2 p + 1 share an accumulator (columns 0 .. 3 and 4 .. 7), the second query's place being empty.
// ---------------------------------------------------------------------------------------------
struct SingleLayout {
    int krow, vrow, warps;
    size_t talk, q, bufs, warp_bytes, total;
};
__host__ __device__ inline SingleLayout single_layout(int G, int dk, int dv) {
    SingleLayout l;
    l.krow = dk > 64 ? 256 : 128;
    l.vrow = dv > 64 ? 256 : 128;
    l.talk = 0;
    l.q = kTalkBytes;
    l.bufs = l.q + (size_t)G * ((dk + 16) / 32) * 32 * 16;
    l.warp_bytes = (size_t)G * 16 * (l.krow + l.vrow);
    const size_t room = (227 * 1024 - l.bufs) / l.warp_bytes;
    l.warps = room > 6 ? 6 : (int)room;
    const size_t sums = 16 * 1024;             // a warp's sums pass through the buffers at the end
    l.total = l.bufs + (l.warps * l.warp_bytes > sums ? l.warps * l.warp_bytes : sums);
    return l;
}

template <int KS, int DT, bool FULL, bool CAP>
__global__ void __launch_bounds__(192, 1) quad_singles_kernel(const QuadArgs a) {
    extern __shared__ __align__(1024) unsigned char smem[];
    const int G = FULL ? kQuads : a.G;
    const SingleLayout L = single_layout(G, a.dk, a.dv);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, threads = L.warps * 32;
    const int seq = blockIdx.x, first = a.cu_seqlens[seq];
    if (a.cu_seqlens[seq + 1] - first != 1) return;            // this kernel serves sequences that bring one token
    const int pos = a.start_pos[seq], kv_hi = pos + 1;
    const int tiles = (kv_hi + 15) / 16, per = tiles_of_range(tiles, a.ranges, kLeastSingle);
    const int lo = blockIdx.y * per, hi = min(tiles, lo + per);
    if (lo >= hi) return;
    const int* table = a.block_table + (size_t)a.slot_of_seq[seq] * a.table_stride;
    const uint4* talk = reinterpret_cast<const uint4*>(smem + L.talk);
    uint4* qf = reinterpret_cast<uint4*>(smem + L.q);
    const int steps = FULL ? KS : a.dk / 16, kp = 2 * steps, vp = FULL ? 2 * DT : a.dv / 8;
    const unsigned ks = smem_at(smem + L.bufs + warp * L.warp_bytes), vs = ks + G * 16 * L.krow;
    const int khead = 16 * L.krow, vhead = 16 * L.vrow;
    const size_t page_elems = (size_t)G * a.page * (a.dk + a.dv);
    auto load_keys = [&](int t, int pg) {
        if (t < hi) {
            const int j0 = t * 16, live = kv_hi - j0;
            const __nv_bfloat16* from = a.pool + (size_t)pg * page_elems + (size_t)(j0 % a.page) * a.dk;
#pragma unroll 8
            for (int e = lane; e < G * 16 * kp; e += 32) {
                const int c = e % kp, j = e / kp % 16, g = e / (kp * 16);
                cp16(ks + g * khead + j * L.krow + (c ^ (j & 7)) * 16, from + ((size_t)g * a.page + j) * a.dk + c * 8, j < live);
            }
        }
        cp_commit();
    };
    auto load_values = [&](int t, int pg) {
        if (t < hi) {
            const int j0 = t * 16, live = kv_hi - j0;
            const __nv_bfloat16* from = a.pool + (size_t)pg * page_elems + (size_t)G * a.page * a.dk + (size_t)(j0 % a.page) * a.dv;
#pragma unroll 8
            for (int e = lane; e < G * 16 * vp; e += 32) {
                const int c = e % vp, j = e / vp % 16, g = e / (vp * 16);
                cp16(vs + g * vhead + j * L.vrow + (c ^ (j & 7)) * 16, from + ((size_t)g * a.page + j) * a.dv + c * 8, j < live);
            }
        }
        cp_commit();
    };
    auto page_of = [&](int t) { return t < hi ? table[t * 16 / a.page] : 0; };
    {
        const int pg = page_of(lo + warp);
        load_keys(lo + warp, pg);
        load_values(lo + warp, pg);
    }
    int ahead = page_of(lo + warp + L.warps);
    stage_talk(reinterpret_cast<uint4*>(smem + L.talk), a, tid, threads);
    stage_queries<KS, FULL>(qf, a, (size_t)first, 1, lane, warp, L.warps);
    const int per_kv = a.H / a.G;
    const WeighConsts consts = weigh_consts(a.scale, a.softcap);
    float begin[kQuads];
#pragma unroll
    for (int u = 0; u < kQuads; ++u)
        begin[u] = weigh_start(a.softcap, a.head_bias && u < G && (lane & 3) < per_kv ? a.head_bias[u * per_kv + (lane & 3)] : 0.f);
    float o[kQuads / 2][DT][4];
#pragma unroll
    for (int p = 0; p < kQuads / 2; ++p)
#pragma unroll
        for (int d = 0; d < DT; ++d) o[p][d][0] = o[p][d][1] = o[p][d][2] = o[p][d][3] = 0.f;
    __syncthreads();
    for (int t = lo + warp; t < hi; t += L.warps) {
        const int pg = ahead;
        ahead = page_of(t + 2 * L.warps);
        cp_wait<1>();
        __syncwarp();
        unsigned p[1][2][2][2];
        mixed_tile<KS, 1, FULL, CAP>(p, ks, L.krow, khead, qf, talk, begin, t * 16 + (lane >> 2), pos, t * 16 + 15 <= pos, consts, G, steps, lane, [&] {
            __syncwarp();
            load_keys(t + L.warps, pg);
        });
        cp_wait<1>();
        __syncwarp();
        const unsigned at = vs + ((lane & 7) + (lane >> 4) * 8) * L.vrow, turn = ((lane >> 3 & 1) ^ (lane & 7)) * 16;
#pragma unroll
        for (int u = 0; u < kQuads; ++u) {
            if (FULL || u < G) {
                const bool mine = (lane >= 16) == (u & 1);
                const unsigned b0 = mine ? p[0][u >> 2][u >> 1 & 1][0] : 0u, b1 = mine ? p[0][u >> 2][u >> 1 & 1][1] : 0u;
#pragma unroll
                for (int d = 0; d < DT; ++d) {
                    if (FULL || d * 16 < a.dv) {
                        unsigned f[4];
                        ldsm_x4_trans(f, at + u * vhead + (turn ^ (d * 32)));
                        mma_bf16(o[u >> 1][d], f, b0, b1);
                    }
                }
            }
        }
        __syncwarp();
        load_values(t + L.warps, pg);
    }
    cp_wait<0>();
    __syncthreads();
    // the warps' sums, in the order of the warps: through the buffers, which are done with
    float* sums = reinterpret_cast<float*>(smem + L.bufs);
    constexpr int kFloats = kQuads / 2 * DT * 4;               // a lane's
    for (int w = 1; w < L.warps; ++w) {
        if (warp == w) {
#pragma unroll
            for (int e = 0; e < kFloats; ++e) sums[e * 32 + lane] = o[e / 4 / DT][e / 4 % DT][e & 3];
        }
        __syncthreads();
        if (warp == 0) {
#pragma unroll
            for (int e = 0; e < kFloats; ++e) o[e / 4 / DT][e / 4 % DT][e & 3] += sums[e * 32 + lane];
        }
        __syncthreads();
    }
    if (warp != 0) return;
    const int HD = a.H * a.dv;
#pragma unroll
    for (int p = 0; p < kQuads / 2; ++p)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int n = 2 * (lane & 3) + e, h = n & 3, g = 2 * p + (n >> 2);
            if (g >= G || h >= per_kv) continue;
            const size_t at = (size_t)first * HD + (g * per_kv + h) * a.dv;
#pragma unroll
            for (int d = 0; d < DT; ++d)
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const int lanev = d * 16 + (lane >> 2) + 8 * r;
                    if (lanev < a.dv) {
                        if (a.ranges > 1) a.partial[(size_t)blockIdx.y * a.n_tokens * HD + at + lanev] = o[p][d][2 * r + e];
                        else a.out[at + lanev] = __float2bfloat16_rn(o[p][d][2 * r + e]);
                    }
                }
        }
}

// out[n, :] = the ranges' partial outputs added in order: as many as the row's block of queries has; rows of no sequence get zeros
__global__ void add_quad_ranges_kernel(const QuadArgs a, int bq, int keys, int least) {
    const int n = blockIdx.x, HD = a.H * a.dv, seq = a.token_seq[n];
    int used = 0;
    if (seq >= 0) {
        const int first = a.cu_seqlens[seq], n_new = a.cu_seqlens[seq + 1] - first, i0 = (n - first) / bq * bq;
        const int tiles = (a.start_pos[seq] + min(i0 + bq, n_new) + keys - 1) / keys, per = tiles_of_range(tiles, a.ranges, least);
        used = (tiles + per - 1) / per;
    }
    for (int e = threadIdx.x * 4; e < HD; e += blockDim.x * 4) {
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int r = 0; r < used; ++r) {
            const float4 v = *reinterpret_cast<const float4*>(a.partial + ((size_t)r * a.n_tokens + n) * HD + e);
            s.x += v.x;
            s.y += v.y;
            s.z += v.z;
            s.w += v.w;
        }
        *reinterpret_cast<uint2*>(a.out + (size_t)n * HD + e) = make_uint2(pack_bf16(s.x, s.y), pack_bf16(s.z, s.w));
    }
}

// Whether these kernels take a shape (bfloat16 alone): at most eight key/value heads with at most four query heads each.
BLM_API int blm_attention_quads_takes(int H, int G, int dk, int dv, int page) {
    if (H < 1 || G < 1 || H % G || G > kQuads || H / G > 4) return 0;
    return dk % 16 == 0 && dk >= 16 && dk <= 128 && dv % 8 == 0 && dv >= 8 && dv <= 128 && page % 32 == 0;
}

// Query rows of a portion block.
BLM_API int blm_attention_quads_rows(int dk, int dv) { return dv > 64 || dk > 64 ? kTeamWarps : 2 * kRowWarps; }

template <typename K>
static int allow_smem(K kernel, size_t smem) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    return e == cudaSuccess ? BLM_OK : blm_fail(BLM_CUDA_ERROR, "attention_quads: %s", cudaGetErrorString(e));
}

BLM_API int blm_attention_quads(const void* q, const void* pool, const int* block_table, int table_stride, const int* cu_seqlens,
                                const int* slot_of_seq, const int* start_pos, const int* token_seq, const float* talk,
                                const float* head_bias, void* out, float* partial, int n_tokens, int n_seqs, int max_q_len, int H, int G,
                                int dk, int dv, int page, long long n_pages, int ranges, float scale, float softcap, int* status,
                                cudaStream_t stream) {
    if (n_tokens == 0 || n_seqs == 0) return BLM_OK;
    BLM_REQUIRE(blm_attention_quads_takes(H, G, dk, dv, page) && max_q_len > 0, "attention_quads: %d heads on %d, %d + %d lanes", H, G, dk, dv);
    BLM_REQUIRE(ranges >= 1 && ranges <= 65535 && (ranges == 1 || partial != nullptr), "attention_quads: several key ranges need a workspace");
    BLM_REQUIRE((((size_t)q | (size_t)pool | (size_t)out | (size_t)partial) & 15) == 0, "attention_quads: tensors start at multiples of 16 bytes");
    QuadArgs a = {(const __nv_bfloat16*)q, (const __nv_bfloat16*)pool, block_table, table_stride, cu_seqlens, slot_of_seq, start_pos, token_seq,
                  talk, head_bias, (__nv_bfloat16*)out, partial, n_tokens, n_seqs, 1, H, G, dk, dv, page, ranges, scale, softcap};
    // the instances without tests of the sizes: eight key/value heads, 64 or 128 lanes
    const bool full = G == kQuads && (dk == 64 || dk == 128) && (dv == 64 || dv == 128);
    int bq = 1, keys = 16;
    if (max_q_len == 1) {
        const SingleLayout l = single_layout(G, dk, dv);
        auto pick = [&](auto cap) {
            constexpr bool CAP = decltype(cap)::value;
            return !full ? quad_singles_kernel<8, 8, false, CAP>
                   : dk == 64 ? (dv == 64 ? quad_singles_kernel<4, 4, true, CAP> : quad_singles_kernel<4, 8, true, CAP>)
                              : (dv == 64 ? quad_singles_kernel<8, 4, true, CAP> : quad_singles_kernel<8, 8, true, CAP>);
        };
        auto k = softcap > 0.f ? pick(std::true_type()) : pick(std::false_type());
        BLM_REQUIRE(l.warps >= 1, "attention_quads: shared memory");
        if (int rc = allow_smem(k, l.total)) return rc;
        k<<<dim3(n_seqs, ranges), l.warps * 32, l.total, stream>>>(a);
    } else {
        const bool wide = dv > 64 || dk > 64;
        bq = blm_attention_quads_rows(dk, dv);
        keys = wide ? kTeamKeys : 16;
        a.q_tiles = (max_q_len + bq - 1) / bq;
        const long long blocks = (long long)n_seqs * a.q_tiles * ranges;
        BLM_REQUIRE(blocks <= 0x7fffffffLL, "attention_quads: grid too large");
        if (wide) {
            const PortionLayout l = portion_layout(G, dk);
            auto pick = [&](auto cap) {
                constexpr bool CAP = decltype(cap)::value;
                return !full || dv == 64 ? quad_portions_kernel<8, false, CAP>
                                         : (dk == 64 ? quad_portions_kernel<4, true, CAP> : quad_portions_kernel<8, true, CAP>);
            };
            auto k = softcap > 0.f ? pick(std::true_type()) : pick(std::false_type());
            BLM_REQUIRE(l.total <= 227 * 1024, "attention_quads: shared memory");
            if (int rc = allow_smem(k, l.total)) return rc;
            k<<<(unsigned)blocks, kTeamWarps * 32, l.total, stream>>>(a);
        } else {
            const RowLayout l = row_layout(G, dk);
            auto k = softcap > 0.f ? (full ? quad_rows_kernel<true, true> : quad_rows_kernel<false, true>)
                                   : (full ? quad_rows_kernel<true, false> : quad_rows_kernel<false, false>);
            // the pages as [page][key/value head][row][lane]; a box is sixteen rows of every head, lanes that are not there read as zero
            const long long page_bytes = (long long)G * page * (dk + dv) * 2;
            CUtensorMap km, vm;
            BLM_REQUIRE(n_pages > 0 &&
                            tc5::make_map_4d(&km, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, a.pool, {dk, page, G, n_pages},
                                             {dk * 2LL, page * dk * 2LL, page_bytes}, {64, 16, G, 1}, CU_TENSOR_MAP_SWIZZLE_128B) &&
                            tc5::make_map_4d(&vm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, a.pool + (size_t)G * page * dk, {dv, page, G, n_pages},
                                             {dv * 2LL, page * dv * 2LL, page_bytes}, {64, 16, G, 1}, CU_TENSOR_MAP_SWIZZLE_128B),
                        "attention_quads: no tensor map for %lld pages of %d heads of %d + %d lanes", n_pages, G, dk, dv);
            BLM_REQUIRE(l.total <= 227 * 1024, "attention_quads: shared memory");
            if (int rc = allow_smem(k, l.total)) return rc;
            k<<<(unsigned)blocks, kRowWarps * 32, l.total, stream>>>(a, km, vm, status);
        }
    }
    if (int rc = blm_check_launch("attention_quads")) return rc;
    if (ranges == 1) return BLM_OK;
    add_quad_ranges_kernel<<<n_tokens, 256, 0, stream>>>(a, bq, keys, max_q_len == 1 ? kLeastSingle : 256 / keys);
    return blm_check_launch("attention_quads (ranges)");
}
