// Long prompts of the state-space scan, sixty-four tokens at a time on tcgen05.
//
// The chunks of sixteen tokens (scan_chunks.cu) are a chain of 128 links for a prompt of 2,048 tokens: 150 to 158 us for 64 heads of 128
// x 64 (eight to one groups that share B and C), whose multiply-adds alone take 58 on the fp32 units.  Here a chunk has 64 tokens, its products run on the tensor cores with every float as three bfloat16 numbers (tcgen05.cuh: 24 bits, six products, sums
// in float32), and a sequence (beyond 4,096 tokens each such segment of it, one after another) is cut into four groups of chunks that
// run side by side: 119 to 125 us.  With P(i..j) the product of the
// decays of the tokens i..j and S the state in front of a chunk:
//     out_j  = P(0..j) S^T C_j + sum_(i <= j) A_ji x_i,     A_ji = (C_j . B_i) P(i+1..j) dt_i  (+ D on the diagonal)
//     S'     = P(0..63) S + Z,     Z = sum_j (P(j+1..63) dt_j B_j) x_j^T
// Every factor is a product of decays, never a quotient of two: nothing overflows however strong a decay is.  Relative errors against 64
// bits, 2,048 tokens of 8 heads that forget within some ten tokens, this / chunks of sixteen / the walk: 1.6e-7 / 1.4e-7 / 1.3e-7, of
// one sign 1.2e-7 / 1.0e-7 / 1.0e-7 (the tensor cores cut their sums off); that forget slowly 1.9e-6 / 1.9e-6 / 2.0e-6.
//
// Three launches.  (1) What does not depend on the state is formed for all chunks at once and left as the tensor cores read it: C,
// B and the 64 x 64 matrices A, split into bfloat16 parts, in the 128-byte swizzle (29 us).  (2) Every group but a segment's last is
// run from an empty state: what it adds to the state (28); the first one also copies the state that the segment starts from.  (3)
// Every group folds the groups in front of it into that copy and runs (59); the last one writes the sequence's state.  The state
// itself is not read in this launch, whose groups run in no order: for an even number of tokens it is what the last group writes (a
// segment of one group reads and writes its own).  A block owns a group and two neighbouring heads that share B and C, whose 2 x 64 columns are the lanes of
// tensor memory.  S lives in registers (a lane a column, half of the rows a warp); its parts, the operand of the read-out, are
// written to tensor memory, and so are x's.
// A chunk takes 10,000 clocks, of which the 120 tcgen05.mma, issued one every 40, take 4,800; the rest are the hand-overs between them
// (x's parts, the reading of A x, of Z and of the output).  That is no faster a chain than sixteen tokens at a time, so only
// long sequences of enough heads gain (kernels.py has the border and both sides' times), and decays per row, whose 64 x 64
// matrices and decayed rows are each head's own (119 us to form them for 32 heads of 128 x 128), do not at all.
#include <algorithm>

#include "tcgen05.cuh"

BLM_API const char* blm_scan_long_last_error() { return g_blm_error; }

using namespace tc5;

constexpr int kT = 64;            // tokens of a chunk
constexpr int kSegment = 64;      // chunks of a segment: a sequence is run segment by segment
constexpr int kGroups = 4;        // groups of a segment: its chunks in even parts
constexpr int kTile = kT * 128;   // bytes of 64 rows of 64 bfloat16 numbers

constexpr int NR = 128, H = NR / 64;      // rows of the state as it lies, and rows of 128 bytes that its parts take

__device__ __forceinline__ float softplus_r(float v) { return fmaxf(v, 0.f) + log1pf(expf(-fabsf(v))); }

// Sequences of `least` or more new tokens are run, in segments of kSegment chunks one after another: what a pass needs of scratch
// does not grow with a sequence, and where a segment begins depends on its own sequence alone, so a sequence has the bits it has alone.
// Chunk c of sequence s has the index cu[s] / 64 + s + c: distinct, and below n_tokens / 64 + n_seqs (a step of one sequence: c).  A pass runs
// the segments whose first chunk has an index from `from` up to from + count; their chunks have indexes below from + count + a
// segment's chunks - 1.  Each has a slot of its own for its groups' sums: sequences begin `gap` indexes apart at least, so every `gap`
// indexes hold the beginning of one at most; where sequences have several segments a pass counts no more than kSegment indexes,
// which hold one at most that is not its sequence's first (slot 0; `later`: there may be both).
struct Chunks {
    const int* cu;
    int n_seqs, least;
    int from, count, gap, later;
};
static long long chunk_bound(int n_tokens, int n_seqs) { return (long long)n_tokens / kT + n_seqs; }
__device__ __forceinline__ int chunk_base(const Chunks& ch, int seq) { return ch.n_seqs > 1 ? ch.cu[seq] / kT + seq : 0; }

// The sequence and chunk of the pass's chunk `idx`; false: there is none.  All threads of the block call it.
__device__ __forceinline__ bool find_chunk(int idx, const Chunks& ch, int* found, int& seq, int& chunk) {
    idx += ch.from;
    if (threadIdx.x == 0) found[0] = -1;
    __syncthreads();
    for (int s = threadIdx.x; s < ch.n_seqs; s += blockDim.x) {
        const int n = ch.cu[s + 1] - ch.cu[s], c = idx - chunk_base(ch, s);
        if (n < ch.least || c < 0 || c >= (n + kT - 1) / kT) continue;
        const int begin = idx - c % kSegment;
        if (begin >= ch.from && begin < ch.from + ch.count) {
            found[0] = s;
            found[1] = c;
        }
    }
    __syncthreads();
    seq = found[0];
    chunk = found[1];
    return seq >= 0;
}

// The sequence and the first chunk of the pass's segment in a slot; false: there is none.  All threads of the block call it.
__device__ __forceinline__ bool find_segment(int slot, const Chunks& ch, int* found, int& seq, int& chunk) {
    if (threadIdx.x == 0) found[0] = -1;
    __syncthreads();
    for (int s = threadIdx.x; s < ch.n_seqs; s += blockDim.x) {
        const int n = ch.cu[s + 1] - ch.cu[s], ahead = max(0, ch.from - chunk_base(ch, s));
        if (n < ch.least) continue;
        const int c = (ahead + kSegment - 1) / kSegment * kSegment, at = chunk_base(ch, s) + c - ch.from;
        if (c < (n + kT - 1) / kT && at < ch.count && slot == (c > 0 ? 0 : ch.later + at / ch.gap)) {
            found[0] = s;
            found[1] = c;
        }
    }
    __syncthreads();
    seq = found[0];
    chunk = found[1];
    return seq >= 0;
}

struct RowsIn {                    // a column range of a float32 [N, *] tensor
    const float* p;
    long long stride;
    int col0;
};

// Scratch: pieces of one kind of every chunk and head, or unit (the heads that share B and C), beside one another.
//   rows   [chunk][unit][C, B][3 parts][NR / 64][64 tokens][64 rows of the state]      bfloat16
//   mats   [chunk][head][3][64 j][64 i]                                                bfloat16
//   nums   [chunk][head][kNums]: 64 factors of the read-out, 64 of what a token writes, the chunk's decay
//   sums   [slot][kGroups - 1][head][column][NR], decays [slot][kGroups - 1][head]
//   firsts [slot][head][column][NR]: the state in front of the segment
constexpr int kNums = 132;
struct Scratch {
    unsigned char *rows, *mats;
    float *nums, *sums, *firsts, *decays;
};
struct Sizes {
    long long rows, mats, nums, sums, firsts, decays;  // bytes
    long long all() const { return rows + mats + nums + sums + firsts + decays; }
};
static Sizes sizes_of(int units, int heads, int dv, long long chunks, long long slots) {
    const long long groups = slots * (kGroups - 1);
    return {chunks * units * 6 * H * kTile, chunks * heads * 3 * kTile, chunks * heads * kNums * 4, groups * heads * dv * NR * 4,
            slots * heads * dv * NR * 4, groups * heads * 4};
}
static Scratch scratch_at(float* base, const Sizes& s) {
    unsigned char *mats = reinterpret_cast<unsigned char*>(base) + s.rows, *nums = mats + s.mats, *sums = nums + s.nums, *firsts = sums + s.sums;
    return {mats - s.rows, mats, (float*)nums, (float*)sums, (float*)firsts, (float*)(firsts + s.firsts)};
}

// where row (8 a multiple of 4) `c` of token t lies in a tile of rows of 128 bytes
__device__ __forceinline__ int swizzled(int t, int c) { return t * 128 + (((c >> 3) ^ (t & 7)) << 4) + (c & 7) * 2; }

// four values of a row into the three parts' tiles, `part` bytes apart
__device__ __forceinline__ void store_parts(unsigned char* to, size_t part, float4 v) {
    uint2 p1, p2, p3;
    split3(v.x, v.y, p1.x, p2.x, p3.x);
    split3(v.z, v.w, p1.y, p2.y, p3.y);
    *reinterpret_cast<uint2*>(to) = p1;
    *reinterpret_cast<uint2*>(to + part) = p2;
    *reinterpret_cast<uint2*>(to + 2 * part) = p3;
}

// a number from its three parts
__device__ __forceinline__ float joined(const unsigned char* at, int part) {
    float w = 0.f;
#pragma unroll
    for (int l = 0; l < 3; ++l) w += __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(at + l * part));
    return w;
}

// ---------------------------------------------------------------------------------------------
// (1) the state-space scan: B and C are shared by the heads of a group and the decay is one number a head and token.  A block per
// (chunk, group, sixteen heads of it).  Products of decays by blocks of eight tokens: what is behind i in its block, whole blocks, what is in front of j.
// ---------------------------------------------------------------------------------------------
struct SsmPrepArgs {
    RowsIn x, dt;                  // x names the tensor; B at b_col0, C at c_col0
    int b_col0, c_col0;
    const float *dt_bias, *A_log, *D;
    Chunks ch;
    int heads, groups, N;          // of all; this pass: `units` groups from group0 on
    int group0, units;
    Scratch s;
};
constexpr int kPrepHeads = 16;     // heads of a block, which forms C . B for itself (one group of 64 heads, 2,048 tokens: 153 us with a block for all)
constexpr int kPrepThreads = 512;
constexpr int kPrepSmem = (2 * kT * (NR + 4) + kT * (kT + 1) + kPrepHeads * (3 * kT + 8)) * 4;

__global__ void __launch_bounds__(kPrepThreads, 2) long_prep_kernel(const SsmPrepArgs a) {
    constexpr int NS = NR + 4;
    extern __shared__ __align__(16) float sm[];
    float *Bs = sm, *Cs = sm + kT * NS, *cb = Cs + kT * NS, *dts = cb + kT * (kT + 1), *decs = dts + kPrepHeads * kT, *suf = decs + kPrepHeads * kT,
          *tot = suf + kPrepHeads * kT;
    __shared__ int found[2];
    const int tid = threadIdx.x, g = a.group0 + blockIdx.y, per = a.heads / a.groups;
    int seq, chunk;
    if (!find_chunk(blockIdx.x, a.ch, found, seq, chunk)) return;
    const int first = a.ch.cu[seq] + chunk * kT, nt = min(kT, a.ch.cu[seq + 1] - first);
    {   // all loads on their way at once (a place that is not there is read from one that is)
        constexpr int kStep = kPrepThreads / NR, kMine = kT / kStep;
        const int n = tid % NR, t0 = tid / NR;
        const float* row = a.x.p + (size_t)first * a.x.stride + (size_t)g * a.N + min(n, a.N - 1);
        float b[kMine], c[kMine];
#pragma unroll
        for (int x = 0; x < kMine; ++x) {
            const size_t at = (size_t)min(t0 + x * kStep, nt - 1) * a.x.stride;
            b[x] = row[at + a.b_col0];
            c[x] = row[at + a.c_col0];
        }
#pragma unroll
        for (int x = 0; x < kMine; ++x) {
            const int t = t0 + x * kStep;
            const bool on = t < nt && n < a.N;
            Bs[t * NS + n] = on ? b[x] : 0.f;
            Cs[t * NS + n] = on ? c[x] : 0.f;
        }
    }
    __syncthreads();
    unsigned char* rows = a.s.rows + ((size_t)blockIdx.x * a.units + blockIdx.y) * 6 * H * kTile;
    for (int e = tid; blockIdx.z == 0 && e < 2 * kT * (NR / 4); e += kPrepThreads) {
        const int n = e % (NR / 4) * 4, t = e / (NR / 4) % kT, which = e / (kT * NR / 4);      // q (C), then k (B)
        const float4 v = *reinterpret_cast<const float4*>((which ? Bs : Cs) + t * NS + n);
        store_parts(rows + (which * 3 * H + n / 64) * kTile + swizzled(t, n % 64), (size_t)H * kTile, v);
    }
    {
        const int tj = tid >> 4, ti = tid & 15;
        float s[2][4] = {}, part[2][4] = {};   // (32 rows at a time: one chain of 128 multiply-adds lost a bit)
#pragma unroll 4
        for (int n = 0; n < NR; n += 4) {
            float4 c4[2], b4[4];
#pragma unroll
            for (int x = 0; x < 2; ++x) c4[x] = *reinterpret_cast<const float4*>(Cs + (tj + 32 * x) * NS + n);
#pragma unroll
            for (int y = 0; y < 4; ++y) b4[y] = *reinterpret_cast<const float4*>(Bs + (ti + 16 * y) * NS + n);
#pragma unroll
            for (int x = 0; x < 2; ++x)
#pragma unroll
                for (int y = 0; y < 4; ++y) {
                    part[x][y] = fmaf(c4[x].x, b4[y].x, part[x][y]);
                    part[x][y] = fmaf(c4[x].y, b4[y].y, part[x][y]);
                    part[x][y] = fmaf(c4[x].z, b4[y].z, part[x][y]);
                    part[x][y] = fmaf(c4[x].w, b4[y].w, part[x][y]);
                }
            if (n % 32 == 28) {
#pragma unroll
                for (int x = 0; x < 2; ++x)
#pragma unroll
                    for (int y = 0; y < 4; ++y) {
                        s[x][y] += part[x][y];
                        part[x][y] = 0.f;
                    }
            }
        }
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int y = 0; y < 4; ++y) cb[(tj + 32 * x) * (kT + 1) + ti + 16 * y] = s[x][y];
    }
    {
        const int h0 = blockIdx.z * kPrepHeads, nh = min(kPrepHeads, per - h0);
        __syncthreads();
        for (int e = tid; e < nh * kT; e += kPrepThreads) {
            const int h = g * per + h0 + e / kT, t = e % kT;
            float dt = 0.f, dec = 1.f;         // a token beyond the chunk's end changes nothing
            if (t < nt) {
                dt = softplus_r(a.dt.p[(size_t)(first + t) * a.dt.stride + a.dt.col0 + h] + a.dt_bias[h]);
                dec = expf(-expf(a.A_log[h]) * dt);
            }
            dts[e] = dt;
            decs[e] = dec;
        }
        __syncthreads();
        for (int e = tid; e < nh * 8; e += kPrepThreads) {
            float p = 1.f;
#pragma unroll
            for (int t = 7; t >= 0; --t) {
                suf[e * 8 + t] = p;            // the tokens behind t, up to the block's end
                p *= decs[e * 8 + t];
            }
            tot[e] = p;
        }
        __syncthreads();
        for (int e = tid; e < nh * 8; e += kPrepThreads) {
            const int hh = e >> 3, b = e & 7;
            float* nums = a.s.nums + ((size_t)blockIdx.x * a.units * per + blockIdx.y * per + h0 + hh) * kNums;
            float before = 1.f, behind = 1.f;
            for (int x = 0; x < b; ++x) before *= tot[hh * 8 + x];
            for (int x = b + 1; x < 8; ++x) behind *= tot[hh * 8 + x];
            if (b == 7) nums[128] = before * tot[e];
#pragma unroll
            for (int t = 0; t < 8; ++t) {
                before *= decs[e * 8 + t];
                nums[b * 8 + t] = before;
                nums[64 + b * 8 + t] = suf[e * 8 + t] * behind * dts[e * 8 + t];
            }
        }
        // A: a thread two neighbouring i and eight j
        const int i = (tid & 31) * 2, jb = tid >> 5 & 7;
        for (int hh = tid >> 8; hh < nh; hh += kPrepThreads / 256) {
            const int h = g * per + h0 + hh;
            unsigned char* mat = a.s.mats + ((size_t)blockIdx.x * a.units * per + blockIdx.y * per + h0 + hh) * 3 * kTile;
            const float* dec = decs + hh * kT;
            float p0 = suf[hh * kT + i], p1 = suf[hh * kT + i + 1];
            for (int x = (i >> 3) + 1; x < jb; ++x) {
                p0 *= tot[hh * 8 + x];
                p1 *= tot[hh * 8 + x];
            }
            const float d0 = dts[hh * kT + i], d1 = dts[hh * kT + i + 1], diag = a.D[h];
            const bool own = jb == i >> 3;
            if (own) p0 = p1 = 1.f;
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const int j = jb * 8 + e;
                if (!own || j > i) p0 *= dec[j];
                if (!own || j > i + 1) p1 *= dec[j];
                const float* c = cb + j * (kT + 1) + i;
                const float v0 = i > j ? 0.f : c[0] * p0 * d0 + (i == j ? diag : 0.f), v1 = i + 1 > j ? 0.f : c[1] * p1 * d1 + (i + 1 == j ? diag : 0.f);
                unsigned w1, w2, w3;
                split3(v0, v1, w1, w2, w3);
                unsigned char* to = mat + swizzled(j, i);
                *reinterpret_cast<unsigned*>(to) = w1;
                *reinterpret_cast<unsigned*>(to + kTile) = w2;
                *reinterpret_cast<unsigned*>(to + 2 * kTile) = w3;
            }
        }
    }
}

// ---------------------------------------------------------------------------------------------
// (2) and (3): a group of chunks
//
// Warp 0 brings the chunk's operands (three barriers: each is asked for as soon as its product of the chunk before is done), one
// thread of warp 1 issues the products, warps 2 to 9 keep the state, warps 10 to 13 split x and write the output.
// A value that is not finite must not reach earlier tokens through a matrix's zeros, so it is taken out of x and joins the later
// tokens' outputs and the state by itself.  An infinite state, B or C has parts that are not numbers, and so is what it reaches, where the
// walk's multiply-adds may leave an infinity; it reaches no more than there.
// ---------------------------------------------------------------------------------------------
struct RunArgs {
    RowsIn v;
    Scratch s;
    Chunks ch;
    const int *slot_of_seq, *start_pos;
    int units, per_unit;           // units of `rows` a chunk, heads of a unit
    int head0, heads;              // this pass: heads from head0 on
    int dv;
    float* y;
    long long y_stride;
    float* state;
    long long slot_stride, copy_stride, state_off;
    int* status;
};

constexpr int kXSlots = 2;        // chunks of x in shared memory
constexpr int kSWarps = 8, kXWarps = 4, kRunThreads = (2 + kSWarps + kXWarps) * 32;
constexpr int kRunSmem = 1024 + 6 * H * kTile + 6 * kTile + kXSlots * kT * 128 * 4 + 256;

// 32 tokens of x (times a factor a token, which the lane of its number has) into their parts in tensor memory; true: there was a value
// that is not finite.
template <bool SCALE>
__device__ __forceinline__ bool put_x(const float* x, unsigned to, float f) {
    unsigned most = 0;
#pragma unroll 1
    for (int t = 0; t < 32; t += 16) {
        float v[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = x[(t + e) * 128];
        unsigned m = 0;
#pragma unroll
        for (int e = 0; e < 16; ++e) m = max(m, __float_as_uint(v[e]) & 0x7fffffffu);
        if (m >= 0x7f800000u) {
#pragma unroll
            for (int e = 0; e < 16; ++e) v[e] = isfinite(v[e]) ? v[e] : 0.f;
        }
        most = max(most, m);
        if (SCALE) {
#pragma unroll
            for (int e = 0; e < 16; ++e) v[e] *= __shfl_sync(0xffffffffu, f, t + e);
        }
        unsigned p[3][8];
#pragma unroll
        for (int e = 0; e < 8; ++e) split3(v[2 * e], v[2 * e + 1], p[0][e], p[1][e], p[2][e]);
#pragma unroll
        for (int l = 0; l < 3; ++l) tmem_st8(to + l * 32 + t / 2, p[l]);
    }
    return most >= 0x7f800000u;
}

template <bool SUMS>
__global__ void __launch_bounds__(kRunThreads, 1) long_run_kernel(const RunArgs a) {
    constexpr int kHalf = NR / 2;
    constexpr unsigned kD = 0, kParts = 128, kX = 320, kOut = 416;         // tensor memory: D, the state's parts, x's parts, the output
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* q_img = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    unsigned char* k_img = q_img + 3 * H * kTile;
    unsigned char* a_img = k_img + 3 * H * kTile;
    float* xs = reinterpret_cast<float*>(a_img + 6 * kTile);   // [kXSlots][64][128]
    unsigned long long* bars = reinterpret_cast<unsigned long long*>(xs + kXSlots * kT * 128);
    unsigned long long *a_full = bars, *q_full = bars + 1, *k_full = bars + 2, *x_full = bars + 3, *xs_full = bars + 4, *s_full = bars + 5,
                       *intra_read = bars + 6, *out_read = bars + 7, *intra_done = bars + 8, *out_done = bars + 9, *upd_done = bars + 10,
                       *d_read = bars + 11, *raw_full = bars + 12;
    unsigned* tmem_slot = reinterpret_cast<unsigned*>(bars + 13);
    int* odd = reinterpret_cast<int*>(tmem_slot + 2);                       // [2][4]: a warp of columns has values that are not finite in the chunk
    int* found = odd + 8;                      // (not beside them: shared memory then begins where addresses are known at compile time)

    const int h = blockIdx.x * 2, slot = blockIdx.y / kGroups, group = blockIdx.y % kGroups;
    int seq, begin;                            // the segment's sequence, and its first chunk
    if (!find_segment(slot, a.ch, found, seq, begin)) return;
    const int n_new = a.ch.cu[seq + 1] - a.ch.cu[seq];
    const int length = min(kSegment, (n_new + kT - 1) / kT - begin), size = (length + kGroups - 1) / kGroups, lo = group * size;      // of the segment
    if (lo >= length || (SUMS && lo + size >= length)) return;
    const int n = min(size, length - lo), base = chunk_base(a.ch, seq) - a.ch.from + begin + lo;
    const int first = a.ch.cu[seq] + (begin + lo) * kT, rest = n_new - (begin + lo) * kT;      // the group's first token, and how many the sequence has from there on
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        mbar_init(a_full, 1);
        mbar_init(q_full, 1);
        mbar_init(k_full, 1);
        mbar_init(x_full, 4);
        mbar_init(xs_full, SUMS ? 4 : 8);
        mbar_init(s_full, 8);
        mbar_init(intra_read, 4);
        mbar_init(out_read, 4);
        mbar_init(intra_done, 1);
        mbar_init(out_done, 1);
        mbar_init(upd_done, 1);
        mbar_init(d_read, 8);
        for (int i = 0; i < kXSlots; ++i) mbar_init(raw_full + i, 32);
        mbar_init_fence();
    }
    if (warp == 1) tmem_alloc(tmem_slot, 512);
    fence_before();
    __syncthreads();
    fence_after();
    const unsigned tmem = *tmem_slot;
    bool ok = true;
    auto wait = [&](unsigned long long* bar, unsigned phase) {
        if (ok && !mbar_wait(bar, phase & 1)) {
            ok = false;
            if (lane == 0) atomicCAS(a.status, TC5_OK, TC5_TIMEOUT_SCAN_LONG);
        }
        return ok;
    };
    auto arrive = [&](unsigned long long* bar) {
        __syncwarp();
        if (lane == 0) mbar_arrive(bar);
    };
    const int hl = h + (warp >> 1 & 1);             // the head of a warp of columns: quarters 0 and 1, 2 and 3
    auto nums_of = [&](int c) { return a.s.nums + ((size_t)(base + c) * a.heads + hl) * kNums; };

    if (warp == 0) {
        // ---------------- the loads ----------------
        const unsigned rows_bytes = 3 * H * kTile;
        auto copy = [&](unsigned char* dst, const unsigned char* src, unsigned bytes, unsigned long long* bar) {
            if (lane == 0) {
                mbar_expect_tx(bar, bytes);
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(smem_u32(dst)), "l"(src),
                             "r"(bytes), "r"(smem_u32(bar))
                             : "memory");
            }
            __syncwarp();
        };
        // x's rows of a chunk; what is not there comes as zeros
        const float* v = a.v.p + a.v.col0 + (size_t)(a.head0 + h) * a.dv;
        const int wide = a.dv;
        const bool vec = (((size_t)v | (size_t)a.v.stride * 4) & 15) == 0 && wide % 4 == 0;
        const int in4 = (lane & 15) * 4, at4 = (lane >> 4) * a.dv + in4;
        auto bring_x = [&](int c) {
            float* to = xs + c % kXSlots * kT * 128;
            const int t0 = first + c * kT, nt = min(kT, rest - c * kT);
            if (vec) {
                const float* src = v + (size_t)t0 * a.v.stride + at4;
#pragma unroll 4
                for (int t = 0; t < kT; ++t, src += a.v.stride) {
                    const int on = t < nt && in4 < wide ? 16 : 0;
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem_u32(to + t * 128 + lane * 4)), "l"(on ? src : a.s.nums), "r"(on) : "memory");
                }
            } else {
                for (int e = lane; e < kT * 128; e += 32) {
                    const int t = e >> 7, i = e & 63, on = t < nt && i < wide ? 4 : 0;
                    const float* src = v + (size_t)(t0 + t) * a.v.stride + i + (e >> 6 & 1) * a.dv;
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(smem_u32(to + e)), "l"(on ? src : a.s.nums), "r"(on) : "memory");
                }
            }
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];\n" ::"r"(smem_u32(raw_full + c % kXSlots)) : "memory");
        };
        bring_x(0);
        int as = 0, ks = 0, qs = 0;            // copies asked for
        for (int c = 0; c < n && ok; ++c) {
            const unsigned char* rows = a.s.rows + ((size_t)(base + c) * a.units + h / a.per_unit) * 6 * H * kTile;
            if (!SUMS) {
                if (c > 0 && !wait(intra_done, c - 1)) break;
                copy(a_img, a.s.mats + ((size_t)(base + c) * a.heads + h) * 3 * kTile, 6 * kTile, a_full);
                ++as;
            }
            if (c > 0 && !wait(upd_done, c - 1)) break;
            copy(k_img, rows + rows_bytes, rows_bytes, k_full);
            ++ks;
            if (c > 0 && !wait(d_read, c - 1)) break;      // (the state may ask for the values of chunk c - 1)
            if (c + 1 < n) bring_x(c + 1);
            if (!SUMS) {
                if (c > 0 && !wait(out_done, c - 1)) break;
                copy(q_img, rows, rows_bytes, q_full);
                ++qs;
            }
        }
        // no copy is on its way when the block ends, not even where a wait ran out
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        if (as > 0) mbar_wait(a_full, (as - 1) & 1);
        if (ks > 0) mbar_wait(k_full, (ks - 1) & 1);
        if (qs > 0) mbar_wait(q_full, (qs - 1) & 1);
    } else if (warp == 1) {
        // ---------------- the products, the smallest first ----------------
        constexpr unsigned of_a = 0x001102, of_b = 0x010120;      // a nibble a product
        const unsigned long long qd = operand(q_img, 2, 1024), kd = operand(k_img, 2, 1024, kTile), ad = operand(a_img, 2, 1024);
        int intra = 0, updates = 0, outs = 0;  // products issued and committed
        for (int c = 0; c < n && ok; ++c) {
            if (!SUMS) {
                if (c > 0) wait(out_read, c - 1);
                wait(a_full, c);
                if (!wait(x_full, c)) break;
                fence_after();
                if (elect()) {
#pragma unroll 1
                    for (int p = 0; p < 6; ++p)
#pragma unroll
                        for (int k = 0; k < kT / 16; ++k)
                            mma_ts(tmem + kOut, tmem + kX + (of_a >> 4 * p & 15) * 32 + 8 * k, ad + (unsigned)((of_b >> 4 * p & 15) * (kTile >> 4) + 2 * k), instruction(64), p > 0 || k > 0);
                }
                __syncwarp();
            }
            if (c > 0) wait(d_read, c - 1);
            if (!SUMS) {                       // the upper head's, where the state's sums have been read and are not yet formed again
                if (!ok) break;
                fence_after();
                if (elect()) {
#pragma unroll 1
                    for (int p = 0; p < 6; ++p)
#pragma unroll
                        for (int k = 0; k < kT / 16; ++k)
                            mma_ts(tmem + kD, tmem + kX + (of_a >> 4 * p & 15) * 32 + 8 * k, ad + (unsigned)(((of_b >> 4 * p & 15) + 3) * (kTile >> 4) + 2 * k),
                                   instruction(64), p > 0 || k > 0);
                    commit(intra_done);
                }
                __syncwarp();
                ++intra;
            }
            if (!SUMS) wait(intra_read, c);
            wait(xs_full, c);
            if (!wait(k_full, c)) break;
            fence_after();
            if (elect()) {
#pragma unroll 1
                for (int p = 0; p < 6; ++p)
#pragma unroll
                    for (int k = 0; k < kT / 16; ++k)
                        mma_ts(tmem + kD, tmem + kX + (of_a >> 4 * p & 15) * 32 + 8 * k, kd + (unsigned)((of_b >> 4 * p & 15) * H * (kTile >> 4) + k * (2048 >> 4)),
                               instruction(NR, false, true), p > 0 || k > 0);
                commit(upd_done);
            }
            __syncwarp();
            ++updates;
            if (!SUMS) {
                wait(q_full, c);
                if (!wait(s_full, c)) break;
                fence_after();
                if (elect()) {
#pragma unroll 1
                    for (int p = 0; p < 6; ++p)
#pragma unroll
                        for (int k = 0; k < NR / 16; ++k)
                            mma_ts(tmem + kOut, tmem + kParts + (of_a >> 4 * p & 15) * kHalf + 8 * k,
                                   qd + (unsigned)(((of_b >> 4 * p & 15) * H + k / 4) * (kTile >> 4) + 2 * (k % 4)), instruction(64), p > 0 || k > 0);
                    commit(out_done);
                }
                __syncwarp();
                ++outs;
            }
        }
        if (!ok) {                             // (those of the lower head may have no commit of their own)
            if (elect()) commit(intra_done);
            __syncwarp();
            ++intra;
        }
        if (intra > 0) mbar_wait(intra_done, (intra - 1) & 1);         // nor are products
        if (updates > 0) mbar_wait(upd_done, (updates - 1) & 1);
        if (outs > 0) mbar_wait(out_done, (outs - 1) & 1);
    } else if (warp < 2 + kSWarps) {
        // ---------------- the state: a lane a column, half of the rows a warp ----------------
        const int quarter = warp & 3, half = warp >= 6, v0 = quarter * 32 + lane, col = v0 & 63;
        const unsigned lanes = (unsigned)(quarter * 32) << 16;
        {
            const bool live = col < a.dv;
            // the half's first eight rows of the column as the state lies, [head][row / 8][column][row % 8]; where the sequence leaves it
            const int start = a.start_pos[seq];
            float* fresh = a.state + (size_t)a.slot_of_seq[seq] * a.slot_stride + a.state_off +
                           (((size_t)(a.head0 + hl) * (NR / 8) + half * (NR / 16)) * a.dv + col) * 8 + (size_t)((start + n_new) & 1) * a.copy_stride;
            const bool lone = size >= length, some = live && (start > 0 || begin > 0);      // (the segment is one group; there is a state)
            // what the segment starts from: the sequence's state, behind another segment what that wrote, and its copy
            const float* old = fresh + (begin > 0 ? 0 : (start & 1) - ((start + n_new) & 1)) * a.copy_stride;
            float* kept = a.s.firsts + (((size_t)slot * a.heads + hl) * a.dv + min(col, a.dv - 1)) * NR + half * kHalf;
            if (SUMS && group == 0 && some) {
#pragma unroll
                for (int r = 0; r < kHalf; ++r) kept[r] = old[r / 8 * 8 * a.dv + r % 8];
            }
            float S[kHalf];
#pragma unroll
            for (int r = 0; r < kHalf; ++r) S[r] = 0.f;
            if (!SUMS) {
                if (some) {
                    const float* from = lone ? old : kept;
                    const int by = lone ? 8 * a.dv : 8;
#pragma unroll
                    for (int r = 0; r < kHalf; ++r) S[r] = from[r / 8 * by + r % 8];
                }
                for (int g = 0; g < group; ++g) {          // the groups in front
                    const size_t i = (size_t)(slot * (kGroups - 1) + g) * a.heads + hl;
                    const float* sum = a.s.sums + (i * a.dv + min(col, a.dv - 1)) * NR + half * kHalf;
                    const float d = a.s.decays[i];
#pragma unroll
                    for (int r = 0; r < kHalf; r += 4) {
                        const float4 s4 = *reinterpret_cast<const float4*>(sum + r);
                        S[r] = fmaf(S[r], d, s4.x);
                        S[r + 1] = fmaf(S[r + 1], d, s4.y);
                        S[r + 2] = fmaf(S[r + 2], d, s4.z);
                        S[r + 3] = fmaf(S[r + 3], d, s4.w);
                    }
                }
            }
            float all = 1.f;                   // the group's decay
            for (int c = 0; c <= n && ok; ++c) {
                if (c > 0) {
                    const float* nums = nums_of(c - 1);
                    const float decay = nums[128];
                    all *= decay;
                    if (!wait(upd_done, c - 1)) break;
                    fence_after();
#pragma unroll
                    for (int r = 0; r < kHalf; r += 16) {
                        float v[16];
                        tmem_ld16(tmem + lanes + kD + half * kHalf + r, v);
                        wait_ld();
#pragma unroll
                        for (int e = 0; e < 16; ++e) S[r + e] = fmaf(S[r + e], decay, v[e]);
                    }
                    if (odd[((c - 1) & 1) * 4 + quarter]) {            // what was taken out of x
                        const unsigned char* k = a.s.rows + ((size_t)(base + c - 1) * a.units + h / a.per_unit) * 6 * H * kTile + 3 * H * kTile;
#pragma unroll 1
                        for (int t = 0; t < kT; ++t) {
                            float x = xs[(c - 1) % kXSlots * kT * 128 + t * 128 + v0];
                            const bool out = !isfinite(x);
                            if (!__any_sync(0xffffffffu, out)) continue;
                            x *= nums[64 + t];
#pragma unroll
                            for (int r = 0; r < kHalf; ++r) {
                                const int row = half * kHalf + r;
                                const float w = joined(k + (row / 64) * kTile + swizzled(t, row % 64), H * kTile);
                                if (out) S[r] = fmaf(w, x, S[r]);
                            }
                        }
                    }
                    fence_before();
                    arrive(d_read);
                }
                if (c == n) break;
                if (SUMS) continue;
                if (c > 0 && !wait(out_done, c - 1)) break;
#pragma unroll
                for (int r = 0; r < kHalf; r += 32) {
                    unsigned p[3][16];
#pragma unroll
                    for (int e = 0; e < 16; ++e) split3(S[r + 2 * e], S[r + 2 * e + 1], p[0][e], p[1][e], p[2][e]);
                    fence_after();
#pragma unroll
                    for (int l = 0; l < 3; ++l) tmem_st16(tmem + lanes + kParts + l * kHalf + half * (kHalf / 2) + r / 2, p[l]);
                }
                wait_st();
                fence_before();
                arrive(s_full);
                {                              // x with the factors of what is written takes the place of x itself: half of the tokens
                    const float f = nums_of(c)[64 + half * 32 + lane];
                    if (!wait(intra_done, c)) break;
                    fence_after();
                    put_x<true>(xs + c % kXSlots * kT * 128 + half * 32 * 128 + v0, tmem + lanes + kX + half * 16, f);
                    wait_st();
                    fence_before();
                    arrive(xs_full);
                }
            }
            if (ok && SUMS) {
                const size_t i = (size_t)(slot * (kGroups - 1) + group) * a.heads + hl;
                if (live) {
                    float* sum = a.s.sums + (i * a.dv + col) * NR + half * kHalf;
#pragma unroll
                    for (int r = 0; r < kHalf; r += 4) *reinterpret_cast<float4*>(sum + r) = make_float4(S[r], S[r + 1], S[r + 2], S[r + 3]);
                }
                if ((quarter & 1) == 0 && half == 0 && lane == 0) a.s.decays[i] = all;
            } else if (ok && lo + n == length && live) {
#pragma unroll
                for (int r = 0; r < kHalf; ++r) fresh[r / 8 * 8 * a.dv + r % 8] = S[r];
            }
        }
    } else {
        // ---------------- x and the output: a lane a column ----------------
        const int quarter = warp & 3, v0 = quarter * 32 + lane, col = v0 & 63;
        const unsigned lanes = (unsigned)(quarter * 32) << 16;
        {
            const bool live = col < a.dv;
            bool some = false;
            auto begin = [&](int c) {          // x of chunk c into its parts, once those of the chunk before have been read
                const float f0 = SUMS ? nums_of(c)[64 + lane] : 1.f, f1 = SUMS ? nums_of(c)[96 + lane] : 1.f;
                wait(raw_full + c % kXSlots, c / kXSlots);
                if (c > 0) wait(upd_done, c - 1);
                if (!ok) return;
                fence_after();
                const float* x = xs + c % kXSlots * kT * 128 + v0;
                const bool low = put_x<SUMS>(x, tmem + lanes + kX, f0), high = put_x<SUMS>(x + 32 * 128, tmem + lanes + kX + 16, f1);
                some = __any_sync(0xffffffffu, low || high);
                wait_st();
                fence_before();
                if (lane == 0) odd[(c & 1) * 4 + quarter] = some;
                arrive(SUMS ? xs_full : x_full);
            };
            begin(0);
            for (int c = 0; c < n && ok; ++c) {
                if (SUMS) {
                    if (c + 1 < n) begin(c + 1);
                    continue;
                }
                const int t0 = first + c * kT, nt = min(kT, rest - c * kT);
                const float* nums = nums_of(c);
                const float* x = xs + c % kXSlots * kT * 128 + v0;
                const bool odd_here = some;
                const float g0 = nums[lane], g1 = nums[32 + lane];
                if (!wait(intra_done, c)) break;
                fence_after();
                float y[kT];
#pragma unroll
                for (int j = 0; j < kT; j += 16) tmem_ld16(tmem + lanes + (quarter >= 2 ? kD : kOut) + j, y + j);
                wait_ld();
                if (odd_here) {
                    const unsigned char* m = a.s.mats + ((size_t)(base + c) * a.heads + hl) * 3 * kTile;
#pragma unroll 1
                    for (int t = 0; t < kT; ++t) {
                        const float bad = x[t * 128];
                        const bool out = !isfinite(bad);
                        if (!__any_sync(0xffffffffu, out)) continue;
#pragma unroll
                        for (int j = 0; j < kT; ++j) {
                            const float w = j < t ? 0.f : joined(m + swizzled(j, t), kTile);
                            if (out && j >= t) y[j] = fmaf(w, bad, y[j]);
                        }
                    }
                }
                fence_before();
                arrive(intra_read);            // (from here on the chunk's x may give way)
                if (c + 1 < n) begin(c + 1);
                if (!wait(out_done, c)) break;
                fence_after();
#pragma unroll
                for (int j = 0; j < kT; j += 16) {
                    float v[16];
                    tmem_ld16(tmem + lanes + kOut + j, v);
                    wait_ld();
                    if (j + 16 == kT) {
                        fence_before();
                        arrive(out_read);
                    }
#pragma unroll
                    for (int e = 0; e < 16; ++e) y[j + e] = fmaf(v[e], __shfl_sync(0xffffffffu, j + e < 32 ? g0 : g1, (j + e) & 31), y[j + e]);
                }
                if (live) {
                    float* out = a.y + (size_t)t0 * a.y_stride + (size_t)(a.head0 + hl) * a.dv + col;
#pragma unroll
                    for (int j = 0; j < kT; ++j) {
                        if (j < nt) *out = y[j];
                        out += a.y_stride;
                    }
                }
            }
        }
    }
    fence_before();
    __syncthreads();
    if (warp == 1) {
        fence_after();
        tmem_free(tmem, 512);
    }
}

template <typename K>
static int allow_smem(K kernel, int smem) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    return e == cudaSuccess ? BLM_OK : blm_fail(BLM_CUDA_ERROR, "scan_long: %s", cudaGetErrorString(e));
}

// How a step is run: passes over the chunks' indexes (Chunks) and over the heads, in whole groups of those that share B and C, so that a
// pass's scratch stays within kMost bytes.  Heads know nothing of one another and segments are their sequences' own: passes change no bit.
// With 64 heads of 128 x 64 and one group a segment of 4,096 tokens is 118 MB.  Passes over heads alone, each over the whole prompt, held fewer blocks
// than the chip and were slower than chunks of sixteen: 64 heads in 8 groups, 16,384 tokens 2,124 us, by segments 895, by chunks of sixteen
// 1,144; 32,768 tokens 7,773, 1,811 and 2,268.
constexpr long long kMost = 256ll << 20;
struct Passes {
    int heads, count, gap, later, slots;
    long long all, chunks;         // indexes of the step, chunks of a pass
    Sizes sizes;
    int number(int of_heads) const { return (int)((all + count - 1) / count) * ((of_heads + heads - 1) / heads); }
};
static bool passes_of(Passes& p, int heads, int unit, int dv, int n_tokens, int n_seqs, int longest, int least) {
    p.all = n_seqs > 1 ? chunk_bound(n_tokens, n_seqs) : (n_tokens + kT - 1) / kT;
    const int longest_chunks = (std::min(longest, n_tokens) + kT - 1) / kT, segment = std::min(kSegment, longest_chunks);
    const bool several = longest_chunks > kSegment;    // sequences of several segments
    p.gap = n_seqs > 1 ? std::min(kSegment, std::max(1, least / kT)) : kSegment;
    p.later = several && n_seqs > 1;
    const long long limit = several ? std::min<long long>(p.all, kSegment) : p.all;
    auto with = [&](long long count) {
        p.count = (int)count;
        p.slots = (int)((count + p.gap - 1) / p.gap) + p.later;
        p.chunks = n_seqs > 1 ? std::min(p.all, count + segment - 1) : count;
        p.sizes = sizes_of(p.heads / unit, p.heads, dv, p.chunks, p.slots);
        return p.sizes.all() <= kMost && p.heads / unit <= 65535 && p.slots * kGroups <= 65535;
    };
    for (p.heads = heads;; p.heads = (p.heads / unit + 1) / 2 * unit) {
        if (with(limit)) return true;
        // as many indexes as fit, in even parts, unless they are few beside the chunks that reach beyond them
        const double chunk = (double)sizes_of(p.heads / unit, p.heads, dv, 1, 0).all(), slot = (double)sizes_of(p.heads / unit, p.heads, dv, 0, 1).all();
        const long long most = (long long)((kMost - chunk * (segment - 1) - slot * (1 + p.later)) / (chunk + slot / p.gap));
        if (n_seqs > 1 && most >= (segment + 1) / 2) {
            const long long parts = (limit + most - 1) / most;
            if (with((limit + parts - 1) / parts)) return true;
        }
        if (p.heads <= unit) return false;
    }
}

// Bytes of scratch; 0: these kernels do not take the step (states of 65 to 128 rows x 33 to 64 columns, an even number of heads that share
// B and C: `unit`; `longest`: no sequence brings more tokens).  And how many kernels are launched.
BLM_API long long blm_scan_long_scratch(int heads, int unit, int rows, int dv, int n_tokens, int n_seqs, int longest, int least) {
    if (rows <= NR / 2 || rows > NR || dv <= 32 || dv > 64 || unit < 2 || unit % 2 || heads % unit || n_seqs < 1 || n_tokens < 1 || longest < 1 || least < 1)
        return 0;
    Passes p;
    return passes_of(p, heads, unit, dv, n_tokens, n_seqs, longest, least) ? p.sizes.all() : 0;
}
BLM_API int blm_scan_long_launches(int heads, int unit, int rows, int dv, int n_tokens, int n_seqs, int longest, int least) {
    Passes p;
    return passes_of(p, heads, unit, dv, n_tokens, n_seqs, longest, least) ? 3 * p.number(heads) : 0;
}

BLM_API int blm_scan_chunks_long_ssm(const float* xbc, long long xbc_stride, int x_col0, int b_col0, int c_col0, const float* dt_raw,
                                     long long dt_stride, int dt_col0, const float* dt_bias, const float* A_log, const float* D, float* y,
                                     long long y_stride, int heads, int groups, int N, int dv, const int* cu_seqlens,
                                     const int* slot_of_seq, const int* start_pos, int n_tokens, int n_seqs, int longest, int least, float* state,
                                     long long slot_stride, long long copy_stride, long long state_off, float* scratch, int* status,
                                     cudaStream_t stream) {
    if (n_seqs == 0 || n_tokens == 0) return BLM_OK;
    BLM_REQUIRE(groups > 0 && heads % groups == 0, "scan_long: bad head counts");
    const int per = heads / groups;
    BLM_REQUIRE(blm_scan_long_scratch(heads, per, N, dv, n_tokens, n_seqs, longest, least) > 0 && status, "scan_long: %d rows, %d columns", N, dv);
    Passes pass;
    passes_of(pass, heads, per, dv, n_tokens, n_seqs, longest, least);
    if (int rc = allow_smem(long_prep_kernel, kPrepSmem)) return rc;
    if (int rc = allow_smem(long_run_kernel<true>, kRunSmem)) return rc;
    if (int rc = allow_smem(long_run_kernel<false>, kRunSmem)) return rc;
    for (int head0 = 0; head0 < heads; head0 += pass.heads)
        for (long long from = 0; from < pass.all; from += pass.count) {
            const Chunks ch = {cu_seqlens, n_seqs, least, (int)from, pass.count, pass.gap, pass.later};
            const int now = std::min(heads - head0, pass.heads);
            const Scratch s = scratch_at(scratch, sizes_of(now / per, now, dv, pass.chunks, pass.slots));
            const SsmPrepArgs p = {{xbc, xbc_stride, x_col0}, {dt_raw, dt_stride, dt_col0}, b_col0, c_col0, dt_bias, A_log, D, ch, heads, groups, N,
                                   head0 / per, now / per, s};
            int rc;
            long_prep_kernel<<<dim3((unsigned)std::min(pass.chunks, pass.all - from), now / per, (per + kPrepHeads - 1) / kPrepHeads), kPrepThreads, kPrepSmem, stream>>>(p);
            if ((rc = blm_check_launch("scan_long (chunks)"))) return rc;
            const RunArgs a = {{xbc, xbc_stride, x_col0}, s, ch, slot_of_seq, start_pos, now / per, per, head0, now, dv, y, y_stride, state, slot_stride, copy_stride, state_off, status};
            const dim3 grid(now / 2, pass.slots * kGroups);
            long_run_kernel<true><<<grid, kRunThreads, kRunSmem, stream>>>(a);
            if ((rc = blm_check_launch("scan_long (sums)"))) return rc;
            long_run_kernel<false><<<grid, kRunThreads, kRunSmem, stream>>>(a);
            if ((rc = blm_check_launch("scan_long (run)"))) return rc;
        }
    return BLM_OK;
}
