// cv_build.cu -- composition-vector construction on the device.
//
// Same result as the reference pipeline of phylogenetics/src/main/cpp/native.cu
// (count_kmers :220-256, totals :317-345, Markov alpha :350-400, nnz/norm
// :402-428, sorted selection :449-458, normalisation :460-468, padding
// :470-474), computed without the dense A^K table:
//
//   A slot a.m.b (a, b single symbols, m the (K-2)-mer in between) can only be
//   nonzero when its prefix a.m and its suffix m.b were both seen as
//   (K-1)-mers (then the middle m was seen too).  So the candidates are, for
//   every seen (K-1)-mer q = a.m in ascending order, the symbols b of the
//   right-extension set R(m) = { b : m.b seen }, a 21-bit mask per
//   (K-2)-mer.  Enumerated in that order the candidate keys q*A + b are
//   already sorted, and the count of every seen K-mer is scattered straight
//   into its candidate slot (rank of b in R(m)) -- no sort and no A^K table.
//
// Pipeline per batch of proteomes (all kernels take the whole batch):
//   k_begin         zeroed counts, bitmaps and totals; tile bases per proteome
//   k_count         (K-2)/(K-1) counts, seen (K-1)-mers (the right-extension
//                   masks are slices of that bitmap), window totals
//   k_cand_count    candidates and seen (K-1)-mers per chunk of bitmap words; in
//                   further blocks the count -> probability and tuple tables
//   k_cand_scan     their offsets; proteome p's candidates start at cbase[p], a
//                   multiple of ALPHA_TILE
//   k_cand_offsets  per-(K-1)-mer candidate offsets and ranks; the key of every candidate
//   k_c0_scatter    (K-1)-mer counts (compact tables) and K-mer counts into candidate
//                   slots (zeroed by k_cand_offsets)
//   k_alpha         Markov alpha (reference double order), flat over the
//                   candidates: a seen candidate's count is replaced in place by
//                   its alpha bits (an unseen one keeps count 0: alpha -1);
//                   survivors counted per segment; norm partials
//   k_norm          per-proteome norm, scale, nnz, and where each CTA's survivors go
//   k_tuple_value   the tuples' normalised values
//   (batches: the host reads nnz)
//   k_compact       survivors' keys and normalised values, segment by segment
//   k_union_mark    (with a key bitmap) the candidate keys of every seen (K-1)-mer
#include "cv_build.cuh"
#include "hostctx.cuh"
#include "rank.cuh"
#include "scan.cuh"

#include <type_traits>

namespace phylo {

constexpr int TILE = 512;            // sequence positions per counting tile (few
                                     // proteomes' tables in flight -> L2 hits)
constexpr int COUNT_THREADS = 256;
constexpr int CHUNK_THREADS = 256;

// ---------------------------------------------------------------------------
// helpers
// ---------------------------------------------------------------------------

// Batch bases (cbase: B + 1 entries) staged in shared memory when they fit, so
// that finding a CTA's proteome is one round of parallel loads instead of a chain
// of dependent ones per thread (k_compact; in the kernels whose tables rely on L1
// the staging measured slower).
constexpr int SMEM_BASES = 256;
__device__ __forceinline__ const uint64_t *stage_bases(const uint64_t *__restrict__ g, int n,
                                                       uint64_t *s) {
    if (n > SMEM_BASES) return g;
    for (int i = threadIdx.x; i <= n; i += blockDim.x) s[i] = g[i];
    __syncthreads();
    return s;
}

__device__ __forceinline__ int find_owner(const uint64_t *__restrict__ base, int n, uint64_t t) {
    // largest p with base[p] <= t, base has n+1 entries, base[0] = 0
    int lo = 0, hi = n;
    while (hi - lo > 1) {
        int mid = (lo + hi) >> 1;
        if (base[mid] <= t) lo = mid; else hi = mid;
    }
    return lo;
}

// Markov alpha with the reference's operation order (native.cu:387-394):
//   p  = full / n0
//   p0 = ((prefix / n1) * (suffix / n1)) / (middle / n2)
//   alpha = float((p - p0) / p0)
// Every operation is an explicitly rounded IEEE double op, so no FMA
// contraction can change the result.
__device__ __forceinline__ float markov_alpha(uint32_t full, uint32_t prefix, uint32_t suffix,
                                              uint32_t middle, uint32_t n0, uint32_t n1,
                                              uint32_t n2) {
    if (full == 0u && n0 != 0u) return -1.0f;  // (0 - p0) / p0 == -1 exactly (p0 > 0 finite)
    double p = __ddiv_rn((double)full, (double)n0);
    double pp = __ddiv_rn((double)prefix, (double)n1);
    double ps = __ddiv_rn((double)suffix, (double)n1);
    double pm = __ddiv_rn((double)middle, (double)n2);
    double p0 = __ddiv_rn(__dmul_rn(pp, ps), pm);
    return __double2float_rn(__ddiv_rn(__dsub_rn(p, p0), p0));
}

// alpha from the quotients p = full/n0, pp = prefix/n1, ps = suffix/n1, pm = middle/n2 and
// ym = RN(1/pm) (see markov_alpha_fast).
__device__ __forceinline__ float markov_alpha_quot(double p, double pp, double ps, double pm,
                                                   double ym) {
    const double a = __dmul_rn(pp, ps);
    const double q0 = __dmul_rn(a, ym);
    const double p0 = __fma_rn(__fma_rn(-q0, pm, a), ym, q0);
    const double d = __dsub_rn(p, p0);
    if (d == 0.0) return 0.0f;
    const double y0 = (double)__frcp_rn(__double2float_rn(p0));
    const double g0 = __dmul_rn(d, y0);
    const double g1 = __fma_rn(__fma_rn(-g0, p0, d), y0, g0);
    const long long low = (long long)(__double_as_longlong(g1) & ((1ll << 29) - 1)) - (1ll << 28);
    if (low <= 256 && low >= -256) return __double2float_rn(__ddiv_rn(d, p0));
    return __double2float_rn(g1);
}

// The same alpha with the FP64 work cut down (GB300 issues FP64 at a small
// fraction of the FP32 rate):
//   * p, prefix/n1, suffix/n1, middle/n2 come from per-proteome tables holding
//     exactly those IEEE quotients for counts below PROB_TABLE;
//   * p0 = RN(a / b) as q0 = RN(a * y), r = a - b*q0 (exact by FMA),
//     RN(q0 + r*y) with y = RN(1/b) from the table -- a correctly rounded
//     quotient (Markstein's reciprocal-correction theorem);
//   * (p - p0) / p0 is only needed rounded to float: a quotient accurate to
//     ~2^-46 from a float reciprocal and one FMA correction gives the same float
//     unless it lies within 256 double ulps of a float rounding midpoint, where
//     the exact IEEE division is used instead.
// Anything outside the tables (large counts, no K-windows) takes markov_alpha.
__device__ __forceinline__ float markov_alpha_fast(uint32_t full, uint32_t prefix,
                                                   uint32_t suffix, uint32_t middle, uint32_t n0,
                                                   uint32_t n1, uint32_t n2,
                                                   const double *__restrict__ prob) {
    if (full == 0u && n0 != 0u) return -1.0f;
    if (n0 == 0u || full >= PROB_TABLE || prefix >= PROB_TABLE || suffix >= PROB_TABLE ||
        middle >= PROB_TABLE)
        return markov_alpha(full, prefix, suffix, middle, n0, n1, n2);
    return markov_alpha_quot(__ldg(&prob[full]), __ldg(&prob[PROB_TABLE + prefix]),
                             __ldg(&prob[PROB_TABLE + suffix]),
                             __ldg(&prob[2 * PROB_TABLE + middle]),
                             __ldg(&prob[3 * PROB_TABLE + middle]));
}
// Sum of non-negative floats as an exact 192-bit fixed-point number in units of
// 2^-96 (terms below 2^-73 lose their lowest bits; such squares need
// |alpha| < 2^-36).  Integer addition makes the result independent of order.
struct U192 {
    uint64_t w0, w1, w2;
};

__device__ __forceinline__ void u192_add(U192 &a, uint64_t p0, uint64_t p1, uint64_t p2) {
    asm("add.cc.u64 %0, %0, %3;\n\taddc.cc.u64 %1, %1, %4;\n\taddc.u64 %2, %2, %5;"
        : "+l"(a.w0), "+l"(a.w1), "+l"(a.w2)
        : "l"(p0), "l"(p1), "l"(p2));
}

// Adds a finite square; returns false for a square too large to hold (>= 2^72).
__device__ __forceinline__ bool u192_add_float(U192 &a, float v) {
    const uint32_t bits = __float_as_uint(v);
    const uint32_t e = bits >> 23;
    uint64_t m = e ? ((bits & 0x7fffffu) | 0x800000u) : (bits & 0x7fffffu);
    if (m == 0) return true;
    int sh = (e ? (int)e : 1) - 150 + 96;  // bit position of m's lowest bit
    if (sh < 0) {
        if (sh <= -24) return true;
        m >>= -sh;
        sh = 0;
    }
    uint64_t p0 = 0, p1 = 0, p2 = 0;
    if (sh < 64) {
        p0 = m << sh;
        p1 = sh ? (m >> (64 - sh)) : 0;
    } else if (sh < 128) {
        const int t = sh - 64;
        p1 = m << t;
        p2 = t ? (m >> (64 - t)) : 0;
    } else if (sh <= 192 - 24) {
        p2 = m << (sh - 128);
    } else {
        return false;
    }
    u192_add(a, p0, p1, p2);
    return true;
}

__device__ __forceinline__ U192 u192_shfl_down(const U192 &a, int d) {
    U192 r;
    r.w0 = __shfl_down_sync(0xffffffffu, a.w0, d);
    r.w1 = __shfl_down_sync(0xffffffffu, a.w1, d);
    r.w2 = __shfl_down_sync(0xffffffffu, a.w2, d);
    return r;
}

// value * 2^-96 rounded to nearest-even double
__device__ double u192_to_double(const U192 &a) {
    uint64_t top, next, rest;
    int base;
    if (a.w2) { top = a.w2; next = a.w1; rest = a.w0; base = 128; }
    else if (a.w1) { top = a.w1; next = a.w0; rest = 0; base = 64; }
    else if (a.w0) { top = a.w0; next = 0; rest = 0; base = 0; }
    else return 0.0;
    const int lz = __clzll(top);
    int pos = base + 63 - lz;  // index of the most significant bit
    const uint64_t hi64 = lz ? ((top << lz) | (next >> (64 - lz))) : top;
    const uint64_t below = lz ? (next << lz) : next;
    uint64_t mant = hi64 >> 11;
    const bool round_bit = (hi64 >> 10) & 1;
    const bool sticky = (hi64 & 0x3ffull) || below || rest;
    if (round_bit && (sticky || (mant & 1))) {
        mant++;
        if (mant == (1ull << 53)) {
            mant >>= 1;
            pos++;
        }
    }
    return ldexp((double)mant, pos - 52 - 96);
}

// Index of (K-1)-mer q of proteome p in the c1 / coff tables: q itself (dense
// rows of T1s entries), or its rank among the batch's seen (K-1)-mers (compact).
__device__ __forceinline__ uint64_t c1_index(const BuildArgs &a, int p, uint32_t q) {
    if (!a.compact1) return (uint64_t)p * a.T1s + q;
    const uint2 t = __ldg(&a.pw1[(uint64_t)p * (a.T1s / 32) + (q >> 5)]);  // {prefix, seen word}
    return (uint64_t)t.x + (uint32_t)__popc(t.y & ((1u << (q & 31u)) - 1u));
}

__device__ __forceinline__ uint32_t c1_load(const BuildArgs &a, uint64_t i) {
    return a.compact1 ? __ldg(&a.cc[i].x) : __ldg(&a.c1[i]);
}

// Index of (K-2)-mer m of proteome p in c2: dense row entry, or its rank among
// the batch's seen (K-2)-mers (compact).
__device__ __forceinline__ uint64_t c2_index(const BuildArgs &a, int p, uint32_t m) {
    if (!a.compact2) return (uint64_t)p * a.T2 + m;
    const uint2 t = __ldg(&a.pw2[(uint64_t)p * (a.T2s / 32) + (m >> 5)]);
    return (uint64_t)t.x + (uint32_t)__popc(t.y & ((1u << (m & 31u)) - 1u));
}

// Right-extension mask of (K-2)-mer m in proteome p: bit b set when the
// (K-1)-mer m.b was seen.  Those are the A bits of the seen bitmap starting at
// bit m * A (the code of m.b is m * A + b), so no separate table is kept.
__device__ __forceinline__ uint32_t ext_mask(const BuildArgs &a, int p, uint32_t m) {
    const uint32_t *sw = a.seen1 + (uint64_t)p * (a.T1s / 32);
    const uint64_t bit = (uint64_t)m * a.A;
    const uint64_t w = bit >> 5;
    const uint32_t off = (uint32_t)bit & 31u;
    uint32_t v = __ldg(&sw[w]) >> off;
    if (off + a.A > 32u) v |= __ldg(&sw[w + 1]) << (32u - off);
    return v & ((1u << a.A) - 1u);
}

// ---------------------------------------------------------------------------
// kernels
// ---------------------------------------------------------------------------

// Zeroes what the counting kernels add to (contiguous in scratch) and the status, and
// sets tile_base[p] = number of TILE-sized tiles of proteomes < p (tile_base[B] =
// total) and, for a single proteome, its offsets and output range.
__global__ void __launch_bounds__(256) k_begin(BuildArgs a) {
    previous_kernel_done();
    const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < a.zero_n8; i += step)
        a.zero[i] = 0;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *a.status = 0u;
        *a.p1_total = 0;
        if (!a.compact2) *a.p2_total = 0;
        if (a.single) {
            a.seq_off_store[0] = 0;
            a.seq_off_store[1] = a.single_len;
            a.dst_base[0] = 0;
            a.dst_cap[0] = a.single_cap;
        }
        uint64_t acc = 0;
        for (int p = 0; p < a.B; p++) {
            a.tile_base[p] = acc;
            acc += div_up(a.single ? a.single_len : a.seq_off[p + 1] - a.seq_off[p], TILE);
        }
        a.tile_base[a.B] = acc;
    }
}

// Blocks of the tables of one proteome (k_cand_count runs them beside its chunks; both
// need only the totals of k_count).
constexpr int PROB_BLOCKS = PROB_TABLE / CHUNK_THREADS;
constexpr int TUPLE_BLOCKS = TUPLE_TABLE / CHUNK_THREADS;

// Block `blk` of proteome p's tables.  prob[p][0][c] = c/n0, [1][c] = c/n1, [2][c] =
// c/n2, [3][c] = 1/(c/n2): the exact IEEE quotients the reference forms for count c.
// atab: alpha of every small count tuple, by the same arithmetic, so that a table hit
// gives the bits the direct path would.
__device__ void table_block(const BuildArgs &a, int p, int blk) {
    const uint32_t n0 = a.tot[p * 4 + 0], n1 = a.tot[p * 4 + 1], n2 = a.tot[p * 4 + 2];
    if (blk < PROB_BLOCKS) {
        const uint32_t c = blk * CHUNK_THREADS + threadIdx.x;
        double *t = a.prob + (uint64_t)p * 4 * PROB_TABLE;
        const double pm = __ddiv_rn((double)c, (double)n2);
        t[c] = __ddiv_rn((double)c, (double)n0);
        t[PROB_TABLE + c] = __ddiv_rn((double)c, (double)n1);
        t[2 * PROB_TABLE + c] = pm;
        t[3 * PROB_TABLE + c] = __ddiv_rn(1.0, pm);
        return;
    }
    // 256 consecutive tuples: one full, one prefix, two suffixes, every middle
    static_assert(CHUNK_THREADS == 2 * TUPLE_MID, "a block holds two suffix counts");
    __shared__ double s_mid[2][TUPLE_MID], s_q[4];
    const uint32_t t0 = (uint32_t)(blk - PROB_BLOCKS) * CHUNK_THREADS, t = t0 + threadIdx.x;
    const uint32_t mid = t % TUPLE_MID, suf = (t / TUPLE_MID) % TUPLE_PS,
                   pre = (t / (TUPLE_MID * TUPLE_PS)) % TUPLE_PS,
                   full = t / (TUPLE_MID * TUPLE_PS * TUPLE_PS);
    if (threadIdx.x < TUPLE_MID) {
        const double pm = __ddiv_rn((double)threadIdx.x, (double)n2);
        s_mid[0][threadIdx.x] = pm;
        s_mid[1][threadIdx.x] = __ddiv_rn(1.0, pm);
    } else if (threadIdx.x < TUPLE_MID + 4) {
        const int j = threadIdx.x - TUPLE_MID;
        const uint32_t c = j == 0 ? full : j == 1 ? pre : (t0 / TUPLE_MID + j - 2) % TUPLE_PS;
        s_q[j] = __ddiv_rn((double)c, (double)(j == 0 ? n0 : n1));
    }
    __syncthreads();
    uint32_t bits = 0;
    if (full >= 1 && pre >= 1 && suf >= 1 && mid >= 1 && n0 != 0)
        bits = __float_as_uint(markov_alpha_quot(s_q[0], s_q[1], s_q[2 + threadIdx.x / TUPLE_MID],
                                                 s_mid[0][mid], s_mid[1][mid]));
    a.atab[(uint64_t)p * TUPLE_TABLE + t] = bits;
}

__device__ __forceinline__ float div_by_scale(float f, double scale, double rs) {
    const double x = (double)f;
    const double q = __dmul_rn(x, rs);
    return __double2float_rn(__fma_rn(__fma_rn(-q, scale, x), rs, q));
}

// Normalised value of every tuple, after the norm is known.  grid = (TUPLE_TABLE / 256, B)
__global__ void k_tuple_value(BuildArgs a) {
    previous_kernel_done();
    const int p = blockIdx.y;
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (uint32_t)TUPLE_TABLE) return;
    const double scale = a.scale[p], rs = a.rscale[p];
    const float f = __uint_as_float(a.atab[(uint64_t)p * TUPLE_TABLE + t]);
    float v;
    if (!(isfinite(scale) && scale > 0.0) || !isfinite(f))
        v = __double2float_rn(__ddiv_rn((double)f, scale));
    else
        v = div_by_scale(f, scale, rs);
    a.vtab[(uint64_t)p * TUPLE_TABLE + t] = v;
}

// Counts (K-2)- and (K-1)-windows, marks right extensions, totals n0/n1/n2.
// A window starting at i counts for length L when its L symbols are all in the
// alphabet and inside the proteome (native.cu:236-252).
template <bool COMPACT>
__global__ void __launch_bounds__(COUNT_THREADS) k_count(BuildArgs a) {
    previous_kernel_done();
    __shared__ uint8_t dig[TILE + 16];
    __shared__ uint32_t ntot[3];
    const int K = a.k;
    const uint32_t A = a.A;
    const uint64_t total_tiles = a.tile_base[a.B];
    for (uint64_t t = blockIdx.x; t < total_tiles; t += gridDim.x) {
        const int p = find_owner(a.tile_base, a.B, t);
        const uint64_t s0 = a.seq_off[p], len = a.seq_off[p + 1] - s0;
        const uint64_t start = (t - a.tile_base[p]) * TILE;
        if (threadIdx.x < 3) ntot[threadIdx.x] = 0;
        for (int j = threadIdx.x; j < TILE + K; j += COUNT_THREADS) {
            uint64_t pos = start + j;
            dig[j] = pos < len ? (uint8_t)char_to_digit(a.alpha, a.seq[s0 + pos]) : (uint8_t)0xff;
        }
        __syncthreads();
        uint32_t *c1 = COMPACT ? nullptr : a.c1 + (uint64_t)p * a.T1s;
        uint32_t *seen = a.seen1 + (uint64_t)p * (a.T1s / 32);
        uint32_t *c2 = a.c2 + (uint64_t)p * a.T2;
        uint32_t *seen2 = a.seen2 + (uint64_t)p * (a.T2s / 32);
        uint32_t cnt0 = 0, cnt1 = 0, cnt2 = 0;
        for (int u = 0; u < TILE / COUNT_THREADS; u++) {
            const int li = u * COUNT_THREADS + threadIdx.x;
            const bool inb = start + li < len;
            uint32_t w = 0, w2 = 0, w1 = 0, last = 0;
            int run = 0;
            if (inb) {
                for (int j = 0; j < K; j++) {
                    uint32_t d = dig[li + j];
                    if (d == 0xffu) break;
                    w = w * A + d;
                    run = j + 1;
                    if (j == K - 3) w2 = w;
                    if (j == K - 2) { w1 = w; last = d; }
                }
            }
            const bool v2 = run >= K - 2, v1 = run >= K - 1, v0 = run >= K;
            cnt2 += v2; cnt1 += v1; cnt0 += v0;
            // counts: reduction atomics (equal keys within a warp are rare, so no
            // aggregation); the first sighting of a (K-1)-mer sets its seen bit,
            // which is also bit `last` of the right-extension mask of its first
            // K-2 symbols (compact tables: only the seen bit here; k_c0_scatter
            // counts once the ranks of the seen (K-1)-mers are known)
            if (v2) {  // compact (K-2)-mer tables: the seen bit; k_c0_scatter counts
                if (a.compact2) atomicOr(&seen2[w2 >> 5], 1u << (w2 & 31u));
                else atomicAdd(&c2[w2], 1u);
            }
            if (v1) {
                if (COMPACT) {
                    atomicOr(&seen[w1 >> 5], 1u << (w1 & 31u));
                } else if (atomicAdd(&c1[w1], 1u) == 0u) {
                    atomicOr(&seen[w1 >> 5], 1u << (w1 & 31u));
                }
            }
        }
        // totals
        cnt0 = __reduce_add_sync(0xffffffffu, cnt0);
        cnt1 = __reduce_add_sync(0xffffffffu, cnt1);
        cnt2 = __reduce_add_sync(0xffffffffu, cnt2);
        if ((threadIdx.x & 31) == 0) {
            atomicAdd(&ntot[0], cnt0);
            atomicAdd(&ntot[1], cnt1);
            atomicAdd(&ntot[2], cnt2);
        }
        __syncthreads();
        if (threadIdx.x < 3 && ntot[threadIdx.x]) atomicAdd(&a.tot[p * 4 + threadIdx.x], ntot[threadIdx.x]);
        __syncthreads();
    }
}

constexpr int MAX_WPT = 8;  // bitmap words per thread of the candidate passes, or one

// Consecutive bitmap words of a warp of the candidate passes.
__device__ __forceinline__ uint32_t warp_words(const BuildArgs &a) { return a.wlanes * a.wpt; }

// Candidates of the seen (K-1)-mers of one word of the seen bitmap (32
// consecutive (K-1)-mers): |R(m)| = popc(ext_mask(m)) for each seen q = a.m.
__device__ __forceinline__ uint32_t word_candidates(const BuildArgs &a, int p, uint32_t q0,
                                                    uint32_t bits) {
    uint32_t s = 0;
    while (bits) {
        const uint32_t j = __ffs(bits) - 1;
        bits &= bits - 1;
        s += __popc(ext_mask(a, p, a.fdT2.mod(q0 + j)));
    }
    return s;
}

// Candidates and seen (K-1)-mers per chunk of bitmap words: each of the CTA's warps has
// warp_words(a) consecutive ones, 32, 8 or 2 of them with 1, 4 or 16 lanes to a word (see
// chunk_lanes); or, WIDE, for the sparse bitmaps of protein K = 7, MAX_WPT times 32, a lane
// taking every 32nd, and only the warps' totals are kept (12 uneven proteomes: 195 -> 148
// us against MAX_WPT neighbouring words per lane and a count per word; k_cand_offsets, which
// then reads coalesced too, 400 -> 365).  grid = (NCH + table blocks, B).  With compact (K-2)-mer tables also zeroes the entries
// in use, which k_c0_scatter counts in.
template <bool WIDE>
__global__ void __launch_bounds__(CHUNK_THREADS) k_cand_count(BuildArgs a) {
    previous_kernel_done();
    const int p = blockIdx.y, c = blockIdx.x;
    if ((uint64_t)c >= a.NCH) {
        table_block(a, p, c - (int)a.NCH);
        return;
    }
    const uint64_t nw = a.T1s / 32;
    const uint32_t lane = threadIdx.x & 31u, shared = 32u / a.wlanes;  // lanes to a word
    const uint64_t wd0 =
        ((uint64_t)c * (CHUNK_THREADS / 32) + threadIdx.x / 32) * warp_words(a) + lane / shared;
    uint32_t s = 0, n = 0;
    for (uint32_t i = 0; i < (WIDE ? MAX_WPT : 1); i++) {
        const uint64_t wd = wd0 + 32 * i;
        uint32_t bits = 0, sw = 0;
        if (wd < nw) {
            bits = a.seen1[(uint64_t)p * nw + wd];
            if (shared > 1) bits &= ((1u << a.wlanes) - 1u) << (lane % shared * a.wlanes);
            if (bits) sw = word_candidates(a, p, (uint32_t)(wd * 32), bits);
        }
        s += sw;
        n += __popc(bits);
        if (WIDE) continue;
        for (uint32_t d = 1; d < shared; d <<= 1) sw += __shfl_xor_sync(0xffffffffu, sw, d);
        if (wd < nw && lane % shared == 0) a.word_cand[(uint64_t)p * nw + wd] = sw;
    }
    s = __reduce_add_sync(0xffffffffu, s);
    n = __reduce_add_sync(0xffffffffu, n);
    __shared__ uint32_t ws[CHUNK_THREADS / 32], wn[CHUNK_THREADS / 32];
    if ((threadIdx.x & 31) == 0) {
        ws[threadIdx.x >> 5] = s;
        wn[threadIdx.x >> 5] = n;
        if (WIDE)
            a.warp_cs[((uint64_t)p * a.NCH + c) * (CHUNK_THREADS / 32) + (threadIdx.x >> 5)] =
                make_uint2(s, n);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t t = 0, u = 0;
        for (int w = 0; w < CHUNK_THREADS / 32; w++) {
            t += ws[w];
            u += wn[w];
        }
        a.chunk_cand[(uint64_t)p * a.NCH + c] = t;
        a.chunk_seen[(uint64_t)p * a.NCH + c] = u;
    }
    if (a.compact2) {
        const uint64_t used = min(*a.p2_total, a.cap2), step = a.NCH * a.B * CHUNK_THREADS;
        for (uint64_t i = ((uint64_t)p * a.NCH + c) * CHUNK_THREADS + threadIdx.x; i < used;
             i += step)
            a.c2[i] = 0u;
    }
}

// Exclusive scans of chunk_cand and chunk_seen over the batch, then cbase[p] = start of
// proteome p's candidates, rounded up to ALPHA_TILE, so that no k_alpha CTA straddles
// two proteomes.  One CTA: a batch of 24 at K = 6 has 12,000 chunks (two rounds), fewer
// than the launches of a wider scan cost.
constexpr int CSCAN_THREADS = 1024, CSCAN_ITEMS = 8;
__global__ void __launch_bounds__(CSCAN_THREADS) k_cand_scan(BuildArgs a) {
    previous_kernel_done();
    __shared__ uint64_t sw[CSCAN_THREADS / 32 + 1];
    const uint64_t nc = (uint64_t)a.B * a.NCH;
    uint64_t cand = 0, seen = 0;  // before the round
    for (uint64_t base = 0; base < nc; base += CSCAN_THREADS * CSCAN_ITEMS) {
        const uint64_t first = base + (uint64_t)threadIdx.x * CSCAN_ITEMS;
        uint32_t vc[CSCAN_ITEMS], vs[CSCAN_ITEMS];
        uint64_t sc = 0, ss = 0, tot;
#pragma unroll
        for (int i = 0; i < CSCAN_ITEMS; i++) {
            vc[i] = first + i < nc ? a.chunk_cand[first + i] : 0u;
            vs[i] = first + i < nc ? a.chunk_seen[first + i] : 0u;
            sc += vc[i];
            ss += vs[i];
        }
        uint64_t ec = cand + block_excl_scan_u64<CSCAN_THREADS>(sc, sw, &tot);
        cand += tot;
        uint64_t es = seen + block_excl_scan_u64<CSCAN_THREADS>(ss, sw, &tot);
        seen += tot;
#pragma unroll
        for (int i = 0; i < CSCAN_ITEMS; i++) {
            if (first + i < nc) {
                a.chunk_cand_off[first + i] = ec;
                a.chunk_seen_off[first + i] = (uint32_t)es;
            }
            ec += vc[i];
            es += vs[i];
        }
    }
    if (threadIdx.x == 0) a.chunk_cand_off[nc] = cand;
    __syncthreads();  // the offsets are read back below
    uint64_t run = 0;
    for (int p0 = 0; p0 < a.B; p0 += CSCAN_THREADS) {
        const int p = p0 + threadIdx.x;
        uint64_t n = 0, tot;
        if (p < a.B)
            n = div_up(a.chunk_cand_off[(uint64_t)(p + 1) * a.NCH] -
                           a.chunk_cand_off[(uint64_t)p * a.NCH], (uint64_t)ALPHA_TILE) * ALPHA_TILE;
        const uint64_t e = run + block_excl_scan_u64<CSCAN_THREADS>(n, sw, &tot);
        if (p < a.B) a.cbase[p] = e;
        run += tot;
    }
    if (threadIdx.x == 0) {
        a.cbase[a.B] = run;
        *a.cand_total = run;
        uint32_t full = run > a.cand_cap;
        if (a.compact1) {
            *a.p1_total = seen;
            full |= seen > a.cap1;
        }
        if (a.compact2) full |= *a.p2_total > a.cap2;
        if (full) *a.status = (uint32_t)DEV_CAPACITY;
    }
}

__device__ __forceinline__ uint32_t warp_incl_scan_u32(uint32_t v) {
    const uint32_t lane = threadIdx.x & 31u;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t o = __shfl_up_sync(0xffffffffu, v, d);
        if (lane >= (uint32_t)d) v += o;
    }
    return v;
}

// The lowest lane k whose (non-decreasing) inclusive scan value incl exceeds i;
// 31 when none does.
__device__ __forceinline__ uint32_t warp_owner(uint32_t incl, uint32_t i) {
    uint32_t k = 0;
#pragma unroll
    for (int step = 16; step > 0; step >>= 1) {
        const uint32_t v = __shfl_sync(0xffffffffu, incl, (int)(k + step - 1));
        if (v <= i) k += step;
    }
    return k;
}

// coff[p][q] = candidate offset of seen (K-1)-mer q within proteome p (entries
// of unseen q are not written); cq = the key q * A + b of every candidate (b over
// the right-extension mask of q's suffix, ascending), c0a zeroed.  A warp owns a
// contiguous run of bitmap words, one per lane of its first wlanes (WIDE: MAX_WPT times
// 32), and their candidates; these and the seen (K-1)-mers start at the exclusive scans of
// the word_cand sums and the words' populations (one scan of packed pairs; WIDE: at the
// totals of the warps before).  With compact tables pw1 gets the ranks of the words that
// hold any.  The warp
// processes its run together: its seen (K-1)-mers, 32 at a time in order (each lane
// finds its own by a search over the scan of the words' populations), load
// their masks together; a warp scan of the mask populations places their
// candidates, each lane writes its candidates into the warp's shared-memory stage
// at that offset, and the warp stores the stage coalesced.  (One lane per word,
// each writing its word's
// 0..32 A candidates, left most lanes idle; a warp per word wasted its scans on
// the sparse words of K = 7; finding each key's (K-1)-mer by a search over the
// scan cost about three times the instructions of the stage.)
// grid = (NCH, B)
template <bool WIDE>
__global__ void __launch_bounds__(CHUNK_THREADS) k_cand_offsets(BuildArgs a) {
    previous_kernel_done();
    __shared__ uint32_t s_stage[CHUNK_THREADS / 32][32 * 21];  // keys of 32 seen (K-1)-mers (A <= 21)
    uint32_t *stage = s_stage[threadIdx.x >> 5];
    const int p = blockIdx.y, c = blockIdx.x;
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t pc = (uint64_t)p * a.NCH + c;
    const uint64_t nw = a.T1s / 32;
    const uint32_t *seen = a.seen1 + (uint64_t)p * nw;
    const uint64_t wbeg =
        ((uint64_t)c * (CHUNK_THREADS / 32) + threadIdx.x / 32) * warp_words(a);
    // the warp's candidates [run, r1) of the proteome, and the rank P of its first seen
    // (K-1)-mer among the batch's
    uint32_t run =
        (uint32_t)(a.chunk_cand_off[pc] - a.chunk_cand_off[(uint64_t)p * a.NCH]);
    uint32_t P = a.chunk_seen_off[pc], r1;
    if constexpr (WIDE) {
        const uint32_t warp = threadIdx.x >> 5;
        const uint2 t =
            lane <= warp ? a.warp_cs[pc * (CHUNK_THREADS / 32) + lane] : make_uint2(0u, 0u);
        run += __reduce_add_sync(0xffffffffu, lane < warp ? t.x : 0u);
        P += __reduce_add_sync(0xffffffffu, lane < warp ? t.y : 0u);
        r1 = run + __shfl_sync(0xffffffffu, t.x, (int)warp);
    } else {
        __shared__ uint64_t sw[CHUNK_THREADS / 32 + 1];
        uint32_t s = 0, npop = 0;
        if (lane < a.wlanes && wbeg + lane < nw) {
            s = a.word_cand[(uint64_t)p * nw + wbeg + lane];
            npop = __popc(seen[wbeg + lane]);
        }
        uint64_t tot;
        const uint64_t ex =
            block_excl_scan_u64<CHUNK_THREADS>((uint64_t)npop << 32 | s, sw, &tot);
        r1 = run + __shfl_sync(0xffffffffu, (uint32_t)ex + s, 31);
        run += __shfl_sync(0xffffffffu, (uint32_t)ex, 0);
        P += __shfl_sync(0xffffffffu, (uint32_t)(ex >> 32), 0);
    }
    const uint64_t gb = a.cbase[p];
    // zero this warp's K-mer count slots (coalesced)
    for (uint64_t i = gb + run + lane; i < gb + r1 && i < a.cand_cap; i += 32) a.c0a[i] = 0u;
    // the warp's words [wbeg, wend), loaded up front (coalesced), lane l holding word
    // wbeg + 32 t + l of group t; the seen (K-1)-mers of a group are taken 32 at a time
    const uint64_t wend = min(wbeg + warp_words(a), nw);
    const uint32_t A = a.A;
    constexpr int WPT = WIDE ? MAX_WPT : 1;
    uint32_t wreg[WPT];
#pragma unroll
    for (int t = 0; t < WPT; t++) {
        const uint64_t w = wbeg + 32 * t + lane;
        wreg[t] = w < wend ? seen[w] : 0u;
    }
#pragma unroll
    for (int t = 0; t < WPT; t++) {
        const uint32_t wbits = wreg[t];
        const uint32_t wincl = warp_incl_scan_u32(__popc(wbits));
        const uint32_t nseen = __shfl_sync(0xffffffffu, wincl, 31);
        if (nseen == 0u) continue;
        const uint64_t wfirst = wbeg + 32 * t;
        // compact tables: P is the rank of the group's first seen (K-1)-mer; the i-th seen
        // (K-1)-mer of the group is then entry P + i
        if (a.compact1 && wfirst + lane < wend)
            a.pw1[(uint64_t)p * nw + wfirst + lane] = make_uint2(P + wincl - __popc(wbits), wbits);
        for (uint32_t sb = 0; sb < nseen; sb += 32) {
            const uint32_t i = sb + lane;
            const uint32_t k = warp_owner(wincl, i);
            const uint32_t wk = __shfl_sync(0xffffffffu, wbits, (int)k);
            const uint32_t ik = __shfl_sync(0xffffffffu, wincl, (int)k);
            const bool ok = i < nseen;
            uint32_t q = 0, mask = 0;
            if (ok) {
                q = (uint32_t)((wfirst + k) * 32) + nth_set_bit(wk, i - (ik - (uint32_t)__popc(wk)));
                mask = ext_mask(a, p, a.fdT2.mod(q));
            }
            const uint32_t n = __popc(mask);
            const uint32_t cincl = warp_incl_scan_u32(n);
            const uint32_t ctot = __shfl_sync(0xffffffffu, cincl, 31);
            // every seen (K-1)-mer, also one without candidates: its offset (the next
            // candidate's) and, with compact tables, its count slot (counted by
            // k_c0_scatter)
            if (ok) {
                const uint64_t qi = a.compact1 ? (uint64_t)P + i : c1_index(a, p, q);
                if (!a.compact1 || qi < a.cap1) {
                    if (a.compact1) a.cc[qi] = make_uint2(0u, run + cincl - n);
                    else a.coff[qi] = run + cincl - n;
                }
            }
            // their candidate keys: each lane writes its own (at most A) into the warp's
            // stage at its scanned offset, then the warp stores them coalesced
            {
                uint32_t e = mask, o = cincl - n;
                while (e) {
                    stage[o++] = q * A + (uint32_t)(__ffs(e) - 1);
                    e &= e - 1;
                }
            }
            __syncwarp();
            for (uint32_t ci = lane; ci < ctot; ci += 32) {
                const uint64_t dst = gb + run + ci;
                if (dst < a.cand_cap) a.cq[dst] = stage[ci];
            }
            __syncwarp();
            run += ctot;
        }
        P += nseen;
    }
}

// Every K-window adds one to the slot of its candidate (native.cu:244); with
// compact (K-1)-mer tables every (K-1)-window also adds one to its count.  A
// thread's windows go through the dependent steps together (codes, rank loads,
// counts, offsets and masks, slot atomics), so their loads are in flight at once.
// The L2 requests, not the latency of the loads, set the pace: four windows per thread
// instead of two measured no faster, and one 64-bit atomic for count and offset instead
// of an atomic and a load took the build of 200 uneven proteomes from 22.2 to 21.0 ms.
__global__ void __launch_bounds__(COUNT_THREADS) k_c0_scatter(BuildArgs a) {
    previous_kernel_done();
    __shared__ uint8_t dig[TILE + 16];
    const int K = a.k;
    const uint32_t A = a.A;
    const uint64_t total_tiles = a.tile_base[a.B];
    for (uint64_t t = blockIdx.x; t < total_tiles; t += gridDim.x) {
        const int p = find_owner(a.tile_base, a.B, t);
        const uint64_t s0 = a.seq_off[p], len = a.seq_off[p + 1] - s0;
        const uint64_t start = (t - a.tile_base[p]) * TILE;
        for (int j = threadIdx.x; j < TILE + K; j += COUNT_THREADS) {
            uint64_t pos = start + j;
            dig[j] = pos < len ? (uint8_t)char_to_digit(a.alpha, a.seq[s0 + pos]) : (uint8_t)0xff;
        }
        __syncthreads();
        const uint64_t cbase = a.cbase[p];
        constexpr int NU = TILE / COUNT_THREADS;
        // phase 1: every window's (K-1)- and (K-2)-mer codes from the staged digits
        uint32_t w[NU], w2[NU], bd[NU];
        int jj[NU];
#pragma unroll
        for (int u = 0; u < NU; u++) {
            const int li = u * COUNT_THREADS + threadIdx.x;
            w[u] = 0;
            w2[u] = 0;
            bd[u] = 0xffu;
            jj[u] = -1;
            if (start + li < len) {
                uint32_t x = 0, x2 = 0;
                int j;
                for (j = 0; j < K - 1; j++) {
                    if (j == K - 2) x2 = x;
                    uint32_t d = dig[li + j];
                    if (d == 0xffu) break;
                    x = x * A + d;
                }
                w[u] = x;
                w2[u] = x2;
                jj[u] = j;
                bd[u] = dig[li + K - 1];
            }
        }
        // phase 2: all rank loads in flight together
        uint64_t wi[NU], mi[NU];
#pragma unroll
        for (int u = 0; u < NU; u++) {
            wi[u] = jj[u] == K - 1 ? c1_index(a, p, w[u]) : ~0ull;
            mi[u] = (a.compact2 && jj[u] >= K - 2) ? c2_index(a, p, w2[u]) : ~0ull;
        }
        // phase 3: counts, then the candidate offsets and extension masks together
        uint32_t co[NU], em[NU];
#pragma unroll
        for (int u = 0; u < NU; u++) {
            co[u] = 0;
            em[u] = 0;
            if (mi[u] < a.cap2) atomicAdd(&a.c2[mi[u]], 1u);
            if (wi[u] != ~0ull) {
                const bool in_cap = !a.compact1 || wi[u] < a.cap1;
                if (a.compact1 && in_cap)
                    co[u] = (uint32_t)(atomicAdd((unsigned long long *)&a.cc[wi[u]], 1ull) >> 32);
                if (!in_cap || bd[u] == 0xffu) wi[u] = ~0ull;
            }
        }
#pragma unroll
        for (int u = 0; u < NU; u++) {
            if (wi[u] != ~0ull) {
                if (!a.compact1) co[u] = __ldg(&a.coff[wi[u]]);
                em[u] = ext_mask(a, p, a.fdT2.mod(w[u]));
            }
        }
#pragma unroll
        for (int u = 0; u < NU; u++) {
            if (wi[u] != ~0ull) {
                const uint64_t slot = cbase + co[u] + __popc(em[u] & ((1u << bd[u]) - 1u));
                if (slot < a.cand_cap) atomicAdd(&a.c0a[slot], 1u);
            }
        }
        __syncthreads();
    }
}

// Markov alpha of every candidate (alpha bits replace the count, as
// native.cu:399 does), flat over the batch's candidate index space: CTA c takes
// candidates [c * ALPHA_TILE, (c + 1) * ALPHA_TILE) of one proteome, warp w the
// segment of SEG candidates starting at c * ALPHA_TILE + w * SEG.  In place: a
// seen candidate's c0a slot receives its alpha bits (or TUPLE_TAG | tuple), or
// CAND_DROP when alpha is 0 (not written out); an unseen one keeps count 0 and
// stands for alpha -1.  seg_surv = survivors per segment.  Per-CTA norm
// partials.  grid = cand_cap / ALPHA_TILE
//
// Most candidates are K-mers that were not seen (count 0): their alpha is -1
// (native.cu:392 with p = 0) and needs no table loads.  The others are listed
// per warp in shared memory and computed densely, 32 lanes on 32 of them, so
// the long path does not run with most lanes idle.
constexpr int ALPHA_ILP = 1;  // listed candidates per lane in flight together
// c0a value of a seen candidate whose alpha is 0: not written out.  No tuple tag
// (tuple indices stay below TUPLE_TABLE) and no alpha (arithmetic NaNs are
// 0x7fffffff) has these bits.
constexpr uint32_t CAND_DROP = 0xffffffffu;
__global__ void __launch_bounds__(CHUNK_THREADS, 6) k_alpha(BuildArgs a) {
    previous_kernel_done();
    __shared__ U192 s_norm[CHUNK_THREADS / 32];
    __shared__ uint32_t s_m1[CHUNK_THREADS / 32], s_bad[CHUNK_THREADS / 32],
        s_surv[CHUNK_THREADS / 32];
    __shared__ uint32_t s_lcnt[CHUNK_THREADS / 32][SEG];   // listed candidates: K-mer count,
    __shared__ uint16_t s_lidx[CHUNK_THREADS / 32][SEG];   // index in the segment
    const uint64_t c = blockIdx.x;
    const uint64_t g0 = c * ALPHA_TILE;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint64_t seg = c * (ALPHA_TILE / SEG) + w;
    const uint64_t total = min(*a.cand_total, a.cand_cap);
    if (g0 >= total) return;  // past the last proteome: k_norm and k_compact stop there too
    // out of room: the ranks below may lie past the count tables, and nothing is kept
    if (*a.status) return;
    const int p = find_owner(a.cbase, a.B, g0);
    const uint32_t np =
        (uint32_t)(a.chunk_cand_off[(uint64_t)(p + 1) * a.NCH] - a.chunk_cand_off[(uint64_t)p * a.NCH]);
    const double *prob = a.prob + (uint64_t)p * 4 * PROB_TABLE;
    const uint32_t *atab = a.atab + (uint64_t)p * TUPLE_TABLE;
    const uint32_t n0 = a.tot[p * 4 + 0], n1 = a.tot[p * 4 + 1], n2 = a.tot[p * 4 + 2];
    const uint32_t A = a.A;
    const uint64_t sbase = g0 + (uint64_t)w * SEG;           // this warp's segment
    const uint32_t loc0 = (uint32_t)(sbase - a.cbase[p]);    // proteome-local index of its start
    U192 acc = {0, 0, 0};
    uint32_t m1 = 0, bad = 0, ndrop = 0;
    constexpr int NI = SEG / 32;  // candidates per lane
    // phase 1: K-mer counts of the whole segment; candidates that need the long path
    // (a seen K-mer, or a proteome without K-windows) are listed
    uint32_t fl[NI];
#pragma unroll
    for (int i = 0; i < NI; i++) {
        const bool ok = loc0 + 32 * i + lane < np;
        fl[i] = ok ? a.c0a[sbase + 32 * i + lane] : 0u;
    }
    uint32_t nlist = 0, nok = 0;
#pragma unroll
    for (int i = 0; i < NI; i++) {
        const bool ok = loc0 + 32 * i + lane < np;
        const bool need = ok && (fl[i] != 0u || n0 == 0u);
        if (ok && !need) m1++;  // an unseen K-mer: alpha -1, square 1
        nok += ok;
        const unsigned bal = __ballot_sync(0xffffffffu, need);
        if (need) {
            const uint32_t pos = nlist + __popc(bal & ((1u << lane) - 1u));
            s_lcnt[w][pos] = fl[i];
            s_lidx[w][pos] = (uint16_t)(32 * i + lane);
        }
        nlist += __popc(bal);
    }
    __syncwarp();
    // phase 2: the listed candidates, ALPHA_ILP per lane with their loads in flight together
    for (uint32_t t0 = 0; t0 < nlist; t0 += 32 * ALPHA_ILP) {
        uint32_t key[ALPHA_ILP], full[ALPHA_ILP], pre[ALPHA_ILP], mid[ALPHA_ILP], suf[ALPHA_ILP];
#pragma unroll
        for (int j = 0; j < ALPHA_ILP; j++) {
            const uint32_t t = t0 + 32 * j + lane;
            const bool ok = t < nlist;
            key[j] = ok ? a.cq[sbase + s_lidx[w][t]] : 0u;
            full[j] = ok ? s_lcnt[w][t] : 0u;
            const uint32_t q = A == 21u ? key[j] / 21u : key[j] >> 2;  // protein or DNA alphabet
            const uint32_t b = key[j] - q * A;
            const uint32_t m = a.fdT2.mod(q);
            const bool seen = ok && full[j] != 0u;
            pre[j] = seen ? c1_load(a, c1_index(a, p, q)) : 0u;
            const uint64_t mi = seen ? c2_index(a, p, m) : 0;
            mid[j] = seen && (!a.compact2 || mi < a.cap2) ? __ldg(&a.c2[mi]) : 0u;
            suf[j] = seen ? c1_load(a, c1_index(a, p, m * A + b)) : 0u;
        }
#pragma unroll
        for (int j = 0; j < ALPHA_ILP; j++) {
            const uint32_t t = t0 + 32 * j + lane;
            if (t >= nlist) continue;
            uint32_t stored;
            float f;
            if (full[j] - 1u < 3u && pre[j] < (uint32_t)TUPLE_PS && suf[j] < (uint32_t)TUPLE_PS &&
                mid[j] < (uint32_t)TUPLE_MID && n0 != 0u) {
                const uint32_t ti =
                    ((full[j] * TUPLE_PS + pre[j]) * TUPLE_PS + suf[j]) * TUPLE_MID + mid[j];
                const uint32_t tb = __ldg(&atab[ti]);
                f = __uint_as_float(tb);
                stored = tb ? (TUPLE_TAG | ti) : 0u;
            } else {
                f = markov_alpha_fast(full[j], pre[j], suf[j], mid[j], n0, n1, n2, prob);
                stored = __float_as_uint(f);
            }
            // in place: the alpha bits (or tuple tag), or CAND_DROP for alpha 0
            a.c0a[sbase + s_lidx[w][t]] = stored ? stored : CAND_DROP;
            ndrop += stored == 0u;
            if (__float_as_uint(f) != 0u) {
                const float sq = __fmul_rn(f, f);  // float square, as native.cu:421-423
                if (sq == 1.0f) m1++;
                else if (isnan(sq)) bad |= 1u;
                else if (isinf(sq) || !u192_add_float(acc, sq)) bad |= 2u;
            }
        }
    }
    // phase 3: survivors of the segment (k_compact copies them out in place order)
    const uint32_t nsurv = __reduce_add_sync(0xffffffffu, nok - ndrop);
    if (lane == 0) a.seg_surv[seg] = nsurv;
    // norm partials (integer: exact and order independent)
    m1 = __reduce_add_sync(0xffffffffu, m1);
    bad = __reduce_or_sync(0xffffffffu, bad);
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        const U192 o = u192_shfl_down(acc, d);
        u192_add(acc, o.w0, o.w1, o.w2);
    }
    if (lane == 0) {
        s_norm[w] = acc; s_m1[w] = m1; s_bad[w] = bad; s_surv[w] = nsurv;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        U192 t = {0, 0, 0};
        uint32_t tm = 0, tb = 0, ts = 0;
        for (int i = 0; i < CHUNK_THREADS / 32; i++) {
            u192_add(t, s_norm[i].w0, s_norm[i].w1, s_norm[i].w2);
            tm += s_m1[i];
            tb |= s_bad[i];
            ts += s_surv[i];
        }
        a.cta_surv[c] = ts;
        a.cta_m1[c] = tm;
        a.cta_bad[c] = tb;
        a.cta_norm[3 * c + 0] = t.w0;
        a.cta_norm[3 * c + 1] = t.w1;
        a.cta_norm[3 * c + 2] = t.w2;
    }
}

// Per proteome: norm = exact sum of the squares rounded once to double
// (native.cu:415-428 sums the same float squares in double, in CUB's order),
// scale = sqrt(norm), its reciprocal, nnz, and cta_out[c] = survivors of the proteome
// before k_alpha CTA c.  grid = B, NORM_THREADS threads (the CTA partials of a proteome
// summed exactly, in any order).
constexpr int NORM_THREADS = 512, NORM_ITEMS = 4;
__global__ void __launch_bounds__(NORM_THREADS) k_norm(BuildArgs a) {
    previous_kernel_done();
    __shared__ U192 s_acc[NORM_THREADS / 32];
    __shared__ uint64_t s_m1[NORM_THREADS / 32], sw[NORM_THREADS / 32 + 1];
    __shared__ uint32_t s_bad[NORM_THREADS / 32];
    const int p = blockIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t ncta = a.cand_cap / ALPHA_TILE;
    const uint64_t c0 = min(a.cbase[p] / ALPHA_TILE, ncta);
    // out of room, k_alpha left no partials: no entries
    const uint64_t c1 = *a.status ? c0 : min(a.cbase[p + 1] / ALPHA_TILE, ncta);
    U192 acc = {0, 0, 0};
    uint64_t m1 = 0, run = 0;
    uint32_t bad = 0;
    for (uint64_t base = c0; base < c1; base += NORM_THREADS * NORM_ITEMS) {
        const uint64_t first = base + (uint64_t)threadIdx.x * NORM_ITEMS;
        uint32_t v[NORM_ITEMS];
        uint64_t s = 0, tot;
#pragma unroll
        for (int i = 0; i < NORM_ITEMS; i++) {
            const uint64_t c = first + i;
            v[i] = 0;
            if (c < c1) {
                u192_add(acc, a.cta_norm[3 * c], a.cta_norm[3 * c + 1], a.cta_norm[3 * c + 2]);
                m1 += a.cta_m1[c];
                bad |= a.cta_bad[c];
                v[i] = a.cta_surv[c];
            }
            s += v[i];
        }
        uint64_t e = run + block_excl_scan_u64<NORM_THREADS>(s, sw, &tot);
        run += tot;
#pragma unroll
        for (int i = 0; i < NORM_ITEMS; i++) {
            if (first + i < c1) a.cta_out[first + i] = (uint32_t)e;
            e += v[i];
        }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        const U192 o = u192_shfl_down(acc, d);
        u192_add(acc, o.w0, o.w1, o.w2);
        m1 += __shfl_down_sync(0xffffffffu, m1, d);
    }
    bad = __reduce_or_sync(0xffffffffu, bad);
    if (lane == 0) {
        s_acc[warp] = acc;
        s_m1[warp] = m1;
        s_bad[warp] = bad;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        acc = s_acc[0];
        m1 = s_m1[0];
        bad = s_bad[0];
        for (int w = 1; w < NORM_THREADS / 32; w++) {
            u192_add(acc, s_acc[w].w0, s_acc[w].w1, s_acc[w].w2);
            m1 += s_m1[w];
            bad |= s_bad[w];
        }
        // each unit square adds 1.0 = 2^96 units: bit 32 of the middle word
        u192_add(acc, 0, m1 << 32, m1 >> 32);
        double norm = u192_to_double(acc);
        if (bad & 1u) norm = __longlong_as_double(0x7ff8000000000000ll);
        else if (bad & 2u) norm = __longlong_as_double(0x7ff0000000000000ll);
        const double scale = __dsqrt_rn(norm);
        a.norm[p] = norm;
        a.scale[p] = scale;
        a.rscale[p] = __ddiv_rn(1.0, scale);
        a.nnz[p] = run;
        if (a.host_result) *a.host_result = {run, norm, *a.cand_total, *a.status, 0u};
    }
}

// Marks in the key bitmap, for every seen (K-1)-mer q of the batch, the keys
// q * A + b of its candidates (b over the right-extension mask of q's suffix):
// one or two atomics per seen (K-1)-mer instead of one per written key.  The
// marked set is a superset of the written keys (a candidate whose alpha is 0 is
// marked but not written), which is all a key-rank bitmap needs: ranks stay
// strictly increasing over the written keys.  grid = (words / (CHUNK_THREADS * wpt), B), or
// WIDE (K = 7) its transpose: the bitmap (225 MB) is larger than L2 there, and the batch's
// proteomes mark the same stretch of it at a time (12 uneven proteomes: 203 -> 162 us; at K =
// 6, where it stays in L2, they would only meet in its words: 111 -> 120).
template <bool WIDE>
__global__ void __launch_bounds__(CHUNK_THREADS) k_union_mark(BuildArgs a) {
    previous_kernel_done();
    const int p = WIDE ? blockIdx.x : blockIdx.y;
    const uint64_t nw = a.T1s / 32;
    const uint64_t wd0 = (uint64_t)(WIDE ? blockIdx.y : blockIdx.x) * CHUNK_THREADS * a.wpt + threadIdx.x;
    for (uint32_t i = 0; i < a.wpt; i++) {
        const uint64_t wd = wd0 + i * CHUNK_THREADS;
        if (wd >= nw) break;
        uint32_t bits = a.seen1[(uint64_t)p * nw + wd];
        while (bits) {
            const uint32_t q = (uint32_t)(wd * 32) + (uint32_t)(__ffs(bits) - 1);
            bits &= bits - 1;
            const uint32_t m = ext_mask(a, p, a.fdT2.mod(q));
            if (!m) continue;
            const uint64_t bit = (uint64_t)q * a.A;
            const uint64_t w = bit >> 5;
            const uint32_t off = (uint32_t)bit & 31u;
            atomicOr(&a.union_bits[w], m << off);
            if (off + a.A > 32u && (m >> (32u - off))) atomicOr(&a.union_bits[w + 1], m >> (32u - off));
        }
    }
}

// Copies every segment's survivors to the output, in key order: keys and
// float(alpha / scale) (native.cu:460-468).  A candidate with count 0 is an
// unseen K-mer (alpha -1); one marked CAND_DROP had alpha 0 and is skipped.  The
// division by the per-proteome constant scale uses its correctly rounded
// reciprocal and one FMA correction (Markstein), which yields the correctly
// rounded double quotient.  Most segments drop nothing and move as they are, eight
// entries per lane in flight; the others place theirs by ballots, at three times the
// instructions (with ballots throughout, 62% of the issue slots: 200 uneven proteomes
// 22.2 -> 21.7 ms).  grid = cand_cap / ALPHA_TILE, and for a single proteome
// a.pad_blocks more, which fill the rest of its output with the padding of
// native.cu:473-474; a single proteome that does not fit leaves its output as it is.
__global__ void __launch_bounds__(CHUNK_THREADS) k_compact(BuildArgs a) {
    previous_kernel_done();
    __shared__ uint64_t s_base[SMEM_BASES + 1];
    if (a.single && (*a.status || a.nnz[0] > a.single_cap)) return;
    const uint64_t c = blockIdx.x, g0 = c * ALPHA_TILE, ncta = a.cand_cap / ALPHA_TILE;
    if (c >= ncta) {
        for (uint64_t i = a.nnz[0] + (c - ncta) * CHUNK_THREADS + threadIdx.x; i < a.single_cap;
             i += (uint64_t)a.pad_blocks * CHUNK_THREADS) {
            a.out_keys[i] = 0xffffffffu;
            a.out_vals[i] = 0.0f;
        }
        return;
    }
    if (g0 >= min(*a.cand_total, a.cand_cap)) return;
    const uint64_t *cb = stage_bases(a.cbase, a.B, s_base);
    const int p = find_owner(cb, a.B, g0);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint64_t seg = c * (ALPHA_TILE / SEG) + w;
    // survivors of the CTA's segments: this warp's come after those of the earlier ones
    const uint32_t nsurv = lane <= w ? a.seg_surv[c * (ALPHA_TILE / SEG) + lane] : 0u;
    if (__shfl_sync(0xffffffffu, nsurv, w) == 0) return;
    const uint32_t before = __reduce_add_sync(0xffffffffu, lane < w ? nsurv : 0u);
    const uint64_t src = seg * SEG;
    const uint32_t np =
        (uint32_t)(a.chunk_cand_off[(uint64_t)(p + 1) * a.NCH] - a.chunk_cand_off[(uint64_t)p * a.NCH]);
    const uint32_t loc0 = (uint32_t)(src - cb[p]);
    const uint32_t nc = loc0 < np ? min((uint32_t)SEG, np - loc0) : 0u;  // its candidates
    const uint64_t dst = a.dst_base[p] + a.cta_out[c] + before;
    const uint64_t dst_end = a.dst_base[p] + a.dst_cap[p];
    const double scale = a.scale[p];
    const double rs = a.rscale[p];
    const float *vtab = a.vtab + (uint64_t)p * TUPLE_TABLE;
    const bool finite = isfinite(scale) && scale > 0.0;
    const float vm1 = __double2float_rn(-rs);  // RN(-1/scale) == -RN(1/scale)
    auto value = [&](uint32_t b) {
        if (b == 0u) return vm1;  // unseen K-mer: alpha -1
        if ((b & TUPLE_TAG) == TUPLE_TAG) return __ldg(&vtab[b & ~TUPLE_TAG]);
        const float f = __uint_as_float(b);
        if (!finite || !isfinite(f)) return __double2float_rn(__ddiv_rn((double)f, scale));
        return f == -1.0f ? vm1 : div_by_scale(f, scale, rs);
    };
    if (__shfl_sync(0xffffffffu, nsurv, w) == nc && dst + nc <= dst_end) {
        // nothing dropped: the segment moves as it is
        constexpr int V = SEG / 32;
        uint32_t bits[V], key[V];
#pragma unroll
        for (int u = 0; u < V; u++) {
            const uint32_t i = 32 * u + lane;
            bits[u] = i < nc ? a.c0a[src + i] : 0u;
            key[u] = i < nc ? a.cq[src + i] : 0u;
        }
#pragma unroll
        for (int u = 0; u < V; u++) {
            const uint32_t i = 32 * u + lane;
            if (i < nc) {
                a.out_keys[dst + i] = key[u];
                a.out_vals[dst + i] = value(bits[u]);
            }
        }
        return;
    }
    // four candidates per lane in flight: loads first, then the stores
    constexpr int U = 4;
    uint32_t out = 0;  // survivors written so far
    for (uint32_t i0 = 0; i0 < nc; i0 += 32 * U) {
        uint32_t bits[U], key[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const uint32_t i = i0 + 32 * u + lane;
            bits[u] = i < nc ? a.c0a[src + i] : CAND_DROP;
            key[u] = i < nc ? a.cq[src + i] : 0u;
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const bool surv = bits[u] != CAND_DROP;
            const unsigned bal = __ballot_sync(0xffffffffu, surv);
            if (surv) {
                const float v = value(bits[u]);
                const uint64_t o = dst + out + __popc(bal & ((1u << lane) - 1u));
                if (o < dst_end) {
                    a.out_keys[o] = key[u];
                    a.out_vals[o] = v;
                }
            }
            out += __popc(bal);
        }
    }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------

int build_geometry(int alpha, int k, BuildGeometry *g) {
    if (alpha != ALPHA_PROTEIN && alpha != ALPHA_DNA) return -1;
    if (k < 3 || k > 10) return -1;
    const uint64_t A = alphabet_size(alpha);
    if (ipow64(A, k) > 0xffffffffull) return -2;  // keys must fit uint32
    g->alpha = alpha;
    g->k = k;
    g->A = (uint32_t)A;
    g->T1 = ipow64(A, k - 1);
    g->T1s = (g->T1 + 31) / 32 * 32;  // whole words of the seen bitmap
    g->T2 = ipow64(A, k - 2);
    g->T2s = (g->T2 + 31) / 32 * 32;
    g->wpt = g->T1s > (1ull << 24) ? MAX_WPT : 1;  // sparse bitmaps: eight words per thread
    return 0;
}

// Lanes with words per warp of the candidate passes for B proteomes: 32, or 8 or 2 where
// that leaves fewer than MIN_CHUNKS CTAs.  A word's (K-1)-mers share all but their last
// symbols, so its work goes with the frequencies of those symbols, and with few CTAs
// the densest words are what the pass waits for (one proteome of 1,500 proteins at K = 6,
// 499 CTAs: k_cand_offsets 30 us at 22% of the warp slots; with 1,995 the whole call
// 141 -> 135 us; 3,000 proteins at K = 5, 24 -> 380 CTAs: 234 -> 180 us).  Proteomes of
// few residues have no such words, and at K = 6 the extra CTAs cost more than they give
// (30 proteins: 97 -> 112 us): build_plan keeps 32 there.
constexpr uint64_t MIN_CHUNKS = 1500, SHORT_PROTEOME = 1u << 18;
static uint32_t chunk_lanes(const BuildGeometry &g, int B) {
    uint32_t lanes = 32;
    if (g.wpt == 1)
        while (lanes > 2 && (uint64_t)B * div_up(g.T1s / 32, CHUNK_THREADS / 32 * lanes) < MIN_CHUNKS)
            lanes /= 4;
    return lanes;
}

// (K-1)-mer tables beyond 2^20 entries per proteome (protein K >= 6) are kept
// compact: one entry per seen (K-1)-mer instead of a dense row.  A batch's
// dense rows (16 MB per proteome at K = 6) would live in DRAM, so every
// (K-1)-window's count would be a DRAM atomic; the compact entries of a batch
// stay in L2, and the zeroing of the dense rows goes away.
static bool compact1_tables(const BuildGeometry &g) { return g.T1s > (1ull << 20); }
// (K-2)-mer counts likewise beyond 2^20 entries (protein K = 7: 16 MB per proteome).
static bool compact2_tables(const BuildGeometry &g) { return g.T2s > (1ull << 20); }

// Candidate capacity rounded up to whole k_alpha CTAs.
static uint64_t cand_cap_rounded(uint64_t cand_cap) {
    return div_up(cand_cap ? cand_cap : 1, (uint64_t)ALPHA_TILE) * ALPHA_TILE;
}

// One description of the scratch for both its size and its addresses: `take` is called
// with every array in order.
template <typename Take>
static void build_layout(const BuildGeometry &g, int B, uint64_t cand_cap, BuildArgs &r, Take &&take) {
    r.wpt = g.wpt;
    r.wlanes = chunk_lanes(g, B);
    r.NCH = div_up(g.T1s / 32, (uint64_t)(CHUNK_THREADS / 32) * r.wlanes * r.wpt);
    const uint64_t nc = (uint64_t)B * r.NCH;
    const uint64_t cap = cand_cap_rounded(cand_cap);
    const uint64_t ncta = cap / ALPHA_TILE, nseg = cap / SEG;
    const uint64_t nw1 = g.T1s / 32 * B, nw2 = g.T2s / 32 * B;
    const bool compact = compact1_tables(g), compact2 = compact2_tables(g);
    r.alpha = g.alpha; r.k = g.k; r.A = g.A; r.T1 = g.T1; r.T2 = g.T2; r.B = B;
    r.T1s = g.T1s;
    r.T2s = g.T2s;
    r.fdT2.set((uint32_t)g.T2);
    r.compact1 = compact ? 1 : 0;
    r.compact2 = compact2 ? 1 : 0;
    r.cap1 = compact ? cap : g.T1s * B;
    r.cap2 = compact2 ? cap : g.T2 * B;
    r.cand_cap = cap;
    // zeroed by k_begin: tot up to c1 (dense) or coff
    take(r.tot, 4 * (uint64_t)B);
    take(r.seen1, nw1);
    take(r.seen2, compact2 ? nw2 : 0);
    if (!compact2) take(r.c2, r.cap2);
    // At the smallest K these and c1 are a few lines that take every window's atomics, and side
    // by side they meet in the L2 or not as the scratch's address has it: 12,000 proteins at
    // K = 3 took 1,012 to 1,448 us over forty addresses, with 4 KB between them 1,002 to 1,141.
    uint32_t *apart = nullptr;
    take(apart, 1024);
    if (!compact) take(r.c1, r.cap1);
    take(r.coff, compact ? 0 : r.cap1);
    take(r.cc, compact ? r.cap1 : 0);
    if (compact2) take(r.c2, r.cap2);
    take(r.pw1, compact ? nw1 : 0);
    take(r.p1_total, 1);
    take(r.word_cand, g.wpt > 1 ? 0 : nw1);
    take(r.warp_cs, g.wpt > 1 ? nc * (CHUNK_THREADS / 32) : 0);
    take(r.pw2, compact2 ? nw2 : 0);
    take(r.p2_partials, compact2 ? bitmap_prefix_partials(nw2) : 0);
    take(r.p2_total, 1);
    take(r.seq_off_store, B + 1);
    take(r.tile_base, B + 1);
    take(r.chunk_cand, nc);
    take(r.chunk_seen, nc);
    take(r.chunk_cand_off, nc + 1);
    take(r.chunk_seen_off, nc);
    take(r.cbase, B + 1);
    take(r.seg_surv, nseg);
    take(r.cta_surv, ncta);
    take(r.cta_out, ncta);
    take(r.cta_m1, ncta);
    take(r.cta_norm, 3 * ncta);
    take(r.cta_bad, ncta);
    take(r.prob, 4 * (uint64_t)PROB_TABLE * B);
    take(r.atab, (uint64_t)TUPLE_TABLE * B);
    take(r.vtab, (uint64_t)TUPLE_TABLE * B);
    take(r.scale, B);
    take(r.rscale, B);
    take(r.dst_base, B);
    take(r.dst_cap, B);
    // the results, as the host reads them: nnz[B] | norm[B] | cand_total | status
    take(r.nnz, 2 * (uint64_t)B + 2);
    take(r.c0a, cap);
    take(r.cq, cap);
}

size_t build_scratch_bytes(const BuildGeometry &g, int B, uint64_t cand_cap) {
    BuildArgs r;
    size_t s = 0;
    build_layout(g, B, cand_cap, r, [&](auto *&p, uint64_t n) { s += round256(n * sizeof(*p)); });
    return s;
}

cudaError_t build_carve(const BuildGeometry &g, int B, uint64_t cand_cap, void *scratch,
                        size_t scratch_size, BuildArgs *a) {
    Scratch sc(scratch, scratch_size);
    BuildArgs &r = *a;
    bool ok = true;
    build_layout(g, B, cand_cap, r, [&](auto *&p, uint64_t n) {
        p = sc.take<std::remove_reference_t<decltype(*p)>>(n);
        ok = ok && p;
    });
    if (!ok) return cudaErrorInvalidValue;  // scratch too small
    r.zero = (uint64_t *)r.tot;
    r.zero_n8 = ((char *)r.coff - (char *)r.tot) / sizeof(uint64_t);
    r.norm = (double *)(r.nnz + B);
    r.cand_total = r.nnz + 2 * (uint64_t)B;
    r.status = (uint32_t *)(r.cand_total + 1);
    return cudaSuccess;
}

// Phase 1: everything up to per-proteome nnz (no host sync inside).
cudaError_t build_plan(BuildArgs &a, cudaStream_t st) {
    if (a.single && a.compact1 && a.wpt == 1 && a.single_len < SHORT_PROTEOME) {
        a.wlanes = 32;
        a.NCH = div_up(a.T1s / 32, (uint64_t)CHUNK_THREADS);
    }
    const int sms = device_sm_count();
    const uint64_t zero_blocks = div_up(a.zero_n8, 4 * 256);
    const unsigned B = (unsigned)a.B, nch = (unsigned)a.NCH;
    PHYLO_CHECK(launch_next(k_begin,
                            (unsigned)max((uint64_t)1, min(zero_blocks, (uint64_t)sms * 8)), 256,
                            st, a));
    const int grid_seq = sms * 8;
    PHYLO_CHECK(launch_next(a.compact1 ? k_count<true> : k_count<false>, grid_seq, COUNT_THREADS,
                            st, a));
    if (a.compact2)  // ranks of the seen (K-2)-mers
        PHYLO_CHECK(bitmap_prefix_pairs(a.seen2, a.T2s / 32 * a.B, a.p2_partials, a.pw2,
                                        a.p2_total, st));
    PHYLO_CHECK(launch_next(a.wpt > 1 ? k_cand_count<true> : k_cand_count<false>,
                            dim3(nch + PROB_BLOCKS + TUPLE_BLOCKS, B), CHUNK_THREADS, st, a));
    PHYLO_CHECK(launch_next(k_cand_scan, 1, CSCAN_THREADS, st, a));
    PHYLO_CHECK(launch_next(a.wpt > 1 ? k_cand_offsets<true> : k_cand_offsets<false>, dim3(nch, B),
                            CHUNK_THREADS, st, a));
    PHYLO_CHECK(launch_next(k_c0_scatter, grid_seq, COUNT_THREADS, st, a));
    PHYLO_CHECK(launch_next(k_alpha, (unsigned)(a.cand_cap / ALPHA_TILE), CHUNK_THREADS, st, a));
    PHYLO_CHECK(launch_next(k_norm, B, NORM_THREADS, st, a));
    PHYLO_CHECK(launch_next(k_tuple_value, dim3(TUPLE_TABLE / 256, B), 256, st, a));
    return cudaGetLastError();
}

// Phase 2: write survivors to out_keys/out_vals at dst_base[p] (capacity dst_cap[p]).
cudaError_t build_emit(BuildArgs &a, cudaStream_t st) {
    const uint64_t ncta = a.cand_cap / ALPHA_TILE;
    if (a.single)
        a.pad_blocks = (unsigned)min(div_up(a.single_cap ? a.single_cap : 1, 8 * CHUNK_THREADS),
                                     (uint64_t)device_sm_count() * 8);
    PHYLO_CHECK(launch_next(k_compact, (unsigned)(ncta + a.pad_blocks), CHUNK_THREADS, st, a));
    if (a.union_bits) {
        const unsigned words = (unsigned)div_up(a.T1s / 32, (uint64_t)CHUNK_THREADS * a.wpt);
        PHYLO_CHECK(a.wpt > 1 ? launch_next(k_union_mark<true>, dim3((unsigned)a.B, words),
                                            CHUNK_THREADS, st, a)
                              : launch_next(k_union_mark<false>, dim3(words, (unsigned)a.B),
                                            CHUNK_THREADS, st, a));
    }
    return cudaGetLastError();
}

// Kernels one batched Plan + Emit launches: plan k_begin, k_count, k_cand_count,
// k_cand_scan, k_cand_offsets, k_c0_scatter, k_alpha, k_norm, k_tuple_value (and three
// for the (K-2)-mer ranks of protein K = 7); emit k_arena_offsets, k_compact,
// k_union_mark (with a key bitmap).
int build_launches_per_batch() { return 9 + 3; }

}  // namespace phylo
