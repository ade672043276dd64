// Products of the sphere Hamiltonians by splitting the Fock word into two
// parts (K20): y = H x without reading one stored element per hop.
//
// A sector word is a primary part P and a secondary part S (one level: the
// high and low orbitals of the word; two levels: the two levels' words).  The
// sector fixes the class (popcount, weight sum) that S must have for a given
// P, so the rows of one P are a contiguous segment of x indexed by the rank
// of S in its class.  A pair hop acts on the two parts separately:
//   <P S|H|P' S'> = sum over gamma of W_gamma(P -> P') s_gamma(S -> S'),
// gamma being what happens to S: nothing, one orbital emptied or filled, or
// one particle moved.  For a given gamma the weight and P' depend on P alone
// and S' and the sign s on S alone, so
//   y[P, S] += s_gamma(S) * sum_alpha W_alpha x[P'_alpha, rank(S'_gamma)]
// where the list of (P'_alpha, W_alpha) is read once for a whole segment of
// rows, and the list of (S, S', sign) is shared by every P of the class.  The
// elements are neither stored nor generated one by one: a list entry stands
// for tens to hundreds of them, the weights are the same for all lanes of a
// warp, and the gathers of x run along a segment.  (The stored-matrix kernels
// are bound by L1 gather wavefronts: a warp's 32 gathers of a CRS row hit
// 12 different lines on average and take 13 of its 19 wavefronts per 32
// elements, 87 % of the L1's rate.)
//
// Two passes cover all hops: the native pass (P = high part, rows in the
// basis order) takes the hops that leave S alone, change one of its orbitals
// or move one of its particles; the transposed pass (P = low part, rows
// ordered low part first) takes the rest: hops inside the low part and those
// that change one orbital of the high part.  Two levels have only the two
// "nothing happens to S" lists (no term mixes the levels).
//
// Arithmetic: ed_fixed.cuh's exact fixed point, as the stored products use
// it: 58-bit weights and x, exact 128-bit sums, one rounding per row, so the
// result does not depend on the order of the hops and equals theirs bit for
// bit (the same exponent bounds).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <numeric>

#include "ed_fixed.cuh"
#include "ed_hop.cuh"
#include "ed_split.h"

namespace edgb {

namespace {

constexpr int kThreads = 64;
constexpr int kWarps = kThreads / 32;
constexpr int kSegRows = 256;        // rows of one segment of a block
constexpr int kIdRows = 2;               // 32-row groups a warp of k_split_keep sums at once

// change-list entries: row | new rank << 8 | sign << 31; move-list entries:
// new rank | weight << 13 | row << 19 | count << 27 | null << 31
constexpr int kRankBits = 13, kWeightShift = 13, kRowShift = 19, kCountShift = 27;
constexpr uint32_t kRankMask = (1u << kRankBits) - 1u;
constexpr uint32_t kNullEntry = 1u << 31;
constexpr int kRowBits = 8;
constexpr int kMaxMovable = 12;      // of kMaxSideBits orbitals, by one distance
static_assert(kSegRows == 1 << kRowBits, "row field");

enum GammaType { kKeep = 0, kEmpty = 1, kFill = 2 };   // and the moves, in lists of their own
constexpr int kKeepParts = 8;        // kKeep's alpha entries are listed in so many parts, one after another
constexpr int kMaxSideBits = 24;     // tables over one part's words (PartArgs::w)

int sms()
{
    int dev = 0, s = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&s, cudaDevAttrMultiProcessorCount, dev);
    return s;
}

// What the generation kernels know of one pass.  Orbital numbers are those
// of the weight table (global for one level, the level's own for two).
struct GenArgs {
    int plo, pbits;                 // primary orbitals plo .. plo + pbits - 1
    int slo, sbits;                 // secondary ones
    int gammas;
    const int* gamma;               // type | o << 4
    int K;                          // weight table: orbitals, values, pair-sum offsets
    const double* w;
    const int* off;
};

__device__ __forceinline__ double hop_weight(const GenArgs& g, int a, int b, int c)
{
    // the stored element's orientation: the lower word's side (hop_bits)
    const int s = a + b, lo = pair_lo(s, g.K), cnt = pair_cnt(s, g.K);
    const int idx = c < a ? (a - lo) * cnt + (c - lo) : (c - lo) * cnt + (a - lo);
    return g.w[g.off[s] + idx];
}

// f(P', weight with the primary part's sign) for every hop of the primary
// word P (local bits) that does gamma to the secondary word.
template <class F>
__device__ __forceinline__ void for_alpha(const GenArgs& g, uint32_t P, int gm, F&& f)
{
    const int type = gm & 15, o = gm >> 4;
    const uint64_t W = (uint64_t)P << g.plo;
    const int plo = g.plo, phi = g.plo + g.pbits;
    auto emit = [&](int a, int b, int c, int d, uint64_t out, uint64_t rest) {
        const double w = hop_weight(g, a, b, c);
        if (w == 0.0) return;
        const int odd = (1 + __popcll(rest & (bits_between(a, b) ^ bits_between(c, d)))) & 1;
        f((uint32_t)(out >> plo), odd ? -w : w);
    };
    if (type == kKeep) {               // part o: every kKeepParts-th pair
        int pair = kKeepParts - o;
        for (uint64_t ta = W; ta; ta &= ta - 1) {
            const int a = __ffsll((long long)ta) - 1;
            for (uint64_t tb = ta & (ta - 1); tb; tb &= tb - 1) {
                if (pair++ % kKeepParts) continue;
                const int b = __ffsll((long long)tb) - 1;
                const uint64_t rest = W ^ (1ull << a) ^ (1ull << b);
                for (uint32_t m = (uint32_t)hop_targets(P, a - plo, b - plo, g.pbits, false); m; m &= m - 1) {
                    const int c = __ffs((int)m) - 1 + plo, d = a + b - c;
                    emit(a, b, c, d, rest | (1ull << c) | (1ull << d), rest);
                }
            }
        }
    } else if (type == kEmpty) {       // removes {x, o}, creates {c, d} in the primary part
        for (uint64_t tx = W; tx; tx &= tx - 1) {
            const int x = __ffsll((long long)tx) - 1, s = x + o;
            const uint64_t rest = W ^ (1ull << x);
            for (int c = max(plo, s - phi + 1); 2 * c < s; ++c) {
                const int d = s - c;
                if (c == x || d == x || ((rest >> c) & 1) || ((rest >> d) & 1)) continue;
                emit(min(x, o), max(x, o), c, d, rest | (1ull << c) | (1ull << d), rest);
            }
        }
    } else {                           // kFill: removes {a, b} from the primary part, creates {x, o}
        for (uint64_t ta = W; ta; ta &= ta - 1) {
            const int a = __ffsll((long long)ta) - 1;
            for (uint64_t tb = ta & (ta - 1); tb; tb &= tb - 1) {
                const int b = __ffsll((long long)tb) - 1, x = a + b - o;
                if (x < plo || x >= phi || ((W >> x) & 1)) continue;
                const uint64_t rest = W ^ (1ull << a) ^ (1ull << b);
                emit(a, b, min(x, o), max(x, o), rest | (1ull << x), rest);
            }
        }
    }
}

// gamma on the secondary word S (local bits): whether it acts, the new word
// and the sign bit of the orbitals its operators pass in S.
__device__ __forceinline__ bool gamma_acts(const GenArgs& g, uint32_t S, int gm, uint32_t& out, int& odd)
{
    const int type = gm & 15, o = (gm >> 4) - g.slo;
    if ((((S >> o) & 1) != 0) != (type == kEmpty)) return false;
    out = S ^ (1u << o);
    // the string to the primary part: the orbitals above o when the primary
    // part is the high one, below o when it is the low one
    const uint32_t mask = g.slo < g.plo ? ~((2u << o) - 1u) : (1u << o) - 1u;
    odd = __popc(S & out & mask) & 1;
    return true;
}

// Words of one part: how many choices of p of the orbitals below b have the
// weight sum s, count[(b (N + 1) + p) span + s].
struct PartArgs {
    int bits, N, span;
    int w[24];
    const int *count, *cls, *start;   // cls: per popcount span + sum, -1 where the sector has none
};

// Every word of a class to its place: classes one after another, ascending
// within a class.  The rank in its class is the sum over its orbitals b of the
// words that agree above b and leave b empty.  base (when wanted): the
// segment's first row in the transposed order, cbase[c] + rank size[c].  (The
// host enumerating the words by popcount and uploading them took 1.6 ms of a
// first product's 4.0 at two levels N=8, 2S=18, with 4e5 words in either part.)
__global__ void k_split_words(PartArgs a, uint32_t* __restrict__ word, int* __restrict__ cls, int* __restrict__ base,
                              const int* __restrict__ cbase, const int* __restrict__ size)
{
    const uint32_t end = 1u << a.bits;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < end; v += gridDim.x * blockDim.x) {
        const int pop = __popc(v);
        if (pop > a.N) continue;
        int sum = 0;
        for (uint32_t m = v; m; m &= m - 1) sum += a.w[__ffs((int)m) - 1];
        const int c = a.cls[pop * a.span + sum];
        if (c < 0) continue;
        int rank = 0, p = pop;
        for (uint32_t m = v; m;) {
            const int b = 31 - __clz((int)m);
            rank += a.count[(b * (a.N + 1) + p) * a.span + sum];
            --p;
            sum -= a.w[b];
            m ^= 1u << b;
        }
        const int at = a.start[c] + rank;
        word[at] = v;
        cls[at] = c;
        if (base) base[at] = cbase[c] + rank * size[c];
    }
}

// table[word] = segment length of the primary word, for the scan of bases
__global__ void k_split_lengths(const uint32_t* __restrict__ pword, const int* __restrict__ pcls,
                                const int* __restrict__ csize, int np, int64_t* __restrict__ table)
{
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < np; p += gridDim.x * blockDim.x)
        table[pword[p]] = csize[pcls[p]];
}

// base of each primary word's segment (from the scan, or given), also by word
__global__ void k_split_bases(const uint32_t* __restrict__ pword, int np, const int64_t* __restrict__ scan,
                              int* __restrict__ pbase, int* __restrict__ by_word)
{
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < np; p += gridDim.x * blockDim.x) {
        if (scan) pbase[p] = (int)scan[pword[p]];
        by_word[pword[p]] = pbase[p];
    }
}

// rank[word] = position of the word in its class
__global__ void k_split_ranks(const uint32_t* __restrict__ word, const int* __restrict__ cls,
                              const int* __restrict__ cstart, int n, int* __restrict__ rank)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        rank[word[i]] = i - cstart[cls[i]];
}

// perm[native row] = transposed row; one warp per native primary word
__global__ void k_split_perm(const int* __restrict__ pbase, const int* __restrict__ pcls,
                             const int* __restrict__ pstart, const int* __restrict__ psize,
                             const int* __restrict__ ssize, const int* __restrict__ cbase, int np,
                             int* __restrict__ perm)
{
    const int lane = threadIdx.x & 31;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    for (int p = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; p < np; p += nw) {
        const int c = pcls[p], rk = p - pstart[c];
        for (int i = lane; i < ssize[c]; i += 32) perm[pbase[p] + i] = cbase[c] + i * psize[c] + rk;
    }
}

// alpha lists, one thread per (primary word, gamma): fill == nullptr counts
// into cnt, else writes the entries (segment base, weight's limb pair) at start
__global__ void __launch_bounds__(128) k_split_alpha(GenArgs g, const uint32_t* __restrict__ pword, int np,
                                                     const int* __restrict__ by_word, int64_t* __restrict__ cnt,
                                                     const int64_t* __restrict__ start, int ea, int4* __restrict__ fill)
{
    const int64_t total = (int64_t)np * g.gammas;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t P = pword[t / g.gammas];
        const int gm = g.gamma[t % g.gammas];
        int64_t k = fill ? start[t] : 0;
        for_alpha(g, P, gm, [&](uint32_t out, double w) {
            const int base = by_word[out];
            if (base < 0) return;
            if (fill) {
                const int64_t q = fix_pair(w, ea);
                fill[k] = make_int4(base, (int)(uint32_t)(q & 0xFFFFFFFF), (int)(q >> 32), 0);
            }
            ++k;
        });
        if (!fill) cnt[t] = k;
    }
}

// Distance of move list i = 0 .. 2 (sbits - 1) - 1: +1, -1, +2, -2, ...
__host__ __device__ __forceinline__ int move_distance(int i) { return (i & 1) ? -(i / 2 + 1) : i / 2 + 1; }

// Moves of one secondary particle by a distance d, one thread per (primary
// word, d), or, filling, per (primary word, d, orbital o): each way the primary
// word makes up for the move (x -> x - d) gets its segment base and two rows of
// weights over the orbital o that the secondary particle leaves (o -> o + d),
// sbits of each sign.
template <bool FILL>
__global__ void __launch_bounds__(128) k_split_moves(GenArgs g, const uint32_t* __restrict__ pword, int np,
                                                     const int* __restrict__ by_word, int64_t* __restrict__ cnt,
                                                     const int64_t* __restrict__ start, int ea, int* __restrict__ base,
                                                     int64_t* __restrict__ weight)
{
    const int nm = 2 * (g.sbits - 1);
    const int64_t total = (int64_t)np * nm * (FILL ? g.sbits : 1);
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t t = FILL ? i / g.sbits : i;
        const int o = FILL ? (int)(i % g.sbits) : 0;
        const uint32_t P = pword[t / nm];
        const int d = move_distance((int)(t % nm)), q = o + d;
        int64_t k = FILL ? start[t] : 0;
        for (uint32_t tx = P; tx; tx &= tx - 1) {
            const int x = __ffs((int)tx) - 1, z = x - d;
            if (z < 0 || z >= g.pbits || ((P >> z) & 1)) continue;
            const int b = by_word[P ^ (1u << x) ^ (1u << z)];
            if (b < 0) continue;
            if (FILL) {
                if (o == 0) base[k] = b;
                const int odd = (1 + __popc(P & ((1u << max(x, z)) - 1u) & ~((2u << min(x, z)) - 1u))) & 1;
                double w = 0.0;
                if (q >= 0 && q < g.sbits) {
                    const int so = g.slo + o, sq = g.slo + q, gx = g.plo + x, gz = g.plo + z;
                    w = hop_weight(g, min(so, gx), max(so, gx), min(sq, gz));
                }
                weight[2 * k * g.sbits + o] = fix_pair(odd ? -w : w, ea);
                weight[(2 * k + 1) * g.sbits + o] = fix_pair(odd ? w : -w, ea);
            }
            ++k;
        }
        if (!FILL) cnt[t] = k;
    }
}

// Secondary lists of the gammas that change one orbital, one warp per (class,
// gamma, segment): entries row | new rank << 8 | sign << 31, rows ascending.
__global__ void __launch_bounds__(256) k_split_lists(GenArgs g, const uint32_t* __restrict__ sword,
                                                     const int* __restrict__ sstart, const int* __restrict__ ssize,
                                                     const int* __restrict__ rank, int nc, int nseg,
                                                     int64_t* __restrict__ cnt, const int64_t* __restrict__ start,
                                                     uint32_t* __restrict__ fill)
{
    const int lane = threadIdx.x & 31;
    const int64_t total = (int64_t)nc * g.gammas * nseg;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t t = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; t < total; t += nw) {
        const int seg = (int)(t % nseg);
        const int gm = g.gamma[(t / nseg) % g.gammas];
        const int c = (int)(t / ((int64_t)nseg * g.gammas));
        int64_t k = fill ? start[t] : 0;
        const int64_t k0 = k;
        if ((gm & 15) != kKeep) {
            const int r1 = min(ssize[c], (seg + 1) * kSegRows);
            for (int rb = seg * kSegRows; rb < r1; rb += 32) {
                const int r = rb + lane;
                uint32_t out = 0;
                int odd = 0;
                const bool acts = r < r1 && gamma_acts(g, sword[sstart[c] + r], gm, out, odd);
                const unsigned m = __ballot_sync(0xffffffffu, acts);
                if (fill && acts)
                    fill[k + __popc(m & ((1u << lane) - 1u))] =
                        (uint32_t)(r - seg * kSegRows) | ((uint32_t)rank[out] << kRowBits) | ((uint32_t)odd << 31);
                k += __popc(m);
            }
        }
        if (!fill && lane == 0) cnt[t] = k - k0;
    }
}

// Secondary lists of the moves, one warp per (class, distance, segment).  The
// rows in which some orbital can move are ordered by how many can (most
// first) and cut into blocks of 32, a lane each; a block holds k entries a
// lane, k its largest count, lane after lane: new rank | weight << 13, the
// weight's index being the orbital left, + sbits for the negative sign.  The
// first entry of a lane also has its row << 19 and k << 27, or the null bit.
__global__ void __launch_bounds__(128) k_split_move_lists(GenArgs g, const uint32_t* __restrict__ sword,
                                                          const int* __restrict__ sstart, const int* __restrict__ ssize,
                                                          const int* __restrict__ rank, int nc, int nseg,
                                                          int64_t* __restrict__ cnt, const int64_t* __restrict__ start,
                                                          uint32_t* __restrict__ fill)
{
    __shared__ short order[4][kSegRows];
    const int nm = 2 * (g.sbits - 1);
    const int64_t total = (int64_t)nc * nm * nseg;
    const uint32_t all = (1u << g.sbits) - 1u;
    const int lane = threadIdx.x & 31;
    short* ord = order[threadIdx.x >> 5];
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t t = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; t < total; t += nw) {
        const int seg = (int)(t % nseg);
        const int d = move_distance((int)((t / nseg) % nm));
        const int c = (int)(t / ((int64_t)nseg * nm));
        const int r0 = seg * kSegRows, rows = max(0, min(ssize[c] - r0, kSegRows));
        const uint32_t* words = sword + sstart[c] + r0;
        // movable orbitals of S: occupied ones whose target is empty
        auto movable = [&](uint32_t S) {
            const uint32_t e = ~S & all;
            return S & (d > 0 ? e >> d : e << -d) & all;
        };
        int found = 0;
        for (int k = kMaxMovable; k >= 1; --k)
            for (int rb = 0; rb < rows; rb += 32) {
                const bool is = rb + lane < rows && __popc(movable(words[rb + lane])) == k;
                const unsigned m = __ballot_sync(0xffffffffu, is);
                if (is) ord[found + __popc(m & ((1u << lane) - 1u))] = (short)(rb + lane);
                found += __popc(m);
            }
        __syncwarp();
        int64_t pos = fill ? start[t] : 0;
        const int64_t pos0 = pos;
        const uint32_t zero = (uint32_t)(d > 0 ? g.sbits - 1 : 0) << kWeightShift;   // no move: weight 0
        for (int b = 0; b < found; b += 32) {
            const int k = __popc(movable(words[ord[b]]));
            if (fill) {
                const bool in = b + lane < found;
                const int r = in ? ord[b + lane] : 0;
                const uint32_t S = words[r];
                uint32_t m = in ? movable(S) : 0u;
                for (int j = 0; j < k; ++j) {
                    uint32_t ent = zero;
                    if (m) {
                        const int o = __ffs((int)m) - 1;
                        m &= m - 1;
                        const uint32_t n = S ^ (1u << o) ^ (1u << (o + d));
                        const int lo = min(o, o + d), hi = max(o, o + d);
                        const int odd = __popc(S & n & ((1u << hi) - 1u) & ~((2u << lo) - 1u)) & 1;
                        ent = (uint32_t)rank[n] | (uint32_t)(o + odd * g.sbits) << kWeightShift;
                    }
                    if (j == 0) ent |= in ? (uint32_t)r << kRowShift : kNullEntry;
                    if (j == 0) ent |= (uint32_t)k << kCountShift;
                    fill[pos + 32 * j + lane] = ent;
                }
            }
            pos += 32 * k;
        }
        __syncwarp();
        if (!fill && lane == 0) cnt[t] = pos - pos0;
    }
}

__global__ void k_split_narrow(const int64_t* __restrict__ in, int64_t n, int* __restrict__ out)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = (int)in[i];
}

// the stored diagonal of each row (0 when none), as limb pairs once E is known
__global__ void k_split_crs_diag(const int64_t* __restrict__ rowptr, const int32_t* __restrict__ col,
                                 const double* __restrict__ val, int64_t n, double* __restrict__ d)
{
    for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < n; r += (int64_t)gridDim.x * blockDim.x) {
        int64_t lo = rowptr[r], hi = rowptr[r + 1];   // columns ascend within a row
        while (lo < hi) {
            const int64_t mid = (lo + hi) >> 1;
            if (col[mid] < r) lo = mid + 1;
            else hi = mid;
        }
        d[r] = lo < rowptr[r + 1] && col[lo] == r ? val[lo] : 0.0;
    }
}

// x in fixed point (its exponent bound the maximum of part, as k_fix_conv)
// in the native order and in the transposed one.
__global__ void __launch_bounds__(256) k_split_conv(const double* __restrict__ v, int64_t n, int* __restrict__ part,
                                                    int nparts, const int* __restrict__ perm, int64_t* __restrict__ q,
                                                    int64_t* __restrict__ qt, bool mark)
{
    __shared__ int sE;
    if (threadIdx.x < 32) {
        int m = 1;
        for (int i = threadIdx.x; i < nparts; i += 32) m = max(m, part[i]);
        m = __reduce_max_sync(0xffffffffu, m);
        if (threadIdx.x == 0) {
            sE = m;
            if (blockIdx.x == 0) atomicMax(part + nparts, m);
        }
    }
    __syncthreads();
    const int E = sE;
    bool lost = false;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double x = v[i];
        const int64_t a = fix_pair(x, E);
        lost |= fix_lost(x, a);
        q[i] = a;
        qt[perm[i]] = a;
    }
    if (mark && lost) atomicMax(part + nparts, kFixLost);
}

using Sum = FixSum;

__device__ __forceinline__ Sum negated(Sum s) { return Sum{~s.hi, (1ull << 60) - s.lo}; }

__device__ __forceinline__ void add_to(Sum& a, Sum b)   // b.lo <= 2^60
{
    const unsigned long long t = a.lo + b.lo;
    a.hi += b.hi + (long long)(t >> 60);
    a.lo = t & kFixLow60;
}

// s[u] += sum over the n entries w of weight * x(entry, u).
template <int NU, class F>
__device__ __forceinline__ void keep_sum(const int4* w, int n, F&& x, Sum (&s)[NU])
{
    for (int i = 0; i < n;) {
        const int e = min(i + kFixFlush, n);
        long long p2[NU], p1[NU], p0[NU];
#pragma unroll
        for (int u = 0; u < NU; ++u) {
            p2[u] = s[u].hi;
            p1[u] = 0;
            p0[u] = (long long)s[u].lo;
        }
#pragma unroll 4
        for (; i < e; ++i) {
            const int4 v = w[i];
#pragma unroll
            for (int u = 0; u < NU; ++u) fix_mac(make_int2(v.y, v.z), x(v, u), p2[u], p1[u], p0[u]);
        }
#pragma unroll
        for (int u = 0; u < NU; ++u) s[u] = fix_carry(p2[u], p1[u], p0[u]);
    }
}

// Finishes native row `row` with its exact sum, or stores a transposed one.
template <bool NATIVE>
__device__ __forceinline__ void finish_row(const SplitArgs& g, int row, Sum v)
{
    if (NATIVE) {
        const ulonglong2 t = g.acct[g.perm[row]];
        add_to(v, Sum{(long long)t.y, t.x});
        const int2 d = __ldg(g.diag + row), x = __ldg(g.x + row);
        long long p2 = 0, p1 = 0, p0 = 0;
        fix_mac(d, x, p2, p1, p0);
        const __int128 s = ((__int128)v.hi << 60) + (__int128)v.lo + fix_combine(p2, p1, p0);
        const int ex = __ldg(g.xexp);
        g.y[row] = ex < 2047 ? round_i128(s, g.ea + ex - 2160) : __longlong_as_double(0x7FF8000000000000ll);
    } else {
        g.acct[row] = make_ulonglong2(v.lo, (unsigned long long)v.hi);
    }
}

// The hops that leave S alone, for NU rows a thread from row `first` on.
template <int NU>
__device__ __forceinline__ void keep_rows(const SplitArgs& g, int a0, int a1, int r0, int first, int rows, Sum* acc)
{
    int at[NU];
    Sum s[NU];
#pragma unroll
    for (int u = 0; u < NU; ++u) {
        at[u] = r0 + min(first + (int)threadIdx.x + u * kThreads, rows - 1);
        s[u] = Sum{0, 0};
    }
    keep_sum<NU>(g.alpha + a0, a1 - a0, [&](const int4& v, int u) { return __ldg(g.x + (v.x + at[u])); }, s);
#pragma unroll
    for (int u = 0; u < NU; ++u) {
        const int r = first + threadIdx.x + u * kThreads;
        if (r < rows) acc[r] = s[u];
    }
}

// One list of a gamma that changes one orbital: U blocks of 32 entries at a
// time, up to kFixFlush alpha entries (the same for all lanes) each.
template <int U>
__device__ __forceinline__ void change_block(const SplitArgs& g, int a0, int a1, int e, int e1, Sum* acc)
{
    uint32_t ent[U];
    int to[U];
    long long p2[U], p1[U], p0[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const bool in = e + 32 * u < e1;
        ent[u] = in ? __ldg(g.list + e + 32 * u) : 0u;
        to[u] = (int)((ent[u] >> kRowBits) & kRankMask);
        p2[u] = p1[u] = p0[u] = 0;
    }
#pragma unroll 2
    for (int a = a0; a < a1; ++a) {
        const int4 w = __ldg(g.alpha + a);
#pragma unroll
        for (int u = 0; u < U; ++u) fix_mac(make_int2(w.y, w.z), __ldg(g.x + (w.x + to[u])), p2[u], p1[u], p0[u]);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
        Sum s = fix_carry(p2[u], p1[u], p0[u]);
        if ((int)ent[u] < 0) s = negated(s);
        if (e + 32 * u < e1) add_to(acc[ent[u] & (kSegRows - 1)], s);
    }
}

__device__ __forceinline__ void change_list(const SplitArgs& g, int a0, int a1, int e0, int e1, Sum* acc)
{
    for (; a0 < a1; a0 += kFixFlush) {
        const int a = min(a1, a0 + kFixFlush);
        int eb = e0, e = e0 + (threadIdx.x & 31);
        for (; eb + 32 < e1; eb += 64, e += 64) change_block<2>(g, a0, a, e, e1, acc);
        if (eb < e1) change_block<1>(g, a0, a, e, e1, acc);
        __syncwarp();
    }
}

// One list of the moves by one distance, for CA ways of the primary word from
// a0: each lane sums its row's entries in registers, taking an entry's weight
// from the way's rows (2 sbits consecutive words), and adds to the row once.
template <int CA>
__device__ __forceinline__ void move_list(const SplitArgs& g, int a0, int e0, int e1, Sum* acc)
{
    constexpr int kSteps = kFixFlush / CA;
    int b[CA];
#pragma unroll
    for (int a = 0; a < CA; ++a) b[a] = __ldg(g.mbase + a0 + a);
    const int2* __restrict__ wr = g.mweight + (int64_t)a0 * 2 * g.sbits;
    const uint32_t* __restrict__ list = g.mlist + e0 + (threadIdx.x & 31);
    uint32_t next = __ldg(list);
    for (int n = (e1 - e0) >> 5; n > 0;) {
        const uint32_t head = next;
        long long p2 = 0, p1 = 0, p0 = 0;
        int left = (int)((head >> kCountShift) & 15);
        n -= left;
        for (int step = kSteps;;) {
            const uint32_t ent = next;
            list += 32;
            next = __ldg(list);           // the list array has a block to spare at its end
            const int to = (int)(ent & kRankMask), wi = (int)((ent >> kWeightShift) & 63);
            int2 x[CA], w[CA];
#pragma unroll
            for (int a = 0; a < CA; ++a) {
                x[a] = __ldg(g.x + (b[a] + to));
                w[a] = __ldg(wr + (wi + 2 * a * g.sbits));
            }
#pragma unroll
            for (int a = 0; a < CA; ++a) fix_mac(w[a], x[a], p2, p1, p0);
            if (--left == 0) break;
            if (--step == 0) {
                const Sum s = fix_carry(p2, p1, p0);
                p2 = s.hi;
                p1 = 0;
                p0 = (long long)s.lo;
                step = kSteps;
            }
        }
        const Sum s = fix_carry(p2, p1, p0);
        if (!(head & kNullEntry)) add_to(acc[(head >> kRowShift) & (kSegRows - 1)], s);
    }
    __syncwarp();
}

__device__ __forceinline__ void move_lists(const SplitArgs& g, int a0, int a1, int e0, int e1, Sum* acc)
{
    for (; a0 < a1; a0 += 4) {
        switch (min(4, a1 - a0)) {
        case 1: move_list<1>(g, a0, e0, e1, acc); break;
        case 2: move_list<2>(g, a0, e0, e1, acc); break;
        case 3: move_list<3>(g, a0, e0, e1, acc); break;
        default: move_list<4>(g, a0, e0, e1, acc); break;
        }
    }
}

// One block per (primary word, segment of at most kSegRows rows).  The hops
// that leave S alone are summed in registers, one to four rows a thread.  The
// lists of the other gammas are taken by the block's warps from a queue; each
// warp keeps its own exact sums of the segment's rows in shared memory, and
// 32 consecutive entries hold 32 different rows, so it adds without atomics.
//
// Instruction issue and shared-memory latency bound it, so the blocks are
// small (64 threads, 18 per SM) to keep many segments in flight.  GB300, both
// passes with the conversion of x, against the element-generating kernel: N=11,
// 2S=30 2.76 -> 0.73 ms, N=12, 2S=33 18.3 -> 4.13 ms; against the stored kernels
// see the dispatch in ed_spmv.cu.  Move lists by (orbital, orbital) instead of
// by distance took 1.53 ms at N=11.
template <bool NATIVE>
__global__ void __launch_bounds__(kThreads, 18) k_split_product(SplitArgs g)
{
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int queue, count;
    Sum* acc = reinterpret_cast<Sum*>(smem);                     // [warp][rows]
    int4* lists = reinterpret_cast<int4*>(acc + kWarps * g.rows);   // alpha and entry ranges of each list
    if (g.gated && __ldg(g.xexp) >= 2047) return;
    const int2 task = g.task[blockIdx.x];
    const int p = task.x, seg = task.y;
    const int c = g.pcls[p];
    const int rows = min(kSegRows, g.ssize[c] - seg * kSegRows);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int* __restrict__ as = g.astart + (int64_t)p * g.gammas;
    const int* __restrict__ ms = g.mstart + (int64_t)p * g.moves;
    if (threadIdx.x == 0) queue = count = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < g.moves + g.gammas - kKeepParts; i += kThreads) {
        // the moves first, the short distances before the long ones: the largest lists
        int4 v;
        if (i < g.moves) {
            const int* l = g.mlstart + ((int64_t)c * g.moves + i) * g.nseg + seg;
            v = make_int4(ms[i], ms[i + 1], l[0], ~l[1]);
        } else {
            const int gm = i - g.moves + kKeepParts;
            const int* l = g.lstart + ((int64_t)c * g.gammas + gm) * g.nseg + seg;
            v = make_int4(as[gm], as[gm + 1], l[0], l[1]);
        }
        if (v.x < v.y && v.z < (v.w < 0 ? ~v.w : v.w)) lists[atomicAdd(&count, 1)] = v;   // any order: the sums are exact
    }
    for (int r = threadIdx.x; r < rows; r += kThreads)
#pragma unroll
        for (int w = 1; w < kWarps; ++w) acc[w * g.rows + r] = Sum{0, 0};
    {
        const int a0 = as[0], a1 = as[kKeepParts], r0 = seg * kSegRows;
        int r = 0;
        for (; r + kThreads < rows; r += 2 * kThreads) keep_rows<2>(g, a0, a1, r0, r, rows, acc);
        if (r < rows) keep_rows<1>(g, a0, a1, r0, r, rows, acc);
    }
    __syncthreads();
    Sum* mine = acc + warp * g.rows;
    const int nl = count;
    for (;;) {
        int i = 0;
        if (lane == 0) i = atomicAdd(&queue, 1);
        i = __shfl_sync(0xffffffffu, i, 0);
        if (i >= nl) break;
        const int4 v = lists[i];
        if (v.w < 0) move_lists(g, v.x, v.y, v.z, ~v.w, mine);
        else change_list(g, v.x, v.y, v.z, v.w, mine);
    }
    __syncthreads();
    const int base = g.pbase[p] + seg * kSegRows;
    for (int r = threadIdx.x; r < rows; r += kThreads) {
        Sum s = acc[r];
#pragma unroll
        for (int w = 1; w < kWarps; ++w) add_to(s, acc[w * g.rows + r]);
        finish_row<NATIVE>(g, base + r, s);
    }
}

// The alpha entries [a0, a1), the same for the whole warp, 32 at a time
// through shared memory, the next 32 loaded meanwhile: no gather of x waits
// for its entry.
template <int NU, class F>
__device__ __forceinline__ void staged_sum(const int4* __restrict__ al, int a0, int a1, F&& x, Sum (&s)[NU], int4* stage)
{
    const int lane = threadIdx.x & 31;
    int4 next = make_int4(0, 0, 0, 0);
    if (a0 + lane < a1) next = __ldg(al + a0 + lane);
    for (; a0 < a1; a0 += 32) {
        stage[lane] = next;
        if (a0 + 32 + lane < a1) next = __ldg(al + a0 + 32 + lane);
        __syncwarp();
        keep_sum<NU>(stage, min(32, a1 - a0), x, s);
        __syncwarp();
    }
}

template <bool NATIVE, int NU>
__device__ __forceinline__ void keep_task(const SplitArgs& g, int p, int size, int r0, int width, bool on, int4* stage)
{
    int at[NU];
    Sum s[NU];
#pragma unroll
    for (int u = 0; u < NU; ++u) {
        at[u] = min(r0 + width * u, size - 1);
        s[u] = Sum{0, 0};
    }
    const int a0 = g.astart[(int64_t)p * kKeepParts], a1 = g.astart[(int64_t)(p + 1) * kKeepParts];
    auto x = [&](const int4& v, int u) { return __ldg(g.x + (v.x + at[u])); };
    if (width == 32) staged_sum<NU>(g.alpha, a0, a1, x, s, stage);
    else keep_sum<NU>(g.alpha + a0, a1 - a0, x, s);
    const int base = g.pbase[p];
#pragma unroll
    for (int u = 0; u < NU; ++u)
        if (on && r0 + width * u < size) finish_row<NATIVE>(g, base + r0 + width * u, s[u]);
}

// Hops that leave S alone only (two levels): a warp takes one primary word
// and 32 * kIdRows rows of its segment, or, where segments are short, up to
// 32 / width words with `width` lanes each.  The gathers of x from L2 bound it:
// GB300, N=8, 2S=18 254 us against 281 of the sliced ELL copy, N=8, 2S=21 760
// against 993; segments staged in shared memory were slower.
template <bool NATIVE>
__global__ void __launch_bounds__(kThreads, 20) k_split_keep(SplitArgs g, int ntasks)
{
    __shared__ int4 stages[kWarps][32];
    const int t = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5);
    if (t >= ntasks || (g.gated && __ldg(g.xexp) >= 2047)) return;
    const int2 task = g.task[t];
    const int lane = threadIdx.x & 31;
    const int width = task.y & 63, cnt = (task.y >> 6) & 63, seg = task.y >> 12;
    const int sub = lane / width;
    const int p = task.x + min(sub, cnt - 1);
    const int size = g.ssize[g.pcls[p]];
    const int r0 = seg * 32 * kIdRows + lane % width;
    int4* stage = stages[threadIdx.x >> 5];
    if (width == 32 && size - seg * 32 * kIdRows > 32) keep_task<NATIVE, kIdRows>(g, p, size, r0, width, sub < cnt, stage);
    else keep_task<NATIVE, 1>(g, p, size, r0, width, sub < cnt, stage);
}

// ------------------------------------------------------------------ the plan

// The words of one part that the sector's classes hold, by class, ascending
// within each (on the device), and the classes' places and sizes.
struct PartWords {
    int count = 0;
    uint32_t* word = nullptr;
    int *cls = nullptr, *base = nullptr;
    std::vector<int> start, size;
};

// count[(b (N + 1) + p) span + s]: choices of p of the first b orbitals with
// weight sum s, b = 0 .. bits
std::vector<int> part_counts(const std::vector<int>& w, int N, int span)
{
    const size_t layer = (size_t)(N + 1) * span;
    std::vector<int> t(layer * (w.size() + 1), 0);
    t[0] = 1;
    for (size_t b = 0; b < w.size(); ++b) {
        const int *from = t.data() + layer * b, wb = w[b];
        int* to = t.data() + layer * (b + 1);
        std::copy(from, from + layer, to);
        for (int p = 1; p <= N; ++p)
            for (int sum = wb; sum < span; ++sum) to[(size_t)p * span + sum] += from[(size_t)(p - 1) * span + sum - wb];
    }
    return t;
}

template <class T>
void upload(DevBuf<T>& d, const std::vector<T>& h, cudaStream_t st)
{
    d.alloc(std::max<size_t>(1, h.size()));
    if (!h.empty()) ED_CUDA(cudaMemcpyAsync(d.p, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice, st));
}

int exponent_of(double v)
{
    uint64_t b;
    std::memcpy(&b, &v, 8);
    const int e = (int)((b >> 52) & 0x7FF);
    return e ? e : 1;
}

int grid_of(int64_t work, int threads)
{
    return (int)std::max<int64_t>(1, std::min<int64_t>((work + threads - 1) / threads, (int64_t)sms() * 16));
}

int exp_parts() { return sms() * 2; }

// Device memory for the build's temporaries: few allocations, freed together.
struct Arena {
    std::vector<DevBuf<char>> blocks;
    size_t used = 0;
    template <class T>
    T* take(size_t count)
    {
        const size_t bytes = (count * sizeof(T) + 255) / 256 * 256;
        if (blocks.empty() || used + bytes > blocks.back().n) {
            blocks.emplace_back(std::max<size_t>(bytes, (size_t)32 << 20));
            used = 0;
        }
        used += bytes;
        return reinterpret_cast<T*>(blocks.back().p + used - bytes);
    }
    template <class T>
    T* put(const std::vector<T>& h, cudaStream_t st)
    {
        T* p = take<T>(std::max<size_t>(1, h.size()));
        if (!h.empty()) ED_CUDA(cudaMemcpyAsync(p, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice, st));
        return p;
    }
};

// One pass: primary words P (by class), secondary words S of the same classes.
// count() sizes the lists (each total's copy to the host waits for its scan),
// fill() allocates them and enqueues their kernels.
struct SideBuild {
    SplitSide& out;
    const PartWords &P, &S;
    GenArgs g;
    const std::vector<int>& gamma;
    bool moves;
    Arena& tmp;
    cudaStream_t st;
    int np = 0, nc = 0, G = 0;
    uint32_t *pword = nullptr, *sword = nullptr;
    int *by_word = nullptr, *sstart = nullptr, *rank = nullptr;
    struct Lists {                 // of one kind
        int64_t n = 0, total = 0;
        int64_t* start = nullptr;
    } alpha, move, list, mlist;

    template <class F>
    void counted(Lists& l, int64_t n, F&& count)
    {
        l.n = n;
        int64_t* cnt = tmp.take<int64_t>((size_t)n);
        l.start = tmp.take<int64_t>((size_t)n + 1);
        count(cnt);
        count_launch();
        exclusive_scan_i64(cnt, l.start, n, tmp.take<int64_t>((size_t)scan_workspace_i64(n)), st);
        ED_CUDA(cudaMemcpyAsync(&l.total, l.start + n, 8, cudaMemcpyDeviceToHost, st));
    }
    // the starts as 32-bit indices
    void starts(const Lists& l, DevBuf<int>& d)
    {
        d.alloc((size_t)l.n + 1);
        k_split_narrow<<<grid_of(l.n + 1, 256), 256, 0, st>>>(l.start, l.n + 1, d.p);
        count_launch();
    }

    // given_base: the segments' bases are P's (transposed pass), else the scan
    // over the primary words in ascending order (native)
    bool count(bool given_base)
    {
        np = P.count;
        nc = (int)P.start.size();
        out.gammas = g.gammas = G = (int)gamma.size();
        int longest = 0;
        for (int c = 0; c < nc; ++c) longest = std::max(longest, S.size[c]);
        const bool lists = G > kKeepParts;
        if (lists && longest > (int)kRankMask) return false;
        out.nseg = (longest + kSegRows - 1) / kSegRows;
        out.rows = (std::min(longest, kSegRows) + 31) / 32 * 32;
        pword = P.word;
        g.gamma = tmp.put(gamma, st);
        out.pcls.alloc(np);
        ED_CUDA(cudaMemcpyAsync(out.pcls.p, P.cls, (size_t)np * 4, cudaMemcpyDeviceToDevice, st));
        upload(out.ssize, S.size, st);
        const int64_t nw = 1ll << g.pbits;
        by_word = tmp.take<int>((size_t)nw);
        ED_CUDA(cudaMemsetAsync(by_word, 0xFF, (size_t)nw * 4, st));
        int64_t* scan = nullptr;
        if (given_base) {
            out.pbase.alloc(np);
            ED_CUDA(cudaMemcpyAsync(out.pbase.p, P.base, (size_t)np * 4, cudaMemcpyDeviceToDevice, st));
        } else {
            int64_t* len = tmp.take<int64_t>((size_t)nw);
            scan = tmp.take<int64_t>((size_t)nw + 1);
            out.pbase.alloc(np);
            ED_CUDA(cudaMemsetAsync(len, 0, (size_t)nw * 8, st));
            k_split_lengths<<<grid_of(np, 256), 256, 0, st>>>(pword, out.pcls.p, out.ssize.p, np, len);
            count_launch();
            exclusive_scan_i64(len, scan, nw, tmp.take<int64_t>((size_t)scan_workspace_i64(nw)), st);
        }
        k_split_bases<<<grid_of(np, 256), 256, 0, st>>>(pword, np, scan, out.pbase.p, by_word);
        count_launch();
        const int64_t na = (int64_t)np * G;
        counted(alpha, na, [&](int64_t* cnt) {
            k_split_alpha<<<grid_of(na, 128), 128, 0, st>>>(g, pword, np, by_word, cnt, nullptr, 0, nullptr);
        });
        if (lists) {
            sword = S.word;
            sstart = tmp.put(S.start, st);
            rank = tmp.take<int>((size_t)1 << g.sbits);
            k_split_ranks<<<grid_of(S.count, 256), 256, 0, st>>>(sword, S.cls, sstart, S.count, rank);
            count_launch();
            counted(list, (int64_t)nc * G * out.nseg, [&](int64_t* cnt) {
                k_split_lists<<<sms() * 8, 256, 0, st>>>(g, sword, sstart, out.ssize.p, rank, nc, out.nseg, cnt, nullptr, nullptr);
            });
        }
        if (moves) {
            out.moves = 2 * (g.sbits - 1);
            out.sbits = g.sbits;
            const int64_t nt = (int64_t)np * out.moves;
            counted(move, nt, [&](int64_t* cnt) {
                k_split_moves<false><<<grid_of(nt, 128), 128, 0, st>>>(g, pword, np, by_word, cnt, nullptr, 0, nullptr, nullptr);
            });
            counted(mlist, (int64_t)nc * out.moves * out.nseg, [&](int64_t* cnt) {
                k_split_move_lists<<<sms() * 16, 128, 0, st>>>(g, sword, sstart, out.ssize.p, rank, nc, out.nseg, cnt, nullptr, nullptr);
            });
        }
        ED_CUDA(cudaGetLastError());
        return true;
    }

    size_t bytes() const
    {
        return (size_t)alpha.total * 16 + (size_t)move.total * (4 + 16 * (size_t)g.sbits) + (size_t)(list.total + mlist.total) * 4 +
               (size_t)(alpha.n + move.n + list.n + mlist.n) * 4;
    }
    bool fits() const
    {
        return std::max(std::max(alpha.total, move.total), std::max(list.total, mlist.total)) < (1ll << 31);
    }

    void fill(int ea)
    {
        const int64_t na = alpha.n;
        out.alpha.alloc((size_t)alpha.total + 1);
        k_split_alpha<<<grid_of(na, 128), 128, 0, st>>>(g, pword, np, by_word, nullptr, alpha.start, ea, out.alpha.p);
        count_launch();
        starts(alpha, out.astart);
        std::vector<int2> task;
        std::vector<int> order(nc);
        for (int c = 0; c < nc; ++c) order[c] = c;
        std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return S.size[a] > S.size[b]; });   // longest first
        if (G == kKeepParts) {
            for (int c : order) {
                const int m = S.size[c], words = P.size[c];
                int width = 32;                       // lanes a word: the fewest that hold its segment
                while (width > 2 && m <= width / 2) width /= 2;
                const int per = 32 / width, rows = width == 32 ? 32 * kIdRows : width;
                for (int i = 0; i < words; i += per)
                    for (int seg = 0; seg * rows < m; ++seg)
                        task.push_back(make_int2(P.start[c] + i, width | std::min(per, words - i) << 6 | seg << 12));
            }
        } else {
            out.list.alloc((size_t)list.total + 1);
            k_split_lists<<<sms() * 8, 256, 0, st>>>(g, sword, sstart, out.ssize.p, rank, nc, out.nseg, nullptr, list.start, out.list.p);
            count_launch();
            starts(list, out.lstart);
            for (int c : order)
                for (int i = 0; i < P.size[c]; ++i)
                    for (int seg = 0; seg * kSegRows < S.size[c]; ++seg) task.push_back(make_int2(P.start[c] + i, seg));
        }
        if (moves) {
            out.mbase.alloc((size_t)move.total + 1);
            out.mweight.alloc((size_t)move.total * 2 * g.sbits + 1);
            k_split_moves<true><<<grid_of(move.n * g.sbits, 128), 128, 0, st>>>(g, pword, np, by_word, nullptr, move.start, ea,
                                                                               out.mbase.p, out.mweight.p);
            count_launch();
            starts(move, out.mstart);
            out.mlist.alloc((size_t)mlist.total + 32);    // the product reads one block past a list
            ED_CUDA(cudaMemsetAsync(out.mlist.p + mlist.total, 0, 32 * 4, st));
            k_split_move_lists<<<sms() * 16, 128, 0, st>>>(g, sword, sstart, out.ssize.p, rank, nc, out.nseg, nullptr, mlist.start,
                                                          out.mlist.p);
            count_launch();
            starts(mlist, out.mlstart);
        }
        ED_CUDA(cudaGetLastError());
        out.ntasks = (int)task.size();
        upload(out.task, task, st);     // pageable: read before the call returns
    }
};

SplitArgs args_of(const SplitPlan& p, const SplitSide& s, const int64_t* x, const SplitPlan::Scratch& sc, double* y, int parts,
                  bool gated)
{
    SplitArgs g;
    g.task = s.task.p;
    g.pbase = s.pbase.p;
    g.pcls = s.pcls.p;
    g.ssize = s.ssize.p;
    g.astart = s.astart.p;
    g.alpha = s.alpha.p;
    g.lstart = s.lstart.p;
    g.list = s.list.p;
    g.mstart = s.mstart.p;
    g.mbase = s.mbase.p;
    g.mweight = reinterpret_cast<const int2*>(s.mweight.p);
    g.mlstart = s.mlstart.p;
    g.mlist = s.mlist.p;
    g.moves = s.moves;
    g.sbits = s.sbits;
    g.gammas = s.gammas;
    g.nseg = s.nseg;
    g.rows = s.rows;
    g.x = reinterpret_cast<const int2*>(x);
    g.xexp = sc.part.p + parts;
    g.acct = sc.acct.p;
    g.perm = p.perm.p;
    g.diag = reinterpret_cast<const int2*>(p.diag.p);
    g.y = y;
    g.ea = p.ea;
    g.gated = gated;
    return g;
}

template <bool NATIVE>
void launch_pass(const SplitSide& s, const SplitArgs& g, cudaStream_t st)
{
    if (s.ntasks == 0) return;
    if (s.gammas == kKeepParts)
        launch(k_split_keep<NATIVE>, (s.ntasks + kWarps - 1) / kWarps, kThreads, 0, st, g, s.ntasks);
    else
        launch(k_split_product<NATIVE>, s.ntasks, kThreads, (size_t)kWarps * sizeof(Sum) * s.rows + sizeof(int4) * (s.moves + s.gammas - kKeepParts), st, g);
}

}  // namespace

static std::unique_ptr<SplitPlan> plan_of(const SplitSource& s, const double* diag, int64_t n, int max_row, cudaStream_t st)
{
    // the low part S-side bits first: one level splits its orbitals in two
    // (the low part one longer for odd counts), two levels by level
    std::vector<int> wl, wh;
    if (s.levels == 1) {
        const int L = (s.norb0 + 1) / 2;
        for (int k = 0; k < s.norb0; ++k) (k < L ? wl : wh).push_back(k);
    } else {
        for (int j = 0; j < s.norb1; ++j) wl.push_back(j);
        for (int i = 0; i < s.norb0; ++i) wh.push_back(i + 1);
    }
    const int B0 = (int)wl.size(), B1 = (int)wh.size();
    if (B0 < 2 || B1 < 2 || B0 > kMaxSideBits || B1 > kMaxSideBits || n < 1 || n >= (1ll << 31)) return nullptr;
    if (max_row <= 0) max_row = s.N * (s.N - 1) / 2 * ((s.norb0 + s.norb1 + 1) / 2) + 1;
    if (max_row > kFixMaxRow) return nullptr;
    int ea = 1;
    double wmax = 0.0;
    for (const HopTables* h : {&s.hop0, &s.hop1})
        for (double w : h->w) {
            ea = std::max(ea, exponent_of(w));
            wmax = std::max(wmax, std::fabs(w));
        }
    // words of both parts by (popcount, weight sum), then the classes the sector joins
    const int lspan = 1 + std::accumulate(wl.begin(), wl.end(), 0), hspan = 1 + std::accumulate(wh.begin(), wh.end(), 0);
    const std::vector<int> ltab = part_counts(wl, s.N, lspan), htab = part_counts(wh, s.N, hspan);
    const int *lcount = ltab.data() + (size_t)B0 * (s.N + 1) * lspan, *hcount = htab.data() + (size_t)B1 * (s.N + 1) * hspan;
    std::vector<int> lclass((size_t)(s.N + 1) * lspan, -1), hclass((size_t)(s.N + 1) * hspan, -1);
    PartWords L, H;
    int64_t rows = 0;
    for (int k = 0; k < (int)lclass.size(); ++k) {
        const int pop = k / lspan, sum = k % lspan;
        const int64_t sh = s.sector_sum - sum;
        if (!lcount[k] || sh < 0 || sh >= hspan) continue;
        const int kh = (s.N - pop) * hspan + (int)sh;
        if (!hcount[kh]) continue;
        lclass[k] = hclass[kh] = (int)L.start.size();
        L.start.push_back(L.count);
        H.start.push_back(H.count);
        L.size.push_back(lcount[k]);
        H.size.push_back(hcount[kh]);
        L.count += lcount[k];
        H.count += hcount[kh];
        rows += (int64_t)lcount[k] * hcount[kh];
    }
    if (rows != n) return nullptr;
    const int nc = (int)L.start.size();
    std::vector<int> cbase(nc);
    int64_t run = 0;
    for (int c = 0; c < nc; ++c) {
        cbase[c] = (int)run;
        run += (int64_t)L.size[c] * H.size[c];
    }

    auto p = std::make_unique<SplitPlan>();
    p->n = n;
    Arena tmp;
    GenArgs gn{}, gt{};
    std::vector<int> gamman, gammat;
    for (int i = 0; i < kKeepParts; ++i) {
        gamman.push_back(kKeep | i << 4);
        gammat.push_back(kKeep | i << 4);
    }
    const double *w0 = tmp.put(s.hop0.w, st), *w1 = tmp.put(s.hop1.w, st);
    const int *off0 = tmp.put(s.hop0.hop_off, st), *off1 = tmp.put(s.hop1.hop_off, st);
    if (s.levels == 1) {
        gn = GenArgs{B0, B1, 0, B0, 0, nullptr, s.norb0, w0, off0};
        gt = GenArgs{0, B0, B0, B1, 0, nullptr, s.norb0, w0, off0};
        for (int o = 0; o < B0 + B1; ++o)
            for (int type : {kEmpty, kFill}) (o < B0 ? gamman : gammat).push_back(type | o << 4);
    } else {
        gn = GenArgs{0, B1, 0, B0, 0, nullptr, s.norb0, w0, off0};
        gt = GenArgs{0, B0, 0, B1, 0, nullptr, s.norb1, w1, off1};
    }
    auto words = [&](PartWords& part, const std::vector<int>& w, int span, const std::vector<int>& tab, const std::vector<int>& cls,
                     bool base) {
        PartArgs a{(int)w.size(), s.N, span, {}, tmp.put(tab, st), tmp.put(cls, st), tmp.put(part.start, st)};
        std::copy(w.begin(), w.end(), a.w);
        part.word = tmp.take<uint32_t>(part.count);
        part.cls = tmp.take<int>(part.count);
        if (base) part.base = tmp.take<int>(part.count);
        launch(k_split_words, grid_of(1ll << a.bits, 256), 256, 0, st, a, part.word, part.cls, part.base,
               base ? tmp.put(cbase, st) : nullptr, base ? tmp.put(H.size, st) : nullptr);
    };
    words(L, wl, lspan, ltab, lclass, true);
    words(H, wh, hspan, htab, hclass, false);
    SideBuild bn{p->native, H, L, gn, gamman, s.levels == 1, tmp, st};
    SideBuild bt{p->trans, L, H, gt, gammat, false, tmp, st};
    if (!bn.count(false) || !bt.count(true)) return nullptr;
    // the diagonal's exponent joins the weights'
    const int parts = exp_parts();
    int* part = tmp.take<int>((size_t)parts + 1);
    launch(k_fix_exp, parts, 256, 0, st, diag, n, part, 1);
    std::vector<int> h(parts);
    ED_CUDA(cudaMemcpyAsync(h.data(), part, (size_t)parts * 4, cudaMemcpyDeviceToHost, st));
    ED_CUDA(cudaStreamSynchronize(st));
    for (int e : h) ea = std::max(ea, e);
    if (ea >= 2047) return nullptr;
    // a row's high limb products fit 63 bits: |w| < ah 2^30 in units of the
    // fixed point, |xh| <= 2^28 (always so where the diagonal, a sum over all
    // pairs, is well above the single weights)
    if ((double)max_row * (std::ldexp(wmax, 1050 - ea) + 1.0) >= std::ldexp(1.0, 34)) return nullptr;
    p->ea = ea;
    // no weight may be lost either (nor, below, an entry of the diagonal)
    for (const HopTables* h : {&s.hop0, &s.hop1})
        for (double w : h->w)
            if (w != 0.0 && std::ldexp(std::fabs(w), 1080 - ea) < 0.5) return nullptr;
    const size_t free_b = device_memory_free();
    if (!bn.fits() || !bt.fits() || (size_t)n * 56 + bn.bytes() + bt.bytes() > free_b / 2) return nullptr;
    p->diag.alloc((size_t)n);
    int bound[2] = {ea, 0};
    ED_CUDA(cudaMemcpyAsync(part, bound, sizeof(bound), cudaMemcpyHostToDevice, st));
    launch(k_fix_conv, sms() * 4, 256, 0, st, diag, n, part, 1, p->diag.p, true);
    ED_CUDA(cudaMemcpyAsync(bound, part, sizeof(bound), cudaMemcpyDeviceToHost, st));
    bn.fill(ea);
    bt.fill(ea);
    p->perm.alloc((size_t)n);
    k_split_perm<<<sms() * 8, 256, 0, st>>>(p->native.pbase.p, p->native.pcls.p, tmp.put(H.start, st), tmp.put(H.size, st),
                                            p->native.ssize.p, tmp.put(cbase, st), H.count, p->perm.p);
    count_launch();
    ED_CUDA(cudaGetLastError());
    ED_CUDA(cudaStreamSynchronize(st));   // the temporaries and the host vectors go
    return bound[1] == kFixLost ? nullptr : std::move(p);
}

std::unique_ptr<SplitPlan> split_build(const SplitSource& s, const double* diag, int64_t n, int max_row, cudaStream_t st)
{
    std::unique_ptr<SplitPlan> p;
    const bool made = if_memory([&] {
        p = plan_of(s, diag, n, max_row, st);
        return p != nullptr;
    });
    return made ? std::move(p) : nullptr;
}

std::unique_ptr<SplitPlan> split_build_crs(const ed_crs& a, cudaStream_t st)
{
    if (!a.source || a.n < 1) return nullptr;
    std::unique_ptr<SplitPlan> p;
    const bool made = if_memory([&] {
        DevBuf<double> d((size_t)a.n);
        k_split_crs_diag<<<grid_of(a.n, 256), 256, 0, st>>>(a.rowptr.p, a.col.p, a.val.p, a.n, d.p);
        count_launch();
        ED_CUDA(cudaGetLastError());
        p = plan_of(*a.source, d.p, a.n, a.upper ? 0 : a.max_row, st);
        return p != nullptr;
    });
    return made ? std::move(p) : nullptr;
}

static SplitPlan::StreamKey stream_key(cudaStream_t st)
{
    int dev = 0;
    ED_CUDA(cudaGetDevice(&dev));
    return {dev, st, st == cudaStreamPerThread ? std::this_thread::get_id() : std::thread::id()};
}

bool split_ready(SplitPlan& p, cudaStream_t st)
{
    const SplitPlan::StreamKey key = stream_key(st);
    std::lock_guard<std::mutex> lk(p.mu);
    if (p.scratch.count(key)) return true;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    ED_CUDA(cudaStreamIsCapturing(st, &cs));
    if (cs != cudaStreamCaptureStatusNone) return false;
    if ((size_t)p.n * 32 > device_memory_free() / 2) return false;
    return if_memory([&] {
        auto sc = std::make_unique<SplitPlan::Scratch>();
        sc->x.alloc((size_t)p.n);
        sc->xt.alloc((size_t)p.n);
        sc->acct.alloc((size_t)p.n);
        sc->part.alloc((size_t)exp_parts() + 1);
        p.scratch.emplace(key, std::move(sc));
        return true;
    });
}

const int* split_product(SplitPlan& p, const double* x, double* y, bool mark, cudaStream_t st)
{
    SplitPlan::Scratch* sc;
    {
        std::lock_guard<std::mutex> lk(p.mu);
        sc = p.scratch.at(stream_key(st)).get();
    }
    const int P = exp_parts();
    launch(k_fix_exp, P, 256, 0, st, x, p.n, sc->part.p, 1);
    launch(k_split_conv, sms() * 4, 256, 0, st, x, p.n, sc->part.p, P, p.perm.p, sc->x.p, sc->xt.p, mark);
    launch_pass<false>(p.trans, args_of(p, p.trans, sc->xt.p, *sc, y, P, mark), st);
    launch_pass<true>(p.native, args_of(p, p.native, sc->x.p, *sc, y, P, mark), st);
    ED_CUDA(cudaGetLastError());
    return sc->part.p + P;
}

void split_release(SplitPlan& p, cudaStream_t st)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return;
    std::lock_guard<std::mutex> lk(p.mu);
    p.scratch.erase({dev, st, std::thread::id()});   // a solver's own stream
}

}  // namespace edgb
