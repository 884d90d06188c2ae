// kernels.cuh -- device data layout and launch wrappers shared by the
// kernels (gen.cu, sieve.cu) and the C ABI implementation (api.cu).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "host.hpp"
#include "pfcsieve.h"

namespace pfc {

constexpr int kSmallPrimes = 29;          // 3..113, the sieve bound of getsegprimes.cl
constexpr int kPatEntries = 1591;         // sum of the 29 primes: one 64-bit mask per residue

// Candidate list of one size class, structure of arrays in HBM.
//   p      : candidate primes
//   s0, s1 : residues (s0: factorial / primorial / compositorial-only;
//            s1: compositorial of the combined search)
//   nnext  : steps walked so far, summed over the candidate's chains; the
//            check kernel compares it with the steps the search needs
template <class W>
struct ClassBuf {
    W *p;
    W *s0;
    W *s1;
    uint32_t *nnext;
    uint32_t cap;
    const uint32_t *count;   // device counter written by the generator
};

struct HitBuf {
    pfc_factor *buf;
    unsigned long long *count;   // total hits (may exceed cap)
    uint64_t cap;
    uint32_t *tag;               // batches: job slot of each hit (else null)
    uint32_t tagval;
};

// Setup program for one quantity: a product of table words with squarings in
// between (Horner form of prod q^e over the bits of e), followed by one
// correction by a power of R.  groups[3k..3k+2] = {word_begin, word_end,
// squarings_before}; `final_sq` squarings follow the last group.
template <class W>
struct Prog {
    const W *words;
    const uint32_t *groups;
    uint32_t ngroups;
    uint32_t final_sq;
    uint64_t corr;           // apply *R^(corr+1) at the end (drift fix)
};

template <class W>
struct SetupArgs {
    unsigned mode;
    Prog<W> a;       // F: e-program; C: (e-1)-program; P: primorial words; FC: (e-1)-program
    Prog<W> b;       // FC only: primorial words continuing from a (factorial = comp * primorial)
    uint32_t nnext0; // nmin for n walks, 0 for the primorial prime index
};

// One walk launch over step indices [lo, hi).  The multiplier of step k is k
// itself (mult == nullptr: the factorial's n) or mult[k - base] (the
// compositorial's table of n at composite n and 1 at prime n, or the
// primorial's list of primes).  With mult2 set the launch also walks the
// candidate's second residue over mult2 (the compositorial chain of the
// combined search, fused with its factorial chain).  Hits record the
// multiplier.
struct WalkArgs {
    uint32_t lo, hi;
    const uint32_t *mult;
    const uint32_t *mult2;
    uint32_t base;      // index of mult[0] and mult2[0]
    int32_t type;       // factor type of chain-0 hits (PFC_TYPE_*)
    int32_t type2;      // factor type of the fused second chain
    int chain;          // single-chain walks: 0 -> residue s0, 1 -> residue s1
};

// A walk over n split into sub-ranges: candidate i's sub-range k covers steps
// [start[k], start[k+1]) and begins from the residue at start[k], in s0/s1 +
// k * pitch.  One launch walks every (candidate, sub-range) pair (grid y = k);
// the last sub-range leaves the candidate's final residue in its state, which
// no sub-range reads (nothing orders the CTAs of a launch: sub-range 0 begins
// from a copy), and every sub-range adds its steps to nnext.
// Candidate sets too small to fill the GPU get more chains this way.
constexpr int kMaxSplit = 8;
template <class W>
struct SplitArgs {
    uint32_t start[kMaxSplit + 1];
    uint32_t n;        // sub-ranges (1 = no split)
    uint32_t pitch;    // stride of the start-residue arrays (the class capacity)
    W *s0, *s1;        // start residues of the sub-ranges
};

// the setup programs of a split walk's boundaries 1..n-1 (n <= kMaxSplit),
// evaluated in one launch (grid y = sub-range; 0 copies the state)
template <class SW>
struct SplitSetup {
    unsigned mode;
    uint32_t n;
    Prog<SW> a[kMaxSplit - 1];
    Prog<SW> b[kMaxSplit - 1];
};

// size classes: class 32 holds p < 2^31, class 64 the rest
constexpr uint64_t kClassSplit = 1ull << 31;
// class-64 segments whose candidates are all below kLazyEnd (3p < 2^64) set
// up with 896-bit table words and walk with lazy one-word steps
constexpr uint64_t kLazyEnd = 0x5555555555555556ull;
constexpr uint64_t kLazyWalkEnd = kLazyEnd;

struct CheckArgs {
    unsigned mode;
    uint32_t nlast;             // nmax - 1
    uint32_t nend;              // steps every candidate must have walked
    unsigned long long *termsum;
    uint32_t *flags;            // bit 0: n-counter validation failure
};

struct GenArgs {
    uint64_t base;     // first odd number of the segment
    uint64_t nodd;     // odd numbers in the segment
    uint32_t *p32;
    uint64_t *p64;
    uint32_t cap32, cap64;
    uint32_t *count;   // [0] class-32 count, [1] class-64 count (may exceed caps)
    const uint64_t *pat;      // kPatEntries sieve masks (device)
    uint32_t bmod[32];        // base mod each of the 29 small primes
    uint32_t share;           // threads per 64-bit word of odd numbers (1, 2 or 4; set by launch_gen)
};

// Launch wrappers (enqueue on `st`); return the number of kernels launched.
int launch_gen(const GenArgs &a, int sms, cudaStream_t st);
int launch_setup32(const ClassBuf<uint32_t> &c, const SetupArgs<WideWord> &a, cudaStream_t st);
int launch_setup64(const ClassBuf<uint64_t> &c, const SetupArgs<uint64_t> &a, cudaStream_t st);
// class 64 below 2^64/3 with 896-bit table words
int launch_setup64w(const ClassBuf<uint64_t> &c, const SetupArgs<WideWord> &a, cudaStream_t st);
// The setup of any class with the table-word fold on the tensor cores
// (setup_tc.cu): each program in its paired form (host.hpp TcProg: 1792-bit
// words, each the product of one or two 896-bit words, merged first groups,
// every group in lanes of its own through all tiles, kTcOne in lanes without a
// word), packed into fp16 digit tiles of tc_tile_words() lanes (tc_tile_bytes()
// each; src[128 t + l] is the word of lane l of tile t), then the setup over
// those tiles with the paired programs' groups (of lanes), final squarings and
// corrections in `a`; a wait that gives up sets bit 1 of *err (the segment then
// fails with PFC_ERR_CUDA)
struct TcTiles {
    const void *tiles;   // device, ntiles * tc_tile_bytes(), 16-byte aligned
    uint32_t ntiles;
};
size_t tc_tile_bytes();
uint32_t tc_tile_words();
int launch_tc_pack(const WideWord *words, const uint32_t *src, uint32_t nw, uint32_t ntiles, void *out,
                   cudaStream_t st);
// class 64: candidate blocks of 32, [block0, block0 + nblocks), nblocks 0 to the
// end (lazy: every candidate is below 2^64/3)
uint32_t tc_setup_blocks(uint32_t cands);
int launch_setup64_tc(const ClassBuf<uint64_t> &c, const SetupArgs<WideWord> &a, const TcTiles &ta,
                      const TcTiles &tb, bool lazy, uint32_t *err, cudaStream_t st, uint32_t block0 = 0,
                      uint32_t nblocks = 0);
// class 32, blocks of 64, on the same tiles (the classes' 896-bit programs are the same)
uint32_t tc_setup_blocks32(uint32_t cands);
// Smallest programs (896-bit words, both programs of the search) set up on the
// tensor cores: below them the kernel's fixed cost per CTA (the position
// residues' planes, TMEM, the first tile's copy and products, the final tree,
// about 18,000 cycles) outweighs what it saves per word.  Measured on GB300
// (factorial searches, 4e6-wide p ranges), integer pipe against tensor cores:
// class 32 at 214 words 0.203 / 0.226 ms, at 304 0.280 / 0.246, at 2,265 1.95 /
// 0.45; class 64 at 145 words 0.28 / 0.39 ms, at 214 0.396 / 0.394, at 304
// 0.54 / 0.44, at 2,265 3.77 / 0.79.
constexpr uint64_t kTcMinWords32 = 240;
constexpr uint64_t kTcMinWords64 = 216;
// From 2^64/3 on, where the integer pipe takes 64-bit words: at 78 words 0.213 /
// 0.255 ms, at 145 0.394 / 0.257, at 2,265 6.52 / 0.58; over a 3e7-wide range
// at 78 words 1.14 / 1.83, at 145 2.16 / 1.84.  Programs for n up to
// kTcMinStartTop do not reach that size (the combined search's do first, from
// nmin 33,504 on).
constexpr uint64_t kTcMinWordsTop = 112;
constexpr uint32_t kTcMinStartTop = 33000;
int launch_setup32_tc(const ClassBuf<uint32_t> &c, const SetupArgs<WideWord> &a, const TcTiles &ta,
                      const TcTiles &tb, uint32_t *err, cudaStream_t st, uint32_t block0 = 0, uint32_t nblocks = 0);
// start residues of a split walk: sub-range k's into s0/s1 + k * c.cap
int launch_split_setup32(const ClassBuf<uint32_t> &c, const SplitSetup<WideWord> &ss, uint32_t *s0, uint32_t *s1,
                         cudaStream_t st);
int launch_split_setup64(const ClassBuf<uint64_t> &c, const SplitSetup<uint64_t> &ss, uint64_t *s0, uint64_t *s1,
                         cudaStream_t st);
int launch_split_setup64w(const ClassBuf<uint64_t> &c, const SplitSetup<WideWord> &ss, uint64_t *s0, uint64_t *s1,
                          cudaStream_t st);
// walk launches: `variant` indexes the walk variants of the size class
// (0 = default; see walk_variant_shape)
// (sp: a split walk, null for the plain one; split walks use each class's
// default shape)
int launch_walk32(const ClassBuf<uint32_t> &c, const WalkArgs &a, const HitBuf &h, cudaStream_t st, int variant,
                  const SplitArgs<uint32_t> *sp = nullptr);
// lazy: every candidate is below 2^64/3 (the walk then takes lazy one-word steps)
int launch_walk64(const ClassBuf<uint64_t> &c, const WalkArgs &a, const HitBuf &h, cudaStream_t st, bool lazy,
                  int variant, const SplitArgs<uint64_t> *sp = nullptr);
// The walk with its tests on the tensor cores (walk_tc.cu): one or two streams
// (the two chains of the combined search) of steps [lo, hi) over every
// candidate, from the tables of words that launch_walk_words laid out for them
// (`top`: the largest multiplier of the tables, which sets the words' shape).
struct WalkTcArgs {
    const unsigned char *words[2];
    const uint32_t *digits[2];   // largest sum of |digit| of a table's words
    const uint32_t *mult[2];   // multipliers of step k at mult[k - base], or k itself (null)
    int32_t type[2];           // factor type of a stream's hits
    uint32_t second[2];        // 1: the stream walks the residue s1
    uint32_t nstreams;
    uint32_t lo, hi, base;           // steps of the first stream,
    uint32_t lo1, hi1, base1;        // and of the second
    uint32_t credit[2];              // steps that a stream adds to the candidates' count (a split walk: its own)
    uint32_t nb, shift11, shift22;   // set by walk_tc_args: steps per block, 2^11, 2^22
};
// (both streams over [lo, hi), each step credited)
void walk_tc_args(WalkTcArgs &a, uint32_t top, uint32_t lo, uint32_t hi, uint32_t base);
// the composite n of [lo, hi) in order (prime flags as launch_cmult)
int launch_composites(uint32_t *out, const uint32_t *primebits, uint32_t nmin, uint32_t lo, uint32_t hi, cudaStream_t st);
uint32_t walk_tc_align(uint32_t top);   // sub-ranges of a split walk start at multiples of this from lo
size_t walk_tc_words_bytes(uint32_t top, uint32_t steps);
// (the table of steps [lo, hi) into `out`, for the walk's stream `stream`)
int launch_walk_words(const uint32_t *mult, uint32_t base, uint32_t lo, uint32_t hi, uint32_t top, unsigned char *out,
                      WalkTcArgs &a, int stream, cudaStream_t st);
// The same over windows of many searches, one launch for the tables and one
// for the walks of a size class and word shape (walk_tc_shape).  Windows are
// ordered by first_cta; a table has walk_tc_words_bytes, its `digits` start at 0.
struct WalkWordsWin {
    const uint32_t *mult;
    unsigned char *out;
    uint32_t *digits;
    uint32_t base, lo, hi, nb, nsuper, first_cta;
};
template <class W>
struct WalkTcWin {
    ClassBuf<W> c;
    WalkTcArgs a;
    uint32_t *err;
    uint32_t first_cta, tag;
};
int walk_tc_shape(uint32_t top);
uint32_t walk_tc_ctas(uint32_t cands);
uint32_t walk_words_ctas(uint32_t top, uint32_t steps);
void walk_words_win(WalkWordsWin &win, const uint32_t *mult, uint32_t base, uint32_t lo, uint32_t hi, uint32_t top,
                    unsigned char *table, uint32_t *digits);
int launch_walk_words_many(const WalkWordsWin *wins, uint32_t n, uint32_t ctas, int shape, cudaStream_t st);
int launch_walk_tc32_many(const WalkTcWin<uint32_t> *wins, uint32_t n, uint32_t ctas, int shape, const HitBuf &h,
                          cudaStream_t st);
int launch_walk_tc64_many(const WalkTcWin<uint64_t> *wins, uint32_t n, uint32_t ctas, int shape, bool lazy,
                          const HitBuf &h, cudaStream_t st);
// a wait that gives up sets bit 2 of *err
int launch_walk_tc32(const ClassBuf<uint32_t> &c, const WalkTcArgs &a, uint32_t top, const HitBuf &h,
                     const SplitArgs<uint32_t> *sp, uint32_t *err, cudaStream_t st);
int launch_walk_tc64(const ClassBuf<uint64_t> &c, const WalkTcArgs &a, uint32_t top, const HitBuf &h,
                     const SplitArgs<uint64_t> *sp, uint32_t *err, cudaStream_t st, bool lazy);
// Which walk, and when it is split.  Times of one walk launch in microseconds,
// fitted to GB300 (factorial searches at p = 1e9, 2^61 and 3 2^62, 2,000 to
// 300,000 candidates x 200 to 10,000 n; the fits are within 15%):
//   tensor cores: CTAs of 128 candidates, one per SM, so whole waves of them,
//     each with a fixed part (the candidates' planes, filling and draining the
//     pipeline, about 1,500 steps' worth) and a part per step; a launch more
//     for the word table;
//   per-step kernels: a rate per candidate-step, and below about one chain per
//     thread the latency of a step.
// Measured, ms, tensor cores / per-step:
//   class 32, 19,000 candidates:  500 n .029 / .026, 1,000 .031 / .038, 10,000 .088 / .169
//            300,000 candidates: 2,000 n .354 / .286, 3,000 .454 / .423, 10,000 1.16 / 1.37
//   class 64, 19,000 candidates:  500 n .034 / .030, 1,000 .037 / .046, 10,000 .116 / .282
//            300,000 candidates: 1,000 n .338 / .296, 2,000 .490 / .563, 10,000 1.58 / 2.70
//   from 2^64/3, 19,000 candidates: 200 n .031 / .025, 500 .033 / .042, 10,000 .125 / .481
//            300,000 candidates: 500 n .287 / .287, 1,000 .363 / .547, 10,000 1.75 / 5.28
struct WalkTimes {
    double fixed, step;            // per wave of the tensor-core walk: fixed part, per step
    double lat, rate0, rate;       // per-step kernels, per step: latency; base and part per candidate
};
constexpr double kTcLaunch = 12.0, kWalkLaunch = 13.0;
constexpr WalkTimes kTimes32 = {9.7, 6.3e-3, 25.3e-3, 12e-3, 4.1e-7}, kTimes64 = {13.2, 8.8e-3, 31e-3, 20e-3, 8.2e-7},
                    kTimesTop = {12.3, 9.6e-3, 58e-3, 8e-3, 1.73e-6};   // (class 64 from 2^64/3)

// Smallest primes the tensor-core walk takes.  Towards small p a growing part
// of the blocks holds a hit or a multiple of p and is replayed; at 2^16 that
// does not show yet (2,700 candidates x 20,000 n: 0.15 ms, per-step 0.62), and
// few searches start below.
constexpr uint64_t kTcMinP = 1u << 16;

// size class 0: p < 2^31, 1: lazy class 64 (p < 2^64/3), 2: other class 64
int walk_variant_count(int cls, bool fused);
int walk_variant_shape(int cls, bool fused, int variant, int *nc, int *b);
// compositorial multipliers of n in [lo, hi): n when composite, 1 when prime
// (bit k of primebits <-> n = nmin + k); `out` is padded with 1 to a multiple of
// 16; `ramp` (may be null) receives n itself, the factorial's multipliers
int launch_cmult(uint32_t *out, uint32_t *ramp, const uint32_t *primebits, uint32_t nmin, uint32_t lo, uint32_t hi,
                 cudaStream_t st);
int launch_check32(const ClassBuf<uint32_t> &c, const CheckArgs &a, cudaStream_t st);
int launch_check64(const ClassBuf<uint64_t> &c, const CheckArgs &a, cudaStream_t st);

// host helper: the sieve pattern table (kPatEntries masks) and prime list
void build_pattern_table(uint64_t *pat, uint32_t *primes29);

// Slow products over k in [lo, hi) modulo the self-check test primes
// (verify.cu): products of the primes and of the composites (plain residues)
// and the prime count.
constexpr int kVerifyPrimes = 3;
constexpr uint64_t kVerifyPrime[kVerifyPrimes] = {2147483647ull, 4611686018427387847ull, 18446744073709551557ull};
struct SlowProducts {
    uint64_t P[kVerifyPrimes], C[kVerifyPrimes], count;
};
}  // namespace pfc
struct pfc_ctx;
namespace pfc {
int slow_products(pfc_ctx *c, uint64_t lo, uint64_t hi, SlowProducts &out);


}  // namespace pfc
