// walk_tc.cu -- the walk over n with its per-step test on the tensor cores
// (tcgen05), for the three size classes (class 32; class 64 below 2^64/3 and
// from there).
//
// walk.cuh multiplies every candidate's residue by every n.  Here the n range
// is cut into blocks of nb multipliers (16, or 12 for n that do not fit the
// word below), and a block's tests use integers that all candidates share:
// with r the residue at the END of the block and N_j the product of the
// block's last j multipliers, the residue j steps before the end is r / N_j,
// so it is +-1 exactly when N_j = +-r (mod p).  Whether that holds is decided
// from a fraction: with X_j = frac(N_j R / p) and A = frac(r R / p) (R the
// Montgomery factor, so that A comes from the residue as it is kept),
// N_j = +-r (mod p) means X_j = +-A (mod 1).  X_j is a contraction over the
// digits of N_j,
//     X_j = sum_b d_b(N_j) f_b (mod 1),   f_b = frac(2^(6b) R / p),
// words x digits by digits x candidates, with balanced 6-bit digits d_b and
// f_b to 24 bits as two 12-bit planes.  Every partial sum is an integer:
// |d| <= 32, |plane| <= 2048 and at most 63 digits give |S| < 2^22, which
// rides on a bias of 1.5 * 2^23 (digit 0 of every word is 4096, of every plane
// 3072), so an fp32 accumulator holds 0x4B400000 + S exactly and the CUDA
// cores read S from its bits.  Per (p, n) they are left with one multiply-add
// (S_hi 2^12 + S_lo), half a byte permute that packs the middle 16 bits of
// two neighbours, and two packed add-and-min (for +A and -A): 2.5
// instructions, against the 10 (class 32) and 21 (class 64) of a step.
//
// The 24-bit f_b are off by at most 0.504 units each and A by 0.045 units of
// 2^-16, so the test takes a window of +-half around +-A, half =
// floor(0.504 / 256 max sum |digit| + 0.045) + 1: every hit passes, and with
// half 2 or 3 one pair in 6,500 or 4,700 passes by chance.  The maximum is
// taken over the table's own words.  A lane that saw a
// pass queues (residue at the block's START, block, candidate) in a ring in
// shared memory, and warps of their own replay the queue with exact
// arithmetic, one entry per lane, so false passes cost time only.  The offsets
// that the biases and the window leave in hi 2^12 + lo ride on the words' last
// digit, which is 1, and the planes' last element.
//
// The residue itself advances once per block, by the whole block product W:
// u = W R' (mod p) comes from a second contraction, the unsigned 6-bit digits
// of W with the residues w_b = 2^(6b) R'' mod p in 11-bit planes (three for
// class 32, six for class 64; digit sums below 63 * 63 * 2047 < 2^23 on a bias
// of 2^23), one Montgomery round reduces the assembled sum to u, and one
// product moves r.  No drift: the power of R is in the planes.
//
// Layout.  A CTA owns 128 candidates (MMA M = 128, one TMEM lane each); the
// words are the N operand, K-major in shared memory, streamed tile by tile
// (four blocks, 64 words; a supertile is four tiles and the 16 words W of
// their blocks) by bulk copies from a table that walk_words_kernel lays out
// once per launch and that stays in L2.  The candidates' planes are the A
// operand: the test's two planes in TMEM (with A in TMEM an MMA of 64 words
// takes 32 cycles, with A in shared memory 48), the residue's in TMEM (class
// 32) or shared memory (class 64, where TMEM is full).  Roles: 16 warps test
// (four groups of a thread per candidate, two groups per buffer, two blocks of
// each tile), in class 32 four warps reduce the block products and four carry
// the residues, in class 64 three groups of four do both in turn, two warps copy
// words and issue the tests' MMAs, one the residues', four (one) replay.  Chain,
// reduction and tests run in units of tiles, handed over through shared memory,
// so that a role waits once per unit and not once per tile.
//
// A launch walks one stream (a chain of each candidate) or the combined
// search's two one after the other, each over its own list of multipliers; one
// stream has kernels of its own, without the second's bookkeeping (2 to 3%).
//
// What bounds it: the CUDA cores' issue slots and their ALU pipe (byte permutes
// and packed minima).  Cycles per 32 candidates and step on an SM's quarter,
// per-step kernels to this one: class 32 (4.8e5 candidates) 17.7 to 12.5 (words
// of 47 digits), 19.6 to 13.4 (63); class 64 (1.2e5) 35.9 to 17.0 (63), 38.3 to
// 17.9 (47), from 2^64/3 (3.0e5) 69.5 to 20.4.  At that rate 66 to 68% of the
// issue slots are used, the ALU 56 to 59% of the time, the fma-heavy pipe 43%
// (class 32) and 58% (class 64), the tensor cores 32 and 40%.
// (The testers' loop runs over whole units, unrolled, and a suspect's residue
// is read only when there is one: a tile at a time took 13.4 cycles in class
// 32, 11% more instructions.)  A CTA's fixed part, about 1,500 steps long, is planes
// (7 to 14 thousand cycles), the first products' way through the roles (5
// thousand), and the last replays.
//
// Every wait is bounded; when one gives up the CTA raises bit 2 of *err,
// waits (bounded) for its copies, frees its TMEM and stores nothing.
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "tcgen05.cuh"
#include "walk.cuh"

namespace pfc {
namespace {

constexpr int kCands = 128;                    // candidates per CTA: MMA M, TMEM lanes
constexpr int kBlocksTile = 4;                 // blocks per tile of test words
constexpr int kRowsTile = 16 * kBlocksTile;    // words per tile: MMA N of the tests
constexpr int kBlocksSuper = 16;               // blocks per supertile of the word table
constexpr int kTilesSuper = kBlocksSuper / kBlocksTile;
constexpr int kBufs = 2;                       // buffers of test sums; tile t takes buffer t % 2
constexpr int kFStages = 2 * kBufs;            // tiles of test words in shared memory, two per buffer
constexpr int kTesterGroups = 4;               // warp groups, two per buffer, each two blocks of its tiles
constexpr int kTestBlocks = 2;
constexpr int kBatches = 16;                   // ring of suspects, in batches of 32
constexpr uint32_t kBiasE = 0x4B000000u;       // fp32 bits of 2^23, under the residues' sums
constexpr uint32_t kTableHead = 128;           // a search's word table begins with its largest sum of |digit| (u32)

// digits per word (KD) and MMA depth (K = KD + 1, the bias digit first)
template <int K>
struct WordShape {
    static constexpr int KD = K - 1;
    static constexpr uint32_t kRowGroup = (K / 8) * 128;               // bytes between 8-row core groups
    static constexpr uint32_t kFTile = (kRowsTile / 8) * kRowGroup;    // 8 KB (K = 64), 6 KB (K = 48)
    static constexpr uint32_t kWTile = (kBlocksSuper / 8) * kRowGroup;
    static constexpr uint32_t kSuper = kWTile + (kBlocksSuper / kBlocksTile) * kFTile;
    static constexpr int kLimbs = (6 * KD + 31) / 32;                  // 32-bit limbs of a word
};

// the value b0 + 2^11 b1 + 2^22 b2 of three sums on their biases.  sh holds
// 2^11 and 2^22 from the launch's arguments: known to the compiler they would
// be shifts and carries, four ALU instructions each, and the ALU is the
// busier pipe here.
__device__ __forceinline__ uint64_t gather(uint32_t b0, uint32_t b1, uint32_t b2, uint2 sh) {
    constexpr uint64_t off = 0ull - (uint64_t)kBiasE * (1u + (1u << 11) + (1u << 22));
    return (uint64_t)b2 * sh.y + ((uint64_t)b1 * sh.x + off) + b0;
}

template <class T>
struct ChainClass;

// class 32: residues signed in (-p, p), R = 2^32
template <>
struct ChainClass<Cls32> {
    using W = uint32_t;
    using M = Mont32;
    using U = int32_t;                         // a block product, reduced
    using Q = uint32_t;                        // p^-1, as reduce and prod take it
    static constexpr int kPlanes = 3;
    static constexpr bool kInTmem = true;      // 3 planes of K / 2 columns
    static constexpr int kBlocksE = 16;        // blocks per MMA of the residues, in
    static constexpr int kBufsE = 2;           // two buffers of sums
    static constexpr int kReduceGroups = 1, kChainGroups = 1, kReplayWarps = 4;
    static constexpr int kUnit = 4, kUUnits = 2, kRUnits = 3;   // tiles the chain takes at a time; units kept
    static constexpr uint32_t kIdle = 0x7FFFFFFFu;
    static constexpr float kScale = 4194304.0f;   // 2^22: |r| < p
    static constexpr int kShift = 6;
    __device__ static __forceinline__ Q qv(const M &m) { return m.pinv; }
    // 2^bits w_0, w_0 = 2^64 (u = T 2^-32 = W 2^32, r u 2^-32 = r W), from the
    // next power of R
    __device__ static __forceinline__ W power(const M &m, uint32_t bits) {
        const uint32_t k = (bits + 64 + 31) / 32;   // R^k
        const W x = m.mont_R_pow(k - 1);            // (R^(e+1))
        return m.mul(x, 1u << (32 * (2 - (int)k) + bits + 32));
    }
    __device__ static __forceinline__ W div64(const M &m, W x) { return m.mul(x, 1u << 26); }
    // x 2^32 mod p
    __device__ static __forceinline__ W step32(const M &m, W x, W) { return m.mul(x, m.r2); }
    __device__ static __forceinline__ W c32(const M &m) { return m.r2; }
    // T < 2^12 p from the three sums: u = hi(T) - hi(m p) with m = lo(T) p^-1
    // read as signed, so |u| <= p/2 + 2^11
    __device__ static __forceinline__ int32_t reduce(const uint32_t (&b)[3], W p, uint32_t pinv, uint2 sh) {
        const uint64_t t = gather(b[0], b[1], b[2], sh);
        const int32_t m = (int32_t)((uint32_t)t * pinv);
        int64_t mp;
        asm("mul.wide.s32 %0, %1, %2;" : "=l"(mp) : "r"(m), "r"(p));
        return (int32_t)(t >> 32) - (int32_t)(mp >> 32);
    }
    // |r| < p, |u| <= p/2 + 2^11: |r u 2^-32| + p/2 < p
    __device__ static __forceinline__ W prod(W r, int32_t u, W p, uint32_t pinv) {
        return (W)redc31s((int32_t)r, (uint32_t)u, (int32_t)p, pinv);
    }
    __device__ static __forceinline__ uint32_t shift(W) { return 0; }
    __device__ static __forceinline__ float value(W r, uint32_t) { return (float)(int32_t)r; }
};

// class 64 below 2^64/3: residues in [0, 2p), R = 2^64
template <>
struct ChainClass<Cls64L> {
    using W = uint64_t;
    using M = Mont64;
    using U = uint64_t;
    using Q = uint32_t;
    static constexpr int kPlanes = 6;
    // 6 planes do not fit in TMEM; with them in shared memory an MMA takes 41
    // cycles for 16 or for 32 blocks (the planes' read), so 32, in one buffer
    static constexpr bool kInTmem = false;
    static constexpr int kBlocksE = 32;
    static constexpr int kBufsE = 1;
    static constexpr int kReduceGroups = 0, kChainGroups = 3, kReplayWarps = 1;
    static constexpr int kUnit = 2, kUUnits = 0, kRUnits = 6;
    static constexpr uint64_t kIdle = 0x1FFFFFFFFFFFFFFFull;
    static constexpr float kScale = 2097152.0f;   // 2^21: r < 2p
    static constexpr int kShift = 5;
    __device__ static __forceinline__ Q qv(const M &m) { return m.q32; }
    __device__ static __forceinline__ W two32(W p) { return p > (1ull << 32) ? (1ull << 32) : (1ull << 32) - p; }
    // 2^bits w_0, w_0 = 2^96 (u = T 2^-32 = W 2^64, r u 2^-64 = r W), from the
    // next power of R down by lazy rounds of 2^-32, in [0, 2p) as are the w_b
    __device__ static __forceinline__ W power(const M &m, uint32_t bits) {
        const uint32_t k = (bits + 96 + 63) / 64, down = 64 * k - (bits + 96);   // down < 64
        W x = m.mont_R_pow(k - 1);
        if (down >= 32) x = redc64l(x, 1u, m.p, m.q32);
        return down % 32 ? redc64l(x, 1u << (32 - down % 32), m.p, m.q32) : x;
    }
    __device__ static __forceinline__ W div64(const M &m, W x) { return redc64l(x, 1u << 26, m.p, m.q32); }
    __device__ static __forceinline__ W c32(const M &m) { return m.to_mont(two32(m.p)); }
    __device__ static __forceinline__ W step32(const M &m, W x, W c96) { return m.mul(x, c96); }
    // T = L + 2^32 H < 2^13 p: u = (T + m p) / 2^32 with m = -T p^-1, u < p + 2^44
    __device__ static __forceinline__ W reduce(const uint32_t (&b)[6], W p, uint32_t q, uint2 sh) {
        const uint64_t L = gather(b[0], b[1], b[2], sh), H = gather(b[3], b[4], b[5], sh);
        const uint32_t m = (uint32_t)L * q;
        // (lo(L) + m p0) / 2^32 exactly: its low word is 0
        const uint64_t c = (uint64_t)m * (uint32_t)p + (uint32_t)L;
        return (uint64_t)m * (uint32_t)(p >> 32) + (H + (L >> 32)) + (c >> 32);
    }
    // two lazy rounds; u < p + 2^44 and p < 2^64/3 leave (3p + 2p u_hi +
    // 2^32 p) / 2^32 < p (1 + 2/3) + small < 2p: no correction
    __device__ static __forceinline__ W prod(W r, W u, W p, uint32_t q) {
        return cios_round(redc64l(r, (uint32_t)u, p, q), r, (uint32_t)(u >> 32), p, q);
    }
    // the top 31 or 32 bits of r (r < 2p): r >> shift, p >> shift below 2^31
    __device__ static __forceinline__ uint32_t shift(W p) { return p >> 31 ? 33 - __clzll((long long)p) : 0; }
    __device__ static __forceinline__ float value(W r, uint32_t sh) {
        return (float)__funnelshift_rc((uint32_t)r, (uint32_t)(r >> 32), sh);
    }
};

// class 64 from 2^64/3: residues in [0, p), R = 2^64
template <>
struct ChainClass<Cls64> {
    using W = uint64_t;
    using M = Mont64;
    using U = uint64_t;
    using Q = uint64_t;
    using L = ChainClass<Cls64L>;
    static constexpr int kPlanes = 6;
    static constexpr bool kInTmem = false;
    static constexpr int kBlocksE = L::kBlocksE, kBufsE = L::kBufsE;
    static constexpr int kReduceGroups = L::kReduceGroups, kChainGroups = L::kChainGroups, kReplayWarps = L::kReplayWarps;
    static constexpr int kUnit = L::kUnit, kUUnits = L::kUUnits, kRUnits = L::kRUnits;
    static constexpr uint64_t kIdle = L::kIdle;
    static constexpr float kScale = 4194304.0f;   // 2^22: r < p
    static constexpr int kShift = 6;
    __device__ static __forceinline__ Q qv(const M &m) { return m.pinv; }
    __device__ static __forceinline__ W power(const M &m, uint32_t bits) {
        const uint32_t k = (bits + 96 + 63) / 64;
        return m.mul(m.mont_R_pow(k - 1), 1ull << (bits + 160 - 64 * k));
    }
    __device__ static __forceinline__ W div64(const M &m, W x) { return m.mul(x, 1ull << 58); }
    __device__ static __forceinline__ W c32(const M &m) { return m.to_mont(1ull << 32); }
    __device__ static __forceinline__ W step32(const M &m, W x, W c96) { return m.mul(x, c96); }
    // T = L + 2^32 H: u = (T + m p) / 2^32 with m = -T p^-1 is a carry of m p
    // (at most p) and T's high part (below 2^46), less p where that passes p
    __device__ static __forceinline__ W reduce(const uint32_t (&b)[6], W p, Q q, uint2 sh) {
        const uint64_t L = gather(b[0], b[1], b[2], sh), H = gather(b[3], b[4], b[5], sh);
        const uint32_t m = 0u - (uint32_t)L * (uint32_t)q;
        const uint64_t c = (uint64_t)m * (uint32_t)p + (uint32_t)L, t = H + (L >> 32);
        const uint64_t u = (uint64_t)m * (uint32_t)(p >> 32) + (c >> 32) + t;
        return u < t || u >= p ? u - p : u;
    }
    __device__ static __forceinline__ W prod(W r, W u, W p, Q q) { return redc64(r, u, p, q); }
    __device__ static __forceinline__ uint32_t shift(W) { return 32; }
    __device__ static __forceinline__ float value(W r, uint32_t) { return (float)(uint32_t)(r >> 32); }
};

// Warp roles, in groups of four warps (a thread per candidate): testers
// (tiles in turn), reducers (class 32), the chain; then single warps: the
// tests' MMAs (one per buffer), the residues' MMAs, replays.
template <class T>
struct Role {
    using C = ChainClass<T>;
    static constexpr int kReduce = 4 * kTesterGroups;
    static constexpr int kChain = kReduce + 4 * C::kReduceGroups;
    static constexpr int kTestMma = kChain + 4 * C::kChainGroups;
    static constexpr int kChainMma = kTestMma + kBufs;
    static constexpr int kReplay = kChainMma + 1;
    static constexpr int kThreads = 32 * (kReplay + C::kReplayWarps);
    static_assert(kThreads <= 1024, "walk_tc roles");
};

template <class T, int K>
struct Lay {
    using W = typename ChainClass<T>::W;
    using S = WordShape<K>;
    static constexpr int kPlanes = ChainClass<T>::kPlanes;
    // TMEM columns
    static constexpr uint32_t kColF = 0;                          // test planes, 2 x K/2
    static constexpr uint32_t kColE = K;                          // residue planes (class 32), 3 x K/2
    static constexpr uint32_t kColDE = kColE + (ChainClass<T>::kInTmem ? kPlanes * K / 2 : 0);
    static constexpr int kBlocksE = ChainClass<T>::kBlocksE, kBufsE = ChainClass<T>::kBufsE;
    static constexpr uint32_t kDE = kPlanes * kBlocksE;           // columns of one residue buffer
    static constexpr uint32_t kColDF = 256;                       // 2 buffers of 2 planes x 64 words
    static constexpr uint32_t kDF = 2 * kRowsTile;
    static_assert(kColDE + kBufsE * kDE <= kColDF && kColDF + kBufs * kDF == 512, "walk_tc TMEM columns");
    // shared memory
    static constexpr uint32_t kPlaneBytes = (kCands / 8) * S::kRowGroup;
    static constexpr uint32_t kOffE = 0;
    static constexpr uint32_t kOffF = kOffE + (ChainClass<T>::kInTmem ? 0 : kPlanes * kPlaneBytes);
    static constexpr uint32_t kWStage = kBlocksE / kBlocksSuper * S::kWTile;
    static constexpr int kWStages = 2 * kBufsE;
    static constexpr uint32_t kOffW = kOffF + kFStages * S::kFTile;
    using C = ChainClass<T>;
    static constexpr uint32_t kRTile = (kBlocksTile + 1) * kCands;         // a tile's residues: block starts, the last one's end
    static constexpr uint32_t kOffR = kOffW + kWStages * kWStage;          // [unit][tile][..][cand] W
    static constexpr uint32_t kOffU = kOffR + C::kRUnits * C::kUnit * kRTile * sizeof(W);   // [unit][block][cand] W
    static constexpr uint32_t kOffQ = kOffU + C::kUUnits * C::kUnit * kBlocksTile * kCands * sizeof(W);  // suspects: W r, then
    static constexpr uint32_t kOffQk = kOffQ + kBatches * 32 * sizeof(W);                 // stream, block, cand
    static constexpr uint32_t kOffQs = kOffQk + kBatches * 32 * 4;                        // written: round + 1
    static constexpr uint32_t kOffP = kOffQs + kBatches * 32 * 4;                         // candidates' p, then q
    static constexpr uint32_t kOffPq = kOffP + kCands * sizeof(W);
    static constexpr uint32_t kOffBar = kOffPq + kCands * sizeof(typename C::Q);
    static constexpr uint32_t kBars = kFStages + kWStages + 2 * kBufs + 2 * C::kRUnits + 2 * kBufsE + 2 * C::kUUnits + kBufs + 1;
    static constexpr uint32_t kOffMisc = kOffBar + kBars * 8;   // failed, TMEM address, suspects, testers done, [batch] rounds replayed
    static constexpr uint32_t kSmem = kOffMisc + 16 + kBatches * 4 + 8;   // and the steps [lo, hi)
    static_assert(kOffF % 128 == 0 && kOffW % 128 == 0 && kOffR % 16 == 0 && kOffBar % 8 == 0, "walk_tc alignment");
    static_assert(kSmem <= 227 * 1024, "walk_tc shared memory");
};

// two integers 0..2047 in the halves of x as fp16: 1024 + (low 10 bits), less
// 1024 where bit 10 is clear (0x400 * 0x19 is the fp16 of 1024)
__device__ __forceinline__ uint32_t f16x2_u11(uint32_t x) {
    return sub_f16x2((x & 0x03FF03FFu) | 0x64006400u, (~x & 0x04000400u) * 0x19u);
}
// two integers -2048..2047 given as v + 2048: bit 11 clear takes off 2048 (0x800 * 0xD)
__device__ __forceinline__ uint32_t f16x2_s12(uint32_t x) {
    return sub_f16x2(f16x2_u11(x & 0x07FF07FFu), (~x & 0x08000800u) * 0xDu);
}

// Exact replay of up to 32 suspects, one per lane: the block's steps from the
// residue at its start, as replay_chain.  (Not from its end: where p divides a
// multiplier of the block the residue at the end is 0 and says nothing of the
// steps before, which hit at n = p - 1 and p - 2.  Such a block is a suspect:
// 0 = +-0.)
template <class T>
__device__ __forceinline__ void replay_suspect(bool act, typename T::W p, typename ChainClass<T>::Q q, typename T::W r, uint32_t k,
                                               uint32_t len, const uint32_t *mult, int32_t type, const HitBuf &h) {
    using W = typename T::W;
    typename T::M m;
    m.p = p;
    W t = 1;
    if constexpr (std::is_same<T, Cls64L>::value) {
        m.q32 = q;
        t = ChainClass<T>::two32(p);
    } else {
        m.pinv = q;
    }
    uint32_t mul[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) mul[j] = (act && (uint32_t)j < len) ? (mult ? __ldg(mult + j) : k + j) : 1u;
    W x = T::canon(m, r);
    unsigned plus = 0, minus = 0;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        if (j) t = T::next_target(m, t);
        x = T::step(m, x, mul[j]);
        if (mul[j] != 1u) {   // at a multiplier of 1 (padding, a prime n of n!/n#) nothing is tested
            if (x == t) plus |= 1u << j;
            else if (x == m.p - t) minus |= 1u << j;
        }
    }
    unsigned any = plus | minus;
    while (__any_sync(kFull, any != 0)) {   // one hit of each lane at a time
        const int j = any ? __ffs(any) - 1 : 0;
        uint32_t n = mul[0];
#pragma unroll
        for (int i = 1; i < 16; ++i)
            if (i == j) n = mul[i];
        append_hit(any != 0, p, (plus >> j) & 1u ? -(int32_t)n : (int32_t)n, type, h);
        any &= any - 1;
    }
}

}  // namespace

// The words of the blocks of steps [lo, hi), padded with multipliers of 1 to
// whole supertiles, in the shared-memory image of the MMA's B operand: per
// supertile the 16 block products W (unsigned 6-bit digits), then four tiles
// of 64 rows, row 16 b + j the product of the last j multipliers of block b
// (balanced digits: the 6-bit digits of N + sum 32 * 64^b, less 32).  One
// thread per word.
template <int K>
__device__ __forceinline__ void walk_words(const WalkWordsWin &win, uint32_t i) {
    using S = WordShape<K>;
    constexpr uint32_t kRows = 17 * kBlocksSuper;
    const uint32_t *mult = win.mult;
    const uint32_t base = win.base, lo = win.lo, hi = win.hi, nb = win.nb, nsuper = win.nsuper;
    unsigned char *out = win.out;
    const uint32_t st = min(i / kRows, nsuper - 1), r = i % kRows;   // (past the end: the last supertile's again)
    const bool whole = r < kBlocksSuper;
    const uint32_t row = r - kBlocksSuper;                      // among the 256 test words
    const uint32_t blk = whole ? r : row / 16;
    const uint32_t cnt = whole ? nb : min(row % 16, nb - 1);    // multipliers of the word
    const uint32_t k0 = lo + (st * kBlocksSuper + blk) * nb;
    uint32_t v[S::kLimbs + 1];
#pragma unroll
    for (int l = 0; l <= S::kLimbs; ++l) v[l] = l == 0 ? 1u : 0u;
    for (uint32_t j = 0; j < cnt; ++j) {
        const uint32_t k = k0 + nb - 1 - j;
        const uint32_t mul = k >= hi ? 1u : mult ? __ldg(mult + (k - base)) : k;
        uint32_t carry = 0;
#pragma unroll
        for (int l = 0; l < S::kLimbs; ++l) {
            const uint64_t t = (uint64_t)v[l] * mul + carry;
            v[l] = (uint32_t)t;
            carry = (uint32_t)(t >> 32);
        }
    }
    uint32_t digits = 0;   // sum of |digit|
    if (!whole) {   // balanced: add 32 to every digit
        uint32_t carry = 0;
#pragma unroll
        for (int l = 0; l < S::kLimbs; ++l) {
            uint32_t c = 0;
#pragma unroll
            for (int s = 0; s < 32; ++s)
                if ((32 * l + s) % 6 == 5 && (32 * l + s) / 6 < S::KD - 1) c |= 1u << s;
            const uint64_t t = (uint64_t)v[l] + c + carry;
            v[l] = (uint32_t)t;
            carry = (uint32_t)(t >> 32);
        }
    }
    const uint32_t off = whole ? 0u : 1056u - 1024u;
    unsigned char *dst = out + (size_t)st * S::kSuper +
                         (whole ? (r / 8) * S::kRowGroup + (r % 8) * 16
                                : S::kWTile + (row / kRowsTile) * S::kFTile + ((row % kRowsTile) / 8) * S::kRowGroup +
                                      (row % 8) * 16);
    const uint32_t less = off ? 0x64206420u : 0x64006400u;   // 1024 + 32, or 1024
#pragma unroll
    for (int k8 = 0; k8 < K / 8; ++k8) {
        uint32_t w[4];
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            uint32_t pair = 0;
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                const int e = 8 * k8 + 2 * h + s;   // element: the bias digit, then digit e - 1
                if (e > 0) {
                    const int bit = 6 * (e - 1), l = bit / 32, sh = bit % 32;
                    const uint32_t d = (sh ? __funnelshift_r(v[l], v[l + 1], sh) : v[l]) & 63u;
                    pair |= d << (16 * s);
                    if (e < K - 1) digits += abs((int)d - 32);
                }
            }
            w[h] = sub_f16x2(pair | 0x64006400u, less);
            if (k8 == 0 && h == 0) w[h] = (w[h] & 0xFFFF0000u) | 0x6C00u;   // 4096
            if (k8 == K / 8 - 1 && h == 3 && !whole) w[h] = (w[h] & 0xFFFFu) | 0x3C000000u;   // 1: the offset's digit
        }
        *reinterpret_cast<uint4 *>(dst + k8 * 128) = make_uint4(w[0], w[1], w[2], w[3]);
    }
    if (whole) digits = 0;
    digits = __reduce_max_sync(kFull, digits);
    if ((threadIdx.x & 31) == 0) atomicMax(win.digits, digits);
}

template <int K>
__global__ void __launch_bounds__(128) walk_words_kernel(WalkWordsWin win) {
    walk_words<K>(win, blockIdx.x * blockDim.x + threadIdx.x);
}

// the last of the windows whose first CTA is not past `cta`
template <class Win>
__device__ __forceinline__ uint32_t window_of(const Win *wins, uint32_t n, uint32_t cta) {
    uint32_t a = 0, b = n;
    while (b - a > 1) {
        const uint32_t mid = (a + b) >> 1;
        if (wins[mid].first_cta <= cta) a = mid;
        else b = mid;
    }
    return a;
}

template <int K>
__global__ void __launch_bounds__(128) walk_words_many_kernel(const WalkWordsWin *wins, uint32_t n) {
    const WalkWordsWin win = wins[window_of(wins, n, blockIdx.x)];
    walk_words<K>(win, (blockIdx.x - win.first_cta) * blockDim.x + threadIdx.x);
}

// one CTA: candidates 128 cta .. of c, sub-range `sub` of a split walk (sp, or
// null); NS 1 for walks of one stream, 2 for one or two
template <class T, int K, int NS>
__device__ __forceinline__ void walk_tc(const ClassBuf<typename T::W> &c, const WalkTcArgs &a, const HitBuf &h,
                                        const SplitArgs<typename T::W> *sp, uint32_t *err, uint32_t cta, uint32_t sub) {
    using C = ChainClass<T>;
    using L = Lay<T, K>;
    using S = WordShape<K>;
    using W = typename T::W;
    extern __shared__ __align__(1024) unsigned char sm[];
    const uint32_t tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
    const uint32_t nstreams = NS == 1 ? 1u : a.nstreams;
    const uint32_t cnt = min(*c.count, c.cap);
    const uint32_t c0 = cta * kCands;
    if (c0 >= cnt) return;   // whole CTA idle

    uint32_t lo = a.lo, hi = a.hi;   // steps of the first stream (of both in a split walk)
    const bool split = sp && sp->n > 1, last = !split || sub + 1 >= sp->n;
#pragma unroll
    for (int k = 0; k < kMaxSplit; ++k)
        if (split && (uint32_t)k == sub) {
            lo = sp->start[k];
            hi = sp->start[k + 1];
        }
    const uint32_t super0 = (lo - a.lo) / (kBlocksSuper * a.nb);   // sub-ranges start at supertiles
    constexpr uint32_t kPer = C::kBlocksE / kBlocksSuper;   // supertiles per buffer of residue sums
    const uint32_t per = kBlocksSuper * a.nb;
    const uint32_t supers = (hi - lo + per - 1) / per;   // supertiles of the first stream, of the second
    const uint32_t supers1 = nstreams < 2 ? 0u : split ? supers : (a.hi1 - a.lo1 + per - 1) / per;
    const uint32_t tiles = supers * kTilesSuper, ntiles = tiles + supers1 * kTilesSuper;   // of the first stream, of both
    const uint32_t nsupers_e = (supers + kPer - 1) / kPer, nge = nsupers_e + (supers1 + kPer - 1) / kPer;
    // the test's window around +-A in units of 2^-16: the f_b are off by up to
    // 0.504 units of 2^-24 each, A by 0.045 of 2^-16
    uint32_t digits = *a.digits[0];
    if (nstreams > 1) digits = max(digits, *a.digits[1]);
    const uint32_t half = (uint32_t)(digits * (0.504f / 256.0f) + 0.045f) + 1u;
    constexpr uint32_t kBlocksUnit = C::kUnit * kBlocksTile, kUnitsE = C::kBlocksE / kBlocksUnit;   // units per buffer of residue sums
    const uint32_t bar = smem_u32(sm + L::kOffBar);
    constexpr uint32_t kB0 = kFStages + L::kWStages, kB1 = kB0 + 2 * kBufs, kB2 = kB1 + 2 * C::kRUnits,
                       kB3 = kB2 + 2 * L::kBufsE, kB4 = kB3 + 2 * C::kUUnits;
    auto bar_f = [&](uint32_t i) { return bar + 8 * i; };                         // test words landed
    auto bar_w = [&](uint32_t i) { return bar + 8 * (kFStages + i); };            // block words landed
    auto bar_t = [&](uint32_t i) { return bar + 8 * (kB0 + i); };                 // a buffer's test sums ready
    auto bar_tf = [&](uint32_t i) { return bar + 8 * (kB0 + kBufs + i); };        // and read
    auto bar_r = [&](uint32_t i) { return bar + 8 * (kB1 + i); };                 // a unit's residues ready
    auto bar_rf = [&](uint32_t i) { return bar + 8 * (kB1 + C::kRUnits + i); };   // and read
    auto bar_e = [&](uint32_t i) { return bar + 8 * (kB2 + i); };                 // residue sums ready
    auto bar_ef = [&](uint32_t i) { return bar + 8 * (kB2 + L::kBufsE + i); };    // and read
    auto bar_u = [&](uint32_t i) { return bar + 8 * (kB3 + i); };                 // a unit's block products reduced
    auto bar_uf = [&](uint32_t i) { return bar + 8 * (kB3 + C::kUUnits + i); };   // and used
    auto bar_end = [&](uint32_t i) { return bar + 8 * (kB4 + i); };               // an MMA warp's last MMAs ended
    uint32_t *misc = reinterpret_cast<uint32_t *>(sm + L::kOffMisc);
    volatile uint32_t *failed = misc;
    const uint32_t fail = smem_u32(misc);
    uint32_t *taddr_slot = misc + 1, *suspects = misc + 2, *testers_done = misc + 3, *replayed = misc + 4;
    const volatile uint32_t *range = misc + 4 + kBatches;   // lo, hi: read where they are rarely needed
    W *cand_p = reinterpret_cast<W *>(sm + L::kOffP);
    auto *cand_q = reinterpret_cast<typename C::Q *>(sm + L::kOffPq);

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(taddr_slot))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (uint32_t i = 0; i < kFStages; ++i) mbar_init(bar_f(i), 1);
        for (uint32_t i = 0; i < L::kWStages; ++i) mbar_init(bar_w(i), 1);
        for (uint32_t i = 0; i < kBufs; ++i) {
            mbar_init(bar_t(i), 1);
            mbar_init(bar_tf(i), 4 * kTesterGroups / kBufs);
        }
        for (uint32_t i = 0; i < C::kRUnits; ++i) {
            mbar_init(bar_r(i), 4);
            mbar_init(bar_rf(i), 4 * kTesterGroups);
        }
        for (uint32_t i = 0; i < L::kBufsE; ++i) {
            mbar_init(bar_e(i), 1);
            mbar_init(bar_ef(i), 4 * (C::kReduceGroups ? C::kReduceGroups : C::kChainGroups));
        }
        for (int i = 0; i < C::kUUnits; ++i) {
            mbar_init(bar_u(i), 4);
            mbar_init(bar_uf(i), 4);
        }
        for (uint32_t i = 0; i <= kBufs; ++i) mbar_init(bar_end(i), 1);
        *failed = 0;
        *suspects = *testers_done = 0;
        for (uint32_t i = 0; i < kBatches; ++i) replayed[i] = 0;
        misc[4 + kBatches] = lo;
        misc[5 + kBatches] = hi;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (uint32_t i = tid; i < kBatches * 32; i += Role<T>::kThreads) reinterpret_cast<uint32_t *>(sm + L::kOffQs)[i] = 0;
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tbase = *taddr_slot;
    const uint32_t lanes = ((warp % 4) * 32u) << 16;          // this warp's TMEM lanes
    const uint32_t cl = (warp % 4) * 32 + lane, ci = c0 + cl;   // this thread's candidate
    const bool act = ci < cnt;

    // copies of the MMA warps: tile t of test words into a stage of its
    // buffer, supertile(s) g of block words; the first ones start here (none
    // after a wait that gave up: a copy may then still be pending on its barrier)
    const unsigned char *tab0 = a.words[0] + (size_t)super0 * S::kSuper;
    const unsigned char *tab1 = nstreams > 1 ? a.words[1] + (size_t)super0 * S::kSuper : nullptr;
    auto load_f = [&](uint32_t t, uint32_t b, uint32_t stage) {
        const bool other = NS > 1 && t >= tiles;   // the second stream's
        const uint32_t tl = other ? t - tiles : t;
        if (elect() && !*failed)
            copy_in(smem_u32(sm + L::kOffF) + (2 * b + stage) * S::kFTile,
                    (other ? tab1 : tab0) + (size_t)(tl / kTilesSuper) * S::kSuper + S::kWTile +
                        (tl % kTilesSuper) * S::kFTile,
                    S::kFTile, bar_f(2 * b + stage));
        __syncwarp();
    };
    auto load_w = [&](uint32_t g) {
        const bool other = NS > 1 && g >= nsupers_e;
        const uint32_t gl = (other ? g - nsupers_e : g) * kPer, n = min(kPer, (other ? supers1 : supers) - gl);
        const uint32_t dst = smem_u32(sm + L::kOffW) + (g % L::kWStages) * L::kWStage, bw = bar_w(g % L::kWStages);
        const unsigned char *src = (other ? tab1 : tab0) + (size_t)gl * S::kSuper;
        if (elect() && !*failed) {
            expect(bw, n * S::kWTile);
            for (uint32_t i = 0; i < n; ++i)
                copy_bulk(dst + i * S::kWTile, src + (size_t)i * S::kSuper, S::kWTile, bw);
        }
        __syncwarp();
    };
    if (warp >= Role<T>::kTestMma && warp < Role<T>::kChainMma) {
        const uint32_t b = warp - Role<T>::kTestMma;
        if (b < ntiles) load_f(b, b, 0);
        if (b + kBufs < ntiles) load_f(b + kBufs, b, 1);
    } else if (warp == Role<T>::kChainMma) {
        for (uint32_t g = 0; g < (uint32_t)L::kBufsE && g < nge; ++g) load_w(g);
    }

    // the candidates' planes: the testers' groups share the residue planes, the
    // reducers' and the chain's the test planes
    typename C::M m;
    if (warp < Role<T>::kTestMma) m.init(act ? c.p[ci] : (W)C::kIdle);
    if (warp < Role<T>::kReduce) {
        // residue planes: elements 8 k8 .. of w_b = 2^(6b) w_0 mod p
        constexpr uint32_t kShare = (K / 8 + kTesterGroups - 1) / kTesterGroups;
        const uint32_t k8a = min((warp / 4) * kShare, (uint32_t)(K / 8)), k8b = min(k8a + kShare, (uint32_t)(K / 8));
        // from the group's last element down, w_b = w_(b+1) / 64
        W x = C::power(m, 6u * (8u * k8b - 2u));
        for (uint32_t k8 = k8b; k8-- > k8a;) {
            W w[8];
#pragma unroll
            for (int j = 7; j >= 0; --j) {   // (element 0 is the bias)
                w[j] = x;
                x = C::div64(m, x);
            }
#pragma unroll
            for (int pl = 0; pl < C::kPlanes; ++pl) {
                const int shift = 32 * (pl / 3) + 11 * (pl % 3);
                const uint32_t mask = pl % 3 == 2 ? 0x3FFu : 0x7FFu;
                uint32_t v[4];
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    v[j] = f16x2_u11(((uint32_t)(w[2 * j] >> shift) & mask) |
                                     (((uint32_t)(w[2 * j + 1] >> shift) & mask) << 16));
                if (k8 == 0) v[0] = (v[0] & 0xFFFF0000u) | 0x6800u;   // 2048
                const uint4 q = make_uint4(v[0], v[1], v[2], v[3]);
                if constexpr (C::kInTmem)
                    st4(tbase + lanes + L::kColE + pl * (K / 2) + 4 * k8, q);
                else
                    *reinterpret_cast<uint4 *>(sm + L::kOffE + pl * L::kPlaneBytes + (cl / 8) * S::kRowGroup +
                                               k8 * 128 + (cl % 8) * 16) = q;
            }
        }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    } else if (warp < Role<T>::kTestMma) {
        if (warp < Role<T>::kReduce + 4) {
            cand_p[cl] = m.p;
            cand_q[cl] = C::qv(m);
        }
        // test planes: the binary expansion of (R mod p) / p, 32 bits per step
        // (w 2^32 = q p + w', so q = -w' p^-1 mod 2^32); f_b is its 24 bits
        // from bit 6b, rounded.  16 elements (96 bits and a look-ahead word)
        // at a time, the groups of warps in turn.
        constexpr uint32_t kGroups = (Role<T>::kTestMma - Role<T>::kReduce) / 4;
        static_assert(kGroups >= 2, "a group's words lie behind those of its turn before");
        const W c96 = C::c32(m);
        W x = m.one;
        auto digits = [&]() {
            x = C::step32(m, x, c96);
            return (uint32_t)(0u - (uint32_t)x * (uint32_t)m.pinv);
        };
        uint32_t at = 0;   // words of the expansion behind x
        for (uint32_t g = (warp - Role<T>::kReduce) / 4; g < K / 16; g += kGroups) {
            // elements 16 g .. 16 g + 15: digit b of element b + 1, so from bit
            // 96 g - 6; the first element of all is the bias
            uint32_t e[5];
            const uint32_t first = g ? 3 * g - 1 : 0;   // word that holds bit 96 g - 6
            for (; at < first; ++at) x = C::step32(m, x, c96);
#pragma unroll
            for (int i = 0; i < 5; ++i) {   // words first .. first + 4 (as if a zero word stood before the expansion)
                if (i == 0 && g == 0) e[i] = 0;
                else {
                    e[i] = digits();
                    ++at;
                }
            }
            uint32_t vh[4], vl[4];
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                const int bit = 26 + 6 * j, l = bit / 32, s = bit % 32;
                const uint32_t t = s ? __funnelshift_l(e[l + 1], e[l], s) : e[l];
                const uint32_t f = (uint32_t)(((uint64_t)t + 0x80u) >> 8);   // up to 2^24 (wraps)
                uint32_t lo12 = (f + 2048u) & 4095u;                         // low digit + 2048
                uint32_t hi12 = (((f + 2048u) >> 12) + 2048u) & 4095u;       // high digit + 2048
                if (j == 15 && g + 1 == K / 16) {
                    // the last element, against the words' 1: takes off the 2^22 that
                    // the biases leave in (hi 2^12 + lo), adds (half + 1) 2^8
                    hi12 = 1024u;
                    lo12 = 2048u + 256u * (half + 1);
                }
                const int i = (j / 2) % 4;
                if (j % 2 == 0) {
                    vh[i] = hi12;
                    vl[i] = lo12;
                } else {
                    vh[i] = f16x2_s12(vh[i] | (hi12 << 16));
                    vl[i] = f16x2_s12(vl[i] | (lo12 << 16));
                    if (j == 1 && g == 0) {   // the bias, 3072
                        vh[0] = (vh[0] & 0xFFFF0000u) | 0x6A00u;
                        vl[0] = (vl[0] & 0xFFFF0000u) | 0x6A00u;
                    }
                    if (i == 3) {
                        const uint32_t k8 = 2 * g + j / 8;
                        st4(tbase + lanes + L::kColF + 4 * k8, make_uint4(vh[0], vh[1], vh[2], vh[3]));
                        st4(tbase + lanes + L::kColF + K / 2 + 4 * k8, make_uint4(vl[0], vl[1], vl[2], vl[3]));
                    }
                }
            }
        }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    fence_before();
    __syncthreads();
    fence_after();

    if (warp < Role<T>::kReduce) {
        // ---------------------------------------------------------- testers
        constexpr int kB = kTestBlocks;
        const uint32_t buf = (warp / 4) % kBufs, b0 = warp / 8 * kB;   // tiles buf, buf + 2, ..; blocks b0, b0 + 1
        W *qr = reinterpret_cast<W *>(sm + L::kOffQ);
        uint32_t *qk = reinterpret_cast<uint32_t *>(sm + L::kOffQk);
        volatile uint32_t *qs = reinterpret_cast<uint32_t *>(sm + L::kOffQs);
        const W *rs = reinterpret_cast<const W *>(sm + L::kOffR) + b0 * kCands + cl;
        const uint32_t col = tbase + lanes + L::kColDF + buf * L::kDF + b0 * 16;
        const uint32_t window = 2 * half, window2 = window * 0x10001u;
        const uint32_t sh = C::shift(m.p);
        const float scale = C::kScale / ldexpf((float)m.p, -(int)sh);
        uint32_t tph = 0, unit = 0, rph = 0;
        for (uint32_t t0 = 0; t0 < ntiles; t0 += C::kUnit) {   // (whole units; a stream's tiles are)
            warp_wait(bar_r(unit), rph, fail);
            const W *ru = rs + unit * (C::kUnit * L::kRTile);
#pragma unroll
            for (uint32_t i = 0; i < (uint32_t)C::kUnit / kBufs; ++i) {   // this group's tiles of the unit
                const W *rt = ru + (buf + i * kBufs) * L::kRTile;   // residues: its blocks' starts, the last one's end
                uint32_t A[kB];   // in both halves (16 bits, from 22 or 21 + 1)
#pragma unroll
                for (int b = 0; b < kB; ++b) {
                    const uint32_t f =
                        __float_as_uint(fmaf(C::value(rt[(b + 1) * kCands], sh), scale, 12582912.0f)) >> C::kShift;
                    A[b] = __byte_perm(f, f, 0x1010);
                }
                warp_wait(bar_t(buf), tph, fail);
                tph ^= 1;
                fence_after();
                uint32_t vh[16], vl[16];
                ld16(col, vh);
                ld16(col + kRowsTile, vl);
                uint32_t mb[kB];
#pragma unroll
                for (int b = 0; b < kB; ++b) {
                    wait_ld();
                    uint32_t w[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j)   // bits 8..23 of two neighbours
                        w[j] = __byte_perm(vh[2 * j] * 4096u + vl[2 * j], vh[2 * j + 1] * 4096u + vl[2 * j + 1], 0x6521);
                    if (b + 1 < kB) {   // the next block's sums arrive meanwhile
                        ld16(col + 16 * (b + 1), vh);
                        ld16(col + kRowsTile + 16 * (b + 1), vl);
                    } else {
                        fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(bar_tf(buf));
                    }
                    uint32_t m0 = ~0u, m1 = ~0u;
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        m0 = __viaddmin_u16x2(w[j], ~A[b], m0);   // X - A + half
                        m1 = __viaddmin_u16x2(w[j], A[b], m1);    // X + A + half + 1
                    }
                    mb[b] = __viaddmin_u16x2(m0, 0u, m1);
                }
                // the least of both halves, in both
                uint32_t least = __viaddmin_u16x2(mb[0], 0u, mb[1]);
                least = __viaddmin_u16x2(least, 0u, __byte_perm(least, least, 0x1032));
                if (__any_sync(kFull, least <= window2)) {   // queue the suspects
                    const uint32_t t = t0 + buf + i * kBufs;
#pragma unroll
                    for (int b = 0; b < kB; ++b) {
                        const unsigned ps = __ballot_sync(kFull, act && min(mb[b] & 0xFFFFu, mb[b] >> 16) <= window);
                        if (!ps) continue;
                        uint32_t at = 0;
                        if (lane == 0) at = atomicAdd(suspects, (uint32_t)__popc(ps));
                        at = __shfl_sync(kFull, at, 0) + __popc(ps & ((1u << lane) - 1u));
                        if ((ps >> lane) & 1u) {
                            const uint32_t round = at / (32 * kBatches), e = at % (32 * kBatches);
                            // room once the batch's previous round has been replayed
                            for (uint32_t it = 0; reinterpret_cast<volatile uint32_t *>(replayed)[e / 32] < round; ++it)
                                if (*failed || it >= 8 * kWaitLimit) {
                                    *failed = 1;
                                    break;
                                }
                            const uint32_t s = NS > 1 && t >= tiles ? 1u : 0u;
                            qr[e] = rt[b * kCands];
                            qk[e] = (s << 31) | (((t - (s ? tiles : 0u)) * kBlocksTile + b0 + b) << 7) | cl;
                            __threadfence_block();
                            qs[e] = round + 1;
                        }
                        __syncwarp();
                    }
                }
            }
            if (lane == 0) mbar_arrive(bar_rf(unit));
            if (++unit == (uint32_t)C::kRUnits) {
                unit = 0;
                rph ^= 1;
            }
        }
        __syncwarp();
        __threadfence_block();
        if (lane == 0) atomicAdd(testers_done, 1u);
    } else if (warp < Role<T>::kTestMma) {
        // ------------------------------------------------ reducers and chain
        const W p = m.p;
        const typename C::Q q = C::qv(m);
        const uint2 shifts = make_uint2(a.shift11, a.shift22);
        W *rs = reinterpret_cast<W *>(sm + L::kOffR) + cl;
        const uint32_t units = tiles / C::kUnit, all_units = ntiles / C::kUnit;   // of the first stream, of both
        // the block products of tile i of unit te of buffer ge
        auto reduce_tile = [&](uint32_t ge, uint32_t te, uint32_t i, typename C::U *u) {
            uint32_t v[C::kPlanes][4];
#pragma unroll
            for (int pl = 0; pl < C::kPlanes; ++pl)
                ld4(tbase + lanes + L::kColDE + ge * L::kDE + pl * C::kBlocksE + te * kBlocksUnit + i * 4, v[pl]);
            wait_ld();
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                uint32_t e[C::kPlanes];
#pragma unroll
                for (int pl = 0; pl < C::kPlanes; ++pl) e[pl] = v[pl][b];
                u[b] = C::reduce(e, p, q, shifts);
            }
        };
        // a stream's first residue, and its last one into place
        auto second = [&](uint32_t s) { return (s ? a.second[1] : a.second[0]) != 0; };
        auto start = [&](uint32_t s) -> W {
            const W *in = second(s) ? c.s1 : c.s0;
            if (split) in = (second(s) ? sp->s1 : sp->s0) + (size_t)sub * sp->pitch;
            return act ? in[ci] : (W)0;
        };
        auto finish = [&](uint32_t s, W r) {
            if (!act || *failed) return;
            if (last) (second(s) ? c.s1 : c.s0)[ci] = T::canon(m, r);
            atomicAdd(c.nnext + ci, split ? range[1] - range[0] : s ? a.credit[1] : a.credit[0]);   // (the streams' ends may fall to two groups)
        };
        if constexpr (C::kReduceGroups != 0) {
            // Class 32: one group reduces, one moves the residues.  A buffer of
            // sums is a unit.
            static_assert(C::kReduceGroups == 0 || kUnitsE == 1, "one unit a buffer");
            typename C::U *us = reinterpret_cast<typename C::U *>(sm + L::kOffU) + cl;
            uint32_t us0 = 0, uph = 0;   // slot of block products, its use
            if (warp < Role<T>::kChain) {
                for (uint32_t un = 0; un < all_units; ++un) {
                    const uint32_t ge = un % L::kBufsE;
                    warp_wait(bar_e(ge), (un / L::kBufsE) & 1, fail);
                    fence_after();
                    if (un >= (uint32_t)C::kUUnits) warp_wait(bar_uf(us0), uph ^ 1, fail);
#pragma unroll
                    for (uint32_t i = 0; i < (uint32_t)C::kUnit; ++i) {
                        typename C::U u[4];
                        reduce_tile(ge, 0, i, u);
#pragma unroll
                        for (int b = 0; b < 4; ++b) us[(us0 * kBlocksUnit + i * 4 + b) * kCands] = u[b];
                    }
                    fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        mbar_arrive(bar_u(us0));
                        mbar_arrive(bar_ef(ge));
                    }
                    if (++us0 == (uint32_t)C::kUUnits) {
                        us0 = 0;
                        uph ^= 1;
                    }
                }
            } else {
                uint32_t un = 0, slot = 0, phase = 1;   // phase of the slot's release before its use
                for (uint32_t s = 0; s < nstreams; ++s) {
                    W r = start(s);
                    const uint32_t end = s ? all_units : units;
                    for (; un < end; ++un) {
                        warp_wait(bar_u(us0), uph, fail);
                        if (un >= (uint32_t)C::kRUnits) warp_wait(bar_rf(slot), phase, fail);
#pragma unroll
                        for (uint32_t i = 0; i < (uint32_t)C::kUnit; ++i) {
                            typename C::U u[4];
#pragma unroll
                            for (int b = 0; b < 4; ++b) u[b] = us[(us0 * kBlocksUnit + i * 4 + b) * kCands];
                            W *rt = rs + (slot * C::kUnit + i) * L::kRTile;
#pragma unroll
                            for (int b = 0; b < 4; ++b) {
                                rt[b * kCands] = r;
                                r = C::prod(r, u[b], p, q);
                            }
                            rt[4 * kCands] = r;
                        }
                        __syncwarp();
                        if (lane == 0) {
                            mbar_arrive(bar_r(slot));
                            mbar_arrive(bar_uf(us0));
                        }
                        if (++slot == (uint32_t)C::kRUnits) {
                            slot = 0;
                            phase ^= 1;
                        }
                        if (++us0 == (uint32_t)C::kUUnits) {
                            us0 = 0;
                            uph ^= 1;
                        }
                    }
                    finish(s, r);
                }
            }
        } else {
            // Class 64: the groups take units in turn, reduce a unit's block
            // products, which waits for no other group, then move the residue
            // on from where the group before left it.  (In class 32 this took
            // 1 to 3% longer than the two roles, here 6% less.)
            static_assert(C::kChainGroups <= C::kRUnits, "a group's next slot is one turn on at most");
            uint32_t ul = (warp - Role<T>::kChain) / 4, s = 0;   // unit of the stream, stream
            uint32_t slot = ul, turn = 0;                        // the unit's slot of residues, its uses before
            uint32_t left = units;                               // units of the stream
            if (NS > 1 && ul >= units) {   // (a stream of two units: the third group starts in the second)
                ul -= units;
                left = all_units - units;
                ++s;
            }
            // a buffer of sums is released by every group, when it has read its
            // last unit there or has none
            uint32_t seen = 0;   // buffers released by this group
            auto pass = [&](uint32_t end) {
                for (; seen < end; ++seen) {
                    warp_wait(bar_e(seen % L::kBufsE), (seen / L::kBufsE) & 1, fail);
                    if (lane == 0) mbar_arrive(bar_ef(seen % L::kBufsE));
                }
            };
            for (uint32_t un = slot; un < all_units; un += C::kChainGroups) {
                const uint32_t g = s * nsupers_e + ul / kUnitsE, te = ul % kUnitsE, ge = g % L::kBufsE;
                pass(g);
                warp_wait(bar_e(ge), (g / L::kBufsE) & 1, fail);
                fence_after();
                typename C::U u[kBlocksUnit];
#pragma unroll
                for (uint32_t i = 0; i < (uint32_t)C::kUnit; ++i) reduce_tile(ge, te, i, u + 4 * i);
                fence_before();
                __syncwarp();
                if (te + C::kChainGroups >= kUnitsE || ul + C::kChainGroups >= left) {
                    if (lane == 0) mbar_arrive(bar_ef(ge));
                    seen = g + 1;
                }
                if (turn) warp_wait(bar_rf(slot), (turn - 1) & 1, fail);
                W r = 0;
                if (un) {   // (at a stream's start too: the units stay in order)
                    const uint32_t before = slot ? slot - 1 : C::kRUnits - 1;
                    warp_wait(bar_r(before), slot ? turn & 1 : (turn - 1) & 1, fail);
                    r = rs[(before * C::kUnit + C::kUnit - 1) * L::kRTile + 4 * kCands];
                }
                if (ul == 0) r = start(s);
                W *ru = rs + slot * (C::kUnit * L::kRTile);
#pragma unroll
                for (uint32_t i = 0; i < (uint32_t)C::kUnit; ++i) {
#pragma unroll
                    for (int b = 0; b < 4; ++b) {
                        ru[i * L::kRTile + b * kCands] = r;
                        r = C::prod(r, u[4 * i + b], p, q);
                    }
                    ru[i * L::kRTile + 4 * kCands] = r;
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_r(slot));
                if (ul + 1 == left) finish(s, r);
                ul += C::kChainGroups;
                while (NS > 1 && ul >= left && s < 2) {
                    ul -= left;
                    left = all_units - units;
                    ++s;
                }
                slot += C::kChainGroups;
                if (slot >= (uint32_t)C::kRUnits) {
                    slot -= C::kRUnits;
                    ++turn;
                }
            }
            pass(nge);
        }
    } else if (warp < Role<T>::kChainMma) {
        // ------------------------------------- the tests' copies and MMAs
        // Warp b serves buffer b: tiles b, b + 2, ...  The whole warp keeps
        // the loop (its operands then stay in uniform registers), one elected
        // lane issues.
        const uint32_t tb = __shfl_sync(kFull, tbase, 0), b = warp - Role<T>::kTestMma;
        const uint32_t f0 = smem_u32(sm + L::kOffF) + b * 2 * S::kFTile;
        const uint32_t d = tb + L::kColDF + b * L::kDF;
        uint32_t stage = 0, sph = 0, fph = 1;
        for (uint32_t t = b; t < ntiles; t += kBufs) {
            warp_wait(bar_f(2 * b + stage), sph, fail);
            if (t >= kBufs) warp_wait(bar_tf(b), fph, fail);   // tile t - 2 read
            fph ^= 1;
            fence_after();
            const uint64_t w = mdesc(f0 + stage * S::kFTile, S::kRowGroup);
            if (elect()) {
#pragma unroll
                for (int pl = 0; pl < 2; ++pl)
#pragma unroll
                    for (int k = 0; k < K / 16; ++k)
                        mma_tmem(d + pl * kRowsTile, tb + L::kColF + pl * (K / 2) + k * 8, w + k * 16,
                                 idesc_n(kRowsTile), k != 0);
                commit(bar_t(b));
            }
            __syncwarp();
            stage ^= 1;
            sph ^= stage == 0;
            if (t >= kBufs && t + kBufs < ntiles) load_f(t + kBufs, b, stage);   // over tile t - 2
        }
        // every MMA has ended before the CTA does
        if (elect()) commit(bar_end(b));
        __syncwarp();
        ended(bar_end(b), 0);
    } else if (warp == Role<T>::kChainMma) {
        // ---------------------------------- the residues' copies and MMAs
        const uint32_t tb = __shfl_sync(kFull, tbase, 0);
        const uint64_t e = mdesc(smem_u32(sm + L::kOffE), S::kRowGroup);
        uint32_t loaded = min((uint32_t)L::kBufsE, nge);
        for (uint32_t g = 0; g < nge; ++g) {
            warp_wait(bar_w(g % L::kWStages), (g / L::kWStages) & 1, fail);
            if (g >= (uint32_t)L::kBufsE)   // the buffer's previous sums read
                warp_wait(bar_ef(g % L::kBufsE), (g / L::kBufsE - 1) & 1, fail);
            fence_after();
            if (loaded < nge) load_w(loaded++);   // over the words of g - kBufsE, whose sums have been read
            const uint64_t w = mdesc(smem_u32(sm + L::kOffW) + (g % L::kWStages) * L::kWStage, S::kRowGroup);
            const uint32_t d = tb + L::kColDE + (g % L::kBufsE) * L::kDE;
            if (elect()) {
#pragma unroll
                for (int pl = 0; pl < C::kPlanes; ++pl)
#pragma unroll
                    for (int k = 0; k < K / 16; ++k) {
                        if constexpr (C::kInTmem)
                            mma_tmem(d + pl * C::kBlocksE, tb + L::kColE + pl * (K / 2) + k * 8, w + k * 16,
                                     idesc_n(C::kBlocksE), k != 0);
                        else
                            mma_smem(d + pl * C::kBlocksE, e + (pl * L::kPlaneBytes + k * 256) / 16, w + k * 16,
                                     idesc_n(C::kBlocksE), k != 0);
                    }
                commit(bar_e(g % L::kBufsE));
            }
            __syncwarp();
        }
        if (elect()) commit(bar_end(kBufs));
        __syncwarp();
        ended(bar_end(kBufs), 0);
    } else {
        // ---------------------------------------------------------- replays
        const W *qr = reinterpret_cast<const W *>(sm + L::kOffQ);
        const uint32_t *qk = reinterpret_cast<const uint32_t *>(sm + L::kOffQk);
        const volatile uint32_t *qs = reinterpret_cast<const uint32_t *>(sm + L::kOffQs);
        const volatile uint32_t *head = suspects, *done = testers_done;
        for (uint32_t b = warp - Role<T>::kReplay;; b += C::kReplayWarps) {   // batches in turn
            uint32_t n = 0;
            bool fin = false;
            while (true) {   // until the batch is full or the testers have ended (each of which waits boundedly)
                fin = *done == (uint32_t)Role<T>::kReduce;
                __threadfence_block();
                const uint32_t got = *head;
                n = got > 32 * b ? min(got - 32 * b, 32u) : 0u;
                const bool go = n == 32 || fin || *failed;
                if (__all_sync(kFull, go)) break;
                __nanosleep(100);
            }
            n = __shfl_sync(kFull, n, 0);
            if (__any_sync(kFull, *failed || n == 0)) break;
            const uint32_t e = (b % kBatches) * 32 + lane, round = b / kBatches;
            const bool mine = lane < n;
            for (uint32_t it = 0; mine && qs[e] != round + 1; ++it)   // reserved, being written
                if (*failed || it >= kWaitLimit) {
                    *failed = 1;
                    break;
                }
            __syncwarp();
            __threadfence_block();
            const uint32_t key = mine ? qk[e] : 0u;
            const W r = mine ? qr[e] : (W)0;
            const uint32_t cand = key & (kCands - 1);
            const bool other = NS > 1 && key >> 31;   // the second stream
            const uint32_t k = (other && !split ? a.lo1 : range[0]) + ((key & 0x7FFFFFFFu) >> 7) * a.nb;
            const uint32_t end = other && !split ? a.hi1 : range[1];
            const uint32_t *mult = other ? a.mult[1] : a.mult[0];
            const bool replay = mine && !*failed;
            __syncwarp();
            if (lane == 0) reinterpret_cast<volatile uint32_t *>(replayed)[b % kBatches] = round + 1;   // entries taken
            replay_suspect<T>(replay, cand_p[cand], cand_q[cand], r, k, k < end ? min(a.nb, end - k) : 0u,
                              mult ? mult + (k - (other ? a.base1 : a.base)) : nullptr, other ? a.type[1] : a.type[0], h);
            if (n < 32) break;
        }
    }
    __syncwarp();
    // (copies still in flight after a wait that gave up; else each was waited for)
    if (*failed)
        for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    fence_before();
    __syncthreads();
    fence_after();
    if (tid == 0 && *failed) atomicOr(err, 4u);
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tbase) : "memory");
}

template <class T, int K, int NS>
__global__ void __launch_bounds__(Role<T>::kThreads, 1)
    walk_tc_kernel(ClassBuf<typename T::W> c, WalkTcArgs a, HitBuf h, SplitArgs<typename T::W> sp, uint32_t *err) {
    walk_tc<T, K, NS>(c, a, h, &sp, err, blockIdx.x, blockIdx.y);
}

// The walks of many searches in one launch (a batch's iteration): each CTA
// finds its window and keeps the window's record in shared memory.
template <class T, int K>
__global__ void __launch_bounds__(Role<T>::kThreads, 1)
    walk_tc_many_kernel(const WalkTcWin<typename T::W> *wins, uint32_t n, HitBuf h) {
    __shared__ WalkTcWin<typename T::W> w;
    if (threadIdx.x == 0) w = wins[window_of(wins, n, blockIdx.x)];
    __syncthreads();
    h.tagval = w.tag;
    walk_tc<T, K, 2>(w.c, w.a, h, nullptr, w.err, blockIdx.x - w.first_cta, 0);
}

// ------------------------------------------------------------------ launches

// Words of 47 digits (K = 48) hold the product of 16 multipliers below 2^17.6,
// words of 63 digits that of 16 below 2^23.6 or of 12 below 2^31.
static int word_depth(uint32_t top) { return top <= 202000u ? 48 : 64; }

uint32_t walk_tc_block(uint32_t top) { return top <= 12900000u ? 16u : 12u; }
uint32_t walk_tc_align(uint32_t top) { return kBlocksSuper * walk_tc_block(top); }

size_t walk_tc_words_bytes(uint32_t top, uint32_t steps) {
    const uint32_t per = walk_tc_align(top);
    const size_t nsuper = ((size_t)steps + per - 1) / per;
    return kTableHead + nsuper * (word_depth(top) == 48 ? WordShape<48>::kSuper : WordShape<64>::kSuper);
}

// One CTA: each thread counts the composites in its share of the flags' words,
// and after a scan over the threads writes them.
static __global__ void __launch_bounds__(1024) composites_kernel(uint32_t *out, const uint32_t *primebits, uint32_t nmin,
                                                                 uint32_t lo, uint32_t hi) {
    __shared__ uint32_t part[32];
    const uint32_t o0 = lo - nmin, o1 = hi - nmin, w0 = o0 / 32, w1 = (o1 + 31) / 32, lane = threadIdx.x % 32;
    const uint32_t per = (w1 - w0 + 1023) / 1024;
    const uint32_t a = min(w0 + threadIdx.x * per, w1), b = min(a + per, w1);
    auto word = [&](uint32_t w) {   // bit k: offset 32 w + k is in the range and composite
        uint32_t v = ~__ldg(primebits + w);
        if (32 * w < o0) v &= ~0u << (o0 - 32 * w);
        if (o1 - 32 * w < 32) v &= ~(~0u << (o1 - 32 * w));
        return v;
    };
    uint32_t count = 0;
    for (uint32_t w = a; w < b; ++w) count += __popc(word(w));
    uint32_t sum = count;   // inclusive over the warp
    for (uint32_t d = 1; d < 32; d <<= 1) {
        const uint32_t v = __shfl_up_sync(kFull, sum, d);
        if (lane >= d) sum += v;
    }
    if (lane == 31) part[threadIdx.x / 32] = sum;
    __syncthreads();
    uint32_t at = sum - count;
    for (uint32_t k = 0; k < threadIdx.x / 32; ++k) at += part[k];
    for (uint32_t w = a; w < b; ++w)
        for (uint32_t v = word(w); v; v &= v - 1) out[at++] = nmin + 32 * w + __ffs(v) - 1;
}
int launch_composites(uint32_t *out, const uint32_t *primebits, uint32_t nmin, uint32_t lo, uint32_t hi, cudaStream_t st) {
    if (hi <= lo) return 0;
    composites_kernel<<<1, 1024, 0, st>>>(out, primebits, nmin, lo, hi);
    return 1;
}

static uint32_t supers_of(uint32_t top, uint32_t steps) {
    const uint32_t per = walk_tc_align(top);
    return (uint32_t)(((uint64_t)steps + per - 1) / per);
}
uint32_t walk_words_ctas(uint32_t top, uint32_t steps) { return (supers_of(top, steps) * 17 * kBlocksSuper + 127) / 128; }
int walk_tc_shape(uint32_t top) { return word_depth(top) == 48 ? 0 : 1; }

void walk_words_win(WalkWordsWin &win, const uint32_t *mult, uint32_t base, uint32_t lo, uint32_t hi, uint32_t top,
                    unsigned char *table, uint32_t *digits) {
    win.mult = mult;
    win.base = base;
    win.lo = lo;
    win.hi = hi;
    win.nb = walk_tc_block(top);
    win.nsuper = supers_of(top, hi - lo);
    win.out = table;
    win.digits = digits;
}

int launch_walk_words(const uint32_t *mult, uint32_t base, uint32_t lo, uint32_t hi, uint32_t top, unsigned char *out,
                      WalkTcArgs &a, int stream, cudaStream_t st) {
    a.words[stream] = out + kTableHead;
    a.digits[stream] = reinterpret_cast<const uint32_t *>(out);
    if (hi <= lo) return 0;
    WalkWordsWin win{};
    walk_words_win(win, mult, base, lo, hi, top, out + kTableHead, reinterpret_cast<uint32_t *>(out));
    const uint32_t blocks = walk_words_ctas(top, hi - lo);
    if (cudaMemsetAsync(out, 0, kTableHead, st) != cudaSuccess) return 0;
    if (word_depth(top) == 48) walk_words_kernel<48><<<blocks, 128, 0, st>>>(win);
    else walk_words_kernel<64><<<blocks, 128, 0, st>>>(win);
    return 1;
}

int launch_walk_words_many(const WalkWordsWin *wins, uint32_t n, uint32_t ctas, int shape, cudaStream_t st) {
    if (!n) return 0;
    if (shape == 0) walk_words_many_kernel<48><<<ctas, 128, 0, st>>>(wins, n);
    else walk_words_many_kernel<64><<<ctas, 128, 0, st>>>(wins, n);
    return 1;
}

void walk_tc_args(WalkTcArgs &a, uint32_t top, uint32_t lo, uint32_t hi, uint32_t base) {
    a.lo = a.lo1 = lo;
    a.hi = a.hi1 = hi;
    a.base = a.base1 = base;
    a.credit[0] = a.credit[1] = hi - lo;
    a.nb = walk_tc_block(top);
    a.shift11 = 1u << 11;
    a.shift22 = 1u << 22;
}

template <class T, int K, int NS>
static int launch_tc(const ClassBuf<typename T::W> &c, const WalkTcArgs &a, const HitBuf &h,
                     const SplitArgs<typename T::W> &sp, uint32_t *err, cudaStream_t st) {
    using L = Lay<T, K>;
    static std::atomic<bool> configured[64];
    if (!configure(walk_tc_kernel<T, K, NS>, L::kSmem, configured)) return 0;
    const dim3 grid((c.cap + kCands - 1) / kCands, sp.n);
    walk_tc_kernel<T, K, NS><<<grid, Role<T>::kThreads, L::kSmem, st>>>(c, a, h, sp, err);
    return 1;
}

template <class T, int K>
static int launch_many(const WalkTcWin<typename T::W> *wins, uint32_t n, uint32_t ctas, const HitBuf &h, cudaStream_t st) {
    using L = Lay<T, K>;
    static std::atomic<bool> configured[64];
    if (!n || !configure(walk_tc_many_kernel<T, K>, L::kSmem, configured)) return 0;
    walk_tc_many_kernel<T, K><<<ctas, Role<T>::kThreads, L::kSmem, st>>>(wins, n, h);
    return 1;
}

uint32_t walk_tc_ctas(uint32_t cands) { return (cands + kCands - 1) / kCands; }

int launch_walk_tc32_many(const WalkTcWin<uint32_t> *wins, uint32_t n, uint32_t ctas, int shape, const HitBuf &h,
                          cudaStream_t st) {
    return shape ? launch_many<Cls32, 64>(wins, n, ctas, h, st) : launch_many<Cls32, 48>(wins, n, ctas, h, st);
}
int launch_walk_tc64_many(const WalkTcWin<uint64_t> *wins, uint32_t n, uint32_t ctas, int shape, bool lazy,
                          const HitBuf &h, cudaStream_t st) {
    if (lazy) return shape ? launch_many<Cls64L, 64>(wins, n, ctas, h, st) : launch_many<Cls64L, 48>(wins, n, ctas, h, st);
    return shape ? launch_many<Cls64, 64>(wins, n, ctas, h, st) : launch_many<Cls64, 48>(wins, n, ctas, h, st);
}

template <class T>
static int launch_tc(const ClassBuf<typename T::W> &c, const WalkTcArgs &a, uint32_t top, const HitBuf &h,
                     const SplitArgs<typename T::W> *sp, uint32_t *err, cudaStream_t st) {
    if (!c.cap || a.hi <= a.lo) return 0;
    SplitArgs<typename T::W> one{};
    one.n = 1;
    const SplitArgs<typename T::W> &parts = sp ? *sp : one;
    if (word_depth(top) == 48)
        return a.nstreams > 1 ? launch_tc<T, 48, 2>(c, a, h, parts, err, st) : launch_tc<T, 48, 1>(c, a, h, parts, err, st);
    return a.nstreams > 1 ? launch_tc<T, 64, 2>(c, a, h, parts, err, st) : launch_tc<T, 64, 1>(c, a, h, parts, err, st);
}

int launch_walk_tc32(const ClassBuf<uint32_t> &c, const WalkTcArgs &a, uint32_t top, const HitBuf &h,
                     const SplitArgs<uint32_t> *sp, uint32_t *err, cudaStream_t st) {
    return launch_tc<Cls32>(c, a, top, h, sp, err, st);
}
int launch_walk_tc64(const ClassBuf<uint64_t> &c, const WalkTcArgs &a, uint32_t top, const HitBuf &h,
                     const SplitArgs<uint64_t> *sp, uint32_t *err, cudaStream_t st, bool lazy) {
    return lazy ? launch_tc<Cls64L>(c, a, top, h, sp, err, st) : launch_tc<Cls64>(c, a, top, h, sp, err, st);
}

}  // namespace pfc
