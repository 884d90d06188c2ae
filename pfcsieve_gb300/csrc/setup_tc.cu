// setup_tc.cu -- the setup of the candidates' residues with the table-word fold
// on the tensor cores (tcgen05), for programs of at least kTcMinWords32 / 64 /
// Top words (kernels.cuh).  The description below is of class 64 below 2^64/3
// (the lazy class); the other classes follow it.
//
// The setup evaluates a program of table words Z (products of primes,
// kernels.cuh Prog) into each candidate's residue.  The costly part on the
// integer pipe is the fold of each word against the candidate's position
// residues, T = sum_b z_b w_b with w_b = 2^(8b+32) mod p: an exact integer
// contraction (words x bytes) x (bytes x candidates).  Here it runs on the
// tensor cores in fp16 with fp32 accumulation and stays exact:
//   * the words are 1792-bit: each is the product of a pair of the program's
//     896-bit words (host.hpp TcProg), so half as many words reach the
//     CUDA cores; a word is 225 balanced base-256 digits z_b (-128..127, the
//     last one a carry of 0 or 1);
//   * a candidate's residues w_b are balanced base-256 digits too, in 8 planes
//     W_a[b];
//   * digits of either sign keep a whole word's sums in one accumulator:
//     S_a[word, cand] = sum_b z_b W_a[b] has |S_a| <= 225 * 128 * 128 < 2^22
//     and rides on a bias of 1.5 * 2^23 (digit 225: 4096 in every word, 3072
//     in every plane), so every partial sum is an integer in [2^23, 2^24),
//     exact in fp32, and the accumulator's bits are 0x4B400000 + S_a;
//   * on the CUDA cores neighbouring planes combine as t_j = S_2j + 256 S_2j+1
//     + 0x8B400000 straight from those bits, which is positive and below 2^32,
//     so T' = sum_j t_j 2^(16j) needs no corrections: digit 226, 1 in every
//     word, carries minus the constant's residue mod p, and T' = Z 2^32 (mod p).
// The programs are first laid out as fp16 tiles of 128 words (A operand, M =
// 128, K = 240, the shared-memory image in three parts of K = 80;
// tc_pack_kernel multiplies the word pairs, once per job).  One CTA owns 32
// candidates: their planes stay in shared memory as the MMA's B operand,
// K-major, one 8-row core group per candidate (row = plane), so that one MMA
// with N = 256 covers the 32 candidates x 8 planes and a candidate's 8 sums are
// adjacent TMEM columns (word = TMEM lane).  Two such buffers of 256 columns.
// A warp copies the tiles' parts (cp.async.bulk) as the MMAs release them, a
// warp issues the MMAs, 15 of K = 16 per tile, and 16 warps take the sums of
// the other buffer: a thread owns one word (TMEM lane) and a quarter of the
// candidates, and keeps a running product for each of those in registers:
// it reduces T' by one Montgomery round, u = (T' + m p) / 2^32 with m = -T' p^-1
// mod 2^32, so u = Z (mod p) up to a power of R and u < 2^48 + p, and multiplies
// it in (two lazy rounds; a product lowers the power of R by one, as a word on
// the integer pipe does).  A lane's words all belong to one group of the
// program, so the squarings between the groups (Horner over exponent bits) wait
// until the program's end, where the lanes' products are multiplied over a tree
// through shared memory.  So a tile needs no barrier among the threads.
// Class 32 (p < 2^31) runs the same kernel with 4 planes, 64 candidates per CTA
// (N = 64 x 4 = 256 again), T' < 2^48 reduced by one 32-bit round and one
// Montgomery product (R = 2^32) per word; class 64 from 2^64/3 on keeps
// canonical residues.  The result equals setup_kernel's: the same product,
// exact arithmetic, canonical residues at the end.  Every wait is bounded; after one that gave up the kernel sets
// bit 1 of `flags`, frees its TMEM and stores nothing.
#include <cuda_runtime.h>

#include <cstdint>

#include "host.hpp"
#include "tcgen05.cuh"
#include "walk.cuh"

namespace pfc {
namespace {

constexpr int kTcWorkers = 512;               // threads that take the sums
constexpr int kTcThreads = kTcWorkers + 64;   // and the warps of the MMAs and of the copies
constexpr uint32_t kTcWords = kTcLanes;       // words per tile: MMA M, TMEM lanes
constexpr uint32_t kTcN = 256;                // MMA N: candidates x planes
constexpr uint32_t kTcDigits = 225;           // digits of a 1792-bit word, with its carry
constexpr uint32_t kTcK = 240;                // MMA K: digits, bias, offset, zeros
constexpr uint32_t kStages = 3;               // parts of a tile
constexpr uint32_t kStageK = kTcK / kStages;
constexpr uint32_t kStageGroup = (kStageK / 8) * 128;             // bytes between 8-row core groups of a part
// and of the planes: 16 bytes more than they take, so that the threads that
// write the same plane of neighbouring candidates hit distinct banks
constexpr uint32_t kRowGroup = (kTcK / 8) * 128 + 16;
constexpr uint32_t kStageBytes = (kTcWords / 8) * kStageGroup;    // 20,480
constexpr uint32_t kATile = kStages * kStageBytes;                // 61,440
constexpr uint32_t kBTile = (kTcN / 8) * kRowGroup;               // 123,392: rows = candidate x plane
constexpr uint32_t kOffA = 0;
constexpr uint32_t kOffB = kOffA + kATile;
constexpr uint32_t kOffU = kOffB + kBTile;
static_assert(kTcDigits + 2 <= kTcK && kStageK % 16 == 0, "setup_tc shape");
static_assert(kStageBytes % 128 == 0 && kBTile % 128 == 0, "setup_tc alignment");
constexpr uint32_t kTBias = 0x8B400000u;      // 257 * 0x4B400000 mod 2^32, in every t_j

// byte offset of the core-matrix row holding elements (r, 8 k8 .. 8 k8 + 7)
__device__ __forceinline__ uint32_t tile_off(uint32_t r, uint32_t k8, uint32_t rowgroup) {
    return (r / 8) * rowgroup + k8 * 128 + (r % 8) * 16;
}

// two bytes (bits 0-7 and 8-15 of x, or 16-23 and 24-31 with hi) -> two fp16
// v - 128: the fp16 of 1024 + v is 0x6400 | v (v < 1024), less 1152
template <bool HI>
__device__ __forceinline__ uint32_t f16x2_of_bytes(uint32_t x) {
    return sub_f16x2(__byte_perm(x, 0x64u, HI ? 0x4342u : 0x4140u), 0x64806480u);
}

// eight bytes -> eight fp16 v - 128 (16 bytes, one core-matrix row)
__device__ __forceinline__ uint4 f16x8(uint64_t bytes8) {
    const uint32_t lo = (uint32_t)bytes8, hi = (uint32_t)(bytes8 >> 32);
    return make_uint4(f16x2_of_bytes<false>(lo), f16x2_of_bytes<true>(lo), f16x2_of_bytes<false>(hi),
                      f16x2_of_bytes<true>(hi));
}

// bytes 0..3 of four words each, transposed
__device__ __forceinline__ void transpose4(uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t (&out)[4]) {
    const uint32_t t0 = __byte_perm(a, b, 0x5140), t1 = __byte_perm(c, d, 0x5140);
    const uint32_t t2 = __byte_perm(a, b, 0x7362), t3 = __byte_perm(c, d, 0x7362);
    out[0] = __byte_perm(t0, t1, 0x5410);
    out[1] = __byte_perm(t0, t1, 0x7632);
    out[2] = __byte_perm(t2, t3, 0x5410);
    out[3] = __byte_perm(t2, t3, 0x7632);
}

// What differs between the size classes: the residue type, its planes, the
// reduction of T' and the product of a reduced word into a running value.
template <class T>
struct TcClass;

// class 64 below 2^64/3: residues in [0, 2p) between squarings, lazy rounds
template <>
struct TcClass<Cls64L> {
    using W = uint64_t;
    using M = Mont64;
    static constexpr int kPlanes = 8;
    static constexpr uint64_t kIdle = 0x1FFFFFFFFFFFFFFFull;   // an idle slot works on 2^61 - 1
    struct __align__(16) Cand {
        W p;
        uint32_t q, pad;   // -p^-1 mod 2^32
    };
    __device__ static __forceinline__ Cand cand(const M &m) { return {m.p, m.q32, 0u}; }
    // 2^bits mod p, from the next power of R down by rounds of 2^-32
    __device__ static __forceinline__ W power(const M &m, uint32_t bits) {
        const uint32_t k = (bits + 63) / 64, down = 64 * k - bits;
        W x = m.mont_R_pow(k - 1);
        if (down >= 32) x = redc64l(x, 1u, m.p, m.q32);
        if (down % 32) x = redc64l(x, 1u << (32 - down % 32), m.p, m.q32);
        return x >= m.p ? x - m.p : x;
    }
    __device__ static __forceinline__ W div256(const M &m, W x) {
        x = redc64l(x, 1u << 24, m.p, m.q32);
        return x >= m.p ? x - m.p : x;
    }
    // kTBias (1 + 2^16) (1 + 2^32) mod p
    __device__ static __forceinline__ W bias(const M &m) {
        const W g = m.to_mont((W)kTBias * 65537u);
        return addmod64(m.mul(g, 1u), m.mul(g, 1ull << 32), m.p);
    }
    // byte pl of w's balanced digits, plus 128 (w below 2^64/3 needs no sign)
    __device__ static __forceinline__ W digits(W w, W) { return w + 0x8080808080808080ull; }
    // T' = L + 2^32 H < 2^80: u = (T' + m p) / 2^32 with m = -T' p^-1 mod 2^32,
    // so u = T' 2^-32 (mod p) and u < 2^48 + p; t0 + lo(m p0) = 2^32 [t0 != 0]
    __device__ static __forceinline__ W reduce(const uint32_t (&t)[4], const Cand &c) {
        const uint64_t L = (uint64_t)t[0] + ((uint64_t)t[1] << 16), H = (uint64_t)t[2] + ((uint64_t)t[3] << 16);
        const uint32_t tw0 = (uint32_t)L;
        const uint64_t Mh = (L >> 32) + H;
        const uint32_t mm = tw0 * c.q;
        const uint64_t lo = (uint64_t)mm * (uint32_t)c.p;
        return Mh + (uint64_t)mm * (uint32_t)(c.p >> 32) + (lo >> 32) + (tw0 != 0 ? 1u : 0u);
    }
    // two lazy rounds, s < 2p: below (3p + 2p u_hi + 2^32 p) / 2^32, which is
    // below 2p for u < 2^48 + p and p < 2^64/3
    __device__ static __forceinline__ W prod(W s, W u, const Cand &c) {
        return cios_round(redc64l(s, (uint32_t)u, c.p, c.q), s, (uint32_t)(u >> 32), c.p, c.q);
    }
    __device__ static __forceinline__ W canon(W s, const Cand &c) { return s >= c.p ? s - c.p : s; }
};

// class 64 from 2^64/3: canonical residues, R = 2^64
template <>
struct TcClass<Cls64> {
    using W = uint64_t;
    using M = Mont64;
    static constexpr int kPlanes = 8;
    static constexpr uint64_t kIdle = TcClass<Cls64L>::kIdle;
    struct __align__(16) Cand {
        W p, q;   // p^-1 mod 2^64
    };
    __device__ static __forceinline__ Cand cand(const M &m) { return {m.p, m.pinv}; }
    __device__ static __forceinline__ W power(const M &m, uint32_t bits) {
        const uint32_t k = (bits + 63) / 64, down = 64 * k - bits;
        const W x = m.mont_R_pow(k - 1);
        return down ? m.mul(x, 1ull << (64 - down)) : x;
    }
    __device__ static __forceinline__ W div256(const M &m, W x) { return m.mul(x, 1ull << 56); }
    __device__ static __forceinline__ W bias(const M &m) { return TcClass<Cls64L>::bias(m); }
    // (eight digits hold -0x8080.. .. 0x7F7F.., 2^64 values)
    __device__ static __forceinline__ W digits(W w, W p) {
        return (w > 0x7F7F7F7F7F7F7F7Full ? w - p : w) + 0x8080808080808080ull;
    }
    // as the lazy class, where (T' mod 2^32 + m p) / 2^32 is at most p and the
    // rest of T' below 2^48: less p where the sum passes it
    __device__ static __forceinline__ W reduce(const uint32_t (&t)[4], const Cand &c) {
        const uint64_t L = (uint64_t)t[0] + ((uint64_t)t[1] << 16), H = (uint64_t)t[2] + ((uint64_t)t[3] << 16);
        const uint32_t tw0 = (uint32_t)L;
        const uint64_t Mh = (L >> 32) + H;
        const uint32_t mm = 0u - tw0 * (uint32_t)c.q;
        const uint64_t lo = (uint64_t)mm * (uint32_t)c.p;
        const uint64_t u = (uint64_t)mm * (uint32_t)(c.p >> 32) + (lo >> 32) + (tw0 != 0 ? 1u : 0u) + Mh;
        return u < Mh || u >= c.p ? u - c.p : u;
    }
    __device__ static __forceinline__ W prod(W s, W u, const Cand &c) { return redc64(s, u, c.p, c.q); }
    __device__ static __forceinline__ W canon(W s, const Cand &) { return s; }
};

// class 32: canonical residues, R = 2^32
template <>
struct TcClass<Cls32> {
    using W = uint32_t;
    using M = Mont32;
    static constexpr int kPlanes = 4;
    static constexpr uint32_t kIdle = 0x7FFFFFFFu;   // an idle slot works on 2^31 - 1
    struct __align__(8) Cand {
        W p;
        uint32_t q;   // p^-1 mod 2^32
    };
    __device__ static __forceinline__ Cand cand(const M &m) { return {m.p, m.pinv}; }
    __device__ static __forceinline__ W power(const M &m, uint32_t bits) {
        const uint32_t k = (bits + 31) / 32, down = 32 * k - bits;
        const W x = m.mont_R_pow(k - 1);
        return down ? m.mul(x, 1u << (32 - down)) : x;
    }
    __device__ static __forceinline__ W div256(const M &m, W x) { return m.mul(x, 1u << 24); }
    // kTBias (1 + 2^16) mod p
    __device__ static __forceinline__ W bias(const M &m) { return (W)((uint64_t)kTBias * 65537u % m.p); }
    // (four digits hold -0x80808080 .. 0x7F7F7F7F)
    __device__ static __forceinline__ W digits(W w, W p) { return (w > 0x7F7F7F7Fu ? w - p : w) + 0x80808080u; }
    // T' < 2^48: with m = lo(T') p^-1 mod 2^32, T' - m p = 0 (mod 2^32), so
    // u = hi(T') - hi(m p) exactly, in (-p, 2^16), plus p when negative:
    // u = T' 2^-32 (mod p), u < 2^31
    __device__ static __forceinline__ W reduce(const uint32_t (&t)[2], const Cand &c) {
        const uint64_t L = (uint64_t)t[0] + ((uint64_t)t[1] << 16);
        const uint32_t m1 = (uint32_t)L * c.q;
        const int32_t u = (int32_t)(uint32_t)(L >> 32) - (int32_t)(((uint64_t)m1 * c.p) >> 32);
        return (W)(u < 0 ? u + (int32_t)c.p : u);
    }
    // s < p and u < 2^31: s u < p 2^32, one canonical round
    __device__ static __forceinline__ W prod(W s, W u, const Cand &c) { return redc32(s, u, c.p, c.q); }
    __device__ static __forceinline__ W canon(W s, const Cand &) { return s; }
};

template <class T>
struct TcLayout {
    using C = TcClass<T>;
    using W = typename C::W;
    static constexpr int kPlanes = C::kPlanes;
    static constexpr int kCands = kTcN / kPlanes;              // candidates per CTA
    static constexpr int kOwn = kCands / 4;                    // running products per thread
    static constexpr int kParts = kTcWorkers / kCands;         // threads per candidate in the planes
    // the lanes' products [cands][kUStride], partial products [parts][cands], p and q, Mont(1), Mont(R^corr)
    // of both programs, the squarings before each lane, all up to it
    static constexpr uint32_t kUStride = kTcWords + 1;   // odd: column reads hit distinct banks
    static constexpr uint32_t kOffPart = kOffU + kCands * kUStride * sizeof(W);
    static constexpr uint32_t kOffCand = kOffPart + kParts * kCands * sizeof(W);
    static constexpr uint32_t kOffOne = kOffCand + kCands * sizeof(typename C::Cand);
    static constexpr uint32_t kOffCorr = kOffOne + kCands * sizeof(W);
    static constexpr uint32_t kOffSq = kOffCorr + 2 * kCands * sizeof(W);
    static constexpr uint32_t kOffBar = kOffSq + 2 * (kTcWords + 1) * 4 + 8;
    static constexpr uint32_t kBars = 2 * kStages + 4 + 1;
    static constexpr uint32_t kOffMisc = kOffBar + 8 * kBars;   // failed, TMEM address
    static constexpr uint32_t kSmemBytes = kOffMisc + 16;
    static constexpr uint32_t kGroupsK = (kTcDigits + 7) / 8;   // groups of 8 elements with digits
    static constexpr uint32_t kChunk = (kGroupsK + kParts - 1) / kParts;
    static_assert(kSmemBytes <= 227 * 1024, "setup_tc shared memory");
    static_assert(kOffBar % 8 == 0 && kOffCand % 16 == 0, "setup_tc alignment");
    static_assert(kOwn * kPlanes == 64, "two loads of 32 columns a tile");
};

}  // namespace

// One thread per word slot of a tile: the 1792-bit word (the product of a
// pair of 896-bit words, one alone, or 1) as fp16 digits in
// the tile's shared-memory image.  The product is formed column by column in
// radix 2^28 (a column sums at most 32 products of 28-bit limbs, below 2^61
// with its carry) and written eight digits at a time (adding 128 to every
// byte makes the bytes of the sum the balanced digits plus 128).
__global__ void tc_pack_kernel(const WideWord *words, const uint32_t *src, uint32_t nw, uint32_t ntiles, uint4 *out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ntiles * kTcWords) return;
    const uint32_t tile = i / kTcWords, slot = i % kTcWords;
    uint32_t x[kWideLimbs], y[kWideLimbs];
    const uint32_t s = i < nw ? __ldg(src + i) : kTcOne;
    const bool have = s != kTcOne, pair = have && (s >> 31);
    const uint32_t w = s & 0x7FFFFFFFu;
#pragma unroll
    for (int k = 0; k < kWideLimbs; ++k) {
        x[k] = have ? words[w].limb[k] : (k == 0 ? 1u : 0u);
        y[k] = pair ? words[w + 1].limb[k] : (k == 0 ? 1u : 0u);
    }
    unsigned char *tb = reinterpret_cast<unsigned char *>(out) + (size_t)tile * kATile;
    auto row = [&](uint32_t k8) {
        constexpr uint32_t per = kStageK / 8;
        return reinterpret_cast<uint4 *>(tb + (k8 / per) * kStageBytes + tile_off(slot, k8 % per, kStageGroup));
    };
    uint64_t carry = 0, bits = 0, up = 0;
    int nbits = 0;
    uint32_t k8 = 0;
    for (int c = 0; c < 2 * kWideLimbs; ++c) {
        uint64_t col = carry;
        for (int a = c < kWideLimbs ? 0 : c - kWideLimbs + 1; a <= c && a < kWideLimbs; ++a)
            col += (uint64_t)x[a] * y[c - a];
        const uint64_t limb = col & ((1ull << kWideRadixBits) - 1u);
        carry = col >> kWideRadixBits;
        // 28 new bits above the nbits (< 64) already gathered
        bits |= limb << nbits;
        if (nbits + kWideRadixBits >= 64) {   // 64 bits complete
            const uint64_t sum = bits + 0x8080808080808080ull + up;
            up = sum < bits ? 1u : 0u;
            *row(k8++) = f16x8(sum);
            const int used = 64 - nbits;      // bits of this limb in the completed group
            bits = used < kWideRadixBits ? limb >> used : 0;
            nbits = kWideRadixBits - used;
        } else {
            nbits += kWideRadixBits;
        }
    }
    // the last carry, the bias's 4096, the offset's 1
    *row(k8++) = make_uint4((up ? 0x3C00u : 0u) | 0x6C000000u, 0x3C00u, 0u, 0u);
    *row(k8) = make_uint4(0u, 0u, 0u, 0u);
}

// What bounds it: the CUDA cores' multiply pipe, which the ten (class 32:
// three) wide multiplies per word and candidate keep busy 79% of the time; the
// tensor cores, 15 MMAs of 128 cycles a tile, are at 65 to 74%.  A tile takes
// about 2,950 cycles (class 64, 20,330 words x 144,000 candidates: 3.96 ms;
// unsigned bytes in two accumulators a plane, one buffer of sums and barriers
// around each tile took 8.01 ms), 2,600 in class 32 (1.69 ms, before 3.59);
// a CTA's fixed part, planes, first tile and the final tree, about 18,000.
template <class T>
__global__ void __launch_bounds__(kTcThreads, 1)
    setup_tc_kernel(ClassBuf<typename TcClass<T>::W> c, SetupArgs<WideWord> a, TcTiles ta, TcTiles tb,
                    uint32_t *flags, uint32_t block0, uint32_t radix) {
    using C = TcClass<T>;
    using Lay = TcLayout<T>;
    using W = typename C::W;
    using Cand = typename C::Cand;
    constexpr int kCands = Lay::kCands, kParts = Lay::kParts, kPlanes = Lay::kPlanes, kOwn = Lay::kOwn;
    extern __shared__ __align__(1024) unsigned char sm[];
    const uint32_t tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
    const uint32_t cnt = min(*c.count, c.cap);
    const uint32_t c0 = (blockIdx.x + block0) * kCands;
    if (c0 >= cnt) return;   // whole CTA idle

    W *U = reinterpret_cast<W *>(sm + kOffU);
    W *part = reinterpret_cast<W *>(sm + Lay::kOffPart);
    Cand *cands = reinterpret_cast<Cand *>(sm + Lay::kOffCand);
    W *ones = reinterpret_cast<W *>(sm + Lay::kOffOne);
    W *corr_pow = reinterpret_cast<W *>(sm + Lay::kOffCorr);
    uint32_t *lane_sq = reinterpret_cast<uint32_t *>(sm + Lay::kOffSq);   // squarings before a lane, of one program
    uint32_t *all_sq = lane_sq + kTcWords;                                // up to and before it [kTcWords + 1]
    uint32_t *misc = reinterpret_cast<uint32_t *>(sm + Lay::kOffMisc);
    volatile uint32_t *failed = misc;
    const uint32_t fail = smem_u32(misc);
    uint32_t *taddr_slot = misc + 1;
    const uint32_t bar = smem_u32(sm + Lay::kOffBar);
    auto bar_full = [&](uint32_t s) { return bar + 8 * s; };                       // a part of a tile landed
    auto bar_free = [&](uint32_t s) { return bar + 8 * (kStages + s); };           // and multiplied
    auto bar_ready = [&](uint32_t b) { return bar + 8 * (2 * kStages + b); };      // a buffer's sums ready
    auto bar_read = [&](uint32_t b) { return bar + 8 * (2 * kStages + 2 + b); };   // and read
    const uint32_t bar_end = bar + 8 * (2 * kStages + 4);

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(taddr_slot))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (uint32_t s = 0; s < 2 * kStages; ++s) mbar_init(bar + 8 * s, 1);
        for (uint32_t b = 0; b < 2; ++b) {
            mbar_init(bar_ready(b), 1);
            mbar_init(bar_read(b), kTcWorkers / 32);
        }
        mbar_init(bar_end, 1);
        *failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tbase = *taddr_slot;
    const int nprog = a.mode == (PFC_FACTORIAL | PFC_COMPOSITORIAL) ? 2 : 1;
    const uint32_t ntiles = ta.ntiles + (nprog == 2 ? tb.ntiles : 0u);

    // a part of tile t (none after a wait that gave up: a copy may then still
    // be pending on its barrier)
    auto load = [&](uint32_t t, uint32_t s) {
        const unsigned char *src = reinterpret_cast<const unsigned char *>(t < ta.ntiles ? ta.tiles : tb.tiles) +
                                   (size_t)(t < ta.ntiles ? t : t - ta.ntiles) * kATile + s * kStageBytes;
        if (elect() && !*failed) copy_in(smem_u32(sm + kOffA) + s * kStageBytes, src, kStageBytes, bar_full(s));
        __syncwarp();
    };

    // this thread's candidate while the planes are built, kParts threads each
    const uint32_t cl = tid % kCands, prt = tid / kCands, ci = c0 + cl;
    const bool act = tid < (uint32_t)kTcWorkers && ci < cnt;
    typename C::M m;
    if (tid < (uint32_t)kTcWorkers) {
        m.init(act ? c.p[ci] : (W)C::kIdle);
        if (prt == 0) {
            cands[cl] = C::cand(m);
            ones[cl] = m.one;
        }
        // w_b = 2^(8b+32) mod p as planes, rows kPlanes c .. kPlanes c + kPlanes
        // - 1: each part writes its share of the groups of 8 digits, from the
        // last digit down, w_b = w_(b+1) / 256
        const uint32_t k8a = min(prt * Lay::kChunk, Lay::kGroupsK), k8b = min(k8a + Lay::kChunk, Lay::kGroupsK);
        W x = k8a < k8b ? C::power(m, 8 * min(8 * k8b - 1, kTcDigits - 1) + 32) : 0;
        unsigned char *rows = sm + kOffB;
        for (uint32_t k8 = k8b; k8-- > k8a;) {
            const bool tail = k8 == kTcDigits / 8;   // one digit, the bias, the offset
            W w[8];
#pragma unroll
            for (int j = 7; j >= 0; --j) {
                w[j] = C::digits(x, m.p);
                if (!tail || j == 0) x = C::div256(m, x);
            }
            if (tail) {
#pragma unroll
                for (int j = 1; j < 8; ++j) w[j] = C::digits(0, m.p);
                const W off = C::bias(m);
                w[2] = C::digits(off ? m.p - off : 0, m.p);
            }
#pragma unroll
            for (int h = 0; h < kPlanes / 4; ++h) {
                uint32_t lo[4], hi[4];
                transpose4((uint32_t)(w[0] >> (32 * h)), (uint32_t)(w[1] >> (32 * h)), (uint32_t)(w[2] >> (32 * h)),
                           (uint32_t)(w[3] >> (32 * h)), lo);
                transpose4((uint32_t)(w[4] >> (32 * h)), (uint32_t)(w[5] >> (32 * h)), (uint32_t)(w[6] >> (32 * h)),
                           (uint32_t)(w[7] >> (32 * h)), hi);
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    uint4 v = f16x8(lo[r] | ((uint64_t)hi[r] << 32));
                    if (tail) v.x = (v.x & 0xFFFFu) | 0x6A000000u;   // 3072
                    *reinterpret_cast<uint4 *>(rows + tile_off(kPlanes * cl + 4 * h + r, k8, kRowGroup)) = v;
                }
            }
        }
        if (prt == (uint32_t)kParts - 1) {   // (the shortest share)
#pragma unroll
            for (int pl = 0; pl < kPlanes; ++pl)
                *reinterpret_cast<uint4 *>(rows + tile_off(kPlanes * cl + pl, kTcK / 8 - 1, kRowGroup)) =
                    make_uint4(0u, 0u, 0u, 0u);
            // the programs' power-of-R corrections
            for (int pi = 0; pi < nprog; ++pi) corr_pow[pi * kCands + cl] = m.mont_R_pow((pi == 0 ? a.a : a.b).corr);
        }
    } else if (warp == kTcThreads / 32 - 1) {
        for (uint32_t s = 0; s < kStages && ntiles; ++s) load(0, s);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();

    if (warp == kTcWorkers / 32) {
        // ------------------------------------------------------------- MMAs
        const uint32_t tb2 = __shfl_sync(kFull, tbase, 0);
        const uint64_t da = mdesc(smem_u32(sm + kOffA), kStageGroup), db = mdesc(smem_u32(sm + kOffB), kRowGroup);
        for (uint32_t t = 0; t < ntiles; ++t) {
            const uint32_t buf = t & 1;
            if (t >= 2) warp_wait(bar_read(buf), ((t >> 1) - 1) & 1, fail);
#pragma unroll 1
            for (uint32_t s = 0; s < kStages; ++s) {
                warp_wait(bar_full(s), t & 1, fail);
                fence_after();
                const uint64_t pa = da + s * (kStageBytes / 16), pb = db + s * (kStageK / 8 * 128 / 16);
                if (elect()) {
#pragma unroll
                    for (uint32_t k = 0; k < kStageK / 16; ++k)
                        mma_smem(tb2 + buf * kTcN, pa + k * 16, pb + k * 16, idesc_n(kTcN), s != 0 || k != 0);
                    commit(bar_free(s));
                    if (s == kStages - 1) commit(bar_ready(buf));
                }
                __syncwarp();
            }
        }
        // every MMA has ended before the CTA does
        if (elect()) commit(bar_end);
        __syncwarp();
        ended(bar_end, 0);
    } else if (warp > kTcWorkers / 32) {
        // ----------------------------------------------------------- copies
        for (uint32_t t = 1; t < ntiles; ++t)
            for (uint32_t s = 0; s < kStages; ++s) {
                warp_wait(bar_free(s), (t - 1) & 1, fail);
                load(t, s);
            }
    } else {
        // ---------------------------------------------------------- workers
        const uint32_t quad = warp % 4, own = warp / 4 * kOwn;   // TMEM lane quadrant, first candidate
        const uint32_t taddr = tbase + ((quad * 32u) << 16) + own * kPlanes;
        W s0 = 0, s1 = 0;
        uint32_t t = 0;
        for (int pi = 0; pi < nprog; ++pi) {
            const Prog<WideWord> &pg = pi == 0 ? a.a : a.b;
            const uint32_t tend = t + (pi == 0 ? ta.ntiles : tb.ntiles);
            W P[kOwn];   // the lane's running products, Montgomery form up to a power of R per word
#pragma unroll
            for (int k = 0; k < kOwn; ++k) P[k] = ones[own + k];
            for (; t < tend; ++t) {
                const uint32_t buf = t & 1;
                warp_wait(bar_ready(buf), (t >> 1) & 1, fail);
                fence_after();
                // 32 sums at a time
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    uint32_t v[32];
                    ld32(taddr + buf * kTcN + 32 * h, v);
                    wait_ld();
                    if (h == 1) {
                        fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(bar_read(buf));
                    }
#pragma unroll
                    for (int j = 0; j < 32 / kPlanes; ++j) {
                        const Cand cd = cands[own + h * (kOwn / 2) + j];
                        uint32_t tj[kPlanes / 2];
#pragma unroll
                        for (int k = 0; k < kPlanes / 2; ++k)   // (radix: 256, kept from becoming a shift)
                            tj[k] = v[kPlanes * j + 2 * k + 1] * radix + v[kPlanes * j + 2 * k];
                        W &y = P[h * (kOwn / 2) + j];
                        y = C::prod(y, C::reduce(tj, cd), cd);
                    }
                }
            }
            // the program's end: the lanes' products through shared memory, each
            // thread those of a share of the lanes of its own candidate, then a
            // tree over the shares; left of a group start go its squarings
#pragma unroll
            for (int k = 0; k < kOwn; ++k) U[(own + k) * Lay::kUStride + quad * 32 + lane] = P[k];
            if (tid < kTcWords) {
                uint32_t sq = 0;
                for (uint32_t g = 0; g < pg.ngroups; ++g)
                    if (__ldg(pg.groups + 3 * g) == tid) sq += __ldg(pg.groups + 3 * g + 2);
                lane_sq[tid] = sq;
            }
            asm volatile("bar.sync 1, %0;" ::"n"(kTcWorkers) : "memory");
            if (tid <= kTcWords) {
                uint32_t sq = 0;
                for (uint32_t k = 0; k < tid; ++k) sq += lane_sq[k];
                all_sq[tid] = sq;
            }
            constexpr uint32_t kShare = kTcWords / kParts;
            const Cand cd = C::cand(m);
            auto square = [&](W y, uint32_t n) {
                for (; n; --n) {
                    y = C::canon(y, cd);
                    y = C::prod(y, y, cd);
                }
                return y;
            };
            const W *row = U + cl * Lay::kUStride + prt * kShare;
            W acc = row[0];
            for (uint32_t k = 1; k < kShare; ++k)
                acc = C::prod(square(acc, lane_sq[prt * kShare + k]), C::canon(row[k], cd), cd);
            for (uint32_t n = 1; n < (uint32_t)kParts; n <<= 1) {
                part[prt * kCands + cl] = acc;
                asm volatile("bar.sync 1, %0;" ::"n"(kTcWorkers) : "memory");
                if ((prt & (2 * n - 1)) == 0)
                    acc = C::prod(square(acc, all_sq[(prt + 2 * n) * kShare] - all_sq[(prt + n) * kShare]),
                                  C::canon(part[(prt + n) * kCands + cl], cd), cd);
            }
            if (prt == 0) {
                // the combined search's second program (primorial words)
                // continues from the first's result
                if (pi) acc = C::prod(square(s1, all_sq[kTcWords]), C::canon(acc, cd), cd);
                acc = C::canon(square(acc, pg.final_sq), cd);
                acc = m.mul(acc, corr_pow[pi * kCands + cl]);
                if (nprog == 2 && pi == 0) s1 = acc;
                else s0 = acc;
            }
        }
        if (tid < (uint32_t)kCands && act && !*failed) {
            c.s0[ci] = s0;
            c.s1[ci] = s1;
            c.nnext[ci] = a.nnext0;
        }
    }
    __syncwarp();
    // (copies still in flight after a wait that gave up; else each was waited for)
    if (*failed)
        for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    fence_before();
    __syncthreads();
    fence_after();
    if (tid == 0 && *failed) atomicOr(flags, 2u);
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tbase) : "memory");
}

size_t tc_tile_bytes() { return kATile; }
uint32_t tc_tile_words() { return kTcWords; }

int launch_tc_pack(const WideWord *words, const uint32_t *src, uint32_t nw, uint32_t ntiles, void *out,
                   cudaStream_t st) {
    if (!ntiles) return 0;
    const uint32_t n = ntiles * kTcWords;
    tc_pack_kernel<<<(n + 127) / 128, 128, 0, st>>>(words, src, nw, ntiles, reinterpret_cast<uint4 *>(out));
    return 1;
}

// One CTA per 32 (class 64) or 64 (class 32) candidates, one
// CTA per SM (shared memory, TMEM); blocks [block0, block0 + nblocks) of the class
// buffer (nblocks 0: to the end).
uint32_t tc_setup_blocks(uint32_t cands) { return (cands + TcLayout<Cls64L>::kCands - 1) / TcLayout<Cls64L>::kCands; }
uint32_t tc_setup_blocks32(uint32_t cands) { return (cands + TcLayout<Cls32>::kCands - 1) / TcLayout<Cls32>::kCands; }

template <class T>
static int launch_tc(const ClassBuf<typename TcClass<T>::W> &c, const SetupArgs<WideWord> &a, const TcTiles &ta,
                     const TcTiles &tb, uint32_t *flags, cudaStream_t st, uint32_t block0, uint32_t nblocks) {
    if (!c.cap) return 0;
    constexpr int kCands = TcLayout<T>::kCands;
    const uint32_t all = (c.cap + kCands - 1) / kCands;
    if (block0 >= all) return 0;
    if (nblocks == 0 || nblocks > all - block0) nblocks = all - block0;
    static std::atomic<bool> configured[64];
    if (!configure(setup_tc_kernel<T>, TcLayout<T>::kSmemBytes, configured)) return 0;
    setup_tc_kernel<T><<<nblocks, kTcThreads, TcLayout<T>::kSmemBytes, st>>>(c, a, ta, tb, flags, block0, 256u);
    return 1;
}

int launch_setup64_tc(const ClassBuf<uint64_t> &c, const SetupArgs<WideWord> &a, const TcTiles &ta,
                      const TcTiles &tb, bool lazy, uint32_t *flags, cudaStream_t st, uint32_t block0, uint32_t nblocks) {
    return lazy ? launch_tc<Cls64L>(c, a, ta, tb, flags, st, block0, nblocks)
                : launch_tc<Cls64>(c, a, ta, tb, flags, st, block0, nblocks);
}

int launch_setup32_tc(const ClassBuf<uint32_t> &c, const SetupArgs<WideWord> &a, const TcTiles &ta,
                      const TcTiles &tb, uint32_t *flags, cudaStream_t st, uint32_t block0, uint32_t nblocks) {
    return launch_tc<Cls32>(c, a, ta, tb, flags, st, block0, nblocks);
}

}  // namespace pfc
