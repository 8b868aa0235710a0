// mps_common.cuh -- shared types of the sm_100a siever kernels.
//
// Device-side layout of one Factor= work item, the BSGS entry handed from
// the prep stage to the solve stage, and the relation record.  Everything is
// plain 64-bit integer data; nothing here touches torch.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace mps {

typedef unsigned long long u64;
typedef long long i64;
typedef unsigned int u32;

// Odd primes 3..65521 (6,541 of them): the sieving primes of the segment
// sieve (same set as gpu_sieve_primes, Math.hpp:342-358).
constexpr u32 kSievePrimes = 6541;
constexpr u32 kSieveMaxPrime = 65521;

// Moduli below this run the FP64-pipe arithmetic (exact for p < 2^49); larger
// ones 64-bit Montgomery.
constexpr u64 kFp64Limit = 1ull << 49;

// The multiplier of the baby-step tables' hash (fq_hash), and that of a launch whose
// primes all lie below kHashLow.
constexpr double kHashK = 1.6180339887498949, kHashKLow = kHashK * 524288.0;
constexpr u64 kHashLow = 1ull << 30;

// Largest baby-step count of one prime (a table of 2^13 slots at load 1/2).
constexpr u32 kMaxBaby = 4096;
// Measured on the B200 (C2 and C3 slices): a baby step (hash, insert) costs
// more than a giant step (hash, probe; 36 and 27 warp instructions), so m = 0.625
// sqrt(jcount) beats the square root, and words filled to 0.625 keys overflow rarely
// enough.
constexpr u32 kDefaultBabyScale = 160;   // m = ceil(sqrt(jcount)) x 160/256
constexpr u32 kDefaultFill = 160;        // fingerprint words: 0.625 keys per word on average

// Item constants, precomputed on the host once per item (all integer, exact).
struct DevItem {
    u64 babs_hi, babs_lo;  // |b| as 128-bit magnitude
    u64 cabs_hi, cabs_lo;  // |c|
    u32 b_neg, c_neg;      // signs
    i64 N0_raw;            // N0 as given (the p | b relation reports it, Math.hpp:496-502)
    i64 N1_raw;            // N1 as given (small-prime path, Math.hpp:506)
    u64 N0;                // max(N0, 0)  (Math.hpp:390)
    u64 N1;
    u64 cm;                // class modulus (>= 1)
    u64 n_start;           // smallest in-class n >= N0 (Math.hpp:393)
    u64 K;                 // in-class n in [n_start, N1): n = n_start + cm*k, k < K
    u32 has_work;          // K > 0
    u32 Q;                 // power-residue split modulus: g = gcd(Q, p - 1)
    u64 Q_rcp;             // floor((2^64 - 1) / Q)
    u32 cmQ;               // cm mod Q
    u32 nsQ;               // n_start mod Q
    u32 max_baby;          // cap on the baby-step count m of this item (<= kMaxBaby)
    u32 baby_scale;        // m = ceil(ceil(sqrt(jcount)) * baby_scale / 256) before the caps
    u32 item_index;
    u32 qf_n;              // prime factors of Q: qf_l[0..qf_n)
    u32 qf_l[9];
    double b_small, t_small;   // b and -c as signed numbers below 2^20, 0 when they are larger
    u32 strong;            // 1: a base-2 strong test screens the survivors (|b| <= 1 proves nothing)
    u32 split_more;        // 1: also split by primes l | p - 1 that Q does not hold (k_dlog)
    // Quadratic-character prefilter (both |b| and |c| below 2^32): for x = b
    // and x = -c, x = (-1)^neg 2^k o with o odd; rcp = floor((2^64-1) / o).
    u32 qr_on;
    u32 qr_neg[2], qr_k[2], qr_o[2];
    u64 qr_rcp[2];
};

// The split by primes l | p - 1 outside the split modulus: the kSplitPrimes
// sieving primes from 5 to kSplitLast; k is an l's index among them.  The first
// kSplitSmall (5 .. 19) have a slot of an entry each; the sieve finds the others,
// one of each of kSplitClasses size classes, a slot a class.  Events queue in
// lists by size, the classes' and one for the small l, for each of the two
// arithmetics (kFp64Limit).
constexpr u32 kSplitBase = 1;                 // 5's place among the sieving primes
constexpr u32 kSplitSmall = 6, kSplitGroups = 18, kSplitPrimes = kSplitSmall + 32 * kSplitGroups;
constexpr u32 kSplitClasses = 4, kSplitSizes = kSplitClasses + 1, kSplitLists = 2 * kSplitSizes, kSplitSlots = kSplitClasses + kSplitSmall;
__host__ __device__ constexpr u32 split_class(u32 k) {       // k >= kSplitSmall; l < 64, 256, 1024
    return k < 16 ? 0u : k < 52 ? 1u : k < 170 ? 2u : 3u;
}
constexpr u32 kSplitLast = 4259;
constexpr u32 primes_from_5(u32 below) {                     // number of primes 5 <= q < below
    u32 n = 0;
    for (u32 q = 5; q < below; q += 2) {
        bool prime = true;
        for (u32 d = 3; d * d <= q && prime; d += 2) prime = q % d != 0;
        n += prime;
    }
    return n;
}
static_assert(primes_from_5(kSplitLast) == kSplitPrimes - 1 && primes_from_5(kSplitLast + 1) == kSplitPrimes, "the last split prime");
static_assert(primes_from_5(20) == kSplitSmall, "5 .. 19");
static_assert(split_class(primes_from_5(64)) == 1 && split_class(primes_from_5(64) - 1) == 0 && split_class(primes_from_5(256)) == 2 &&
                  split_class(primes_from_5(256) - 1) == 1 && split_class(primes_from_5(1024)) == 3 &&
                  split_class(primes_from_5(1024) - 1) == 2, "the size classes");
__host__ __device__ constexpr u32 slot_list(u32 slot) { return slot < kSplitClasses ? slot : kSplitClasses; }

// One prime that reached the discrete-log stages: the candidates left are
// n = n_first + j*L, j in [0, jcount).  The prep writes p, n_first, L, jcount,
// item and the primes l | p - 1 to split the candidates by; k_dlog resolves those; k_setup applies them and fills t, G0,
// B, Bm and m for the solve of G0 * B^j == t (mod p).
struct Entry {
    u64 p;
    u64 t;                // -c
    u64 G0;               // b^n_first
    u64 B;                // b^L
    u64 Bm;               // B^m
    double pinv;          // 1/p (p < 2^49)
    u32 jcount;           // <= 10^7 (the width of the N range)
    u32 m;                // baby steps (<= kMaxBaby)
    u32 G;                // giant steps: ceil((jcount - 1) / m)
    u32 tw;               // log2 of the fingerprint table's words
    u64 n_first;          // smallest candidate n
    u64 L;
    u32 item;             // item index (batched runs)
    u32 pad;
    unsigned short k[kSplitClasses];   // the index of the l in each class's slot (a small l's is its slot - kSplitClasses)
    u32 ev[kSplitSlots];  // 0: no l in this slot, else what is known of j mod l (kEv*)
};
constexpr u32 kEvQueued = 1u << 31;   // an l is in the slot
constexpr u32 kEvValue = 0x1FFFu;     // j mod l, or one of
constexpr u32 kEvUnknown = 0x1FFFu;   //   nothing learned: b is an l-th power residue and so is t
constexpr u32 kEvReject = 0x1FFEu;    //   no n solves it: b is an l-th power residue and t is not
constexpr u32 kEvInvShift = 13;       // above it: the inverse mod l of the product of the earlier slots' primes
__host__ __device__ constexpr u32 slot_small(u32 slot) { return slot - kSplitClasses; }

// A prime l | p - 1 of an entry, queued for k_dlog.
struct SplitEvent {
    u32 entry;            // entry index
    u32 which;            // l's index << 16 | slot
};

// What a solve needs of an entry (plain residues in [0, p)): the smallest j in
// [0, jcount) with G0 * B^j == t (mod p), with m baby steps.
struct Solve {
    u64 p, t, G0, B, Bm;
    u64 jcount;
    u32 m;
};

// A relation before its order is known (q == 0 means "compute it").
struct RawRelation {
    u64 p, M, q;
    u32 item;
    u32 pad;
};

// Per-run device counters (one cache line each to keep atomics apart).
struct Counters {
    unsigned long long survivors;  u64 pad0[7];
    unsigned long long entries;    u64 pad1[7];
    unsigned long long relations;  u64 pad2[7];
    unsigned long long work_next;  u64 pad3[7];
    unsigned long long status;     u64 pad4[7];   // nonzero: an error bit set by a kernel
    unsigned long long primes;     u64 pad5[7];   // prime count (counting kernel only)
    unsigned long long steps;      u64 pad6[7];   // baby + giant steps executed by the BSGS
    unsigned long long prep_next;  u64 pad7[7];   // next survivor the prep's warps claim
    unsigned long long baby;       u64 pad8[7];   // the baby steps among `steps`
    unsigned long long events[kSplitLists]; u64 pad9[16 - kSplitLists];   // split events queued, by list
    unsigned long long setup_next; u64 pad10[7];  // next entry the set-up's warps claim
    unsigned long long dlog_next;  u64 pad12[7];  // next unit of 32 events k_dlog's warps claim
    unsigned long long big;        u64 pad11[7];  // entries left for a warp each (k_bsgs)
};

// Status bits a kernel may set (host turns them into error codes).
constexpr u64 kStatusSurvivorOverflow = 1ull << 0;
constexpr u64 kStatusEntryOverflow    = 1ull << 1;
constexpr u64 kStatusRelationOverflow = 1ull << 2;
constexpr u64 kStatusOrderFailed      = 1ull << 3;
constexpr u64 kStatusBadLaunch        = 1ull << 4;   // an entry the launch's kernel cannot take (host sizing error)

}  // namespace mps
