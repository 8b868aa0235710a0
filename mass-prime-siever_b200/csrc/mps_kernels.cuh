// mps_kernels.cuh -- launchers of the sm_100a siever kernels (mps_kernels.cu).
#pragma once

#include "mps_common.cuh"

namespace mps {

// Sieving-prime tables (device, built once per context).
struct SieveTables {
    const u32* sp;      // odd primes 3..65521
    const u64* rcp;     // floor((2^64 - 1) / q)
    const u64* inv;     // q^-1 mod 2^64
};

// Segment sieve of the odd numbers of [lo, hi) by the odd primes <= 65521:
// every survivor (an odd v >= 3 with no odd prime factor q <= min(65521,
// sqrt(hi)) other than itself) is appended to surv[].  include_two adds 2.
struct SieveArgs {
    u64 lo_odd;        // first odd >= max(lo, 3)
    u64 n_odds;        // odd numbers to sieve
    u64 hi;            // exclusive bound
    u32 include_two;
    u32 n_primes;      // sieving primes to use (those with q*q < hi, at most 6541)
    u32 n_split;       // split primes to look for in p - 1 (at most kSplitPrimes; 0: none)
    u32 item;          // item index stored with the survivors
};

// Where the survivors go: surv[], their items (or nullptr), and the split
// primes l | p - 1 of each (nullptr: not looked for): one 16-bit l index + 1
// per size class, 0 where there is none.
struct SurvOut {
    u64* surv;
    u32* item;
    u64* split;
    u64 cap;
};

// seg_words: segment bitmap words (1024, 2048 or 4096; 32 odd numbers each).  A range or
// wave of fewer than kFewSegs segments is cut into smaller ones, down to kLeastSegWords
// (2^20 integers at 10^9 as a chunk: 8 blocks, 40 us of sieve; now 64 blocks, 15 us.
// Switching at 296 segments instead costs 2^24 integers 48 us against 40: a segment has
// the same set-up for its 6,541 primes whatever its length).
constexpr u64 kFewSegs = 148;
constexpr u32 kLeastSegWords = 256;
constexpr u32 kDefaultSegWords = 2048;
cudaError_t launch_sieve(const SieveArgs& a, const SieveTables& t, const SurvOut& o, Counters* ctr, cudaStream_t s,
                         u32 seg_words = kDefaultSegWords, bool fit = true);   // fit: cut a short range smaller

// A wave: several runs (odd ranges of possibly different items) sieved by
// one launch; kept in device memory so that a captured graph is replayable.
constexpr u32 kMaxRuns = 512;
struct SieveRun {
    u64 lo_odd;        // first odd >= max(lo, 3)
    u64 n_odds;
    u64 seg_begin;     // index of this run's first segment in the wave
    u64 hi;            // end of the run's integer range (lo .. hi)
    u32 n_primes;
    u32 include_two;
    u32 item;
    u32 n_split;
};

// Device-resident state of one item: every P below p_done is sieved once the
// wave that covered it has committed; n_rel relations found, the first rel_cap
// of them kept in rel_buf (the item's reservation in a server's device pool;
// nullptr when the relations are not kept on the device).
struct ItemState {
    unsigned long long p_done;
    unsigned long long n_rel;
    unsigned long long waves;
    unsigned long long rel_cap;
    RawRelation* rel_buf;
    unsigned long long pad[3];
};
struct WaveDesc {
    u32 n_runs;
    u32 pad;
    u64 total_segs;
    SieveRun runs[kMaxRuns];
};
// After a wave: advance each run's item to the run's end, count relations.
cudaError_t launch_commit(const WaveDesc* w, const RawRelation* rel, const Counters* ctr, u64 rel_cap,
                          ItemState* st, cudaStream_t s);
// A run of an overflowed wave, redone on the host path: p_done = max(p_done, hi),
// its n relations rel[0..n) appended to the item's state.
cudaError_t launch_state_add(ItemState* st, u32 item, u64 hi, const RawRelation* rel, u64 n, cudaStream_t s);
// The wave's runs' seg_begin must count segments of seg_words * 32 odd numbers (seg_words
// 256, 512, 1024, 2048 or 4096).
cudaError_t launch_sieve_wave(const WaveDesc* w, const SieveTables& t, const SurvOut& o, Counters* ctr, int grid,
                              cudaStream_t s, u32 seg_words = kDefaultSegWords);

// Prep: filters, primality screen and class combination for every survivor
// (k_prep), the split by larger primes l | p - 1 (k_dlog; k_split finds them
// where the sieve has not), and the BSGS set-up, which also solves the primes
// with few candidates left (k_setup).
struct PrepArgs {
    const u64* surv;
    u64 surv_cap;
    const u32* surv_item;      // nullptr: every survivor belongs to `item0`
    const u64* surv_split;     // the sieve's split primes (SurvOut::split); nullptr: k_split finds them
    u32 split;                 // 0: no item has split_more, so there are no split events
    SieveTables tables;
    u32 item0;
    const DevItem* items;
    Entry* ent;
    u64 ent_cap;               // < 2^32
    SplitEvent* events;        // the lists of split events (set_event_lists)
    u32 ev_at[kSplitLists];    //   the place of each
    u32 ev_cap, ev_small;      //   events of a size class's list, and of a small-l list
    u32 two_fields;            // 0: kSplitSizes lists only, shared by both arithmetics
    u32* big;                  // ent_cap indices: the entries k_bsgs solves
    RawRelation* rel;
    u64 rel_cap;
    u32 full_mr;               // 1: 12-base Miller-Rabin on every survivor that passes the filters
    u32 m_cap;                 // baby steps per prime at most (what the launch's BSGS tables hold)
    u32 m_round;               // baby steps rounded up to a multiple of this (the BSGS iteration width)
    u32 tbits, fill;           // the BSGS launch's tables (BsgsArgs)
    u64 prime_below;           // survivors below this are prime (sieved by every prime up to their
                               // square root: 65521^2 for the sieve's survivors, 0 for caller-given numbers)
};
// Survivors of the sieve and entries of a range of that many odd numbers: the primes of
// any such range (the first one holds the most: pi(2 odds) stays below this, by 2% at
// 2^24 .. 2^26).  Beyond 65521^2 the survivors are 0.101 of the odd numbers.  168 B an
// entry (Entry, events, BSGS list) and 16 a survivor: 23 B an odd number.  (A range
// that has more all the same is halved.)
constexpr u64 entry_cap(u64 odds) { return odds / 8 + (1u << 17); }
// Events of a size class's list and of a small-l list for ent_cap entries: a prime has
// an l of a class with chance 1/4 at most (0.25 for 67 .. 251) and 0.72 small l on
// average, so neither fills up unless the caller's own primes were chosen for it; a
// full list loses splits, never relations.
constexpr u64 split_event_cap(u64 ent_cap) { return ent_cap / 4; }
constexpr u64 split_small_cap(u64 ent_cap) { return ent_cap / 4 * 3; }
constexpr u64 split_events(u64 ev_cap, u64 ev_small, u32 fields) { return fields * (kSplitClasses * ev_cap + ev_small); }
// Lays the lists out in events (split_events of them, below 2^32): the sizes' lists of one arithmetic, then of the other.
inline void set_event_lists(PrepArgs* a, SplitEvent* events, u64 ev_cap, u64 ev_small, u32 fields) {
    a->events = events;
    a->ev_cap = (u32)ev_cap;
    a->ev_small = (u32)ev_small;
    a->two_fields = fields == 2;
    for (u32 c = 0; c < kSplitLists; ++c)
        a->ev_at[c] = (u32)(c % kSplitSizes * ev_cap + c / kSplitSizes % fields * (kSplitClasses * ev_cap + ev_small));
}
// Split primes to look for in the range of an item with K in-class exponents.
u32 split_primes_for(u64 K);
constexpr u64 kSievedPrimeBelow = (u64)kSieveMaxPrime * kSieveMaxPrime;
// kernels of one launch_prep
constexpr u32 prep_launches(bool split, bool sieved) { return 2 + (split ? sieved ? 1 : 2 : 0); }
cudaError_t launch_prep(const PrepArgs& a, Counters* ctr, int grid, int num_sms, cudaStream_t s);

// Exact BSGS, one warp per entry.
struct BsgsArgs {
    const Entry* ent;
    const u32* big;            // indices of the entries to solve (ctr->big of them)
    u64 ent_cap;
    RawRelation* rel;
    u64 rel_cap;
    u32 tbits;                 // baby-step table of 2^tbits slots per warp
    u32 warps_per_block;
    u32 persistent;            // 1: work-stealing warps; 0: one warp per entry
    u32 chains;                // FP64 solve: independent chains per lane (1, 2, 4)
    u64 max_p;                 // largest p of the entries (>= 2^49: integer solve)
    u32 table_kind;            // FP64 solve: 0 = fingerprint words, 1 = 32-bit slots, 2 = 16-bit slots
    u32 load_shift;            // table kind 2: at most 2^-load_shift of a prime's slots are used
    u32 lanes;                 // table kind 2: lanes per prime, 32 (a warp) or 16 / 8 (groups; every
                               // entry must have p < 2^49, max_p > 0 and < 2^49 or the caller's guarantee)
    u32 low;                   // 1: every prime is below kHashLow (table kinds 0 and 3: kHashKLow instead of kHashK)
    u32 fill;                  // table kinds 0 and 3: a prime's table has at least m * 256 / fill words
                               // (1..256; 0 counts as 256), within the launch's 2^(tbits-1)
};
constexpr u32 kDefaultLoadShift = 2;
cudaError_t launch_bsgs(const BsgsArgs& a, Counters* ctr, int grid, cudaStream_t s);
cudaError_t bsgs_reserve_smem(size_t smem);   // call before capturing a launch_bsgs

// Order q = ord_p(b) and the exact 12-base primality check of every relation.
struct OrderArgs {
    RawRelation* rel;
    u64 rel_cap;
    const DevItem* items;
    SieveTables tables;
};
cudaError_t launch_order(const OrderArgs& a, Counters* ctr, int grid, cudaStream_t s);

// Counts the primes among the survivors (exact 12-base test) into ctr->primes.
cudaError_t launch_count_primes(const u64* surv, u64 surv_cap, Counters* ctr, int grid, cudaStream_t s);

// Roofline probes: 256 x grid threads x 8 independent chains x iters operations.
cudaError_t launch_mmul_peak(u64 p, u32 iters, int grid, u64* sink, cudaStream_t s);
cudaError_t launch_imad_peak(u32 iters, int grid, u32* sink, cudaStream_t s);
cudaError_t launch_fmul_peak(u64 p, u32 iters, int grid, u64* sink, cudaStream_t s);
cudaError_t launch_smem_or_peak(u32 iters, int grid, u32* sink, cudaStream_t s);   // 256 x grid x 8 x iters

// Test hooks: raw kernels on given inputs.
cudaError_t launch_is_prime(const u64* n, u32* out, u64 count, cudaStream_t s);
cudaError_t launch_bsgs_direct(const u64* cases /* p,B,G0,t,jcount */, u64* j_out, u64 count, u32 tbits,
                               u32 table_kind, cudaStream_t s);
cudaError_t launch_order_direct(const u64* bp /* b,p pairs */, u64* q_out, u64 count, SieveTables t,
                                cudaStream_t s);

// Dynamic shared memory of a BSGS launch: 4 << tbits bytes of table per warp,
// and for table kind 3 one count byte per eight bytes of table.
size_t bsgs_smem_bytes(u32 tbits, u32 warps_per_block, u32 table_kind);

}  // namespace mps
