// mps_kernels.cu -- the sm_100a kernels of the siever hot path.
//
//   k_sieve  segment sieve of the odd numbers by the odd primes <= 65521,
//            bitmap in shared memory, survivors compacted to global memory
//            (what psieve does, Gpu.hpp:385-455, sized for 148 SMs)
//   k_prep   per survivor: residues of b and -c, quadratic-character filter,
//            power-residue split over g = gcd(Q, p - 1) (Gpu.hpp:465-589,
//            Math.hpp:410-433), class combination; staged through shared-memory
//            queues so that every stage runs with full warps
//   k_dlog   per prime and l | p - 1 (5 .. 4259, found by the sieve, or by
//            k_split for given primes): the candidates' residue mod l
//   k_setup  applies those, sets the solve up, and solves entries with few
//            candidates left, one lane each
//   k_bsgs   exact baby-step giant-step, one warp per prime: baby-step table
//            of fingerprints + indices in shared memory, giant steps probed by
//            every lane, the smallest j found with a warp min-reduction
//            (the exact form of bsgs_wg / bsgs_wq, Gpu.hpp:329-383,600-650,
//            with run_bsgs's smallest-solution semantics, Math.hpp:439-483)
//   k_order  exact 12-base primality of each relation's p and q = ord_p(b)
//            (Math.hpp:209-251, 253-310), on the device
//
// All arithmetic is exact integer arithmetic; the relations equal those of
// the reference's CPU path.
#include "arith.cuh"
#include "mps_kernels.cuh"

#include <algorithm>
#include <cstddef>
#include <cuda_fp16.h>
#include <mutex>

namespace mps {

constexpr u32 FULL = 0xFFFFFFFFu;

#ifndef MPS_BSGS_MINB
#define MPS_BSGS_MINB 3      // resident 256-thread BSGS blocks per SM the register budget is cut for
#endif

// ---------------------------------------------------------------- helpers --

// |x| mod p for the 128-bit magnitude hi:lo (shift-and-subtract for the rare
// wide values), then the sign.
__device__ __forceinline__ u64 residue128(u64 hi, u64 lo, u32 neg, u64 p) {
    u64 r;
    if (hi == 0) {
        r = lo < p ? lo : lo % p;
    } else {
        r = hi % p;
        for (int bit = 63; bit >= 0; --bit) {
            r = (r << 1) | ((lo >> bit) & 1ull);
            if (r >= p) r -= p;
        }
    }
    return (neg && r) ? p - r : r;
}

__device__ __forceinline__ u64 isqrt_ceil_dev(u64 x) {
    if (x == 0) return 0;
    u64 r = (u64)sqrt((double)x);
    while (r > 0 && r * r >= x) --r;
    while (r * r < x) ++r;
    return r;
}

__device__ __forceinline__ void emit_relation(u64 p, u64 M, u64 q, u32 item, RawRelation* rel, u64 cap,
                                              Counters* ctr) {
    const u64 slot = atomicAdd(&ctr->relations, 1ull);
    if (slot < cap) {
        RawRelation r;
        r.p = p; r.M = M; r.q = q; r.item = item; r.pad = 0;
        rel[slot] = r;
    } else {
        atomicOr(&ctr->status, kStatusRelationOverflow);
    }
}

// -------------------------------------------------------------- the sieve --

// A segment is W words of shared-memory bitmap (W * 32 odd numbers); W is a
// template parameter (256, 512, 1024, 2048 or 4096 words: 1 .. 16 KB), chosen per
// launch.  kSegWords is the default.
constexpr u32 kSegWords = 2048;
constexpr u32 kSieveThreads = 256;
constexpr u32 kNumPattern = 10;               // 3..31: whole-word patterns, no atomics
constexpr u32 kSplitShared = 170;             // split primes below 1024: a warp's lanes share each
constexpr u32 kNumMedium = 171;               // primes below 1024: a warp's lanes share each prime

// Index j >= 0 of the first odd multiple v0 + 2j of q with v0 + 2j >= v0 (v0 odd).
__device__ __forceinline__ u32 first_odd_multiple(u64 v0, u32 q, u64 rcp) {
    const u64 qh = __umul64hi(v0, rcp);
    u64 r = v0 - qh * q;
    if (r >= q) r -= q;
    const u32 rr = (u32)r;
    return rr == 0 ? 0u : ((rr & 1u) ? (q - rr) >> 1 : q - (rr >> 1));
}

// Same, but never below q^2 (so q itself is never struck).
__device__ __forceinline__ u64 first_strike(u64 v0, u32 q, u64 rcp) {
    u64 j = first_odd_multiple(v0, q, rcp);
    const u64 qq = (u64)q * q;
    if (v0 + 2 * j < qq) j = (qq - v0) >> 1;
    return j;
}

template <u32 W>
struct SieveShared {
    u32 bits[W];
    u32 med_start[kNumMedium];
    u32 warp_sum[kSieveThreads / 32];
    unsigned long long block_base;
    unsigned short before[W];                 // survivors of the segment before each word
    unsigned short split_start[kSplitPrimes];
};

__device__ __forceinline__ void emit_two(u32 item, const SurvOut& o, Counters* ctr) {
    const u64 slot = atomicAdd(&ctr->survivors, 1ull);
    if (slot < o.cap) {
        o.surv[slot] = 2;
        if (o.item) o.item[slot] = item;
        if (o.split) o.split[slot] = 0;
    } else {
        atomicOr(&ctr->status, kStatusSurvivorOverflow);
    }
}

// One segment of len <= W * 32 odd numbers v0, v0 + 2, ... (v0 odd, >= 3),
// sieved by the first n_primes odd primes; survivors appended to o, with the
// first n_split split primes l | v - 1 of each.  Called by all threads of the block.
template <u32 W>
__device__ void sieve_segment(SieveShared<W>& sh, u64 v0, u32 len, u32 n_primes, u32 n_split, u32 item,
                              const SieveTables& t, const SurvOut& o, Counters* ctr) {
    constexpr u32 kSegOdds = W * 32, kWordsPerThread = W / kSieveThreads;
    const u32 tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const u32 n_med = min(n_primes, kNumMedium);
    // 1. primes 3..31: each thread writes whole words (pattern << offset).
    {
        u32 pat[kNumPattern], off[kNumPattern], step[kNumPattern], qs[kNumPattern];
#pragma unroll
        for (u32 k = 0; k < kNumPattern; ++k) {
            const u32 q = t.sp[k];
            qs[k] = q;
            u32 pm = 0;
            for (u32 b = 0; b < 32; b += q) pm |= 1u << b;
            pat[k] = pm;
            const u32 j0 = first_odd_multiple(v0, q, t.rcp[k]);
            int o = (int)j0 - (int)((32u * tid) % q);   // word w = tid first
            if (o < 0) o += (int)q;
            off[k] = (u32)o;
            step[k] = (32u * kSieveThreads) % q;
        }
        for (u32 w = tid; w < W; w += kSieveThreads) {
            u32 word = 0;
#pragma unroll
            for (u32 k = 0; k < kNumPattern; ++k) {
                word |= pat[k] << off[k];
                int o = (int)off[k] - (int)step[k];
                if (o < 0) o += (int)qs[k];
                off[k] = (u32)o;
            }
            sh.bits[w] = word;
        }
    }
    if (tid >= kNumPattern && tid < n_med)
        sh.med_start[tid] = (u32)min(first_strike(v0, t.sp[tid], t.rcp[tid]), (u64)kSegOdds);
    __syncthreads();
    // the pattern struck 3..31 themselves when they lie in this segment
    if (v0 <= 31 && tid < kNumPattern) {
        const u32 q = t.sp[tid];
        if (q >= v0) {
            const u32 i = (u32)((q - v0) >> 1);
            if (i < len) atomicAnd(&sh.bits[i >> 5], ~(1u << (i & 31)));
        }
    }
    // 2. primes 37..1021: the lanes of a warp share each prime, every eighth
    // prime a warp (all threads on each prime leaves most of them without a
    // multiple from q = 256 on, in a segment of 65,536: 2^28 integers at 10^12
    // took 219 us, now 175).
    for (u32 k = kNumPattern + warp; k < n_med; k += kSieveThreads / 32) {
        const u32 q = t.sp[k];
        for (u32 i = sh.med_start[k] + lane * q; i < len; i += 32 * q)
            atomicOr(&sh.bits[i >> 5], 1u << (i & 31));
    }
    // 3. primes 1031..65521: one thread per prime.
    // (the next prime's loads are in flight while this one strikes)
    u32 q = 0;
    u64 rcp = 0;
    if (kNumMedium + tid < n_primes) {
        q = t.sp[kNumMedium + tid];
        rcp = t.rcp[kNumMedium + tid];
    }
    for (u32 k = kNumMedium + tid; k < n_primes; k += kSieveThreads) {
        const u32 next = min(k + kSieveThreads, n_primes - 1);
        const u32 q_next = t.sp[next];
        const u64 rcp_next = t.rcp[next];
        const u64 j = first_strike(v0, q, rcp);
        for (u64 i = j; i < len; i += q) atomicOr(&sh.bits[(u32)i >> 5], 1u << ((u32)i & 31));
        q = q_next;
        rcp = rcp_next;
    }
    __syncthreads();

    // 4. survivors: contiguous words per thread, block scan, one global atomic.
    const u32 w0 = tid * kWordsPerThread;
    u32 mine = 0;
#pragma unroll
    for (u32 k = 0; k < kWordsPerThread; ++k) {
        const u32 w = w0 + k;
        u32 x = ~sh.bits[w];
        const u32 first = w * 32;
        if (first >= len) x = 0;
        else if (len - first < 32) x &= (1u << (len - first)) - 1u;
        mine += __popc(x);
    }
    u32 incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const u32 y = __shfl_up_sync(FULL, incl, o);
        if (lane >= (u32)o) incl += y;
    }
    if (lane == 31) sh.warp_sum[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        u32 ws = lane < kSieveThreads / 32 ? sh.warp_sum[lane] : 0;
        u32 wincl = ws;
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            const u32 y = __shfl_up_sync(FULL, wincl, o);
            if (lane >= (u32)o) wincl += y;
        }
        if (lane < kSieveThreads / 32) sh.warp_sum[lane] = wincl - ws;   // exclusive
        if (lane == kSieveThreads / 32 - 1) sh.block_base = atomicAdd(&ctr->survivors, (unsigned long long)wincl);
    }
    __syncthreads();
    const u64 base = sh.block_base;
    u32 rank = sh.warp_sum[warp] + (incl - mine);
    for (u32 k = 0; k < kWordsPerThread; ++k) {
        const u32 w = w0 + k;
        u32 x = ~sh.bits[w];
        const u32 first = w * 32;
        if (first >= len) x = 0;
        else if (len - first < 32) x &= (1u << (len - first)) - 1u;
        sh.before[w] = (unsigned short)rank;
        while (x) {
            const u32 b = __ffs(x) - 1;
            x &= x - 1;
            const u64 pos = base + rank;
            if (pos < o.cap) {
                o.surv[pos] = v0 + 2ull * (first + b);
                if (o.item) o.item[pos] = item;
                if (o.split) o.split[pos] = 0;
            }
            ++rank;
        }
    }
    if (base + rank > o.cap) atomicOr(&ctr->status, kStatusSurvivorOverflow);
    if (o.split && n_split > kSplitSmall) {
        // 5. the split primes l | v - 1: the bitmap walked once more, from the
        // first v == 1 (mod l), a warp's lanes sharing each l below 1024 (the
        // first three classes), one thread each of the others.  A survivor keeps one
        // l of each size class (a second one of a class, 4% of them, overwrites
        // the first).  This costs 1/l visits an odd number, about a tenth of
        // trying the primes on each entry (k_split).
        for (u32 k = kSplitSmall + tid; k < n_split; k += kSieveThreads) {
            const u32 q = t.sp[kSplitBase + k];
            u32 r = (u32)(v0 - __umul64hi(v0, t.rcp[kSplitBase + k]) * q);
            if (r >= q) r -= q;
            const u32 d = r <= 1 ? 1 - r : q + 1 - r;              // 2 j == 1 - v0 (mod q)
            sh.split_start[k] = (unsigned short)((d & 1u) ? (d + q) >> 1 : d >> 1);
        }
        __syncthreads();
        unsigned short* out = reinterpret_cast<unsigned short*>(o.split + base);
        const u32 room = base < o.cap ? (u32)min(o.cap - base, (u64)~0u) : 0u;
        auto visit = [&](u32 i, u32 c, u32 k) {
            const u32 w = ~sh.bits[i >> 5] << (31 - (i & 31));     // bit i on top
            if ((int)w < 0) {
                const u32 r = sh.before[i >> 5] + __popc(w) - 1;
                if (r < room) out[4 * r + c] = (unsigned short)(k + 1);
            }
        };
        const u32 n_shared = min(n_split, kSplitShared);
        for (u32 k = kSplitSmall + warp; k < n_shared; k += kSieveThreads / 32) {
            const u32 q = t.sp[kSplitBase + k], c = split_class(k);
#pragma unroll 4
            for (u32 i = sh.split_start[k] + lane * q; i < len; i += 32 * q) visit(i, c, k);
        }
        for (u32 k = kSplitShared + tid; k < n_split; k += kSieveThreads) {
            const u32 q = t.sp[kSplitBase + k];
#pragma unroll 4
            for (u32 i = sh.split_start[k]; i < len; i += q) visit(i, kSplitClasses - 1, k);
        }
    }
    __syncthreads();
}
static_assert(offsetof(Entry, k) % 8 == 0, "k_dlog reads the classes' indices as one word");
static_assert(kSplitClasses == 4 && split_class(kSplitShared - 1) == 2 && split_class(kSplitShared) == 3, "a survivor's split primes fill one 64-bit word");

template <u32 W>
__global__ void __launch_bounds__(kSieveThreads) k_sieve(SieveArgs a, SieveTables t, SurvOut o, Counters* ctr) {
    constexpr u32 kSegOdds = W * 32;
    __shared__ SieveShared<W> sh;
    if (blockIdx.x == 0 && threadIdx.x == 0 && a.include_two) emit_two(a.item, o, ctr);
    for (u64 seg = blockIdx.x; seg * kSegOdds < a.n_odds; seg += gridDim.x) {
        const u64 base = seg * kSegOdds;
        sieve_segment(sh, a.lo_odd + 2 * base, (u32)min((u64)kSegOdds, a.n_odds - base), a.n_primes, a.n_split, a.item, t, o,
                      ctr);
    }
}

// The same over a wave of runs (ranges of possibly different items), read
// from device memory so that a captured graph can be replayed per wave.
template <u32 W>
__global__ void __launch_bounds__(kSieveThreads) k_sieve_wave(const WaveDesc* w, SieveTables t, SurvOut o,
                                                              Counters* ctr) {
    constexpr u32 kSegOdds = W * 32;
    __shared__ SieveShared<W> sh;
    const u32 n_runs = w->n_runs;
    const u64 total = w->total_segs;
    if (blockIdx.x == 0 && threadIdx.x == 0)
        for (u32 r = 0; r < n_runs; ++r)
            if (w->runs[r].include_two) emit_two(w->runs[r].item, o, ctr);
    for (u64 seg = blockIdx.x; seg < total; seg += gridDim.x) {
        u32 lo = 0, hi = n_runs;                        // last run with seg_begin <= seg
        while (hi - lo > 1) {
            const u32 mid = (lo + hi) >> 1;
            if (w->runs[mid].seg_begin <= seg) lo = mid;
            else hi = mid;
        }
        const SieveRun& run = w->runs[lo];
        const u64 base = (seg - run.seg_begin) * kSegOdds;
        if (base >= run.n_odds) continue;               // (a run with no odd numbers)
        sieve_segment(sh, run.lo_odd + 2 * base, (u32)min((u64)kSegOdds, run.n_odds - base), run.n_primes, run.n_split,
                      run.item, t, o, ctr);
    }
}

// ------------------------------------------------------------ the fields --

// Two exact arithmetics behind one interface: FP64 (p < 2^49, the FP64 pipe)
// and 64-bit Montgomery (p < 2^62, the integer pipe).  V is the value type;
// key() gives the canonical integer (the table key) of a canonical value;
// eq(a, c) compares a product (or one()) with a canonical value c without
// leaving the field's representation.

// a^e two bits at a time (a product for every two squarings, chosen from 1, a,
// a^2, a^3 without a branch).
template <class F>
__device__ __forceinline__ typename F::V pow_window(const F& f, typename F::V a, u64 e) {
    typedef typename F::V V;
    const V one = f.one();
    if (e == 0) return one;
    const V a2 = f.mul(a, a), a3 = f.mul(a2, a);
    int k = (63 - __clzll((long long)e)) & ~1;
    const u32 top = (u32)(e >> k) & 3u;
    V x = top == 1 ? a : top == 2 ? a2 : a3;
    for (k -= 2; k >= 0; k -= 2) {
        const u32 dgt = (u32)(e >> k) & 3u;
        const V lo = dgt & 1u ? a : one, hi = dgt & 1u ? a3 : a2;
        x = f.mul(x, x);
        x = f.mul(x, x);
        x = f.mul(x, dgt & 2u ? hi : lo);
    }
    return x;
}

struct FieldF {
    typedef double V;
    Fp64 f;
    __device__ __forceinline__ void init(u64 p) { f.init(p); }
    __device__ __forceinline__ V mul(V a, V b) const { return f.mul(a, b); }
    __device__ __forceinline__ V canon(V a) const { return f.canon(a); }          // units: (-p, p) -> [0, p)
    __device__ __forceinline__ u64 key(V c) const { return f.bits(c); }
    // the low word of a unit's canonical integer (|a| < p, a != 0): 2^52 is added to a or to a + p in one step
    __device__ __forceinline__ u32 key32(V a) const {
        const double c = 4503599627370496.0;
        return (u32)__double2loint(__dadd_rn(a, a < 0.0 ? __dadd_rn(c, f.p) : c));
    }
    __device__ __forceinline__ u64 residue(V a) const { return f.residue(a); }   // any lazy value
    __device__ __forceinline__ V from_u64(u64 x) const { return (double)x; }
    __device__ __forceinline__ V one() const { return 1.0; }
    __device__ __forceinline__ double reciprocal() const { return f.pinv; }
    __device__ __forceinline__ V dbl(V a) const { return __dadd_rn(a, a); }      // (-p, p) -> (-2p, 2p)
    __device__ __forceinline__ V pow(V b, u64 e) const { return f.pow(b, e); }
    __device__ __forceinline__ bool eq(V a, V c) const { return a == c || a == c - f.p; }   // a in (-p, p)

    // Powers of a small base s (|s| p <= 2^50), from the top bit down: x <- x^2 s^bit
    // as (x s) x, where x s is exact (below 2^53), so a bit costs one product more
    // than a squaring's six instead of six.  The quotient of (x s) x by p is below
    // 0.43 * 2^50 and its estimate off by at most 1/2 + 2^-52 of that, so with
    // |x| <= 0.66 p, |x'| <= p (1/2 + 0.43 * 2^-2) <= 0.61 p: the values stay small
    // (the first one, s itself, is below p, and its square below 3/4 p, then
    // 0.65 p).  About 10 issue slots a bit against 16 for square-and-multiply.
    __device__ __forceinline__ bool small(double s) const { return s != 0.0 && fabs(s) * f.p <= 1125899906842624.0 && fabs(s) < f.p; }
    // (A small s has no bits in its low word: the factor s^bit is one select.)
    __device__ __forceinline__ static double factor(bool bit, int s_hi) { return __hiloint2double(bit ? s_hi : 0x3FF00000, 0); }
    __device__ __forceinline__ V pow_small(double s, u64 e) const {
        if (e == 0) return 1.0;
        const int lead = __clzll((long long)e), hi = __double2hiint(s);
        double x = s;
        e <<= lead;
        for (int k = 63 - lead; k > 0; --k) {
            e <<= 1;
            const bool bit = (long long)e < 0;
            x = f.mul(__dmul_rn(x, factor(bit, hi)), x);
        }
        return x;
    }
    // b^e and t^e (t = -c) for e > 0.
    __device__ __forceinline__ void powers(const DevItem& it, u64 e, V& w, V& u) const {
        const double bs = it.b_small, ts = it.t_small;
        if (small(bs) && small(ts)) {
            const int lead = __clzll((long long)e), bh = __double2hiint(bs), th = __double2hiint(ts);
            w = bs;
            u = ts;
            e <<= lead;
            for (int k = 63 - lead; k > 0; --k) {
                e <<= 1;
                const bool bit = (long long)e < 0;
                w = f.mul(__dmul_rn(w, factor(bit, bh)), w);
                u = f.mul(__dmul_rn(u, factor(bit, th)), u);
            }
            return;
        }
        w = b_power(it, e);
        u = small(ts) ? pow_small(ts, e) : pow_window(*this, from_u64(f.pi - residue128(it.cabs_hi, it.cabs_lo, it.c_neg, f.pi)), e);
    }
    __device__ __forceinline__ V b_power(const DevItem& it, u64 e) const {
        return small(it.b_small) ? pow_small(it.b_small, e)
                                 : pow_window(*this, from_u64(residue128(it.babs_hi, it.babs_lo, it.b_neg, f.pi)), e);
    }
};

struct FieldM {
    typedef u64 V;
    Mont M;
    u64 rr;
    __device__ __forceinline__ void init(u64 p) {
        M.init(p);
        rr = M.r2();
    }
    __device__ __forceinline__ V mul(V a, V b) const { return M.mul(a, b); }
    __device__ __forceinline__ V canon(V a) const { return M.norm(a); }
    __device__ __forceinline__ u64 key(V c) const { return c; }
    __device__ __forceinline__ u32 key32(V a) const { return (u32)M.norm(a); }
    __device__ __forceinline__ u64 residue(V a) const { return M.from_mont(a); }
    __device__ __forceinline__ V from_u64(u64 x) const { return M.to_mont(x, rr); }
    __device__ __forceinline__ V one() const { return M.one; }
    __device__ __forceinline__ double reciprocal() const { return 0.0; }
    __device__ __forceinline__ V dbl(V a) const { return M.dbl(a); }
    __device__ __forceinline__ V pow(V b, u64 e) const { return M.pow(b, e); }
    __device__ __forceinline__ bool eq(V a, V c) const { return a == c || a == c + M.p; }   // a in [0, 2p)
    __device__ __forceinline__ void powers(const DevItem& it, u64 e, V& w, V& u) const {
        w = b_power(it, e);
        u = pow_window(*this, from_u64(M.p - residue128(it.cabs_hi, it.cabs_lo, it.c_neg, M.p)), e);
    }
    __device__ __forceinline__ V b_power(const DevItem& it, u64 e) const {
        return pow_window(*this, from_u64(residue128(it.babs_hi, it.babs_lo, it.b_neg, M.p)), e);
    }
};

// --------------------------------------------------------------- the prep --

// log2 of the fingerprint-table words (the BSGS) a prime with m baby steps gets: at least m * 256 / fill
// words (fill 1..256; 0 counts as 256) and at least 32, at most 2^(tbits-1).
__device__ __forceinline__ u32 fq_words_log(u32 m, u32 fill, u32 tbits) {
    const u32 f = fill - 1u < 256u ? fill : 256u;
    const u32 keys = max(m, 2u) * 256u;                // m <= 4096: fits 32 bits
    u32 t = 32u - __clz(max(m, 2u) - 1);               // 2^t >= m; 2^t f >= 256 m needs at most 8 more
    while ((f << t) < keys) ++t;                       // no division: f << t <= 2^28
    return min(tbits - 1, max(5u, t));
}


// p < 1000: the reference's direct BSGS over n in [0, m*m), m = ceil(sqrt(min(p, N1)))
// (Math.hpp:488-542), which yields the smallest such n; a walk gives the same n.
__device__ __noinline__ void small_prime(u64 p, u64 b_mod, u64 t, const DevItem& it, const PrepArgs& a, Counters* ctr) {
    const i64 lim = ((i64)p > it.N1_raw) ? it.N1_raw : (i64)p;
    if (lim <= 0) return;
    const u64 m = isqrt_ceil_dev((u64)lim);
    const u64 mm = m * m;
    u64 v = 1 % p;
    for (u64 n = 0; n < mm; ++n) {
        if (v == t) {
            emit_relation(p, n, 0, it.item_index, a.rel, a.rel_cap, ctr);
            return;
        }
        v = (v * b_mod) % p;
    }
}

// Strong probable-prime test to base 2 in field F (square-and-double).
template <class F>
__device__ __forceinline__ bool sprp2_f(const F& f, u64 p) {
    const u64 pm1 = p - 1;
    const int s = __ffsll((long long)pm1) - 1;
    const u64 d = pm1 >> s;
    int k = 63 - __clzll((long long)d);
    typename F::V x = f.dbl(f.one());               // 2 (top bit of d)
    for (--k; k >= 0; --k) {
        x = f.mul(x, x);
        if ((d >> k) & 1) x = f.dbl(x);
    }
    u64 y = f.residue(x);
    if (y == 1 || y == pm1) return true;
    for (int r = 1; r < s; ++r) {
        x = f.mul(x, x);
        y = f.residue(x);
        if (y == pm1) return true;
        if (y == 1) return false;
    }
    return false;
}

// Residues of b and -c for the survivor p, and the cases that never reach
// the field arithmetic: p | b (Math.hpp:383-385, 496-503), p < 1000
// (Math.hpp:488-542), p | c or no candidate n (Math.hpp:386-396).
// Returns true when p continues to the main path.
__device__ __forceinline__ bool prep_special(u64 p, const DevItem& it, const PrepArgs& a, Counters* ctr, u64& b_mod,
                                             u64& t) {
    b_mod = residue128(it.babs_hi, it.babs_lo, it.b_neg, p);
    const u64 c_mod = residue128(it.cabs_hi, it.cabs_lo, it.c_neg, p);
    t = c_mod == 0 ? 0 : p - c_mod;                     // -c mod p
    if (b_mod == 0) {
        if (t == 0) emit_relation(p, (u64)it.N0_raw, 1, it.item_index, a.rel, a.rel_cap, ctr);
        return false;
    }
    if (p < 1000) {
        small_prime(p, b_mod, t, it, a, ctr);
        return false;
    }
    return t != 0 && it.has_work;
}

// Quadratic-character prefilter (the reference's Jacobi filter, Gpu.hpp:
// 247-263, restated): b^n == t (mod p) forces (b/p)^n == (t/p).  With every
// in-class n == n_start (mod cm): for even cm the parity of n is fixed, so
// (b/p)^(n_start mod 2) must equal (t/p); for odd cm, (b/p) = 1 forces
// (t/p) = 1.  True when p can be dropped: a prime p then has no in-class
// solution, and a composite p never gives a relation.  Costs two Jacobi
// symbols of 32-bit numbers, before any modular exponentiation.
__device__ __forceinline__ bool qr_reject(u64 p, const DevItem& it) {
    if (!it.qr_on) return false;
    int jb = 0, jt = 0;
#pragma unroll 1
    for (int i = 0; i < 2; ++i) {                      // (one copy of the code)
        jb = jt;
        jt = jacobi_small(p, it.qr_neg[i], it.qr_k[i], it.qr_o[i], it.qr_rcp[i]);
    }
    if (jb == 0 || jt == 0) return false;              // p shares a factor with b or c: the exact path decides
    if ((it.cm & 1) == 0) return (it.n_start & 1) ? jb != jt : jt != 1;
    return jb == 1 && jt != 1;
}

// e = (p - 1) / g exactly, g | p - 1.
__device__ __forceinline__ u64 exact_quotient(u64 pm1, u32 g) {
    const int tz = __ffs(g) - 1;
    return (pm1 >> tz) * (0 - Mont::neg_inverse((u64)(g >> tz)));
}

// gcd(Q, p - 1): the power of two by counting zeros, the odd parts by the
// binary algorithm (no divisions).
__device__ __forceinline__ u32 gcd_Q(const DevItem& it, u64 pm1) {
    const u64 qh = __umul64hi(pm1, it.Q_rcp);
    u32 rem = (u32)(pm1 - qh * it.Q);
    if (rem >= it.Q) rem -= it.Q;
    if (rem == 0) return it.Q;
    const int zq = __ffs((int)it.Q) - 1, zr = __ffs((int)rem) - 1;
    u32 x = it.Q >> zq, y = rem >> zr;
    while (x != y) {
        const u32 d = x > y ? x - y : y - x;
        y = min(x, y);
        x = d >> (__ffs((int)d) - 1);
    }
    return x << min(zq, zr);
}

// Stage 2: with g = gcd(Q, p - 1) and e = (p - 1) / g, w = b^e and u = t^e
// are g-th roots of unity and b^n == t forces w^n == u, i.e. n == r (mod d),
// d = ord(w) -- or there is no solution.  Returns 0 (no solution), 1 (d, r
// found within `walk` steps) or 2 (longer: deferred, with the residues of w
// and u in w_out, u_out for stage 2b).  This is the primality screen too: a
// composite p has w^g != 1 but for the rare pseudoprimes to base b, which the
// order stage drops.
//
// The orders and logarithms are found S at a time: with w^(S k) (k = 1,
// 2, ..) compared with w^i and u w^i, i < S, the largest match i gives the
// smallest exponent S k - i.  (S = 8 takes as many instructions and 16 more
// registers, a block less per SM: 2% of the prep.)
//
// Against a base-2 strong test of every survivor, the two powers by squaring
// from the low bit and a walk one step at a time, with 5 .. 19 in Q: k_prep on
// 2^27 integers at 10^12 0.90 -> 0.55 ms (and k_dlog, which took 5 .. 19 over,
// 0.21 -> 0.28).
template <class F>
__device__ __forceinline__ int power_split(const F& f, u64 p, const DevItem& it, u32 walk, u32& d, u32& r, u64& w_out,
                                           u64& u_out) {
    typedef typename F::V V;
    constexpr u32 S = 4;
    const u64 pm1 = p - 1;
    const u32 g = gcd_Q(it, pm1);
    V w, u;
    f.powers(it, exact_quotient(pm1, g), w, u);
    V wi[S], ui[S];                                    // w^i, u w^i (canonical)
    wi[0] = f.canon(f.one());
    ui[0] = f.canon(u);
    V x = w, y = f.mul(u, w);
#pragma unroll
    for (u32 i = 1; i < S; ++i) {
        wi[i] = f.canon(x);
        ui[i] = f.canon(y);
        x = f.mul(x, w);
        y = f.mul(y, w);
    }
    const V step = x;                                  // w^S
    const u32 lim = min(g, walk);
    u32 log = ui[0] == wi[0] ? 0 : ~0u, ord = ~0u;
    for (u32 k = S; k < lim + S && ord == ~0u; k += S) {
        const V c = f.canon(x);
        x = f.mul(x, step);
        u32 mu = 0, mw = 0;                            // the largest i + 1 that matches
#pragma unroll
        for (u32 i = 0; i < S; ++i) {
            if (ui[i] == c) mu = i + 1;
            if (wi[i] == c) mw = i + 1;
        }
        if (mu && log == ~0u) log = k + 1 - mu;
        if (mw) ord = k + 1 - mw;
    }
    if (ord <= lim) {
        d = ord;
        r = log;
        return log < ord ? 1 : 0;
    }
    if (lim == g) return 0;                            // w^g != 1: p is not prime
    w_out = f.residue(w);
    u_out = f.residue(u);
    return 2;
}

// Stage 2b: the same split for long orders, one prime power of g at a time,
// from stage 2's w and u (residues): w_l = w^(g/l^c), u_l = u^(g/l^c) in the
// l^c-th roots of unity, a walk of at most l^c steps each, combined by the
// Chinese remainder theorem.
template <class F>
__device__ bool power_split_pp(const F& f, u64 p, u64 w_res, u64 u_res, const DevItem& it, u32& d, u32& r) {
    typedef typename F::V V;
    const u32 g = gcd_Q(it, p - 1);
    const V w = f.from_u64(w_res), u = f.from_u64(u_res);
    d = 1;
    r = 0;
    for (u32 i = 0; i < it.qf_n; ++i) {
        const u32 l = it.qf_l[i];
        if (g % l) continue;
        u32 lc = l;
        while (g % (lc * l) == 0) lc *= l;
        const u32 k = g / lc;
        const V wl = f.pow(w, k), uc = f.canon(f.pow(u, k)), one = f.one();
        V x = one;
        bool found = false;
        u32 xr = 0, dl = 0;
        for (u32 y = 0; y < lc; ++y) {
            if (!found && f.eq(x, uc)) {
                xr = y;
                found = true;
            }
            x = f.mul(x, wl);
            if (f.eq(x, one)) {
                dl = y + 1;
                break;
            }
        }
        if (!found || dl == 0) return false;               // (dl == 0: p is not prime)
        // r' == r (mod d), r' == xr (mod dl); d, dl coprime
        u32 step = 0;                                      // d * dl <= g <= Q <= 2^28
        while ((r + d * step) % dl != xr) ++step;
        r += d * step;
        d *= dl;
    }
    return true;
}

// a^-1 mod m for gcd(a, m) = 1, 0 < a < m < 2^13: extended Euclid with the
// quotients by single-precision division, off by one at most and set right.  (At
// most 18 steps: the remainders fall as fast as Fibonacci numbers.)
__device__ __forceinline__ u32 inv_mod_small(u32 a, u32 m) {
    int r0 = (int)m, r1 = (int)a, s0 = 0, s1 = 1;
    for (int step = 0; step < 20 && r1 > 0; ++step) {
        int q = (int)__fdividef((float)r0, (float)r1);
        int r2 = r0 - q * r1;
        if (r2 < 0) {
            --q;
            r2 += r1;
        } else if (r2 >= r1) {
            ++q;
            r2 -= r1;
        }
        const int s2 = s0 - q * s1;
        r0 = r1;
        r1 = r2;
        s0 = s1;
        s1 = s2;
    }
    const int x = s0 % (int)m;
    return (u32)(x < 0 ? x + (int)m : x);
}

// a / m and a % m for a < 2^24, 0 < m < 2^13 and a quotient below 2^23, by single-precision
// division: its error of 2 units in the last place is 1 at most there, so the quotient is
// off by one at most, and set right.
__device__ __forceinline__ u32 div_small(u32 a, u32 m, u32& rem) {
    int q = (int)__fdividef((float)a, (float)m), r = (int)a - q * (int)m;
    if (r < 0) {
        --q;
        r += (int)m;
    } else if (r >= (int)m) {
        ++q;
        r -= (int)m;
    }
    rem = (u32)r;
    return (u32)q;
}
__device__ __forceinline__ u32 mod_small24(u32 a, u32 m) {
    u32 r;
    div_small(a, m, r);
    return r;
}

// Stage 3: n = n_start + cm*k (in class) with n == r (mod d): the candidates
// n_first + j*L, j < jcount.  False when there is none.
__device__ __forceinline__ bool combine_class(u64 p, const DevItem& it, u32 d, u32 r, Entry& e) {
    // the smallest k0 >= 0 with n_start + cm*k0 == r (mod d): k0*cmd == want
    // (mod d) is solvable iff h = gcd(cmd, d) divides want, and then its
    // solutions are k0 + per*i with per = d/h, k0 = (want/h)(cmd/h)^-1 mod per
    u32 per, k0;                                       // period of k
    u64 jcount;
    if (it.Q <= 4096) {
        // (every value here is below 2^24, where a quotient by single precision costs
        // half of an integer division: the prep kernels -0.8%)
        const u32 cmd = mod_small24(it.cmQ, d);        // d | Q
        const u32 want = mod_small24(r + d - mod_small24(it.nsQ, d), d);
        u32 h = d, x = cmd, rem;                       // h = gcd(cmd, d), gcd(0, d) = d
        for (int step = 0; step < 20 && x != 0; ++step) {
            const u32 y = mod_small24(h, x);
            h = x;
            x = y;
        }
        const u32 wh = div_small(want, h, rem);
        if (rem) return false;
        per = div_small(d, h, rem);
        const u32 ch = mod_small24(div_small(cmd, h, rem), per);
        k0 = per == 1 ? 0u : mod_small24(wh * inv_mod_small(ch, per), per);
        if (k0 >= it.K) return false;
        const u32 left = (u32)it.K - k0;               // K <= 10^7: above 2^23 only when undivided
        jcount = per == 1 ? left : div_small(left + per - 1, per, rem);
    } else {
        const u32 cmd = it.cmQ % d;
        const u32 want = (r + d - it.nsQ % d) % d;
        const u32 h = gcd32(cmd, d);
        if (want % h) return false;
        per = d / h;
        k0 = (u32)((u64)(want / h) * inv_mod32((cmd / h) % per, per) % per);
        if (k0 >= it.K) return false;
        jcount = ((u32)it.K - k0 + per - 1) / per;
    }
    if (jcount > p) jcount = p;                        // ord(B) < p (Math.hpp:398-400)
    e.jcount = (u32)jcount;
    e.L = it.cm * per;
    e.n_first = it.n_start + it.cm * k0;
    return true;
}

// ---- the split by larger primes ----
//
// A prime l | p - 1 outside Q splits an entry's candidates the same way: with
// w = b^((p-1)/l) and u = t^((p-1)/l), b^n == t forces w^n == u, so n is known
// mod l (or, when b is an l-th power residue, t has to be one too).  One
// discrete logarithm in a group of l elements divides the candidates by l and
// the baby and giant steps by sqrt(l); a prime has an l of 5 .. 4259 with
// chance 1/(l-1), 1.7 in all.  Those of 5 .. 19 are tried on each entry, finding
// the others costs a second walk of the sieve's bitmap (sieve_segment); a
// logarithm costs about 700 lane instructions for the powers and 1.2 l for the
// walk (k_dlog), so only entries with enough candidates have it.
// On 2^27 integers of b = 10, c = 111 at 10^12 (1.36 M entries), against the split
// by lcm(mod, 232792560) alone: BSGS steps 2.10e9 -> 0.87e9 and, with the later
// changes of the step itself, k_bsgs 3.44 -> 1.28 ms, for 0.13 ms of sieve, 0.28 of
// k_dlog and 0.17 of k_setup (which took the set-up over from k_prep and solves
// the smallest entries).

// How many primes of the table an entry with J candidates is split by.  (The
// optimum is flat: splitting from 512 candidates on, by all primes from 4096,
// costs an item of K = 10^4 4% and one of K = 10^6 nothing; stopping at half as
// many primes for each size loses as much.)
__host__ __device__ constexpr u32 split_limit(u32 J) {
    return J < 1536 ? 0u : J < 4096 ? 32u : J < 16384 ? 100u : J < 65536 ? 300u : kSplitPrimes;
}
u32 split_primes_for(u64 K) { return split_limit((u32)min(K, (u64)~0u)); }

// Queues the split events of the warp's entries (idx, lanes with ok) in slots
// S0 .. S1 - 1: k[slot] is the index + 1 of the entry's l, 0 for none.  One
// atomic per list and warp; a full list drops the event.
template <u32 S0, u32 S1>
__device__ __forceinline__ void queue_events(bool ok, u64 idx, u64 p, const u32 (&k)[kSplitSlots], const PrepArgs& a,
                                             Counters* ctr) {
    const u32 lane = threadIdx.x & 31, below = (1u << lane) - 1;
    const u32 field = a.two_fields && p >= kFp64Limit ? kSplitSizes : 0u;
    const u32 second = __ballot_sync(FULL, field != 0), mine_field = field ? second : ~second;
    u32 pos[kSplitSlots], n[kSplitLists] = {}, mine = 0;
#pragma unroll
    for (u32 s = S0; s < S1; ++s) {
        const u32 bal = __ballot_sync(FULL, ok && k[s] != 0), c = slot_list(s);
        pos[s] = (field ? n[c + kSplitSizes] : n[c]) + __popc(bal & mine_field & below);
        n[c] += __popc(bal & ~second);
        n[c + kSplitSizes] += __popc(bal & second);
    }
#pragma unroll
    for (u32 c = 0; c < kSplitLists; ++c)
        if (lane == c) mine = n[c];
    u64 at0 = 0;
    if (mine) at0 = atomicAdd(&ctr->events[lane], (unsigned long long)mine);
#pragma unroll
    for (u32 s = S0; s < S1; ++s) {
        const u64 at = __shfl_sync(FULL, at0, slot_list(s) + field) + pos[s];
        if (!ok) continue;
        const bool in = k[s] != 0 && at < (s < kSplitClasses ? a.ev_cap : a.ev_small);
        const u32 list = field ? a.ev_at[slot_list(s) + kSplitSizes] : a.ev_at[slot_list(s)];
        if (in) a.events[list + (u32)at] = SplitEvent{(u32)idx, (k[s] - 1) << 16 | s};
        a.ent[idx].ev[s] = in ? kEvQueued | kEvUnknown : 0u;
        if (s < kSplitClasses) a.ent[idx].k[s] = (unsigned short)(k[s] - 1);
    }
}

// Whether l divides x, l^-1 mod 2^64 and floor((2^64 - 1) / l) folded at compile time.
template <u32 L>
__device__ __forceinline__ bool divides(u64 x) {
    constexpr u64 i0 = (3ull * L) ^ 2, i1 = i0 * (2 - L * i0), i2 = i1 * (2 - L * i1), i3 = i2 * (2 - L * i2),
                  inv = i3 * (2 - L * i3);
    static_assert(inv * L == 1, "inverse");
    return x * inv <= ~0ull / L;
}

// Two 16-bit halves of a compared with those of b as half-precision numbers
// (two FMA-pipe compares in one instruction): 0xFFFF where equal.
__device__ __forceinline__ u32 equal_halves(u32 a, u32 b) {
    return __heq2_mask(*reinterpret_cast<const __half2*>(&a), *reinterpret_cast<const __half2*>(&b));
}

// The largest i < M with t * B^i == g as base + M - i, ~0 when there is none.
template <u32 M, class F>
__device__ __forceinline__ u32 lane_match(const F& f, typename F::V t, typename F::V B, typename F::V g, u32 base) {
    const typename F::V c = f.canon(g);
    typename F::V x = t;
    u32 best = ~0u;
#pragma unroll 4
    for (u32 i = 0; i < M; ++i) {
        if (f.canon(x) == c) best = base + M - i;
        x = f.mul(x, B);
    }
    return best;
}

// The smallest j in [1, J) with G0 * B^j == t, by one lane (~0: none): M baby
// steps t * B^i, giant steps G0 * B^(M g) each compared with all of them, a
// match resolved exactly after the loop.  t canonical.  The lanes leave the loop
// at different times and are brought together by __syncwarp before the
// resolution; without it each group that leaves runs the resolution on its own
// (k_dlog: 0.58 ms instead of 0.29 on 2^27 integers at 10^12).
//   16 baby steps (small J): their low words in registers, a compare each; the
//     walk ends at the first match (a wrong one, 2^-28, goes on from there).
//   32 baby steps: the low 14 bits and bit 15 of their low words, two to a
//     register, as finite half-precision numbers, so that a giant step costs 16
//     FMA-pipe compares and 8 ORs where 32 integer compares would take twice the
//     ALU's time.  One giant step in 1,000 matches by chance: the walk goes on,
//     keeping the last two matches (a third one has the first resolved at once).
template <class F>
__device__ __noinline__ u32 lane_rest(F f, typename F::V t, typename F::V B, typename F::V S, typename F::V g,
                                      u32 base, u32 M, u32 J) {
    for (; base + 1 < J; base += M) {                  // every giant step resolved in full
        const typename F::V c = f.canon(g);
        typename F::V x = t;
        u32 best = ~0u;
        for (u32 i = 0; i < M; ++i) {
            if (f.canon(x) == c) best = base + M - i;
            x = f.mul(x, B);
        }
        if (best != ~0u) return best < J ? best : ~0u;
        g = f.mul(g, S);
    }
    return ~0u;
}

template <class F>
__device__ __forceinline__ u32 lane_solve16(const F& f, typename F::V t, typename F::V G0, typename F::V B, u32 J) {
    typedef typename F::V V;
    constexpr u32 M = 16;
    const u32 together = __activemask();
    u32 key[M];
    V x = t;
#pragma unroll
    for (u32 i = 0; i < M; ++i) {
        key[i] = f.key32(x);
        x = f.mul(x, B);
    }
    V S = f.mul(B, B);
#pragma unroll
    for (u32 i = 2; i < M; i <<= 1) S = f.mul(S, S);
    V g = f.mul(G0, S);
    u32 base = 0;
    bool hit = false;
    for (; base + 1 < J; base += M) {                  // g = G0 B^(base + M): j in (base, base + M]
        const u32 k = f.key32(g);
        const V next = f.mul(g, S);
#pragma unroll
        for (u32 i = 0; i < M; ++i) hit |= key[i] == k;
        if (hit) break;
        g = next;
    }
    __syncwarp(together);
    u32 best = ~0u;
    if (hit) {
        best = lane_match<M>(f, t, B, g, base);
        if (best == ~0u) best = lane_rest(f, t, B, S, f.mul(g, S), base + M, M, J);
    }
    return best < J ? best : ~0u;
}

template <class F>
__device__ __forceinline__ u32 lane_solve32(const F& f, typename F::V t, typename F::V G0, typename F::V B, u32 J) {
    typedef typename F::V V;
    constexpr u32 M = 32;
    const u32 together = __activemask();
    u32 key[M / 2];
    V x = t;
#pragma unroll
    for (u32 i = 0; i < M; i += 2) {
        const u32 k0 = f.key32(x);
        x = f.mul(x, B);
        const u32 k1 = f.key32(x);
        x = f.mul(x, B);
        key[i / 2] = __byte_perm(k0, k1, 0x5410) & 0xBFFFBFFFu;
    }
    V S = f.mul(B, B);
#pragma unroll
    for (u32 i = 2; i < M; i <<= 1) S = f.mul(S, S);
    V g = f.mul(G0, S), g0 = g, g1 = g;
    u32 n = 0, b0 = 0, b1 = 0, best = ~0u;
    for (u32 base = 0; base + 1 < J; base += M) {      // g = G0 B^(base + M): j in (base, base + M]
        const u32 k = f.key32(g), rep = __byte_perm(k, k, 0x1010) & 0xBFFFBFFFu;
        const V next = f.mul(g, S);
        u32 z = 0;
#pragma unroll
        for (u32 i = 0; i < M / 2; ++i) z |= equal_halves(key[i], rep);
        if (z) {
            if (n == 2) {
                best = lane_match<32>(f, t, B, g0, b0);
                if (best != ~0u) break;
                g0 = g1;
                b0 = b1;
                n = 1;
            }
            if (n == 0) {
                g0 = g;
                b0 = base;
            } else {
                g1 = g;
                b1 = base;
            }
            ++n;
        }
        g = next;
    }
    __syncwarp(together);
    if (best == ~0u && n > 0) best = lane_match<32>(f, t, B, g0, b0);
    if (best == ~0u && n > 1) best = lane_match<32>(f, t, B, g1, b1);
    return best < J ? best : ~0u;
}

// What stage 1 tests of primality itself: a base-2 strong test where the powers
// of b prove nothing (|b| <= 1), all 12 bases when the caller asks for them.
template <class F>
__device__ __forceinline__ bool stage1_in(u64 p, const DevItem& it, const PrepArgs& a) {
    if (it.strong) {
        F f;
        f.init(p);
        if (!sprp2_f(f, p)) return false;
    }
    return !a.full_mr || is_prime64(p);
}

constexpr u32 kPrepThreads = 256;
constexpr u32 kWalk = 48;                              // stage-2 walk before deferring

// Warp-aggregated push onto a shared-memory queue.
__device__ __forceinline__ u32 queue_slot(u32* count, bool want) {
    const u32 bal = __ballot_sync(FULL, want);
    if (!bal) return 0;
    const u32 lane = threadIdx.x & 31;
    const int leader = __ffs(bal) - 1;
    u32 base = 0;
    if ((int)lane == leader) base = atomicAdd(count, __popc(bal));
    base = __shfl_sync(FULL, base, leader);
    return base + __popc(bal & ((1u << lane) - 1));
}

// The prep: one persistent kernel without block barriers.  Every warp claims
// 32 survivors at a time and carries them through the stages on its own,
// with three warp-private queues in shared memory between the stages
// (survivors that passed stage 1; primes with their (d, r) for stage 3;
// primes deferred to stage 2b).  A queue is drained whenever it holds 32
// entries, so every stage runs with full warps, and a warp never waits for
// another; the partial queues are drained at the end.  A queue never holds
// more than 63 entries: a stage pushes at most 32 into a queue that held
// fewer than 32.
constexpr u32 kPrepWarps = kPrepThreads / 32;

struct PrepQueues {
    u64 p1[64];
    u32 i1[64], s1[64];                            // item, survivor index (surv_split's)
    u64 p2[64];
    u32 i2[64], s2[64], d2[64], r2[64];
    u64 pd[64];
    u64 wd[64], ud[64];                            // stage 2's w and u of a deferred prime
    u32 id[64], sd[64];
};

// Appends the lanes with want to a warp queue of n entries (n warp-uniform).
__device__ __forceinline__ void qpush(bool want, u32& n, u32* slot_out) {
    const u32 lane = threadIdx.x & 31;
    const u32 bal = __ballot_sync(FULL, want);
    *slot_out = n + __popc(bal & ((1u << lane) - 1));
    n += __popc(bal);
}

template <class F>
__device__ __forceinline__ int split_in(const DevItem& it, u64 p, u32& d, u32& r, u64& w, u64& u) {
    F f;
    f.init(p);
    return power_split(f, p, it, kWalk, d, r, w, u);
}

// The rare paths are out of line: with everything inline the kernel's warps, each
// at another stage, waited for instruction fetches more than for anything else
// but their own arithmetic (2.25 stalls an issue).
__device__ __noinline__ int split_in_m(const DevItem& it, u64 p, u32& d, u32& r, u64& w, u64& u) {
    return split_in<FieldM>(it, p, d, r, w, u);
}
__device__ __noinline__ bool split_pp_in(const DevItem& it, u64 p, u64 w, u64 u, u32& d, u32& r) {
    if (p < kFp64Limit) {
        FieldF f;
        f.init(p);
        return power_split_pp(f, p, w, u, it, d, r);
    }
    FieldM f;
    f.init(p);
    return power_split_pp(f, p, w, u, it, d, r);
}
__device__ __noinline__ bool stage1(u64 p, const DevItem& it, const PrepArgs& a) {
    return p < kFp64Limit ? stage1_in<FieldF>(p, it, a) : stage1_in<FieldM>(p, it, a);
}

__global__ void __launch_bounds__(kPrepThreads, 4) k_prep(PrepArgs a, Counters* ctr) {
    __shared__ PrepQueues qs[kPrepWarps];
    PrepQueues& Q = qs[threadIdx.x >> 5];
    const u32 lane = threadIdx.x & 31;
    const u64 n_surv = min((u64)*(volatile unsigned long long*)&ctr->survivors, a.surv_cap);
    u32 n1 = 0, n2 = 0, nd = 0;                          // queue lengths (warp-uniform)
    bool inputs = true;
    for (;;) {
        if (n2 >= 32 || (!inputs && n1 == 0 && nd == 0 && n2 > 0)) {
            // stage 3: class combination, and the entries' way out
            const u32 cnt = min(n2, 32u);
            Entry e;
            bool ok = false;
            u32 sv = 0;
            if (lane < cnt) {
                const u32 k = n2 - cnt + lane;
                e.p = Q.p2[k];
                e.item = Q.i2[k];
                sv = Q.s2[k];
                ok = combine_class(e.p, a.items[e.item], Q.d2[k], Q.r2[k], e);
            }
            n2 -= cnt;
            __syncwarp();
            const u32 bal = __ballot_sync(FULL, ok);
            if (bal) {
                u64 base = 0;
                if (lane == 0) base = atomicAdd(&ctr->entries, (unsigned long long)__popc(bal));
                const u64 slot = __shfl_sync(FULL, base, 0) + __popc(bal & ((1u << lane) - 1));
                if (ok && slot >= a.ent_cap) {
                    atomicOr(&ctr->status, kStatusEntryOverflow);
                    ok = false;
                }
                if (ok) {
                    Entry& d = a.ent[slot];
                    d.p = e.p; d.n_first = e.n_first; d.L = e.L; d.jcount = e.jcount; d.item = e.item;
                }
                // the primes l | p - 1 to split by: 5 .. 19 here, the others from the sieve
                u32 k[kSplitSlots] = {};
                if (ok && a.items[e.item].split_more) {
                    const u32 limit = split_limit(e.jcount), modulus = a.items[e.item].Q;
                    const u64 found = a.surv_split ? a.surv_split[sv] : 0;
#pragma unroll
                    for (u32 c = 0; c < kSplitClasses; ++c) {
                        k[c] = (u32)(found >> (16 * c)) & 0xFFFFu;
                        if (k[c] > limit) k[c] = 0;
                    }
                    if (limit) {
                        const u64 pm1 = e.p - 1;
                        if (divides<5>(pm1)) k[kSplitClasses] = 1;
                        if (divides<7>(pm1)) k[kSplitClasses + 1] = 2;
                        if (divides<11>(pm1)) k[kSplitClasses + 2] = 3;
                        if (divides<13>(pm1)) k[kSplitClasses + 3] = 4;
                        if (divides<17>(pm1)) k[kSplitClasses + 4] = 5;
                        if (divides<19>(pm1)) k[kSplitClasses + 5] = 6;
                    }
#pragma unroll
                    for (u32 s = 0; s < kSplitSlots; ++s)
                        if (k[s] && modulus % a.tables.sp[kSplitBase + k[s] - 1] == 0) k[s] = 0;   // Q splits by it
                }
                queue_events<0, kSplitSlots>(ok, slot, ok ? e.p : 0, k, a, ctr);
            }
            continue;
        }
        if (nd >= 32 || (!inputs && n1 == 0 && nd > 0)) {
            // stage 2b: long orders, one prime power at a time
            const u32 cnt = min(nd, 32u);
            bool ok = false;
            u32 d = 1, r = 0, item = 0, sv = 0;
            u64 p = 0;
            if (lane < cnt) {
                const u32 k = nd - cnt + lane;
                p = Q.pd[k];
                item = Q.id[k];
                sv = Q.sd[k];
                const DevItem& it = a.items[item];
                const u64 w = Q.wd[k], u = Q.ud[k];
                ok = split_pp_in(it, p, w, u, d, r);
            }
            nd -= cnt;
            __syncwarp();
            u32 s2;
            qpush(ok, n2, &s2);
            if (ok) {
                Q.p2[s2] = p;
                Q.i2[s2] = item;
                Q.s2[s2] = sv;
                Q.d2[s2] = d;
                Q.r2[s2] = r;
            }
            __syncwarp();
            continue;
        }
        if (n1 >= 32 || (!inputs && n1 > 0)) {
            // stage 2: power-residue split with a short walk
            const u32 cnt = min(n1, 32u);
            int res = 0;
            u32 d = 1, r = 0, item = 0, sv = 0;
            u64 p = 0, w = 0, u = 0;
            if (lane < cnt) {
                const u32 k = n1 - cnt + lane;
                p = Q.p1[k];
                item = Q.i1[k];
                sv = Q.s1[k];
                const DevItem& it = a.items[item];
                res = p < kFp64Limit ? split_in<FieldF>(it, p, d, r, w, u) : split_in_m(it, p, d, r, w, u);
            }
            n1 -= cnt;
            __syncwarp();
            u32 s2, sd;
            qpush(res == 1, n2, &s2);
            qpush(res == 2, nd, &sd);
            if (res == 1) {
                Q.p2[s2] = p;
                Q.i2[s2] = item;
                Q.s2[s2] = sv;
                Q.d2[s2] = d;
                Q.r2[s2] = r;
            } else if (res == 2) {
                Q.pd[sd] = p;
                Q.wd[sd] = w;
                Q.ud[sd] = u;
                Q.id[sd] = item;
                Q.sd[sd] = sv;
            }
            __syncwarp();
            continue;
        }
        if (!inputs) break;
        // stage 1: claim 32 survivors; special cases and the quadratic-character prefilter
        u64 first = 0;
        if (lane == 0) first = atomicAdd(&ctr->prep_next, 32ull);
        first = __shfl_sync(FULL, first, 0);
        if (first >= n_surv) {
            inputs = false;
            continue;
        }
        const u64 k = first + lane;
        bool keep = false;
        u64 p = 0;
        u32 item = a.item0;
        if (k < n_surv) {
            p = a.surv[k];
            if (a.surv_item) item = a.surv_item[k];
            u64 bm, t;
            if (prep_special(p, a.items[item], a, ctr, bm, t) && !qr_reject(p, a.items[item]))
                // (below prime_below the sieve removed every composite)
                keep = p < a.prime_below || !(a.items[item].strong || a.full_mr) || stage1(p, a.items[item], a);
        }
        u32 s1;
        qpush(keep, n1, &s1);
        if (keep) {
            Q.p1[s1] = p;
            Q.i1[s1] = item;
            Q.s1[s1] = (u32)k;
        }
        __syncwarp();
    }
}

// ---- k_split: the primes l | p - 1 of entries whose primes did not come from the sieve ----

// A warp takes up to 32 entries; the lanes hold the table's primes (kSplitGroups
// each, in registers for the whole launch) and try them against one entry after
// another: four integer instructions a prime and no loads.
__global__ void __launch_bounds__(256, 2) k_split(PrepArgs a, Counters* ctr) {
    const u32 lane = threadIdx.x & 31;
    const u64 n_ent = min((u64)*(volatile unsigned long long*)&ctr->entries, a.ent_cap);
    const u64 warps = (u64)gridDim.x * (blockDim.x >> 5);
    u32 inv_lo[kSplitGroups], inv_hi[kSplitGroups], lim[kSplitGroups];
#pragma unroll
    for (u32 g = 0; g < kSplitGroups; ++g) {
        const u64 inv = a.tables.inv[kSplitBase + kSplitSmall + 32 * g + lane];
        inv_lo[g] = (u32)inv;
        inv_hi[g] = (u32)(inv >> 32);
        lim[g] = (u32)(a.tables.rcp[kSplitBase + kSplitSmall + 32 * g + lane] >> 32);
    }
    // few entries: fewer than 32 a warp, so that every warp has some
    const u32 per = (u32)min((u64)32, max((u64)1, n_ent / warps));
    for (u64 first = ((u64)(threadIdx.x >> 5) * gridDim.x + blockIdx.x) * per; first < n_ent; first += warps * per) {
        const u64 idx = first + lane;
        const bool ok = lane < per && idx < n_ent;
        u32 lo = 0, hi = 0, limit = 0;
        if (ok) {
            const Entry& e = a.ent[idx];
            const u64 pm1 = e.p - 1;
            lo = (u32)pm1;
            hi = (u32)(pm1 >> 32);
            limit = a.items[e.item].split_more ? split_limit(e.jcount) : 0u;
        }
        u32 found[kSplitSlots] = {};
        for (u32 i = 0; i < per; ++i) {
            const u32 n = __shfl_sync(FULL, limit, i);
            const u32 xl = __shfl_sync(FULL, lo, i), xh = __shfl_sync(FULL, hi, i);
            u32 div = 0;
#pragma unroll
            for (u32 g = 0; g < kSplitGroups; ++g) {
                if (kSplitSmall + 32 * g >= n) break;
                // y = x l^-1 mod 2^64 is x / l when l | x, below 2^62 / l, and at least
                // 2^64 / l when not (l y = x + i 2^64, i >= 1): the high words decide
                if (__umulhi(xl, inv_lo[g]) + xl * inv_hi[g] + xh * inv_lo[g] < lim[g]) div |= 1u << g;
            }
            u32 bal = __ballot_sync(FULL, div != 0);
            while (bal) {                                      // one prime of each lane
                const u32 src = (u32)__ffs((int)bal) - 1;
                bal &= bal - 1;
                const u32 k = kSplitSmall + 32 * ((u32)__ffs((int)__shfl_sync(FULL, div, src)) - 1) + src;
#pragma unroll
                for (u32 c = 0; c < kSplitClasses; ++c)
                    if (lane == i && split_class(k) == c) found[c] = k + 1;
            }
        }
        queue_events<0, kSplitClasses>(ok, idx, ok ? a.ent[idx].p : 0, found, a, ctr);
    }
}

// ---- k_dlog: the split events ----

// n mod l for an entry's p: dlog of u = t^((p-1)/l) to w = b^((p-1)/l), or
// kEvUnknown / kEvReject.  together: the lanes that call this; they are brought
// together after the powers, whose lengths differ.
template <class F>
__device__ __forceinline__ u32 split_solve(u64 p, const DevItem& it, u32 l, u64 l_inv, bool large, u32 together) {
    typedef typename F::V V;
    F f;
    f.init(p);
    const u64 e = (p - 1) * l_inv;                     // (p - 1) / l, if l divides p - 1 at all
    V w, u;
    f.powers(it, e, w, u);
    __syncwarp(together);
    const V one = f.one();
    const bool w1 = f.eq(w, one), u1 = f.eq(u, one);
    u32 x = w1 ? (u1 ? kEvUnknown : kEvReject) : 0u;
    if (!w1 && !u1) {
        x = large ? lane_solve32(f, f.canon(u), one, w, l) : lane_solve16(f, f.canon(u), one, w, l);
        if (x == ~0u) x = kEvUnknown;                  // p is not prime; the order stage drops it
    }
    return __umul64hi(e, l) == 0 ? x : kEvUnknown;
}

__device__ __noinline__ u32 split_solve_m(u64 p, const DevItem& it, u32 l, u64 l_inv, bool large, u32 together) {
    return split_solve<FieldM>(p, it, l, l_inv, large, together);   // out of line: the FP64 path sets the registers
}

// One lane per event, a list after the other, the longest walks first.
__global__ void __launch_bounds__(256, 4) k_dlog(PrepArgs a, Counters* ctr) {
    const u32 lane = threadIdx.x & 31;
    constexpr u32 order[kSplitLists] = {8, 3, 7, 2, 6, 1, 5, 0, 9, 4};
    static_assert(kSplitSizes == 5, "the lists' order");
    u64 count[kSplitLists], total = 0;
#pragma unroll
    for (u32 i = 0; i < kSplitLists; ++i) {
        count[i] = min((u64)*(volatile unsigned long long*)&ctr->events[order[i]],
                       (u64)(order[i] % kSplitSizes == kSplitClasses ? a.ev_small : a.ev_cap));
        total += (count[i] + 31) / 32;
    }
    // the first unit of a warp is fixed, block by block, so that the longest walks
    // start on all SMs (claimed like the others, they went to the SMs whose blocks
    // started first: 2^20 integers at 10^9, 64 us instead of 27)
    const u64 warps = (u64)gridDim.x * (blockDim.x >> 5);
    for (u64 unit = (u64)(threadIdx.x >> 5) * gridDim.x + blockIdx.x; unit < total;) {
        u64 k = unit, idx = 0;
        if (lane == 0) unit = warps + atomicAdd(&ctr->dlog_next, 1ull);
        unit = __shfl_sync(FULL, unit, 0);
        bool placed = false, live = false, large = false;
#pragma unroll
        for (u32 i = 0; i < kSplitLists; ++i) {
            const u64 units = (count[i] + 31) / 32;
            if (!placed && k < units) {
                idx = a.ev_at[order[i]] + k * 32 + lane;
                live = k * 32 + lane < count[i];
                large = i < 4;                         // l > 256
                placed = true;
            }
            k -= units;
        }
        const u32 together = __ballot_sync(FULL, live);
        if (live) {
            const SplitEvent s = a.events[idx];
            Entry& e = a.ent[s.entry];
            const u64 p = e.p;
            u32 slots = 0;                             // the slots with an l (their loads go together)
#pragma unroll
            for (u32 i = 0; i < kSplitSlots; ++i)
                if (e.ev[i] != 0) slots |= 1u << i;
            const u64 classes = *reinterpret_cast<const u64*>(e.k);
            const u32 together_f = __ballot_sync(together, p < kFp64Limit);
            const DevItem& it = a.items[e.item];
            const u32 li = s.which >> 16, l = a.tables.sp[kSplitBase + li];
            const u64 l_inv = a.tables.inv[kSplitBase + li], rcp = a.tables.rcp[kSplitBase + li];
            u32 x = p < kFp64Limit ? split_solve<FieldF>(p, it, l, l_inv, large, together_f)
                                   : split_solve_m(p, it, l, l_inv, large, together & ~together_f);
            __syncwarp(together);
            // n_first + j L == x (mod l) for j, and the inverse that k_setup combines
            // it with, that of the earlier slots' primes' product M: from one
            // inverse, of L M.  L is prime to l unless the class modulus holds l
            const u32 slot = s.which & 0xFFFFu;
            const u32 Lm = mod_small(e.L, l, rcp), nm = mod_small(e.n_first, l, rcp);
            u32 Mm = 1, inv = 0;
            for (u32 before = slots & ((1u << slot) - 1); before; before &= before - 1) {
                const u32 i = (u32)__ffs((int)before) - 1;
                const u32 k = i < kSplitClasses ? (u32)(classes >> (16 * i)) & 0xFFFFu : slot_small(i);
                Mm = Mm * a.tables.sp[kSplitBase + k] % l;
            }
            if (x < kEvReject) {
                if (Lm != 0) {
                    const u32 lm = inv_mod_small(Lm * Mm % l, l);
                    x = (x >= nm ? x - nm : x + l - nm) * (lm * Mm % l) % l;
                    inv = lm * Lm % l;
                } else {
                    x = x == nm ? kEvUnknown : kEvReject;
                }
            }
            e.ev[slot] = kEvQueued | inv << kEvInvShift | x;
        }
        __syncwarp();
    }
}

// ---- k_setup: the solve's set-up, and the solve of primes with few candidates ----

// Applies what k_dlog found to the entry's candidates; false when none is
// left.  ev: the entry's slots in memory, each lane taking its own next one (an
// entry has 1.7 on average, so a loop over the slots would mostly idle).  The
// residues are combined one after the other with the inverses that k_dlog left;
// these are those of all earlier slots' primes, so after a slot that taught
// nothing (1 in l^2) they are computed here.
__device__ __forceinline__ bool apply_events(Entry& e, const Entry& mem, const SieveTables& t) {
    u32 mask = 0;
#pragma unroll
    for (u32 i = 0; i < kSplitSlots; ++i)
        if (e.ev[i] != 0) mask |= 1u << i;
    u64 j = 0, M = 1;                                  // the j left: == j (mod M)
    bool whole = true;                                 // M is the product of all earlier slots' primes
    while (mask) {
        const u32 slot = (u32)__ffs((int)mask) - 1, v = mem.ev[slot], x = v & kEvValue;
        mask &= mask - 1;
        if (x == kEvReject) return false;
        if (x == kEvUnknown) {
            whole = false;
            continue;
        }
        const u32 k = kSplitBase + (slot < kSplitClasses ? mem.k[slot] : slot_small(slot)), l = t.sp[k];
        const u64 rcp = t.rcp[k];
        const u32 jm = mod_small(j, l, rcp);
        const u32 diff = x >= jm ? x - jm : x + l - jm;
        if (M >= e.jcount) {                           // one candidate at most: check it
            if (diff) return false;
            whole = false;
        } else {
            const u32 inv = whole ? v >> kEvInvShift & kEvValue : inv_mod_small(mod_small(M, l, rcp), l);
            j += M * mod_small((u64)diff * inv, l, rcp);
            M *= l;
        }
        if (j >= e.jcount) return false;
    }
    e.n_first += j * e.L;
    const u32 left = e.jcount - (u32)j;                // >= 1
    e.jcount = M >= left ? 1 : (left + (u32)M - 1) / (u32)M;
    if (e.jcount > 1) e.L *= M;
    return true;
}

// The set-up of one entry: false when it needs no solve (its only candidate
// decided, or n_first already a solution).
template <class F>
__device__ __forceinline__ bool setup_entry(Entry& e, const DevItem& it, const PrepArgs& a, Counters* ctr, bool small) {
    typedef typename F::V V;
    F f;
    f.init(e.p);
    e.t = e.p - residue128(it.cabs_hi, it.cabs_lo, it.c_neg, e.p);
    const V gv = f.b_power(it, e.n_first);
    e.G0 = f.residue(gv);
    if (e.G0 == e.t) {                                 // j = 0
        emit_relation(e.p, e.n_first, 0, e.item, a.rel, a.rel_cap, ctr);
        return false;
    }
    if (e.jcount <= 1) return false;
    const V Bv = f.b_power(it, e.L);
    e.B = f.residue(Bv);
    // B = 1 or -1: G0 B^j takes G0 and -G0 only.  (Every prime of an item with |b| = 1 is
    // one; all its baby steps would share one or two words of the table, each walking
    // past all the earlier ones: 2^20 integers at 10^9 with b = -1, K = 10^7, took 26 ms.)
    if (e.B == 1 || e.B == e.p - 1) {
        if (e.B != 1 && e.G0 + e.t == e.p)             // j = 1
            emit_relation(e.p, e.n_first + e.L, 0, e.item, a.rel, a.rel_cap, ctr);
        return false;
    }
    if (small) return true;
    u32 m = (u32)isqrt_ceil_dev(e.jcount);
    if (it.baby_scale != 256) m = max(1u, (u32)(((u64)m * it.baby_scale + 255) >> 8));
    // a whole number of baby iterations (lanes x chains per prime): the last
    // iteration's lanes then all insert, and the extra baby steps save giant steps
    if (a.m_round > 1) m = (m + a.m_round - 1) / a.m_round * a.m_round;
    if (m > it.max_baby) m = it.max_baby;
    if (m > a.m_cap) m = a.m_cap;                      // never more than the launch's tables hold
    e.m = m;
    e.G = (e.jcount - 1 + m - 1) / m;                  // g = 1..G covers j in [1, G*m]
    e.tw = fq_words_log(m, a.fill, a.tbits);
    e.pinv = f.reciprocal();
    e.Bm = f.residue(f.pow(Bv, m));
    return true;
}

template <class F>
__device__ __forceinline__ u32 lane_solve_entry(const Entry& e, bool large) {
    F f;
    f.init(e.p);
    return large ? lane_solve32(f, f.from_u64(e.t), f.from_u64(e.G0), f.from_u64(e.B), e.jcount)
                 : lane_solve16(f, f.from_u64(e.t), f.from_u64(e.G0), f.from_u64(e.B), e.jcount);
}

__device__ __noinline__ u32 lane_solve_entry_m(const Entry& e, bool large) { return lane_solve_entry<FieldM>(e, large); }

// Entries with at most kLaneMax candidates are solved here, one lane each:
// 1.2 lane instructions a candidate against about 290 warp instructions of
// per-prime set-up in k_bsgs and its partly filled iterations.  A warp's lanes walk together, so the entries
// wait in queues by size (a factor of two each) and arithmetic until one holds 32.
constexpr u32 kLaneSizes = 6, kLaneQueues = 2 * kLaneSizes, kLaneMax = 2048, kLaneMin = 64;   // J <= 64, 128, .. 2048
constexpr u32 kLaneFew = 1u << 16, kLaneMaxFew = 256;            // (2^19 integers at 10^9: 248 us with 2048, 231 with 256)

constexpr u32 kSetupWarps = 4;
__global__ void __launch_bounds__(kSetupWarps * 32, 7) k_setup(PrepArgs a, Counters* ctr) {
    __shared__ u32 queues[kSetupWarps][kLaneQueues][64];
    u32(&Q)[kLaneQueues][64] = queues[threadIdx.x >> 5];
    const u32 lane = threadIdx.x & 31, below = (1u << lane) - 1;
    const u64 n_ent = min((u64)*(volatile unsigned long long*)&ctr->entries, a.ent_cap);
    // few entries: a lane's walk is then what the launch waits for
    const u32 lane_max = n_ent < kLaneFew ? kLaneMaxFew : kLaneMax;
    u32 n[kLaneQueues] = {};                           // queue lengths (warp-uniform)
    bool inputs = true;
    for (;;) {
        // a queue that holds 32 is drained; once the inputs are used up, the
        // last 32 entries of all the queues together, the longest first
        u32 q = kLaneQueues, idx = ~0u;
#pragma unroll
        for (u32 k = 0; k < kLaneQueues; ++k)
            if (n[k] >= 32) q = k;
        if (q < kLaneQueues) {
#pragma unroll
            for (u32 k = 0; k < kLaneQueues; ++k)
                if (k == q) {
                    n[k] -= 32;
                    idx = Q[k][n[k] + lane];
                }
        } else if (!inputs) {
            u32 taken = 0;
#pragma unroll
            for (u32 k = kLaneQueues; k-- > 0;) {
                const u32 cnt = min(n[k], 32 - taken);
                if (lane >= taken && lane - taken < cnt) idx = Q[k][n[k] - cnt + lane - taken];
                n[k] -= cnt;
                taken += cnt;
            }
            if (taken == 0) break;
        }
        if (q < kLaneQueues || !inputs) {
            // the two smallest sizes with 16 baby steps
            const bool large = q < kLaneQueues ? q % kLaneSizes >= 2 : lane_max > kLaneMaxFew;
            if (idx != ~0u) {
                const Entry& e = a.ent[idx];
                const u32 j = e.p < kFp64Limit ? lane_solve_entry<FieldF>(e, large) : lane_solve_entry_m(e, large);
                if (j != ~0u) emit_relation(e.p, e.n_first + (u64)j * e.L, 0, e.item, a.rel, a.rel_cap, ctr);
            }
            __syncwarp();
            continue;
        }
        u64 first = 0;
        if (lane == 0) first = atomicAdd(&ctr->setup_next, 32ull);
        first = __shfl_sync(FULL, first, 0);
        if (first >= n_ent) {
            inputs = false;
            continue;
        }
        idx = (u32)first + lane;
        u32 cls = kLaneQueues + 1;                     // kLaneQueues: for k_bsgs
        // (the lanes leave apply_events at different times: together again for the powers)
        Entry e;
        bool ok = false;
        if (first + lane < n_ent) {
            e = a.ent[idx];
            ok = apply_events(e, a.ent[idx], a.tables);
        }
        __syncwarp();
        if (ok) {
            const DevItem& it = a.items[e.item];
            const bool small = e.jcount <= lane_max;
            if (e.p < kFp64Limit ? setup_entry<FieldF>(e, it, a, ctr, small)
                                 : setup_entry<FieldM>(e, it, a, ctr, small)) {
                Entry& d = a.ent[idx];
                d.t = e.t; d.G0 = e.G0; d.B = e.B; d.Bm = e.Bm; d.jcount = e.jcount; d.m = e.m;
                d.pinv = e.pinv; d.G = e.G; d.tw = e.tw;
                d.n_first = e.n_first; d.L = e.L;
                cls = kLaneQueues;
                if (small) {
                    cls = 0;
                    while (e.jcount > (kLaneMin << cls)) ++cls;
                    if (e.p >= kFp64Limit) cls += kLaneSizes;
                }
            }
        }
        __syncwarp();
#pragma unroll
        for (u32 k = 0; k < kLaneQueues; ++k) {
            const u32 bal = __ballot_sync(FULL, cls == k);
            if (cls == k) Q[k][n[k] + __popc(bal & below)] = idx;
            n[k] += __popc(bal);
        }
        const u32 bal = __ballot_sync(FULL, cls == kLaneQueues);
        if (bal) {
            u64 base = 0;
            if (lane == 0) base = atomicAdd(&ctr->big, (unsigned long long)__popc(bal));
            base = __shfl_sync(FULL, base, 0);
            if (cls == kLaneQueues) a.big[base + __popc(bal & below)] = idx;
        }
        __syncwarp();
    }
}

// --------------------------------------------------------------- the BSGS --
//
// One warp per prime.  The baby-step table holds a 16-bit fingerprint per
// slot (0 = empty; linear probing); a giant value whose fingerprint matches
// is resolved exactly by recomputing the baby steps, which is rare (true
// solutions, and fingerprint collisions at ~2^-15 per compare).

__device__ __forceinline__ void table_hash(u64 key, u32 tbits, u32& slot, u32& fp) {
    const u32 lo = (u32)key, hi = (u32)(key >> 32);
    const u32 x = (lo ^ (hi * 0x9E3779B1u)) * 0x85EBCA6Bu;
    slot = x >> (32 - tbits);
    fp = (x & 0xFFFFu) | 1u;
}

__device__ __forceinline__ void table_insert(unsigned short* tab, u32 mask, u32 tbits, u64 key) {
    u32 s, fp;
    table_hash(key, tbits, s, fp);
    while (atomicCAS(&tab[s], (unsigned short)0, (unsigned short)fp) != 0) s = (s + 1) & mask;
}

__device__ __forceinline__ bool table_maybe(const unsigned short* tab, u32 mask, u32 tbits, u64 key) {
    u32 s, fp;
    table_hash(key, tbits, s, fp);
    for (;;) {
        const u32 e = tab[s];
        if (e == fp) return true;
        if (e == 0) return false;
        s = (s + 1) & mask;
    }
}

// Smallest i in [lo, limit) with key(t * B^i) == key, or -1 (warp-cooperative;
// tbl = t * B^lane, B32 = B^32).
template <class F>
__device__ __noinline__ int find_baby_index(F f, typename F::V tbl, typename F::V B32, u32 lo, u32 limit, u64 key) {
    const u32 lane = threadIdx.x & 31;
    typename F::V v = tbl;
    for (u32 base = 0; base < limit; base += 32) {
        const u32 i = base + lane;
        const bool hit = i >= lo && i < limit && f.key(f.canon(v)) == key;
        const u32 bal = __ballot_sync(FULL, hit);
        if (bal) return (int)(base + __ffs(bal) - 1);
        v = f.mul(v, B32);
    }
    return -1;
}

// A solve's step counts for its caller: giant steps in the high 32 bits,
// baby steps in the low 32 (baby <= kMaxBaby, giant <= jcount <= 10^7).
__device__ __forceinline__ u64 pack_steps(u64 baby, u64 giant) { return (giant << 32) | baby; }

// Solves one entry with the 32 lanes of the calling warp; returns the
// smallest j (< jcount) or ~0ull.  Two interleaved chains per lane: baby
// indices i = l + 64k and l + 32 + 64k, giant steps g = 1 + l + 64k and
// 33 + l + 64k.
template <class F>
__device__ u64 solve_entry(const Solve& e, unsigned short* tab, u32 tbits, u64* steps_out) {
    typedef typename F::V V;
    const u32 lane = threadIdx.x & 31;
    F f;
    f.init(e.p);
    const u32 m = e.m;
    const u32 T = 1u << tbits, mask = T - 1;
    const V B = f.from_u64(e.B), Bm = f.from_u64(e.Bm), tv = f.from_u64(e.t), G0 = f.from_u64(e.G0);
    const u64 tkey = f.key(f.canon(tv));

    // lane powers by an inclusive scan: xb = B^(l+1), xg = Bm^(l+1)
    V xb = B, xg = Bm;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const V yb = __shfl_up_sync(FULL, xb, off), yg = __shfl_up_sync(FULL, xg, off);
        if (lane >= (u32)off) {
            xb = f.mul(xb, yb);
            xg = f.mul(xg, yg);
        }
    }
    const V B32 = __shfl_sync(FULL, xb, 31), Bm32 = __shfl_sync(FULL, xg, 31);
    V bl = __shfl_up_sync(FULL, xb, 1);
    if (lane == 0) bl = f.one();                       // B^l
    const V B64 = f.mul(B32, B32), Bm64 = f.mul(Bm32, Bm32);
    const V tbl = f.mul(tv, bl);                       // t B^l
    V baby0 = tbl, baby1 = f.mul(tbl, B32);
    V gi0 = f.mul(G0, xg), gi1 = f.mul(gi0, Bm32);

    uint4* t4 = reinterpret_cast<uint4*>(tab);
    for (u32 k = lane; k < T / 8; k += 32) t4[k] = make_uint4(0, 0, 0, 0);
    __syncwarp();

    // baby steps t*B^i, stopping at a cycle B^d == 1 (d < m)
    u32 cyc = 0;
    u64 steps = 0, baby_steps = 0;
    for (u32 base = 0; base < m; base += 64) {
        const u32 i0 = base + lane, i1 = base + 32 + lane;
        const u64 k0 = f.key(f.canon(baby0)), k1 = f.key(f.canon(baby1));
        const u32 b0 = __ballot_sync(FULL, i0 > 0 && i0 < m && k0 == tkey);
        const u32 b1 = __ballot_sync(FULL, i1 < m && k1 == tkey);
        u32 lim = m;
        if (b0 | b1) {
            cyc = b0 ? base + __ffs(b0) - 1 : base + 32 + __ffs(b1) - 1;
            lim = cyc;
        }
        if (i0 < lim) table_insert(tab, mask, tbits, k0);
        if (i1 < lim) table_insert(tab, mask, tbits, k1);
        steps += min(64u, lim - base);
        baby_steps += min(64u, lim - base);
        if (cyc) break;
        baby0 = f.mul(baby0, B64);
        baby1 = f.mul(baby1, B64);
    }
    __syncwarp();

    u64 best = ~0ull;
    if (cyc) {
        // ord(B) = cyc < m: the answer is the j in [1, cyc) with G0 == t*B^(cyc-j)
        // (j = 0 was ruled out by the prep); t*B^i, i < cyc, are distinct.
        const int i = find_baby_index(f, tbl, B32, 1, cyc, f.key(f.canon(G0)));
        if (i > 0) best = cyc - (u32)i;
    } else {
        const u64 G = (e.jcount - 1 + m - 1) / m;      // giant steps g = 1..G cover j in [1, G*m]
        for (u64 base = 0; base < G; base += 64) {
            const u64 g0 = base + 1 + lane, g1 = base + 33 + lane;
            const u64 k0 = f.key(f.canon(gi0)), k1 = f.key(f.canon(gi1));
            const bool h0 = g0 <= G && table_maybe(tab, mask, tbits, k0);
            const bool h1 = g1 <= G && table_maybe(tab, mask, tbits, k1);
            const u32 bal0 = __ballot_sync(FULL, h0), bal1 = __ballot_sync(FULL, h1);
            steps += min((u64)64, G - base);
            if (bal0 | bal1) {
                // candidates in increasing g: the first exact one is the smallest j
                u64 jb = ~0ull;
                for (int pass = 0; pass < 2 && jb == ~0ull; ++pass) {
                    u32 bal = pass == 0 ? bal0 : bal1;
                    while (bal && jb == ~0ull) {
                        const int src = __ffs(bal) - 1;
                        bal &= bal - 1;
                        const u64 kk = __shfl_sync(FULL, pass == 0 ? k0 : k1, src);
                        const u64 gg = base + (pass == 0 ? 1 : 33) + (u64)src;
                        const int i = find_baby_index(f, tbl, B32, 0, m, kk);
                        if (i >= 0) jb = gg * m - (u64)i;
                    }
                }
                if (jb != ~0ull) {
                    best = jb;
                    break;
                }
            }
            gi0 = f.mul(gi0, Bm64);
            gi1 = f.mul(gi1, Bm64);
        }
    }
    __syncwarp();
    if (steps_out) *steps_out = pack_steps(baby_steps, steps - baby_steps);
    return best < e.jcount ? best : ~0ull;
}

// ---- the FP64 solve (p < 2^49): the hot loop of the whole path ----
//
// Table: 2^tbits 32-bit slots per warp.  A key's home slot is the top tbits
// of a multiplicative hash h of the canonical value's two 32-bit halves; the
// slot word is (h & ~1) | 2 (never 0) plus bit 0, the overflow bit, set on a
// home slot when a key homed there had to move further (linear probing).  A
// probe therefore reads one slot: a match, an empty slot, or an occupied slot
// without the overflow bit all end it; only an overflowed home (rare at the
// load factors used) walks the chain, in a ballot-guarded slow path.  A match
// is resolved exactly by recomputation (ffind_baby): true solutions, and hash
// collisions at about 2^-20 per compare.

__device__ __forceinline__ u32 fhash(double v) {
    return (u32)(__double2loint(v) ^ __double2hiint(v)) * 0x9E3779B1u;
}

__device__ __forceinline__ u32 fword(u32 h) { return (h & ~3u) | 2u; }

__device__ __forceinline__ void ftable_insert(u32* tab, u32 mask, u32 shift, u32 h) {
    u32 s = h >> shift;
    const u32 w = fword(h);
    if (atomicCAS(&tab[s], 0u, w) == 0u) return;
    atomicOr(&tab[s], 1u);                         // a key homed here moves on
    do s = (s + 1) & mask;
    while (atomicCAS(&tab[s], 0u, w) != 0u);
}

// Continues a probe past an overflowed home slot s.
__device__ __forceinline__ bool ftable_walk(const u32* tab, u32 mask, u32 s, u32 w) {
    for (;;) {
        s = (s + 1) & mask;
        const u32 e = tab[s];
        if (e == 0u) return false;
        if ((e & ~1u) == w) return true;
    }
}

// Smallest i in [lo, limit) with t * B^i == v (canonical doubles compared
// exactly); -1 when there is none.  Warp-cooperative: tbl = t * B^lane.
__device__ __noinline__ int ffind_baby(Fp64 f, double tbl, double B32, u32 lo, u32 limit, double v) {
    const u32 lane = threadIdx.x & 31;
    double x = tbl;
    for (u32 base = 0; base < limit; base += 32) {
        const u32 i = base + lane;
        const bool hit = i >= lo && i < limit && f.canon(x) == v;
        const u32 bal = __ballot_sync(FULL, hit);
        if (bal) return (int)(base + __ffs(bal) - 1);
        x = f.mul(x, B32);
    }
    return -1;
}

// CH interleaved chains per lane: baby index i = lane + 32c + 32*CH*k,
// giant step g = 1 + lane + 32c + 32*CH*k.
template <int CH>
__device__ u64 solve_fp64(const Solve& e, u32* tab, u32 tbits, u64* steps_out) {
    const u32 lane = threadIdx.x & 31;
    Fp64 f;
    f.init(e.p);
    const u32 m = e.m;
    const u32 jc = (u32)e.jcount;                      // jcount <= 10^7
    // this prime's table: 2^tb slots for m baby steps (load <= ~1/5), at most the launch's
    tbits = min(tbits, max(6u, 32u - __clz(5 * m - 1)));
    const u32 mask = (1u << tbits) - 1, shift = 32 - tbits;
    const double B = (double)e.B, Bm = (double)e.Bm, tv = (double)e.t, G0 = (double)e.G0;

    double xb = B, xg = Bm;                            // B^(l+1), Bm^(l+1)
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const double yb = __shfl_up_sync(FULL, xb, off), yg = __shfl_up_sync(FULL, xg, off);
        if (lane >= (u32)off) {
            xb = f.mul(xb, yb);
            xg = f.mul(xg, yg);
        }
    }
    const double B32 = __shfl_sync(FULL, xb, 31), Bm32 = __shfl_sync(FULL, xg, 31);
    double bl = __shfl_up_sync(FULL, xb, 1);
    if (lane == 0) bl = 1.0;
    double Bstep = B32, Gstep = Bm32;                  // B^(32 CH), Bm^(32 CH)
#pragma unroll
    for (int c = 1; c < CH; c <<= 1) {
        Bstep = f.mul(Bstep, Bstep);
        Gstep = f.mul(Gstep, Gstep);
    }
    const double tbl = f.mul(tv, bl);
    double bx[CH], gx[CH];
    bx[0] = tbl;
    gx[0] = f.mul(G0, xg);
#pragma unroll
    for (int c = 1; c < CH; ++c) {
        bx[c] = f.mul(bx[c - 1], B32);
        gx[c] = f.mul(gx[c - 1], Bm32);
    }

    uint4* t4 = reinterpret_cast<uint4*>(tab);
    for (u32 k = lane; k <= mask / 4; k += 32) t4[k] = make_uint4(0, 0, 0, 0);
    __syncwarp();

    // baby steps, stopping at a cycle B^d == 1 (d < m)
    u32 cyc = 0, baby_done = m;
    for (u32 base = 0; base < m; base += 32 * CH) {
        double cv[CH];
        u32 cb = 0;
#pragma unroll
        for (int c = 0; c < CH; ++c) {
            cv[c] = f.canon(bx[c]);
            const u32 i = base + 32 * c + lane;
            const u32 bc = __ballot_sync(FULL, i > 0 && i < m && cv[c] == tv);
            if (bc && !cb) cb = base + 32 * c + __ffs(bc) - 1;
        }
        const u32 lim = cb ? cb : m;
#pragma unroll
        for (int c = 0; c < CH; ++c) {
            const u32 i = base + 32 * c + lane;
            if (i < lim) ftable_insert(tab, mask, shift, fhash(cv[c]));
        }
        if (cb) {
            cyc = cb;
            baby_done = cb;
            break;
        }
#pragma unroll
        for (int c = 0; c < CH; ++c) bx[c] = f.mul(bx[c], Bstep);
    }
    __syncwarp();

    u64 best = ~0ull;
    u32 giant_done = 0;
    if (cyc) {
        const int i = ffind_baby(f, tbl, B32, 1, cyc, G0);
        if (i > 0) best = cyc - (u32)i;
    } else {
        const u32 G = (jc - 1 + m - 1) / m;            // g = 1..G covers j in [1, G*m]
        giant_done = G;
        for (u32 base = 0; base < G; base += 32 * CH) {
            double cv[CH];
            u32 hit = 0;
#pragma unroll
            for (int c = 0; c < CH; ++c) {
                cv[c] = f.canon(gx[c]);
                const u32 h = fhash(cv[c]);
                const u32 s0 = h >> shift;
                const u32 w1 = (h & ~3u) | 3u;         // the slot word with the overflow bit forced
                const u32 e = tab[s0];
                bool m1 = (e | 1u) == w1;
                if (!m1 && (e & 1u)) m1 = ftable_walk(tab, mask, s0, w1 & ~1u);
                hit |= m1 ? (1u << c) : 0u;
            }
            if (__any_sync(FULL, hit)) {
                u32 bal[CH];
#pragma unroll
                for (int c = 0; c < CH; ++c)
                    bal[c] = __ballot_sync(FULL, ((hit >> c) & 1u) && base + 32 * c + lane + 1 <= G);
                // candidates in increasing g: the first exact one gives the smallest j
                u64 jb = ~0ull;
#pragma unroll
                for (int c = 0; c < CH; ++c) {
                    u32 bb = bal[c];
                    while (bb && jb == ~0ull) {
                        const int src = __ffs(bb) - 1;
                        bb &= bb - 1;
                        const double v = __shfl_sync(FULL, cv[c], src);
                        const u64 g = base + 32 * c + (u32)src + 1;
                        const int i = ffind_baby(f, tbl, B32, 0, m, v);
                        if (i >= 0) jb = g * m - (u64)i;
                    }
                }
                if (jb != ~0ull) {
                    best = jb;
                    giant_done = min(G, base + 32 * CH);
                    break;
                }
            }
#pragma unroll
            for (int c = 0; c < CH; ++c) gx[c] = f.mul(gx[c], Gstep);
        }
    }
    __syncwarp();
    if (steps_out) *steps_out = pack_steps(baby_done, giant_done);
    return best < e.jcount ? best : ~0ull;
}

// ---- the FP64 solve with a fingerprint table (the default) ----
//
// Table: 2^tw 64-bit words per warp, each holding up to four 16-bit halves
// filled in order (half k = bits 16k..16k+15): bit 15 of a half marks it
// used, bits 0..13 hold a 14-bit fingerprint of the key; bit 14 of half 0 is
// the word's overflow bit, set when a key homed at this word found it full
// and moved on (linear probing over words).  For m baby steps tw =
// ceil(log2(m * 256 / fill)), so a word holds at most fill/256 keys on average
// (fill 160: 0.6, and about 0.1% of the words overflow).
//
// The step is bound by instruction issue and the ALU pipe, with the FP64 pipe
// a third busy, so its work sits where there is room.  The hash is one FP64
// multiply-add of the canonical residue c (fq_hash): the low mantissa word of
// c k + 2^51, 32 mixed bits of the fixed-point product.  Its bits 3 .. tw + 2
// are the home word's byte offset as they stand and its bits 16 .. 29 the
// fingerprint.  The four halves of a word are compared with the fingerprint as
// half-precision numbers, two instructions of the FMA pipe: a used half is a
// negative finite number (bit 14 clear), so equality is that of the bits, but
// for fingerprint 0, -0, which an empty half also equals (one probe in 16,384).
// A home with its overflow bit set also counts as a candidate.  The next giant
// value is multiplied before the probe of the current one, so the multiply's
// latency overlaps the shared-memory load.  Candidates leave the hot loop: the
// lane walks the overflow chain, and a fingerprint found is resolved exactly by
// recomputation (ffind_last).
//
// Measured on 2^27 integers of b = 10, c = 111 at 10^12: 1.61 -> 1.32 ms (the
// hash, the half-precision compare and the cycle check left out: 1,358 -> 1,162 M
// warp instructions; the set-up from k_setup and the half-warp scan: 1,100 M).
// Per 32 steps a giant step is 27 instructions (9 FP64, 12 ALU), a baby step 36,
// and a prime costs 290 besides.
//
// A cycle B^d == 1 with d < m needs no care for the result: the baby steps then
// repeat, the table holds some keys several times, and the largest i of the
// smallest g still gives the smallest j = g m - i.  It costs a walk of about
// m / 4d words an insertion, so k_setup decides the entries with d <= 2 itself;
// larger orders as small as that are left to chance (p divides b^k - 1 for a k
// of at most d L).

constexpr u64 kQValid = 0x8000800080008000ull;
constexpr u32 kQOvf = 0x4000u;

__device__ __forceinline__ u32 fq_fingerprints(u32 h) {        // in both halves
    return (__byte_perm(h, h, 0x3232) & 0x3FFF3FFFu) | 0x80008000u;
}

__device__ __forceinline__ bool fq_word_has(u64 w, u32 pat) {
    const u32 lo = (u32)w & ~kQOvf, hi = (u32)(w >> 32);
    return (lo & 0xFFFFu) == pat || (lo >> 16) == pat || (hi & 0xFFFFu) == pat || (hi >> 16) == pat;
}

// One compare-and-swap per key (table kind 0).
__device__ __forceinline__ void fq_insert(unsigned long long* tab, u32 mask, u32 home, u32 pat) {
    volatile unsigned long long* vt = tab;
    u32 s = home;
    unsigned long long w = vt[s];
    for (;;) {
        if (w >> 63) {                               // full: move on (marking the home once)
            if (s == home && !(w & kQOvf)) atomicOr(&tab[home], (unsigned long long)kQOvf);
            s = (s + 1) & mask;
            w = vt[s];
            continue;
        }
        const u32 k = __popcll(w & kQValid);
        const unsigned long long nw = w | ((unsigned long long)pat << (16 * k));
        const unsigned long long old = atomicCAS(&tab[s], w, nw);
        if (old == w) return;
        w = old;
    }
}

// Whether the key (home, pat) is in the table: its home word, then the
// overflow chain up to the first word that is not full.
__device__ __forceinline__ bool fq_contains(const unsigned long long* tab, u32 mask, u32 home, u32 pat) {
    u64 w = tab[home];
    if (fq_word_has(w, pat)) return true;
    if (!(w & kQOvf)) return false;
    for (u32 s = (home + 1) & mask, n = 0; n <= mask; s = (s + 1) & mask, ++n) {
        w = tab[s];
        if (fq_word_has(w, pat)) return true;
        if (!(w >> 63)) return false;
    }
    return false;
}

// Table kind 3: the fingerprint words of kind 0 with a count byte per word
// (after the launch's words: one byte per eight of table).  A key claims the
// next half of its home word by one shared-memory atomic add on the word's count
// and writes its fingerprint with a plain 16-bit store (every claimed half is
// distinct).  A claim that finds the word full (count >= 4) is taken back at
// once, so a count rests at 4 at most and never passes 4 + 32 * CH in flight (a
// byte cannot wrap).  The rare keys whose home was full then walk on, word by
// word, in rounds of the whole warp, as in kind 0's walk; the overflow bits of
// their homes are set after every store of the call, so a store to half 0
// never clears one.  off: the word's byte offset.
__device__ __forceinline__ u32 fq_claim(unsigned char* cnt, u32 off) {
    const u32 sh = off & 24u;                          // 8 x (word mod 4)
    u32* c32 = reinterpret_cast<u32*>(cnt) + (off >> 5);
    return (atomicAdd(c32, 1u << sh) >> sh) & 0xFFu;
}
__device__ __forceinline__ void fq_unclaim(unsigned char* cnt, u32 off) {
    atomicSub(reinterpret_cast<u32*>(cnt) + (off >> 5), 1u << (off & 24u));
}

template <int CH>
__device__ __forceinline__ void fq_insert_count(unsigned char* tab, unsigned char* cnt, u32 mask8, u32 want,
                                                const u32 (&h)[CH]) {
    u32 k[CH], pend = 0;                               // bit c: chain c found its home full
#pragma unroll
    for (int c = 0; c < CH; ++c) k[c] = (want >> c) & 1u ? fq_claim(cnt, h[c] & mask8) : 0u;
#pragma unroll
    for (int c = 0; c < CH; ++c) {
        if (!((want >> c) & 1u)) continue;
        if (k[c] < 4u) *reinterpret_cast<unsigned short*>(tab + (h[c] & mask8) + 2 * k[c]) = (unsigned short)fq_fingerprints(h[c]);
        else pend |= 1u << c;
    }
    if (!__any_sync(FULL, pend)) return;
    const u32 ovf = pend;
    u32 s[CH];
#pragma unroll
    for (int c = 0; c < CH; ++c) {
        s[c] = h[c] & mask8;
        if ((pend >> c) & 1u) fq_unclaim(cnt, s[c]);
        s[c] = (s[c] + 8) & mask8;
    }
    while (__any_sync(FULL, pend)) {
#pragma unroll
        for (int c = 0; c < CH; ++c) k[c] = (pend >> c) & 1u ? fq_claim(cnt, s[c]) : 4u;
#pragma unroll
        for (int c = 0; c < CH; ++c) {
            if (!((pend >> c) & 1u)) continue;
            if (k[c] < 4u) {
                *reinterpret_cast<unsigned short*>(tab + s[c] + 2 * k[c]) = (unsigned short)fq_fingerprints(h[c]);
                pend &= ~(1u << c);
            } else {
                fq_unclaim(cnt, s[c]);
                s[c] = (s[c] + 8) & mask8;
            }
        }
    }
    __syncwarp();
#pragma unroll
    for (int c = 0; c < CH; ++c)
        if ((ovf >> c) & 1u) atomicOr(reinterpret_cast<u32*>(tab + (h[c] & mask8)), kQOvf);
}

// The largest i in [0, m) with t * B^i == v (canonical doubles compared
// exactly); -1 when there is none.  Warp-cooperative: tbl = t * B^lane.
__device__ __noinline__ int ffind_last(Fp64 f, double tbl, double B32, u32 m, double v) {
    const u32 lane = threadIdx.x & 31;
    double x = tbl;
    int last = -1;
    for (u32 base = 0; base < m; base += 32) {
        const u32 bal = __ballot_sync(FULL, base + lane < m && f.canon(x) == v);
        if (bal) last = (int)(base + 31 - __clz((int)bal));
        x = f.mul(x, B32);
    }
    return last;
}

// What the fingerprint-table solve needs of an entry, as k_setup left it.
struct SolveF {
    Fp64 f;                                            // p and 1/p
    double t, G0, B, Bm;
    u32 jcount, m, G, tw;
};
__device__ __forceinline__ SolveF solve_f(const Solve& e, u32 tbits, u32 fill) {
    SolveF s;
    s.f.init(e.p);
    s.t = (double)e.t; s.G0 = (double)e.G0; s.B = (double)e.B; s.Bm = (double)e.Bm;
    s.jcount = (u32)e.jcount;                          // <= 10^7
    s.m = e.m;
    s.G = (s.jcount - 1 + e.m - 1) / e.m;
    s.tw = fq_words_log(e.m, fill, tbits);
    return s;
}

// WI: baby steps inserted by fq_insert_count (table kind 3, count bytes
// after the words) instead of one compare-and-swap each (table kind 0); the
// words and the probes are the same.  The words are 2^tw of the launch's
// 2^(tbits-1).
template <int CH, bool WI, bool LOW>
__device__ u64 solve_fp64q(const SolveF& e, unsigned long long* tab, u32 tbits, u64* steps_out) {
    const u32 lane = threadIdx.x & 31, lo = lane & 15;
    const Fp64 f = e.f;
    const u32 m = e.m, G = e.G;
    const u32 mask = (1u << e.tw) - 1, mask8 = mask << 3;

    // the lanes' powers: lanes 0..15 scan to B^(lo+1), lanes 16..31 to Bm^(lo+1)
    // in four steps; B^lane and Bm^(lane+1) are then one product away at most
    double y = lane < 16 ? e.B : e.Bm;
#pragma unroll
    for (int off = 1; off < 16; off <<= 1) {
        const double z = __shfl_up_sync(FULL, y, off, 16);
        if (lo >= (u32)off) y = f.mul(y, z);
    }
    const double B16 = __shfl_sync(FULL, y, 15), Bm16 = __shfl_sync(FULL, y, 31);
    double bl = __shfl_sync(FULL, y, (int)((lo - 1) & 15)), gl = __shfl_sync(FULL, y, (int)(16 + lo));
    if (lo == 0) bl = 1.0;
    if (lane >= 16) {
        bl = f.mul(bl, B16);
        gl = f.mul(gl, Bm16);
    }
    const double B32 = f.mul(B16, B16), Bm32 = f.mul(Bm16, Bm16);
    double Bstep = B32, Gstep = Bm32;                  // B^(32 CH), Bm^(32 CH)
#pragma unroll
    for (int c = 1; c < CH; c <<= 1) {
        Bstep = f.mul(Bstep, Bstep);
        Gstep = f.mul(Gstep, Gstep);
    }
    const double tbl = f.mul(e.t, bl);
    double bx[CH], gx[CH];
    bx[0] = tbl;
    gx[0] = f.mul(e.G0, gl);
#pragma unroll
    for (int c = 1; c < CH; ++c) {
        bx[c] = f.mul(bx[c - 1], B32);
        gx[c] = f.mul(gx[c - 1], Bm32);
    }

    unsigned char* bytes = reinterpret_cast<unsigned char*>(tab);
    unsigned char* cnt = bytes + (4u << tbits);        // kind 3 only
    uint4* t4 = reinterpret_cast<uint4*>(tab);
#pragma unroll 4
    for (u32 k = lane; k <= mask / 2; k += 32) t4[k] = make_uint4(0, 0, 0, 0);
    if (WI)
        for (u32 k = lane; k <= mask / 16; k += 32) reinterpret_cast<uint4*>(cnt)[k] = make_uint4(0, 0, 0, 0);
    __syncwarp();

    for (u32 base = 0; base < m; base += 32 * CH) {
        u32 h[CH], want = 0;
#pragma unroll
        for (int c = 0; c < CH; ++c) {
            h[c] = fq_hash(f.canon(bx[c]), LOW ? kHashKLow : kHashK);
            bx[c] = f.mul(bx[c], Bstep);               // the next value, independent of the insert
            if (base + 32 * c + lane < m) want |= 1u << c;
        }
        if (WI) {
            // (whole iterations but for the last one: want is then a constant)
            if (base + 32 * CH <= m) fq_insert_count<CH>(bytes, cnt, mask8, (1u << CH) - 1, h);
            else fq_insert_count<CH>(bytes, cnt, mask8, want, h);
        } else {
#pragma unroll
            for (int c = 0; c < CH; ++c)
                if ((want >> c) & 1u) fq_insert(tab, mask, (h[c] & mask8) >> 3, fq_fingerprints(h[c]) & 0xFFFFu);
        }
    }
    __syncwarp();

    u64 best = ~0ull;
    u32 giant_done = G;                                // g = 1..G covers j in [1, G*m]
    for (u32 base = 0; base < G; base += 32 * CH) {
        double cv[CH], nx[CH];
        u32 hs[CH];
        u32 z = 0;
#pragma unroll
        for (int c = 0; c < CH; ++c) {
            cv[c] = f.canon(gx[c]);
            hs[c] = fq_hash(cv[c], LOW ? kHashKLow : kHashK);
            nx[c] = f.mul(gx[c], Gstep);                  // the next value, independent of the probe
            const uint2 w = *reinterpret_cast<const uint2*>(bytes + (hs[c] & mask8));
            const u32 rep = fq_fingerprints(hs[c]);
            z |= equal_halves(w.x, rep) | equal_halves(w.y, rep) | (w.x & kQOvf);
        }
        if (__any_sync(FULL, z)) {
            // the rare path: walk overflowed homes, then resolve exact matches in increasing g
            u32 real = 0;
            if (z) {
#pragma unroll
                for (int c = 0; c < CH; ++c)
                    if (base + 32 * c + lane + 1 <= G &&
                        fq_contains(tab, mask, (hs[c] & mask8) >> 3, fq_fingerprints(hs[c]) & 0xFFFFu))
                        real |= 1u << c;
            }
            u64 jb = ~0ull;
            if (__any_sync(FULL, real)) {
#pragma unroll
                for (int c = 0; c < CH; ++c) {
                    u32 bb = __ballot_sync(FULL, (real >> c) & 1u);
                    while (bb && jb == ~0ull) {
                        const int src = __ffs(bb) - 1;
                        bb &= bb - 1;
                        const double v = __shfl_sync(FULL, cv[c], src);
                        const u64 g = base + 32 * c + (u32)src + 1;
                        const int i = ffind_last(f, tbl, B32, m, v);
                        if (i >= 0) jb = g * m - (u64)i;
                    }
                }
            }
            if (jb != ~0ull) {
                best = jb;
                giant_done = min(G, base + 32 * CH);
                break;
            }
        }
#pragma unroll
        for (int c = 0; c < CH; ++c) gx[c] = nx[c];
    }
    __syncwarp();
    if (steps_out) *steps_out = pack_steps(m, giant_done);
    return best < e.jcount ? best : ~0ull;
}

// ---- the FP64 solve with a 16-bit slot table ----
//
// Table: 2^(tbits+1) 16-bit slots per warp (4 << tbits bytes), of which a
// prime with m baby steps uses 2^tw, tw = ceil(log2 m) + load_shift (load at
// most 2^-load_shift).  A key -- the canonical residue x of a baby step -- is
// hashed from the low 32 bits of x, which the FP64 pipe exposes with one add
// (x + 2^52 has x in its low mantissa bits): h = lo32(x) * kHashMul, a
// bijection of lo32(x).  The home slot is the top tw bits of h and holds the
// 15-bit fingerprint (h & 0x7FFF) | 1 (never 0; 0 is an empty slot).  Bit 15
// of a slot is its overflow flag, set when a key homed there found it taken
// and moved on (linear probing).  A probe reads its home slot only: equal
// fingerprints make a candidate; a set overflow flag sends the lane to the
// warp's slow path, which walks the chain.  Candidates are resolved exactly by
// recomputing the baby steps, so fingerprint collisions (about 2^-14 per
// occupied probe) never change a result.

constexpr u32 kHashMul = 0x9E3779B1u;

__device__ __forceinline__ u32 hkey_canon(double x) {          // x canonical in [0, p), p < 2^49
    return (u32)__double2loint(__dadd_rn(x, 4503599627370496.0)) * kHashMul;
}

__device__ __forceinline__ u32 hfp(u32 h) { return (h & 0x7FFFu) | 1u; }

__device__ __forceinline__ void h_insert(unsigned short* tab, u32 mask, u32 shift, u32 h) {
    u32 s = h >> shift;
    const unsigned short f = (unsigned short)hfp(h);
    if (atomicCAS(&tab[s], (unsigned short)0, f) == 0) return;
    atomicOr(reinterpret_cast<u32*>(tab) + (s >> 1), 0x8000u << (16 * (s & 1)));   // flag the home slot
    do s = (s + 1) & mask;
    while (atomicCAS(&tab[s], (unsigned short)0, f) != 0);
}

// Whether a key with hash h may be in the table: its home slot, then (when the
// home's overflow flag is set) the chain up to the first empty slot.
__device__ __forceinline__ bool h_contains(const unsigned short* tab, u32 mask, u32 shift, u32 h) {
    u32 s = h >> shift;
    const u32 f = hfp(h);
    u32 e = tab[s];
    if (((e ^ f) & 0x7FFFu) == 0) return true;
    if (!(e & 0x8000u)) return false;
    for (u32 n = 0; n < mask; ++n) {
        s = (s + 1) & mask;
        e = tab[s];
        if (e == 0) return false;
        if (((e ^ f) & 0x7FFFu) == 0) return true;
    }
    return false;
}

template <int CH>
__device__ u64 solve_fp64h(const Solve& e, unsigned short* tab, u32 tbits, u32 load_shift, u64* steps_out) {
    const u32 lane = threadIdx.x & 31;
    Fp64 f;
    f.init(e.p);
    const u32 m = e.m;
    const u32 jc = (u32)e.jcount;                      // jcount <= 10^7
    const u32 tw = min(tbits + 1, max(6u, 32u - __clz(max(m, 2u) - 1) + load_shift));
    const u32 mask = (1u << tw) - 1, shift = 32 - tw;
    const double B = (double)e.B, Bm = (double)e.Bm, tv = (double)e.t, G0 = (double)e.G0;

    double xb = B, xg = Bm;                            // B^(l+1), Bm^(l+1)
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const double yb = __shfl_up_sync(FULL, xb, off), yg = __shfl_up_sync(FULL, xg, off);
        if (lane >= (u32)off) {
            xb = f.mul(xb, yb);
            xg = f.mul(xg, yg);
        }
    }
    const double B32 = __shfl_sync(FULL, xb, 31), Bm32 = __shfl_sync(FULL, xg, 31);
    double bl = __shfl_up_sync(FULL, xb, 1);
    if (lane == 0) bl = 1.0;
    double Bstep = B32, Gstep = Bm32;                  // B^(32 CH), Bm^(32 CH)
#pragma unroll
    for (int c = 1; c < CH; c <<= 1) {
        Bstep = f.mul(Bstep, Bstep);
        Gstep = f.mul(Gstep, Gstep);
    }
    const double tbl = f.mul(tv, bl);
    double bx[CH], gx[CH];
    bx[0] = tbl;
    gx[0] = f.mul(G0, xg);
#pragma unroll
    for (int c = 1; c < CH; ++c) {
        bx[c] = f.mul(bx[c - 1], B32);
        gx[c] = f.mul(gx[c - 1], Bm32);
    }

    uint4* t4 = reinterpret_cast<uint4*>(tab);
    for (u32 k = lane; k <= (mask >> 3); k += 32) t4[k] = make_uint4(0, 0, 0, 0);
    __syncwarp();

    // baby steps, stopping at a cycle B^d == 1 (d < m)
    u32 cyc = 0, baby_done = m;
    for (u32 base = 0; base < m; base += 32 * CH) {
        double cv[CH];
        u32 cb = 0;
#pragma unroll
        for (int c = 0; c < CH; ++c) {
            cv[c] = f.canon(bx[c]);
            const u32 i = base + 32 * c + lane;
            const u32 bc = __ballot_sync(FULL, i > 0 && i < m && cv[c] == tv);
            if (bc && !cb) cb = base + 32 * c + __ffs(bc) - 1;
        }
        const u32 lim = cb ? cb : m;
#pragma unroll
        for (int c = 0; c < CH; ++c)
            if (base + 32 * c + lane < lim) h_insert(tab, mask, shift, hkey_canon(cv[c]));
        if (cb) {
            cyc = cb;
            baby_done = cb;
            break;
        }
#pragma unroll
        for (int c = 0; c < CH; ++c) bx[c] = f.mul(bx[c], Bstep);
    }
    __syncwarp();

    u64 best = ~0ull;
    u32 giant_done = 0;
    if (cyc) {
        const int i = ffind_baby(f, tbl, B32, 1, cyc, G0);
        if (i > 0) best = cyc - (u32)i;
    } else {
        const u32 G = (jc - 1 + m - 1) / m;            // g = 1..G covers j in [1, G*m]
        giant_done = G;
        for (u32 base = 0; base < G; base += 32 * CH) {
            u32 hs[CH];
            bool flag = false;
#pragma unroll
            for (int c = 0; c < CH; ++c) {
                hs[c] = hkey_canon(f.canon(gx[c]));
                const u32 slot = tab[hs[c] >> shift];
                flag |= (((slot ^ hfp(hs[c])) & 0x7FFFu) == 0) | ((slot & 0x8000u) != 0);
            }
            if (__any_sync(FULL, flag)) {
                // the slow path: walk overflowed homes, then resolve candidates in increasing g
                u32 real = 0;
#pragma unroll
                for (int c = 0; c < CH; ++c)
                    if (base + 32 * c + lane + 1 <= G && h_contains(tab, mask, shift, hs[c])) real |= 1u << c;
                u64 jb = ~0ull;
#pragma unroll
                for (int c = 0; c < CH; ++c) {
                    u32 bb = __ballot_sync(FULL, (real >> c) & 1u);
                    while (bb && jb == ~0ull) {
                        const int src = __ffs(bb) - 1;
                        bb &= bb - 1;
                        const double v = __shfl_sync(FULL, f.canon(gx[c]), src);
                        const u64 g = base + 32 * c + (u32)src + 1;
                        const int i = ffind_baby(f, tbl, B32, 0, m, v);
                        if (i >= 0) jb = g * m - (u64)i;
                    }
                }
                if (jb != ~0ull) {
                    best = jb;
                    giant_done = min(G, base + 32 * CH);
                    break;
                }
            }
#pragma unroll
            for (int c = 0; c < CH; ++c) gx[c] = f.mul(gx[c], Gstep);
        }
    }
    __syncwarp();
    if (steps_out) *steps_out = pack_steps(baby_done, giant_done);
    return best < e.jcount ? best : ~0ull;
}

template <int CH, int QT, bool LOW>
__device__ __forceinline__ u64 solve_any(const Solve& e, void* tab, u32 tbits, u32 load_shift, u32 fill, u64* steps) {
    if (CH == 0 || e.p >= kFp64Limit) return solve_entry<FieldM>(e, (unsigned short*)tab, tbits + 1, steps);
    if (QT == 0) return solve_fp64q<CH ? CH : 1, false, LOW>(solve_f(e, tbits, fill), (unsigned long long*)tab, tbits, steps);
    if (QT == 2) return solve_fp64h<CH ? CH : 1>(e, (unsigned short*)tab, tbits, load_shift, steps);
    if (QT == 3) return solve_fp64q<CH ? CH : 1, true, LOW>(solve_f(e, tbits, fill), (unsigned long long*)tab, tbits, steps);
    return solve_fp64<CH ? CH : 1>(e, (u32*)tab, tbits, steps);
}

// Whether a prime's baby steps fit the table its solve will use (at most half
// of its keys' room), so that every insertion finds a free slot.
template <int CH, int QT>
__device__ __forceinline__ bool fits_table(u64 p, u32 m, u32 tbits) {
    if (CH == 0 || p >= kFp64Limit) return m <= (1u << tbits);              // 2^(tbits+1) 16-bit slots
    if (QT == 0 || QT == 3) return m <= (1u << tbits);                      // 2^(tbits-1) words of four
    if (QT == 2) return m <= (1u << tbits);                                 // 2^(tbits+1) 16-bit slots
    return m < (1u << tbits);                                              // 2^tbits 32-bit slots
}

__device__ __forceinline__ Solve solve_of(const Entry& g) {
    Solve e;
    e.p = g.p; e.t = g.t; e.G0 = g.G0; e.B = g.B; e.Bm = g.Bm;
    e.jcount = g.jcount; e.m = g.m;
    return e;
}

// CH > 0: every entry has p < 2^49 (FP64 solve with CH chains per lane);
// CH == 0: any p (integer Montgomery solve).  LOW: every p is below
// kHashLow.
template <int CH, int QT, bool LOW = false>
__global__ void __launch_bounds__(256, MPS_BSGS_MINB) k_bsgs(BsgsArgs a, Counters* ctr) {
    extern __shared__ __align__(16) u32 smem32[];
    const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // per warp 4 << tbits bytes of table (kind 3: and one count byte per eight)
    u32* tab = smem32 + (size_t)warp * ((1u << a.tbits) + (QT == 3 ? (1u << a.tbits) / 8 : 0u));
    const u64 n_ent = *(volatile unsigned long long*)&ctr->big;
    u64 my_steps = 0, my_baby = 0;
    if (a.persistent) {
        // A warp claims the entry after the one it solves, and lanes 0..7 load
        // that entry's words while the current one is solved, so neither the
        // claim nor the load is waited for between entries.  What is the same
        // for every lane of a solve (1/p, G, the table's width) comes from
        // k_setup, a lane's work there instead of a warp's here, and the five
        // residues are converted where they are staged, one lane each.
        static_assert(offsetof(Entry, pinv) == 40 && offsetof(Entry, jcount) == 48 && offsetof(Entry, G) == 56,
                      "entry staging assumes p, t, G0, B, Bm, 1/p, (jcount, m), (G, tw)");
        u64 cur = 0;
        if (lane == 0) cur = atomicAdd(&ctr->work_next, 1ull);
        cur = __shfl_sync(FULL, cur, 0);
        u64 claim = 0;                                          // lane 0: the entry after cur
        if (lane == 0 && cur < n_ent) claim = atomicAdd(&ctr->work_next, 1ull);
        u32 idx = cur < n_ent ? a.big[cur] : 0u;
        u64 stage = cur < n_ent && lane < 8 ? reinterpret_cast<const u64*>(a.ent + idx)[lane] : 0;
        while (cur < n_ent) {
            const u64 mine = stage, p = __shfl_sync(FULL, mine, 0);
            const u64 jm = __shfl_sync(FULL, mine, 6), gt = __shfl_sync(FULL, mine, 7);   // little-endian pairs
            const u32 this_idx = idx, m = (u32)(jm >> 32);
            const u64 next = __shfl_sync(FULL, claim, 0);
            idx = next < n_ent ? a.big[next] : 0u;
            stage = next < n_ent && lane < 8 ? reinterpret_cast<const u64*>(a.ent + idx)[lane] : 0;
            if (lane == 0 && next < n_ent) claim = atomicAdd(&ctr->work_next, 1ull);
            cur = next;
            if (!fits_table<CH, QT>(p, m, a.tbits)) {           // host sizing error: never overfill a table
                if (lane == 0) atomicOr(&ctr->status, kStatusBadLaunch);
                continue;
            }
            u64 steps = 0, j;
            if (CH > 0 && (QT == 0 || QT == 3) && p < kFp64Limit) {
                const double v = lane < 5 ? (double)mine : __longlong_as_double((long long)mine);
                SolveF e;
                e.f.p = __shfl_sync(FULL, v, 0);
                e.t = __shfl_sync(FULL, v, 1);
                e.G0 = __shfl_sync(FULL, v, 2);
                e.B = __shfl_sync(FULL, v, 3);
                e.Bm = __shfl_sync(FULL, v, 4);
                e.f.pinv = __shfl_sync(FULL, v, 5);
                e.f.pi = p;
                e.jcount = (u32)jm;
                e.m = m;
                e.G = (u32)gt;
                e.tw = min((u32)(gt >> 32), a.tbits - 1);
                j = solve_fp64q<CH ? CH : 1, QT == 3, LOW>(e, (unsigned long long*)tab, a.tbits, &steps);
            } else {
                Solve e;
                e.p = p;
                e.t = __shfl_sync(FULL, mine, 1);
                e.G0 = __shfl_sync(FULL, mine, 2);
                e.B = __shfl_sync(FULL, mine, 3);
                e.Bm = __shfl_sync(FULL, mine, 4);
                e.jcount = (u32)jm;
                e.m = m;
                j = solve_any<CH, QT, LOW>(e, tab, a.tbits, a.load_shift, a.fill, &steps);
            }
            if (lane == 0) {
                if (j != ~0ull) {
                    const Entry& g = a.ent[this_idx];
                    emit_relation(g.p, g.n_first + j * g.L, 0, g.item, a.rel, a.rel_cap, ctr);
                }
                my_steps += (steps & 0xFFFFFFFFull) + (steps >> 32);
                my_baby += steps & 0xFFFFFFFFull;
            }
        }
        if (lane == 0 && my_steps) {
            atomicAdd(&ctr->steps, (unsigned long long)my_steps);
            atomicAdd(&ctr->baby, (unsigned long long)my_baby);
        }
    } else {
        const u64 k = (u64)blockIdx.x * a.warps_per_block + warp;
        if (k >= n_ent) return;
        const Entry& g = a.ent[a.big[k]];
        const Solve e = solve_of(g);
        if (!fits_table<CH, QT>(e.p, e.m, a.tbits)) {
            if (lane == 0) atomicOr(&ctr->status, kStatusBadLaunch);
            return;
        }
        u64 steps = 0;
        const u64 j = solve_any<CH, QT, LOW>(e, tab, a.tbits, a.load_shift, a.fill, &steps);
        if (lane == 0) {
            if (j != ~0ull) emit_relation(e.p, g.n_first + j * g.L, 0, g.item, a.rel, a.rel_cap, ctr);
            atomicAdd(&ctr->steps, (unsigned long long)((steps & 0xFFFFFFFFull) + (steps >> 32)));
            atomicAdd(&ctr->baby, (unsigned long long)(steps & 0xFFFFFFFFull));
        }
    }
}

// ---- lanes per prime: L-lane groups, 32/L primes per warp in lockstep ----
//
// For primes with few baby and giant steps a whole warp per prime spends
// most of its time on per-prime set-up (the lane-power scan, the table
// clear).  Here a warp takes 32/L entries at once and each group of L lanes
// solves one with its own 16-bit slot table (a 1/(32/L) share of the warp's
// table memory); the loops run to the largest bound among the warp's primes
// with per-group predicates, so the groups never diverge.  Same tables, same
// exact resolution and the same smallest-j result as solve_fp64h.

// Smallest i in [lo, limit) with t * B^i == v within the group (-1: none).
// Warp-uniform control flow: a group with want == false only keeps pace.
template <int L>
__device__ int gfind_baby(const Fp64& f, double tbl, double BL, u32 lo, u32 limit, double v, bool want, u32 gl,
                          u32 gshift, u32 gbits) {
    const u32 lim_max = __reduce_max_sync(FULL, want ? limit : 0u);
    double x = tbl;
    int res = -1;
    for (u32 base = 0; base < lim_max; base += L) {
        const u32 i = base + gl;
        const bool hit = want && res < 0 && i >= lo && i < limit && f.canon(x) == v;
        const u32 gb = (__ballot_sync(FULL, hit) >> gshift) & gbits;
        if (gb && res < 0) res = (int)(base + __ffs(gb) - 1);
        if (__all_sync(FULL, !want || res >= 0 || base + L >= limit)) break;
        x = f.mul(x, BL);
    }
    return res;
}

template <int L, int CH>
__global__ void __launch_bounds__(256, MPS_BSGS_MINB) k_bsgs_groups(BsgsArgs a, Counters* ctr) {
    constexpr u32 NG = 32 / L;
    constexpr u32 NG_LOG = NG == 4 ? 2 : NG == 2 ? 1 : 0;
    extern __shared__ __align__(16) u32 smem32[];
    const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const u32 grp = lane / L, gl = lane % L, gshift = grp * L;
    const u32 gbits = L == 32 ? FULL : (1u << L) - 1u;
    const u32 group_slots = (2u << a.tbits) >> NG_LOG;          // 16-bit slots per group
    unsigned short* tab = reinterpret_cast<unsigned short*>(smem32 + (size_t)warp * (1u << a.tbits)) +
                          (size_t)grp * group_slots;
    const u32 tw_max = a.tbits + 1 - NG_LOG;
    const u64 n_ent = *(volatile unsigned long long*)&ctr->big;
    u64 my_steps = 0, my_baby = 0;
    for (;;) {
        u64 first = 0;
        if (lane == 0) first = atomicAdd(&ctr->work_next, (unsigned long long)NG);
        first = __shfl_sync(FULL, first, 0);
        if (first >= n_ent) break;
        const u64 idx = first + grp;
        const Entry& g = a.ent[a.big[idx < n_ent ? idx : n_ent - 1]];
        const Solve e = solve_of(g);
        bool active = idx < n_ent;
        // the host sends only p < 2^49 and at most half a group table of baby steps here
        if (active && (e.p >= kFp64Limit || e.m > (1u << (tw_max - 1)))) {
            if (gl == 0) atomicOr(&ctr->status, kStatusBadLaunch);
            active = false;
        }
        Fp64 f;
        f.init(active ? e.p : 1000003ull);
        const u32 m = active ? e.m : 0;
        const u32 jc = active ? (u32)e.jcount : 0;
        const u32 tw = min(tw_max, max(6u, 32u - __clz(max(m, 2u) - 1) + a.load_shift));
        const u32 mask = (1u << tw) - 1, shift = 32 - tw;
        const double B = active ? (double)e.B : 1.0, Bm = active ? (double)e.Bm : 1.0;
        const double tv = active ? (double)e.t : 1.0, G0 = active ? (double)e.G0 : 1.0;

        double xb = B, xg = Bm;                                 // B^(gl+1), Bm^(gl+1)
#pragma unroll
        for (int off = 1; off < L; off <<= 1) {
            const double yb = __shfl_up_sync(FULL, xb, off, L), yg = __shfl_up_sync(FULL, xg, off, L);
            if (gl >= (u32)off) {
                xb = f.mul(xb, yb);
                xg = f.mul(xg, yg);
            }
        }
        const double BL = __shfl_sync(FULL, xb, L - 1, L), BmL = __shfl_sync(FULL, xg, L - 1, L);
        double bl = __shfl_up_sync(FULL, xb, 1, L);
        if (gl == 0) bl = 1.0;
        double Bstep = BL, Gstep = BmL;                         // B^(L CH), Bm^(L CH)
#pragma unroll
        for (int c = 1; c < CH; c <<= 1) {
            Bstep = f.mul(Bstep, Bstep);
            Gstep = f.mul(Gstep, Gstep);
        }
        const double tbl = f.mul(tv, bl);
        double bx[CH], gx[CH];
        bx[0] = tbl;
        gx[0] = f.mul(G0, xg);
#pragma unroll
        for (int c = 1; c < CH; ++c) {
            bx[c] = f.mul(bx[c - 1], BL);
            gx[c] = f.mul(gx[c - 1], BmL);
        }
        uint4* t4 = reinterpret_cast<uint4*>(tab);
        for (u32 k = gl; k <= (mask >> 3); k += L) t4[k] = make_uint4(0, 0, 0, 0);
        __syncwarp();

        // baby steps, each group stopping at its own cycle B^d == 1 (d < m)
        u32 cyc = 0, baby_done = m;
        bool bdone = m == 0;
        const u32 m_max = __reduce_max_sync(FULL, m);
        for (u32 base = 0; base < m_max; base += L * CH) {
            double cv[CH], nb[CH];
            bool hit = false;
#pragma unroll
            for (int c = 0; c < CH; ++c) {
                cv[c] = f.canon(bx[c]);
                nb[c] = f.mul(bx[c], Bstep);               // the next value, independent of the inserts
                hit |= !bdone && base + L * c + gl - 1u < m - 1u && cv[c] == tv;
            }
            u32 cb = 0;
            if (__any_sync(FULL, hit)) {                    // a cycle in some group: locate it exactly
#pragma unroll
                for (int c = 0; c < CH; ++c) {
                    const u32 i = base + L * c + gl;
                    const u32 gb = (__ballot_sync(FULL, !bdone && i > 0 && i < m && cv[c] == tv) >> gshift) & gbits;
                    if (gb && !cb) cb = base + L * c + __ffs(gb) - 1;
                }
            }
            const u32 lim = cb ? cb : m;
#pragma unroll
            for (int c = 0; c < CH; ++c)
                if (!bdone && base + L * c + gl < lim) h_insert(tab, mask, shift, hkey_canon(cv[c]));
            if (cb && !bdone) {
                cyc = cb;
                baby_done = cb;
            }
            bdone = bdone || cb != 0 || base + L * CH >= m;
            if (__all_sync(FULL, bdone)) break;
#pragma unroll
            for (int c = 0; c < CH; ++c) bx[c] = nb[c];
        }
        __syncwarp();

        u64 best = ~0ull;
        // a cycle: the j in [1, cyc) with G0 == t B^(cyc - j)
        {
            const int i = gfind_baby<L>(f, tbl, BL, 1, cyc, G0, cyc != 0, gl, gshift, gbits);
            if (cyc && i > 0) best = cyc - (u32)i;
        }
        const u32 G = (active && !cyc && jc > 1) ? (jc - 1 + m - 1) / m : 0;   // g = 1..G covers j in [1, G*m]
        u32 giant_done = G;
        bool gdone = G == 0;
        const u32 G_max = __reduce_max_sync(FULL, G);
        for (u32 base = 0; base < G_max; base += L * CH) {
            u32 hs[CH];
            double nx[CH];
            bool flag = false;
#pragma unroll
            for (int c = 0; c < CH; ++c) {
                hs[c] = hkey_canon(f.canon(gx[c]));
                nx[c] = f.mul(gx[c], Gstep);                   // the next value, independent of the probe
                const u32 slot = tab[hs[c] >> shift];
                flag |= !gdone && ((((slot ^ hfp(hs[c])) & 0x7FFFu) == 0) | ((slot & 0x8000u) != 0));
            }
            if (__any_sync(FULL, flag)) {
                u32 real = 0;
#pragma unroll
                for (int c = 0; c < CH; ++c)
                    if (!gdone && base + L * c + gl + 1 <= G && h_contains(tab, mask, shift, hs[c])) real |= 1u << c;
                u64 jb = ~0ull;
#pragma unroll
                for (int c = 0; c < CH; ++c) {
                    u32 gb = (__ballot_sync(FULL, (real >> c) & 1u) >> gshift) & gbits;
                    const double cvc = f.canon(gx[c]);
                    while (__any_sync(FULL, gb != 0 && jb == ~0ull)) {
                        const bool mine = gb != 0 && jb == ~0ull;
                        const int src = mine ? __ffs(gb) - 1 : 0;
                        const double v = __shfl_sync(FULL, cvc, gshift + (u32)src);
                        const int i = gfind_baby<L>(f, tbl, BL, 0, m, v, mine, gl, gshift, gbits);
                        if (mine) {
                            gb &= gb - 1;
                            if (i >= 0) jb = (u64)(base + L * c + (u32)src + 1) * m - (u64)i;
                        }
                    }
                }
                if (jb != ~0ull && !gdone) {
                    best = jb;
                    giant_done = min(G, base + L * CH);
                    gdone = true;
                }
            }
            gdone = gdone || base + L * CH >= G;
            if (__all_sync(FULL, gdone)) break;
#pragma unroll
            for (int c = 0; c < CH; ++c) gx[c] = nx[c];
        }
        __syncwarp();
        if (gl == 0 && active) {
            if (best < e.jcount) emit_relation(e.p, g.n_first + best * g.L, 0, g.item, a.rel, a.rel_cap, ctr);
            my_steps += (u64)baby_done + giant_done;
            my_baby += baby_done;
        }
    }
    if (gl == 0 && my_steps) {
        atomicAdd(&ctr->steps, (unsigned long long)my_steps);
        atomicAdd(&ctr->baby, (unsigned long long)my_baby);
    }
}

// -------------------------------------------------------------- the order --

// y^2 + c in [0, n) (Montgomery squaring; any polynomial map serves rho).
__device__ __forceinline__ u64 rho_step(const Mont& R, u64 y, u64 c) {
    u64 z = R.norm(R.mul(y, y)) + c;
    return z >= R.p ? z - R.p : z;
}

// Pollard-Brent rho with the 32 lanes of a warp walking 32 different maps
// y -> y^2 + c (c = c0 + lane) in lockstep; the first lane whose batch gcd
// gives a nontrivial factor wins (a batch that overshoots to n is replayed
// step by step from its start).  Returns a nontrivial factor of the odd
// composite n < 2^62, or 0 after four rounds of 32 maps.  Warp-uniform.
__device__ u64 warp_rho_factor(u64 n) {
    const u32 lane = threadIdx.x & 31;
    Mont R;
    R.init(n);
    for (u64 c0 = 1; c0 < 1 + 32 * 4; c0 += 32) {
        const u64 c = c0 + lane;
        u64 y = R.one, q = R.one, x = 0, ys = 0, g = 1;
        bool stop = false;
        for (u64 r = 1; r <= (1ull << 24) && !stop; r <<= 1) {
            if (g == 1) x = y;                         // a lane that found g keeps its x and ys for the replay
            for (u64 i = 0; i < r; ++i) y = rho_step(R, y, c);
            for (u64 k = 0; k < r && !stop; k += 128) {
                if (g == 1) ys = y;
                const u64 lim = min((u64)128, r - k);
                for (u64 i = 0; i < lim; ++i) {
                    y = rho_step(R, y, c);
                    q = R.mul(q, x > y ? x - y : y - x);
                }
                if (g == 1) g = gcd64(R.norm(q), n);
                stop = __any_sync(FULL, g != 1 && g != n) || __all_sync(FULL, g != 1);
            }
        }
        if (g == n) {                                  // replay this lane's last batch one step at a time
            g = 1;
            for (u32 it = 0; it < 128 && g == 1; ++it) {
                ys = rho_step(R, ys, c);
                g = gcd64(x > ys ? x - ys : ys - x, n);
            }
        }
        const u32 good = __ballot_sync(FULL, g != 1 && g != n);
        if (good) return __shfl_sync(FULL, g, __ffs(good) - 1);
    }
    return 0;
}

// Exact 12-base Miller-Rabin (Math.hpp:209-251) with the bases spread over
// the lanes of a warp: lane k < 12 tries base k.  Warp-uniform result.
__device__ bool warp_is_prime64(u64 n) {
    const u32 lane = threadIdx.x & 31;
    const u32 bases[12] = {2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31, 37};
    if (n < 2) return false;
    for (int i = 0; i < 12; ++i) {
        if (n == bases[i]) return true;
        if (n % bases[i] == 0) return false;
    }
    bool ok = true;
    if (lane < 12) {
        Mont M;
        M.init(n);
        ok = sprp(M, bases[lane], M.r2());
    }
    return __all_sync(FULL, ok);
}

// q = ord_p(b), b mod p != 0, p prime (Math.hpp:294-310), one warp: the
// lanes split the trial division of p - 1 by the sieving primes (divisibility
// by multiplicative inverses, the loads of 256 primes in flight at once: a
// lone relation's order is bound by their latency, not by its arithmetic); the cofactor is finished by Miller-Rabin /
// Pollard rho; then each prime factor is stripped from the order.
__device__ u64 warp_mult_order(u64 b, u64 p, const SieveTables& t, bool* failed) {
    const u32 lane = threadIdx.x & 31;
    if (p < 1000) {
        u64 x = b % p, k = 1;
        while (x != 1) {
            x = (x * (b % p)) % p;
            ++k;
        }
        return k;
    }
    u64 f[24];
    int nf = 0;
    const u64 pm1 = p - 1;
    const u64 n0 = pm1 >> (__ffsll((long long)pm1) - 1);    // odd part
    f[nf++] = 2;
    // kAhead groups of 32 primes at a time: their loads are in flight together
    // (one group at a time, the loop is a chain of 205 global-memory latencies:
    // k_order on 38 relations at 10^9 took 52 us, with eight groups ahead 25 us;
    // on 17 at 10^12, 257 and 94 us)
    constexpr u32 kAhead = 8;
    const u32 pad = kSievePrimes - 1;
    for (u32 base = 0; base < kSievePrimes; base += 32 * kAhead) {
        u64 q[kAhead], inv[kAhead], rcp[kAhead];
#pragma unroll
        for (u32 g = 0; g < kAhead; ++g) {
            const u32 k = min(base + 32 * g + lane, pad);
            q[g] = t.sp[k];
            inv[g] = t.inv[k];
            rcp[g] = t.rcp[k];
        }
        u32 div = 0;
#pragma unroll
        for (u32 g = 0; g < kAhead; ++g)
            if (base + 32 * g + lane <= pad && q[g] * q[g] <= n0 && n0 * inv[g] <= rcp[g]) div |= 1u << g;
        if (__any_sync(FULL, div)) {
#pragma unroll
            for (u32 g = 0; g < kAhead; ++g) {
                u32 bal = __ballot_sync(FULL, (div >> g) & 1u);
                while (bal) {
                    const int src = __ffs(bal) - 1;
                    bal &= bal - 1;
                    const u64 qf = __shfl_sync(FULL, q[g], src);
                    if (nf < 24) f[nf++] = qf;
                }
            }
        }
        // lane 31's last prime is the largest of the round
        if (__shfl_sync(FULL, q[kAhead - 1] * q[kAhead - 1] > n0, 31)) break;
    }
    // the cofactor of n0 by the small factors found
    u64 c = n0;
    for (int i = 1; i < nf; ++i)
        while (c % f[i] == 0) c /= f[i];
    if (c > 1) {
        u64 stack[8];
        int sp = 0;
        stack[sp++] = c;
        while (sp > 0) {
            const u64 x = stack[--sp];
            if (x == 1) continue;
            if (x < (u64)kSieveMaxPrime * kSieveMaxPrime || warp_is_prime64(x)) {
                bool dup = false;
                for (int i = 0; i < nf; ++i) dup |= f[i] == x;
                if (!dup && nf < 24) f[nf++] = x;
                continue;
            }
            const u64 dv = warp_rho_factor(x);
            if (dv == 0 || sp + 2 > 8) {
                *failed = true;
                return 0;
            }
            stack[sp++] = dv;
            stack[sp++] = x / dv;
        }
    }
    // the order, one prime factor q of p - 1 per lane (nf <= 24): with q^k the
    // power of q in p - 1, x = b^((p-1)/q^k) has order q^j, the q-part of
    // ord_p(b); the order is the product of the lanes' parts
    Mont M;
    M.init(p);
    const u64 bm = M.to_mont(b % p, M.r2());
    u64 q = 0;
#pragma unroll
    for (int i = 0; i < 24; ++i)
        if (i < nf && (u32)i == lane) q = f[i];
    u64 part = 1;
    if (q) {
        u64 t = pm1;
        while (t % q == 0) t /= q;                     // t = (p - 1) / q^k
        u64 x = M.pow(bm, t);
        while (x != M.one) {
            x = M.pow(x, q);
            part *= q;
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) part *= __shfl_xor_sync(FULL, part, off);
    return part;
}

// One warp per relation: exact primality of p (composite survivors are
// dropped, q = ~0) and q = ord_p(b).
__global__ void __launch_bounds__(128) k_order(OrderArgs a, Counters* ctr) {
    const u64 n = min((u64)*(volatile unsigned long long*)&ctr->relations, a.rel_cap);
    const u32 lane = threadIdx.x & 31;
    const u64 w0 = (blockIdx.x * (u64)blockDim.x + threadIdx.x) >> 5;
    const u64 nw = ((u64)gridDim.x * blockDim.x) >> 5;
    for (u64 i = w0; i < n; i += nw) {
        RawRelation r = a.rel[i];
        if (!warp_is_prime64(r.p)) {
            r.q = ~0ull;
        } else if (r.q == 0) {
            const DevItem& it = a.items[r.item];
            const u64 b_mod = residue128(it.babs_hi, it.babs_lo, it.b_neg, r.p);
            bool failed = false;
            r.q = warp_mult_order(b_mod, r.p, a.tables, &failed);
            if (failed && lane == 0) atomicOr(&ctr->status, kStatusOrderFailed);
        }
        if (lane == 0) a.rel[i] = r;
    }
}

// ------------------------------------------------------- served-item state --

// A wave whose buffers overflowed commits nothing: the host redoes its runs
// and records them with k_state_add.
__global__ void k_commit(const WaveDesc* w, const RawRelation* rel, const Counters* ctr, u64 rel_cap, ItemState* st) {
    if (ctr->status & (kStatusSurvivorOverflow | kStatusEntryOverflow | kStatusRelationOverflow)) return;
    const u32 tid = blockIdx.x * blockDim.x + threadIdx.x;
    const u32 n_runs = w->n_runs;
    if (tid < n_runs) {
        const SieveRun& r = w->runs[tid];
        atomicMax(&st[r.item].p_done, (unsigned long long)r.hi);
        atomicAdd(&st[r.item].waves, 1ull);
    }
    const u64 n = min((u64)ctr->relations, rel_cap);
    for (u64 i = tid; i < n; i += (u64)gridDim.x * blockDim.x) {
        const RawRelation r = rel[i];
        if (r.q == ~0ull) continue;                     // a composite survivor
        ItemState& s = st[r.item];
        const u64 k = atomicAdd(&s.n_rel, 1ull);
        if (s.rel_buf && k < s.rel_cap) s.rel_buf[k] = r;
    }
}

// One run redone on the host path: advance the item to hi, append its relations.
__global__ void k_state_add(ItemState* st, u32 item, u64 hi, const RawRelation* rel, u64 n) {
    ItemState& s = st[item];
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        atomicMax(&s.p_done, (unsigned long long)hi);
        atomicAdd(&s.waves, 1ull);
    }
    for (u64 i = blockIdx.x * (u64)blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x) {
        const u64 k = atomicAdd(&s.n_rel, 1ull);
        if (s.rel_buf && k < s.rel_cap) s.rel_buf[k] = rel[i];
    }
}

// ------------------------------------------------------ prime counting --

// Strong probable-prime test of p to base a (a < p) in field F.
template <class F>
__device__ __forceinline__ bool sprp_f(const F& f, u64 p, u64 a) {
    const u64 pm1 = p - 1;
    const int s = __ffsll((long long)pm1) - 1;
    typename F::V x = f.pow(f.from_u64(a), pm1 >> s);
    u64 y = f.residue(x);
    if (y == 1 || y == pm1) return true;
    for (int r = 1; r < s; ++r) {
        x = f.mul(x, x);
        y = f.residue(x);
        if (y == pm1) return true;
        if (y == 1) return false;
    }
    return false;
}

// Exact primality of an odd p > 37 with no factor <= 37: strong tests to the
// 12 bases 2..37 (the set of is_prime64, Math.hpp:209-251), in field F.
template <class F>
__device__ bool is_prime_f(u64 p) {
    const u32 bases[12] = {2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31, 37};
    F f;
    f.init(p);
    for (int i = 0; i < 12; ++i)
        if (!sprp_f(f, p, bases[i])) return false;
    return true;
}

__global__ void __launch_bounds__(256) k_count_primes(const u64* surv, u64 surv_cap, Counters* ctr) {
    const u64 n = min((u64)*(volatile unsigned long long*)&ctr->survivors, surv_cap);
    u32 mine = 0;
    for (u64 i = blockIdx.x * (u64)blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x) {
        const u64 p = surv[i];
        bool prime;
        if (p < 65536ull * 65536ull) {
            prime = true;                               // survivors below 65536^2 are the primes
        } else {
            prime = p < kFp64Limit ? is_prime_f<FieldF>(p) : is_prime_f<FieldM>(p);
        }
        mine += prime ? 1u : 0u;
    }
    const u32 warp_total = __reduce_add_sync(FULL, mine);
    if ((threadIdx.x & 31) == 0 && warp_total) atomicAdd(&ctr->primes, (unsigned long long)warp_total);
}

// ------------------------------------------------------- roofline probes --

// Independent Montgomery multiplies: 8 chains per thread, no memory traffic;
// the arithmetic ceiling of the BSGS step.
__global__ void __launch_bounds__(256) k_mmul_peak(u64 p0, u32 iters, u64* sink) {
    Mont M;
    M.p = p0 | 1;
    M.ninv = Mont::neg_inverse(M.p);
    M.one = 1;
    u64 x[8];
    const u64 y = (0x9E3779B97F4A7C15ull ^ threadIdx.x) % M.p;
#pragma unroll
    for (int k = 0; k < 8; ++k) x[k] = (blockIdx.x * 8191ull + threadIdx.x * 31ull + k) % M.p;
    for (u32 i = 0; i < iters; ++i) {
#pragma unroll
        for (int k = 0; k < 8; ++k) x[k] = M.mul(x[k], y);
    }
    u64 acc = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) acc ^= x[k];
    if (acc == 0x123456789ull) sink[0] = acc;
}

// Independent exact FP64 modular multiplies (p < 2^49): 8 chains per thread.
__global__ void __launch_bounds__(256) k_fmul_peak(u64 p0, u32 iters, u64* sink) {
    Fp64 f;
    f.init(p0 | 1);
    double x[8];
    const double y = (double)((0x9E3779B97F4A7C15ull ^ threadIdx.x) % f.pi);
#pragma unroll
    for (int k = 0; k < 8; ++k) x[k] = (double)((blockIdx.x * 8191ull + threadIdx.x * 31ull + k) % f.pi);
    for (u32 i = 0; i < iters; ++i) {
#pragma unroll
        for (int k = 0; k < 8; ++k) x[k] = f.mul(x[k], y);
    }
    double acc = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) acc += x[k];
    if (acc == 123.0) sink[0] = (u64)acc;
}

// Independent 32-bit multiply-adds: 8 chains per thread.
__global__ void __launch_bounds__(256) k_imad_peak(u32 iters, u32* sink) {
    u32 x[8];
    const u32 a = 0x9E3779B1u ^ threadIdx.x, b = 0x85EBCA6Bu + blockIdx.x;
#pragma unroll
    for (int k = 0; k < 8; ++k) x[k] = threadIdx.x + k;
    for (u32 i = 0; i < iters; ++i) {
#pragma unroll
        for (int k = 0; k < 8; ++k) x[k] = x[k] * a + b;
    }
    u32 acc = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) acc ^= x[k];
    if (acc == 0x12345u) sink[0] = acc;
}

// Conflict-free shared-memory atomicOr: lane l of every warp always hits
// bank l of an 8 KB bitmap (the sieve's segment), 8 independent words per
// thread per iteration.
__global__ void __launch_bounds__(256) k_smem_or_peak(u32 iters, u32* sink) {
    __shared__ u32 bits[kSegWords];
    const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (u32 w = threadIdx.x; w < kSegWords; w += blockDim.x) bits[w] = 0;
    __syncthreads();
    for (u32 i = 0; i < iters; ++i) {
#pragma unroll
        for (u32 k = 0; k < 8; ++k) atomicOr(&bits[lane + 32 * ((warp * 8 + k + i) & 63)], 1u << ((i + k) & 31));
    }
    __syncthreads();
    if (bits[threadIdx.x] == 0x12345u) sink[0] = bits[threadIdx.x];
}

// ------------------------------------------------------------- test hooks --

__global__ void k_is_prime(const u64* n, u32* out, u64 count) {
    for (u64 i = blockIdx.x * (u64)blockDim.x + threadIdx.x; i < count; i += (u64)gridDim.x * blockDim.x)
        out[i] = is_prime64(n[i]) ? 1u : 0u;
}

// cases[5i..5i+4] = p, B, G0, t, jcount (plain residues); one warp per case.
__global__ void k_bsgs_direct(const u64* cases, u64* j_out, u64 count, u32 tbits, u32 table_kind) {
    extern __shared__ __align__(16) u32 smem32[];
    const u64 idx = blockIdx.x;
    if (idx >= count) return;
    const u64* c = cases + 5 * idx;
    const u64 p = c[0];
    Solve e;
    e.p = p; e.B = c[1] % p; e.G0 = c[2] % p; e.t = c[3] % p; e.jcount = c[4];
    u64 result;
    if (e.jcount == 0) {
        result = ~0ull;
    } else if (e.G0 == e.t) {
        result = 0;
    } else if (e.jcount == 1) {
        result = ~0ull;
    } else {
        u32 m = (u32)isqrt_ceil_dev(e.jcount);
        // the table loads of the sieving path
        const u32 cap = min(kMaxBaby, table_kind == 0 || table_kind == 3 ? 1u << (tbits - 1)
                                      : table_kind == 2                    ? 1u << (tbits + 1 - kDefaultLoadShift)
                                                                           : max(1u, (1u << tbits) / 5));
        if (m > cap) m = cap;
        e.m = m;
        Mont M;
        M.init(p);
        const u64 rr = M.r2();
        e.Bm = M.from_mont(M.pow(M.to_mont(e.B, rr), m));
        if (e.p >= kFp64Limit) result = solve_any<0, 0, false>(e, smem32, tbits, kDefaultLoadShift, kDefaultFill, nullptr);
        else if (table_kind == 0) result = solve_any<2, 0, false>(e, smem32, tbits, kDefaultLoadShift, kDefaultFill, nullptr);
        else if (table_kind == 2) result = solve_any<2, 2, false>(e, smem32, tbits, kDefaultLoadShift, kDefaultFill, nullptr);
        else if (table_kind == 3) result = solve_any<2, 3, false>(e, smem32, tbits, 0, kDefaultFill, nullptr);
        else result = solve_any<2, 1, false>(e, smem32, tbits, kDefaultLoadShift, kDefaultFill, nullptr);
    }
    if (threadIdx.x == 0) j_out[idx] = result;
}

__global__ void k_order_direct(const u64* bp, u64* q_out, u64 count, SieveTables t) {
    const u64 w0 = (blockIdx.x * (u64)blockDim.x + threadIdx.x) >> 5;
    const u64 nw = ((u64)gridDim.x * blockDim.x) >> 5;
    for (u64 i = w0; i < count; i += nw) {
        bool failed = false;
        const u64 q = warp_mult_order(bp[2 * i], bp[2 * i + 1], t, &failed);
        if ((threadIdx.x & 31) == 0) q_out[i] = failed ? 0 : q;
    }
}

// -------------------------------------------------------------- launchers --

size_t bsgs_smem_bytes(u32 tbits, u32 warps_per_block, u32 table_kind) {
    const size_t per_warp = (size_t)(4u << tbits);
    return (size_t)warps_per_block * (table_kind == 3 ? per_warp + per_warp / 8 : per_warp);
}

bool valid_seg_words(u32 seg_words) { return seg_words == 1024 || seg_words == 2048 || seg_words == 4096; }

// The segment size of one range.
u32 range_seg_words(u32 seg_words, u64 n_odds) {
    while (seg_words > kLeastSegWords && n_odds < kFewSegs * seg_words * 32) seg_words /= 2;
    return seg_words;
}

cudaError_t launch_sieve(const SieveArgs& a, const SieveTables& t, const SurvOut& o, Counters* ctr, cudaStream_t s,
                         u32 seg_words, bool fit) {
    if (!valid_seg_words(seg_words)) return cudaErrorInvalidValue;
    if (fit) seg_words = range_seg_words(seg_words, a.n_odds);
    const u64 seg_odds = (u64)seg_words * 32;
    const u64 segs = (a.n_odds + seg_odds - 1) / seg_odds;
    if (segs == 0 && !a.include_two) return cudaSuccess;
    const u64 grid = segs == 0 ? 1 : min(segs, (u64)148 * 8);
    auto go = [&](auto kern) {
        kern<<<(unsigned)grid, kSieveThreads, 0, s>>>(a, t, o, ctr);
        return cudaGetLastError();
    };
    switch (seg_words) {
        case 256: return go(k_sieve<256>);
        case 512: return go(k_sieve<512>);
        case 1024: return go(k_sieve<1024>);
        case 4096: return go(k_sieve<4096>);
        default: return go(k_sieve<2048>);
    }
}

cudaError_t launch_sieve_wave(const WaveDesc* w, const SieveTables& t, const SurvOut& o, Counters* ctr, int grid,
                              cudaStream_t s, u32 seg_words) {
    auto go = [&](auto kern) {
        kern<<<grid, kSieveThreads, 0, s>>>(w, t, o, ctr);
        return cudaGetLastError();
    };
    switch (seg_words) {
        case 256: return go(k_sieve_wave<256>);
        case 512: return go(k_sieve_wave<512>);
        case 1024: return go(k_sieve_wave<1024>);
        case 2048: return go(k_sieve_wave<2048>);
        case 4096: return go(k_sieve_wave<4096>);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_prep(const PrepArgs& a, Counters* ctr, int grid, int num_sms, cudaStream_t s) {
    k_prep<<<grid, kPrepThreads, 0, s>>>(a, ctr);
    if (a.split && !a.surv_split) k_split<<<num_sms * 2, 256, 0, s>>>(a, ctr);
    if (a.split) k_dlog<<<num_sms * 4, 256, 0, s>>>(a, ctr);
    k_setup<<<num_sms * 7, kSetupWarps * 32, 0, s>>>(a, ctr);
    return cudaGetLastError();
}

// Dynamic shared memory limit of every k_bsgs variant on the current device
// (the attribute is per device; set once per size and device, before any
// graph capture, so that a captured launch never needs it).
cudaError_t bsgs_reserve_smem(size_t smem) {
    constexpr int kDevices = 64;
    static std::mutex lock;
    static size_t done[kDevices] = {};
    int dev = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess) return err;
    if (dev < 0 || dev >= kDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> g(lock);
    if (smem <= done[dev]) return cudaSuccess;
    for (auto kern : {k_bsgs<0, 0>, k_bsgs<1, 0>, k_bsgs<2, 0>, k_bsgs<4, 0>, k_bsgs<1, 1>, k_bsgs<2, 1>,
                      k_bsgs<4, 1>, k_bsgs<1, 2>, k_bsgs<2, 2>, k_bsgs<4, 2>, k_bsgs<1, 3>, k_bsgs<2, 3>,
                      k_bsgs<4, 3>, k_bsgs<1, 0, true>, k_bsgs<2, 0, true>, k_bsgs<4, 0, true>, k_bsgs<1, 3, true>,
                      k_bsgs<2, 3, true>, k_bsgs<4, 3, true>, k_bsgs_groups<8, 1>, k_bsgs_groups<8, 2>,
                      k_bsgs_groups<16, 1>, k_bsgs_groups<16, 2>}) {
        err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (err != cudaSuccess) return err;
    }
    done[dev] = smem;
    return cudaSuccess;
}

cudaError_t launch_bsgs(const BsgsArgs& a, Counters* ctr, int grid, cudaStream_t s) {
    const size_t smem = bsgs_smem_bytes(a.tbits, a.warps_per_block,
                                        a.max_p >= kFp64Limit || (a.table_kind == 2 && a.lanes != 32) ? 0 : a.table_kind);
    cudaError_t err = bsgs_reserve_smem(smem);
    if (err != cudaSuccess) return err;
    auto go = [&](auto kern) {
        kern<<<grid, a.warps_per_block * 32, smem, s>>>(a, ctr);
        return cudaGetLastError();
    };
    if (a.max_p >= kFp64Limit) return go(k_bsgs<0, 0>);
    if (a.table_kind == 2 && (a.lanes == 8 || a.lanes == 16)) {
        // groups of lanes per prime: FP64 arithmetic only (the caller checked p < 2^49)
        if (a.lanes == 8) return a.chains == 1 ? go(k_bsgs_groups<8, 1>) : go(k_bsgs_groups<8, 2>);
        return a.chains == 1 ? go(k_bsgs_groups<16, 1>) : go(k_bsgs_groups<16, 2>);
    }
    if (a.table_kind == 3) {
        if (a.chains == 4) return a.low ? go(k_bsgs<4, 3, true>) : go(k_bsgs<4, 3>);
        if (a.chains == 1) return a.low ? go(k_bsgs<1, 3, true>) : go(k_bsgs<1, 3>);
        return a.low ? go(k_bsgs<2, 3, true>) : go(k_bsgs<2, 3>);
    }
    if (a.table_kind == 2) {
        if (a.chains == 4) return go(k_bsgs<4, 2>);
        if (a.chains == 1) return go(k_bsgs<1, 2>);
        return go(k_bsgs<2, 2>);
    }
    if (a.table_kind == 1) {
        if (a.chains == 4) return go(k_bsgs<4, 1>);
        if (a.chains == 1) return go(k_bsgs<1, 1>);
        return go(k_bsgs<2, 1>);
    }
    if (a.chains == 4) return a.low ? go(k_bsgs<4, 0, true>) : go(k_bsgs<4, 0>);
    if (a.chains == 1) return a.low ? go(k_bsgs<1, 0, true>) : go(k_bsgs<1, 0>);
    return a.low ? go(k_bsgs<2, 0, true>) : go(k_bsgs<2, 0>);
}

cudaError_t launch_order(const OrderArgs& a, Counters* ctr, int grid, cudaStream_t s) {
    k_order<<<grid, 128, 0, s>>>(a, ctr);
    return cudaGetLastError();
}

cudaError_t launch_commit(const WaveDesc* w, const RawRelation* rel, const Counters* ctr, u64 rel_cap,
                          ItemState* st, cudaStream_t s) {
    k_commit<<<4, 128, 0, s>>>(w, rel, ctr, rel_cap, st);
    return cudaGetLastError();
}

cudaError_t launch_state_add(ItemState* st, u32 item, u64 hi, const RawRelation* rel, u64 n, cudaStream_t s) {
    k_state_add<<<(unsigned)std::min<u64>((n + 255) / 256 + 1, 256), 256, 0, s>>>(st, item, hi, rel, n);
    return cudaGetLastError();
}

cudaError_t launch_count_primes(const u64* surv, u64 surv_cap, Counters* ctr, int grid, cudaStream_t s) {
    k_count_primes<<<grid, 256, 0, s>>>(surv, surv_cap, ctr);
    return cudaGetLastError();
}

cudaError_t launch_mmul_peak(u64 p, u32 iters, int grid, u64* sink, cudaStream_t s) {
    k_mmul_peak<<<grid, 256, 0, s>>>(p, iters, sink);
    return cudaGetLastError();
}

cudaError_t launch_fmul_peak(u64 p, u32 iters, int grid, u64* sink, cudaStream_t s) {
    k_fmul_peak<<<grid, 256, 0, s>>>(p, iters, sink);
    return cudaGetLastError();
}

cudaError_t launch_imad_peak(u32 iters, int grid, u32* sink, cudaStream_t s) {
    k_imad_peak<<<grid, 256, 0, s>>>(iters, sink);
    return cudaGetLastError();
}

cudaError_t launch_smem_or_peak(u32 iters, int grid, u32* sink, cudaStream_t s) {
    k_smem_or_peak<<<grid, 256, 0, s>>>(iters, sink);
    return cudaGetLastError();
}

cudaError_t launch_is_prime(const u64* n, u32* out, u64 count, cudaStream_t s) {
    if (count == 0) return cudaSuccess;
    k_is_prime<<<(unsigned)min((count + 127) / 128, (u64)4096), 128, 0, s>>>(n, out, count);
    return cudaGetLastError();
}

cudaError_t launch_bsgs_direct(const u64* cases, u64* j_out, u64 count, u32 tbits, u32 table_kind, cudaStream_t s) {
    if (count == 0) return cudaSuccess;
    const size_t smem = bsgs_smem_bytes(tbits, 1, table_kind);
    cudaError_t err = cudaFuncSetAttribute(k_bsgs_direct, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (err != cudaSuccess) return err;
    k_bsgs_direct<<<(unsigned)count, 32, smem, s>>>(cases, j_out, count, tbits, table_kind);
    return cudaGetLastError();
}

cudaError_t launch_order_direct(const u64* bp, u64* q_out, u64 count, SieveTables t, cudaStream_t s) {
    if (count == 0) return cudaSuccess;
    k_order_direct<<<(unsigned)min((count + 3) / 4, (u64)4096), 128, 0, s>>>(bp, q_out, count, t);
    return cudaGetLastError();
}

}  // namespace mps
