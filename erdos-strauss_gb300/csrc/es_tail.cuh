// es_tail.cuh -- warp-cooperative survivor tail: Miller-Rabin, factorization, the rung DP.
//
// One prime's rung walk is a chain of dependent steps (trial division, a primality test,
// sometimes Brent's rho, then a divisor DP), so a thread per prime is latency-bound: the
// slowest prime sets the time of the whole window. Here every step is spread over a warp:
//   trial division   lane i tests the odd primes i, i+32, ... below 2^16 against n by
//                    multiplicative inverse; hits are gathered by ballot and divided out of
//                    the cofactor with one warp-wide product of inverses per chunk
//   primality        lanes 0..11 each run one of the 12 strong-probable-prime rounds
//   Brent's rho      all 32 lanes walk with different constants c; the first split wins
//                    (the factorization is unique, so which lane wins cannot change it)
//   ECM              in the latency-bound tail, a cofactor rho has not split after ECM_AFTER
//                    steps gets rounds of one elliptic curve per lane (es_ecm.cuh), the first
//                    divisor wins
//   rung DP          the least divisor up to 65536 in the rung's class by 32-bit values; if there is
//                    none, whether any divisor is in the class; only then the least of all: lanes
//                    own residue classes t mod r and gather
//                    nxt[t] = min_j cur[t * pr^-j] * pr^j over j <= e with the bound <= q
// and a team of four warps walks successive rungs of one prime concurrently, keeping the
// smallest rung that certifies (the reference's emission rule, sieve/rung_scan3.cpp:574-603).
//
// Code size bounds the bulk of it: the warps of an SM are at different places of a long walk, so
// what they run has to fit the instruction cache. With the compiler's own unrolling of these loops
// 32-41 % of the fetches missed it and waiting for instructions was the first stall (5.8-8.9 warps a
// cycle); so the loops that are a chain anyway (multiplies of a power or a walk, lanes' tables) stay
// rolled (unroll 1) and rare paths are out of line. With that and one sieve a prime in the bulk
// (td_sieve), stage D of a window of 2^41 integers at 1e15 takes 1.78 ms for 2.88. Calls in the place
// of whole inlined steps cost more than the misses that they save.
#pragma once
#include "es_arith.cuh"
#include "es_ecm.cuh"

namespace es {

constexpr unsigned FULL = 0xFFFFFFFFu;
constexpr int TD_CHUNKS = (NTD + 31) / 32;     // 205 chunks of 32 primes
constexpr u64 WARP_RHO_STEPS = 1ull << 24;     // per lane, per split

struct WarpFac {          // shared memory, one per warp
  u64 pr[MAXF];
  u32 ex[MAXF];
  int k;
  int overflow;
};

// Append prime p with exponent e (merging a repeat). Lane 0 writes; all lanes call.
__device__ __forceinline__ void wf_add(WarpFac &F, u64 p, int e, u32 lane) {
  if (lane == 0) {
    int i = 0;
    for (; i < F.k; ++i) if (F.pr[i] == p) { F.ex[i] += e; break; }
    if (i == F.k) {
      if (F.k < MAXF) { F.pr[F.k] = p; F.ex[F.k] = e; ++F.k; } else F.overflow = 1;
    }
  }
  __syncwarp();
}

// One strong-probable-prime round on an odd n > 37 to a prime base b <= 37. No division by the base
// first: one that divides n has only multiples of itself as powers mod n, never +-1, so the round
// fails. The base's Montgomery form by doublings of 1's.
__device__ __forceinline__ bool sprp_round(const Mont &M, u32 b) {
  u64 bm = 0;
  for (int i = 5; i >= 0; --i) {
    bm = addmod(bm, bm, M.n);
    if (b >> i & 1) bm = addmod(bm, M.one, M.n);
  }
  u64 d = M.n - 1;
  const int s = __ffsll((long long)d) - 1;
  d >>= s;
  return M.n < LazyArith::NMAX ? sprp_ar<LazyArith>(bm, d, s, M) : sprp_mont(bm, d, s, M);
}

// The 12-base deterministic test (census/rung_scan.cpp:76-92) with one base per lane.
// All lanes must call; returns the same verdict in every lane.
__device__ inline bool warp_is_prime(u64 n, u32 lane) {
  bool ok = true;
  if (n < 2) return false;
  if (n <= 37) {
    bool isb = false;
    #pragma unroll
    for (int i = 0; i < 12; ++i) isb |= (n == MR_BASES[i]);
    return isb;
  }
  if (!(n & 1)) return false;
  if (lane < 12) {
    ok = sprp_round(mont_one(n), (u32)MR_BASES[lane]);
  }
  return __all_sync(FULL, ok);
}

// The primes among the 32 numbers of a warp's threads (where `valid`), as a mask in every lane: the
// base-2 round of each thread's own number, which nearly every composite fails, then the other 11
// bases of the numbers that passed, a (number, base) pair per lane, so that no lane idles while
// another's number is tested. All lanes call.
__device__ inline unsigned warp_primes(u64 n, bool valid, u32 lane) {
  bool pass = valid && n >= 2 && ((n & 1) || n == 2);
  Mont M{3, 0, 0, 0};
  if (pass && n > 37) {
    M = mont_one(n);
    pass = sprp2_round(M);
  } else if (pass) {
    pass = false;
    #pragma unroll
    for (int i = 0; i < 12; ++i) pass |= n == MR_BASES[i];
  }
  unsigned primes = __ballot_sync(FULL, pass);
  const unsigned test = __ballot_sync(FULL, pass && n > 37);
  const u32 pairs = 11 * __popc(test);
  for (u32 i0 = 0; i0 < pairs; i0 += 32) {
    const u32 i = min(i0 + lane, pairs - 1);
    unsigned m = test;
    for (u32 skip = i / 11; skip; --skip) m &= m - 1;
    const int src = __ffs(m) - 1;
    Mont Q;
    Q.n = __shfl_sync(FULL, M.n, src);
    Q.ninv = __shfl_sync(FULL, M.ninv, src);
    Q.one = __shfl_sync(FULL, M.one, src);
    Q.r2 = 0;
    const bool ok = sprp_round(Q, (u32)MR_BASES[1 + i % 11]);
    primes &= ~__reduce_or_sync(FULL, ok ? 0u : 1u << src);
  }
  return primes;
}

// Brent's backtrack from ys: step one at a time until gcd(|x - ys|, n) > 1 (bounded by the
// longest batch).
constexpr u32 RHO_BATCH_MAX_BACKTRACK = 512;
template <class Ar>
__device__ __forceinline__ u64 rho_backtrack(u64 x, u64 ys, u64 cm, u64 n, const Mont &M) {
  u64 g = 1;
  for (u32 guard = 0; g == 1 && guard <= RHO_BATCH_MAX_BACKTRACK; ++guard) {
    ys = Ar::add(Ar::mul(ys, ys, M), cm, M);
    const u64 diff = x > ys ? x - ys : ys - x;
    g = gcd64(diff ? diff : n, n);
  }
  return g;
}

// Brent's rho, one walk per lane (constants c = 1 + lane + 32j for successive tries): the
// schedule of sieve/rung_scan3.cpp:333-369 -- y -> y^2 + c in Montgomery form, products of
// |x - y| accumulated between gcds, the comparison window doubling -- with two changes that
// cannot change a result, only when a factor is found: the first window is 16 steps instead
// of 1 (every cofactor that reaches rho has all its primes above 2^16, so its cycles are far
// longer) and gcds come every 256 steps, across windows, instead of 128 (a 64-bit binary gcd costs
// as much as 25 steps here). More walks per lane would only add work: the latency-optimal split
// is one walk per lane.
// The lanes run in lockstep (one window schedule for the warp), so that the warp can stop as
// soon as any lane has a divisor, poll for one from outside every RHO_POLL steps and be cancelled
// there. A lane whose product shares all of n goes on with its next constant, and the warp then
// takes gcds within windows, where a lane can backtrack one step at a time from the batch start (as
// it does from the first for n < 2^40, whose two primes may well be met in one batch).
// Returns a nontrivial factor of the odd composite n (the same value in every lane), or 0
// when the budget ran out or the warp was cancelled. The factorization is unique, so which
// walk wins cannot change any result.
constexpr u64 RHO_R0 = 16;      // first comparison window
constexpr u64 RHO_BATCH = 256;  // steps between gcds
constexpr u64 RHO_POLL = 64;    // steps between polls

// cancel/my_k: the warp is working for rung index my_k of a block whose best certifying rung
// so far is *cancel; once that drops below my_k nothing this warp finds can matter and it stops
// (returning 0 without an error). cancel may be null.
__device__ __forceinline__ bool cancelled(const volatile int *cancel, int my_k) {
  return cancel && *cancel < my_k;
}

// A block's hard cofactors (shared memory): a warp that has to split a cofactor posts it in its own
// slot, and warps of the block with nothing else to do -- block-mates that have finished their own
// rungs, and all warps of a team that found the prime queue empty -- run rounds of elliptic curves on
// it while the owner walks rho and then curves of its own; the first divisor found ends the search
// (the owner checks it divides n). Only speed depends on the helpers.
// More curves at once on one SM pay little: two warps on a scheduler take 1.5 times as long as one for
// a step of a curve (820 and 1217 cycles) and slow the owners' rho and the other rungs as much. So
// at most CURVE_WARPS helpers, on cofactors that have outlasted rho; in a run of few primes (its
// cofactors are posted at once, and done SMs help through the board) CURVE_WARPS_FEW. Mean stage-D
// time of the 4096-window batch at 1e19 (gpu table): 0.80, 0.50, 0.46, 0.46 ms with 0, 3, 5, 8; of the
// batch over all heights 0.29, 0.32, 0.31, 0.35; of 2^34 windows at 1.8e19 in the few-primes form
// 0.27, 0.23, 0.25, 0.28 with 0, 1, 3, 8.
constexpr int BLOCK_WARPS = 16;
constexpr u32 CURVE_WARPS = 5, CURVE_WARPS_FEW = 1;
// The grid's hard cofactors (device memory, all free between runs): in a run of few primes, where
// most blocks are soon done, an owner that turns to curves posts its cofactor here too, and the done
// blocks run curves on it, one warp per scheduler.
constexpr u32 BOARD_SLOTS = 64;
struct BoardSlot {
  unsigned long long n, found;
  unsigned int state, pad;                     // 0 free, 1 being written, 2 posted
  unsigned long long pad2;
};
struct Board {
  BoardSlot *slot;                             // [BOARD_SLOTS]
  unsigned long long *sessions, *done;         // curve rounds started on it, primes finished
};
struct BlockHelp {
  Board board;                                 // slot null: not in this run
  unsigned long long n[BLOCK_WARPS], found[BLOCK_WARPS];   // the posted cofactor (0: none), a divisor of it
  unsigned int curves;                         // helpers at work
  unsigned int sessions;                       // curve rounds started by helpers (distinct sigmas)
  unsigned int working;                        // teams that may still post
};

__device__ __forceinline__ u64 ld_volatile(const unsigned long long *p) { return *(const volatile unsigned long long *)p; }
__device__ __forceinline__ u32 ld_volatile(const unsigned int *p) { return *(const volatile unsigned int *)p; }
__device__ __forceinline__ void st_volatile(unsigned long long *p, u64 v) { *(volatile unsigned long long *)p = v; }

// The lockstep walk shared by the owner and its helpers. c0: this lane's first constant,
// cstep: the distance to its next one. poll() is called by every lane between batches (warp-
// uniform) and returns a divisor handed in from outside, ~0 to stop, or 0 to go on. Ar is the
// arithmetic (es_arith.cuh): LazyArith for n < 2^62, ExactArith above.
template <class Ar, class Poll>
__device__ __forceinline__ u64 rho_walk(u64 n, const Mont &M, u64 c0, u64 cstep, u64 budget, u32 lane, Poll poll,
                                        u64 r0 = RHO_R0) {
  const u64 y0 = to_mont(2, M);
  u64 c = c0;
  u64 cm = to_mont(c, M);
  u64 y = y0, x = y0, ys = y0, q = M.one;
  u64 steps = 0, since = 0;                            // since: steps in q
  bool fine = n < 1ull << 40;                          // gcds within windows, with backtracking
  // gcd of the batch in every lane; a divisor found by any lane, or 0
  auto test = [&]() -> u64 {
    u64 mine = 0;
    bool spent = false;
    const u64 g = gcd64(q, n);
    if (g != 1) {
      if (g != n) mine = g;
      else {
        const u64 gb = fine ? rho_backtrack<Ar>(x, ys, cm, n, M) : n;
        if (gb != 1 && gb != n) mine = gb;
        else {                                          // this walk is spent: next constant
          spent = true;
          c += cstep;
          cm = to_mont(c, M);
          y = y0; x = y0; q = M.one;
        }
      }
    }
    since = 0;
    const unsigned has = __ballot_sync(FULL, mine != 0);
    fine = __any_sync(FULL, spent) || fine;
    return has ? __shfl_sync(FULL, mine, __ffs(has) - 1) : 0;
  };
  #pragma unroll 1
  for (u64 r = r0;; r <<= 1) {
    x = y;
    if (steps + 2 * r > budget) return since ? test() : 0;
    for (u64 i = 0; i < r;) {
      const u64 lim = RHO_POLL < r - i ? RHO_POLL : r - i;
      #pragma unroll 1
      for (u32 k = 0; k < (u32)lim; ++k) y = Ar::add(Ar::mul(y, y, M), cm, M);
      i += lim;
      const u64 ext = poll();
      if (ext) return ext == ~0ull ? 0 : ext;
    }
    steps += r;
    for (u64 k = 0; k < r;) {
      const u64 lim = RHO_POLL < r - k ? RHO_POLL : r - k;
      if (!since) ys = y;
      // q takes y while the next y is computed: two independent multiplies in flight
      y = Ar::add(Ar::mul(y, y, M), cm, M);
      #pragma unroll 1
      for (u32 i = 1; i < (u32)lim; ++i) {
        const u64 next = Ar::add(Ar::mul(y, y, M), cm, M);
        q = Ar::mul(q, x > y ? x - y : y - x, M);     // a closed cycle makes q = 0 mod n
        y = next;
      }
      q = Ar::mul(q, x > y ? x - y : y - x, M);
      k += lim;
      steps += lim;
      since += lim;
      if (since >= RHO_BATCH || (fine && k == r)) {
        const u64 d = test();
        if (d) return d;
      }
      const u64 ext = poll();
      if (ext) return ext == ~0ull ? 0 : ext;
    }
  }
}

// When a warp's round of curves on n may stop: its slot was withdrawn or split, its rung became
// moot, or its team is done. Null pointers ask nothing.
struct CurveStop {
  const unsigned long long *n_at, *found, *found2;
  u64 n;
  const unsigned int *busy;
  const volatile int *cancel;
  int my_k;
};

// One round of elliptic curves on n < 2^62, one per lane: lane l takes sigma0 + l. Returns the first
// divisor a lane found (the same value in every lane), or 0. Not inlined: one copy of the curve's
// code serves owners and helpers, so that it stays in the instruction cache.
static __device__ __noinline__ u64 warp_ecm(const Mont M, u64 sigma0, u32 lane, const CurveStop stop) {
  auto poll = [&]() -> bool {
    int end = 0;
    if (lane == 0)
      end = (stop.n_at && ld_volatile(stop.n_at) != stop.n) || (stop.found && ld_volatile(stop.found) != 0) || (stop.found2 && ld_volatile(stop.found2) != 0) ||
            (stop.busy && ld_volatile(stop.busy) == 0) || cancelled(stop.cancel, stop.my_k);
    return __shfl_sync(FULL, end, 0) != 0;
  };
  const u64 d = ecm_curve<LazyArith>(sigma0 + lane, M, poll);
  const unsigned has = __ballot_sync(FULL, d != 0);
  return has ? __shfl_sync(FULL, d, __ffs(has) - 1) : 0;
}

// Rho steps per lane before the owner of a cofactor turns to ECM: rho is the cheaper method for a
// prime factor below ~2^20 (its expected walk over 32 lanes is a few hundred steps), ECM above.
// 230 takes the windows of 16, 32 and 64 steps: 28 us, half a round of curves. Against 512 steps the
// 2^34 windows at 1e15 took 0.164 instead of 0.185 ms of stage D.
constexpr u64 ECM_AFTER = 230;
constexpr u32 ECM_OWNER_ROUNDS = 32;     // 1024 curves: a 31-bit factor survives them w.p. ~2e-7
constexpr u64 ECM_SIGMA_OWNER = 6;       // owner round r: sigma = 6 + 32 r + lane
constexpr u64 ECM_SIGMA_HELP = 1ull << 22;    // helper session t: sigma = 2^22 + 32 t + lane
constexpr u64 ECM_SIGMA_BOARD = 1ull << 32;   // board session t: sigma = 2^32 + 32 t + lane
constexpr u32 HELP_POLLS = 1u << 16;     // empty polls (0.5 us apart) before a helper stops
constexpr u32 BOARD_POLLS = 256;         // the same for the board
constexpr u32 HELP_ROUNDS = 1u << 12;    // curve rounds per helper and wait, at most

// A divisor of n >= 2^62 (factorization probes), without helpers: 230 rho steps in exact arithmetic, the
// owner's rounds of curves, rho again. Two 32-bit primes took 1.5 to 3 ms by rho alone (8 K
// integers of up to 64 bits 2.7 -> 1.2 ms). Out of line, and not in stage D, whose cofactors are
// below 2^62 but for the last primes below 2^64: the call put k_rung's spills from 500 to 900 bytes.
static __device__ __noinline__ u64 warp_split_exact(const Mont M, u32 lane, u64 budget, bool use_ecm,
                                                    const volatile int *cancel, int my_k) {
  bool stop = false;
  auto poll = [&]() -> u64 {
    stop = __shfl_sync(FULL, lane == 0 && cancelled(cancel, my_k) ? 1 : 0, 0) != 0;
    return stop ? ~0ull : 0;
  };
  const bool ecm = use_ecm && budget >= ECM_AFTER + ECM_ROUND_STEPS;
  u64 steps = ecm ? ECM_AFTER : budget;
  u64 f = rho_walk<ExactArith>(M.n, M, 1 + lane, 32, steps, lane, poll);
  if (!ecm) return f;
  for (u32 round = 0; !f && !stop && round < ECM_OWNER_ROUNDS && steps + ECM_ROUND_STEPS <= budget; ++round) {
    const u64 d = ecm_curve<ExactArith>(ECM_SIGMA_OWNER + 32 * (u64)round + lane, M, [&]() { return poll() != 0; });
    const unsigned has = __ballot_sync(FULL, d != 0);
    if (has) f = __shfl_sync(FULL, d, __ffs(has) - 1);
    steps += ECM_ROUND_STEPS;
  }
  if (!f && !stop && steps < budget)
    f = rho_walk<ExactArith>(M.n, M, 1 + lane + 32 * 1024, 32, budget - steps, lane, poll);
  return f;
}

// BIG: n is often 2^62 or more.
template <bool BIG>
__device__ inline u64 warp_rho(u64 n, u32 lane, volatile u64 *found, u32 *status, const volatile int *cancel = nullptr,
                               int my_k = 0, BlockHelp *bh = nullptr, u32 slot = 0, u64 budget = WARP_RHO_STEPS,
                               bool use_ecm = true) {
  const Mont M = mont_init(n);
  const bool posted = bh && n < LazyArith::NMAX;
  bool stop = false;                               // cancelled (warp-uniform)
  const bool few = bh && bh->board.slot;
  auto post = [&]() {
    if (!posted || lane) return;
    st_volatile(&bh->found[slot], 0);
    __threadfence_block();
    st_volatile(&bh->n[slot], n);
  };
  if (few) post();
  BoardSlot *far = nullptr;                        // this warp's slot on the board
  auto poll = [&]() -> u64 {
    u64 ext = 0;
    if (lane == 0) {
      if (far) {
        const u64 d = ld_volatile(&far->found);
        if (d > 1 && d < n && n % d == 0) ext = d;
      }
      if (posted && !ext) {
        const u64 d = ld_volatile(&bh->found[slot]);
        if (d > 1 && d < n && n % d == 0) ext = d;
        else if (d) st_volatile(&bh->found[slot], 0);       // of an earlier cofactor
      }
      if (!ext && cancelled(cancel, my_k)) ext = ~0ull;
    }
    ext = __shfl_sync(FULL, ext, 0);
    if (ext == ~0ull) stop = true;
    return ext;
  };
  // Brent's rho first; a cofactor it has not split goes to ECM rounds (charged against the same
  // budget), and rho resumes with fresh constants for whatever budget remains after them. Every
  // stage-D cofactor is below 2^62 (A = (p + r)/4 with p below 2^64) and takes the lazy
  // arithmetic; larger n go to warp_split_exact where there are many, else they walk rho.
  u64 f = 0;
  if (n >= LazyArith::NMAX) {
    f = BIG ? warp_split_exact(M, lane, budget, use_ecm, cancel, my_k)
            : rho_walk<ExactArith>(n, M, 1 + lane, 32, budget, lane, poll);
  } else {
    const bool ecm = use_ecm && budget >= ECM_AFTER + ECM_ROUND_STEPS;
    u64 steps = 0;
    for (u32 part = 0; !f && !stop && part < 2; ++part) {            // rho, curves, rho again
      const u64 lim = part == 0 && ecm ? ECM_AFTER : budget - steps;
      if (part == 0 || steps < budget) f = rho_walk<LazyArith>(n, M, 1 + lane + 32 * 1024 * part, 32, lim, lane, poll);
      steps += lim;
      if (!ecm) break;
      if (!few && !f && !stop && part == 0) post();
      if (few && !f && !stop && part == 0 && posted && lane == 0) {
        for (u32 j = 0; j < BOARD_SLOTS && !far; ++j) {
          BoardSlot *const b = bh->board.slot + (slot + blockIdx.x + j) % BOARD_SLOTS;
          if (atomicCAS(&b->state, 0u, 1u) != 0u) continue;
          far = b;
          st_volatile(&b->found, 0);
          st_volatile(&b->n, n);
          __threadfence();
          atomicExch(&b->state, 2u);
        }
      }
      const CurveStop cs{nullptr, posted ? &bh->found[slot] : nullptr, far ? &far->found : nullptr, n, nullptr, cancel, my_k};
      for (u32 round = 0; part == 0 && !f && !stop && round < ECM_OWNER_ROUNDS && steps + ECM_ROUND_STEPS <= budget; ++round) {
        f = warp_ecm(M, ECM_SIGMA_OWNER + 32 * (u64)round, lane, cs);
        steps += ECM_ROUND_STEPS;
        if (f) break;
        const u64 ext = poll();
        if (ext && ext != ~0ull) f = ext;
      }
    }
  }
  if (lane == 0 && far) {                          // withdraw n
    atomicExch(&far->state, 1u);
    st_volatile(&far->n, 0);
    st_volatile(&far->found, 0);
    __threadfence();
    atomicExch(&far->state, 0u);
  }
  if (lane == 0 && posted) {
    st_volatile(&bh->n[slot], 0);
    __threadfence_block();
    st_volatile(&bh->found[slot], 0);
  }
  if (lane == 0) *found = f;
  __syncwarp();
  if (!f && lane == 0 && !cancelled(cancel, my_k)) atomicOr(status, ST_RHO_BUDGET);
  return f;
}

// A warp with no rung of its own helps the block's posted cofactors until *done is zero: rounds of
// curves with sigmas of their own, the open slots in turn by session, at most CURVE_WARPS warps at a
// time, each round polling its slot every few ladder bits. `busy`: the round stops when it is zero
// too. Bounded: HELP_POLLS empty polls at most, and every round is bounded. All lanes call.
__device__ inline void warp_help(BlockHelp *bh, const unsigned int *done, const unsigned int *busy, u32 lane) {
  for (u32 idle = 0, rounds = 0; idle < HELP_POLLS && rounds < HELP_ROUNDS;) {
    if (!__shfl_sync(FULL, ld_volatile(done), 0)) return;
    // lane i looks at slot i: a cofactor not split yet, with the fewest helpers
    const u64 mine = lane < BLOCK_WARPS ? ld_volatile(&bh->n[lane]) : 0;
    unsigned open = __ballot_sync(FULL, mine && !ld_volatile(&bh->found[lane % BLOCK_WARPS]));
    u32 go = 0, ses = 0;
    if (open && lane == 0) {
      go = atomicAdd(&bh->curves, 1u) < (bh->board.slot ? CURVE_WARPS_FEW : CURVE_WARPS);
      if (go) ses = atomicAdd(&bh->sessions, 1u);
      else atomicSub(&bh->curves, 1u);
    }
    go = __shfl_sync(FULL, go, 0);
    if (!go) { ++idle; __nanosleep(500); continue; }
    ++rounds;
    ses = __shfl_sync(FULL, ses, 0);
    for (u32 skip = ses % __popc(open); skip; --skip) open &= open - 1;
    const u32 j = __ffs(open) - 1;
    const u64 n = __shfl_sync(FULL, mine, j);
    const Mont M = mont_init(n);
    const u64 d = warp_ecm(M, ECM_SIGMA_HELP + 32 * (u64)ses, lane, CurveStop{&bh->n[j], &bh->found[j], nullptr, n, busy, nullptr, 0});
    if (lane == 0) {
      if (d > 1 && d < n && n % d == 0 && ld_volatile(&bh->n[j]) == n) atomicCAS(&bh->found[j], 0ull, (unsigned long long)d);
      atomicSub(&bh->curves, 1u);
    }
    __syncwarp();
  }
}

// A warp of a block that is done helps the board's cofactors until all `total` primes are. Bounded as
// warp_help. All lanes call.
__device__ inline void warp_help_board(const Board &B, u64 total, u32 lane) {
  for (u32 idle = 0, rounds = 0; idle < BOARD_POLLS && rounds < HELP_ROUNDS;) {
    if (__shfl_sync(FULL, ld_volatile(B.done), 0) >= total) return;
    unsigned open[BOARD_SLOTS / 32];
    u32 count = 0;
    #pragma unroll
    for (u32 i = 0; i < BOARD_SLOTS / 32; ++i) {
      const BoardSlot *b = B.slot + 32 * i + lane;
      open[i] = __ballot_sync(FULL, ld_volatile(&b->state) == 2u && !ld_volatile(&b->found));
      count += __popc(open[i]);
    }
    if (!count) { ++idle; __nanosleep(500); continue; }
    ++rounds;
    u64 ses = 0;
    if (lane == 0) ses = atomicAdd(B.sessions, 1ull);
    ses = __shfl_sync(FULL, ses, 0);
    u32 skip = (u32)(ses % count), i = 0;
    while (skip >= (u32)__popc(open[i])) skip -= __popc(open[i++]);
    unsigned m = open[i];
    for (; skip; --skip) m &= m - 1;
    BoardSlot *const b = B.slot + 32 * i + (__ffs(m) - 1);
    u64 n = ld_volatile(&b->n);
    __threadfence();
    if (ld_volatile(&b->state) != 2u) n = 0;
    n = __shfl_sync(FULL, n, 0);
    if (n <= 0xFFFFFFFFull || n >= LazyArith::NMAX || !(n & 1)) continue;
    const u64 d = warp_ecm(mont_init(n), ECM_SIGMA_BOARD + 32 * ses, lane, CurveStop{&b->n, &b->found, nullptr, n, nullptr, nullptr, 0});
    if (lane == 0 && d > 1 && d < n && n % d == 0 && ld_volatile(&b->n) == n) atomicCAS(&b->found, 0ull, (unsigned long long)d);
    __syncwarp();
  }
}

// The prime factors of a cofactor v0 > 2^32 with no prime factor below 2^16 (so at most three
// of them), appended to F: primes and squares at once, anything else split by warp_rho. `composite`:
// v0 is known to be neither a prime nor a square. All lanes call. Returns false when a bound was hit
// (status says which) or on cancellation.
template <bool BIG = false>
__device__ inline bool warp_factor_cofactor(u64 v0, WarpFac &F, u32 *status, u32 lane, volatile u64 *rho_slot,
                                            const volatile int *cancel, int my_k, BlockHelp *bh, u32 slot,
                                            u64 rho_budget, bool use_ecm, bool composite) {
  u64 stack[4];
  int sp = 0;
  stack[sp++] = v0;
  for (int guard = 0; sp > 0; ++guard) {
    if (guard > 16) { if (lane == 0) atomicOr(status, ST_STACK_OVERFLOW); return false; }
    const u64 v = stack[--sp];
    if (v == 1) continue;
    if (cancel && __shfl_sync(FULL, cancelled(cancel, my_k) ? 1 : 0, 0)) return false;
    if (!composite || guard) {
      if (v <= 0xFFFFFFFFull || warp_is_prime(v, lane)) { wf_add(F, v, 1, lane); continue; }
      const u64 s = isqrt64(v);
      if (s * s == v) { wf_add(F, s, 2, lane); continue; }
    }
    const u64 d = warp_rho<BIG>(v, lane, rho_slot, status, cancel, my_k, bh, slot, rho_budget, use_ecm);
    if (d == 0) return false;                  // budget (status set) or cancelled
    if (sp + 2 > 4) { if (lane == 0) atomicOr(status, ST_STACK_OVERFLOW); return false; }
    stack[sp++] = d;
    stack[sp++] = v / d;
  }
  __syncwarp();
  if (F.overflow) { if (lane == 0) atomicOr(status, ST_FAC_OVERFLOW); return false; }
  return true;
}

// The odd primes below 2^16 dividing each rung of one prime, found for all rungs at once:
// rung k's A is A_k = floor(p/4) + 1 + k (A = (p + r)/4 with r = r0 + 4k and p + r0 = 4
// floor(p/4) + 4), so q | A_k exactly when k = -A_0 (mod q), and one residue A_0 mod q per
// prime q replaces trial division of every rung by q. The 17 primes below TD_RUNGS divide many
// rungs each and are kept as a bit mask per rung; every larger prime divides at most one of
// the 64 rungs and goes into that rung's list. Rung k then divides out only its own primes; a
// list longer than TD_LIST_CAP is marked incomplete and that rung trial-divides.
constexpr int TD_RUNGS = 64;            // rung indices 0 .. 63 (r = r0 + 4k <= RCAP)
constexpr int TD_SMALL = 17;            // odd primes below TD_RUNGS: 3 .. 61, tdp[0 .. 16]
constexpr int TD_LIST_CAP = 15;         // with TD_SMALL, at most 32: one prime per lane
struct TdSieve {                        // shared memory: a warp's in the bulk, then a team's
  u16 idx[TD_RUNGS][TD_LIST_CAP];       // indices into tdp of the primes above 61 dividing A_k
  u32 n[TD_RUNGS];                      // their count (above TD_LIST_CAP: the list is incomplete)
  u32 small[TD_RUNGS];                  // bit i: tdp[i] divides A_k, i < TD_SMALL
  uint2 qm[TD_SMALL];                   // tdp[i] and floor(2^32 / tdp[i])
  u32 rs[TD_SMALL];                     // A_0 mod tdp[i]
};

// x mod q for x < 2^32 and an odd prime q < 2^16, m = floor(2^32 / q) (Barrett: the
// quotient estimate umulhi(x, m) is low by at most one).
__device__ __forceinline__ u32 mod_q16(u32 x, u32 q, u32 m) {
  const u32 r = x - __umulhi(x, m) * q;
  return r >= q ? r - q : r;
}
__device__ __forceinline__ u32 mod_a0(u32 hi, u32 mid, u32 lo, u32 q, u32 m) {   // A0 mod q, 16 bits at a time
  u32 r = mod_q16(hi, q, m);
  r = mod_q16((r << 16) | mid, q, m);
  return mod_q16((r << 16) | lo, q, m);
}

// S for A_k = A0 + k, k < TD_RUNGS, A0 < 2^64, from tdqm[i] = {d_i, floor(2^32 / d_i)} over
// the odd primes d_i below 2^16. Each thread takes SIEVE_BATCH primes at a time, the next batch's
// table entries in flight while one is used. Every thread of the team (THREADS = TEAM_THREADS, tid
// its place, `bar` its barrier) or warp (THREADS = 32) calls; they synchronize on entry and exit.
constexpr int TEAM_WARPS = 4, TEAM_THREADS = 32 * TEAM_WARPS;
// Barrier of a team: hardware barrier `bar` over its threads.
__device__ __forceinline__ void team_sync(u32 bar) { asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(TEAM_THREADS) : "memory"); }
// In the bulk a warp sieves for its own prime too, in the place of a trial division on each of its
// rungs (2^43 integers at 1e16, 88 K primes: stage D 9.2 -> 5.2 ms with the rolled loops). 4 entries in
// flight: 8 spill (2^41 integers at 1e15 1.86 ms for 1.78), 2 are no faster than 4.
constexpr int SIEVE_BATCH = 4;
template <int THREADS>
static __device__ inline void td_sieve(u64 A0, const uint2 *__restrict__ tdqm, TdSieve &S, u32 tid, u32 bar) {
  auto sync = [&]() { if (THREADS == 32) __syncwarp(); else team_sync(bar); };
  const u32 hi = (u32)(A0 >> 32), mid = (u32)(A0 >> 16) & 0xFFFFu, lo = (u32)A0 & 0xFFFFu;
  for (u32 k = tid; k < TD_RUNGS; k += THREADS) S.n[k] = 0;
  if (tid < TD_SMALL) {
    const uint2 e = __ldg(tdqm + tid);
    S.qm[tid] = e;
    S.rs[tid] = mod_a0(hi, mid, lo, e.x, e.y);
  }
  sync();
  for (u32 k = tid; k < TD_RUNGS; k += THREADS) {   // the small primes, rung by rung
    u32 mask = 0;
    #pragma unroll
    for (int i = 0; i < TD_SMALL; ++i) {
      const uint2 e = S.qm[i];
      if (mod_q16(S.rs[i] + k, e.x, e.y) == 0) mask |= 1u << i;
    }
    S.small[k] = mask;
  }
  uint2 e[SIEVE_BATCH], nx[SIEVE_BATCH];
  auto load = [&](int i0, uint2 (&to)[SIEVE_BATCH]) {
    #pragma unroll
    for (int j = 0; j < SIEVE_BATCH; ++j) {
      const int i = i0 + j * THREADS;
      to[j] = i < NTD ? __ldg(tdqm + i) : make_uint2(1u, ~0u);       // 1: residue 0, never a listed prime
    }
  };
  load(TD_SMALL + tid, nx);
  #pragma unroll 1
  for (int i0 = TD_SMALL + tid; i0 < NTD; i0 += SIEVE_BATCH * THREADS) {
    #pragma unroll
    for (int j = 0; j < SIEVE_BATCH; ++j) e[j] = nx[j];
    load(i0 + SIEVE_BATCH * THREADS, nx);
    u32 k[SIEVE_BATCH];
    #pragma unroll
    for (int j = 0; j < SIEVE_BATCH; ++j) {
      const u32 r = mod_a0(hi, mid, lo, e[j].x, e[j].y);
      k[j] = r ? e[j].x - r : (e[j].x == 1 ? ~0u : 0u);                // q > TD_RUNGS: one rung at most
    }
    #pragma unroll
    for (int j = 0; j < SIEVE_BATCH; ++j)
      if (k[j] < (u32)TD_RUNGS) {
        const u32 s = atomicAdd(&S.n[k[j]], 1u);
        if (s < (u32)TD_LIST_CAP) S.idx[k[j]][s] = (u16)(i0 + j * THREADS);
      }
  }
  sync();
}

// Records in F the primes d (one per lane, where `hit`: x = n / d exactly, iv = d^-1 mod 2^64) with
// their full powers in n; returns the product of the inverses of those powers.
static __device__ __noinline__ u64 take_primes(WarpFac &F, bool hit, u64 x, u64 iv, u32 d, u32 lane) {
  const unsigned mask = __ballot_sync(FULL, hit);
  u64 f = 1;
  int e = 0;
  if (hit) {
    u64 m = x;
    e = 1;
    f = iv;
    #pragma unroll 1
    for (int g = 0; g < 64; ++g) {
      x = m * iv;
      if (__umul64hi(x, (u64)d)) break;
      m = x; ++e; f *= iv;
    }
  }
  const int base = F.k;
  __syncwarp();
  if (hit) {
    const int pos = base + __popc(mask & ((1u << lane) - 1));
    if (pos < MAXF) { F.pr[pos] = d; F.ex[pos] = e; }
  }
  #pragma unroll
  for (int o = 16; o; o >>= 1) f *= __shfl_xor_sync(FULL, f, o);
  __syncwarp();
  if (lane == 0) {
    const int nk = base + __popc(mask);
    if (nk > MAXF) F.overflow = 1;
    F.k = nk > MAXF ? MAXF : nk;
  }
  __syncwarp();
  return f;                                        // exact: n times it has every d^e divided out
}

// Complete factorization of n >= 1 into F (prime order as found). All lanes call.
// Returns false when a bound was hit (status says which). With hard_left, a composite
// cofactor that would need rho (no prime factor below 2^16, not a square) is not factored:
// it is left in *hard_left (0 otherwise) and F holds the other prime factors; the caller
// finishes with warp_factor_cofactor if it needs the rest.
template <bool BIG = false>
__device__ inline bool warp_factor(u64 n, WarpFac &F, const u32 *__restrict__ tdp, const u64 *__restrict__ tdi,
                                   u32 *status, u32 lane, volatile u64 *rho_slot,
                                   const volatile int *cancel = nullptr, int my_k = 0,
                                   BlockHelp *bh = nullptr, u32 slot = 0, u64 rho_budget = WARP_RHO_STEPS,
                                   bool use_ecm = true, u64 *hard_left = nullptr,
                                   const u16 *td_list = nullptr, u32 td_n = ~0u, u32 td_small = 0) {
  if (hard_left) *hard_left = 0;
  if (lane == 0) { F.k = 0; F.overflow = 0; }
  __syncwarp();
  if (n <= 1) return true;
  const int tz = __ffsll((long long)n) - 1;
  if (tz) { n >>= tz; wf_add(F, 2, tz, lane); }
  u64 cur = n;                 // n with every prime found so far divided out
  bool complete = true;        // every odd prime < 2^16 was tested
  // Blocks of TD_UNROLL chunks of 32 primes, lane i of chunk c testing prime 32c + i: n is
  // divisible by an odd prime d iff x = n * d^-1 (mod 2^64) satisfies x * d < 2^64, i.e.
  // umul64hi(x, d) == 0 (then x = n / d exactly). The table holds only d (tdp) and d^-1 (tdi),
  // 12 bytes a prime, 78 KB in all, small enough to stay in L1; the loads of the next block
  // are issued before the current block is tested, so the loop pays one load latency rather
  // than one per block. Testing primes past the point where d^2 > cur is harmless (each prime
  // is tested once, against n, and a hit is a genuine factor), so the early exit is checked
  // once per block.
  auto take = [&](bool hit, u64 x, u64 iv, u32 d) {
    if (__any_sync(FULL, hit)) cur *= take_primes(F, hit, x, iv, d, lane);   // rare: a prime below 2^16 divides n
  };
  if (td_list && td_n <= (u32)TD_LIST_CAP) {       // the block's sieve listed n's odd primes < 2^16
    const u32 ns = __popc(td_small);               // lanes [0, ns): the small ones, then the list
    bool mine = false;
    u32 i = 0;
    if (lane < ns) {
      u32 m = td_small;
      for (u32 t = 0; t < lane; ++t) m &= m - 1;
      i = (u32)(__ffs(m) - 1);
      mine = true;
    } else if (lane < ns + td_n) {
      i = (u32)td_list[lane - ns];
      mine = true;
    }
    const u64 iv = mine ? __ldg(tdi + i) : 0;
    const u32 d = mine ? __ldg(tdp + i) : 0u;
    const u64 x = n * iv;
    take(mine && __umul64hi(x, (u64)d) == 0, x, iv, d);
  } else {
  constexpr int TD_UNROLL = 8;
  u64 inv[TD_UNROLL], ninv[TD_UNROLL];
  u32 pr[TD_UNROLL], npr[TD_UNROLL];
  auto load_block = [&](int cb, u64 (&iv)[TD_UNROLL], u32 (&pv)[TD_UNROLL]) {
    #pragma unroll
    for (int j = 0; j < TD_UNROLL; ++j) {
      const int i = (cb + j) * 32 + lane;
      iv[j] = i < NTD ? __ldg(tdi + i) : 0;
      pv[j] = i < NTD ? __ldg(tdp + i) : 0;
    }
  };
  load_block(0, inv, pr);
  #pragma unroll 1
  for (int cb = 0; cb < TD_CHUNKS; cb += TD_UNROLL) {
    if (cb + TD_UNROLL < TD_CHUNKS) load_block(cb + TD_UNROLL, ninv, npr);
    const int nx = (cb + TD_UNROLL) * 32;
    #pragma unroll
    for (int j = 0; j < TD_UNROLL; ++j) {
      const int i = (cb + j) * 32 + lane;
      const u64 x = n * inv[j];
      take(i < NTD && __umul64hi(x, (u64)pr[j]) == 0, x, inv[j], pr[j]);
    }
    if (nx >= NTD) break;
    const u64 dn = __shfl_sync(FULL, (u64)npr[0], 0);   // the next block's first prime
    if (dn * dn > cur) { complete = false; break; }   // cur is 1 or prime
    if (cancel && __shfl_sync(FULL, cancelled(cancel, my_k) ? 1 : 0, 0)) return false;   // moot rung
    #pragma unroll
    for (int j = 0; j < TD_UNROLL; ++j) { inv[j] = ninv[j]; pr[j] = npr[j]; }
  }
  }
  if (cur > 1) {
    if (!complete || cur <= 0xFFFFFFFFull) {
      wf_add(F, cur, 1, lane);
    } else if (hard_left) {
      const u64 s = isqrt64(cur);
      if (warp_is_prime(cur, lane)) wf_add(F, cur, 1, lane);
      else if (s * s == cur) wf_add(F, s, 2, lane);     // s is prime: no factor of cur is below 2^16
      else *hard_left = cur;                             // needs rho: left to the caller
    } else {
      return warp_factor_cofactor<BIG>(cur, F, status, lane, rho_slot, cancel, my_k, bh, slot, rho_budget, use_ecm, false);
    }
  }
  __syncwarp();
  if (F.overflow) { if (lane == 0) atomicOr(status, ST_FAC_OVERFLOW); return false; }
  return true;
}

// 128-bit product bound: a*b <= q for a, b < 2^128, q < 2^128 (one of a, b must be below
// 2^64 for the product to fit at all).
__device__ __forceinline__ bool mul_le128(U128 a, U128 b, U128 q, U128 &out) {
  if (a.hi && b.hi) return false;
  if (a.hi) { const U128 t = a; a = b; b = t; }     // now a < 2^64
  bool over;
  out = mul128_64(b, a.lo, over);
  return !over && !lt128(q, out);
}

struct DPWarp {            // shared memory, one per warp: the DP's table and the next one, in turn
  U128 v[2][RCAP + 1];
};

// Residues modulo a rung's r (1 <= r <= RCAP) without a division per residue: Barrett
// reduction of 32-bit values with m = floor((2^32 - 1) / r) (the quotient estimate umulhi(x, m)
// is low by at most one, r = 1 and powers of two included), and 64-bit values from their
// halves with c = 2^32 mod r.
struct ModR {
  u32 r, m, c;
  __device__ __forceinline__ explicit ModR(u32 r_) : r(r_), m(0xFFFFFFFFu / r_) {
    const u32 rem = 0xFFFFFFFFu - m * r_;
    c = rem + 1 == r_ ? 0u : rem + 1;
  }
  __device__ __forceinline__ u32 mod32(u32 x) const {
    const u32 v = x - __umulhi(x, m) * r;
    return v >= r ? v - r : v;
  }
  __device__ __forceinline__ u32 mod64(u64 x) const {
    return mod32(mod32((u32)(x >> 32)) * c + mod32((u32)x));   // below RCAP^2 + RCAP < 2^32
  }
};

// Residues of the divisors of a rung, in two forms that are cheaper than the table of least divisors
// below (10 us of a rung's latency, most of it 128-bit products): `small` is the least divisor up
// to 65536 in each residue class, from the primes below 2^16 alone (p and every other prime are
// larger); `met` the classes that any divisor of q^2 lies in. Both push a class's value along its
// multiples by a prime, in shared memory.
constexpr u32 SMALL_U = 65536;

// The least divisor u <= SMALL_U of q^2 with u == target (mod r), p > SMALL_U; 0 if there is none.
__device__ inline u32 warp_small_divisor(const WarpFac &F, const ModR &R, u32 target, DPWarp &D, u32 lane) {
  u32 *v = reinterpret_cast<u32 *>(D.v[0]), *w = reinterpret_cast<u32 *>(D.v[1]);
  const u32 r = R.r;
  #pragma unroll 1
  for (u32 t = lane; t < r; t += 32) v[t] = t == (r == 1 ? 0u : 1u) ? 1u : ~0u;
  __syncwarp();
  const u64 mine = lane < (u32)F.k ? F.pr[lane] : ~0ull;
  const u32 my_res = mine < SMALL_U ? R.mod32((u32)mine) : 0u;
  for (int idx = 0; idx < F.k; ++idx) {
    const u32 pr = (u32)min(__shfl_sync(FULL, mine, idx), (u64)SMALL_U), res = __shfl_sync(FULL, my_res, idx);
    if (pr >= SMALL_U) continue;
    const int e = 2 * (int)F.ex[idx];
    #pragma unroll 1
    for (u32 t = lane; t < r; t += 32) w[t] = v[t];
    __syncwarp();
    #pragma unroll 1
    for (u32 t = lane; t < r; t += 32) {
      u32 x = v[t], s = t;
      if (x == ~0u) continue;
      #pragma unroll 1
      for (int j = 0; j < e; ++j) {
        x *= pr;                                       // below 2^16 2^16
        if (x > SMALL_U) break;
        s = R.mod32(s * res);
        atomicMin(w + s, x);
      }
    }
    __syncwarp();
    u32 *const t = v; v = w; w = t;
  }
  const u32 u = v[target];
  __syncwarp();
  return u == ~0u ? 0u : u;
}

// Whether a divisor of q^2 = (p A)^2, A's factorization complete in F, is == target (mod r). With
// target == -q, u and q^2 / u are in the class together and one of them is at most q: the least
// divisor u <= q in the class exists exactly when the class is met.
__device__ inline bool warp_class_met(u64 p, const WarpFac &F, const ModR &R, u32 target, DPWarp &D, u32 lane) {
  unsigned char *v = reinterpret_cast<unsigned char *>(D.v[0]), *w = reinterpret_cast<unsigned char *>(D.v[1]);
  const u32 r = R.r;
  #pragma unroll 1
  for (u32 t = lane; t < r; t += 32) v[t] = t == (r == 1 ? 0u : 1u);
  __syncwarp();
  const u32 my_res = R.mod64(lane < (u32)F.k ? F.pr[lane] : p);    // lane F.k <= MAXF: p
  for (int idx = 0; idx <= F.k; ++idx) {
    const u32 res = __shfl_sync(FULL, my_res, idx);
    const int e = idx < F.k ? 2 * (int)F.ex[idx] : 2;
    #pragma unroll 1
    for (u32 t = lane; t < r; t += 32) w[t] = v[t];
    __syncwarp();
    #pragma unroll 1
    for (u32 t = lane; t < r; t += 32) {
      if (!v[t]) continue;
      u32 s = t;
      #pragma unroll 1
      for (int j = 0; j < e; ++j) { s = R.mod32(s * res); w[s] = 1; }
    }
    __syncwarp();
    unsigned char *const t = v; v = w; w = t;
  }
  const bool met = v[target] != 0;
  __syncwarp();
  return met;
}

// min_div_res (sieve/rung_scan3.cpp:544-565), lanes over residue classes. Returns the
// least divisor u <= q of q^2 with u == target (mod r), or 0.
__device__ inline U128 warp_min_div_res(u64 p, const WarpFac &F, U128 q, u32 r, u32 target, DPWarp &D, u32 lane) {
  const U128 INF{~0ull, ~0ull};
  const ModR R(r);
  const u32 one = r == 1 ? 0u : 1u;              // 1 mod r
  // p's own stage: q = pA with A < p, so p^2 > q and p enters with exponent 0 or 1 -- the
  // divisors 1 and p (this one only when p is within the bound)
  const u32 pm = R.mod64(p);
  const bool p_fits = !lt128(q, U128{p, 0});
  u32 ph = 0;                                     // D.v[ph] is the current table
  #pragma unroll 1
  for (u32 t = lane; t < r; t += 32)
    D.v[0][t] = (t == one) ? U128{1, 0} : (p_fits && t == pm) ? U128{p, 0} : INF;
  __syncwarp();
  #pragma unroll 1
  for (int idx = 0; idx < F.k; ++idx) {
    const u64 pr = F.pr[idx];
    const int e = 2 * (int)F.ex[idx];
    const u32 prm = R.mod64(pr);
    u32 inv = 0;                                 // prm^-1 mod r (prm is a unit: gcd(q, r) = 1)
    #pragma unroll 1
    for (u32 base = 0; base < r; base += 32) {
      const u32 x = base + lane;
      const unsigned m = __ballot_sync(FULL, x < r && R.mod32(prm * x) == one);
      if (m) { inv = base + __ffs(m) - 1; break; }
    }
    #pragma unroll 1
    for (u32 t = lane; t < r; t += 32) {
      U128 best = INF;
      u32 s = t;
      U128 pw{1, 0};
      #pragma unroll 1
      for (int j = 0; j <= e; ++j) {
        if (j) {
          bool over;
          pw = mul128_64(pw, pr, over);
          if (over || lt128(q, pw)) break;       // pr^j > q: nothing further fits
          s = R.mod32(s * inv);
        }
        const U128 v = D.v[ph][s];
        if (v.lo == ~0ull && v.hi == ~0ull) continue;
        U128 cand;
        if (mul_le128(v, pw, q, cand) && lt128(cand, best)) best = cand;
      }
      D.v[ph ^ 1][t] = best;
    }
    __syncwarp();                                  // every lane has read D.v[ph]: swap
    ph ^= 1;
  }
  const U128 u = D.v[ph][target];
  __syncwarp();
  return (u.lo == ~0ull && u.hi == ~0ull) ? U128{0, 0} : u;
}

struct RungResult { u64 A; u32 r, k; U128 u; };

// Rung k of p's walk (the loop body of solve_rung3, sieve/rung_scan3.cpp:578-603): r = r0 + 4k
// with r0 the least positive r = -p (mod 4), A = (p + r) / 4, q = pA, and the residue the
// divisor must have, target = -q (mod r). False when the rung does not apply (r > RCAP, A = 0,
// or q not prime to r).
struct Rung { u64 A; U128 q; u32 r, target; };
__device__ __forceinline__ u32 rung_r0(u64 p) { return 4 - (u32)(p & 3); }
__device__ __forceinline__ bool rung_of(u64 p, u32 k, Rung &g) {
  const u32 r = rung_r0(p) + 4 * k;
  if (k > RCAP || r > RCAP) return false;
  const u64 A = (p >> 2) + ((u64)(p & 3) + r) / 4;
  if (!A) return false;
  const ModR R(r);
  const u32 qm = R.mod32(R.mod64(p) * R.mod64(A));
  if (r > 1 && gcd64(qm, r) != 1) return false;
  g = Rung{A, U128{p * A, __umul64hi(p, A)}, r, qm ? r - qm : 0};
  return true;
}

// min_div_res of one rung (sieve/rung_scan3.cpp:544-565): the least divisor u <= q of q^2,
// q = pA, with u == target (mod r), or u = 0 when there is none. A is factored by trial
// division first; when that leaves a composite cofactor C (prime factors all >= 65537), the
// divisors of q^2 up to 65536 are exactly those of S^2, S = A / C, so the least qualifying
// one among them -- found from S's primes alone -- is the answer whenever it exists, and C is
// factored (rho, ECM) only when it does not. The table of least divisors is made only when the
// class holds a divisor and none up to 65536. Returns false when a bound was hit or the rung was
// cancelled.
__device__ inline bool rung_divisor(u64 p, u64 A, U128 q, u32 r, u32 target, WarpFac &F, DPWarp &D,
                                    const u32 *tdp, const u64 *tdi, u32 *status, u32 lane,
                                    volatile u64 *rho_slot, const volatile int *cancel, int my_k,
                                    BlockHelp *bh, u32 slot, u64 rho_budget, bool use_ecm, U128 &u,
                                    const u16 *td_list = nullptr, u32 td_n = ~0u, u32 td_small = 0) {
  const ModR R(r);
  u64 hard = 0;
  if (p <= SMALL_U) {                                  // probes only: the scans' floors are far above
    if (!warp_factor(A, F, tdp, tdi, status, lane, rho_slot, cancel, my_k, bh, slot, rho_budget, use_ecm, nullptr,
                     td_list, td_n, td_small))
      return false;
    u = warp_min_div_res(p, F, q, r, target, D, lane);
    return true;
  }
  if (!warp_factor(A, F, tdp, tdi, status, lane, rho_slot, cancel, my_k, bh, slot, rho_budget, use_ecm, &hard, td_list,
                   td_n, td_small))
    return false;
  u = U128{warp_small_divisor(F, R, target, D, lane), 0};
  if (u.lo) return true;
  if (hard &&
      !warp_factor_cofactor(hard, F, status, lane, rho_slot, cancel, my_k, bh, slot, rho_budget, use_ecm, true))
    return false;
  if (warp_class_met(p, F, R, target, D, lane)) u = warp_min_div_res(p, F, q, r, target, D, lane);
  return true;
}

// The rung walk of one prime by one warp, rung after rung (solve_rung3,
// sieve/rung_scan3.cpp:578-603, in its own order): the throughput form of team_solve_rung
// below, for while there are more primes than warps. Returns true in every lane when a rung
// certifies p, with the result in *out (written by lane 0). use_ecm = false keeps the hard
// cofactors on rho: with every warp of the GPU busy, a round of curves costs more issue slots
// than the rho steps it saves (a 10^14-integer window at 10^16, a million primes: 108 ms of
// stage D with rho alone, 179 ms with ECM), while ECM pays in the latency-bound tail.
__device__ inline bool warp_solve_rung(u64 p, const u32 *tdp, const u64 *tdi, const uint2 *tdqm, u32 *status, WarpFac &F,
                                       DPWarp &D, TdSieve &S, volatile u64 *rho_slot, RungResult *out,
                                       u64 rho_budget = WARP_RHO_STEPS, bool use_ecm = true) {
  const u32 lane = threadIdx.x & 31;
  const u32 r0 = rung_r0(p);
  td_sieve<32>((p >> 2) + 1, tdqm, S, lane, 0);
  for (u32 k = 0; r0 + 4 * k <= RCAP; ++k) {
    Rung g;
    if (!rung_of(p, k, g)) continue;
    U128 u;
    if (!rung_divisor(p, g.A, g.q, g.r, g.target, F, D, tdp, tdi, status, lane, rho_slot, nullptr, 0, nullptr, 0,
                      rho_budget, use_ecm, u, S.idx[k], S.n[k], S.small[k]))
      return false;
    if (u.lo == 0 && u.hi == 0) continue;
    if (lane == 0) *out = RungResult{g.A, g.r, k, u};
    __syncwarp();
    return true;
  }
  return false;
}

// The rung walk of one prime by a team of four warps (solve_rung3, sieve/rung_scan3.cpp:
// 578-603). Warp w takes rung indices k = w, w+4, ... (r = r0 + 4k) in increasing order and
// stops once k passes the best certifying index found by any warp. The team first lists the odd
// primes below 2^16 of all the prime's rungs at once (td_sieve), and each rung divides out
// only its own. Returns true in every thread when some rung certifies p; the team's result is
// then in *out. F, D, rho_slot and slot are the team's four, warp0 its first slot in *bh, *busy
// the count of its warps still on their rungs.
struct Team {
  WarpFac *F;
  DPWarp *D;
  u64 *rho_slot;
  RungResult *slot, *out;
  TdSieve *S;
  int *best_k;
  unsigned int *busy;
  BlockHelp *bh;
  u32 warp0, bar;
};
__device__ inline bool team_solve_rung(u64 p, const u32 *tdp, const u64 *tdi, const uint2 *tdqm, u32 *status,
                                       const Team &T, u64 rho_budget) {
  const u32 lane = threadIdx.x & 31, tid = threadIdx.x % TEAM_THREADS, w = tid >> 5;
  if (tid == 0) {
    *T.best_k = 0x7FFFFFFF;
    *T.busy = TEAM_WARPS;
  }
  if (lane == 0) T.slot[w].k = 0x7FFFFFFF;
  team_sync(T.bar);
  td_sieve<TEAM_THREADS>((p >> 2) + 1, tdqm, *T.S, tid, T.bar);   // A_0 = floor(p/4) + 1
  const u32 r0 = rung_r0(p);
  for (u32 k = w; r0 + 4 * k <= RCAP; k += TEAM_WARPS) {
    // warp-uniform: every lane must take the same branch before the warp collectives below
    if ((int)k >= __shfl_sync(FULL, *(volatile int *)T.best_k, 0)) break;
    Rung g;
    if (!rung_of(p, k, g)) continue;
    U128 u;
    if (!rung_divisor(p, g.A, g.q, g.r, g.target, T.F[w], T.D[w], tdp, tdi, status, lane, T.rho_slot + w, T.best_k,
                      (int)k, T.bh, T.warp0 + w, rho_budget, true, u, T.S->idx[k], T.S->n[k], T.S->small[k]))
      break;
    if (u.lo == 0 && u.hi == 0) continue;
    if (lane == 0) {
      T.slot[w] = RungResult{g.A, g.r, k, u};
      atomicMin(T.best_k, (int)k);
    }
    break;
  }
  if (lane == 0) atomicSub(T.busy, 1u);           // done with this prime's rungs: help the others
  __syncwarp();
  warp_help(T.bh, T.busy, T.busy, lane);
  team_sync(T.bar);
  const int bk = *(volatile int *)T.best_k;
  bool ok = false;
  if (bk != 0x7FFFFFFF) {
    ok = true;
    if (tid == 0)
      for (int i = 0; i < TEAM_WARPS; ++i) if ((int)T.slot[i].k == bk) *T.out = T.slot[i];
  }
  team_sync(T.bar);
  return ok;
}

}  // namespace es
