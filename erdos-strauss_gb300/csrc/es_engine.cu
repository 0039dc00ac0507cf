// es_engine.cu -- the GB300 engine: device tables, the funnel kernels, and the C ABI.
//
// Data layout in HBM (resident for the engine's lifetime):
//   rho[L]            u32  lane classes mod M in wheel order
//   K0[L][ldk]        u16  per (lane, filter): the residue K0 = K mod s at which filter f
//                          kills lane l (p = rho_l + M*K), or K0_MISS; 2308 x 3752 x 2 B
//                          = 17.3 MB for the M = 2042040 table, read coalesced row by row
//   tdense            per group of 128 lanes, the rows of the dense strides: 16 bytes a row, the
//                     lanes that some filter of stride s kills at K == x (mod s) (209 KB a group,
//                     4 MB for the M = 2042040 table)
//   tlane[L]          u32  per lane, the other strides' bits 0 .. s - 1 (26 KB a lane, 60 MB)
//   mdesc             per stride with a table (densest first): s, its reduction constants, its place
//   fdesc[nf]         u32  per filter: stride s = mod/gcd(M,mod) and its Qm column
//   tdp/tde                trial-division table: 6541 odd primes < 2^16 with inverses
// Per run: window descriptors, row pieces and rows, candidate chunks, Qm[window][stride] =
// (lo / M) mod s where windows are marked by segments, the survivor list, prime/direct index lists, records and counters.
//
// Pipeline per run (one CUDA stream, replayed as a CUDA graph for batches):
//   k_rows        the windows cut into rows (one K, all lanes) and pieces of 32 rows, with each
//                 piece's place in every dense stride's table
//   k_mark_short  a lane group's dense slice in an SM's shared memory; a thread per row ORs one
//                 16-byte read per dense stride: the 0.2% of positions left become candidates
//   k_sift        the candidates against the other strides; survivors appended
//   k_prep, k_mark  the alternative for long windows: a byte map per segment in shared memory,
//                 each filter clears its progression, warp-aggregated compaction
//   k_mr          Miller-Rabin: the base-2 round by a thread per survivor, the other bases by the
//                 warp (few survivors: a warp each, one base per lane)
//   k_rung        stage D: a warp per prime while primes outnumber the grid's warps, then a
//                 team of four warps per prime over successive rungs; warp trial division,
//                 Miller-Rabin, Brent's rho, ECM rounds (es_tail.cuh, es_ecm.cuh), the rung
//                 DP, and the exact certificate check (es_check.cuh) before a record is
//                 written
//   k_search      engines without rungs: the direct search of every prime, else SURVIVOR
//   k_direct      the direct search of primes left over by rungs; the results to pinned memory
// Records come back unordered; the host puts them in (window, lane, J) order, the
// reference's lane-major order per window.
#include "../../include/es_sieve.h"
#include "es_arith.cuh"
#include "es_check.cuh"
#include "es_kernels.cuh"
#include "es_tail.cuh"
#include "es_wheel.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>
#include <chrono>
#include <cinttypes>
#include <cmath>
#include <condition_variable>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <map>
#include <mutex>
#include <string>
#include <thread>
#include <unordered_map>
#include <vector>

namespace es {

constexpr size_t CTR_BYTES = CTR_OUT * sizeof(unsigned long long) + BOARD_SLOTS * sizeof(BoardSlot);

// ============================================================================ kernels

// K0 table: for lane l and filter f, p = rho + M*K == res (mod mod) iff
// g | (res - rho) and K == ((res - rho) mod mod)/g * inv((M/g) mod s, s) (mod s).
// This is the per-(lane, filter) setup of sieve/rung_scan3.cpp:719-728 moved from the
// window's first position to K = 0, so it no longer depends on the window at all.
__global__ void k_build_k0(const u32 *__restrict__ rho, u32 L, const u64 *__restrict__ mods,
                           const u64 *__restrict__ ress, const u32 *__restrict__ gs,
                           const u32 *__restrict__ invs, const u32 *__restrict__ fdesc, u32 nf,
                           u32 ldk, u16 *__restrict__ K0) {
  const u64 idx = (u64)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (u64)L * ldk) return;
  const u32 l = (u32)(idx / ldk), f = (u32)(idx % ldk);
  if (f >= nf) { K0[idx] = K0_MISS; return; }
  const u64 mod = mods[f];
  const u64 d = (ress[f] % mod + mod - rho[l] % mod) % mod;
  const u32 g = gs[f], s = fdesc[f] & 0xFFFFu;
  if (d % g) { K0[idx] = K0_MISS; return; }
  K0[idx] = (u16)((d / g) * (u64)invs[f] % s);
}


// Clear the progression of every filter in [from, to) over alive[0, n) of one lane.
template <int BLOCK>
__device__ __forceinline__ void mark_lane(const u16 *__restrict__ K0row, const u32 *__restrict__ fdesc,
                                          const u16 *R, unsigned char *alive, u32 from, u32 to, u32 n) {
  for (u32 f = from + threadIdx.x; f < to; f += BLOCK) {
    const u32 k0 = K0row[f];
    if (k0 == K0_MISS) continue;
    const u32 fd = __ldg(fdesc + f);
    const u32 s = fd & 0xFFFFu;
    int off = (int)k0 - (int)R[fd >> 16];
    if (off < 0) off += (int)s;
    for (u32 j = (u32)off; j < n; j += s) alive[j] = 0;
  }
}

template <int BLOCK>
__device__ __forceinline__ u32 block_sum(u32 v, u32 *red) {
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
  const int wid = threadIdx.x >> 5, ln = threadIdx.x & 31;
  __syncthreads();
  if (ln == 0) red[wid] = v;
  __syncthreads();
  u32 t = 0;
  if (threadIdx.x < 32) {
    t = threadIdx.x < BLOCK / 32 ? red[threadIdx.x] : 0;
    for (int o = 16; o; o >>= 1) t += __shfl_xor_sync(0xFFFFFFFFu, t, o);
  }
  return t;   // valid in thread 0
}

struct ItemInfo {
  u64 J0;                 // position index of the segment start within each lane
  u64 first[GROUP];       // first position p of each lane in the window
  u32 n[GROUP];           // positions of each lane in this segment (0 = inactive)
  u32 lane_base, win, G, bmask, valid;
};

// Per-window residues (lo / M) mod s_d for every distinct stride: computed once per window
// here, instead of once per (window, lane) item.
// Qm[w][d] = Q_w mod s_d. A thread keeps its strides d = threadIdx.x + k blockDim over the
// block's windows, with the Barrett constant of each stride taken once: Q < 2^64 / M, so Q mod
// s for s < 2^16 is three 16-bit steps of a 32-bit reduction (the quotient estimate
// umulhi(x, m), m = floor((2^32 - 1) / s), is low by at most one).
__global__ void k_prep(const BatchHdr *__restrict__ hdr, const WinDev *__restrict__ win,
                       const u32 *__restrict__ sdist, u32 D, u32 Dq, u16 *__restrict__ Qm) {
  const u32 nwin = hdr->nwin;
  for (u32 d = threadIdx.x; d < D; d += blockDim.x) {
    const u32 sd = sdist[d], m = 0xFFFFFFFFu / sd;
    auto mod = [&](u32 x) { const u32 v = x - __umulhi(x, m) * sd; return v >= sd ? v - sd : v; };
    for (u32 w = blockIdx.x; w < nwin; w += gridDim.x) {
      const u64 Q = win[w].Q;
      u32 r = mod((u32)(Q >> 32));
      r = mod((r << 16) | ((u32)(Q >> 16) & 0xFFFFu));
      r = mod((r << 16) | ((u32)Q & 0xFFFFu));
      Qm[(size_t)w * Dq + d] = (u16)r;
    }
  }
}

// Items are dealt from an atomic queue (persistent schedule: gridDim = resident CTAs) or
// one per CTA (gridDim = items).
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK) k_mark(const MarkParams P, int persistent) {
  extern __shared__ __align__(16) unsigned char smem[];
  u16 *R0 = reinterpret_cast<u16 *>(smem);          // G = 1: R; G = GROUP: residues at K = Q
  u16 *R1 = R0 + P.D;                                // G = GROUP: residues at K = Q + 1
  unsigned char *alive = smem + P.r_bytes;
  u32 *alive32 = reinterpret_cast<u32 *>(alive);
  __shared__ ItemInfo it;
  __shared__ u32 red[BLOCK / 32];
  __shared__ u64 s_item;
  const u32 lane_id = threadIdx.x & 31;
  stamp(P.ctr, 2);
  const u64 total_items = P.hdr->total_items;
  const u32 nwin = P.hdr->nwin;
  u64 next = blockIdx.x;
  for (;;) {
    if (threadIdx.x == 0) {
      const u64 item = persistent ? atomicAdd(reinterpret_cast<unsigned long long *>(P.queue), 1ull) : next;
      s_item = item;
      it.valid = 0;
      if (item < total_items) {
        u32 lo = 0, hi = nwin;                     // last window with item0 <= item
        while (hi - lo > 1) {
          const u32 mid = (lo + hi) >> 1;
          if (P.win[mid].item0 <= item) lo = mid; else hi = mid;
        }
        const WinDev &W = P.win[lo];
        const u64 rem = item - W.item0;
        it.win = lo;
        it.G = W.G;
        it.lane_base = W.lane0 + (u32)(rem % W.groups) * W.G;
        it.J0 = (rem / W.groups) * W.seg;
        it.valid = 1;
      }
    }
    __syncthreads();
    const u64 item = s_item;
    if (item >= total_items) break;
    next += gridDim.x;
    const u32 win = it.win, G = it.G, lane_base = it.lane_base;
    const u64 J0 = it.J0;
    const WinDev &W = P.win[win];
    if (threadIdx.x < G) {
      const u32 lane = lane_base + threadIdx.x;
      u32 n = 0;
      u64 first = 0;
      bool b = false;
      if (lane < P.L) {
        const u64 rho = P.rho[lane];
        b = rho < W.lomod;
        const u64 Kfirst = W.Q + (b ? 1 : 0);
        first = rho + P.M * Kfirst;
        if (first < W.hi) {
          const u64 npos = (W.hi - first - 1) / P.M + 1;
          if (J0 < npos) n = (u32)min((u64)W.seg, npos - J0);
        }
      }
      it.n[threadIdx.x] = n;
      it.first[threadIdx.x] = first;
      const unsigned bm = __ballot_sync(0xFFFFFFFFu >> (32 - (G < 32 ? G : 32)), b);
      if (threadIdx.x == 0) it.bmask = bm;
    }
    __syncthreads();
    u32 ntot = 0;
    #pragma unroll
    for (int g = 0; g < (int)GROUP; ++g) ntot += (g < (int)G) ? it.n[g] : 0;
    if (ntot == 0) { __syncthreads(); continue; }
    // segment-start residues of K modulo every distinct stride
    const u16 *Qm = P.Qm + (size_t)win * P.Dq;
    if (G == 1) {
      const u32 b = it.bmask & 1;
      for (u32 d = threadIdx.x; d < P.D; d += BLOCK) {
        const u32 s = P.sdist[d];
        u32 r = (u32)Qm[d] + b + (J0 ? (u32)(J0 % s) : 0u);
        r = r >= s ? r - s : r;
        r = r >= s ? r - s : r;
        R0[d] = (u16)r;
      }
    } else {
      for (u32 d = threadIdx.x; d < P.D; d += BLOCK) {
        const u32 s = P.sdist[d], q = Qm[d];
        R0[d] = (u16)q;
        R1[d] = (u16)(q + 1 == s ? 0 : q + 1);
      }
    }
    // alive bytes: 1 for the segment's positions, 0 beyond
    const u32 nw = G == 1 ? (it.n[0] + 3) >> 2 : GROUP * (SEG_SMALL / 4);
    for (u32 w = threadIdx.x; w < nw; w += BLOCK) {
      const u32 g = G == 1 ? 0 : w / (SEG_SMALL / 4);
      const u32 jb = (G == 1 ? w : w % (SEG_SMALL / 4)) * 4;
      const u32 n = it.n[g];
      const u32 left = n > jb ? n - jb : 0;
      alive32[w] = left >= 4 ? 0x01010101u : (0x01010101u & ((1u << (8 * left)) - 1u));
    }
    __syncthreads();
    u32 ng[GROUP];
    #pragma unroll
    for (int g = 0; g < (int)GROUP; ++g) ng[g] = (g < (int)G) ? it.n[g] : 0;
    for (int phase = 0; phase < 2; ++phase) {
      const u32 from = phase ? P.ncov : 0, to = phase ? P.nf : P.ncov;
      if (phase) {                                  // stage B': count survivors of the covers
        if (P.nf == P.ncov) break;
        u32 c = 0;
        for (u32 w = threadIdx.x; w < nw; w += BLOCK) c += __popc(alive32[w]);
        c = block_sum<BLOCK>(c, red);
        if (threadIdx.x == 0) atomicAdd(&P.cnt[win].after_covers, (unsigned long long)c);
      }
      mark_lane<BLOCK>(P.K0 + (size_t)lane_base * P.ldk, P.fdesc, R0, alive, from, to, ng[0]);   // G == 1
      __syncthreads();
    }
    // Compaction: each warp takes 32 consecutive words per step; an inclusive warp scan of
    // the per-word popcounts gives each lane its slot, and one atomicAdd per warp reserves
    // the warp's block in the survivor list.
    u32 mine = 0;
    const u32 wid = threadIdx.x >> 5;
    for (u32 base = wid * 32; base < nw; base += BLOCK) {
      const u32 w = base + lane_id;
      u32 x = w < nw ? alive32[w] : 0u;
      const u32 c = __popc(x);
      u32 incl = c;
      #pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const u32 t = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane_id >= (u32)o) incl += t;
      }
      const u32 tot = __shfl_sync(0xFFFFFFFFu, incl, 31);
      if (tot) {
        unsigned long long gbase = 0;
        if (lane_id == 0) gbase = atomicAdd(P.surv_count, (unsigned long long)tot);
        gbase = __shfl_sync(0xFFFFFFFFu, gbase, 0);
        u64 slot = gbase + incl - c;
        const u32 g = G == 1 ? 0 : w / (SEG_SMALL / 4);
        const u32 jb = (G == 1 ? w : w % (SEG_SMALL / 4)) * 4;
        while (x) {
          const u32 k = __ffs(x) - 1;
          x &= x - 1;
          if (slot < P.surv_cap) {
            const u64 J = J0 + jb + (k >> 3);
            Surv sv;
            sv.p = it.first[g] + P.M * J;
            sv.J = J;
            sv.win = win;
            sv.lane = lane_base + g;
            P.surv[slot] = sv;
          }
          ++slot;
        }
        mine += tot;
      }
    }
    if (lane_id == 0 && mine) atomicAdd(&P.cnt[win].surv, (unsigned long long)mine);
    __syncthreads();
  }
}

// ---------------------------------------------------------------- marking by rows
// A row is one K of one window: the positions p = rho_l + M K of all lanes l (contiguous in
// integer order, so a window is a run of rows whose first and last are cut at a lane). For a
// stride s the filters kill the lanes of row K by a bit vector that depends on K mod s alone.
// Dense strides (the first n1, densest first) keep these vectors by group of GROUP_LANES lanes,
// each stride's rows 0 .. s - 1 followed by PIECE_ROWS - 1 repeats, so that the rows of a piece (at
// most PIECE_ROWS consecutive K of one window) that starts at K0 are consecutive from K0 mod s; one
// group's slice fits an SM's shared memory. The other strides keep, per lane, the bits 0 .. s - 1.

// x mod s for x < 2^32, m = floor((2^32 - 1) / s) (the quotient estimate is low by at most one)
__device__ __forceinline__ u32 mod_s(u32 x, u32 s, u32 m) {
  const u32 v = x - __umulhi(x, m) * s;
  return min(v, v - s);
}
// K mod s for d = {s, m, 2^32 mod s, ..}; wide: K may reach 2^48
__device__ __forceinline__ u32 mod_stride(u64 K, const uint4 &d, bool wide) {
  u32 hi = (u32)(K >> 32);
  if (wide) hi = mod_s(hi, d.x, d.y);
  return mod_s(hi * d.z + mod_s((u32)K, d.x, d.y), d.x, d.y);        // below 2^16 (2^16 - 1) + 2^16
}

// The run's first kernel. It reads the header and the window descriptors from pinned host memory
// itself, copies them for the kernels that follow and clears the run's counters (three memsets and
// three copies as nodes of the graph cost 12 us), and cuts the windows marked by rows into pieces:
// a block takes a run of pieces, finds their first window (32-way search over the windows' first
// pieces, which are in host memory too: as few dependent reads as possible) and goes on 32 windows
// at a time; a warp per piece writes the piece, its rows, and per dense stride the slice row of the
// piece's first K. Bound by the latency of its few dependent loads.
__global__ void __launch_bounds__(256) k_rows(const RowParams P) {
  __shared__ BatchHdr s_hdr;
  __shared__ RowWin s_win[32];
  __shared__ u32 s_first;
  const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x < sizeof(BatchHdr) / 8)
    reinterpret_cast<u64 *>(&s_hdr)[threadIdx.x] = reinterpret_cast<const volatile u64 *>(P.h_hdr)[threadIdx.x];
  __syncthreads();
  const u32 nw = s_hdr.nshort, npieces = s_hdr.npieces, nwin = s_hdr.nwin;
  const u32 tid = blockIdx.x * blockDim.x + threadIdx.x, threads = gridDim.x * blockDim.x;
  if (blockIdx.x == 0) {
    if (threadIdx.x < sizeof(BatchHdr) / 8) reinterpret_cast<u64 *>(P.hdr)[threadIdx.x] = reinterpret_cast<u64 *>(&s_hdr)[threadIdx.x];
    if (threadIdx.x == 0) *P.status = 0;
    for (u32 i = threadIdx.x; i < CTR_BYTES / 8; i += blockDim.x)
      if (i != STAMP0) P.ctr[i] = 0;
    stamp(P.ctr, 0);
  }
  for (u32 i = tid; i < nwin * (sizeof(WinCount) / 16); i += threads)
    reinterpret_cast<uint4 *>(P.cnt)[i] = make_uint4(0, 0, 0, 0);
  for (u32 i = tid; i < nwin * (sizeof(WinDev) / 8); i += threads)
    reinterpret_cast<u64 *>(P.win)[i] = reinterpret_cast<const volatile u64 *>(P.h_win)[i];
  const u32 share = (npieces + gridDim.x - 1) / gridDim.x;
  u32 pc0 = min(blockIdx.x * share, npieces);
  const u32 pc1 = min(pc0 + share, npieces);
  if (pc0 == pc1) return;
  const RowWin *hw = P.h_roww;
  auto piece0 = [&](u32 w) { return *reinterpret_cast<const volatile u32 *>(&hw[w].piece0); };
  if (warp == 0) {
    u32 w0 = 0, cnt = nw;                            // the last window whose first piece is <= pc0
    while (cnt > 1) {
      const u32 step = (cnt + 31) / 32, off = lane * step;
      const bool le = off < cnt && piece0(w0 + off) <= pc0;
      const u32 k = __popc(__ballot_sync(FULL, le)) - 1;          // lane 0 always holds
      w0 += k * step;
      cnt = min(step, cnt - k * step);
    }
    if (lane == 0) s_first = w0;
  }
  __syncthreads();
  for (u32 w0 = s_first; pc0 < pc1; w0 += 32) {
    const u32 have = min(nw - w0, 32u);
    for (u32 i = threadIdx.x; i < have * (sizeof(RowWin) / 8); i += blockDim.x)
      reinterpret_cast<u64 *>(s_win)[i] = reinterpret_cast<const volatile u64 *>(hw + w0)[i];
    __syncthreads();
    const RowWin &Z = s_win[have - 1];
    const u32 end = min(pc1, Z.piece0 + (Z.nrows + PIECE_ROWS - 1) / PIECE_ROWS);   // these windows' last piece
    const u32 mine = lane < have ? s_win[lane].piece0 : ~0u;
    for (u32 pc = pc0 + warp; pc < end; pc += blockDim.x / 32) {
      const RowWin W = s_win[__popc(__ballot_sync(FULL, mine <= pc)) - 1];
      const u32 t = pc - W.piece0;
      Piece x;
      x.K0 = W.K0 + (u64)t * PIECE_ROWS;
      x.row0 = W.row0 + t * PIECE_ROWS;
      x.win = W.wi;
      x.n = min(PIECE_ROWS, W.nrows - t * PIECE_ROWS);
      const bool last = t * PIECE_ROWS + x.n == W.nrows;
      x.la = t == 0 ? W.la : 0;
      x.lb = last ? W.lb : P.L;
      x.pad = 0;
      if (lane == 0) P.piece[pc] = x;
      if (lane < x.n) {
        const bool cut = (lane == 0 && x.la) || (lane == x.n - 1 && x.lb < P.L);
        P.rowinfo[x.row0 + lane] = pc * PIECE_ROWS + lane + (cut ? ROW_CUT : 0u);
      }
      for (u32 m = lane; m < P.n1p; m += 32) {
        const uint4 d = __ldg(P.mdesc + m);
        P.pidx[(size_t)pc * P.n1p + m] = (u16)(d.w + mod_stride(x.K0, d, P.wide));
      }
    }
    pc0 = end;
    __syncthreads();
  }
}

// Bulk copies into shared memory, and the bounded wait for them.
__device__ __forceinline__ u32 smem_addr(const void *p) { return (u32)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void bar_init(u32 bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void bar_expect(u32 bar, u32 bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_copy(u32 dst, const void *src, u32 bytes, u32 bar) {   // bytes: a multiple of 16
  for (u32 o = 0; o < bytes; o += BULK_COPY)
    asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst + o),
                 "l"((const char *)src + o), "r"(min(BULK_COPY, bytes - o)), "r"(bar)
                 : "memory");
}
// Every thread of the block waits for the barrier's phase; false (never: the copies take
// microseconds) when one gave up, with the status set and the copies waited for once more.
__device__ __forceinline__ bool bulk_wait(u32 bar, u32 parity, u32 *status) {
  auto wait = [&]() {
    u32 ok = 0;
    for (u32 i = 0; !ok && i < (1u << 20); ++i)
      asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                   : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok;
  };
  if (__syncthreads_and(wait())) return true;
  if (threadIdx.x == 0) atomicOr(status, ST_QUEUE_TIMEOUT);
  wait();
  return false;
}

// The lanes of word w of group g that have a position in the row `ri`.
__device__ __forceinline__ void row_lanes(const RowParams &P, u32 ri, u32 g, u32 (&al)[GROUP_WORDS]) {
  u32 a = 0, b = ri == ROW_NONE ? 0 : P.L;
  if (ri != ROW_NONE && (ri & ROW_CUT)) {
    const u32 j = ri % PIECE_ROWS;
    const Piece x = P.piece[(ri & ~ROW_CUT) / PIECE_ROWS];
    if (j == 0) a = x.la;
    if (j == x.n - 1) b = x.lb;
  }
  #pragma unroll
  for (u32 w = 0; w < GROUP_WORDS; ++w) {              // bits [a, b) of lanes l0 .. l0 + 31
    const u32 l0 = g * GROUP_LANES + w * 32;
    const u32 lo = a > l0 ? min(a - l0, 32u) : 0u, hi = b > l0 ? min(b - l0, 32u) : 0u;
    al[w] = lo < hi ? (~0u << lo) & (~0u >> (32 - hi)) : 0u;
  }
}

// A warp's n <= 32 candidates of group g as a chunk. Chunks past the capacity are counted only
// (the host runs again with room for them).
__device__ __forceinline__ void put_chunk(const RowParams &P, u32 g, const uint2 *buf, u32 n, u32 lane) {
  u64 id = 0;
  if (lane == 0) id = atomicAdd(P.chunk_count, 1ull);
  id = __shfl_sync(FULL, id, 0);
  if (id >= P.chunk_cap) return;
  if (lane == 0) P.chunk[id] = g << 8 | n;
  if (lane < n) P.cand[id * 32 + lane] = buf[lane];
}

// Marks the tiles (32 consecutive rows of the batch, one per thread of a warp) of every lane
// group by the dense strides. The (group, tile) items are dealt to the CTAs (one per SM) in equal
// runs, so a CTA holds one group's slice or two in turn; its warps take tiles from a counter, the
// next tile's rows loaded while one is marked. Per tile a thread ORs its row's bit vectors over the
// strides: one 16-byte shared-memory read per stride decides GROUP_LANES positions, and consecutive
// rows read consecutive words. The positions left (0.2% with the gpu table) go to k_sift in chunks
// of up to 32 of one group.
// Bound by shared-memory bandwidth: on a 2^40-integer window (1.24e9 positions) 0.257 ms at 94% of
// the LSU data pipe's peak; the 4096-window batch takes 0.052 ms. Per-lane masks of one stride per
// lane of a warp, which this replaced, took 1.9 ms and 0.83 ms with the survivors' other strides
// included. Rows of 8 bytes hold 64 strides in a slice but were bound by address arithmetic (0.47
// ms with next to no candidates left); with 16-byte rows and k_sift, 40, 48 and 56 dense strides
// (the last cut to 50 by the slice) took 0.71, 0.60 and 0.61 ms together on that window.
__global__ void __launch_bounds__(ROW_THREADS, 1) k_mark_short(const RowParams P) {
  extern __shared__ __align__(128) unsigned char rowmem[];
  __shared__ __align__(8) u64 s_bar;
  __shared__ u32 s_next;
  const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  stamp(P.ctr, 1);
  const u32 nrows = P.hdr->nrows;
  const u32 ntiles = (nrows + 31) / 32;
  const u64 items = (u64)ntiles * P.ngroups;
  u64 item = items * blockIdx.x / gridDim.x;
  const u64 end = items * (blockIdx.x + 1) / gridDim.x;
  if (item >= end) return;
  uint2 *buf = reinterpret_cast<uint2 *>(rowmem + P.slice_bytes) + warp * 64;   // fewer than 32, then at most 32 more
  const u32 bar = smem_addr(&s_bar), tab = smem_addr(rowmem);
  if (threadIdx.x == 0) bar_init(bar);
  u32 parity = 0;
  auto row_at = [&](u32 t, u32 t1) {
    const u32 row = t * 32 + lane;
    return t < t1 && row < nrows ? __ldg(P.rowinfo + row) : ROW_NONE;
  };
  while (item < end) {
    const u32 g = (u32)(item / ntiles), t0 = (u32)(item % ntiles);
    const u32 t1 = (u32)min((u64)ntiles, t0 + (end - item));
    item += t1 - t0;
    u32 al[GROUP_WORDS];
    // A run no longer than the warps may hold no position of the group at all (windows shorter
    // than M): then its slice is not needed. The barrier also ends the previous run's reads.
    bool some = true;
    u32 t = t0 + warp, ri = row_at(t, t1);
    if (t1 - t0 <= ROW_THREADS / 32) {
      row_lanes(P, ri, g, al);
      some = al[0] | al[1] | al[2] | al[3];
    }
    if (!__syncthreads_or(some)) continue;
    if (threadIdx.x == 0) {
      s_next = t0 + ROW_THREADS / 32;
      bar_expect(bar, P.slice_bytes);
      bulk_copy(tab, P.tdense + (size_t)g * P.slice_bytes, P.slice_bytes, bar);
    }
    if (!bulk_wait(bar, parity, P.status)) return;
    parity ^= 1;
    u32 nbuf = 0;                                      // candidates in the warp's buffer
    while (t < t1) {
      const u32 now = ri;
      if (lane == 0) t = atomicAdd(&s_next, 1u);
      t = __shfl_sync(FULL, t, 0);
      ri = row_at(t, t1);
      row_lanes(P, now, g, al);
      if (!__any_sync(FULL, al[0] | al[1] | al[2] | al[3])) continue;
      const u32 pj = now == ROW_NONE ? 0 : now & ~ROW_CUT, j = pj % PIECE_ROWS;
      const uint4 *ip = reinterpret_cast<const uint4 *>(P.pidx + (size_t)(pj / PIECE_ROWS) * P.n1p);
      const u32 base = tab + j * 16;
      u32 a0 = 0, a1 = 0, a2 = 0, a3 = 0;
      auto take = [&](u32 row) {
        u32 x, y, z, w;
        asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(x), "=r"(y), "=r"(z), "=r"(w) : "r"(base + row * 16));
        a0 |= x; a1 |= y; a2 |= z; a3 |= w;
      };
      uint4 nx = P.n1p ? __ldg(ip) : make_uint4(0, 0, 0, 0);
      for (u32 m = 0; m < P.n1p; m += 8) {
        const uint4 c = nx;
        if (m + 8 < P.n1p) nx = __ldg(ip + m / 8 + 1);
        take(c.x & 0xFFFFu); take(c.x >> 16);
        take(c.y & 0xFFFFu); take(c.y >> 16);
        take(c.z & 0xFFFFu); take(c.z >> 16);
        take(c.w & 0xFFFFu); take(c.w >> 16);
      }
      al[0] &= ~a0; al[1] &= ~a1; al[2] &= ~a2; al[3] &= ~a3;
      #pragma unroll
      for (u32 w = 0; w < GROUP_WORDS; ++w)
        for (unsigned who; (who = __ballot_sync(FULL, al[w] != 0));) {
          if (al[w]) {
            buf[nbuf + __popc(who & ((1u << lane) - 1))] = make_uint2(pj / PIECE_ROWS, j * GROUP_LANES + w * 32 + __ffs(al[w]) - 1);
            al[w] &= al[w] - 1;
          }
          nbuf += __popc(who);
          __syncwarp();
          if (nbuf < 32) continue;
          nbuf -= 32;
          put_chunk(P, g, buf + nbuf, 32, lane);
          __syncwarp();
        }
    }
    if (nbuf) put_chunk(P, g, buf, nbuf, lane);
    __syncwarp();
  }
}

// A position the strides so far left: lane l at K, of window win.
struct __align__(16) Cand {
  u64 K;
  u32 win, l;
};

// Kill bit of stride d = {s, m, c, first word} at K in a lane's table: NEAR, in shared memory from
// word `at` of the dynamic part on; else in L2, from word `at` of P.tlane on.
template <bool NEAR>
__device__ __forceinline__ u32 stride_kills(const RowParams &P, const uint4 &d, u64 K, size_t at) {
  extern __shared__ __align__(128) unsigned char rowmem[];
  const u32 r = mod_stride(K, d, P.wide);
  const u32 x = NEAR ? reinterpret_cast<const u32 *>(rowmem)[(u32)at + d.w + (r >> 5)] : __ldg(P.tlane + at + d.w + (r >> 5));
  return __funnelshift_r(x, 0, r) & 1u;
}

// The strides sdesc[m0, m1) against candidates c[0, N), whose tables start at word at[i], a stride
// per lane of the warp: one round of 32, which half of them die in, then four rounds at a time, the
// loads of all candidates in flight together (past m1 the last stride is read again). Returns the
// candidates of `mask` left, in every lane.
template <bool NEAR, int N>
__device__ __forceinline__ u32 strides_leave(const RowParams &P, const uint4 *sdesc, u32 m0, u32 m1, const Cand (&c)[N],
                                             const size_t (&at)[N], u32 mask, u32 lane) {
  for (u32 mb = m0; mb < m1 && mask;) {
    u32 kill[N];
    #pragma unroll
    for (int i = 0; i < N; ++i) kill[i] = 0;
    auto round = [&]() {
      const uint4 d = sdesc[min(mb + lane, m1 - 1)];
      #pragma unroll
      for (int i = 0; i < N; ++i) kill[i] |= stride_kills<NEAR>(P, d, c[i].K, at[i]);
      mb += 32;
    };
    if (mb == m0) round();
    else {
      #pragma unroll
      for (u32 r = 0; r < 4; ++r) round();
    }
    #pragma unroll
    for (int i = 0; i < N; ++i)
      if (__any_sync(FULL, kill[i])) mask &= ~(1u << i);
  }
  return mask;
}

// Whether one of the filters lfil[l0, l1) (strides with no table) kills lane l at K.
__device__ __forceinline__ bool list_kills(const RowParams &P, u32 l0, u32 l1, u64 K, u32 l, u32 lane) {
  u32 kill = 0;
  for (u32 k = l0 + lane; k < l1; k += 32) {
    const u32 f = P.lfil[k], s = P.fdesc[f] & 0xFFFFu;
    kill |= (u32)P.K0[(size_t)l * P.ldk + f] == (u32)(K % s);       // K0_MISS is no residue
  }
  return __any_sync(FULL, kill);
}

// The root of a perfect square p, else 0: a float root (off by less than 2^10 for p < 2^64) and one
// Newton step, whose error is then below 2^-12.
__device__ __forceinline__ u64 square_root(u64 p) {
  const float f = sqrtf((float)p);
  u64 s = (u64)f;
  const float d = (float)(long long)(p - s * s) / (2.0f * f);       // wraps at s = 2^32: still p - s^2
  s += (u64)(long long)rintf(d);
  return s * s == p ? s : 0;
}
// Whether p = rho_l + M K is a square that passes every cover (see k_square_mask): n is prime to
// the listed primes q (n < 2^32 is a multiple of q when n / q, as a product with q's inverse mod
// 2^32, does not exceed (2^32 - 1) / q).
__device__ __forceinline__ bool free_square(const RowParams &P, u64 K, u32 l) {
  if (!P.squares) return false;
  const u32 n = (u32)square_root(P.rho[l] + P.M * K);
  bool ok = n != 0;
  if (ok)
    for (u32 i = 0; i < P.nsq; ++i) ok = ok && n * P.sq_inv[i] > P.sq_lim[i];
  return ok;
}

// A chunk's candidate as a position.
__device__ __forceinline__ Cand cand_of(const RowParams &P, uint2 e, u32 g) {
  const Piece &x = P.piece[e.x];
  return Cand{x.K0 + e.y / GROUP_LANES, x.win, g * GROUP_LANES + e.y % GROUP_LANES};
}

// Candidates c[0, n) against the covers' strides from m0 on (those below n2 in shared memory, from
// word near[i] on), the filters without tables and stage B'; what is left is appended to the
// survivors. The whole warp calls.
constexpr int CAND_ILP = 2;
__device__ __forceinline__ void take_candidates(const RowParams &P, const uint4 *sdesc, u32 m0, u32 n2,
                                                const Cand (&c)[CAND_ILP], const size_t (&near)[CAND_ILP], int n,
                                                u32 lane) {
  u32 left = (1u << n) - 1;
  if (m0 < n2) left = strides_leave<true>(P, sdesc, m0, n2, c, near, left, lane);
  size_t far[CAND_ILP];
  #pragma unroll
  for (int i = 0; i < CAND_ILP; ++i) far[i] = (size_t)c[i].l * P.lane_words;
  left = strides_leave<false>(P, sdesc, max(m0, n2), P.nm_cov, c, far, left, lane);
  while (left) {
    const int k = __ffs(left) - 1;
    left &= left - 1;
    Cand x[1] = {c[0]};
    size_t y[1] = {far[0]};
    #pragma unroll
    for (int i = 1; i < CAND_ILP; ++i)
      if (k == i) { x[0] = c[i]; y[0] = far[i]; }
    const u64 K = x[0].K;
    const u32 l = x[0].l, win = x[0].win;
    if (P.nl_cov && list_kills(P, 0, P.nl_cov, K, l, lane)) continue;
    if (P.nm_all > P.nm_cov || P.nl_all > P.nl_cov) {                 // stage B'
      if (lane == 0) atomicAdd(&P.cnt[win].after_covers, 1ull);
      if (!strides_leave<false>(P, sdesc, P.nm_cov, P.nm_all, x, y, 1, lane)) continue;
      if (P.nl_all > P.nl_cov && list_kills(P, P.nl_cov, P.nl_all, K, l, lane)) continue;
    }
    if (lane == 0) {
      const u64 slot = atomicAdd(P.surv_count, 1ull);
      atomicAdd(&P.cnt[win].surv, 1ull);
      if (slot < P.surv_cap) {
        const WinDev &W = P.win[win];
        const u32 rho = P.rho[l];
        Surv sv;
        sv.p = rho + P.M * K;
        sv.J = K - W.Q - (rho < W.lomod ? 1 : 0);                     // lane l starts at K = Q or Q + 1
        sv.win = win;
        sv.lane = l;
        P.surv[slot] = sv;
      }
    }
  }
}

// Whether strides sdesc[m0, m1) leave a thread's candidate (where `on`; x is some position
// elsewhere), its lane's table at word `at`; the warp stops when none is left.
template <bool NEAR>
__device__ __forceinline__ bool thread_leaves(const RowParams &P, const uint4 *sdesc, u32 m0, u32 m1, const Cand &x,
                                              size_t at, bool on) {
  for (u32 m = m0; m < m1 && __any_sync(FULL, on); m += 8) {
    u32 kill = 0;
    #pragma unroll
    for (u32 i = 0; i < 8; ++i) kill |= stride_kills<NEAR>(P, sdesc[min(m + i, m1 - 1)], x.K, at);
    on = on && !kill;
  }
  return on;
}

// The candidates `left` of a warp's threads, strides below m0 done, by the whole warp.
template <bool NEAR>
__device__ __forceinline__ void take_left(const RowParams &P, const uint4 *sdesc, u32 m0, u32 n2, const Cand &x, size_t at,
                                          unsigned left, u32 lane) {
  while (left) {
    Cand c[CAND_ILP];
    size_t near[CAND_ILP];
    int n = 0;
    #pragma unroll
    for (int i = 0; i < CAND_ILP; ++i) {
      const int src = left ? __ffs(left) - 1 : 0;
      n += left != 0;
      left &= left - 1;
      c[i].K = __shfl_sync(FULL, x.K, src);
      c[i].win = __shfl_sync(FULL, x.win, src);
      c[i].l = __shfl_sync(FULL, x.l, src);
      near[i] = NEAR ? __shfl_sync(FULL, (u32)at, src) : 0;
    }
    take_candidates(P, sdesc, m0, NEAR ? n2 : 0, c, near, n, lane);
  }
}

// Whether a thread's candidate needs no test because it is a square; if so it is counted.
__device__ __forceinline__ bool take_square(const RowParams &P, const Cand &x) {
  const bool sq = free_square(P, x.K, x.l);
  if (sq) atomicAdd(&P.cnt[x.win].surv, 1ull);
  return sq;
}

// The candidates against the other strides. Up to two per warp of the grid: a warp each. Up to
// SIFT_FAR chunks: a thread each, reading the lanes' tables (60 MB) from L2, for THREAD_STRIDES[0]
// strides, then the whole warp for the quarter that is left. Beyond: the CTAs take parts of SIFT_LANES
// lanes, copy their tables to shared memory, and pick those lanes' candidates out of their
// group's chunks; where there are fewer parts than CTAs (the 120120 wheel's 220 lanes make 28), each is
// taken by several, every nslices'th 32 chunks each: marking of 2^34 and 2^40 windows with that wheel's
// table 322 us and 15.8 ms with a CTA a part, 120 us and 4.0 ms so (5.3 ms where a slice was a run of chunks,
// which lie by group). In a part a warp walks THREAD_STRIDES[0] strides when it has gathered 32, gathers what is
// left in a second buffer, walks THREAD_STRIDES[1] more when that holds 32, and takes the few that
// are left together. The lines: reading tables from L2 costs a sector per test, so beyond a few
// candidates a thread their traffic is the bound (one kernel without the shared-memory pass took 0.65
// ms on a 2^40-integer window and 0.55 ms on the 4096-window batch, against 0.60 and 0.21 ms for
// the two), while copying all lane tables costs 15 us whatever the count: a 2^34 window's 5 K part-
// filled chunks took 15 us more with them. Bound by instruction issue (58% of peak issue on the 2^40
// window: 0.35 ms for 2.3 M candidates).
constexpr u32 SIFT_FAR = 8192;
constexpr u32 THREAD_STRIDES[2] = {32, 64};
__global__ void __launch_bounds__(ROW_THREADS, 1) k_sift(const RowParams P) {
  extern __shared__ __align__(128) unsigned char rowmem[];
  __shared__ __align__(8) u64 s_bar;
  const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const u32 nchunks = (u32)min(*P.chunk_count, (unsigned long long)P.chunk_cap);
  if (!nchunks) return;
  uint4 *sdesc = reinterpret_cast<uint4 *>(rowmem + 2 * CAND_SMEM) - P.n1;              // indexed from n1
  constexpr u32 near = (2 * CAND_SMEM + STRIDES_MAX * 16) / 4;                          // the tables' first word
  for (u32 m = P.n1 + threadIdx.x; m < P.nm_all; m += ROW_THREADS) sdesc[m] = P.mdesc[P.n1p - P.n1 + m];
  const u32 warps = gridDim.x * (ROW_THREADS / 32), w0 = blockIdx.x + warp * gridDim.x;   // spread over the SMs
  __syncthreads();
  if (nchunks * 32 <= 2 * warps) {
    for (u32 i = w0; i < nchunks * 32; i += warps) {
      const u32 h = P.chunk[i / 32];
      if (i % 32 >= (h & 255u)) continue;
      const Cand x = cand_of(P, P.cand[i], h >> 8), c[CAND_ILP] = {x, x};
      const size_t none[CAND_ILP] = {};
      if (free_square(P, c[0].K, c[0].l)) {
        if (lane == 0) atomicAdd(&P.cnt[c[0].win].surv, 1ull);
        continue;
      }
      take_candidates(P, sdesc, P.n1, 0, c, none, 1, lane);
    }
    return;
  }
  if (nchunks <= SIFT_FAR) {
    const u32 m1 = min(P.n1 + THREAD_STRIDES[0], P.nm_cov);
    for (u32 i = w0; i < nchunks; i += warps) {
      const u32 h = P.chunk[i];
      bool on = lane < (h & 255u);
      Cand x{0, 0, 0};
      if (on) x = cand_of(P, P.cand[(size_t)i * 32 + lane], h >> 8);
      const size_t far = (size_t)x.l * P.lane_words;
      on = on && !take_square(P, x);
      on = thread_leaves<false>(P, sdesc, P.n1, m1, x, far, on);
      take_left<false>(P, sdesc, m1, 0, x, far, __ballot_sync(FULL, on), lane);
    }
    return;
  }
  uint2 *buf = reinterpret_cast<uint2 *>(rowmem) + warp * 128, *buf2 = buf + 64;
  const u32 bar = smem_addr(&s_bar);
  if (threadIdx.x == 0) bar_init(bar);
  u32 parity = 0;
  // the words of the strides below n2, whole 16-byte units (a lane's table is one too)
  const u32 n2 = min(P.n2, P.nm_cov);
  const u32 nwords = P.n2 < P.nm_all ? P.mdesc[P.n1p - P.n1 + P.n2].w & ~3u : P.lane_words;
  const u32 m1 = min(P.n1 + THREAD_STRIDES[0], n2), m2 = min(m1 + THREAD_STRIDES[1], n2);
  const u32 nparts = (P.L + SIFT_LANES - 1) / SIFT_LANES, nslices = max(1u, gridDim.x / nparts);
  for (u32 item = blockIdx.x; item < nparts * nslices; item += gridDim.x) {
    const u32 l0 = item % nparts * SIFT_LANES, slice = item / nparts;
    __syncthreads();                                   // the barrier's init, the previous lanes' reads
    if (threadIdx.x == 0) {
      const u32 nl = min(SIFT_LANES, P.L - l0);
      bar_expect(bar, nl * nwords * 4);
      for (u32 q = 0; q < nl; ++q)
        bulk_copy(smem_addr(rowmem) + (near + q * nwords) * 4, P.tlane + (size_t)(l0 + q) * P.lane_words, nwords * 4, bar);
    }
    if (!bulk_wait(bar, parity, P.status)) return;
    parity ^= 1;
    const u32 g = l0 / GROUP_LANES, o0 = l0 % GROUP_LANES / SIFT_LANES;
    u32 nbuf = 0, nbuf2 = 0;                           // fewer than 32, then at most 32 more
    auto load = [&](const uint2 *from, u32 n, uint2 &e, Cand &x) {
      e = make_uint2(0, 0);
      x = Cand{0, 0, l0};
      if (lane < n) { e = from[lane]; x = cand_of(P, e, g); }
      __syncwarp();
      return near + (x.l - l0) * nwords;
    };
    auto drain2 = [&](u32 n) {
      uint2 e;
      Cand x;
      nbuf2 -= n;
      const u32 at = load(buf2 + nbuf2, n, e, x);
      const bool on = thread_leaves<true>(P, sdesc, m1, m2, x, at, lane < n);
      take_left<true>(P, sdesc, m2, n2, x, at, __ballot_sync(FULL, on), lane);
    };
    auto drain = [&](u32 n) {
      uint2 e;
      Cand x;
      nbuf -= n;
      const u32 at = load(buf + nbuf, n, e, x);
      bool on = lane < n && !take_square(P, x);
      on = thread_leaves<true>(P, sdesc, P.n1, m1, x, at, on);
      const unsigned left = __ballot_sync(FULL, on);
      if (on) buf2[nbuf2 + __popc(left & ((1u << lane) - 1))] = e;
      nbuf2 += __popc(left);
      __syncwarp();
      if (nbuf2 >= 32) drain2(32);
    };
    for (u32 c0 = (warp * nslices + slice) * 32; c0 < nchunks; c0 += ROW_THREADS * nslices) {
      const u32 h = c0 + lane < nchunks ? __ldg(P.chunk + c0 + lane) : ~0u;
      unsigned mine = __ballot_sync(FULL, h >> 8 == g);
      auto entry = [&](int k) {                        // of chunk c0 + k, no lane's past its end
        const u32 n = __shfl_sync(FULL, h, k) & 255u;
        return lane < n ? __ldg(P.cand + (size_t)(c0 + k) * 32 + lane) : make_uint2(0, ~0u);
      };
      uint2 next = mine ? entry(__ffs(mine) - 1) : make_uint2(0, ~0u);
      while (mine) {
        const uint2 e = next;
        mine &= mine - 1;
        if (mine) next = entry(__ffs(mine) - 1);       // loaded while this chunk is taken
        const unsigned hit = __ballot_sync(FULL, e.y != ~0u && e.y % GROUP_LANES / SIFT_LANES == o0);
        if (hit >> lane & 1) buf[nbuf + __popc(hit & ((1u << lane) - 1))] = e;
        nbuf += __popc(hit);
        __syncwarp();
        if (nbuf >= 32) drain(32);
      }
    }
    if (nbuf) drain(nbuf);
    if (nbuf2) drain2(nbuf2);
  }
}

// The tables' bits from the first-hit table, a thread per (lane, filter) that hits: in the
// dense slices every row x == K0 (mod s) of the stride's s + PIECE_ROWS - 1, elsewhere one bit.
__global__ void k_build_rows(const u16 *__restrict__ K0, u32 L, u32 ldk, u32 nf, const int *__restrict__ fmask,
                             const uint4 *__restrict__ mdesc, u32 n1, u32 n1p, u32 slice_rows, u32 lane_words,
                             u32 *__restrict__ tdense, u32 *__restrict__ tlane) {
  const u64 idx = (u64)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (u64)L * nf) return;
  const u32 l = (u32)(idx / nf), f = (u32)(idx % nf);
  const int m = fmask[f];
  if (m < 0) return;
  const u32 k0 = K0[(size_t)l * ldk + f];
  if (k0 == K0_MISS) return;
  if ((u32)m < n1) {
    const uint4 d = mdesc[m];
    u32 *slice = tdense + (size_t)(l / GROUP_LANES) * slice_rows * GROUP_WORDS + l % GROUP_LANES / 32;
    for (u32 x = k0; x < d.x + PIECE_ROWS - 1; x += d.x) atomicOr(slice + (size_t)(d.w + x) * GROUP_WORDS, 1u << (l & 31));
  } else {
    atomicOr(tlane + (size_t)l * lane_words + mdesc[n1p - n1 + m].w + (k0 >> 5), 1u << (k0 & 31));
  }
}

// Adds to sum[0], 32 lanes a block, the share of a lane's positions that no stride of the tables kills, were
// the strides independent, and to sum[1] that of the dense strides alone: what the buffers of survivors and
// of candidates are sized by. A lane's own product and not the product of the strides' means, since lanes
// differ: few of them hold most of what is left. A warp takes every RATE_WARPS'th stride: 0.20 ms of es_open,
// latency of the reads (a thread for all of a lane's 1.4).
constexpr u32 RATE_WARPS = 16;
__global__ void k_lane_rate(const u32 *__restrict__ tdense, const u32 *__restrict__ tlane, const uint4 *__restrict__ mdesc,
                            u32 n1, u32 n1p, u32 nm, u32 slice_rows, u32 lane_words, u32 L, double *__restrict__ sum) {
  __shared__ double part[2][RATE_WARPS][32];
  const u32 lane = threadIdx.x & 31, w = threadIdx.x >> 5, l = blockIdx.x * 32 + lane;
  double r = 1, dense = 1;
  if (l < L) {
    const u32 *slice = tdense + (size_t)(l / GROUP_LANES) * slice_rows * GROUP_WORDS + l % GROUP_LANES / 32;
    for (u32 m = w; m < nm; m += RATE_WARPS) {
      const uint4 d = mdesc[m < n1 ? m : n1p - n1 + m];
      u32 c = 0;
      if (m < n1) {
        #pragma unroll 8
        for (u32 x = 0; x < d.x; ++x) c += slice[(size_t)(d.w + x) * GROUP_WORDS] >> lane & 1u;
        dense *= 1.0 - (double)c / d.x;
      } else {
        #pragma unroll 4
        for (u32 x = 0; x < (d.x + 31) / 32; ++x) c += __popc(tlane[(size_t)l * lane_words + d.w + x]);
      }
      r *= 1.0 - (double)c / d.x;
    }
  }
  part[0][w][lane] = l < L ? r : 0;
  part[1][w][lane] = l < L ? dense : 0;
  __syncthreads();
  if (w >= 2) return;                                  // a warp for each sum
  r = part[w][0][lane];
  for (u32 i = 1; i < RATE_WARPS; ++i) r *= part[w][i][lane];
  #pragma unroll
  for (int o = 16; o; o >>= 1) r += __shfl_xor_sync(FULL, r, o);
  if (lane == 0) atomicAdd(sum + w, r);
}

// Whether a filter (mod, res) can kill a perfect square: a thread per (filter, x mod mod), hits
// x^2 == res (mod mod). Such an x shares a factor g with mod, and a square n^2 that the filter kills
// has n == x, so n shares it too: its least odd prime factor q goes into `primes` as bit q. A hit
// with no such q below 64 sets bit 0: squares then get no shortcut.
__global__ void k_square_mask(const u64 *__restrict__ mods, const u64 *__restrict__ ress, u32 nf,
                              unsigned long long *__restrict__ primes) {
  for (u32 f = blockIdx.x; f < nf; f += gridDim.x) {
    const u64 mod = mods[f], res = ress[f] % mod;
    for (u64 x = threadIdx.x; x < mod; x += blockDim.x) {
      if (x * x % mod != res) continue;                // mod < 2^32
      const u64 g = gcd64(x, mod);
      u64 q = 3;
      while (q < 64 && g % q) q += 2;
      atomicOr(primes, q < 64 ? 1ull << q : 1ull);
    }
  }
}

// Miller-Rabin of the survivors (sprp2, sieve/rung_scan3.cpp:680-689, and the 12-base test,
// census/rung_scan.cpp:76-92; a prime passes base 2, so the two give exactly is_prime). Up to one warp
// a scheduler, a survivor per warp: all 12 bases at once, one per lane, for the latency of one round.
// Beyond, each warp takes several survivors, a thread each for base 2 and the warp's lanes for the
// rest (warp_primes): up to 12 while the list is short enough that latency counts (a warp's survivors
// share one round to each base pass, and 12 rarely fill a second pass of pairs), else 32.
// Integer-multiply bound on long lists. With its launch: 6 us with no survivor, 10 for 33 survivors, 18
// for the 1 K of a 2^34 window at 1e15 and 40 for the 7 K of the 4096-window batch at 1e19; two kernels
// with a list between them, which this replaced, took 9, 16, 22 and 38; with 32 a warp from the first
// the last two are 38 and 55.
constexpr u32 MR_BLOCKS_PER_SM = 6;
// Numbers a warp takes at a time, of n in all.
__device__ __forceinline__ u32 mr_share(u64 n) {
  const u64 warps = (u64)gridDim.x / MR_BLOCKS_PER_SM * 4, share = (n + warps - 1) / warps;
  return share > 48 ? 32u : (u32)min(share, 12ull);
}
// This warp's place among the grid's: the first of every block, on the schedulers in turn, then the
// second of every block and so on.
__device__ __forceinline__ u64 mr_warp() {
  const u32 turn = blockIdx.x / (gridDim.x / MR_BLOCKS_PER_SM);
  return ((threadIdx.x / 32 + 8 - turn % 8) % 8) * (u64)gridDim.x + blockIdx.x;
}
__global__ void __launch_bounds__(256, MR_BLOCKS_PER_SM) k_mr(const TailParams T) {
  const u32 lane = threadIdx.x & 31;
  const u64 warps = (u64)gridDim.x * blockDim.x / 32, w = mr_warp();
  stamp(T.ctr, 3);
  const u64 n = min((u64)*T.surv_count, T.cap);
  const u32 share = mr_share(n);
  for (u64 i0 = w * share; i0 < n; i0 += warps * share) {
    const u64 i = i0 + lane;
    const bool valid = lane < share && i < n;
    const unsigned m = share == 1 ? (u32)warp_is_prime(T.surv[i0].p, lane) : warp_primes(valid ? T.surv[i].p : 0, valid, lane);
    if (!m) continue;
    unsigned long long k = 0;
    if (lane == 0) k = atomicAdd(T.prime_count, (unsigned long long)__popc(m));
    k = __shfl_sync(FULL, k, 0) + __popc(m & ((1u << lane) - 1));
    if ((m >> lane & 1) && k < T.cap) T.primes[k] = (u32)i;
  }
}

__device__ __forceinline__ void put_record(const TailParams &T, const RecDev &r) {
  const unsigned long long k = atomicAdd(T.rec_count, 1ull);
  if (k < T.cap) T.recs[k] = r;
}

// Shared memory of a stage-D block of TEAMS teams.
template <int TEAMS, int SIEVES = TEAMS>
struct RungShared {
  WarpFac F[TEAMS * TEAM_WARPS];
  DPWarp D[TEAMS * TEAM_WARPS];
  u64 rho_slot[TEAMS * TEAM_WARPS];
  RungResult slot[TEAMS * TEAM_WARPS], out[TEAMS];
  TdSieve tds[SIEVES];                             // a team's: its first warp's, which has a prime of its own first
  BlockHelp help;
  unsigned long long next[TEAMS];
  int best_k[TEAMS];
  unsigned int busy[TEAMS];
  __device__ Team team(int t) {
    return Team{F + TEAM_WARPS * t, D + TEAM_WARPS * t, rho_slot + TEAM_WARPS * t, slot + TEAM_WARPS * t, out + t,
                tds + SIEVES / TEAMS * t, best_k + t, busy + t, &help, (u32)(TEAM_WARPS * t), (u32)t + 1};
  }
  __device__ void init() {                         // every thread calls; the caller synchronizes
    for (u32 i = threadIdx.x; i < sizeof(BlockHelp) / 4; i += blockDim.x) reinterpret_cast<u32 *>(&help)[i] = 0;
  }
};
constexpr int RUNG_TEAMS = BLOCK_WARPS / TEAM_WARPS, RUNG_THREADS = 32 * BLOCK_WARPS;
typedef RungShared<RUNG_TEAMS, BLOCK_WARPS> RungBlock;
// Every fourth block stays to help the board when it is done: all of them keep their SMs from the next
// batch's marking (three pipelined batches at 1e19 1.26-1.36 ms against 1.48-1.60 with every block and
// 1.33-1.51 with none; a 2^34 window at 1.8e19 with the tuned table 0.29-0.35, 0.28-0.35, 0.34-0.40).
constexpr u32 BOARD_BLOCKS_DIV = 4;
constexpr u32 FEW_PRIMES_PER_BLOCK = 2;        // up to two a block: the board is on (4 measured the same)

// Stage D, in blocks of four teams of four warps (one block per SM resident). While more primes
// remain than the grid has warps, every warp takes a prime of its own from a queue and walks its
// rungs in order (warp_solve_rung: no barrier, no speculative rungs); the last gridDim.x *
// BLOCK_WARPS primes go to teams that try four rungs of one prime at a time (team_solve_rung), so
// that the run ends on short latencies. The later teams of a block come to the queue a little
// later, so that few primes have an SM each. A team that finds the queue empty turns its warps into
// helpers on the block's hard cofactors until the block's other teams are done.
__device__ __forceinline__ void rung_result(const TailParams &T, const Surv &s, u32 si, bool ok,
                                            const RungResult &res) {
  if (ok && !check_rung_cert(s.p, res.A, res.r, res.u)) {
    atomicOr(T.status, ST_CERT_BAD);                // never emitted
  } else if (ok) {
    RecDev rec{ES_REC_RUNG, s.win, s.lane, 0, s.J, s.p, res.A, res.r, res.u.lo, res.u.hi};
    put_record(T, rec);
    atomicAdd(&T.cnt[s.win].rung, 1ull);
  } else {
    const unsigned long long k = atomicAdd(T.direct_count, 1ull);
    if (k < T.cap) T.direct[k] = si;
  }
  __threadfence();
  atomicAdd(T.rung_done, 1ull);
}

__global__ void __launch_bounds__(RUNG_THREADS, 1) k_rung(const TailParams T, int no_rung) {
  extern __shared__ __align__(16) unsigned char rungmem[];
  RungBlock &H = *reinterpret_cast<RungBlock *>(rungmem);
  stamp(T.ctr, 4);
  const u64 n = min((u64)*T.prime_count, T.cap);
  if (!n) return;
  const u32 lane = threadIdx.x & 31, w = threadIdx.x >> 5, t = w / TEAM_WARPS;
  const u64 tail = min(n, (u64)gridDim.x * BLOCK_WARPS);
  const u64 nw = n - tail;                           // primes [0, nw): a warp each
  H.init();
  const bool few = n <= FEW_PRIMES_PER_BLOCK * (u64)gridDim.x;
  const Board board{few ? T.board : nullptr, T.help_sessions, T.rung_done};
  __syncthreads();
  if (threadIdx.x == 0) {
    H.help.working = RUNG_TEAMS;
    H.help.board = board;
  }
  __syncthreads();
  for (;;) {
    u64 i = nw;
    if (nw && lane == 0) i = atomicAdd(T.rung_next_warp, 1ull);
    i = __shfl_sync(0xFFFFFFFFu, i, 0);
    if (i >= nw) break;
    const u32 si = T.primes[i];
    const Surv s = T.surv[si];
    const bool ok = !no_rung && warp_solve_rung(s.p, T.tdp, T.tdi, T.tdqm, T.status, H.F[w], H.D[w], H.tds[w], H.rho_slot + w,
                                                &H.slot[w], T.rho_budget, /*use_ecm=*/false);
    if (lane == 0) rung_result(T, s, si, ok, H.slot[w]);
    __syncwarp();
  }
  const Team team = H.team(t);
  const bool first = threadIdx.x % TEAM_THREADS == 0;
  __nanosleep(1500 * t);
  for (;;) {                                         // primes [nw, n): a team each
    if (first) H.next[t] = nw + atomicAdd(T.rung_next, 1ull);
    team_sync(team.bar);
    const u64 i = H.next[t];
    if (i >= n) break;
    const u32 si = T.primes[i];
    const Surv s = T.surv[si];
    const bool ok = !no_rung && team_solve_rung(s.p, T.tdp, T.tdi, T.tdqm, T.status, team, T.rho_budget);
    if (first) rung_result(T, s, si, ok, *team.out);
    team_sync(team.bar);
  }
  if (first) atomicSub(&H.help.working, 1u);
  __syncwarp();
  if (no_rung) return;
  warp_help(&H.help, &H.help.working, nullptr, lane);
  if (few && t == 0 && blockIdx.x % BOARD_BLOCKS_DIV == 0) warp_help_board(board, n, lane);
}

// The direct search of one prime that no rung certified.
__device__ __forceinline__ void direct_one(const TailParams &T, u64 i) {
  const Surv s = T.surv[T.direct[i]];
  u64 a, c, d, k;
  if (solve_direct(s.p, a, c, d, k, T.tdp, T.tde, T.status)) {
    if (!check_solved_cert(s.p, a, c, d, k)) { atomicOr(T.status, ST_CERT_BAD); return; }
    RecDev rec{ES_REC_SOLVED, s.win, s.lane, 0, s.J, s.p, a, c, d, k};
    put_record(T, rec);
    atomicAdd(&T.cnt[s.win].direct, 1ull);
  } else {
    RecDev rec{ES_REC_SURVIVOR, s.win, s.lane, 0, s.J, s.p, 0, 0, 0, 0};
    put_record(T, rec);
    atomicAdd(&T.cnt[s.win].unsolved, 1ull);
  }
}

// The direct search of an engine without rungs (ES_FLAG_NO_RUNG), where every prime takes it: a prime a warp
// while there are warps, then as many lanes of each as it takes. Bound by the latency of one thread's trial
// divisions and rho, and lanes of a warp that part company wait for each other: with 32 to a warp the 2^34
// windows of the 120120 table at 1e9, 1e12 and 1e15 take 13.3, 26.6 and 26.6 ms, with 4 12.0, 24.3 and 23.6,
// with one 10.5, 21.5 and 20.8. A kernel of its own because the search in k_direct's blocks of 256 compiles
// to a slower chain: 4 primes at 1e12 11.7 ms there, 8.9 here.
__global__ void k_search(const TailParams T) {
  stamp(T.ctr, 5);
  const u64 n = min((u64)*T.direct_count, T.cap);
  const u32 share = (u32)min((n + gridDim.x - 1) / gridDim.x, 32ull);
  if (threadIdx.x >= share) return;
  for (u64 i = (u64)blockIdx.x * share + threadIdx.x; i < n; i += (u64)gridDim.x * share) direct_one(T, i);
}

// The run's last kernel: the direct search, a thread per prime that no rung certified (none in
// scans; `searched`: k_search has done it), then the run's counters, the windows' counters and the records
// written to pinned host memory (four copies as nodes of the graph cost 8 us, and a fifth with a second
// wait brought the records past the first 4096). Without direct primes every block writes its share at
// once; else the last block to finish them writes all.
__global__ void __launch_bounds__(256) k_direct(const TailParams T, int searched) {
  __shared__ bool s_last;
  if (!searched) stamp(T.ctr, 5);
  const u64 n = searched ? 0 : min((u64)*T.direct_count, T.cap);
  u32 block = blockIdx.x, blocks = gridDim.x;
  if (n) {
    for (u64 i = (u64)threadIdx.x * gridDim.x + blockIdx.x; i < n; i += (u64)gridDim.x * blockDim.x) direct_one(T, i);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(T.ctr + 5, 1ull) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    block = 0; blocks = 1;
  }
  const u64 threads = (u64)blocks * blockDim.x, first = (u64)block * blockDim.x + threadIdx.x;
  const u64 nrec = min((u64)__ldcg(T.rec_count), T.cap), nwin = T.hdr->nwin;
  const uint4 *cnt = reinterpret_cast<const uint4 *>(T.cnt), *recs = reinterpret_cast<const uint4 *>(T.recs);
  for (u64 i = first; i < nwin * (sizeof(WinCount) / 16); i += threads) reinterpret_cast<uint4 *>(T.out.cnt)[i] = __ldcg(cnt + i);
  for (u64 i = first; i < nrec * (sizeof(RecDev) / 16); i += threads) reinterpret_cast<uint4 *>(T.out.recs)[i] = __ldcg(recs + i);
  if (block == 0) {
    if (threadIdx.x == 0) { *T.out.status = __ldcg(T.status); }
    __syncthreads();
    if (threadIdx.x == 0) {
      unsigned long long t;
      asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
      T.ctr[STAMP0 + 6] = t;
    }
    __syncthreads();
    if (threadIdx.x < CTR_OUT) T.out.ctr[threadIdx.x] = __ldcg(T.ctr + threadIdx.x);
  }
}

// ---------------------------------------------------------------- probe kernels
// Exact re-check of caller records (es_check_records): ok[i] = 1 for a RUNG or SOLVED
// record whose identity holds, 0 otherwise (SURVIVOR and unknown kinds included).
__global__ void k_probe_check(const RecDev *r, u64 count, unsigned char *ok) {
  for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (u64)gridDim.x * blockDim.x) {
    const RecDev x = r[i];
    bool good = false;
    if (x.kind == ES_REC_RUNG) good = check_rung_cert(x.p, x.a, x.b, U128{x.c, x.d});
    else if (x.kind == ES_REC_SOLVED) good = check_solved_cert(x.p, x.a, x.b, x.c, x.d);
    ok[i] = good;
  }
}

// As k_mr: 200 K odd numbers take 0.13 ms, 1.25 ms with a warp each.
__global__ void __launch_bounds__(256, MR_BLOCKS_PER_SM) k_probe_prime(const u64 *n, u64 count, unsigned char *out) {
  const u32 lane = threadIdx.x & 31;
  const u64 warps = (u64)gridDim.x * blockDim.x / 32, w = mr_warp();
  const u32 share = mr_share(count);
  for (u64 i0 = w * share; i0 < count; i0 += warps * share) {
    const u64 i = i0 + lane;
    const bool valid = lane < share && i < count;
    const unsigned m = share == 1 ? (u32)warp_is_prime(n[i0], lane) : warp_primes(valid ? n[i] : 0, valid, lane);
    if (valid) out[i] = m >> lane & 1;
  }
}
__global__ void __launch_bounds__(TEAM_THREADS, 4) k_probe_rung(const u64 *p, u64 count, RecDev *out,
                                                               unsigned char *found, const u32 *tdp,
                                                               const u64 *tdi, const uint2 *tdqm, u32 *status,
                                                               u64 rho_budget) {
  __shared__ RungShared<1> H;
  H.init();
  __syncthreads();
  const Team team = H.team(0);
  for (u64 i = blockIdx.x; i < count; i += gridDim.x) {
    bool ok = team_solve_rung(p[i], tdp, tdi, tdqm, status, team, rho_budget);
    if (threadIdx.x == 0) {
      const RungResult &res = *team.out;
      if (ok && !check_rung_cert(p[i], res.A, res.r, res.u)) { atomicOr(status, ST_CERT_BAD); ok = false; }
      found[i] = ok;
      out[i] = ok ? RecDev{ES_REC_RUNG, 0, 0, 0, 0, p[i], res.A, res.r, res.u.lo, res.u.hi}
                  : RecDev{0, 0, 0, 0, 0, p[i], 0, 0, 0, 0};
    }
    __syncthreads();
  }
}
__global__ void k_probe_direct(const u64 *p, u64 count, RecDev *out, unsigned char *found,
                               const u32 *tdp, const TdEntry *tde, u32 *status) {
  for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (u64)gridDim.x * blockDim.x) {
    u64 a, c, d, k;
    bool ok = solve_direct(p[i], a, c, d, k, tdp, tde, status);
    if (ok && !check_solved_cert(p[i], a, c, d, k)) { atomicOr(status, ST_CERT_BAD); ok = false; }
    found[i] = ok;
    out[i] = ok ? RecDev{ES_REC_SOLVED, 0, 0, 0, 0, p[i], a, c, d, k} : RecDev{0, 0, 0, 0, 0, p[i], 0, 0, 0, 0};
  }
}
// The production factorization (warp_factor), one warp per value; primes sorted ascending. A block's
// warps take its values (every gridDim-th) as they come free, and one that finds none left runs
// curves for the others' cofactors, as stage D's do: 8 K integers of up to 62 bits 585 -> 435 us, 16 of
// them 281 -> 148.
struct FactorShared {
  WarpFac F[BLOCK_WARPS];
  u64 rho_slot[BLOCK_WARPS];
  BlockHelp help;
  unsigned int next;
};
__global__ void __launch_bounds__(RUNG_THREADS, 1) k_probe_factor(const u64 *n, u64 count, u64 *pr, unsigned char *ex,
                                                                  unsigned char *k, const u32 *tdp, const u64 *tdi,
                                                                  u32 *status, u64 rho_budget) {
  __shared__ __align__(16) FactorShared H;
  const u32 lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (u32 i = threadIdx.x; i < sizeof(BlockHelp) / 4; i += blockDim.x) reinterpret_cast<u32 *>(&H.help)[i] = 0;
  __syncthreads();
  if (threadIdx.x == 0) { H.help.working = BLOCK_WARPS; H.next = 0; }
  __syncthreads();
  for (;;) {
    u32 j = 0;
    if (lane == 0) j = atomicAdd(&H.next, 1u);
    const u64 i = blockIdx.x + (u64)gridDim.x * __shfl_sync(FULL, j, 0);
    if (i >= count) break;
    WarpFac &f = H.F[w];
    const bool ok = warp_factor<true>(n[i], f, tdp, tdi, status, lane, H.rho_slot + w, nullptr, 0, &H.help, w, rho_budget);
    const u32 kk = ok ? (u32)f.k : 0;
    const bool mine = lane < kk;
    const u64 p = mine ? f.pr[lane] : 0;
    u32 at = lane;                                   // an empty place, or the prime's rank
    if (mine) {
      at = 0;
      for (u32 b = 0; b < kk; ++b) at += f.pr[b] < p || (f.pr[b] == p && b < lane);
    }
    if (lane < (u32)MAXF) {
      pr[i * MAXF + at] = p;
      ex[i * MAXF + at] = mine ? (unsigned char)f.ex[lane] : 0;
    }
    if (lane == 0) k[i] = (unsigned char)kk;
    __syncwarp();
  }
  if (lane == 0) atomicSub(&H.help.working, 1u);
  __syncwarp();
  warp_help(&H.help, &H.help.working, nullptr, lane);
}

// ============================================================================ host engine

constexpr int MARK_BLOCK = 128;
}  // namespace es

namespace es {
// Everything one run needs besides the resident tables: a stream, its events, the per-run
// device buffers and their pinned host staging, and the captured graph. An engine has one
// slot for its synchronous calls and SERVE_SLOTS more for the serving workers, so that
// several batches can be in flight on their own streams.
struct RecKey {                         // a record's place in its window
  u64 J;
  u32 lane, idx;
  bool operator<(const RecKey &o) const { return lane != o.lane ? lane < o.lane : J < o.J; }
};
struct Slot {
  cudaStream_t stream = nullptr;
  cudaEvent_t ev[12] = {};
  BatchHdr *d_hdr = nullptr, *h_hdr = nullptr;
  WinDev *h_win = nullptr;
  RowWin *h_roww = nullptr;
  WinCount *h_cnt = nullptr;
  unsigned long long *h_ctr = nullptr;
  u32 *h_status = nullptr;
  RecDev *h_recs = nullptr;
  // The persistent schedule, captured once per capacity. A serving slot has two graphs, the front
  // (marking, Miller-Rabin) and the tail (stage D, stage E, results written out). ev[11] is
  // recorded between them on the slot's stream: the next slot's front waits for it (marking runs
  // one batch at a time, in launch order) while this slot's tail overlaps the next batch's
  // marking. The synchronous slot has one graph of both, ev[11] recorded inside.
  cudaGraph_t graph = nullptr, graph2 = nullptr;
  cudaGraphExec_t gexec = nullptr, gexec2 = nullptr;
  WinDev *d_win = nullptr; size_t win_cap = 0;
  WinCount *d_cnt = nullptr;
  Piece *d_piece = nullptr; u16 *d_pidx = nullptr; u32 *d_rowinfo = nullptr; size_t piece_cap = 0;
  uint2 *d_cand = nullptr; u32 *d_chunk = nullptr; size_t chunk_cap = 0;
  u16 *d_Qm = nullptr; size_t qm_cap = 0;
  Surv *d_surv = nullptr;
  u32 *d_primes = nullptr, *d_direct = nullptr;
  RecDev *d_recs = nullptr;
  size_t cap = 0;
  u64 graph_launches = 0;               // its kernels
  unsigned long long *d_ctr = nullptr;  // run counters (es_kernels.cuh) and stage D's board
  u32 *d_status = nullptr;
  unsigned char *d_probe = nullptr; size_t probe_cap = 0;
  es_timing_t timing{};
  struct HostScratch {                  // per-run host vectors, kept with their capacity
    std::vector<WinDev> wd;
    std::vector<RowWin> roww;
    std::vector<u64> npos;
    std::vector<RecDev> hr;             // the plain schedule's records, unordered
    std::vector<RecKey> key, bin;       // order_records
    std::vector<u32> start, pos, bstart;
    std::vector<es_window> dw;          // runs in passes (run_windows)
    std::vector<std::pair<u32, u64>> dmap;
    std::vector<es_counters> pc;
    std::vector<RecDev> all;            // and their records
  } hs;
  std::mutex mu;                        // one run at a time per slot
};

constexpr int SERVE_SLOTS = 2;
// A serving request: windows in, counters and records out.
struct Request {
  uint64_t ticket = 0;
  std::vector<es_window> w;
  std::vector<es_counters> cnt;
  std::vector<es_record> recs;
  es_status st = ES_OK;
  std::string err;
  bool done = false;
  bool claimed = false;                 // an es_poll is waiting on it (one poller per ticket)
  bool solo = false;                    // es_submit_batch: runs as a batch of its own
  u64 mem = 0;                          // admitted device-memory estimate
};
}  // namespace es

struct es_engine {
  // configuration and derived tables
  es::u64 M = 0, mmax = 0, sieve_p = 0;
  uint32_t flags = 0;
  std::vector<es::u64> classes;
  // host arithmetic on window bounds: classes below residue x are lane_at[x >> LANE_BLOCK_BITS]
  // plus the few classes of x's block that lie below x; inv_M estimates division by M
  std::vector<uint32_t> lane_at;
  double inv_M = 0;
  es::u64 wheel_pmin = 0, cover_pmax = 0, class_fnv = 0, filter_fnv = 0;
  const es::ClassPin *pin = nullptr;
  std::vector<es::u64> mods, ress;     // certified filters [0,ncov) then stage-B' primes
  size_t ncov = 0;
  // marking order: filters sorted by stride within each phase
  std::vector<uint32_t> order;
  uint32_t nf = 0, ldk = 0, D = 0, Dq = 0;
  es_schedule sched{es::SEG_SMALL, 6, 1, {0, 0, 0, 0, 0}};   // es_set_schedule / es_autotune
  es::u64 rho_budget = es::WARP_RHO_STEPS;                      // ES_FLAG_TEST_RHO_BUDGET: 64
  int device = 0, sm_count = 0, mark_occupancy = 0;
  // resident device tables
  es::u32 *d_rho = nullptr, *d_fdesc = nullptr, *d_sdist = nullptr, *d_tdp = nullptr;
  es::u16 *d_K0 = nullptr;
  // the row tables: dense slices by lane group, the other strides' rows, the strides' descriptors
  // ([0, n1) dense, padded to n1p, then the others), the filters of the strides without rows
  unsigned char *d_tdense = nullptr;
  es::u32 *d_tlane = nullptr;
  uint4 *d_mdesc = nullptr;
  es::u32 *d_lfil = nullptr;
  bool squares = false;                 // see RowParams
  std::vector<uint32_t> sq;             // the primes a root has to avoid
  es::u64 pass_rows = 0;                // rows a run marks at a time (run_windows)
  double surv_rate = 0;                 // survivors per position, estimated (k_lane_rate)
  double cand_rate = 0;                 // candidates per position after the dense strides, estimated
  uint32_t lane_words = 0, n2 = 0, ngroups = 0, n1 = 0, n1p = 0, slice_rows = 0, nm_cov = 0, nm_all = 0, nl_cov = 0, nl_all = 0;
  es::TdEntry *d_tde = nullptr;
  es::u64 *d_tdi = nullptr;
  uint2 *d_tdqm = nullptr;              // {d, floor(2^32 / d)} for the same primes
  // slot 0: es_run_window / es_run_batch / probes; slots 1..SERVE_SLOTS: serving workers
  es::Slot slots[1 + es::SERVE_SLOTS];
  std::string last_error;
  std::mutex err_mu;
  // serving
  size_t mem_budget = 0;
  std::mutex qmu;
  std::condition_variable qcv, dcv;
  std::deque<es::Request *> queue;
  std::map<uint64_t, es::Request *> reqs;
  uint64_t next_ticket = 1;
  es::u64 mem_in_use = 0;
  size_t queued_windows = 0;
  int pollers = 0;                      // es_poll calls inside the engine (es_close waits for them)
  std::vector<std::thread> workers;
  bool stopping = false;
  // persistent runs of every slot: the slot whose front graph was launched last (its ev[11]
  // marks the end of that front), so that fronts run one after another in launch order
  std::mutex front_mu;
  es::Slot *last_front = nullptr;
};

namespace es {

static es_status fail(es_engine *e, es_status s, const std::string &msg) {
  if (e) { std::lock_guard<std::mutex> lk(e->err_mu); e->last_error = msg; }
  return s;
}

// The failure is this call's alone: the runtime forgets it, or the next call would take it for one
// of its own launches'.
#define CU(call)                                                                           \
  do {                                                                                     \
    cudaError_t err_ = (call);                                                             \
    if (err_ != cudaSuccess) {                                                             \
      cudaGetLastError();                                                                  \
      return fail(e, ES_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(err_));   \
    }                                                                                      \
  } while (0)

static void drop_graph(Slot *sl) {
  if (sl->gexec) cudaGraphExecDestroy(sl->gexec);
  if (sl->graph) cudaGraphDestroy(sl->graph);
  if (sl->gexec2) cudaGraphExecDestroy(sl->gexec2);
  if (sl->graph2) cudaGraphDestroy(sl->graph2);
  sl->gexec = sl->gexec2 = nullptr;
  sl->graph = sl->graph2 = nullptr;
}

// Capacities go in doublings from a floor, so that calls a little larger than the last do not each make
// their own buffers and graph: 24 windows from 2^28 integers on, each 5% longer than the last, took 8.9 ms
// (120120 wheel) and 8.3 (gpu table) with exact sizes for chunks and windows and a quarter of slack for
// pieces, 4.7 and 4.4 so; 40 batches of 100 to 880 windows 41.7 and 35.2.
static size_t grown(size_t need, size_t floor) {
  while (floor < need) floor <<= 1;
  return floor;
}

// Device buffers for nwin windows, npieces row pieces, nchunks candidate chunks and a survivor
// capacity of cap, with their pinned host
// staging. Growing any of them invalidates the captured graph (its copies and kernel
// parameters name the old buffers and sizes). A group that grows counts as empty until its last
// allocation has succeeded: after a failure the next call makes all of it again.
static es_status ensure_capacity(es_engine *e, Slot *sl, size_t nwin, size_t npieces, size_t nchunks, size_t cap) {
  if (!sl->d_hdr) CU(cudaMalloc(&sl->d_hdr, sizeof(BatchHdr)));
  if (!sl->h_hdr) CU(cudaMallocHost(&sl->h_hdr, sizeof(BatchHdr)));
  if (!sl->h_ctr) CU(cudaMallocHost(&sl->h_ctr, CTR_OUT * sizeof(unsigned long long)));
  if (!sl->h_status) CU(cudaMallocHost(&sl->h_status, sizeof(u32)));
  if (nwin > sl->win_cap) {
    drop_graph(sl);
    cudaFree(sl->d_win); cudaFree(sl->d_cnt); cudaFree(sl->d_Qm);
    cudaFreeHost(sl->h_win); cudaFreeHost(sl->h_roww); cudaFreeHost(sl->h_cnt);
    sl->d_win = nullptr; sl->d_cnt = nullptr; sl->d_Qm = nullptr;
    sl->h_win = nullptr; sl->h_roww = nullptr; sl->h_cnt = nullptr;
    sl->win_cap = 0;
    const size_t want = grown(nwin, 64);
    CU(cudaMalloc(&sl->d_win, want * sizeof(WinDev)));
    CU(cudaMalloc(&sl->d_cnt, want * sizeof(WinCount)));
    CU(cudaMalloc(&sl->d_Qm, want * std::max<u32>(e->Dq, 8) * sizeof(u16)));
    CU(cudaMallocHost(&sl->h_win, want * sizeof(WinDev)));
    CU(cudaMallocHost(&sl->h_roww, want * sizeof(RowWin)));
    CU(cudaMallocHost(&sl->h_cnt, want * sizeof(WinCount)));
    sl->win_cap = want;
    sl->qm_cap = want * std::max<u32>(e->Dq, 8);
  }
  if (npieces > sl->piece_cap) {
    drop_graph(sl);
    cudaFree(sl->d_piece); cudaFree(sl->d_pidx); cudaFree(sl->d_rowinfo);
    sl->d_piece = nullptr; sl->d_pidx = nullptr; sl->d_rowinfo = nullptr;
    sl->piece_cap = 0;
    const size_t want = grown(npieces, 256);
    CU(cudaMalloc(&sl->d_piece, want * sizeof(Piece)));
    CU(cudaMalloc(&sl->d_pidx, want * std::max<u32>(e->n1p, 8) * sizeof(u16)));
    CU(cudaMalloc(&sl->d_rowinfo, want * PIECE_ROWS * sizeof(u32)));
    sl->piece_cap = want;
  }
  if (nchunks > sl->chunk_cap) {
    drop_graph(sl);
    cudaFree(sl->d_cand); cudaFree(sl->d_chunk);
    sl->d_cand = nullptr; sl->d_chunk = nullptr;
    sl->chunk_cap = 0;
    CU(cudaMalloc(&sl->d_cand, nchunks * 32 * sizeof(uint2)));
    CU(cudaMalloc(&sl->d_chunk, nchunks * sizeof(u32)));
    sl->chunk_cap = nchunks;
  }
  if (cap > sl->cap) {
    drop_graph(sl);
    cudaFree(sl->d_surv); cudaFree(sl->d_primes); cudaFree(sl->d_direct); cudaFree(sl->d_recs);
    cudaFreeHost(sl->h_recs);
    sl->d_surv = nullptr; sl->d_primes = sl->d_direct = nullptr; sl->d_recs = nullptr; sl->h_recs = nullptr;
    sl->cap = 0;
    CU(cudaMalloc(&sl->d_surv, cap * sizeof(Surv)));
    CU(cudaMalloc(&sl->d_primes, cap * sizeof(u32)));
    CU(cudaMalloc(&sl->d_direct, cap * sizeof(u32)));
    CU(cudaMalloc(&sl->d_recs, cap * sizeof(RecDev)));
    CU(cudaMallocHost(&sl->h_recs, cap * sizeof(RecDev)));
    sl->cap = cap;
  }
  return ES_OK;
}

static MarkParams mark_params(const es_engine *e, const Slot *sl) {
  MarkParams P;
  P.rho = e->d_rho; P.K0 = e->d_K0; P.fdesc = e->d_fdesc; P.sdist = e->d_sdist;
  P.Qm = sl->d_Qm;
  P.win = sl->d_win; P.queue = reinterpret_cast<u64 *>(sl->d_ctr + 0);
  P.surv = sl->d_surv; P.surv_count = sl->d_ctr + 1; P.cnt = sl->d_cnt;
  P.hdr = sl->d_hdr; P.ctr = sl->d_ctr; P.surv_cap = sl->cap; P.M = e->M;
  P.L = (u32)e->classes.size(); P.ldk = e->ldk; P.nf = e->nf; P.ncov = (u32)e->ncov;
  P.D = e->D; P.Dq = e->Dq;
  P.r_bytes = (4 * e->D + 15) & ~15u;
  return P;
}

static TailParams tail_params(const es_engine *e, const Slot *sl) {
  TailParams T;
  T.ctr = sl->d_ctr; T.hdr = sl->d_hdr; T.out = HostOut{sl->h_ctr, sl->h_status, sl->h_cnt, sl->h_recs};
  T.surv = sl->d_surv; T.surv_count = sl->d_ctr + 1;
  T.primes = sl->d_primes; T.prime_count = sl->d_ctr + 2;
  T.direct = sl->d_direct; T.direct_count = sl->d_ctr + 3;
  T.recs = sl->d_recs; T.rec_count = sl->d_ctr + 4;
  T.rung_next = sl->d_ctr + 6; T.rung_done = sl->d_ctr + 7; T.help_sessions = sl->d_ctr + 8;
  T.board = reinterpret_cast<BoardSlot *>(sl->d_ctr + CTR_OUT);
  T.rung_next_warp = sl->d_ctr + 9;
  T.rho_budget = e->rho_budget;
  T.cnt = sl->d_cnt; T.tdp = e->d_tdp; T.tde = e->d_tde; T.tdi = e->d_tdi; T.tdqm = e->d_tdqm; T.status = sl->d_status;
  T.cap = sl->cap;
  return T;
}

static RowParams row_params(const es_engine *e, const Slot *sl) {
  RowParams S;
  S.rho = e->d_rho; S.K0 = e->d_K0; S.fdesc = e->d_fdesc; S.tdense = e->d_tdense; S.tlane = e->d_tlane;
  S.mdesc = e->d_mdesc; S.lfil = e->d_lfil; S.win = sl->d_win; S.piece = sl->d_piece;
  S.h_hdr = sl->h_hdr; S.h_win = sl->h_win; S.h_roww = sl->h_roww; S.ctr = sl->d_ctr;
  S.pidx = sl->d_pidx; S.rowinfo = sl->d_rowinfo; S.cand = sl->d_cand; S.chunk = sl->d_chunk;
  S.chunk_count = sl->d_ctr + 10; S.chunk_cap = (u32)sl->chunk_cap;
  S.surv = sl->d_surv; S.surv_count = sl->d_ctr + 1; S.cnt = sl->d_cnt; S.surv_cap = sl->cap; S.M = e->M;
  S.status = sl->d_status; S.hdr = sl->d_hdr;
  S.L = (u32)e->classes.size(); S.ldk = e->ldk; S.lane_words = e->lane_words; S.ngroups = e->ngroups;
  S.slice_bytes = e->slice_rows * 4 * GROUP_WORDS; S.n1 = e->n1; S.n1p = e->n1p; S.n2 = e->n2;
  S.nm_cov = e->nm_cov; S.nm_all = e->nm_all; S.nl_cov = e->nl_cov; S.nl_all = e->nl_all;
  S.wide = (DIRECT_PMAX / e->M) >> 48 != 0;
  S.squares = e->squares;
  S.nsq = (u32)e->sq.size();
  for (u32 i = 0; i < S.nsq; ++i) {
    const u32 q = e->sq[i];
    u32 v = q;                                       // q^-1 mod 2^32 by Newton, from 3 bits
    for (int k = 0; k < 4; ++k) v *= 2 - q * v;
    S.sq_inv[i] = v;
    S.sq_lim[i] = ~0u / q;
  }
  return S;
}

static size_t mark_smem(const es_engine *e) {
  return ((4 * e->D + 15) & ~15u) + std::max<u32>(SEG_BIG, GROUP * SEG_SMALL) + 16;
}

constexpr int LANE_BLOCK_BITS = 9;

// Number of classes below x, 0 <= x <= M (lower_bound over the sorted classes, by table).
static u64 classes_below(const es_engine *e, u64 x) {
  u64 i = e->lane_at[x >> LANE_BLOCK_BITS];
  while (i < e->classes.size() && e->classes[i] < x) ++i;
  return i;
}

// x / M and x mod M for any 64-bit x: a double estimate of the quotient, corrected exactly (its
// relative error is below 2^-51: off by at most one while x / M < 2^51, by a few for smaller M).
static void divmod_M(const es_engine *e, u64 x, u64 &q, u64 &r) {
  const u64 M = e->M;
  q = (u64)((double)x * e->inv_M);
  unsigned __int128 qm = (unsigned __int128)q * M;
  for (; qm > x; qm -= M) --q;
  for (r = x - (u64)qm; r >= M; r -= M) ++q;
}

static void build_lane_index(es_engine *e) {
  const u64 nb = (e->M >> LANE_BLOCK_BITS) + 2;
  e->lane_at.assign(nb, 0);
  size_t i = 0;
  for (u64 b = 0; b < nb; ++b) {
    while (i < e->classes.size() && e->classes[i] < (b << LANE_BLOCK_BITS)) ++i;
    e->lane_at[b] = (uint32_t)i;
  }
  e->inv_M = 1.0 / (double)e->M;
}

// Window descriptors and their marking work. Windows marked by rows (all of them with
// sched.long_split, else those with at most sched.short_max positions in any lane) get their run
// of rows: K = lo / M from the first class at or above lo mod M on, to the last class below hi.
// The others get one lane per item and segments of SEG_BIG positions in k_mark. npos[i] is the
// window's wheel positions; the totals go to `run`.
struct RunShape {
  u64 items = 0, rows = 0, pieces = 0;
  u64 positions = 0, row_positions = 0;    // of all windows, of those marked by rows
};
static RunShape describe(const es_engine *e, const es_window *w, size_t n, std::vector<WinDev> &out,
                         std::vector<RowWin> &roww, std::vector<u64> &npos) {
  out.resize(n);
  npos.resize(n);
  roww.clear();
  roww.reserve(n);
  RunShape run;
  const u64 L = e->classes.size();
  for (size_t i = 0; i < n; ++i) {
    WinDev &d = out[i];
    d.lo = w[i].lo; d.hi = std::max(w[i].lo, w[i].hi);
    u64 q, r, qh, rh;
    divmod_M(e, d.lo, q, r);
    divmod_M(e, d.hi, qh, rh);
    d.Q = q;
    d.lomod = (u32)r;
    d.item0 = run.items;
    d.G = 1; d.lane0 = 0;
    d.seg = SEG_SMALL; d.nseg = 0; d.groups = 0;
    // positions before lo and before hi, both counted from K = q
    const u64 before = classes_below(e, r), upto = (qh - q) * L + classes_below(e, rh);
    npos[i] = upto - before;
    run.positions += npos[i];
    if (!npos[i]) continue;
    u64 maxpos, rem_;                                    // most positions any lane can hold
    divmod_M(e, d.hi - d.lo - 1, maxpos, rem_);
    ++maxpos;
    if (e->sched.long_split || maxpos <= e->sched.short_max) {
      const u64 k0 = before / L, k1 = (upto - 1) / L;    // first and last row holding a position, from q
      RowWin x;
      x.K0 = q + k0;
      x.nrows = (u32)(k1 - k0 + 1);
      x.la = (u32)(before - k0 * L);
      x.lb = (u32)(upto - k1 * L);
      x.wi = (u32)i;
      x.row0 = (u32)run.rows;
      x.piece0 = (u32)run.pieces;
      roww.push_back(x);
      run.rows += x.nrows;
      run.row_positions += npos[i];
      run.pieces += (x.nrows + PIECE_ROWS - 1) / PIECE_ROWS;
    } else {
      d.seg = SEG_BIG; d.nseg = (u32)((maxpos + SEG_BIG - 1) / SEG_BIG); d.groups = (u32)L;
      run.items += (u64)d.groups * d.nseg;
    }
  }
  return run;
}

// Wheel positions in [lo, hi): L per full period of M, plus the classes among the residues
// of the remainder (the sum over lanes of sieve/rung_scan3.cpp:716's npos).
static u64 positions_in(const es_engine *e, u64 lo, u64 hi) {
  if (hi <= lo) return 0;
  const u64 M = e->M;
  u64 qa, a, ql, rem;
  divmod_M(e, lo, qa, a);
  divmod_M(e, hi - lo, ql, rem);
  u64 part = a + rem <= M ? classes_below(e, a + rem) - classes_below(e, a)
                          : (e->classes.size() - classes_below(e, a)) + classes_below(e, a + rem - M);
  return ql * e->classes.size() + part;
}

// The funnel's front on the engine's stream: k_rows (which takes the header and the window
// descriptors from pinned staging and clears the counters), the marking kernels and Miller-Rabin.
// With `capture` the event record is an external graph node, so that the run can be timed when the
// sequence is a graph. `rows`, `segments`: some windows may be marked by rows, by segments (k_mark,
// sized by `items_hint` in the plain schedule). Adds its kernel launches to `launches`.
static es_status enqueue_front(es_engine *e, Slot *sl, bool persistent, WinCount *cnt, bool rows, bool segments,
                               u64 items_hint, bool capture, u64 &launches) {
  MarkParams P = mark_params(e, sl);
  TailParams T = tail_params(e, sl);
  P.cnt = cnt;
  T.cnt = cnt;
  cudaStream_t st = sl->stream;
  CU(capture ? cudaEventRecordWithFlags(sl->ev[0], st, cudaEventRecordExternal) : cudaEventRecord(sl->ev[0], st));
  RowParams S = row_params(e, sl);
  S.cnt = cnt;
  k_rows<<<e->sm_count * 4, 256, 0, st>>>(S);
  CU(cudaGetLastError());
  ++launches;
  if (segments) {
    k_prep<<<e->sm_count * 4, 256, 0, st>>>(sl->d_hdr, sl->d_win, e->d_sdist, e->D, e->Dq, sl->d_Qm);
    CU(cudaGetLastError());
    ++launches;
  }
  if (rows) {
    k_mark_short<<<e->sm_count, ROW_THREADS, e->slice_rows * 4 * GROUP_WORDS + CAND_SMEM, st>>>(S);
    CU(cudaGetLastError());
    k_sift<<<e->sm_count, ROW_THREADS, ROW_SMEM, st>>>(S);
    CU(cudaGetLastError());
    launches += 2;
  }
  if (segments) {
    const unsigned grid = persistent ? (unsigned)((u64)e->sm_count * e->mark_occupancy)
                                     : (unsigned)std::max<u64>(1, std::min<u64>(items_hint, 0x7FFFFFFFull));
    k_mark<MARK_BLOCK><<<grid, MARK_BLOCK, mark_smem(e), st>>>(P, persistent ? 1 : 0);
    CU(cudaGetLastError());
    ++launches;
  }
  k_mr<<<e->sm_count * MR_BLOCKS_PER_SM, 256, 0, st>>>(T);
  CU(cudaGetLastError());
  ++launches;
  return ES_OK;
}

// The funnel's tail on the slot's stream: stage D, stage E, the results written to pinned memory
// (the windows' counters at out_cnt). Adds its kernel launches to `launches`.
static es_status enqueue_tail(es_engine *e, Slot *sl, WinCount *cnt, WinCount *out_cnt, bool capture, u64 &launches) {
  TailParams T = tail_params(e, sl);
  T.cnt = cnt;
  T.out.cnt = out_cnt;
  cudaStream_t st = sl->stream;
  const u32 teams = e->sm_count * std::min<u32>(e->sched.rung_blocks_per_sm, RUNG_TEAMS);
  const int no_rung = (e->flags & ES_FLAG_NO_RUNG) ? 1 : 0;
  k_rung<<<(teams + RUNG_TEAMS - 1) / RUNG_TEAMS, RUNG_THREADS, sizeof(RungBlock), st>>>(T, no_rung);
  CU(cudaGetLastError());
  if (no_rung) {
    k_search<<<e->sm_count * 16, 32, 0, st>>>(T);
    CU(cudaGetLastError());
  }
  k_direct<<<e->sm_count, 256, 0, st>>>(T, no_rung);
  CU(cudaGetLastError());
  launches += 2 + no_rung;
  CU(capture ? cudaEventRecordWithFlags(sl->ev[4], st, cudaEventRecordExternal) : cudaEventRecord(sl->ev[4], st));
  return ES_OK;
}

// The end of the front (ev[11], which a serving slot's front waits for) inside the synchronous slot's
// single graph: a leaf of its own beside stage D. As a node between Miller-Rabin and stage D it took
// 2.2 us of a small window's 39; recorded after the graph, as it was, it made a served request wait for
// stage D and the results (a request beside a call of 11.7 ms of direct search: 23.6 ms for both, 14.0 so).
static es_status capture_front_end(es_engine *e, Slot *sl) {
  cudaStreamCaptureStatus status;
  unsigned long long id;
  cudaGraph_t g;
  const cudaGraphNode_t *deps;
  const cudaGraphEdgeData *edges;
  size_t n;
  CU(cudaStreamGetCaptureInfo(sl->stream, &status, &id, &g, &deps, &edges, &n));
  cudaGraphNode_t node;
  CU(cudaGraphAddEventRecordNode(&node, g, deps, n, sl->ev[11]));
  return ES_OK;
}

// The persistent schedule as CUDA graphs, captured once and replayed per batch: for a serving slot
// two, the funnel up to Miller-Rabin, and stage D and E with the results written out; for the
// synchronous slot one, with the front's end recorded inside (the gap between two is 5 us of a small window's 50).
static es_status capture_graph(es_engine *e, Slot *sl) {
  drop_graph(sl);
  struct Undo {                                    // a front without its tail is none, on every return path
    Slot *sl;
    ~Undo() { if (sl) drop_graph(sl); }
  } undo{sl};
  const bool one = sl == &e->slots[0];
  u64 launches = 0;
  for (int part = 0; part < (one ? 1 : 2); ++part) {
    CU(cudaStreamBeginCapture(sl->stream, cudaStreamCaptureModeThreadLocal));
    es_status s = ES_OK;
    if (part == 0) s = enqueue_front(e, sl, true, sl->d_cnt, true, !e->sched.long_split, 0, true, launches);
    if (s == ES_OK && one) s = capture_front_end(e, sl);
    if (s == ES_OK && (one || part == 1)) s = enqueue_tail(e, sl, sl->d_cnt, sl->h_cnt, true, launches);
    cudaGraph_t g = nullptr;
    const cudaError_t end = cudaStreamEndCapture(sl->stream, &g);
    if (end != cudaSuccess) cudaGetLastError();
    if (s != ES_OK) { if (g) cudaGraphDestroy(g); return s; }
    if (end != cudaSuccess) return fail(e, ES_ERR_CUDA, std::string("capture: ") + cudaGetErrorString(end));
    (part == 0 ? sl->graph : sl->graph2) = g;
    CU(cudaGraphInstantiate(part == 0 ? &sl->gexec : &sl->gexec2, g, 0));
  }
  undo.sl = nullptr;
  sl->graph_launches = launches;
  return ES_OK;
}

// Launches a captured persistent run on the slot's stream. The front waits for the front
// most recently launched on any other slot, so batches are marked one at a time in launch
// order, and a batch's stage-D tail (a few latency-bound factorizations on a handful of SMs)
// runs beside the next batch's marking instead of leaving the GPU idle.
static es_status launch_persistent(es_engine *e, Slot *sl) {
  {
    std::lock_guard<std::mutex> lk(e->front_mu);
    if (e->last_front && e->last_front != sl) CU(cudaStreamWaitEvent(sl->stream, e->last_front->ev[11], 0));
    CU(cudaGraphLaunch(sl->gexec, sl->stream));
    if (sl->gexec2) CU(cudaEventRecord(sl->ev[11], sl->stream));
    e->last_front = sl;
  }
  if (sl->gexec2) CU(cudaGraphLaunch(sl->gexec2, sl->stream));
  return ES_OK;
}

static float ev_ms(cudaEvent_t a, cudaEvent_t b) {
  float ms = 0;
  if (cudaEventElapsedTime(&ms, a, b) != cudaSuccess) { (void)cudaGetLastError(); ms = 0; }
  return ms;
}

static std::string status_text(u32 st) {
  std::string s;
  if (st & ST_RHO_BUDGET) s += " rho-budget";
  if (st & ST_FAC_OVERFLOW) s += " factor-overflow";
  if (st & ST_STACK_OVERFLOW) s += " factor-stack";
  if (st & ST_QUEUE_TIMEOUT) s += " queue-timeout";
  if (st & ST_BAD_INPUT) s += " bad-input";
  if (st & ST_CERT_BAD) s += " certificate-self-check";
  return s;
}

static double ms_since(std::chrono::steady_clock::time_point t) {
  return std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t).count();
}

constexpr size_t ORDER_BINS_MIN = 64;
// The caller's copy of m records of n windows, in (window, lane, J) order. What is sorted are
// 16-byte keys, dealt out by window and, in a window of many, by lane into about as many bins as it
// has records; each record is then copied once, from where the device wrote it. 88 K records
// (one window of 2^43 integers at 1e16): 2.4 ms, where sorting the records themselves took 6.2.
// Below ORDER_BINS_MIN the bins' own passes cost as much as the comparisons that they save.
static es_status order_records(es_engine *e, Slot *sl, const RecDev *src, size_t m, size_t n, es_records *recs) {
  static_assert(sizeof(RecDev) == sizeof(es_record), "record layout");
  recs->n = m;
  recs->recs = (es_record *)malloc(std::max<size_t>(m, 1) * sizeof(es_record));
  if (!recs->recs) return fail(e, ES_ERR_NOMEM, "host records");
  std::vector<u32> &start = sl->hs.start, &pos = sl->hs.pos, &bstart = sl->hs.bstart;
  std::vector<RecKey> &key = sl->hs.key, &bin = sl->hs.bin;
  start.assign(n + 1, 0);
  pos.resize(m);
  bin.resize(m);
  for (size_t i = 0; i < m; ++i) {                   // one read of what the device wrote, in its order
    const RecDev &r = src[i];
    bin[i] = RecKey{r.J, r.lane, (u32)i};
    pos[i] = (u32)std::min<size_t>(r.win, n - 1);
    ++start[pos[i] + 1];
  }
  for (size_t i = 0; i < n; ++i) start[i + 1] += start[i];
  if (n == 1) {
    key.swap(bin);
  } else {
    key.resize(m);
    bstart.assign(start.begin(), start.end() - 1);
    for (size_t i = 0; i < m; ++i) key[bstart[pos[i]]++] = bin[i];
  }
  const size_t lanes = std::max<size_t>(e->classes.size(), 1);
  for (size_t i = 0; i < n; ++i) {
    RecKey *k = key.data() + start[i];
    const size_t c = start[i + 1] - start[i];
    if (c > ORDER_BINS_MIN) {
      u32 shift = 0;
      while ((lanes - 1) >> shift >= c) ++shift;
      const size_t bins = ((lanes - 1) >> shift) + 1;
      auto bin_of = [&](const RecKey &x) { return std::min<size_t>(x.lane >> shift, bins - 1); };
      bstart.assign(bins + 1, 0);
      for (size_t j = 0; j < c; ++j) ++bstart[bin_of(k[j]) + 1];
      for (size_t b = 0; b < bins; ++b) bstart[b + 1] += bstart[b];
      bin.assign(k, k + c);
      for (const RecKey &x : bin) k[bstart[bin_of(x)]++] = x;      // bstart[b] is now bin b's end
      size_t from = 0;
      for (size_t b = 0; b < bins; from = bstart[b++])
        if (bstart[b] - from > 1) std::sort(k + from, k + bstart[b]);
    } else if (c > 1) {
      std::sort(k, k + c);
    }
  }
  RecDev *out = reinterpret_cast<RecDev *>(recs->recs);
  for (size_t i = 0; i < m; ++i) {
    if (i + 16 < m) __builtin_prefetch(&src[key[i + 16].idx]);
    out[i] = src[key[i].idx];
  }
  return ES_OK;
}

// Survivors that a run's buffers are made for: SURV_ROOM times the tables' estimate and, where squares
// get no shortcut, the squares (they survive what the estimate takes for random), at most all the
// positions; in powers of two, so that batches a little larger than the last do not each make their
// own. Over 2^34 to 2^43 integers at 1e12 to 1e19 and three tables 0.6 to 2.2 times the estimate
// came (up to 15 times at 1e12 with 91 expected, where the squares are most of it). A window of 2^43
// integers at 1e16 takes 8 M records of room where 1/64 of its positions took 67 M, 4.3 GB of it
// pinned: the first call of an engine 161 -> 25 ms, the 4096-window batch's 6.9 -> 1.7 ms.
constexpr double SURV_ROOM = 8;
constexpr size_t SURV_MIN = 1 << 16;
static size_t surv_need(const es_engine *e, const es_window *w, size_t n, u64 positions) {
  double want = SURV_ROOM * e->surv_rate * (double)positions;
  for (size_t i = 0; i < n && !e->squares; ++i)
    if (w[i].hi > w[i].lo) want += std::sqrt((double)w[i].hi) - std::sqrt((double)w[i].lo) + 1;
  return (size_t)std::min(std::min(want, (double)positions) + 1024, (double)(1u << 26));
}
// Candidate chunks: half as many again as the tables' estimate. CHUNKS_MIN holds those of 5 G integers with
// the 120120 wheel's table, 80 G with the gpu table.
constexpr size_t CHUNKS_MIN = 8192;
static size_t chunk_need(const es_engine *e, u64 row_positions) {
  return (size_t)(1.5 * e->cand_rate * (double)row_positions / 32);
}
// Rows of [lo, hi), at most; 0 for a window that goes to the segment marking.
static u64 window_rows(const es_schedule &sched, u64 M, u64 lo, u64 hi) {
  const u64 len = hi > lo ? hi - lo : 0;
  return sched.long_split || len <= sched.short_max * M ? len / M + 2 : 0;
}

// Runs windows through the funnel and collects counters; the records are left unordered at *src
// (the slot's, until its next run). Re-runs with larger buffers when the survivor list overflowed
// (the count is exact even then).
static es_status run_device_windows(es_engine *e, Slot *sl, const es_window *w, size_t n, int schedule,
                                    es_counters *per_window, const RecDev **src, size_t *nsrc) {
  const auto t_start = std::chrono::steady_clock::now();
  double setup_ms = 0, device_ms = 0;
  const u64 floor_ = std::max(e->wheel_pmin, e->cover_pmax);
  for (size_t i = 0; i < n; ++i) {
    if (w[i].hi > DIRECT_PMAX)
      return fail(e, ES_ERR_RANGE, "HI must not exceed the stage-E ceiling " + std::to_string(DIRECT_PMAX));
    if (w[i].lo <= floor_)
      return fail(e, ES_ERR_RANGE, "LO must exceed max pmin of the filter table (" + std::to_string(floor_) + ")");
  }
  std::vector<WinDev> &wd = sl->hs.wd;
  std::vector<RowWin> &roww = sl->hs.roww;
  std::vector<u64> &npos = sl->hs.npos;
  const RunShape shape = describe(e, w, n, wd, roww, npos);
  size_t cap = std::max(grown(surv_need(e, w, n, shape.positions), SURV_MIN), sl->cap);
  size_t chunks = grown(chunk_need(e, shape.row_positions), CHUNKS_MIN) +
                  4 * (size_t)e->sm_count * (ROW_THREADS / 32);       // a part-filled one per warp and run
  const bool persistent = schedule == ES_SCHED_PERSISTENT;
  std::vector<RecDev> &hr = sl->hs.hr;   // the plain schedule's
  size_t nrec = 0;
  bool done = false;
  u64 launches = 0;                      // of all attempts
  for (int attempt = 0; attempt < 4 && !done; ++attempt) {
    es_status s = ensure_capacity(e, sl, n, shape.pieces, chunks, cap);
    if (s) return s;
    double total_ms = 0, mark_ms = 0, mr_ms = 0, rung_ms = 0, direct_ms = 0, prep_ms = 0, short_ms = 0, long_ms = 0;
    u64 surv_max = 0, chunk_max = 0, prime_total = 0;
    u32 status = 0;
    hr.clear();
    auto collect = [&]() -> es_status {   // after a pass: timings, counts, records
      total_ms += ev_ms(sl->ev[0], sl->ev[4]);
      // a stage runs from its first kernel's start to the next stage's; 0 marks one not launched
      const unsigned long long *t = sl->h_ctr + STAMP0;
      auto ms = [](u64 a, u64 b) { return b > a ? (double)(b - a) * 1e-6 : 0.0; };
      const u64 longs = t[2] ? t[2] : t[3], rows = t[1] ? t[1] : longs;
      prep_ms += ms(t[0], rows); short_ms += ms(rows, longs); long_ms += ms(longs, t[3]);
      mark_ms += ms(t[0], t[3]); mr_ms += ms(t[3], t[4]);
      rung_ms += ms(t[4], t[5]); direct_ms += ms(t[5], t[6]);
      const unsigned long long *ctr = sl->h_ctr;
      surv_max = std::max<u64>(surv_max, ctr[1]);
      chunk_max = std::max<u64>(chunk_max, ctr[10]);
      prime_total += ctr[2];
      status |= *sl->h_status;
      if (ctr[1] > sl->cap) return ES_OK;
      nrec = (size_t)std::min<u64>(ctr[4], sl->cap);
      return ES_OK;
    };
    if (persistent) {
      sl->h_hdr->total_items = shape.items;
      sl->h_hdr->nwin = (u32)n;
      sl->h_hdr->nshort = (u32)roww.size();
      sl->h_hdr->nrows = (u32)shape.rows;
      sl->h_hdr->npieces = (u32)shape.pieces;
      memcpy(sl->h_win, wd.data(), n * sizeof(WinDev));
      if (!roww.empty()) memcpy(sl->h_roww, roww.data(), roww.size() * sizeof(RowWin));
      if (!sl->gexec) { s = capture_graph(e, sl); if (s) return s; }
      setup_ms = ms_since(t_start);
      const auto t_launch = std::chrono::steady_clock::now();
      s = launch_persistent(e, sl);
      if (s) return s;
      CU(cudaStreamSynchronize(sl->stream));
      device_ms = ms_since(t_launch);
      launches += sl->graph_launches;
      s = collect();
      if (s) return s;
    } else {
      // The plain schedule: the same kernels, one launch sequence per window.
      size_t k = 0;                      // next window marked by rows (describe emits them in order)
      for (size_t i = 0; i < n; ++i) {
        sl->h_win[0] = wd[i];
        sl->h_win[0].item0 = 0;
        const u64 items = (u64)wd[i].nseg * wd[i].groups;
        BatchHdr &h = *sl->h_hdr;
        h.total_items = items; h.nwin = 1; h.nshort = h.nrows = h.npieces = 0;
        if (k < roww.size() && roww[k].wi == i) {
          RowWin &x = sl->h_roww[0];
          x = roww[k++];
          x.wi = x.row0 = x.piece0 = 0;
          h.nshort = 1; h.nrows = x.nrows; h.npieces = (x.nrows + PIECE_ROWS - 1) / PIECE_ROWS;
        }
        s = enqueue_front(e, sl, false, sl->d_cnt + i, h.nshort != 0, items != 0, items, false, launches);
        if (s) return s;
        s = enqueue_tail(e, sl, sl->d_cnt + i, sl->h_cnt + i, false, launches);
        if (s) return s;
        CU(cudaStreamSynchronize(sl->stream));
        nrec = 0;
        s = collect();
        if (s) return s;
        if (surv_max > sl->cap || chunk_max > sl->chunk_cap) break;
        for (size_t r = 0; r < nrec; ++r) {
          hr.push_back(sl->h_recs[r]);
          hr.back().win = (u32)i;
        }
      }
    }
    if (surv_max > sl->cap || chunk_max > sl->chunk_cap) {   // overflow: grow to the exact need and re-run
      if (surv_max > sl->cap) cap = (size_t)(surv_max + surv_max / 4 + 1024);
      if (chunk_max > sl->chunk_cap) chunks = (size_t)(chunk_max + chunk_max / 4);
      continue;
    }
    if (status) return fail(e, ES_ERR_DEVICE_STATUS, "device status:" + status_text(status));
    sl->timing.total_ms = total_ms;
    sl->timing.mark_ms = mark_ms; sl->timing.mr_ms = mr_ms;
    sl->timing.prep_ms = prep_ms; sl->timing.mark_short_ms = short_ms; sl->timing.mark_long_ms = long_ms;
    sl->timing.short_pairs = (u64)roww.size() * e->classes.size();
    sl->timing.mask_bytes = roww.empty() ? 0 : (u64)e->ngroups * e->slice_rows * 4 * GROUP_WORDS;
    sl->timing.rung_ms = rung_ms; sl->timing.direct_ms = direct_ms;
    sl->timing.marks_kernel_launches = persistent ? 1 : n;
    sl->timing.kernel_launches = launches;
    sl->timing.mark_items = shape.items;
    sl->timing.primes = prime_total;
    done = true;
  }
  if (!done) return fail(e, ES_ERR_NOMEM, "survivor list kept overflowing");
  sl->timing.survivors = 0;
  for (size_t i = 0; i < n; ++i) {      // the SUMMARY counters (sieve/rung_scan3.cpp:764-772)
    const WinCount &c = sl->h_cnt[i];
    es_counters &o = per_window[i];
    o.positions = npos[i];
    sl->timing.survivors += c.surv;
    if (e->nf == e->ncov) { o.covered = o.positions - c.surv; o.sieved = 0; }
    else { o.covered = o.positions - c.after_covers; o.sieved = c.after_covers - c.surv; }
    // every prime survivor ends as a rung record, a direct one or an unsolved one, so the
    // composites are the rest (a run where that fails is refused by its status)
    const unsigned long long primes_w = c.rung + c.direct + c.unsolved;
    o.mr = c.surv; o.composite = c.surv >= primes_w ? c.surv - primes_w : 0; o.rung = c.rung; o.direct = c.direct;
    o.survivors = c.unsolved;
  }
  *src = persistent ? sl->h_recs : hr.data();
  *nsrc = persistent ? nrec : hr.size();
  sl->timing.host_setup_ms = setup_ms;
  sl->timing.host_device_ms = device_ms;
  sl->timing.host_collect_ms = ms_since(t_start) - setup_ms - device_ms;
  return ES_OK;
}

// Runs windows in passes of at most e->pass_rows rows. A window
// that does not fit the pass is cut at whole multiples of M: a part that starts t M
// integers into the window starts t positions into every lane, so its records map back by J += t,
// and its counters add up to the window's (every counter is a sum over positions). Every caller
// passes per_window zeroed.
static es_status run_windows(es_engine *e, Slot *sl, const es_window *w, size_t n, int schedule,
                             es_counters *per_window, es_records *recs) {
  const u64 M = e->M;
  const u64 floor_ = std::max(e->wheel_pmin, e->cover_pmax);
  u64 rows = 0;
  for (size_t i = 0; i < n; ++i) {                 // refuse what a run would refuse, first
    if (w[i].hi > DIRECT_PMAX)
      return fail(e, ES_ERR_RANGE, "HI must not exceed the stage-E ceiling " + std::to_string(DIRECT_PMAX));
    if (w[i].lo <= floor_)
      return fail(e, ES_ERR_RANGE, "LO must exceed max pmin of the filter table (" + std::to_string(floor_) + ")");
    rows += window_rows(e->sched, M, w[i].lo, w[i].hi);
  }
  const RecDev *src = nullptr;
  size_t nsrc = 0;
  const auto t_start = std::chrono::steady_clock::now();
  auto finish = [&](const RecDev *from, size_t m) -> es_status {     // the records, ordered
    if (recs) {
      es_status st;
      try {
        st = order_records(e, sl, from, m, n, recs);
      } catch (const std::bad_alloc &) {
        es_free_records(recs);
        st = fail(e, ES_ERR_NOMEM, "host records");
      }
      if (st != ES_OK) return st;
    }
    sl->timing.host_collect_ms = ms_since(t_start) - sl->timing.host_setup_ms - sl->timing.host_device_ms;
    return ES_OK;
  };
  if (rows <= e->pass_rows) {
    const es_status st = run_device_windows(e, sl, w, n, schedule, per_window, &src, &nsrc);
    return st != ES_OK ? st : finish(src, nsrc);
  }
  std::vector<RecDev> &all = sl->hs.all;
  all.clear();
  es_timing_t tot{};
  std::vector<es_window> &dw = sl->hs.dw;
  std::vector<std::pair<u32, u64>> &dmap = sl->hs.dmap;   // (window, position offset) per device window
  std::vector<es_counters> &pc = sl->hs.pc;
  size_t i = 0;
  u64 t = 0;                                         // window i is done up to t M integers
  while (i < n) {
    dw.clear();
    dmap.clear();
    for (u64 left = e->pass_rows; i < n;) {
      const u64 lo = w[i].lo + t * M, hi = std::max(w[i].lo, w[i].hi), need = window_rows(e->sched, M, lo, hi);
      if (need <= left) {
        dw.push_back({lo, hi});
        dmap.push_back({(u32)i, t});
        left -= need;
        ++i;
        t = 0;
        continue;
      }
      if (e->sched.long_split && left > 2) {         // need > left: (left - 2) M is below hi - lo
        dw.push_back({lo, lo + (left - 2) * M});
        dmap.push_back({(u32)i, t});
        t += left - 2;
      }
      break;
    }
    const size_t m = dw.size();
    pc.resize(m);
    const es_status st = run_device_windows(e, sl, dw.data(), m, schedule, pc.data(), &src, &nsrc);
    if (st != ES_OK) return st;
    for (size_t k = 0; k < m; ++k) {
      es_counters &o = per_window[dmap[k].first];
      const es_counters &c = pc[k];
      o.positions += c.positions; o.covered += c.covered; o.sieved += c.sieved; o.mr += c.mr;
      o.composite += c.composite; o.rung += c.rung; o.direct += c.direct; o.survivors += c.survivors;
    }
    for (size_t r = 0; recs && r < nsrc; ++r) {
      all.push_back(src[r]);
      RecDev &x = all.back();
      const auto &mp = dmap[std::min<size_t>(x.win, m - 1)];
      x.win = mp.first;
      x.J += mp.second;
    }
    const es_timing_t &tt = sl->timing;
    tot.total_ms += tt.total_ms; tot.mark_ms += tt.mark_ms; tot.mr_ms += tt.mr_ms; tot.rung_ms += tt.rung_ms;
    tot.direct_ms += tt.direct_ms; tot.prep_ms += tt.prep_ms; tot.mark_short_ms += tt.mark_short_ms;
    tot.mark_long_ms += tt.mark_long_ms; tot.marks_kernel_launches += tt.marks_kernel_launches;
    tot.kernel_launches += tt.kernel_launches; tot.mark_items += tt.mark_items; tot.survivors += tt.survivors;
    tot.primes += tt.primes; tot.short_pairs += tt.short_pairs; tot.mask_bytes += tt.mask_bytes;
    tot.host_setup_ms += tt.host_setup_ms; tot.host_device_ms += tt.host_device_ms;
  }
  sl->timing = tot;
  return finish(all.data(), all.size());
}

static es_status build_tables(es_engine *e) {
  const u64 M = e->M;
  const u32 L = (u32)e->classes.size();
  const size_t nf = e->mods.size();
  // Per filter: g = gcd(M, mod), s = mod/g, inv = ((M/g) mod s)^-1 mod s.
  std::vector<u32> g(nf), s(nf), inv(nf);
  for (size_t i = 0; i < nf; ++i) {
    const u64 mod = e->mods[i];
    if (mod == 0) return fail(e, ES_ERR_FILTERS, "filter with modulus 0");
    if (mod > 0xFFFFFFFFull) return fail(e, ES_ERR_ARG, "filter modulus above 2^32 is not supported");
    const u64 gg = gcd_u64(M, mod), ss = mod / gg;
    if (ss > 0xFFFFull) return fail(e, ES_ERR_ARG, "filter stride mod/gcd(M,mod) above 65535 is not supported");
    bool ok;
    const u64 iv = ss == 1 ? 0 : inv_mod((M / gg) % ss, ss, ok);
    if (ss != 1 && !ok) return fail(e, ES_ERR_ARG, "non-invertible stride (impossible for g = gcd)");
    g[i] = (u32)gg; s[i] = (u32)ss; inv[i] = (u32)iv;
  }
  // Marking order: by stride within each phase, so that a warp's 32 filters have similar
  // trip counts. Marking is idempotent, so the order cannot change the result.
  e->order.resize(nf);
  for (size_t i = 0; i < nf; ++i) e->order[i] = (u32)i;
  std::stable_sort(e->order.begin(), e->order.begin() + e->ncov, [&](u32 a, u32 b) { return s[a] < s[b]; });
  std::stable_sort(e->order.begin() + e->ncov, e->order.end(), [&](u32 a, u32 b) { return s[a] < s[b]; });
  std::vector<u32> sd;
  for (size_t i = 0; i < nf; ++i) sd.push_back(s[i]);
  std::sort(sd.begin(), sd.end());
  sd.erase(std::unique(sd.begin(), sd.end()), sd.end());
  if (sd.size() > (size_t)DMAX) return fail(e, ES_ERR_ARG, "more than 8192 distinct filter strides");
  e->D = (u32)sd.size();
  e->Dq = (e->D + 7) & ~7u;                        // Qm rows: whole 16-byte chunks
  std::vector<u64> om(nf), orr(nf);
  std::vector<u32> og(nf), oinv(nf), fdesc(nf);
  for (size_t k = 0; k < nf; ++k) {
    const u32 i = e->order[k];
    om[k] = e->mods[i]; orr[k] = e->ress[i]; og[k] = g[i]; oinv[k] = inv[i];
    const u32 di = (u32)(std::lower_bound(sd.begin(), sd.end(), s[i]) - sd.begin());
    fdesc[k] = s[i] | (di << 16);
  }
  e->nf = (u32)nf;
  e->ldk = (u32)((nf + 7) & ~7ull);
  std::vector<u32> rho(L);
  for (u32 l = 0; l < L; ++l) rho[l] = (u32)e->classes[l];
  // trial-division table
  std::vector<u32> tdp;
  std::vector<TdEntry> tde;
  {
    std::vector<uint8_t> comp(65537, 0);
    for (u64 i = 2; i <= 65536; ++i) {
      if (comp[i]) continue;
      for (u64 j = i * i; j <= 65536; j += i) comp[j] = 1;
      if (i == 2) continue;
      u64 x = i;
      for (int k = 0; k < 5; ++k) x *= 2 - i * x;
      tdp.push_back((u32)i);
      tde.push_back(TdEntry{x, ~0ull / i});
    }
    if ((int)tdp.size() != NTD) return fail(e, ES_ERR_ARG, "trial-division table size");
  }
  // temporaries of the table build, freed on every return path
  struct Temps {
    void *p[7] = {};
    ~Temps() { for (void *x : p) cudaFree(x); }
  } temps;
  u64 *d_mods = nullptr, *d_ress = nullptr;
  u32 *d_g = nullptr, *d_inv = nullptr;
  CU(cudaMalloc(&e->d_rho, L * sizeof(u32)));
  CU(cudaMalloc(&e->d_fdesc, std::max<size_t>(nf, 1) * sizeof(u32)));
  CU(cudaMalloc(&e->d_sdist, std::max<size_t>(sd.size(), 1) * sizeof(u32)));
  CU(cudaMalloc(&e->d_K0, (size_t)L * e->ldk * sizeof(u16)));
  CU(cudaMalloc(&e->d_tdp, tdp.size() * sizeof(u32)));
  CU(cudaMalloc(&e->d_tde, tde.size() * sizeof(TdEntry)));
  CU(cudaMalloc(&e->d_tdi, tde.size() * sizeof(u64)));
  CU(cudaMalloc(&e->d_tdqm, tdp.size() * sizeof(uint2)));
  CU(cudaMalloc(&d_mods, std::max<size_t>(nf, 1) * sizeof(u64)));
  temps.p[0] = d_mods;
  CU(cudaMalloc(&d_ress, std::max<size_t>(nf, 1) * sizeof(u64)));
  temps.p[1] = d_ress;
  CU(cudaMalloc(&d_g, std::max<size_t>(nf, 1) * sizeof(u32)));
  temps.p[2] = d_g;
  CU(cudaMalloc(&d_inv, std::max<size_t>(nf, 1) * sizeof(u32)));
  temps.p[3] = d_inv;
  // The table copies go on the stream the build kernels run on (slot 0's, non-blocking, so not
  // ordered after the legacy stream); the host vectors they read outlive the synchronisation
  // at the end of this function.
  cudaStream_t bs = e->slots[0].stream;
  CU(cudaMemcpyAsync(e->d_rho, rho.data(), L * sizeof(u32), cudaMemcpyHostToDevice, bs));
  CU(cudaMemcpyAsync(e->d_fdesc, fdesc.data(), nf * sizeof(u32), cudaMemcpyHostToDevice, bs));
  CU(cudaMemcpyAsync(e->d_sdist, sd.data(), sd.size() * sizeof(u32), cudaMemcpyHostToDevice, bs));
  CU(cudaMemcpyAsync(e->d_tdp, tdp.data(), tdp.size() * sizeof(u32), cudaMemcpyHostToDevice, bs));
  CU(cudaMemcpyAsync(e->d_tde, tde.data(), tde.size() * sizeof(TdEntry), cudaMemcpyHostToDevice, bs));
  std::vector<u64> tdi(tde.size());
  for (size_t i = 0; i < tde.size(); ++i) tdi[i] = tde[i].inv;
  CU(cudaMemcpyAsync(e->d_tdi, tdi.data(), tdi.size() * sizeof(u64), cudaMemcpyHostToDevice, bs));
  std::vector<uint2> tdqm(tdp.size());
  for (size_t i = 0; i < tdp.size(); ++i) tdqm[i] = make_uint2(tdp[i], (u32)((1ull << 32) / tdp[i]));
  CU(cudaMemcpyAsync(e->d_tdqm, tdqm.data(), tdqm.size() * sizeof(uint2), cudaMemcpyHostToDevice, bs));
  CU(cudaMemcpyAsync(d_mods, om.data(), nf * sizeof(u64), cudaMemcpyHostToDevice, bs));
  CU(cudaMemcpyAsync(d_ress, orr.data(), nf * sizeof(u64), cudaMemcpyHostToDevice, bs));
  CU(cudaMemcpyAsync(d_g, og.data(), nf * sizeof(u32), cudaMemcpyHostToDevice, bs));
  CU(cudaMemcpyAsync(d_inv, oinv.data(), nf * sizeof(u32), cudaMemcpyHostToDevice, bs));
  const u64 total = (u64)L * e->ldk;
  k_build_k0<<<(unsigned)((total + 255) / 256), 256, 0, bs>>>(e->d_rho, L, d_mods, d_ress, d_g, d_inv,
                                                              e->d_fdesc, (u32)nf, e->ldk, e->d_K0);
  CU(cudaGetLastError());
  // The strides that get rows: within each phase (covers, then stage-B' primes) the smallest,
  // while their rows fit the budget; the filters of the remaining strides are checked one by one
  // from the first-hit table. The strides are then ordered by how many positions they kill -- the
  // sum over lanes and filters of 1/s where the filter hits the lane (rho == res mod g) -- and the
  // densest covers whose rows fit a slice become the dense strides. Kills are ORed, so the order
  // cannot change a result.
  {
    std::vector<u32> ms;                               // strides with rows, in marking order
    std::vector<int> fmask(nf, -1);
    std::vector<u32> lfil_cov, lfil_siv;
    std::map<u32, std::unordered_map<u32, u32>> lanes_mod;     // g -> (rho mod g -> lanes)
    for (size_t k = 0; k < nf; ++k) {
      auto &h = lanes_mod[og[k]];
      if (h.empty())
        for (u32 l = 0; l < L; ++l) ++h[rho[l] % og[k]];
    }
    std::vector<double> kills(65536, 0.0);
    for (size_t k = 0; k < nf; ++k) {
      const auto &h = lanes_mod[og[k]];
      const auto it = h.find((u32)(orr[k] % og[k]));
      if (it != h.end()) kills[fdesc[k] & 0xFFFFu] += (double)it->second / (double)(fdesc[k] & 0xFFFFu);
    }
    u64 bits = 0;
    u32 dense_rows = PIECE_ROWS;                       // the padding's rows
    for (int phase = 0; phase < 2; ++phase) {
      const size_t f0 = phase ? e->ncov : 0, f1 = phase ? nf : e->ncov;
      std::vector<u32> strides;
      for (size_t k = f0; k < f1; ++k) strides.push_back(fdesc[k] & 0xFFFFu);
      std::sort(strides.begin(), strides.end());
      strides.erase(std::unique(strides.begin(), strides.end()), strides.end());
      const size_t m_first = ms.size();
      for (u32 st : strides) {
        if (bits + st > 8ull * MASK_BYTES_MAX || ms.size() >= STRIDES_MAX) break;
        ms.push_back(st);
        bits += st;
      }
      std::stable_sort(ms.begin() + m_first, ms.end(), [&](u32 x, u32 y) { return kills[x] > kills[y]; });
      if (phase == 0) {
        std::vector<u32> dense, rest;
        for (u32 st : ms) {
          const u32 need = st + PIECE_ROWS - 1;
          const bool fits = dense.size() < DENSE_MAX && dense_rows + need <= SLICE_ROWS_MAX;
          (fits ? dense : rest).push_back(st);
          if (fits) dense_rows += need;
        }
        e->n1 = (u32)dense.size();
        ms = dense;
        ms.insert(ms.end(), rest.begin(), rest.end());
        e->nm_cov = (u32)ms.size();
      }
      std::vector<int> slot_of(65536, -1);
      for (size_t m = m_first; m < ms.size(); ++m) slot_of[ms[m]] = (int)m;
      for (size_t k = f0; k < f1; ++k) {
        const int m = slot_of[fdesc[k] & 0xFFFFu];
        fmask[k] = m;
        if (m < 0) (phase ? lfil_siv : lfil_cov).push_back((u32)k);
      }
    }
    e->nm_all = (u32)ms.size();
    e->n1p = (e->n1 + 7) & ~7u;
    e->slice_rows = (dense_rows + 7) & ~7u;            // a slice is whole 128-byte lines
    e->ngroups = (L + GROUP_LANES - 1) / GROUP_LANES;
    std::vector<uint4> md(e->n1p + e->nm_all - e->n1);
    auto desc = [](u32 st, u32 at) { return make_uint4(st, 0xFFFFFFFFu / st, (u32)((1ull << 32) % st), at); };
    u32 row = PIECE_ROWS, word = 0;
    for (u32 m = 0; m < e->n1; ++m) { md[m] = desc(ms[m], row); row += ms[m] + PIECE_ROWS - 1; }
    for (u32 m = e->n1; m < e->n1p; ++m) md[m] = desc(1, 0);
    e->n2 = e->nm_all;
    for (u32 m = e->n1; m < e->nm_all; ++m) {
      const u32 wd = (ms[m] + 31) / 32;
      if (e->n2 == e->nm_all && ((word + wd + 3) & ~3u) > SIFT_WORDS_MAX) {   // k_sift's copy ends here
        e->n2 = m;
        word = (word + 3) & ~3u;
      }
      md[e->n1p - e->n1 + m] = desc(ms[m], word);
      word += wd;
    }
    e->lane_words = std::max(4u, (word + 3) & ~3u);
    e->nl_cov = (u32)lfil_cov.size();
    e->nl_all = (u32)(lfil_cov.size() + lfil_siv.size());
    std::vector<u32> lfil(lfil_cov);
    lfil.insert(lfil.end(), lfil_siv.begin(), lfil_siv.end());
    int *d_fmask = nullptr;
    const size_t dense_bytes = (size_t)e->ngroups * e->slice_rows * 4 * GROUP_WORDS;
    const size_t lane_bytes = (size_t)L * e->lane_words * sizeof(u32);
    CU(cudaMalloc(&e->d_tdense, dense_bytes));
    CU(cudaMalloc(&e->d_tlane, lane_bytes));
    CU(cudaMalloc(&e->d_mdesc, std::max<size_t>(md.size(), 1) * sizeof(uint4)));
    CU(cudaMalloc(&e->d_lfil, std::max<size_t>(lfil.size(), 1) * sizeof(u32)));
    CU(cudaMalloc(&d_fmask, std::max<size_t>(nf, 1) * sizeof(int)));
    temps.p[4] = d_fmask;
    CU(cudaMemsetAsync(e->d_tdense, 0, dense_bytes, bs));
    CU(cudaMemsetAsync(e->d_tlane, 0, lane_bytes, bs));
    if (!md.empty()) CU(cudaMemcpyAsync(e->d_mdesc, md.data(), md.size() * sizeof(uint4), cudaMemcpyHostToDevice, bs));
    if (!lfil.empty()) CU(cudaMemcpyAsync(e->d_lfil, lfil.data(), lfil.size() * sizeof(u32), cudaMemcpyHostToDevice, bs));
    if (nf) CU(cudaMemcpyAsync(d_fmask, fmask.data(), nf * sizeof(int), cudaMemcpyHostToDevice, bs));
    if (nf && e->nm_all) {
      const u64 tt = (u64)L * nf;
      k_build_rows<<<(unsigned)((tt + 255) / 256), 256, 0, bs>>>(e->d_K0, L, e->ldk, (u32)nf, d_fmask, e->d_mdesc, e->n1,
                                                                 e->n1p, e->slice_rows, e->lane_words,
                                                                 (u32 *)e->d_tdense, e->d_tlane);
      CU(cudaGetLastError());
    }
    double rate[2] = {};
    CU(cudaMalloc(&temps.p[6], sizeof rate));
    CU(cudaMemsetAsync(temps.p[6], 0, sizeof rate, bs));
    k_lane_rate<<<(L + 31) / 32, 32 * RATE_WARPS, 0, bs>>>((const u32 *)e->d_tdense, e->d_tlane, e->d_mdesc, e->n1, e->n1p,
                                                 e->nm_all, e->slice_rows, e->lane_words, L, (double *)temps.p[6]);
    CU(cudaGetLastError());
    CU(cudaMemcpyAsync(rate, temps.p[6], sizeof rate, cudaMemcpyDeviceToHost, bs));
    // Stage B' primes kill squares by their own rule, and moduli past 2^16 are not searched.
    unsigned long long hit = 1;
    if (nf && nf == e->ncov && *std::max_element(om.begin(), om.end()) <= 65536) {
      CU(cudaMalloc(&temps.p[5], sizeof hit));
      CU(cudaMemsetAsync(temps.p[5], 0, sizeof hit, bs));
      k_square_mask<<<(unsigned)std::min<size_t>(nf, 65535), 128, 0, bs>>>(d_mods, d_ress, (u32)nf,
                                                                          (unsigned long long *)temps.p[5]);
      CU(cudaGetLastError());
      CU(cudaMemcpyAsync(&hit, temps.p[5], sizeof hit, cudaMemcpyDeviceToHost, bs));
    }
    CU(cudaStreamSynchronize(bs));
    e->surv_rate = rate[0] / L;
    e->cand_rate = rate[1] / L;
    // a pass of 2^23 full rows holds 60 MB of rows and pieces and, with the tables for wheel 2042040,
    // up to 450 MB of candidates; tables that leave more candidates take shorter passes
    e->pass_rows = (u64)std::min(8388608.0, std::max(4096.0, 32.0 * 2097152.0 / (1.5 * e->cand_rate * L + 1e-9)));
    e->squares = !(hit & 1);
    for (u32 q = 3; q < 64; ++q)
      if (hit >> q & 1) e->sq.push_back(q);
    CU(cudaFuncSetAttribute(k_mark_short, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ROW_SMEM));
    CU(cudaFuncSetAttribute(k_sift, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ROW_SMEM));
  }
  CU(cudaStreamSynchronize(e->slots[0].stream));
  // Stage D's trial division streams its 78 KB prime table once per factorization: ask for
  // the smallest shared-memory carveout that still holds the resident blocks' shared memory,
  // so that the rest of the SM's 256 KB stays L1 and the table stays in it.
  {
    int max_smem = 0;
    CU(cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerMultiprocessor, e->device));
    CU(cudaFuncSetAttribute(k_rung, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(RungBlock)));
    const std::pair<const void *, size_t> resident[] = {{(const void *)k_rung, sizeof(RungBlock)},
                                                        {(const void *)k_probe_rung, 4 * sizeof(RungShared<1>)}};
    for (const auto &[f, bytes] : resident) {
      const int pct = std::min(100, (int)(100.0 * (bytes + 4096) / std::max(max_smem, 1)) + 1);
      CU(cudaFuncSetAttribute(f, cudaFuncAttributePreferredSharedMemoryCarveout, pct));
    }
  }
  // k_mark's shared memory: the attribute is per function and process-wide, so it is the largest
  // size any engine can ask for (DMAX strides), never this engine's own, or a second engine with
  // fewer strides would shrink it under the first; its occupancy sizes the persistent grid.
  const size_t smem = mark_smem(e);
  const size_t smem_max = ((4 * DMAX + 15) & ~15u) + std::max<u32>(SEG_BIG, GROUP * SEG_SMALL) + 16;
  CU(cudaFuncSetAttribute(k_mark<MARK_BLOCK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_max));
  int occ = 0;
  CU(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_mark<MARK_BLOCK>, MARK_BLOCK, smem));
  e->mark_occupancy = std::max(occ, 1);
  return ES_OK;
}

constexpr size_t SERVE_QUEUE_WINDOWS = 1 << 20;   // windows waiting, across requests
constexpr size_t SERVE_BATCH_WINDOWS = 8192;      // windows per batch a worker takes

// Device bytes a request's windows need in a slot: twice what run_device_windows asks for (its capacities
// go in doublings), of at most a pass; the floors that every slot has are not a request's.
static u64 request_bytes(const es_engine *e, const es_schedule &sched, const es_window *w, size_t n) {
  const u64 L = e->classes.size();
  u64 pos = 0, row_pos = 0, rows = 0;
  for (size_t i = 0; i < n; ++i) {
    const u64 p = positions_in(e, w[i].lo, w[i].hi), r = window_rows(sched, e->M, w[i].lo, w[i].hi);
    pos += p;
    rows += r;
    if (r) row_pos += p;
  }
  pos -= row_pos;                                      // those marked by segments
  rows = std::min(rows, e->pass_rows);
  row_pos = std::min(row_pos, rows * L);
  pos += row_pos;
  return 2 * (n * (sizeof(WinDev) + sizeof(WinCount) + 2ull * e->Dq) +
              (rows / PIECE_ROWS + n) * (sizeof(Piece) + 2ull * e->n1p + PIECE_ROWS * sizeof(u32)) +
              chunk_need(e, row_pos) * (32 * sizeof(uint2) + sizeof(u32)) +
              surv_need(e, w, n, pos) * (sizeof(Surv) + 2 * sizeof(u32) + sizeof(RecDev)));
}

// A serving worker owns slot k: whenever its slot is free it takes every queued request
// that fits one batch (continuous batching -- requests that arrive while other batches run
// join the next one), runs the batch on its own stream, and hands each request its windows'
// counters and records. Workers of different slots run their batches concurrently.
static void serve_worker(es_engine *e, int k) {
  cudaSetDevice(e->device);
  Slot *sl = &e->slots[k];
  for (;;) {
    std::vector<Request *> batch;
    {
      std::unique_lock<std::mutex> lk(e->qmu);
      e->qcv.wait(lk, [&] { return e->stopping || !e->queue.empty(); });
      if (e->stopping && e->queue.empty()) return;
      size_t nw = 0;
      // a solo request (es_submit_batch) is a batch of its own, of any size
      while (!e->queue.empty() &&
             (batch.empty() || (!batch[0]->solo && !e->queue.front()->solo &&
                                nw + e->queue.front()->w.size() <= SERVE_BATCH_WINDOWS))) {
        Request *r = e->queue.front();
        e->queue.pop_front();
        nw += r->w.size();
        e->queued_windows -= r->w.size();
        batch.push_back(r);
      }
    }
    std::vector<es_window> wins;
    for (Request *r : batch) wins.insert(wins.end(), r->w.begin(), r->w.end());
    std::vector<es_counters> cnt(wins.size());
    es_records recs{nullptr, 0};
    es_status st = ES_OK;
    std::string err;
    if (!wins.empty()) {
      std::lock_guard<std::mutex> lk(sl->mu);
      st = run_windows(e, sl, wins.data(), wins.size(), ES_SCHED_PERSISTENT, cnt.data(), &recs);
      if (st != ES_OK) { std::lock_guard<std::mutex> el(e->err_mu); err = e->last_error; }
    }
    // split the batch back into its requests (records are sorted by window)
    size_t w0 = 0, r0 = 0;
    for (Request *r : batch) {
      const size_t n = r->w.size();
      r->st = st;
      r->err = err;
      if (st == ES_OK) {
        r->cnt.assign(cnt.begin() + w0, cnt.begin() + w0 + n);
        size_t r1 = r0;
        while (r1 < recs.n && recs.recs[r1].window < w0 + n) ++r1;
        r->recs.assign(recs.recs + r0, recs.recs + r1);
        for (es_record &x : r->recs) x.window -= (uint32_t)w0;
        r0 = r1;
      }
      w0 += n;
    }
    free(recs.recs);
    {
      std::lock_guard<std::mutex> lk(e->qmu);
      for (Request *r : batch) { r->done = true; e->mem_in_use -= r->mem; }
    }
    e->dcv.notify_all();
  }
}

}  // namespace es

using namespace es;

namespace es {
// Probes: copy in, one kernel, copy out. Small and synchronous. The buffer stays with the engine up to
// PROBE_KEEP bytes: an allocation and its release a call took 150 us (the primality of 200 K values
// 366 -> 217 us, 8 K factorizations 828 -> 677).
constexpr size_t PROBE_KEEP = 64u << 20;
template <typename Launch>
static es_status probe(es_engine *e, Slot *sl, size_t count, size_t in_bytes, const void *in, size_t out_bytes,
                       std::vector<std::pair<void *, size_t>> outs, Launch launch) {
  std::lock_guard<std::mutex> lk(sl->mu);
  cudaSetDevice(e->device);
  auto unit = [](size_t b) { return (std::max<size_t>(b, 8) + 255) & ~(size_t)255; };
  size_t total = unit(in_bytes);
  for (const auto &o : outs) total += unit(o.second);
  struct Release {                                   // what is too large to stay, on every return path
    Slot *sl;
    ~Release() {
      if (sl->probe_cap <= PROBE_KEEP) return;
      cudaFree(sl->d_probe);
      sl->d_probe = nullptr;
      sl->probe_cap = 0;
    }
  } release{sl};
  if (total > sl->probe_cap) {
    cudaFree(sl->d_probe);
    sl->d_probe = nullptr;
    sl->probe_cap = 0;
    CU(cudaMalloc(&sl->d_probe, total));
    sl->probe_cap = total;
  }
  void *d_in = sl->d_probe;
  std::vector<void *> d_outs(outs.size(), nullptr);
  size_t at = unit(in_bytes);
  for (size_t i = 0; i < outs.size(); ++i) { d_outs[i] = sl->d_probe + at; at += unit(outs[i].second); }
  // Every copy is queued on the probe's own stream (a non-blocking stream is not ordered after
  // the legacy stream that a plain cudaMemcpy uses), and the host waits for that stream before
  // it reads anything back.
  CU(cudaMemcpyAsync(d_in, in, in_bytes, cudaMemcpyHostToDevice, sl->stream));
  CU(cudaMemsetAsync(sl->d_status, 0, sizeof(u32), sl->stream));
  CU(cudaEventRecord(sl->ev[9], sl->stream));
  launch(d_in, d_outs);
  CU(cudaGetLastError());
  CU(cudaEventRecord(sl->ev[10], sl->stream));
  for (size_t i = 0; i < outs.size(); ++i)
    CU(cudaMemcpyAsync(outs[i].first, d_outs[i], outs[i].second, cudaMemcpyDeviceToHost, sl->stream));
  u32 st = 0;
  CU(cudaMemcpyAsync(&st, sl->d_status, sizeof st, cudaMemcpyDeviceToHost, sl->stream));
  CU(cudaStreamSynchronize(sl->stream));
  sl->timing.total_ms = ev_ms(sl->ev[9], sl->ev[10]);   // the probe kernel alone
  (void)count;
  if (st) return fail(e, ES_ERR_DEVICE_STATUS, "device status:" + status_text(st));
  return ES_OK;
}

}  // namespace es

// ============================================================================ C ABI

extern "C" {

const char *es_status_str(es_status s) {
  switch (s) {
    case ES_OK: return "ok";
    case ES_ERR_ARG: return "invalid argument";
    case ES_ERR_PIN: return "class table digest mismatch";
    case ES_ERR_RANGE: return "range outside floor/ceiling";
    case ES_ERR_FILTERS: return "bad filter file";
    case ES_ERR_CUDA: return "CUDA error";
    case ES_ERR_DEVICE_STATUS: return "device status error";
    case ES_ERR_NOMEM: return "out of memory";
    case ES_ERR_TIMEOUT: return "timeout";
    case ES_ERR_BUSY: return "busy";
  }
  return "unknown status";
}

static thread_local std::string g_open_error;   // why the last es_open on this thread failed

const char *es_last_error(const es_engine *e) { return e ? e->last_error.c_str() : g_open_error.c_str(); }

es_status es_load_filters(const char *path, uint64_t **mods, uint64_t **ress, size_t *n) {
  if (!path || !mods || !ress || !n) return ES_ERR_ARG;
  FILE *fp = fopen(path, "r");
  if (!fp) return ES_ERR_FILTERS;
  std::vector<uint64_t> m, r;
  char line[256];
  while (fgets(line, sizeof line, fp)) {
    unsigned long long a, b;
    if (sscanf(line, "FILTER %llu %llu", &a, &b) == 2) { m.push_back(a); r.push_back(b); }
  }
  fclose(fp);
  if (m.empty()) return ES_ERR_FILTERS;
  *mods = (uint64_t *)malloc(m.size() * sizeof(uint64_t));
  *ress = (uint64_t *)malloc(r.size() * sizeof(uint64_t));
  if (!*mods || !*ress) { free(*mods); free(*ress); return ES_ERR_NOMEM; }
  memcpy(*mods, m.data(), m.size() * sizeof(uint64_t));
  memcpy(*ress, r.data(), r.size() * sizeof(uint64_t));
  *n = m.size();
  return ES_OK;
}

void es_free_u64(uint64_t *p) { free(p); }

es_status es_open(const es_config *cfg, es_engine **out) {
  if (!cfg || !out) return ES_ERR_ARG;
  *out = nullptr;
  es_engine *e = new (std::nothrow) es_engine();
  if (!e) return ES_ERR_NOMEM;
  e->M = cfg->wheel_M ? cfg->wheel_M : 2042040;
  e->mmax = cfg->mmax ? cfg->mmax : 10000;
  e->sieve_p = cfg->sieve_p;
  e->device = cfg->device;
  e->flags = cfg->flags;
  if (e->flags & ES_FLAG_TEST_RHO_BUDGET) e->rho_budget = 64;
  if (e->M < 2 || e->M > 0x7FFFFFFFull) { g_open_error = "wheel modulus must be below 2^31"; delete e; return ES_ERR_ARG; }
  const std::vector<Cover> covers = gen_covers(e->mmax);
  const Wheel w = build_wheel(e->M, gen_wheel_covers(e->M), gen_ucerts(UCERT_RMAX, UCERT_UMAX));
  e->classes = w.classes;
  build_lane_index(e);
  e->wheel_pmin = w.max_pmin;
  for (const Cover &f : covers) e->cover_pmax = std::max(e->cover_pmax, f.pmin);
  e->class_fnv = fnv64_classes(e->classes);
  e->pin = class_pin(e->M);
  if (e->pin && e->class_fnv != e->pin->fnv64) {
    char buf[200];
    snprintf(buf, sizeof buf, "class table digest mismatch at M=%llu -- derived fnv64 %016llx, expected %016llx",
             e->M, e->class_fnv, e->pin->fnv64);
    g_open_error = buf;
    delete e;
    return ES_ERR_PIN;
  }
  if (e->classes.empty()) { delete e; return ES_ERR_ARG; }
  if (cfg->filter_mods) {
    if (!cfg->filter_ress || cfg->n_filters == 0) { delete e; return ES_ERR_FILTERS; }
    e->mods.assign(cfg->filter_mods, cfg->filter_mods + cfg->n_filters);
    e->ress.assign(cfg->filter_ress, cfg->filter_ress + cfg->n_filters);
  } else {
    for (const Cover &f : covers)
      if (e->M % f.mod) { e->mods.push_back(f.mod); e->ress.push_back(f.res); }
  }
  e->ncov = e->mods.size();
  if (e->sieve_p)
    for (u64 q : small_primes(e->sieve_p, e->M)) { e->mods.push_back(q); e->ress.push_back(0); }
  e->filter_fnv = fnv64_filters(e->mods, e->ress, e->ncov);
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev <= e->device || e->device < 0) {
    g_open_error = "no CUDA device " + std::to_string(e->device);
    delete e;
    return ES_ERR_CUDA;
  }
  if (cudaSetDevice(e->device) != cudaSuccess) { g_open_error = "cudaSetDevice failed"; delete e; return ES_ERR_CUDA; }
  cudaDeviceGetAttribute(&e->sm_count, cudaDevAttrMultiProcessorCount, e->device);
  for (Slot &sl : e->slots) {
    if (cudaStreamCreateWithFlags(&sl.stream, cudaStreamNonBlocking) != cudaSuccess ||
        cudaMalloc(&sl.d_ctr, CTR_BYTES) != cudaSuccess ||
        cudaMalloc(&sl.d_status, sizeof(u32)) != cudaSuccess) {
      g_open_error = "stream or counter allocation failed";
      cudaGetLastError();
      es_close(e);
      return ES_ERR_CUDA;
    }
    for (auto &ev : sl.ev) cudaEventCreate(&ev);
  }
  {
    size_t fr = 0, tot = 0;
    cudaMemGetInfo(&fr, &tot);
    e->mem_budget = cfg->mem_budget ? cfg->mem_budget : fr / 4;   // serving admission budget
  }
  const es_status s = build_tables(e);
  if (s != ES_OK) {
    g_open_error = e->last_error;
    es_close(e);
    return s;
  }
  *out = e;
  return ES_OK;
}

es_status es_close(es_engine *e) {
  if (!e) return ES_OK;
  {
    std::lock_guard<std::mutex> lk(e->qmu);
    e->stopping = true;
  }
  e->qcv.notify_all();
  for (std::thread &t : e->workers) t.join();
  {
    // the workers finished every queued request; a poller still inside es_poll has been woken
    // and owns its request until it returns
    std::unique_lock<std::mutex> lk(e->qmu);
    e->dcv.notify_all();
    e->dcv.wait(lk, [&] { return e->pollers == 0; });
  }
  for (auto &kv : e->reqs) delete kv.second;
  cudaSetDevice(e->device);
  for (Slot &sl : e->slots) {
    if (sl.stream) cudaStreamSynchronize(sl.stream);
    drop_graph(&sl);
    cudaFree(sl.d_win); cudaFree(sl.d_cnt); cudaFree(sl.d_Qm);
    cudaFree(sl.d_piece); cudaFree(sl.d_pidx); cudaFree(sl.d_rowinfo); cudaFree(sl.d_cand); cudaFree(sl.d_chunk);
    cudaFree(sl.d_surv); cudaFree(sl.d_primes); cudaFree(sl.d_direct); cudaFree(sl.d_recs);
    cudaFree(sl.d_ctr); cudaFree(sl.d_status); cudaFree(sl.d_hdr); cudaFree(sl.d_probe);
    cudaFreeHost(sl.h_hdr); cudaFreeHost(sl.h_win); cudaFreeHost(sl.h_roww); cudaFreeHost(sl.h_cnt);
    cudaFreeHost(sl.h_ctr); cudaFreeHost(sl.h_status); cudaFreeHost(sl.h_recs);
    for (auto &ev : sl.ev) if (ev) cudaEventDestroy(ev);
    if (sl.stream) cudaStreamDestroy(sl.stream);
  }
  cudaFree(e->d_rho); cudaFree(e->d_fdesc); cudaFree(e->d_sdist); cudaFree(e->d_tdp);
  cudaFree(e->d_K0); cudaFree(e->d_tde); cudaFree(e->d_tdi); cudaFree(e->d_tdqm);
  cudaFree(e->d_tdense); cudaFree(e->d_tlane); cudaFree(e->d_mdesc); cudaFree(e->d_lfil);
  delete e;
  return ES_OK;
}

es_status es_run_window(es_engine *e, uint64_t lo, uint64_t hi, es_counters *out, es_records *recs) {
  if (!e || !out) return ES_ERR_ARG;
  std::lock_guard<std::mutex> lk(e->slots[0].mu);
  cudaSetDevice(e->device);
  const auto t0 = std::chrono::steady_clock::now();
  es_window w{lo, hi};
  memset(out, 0, sizeof *out);
  if (recs) { recs->recs = nullptr; recs->n = 0; }
  const es_status st = run_windows(e, &e->slots[0], &w, 1, ES_SCHED_PERSISTENT, out, recs);
  e->slots[0].timing.host_total_ms = ms_since(t0);
  return st;
}

es_status es_run_batch(es_engine *e, const es_window *w, size_t n, int schedule, es_counters *per_window,
                       es_records *recs) {
  if (!e || (!w && n) || !per_window) return ES_ERR_ARG;
  if (schedule != ES_SCHED_PLAIN && schedule != ES_SCHED_PERSISTENT) return ES_ERR_ARG;
  std::lock_guard<std::mutex> lk(e->slots[0].mu);
  const auto t0 = std::chrono::steady_clock::now();
  cudaSetDevice(e->device);
  memset(per_window, 0, n * sizeof(es_counters));
  if (recs) { recs->recs = nullptr; recs->n = 0; }
  if (n == 0) return ES_OK;
  const es_status st = run_windows(e, &e->slots[0], w, n, schedule, per_window, recs);
  e->slots[0].timing.host_total_ms = ms_since(t0);
  return st;
}

es_status es_free_records(es_records *r) {
  if (!r) return ES_ERR_ARG;
  free(r->recs);
  r->recs = nullptr;
  r->n = 0;
  return ES_OK;
}

static char *put_u64(char *o, unsigned long long v) {
  char b[20];
  int n = 0;
  do { b[n++] = (char)('0' + (int)(v % 10)); v /= 10; } while (v);
  while (n) *o++ = b[--n];
  return o;
}

static char *put_u128(char *o, unsigned long long lo, unsigned long long hi) {
  if (!hi) return put_u64(o, lo);
  const unsigned __int128 v = ((unsigned __int128)hi << 64) | lo;
  const unsigned long long P19 = 10000000000000000000ull;
  const unsigned __int128 q = v / P19;                 // below 2^64 for every u < 2^127
  unsigned long long r = (unsigned long long)(v % P19);
  o = q >> 64 ? put_u128(o, (unsigned long long)q, (unsigned long long)(q >> 64)) : put_u64(o, (unsigned long long)q);
  char b[19];
  for (int i = 18; i >= 0; --i) { b[i] = (char)('0' + (int)(r % 10)); r /= 10; }
  memcpy(o, b, 19);
  return o + 19;
}

size_t es_format_record(const es_record *r, char *buf, size_t cap) {
  if (!r || !buf) return 0;
  char line[192];
  char *o = line;
  auto put = [&](const char *s, size_t n) { memcpy(o, s, n); o += n; };
  if (r->kind == ES_REC_RUNG) {
    put("RUNG ", 5);
    o = put_u64(o, r->p); *o++ = ' ';
    o = put_u64(o, r->a); *o++ = ' ';
    o = put_u64(o, r->b); *o++ = ' ';
    o = put_u128(o, r->c, r->d);
  } else if (r->kind == ES_REC_SOLVED) {
    put("SOLVED ", 7);
    o = put_u64(o, r->p); *o++ = ' ';
    o = put_u64(o, r->a); *o++ = ' ';
    o = put_u64(o, r->b); *o++ = ' ';
    o = put_u64(o, r->c); *o++ = ' ';
    o = put_u64(o, r->d);
  } else if (r->kind == ES_REC_SURVIVOR) {
    put("SURVIVOR ", 9);
    o = put_u64(o, r->p);
  } else {
    return 0;
  }
  *o++ = '\n';
  const size_t k = (size_t)(o - line);
  if (k >= cap) return 0;
  memcpy(buf, line, k);
  buf[k] = 0;
  return k;
}

size_t es_format_summary(const es_engine *e, uint64_t lo, uint64_t hi, const es_counters *c, char *buf, size_t cap) {
  if (!e || !c || !buf) return 0;
  const int k = snprintf(buf, cap,
                         "SUMMARY lo=%llu hi=%llu wheelM=%llu lanes=%zu mmax=%llu ucert_rmax=%u ucert_umax=%u "
                         "wheel_pmin=%llu classes_sha256=%s positions=%llu covered=%llu sieved=%llu mr=%llu "
                         "composite=%llu rung=%llu direct=%llu survivors=%llu\n",
                         (unsigned long long)lo, (unsigned long long)hi, e->M, e->classes.size(), e->mmax,
                         UCERT_RMAX, UCERT_UMAX, e->wheel_pmin, e->pin ? e->pin->sha256 : "unpinned",
                         (unsigned long long)c->positions, (unsigned long long)c->covered,
                         (unsigned long long)c->sieved, (unsigned long long)c->mr, (unsigned long long)c->composite,
                         (unsigned long long)c->rung, (unsigned long long)c->direct,
                         (unsigned long long)c->survivors);
  return (k > 0 && (size_t)k < cap) ? (size_t)k : 0;
}

es_status es_get_schedule(const es_engine *e, es_schedule *o) {
  if (!e || !o) return ES_ERR_ARG;
  *o = e->sched;
  return ES_OK;
}

es_status es_set_schedule(es_engine *e, const es_schedule *s) {
  if (!e || !s) return ES_ERR_ARG;
  if (s->short_max < 1 || s->short_max > es::SEG_SMALL)
    return fail(e, ES_ERR_ARG, "short_max must be in 1.." + std::to_string(es::SEG_SMALL));
  if (s->rung_blocks_per_sm < 1 || s->rung_blocks_per_sm > 16)
    return fail(e, ES_ERR_ARG, "rung_blocks_per_sm must be in 1..16");
  if (s->long_split > 1) return fail(e, ES_ERR_ARG, "long_split must be 0 or 1");
  for (uint32_t r : s->reserved)
    if (r) return fail(e, ES_ERR_ARG, "reserved schedule fields must be zero");
  // every slot idle while the schedule changes; their graphs hold the old launch shapes
  std::vector<std::unique_lock<std::mutex>> locks;
  for (Slot &sl : e->slots) locks.emplace_back(sl.mu);
  cudaSetDevice(e->device);
  {
    std::lock_guard<std::mutex> lk(e->qmu);
    e->sched = *s;
  }
  for (Slot &sl : e->slots) drop_graph(&sl);
  return ES_OK;
}

es_status es_autotune(es_engine *e, const es_window *w, size_t n, int repeats, es_schedule *chosen) {
  if (!e || !w || n == 0 || repeats < 1 || repeats > 1000) return ES_ERR_ARG;
  // {long_split, short_max}: the schedules that launch different work. Stage D's grid is full from four teams an
  // SM on, and with long_split = 1 every window is marked by rows.
  static const uint32_t CAND[][2] = {{1, SEG_SMALL}, {0, SEG_SMALL / 4}, {0, SEG_SMALL / 2}, {0, SEG_SMALL}};
  const es_schedule before = e->sched;
  std::vector<es_counters> base(n), cur(n);
  es_records rbase{nullptr, 0};
  es_schedule best = before;
  double best_ms = 1e300;
  bool first = true;
  es_status st = ES_OK;
  for (const auto &cand : CAND) {
    es_schedule c = before;
    c.long_split = cand[0];
    c.short_max = cand[1];
    c.rung_blocks_per_sm = RUNG_TEAMS;
    if ((st = es_set_schedule(e, &c)) != ES_OK) break;
    double ms = 0;                               // mean device time of the timed runs
    for (int r = 0; r <= repeats && st == ES_OK; ++r) {
      es_records rc{nullptr, 0};
      st = es_run_batch(e, w, n, ES_SCHED_PERSISTENT, cur.data(), &rc);
      if (st != ES_OK) break;
      if (first) {                               // the first run defines the results
        base = cur;
        rbase = rc;
        first = false;
        continue;
      }
      const bool same = memcmp(cur.data(), base.data(), n * sizeof(es_counters)) == 0 && rc.n == rbase.n &&
                        (rc.n == 0 || memcmp(rc.recs, rbase.recs, rc.n * sizeof(es_record)) == 0);
      es_free_records(&rc);
      if (!same) st = fail(e, ES_ERR_DEVICE_STATUS, "autotune: a schedule changed a result");
      // run 0 warms up (graph capture). The mean, not the best, of the timed runs: stage D's
      // time varies from run to run with which walk splits the hardest cofactor first, and
      // the fastest of a few runs rewards a lucky tail rather than a better schedule.
      if (r > 0) ms += e->slots[0].timing.total_ms / repeats;
    }
    if (st != ES_OK) break;
    if (ms < best_ms) { best_ms = ms; best = c; }
  }
  es_free_records(&rbase);
  if (st != ES_OK) { es_set_schedule(e, &before); return st; }
  st = es_set_schedule(e, &best);
  if (st == ES_OK && chosen) *chosen = best;
  return st;
}

es_status es_info(const es_engine *e, es_info_t *o) {
  if (!e || !o) return ES_ERR_ARG;
  memset(o, 0, sizeof *o);
  o->wheel_M = e->M; o->lanes = e->classes.size(); o->wheel_pmin = e->wheel_pmin;
  o->cover_pmax = e->cover_pmax; o->floor = std::max(e->wheel_pmin, e->cover_pmax);
  o->ceiling = DIRECT_PMAX; o->class_fnv64 = e->class_fnv; o->filter_fnv64 = e->filter_fnv;
  o->n_certified = e->ncov; o->n_filters = e->mods.size(); o->mmax = e->mmax;
  o->short_max_limit = es::SEG_SMALL;
  o->pinned = e->pin != nullptr;
  snprintf(o->classes_sha256, sizeof o->classes_sha256, "%s", e->pin ? e->pin->sha256 : "unpinned");
  return ES_OK;
}

es_status es_classes(const es_engine *e, uint64_t *out, size_t cap) {
  if (!e || !out) return ES_ERR_ARG;
  for (size_t i = 0; i < e->classes.size() && i < cap; ++i) out[i] = e->classes[i];
  return ES_OK;
}

es_status es_timing(const es_engine *e, es_timing_t *o) {
  if (!e || !o) return ES_ERR_ARG;
  *o = e->slots[0].timing;
  return ES_OK;
}

es_status es_is_prime_batch(es_engine *e, const uint64_t *n, size_t count, uint8_t *out) {
  if (!e || (!n && count) || (!out && count)) return ES_ERR_ARG;
  if (!count) return ES_OK;
  return probe(e, &e->slots[0], count, count * 8, n, count, {{out, count}}, [&](void *in, std::vector<void *> &o) {
    k_probe_prime<<<e->sm_count * MR_BLOCKS_PER_SM, 256, 0, e->slots[0].stream>>>((const u64 *)in, count, (unsigned char *)o[0]);
  });
}

es_status es_solve_rung_batch(es_engine *e, const uint64_t *p, size_t count, es_record *out, uint8_t *found) {
  if (!e || (!p && count) || (!out && count) || (!found && count)) return ES_ERR_ARG;
  if (!count) return ES_OK;
  return probe(e, &e->slots[0], count, count * 8, p, 0, {{out, count * sizeof(es_record)}, {found, count}},
               [&](void *in, std::vector<void *> &o) {
                 k_probe_rung<<<e->sm_count * 4, TEAM_THREADS, 0, e->slots[0].stream>>>((const u64 *)in, count, (RecDev *)o[0],
                                                                     (unsigned char *)o[1], e->d_tdp, e->d_tdi, e->d_tdqm,
                                                                     e->slots[0].d_status, e->rho_budget);
               });
}

es_status es_solve_direct_batch(es_engine *e, const uint64_t *p, size_t count, es_record *out, uint8_t *found) {
  if (!e || (!p && count) || (!out && count) || (!found && count)) return ES_ERR_ARG;
  if (!count) return ES_OK;
  return probe(e, &e->slots[0], count, count * 8, p, 0, {{out, count * sizeof(es_record)}, {found, count}},
               [&](void *in, std::vector<void *> &o) {
                 k_probe_direct<<<e->sm_count * 4, 32, 0, e->slots[0].stream>>>((const u64 *)in, count, (RecDev *)o[0],
                                                                       (unsigned char *)o[1], e->d_tdp, e->d_tde,
                                                                       e->slots[0].d_status);
               });
}

es_status es_factor_batch(es_engine *e, const uint64_t *n, size_t count, uint64_t *pr, uint8_t *ex, uint8_t *k) {
  if (!e || (!n && count) || (!pr && count) || (!ex && count) || (!k && count)) return ES_ERR_ARG;
  if (!count) return ES_OK;
  return probe(e, &e->slots[0], count, count * 8, n, 0, {{pr, count * MAXF * 8}, {ex, count * MAXF}, {k, count}},
               [&](void *in, std::vector<void *> &o) {
                 k_probe_factor<<<e->sm_count, RUNG_THREADS, 0, e->slots[0].stream>>>((const u64 *)in, count, (u64 *)o[0],
                                                                       (unsigned char *)o[1], (unsigned char *)o[2],
                                                                       e->d_tdp, e->d_tdi, e->slots[0].d_status,
                                                                       e->rho_budget);
               });
}

es_status es_check_records(es_engine *e, const es_record *r, size_t count, uint8_t *ok) {
  if (!e || (!r && count) || (!ok && count)) return ES_ERR_ARG;
  if (!count) return ES_OK;
  return probe(e, &e->slots[0], count, count * sizeof(es_record), r, 0, {{ok, count}},
               [&](void *in, std::vector<void *> &o) {
                 k_probe_check<<<e->sm_count * 4, 256, 0, e->slots[0].stream>>>((const RecDev *)in, count,
                                                                              (unsigned char *)o[0]);
               });
}

static es_status submit(es_engine *e, const es_window *w, size_t n, uint64_t *ticket, bool solo) {
  if (!e || !ticket || (!w && n)) return ES_ERR_ARG;
  *ticket = 0;
  const u64 floor_ = std::max(e->wheel_pmin, e->cover_pmax);
  for (size_t i = 0; i < n; ++i) {                 // refuse what a run would refuse, now
    if (w[i].hi > DIRECT_PMAX) return fail(e, ES_ERR_RANGE, "HI above the stage-E ceiling");
    if (w[i].lo <= floor_) return fail(e, ES_ERR_RANGE, "LO at or below the pmin floor");
  }
  Request *r = new (std::nothrow) Request();
  if (!r) return ES_ERR_NOMEM;
  r->w.assign(w, w + n);
  r->solo = solo;
  es_schedule sched;
  {
    std::lock_guard<std::mutex> lk(e->qmu);            // es_set_schedule writes it under qmu
    sched = e->sched;
  }
  r->mem = request_bytes(e, sched, w, n);
  {
    std::lock_guard<std::mutex> lk(e->qmu);
    if (e->stopping) { delete r; return ES_ERR_ARG; }
    // admission: a bounded queue, and device memory for the request's buffers within the
    // engine's budget (what is queued or in flight counts against it)
    if (e->queued_windows + n > SERVE_QUEUE_WINDOWS || e->mem_in_use + r->mem > e->mem_budget) {
      delete r;
      return fail(e, ES_ERR_BUSY, "admission refused: queue or device-memory budget full");
    }
    if (e->workers.empty())
      for (int k = 1; k <= SERVE_SLOTS; ++k) e->workers.emplace_back(serve_worker, e, k);
    r->ticket = e->next_ticket++;
    e->mem_in_use += r->mem;
    e->queued_windows += n;
    e->reqs[r->ticket] = r;
    e->queue.push_back(r);
    *ticket = r->ticket;
  }
  e->qcv.notify_one();
  return ES_OK;
}

es_status es_submit(es_engine *e, const es_window *w, size_t n, uint64_t *ticket) {
  return submit(e, w, n, ticket, false);
}

es_status es_submit_batch(es_engine *e, const es_window *w, size_t n, uint64_t *ticket) {
  return submit(e, w, n, ticket, true);
}

es_status es_poll(es_engine *e, uint64_t ticket, es_counters *per_window, es_records *recs, int timeout_ms) {
  if (!e) return ES_ERR_ARG;
  if (recs) { recs->recs = nullptr; recs->n = 0; }
  std::unique_lock<std::mutex> lk(e->qmu);
  auto it = e->reqs.find(ticket);
  if (it == e->reqs.end()) return fail(e, ES_ERR_ARG, "unknown ticket");
  Request *r = it->second;
  // One poller per ticket: a second one would read the request while the first deletes it.
  if (r->claimed) return fail(e, ES_ERR_ARG, "ticket is already being polled");
  r->claimed = true;
  ++e->pollers;
  auto ready = [&] { return r->done; };
  bool done = true;
  if (timeout_ms < 0) e->dcv.wait(lk, ready);
  else done = e->dcv.wait_for(lk, std::chrono::milliseconds(timeout_ms), ready);
  --e->pollers;
  if (!done) {
    r->claimed = false;                  // the ticket stays valid; the caller may poll again
    e->dcv.notify_all();
    return ES_ERR_TIMEOUT;
  }
  e->reqs.erase(r->ticket);
  e->dcv.notify_all();                   // es_close may be waiting for the last poller
  lk.unlock();
  const es_status st = r->st;
  if (st == ES_OK) {
    if (per_window) memcpy(per_window, r->cnt.data(), r->cnt.size() * sizeof(es_counters));
    if (recs) {
      recs->n = r->recs.size();
      recs->recs = (es_record *)malloc(std::max<size_t>(r->recs.size(), 1) * sizeof(es_record));
      if (!recs->recs) { delete r; return ES_ERR_NOMEM; }
      memcpy(recs->recs, r->recs.data(), r->recs.size() * sizeof(es_record));
    }
  } else {
    fail(e, st, r->err);
  }
  delete r;
  return st;
}

}  // extern "C"
