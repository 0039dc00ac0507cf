// es_kernels.cuh -- device-side layouts shared by the kernels and the host engine.
#pragma once
#include <cstdint>
#include "es_arith.cuh"

namespace es {

constexpr u16 K0_MISS = 0xFFFF;     // the filter never hits this lane
constexpr int DMAX = 8192;          // distinct strides held in shared memory per CTA

// One scan window as the device sees it. Lane l's positions are p = rho_l + M*K for
// K = Kfirst .. Kfirst + npos - 1, with Kfirst = Q + (rho_l < lo mod M). Segment-marking
// items (k_mark) are (lane, segment) pairs with segments of SEG_BIG positions; they take the
// windows that are not marked by rows (k_mark_short): with es_schedule.long_split = 0, those with
// more than short_max (at most SEG_SMALL) positions in a lane.
constexpr u32 GROUP = 16;
constexpr u32 SEG_SMALL = 128;
constexpr u32 SEG_BIG = 16384;

struct WinDev {
  u64 lo, hi;
  u64 Q;          // lo / M
  u64 item0;      // first marking item of this window in the batch's item space
  u32 lomod;      // lo % M
  u32 G;          // lanes per item (1 or GROUP)
  u32 seg;        // positions per segment
  u32 nseg;       // segments
  u32 lane0;      // first lane of the active range (a multiple of G)
  u32 groups;     // lane groups per segment
};

// Sizes of the batch in flight, read by the marking kernels from device memory so that one
// captured launch sequence (a CUDA graph) serves every batch up to the buffers' capacity.
struct BatchHdr {
  u64 total_items;   // long-window marking items
  u32 nwin, nshort;  // windows; windows marked by rows
  u32 nrows, npieces;
};

// A position that no filter killed: (window, lane, J) is its key in the output order.
struct Surv {
  u64 p;
  u64 J;
  u32 win, lane;
};

// Per-window device counters; covered/sieved/mr are derived on the host from
// positions, alive-after-covers and survivors, which are sums over segments, and the
// composites from the survivors less the primes (rung + direct + unsolved).
struct WinCount {
  unsigned long long positions, after_covers, surv, spare, rung, direct, unsolved, pad;
};

// Device record: the layout of es_record.
struct RecDev {
  u32 kind, win, lane, reserved;
  u64 J, p, a, b, c, d;
};

struct MarkParams {
  const u32 *rho;          // [L] lane classes
  const u16 *K0;           // [L][ldk] first hit K mod s per (lane, filter), or K0_MISS
  const u32 *fdesc;        // [nf] stride s (low 16 bits) | index of s among distinct strides
  const u32 *sdist;        // [D] distinct strides
  const u16 *Qm;           // [nwin][Dq] (lo / M) mod s_d per window (rows of Dq >= D, 16-byte multiples)
  const WinDev *win;       // [nwin]
  u64 *queue;              // work-queue head (persistent schedule)
  Surv *surv;              // survivor list
  unsigned long long *surv_count;
  WinCount *cnt;           // [nwin]
  const BatchHdr *hdr;     // total_items, nwin
  unsigned long long *ctr;
  u64 surv_cap;
  u64 M;
  u32 L, ldk, nf, ncov, D, Dq;
  u32 r_bytes;             // shared bytes for the stride residues (16-aligned)
};

// Marking by rows (k_mark_short). A row is one K of one window: the positions rho_l + M K of all
// lanes l in [la, lb); a piece is at most PIECE_ROWS consecutive rows of one window.
constexpr u32 MASK_BYTES_MAX = 48 * 1024;   // stride table budget per lane (strides past it are not tabled)
constexpr u32 STRIDES_MAX = 512;            // strides with tables, at most
constexpr u32 PIECE_ROWS = 32;
constexpr u32 GROUP_WORDS = 4;              // 32-bit words of a dense row
constexpr u32 GROUP_LANES = 32 * GROUP_WORDS;
constexpr u32 ROW_THREADS = 1024;           // threads of k_mark_short and k_sift, one CTA of each per SM
constexpr u32 DENSE_MAX = 48;     // dense strides, at most
constexpr u32 BULK_COPY = 16384;            // bytes per bulk copy into shared memory
// Shared memory of a CTA (the rest of the 227 KB an SM can give one is static): per warp 64
// candidates of 8 bytes (k_sift: twice); k_mark_short's group slice, or k_sift's stride descriptors
// and lane tables.
constexpr u32 ROW_SMEM = 226 * 1024;
constexpr u32 CAND_SMEM = ROW_THREADS / 32 * 64 * 8;
constexpr u32 SLICE_ROWS_MAX = (ROW_SMEM - CAND_SMEM) / (4 * GROUP_WORDS);
constexpr u32 SIFT_LANES = 8;               // lanes whose tables k_sift holds at a time
constexpr u32 SIFT_WORDS_MAX = (ROW_SMEM - 2 * CAND_SMEM - STRIDES_MAX * 16) / (4 * SIFT_LANES);
static_assert(SLICE_ROWS_MAX < 65536, "slice rows are 16-bit indices");

// A window marked by rows: K0, K0 + 1, .. K0 + nrows - 1, the first from lane la on, the last up
// to lane lb; row0 and piece0 count the rows and pieces of the windows before it.
struct RowWin {
  u64 K0;
  u32 wi, row0, piece0, nrows, la, lb;
};
struct __align__(16) Piece {
  u64 K0;
  u32 row0, win, n, la, lb, pad;
};
// rowinfo: the row's piece and its place in it, and whether the row is cut (la, lb)
constexpr u32 ROW_CUT = 1u << 31, ROW_NONE = ~0u;

// Run counters: [0] k_mark's queue [1] survivors [2] primes [3] direct [4] records [5] k_direct's blocks
// done [6] rung queue (teams) [7] rung primes done [8] board sessions [9] rung queue (warps)
// [10] candidate chunks, [STAMP0 + i] the device clock in ns at the start of k_rows, k_mark_short,
// k_mark, k_mr, k_rung and k_search or k_direct and at the latter's end; then stage D's board.
constexpr u32 STAMP0 = 16, CTR_OUT = 24;
__device__ __forceinline__ void stamp(unsigned long long *ctr, u32 i) {
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    ctr[STAMP0 + i] = t;
  }
}

struct RowParams {
  const u32 *rho;
  const u16 *K0;
  const u32 *fdesc;
  const unsigned char *tdense;   // [ngroups][slice_bytes]: row x of dense stride m at mdesc[m].w + x
  const u32 *tlane;         // [L][lane_words]: bit x of another stride at mdesc.w + x / 32
  const uint4 *mdesc;       // {s, floor((2^32 - 1) / s), 2^32 mod s, first row or word}: n1 dense
                            // strides padded to n1p with rows that hold no bit, then the covers'
                            // others up to nm_cov and stage B''s up to nm_all
  const u32 *lfil;          // filters of strides without tables: covers [0, nl_cov), then B' [nl_cov, nl_all)
  WinDev *win;
  // the run's pinned host staging: header, window descriptors, windows marked by rows
  const BatchHdr *h_hdr;
  const WinDev *h_win;
  const RowWin *h_roww;     // [hdr->nshort]
  unsigned long long *ctr;  // the run's counters (CTR_WORDS), cleared by k_rows
  Piece *piece;             // [hdr->npieces]
  u16 *pidx;                // [npieces][n1p] slice row of the piece's first K per dense stride
  u32 *rowinfo;             // [nrows]
  uint2 *cand;              // [chunk_cap][32] positions the dense strides left: piece, place * GROUP_LANES + lane
  u32 *chunk;               // [chunk_cap] group << 8 | candidates
  unsigned long long *chunk_count;
  Surv *surv;
  unsigned long long *surv_count;
  WinCount *cnt;
  u64 surv_cap, M;
  BatchHdr *hdr;
  u32 *status;
  bool wide;                // K may reach 2^48
  bool squares;             // n^2 passes every cover when n is prime to the nsq primes with these inverses
  u32 nsq, sq_inv[18], sq_lim[18];   // mod 2^32 and quotients of 2^32 - 1 (odd primes below 64)
  u32 L, ldk, ngroups, slice_bytes, lane_words, chunk_cap;
  u32 n1, n1p, n2, nm_cov, nm_all, nl_cov, nl_all;   // the first words of strides [n1, n2) fit SIFT_WORDS_MAX
};

struct BoardSlot;

// Where a run's results go: pinned host memory, written by k_direct.
struct HostOut {
  unsigned long long *ctr;
  u32 *status;
  WinCount *cnt;
  RecDev *recs;
};

struct TailParams {
  unsigned long long *ctr;
  const BatchHdr *hdr;
  HostOut out;
  Surv *surv;
  unsigned long long *surv_count;
  u32 *primes;             // indices into surv
  unsigned long long *prime_count;
  u32 *direct;             // indices into surv, primes that no rung certified
  unsigned long long *direct_count;
  RecDev *recs;
  unsigned long long *rec_count;
  WinCount *cnt;
  const u32 *tdp;          // odd primes < 2^16
  const TdEntry *tde;      // their inverses mod 2^64 and division limits (thread-per-value paths)
  const u64 *tdi;          // their inverses mod 2^64 alone (warp trial division)
  const uint2 *tdqm;       // {d, floor(2^32 / d)} (the rung sieve's residues)
  u32 *status;
  u64 cap;                 // capacity of surv/primes/direct/recs
  unsigned long long *rung_next;      // k_rung's prime queue head, a team per prime (the tail)
  unsigned long long *rung_done;      // primes k_rung has finished
  unsigned long long *help_sessions;  // curve rounds started on the board
  struct BoardSlot *board;            // [BOARD_SLOTS] hard cofactors of a run of few primes
  unsigned long long *rung_next_warp; // k_rung's prime queue head, one warp per prime
  u64 rho_budget;                     // Brent steps per lane before a factorization gives up
};

}  // namespace es
