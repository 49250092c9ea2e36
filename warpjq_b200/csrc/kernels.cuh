// The sm_100a scan kernels.
//
// The hot path of the reference's k_nl_count / k_nl_write / k_build_lines /
// k_eval / DeviceSelect / k_row_len / k_emit chain (warpjq_kernels.cu:
// 1117-1849) as one scan pass plus, for row output, two small passes:
//
//   k_scan      One warp per CTA.  A warp takes the next tile from a work
//               ticket and stages tile + halo into shared memory with one
//               bulk (TMA) copy.  Stage 1 is lane-parallel over 32-byte
//               chunks: each chunk's "special" bytes ('"', '\\', < 0x20)
//               become a bit mask, its newlines line starts.  Stage 2 walks
//               the lines one per lane (walker.cuh), by the run's line
//               template where it fits, else from special byte to special
//               byte of the mask: validation, path
//               resolution, the filter, and either the aggregate or a
//               compact record per selected row (line offset, row length,
//               field spans).
//   k_tail      Group results, the exclusive prefix over the tiles' (rows,
//               bytes, lines) totals, first bad lines and FP totals.
//   k_rows_emit Rows only: copies them in line order from the input to the
//               output.
//
// No host synchronisation happens inside a run and no kernel waits on
// another CTA.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include <algorithm>

#include "../../include/warpjq_ext.h"
#include "../../include/warpjq_kernels.h"
#include "devutil.cuh"
#include "fixsum.cuh"
#include "plan.h"
#include "walker.cuh"

namespace wjq {

constexpr int kThreads = 32;                 // one warp per CTA; each warp owns its tile
constexpr uint32_t kMaxLinesPerPass = 128;   // line-start list capacity per pass
// Register budgets of k_scan (CTAs of one warp per SM), measured per variant
// on 1 GB of the nginx workload: the ungrouped aggregate at 20 (96 registers,
// then 8 bytes of spills: 685 us; at 24, with 144 bytes, 713; at 16, 775; since
// wide tiles note their lines too, 52 bytes and 702 us), the row variant at 20
// and the group-by variant at 16 (128).  What the warps have in
// common is the instruction cache: the body's loops are kept rolled and the
// rare walks out of line, which took the same scan from 840 us to 685 with the
// same work (misses had kept the next cache level 56% busy; 34% then).
constexpr int kScanBlocksPerSM = 20;
constexpr int kScanBlocksPerSMRows = 20;
constexpr int kScanBlocksPerSMGrouped = 16;

// A CTA's line counts and ungrouped aggregate, in shared memory: each round
// of up to 32 lines is reduced in the warp (ballots, warp reductions) and
// lane 0 adds the round's totals here, so no lane keeps accumulators in
// registers through the walk.  Flushed to the run's counters at the end of
// the CTA (or of each tile, in a batch).
struct CtaAcc {
  unsigned long long lines, blank, invalid, type, sel;
  unsigned long long numeric, n_int;
  unsigned long long isum_lo, isum_hi;  // exact 128-bit sum of the integer values
  unsigned long long min_bits, max_bits;
  uint32_t saw;  // a selected line had a non-numeric, non-null value
  uint32_t pad;
  __device__ void clear() {
    lines = blank = invalid = type = sel = numeric = n_int = isum_lo = isum_hi = 0;
    min_bits = ~0ull;
    max_bits = 0;
    saw = 0;
  }
};

static_assert(sizeof(CtaAcc) % 16 == 0, "the template after it is 16-byte aligned");

// Readable bytes kept past a window's data: the end sentinel, the walker's
// word reads after a line's newline, and the last chunk's 32-byte read.
constexpr uint32_t kWinSlack = 64;

// Shared-memory layout of k_scan for tile T and halo H: the window bytes,
// then the special mask (one word per 32-byte chunk, the sentinel's chunk and
// one more included), the CTA's exact FP sum, its counts, the line template,
// the mbarrier the tile copies complete on, the line-start list, and for
// grouped aggregates the group cache.  Nothing is static, so the dynamic size may be raised
// to the device's whole opt-in limit.
__host__ __device__ inline uint32_t scan_win_bytes(uint32_t T, uint32_t H) {
  return (T + H + kWinSlack + 15u) & ~15u;
}
__host__ __device__ inline uint32_t scan_chunk_words(uint32_t T, uint32_t H) {
  return ((T + H) / 32 + 2 + 3) & ~3u;
}
__host__ __device__ inline size_t scan_smem_base(uint32_t T, uint32_t H) {
  size_t s = scan_win_bytes(T, H);
  s += (size_t)scan_chunk_words(T, H) * sizeof(uint32_t);
  s += kFixDigits * sizeof(long long);
  s += sizeof(CtaAcc);
  s += sizeof(Template);
  s += sizeof(unsigned long long);  // the mbarrier of the tile copies
  s += (kMaxLinesPerPass + 2) * sizeof(uint16_t);
  return (s + 15) & ~(size_t)15;
}

// Record of one selected row, appended to the CTA's record arena for k_rows_emit.
struct RowRec {
  unsigned long long line_start;  // absolute offset of the line
  uint32_t line_len;              // without '\n' and without a trailing '\r'
  uint32_t ordinal;               // line index within the tile
  uint32_t local_off;             // row offset within the tile's output
  uint32_t row_len;
  uint32_t pad[2];
  // followed by n_fields x {uint32 off (relative to line), uint32 len|kind<<28|esc<<27}
};
static_assert(sizeof(RowRec) == kRowRecBytes, "row record header size");

// One group key's accumulators, 128 bytes: the counts, the exact integer
// sum and min/max in the first 64, the exact sum of the non-integer values
// (fixsum.cuh) in the second.
struct GroupAcc {
  unsigned long long count, numeric, isum_lo, isum_hi, n_int, min_bits, max_bits;
  double fbig;                // non-integer values of magnitude >= 2^128
  long long fix[kFixDigits];  // the other non-integer values, exactly
};
static_assert(sizeof(GroupAcc) == 128, "group accumulator record");

__device__ __forceinline__ void group_acc_init(GroupAcc &a) {
  a.count = a.numeric = a.isum_lo = a.isum_hi = a.n_int = 0;
  a.min_bits = ~0ull;
  a.max_bits = 0;
  a.fbig = 0.0;
#pragma unroll
  for (int k = 0; k < kFixDigits; k++) a.fix[k] = 0;
}

// Adds a non-integer value to exact limbs (global or shared memory) with
// independent atomics; values too large for the limbs go to *big.
__device__ __forceinline__ void fix_atomic_add(long long *limbs, double *big, double v) {
  const FixParts pr = fix_split(v);
  if (pr.d == -2) {
    atomicAdd(big, v);
    return;
  }
  if (pr.d < 0) return;
#pragma unroll
  for (int k = 0; k < 3; k++)
    if (pr.part[k] && pr.d + k < kFixDigits)
      atomicAdd((unsigned long long *)&limbs[pr.d + k], (unsigned long long)pr.part[k]);
}

// Where a group key's bytes are (the first line that inserted it).
struct GroupKeyDesc {
  unsigned long long off;  // absolute input offset of the key bytes (string: body)
  uint32_t len;
  uint32_t input;           // batch input the key belongs to (0 for one input)
  uint8_t kind;
  uint8_t esc;
  uint8_t pad[6];
};
static_assert(sizeof(GroupKeyDesc) == 24, "group key descriptor");

// A CTA's own record of the first 32 short keys it meets, by their hash (the
// place it names, or the next free one) and bytes, with their accumulators: a key that
// comes again costs no probe of the table in global memory (a slot, the key's
// descriptor and its bytes, one after another) and no global atomics, where
// the hot keys of all CTAs would meet.  Sums and averages keep 16 keys with
// whole accumulators, the others 32 with their first halves.  Entries hold
// keys of one input; a batch's next input starts over.
//
// Once no place is free the record stays as it is and no key asks for one
// (an atomic a place and line, with each key that is not in it: 96 MB of lines
// over 200 keys, scan of max 823 us that way, 480 so; 256 MB over 959,000 keys
// 1,500 and 1,447).
//
// Most rounds are counts, extremes and sums of plain integers: those go by
// 32-bit shared atomics into n, num, lo and hi (a sum's values as two halves;
// for extremes, lo counts the integers), which hold kFoldLines lines before
// they are folded into the accumulators.  (group_by(.path) | count over 500 MB,
// 32 keys: 546 us; with accumulators for 16 key ids and every round's keys
// looked up in the table, 675.)
constexpr uint32_t kKeyCache = 32;       // one lane clears one
constexpr uint32_t kKeyCacheBytes = 24;  // longest key kept
constexpr uint32_t kKeyAccBytes = 2048;
constexpr uint32_t kFoldLines = 32768;   // lo, 65,535 a line at most, holds 65,537
struct KeyCache {
  uint32_t hash[kKeyCache];  // 0: free
  uint32_t meta[kKeyCache];  // length | kind << 24
  uint32_t kid[kKeyCache];
  uint32_t bytes[kKeyCache][kKeyCacheBytes / 4];  // zero past the key's end
  uint32_t n[kKeyCache], num[kKeyCache], lo[kKeyCache], hi[kKeyCache];
  unsigned long long acc[kKeyAccBytes / 8];
  __device__ __forceinline__ GroupAcc &at(uint32_t e, bool whole) {
    return *(GroupAcc *)((uint8_t *)acc + e * (whole ? 128u : 64u));
  }
};
static_assert(offsetof(GroupAcc, fix) == 64, "the first half is all but the limbs");

__host__ __device__ inline size_t scan_smem_bytes(uint32_t T, uint32_t H, bool groups) {
  return scan_smem_base(T, H) + (groups ? sizeof(KeyCache) : 0);
}

struct GroupTable {
  unsigned long long *slots;  // 0 = empty, else (hash << 32) | (key_id + 1)
  uint32_t cap_mask;
  uint32_t key_cap;
  GroupKeyDesc *keys;
  GroupAcc *acc;
};

// Per-tile totals of a rows run.
struct RowTile {
  unsigned long long rec_begin;  // the tile's first record in the record arena
  unsigned long long bytes;      // output bytes of the tile's rows
  uint32_t rows;
  uint32_t pad;
};

// A run's line template in device memory (one per plan of a mixed batch):
// made by the first CTA that can from a line it walked, taken over by the
// others as they see it.  It only decides how fast a line is walked, so no
// result depends on who made it, when, or from which line.
struct TemplateBuf {
  uint32_t state;  // kTmpl*, set to kTmplNone before the run
  uint32_t tries;  // lines that had no template
  uint32_t misses;  // rounds that missed a line by it
  Template t;
};
constexpr uint32_t kTmplNone = 0, kTmplBuilding = 1, kTmplReady = 2, kTmplOff = 3;
// Lines tried before the run goes on without one.  (1 or 64 measure much the same: 96 MB of
// lines, an array in half or nine tenths of them, 197 to 204 us with 1, 209 to 219
// with 4, 209 to 216 with 64; 4 finds one where a few lines of another kind come first.)
constexpr uint32_t kTmplTries = 4;
constexpr uint32_t kTmplMisses = 3;  // rounds that missed a line, past every second one, before a CTA stops using it
// The run gives the template up when more than kTmplDrop tenths of its rounds
// miss a line: such a round walks the template and the line, with the other
// lanes waiting.  k_scan, us, of 600 MB of access-log lines with an optional
// member in some: never given up 0.5% of the lines (15% of the rounds) 518, 1%
// (28%) 562, 2% (48%) 629, 5% (81%) 723; no template 570 to 580.  (Each CTA by
// itself needed some ten rounds to see it: 648 at 2%, 642 at 5%; so 588 and 589.)
constexpr uint32_t kTmplDrop = 3;
constexpr uint32_t kTmplFirst = 64;  // rounds that may miss before that

struct ScanParams {
  const uint8_t *data;
  unsigned long long n;
  uint32_t tile_bytes;
  uint32_t halo_bytes;
  unsigned long long n_tiles;
  RunCounters *ctr;
  TileDesc *tiles;
  // rows mode: per-tile totals and the record arena (rec_cap_per_cta
  // records per CTA, appended over all the CTA's tiles)
  RowTile *row_tiles;
  uint8_t *rec_scratch;
  unsigned long long rec_cap_per_cta;
  GroupTable g;
  // deep-nesting scratch, per CTA
  uint32_t *deep_words;
  unsigned long long deep_levels_per_cta;
  // Batched runs (tile_input null for one input): input i is
  // data[in_start[i], in_end[i]) and owns tiles [in_tile0[i], in_tile0[i+1]);
  // its counters and aggregate go to in_ctr[i].
  const uint32_t *tile_input;
  const unsigned long long *in_start;
  const unsigned long long *in_end;
  const unsigned long long *in_tile0;
  RunCounters *in_ctr;
  uint32_t any_rows;    // a mixed batch one of whose plans prints rows (its
                        // aggregate launches write empty row tiles)
  uint32_t rec_stride;  // bytes per row record (a mixed batch: the largest of its plans')
  // A mixed batch runs as one launch per distinct plan: this launch takes
  // its tiles from tile_list[0, n_list) (null: every tile) by tickets from
  // *ticket (null: ctr->next_tile), and a CTA's records follow those its
  // earlier launches of the batch appended (rec_cursor, one count per CTA,
  // read at the start and written back at the end; null: none).
  const uint32_t *tile_list;
  unsigned long long n_list;
  unsigned long long *ticket;
  unsigned long long *rec_cursor;
  TemplateBuf *tmpl;  // the run's line template (null: none is used)
};

// Rows emission.
struct EmitParams {
  const uint8_t *data;
  // A mixed batch: tile t's rows are rendered by plans[in_plan[tile_input[t]]]
  // (null otherwise: the kernel's own plan).
  const DevPlan *plans;
  const uint32_t *in_plan;
  const uint32_t *tile_input;
  uint32_t rec_stride;
  const RowTile *row_tiles;
  const TileDesc *tiles;
  unsigned long long n_tiles;
  const unsigned long long *block_prefix;  // 3 per block of tiles_per_block tiles
  uint32_t tiles_per_block;
  const uint8_t *recs;
  uint8_t *out;
  unsigned long long out_cap;
  unsigned long long *row_off;   // rows_cap + 1
  unsigned long long *line_idx;  // rows_cap
  unsigned long long rows_cap;
  RunCounters *ctr;
};

// ---------------------------------------------------------------------------
// Group table (open addressing; the key is published with one 64-bit CAS
// that carries its hash and a dense key id whose descriptor was written and
// fenced before the CAS).
// ---------------------------------------------------------------------------

struct KeyRef {
  const uint8_t *p;  // key bytes (string: body)
  uint32_t len;
  uint8_t kind;      // JK_NULL for missing/null keys
  uint8_t esc;
  uint32_t input;    // batch input of the line (keys of different inputs differ)
  unsigned long long abs_off;
};

__device__ __forceinline__ bool key_bytes_equal(const KeyRef &a, const uint8_t *bp, uint32_t blen,
                                                uint8_t besc) {
  if (!a.esc && !besc) {
    if (a.len != blen) return false;
#pragma unroll 1
    for (uint32_t k = 0; k < blen; k++)
      if (a.p[k] != bp[k]) return false;
    return true;
  }
  StrDecoder x(a.p, a.len), y(bp, blen);
#pragma unroll 1
  for (;;) {
    int u = x.next(), w = y.next();
    if (u != w) return false;
    if (u < 0) return true;
  }
}

// The mask of the bytes of a key's word k (of a key of len bytes).
__device__ __forceinline__ uint32_t key_word_mask(uint32_t len, uint32_t k) {
  return 4 * k + 4 <= len ? 0xFFFFFFFFu : 0xFFFFFFFFu >> (8 * (4 * k + 4 - len));
}

// Whether n bytes at a and b are the same: four words of each a turn, their
// loads in flight together.  Up to seven bytes past both are read.
__device__ __forceinline__ bool key_words_equal(const uint8_t *a, const uint8_t *b, uint32_t n) {
  const uint32_t *qa = (const uint32_t *)((uintptr_t)a & ~(uintptr_t)3), *qb = (const uint32_t *)((uintptr_t)b & ~(uintptr_t)3);
  const uint32_t sa = ((uint32_t)(uintptr_t)a & 3u) * 8u, sb = ((uint32_t)(uintptr_t)b & 3u) * 8u;
#pragma unroll 1
  for (uint32_t k = 0; 4 * k < n; k += 4) {
    uint32_t diff = 0;
#pragma unroll
    for (uint32_t i = k; i < k + 4; i++)
      if (4 * i < n)
        diff |= (__funnelshift_r(qa[i], qa[i + 1], sa) ^ __funnelshift_r(qb[i], qb[i + 1], sb)) & key_word_mask(n, i);
    if (diff) return false;
  }
  return true;
}

// The hash of a key's (decoded) bytes, four at a time, zero past the end.
struct KeyHasher {
  uint32_t h = 0x811C9DC5u;
  __device__ __forceinline__ void word(uint32_t w) {
    h = (h ^ w) * 0x9E3779B1u;
    h ^= h >> 15;
  }
  __device__ __forceinline__ uint32_t done(uint32_t len, uint32_t kind, uint32_t input) {
    h ^= len * 0x85EBCA6Bu ^ kind * 0xC2B2AE35u ^ input * 0x27D4EB2Fu;
    h = (h ^ (h >> 16)) * 0x7FEB352Du;
    h ^= h >> 15;
    return h ? h : 1u;
  }
};

// The bytes of a key of up to kKeyCacheBytes at w[off, off + len) of a window,
// zero past its end.
__device__ __forceinline__ void key_words(const uint8_t *w, uint32_t off, uint32_t len,
                                          uint32_t kw[kKeyCacheBytes / 4]) {
  const uint32_t *q = (const uint32_t *)w + (off >> 2);
  const uint32_t sh = (off & 3u) * 8u;
  uint32_t lo = q[0];
#pragma unroll
  for (uint32_t k = 0; k < kKeyCacheBytes / 4; k++) {
    const uint32_t hi = q[k + 1];
    kw[k] = 4 * k < len ? __funnelshift_r(lo, hi, sh) & key_word_mask(len, k) : 0u;
    lo = hi;
  }
}

// kcache without keys.
__device__ __noinline__ void keys_clear(KeyCache &c, bool whole, int lane) {
  __syncwarp();
  c.hash[lane] = c.n[lane] = c.num[lane] = c.lo[lane] = c.hi[lane] = 0;
  if (whole) {
    if (lane < (int)kKeyCache / 2) group_acc_init(c.at(lane, true));
  } else {
    GroupAcc &a = c.at(lane, false);
    a.count = a.numeric = a.isum_lo = a.isum_hi = a.n_int = 0;
    a.min_bits = ~0ull;
    a.max_bits = 0;
    a.fbig = 0.0;
  }
  __syncwarp();
}

// The 32-bit sums into the accumulators they belong to.
__device__ __noinline__ void keys_fold(KeyCache &c, bool whole, int lane) {
  __syncwarp();
  if (c.n[lane]) {
    GroupAcc &a = c.at(lane, whole);
    a.count += c.n[lane];
    a.numeric += c.num[lane];
    a.n_int += whole ? c.num[lane] : c.lo[lane];
    if (whole) {
      const unsigned long long x = c.lo[lane] + ((unsigned long long)c.hi[lane] << 16), lo = a.isum_lo + x;
      a.isum_hi += lo < x ? 1ull : 0ull;
      a.isum_lo = lo;
    }
    c.n[lane] = c.num[lane] = c.lo[lane] = c.hi[lane] = 0;
  }
  __syncwarp();
}

// Adds kcache's accumulators to the keys' global records.
__device__ __noinline__ void keys_flush(KeyCache &c, const GroupTable &g, bool whole, int lane) {
  keys_fold(c, whole, lane);
  if (lane >= (int)(whole ? kKeyCache / 2 : kKeyCache) || !c.hash[lane]) return;
  const GroupAcc &x = c.at(lane, whole);
  GroupAcc &a = g.acc[c.kid[lane]];
  if (x.count) atomicAdd(&a.count, x.count);
  if (x.numeric) {
    atomicAdd(&a.numeric, x.numeric);
    atomicMin(&a.min_bits, x.min_bits);
    atomicMax(&a.max_bits, x.max_bits);
  }
  if (x.n_int) {
    const unsigned long long old = atomicAdd(&a.isum_lo, x.isum_lo);
    const unsigned long long carry = (old + x.isum_lo) < old ? 1ull : 0ull;
    if (x.isum_hi + carry) atomicAdd(&a.isum_hi, x.isum_hi + carry);
    atomicAdd(&a.n_int, x.n_int);
  }
  if (whole) {  // whatever numeric says: a line that led the key's round may have counted in the global record
#pragma unroll 1
    for (int d = 0; d < kFixDigits; d++)
      if (x.fix[d]) atomicAdd((unsigned long long *)&a.fix[d], (unsigned long long)x.fix[d]);
    if (x.fbig != 0.0) atomicAdd(&a.fbig, x.fbig);
  }
}

// Any key, byte by byte: the same hash for the same decoded bytes.
__device__ __noinline__ uint32_t hash_key_far(const uint8_t *p, uint32_t len, bool esc, uint32_t kind,
                                              uint32_t input) {
  KeyHasher x;
  uint32_t w = 0, n = 0;
  auto put = [&](uint32_t c) {
    w |= c << (8 * (n & 3u));
    if ((++n & 3u) == 0) {
      x.word(w);
      w = 0;
    }
  };
  if (esc) {
    StrDecoder d(p, len);
#pragma unroll 1
    for (int c; (c = d.next()) >= 0;) put((uint32_t)c);
  } else {
#pragma unroll 1
    for (uint32_t k = 0; k < len; k++) put(p[k]);
  }
  if (n & 3u) x.word(w);
  return x.done(n, kind, input);
}

// Returns the key id, or 0xFFFFFFFF when the table is full (the overflow flag
// is raised and the run is repeated with a bigger table).
__device__ __noinline__ uint32_t group_find_or_insert(const ScanParams &sp, const KeyRef &k, uint32_t h) {
  const GroupTable &g = sp.g;
  uint32_t pos = h & g.cap_mask;
  uint32_t mine = 0xFFFFFFFFu;
#pragma unroll 1
  for (uint32_t probe = 0; probe <= g.cap_mask; probe++) {
    unsigned long long w = *(volatile unsigned long long *)&g.slots[pos];
    if (w == 0) {
      if (mine == 0xFFFFFFFFu) {
        mine = atomicAdd(&sp.ctr->n_keys, 1u);
        if (mine >= g.key_cap) {
          atomicOr(&sp.ctr->overflow, 4u);
          return 0xFFFFFFFFu;
        }
        GroupKeyDesc d = {};
        d.off = k.abs_off;
        d.len = k.len;
        d.input = k.input;
        d.kind = k.kind;
        d.esc = k.esc;
        g.keys[mine] = d;
        group_acc_init(g.acc[mine]);  // a key's accumulators start when it gets its id
        __threadfence();
      }
      unsigned long long want = ((unsigned long long)h << 32) | (mine + 1ull);
      unsigned long long old = atomicCAS(&g.slots[pos], 0ull, want);
      if (old == 0) return mine;
      w = old;
    }
    if ((uint32_t)(w >> 32) == h) {
      uint32_t kid = (uint32_t)w - 1;
      __threadfence();
      const GroupKeyDesc d = g.keys[kid];
      if (d.kind == k.kind && d.input == k.input) {
        // by words, unless that would read past the input (96 MB of lines over
        // 200 keys of 40 bytes: scan 547 us a byte a step, 462 so)
        const unsigned long long end = sp.tile_input ? sp.in_end[k.input] : sp.n;
        const bool words = !k.esc && !d.esc && max(k.abs_off, d.off) + d.len + 7 <= end;
        if (words ? k.len == d.len && key_words_equal(k.p, sp.data + d.off, d.len)
                  : key_bytes_equal(k, sp.data + d.off, d.len, d.esc))
          return kid;
      }
    }
    pos = (pos + 1) & g.cap_mask;
  }
  atomicOr(&sp.ctr->overflow, 4u);
  return 0xFFFFFFFFu;
}

// ---------------------------------------------------------------------------
// Row rendering.
// ---------------------------------------------------------------------------

__device__ __forceinline__ uint32_t csv_cell_len(const uint8_t *p, uint32_t n, bool decode) {
  // RFC 4180 quoting as output.rs:45-61 does it, over raw or decoded bytes.
  uint32_t len = 0, quotes = 0;
  bool need = false;
  if (!decode) {
#pragma unroll 1
    for (uint32_t k = 0; k < n; k++) {
      uint32_t c = p[k];
      if (c == '"') quotes++;
      if (c == ',' || c == '"' || c == '\n' || c == '\r') need = true;
    }
    len = n;
  } else {
    StrDecoder d(p, n);
#pragma unroll 1
    for (int c; (c = d.next()) >= 0;) {
      len++;
      if (c == '"') quotes++;
      if (c == ',' || c == '"' || c == '\n' || c == '\r') need = true;
    }
  }
  return need ? len + quotes + 2 : len;
}

__device__ __forceinline__ uint32_t csv_cell_write(uint8_t *dst, const uint8_t *p, uint32_t n,
                                                   bool decode, uint32_t expect_len) {
  // expect_len tells whether quoting applies (it differs from the bare length).
  uint32_t w = 0;
  uint32_t bare = 0;
  if (!decode) bare = n;
  else {
    StrDecoder d(p, n);
#pragma unroll 1
    while (d.next() >= 0) bare++;
  }
  bool quote = expect_len != bare;
  if (quote) dst[w++] = '"';
  if (!decode) {
#pragma unroll 1
    for (uint32_t k = 0; k < n; k++) {
      if (quote && p[k] == '"') dst[w++] = '"';
      dst[w++] = p[k];
    }
  } else {
    StrDecoder d(p, n);
#pragma unroll 1
    for (int c; (c = d.next()) >= 0;) {
      if (quote && c == '"') dst[w++] = '"';
      dst[w++] = (uint8_t)c;
    }
  }
  if (quote) dst[w++] = '"';
  return w;
}

// Length of a value cell in CSV mode (output.rs:65-81).
__device__ __forceinline__ uint32_t csv_value_len(const uint8_t *line, const SlotVal &s) {
  if (s.kind == JK_MISSING || s.kind == JK_NULL) return 0;
  if (s.kind == JK_STR) return csv_cell_len(line + s.off + 1, s.len - 2, s.esc);
  return csv_cell_len(line + s.off, s.len, false);
}

// Computes the row length of a selected line.
__device__ __forceinline__ uint32_t row_length(const DevPlan &P, const uint8_t *line,
                                               uint32_t line_len, const SlotVal *slots) {
  switch (P.output_kind) {
    case 0:  // passthrough (output.rs:204-217)
      return (P.csv_mode ? csv_cell_len(line, line_len, false) : line_len) + 1;
    case 1: {  // single value (output.rs:220-231)
      const SlotVal &s = slots[P.out_slot];
      if (P.csv_mode) return csv_value_len(line, s) + 1;
      return (s.kind == JK_MISSING ? 4 : s.len) + 1;
    }
    default: {  // projection (output.rs:234-264, prefixes rendered by lower.rs:63-87)
      uint32_t len = P.suffix_len + 1;
      for (uint32_t f = 0; f < P.n_fields; f++) {
        const SlotVal &s = slots[P.field_slot[f]];
        len += P.prefix_len[f];
        if (P.csv_mode) len += csv_value_len(line, s);
        else len += s.kind == JK_MISSING ? 4 : s.len;
      }
      return len;
    }
  }
}

// Rows are copied by groups of kEmitLanes lanes, a row a group.
constexpr uint32_t kEmitLanes = 8;

// Copies n bytes with one group (lane g of it): whole aligned words of the
// output, each from the two source words it straddles, four a lane in flight,
// and single bytes at both ends.  No word past the source's last is read.
__device__ __forceinline__ void group_copy(uint8_t *dst, const uint8_t *src, uint32_t n, uint32_t g) {
  const uint32_t head = min(n, (uint32_t)(-(uintptr_t)dst & 3u));
  const uint32_t sh = (uint32_t)((uintptr_t)(src + head) & 3u) * 8u;
  const uint32_t *sw = (const uint32_t *)((uintptr_t)(src + head) & ~(uintptr_t)3);
  uint32_t *dw = (uint32_t *)(dst + head);
  // output word k needs source words k and k + 1, which must end within it
  const uint32_t avail = (uint32_t)((uintptr_t)(src + n) - (uintptr_t)sw) / 4u;
  const uint32_t words = avail > 1u && n > head ? min((n - head) / 4u, avail - 1u) : 0u;
#pragma unroll 1
  for (uint32_t k0 = g; k0 < words; k0 += 4 * kEmitLanes) {
    uint32_t x[4];
#pragma unroll
    for (uint32_t j = 0; j < 4; j++) {
      const uint32_t k = k0 + j * kEmitLanes;
      x[j] = k < words ? __funnelshift_r(__ldg(sw + k), __ldg(sw + k + 1), sh) : 0u;
    }
#pragma unroll
    for (uint32_t j = 0; j < 4; j++) {
      const uint32_t k = k0 + j * kEmitLanes;
      if (k < words) dw[k] = x[j];
    }
  }
  if (g < head) dst[g] = src[g];
#pragma unroll 1
  for (uint32_t k = head + 4 * words + g; k < n; k += kEmitLanes) dst[k] = src[k];
}

// Writes a row of cells or values, one thread: a value, or a projection's
// prefixes and values, as CSV (output.rs:45-81) or JSON; or a whole line as
// one CSV cell.
__device__ __forceinline__ void emit_row(const DevPlan &P, const uint8_t *line, const RowRec &r,
                                         const uint32_t *fields, uint8_t *dst) {
  uint32_t w = 0;
  if (P.output_kind == 0) {
    w = csv_cell_write(dst, line, r.line_len, false, r.row_len - 1);
    dst[w] = '\n';
    return;
  }
  const bool proj = P.output_kind == 2;
  const uint32_t nf = proj ? P.n_fields : 1;
#pragma unroll 1
  for (uint32_t f = 0; f < nf; f++) {
    const uint32_t off = fields[2 * f], lk = fields[2 * f + 1];
    const uint32_t kind = lk >> 28, esc = (lk >> 27) & 1, len = lk & 0x07FFFFFFu;
    const uint8_t *vp = line + off;
    if (proj) {
      const uint32_t n = P.prefix_len[f], at = P.prefix_off[f];
      for (uint32_t k = 0; k < n; k++) dst[w + k] = P.blob[at + k];
      w += n;
    }
    if (!P.csv_mode) {
      if (kind == JK_MISSING) {
        dst[w] = 'n';
        dst[w + 1] = 'u';
        dst[w + 2] = dst[w + 3] = 'l';
        w += 4;
      } else {
#pragma unroll 4
        for (uint32_t k = 0; k < len; k++) dst[w + k] = vp[k];
        w += len;
      }
    } else if (kind != JK_MISSING && kind != JK_NULL) {
      const bool str = kind == JK_STR;
      const uint8_t *cp = str ? vp + 1 : vp;
      const uint32_t n = str ? len - 2 : len;
      w += csv_cell_write(dst + w, cp, n, str && esc, csv_cell_len(cp, n, str && esc));
    }
  }
  if (proj && !P.csv_mode) {
    const uint32_t n = P.suffix_len, at = P.suffix_off;
    for (uint32_t k = 0; k < n; k++) dst[w + k] = P.blob[at + k];
    w += n;
  }
  dst[w] = '\n';
}

// emit_row for JSON values and projections by a group of lanes (lane g of it).
__device__ __forceinline__ void emit_row_group(const DevPlan &P, const uint8_t *line, const uint32_t *fields,
                                               uint8_t *dst, uint32_t g) {
  uint32_t w = 0;
  auto text = [&](uint32_t at, uint32_t n) {  // of the plan's
#pragma unroll 1
    for (uint32_t k = g; k < n; k += kEmitLanes) dst[w + k] = P.blob[at + k];
    w += n;
  };
  const bool proj = P.output_kind == 2;
  const uint32_t nf = proj ? P.n_fields : 1;
#pragma unroll 1
  for (uint32_t f = 0; f < nf; f++) {
    const uint32_t off = fields[2 * f], lk = fields[2 * f + 1], len = lk & 0x07FFFFFFu;
    if (proj) text(P.prefix_off[f], P.prefix_len[f]);
    if (lk >> 28 == JK_MISSING) {
      if (g < 4) dst[w + g] = (uint8_t)(0x6C6C756Eu >> (8 * g));  // "null"
      w += 4;
    } else {
      group_copy(dst + w, line + off, len, g);
      w += len;
    }
  }
  if (proj) text(P.suffix_off, P.suffix_len);
  if (g == 0) dst[w] = '\n';
}

// ---------------------------------------------------------------------------
// The scan kernel.
// ---------------------------------------------------------------------------

// The 128-bit sum over the lanes of `grp` of their signed 64-bit values
// (0 where `on` is false): three parts of at most 22 bits, which cannot
// overflow 32 bits over 32 lanes, recombined with the negatives' borrow.
__device__ __forceinline__ void group_sum128(unsigned grp, bool on, long long v, unsigned long long &lo,
                                             unsigned long long &hi) {
  const unsigned long long u = on ? (unsigned long long)v : 0ull;
  const uint32_t p0 = __reduce_add_sync(grp, (uint32_t)(u & 0x1FFFFFu));
  const uint32_t p1 = __reduce_add_sync(grp, (uint32_t)((u >> 21) & 0x1FFFFFu));
  const uint32_t p2 = __reduce_add_sync(grp, (uint32_t)(u >> 42));
  const uint32_t nneg = __popc(__ballot_sync(0xffffffffu, on && v < 0) & grp);
  const unsigned __int128 t = (unsigned __int128)p0 + ((unsigned __int128)p1 << 21) +
                              ((unsigned __int128)p2 << 42) - ((unsigned __int128)nneg << 64);
  lo = (unsigned long long)t;
  hi = (unsigned long long)(t >> 64);
}

// The extreme (min or max) over the lanes of `grp` of 64-bit keys (lanes
// with `on` false hold none): the high words first, then the low words of
// the lanes holding the extreme high word.
__device__ __forceinline__ unsigned long long group_extreme(unsigned grp, bool on, unsigned long long ob,
                                                            bool mn) {
  const uint32_t none = mn ? 0xFFFFFFFFu : 0u;
  const uint32_t h = on ? (uint32_t)(ob >> 32) : none;
  const uint32_t eh = mn ? __reduce_min_sync(grp, h) : __reduce_max_sync(grp, h);
  const uint32_t l = (on && h == eh) ? (uint32_t)ob : none;
  const uint32_t el = mn ? __reduce_min_sync(grp, l) : __reduce_max_sync(grp, l);
  return ((unsigned long long)eh << 32) | el;
}

// Adds the warp's fractional values (of the lanes with `on`) to the limbs in
// the CTA's shared memory.  Values of like magnitude start at the same limb:
// then each of their three parts is summed in the warp (a part's 64 bits as
// two 16-bit pieces and a sign, which cannot overflow over 32 lanes) and one
// lane adds the sums; adding lane by lane, every lane waits for the others at
// the same three limbs (avg over 500 MB of lines: 499 us so, 390 reduced).
__device__ __forceinline__ void warp_fix_add(long long *limbs, double *big, bool on, double v, int lane) {
  FixParts pr;
  pr.d = -1;
  if (on) pr = fix_split(v);
  const unsigned m = __ballot_sync(0xffffffffu, pr.d != -1);
  if (!m) return;
  const int d = __shfl_sync(0xffffffffu, pr.d, __ffs(m) - 1);
  if (d >= 0 && d + 2 < kFixDigits && __all_sync(0xffffffffu, pr.d == -1 || pr.d == d)) {
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const unsigned long long u = pr.d == -1 ? 0ull : (unsigned long long)pr.part[k];
      const uint32_t lo = __reduce_add_sync(0xffffffffu, (uint32_t)u & 0xFFFFu);
      const uint32_t hi = __reduce_add_sync(0xffffffffu, (uint32_t)u >> 16);
      const uint32_t neg = __popc(__ballot_sync(0xffffffffu, (long long)u < 0));
      if (lane == 0)
        limbs[d + k] += (long long)((unsigned long long)lo + ((unsigned long long)hi << 16) -
                                    ((unsigned long long)neg << 32));
    }
  } else if (on) {
    fix_atomic_add(limbs, big, v);
  }
  __syncwarp();
}

// One-CTA mbarrier (a tile's bulk copy completes on it) and the 1-D bulk
// (TMA) copy from this GPU's own global memory into shared memory.  The
// copy is single-CTA, with no cluster multicast.
constexpr uint32_t kWaitLimit = 1u << 22;  // try_wait rounds before a wait gives up

__device__ __forceinline__ void mbar_init(uint32_t bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(bar) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
}

// Issued by one lane: expects `bytes` (a multiple of 16, src and dst 16-byte
// aligned) on the barrier, then starts the copy.  The proxy fence orders the
// warp's earlier generic reads of `dst` before the copy's writes.
__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes, uint32_t bar) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(d),
      "l"(src), "r"(bytes), "r"(bar)
      : "memory");
}

// Hint: bring `bytes` (a multiple of 16, src 16-byte aligned) of this GPU's
// global memory into L2; nothing waits for it.
__device__ __forceinline__ void l2_prefetch(const void *src, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;\n" ::"l"(src), "r"(bytes) : "memory");
}

// Waits (bounded) for the barrier's phase of parity `phase` to complete.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t phase) {
  for (uint32_t it = 0; it < kWaitLimit; it++) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(bar), "r"(phase)
        : "memory");
    if (done) return true;
  }
  return false;
}

// Exclusive warp scan of (a, b) in lane order, with the warp totals.
__device__ __forceinline__ void warp_scan2(uint32_t a, unsigned long long b, uint32_t &ea,
                                           unsigned long long &eb, uint32_t &ta,
                                           unsigned long long &tb) {
  const int lane = threadIdx.x & 31;
  uint32_t ia = a;
  unsigned long long ib = b;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    uint32_t xa = __shfl_up_sync(0xffffffffu, ia, d);
    unsigned long long xb = __shfl_up_sync(0xffffffffu, ib, d);
    if (lane >= d) {
      ia += xa;
      ib += xb;
    }
  }
  ea = ia - a;
  eb = ib - b;
  ta = __shfl_sync(0xffffffffu, ia, 31);
  tb = __shfl_sync(0xffffffffu, ib, 31);
}

// Adds the CTA's counts and (ungrouped) aggregate to `dst` and clears them;
// `also` (a batch's totals, may be null) receives the line counts too.  The
// non-integer values' exact sum, gathered in the CTA's shared limbs
// `cta_fix`, goes into dst's limbs (and the shared limbs are cleared).
__device__ __noinline__ void flush_counts(RunCounters *dst, RunCounters *also, const DevPlan &P, bool rows,
                                          int lane, CtaAcc *acc, long long *cta_fix) {
  __syncwarp();
  if (lane == 0) {
    for (RunCounters *c : {dst, also}) {
      if (!c) continue;
      if (acc->lines) atomicAdd(&c->n_lines, acc->lines);
      if (acc->blank) atomicAdd(&c->n_blank, acc->blank);
      if (acc->invalid) atomicAdd(&c->n_invalid, acc->invalid);
      if (acc->type) atomicAdd(&c->n_type_error, acc->type);
      if (acc->sel) atomicAdd(&c->n_selected, acc->sel);
    }
    if (!rows && P.group_slot < 0 && P.output_kind == 3) {
      if (acc->sel) atomicAdd(&dst->agg_count, acc->sel);  // an ungrouped aggregate counts every selected line
      if (acc->numeric) atomicAdd(&dst->agg_numeric, acc->numeric);
      if (acc->n_int) atomicAdd(&dst->agg_n_int, acc->n_int);
      const unsigned long long lo = acc->isum_lo, hi = acc->isum_hi;
      if (lo || hi) {
        const unsigned long long old = atomicAdd(&dst->agg_isum_lo, lo);
        const unsigned long long carry = (old + lo) < old;
        if (hi + carry) atomicAdd(&dst->agg_isum_hi, hi + carry);
      }
      if (acc->numeric) {
        atomicMin(&dst->agg_min_bits, acc->min_bits);
        atomicMax(&dst->agg_max_bits, acc->max_bits);
      }
    }
    if (!rows && acc->saw) atomicOr(&dst->agg_saw_non_numeric, 1u);
    acc->clear();
  }
  if (!rows && P.group_slot < 0 && P.output_kind == 3 && lane < kFixDigits) {
    const long long v = cta_fix[lane];
    cta_fix[lane] = 0;
    if (v) atomicAdd((unsigned long long *)&dst->fix[lane], (unsigned long long)v);
  }
  __syncwarp();
}

// The first '\n' of d[q, end), or end: the end of a line longer than its window,
// looked for sixteen bytes a load (96 MB of lines of 200 KB: scan 13.2 ms; a byte
// a load, one waiting for the last, 34.7).
__device__ __noinline__ unsigned long long far_newline(const uint8_t *d, unsigned long long q, unsigned long long end) {
#pragma unroll 1
  for (; q < end && ((uintptr_t)(d + q) & 15u); q++)
    if (d[q] == '\n') return q;
  for (; q + 16 <= end; q += 16) {
    const uint4 v = *(const uint4 *)(d + q);
    if (flags_newline(v.x) | flags_newline(v.y) | flags_newline(v.z) | flags_newline(v.w)) break;
  }
#pragma unroll 1
  while (q < end && d[q] != '\n') q++;
  return q;
}

// One more round missed a line by the template, in a tile of n_lines lines:
// whether the run is better off without it.  `next` is the CTA's next ticket.
__device__ __noinline__ bool template_missed(TemplateBuf *t, unsigned long long next, uint32_t n_lines) {
  const unsigned long long m = atomicAdd(&t->misses, 1u) + 1ull;
  if (*(volatile uint32_t *)&t->state == kTmplOff) return true;
  // tiles walked by it: all that are taken, but every CTA's first and next
  const unsigned long long taken = 2ull * gridDim.x, tiles = next > taken ? next - taken : 0ull;
  if (10 * m <= 10 * kTmplFirst + kTmplDrop * tiles * ((n_lines + 31u) >> 5)) return false;
  atomicExch(&t->state, kTmplOff);
  return true;
}

// The plan is a kernel parameter (constant bank): fields at fixed offsets
// are instruction operands, and no plan read goes through global memory.
// kGroups: the group-by path is compiled in (grouped aggregates); without
// it the kernel is lighter for every other query.
template <bool kRows, bool kGroups = false>
__global__ void __launch_bounds__(kThreads, kGroups ? kScanBlocksPerSMGrouped : (kRows ? kScanBlocksPerSMRows : kScanBlocksPerSM))
    k_scan(const __grid_constant__ ScanParams sp, const __grid_constant__ DevPlan plan) {
  extern __shared__ __align__(16) uint8_t smem[];
  const DevPlan &P = plan;
  const uint32_t T = sp.tile_bytes, H = sp.halo_bytes;
  const uint32_t nwords = scan_chunk_words(T, H);
  uint8_t *win = smem;                                              // window bytes (+ slack)
  uint32_t *smask = (uint32_t *)(smem + scan_win_bytes(T, H));      // special bytes per chunk
  long long *cta_fix = (long long *)(smask + nwords);               // the CTA's exact FP sum
  CtaAcc *acc = (CtaAcc *)(cta_fix + kFixDigits);                   // the CTA's counts and aggregate
  Template *tmpl = (Template *)(acc + 1);                           // the run's line template, once seen
  unsigned long long *s_bar = (unsigned long long *)(tmpl + 1);      // tile copies' mbarrier
  uint16_t *lstart = (uint16_t *)(s_bar + 1);                       // kMaxLinesPerPass + 2
  KeyCache *kcache = (KeyCache *)(smem + scan_smem_base(T, H));      // grouped aggregates only
  const bool whole = P.agg_kind == WARPJQ_AGG_SUM || P.agg_kind == WARPJQ_AGG_AVG;
  const uint32_t n_places = whole ? kKeyCache / 2 : kKeyCache;

  const int lane = threadIdx.x;
  const uint32_t rec_stride = sp.rec_stride;
  uint8_t *my_recs = sp.rec_scratch + (unsigned long long)blockIdx.x * sp.rec_cap_per_cta * rec_stride;
  DeepStack deep;
  deep.words = sp.deep_words + (unsigned long long)blockIdx.x * (sp.deep_levels_per_cta / 32);
  deep.cap_levels = sp.deep_levels_per_cta;

  // records this CTA has appended (rows mode)
  unsigned long long cta_recs = (kRows && sp.rec_cursor) ? sp.rec_cursor[blockIdx.x] : 0;
  NodeVals nv;
  SlotVal slots[kMaxSlots];

  if (lane < kFixDigits) cta_fix[lane] = 0;
  if (lane == 0) acc->clear();
  const bool grouped = kGroups && !kRows && P.group_slot >= 0;
  if (grouped) keys_clear(*kcache, whole, lane);
  uint32_t fold_lines = 0;  // lines added to kcache's 32-bit sums since the last fold
  uint32_t key_input = 0;  // the batch input whose keys kcache holds
  bool keys_full = false;  // kcache has no free place
  const uint32_t bar = (uint32_t)__cvta_generic_to_shared(s_bar);
  if (lane == 0) mbar_init(bar);
  __syncwarp();
  uint32_t phase = 0;  // parity of the barrier's current phase
  // What this CTA last saw of the run's template, and the rounds that missed
  // a line by it, less half of all rounds since.
  uint32_t tstate = sp.tmpl ? kTmplNone : kTmplOff, tmisses = 0;

  // The first tile is the CTA's own; the others' tickets are taken one tile
  // ahead, so the atomic's latency overlaps a tile's work.  (With every
  // ticket from the counter, the CTAs that start first take two tiles each
  // of an input with one per CTA, and the others none.)
  unsigned long long *const ticket_ctr = sp.ticket ? sp.ticket : &sp.ctr->next_tile;
  unsigned long long next_ticket = blockIdx.x;
  const unsigned long long n_work = sp.tile_list ? sp.n_list : sp.n_tiles;
  for (;;) {
    const unsigned long long ticket = __shfl_sync(0xffffffffu, next_ticket, 0);
    if (ticket >= n_work) break;
    const unsigned long long tile = sp.tile_list ? sp.tile_list[ticket] : ticket;
    if (lane == 0) next_ticket = gridDim.x + atomicAdd(ticket_ctr, 1ull);
    // The tile's input: the whole data, or one input of a batch (a window
    // never reaches past its input's end).
    uint32_t input = 0;
    unsigned long long data_start = 0, data_end = sp.n, ts = tile * T;
    RunCounters *ctr_in = sp.ctr;
    if (sp.tile_input) {
      input = sp.tile_input[tile];
      data_start = sp.in_start[input];
      data_end = sp.in_end[input];
      ts = data_start + (tile - sp.in_tile0[input]) * T;
      ctr_in = sp.in_ctr + input;
      if (kGroups && input != key_input) {
        keys_flush(*kcache, sp.g, whole, lane);
        keys_clear(*kcache, whole, lane);
        key_input = input;
        fold_lines = 0;
        keys_full = false;
      }
    }
    const uint32_t nf = P.output_kind == 2 ? P.n_fields : (P.output_kind == 1 ? 1u : 0u);
    const unsigned long long te = min(ts + T, data_end);
    const uint32_t tlen = (uint32_t)(te - ts);
    const uint32_t wlen = (uint32_t)min((unsigned long long)T + H, data_end - ts);
    const bool win_reaches_end = ts + wlen == data_end;

    // The run's template, until this CTA has it or the run goes without.
    uint32_t tsee = 0;
    if (tstate < kTmplReady && lane == 0)
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];\n" : "=r"(tsee) : "l"(&sp.tmpl->state) : "memory");

    // 1. Stage tile + halo: the window's 16-byte multiple by one bulk copy
    //    (inputs and tiles start 16-byte aligned), its last 0-15 bytes by
    //    plain loads, so nothing past the input is read.
    const uint32_t body = wlen & ~15u;
    __syncwarp();  // the previous tile's reads of the window are done
    if (lane == 0 && body) bulk_load(win, sp.data + ts, body, bar);
    if (lane < (wlen & 15u)) win[body + lane] = sp.data[ts + body + lane];
    const uint32_t prev_nl = (ts == data_start || sp.data[ts - 1] == '\n') ? 1u : 0u;
    if (body) {
      if (!mbar_wait(bar, phase)) {
        // the copy did not complete within the wait limit: report, give it
        // another bounded wait (it writes this CTA's shared memory), stop
        if (lane == 0) atomicOr(&sp.ctr->error, 2u);
        mbar_wait(bar, phase);
        return;
      }
      phase ^= 1u;
    }
    if (lane == 0 && win_reaches_end) win[wlen] = '\n';  // ends the last line for the walker
    if (tstate < kTmplReady) {
      tstate = __shfl_sync(0xffffffffu, tsee, 0);
      __syncwarp();  // the other lanes' reads come after lane 0's acquire (a tile under 16 bytes has no copy to wait for)
      if (tstate == kTmplReady)
#pragma unroll 1
        for (uint32_t k = lane; k < sizeof(Template) / 4; k += 32)
          ((uint32_t *)tmpl)[k] = __ldcg((const uint32_t *)&sp.tmpl->t + k);
    }
    __syncwarp();

    // 2. Stage 1, lane-parallel: every 32-byte chunk of the window (the end
    //    sentinel's too) becomes its special mask; lane l owns chunks
    //    [l*K, l*K + K) and notes the newlines among them that start a line of
    //    the tile in one 64-bit word (the last ones found lowest): eight
    //    positions of 8 bits, or, where a lane owns more than eight chunks
    //    (the tiles of lines of 300 bytes and more), four of 16.  (With those
    //    tiles' chunks classified again instead: lines of 1,000 bytes, 96 MB,
    //    scan 88 us, 79 so.)  Bytes past the window's data are stale: no walk gets
    //    past its line's newline, so their mask bits are never looked at.
    const uint32_t limit = wlen + (win_reaches_end ? 1u : 0u);  // classified bytes
    const uint32_t nchunks = (limit + 31) >> 5;
    const uint32_t K = (nchunks + 31) >> 5;
    const uint32_t c0 = lane * K;
    const uint32_t nl_limit = tlen - 1;  // newlines below this start a line in the tile
    // the newlines of chunk c that start a line of the tile
    auto listed = [&](uint32_t c, uint32_t m) -> uint32_t {
      const int left = max((int)nl_limit - (int)(c * 32), 0);
      return m & ~__funnelshift_lc(0u, 0xFFFFFFFFu, (uint32_t)left);  // all bits from 32 on
    };
    uint32_t my_nl = 0;
    const uint32_t pos_bits = K <= 8 ? 8u : 16u;
    unsigned long long nl_pos = 0;  // positions within the lane's chunks, pos_bits each
    const uint32_t c1 = min(c0 + K, nchunks);
#pragma unroll 1
    for (uint32_t c = c0; c < c1; c++) {
      const uint4 u = ((const uint4 *)win)[2 * c];
      const uint4 v = ((const uint4 *)win)[2 * c + 1];
      const uint32_t w8[8] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w};
      uint32_t sm_c;
      uint32_t m = listed(c, classify_chunk(w8, &sm_c));
      smask[c] = sm_c;
#pragma unroll 1
      for (; m; m &= m - 1u, my_nl++) nl_pos = nl_pos << pos_bits | ((c - c0) * 32u + (uint32_t)__ffs(m) - 1u);
    }

    // The next tile's window is fetched into L2 now (its ticket has
    // arrived), so its bulk copy reads from L2 rather than waiting on HBM.
    if (lane == 0 && next_ticket < n_work) {
      const unsigned long long nt = sp.tile_list ? sp.tile_list[next_ticket] : next_ticket;
      {
        unsigned long long ns = nt * T, ne = sp.n;
        if (sp.tile_input) {
          const uint32_t ni = sp.tile_input[nt];
          ns = sp.in_start[ni] + (nt - sp.in_tile0[ni]) * T;
          ne = sp.in_end[ni];
        }
        const uint32_t nb = (uint32_t)min((unsigned long long)T + H, ne - ns) & ~15u;
        if (nb) l2_prefetch(sp.data + ns, nb);
      }
    }

    // 3. Lines starting in the tile: ts itself (after a newline) and q+1 for
    //    every newline q in [ts, te-1).
    uint32_t first_nl = my_nl;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t x = __shfl_up_sync(0xffffffffu, first_nl, d);
      if (lane >= d) first_nl += x;
    }
    const uint32_t tot_nl = __shfl_sync(0xffffffffu, first_nl, 31);
    first_nl -= my_nl;
    const uint32_t lead = prev_nl;
    const uint32_t n_lines_tile = tot_nl + lead;
    // whether every lane's newlines are noted (else they are found again)
    const bool noted = !__any_sync(0xffffffffu, my_nl * pos_bits > 64u);
    // The tile's last line ends at the first newline at or after te - 1 (the
    // sentinel's, when the window reaches the data's end): looked for 512
    // bytes at a time, 16 a lane.
    uint32_t last_end = 0xFFFFFFFFu;  // none: the line is longer than the window
#pragma unroll 1
    for (uint32_t base = nl_limit & ~15u; base < limit && last_end == 0xFFFFFFFFu; base += 512) {
      const uint32_t at = base + 16 * lane;
      uint32_t first = 0xFFFFFFFFu;
      if (at < limit) {
        const uint4 u = *(const uint4 *)(win + at);
        uint32_t m = flags_push(flags_push(flags_push(flags_push(0, flags_newline(u.w)), flags_newline(u.z)),
                                           flags_newline(u.y)), flags_newline(u.x));
        if (at < nl_limit) m &= 0xFFFFFFFFu << (nl_limit - at);
        if (limit - at < 16) m &= (1u << (limit - at)) - 1u;
        if (m) first = at + (uint32_t)__ffs(m) - 1u;
      }
      last_end = __reduce_min_sync(0xffffffffu, first);
    }

    // 4. Walk the lines, one per lane, in passes of the list's capacity.
    unsigned long long tile_rows = 0, tile_bytes = 0;
    const unsigned long long tile_rec0 = cta_recs;
    uint32_t tile_first_invalid = 0xFFFFFFFFu, tile_first_type = 0xFFFFFFFFu, tile_sel = 0;
#pragma unroll 1
    for (uint32_t base = 0; base < n_lines_tile; base += kMaxLinesPerPass) {
      const uint32_t cnt = min(n_lines_tile - base, kMaxLinesPerPass);
      // list line starts [base, base + cnt] (one extra as the end marker)
      if (lead && lane == 0 && base == 0) lstart[0] = 0;
      {
        const uint32_t idx = first_nl + lead;  // of this lane's first newline
        if (noted) {
#pragma unroll 1
          for (uint32_t k = 0; k < my_nl; k++) {
            const uint32_t i = idx + my_nl - 1u - k - base;
            if (i <= cnt) lstart[i] = (uint16_t)(c0 * 32u + ((uint32_t)(nl_pos >> (pos_bits * k)) & ((1u << pos_bits) - 1u)) + 1u);
          }
        } else if (my_nl && idx <= base + cnt && idx + my_nl > base) {
          uint32_t i = idx - base;  // wraps below the pass
#pragma unroll 1
          for (uint32_t c = c0; c < c1; c++) {
            const uint4 u = ((const uint4 *)win)[2 * c];
            const uint4 v = ((const uint4 *)win)[2 * c + 1];
            const uint32_t w8[8] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w};
            uint32_t unused;
#pragma unroll 1
            for (uint32_t m = listed(c, classify_chunk(w8, &unused)); m; m &= m - 1u, i++)
              if (i <= cnt) lstart[i] = (uint16_t)(c * 32u + (uint32_t)__ffs(m));
          }
        }
      }
      __syncwarp();
#pragma unroll 1
      for (uint32_t b0 = 0; b0 < cnt; b0 += 32) {
        const uint32_t li = b0 + lane;  // line index within the pass
        int status = -1;
        uint32_t has_row = 0, row_len = 0;
        const uint32_t ordinal = base + li;
        uint32_t s = 0, e = 0;  // window offsets of the line and of its newline
        bool found = false;     // the line lies in the window
        const uint8_t *lp = nullptr;
        uint32_t line_len = 0;
        bool has_group = false;
        KeyRef gk;
        uint32_t gh = 0, key_off = 0;  // the key's hash; its window offset
        uint32_t kw[kKeyCacheBytes / 4];  // a short key's bytes
        bool odd_key = false;  // escaped, long, or of a line outside the window
        SlotVal aggv;
        aggv.kind = JK_MISSING;
        if (li < cnt) {
          s = lstart[li];
          // the next line's start is listed (the list keeps one entry past
          // the pass for exactly this), except after the tile's last line
          e = base + li + 1 < n_lines_tile ? (uint32_t)lstart[li + 1] - 1u : last_end;
          found = e != 0xFFFFFFFFu;
        }
        const unsigned long long line_abs = ts + s;

        // The walk.  A slot's value ends up in slots[]; bad_slots says which
        // of them are type errors (resolve_slots).
        uint32_t bad_slots = 0;
        bool walk = found;  // not decided by the template
        if (tstate == kTmplReady) {
          SlotVal none;
          none.off = none.len = 0;
          none.state = SS_MISSING;
          none.kind = JK_MISSING;
          none.esc = 0;
#pragma unroll 1
          for (uint32_t k = 0; k < P.n_slots; k++) slots[k] = none;
          const int st = walk_template(tmpl, win, smask, s, e, found, slots);  // every lane
          walk = found && st != LS_OK;
          if (found) status = LS_OK;
        }
        if (found) {
          lp = win + s;
          line_len = e - s;
        }
        // Everything below, to the next bracket, is for lines no template fits.
        if (__any_sync(0xffffffffu, walk || (li < cnt && !found))) {
          const bool far = li < cnt && !found;
          if (walk) {
            status = walk_objects(P, win, smask, s, e, nv);
            if (status == LS_FALLBACK) status = walk_masked(P, win, smask, s, e, nv);
          }
          if (far) {
            // longer than the window: walk it from global memory
            const unsigned long long q = far_newline(sp.data, ts + wlen, data_end);
            lp = sp.data + line_abs;
            line_len = (uint32_t)(q - line_abs);
            status = walk_line(P, lp, line_len, nv, nullptr);
          }
          __syncwarp();
          const unsigned ok = __ballot_sync(0xffffffffu, walk && status == LS_OK);
          if (tstate == kTmplReady) {
            // a template that many rounds miss a line of costs more than it saves
            if (ok) {
              const bool off = lane == 0 && template_missed(sp.tmpl, next_ticket, n_lines_tile);
              if (__any_sync(0xffffffffu, off) || (tmisses += 2) > 2 * kTmplMisses) tstate = kTmplOff;
            }
          } else if (tstate == kTmplNone) {
            // one line is enough, and only a CTA with another tile to walk tries
            const bool more = __shfl_sync(0xffffffffu, next_ticket < n_work ? 1u : 0u, 0);
            if (ok && more) {
              tstate = kTmplBuilding;  // by this CTA or another: looked up at the next tile
              if (lane == __ffs(ok) - 1 && atomicCAS(&sp.tmpl->state, kTmplNone, kTmplBuilding) == kTmplNone) {
                uint32_t next = kTmplReady;
                if (!build_template(P, win, smask, s, e, tmpl))
                  next = atomicAdd(&sp.tmpl->tries, 1u) + 1u < kTmplTries ? kTmplNone : kTmplOff;  // CTAs take turns at it
                else
                  sp.tmpl->t = *tmpl;
                __threadfence();
                atomicExch(&sp.tmpl->state, next);
              }
            }
          }
          // Lines nesting past 64 levels share this CTA's deep stack, so they
          // are walked one at a time.
          if (__any_sync(0xffffffffu, status == LS_DEEP)) {
#pragma unroll 1
            for (int t = 0; t < 32; t++) {
              if (lane == t && status == LS_DEEP) {
                status = walk_line(P, lp, line_len, nv, &deep);
                if (status == LS_DEEP_FULL) {
                  atomicOr(&sp.ctr->overflow, 8u);
                  status = LS_INVALID;
                }
              }
              __syncwarp();
            }
          }
          if ((walk || far) && status == LS_OK) bad_slots = resolve_slots(P, nv, slots);
          __syncwarp();
        }
        if (tmisses) tmisses--;
        // `out_len`: the line without a trailing '\r' (chunk.rs:433-435).
        uint32_t out_len = line_len;
        if (status >= 0 && out_len && lp[out_len - 1] == '\r') out_len--;

        if (status == LS_OK) {
          if (bad_slots & 1u) {
            status = LS_TYPE_ERROR;
          } else if (P.has_filter && !(found ? eval_filter_win(P, win, s, slots) : eval_filter_far(P, lp, slots))) {
            status = 100;  // filtered out
          } else if (bad_slots) {
            status = LS_TYPE_ERROR;
          } else {
            status = 101;  // selected
          }
        }
        if (status == LS_INVALID) {
          tile_first_invalid = min(tile_first_invalid, ordinal);
        } else if (status == LS_TYPE_ERROR) {
          tile_first_type = min(tile_first_type, ordinal);
        } else if (status == 101) {
          if (kRows) {
            has_row = 1;
            row_len = row_length(P, lp, out_len, slots);
          } else {
            // aggregate (exec/cpu.rs:358-369, agg.rs:44-71)
            if (P.agg_slot >= 0) aggv = slots[P.agg_slot];
            if (kGroups && P.group_slot >= 0) {
              const SlotVal &g = slots[P.group_slot];
              has_group = true;
              gk.esc = 0;
              gk.input = input;
              if (g.kind == JK_MISSING || g.kind == JK_NULL) {
                gk.kind = JK_NULL;
                gk.p = lp;
                gk.len = 0;
                gk.abs_off = line_abs;
              } else if (g.kind == JK_STR) {
                gk.kind = JK_STR;
                gk.p = lp + g.off + 1;
                gk.len = g.len - 2;
                gk.esc = g.esc;
                gk.abs_off = line_abs + g.off + 1;
              } else {
                gk.kind = g.kind;
                gk.p = lp + g.off;
                gk.len = g.len;
                gk.abs_off = line_abs + g.off;
              }
              odd_key = !found || gk.esc || gk.len > kKeyCacheBytes;
              key_off = (uint32_t)(gk.abs_off - ts);
              if (odd_key) {
                gh = hash_key_far(gk.p, gk.len, gk.esc, gk.kind, input);
              } else {
                KeyHasher x;
                key_words(win, key_off, gk.len, kw);
#pragma unroll
                for (uint32_t k = 0; k < kKeyCacheBytes / 4; k++)
                  if (4 * k < gk.len) x.word(kw[k]);
                gh = x.done(gk.len, gk.kind, input);
              }
            }
          }
        }

        // Aggregate contribution of this line.
        bool contrib = !kRows && status == 101;
        long long iv = 0;
        double fv = 0.0;
        bool is_int = false, is_num = false;
        bool saw = false;
        if (contrib && P.agg_slot >= 0) {
          if (aggv.kind == JK_NUM) {
            fv = found ? detail::parse_number_win(win, s + aggv.off, aggv.len, is_int, iv)
                       : detail::parse_number_far(lp + aggv.off, aggv.len, is_int, iv);
            is_num = true;
          } else if (aggv.kind != JK_MISSING && aggv.kind != JK_NULL) {
            saw = true;
          }
        }
        // The round's counts and ungrouped aggregate, reduced in the warp
        // and added to the CTA's shared accumulator by lane 0.
        {
          const unsigned full = 0xffffffffu;
          if (__any_sync(full, status >= 0 && status < 100)) {  // neither selected nor filtered out
            const unsigned m_blank = __ballot_sync(full, status == LS_BLANK);
            const unsigned m_inv = __ballot_sync(full, status == LS_INVALID);
            const unsigned m_type = __ballot_sync(full, status == LS_TYPE_ERROR);
            if (lane == 0) {
              acc->blank += __popc(m_blank);
              acc->invalid += __popc(m_inv);
              acc->type += __popc(m_type);
            }
          }
          const unsigned m_sel = __ballot_sync(full, status == 101);
          tile_sel += __popc(m_sel);
        }
        if (!kRows && P.agg_slot >= 0 && __any_sync(0xffffffffu, contrib)) {
          const unsigned full = 0xffffffffu;
          const unsigned m_saw = __ballot_sync(full, saw);
          const bool ung = contrib && !has_group;
          const unsigned m_num = __ballot_sync(full, ung && is_num);
          const unsigned m_int = __ballot_sync(full, ung && is_num && is_int);
          unsigned long long s_lo = 0, s_hi = 0, ext = 0;
          const uint32_t ak = P.agg_kind;
          if (m_int && (ak == WARPJQ_AGG_SUM || ak == WARPJQ_AGG_AVG))
            group_sum128(full, ung && is_num && is_int, iv, s_lo, s_hi);
          if (m_num && (ak == WARPJQ_AGG_MIN || ak == WARPJQ_AGG_MAX))
            ext = group_extreme(full, ung && is_num, order_bits(fv), ak == WARPJQ_AGG_MIN);
          if (ak == WARPJQ_AGG_SUM || ak == WARPJQ_AGG_AVG)
            warp_fix_add(cta_fix, &ctr_in->fbig, ung && is_num && !is_int, fv, lane);  // exact, in the CTA's limbs
          if (lane == 0) {
            if (m_saw) acc->saw = 1;
            if (m_num) {
              acc->numeric += __popc(m_num);
              acc->n_int += __popc(m_int);
              if (s_lo || s_hi) {
                const unsigned long long o = acc->isum_lo;
                acc->isum_lo = o + s_lo;
                acc->isum_hi += s_hi + (acc->isum_lo < o ? 1ull : 0ull);
              }
              if (ak == WARPJQ_AGG_MIN) acc->min_bits = min(acc->min_bits, ext);
              if (ak == WARPJQ_AGG_MAX) acc->max_bits = max(acc->max_bits, ext);
            }
          }
        }
        if (kGroups && !kRows && P.group_slot >= 0) {
          // A short key is looked up among the CTA's own first.
          constexpr uint32_t kNone = 0xFFFFFFFFu;
          uint32_t kid = kNone, ke = kNone;  // the key's id; its place in kcache
          const uint32_t meta = gk.len | (uint32_t)gk.kind << 24;
          if (has_group && !odd_key) {
#pragma unroll 1
            for (uint32_t j = 0; j < n_places; j++) {
              const uint32_t e = (gh + j) & (n_places - 1u), hv = kcache->hash[e];
              if (!hv) break;
              if (hv != gh || kcache->meta[e] != meta) continue;
              uint32_t diff = 0;
#pragma unroll
              for (uint32_t k = 0; k < kKeyCacheBytes / 4; k++) diff |= kcache->bytes[e][k] ^ kw[k];
              if (!diff) {
                kid = kcache->kid[e];
                ke = e;
                break;
              }
            }
          }
          const bool look = has_group && kid == kNone;
          if (__any_sync(0xffffffffu, look)) {
            // Lanes whose keys hash alike compare their key bytes with the
            // lowest such lane; only lanes that differ from it look up the
            // table themselves.
            const unsigned peers = __match_any_sync(0xffffffffu, look ? gh : 0u);
            const int leader = __ffs(peers) - 1;
            const unsigned long long lp = __shfl_sync(0xffffffffu, (unsigned long long)gk.p, leader);
            const uint32_t lmeta = __shfl_sync(0xffffffffu, meta, leader);
            const uint32_t llen = __shfl_sync(0xffffffffu, gk.len, leader);
            const uint32_t lesc = __shfl_sync(0xffffffffu, (uint32_t)gk.esc, leader);
            const bool same = look && lane != leader && gk.kind == lmeta >> 24 &&
                              key_bytes_equal(gk, (const uint8_t *)lp, llen, (uint8_t)lesc);
            bool full = false;
            if (look && !same) {
              kid = group_find_or_insert(sp, gk, gh);
              if (!odd_key && kid != kNone && !keys_full) {  // kept in the first free of its places
                full = true;
#pragma unroll 1
                for (uint32_t j = 0; j < n_places; j++) {
                  const uint32_t e = (gh + j) & (n_places - 1u);
                  if (atomicCAS(&kcache->hash[e], 0u, gh) != 0u) continue;
                  full = false;
#pragma unroll
                  for (uint32_t k = 0; k < kKeyCacheBytes / 4; k++) kcache->bytes[e][k] = kw[k];
                  kcache->meta[e] = meta;
                  kcache->kid[e] = kid;
                  ke = e;
                  break;
                }
              }
            }
            keys_full = keys_full || __any_sync(0xffffffffu, full);
            const uint32_t lkid = __shfl_sync(0xffffffffu, kid, leader), lke = __shfl_sync(0xffffffffu, ke, leader);
            if (same) {
              kid = lkid;
              ke = lke;
            }
          }
          const uint32_t ak = P.agg_kind;
          const bool minmax = ak == WARPJQ_AGG_MIN || ak == WARPJQ_AGG_MAX;
          const bool plain = !has_group || (ke != kNone && (!is_num || minmax || (is_int && iv >= 0 && iv < (1ll << 31))));
          if (__all_sync(0xffffffffu, plain)) {
            if (has_group) {
              atomicAdd(&kcache->n[ke], 1u);
              if (is_num) {
                atomicAdd(&kcache->num[ke], 1u);
                if (minmax) {
                  if (is_int) atomicAdd(&kcache->lo[ke], 1u);
                  // few values still move a key's extreme
                  GroupAcc &a = kcache->at(ke, false);
                  const unsigned long long ob = order_bits(fv);
                  if (ak == WARPJQ_AGG_MIN) {
                    if (ob < a.min_bits) atomicMin(&a.min_bits, ob);
                  } else if (ob > a.max_bits) {
                    atomicMax(&a.max_bits, ob);
                  }
                } else {
                  atomicAdd(&kcache->lo[ke], (uint32_t)iv & 0xFFFFu);
                  atomicAdd(&kcache->hi[ke], (uint32_t)iv >> 16);
                }
              }
            }
            if ((fold_lines += 32) >= kFoldLines) {
              keys_fold(*kcache, whole, lane);
              fold_lines = 0;
            }
          } else {
            // Lanes holding the same key add up their contributions in the
            // warp first; one lane per key then updates its accumulators
            // (counts, the exact integer sum, min or max).  Fractional values
            // go in per lane, exactly (fixsum.cuh).  kcache's are this warp's,
            // and one lane of it leads a key, so its adds need no atomics.
            const unsigned grp = __match_any_sync(0xffffffffu, kid);
            const bool lead = kid != kNone && lane == __ffs(grp) - 1;
            const bool num_int = is_num && is_int;
            const unsigned m_num = __ballot_sync(0xffffffffu, is_num) & grp;
            const unsigned m_int = __ballot_sync(0xffffffffu, num_int) & grp;
            unsigned long long s_lo = 0, s_hi = 0, ext = 0;
            if (whole && __any_sync(0xffffffffu, num_int)) group_sum128(grp, num_int, iv, s_lo, s_hi);
            if (minmax && __any_sync(0xffffffffu, is_num))
              ext = group_extreme(grp, is_num, order_bits(fv), ak == WARPJQ_AGG_MIN);
            const bool frac = is_num && !is_int && whole;
            if (kid == kNone) {  // no key, or the table is full
            } else if (ke != kNone) {
              GroupAcc &a = kcache->at(ke, whole);
              if (lead) {
                a.count += __popc(grp);
                a.numeric += __popc(m_num);
                a.n_int += __popc(m_int);
                const unsigned long long lo = a.isum_lo + s_lo;
                a.isum_hi += s_hi + (lo < s_lo ? 1ull : 0ull);
                a.isum_lo = lo;
                if (m_num && ak == WARPJQ_AGG_MIN) a.min_bits = min(a.min_bits, ext);
                if (m_num && ak == WARPJQ_AGG_MAX) a.max_bits = max(a.max_bits, ext);
              }
              if (frac) fix_atomic_add(a.fix, &a.fbig, fv);
            } else {
              GroupAcc &a = sp.g.acc[kid];
              if (lead) {
                atomicAdd(&a.count, (unsigned long long)__popc(grp));
                if (m_num) atomicAdd(&a.numeric, (unsigned long long)__popc(m_num));
                if (m_int) {
                  atomicAdd(&a.n_int, (unsigned long long)__popc(m_int));
                  if (s_lo || s_hi) {
                    const unsigned long long old = atomicAdd(&a.isum_lo, s_lo);
                    const unsigned long long carry = (old + s_lo) < old ? 1ull : 0ull;
                    if (s_hi + carry) atomicAdd(&a.isum_hi, s_hi + carry);
                  }
                }
                if (m_num && ak == WARPJQ_AGG_MIN) atomicMin(&a.min_bits, ext);
                if (m_num && ak == WARPJQ_AGG_MAX) atomicMax(&a.max_bits, ext);
              }
              if (frac) fix_atomic_add(a.fix, &a.fbig, fv);
            }
          }
          __syncwarp();  // kcache's keys and sums are there for the lanes that look in the next round
        }

        if (kRows) {
          uint32_t er, tr;
          unsigned long long eb, tb;
          warp_scan2(has_row, (unsigned long long)row_len, er, eb, tr, tb);
          if (has_row) {
            unsigned long long ri = cta_recs + er;
            if (ri < sp.rec_cap_per_cta) {
              RowRec *r = (RowRec *)(my_recs + ri * rec_stride);
              r->line_start = line_abs;
              r->line_len = out_len;
              r->ordinal = ordinal;
              r->local_off = (uint32_t)(tile_bytes + eb);
              r->row_len = row_len;
              uint32_t *fl = (uint32_t *)(r + 1);
#pragma unroll 1
              for (uint32_t f = 0; f < nf; f++) {
                const SlotVal &s = slots[P.output_kind == 1 ? P.out_slot : P.field_slot[f]];
                fl[2 * f] = s.off;
                fl[2 * f + 1] = s.len | ((uint32_t)s.kind << 28) | ((uint32_t)s.esc << 27);
              }
            } else {
              atomicOr(&sp.ctr->overflow, 1u);
            }
          }
          tile_rows += tr;
          tile_bytes += tb;
          cta_recs += tr;
        }
      }
      __syncwarp();
    }
    if (lane == 0) {
      acc->lines += n_lines_tile;
      acc->sel += tile_sel;
    }

    // Per-tile bookkeeping.
    tile_first_invalid = __reduce_min_sync(0xffffffffu, tile_first_invalid);
    tile_first_type = __reduce_min_sync(0xffffffffu, tile_first_type);
    if (lane == 0) {
      sp.tiles[tile].n_lines = n_lines_tile;
      sp.tiles[tile].first_invalid = tile_first_invalid;
      sp.tiles[tile].first_type_error = tile_first_type;
      if (tile_first_invalid != 0xFFFFFFFFu) {
        atomicMin(&sp.ctr->first_invalid_tile, tile);
        if (sp.tile_input) atomicMin(&ctr_in->first_invalid_tile, tile);
      }
      if (tile_first_type != 0xFFFFFFFFu) {
        atomicMin(&sp.ctr->first_type_tile, tile);
        if (sp.tile_input) atomicMin(&ctr_in->first_type_tile, tile);
      }
    }
    if (kRows || sp.any_rows) {  // an aggregate tile of a batch with rows has none
      if (lane == 0) {
        RowTile rt;
        rt.rec_begin = (unsigned long long)blockIdx.x * sp.rec_cap_per_cta + tile_rec0;
        rt.bytes = tile_bytes;
        rt.rows = (uint32_t)tile_rows;
        rt.pad = 0;
        sp.row_tiles[tile] = rt;
      }
    }
    // A batch input's counts and aggregate go to its own record, tile by tile.
    if (sp.tile_input)
      flush_counts(ctr_in, sp.ctr, P, kRows, lane, acc, cta_fix);
  }

  // Merge this CTA's own group accumulators into the global records.
  if (grouped) keys_flush(*kcache, sp.g, whole, lane);

  if (kRows && sp.rec_cursor && lane == 0) sp.rec_cursor[blockIdx.x] = cta_recs;
  // Flush this CTA's counters (a batch's were flushed per tile).
  flush_counts(sp.ctr, nullptr, P, kRows, lane, acc, cta_fix);
}

// The run's FP totals from its exact limbs (the integer sum joins them
// before the one rounding of sum_total).
__device__ __forceinline__ void finalize_sums(RunCounters &c) {
  c.fsum_total = fix_to_double(c.fix, 0, 0) + c.fbig;
  c.sum_total = fix_to_double(c.fix, c.agg_isum_lo, c.agg_isum_hi) + c.fbig;
}

// The keys that hold lines (not the ids that inserts racing for a key left
// unused), as the results the host hands on: exact sums rounded once
// (fixsum.cuh), minima and maxima decoded.  Their order is any, like the ids'.
// Compacting and rounding them here leaves the host one copy of 88 bytes a
// group: some 160 ns a group before (the raw descriptors and accumulators of every
// id, 152 bytes each, through pageable memory, then two roundings).
__device__ __forceinline__ void compact_groups(RunCounters *ctr, const GroupKeyDesc *keys, const GroupAcc *acc,
                                               uint32_t key_cap, warpjq_group_ext *out, uint32_t *out_input) {
  const uint32_t nk = min(ctr->n_keys, key_cap);
  for (uint32_t k0 = blockIdx.x * blockDim.x; k0 < nk; k0 += gridDim.x * blockDim.x) {
    const uint32_t k = k0 + threadIdx.x;
    const bool on = k < nk && acc[k].count != 0;
    const unsigned m = __ballot_sync(0xffffffffu, on);
    if (!m) continue;
    uint32_t at = 0;
    const int lane = threadIdx.x & 31;
    if (lane == 0) at = atomicAdd(&ctr->n_groups, (uint32_t)__popc(m));
    at = __shfl_sync(0xffffffffu, at, 0) + __popc(m & ((1u << lane) - 1u));
    if (!on) continue;
    const GroupAcc &a = acc[k];
    const GroupKeyDesc &d = keys[k];
    warpjq_group_ext g;
    g.key_off = d.off;
    g.key_len = d.len;
    g.key_kind = d.kind;
    g.count = a.count;
    g.numeric = a.numeric;
    g.isum_lo = a.isum_lo;
    g.isum_hi = a.isum_hi;
    g.n_int = a.n_int;
    g.fsum = fix_to_double(a.fix, 0, 0) + a.fbig;
    g.min = a.numeric ? min_of_bits(a.min_bits) : __builtin_huge_val();
    g.max = a.numeric ? max_of_bits(a.max_bits) : -__builtin_huge_val();
    g.sum = fix_to_double(a.fix, a.isum_lo, a.isum_hi) + a.fbig;
    out[at] = g;
    out_input[at] = d.input;
  }
}

// Batched runs: every input's record starts like a fresh run's.
__global__ void k_batch_reset(RunCounters *in_ctr, uint32_t n_inputs) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n_inputs; i += gridDim.x * blockDim.x) {
    RunCounters z;
    memset(&z, 0, sizeof(z));
    z.first_invalid_tile = ~0ull;
    z.first_type_tile = ~0ull;
    z.agg_min_bits = ~0ull;
    z.first_invalid = ~0ull;
    z.first_type_error = ~0ull;
    in_ctr[i] = z;
  }
}

// The largest i in [0, n) with a[i] <= t (a[0] <= t, a ascending).
__device__ __forceinline__ uint32_t last_at_or_below(const unsigned long long *a, uint32_t n,
                                                     unsigned long long t) {
  uint32_t lo = 0, hi = n;
  while (hi - lo > 1) {
    const uint32_t mid = lo + (hi - lo) / 2;
    if (a[mid] <= t) lo = mid;
    else hi = mid;
  }
  return lo;
}

// A batch's per-tile tables, built on the device from its per-input ones
// (host work stays proportional to the inputs, not the tiles): tile t
// belongs to the input i with in_tile0[i] <= t < in_tile0[i + 1] (an empty
// input owns none, so the last input starting at or below t is its owner).
// A mixed batch also lists, plan after plan, the tiles of each plan's
// inputs: position p of list_tiles is tile p - list_tile0[j] of input
// list_inputs[j] (list_tile0 running over the inputs in list order).
__global__ void k_batch_expand(unsigned long long n_tiles, uint32_t n_inputs, const unsigned long long *in_tile0,
                               uint32_t *tile_input, const uint32_t *list_inputs,
                               const unsigned long long *list_tile0, uint32_t *list_tiles) {
  for (unsigned long long t = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; t < n_tiles;
       t += (unsigned long long)gridDim.x * blockDim.x) {
    tile_input[t] = last_at_or_below(in_tile0, n_inputs, t);
    if (list_tiles) {
      const uint32_t j = last_at_or_below(list_tile0, n_inputs, t);
      const uint32_t i = list_inputs[j];
      list_tiles[t] = (uint32_t)(in_tile0[i] + (t - list_tile0[j]));
    }
  }
}

// Batched runs, one warp per input: the input's first invalid / type-error
// line (lane l sums a contiguous slice of the input's tiles' line counts)
// and its FP totals.
__global__ void k_batch_finalize(const TileDesc *tiles, const unsigned long long *in_tile0,
                                 RunCounters *in_ctr, uint32_t n_inputs) {
  const int lane = threadIdx.x & 31;
  const unsigned long long i = ((unsigned long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (i >= n_inputs) return;  // uniform per warp
  const unsigned long long t0 = in_tile0[i], t1 = in_tile0[i + 1];
  RunCounters &c = in_ctr[i];
  const unsigned long long cut = c.first_invalid_tile, cut_t = c.first_type_tile;
  const unsigned long long per = (t1 - t0 + 31) / 32;
  const unsigned long long a = min(t0 + lane * per, t1), b = min(a + per, t1);
  unsigned long long lines = 0, lines_t = 0;
  for (unsigned long long t = a; t < b && (t < cut || t < cut_t); t++) {
    if (t < cut) lines += tiles[t].n_lines;
    if (t < cut_t) lines_t += tiles[t].n_lines;
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    lines += __shfl_down_sync(0xffffffffu, lines, d);
    lines_t += __shfl_down_sync(0xffffffffu, lines_t, d);
  }
  if (lane != 0) return;
  finalize_sums(c);
  c.first_invalid = cut == ~0ull ? ~0ull : lines + tiles[cut].first_invalid;
  c.first_type_error = cut_t == ~0ull ? ~0ull : lines_t + tiles[cut_t].first_type_error;
}

// ---------------------------------------------------------------------------
// Rows: prefix over the per-tile totals, then emission in line order.
// ---------------------------------------------------------------------------

// Tiles per block of the rows passes, at most a thread each.  A row costs a
// few microseconds of dependent loads, whoever copies it, so what counts is
// how many are in flight: small inputs take 8 tiles a block, up to 262,144
// tiles 64 (whole lines: 470 us a pass with 64 tiles, 475 with 32, 483 with
// 128), the largest 128, so the one block that scans the block sums stays
// short.
constexpr int kEmitThreads = 128;
__host__ __device__ inline uint32_t rows_tiles_per_block(unsigned long long n_tiles) {
  return n_tiles < 148ull * 8 ? 8u : n_tiles < 262144ull ? 64u : 128u;
}
// Exclusive block scan of three u64 values in thread order, with totals.
template <int NT>
__device__ __forceinline__ void block_scan3(const unsigned long long v[3], unsigned long long ex[3],
                                            unsigned long long tot[3],
                                            unsigned long long (*s_w)[NT / 32]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned long long inc[3] = {v[0], v[1], v[2]};
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
#pragma unroll
    for (int k = 0; k < 3; k++) {
      unsigned long long x = __shfl_up_sync(0xffffffffu, inc[k], d);
      if (lane >= d) inc[k] += x;
    }
  }
  if (lane == 31)
    for (int k = 0; k < 3; k++) s_w[k][warp] = inc[k];
  __syncthreads();
  for (int k = 0; k < 3; k++) {
    unsigned long long before = 0, all = 0;
    for (int w = 0; w < NT / 32; w++) {
      if (w < warp) before += s_w[k][w];
      all += s_w[k][w];
    }
    ex[k] = before + inc[k] - v[k];
    tot[k] = all;
  }
  __syncthreads();
}

// The run's last pass over its tiles, in blocks of `tpb` of them: the group
// results, sums of (rows, bytes, lines) per block, and in the block that is
// through last everything that needs them all: for rows the exclusive prefix
// over the blocks (in place; output that does not fit raises the overflow
// flag, and the run is repeated with room), the indexes of the first invalid
// and type-error line, and the FP totals.  One launch where the same took four
// (two without rows): a run of 4 KB spent 9 of its 23 us on the device there.
struct TailParams {
  unsigned long long n_tiles;
  uint32_t tpb;
  const TileDesc *tiles;
  const RowTile *row_tiles;  // null: no rows
  unsigned long long *bsum;  // 3 per block
  RunCounters *ctr;
  RunCounters *mirror;  // page-locked host memory that gets the finished counters (null: none)
  unsigned long long *row_off;
  unsigned long long rows_cap, out_cap;
  const GroupKeyDesc *keys;  // null: no groups
  const GroupAcc *acc;
  uint32_t key_cap;
  warpjq_group_ext *ext;
  uint32_t *ext_input;
};
constexpr int kTailThreads = 256;
constexpr unsigned kTailBlocks = 256;  // of a run without rows, at most

__global__ void __launch_bounds__(kTailThreads) k_tail(const __grid_constant__ TailParams tp) {
  __shared__ unsigned long long s_w[3][kTailThreads / 32];
  __shared__ uint32_t s_last;
  RunCounters &c = *tp.ctr;
  if (tp.keys) {
    compact_groups(tp.ctr, tp.keys, tp.acc, tp.key_cap, tp.ext, tp.ext_input);
    __syncthreads();  // all of the block's groups are counted before thread 0 says that it is through
  }
  const unsigned long long cut[2] = {c.first_invalid_tile, c.first_type_tile};
  const bool bad = cut[0] != ~0ull || cut[1] != ~0ull, sums = tp.row_tiles || bad;
  unsigned long long v[3] = {0, 0, 0}, ex[3], tot[3];
  if (sums) {
    const unsigned long long t0 = (unsigned long long)blockIdx.x * tp.tpb, t1 = min(t0 + tp.tpb, tp.n_tiles);
    for (unsigned long long t = t0 + threadIdx.x; t < t1; t += kTailThreads) {
      if (tp.row_tiles) {
        v[0] += tp.row_tiles[t].rows;
        v[1] += tp.row_tiles[t].bytes;
      }
      v[2] += tp.tiles[t].n_lines;
    }
    block_scan3<kTailThreads>(v, ex, tot, s_w);
  }
  if (threadIdx.x == 0) {
    if (sums)
      for (int k = 0; k < 3; k++) tp.bsum[blockIdx.x * 3 + k] = tot[k];
    __threadfence();
    s_last = atomicAdd(&c.tail_done, 1u) + 1 == gridDim.x;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();  // the other blocks' sums are there
  if (sums) {
    const unsigned nb = gridDim.x, per = (nb + kTailThreads - 1) / kTailThreads;
    const unsigned b0 = min(threadIdx.x * per, nb), b1 = min(b0 + per, nb);
    v[0] = v[1] = v[2] = 0;
    for (unsigned b = b0; b < b1; b++)
      for (int k = 0; k < 3; k++) v[k] += __ldcg(tp.bsum + b * 3 + k);
    block_scan3<kTailThreads>(v, ex, tot, s_w);
    for (unsigned b = b0; b < b1; b++)
      for (int k = 0; k < 3; k++) {
        const unsigned long long x = __ldcg(tp.bsum + b * 3 + k);
        tp.bsum[b * 3 + k] = ex[k];
        ex[k] += x;
      }
    if (threadIdx.x == 0 && tp.row_tiles) {
      c.out_len = tot[1];
      if (tot[0] > tp.rows_cap || tot[1] > tp.out_cap) atomicOr(&c.overflow, 2u);
      else tp.row_off[tot[0]] = tot[1];
    }
    __syncthreads();
  }
  if (bad) {  // lines before the first tile that holds one: of the blocks before its block, then of its tiles
    v[0] = v[1] = v[2] = 0;
    for (int k = 0; k < 2; k++)
      if (cut[k] != ~0ull)
        for (unsigned long long t = cut[k] / tp.tpb * tp.tpb + threadIdx.x; t < cut[k]; t += kTailThreads)
          v[k] += tp.tiles[t].n_lines;
    block_scan3<kTailThreads>(v, ex, tot, s_w);
  }
  if (threadIdx.x == 0) {
    finalize_sums(c);
    c.first_invalid = cut[0] == ~0ull ? ~0ull : tp.bsum[cut[0] / tp.tpb * 3 + 2] + tot[0] + tp.tiles[cut[0]].first_invalid;
    c.first_type_error =
        cut[1] == ~0ull ? ~0ull : tp.bsum[cut[1] / tp.tpb * 3 + 2] + tot[1] + tp.tiles[cut[1]].first_type_error;
    __threadfence();
  }
  // The host reads the counters once the stream is done, with no copy of its
  // own behind the kernel (5 us of a 4 KB run).
  __syncthreads();
  static_assert(sizeof(RunCounters) % 8 == 0, "copied by words");
  if (tp.mirror && threadIdx.x < sizeof(RunCounters) / 8)
    ((unsigned long long *)tp.mirror)[threadIdx.x] = __ldcg((const unsigned long long *)tp.ctr + threadIdx.x);
}

// Tiles per block of k_tail, and its blocks.
inline uint32_t tail_tiles_per_block(unsigned long long n_tiles, bool rows) {
  return rows ? rows_tiles_per_block(n_tiles)
              : (uint32_t)std::max<unsigned long long>(32, (n_tiles + kTailBlocks - 1) / kTailBlocks);
}
inline unsigned tail_blocks(unsigned long long n_tiles, uint32_t tpb) { return (unsigned)((n_tiles + tpb - 1) / tpb); }

// The rows' copy: each block takes its `tiles_per_block` tiles: per-tile prefixes by a
// block scan, then the block's rows, in order.  Whole lines are copied a row a
// group of lanes.  Rows of values take a thread each while they are short, which
// puts its bytes into shared memory; the block then writes the batch's rows,
// which are contiguous in the output, in whole words.  (768 MB of access-log
// lines, 6% of them selected: 66 us with a group of lanes a row, 43 so; a warp
// a row, a tile's rows one after another, took 198.)  Rows of JSON longer than
// kEmitOwn, and all of a batch that does not fit, are written by groups of lanes
// too.  (Rows of 100 bytes, 96 MB of them: a thread a row, unstaged, 985 us, so
// 417; of 1,000 bytes 1,420 and 394.  64 or 256 in kEmitOwn's place measure the
// same; 16 KB of kEmitStage, with half the blocks in flight, 854 and 404.)
// A CSV row's cells are a thread's, staged or not: their quoting is a byte's work.
constexpr uint32_t kEmitStage = 8192;  // bytes of a batch of rows kept in shared memory
constexpr uint32_t kEmitOwn = 128;     // longest row a thread writes there by itself

template <bool kMixed>
__global__ void __launch_bounds__(kEmitThreads) k_rows_emit(EmitParams ep, const __grid_constant__ DevPlan plan) {
  __shared__ unsigned long long s_w[3][kEmitThreads / 32];
  __shared__ unsigned long long s_byte[kEmitThreads], s_line[kEmitThreads], s_rec[kEmitThreads];
  __shared__ uint32_t s_row[kEmitThreads];  // rows of the block's tiles before this one
  __shared__ unsigned long long s_span[2];  // output bytes of a batch of rows
  __shared__ __align__(16) uint8_t s_out[kEmitStage];
  if (ep.ctr->overflow & 3u) return;  // the run is repeated with bigger buffers
  const uint32_t rec_stride = ep.rec_stride, tpb = ep.tiles_per_block;
  const unsigned long long t0 = (unsigned long long)blockIdx.x * tpb, t = t0 + threadIdx.x;
  unsigned long long v[3] = {0, 0, 0};
  unsigned long long rec = 0;
  if (threadIdx.x < tpb && t < ep.n_tiles) {
    const RowTile rt = ep.row_tiles[t];
    v[0] = rt.rows;
    v[1] = rt.bytes;
    v[2] = ep.tiles[t].n_lines;
    rec = rt.rec_begin;
  }
  const unsigned long long row0 = ep.block_prefix[blockIdx.x * 3], byte0 = ep.block_prefix[blockIdx.x * 3 + 1],
                           line0 = ep.block_prefix[blockIdx.x * 3 + 2];
  unsigned long long ex[3], tot[3];
  block_scan3<kEmitThreads>(v, ex, tot, s_w);
  s_row[threadIdx.x] = (uint32_t)ex[0];
  s_byte[threadIdx.x] = byte0 + ex[1];
  s_line[threadIdx.x] = line0 + ex[2];
  s_rec[threadIdx.x] = rec;
  __syncthreads();
  const uint32_t rows = (uint32_t)tot[0];
  // row r's tile: the last with at most r rows before it
  auto tile_of = [&](uint32_t r) {
    uint32_t i = 0;
#pragma unroll
    for (uint32_t d = kEmitThreads / 2; d; d >>= 1)
      if (i + d < tpb && s_row[i + d] <= r) i += d;
    return i;
  };
  if (kMixed || (plan.output_kind == 0 && !plan.csv_mode)) {
    // whole lines; in a mixed batch, rows of any kind
    const uint32_t g = threadIdx.x % kEmitLanes;
#pragma unroll 1
    for (uint32_t r = threadIdx.x / kEmitLanes; r < rows; r += kEmitThreads / kEmitLanes) {
      const uint32_t i = tile_of(r);
      const RowRec *rr = (const RowRec *)(ep.recs + (s_rec[i] + (r - s_row[i])) * rec_stride);
      const RowRec h = *rr;
      const unsigned long long at = s_byte[i] + h.local_off;
      const uint8_t *line = ep.data + h.line_start;
      if (kMixed) {
        const DevPlan &P = ep.plans[ep.in_plan[ep.tile_input[t0 + i]]];
        if (P.output_kind != 0 || P.csv_mode) {
          if (!P.csv_mode) emit_row_group(P, line, (const uint32_t *)(rr + 1), ep.out + at, g);
          else if (g == 0) emit_row(P, line, h, (const uint32_t *)(rr + 1), ep.out + at);
          if (g == 0) {
            ep.row_off[row0 + r] = at;
            ep.line_idx[row0 + r] = s_line[i] + h.ordinal;
          }
          continue;
        }
      }
      group_copy(ep.out + at, line, h.line_len, g);
      if (g == 0) {
        ep.out[at + h.line_len] = '\n';
        ep.row_off[row0 + r] = at;
        ep.line_idx[row0 + r] = s_line[i] + h.ordinal;
      }
    }
    return;
  }
  if constexpr (!kMixed)
#pragma unroll 1
  for (uint32_t r0 = 0; r0 < rows; r0 += kEmitThreads) {
    const uint32_t r = r0 + threadIdx.x;
    RowRec h = {};
    const uint32_t *fl = nullptr;
    unsigned long long at = 0;
    if (r < rows) {
      const uint32_t i = tile_of(r);
      const RowRec *rr = (const RowRec *)(ep.recs + (s_rec[i] + (r - s_row[i])) * rec_stride);
      h = *rr;
      fl = (const uint32_t *)(rr + 1);
      at = s_byte[i] + h.local_off;
      ep.row_off[row0 + r] = at;
      ep.line_idx[row0 + r] = s_line[i] + h.ordinal;
      if (threadIdx.x == 0) s_span[0] = at;
      if (r + 1 == rows || threadIdx.x == kEmitThreads - 1) s_span[1] = at + h.row_len;
    }
    __syncthreads();
    // the batch's place in the output and, from the word it starts in, in s_out
    const unsigned long long b0 = s_span[0], b1 = s_span[1];
    const uint32_t lead = (uint32_t)((uintptr_t)(ep.out + b0) & 3u);
    const bool staged = b1 - b0 + 4 <= kEmitStage;
    uint8_t *const dst = staged ? s_out + lead + (uint32_t)(at - b0) : ep.out + at;
    const bool mine = plan.csv_mode || (staged && h.row_len <= kEmitOwn);
    if (r < rows && mine) emit_row(plan, ep.data + h.line_start, h, fl, dst);
    if (!plan.csv_mode) {  // the others by groups of lanes, each group its own lanes' rows
      const uint32_t g = threadIdx.x % kEmitLanes;
      const unsigned todo = __ballot_sync(0xffffffffu, r < rows && !mine);
#pragma unroll 1
      for (uint32_t k = 0; k < kEmitLanes && todo; k++) {
        const uint32_t from = (threadIdx.x & 31u) - g + k;
        const unsigned long long line = __shfl_sync(0xffffffffu, h.line_start, from);
        const uint32_t *const ffl = (const uint32_t *)__shfl_sync(0xffffffffu, (unsigned long long)fl, from);
        uint8_t *const fdst = (uint8_t *)__shfl_sync(0xffffffffu, (unsigned long long)dst, from);
        if (todo >> from & 1u) emit_row_group(plan, ep.data + line, ffl, fdst, g);
      }
    }
    __syncthreads();
    if (staged) {
      uint8_t *const w0 = ep.out + b0 - lead;  // a word boundary
      const uint32_t end = lead + (uint32_t)(b1 - b0);
      for (uint32_t k = 4 * threadIdx.x; k < end; k += 4 * kEmitThreads) {
        if (k >= lead && k + 4 <= end) {
          *(uint32_t *)(w0 + k) = *(const uint32_t *)(s_out + k);
        } else {
          for (uint32_t j = max(k, lead); j < min(k + 4, end); j++) w0[j] = s_out[j];
        }
      }
      __syncthreads();
    }
  }
}

}  // namespace wjq
