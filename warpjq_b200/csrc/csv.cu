// CSV input: converts RFC 4180 CSV to NDJSON in device memory, so the scan
// kernels run on it unchanged.  The reference reads only NDJSON (its --csv
// flag is an output format, crates/warpjq-core/src/output.rs:45-85); this
// mapping is this library's own:
//
//   - a '\n' ends a row when the number of '"' bytes before it (from the
//     start of the input) is even; a '\r' just before it is dropped;
//   - the first row is the header; every later row becomes one NDJSON line,
//     an empty row an empty line (which the scan skips as blank);
//   - fields are separated by ','; a field that starts with '"' is quoted:
//     it runs to the next '"' not followed by another '"', a doubled '""'
//     inside stands for '"', and bytes after the closing quote up to the
//     next ',' are kept as they are; other fields run to the next ',';
//   - a row becomes an object with the header's names as keys, in order,
//     from its first min(fields, names) fields: missing trailing fields are
//     left out, extra fields are dropped;
//   - a value is the field's text as a JSON number when the field is not
//     quoted and its text is a JSON number; null when it is not quoted and
//     empty; else a JSON string ('"' and '\' escaped, control bytes as
//     \n \r \t \b \f or \u00XX, other bytes as they are).  Header names are
//     escaped the same way; a UTF-8 byte-order mark before the header is
//     dropped.
//
// Passes, none waiting on another CTA:
//   k_csv_stats     per 256-byte run: quote parity, newline count, newlines
//                   outside quotes if the run starts outside; per 64 KiB
//                   tile the same (16-byte loads, SWAR byte masks, a prefix
//                   XOR over the quote mask for the in-quote state)
//   k_csv_tiles     one block: each tile's start state and first row
//   k_csv_row_ends  each row's end offset
//   k_csv_close     the last row, the consumed length, the header's end
//   k_csv_json<0>   every row's NDJSON length, 32 rows a warp
//   (exclusive scan of the lengths)
//   k_csv_json<1>   every row's NDJSON bytes, 32 rows a warp
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <new>
#include <string>
#include <vector>

#include "../../include/warpjq_ext.h"
#include "csv_rows.cuh"

// The window helpers of the scan, with internal linkage.
namespace {
#include "walker.cuh"
}

using namespace wjq_csv;

namespace {

constexpr uint32_t kRun = 256;                     // bytes a thread owns in the row passes
constexpr int kCsvThreads = 256;                   // threads per tile
constexpr uint32_t kCsvTile = kRun * kCsvThreads;  // 64 KiB
constexpr int kScanBlock = 1024;                   // elements per block of the u64 scan

void csv_err(char *err, size_t len, const char *fmt, ...) {
  if (!err || !len) return;
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(err, len, fmt, ap);
  va_end(ap);
}

#define CSV_CK(call, what)                                                         \
  do {                                                                              \
    cudaError_t e_ = (call);                                                        \
    if (e_ != cudaSuccess) {                                                        \
      csv_err(err, err_len, "%s: %s", what, cudaGetErrorString(e_));                \
      return e_ == cudaErrorMemoryAllocation ? WARPJQ_ERR_OOM : WARPJQ_ERR_CUDA;    \
    }                                                                               \
  } while (0)

// Block-wide exclusive scan (+ or ^) of one u64 per thread; `total` gets
// the whole block's.  Every thread of the block must call it.
template <bool kXor>
__device__ u64 block_excl(u64 v, u64 &total) {
  __shared__ u64 s_w[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  u64 inc = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const u64 x = __shfl_up_sync(0xffffffffu, inc, d);
    if (lane >= d) inc = kXor ? (inc ^ x) : (inc + x);
  }
  if (lane == 31) s_w[warp] = inc;
  __syncthreads();
  u64 before = 0, all = 0;
  for (int w = 0; w < nw; w++) {
    if (w < warp) before = kXor ? (before ^ s_w[w]) : (before + s_w[w]);
    all = kXor ? (all ^ s_w[w]) : (all + s_w[w]);
  }
  total = all;
  __syncthreads();
  return kXor ? (before ^ inc ^ v) : (before + inc - v);
}

// Quote and newline masks of the 16-byte aligned block at `blk`.
__device__ __forceinline__ void block_masks(const uint8_t *blk, uint32_t &q, uint32_t &nl) {
  const uint4 v = __ldg(reinterpret_cast<const uint4 *>(blk));
  q = eq4(v.x, 0x22222222u) | eq4(v.y, 0x22222222u) << 4 | eq4(v.z, 0x22222222u) << 8 |
      eq4(v.w, 0x22222222u) << 12;
  nl = eq4(v.x, 0x0A0A0A0Au) | eq4(v.y, 0x0A0A0A0Au) << 4 | eq4(v.z, 0x0A0A0A0Au) << 8 |
       eq4(v.w, 0x0A0A0A0Au) << 12;
}

// Inclusive prefix XOR of a 16-bit mask: bit j = parity of bits 0..j.
__device__ __forceinline__ uint32_t pxor16(uint32_t x) {
  x ^= x << 1;
  x ^= x << 2;
  x ^= x << 4;
  x ^= x << 8;
  return x & 0xFFFFu;
}

// Walks the bytes [a, b) of `d` in 16-byte aligned blocks (a block that
// holds one byte of the range lies in the same page as that byte, so the
// aligned loads stay in mapped memory).  For each block: f(block offset
// from d, quote mask, newline mask), both limited to the range.
template <typename F>
__device__ __forceinline__ void for_blocks(const uint8_t *d, u64 a, u64 b, F &&f) {
  if (a >= b) return;
  const uintptr_t pa = (uintptr_t)(d + a), pb = (uintptr_t)(d + b);
  for (uintptr_t blk = pa & ~(uintptr_t)15; blk < pb; blk += 16) {
    const uint32_t lo = blk < pa ? (uint32_t)(pa - blk) : 0;
    const uint32_t hi = pb - blk < 16 ? (uint32_t)(pb - blk) : 16;
    const uint32_t valid = ((1u << hi) - 1) & ~((1u << lo) - 1);
    uint32_t q, nl;
    block_masks(reinterpret_cast<const uint8_t *>(blk), q, nl);
    f((long long)(blk - (uintptr_t)d), q & valid, nl & valid);
  }
}

// Per run (u32): bit 0 quote parity, bits 1..11 newlines outside quotes
// when the run starts outside, bits 12..22 all newlines.  Per tile (u64):
// bit 0 parity, bits 1..31 the same outside count, bits 32..63 all newlines.
__global__ void __launch_bounds__(kCsvThreads) k_csv_stats(const uint8_t *d, u64 n, uint32_t *run_stat,
                                                           u64 *tile_stat) {
  const u64 a = (u64)blockIdx.x * kCsvTile + (u64)threadIdx.x * kRun;
  const u64 b = a + kRun < n ? a + kRun : n;
  uint32_t s = 0, c0 = 0, nlt = 0;
  for_blocks(d, a, b, [&](long long, uint32_t q, uint32_t nl) {
    const uint32_t inq = pxor16(q) ^ (s ? 0xFFFFu : 0u);
    c0 += __popc(nl & ~inq);
    nlt += __popc(nl);
    s ^= __popc(q) & 1;
  });
  run_stat[(u64)blockIdx.x * kCsvThreads + threadIdx.x] = s | c0 << 1 | nlt << 12;
  u64 ptot, ctot, ntot;
  const u64 sb = block_excl<true>(s, ptot);  // quote parity before this run, within the tile
  block_excl<false>(sb ? nlt - c0 : c0, ctot);
  block_excl<false>(nlt, ntot);
  if (threadIdx.x == 0) tile_stat[blockIdx.x] = (ptot & 1) | ctot << 1 | ntot << 32;
}

// One block: each tile's start state (inside quotes or not) and the rows
// ended before it; info[0] = rows ended by a newline.
__global__ void __launch_bounds__(1024) k_csv_tiles(const u64 *tile_stat, u64 n_tiles, uint32_t *tile_state,
                                                    u64 *tile_row, u64 *info) {
  const u64 per = (n_tiles + blockDim.x - 1) / blockDim.x;
  const u64 a = threadIdx.x * per < n_tiles ? threadIdx.x * per : n_tiles;
  const u64 b = a + per < n_tiles ? a + per : n_tiles;
  u64 p = 0;
  for (u64 t = a; t < b; t++) p ^= tile_stat[t] & 1;
  u64 ptot;
  const uint32_t s0 = (uint32_t)block_excl<true>(p, ptot);
  uint32_t s = s0;
  u64 rows = 0;
  for (u64 t = a; t < b; t++) {
    const u64 ts = tile_stat[t];
    const u64 c0 = (ts >> 1) & 0x7FFFFFFFull, nlt = ts >> 32;
    rows += s ? nlt - c0 : c0;
    s ^= (uint32_t)(ts & 1);
  }
  u64 rtot;
  u64 base = block_excl<false>(rows, rtot);
  s = s0;
  for (u64 t = a; t < b; t++) {
    const u64 ts = tile_stat[t];
    const u64 c0 = (ts >> 1) & 0x7FFFFFFFull, nlt = ts >> 32;
    tile_state[t] = s;
    tile_row[t] = base;
    base += s ? nlt - c0 : c0;
    s ^= (uint32_t)(ts & 1);
  }
  if (threadIdx.x == 0) info[0] = rtot;
}

// Writes the offset of every row-ending newline, in order.
__global__ void __launch_bounds__(kCsvThreads) k_csv_row_ends(const uint8_t *d, u64 n, const uint32_t *run_stat,
                                                              const uint32_t *tile_state, const u64 *tile_row,
                                                              u64 *row_end) {
  const u64 a = (u64)blockIdx.x * kCsvTile + (u64)threadIdx.x * kRun;
  const u64 b = a + kRun < n ? a + kRun : n;
  const uint32_t st = run_stat[(u64)blockIdx.x * kCsvThreads + threadIdx.x];
  const uint32_t p = st & 1, c0 = (st >> 1) & 0x7FF, nlt = (st >> 12) & 0x7FF;
  u64 tot;
  uint32_t s = (uint32_t)block_excl<true>(p, tot) ^ tile_state[blockIdx.x];
  u64 idx = block_excl<false>(s ? nlt - c0 : c0, tot) + tile_row[blockIdx.x];
  for_blocks(d, a, b, [&](long long off, uint32_t q, uint32_t nl) {
    const uint32_t inq = pxor16(q) ^ (s ? 0xFFFFu : 0u);
    uint32_t m = nl & ~inq;
    while (m) {
      const int j = __ffs(m) - 1;
      m &= m - 1;
      row_end[idx++] = (u64)(off + j);
    }
    s ^= __popc(q) & 1;
  });
}

// info[0] (rows ended by a newline) -> rows; info[1] = bytes consumed (up
// to and with the last row's newline, or all when `final`); info[2] = the
// first row's end.  With `final`, a last row without a newline ends at n.
__global__ void k_csv_close(u64 *row_end, u64 n, int final_, u64 *info) {
  u64 r = info[0];
  const u64 start = r ? row_end[r - 1] + 1 : 0;
  if (final_ && start < n) row_end[r++] = n;
  info[0] = r;
  info[1] = final_ ? n : start;
  info[2] = r ? row_end[0] : 0;
}

// Rows to NDJSON, 32 rows a warp (one warp a block), a lane a row.  The rows'
// bytes are staged in shared memory (they are contiguous, so the loads are
// whole blocks), and every 32 of them become a mask of the bytes a row's walk
// has to look at: ',' '"' '\\' and control bytes.  A lane then steps from hit
// to hit, takes a field's kind from its first byte and its end, and moves
// everything else a word at a time; the lines, contiguous too, are put
// together in shared memory and written out as whole blocks.  A thread a row
// over global memory, stepping a word at a time through every byte, was bound
// by its instructions: 256 MB of CSV took 762 us for the lengths and 1,111 us
// for the bytes; 179 and 783 so.  What bounds the second now is latency: 14 KB
// of windows leave 15 warps an SM, and the lanes' escapes fall on different
// bytes.  (Copying short pieces byte by byte took 857, byte by byte through
// the fields with escapes 938.)
constexpr uint32_t kCsvWin = 5120;   // staged input bytes, at most
constexpr uint32_t kCsvOut = 8192;   // staged output bytes, at most

// The windows of one launch: room for 32 rows of the average length and a
// quarter, so that short rows leave shared memory for more warps (64 MB of rows
// of 30 bytes: 562 us with the largest windows, 434 so).  Both 0: every row goes
// by row_json.
struct CsvWin {
  uint32_t in, out;  // bytes; out 0: no output is staged
  __host__ __device__ uint32_t mask_words() const { return (in / 32 + 2 + 3) & ~3u; }
  __host__ __device__ uint32_t out_at() const { return in + 64 + mask_words() * 4; }
  __host__ __device__ uint32_t smem() const { return out_at() + (out ? out + 16 : 0u); }
};
uint32_t csv_room(u64 bytes, u64 rows, uint32_t most) {
  return (uint32_t)std::min<u64>(most, std::max<u64>(1024, (40 * bytes / rows + 127) & ~(u64)31));
}

// Whether lines are better written by row_json, a lane a row over global memory.
// With fewer rows in a window than lanes, what the windows save at each field's
// bytes is lost on the lanes that wait through its steps.  Measured on 64 MB,
// the windows against row_json, us: 50 columns of 7 bytes, lines of 950 bytes
// 1,373 and 897; 30 of 25 bytes, lines of 1,000, 855 and 551; 40 of 3 bytes,
// lines of 430, 957 and 689; 10 of 3 bytes, lines of 110, 533 and 673; 4 of 75
// bytes 308 and 486, of 250 bytes 359 and 743.
bool csv_direct(u64 in, u64 out, u64 rows, u64 columns) {
  return columns > 8 && out > rows * (in < 6 * columns * rows ? 320u : 560u);
}

// The hits of eight words: ',' '"' '\\' and bytes below 0x20 (devutil.cuh
// flags_special, with ',').
__device__ __forceinline__ uint32_t csv_hits(const uint32_t w[8]) {
  uint32_t f[8];
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const uint32_t t = (w[k] ^ 0x02020202u) & 0x7F7F7F7Fu;
    const uint32_t sq = t + 0x5F5F5F5Fu, sb = (t ^ 0x5E5E5E5Eu) + 0x7F7F7F7Fu, sc = (t ^ 0x2E2E2E2Eu) + 0x7F7F7F7Fu;
    f[k] = ~((sq & sb & sc) | w[k]) & 0x80808080u;
  }
  return wjq::flags_gather(f);
}

// Output into shared memory from byte `at` on, a word at a time; the words a
// line shares with its neighbours are written bytewise.
struct LineOut {
  uint32_t *o;
  uint32_t first;   // the word the line starts in, when it starts within it
  uint32_t skip;    // that word's bytes before the line
  uint32_t w, off;  // the word being filled, its bytes so far
  uint32_t acc;     // and those
  __device__ __forceinline__ LineOut(uint32_t *o_, uint32_t at)
      : o(o_), first(at & 3 ? at >> 2 : 0xFFFFFFFFu), skip(at & 3), w(at >> 2), off(at & 3), acc(0) {}
  __device__ __forceinline__ void bytes(uint32_t x, uint32_t n) {  // bytes up to n of word w
    for (uint32_t j = w == first ? skip : 0u; j < n; j++) ((uint8_t *)o)[4 * w + j] = (uint8_t)(x >> (8 * j));
  }
  __device__ __forceinline__ void put(uint32_t v, uint32_t k) {  // the k (1..4) low bytes of v, the others zero
    const uint32_t x = acc | v << (8 * off);
    const uint32_t n = off + k;
    if (n < 4) {
      acc = x;
      off = n;
    } else {
      if (w == first) bytes(x, 4);
      else o[w] = x;
      w++;
      acc = __funnelshift_l(v, 0u, 8 * off);  // what did not fit
      off = n - 4;
    }
  }
  __device__ __forceinline__ void flush() { bytes(acc, off); }
  // Bytes [a, b) of the window: up to the next word of the output, then whole
  // words straight across, then the rest.
  __device__ __forceinline__ void copy(const uint8_t *win, uint32_t a, uint32_t b) {
    if (off && a < b) {
      const uint32_t k = min(4 - off, b - a);
      put(wjq::detail::load4(win, a) & (0xFFFFFFFFu >> (32 - 8 * k)), k);
      a += k;
    }
    if (a >= b) return;
    const uint32_t *q = (const uint32_t *)win + (a >> 2);
    const uint32_t sh = (a & 3u) * 8u;
    uint32_t lo = *q;
#pragma unroll 1
    for (; a + 4 <= b; a += 4) {
      const uint32_t hi = *++q;
      o[w++] = __funnelshift_r(lo, hi, sh);
      lo = hi;
    }
    off = b - a;
    acc = off ? __funnelshift_r(lo, q[1], sh) & (0xFFFFFFFFu >> (32 - 8 * off)) : 0u;
  }
  __device__ __forceinline__ void escape(uint32_t c) {
    const uint32_t two = c == '\n' ? 'n' : c == '\r' ? 'r' : c == '\t' ? 't' : c == 8 ? 'b' : c == 12 ? 'f'
                         : c >= 0x20 ? c : 0u;
    if (two) {
      put('\\' | two << 8, 2);
    } else {
      const uint32_t l = c & 15;
      put('\\' | 'u' << 8 | '0' << 16 | (uint32_t)'0' << 24, 4);
      put((uint32_t)('0' + (c >> 4)) | (uint32_t)(l < 10 ? '0' + l : 'a' + l - 10) << 8, 2);
    }
  }
};

// One row w[s, e) of a window (hits in sm; w[e] is a hit): its NDJSON length,
// and with kWrite its bytes.  The fields' rules are row_json's.
template <bool kWrite>
__device__ __forceinline__ uint32_t row_line(const uint8_t *w, const uint32_t *sm, uint32_t s, uint32_t e, bool on,
                                             const KeySet &ks, LineOut &o) {
  if (on && e > s && w[e - 1] == '\r') e--;
  const bool empty = e == s;
  uint32_t len = 3, p = s;  // "{" "}\n"
  bool more = on && !empty;
  if (kWrite && more) o.put('{', 1);
#pragma unroll 1
  for (uint32_t k = 0; k < ks.n && __any_sync(0xffffffffu, more); k++) {
    const uint32_t kw = __ldg(ks.meta + 2 * k), kl = __ldg(ks.meta + 2 * k + 1);
    if (more) {
      len += kl;
      if (kWrite)
#pragma unroll 1
        for (uint32_t j = 0; j < kl; j += 4) o.put(__ldg(ks.text + kw + (j >> 2)), min(kl - j, 4u));
    }
    __syncwarp();
    // the field's text [a, b), and whether it holds bytes to escape
    const uint32_t c = more && p < e ? w[p] : 0u;
    const bool quoted = c == '"';
    const uint32_t a = quoted ? p + 1 : p;
    uint32_t b = a, extra = 0;
    bool esc = false, go = more;
#pragma unroll 1
    while (go) {
      b = min(wjq::detail::next_special(sm, b), e);
      const uint32_t x = w[b];
      if (b == e) {
        go = false;
      } else if (x == ',') {
        go = quoted;
        b += quoted;
      } else if (x != '"') {
        esc = true;
        extra += esc_len((uint8_t)x) - 1;
        b++;
      } else if (!quoted) {
        esc = true;
        extra++;
        b++;
      } else if (b + 1 < e && w[b + 1] == '"') {  // a doubled quote stays two bytes
        esc = true;
        b += 2;
      } else {
        go = false;
      }
    }
    __syncwarp();
    if (more) {
      p = quoted && b < e ? b + 1 : b;  // past the closing quote
      // bytes after it, kept up to the next ',': [p, t)
      uint32_t t = p;
      if (quoted)
#pragma unroll 1
        while (t < e && w[t] != ',') {
          const uint32_t h = min(wjq::detail::next_special(sm, t), e);
          if (h < e && w[h] != ',') extra += esc_len(w[h]) - 1;
          t = h + (h < e && w[h] != ',');
        }
      const bool null = !quoted && b == a;
      const bool number = !quoted && !esc && !null && (c == '-' || c - '0' < 10u) && wjq::detail::win_number(w, a, c) == b;
      const bool str = !null && !number;
      len += null ? 4u : b - a + (t - p) + extra + (str ? 2u : 0u);
      if (kWrite) {
        if (null) o.put('n' | 'u' << 8 | 'l' << 16 | (uint32_t)'l' << 24, 4);
        if (str) o.put('"', 1);
        auto escaped = [&](uint32_t q, uint32_t end, bool doubled) {
#pragma unroll 1
          while (q < end) {
            const uint32_t h = min(wjq::detail::next_special(sm, q), end);
            o.copy(w, q, h);
            q = h;
            if (h < end) {
              const uint32_t x = w[h];
              if (x == ',') o.put(',', 1);
              else o.escape(x);
              q += x == '"' && doubled ? 2 : 1;
            }
          }
        };
        if (esc) escaped(a, b, quoted);
        else if (!null) o.copy(w, a, b);
        if (t > p) escaped(p, t, false);
        if (str) o.put('"', 1);
      }
      more = t < e;  // a ',' follows
      p = t + 1;
    }
    __syncwarp();
  }
  if (kWrite && on) {
    if (empty) o.put('\n', 1);
    else o.put('}' | '\n' << 8, 2);
    o.flush();
  }
  return empty ? 1u : len;
}

// A row by row_json over global memory, out of line: the rows of the windows
// lose registers to it otherwise (64 MB of rows of 600 bytes: 357 us inline, 333 so).
template <bool kWrite>
__device__ __noinline__ u64 row_far(const uint8_t *d, u64 s, u64 e, KeySet ks, uint8_t *to) {
  WordIn in(d);
  WordOut wo(to);
  const u64 len = row_json<kWrite>(in, s, e, ks, wo);
  if (kWrite) wo.flush();
  return len;
}

// Rows [row0, rows) of the chunk: pass 0 writes the NDJSON length of line r -
// row0 to len_off, pass 1 writes the line at out + len_off[r - row0] (len_off
// by then an exclusive prefix, *total the end of the last line).  A warp takes
// as many of its 32 rows at once as fit the staged windows, after those that fit
// none alone, which go by row_json all at once (one after another, 64 MB of rows
// of 8,000 bytes took 34.7 ms; 5.2 so).
template <bool kWrite>
__global__ void __launch_bounds__(32) k_csv_json(const uint8_t *d, const u64 *row_end, u64 row0, u64 rows, KeySet ks,
                                                 u64 *len_off, uint8_t *out, const u64 *total, CsvWin room) {
  extern __shared__ __align__(16) uint8_t csv_sm[];
  uint8_t *win = csv_sm;
  uint32_t *mask = (uint32_t *)(csv_sm + room.in + 64);
  uint32_t *obuf = (uint32_t *)(csv_sm + room.out_at());
  const uint32_t lane = threadIdx.x;
  for (u64 base = row0 + blockIdx.x * 32ull; base < rows; base += gridDim.x * 32ull) {
    const u64 r = base + lane;
    const uint32_t n_here = (uint32_t)min((u64)32, rows - base);
    const bool mine = lane < n_here;
    u64 s = 0, e = 0, o0 = 0, o1 = 0;  // the row, and its line in the output
    if (mine) {
      s = r ? __ldg(row_end + r - 1) + 1 : 0;
      e = __ldg(row_end + r);
      if (kWrite) {
        o0 = len_off[r - row0];
        o1 = r + 1 < rows ? len_off[r + 1 - row0] : *total;
      }
    }
    // Rows too long for the windows go by row_json, each lane its own, and with
    // them those that a window holds few of.
    bool big = mine && (e - s + 15 >= room.in || (kWrite && o1 - o0 + 15 > room.out));
    if (__any_sync(0xffffffffu, big)) big = big || (mine && 4 * (e - s) >= room.in);
    if (big) {
      const u64 len = row_far<kWrite>(d, s, e, ks, kWrite ? out + o0 : nullptr);
      if (!kWrite) len_off[r - row0] = len;
    }
    const unsigned gone = __ballot_sync(0xffffffffu, big);
    for (uint32_t lo = 0; lo < n_here;) {
      if (gone >> lo & 1u) {
        lo++;
        continue;
      }
      const u64 s_lo = __shfl_sync(0xffffffffu, s, lo), o_lo = __shfl_sync(0xffffffffu, o0, lo);
      const u64 w0 = (u64)((uintptr_t)(d + s_lo) & 15u);  // the window starts at a block
      const uint32_t lead = (uint32_t)((uintptr_t)(out + o_lo) & 15u);
      const bool fits = mine && !big && lane >= lo && e - s_lo + w0 < room.in && (!kWrite || o1 - o_lo + lead <= room.out);
      const unsigned m = __ballot_sync(0xffffffffu, fits) >> lo;
      const uint32_t take = m == 0xFFFFFFFFu ? 32u : (uint32_t)__ffs(~m) - 1u;  // rows lo .. lo + take fit, one at least
      const bool on = fits && lane < lo + take;
      const uint32_t hi = lo + take - 1;
      const uint32_t n_win = (uint32_t)(__shfl_sync(0xffffffffu, e, hi) - s_lo + w0);
      const uint4 *src = (const uint4 *)((uintptr_t)(d + s_lo) & ~(uintptr_t)15);
      // whole blocks, each holding a byte of the rows
      for (uint32_t k = lane; 16 * k < n_win; k += 32) ((uint4 *)win)[k] = __ldg(src + k);
      __syncwarp();
      if (lane == 0) win[n_win] = '\n';  // ends the last row
      __syncwarp();
      for (uint32_t k = lane; 32 * k <= n_win; k += 32) {
        const uint4 u = ((const uint4 *)win)[2 * k], v = ((const uint4 *)win)[2 * k + 1];
        const uint32_t w8[8] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w};
        mask[k] = csv_hits(w8);
      }
      __syncwarp();
      const uint32_t ws = on ? (uint32_t)(s - s_lo + w0) : 0u, we = on ? (uint32_t)(e - s_lo + w0) : 0u;
      const uint32_t at = on ? (uint32_t)(o0 - o_lo) + lead : 0u;
      LineOut o(obuf, at);
      const uint32_t len = row_line<kWrite>(win, mask, ws, we, on, ks, o);
      __syncwarp();
      if (!kWrite) {
        if (on) len_off[r - row0] = len;
      } else {
        // whole blocks, and the bytes around them
        const uint32_t end = (uint32_t)(__shfl_sync(0xffffffffu, o1, hi) - o_lo) + lead;
        uint8_t *dst = out + o_lo - lead;
        for (uint32_t k = 16 * lane; k < end; k += 512) {
          if (k >= lead && k + 16 <= end) {
            *(uint4 *)(dst + k) = *(const uint4 *)((const uint8_t *)obuf + k);
          } else {
            for (uint32_t j = max(k, lead); j < min(k + 16, end); j++) dst[j] = ((const uint8_t *)obuf)[j];
          }
        }
        __syncwarp();
      }
      lo += take;
    }
  }
}

// Exclusive prefix sum of v[0, m) in place, as block totals, one block over
// the totals, and a per-block add; the grand total goes to *total.
__global__ void __launch_bounds__(256) k_sum_blocks(u64 *v, u64 m, u64 *bt) {
  const u64 i0 = (u64)blockIdx.x * kScanBlock + threadIdx.x * (kScanBlock / 256);
  u64 loc[kScanBlock / 256];
  u64 s = 0;
#pragma unroll
  for (int k = 0; k < kScanBlock / 256; k++) {
    loc[k] = i0 + k < m ? v[i0 + k] : 0;
    s += loc[k];
  }
  u64 tot;
  u64 ex = block_excl<false>(s, tot);
#pragma unroll
  for (int k = 0; k < kScanBlock / 256; k++) {
    if (i0 + k < m) v[i0 + k] = ex;
    ex += loc[k];
  }
  if (threadIdx.x == 0) bt[blockIdx.x] = tot;
}

__global__ void __launch_bounds__(1024) k_sum_totals(u64 *bt, u64 nb, u64 *total) {
  const u64 per = (nb + blockDim.x - 1) / blockDim.x;
  const u64 a = threadIdx.x * per < nb ? threadIdx.x * per : nb;
  const u64 b = a + per < nb ? a + per : nb;
  u64 s = 0;
  for (u64 i = a; i < b; i++) s += bt[i];
  u64 tot;
  u64 ex = block_excl<false>(s, tot);
  for (u64 i = a; i < b; i++) {
    const u64 x = bt[i];
    bt[i] = ex;
    ex += x;
  }
  if (threadIdx.x == 0) *total = tot;
}

__global__ void __launch_bounds__(256) k_sum_add(u64 *v, u64 m, const u64 *bt) {
  const u64 i0 = (u64)blockIdx.x * kScanBlock + threadIdx.x;
  const u64 base = bt[blockIdx.x];
#pragma unroll
  for (int k = 0; k < kScanBlock; k += 256)
    if (i0 + k < m) v[i0 + k] += base;
}

// Copies slices src[off[i], off[i] + len[i]) to dst[dst_off[i], ...), a warp per slice.
__global__ void k_gather(const uint8_t *src, const u64 *off, const uint32_t *len, const u64 *dst_off, u64 n,
                         uint8_t *dst) {
  const u64 wid = (blockIdx.x * (u64)blockDim.x + threadIdx.x) >> 5;
  const uint32_t lane = threadIdx.x & 31;
  for (u64 i = wid; i < n; i += ((u64)gridDim.x * blockDim.x) >> 5)
    for (uint32_t j = lane; j < len[i]; j += 32) dst[dst_off[i] + j] = src[off[i] + j];
}

template <typename T>
struct DBuf {  // device buffer that only grows
  T *p = nullptr;
  size_t n = 0;
  cudaError_t ensure(size_t want) {  // grows by at least 1.5x (cudaFree synchronises the device)
    if (want <= n) return cudaSuccess;
    want = std::max(want + want / 8, n + n / 2);
    if (p) cudaFree(p);
    p = nullptr;
    n = 0;
    cudaError_t e = cudaMalloc((void **)&p, want * sizeof(T));
    if (e == cudaSuccess) n = want;
    return e;
  }
  void release() {
    if (p) cudaFree(p);
    p = nullptr;
    n = 0;
  }
};

}  // namespace

struct warpjq_csv {
  DBuf<uint8_t> in;  // device copy of host input
  DBuf<uint32_t> run_stat, tile_state, keys, key_off, g_len;  // keys: key texts by words; key_off: their meta
  DBuf<u64> tile_stat, tile_row, row_end, lens, bt, info, g_off, g_dst;
  DBuf<uint8_t> out, g_out;
  bool have_header = false;  // header names taken from an earlier chunk
  std::string key_text;
  std::vector<uint32_t> key_offs, key_words, key_meta;
  // chunks staged from host memory on a copy stream of their own
  DBuf<uint8_t> stage[2];
  cudaStream_t copy = nullptr;
  cudaEvent_t staged[2] = {nullptr, nullptr};
  ~warpjq_csv() {
    if (copy) cudaStreamSynchronize(copy);
    for (int b = 0; b < 2; b++) {
      stage[b].release();
      if (staged[b]) cudaEventDestroy(staged[b]);
    }
    if (copy) cudaStreamDestroy(copy);
    in.release();
    run_stat.release();
    tile_state.release();
    key_off.release();
    g_len.release();
    tile_stat.release();
    tile_row.release();
    row_end.release();
    lens.release();
    bt.release();
    info.release();
    g_off.release();
    g_dst.release();
    keys.release();
    out.release();
    g_out.release();
  }
};

extern "C" {

warpjq_status warpjq_csv_create(warpjq_csv **out) {
  if (!out) return WARPJQ_ERR_INVALID_ARG;
  *out = new (std::nothrow) warpjq_csv();
  return *out ? WARPJQ_OK : WARPJQ_ERR_OOM;
}

void warpjq_csv_destroy(warpjq_csv *c) { delete c; }

void warpjq_csv_reset(warpjq_csv *c) {
  if (!c) return;
  c->have_header = false;
  c->key_text.clear();
  c->key_offs.clear();
  c->key_words.clear();
  c->key_meta.clear();
}

warpjq_status warpjq_csv_convert(warpjq_csv *c, const uint8_t *src, uint64_t n, uint32_t flags, void *stream,
                                 const uint8_t **d_ndjson, uint64_t *ndjson_len, uint64_t *consumed,
                                 uint64_t *records, char *err, size_t err_len) {
  if (!c || (!src && n) || !d_ndjson || !ndjson_len || !consumed) {
    csv_err(err, err_len, "invalid argument");
    return WARPJQ_ERR_INVALID_ARG;
  }
  cudaStream_t st = (cudaStream_t)stream;
  const bool final_ = (flags & WARPJQ_CSV_FINAL) != 0;
  *d_ndjson = nullptr;
  *ndjson_len = 0;
  *consumed = 0;
  if (records) *records = 0;
  if (n == 0) return WARPJQ_OK;
  const uint8_t *d = src;
  for (int b = 0; b < 2; b++)
    if ((flags & (WARPJQ_CSV_AFTER_STAGE0 << b)) && c->staged[b])
      CSV_CK(cudaStreamWaitEvent(st, c->staged[b], 0), "wait for a staged chunk");
  if (flags & WARPJQ_CSV_HOST_INPUT) {
    CSV_CK(c->in.ensure(n + 16), "device memory for the CSV input");
    CSV_CK(cudaMemcpyAsync(c->in.p, src, n, cudaMemcpyHostToDevice, st), "copy of the CSV input");
    d = c->in.p;
  }
  const u64 tiles = (n + kCsvTile - 1) / kCsvTile;
  CSV_CK(c->run_stat.ensure(tiles * kCsvThreads), "device memory for CSV rows");
  CSV_CK(c->tile_stat.ensure(tiles), "device memory for CSV rows");
  CSV_CK(c->tile_state.ensure(tiles), "device memory for CSV rows");
  CSV_CK(c->tile_row.ensure(tiles), "device memory for CSV rows");
  CSV_CK(c->info.ensure(4), "device memory for CSV rows");
  // rows ended by a newline outside quotes
  k_csv_stats<<<(unsigned)tiles, kCsvThreads, 0, st>>>(d, n, c->run_stat.p, c->tile_stat.p);
  k_csv_tiles<<<1, 1024, 0, st>>>(c->tile_stat.p, tiles, c->tile_state.p, c->tile_row.p, c->info.p);
  CSV_CK(cudaGetLastError(), "CSV row count");
  u64 nl_rows = 0;
  CSV_CK(cudaMemcpyAsync(&nl_rows, c->info.p, 8, cudaMemcpyDeviceToHost, st), "CSV row count");
  CSV_CK(cudaStreamSynchronize(st), "CSV row count");
  CSV_CK(c->row_end.ensure(nl_rows + 1), "device memory for CSV rows");
  k_csv_row_ends<<<(unsigned)tiles, kCsvThreads, 0, st>>>(d, n, c->run_stat.p, c->tile_state.p, c->tile_row.p,
                                                          c->row_end.p);
  k_csv_close<<<1, 1, 0, st>>>(c->row_end.p, n, final_ ? 1 : 0, c->info.p);
  CSV_CK(cudaGetLastError(), "CSV row ends");
  u64 info[3];
  CSV_CK(cudaMemcpyAsync(info, c->info.p, 24, cudaMemcpyDeviceToHost, st), "CSV row ends");
  CSV_CK(cudaStreamSynchronize(st), "CSV row ends");
  const u64 rows = info[0];
  u64 row0 = 0;
  if (!c->have_header) {
    if (rows == 0) return WARPJQ_OK;  // no whole row yet: the caller passes more bytes
    const u64 h_end = info[2];
    std::vector<uint8_t> head(h_end);
    if (h_end) {
      if (flags & WARPJQ_CSV_HOST_INPUT) memcpy(head.data(), src, h_end);
      else CSV_CK(cudaMemcpy(head.data(), d, h_end, cudaMemcpyDeviceToHost), "copy of the CSV header");
    }
    parse_header(head.data(), head.size(), c->key_text, c->key_offs);
    pack_keys(c->key_text, c->key_offs, c->key_words, c->key_meta);
    CSV_CK(c->keys.ensure(c->key_words.size() + 1), "device memory for CSV keys");
    CSV_CK(c->key_off.ensure(c->key_meta.size() + 1), "device memory for CSV keys");
    if (!c->key_words.empty())
      CSV_CK(cudaMemcpyAsync(c->keys.p, c->key_words.data(), c->key_words.size() * 4, cudaMemcpyHostToDevice, st),
             "copy of the CSV keys");
    if (!c->key_meta.empty())
      CSV_CK(cudaMemcpyAsync(c->key_off.p, c->key_meta.data(), c->key_meta.size() * 4, cudaMemcpyHostToDevice, st),
             "copy of the CSV keys");
    c->have_header = true;
    row0 = 1;
  }
  *consumed = info[1];
  const u64 m = rows - row0;
  if (records) *records = m;
  if (m == 0) return WARPJQ_OK;
  KeySet ks{c->keys.p, c->key_off.p, (uint32_t)(c->key_meta.size() / 2)};
  CSV_CK(c->lens.ensure(m + 1), "device memory for CSV lines");
  const unsigned grid = (unsigned)std::min<u64>((m + 31) / 32, 148ull * 256);
  CsvWin room{csv_room(n, rows, kCsvWin), 0};
  k_csv_json<false><<<grid, 32, room.smem(), st>>>(d, c->row_end.p, row0, rows, ks, c->lens.p, nullptr, nullptr, room);
  const u64 nb = (m + kScanBlock - 1) / kScanBlock;
  CSV_CK(c->bt.ensure(nb), "device memory for CSV lines");
  k_sum_blocks<<<(unsigned)nb, 256, 0, st>>>(c->lens.p, m, c->bt.p);
  k_sum_totals<<<1, 1024, 0, st>>>(c->bt.p, nb, c->info.p + 3);
  k_sum_add<<<(unsigned)nb, 256, 0, st>>>(c->lens.p, m, c->bt.p);
  CSV_CK(cudaGetLastError(), "CSV line lengths");
  u64 total = 0;
  CSV_CK(cudaMemcpyAsync(&total, c->info.p + 3, 8, cudaMemcpyDeviceToHost, st), "CSV line lengths");
  CSV_CK(cudaStreamSynchronize(st), "CSV line lengths");
  CSV_CK(c->out.ensure(total + 16), "device memory for the NDJSON");
  room.out = csv_room(total, m, kCsvOut);
  if (csv_direct(n, total, m, ks.n)) room.in = room.out = 0;
  k_csv_json<true><<<grid, 32, room.smem(), st>>>(d, c->row_end.p, row0, rows, ks, c->lens.p, c->out.p,
                                                  c->info.p + 3, room);
  CSV_CK(cudaGetLastError(), "CSV to NDJSON");
  *d_ndjson = c->out.p;
  *ndjson_len = total;
  return WARPJQ_OK;
}

warpjq_status warpjq_csv_stage(warpjq_csv *c, uint32_t buf, uint64_t at, const uint8_t *h_src, uint64_t n,
                               uint8_t **d_buf, char *err, size_t err_len) {
  if (!c || buf > 1 || (!h_src && n) || !d_buf) {
    csv_err(err, err_len, "invalid argument");
    return WARPJQ_ERR_INVALID_ARG;
  }
  if (!c->copy) {
    CSV_CK(cudaStreamCreateWithFlags(&c->copy, cudaStreamNonBlocking), "copy stream");
    for (int b = 0; b < 2; b++) CSV_CK(cudaEventCreateWithFlags(&c->staged[b], cudaEventDisableTiming), "copy event");
  }
  if (c->stage[buf].n < at + n + 16) {  // the buffer's bytes do not survive growth
    CSV_CK(cudaStreamSynchronize(c->copy), "copy stream");
    CSV_CK(c->stage[buf].ensure(at + n + 16), "device memory for a staged chunk");
  }
  if (n) CSV_CK(cudaMemcpyAsync(c->stage[buf].p + at, h_src, n, cudaMemcpyHostToDevice, c->copy), "staging copy");
  CSV_CK(cudaEventRecord(c->staged[buf], c->copy), "staging copy");
  *d_buf = c->stage[buf].p;
  return WARPJQ_OK;
}

warpjq_status warpjq_csv_stage_wait(warpjq_csv *c, uint32_t buf, char *err, size_t err_len) {
  if (!c || buf > 1) return WARPJQ_ERR_INVALID_ARG;
  if (c->staged[buf]) CSV_CK(cudaEventSynchronize(c->staged[buf]), "staging copy");
  return WARPJQ_OK;
}

warpjq_status warpjq_csv_carry(warpjq_csv *c, const uint8_t *d_src, uint64_t n, uint32_t buf, uint64_t at,
                               void *stream, char *err, size_t err_len) {
  if (!c || buf > 1 || (!d_src && n) || at + n + 16 > c->stage[buf].n) {
    csv_err(err, err_len, "invalid argument");
    return WARPJQ_ERR_INVALID_ARG;
  }
  if (n)
    CSV_CK(cudaMemcpyAsync(c->stage[buf].p + at, d_src, n, cudaMemcpyDeviceToDevice, (cudaStream_t)stream),
           "carried row copy");
  return WARPJQ_OK;
}

warpjq_status warpjq_csv_gather(warpjq_csv *c, const uint8_t *d_src, const uint64_t *offsets,
                                const uint32_t *lengths, uint64_t n, uint8_t *h_dst, void *stream, char *err,
                                size_t err_len) {
  if (!c || (n && (!offsets || !lengths || !h_dst))) {  // d_src null: offsets are addresses
    csv_err(err, err_len, "invalid argument");
    return WARPJQ_ERR_INVALID_ARG;
  }
  if (!n) return WARPJQ_OK;
  cudaStream_t st = (cudaStream_t)stream;
  std::vector<u64> dst(n);
  u64 total = 0;
  for (u64 i = 0; i < n; i++) {
    dst[i] = total;
    total += lengths[i];
  }
  CSV_CK(c->g_off.ensure(n), "device memory for a gather");
  CSV_CK(c->g_dst.ensure(n), "device memory for a gather");
  CSV_CK(c->g_len.ensure(n), "device memory for a gather");
  CSV_CK(c->g_out.ensure(total + 1), "device memory for a gather");
  CSV_CK(cudaMemcpyAsync(c->g_off.p, offsets, n * 8, cudaMemcpyHostToDevice, st), "gather offsets");
  CSV_CK(cudaMemcpyAsync(c->g_dst.p, dst.data(), n * 8, cudaMemcpyHostToDevice, st), "gather offsets");
  CSV_CK(cudaMemcpyAsync(c->g_len.p, lengths, n * 4, cudaMemcpyHostToDevice, st), "gather offsets");
  const unsigned grid = (unsigned)std::min<u64>((n + 7) / 8, 148ull * 16);
  k_gather<<<grid, 256, 0, st>>>(d_src, c->g_off.p, c->g_len.p, c->g_dst.p, n, c->g_out.p);
  CSV_CK(cudaGetLastError(), "gather");
  if (total) CSV_CK(cudaMemcpyAsync(h_dst, c->g_out.p, total, cudaMemcpyDeviceToHost, st), "gather copy");
  CSV_CK(cudaStreamSynchronize(st), "gather");
  return WARPJQ_OK;
}

warpjq_status warpjq_device_read(void *h_dst, const void *d_src, uint64_t n, void *stream, char *err,
                                 size_t err_len) {
  if (!n) return WARPJQ_OK;
  if (!h_dst || !d_src) return WARPJQ_ERR_INVALID_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  CSV_CK(cudaMemcpyAsync(h_dst, d_src, n, cudaMemcpyDeviceToHost, st), "device to host copy");
  CSV_CK(cudaStreamSynchronize(st), "device to host copy");
  return WARPJQ_OK;
}

}  // extern "C"
