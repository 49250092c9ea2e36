// Per-line walker: one thread validates one NDJSON line end to end and, in
// the same pass, records the value of every trie node of the query plan.
//
// Semantics restated from the reference CPU engine:
//   - strict RFC 8259 validation of exactly one value per line
//     (json.rs:198-421): strings reject raw bytes < 0x20 and bad escapes,
//     numbers follow the JSON grammar, literals must be exact, brackets must
//     match;
//   - blank lines are those made only of ASCII whitespace including form
//     feed (chunk.rs:436);
//   - path resolution follows json.rs:444-508: last duplicate key wins,
//     missing/null propagate as Missing, indexing a scalar is a type error,
//     and an invalid line beats a type error.
// The walk is iterative; container depth is tracked in a 64-bit register
// and, for the rare deeper line, in a caller-provided bit stack.
#pragma once

#include "devutil.cuh"
#include "plan.h"

namespace wjq {

enum LineStatus : int {
  LS_OK = 0,
  LS_INVALID = 1,
  LS_TYPE_ERROR = 2,
  LS_BLANK = 4,
  LS_DEEP = 5,       // deeper than the register stack; caller retries with a deep stack
  LS_DEEP_FULL = 6,  // deeper than the deep stack provided
  LS_FALLBACK = 7,   // not the fast path's shape; the general walker decides
};

// Values recorded per trie node for one line; offsets are relative to the
// line start.
struct NodeVals {
  alignas(4) uint8_t kind[kMaxNodes];
  uint8_t esc[kMaxNodes];
  uint32_t off[kMaxNodes];
  uint32_t len[kMaxNodes];
};

// A deep bit stack for levels >= 64 (bit = 1 for arrays), in global memory.
struct DeepStack {
  uint32_t *words;
  uint64_t cap_levels;
};

namespace detail {

enum Expect : int {
  EX_VALUE = 0,
  EX_KEY_OR_CLOSE = 1,
  EX_KEY = 2,
  EX_COLON = 3,
  EX_COMMA_OR_CLOSE = 4,
  EX_VALUE_OR_CLOSE = 5,
  EX_END = 6,
};

// Scans the string whose opening quote is at `s`.  Returns the index of the
// closing quote, or -1 when the string is malformed or unterminated.
__device__ __forceinline__ long long scan_string_bytes(const uint8_t *line, uint32_t n, uint32_t s,
                                                       bool &esc) {
  uint32_t j = s + 1;
  esc = false;
#pragma unroll 1
  for (;;) {
    // Aligned word steps over runs of ordinary bytes.
#pragma unroll 1
    while (((uintptr_t)(line + j) & 3u) == 0 && j + 4 <= n &&
           swar_string_special(*(const uint32_t *)(line + j)) == 0)
      j += 4;
    if (j >= n) return -1;
    uint32_t c = line[j];
    if (c == '"') return j;
    if (c == '\\') {
      if (j + 1 >= n) return -1;
      uint32_t e = line[j + 1];
      esc = true;
      if (e == '"' || e == '\\' || e == '/' || e == 'b' || e == 'f' || e == 'n' || e == 'r' ||
          e == 't') {
        j += 2;
      } else if (e == 'u') {
        if (j + 6 > n) return -1;
        if (hex_val(line[j + 2]) < 0 || hex_val(line[j + 3]) < 0 || hex_val(line[j + 4]) < 0 ||
            hex_val(line[j + 5]) < 0)
          return -1;
        j += 6;
      } else {
        return -1;
      }
      continue;
    }
    if (c < 0x20) return -1;
    j++;
  }
}

// Validates an atom (number or literal) occupying [s, e).
__device__ __forceinline__ bool valid_atom(const uint8_t *p, uint32_t n) {
  uint32_t c = p[0];
  if (c == 't') return n == 4 && p[1] == 'r' && p[2] == 'u' && p[3] == 'e';
  if (c == 'f') return n == 5 && p[1] == 'a' && p[2] == 'l' && p[3] == 's' && p[4] == 'e';
  if (c == 'n') return n == 4 && p[1] == 'u' && p[2] == 'l' && p[3] == 'l';
  // number: -?(0|[1-9][0-9]*)(\.[0-9]+)?([eE][+-]?[0-9]+)?   (json.rs:370-410)
  uint32_t i = 0;
  if (c == '-') i = 1;
  if (i >= n || !is_digit(p[i])) return false;
  if (p[i] == '0') {
    i++;
  } else {
#pragma unroll 1
    while (i < n && is_digit(p[i])) i++;
  }
  if (i < n && p[i] == '.') {
    i++;
    if (i >= n || !is_digit(p[i])) return false;
#pragma unroll 1
    while (i < n && is_digit(p[i])) i++;
  }
  if (i < n && (p[i] == 'e' || p[i] == 'E')) {
    i++;
    if (i < n && (p[i] == '+' || p[i] == '-')) i++;
    if (i >= n || !is_digit(p[i])) return false;
#pragma unroll 1
    while (i < n && is_digit(p[i])) i++;
  }
  return i == n;
}

__device__ __forceinline__ uint8_t kind_of(uint32_t c) {
  switch (c) {
    case '{': return JK_OBJ;
    case '[': return JK_ARR;
    case '"': return JK_STR;
    case 't': case 'f': return JK_BOOL;
    case 'n': return JK_NULL;
    default: return JK_NUM;
  }
}

// Key child of `node` whose decoded key equals the key body, or kNoNode.
__device__ __forceinline__ uint8_t match_key(const DevPlan &P, uint8_t node, const uint8_t *body,
                                             uint32_t len, bool esc) {
#pragma unroll 1
  for (uint8_t c = P.nodes[node].first_child; c != kNoNode; c = P.nodes[c].next_sibling) {
    const PlanNode &nd = P.nodes[c];
    if (nd.is_index) continue;
    if (!esc) {
      if (nd.key_len != len) continue;
      if (len && body[0] != nd.key_first) continue;
      const uint8_t *k = P.blob + nd.key_off;
      uint32_t t = 1;
#pragma unroll 1
      while (t < len && body[t] == k[t]) t++;
      if (t >= len) return c;
    } else if (cmp_str_body(body, len, true, P.blob + nd.key_off, nd.key_len) == 0) {
      return c;
    }
  }
  return kNoNode;
}

__device__ __forceinline__ uint8_t index_child(const DevPlan &P, uint8_t node, uint32_t idx) {
  if (node == kNoNode || !P.nodes[node].has_index_children) return kNoNode;
#pragma unroll 1
  for (uint8_t c = P.nodes[node].first_child; c != kNoNode; c = P.nodes[c].next_sibling) {
    const PlanNode &nd = P.nodes[c];
    if (nd.is_index && nd.index == idx) return c;
  }
  return kNoNode;
}

}  // namespace detail

// Walks `line[0, n)` (no newline; a trailing '\r' is JSON whitespace).
// `deep` may be null: a line nesting past 64 levels then returns LS_DEEP.
__device__ __noinline__ int walk_line(const DevPlan &P, const uint8_t *line, uint32_t n,
                                      NodeVals &v, const DeepStack *deep) {
  using namespace detail;
  const uint32_t n_nodes = P.n_nodes;
#pragma unroll 1
  for (uint32_t k = 0; k < n_nodes; k++) v.kind[k] = JK_MISSING;

  uint32_t i = 0;
#pragma unroll 1
  while (i < n && is_ws(line[i])) i++;
  if (i == n) return LS_BLANK;
  if (line[i] == 0x0C) {  // form feed counts toward a blank line, not toward JSON
#pragma unroll 1
    for (uint32_t j = i; j < n; j++) {
      uint32_t c = line[j];
      if (!(c == ' ' || c == '\t' || c == '\r' || c == 0x0C)) return LS_INVALID;
    }
    return LS_BLANK;
  }

  uint8_t node_at[kMaxDepthFast];  // trie node of the open container at each level
  uint32_t arr_idx[kMaxDepthFast];
  uint64_t stk = 0;                // bit d: container at level d is an array
  uint64_t depth = 0;
  uint8_t pending = n_nodes ? 0 : kNoNode;  // node the next value lands on
  int expect = EX_VALUE;

#pragma unroll 1
  for (;;) {
#pragma unroll 1
    while (i < n && is_ws(line[i])) i++;
    if (i >= n) break;
    uint32_t c = line[i];
    bool close = false;

    if (expect == EX_COLON) {
      if (c != ':') return LS_INVALID;
      i++;
      expect = EX_VALUE;
      continue;
    }
    if (expect == EX_KEY_OR_CLOSE || expect == EX_KEY) {
      if (c == '}' && expect == EX_KEY_OR_CLOSE) {
        close = true;
      } else {
        if (c != '"') return LS_INVALID;
        bool esc;
        long long e = scan_string_bytes(line, n, i, esc);
        if (e < 0) return LS_INVALID;
        uint8_t parent = depth <= kMaxDepthFast ? node_at[depth - 1] : kNoNode;
        pending = kNoNode;
        if (parent != kNoNode && P.nodes[parent].has_key_children)
          pending = match_key(P, parent, line + i + 1, (uint32_t)e - i - 1, esc);
        i = (uint32_t)e + 1;
        expect = EX_COLON;
        continue;
      }
    } else if (expect == EX_COMMA_OR_CLOSE) {
      uint32_t lvl = (uint32_t)depth - 1;
      bool arr;
      if (lvl < 64) {
        arr = (stk >> lvl) & 1;
      } else {
        uint64_t b = lvl - 64;
        arr = (deep->words[b >> 5] >> (b & 31)) & 1;
      }
      if (c == ',') {
        i++;
        if (arr) {
          pending = kNoNode;
          if (lvl < kMaxDepthFast) {
            uint32_t idx = ++arr_idx[lvl];
            pending = index_child(P, node_at[lvl], idx);
          }
          expect = EX_VALUE;
        } else {
          expect = EX_KEY;
        }
        continue;
      }
      if ((c == '}' && !arr) || (c == ']' && arr)) {
        close = true;
      } else {
        return LS_INVALID;
      }
    } else if (expect == EX_END) {
      return LS_INVALID;
    } else if (expect == EX_VALUE_OR_CLOSE && c == ']') {
      close = true;
    }

    if (close) {
      depth--;
      if (depth < kMaxDepthFast) {
        uint8_t cn = node_at[depth];
        if (cn != kNoNode) v.len[cn] = i + 1 - v.off[cn];
      }
      i++;
      expect = depth == 0 ? EX_END : EX_COMMA_OR_CLOSE;
      continue;
    }

    // A value starts at i (expect is EX_VALUE or EX_VALUE_OR_CLOSE).
    uint8_t vn = pending;
    if (vn != kNoNode) {
#pragma unroll 1
      for (uint32_t k = vn + 1u; k < P.nodes[vn].subtree_end; k++) v.kind[k] = JK_MISSING;
      v.kind[vn] = kind_of(c);
      v.off[vn] = i;
      v.esc[vn] = 0;
    }
    if (c == '{' || c == '[') {
      bool arr = c == '[';
      if (depth < 64) {
        if (arr) stk |= 1ull << depth;
        else stk &= ~(1ull << depth);
      } else {
        if (!deep) return LS_DEEP;
        uint64_t b = depth - 64;
        if (b >= deep->cap_levels) return LS_DEEP_FULL;
        uint32_t m = 1u << (b & 31);
        if (arr) deep->words[b >> 5] |= m;
        else deep->words[b >> 5] &= ~m;
      }
      if (depth < kMaxDepthFast) {
        node_at[depth] = vn;
        arr_idx[depth] = 0;
      }
      pending = arr ? index_child(P, vn, 0) : kNoNode;
      depth++;
      i++;
      expect = arr ? EX_VALUE_OR_CLOSE : EX_KEY_OR_CLOSE;
      continue;
    }
    uint32_t vend;
    if (c == '"') {
      bool esc;
      long long e = scan_string_bytes(line, n, i, esc);
      if (e < 0) return LS_INVALID;
      vend = (uint32_t)e + 1;
      if (vn != kNoNode) v.esc[vn] = esc;
    } else {
      uint32_t j = i + 1;
#pragma unroll 1
      while (j < n && !ends_atom(line[j])) j++;
      if (!valid_atom(line + i, j - i)) return LS_INVALID;
      vend = j;
    }
    if (vn != kNoNode) v.len[vn] = vend - i;
    i = vend;
    expect = depth == 0 ? EX_END : EX_COMMA_OR_CLOSE;
  }
  return expect == EX_END ? LS_OK : LS_INVALID;
}

// ---------------------------------------------------------------------------
// The window walker: the same semantics as walk_line for a line staged in a
// shared-memory window, where the line's own newline (or one stored after
// the data end) terminates every scan, so no step needs a bounds check.
// ---------------------------------------------------------------------------

namespace detail {

// JSON whitespace inside a line ('\n' ends the line).
__device__ __forceinline__ bool is_ws3(uint32_t c) { return c == ' ' || c == '\t' || c == '\r'; }

__device__ __forceinline__ uint32_t skip_ws3(const uint8_t *w, uint32_t i) {
#pragma unroll 1
  while (is_ws3(w[i])) i++;
  return i;
}

// Index of the lowest set bit of a nonzero word.
__device__ __forceinline__ uint32_t low_bit64(unsigned long long x) {
  const uint32_t lo = (uint32_t)x;
  return lo ? (uint32_t)__ffs(lo) - 1u : 31u + (uint32_t)__ffs((uint32_t)(x >> 32));
}

// Four bytes at any offset of a 4-byte-aligned window.
__device__ __forceinline__ uint32_t load4(const uint8_t *w, uint32_t i) {
  const uint32_t *p = (const uint32_t *)(w + (i & ~3u));
  return __funnelshift_r(p[0], p[1], (i & 3u) * 8u);
}

// Number of ASCII digits starting at w[j]; `term` receives the byte after
// them.
__device__ __forceinline__ uint32_t digit_run(const uint8_t *w, uint32_t j, uint32_t &term) {
  uint32_t n = 0;
#pragma unroll 1
  for (;;) {
    uint32_t x = load4(w, j + n);
    // flags the bytes that are no digit: x ^ '0' is at most 9 for a digit
    const uint32_t nd = ((((x ^ 0x30303030u) & 0x7F7F7F7Fu) + 0x76767676u) | x) & 0x80808080u;
    if (nd) {
      const uint32_t sh = (uint32_t)__ffs(nd) - 8u;
      term = (x >> sh) & 0xFFu;
      return n + (sh >> 3);
    }
    n += 4;
  }
}

// The value of a validated number too long or too odd for the window forms
// below (signs, exponents, more than eight bytes).
__device__ __noinline__ double parse_number_far(const uint8_t *p, uint32_t n, bool &is_int, long long &iv) {
  return parse_number(p, n, is_int, iv);
}

// Four decimal digit values (the first digit in the low byte) as a number:
// pairs by one multiply by 10, their sum by one multiply by 100.
__device__ __forceinline__ uint32_t four_digits(uint32_t y) {
  const uint32_t t = (y * 10u + (y >> 8)) & 0x00FF00FFu;
  return (t * 100u + (t >> 16)) & 0xFFFFu;
}

// parse_number for the n bytes at w[o, o + n) of a window (the 12 bytes from
// o on readable): up to eight bytes of digits, with one '.' or none, take a
// fixed number of steps for every lane, instead of one step a digit.
__device__ __forceinline__ double parse_number_win(const uint8_t *w, uint32_t o, uint32_t n, bool &is_int,
                                                   long long &iv) {
  if (n <= 8) {
    // the bytes xor '0' in the top n bytes of y, first byte lowest: zeros
    // (the digit 0) before the first
    const uint32_t x0 = load4(w, o) ^ 0x30303030u, x1 = load4(w, o + 4) ^ 0x30303030u;
    unsigned long long y = ((unsigned long long)x1 << 32 | x0) << (64u - 8u * n);
    const unsigned long long k7 = 0x7F7F7F7F7F7F7F7Full, k8 = 0x8080808080808080ull;
    unsigned long long odd = (((y & k7) + 0x7676767676767676ull) | y) & k8;  // bytes that are no digit
    uint32_t frac = 0;
    if (odd && !(odd & (odd - 1))) {  // one of them: a '.' is taken out
      const uint32_t at = low_bit64(odd) - 7u;  // its lowest bit
      if (((y >> at) & 0xFFu) == ('.' ^ '0')) {
        frac = 7u - (at >> 3);
        const unsigned long long low = y & ((1ull << at) - 1ull);
        y = (y & ~((2ull << (at + 7u)) - 1ull)) | low << 8;
        odd = 0;
      }
    }
    if (!odd) {
      const uint32_t v = four_digits((uint32_t)y) * 10000u + four_digits((uint32_t)(y >> 32));
      is_int = !frac;
      iv = (long long)v;
      // a fraction has at most seven digits before and after the '.': one
      // correctly rounded division by an exact power of ten
      return frac ? (double)v / exact_pow10((int)frac) : (double)v;
    }
  }
  return parse_number_far(w + o, n, is_int, iv);
}

// One of " \ / b f n r t: a bit per letter, the letters' columns 0x20-0x3F,
// 0x40-0x5F and 0x60-0x7F picked by their high bits.
__device__ __forceinline__ bool simple_escape(uint32_t e) {
  const uint32_t row = e >> 5;
  const uint32_t set = row == 1 ? (1u << ('"' & 31) | 1u << ('/' & 31))
                       : row == 2 ? 1u << ('\\' & 31)
                       : row == 3 ? (1u << ('b' & 31) | 1u << ('f' & 31) | 1u << ('n' & 31) | 1u << ('r' & 31) |
                                     1u << ('t' & 31))
                                  : 0u;
  return (set >> (e & 31u)) & 1u;
}

// Closing quote of the string opened at w[i], or 0 when the string is
// malformed (a bad escape, a raw control byte) or reaches the newline.
// `esc` reports whether the body holds a backslash.  `sm` has one bit per
// window byte that is '"', '\\' or below 0x20 (the stage-1 special mask), so
// the scan jumps from one such byte to the next: ordinary bytes are never
// looked at.  The line's own newline is such a byte, so no search passes
// it: every escape that moves past a byte has checked that byte first.
__device__ __forceinline__ uint32_t mask_string(const uint8_t *w, const uint32_t *sm, uint32_t i,
                                                bool &esc) {
  uint32_t p = i + 1;
  esc = false;
#pragma unroll 1
  for (;;) {
    uint32_t k = p >> 5;
    uint32_t m = sm[k] & (0xFFFFFFFFu << (p & 31u));
#pragma unroll 1
    while (!m) m = sm[++k];
    p = (k << 5) + (uint32_t)__ffs(m) - 1u;
    const uint32_t c = w[p];
    if (c == '"') return p;
    if (c != '\\') return 0;  // a byte below 0x20
    esc = true;
    const uint32_t e = w[p + 1];
    if (e == 'u') {
      if (hex_val(w[p + 2]) < 0 || hex_val(w[p + 3]) < 0 || hex_val(w[p + 4]) < 0 ||
          hex_val(w[p + 5]) < 0)
        return 0;
      p += 6;
    } else {
      if (!simple_escape(e)) return 0;
      p += 2;
    }
  }
}

// End (exclusive) of the number starting at w[i] == c, or 0 when it is
// malformed: -?(0|[1-9][0-9]*)(\.[0-9]+)?([eE][+-]?[0-9]+)?  (json.rs:370-410).
// The byte after it is checked by the caller.
__device__ __forceinline__ uint32_t win_number(const uint8_t *w, uint32_t i, uint32_t c) {
  uint32_t j = i;
  if (c == '-') c = w[++j];
  if (c - '0' >= 10u) return 0;
  uint32_t t;
  uint32_t d = digit_run(w, j, t);
  if (c == '0' && d > 1) return 0;
  j += d;
  if (t == '.') {
    d = digit_run(w, j + 1, t);
    if (!d) return 0;
    j += 1 + d;
  }
  if ((t | 0x20u) == 'e') {
    uint32_t sgn = w[++j];
    if (sgn == '+' || sgn == '-') j++;
    d = digit_run(w, j, t);
    if (!d) return 0;
    j += d;
  }
  return j;
}

// End (exclusive) of the number or literal starting at w[i] == c, or 0 when
// it is malformed.
__device__ __forceinline__ uint32_t win_atom(const uint8_t *w, uint32_t i, uint32_t c) {
  if (c <= '9') return win_number(w, i, c);
  if (c == 't') return load4(w, i) == 0x65757274u ? i + 4 : 0;      // "true"
  if (c == 'n') return load4(w, i) == 0x6C6C756Eu ? i + 4 : 0;      // "null"
  if (c == 'f') return load4(w, i + 1) == 0x65736C61u ? i + 5 : 0;  // "alse"
  return 0;
}

// match_key for a key body at w[off, off + len) of a window: keys of up to
// 8 bytes compare as two words.
__device__ __forceinline__ uint8_t match_key_win(const DevPlan &P, uint8_t node, const uint8_t *w,
                                                 uint32_t off, uint32_t len, bool esc) {
  if (esc) return match_key(P, node, w + off, len, esc);
  const uint32_t w0 = load4(w, off), w1 = load4(w, off + 4);
  const uint32_t m0 = len >= 4 ? 0xFFFFFFFFu : (1u << (8 * len)) - 1u;
  const uint32_t m1 = len >= 8 ? 0xFFFFFFFFu : len > 4 ? (1u << (8 * (len - 4))) - 1u : 0u;
#pragma unroll 1
  for (uint8_t c = P.nodes[node].first_child; c != kNoNode; c = P.nodes[c].next_sibling) {
    const PlanNode &nd = P.nodes[c];
    if (nd.is_index || nd.key_len != len) continue;
    if ((w0 & m0) != nd.key_w[0] || (w1 & m1) != nd.key_w[1]) continue;
    if (len <= 8) return c;
    const uint8_t *k = P.blob + nd.key_off;
    uint32_t t = 8;
#pragma unroll 1
    while (t < len && w[off + t] == k[t]) t++;
    if (t >= len) return c;
  }
  return kNoNode;
}

}  // namespace detail

// Walks the line w[s, e) of a window.  w must be 4-byte aligned, w[e] must
// be '\n' and the 32 bytes after it readable; `sm` is the window's special
// mask (bit j of sm[j / 32]: byte j is '"', '\\' or below 0x20), complete at
// least up to e.  Offsets recorded in `v` are relative to s.  Lines nesting
// past 64 levels return LS_DEEP.
__device__ __noinline__ int walk_masked(const DevPlan &P, const uint8_t *w, const uint32_t *sm,
                                           uint32_t s, uint32_t e, NodeVals &v) {
  using namespace detail;
  const uint32_t n_nodes = P.n_nodes;
#pragma unroll 1
  for (uint32_t k = 0; k < n_nodes; k++) v.kind[k] = JK_MISSING;

  uint32_t i = s;
  uint32_t c = w[i];
  if (is_ws3(c)) {
    i = skip_ws3(w, i);
    c = w[i];
  }
  if (c == '\n') return LS_BLANK;
  if (c == 0x0C) {  // form feed counts toward a blank line, not toward JSON
#pragma unroll 1
    for (; i < e; i++) {
      c = w[i];
      if (!(is_ws3(c) || c == 0x0C)) return LS_INVALID;
    }
    return LS_BLANK;
  }

  uint64_t arrs = 0;  // bit d: the container open at depth d is an array
  uint32_t depth = 0;
  uint32_t cur = kNoNode, idx = 0;  // trie node and element index of the innermost container
  unsigned long long cur_lm = 0;    // key_len_mask of cur (0: no key is looked up)
  uint8_t stk_node[kMaxDepthFast];
  uint32_t stk_idx[kMaxDepthFast];
  uint32_t vn = n_nodes ? 0u : kNoNode;  // node the next value lands on
  bool want_key = false;

#pragma unroll 1
  for (;;) {
    if (want_key) {
      if (c != '"') return LS_INVALID;
      bool esc;
      const uint32_t q = mask_string(w, sm, i, esc);
      if (!q) return LS_INVALID;
      vn = kNoNode;
      if (cur_lm) {
        const uint32_t kl = q - i - 1;
        if (esc || ((cur_lm >> (kl < 63u ? kl : 63u)) & 1ull))
          vn = match_key_win(P, (uint8_t)cur, w, i + 1, kl, esc);
      }
      // ':' and the value's first byte, usually in one read
      const uint32_t la = load4(w, q + 1);
      if ((la & 0xFFu) == ':') {
        i = q + 2;
        c = (la >> 8) & 0xFFu;
      } else {
        i = skip_ws3(w, q + 1);
        if (w[i] != ':') return LS_INVALID;
        c = w[++i];
      }
      if (is_ws3(c)) {
        i = skip_ws3(w, i);
        c = w[i];
      }
    }
    // A value starts at w[i] == c.
    if (vn != kNoNode) {
#pragma unroll 1
      for (uint32_t k = vn + 1u; k < P.nodes[vn].subtree_end; k++) v.kind[k] = JK_MISSING;
      v.kind[vn] = kind_of(c);
      v.off[vn] = i - s;
      v.esc[vn] = 0;
    }
    if (c == '{' || c == '[') {
      if (depth >= kMaxDepthFast) return LS_DEEP;
      const bool arr = c == '[';
      if (arr) arrs |= 1ull << depth;
      else arrs &= ~(1ull << depth);
      stk_node[depth] = (uint8_t)cur;
      stk_idx[depth] = idx;
      depth++;
      cur = vn;
      idx = 0;
      cur_lm = (!arr && vn != kNoNode) ? P.nodes[vn].key_len_mask : 0ull;
      c = w[++i];
      if (is_ws3(c)) {
        i = skip_ws3(w, i);
        c = w[i];
      }
      if (c != (arr ? (uint32_t)']' : (uint32_t)'}')) {
        want_key = !arr;
        vn = arr ? index_child(P, (uint8_t)cur, 0) : kNoNode;
        continue;
      }
      // an empty container: its close is taken below
    } else {
      uint32_t j;
      if (c == '"') {
        bool esc;
        j = mask_string(w, sm, i, esc);
        if (!j) return LS_INVALID;
        j++;
        if (vn != kNoNode) v.esc[vn] = esc;
      } else {
        j = win_atom(w, i, c);
        if (!j) return LS_INVALID;
      }
      if (vn != kNoNode) v.len[vn] = j - i;
      i = j;
    }
    // After a value: commas and closing brackets, with the next bytes read
    // four at a time.
    uint32_t la = load4(w, i);
#pragma unroll 1
    for (;;) {
      c = la & 0xFFu;
      if (is_ws3(c)) {
        i = skip_ws3(w, i);
        la = load4(w, i);
        c = la & 0xFFu;
      }
      if (depth == 0) return c == '\n' ? LS_OK : LS_INVALID;
      const bool arr = (arrs >> (depth - 1)) & 1;
      if (c == ',') {
        i++;
        c = (la >> 8) & 0xFFu;
        if (is_ws3(c)) {
          i = skip_ws3(w, i);
          c = w[i];
        }
        if (arr) {
          idx++;
          vn = index_child(P, (uint8_t)cur, idx);
        }
        want_key = !arr;
        break;
      }
      if (c != (arr ? (uint32_t)']' : (uint32_t)'}')) return LS_INVALID;
      if (cur != kNoNode) v.len[cur] = i + 1 - s - v.off[cur];
      depth--;
      cur = stk_node[depth];
      idx = stk_idx[depth];
      const bool parent_obj = depth > 0 && !((arrs >> (depth - 1)) & 1);
      cur_lm = (parent_obj && cur != kNoNode) ? P.nodes[cur].key_len_mask : 0ull;
      i++;
      la = load4(w, i);
    }
  }
}

namespace detail {

// Four hex digits at w[i..i+3].
__device__ __forceinline__ bool hex4_at(const uint8_t *w, uint32_t i) {
  return hex_val(w[i]) >= 0 && hex_val(w[i + 1]) >= 0 && hex_val(w[i + 2]) >= 0 && hex_val(w[i + 3]) >= 0;
}

// Position of the first special byte at or after p (a set bit of the window's
// special mask).  The line's newline is special, so no search from within a
// line passes it.
__device__ __forceinline__ uint32_t next_special(const uint32_t *sm, uint32_t p) {
  for (;;) {
    const uint32_t k = p >> 5, m = __funnelshift_r(sm[k], sm[k + 1], p & 31u);
    if (m) return p + (uint32_t)__ffs(m) - 1u;
    p += 32;
  }
}

}  // namespace detail

// The lanes of a warp meet here; whether any of them says so.
__device__ __forceinline__ void warp_meet() {
#ifdef __CUDA_ARCH__
  __syncwarp();
#endif
}
__device__ __forceinline__ bool warp_any(bool x) {
#ifdef __CUDA_ARCH__
  return __any_sync(0xffffffffu, x);
#else
  return x;
#endif
}

// The fast path of the window walk, for the common shape of a log line: one
// object whose members are separated by single ',' and ':' with no
// whitespace, keys without escapes, and values that are scalars or objects
// of the same shape, at most 8 deep (no arrays).  It steps from special byte
// to special byte: a key is its two quotes, a string value its quotes and
// escapes, and only the bytes right after them are read ('"' ':' value, ','
// or '}').  Lines of that shape get exactly walk_masked's verdict and node
// values; a line that breaks off from it where nothing valid goes on is
// LS_INVALID without the general walk; for any other line (whitespace, arrays,
// empty objects, escaped keys, deeper nesting) it returns LS_FALLBACK and
// records nothing that walk_masked does not overwrite.  (One line left to
// walk_masked costs its warp a walk of its own, so malformed lines are worth
// deciding here.)  Same window contract as walk_masked.
//
// Each lane walks its own line and leaves as soon as its verdict is known.  What
// bounds it is instructions.  (Taking one member a turn with the warp together,
// meeting after its key and after its value, cost a quarter more of them on
// lines of one member order: scan of 192 MB of lines of 24 members, too long
// for a template, 368 us that way and 275 so; of two interleaved shapes 286 and
// 262; 256 MB of members in any order, 2% of the lines malformed, 883 and 882.)
__device__ __noinline__ int walk_objects(const DevPlan &P, const uint8_t *w, const uint32_t *sm, uint32_t s,
                                         uint32_t e, NodeVals &v) {
  using namespace detail;
  if (w[s] != '{') return LS_FALLBACK;
  const uint32_t n_nodes = P.n_nodes;
#pragma unroll 1
  for (uint32_t k = 0; k < n_nodes; k += 4) *(uint32_t *)(v.kind + k) = 0;  // JK_MISSING, four nodes a store
  unsigned long long seen = 1;  // nodes a value has landed on
  uint32_t cur = n_nodes ? 0u : kNoNode;  // trie node of the innermost open object
  unsigned long long lm = 0;             // its key_len_mask (0: no key is looked up)
  if (cur != kNoNode) {
    v.kind[0] = JK_OBJ;
    v.off[0] = 0;
    v.esc[0] = 0;
    lm = P.nodes[0].key_len_mask;
  }
  unsigned long long stack = 0;  // trie nodes of the enclosing objects, 8 bits a level
  uint32_t depth = 1;
  uint32_t p = s + 1;  // where the next key's opening quote must be
  if (w[p] == '}') return LS_FALLBACK;
#pragma unroll 1
  for (;;) {
    if (w[p] != '"') return is_ws3(w[p]) ? LS_FALLBACK : LS_INVALID;
    const uint32_t q = next_special(sm, p + 1);
    const uint32_t la = load4(w, q + 1);
    if (w[q] != '"') return w[q] == '\\' ? LS_FALLBACK : LS_INVALID;
    if ((la & 0xFFu) != ':') return is_ws3(la & 0xFFu) ? LS_FALLBACK : LS_INVALID;
    const uint32_t vs = q + 2;
    const uint32_t c = (la >> 8) & 0xFFu;
    const uint32_t kl = q - p - 1;
    uint32_t vn = kNoNode;
    if ((lm >> (kl < 63u ? kl : 63u)) & 1ull) vn = match_key_win(P, (uint8_t)cur, w, p + 1, kl, false);
    if (vn != kNoNode) {
      // a key that comes again replaces what its first value held below it
      if ((seen >> vn) & 1ull)
#pragma unroll 1
        for (uint32_t x = vn + 1u; x < P.nodes[vn].subtree_end; x++) v.kind[x] = JK_MISSING;
      seen |= 1ull << vn;
      v.kind[vn] = kind_of(c);
      v.off[vn] = vs - s;
      v.esc[vn] = 0;
    }
    uint32_t ve;
    if (c == '"') {
      ve = vs + 1;
      bool esc = false;
#pragma unroll 1
      for (;;) {
        ve = next_special(sm, ve);
        const uint32_t x = w[ve];
        if (x == '"') break;
        if (x != '\\') return LS_INVALID;  // a control byte, the newline among them
        const uint32_t y = w[ve + 1];
        esc = true;
        if (!simple_escape(y) && !(y == 'u' && hex4_at(w, ve + 2))) return LS_INVALID;
        ve += 2;
      }
      ve++;
      if (esc && vn != kNoNode) v.esc[vn] = 1;
    } else if (c == '{') {
      if (depth >= 8 || w[vs + 1] == '}') return LS_FALLBACK;
      stack = (stack << 8) | cur;
      depth++;
      cur = vn;
      lm = vn != kNoNode ? P.nodes[vn].key_len_mask : 0ull;
      p = vs + 1;
      continue;
    } else {
      if (c == '[') return LS_FALLBACK;
      ve = win_atom(w, vs, c);
      if (!ve) return is_ws3(c) ? LS_FALLBACK : LS_INVALID;
    }
    if (vn != kNoNode) v.len[vn] = ve - vs;
    // after a value: ',' and the next key, or '}' closing one or more objects
    uint32_t t = w[ve];
    if (t == '}') {
#pragma unroll 1
      do {
        ve++;
        if (cur != kNoNode) v.len[cur] = ve - s - v.off[cur];
        if (--depth == 0) return ve == e ? LS_OK : is_ws3(w[ve]) ? LS_FALLBACK : LS_INVALID;
        cur = (uint32_t)(stack & 0xFFu);
        stack >>= 8;
        t = w[ve];
      } while (t == '}');
      lm = cur != kNoNode ? P.nodes[cur].key_len_mask : 0ull;
    }
    if (t != ',') return is_ws3(t) ? LS_FALLBACK : LS_INVALID;
    p = ve + 1;
  }
}

// ---------------------------------------------------------------------------
// Evaluation of a walked line.
// ---------------------------------------------------------------------------

enum SlotState : uint8_t { SS_FOUND = 0, SS_MISSING = 1, SS_TYPE_ERROR = 2 };

struct alignas(16) SlotVal {  // one 16-byte load or store
  uint32_t off;
  uint32_t len;
  uint8_t state;  // SlotState
  uint8_t kind;   // JKind (JK_MISSING when not found)
  uint8_t esc;
};

// Resolves slot `s` from the node values (json.rs:461-507).  Walking up from
// the terminal node, the shallowest failing step decides Missing vs type
// error, exactly as the top-down lookup does.
__device__ __forceinline__ SlotVal resolve_slot(const DevPlan &P, const NodeVals &v, uint32_t s) {
  SlotVal r;
  uint8_t t = P.slot_node[s];
  uint8_t st = SS_FOUND;
#pragma unroll 1
  for (uint8_t c = t; c != 0;) {
    uint8_t p = P.nodes[c].parent;
    uint8_t kp = v.kind[p];
    if (kp == JK_MISSING || kp == JK_NULL) st = SS_MISSING;
    else if (!P.nodes[c].is_index && kp != JK_OBJ) st = SS_TYPE_ERROR;
    else if (P.nodes[c].is_index && kp != JK_ARR) st = SS_TYPE_ERROR;
    c = p;
  }
  r.state = st;
  if (st == SS_FOUND && v.kind[t] != JK_MISSING) {
    r.kind = v.kind[t];
    r.esc = v.esc[t];
    r.off = v.off[t];
    r.len = v.len[t];
  } else {
    if (st == SS_FOUND) r.state = SS_MISSING;
    r.kind = JK_MISSING;
    r.esc = 0;
    r.off = 0;
    r.len = 0;
  }
  return r;
}

__device__ __forceinline__ uint32_t slot_rank(const uint8_t *line, const SlotVal &s) {
  switch (s.kind) {
    case JK_MISSING: case JK_NULL: return 0;
    case JK_BOOL: return line[s.off] == 't' ? 2 : 1;
    case JK_NUM: return 3;
    case JK_STR: return 4;
    case JK_ARR: return 5;
    default: return 6;
  }
}

// Three-way compare of a slot with a literal (json.rs:662-693).
__device__ __forceinline__ int compare_slot(const DevPlan &P, const uint8_t *line, const SlotVal &s,
                                            const PlanCmp &c) {
  uint32_t sr = slot_rank(line, s);
  if (sr != c.lit_rank) return sr < c.lit_rank ? -1 : 1;
  if (c.lit_kind == 3 /* NUM */) {
    bool is_int;
    long long iv;
    double d = parse_number(line + s.off, s.len, is_int, iv);
    if (d < c.lit_num) return -1;
    if (d > c.lit_num) return 1;
    return 0;
  }
  if (c.lit_kind == 4 /* STR */)
    return cmp_str_body(line + s.off + 1, s.len - 2, s.esc, P.blob + c.lit_off, c.lit_len);
  return 0;
}

__device__ __forceinline__ bool op_accepts(uint32_t op, int o) {
  switch (op) {
    case 0: return o == 0;
    case 1: return o != 0;
    case 2: return o < 0;
    case 3: return o <= 0;
    case 4: return o > 0;
    default: return o >= 0;
  }
}

__device__ __forceinline__ bool truthy(const uint8_t *line, const SlotVal &s) {
  if (s.kind == JK_MISSING || s.kind == JK_NULL) return false;
  return !(s.kind == JK_BOOL && line[s.off] == 'f');
}

// Evaluates the RPN condition (exec/cpu.rs:443-453; And/Or short-circuit
// has no side effects here, so a strict evaluation gives the same verdict).
__device__ __forceinline__ bool eval_filter(const DevPlan &P, const uint8_t *line,
                                            const SlotVal *slots) {
  uint64_t st = 0;  // bit stack, top at bit 0
#pragma unroll 1
  for (uint32_t k = 0; k < P.n_cond; k++) {
    const PlanCond &o = P.cond[k];
    switch (o.op) {
      case 0: {
        const PlanCmp &c = P.cmps[o.arg];
        bool r = op_accepts(c.op, compare_slot(P, line, slots[c.slot], c));
        st = (st << 1) | (r ? 1u : 0u);
        break;
      }
      case 1:
        st = (st << 1) | (truthy(line, slots[o.arg]) ? 1u : 0u);
        break;
      case 2: {
        uint64_t b = st & 1, a = (st >> 1) & 1;
        st = (st >> 2 << 1) | (a & b);
        break;
      }
      case 3: {
        uint64_t b = st & 1, a = (st >> 1) & 1;
        st = (st >> 2 << 1) | (a | b);
        break;
      }
      default:
        st ^= 1;
    }
  }
  return st & 1;
}

// compare_slot for a line at w + s of a window (its number and string reads
// stay in the window).
__device__ __forceinline__ int compare_slot_win(const DevPlan &P, const uint8_t *w, uint32_t s, const SlotVal &v,
                                                const PlanCmp &c) {
  using namespace detail;
  // the kinds from JK_NUM on are their jq ranks; null and missing rank 0
  const uint32_t sr = v.kind == JK_BOOL ? (w[s + v.off] == 't' ? 2u : 1u) : v.kind <= JK_NULL ? 0u : v.kind;
  if (sr != c.lit_rank) return sr < c.lit_rank ? -1 : 1;
  if (c.lit_kind == 3 /* NUM */) {
    bool is_int;
    long long iv;
    const double d = parse_number_win(w, s + v.off, v.len, is_int, iv);
    return d < c.lit_num ? -1 : d > c.lit_num ? 1 : 0;
  }
  if (c.lit_kind == 4 /* STR */) {
    const uint32_t o = s + v.off + 1, n = v.len - 2;
    if (c.op <= 1 && !v.esc) {  // equality: the length, then the first eight bytes
      if (n != c.lit_len) return 1;
      const uint32_t m0 = n >= 4 ? 0xFFFFFFFFu : (1u << (8 * n)) - 1u;
      const uint32_t m1 = n >= 8 ? 0xFFFFFFFFu : n > 4 ? (1u << (8 * (n - 4))) - 1u : 0u;
      if ((load4(w, o) & m0) != c.lit_w[0] || (load4(w, o + 4) & m1) != c.lit_w[1]) return 1;
      if (n <= 8) return 0;
    }
    return cmp_str_body(w + o, n, v.esc, P.blob + c.lit_off, c.lit_len);
  }
  return 0;
}

// eval_filter for a line at w + s of a window.
__device__ __forceinline__ bool eval_filter_win(const DevPlan &P, const uint8_t *w, uint32_t s, const SlotVal *slots) {
  uint64_t st = 0;  // bit stack, top at bit 0
#pragma unroll 1
  for (uint32_t k = 0; k < P.n_cond; k++) {
    const PlanCond &o = P.cond[k];
    if (o.op == 0) {
      const PlanCmp &c = P.cmps[o.arg];
      st = (st << 1) | (op_accepts(c.op, compare_slot_win(P, w, s, slots[c.slot], c)) ? 1u : 0u);
    } else if (o.op == 1) {
      st = (st << 1) | (truthy(w + s, slots[o.arg]) ? 1u : 0u);
    } else if (o.op == 2 || o.op == 3) {
      const uint64_t b = st & 1, a = (st >> 1) & 1;
      st = (st >> 2 << 1) | (o.op == 2 ? a & b : a | b);
    } else {
      st ^= 1;
    }
  }
  return st & 1;
}

// eval_filter out of line, for lines outside the window (long ones).
__device__ __noinline__ bool eval_filter_far(const DevPlan &P, const uint8_t *line, const SlotVal *slots) {
  return eval_filter(P, line, slots);
}

// The slots of a walked line: bit 0 of the result where one that the filter
// reads is a type error, bit 1 where another is.
__device__ __noinline__ uint32_t resolve_slots(const DevPlan &P, const NodeVals &v, SlotVal *slots) {
  uint32_t bad = 0;
#pragma unroll 1
  for (uint32_t k = 0; k < P.n_slots; k++) {
    slots[k] = resolve_slot(P, v, k);
    if (slots[k].state == SS_TYPE_ERROR) bad |= ((P.filter_slot_mask >> k) & 1) ? 1u : 2u;
  }
  return bad;
}

// ---------------------------------------------------------------------------
// Line templates: log lines of one source repeat the same text around their
// values, so a line is mostly a comparison.
//
// A template is the text of one valid line with its scalar values taken out:
// literal 0, value, literal 1, value, ..., last literal.  A literal holds
// everything between two values -- punctuation, keys, whitespace, opened and
// closed objects, and a string value's own quotes.  A line that consists of
// the same literals with any string body or any number, true, false or null
// at the values' places is valid JSON with the template line's structure, so
// each value's trie node and the kind of every object node are the
// template's.  Any other line is left to the walkers below it.
//
// What bounds the walk is instructions, most of them spent finding and
// checking keys and punctuation one member at a time; comparing them sixteen
// bytes at a time took the scan of 1 GB of access-log lines from 970 us
// (walk_objects on every line) to 695.
// ---------------------------------------------------------------------------

constexpr uint32_t kTmplSteps = 24;       // steps per line
constexpr uint32_t kTmplStepBytes = 16;   // literal bytes per step (a longer literal takes several)
constexpr uint32_t kTmplNodes = 32;       // trie nodes of the plan

enum TmplValue : uint32_t { TV_NONE = 0, TV_STR = 1, TV_ATOM = 2 };

constexpr uint32_t kNoSlot = 0xFF;

// One step: up to 16 literal bytes, compared as four words under a byte mask
// (always four: a flat compare has no loop, and its loads are in flight
// together), then a value or none.
struct alignas(16) Template {
  uint32_t lit[kTmplSteps][4];
  uint32_t mask[kTmplSteps][4];
  uint32_t desc[kTmplSteps];  // literal bytes (bits 0-7), TmplValue (8-15), the value's slot (16-23)
  uint32_t n_steps;
  uint32_t pad[3];
};


// Makes the template of the line w[s, e), which must be a valid one (same
// window contract as walk_masked).  False when the line has none: no object,
// arrays, duplicate wanted keys, an object as a wanted value, a scalar where
// a wanted path goes on (whose slot is missing or a type error, depending on
// the value), or too large.
__device__ __noinline__ bool build_template(const DevPlan &P, const uint8_t *w, const uint32_t *sm, uint32_t s,
                                            uint32_t e, Template *t) {
  using namespace detail;
  const uint32_t n_nodes = P.n_nodes;
  if (n_nodes > kTmplNodes) return false;
  uint8_t seen[kTmplNodes];  // kinds of the nodes met: JK_OBJ, else JK_NUM for any scalar
#pragma unroll 1
  for (uint32_t k = 0; k < n_nodes; k++) seen[k] = JK_MISSING;
  uint32_t ns = 0, lit0 = s, depth = 0;
  uint8_t stk[8];
  uint32_t vn = n_nodes ? 0u : kNoNode;  // node of the next value
  bool key = false;                     // a key (not a value) comes next
  // the steps of the literal [lit0, end) and the value after it
  auto close_literal = [&](uint32_t end, uint32_t value, uint32_t node) -> bool {
    uint32_t at = lit0, slot = kNoSlot;
#pragma unroll 1
    for (uint32_t k = 0; k < P.n_slots && node != kNoNode; k++)
      if (P.slot_node[k] == node) {
        if (slot != kNoSlot) return false;
        slot = k;
      }
    do {
      if (ns >= kTmplSteps) return false;
      const uint32_t nb = end - at < kTmplStepBytes ? end - at : kTmplStepBytes;
#pragma unroll 1
      for (uint32_t k = 0; k < 4; k++) {
        const uint32_t m = nb >= 4 * k + 4 ? 0xFFFFFFFFu : nb <= 4 * k ? 0u : 0xFFFFFFFFu >> (8 * (4 * k + 4 - nb));
        t->lit[ns][k] = load4(w, at + 4 * k) & m;
        t->mask[ns][k] = m;
      }
      at += nb;
      t->desc[ns++] = nb | (at == end ? value << 8 | slot << 16 : TV_NONE << 8 | kNoSlot << 16);
    } while (at < end);
    return true;
  };
#pragma unroll 1
  for (uint32_t i = s; i < e;) {
    const uint32_t c = w[i];
    if (is_ws3(c) || c == ':') {
      i++;
    } else if (c == '{') {
      if (depth >= 8) return false;
      if (vn != kNoNode) {
        if (seen[vn]) return false;
        seen[vn] = JK_OBJ;
#pragma unroll 1
        for (uint32_t k = 0; k < P.n_slots; k++)
          if (P.slot_node[k] == vn) return false;
      }
      stk[depth++] = (uint8_t)vn;
      key = true;
      i++;
    } else if (c == '}') {
      if (!depth) return false;
      depth--;
      i++;
    } else if (c == ',') {
      key = true;
      i++;
    } else if (c == '[' || c == ']' || !depth) {
      return false;
    } else if (key) {
      bool esc;
      const uint32_t q = mask_string(w, sm, i, esc);
      if (c != '"' || !q) return false;
      const uint32_t cur = stk[depth - 1];
      vn = kNoNode;
      if (cur != kNoNode && P.nodes[cur].has_key_children)
        vn = match_key_win(P, (uint8_t)cur, w, i + 1, q - i - 1, esc);
      key = false;
      i = q + 1;
    } else {
      if (vn != kNoNode) {
        if (seen[vn]) return false;
        seen[vn] = JK_NUM;
      }
      uint32_t end;
      if (c == '"') {
        bool esc;
        end = mask_string(w, sm, i, esc);
        if (!close_literal(i + 1, TV_STR, vn)) return false;
      } else {
        end = win_atom(w, i, c);
        if (!close_literal(i, TV_ATOM, vn)) return false;
      }
      if (!end) return false;
      lit0 = i = end;
      if (c == '"') i++;
    }
  }
  if (depth || !close_literal(e, TV_NONE, kNoNode)) return false;
  // every path runs through objects of the line up to its value, or to a
  // member that is not there
#pragma unroll 1
  for (uint32_t k = 0; k < P.n_slots; k++)
#pragma unroll 1
    for (uint32_t c = P.slot_node[k]; c != 0; c = P.nodes[c].parent) {
      const uint32_t kp = seen[P.nodes[c].parent];
      if (kp != JK_MISSING && (kp != JK_OBJ || P.nodes[c].is_index)) return false;
    }
  t->n_steps = ns;
  return true;
}

// Walks w[s, e) by the template t (same window contract as walk_masked):
// LS_OK with the slots' values (those of the template's line; the caller
// sets the others to missing), or LS_FALLBACK for a line of another shape,
// malformed ones among them.  All lanes of the warp call it together, with
// `on` where the lane has a line (the others read at the window's start):
// the steps are the same for every lane, so their loads are broadcasts, and
// the lanes meet again after every value (no lane leaves the loop alone, or
// the compiler would let the others run on apart from it).  A lane never
// steps past e, and reads at most 20 bytes from where it is.
__device__ __forceinline__ int walk_template(const Template *t, const uint8_t *w, const uint32_t *sm, uint32_t s,
                                             uint32_t e, bool on, SlotVal *slots) {
  using namespace detail;
  const uint32_t ns = t->n_steps;
  uint32_t p = on ? s : 0;
#pragma unroll 1
  for (uint32_t j = 0; j < ns; j++) {
    const uint32_t d = t->desc[j];
    {
      const uint32_t *q = (const uint32_t *)w + (p >> 2);
      const uint4 L = *(const uint4 *)t->lit[j], M = *(const uint4 *)t->mask[j];
      const uint32_t sh = (p & 3u) * 8u;
      const uint32_t a = q[0], b = q[1], c = q[2], f = q[3], g = q[4];
      const uint32_t bad = ((__funnelshift_r(a, b, sh) ^ L.x) & M.x) | ((__funnelshift_r(b, c, sh) ^ L.y) & M.y) |
                           ((__funnelshift_r(c, f, sh) ^ L.z) & M.z) | ((__funnelshift_r(f, g, sh) ^ L.w) & M.w);
      // no literal holds a newline, so one that fits ends at or before e
      on = on && !bad;
      if (on) p += d & 0xFFu;
    }
    if (!warp_any(on)) break;
    const uint32_t value = (d >> 8) & 0xFFu, slot = (d >> 16) & 0xFFu, b = p;
    bool esc = false;
    if (value == TV_STR) {
      // from special byte to special byte of the stage-1 mask, 32 bytes at
      // a time, until one that is not an escape's backslash
      bool go = on;
#pragma unroll 1
      while (go) {
        const uint32_t k = p >> 5, m = __funnelshift_r(sm[k], sm[k + 1], p & 31u);
        if (!m) {
          p += 32;
        } else {
          p += (uint32_t)__ffs(m) - 1u;
          const uint32_t c = w[p];
          go = c == '\\';
          on = go || c == '"';  // else a byte below 0x20, the newline among them
          if (go) {
            const uint32_t x = w[p + 1];
            esc = true;
            if (!simple_escape(x)) on = go = x == 'u' && hex4_at(w, p + 2);
            p += 2;
          }
        }
      }
      warp_meet();
    } else if (value == TV_ATOM) {
      if (on) {
        p = win_atom(w, b, w[b]);
        on = p != 0;
      }
      warp_meet();
    }
    if (slot != kNoSlot && on) {
      const uint32_t q = value == TV_STR ? 1u : 0u;  // a string's span includes its quotes
      SlotVal r;
      r.state = SS_FOUND;
      r.kind = q ? (uint8_t)JK_STR : kind_of(w[b]);
      r.esc = esc;
      r.off = b - q - s;
      r.len = p - b + 2 * q;
      slots[slot] = r;
    }
  }
  return on && p == e ? LS_OK : LS_FALLBACK;
}

}  // namespace wjq
