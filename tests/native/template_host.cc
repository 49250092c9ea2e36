// TEST HARNESS (CPU): the line templates of warpjq_b200/csrc/walker.cuh
// (build_template, walk_template), compiled for the host like the other
// walkers.
#include "walker_host.cc"

extern "C" {

// Every line walked by the template of line `from` (the first line at or
// after it that has one; 0-based) when it fits it, else by walk_masked.  One
// output line per input line, as wh_eval's; *hits counts the lines the
// template decided, *made is 1 when there was a template.
int th_eval(const char *query, const uint8_t *data, size_t len, size_t from, char **out, size_t *out_len,
            size_t *hits, int *made) {
  wjqh::Program prog;
  wjqh::QueryError qe;
  if (!wjqh::parse(query, prog, qe)) return 2;
  wjqh::Lowered low;
  low.build(prog, false);
  static DevPlan P;
  char err[256];
  if (build_plan(&low.prog, P, err, sizeof err) != WARPJQ_OK) return 3;
  std::vector<uint32_t> deep_words(1 << 16);
  DeepStack deep{deep_words.data(), (uint64_t)deep_words.size() * 32};
  static NodeVals nv;
  static Template T;
  std::memset(&T, 0xEE, sizeof T);
  std::vector<uint32_t> winbuf, smask;
  uint32_t s = 0;
  auto window = [&](const uint8_t *line, uint32_t n, size_t no) -> const uint8_t * {
    s = (uint32_t)(no * 7 % 48);
    const uint32_t W = (s + n + 64 + 31) / 32 * 32;
    winbuf.assign(W / 4 + 8, 0);
    uint8_t *w = (uint8_t *)winbuf.data();
    std::memcpy(w + s, line, n);
    w[s + n] = '\n';
    for (uint32_t k = 1; k < 40; k++) w[s + n + k] = "\"\\9"[k % 3];
    smask.assign(W / 32 + 1, 0);
    for (uint32_t c = 0; c < W / 32; c++) classify_chunk(winbuf.data() + 8 * c, &smask[c]);
    return w;
  };
  auto each = [&](auto &&f) {
    size_t no = 0;
    for (size_t pos = 0; pos < len; no++) {
      const uint8_t *nl = (const uint8_t *)std::memchr(data + pos, '\n', len - pos);
      const size_t end = nl ? (size_t)(nl - data) : len;
      if (!f(data + pos, (uint32_t)(end - pos), no)) return;
      pos = end + 1;
    }
  };
  bool have = false;
  each([&](const uint8_t *line, uint32_t n, size_t no) {
    if (no < from) return true;
    const uint8_t *w = window(line, n, no);
    if (walk_masked(P, w, smask.data(), s, s + n, nv) == LS_OK)
      have = build_template(P, w, smask.data(), s, s + n, &T);
    return !have;
  });
  *made = have;
  *hits = 0;
  std::string o;
  each([&](const uint8_t *src, uint32_t n, size_t no) {
    const uint8_t *w = window(src, n, no + 3), *line = w + s;
    SlotVal slots[kMaxSlots];
    for (SlotVal &x : slots) x = SlotVal{0, 0, SS_MISSING, JK_MISSING, 0};
    int st = have ? walk_template(&T, w, smask.data(), s, s + n, true, slots) : LS_FALLBACK;
    const bool hit = st != LS_FALLBACK;
    if (hit) ++*hits;
    else st = walk_masked(P, w, smask.data(), s, s + n, nv);
    if (st == LS_DEEP) st = walk_line(P, line, n, nv, &deep);
    if (st != LS_OK) {
      o += st == LS_BLANK ? "blank\n" : "invalid\n";
      return true;
    }
    const uint32_t bad = hit ? 0u : resolve_slots(P, nv, slots);
    if (bad & 1u) {
      o += "type\n";
    } else if (P.has_filter && !eval_filter_win(P, w, s, slots)) {
      o += "filtered\n";
    } else if (bad) {
      o += "type\n";
    } else {
      o += "selected";
      for (uint32_t k = 0; k < P.n_slots; k++) {
        o += "\t" + std::to_string(slots[k].kind) + ":";
        if (slots[k].kind != JK_MISSING) o.append((const char *)line + slots[k].off, slots[k].len);
        if (slots[k].kind == JK_NUM) {
          bool is_int;
          long long iv;
          char b[64];
          std::snprintf(b, sizeof b, "=%a", detail::parse_number_win(w, s + slots[k].off, slots[k].len, is_int, iv));
          o += b;
        }
      }
      o += "\n";
    }
    return true;
  });
  *out = (char *)std::malloc(o.size() + 1);
  std::memcpy(*out, o.data(), o.size());
  *out_len = o.size();
  return 0;
}

}  // extern "C"
