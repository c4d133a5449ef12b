// sr_share.cpp — equal expressions, constant subtrees and frequent subtrees of
// a population (sr_share.hpp).
//
// Three passes.  (1) On the workers: a structural hash and size per token,
// from the right, and a count per distinct subtree in one open-addressed table
// (keys are claimed with a compare-and-swap; a hash is only ever a hint, every
// use compares the tokens).  (2) On the caller: the rows, chosen greedily by
// the evaluations they save, most first; choosing one takes its occurrences
// away from the subtrees inside it and its cost from the subtrees around it.
// (3) While compiling: each expression's tokens are marked, outermost first.
#include "sr_share.hpp"

#include <algorithm>
#include <cstring>
#include <new>

#include "sr_internal.hpp"
#include "sr_program.hpp"

namespace sr {

namespace {

inline uint64_t mix(uint64_t z) {
  z *= 0x9E3779B97F4A7C15ull;
  z ^= z >> 32;
  z *= 0xD6E8FEB86659FD93ull;
  return z ^ (z >> 29);
}

inline uint32_t bits_of(double v) {
  const float f = static_cast<float>(v);
  uint32_t u;
  std::memcpy(&u, &f, sizeof u);
  return u;
}

inline int64_t index_of(double v) {
  return v > -2147483648.0 && v < 2147483648.0 ? static_cast<int64_t>(v) : -1;
}

// Device cost of one operator instruction in warp instructions per 8
// datapoints a lane: its arithmetic and about 25 of dispatch.
inline float token_cost(int t) { return 25.0f + 6.0f * op_cost(t); }
constexpr float kRowLoadCost = 8.0f;  // reading a row instead

constexpr uint64_t kRootSalt = 0x9E3779B97F4A7C15ull;

}  // namespace

bool mark_constant_subtrees(const int32_t *tok, int len, int32_t *hints) {
  // size: tokens of the subtree at each position, negative when constant.
  int16_t size[SR_MAX_TOKENS];
  if (len > SR_MAX_TOKENS) return false;
  int depth = 0;
  for (int i = len - 1; i >= 0; --i) {
    const int32_t t = tok[i];
    if (t == SR_TOK_CONST || t == SR_TOK_VAR) {
      ++depth;
      size[i] = t == SR_TOK_CONST ? -1 : 1;
      continue;
    }
    const bool binary = is_binary_token(t);
    if (binary ? --depth < 1 : !is_unary_token(t) || depth < 1) return false;
    const int16_t a = size[i + 1];
    int n = 1 + (a < 0 ? -a : a);
    bool constant = a < 0;
    if (binary) {
      const int16_t b = size[i + n];
      n += b < 0 ? -b : b;
      constant = constant && b < 0;
    }
    size[i] = static_cast<int16_t>(constant ? -n : n);
  }
  if (depth != 1) return false;
  bool any = false;
  for (int i = 0; i < len;) {
    hints[i] = -1;
    const int n = -size[i];
    if (n < 2 || n > kMaxSharedTokens) {
      ++i;
      continue;
    }
    any = true;
    hints[i] = kHintFold;
    for (int k = 1; k < n; ++k) hints[i + k] = -2;
    i += n;
  }
  return any;
}

void merge_hints(const int32_t *hints, int len, int32_t *marks) {
  for (int i = 0; i < len;) {
    if (marks[i] == kHintFold) {  // over whatever is cached inside
      for (++i; i < len && marks[i] == -2; ++i) {
      }
    } else if (hints[i] >= 0) {   // over whatever would be folded inside
      marks[i] = hints[i];
      for (++i; i < len && hints[i] == -2; ++i) marks[i] = -2;
    } else {
      ++i;
    }
  }
}

// A worker's own counts of the subtrees it met last: the frequent ones (sin x0)
// would otherwise have every worker add to the same few words.
struct Sharing::Local {
  static constexpr int kSlots = 256;
  uint64_t key[kSlots] = {};
  uint32_t count[kSlots] = {};
  uint32_t at[kSlots] = {};
  std::vector<uint32_t> frequent;  // table entries that reached min_count_
};

void Sharing::flush(Local &local, int s) {
  if (local.count[s] == 0) return;
  Entry *e = insert(local.key[s]);
  const uint32_t before = e->count.fetch_add(local.count[s], std::memory_order_relaxed);
  if (before == 0) e->at.store(local.at[s], std::memory_order_relaxed);
  if (before < min_count_ && before + local.count[s] >= min_count_)
    local.frequent.push_back(static_cast<uint32_t>(e - table_.get()));
  local.count[s] = 0;
}

Sharing::Entry *Sharing::insert(uint64_t key) {
  size_t i = key & mask_;
  for (;;) {
    uint64_t k = table_[i].key.load(std::memory_order_relaxed);
    if (k == key) return &table_[i];
    if (k == 0 &&
        (table_[i].key.compare_exchange_strong(k, key, std::memory_order_relaxed) || k == key))
      return &table_[i];
    i = (i + 1) & mask_;
  }
}

const Sharing::Entry *Sharing::lookup(uint64_t key) const {
  for (size_t i = key & mask_;; i = (i + 1) & mask_) {
    const uint64_t k = table_[i].key.load(std::memory_order_relaxed);
    if (k == key) return &table_[i];
    if (k == 0) return nullptr;
  }
}

// Same operators, same constants (as floats, bit for bit), same variables.
bool Sharing::equal_runs(int64_t a, int64_t b, int32_t n) const {
  for (int32_t i = 0; i < n; ++i) {
    const int32_t t = tok_[a + i];
    if (t != tok_[b + i]) return false;
    if (t == SR_TOK_CONST && bits_of(val_[a + i]) != bits_of(val_[b + i])) return false;
    if (t == SR_TOK_VAR && index_of(val_[a + i]) != index_of(val_[b + i])) return false;
  }
  return true;
}

bool Sharing::hash_expression(int x, Local &local) {
  const int64_t o = off_[x];
  const int len = static_cast<int>(off_[x + 1] - o);
  int depth = 0;  // values to the right: an operator finds its operands there
  for (int i = len - 1; i >= 0; --i) {
    const int64_t p = o + i;
    const int32_t t = tok_[p];
    if (t == SR_TOK_CONST || t == SR_TOK_VAR) {
      ++depth;
    } else if (is_binary_token(t)) {
      if (--depth < 1) return false;
    } else if (!is_unary_token(t) || depth < 1) {
      return false;
    }
    if (t == SR_TOK_CONST) {
      hash_[static_cast<size_t>(p)] = mix(0x100000000ull | bits_of(val_[p]));
      size_[static_cast<size_t>(p)] = -1;
      continue;
    }
    if (t == SR_TOK_VAR) {
      hash_[static_cast<size_t>(p)] = mix(0x200000000ull ^ static_cast<uint64_t>(index_of(val_[p])));
      size_[static_cast<size_t>(p)] = 1;
      continue;
    }
    const int16_t sl = size_[static_cast<size_t>(p + 1)];
    const int nl = sl < 0 ? -sl : sl;
    uint64_t h = hash_[static_cast<size_t>(p + 1)] + 0x632BE59BD9B4E019ull * static_cast<uint64_t>(t);
    int n = 1 + nl;
    bool constant = sl < 0;
    if (is_binary_token(t)) {
      const int16_t sr = size_[static_cast<size_t>(p + 1 + nl)];
      n += sr < 0 ? -sr : sr;
      constant = constant && sr < 0;
      const uint64_t r = hash_[static_cast<size_t>(p + 1 + nl)];
      h = mix(h) ^ ((r << 23) | (r >> 41));
    }
    h = mix(h) | 1;  // never 0, the table's empty key
    hash_[static_cast<size_t>(p)] = h;
    size_[static_cast<size_t>(p)] = static_cast<int16_t>(constant ? -n : n);
    if (constant || n > kMaxSharedTokens) continue;
    const int slot = static_cast<int>((h >> 1) & (Local::kSlots - 1));
    if (local.key[slot] != h) {
      flush(local, slot);
      local.key[slot] = h;
      local.at[slot] = static_cast<uint32_t>(p);
    }
    ++local.count[slot];
  }
  // The expression itself: the lowest index of each distinct one.
  Entry *e = insert(mix(hash_[static_cast<size_t>(o)] ^ kRootSalt) | 1);
  uint32_t cur = e->at.load(std::memory_order_relaxed);
  const uint32_t mine = static_cast<uint32_t>(x) + 1;  // 0: not set yet
  while ((cur == 0 || mine < cur) &&
         !e->at.compare_exchange_weak(cur, mine, std::memory_order_relaxed)) {
  }
  return depth == 1;
}

void Sharing::choose(std::vector<uint32_t> &frequent, int max_rows) {
  drop_rows();
  struct Candidate {
    uint64_t key;
    int64_t at;
    int32_t n;
    float occ, cost;
    bool taken;
  };
  std::vector<Candidate> cs;
  cs.reserve(frequent.size());
  for (const uint32_t i : frequent) {
    const Entry &e = table_[i];
    Candidate c{};
    c.key = e.key.load(std::memory_order_relaxed);
    c.at = e.at.load(std::memory_order_relaxed);
    if (c.at >= n_tokens_ || hash_[static_cast<size_t>(c.at)] != c.key) continue;
    c.n = size_[static_cast<size_t>(c.at)];
    if (c.n < 2) continue;
    c.occ = static_cast<float>(e.count.load(std::memory_order_relaxed));
    for (int32_t q = 0; q < c.n;) {
      const int16_t s = size_[static_cast<size_t>(c.at + q)];
      if (s < -1) {
        q += -s;  // folded
        continue;
      }
      if (tok_[c.at + q] > 0) c.cost += token_cost(tok_[c.at + q]);
      ++q;
    }
    cs.push_back(c);
  }
  // Most saving first; the hash breaks ties, so the choice does not depend on
  // which worker met a subtree first.
  const auto gain = [](const Candidate &c) { return (c.occ - 1.0f) * (c.cost - kRowLoadCost); };
  const auto before = [&](const Candidate &a, const Candidate &b) {
    const float ga = gain(a), gb = gain(b);
    return ga != gb ? ga > gb : a.key < b.key;
  };
  // The rows come from the first of them: choosing one only lowers the others.
  constexpr size_t kCandidates = 128;
  if (cs.size() > kCandidates) {
    std::nth_element(cs.begin(), cs.begin() + kCandidates, cs.end(), before);
    cs.resize(kCandidates);
  }
  // Candidates by hash, open-addressed.
  int16_t of_key[512];
  std::memset(of_key, 0xff, sizeof of_key);
  for (size_t i = 0; i < cs.size(); ++i) {
    size_t k = cs[i].key & 511;
    while (of_key[k] >= 0) k = (k + 1) & 511;
    of_key[k] = static_cast<int16_t>(i);
  }
  const auto find_candidate = [&](uint64_t key) -> Candidate * {
    for (size_t k = key & 511; of_key[k] >= 0; k = (k + 1) & 511)
      if (cs[static_cast<size_t>(of_key[k])].key == key) return &cs[static_cast<size_t>(of_key[k])];
    return nullptr;
  };
  while (static_cast<int>(rows_.size()) < max_rows) {
    Candidate *best = nullptr;
    for (auto &c : cs)
      if (!c.taken && (!best || before(c, *best))) best = &c;
    // A row costs its own evaluation and a copy per group of expressions: it
    // has to save several of them.
    if (!best || best->occ < static_cast<float>(min_count_) || best->cost <= 2.0f * kRowLoadCost)
      break;
    best->taken = true;
    const int r = static_cast<int>(rows_.size());
    rows_.push_back(Row{best->at, best->n, static_cast<int32_t>(best->occ)});
    enter_row(best->key, r);
    const auto is_row = [&](uint64_t key) {
      for (size_t i = key & 255; row_key_[i] != 0; i = (i + 1) & 255)
        if (row_key_[i] == key) return true;
      return false;
    };
    // Inside it: those occurrences go.
    for (int32_t q = 1; q < best->n;) {
      const size_t p = static_cast<size_t>(best->at + q);
      const int16_t s = size_[p];
      if (s < 0 || tok_[p] <= 0) {
        q += s < 0 ? -s : 1;
        continue;
      }
      if (is_row(hash_[p])) {
        q += s;
        continue;
      }
      if (Candidate *c = find_candidate(hash_[p])) c->occ -= best->occ;
      ++q;
    }
    // Around it: it is read, not evaluated.
    const float saved = best->cost - kRowLoadCost;
    for (auto &c : cs) {
      if (c.taken || c.n <= best->n) continue;
      for (int32_t q = 1; q + best->n <= c.n; ++q)
        if (hash_[static_cast<size_t>(c.at + q)] == best->key) c.cost -= saved;
    }
  }
}

void Sharing::enter_row(uint64_t key, int r) {
  size_t slot = key & 255;
  while (row_key_[slot] != 0) slot = (slot + 1) & 255;
  row_key_[slot] = key;
  row_of_[slot] = static_cast<int16_t>(r);
  max_row_size_ = std::max(max_row_size_, rows_[static_cast<size_t>(r)].size);
}

void Sharing::keep_rows(int n) {
  if (static_cast<int>(rows_.size()) > n) rows_.resize(static_cast<size_t>(n));
  max_row_size_ = 0;
  std::memset(row_key_, 0, sizeof row_key_);
  for (size_t r = 0; r < rows_.size(); ++r)
    enter_row(hash_[static_cast<size_t>(rows_[r].tok)], static_cast<int>(r));
}

bool Sharing::find(int E, const int32_t *tok, const double *val, const int64_t *off, int max_rows,
                   WorkerPool &pool, int threads) {
  // Sharing is an option: a population whose hashes and table (up to about 50
  // bytes a token) do not fit host memory is evaluated without it.
  try {
    return search(E, tok, val, off, max_rows, pool, threads);
  } catch (const std::bad_alloc &) {
    drop_rows();
    std::vector<uint64_t>().swap(hash_);
    std::vector<int16_t>().swap(size_);
    table_.reset();
    cap_ = 0;
    return false;
  }
}

bool Sharing::search(int E, const int32_t *tok, const double *val, const int64_t *off,
                     int max_rows, WorkerPool &pool, int threads) {
  tok_ = tok;
  val_ = val;
  off_ = off;
  drop_rows();
  const size_t T = static_cast<size_t>(off[E]);
  if (T >= (1ull << 31)) return false;
  n_tokens_ = static_cast<int64_t>(T);
  if (hash_.size() < T) hash_.resize(T);
  if (size_.size() < T) size_.resize(T);
  // Room for every operator and expression, were they all different.
  size_t n_ops = 0;
  for (size_t i = 0; i < T; ++i) n_ops += tok[i] > 0 ? 1 : 0;
  size_t cap = 1024;
  while (cap * 7 < (n_ops + static_cast<size_t>(E)) * 8) cap *= 2;
  if (cap > cap_) {
    table_.reset();
    cap_ = 0;
    table_.reset(new Entry[cap]);
    cap_ = cap;
  }
  mask_ = cap - 1;
  // Rows serve every group of expressions; one used by few is no gain.
  min_count_ = static_cast<uint32_t>(std::max(4, E / 512));
  const int chunks = static_cast<int>(
      std::max<int64_t>(1, std::min<int64_t>({threads, E, static_cast<int64_t>(T) / 2500})));
  Entry *table = table_.get();
  const int zero_chunks = cap < 65536 ? 1 : chunks;  // 1 MB
  pool.run(zero_chunks, threads, [&](int c) {
    const size_t a = cap * static_cast<size_t>(c) / zero_chunks, b = cap * (static_cast<size_t>(c) + 1) / zero_chunks;
    std::memset(static_cast<void *>(table + a), 0, (b - a) * sizeof(Entry));
  });
  std::vector<Local> locals(static_cast<size_t>(chunks));
  std::vector<char> bad(static_cast<size_t>(chunks), 0);
  pool.run(chunks, threads, [&](int c) {
    const int x0 = static_cast<int>(static_cast<int64_t>(E) * c / chunks);
    const int x1 = static_cast<int>(static_cast<int64_t>(E) * (c + 1) / chunks);
    Local &local = locals[static_cast<size_t>(c)];
    for (int x = x0; x < x1; ++x)
      if (!hash_expression(x, local)) {
        bad[static_cast<size_t>(c)] = 1;
        return;
      }
    for (int k = 0; k < Local::kSlots; ++k) flush(local, k);
  });
  if (std::find(bad.begin(), bad.end(), 1) != bad.end()) return false;
  std::vector<uint32_t> all;
  for (const auto &l : locals) all.insert(all.end(), l.frequent.begin(), l.frequent.end());
  choose(all, max_rows);
  return true;
}

bool Sharing::mark(int x, int32_t *hints) const {
  const int64_t o = off_[x];
  const int len = static_cast<int>(off_[x + 1] - o);
  bool any = false;
  for (int i = 0; i < len;) {
    const size_t p = static_cast<size_t>(o + i);
    hints[i] = -1;
    const int16_t s = size_[p];
    int32_t mark = -1;
    int n = s < 0 ? -s : s;
    if (tok_[p] > 0 && n <= kMaxSharedTokens) {
      if (s < 0) {
        mark = kHintFold;
      } else if (n <= max_row_size_) {
        const uint64_t key = hash_[p];
        for (size_t k = key & 255; row_key_[k] != 0; k = (k + 1) & 255)
          if (row_key_[k] == key) {
            const Row &r = rows_[static_cast<size_t>(row_of_[k])];
            if (r.size == n && equal_runs(r.tok, o + i, n)) mark = kHintRow0 - row_of_[k];
            break;
          }
      }
    }
    if (mark == -1) {
      ++i;
      continue;
    }
    any = true;
    hints[i] = mark;
    for (int k = 1; k < n; ++k) hints[i + k] = -2;
    i += n;
  }
  return any;
}

void Sharing::mark_row(const Row &r, int32_t *hints) const {
  for (int i = 0; i < r.size;) {
    const size_t p = static_cast<size_t>(r.tok + i);
    const int16_t s = size_[p];
    hints[i] = -1;
    if (s < -1) {
      hints[i] = kHintFold;
      for (int k = 1; k < -s; ++k) hints[i + k] = -2;
      i += -s;
    } else {
      ++i;
    }
  }
}

int Sharing::rep(int x) const {
  const int64_t o = off_[x];
  const Entry *e = lookup(mix(hash_[static_cast<size_t>(o)] ^ kRootSalt) | 1);
  if (!e) return x;
  const int first = static_cast<int>(e->at.load(std::memory_order_relaxed)) - 1;
  const int64_t n = off_[x + 1] - o;
  if (first < 0 || first >= x || off_[first + 1] - off_[first] != n) return x;
  return equal_runs(off_[first], o, static_cast<int32_t>(n)) ? first : x;
}

}  // namespace sr
