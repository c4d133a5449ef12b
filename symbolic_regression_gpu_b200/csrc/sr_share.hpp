// sr_share.hpp — shared work of a population: equal expressions, constant
// subtrees and frequent subtrees, found once per prepared population.
//
//   * equal expressions are evaluated once (rep: the first equal one);
//   * a subtree of constants has one value: it becomes a constant leaf whose
//     value the device computes (fold_kernel), with the interpreter's own
//     arithmetic;
//   * the subtrees whose repeated evaluation costs most become derived rows: a
//     launch over the few of them writes their values beside the variables,
//     and every other program reads them as it reads a variable.
//
// Every operator still gets the operand values it had, so results do not
// change.  (The subtree cache of the reference, detect.cpp:120-387, serves
// repeated generations; this serves one launch, keeps nothing and costs a few
// rows of memory.)
#pragma once
#include <cstdint>
#include <memory>
#include <atomic>
#include <vector>

#include "sr_parallel.hpp"

namespace sr {

// Token marks for compile_expression's hints besides the cache's (>= 0 cached
// subtree, -1 none, -2 inside a collapsed one).
constexpr int32_t kHintFold = -3;      // root of a subtree of constants
constexpr int32_t kHintRow0 = -16;     // root of derived row r: kHintRow0 - r

constexpr int kMaxDerivedRows = 24;
constexpr int kMaxSharedTokens = 64;   // largest subtree folded or made a row

// Marks the maximal subtrees of constants of one expression (operators over
// constants only, at most kMaxSharedTokens tokens) for folding; returns
// whether there is one, false as well for a malformed expression.
bool mark_constant_subtrees(const int32_t *tok, int len, int32_t *hints);

// Adds an expression's cache hints to its fold marks: cached subtrees outside
// the folded ones stay collapsed.
void merge_hints(const int32_t *hints, int len, int32_t *marks);

class Sharing {
 public:
  struct Row {
    int64_t tok;   // first token of its representative
    int32_t size;
    int32_t occ;   // evaluations it replaces
  };

  // Hashes, counts and chooses up to max_rows rows for expressions [0, E) of a
  // CSR population.  False when an expression is malformed (compiling it
  // reports how) or host memory runs out.  The arrays are read until the last mark() / rep().
  bool find(int E, const int32_t *tok, const double *val, const int64_t *off, int max_rows,
            WorkerPool &pool, int threads);
  // Marks expression x's tokens (hints has its length) and returns whether
  // any is marked.
  bool mark(int x, int32_t *hints) const;
  // The row's own tokens (r.size of them), marked for folding only.
  void mark_row(const Row &r, int32_t *hints) const;
  // First expression equal to x (x itself when none is before it).
  int rep(int x) const;

  const std::vector<Row> &rows() const { return rows_; }
  void drop_rows() { keep_rows(0); }
  // The first n rows only (the most saving ones).
  void keep_rows(int n);

 private:
  struct Entry {
    std::atomic<uint64_t> key;
    std::atomic<uint32_t> count;
    std::atomic<uint32_t> at;   // token index of a representative / expression
  };
  Entry *insert(uint64_t key);
  const Entry *lookup(uint64_t key) const;
  bool equal_runs(int64_t a, int64_t b, int32_t n) const;
  struct Local;
  bool search(int E, const int32_t *tok, const double *val, const int64_t *off, int max_rows,
              WorkerPool &pool, int threads);
  bool hash_expression(int x, Local &local);
  void flush(Local &local, int slot);
  void choose(std::vector<uint32_t> &frequent, int max_rows);

  const int32_t *tok_ = nullptr;
  const double *val_ = nullptr;
  const int64_t *off_ = nullptr;
  int64_t n_tokens_ = 0;
  uint32_t min_count_ = 4;
  std::vector<uint64_t> hash_;   // per token: hash of the subtree rooted there
  std::vector<int16_t> size_;    // its tokens, negative when all its leaves are constants
  std::unique_ptr<Entry[]> table_;
  size_t cap_ = 0, mask_ = 0;
  std::vector<Row> rows_;
  int max_row_size_ = 0;
  void enter_row(uint64_t key, int r);
  uint64_t row_key_[256];        // open-addressed set of the rows' hashes
  int16_t row_of_[256];
};

}  // namespace sr
