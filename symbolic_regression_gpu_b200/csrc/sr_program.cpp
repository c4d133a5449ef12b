// sr_program.cpp — validation and bytecode compilation of prefix expressions.
//
// Semantics follow the reference CPU evaluator evaluate_single_expr
// (src/cleaned/cl_cpu_eval.cpp:59-90): tokens are consumed right to left, a
// constant pushes (float)value, a variable pushes x[(int)value] (0 when the
// index is not a valid input variable, cl_cpu_eval.cpp:70-76), an operator pops
// its left operand first (cl_gpu_eval.cu:98-101).
//
// The compiler builds the expression tree, labels every node with the number
// of spill slots its evaluation needs (Sethi-Ullman numbering: the child that
// needs more slots is evaluated first, which bounds the slots of a
// 127-token tree by 5), and emits one instruction per operator node with its
// leaf children folded in as operands.  Reordering the evaluation of two
// independent subtrees changes no floating-point result: every operator still
// receives exactly the same operand values.
#include "sr_program.hpp"

#include "sr_share.hpp"

#include <cmath>
#include <cstring>

namespace sr {

void subtree_sizes(const int32_t *tok, int len, int32_t *sizes) {
  // Reverse pass: children of position i start at i+1.
  for (int i = len - 1; i >= 0; --i) {
    const int t = tok[i];
    if (t <= 0) {
      sizes[i] = 1;
      continue;
    }
    const int arity = (t < 10) ? 2 : 1;
    int size = 1, pos = i + 1;
    for (int k = 0; k < arity && pos < len; ++k) {
      size += sizes[pos];
      pos += sizes[pos];
    }
    sizes[i] = size;
  }
}

void declared_op_work(int tok, double *sfu, double *fp32) {
  double s = 0, f = 0;
  switch (tok) {
    case SR_OP_ADD: case SR_OP_SUB: case SR_OP_MUL: case SR_OP_NEG:
    case SR_OP_ABS: case SR_OP_MIN: case SR_OP_MAX:
      f = 1; break;
    case SR_OP_LOOSE_DIV: case SR_OP_DIV: case SR_OP_INV: case SR_OP_LOOSE_INV:
      s = 1; f = 1; break;
    case SR_OP_LOOSE_SQRT: case SR_OP_SQRT:
      s = 1; break;
    case SR_OP_SIN: case SR_OP_COS:
      s = 1; f = 1; break;
    case SR_OP_EXP: case SR_OP_EXP_CLAMP:
      s = 1; f = 2; break;
    case SR_OP_LOG: case SR_OP_LOOSE_LOG:
      s = 1; f = 1; break;
    case SR_OP_POW: case SR_OP_LOOSE_POW:
      s = 2; f = 2; break;
    case SR_OP_TAN:
      s = 3; f = 2; break;
    case SR_OP_SINH: case SR_OP_COSH: case SR_OP_TANH:
      s = 2; f = 3; break;
    case SR_OP_ASIN: case SR_OP_ACOS: case SR_OP_ATAN:
      s = 1; f = 8; break;
    default: break;  // leaves
  }
  *sfu = s;
  *fp32 = f;
}

float op_cost(int tok) { return operator_cost(tok); }

namespace {

// Cost and declared work per device opcode (reversed opcodes like their
// operator), looked up once per instruction.
struct OpTables {
  float cost[64];
  float sfu[64], fp32[64];
  OpTables() {
    for (int k = 0; k < 64; ++k) {
      const int op = k > static_cast<int>(kOpReversed) ? k - static_cast<int>(kOpReversed) : k;
      double s, f;
      declared_op_work(op, &s, &f);
      cost[k] = 2.0f + op_cost(op);
      sfu[k] = static_cast<float>(s);
      fp32[k] = static_cast<float>(f);
    }
  }
};

struct Node {
  bool leaf = false;
  int32_t op = 0;          // operator token
  uint32_t lk = kLeafC;    // leaf kind (kLeafX / kLeafC / kLeafR)
  uint32_t lp = 0;         // leaf payload
  uint32_t lconst = kNoConst;
  int32_t fold = -1;       // token of a folded subtree this leaf stands for
  int32_t left = -1;       // first popped operand (operators)
  int32_t right = -1;      // second popped operand (binary)
  int32_t need = 0;
};

inline uint32_t float_bits(float f) {
  uint32_t u;
  std::memcpy(&u, &f, sizeof u);
  return u;
}

// (int)value with the reference's truncation; values that cannot be an int
// (NaN, huge) map to -1 = "not an input variable".
inline int var_index(double v) {
  if (!(v > -2147483648.0 && v < 2147483648.0)) return -1;
  return static_cast<int>(v);
}

inline uint32_t b_kind_of_leaf(uint32_t lk) {
  return lk == kLeafX ? kBX : (lk == kLeafC ? kBC : kBR);
}

// Opcode computing T = f(b, T) for binary token f.
inline uint32_t reversed(int tok) {
  return is_commutative_token(tok) ? static_cast<uint32_t>(tok)
                                   : kOpReversed + static_cast<uint32_t>(tok);
}

// Writes one program (its instruction count is known: one per operator node,
// one for a single leaf) and adds up its modelled cost.
struct Emitter {
  const Node *nodes;
  const OpTables &tab;
  int n_const;               // constants of the expression
  std::vector<FoldRef> *folds;
  Instr *out;                // the program's first instruction
  int count = 0;
  float cost = 0.f, sfu = 0.f, fp32 = 0.f;
  int pending_spill = -1;
  int sp = 0;
  int spill_at[kMaxSpillSlots + 1] = {};  // instruction that spilled into each slot

  // Constants are numbered in token order; the parse meets them from the right.
  uint32_t const_index(uint32_t from_right) const {
    return from_right == kNoConst ? kNoConst
                                  : static_cast<uint32_t>(n_const - 1) - from_right;
  }

  // [spill] [T = load] [b = operand] T = op(T, b)
  void emit(uint32_t op, const Node *load, uint32_t bk, uint32_t bp, uint32_t bc) {
    Instr ins;
    ins.w = (op & 63u) | ((bk & 7u) << 9);
    uint32_t ac = kNoConst;
    ins.a = 0;
    cost += tab.cost[op & 63u];
    sfu += tab.sfu[op & 63u];
    fp32 += tab.fp32[op & 63u];
    if (load) {
      ins.w |= kLoadBit | ((load->lk & 3u) << 7);
      ins.a = load->lp;
      ac = const_index(load->lconst);
      if (load->lk != kLeafC) cost += 0.5f;
      if (load->fold >= 0) folds->push_back(FoldRef{load->fold, count << 1});
    }
    if (pending_spill >= 0) {
      ins.w |= kSpillBit | (static_cast<uint32_t>(pending_spill) << 13);
      spill_at[pending_spill] = count;
      pending_spill = -1;
      cost += 0.5f;
    }
    if (bk == kBS || bk == kBX || bk == kBR) cost += 0.5f;
    ins.b = bp;
    // A spilled operand is the accumulator value right before its spill.
    const uint32_t producer = (bk == kBS) ? static_cast<uint32_t>(spill_at[bp] - 1) : 0u;
    ins.c = (ac & 0x3FFu) | ((const_index(bc) & 0x3FFu) << 10) | ((producer & 0x3FFu) << 20);
    out[count++] = ins;
  }

  void emit_b_leaf(uint32_t op, const Node *load, const Node &b) {
    if (b.fold >= 0) folds->push_back(FoldRef{b.fold, (count << 1) | 1});
    emit(op, load, b_kind_of_leaf(b.lk), b.lp, b.lconst);
  }

  void gen(int n) {
    const Node &nd = nodes[n];
    if (nd.leaf) {
      emit(kOpNone, &nd, kBNone, 0, kNoConst);
      return;
    }
    const Node &L = nodes[nd.left];
    const uint32_t op = static_cast<uint32_t>(nd.op);
    if (nd.right < 0) {  // unary
      if (L.leaf) {
        emit(op, &L, kBNone, 0, kNoConst);
      } else {
        gen(nd.left);
        emit(op, nullptr, kBNone, 0, kNoConst);
      }
      return;
    }
    const Node &R = nodes[nd.right];
    if (L.leaf && R.leaf) {
      emit_b_leaf(op, &L, R);              // T = L; T = f(T, R)
    } else if (R.leaf) {
      gen(nd.left);
      emit_b_leaf(op, nullptr, R);         // T = f(T=L, R)
    } else if (L.leaf) {
      gen(nd.right);
      emit_b_leaf(reversed(nd.op), nullptr, L);  // T = f(L, T=R)
    } else {
      // Both operands are operator subtrees: evaluate the one needing more
      // spill slots first (ties: the right one, the reference's own order),
      // park it in S[sp], evaluate the other into T, combine.
      const bool left_first = L.need > R.need;
      gen(left_first ? nd.left : nd.right);
      const int slot = sp++;
      pending_spill = slot;
      gen(left_first ? nd.right : nd.left);
      --sp;
      if (left_first)
        emit(reversed(nd.op), nullptr, kBS, static_cast<uint32_t>(slot), kNoConst);  // f(S, T)
      else
        emit(op, nullptr, kBS, static_cast<uint32_t>(slot), kNoConst);  // f(T, S)
    }
  }
};

const OpTables &op_tables() {
  static const OpTables tab;
  return tab;
}

}  // namespace

sr_status compile_expression(const int32_t *tok, const double *val, int len,
                             int num_vars, const int32_t *hints,
                             std::vector<Instr> &out, ExprInfo &info,
                             std::string *err, int first_row, std::vector<FoldRef> *folds) {
  info = ExprInfo{};
  info.n_tokens = len;
  if (len <= 0) {
    if (err) *err = "empty expression";
    return SR_ERR_MALFORMED_EXPRESSION;
  }
  if (len > SR_MAX_TOKENS) {
    if (err) *err = "expression has " + std::to_string(len) + " tokens (max " +
                    std::to_string(SR_MAX_TOKENS) + ")";
    return SR_ERR_EXPRESSION_TOO_LONG;
  }
  // One pass from the right: validation of the original token stream (known
  // tokens, no underflow, exactly one value left), constant numbering and the
  // tree, with cached subtrees (hints) collapsed to one leaf at their root.
  // Children get lower node ids than their parent, and a node's spill-slot
  // label (Sethi-Ullman) is known when it is made.
  const OpTables &tab = op_tables();
  thread_local std::vector<Node> node_store;
  thread_local std::vector<int32_t> stack_store;
  if (static_cast<int>(node_store.size()) < len) {
    node_store.resize(static_cast<size_t>(len));
    stack_store.resize(static_cast<size_t>(len) + 1);
  }
  Node *nodes = node_store.data();
  int32_t *stk = stack_store.data();
  int n_nodes = 0, sp = 0, depth = 0, n_ops = 0;
  uint32_t n_const = 0;
  bool bad_skeleton = false;
  // The leaf a collapsed subtree becomes.
  const auto collapse = [&](Node &nd, int hint, int i) {
    nd.leaf = true;
    nd.need = 0;
    nd.lconst = kNoConst;
    nd.fold = -1;
    if (hint >= 0) {
      nd.lk = kLeafR;
      nd.lp = static_cast<uint32_t>(hint);
    } else if (hint == kHintFold) {
      nd.lk = kLeafC;
      nd.lp = 0;
      nd.fold = i;
    } else {
      nd.lk = kLeafX;
      nd.lp = static_cast<uint32_t>(first_row + (kHintRow0 - hint));
    }
  };
  for (int i = len - 1; i >= 0; --i) {
    const int t = tok[i];
    const int hint = hints ? hints[i] : -1;
    const bool collapsed = hint >= 0 || hint == kHintFold || hint <= kHintRow0;
    // -2: inside a collapsed subtree; -1: neither.
    if (t == SR_TOK_CONST || t == SR_TOK_VAR) {
      ++depth;
      const uint32_t ci = n_const;
      if (t == SR_TOK_CONST) ++n_const;
      if (hint == -2) continue;
      Node &nd = nodes[n_nodes];
      nd.leaf = true;
      nd.need = 0;
      nd.lconst = kNoConst;
      nd.fold = -1;
      if (collapsed) {
        collapse(nd, hint, i);
      } else if (t == SR_TOK_CONST) {
        nd.lk = kLeafC;
        nd.lp = float_bits(static_cast<float>(val[i]));
        nd.lconst = ci;
      } else {
        const int v = var_index(val[i]);
        const bool ok = v >= 0 && v < num_vars;
        nd.lk = ok ? kLeafX : kLeafC;  // reference CPU pushes 0.0f (cl_cpu_eval.cpp:73-75)
        nd.lp = ok ? static_cast<uint32_t>(v) : float_bits(0.0f);
      }
      stk[sp++] = n_nodes++;
      continue;
    }
    const bool binary = is_binary_token(t);
    if (!binary && !is_unary_token(t)) {
      if (err) *err = "unknown token " + std::to_string(t) + " at position " + std::to_string(i);
      return SR_ERR_BAD_TOKEN;
    }
    if (depth < (binary ? 2 : 1)) {
      if (err) *err = "stack underflow at token " + std::to_string(i);
      return SR_ERR_MALFORMED_EXPRESSION;
    }
    if (binary) --depth;
    if (hint == -2 || bad_skeleton) continue;
    Node &nd = nodes[n_nodes];
    nd.lconst = kNoConst;
    nd.fold = -1;
    if (collapsed) {
      collapse(nd, hint, i);
      stk[sp++] = n_nodes++;
      continue;
    }
    if (sp < (binary ? 2 : 1)) {
      bad_skeleton = true;
      continue;
    }
    nd.leaf = false;
    nd.op = t;
    nd.left = stk[--sp];
    nd.right = -1;
    const Node &L = nodes[nd.left];
    nd.need = L.need;  // a leaf's is 0
    if (binary) {
      nd.right = stk[--sp];
      const Node &R = nodes[nd.right];
      if (R.leaf) nd.need = L.need;
      else if (L.leaf) nd.need = R.need;
      else nd.need = (L.need == R.need) ? L.need + 1 : std::max(L.need, R.need);
    }
    ++n_ops;
    stk[sp++] = n_nodes++;
  }
  if (depth != 1) {
    if (err) *err = "expression leaves " + std::to_string(depth) + " values on the stack";
    return SR_ERR_MALFORMED_EXPRESSION;
  }
  if (bad_skeleton || sp != 1) {
    if (err) *err = "cache marking produced an invalid skeleton";
    return SR_ERR_MALFORMED_EXPRESSION;
  }
  const int root = stk[0];
  info.n_const = static_cast<int>(n_const);
  info.n_executed = n_nodes;
  info.need = nodes[root].need;
  if (info.need > kMaxSpillSlots) {
    if (err) *err = "expression needs " + std::to_string(info.need) +
                    " spill slots (max " + std::to_string(kMaxSpillSlots) + ")";
    return SR_ERR_EXPRESSION_TOO_LONG;
  }

  const size_t first = out.size();
  info.n_instr = std::max(n_ops, 1);
  out.resize(first + static_cast<size_t>(info.n_instr));
  Emitter em{nodes, tab, info.n_const, folds, out.data() + first};
  em.gen(root);
  info.cost = em.cost + 6.0f;           // epilogue
  info.sfu_ops = em.sfu;
  info.fp32_ops = em.fp32 + 3.0;        // MSE epilogue per datapoint (declared model)
  return SR_OK;
}

}  // namespace sr
