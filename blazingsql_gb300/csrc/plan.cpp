// plan.cpp -- expression DAG + CUDA code generation (see plan.h).
#include "plan.h"

#include "fp64emu.cuh"

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <set>
#include <sstream>

namespace gx {
namespace {

std::string hex64(uint64_t v) {
  char buf[32];
  std::snprintf(buf, sizeof buf, "0x%016llxull", (unsigned long long)v);
  return buf;
}

struct Builder {
  Plan& p;
  std::map<std::string, int> memo;
  int rand_counter = 0;
  bool rand_out_row = false;

  int push(Node n, const std::string& key) {
    if (!key.empty()) {
      auto it = memo.find(key);
      if (it != memo.end()) return it->second;
    }
    p.nodes.push_back(n);
    int id = (int)p.nodes.size() - 1;
    if (!key.empty()) memo[key] = id;
    return id;
  }

  int add(const ExprPtr& e) {
    if (e->kind == Expr::COL) {
      Node n;
      n.kind = Node::COL;
      n.col = e->col;
      n.vtype = e->vtype;
      n.ktype = e->ktype;
      return push(n, "c" + std::to_string(e->col));
    }
    if (e->kind == Expr::LIT) {
      Node n;
      n.kind = Node::LIT;
      n.lit_type = e->lit_type;
      n.lit_valid = e->lit_valid;
      n.lit_bits = e->lit_bits;
      n.vtype = e->vtype;
      n.ktype = e->ktype;
      return push(n, "l" + std::to_string(e->vtype) + ":" + std::to_string(e->ktype) + ":" +
                         std::to_string(e->lit_valid) + ":" + std::to_string(e->lit_bits));
    }
    // every operand is visited (RAND ordinals follow the reference's post-order
    // visit, which also walks the extra operands of an un-nested OR)
    std::vector<int> kids;
    for (const auto& c : e->ch) kids.push_back(add(c));
    Node n;
    n.kind = Node::OP;
    n.op = e->op;
    n.vtype = e->vtype;
    n.ktype = e->ktype;
    if (!kids.empty()) n.a = kids[0];
    if (op_is_binary(e->op) && kids.size() > 1) n.b = kids[1];
    if (e->op == OP_RAND) {
      n.rand_id = rand_counter++;
      n.rand_out_row = rand_out_row;
      return push(n, "");  // never shared
    }
    return push(n, "o" + std::to_string(n.op) + ":" + std::to_string(n.a) + ":" + std::to_string(n.b) + ":" +
                       std::to_string(n.vtype) + ":" + std::to_string(n.ktype));
  }
};

void flatten_and(const Plan& p, int id, std::vector<int>& out) {
  const Node& n = p.nodes[id];
  if (n.kind == Node::OP && n.op == OP_AND) {
    flatten_and(p, n.a, out);
    flatten_and(p, n.b, out);
  } else {
    out.push_back(id);
  }
}

}  // namespace

uint64_t OutSpec::lit_bits_as_element() const {
  if (type == FLOAT32) {
    double d;
    std::memcpy(&d, &lit_bits, 8);
    const float f = (float)d;
    uint32_t u;
    std::memcpy(&u, &f, 4);
    return u;
  }
  if (type == BOOL8) return lit_bits != 0;
  return lit_bits;
}

bool Plan::needs_kernel() const {
  if (has_filter()) return true;
  for (const auto& o : outputs)
    if (o.kind == OutSpec::NODE) return true;
  return false;
}

Plan build_plan(const std::vector<int>& schema, const std::vector<bool>& nullable, const std::string& condition,
                const std::vector<std::string>& expressions, bool filter_all, bool rand_by_output_row,
                int first_rand_id, int* rand_count, bool all_nodes) {
  Plan p;
  p.schema = schema;
  p.nullable = nullable;
  Builder b{p};
  if (!condition.empty()) {
    ExprPtr c = compile_expression(condition, schema);
    if (c->vtype != BOOL8) fail(GX_ERR_TYPE, "Expression does not evaluate to a boolean mask");
    p.predicate = b.add(c);
    flatten_and(p, p.predicate, p.conjuncts);
  }
  b.rand_counter = first_rand_id;
  b.rand_out_row = rand_by_output_row && !condition.empty();
  if (filter_all) {
    p.filter_copies_all = true;
    for (size_t i = 0; i < schema.size(); i++) {
      OutSpec o;
      o.kind = OutSpec::COPY;
      o.col = (int)i;
      o.type = schema[i];
      p.outputs.push_back(o);
    }
  } else {
    for (const auto& text : expressions) {
      ExprPtr e = compile_expression(text, schema);
      OutSpec o;
      if (e->kind == Expr::LIT && all_nodes) {
        fail(GX_ERR_UNSUPPORTED, "a literal aggregation input");
      } else if (e->kind == Expr::LIT) {
        o.kind = OutSpec::BROADCAST;
        o.type = e->lit_type;
        o.lit_bits = e->lit_bits;
        o.lit_valid = e->lit_valid;
        if (o.type == EMPTY || type_size(o.type) == 0) fail(GX_ERR_TYPE, "a bare null literal has no column type");
      } else if (e->kind == Expr::COL && !all_nodes) {
        o.kind = OutSpec::COPY;
        o.col = e->col;
        o.type = schema[e->col];
      } else {
        o.kind = OutSpec::NODE;
        o.node = b.add(e);
        o.type = e->vtype;
        if (type_size(o.type) == 0) fail(GX_ERR_TYPE, "expression has no fixed-width output type");
      }
      p.outputs.push_back(o);
    }
  }
  if (rand_count) *rand_count = b.rand_counter - first_rand_id;
  if (p.outputs.size() > (size_t)GX_MAX_OUTS) fail(GX_ERR_UNSUPPORTED, "too many output columns in one plan");
  if (schema.size() > (size_t)GX_MAX_COLS) fail(GX_ERR_UNSUPPORTED, "too many input columns in one plan");
  // data under NULL is observable where it reaches CASE's magic-number test
  for (int i = (int)p.nodes.size() - 1; i >= 0; i--) {
    Node& n = p.nodes[i];
    if (n.kind != Node::OP) continue;
    if (n.op == OP_MAGIC_IF_NOT && n.b >= 0) p.nodes[n.b].exact_null = true;
    if (n.op == OP_FIRST_NON_MAGIC) {
      p.nodes[n.a].exact_null = true;
      if (n.exact_null) p.nodes[n.b].exact_null = true;
    }
  }
  return p;
}

// =============================================================== code generation
namespace {

const char* load_fn(int t) {
  switch (t) {
    case INT8: return "gx_ld_i8";
    case UINT8: case BOOL8: return "gx_ld_u8";
    case INT16: return "gx_ld_i16";
    case UINT16: return "gx_ld_u16";
    case INT32: case TIMESTAMP_DAYS: case DURATION_DAYS: return "gx_ld_i32";
    case UINT32: return "gx_ld_u32";
    case FLOAT32: return "gx_ld_f32";
    default: return "gx_ld_64";
  }
}

const char* load_fn_emu(int t) { return t == FLOAT32 ? "gx_ld_f32e" : load_fn(t); }

// store of 64-bit value bits into an output column of type t
// (device_ptr_write_from_buffer, interpreter_ops.cuh:329-395)
std::string store_stmt(int t, const std::string& ptr, const std::string& idx, const std::string& bits) {
  switch (t) {
    case BOOL8: return "gx_st_8(" + ptr + ", " + idx + ", (u64)((" + bits + ") != 0ull));";
    case INT8: case UINT8: return "gx_st_8(" + ptr + ", " + idx + ", " + bits + ");";
    case INT16: case UINT16: return "gx_st_16(" + ptr + ", " + idx + ", " + bits + ");";
    case INT32: case UINT32: case TIMESTAMP_DAYS: case DURATION_DAYS:
      return "gx_st_32(" + ptr + ", " + idx + ", " + bits + ");";
    case FLOAT32: return "gx_st_f32(" + ptr + ", " + idx + ", " + bits + ");";
    default: return "gx_st_64(" + ptr + ", " + idx + ", " + bits + ");";
  }
}

// raw element copy for COPY outputs of filter kernels
std::string raw_type(int t) {
  switch (type_size(t)) {
    case 1: return "unsigned char";
    case 2: return "unsigned short";
    case 4: return "unsigned int";
    default: return "unsigned long long";
  }
}

double bits_double(uint64_t u) {
  double d;
  std::memcpy(&d, &u, 8);
  return d;
}

uint64_t magic_double_bits() {
  const double m = 1.7976931348623123e+308;  // interpreter_ops.cuh:47
  uint64_t u;
  std::memcpy(&u, &m, 8);
  return u;
}

int64_t ns_per_unit(int t) {
  switch (t) {
    case TIMESTAMP_DAYS: case DURATION_DAYS: return 86400000000000LL;
    case TIMESTAMP_SECONDS: case DURATION_SECONDS: return 1000000000LL;
    case TIMESTAMP_MILLISECONDS: case DURATION_MILLISECONDS: return 1000000LL;
    case TIMESTAMP_MICROSECONDS: case DURATION_MICROSECONDS: return 1000LL;
    default: return 1;
  }
}

class Gen {
 public:
  Gen(const Plan& p, const KernelConfig& c) : p_(p), cfg_(c) {
    for (int r : p.conjuncts) {
      const Node& n = p.nodes[r];
      // IS NOT NULL proves its operand valid where it is true: as a conjunct
      prove_valid(n.kind == Node::OP && n.op == OP_IS_NOT_NULL ? n.a : r);
    }
  }

  // Columns that are valid in every row a conjunct keeps: a kept row's
  // conjunct is valid and true, and an operator that is NULL whenever an
  // operand is makes its operands valid too.  The walk carries validity only,
  // so it ends at operators that are valid whatever their operands are: under
  // NOT or a comparison, IS NOT NULL($0) may be false in a kept row.
  void prove_valid(int id) {
    const Node& n = p_.nodes[id];
    if (n.kind == Node::COL) { proven_.insert(n.col); return; }
    if (n.kind != Node::OP) return;
    switch (n.op) {
      case OP_OR: case OP_IS_NULL: case OP_IS_NOT_NULL: case OP_IS_TRUE: case OP_IS_NOT_TRUE: case OP_IS_NOT_FALSE:
      case OP_IS_NOT_DISTINCT_FROM: case OP_MAGIC_IF_NOT: case OP_FIRST_NON_MAGIC: case OP_RAND: case OP_ROW_INDEX:
        return;
      default: break;
    }
    if (n.a >= 0) prove_valid(n.a);
    if (n.b >= 0) prove_valid(n.b);
  }

  // operand views for node id in word-slot k
  std::string B(int id) const { return value_bits(id); }
  std::string V(int id) const { return value_valid(id); }

  std::string value_bits(int id) const {
    const Node& n = p_.nodes[id];
    if (n.kind == Node::LIT) return n.lit_valid ? hex64(n.lit_bits) : std::string("0ull");
    return "b" + std::to_string(id) + "[k]";
  }
  std::string value_valid(int id) const {
    const Node& n = p_.nodes[id];
    if (n.kind == Node::LIT) return n.lit_valid ? "true" : "false";
    return "v" + std::to_string(id) + "[k]";
  }
  bool kind_f(int id) const { return is_float(p_.nodes[id].ktype); }
  // Bound on an integer-kind node's values: |v| < 2^bits (64: none known).
  // Plans do not narrow at CASTs, so a CAST keeps its operand's bound; data
  // under NULL is bounded like any other (columns are sign- or zero-extended
  // from their storage type, and an unselected row reads 0).
  int int_bits(int id) const {
    const Node& n = p_.nodes[id];
    if (kind_f(id)) return 64;
    if (n.kind == Node::LIT) {
      const int64_t v = n.lit_valid ? (int64_t)n.lit_bits : 0;
      const uint64_t u = v < 0 ? 0ull - (uint64_t)v : (uint64_t)v;
      return u == 0 ? 1 : 64 - __builtin_clzll(u);
    }
    if (n.kind == Node::COL) {
      switch (p_.schema[n.col]) {
        case INT8: case UINT8: case BOOL8: return 8;
        case INT16: case UINT16: return 16;
        case INT32: case UINT32: case TIMESTAMP_DAYS: case DURATION_DAYS: return 32;
        default: return 64;
      }
    }
    switch (n.op) {
      case OP_EQ: case OP_NE: case OP_LT: case OP_GT: case OP_LE: case OP_GE: case OP_AND: case OP_NOT:
      case OP_IS_NULL: case OP_IS_NOT_NULL: case OP_IS_NOT_TRUE: case OP_IS_NOT_FALSE:
      case OP_IS_NOT_DISTINCT_FROM:
        return 1;
      case OP_CAST_TINYINT: case OP_CAST_SMALLINT: case OP_CAST_INTEGER: case OP_CAST_BIGINT: case OP_ABS:
        return int_bits(n.a);
      case OP_MOD:
        if (kind_f(n.a) || kind_f(n.b)) return 64;
        return p_.nodes[n.b].kind == Node::LIT ? std::min(int_bits(n.a), int_bits(n.b)) : int_bits(n.a);
      case OP_ADD: case OP_SUB:
        if (kind_f(n.a) || kind_f(n.b)) return 64;
        return std::min(64, std::max(int_bits(n.a), int_bits(n.b)) + 1);
      case OP_MUL:
        if (kind_f(n.a) || kind_f(n.b)) return 64;
        return std::min(64, int_bits(n.a) + int_bits(n.b));
      default: return 64;
    }
  }
  // (double) of an integer-kind node on the integer pipes, as bits; 31 bits
  // and a sign (INT32's lowest value included) take the 32-bit form
  std::string int_to_double(int id) const {
    const Node& n = p_.nodes[id];
    if (n.kind == Node::LIT) return hex64(n.lit_valid ? literal_double_bits(id) : 0ull);
    const bool i32 = n.kind == Node::COL && p_.schema[n.col] != UINT32 && int_bits(id) <= 32;
    if (i32 || int_bits(id) <= 31) return "gxe_i2d32((int)(" + B(id) + "))";
    return "gxe_i2d((i64)(" + B(id) + "))";
  }
  // operand as a double value (native FP64 arithmetic follows)
  std::string asD(int id) const {
    if (kind_f(id)) return "gx_D(" + B(id) + ")";
    return emu_op(kNativeConvert) ? "gx_D(" + int_to_double(id) + ")" : "gx_I2D(" + B(id) + ")";
  }
  // operand as the bits of its double value (integer-pipe binary64 routines follow)
  std::string asDB(int id) const {
    if (kind_f(id)) return B(id);
    return emu_op(kNativeConvert) ? int_to_double(id) : "gx_B(gx_I2D(" + B(id) + "))";
  }
  std::string asI(int id) const {
    if (!kind_f(id)) return "(i64)(" + B(id) + ")";
    return emu_op(kNativeConvert) ? "gxe_d2ll(" + B(id) + ")" : "gx_D2LL(gx_D(" + B(id) + "))";
  }
  std::string nz(int id) const {
    if (!kind_f(id)) return "(" + B(id) + " != 0ull)";
    return emu() ? "gxe_nz(" + B(id) + ")" : "(gx_D(" + B(id) + ") != 0.0)";
  }
  bool emu() const { return cfg_.emulate_fp64; }
  // this class of binary64 operation runs on the integer pipes
  bool emu_op(int cls) const { return cfg_.emulate_fp64 && !(cfg_.native_f64_ops & cls); }

  // a valid literal's value as binary64 bits (integer literals converted exactly
  // as the kernels convert them)
  uint64_t literal_double_bits(int id) const {
    const Node& n = p_.nodes[id];
    return kind_f(id) ? n.lit_bits : gxe_i2d((gxe_i64)n.lit_bits);
  }
  // A node whose value is an integer (an integer-kind node, or its CAST to
  // DOUBLE / FLOAT, which keeps the exact value inside a plan): the node
  // holding that integer, or -1.  A CAST whose data under NULL is observable
  // reads as 0 there, which the integer would not, so it counts as a double.
  int int_source(int y) const {
    const Node& n = p_.nodes[y];
    if (n.kind == Node::LIT) return -1;
    if (!kind_f(y)) return y;
    if (n.kind == Node::OP && (n.op == OP_CAST_DOUBLE || n.op == OP_CAST_FLOAT) && !kind_f(n.a) && !n.exact_null &&
        p_.nodes[n.a].kind != Node::LIT)
      return n.a;
    return -1;
  }
  // a division by an integer value reads the divisor's reciprocal from a table
  bool small_div(int id) const {
    const Node& n = p_.nodes[id];
    return n.kind == Node::OP && n.op == OP_DIV && (kind_f(n.a) || kind_f(n.b)) && emu_op(kNativeDiv) &&
           !const_divisor(n.b) && int_source(n.b) >= 0;
  }
  // The reciprocal table of the plan's divisions by an integer value, when it
  // has one: 64-bit reciprocals of the integers' significands rounded down
  // (gxe_div_k), or RN(1 / k) as binary64 (gxe_div_small on the FMA unit).
  void emit_rcp_table(std::ostringstream& o) const {
    bool any = false;
    for (size_t i = 0; i < p_.nodes.size() && !any; i++) any = small_div((int)i);
    if (!any) return;
    if (emu_op(kNativeIntDiv)) {
      static const std::string fixed = rcp_table(true);
      o << fixed;
    } else {
      static const std::string binary64 = rcp_table(false);
      o << binary64;
    }
  }
  static std::string rcp_table(bool fixed) {
    std::ostringstream o;
    o << "#define GX_RCP_N " << kRcpTable << "\n__device__ const unsigned long long gx_rcp_[GX_RCP_N] = {";
    for (int k = 1; k <= kRcpTable; k++) {
      const double y = fixed ? (double)k : 1.0 / (double)k;
      uint64_t b;
      std::memcpy(&b, &y, 8);
      if (fixed) b = gxe_recip_floor((b & GXE_FRAC) | GXE_HIDDEN);
      o << (k > 1 ? "," : "") << (k % 8 == 1 ? "\n  " : "") << hex64(b);
    }
    o << "};\n";
    return o.str();
  }
  static constexpr int kRcpTable = 1024;
  // a literal divisor that is a normal finite nonzero double
  bool const_divisor(int id) const {
    const Node& n = p_.nodes[id];
    if (n.kind != Node::LIT || !n.lit_valid) return false;
    const int e = (int)((literal_double_bits(id) >> 52) & 0x7FF);
    return e >= 1 && e <= 2046;
  }

  // the load of a column's element at `row` (data pointers start at the batch's first row)
  std::string load_call(int c) const {
    std::string fn = emu() ? load_fn_emu(p_.schema[c]) : load_fn(p_.schema[c]);
    // a kept-row round starts and ends inside a sector that its neighbours read
    // too, so it loads with the default policy (order-line plan 2^27: 1.75 ms
    // against 1.89 with evict-first loads)
    if (reread_cols_.count(c) || masks_ == Masks::KEPT) fn = "gx_ldg_" + fn.substr(6);  // gx_ld_X -> gx_ldg_X
    return fn + "(a.in_data[" + std::to_string(c) + "], row)";
  }
  // where a row's validity bit is read from
  enum class Masks {
    GLOBAL,  // the mask, by row
    WORDS,   // lane l holds word l of the warp's words (mw_<c>); slot k, bit `lane`
    KEPT,    // the same words; the row's offset within the warp's rows is kp_, and
             // the condition has made the proven_ columns valid
  };
  mutable Masks masks_ = Masks::GLOBAL;
  // a warp of more than 32 words has more of them than lanes: rows read their bits from the mask
  bool lane_words() const { return cfg_.words <= 32; }
  bool masked(int c) const { return p_.nullable[c] && !(masks_ == Masks::KEPT && proven_.count(c)); }
  // validity of column c for the lane's row
  std::string col_valid(int c) const {
    const std::string cs = std::to_string(c);
    if (!masked(c)) return "inr";
    switch (lane_words() ? masks_ : Masks::GLOBAL) {
      case Masks::WORDS: return "(gx_wbit(mw_" + cs + ", k, lane) && inr)";
      case Masks::KEPT: return "(gx_wbit(mw_" + cs + ", kp_ >> 5, kp_ & 31u) && inr)";
      default: return "(inr && gx_valid(a.in_mask[" + cs + "], a.in_off[" + cs + "] + row))";
    }
  }
  // the validity words that the rows of `ids` and of the columns `more` need,
  // one word per lane (words w0 .. w0 + GX_V - 1)
  void emit_mask_words(std::ostringstream& o, const std::vector<int>& ids, const std::vector<int>& more,
                       const std::string& ind) const {
    if (!lane_words()) return;
    std::set<int> cols(more.begin(), more.end());
    for (int id : ids)
      if (p_.nodes[id].kind == Node::COL) cols.insert(p_.nodes[id].col);
    for (int c : cols)
      if (masked(c))
        o << ind << "const u32 mw_" << c << " = lane < GX_V ? gx_mask_word(a.in_mask[" << c << "], a.in_off[" << c
          << "], w0 + lane, a.n) : 0u;\n";
  }

  // statements computing node id for slot k; row / out-row expressions given
  void emit_node(std::ostringstream& o, int id, const std::string& ind) const {
    const Node& n = p_.nodes[id];
    const std::string b = "b" + std::to_string(id) + "[k]", v = "v" + std::to_string(id) + "[k]";
    if (n.kind == Node::LIT) return;
    if (n.kind == Node::COL) {
      const int c = n.col;
      if (tile_mode_) {
        // the tile's rows of column c are in shared memory: element trow at
        // byte offset sd_<c> + trow * width, validity bit trow of the tile's
        // re-aligned mask words vmw_<c>
        const std::string gfn = emu() ? load_fn_emu(p_.schema[c]) : load_fn(p_.schema[c]);
        const std::string sfn = "gx_sld_" + gfn.substr(6);  // gx_ld_X -> gx_sld_X
        o << ind << b << " = inr ? (u64)" << sfn << "(sd_" << c << " + trow * " << type_size(p_.schema[c])
          << "u) : 0ull;\n";
        if (p_.nullable[c]) o << ind << v << " = inr && ((vmw_" << c << "[trow >> 5] >> (trow & 31u)) & 1u);\n";
        else o << ind << v << " = inr;\n";
        return;
      }
      auto st = staged_.find(c);
      if (st != staged_.end()) {
        // full words are staged in shared memory at (buffer, index); a partial
        // last word is read from global memory
        const std::string gfn = emu() ? load_fn_emu(p_.schema[c]) : load_fn(p_.schema[c]);
        const std::string sfn = "gx_lds_" + gfn.substr(6);  // gx_ld_X -> gx_lds_X
        o << ind << b << " = inr ? (full_word_ ? (u64)" << sfn << "(" << st->second.first << ", " << st->second.second
          << ") : (u64)" << gfn << "(a.in_data[" << c << "], row)) : 0ull;\n";
      } else {
        o << ind << b << " = inr ? (u64)" << load_call(c) << " : 0ull;\n";
      }
      o << ind << v << " = " << col_valid(c) << ";\n";
      return;
    }
    std::string r, vv;
    const Op op = n.op;
    if (op == OP_RAND) {
      o << ind << b << " = gx_B(gx_philox_uniform(a.seed, " << n.rand_id << "u, (u64)("
        << (n.rand_out_row ? "orow" : "row") << ")));\n";
      o << ind << v << " = true;\n";
      return;
    }
    if (op == OP_ROW_INDEX) {
      o << ind << b << " = (u64)row;\n";
      o << ind << v << " = true;\n";
      return;
    }
    if (op_is_unary(op)) {
      const int x = n.a;
      const int lt = p_.nodes[x].ktype;
      const bool lf = kind_f(x);
      const std::string X = B(x), XV = V(x);
      bool always_valid = false;
      switch (op) {
        case OP_IS_NOT_TRUE:
          r = "(u64)(!(" + XV + " && " + (lf ? "(" + X + ") == 0x3ff0000000000000ull" : "(i64)(" + X + ") == 1LL") +
              "))";
          always_valid = true;
          break;
        case OP_IS_NOT_FALSE:
          r = "(u64)(!(" + XV + " && " + (lf ? "((" + X + ") << 1) == 0ull" : "(i64)(" + X + ") == 0LL") + "))";
          always_valid = true;
          break;
        case OP_IS_NULL: r = "(u64)(!" + XV + ")"; always_valid = true; break;
        case OP_IS_NOT_NULL: r = "(u64)(" + XV + ")"; always_valid = true; break;
        case OP_FLOOR: r = emu_op(kNativeRound) ? "gxe_floor(" + asDB(x) + ")" : "gx_B(floor(" + asD(x) + "))"; break;
        case OP_CEIL: r = emu_op(kNativeRound) ? "gxe_ceil(" + asDB(x) + ")" : "gx_B(ceil(" + asD(x) + "))"; break;
        case OP_SIN: r = "gx_B(sin(" + asD(x) + "))"; break;
        case OP_COS: r = "gx_B(cos(" + asD(x) + "))"; break;
        case OP_ASIN: r = "gx_B(asin(" + asD(x) + "))"; break;
        case OP_ACOS: r = "gx_B(acos(" + asD(x) + "))"; break;
        case OP_TAN: r = "gx_B(tan(" + asD(x) + "))"; break;
        case OP_COTAN: r = "gx_B(cos(" + asD(x) + ") / sin(" + asD(x) + "))"; break;
        case OP_ATAN: r = "gx_B(atan(" + asD(x) + "))"; break;
        case OP_LN: r = "gx_B(log(" + asD(x) + "))"; break;
        case OP_LOG10: r = "gx_B(log10(" + asD(x) + "))"; break;
        case OP_EXP: r = "gx_B(exp(" + asD(x) + "))"; break;
        case OP_ABS:
          r = lf ? "((" + X + ") & 0x7fffffffffffffffull)" : "((i64)(" + X + ") < 0LL ? 0ull - (" + X + ") : (" + X + "))";
          break;
        case OP_NOT: r = "(u64)(!" + nz(x) + ")"; break;
        case OP_IS_TRUE: r = "(u64)" + asI(x); break;
        case OP_YEAR: case OP_MONTH: case OP_DAY: case OP_DAYOFWEEK: case OP_HOUR: case OP_MINUTE: case OP_SECOND: {
          if (!is_timestamp(lt)) { r = "0ull"; break; }
          const int which = op == OP_YEAR ? 0 : op == OP_MONTH ? 1 : op == OP_DAY ? 2 : op == OP_DAYOFWEEK ? 3
                          : op == OP_HOUR ? 4 : op == OP_MINUTE ? 5 : 6;
          const long long per_day = lt == TIMESTAMP_DAYS ? 1LL : 86400000000000LL / ns_per_unit(lt);
          const std::string cnt = lt == TIMESTAMP_DAYS ? "gx_days32((i64)(" + X + "))" : "(i64)(" + X + ")";
          if (per_day == 1 && which <= 2)  // a DATE's parts in 32-bit arithmetic
            r = "(u64)gx_civil32((int)(" + X + "), " + std::to_string(which) + ")";
          else
            r = "(u64)gx_extract(" + cnt + ", " + std::to_string(per_day) + "LL, " + std::to_string(which) + ")";
          break;
        }
        case OP_CAST_TINYINT: case OP_CAST_SMALLINT: case OP_CAST_INTEGER: case OP_CAST_BIGINT:
          r = "(u64)" + asI(x);
          break;
        case OP_CAST_FLOAT: case OP_CAST_DOUBLE: r = asDB(x); break;
        case OP_CAST_DATE: {
          long long div = lt == TIMESTAMP_SECONDS ? 86400LL : lt == TIMESTAMP_MILLISECONDS ? 86400000LL
                        : lt == TIMESTAMP_MICROSECONDS ? 86400000000LL : lt == TIMESTAMP_NANOSECONDS ? 86400000000000LL : 1;
          r = div == 1 ? "(u64)(i64)(int)" + asI(x) : "(u64)(i64)(int)(" + asI(x) + " / " + std::to_string(div) + "LL)";
          break;
        }
        case OP_CAST_TIMESTAMP_SECONDS: case OP_CAST_TIMESTAMP_MILLISECONDS: case OP_CAST_TIMESTAMP_MICROSECONDS:
        case OP_CAST_TIMESTAMP:
          if (is_timestamp(lt)) {
            const std::string cnt = lt == TIMESTAMP_DAYS ? "(u64)gx_days32(" + asI(x) + ")" : "(u64)" + asI(x);
            r = "(" + cnt + " * " + std::to_string(ns_per_unit(lt)) + "ull)";
          } else {
            r = "(u64)" + asI(x);
          }
          break;
        default: fail(GX_ERR_UNSUPPORTED, "no code for unary operator");
      }
      vv = always_valid ? "true" : XV;
      if (!always_valid && n.exact_null) r = "(" + vv + " ? " + r + " : 0ull)";
      o << ind << b << " = " << r << ";\n" << ind << v << " = " << vv << ";\n";
      return;
    }
    // binary
    const int x = n.a, y = n.b;
    const bool lf = kind_f(x), rf = kind_f(y), anyf = lf || rf;
    const int lt = p_.nodes[x].ktype, rt = p_.nodes[y].ktype;
    const std::string X = B(x), Y = B(y), XV = V(x), YV = V(y);
    switch (op) {
      case OP_MAGIC_IF_NOT: {
        const std::string cond = "(" + XV + " && " + nz(x) + ")";
        o << ind << "{ const bool c_ = " << cond << ";\n";
        o << ind << "  " << b << " = c_ ? " << Y << " : " << (rf ? "gx_B(GX_MAGIC_D)" : "(u64)GX_MAGIC_I")
          << ";\n";
        o << ind << "  " << v << " = c_ ? " << YV << " : false; }\n";
        return;
      }
      case OP_FIRST_NON_MAGIC: {
        // double equality with the (non-zero, finite) magic value is bit equality
        const std::string magic = lf ? "((" + X + ") == " + hex64(magic_double_bits()) + ")"
                                     : "((i64)(" + X + ") == GX_MAGIC_I)";
        o << ind << "{ const bool m_ = " << magic << ";\n";
        o << ind << "  " << b << " = m_ ? " << Y << " : " << X << ";\n";
        o << ind << "  " << v << " = m_ ? " << YV << " : " << XV << "; }\n";
        return;
      }
      case OP_OR:
        o << ind << b << " = (" << XV << " && " << YV << ") ? (u64)(" << nz(x) << " || " << nz(y) << ") : (" << XV
          << " ? " << X << " : (" << YV << " ? " << Y << " : 0ull));\n";
        o << ind << v << " = (" << XV << " && " << YV << ") || (" << XV << " ? " << nz(x) << " : " << YV << ");\n";
        return;
      case OP_IS_NOT_DISTINCT_FROM: {
        const std::string eq = !anyf ? "(" + X + " == " + Y + ")"
                               : emu_op(kNativeCompare) ? "gxe_eq(" + asDB(x) + ", " + asDB(y) + ")"
                                       : "(" + asD(x) + " == " + asD(y) + ")";
        o << ind << b << " = (u64)((!" << XV << " && !" << YV << ") || (" << XV << " && " << YV << " && " << eq
          << "));\n";
        o << ind << v << " = true;\n";
        return;
      }
      default: break;
    }
    vv = "(" + XV + " && " + YV + ")";
    const bool ts_cmp = is_timestamp(lt) && is_timestamp(rt);
    auto cmp = [&](const char* opstr) -> std::string {
      if (ts_cmp) {
        auto to_ns = [&](int id, int t) {
          const std::string cnt = t == TIMESTAMP_DAYS ? "(u64)gx_days32((i64)(" + B(id) + "))" : "(u64)(" + B(id) + ")";
          return "(i64)(" + cnt + " * " + std::to_string(ns_per_unit(t)) + "ull)";
        };
        return std::string("(u64)(") + to_ns(x, lt) + " " + opstr + " " + to_ns(y, rt) + ")";
      }
      if (anyf && emu() && p_.nodes[y].kind == Node::LIT && p_.nodes[y].lit_valid && kind_f(x) &&
          !gxe_isnan_(literal_double_bits(y))) {  // ranges of x's bits: no FP64-pipe compare
        const std::string C = hex64(literal_double_bits(y)), o2 = opstr;
        if (o2 == "!=") return "(u64)(!gxe_eqc(" + X + ", " + C + "))";
        return "(u64)" + std::string(o2 == "<" ? "gxe_ltc(" : o2 == ">" ? "gxe_gtc(" : o2 == "<=" ? "gxe_lec("
                                     : o2 == ">=" ? "gxe_gec(" : "gxe_eqc(") + X + ", " + C + ")";
      }
      if (anyf && emu_op(kNativeCompare)) {
        const std::string X2 = asDB(x), Y2 = asDB(y), o2 = opstr;
        if (o2 == "<") return "(u64)gxe_lt(" + X2 + ", " + Y2 + ")";
        if (o2 == ">") return "(u64)gxe_lt(" + Y2 + ", " + X2 + ")";
        if (o2 == "<=") return "(u64)gxe_le(" + X2 + ", " + Y2 + ")";
        if (o2 == ">=") return "(u64)gxe_le(" + Y2 + ", " + X2 + ")";
        if (o2 == "==") return "(u64)gxe_eq(" + X2 + ", " + Y2 + ")";
        return "(u64)(!gxe_eq(" + X2 + ", " + Y2 + "))";
      }
      if (anyf) return std::string("(u64)(") + asD(x) + " " + opstr + " " + asD(y) + ")";
      return std::string("(u64)((i64)(") + X + ") " + opstr + " (i64)(" + Y + "))";
    };
    switch (op) {
      case OP_AND: r = "(u64)(" + nz(x) + " && " + nz(y) + ")"; break;
      case OP_ADD:
        r = !anyf ? "(" + X + " + " + Y + ")"
            : emu_op(kNativeAddSub) ? "gxe_add(" + asDB(x) + ", " + asDB(y) + ")" : "gx_B(" + asD(x) + " + " + asD(y) + ")";
        break;
      case OP_SUB:
        r = !anyf ? "(" + X + " - " + Y + ")"
            : emu_op(kNativeAddSub) ? "gxe_sub(" + asDB(x) + ", " + asDB(y) + ")" : "gx_B(" + asD(x) + " - " + asD(y) + ")";
        break;
      case OP_MUL:
        r = !anyf ? "(" + X + " * " + Y + ")"
            : emu_op(kNativeMul) ? "gxe_mul(" + asDB(x) + ", " + asDB(y) + ")" : "gx_B(" + asD(x) + " * " + asD(y) + ")";
        break;
      case OP_DIV:
        if (anyf && emu_op(kNativeDiv) && const_divisor(y) && !emu_op(kNativeConstDiv)) {
          // the FMA unit's correctly rounded constant division, the integer
          // pipes' form outside its exponent window
          const uint64_t db = literal_double_bits(y);
          double bd, yd;
          std::memcpy(&bd, &db, 8);
          yd = 1.0 / bd;
          uint64_t yb;
          std::memcpy(&yb, &yd, 8);
          int lo = 0, hi = 0;
          gxe_div_c_window((int)((db >> 52) & 0x7FF), &lo, &hi);
          r = "gxe_div_c(" + asDB(x) + ", " + hex64(db) + ", " + hex64(gxe_recip_fixed((db & GXE_FRAC) | GXE_HIDDEN)) +
              ", " + hex64(yb) + ", " + std::to_string(lo) + ", " + std::to_string(hi) + ")";
        } else if (small_div(id)) {  // an integer divisor: RN(1/|k|) from the table for small |k|
          const std::string k = "(i64)(" + B(int_source(y)) + "), gx_rcp_, GX_RCP_N)";
          if (!emu_op(kNativeIntDiv)) r = "gxe_div_small(" + asDB(x) + ", " + k;
          else if (int_source(x) >= 0) r = "gxe_divi_k((i64)(" + B(int_source(x)) + "), " + k;
          else r = "gxe_div_k(" + asDB(x) + ", " + k;
        } else if (anyf && emu_op(kNativeDiv) && const_divisor(y)) {
          // constant divisor: its reciprocal is computed here
          const uint64_t db = literal_double_bits(y);
          const std::string c = hex64(db) + ", " + hex64(gxe_recip_floor((db & GXE_FRAC) | GXE_HIDDEN)) + ")";
          r = int_source(x) >= 0 ? "gxe_divi_lit((i64)(" + B(int_source(x)) + "), " + c : "gxe_div_lit(" + asDB(x) + ", " + c;
        } else {
          r = !anyf ? "gx_div_ii(" + X + ", " + Y + ")"
              : emu_op(kNativeDiv) ? "gxe_div(" + asDB(x) + ", " + asDB(y) + ")" : "gx_B(" + asD(x) + " / " + asD(y) + ")";
        }
        if (const_divisor(y)) break;  // never zero
        if (rf && emu() && int_source(y) >= 0) vv = "(" + vv + " && (i64)(" + B(int_source(y)) + ") != 0LL)";
        else vv = "(" + vv + " && " + (rf ? nz(y) : "(i64)(" + Y + ") != 0LL") + ")";
        break;
      case OP_MOD:
        if (anyf) {
          r = "gx_B(fmod(" + asD(x) + ", " + asD(y) + "))";
        } else if (int_bits(x) <= 31 && int_bits(y) <= 31) {  // 32-bit remainder
          r = "gx_mod_32((int)(" + X + "), (int)(" + Y + "))";
          vv = "(" + vv + " && (i64)(" + Y + ") != 0LL)";
        } else {
          r = "gx_mod_ii(" + X + ", " + Y + ")";
          vv = "(" + vv + " && (i64)(" + Y + ") != 0LL)";
        }
        break;
      case OP_POW: r = "gx_B(pow(" + asD(x) + ", " + asD(y) + "))"; break;
      case OP_ROUND: {
        // a literal integral digit count of at most 22: the scale is the
        // literal 10^d, the rounding and the division stay on the integer pipes
        const double d = p_.nodes[y].kind == Node::LIT && p_.nodes[y].lit_valid ? bits_double(literal_double_bits(y)) : 99.0;
        if (emu_op(kNativeDiv) && emu_op(kNativeRound) && d >= -22.0 && d <= 22.0 && d == std::floor(d)) {
          const std::string f = "1e" + std::to_string((int)d);
          const double fv = std::strtod(f.c_str(), nullptr);
          uint64_t fb;
          std::memcpy(&fb, &fv, 8);
          r = "gxe_div_lit(gxe_round(gx_B(" + asD(x) + " * gx_D(" + hex64(fb) + "))), " + hex64(fb) + ", " +
              hex64(gxe_recip_floor((fb & GXE_FRAC) | GXE_HIDDEN)) + ")";
        } else {
          r = "gx_B(gx_round_to(" + asD(x) + ", " + asD(y) + "))";
        }
        break;
      }
      case OP_EQ: r = cmp("=="); break;
      case OP_NE: r = cmp("!="); break;
      case OP_LT: r = cmp("<"); break;
      case OP_GT: r = cmp(">"); break;
      case OP_LE: r = cmp("<="); break;
      case OP_GE: r = cmp(">="); break;
      default: fail(GX_ERR_UNSUPPORTED, "no code for binary operator");
    }
    if (n.exact_null) {
      o << ind << v << " = " << vv << ";\n";
      o << ind << b << " = " << v << " ? " << r << " : 0ull;\n";
    } else {
      o << ind << b << " = " << r << ";\n" << ind << v << " = " << vv << ";\n";
    }
  }

  // ids of OP / COL nodes reachable from roots, ascending (topological)
  std::vector<int> cone(const std::vector<int>& roots) const {
    std::set<int> seen;
    std::function<void(int)> go = [&](int id) {
      if (id < 0 || seen.count(id)) return;
      seen.insert(id);
      const Node& n = p_.nodes[id];
      if (n.kind == Node::OP) { go(n.a); go(n.b); }
    };
    for (int r : roots) go(r);
    std::vector<int> v;
    for (int id : seen)
      if (p_.nodes[id].kind != Node::LIT) v.push_back(id);
    return v;
  }

  void decl(std::ostringstream& o, const std::vector<int>& ids, const std::string& ind) const {
    for (int id : ids) o << ind << "u64 b" << id << "[GX_V]; bool v" << id << "[GX_V];\n";
  }

  // keep expression of conjunct c (index into p_.conjuncts) for slot k
  std::string conj_keep(int cid) const {
    if (cid < 0) return "true";
    const Node& n = p_.nodes[cid];
    if (n.kind == Node::LIT) return (n.lit_valid && n.lit_bits != 0) ? "inr" : "false";
    if (p_.conjuncts.size() == 1 && cid == p_.predicate)  // the root itself: BOOL8 column semantics
      return "(" + V(cid) + " && " + B(cid) + " != 0ull)";
    return "(" + V(cid) + " && " + nz(cid) + ")";
  }

  // Evaluates nodes `ids` for the warp's GX_V words: first a loop issuing every
  // column load of every word (so the loads are in flight together), then a
  // loop computing the operators and `tail` (a statement per word).  `inr` is
  // the per-row condition that loads are predicated on.
  void emit_words(std::ostringstream& o, const std::vector<int>& ids, const std::string& ind, const std::string& inr,
                  const std::string& tail) const {
    const std::string rowdef =
        tile_mode_ ? "const u32 trow = (u32)(wl0 + k) * 32u + (u32)lane; const i64 row = tb0 + (i64)trow; "
                     "const bool inr = " + inr + "; (void)inr; (void)row;\n"
                   : "const i64 row = (w0 + k) * 32 + lane; const bool inr = " + inr + "; (void)inr;\n";
    bool any_col = false;
    for (int id : ids) any_col |= p_.nodes[id].kind == Node::COL;
    const Masks was = masks_;
    if (!tile_mode_) {
      masks_ = Masks::WORDS;
      emit_mask_words(o, ids, {}, ind);
    }
    if (any_col) {
      o << ind << "#pragma unroll\n" << ind << "for (int k = 0; k < GX_V; k++) {\n" << ind << "  " << rowdef;
      for (int id : ids)
        if (p_.nodes[id].kind == Node::COL) emit_node(o, id, ind + "  ");
      o << ind << "}\n";
    }
    o << ind << "#pragma unroll\n" << ind << "for (int k = 0; k < GX_V; k++) {\n" << ind << "  " << rowdef;
    for (int id : ids)
      if (p_.nodes[id].kind != Node::COL) emit_node(o, id, ind + "  ");
    if (!tail.empty()) o << ind << "  " << tail << "\n";
    o << ind << "}\n";
    masks_ = was;
  }

  // predicate phase: fills keep bits bal[k]; with short-circuit, conjuncts are
  // evaluated in cfg order and later conjuncts skipped for all-dead warps
  void emit_predicate(std::ostringstream& o, const std::string& ind) const {
    std::vector<int> order;
    if (!cfg_.conjunct_order.empty()) {
      for (int i : cfg_.conjunct_order) order.push_back(p_.conjuncts.at(i));
    } else {
      order = p_.conjuncts;
    }
    o << ind << "bool alive[GX_V];\n";
    if (!tile_mode_)  // rows of the warp's words that exist, 0 .. 32 GX_V
      o << ind << "const int nrow_ = (int)max(min(a.n - w0 * 32, (i64)(GX_V * 32)), (i64)0);\n";
    o << ind << "#pragma unroll\n" << ind << "for (int k = 0; k < GX_V; k++) alive[k] = "
      << (tile_mode_ ? "(w0 + k) * 32 + lane < a.n" : "k * 32 + lane < nrow_") << ";\n";
    if (cfg_.runtime_order) {
      if (cfg_.stream_slots > 0 && streamable())
        emit_predicate_stream(o, ind);
      else
        emit_predicate_runtime_order(o, ind);
      return;
    }
    std::set<int> done;
    if (!cfg_.short_circuit) {
      // fixed order: evaluate every conjunct for every row
      std::string keep = "inr";
      for (int c : order) keep += " && " + conj_keep(c);
      emit_words(o, cone(order), ind, tile_mode_ ? "row < a.n" : "k * 32 + lane < nrow_", "alive[k] = " + keep + ";");
      return;
    }
    o << ind << "bool any_alive = true;\n";
    for (size_t j = 0; j < order.size(); j++) {
      std::vector<int> ids;
      for (int id : cone({order[j]}))
        if (!done.count(id)) ids.push_back(id);
      // loads predicated on the row being alive, issued for all words before
      // the ballots
      o << ind << "if (any_alive) {\n";
      emit_words(o, ids, ind + "  ", "alive[k]", "alive[k] = alive[k] && " + conj_keep(order[j]) + ";");
      o << ind << "  u32 any_ = 0;\n";
      o << ind << "  #pragma unroll\n" << ind << "  for (int k = 0; k < GX_V; k++) any_ |= __ballot_sync(GX_FULL, alive[k]);\n";
      o << ind << "  any_alive = any_ != 0u;\n";
      o << ind << "}\n";
      for (int id : ids) done.insert(id);
    }
  }

  // Short-circuit evaluation in the order a.order[] given at launch: one
  // warp-uniform switch per conjunct, each case evaluating its conjunct's whole
  // cone (no value crosses conjuncts) for the warp's GX_V words.  Column loads
  // are predicated on the row still being alive, so sectors whose rows all
  // died are not read; the words' loads are issued together (no ballot between
  // them), and the warp stops once none of its rows is alive.
  void emit_predicate_runtime_order(std::ostringstream& o, const std::string& ind) const {
    const int nc = (int)p_.conjuncts.size();
    o << ind << "u32 live_[GX_V];\n";
    o << ind << "#pragma unroll\n" << ind << "for (int k = 0; k < GX_V; k++) live_[k] = __ballot_sync(GX_FULL, alive[k]);\n";
    o << ind << "for (int j_ = 0; j_ < " << nc << "; j_++) {\n";
    o << ind << "  bool keep_[GX_V];\n";
    o << ind << "  switch (a.order_dev ? __ldg(a.order_dev + j_) : a.order[j_]) {\n";
    for (int c = 0; c < nc; c++) {
      const int cid = p_.conjuncts[c];
      o << ind << "    case " << c << ": {\n";
      std::vector<int> ids = cone({cid});
      decl(o, ids, ind + "      ");
      emit_words(o, ids, ind + "      ", "alive[k]", "keep_[k] = " + conj_keep(cid) + ";");
      o << ind << "      break; }\n";
    }
    o << ind << "    default:\n";
    o << ind << "      #pragma unroll\n" << ind << "      for (int k = 0; k < GX_V; k++) keep_[k] = false;\n";
    o << ind << "  }\n";
    o << ind << "  u32 any_ = 0u;\n";
    o << ind << "  #pragma unroll\n" << ind << "  for (int k = 0; k < GX_V; k++) {\n";
    o << ind << "    alive[k] = alive[k] && keep_[k];\n";
    o << ind << "    live_[k] = __ballot_sync(GX_FULL, alive[k]);\n";
    o << ind << "    any_ |= live_[k];\n";
    o << ind << "  }\n";
    o << ind << "  if (any_ == 0u) break;\n";
    o << ind << "}\n";
  }

  // every conjunct reads exactly one column (or none)
  bool streamable() const {
    for (size_t c = 0; c < p_.conjuncts.size(); c++)
      if (conjunct_columns(p_, (int)c).size() > 1) return false;
    return true;
  }

  // Streaming short-circuit in the launch order: the warp keeps S word slots in
  // flight, each at its own conjunct step; a slot whose word has no live row
  // left, or has passed every conjunct, takes the warp's next word.  Each round
  // issues the loads of every slot before evaluating any, so the warp always has
  // S words' loads outstanding instead of a shrinking lockstep set, and the
  // number of dependent load rounds is about (words x steps per word) / S
  // rather than the longest chain per group of words.  Word masks live in shared
  // memory (indexed by a slot's word).
  void emit_predicate_stream(std::ostringstream& o, const std::string& ind) const {
    const int nc = (int)p_.conjuncts.size();
    const int S = cfg_.stream_slots;
    std::vector<int> col_of(nc, -1);
    for (int c = 0; c < nc; c++) {
      const std::vector<int> cols = conjunct_columns(p_, c);
      if (!cols.empty()) col_of[c] = cols[0];
    }
    const std::string S_ = std::to_string(S);
    o << ind << "__shared__ u32 s_aw_[GX_WARPS][GX_V];\n";
    o << ind << "#pragma unroll\n" << ind << "for (int k = 0; k < GX_V; k++) {\n";
    o << ind << "  const u32 m_ = __ballot_sync(GX_FULL, alive[k]);\n";
    o << ind << "  if (lane == 0) s_aw_[warp][k] = m_;\n";
    o << ind << "}\n";
    o << ind << "__syncwarp();\n";
    o << ind << "int sw_[" << S_ << "], sj_[" << S_ << "]; u64 val_[" << S_ << "]; bool vv_[" << S_ << "];\n";
    o << ind << "int nx_ = 0;\n";
    o << ind << "#pragma unroll\n" << ind << "for (int q = 0; q < " << S_ << "; q++) {\n";
    o << ind << "  sw_[q] = -1; sj_[q] = 0; val_[q] = 0ull; vv_[q] = false;\n";
    o << ind << "  while (nx_ < GX_V && s_aw_[warp][nx_] == 0u) nx_++;\n";
    o << ind << "  if (nx_ < GX_V) { sw_[q] = nx_; nx_++; }\n";
    o << ind << "}\n";
    o << ind << "while (true) {\n";
    o << ind << "  bool act_ = false;\n";
    o << ind << "  #pragma unroll\n" << ind << "  for (int q = 0; q < " << S_ << "; q++) act_ |= sw_[q] >= 0;\n";
    o << ind << "  if (!act_) break;\n";
    // loads of every slot
    o << ind << "  #pragma unroll\n" << ind << "  for (int q = 0; q < " << S_ << "; q++) {\n";
    o << ind << "    if (sw_[q] < 0) continue;\n";
    o << ind << "    const int wk_ = sw_[q];\n";
    o << ind << "    const i64 row = (w0 + wk_) * 32 + lane;\n";
    o << ind << "    const bool inr = ((s_aw_[warp][wk_] >> lane) & 1u) != 0u;\n";
    o << ind << "    switch (a.order_dev ? __ldg(a.order_dev + sj_[q]) : a.order[sj_[q]]) {\n";
    for (int c = 0; c < nc; c++) {
      const int col = col_of[c];
      if (col < 0) continue;
      const std::string gfn = emu() ? load_fn_emu(p_.schema[col]) : load_fn(p_.schema[col]);
      o << ind << "      case " << c << ": val_[q] = inr ? (u64)" << gfn << "(a.in_data[" << col
        << "], row) : 0ull; vv_[q] = inr" << (p_.nullable[col] ? " && gx_valid(a.in_mask[" + std::to_string(col) +
                                                                      "], a.in_off[" + std::to_string(col) + "] + row)"
                                                                : std::string())
        << "; break;\n";
    }
    o << ind << "      default: break;\n    }\n";
    o << ind << "  }\n";
    // evaluation, mask update, refill
    o << ind << "  #pragma unroll\n" << ind << "  for (int q = 0; q < " << S_ << "; q++) {\n";
    o << ind << "    if (sw_[q] < 0) continue;\n";
    o << ind << "    const int wk_ = sw_[q];\n";
    o << ind << "    const i64 row = (w0 + wk_) * 32 + lane; (void)row;\n";
    o << ind << "    const bool inr = ((s_aw_[warp][wk_] >> lane) & 1u) != 0u;\n";
    o << ind << "    const int k = 0;\n";
    o << ind << "    bool keep_ = false;\n";
    o << ind << "    switch (a.order_dev ? __ldg(a.order_dev + sj_[q]) : a.order[sj_[q]]) {\n";
    for (int c = 0; c < nc; c++) {
      const int cid = p_.conjuncts[c];
      o << ind << "      case " << c << ": {\n";
      const std::vector<int> ids = cone({cid});
      for (int id : ids) o << ind << "        u64 b" << id << "[1]; bool v" << id << "[1];\n";
      for (int id : ids) {
        if (p_.nodes[id].kind == Node::COL)
          o << ind << "        b" << id << "[0] = val_[q]; v" << id << "[0] = vv_[q];\n";
      }
      for (int id : ids)
        if (p_.nodes[id].kind != Node::COL) emit_node(o, id, ind + "        ");
      o << ind << "        keep_ = " << conj_keep(cid) << ";\n";
      o << ind << "        break; }\n";
    }
    o << ind << "      default: break;\n    }\n";
    o << ind << "    const u32 m_ = s_aw_[warp][wk_] & __ballot_sync(GX_FULL, inr && keep_);\n";
    o << ind << "    __syncwarp();\n";
    o << ind << "    if (lane == 0) s_aw_[warp][wk_] = m_;\n";
    o << ind << "    __syncwarp();\n";
    o << ind << "    sj_[q]++;\n";
    o << ind << "    if (m_ == 0u || sj_[q] >= " << nc << ") {\n";
    o << ind << "      sw_[q] = -1; sj_[q] = 0;\n";
    o << ind << "      while (nx_ < GX_V && s_aw_[warp][nx_] == 0u) nx_++;\n";
    o << ind << "      if (nx_ < GX_V) { sw_[q] = nx_; nx_++; }\n";
    o << ind << "    }\n";
    o << ind << "  }\n";
    o << ind << "}\n";
    o << ind << "#pragma unroll\n" << ind << "for (int k = 0; k < GX_V; k++) alive[k] = ((s_aw_[warp][k] >> lane) & 1u) != 0u;\n";
    o << ind << "__syncwarp();\n";  // s_aw_ is rewritten by the warp's next tile
  }

  // per-conjunct pass counts of this warp's rows, accumulated in shared memory
  void emit_conj_stats(std::ostringstream& o, const std::string& ind) const {
    const int nc = (int)p_.conjuncts.size();
    o << ind << "#pragma unroll\n" << ind << "for (int k = 0; k < GX_V; k++) {\n";
    o << ind << "  const i64 row = (w0 + k) * 32 + lane; const bool inr = row < a.n; (void)inr;\n";
    for (int c = 0; c < nc; c++) {
      o << ind << "  { const u32 b_ = __ballot_sync(GX_FULL, inr && " << conj_keep(p_.conjuncts[c]) << ");\n";
      o << ind << "    if (lane == 0) atomicAdd(&s_conj[" << c << "], (unsigned long long)__popc(b_)); }\n";
    }
    o << ind << "}\n";
  }

  std::vector<int> predicate_cone() const { return p_.has_filter() ? cone(p_.conjuncts) : std::vector<int>{}; }

  // ids of OP / COL nodes reachable from roots without descending below the
  // nodes in `stop` (which are included themselves), ascending
  std::vector<int> cone_stop(const std::vector<int>& roots, const std::set<int>& stop) const {
    std::set<int> seen;
    std::function<void(int)> go = [&](int id) {
      if (id < 0 || seen.count(id)) return;
      seen.insert(id);
      const Node& n = p_.nodes[id];
      if (n.kind == Node::OP && !stop.count(id)) { go(n.a); go(n.b); }
    };
    for (int r : roots) go(r);
    std::vector<int> v;
    for (int id : seen)
      if (p_.nodes[id].kind != Node::LIT) v.push_back(id);
    return v;
  }

  // A CASE branch (the value operand of a MAGIC_IF_NOT) whose subtree is used
  // by nothing else, reads only columns and literals, and is expensive
  // (transcendentals, divisions): the dense phase evaluates it only for the
  // kept rows whose condition selects it, packed into full warps.  Rows whose
  // condition is false take the magic value whatever the branch computes, so
  // skipping them changes no result.
  struct Lazy {
    int consumer = -1;  // the MAGIC_IF_NOT node
    int cond = -1;      // its condition operand
    int root = -1;      // the branch value operand
    std::vector<int> nodes;  // OP and COL nodes of the branch, ascending
  };

  static int op_cost(Op op) {
    switch (op) {
      case OP_LN: case OP_LOG10: case OP_EXP: case OP_POW: case OP_SIN: case OP_COS: case OP_TAN: case OP_ASIN:
      case OP_ACOS: case OP_ATAN: case OP_COTAN:
        return 64;
      case OP_DIV: case OP_MOD: case OP_ROUND:
        return 16;
      default:
        return 1;
    }
  }

  std::vector<Lazy> lazy_branches(const std::vector<int>& roots) const {
    std::vector<Lazy> out;
    if (!cfg_.lazy_case) return out;
    const std::vector<int> all = cone(roots);
    std::map<int, std::vector<int>> users;
    for (int id : all) {
      const Node& n = p_.nodes[id];
      if (n.kind != Node::OP) continue;
      if (n.a >= 0) users[n.a].push_back(id);
      if (n.b >= 0 && n.b != n.a) users[n.b].push_back(id);
    }
    const std::set<int> external(roots.begin(), roots.end());
    std::set<int> taken;
    // outermost consumers first (a parent's id is above its operands')
    for (auto it = all.rbegin(); it != all.rend(); ++it) {
      const int m = *it;
      const Node& mn = p_.nodes[m];
      if (mn.kind != Node::OP || mn.op != OP_MAGIC_IF_NOT || taken.count(m)) continue;
      const int y = mn.b;
      if (y < 0 || p_.nodes[y].kind != Node::OP || external.count(y) || taken.count(y)) continue;
      if (users[y].size() != 1 || users[y][0] != m) continue;
      const std::vector<int> ycone = cone({y});
      std::set<int> S{y};
      for (bool grown = true; grown;) {
        grown = false;
        for (int id : ycone) {
          if (S.count(id) || p_.nodes[id].kind != Node::OP || external.count(id)) continue;
          bool excl = true;
          for (int u : users[id])
            if (!S.count(u)) { excl = false; break; }
          if (excl) { S.insert(id); grown = true; }
        }
      }
      bool ok = true;
      int cost = 0;
      for (int id : ycone) {
        const Node& n = p_.nodes[id];
        if (n.kind != Node::OP) continue;
        if (!S.count(id) || taken.count(id)) { ok = false; break; }
        cost += op_cost(n.op);
      }
      if (!ok || cost < 32) continue;
      Lazy lz;
      lz.consumer = m;
      lz.cond = mn.a;
      lz.root = y;
      lz.nodes = ycone;
      for (int id : ycone)
        if (p_.nodes[id].kind == Node::OP) taken.insert(id);
      out.push_back(lz);
    }
    return out;
  }

  std::vector<int> output_roots() const {
    std::vector<int> r;
    for (const auto& o : p_.outputs)
      if (o.kind == OutSpec::NODE) r.push_back(o.node);
    return r;
  }

  const Plan& p_;
  const KernelConfig& cfg_;
  // columns read from a shared-memory staging buffer: col -> (buffer, index)
  mutable std::map<int, std::pair<std::string, std::string>> staged_;
  // tile-staged kernels: every column is read from the tile's shared-memory
  // stage (row trow of the tile; see emit_fused_tma)
  mutable bool tile_mode_ = false;
  // columns whose data both the predicate and the projections read: loaded
  // with the default cache policy so the projections' re-read hits L2
  mutable std::set<int> reread_cols_;
  std::set<int> proven_;  // columns valid in every kept row (prove_valid)

  // validity of node id is true for every row the filter keeps (no NULL can
  // arise): non-nullable columns, columns the condition proves valid, valid literals, and operators that propagate only
  // their operands' validity or divide by a nonzero literal
  bool never_null(int id) const {
    const Node& n = p_.nodes[id];
    if (n.kind == Node::LIT) return n.lit_valid;
    if (n.kind == Node::COL) return !p_.nullable[n.col] || proven_.count(n.col);
    switch (n.op) {
      case OP_RAND: case OP_ROW_INDEX:
      case OP_IS_NOT_TRUE: case OP_IS_NOT_FALSE: case OP_IS_NULL: case OP_IS_NOT_NULL: case OP_IS_NOT_DISTINCT_FROM:
        return true;
      case OP_MAGIC_IF_NOT: return false;
      default: break;
    }
    if (op_is_unary(n.op)) return never_null(n.a);
    if (!never_null(n.a) || !never_null(n.b)) return false;
    if (n.op == OP_DIV || (n.op == OP_MOD && !kind_f(n.a) && !kind_f(n.b))) {
      const Node& d = p_.nodes[n.b];
      return d.kind == Node::LIT && d.lit_valid && (d.lit_bits & 0x7fffffffffffffffull) != 0;
    }
    return true;
  }
};

void emit_prelude(std::ostringstream& o, const KernelConfig& cfg) {
  o << "#define GX_V " << cfg.words << "\n#define GX_WARPS " << cfg.warps << "\n";
  // a register cap becomes a resident-block count in the launch bounds; without
  // one the bounds name the block size only (a minimum of one block lets ptxas
  // take more registers than its default choice)
  if (cfg.max_regs > 0)
    o << "#define GX_LB __launch_bounds__(GX_WARPS * 32, "
      << std::max(1, 65536 / (cfg.max_regs * cfg.warps * 32)) << ")\n";
  else
    o << "#define GX_LB __launch_bounds__(GX_WARPS * 32)\n";
  o << "#define GX_TILE_WORDS (GX_WARPS * GX_V)\n";
  o << "#define GX_MAX_COLS " << GX_MAX_COLS << "\n#define GX_MAX_OUTS " << GX_MAX_OUTS << "\n";
  o << "struct GxArgs {\n"
       "  const void* in_data[GX_MAX_COLS]; const u32* in_mask[GX_MAX_COLS]; i64 in_off[GX_MAX_COLS];\n"
       "  void* out_data[GX_MAX_OUTS]; u32* out_mask[GX_MAX_OUTS];\n"
       "  i64 n; i64 capacity; u64* tile_status; unsigned long long* tile_counter; unsigned long long* out_count;\n"
       "  int* err; u64 seed; unsigned long long* conj_counts; int order[16]; const int* order_dev;\n"
       "  u32 spin_limit;\n};\n"
       // polls a bounded wait makes before it gives up (0: the default)
       "#define GX_SPINS (a.spin_limit ? a.spin_limit : (1u << 22))\n";
}

// phase 2 of the filter kernels: projections for the kept rows of each word,
// written at positions pos.. (warp-uniform), plus validity bit streams.
// Stores output j for the current lane (dense rounds) and returns its validity
// expression for the round's ballot ("" for a broadcast output, filled after
// the launch).
std::string emit_dense_store(std::ostringstream& o, const Gen& g, const Plan& p, size_t j, const std::string& ind) {
  const OutSpec& os = p.outputs[j];
  if (os.kind == OutSpec::NODE) {
    o << ind << "if (wr) " << store_stmt(os.type, "a.out_data[" + std::to_string(j) + "]", "orow", g.B(os.node)) << "\n";
    return g.V(os.node);
  }
  if (os.kind != OutSpec::COPY) return "";
  const int c = os.col;
  const std::string rt = raw_type(p.schema[c]);
  o << ind << "if (wr) __stcs((" << rt << "*)a.out_data[" << j << "] + orow, r" << j << "_);\n";
  return g.col_valid(c);
}

// outputs that carry a validity bit stream (broadcasts are filled after the launch)
std::vector<size_t> masked_outputs(const Plan& p) {
  std::vector<size_t> v;
  for (size_t j = 0; j < p.outputs.size(); j++)
    if (p.outputs[j].kind != OutSpec::BROADCAST) v.push_back(j);
  return v;
}

// The warp's kept rows in order, from its keep masks `bal`: offsets from its
// first row, listed in `list` (GX_V * 32 entries of shared memory) by kept rank;
// declares and counts `total`.
void emit_kept_list(std::ostringstream& o, const std::string& bal, const std::string& list, const std::string& total,
                    const std::string& ind) {
  o << ind << "#pragma unroll\n" << ind << "for (int kk = 0; kk < GX_V; kk++) {\n";
  o << ind << "  if ((" << bal << "[kk] >> lane) & 1u) " << list << "[" << total << " + __popc(" << bal
    << "[kk] & ((1u << lane) - 1u))] = (unsigned short)(kk * 32 + lane);\n";
  o << ind << "  " << total << " += __popc(" << bal << "[kk]);\n";
  o << ind << "}\n";
}

// statements mapping kept rank t_ of the warp (0 <= t_ < total_) to its row
// through the warp's kept-row list kl_ in shared memory
void emit_rank_to_row(std::ostringstream& o, const std::string& ind) {
  o << ind << "const u32 kp_ = act ? (u32)kl_[t_] : 0u; const i64 row = w0 * 32 + kp_; const bool inr = act; (void)inr;\n";
  o << ind << "const i64 orow = (i64)pos + (i64)t_; (void)orow;\n";
  o << ind << "const int k = 0;\n";
}

// nodes ids for one row per lane: gathers first, then operators; lazy branch
// roots (lz_root -> index) are read from the branch results in shared memory
void emit_row_nodes(std::ostringstream& o, const Gen& g, const Plan& p, const std::vector<int>& ids,
                    const std::map<int, int>& lz_root, const std::string& ind) {
  g.decl(o, ids, ind);
  for (int id : ids)
    if (p.nodes[id].kind == Node::COL) g.emit_node(o, id, ind);
  for (int id : ids) {
    if (p.nodes[id].kind == Node::COL) continue;
    auto it = lz_root.find(id);
    if (it != lz_root.end()) {
      o << ind << "b" << id << "[k] = s_lzb_[" << it->second << "][warp][t_]; v" << id << "[k] = s_lzv_["
        << it->second << "][warp][t_] != 0;\n";
    } else {
      g.emit_node(o, id, ind);
    }
  }
}

// Dense phase 2: the warp's kept rows, in row order, are dealt to lanes in
// rounds of 32 (lane l of round r takes the warp's (32r + l)-th kept row), so
// projections are computed only for surviving rows and every output store and
// validity word of a round is contiguous.  Operands are re-read with the
// gathered row index (predicate columns hit L1/L2).  Expensive CASE branches
// (Gen::lazy_branches) are first evaluated for the kept rows whose condition
// selects them, packed into full warps, into shared memory.
//
// What bounds it is instructions and load latency (order-line plan, ncu: IPC
// 1.7, 340 instructions per 32 rows, most of them addresses and validity).  So
// a round keeps both small: columns share one row index (bind_column folds the
// view's offset into the pointers); validity comes by shuffle from words that
// the warp's lanes loaded once per tile, and not at all for columns that the
// condition proves valid; output validity bits stay in lane r until the warp
// has done its rounds, then go out one coalesced store per mask instead of one
// lane's store per mask and round.  340 -> 285 instructions, call time at 2^27
// rows 2.43 -> 2.08 ms; deep plan 2^26 1.70 -> 1.47; process_filter of six
// columns 2^23 0.346 -> 0.274.
// The list kl_ of the warp's total_ kept rows is made here from bal[], unless the
// caller has made it (`listed`).
void emit_filter_writes_dense(std::ostringstream& o, const Gen& g, const Plan& p, const std::string& ind,
                              bool listed = false) {
  const std::vector<int> roots = g.output_roots();
  const std::vector<Gen::Lazy> lz = g.lazy_branches(roots);
  std::map<int, int> lz_root;
  std::set<int> stop;
  for (size_t i = 0; i < lz.size(); i++) {
    lz_root[lz[i].root] = (int)i;
    stop.insert(lz[i].root);
  }
  const std::vector<int> proj = g.cone_stop(roots, stop);
  const Gen::Masks was = g.masks_;
  g.masks_ = Gen::Masks::KEPT;
  {
    std::vector<int> copied;
    for (const auto& os : p.outputs)
      if (os.kind == OutSpec::COPY) copied.push_back(os.col);
    g.emit_mask_words(o, g.cone(roots), copied, ind);
  }
  if (!listed) {
    o << ind << "__shared__ unsigned short s_kept_[GX_WARPS][GX_V * 32];\n";
    o << ind << "unsigned short* const kl_ = s_kept_[warp];\n";
    o << ind << "u32 total_ = 0u;\n";
    emit_kept_list(o, "bal", "kl_", "total_", ind);
    o << ind << "__syncwarp();\n";
  }
  if (!lz.empty()) {
    const int nl = (int)lz.size();
    o << ind << "__shared__ u64 s_lzb_[" << nl << "][GX_WARPS][GX_V * 32];\n";
    o << ind << "__shared__ unsigned char s_lzv_[" << nl << "][GX_WARPS][GX_V * 32];\n";
    // pass 1: which kept rows select each branch
    std::vector<int> conds;
    for (const auto& l : lz) conds.push_back(l.cond);
    const std::vector<int> cond_ids = g.cone(conds);
    o << ind << "u32 dmd_[" << nl << "][GX_V];\n";
    o << ind << "__shared__ unsigned short s_dem_[GX_WARPS][GX_V * 32];\n";
    o << ind << "#pragma unroll\n" << ind << "for (int r_ = 0; r_ < GX_V; r_++) {\n";
    const std::string i2 = ind + "  ";
    o << i2 << "#pragma unroll\n" << i2 << "for (int l_ = 0; l_ < " << nl << "; l_++) dmd_[l_][r_] = 0u;\n";
    o << i2 << "if ((u32)r_ * 32u < total_) {\n";
    const std::string i3 = i2 + "  ";
    o << i3 << "const u32 t_ = (u32)r_ * 32u + (u32)lane; const bool act = t_ < total_;\n";
    emit_rank_to_row(o, i3);
    emit_row_nodes(o, g, p, cond_ids, {}, i3);
    for (int i = 0; i < nl; i++) {
      const int c = lz[i].cond;
      o << i3 << "dmd_[" << i << "][r_] = __ballot_sync(GX_FULL, act && (" << g.V(c) << " && " << g.nz(c) << "));\n";
    }
    o << i2 << "}\n";
    o << ind << "}\n";
    // pass 2: each branch over its selecting rows, 32 at a time
    for (int i = 0; i < nl; i++) {
      o << ind << "{\n";
      // the kept ranks selecting branch i, in order, listed in shared memory
      o << i2 << "u32 dtot_ = 0u;\n";
      o << i2 << "#pragma unroll\n" << i2 << "for (int r_ = 0; r_ < GX_V; r_++) {\n";
      o << i2 << "  const u32 db_ = dmd_[" << i << "][r_];\n";
      o << i2 << "  if ((db_ >> lane) & 1u) s_dem_[warp][dtot_ + __popc(db_ & ((1u << lane) - 1u))] = (unsigned short)(r_ * 32 + lane);\n";
      o << i2 << "  dtot_ += __popc(db_);\n";
      o << i2 << "}\n";
      o << i2 << "__syncwarp();\n";
      o << i2 << "for (u32 db_ = 0; db_ < dtot_; db_ += 32u) {\n";
      o << i3 << "const u32 q_ = db_ + (u32)lane; const bool act = q_ < dtot_;\n";
      o << i3 << "const u32 t_ = act ? (u32)s_dem_[warp][q_] : 0u;\n";
      emit_rank_to_row(o, i3);
      emit_row_nodes(o, g, p, lz[i].nodes, {}, i3);
      o << i3 << "if (act) { s_lzb_[" << i << "][warp][t_] = " << g.B(lz[i].root) << "; s_lzv_[" << i
        << "][warp][t_] = " << g.V(lz[i].root) << " ? 1 : 0; }\n";
      o << i2 << "}\n";
      o << i2 << "__syncwarp();\n";  // s_dem_ is rewritten for the next branch
      o << ind << "}\n";
    }
    o << ind << "__syncwarp();\n";
  }
  // validity bits: lane r keeps round r's ballot of each output whose validity
  // varies (outputs that are never NULL need none), and the warp writes every
  // mask once, after its rounds (gx_put_bits)
  const std::vector<size_t> mo = masked_outputs(p);
  std::vector<int> slot(p.outputs.size(), -1);
  int nslots = 0;
  for (size_t j : mo) {
    const OutSpec& os = p.outputs[j];
    if (os.kind == OutSpec::COPY ? g.masked(os.col) : !g.never_null(os.node)) slot[j] = nslots++;
  }
  if (!g.lane_words()) o << ind << "const i64 cap_words = (a.capacity + 31) >> 5;\n";
  else
    for (int sl = 0; sl < nslots; sl++) o << ind << "u32 vb" << sl << "_ = 0u;\n";
  o << ind << "const u32 wmax_ = (u32)max((i64)0, min((i64)total_, a.capacity - (i64)pos));\n";
  o << ind << "for (u32 base_ = 0; base_ < total_; base_ += 32u) {\n";
  const std::string in2 = ind + "  ";
  o << in2 << "const u32 t_ = base_ + (u32)lane; const bool act = t_ < total_;\n";
  emit_rank_to_row(o, in2);
  // the copied columns' loads go out with the projections'
  for (size_t j = 0; j < p.outputs.size(); j++) {
    if (p.outputs[j].kind != OutSpec::COPY) continue;
    const int c = p.outputs[j].col;
    const std::string rt = raw_type(p.schema[c]);
    o << in2 << "const " << rt << " r" << j << "_ = act ? __ldg((const " << rt << "*)a.in_data[" << c << "] + row) : ("
      << rt << ")0;\n";
  }
  emit_row_nodes(o, g, p, proj, lz_root, in2);
  o << in2 << "const bool wr = t_ < wmax_;\n";
  for (size_t j = 0; j < p.outputs.size(); j++) {
    const std::string v = emit_dense_store(o, g, p, j, in2);
    if (slot[j] < 0) continue;
    o << in2 << "{ const u32 b_ = __ballot_sync(GX_FULL, " << v << " && act); ";
    if (g.lane_words())
      o << "if ((u32)lane == base_ >> 5) vb" << slot[j] << "_ = b_; }\n";
    else  // more rounds than lanes: each round writes its own bits
      o << "gx_put_bits(a.out_mask[" << j << "], (i64)pos + base_, min(32u, total_ - base_), lane == 0 ? b_ : 0u, cap_words); }\n";
  }
  o << ind << "}\n";
  o << ind << "__syncwarp();\n";  // the kept-row list and branch results are rewritten by the next tile
  if (g.lane_words()) o << ind << "const i64 cap_words = (a.capacity + 31) >> 5;\n";
  for (size_t j : mo) {
    if (slot[j] >= 0 && g.lane_words())
      o << ind << "gx_put_bits(a.out_mask[" << j << "], (i64)pos, total_, vb" << slot[j] << "_, cap_words);\n";
    else if (slot[j] < 0 && !listed)  // else the block writes its tile's (emit_tile_ones)
      o << ind << "gx_put_ones(a.out_mask[" << j << "], (i64)pos, total_, cap_words);\n";
  }
  g.masks_ = was;
}

// The validity bits of the outputs that are never NULL, for a whole tile: its
// rows' bits are all ones from the tile's base on, so the block's warps share
// the masks out, one warp per mask.
void emit_tile_ones(std::ostringstream& o, const Gen& g, const Plan& p, const std::string& base, const std::string& total,
                    const std::string& ind) {
  const Gen::Masks was = g.masks_;
  g.masks_ = Gen::Masks::KEPT;
  int i = 0;
  for (size_t j : masked_outputs(p)) {
    const OutSpec& os = p.outputs[j];
    if (os.kind == OutSpec::COPY ? g.masked(os.col) : !g.never_null(os.node)) continue;
    o << ind << "if (warp == " << i++ << " % GX_WARPS) gx_put_ones(a.out_mask[" << j << "], (i64)" << base << ", " << total
      << ", (a.capacity + 31) >> 5);\n";
  }
  g.masks_ = was;
}

void emit_filter_writes(std::ostringstream& o, const Gen& g, const Plan& p, const std::vector<int>& pred_ids,
                        const std::string& ind) {
  if (g.cfg_.dense) {
    emit_filter_writes_dense(o, g, p, ind);
    return;
  }
  std::vector<int> proj = g.cone(g.output_roots());
  std::set<int> have(pred_ids.begin(), pred_ids.end());
  std::vector<int> fresh;
  for (int id : proj)
    if (!have.count(id)) fresh.push_back(id);
  g.decl(o, fresh, ind);
  o << ind << "GxBitWriter bw_[" << p.outputs.size() << "];\n";
  o << ind << "#pragma unroll\n" << ind << "for (int j = 0; j < " << p.outputs.size() << "; j++) bw_[j].init((i64)pos);\n";
  o << ind << "const i64 cap_words = (a.capacity + 31) >> 5;\n";
  o << ind << "#pragma unroll\n" << ind << "for (int k = 0; k < GX_V; k++) {\n";
  o << ind << "  const u32 bk = bal[k];\n";
  o << ind << "  if (bk == 0u) continue;\n";
  o << ind << "  const i64 row = (w0 + k) * 32 + lane; const bool inr = row < a.n; (void)inr;\n";
  o << ind << "  const bool keep = (bk >> lane) & 1u;\n";
  o << ind << "  const i64 orow = (i64)pos + __popc(bk & ((1u << lane) - 1u)); (void)orow;\n";
  for (int id : fresh) g.emit_node(o, id, ind + "  ");
  o << ind << "  const bool wr = keep && orow < a.capacity;\n";
  o << ind << "  const int nb = __popc(bk);\n";
  o << ind << "  const int q = (int)(orow - (i64)pos);\n";
  for (size_t j = 0; j < p.outputs.size(); j++) {
    const OutSpec& os = p.outputs[j];
    std::string vexpr;
    if (os.kind == OutSpec::NODE) {
      o << ind << "  if (wr) " << store_stmt(os.type, "a.out_data[" + std::to_string(j) + "]", "orow", g.B(os.node))
        << "\n";
      vexpr = g.V(os.node);
    } else if (os.kind == OutSpec::COPY) {
      const int c = os.col;
      const std::string rt = raw_type(p.schema[c]);
      o << ind << "  if (wr) ((" << rt << "*)a.out_data[" << j << "])[orow] = __ldcs((const " << rt << "*)a.in_data[" << c
        << "] + row);\n";
      vexpr = p.nullable[c] ? "gx_valid(a.in_mask[" + std::to_string(c) + "], a.in_off[" + std::to_string(c) + "] + row)"
                            : "true";
    } else {
      continue;  // broadcast outputs are filled after the launch
    }
    o << ind << "  { const u32 vb_ = __reduce_or_sync(GX_FULL, (keep && " << vexpr << ") ? (1u << (q & 31)) : 0u);\n";
    o << ind << "    if (bw_[" << j << "].word < cap_words) bw_[" << j << "].append(a.out_mask[" << j
      << "], vb_, nb); else { bw_[" << j << "].fill = 0; } }\n";
  }
  o << ind << "  pos += (u64)nb;\n";
  o << ind << "}\n";
  for (size_t j = 0; j < p.outputs.size(); j++) {
    if (p.outputs[j].kind == OutSpec::BROADCAST) continue;
    o << ind << "if (bw_[" << j << "].word < cap_words) bw_[" << j << "].flush(a.out_mask[" << j << "]);\n";
  }
}

// The tile pipeline's kept-row lists, in shared memory: one of each tile in
// flight, made with the tile's predicate.  A block whose rows (or expensive CASE
// branches) leave no room for two of them in the 227 KB that it may have keeps the
// next tile's keep masks, a 16th of the size, and lists them when it writes.
struct KeptLists {
  bool two = true;
  KeptLists(const Gen& g) {
    const size_t rows = (size_t)g.cfg_.warps * g.cfg_.words * 32, branches = g.lazy_branches(g.output_roots()).size();
    const size_t others = (size_t)g.cfg_.warps * (24 + 4 * g.cfg_.words) + 256;  // counts, offsets, the tile's words
    two = rows * (4 + (branches ? 2 : 0) + 9 * branches) + others <= 227 * 1024;
  }
  void decl(std::ostringstream& o) const {
    o << "  __shared__ unsigned short s_kept_[" << (two ? 2 : 1) << "][GX_WARPS][GX_V * 32];\n";
    if (!two) o << "  __shared__ u32 s_bal_[2][GX_WARPS][GX_V];\n";
  }
  // keeps the warp's rows of bal[] for tile slot `buf`, counting them in `cnt`
  void keep(std::ostringstream& o, const std::string& buf, const std::string& cnt, const std::string& ind) const {
    if (two) return emit_kept_list(o, "bal", "s_kept_[" + buf + "][warp]", cnt, ind);
    o << ind << "#pragma unroll\n" << ind << "for (int kk = 0; kk < GX_V; kk++) {\n";
    o << ind << "  if (lane == 0) s_bal_[" << buf << "][warp][kk] = bal[kk];\n" << ind << "  " << cnt
      << " += __popc(bal[kk]);\n" << ind << "}\n";
    o << ind << "__syncwarp();\n";
  }
  // kl_ and total_ of the tile in slot par
  void list(std::ostringstream& o, const std::string& ind) const {
    if (!two) {
      o << ind << "u32 listed_ = 0u; u32 wb_[GX_V];\n";
      o << ind << "#pragma unroll\n" << ind << "for (int kk = 0; kk < GX_V; kk++) wb_[kk] = s_bal_[par][warp][kk];\n";
      emit_kept_list(o, "wb_", "s_kept_[0][warp]", "listed_", ind);
      o << ind << "__syncwarp();\n";
    }
    o << ind << "const unsigned short* const kl_ = s_kept_[" << (two ? "par" : "0") << "][warp]; const u32 total_ = wcnt;\n";
  }
};

// Fused single-pass filter (dense projections) as a two-stage tile pipeline:
// a block evaluates tile t+1's predicate before it resolves tile t's output
// offset by look-back, so the look-back of t waits on tiles that had a whole
// tile's time to publish, and the next tile's loads are in flight meanwhile.
// Between the stages tile t is its warps' kept-row lists in shared memory
// (dense projections recompute outputs from the gathered rows).
//
// The block is bound by what its warps wait for, so they wait for little: the
// ticket of tile t+2 is drawn while t+1 is evaluated (an atomic's round trip to
// L2 otherwise starts every tile), warps other than the first only announce
// their counts (bar.arrive) and go on, and meet the first one once per tile,
// when the offset is known.  No deadlock: the block that holds the first
// unpublished tile waits at most for earlier tiles, all of them published, so
// it comes to evaluate and publish it.
void emit_fused_pipelined(std::ostringstream& o, const Gen& g, const Plan& p, const std::vector<int>& pred_ids) {
  // with conj_stats (fixed order, every conjunct evaluated for every row): each
  // conjunct's passing rows, counted per warp in registers and added to
  // a.conj_counts once per warp at the end
  const bool stats = g.cfg_.conj_stats && !g.cfg_.runtime_order && !g.cfg_.short_circuit;
  const int nc = (int)p.conjuncts.size();
  auto count_conjuncts = [&](const std::string& ind) {
    if (!stats) return;
    o << ind << "#pragma unroll\n" << ind << "for (int k = 0; k < GX_V; k++) {\n";
    o << ind << "  const i64 row = (w0 + k) * 32 + lane; const bool inr = row < a.n; (void)inr;\n";
    for (int c = 0; c < nc; c++)
      o << ind << "  cst_[" << c << "] += (u32)__popc(__ballot_sync(GX_FULL, inr && " << g.conj_keep(p.conjuncts[c])
        << "));\n";
    o << ind << "}\n";
  };
  if (stats) o << "  u32 cst_[" << nc << "] = {};\n";
  o << "  __shared__ unsigned long long s_claim;\n";
  o << "  __shared__ u32 s_cnt[2][GX_WARPS];\n";
  o << "  __shared__ u64 s_off[2][GX_WARPS];\n";
  o << "  __shared__ u64 s_base, s_total;\n";
  const KeptLists kept(g);
  kept.decl(o);
  o << "  const i64 ntiles = (nwords + GX_TILE_WORDS - 1) / GX_TILE_WORDS;\n";
  o << "  if (threadIdx.x == 0) s_claim = atomicAdd(a.tile_counter, 1ull);\n";
  o << "  __syncthreads();\n";
  o << "  i64 tile = (i64)s_claim;\n";
  o << "  if (tile >= ntiles) return;\n";
  o << "  __syncthreads();\n";  // s_claim is rewritten below
  o << "  u32 wcnt = 0u; int par = 0; u64 ptotal = 0ull; unsigned long long ahead_ = 0ull;\n";
  o << "  i64 known_ = -1; u64 known_incl_ = 0ull;\n";  // the block's last resolved tile and its inclusive prefix
  o << "  if (threadIdx.x == 0) ahead_ = atomicAdd(a.tile_counter, 1ull);\n";
  o << "  {\n";
  o << "    const i64 w0 = tile * GX_TILE_WORDS + (i64)warp * GX_V;\n";
  auto predicate = [&](const std::string& buf, const std::string& cnt, const std::string& ind) {
    g.decl(o, pred_ids, ind);
    g.emit_predicate(o, ind);
    count_conjuncts(ind);
    o << ind << "u32 bal[GX_V];\n";
    o << ind << "#pragma unroll\n" << ind << "for (int k = 0; k < GX_V; k++) bal[k] = __ballot_sync(GX_FULL, alive[k]);\n";
    kept.keep(o, buf, cnt, ind);
    o << ind << "if (lane == 0) s_cnt[" << buf << "][warp] = " << cnt << ";\n";
  };
  predicate("0", "wcnt", "    ");
  o << "  }\n";
  o << "  if (threadIdx.x == 0) s_claim = ahead_;\n";
  o << "  __syncthreads();\n";
  o << "  if (warp == 0) ptotal = gx_tile_publish(a.tile_status, tile, s_cnt[0], s_off[0], GX_WARPS);\n";
  o << "  while (true) {\n";
  o << "    const i64 next = (i64)s_claim;\n";
  o << "    if (threadIdx.x == 0 && next < ntiles) ahead_ = atomicAdd(a.tile_counter, 1ull);\n";
  o << "    const int npar = par ^ 1;\n";
  o << "    u32 nwcnt = 0u;\n";
  o << "    if (next < ntiles) {\n";
  o << "      const i64 w0 = next * GX_TILE_WORDS + (i64)warp * GX_V;\n";
  predicate("npar", "nwcnt", "      ");
  o << "    }\n";
  o << "    gx_bar_counts(warp, GX_WARPS);\n";  // the first warp waits for every warp's count
  o << "    if (warp == 0) {\n";
  o << "      u64 ntotal = 0ull;\n";
  o << "      if (next < ntiles) ntotal = gx_tile_publish(a.tile_status, next, s_cnt[npar], s_off[npar], GX_WARPS);\n";
  o << "      const u64 excl = gx_lookback_resolve(a.tile_status, tile, ptotal, a.err, GX_SPINS, known_, known_incl_);\n";
  o << "      if (lane == 0) {\n";
  o << "        s_base = excl; s_total = ptotal; s_claim = ahead_;\n";
  o << "        if (tile == ntiles - 1 && excl != ~0ull) *a.out_count = excl + ptotal;\n";
  o << "      }\n";
  o << "      known_ = tile; known_incl_ = excl + ptotal;\n";
  o << "      ptotal = ntotal;\n";
  o << "    }\n";
  o << "    __syncthreads();\n";
  o << "    const u64 base_t = s_base;\n";
  o << "    if (base_t == ~0ull) break;\n";  // look-back gave up: error already recorded
  emit_tile_ones(o, g, p, "base_t", "s_total", "    ");
  o << "    if (wcnt != 0u) {\n";
  o << "      u64 pos = base_t + s_off[par][warp];\n";
  o << "      const i64 w0 = tile * GX_TILE_WORDS + (i64)warp * GX_V;\n";
  kept.list(o, "      ");
  emit_filter_writes_dense(o, g, p, "      ", true);
  o << "    }\n";
  o << "    if (next >= ntiles) break;\n";
  o << "    tile = next; par = npar; wcnt = nwcnt;\n";
  o << "  }\n";
  if (stats) {
    o << "  if (lane == 0) {\n";
    for (int c = 0; c < nc; c++)
      o << "    if (cst_[" << c << "]) atomicAdd(&a.conj_counts[" << c << "], (unsigned long long)cst_[" << c << "]);\n";
    o << "  }\n";
  }
  o << "}\n";
}

// Columns read by the predicate and the outputs (COPY outputs included), ascending.
std::vector<int> referenced_columns(const Plan& p) {
  std::set<int> cols, seen;
  std::function<void(int)> go = [&](int id) {
    if (id < 0 || seen.count(id)) return;
    seen.insert(id);
    const Node& n = p.nodes[id];
    if (n.kind == Node::COL) cols.insert(n.col);
    if (n.kind == Node::OP) { go(n.a); go(n.b); }
  };
  if (p.has_filter()) go(p.predicate);
  for (const auto& os : p.outputs) {
    if (os.kind == OutSpec::NODE) go(os.node);
    if (os.kind == OutSpec::COPY) cols.insert(os.col);
  }
  return std::vector<int>(cols.begin(), cols.end());
}

// Store of an output value into its shared-memory staging slot at byte
// offset `off`, with the conversion store_stmt applies to a global store.
std::string sstore_stmt(int t, const std::string& off, const std::string& bits) {
  const std::string at = "(gx_smem + " + off + ")";
  switch (t) {
    case BOOL8: return "*(unsigned char*)" + at + " = (unsigned char)((" + bits + ") != 0ull);";
    case INT8: case UINT8: return "*(unsigned char*)" + at + " = (unsigned char)(" + bits + ");";
    case INT16: case UINT16: return "*(unsigned short*)" + at + " = (unsigned short)(" + bits + ");";
    case INT32: case UINT32: case TIMESTAMP_DAYS: case DURATION_DAYS:
      return "*(unsigned*)" + at + " = (unsigned)(" + bits + ");";
    case FLOAT32: return "*(float*)" + at + " = (float)gx_D(" + bits + ");";
    default: return "*(u64*)" + at + " = (" + bits + ");";
  }
}

// kept rank t_ of the consumer warp -> its tile row, and its rank tk_ among
// the tile's kept rows
void emit_ws_rank_row(std::ostringstream& o, const std::string& in) {
  o << in << "const u32 trow = act ? (u32)s_kept_w[warp][t_] : 0u; const i64 row = tb0 + (i64)trow; const bool inr = act;"
             " (void)row; (void)inr;\n";
  o << in << "const u32 tk_ = woff + t_; (void)tk_;\n";
  o << in << "const int k = 0;\n";
}

// Projections of one consumer warp's kept rows of a tile (wcnt rows, tile
// rows in s_kept_w[warp]), computed in rounds of 32 and staged in shared
// memory at the rows' tile-level kept ranks (woff + rank): data in the output's
// slot, validity as one byte per row.  Expensive CASE branches are first
// evaluated for the warp's kept rows whose condition selects them, packed into
// full rounds (per-warp lists, no block barrier).
void emit_ws_dense(std::ostringstream& o, const Gen& g, const Plan& p, const TileLayout& L, const std::string& ind) {
  const std::vector<int> roots = g.output_roots();
  const std::vector<Gen::Lazy> lz = g.lazy_branches(roots);
  std::map<int, int> lz_root;
  std::set<int> stop;
  for (size_t i = 0; i < lz.size(); i++) {
    lz_root[lz[i].root] = (int)i;
    stop.insert(lz[i].root);
  }
  const std::vector<int> proj = g.cone_stop(roots, stop);
  const std::string i2 = ind + "  ", i3 = i2 + "  ";
  if (!lz.empty()) {
    const int nl = (int)lz.size();
    std::vector<int> conds;
    for (const auto& l : lz) conds.push_back(l.cond);
    const std::vector<int> cond_ids = g.cone(conds);
    o << ind << "u32 dmd_[" << nl << "][GX_V];\n";
    o << ind << "#pragma unroll\n" << ind << "for (int r_ = 0; r_ < GX_V; r_++) {\n";
    o << i2 << "#pragma unroll\n" << i2 << "for (int l_ = 0; l_ < " << nl << "; l_++) dmd_[l_][r_] = 0u;\n";
    o << i2 << "if ((u32)r_ * 32u < wcnt) {\n";
    o << i3 << "const u32 t_ = (u32)r_ * 32u + (u32)lane; const bool act = t_ < wcnt;\n";
    emit_ws_rank_row(o, i3);
    emit_row_nodes(o, g, p, cond_ids, {}, i3);
    for (int i = 0; i < nl; i++) {
      const int c = lz[i].cond;
      o << i3 << "dmd_[" << i << "][r_] = __ballot_sync(GX_FULL, act && (" << g.V(c) << " && " << g.nz(c) << "));\n";
    }
    o << i2 << "}\n";
    o << ind << "}\n";
    for (int i = 0; i < nl; i++) {
      o << ind << "{\n";
      o << i2 << "u32 dtot_ = 0u;\n";
      o << i2 << "#pragma unroll\n" << i2 << "for (int r_ = 0; r_ < GX_V; r_++) {\n";
      o << i3 << "const u32 db_ = dmd_[" << i << "][r_];\n";
      o << i3 << "if ((db_ >> lane) & 1u) s_dem_[warp][dtot_ + __popc(db_ & ((1u << lane) - 1u))] = "
                 "(unsigned short)(r_ * 32 + lane);\n";
      o << i3 << "dtot_ += __popc(db_);\n";
      o << i2 << "}\n";
      o << i2 << "__syncwarp();\n";
      o << i2 << "for (u32 db_ = 0; db_ < dtot_; db_ += 32u) {\n";
      o << i3 << "const u32 q_ = db_ + (u32)lane; const bool act = q_ < dtot_;\n";
      o << i3 << "const u32 t_ = act ? (u32)s_dem_[warp][q_] : 0u;\n";
      emit_ws_rank_row(o, i3);
      emit_row_nodes(o, g, p, lz[i].nodes, {}, i3);
      o << i3 << "if (act) { s_lzb_[" << i << "][warp][t_] = " << g.B(lz[i].root) << "; s_lzv_[" << i
        << "][warp][t_] = " << g.V(lz[i].root) << " ? 1 : 0; }\n";
      o << i2 << "}\n";
      o << i2 << "__syncwarp();\n";  // s_dem_ is rewritten for the next branch
      o << ind << "}\n";
    }
  }
  o << ind << "for (u32 base_ = 0; base_ < wcnt; base_ += 32u) {\n";
  o << i2 << "const u32 t_ = base_ + (u32)lane; const bool act = t_ < wcnt;\n";
  emit_ws_rank_row(o, i2);
  emit_row_nodes(o, g, p, proj, lz_root, i2);
  for (size_t j = 0; j < p.outputs.size(); j++) {
    const OutSpec& os = p.outputs[j];
    if (os.kind == OutSpec::BROADCAST) continue;
    const std::string w = std::to_string(L.out_width[j]);
    const std::string doff = "ost + " + std::to_string(L.out_off[j]) + "u + tk_ * " + w + "u";
    const std::string voff = "ost + " + std::to_string(L.out_valid_off[j]) + "u + tk_";
    if (os.kind == OutSpec::NODE) {
      o << i2 << "if (act) { " << sstore_stmt(os.type, doff, g.B(os.node)) << " gx_smem[" << voff << "] = "
        << g.V(os.node) << " ? 1 : 0; }\n";
    } else {
      const int c = os.col;
      const std::string cs = std::to_string(c), rt = raw_type(p.schema[c]);
      const std::string vexpr = p.nullable[c] ? "((vmw_" + cs + "[trow >> 5] >> (trow & 31u)) & 1u)" : "1u";
      o << i2 << "if (act) { *(" << rt << "*)(gx_smem + " << doff << ") = *(const " << rt << "*)(gx_smem + sd_" << cs
        << " + trow * " << w << "u); gx_smem[" << voff << "] = (unsigned char)" << vexpr << "; }\n";
    }
  }
  o << ind << "}\n";
}

// Write-out of a tile's staged outputs (K_w rows at output rows base_w..) by
// every consumer warp: data element by element (coalesced), validity words
// rebuilt from the staged bytes by ballots; the first and last words of the
// tile's range may be shared with the neighbouring tiles and are OR-ed in
// atomically (the masks were zeroed before the launch).
void emit_ws_writeout(std::ostringstream& o, const Plan& p, const TileLayout& L, const std::string& ind) {
  const std::string i2 = ind + "  ";
  o << ind << "const u32 tid_ = (u32)warp * 32u + (u32)lane;\n";
  for (size_t j = 0; j < p.outputs.size(); j++) {
    if (p.outputs[j].kind == OutSpec::BROADCAST) continue;
    const std::string rt = raw_type(p.outputs[j].kind == OutSpec::COPY ? p.schema[p.outputs[j].col] : p.outputs[j].type);
    o << ind << "for (u32 t = tid_; t < K_w; t += GX_WARPS * 32u) {\n";
    o << i2 << "const i64 orow = (i64)base_w + (i64)t;\n";
    o << i2 << "if (orow < a.capacity) __stcs((" << rt << "*)a.out_data[" << j << "] + orow, *(const " << rt
      << "*)(gx_smem + osw + " << L.out_off[j] << "u + t * " << L.out_width[j] << "u));\n";
    o << ind << "}\n";
  }
  o << ind << "const u32 bf_ = (u32)(base_w & 31ull); const u32 nw_ = K_w ? (bf_ + K_w + 31u) >> 5 : 0u;\n";
  o << ind << "const i64 w0_ = (i64)(base_w >> 5); const i64 cap_words = (a.capacity + 31) >> 5;\n";
  o << ind << "for (u32 kw = (u32)warp; kw < nw_; kw += GX_WARPS) {\n";
  o << i2 << "const int t = (int)(kw * 32u + (u32)lane) - (int)bf_;\n";
  o << i2 << "const bool in_ = t >= 0 && (u32)t < K_w;\n";
  o << i2 << "const bool shared_ = (kw == 0u && bf_ != 0u) || kw + 1u == nw_;\n";
  for (size_t j = 0; j < p.outputs.size(); j++) {
    if (p.outputs[j].kind == OutSpec::BROADCAST) continue;
    o << i2 << "{ const u32 word_ = __ballot_sync(GX_FULL, in_ && gx_smem[osw + " << L.out_valid_off[j]
      << "u + (u32)(in_ ? t : 0)] != 0);\n";
    o << i2 << "  if (lane == 0 && w0_ + (i64)kw < cap_words) { if (shared_) atomicOr(a.out_mask[" << j
      << "] + w0_ + kw, word_); else a.out_mask[" << j << "][w0_ + kw] = word_; } }\n";
  }
  o << ind << "}\n";
}

// Tile-staged fused filter + project (single pass, stable order), with the
// warps of a block in three roles.
//
//  * warp 0 (producer): claims tiles in order from the ticket and, for each,
//    issues one bulk copy per column (its data bytes, and its mask words when
//    it has a mask) into the next free stage of a GX_NS-stage ring in shared
//    memory, completing on the stage's "full" mbarrier; it reuses a stage once
//    every consumer warp has arrived on the stage's "empty" mbarrier.
//  * warp 1 (resolver): for each tile, once the consumers have published its
//    aggregate and the block's next tile has been counted too, resolves its
//    output offset by decoupled look-back -- a 256-wide window per poll that
//    stops at the block's previous tile, whose inclusive prefix it already
//    has -- and hands it back through a "based" mbarrier.
//  * warps 2.. (consumers): slot j of their loop evaluates the predicate of
//    the block's j-th tile from shared memory (lane per row; the mask words are
//    first re-aligned to the tile's rows), lists each warp's kept rows, meets
//    at one named barrier to total the tile (one thread publishes the
//    aggregate and passes it to the resolver); then computes the projections
//    of the (j-1)-th tile's kept rows into a ring of shared-memory output
//    staging buffers and releases that tile's stage; then writes the
//    (j - GX_NR)-th tile's staged outputs to their final rows.
//
// A block thus publishes its newest aggregate before it waits on any
// look-back, and a tile's look-back waits only on earlier tiles, so the kernel
// cannot deadlock.  Every wait is bounded: a look-back that gives up records
// error 1 (the block goes on without writing that tile); a copy or hand-over
// wait that gives up records error 2, and the consumers wait (bounded) for the
// copies still in flight to land before the block returns.
void emit_fused_tma(std::ostringstream& o, const Gen& g, const Plan& p, const TileLayout& L, const std::string& name) {
  g.tile_mode_ = true;
  const std::vector<int> pred_ids = g.predicate_cone();
  const std::vector<Gen::Lazy> lz = g.lazy_branches(g.output_roots());
  const int nl = (int)lz.size();
  o << "#undef GX_LB\n#define GX_LB __launch_bounds__((GX_WARPS + 2) * 32)\n";
  o << "#define GX_TR " << L.tile_rows << "\n#define GX_NS " << L.stages << "\n#define GX_STAGE " << L.stage_bytes
    << "u\n#define GX_OBASE " << L.out_base << "u\n#define GX_OSTAGE " << L.out_stage_bytes << "u\n#define GX_NR "
    << L.out_stages << "\n#define GX_RR (GX_NR + 1)\n";
  o << "#define GX_WAIT (1u << 21)\n";
  // the copies of one tile into the stage at shared address stg
  o << "__device__ __forceinline__ void gx_issue_tile_(const GxArgs& a, long long t, u32 stg, u64* bar) {\n";
  o << "  const i64 r0 = (i64)t * GX_TR; const i64 r1 = min(a.n, r0 + (i64)GX_TR);\n";
  for (size_t i = 0; i < L.cols.size(); i++) {
    const int c = L.cols[i];
    const std::string cs = std::to_string(c), w = std::to_string(type_size(p.schema[c]));
    o << "  const u64 lo" << cs << " = (u64)a.in_data[" << cs << "] + (u64)r0 * " << w
      << "ull, hi" << cs << " = (u64)a.in_data[" << cs << "] + (u64)r1 * " << w << "ull;\n";
    if (L.mask_off[i] != UINT32_MAX)
      o << "  const u64 mlo" << cs << " = (u64)(a.in_mask[" << cs << "] + ((a.in_off[" << cs << "] + r0) >> 5)), mhi"
        << cs << " = (u64)(a.in_mask[" << cs << "] + ((a.in_off[" << cs << "] + r1 - 1) >> 5) + 1);\n";
  }
  o << "  u32 tot = 0u;\n";
  for (size_t i = 0; i < L.cols.size(); i++) {
    const std::string cs = std::to_string(L.cols[i]);
    o << "  tot += gx_bulk_span(0u, lo" << cs << ", hi" << cs << ", bar, false);\n";
    if (L.mask_off[i] != UINT32_MAX) o << "  tot += gx_bulk_span(0u, mlo" << cs << ", mhi" << cs << ", bar, false);\n";
  }
  o << "  gx_mbar_arrive_tx(bar, tot);\n";
  for (size_t i = 0; i < L.cols.size(); i++) {
    const std::string cs = std::to_string(L.cols[i]);
    o << "  gx_bulk_span(stg + " << L.data_off[i] << "u, lo" << cs << ", hi" << cs << ", bar, true);\n";
    if (L.mask_off[i] != UINT32_MAX)
      o << "  gx_bulk_span(stg + " << L.mask_off[i] << "u, mlo" << cs << ", mhi" << cs << ", bar, true);\n";
  }
  o << "}\n";

  o << "extern \"C\" __global__ void GX_LB " << name << "(const GxArgs a) {\n";
  o << "  const int lane = threadIdx.x & 31; const int wid_ = threadIdx.x >> 5;\n";
  o << "  const i64 ntiles = (a.n + GX_TR - 1) / GX_TR;\n";
  o << "  __shared__ __align__(8) u64 s_full_[GX_NS];\n";
  o << "  __shared__ __align__(8) u64 s_empty_[GX_NS];\n";
  o << "  __shared__ __align__(8) u64 s_counted_[GX_RR];\n";
  o << "  __shared__ __align__(8) u64 s_based_[GX_RR];\n";
  o << "  __shared__ long long s_tile_[GX_NS];\n";
  o << "  __shared__ long long s_rtile_[GX_RR];\n";
  o << "  __shared__ u64 s_ragg_[GX_RR];\n";
  o << "  __shared__ u64 s_base_[GX_RR];\n";
  o << "  __shared__ u32 s_cnt_[2][GX_WARPS];\n";
  o << "  __shared__ unsigned short s_kept_[2][GX_WARPS][GX_V * 32];\n";
  if (L.num_masked > 0) o << "  __shared__ u32 s_vm_[2][" << L.num_masked << "][GX_TR / 32];\n";
  if (nl > 0) {
    o << "  __shared__ unsigned short s_dem_[GX_WARPS][GX_V * 32];\n";
    o << "  __shared__ u64 s_lzb_[" << nl << "][GX_WARPS][GX_V * 32];\n";
    o << "  __shared__ unsigned char s_lzv_[" << nl << "][GX_WARPS][GX_V * 32];\n";
  }
  o << "  const u32 smem0_ = gx_saddr(gx_smem);\n";
  // bulk copies land on 16-byte boundaries of the dynamic shared memory
  o << "  if ((smem0_ & 15u) != 0u) { if (threadIdx.x == 0) gx_set_err(a.err, 3); return; }\n";
  o << "  if (threadIdx.x == 0) {\n";
  o << "    for (int q = 0; q < GX_NS; q++) { gx_mbar_init(&s_full_[q], 1u); gx_mbar_init(&s_empty_[q], GX_WARPS); }\n";
  o << "    for (int q = 0; q < GX_RR; q++) { gx_mbar_init(&s_counted_[q], 1u); gx_mbar_init(&s_based_[q], 1u); }\n";
  o << "    gx_mbar_init_fence();\n";
  o << "  }\n";
  o << "  __syncthreads();\n";
  // ---- producer
  o << "  if (wid_ == 0) {\n";
  o << "    if (lane == 0) {\n";
  o << "      for (int j = 0; ; j++) {\n";
  o << "        const int q = j % GX_NS;\n";
  o << "        if (j >= GX_NS && !gx_mbar_wait(&s_empty_[q], (u32)(j / GX_NS - 1) & 1u, GX_WAIT)) {\n";
  o << "          gx_set_err(a.err, 2);\n";
  o << "          break;\n";
  o << "        }\n";
  o << "        long long t = (long long)atomicAdd(a.tile_counter, 1ull);\n";
  o << "        if (t >= ntiles) t = -1;\n";
  o << "        s_tile_[q] = t;\n";
  o << "        if (t < 0) { gx_mbar_arrive(&s_full_[q]); break; }\n";
  o << "        gx_fence_async_smem();\n";
  o << "        gx_issue_tile_(a, t, smem0_ + (u32)q * GX_STAGE, &s_full_[q]);\n";
  o << "      }\n";
  o << "    }\n";
  o << "    return;\n";
  o << "  }\n";
  // ---- resolver
  o << "  if (wid_ == 1) {\n";
  o << "    long long tk = -1; u64 pk = 0ull;\n";  // the block's last resolved tile and its inclusive prefix
  o << "    for (int j = 0; ; j++) {\n";
  o << "      const int b = j % GX_RR;\n";
  o << "      if (!gx_mbar_wait(&s_counted_[b], (u32)(j / GX_RR) & 1u, GX_WAIT)) {\n";
  o << "        if (lane == 0) gx_set_err(a.err, 2);\n";
  o << "        return;\n";
  o << "      }\n";
  o << "      const long long t = s_rtile_[b]; const u64 agg = s_ragg_[b];\n";
  o << "      if (t < 0) return;\n";
  // start once the block's next tile is counted too: by then the tiles other
  // blocks claimed before this one have mostly published their aggregates
  o << "      gx_mbar_wait(&s_counted_[(j + 1) % GX_RR], (u32)((j + 1) / GX_RR) & 1u, GX_WAIT);\n";
  o << "      const u64 ex = gx_lookback_wide<8>(a.tile_status, t, agg, a.err, GX_SPINS, tk, pk);\n";
  o << "      if (ex != ~0ull) { tk = t; pk = ex + agg; } else { tk = -1; pk = 0ull; }\n";
  o << "      if (lane == 0) {\n";
  o << "        s_base_[b] = ex;\n";
  o << "        if (t == ntiles - 1 && ex != ~0ull) *a.out_count = ex + agg;\n";
  o << "        gx_mbar_arrive(&s_based_[b]);\n";
  o << "      }\n";
  o << "      __syncwarp();\n";
  o << "    }\n";
  o << "  }\n";
  // ---- consumers
  o << "  const int warp = wid_ - 2;\n";
  // per-column shifts: the byte of element 0 within its 16-byte block, and
  // for masks the byte of the first word within its block and the bit of row
  // 0 within that word -- the same for every tile (tiles are multiples of 128 rows)
  for (size_t i = 0; i < L.cols.size(); i++) {
    const int c = L.cols[i];
    const std::string cs = std::to_string(c);
    o << "  const u32 h_" << cs << " = (u32)((u64)a.in_data[" << cs << "] & 15ull);\n";
    if (L.mask_off[i] != UINT32_MAX) {
      o << "  const u32 mh_" << cs << " = (u32)((u64)(a.in_mask[" << cs << "] + (a.in_off[" << cs << "] >> 5)) & 15ull);\n";
      o << "  const u32 ms_" << cs << " = (u32)(a.in_off[" << cs << "] & 31);\n";
    }
  }
  o << "  long long tile_p = -1; u32 wcnt_p = 0u, woff_p = 0u;\n";  // the (j-1)-th tile, awaiting its projections
  o << "  for (int j = 0; ; j++) {\n";
  o << "    const int q = j % GX_NS; const int vp = j & 1; const int rr = j % GX_RR;\n";
  o << "    const bool ok_ = gx_mbar_wait(&s_full_[q], (u32)(j / GX_NS) & 1u, GX_WAIT);\n";
  o << "    const long long tile = ok_ ? s_tile_[q] : -1;\n";
  o << "    u32 wcnt = 0u;\n";
  o << "    if (tile >= 0) {\n";
  o << "      const i64 tb0 = (i64)tile * GX_TR; const int wl0 = warp * GX_V;\n";
  o << "      const u32 stg = (u32)q * GX_STAGE;\n";
  for (size_t i = 0; i < L.cols.size(); i++) {
    const std::string cs = std::to_string(L.cols[i]);
    o << "      const u32 sd_" << cs << " = stg + " << L.data_off[i] << "u + h_" << cs << "; (void)sd_" << cs << ";\n";
    if (L.mask_off[i] != UINT32_MAX) {
      o << "      const u32* vmw_" << cs << " = s_vm_[vp][" << L.mask_index[i] << "]; (void)vmw_" << cs << ";\n";
      o << "      if (lane < GX_V) {\n";
      o << "        const u32 wk_ = (u32)(wl0 + lane);\n";
      o << "        const u32* raw_ = (const u32*)(gx_smem + stg + " << L.mask_off[i] << "u + mh_" << cs << ");\n";
      o << "        s_vm_[vp][" << L.mask_index[i] << "][wk_] = __funnelshift_r(raw_[wk_], raw_[wk_ + 1], ms_" << cs
        << ");\n";
      o << "      }\n";
    }
  }
  o << "      __syncwarp();\n";
  o << "      const i64 w0 = (i64)tile * GX_TILE_WORDS + wl0;\n";
  g.decl(o, pred_ids, "      ");
  g.emit_predicate(o, "      ");
  o << "      u32 r_ = 0u;\n";
  o << "      #pragma unroll\n      for (int k = 0; k < GX_V; k++) {\n";
  o << "        const u32 bk_ = __ballot_sync(GX_FULL, alive[k]);\n";
  o << "        if ((bk_ >> lane) & 1u) s_kept_[vp][warp][r_ + __popc(bk_ & ((1u << lane) - 1u))] = "
       "(unsigned short)((wl0 + k) * 32 + lane);\n";
  o << "        r_ += __popc(bk_);\n";
  o << "      }\n";
  o << "      wcnt = r_;\n";
  o << "      __syncwarp();\n";
  o << "    }\n";
  o << "    if (lane == 0) s_cnt_[vp][warp] = wcnt;\n";
  o << "    if (!gx_bar_and(ok_, GX_WARPS * 32)) {\n";
  // a copy never landed: wait (bounded) for the copies in flight, then leave
  o << "      if (warp == 0 && lane == 0) gx_set_err(a.err, 2);\n";
  o << "      for (int d_ = 0; d_ < GX_NS; d_++) gx_mbar_wait(&s_full_[(j + d_) % GX_NS], (u32)((j + d_) / GX_NS) & 1u, "
       "GX_WAIT);\n";
  o << "      return;\n";
  o << "    }\n";
  o << "    u32 tot_ = 0u, woff = 0u;\n";
  o << "    if (tile >= 0) woff = gx_block_excl(s_cnt_[vp], GX_WARPS, &tot_, warp);\n";
  o << "    if (warp == 0 && lane == 0) {\n";
  o << "      if (tile >= 0) gx_st_status(a.tile_status + tile, (tile == 0 ? GX_ST_PFX : GX_ST_AGG) | (u64)tot_);\n";
  o << "      s_rtile_[rr] = tile; s_ragg_[rr] = (u64)tot_;\n";
  o << "      gx_mbar_arrive(&s_counted_[rr]);\n";
  o << "    }\n";
  // projections of the previous slot's tile
  o << "    if (tile_p >= 0) {\n";
  o << "      const int jp = j - 1; const int qp = jp % GX_NS; const int pp = jp & 1;\n";
  o << "      const u32 ost = GX_OBASE + (u32)(jp % GX_NR) * GX_OSTAGE;\n";
  o << "      const u32 wcnt = wcnt_p, woff = woff_p;\n";
  o << "      const i64 tb0 = (i64)tile_p * GX_TR;\n";
  o << "      const u32 stg = (u32)qp * GX_STAGE;\n";
  o << "      const unsigned short (*s_kept_w)[GX_V * 32] = s_kept_[pp];\n";
  for (size_t i = 0; i < L.cols.size(); i++) {
    const std::string cs = std::to_string(L.cols[i]);
    o << "      const u32 sd_" << cs << " = stg + " << L.data_off[i] << "u + h_" << cs << "; (void)sd_" << cs << ";\n";
    if (L.mask_off[i] != UINT32_MAX)
      o << "      const u32* vmw_" << cs << " = s_vm_[pp][" << L.mask_index[i] << "]; (void)vmw_" << cs << ";\n";
  }
  emit_ws_dense(o, g, p, L, "      ");
  o << "      __syncwarp();\n";
  o << "      if (lane == 0) gx_mbar_arrive(&s_empty_[qp]);\n";
  o << "    }\n";
  // after the last tile every staged tile is written out, the one just
  // projected included: all consumer warps must have staged it first
  o << "    if (tile < 0) gx_bar_and(true, GX_WARPS * 32);\n";
  o << "    for (int jw = j - GX_NR; jw <= (tile >= 0 ? j - GX_NR : j - 1); jw++) {\n";
  o << "      if (jw < 0) continue;\n";
  o << "      const int pr = jw % GX_RR;\n";
  o << "      if (s_rtile_[pr] < 0) continue;\n";
  o << "      const bool okb = gx_mbar_wait(&s_based_[pr], (u32)(jw / GX_RR) & 1u, GX_WAIT);\n";
  o << "      if (!okb && warp == 0 && lane == 0) gx_set_err(a.err, 2);\n";
  o << "      const u64 base_w = okb ? s_base_[pr] : ~0ull;\n";
  o << "      if (base_w != ~0ull) {\n";
  o << "        const u32 K_w = (u32)s_ragg_[pr]; const u32 osw = GX_OBASE + (u32)(jw % GX_NR) * GX_OSTAGE;\n";
  emit_ws_writeout(o, p, L, "        ");
  o << "      }\n";
  o << "    }\n";
  o << "    if (tile < 0) break;\n";
  o << "    tile_p = tile; wcnt_p = wcnt; woff_p = woff;\n";
  o << "  }\n";
  o << "}\n";
  g.tile_mode_ = false;
}

// Batched persistent form of the pipelined fused filter: one launch runs a
// whole table of batches (GxArgs per batch).  Batch b owns the tiles
// [tile_base[b], tile_base[b + 1]) of one tile sequence that blocks claim in
// order from one counter; every batch has its own look-back segment and row
// counter, so a block's pending and next tiles may belong to different
// batches, and each batch's result is exactly that of running it alone.
// (streaming: the host appends batches while the kernel runs -- descriptors,
// tile offsets, then the published tile count, each by an ordered copy -- and
// closes the queue by setting hdr->pad; a block that claims a tile past the
// published count waits for it (bounded: `wait_polls` polls 2 us apart, then
// *werr = 1) or, once the queue is closed without it, stops.  Tile offsets of
// unpublished batches hold INT64_MAX, so a lookup never passes the last
// published batch.)
void emit_fused_batched(std::ostringstream& o, const Gen& g, const Plan& p, const std::vector<int>& pred_ids,
                        const std::string& name, bool streaming = false) {
  o << "struct GxBatchHdr { unsigned long long tile_counter; long long total_tiles; int nbatch; int pad; };\n";
  // a batch's descriptor: streaming descriptors sit kArgsStride bytes apart,
  // so that no cache line holds two of them (one is written while the kernel
  // may have read its neighbour)
  if (streaming)
    o << "#define GX_BATCH(b) (*(const GxArgs*)((const char*)A + (size_t)(b) * " << kStreamArgsStride << "u))\n";
  else
    o << "#define GX_BATCH(b) (A[(b)])\n";
  if (streaming) {
    o << "extern \"C\" __global__ void GX_LB " << name
      << "(const GxArgs* A, const volatile long long* tile_base, GxBatchHdr* hdr, int* werr, unsigned wait_polls) {\n";
    o << "  const int nbatch = 0x7fffffff; (void)nbatch;\n";
    // claim a tile; -1 once the queue is closed below it (or the wait gave up)
    o << "  auto claim_ = [&]() -> long long {\n";
    o << "    long long t = (long long)atomicAdd(&hdr->tile_counter, 1ull);\n";
    o << "    unsigned polls = 0;\n";
    o << "    while (true) {\n";
    o << "      if (t < *(volatile long long*)&hdr->total_tiles) break;\n";
    o << "      if (*(volatile int*)&hdr->pad != 0) {\n";  // closed: the published count is final
    o << "        if (t < *(volatile long long*)&hdr->total_tiles) break;\n";
    o << "        return -1;\n";
    o << "      }\n";
    o << "      if (*(volatile int*)werr != 0) return -1;\n";
    o << "      if (++polls > wait_polls) { atomicExch(werr, 1); return -1; }\n";
    o << "      __nanosleep(2000);\n";
    o << "    }\n";
    o << "    __threadfence();\n";  // the batch's descriptor and tile offsets were copied before its tiles were published
    o << "    return t;\n";
    o << "  };\n";
  } else {
    o << "extern \"C\" __global__ void GX_LB " << name
      << "(const GxArgs* __restrict__ A, const long long* __restrict__ tile_base, GxBatchHdr* hdr) {\n";
    o << "  const i64 total_tiles = hdr->total_tiles; const int nbatch = hdr->nbatch;\n";
  }
  o << "  const int lane = threadIdx.x & 31; const int warp = threadIdx.x >> 5;\n";
  o << "  __shared__ unsigned long long s_claim;\n";
  o << "  __shared__ u32 s_cnt[2][GX_WARPS];\n";
  o << "  __shared__ u64 s_off[2][GX_WARPS];\n";
  o << "  __shared__ u64 s_base, s_total;\n";
  const KeptLists kept(g);
  kept.decl(o);
  // the batch of global tile gt, at or after batch b
  auto find = [&](const std::string& b, const std::string& gt, const std::string& ind) {
    if (streaming) o << ind << "while (" << b << " + 1 < nbatch && tile_base[" << b << " + 1] <= " << gt << ") " << b << "++;\n";
    else o << ind << b << " = gx_find_batch(tile_base, " << b << ", nbatch, " << gt << ");\n";
  };
  if (streaming) {
    o << "  if (threadIdx.x == 0) s_claim = (unsigned long long)claim_();\n";
    o << "  __syncthreads();\n";
    o << "  const i64 gt0 = (i64)s_claim;\n";
    o << "  if (gt0 < 0) return;\n";
  } else {
    o << "  if (threadIdx.x == 0) s_claim = atomicAdd(&hdr->tile_counter, 1ull);\n";
    o << "  __syncthreads();\n";
    o << "  const i64 gt0 = (i64)s_claim;\n";
    o << "  if (gt0 >= total_tiles) return;\n";
  }
  o << "  __syncthreads();\n";  // s_claim is rewritten below
  // the ticket after next is drawn ahead (as emit_fused_pipelined), but for a
  // queue that the host extends: there a claim may wait for the host
  if (!streaming) {
    o << "  unsigned long long ahead_ = 0ull;\n";
    o << "  if (threadIdx.x == 0) ahead_ = atomicAdd(&hdr->tile_counter, 1ull);\n";
  }
  o << "  int pb = 0;\n";
  find("pb", "gt0", "  ");
  o << "  i64 tile = gt0 - tile_base[pb];\n";
  o << "  u32 wcnt = 0u; int par = 0; u64 ptotal = 0ull;\n";
  o << "  i64 known_ = -1; u64 known_incl_ = 0ull;\n";  // the block's last resolved tile of this batch
  auto predicate = [&](const std::string& buf, const std::string& cnt, const std::string& ind) {
    g.decl(o, pred_ids, ind);
    g.emit_predicate(o, ind);
    o << ind << "u32 bal[GX_V];\n";
    o << ind << "#pragma unroll\n" << ind << "for (int k = 0; k < GX_V; k++) bal[k] = __ballot_sync(GX_FULL, alive[k]);\n";
    kept.keep(o, buf, cnt, ind);
    o << ind << "if (lane == 0) s_cnt[" << buf << "][warp] = " << cnt << ";\n";
  };
  o << "  {\n";
  o << "    const GxArgs& a = GX_BATCH(pb);\n";
  o << "    const i64 w0 = tile * GX_TILE_WORDS + (i64)warp * GX_V;\n";
  predicate("0", "wcnt", "    ");
  o << "  }\n";
  if (!streaming) o << "  if (threadIdx.x == 0) s_claim = ahead_;\n";
  o << "  __syncthreads();\n";
  o << "  if (warp == 0) ptotal = gx_tile_publish(GX_BATCH(pb).tile_status, tile, s_cnt[0], s_off[0], GX_WARPS);\n";
  o << "  while (true) {\n";
  if (streaming) {
    o << "    if (threadIdx.x == 0) s_claim = (unsigned long long)claim_();\n";
    o << "    __syncthreads();\n";
  }
  o << "    const i64 ngt = (i64)s_claim;\n";
  o << "    int nb = pb; i64 next = -1;\n";
  o << "    if (" << (streaming ? "ngt >= 0" : "ngt < total_tiles") << ") {\n";
  if (!streaming) o << "      if (threadIdx.x == 0) ahead_ = atomicAdd(&hdr->tile_counter, 1ull);\n";
  find("nb", "ngt", "      ");
  o << "      next = ngt - tile_base[nb];\n";
  o << "    }\n";
  o << "    const int npar = par ^ 1;\n";
  o << "    u32 nwcnt = 0u;\n";
  o << "    if (next >= 0) {\n";
  o << "      const GxArgs& a = GX_BATCH(nb);\n";
  o << "      const i64 w0 = next * GX_TILE_WORDS + (i64)warp * GX_V;\n";
  predicate("npar", "nwcnt", "      ");
  o << "    }\n";
  o << "    gx_bar_counts(warp, GX_WARPS);\n";
  o << "    if (warp == 0) {\n";
  o << "      u64 ntotal = 0ull;\n";
  o << "      if (next >= 0) ntotal = gx_tile_publish(GX_BATCH(nb).tile_status, next, s_cnt[npar], s_off[npar], GX_WARPS);\n";
  o << "      const GxArgs& a = GX_BATCH(pb);\n";
  o << "      const i64 ntiles = (((a.n + 31) >> 5) + GX_TILE_WORDS - 1) / GX_TILE_WORDS;\n";
  o << "      const u64 excl = gx_lookback_resolve(a.tile_status, tile, ptotal, a.err, GX_SPINS, known_, known_incl_);\n";
  o << "      if (lane == 0) {\n";
  o << "        s_base = excl; s_total = ptotal;" << (streaming ? "" : " s_claim = ahead_;") << "\n";
  o << "        if (tile == ntiles - 1 && excl != ~0ull) *a.out_count = excl + ptotal;\n";
  o << "      }\n";
  o << "      known_ = nb == pb ? tile : -1; known_incl_ = nb == pb ? excl + ptotal : 0ull;\n";
  o << "      ptotal = ntotal;\n";
  o << "    }\n";
  o << "    __syncthreads();\n";
  o << "    const u64 base_t = s_base;\n";
  o << "    if (base_t == ~0ull) break;\n";  // look-back gave up: error already recorded
  o << "    {\n      const GxArgs& a = GX_BATCH(pb);\n";
  emit_tile_ones(o, g, p, "base_t", "s_total", "      ");
  o << "    }\n";
  o << "    if (wcnt != 0u) {\n";
  o << "      const GxArgs& a = GX_BATCH(pb);\n";
  o << "      u64 pos = base_t + s_off[par][warp];\n";
  o << "      const i64 w0 = tile * GX_TILE_WORDS + (i64)warp * GX_V;\n";
  kept.list(o, "      ");
  emit_filter_writes_dense(o, g, p, "      ", true);
  o << "    }\n";
  o << "    if (next < 0) break;\n";
  o << "    tile = next; pb = nb; par = npar; wcnt = nwcnt;\n";
  o << "  }\n";
  o << "}\n";
}

// Staged short-circuit filter (runtime conjunct order, dense projections).
// Each block keeps GX_D tiles in flight.  A tile's conjuncts are evaluated one
// at a time in the launch order; before each step, warp 0 copies the 32-row
// words of that conjunct's columns that still have a live row into the tile's
// shared-memory slot with asynchronous copies (completion on the slot's
// mbarrier) and the block moves on to the next slot, so the copies of several
// tiles are in flight while it evaluates one.  (Bulk copies of one 256-byte
// word each were measured an order of magnitude slower than 16-byte
// asynchronous copies spread over the warp: small bulk copies serialise.)  A tile whose rows are all dead, or that has
// passed every conjunct, publishes its aggregate at once; tiles are resolved
// (look-back) and written in claim order, so a block never waits on one of its
// own unpublished tiles.  A partial last word is read from global memory
// directly.  Every column a conjunct reads must start on a 16-byte boundary
// (the host checks and otherwise runs the unstaged kernel).
void emit_staged_filter(std::ostringstream& o, const Gen& g, const Plan& p, const std::string& name) {
  const int nc = (int)p.conjuncts.size();
  std::vector<std::vector<int>> cc(nc);
  std::vector<std::vector<int>> coff(nc);  // byte offset of each column's region in a slot, per word
  std::vector<int> cwb(nc, 0);             // bytes per word of all the conjunct's columns
  int wbmax = 16;
  for (int c = 0; c < nc; c++) {
    cc[c] = conjunct_columns(p, c);
    for (int col : cc[c]) {
      coff[c].push_back(cwb[c]);
      cwb[c] += 32 * type_size(p.schema[col]);
    }
    wbmax = std::max(wbmax, cwb[c]);
  }
  o << "#define GX_T (GX_WARPS * GX_V)\n#define GX_D 4\n";
  o << "extern \"C\" __global__ void GX_LB " << name << "(const GxArgs a) {\n";
  o << "  const int lane = threadIdx.x & 31; const int warp = threadIdx.x >> 5;\n";
  o << "  const i64 nwords = (a.n + 31) >> 5;\n";
  o << "  const i64 ntiles = (nwords + GX_T - 1) / GX_T;\n";
  // slot layout for conjunct c: column i's words at GX_T * coff[c][i] + kw * 32 * w
  o << "  __shared__ __align__(128) unsigned char s_buf[GX_D][GX_T * " << wbmax << "];\n";
  o << "  __shared__ __align__(8) u64 s_bar[GX_D];\n";
  o << "  __shared__ long long s_tile[GX_D];\n";
  o << "  __shared__ int s_step[GX_D], s_done[GX_D], s_pend[GX_D], s_seq[GX_D];\n";
  o << "  __shared__ u32 s_par[GX_D];\n";
  o << "  __shared__ u32 s_alive[GX_D][GX_T];\n";
  o << "  __shared__ u32 s_cnt[GX_WARPS];\n";
  o << "  __shared__ u64 s_off[GX_D][GX_WARPS];\n";
  o << "  __shared__ u64 s_total[GX_D];\n";
  o << "  __shared__ u64 s_base;\n";
  o << "  __shared__ int s_cseq, s_rseq, s_abort, s_ready;\n";
  o << "  __shared__ long long s_lbpred;\n";   // look-back progress of the oldest tile
  o << "  __shared__ u64 s_lbexcl;\n";
  o << "  __shared__ u32 s_lbpolls;\n";
  o << "  const u32 spin_limit = 1u << 22;\n";
  o << "  const u32 mbar_limit = 1u << 20;  // polls of a slot's barrier (each try_wait may suspend briefly)\n";

  // warp 0: copies of conjunct order[step]'s live full words of slot s, as
  // 16-byte asynchronous copies spread over the warp's lanes; every lane then
  // arrives on the slot's barrier when its copies have landed (32 arrivals)
  o << "  auto issue_ = [&](int s, long long tile, int step) {\n";
  o << "    const int cj = a.order_dev ? __ldg(a.order_dev + step) : a.order[step];\n";
  o << "    int nwt_ = 0;\n";
  o << "    for (int kb = 0; kb < GX_T; kb += 32) {\n";
  o << "      const int kw = kb + lane;\n";
  o << "      const i64 wd = tile * GX_T + kw;\n";
  o << "      nwt_ += __popc(__ballot_sync(GX_FULL, kw < GX_T && s_alive[s][kw] != 0u && (wd + 1) * 32 <= a.n));\n";
  o << "    }\n";
  o << "    if (lane == 0) s_pend[s] = nwt_ != 0 ? 1 : 0;\n";
  o << "    if (nwt_ == 0) return;\n";
  o << "    gx_fence_async_smem();\n";
  o << "    for (int kb = 0; kb < GX_T; kb += 32) {\n";
  o << "      const int kwl = kb + lane;\n";
  o << "      const u32 wm_ = __ballot_sync(GX_FULL, kwl < GX_T && s_alive[s][kwl] != 0u && (tile * GX_T + kwl + 1) * 32 <= a.n);\n";
  o << "      const int nw_ = __popc(wm_);\n";
  o << "      switch (cj) {\n";
  for (int c = 0; c < nc; c++) {
    const int ch = cwb[c] / 16;  // 16-byte chunks per word, all the conjunct's columns
    o << "        case " << c << ":\n";
    o << "          for (int q = lane; q < nw_ * " << ch << "; q += 32) {\n";
    o << "            const int kw = kb + (int)__fns(wm_, 0u, q / " << ch << " + 1);\n";
    o << "            const int ck = q % " << ch << ";\n";
    o << "            const i64 wd = tile * GX_T + kw;\n";
    int chk = 0;
    for (size_t i = 0; i < cc[c].size(); i++) {
      const int col = cc[c][i];
      const int w = type_size(p.schema[col]);
      const int cn = 2 * w;  // chunks of this column per word (32 * w / 16)
      o << "            " << (i ? "else " : "") << "if (ck < " << chk + cn << ") gx_cp16(s_buf[s] + GX_T * " << coff[c][i]
        << " + kw * " << 32 * w << " + (ck - " << chk << ") * 16, (const char*)a.in_data[" << col
        << "] + (wd * 32) * " << w << " + (ck - " << chk << ") * 16);\n";
      chk += cn;
    }
    o << "          }\n";
    o << "          break;\n";
  }
  o << "        default: break;\n      }\n    }\n";
  o << "    gx_cp_arrive(&s_bar[s]);\n";
  o << "  };\n";

  // thread 0: claim the next tile into slot s; returns whether one was claimed
  o << "  auto claim_ = [&](int s) {\n";
  o << "    const long long t = (long long)atomicAdd(a.tile_counter, 1ull);\n";
  o << "    if (t >= ntiles) { s_tile[s] = -1; return; }\n";
  o << "    s_tile[s] = t; s_step[s] = 0; s_done[s] = 0; s_pend[s] = 0; s_seq[s] = s_cseq++;\n";
  o << "  };\n";
  // warp 0: alive masks of a newly claimed tile (rows < n)
  o << "  auto init_alive_ = [&](int s, long long tile) {\n";
  o << "    for (int kw = lane; kw < GX_T; kw += 32) {\n";
  o << "      const i64 r0 = (tile * GX_T + kw) * 32;\n";
  o << "      const i64 left = a.n - r0;\n";
  o << "      s_alive[s][kw] = left >= 32 ? 0xffffffffu : (left <= 0 ? 0u : ((1u << left) - 1u));\n";
  o << "    }\n";
  o << "    __syncwarp();\n";
  o << "  };\n";

  // setup: barriers and the first GX_D tiles
  o << "  if (threadIdx.x == 0) {\n";
  o << "    s_cseq = 0; s_rseq = 0; s_abort = 0;\n";
  o << "    for (int s = 0; s < GX_D; s++) { gx_mbar_init(&s_bar[s], 32u); s_par[s] = 0u; }\n";
  o << "    gx_mbar_init_fence();\n";
  o << "    for (int s = 0; s < GX_D; s++) claim_(s);\n";
  o << "  }\n";
  o << "  __syncthreads();\n";
  o << "  if (warp == 0) {\n";
  o << "    for (int s = 0; s < GX_D; s++) {\n";
  o << "      const long long t = s_tile[s];\n";
  o << "      if (t < 0) continue;\n";
  o << "      init_alive_(s, t);\n";
  o << "      issue_(s, t, 0);\n";
  o << "    }\n";
  o << "  }\n";

  o << "  while (true) {\n";
  o << "    __syncthreads();\n";
  o << "    bool any_ = false;\n";
  o << "    #pragma unroll\n    for (int s = 0; s < GX_D; s++) any_ |= s_tile[s] >= 0;\n";
  o << "    if (!any_ || s_abort) break;\n";
  o << "    for (int s = 0; s < GX_D; s++) {\n";
  o << "      __syncthreads();\n";
  o << "      const long long tile = s_tile[s];\n";
  o << "      if (tile < 0) continue;\n";
  // ---- one conjunct step
  o << "      if (s_done[s] == 0) {\n";
  o << "        if (s_pend[s]) {\n";
  o << "          const u32 par_ = s_par[s];\n";
  o << "          u32 sp_ = 0u;\n";
  o << "          while (!gx_mbar_try_wait(&s_bar[s], par_)) {\n";
  o << "            if (++sp_ > mbar_limit) { gx_set_err(a.err, 1); s_abort = 1; break; }\n";
  o << "            __nanosleep(20);\n";
  o << "          }\n";
  o << "        }\n";
  o << "        const int cj = a.order_dev ? __ldg(a.order_dev + s_step[s]) : a.order[s_step[s]];\n";
  o << "        bool keep_[GX_V];\n";
  o << "        bool inr_[GX_V];\n";
  o << "        switch (cj) {\n";
  for (int c = 0; c < nc; c++) {
    const int cid = p.conjuncts[c];
    o << "          case " << c << ": {\n";
    g.staged_.clear();
    for (size_t i = 0; i < cc[c].size(); i++)
      g.staged_[cc[c][i]] = {"(const void*)(s_buf[s] + GX_T * " + std::to_string(coff[c][i]) + ")",
                             "(i64)(kw * 32 + lane)"};
    const std::vector<int> ids = g.cone({cid});
    g.decl(o, ids, "            ");
    o << "            #pragma unroll\n            for (int k = 0; k < GX_V; k++) {\n";
    o << "              const int kw = warp * GX_V + k;\n";
    o << "              const i64 row = (tile * GX_T + kw) * 32 + lane;\n";
    o << "              const bool full_word_ = (tile * GX_T + kw + 1) * 32 <= a.n; (void)full_word_;\n";
    o << "              const bool inr = ((s_alive[s][kw] >> lane) & 1u) != 0u;\n";
    for (int id : ids)
      if (p.nodes[id].kind == Node::COL) g.emit_node(o, id, "              ");
    for (int id : ids)
      if (p.nodes[id].kind != Node::COL) g.emit_node(o, id, "              ");
    o << "              keep_[k] = " << g.conj_keep(cid) << "; inr_[k] = inr;\n";
    o << "            }\n";
    o << "            break; }\n";
  }
  g.staged_.clear();
  o << "          default:\n";
  o << "            #pragma unroll\n            for (int k = 0; k < GX_V; k++) { keep_[k] = false; inr_[k] = false; }\n";
  o << "        }\n";
  o << "        #pragma unroll\n        for (int k = 0; k < GX_V; k++) {\n";
  o << "          const u32 nb_ = __ballot_sync(GX_FULL, inr_[k] && keep_[k]);\n";
  o << "          if (lane == 0) s_alive[s][warp * GX_V + k] &= nb_;\n";
  o << "        }\n";
  o << "        __syncthreads();\n";
  // warp 0: next step or done
  o << "        if (warp == 0) {\n";
  o << "          if (lane == 0) { if (s_pend[s]) s_par[s] ^= 1u; s_step[s] += 1; }\n";
  o << "          __syncwarp();\n";
  o << "          u32 live_ = 0u;\n";
  o << "          for (int kw = lane; kw < GX_T; kw += 32) live_ |= s_alive[s][kw];\n";
  o << "          const bool anyl_ = __any_sync(GX_FULL, live_ != 0u);\n";
  o << "          if (!anyl_ || s_step[s] >= " << nc << ") {\n";
  o << "            if (lane == 0) { s_done[s] = 1; s_pend[s] = 0; }\n";
  o << "          } else {\n";
  o << "            issue_(s, tile, s_step[s]);\n";
  o << "          }\n";
  o << "        }\n";
  o << "        __syncthreads();\n";
  o << "      }\n";
  // ---- publish the aggregate of a finished tile
  o << "      if (s_done[s] == 1) {\n";
  o << "        u32 c_ = 0u;\n";
  o << "        #pragma unroll\n        for (int k = 0; k < GX_V; k++) c_ += __popc(s_alive[s][warp * GX_V + k]);\n";
  o << "        if (lane == 0) s_cnt[warp] = c_;\n";
  o << "        __syncthreads();\n";
  o << "        if (warp == 0) {\n";
  o << "          const u64 tot_ = gx_tile_publish(a.tile_status, tile, s_cnt, s_off[s], GX_WARPS);\n";
  o << "          if (lane == 0) { s_total[s] = tot_; s_done[s] = 2; }\n";
  o << "          if (lane == 0 && s_seq[s] == s_rseq) { s_lbpred = tile - 1; s_lbexcl = 0ull; s_lbpolls = 0u; }\n";
  o << "        }\n";
  o << "        __syncthreads();\n";
  o << "      }\n";
  // ---- resolve and write, in claim order
  // the oldest tile's look-back is polled, never waited on: while predecessors
  // are missing the block goes on with its other tiles, whose aggregates other
  // blocks may be waiting for
  o << "      if (s_done[s] == 2 && s_seq[s] == s_rseq) {\n";
  o << "        if (warp == 0) {\n";
  o << "          long long pr_ = s_lbpred; u64 ex_ = s_lbexcl;\n";
  o << "          const bool ok_ = gx_lookback_poll(a.tile_status, tile, s_total[s], &pr_, &ex_);\n";
  o << "          if (lane == 0) {\n";
  o << "            s_lbpred = pr_; s_lbexcl = ex_; s_ready = ok_ ? 1 : 0;\n";
  o << "            if (ok_) {\n";
  o << "              s_base = ex_;\n";
  o << "              if (tile == ntiles - 1) *a.out_count = ex_ + s_total[s];\n";
  o << "            } else if (++s_lbpolls > spin_limit) {\n";
  o << "              gx_set_err(a.err, 1); s_abort = 1;\n";
  o << "            } else {\n";
  o << "              __nanosleep(64);\n";
  o << "            }\n";
  o << "          }\n";
  o << "        }\n";
  o << "        __syncthreads();\n";
  o << "        if (!s_ready) continue;\n";
  o << "        {\n";
  o << "          u32 bal[GX_V]; u32 wcnt = 0u;\n";
  o << "          #pragma unroll\n          for (int k = 0; k < GX_V; k++) { bal[k] = s_alive[s][warp * GX_V + k]; wcnt += __popc(bal[k]); }\n";
  o << "          if (wcnt != 0u) {\n";
  o << "            u64 pos = s_base + s_off[s][warp];\n";
  o << "            const i64 w0 = tile * GX_T + (i64)warp * GX_V;\n";
  emit_filter_writes_dense(o, g, p, "            ");
  o << "          }\n";
  o << "        }\n";
  o << "        __syncthreads();\n";
  o << "        if (threadIdx.x == 0) {\n";
  o << "          s_rseq++;\n";
  o << "          claim_(s);\n";
  o << "          for (int q = 0; q < GX_D; q++)  // the next oldest, if already published\n";
  o << "            if (s_tile[q] >= 0 && s_done[q] == 2 && s_seq[q] == s_rseq) { s_lbpred = s_tile[q] - 1; s_lbexcl = 0ull; s_lbpolls = 0u; }\n";
  o << "        }\n";
  o << "        __syncthreads();\n";
  o << "        if (warp == 0 && s_tile[s] >= 0) {\n";
  o << "          init_alive_(s, s_tile[s]);\n";
  o << "          issue_(s, s_tile[s], 0);\n";
  o << "        }\n";
  o << "      }\n";
  o << "    }\n";
  o << "  }\n";
  // an abandoned run (a wait gave up): let copies still in flight land before exit
  o << "  __syncthreads();\n";
  o << "  if (s_abort && threadIdx.x == 0) {\n";
  o << "    for (int s = 0; s < GX_D; s++) {\n";
  o << "      if (s_tile[s] < 0 || !s_pend[s] || s_done[s] != 0) continue;\n";
  o << "      u32 sp_ = 0u;\n";
  o << "      while (!gx_mbar_try_wait(&s_bar[s], s_par[s]) && ++sp_ < mbar_limit) __nanosleep(20);\n";
  o << "    }\n";
  o << "  }\n";
  o << "}\n";
}

}  // namespace

TileLayout tile_layout(const Plan& p, int warps, int words, int stages) {
  TileLayout L;
  L.tile_rows = warps * words * 32;
  L.stages = stages;
  if (L.tile_rows % 128 != 0) fail(GX_ERR_INVALID, "tile-staged kernels need tiles of a multiple of 128 rows");
  if (stages < 2) fail(GX_ERR_INVALID, "tile-staged kernels need at least 2 stages");
  if (warps > 32) fail(GX_ERR_INVALID, "tile-staged kernels take at most 32 consumer warps");
  L.cols = referenced_columns(p);
  uint32_t off = 0;
  for (int c : L.cols) {
    // data: the tile's bytes from the 16-byte block of its first element up to
    // the block past its last; mask: its words plus the next one (re-alignment
    // to the tile's rows reads one word ahead), from the first word's block
    L.data_off.push_back(off);
    off += (uint32_t)L.tile_rows * (uint32_t)type_size(p.schema[c]) + 32u;
    if (p.nullable[c]) {
      L.mask_off.push_back(off);
      L.mask_index.push_back(L.num_masked++);
      off += (uint32_t)L.tile_rows / 8u + 32u;
    } else {
      L.mask_off.push_back(UINT32_MAX);
      L.mask_index.push_back(-1);
    }
  }
  L.stage_bytes = (off + 127u) & ~127u;
  // output staging: per non-literal output its data slot and one validity
  // byte per row, by the row's kept rank within the tile
  uint32_t oo = 0;
  for (const auto& os : p.outputs) {
    const int t = os.kind == OutSpec::COPY ? p.schema[os.col] : os.type;
    const uint32_t w = os.kind == OutSpec::BROADCAST ? 0u : (uint32_t)type_size(t);
    L.out_width.push_back(w);
    L.out_off.push_back(oo);
    oo += ((uint32_t)L.tile_rows * w + 15u) & ~15u;
    L.out_valid_off.push_back(oo);
    if (os.kind != OutSpec::BROADCAST) oo += (uint32_t)L.tile_rows;
  }
  L.out_stage_bytes = (oo + 127u) & ~127u;
  L.out_base = L.stage_bytes * (uint32_t)stages;
  L.dyn_smem = L.out_base + (uint32_t)L.out_stages * L.out_stage_bytes;
  return L;
}

std::vector<int> conjunct_columns(const Plan& p, int c) {
  std::set<int> cols;
  std::function<void(int)> go = [&](int id) {
    if (id < 0) return;
    const Node& n = p.nodes[id];
    if (n.kind == Node::COL) cols.insert(n.col);
    if (n.kind == Node::OP) { go(n.a); go(n.b); }
  };
  go(p.conjuncts.at(c));
  return std::vector<int>(cols.begin(), cols.end());
}

// Which binary64 operation classes go to the FP64 pipe when the plan leaves it
// to the library.  Both forms are exact; the choice balances the two pipes.
// The FP64 pipe takes a warp instruction every 16 clocks per SM, the ALU and
// IMAD pipes two a clock each.  Add, subtract and multiply are one FP64
// instruction or about 25 integer ones (12 clocks), close enough that the
// otherwise idle FP64 pipe takes them.  Conversions (10 to 20 integer
// instructions), compares with a literal (4) and divisions by a literal or an
// integer (about 30, against a multiply, two FMAs and the conversions of the
// operands) are far cheaper on the integer pipes.  Measured at 2^26 rows of the
// deep plan: 1.30 ms, 1.42 ms with conversions and 1.47 ms with literal
// divisions on the FP64 pipe; the order-line plan's two divisions at 2^27 rows
// cost the same either way (1.88 ms), its aggregation 1.48 ms against 1.64 ms.
int auto_native_f64_ops() { return kNativeAddSub | kNativeMul; }

// Projection kernels wait for memory, so one more block of warps per SM is worth
// more than the compiler's last registers: five outputs over five columns, 2^25
// rows, 88 registers 499 us, capped at 80 474 (72 477, 64 478, 56 513 with spills).
// Held to the cap are plans whose loads of a warp's words leave half of it and that
// call no transcendental function (those keep polynomials and the call's own
// state live).
constexpr int kProjectRegs = 80;
static bool project_fits_cap(const Plan& p, const KernelConfig& cfg) {
  std::set<int> seen;
  int regs = 0;
  bool fits = true;
  std::function<void(int)> go = [&](int id) {
    if (id < 0 || !seen.insert(id).second) return;
    const Node& n = p.nodes[id];
    if (n.kind == Node::COL) regs += cfg.words * std::max(1, type_size(p.schema[n.col]) / 4);
    if (n.kind != Node::OP) return;
    fits = fits && Gen::op_cost(n.op) < 64;
    go(n.a);
    go(n.b);
  };
  for (const auto& o : p.outputs)
    if (o.kind == OutSpec::NODE) go(o.node);
  return fits && regs <= kProjectRegs / 2;
}

bool copies_only(const Plan& p) {
  for (const auto& o : p.outputs)
    if (o.kind != OutSpec::COPY) return false;
  return true;
}

// The learner's ordered kernel waits on one load per conjunct and word, so
// resident warps are what hides it: with outputs that are column copies, few
// values are live, and 32 registers (64 warps per SM) suffice for conjuncts that
// compare and add.  Validity and divisions keep more alive, and 48 registers then
// spill less than the lost warps cost; a transcendental function's own state spills
// at either, and 40 keep more warps.  Queues of eight batches of 2^22 rows, us
// at 32 / 40 / 48 registers / uncapped: the skewed-range conjuncts 481 / 521 / 537
// / 888, over nullable columns 641 / 553 / 543 / 840; sums 728 / 837 / 810 / 1374
// and 976 / 881 / 851 / 1803; divisions 1782 / 1620 / 1527 / 1737 and 1949 / 1876 /
// 1753 / 3177; LN and EXP 3771 / 3577 / 3757 / 3662 and 3832 / 3610 / 3722 / 3781.
static int ordered_regs(const Plan& p) {
  bool nulls = false;
  int most = 0;  // the dearest operator's cost
  std::function<void(int)> go = [&](int id) {
    if (id < 0) return;
    const Node& n = p.nodes[id];
    if (n.kind == Node::COL) nulls = nulls || p.nullable[n.col];
    if (n.kind != Node::OP) return;
    most = std::max(most, Gen::op_cost(n.op));
    go(n.a);
    go(n.b);
  };
  for (int c : p.conjuncts) go(c);
  return most >= 64 ? 40 : most >= 16 || nulls ? 48 : 32;
}

std::string generate_kernel(const Plan& p, KernelKind kind, const KernelConfig& cfg_in, const std::string& name) {
  KernelConfig cfg = cfg_in;
  if (cfg.runtime_order && cfg.max_regs == 0 && copies_only(p)) cfg.max_regs = ordered_regs(p);
  if (cfg.native_f64_ops < 0) cfg.native_f64_ops = auto_native_f64_ops();
  if (kind == KernelKind::PROJECT && cfg.max_regs == 0 && project_fits_cap(p, cfg)) cfg.max_regs = kProjectRegs;
  Gen g(p, cfg);
  if (p.has_filter() && cfg.dense) {
    // columns whose data the predicate reads (not only their validity, as
    // IS [NOT] NULL does) and the dense projections read again by kept row
    std::set<int> pred_cols;
    const std::vector<int> pc = g.predicate_cone();
    for (int id : pc) {
      const Node& n = p.nodes[id];
      if (n.kind != Node::OP || n.op == OP_IS_NULL || n.op == OP_IS_NOT_NULL) continue;
      for (int x : {n.a, n.b})
        if (x >= 0 && p.nodes[x].kind == Node::COL) pred_cols.insert(p.nodes[x].col);
    }
    for (int c : p.conjuncts)  // a BOOL8 column as a conjunct is read as data
      if (p.nodes[c].kind == Node::COL) pred_cols.insert(p.nodes[c].col);
    for (int id : g.cone(g.output_roots()))
      if (p.nodes[id].kind == Node::COL && pred_cols.count(p.nodes[id].col)) g.reread_cols_.insert(p.nodes[id].col);
    for (const auto& os : p.outputs)
      if (os.kind == OutSpec::COPY && pred_cols.count(os.col)) g.reread_cols_.insert(os.col);
  }
  std::ostringstream o;
  emit_prelude(o, cfg);
  g.emit_rcp_table(o);
  if (kind == KernelKind::FUSED_STAGED) {
    if (!p.has_filter() || p.conjuncts.size() > 16) fail(GX_ERR_INVALID, "the staged kernel runs filters of at most 16 conjuncts");
    KernelConfig c = cfg;
    c.dense = true;
    c.runtime_order = true;
    Gen gs(p, c);
    emit_staged_filter(o, gs, p, name);
    return o.str();
  }
  if (kind == KernelKind::FUSED_TMA) {
    if (!p.has_filter()) fail(GX_ERR_INVALID, "the tile-staged kernel runs filter plans");
    if (cfg.runtime_order || cfg.short_circuit || !cfg.dense)
      fail(GX_ERR_INVALID, "the tile-staged kernel evaluates conjuncts in plan order with dense projections");
    const TileLayout L = tile_layout(p, cfg.warps, cfg.words, cfg.stages);
    emit_fused_tma(o, g, p, L, name);
    return o.str();
  }
  if (kind == KernelKind::FUSED_BATCHED || kind == KernelKind::FUSED_STREAM) {
    if (!p.has_filter()) fail(GX_ERR_INVALID, "the batched kernel runs filter plans");
    if (cfg.runtime_order || cfg.short_circuit) fail(GX_ERR_INVALID, "the batched kernel evaluates conjuncts in plan order");
    KernelConfig c = cfg;
    c.dense = true;
    Gen gb(p, c);
    gb.reread_cols_ = g.reread_cols_;
    emit_fused_batched(o, gb, p, gb.predicate_cone(), name, kind == KernelKind::FUSED_STREAM);
    return o.str();
  }
  o << "extern \"C\" __global__ void GX_LB " << name << "(const GxArgs a) {\n";
  o << "  const int lane = threadIdx.x & 31; const int warp = threadIdx.x >> 5;\n";
  o << "  const i64 nwords = (a.n + 31) >> 5;\n";
  if (kind == KernelKind::PROJECT) {
    std::vector<int> ids = g.cone(g.output_roots());
    o << "  for (i64 w0 = ((i64)blockIdx.x * GX_WARPS + warp) * GX_V; w0 < nwords;"
         " w0 += (i64)gridDim.x * GX_WARPS * GX_V) {\n";
    g.decl(o, ids, "    ");
    g.masks_ = Gen::Masks::WORDS;
    g.emit_mask_words(o, ids, {}, "    ");
    // every column load of the warp's words first, then operators and stores
    o << "    #pragma unroll\n    for (int k = 0; k < GX_V; k++) {\n";
    o << "      const i64 row = (w0 + k) * 32 + lane; const bool inr = row < a.n; (void)inr;\n";
    for (int id : ids)
      if (p.nodes[id].kind == Node::COL) g.emit_node(o, id, "      ");
    o << "    }\n";
    o << "    #pragma unroll\n    for (int k = 0; k < GX_V; k++) {\n";
    o << "      const i64 row = (w0 + k) * 32 + lane; const bool inr = row < a.n; (void)inr;\n";
    o << "      const i64 orow = row; (void)orow;\n";
    for (int id : ids)
      if (p.nodes[id].kind != Node::COL) g.emit_node(o, id, "      ");
    for (size_t j = 0; j < p.outputs.size(); j++) {
      const OutSpec& os = p.outputs[j];
      if (os.kind != OutSpec::NODE) continue;
      o << "      if (inr) " << store_stmt(os.type, "a.out_data[" + std::to_string(j) + "]", "row", g.B(os.node)) << "\n";
      o << "      { const u32 vb_ = __ballot_sync(GX_FULL, inr && " << g.V(os.node) << ");\n";
      o << "        if (lane == 0 && w0 + k < nwords) a.out_mask[" << j << "][w0 + k] = vb_; }\n";
    }
    o << "    }\n  }\n}\n";
    return o.str();
  }

  if ((cfg.runtime_order || cfg.conj_stats) && p.conjuncts.size() > 16)
    fail(GX_ERR_UNSUPPORTED, "learned ordering supports at most 16 AND conjuncts");
  // dense phase 2 recomputes every output from the gathered row; the word mode
  // would reuse predicate values that a runtime-ordered predicate never computed
  if (cfg.runtime_order && !cfg.dense) fail(GX_ERR_INVALID, "runtime conjunct order needs dense projections");
  const std::vector<int> pred_ids = g.predicate_cone();
  // per-conjunct pass counts (training labels) only in the plain fixed-order count pass
  const bool stats = kind == KernelKind::COUNT_FILTER && cfg.conj_stats && !cfg.runtime_order && !cfg.short_circuit;
  if (stats) {
    o << "  __shared__ unsigned long long s_conj[16];\n";
    o << "  if (threadIdx.x < 16) s_conj[threadIdx.x] = 0ull;\n";
    o << "  __syncthreads();\n";
  }
  if (kind == KernelKind::FUSED_FILTER && cfg.dense) {
    emit_fused_pipelined(o, g, p, pred_ids);
    return o.str();
  }
  o << "  __shared__ unsigned long long s_tile;\n";
  o << "  __shared__ u64 s_w[GX_WARPS];\n";
  o << "  const i64 ntiles = (nwords + GX_TILE_WORDS - 1) / GX_TILE_WORDS;\n";
  if (kind == KernelKind::FUSED_FILTER) {
    o << "  while (true) {\n";
    o << "    if (threadIdx.x == 0) s_tile = atomicAdd(a.tile_counter, 1ull);\n";
    o << "    __syncthreads();\n";
    o << "    const i64 tile = (i64)s_tile;\n";
    o << "    if (tile >= ntiles) break;\n";
  } else {
    o << "  for (i64 tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {\n";
  }
  o << "    const i64 w0 = tile * GX_TILE_WORDS + (i64)warp * GX_V;\n";
  g.decl(o, pred_ids, "    ");
  g.emit_predicate(o, "    ");
  if (stats) g.emit_conj_stats(o, "    ");
  o << "    u32 bal[GX_V]; u32 wcnt = 0;\n";
  o << "    #pragma unroll\n    for (int k = 0; k < GX_V; k++) { bal[k] = __ballot_sync(GX_FULL, alive[k]); wcnt += __popc(bal[k]); }\n";
  // per-warp exclusive offsets within the tile
  o << "    if (lane == 0) s_w[warp] = wcnt;\n";
  o << "    __syncthreads();\n";
  o << "    if (warp == 0) {\n";
  o << "      u64 c = lane < GX_WARPS ? s_w[lane] : 0ull; u64 incl = c;\n";
  o << "      #pragma unroll\n      for (int d = 1; d < 32; d <<= 1) { u64 t = __shfl_up_sync(GX_FULL, incl, d); if (lane >= d) incl += t; }\n";
  o << "      const u64 total = __shfl_sync(GX_FULL, incl, 31);\n";
  if (kind == KernelKind::FUSED_FILTER) {
    o << "      const u64 excl_tile = gx_lookback(a.tile_status, tile, total, a.err, GX_SPINS);\n";
    o << "      if (tile == ntiles - 1 && lane == 0 && excl_tile != ~0ull) *a.out_count = excl_tile + total;\n";
  } else if (kind == KernelKind::COUNT_FILTER) {
    o << "      if (lane == 0) a.tile_status[tile] = total;\n";
    o << "      const u64 excl_tile = 0ull;\n";
  } else {
    o << "      const u64 excl_tile = a.tile_status[tile];\n";
  }
  o << "      if (lane < GX_WARPS) s_w[lane] = excl_tile == ~0ull ? ~0ull : excl_tile + incl - c;\n";
  o << "    }\n";
  o << "    __syncthreads();\n";
  if (kind != KernelKind::COUNT_FILTER) {
    o << "    u64 pos = s_w[warp];\n";
    o << "    if (pos == ~0ull) break;\n";  // look-back gave up: error already recorded
    o << "    if (wcnt != 0u) {\n";
    emit_filter_writes(o, g, p, pred_ids, "      ");
    o << "    }\n";
  }
  o << "    __syncthreads();\n";  // s_tile / s_w reuse by the next tile
  o << "  }\n";
  if (stats) {
    o << "  __syncthreads();\n";
    o << "  if (threadIdx.x < " << p.conjuncts.size() << ") atomicAdd(&a.conj_counts[threadIdx.x], s_conj[threadIdx.x]);\n";
  }
  o << "}\n";
  return o.str();
}


// ------------------------------------------------------------ aggregation
// Fused filter + group-by aggregation kernel (gx_filter_aggregate).  One block
// per SM; its warps draw chunks of GX_V words, evaluate the condition, list
// their kept rows, and deal them to lanes in rounds of 32.  A lane computes its
// row's keys and aggregation inputs and adds them to its group, in one of two
// ways:
//
// 1. Few groups.  Every warp has accumulators of its own in shared memory for
//    each of the first warp_groups groups the block meets, `replicas` of each, so
//    that as many lanes of one group update them side by side: a load, one
//    operation and a store per accumulator, no combining and no atomic, repeated
//    while a round holds more lanes of a group.  Rounds with more than three
//    passes' worth combine over a tree within the warp first.  The tree alone took
//    280 of 640 instructions per 32 rows and five FP64 instructions per sum, the
//    passes take about 90 and two: order-line rows by two flags (four groups, nine
//    aggregations), 2^26 rows: 1.48 -> 1.30 ms.  The room goes to 8 or
//    more groups with up to 16 replicas first, so that a round's largest group
//    mostly takes one pass (four groups, 6 / 9 / 12 / 16 replicas: 1362 / 1246 /
//    1229 / 1126 us; 1142 with the number read from shared memory).  A block that
//    meets more groups merges what it has and goes on with half the replicas, or
//    fewer, for more groups, down to one, unless 32 of its rows held more than 28:
//    then there are hundreds.  2^24 rows, nine aggregations, call us with 18 / 30 /
//    45 groups: 373 / 362 / 493; through the table 1018 / 907 and more.
// 2. Many groups.  When a group finds no room there, the block's warps finish
//    their chunks, the warps' accumulators go to the global table, and the block
//    goes on with one hash table in the same shared memory (thousands of groups),
//    updated by shared-memory atomics; the tree runs only for rounds that hold
//    more than two rows of one group.  A row whose group finds no room in it
//    goes to the global table directly.  By ship date (2557 groups, four
//    accumulators, 2^24 rows) 1.40 -> 0.55 ms, where one-warp blocks with 8 KB
//    tables sent most rows to the global table.
//
// When the chunks run out, each block merges its accumulators into the global
// table.
static std::string agg_identity(int kind, bool flt) {
  if (kind == 2) return "0x7FFFFFFFFFFFFFFFull";                 // MIN: +largest (ordered)
  if (kind == 3) return "0x8000000000000000ull";                 // MAX: -largest (ordered)
  (void)flt;
  return "0ull";                                                 // sums (0 and +0.0 share bits)
}

uint64_t agg_counts_are_rows(const Plan& p, const AggLayout& L) {
  KernelConfig cfg;
  cfg.native_f64_ops = 0;
  Gen g(p, cfg);
  uint64_t m = 0;
  for (size_t j = 0; j < L.in_nodes.size() && j < 64; j++)
    if (L.in_nodes[j] >= 0 && g.never_null(L.in_nodes[j])) m |= 1ull << j;
  return m;
}

// Bits of group key j (an integer, date or BOOL8 column) as a field of a packed key
static int agg_key_bits(const Plan& p, const AggLayout& L, int j) {
  return 8 * type_size(p.schema[p.nodes[L.key_nodes[j]].col]);
}
// One group key of 64 bits
static bool agg_one_word_key(const Plan& p, const AggLayout& L) {
  return L.key_nodes.size() == 1 && agg_key_bits(p, L, 0) == 64;
}
// All keys, their null bits and one bit that is always set fit a 64-bit word: a
// group then is one word in shared memory, claimed by one compare-and-swap and
// compared by one load (else: a state word, a null word and a word per key, with
// a wait while another lane writes them).  One 64-bit key is packed too: it is
// XORed with a constant, so that the words that mean "empty" and NULL stand for
// two keys of its 2^64; rows of these two go to the global table (2557 groups, nine
// aggregations, 2^24 rows: 1260 us as separate words, 645 as one).
static bool agg_packs_keys(const Plan& p, const AggLayout& L) {
  int bits = 1 + (int)L.key_nodes.size();
  for (size_t j = 0; j < L.key_nodes.size(); j++) bits += agg_key_bits(p, L, (int)j);
  return bits <= 64 || agg_one_word_key(p, L);
}

AggShared agg_shared(const Plan& p, const AggLayout& L, const KernelConfig& cfg) {
  const int nk = std::max<int>(1, (int)L.key_nodes.size()), na = (int)L.kinds.size();
  const uint64_t rows_cnt = agg_counts_are_rows(p, L);
  AggShared s;
  s.packed = agg_packs_keys(p, L);
  s.acc_cell.assign(na, -1);
  s.cnt_cell.assign(na, -1);
  s.acc_slot.assign(na, -1);
  s.cnt_slot.assign(na, -1);
  int cnts = 0;
  s.rows_cell = s.cells++;
  for (int j = 0; j < na; j++) {
    if (L.kinds[j] != 4 && L.kinds[j] != 5) {
      s.acc_cell[j] = s.cells++;
      s.acc_slot[j] = s.accs++;
    }
    if (!((rows_cnt >> j) & 1ull)) {
      s.cnt_cell[j] = s.cells++;
      s.cnt_slot[j] = cnts++;
    }
  }
  s.dict_bytes = (kAggDict * (8 * (nk + 1) + 12) + 15) / 16 * 16;
  const int budget = std::max(L.smem_bytes - s.dict_bytes, 8 * 1024);  // small blocks keep a table of some size
  const int room = budget / (cfg.warps * s.cells * 8);  // words of a cell per warp
  s.replicas = std::max(1, std::min(16, room / L.first_groups));
  s.warp_groups = std::min(kAggGroups, room / s.replicas);
  s.cell_words = std::min(room, s.replicas * kAggGroups);
  const int slot_bytes = 8 * ((s.packed ? 1 : nk) + s.accs) + 4 * ((s.packed ? 1 : 3) + cnts);
  s.slots = std::max(16, std::min(8192, budget / slot_bytes) / 8 * 8);
  s.dyn_bytes = s.dict_bytes + std::max(s.cell_words * cfg.warps * s.cells * 8, s.slots * slot_bytes);
  return s;
}

std::string generate_agg_kernel(const Plan& p, const AggLayout& L, const KernelConfig& cfg_in,
                                const std::string& name) {
  KernelConfig cfg = cfg_in;
  if (cfg.native_f64_ops < 0) cfg.native_f64_ops = auto_native_f64_ops();
  cfg.short_circuit = false;
  cfg.runtime_order = false;
  cfg.conjunct_order.clear();
  Gen g(p, cfg);
  std::ostringstream o;
  emit_prelude(o, cfg);
  g.emit_rcp_table(o);
  const int nk = (int)L.key_nodes.size(), na = (int)L.kinds.size();
  const uint64_t rows_cnt = agg_counts_are_rows(p, L);
  const AggShared sh = agg_shared(p, L, cfg);
  // (a row that finds no place in 8 probes of the table goes to the global one: 32
  // probes of a full table cost 100,000 groups 4757 us, 8 take 4442)
  const bool two = sh.replicas > 1 && sh.warp_groups < kAggGroups;  // fewer replicas hold more groups
  o << "#define GXA_S " << sh.slots << "\n#define GXA_G " << sh.warp_groups << "\n#define GXA_R " << sh.replicas << "\n#define GXA_GMAX "
    << kAggGroups << "\n#define GXA_GMANY 28\n#define GXA_GR " << sh.cell_words << "\n#define GXA_CS (GX_WARPS * GXA_GR)\n"
    << "#define GXA_D " << kAggDict
    << "\n#define GXA_NK " << std::max(nk, 1) << "\n#define GXA_PROBES 8\n";
  // key hash (null keys hash as zero with their null bit set)
  // (32-bit multiplies by odd constants, a key's high half only where it has
  // one; the finaliser spreads to both the high bits, which place a group in
  // shared memory, and the low ones, which do in the global table)
  o << "__device__ __forceinline__ u64 gxa_hash(const u64* kv, u32 kn) {\n"
       "  u32 h = kn * 0x9E3779B1u + 0x85EBCA77u;\n";
  for (int j = 0; j < nk; j++) {
    o << "  h = (h ^ (u32)kv[" << j << "]) * 0x9E3779B1u; h ^= h >> 15;\n";
    if (type_size(p.schema[p.nodes[L.key_nodes[j]].col]) == 8) o << "  h = (h ^ (u32)(kv[" << j << "] >> 32)) * 0xC2B2AE35u; h ^= h >> 13;\n";
  }
  o << "  h *= 0x27D4EB2Fu; return (u64)(h ^ (h >> 16));\n}\n";
  auto same_keys = [&](const std::string& ks, const std::string& stride, const std::string& pos) {
    std::string r = "true";
    for (int j = 0; j < nk; j++)
      r += " && *(volatile u64*)(" + ks + " + " + std::to_string(j) + "ull * " + stride + " + " + pos + ") == kv[" +
           std::to_string(j) + "]";
    return r;
  };
  auto write_keys = [&](std::ostringstream& os, const std::string& ks, const std::string& stride,
                        const std::string& pos, const std::string& ind) {
    for (int j = 0; j < nk; j++)
      os << ind << ks << "[" << j << "ull * " << stride << " + " << pos << "] = kv[" << j << "];\n";
  };
  if (two)
    // the next split of the accumulators' room, when a block met `need` groups in
    // 32 rows: fewer replicas, more groups (replicas 0: the table is next)
    o << "__device__ __noinline__ void gxa_next_split(u32* room, int* rep, u32 need) {\n"
         "  int r = *rep; u32 g = *room;\n"
         "  while (r > 1 && (g == *room || g < need + need / 4u)) { r /= 2; g = min((u32)GXA_GMAX, (u32)GXA_GR / (u32)r); }\n"
         "  if (g > *room && need <= GXA_GMANY) { *room = g; *rep = r; } else { *rep = 0; }\n"
         "}\n";
  if (sh.packed) {
    // a group as one word, and back; its place in shared memory is the key times
    // 2^32 over the golden ratio (Knuth's multiplicative hashing): consecutive
    // keys -- dates, numbered rows -- fall evenly over the table, so the longest
    // probe of a warp's 32 lanes, which all of them wait for, stays short
    const bool one = agg_one_word_key(p, L);
    if (one) {
      o << "__device__ __forceinline__ u64 gxa_pack(const u64* kv, u32 kn) {\n"
           "  const u64 pk = kv[0] ^ 0x9E3779B97F4A7C15ull;\n"
           "  return kn ? 1ull : pk == 1ull ? 0ull : pk;\n}\n"
           "__device__ __forceinline__ u32 gxa_unpack(u64 pk, u64* kv) {\n"
           "  kv[0] = pk == 1ull ? 0ull : pk ^ 0x9E3779B97F4A7C15ull;\n  return pk == 1ull ? 1u : 0u;\n}\n"
           "__device__ __forceinline__ u32 gxa_place(u64 pk) {\n"
           "  const u32 h = (u32)pk * 0x9E3779B1u;\n"
           "  return (h ^ (h >> 15) ^ (u32)(pk >> 32)) * 0x9E3779B1u;\n}\n";
    } else {
      int off = 1 + nk;
      std::string pack = "1ull | ((u64)kn << 1)", unpack;
      for (int j = 0; j < nk; j++) {
        const int w = agg_key_bits(p, L, j);
        const std::string m = "0x" + [&] { std::ostringstream h; h << std::hex << (w == 64 ? ~0ull : (1ull << w) - 1ull); return h.str(); }() + "ull";
        pack += " | ((kv[" + std::to_string(j) + "] & " + m + ") << " + std::to_string(off) + ")";
        const bool sgn = std::string(load_fn(p.schema[p.nodes[L.key_nodes[j]].col])).find("_u") == std::string::npos;
        const std::string lsh = std::to_string(64 - off - w), rsh = std::to_string(64 - w);
        unpack += " kv[" + std::to_string(j) + "] = " + (sgn ? "(u64)((i64)(pk << " + lsh + ") >> " + rsh + ")" : "(pk << " + lsh + ") >> " + rsh) + ";";
        off += w;
      }
      o << "__device__ __forceinline__ u64 gxa_pack(const u64* kv, u32 kn) { return " << pack << "; }\n";
      o << "__device__ __forceinline__ u32 gxa_unpack(u64 pk, u64* kv) { kv[0] = 0ull;" << unpack << " return (u32)(pk >> 1) & "
        << ((1u << nk) - 1u) << "u; }\n";
      o << "__device__ __forceinline__ u32 gxa_place(u64 pk) {\n  u32 h = (u32)(pk >> " << 1 + nk << ") * 0x9E3779B1u;\n";
      if (off - 1 - nk > 32) o << "  h = (h ^ (h >> 15) ^ (u32)(pk >> " << 33 + nk << ")) * 0x9E3779B1u;\n";
      if (nk) o << "  h += ((u32)(pk >> 1) & " << ((1u << nk) - 1u) << "u) * 0x27D4EB2Fu;\n";
      o << "  return h;\n}\n";
    }
    const std::string none = one ? "  if (key == 0ull) return -1;\n" : "";  // not held in shared memory
    o << "__device__ int gxa_find_table(u64* pk, u64 key) {\n" << none
      << "  u32 pos = __umulhi(gxa_place(key), (u32)GXA_S);\n"
         "  for (int pr = 0; pr < GXA_PROBES; pr++) {\n"
         "    u64 v = *(volatile u64*)(pk + pos);\n"
         "    if (v == 0ull) v = atomicCAS((unsigned long long*)(pk + pos), 0ull, (unsigned long long)key);\n"
         "    if (v == 0ull || v == key) return (int)pos;\n"
         "    pos = pos + 1u == GXA_S ? 0u : pos + 1u;\n"
         "  }\n"
         "  return -1;\n"
         "}\n";
    o << "__device__ int gxa_find_dict(u32* st, u64* pk, u32* at, u32* ng, const u32* room, u64 key, int* err) {\n" << none
      << "  u32 pos = __umulhi(gxa_place(key), (u32)GXA_D);\n"
         "  for (int pr = 0; pr < GXA_D; pr++) {\n"
         "    u64 v = *(volatile u64*)(pk + pos);\n"
         "    if (v == 0ull) {\n"
         "      if (*(volatile u32*)ng >= *(volatile const u32*)room) return -1;\n"
         "      v = atomicCAS((unsigned long long*)(pk + pos), 0ull, (unsigned long long)key);\n"
         "      if (v == 0ull) {\n"
         "        const u32 i = atomicAdd(ng, 1u);\n"
         "        if (i >= *(volatile const u32*)room) { atomicExch(st + pos, 0xffffffffu); return -1; }\n"  // lost the last place
         "        at[i] = pos;\n"
         "        __threadfence_block();\n"
         "        atomicExch(st + pos, 2u + i);\n"
         "        return (int)i;\n"
         "      }\n"
         "    }\n"
         "    if (v == key) {\n"
         "      u32 s = gx_lds_acquire(st + pos), spins = 0;\n"
         "      while (s == 0u) {\n"
         "        if (++spins > (1u << 20)) { atomicExch(err, 1); return -2; }\n"
         "        __nanosleep(16);\n"
         "        s = gx_lds_acquire(st + pos);\n"
         "      }\n"
         "      return s == 0xffffffffu ? -1 : (int)s - 2;\n"
         "    }\n"
         "    pos = (pos + 1u) & (GXA_D - 1);\n"
         "  }\n"
         "  return -1;\n"
         "}\n";
  } else {
    // the block's table: -1 when the probe finds no room, -2 after a wait gave up
    o << "__device__ int gxa_find_smem(u32* st, u32* nm, u64* ks, const u64* kv, u32 kn, u64 h, int* err) {\n"
         "  u32 pos = __umulhi((u32)h, (u32)GXA_S);\n"
         "  for (int pr = 0; pr < GXA_PROBES; pr++) {\n"
         "    u32 s = gx_lds_acquire(st + pos);\n"
         "    if (s == 0u) {\n"
         "      s = atomicCAS(st + pos, 0u, 1u);\n"
         "      if (s == 0u) {\n";
    write_keys(o, "ks", "GXA_S", "pos", "        ");
    o << "        nm[pos] = kn;\n"
         "        __threadfence_block();\n"
         "        atomicExch(st + pos, 2u);\n"
         "        return (int)pos;\n"
         "      }\n"
         "    }\n"
         "    u32 spins = 0;\n"
         "    while (s == 1u) {\n"
         "      if (++spins > (1u << 20)) { atomicExch(err, 1); return -2; }\n"
         "      __nanosleep(16);\n"
         "      s = gx_lds_acquire(st + pos);\n"
         "    }\n"
         "    if (*(volatile u32*)(nm + pos) == kn && " << same_keys("ks", "GXA_S", "pos") << ") return (int)pos;\n"
         "    pos = pos + 1u == GXA_S ? 0u : pos + 1u;\n"
         "  }\n"
         "  return -1;\n"
         "}\n";
    // the block's dictionary of groups with warp accumulators: the group's index,
    // -1 when it has none and no room is left, -2 after a wait gave up
    o << "__device__ int gxa_find_warp(u32* st, u32* nm, u64* ks, u32* at, u32* ng, const u32* room, const u64* kv, u32 kn, u64 h, int* err) {\n"
         "  u32 pos = (u32)h & (GXA_D - 1);\n"
         "  for (int pr = 0; pr < GXA_D; pr++) {\n"
         "    u32 s = gx_lds_acquire(st + pos);\n"
         "    if (s == 0u) {\n"
         "      if (*(volatile u32*)ng >= *(volatile const u32*)room) return -1;\n"
         "      s = atomicCAS(st + pos, 0u, 1u);\n"
         "      if (s == 0u) {\n"
         "        const u32 i = atomicAdd(ng, 1u);\n"
         "        if (i >= *(volatile const u32*)room) { atomicExch(st + pos, 0xffffffffu); return -1; }\n";  // lost the last place
    write_keys(o, "ks", "GXA_D", "pos", "        ");
    o << "        nm[pos] = kn; at[i] = pos;\n"
         "        __threadfence_block();\n"
         "        atomicExch(st + pos, 2u + i);\n"
         "        return (int)i;\n"
         "      }\n"
         "    }\n"
         "    u32 spins = 0;\n"
         "    while (s == 1u) {\n"
         "      if (++spins > (1u << 20)) { atomicExch(err, 1); return -2; }\n"
         "      __nanosleep(16);\n"
         "      s = gx_lds_acquire(st + pos);\n"
         "    }\n"
         "    if (s != 0xffffffffu && *(volatile u32*)(nm + pos) == kn && " << same_keys("ks", "GXA_D", "pos") << ") return (int)s - 2;\n"
         "    pos = (pos + 1u) & (GXA_D - 1);\n"
         "  }\n"
         "  return -1;\n"
         "}\n";
  }
  // the global table: -1 when the whole table was probed (overflow) or a wait gave
  // up.  A slot's state is read with acquire semantics: a fence instead would wait
  // for the atomics of the lane's earlier rows (100,000 groups, nine aggregations,
  // 2^24 rows 4456 -> 3277 us).  A slot's words lie in separate arrays: side by
  // side, a row's atomics meet in one sector and take turns (10,000 groups 1772 us,
  // 2644 side by side).
  o << "__device__ long long gxa_find_global(const GxAggArgs& g, const u64* kv, u32 kn, u64 h) {\n"
       "  u64 pos = h & (g.cap - 1ull);\n"
       "  for (u64 pr = 0; pr < g.cap; pr++) {\n"
       "    if ((pr & 63ull) == 63ull && *(volatile int*)g.overflow != 0) return -1;\n"  // the pass is repeated anyway
       "    u32 s = gx_ldg_acquire(g.state + pos);\n"
       "    if (s == 0u) {\n"
       "      s = atomicCAS(g.state + pos, 0u, 1u);\n"
       "      if (s == 0u) {\n";
  write_keys(o, "g.keys", "g.cap", "pos", "        ");
  for (int j = 0; j < na; j++)  // the table is not cleared: a claimed slot starts its accumulators
    o << "        g.acc[" << j << "ull * g.cap + pos] = " << agg_identity(L.kinds[j], false) << "; g.cnt[" << j
      << "ull * g.cap + pos] = 0ull;\n";
  o << "        g.nullm[pos] = kn; g.rows[pos] = 0ull;\n"
       "        g.list[atomicAdd(g.groups, 1ull)] = (u32)pos;\n"
       "        __threadfence();\n"
       "        atomicExch(g.state + pos, 2u);\n"
       "        return (long long)pos;\n"
       "      }\n"
       "      s = gx_ldg_acquire(g.state + pos);\n"
       "    }\n"
       "    u32 spins = 0;\n"
       "    while (s == 1u) {\n"
       "      if (++spins > (1u << 22)) { atomicExch(g.err, 1); return -1; }\n"
       "      __nanosleep(32);\n"
       "      s = gx_ldg_acquire(g.state + pos);\n"
       "    }\n"
       "    if (*(volatile u32*)(g.nullm + pos) == kn && " << same_keys("g.keys", "g.cap", "pos") << ") return (long long)pos;\n"
       "    pos = (pos + 1ull) & (g.cap - 1ull);\n"
       "  }\n"
       "  atomicExch(g.overflow, 1);\n"
       "  return -1;\n"
       "}\n";

  // per aggregation: value type, input value, identity, combine, atomic update
  struct AggCode {
    std::string ty, val, id, comb, atom;  // atom: format with @A@ (address) and @X@ (value)
  };
  std::vector<AggCode> ac(na);
  for (int j = 0; j < na; j++) {
    const int kind = L.kinds[j], in = L.in_nodes[j];
    const bool flt = in >= 0 && g.kind_f(in);
    AggCode& c = ac[j];
    if (kind == 4 || kind == 5) continue;  // counts only
    if (kind == 2 || kind == 3) {
      c.ty = "long long";
      c.val = flt ? "gx_ord64(" + g.B(in) + ")" : "(long long)(" + g.B(in) + ")";
      c.id = kind == 2 ? "(long long)0x7FFFFFFFFFFFFFFFull" : "(long long)0x8000000000000000ull";
      c.comb = kind == 2 ? "min" : "max";
      c.atom = kind == 2 ? "atomicMin((long long*)(@A@), @X@);" : "atomicMax((long long*)(@A@), @X@);";
    } else if (flt) {
      c.ty = "double";
      c.val = "__longlong_as_double((long long)(" + g.B(in) + "))";
      c.id = "0.0";
      c.comb = "+";
      c.atom = "atomicAdd((double*)(@A@), @X@);";
    } else {
      c.ty = "u64";
      c.val = "(u64)(" + g.B(in) + ")";
      c.id = "0ull";
      c.comb = "+";
      c.atom = "atomicAdd((unsigned long long*)(@A@), (unsigned long long)(@X@));";
    }
  }
  // the same in shared memory: 64-bit sums as two 32-bit atomics with the carry
  auto satom = [&](int j, const std::string& addr, const std::string& x) {
    if (ac[j].ty == "u64") return "gx_sadd64(" + addr + ", (u64)(" + x + "));";
    std::string r = ac[j].atom;
    r.replace(r.find("@A@"), 3, addr);
    r.replace(r.find("@X@"), 3, x);
    return r;
  };
  auto atom = [&](int j, const std::string& addr, const std::string& x) {
    std::string a = ac[j].atom;
    a.replace(a.find("@A@"), 3, addr);
    a.replace(a.find("@X@"), 3, x);
    return a;
  };
  auto combine = [&](int j, const std::string& x, const std::string& t) {
    if (ac[j].comb == "+") return x + " += " + t + ";";
    return x + " = " + ac[j].comb + "(" + x + ", " + t + ");";
  };
  std::vector<int> roots = L.key_nodes;
  for (int in : L.in_nodes)
    if (in >= 0) roots.push_back(in);
  const std::vector<int> row_ids = g.cone(roots);
  const std::vector<int> pred_ids = g.predicate_cone();

  o << "extern \"C\" __global__ void GX_LB " << name
    << "(const GxArgs a, const GxAggArgs ga) {\n";
  o << "  const int lane = threadIdx.x & 31; const int warp = threadIdx.x >> 5;\n";
  o << "  const i64 nwords = (a.n + 31) >> 5;\n";
  // ---- shared memory: the dictionary, then the warps' accumulators or the table
  // a cell: one 8-byte word per warp, group and replica, cell after cell
  o << "  const i64 nchunks = (nwords + GX_V - 1) / GX_V;\n";
  o << "  __shared__ unsigned short s_kept_[GX_WARPS][GX_V * 32];\n";
  o << "  __shared__ u32 s_ng_; __shared__ int s_over_;\n";
  o << "  u64* const d_ks_ = (u64*)gx_smem; u64* const d_gs_ = d_ks_ + GXA_NK * GXA_D;\n";
  o << "  u32* const d_st_ = (u32*)(d_gs_ + GXA_D); u32* const d_nm_ = d_st_ + GXA_D; u32* const d_at_ = d_nm_ + GXA_D;\n";
  o << "  u64* const s_warp_ = (u64*)(gx_smem + " << sh.dict_bytes << ");\n";
  if (sh.packed) {
    o << "  u64* const s_pk_ = s_warp_; u64* const s_acc_ = s_pk_ + GXA_S;\n";
    o << "  u32* const s_rows_ = (u32*)(s_acc_ + " << sh.accs << " * GXA_S); u32* const s_cnt_ = s_rows_ + GXA_S;\n";
  } else {
    o << "  u64* const s_ks_ = s_warp_; u64* const s_acc_ = s_ks_ + GXA_NK * GXA_S;\n";
    o << "  u32* const s_st_ = (u32*)(s_acc_ + " << sh.accs << " * GXA_S); u32* const s_nm_ = s_st_ + GXA_S;\n";
    o << "  u32* const s_rows_ = s_nm_ + GXA_S; u32* const s_cnt_ = s_rows_ + GXA_S;\n";
  }
  o << "  int mode_ = GXA_G > 0 ? 1 : 2;\n";
  // the split in use, groups and replicas of each (shared: it takes no register)
  o << "  __shared__ u32 s_room_; __shared__ int s_rep_;\n";
  o << "  if (threadIdx.x == 0) { s_room_ = GXA_G; s_rep_ = GXA_R; }\n";
  if (two) o << "  __shared__ u32 s_need_;\n";
  o << "  auto warps_init_ = [&]() {\n";
  o << "  for (int i = threadIdx.x; i < GXA_D; i += blockDim.x) { d_st_[i] = 0u;" << (sh.packed ? " d_ks_[i] = 0ull;" : "") << " }\n";
  o << "  if (threadIdx.x == 0) { s_ng_ = 0u; s_over_ = 0;" << (two ? " s_need_ = 0u;" : "") << " }\n";
  o << "  if (mode_ == 1) {\n";
  o << "    for (int i = threadIdx.x; i < GX_WARPS * GXA_GR; i += blockDim.x) {\n";
  for (int j = 0; j < na; j++) {
    if (sh.acc_cell[j] >= 0) o << "      s_warp_[" << sh.acc_cell[j] << " * GXA_CS + i] = " << agg_identity(L.kinds[j], false) << ";\n";
    if (sh.cnt_cell[j] >= 0) o << "      s_warp_[" << sh.cnt_cell[j] << " * GXA_CS + i] = 0ull;\n";
  }
  o << "      s_warp_[" << sh.rows_cell << " * GXA_CS + i] = 0ull;\n";
  o << "    }\n  }\n  };\n  warps_init_();\n";
  o << "  auto table_init_ = [&]() {\n";
  o << "    for (int i = threadIdx.x; i < GXA_S; i += blockDim.x) {\n";
  o << "      " << (sh.packed ? "s_pk_[i] = 0ull" : "s_st_[i] = 0u") << "; s_rows_[i] = 0u;\n";
  for (int j = 0; j < na; j++) {
    if (sh.acc_slot[j] >= 0) o << "      s_acc_[" << sh.acc_slot[j] << " * GXA_S + i] = " << agg_identity(L.kinds[j], false) << ";\n";
    if (sh.cnt_slot[j] >= 0) o << "      s_cnt_[" << sh.cnt_slot[j] << " * GXA_S + i] = 0u;\n";
  }
  o << "    }\n  };\n";
  o << "  if (mode_ == 2) table_init_();\n";
  o << "  __syncthreads();\n";
  // chunk tickets are drawn by lane 0, one ahead of their use
  o << "  unsigned long long tk_ = 0ull;\n";
  o << "  if (lane == 0) tk_ = atomicAdd(a.tile_counter, 1ull);\n";
  o << "  i64 chunk_ = (i64)__shfl_sync(GX_FULL, tk_, 0);\n";
  // a chunk left in its middle for the block's change to its table: its ticket
  // is kept, and its first skip_ kept rows are done
  o << "  u32 skip_ = 0u; bool full_ = false;\n";
  o << "  while (true) {\n";
  o << "  while (chunk_ < nchunks) {\n";
  o << "    if (mode_ == 1 && __any_sync(GX_FULL, *(volatile int*)&s_over_ != 0)) break;\n";
  o << "    if (lane == 0 && !full_) tk_ = atomicAdd(a.tile_counter, 1ull);\n";
  o << "    const i64 w0 = chunk_ * GX_V;\n";
  o << "    u32 bal[GX_V];\n";
  o << "    {\n";
  if (p.has_filter()) {
    g.decl(o, pred_ids, "      ");
    g.emit_predicate(o, "      ");
  } else {
    o << "      bool alive[GX_V];\n";
    o << "      #pragma unroll\n      for (int k = 0; k < GX_V; k++) alive[k] = (w0 + k) * 32 + lane < a.n;\n";
  }
  o << "      #pragma unroll\n      for (int k = 0; k < GX_V; k++) bal[k] = __ballot_sync(GX_FULL, alive[k]);\n";
  o << "    }\n";
  o << "    u32 total_ = 0u;\n";
  o << "    unsigned short* const kl_ = s_kept_[warp];\n";
  emit_kept_list(o, "bal", "kl_", "total_", "    ");
  o << "    __syncwarp();\n";
  {
    std::vector<int> cols;
    for (const auto& ids : {pred_ids, row_ids})
      for (int id : ids)
        if (p.nodes[id].kind == Node::COL && std::find(cols.begin(), cols.end(), p.nodes[id].col) == cols.end())
          cols.push_back(p.nodes[id].col);
    // The next chunk's columns are brought into L2 while this one's rows are
    // combined: with 32 warps on an SM (one block, whose tables fill its shared
    // memory) a round mostly waits for its loads.  Lane i takes column i; not for
    // a chunk of which less than a quarter is kept, where most bytes would go
    // unread.  Kernel us without and with: 2557 dates 340 / 332, two flag columns
    // at 2^26 rows 1270 / 1243.
    if (!cols.empty() && cols.size() <= 32) {
      o << "    {\n      const i64 nx_ = (i64)__shfl_sync(GX_FULL, tk_, 0);\n";
      o << "      if (total_ >= GX_V * 8u && (nx_ + 1) * (GX_V * 32) <= a.n) {\n";
      o << "        const char* q_ = nullptr; u32 w_ = 0u;\n";
      for (size_t i = 0; i < cols.size(); i++)
        o << "        if (lane == " << i << ") { q_ = (const char*)a.in_data[" << cols[i] << "]; w_ = "
          << type_size(p.schema[cols[i]]) << "u; }\n";
      o << "        if (w_) gx_prefetch_l2(q_ + nx_ * (i64)(GX_V * 32u * w_), GX_V * 32u * w_);\n";
      o << "      }\n    }\n";
    }
  }
  g.masks_ = Gen::Masks::KEPT;
  g.emit_mask_words(o, row_ids, {}, "    ");
  o << "    full_ = false;\n";
  o << "    for (u32 base_ = skip_; base_ < total_; base_ += 32u) {\n";
  const std::string in2 = "      ";
  o << in2 << "const u32 t_ = base_ + (u32)lane; const bool act = t_ < total_;\n";
  o << in2 << "const u64 pos = 0ull;\n";
  emit_rank_to_row(o, in2);
  emit_row_nodes(o, g, p, row_ids, {}, in2);
  o << in2 << "u64 kv[GXA_NK]; u32 kn_ = 0u; kv[0] = 0ull;\n";
  for (int j = 0; j < nk; j++) {
    const int id = L.key_nodes[j];
    o << in2 << "kv[" << j << "] = " << g.V(id) << " ? (u64)(" << g.B(id) << ") : 0ull; if (!(" << g.V(id)
      << ")) kn_ |= " << (1u << j) << "u;\n";
  }
  o << in2 << (sh.packed ? "const u64 pk_ = gxa_pack(kv, kn_);\n" : "const u64 h_ = gxa_hash(kv, kn_);\n");
  for (int j = 0; j < na; j++) {
    const int in = L.in_nodes[j];
    o << in2 << "const bool ok" << j << "_ = " << (in >= 0 ? g.V(in) : std::string("true")) << ";\n";
    if (!ac[j].ty.empty()) o << in2 << "const " << ac[j].ty << " in" << j << "_ = " << ac[j].val << ";\n";
  }
  auto in_ = [](int j) { return "in" + std::to_string(j) + "_"; };
  auto ok_ = [](int j) { return "ok" + std::to_string(j) + "_"; };
  o << in2 << "int sl_ = -3;\n";
  if (sh.packed)
    o << in2 << "if (act) sl_ = mode_ == 1 ? gxa_find_dict(d_st_, d_ks_, d_at_, &s_ng_, &s_room_, pk_, ga.err) : gxa_find_table(s_pk_, pk_);\n";
  else
    o << in2 << "if (act) sl_ = mode_ == 1 ? gxa_find_warp(d_st_, d_nm_, d_ks_, d_at_, &s_ng_, &s_room_, kv, kn_, h_, ga.err)\n"
      << in2 << "                          : gxa_find_smem(s_st_, s_nm_, s_ks_, kv, kn_, h_, ga.err);\n";
  // a group without warp accumulators: the round is left for the table
  o << in2 << "if (mode_ == 1 && __any_sync(GX_FULL, sl_ == -1 || *(volatile int*)&s_over_ != 0)) {\n";
  o << in2 << "  *(volatile int*)&s_over_ = 1; skip_ = base_; full_ = true;\n";
  if (two) {  // the groups of these 32 rows tell how many there may be
    o << in2 << "  const u32 same_ = __match_any_sync(GX_FULL, " << (sh.packed ? "pk_" : "h_") << ");\n";
    o << in2 << "  const u32 seen_ = (u32)__popc(__ballot_sync(GX_FULL, act && (same_ & ((1u << lane) - 1u)) == 0u));\n";
    o << in2 << "  if (lane == 0) atomicMax(&s_need_, seen_);\n";
  }
  o << in2 << "  break;\n" << in2 << "}\n";
  o << in2 << "const bool sm_ = sl_ >= 0;\n";
  auto direct = [&](const std::string& ind) {
    o << ind << "if (sm_) {\n";
    o << ind << "  atomicAdd(&s_rows_[sl_], 1u);\n";
    for (int j = 0; j < na; j++) {
      const bool never = (rows_cnt >> j) & 1ull;
      o << ind << "  " << (never ? "{" : "if (" + ok_(j) + ") {");
      if (sh.cnt_slot[j] >= 0) o << " atomicAdd(&s_cnt_[" << sh.cnt_slot[j] << " * GXA_S + sl_], 1u);";
      if (sh.acc_slot[j] >= 0) o << " " << satom(j, "&s_acc_[" + std::to_string(sh.acc_slot[j]) + " * GXA_S + sl_]", in_(j));
      o << " }\n";
    }
    o << ind << "}\n";
  };
  o << in2 << "const u32 peers_ = __match_any_sync(GX_FULL, sm_ ? (u32)sl_ : (0x80000000u | (u32)lane));\n";
  o << in2 << "const int mx_ = (int)__reduce_max_sync(GX_FULL, (u32)__popc(peers_));\n";
  auto update = [&](const std::string& ind, const std::string& rows, const std::string& cnt,
                    const std::string& val, bool guard) {
    o << ind << "c_[" << sh.rows_cell << " * GXA_CS] += " << rows << ";\n";
    for (int j = 0; j < na; j++) {
      const std::string js = std::to_string(j) + "_";
      const bool g2 = guard && !((rows_cnt >> j) & 1ull);
      if (g2) o << ind << "if (ok" << js << ") {\n";
      if (sh.cnt_cell[j] >= 0) o << ind << "c_[" << sh.cnt_cell[j] << " * GXA_CS] += " << (guard ? "1ull" : "(u64)" + cnt + js) << ";\n";
      if (sh.acc_cell[j] >= 0) {
        const std::string x = val + js;
        o << ind << "{ " << ac[j].ty << "* const q_ = (" << ac[j].ty << "*)(c_ + " << sh.acc_cell[j] << " * GXA_CS); *q_ = "
          << (ac[j].comb == "+" ? "*q_ + " + x : ac[j].comb + "(*q_, " + x + ")") << "; }\n";
      }
      if (g2) o << ind << "}\n";
    }
  };
  o << in2 << "const int rep_ = " << (two ? "*(volatile int*)&s_rep_" : "GXA_R") << ";\n";
  o << in2 << "if (mode_ == 1 && mx_ <= 3 * rep_) {\n";
  o << in2 << "  const int rank_ = __popc(peers_ & ((1u << lane) - 1u));\n";
  o << in2 << "  for (int p_ = 0; p_ < mx_; p_ += rep_) {\n";
  o << in2 << "    if (sm_ && (u32)(rank_ - p_) < (u32)rep_) {\n";
  o << in2 << "      u64* const c_ = s_warp_ + warp * GXA_GR + sl_ * rep_ + (rank_ - p_);\n";
  update(in2 + "      ", "1ull", "", "in", true);
  o << in2 << "    }\n";
  o << in2 << "    __syncwarp();\n";  // the next pass's lanes update the same words
  o << in2 << "  }\n";
  o << in2 << "} else if (mode_ == 2 && " << (L.warp_combine ? "mx_ <= 2" : "true") << ") {\n";
  direct(in2 + "  ");
  o << in2 << "} else {\n";
  {
    const std::string i4 = in2 + "  ";
    o << i4 << "GxPeers pr_; pr_.init(peers_);\n";
    for (int j = 0; j < na; j++) {
      o << i4 << "const bool vl" << j << "_ = sm_ && " << ok_(j) << ";\n";
      if (sh.cnt_slot[j] >= 0)
        o << i4 << "const u32 c" << j << "_ = (u32)__popc(__ballot_sync(GX_FULL, vl" << j << "_) & peers_);\n";
      if (!ac[j].ty.empty())
        o << i4 << ac[j].ty << " x" << j << "_ = vl" << j << "_ ? " << in_(j) << " : " << ac[j].id << ";\n";
    }
    // a tree over each group's lanes: log2 of the largest group's lanes steps
    o << i4 << "#pragma unroll\n" << i4 << "for (int s_ = 1; s_ < 32; s_ <<= 1) {\n";
    o << i4 << "  if (s_ >= mx_) break;\n";
    o << i4 << "  const int src_ = pr_.partner(); const bool rcv_ = pr_.receives(s_);\n";
    for (int j = 0; j < na; j++) {
      if (ac[j].ty.empty()) continue;
      o << i4 << "  { const " << ac[j].ty << " t2_ = __shfl_sync(GX_FULL, x" << j << "_, src_); if (rcv_) "
        << combine(j, "x" + std::to_string(j) + "_", "t2_") << " }\n";
    }
    o << i4 << "  pr_.step(s_);\n";
    o << i4 << "}\n";
    o << i4 << "if (sm_ && pr_.rank == 0) {\n";
    o << i4 << "  if (mode_ == 1) {\n";
    o << i4 << "    u64* const c_ = s_warp_ + warp * GXA_GR + sl_ * rep_;\n";
    update(i4 + "    ", "(u64)__popc(peers_)", "c", "x", false);
    o << i4 << "  } else {\n";
    o << i4 << "    atomicAdd(&s_rows_[sl_], (u32)__popc(peers_));\n";
    for (int j = 0; j < na; j++) {
      const std::string xj = "x" + std::to_string(j) + "_";
      if (sh.cnt_slot[j] >= 0)
        o << i4 << "    if (c" << j << "_ != 0u) atomicAdd(&s_cnt_[" << sh.cnt_slot[j] << " * GXA_S + sl_], c" << j << "_);\n";
      if (sh.acc_slot[j] >= 0)
        o << i4 << "    " << satom(j, "&s_acc_[" + std::to_string(sh.acc_slot[j]) + " * GXA_S + sl_]", xj) << "\n";
    }
    o << i4 << "  }\n";
    o << i4 << "}\n";
    o << i4 << "__syncwarp();\n";  // a slot's next update in this warp comes from another lane
  }
  o << in2 << "}\n";
  // rows whose group found no room in the block go to the global table
  o << in2 << "if (mode_ == 2 && act && sl_ == -1) {\n";
  o << in2 << "  const long long gs_ = gxa_find_global(ga, kv, kn_, " << (sh.packed ? "gxa_hash(kv, kn_)" : "h_") << ");\n";
  o << in2 << "  if (gs_ >= 0) {\n";
  o << in2 << "    atomicAdd((unsigned long long*)(ga.rows + gs_), 1ull);\n";
  for (int j = 0; j < na; j++) {
    o << in2 << "    if (" << ok_(j) << ") {\n";
    if (!((rows_cnt >> j) & 1ull))
      o << in2 << "      atomicAdd((unsigned long long*)(ga.cnt + " << j << "ull * ga.cap + gs_), 1ull);\n";
    if (!ac[j].ty.empty())
      o << in2 << "      " << atom(j, "ga.acc + " + std::to_string(j) + "ull * ga.cap + gs_", in_(j)) << "\n";
    o << in2 << "    }\n";
  }
  o << in2 << "  }\n";
  o << in2 << "}\n";
  o << "    }\n";  // rounds
  o << "    __syncwarp();\n";  // the kept-row list is rewritten by the next chunk
  o << "    if (full_) break;\n";
  o << "    skip_ = 0u;\n";
  o << "    chunk_ = (i64)__shfl_sync(GX_FULL, tk_, 0);\n";
  o << "  }\n";  // chunks
  o << "  __syncthreads();\n";
  // ---- merge into the global table
  o << "  if (mode_ == 1) {\n";
  o << "    const int ng_ = (int)min(s_ng_, s_room_); const int rep_ = s_rep_;\n";
  // a thread per group (a block of one warp has fewer threads than groups, so it goes round)
  o << (cfg.warps * 32 >= kAggGroups ? "    if ((int)threadIdx.x < ng_) {\n      const int gi = (int)threadIdx.x;\n"
                                     : "    for (int gi = (int)threadIdx.x; gi < ng_; gi += GX_WARPS * 32) {\n");
  o << "      const u32 i = d_at_[gi];\n";
  o << "      u64 rows_ = 0ull;\n";  // none: its only round was left for the table
  o << "      for (int w = 0; w < GX_WARPS; w++)\n        for (int r = 0; r < rep_; r++)\n"
       "          rows_ += s_warp_[" << sh.rows_cell << " * GXA_CS + w * GXA_GR + gi * rep_ + r];\n";
  o << "      u64 kv[GXA_NK]; kv[0] = 0ull;\n";
  if (sh.packed) {
    o << "      const u32 kn_ = gxa_unpack(d_ks_[i], kv);\n";
  } else {
    for (int j = 0; j < nk; j++) o << "      kv[" << j << "] = d_ks_[" << j << " * GXA_D + i];\n";
    o << "      const u32 kn_ = d_nm_[i];\n";
  }
  o << "      d_gs_[gi] = rows_ ? (u64)gxa_find_global(ga, kv, kn_, gxa_hash(kv, kn_)) : ~0ull;\n";
  o << "    }\n";
  o << "    __syncthreads();\n";
  // one warp per group and cell: lane w takes warp w's replicas, then a tree over lanes
  auto merge_warps = [&](const std::string& ty, const std::string& id, const std::string& comb, int cell,
                         const std::string& store) {
    o << "    for (int gi = (warp + " << cell << ") % GX_WARPS; gi < ng_; gi += GX_WARPS) {\n";
    o << "      const long long gs_ = (long long)d_gs_[gi];\n";
    o << "      " << ty << " x = " << id << ";\n";
    o << "      if (lane < GX_WARPS) for (int r = 0; r < rep_; r++) { const " << ty << " y = *(const " << ty << "*)(s_warp_ + "
      << cell << " * GXA_CS + lane * GXA_GR + gi * rep_ + r); x = " << (comb == "+" ? "x + y" : comb + "(x, y)") << "; }\n";
    o << "      #pragma unroll\n      for (int d = 16; d > 0; d >>= 1) { const " << ty
      << " y = __shfl_xor_sync(GX_FULL, x, d); x = " << (comb == "+" ? "x + y" : comb + "(x, y)") << "; }\n";
    o << "      if (lane == 0 && gs_ >= 0) " << store << "\n";
    o << "    }\n";
  };
  merge_warps("u64", "0ull", "+", sh.rows_cell, "atomicAdd((unsigned long long*)(ga.rows + gs_), (unsigned long long)x);");
  for (int j = 0; j < na; j++) {
    if (sh.cnt_cell[j] >= 0)
      merge_warps("u64", "0ull", "+", sh.cnt_cell[j],
                 "atomicAdd((unsigned long long*)(ga.cnt + " + std::to_string(j) + "ull * ga.cap + gs_), (unsigned long long)x);");
    if (sh.acc_cell[j] >= 0)
      merge_warps(ac[j].ty, ac[j].id, ac[j].comb, sh.acc_cell[j],
                 atom(j, "ga.acc + " + std::to_string(j) + "ull * ga.cap + gs_", "x"));
  }
  o << "  } else {\n";
  o << "    for (int i = threadIdx.x; i < GXA_S; i += blockDim.x) {\n";
  o << "      if (s_rows_[i] == 0u" << (sh.packed ? "" : " || s_st_[i] != 2u") << ") continue;\n";
  o << "      u64 kv[GXA_NK]; kv[0] = 0ull;\n";
  if (sh.packed) {
    o << "      const u32 kn_ = gxa_unpack(s_pk_[i], kv);\n";
  } else {
    for (int j = 0; j < nk; j++) o << "      kv[" << j << "] = s_ks_[" << j << " * GXA_S + i];\n";
    o << "      const u32 kn_ = s_nm_[i];\n";
  }
  o << "      const long long gs_ = gxa_find_global(ga, kv, kn_, gxa_hash(kv, kn_));\n";
  o << "      if (gs_ < 0) continue;\n";
  o << "      atomicAdd((unsigned long long*)(ga.rows + gs_), (unsigned long long)s_rows_[i]);\n";
  for (int j = 0; j < na; j++) {
    if (sh.cnt_slot[j] >= 0)
      o << "      if (s_cnt_[" << sh.cnt_slot[j] << " * GXA_S + i] != 0u) atomicAdd((unsigned long long*)(ga.cnt + " << j
        << "ull * ga.cap + gs_), (unsigned long long)s_cnt_[" << sh.cnt_slot[j] << " * GXA_S + i]);\n";
    if (sh.acc_slot[j] < 0) continue;
    const std::string c = "s_acc_[" + std::to_string(sh.acc_slot[j]) + " * GXA_S + i]";
    const std::string x = ac[j].ty == "double" ? "__longlong_as_double((long long)" + c + ")"
                        : ac[j].ty == "long long" ? "(long long)" + c : c;
    o << "      " << atom(j, "ga.acc + " + std::to_string(j) + "ull * ga.cap + gs_", x) << "\n";
  }
  o << "    }\n";
  o << "  }\n";
  o << "  if (mode_ == 2 || s_over_ == 0) break;\n";
  if (two) {
    o << "  __syncthreads();\n";
    o << "  if (threadIdx.x == 0) gxa_next_split(&s_room_, &s_rep_, s_need_);\n";
    o << "  __syncthreads();\n";
    o << "  if (s_rep_ > 0) warps_init_();\n";
    o << "  else { mode_ = 2; table_init_(); }\n";
  } else {
    o << "  __syncthreads();\n";
    o << "  mode_ = 2;\n";
    o << "  table_init_();\n";
  }
  o << "  __syncthreads();\n";
  o << "  }\n";
  o << "}\n";
  return o.str();
}
}  // namespace gx
