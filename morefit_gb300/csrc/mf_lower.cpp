// Lowering of MoreFit kernel expressions to CUDA C (see mf_lower.h).
#include "mf_lower.h"

#include <cctype>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <functional>
#include <set>
#include <sstream>
#include <stdexcept>

namespace mf {

// REDUCE kernels with more than kAccRegMax outputs keep the per-thread
// partials of as many outputs as fit in kAccSmemBytes of shared memory per
// block there (the last ones), and at least kAccRegMin in registers.
constexpr int kAccRegMax = 64, kAccRegMin = 8;
constexpr size_t kAccSmemBytes = 40 * 1024;

namespace {

bool is_unary_fn(Op op) {
  switch (op) {
    case Op::Exp: case Op::Log: case Op::Sqrt: case Op::Sin: case Op::Cos: case Op::Tan:
    case Op::Asin: case Op::Acos: case Op::Atan: case Op::Erf:
      return true;
    default:
      return false;
  }
}

double apply_unary(Op op, double x) {
  switch (op) {
    case Op::Neg: return -x;
    case Op::Rcp: return 1.0 / x;
    case Op::Exp: return std::exp(x);
    case Op::Log: return std::log(x);
    case Op::Sqrt: return std::sqrt(x);
    case Op::Sin: return std::sin(x);
    case Op::Cos: return std::cos(x);
    case Op::Tan: return std::tan(x);
    case Op::Asin: return std::asin(x);
    case Op::Acos: return std::acos(x);
    case Op::Atan: return std::atan(x);
    case Op::Erf: return std::erf(x);
    default: throw std::runtime_error("not a unary op");
  }
}

double apply_binary(Op op, double a, double b) {
  switch (op) {
    case Op::Add: return a + b;
    case Op::Sub: return a - b;
    case Op::Mul: return a * b;
    case Op::Div: return a / b;
    case Op::Pow: return std::pow(a, b);
    default: throw std::runtime_error("not a binary op");
  }
}

bool apply_cmp(CmpOp c, double a, double b) {
  switch (c) {
    case CmpOp::Eq: return a == b;
    case CmpOp::Ne: return a != b;
    case CmpOp::Gt: return a > b;
    case CmpOp::Lt: return a < b;
    case CmpOp::Ge: return a >= b;
    case CmpOp::Le: return a <= b;
  }
  return false;
}

// ---------------------------------------------------------------- parser --
class Parser {
 public:
  Parser(Dag& dag, const std::string& s) : dag_(dag), s_(s) {}
  int run() {
    int r = expr();
    skip();
    if (p_ != s_.size()) fail("trailing characters");
    return r;
  }

 private:
  [[noreturn]] void fail(const std::string& what) {
    std::ostringstream m;
    m << "expression parse error (" << what << ") at offset " << p_ << " of \"" << s_.substr(0, 200)
      << (s_.size() > 200 ? "..." : "") << "\"";
    throw std::runtime_error(m.str());
  }
  void skip() {
    while (p_ < s_.size() && std::isspace((unsigned char)s_[p_])) p_++;
  }
  bool eat(const char* t) {
    skip();
    size_t n = std::strlen(t);
    if (s_.compare(p_, n, t) == 0) {
      p_ += n;
      return true;
    }
    return false;
  }
  int expr() {
    int c = comparison();
    if (eat("?")) {
      int a = expr();
      if (!eat(":")) fail("expected ':'");
      int b = expr();
      return dag_.select(c, a, b);
    }
    return c;
  }
  int comparison() {
    int a = additive();
    skip();
    static const struct { const char* t; CmpOp c; } ops[] = {{"==", CmpOp::Eq}, {"!=", CmpOp::Ne},
                                                             {">=", CmpOp::Ge}, {"<=", CmpOp::Le},
                                                             {">", CmpOp::Gt},  {"<", CmpOp::Lt}};
    for (auto& o : ops)
      if (eat(o.t)) return dag_.compare(o.c, a, additive());
    return a;
  }
  int additive() {
    int a = multiplicative();
    for (;;) {
      if (eat("+"))
        a = dag_.binary(Op::Add, a, multiplicative());
      else if (peek_binary_minus())
        a = dag_.binary(Op::Sub, a, multiplicative());
      else
        return a;
    }
  }
  bool peek_binary_minus() {
    skip();
    if (p_ < s_.size() && s_[p_] == '-') {
      p_++;
      return true;
    }
    return false;
  }
  int multiplicative() {
    int a = unary();
    for (;;) {
      if (eat("*"))
        a = dag_.binary(Op::Mul, a, unary());
      else if (eat("/"))
        a = dag_.binary(Op::Div, a, unary());
      else
        return a;
    }
  }
  int unary() {
    skip();
    if (eat("-")) return dag_.unary(Op::Neg, unary());
    if (eat("+")) return unary();
    return primary();
  }
  int primary() {
    skip();
    if (p_ >= s_.size()) fail("unexpected end");
    char ch = s_[p_];
    if (ch == '(') {
      p_++;
      int r = expr();
      if (!eat(")")) fail("expected ')'");
      return r;
    }
    if (std::isdigit((unsigned char)ch) || ch == '.') return number();
    if (std::isalpha((unsigned char)ch) || ch == '_') {
      size_t b = p_;
      while (p_ < s_.size() && (std::isalnum((unsigned char)s_[p_]) || s_[p_] == '_')) p_++;
      std::string id = s_.substr(b, p_ - b);
      skip();
      if (p_ < s_.size() && s_[p_] == '(') {
        p_++;
        std::vector<int> args;
        args.push_back(expr());
        while (eat(",")) args.push_back(expr());
        if (!eat(")")) fail("expected ')' after arguments");
        return call(id, args);
      }
      return variable(id);
    }
    fail(std::string("unexpected character '") + ch + "'");
  }
  int number() {
    const char* start = s_.c_str() + p_;
    char* end = nullptr;
    double v = std::strtod(start, &end);
    if (end == start) fail("bad number");
    p_ += size_t(end - start);
    return dag_.constant(v);
  }
  int call(const std::string& f, const std::vector<int>& a) {
    static const std::map<std::string, Op> fns = {
        {"exp", Op::Exp},   {"log", Op::Log},   {"sqrt", Op::Sqrt}, {"sin", Op::Sin},   {"cos", Op::Cos},
        {"tan", Op::Tan},   {"asin", Op::Asin}, {"acos", Op::Acos}, {"atan", Op::Atan}, {"erf", Op::Erf}};
    auto it = fns.find(f);
    if (it != fns.end()) {
      if (a.size() != 1) fail("wrong argument count for " + f);
      return dag_.unary(it->second, a[0]);
    }
    if (f == "pow") {
      if (a.size() != 2) fail("pow takes two arguments");
      return dag_.binary(Op::Pow, a[0], a[1]);
    }
    fail("unknown function " + f);
  }
  int variable(const std::string& id);

  Dag& dag_;
  const std::string& s_;
  size_t p_ = 0;
};

}  // namespace

// ------------------------------------------------------------------- DAG --
Dag::Dag(const std::vector<std::string>& inputs, const std::vector<std::string>& params)
    : inputs_(inputs), params_(params) {
  for (size_t i = 0; i < inputs.size(); i++) input_idx_[inputs[i]] = int(i);
  for (size_t i = 0; i < params.size(); i++)
    if (!param_idx_.count(params[i])) param_idx_[params[i]] = int(i);
}

int Parser::variable(const std::string& id) {
  // Input columns shadow parameters of the same name (the reference declares
  // parameters first and events inside the loop, compute_llvm.hh:601-646).
  auto& in = dag_.input_names();
  for (size_t i = 0; i < in.size(); i++)
    if (in[i] == id) return dag_.unary(Op::Input, int(i));
  auto& pa = dag_.param_names();
  for (size_t i = 0; i < pa.size(); i++)
    if (pa[i] == id) return dag_.unary(Op::Param, int(i));
  fail("unknown variable '" + id + "'");
}

// A node's fields as bytes.
static std::string node_key(const Node& n) {
  uint64_t bits;
  std::memcpy(&bits, &n.value, sizeof bits);
  const uint64_t k[4] = {(uint64_t(n.op) << 8) | uint64_t(n.cmp), bits,
                         (uint64_t(uint32_t(n.index)) << 32) | uint32_t(n.a),
                         (uint64_t(uint32_t(n.b)) << 32) | uint32_t(n.c)};
  return std::string(reinterpret_cast<const char*>(k), sizeof k);
}

int Dag::find(const Node& n) const {
  auto it = table_.find(node_key(n));
  return it != table_.end() ? it->second : -1;
}

int Dag::intern(const Node& n) {
  const std::string key = node_key(n);
  auto it = table_.find(key);
  if (it != table_.end()) return it->second;
  nodes_.push_back(n);
  int id = int(nodes_.size()) - 1;
  table_[key] = id;
  return id;
}

int Dag::constant(double v) {
  Node n;
  n.op = Op::Const;
  n.value = v;
  return intern(n);
}

static bool is_const(const std::vector<Node>& ns, int id, double v) {
  return ns[id].op == Op::Const && ns[id].value == v;
}

int Dag::unary(Op op, int a) {
  if (op == Op::Input || op == Op::Param) {
    Node n;
    n.op = op;
    n.index = a;
    n.uniform = (op == Op::Param);
    return intern(n);
  }
  const Node& x = nodes_[a];
  if (x.op == Op::Const) return constant(apply_unary(op, x.value));
  if (op == Op::Neg && x.op == Op::Neg) return x.a;  // -(-y) = y exactly
  Node n;
  n.op = op;
  n.a = a;
  n.uniform = x.uniform;
  return intern(n);
}

int Dag::binary(Op op, int a, int b) {
  const Node& x = nodes_[a];
  const Node& y = nodes_[b];
  if (x.op == Op::Const && y.op == Op::Const) return constant(apply_binary(op, x.value, y.value));
  switch (op) {
    case Op::Add:
      if (y.op == Op::Neg) return binary(Op::Sub, a, y.a);  // a + (-b) = a - b exactly
      break;
    case Op::Mul:
      if (is_const(nodes_, b, 1.0)) return a;  // exact
      if (is_const(nodes_, a, 1.0)) return b;
      if (is_const(nodes_, b, -1.0)) return unary(Op::Neg, a);
      if (is_const(nodes_, a, -1.0)) return unary(Op::Neg, b);
      break;
    case Op::Div:
      if (is_const(nodes_, b, 1.0)) return a;
      // x / y -> x * (1/y): the reciprocal of a shared denominator (the
      // density in every gradient output) is computed once per event.
      if (is_const(nodes_, a, 1.0)) return unary(Op::Rcp, b);
      return binary(Op::Mul, a, unary(Op::Rcp, b));
    case Op::Pow:
      if (is_const(nodes_, b, 1.0)) return a;
      if (is_const(nodes_, b, 2.0)) return binary(Op::Mul, a, a);  // pow(x,2) and x*x round identically
      break;
    default:
      break;
  }
  Node n;
  n.op = op;
  n.a = a;
  n.b = b;
  n.uniform = x.uniform && y.uniform;
  if (share_exchanged && (op == Op::Add || op == Op::Mul)) {  // the same sum or product with its operands exchanged
    Node m = n;
    m.a = b;
    m.b = a;
    const int known = find(m);
    if (known >= 0) return known;
  }
  return intern(n);
}

int Dag::compare(CmpOp c, int a, int b) {
  const Node& x = nodes_[a];
  const Node& y = nodes_[b];
  if (x.op == Op::Const && y.op == Op::Const) return constant(apply_cmp(c, x.value, y.value) ? 1.0 : 0.0);
  Node n;
  n.op = Op::Cmp;
  n.cmp = c;
  n.a = a;
  n.b = b;
  n.uniform = x.uniform && y.uniform;
  return intern(n);
}

int Dag::select(int cond, int a, int b) {
  const Node& c = nodes_[cond];
  if (c.op == Op::Const) return c.value != 0.0 ? a : b;
  if (a == b) return a;
  Node n;
  n.op = Op::Select;
  n.a = cond;
  n.b = a;
  n.c = b;
  n.uniform = c.uniform && nodes_[a].uniform && nodes_[b].uniform;
  return intern(n);
}

int Dag::parse(const std::string& expr) {
  Parser p(*this, expr);
  return p.run();
}

void Dag::eval_all(const double* pa, size_t np, std::vector<double>& v) const {
  v.resize(nodes_.size());
  for (size_t i = 0; i < nodes_.size(); i++) {
    const Node& n = nodes_[i];
    switch (n.op) {
      case Op::Const: v[i] = n.value; break;
      case Op::Input: v[i] = 0.0; break;
      case Op::Param: v[i] = size_t(n.index) < np ? pa[n.index] : 0.0; break;
      case Op::Add: case Op::Sub: case Op::Mul: case Op::Div: case Op::Pow:
        v[i] = apply_binary(n.op, v[n.a], v[n.b]);
        break;
      case Op::Cmp: v[i] = apply_cmp(n.cmp, v[n.a], v[n.b]) ? 1.0 : 0.0; break;
      case Op::Select: v[i] = v[n.a] != 0.0 ? v[n.b] : v[n.c]; break;
      default: v[i] = apply_unary(n.op, v[n.a]); break;
    }
  }
}

double Dag::eval(int id, const std::vector<double>& in, const std::vector<double>& pa) const {
  const Node& n = nodes_[id];
  switch (n.op) {
    case Op::Const: return n.value;
    case Op::Input: return in.at(n.index);
    case Op::Param: return pa.at(n.index);
    case Op::Add: case Op::Sub: case Op::Mul: case Op::Div: case Op::Pow:
      return apply_binary(n.op, eval(n.a, in, pa), eval(n.b, in, pa));
    case Op::Cmp: return apply_cmp(n.cmp, eval(n.a, in, pa), eval(n.b, in, pa)) ? 1.0 : 0.0;
    case Op::Select: return eval(n.a, in, pa) != 0.0 ? eval(n.b, in, pa) : eval(n.c, in, pa);
    default: return apply_unary(n.op, eval(n.a, in, pa));
  }
}

// -------------------------------------------------------------- emitter --
namespace {

std::string fmt_const(double v, bool f32) {
  char buf[64];
  if (std::isnan(v)) return f32 ? "__int_as_float(0x7fc00000)" : "__longlong_as_double(0x7ff8000000000000ULL)";
  if (std::isinf(v)) {
    if (f32) return v > 0 ? "__int_as_float(0x7f800000)" : "__int_as_float(0xff800000)";
    return v > 0 ? "__longlong_as_double(0x7ff0000000000000ULL)" : "__longlong_as_double(0xfff0000000000000ULL)";
  }
  if (f32)
    std::snprintf(buf, sizeof buf, "%.9ef", double(float(v)));
  else
    std::snprintf(buf, sizeof buf, "%.17e", v);
  std::string s(buf);
  return v < 0 ? "(" + s + ")" : s;
}

const char* fn_name(Op op, bool f32) {
  switch (op) {
    case Op::Exp: return f32 ? "expf" : "exp";
    case Op::Log: return f32 ? "logf" : "log";
    case Op::Sqrt: return f32 ? "sqrtf" : "sqrt";
    case Op::Sin: return f32 ? "sinf" : "sin";
    case Op::Cos: return f32 ? "cosf" : "cos";
    case Op::Tan: return f32 ? "tanf" : "tan";
    case Op::Asin: return f32 ? "asinf" : "asin";
    case Op::Acos: return f32 ? "acosf" : "acos";
    case Op::Atan: return f32 ? "atanf" : "atan";
    case Op::Erf: return f32 ? "erff" : "erf";
    case Op::Pow: return f32 ? "powf" : "pow";
    case Op::Rcp: return f32 ? "__frcp_rn" : "__drcp_rn";
    default: return "?";
  }
}

const char* cmp_str(CmpOp c) {
  switch (c) {
    case CmpOp::Eq: return "==";
    case CmpOp::Ne: return "!=";
    case CmpOp::Gt: return ">";
    case CmpOp::Lt: return "<";
    case CmpOp::Ge: return ">=";
    case CmpOp::Le: return "<=";
  }
  return "==";
}

// Marks the nodes reachable from `roots`.
std::vector<char> reachable(const std::vector<Node>& ns, const std::vector<int>& roots) {
  std::vector<char> r(ns.size(), 0);
  std::vector<int> st(roots.begin(), roots.end());
  while (!st.empty()) {
    int id = st.back();
    st.pop_back();
    if (id < 0 || r[id]) continue;
    r[id] = 1;
    const Node& n = ns[id];
    if (n.op == Op::Input || n.op == Op::Param || n.op == Op::Const) continue;
    st.push_back(n.a);
    st.push_back(n.b);
    st.push_back(n.c);
  }
  return r;
}

// Operands of which both sin and cos are live per-event values: operand -> (sin node, cos node).
std::map<int, std::pair<int, int>> sincos_pairs(const std::vector<Node>& ns, const std::vector<char>& live) {
  std::map<int, int> sin_of, cos_of;
  std::map<int, std::pair<int, int>> r;
  for (size_t i = 0; i < ns.size(); i++) {
    if (!live[i] || ns[i].uniform) continue;
    if (ns[i].op == Op::Sin) sin_of[ns[i].a] = int(i);
    if (ns[i].op == Op::Cos) cos_of[ns[i].a] = int(i);
  }
  for (auto& [a, si] : sin_of) {
    auto c = cos_of.find(a);
    if (c != cos_of.end()) r[a] = {si, c->second};
  }
  return r;
}

struct Emitter {
  const std::vector<Node>& ns;
  bool f32;  // arithmetic type float
  std::string T() const { return f32 ? "float" : "double"; }
  std::string ref(int id, const std::string& pfx) const {
    const Node& n = ns[id];
    if (n.op == Op::Const) return fmt_const(n.value, f32);
    if (n.op == Op::Input) return "x" + std::to_string(n.index);
    if (n.op == Op::Param) return "p" + std::to_string(n.index);
    return (n.uniform ? std::string("u") : pfx) + std::to_string(id);
  }
  // One SSA statement for node id (not for leaves).
  std::string stmt(int id, const std::string& pfx) const {
    const Node& n = ns[id];
    std::string lhs = "const " + std::string(n.op == Op::Cmp ? "bool" : T()) + " " + ref(id, pfx) + " = ";
    auto A = [&](int k) { return ref(k, pfx); };
    switch (n.op) {
      case Op::Add: return lhs + A(n.a) + " + " + A(n.b) + ";";
      case Op::Sub: return lhs + A(n.a) + " - " + A(n.b) + ";";
      case Op::Mul: return lhs + A(n.a) + " * " + A(n.b) + ";";
      case Op::Div: return lhs + A(n.a) + " / " + A(n.b) + ";";
      case Op::Neg: return lhs + "-" + A(n.a) + ";";
      case Op::Rcp: return lhs + fn_name(Op::Rcp, f32) + "(" + A(n.a) + ");";
      case Op::Pow: return lhs + fn_name(Op::Pow, f32) + "(" + A(n.a) + ", " + A(n.b) + ");";
      case Op::Cmp: return lhs + "(" + A(n.a) + " " + cmp_str(n.cmp) + " " + A(n.b) + ");";
      case Op::Select: return lhs + "(" + A(n.a) + " ? " + A(n.b) + " : " + A(n.c) + ");";
      case Op::Exp:
      case Op::Log:
      case Op::Sqrt:
      case Op::Sin:
      case Op::Cos: return lhs + fn_name(n.op, f32) + "(" + A(n.a) + ");";
      default:
        if (is_unary_fn(n.op)) return lhs + fn_name(n.op, f32) + "(" + A(n.a) + ");";
        throw std::runtime_error("emit: unexpected node");
    }
  }
};

const char* kPrelude = R"CUDA(
typedef unsigned long long mf_u64;
#define MF_FULL 0xffffffffu
__device__ __forceinline__ double mf_warp_sum(double x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(MF_FULL, x, o);
  return x;
}
// Neumaier-compensated add (fixed-order combine of block partials).
__device__ __forceinline__ void mf_neumaier(double& s, double& c, double x) {
  const double t = s + x;
  c += (fabs(s) >= fabs(x)) ? ((s - t) + x) : ((x - t) + s);
  s = t;
}
// Programmatic dependent launch (PTX griddepcontrol): no-ops unless the grid
// was launched with programmatic stream serialization.
__device__ __forceinline__ void mf_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void mf_grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// Device-scope fetch-and-add with acquire-release semantics.
__device__ __forceinline__ unsigned mf_atom_add_acq_rel(unsigned* p, unsigned v) {
  unsigned old;
  asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
  return old;
}
// Kahan step for FP32 per-thread partials (compute_llvm.hh:556-568 semantics).
__device__ __forceinline__ void mf_kahan_f32(float& s, float& c, float x) {
  const float y = __fsub_rn(x, c);
  const float t = __fadd_rn(s, y);
  c = __fsub_rn(__fsub_rn(t, s), y);
  s = t;
}
)CUDA";

// Double-float ("double-word") arithmetic on pairs of FP32 values, used by
// FP64 REDUCE kernels. GB300 issues FP32 at 64x its FP64 rate; a value is
// kept as an unevaluated sum h + l of two floats (|l| <= ulp(h)/2, ~48
// significant bits) and combined with error-free transforms: TwoSum (Knuth),
// FastTwoSum (Dekker 1971) and the FMA-based TwoProd; addition and
// multiplication follow the double-word algorithms analysed by Joldes, Muller
// and Popescu (ACM TOMS 44, 2017). The logarithm is table driven in the manner
// of Tang (ACM TOMS 16, 1990): log y = E ln2 + ln c_j + ln(1+t) with c_j the
// centre of one of 128 mantissa intervals, |t| <= 2^-8 and a short series.
// Operations without a double-float form fall back to FP64 on the value.
const char* kDwPrelude = R"CUDA(
struct mf_dw { float h, l; };
__device__ __forceinline__ mf_dw mf_dw_make(float h, float l) { mf_dw r; r.h = h; r.l = l; return r; }
__device__ __forceinline__ mf_dw mf_two_sum(float a, float b) {
  const float s = __fadd_rn(a, b);
  const float bb = __fsub_rn(s, a);
  return mf_dw_make(s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb)));
}
__device__ __forceinline__ mf_dw mf_fast_two_sum(float a, float b) {
  const float s = __fadd_rn(a, b);
  return mf_dw_make(s, __fsub_rn(b, __fsub_rn(s, a)));
}
__device__ __forceinline__ mf_dw mf_dw_add(mf_dw a, mf_dw b) {
  const mf_dw s = mf_two_sum(a.h, b.h);
  return mf_fast_two_sum(s.h, __fadd_rn(__fadd_rn(a.l, b.l), s.l));
}
__device__ __forceinline__ mf_dw mf_dw_neg(mf_dw a) { return mf_dw_make(-a.h, -a.l); }
__device__ __forceinline__ mf_dw mf_dw_sub(mf_dw a, mf_dw b) { return mf_dw_add(a, mf_dw_neg(b)); }
__device__ __forceinline__ mf_dw mf_dw_mul(mf_dw a, mf_dw b) {
  const float p = __fmul_rn(a.h, b.h);
  const float e = __fmaf_rn(a.h, b.l, __fmaf_rn(a.l, b.h, __fmaf_rn(a.h, b.h, -p)));
  return mf_fast_two_sum(p, e);
}
__device__ __forceinline__ mf_dw mf_dw_rcp(mf_dw a) {
  // r = 1/a.h, then the correction r (e + e^2) with the residual e = 1 - a*r
  // formed exactly to first order; without e^2 (2^-48 at most, never negative)
  // every reciprocal is a little small, and sums over events keep that.
  const float r = __frcp_rn(a.h);
  const float p = __fmul_rn(a.h, r);
  const float pe = __fmaf_rn(a.h, r, -p);
  const float e = __fsub_rn(__fsub_rn(__fsub_rn(1.0f, p), pe), __fmul_rn(a.l, r));
  return mf_fast_two_sum(r, __fmul_rn(r, __fmaf_rn(e, e, e)));
}
// An infinite high word is the value (its low word is NaN after inf - inf
// in the error terms of a sum).
__device__ __forceinline__ double mf_dw_to_double(mf_dw a) {
  return isinf(a.h) ? (double)a.h : (double)a.h + (double)a.l;
}
__device__ __forceinline__ mf_dw mf_dw_from_double(double x) {
  const float h = __double2float_rn(x);
  return mf_dw_make(h, __double2float_rn(x - (double)h));
}
// Splits an FP64 value into h + l with integer and FP32 operations only (no
// FP64 pipe, no conversion instructions, no branch): h keeps the top 24
// significand bits (truncated), l the next 23. Magnitudes below 2^-126 give
// h = l = 0 (an absolute error below 1.2e-38), l underflows to 0 below
// 2^-81, magnitudes from 2^128 on give +-inf, NaN stays NaN.
__device__ __forceinline__ mf_dw mf_dw_split(double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const unsigned hi32 = (unsigned)(b >> 32), lo32 = (unsigned)b;
  const unsigned e = (hi32 >> 20) & 0x7ffu;
  const unsigned sign = hi32 & 0x80000000u;
  const unsigned hnorm = sign | ((e - 896u) << 23) | ((hi32 & 0xfffffu) << 3) | (lo32 >> 29);
  const unsigned hbig = sign | 0x7f800000u | ((e == 2047u && ((hi32 & 0xfffffu) | lo32)) ? 0x400000u : 0u);
  const unsigned hb = e > 1150u ? hbig : (e >= 897u ? hnorm : sign);
  // top 23 of the 29 remaining bits as an exact float (exponent-field trick), scaled by 2^(e - 1069)
  const float r23 = __fsub_rn(__uint_as_float(0x4b000000u | ((lo32 & 0x1fffffffu) >> 6)), 8388608.0f);
  const unsigned sb = (e >= 943u && e <= 1150u) ? ((e - 942u) << 23) : 0u;
  const float l = __fmul_rn(r23, __uint_as_float(sb));
  return mf_dw_make(__uint_as_float(hb), __uint_as_float(__float_as_uint(l) | sign));
}
__device__ __forceinline__ mf_dw mf_dw_pair(float2 t) { return mf_dw_make(t.x, t.y); }
// Lazy double-float accumulation (per-thread partials, dot products): TwoSum
// of the high words, the low words and the rounding error added in FP32;
// mf_dw_renorm restores a normalized pair (|l| <= ulp(h)/2) at the end.
__device__ __forceinline__ void mf_dw_acc(mf_dw& a, mf_dw x) {
  const mf_dw s = mf_two_sum(a.h, x.h);
  a.h = s.h;
  a.l = __fadd_rn(a.l, __fadd_rn(s.l, x.l));
}
// a += x * y (the product's error terms formed with FMA, as in mf_dw_mul)
__device__ __forceinline__ void mf_dw_acc_mul(mf_dw& a, mf_dw x, mf_dw y) {
  const float p = __fmul_rn(x.h, y.h);
  const float e = __fmaf_rn(x.h, y.l, __fmaf_rn(x.l, y.h, __fmaf_rn(x.h, y.h, -p)));
  const mf_dw s = mf_two_sum(a.h, p);
  a.h = s.h;
  a.l = __fadd_rn(a.l, __fadd_rn(s.l, e));
}
// x * y as such a sum begins: acc_mul onto zero (not renormalized)
__device__ __forceinline__ mf_dw mf_dw_prod(mf_dw x, mf_dw y) {
  const float p = __fmul_rn(x.h, y.h);
  return mf_dw_make(p, __fmaf_rn(x.h, y.l, __fmaf_rn(x.l, y.h, __fmaf_rn(x.h, y.h, -p))));
}
// a += x * y for FP32 operands: the product is exact as p + e (FMA), so a
// dot product of FP32 values accumulated this way is as accurate as one
// computed in double-float (the compensated dot product of Ogita, Rump and
// Oishi, SIAM J. Sci. Comput. 26, 2005, with a lazily renormalised sum).
__device__ __forceinline__ mf_dw mf_dw_prodf(float x, float y) {
  const float p = __fmul_rn(x, y);
  return mf_dw_make(p, __fmaf_rn(x, y, -p));
}
// The same with a double-float factor c = c.h + c.l (a parameter-only
// coefficient kept to ~48 bits): x * c.h exact as p + e, plus x * c.l.
__device__ __forceinline__ mf_dw mf_dw_prodfw(float x, mf_dw c) {
  const float p = __fmul_rn(x, c.h);
  return mf_dw_make(p, __fmaf_rn(x, c.l, __fmaf_rn(x, c.h, -p)));
}
__device__ __forceinline__ void mf_dw_acc_mulfw(mf_dw& a, float x, mf_dw c) {
  const float p = __fmul_rn(x, c.h);
  const float e = __fmaf_rn(x, c.l, __fmaf_rn(x, c.h, -p));
  const mf_dw s = mf_two_sum(a.h, p);
  a.h = s.h;
  a.l = __fadd_rn(a.l, __fadd_rn(s.l, e));
}
__device__ __forceinline__ void mf_dw_acc_mulf(mf_dw& a, float x, float y) {
  const float p = __fmul_rn(x, y);
  const float e = __fmaf_rn(x, y, -p);
  const mf_dw s = mf_two_sum(a.h, p);
  a.h = s.h;
  a.l = __fadd_rn(a.l, __fadd_rn(s.l, e));
}
__device__ __forceinline__ mf_dw mf_dw_renorm(mf_dw a) { return mf_two_sum(a.h, a.l); }
// Round-to-nearest split with integer operations only: h = x rounded to 24
// bits, l = x - h rounded to 24 bits, |x - h - l| <= 2^-48 |x| for |x| from
// 2^-100 to 2^127 (below 2^-100 l loses bits to the FP32 exponent range).
// Magnitudes outside [2^-126, 2^127) (and zero, inf, NaN) take the
// truncating split. No FP64 instruction on any path: a short FP64 fallback
// would be if-converted and executed for every value.
__device__ __forceinline__ mf_dw mf_dw_split_rn(double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const unsigned e = (unsigned)(b >> 52) & 0x7ffu;
  if (e < 897u || e > 1149u) return mf_dw_split(x);
  const unsigned sign = (unsigned)(b >> 32) & 0x80000000u;
  const unsigned long long M = (b & 0xfffffffffffffull) | 0x10000000000000ull;  // 53-bit significand
  const unsigned long long H = (M + 0x10000000ull) >> 29;                       // nearest 24-bit value
  const long long L = (long long)M - (long long)(H << 29);                      // |L| <= 2^28
  const unsigned carry = (unsigned)(H >> 24);                                   // H = 2^24: next binade
  const float h = __uint_as_float(sign | ((e - 896u + carry) << 23) | (carry ? 0u : ((unsigned)H & 0x7fffffu)));
  const unsigned al = (unsigned)(L < 0 ? -L : L);
  // |L| rounded to its top 24 bits as an exact float (exponent-field trick),
  // scaled by 2^(e - 1070) (as 2^(e - 1006) * 2^-64 where e - 1070 < -126)
  const float m = __fsub_rn(__uint_as_float(0x4b000000u | ((al + 16u) >> 5)), 8388608.0f);
  const bool low = e < 944u;
  const float lm = __fmul_rn(__fmul_rn(m, __uint_as_float((low ? e - 879u : e - 943u) << 23)),
                             low ? 0x1p-64f : 1.0f);
  return mf_dw_make(h, __uint_as_float(__float_as_uint(lm) | (sign ^ (L < 0 ? 0x80000000u : 0u))));
}
// A normalized pair (|l| <= ulp(h)/2, as every operation here returns) as an
// FP64 value without the FP64 pipe: the double of h from its bits, moved by l
// in units of the double's last place (one exact scaling and one conversion to
// an integer, |l| <= 2^28 units, rounded to nearest) as an integer step of the
// bit pattern, which cannot leave h's binade upwards. Powers of two, whose
// lower neighbours are half as far apart, magnitudes below 2^-75, zero, inf
// and NaN take the general form, out of line: zero or subnormal h gives a
// signed zero (an absolute error below 2^-125), inf and NaN carry over.
__device__ __noinline__ double mf_dw_to_double_rare(float h, float l) {
  const unsigned hb = __float_as_uint(h), sign = hb & 0x80000000u;
  const int eh = (int)((hb >> 23) & 0xffu);
  const float up = sign ? -l : l;  // away from zero
  // times 2^(179 - eh), twice that below a power of two, in two exact steps
  const int sh = 179 - eh + ((hb & 0x7fffffu) == 0u && up < 0.0f ? 1 : 0), s1 = sh / 2;
  const float units = __fmul_rn(__fmul_rn(up, __uint_as_float((unsigned)(127 + s1) << 23)),
                                __uint_as_float((unsigned)(127 + sh - s1) << 23));
  const int li = eh != 0 && eh != 255 ? __float2int_rn(units) : 0;
  long long bits = ((long long)(hb & 0x7fffffffu) << 29) + (896ll << 52) + (long long)li;
  if (eh == 0) bits = 0;
  if (eh == 255) bits = (0x7ffll << 52) | ((hb & 0x7fffffu) ? (1ll << 51) : 0ll);
  return __longlong_as_double(bits | ((long long)sign << 32));
}
__device__ __forceinline__ double mf_dw_to_double_bits(mf_dw a) {
  const unsigned hb = __float_as_uint(a.h), e = hb & 0x7f800000u, sign = hb & 0x80000000u;
  if ((hb & 0x7fffffu) == 0u || e - (52u << 23) >= (203u << 23)) return mf_dw_to_double_rare(a.h, a.l);
  // l * 2^(179 - eh), negated where h is negative
  const int li = __float2int_rn(__fmul_rn(a.l, __uint_as_float(((306u << 23) - e) ^ sign)));
  const unsigned long long h = ((unsigned long long)((((hb & 0x7fffffffu) >> 3) + 0x38000000u) | sign) << 32) | (hb << 29);
  return __longlong_as_double((long long)h + (long long)li);
}
// Square root: s = a.h / sqrt(a.h) and h = 1 / (2 sqrt(a.h)) in FP32, each
// corrected once (Goldschmidt's iteration), then the series sqrt(s^2 + r) =
// s + d - d^2/(2s) + ..., d = r/(2s). d reaches 2^-23 s, so the residual
// r = a - s^2 (s^2 exact by FMA) and d are kept as double-float values, d by
// the reciprocal h and one correction; the next term, d^3/(2s^2), is below
// 2^-70 s. sqrt(0) = 0, negative or NaN -> NaN, +inf -> +inf.
__device__ __forceinline__ mf_dw mf_dw_sqrt(mf_dw a) {
  if (!(a.h > 0.0f) || a.h == __int_as_float(0x7f800000))
    return mf_dw_make(a.h == 0.0f ? 0.0f : (a.h > 0.0f ? a.h : __int_as_float(0x7fc00000)), 0.0f);
  const float y = rsqrtf(a.h);
  const float s0 = __fmul_rn(a.h, y), h0 = __fmul_rn(0.5f, y);
  const float c = __fmaf_rn(-s0, h0, 0.5f);
  const float s = __fmaf_rn(s0, c, s0), h = __fmaf_rn(h0, c, h0);
  const float p = __fmul_rn(s, s);
  const float pe = __fmaf_rn(s, s, -p);
  // a.h - p is exact (Sterbenz); the rest of the residual in double-float
  const mf_dw r0 = mf_two_sum(__fsub_rn(a.h, p), -pe), r = mf_two_sum(r0.h, a.l);
  const float rl = __fadd_rn(r0.l, r.l);
  const float dh = __fmul_rn(__fadd_rn(r.h, rl), h);
  const float dl = __fmul_rn(__fadd_rn(__fmaf_rn(-dh, __fadd_rn(s, s), r.h), rl), h);
  const float q = __fmul_rn(__fmul_rn(dh, dh), h);
  const mf_dw t = mf_fast_two_sum(s, dh);
  return mf_fast_two_sum(t.h, __fadd_rn(t.l, __fsub_rn(dl, q)));
}
// c + x * q for |x q| < |c|, not renormalized
__device__ __forceinline__ mf_dw mf_dw_horner(mf_dw c, mf_dw x, mf_dw q) {
  const float p = __fmul_rn(x.h, q.h);
  const float e = __fmaf_rn(x.h, q.l, __fmaf_rn(x.l, q.h, __fmaf_rn(x.h, q.h, -p)));
  const float s = __fadd_rn(c.h, p);
  return mf_dw_make(s, __fadd_rn(__fsub_rn(p, __fsub_rn(s, c.h)), __fadd_rn(c.l, e)));
}
// the same with the product normalized first
__device__ __forceinline__ mf_dw mf_dw_horner_last(mf_dw c, mf_dw x, mf_dw q) {
  const mf_dw p = mf_dw_mul(x, q);
  const float s = __fadd_rn(c.h, p.h);
  return mf_dw_make(s, __fadd_rn(__fsub_rn(p.h, __fsub_rn(s, c.h)), __fadd_rn(c.l, p.l)));
}
// sin and cos of a double-float. a = k*(pi/2) + r, |r| <~ pi/4, by a
// four-part Cody-Waite reduction: pi/2 = C1 + C2 + C3 + C4 with C1 and C2 of
// 12 significant bits (k*C1, k*C2 exact for |k| < 2^12) and a remainder below
// 4e-22. sin r and cos r are their Taylor series, the terms above 2^-26 in
// double-float (Horner), the rest in FP32; the first omitted term is below
// 2e-16 relative. A Horner step adds a product to a coefficient at least 16
// times as large, so it needs neither an ordered sum nor a renormalized
// result: nine operations (mf_dw_horner). The last step of each, whose product
// is not as small, normalizes it: sin r within 2^-46.57 (rms 2^-49.60) and cos r
// within 2^-47.07 (2^-50.37), as with normalized operations throughout;
// without, 2^-46.54 and 2^-46.71. Arguments beyond |a| = 6000 (and inf/NaN)
// use FP64.
__device__ __forceinline__ void mf_dw_sincos(mf_dw a, mf_dw* sn, mf_dw* cs) {
  if (!(fabsf(a.h) <= 6000.0f)) {
    const double x = mf_dw_to_double(a);
    *sn = mf_dw_from_double(sin(x));
    *cs = mf_dw_from_double(cos(x));
    return;
  }
  const float k = rintf(__fmul_rn(a.h, 0x1.45f306p-1f));
  const float t1 = __fmaf_rn(-k, 0x1.92p+0f, a.h);  // exact
  mf_dw r = mf_two_sum(t1, -__fmul_rn(k, 0x1.fb4p-12f));
  const float p3 = __fmul_rn(k, 0x1.4442dp-24f);
  r = mf_dw_sub(r, mf_dw_make(p3, __fmaf_rn(k, 0x1.4442dp-24f, -p3)));
  r = mf_dw_add(r, mf_dw_make(__fmaf_rn(-k, 0x1.846988p-48f, a.l), 0.0f));
  const mf_dw r2 = mf_dw_mul(r, r);
  const float z = r2.h;
  // sin r = r + r^3 (c3 + r^2 (c5 + r^2 (c7 + r^2 (c9 + r^2 T)))), c_n = (-1)^((n-1)/2) / n!
  const float T = __fmaf_rn(z, __fmaf_rn(z, -0x1.ae7f3ep-41f, 0x1.612462p-33f), -0x1.ae6456p-26f);
  mf_dw q = mf_dw_horner(mf_dw_make(0x1.71de3ap-19f, 0x1.55b1ccp-45f), r2, mf_dw_make(T, 0.0f));
  q = mf_dw_horner(mf_dw_make(-0x1.a01a02p-13f, 0x1.7f97fap-39f), r2, q);
  q = mf_dw_horner(mf_dw_make(0x1.111112p-7f, -0x1.dddddep-32f), r2, q);
  q = mf_dw_horner(mf_dw_make(-0x1.555556p-3f, 0x1.555556p-28f), r2, q);
  mf_dw sr = mf_dw_horner_last(r, mf_dw_mul(r, r2), q);
  sr = mf_fast_two_sum(sr.h, sr.l);
  // cos r = 1 + r^2 (c2 + r^2 (c4 + r^2 (c6 + r^2 (c8 + r^2 (c10 + r^2 T2))))), c_n = (-1)^(n/2) / n!
  const float T2 = __fmaf_rn(z, __fmaf_rn(z, 0x1.ae7f3ep-45f, -0x1.93974ap-37f), 0x1.1eed8ep-29f);
  mf_dw u = mf_dw_horner(mf_dw_make(-0x1.27e4fcp-22f, 0x1.10ec14p-47f), r2, mf_dw_make(T2, 0.0f));
  u = mf_dw_horner(mf_dw_make(0x1.a01a02p-16f, -0x1.7f97fap-42f), r2, u);
  u = mf_dw_horner(mf_dw_make(-0x1.6c16c2p-10f, 0x1.27d27ep-35f), r2, u);
  u = mf_dw_horner(mf_dw_make(0x1.555556p-5f, -0x1.555556p-30f), r2, u);
  u = mf_dw_horner(mf_dw_make(-0.5f, 0.0f), r2, u);
  u = mf_dw_horner_last(mf_dw_make(1.0f, 0.0f), r2, u);
  const mf_dw cr = mf_fast_two_sum(u.h, u.l);
  const int quad = ((int)k) & 3;
  const mf_dw s0 = (quad & 1) ? cr : sr, c0 = (quad & 1) ? sr : cr;
  *sn = (quad & 2) ? mf_dw_neg(s0) : s0;
  *cs = ((quad + 1) & 2) ? mf_dw_neg(c0) : c0;
}
__device__ __forceinline__ mf_dw mf_dw_sin(mf_dw a) { mf_dw s, c; mf_dw_sincos(a, &s, &c); return s; }
__device__ __forceinline__ mf_dw mf_dw_cos(mf_dw a) { mf_dw s, c; mf_dw_sincos(a, &s, &c); return c; }
// ln of a positive double-float (see above); zero gives -inf, negative or
// NaN gives NaN, +inf gives +inf, subnormal h is rescaled by 2^64 first.
__device__ __forceinline__ mf_dw mf_dw_log(mf_dw a, const float4* __restrict__ tab) {
  const bool sub = a.h > 0.0f && a.h < 1.17549435e-38f;
  const float ah = sub ? __fmul_rn(a.h, 18446744073709551616.0f) : a.h;
  const float al = sub ? __fmul_rn(a.l, 18446744073709551616.0f) : a.l;
  const unsigned bits = __float_as_uint(ah);
  const int E = (int)((bits >> 23) & 0xffu) - 127;
  const float m = __uint_as_float((bits & 0x007fffffu) | 0x3f800000u);
  const float4 T = tab[(bits >> 16) & 0x7fu];  // {ln c hi, ln c lo, 1/c, c}
  const unsigned se = (unsigned)(127 - E);
  const float yl = __fmul_rn(al, __uint_as_float(se >= 1u && se <= 254u ? (se << 23) : 0u));
  const mf_dw N = mf_two_sum(__fsub_rn(m, T.w), yl);
  const float th = __fmul_rn(N.h, T.z);
  const float tl = __fmul_rn(__fadd_rn(__fmaf_rn(-th, T.w, N.h), N.l), T.z);
  const float sh = __fmul_rn(th, th);
  const float sl = __fmaf_rn(2.0f * th, tl, __fmaf_rn(th, th, -sh));
  mf_dw lt = mf_dw_sub(mf_dw_make(th, tl), mf_dw_make(0.5f * sh, 0.5f * sl));
  const float P = __fmaf_rn(th, __fmaf_rn(th, __fmaf_rn(th, __fmaf_rn(th, 0.142857143f, -0.166666667f), 0.2f), -0.25f),
                            0.333333333f);
  lt = mf_dw_add(lt, mf_dw_make(__fmul_rn(__fmul_rn(sh, th), P), 0.0f));
  const int Et = E - (sub ? 64 : 0);
  const float Ef = __fsub_rn(__int_as_float(0x4b400000 + Et), 12582912.0f);  // (float)Et without a conversion
  // E*ln2 with ln2 = L1 + L2 + L3 (L1 of 12 bits: E*L1 exact; remainder of L3 below 1e-19)
  const float e1 = __fmul_rn(Ef, 0x1.62ep-1f);
  const float e2 = __fmul_rn(Ef, 0x1.0bfbe8p-15f);
  const mf_dw e12 = mf_two_sum(e1, e2);
  const mf_dw el = mf_fast_two_sum(
      e12.h, __fadd_rn(e12.l, __fmaf_rn(Ef, 0x1.cf79aap-40f, __fmaf_rn(Ef, 0x1.0bfbe8p-15f, -e2))));
  mf_dw r = mf_dw_add(mf_dw_add(el, mf_dw_make(T.x, T.y)), lt);
  const float inf = __uint_as_float(0x7f800000u);
  if (a.h == 0.0f) r = mf_dw_make(-inf, 0.0f);
  if (!(a.h >= 0.0f)) r = mf_dw_make(__uint_as_float(0x7fc00000u), 0.0f);
  if (a.h == inf) r = mf_dw_make(inf, 0.0f);
  return r;
}
// exp of a double-float value by Tang's table-driven method (P. T. P. Tang,
// ACM TOMS 15 (1989) 144-157): x = (64k + j) ln2/64 + r with ln2/64 split as
// C1 + C2 + C3 (C1 of 9 significant bits, so N*C1 is exact for |N| < 2^13),
// |r| <= ln2/128 (+ a rounding); exp(r) - 1 = r + r^2/2 + r^3/6 in
// double-float plus r^4/24 + r^5/120 + r^6/720 in FP32 (below 4e-11);
// exp(x) = 2^k * T_j * (1 + (exp(r) - 1)) with T_j = 2^(j/64) from the table,
// 2^k applied as two exact power-of-two factors. Relative error ~2^-46 for
// results from 2^-100 to 2^128 (where the low word is a normal float); below
// 2^-100 the low word loses bits (an absolute error of a few 2^-149, the
// resolution of any double-float value there) and results under 2^-149 are
// 0; above 2^128 the result is +inf; NaN stays NaN.
__device__ __forceinline__ mf_dw mf_dw_exp(mf_dw a, const float2* __restrict__ tab) {
  const float x = fminf(fmaxf(a.h, -104.0f), 89.0f);
  // N = x * 64/ln2 rounded to an integer (|N| < 2^14) without a conversion:
  // adding 1.5*2^23 leaves the integer in the low significand bits
  const float tn = __fmaf_rn(x, 0x1.715476p+6f, 12582912.0f);
  const int Ni = __float_as_int(tn) - 0x4b400000;
  const float N = __fsub_rn(tn, 12582912.0f);
  const int j = Ni & 63;
  const int k = (Ni - j) >> 6;
  const float t1 = __fmaf_rn(-N, 0x1.63p-7f, x);  // exact
  const float p2 = __fmul_rn(N, -0x1.bd0106p-19f);
  const float p2e = __fmaf_rn(N, -0x1.bd0106p-19f, -p2);
  mf_dw r = mf_two_sum(t1, -p2);
  r = mf_fast_two_sum(r.h, __fadd_rn(r.l, __fsub_rn(__fmaf_rn(-N, 0x1.cf79acp-46f, a.l), p2e)));
  const mf_dw r2 = mf_dw_mul(r, r);
  const mf_dw r3 = mf_dw_mul(r2, r);
  mf_dw t3 = mf_dw_mul(r3, mf_dw_make(0x1.555556p-3f, -0x1.555556p-28f));
  const float q = __fmul_rn(__fmul_rn(r2.h, r2.h),
                            __fmaf_rn(r.h, __fmaf_rn(r.h, 0x1.6c16c2p-10f, 0x1.111112p-7f), 0x1.555556p-5f));
  t3 = mf_fast_two_sum(t3.h, __fadd_rn(t3.l, q));
  mf_dw e = mf_dw_add(r, mf_dw_make(0.5f * r2.h, 0.5f * r2.l));
  e = mf_dw_add(e, t3);
  const float2 T = tab[j];
  const mf_dw Tj = mf_dw_make(T.x, T.y);
  mf_dw y = mf_dw_add(Tj, mf_dw_mul(Tj, e));
  const int k1 = k >> 1, k2 = k - k1;  // both in [-76, 64]
  const float s1 = __int_as_float((k1 + 127) << 23), s2 = __int_as_float((k2 + 127) << 23);
  y = mf_dw_make(__fmul_rn(__fmul_rn(y.h, s1), s2), __fmul_rn(__fmul_rn(y.l, s1), s2));
  if (a.h > 89.0f) y = mf_dw_make(__int_as_float(0x7f800000), 0.0f);
  if (a.h < -104.0f) y = mf_dw_make(0.0f, 0.0f);
  if (a.h != a.h) y = mf_dw_make(a.h, a.h);
  return y;
}
// a^b = exp(b ln|a|) in double-float. a < 0: for integer b the sign follows
// b's parity, otherwise NaN; a = 0: 0 for b > 0, +inf for b < 0; b = 0: 1
// (also for a NaN). Relative error ~|b ln a| 2^-46.
// `la` is ln|a| (mf_dw_logabs), which the powers of one base and its logarithm share.
__device__ __forceinline__ mf_dw mf_dw_logabs(mf_dw a, const float4* __restrict__ tab) {
  return mf_dw_log(a.h < 0.0f ? mf_dw_neg(a) : a, tab);
}
__device__ __forceinline__ mf_dw mf_dw_log_of(mf_dw a, mf_dw la) {  // ln a from ln|a|
  return a.h < 0.0f ? mf_dw_make(__uint_as_float(0x7fc00000u), 0.0f) : la;
}
__device__ __forceinline__ mf_dw mf_dw_pow(mf_dw a, mf_dw b, mf_dw la, const float2* __restrict__ etab) {
  const bool neg = a.h < 0.0f;
  mf_dw r = mf_dw_exp(mf_dw_mul(b, la), etab);
  // integer b and its parity from the significand bits (|v| < 2^23: v + 2^23
  // holds v's integer part in its last bits; |v| >= 2^23 is an integer)
  const float bh = fabsf(b.h), bl = fabsf(b.l);
  const float th = __fadd_rn(bh, 8388608.0f), tl = __fadd_rn(bl, 8388608.0f);
  const bool int_h = bh >= 8388608.0f || __fsub_rn(th, 8388608.0f) == bh;
  const bool int_l = bl >= 8388608.0f || __fsub_rn(tl, 8388608.0f) == bl;
  const bool int_b = int_h && int_l;
  const bool odd = bh < 8388608.0f ? (__float_as_int(th) & 1) != 0
                                   : (bh < 16777216.0f ? (__float_as_int(b.h) & 1) != 0
                                                       : (bl < 8388608.0f && (__float_as_int(tl) & 1) != 0));
  if (neg) r = int_b ? (odd ? mf_dw_neg(r) : r) : mf_dw_make(__int_as_float(0x7fc00000), 0.0f);
  if (a.h == 0.0f) r = mf_dw_make(b.h > 0.0f ? 0.0f : __int_as_float(0x7f800000), 0.0f);
  if (b.h == 0.0f) r = mf_dw_make(1.0f, 0.0f);
  return r;
}
// Comparisons of normalized double-float values (lexicographic on (h, l)).
__device__ __forceinline__ bool mf_dw_gt(mf_dw a, mf_dw b) { return a.h > b.h || (a.h == b.h && a.l > b.l); }
__device__ __forceinline__ bool mf_dw_lt(mf_dw a, mf_dw b) { return a.h < b.h || (a.h == b.h && a.l < b.l); }
__device__ __forceinline__ bool mf_dw_ge(mf_dw a, mf_dw b) { return a.h > b.h || (a.h == b.h && a.l >= b.l); }
__device__ __forceinline__ bool mf_dw_le(mf_dw a, mf_dw b) { return a.h < b.h || (a.h == b.h && a.l <= b.l); }
__device__ __forceinline__ bool mf_dw_eq(mf_dw a, mf_dw b) { return a.h == b.h && a.l == b.l; }
// A sum of logarithms as the logarithm of a running product (per thread):
// m * 2^e with m kept in [1, 2) by an exact power-of-two rescaling and the
// binary exponent e in an integer, so each factor costs one double-float
// product instead of a logarithm. A factor that is not positive (or NaN), or
// a product outside the FP32 normal range, makes m NaN for good; the
// thread's sum is then NaN, as a sum of the logs would be non-finite.
__device__ __forceinline__ void mf_dw_logprod(mf_dw& m, int& e, mf_dw p) {
  const mf_dw q = mf_dw_mul(m, p);
  const int ex = (int)((__float_as_uint(q.h) >> 23) & 0xffu);
  const float sc = __uint_as_float((unsigned)(254 - ex) << 23);  // 2^(127 - ex) for ex in [1, 253]
  const bool ok = p.h > 0.0f && ex > 0 && ex < 254;
  m = ok ? mf_dw_make(__fmul_rn(q.h, sc), __fmul_rn(q.l, sc)) : mf_dw_make(__int_as_float(0x7fc00000), 0.0f);
  e += ex - 127;
}
// log(m * 2^e) = log(m) + e ln2, ln2 as a double-float pair (e exact in FP32);
// a thread without factors (m = 1, e = 0) contributes exactly 0.
__device__ __forceinline__ mf_dw mf_dw_logprod_log(mf_dw m, int e, const float4* __restrict__ tab) {
  if (e == 0 && m.h == 1.0f && m.l == 0.0f) return mf_dw_make(0.0f, 0.0f);
  const mf_dw el = mf_dw_mul(mf_dw_make((float)e, 0.0f), mf_dw_make(MF_LN2_HI, MF_LN2_LO));
  return mf_dw_add(mf_dw_log(m, tab), el);
}
__device__ __forceinline__ mf_dw mf_dw_shfl_xor(mf_dw a, int o) {
  return mf_dw_make(__shfl_xor_sync(0xffffffffu, a.h, o), __shfl_xor_sync(0xffffffffu, a.l, o));
}
)CUDA";

// Cross-thread sums of REDUCE kernels: double-float adds in a fixed order.
// mf_sum_rows: the sums of `nb` partial rows, `step` rows apart, into sums[]
// (shared, complete for every thread on return). Thread (g, o) takes rows g,
// g + MF_GRP, ... of output o, so that a warp's loads are contiguous and a
// round of loads covers MF_Q rows per thread, added as a tree; then the MF_GRP
// partials per output are added as a tree, by one thread (few) or a warp. All
// of the block's threads take rows of a single output: its kernels are small,
// so their full grids have up to 1216 rows, two and three rounds of loads for
// 32 threads (1M events, FP32 values mass 22.1 -> 19.4 us, Crystal Ball 25.9 ->
// 23.3, FP64 mass 26.0 -> 24.7). Two to seven outputs keep 32 threads each: the
// mass gradient's registers (FP32 40 -> 42, FP64 48 -> 54) would cost a block
// per SM. Measured as part of a lone launch, one thread per row and a shuffle
// tree per output took 18 us of the P-wave Hessian's 54 (36 outputs, 152 rows,
// ncu) and 100 of the S+P wave's 163 (105 outputs, 608 rows). A lone small
// evaluation waits for every add in turn (about 60 cycles): trees instead of
// chains here and across a block's warps, and no tree of empty rows for grids
// of up to MF_GRP blocks, 14.6 -> 14.3 us (P-wave NLL in FP32, 30011 events)
// and 15.7 -> 15.3 (mass gradient, 1000).
const char* kCombine = R"CUDA(
template <int N> __device__ __forceinline__ void mf_warp_sums(mf_dw (&v)[N], int lane) {
  int o = 16;
#pragma unroll
  for (int h = N / 2; h > 0; h >>= 1, o >>= 1) {
    const bool up = (lane & o) != 0;  // keep the upper half of the outputs
#pragma unroll
    for (int c = 0; c < h; c++) {
      const mf_dw keep = up ? v[c + h] : v[c], give = up ? v[c] : v[c + h];
      v[c] = mf_dw_add(keep, mf_dw_shfl_xor(give, o));
    }
  }
#pragma unroll
  for (; o > 0; o >>= 1) v[0] = mf_dw_add(v[0], mf_dw_shfl_xor(v[0], o));
}
// t[0] = the sum of t[0..N)
template <int N> __device__ __forceinline__ void mf_tree_sum(mf_dw (&t)[N]) {
#pragma unroll
  for (int s = 1; s < N; s *= 2)
#pragma unroll
    for (int q = 0; q + s < N; q += 2 * s) t[q] = mf_dw_add(t[q], t[q + s]);
}
// the sum of one output over the block's warps (rows of MF_NOUT), in eights
__device__ __forceinline__ mf_dw mf_sum_warps(const float2* p) {
  mf_dw a;
  for (int w0 = 0; w0 < MF_BLOCK / 32; w0 += 8) {
    mf_dw t[MF_BLOCK / 32 < 8 ? MF_BLOCK / 32 : 8];
#pragma unroll
    for (int w = 0; w < (MF_BLOCK / 32 < 8 ? MF_BLOCK / 32 : 8); w++)
      t[w] = w0 + w < MF_BLOCK / 32 ? mf_dw_pair(p[(w0 + w) * MF_NOUT]) : mf_dw_make(0.0f, 0.0f);
    mf_tree_sum(t);
    a = w0 == 0 ? t[0] : mf_dw_add(a, t[0]);
  }
  return a;
}
__device__ __forceinline__ void mf_sum_rows(const float2* rows, unsigned nb, unsigned step, float2* part, float2* sums) {
  const mf_u64 stride = (mf_u64)step * MF_NOUT;
#if MF_GRP > 1
  const int g = threadIdx.x / MF_NOUT, o = threadIdx.x - g * MF_NOUT;
  if (g < MF_GRP) {
#else
  const int g = 0;
  for (int o = threadIdx.x; o < MF_NOUT; o += MF_BLOCK) {
#endif
    mf_dw a;
    if (nb <= MF_GRP) {  // a row each at most
      a = g < nb ? mf_dw_pair(__ldcg(rows + g * stride + o)) : mf_dw_make(0.0f, 0.0f);
    } else {
      for (unsigned r0 = g; r0 == g || r0 < nb; r0 += MF_GRP * MF_Q) {
        float2 v[MF_Q];
#pragma unroll
        for (int q = 0; q < MF_Q; q++) {
          const unsigned r = r0 + q * MF_GRP;
          v[q] = r < nb ? __ldcg(rows + r * stride + o) : make_float2(0.0f, 0.0f);
        }
        mf_dw t[MF_Q];
#pragma unroll
        for (int q = 0; q < MF_Q; q++) t[q] = mf_dw_pair(v[q]);
        mf_tree_sum<MF_Q>(t);
        a = r0 == g ? t[0] : mf_dw_add(a, t[0]);
      }
    }
#if MF_GRP > 1
    part[g * MF_NOUT + o] = make_float2(a.h, a.l);
  }
  __syncthreads();
#if MF_GRP <= 8
  if (threadIdx.x < MF_NOUT) {
    mf_dw t[MF_GRP];
#pragma unroll
    for (int q = 0; q < MF_GRP; q++) t[q] = mf_dw_pair(part[q * MF_NOUT + threadIdx.x]);
    mf_tree_sum<MF_GRP>(t);
    sums[threadIdx.x] = make_float2(t[0].h, t[0].l);
  }
#else
  for (int j = threadIdx.x >> 5; j < MF_NOUT; j += MF_BLOCK / 32) {
    const int q = threadIdx.x & 31;
    mf_dw a = q < MF_GRP ? mf_dw_pair(part[q * MF_NOUT + j]) : mf_dw_make(0.0f, 0.0f);
#if MF_GRP > 32
    if (nb > 32u) {
      mf_dw t[(MF_GRP + 31) / 32];
#pragma unroll
      for (int r = 0; r < (MF_GRP + 31) / 32; r++)
        t[r] = q + 32 * r < MF_GRP ? mf_dw_pair(part[(q + 32 * r) * MF_NOUT + j]) : mf_dw_make(0.0f, 0.0f);
      mf_tree_sum(t);
      a = t[0];
    }
#endif
#pragma unroll
    for (int w = MF_GRP > 16 ? 16 : 8; w > 0; w >>= 1) a = mf_dw_add(a, mf_dw_shfl_xor(a, w));
    if (q == 0) sums[j] = make_float2(a.h, a.l);
  }
#endif
#else
    sums[o] = make_float2(a.h, a.l);
  }
#endif
  __syncthreads();
}
)CUDA";

// FP32 values with a running bound of their error, for the generator's accept
// test: the exact value of the expression lies within e of v. Every operation
// adds to the propagated bounds of its operands the rounding of its own result
// (kept at twice 2^-24 relative, which also covers the rounding of the bounds
// themselves, plus 2^-126 for results that underflow); the functions' results
// are taken as within 4 units of 2^-23 (CUDA's documented maximum errors are
// smaller), and their slopes are bounded over the whole interval the operand
// may lie in, or the bound is infinite where it may reach a pole or a branch.
// The caller tests the final bound with 1% to spare.
const char* kEfPrelude = R"CUDA(
struct mf_ef { float v, e; };
#define MF_EF_INF __int_as_float(0x7f800000)
__device__ __forceinline__ mf_ef mf_ef_make(float v, float e) { mf_ef r; r.v = v; r.e = e; return r; }
__device__ __forceinline__ mf_ef mf_ef_from(double x) {
  const float v = (float)x;
  return mf_ef_make(v, fabsf(v) * 0x1p-23f + 0x1p-126f);
}
__device__ __forceinline__ mf_ef mf_ef_neg(mf_ef a) { return mf_ef_make(-a.v, a.e); }
__device__ __forceinline__ mf_ef mf_ef_add(mf_ef a, mf_ef b) {
  const float v = a.v + b.v;
  return mf_ef_make(v, fmaf(fabsf(v), 0x1p-23f, a.e + b.e));
}
__device__ __forceinline__ mf_ef mf_ef_sub(mf_ef a, mf_ef b) { return mf_ef_add(a, mf_ef_neg(b)); }
__device__ __forceinline__ mf_ef mf_ef_mul(mf_ef a, mf_ef b) {
  const float v = a.v * b.v;
  return mf_ef_make(v, fmaf(fabsf(a.v) + a.e, b.e, fmaf(fabsf(b.v), a.e, fmaf(fabsf(v), 0x1p-23f, 0x1p-126f))));
}
__device__ __forceinline__ mf_ef mf_ef_rcp(mf_ef a) {  // |1/(a+d) - 1/a| <= e r^2 / (1 - e r)
  const float r = __frcp_rn(a.v), er = a.e * fabsf(r);
  return mf_ef_make(r, er < 0.25f ? fmaf(fabsf(r), fmaf(er, 1.34f, 0x1p-23f), 0x1p-126f) : MF_EF_INF);
}
// 4 units of 2^-23 of a function's result
#define MF_EF_FN 0x1p-21f
__device__ __forceinline__ mf_ef mf_ef_exp(mf_ef a) {  // e^d - 1 <= 1.07 d for d < 1/8
  const float v = expf(a.v);
  return mf_ef_make(v, a.e < 0.125f ? fmaf(v, fmaf(a.e, 1.07f, MF_EF_FN), 0x1p-126f) : MF_EF_INF);
}
__device__ __forceinline__ mf_ef mf_ef_log(mf_ef a) {
  const float v = logf(a.v);
  return mf_ef_make(v, a.v > 4.0f * a.e ? fmaf(fabsf(v), MF_EF_FN, 1.34f * a.e / a.v) : MF_EF_INF);
}
__device__ __forceinline__ mf_ef mf_ef_sqrt(mf_ef a) {  // |d| / (s + s') <= e / s
  const float v = sqrtf(a.v);
  return mf_ef_make(v, a.v > 2.0f * a.e ? fmaf(v, MF_EF_FN, 1.01f * a.e * rsqrtf(a.v)) : MF_EF_INF);
}
__device__ __forceinline__ void mf_ef_sincos(mf_ef a, mf_ef* s, mf_ef* c) {
  sincosf(a.v, &s->v, &c->v);
  s->e = fmaf(fabsf(s->v), MF_EF_FN, a.e) + 0x1p-126f;
  c->e = fmaf(fabsf(c->v), MF_EF_FN, a.e) + 0x1p-126f;
}
__device__ __forceinline__ mf_ef mf_ef_sin(mf_ef a) {
  const float v = sinf(a.v);
  return mf_ef_make(v, fmaf(fabsf(v), MF_EF_FN, a.e) + 0x1p-126f);
}
__device__ __forceinline__ mf_ef mf_ef_cos(mf_ef a) {
  const float v = cosf(a.v);
  return mf_ef_make(v, fmaf(fabsf(v), MF_EF_FN, a.e) + 0x1p-126f);
}
__device__ __forceinline__ mf_ef mf_ef_tan(mf_ef a) {  // slope 1 + t^2, below 1.5 times that while e (1 + |t|) < 1/8
  const float v = tanf(a.v);
  return mf_ef_make(v, a.e * (1.0f + fabsf(v)) < 0.125f
                           ? fmaf(fabsf(v), MF_EF_FN, a.e * fmaf(v, v, 1.0f) * 1.5f) + 0x1p-126f : MF_EF_INF);
}
__device__ __forceinline__ float mf_ef_arc(mf_ef a) {  // slope 1 / sqrt(1 - x^2) at the end of the interval nearest 1
  const float y = (1.0f - fabsf(a.v)) - a.e;
  return y > 1e-5f ? 1.01f * a.e * rsqrtf(y) : MF_EF_INF;
}
__device__ __forceinline__ mf_ef mf_ef_asin(mf_ef a) {
  const float v = asinf(a.v);
  return mf_ef_make(v, fmaf(fabsf(v), MF_EF_FN, mf_ef_arc(a)) + 0x1p-126f);
}
__device__ __forceinline__ mf_ef mf_ef_acos(mf_ef a) {
  const float v = acosf(a.v);
  return mf_ef_make(v, fmaf(fabsf(v), MF_EF_FN, mf_ef_arc(a)) + 0x1p-126f);
}
__device__ __forceinline__ mf_ef mf_ef_atan(mf_ef a) {
  const float v = atanf(a.v);
  return mf_ef_make(v, fmaf(fabsf(v), MF_EF_FN, a.e) + 0x1p-126f);
}
__device__ __forceinline__ mf_ef mf_ef_erf(mf_ef a) {
  const float v = erff(a.v);
  return mf_ef_make(v, fmaf(fabsf(v), MF_EF_FN, 1.13f * a.e) + 0x1p-126f);
}
// a^b for a > 0: ln of it moves by |b| de/a + |ln a| db; any other base in FP64
__device__ __forceinline__ mf_ef mf_ef_pow(mf_ef a, mf_ef b) {
  const float v = powf(a.v, b.v);
  const float d = fmaf((fabsf(b.v) + b.e) * 1.34f, a.e / a.v, fabsf(logf(a.v)) * b.e * 1.01f);
  return mf_ef_make(v, a.v > 4.0f * a.e && d < 0.125f ? fmaf(v, fmaf(d, 1.07f, 2.0f * MF_EF_FN), 0x1p-126f) : MF_EF_INF);
}
// whether the order of two values is uncertain
__device__ __forceinline__ bool mf_ef_near(mf_ef a, mf_ef b) { return !(fabsf(a.v - b.v) > 1.01f * (a.e + b.e)); }
)CUDA";

// Bulk asynchronous global->shared copies completed on an mbarrier (sm_90+
// PTX: cp.async.bulk, mbarrier.*). Both addresses 16-byte aligned, sizes a
// multiple of 16 bytes.
const char* kBulkPrelude = R"CUDA(
__device__ __forceinline__ unsigned mf_smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mf_mbar_init(unsigned long long* b, unsigned cnt) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(mf_smem_u32(b)), "r"(cnt) : "memory");
}
__device__ __forceinline__ void mf_fence_mbar_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void mf_fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void mf_mbar_expect_tx(unsigned long long* b, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mf_smem_u32(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mf_bulk_g2s(void* dst, const void* src, unsigned bytes, unsigned long long* b) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(mf_smem_u32(dst)), "l"(src), "r"(bytes), "r"(mf_smem_u32(b)) : "memory");
}
__device__ __forceinline__ unsigned mf_mbar_try_wait(unsigned long long* b, unsigned parity) {
  unsigned ok;
  asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
               : "=r"(ok) : "r"(mf_smem_u32(b)), "r"(parity) : "memory");
  return ok;
}
// Bounded wait: false after MF_SPIN_LIMIT unsuccessful polls.
#define MF_SPIN_LIMIT (1u << 22)
__device__ __forceinline__ bool mf_mbar_wait_bounded(unsigned long long* b, unsigned parity) {
  for (unsigned i = 0; i < MF_SPIN_LIMIT; i++)
    if (mf_mbar_try_wait(b, parity)) return true;
  return false;
}
)CUDA";

// 2^(j/64), j = 0..63, as double-float pairs {hi, lo} (hi the nearest float,
// lo the nearest float to the remainder), computed in 60-digit decimal
// arithmetic: the table of mf_dw_exp.
const char* const kExp2Table[64] = {
    "{0x1p+0f, 0x0p+0f}", "{0x1.02c9a4p+0f, -0x1.887fap-28f}",
    "{0x1.059b0ep+0f, -0x1.9d4f52p-25f}", "{0x1.087452p+0f, -0x1.e2990ep-26f}",
    "{0x1.0b5586p+0f, 0x1.9f3122p-25f}", "{0x1.0e3ec4p+0f, -0x1.a585ccp-25f}",
    "{0x1.11301ep+0f, -0x1.fdb496p-25f}", "{0x1.1429aap+0f, 0x1.d525bcp-25f}",
    "{0x1.172b84p+0f, -0x1.c15742p-27f}", "{0x1.1a35bep+0f, 0x1.6df96ep-25f}",
    "{0x1.1d4874p+0f, -0x1.d2e8cap-25f}", "{0x1.2063b8p+0f, 0x1.0c519ap-25f}",
    "{0x1.2387a6p+0f, 0x1.ceac48p-25f}", "{0x1.26b456p+0f, 0x1.789f38p-26f}",
    "{0x1.29e9ep+0f, -0x1.5c0424p-25f}", "{0x1.2d285ap+0f, 0x1.b900c2p-26f}",
    "{0x1.306fep+0f, 0x1.4636e2p-25f}", "{0x1.33c08cp+0f, -0x1.b37d2p-25f}",
    "{0x1.371a74p+0f, -0x1.18aac6p-25f}", "{0x1.3a7db4p+0f, -0x1.634c02p-25f}",
    "{0x1.3dea64p+0f, 0x1.824684p-25f}", "{0x1.4160a2p+0f, 0x1.f72e2ap-28f}",
    "{0x1.44e086p+0f, 0x1.8624b4p-30f}", "{0x1.486a2cp+0f, -0x1.47d866p-25f}",
    "{0x1.4bfdaep+0f, -0x1.593abcp-25f}", "{0x1.4f9b28p+0f, -0x1.2c5a6cp-25f}",
    "{0x1.5342b6p+0f, -0x1.2c561p-25f}", "{0x1.56f474p+0f, -0x1.295b04p-25f}",
    "{0x1.5ab07ep+0f, -0x1.5bd5ecp-27f}", "{0x1.5e76f2p+0f, -0x1.4a5bd6p-25f}",
    "{0x1.6247ecp+0f, -0x1.f8b55p-25f}", "{0x1.662388p+0f, 0x1.2a9112p-27f}",
    "{0x1.6a09e6p+0f, 0x1.9fcef4p-26f}", "{0x1.6dfb24p+0f, -0x1.cd72e8p-27f}",
    "{0x1.71f75ep+0f, 0x1.1d8beep-25f}", "{0x1.75feb6p+0f, -0x1.37b306p-25f}",
    "{0x1.7a1148p+0f, -0x1.829fdp-25f}", "{0x1.7e2f34p+0f, -0x1.261634p-25f}",
    "{0x1.82589ap+0f, -0x1.accc7cp-26f}", "{0x1.868d9ap+0f, -0x1.2edb44p-26f}",
    "{0x1.8ace54p+0f, 0x1.15506ep-27f}", "{0x1.8f1aeap+0f, -0x1.baa232p-26f}",
    "{0x1.93737cp+0f, -0x1.e64744p-25f}", "{0x1.97d82ap+0f, -0x1.0d8d84p-31f}",
    "{0x1.9c4918p+0f, 0x1.51f848p-27f}", "{0x1.a0c668p+0f, -0x1.2886a6p-26f}",
    "{0x1.a5503cp+0f, -0x1.b83b54p-25f}", "{0x1.a9e6b6p+0f, -0x1.50c048p-25f}",
    "{0x1.ae89fap+0f, -0x1.a94b14p-26f}", "{0x1.b33a2cp+0f, -0x1.ec3a82p-26f}",
    "{0x1.b7f77p+0f, -0x1.a09438p-25f}", "{0x1.bcc1eap+0f, -0x1.f687c6p-25f}",
    "{0x1.c199bep+0f, -0x1.3d56b2p-27f}", "{0x1.c67f12p+0f, 0x1.cafa2ap-25f}",
    "{0x1.cb720ep+0f, -0x1.8837ccp-27f}", "{0x1.d072d4p+0f, 0x1.40f13p-25f}",
    "{0x1.d5818ep+0f, -0x1.822dbcp-27f}", "{0x1.da9e6p+0f, 0x1.ed9942p-27f}",
    "{0x1.dfc974p+0f, -0x1.908c94p-25f}", "{0x1.e502eep+0f, 0x1.e2cffep-26f}",
    "{0x1.ea4afap+0f, 0x1.52486cp-27f}", "{0x1.efa1bep+0f, 0x1.cc2b44p-25f}",
    "{0x1.f50766p+0f, -0x1.246ebp-26f}", "{0x1.fa7c18p+0f, 0x1.9e90d8p-28f}"};

// The 128-entry table of mf_dw_log: for c_j = 1 + (2j+1)/256,
// {hi(ln c_j), lo(ln c_j), 1/c_j, c_j} as exact float literals; and the
// 64-entry table of mf_dw_exp.
std::string dw_log_table() {
  std::ostringstream o;
  {
    const double ln2 = std::log(2.0);
    const float hi = float(ln2), lo = float(ln2 - double(hi));
    char b[160];
    std::snprintf(b, sizeof b, "#define MF_LN2_HI %af\n#define MF_LN2_LO %af\n", double(hi), double(lo));
    o << b;
  }
  o << "__device__ const float4 mf_dw_logtab_g[128] = {\n";
  for (int j = 0; j < 128; j++) {
    const double c = 1.0 + (2.0 * j + 1.0) / 256.0;
    const double L = std::log(c);
    const float lh = float(L);
    const float ll = float(L - double(lh));
    const float ic = float(1.0 / c);
    char b[200];
    std::snprintf(b, sizeof b, "  {%af, %af, %af, %af},\n", double(lh), double(ll), double(ic), c);
    o << b;
  }
  o << "};\n";
  o << "__device__ const float2 mf_dw_exptab_g[64] = {\n";
  for (const char* row : kExp2Table) o << "  " << row << ",\n";
  o << "};\n";
  return o.str();
}

}  // namespace

OpCount count_ops(const std::vector<std::string>& inputs, const std::vector<std::string>& params,
                  const std::vector<std::string>& exprs) {
  Dag dag(inputs, params);
  std::vector<int> roots;
  for (auto& e : exprs) roots.push_back(dag.parse(e));
  auto live = reachable(dag.nodes(), roots);
  OpCount c;
  for (size_t i = 0; i < dag.nodes().size(); i++) {
    if (!live[i]) continue;
    const Node& n = dag.nodes()[i];
    if (n.op == Op::Const || n.op == Op::Input || n.op == Op::Param) continue;
    c.nodes++;
    if (n.uniform) {
      c.uniform++;
      continue;
    }
    c.per_event++;
    if (is_unary_fn(n.op) || n.op == Op::Pow) c.transcendental++;
    if (n.op == Op::Rcp || n.op == Op::Div) c.divisions++;
  }
  return c;
}

LoweredKernel lower(const std::string& name, Kind kind, Elem elem, const std::vector<std::string>& inputs,
                    const std::vector<std::string>& params, const std::vector<std::string>& exprs,
                    const GenerateSpec* gen, bool native_f64, int vec_req, int block_req, bool f32_arith,
                    bool direct_loads, int stages_req, const std::vector<std::string>& param_defs) {
  std::vector<std::string> in_names = inputs;
  if (kind == Kind::Generate) {
    if (!gen) throw std::runtime_error("generate kernel without generate spec");
    in_names = gen->dims;
  }
  Dag dag(in_names, params);
  // FP32 arithmetic keeps the text's own operations: which products the
  // compiler fuses into sums, and so the last bit, follows them
  dag.share_exchanged = elem == Elem::F64 && !f32_arith;
  std::vector<int> roots0;
  for (auto& e : exprs) roots0.push_back(dag.parse(e));
  std::vector<int> source_inputs;
  {
    const auto& n0 = dag.nodes();
    const auto l0 = reachable(n0, roots0);
    std::set<int> u;
    for (size_t i = 0; i < n0.size(); i++)
      if (l0[i] && n0[i].op == Op::Input) u.insert(n0[i].index);
    source_inputs.assign(u.begin(), u.end());
  }
  const bool st32 = (elem == Elem::F32);
  // REDUCE kernels read prepared columns when that pays: double-float
  // kernels always (FP64 values stored pre-split as float pairs, so the event
  // loop does no splitting), FP32 and native FP64 kernels when linearly
  // dependent columns fold. FP32-over-FP64 kernels read the source columns.
  FoldResult fold;
  int prep = LoweredKernel::PrepNone;
  if (kind == Kind::Reduce && !f32_arith) {
    fold = fold_columns(dag, roots0, param_defs);
    const bool dw = !st32 && !native_f64;
    if (fold.rewritten && (dw || fold.folded))
      prep = dw ? LoweredKernel::PrepPair : st32 ? LoweredKernel::PrepF32 : LoweredKernel::PrepF64;
  }
  const Dag& G = prep ? *fold.dag : dag;
  const std::vector<int>& roots = prep ? fold.roots : roots0;
  const auto& ns = G.nodes();
  auto live = reachable(ns, roots);

  // Arithmetic type: REDUCE kernels compute in the element type (the FP32
  // variant is the mixed-precision path); STORE kernels (event-only
  // precompute) compute in FP64 and round once on store; GENERATE kernels
  // compute in the element type like the reference's generate kernel.
  const bool ar32 = st32 && kind != Kind::Store;
  Emitter em{ns, ar32};
  const std::string ST = st32 ? "float" : "double";
  const std::string AT = ar32 ? "float" : "double";

  LoweredKernel out;
  out.entry = "mf_" + std::string(kind == Kind::Reduce ? "reduce" : kind == Kind::Store ? "store" : "generate");
  // GENERATE and STORE: small blocks, whose ends leave less of an SM idle
  // (S+P-wave precompute, 1M events: 71.8 us in blocks of 256, 68.9 of 128)
  out.block = kind == Kind::Reduce ? 256 : 128;
  out.vec = (kind == Kind::Generate) ? 1 : (st32 ? 4 : 2);
  if (kind == Kind::Reduce) {
    out.pipelined = !direct_loads;
    // double-float bodies: one event per thread per iteration, 512 threads
    // (measured fastest on GB300 for the K*mumu gradient kernel)
    const bool dw_default = !st32 && !native_f64 && !f32_arith;
    if (dw_default) {
      // two events per thread (one 16-byte load per prepared column) for
      // gradient-sized kernels, measured fastest on GB300 for the K*mumu
      // gradient; many-output kernels (Hessians) take one event per thread so
      // their accumulators stay in registers
      out.vec = (!out.pipelined && exprs.size() <= 16) ? 2 : 1;
    }
    // FP32 Hessian-sized kernels: one event per thread as well (measured on
    // GB300: K*mumu P-wave Hessian 12.1 vs 13.4 us at four events per thread,
    // S+P-wave Hessian, 105 outputs, 58.7 vs 70.6 us per 1M events)
    if (st32 && !out.pipelined && exprs.size() > 16) out.vec = 1;
    if (vec_req == 1 || vec_req == 2 || (vec_req == 4 && st32)) out.vec = vec_req;
    if (block_req >= 64 && block_req <= 1024 && block_req % 32 == 0) out.block = block_req;
    // bulk-copy pipeline: shared-memory stages; direct loads: loop unroll
    // factor (1 = none). Gradient-sized kernels (at most 16 outputs) unroll
    // twice by default: with batched evaluations overlapping, the next
    // iteration's loads issued before this one's arithmetic measured fastest
    // on GB300 (K*mumu gradient 11.4 vs 12.1 us per 1M-event evaluation in
    // double-float, 5.9 vs 6.5 us in FP32); Hessian-sized kernels keep their
    // accumulators in registers with one iteration in flight.
    // Many-output double-float kernels (the S+P-wave Hessian: 105 outputs)
    // cannot keep every per-thread partial in registers: the outputs beyond
    // acc_reg keep theirs in shared memory instead (each thread its own
    // column, 8 bytes per output), in blocks of 64 threads unless a block
    // size is asked for, so that the kernel neither spills nor reads the
    // dataset more than once (S+P-wave Hessian at 1M events, batched: 157 us,
    // against 301 us spilling and 189 us as three register-only kernels).
    // FP32 partials are cheap enough that the shared-memory traffic costs more
    // than it saves (85 us against 49 us as three kernels): not for FP32.
    if (!out.pipelined && int(exprs.size()) > kAccRegMax && dw_default) {
      if (block_req == 0) out.block = 64;
      const int room = int(kAccSmemBytes / (8 * size_t(out.block)));
      out.acc_reg = std::max(int(exprs.size()) - room, kAccRegMin);
    }
    if (out.pipelined)
      out.stages = stages_req >= 2 && stages_req <= 8 ? stages_req : (dw_default ? 3 : 4);
    else
      out.stages = stages_req >= 1 && stages_req <= 4 ? stages_req
                                                     : (!native_f64 && exprs.size() <= 16 ? 2 : 1);
    out.tile = out.block * out.vec;
  }
  const int V = out.vec;
  const int M = int(exprs.size());
  const int NP = std::max<int>(1, int(params.size()));

  std::set<int> used;
  for (size_t i = 0; i < ns.size(); i++)
    if (live[i] && ns[i].op == Op::Input) used.insert(ns[i].index);
  out.used_inputs.assign(used.begin(), used.end());
  out.source_inputs = source_inputs;
  out.prep = prep;
  if (prep) out.prep_cols = fold.cols;
  const bool pair = prep == LoweredKernel::PrepPair;
  if (pair && V != 1 && V != 2) throw std::runtime_error("double-float kernels take 1 or 2 events per thread");

  std::ostringstream s;
  s << "// MoreFit CUDA backend: generated kernel '" << name << "' (" << (kind == Kind::Reduce ? "reduce"
                                                                          : kind == Kind::Store ? "store"
                                                                                                : "generate")
    << ", " << ST << " storage, "
    << (kind == Kind::Reduce && !st32 && !native_f64 ? std::string("double-float") : AT) << " arithmetic)\n";
  if (prep) {
    s << "// reads " << fold.cols.size() << " prepared columns (" << (pair ? "FP64 as float pairs" : st32 ? "FP32" : "FP64")
      << ") derived from " << fold.source_columns << " source columns:\n";
    for (size_t m = 0; m < fold.cols.size(); m++) {
      s << "//   y" << m << " =";
      for (auto& [col, c] : fold.cols[m]) s << " + " << c << "*" << in_names[col];
      s << "\n";
    }
  }
  s << "// outputs:\n";
  for (size_t j = 0; j < exprs.size(); j++) s << "//   [" << j << "] " << exprs[j].substr(0, 160) << "\n";
  s << kPrelude;
  if (out.acc_reg <= 0 || out.acc_reg > M) out.acc_reg = M;
  const int NREG = out.acc_reg;
  s << "#define MF_BLOCK " << out.block << "\n#define MF_NOUT " << M << "\n#define MF_NPAR " << NP << "\n";
  // per-thread partials of outputs [0, MF_NREG) in registers, the rest in shared memory
  s << "#define MF_NREG " << NREG << "\n";
  // launch bounds of the event-loop entries
  s << "#define MF_BOUNDS __launch_bounds__(MF_BLOCK)\n";
  // combine of block partial rows: MF_GRP threads (a warp's lanes at most, the
  // whole block for a single output) share an output's rows, each with MF_Q
  // loads in flight; kernels of many outputs, whose grids of small blocks leave
  // hundreds of rows, combine them in groups of MF_ROWS blocks first
  const int grp = M == 1 ? out.block : std::max(1, std::min(32, out.block / M));
  int q = 2;  // a power of two: the rows of a round are added as a tree
  while (q < 16 && q * grp < (M == 1 ? 8 * 152 : 608)) q *= 2;
  s << "#define MF_GRP " << grp << "\n#define MF_Q " << q << "\n";
  s << "#define MF_ROWS " << (M > kAccRegMax ? kCombineRows : 0) << "\n";
  // shared scratch of the block reduction (a row per warp) and the combine (MF_GRP rows)
  s << "#define MF_PART " << std::max(out.block / 32, grp) * M << "\n";
  s << "struct mf_par { double v[MF_NPAR]; };\n";

  // Parameter-only prologue (u*), emitted once per thread.
  auto emit_params_and_uniform = [&](std::ostringstream& o, const std::string& src) {
    std::set<int> used_params;
    for (size_t i = 0; i < ns.size(); i++)
      if (live[i] && ns[i].op == Op::Param) used_params.insert(ns[i].index);
    for (int k : used_params) o << "  const " << AT << " p" << k << " = (" << AT << ")" << src << "[" << k << "];\n";
    for (size_t i = 0; i < ns.size(); i++) {
      if (!live[i] || !ns[i].uniform) continue;
      Op op = ns[i].op;
      if (op == Op::Const || op == Op::Param) continue;
      o << "  " << em.stmt(int(i), "u") << "\n";
    }
  };
  // Per-event body: x<k> already defined; defines e<id> and r<j>.
  auto emit_body = [&](std::ostringstream& o, const std::string& indent) {
    for (size_t i = 0; i < ns.size(); i++) {
      if (!live[i] || ns[i].uniform) continue;
      Op op = ns[i].op;
      if (op == Op::Input) continue;
      o << indent << em.stmt(int(i), "e") << "\n";
    }
    for (int j = 0; j < M; j++) o << indent << "const " << AT << " r" << j << " = " << em.ref(roots[j], "e") << ";\n";
  };

  if (kind == Kind::Reduce || (kind == Kind::Store && !native_f64)) {
    // Arithmetic of the per-event body: FP32 (mixed precision), FP64, or
    // double-float on FP32 pairs (the default for FP64 storage, and for
    // STORE kernels unless native FP64 is asked for).
    // F32S: FP64 storage, FP32 arithmetic, except that a sum or difference of
    // an input column and a parameter-only value is formed in FP64 before it
    // is rounded (keeps m - mu exact for observables with a large offset).
    enum class Ar { F32, F64, DW, F32S } ar =
        kind == Kind::Store ? Ar::DW : st32 ? Ar::F32 : (f32_arith ? Ar::F32S : (native_f64 ? Ar::F64 : Ar::DW));
    auto is_leafish = [&](int k) {
      const Op o = ns[k].op;
      return o == Op::Input || ns[k].uniform;
    };
    // per-event nodes evaluated in FP64 under F32S
    std::vector<char> dnode(ns.size(), 0);
    if (ar == Ar::F32S)
      for (size_t i = 0; i < ns.size(); i++) {
        const Node& n = ns[i];
        if (!live[i] || n.uniform || (n.op != Op::Add && n.op != Op::Sub)) continue;
        if (is_leafish(n.a) && is_leafish(n.b) && (ns[n.a].op == Op::Input || ns[n.b].op == Op::Input)) dnode[i] = 1;
      }
    // Double-float exp and pow (table-driven, FP32 pipe) in REDUCE kernels,
    // whose non-finite sums are re-evaluated in native FP64 by the runtime;
    // STORE kernels write columns and keep FP64 exp / pow (full FP64 range).
    const bool dw_exp = kind == Kind::Reduce;
    bool has_log = false, has_exp = false;
    for (size_t i = 0; i < ns.size(); i++) {
      if (!live[i] || ns[i].uniform) continue;
      if (ns[i].op == Op::Log || (dw_exp && ns[i].op == Op::Pow)) has_log = true;
      if (dw_exp && (ns[i].op == Op::Exp || ns[i].op == Op::Pow)) has_exp = true;
    }
    // The double-float library is always present: every cross-thread sum
    // (warp, block, grid) runs in double-float on the FP32 pipe.
    s << dw_log_table() << kDwPrelude << (kind == Kind::Reduce ? kBulkPrelude : "");
    // ---- leaves and statements of the per-event body ----
    auto eref = [&](int id) -> std::string {
      const Node& n = ns[id];
      if (ar == Ar::F32S) {  // float view of any node
        if (n.op == Op::Const) return fmt_const(n.value, true);
        if (n.op == Op::Input) return "(float)x" + std::to_string(n.index);
        if (n.op == Op::Param) return "pf" + std::to_string(n.index);
        if (n.uniform) return "uf" + std::to_string(id);
        if (dnode[id]) return "(float)e" + std::to_string(id);
        return "e" + std::to_string(id);
      }
      if (n.op == Op::Const) {
        if (ar == Ar::F32) return fmt_const(n.value, true);
        if (ar == Ar::F64) return fmt_const(n.value, false);
        const float h = float(n.value);
        const float l = float(n.value - double(h));
        char b[96];
        std::snprintf(b, sizeof b, "mf_dw_make(%af, %af)", double(h), double(l));
        return b;
      }
      if (n.op == Op::Input) return "x" + std::to_string(n.index);
      const std::string sfx = ar == Ar::F32 ? "f" : ar == Ar::DW ? "w" : "";
      if (n.op == Op::Param) return "p" + sfx + std::to_string(n.index);
      if (n.uniform) return "u" + sfx + std::to_string(id);
      return "e" + std::to_string(id);
    };
    auto dref = [&](int k) -> std::string {  // FP64 view of an input / uniform / constant (F32S only)
      const Node& n = ns[k];
      if (n.op == Op::Const) return fmt_const(n.value, false);
      if (n.op == Op::Input) return "x" + std::to_string(n.index);
      if (n.op == Op::Param) return "p" + std::to_string(n.index);
      return "u" + std::to_string(k);
    };
    std::map<int, std::pair<int, int>> sincos_pair;  // operand -> (sin node, cos node)
    if (ar == Ar::DW) sincos_pair = sincos_pairs(ns, live);
    // Double-float REDUCE bodies: sums of (value x parameter-only factor)
    // terms become compensated dot products, and an output that is a product
    // used nowhere else is multiplied straight into its accumulator.
    std::vector<int> uses(ns.size(), 0), consumer(ns.size(), -1);
    std::vector<char> skip(ns.size(), 0);
    std::map<int, std::vector<std::pair<int, int>>> chains;  // chain root -> its terms (a, b)
    std::vector<std::pair<int, int>> fused(roots.size(), {-1, -1});
    std::vector<int> logprod(roots.size(), -1);  // output j = log(node) summed as a running product
    // ... plus (or minus) a parameter-only value per event (the normalisation
    // term of logprob_normalised, pdf.hh:103-106): log(x) + u or log(x) - u
    std::vector<int> logadd(roots.size(), -1), logsign(roots.size(), 0), lognode(roots.size(), -1);
    // Double-float outputs x + u or x - u with u parameter-only (the
    // normalisation terms of Hessian outputs): x is accumulated and the
    // thread's event count times u added once, before the block reduction.
    std::vector<int> addu(roots.size(), -1), addsign(roots.size(), 0), accnode(roots);
    // Double-float outputs x * u with u parameter-only: x is accumulated and
    // multiplied by u once (the S+P-wave Hessian scales 36 of its 105 outputs
    // by (1 - FS): a product per event and output less).
    std::vector<std::vector<int>> scale(roots.size());
    // FP32 REDUCE bodies (mixed precision) whose only output is the logarithm
    // of a dot product of per-event values with parameter-only factors (the
    // fitter's NLL kernel for a density linear in its prepared columns): that
    // dot product is kept as a compensated double-float value and its
    // logarithm summed as a double-float running product, so the NLL carries
    // no per-event FP32 rounding. Minuit2 takes function values from this
    // kernel (minuit2_grad_fcn::DoEval, fitter.hh:131-136) and compares them
    // in its line searches, which FP32 rounding noise of ~1e-7 per event
    // (1e-4 in the NLL of 1M events) would disturb. Kernels with gradient
    // outputs keep plain FP32 arithmetic: Minuit2 discards their NLL value
    // (fitter.hh:138-144), and their cost per event stays at the FP32 rate.
    std::set<int> f32_dw_chain;  // chain roots evaluated in double-float under F32
    if ((ar == Ar::DW || ar == Ar::F32) && kind == Kind::Reduce) {
      for (size_t i = 0; i < ns.size(); i++) {
        if (!live[i] || ns[i].uniform || ns[i].op == Op::Input) continue;
        for (int c : {ns[i].a, ns[i].b, ns[i].c})
          if (c >= 0) {
            uses[c]++;
            consumer[c] = int(i);
          }
      }
      for (int r : roots) {
        uses[r]++;
        consumer[r] = -1;
      }
      auto is_term = [&](int k) {
        const Node& n = ns[k];
        return n.op == Op::Mul && !n.uniform && uses[k] == 1 && (ns[n.a].uniform || ns[n.b].uniform);
      };
      std::vector<char> chain(ns.size(), 0);
      for (size_t i = 0; i < ns.size(); i++) {
        const Node& n = ns[i];
        if (!live[i] || n.uniform || n.op != Op::Add) continue;
        auto part = [&](int c) { return is_term(c) || (chain[c] && uses[c] == 1); };
        if (part(n.a) && part(n.b)) chain[i] = 1;
      }
      std::function<void(int, std::vector<std::pair<int, int>>&)> collect = [&](int k, auto& terms) {
        if (chain[k]) {
          collect(ns[k].a, terms);
          collect(ns[k].b, terms);
        } else {
          terms.push_back({ns[k].a, ns[k].b});
        }
      };
      // Output r as log(x) [+ or - u]: the Log node (used only there), u, sign.
      auto log_form = [&](int r, int& lg, int& u, int& sign) {
        lg = -1;
        u = -1;
        sign = 0;
        const Node& n = ns[r];
        if (n.uniform || uses[r] != 1) return false;
        auto is_log = [&](int k) { return ns[k].op == Op::Log && !ns[k].uniform && uses[k] == 1; };
        if (is_log(r)) {
          lg = r;
          return true;
        }
        if (n.op == Op::Add || n.op == Op::Sub) {
          if (is_log(n.a) && ns[n.b].uniform) {
            lg = n.a;
            u = n.b;
            sign = n.op == Op::Add ? 1 : -1;
            return true;
          }
          if (n.op == Op::Add && is_log(n.b) && ns[n.a].uniform) {
            lg = n.b;
            u = n.a;
            sign = 1;
            return true;
          }
        }
        return false;
      };
      if (ar == Ar::F32) {
        // only the chain that is the argument of the single output's logarithm
        std::set<int> wanted;
        for (int r : roots) {
          int lg, u, sg;
          if (M == 1 && log_form(r, lg, u, sg) && chain[ns[lg].a]) wanted.insert(ns[lg].a);
        }
        for (size_t i = 0; i < ns.size(); i++)
          if (chain[i] && !wanted.count(int(i))) {
            // keep chain marks only below a wanted root
            bool below = false;
            for (int c = consumer[i]; c >= 0 && !below; c = (uses[c] == 1 && chain[c]) ? consumer[c] : -1)
              below = wanted.count(c) > 0;
            if (!below) chain[i] = 0;
          }
        f32_dw_chain = wanted;
      }
      for (size_t i = 0; i < ns.size(); i++) {
        if (!chain[i]) continue;
        const bool absorbed = uses[i] == 1 && consumer[i] >= 0 && chain[consumer[i]];
        if (absorbed) continue;
        std::vector<std::pair<int, int>> terms;
        collect(int(i), terms);
        chains[int(i)] = terms;
        // every node of the chain below its root is folded into the root's statement
        std::function<void(int)> mark = [&](int k) {
          if (k != int(i)) skip[k] = 1;
          if (chain[k]) {
            mark(ns[k].a);
            mark(ns[k].b);
          }
        };
        mark(int(i));
      }
      for (size_t j = 0; j < roots.size(); j++) {
        const int r = roots[j];
        const Node& n = ns[r];
        int lg = -1, u = -1, sg = 0;
        const bool lf = !skip[r] && log_form(r, lg, u, sg);
        if (ar == Ar::F32) {
          if (lf && f32_dw_chain.count(ns[lg].a)) {
            logprod[j] = ns[lg].a;
            logadd[j] = u;
            logsign[j] = sg;
            lognode[j] = lg;
            skip[r] = 1;
            skip[lg] = 1;
          }
          continue;
        }
        // what output j accumulates of node x: parameter-only factors aside, a
        // product multiplied straight into the accumulator
        auto accumulate = [&](int x) {
          auto product = [&](int k) {
            return ns[k].op == Op::Mul && !ns[k].uniform && uses[k] == 1 && !chains.count(k) && !skip[k];
          };
          while (product(x) && ns[ns[x].a].uniform != ns[ns[x].b].uniform) {
            const bool first = ns[ns[x].a].uniform;
            scale[j].push_back(first ? ns[x].a : ns[x].b);
            skip[x] = 1;
            x = first ? ns[x].b : ns[x].a;
          }
          accnode[j] = x;
          if (product(x)) {
            fused[j] = {ns[x].a, ns[x].b};
            skip[x] = 1;
          }
        };
        if (n.op == Op::Mul && !n.uniform && uses[r] == 1 && !chains.count(r) && !skip[r]) accumulate(r);
        if (ar == Ar::DW && !lf && !skip[r] && uses[r] == 1 && !n.uniform && (n.op == Op::Add || n.op == Op::Sub)) {
          int x = -1, u = -1, sg = 0;
          if (ns[n.b].uniform && !ns[n.a].uniform) {
            x = n.a;
            u = n.b;
            sg = n.op == Op::Add ? 1 : -1;
          } else if (n.op == Op::Add && ns[n.a].uniform && !ns[n.b].uniform) {
            x = n.b;
            u = n.a;
            sg = 1;
          }
          if (x >= 0 && !skip[x] && !chains.count(x)) {
            addu[j] = u;
            addsign[j] = sg;
            skip[r] = 1;
            accumulate(x);
          }
        }
        // an output that is the logarithm of a per-event value (plus or minus a
        // parameter-only value), used nowhere else: sum of logs = log of the
        // product (one multiply per event), plus the event count times u
        if (lf && !skip[r]) {
          logprod[j] = ns[lg].a;
          logadd[j] = u;
          logsign[j] = sg;
          lognode[j] = lg;
          skip[r] = 1;
          skip[lg] = 1;
        }
      }
    }
    bool has_addu = false;
    for (int u : addu) has_addu = has_addu || u >= 0;
    // Double-float REDUCE bodies: the powers of one per-event base, and its
    // logarithm, share ln|base| (a third of a pow's instructions): base ->
    // the first statement that uses it, which defines la<base>.
    std::map<int, int> pow_base;
    if (ar == Ar::DW && dw_exp) {
      for (size_t i = 0; i < ns.size(); i++)
        if (live[i] && !ns[i].uniform && ns[i].op == Op::Pow && !ns[ns[i].a].uniform) pow_base[ns[i].a] = -1;
      for (size_t i = 0; i < ns.size(); i++)
        if (live[i] && !ns[i].uniform && !skip[i] && (ns[i].op == Op::Pow || ns[i].op == Op::Log)) {
          auto it = pow_base.find(ns[i].a);
          if (it != pow_base.end() && it->second < 0) it->second = int(i);
        }
    }
    auto rcp_of = [&](int a) {  // the live per-event reciprocal of node a, or -1
      for (size_t i = 0; i < ns.size(); i++)
        if (live[i] && !ns[i].uniform && ns[i].op == Op::Rcp && ns[i].a == a) return int(i);
      return -1;
    };
    auto logabs = [&](int id) -> std::string {  // defined with its first use
      const int b = ns[id].a;
      if (pow_base.at(b) != id) return "";
      return "const mf_dw la" + std::to_string(b) + " = mf_dw_logabs(" + eref(b) + ", mf_logtab); ";
    };
    auto estmt = [&](int id) -> std::string {
      const Node& n = ns[id];
      if (ar == Ar::F32S && dnode[id])
        return "const double e" + std::to_string(id) + " = " + dref(n.a) + (n.op == Op::Add ? " + " : " - ") + dref(n.b) +
               ";";
      const std::string T = ar == Ar::F32 || ar == Ar::F32S ? "float" : ar == Ar::F64 ? "double" : "mf_dw";
      const std::string lhs = "const " + std::string(n.op == Op::Cmp ? "bool" : T) + " e" + std::to_string(id) + " = ";
      const std::string A = n.a >= 0 ? eref(n.a) : "", B = n.b >= 0 ? eref(n.b) : "", Cc = n.c >= 0 ? eref(n.c) : "";
      if (ar == Ar::F32 && skip[id]) return "";
      if (ar == Ar::F32 && chains.count(id)) {
        // terms value x factor, the parameter-only factor as a double-float
        // pair (so that the sum follows the FP64 parameters smoothly)
        const std::string e = "e" + std::to_string(id);
        const auto& terms = chains.at(id);
        std::string c = "mf_dw w" + e + "; { mf_dw t_;";
        for (size_t q = 0; q < terms.size(); q++) {
          const bool a_uni = ns[terms[q].first].uniform;
          const int u = a_uni ? terms[q].first : terms[q].second, v = a_uni ? terms[q].second : terms[q].first;
          std::string cw;
          if (ns[u].op == Op::Const) {
            const float h = float(ns[u].value);
            char b[96];
            std::snprintf(b, sizeof b, "mf_dw_make(%af, %af)", double(h), double(float(ns[u].value - double(h))));
            cw = b;
          } else {
            cw = "uw" + std::to_string(u);
          }
          c += q == 0 ? " t_ = mf_dw_prodfw(" + eref(v) + ", " + cw + ");"
                      : " mf_dw_acc_mulfw(t_, " + eref(v) + ", " + cw + ");";
        }
        return c + " w" + e + " = mf_dw_renorm(t_); } const float " + e + " = w" + e + ".h;";
      }
      if (ar != Ar::DW) {
        const bool f = ar == Ar::F32 || ar == Ar::F32S;
        switch (n.op) {
          case Op::Add: return lhs + A + " + " + B + ";";
          case Op::Sub: return lhs + A + " - " + B + ";";
          case Op::Mul: return lhs + A + " * " + B + ";";
          case Op::Div: return lhs + A + " / " + B + ";";
          case Op::Neg: return lhs + "-" + A + ";";
          case Op::Rcp: return lhs + fn_name(Op::Rcp, f) + "(" + A + ");";
          case Op::Pow: return lhs + fn_name(Op::Pow, f) + "(" + A + ", " + B + ");";
          case Op::Cmp: return lhs + "(" + A + " " + cmp_str(n.cmp) + " " + B + ");";
          case Op::Select: return lhs + "(" + A + " ? " + B + " : " + Cc + ");";
          default:
            if (is_unary_fn(n.op)) return lhs + fn_name(n.op, f) + "(" + A + ");";
        }
        throw std::runtime_error("emit: unexpected node");
      }
      auto D = [](const std::string& v) { return "mf_dw_to_double(" + v + ")"; };
      if (skip[id]) return "";
      auto ch = chains.find(id);
      if (ch != chains.end()) {
        std::string c = "mf_dw e" + std::to_string(id) + "; {";
        for (auto& [ta, tb] : ch->second)
          c += (&ta == &ch->second.front().first ? " mf_dw t_ = mf_dw_prod(" : " mf_dw_acc_mul(t_, ") + eref(ta) + ", " +
               eref(tb) + ");";
        return c + " e" + std::to_string(id) + " = mf_dw_renorm(t_); }";
      }
      switch (n.op) {
        case Op::Add: return lhs + "mf_dw_add(" + A + ", " + B + ");";
        case Op::Sub: return lhs + "mf_dw_sub(" + A + ", " + B + ");";
        case Op::Mul: return lhs + "mf_dw_mul(" + A + ", " + B + ");";
        case Op::Div: return lhs + "mf_dw_mul(" + A + ", mf_dw_rcp(" + B + "));";
        case Op::Neg: return lhs + "mf_dw_neg(" + A + ");";
        case Op::Rcp:
          // 1/a^2 where 1/a is there already: its square
          if (ns[n.a].op == Op::Mul && ns[n.a].a == ns[n.a].b) {
            const int r = rcp_of(ns[n.a].a);
            if (r >= 0 && r < id && !skip[r]) return lhs + "mf_dw_mul(" + eref(r) + ", " + eref(r) + ");";
          }
          return lhs + "mf_dw_rcp(" + A + ");";
        case Op::Log:
          if (pow_base.count(n.a)) return logabs(id) + lhs + "mf_dw_log_of(" + A + ", la" + std::to_string(n.a) + ");";
          return lhs + "mf_dw_log(" + A + ", mf_logtab);";
        case Op::Sqrt: return lhs + "mf_dw_sqrt(" + A + ");";
        case Op::Sin:
        case Op::Cos: {
          // sin and cos of the same operand share one reduction and both polynomials
          auto it = sincos_pair.find(n.a);
          if (it == sincos_pair.end()) return lhs + (n.op == Op::Sin ? "mf_dw_sin(" : "mf_dw_cos(") + A + ");";
          const int first = std::min(it->second.first, it->second.second);
          if (id != first) return "";  // defined with the first of the two
          const std::string sn = "e" + std::to_string(it->second.first), cn = "e" + std::to_string(it->second.second);
          return "mf_dw " + sn + ", " + cn + "; mf_dw_sincos(" + A + ", &" + sn + ", &" + cn + ");";
        }
        case Op::Pow:
          if (dw_exp && pow_base.count(n.a))
            return logabs(id) + lhs + "mf_dw_pow(" + A + ", " + B + ", la" + std::to_string(n.a) + ", mf_exptab);";
          if (dw_exp)  // a parameter-only base
            return lhs + "mf_dw_pow(" + A + ", " + B + ", mf_dw_logabs(" + A + ", mf_logtab), mf_exptab);";
          return lhs + "mf_dw_from_double(pow(" + D(A) + ", " + D(B) + "));";
        case Op::Exp:
          if (dw_exp) return lhs + "mf_dw_exp(" + A + ", mf_exptab);";
          return lhs + "mf_dw_from_double(exp(" + D(A) + "));";
        case Op::Cmp:
          switch (n.cmp) {
            case CmpOp::Gt: return lhs + "mf_dw_gt(" + A + ", " + B + ");";
            case CmpOp::Lt: return lhs + "mf_dw_lt(" + A + ", " + B + ");";
            case CmpOp::Ge: return lhs + "mf_dw_ge(" + A + ", " + B + ");";
            case CmpOp::Le: return lhs + "mf_dw_le(" + A + ", " + B + ");";
            case CmpOp::Eq: return lhs + "mf_dw_eq(" + A + ", " + B + ");";
            case CmpOp::Ne: return lhs + "!mf_dw_eq(" + A + ", " + B + ");";
          }
          break;
        case Op::Select: return lhs + "(" + A + " ? " + B + " : " + Cc + ");";
        default:
          if (is_unary_fn(n.op)) return lhs + "mf_dw_from_double(" + fn_name(n.op, false) + "(" + D(A) + "));";
      }
      throw std::runtime_error("emit: unexpected node");
    };
    if (kind == Kind::Store) {
      // Event-only precompute in double-float: inputs split with rounding
      // and outputs joined by integer operations (the FP64 pipe, 1/64 of the
      // FP32 rate on GB300, is not used per event), parameter-only values
      // evaluated in FP64 once per thread. Bound by instruction issue, most
      // of it on the half-rate integer pipe: the P wave's 1M events took 67.6
      // us at about 1900 instructions per event and take 43.3 at about 1200
      // (136 MB are 20 us at the copy rate); the S+P wave 99.2 and 68.9. What
      // went: the divisions of the square root, the ordered and renormalized
      // sums of the sine's and cosine's Horner steps, and the shifts and
      // special cases of joining a pair.
      std::set<int> uni;
      for (size_t i = 0; i < ns.size(); i++) {
        if (!live[i] || ns[i].uniform || ns[i].op == Op::Input) continue;
        for (int c : {ns[i].a, ns[i].b, ns[i].c})
          if (c >= 0 && ns[c].uniform && ns[c].op != Op::Const) uni.insert(c);
      }
      for (int r : roots)
        if (ns[r].uniform && ns[r].op != Op::Const) uni.insert(r);
      s << "extern \"C\" __global__ void __launch_bounds__(MF_BLOCK) " << out.entry << "(const " << ST
        << "* __restrict__ data, mf_u64 stride, mf_u64 n, mf_par P, " << ST
        << "* __restrict__ outp, mf_u64 out_stride) {\n";
      if (has_log)
        s << "  __shared__ float4 mf_logtab[128];\n"
          << "  for (int q = threadIdx.x; q < 128; q += MF_BLOCK) mf_logtab[q] = mf_dw_logtab_g[q];\n"
          << "  __syncthreads();\n";
      emit_params_and_uniform(s, "P.v");
      for (int k : uni)
        s << "  const mf_dw " << eref(k) << " = mf_dw_from_double(" << dref(k) << ");\n";
      s << "  const mf_u64 step = (mf_u64)gridDim.x * MF_BLOCK;\n";
      s << "  for (mf_u64 i = (mf_u64)blockIdx.x * MF_BLOCK + threadIdx.x; i < n; i += step) {\n";
      for (int k : out.used_inputs)
        s << "    const mf_dw x" << k << " = mf_dw_split_rn((double)data[(mf_u64)" << k << " * stride + i]);\n";
      for (size_t i = 0; i < ns.size(); i++) {
        if (!live[i] || ns[i].uniform || ns[i].op == Op::Input) continue;
        const std::string st = estmt(int(i));
        if (!st.empty()) s << "    " << st << "\n";
      }
      for (int j = 0; j < M; j++) {
        const Node& r = ns[roots[j]];
        if (r.op == Op::Input)  // a copied column stays bit-exact
          s << "    outp[(mf_u64)" << j << " * out_stride + i] = data[(mf_u64)" << r.index << " * stride + i];\n";
        else if (st32)  // h + l rounded once
          s << "    { const mf_dw o = " << eref(roots[j]) << "; outp[(mf_u64)" << j
            << " * out_stride + i] = __fadd_rn(o.h, o.l); }\n";
        else
          s << "    outp[(mf_u64)" << j << " * out_stride + i] = mf_dw_to_double_bits(" << eref(roots[j]) << ");\n";
      }
      s << "  }\n}\n";
      out.source = s.str();
      return out;
    }
    // Uniform (parameter-only) values referenced by the per-event body or by an output.
    std::set<int> uni_used;
    auto note_uniform = [&](int k) {
      if (k >= 0 && ns[k].uniform && ns[k].op != Op::Const) uni_used.insert(k);
    };
    for (size_t i = 0; i < ns.size(); i++) {
      if (!live[i] || ns[i].uniform || ns[i].op == Op::Input || dnode[i]) continue;
      note_uniform(ns[i].a);
      note_uniform(ns[i].b);
      note_uniform(ns[i].c);
    }
    for (int r : roots) note_uniform(r);
    // Parameter-only values: evaluated once per launch on the host and passed
    // pre-rounded in the argument struct (no FP64 work in the kernel, where
    // FP64 issues at 1/64 of the FP32 rate).
    std::map<int, std::string> slot_names;  // node -> C name in the body
    {
      std::vector<UniformSlot> slots;
      int nd = 0, nf = 0;
      auto add_slot = [&](int k, int kind) {
        UniformSlot sl{k, kind, kind == UniformSlot::Double ? nd : nf};
        if (kind == UniformSlot::Double)
          nd++;
        else
          nf += kind == UniformSlot::DwPair ? 2 : 1;
        slots.push_back(sl);
      };
      std::set<int> dslots;  // nodes needed as doubles
      if (ar == Ar::F64) dslots = uni_used;
      if (ar == Ar::F32S)
        for (size_t i = 0; i < ns.size(); i++)
          if (dnode[i]) {
            if (ns[ns[i].a].uniform && ns[ns[i].a].op != Op::Const) dslots.insert(ns[i].a);
            if (ns[ns[i].b].uniform && ns[ns[i].b].op != Op::Const) dslots.insert(ns[i].b);
          }
      for (int k : dslots) {
        add_slot(k, UniformSlot::Double);
        slot_names[k] = ns[k].op == Op::Param ? "p" + std::to_string(ns[k].index) : "u" + std::to_string(k);
      }
      if (ar != Ar::F64)
        for (int k : uni_used)
          add_slot(k, ns[k].op == Op::Cmp ? UniformSlot::Bool : ar == Ar::DW ? UniformSlot::DwPair : UniformSlot::Float);
      if (ar == Ar::F32) {  // double-float factors of the compensated NLL dot product ("uw<node>")
        std::set<int> fac;
        for (auto& [root, terms] : chains)
          for (auto& [ta, tb] : terms) {
            const int u = ns[ta].uniform ? ta : tb;
            if (ns[u].op != Op::Const) fac.insert(u);
          }
        for (int j = 0; j < M; j++)
          if (logadd[j] >= 0 && ns[logadd[j]].op != Op::Const) fac.insert(logadd[j]);
        for (int k : fac) {
          add_slot(k, UniformSlot::DwPair);
          slot_names[k] = "uw" + std::to_string(k);
        }
      }
      out.host_args = true;
      out.nodes = ns;
      out.slots = slots;
      {
        // nodes reachable from the slots, in id order: a node's operands
        // always have smaller ids (hash-consed construction)
        std::vector<char> need(ns.size(), 0);
        for (const auto& sl : slots) need[sl.node] = 1;
        for (size_t i = ns.size(); i-- > 0;) {
          if (!need[i]) continue;
          for (int c : {ns[i].a, ns[i].b, ns[i].c}) {
            if (c >= int(i)) throw std::runtime_error("lowering: operand after its node");
            if (c >= 0) need[c] = 1;
          }
        }
        for (size_t i = 0; i < ns.size(); i++)
          if (need[i]) out.eval_order.push_back(int(i));
      }
      out.nd = std::max(1, nd);
      out.nf = std::max(1, nf);
    }
    auto prologue = [&](std::ostringstream& o, const std::string& P) {
      for (const auto& sl : out.slots) {
        const int k = sl.node;
        const std::string off = std::to_string(sl.offset);
        switch (sl.kind) {
          case UniformSlot::Double: o << "  const double " << slot_names[k] << " = " << P << "d[" << off << "];\n"; break;
          case UniformSlot::Float: o << "  const float " << eref(k) << " = " << P << "f[" << off << "];\n"; break;
          case UniformSlot::Bool: o << "  const bool " << eref(k) << " = " << P << "f[" << off << "] != 0.0f;\n"; break;
          case UniformSlot::DwPair:
            o << "  const mf_dw " << (ar == Ar::F32 ? slot_names[k] : eref(k)) << " = mf_dw_make(" << P << "f["
              << off << "], " << P << "f[" << sl.offset + 1 << "]);\n";
            break;
        }
      }
    };
    auto body = [&](std::ostringstream& o, const std::string& ind) {
      for (size_t i = 0; i < ns.size(); i++) {
        if (!live[i] || ns[i].uniform || ns[i].op == Op::Input) continue;
        const std::string st = estmt(int(i));
        if (!st.empty()) o << ind << st << "\n";
      }
    };
    // Accumulation of output j from the body's value (per thread).
    auto acc_decl = [&](std::ostringstream& o) {
      if (ar == Ar::F32 || ar == Ar::F32S)
        o << "  float acc[MF_NREG], cmp[MF_NREG];\n#pragma unroll\n  for (int j = 0; j < MF_NREG; j++) { acc[j] = 0.0f; cmp[j] = 0.0f; }\n";
      else if (ar == Ar::F64)
        o << "  double acc[MF_NREG];\n#pragma unroll\n  for (int j = 0; j < MF_NREG; j++) acc[j] = 0.0;\n";
      else
        o << "  mf_dw acc[MF_NREG];\n#pragma unroll\n  for (int j = 0; j < MF_NREG; j++) acc[j] = mf_dw_make(0.0f, 0.0f);\n";
      if (NREG < M) {  // this thread's column of the shared partials
        if (ar == Ar::F32 || ar == Ar::F32S)
          o << "  __shared__ float mf_sacc[MF_NOUT - MF_NREG][MF_BLOCK], mf_scmp[MF_NOUT - MF_NREG][MF_BLOCK];\n"
            << "  for (int j = 0; j < MF_NOUT - MF_NREG; j++) { mf_sacc[j][threadIdx.x] = 0.0f; "
               "mf_scmp[j][threadIdx.x] = 0.0f; }\n";
        else if (ar == Ar::F64)
          o << "  __shared__ double mf_sacc[MF_NOUT - MF_NREG][MF_BLOCK];\n"
            << "  for (int j = 0; j < MF_NOUT - MF_NREG; j++) mf_sacc[j][threadIdx.x] = 0.0;\n";
        else
          o << "  __shared__ mf_dw mf_sacc[MF_NOUT - MF_NREG][MF_BLOCK];\n"
            << "  for (int j = 0; j < MF_NOUT - MF_NREG; j++) mf_sacc[j][threadIdx.x] = mf_dw_make(0.0f, 0.0f);\n";
      }
      for (int j = 0; j < M; j++)
        if (logprod[j] >= 0) {
          o << "  mf_dw lpm" << j << " = mf_dw_make(1.0f, 0.0f);\n  int lpe" << j << " = 0;\n";
          if (logadd[j] >= 0) o << "  int lpc" << j << " = 0;\n";
        }
      if (has_addu) o << "  int mf_cnt = 0;  // events of this thread (for the x + u outputs)\n";
    };
    // A thread's partial of output j (and its FP32 compensation): a register
    // or the thread's slot of the shared partials.
    auto accref = [&](int j) {
      return j < NREG ? "acc[" + std::to_string(j) + "]"
                      : "mf_sacc[" + std::to_string(j - NREG) + "][threadIdx.x]";
    };
    auto cmpref = [&](int j) {
      return j < NREG ? "cmp[" + std::to_string(j) + "]"
                      : "mf_scmp[" + std::to_string(j - NREG) + "][threadIdx.x]";
    };
    // Per-thread partials of the log-product outputs, before the block reduction.
    auto acc_finish = [&](std::ostringstream& o) {
      for (int j = 0; j < M; j++) {
        for (size_t q = 0; q < scale[j].size(); q++)
          o << "  " << accref(j) << " = mf_dw_mul(" << (q ? "" : "mf_dw_renorm(") << accref(j) << (q ? "" : ")") << ", "
            << eref(scale[j][q]) << ");\n";
      }
      for (int j = 0; j < M; j++)
        if (addu[j] >= 0)
          o << "  " << accref(j) << " = " << (addsign[j] > 0 ? "mf_dw_add" : "mf_dw_sub") << "(mf_dw_renorm("
            << accref(j) << "), mf_dw_mul(mf_dw_make((float)mf_cnt, 0.0f), " << eref(addu[j]) << "));\n";
      for (int j = 0; j < M; j++) {
        if (logprod[j] < 0) continue;
        const std::string J = std::to_string(j);
        o << "  { mf_dw q_ = mf_dw_logprod_log(lpm" << J << ", lpe" << J << ", mf_logtab);\n";
        if (logadd[j] >= 0) {
          // plus (minus) the thread's event count times u, the count exact in FP32
          std::string uw;
          if (ns[logadd[j]].op == Op::Const) {
            const float h = float(ns[logadd[j]].value);
            char b[96];
            std::snprintf(b, sizeof b, "mf_dw_make(%af, %af)", double(h),
                          double(float(ns[logadd[j]].value - double(h))));
            uw = b;
          } else {
            uw = ar == Ar::F32 ? "uw" + std::to_string(logadd[j]) : eref(logadd[j]);
          }
          o << "    const mf_dw c_ = mf_dw_mul(mf_dw_make((float)lpc" << J << ", 0.0f), " << uw << ");\n"
            << "    q_ = " << (logsign[j] > 0 ? "mf_dw_add" : "mf_dw_sub") << "(q_, c_);\n";
        }
        if (ar == Ar::F32)  // as a compensated FP32 partial: (acc, -cmp) = (h, l)
          o << "    " << accref(j) << " = q_.h; " << cmpref(j) << " = -q_.l; }\n";
        else
          o << "    " << accref(j) << " = q_; }\n";
      }
    };
    // `fresh` (double-float): the thread's first event, whose value is the partial
    auto acc_one = [&](std::ostringstream& o, const std::string& ind, int j, bool fresh = false) {
      {
        if (logadd[j] >= 0) o << ind << "lpc" << j << "++;\n";
        if (ar == Ar::F32 && logprod[j] >= 0) {
          o << ind << "mf_dw_logprod(lpm" << j << ", lpe" << j << ", we" << logprod[j] << ");\n";
          return;
        }
        const std::string r = eref(accnode[j]);
        if (ar == Ar::F32 || ar == Ar::F32S)
          o << ind << "mf_kahan_f32(" << accref(j) << ", " << cmpref(j) << ", " << r << ");\n";
        else if (ar == Ar::F64)
          o << ind << accref(j) << " += " << r << ";\n";
        else if (logprod[j] >= 0)
          o << ind << "mf_dw_logprod(lpm" << j << ", lpe" << j << ", " << eref(logprod[j]) << ");\n";
        else if (fresh)
          o << ind << accref(j) << " = "
            << (fused[j].first >= 0 ? "mf_dw_prod(" + eref(fused[j].first) + ", " + eref(fused[j].second) + ")" : r)
            << ";\n";
        else if (fused[j].first >= 0)
          o << ind << "mf_dw_acc_mul(" << accref(j) << ", " << eref(fused[j].first) << ", "
            << eref(fused[j].second) << ");\n";
        else
          o << ind << "mf_dw_acc(" << accref(j) << ", " << r << ");\n";
      }
    };
    auto acc_add = [&](std::ostringstream& o, const std::string& ind) {
      for (int j = 0; j < M; j++) acc_one(o, ind, j);
    };
    // Kernels with many outputs (Hessians) accumulate each output as soon as
    // the values it needs exist, instead of after the whole body: the outputs'
    // values then need not all be live at once (105 for the S+P-wave Hessian,
    // two registers each in double-float). Same operations in the same order
    // per output, so the same sums.
    const bool interleave = M > 16;
    std::vector<std::vector<int>> ready_after(ns.size() + 1);  // [ns.size()]: before the first statement
    if (interleave) {
      auto in_body = [&](int id) { return id >= 0 && live[id] && !ns[id].uniform && ns[id].op != Op::Input; };
      for (int j = 0; j < M; j++) {
        std::vector<int> deps{accnode[j]};
        if (ar == Ar::F32 && logprod[j] >= 0)
          deps = {logprod[j]};
        else if (ar == Ar::DW && logprod[j] >= 0)
          deps = {logprod[j]};
        else if (ar == Ar::DW && fused[j].first >= 0)
          deps = {fused[j].first, fused[j].second};
        int at = -1;
        for (int d : deps)
          if (in_body(d)) at = std::max(at, d);
        ready_after[at < 0 ? ns.size() : size_t(at)].push_back(j);
      }
    }
    // The body and the accumulation of every output; `guard` (a condition, or
    // empty) decides whether this event counts.
    auto body_acc = [&](std::ostringstream& o, const std::string& ind, const std::string& guard, bool fresh = false) {
      if (has_addu) o << ind << (guard.empty() ? "" : "if (" + guard + ") ") << "mf_cnt++;\n";
      auto accs = [&](const std::vector<int>& js) {
        if (js.empty()) return;
        if (!guard.empty()) o << ind << "if (" << guard << ") {\n";
        for (int j : js) acc_one(o, guard.empty() ? ind : ind + "  ", j, fresh);
        if (!guard.empty()) o << ind << "}\n";
      };
      if (!interleave) {
        body(o, ind);
        std::vector<int> all(M);
        for (int j = 0; j < M; j++) all[j] = j;
        accs(all);
        return;
      }
      accs(ready_after[ns.size()]);
      for (size_t i = 0; i < ns.size(); i++) {
        if (!live[i] || ns[i].uniform || ns[i].op == Op::Input) continue;
        const std::string st = estmt(int(i));
        if (!st.empty()) o << ind << st << "\n";
        accs(ready_after[i]);
      }
    };
    // A thread's partial of output j as a double-float value (expression).
    auto thread_dw = [&](int j) -> std::string {
      if (ar == Ar::F32 || ar == Ar::F32S) return "mf_two_sum(" + accref(j) + ", -" + cmpref(j) + ")";
      if (ar == Ar::F64) return "mf_dw_split(" + accref(j) + ")";
      return "mf_dw_renorm(" + accref(j) + ")";
    };
    // Block reduction of every output into mf_blk[] (shared). A warp sums N
    // outputs at once by a butterfly that halves the outputs a lane holds at
    // every step (mf_warp_sums: N - 1 exchanges instead of 5 N), outputs going
    // in chunks of 32, 16, 8, ... so that the fewest exchanges are made; then
    // one thread per output adds the warps in order. One barrier, where
    // staging eight outputs at a time through shared memory took two per
    // chunk and one warp's serial sum each: the P-wave Hessian's 36 outputs
    // were five such rounds, the S+P wave's 105 in blocks of two warps 53.
    // The order is fixed, so the result is reproducible.
    const std::vector<int> chunks = [&] {
      auto cost = [](int n) {  // exchanges of a chunk of n = 2^k outputs
        int k = 0;
        while ((1 << k) < n) k++;
        return n - 1 + 5 - k;
      };
      std::vector<int> best(M + 1, 0), pick(M + 1, 0);
      for (int r = 1; r <= M; r++)
        for (int n = 1; n <= 32; n *= 2) {
          const int c = cost(n) + best[std::max(0, r - n)];
          if (!pick[r] || c < best[r]) {
            best[r] = c;
            pick[r] = n;
          }
        }
      std::vector<int> v;
      for (int r = M; r > 0; r -= pick[r]) v.push_back(pick[r]);
      return v;
    }();
    // Partials in shared memory: nothing of a chunk is loaded before the one
    // before is done. ptxas otherwise loads all of them at once and spills, and
    // callers split a Hessian that spills. Of a density linear in p + 1 columns,
    // bytes a thread and one call at 1M events, without and with the barrier:
    // p = 15 (120 outputs) 376 / 0, 194 / 161 us; p = 16 992 / 0, 229 / 196;
    // p = 18 2144 / 568, 336 / 381; p = 20 2584 / 1304, 546 / 527. Up to 32
    // partials in registers there is no spill either way: the S+P wave's 105
    // outputs (25) take 71.5 / 76.3 us at 333333 events, 152 / 148 at 1M.
    auto warp_reduce = [&](std::ostringstream& o) {  // into row `warp` of part[]
      int j0 = 0;
      for (int n : chunks) {
        if (NREG < M && NREG > 32) o << "  asm volatile(\"\" ::: \"memory\");\n";
        o << "  {\n    mf_dw v[" << n << "];\n";
        for (int c = 0; c < n; c++)
          o << "    v[" << c << "] = " << (j0 + c < M ? thread_dw(j0 + c) : "mf_dw_make(0.0f, 0.0f)") << ";\n";
        o << "    mf_warp_sums<" << n << ">(v, lane);\n"
          << "    const int j = " << j0 << " + lane / " << 32 / n << ";\n"
          << "    if (lane % " << 32 / n << " == 0 && j < MF_NOUT) part[warp * MF_NOUT + j] = make_float2(v[0].h, v[0].l);\n"
          << "  }\n";
        j0 += n;
      }
    };
    // Up to eight outputs (256 threads) of FP32 kernels, a warp each: through
    // shared memory, so that a block does M warps' sums instead of M outputs'
    // butterflies in each of its eight warps (1370 instructions for 5 outputs,
    // 1070 so); batched gradients of 250k events, FP32 mass 2.23 -> 2.02 us an
    // evaluation, weighted 2.38 -> 2.18. Double-float kernels share the
    // butterfly's order with their _batch entry.
    const bool staged = (ar == Ar::F32 || ar == Ar::F32S) && M <= out.block / 32 && M * out.block <= 2048;  // 16 KB
    auto block_reduce = [&](std::ostringstream& o) {
      if (staged) {
        o << "  __shared__ float2 mf_stage[MF_NOUT][MF_BLOCK];\n"
          << "  __shared__ float2 mf_part[MF_PART];\n  __shared__ float2 mf_blk[MF_NOUT];\n"
          << "  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;\n";
        for (int j = 0; j < M; j++)
          o << "  { const mf_dw t = " << thread_dw(j) << "; mf_stage[" << j << "][threadIdx.x] = make_float2(t.h, t.l); }\n";
        o << "  __syncthreads();\n  if (warp < MF_NOUT) {\n    mf_dw t[MF_BLOCK / 32];\n"
          << "#pragma unroll\n    for (int k = 0; k < MF_BLOCK / 32; k++) t[k] = mf_dw_pair(mf_stage[warp][lane + 32 * k]);\n"
          << "    mf_tree_sum(t);\n"
          << "#pragma unroll\n    for (int o = 16; o > 0; o >>= 1) t[0] = mf_dw_add(t[0], mf_dw_shfl_xor(t[0], o));\n"
          << "    if (lane == 0) mf_blk[warp] = make_float2(t[0].h, t[0].l);\n  }\n  __syncthreads();\n";
        return;
      }
      o << "  __shared__ float2 mf_part[MF_PART];\n  __shared__ float2 mf_blk[MF_NOUT];\n"
        << "  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;\n  float2* const part = mf_part;\n";
      warp_reduce(o);
      o << "  __syncthreads();\n"
        << "  for (int j = threadIdx.x; j < MF_NOUT; j += MF_BLOCK) {\n"
        << "    const mf_dw a = mf_sum_warps(mf_part + j);\n"
        << "    mf_blk[j] = make_float2(a.h, a.l);\n  }\n  __syncthreads();\n";
    };
    bool f32_logprod = false;
    for (int j = 0; j < M; j++) f32_logprod = f32_logprod || (ar == Ar::F32 && logprod[j] >= 0);
    auto load_table = [&](std::ostringstream& o) {
      if (f32_logprod) {
        o << "  __shared__ float4 mf_logtab[128];\n"
          << "  for (int q = threadIdx.x; q < 128; q += MF_BLOCK) mf_logtab[q] = mf_dw_logtab_g[q];\n"
          << "  __syncthreads();\n";
        return;
      }
      if (ar != Ar::DW || (!has_log && !has_exp)) return;
      if (has_log)
        o << "  __shared__ float4 mf_logtab[128];\n"
          << "  for (int q = threadIdx.x; q < 128; q += MF_BLOCK) mf_logtab[q] = mf_dw_logtab_g[q];\n";
      if (has_exp)
        o << "  __shared__ float2 mf_exptab[64];\n"
          << "  for (int q = threadIdx.x; q < 64; q += MF_BLOCK) mf_exptab[q] = mf_dw_exptab_g[q];\n";
      o << "  __syncthreads();\n";
    };
    auto input_value = [&](const std::string& raw) {
      if (ar == Ar::DW) return (pair ? "mf_dw_pair(" : "mf_dw_split(") + raw + ")";
      return raw;
    };
    const std::string DT = pair ? "float2" : ST;  // element type the REDUCE entries read
    const std::string XT = ar == Ar::F32 ? "float" : (ar == Ar::F64 || ar == Ar::F32S) ? "double" : "mf_dw";

    s << "__device__ __forceinline__ void mf_prefetch_l2(const void* p) {\n"
      << "  asm volatile(\"prefetch.global.L2 [%0];\" ::\"l\"(p));\n}\n";
    s << "struct mf_args { double d[" << out.nd << "]; float f[" << out.nf << "]; };\n";
    s << kCombine;
    const int NC = int(out.used_inputs.size());
    const std::string VT = V == 1 ? DT : pair ? "float4" : st32 ? (V == 4 ? "float4" : "float2") : "double2";
    auto load_at = [&](int k, const std::string& at) {
      return "__ldg(reinterpret_cast<const " + VT + "*>(data + (mf_u64)" + std::to_string(k) + " * stride + " + at + "))";
    };
    const char* comp[4] = {"x", "y", "z", "w"};
    // event v of the vector loaded into l<k>
    auto lane_of = [&](int k, int v) -> std::string {
      const std::string l = "l" + std::to_string(k);
      if (pair) return V == 1 ? l : "make_float2(" + l + "." + comp[2 * v] + ", " + l + "." + comp[2 * v + 1] + ")";
      return V == 1 ? l : l + "." + comp[v];
    };
    // the vector's events (loaded here from src(k), or l<k> defined already)
    auto emit_events = [&](std::ostringstream& s, const std::string& ind, const std::string& valid_base,
                           const std::function<std::string(int)>& src, bool fresh = false) {
      for (int k : out.used_inputs)
        if (src) s << ind << "const " << VT << " l" << k << " = " << src(k) << ";\n";
      for (int v = 0; v < V; v++) {
        s << ind << "{\n";
        for (int k : out.used_inputs)
          s << ind << "  const " << XT << " x" << k << " = " << input_value(lane_of(k, v)) << ";\n";
        body_acc(s, ind + "  ", valid_base + " + " + std::to_string(v) + " < n", fresh && v == 0);
        s << ind << "}\n";
      }
    };
    // y = one event's value of a prepared column, from the columns src(k) it folds
    auto emit_fold = [&](std::ostringstream& s, const std::string& ind, const std::string& y, const auto& terms,
                         const std::function<std::string(int)>& src) {
      s << ind << "double " << y << " = " << src(terms[0].first) << ";\n";
      for (size_t t = 1; t < terms.size(); t++) {
        const double c = terms[t].second;
        if (c == 1.0)
          s << ind << y << " = __dadd_rn(" << y << ", " << src(terms[t].first) << ");\n";
        else if (c == -1.0)
          s << ind << y << " = __dsub_rn(" << y << ", " << src(terms[t].first) << ");\n";
        else
          s << ind << y << " = __fma_rn(" << fmt_const(c, false) << ", " << src(terms[t].first) << ", " << y << ");\n";
      }
    };
    // The per-block work of the single-evaluation and the batched entry: the
    // event loop and the block reduction. `prefetch`: a thread's next events
    // are loaded while it computes its present ones, the first before the
    // tables (the same events in the same order, so the same sums).
    // `first`: the dataset's columns, unprepared: every vector of them is
    // prepared here as the _prep entry does and stored for later evaluations.
    auto block_work = [&](std::ostringstream& s, const bool prefetch, const bool first = false) {
      if (!first)
        s << "  mf_launch_dependents();  // the next evaluation may start its event loop on SMs this grid frees\n";
      std::set<int> raw_cols;
      const std::string RT = V == 1 ? "double" : "double2";
      auto raw_at = [&](int k, const std::string& at) {
        return "__ldg(reinterpret_cast<const " + RT + "*>(raw + (mf_u64)" + std::to_string(k) + " * stride + " + at + "))";
      };
      if (first) {
        for (const auto& terms : fold.cols)
          for (const auto& t : terms) raw_cols.insert(t.first);
        s << "  const mf_u64 step = (mf_u64)gridDim.x * MF_BLOCK * " << V << ";\n"
          << "  mf_u64 base = ((mf_u64)blockIdx.x * MF_BLOCK + threadIdx.x) * " << V << ";\n";
        for (int k : raw_cols)
          s << "  " << RT << " c" << k << " = base < stride ? " << raw_at(k, "base") << " : " << RT << "();\n";
      } else if (prefetch) {
        s << "  const mf_u64 step = (mf_u64)gridDim.x * MF_BLOCK * " << V << ";\n"
          << "  mf_u64 base = ((mf_u64)blockIdx.x * MF_BLOCK + threadIdx.x) * " << V << ";\n";
        for (int k : out.used_inputs)
          s << "  " << VT << " c" << k << " = base < n ? " << load_at(k, "base") << " : " << VT << "();\n";
      }
      load_table(s);
      prologue(s, "P.");
      acc_decl(s);
      if (out.pipelined && NC > 0) {
        // Persistent blocks; tile t (events [t*MF_TILE, (t+1)*MF_TILE) of every
        // column read by the body) goes to block t % gridDim.x. Thread 0 keeps
        // MF_STAGES - 1 tiles in flight with bulk asynchronous copies into a
        // ring of shared-memory stages; all threads wait on the stage's
        // mbarrier (bounded), compute from shared memory and release the stage.
        const size_t es = st32 ? 4 : 8;  // float pairs are 8 bytes too
        out.smem_bytes = size_t(out.stages) * NC * out.tile * es;
        s << "#define MF_TILE " << out.tile << "\n#define MF_STAGES " << out.stages << "\n#define MF_NC " << NC << "\n";
        s << "  extern __shared__ __align__(128) unsigned char mf_dyn[];\n";
        s << "  " << DT << "* __restrict__ stage = reinterpret_cast<" << DT << "*>(mf_dyn);\n";
        s << "  __shared__ __align__(8) unsigned long long mf_bar[MF_STAGES];\n";
        s << "  const mf_u64 ntiles = (n + MF_TILE - 1) / MF_TILE;\n";
        s << "  if (threadIdx.x == 0) {\n    for (int q = 0; q < MF_STAGES; q++) mf_mbar_init(&mf_bar[q], 1u);\n"
          << "    mf_fence_mbar_init();\n  }\n  __syncthreads();\n";
        // issue lambda as a macro-like block
        std::ostringstream issue;
        issue << "{ const mf_u64 t0 = (TL) * (mf_u64)MF_TILE; mf_u64 cnt = stride - t0; if (cnt > MF_TILE) cnt = MF_TILE;\n"
              << "          const unsigned bytes = (unsigned)(cnt * sizeof(" << DT << "));\n"
              << "          mf_mbar_expect_tx(&mf_bar[SL], bytes * MF_NC);\n";
        for (int ci = 0; ci < NC; ci++)
          issue << "          mf_bulk_g2s(stage + ((mf_u64)(SL) * MF_NC + " << ci << ") * MF_TILE, data + (mf_u64)"
                << out.used_inputs[ci] << " * stride + t0, bytes, &mf_bar[SL]);\n";
        issue << "        }";
        auto issue_code = [&](const std::string& tl, const std::string& sl) {
          std::string c = issue.str();
          for (size_t p; (p = c.find("(TL)")) != std::string::npos;) c.replace(p, 4, "(" + tl + ")");
          for (size_t p; (p = c.find("SL")) != std::string::npos;) c.replace(p, 2, sl);
          return c;
        };
        s << "  unsigned issued = 0;  // tiles issued by thread 0 (valid in thread 0)\n";
        s << "  if (threadIdx.x == 0)\n    for (int q = 0; q < MF_STAGES - 1; q++) {\n"
          << "      const mf_u64 tl = blockIdx.x + (mf_u64)q * gridDim.x;\n      if (tl < ntiles) {\n        "
          << issue_code("tl", "q") << "\n        issued++;\n      }\n    }\n";
        s << "  unsigned it = 0;\n  bool aborted = false;\n";
        s << "  for (mf_u64 tile = blockIdx.x; tile < ntiles; tile += gridDim.x, it++) {\n";
        s << "    const unsigned sl = it % MF_STAGES, par = (it / MF_STAGES) & 1u;\n";
        s << "    if (threadIdx.x == 0) {\n      const mf_u64 nt = tile + (mf_u64)(MF_STAGES - 1) * gridDim.x;\n"
          << "      if (nt < ntiles) {\n        const unsigned ns = (it + MF_STAGES - 1) % MF_STAGES;\n"
          << "        mf_fence_proxy_async();\n        " << issue_code("nt", "ns") << "\n        issued++;\n      }\n    }\n";
        s << "    const bool ok = mf_mbar_wait_bounded(&mf_bar[sl], par);\n";
        s << "    if (__syncthreads_or(!ok)) { aborted = true; break; }\n";
        s << "    const " << DT << "* __restrict__ sb = stage + (mf_u64)sl * MF_NC * MF_TILE;\n";
        s << "    const mf_u64 tbase = tile * (mf_u64)MF_TILE;\n";
        s << "    {\n      const int e0 = threadIdx.x * " << V << ";\n";
        std::map<int, int> colpos;
        for (int ci = 0; ci < NC; ci++) colpos[out.used_inputs[ci]] = ci;
        emit_events(s, "      ", "tbase + e0", [&](int k) {
          return "*reinterpret_cast<const " + VT + "*>(sb + " + std::to_string(colpos[k]) + " * MF_TILE + e0)";
        });
        s << "    }\n    __syncthreads();\n  }\n";
        // abort: report, drain this block's copies still in flight (bounded), continue to the reduction
        s << "  if (aborted && threadIdx.x == 0) {\n    atomicOr(status, 1u);\n"
          << "    for (unsigned k = it; k < issued; k++) mf_mbar_wait_bounded(&mf_bar[k % MF_STAGES], (k / MF_STAGES) & 1u);\n"
          << "  }\n";
      } else if (first) {
        s << "  for (; base < stride; base += step) {\n    const mf_u64 ahead = base + step;\n";
        for (int k : raw_cols)
          s << "    const " << RT << " s" << k << " = c" << k << ";\n    c" << k << " = ahead < stride ? "
            << raw_at(k, "ahead") << " : " << RT << "();\n";
        for (size_t m = 0; m < fold.cols.size(); m++) {
          s << "    " << VT << " l" << m << ";\n    {\n";
          for (int v = 0; v < V; v++) {
            const std::string y = "y" + std::to_string(v), w = "w" + std::to_string(v);
            emit_fold(s, "      ", y, fold.cols[m],
                      [&](int k) { return "s" + std::to_string(k) + (V == 1 ? "" : v == 0 ? ".x" : ".y"); });
            s << "      const mf_dw " << w << " = mf_dw_split(" << y << ");\n";
          }
          s << "      l" << m << " = "
            << (V == 1 ? "make_float2(w0.h, w0.l)" : "make_float4(w0.h, w0.l, w1.h, w1.l)") << ";\n    }\n"
            << "    *reinterpret_cast<" << VT << "*>(prepared + (mf_u64)" << m << " * stride + base) = l" << m << ";\n";
        }
        s << "    if (base < n) {\n";
        emit_events(s, "      ", "base", nullptr);
        s << "    }\n  }\n";
      } else if (prefetch) {
        if (out.stages > 1) s << "#pragma unroll " << out.stages << "\n";
        s << "  for (; base < n; base += step) {\n    const mf_u64 ahead = base + step;\n";
        for (int k : out.used_inputs) s << "    const " << VT << " l" << k << " = c" << k << ";\n";
        for (int k : out.used_inputs)
          s << "    c" << k << " = ahead < n ? " << load_at(k, "ahead") << " : " << VT << "();\n";
        if (M > 16) {  // the events after those on their way into L2
          s << "    if (ahead + step < n) {\n";
          for (int k : out.used_inputs)
            s << "      mf_prefetch_l2(data + (mf_u64)" << k << " * stride + ahead + step);\n";
          s << "    }\n";
        }
        emit_events(s, "    ", "base", nullptr);
        s << "  }\n";
      } else {
        s << "  const mf_u64 step = (mf_u64)gridDim.x * MF_BLOCK * " << V << ";\n";
        // unrolled: the next iteration's loads are issued before this one's arithmetic
        if (out.stages > 1) s << "#pragma unroll " << out.stages << "\n";
        s << "  for (mf_u64 base = ((mf_u64)blockIdx.x * MF_BLOCK + threadIdx.x) * " << V
          << "; base < n; base += step) {\n";
        emit_events(s, "    ", "base", [&](int k) { return load_at(k, "base"); });
        s << "  }\n";
      }
      s << "  __shared__ bool am_last;\n";
      acc_finish(s);
      block_reduce(s);
    };
    // Prefetching pays where one launch must hide its own latency (a lone
    // evaluation: the P-wave Hessian's eight warps per SM keep 18 KB of loads
    // in flight without it, which is 2.8 TB/s) and the next events fit in
    // registers beside the accumulators at the same blocks per SM. Lone calls,
    // 1M events, without and with: P wave gradient 30.4 / 27.3 us, value 26.5
    // / 25.9, Hessian 54.8 / 45.5, S+P gradient 52.6 / 45.6, value 33.8 /
    // 32.4; the S+P Hessian spills. FP32 kernels keep the plain loop: they are
    // nearer the copy rate (S+P gradient, 3M: 44.4 us without, 50.1 with), and
    // which of their products the compiler fuses into a sum, and so their last
    // bit, follows the loop's form. Batched evaluations overlap their
    // neighbours instead and keep the registers (P-wave gradient, 64 points of
    // 100k events: 175 without, 190 with).
    // Of more than 16 outputs (one event per thread and turn, eight warps per
    // SM) a turn is still shorter than a loaded memory's latency: the events
    // after the next are asked for in L2 (P-wave Hessian, 1M events 45.3 ->
    // 42.4 us, 3M 100 -> 93.8; a ring of three turns in shared memory, 42.7;
    // the gradients, 16 warps per SM and more, lose 3 us by either).
    //
    // "Fits" is two vectors of the columns, the partials, and 30 registers for
    // the body (60 for Hessians, one event per turn) within 40 of the registers
    // of a thread, 65536 over the block or 255: some spilled events cost less
    // than the waits. Lone calls of 1M events, plain and prefetching (estimate
    // at 256 threads): values of 31 columns 74 / 66 us (280), of 37 60 / 97
    // (328), of 48 74 / 142 (416), of 64 134 / 1052 (544: 13 KB of spill);
    // first evaluations of 31 columns 152 / 131, of 48 197 / 1506. The P-wave
    // Hessian in blocks of 512 (168) spills 384 bytes, none with the plain loop.
    auto fits = [&](int columns, int events) {
      return 4 * columns * events + 2 * M + (events == 1 ? 60 : 30) < std::min(256, 65536 / out.block / 8 * 8) + 40;
    };
    const bool lone_prefetch = !out.pipelined && NC > 0 && ar == Ar::DW && M <= kAccRegMax && fits(NC, V);
    auto replace_all = [](std::string& t, const std::string& from, const std::string& to) {
      for (size_t p = t.find(from); p != std::string::npos; p = t.find(from, p + to.size())) t.replace(p, from.size(), to);
    };
    std::ostringstream lone_work, part_work;
    block_work(lone_work, lone_prefetch);
    block_work(part_work, false);
    const auto entry_mark = s.tellp();
    // ---- single-dataset reduce ----
    s << "extern \"C\" __global__ void MF_BOUNDS " << out.entry << "(const " << DT
      << "* __restrict__ data, mf_u64 stride, mf_u64 n, mf_args P, float2* __restrict__ partials,"
      << " unsigned* __restrict__ counter, double* __restrict__ out, unsigned* __restrict__ status, unsigned seq) {\n";
    const auto body_mark = s.tellp();
    s << lone_work.str();
    s << R"CUDA(  // Launched as a programmatic dependent of the previous evaluation on the
  // stream (batched evaluations), this grid ran its event loop while that
  // one finished; the scratch below is shared, so wait for it to complete.
  mf_grid_dependency_wait();
  // Completion counts with release/acquire semantics: the barrier orders the
  // block's row before thread 0's release; the last block's acquire plus the
  // barrier orders its reads of every row after. A grid of one block has
  // nothing to combine.
  if (gridDim.x > 1u) {
    for (int j = threadIdx.x; j < MF_NOUT; j += MF_BLOCK) partials[(mf_u64)blockIdx.x * MF_NOUT + j] = mf_blk[j];
    __syncthreads();
#if MF_ROWS > 0
    const unsigned mf_g = blockIdx.x / MF_ROWS, mf_first = mf_g * MF_ROWS;
    const unsigned mf_nr = gridDim.x - mf_first < MF_ROWS ? gridDim.x - mf_first : MF_ROWS;
    if (threadIdx.x == 0) am_last = (mf_atom_add_acq_rel(counter + 1 + mf_g, 1u) == mf_nr - 1);
    __syncthreads();
    if (!am_last) return;
    mf_sum_rows(partials + (mf_u64)mf_first * MF_NOUT, mf_nr, 1u, mf_part, mf_blk);
    for (int j = threadIdx.x; j < MF_NOUT; j += MF_BLOCK) partials[(mf_u64)mf_first * MF_NOUT + j] = mf_blk[j];
    if (threadIdx.x == 0) counter[1 + mf_g] = 0u;
    __syncthreads();
    const unsigned mf_nb = (gridDim.x + MF_ROWS - 1) / MF_ROWS, mf_step = MF_ROWS;
#else
    const unsigned mf_nb = gridDim.x, mf_step = 1u;
#endif
    if (threadIdx.x == 0) am_last = (mf_atom_add_acq_rel(counter, 1u) == mf_nb - 1);
    __syncthreads();
    if (!am_last) return;
    mf_sum_rows(partials, mf_nb, mf_step, mf_part, mf_blk);
    if (threadIdx.x == 0) *counter = 0u;
  }
  for (int j = threadIdx.x; j < MF_NOUT; j += MF_BLOCK) out[j] = mf_dw_to_double(mf_dw_pair(mf_blk[j]));
  // Synchronous evaluation (seq != 0): out[] is mapped host memory; publish
  // completion in the mapped word status[1] after every output is visible
  // system-wide, so the host can read the sums without a stream synchronize.
  if (seq != 0u) {
    __threadfence_system();
    __syncthreads();
    if (threadIdx.x == 0) *reinterpret_cast<volatile unsigned*>(status + 1) = seq;
  }
)CUDA";
    const std::string lone_tail = s.str().substr(size_t(body_mark) + lone_work.str().size());
    if (!out.pipelined) {
      auto resident = [&](std::string work) {
        replace_all(work, "blockIdx.x", "mf_vb");
        replace_all(work, "gridDim.x", "mf_grid");
        return "__device__ __forceinline__ void mf_rbody(const " + DT +
               "* __restrict__ data, mf_u64 stride, mf_u64 n, const mf_args& P, float2* __restrict__ "
               "partials, unsigned* __restrict__ counter, double* __restrict__ out, unsigned* "
               "__restrict__ status, unsigned seq, unsigned mf_vb, unsigned mf_grid) {\n" +
               work + "}\n";
      };
      out.resident_prefix = s.str().substr(0, size_t(entry_mark));
      out.resident_data_type = DT;
      out.resident_body = resident(lone_work.str() + lone_tail);
      out.resident_plain = resident(part_work.str() + lone_tail);
    }
    s << "}\n";
    // ---- the first evaluation of a dataset ----
    // Preparing the columns in a pass of its own writes them only for the
    // event loop to read them again. This entry is the event loop over the
    // columns as they are: each thread prepares the events it evaluates (the
    // padding up to `stride` as well) and stores them for the evaluations to
    // come. The same events, operations and grid as the entry above, so the
    // same sums bit for bit. Bound by the columns' bytes and by latency at 16
    // warps per SM: for 1M K*mumu P-wave events (88 MB read, 72 MB written)
    // the pass and the gradient took 20.2 + 18.4 us (ncu), this entry 32.4
    // with the next columns' loads in flight and 36 without; a new dataset
    // with its precompute and first gradient 111.5 -> 98.9 us. For
    // gradient-sized kernels; Hessians are issue-bound and seldom first.
    // Only where the columns as they are, two vectors of them beside one of the
    // prepared ones, fit as above.
    std::set<int> raw_columns;
    for (const auto& terms : fold.cols)
      for (const auto& t : terms) raw_columns.insert(t.first);
    out.first = prep && pair && ar == Ar::DW && !st32 && !out.pipelined && NC > 0 && M <= 16 &&
                fits(std::max(NC, int(raw_columns.size())), V);
    if (out.first) {
      std::ostringstream first_work;
      block_work(first_work, false, true);
      s << "extern \"C\" __global__ void MF_BOUNDS " << out.entry
        << "_first(const double* __restrict__ raw, mf_u64 stride, mf_u64 n, mf_args P, float2* __restrict__ partials,"
        << " unsigned* __restrict__ counter, double* __restrict__ out, unsigned* __restrict__ status, unsigned seq, "
        << DT << "* __restrict__ prepared) {\n"
        << first_work.str() << lone_tail << "}\n";
    }
    // ---- batched evaluations: per-block partials only, then one combine ----
    // Evaluation e of a batch writes its partial rows to its own slot of the
    // batch's partial buffer without counting or combining, so consecutive
    // evaluations' grids overlap (each waits for its predecessor only after
    // its own work); <entry>_combine then reduces every evaluation's rows
    // (one block each, the same fixed order: the sums equal the
    // single-evaluation entry's).
    //
    // Consecutive grids of two blocks per SM overlap in the slot of a third
    // where the registers leave one: asked for (80 registers) where one
    // vector of the columns and the partials take at most 56, which costs the
    // P-wave gradient 12 bytes of spill. Datasets in turn from HBM, 1M events:
    // 13.2 us an evaluation at the 86 registers it takes of itself, 11.0 at
    // 80. The S+P wave (16 columns) would spill its events.
    // Kernels of one column take fewer than 80 of themselves, and the bound raises
    // them (mass value 48 -> 56, gradient 48 -> 64): a block per SM less.
    const bool three = ar == Ar::DW && out.block == 256 && NC > 1 && 2 * (NC * V + M) <= 56;
    s << "extern \"C\" __global__ void " << (three ? "__launch_bounds__(MF_BLOCK, 3) " : "MF_BOUNDS ") << out.entry
      << "_part(const " << DT
      << "* __restrict__ data, mf_u64 stride, mf_u64 n, mf_args P, float2* __restrict__ partials,"
      << " unsigned* __restrict__ status) {\n"
      << part_work.str()
      << "  for (int j = threadIdx.x; j < MF_NOUT; j += MF_BLOCK) partials[(mf_u64)blockIdx.x * MF_NOUT + j] = mf_blk[j];\n"
      << "  // complete only after the previous evaluation's grid: completions stay in\n"
      << "  // stream order, so the combine launch after the last evaluation sees every partial\n"
      << "  mf_grid_dependency_wait();\n"
      << "}\n";
    // ---- many small evaluations in one launch ----
    // For evaluations of less than one grid of the device, where a thread has
    // one vector of events at most and a launch each costs the host more than
    // the device: block (vb, q) does block vb of evaluations [q * group, ...)
    // of the launch, one after the other, its events kept in registers while
    // they stay the same (a scan of one dataset), one table load and one
    // barrier for all. Each row of partials is the _part entry's, and
    // <entry>_combine follows the same way. The evaluations' columns, sizes
    // and parameters are the launch's own argument (constant memory).
    // Double-float kernels only: their operations are fixed one by one, an
    // FP32 body's last bit follows the form of the loop around it.
    if (!out.pipelined && NC > 0 && ar == Ar::DW && M <= 16) {
      out.batch_max = int(std::min<size_t>(64, 24576 / (32 + out.args_bytes())));
      s << "#define MF_GROUP " << kBatchGroup << "\n"
        << "struct mf_job { const " << DT << "* data; mf_u64 stride, n, grid; mf_args P; };\n"
        << "struct mf_batch { mf_job job[" << out.batch_max << "]; };\n"
        << "extern \"C\" __global__ void MF_BOUNDS " << out.entry
        << "_batch(const __grid_constant__ mf_batch B, float2* __restrict__ partials_all, mf_u64 pstride,"
        << " unsigned count, unsigned group) {\n"
        << "  __shared__ float2 mf_warps[MF_GROUP][MF_BLOCK / 32 * MF_NOUT];\n"
        << "  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;\n"
        << "  const unsigned first = blockIdx.y * group, last = first + group < count ? first + group : count;\n"
        << "  const mf_u64 base = ((mf_u64)blockIdx.x * MF_BLOCK + threadIdx.x) * " << V << ";\n"
        << "  const " << DT << "* __restrict__ data = B.job[first].data;\n"
        << "  mf_u64 stride = B.job[first].stride, n = B.job[first].n;\n";
      for (int k : out.used_inputs)
        s << "  " << VT << " l" << k << " = base < n ? " << load_at(k, "base") << " : " << VT << "();\n";
      load_table(s);
      s << "  for (unsigned e = first; e < last; e++) {\n    const mf_job& J = B.job[e];\n"
        << "    if (blockIdx.x >= J.grid) continue;\n    const mf_args& P = J.P;\n"
        << "    if (J.data != data || J.stride != stride || J.n != n) {  // another dataset\n"
        << "      data = J.data; stride = J.stride; n = J.n;\n";
      for (int k : out.used_inputs)
        s << "      l" << k << " = base < n ? " << load_at(k, "base") << " : " << VT << "();\n";
      s << "    }\n    float2* const part = mf_warps[e - first];\n";
      prologue(s, "P.");
      acc_decl(s);
      s << "    if (base < n) {\n";
      emit_events(s, "      ", "base", nullptr, true);
      s << "    }\n";
      acc_finish(s);
      warp_reduce(s);
      s << R"CUDA(  }
  __syncthreads();
  for (unsigned q = threadIdx.x; q < (last - first) * MF_NOUT; q += MF_BLOCK) {
    const unsigned e = q / MF_NOUT, j = q - e * MF_NOUT;
    if (blockIdx.x >= B.job[first + e].grid) continue;
    const mf_dw a = mf_sum_warps(mf_warps[e] + j);
    partials_all[(first + e) * pstride + (mf_u64)blockIdx.x * MF_NOUT + j] = make_float2(a.h, a.l);
  }
}
)CUDA";
    }
    s << "extern \"C\" __global__ void __launch_bounds__(MF_BLOCK) " << out.entry
      << "_combine(float2* __restrict__ partials_all, mf_u64 pstride, const unsigned* __restrict__ grids,"
      << " double* __restrict__ out_all, unsigned count, unsigned grid_all) {\n"
      << "  // launched as a programmatic dependent of the last evaluation: its partials\n"
      << "  // (and every earlier one's) are complete and visible after this\n"
      << "  mf_grid_dependency_wait();\n"
      << "  const unsigned e = blockIdx.x;\n  if (e >= count) return;\n"
      << "  // every evaluation's grid size, or (grids null) the one they all share\n"
      << "  const unsigned mf_nb = grids ? grids[e] : grid_all;\n"
      << "  float2* __restrict__ partials = partials_all + (mf_u64)e * pstride;\n"
      << "  double* __restrict__ out = out_all + (mf_u64)e * MF_NOUT;\n"
      << R"CUDA(  __shared__ float2 mf_part[MF_PART];
  __shared__ float2 mf_blk[MF_NOUT];
  unsigned mf_rows = mf_nb, mf_step = 1u;
#if MF_ROWS > 0
  if (mf_nb > 1u) {  // the single-evaluation entry's groups first
    for (unsigned f = 0; f < mf_nb; f += MF_ROWS) {
      mf_sum_rows(partials + (mf_u64)f * MF_NOUT, mf_nb - f < MF_ROWS ? mf_nb - f : MF_ROWS, 1u, mf_part, mf_blk);
      for (int j = threadIdx.x; j < MF_NOUT; j += MF_BLOCK) partials[(mf_u64)f * MF_NOUT + j] = mf_blk[j];
      __syncthreads();
    }
    mf_rows = (mf_nb + MF_ROWS - 1) / MF_ROWS;
    mf_step = MF_ROWS;
  }
#endif
  mf_sum_rows(partials, mf_rows, mf_step, mf_part, mf_blk);
  for (int j = threadIdx.x; j < MF_NOUT; j += MF_BLOCK) out[j] = mf_dw_to_double(mf_dw_pair(mf_blk[j]));
}
)CUDA";

    // Event loop and block reduction of a block that owns events [first,
    // first + cnt) of its columns, its parameters in `P`: one event per thread
    // and round, the next round's event loaded while this one is computed (the
    // first before the tables): a block is alone with its segment and its few
    // warps hide little latency. Toys of 2000 P-wave events, one call, plain
    // and so: value of 1 toy 52 / 37 us, of 1000 144 / 112, of 4096 388 / 315;
    // F, gradient and Hessian of 1000 toys 311 / 304. Kernels whose partials
    // fill the registers (more than kAccRegMax outputs) and FP32 ones keep the
    // plain loop, and those whose events do not fit (see lone_prefetch).
    const bool seg_prefetch = ar == Ar::DW && M <= kAccRegMax && fits(NC, 1);
    auto segment_work = [&](std::ostringstream& o) {
      auto load_event = [&](int k, const std::string& at) {
        return "__ldg(data + (mf_u64)" + std::to_string(k) + " * stride + first + " + at + ")";
      };
      if (seg_prefetch)
        for (int k : out.used_inputs)
          o << "  " << DT << " c" << k << " = threadIdx.x < cnt ? " << load_event(k, "threadIdx.x") << " : " << DT
            << "();\n";
      load_table(o);
      prologue(o, "P.");
      acc_decl(o);
      // from the last turn to cnt itself: i + MF_BLOCK would wrap for counts
      // near 2^32, and the loop not end
      o << "  for (unsigned i = threadIdx.x; i < cnt; i = cnt - i > MF_BLOCK ? i + MF_BLOCK : cnt) {\n";
      if (seg_prefetch) {
        for (int k : out.used_inputs) o << "    const " << DT << " l" << k << " = c" << k << ";\n";
        o << "    const bool more = cnt - i > MF_BLOCK;\n";
        for (int k : out.used_inputs)
          o << "    c" << k << " = more ? " << load_event(k, "(i + MF_BLOCK)") << " : " << DT << "();\n";
      }
      for (int k : out.used_inputs)
        o << "    const " << XT << " x" << k << " = "
          << input_value(seg_prefetch ? "l" + std::to_string(k) : load_event(k, "i")) << ";\n";
      body_acc(o, "    ", "");
      o << "  }\n";
      acc_finish(o);
      block_reduce(o);
    };
    // ---- ragged segments: one block per segment ----
    s << "extern \"C\" __global__ void __launch_bounds__(MF_BLOCK) " << out.entry << "_segments(const " << DT
      << "* __restrict__ data, mf_u64 stride, const mf_u64* __restrict__ seg_begin,"
      << " const unsigned* __restrict__ seg_count, const mf_args* __restrict__ args,"
      << " double* __restrict__ out) {\n";
    s << "  const unsigned seg = blockIdx.x;\n  const mf_u64 first = seg_begin[seg];\n"
      << "  const unsigned cnt = seg_count[seg];\n  const mf_args& P = args[seg];\n";
    segment_work(s);
    s << R"CUDA(  for (int j = threadIdx.x; j < MF_NOUT; j += MF_BLOCK)
    out[(mf_u64)seg * MF_NOUT + j] = mf_dw_to_double(mf_dw_make(mf_blk[j].x, mf_blk[j].y));
}
)CUDA";
    // ---- many datasets in one launch: one block per segment ----
    // A segment is a run of at most MF_MULTI_CHUNK events of one dataset
    // (its own columns, stride and parameter row); the block writes its
    // partial row to `row` of the partial buffer, and <entry>_combine then
    // reduces each dataset's rows in a fixed order. A dataset's sums depend
    // only on its own events, parameters and size (segments are cut at fixed
    // multiples of MF_MULTI_CHUNK), never on what else shares the launch.
    s << "struct mf_seg { const void* data; mf_u64 stride; mf_u64 first; unsigned count; unsigned req; unsigned row;"
         " unsigned pad; };\n";
    s << "extern \"C\" __global__ void __launch_bounds__(MF_BLOCK) " << out.entry
      << "_multi(const mf_seg* __restrict__ segs, const mf_args* __restrict__ args,"
      << " float2* __restrict__ partials) {\n";
    s << "  const mf_seg S = segs[blockIdx.x];\n"
      << "  const " << DT << "* __restrict__ data = static_cast<const " << DT << "*>(S.data);\n"
      << "  const mf_u64 stride = S.stride, first = S.first;\n  const unsigned cnt = S.count;\n"
      << "  const mf_args& P = args[S.req];\n";
    segment_work(s);
    s << R"CUDA(  for (int j = threadIdx.x; j < MF_NOUT; j += MF_BLOCK) partials[(mf_u64)S.row * MF_NOUT + j] = mf_blk[j];
}
)CUDA";
    // ---- per-dataset preparation of the columns the entries above read ----
    if (prep) {
      const std::string PT = pair ? "float2" : ST;
      s << "extern \"C\" __global__ void __launch_bounds__(256) " << out.entry << "_prep(const " << ST
        << "* __restrict__ data, mf_u64 stride, mf_u64 n, " << PT << "* __restrict__ outp) {\n"
        << "  for (mf_u64 i = (mf_u64)blockIdx.x * 256 + threadIdx.x; i < stride; i += (mf_u64)gridDim.x * 256) {\n"
        << "    const bool v = i < n;  // padding events are written as zeros\n";
      auto src = [&](int col) {
        return "(double)__ldg(data + (mf_u64)" + std::to_string(col) + " * stride + i)";
      };
      for (size_t m = 0; m < fold.cols.size(); m++) {
        s << "    {\n      double y = 0.0;\n      if (v) {\n";
        emit_fold(s, "        ", "f", fold.cols[m], src);
        s << "        y = f;\n      }\n";
        if (pair)
          s << "      const mf_dw w = mf_dw_split(y);\n      outp[(mf_u64)" << m << " * stride + i] = make_float2(w.h, w.l);\n";
        else
          s << "      outp[(mf_u64)" << m << " * stride + i] = (" << PT << ")y;\n";
        s << "    }\n";
      }
      s << "  }\n}\n";
    }
  } else if (kind == Kind::Store) {
    s << "extern \"C\" __global__ void __launch_bounds__(MF_BLOCK) " << out.entry << "(const " << ST
      << "* __restrict__ data, mf_u64 stride, mf_u64 n, mf_par P, " << ST
      << "* __restrict__ outp, mf_u64 out_stride) {\n";
    emit_params_and_uniform(s, "P.v");
    s << "  const mf_u64 step = (mf_u64)gridDim.x * MF_BLOCK;\n";
    s << "  for (mf_u64 i = (mf_u64)blockIdx.x * MF_BLOCK + threadIdx.x; i < n; i += step) {\n";
    for (int k : out.used_inputs)
      s << "    const " << AT << " x" << k << " = (" << AT << ")data[(mf_u64)" << k << " * stride + i];\n";
    emit_body(s, "    ");
    for (int j = 0; j < M; j++) s << "    outp[(mf_u64)" << j << " * out_stride + i] = (" << ST << ")r" << j << ";\n";
    s << "  }\n}\n";
  } else {
    // GENERATE: accept-reject generation, one xoshiro128++ stream per
    // `lanes` threads of a warp (a power of two up to 32, chosen at launch).
    // Stream t owns events [t*nper, min((t+1)*nper, n)) and makes them from
    // its proposals in order. In a turn, lane j of the stream's lanes tests
    // proposals j*chunk ... (j+1)*chunk - 1 of the next lanes*chunk, and the
    // accepted ones take the stream's next events in the order of the
    // proposals, so the events are those of one thread walking the stream,
    // and no lane waits for another stream's next acceptance.
    //
    // What bounds it: instructions, of which a third skipped the other lanes'
    // draws (six logic instructions a draw, (D+1) * (lanes - 1) draws after
    // each proposal) while a turn was one proposal a lane. With chunk > 1 a
    // lane jumps over them by a table of its own fixed number of steps, a
    // linear map of the 128-bit state: 64 loads and about 200 instructions
    // for `chunk` proposals and any number of lanes. The table is 8 KB of
    // shared memory, two words an entry so that the 16 values of a nibble lie
    // in all 32 banks once (with four words an entry the loads' bank
    // conflicts took twice the time), and every block makes it for itself.
    // K*mumu P wave, 1M events: 337 -> 215 us. chunk = 1 keeps the stepping,
    // for streams too short to pay for the table. Both forms measured, and
    // where the line lies: generator_shape() in mf_runtime.cpp.
    const int D = int(gen->dims.size());
    s << R"CUDA(__device__ __forceinline__ unsigned mf_rotl(unsigned x, int k) { return (x << k) | (x >> (32 - k)); }
struct mf_rng { unsigned s0, s1, s2, s3; };
__device__ __forceinline__ void mf_rng_step(mf_rng& s) {
  const unsigned t = s.s1 << 9, a = s.s2 ^ s.s0, b = s.s3 ^ s.s1;
  s.s1 ^= a; s.s0 ^= b; s.s2 = a ^ t; s.s3 = mf_rotl(b, 11);
}
__device__ __forceinline__ unsigned mf_rng_draw(mf_rng& s) {
  const unsigned r = mf_rotl(s.s0 + s.s3, 7) + s.s0;
  mf_rng_step(s);
  return r;
}
// A fixed number of steps is a 128 x 128 matrix over GF(2); `tab` holds, for
// each of the state's 32 nibbles and each value of it, the columns it adds.
__device__ __forceinline__ mf_rng mf_rng_jump(const uint2 (*tab)[512], const mf_rng s) {
  unsigned w[4] = {s.s0, s.s1, s.s2, s.s3};
  mf_rng r = {0u, 0u, 0u, 0u};
#pragma unroll 1
  for (int k = 0; k < 4; k++) {
#pragma unroll
    for (int q = 0; q < 8; q++) {
      const unsigned v = k * 128 + q * 16 + ((w[0] >> (4 * q)) & 15u);
      const uint2 e = tab[0][v], f = tab[1][v];
      r.s0 ^= e.x; r.s1 ^= e.y; r.s2 ^= f.x; r.s3 ^= f.y;
    }
    w[0] = w[1]; w[1] = w[2]; w[2] = w[3];
  }
  return r;
}
// Lane `sub` of a stream goes `sub * steps` steps ahead, and `tab` becomes the
// table of `lanes * steps` steps. Column threadIdx.x of the matrix is stepped
// from its unit vector; applying a table to its own columns doubles the steps.
// All threads of a block of MF_BLOCK >= 128 call this together.
__device__ __forceinline__ mf_rng mf_rng_spread(mf_rng st, unsigned steps, unsigned sub, unsigned lanes, uint4* col,
                                                uint2 (*tab)[512]) {
  const unsigned t = threadIdx.x & 127u, bit = 1u << (t & 31u);
  mf_rng c = {t < 32u ? bit : 0u, (t >> 5) == 1u ? bit : 0u, (t >> 5) == 2u ? bit : 0u, t >= 96u ? bit : 0u};
  for (unsigned k = 0; k < steps; k++) mf_rng_step(c);
  for (unsigned b = 1;; b *= 2) {
    if (threadIdx.x < 128u) col[t] = make_uint4(c.s0, c.s1, c.s2, c.s3);
    __syncthreads();
    if (threadIdx.x < 128u) {
      // four values of nibble t / 4: the upper two bits are those of t
      const uint4* n = col + (t & ~3u);
      const uint4 p = n[0], q = n[1], u = n[2], v = n[3];
      const unsigned mu = (t & 1u) ? MF_FULL : 0u, mv = (t & 2u) ? MF_FULL : 0u;
      const uint2 z0 = make_uint2((u.x & mu) ^ (v.x & mv), (u.y & mu) ^ (v.y & mv));
      const uint2 z1 = make_uint2((u.z & mu) ^ (v.z & mv), (u.w & mu) ^ (v.w & mv));
      uint2 *lo = tab[0] + 4u * t, *hi = tab[1] + 4u * t;
      lo[0] = z0;
      lo[1] = make_uint2(z0.x ^ p.x, z0.y ^ p.y);
      lo[2] = make_uint2(z0.x ^ q.x, z0.y ^ q.y);
      lo[3] = make_uint2(z0.x ^ p.x ^ q.x, z0.y ^ p.y ^ q.y);
      hi[0] = z1;
      hi[1] = make_uint2(z1.x ^ p.z, z1.y ^ p.w);
      hi[2] = make_uint2(z1.x ^ q.z, z1.y ^ q.w);
      hi[3] = make_uint2(z1.x ^ p.z ^ q.z, z1.y ^ p.w ^ q.w);
    }
    __syncthreads();
    if (b >= lanes) return st;
    if (sub & b) st = mf_rng_jump(tab, st);
    c = mf_rng_jump(tab, c);
  }
}
)CUDA";
    if (!ar32) s << kEfPrelude;
    // The reference prints min, max-min and maxprob with "%.15e" into its
    // generate kernel (compute_llvm.hh:466-478,485-489) and evaluates
    // min + delta*u and maxprob*u with one rounding per operation; the
    // explicit _rn intrinsics keep the compiler from fusing them, so the
    // proposals are bit-identical to the reference's.
    auto printed15 = [](double v) {
      char b[64];
      std::snprintf(b, sizeof b, "%.15e", v);
      return std::strtod(b, nullptr);
    };
    const char* mul = ar32 ? "__fmul_rn" : "__dmul_rn";
    const char* add = ar32 ? "__fadd_rn" : "__dadd_rn";
    // coordinate d from its draw (an expression), in the generated type; a
    // draw times 2^-32 is exact in FP64 and one rounding of the draw in FP32
    auto coordinate = [&](int d, const std::string& draw) {
      return std::string(add) + "(" + fmt_const(printed15(gen->lo[d]), ar32) + ", " + mul + "(" +
             fmt_const(printed15(gen->hi[d] - gen->lo[d]), ar32) + ", " +
             (ar32 ? "(float)" + draw + " * 2.3283064365386963e-10f" : draw + " * 2.3283064365386963e-10") + "))";
    };
    // FP64 generation decides maxprob*u < p in FP32 wherever that is certain:
    // the density is evaluated in FP32 together with a bound of its error
    // (kEfPrelude), and only where |maxprob*u - p| is within the bounds of
    // both sides, or anything is not finite, are the coordinates and the
    // density formed in FP64 (the code the reference runs) and compared. Every
    // decision, and so every event, equals the FP64 one; GB300 issues FP64 at
    // 1/64 of its FP32 rate. The accepted draws are stored in place of the
    // coordinates and turned into coordinates, FP64 as the reference forms
    // them, when the stream is complete (full warps instead of the few lanes
    // that accept).
    const bool filter = !ar32;
    // A bound as an FP32 literal, 0 or at least 2^-126: a smaller one is out of
    // range for the compiler, and results that underflow are off by up to 2^-150.
    auto bound_f = [](double e) {
      char b[48];
      std::snprintf(b, sizeof b, "%.9ef", e > 0.0 ? e + 0x1p-126 : 0.0);
      return std::string(b);
    };
    std::string filter_call;
    std::vector<int> filter_uniform;
    if (filter) {
      std::set<int> uni;
      auto note = [&](int k) {
        if (k >= 0 && ns[k].uniform && ns[k].op != Op::Const) uni.insert(k);
      };
      std::set<int> conditions;  // parameter-only conditions of selects, exact
      for (size_t i = 0; i < ns.size(); i++) {
        if (!live[i] || ns[i].uniform || ns[i].op == Op::Input) continue;
        const bool cond = ns[i].op == Op::Select && ns[ns[i].a].uniform;
        if (cond) conditions.insert(ns[i].a);
        if (!cond) note(ns[i].a);
        note(ns[i].b);
        note(ns[i].c);
      }
      for (int r : roots) note(r);
      auto eref = [&](int id) -> std::string {
        const Node& n = ns[id];
        if (n.op == Op::Const) {
          const float v = float(n.value);
          if (!std::isfinite(v)) return "mf_ef_make(0.0f, MF_EF_INF)";  // decided in FP64
          // the rounding of the constant, bounded (0 when it is exact)
          const double e = std::fabs(n.value - double(v)) * 1.0000005;
          return "mf_ef_make(" + fmt_const(n.value, true) + ", " + bound_f(e) + ")";
        }
        if (n.op == Op::Input) return "x" + std::to_string(n.index);
        return (n.uniform ? "uf" : "f") + std::to_string(id);
      };
      s << "// The density in FP32 and a bound of its error; `amb` is set where a comparison is uncertain.\n"
        << "__device__ __forceinline__ mf_ef mf_filter(";
      for (int d = 0; d < D; d++) s << "mf_ef x" << d << ", ";
      for (int k : uni) s << "mf_ef uf" << k << ", ";
      for (int k : conditions) s << "bool uc" << k << ", ";
      s << "bool& amb) {\n";
      std::map<int, std::pair<int, int>> pair_of = sincos_pairs(ns, live);
      for (size_t i = 0; i < ns.size(); i++) {
        const Node& n = ns[i];
        if (!live[i] || n.uniform || n.op == Op::Input) continue;
        const std::string A = n.a >= 0 ? eref(n.a) : "", B = n.b >= 0 ? eref(n.b) : "", C = n.c >= 0 ? eref(n.c) : "";
        const std::string lhs = "  const mf_ef f" + std::to_string(i) + " = ";
        switch (n.op) {
          case Op::Add: s << lhs << "mf_ef_add(" << A << ", " << B << ");\n"; break;
          case Op::Sub: s << lhs << "mf_ef_sub(" << A << ", " << B << ");\n"; break;
          case Op::Mul: s << lhs << "mf_ef_mul(" << A << ", " << B << ");\n"; break;
          case Op::Div: s << lhs << "mf_ef_mul(" << A << ", mf_ef_rcp(" << B << "));\n"; break;
          case Op::Neg: s << lhs << "mf_ef_neg(" << A << ");\n"; break;
          case Op::Pow: s << lhs << "mf_ef_pow(" << A << ", " << B << ");\n"; break;
          case Op::Cmp:
            s << "  amb = amb || mf_ef_near(" << A << ", " << B << ");\n  const bool f" << i << " = " << A << ".v "
              << cmp_str(n.cmp) << " " << B << ".v;\n";
            break;
          case Op::Select:
            // a condition that is not a comparison tests a value against zero
            if (ns[n.a].uniform)
              s << lhs << "uc" << n.a << " ? " << B << " : " << C << ";\n";
            else if (ns[n.a].op == Op::Cmp)
              s << lhs << A << " ? " << B << " : " << C << ";\n";
            else
              s << "  amb = amb || mf_ef_near(" << A << ", mf_ef_make(0.0f, 0.0f));\n"
                << lhs << A << ".v != 0.0f ? " << B << " : " << C << ";\n";
            break;
          case Op::Sin:
          case Op::Cos: {
            auto it = pair_of.find(n.a);
            if (it == pair_of.end()) {
              s << lhs << (n.op == Op::Sin ? "mf_ef_sin(" : "mf_ef_cos(") << A << ");\n";
            } else if (int(i) == std::min(it->second.first, it->second.second)) {
              s << "  mf_ef f" << it->second.first << ", f" << it->second.second << ";\n  mf_ef_sincos(" << A << ", &f"
                << it->second.first << ", &f" << it->second.second << ");\n";
            }
            break;
          }
          default:
            if (n.op != Op::Rcp && !is_unary_fn(n.op)) throw std::runtime_error("emit: unexpected node");
            s << lhs << "mf_ef_" << (n.op == Op::Rcp ? "rcp" : fn_name(n.op, false)) << "(" << A << ");\n";
        }
      }
      s << "  return " << eref(roots[0]) << ";\n}\n";
      filter_call = "mf_filter(";
      for (int d = 0; d < D; d++) filter_call += "xe" + std::to_string(d) + ", ";
      for (int k : uni) filter_call += "uf" + std::to_string(k) + ", ";
      for (int k : conditions) filter_call += "(" + em.ref(k, "u") + ") != 0.0, ";
      filter_call += "amb)";
      for (int k : uni) filter_uniform.push_back(k);
    }
    // one stream's events, `lanes` threads a stream; from, to, maxprob and
    // the parameter-only values are defined
    // A chunk's accepted proposals wait in shared memory (at most 24 KB) for
    // their events' places.
    const unsigned chunk_max = out.gen_chunk = std::max(1u, std::min(8u, 48u / unsigned(D)));
    auto draw = [](int d) { return "d" + std::to_string(d); };
    auto slot = [](int d) { return "outp[(mf_u64)" + std::to_string(d) + " * out_stride + at]"; };
    // acc = the decision on the proposal with the draws d0...
    auto decide = [&]() {
      for (int d = 0; d <= D; d++) s << "      const unsigned d" << d << " = mf_rng_draw(st);\n";
      s << "      bool acc = false;\n"
        << "      if (run && tried + at_try < max_tries) {\n";
      if (filter) {
        for (int d = 0; d < D; d++) {
          const double lo = printed15(gen->lo[d]), del = printed15(gen->hi[d] - gen->lo[d]);
          // an end or a width that FP32 cannot hold: decided in FP64
          const bool fits = std::isfinite(float(lo)) && std::isfinite(float(del)) && std::isfinite(float(lo + del));
          s << "        const mf_ef xe" << d << " = mf_ef_make("
            << (fits ? "__fmaf_rn(" + fmt_const(del, true) + ", (float)d" + std::to_string(d) +
                           " * 2.3283064365386963e-10f, " + fmt_const(lo, true) + ")"
                     : std::string("0.0f"))
            << ", " << (fits ? bound_f((std::fabs(lo) + std::fabs(del)) * 0x1p-22) : "MF_EF_INF") << ");\n";
        }
        s << "        bool amb = false;\n        const mf_ef p = " << filter_call << ";\n"
          << "        const mf_ef ug = mf_ef_mul(maxprob_f, mf_ef_make((float)d" << D
          << " * 2.3283064365386963e-10f, 0x1p-24f));\n"
          << "        const float gap = __fsub_rn(p.v, ug.v);\n"
          << "        acc = gap > 0.0f;\n"
          << "        if (amb || !(fabsf(gap) > 1.01f * (p.e + ug.e) + 0x1p-23f * fabsf(gap))) {  // in FP64\n";
        for (int d = 0; d < D; d++) s << "          const double x" << d << " = " << coordinate(d, draw(d)) << ";\n";
        emit_body(s, "          ");
        s << "          acc = __dmul_rn(maxprob, d" << D << " * 2.3283064365386963e-10) < r0;\n        }\n";
      } else {
        for (int d = 0; d < D; d++) s << "        const float x" << d << " = " << coordinate(d, draw(d)) << ";\n";
        emit_body(s, "        ");
        s << "        acc = __fmul_rn(maxprob, (float)d" << D << " * 2.3283064365386963e-10f) < r0;\n";
      }
      s << "      }\n";
    };
    auto keep_event = [&](const std::string& pad, const std::function<std::string(int)>& w) {
      for (int d = 0; d < D; d++)
        s << pad << slot(d) << " = "
          << (filter ? "__longlong_as_double((long long)" + w(d) + ")" : coordinate(d, w(d))) << ";\n";
    };
    auto end_of_turn = [&]() {
      s << "      if (run && i >= to) {\n        run = false;\n      } else if (run && tried >= max_tries) {\n"
        << "        run = false;\n        if (sub == 0u) atomicOr(status, 1u);\n      }\n    }\n";
    };
    auto accept_reject = [&]() {
      if (chunk_max > 1)
        s << "  __shared__ uint4 mf_col[MF_BLOCK];\n  __shared__ uint2 mf_tab[2][512];\n  __shared__ unsigned mf_kept["
          << chunk_max * D << " * MF_BLOCK];\n";
      for (int k : filter_uniform)
        s << "  const mf_ef uf" << k << " = mf_ef_from(" << em.ref(k, "u") << ");\n";
      if (filter) s << "  const mf_ef maxprob_f = mf_ef_from(maxprob);\n";
      s << "  const unsigned sub = threadIdx.x & (lanes - 1u);\n"
        << "  mf_u64 i = from, tried = 0;\n  bool run = i < to;\n";
      if (chunk_max > 1) {
        s << "  if (chunk > 1u) {\n    st = mf_rng_spread(st, chunk * " << D + 1 << "u, sub, lanes, mf_col, mf_tab);\n"
          << "    while (__any_sync(MF_FULL, run)) {\n      mf_col[threadIdx.x] = make_uint4(st.s0, st.s1, st.s2, st.s3);\n"
          << "      unsigned c = 0;\n#pragma unroll 1\n"
          << "      for (unsigned q = 0; q < chunk; q++) {\n      const unsigned at_try = sub * chunk + q;\n";
        decide();
        s << "      if (acc) {\n";
        const std::string KD = " * " + std::to_string(D) + "u + ";
        for (int d = 0; d < D; d++)
          s << "        mf_kept[(c" << KD << d << "u) * MF_BLOCK + threadIdx.x] = d" << d << ";\n";
        s << "        c++;\n      }\n      }\n      const uint4 w = mf_col[threadIdx.x];\n"
          << "      st = mf_rng_jump(mf_tab, mf_rng{w.x, w.y, w.z, w.w});\n"
          << "      unsigned upto = c;  // events of this and the stream's earlier lanes\n"
          << "      for (unsigned o = 1; o < lanes; o *= 2) {\n"
          << "        const unsigned v = __shfl_up_sync(MF_FULL, upto, o, lanes);\n        if (sub >= o) upto += v;\n"
          << "      }\n      for (unsigned j = 0; j < c; j++) {\n        const mf_u64 at = i + (upto - c) + j;\n"
          << "        if (at < to) {\n";
        keep_event("          ", [&](int d) {
          return "mf_kept[(j" + KD + std::to_string(d) + "u) * MF_BLOCK + threadIdx.x]";
        });
        s << "        }\n      }\n      i += __shfl_sync(MF_FULL, upto, lanes - 1u, lanes);\n      tried += lanes * chunk;\n";
        end_of_turn();
        s << "  } else {\n";
      } else {
        s << "  {\n";
      }
      s << "    const unsigned first = (threadIdx.x & 31u) - sub;\n"
        << "    const unsigned mine = lanes == 32u ? MF_FULL : ((1u << lanes) - 1u);\n"
        << "    for (unsigned k = 0; k < sub; k++) {\n#pragma unroll\n      for (int q = 0; q < " << D + 1
        << "; q++) mf_rng_step(st);\n    }\n"
        << "    while (__any_sync(MF_FULL, run)) {\n      const unsigned at_try = sub;\n";
      decide();
      s << "      for (unsigned k = 1; k < lanes; k++) {\n#pragma unroll\n        for (int q = 0; q < " << D + 1
        << "; q++) mf_rng_step(st);\n      }\n"
        << "      const unsigned m = (__ballot_sync(MF_FULL, acc) >> first) & mine;\n"
        << "      if (acc) {\n        const mf_u64 at = i + __popc(m & ((1u << sub) - 1u));\n        if (at < to) {\n";
      keep_event("          ", draw);
      s << "        }\n      }\n      i += __popc(m);\n      tried += lanes;\n";
      end_of_turn();
      s << "  }\n";
      if (filter) {
        s << "  // the stored draws become coordinates\n  __syncwarp();\n  if (i > to) i = to;\n"
          << "  for (mf_u64 at = from + sub; at < i; at += lanes) {\n";
        for (int d = 0; d < D; d++)
          s << "    { const unsigned w = (unsigned)__double_as_longlong(" << slot(d) << ");\n      " << slot(d) << " = "
            << coordinate(d, "w") << "; }\n";
        s << "  }\n";
      }
      s << "}\n";
    };
    s << "extern \"C\" __global__ void __launch_bounds__(MF_BLOCK) " << out.entry
      << "(const unsigned* __restrict__ seeds, unsigned nseeds, mf_u64 n, mf_u64 nper, mf_par P, " << ST
      << "* __restrict__ outp, mf_u64 out_stride, unsigned* __restrict__ status, unsigned long long max_tries,"
      << " unsigned long long splitmix_seed, unsigned lanes, unsigned chunk) {\n";
    // whole warps stay in the loop: threads beyond the last stream have no events
    s << "  const mf_u64 thread = (mf_u64)blockIdx.x * MF_BLOCK + threadIdx.x;\n"
      << "  const bool have = thread / lanes < nseeds;\n"
      << "  const unsigned t = have ? (unsigned)(thread / lanes) : 0u;\n";
    // the stream's xoshiro128++ state: from the seed table, or (seeds null)
    // made here as mf_splitmix_seed_rows makes row t: the upper halves of four
    // SplitMix64 outputs (Steele, Lea and Flood, OOPSLA 2014) from
    // (seed mod 2^32) * 2^32 + t
    s << "  unsigned w[4];\n"
      << "  if (seeds) {\n#pragma unroll\n    for (int k = 0; k < 4; k++) w[k] = seeds[(mf_u64)k * nseeds + t];\n"
      << "  } else {\n    unsigned long long sm = (splitmix_seed & 0xffffffffull) * 4294967296ull + t;\n"
      << "#pragma unroll\n    for (int k = 0; k < 4; k++) {\n"
      << "      unsigned long long z = (sm += 0x9e3779b97f4a7c15ull);\n"
      << "      z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;\n"
      << "      z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;\n"
      << "      w[k] = (unsigned)((z ^ (z >> 31)) >> 32);\n    }\n  }\n"
      << "  mf_rng st = {w[0], w[1], w[2], w[3]};\n";
    emit_params_and_uniform(s, "P.v");
    s << "  const " << AT << " maxprob = " << fmt_const(printed15(gen->maxprob), ar32) << ";\n";
    s << "  const mf_u64 from = have ? (mf_u64)t * nper : 0;\n"
      << "  mf_u64 to = have ? from + nper : 0; if (to > n) to = n;\n";
    accept_reject();
    // Segments (toy studies): `threads_per_seg` streams per segment; segment
    // s owns events [seg_begin[s], seg_begin[s] + seg_count[s]) and generates
    // them with its own parameter row and bound (stream r of the segment
    // takes the r-th block of ceil(count / threads_per_seg) events).
    s << "extern \"C\" __global__ void __launch_bounds__(MF_BLOCK) " << out.entry
      << "_segments(const unsigned* __restrict__ seeds, unsigned nthreads, unsigned threads_per_seg,"
      << " const mf_u64* __restrict__ seg_begin, const unsigned* __restrict__ seg_count,"
      << " const mf_par* __restrict__ seg_params, const double* __restrict__ seg_maxprob, " << ST
      << "* __restrict__ outp, mf_u64 out_stride, unsigned* __restrict__ status, unsigned long long max_tries,"
      << " unsigned lanes, unsigned chunk) {\n";
    s << "  const mf_u64 thread = (mf_u64)blockIdx.x * MF_BLOCK + threadIdx.x;\n"
      << "  const bool have = thread / lanes < nthreads;\n"
      << "  const unsigned t = have ? (unsigned)(thread / lanes) : 0u;\n"
      << "  const unsigned seg = t / threads_per_seg, r = t - seg * threads_per_seg;\n";
    s << "  mf_rng st = {seeds[t], seeds[(mf_u64)nthreads + t], seeds[2 * (mf_u64)nthreads + t], "
         "seeds[3 * (mf_u64)nthreads + t]};\n";
    s << "  const mf_par& P = seg_params[seg];\n";
    emit_params_and_uniform(s, "P.v");
    s << "  const " << AT << " maxprob = (" << AT << ")seg_maxprob[seg];\n";
    s << "  const mf_u64 cnt = have ? seg_count[seg] : 0, per = (cnt + threads_per_seg - 1) / threads_per_seg;\n";
    s << "  const mf_u64 end = seg_begin[seg] + cnt, from = seg_begin[seg] + (mf_u64)r * per;\n";
    s << "  mf_u64 to = from + per; if (to > end) to = end;\n";
    accept_reject();
  }
  out.source = s.str();
  return out;
}


void LoweredKernel::fill_args(const double* params, size_t np, unsigned char* out) const {
  fill_args_many(params, np, 1, out);
}

void LoweredKernel::fill_args_many(const double* params, size_t np, size_t count, unsigned char* out) const {
  // Straight-line evaluation of the nodes the slots read (both arms of a
  // select are evaluated; their values only feed the select), into a scratch
  // array of which only those entries are written and read; one scratch for
  // all rows.
  std::vector<double> val(nodes.size());
  const size_t ab = args_bytes();
  for (size_t r = 0; r < count; r++) {
    const double* pr = params + r * np;
    unsigned char* o = out + r * ab;
    std::memset(o, 0, ab);
    for (int id : eval_order) {
      const Node& n = nodes[id];
      double v;
      switch (n.op) {
        case Op::Const: v = n.value; break;
        case Op::Param: v = size_t(n.index) < np ? pr[n.index] : 0.0; break;
        case Op::Input: throw std::runtime_error("input column in a parameter-only value");
        case Op::Add: v = val[n.a] + val[n.b]; break;
        case Op::Sub: v = val[n.a] - val[n.b]; break;
        case Op::Mul: v = val[n.a] * val[n.b]; break;
        case Op::Div: case Op::Pow: v = apply_binary(n.op, val[n.a], val[n.b]); break;
        case Op::Cmp: v = apply_cmp(n.cmp, val[n.a], val[n.b]) ? 1.0 : 0.0; break;
        case Op::Select: v = val[n.a] != 0.0 ? val[n.b] : val[n.c]; break;
        default: v = apply_unary(n.op, val[n.a]); break;
      }
      val[id] = v;
    }
    double* d = reinterpret_cast<double*>(o);
    float* f = reinterpret_cast<float*>(o + size_t(nd) * 8);
    for (const auto& sl : slots) {
      const double v = val[sl.node];
      switch (sl.kind) {
        case UniformSlot::Double: d[sl.offset] = v; break;
        case UniformSlot::Float: f[sl.offset] = float(v); break;
        case UniformSlot::Bool: f[sl.offset] = v != 0.0 ? 1.0f : 0.0f; break;
        case UniformSlot::DwPair: {
          const float h = float(v);
          f[sl.offset] = h;
          f[sl.offset + 1] = float(v - double(h));
          break;
        }
      }
    }
  }
}

}  // namespace mf
