// Routine compilation: cut the body into stages, find the parallel loops of each stage and
// generate its kernel.  See compile.hpp.
//
// The reference runs a routine as ONE sequential function (cc: arrayjit/lib/cc_backend.ml:325-343;
// cuda: one thread of one block, arrayjit/lib/cuda_backend.ml:357-360,1043).  Here every
// top-level loop nest (`loop_accum` emits one per assignment, arrayjit/lib/assignments.ml:311-488)
// becomes a kernel whose threads own disjoint iterations of the nest's independent loops.
#include "compile.hpp"

#include <algorithm>
#include <cmath>
#include <functional>
#include <set>
#include <sstream>

#include "emit.hpp"

namespace b200 {

bool match_attention(const Program& P, const std::vector<StmtP>& flat, size_t at, const CompileOptions& opt, int* n_absorbed,
                     Stage* out);
std::string attn_translation_unit(const Program& P, Stage& st, const std::string& kernel_name);
bool match_gemm(const Program& P, const std::vector<LoopDim>& nest, const Stmt& body, bool zeroed_before,
                const CompileOptions& opt, const std::vector<Follower>& followers, int* n_fused,
                Stage* out);  // gemm_match.cpp
void group_contractions(Code& code, const CompileOptions& opt);
std::string gemm_translation_unit(const Program& P, Stage& st, const std::string& kernel_name,
                                  const CompileOptions& opt);

namespace {

// ---- walking helpers
void walk_scalar(const Scalar& e, const std::function<void(const Scalar&)>& fs,
                 const std::function<void(const Stmt&)>& ft);
void walk_stmt(const Stmt& s, const std::function<void(const Scalar&)>& fs, const std::function<void(const Stmt&)>& ft) {
  ft(s);
  switch (s.kind) {
    case Stmt::Seq:
      for (auto& x : s.items) walk_stmt(*x, fs, ft);
      break;
    case Stmt::For: walk_stmt(*s.body, fs, ft); break;
    case Stmt::Set:
    case Stmt::SetLocal: walk_scalar(*s.value, fs, ft); break;
    default: break;
  }
}
void walk_scalar(const Scalar& e, const std::function<void(const Scalar&)>& fs,
                 const std::function<void(const Stmt&)>& ft) {
  fs(e);
  if (e.kind == Scalar::LocalScope) walk_stmt(*e.body, fs, ft);
  for (auto& a : e.args) walk_scalar(*a.s, fs, ft);
}

// Nodes whose values are compared, gate something or are truncated, and those that they are computed from: a change in the
// last bits of such a value may change a result by a whole step.  (A position read by a value, `GetDyn`, is one too.)  A sum
// that is decided on by the assignment that holds it counts as that assignment's node.  What another routine does with a
// node is not known here: a forward pass compiled by itself may add in another order than the step that gates its values.
std::set<int> find_deciding(const Program& P) {
  static const std::set<std::string> first = {"relu_gate", "sat01_gate", "where", "trunc", "not"},
                                     both = {"lt", "eq", "ne", "or", "and", "mod"};
  std::set<int> found;
  std::map<int, std::set<int>> made_from;
  auto local = [](int scope_id) { return -1 - scope_id; };   // scalar locals stand beside the nodes
  walk_stmt(*P.body, [](const Scalar&) {}, [&](const Stmt& st) {
    if (st.kind != Stmt::Set && st.kind != Stmt::SetLocal) return;
    const int target = st.kind == Stmt::Set ? st.tn : local(st.scope_id);
    std::set<int> all;
    bool open = is_int_prec(P.tn(st.tn).prec);   // values of scopes are followed to the whole assignment
    bool own = open;                             // a sum of this assignment decides something
    auto reads = [&](const Scalar& e, std::set<int>& into) {
      walk_scalar(e, [&](const Scalar& x) {
        if (x.kind == Scalar::Get || x.kind == Scalar::GetDyn || x.kind == Scalar::GetMerge) into.insert(x.tn);
        if (x.kind == Scalar::GetLocal) {
          into.insert(local(x.scope_id));
          open = open || &into == &found;
        }
        if (x.kind == Scalar::GetLocal || x.kind == Scalar::LocalScope) own = own || &into == &found;
      }, [](const Stmt&) {});
    };
    reads(*st.value, all);
    walk_scalar(*st.value, [&](const Scalar& x) {
      const bool truncated = x.kind == Scalar::LocalScope && is_int_prec(P.tn(x.tn).prec);
      if (x.kind == Scalar::GetDyn || truncated) open = true;
      own = own || truncated;
      for (size_t a = 0; a < x.args.size(); ++a)
        if (both.count(x.op) || (a == 0 && first.count(x.op))) reads(*x.args[a].s, found);
    }, [](const Stmt&) {});
    if (open) found.insert(all.begin(), all.end());
    if (own) found.insert(target);
    made_from[target].insert(all.begin(), all.end());
  });
  std::vector<int> todo(found.begin(), found.end());
  while (!todo.empty()) {
    const int n = todo.back();
    todo.pop_back();
    for (int m : made_from[n])
      if (found.insert(m).second) todo.push_back(m);
  }
  return found;
}

// Is loop symbol `s` safe to run in parallel over `body`?  Sufficient condition: every
// node written in the body is written only at positions that carry `s` as a plain iterator
// on one fixed axis, and every read of such a node carries `s` on that same axis — so
// distinct values of `s` touch disjoint slices of everything that is written.
bool parallel_safe(const std::string& s, const Stmt& body) {
  std::map<int, int> axis_of;  // written node -> axis that carries s
  std::map<int, Index> index_of;  // written node -> the index on that axis
  bool ok = true;
  // an index is one-to-one in s when it is s itself or c * s + fixed with c != 0 (a padded
  // node addressed past its margin)
  auto one_to_one = [&](const Index& ix) {
    return (ix.kind == Index::Iter && ix.sym == s) ||
           (ix.kind == Index::Affine && ix.terms.size() == 1 && ix.terms[0].second == s && ix.terms[0].first != 0);
  };
  auto same_index = [](const Index& a, const Index& b) {
    return a.kind == b.kind && a.sym == b.sym && a.fixed == b.fixed && a.terms == b.terms;
  };
  auto axis_with = [&](const Indices& idcs) {
    for (size_t a = 0; a < idcs.size(); ++a)
      if (one_to_one(idcs[a])) return (int)a;
    return -1;
  };
  walk_stmt(
      body, [](const Scalar&) {},
      [&](const Stmt& st) {
        if (st.kind == Stmt::ZeroOut) ok = false;
        if (st.kind == Stmt::Set) {
          int a = axis_with(st.idcs);
          if (st.vec_len > 0 && a >= 0 && st.idcs[a].kind == Index::Affine) a = -1;  // judged by the rule below
          if (a < 0 && st.vec_len > 0 && !st.idcs.empty()) {
            // a vector store whose last index is c * s (+ fixed) with c >= the vector length
            // writes disjoint runs for distinct s
            const Index& last = st.idcs.back();
            if (last.kind == Index::Affine && last.terms.size() == 1 && last.terms[0].second == s &&
                last.terms[0].first >= st.vec_len)
              a = (int)st.idcs.size() - 1;
          } else if (a >= 0 && st.vec_len > 1 && a == (int)st.idcs.size() - 1) {
            a = -1;  // runs of neighbouring elements would overlap
          }
          if (a < 0) { ok = false; return; }
          // the symbol must not appear on any other axis of the write
          for (size_t k = 0; k < st.idcs.size(); ++k)
            if ((int)k != a && st.idcs[k].uses(s)) ok = false;
          auto it = axis_of.find(st.tn);
          if (it == axis_of.end()) { axis_of[st.tn] = a; index_of[st.tn] = st.idcs[a]; }
          else if (it->second != a || !same_index(index_of[st.tn], st.idcs[a])) ok = false;
        }
      });
  if (!ok) return false;
  walk_stmt(
      body,
      [&](const Scalar& e) {
        if (e.kind == Scalar::Get || e.kind == Scalar::GetDyn) {
          auto it = axis_of.find(e.tn);
          if (it == axis_of.end()) return;
          if (e.kind == Scalar::GetDyn) { ok = false; return; }
          int a = it->second;
          if (a >= (int)e.idcs.size() || !same_index(e.idcs[a], index_of[e.tn])) ok = false;
          for (size_t k = 0; k < e.idcs.size(); ++k)
            if ((int)k != a && e.idcs[k].uses(s)) ok = false;
        }
      },
      [](const Stmt&) {});
  return ok;
}

// `t[p] := fma(a, b, t[p])` or `t[p] := t[p] + term` (either order) where neither a, b nor the
// term read t or hold a local scope.
bool accumulates_into_self(const Stmt& set) {
  if (set.kind != Stmt::Set || !set.value) return false;
  const Scalar& v = *set.value;
  auto is_self = [&](const Scalar& e) {
    if (e.kind != Scalar::Get || e.tn != set.tn || e.idcs.size() != set.idcs.size()) return false;
    for (size_t i = 0; i < e.idcs.size(); ++i)
      if (e.idcs[i].kind != set.idcs[i].kind || e.idcs[i].sym != set.idcs[i].sym || e.idcs[i].fixed != set.idcs[i].fixed ||
          e.idcs[i].terms != set.idcs[i].terms)
        return false;
    return true;
  };
  auto plain = [&](const Scalar& e) {
    bool ok = true;
    walk_scalar(e, [&](const Scalar& x) {
      if ((x.kind == Scalar::Get || x.kind == Scalar::GetDyn) && x.tn == set.tn) ok = false;
      if (x.kind == Scalar::LocalScope) ok = false;
    }, [](const Stmt&) {});
    return ok;
  };
  if (v.kind == Scalar::Tern && v.op == "fma")
    return is_self(*v.args[2].s) && plain(*v.args[0].s) && plain(*v.args[1].s);
  if (v.kind == Scalar::Bin && v.op == "add")
    return (is_self(*v.args[0].s) && plain(*v.args[1].s)) || (is_self(*v.args[1].s) && plain(*v.args[0].s));
  return false;
}

// Innermost iterations one execution of a statement takes (loops and reductions inside it multiplied out).
double iterations(const Stmt& s);
double iterations(const Scalar& e) {
  double n = e.kind == Scalar::LocalScope ? iterations(*e.body) : 0.0;
  for (auto& a : e.args) n += iterations(*a.s);
  return n;
}
double iterations(const Stmt& s) {
  switch (s.kind) {
    case Stmt::Seq: {
      double n = 0;
      for (auto& x : s.items) n += iterations(*x);
      return n;
    }
    case Stmt::For: return (double)std::max<int64_t>(0, s.to - s.from + 1) * iterations(*s.body);
    case Stmt::Set:
    case Stmt::SetLocal: return 1.0 + iterations(*s.value);
    default: return 0.0;
  }
}

bool body_has_set(const Stmt& s) {
  bool any = false;
  walk_stmt(s, [](const Scalar&) {}, [&](const Stmt& st) {
    if (st.kind == Stmt::Set || st.kind == Stmt::ZeroOut) any = true;
  });
  return any;
}

// Does the statement tree mention a function-scope scalar local (declared outside it)?
void collect_scopes(const Stmt& s, std::set<std::pair<int, int>>& declared, std::set<std::pair<int, int>>& used) {
  walk_stmt(
      s,
      [&](const Scalar& e) {
        if (e.kind == Scalar::LocalScope) declared.insert({e.scope_id, e.tn});
        if (e.kind == Scalar::GetLocal) used.insert({e.scope_id, e.tn});
      },
      [&](const Stmt& st) {
        if (st.kind == Stmt::DeclareLocal) declared.insert({st.scope_id, st.tn});
        if (st.kind == Stmt::SetLocal) used.insert({st.scope_id, st.tn});
      });
}

// Cooperative row reduction: the stage's body is `Set t[..] := E` where E holds Local_scope
// reductions `v := neutral; for k { v := v (+|max|min) f(k) }` over loops long enough that a
// warp per output element pays.  Returns the lane-strided symbol or "".
struct CoopInfo {
  std::string sym;
  int width = 32;  // threads cooperating on one output element
  int64_t extent = 0;   // terms of the reduction
  int grid_blocks = 0;  // >0: two-kernel grid-wide reduction with this many blocks in pass 1
  std::vector<std::pair<int, std::string>> scopes;  // (scope id, combine op)
};

bool accum_form(const Stmt& st, int sid, int tn, std::string* op) {
  // Set_local(id, Binop(op, Get_local id, x)) | Binop(op, x, Get_local id) | FMA(a, b, Get_local id)
  if (st.kind != Stmt::SetLocal || st.scope_id != sid || st.tn != tn) return false;
  const Scalar& v = *st.value;
  auto is_self = [&](const Scalar& e) { return e.kind == Scalar::GetLocal && e.scope_id == sid && e.tn == tn; };
  auto mentions_self = [&](const Scalar& e) {
    bool m = false;
    walk_scalar(e, [&](const Scalar& x) { if (is_self(x)) m = true; }, [](const Stmt&) {});
    return m;
  };
  if (v.kind == Scalar::Tern && v.op == "fma") {
    if (is_self(*v.args[2].s) && !mentions_self(*v.args[0].s) && !mentions_self(*v.args[1].s)) {
      *op = "add";
      return true;
    }
    return false;
  }
  if (v.kind == Scalar::Bin && (v.op == "add" || v.op == "max" || v.op == "min")) {
    if (is_self(*v.args[0].s) && !mentions_self(*v.args[1].s)) { *op = v.op; return true; }
    if (is_self(*v.args[1].s) && !mentions_self(*v.args[0].s)) { *op = v.op; return true; }
  }
  return false;
}

}  // namespace

int64_t PackOp::rows() const {
  int64_t r = kmajor ? 1 : seg * (split ? 2 : 1);
  if (kmajor)
    for (auto& a : mn) r *= a.extent;
  for (auto& a : batch) r *= a.extent;
  return r;
}
int64_t PackOp::bytes() const { return rows() * ld * prec_bytes(prec); }
std::string PackOp::key() const {
  std::ostringstream o;
  // (rows along m or n of values along k, or the other way round: the same copy, where a value is one part)
  o << tn << ":" << off << ":" << (split ? 1 + kmajor : 0) << ":" << ld << ":" << (split ? seg : 0);
  for (auto* v : {&batch, kmajor ? &mn : &k, kmajor ? &k : &mn}) {
    o << ";";
    for (auto& a : *v) o << a.extent << "," << a.stride << " ";
  }
  return o.str();
}

double GemmPlan::flops() const {
  double f = 2.0 * (double)m.extent * (double)n.extent * (double)k.extent;
  for (auto& b : batch) f *= (double)b.extent;
  return f;
}

std::string Code::describe() const {
  std::ostringstream o;
  o << "{\"name\":\"" << prog.name << "\",\"stages\":[";
  for (size_t i = 0; i < stages.size(); ++i) {
    const Stage& s = stages[i];
    if (i) o << ",";
    o << "{\"kind\":\"" << (s.kind == Stage::Memset || s.clears ? "memset" : s.kind == Stage::Gemm ? "gemm" : s.kind == Stage::Attn ? (s.attn.rows_kernel ? "row attention" : "attention") : "generic") << "\"";
    o << ",\"kernel\":\"" << s.kernel << "\",\"total\":" << s.total << ",\"coop\":" << s.coop;
    if (s.kind == Stage::Gemm) {
      o << ",\"m\":" << s.gemm.m.extent << ",\"n\":" << s.gemm.n.extent << ",\"k\":" << s.gemm.k.extent;
      int64_t b = 1;
      for (auto& d : s.gemm.batch) b *= d.extent;
      o << ",\"batch\":" << b << ",\"a_kmajor\":" << (s.gemm.a_kmajor ? 1 : 0) << ",\"b_kmajor\":" << (s.gemm.b_kmajor ? 1 : 0)
        << ",\"accumulate\":" << (s.gemm.accumulate ? 1 : 0) << ",\"flops\":" << s.gemm.flops();
    }
    if (s.kind == Stage::Attn) {
      const AttnPlan& a = s.attn;
      // both contractions: queries x keys x head dimension, twice
      o << ",\"queries\":" << a.S << ",\"keys\":" << a.T << ",\"head_dim\":" << a.E << ",\"batch\":" << a.B0 * a.B1
        << ",\"flops\":" << 4.0 * (double)(a.B0 * a.B1) * (double)a.S * (double)a.T * (double)a.E;
    }
    if (s.kind != Stage::Memset) {
      // bytes of every node the stage touches, each counted once: the stage's algorithmic traffic
      long long bytes = 0;
      for (auto& a : s.args)
        if (a.kind == KArg::Node) bytes += prog.tn(a.tn).bytes();
      if (s.kind == Stage::Gemm) bytes += prog.tn(s.gemm.a_tn).bytes() + prog.tn(s.gemm.b_tn).bytes();
      if (s.kind == Stage::Attn) bytes += prog.tn(s.attn.q_tn).bytes() + prog.tn(s.attn.k_tn).bytes() + prog.tn(s.attn.v_tn).bytes();
      o << ",\"bytes\":" << bytes;
    } else {
      o << ",\"bytes\":" << prog.tn(s.memset_tn).bytes();
    }
    o << ",\"note\":\"" << s.note << "\"}";
  }
  o << "]}";
  return o.str();
}

namespace {

// What generic_stage knows about a stage before its kernel text is written.
// First statements of every generated kernel: let the next kernel in the stream be placed, then
// wait until the grids before this one have completed and their writes are visible.
static const char* kGridEntry =
    "  asm volatile(\"griddepcontrol.launch_dependents;\");\n  asm volatile(\"griddepcontrol.wait;\" ::: \"memory\");\n";

struct Piece {
  bool fusable = false;
  std::string decomp, body_text;
  std::set<int> used, written;
  bool uses_merge = false;
  // row fusion: the outermost parallel loop ("row") and the work of one of its iterations
  StmtP body;
  std::string row_sym;
  int64_t rows = 0, per_row = 0;
  // warp-per-row fusion: the stage's parallel loops, whether a warp cooperates on each output
  // element (its reductions are warp-wide), whether a thread takes pairs of the innermost loop
  StmtP any_body;
  std::vector<LoopDim> par;
  int coop = 0;
  bool pairs = false;
  int64_t ser_work = 1;
  std::vector<int> staged;   // small read-only nodes the kernel first copies into shared memory
  std::string alone;         // the body's text in a kernel of its own, where it differs
  std::string whole;         // the kernel's body where it is not the grid-stride loop over the stage's iterations
  // a sum kept in `b200_self` over the serial loops (`t[p] := t[p] + term`): its parts, so that several
  // lanes may share one sum
  bool sum = false;
  std::string self_type, self_init, zero, inner, after;
  std::vector<LoopDim> ser;
};

struct Builder {
  Code& code;
  const CompileOptions& opt;
  std::ostringstream src;
  int next_kernel = 0;
  int cur_origin = -1;             // index of the top-level statement being planned
  std::map<size_t, Piece> pieces;  // by index into code.stages
  bool pairs_here() const { return opt.enable_pairs && !opt.no_pairs_at.count(cur_origin); }
  bool gemm_at(size_t i) const { return opt.enable_gemm && !opt.no_gemm_at.count((int)i); }

  std::string kernel_name() { return code.prog.name + "_s" + std::to_string(next_kernel++); }

  void emit_params(std::ostringstream& o, Stage& st, const Emitter& em, const std::set<int>& written) {
    // parameters in node declaration order, then the static-index table, then the merge buffer
    bool first = true;
    for (auto& t : code.prog.tnodes) {
      if (!em.used_nodes.count(t.id)) continue;
      if (t.mode == Mode::Virtual) continue;
      if (!first) o << ", ";
      first = false;
      const bool ro = !written.count(t.id);
      o << (ro ? "const " : "") << Emitter::ctype(t.prec) << "* " << (ro ? "__restrict__ " : "") << t.ident;
      st.args.push_back({KArg::Node, t.id});
    }
    if (em.uses_statics) {
      if (!first) o << ", ";
      first = false;
      o << "const unsigned int* __restrict__ b200_statics";
      st.args.push_back({KArg::Statics, -1});
    }
    if (em.uses_merge) {
      if (!first) o << ", ";
      first = false;
      o << "const " << Emitter::ctype(code.prog.tn(code.prog.merge_node).prec) << "* __restrict__ merge_buffer";
      st.args.push_back({KArg::Merge, -1});
    }
  }

  std::string static_prologue(const std::string& body_text, Emitter& em, int ind) {
    // static index symbols are read from the table the launcher fills
    std::string out;
    for (size_t i = 0; i < code.prog.statics.size(); ++i) {
      const std::string& s = code.prog.statics[i].sym;
      // whole-word search
      size_t p = 0;
      bool found = false;
      while ((p = body_text.find(s, p)) != std::string::npos) {
        auto isid = [](char c) { return isalnum((unsigned char)c) || c == '_'; };
        bool l = p == 0 || !isid(body_text[p - 1]);
        bool r = p + s.size() >= body_text.size() || !isid(body_text[p + s.size()]);
        if (l && r) { found = true; break; }
        p += s.size();
      }
      if (found) {
        out += std::string((size_t)ind, ' ') + "const unsigned int " + s + " = b200_statics[" + std::to_string(i) + "];\n";
        em.uses_statics = true;
      }
    }
    return out;
  }

  // Cooperative reduction: the stage's assignment holds Local_scope reductions
  // `v := neutral; for k1 { for k2 .. { v := v (+|max|min) f(k..) } }`.  A group of threads (a
  // warp, or a whole block when there are few outputs and much to reduce) strides over the
  // flattened reduction space of one output element and combines its partial results.
  // From here on a single output's sum is spread over many blocks.
  static constexpr int64_t kGridSum = 32768;
  CoopInfo find_coop(const Stmt& body, int64_t par_total) {
    CoopInfo ci;
    if (!opt.enable_coop) return ci;
    if (body.kind != Stmt::Set) return ci;
    std::vector<const Scalar*> scopes;
    bool nested = false;
    std::function<void(const Scalar&, int)> rec = [&](const Scalar& e, int depth) {
      if (e.kind == Scalar::LocalScope) {
        if (depth > 0) nested = true;
        scopes.push_back(&e);
        walk_stmt(*e.body, [&](const Scalar& x) { if (x.kind == Scalar::LocalScope) nested = true; }, [](const Stmt&) {});
        return;
      }
      for (auto& a : e.args) rec(*a.s, depth);
    };
    rec(*body.value, 0);
    if (scopes.empty() || nested) return ci;
    int64_t extent = -1;
    for (auto* sc : scopes) {
      const Stmt& b = *sc->body;
      const Stmt* loop = nullptr;
      const Stmt* init = nullptr;
      if (b.kind == Stmt::For) loop = &b;
      else if (b.kind == Stmt::Seq && b.items.size() == 2 && b.items[0]->kind == Stmt::SetLocal && b.items[1]->kind == Stmt::For) {
        init = b.items[0].get();
        loop = b.items[1].get();
      } else return CoopInfo{};
      if (init && (init->scope_id != sc->scope_id || init->value->kind != Scalar::Const)) return CoopInfo{};
      int64_t ext = 1;
      const Stmt* inner = loop;
      while (inner->kind == Stmt::For) {
        ext *= inner->to - inner->from + 1;
        inner = inner->body.get();
      }
      std::string op;
      if (!accum_form(*inner, sc->scope_id, sc->tn, &op)) return CoopInfo{};
      Prec p = code.prog.tn(sc->tn).prec;
      if (p != Prec::Single && !(p == Prec::Double && op == "add")) return CoopInfo{};
      // the initial value must be the neutral element of the combine
      double want = op == "add" ? 0.0 : (op == "max" ? -INFINITY : INFINITY);
      if (init && init->value->cval != want) return CoopInfo{};
      if (!init && op != "add") return CoopInfo{};
      if (extent < 0) extent = ext;
      else if (ext != extent) return CoopInfo{};
      ci.scopes.push_back({sc->scope_id, op});
    }
    if (extent < 32) return CoopInfo{};
    ci.extent = extent;
    ci.sym = "*";
    // few outputs and a long reduction: a whole block per output element
    // (a single one, a loss, from 256 on: one warp took 8 us for 2130 terms)
    ci.width = (par_total <= 256 && extent >= 4096) || (par_total == 1 && extent >= 256) ? 1024 : 32;
    // a single output fed by a very long reduction: many blocks write partial results to
    // scratch and a second, single-block kernel combines them
    if (par_total == 1 && extent >= kGridSum) {
      ci.width = 1024;
      ci.grid_blocks = (int)std::min<int64_t>(296, (extent + 1023) / 1024);
    }
    return ci;
  }

  // Grid-wide reduction of a single output element in one launch.  Every block reduces a strided
  // slice of each Local_scope's flattened loop space and writes one partial per scope to
  // scratch[scope_index * blocks + block]; the block that takes the last ticket of a counter in
  // scratch (zero at link time, reset here) then combines the partials in block order -- a fixed
  // order, so the result does not depend on scheduling -- and evaluates the assignment.
  void grid_reduce_stage(const StmtP& body, const CoopInfo& ci) {
    const Stmt& set = *body;
    const Tnode& t = code.prog.tn(set.tn);
    const int G = ci.grid_blocks;
    const size_t scratch_off = code.reduce_scratch_bytes;
    const size_t counter_off = (size_t)G * ci.scopes.size() * 8;
    code.reduce_scratch_bytes += counter_off + 8;
    code.reduce_scratch_bytes = (code.reduce_scratch_bytes + 255) & ~(size_t)255;

    Stage a;
    a.kind = Stage::Generic;
    a.kernel = kernel_name();
    a.total = 1;
    a.block = 1024;
    a.coop = 1024;
    a.grid_override = G;

    Emitter ea(code.prog), eb(code.prog);
    ea.large_models = eb.large_models = opt.large_models;
    std::string pass1, pass2;
    int si = 0;
    std::function<void(const Scalar&)> rec = [&](const Scalar& e) {
      if (e.kind == Scalar::LocalScope) {
        std::string op;
        for (auto& s : ci.scopes)
          if (s.first == e.scope_id) op = s.second;
        Prec p = code.prog.tn(e.tn).prec;
        const Stmt& sb = *e.body;
        const Stmt* loop = sb.kind == Stmt::For ? &sb : sb.items[1].get();
        std::vector<LoopDim> red;
        const Stmt* inner = loop;
        while (inner->kind == Stmt::For) {
          red.push_back({inner->index, inner->from, inner->to});
          inner = inner->body.get();
        }
        int64_t total = 1;
        for (auto& d : red) total *= d.extent();
        const std::string name = ea.scope_name(e.scope_id, e.tn);
        const std::string T = Emitter::ctype(p);
        const double neutral = op == "add" ? 0.0 : (op == "max" ? -INFINITY : INFINITY);
        const std::string fn = op == "add" ? "sum" : op;
        const std::string at = "(b200_partials + " + std::to_string((size_t)si * G * 8) + "))";
        const std::string slot = "((" + T + "*)" + at, vslot = "((volatile " + T + "*)" + at;
        pass1 += "  {\n    " + T + " " + name + " = " + ea.constant(neutral, p) + ";\n";
        // Every thread takes the same whole number of steps and at most one more, so that the loads of eight steps are
        // under way together (a step after the other cost their latency each: the 2 M squared differences of 64 images
        // of 32 x 32 x 32, 10.0 us -> 8.5, most of it cold reads).
        const bool narrow = total < (1ll << 31);
        const std::string IT = narrow ? "unsigned int" : "unsigned long long", SUF = narrow ? "u" : "ull";
        const int64_t stride = (int64_t)G * 1024, whole = total / stride;
        std::string step;
        std::string rem = "b200_l";
        for (size_t i = red.size(); i-- > 0;) {
          const LoopDim& d = red[i];
          std::string ext = std::to_string(d.extent()) + SUF;
          std::string val = i == 0 ? rem : "(" + rem + " % " + ext + ")";
          step += "      const unsigned int " + d.sym + " = (unsigned int)" + val +
                  (d.from ? " + " + std::to_string(d.from) : std::string()) + ";\n";
          if (i != 0) {
            std::string nr = "b200_q" + std::to_string(i);
            step += "      const " + IT + " " + nr + " = " + rem + " / " + ext + ";\n";
            rem = nr;
          }
        }
        step += ea.stmt(*inner, 6);
        pass1 += "    const " + IT + " b200_first = blockIdx.x * 1024u + threadIdx.x;\n#pragma unroll 8\n    for (unsigned int b200_k = 0; b200_k < " +
                 std::to_string(whole) + "u; ++b200_k) {\n      const " + IT + " b200_l = b200_first + b200_k * " + std::to_string(stride) + SUF + ";\n" + step + "    }\n";
        if (total % stride)
          pass1 += "    if (b200_first < " + std::to_string(total % stride) + SUF + ") {\n      const " + IT + " b200_l = b200_first + " +
                   std::to_string(whole * stride) + SUF + ";\n" + step + "    }\n";
        pass1 += "    " + name + " = b200_block_" + fn + "(" + name + ", b200_red);\n";
        pass1 += "    if (threadIdx.x == 0) " + slot + "[blockIdx.x] = " + name + ";\n  }\n";
        // combine: the partials in block order
        pass2 += "  " + T + " " + name + " = " + eb.constant(neutral, p) + ";\n";
        pass2 += "  for (unsigned int b200_i = threadIdx.x; b200_i < " + std::to_string(G) + "u; b200_i += blockDim.x) " + name + " = ";
        if (op == "add") pass2 += name + " + " + vslot + "[b200_i];\n";
        else pass2 += std::string("f") + op + (p == Prec::Double ? "(" : "f(") + name + ", " + vslot + "[b200_i]);\n";
        pass2 += "  " + name + " = b200_block_" + fn + "(" + name + ", b200_red);\n";
        eb.scope_subst[e.scope_id] = name;
        ++si;
        return;
      }
      for (auto& x : e.args) rec(*x.s);
    };
    rec(*set.value);
    Emitter::Res v = eb.scalar(t.prec, *set.value);
    eb.used_nodes.insert(set.tn);
    pass2 += "  if (threadIdx.x == 0) {\n    " + t.ident + "[" + eb.offset(set.idcs, t.dims) + "] = " + Emitter::store_wrap(t.prec, v.expr) +
             ";\n    *b200_ticket = 0u;\n  }\n";

    std::set<int> written = {set.tn};
    Emitter eu(code.prog);
    eu.used_nodes = ea.used_nodes;
    eu.used_nodes.insert(eb.used_nodes.begin(), eb.used_nodes.end());
    eu.uses_merge = ea.uses_merge || eb.uses_merge;
    std::ostringstream ka;
    std::string statics = static_prologue(pass1 + pass2, eu, 2);
    ka << "extern \"C\" __global__ void __launch_bounds__(1024) " << a.kernel << "(";
    emit_params(ka, a, eu, written);
    ka << (a.args.empty() ? "" : ", ") << "unsigned char* b200_partials) {\n" << kGridEntry << "  __shared__ double b200_red[32];\n"
       << "  __shared__ unsigned int b200_last;\n  unsigned int* b200_ticket = (unsigned int*)(b200_partials + " << counter_off << ");\n"
       << statics << pass1
       << "  __threadfence();\n  __syncthreads();\n"
       << "  if (threadIdx.x == 0) b200_last = atomicAdd(b200_ticket, 1u) == gridDim.x - 1u ? 1u : 0u;\n"
       << "  __syncthreads();\n  if (!b200_last) return;\n  __threadfence();\n"
       << pass2 << "}\n\n";
    a.args.push_back({KArg::Scratch, (int)scratch_off});
    src << ka.str();
    a.note = "grid-wide reduction (" + std::to_string(G) + " blocks, the last one combines)";
    a.writes = {set.tn};
    code.stages.push_back(a);
  }

  // Accumulation whose reduced loops are OUTSIDE the output loops (back-propagation keeps the
  // forward loop order: `for b { for o { g[o] := g[o] + dz[b, o] } }`, or the fma form with two
  // factors).  A block owns up to 128 neighbouring outputs (or pairs) and splits the flattened serial
  // loop space over its other threads; partial sums meet through shuffles and shared memory.
  // dW of a 10-class output layer over 8192 rows and 1024 inputs: 33 us with one pair per thread, whose ten
  // factors were then loaded for two products each.
  bool ser_split_stage(Stage st, const Stmt& set) {
    if (set.kind != Stmt::Set) return false;
    const Tnode& t = code.prog.tn(set.tn);
    if (t.prec != Prec::Single && t.prec != Prec::Double) return false;
    int64_t ser_total = 1;
    for (auto& d : st.ser) ser_total *= d.extent();
    if (ser_total < 256) return false;
    // the written position must not move with a serial loop (an affine output position
    // `stride * o + k` of a convolution's input gradient does): then this is no reduction
    for (auto& d : st.ser)
      for (auto& ix : set.idcs)
        if (ix.uses(d.sym)) return false;
    const Scalar& v = *set.value;
    auto is_self = [&](const Scalar& e) {
      if (e.kind != Scalar::Get || e.tn != set.tn || e.idcs.size() != set.idcs.size()) return false;
      for (size_t i = 0; i < e.idcs.size(); ++i)
        if (e.idcs[i].kind != set.idcs[i].kind || e.idcs[i].sym != set.idcs[i].sym || e.idcs[i].fixed != set.idcs[i].fixed ||
            e.idcs[i].terms != set.idcs[i].terms)
          return false;
      return true;
    };
    auto reads_node = [&](const Scalar& e) {
      bool m = false;
      walk_scalar(e, [&](const Scalar& x) {
        if ((x.kind == Scalar::Get || x.kind == Scalar::GetDyn) && x.tn == set.tn) m = true;
        if (x.kind == Scalar::LocalScope) m = true;  // keep this path to plain terms
      }, [](const Stmt&) {});
      return m;
    };
    const Scalar *fa = nullptr, *fb = nullptr, *term = nullptr;
    if (v.kind == Scalar::Tern && v.op == "fma" && is_self(*v.args[2].s)) {
      fa = v.args[0].s.get();
      fb = v.args[1].s.get();
      if (reads_node(*fa) || reads_node(*fb)) return false;
    } else if (v.kind == Scalar::Bin && v.op == "add") {
      if (is_self(*v.args[0].s)) term = v.args[1].s.get();
      else if (is_self(*v.args[1].s)) term = v.args[0].s.get();
      if (!term || reads_node(*term)) return false;
    } else {
      return false;
    }
    Emitter em(code.prog);
    em.large_models = opt.large_models;
    // Pairs: a thread owns two neighbouring outputs along the innermost output loop when that loop
    // runs along the last axis of the fp32 node; the factors are then read as 4- and 8-byte words.
    bool pairs = false;
    if (pairs_here() && t.prec == Prec::Single && !st.par.empty() && !set.idcs.empty()) {
      const LoopDim& p = st.par.back();
      bool ok = p.from == 0 && p.extent() % 2 == 0 && set.idcs.back().kind == Index::Iter && set.idcs.back().sym == p.sym &&
                t.dims.back() % 2 == 0;
      for (size_t a = 0; ok && a + 1 < set.idcs.size(); ++a)
        if (set.idcs[a].uses(p.sym)) ok = false;
      if (ok && (term ? em.pair_supported(*term) : em.pair_supported(*fa) && em.pair_supported(*fb))) {
        pairs = true;
        em.pair = true;
        em.pair_sym = p.sym;
        em.pair_vector_loads = true;
      }
    }
    const std::string T = pairs ? "b200_f2" : Emitter::ctype(t.prec);
    const std::string zero = pairs ? "b200_f2{0.0f, 0.0f}" : "0";
    std::string step;
    if (pairs) {
      std::string pre;
      if (term) {
        const std::string v = em.pair_scalar(t.prec, *term, pre);
        step = "{\n" + pre + "          b200_acc = b200_f2{b200_acc.x + " + v + ".x, b200_acc.y + " + v + ".y};\n          }";
      } else {
        const std::string a = em.pair_scalar(t.prec, *fa, pre), b = em.pair_scalar(t.prec, *fb, pre);
        step = "{\n" + pre + "          b200_acc = b200_f2{fmaf(" + a + ".x, " + b + ".x, b200_acc.x), fmaf(" + a + ".y, " + b +
               ".y, b200_acc.y)};\n          }";
      }
      st.min_align = 8;
    } else if (term) {
      Emitter::Res r = em.scalar(t.prec, *term);
      if (!r.defs.empty()) return false;
      step = "b200_acc = b200_acc + " + r.expr + ";";
    } else {
      Emitter::Res ra = em.scalar(t.prec, *fa), rb = em.scalar(t.prec, *fb);
      if (!ra.defs.empty() || !rb.defs.empty()) return false;
      step = std::string("b200_acc = ") + (t.prec == Prec::Double ? "fma(" : "fmaf(") + ra.expr + ", " + rb.expr + ", b200_acc);";
    }
    em.used_nodes.insert(set.tn);
    for (auto& d : st.par) if (d.from != 0) return false;
    for (auto& d : st.ser) if (d.from != 0) return false;
    // Register tiling: a short outermost output loop (the 10 classes of `dW[o, i] += dz[b, o] * h[b, i]`)
    // stays inside the thread, which then reads the other factor once for all of its values.
    const bool tiled = !term && st.par.size() >= 2 && st.par[0].extent() <= 16;
    const int64_t e0 = tiled ? st.par[0].extent() : 1;
    const size_t first_par = tiled ? 1 : 0;
    const int64_t outputs = st.total / e0 / (pairs ? 2 : 1);   // output elements (or pairs) spread over the columns
    // A block is 32 lanes x BY rows of threads.  CW lanes take neighbouring outputs, Q of them each, CW
    // apart (what does not depend on the output -- the other factor of every tiled value -- is then loaded
    // once for Q outputs); the 32 / CW lane groups and the BY rows share out the serial loop space.  Few
    // outputs (the 24 channels of a convolution's bias) thus keep whole warps busy.
    int64_t CW = 1;
    while (CW < 32 && CW < outputs) CW *= 2;
    // (at most 80 accumulator registers per thread)
    const int64_t q_max = std::max<int64_t>(1, 80 / (e0 * (pairs ? 2 : 1)));
    const int64_t Q = outputs >= 4 * CW && q_max >= 4 ? 4 : (outputs >= 2 * CW && q_max >= 2 ? 2 : 1);
    const int64_t XR = 32 / CW, BY = tiled ? 16 : 32, SUBS = BY * XR;
    std::string decomp, sdecomp;
    {
      std::string rem = "b200_g";
      for (size_t i = st.par.size(); i-- > first_par;) {
        const LoopDim& d = st.par[i];
        const bool pair_dim = pairs && i + 1 == st.par.size();
        std::string ext = std::to_string(pair_dim ? d.extent() / 2 : d.extent()) + "u";
        decomp += "          const unsigned int " + d.sym + " = " + (pair_dim ? "2u * " : "") +
                  (i == first_par ? rem : "(" + rem + " % " + ext + ")") + ";\n";
        if (i != first_par) {
          decomp += "          const unsigned int b200_r" + std::to_string(i) + " = " + rem + " / " + ext + ";\n";
          rem = "b200_r" + std::to_string(i);
        }
      }
      rem = "b200_l";
      for (size_t i = st.ser.size(); i-- > 0;) {
        const LoopDim& d = st.ser[i];
        std::string ext = std::to_string(d.extent()) + "u";
        sdecomp += "        const unsigned int " + d.sym + " = " + (i == 0 ? rem : "(" + rem + " % " + ext + ")") + ";\n";
        if (i != 0) {
          sdecomp += "        const unsigned int b200_q" + std::to_string(i) + " = " + rem + " / " + ext + ";\n";
          rem = "b200_q" + std::to_string(i);
        }
      }
    }
    if (st.total >= (1ll << 31) || ser_total >= (1ll << 31)) return false;   // (positions are counted in 32 bits)
    const std::string off = em.offset(set.idcs, t.dims);
    std::string text = decomp + sdecomp + step + off;
    std::string statics = static_prologue(text, em, 2);
    // Few output groups leave most SMs idle: the serial loop space is then also cut into Z slices,
    // one block per (group, slice), and the slices meet in the output through atomic adds (their
    // order is not fixed; the node is fp32 or fp64 and already holds the value being added to).
    const int64_t groups = (outputs + CW * Q - 1) / (CW * Q);
    int64_t Z = 1;
    if (groups < 2 * 148) Z = std::max<int64_t>(1, std::min<int64_t>(((tiled ? 148 : 2 * 148) + groups - 1) / groups, ser_total / std::max<int64_t>(2 * SUBS, 128)));
    st.block = 32;
    st.block_y = (int)BY;
    st.coop = 32;  // several threads per output element
    st.grid_override = (int)std::min<int64_t>(groups * Z, 148 * 8);
    std::set<int> written = {set.tn};
    const std::string o_sym = tiled ? st.par[0].sym : std::string();
    const std::string E0 = std::to_string(e0), QS = std::to_string(Q), CWS = std::to_string(CW);
    auto sum_of = [&](const std::string& a, const std::string& b) {
      return pairs ? "b200_f2{" + a + ".x + " + b + ".x, " + a + ".y + " + b + ".y}" : a + " + " + b;
    };
    // Values of the tiled loop that are combined at a time, between two barriers: as many as 40 KB of partials hold.  (One at
    // a time, ten outputs over 500 rows spent most of their 10 us there, ten times two barriers and a chain of 16 sums.  A
    // half-moons step of 257 points with 9 hidden units 24.7 us so, now 22.7; 8192 rows unchanged.)
    const int64_t per = std::max<int64_t>(1, std::min<int64_t>(e0, 40960 / (BY * Q * CW * (pairs ? 8 : prec_bytes(t.prec)))));
    std::ostringstream k;
    k << "extern \"C\" __global__ void __launch_bounds__(" << 32 * BY << ") " << st.kernel << "(";
    emit_params(k, st, em, written);
    k << ") {\n" << kGridEntry << statics << "  __shared__ " << T << " b200_part[" << BY << "][" << per * Q * CW + 1 << "];\n"
      << "  const unsigned int b200_c = threadIdx.x % " << CWS << "u, b200_sub = threadIdx.y * " << XR << "u + threadIdx.x / " << CWS << "u;\n"
      << "  for (unsigned int b200_u = blockIdx.x; b200_u < " << groups * Z << "u; b200_u += gridDim.x) {\n"
      << "    const unsigned int b200_g0 = (b200_u % " << groups << "u) * " << Q * CW << "u, b200_z = b200_u / " << groups << "u;\n"
      << "    const unsigned int b200_l0 = (unsigned int)(b200_z * " << ser_total << "ull / " << Z << "ull), b200_l1 = (unsigned int)((b200_z + 1ull) * "
      << ser_total << "ull / " << Z << "ull);\n"
      << "    " << T << " b200_accs[" << QS << "][" << E0 << "];\n#pragma unroll\n    for (int b200_q = 0; b200_q < " << QS
      << "; ++b200_q)\n#pragma unroll\n      for (int b200_o = 0; b200_o < " << E0 << "; ++b200_o) b200_accs[b200_q][b200_o] = " << zero << ";\n"
      << "#pragma unroll " << (Q * e0 <= 8 ? 4 : (Q * e0 <= 16 ? 2 : 1)) << "\n      for (unsigned int b200_l = b200_l0 + b200_sub; b200_l < b200_l1; b200_l += " << SUBS << "u) {\n" << sdecomp
      << "#pragma unroll\n        for (unsigned int b200_q = 0; b200_q < " << QS << "u; ++b200_q) {\n"
      // (columns past the end repeat the last one; nothing of them is added to the output)
      << "          const unsigned int b200_g = min(b200_g0 + b200_q * " << CWS << "u + b200_c, " << outputs - 1 << "u);\n" << decomp
      << "#pragma unroll\n          for (unsigned int " << (tiled ? o_sym : std::string("b200_one")) << " = 0; " << (tiled ? o_sym : std::string("b200_one")) << " < " << E0 << "u; ++"
      << (tiled ? o_sym : std::string("b200_one")) << ") {\n"
      << "            " << T << " b200_acc = b200_accs[b200_q][" << (tiled ? o_sym : std::string("0")) << "];\n            " << step << "\n            b200_accs[b200_q]["
      << (tiled ? o_sym : std::string("0")) << "] = b200_acc;\n          }\n        }\n      }\n";
    // combine: lane groups by shuffles, then the BY rows through shared memory, `per` values of the tiled loop at a time
    k << "#pragma unroll\n    for (unsigned int b200_o0 = 0; b200_o0 < " << E0 << "u; b200_o0 += " << per << "u) {\n"
      << "#pragma unroll\n      for (unsigned int b200_oo = 0; b200_oo < " << per << "u; ++b200_oo) {\n        if (b200_o0 + b200_oo >= " << E0 << "u) break;\n"
      << "#pragma unroll\n      for (int b200_q = 0; b200_q < " << QS << "; ++b200_q) {\n        " << T << " b200_acc = b200_accs[b200_q][b200_o0 + b200_oo];\n";
    if (XR > 1) {
      k << "#pragma unroll\n        for (unsigned int b200_s = " << CWS << "u; b200_s < 32u; b200_s <<= 1) {\n";
      if (pairs)
        k << "          const " << T << " b200_w = {__shfl_xor_sync(0xffffffffu, b200_acc.x, b200_s), __shfl_xor_sync(0xffffffffu, b200_acc.y, b200_s)};\n";
      else
        k << "          const " << T << " b200_w = __shfl_xor_sync(0xffffffffu, b200_acc, b200_s);\n";
      k << "          b200_acc = " << sum_of("b200_acc", "b200_w") << ";\n        }\n";
    }
    k << "        if (threadIdx.x < " << CWS << "u) b200_part[threadIdx.y][(b200_oo * " << QS << " + b200_q) * " << CWS << " + b200_c] = b200_acc;\n      }\n      }\n      __syncthreads();\n"
      << "      for (unsigned int b200_i = threadIdx.y * 32u + threadIdx.x; b200_i < " << per * Q * CW << "u; b200_i += " << 32 * BY << "u) {\n"
      << "        const unsigned int b200_g = b200_g0 + b200_i % " << Q * CW << "u, " << (tiled ? o_sym : std::string("b200_one")) << " = b200_o0 + b200_i / " << Q * CW
      << "u;\n        if (b200_g < " << outputs << "u && " << (tiled ? o_sym : std::string("b200_one")) << " < " << E0 << "u) {\n" << decomp
      << "          " << T << " b200_s = b200_part[0][b200_i];\n#pragma unroll\n          for (int b200_y = 1; b200_y < " << BY << "; ++b200_y) b200_s = "
      << sum_of("b200_s", "b200_part[b200_y][b200_i]") << ";\n";
    if (pairs) {
      if (Z > 1) k << "          b200_red2(" << t.ident << " + (" << off << "), b200_s.x, b200_s.y);\n";
      else k << "          " << t.ident << "[" << off << "] = " << t.ident << "[" << off << "] + b200_s.x;\n          " << t.ident << "[(" << off
             << ") + 1] = " << t.ident << "[(" << off << ") + 1] + b200_s.y;\n";
    } else {
      if (Z > 1) k << "          atomicAdd(&" << t.ident << "[" << off << "], b200_s);\n";
      else k << "          " << t.ident << "[" << off << "] = " << t.ident << "[" << off << "] + b200_s;\n";
    }
    k << "        }\n      }\n      __syncthreads();\n    }\n  }\n}\n\n";
    src << k.str();
    st.note = "par=" + std::to_string(st.par.size()) + " ser=" + std::to_string(st.ser.size()) + " serial loops split over a 32x" + std::to_string(BY) + " block" +
              (Z > 1 ? ", " + std::to_string(Z) + " slices per output group (atomic adds)" : std::string()) +
              (tiled ? ", outer loop of " + E0 + " kept in registers" : std::string()) + (pairs ? ", pairs" : std::string());
    st.writes = {set.tn};
    code.stages.push_back(st);
    return true;
  }

  // Does `set` write every element of its node exactly once over `loops` (each axis a distinct
  // loop symbol running over the whole axis, or a fixed 0 on an axis of extent 1)?
  bool covers_node(const Stmt& set, const std::vector<LoopDim>& loops) {
    const Tnode& t = code.prog.tn(set.tn);
    if (set.kind != Stmt::Set || set.vec_len > 0 || set.idcs.size() != t.dims.size()) return false;
    std::set<std::string> seen;
    for (size_t a = 0; a < set.idcs.size(); ++a) {
      const Index& ix = set.idcs[a];
      if (ix.kind == Index::Fixed) {
        if (ix.fixed != 0 || t.dims[a] != 1) return false;
        continue;
      }
      if (ix.kind != Index::Iter || !seen.insert(ix.sym).second) return false;
      bool found = false;
      for (auto& d : loops)
        if (d.sym == ix.sym && d.from == 0 && d.extent() == t.dims[a]) found = true;
      if (!found) return false;
    }
    return true;
  }

  // The part of its node that a stage overwrites without reading any of it, an interval per axis (empty: not known).
  using Box = std::vector<std::pair<int64_t, int64_t>>;
  Box written_box(const Piece& pc) {
    if (!pc.any_body || pc.any_body->kind != Stmt::Set || pc.any_body->vec_len > 0 || pc.sum) return {};
    const Stmt& set = *pc.any_body;
    bool reads = false;
    walk_scalar(*set.value, [&](const Scalar& e) {
      if ((e.kind == Scalar::Get || e.kind == Scalar::GetDyn) && e.tn == set.tn) reads = true;
    }, [](const Stmt&) {});
    if (reads) return {};
    Box box;
    for (auto& ix : set.idcs) {
      int64_t lo = ix.kind == Index::Iter ? 0 : ix.fixed, hi = lo;
      auto add = [&](int64_t k, const std::string& sym) {
        for (auto* loops : {&pc.par, &pc.ser})
          for (auto& d : *loops)
            if (d.sym == sym) {
              const int64_t a = k * d.from, b = k * (d.from + d.extent() - 1);
              lo += std::min(a, b);
              hi += std::max(a, b);
              return true;
            }
        return false;
      };
      bool known = ix.kind != Index::SubAxis;
      if (ix.kind == Index::Iter) known = add(1, ix.sym);
      if (ix.kind == Index::Affine)
        for (auto& t : ix.terms) known = known && add(t.first, t.second);
      if (!known) return {};
      box.push_back({lo, hi});
    }
    return box;
  }
  static bool apart(const Box& a, const Box& b) {
    for (size_t i = 0; i < a.size() && i < b.size(); ++i)
      if (a[i].second < b[i].first || b[i].second < a[i].first) return true;
    return false;
  }

  // A single-precision sum of products whose one factor is a small table (the kernel of a convolution, at most
  // 40 KB) and whose other factor is looked up at moving positions.  The table lies in shared memory with its
  // outputs next to one another; a thread sums T outputs at P neighbouring positions, so that T table entries and
  // P looked-up values, T / 4 + P loads, serve T P multiplications.  Sums run in the order of the loops.
  // On the tensor cores the same sum would need three products of two-part operands, and a copy of every
  // window in memory: 64 images of 32 x 32 x 3, 32 outputs of 3 x 3: 14.6 us, 6 us here.
  // T P is as large as leaves 12 warps per SM; below four outputs per thread the plain kernel is as good.
  bool table_stage(const std::vector<LoopDim>& nest, const StmtP& body) {
    if (opt.bounds || body->kind != Stmt::Set || body->vec_len > 0 || nest.size() < 2) return false;
    const Tnode& out = code.prog.tn(body->tn);
    if (out.prec != Prec::Single) return false;
    for (auto& d : nest)
      if (d.extent() <= 0 || !parallel_safe(d.sym, *body)) return false;
    // the one local sum of the assigned value
    const Scalar* scope = nullptr;
    int scopes = 0;
    bool plain = true;
    walk_scalar(*body->value, [&](const Scalar& e) {
      if (e.kind == Scalar::LocalScope) { scope = &e; ++scopes; }
      if (e.kind == Scalar::GetDyn || e.kind == Scalar::GetMerge || (e.kind == Scalar::Get && e.tn == body->tn)) plain = false;
    }, [](const Stmt&) {});
    if (scopes != 1 || !plain || code.prog.tn(scope->tn).prec != Prec::Single) return false;
    const Stmt* at = scope->body.get();
    if (!at || at->kind != Stmt::Seq || at->items.size() != 2) return false;
    const Stmt* init = at->items[0].get();
    if (init->kind != Stmt::SetLocal || init->scope_id != scope->scope_id || init->value->kind != Scalar::Const) return false;
    std::vector<LoopDim> red;
    for (at = at->items[1].get(); at->kind == Stmt::For; at = at->body.get()) {
      LoopDim d;
      d.sym = at->index; d.from = at->from; d.to = at->to;
      if (d.extent() <= 0) return false;
      red.push_back(d);
      if (!at->body) return false;
    }
    if (red.empty() || at->kind != Stmt::SetLocal || at->scope_id != scope->scope_id) return false;
    const Scalar& step = *at->value;
    if (step.kind != Scalar::Tern || step.op != "fma" || step.args[2].s->kind != Scalar::GetLocal || step.args[2].s->scope_id != scope->scope_id) return false;
    const LoopDim& c = nest.back();
    auto uses_sym = [](const Scalar& e, const std::string& sym) {
      for (auto& ix : e.idcs)
        if (ix.uses(sym)) return true;
      return false;
    };
    const Scalar* W = step.args[0].s.get();
    const Scalar* X = step.args[1].s.get();
    for (auto* e : {W, X})
      if (e->kind != Scalar::Get || code.prog.tn(e->tn).prec != Prec::Single || e->tn == body->tn) return false;
    if (!uses_sym(*W, c.sym)) std::swap(W, X);
    if (!uses_sym(*W, c.sym) || uses_sym(*X, c.sym)) return false;
    for (size_t i = 0; i + 1 < nest.size(); ++i)
      if (uses_sym(*W, nest[i].sym)) return false;
    bool moving = false;
    for (auto& ix : X->idcs) moving = moving || ix.kind == Index::Affine;
    for (auto& ix : W->idcs)
      if (ix.kind == Index::SubAxis) return false;
    for (auto& ix : X->idcs)
      if (ix.kind == Index::SubAxis) return false;
    if (!moving) return false;
    int64_t K = 1, outputs = 1;
    for (auto& d : red) K *= d.extent();
    for (auto& d : nest) outputs *= d.extent();
    const LoopDim& w = nest[nest.size() - 2];
    const int64_t C = c.extent();
    int T = 0, P = 0;
    for (auto tp : {std::pair<int, int>{16, 4}, {16, 2}, {8, 4}, {8, 2}, {16, 1}, {8, 1}, {4, 2}, {4, 1}}) {
      const int64_t padded = (C + tp.first - 1) / tp.first * tp.first;
      // (no more than a fifth of the sums for columns that do not exist)
      if (w.extent() % tp.second || padded * 4 > C * 5 || padded * K * 4 > 40960) continue;
      if (outputs / C * (padded / tp.first) / tp.second < 148 * 384) continue;
      T = tp.first;
      P = tp.second;
      break;
    }
    if (!T || outputs >= (1ll << 31)) return false;
    const int64_t Cp = (C + T - 1) / T * T, G = Cp / T, threads = outputs / C * G / P;

    Emitter em(code.prog);
    Emitter::Res wr = em.scalar(Prec::Single, *W), xr = em.scalar(Prec::Single, *X);
    em.scope_subst[scope->scope_id] = "b200_acc[b200_p][b200_q]";
    Emitter::Res vr = em.scalar(Prec::Single, *body->value);
    if (!wr.defs.empty() || !xr.defs.empty() || !vr.defs.empty()) return false;
    em.used_nodes.insert(body->tn);
    auto u = [](int64_t v) { return std::to_string(v) + "u"; };
    auto plus = [&](const LoopDim& d) { return d.from ? " + " + u(d.from) : std::string(); };
    std::ostringstream o;
    o << "  __shared__ __align__(16) float b200_table[" << K * Cp << "];\n"
      << "  for (unsigned int b200_i = threadIdx.x; b200_i < " << u(K * Cp) << "; b200_i += blockDim.x) {\n    const unsigned int b200_c = b200_i % " << u(Cp)
      << ", " << c.sym << " = b200_c" << plus(c) << ";\n    unsigned int b200_k = b200_i / " << u(Cp) << ";\n";
    for (size_t i = red.size(); i-- > 0;) {
      o << "    const unsigned int " << red[i].sym << " = " << (i ? "b200_k % " + u(red[i].extent()) : std::string("b200_k")) << plus(red[i]) << ";\n";
      if (i) o << "    b200_k /= " << u(red[i].extent()) << ";\n";
    }
    o << "    b200_table[b200_i] = b200_c < " << u(C) << " ? " << wr.expr << " : 0.0f;\n  }\n  __syncthreads();\n"
      << "  for (unsigned int b200_g = blockIdx.x * blockDim.x + threadIdx.x; b200_g < " << u(threads) << "; b200_g += gridDim.x * blockDim.x) {\n"
      << "    const unsigned int b200_c0 = b200_g % " << u(G) << " * " << u(T) << ";\n    unsigned int b200_r = b200_g / " << u(G) << ";\n";
    o << "    const unsigned int b200_w0 = b200_r % " << u(w.extent() / P) << " * " << u(P) << plus(w) << ";\n    b200_r /= " << u(w.extent() / P) << ";\n";
    for (size_t i = nest.size() - 2; i-- > 0;) {
      o << "    const unsigned int " << nest[i].sym << " = " << (i ? "b200_r % " + u(nest[i].extent()) : std::string("b200_r")) << plus(nest[i]) << ";\n";
      if (i) o << "    b200_r /= " << u(nest[i].extent()) << ";\n";
    }
    o << "    float b200_acc[" << P << "][" << T << "];\n#pragma unroll\n    for (int b200_p = 0; b200_p < " << P << "; ++b200_p)\n#pragma unroll\n      for (int b200_q = 0; b200_q < "
      << T << "; ++b200_q) b200_acc[b200_p][b200_q] = " << em.constant(init->value->cval, Prec::Single) << ";\n";
    // the innermost loops without jumps, up to 32 steps
    std::vector<bool> flat(red.size(), false);
    int64_t steps = 1;
    for (size_t i = red.size(); i-- > 0 && steps * red[i].extent() <= 32;) {
      steps *= red[i].extent();
      flat[i] = true;
    }
    std::string k = "0u";
    for (size_t i = 0; i < red.size(); ++i) {
      o << (flat[i] ? "#pragma unroll\n" : i + 1 == red.size() ? "#pragma unroll 8\n" : "#pragma unroll 1\n") << "    for (unsigned int " << red[i].sym << " = " << u(red[i].from) << "; " << red[i].sym << " <= " << u(red[i].to)
        << "; ++" << red[i].sym << ") {\n";
      k = "(" + k + " * " + u(red[i].extent()) + " + " + red[i].sym + (red[i].from ? " - " + u(red[i].from) : std::string()) + ")";
    }
    o << "      float b200_w[" << T << "];\n#pragma unroll\n      for (int b200_q = 0; b200_q < " << T << "; b200_q += 4) {\n        const float4 b200_v = *(const float4*)(b200_table + "
      << k << " * " << u(Cp) << " + b200_c0 + b200_q);\n        b200_w[b200_q] = b200_v.x; b200_w[b200_q + 1] = b200_v.y; b200_w[b200_q + 2] = b200_v.z; b200_w[b200_q + 3] = b200_v.w;\n      }\n"
      << "#pragma unroll\n      for (int b200_p = 0; b200_p < " << P << "; ++b200_p) {\n        const unsigned int " << w.sym << " = b200_w0 + b200_p;\n        const float b200_x = " << xr.expr
      << ";\n#pragma unroll\n        for (int b200_q = 0; b200_q < " << T << "; ++b200_q) b200_acc[b200_p][b200_q] = fmaf(b200_w[b200_q], b200_x, b200_acc[b200_p][b200_q]);\n      }\n";
    for (size_t i = 0; i < red.size(); ++i) o << "    }\n";
    o << "#pragma unroll\n    for (int b200_p = 0; b200_p < " << P << "; ++b200_p) {\n      const unsigned int " << w.sym << " = b200_w0 + b200_p;\n      float b200_v[" << T
      << "];\n#pragma unroll\n      for (int b200_q = 0; b200_q < " << T << "; ++b200_q) {\n        b200_v[b200_q] = 0.0f;\n        if (" << (Cp == C ? std::string("true") : "b200_c0 + b200_q < " + u(C)) << ") {\n          const unsigned int " << c.sym << " = b200_c0 + b200_q"
      << plus(c) << ";\n          b200_v[b200_q] = " << vr.expr << ";\n        }\n      }\n";
    Indices first = body->idcs;
    const std::string off = em.offset(first, out.dims);
    const bool unit = !first.empty() && first.back().kind == Index::Iter && first.back().sym == c.sym && C % 4 == 0;
    o << "#pragma unroll\n      for (int b200_q = 0; b200_q < " << T << "; b200_q += " << (unit ? 4 : 1) << ") {\n        const unsigned int " << c.sym << " = b200_c0 + b200_q" << plus(c)
      << ";\n        float* const b200_to = " << out.ident << " + (" << off << ");\n";
    if (unit)
      o << "        if (b200_c0 + b200_q >= " << u(C) << ") break;\n        if (((unsigned long long)b200_to & 15ull) == 0ull) *(float4*)b200_to = make_float4(b200_v[b200_q], b200_v[b200_q + 1], b200_v[b200_q + 2], b200_v[b200_q + 3]);\n"
        << "        else { b200_to[0] = b200_v[b200_q]; b200_to[1] = b200_v[b200_q + 1]; b200_to[2] = b200_v[b200_q + 2]; b200_to[3] = b200_v[b200_q + 3]; }\n";
    else
      o << "        if (b200_c0 + b200_q < " << u(C) << ") *b200_to = b200_v[b200_q];\n";
    o << "      }\n    }\n  }\n";

    Stage st;
    st.kind = Stage::Generic;
    st.kernel = kernel_name();
    st.par = nest;
    st.total = threads;
    st.block = 256;
    st.grid_override = (int)std::min<int64_t>((threads + 255) / 256, 148 * 4);
    st.note = "table of " + std::to_string(K) + " x " + std::to_string(C) + " in shared memory, " + std::to_string(T) + " outputs at " + std::to_string(P) + " positions per thread";
    st.writes = {body->tn};
    Piece pc;
    pc.whole = o.str();
    pc.used = em.used_nodes;
    pc.written = {body->tn};
    pieces[code.stages.size()] = pc;
    code.stages.push_back(st);
    return true;
  }

  // Accumulations at few moving positions, by position.  `t[.., c * o + k, ..] := t[same] + term`: a thread takes one
  // position of t and walks the loops in their order, without the innermost symbol of every moving axis: the position
  // gives that one.  Every position so gets its terms one after the other in the order of the loops, as when a thread
  // walks all of them by itself, and the sums have the same bits from run to run, which atomic adds would not give.
  // The loop that fixes the given symbol covers the iterations that reach the position and no others: threads of a warp, whose
  // positions differ, then walk side by side (with a test in each iteration instead they took turns).
  // A chain of dependent additions with its loads in between bounds it: 16 steps unrolled, blocks of one warp, on as many
  // SMs as there are.  Convolution steps, one thread / atomic adds / by position, us: 1 image of 8 x 8 under 50 kernels of
  // 5 x 5 590 / 15 / 34, 3 of 16 x 16 x 3 under 56 of 3 x 3, stride 2, 645 / 31 / 33, 19 of 9 x 9 under 38, stride 2,
  // 695 / 10.4 / 10.4, 1 of 8 x 8 x 32 under 16 20.7 / 16.6 / 16.6.  (First case with 8 steps unrolled 43, with
  // blocks of 256 threads 52.)
  struct Solved {
    size_t within = 0;        // the serial loop that fixes the symbol
    std::string ahead;        // ahead of that loop: what is left of the position
    std::string from, to;     // the iterations of that loop
    std::string text;         // in the loop: declares the symbol
  };
  bool positions_of(Stage& st, const Stmt& set, std::vector<Solved>* solved, Indices* at) {
    if (opt.bounds) return false;   // (an access outside the node has to be seen)
    const Tnode& t = code.prog.tn(set.tn);
    const int64_t limit = 1 << 28;  // keeps the arithmetic on positions in 32 bits
    std::map<std::string, int> axes;   // serial symbol -> axes it is on
    auto terms = [&](const Index& ix) {
      std::vector<std::pair<int64_t, std::string>> v = ix.terms;
      if (ix.kind == Index::Iter) v = {{1, ix.sym}};
      if (ix.kind != Index::Iter && ix.kind != Index::Affine) v.clear();
      return v;
    };
    auto serial = [&](const std::string& s) {
      for (size_t i = 0; i < st.ser.size(); ++i)
        if (st.ser[i].sym == s) return (int)i;
      return -1;
    };
    for (auto& ix : set.idcs)
      for (auto& d : st.ser) axes[d.sym] += ix.uses(d.sym);
    std::vector<LoopDim> par;
    std::set<std::string> given;
    *at = set.idcs;
    for (size_t a = 0; a < set.idcs.size(); ++a) {
      const auto on = terms(set.idcs[a]);
      int last = -1, outer = -1;      // the symbol that the position gives; the innermost of the others
      int64_t c = 0, most = std::abs(set.idcs[a].fixed) + t.dims[a];
      std::set<std::string> seen;
      for (auto& v : on) {
        if (!seen.insert(v.second).second) return false;
        const int i = serial(v.second);
        if (i < 0) {
          for (auto& d : st.par)
            if (d.sym == v.second) par.push_back(d);
          continue;
        }
        if (st.ser[(size_t)i].from < 0 || std::abs(v.first) > limit || st.ser[(size_t)i].to > limit) return false;
        most += std::abs(v.first) * st.ser[(size_t)i].to;
        if (i > last) { last = i; c = v.first; }
      }
      if (last < 0) continue;
      if (axes[st.ser[(size_t)last].sym] != 1 || c == 0 || most > limit) return false;
      for (auto& v : on) {
        const int i = serial(v.second);
        if (i != last) outer = std::max(outer, i);
      }
      if (outer < 0 || on.size() != seen.size()) return false;
      const LoopDim& e = st.ser[(size_t)last];
      const std::string pos = "b200_at" + std::to_string(a), n = "b200_n" + std::to_string(a);
      Solved v;
      v.within = (size_t)outer;
      int64_t co = 0;
      v.ahead = "const int " + n + " = (int)" + pos + " - (" + std::to_string(set.idcs[a].fixed);
      for (auto& x : on)
        if (x.second == st.ser[(size_t)outer].sym) co = x.first;
        else if (x.second != e.sym) v.ahead += " + " + std::to_string(x.first) + " * (int)" + x.second;
      v.ahead += ");\n";
      if (co == 0) return false;
      // c * symbol = n - co * loop, with the symbol between its ends: the loop lies between two quotients
      auto less = [&](int64_t by) { return by ? n + " - " + std::to_string(by) : n; };
      std::string low = less(c > 0 ? c * e.to : c * e.from), high = less(c > 0 ? c * e.from : c * e.to);
      if (co < 0) {
        const std::string was = low;
        low = "-(" + high + ")";
        high = "-(" + was + ")";
      }
      const std::string by = std::to_string(std::abs(co));
      v.from = by == "1" ? low : "-b200_floor_div(-(" + low + "), " + by + ")";
      v.to = by == "1" ? high : "b200_floor_div(" + high + ", " + by + ")";
      const std::string m = "b200_m" + std::to_string(a);
      const std::string pad(6 + 2 * (size_t)outer, ' ');
      v.text = pad + "const int " + m + " = " + n + " - " + std::to_string(co) + " * (int)" + st.ser[(size_t)outer].sym + ";\n";
      if (std::abs(c) != 1) v.text += pad + "if (" + m + " % " + std::to_string(c) + " != 0) continue;\n";
      v.text += pad + "const unsigned int " + e.sym + " = (unsigned int)(" + m + (c == 1 ? "" : " / " + std::to_string(c)) + ");\n";
      solved->push_back(v);
      given.insert(e.sym);
      (*at)[a] = Index();
      (*at)[a].kind = Index::Iter;
      (*at)[a].sym = pos;
      par.push_back({pos, 0, t.dims[a] - 1});
    }
    if (given.empty()) return false;
    // the loops that remain, and where among them each symbol is fixed
    std::vector<LoopDim> ser;
    std::vector<size_t> place(st.ser.size(), 0);
    for (size_t i = 0; i < st.ser.size(); ++i) {
      place[i] = ser.size();
      if (!given.count(st.ser[i].sym)) ser.push_back(st.ser[i]);
    }
    for (auto& v : *solved) {
      if (given.count(st.ser[v.within].sym)) return false;   // (fixed by a symbol that a position gives itself)
      v.within = place[v.within];
    }
    int64_t total = 1;
    for (auto& d : par) {
      total *= d.extent();
      if (total > (1 << 20)) return false;
    }
    st.par = par;
    st.ser = ser;
    st.total = total;
    return true;
  }

  // `lhs_zero`: the node the body assigns is known to be all zero when the stage starts.
  // Returns true when the stage made an earlier zero_out of that node unnecessary.
  bool generic_stage(const std::vector<LoopDim>& nest, const StmtP& body, bool lhs_zero = false) {
    bool zero_out_dead = false;
    Stage st;
    st.kind = Stage::Generic;
    st.kernel = kernel_name();
    // which loops are independent
    std::vector<bool> par(nest.size(), false);
    for (size_t i = 0; i < nest.size(); ++i) par[i] = nest[i].extent() > 0 && parallel_safe(nest[i].sym, *body);
    for (size_t i = 0; i < nest.size(); ++i) (par[i] ? st.par : st.ser).push_back(nest[i]);
    st.total = 1;
    for (auto& d : st.par) st.total *= d.extent();
    for (auto& d : nest)
      if (d.extent() <= 0) st.total = 0;

    Emitter em(code.prog);
    em.large_models = opt.large_models;

    // Scatter accumulation: `t[.., c * o + k, ..] := t[same] + term` where the written position
    // moves with loops that therefore cannot run in parallel (the input gradient of a
    // convolution).  Those loops are spread over threads all the same: a thread sums over the
    // loops that do not move the position and adds its partial sum with one atomic add.
    // Few of them, and each thread would walk far: a thread per position instead (positions_of).
    bool scatter = false, by_position = false;
    std::vector<Solved> solved;
    Indices at;
    if (opt.enable_coop && !st.ser.empty() && st.total > 0 && body->kind == Stmt::Set && body->vec_len == 0 &&
        accumulates_into_self(*body)) {
      const Tnode& t = code.prog.tn(body->tn);
      std::vector<LoopDim> spread, kept;
      for (auto& d : nest) {
        bool in_par = false, moves = false;
        for (auto& q : st.par) in_par = in_par || q.sym == d.sym;
        for (auto& ix : body->idcs) moves = moves || ix.uses(d.sym);
        (in_par || moves ? spread : kept).push_back(d);
      }
      int64_t total = 1;
      for (auto& d : spread) total *= d.extent();
      int64_t walk = 1;
      for (auto& d : st.ser) walk *= d.extent();
      if ((t.prec == Prec::Single || t.prec == Prec::Double) && t.mode != Mode::Virtual && spread.size() > st.par.size()) {
        if (total >= 4096) {
          scatter = true;
          st.par = spread;
          st.ser = kept;
          st.total = total;
        } else if (walk >= 256) {
          by_position = positions_of(st, *body, &solved, &at);
        }
      }
    }
    const bool moving = scatter || by_position;
    if (by_position) st.block = 32;

    if (!moving && !st.ser.empty() && st.total > 0 && opt.enable_coop && ser_split_stage(st, *body)) return false;

    CoopInfo ci;
    if (st.ser.empty() && st.total > 0) ci = find_coop(*body, st.total);
    if (ci.grid_blocks > 0) {
      --next_kernel;  // the name reserved above is re-issued to the first pass
      grid_reduce_stage(body, ci);
      return false;
    }
    std::set<int> written;
    walk_stmt(*body, [](const Scalar&) {}, [&](const Stmt& s) {
      if (s.kind == Stmt::Set || s.kind == Stmt::ZeroOut) written.insert(s.tn);
    });

    // Pairs.  When the stage is one assignment whose innermost parallel loop runs along the last
    // axis of the written node, and everything in it is fp32, bf16 or half, a thread takes TWO
    // neighbouring iterations of that loop: 4- and 8-byte accesses, packed 16-bit arithmetic.
    bool pairs = false;
    if (pairs_here() && !moving && ci.sym.empty() && body->kind == Stmt::Set && body->vec_len == 0 && !st.par.empty() && st.total > 0) {
      const Stmt& set = *body;
      const Tnode& t = code.prog.tn(set.tn);
      const LoopDim& p = st.par.back();
      bool ok = p.from == 0 && p.extent() % 2 == 0 && Emitter::pair_prec(t.prec) && t.mode != Mode::Virtual && !set.idcs.empty() &&
                set.idcs.back().kind == Index::Iter && set.idcs.back().sym == p.sym && t.dims.back() % 2 == 0;
      for (size_t a = 0; ok && a + 1 < set.idcs.size(); ++a)
        if (set.idcs[a].uses(p.sym)) ok = false;
      // reads of the written node only at the written position (they become the promoted register)
      walk_scalar(*set.value, [&](const Scalar& e) {
        if (e.kind == Scalar::GetDyn && e.tn == set.tn) ok = false;
      }, [](const Stmt&) {});
      if (ok && em.pair_supported(*set.value)) {
        pairs = true;
        em.pair = true;
        em.pair_sym = p.sym;
        em.pair_vector_loads = true;
      }
    }
    // Accumulator promotion: `t[p] := f(t[p], ...)` under serial loops that do not move p keeps
    // t[p] in a register across those loops (one load, or none when the node is known to be zero,
    // and one store) instead of a read-modify-write of memory per iteration.
    std::string before, after, self_type, self_init;
    if (scatter) {
      const Stmt& set = *body;
      const Tnode& t = code.prog.tn(set.tn);
      em.used_nodes.insert(set.tn);
      before = std::string("    ") + Emitter::ctype(t.prec) + " b200_self = 0;\n";
      after = "    atomicAdd(&" + t.ident + "[" + em.offset(set.idcs, t.dims) + "], b200_self);\n";
      em.forwarded[set.tn] = {set.idcs, "b200_self"};
      em.set_redirect[set.tn] = {set.idcs, "b200_self"};
    } else if (by_position) {
      const Stmt& set = *body;
      const Tnode& t = code.prog.tn(set.tn);
      em.used_nodes.insert(set.tn);
      const std::string lv = t.ident + "[" + em.offset(at, t.dims) + "]";
      before = std::string("    ") + Emitter::ctype(t.prec) + " b200_self = " + lv + ";\n";
      after = "    " + lv + " = b200_self;\n";
      em.forwarded[set.tn] = {set.idcs, "b200_self"};
      em.set_redirect[set.tn] = {set.idcs, "b200_self"};
    } else if (ci.sym.empty() && (pairs || !st.ser.empty()) && body->kind == Stmt::Set && body->vec_len == 0) {
      const Stmt& set = *body;
      const Tnode& t = code.prog.tn(set.tn);
      bool ok = t.mode != Mode::Virtual && t.prec != Prec::Uint4x32;
      for (auto& ix : set.idcs)
        for (auto& d : st.ser)
          if (ix.uses(d.sym)) ok = false;
      int self_reads = 0;
      walk_scalar(*set.value, [&](const Scalar& e) {
        if (e.kind == Scalar::LocalScope) ok = false;
        if ((e.kind == Scalar::Get || e.kind == Scalar::GetDyn) && e.tn == set.tn) {
          bool same = e.kind == Scalar::Get && e.idcs.size() == set.idcs.size();
          for (size_t i = 0; same && i < e.idcs.size(); ++i)
            if (e.idcs[i].kind != set.idcs[i].kind || e.idcs[i].sym != set.idcs[i].sym || e.idcs[i].fixed != set.idcs[i].fixed ||
                e.idcs[i].terms != set.idcs[i].terms)
              same = false;
          if (same) ++self_reads; else ok = false;
        }
      }, [](const Stmt&) {});
      if (ok && self_reads > 0) {
        const std::string off = em.offset(set.idcs, t.dims);
        const std::string lv = t.ident + "[" + off + "]";
        em.used_nodes.insert(set.tn);
        if (pairs) {
          const std::string PT = Emitter::pair_type(t.prec);
          const std::string at = "(" + t.ident + " + " + off + ")";
          self_type = PT;
          self_init = lhs_zero ? (t.prec == Prec::Single ? std::string("b200_f2{0.0f, 0.0f}") : std::string("0u")) : "*(const " + PT + "*)" + at;
          before = "    " + PT + " b200_self = " + self_init + ";\n";
          after = "    *(" + PT + "*)" + at + " = b200_self;\n";
        } else {
          self_type = Emitter::rtype(t.prec);
          self_init = lhs_zero ? em.constant(0.0, t.prec) : Emitter::load_wrap(t.prec, lv);
          before = "    " + self_type + " b200_self = " + self_init + ";\n";
          after = "    " + lv + " = " + Emitter::store_wrap(t.prec, "b200_self") + ";\n";
        }
        em.forwarded[set.tn] = {set.idcs, "b200_self"};
        em.set_redirect[set.tn] = {set.idcs, "b200_self"};
        zero_out_dead = lhs_zero && covers_node(set, st.par);
      }
    }
    if (pairs && before.empty()) {
      // without promotion a read of the written node would be a plain (unpaired) memory access
      bool self = false;
      walk_scalar(*body->value, [&](const Scalar& e) {
        if ((e.kind == Scalar::Get || e.kind == Scalar::GetDyn) && e.tn == body->tn) self = true;
      }, [](const Stmt&) {});
      if (self) {
        pairs = false;
        em.pair = false;
        em.pair_vector_loads = false;
      }
    }
    if (pairs) {
      st.total /= 2;      // one thread per pair
      st.min_align = 8;   // pairs are read and written as 4- and 8-byte words
    }
    // Small tables read over and over.  A read-only node of at most 32 KB that the stage reads inside
    // a reduction or serial loop, many times per element (the 512 x 27 embedding table of a one-hot
    // contraction with K = 27: rows of 54 bytes, no tensor-map can describe them) is copied into
    // shared memory once per block; the strided reads then hit shared-memory banks instead of L1
    // sectors.  Such a stage keeps its own kernel (few blocks, each looping over many elements).
    std::vector<int> staged;
    if (opt.enable_coop && !moving && !pairs && ci.sym.empty() && body->kind == Stmt::Set && st.total > 0) {
      int64_t work = st.total;
      for (auto& d : st.ser) work *= std::max<int64_t>(1, d.extent());
      std::set<std::string> inner_syms;
      for (auto& d : st.ser) inner_syms.insert(d.sym);
      walk_stmt(*body, [](const Scalar&) {}, [&](const Stmt& x) { if (x.kind == Stmt::For) inner_syms.insert(x.index); });
      int64_t inner_iters = 1;
      walk_stmt(*body, [](const Scalar&) {}, [&](const Stmt& x) { if (x.kind == Stmt::For) inner_iters *= std::max<int64_t>(1, x.to - x.from + 1); });
      std::set<int> cand;
      size_t bytes = 0;
      walk_scalar(*body->value, [&](const Scalar& e) {
        if (e.kind != Scalar::Get) return;
        const Tnode& t = code.prog.tn(e.tn);
        if (!t.read_only || t.mode == Mode::Virtual || written.count(e.tn) || t.bytes() > 32768 || t.prec == Prec::Uint4x32) return;
        bool in_loop = false;
        for (auto& ix : e.idcs)
          for (auto& sy : inner_syms) in_loop = in_loop || ix.uses(sy);
        if (in_loop && work * inner_iters >= 256 * t.num_elems()) cand.insert(e.tn);
      }, [](const Stmt&) {});
      // first the nodes indexed by the innermost parallel loop: their reads differ from thread to
      // thread (a read that is the same for a whole warp is one broadcast access anyway)
      std::vector<int> order(cand.begin(), cand.end());
      auto strided = [&](int tn) {
        bool u = false;
        walk_scalar(*body->value, [&](const Scalar& e) {
          if (e.kind == Scalar::Get && e.tn == tn && !st.par.empty())
            for (auto& ix : e.idcs) u = u || ix.uses(st.par.back().sym);
        }, [](const Stmt&) {});
        return u;
      };
      std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return strided(a) > strided(b); });
      for (int tn : order) {
        if (bytes + (size_t)code.prog.tn(tn).bytes() > 40960) continue;
        bytes += (size_t)code.prog.tn(tn).bytes();
        staged.push_back(tn);
        em.node_alias[tn] = "b200_sm_" + code.prog.tn(tn).ident;
      }
      if (!staged.empty() && inner_iters < 8) {   // nothing is re-read often enough
        staged.clear();
        em.node_alias.clear();
      }
    }
    std::string inner, alone;
    int ind = 4 + 2 * (int)st.ser.size();
    if (!ci.sym.empty()) {
      st.coop = ci.width;
      if (ci.width > 32) st.block = ci.width;
      // (few warps in single precision: with many, or 16-bit values to convert, there is nothing to wait for; 31 rows of
      // 777-472-66-2, a training step, 33.9 us and 35.4, two rows of 80-1832-382-55 in half precision 14.9 and 15.7)
      bool wide_values = true;
      walk_scalar(*body->value, [&](const Scalar& e) { if (e.kind == Scalar::Get) wide_values = wide_values && code.prog.tn(e.tn).prec == Prec::Single; }, [](const Stmt&) {});
      if (ci.width > 32 || (ci.extent >= 256 && st.total <= 148 * 32 && wide_values)) alone = coop_body(em, *body, ci, ind, true);
      inner = coop_body(em, *body, ci, ind, ci.width > 32);
    } else {
      inner = em.stmt(*body, ind);
    }
    // serial loops wrap the body in their original order
    std::string open, close;
    int k = 4;
    for (size_t i = 0; i < st.ser.size(); ++i) {
      const LoopDim& d = st.ser[i];
      const std::string pad((size_t)k, ' ');
      std::string from, to;
      for (auto& v : solved)
        if (v.within == i) {
          open += pad + v.ahead;
          from = "max(" + (from.empty() ? std::to_string(d.from) : from) + ", " + v.from + ")";
          to = "min(" + (to.empty() ? std::to_string(d.to) : to) + ", " + v.to + ")";
        }
      if (!from.empty()) {
        const std::string last = "b200_last" + std::to_string(i);
        open += pad + "const int " + last + " = " + to + ";\n" + pad + "for (unsigned int " + d.sym + " = (unsigned int)" + from + "; (int)" + d.sym + " <= " + last + "; ++" + d.sym + ") {\n";
      } else {
        // (by position: the terms are added one after the other, but the loads of sixteen of them are under way together)
        if (by_position && i + 1 == st.ser.size()) open += "#pragma unroll 16\n";
        open += pad + "for (unsigned int " + d.sym + " = " + std::to_string(d.from) + "; " + d.sym + " <= " + std::to_string(d.to) + "; ++" + d.sym + ") {\n";
      }
      k += 2;
      for (auto& v : solved)
        if (v.within == i) open += v.text;
    }
    for (size_t i = st.ser.size(); i-- > 0;) {
      k -= 2;
      close += std::string((size_t)k, ' ') + "}\n";
    }
    std::string body_text = before + open + inner + close + after;

    // index decomposition: the innermost parallel loop varies fastest across threads
    // (in 32-bit arithmetic when the flattened count fits: 64-bit divisions by constants cost
    // several times as many instructions, and pointwise kernels are made of little else)
    std::string decomp;
    {
      const bool narrow = st.total < (1ll << 31);
      const std::string IT = narrow ? "unsigned int" : "unsigned long long", SUF = narrow ? "u" : "ull";
      std::string rem = "b200_g";
      if (narrow && st.par.size() > 1) {
        decomp += "    const unsigned int b200_g32 = (unsigned int)b200_g;\n";
        rem = "b200_g32";
      }
      for (size_t i = st.par.size(); i-- > 0;) {
        const LoopDim& d = st.par[i];
        const bool pair_dim = pairs && i + 1 == st.par.size();   // iterations of this loop are taken two at a time
        std::string ext = std::to_string(pair_dim ? d.extent() / 2 : d.extent()) + SUF;
        std::string val = i == 0 ? rem : "(" + rem + " % " + ext + ")";
        decomp += "    const unsigned int " + d.sym + " = " + (pair_dim ? "2u * " : "") + "(unsigned int)" + val +
                  (d.from ? " + " + std::to_string(d.from) : std::string()) + ";\n";
        if (i != 0) {
          std::string nr = "b200_r" + std::to_string(i);
          decomp += "    const " + IT + " " + nr + " = " + rem + " / " + ext + ";\n";
          rem = nr;
        }
      }
    }
    // the kernel text is assembled at the end of the routine (emit_kernels), when it is known
    // which neighbouring stages are small enough to share one launch
    Piece pc;
    pc.decomp = decomp;
    pc.body_text = body_text;
    if (!alone.empty()) pc.alone = before + open + alone + close + after;
    pc.used = em.used_nodes;
    pc.written = written;
    pc.uses_merge = em.uses_merge;
    int64_t ser_work = 1;
    for (auto& d : st.ser) ser_work *= std::max<int64_t>(1, d.extent());
    // (a single output that a whole block sums up fits the block that other small stages share)
    const bool block_sum = st.coop == 1024 && st.total == 1;
    pc.fusable = opt.enable_fuse && st.total > 0 && (st.coop == 0 || st.coop == 32 || block_sum) &&
                 st.total * std::max(1, st.coop) <= 16384 && ser_work <= 4096;
    if (moving) pc.fusable = false;
    {
      // A stage shares the single block of small stages only while that block gets through it in less
      // than what leaving it out costs: its own launch, and a second one for the block's other half (8 us,
      // 16000 cycles, with the stage's own time on many SMs).  Each of a thread's iterations takes the
      // latency of its loads or, with many warps, their issue, about six instructions per warp and
      // scheduler, twice that for pairs.  (The 37 x 10 logits over 1024 hidden units took 25 us of one block.)
      const double threads = (double)st.total * std::max(1, st.coop);
      const double rounds = std::ceil(threads / 1024.0), warps = std::ceil(std::min(threads, 1024.0) / 32.0);
      const double iters = rounds * (double)ser_work * iterations(*body) / std::max(1, st.coop);
      // A warp's sums over a node that does not fit into shared memory wait for memory at every step (one row of 160-552-177-35:
      // 23 us with the second layer in the block, 8 us without; 300 cycles a step).
      bool far = false;
      for (int n : em.used_nodes) far = far || (st.coop && code.prog.tn(n).bytes() > 12288);
      if (iters * std::max(far ? 300.0 : 30.0, (pairs ? 12.0 : 6.0) * warps / 4.0) > 16000.0) pc.fusable = false;
    }
    if (opt.enable_fuse && !moving && st.coop == 0 && st.total > 0 && !st.par.empty() && st.par[0].from == 0 && !(pairs && st.par.size() == 1)) {
      pc.body = body;
      pc.row_sym = st.par[0].sym;
      pc.rows = st.par[0].extent();
      pc.per_row = st.total / pc.rows * ser_work;
    }
    if (!moving) pc.any_body = body;
    if (!self_type.empty() && ser_work > 1 && (code.prog.tn(body->tn).prec == Prec::Single || code.prog.tn(body->tn).prec == Prec::Double) &&
        accumulates_into_self(*body)) {
      pc.sum = true;
      pc.self_type = self_type;
      pc.self_init = self_init;
      pc.zero = pairs ? "b200_f2{0.0f, 0.0f}" : "0";
      pc.inner = inner;
      pc.after = after;
      pc.ser = st.ser;
    }
    if (!staged.empty()) {      // keeps a kernel of its own
      pc.staged = staged;
      pc.fusable = false;
      pc.body = nullptr;
      pc.any_body = nullptr;
      st.grid_override = 148 * 4;
      st.block = 512;
    }
    pc.par = st.par;
    pc.coop = st.coop;
    pc.pairs = pairs;
    pc.ser_work = ser_work;
    std::ostringstream note;
    note << "par=" << st.par.size() << " ser=" << st.ser.size()
         << (st.coop > 32 ? " block-per-element" : st.coop ? " warp-per-element" : "") << (pairs ? " pairs" : "")
         << (scatter ? " scatter accumulation (atomic adds)" : by_position ? " accumulation by position" : "") << (staged.empty() ? "" : " small table staged in shared memory");
    st.note = note.str();
    pieces[code.stages.size()] = pc;
    st.writes.assign(written.begin(), written.end());
    code.stages.push_back(st);
    return zero_out_dead;
  }

  // Text of one stand-alone generic kernel (grid-stride over the stage's parallel iterations).
  void emit_single(Stage& st, const Piece& pc) {
    Emitter em(code.prog);
    em.used_nodes = pc.used;
    em.uses_merge = pc.uses_merge;
    std::string statics = static_prologue(pc.body_text + pc.decomp + pc.whole, em, 2);
    std::ostringstream k_src;
    k_src << "extern \"C\" __global__ void __launch_bounds__(" << st.block << ") " << st.kernel << "(";
    emit_params(k_src, st, em, pc.written);
    k_src << ") {\n" << kGridEntry << statics;
    if (!pc.whole.empty()) {
      src << k_src.str() << pc.whole << "}\n\n";
      return;
    }
    for (int tn : pc.staged) {
      const Tnode& t = code.prog.tn(tn);
      const std::string sm = "b200_sm_" + t.ident;
      k_src << "  __shared__ " << Emitter::ctype(t.prec) << " " << sm << "[" << t.num_elems() << "];\n"
            << "  for (unsigned int b200_i = threadIdx.x; b200_i < " << t.num_elems() << "u; b200_i += blockDim.x) " << sm
            << "[b200_i] = " << t.ident << "[b200_i];\n";
    }
    if (!pc.staged.empty()) k_src << "  __syncthreads();\n";
    if (st.coop > 32) {
      k_src << "  __shared__ double b200_red[32];\n";
      k_src << "  const unsigned int b200_t = threadIdx.x;\n";
      k_src << "  for (unsigned long long b200_g = blockIdx.x; b200_g < " << st.total << "ull; b200_g += gridDim.x) {\n";
    } else if (st.coop) {
      k_src << "  const unsigned int b200_t = threadIdx.x & 31u;\n";
      k_src << "  const unsigned long long b200_warp = ((unsigned long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;\n";
      k_src << "  const unsigned long long b200_nwarps = ((unsigned long long)gridDim.x * blockDim.x) >> 5;\n";
      k_src << "  for (unsigned long long b200_g = b200_warp; b200_g < " << st.total << "ull; b200_g += b200_nwarps) {\n";
    } else {
      k_src << "  for (unsigned long long b200_g = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; b200_g < "
            << st.total << "ull; b200_g += (unsigned long long)gridDim.x * blockDim.x) {\n";
    }
    k_src << pc.decomp << (pc.alone.empty() ? pc.body_text : pc.alone) << "  }\n}\n\n";
    src << k_src.str();
  }

  // Several small consecutive stages (and small zero_outs) as ONE kernel of a single
  // 1024-thread block: each stage strides its iterations over the block, __syncthreads()
  // separates the stages.  Launch latency, not work, dominates such routines (the 2-16-16-1
  // training step is ~30 stages of a few hundred iterations each).
  void merge_origins(Stage& f, const std::vector<size_t>& idx) {
    std::set<int> all;
    std::set<int> w;
    for (size_t i : idx) {
      all.insert(code.stages[i].origins.begin(), code.stages[i].origins.end());
      w.insert(code.stages[i].writes.begin(), code.stages[i].writes.end());
    }
    f.origins.assign(all.begin(), all.end());
    f.writes.assign(w.begin(), w.end());
  }

  // Nodes small enough live in shared memory for the length of the block: read once at its start, written
  // back at its end, and routine-local ones that no other stage touches never reach memory at all.  A stage
  // then waits some 30 cycles for what the one before it wrote instead of some 300.  The barrier
  // between two stages is left out when neither writes what the other touches; a long sum with few outputs
  // (a gradient over the batch) is shared by up to four lanes of a warp.  (The 25 stages of the
  // 2-16-16-1 training step: 11.6 us through memory.)
  std::map<int, std::set<size_t>> node_stages;   // node -> stages that touch it, by index into code.stages
  void note_node_stages() {
    node_stages.clear();
    for (size_t i = 0; i < code.stages.size(); ++i) {
      const Stage& st = code.stages[i];
      if (st.kind == Stage::Memset) node_stages[st.memset_tn].insert(i);
      auto it = pieces.find(i);
      if (it != pieces.end())
        for (int n : it->second.used) node_stages[n].insert(i);
      for (auto& a : st.args)
        if (a.kind == KArg::Node) node_stages[a.tn].insert(i);
      if (st.kind == Stage::Gemm)
        for (int n : {st.gemm.a_tn, st.gemm.b_tn, st.gemm.d_tn}) node_stages[n].insert(i);
      if (st.kind == Stage::Attn)
        for (int n : {st.attn.q_tn, st.attn.k_tn, st.attn.v_tn}) node_stages[n].insert(i);
      for (int n : st.writes) node_stages[n].insert(i);
    }
  }

  // Short innermost loops of a known number of steps are unrolled 32 times: one block has too few warps to hide
  // the latency of a load per step, and how far the compiler unrolls by itself changes with the size of the kernel
  // around the loop (64 points through 2-64-64-1: 26.7 us or 30.7; 150 through 2-40-40-1: 41.0, 33.1 so).
  static std::string unrolled(const std::string& text) {
    std::vector<std::string> lines;
    std::istringstream in(text);
    for (std::string line; std::getline(in, line);) lines.push_back(line);
    std::string out;
    for (size_t i = 0; i < lines.size(); ++i) {
      const size_t at = lines[i].find_first_not_of(' ');
      if (at != std::string::npos && lines[i].compare(at, 4, "for ") == 0 && lines[i].back() == '{' &&
          (lines[i].find(" <= ") != std::string::npos || lines[i].find("b200_k < ") != std::string::npos)) {
        size_t j = i + 1;
        while (j < lines.size() && lines[j].find("for (") == std::string::npos && lines[j].find_first_not_of(' ') != std::string::npos &&
               lines[j][lines[j].find_first_not_of(' ')] != '}')
          ++j;
        if (j < lines.size() && j - i <= 9 && lines[j].find("for (") == std::string::npos) out += "#pragma unroll 32\n";
      }
      out += lines[i] + "\n";
    }
    return out;
  }

  Stage emit_fused(const std::vector<size_t>& idx) {
    Stage f;
    merge_origins(f, idx);
    f.kind = Stage::Generic;
    f.kernel = code.stages[idx.front()].kernel.empty() ? kernel_name() : code.stages[idx.front()].kernel;
    f.block = 1024;
    f.grid_override = 1;
    f.total = 1;
    Emitter em(code.prog);
    std::set<int> written;
    std::string text;
    int64_t most = 1;                 // threads the widest stage could use
    bool ordered = false;             // some stage depends on another
    bool block_sums = false;          // some stage sums with the whole block
    std::set<int> fresh_w, fresh_r;   // written / read since the last barrier
    // (stages that overwrite different parts of one node, the margins of a padded image, do not depend on one another)
    std::map<int, std::vector<Box>> fresh_boxes;   // node -> the parts overwritten since the last barrier, where all are known
    auto barrier_for = [&](const std::set<int>& used, const std::set<int>& writes, int boxed = -1, const Box& box = {}) {
      bool need = false;
      auto clear_of_all = [&](int n) {
        if (n != boxed || box.empty() || fresh_boxes[n].empty()) return false;
        for (auto& b : fresh_boxes[n])
          if (b.empty() || !apart(b, box)) return false;
        return true;
      };
      for (int n : used) need = need || (fresh_w.count(n) && !clear_of_all(n));
      for (int n : writes) need = need || (fresh_r.count(n) && !(fresh_w.count(n) && clear_of_all(n)));
      if (need) {
        ordered = true;
        text += "  __syncthreads();\n";
        fresh_w.clear();
        fresh_r.clear();
        fresh_boxes.clear();
      } else if (!text.empty()) {
        text += "  // __syncthreads() left out: neither stage writes what the other touches\n";
      }
      fresh_r.insert(used.begin(), used.end());
      fresh_w.insert(writes.begin(), writes.end());
      for (int n : used) fresh_boxes[n].push_back(n == boxed ? box : Box());
    };
    std::set<int> first_cleared;   // nodes whose first use here overwrites them
    std::set<int> moving;          // nodes read at a static index: a slice of something larger
    std::set<std::string> statics_syms;
    for (auto& sy : code.prog.statics) statics_syms.insert(sy.sym);
    for (size_t i : idx) {
      const Stage& st = code.stages[i];
      if (st.kind == Stage::Memset) {
        const Tnode& t = code.prog.tn(st.memset_tn);
        if (!em.used_nodes.count(t.id)) first_cleared.insert(t.id);
        barrier_for({t.id}, {t.id});
        em.used_nodes.insert(t.id);
        written.insert(t.id);
        most = std::max<int64_t>(most, t.num_elems());
        text += "  for (unsigned int b200_z = B200_FIRST; b200_z < " + std::to_string(t.num_elems()) +
                "u; b200_z += B200_STEP) " + t.ident + "[b200_z] = " + em.storage_zero(t.prec) + ";\n";
      } else {
        const Piece& pc = pieces[i];
        const Box box = written_box(pc);
        barrier_for(pc.used, pc.written, box.empty() ? -1 : pc.any_body->tn, box);
        if (pc.any_body && pc.any_body->kind == Stmt::Set && !em.used_nodes.count(pc.any_body->tn) && !pc.sum && covers_node(*pc.any_body, pc.par)) {
          bool reads = false;
          walk_scalar(*pc.any_body->value, [&](const Scalar& e) {
            if ((e.kind == Scalar::Get || e.kind == Scalar::GetDyn) && e.tn == pc.any_body->tn) reads = true;
          }, [](const Stmt&) {});
          if (!reads) first_cleared.insert(pc.any_body->tn);   // written in full before anything reads it
        }
        f.min_align = std::max(f.min_align, st.min_align);
        em.used_nodes.insert(pc.used.begin(), pc.used.end());
        written.insert(pc.written.begin(), pc.written.end());
        em.uses_merge |= pc.uses_merge;
        if (pc.any_body)
          walk_stmt(*pc.any_body, [&](const Scalar& e) {
            if (e.kind == Scalar::Get || e.kind == Scalar::GetDyn)
              for (auto& ix : e.idcs)
                for (auto& sy : statics_syms)
                  if (ix.uses(sy)) moving.insert(e.tn);
          }, [&](const Stmt& w) {
            if (w.kind == Stmt::Set)
              for (auto& ix : w.idcs)
                for (auto& sy : statics_syms)
                  if (ix.uses(sy)) moving.insert(w.tn);
          });
        int64_t ser_total = 1;
        for (auto& d : pc.ser) ser_total *= d.extent();
        // Lanes per sum: two or four, 16 steps each at least.  Neighbouring lanes keep neighbouring outputs, so that a
        // step reads stretches of a row.  (Training steps of points x hidden units, us.  No sharing, up to 4 lanes, up
        // to 32: 200 x 16 23.1, 18.5, 23.0; 100 x 100 35.0, 30.7, 30.9; 8 x 128 16.8, 17.2, 19.4; 64 x 64 26.7, 28.7, 34.9;
        // with two steps a lane 12 x 112 takes 22.0 instead of 18.8.)
        int64_t share = 1;
        if (pc.sum)
          while (share < 4 && share * 2 * st.total <= 1024 && share * 32 <= ser_total) share *= 2;
        most = std::max<int64_t>(most, st.total * std::max(1, st.coop));
        if (share > 1) {
          ordered = true;
          const std::string S = std::to_string(share) + "u", O = std::to_string(32 / share) + "u";
          text += "  {\n  const unsigned int b200_s = threadIdx.x % 32u / " + O + ", b200_gq = threadIdx.x / 32u * " + O + " + threadIdx.x % " + O + ";\n  const bool b200_on = b200_gq < " +
                  std::to_string(st.total) + "u;\n  const unsigned int b200_g = b200_on ? b200_gq : 0u;\n" + pc.decomp + "    " + pc.self_type + " b200_self = " +
                  pc.zero + ";\n    if (b200_on) {\n      if (b200_s == 0u) b200_self = " + pc.self_init + ";\n";
          std::string term, rem = "b200_l";
          for (size_t q = pc.ser.size(); q-- > 0;) {
            const LoopDim& d = pc.ser[q];
            const std::string ext = std::to_string(d.extent()) + "u";
            term += "        const unsigned int " + d.sym + " = " + (q == 0 ? rem : rem + " % " + ext) + (d.from ? " + " + std::to_string(d.from) + "u" : std::string()) + ";\n";
            if (q) {
              term += "        const unsigned int b200_lq" + std::to_string(q) + " = " + rem + " / " + ext + ";\n";
              rem = "b200_lq" + std::to_string(q);
            }
          }
          term += pc.inner;
          // (a number of steps that is the same for every lane, and known: the loads of many steps are under way together)
          text += "      for (unsigned int b200_k = 0; b200_k < " + std::to_string(ser_total / share) + "u; ++b200_k) {\n        const unsigned int b200_l = b200_k * " + S +
                  " + b200_s;\n" + term + "      }\n";
          if (ser_total % share)
            text += "      if (b200_s < " + std::to_string(ser_total % share) + "u) {\n        const unsigned int b200_l = " + std::to_string(ser_total / share * share) +
                    "u + b200_s;\n" + term + "      }\n";
          text += "    }\n#pragma unroll\n    for (unsigned int b200_o = " + O + "; b200_o < 32u; b200_o <<= 1) ";
          if (pc.pairs)
            text += "{\n      const b200_f2 b200_w = {__shfl_xor_sync(0xffffffffu, b200_self.x, b200_o), __shfl_xor_sync(0xffffffffu, b200_self.y, b200_o)};\n"
                    "      b200_self = b200_f2{b200_self.x + b200_w.x, b200_self.y + b200_w.y};\n    }\n";
          else
            text += "b200_self = b200_self + __shfl_xor_sync(0xffffffffu, b200_self, b200_o);\n";
          text += "    if (b200_on && b200_s == 0u) {\n" + pc.after + "    }\n  }\n";
        } else {
          text += "  {\n";
          if (st.coop > 32) {
            ordered = true;
            block_sums = true;
            text += "  const unsigned int b200_t = threadIdx.x;\n  {\n  const unsigned int b200_g = 0u;\n";
          } else if (st.coop) {
            text += "  const unsigned int b200_t = threadIdx.x & 31u;\n";
            text += "  for (unsigned int b200_g = B200_FIRST >> 5; b200_g < " + std::to_string(st.total) + "u; b200_g += B200_STEP >> 5) {\n";
          } else {
            text += "  for (unsigned int b200_g = B200_FIRST; b200_g < " + std::to_string(st.total) + "u; b200_g += B200_STEP) {\n";
          }
          text += pc.decomp + pc.body_text + "  }\n  }\n";
        }
      }
    }
    // Stages that do not depend on one another (the updates of several parameters, the margins of a padded
    // image) need no single block: every stage is spread over the whole grid.
    const bool wide = !ordered && most > 1024;
    if (!wide) text = unrolled(text);
    {
      auto put = [&](const std::string& what, const std::string& by) {
        for (size_t q = 0; (q = text.find(what, q)) != std::string::npos; q += by.size()) text.replace(q, what.size(), by);
      };
      put("B200_FIRST", wide ? "(blockIdx.x * 256u + threadIdx.x)" : "threadIdx.x");
      put("B200_STEP", wide ? "(gridDim.x * 256u)" : "blockDim.x");
    }
    // which nodes move into shared memory: the smallest first
    std::vector<int> small;
    if (!opt.bounds && !wide)
      for (int n : em.used_nodes) {
        const Tnode& t = code.prog.tn(n);
        if (t.mode != Mode::Virtual && t.prec != Prec::Uint4x32 && t.bytes() <= 12288 && !moving.count(n)) small.push_back(n);
      }
    std::sort(small.begin(), small.end(), [&](int a, int b) { return code.prog.tn(a).bytes() < code.prog.tn(b).bytes() || (code.prog.tn(a).bytes() == code.prog.tn(b).bytes() && a < b); });
    std::string decls, load, land, store;
    if (block_sums) decls = "  __shared__ double b200_red[32];\n";
    size_t bytes = 0;
    for (int n : small) {
      const Tnode& t = code.prog.tn(n);
      const size_t sz = ((size_t)t.bytes() + 15) & ~(size_t)15;
      if (bytes + sz > 45056) break;
      const std::string T = Emitter::ctype(t.prec), count = std::to_string(t.num_elems()) + "u";
      bool mine = t.mode == Mode::Local;   // a routine-local node no other stage touches
      for (size_t i : node_stages[n]) mine = mine && std::count(idx.begin(), idx.end(), i);
      decls += "  __shared__ __align__(16) " + T + " b200_sm_" + t.ident + "[" + std::to_string(t.num_elems()) + "];\n";
      const std::string each = "  for (unsigned int b200_z = threadIdx.x; b200_z < " + count + "; b200_z += 1024u) ";
      if (mine) {
        if (t.zero_init && !first_cleared.count(n)) load += each + "b200_sm_" + t.ident + "[b200_z] = " + em.storage_zero(t.prec) + ";\n";
        em.used_nodes.erase(n);
      } else {
        // (all of the block's loads are in flight before the first of them is stored)
        if (!first_cleared.count(n))
          for (int64_t q = 0; q * 1024 < t.num_elems(); ++q) {
            const std::string v = "b200_in" + std::to_string(n) + "_" + std::to_string(q), at = "threadIdx.x + " + std::to_string(q * 1024) + "u";
            const std::string in = at + " < " + count;
            load += "  " + T + " " + v + " = 0;\n  if (" + in + ") " + v + " = " + t.ident + "__g[" + at + "];\n";
            land += "  if (" + in + ") b200_sm_" + t.ident + "[" + at + "] = " + v + ";\n";
          }
        if (written.count(n)) store += each + t.ident + "__g[b200_z] = b200_sm_" + t.ident + "[b200_z];\n";
      }
      decls += "  " + T + "* const " + t.ident + " = b200_sm_" + t.ident + ";\n";
      bytes += sz;
      moved_to_shared.insert(n);
    }
    std::string statics = static_prologue(text, em, 2);
    std::ostringstream params, k_src;
    emit_params(params, f, em, written);
    // parameters of the nodes that moved get another name; the node's own name is its copy
    std::string ps = params.str();
    for (int n : moved_to_shared) {
      const std::string& id = code.prog.tn(n).ident;
      for (size_t q = 0; (q = ps.find(id, q)) != std::string::npos; q += id.size()) {
        const bool l = q > 0 && ps[q - 1] == ' ', r = q + id.size() == ps.size() || ps[q + id.size()] == ',';
        if (l && r) ps.insert(q + id.size(), "__g");
      }
    }
    moved_to_shared.clear();
    if (wide) {
      f.block = 256;
      f.grid_override = (int)std::min<int64_t>((most + 255) / 256, 148 * 8);
    }
    k_src << "extern \"C\" __global__ void __launch_bounds__(" << f.block << ") " << f.kernel << "(" << ps << ") {\n" << kGridEntry << decls << statics << load << land
          << (load.empty() ? "" : "  __syncthreads();\n") << text << (store.empty() ? "" : "  __syncthreads();\n") << store << "}\n\n";
    src << k_src.str();
    f.note = "fused " + std::to_string(idx.size()) + (wide ? " small stages over one grid" : " small stages in one block");
    return f;
  }
  std::set<int> moved_to_shared;

  // Warp-per-row fusion.  A run of stages that share their L outermost parallel loops ("the
  // row": (batch, position, head) of an attention softmax), some of which reduce over the rest of
  // the row with a warp per output element while others are pointwise along it, and which hand
  // data to one another only within a row, runs as ONE kernel: a warp takes a row and executes
  // the stages one after the other, its lanes striding over the row.  Row max, exponentials, row
  // sum and the division of a softmax are one launch; the row stays in L1 / L2 between them.
  bool rows_independent_prefix(const std::vector<size_t>& run, size_t L) {
    std::map<int, int> writers, users;
    for (size_t i : run) {
      const Piece& pc = pieces[i];
      for (int n : pc.written) writers[n]++;
      for (int n : pc.used) users[n]++;
    }
    std::map<std::pair<int, size_t>, int> axis;  // (shared node, prefix position) -> axis carrying that loop's symbol
    bool ok = true;
    for (size_t i : run) {
      const Piece& pc = pieces[i];
      auto check = [&](int tn, const Indices& idcs) {
        if (!writers.count(tn) || users[tn] < 2) return;
        for (size_t q = 0; q < L; ++q) {
          if (pc.par[q].extent() == 1) continue;   // a loop of one iteration separates nothing
          const std::string& sym = pc.par[q].sym;
          int a = -1;
          for (size_t k = 0; k < idcs.size(); ++k) {
            if (idcs[k].kind == Index::Iter && idcs[k].sym == sym && a < 0) a = (int)k;
            else if (idcs[k].uses(sym)) ok = false;
          }
          if (a < 0) { ok = false; return; }
          auto it = axis.find({tn, q});
          if (it == axis.end()) axis[{tn, q}] = a;
          else if (it->second != a) ok = false;
        }
      };
      walk_stmt(
          *pc.any_body,
          [&](const Scalar& e) {
            if (e.kind == Scalar::Get) check(e.tn, e.idcs);
            if (e.kind == Scalar::GetDyn && writers.count(e.tn) && users[e.tn] >= 2) ok = false;
          },
          [&](const Stmt& st) {
            if (st.kind == Stmt::Set) {
              if (st.vec_len > 0 && writers.count(st.tn) && users[st.tn] >= 2) ok = false;
              check(st.tn, st.idcs);
            }
            if (st.kind == Stmt::ZeroOut) ok = false;
          });
    }
    return ok;
  }

  // can stage i join a warp-per-row group whose rows are the first L parallel loops of `like`?
  bool warp_row_member(size_t i, size_t L, const Piece* like) {
    auto it = pieces.find(i);
    if (it == pieces.end() || !it->second.any_body) return false;
    const Piece& pc = it->second;
    if (pc.coop != 0 && pc.coop != 32) return false;
    if (pc.par.size() < L || (pc.coop == 32 && pc.par.size() != L)) return false;
    if (pc.pairs && pc.par.size() == L) return false;   // the pair loop must lie inside the row
    for (size_t q = 0; q < L; ++q) {
      if (pc.par[q].from != 0) return false;
      if (like && pc.par[q].extent() != like->par[q].extent()) return false;
    }
    return true;
  }

  Stage emit_warp_rows(const std::vector<size_t>& run, size_t L) {
    Stage f;
    merge_origins(f, run);
    f.kind = Stage::Generic;
    f.kernel = code.stages[run.front()].kernel;
    f.block = 256;
    int64_t rows = 1;
    for (size_t q = 0; q < L; ++q) rows *= pieces[run.front()].par[q].extent();
    f.total = rows;
    f.coop = 32;   // launch arithmetic: 32 threads per row
    Emitter em(code.prog);
    std::set<int> written;
    std::string text;
    for (size_t i : run) {
      const Stage& st = code.stages[i];
      const Piece& pc = pieces[i];
      f.min_align = std::max(f.min_align, st.min_align);
      em.used_nodes.insert(pc.used.begin(), pc.used.end());
      written.insert(pc.written.begin(), pc.written.end());
      em.uses_merge |= pc.uses_merge;
      if (pc.coop == 32) {
        text += "    {\n    const unsigned long long b200_g = b200_row;\n" + pc.decomp + pc.body_text + "    }\n";
      } else {
        const std::string inner = std::to_string(st.total / rows) + "ull";
        text += "    for (unsigned long long b200_g = b200_row * " + inner + " + b200_t; b200_g < (b200_row + 1ull) * " + inner +
                "; b200_g += 32ull) {\n" + pc.decomp + pc.body_text + "    }\n";
      }
      text += "    __syncwarp();\n";   // orders the row's stores before the next stage's loads
    }
    std::string statics = static_prologue(text, em, 2);
    std::ostringstream k_src;
    k_src << "extern \"C\" __global__ void __launch_bounds__(" << f.block << ") " << f.kernel << "(";
    emit_params(k_src, f, em, written);
    k_src << ") {\n" << kGridEntry << statics
          << "  const unsigned int b200_t = threadIdx.x & 31u;\n"
          << "  const unsigned long long b200_warp = ((unsigned long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;\n"
          << "  const unsigned long long b200_nwarps = ((unsigned long long)gridDim.x * blockDim.x) >> 5;\n"
          << "  for (unsigned long long b200_row = b200_warp; b200_row < " << rows << "ull; b200_row += b200_nwarps) {\n"
          << text << "  }\n}\n\n";
    src << k_src.str();
    f.note = "row-fused " + std::to_string(run.size()) + " stages, one warp per row";
    return f;
  }

  // ---- register-resident rows.  The warp-per-row kernel above lets its stages meet through memory:
  // every stage strides the row again, decomposes indices again and reloads from L1 what the
  // stage before stored.  When every stage is one assignment and touches the shared nodes only at
  // "the row's element t" (t on the node's last, contiguous axis) or at one value per row, a lane
  // instead owns R / 32 CONSECUTIVE elements of the row for the whole kernel: inputs are loaded
  // once with 16-byte accesses into register arrays, reductions run over the lane's registers
  // and one shuffle tree, every produced row is kept in registers for the stages after it and
  // stored once, with 16-byte accesses.  (Softmax over 256 keys: the scores are read once, the
  // exponentials and the weights written once each; layer norm over 512 features likewise.)
  static StmtP rename_stmt(const StmtP& s, const std::map<std::string, std::string>& ren) {
    auto c = std::make_shared<Stmt>(*s);
    rename_idcs(c->idcs, ren);
    auto it = ren.find(c->index);
    if (it != ren.end()) c->index = it->second;
    for (auto& x : c->items) x = rename_stmt(x, ren);
    if (c->body) c->body = rename_stmt(c->body, ren);
    if (c->value) c->value = rename_scalar(c->value, ren);
    return c;
  }
  static void rename_idcs(Indices& idcs, const std::map<std::string, std::string>& ren) {
    for (auto& ix : idcs) {
      if (ix.kind == Index::Iter) {
        auto it = ren.find(ix.sym);
        if (it != ren.end()) ix.sym = it->second;
      } else if (ix.kind == Index::Affine) {
        for (auto& t : ix.terms) {
          auto it = ren.find(t.second);
          if (it != ren.end()) t.second = it->second;
        }
      }
    }
  }
  static ScalarP rename_scalar(const ScalarP& e, const std::map<std::string, std::string>& ren) {
    auto c = std::make_shared<Scalar>(*e);
    rename_idcs(c->idcs, ren);
    {
      Indices one = {c->idx};
      rename_idcs(one, ren);
      c->idx = one[0];
    }
    if (c->body) c->body = rename_stmt(c->body, ren);
    for (auto& a : c->args) a.s = rename_scalar(a.s, ren);
    return c;
  }

  struct RegRowStage {
    StmtP set;                       // the assignment, row symbols renamed to the canonical ones
    bool coop = false;
    std::string t_sym;               // pointwise: the stage's element loop
    std::vector<std::pair<int, std::string>> scopes;   // coop: (scope id, combine op)
    std::vector<std::string> scope_syms;               // coop: each scope's element loop
  };

  bool emit_warp_rows_reg(const std::vector<size_t>& run, size_t L, Stage* out) {
    if (!opt.enable_pairs) return false;
    const Piece& first = pieces[run.front()];
    std::vector<std::string> canon;
    int64_t rows = 1;
    for (size_t q = 0; q < L; ++q) {
      canon.push_back("b200_r" + std::to_string(q) + "_" + first.par[q].sym);
      rows *= first.par[q].extent();
    }
    int64_t R = -1;
    std::vector<RegRowStage> stages;
    for (size_t i : run) {
      if (opt.no_pairs_at.count(code.stages[i].origins.empty() ? -1 : code.stages[i].origins[0])) return false;
      const Piece& pc = pieces[i];
      if (!pc.any_body || pc.any_body->kind != Stmt::Set || pc.any_body->vec_len > 0) return false;
      RegRowStage st;
      std::map<std::string, std::string> ren;
      for (size_t q = 0; q < L; ++q) ren[pc.par[q].sym] = canon[q];
      st.set = rename_stmt(pc.any_body, ren);
      if (pc.coop == 32) {
        st.coop = true;
        if (pc.par.size() != L) return false;
        CoopInfo ci = find_coop(*pc.any_body, 1 << 20);
        if (ci.sym.empty() || ci.width != 32) return false;
        st.scopes = ci.scopes;
        // every scope: [v := neutral;] for k = 0 .. R-1 { v := v op term }
        bool ok = true;
        std::function<void(const Scalar&)> rec = [&](const Scalar& e) {
          if (e.kind == Scalar::LocalScope) {
            const Stmt* b = e.body.get();
            if (b->kind == Stmt::Seq) b = b->items[1].get();
            if (b->kind != Stmt::For || b->from != 0 || b->body->kind == Stmt::For) { ok = false; return; }
            const int64_t ext = b->to + 1;
            if (R < 0) R = ext;
            if (ext != R) ok = false;
            st.scope_syms.push_back(b->index);
            return;
          }
          for (auto& a : e.args) rec(*a.s);
        };
        rec(*st.set->value);
        if (!ok || st.scope_syms.size() != st.scopes.size()) return false;
      } else {
        if (pc.coop != 0 || pc.par.size() != L + 1 || pc.ser_work != 1) return false;
        const LoopDim& t = pc.par[L];
        if (t.from != 0) return false;
        if (R < 0) R = t.extent();
        if (t.extent() != R) return false;
        st.t_sym = t.sym;
        bool scopes = false;
        walk_scalar(*st.set->value, [&](const Scalar& e) { if (e.kind == Scalar::LocalScope || e.kind == Scalar::GetLocal) scopes = true; },
                    [](const Stmt&) {});
        if (scopes) return false;
      }
      stages.push_back(st);
    }
    if (R < 32 || R > 1024) return false;
    const int EPL = (int)((R + 31) / 32);
    const bool dealt = R % 128 == 0 && EPL <= 16, pairwise = R == 64;
    const bool strided = !dealt && !pairwise;   // one element per lane and step, the last step perhaps partly filled
    const bool tail = strided && R % 32 != 0;

    // ---- classify every access
    struct RowNode { Indices idcs; Prec prec; bool loaded = false, produced = false; int writer = -1; };
    std::map<int, RowNode> rownodes;        // nodes touched at (row.., t)
    std::map<int, std::pair<Indices, int>> scalars;   // nodes written once per row: (indices, writing stage)
    auto uses_any = [&](const Indices& idcs, const std::set<std::string>& syms) {
      for (auto& ix : idcs)
        for (auto& sy : syms)
          if (ix.uses(sy)) return true;
      return false;
    };
    bool ok = true;
    std::set<int> written_nodes;
    for (size_t k = 0; k < stages.size(); ++k) {
      const RegRowStage& st = stages[k];
      std::set<std::string> tsyms(st.scope_syms.begin(), st.scope_syms.end());
      if (!st.t_sym.empty()) tsyms.insert(st.t_sym);
      auto row_position = [&](int tn, const Indices& idcs) {
        // last index is exactly an element symbol, on a last axis of extent R; no other use of it
        const Tnode& t = code.prog.tn(tn);
        if (idcs.empty() || idcs.size() != t.dims.size()) return false;
        const Index& last = idcs.back();
        if (last.kind != Index::Iter || !tsyms.count(last.sym) || t.dims.back() != R) return false;
        Indices rest(idcs.begin(), idcs.end() - 1);
        if (uses_any(rest, tsyms)) return false;
        for (auto& ix : rest)
          if (ix.kind != Index::Iter && ix.kind != Index::Fixed) return false;
        return t.prec == Prec::Single || t.prec == Prec::Bfloat16 || t.prec == Prec::Half;
      };
      auto note_row = [&](int tn, const Indices& idcs, bool write) {
        Indices key(idcs.begin(), idcs.end() - 1);
        auto it = rownodes.find(tn);
        if (it == rownodes.end()) {
          RowNode rn;
          rn.idcs = key;
          rn.prec = code.prog.tn(tn).prec;
          it = rownodes.emplace(tn, rn).first;
        } else {
          if (it->second.idcs.size() != key.size()) { ok = false; return; }
          for (size_t a = 0; a < key.size(); ++a)
            if (key[a].kind != it->second.idcs[a].kind || key[a].sym != it->second.idcs[a].sym || key[a].fixed != it->second.idcs[a].fixed) ok = false;
        }
        if (write) {
          if (it->second.produced || it->second.loaded) ok = false;    // written twice, or read before it is written
          it->second.produced = true;
          it->second.writer = (int)k;
        } else if (!it->second.produced) {
          it->second.loaded = true;
        }
      };
      // reads
      walk_scalar(*st.set->value, [&](const Scalar& e) {
        if (e.kind == Scalar::GetDyn || e.kind == Scalar::GetMerge) { ok = false; return; }
        if (e.kind != Scalar::Get) return;
        if (uses_any(e.idcs, tsyms)) {
          if (!row_position(e.tn, e.idcs)) {
            // an element-dependent read of a node this kernel does not write may stay a plain load
            if (written_nodes.count(e.tn)) ok = false;
            bool later = false;
            for (size_t k2 = k; k2 < stages.size(); ++k2) later = later || stages[k2].set->tn == e.tn;
            if (later) ok = false;
            return;
          }
          note_row(e.tn, e.idcs, false);
        } else if (written_nodes.count(e.tn)) {
          auto it = scalars.find(e.tn);
          if (it == scalars.end()) { ok = false; return; }
          if (e.idcs.size() != it->second.first.size()) { ok = false; return; }
          for (size_t a = 0; a < e.idcs.size(); ++a)
            if (e.idcs[a].kind != it->second.first[a].kind || e.idcs[a].sym != it->second.first[a].sym ||
                e.idcs[a].fixed != it->second.first[a].fixed)
              ok = false;
        }
      }, [](const Stmt&) {});
      // the write
      const Stmt& set = *st.set;
      if (st.coop) {
        if (uses_any(set.idcs, tsyms) || written_nodes.count(set.tn) || rownodes.count(set.tn)) ok = false;
        for (auto& ix : set.idcs)
          if (ix.kind != Index::Iter && ix.kind != Index::Fixed) ok = false;
        scalars[set.tn] = {set.idcs, (int)k};
      } else {
        if (!row_position(set.tn, set.idcs) || written_nodes.count(set.tn)) ok = false;
        else note_row(set.tn, set.idcs, true);
      }
      written_nodes.insert(set.tn);
      if (!ok) return false;
    }
    if ((int64_t)rownodes.size() * EPL > 160) return false;   // the rows have to fit the registers
    // a node read at other positions by a LATER plain load after being written here was refused above;
    // a row node that is both loaded and produced was refused as well

    // ---- emit
    Stage f;
    f.kind = Stage::Generic;
    f.kernel = code.stages[run.front()].kernel;
    f.block = 256;
    f.total = rows;
    f.coop = 32;
    merge_origins(f, run);
    Emitter em(code.prog);
    em.large_models = opt.large_models;
    em.unroll_loops = true;
    std::set<int> written;
    for (size_t i : run) {
      const Piece& pc = pieces[i];
      em.used_nodes.insert(pc.used.begin(), pc.used.end());
      written.insert(pc.written.begin(), pc.written.end());
      em.uses_merge |= pc.uses_merge;
    }
    int max_bytes = 4;
    auto reg = [](int tn) { return "b200_row" + std::to_string(tn); };
    // Which elements of a row a lane owns.  Four at a time, dealt round the warp (element
    // (k * 32 + lane) * 4 + j in register 4 k + j) when the lane's share is a multiple of four: every
    // access of the warp then covers one contiguous stretch of the row.  A share of two elements stays
    // consecutive (lane * 2 + e).  Rows of any other length go one element per lane and step (element e * 32 +
    // lane in register e), the lanes beyond the row's end idle in the last step.
    const std::string own = dealt ? "(((b200_e >> 2) * 32u + b200_t) * 4u + (b200_e & 3u))" : strided ? "(b200_e * 32u + b200_t)" : "(b200_t0 + b200_e)";
    const std::string Rs = std::to_string(R);
    auto row_ptr = [&](int tn, const RowNode& rn) {
      const Tnode& t = code.prog.tn(tn);
      Indices at = rn.idcs;
      Index zero;
      at.push_back(zero);
      return t.ident + " + (" + em.offset(at, t.dims) + ")" + (pairwise ? " + b200_t0" : "");
    };
    auto ld = [&](int tn, const RowNode& rn) {
      const std::string n = std::to_string(EPL);
      if (strided)
        return "#pragma unroll\n    for (unsigned int b200_e = 0; b200_e < " + n + "u; ++b200_e) " + reg(tn) + "[b200_e] = " + (tail ? own + " < " + Rs + "u ? " : std::string()) +
               Emitter::load_wrap(rn.prec, "(" + row_ptr(tn, rn) + ")[" + own + "]") + (tail ? " : 0.0f" : "") + ";\n";
      max_bytes = std::max(max_bytes, dealt ? 4 * prec_bytes(rn.prec) : std::min(16, EPL * prec_bytes(rn.prec)));
      const std::string lane = dealt ? "b200_t, " : "";
      if (rn.prec == Prec::Single) return std::string("    b200_ld_row") + (dealt ? "v<" : "<") + n + ">(" + row_ptr(tn, rn) + ", " + lane + reg(tn) + ");\n";
      return std::string("    b200_ld_row") + (dealt ? "v16<" : "16<") + n + ", " + (rn.prec == Prec::Half ? "true" : "false") + ">(" + row_ptr(tn, rn) + ", " + lane + reg(tn) + ");\n";
    };
    auto stv = [&](int tn, const RowNode& rn) {
      const std::string n = std::to_string(EPL);
      if (strided)
        return "#pragma unroll\n    for (unsigned int b200_e = 0; b200_e < " + n + "u; ++b200_e)" + (tail ? " if (" + own + " < " + Rs + "u)" : std::string()) + " (" + row_ptr(tn, rn) + ")[" + own +
               "] = " + Emitter::store_wrap(rn.prec, reg(tn) + "[b200_e]") + ";\n";
      max_bytes = std::max(max_bytes, dealt ? 4 * prec_bytes(rn.prec) : std::min(16, EPL * prec_bytes(rn.prec)));
      const std::string lane = dealt ? "b200_t, " : "";
      if (rn.prec == Prec::Single) return std::string("    b200_st_row") + (dealt ? "v<" : "<") + n + ">(" + row_ptr(tn, rn) + ", " + lane + reg(tn) + ");\n";
      return std::string("    b200_st_row") + (dealt ? "v16<" : "16<") + n + ", " + (rn.prec == Prec::Half ? "true" : "false") + ">(" + row_ptr(tn, rn) + ", " + lane + reg(tn) + ");\n";
    };
    // rows that are the same for every row of the kernel (a scale, a shift: no row symbol in their
    // position) are loaded once per warp, before the loop over the warp's rows
    auto row_invariant = [&](const RowNode& rn) {
      if (rn.produced) return false;
      for (auto& ix : rn.idcs)
        if (ix.kind != Index::Fixed) return false;
      return true;
    };
    std::string text, decls, pre_decls, pre_text;
    bool any_invariant = false;
    for (auto& kv : rownodes) {
      const std::string d = "    float " + reg(kv.first) + "[" + std::to_string(EPL) + "];\n";
      if (row_invariant(kv.second)) { pre_decls += d; any_invariant = true; }
      else decls += d;
    }
    std::set<int> have;
    auto forwards = [&]() {
      em.row_forwards.clear();
      for (auto& kv : rownodes) {
        Indices idcs = kv.second.idcs;
        Index any;
        idcs.push_back(any);
        em.row_forwards.push_back({kv.first, idcs, (int)idcs.size() - 1, reg(kv.first), " - b200_t0", "b200_e"});   // (every element loop below runs over b200_e)
      }
    };
    forwards();
    for (size_t k = 0; k < stages.size(); ++k) {
      const RegRowStage& st = stages[k];
      const Stmt& set = *st.set;
      const Tnode& T = code.prog.tn(set.tn);
      // rows this stage reads that are not in registers yet
      walk_scalar(*set.value, [&](const Scalar& e) {
        if (e.kind != Scalar::Get) return;
        auto it = rownodes.find(e.tn);
        if (it == rownodes.end() || it->second.produced || have.count(e.tn)) return;
        bool positional = !e.idcs.empty() && e.idcs.back().kind == Index::Iter &&
                          (e.idcs.back().sym == st.t_sym || std::count(st.scope_syms.begin(), st.scope_syms.end(), e.idcs.back().sym));
        if (!positional) return;
        if (row_invariant(it->second)) pre_text += ld(e.tn, it->second);
        else text += ld(e.tn, it->second);
        have.insert(e.tn);
      }, [](const Stmt&) {});
      if (st.coop) {
        text += "    {\n";
        size_t si = 0;
        std::function<void(const Scalar&)> rec = [&](const Scalar& e) {
          if (e.kind == Scalar::LocalScope) {
            std::string op;
            for (auto& sc : st.scopes)
              if (sc.first == e.scope_id) op = sc.second;
            const Prec p = code.prog.tn(e.tn).prec;
            const Stmt* b = e.body.get();
            if (b->kind == Stmt::Seq) b = b->items[1].get();
            const std::string name = em.scope_name(e.scope_id, e.tn);
            const double neutral = op == "add" ? 0.0 : (op == "max" ? -INFINITY : INFINITY);
            text += "      " + std::string(Emitter::ctype(p)) + " " + name + " = " + em.constant(neutral, p) + ";\n";
            text += "#pragma unroll\n      for (unsigned int b200_e = 0; b200_e < " + std::to_string(EPL) + "u; ++b200_e) {\n"
                    "        const unsigned int " + b->index + " = " + own + ";\n" + (tail ? "        if (" + b->index + " < " + Rs + "u) {\n" : std::string()) +
                    em.stmt(*b->body, 8) + (tail ? "        }\n" : "") + "      }\n";
            text += "      " + name + " = b200_warp_" + (op == "add" ? std::string("sum") : op) + "(" + name + ");\n";
            em.scope_subst[e.scope_id] = name;
            ++si;
            return;
          }
          for (auto& a : e.args) rec(*a.s);
        };
        rec(*set.value);
        Emitter::Res v = em.scalar(T.prec, *set.value);
        em.scope_subst.clear();
        const std::string sname = "b200_val" + std::to_string(set.tn);
        decls += "    " + std::string(Emitter::rtype(T.prec)) + " " + sname + ";\n";
        text += "      " + sname + " = " + v.expr + ";\n";
        text += "      if (b200_t == 0u) " + T.ident + "[" + em.offset(set.idcs, T.dims) + "] = " + Emitter::store_wrap(T.prec, sname) + ";\n";
        text += "    }\n";
        em.forwarded[set.tn] = {set.idcs, sname};     // every lane holds the value after the shuffle tree
      } else {
        em.set_redirect[set.tn] = {set.idcs, reg(set.tn) + "[b200_e]"};
        const std::string loop_head = "#pragma unroll\n    for (unsigned int b200_e = 0; b200_e < " + std::to_string(EPL) + "u; ++b200_e) {\n"
                                      "      const unsigned int " + st.t_sym + " = " + own + ";\n";
        // divisors that are the same for the whole row (a standard deviation, a sum) are prepared
        // once: reciprocal and range check per row, a short exact sequence per element
        std::vector<std::string> probe;
        em.divisor_probe = &probe;
        const std::string body_plain = em.stmt(set, 6);
        em.divisor_probe = nullptr;
        std::vector<std::string> inv;
        for (auto& d : probe)
          if (d.find('[') == std::string::npos && d.find(st.t_sym) == std::string::npos && d.find("b200_e") == std::string::npos &&
              std::find(inv.begin(), inv.end(), d) == inv.end())
            inv.push_back(d);
        if (!inv.empty()) {
          std::string all_fast;
          text += "    {\n";
          for (size_t q = 0; q < inv.size(); ++q) {
            const std::string nm = "b200_dv" + std::to_string(set.tn) + "_" + std::to_string(q);
            text += "    const b200_divisor " + nm + " = b200_divisor_of(" + inv[q] + ");\n";
            em.divisor_vars[inv[q]] = nm;
            all_fast += (q ? " && " : "") + nm + ".fast";
          }
          const std::string body_fast = em.stmt(set, 6);
          em.divisor_vars.clear();
          text += "    if (" + all_fast + ") {\n" + loop_head + body_fast + "    }\n    } else {\n" + loop_head + body_plain + "    }\n    }\n    }\n";
        } else {
          text += loop_head + body_plain + "    }\n";
        }
        em.set_redirect.erase(set.tn);
        text += stv(set.tn, rownodes[set.tn]);
        have.insert(set.tn);
      }
    }
    f.min_align = strided ? 0 : max_bytes;
    std::string statics = static_prologue(text, em, 2);
    std::ostringstream k_src;
    k_src << "extern \"C\" __global__ void __launch_bounds__(" << f.block << ") " << f.kernel << "(";
    emit_params(k_src, f, em, written);
    k_src << ") {\n" << kGridEntry << statics
          << "  const unsigned int b200_t = threadIdx.x & 31u;\n  const unsigned int b200_t0 = b200_t * " << EPL << "u;\n"
          << "  const unsigned long long b200_warp = ((unsigned long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;\n"
          << "  const unsigned long long b200_nwarps = ((unsigned long long)gridDim.x * blockDim.x) >> 5;\n"
          << pre_decls << pre_text
          << "  for (unsigned long long b200_row = b200_warp; b200_row < " << rows << "ull; b200_row += b200_nwarps) {\n";
    {
      std::string rem = "b200_row";
      for (size_t q = L; q-- > 0;) {
        const std::string ext = std::to_string(first.par[q].extent()) + "ull";
        k_src << "    const unsigned int " << canon[q] << " = (unsigned int)" << (q == 0 ? rem : "(" + rem + " % " + ext + ")") << ";\n";
        if (q != 0) {
          k_src << "    const unsigned long long b200_q" << q << " = " << rem << " / " << ext << ";\n";
          rem = "b200_q" + std::to_string(q);
        }
      }
    }
    k_src << decls << text << "  }\n}\n\n";
    src << k_src.str();
    // with rows loaded once per warp, a warp takes several rows: as many blocks as stay resident on 148
    // SMs (three of 256 threads at this kernel's register use), each warp striding over the rows
    if (any_invariant && rows >= 2 * 148 * 3 * 8) f.grid_override = 148 * 3;
    f.note = "row-fused " + std::to_string(run.size()) + " stages, one warp per row, rows in registers (" + std::to_string(EPL) +
             " elements per lane" + (dealt ? ", dealt four at a time" : strided ? ", one per step" : "") + ")";
    *out = f;
    return true;
  }

  // Row fusion.  Consecutive stages whose outermost parallel loop has the same extent, and which
  // hand data to one another only within one iteration of that loop (every node written by one
  // of them and touched by another is indexed by the row symbol on one fixed axis, nowhere else),
  // run as ONE kernel: a thread takes a row and executes the stages one after the other for it,
  // the inner parallel loops of each stage becoming short serial loops.  A softmax over ten
  // logits (row max, exponentials, row sum) is one launch and one pass instead of three.
  bool rows_independent(const std::vector<size_t>& run) {
    std::map<int, int> writers, users;  // node -> number of stages writing / touching it
    for (size_t i : run) {
      const Piece& pc = pieces[i];
      for (int n : pc.written) writers[n]++;
      for (int n : pc.used) users[n]++;
    }
    std::map<int, int> axis;  // shared node -> axis that carries the row symbol
    bool ok = true;
    for (size_t i : run) {
      const Piece& pc = pieces[i];
      auto check = [&](int tn, const Indices& idcs) {
        if (!writers.count(tn) || users[tn] < 2) return;   // private to one stage, or only read
        int a = -1;
        for (size_t k = 0; k < idcs.size(); ++k) {
          if (idcs[k].kind == Index::Iter && idcs[k].sym == pc.row_sym && a < 0) a = (int)k;
          else if (idcs[k].uses(pc.row_sym)) ok = false;
        }
        if (a < 0) { ok = false; return; }
        auto it = axis.find(tn);
        if (it == axis.end()) axis[tn] = a;
        else if (it->second != a) ok = false;
      };
      walk_stmt(
          *pc.body,
          [&](const Scalar& e) {
            if (e.kind == Scalar::Get) check(e.tn, e.idcs);
            if (e.kind == Scalar::GetDyn && writers.count(e.tn) && users[e.tn] >= 2) ok = false;
          },
          [&](const Stmt& st) {
            if (st.kind == Stmt::Set) {
              if (st.vec_len > 0 && writers.count(st.tn) && users[st.tn] >= 2) ok = false;
              check(st.tn, st.idcs);
            }
            if (st.kind == Stmt::ZeroOut) ok = false;
          });
    }
    return ok;
  }

  Stage emit_rows(const std::vector<size_t>& run) {
    Stage f;
    merge_origins(f, run);
    f.kind = Stage::Generic;
    f.kernel = code.stages[run.front()].kernel;
    f.block = 128;
    f.total = pieces[run.front()].rows;
    Emitter em(code.prog);
    std::set<int> written;
    std::string text;
    for (size_t i : run) {
      const Stage& st = code.stages[i];
      const Piece& pc = pieces[i];
      f.min_align = std::max(f.min_align, st.min_align);
      em.used_nodes.insert(pc.used.begin(), pc.used.end());
      written.insert(pc.written.begin(), pc.written.end());
      em.uses_merge |= pc.uses_merge;
      const std::string inner = std::to_string(st.total / pc.rows) + "ull";
      text += "    for (unsigned long long b200_g = b200_row * " + inner + "; b200_g < (b200_row + 1ull) * " + inner +
              "; ++b200_g) {\n" + pc.decomp + pc.body_text + "    }\n";
    }
    std::string statics = static_prologue(text, em, 2);
    std::ostringstream k_src;
    k_src << "extern \"C\" __global__ void __launch_bounds__(" << f.block << ") " << f.kernel << "(";
    emit_params(k_src, f, em, written);
    k_src << ") {\n" << kGridEntry << statics
          << "  for (unsigned long long b200_row = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; b200_row < "
          << f.total << "ull; b200_row += (unsigned long long)gridDim.x * blockDim.x) {\n"
          << text << "  }\n}\n\n";
    src << k_src.str();
    f.note = "row-fused " + std::to_string(run.size()) + " stages, one thread per row";
    return f;
  }

  // Pointwise chain.  Consecutive stages over the SAME parallel loops (no serial loops, no
  // cooperative reductions) that hand data to one another only at one position of those loops
  // run as one kernel: a thread executes the stages one after the other for its element (or
  // pair).  What one stage stores the next reads back from L1 / L2 instead of DRAM, and a
  // momentum SGD step (delta, momentum, Nesterov correction, parameter) is one launch per
  // parameter instead of four.
  bool pointwise_member(size_t i, const Piece* like) {
    auto it = pieces.find(i);
    if (it == pieces.end() || !it->second.any_body) return false;
    const Piece& pc = it->second;
    if (pc.coop != 0 || pc.ser_work != 1 || pc.par.empty() || code.stages[i].total <= 0) return false;
    for (auto& d : pc.par)
      if (d.from != 0) return false;
    if (like) {
      if (pc.par.size() != like->par.size() || pc.pairs != like->pairs) return false;
      for (size_t q = 0; q < pc.par.size(); ++q)
        if (pc.par[q].extent() != like->par[q].extent()) return false;
    }
    return true;
  }

  Stage emit_pointwise_chain(const std::vector<size_t>& run) {
    Stage f = code.stages[run.front()];
    merge_origins(f, run);
    Emitter em(code.prog);
    std::set<int> written;
    std::string text;
    for (size_t i : run) {
      const Piece& pc = pieces[i];
      f.min_align = std::max(f.min_align, code.stages[i].min_align);
      em.used_nodes.insert(pc.used.begin(), pc.used.end());
      written.insert(pc.written.begin(), pc.written.end());
      em.uses_merge |= pc.uses_merge;
      text += "    {\n" + pc.decomp + pc.body_text + "    }\n";
    }
    std::string statics = static_prologue(text, em, 2);
    std::ostringstream k_src;
    k_src << "extern \"C\" __global__ void __launch_bounds__(" << f.block << ") " << f.kernel << "(";
    emit_params(k_src, f, em, written);
    k_src << ") {\n" << kGridEntry << statics
          << "  for (unsigned long long b200_g = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; b200_g < "
          << f.total << "ull; b200_g += (unsigned long long)gridDim.x * blockDim.x) {\n"
          << text << "  }\n}\n\n";
    src << k_src.str();
    f.note = "pointwise chain of " + std::to_string(run.size()) + " stages" + (pieces[run.front()].pairs ? ", pairs" : "");
    return f;
  }

  // Pointwise chains that do not depend on one another -- the updates of a routine's parameters -- as one launch.  Small ones
  // over their concatenated iterations, every chain beginning at a multiple of a warp's 32.  Where a chain has more
  // than a few rounds of a launch's threads, each has a range of the blocks instead, as many as its own launch would have, and
  // the loop that it would have there: one that tells the chains apart in its body is not unrolled.  (Updates of
  // n-n-n-10, us, a launch each / concatenated / ranges: n = 1024 in bf16 9.9 / 5.3 / 5.5, 1448 10.4 / 5.5 / 6.6, 1023 11.7 /
  // 6.2 / 7.4; 2048 14.0 / 9.3 / 7.7, 2047 18.6 / 19.0 / 14.8, 2895 35.6 / 42.2 / 35.1, 4096 47.8 / 53.1 / 48.5; with
  // momentum 4096 131.8 / 132.1 / 128.4.  Working sets next to the size of L2 may be better off one by one: 2895 in single
  // precision 36.7 / 49.1 / 44.0.)  The plan lists what is in it as stages: a large chain each, neighbouring small ones together.
  void emit_pointwise_group(const std::vector<std::vector<size_t>>& parts, std::vector<Stage>* out) {
    std::vector<size_t> all;
    for (auto& run : parts) all.insert(all.end(), run.begin(), run.end());
    Stage f = code.stages[all.front()];
    f.min_align = 0;
    merge_origins(f, all);
    Emitter em(code.prog);
    std::set<int> written;
    std::string text;
    int64_t most = 0, threads = 0, first = 0;   // iterations of a chain, of all of them; blocks
    for (auto& run : parts) most = std::max(most, code.stages[run.front()].total);
    const bool ranges = most > 3 << 19;
    for (auto& run : parts) {
      const int64_t total = code.stages[run.front()].total, blocks = std::min<int64_t>((total + f.block - 1) / f.block, 148 * 16);
      text += std::string("    ") + (first ? "else " : "");
      if (ranges)
        text += "if (blockIdx.x < " + std::to_string(first + blocks) + "u) {\n    for (unsigned long long b200_g = (unsigned long long)(blockIdx.x - " + std::to_string(first) +
                "u) * blockDim.x + threadIdx.x; b200_g < " + std::to_string(total) + "ull; b200_g += " + std::to_string(blocks) + "ull * blockDim.x) {\n";
      else
        text += "if (b200_i < " + std::to_string(threads + total) + "ull) {\n    if (b200_i >= " + std::to_string(threads) + "ull) {\n    const unsigned long long b200_g = b200_i - " +
                std::to_string(threads) + "ull;\n";
      // (a parameter off its boundary takes its own chain's pairs away, not those of the others in the launch)
      Stage::AlignNeed need{0, {}, {}};
      for (size_t i : run) {
        const Piece& pc = pieces[i];
        need.bytes = std::max(need.bytes, code.stages[i].min_align);
        need.nodes.insert(need.nodes.end(), pc.used.begin(), pc.used.end());
        need.origins.insert(need.origins.end(), code.stages[i].origins.begin(), code.stages[i].origins.end());
        em.used_nodes.insert(pc.used.begin(), pc.used.end());
        written.insert(pc.written.begin(), pc.written.end());
        em.uses_merge |= pc.uses_merge;
        text += "    {\n" + pc.decomp + pc.body_text + "    }\n";
      }
      if (need.bytes > 1) f.needs.push_back(need);
      text += "    }\n    }\n";
      threads = (threads + total + 31) / 32 * 32;
      first += blocks;
    }
    if (ranges) f.grid_override = (int)first;
    std::string statics = static_prologue(text, em, 2);
    std::ostringstream k_src;
    k_src << "extern \"C\" __global__ void __launch_bounds__(" << f.block << ") " << f.kernel << "(";
    emit_params(k_src, f, em, written);
    k_src << ") {\n" << kGridEntry << statics;
    if (!ranges)
      k_src << "  for (unsigned long long b200_i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; b200_i < " << threads
            << "ull; b200_i += (unsigned long long)gridDim.x * blockDim.x) {\n";
    k_src << text << (ranges ? "}\n\n" : "  }\n}\n\n");
    src << k_src.str();
    std::vector<std::vector<size_t>> listed;
    bool small_before = false;
    for (auto& run : parts) {
      const bool small = small_chain(run);
      if (small && small_before) listed.back().insert(listed.back().end(), run.begin(), run.end());
      else listed.push_back(run);
      small_before = small;
    }
    f.group = (int)listed.size();
    for (size_t k = 0; k < listed.size(); ++k) {
      const std::vector<size_t>& run = listed[k];
      Stage st = code.stages[run.front()];
      std::set<int> used;
      for (size_t i : run) used.insert(pieces[i].used.begin(), pieces[i].used.end());
      merge_origins(st, run);
      if (small_chain(run) && run.size() > 1) st.note = "fused " + std::to_string(run.size()) + " small stages";
      else if (run.size() > 1) st.note = "pointwise chain of " + std::to_string(run.size()) + " stages" + (pieces[run.front()].pairs ? ", pairs" : "");
      if (k == 0) {
        f.note = st.note;
        f.total = threads;
        out->push_back(f);
      } else {
        st.note += " (in the launch of " + f.kernel + ")";
        st.in_group = true;
        st.min_align = 0;
        st.args.clear();
        for (int n : used) st.args.push_back({KArg::Node, n});
        out->push_back(st);
      }
    }
  }
  // a chain that one block could take with others
  bool small_chain(const std::vector<size_t>& run) {
    bool small = true;
    for (size_t i : run) small = small && pieces[i].fusable && code.stages[i].total < 8192;
    return small;
  }

  // Decides which stages share a launch and writes the kernels' text.
  void emit_kernels() {
    {
      // zero_outs that later stages made unnecessary leave the list (pieces are keyed by stage index)
      std::vector<Stage> kept;
      std::map<size_t, Piece> moved;
      for (size_t i = 0; i < code.stages.size(); ++i) {
        if (code.stages[i].kind == Stage::Memset && code.stages[i].memset_tn < 0) continue;
        auto it = pieces.find(i);
        if (it != pieces.end()) moved[kept.size()] = it->second;
        kept.push_back(code.stages[i]);
      }
      code.stages.swap(kept);
      pieces.swap(moved);
    }
    note_node_stages();
    std::vector<Stage> out;
    auto fusable = [&](size_t i) {
      const Stage& st = code.stages[i];
      if (st.kind == Stage::Memset) {
        const Tnode& t = code.prog.tn(st.memset_tn);
        return opt.enable_fuse && t.bytes() <= 262144 && prec_bytes(t.prec) <= 8 && t.prec != Prec::Uint4x32;
      }
      auto it = pieces.find(i);
      return it != pieces.end() && it->second.fusable;
    };
    // The pointwise chain that starts at stage i.  Where one block could take the stages too, a chain counts
    // from three stages over 8192 threads on: the momentum update of a 300 x 100 layer took that block 30 us.
    auto chain_from = [&](size_t i) {
      std::vector<size_t> run;
      const bool long_chain = code.stages[i].kind == Stage::Generic && code.stages[i].total >= 8192;
      if ((fusable(i) && !long_chain) || !pointwise_member(i, nullptr)) return run;
      const Piece& first = pieces[i];
      run = {i};
      size_t j = i + 1;
      while (j < code.stages.size() && run.size() < 8 && pointwise_member(j, &first)) {
        run.push_back(j);
        if (!rows_independent_prefix(run, first.par.size())) { run.pop_back(); break; }
        ++j;
      }
      return run;
    };
    // Chains that do not depend on one another, from stage i on, where at least one is too large for a block: one launch
    // instead of a kernel each and a block for the small ones in between.
    auto group_from = [&](size_t i) {
      std::vector<std::vector<size_t>> parts;
      std::set<int> used, written;
      bool large = false;
      size_t j = opt.bounds ? code.stages.size() : i;
      while (j < code.stages.size() && parts.size() < 16 && pointwise_member(j, nullptr)) {
        std::vector<size_t> run = {j};
        const Piece& first = pieces[j];
        for (size_t k = j + 1; k < code.stages.size() && run.size() < 8 && pointwise_member(k, &first); ++k) {
          run.push_back(k);
          if (!rows_independent_prefix(run, first.par.size())) { run.pop_back(); break; }
        }
        bool apart_from_others = true;
        for (size_t k : run) {
          for (int n : pieces[k].written) apart_from_others = apart_from_others && !used.count(n) && !written.count(n);
          for (int n : pieces[k].used) apart_from_others = apart_from_others && !written.count(n);
        }
        if (!apart_from_others) break;
        for (size_t k : run) {
          used.insert(pieces[k].used.begin(), pieces[k].used.end());
          written.insert(pieces[k].written.begin(), pieces[k].written.end());
        }
        large = large || !small_chain(run);
        parts.push_back(run);
        j = run.back() + 1;
      }
      if (!large || parts.size() < 2) parts.clear();
      return parts;
    };
    auto row_candidate = [&](size_t i) {
      auto it = pieces.find(i);
      return it != pieces.end() && it->second.body && it->second.rows >= 256 && it->second.per_row <= 64;
    };
    for (size_t i = 0; i < code.stages.size();) {
      if (opt.enable_fuse && pieces.count(i) && pieces[i].any_body && (pieces[i].coop == 0 || pieces[i].coop == 32)) {
        // the row is given by the first warp-cooperative stage of the run
        size_t L = 0;
        for (size_t j = i; j < code.stages.size() && j < i + 16; ++j) {
          auto it = pieces.find(j);
          if (it == pieces.end()) break;
          if (it->second.coop == 32) { L = it->second.par.size(); break; }
          if (it->second.coop != 0) break;
        }
        if (L > 0 && warp_row_member(i, L, nullptr)) {
          const Piece& first = pieces[i];
          int64_t rows = 1;
          for (size_t q = 0; q < L; ++q) rows *= first.par[q].extent();
          std::vector<size_t> run = {i};
          bool has_coop = first.coop == 32;
          size_t j = i + 1;
          while (j < code.stages.size() && run.size() < 16 && warp_row_member(j, L, &first)) {
            run.push_back(j);
            if (!rows_independent_prefix(run, L)) { run.pop_back(); break; }
            has_coop = has_coop || pieces[j].coop == 32;
            ++j;
          }
          // a trailing pointwise stage gains nothing from the warp form unless it follows a reduction
          // Fewer than 128 rows may go to one block, whose four passes over 100 rows of 256 take 8 us longer than a warp
          // a row in registers (decoders of two layers, 100 x 256: 93.7 -> 60.5 us; 16 x 128: 47.4 -> 39.0).  It is left to the
          // block when that takes stages behind the rows as well (a loss) and the rows are short: a launch
          // less then counts more (20 rows of 40: 13.7 us, 16.4 with a warp a row; 100 of 64: 18.5 and 16.4).
          const bool block_goes_on = run.back() + 1 < code.stages.size() && fusable(run.back()) && fusable(run.back() + 1);
          const int64_t elems = rows * std::max(code.stages[i].total / rows, code.stages[run.back()].total / rows);
          if (run.size() >= 2 && has_coop && (rows >= 128 || (rows >= 8 && (!block_goes_on || elems >= 4096)))) {
            Stage reg_form;
            const bool in_registers = emit_warp_rows_reg(run, L, &reg_form);
            if (in_registers || rows >= 128) {
              out.push_back(in_registers ? reg_form : emit_warp_rows(run, L));
              i = run.back() + 1;
              continue;
            }
          }
        }
      }
      if (opt.enable_fuse) {
        const std::vector<std::vector<size_t>> parts = group_from(i);
        if (!parts.empty()) {
          emit_pointwise_group(parts, &out);
          i = parts.back().back() + 1;
          continue;
        }
      }
      if (row_candidate(i)) {
        // the longest run that stays row-independent; runs made only of small stages are left to
        // the single-block fusion below, which also takes stages of unrelated shapes
        std::vector<size_t> run = {i};
        size_t j = i + 1;
        bool all_small = fusable(i);
        while (j < code.stages.size() && row_candidate(j) && pieces[j].rows == pieces[i].rows && run.size() < 16) {
          run.push_back(j);
          if (!rows_independent(run)) { run.pop_back(); break; }
          all_small = all_small && fusable(j);
          ++j;
        }
        if (run.size() >= 2 && !all_small) {
          out.push_back(emit_rows(run));
          i = run.back() + 1;
          continue;
        }
      }
      // (a long chain over thousands of elements -- the momentum update of a 300 x 100 layer -- is a kernel of
      // its own even where one block could take it: that block spent 30 us on four passes over it)
      if (opt.enable_fuse) {
        const std::vector<size_t> run = chain_from(i);
        if (run.size() >= (fusable(i) ? 3u : 2u)) {
          out.push_back(emit_pointwise_chain(run));
          i = run.back() + 1;
          continue;
        }
      }
      // Clears in a row are one kernel, which nothing before them holds up: in a captured graph every clear of its own was a
      // node on some branch (2706 rows through 141-82-270-5, a training step: 65 us with five of them, 53 so; 8192 of 784-1024-1024-10 143.1 and 133.4).
      // Not the largest: the driver's clear has the higher bandwidth (two nodes each, us, by the driver / as a kernel: 2^23 floats
      // 12.4 / 10.5, 2^24 21.0 / 22.0, 2^26 76 / 90; 2^24 values of 16 bits 12.5 / 11.3, 2^25 22.3 / 23.0; 2^24 bytes 8.3 / 7.8, 2^25 12.5 / 14.0).
      if (opt.enable_fuse && code.stages[i].kind == Stage::Memset) {
        std::vector<size_t> run;
        std::set<int> cleared;   // (a second clear of the same node has to wait for the first: one block would do both)
        size_t j = i;
        for (; j < code.stages.size() && code.stages[j].kind == Stage::Memset; ++j) {
          const Tnode& t = code.prog.tn(code.stages[j].memset_tn);
          if (prec_bytes(t.prec) > 8 || t.prec == Prec::Uint4x32 || t.num_elems() > (1 << 24) || t.bytes() > (1 << 25) || !cleared.insert(t.id).second) break;
          run.push_back(j);
        }
        // (those that stages behind them join share a launch with these anyway)
        if (run.size() >= 2 && !(j < code.stages.size() && fusable(j) && code.stages[j].kind != Stage::Memset)) {
          Stage lead = emit_fused(run);
          lead.clears = true;
          lead.group = (int)run.size();
          lead.note = "zero_out";
          out.push_back(lead);
          for (size_t k = 1; k < run.size(); ++k) {   // listed as the clears they are
            Stage st = code.stages[run[k]];
            st.kind = Stage::Generic;
            st.clears = st.in_group = true;
            st.writes = {st.memset_tn};
            st.note = "zero_out (in the launch of " + lead.kernel + ")";
            out.push_back(st);
          }
          i = j;
          continue;
        }
      }
      if (fusable(i)) {
        // A sum by the whole block joins the stages whose values it sums; where it comes first, only what reads it follows
        // (the first pointwise steps of a gradient have nothing to do with the loss and are better off over a grid).
        std::vector<size_t> run;
        std::set<int> run_writes;
        auto depends = [&](size_t k) {
          auto p = pieces.find(k);
          if (p == pieces.end()) return false;
          for (int n : p->second.used)
            if (run_writes.count(n)) return true;
          return false;
        };
        size_t j = i;
        while (j < code.stages.size() && fusable(j) && (j == i || (chain_from(j).size() < 3 && group_from(j).empty()))) {
          if (j > i && (code.stages[i].coop > 32 || code.stages[j].coop > 32) && !depends(j)) break;
          run_writes.insert(code.stages[j].writes.begin(), code.stages[j].writes.end());
          if (code.stages[j].kind == Stage::Memset) run_writes.insert(code.stages[j].memset_tn);
          run.push_back(j++);
        }
        int kernels = 0;
        for (size_t k : run) kernels += code.stages[k].kind != Stage::Memset;
        if (run.size() >= 2 && kernels >= 1) {
          out.push_back(emit_fused(run));
          i = j;
          continue;
        }
      }
      Stage st = code.stages[i];
      auto it = pieces.find(i);
      if (it != pieces.end()) emit_single(st, it->second);
      out.push_back(st);
      ++i;
    }
    code.stages = out;
  }

  // A group of threads per output element: each Local_scope reduction runs over its flattened
  // loop space strided by the group width, partial results are combined with shuffles (and
  // shared memory across warps), and thread 0 of the group evaluates and stores the rest.
  std::string coop_body(Emitter& em, const Stmt& set, const CoopInfo& ci, int ind, bool unroll) {
    std::string out;
    std::string padding((size_t)ind, ' ');
    const Tnode& t = code.prog.tn(set.tn);
    std::function<void(const Scalar&)> rec = [&](const Scalar& e) {
      if (e.kind == Scalar::LocalScope) {
        std::string op;
        for (auto& s : ci.scopes)
          if (s.first == e.scope_id) op = s.second;
        Prec p = code.prog.tn(e.tn).prec;
        const Stmt& b = *e.body;
        const Stmt* loop = b.kind == Stmt::For ? &b : b.items[1].get();
        std::vector<LoopDim> red;
        const Stmt* inner = loop;
        while (inner->kind == Stmt::For) {
          red.push_back({inner->index, inner->from, inner->to});
          inner = inner->body.get();
        }
        int64_t total = 1;
        for (auto& d : red) total *= d.extent();
        std::string name = em.scope_name(e.scope_id, e.tn);
        double neutral = op == "add" ? 0.0 : (op == "max" ? -INFINITY : INFINITY);
        out += padding + Emitter::ctype(p) + " " + name + " = " + em.constant(neutral, p) + ";\n";
        std::string lv = "b200_l" + std::to_string(e.scope_id);
        const bool narrow = total < (1ll << 31);
        const std::string IT = narrow ? "unsigned int" : "unsigned long long", SUF = narrow ? "u" : "ull";
        std::string step;
        std::string rem = lv;
        for (size_t i = red.size(); i-- > 0;) {
          const LoopDim& d = red[i];
          std::string ext = std::to_string(d.extent()) + SUF;
          std::string val = i == 0 ? rem : "(" + rem + " % " + ext + ")";
          step += padding + "  const unsigned int " + d.sym + " = (unsigned int)" + val +
                  (d.from ? " + " + std::to_string(d.from) : std::string()) + ";\n";
          if (i != 0) {
            std::string nr = "b200_q" + std::to_string(e.scope_id) + "_" + std::to_string(i);
            step += padding + "  const " + IT + " " + nr + " = " + rem + " / " + ext + ";\n";
            rem = nr;
          }
        }
        step += em.stmt(*inner, ind + 2);
        // The lanes take the same whole number of steps, so that the loads of eight are under way together, and a shorter last
        // one: sums by a block, and a warp's of 256 terms and more in a kernel of their own (10 rows of 496-2032-200-14 in single precision 34 -> 19 us).
        // Not among other small stages, whose code runs once: two rows of 80-1832-382-55 took 16.6 us instead of 15.0.
        const int64_t whole = unroll ? total / ci.width : 0, rest = unroll ? total % ci.width : 0;
        if (!unroll)
          out += padding + "for (" + IT + " " + lv + " = b200_t; " + lv + " < " + std::to_string(total) + SUF + "; " + lv + " += " + std::to_string(ci.width) + "u) {\n" +
                 step + padding + "}\n";
        if (whole > 0) {
          out += "#pragma unroll 8\n" + padding + "for (" + IT + " " + lv + "_k = 0; " + lv + "_k < " + std::to_string(whole) + SUF + "; ++" + lv + "_k) {\n" + padding +
                 "  const " + IT + " " + lv + " = " + lv + "_k * " + std::to_string(ci.width) + SUF + " + b200_t;\n" + step + padding + "}\n";
        }
        if (rest > 0)
          out += padding + "if (b200_t < " + std::to_string(rest) + "u) {\n" + padding + "  const " + IT + " " + lv + " = " + std::to_string(whole * ci.width) + SUF +
                 " + b200_t;\n" + step + padding + "}\n";
        const std::string fn = op == "add" ? "sum" : op;
        if (ci.width > 32) out += padding + name + " = b200_block_" + fn + "(" + name + ", b200_red);\n";
        else out += padding + name + " = b200_warp_" + fn + "(" + name + ");\n";
        em.scope_subst[e.scope_id] = name;
        return;
      }
      for (auto& a : e.args) rec(*a.s);
    };
    rec(*set.value);
    Emitter::Res v = em.scalar(t.prec, *set.value);
    em.used_nodes.insert(set.tn);
    out += padding + "if (b200_t == 0) " + t.ident + "[" + em.offset(set.idcs, t.dims) + "] = " + Emitter::store_wrap(t.prec, v.expr) + ";\n";
    em.scope_subst.clear();
    return out;
  }

  // A node that a later stage only tests against zero (the mask of an attention stage), packed to
  // one bit per element: bit (i % 32) of word (i / 32) of its row's words = (element i != 0).  The bits
  // live in the routine's scratch; for a read-only node they are made once per run and shared by
  // every stage that asks for them.  Returns the byte offset in the reduction scratch.
  std::map<int, size_t> packed_bits;
  size_t pack_bits_stage(int tn) {
    const Tnode& t = code.prog.tn(tn);
    if (t.read_only) {
      auto it = packed_bits.find(tn);
      if (it != packed_bits.end()) return it->second;
    }
    // the bits of every row (last axis) start on a word of their own
    const long long len = t.dims.back(), row_words = (len + 31) / 32, words = t.num_elems() / len * row_words;
    const size_t off = code.reduce_scratch_bytes;
    code.reduce_scratch_bytes = (code.reduce_scratch_bytes + (size_t)words * 4 + 255) & ~(size_t)255;
    Stage st;
    st.kind = Stage::Generic;
    st.kernel = kernel_name();
    st.args = {{KArg::Node, tn}, {KArg::Scratch, (int)off}};
    st.total = words * 32;
    st.block = 256;
    st.note = "one bit per element: (value != 0), for the stages that only test this node";
    src << "extern \"C\" __global__ void __launch_bounds__(256) " << st.kernel << "(const " << Emitter::ctype(t.prec) << "* __restrict__ "
        << t.ident << ", unsigned char* b200_bits) {\n" << kGridEntry
        << "  unsigned int* b200_words = (unsigned int*)b200_bits;\n"
        << "  for (unsigned long long b200_i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; b200_i < " << words * 32
        << "ull; b200_i += (unsigned long long)gridDim.x * blockDim.x) {\n"
        << "    const unsigned long long b200_row = b200_i / " << row_words * 32 << "ull, b200_col = b200_i % " << row_words * 32 << "ull;\n"
        << "    const unsigned long long b200_at = b200_row * " << len << "ull + b200_col;\n"
        << "    const bool b200_nz = b200_col < " << len << "ull && " << Emitter::load_wrap(t.prec, t.ident + "[b200_at]") << " != 0;\n"
        << "    const unsigned int b200_w = __ballot_sync(0xffffffffu, b200_nz);\n"
        << "    if ((threadIdx.x & 31u) == 0u) b200_words[b200_i >> 5] = b200_w;\n  }\n}\n\n";
    code.stages.push_back(st);
    if (t.read_only) packed_bits[tn] = off;
    return off;
  }

  // Operands of a contraction that have to be gathered first (PackOp): one kernel fills the slots of both.
  // A thread owns 16 bytes of a packed row: it takes the row apart into the operand's loops once and
  // reads its 8 (4) elements one by one, so neither the alignment nor the layout of the node matters;
  // neighbouring threads read neighbouring elements wherever the node has a contiguous axis.
  // Contents are shared by the contractions of a routine (the three projections of an attention layer
  // read one input) until some stage writes the node.
  std::map<std::string, std::pair<int, size_t>> packed;   // key -> (slot, index of the stage that filled it)
  void pack_stage(Stage& g) {
    std::vector<const PackOp*> todo;
    std::vector<int> slots;
    for (auto& op : g.gemm.packs) {
      const std::string key = op.key();
      int slot = -1;
      auto it = packed.find(key);
      if (it != packed.end()) {
        slot = it->second.first;
        for (size_t i = it->second.second + 1; i < code.stages.size() && slot >= 0; ++i) {
          const Stage& st = code.stages[i];
          if (std::count(st.writes.begin(), st.writes.end(), op.tn)) slot = -1;
        }
      }
      if (slot < 0) {
        slot = (int)code.pack_bytes.size();
        code.pack_bytes.push_back((size_t)op.bytes());
        packed[key] = {slot, code.stages.size()};
        todo.push_back(&op);
        slots.push_back(slot);
      }
      (&op == &g.gemm.packs[0] && g.gemm.pack_a ? g.gemm.a_slot : g.gemm.b_slot) = slot;
    }
    g.copies = g.gemm.pack_a || g.gemm.pack_b;
    if (todo.empty()) return;
    // An operand that a pointwise stage makes, element by element, is gathered where it is made: the kernel takes that
    // stage's place, evaluates its expression, and stores the node as well as the copy.  (The embedding ahead of a
    // 30-200-27 character model, 4096 rows: 16.6 us -> 14.5; a convolution step of 64 images 68.6 -> 57.)
    Emitter em(code.prog);
    em.large_models = opt.large_models;
    int folded = -1;
    size_t at_stage = code.stages.size();
    Emitter::Res made;
    for (size_t i = 0; opt.enable_fuse && i < todo.size() && folded < 0; ++i) {
      const int j = pointwise_maker(*todo[i]);
      bool fits = j >= 0;
      for (auto* op : todo)
        for (size_t k = (size_t)std::max(j, 0); fits && k < code.stages.size(); ++k)
          if (op != todo[i] && (std::count(code.stages[k].writes.begin(), code.stages[k].writes.end(), op->tn) ||
                                (code.stages[k].kind == Stage::Memset && code.stages[k].memset_tn == op->tn)))
            fits = false;
      if (!fits) continue;
      made = em.scalar(code.prog.tn(todo[i]->tn).prec, *pieces[(size_t)j].any_body->value);
      if (!made.defs.empty()) { em.used_nodes.clear(); continue; }
      folded = (int)i;
      at_stage = (size_t)j;
    }
    Stage st;
    st.kind = Stage::Generic;
    st.kernel = folded >= 0 ? code.stages[at_stage].kernel : kernel_name();
    st.block = 256;
    std::ostringstream params, body;
    std::set<int> nodes = em.used_nodes;
    for (auto* op : todo) nodes.insert(op->tn);
    for (auto& t : code.prog.tnodes)
      if (nodes.count(t.id)) {
        const bool stored = folded >= 0 && t.id == todo[(size_t)folded]->tn;
        params << (params.tellp() > 0 ? ", " : "") << (stored ? "" : "const ") << Emitter::ctype(t.prec) << "* " << (stored ? "" : "__restrict__ ") << t.ident;
        st.args.push_back({KArg::Node, t.id});
      }
    int64_t total = 0;
    std::string what;
    for (size_t i = 0; i < todo.size(); ++i) {
      const PackOp& op = *todo[i];
      const std::string dst = "b200_pack" + std::to_string(slots[i]);
      params << ", uint4* __restrict__ " << dst;
      st.args.push_back({KArg::Pack, slots[i]});
      st.pack_writes.push_back(slots[i]);
      const int64_t first = total;
      total += op.rows() * op.ld * prec_bytes(op.prec) / ((int)i == folded ? 4 : 16) / (op.split ? 2 : 1);   // (a thread writes both parts)
      body << "    " << (i ? "else " : "") << "if (b200_g < " << total << "ull) {\n" << pack_body(op, dst, first, (int)i == folded ? &made : nullptr, at_stage) << "    }\n";
      what += (i ? ", " : "") + code.prog.tn(op.tn).label;
    }
    st.total = total;
    st.note = "gathers operands of the next contraction into padded rows" + std::string(g.gemm.tf32_pairs ? " (tf32 pairs)" : "") + ": " + what;
    src << "extern \"C\" __global__ void __launch_bounds__(256) " << st.kernel << "(" << params.str() << ") {\n" << kGridEntry
        << "  for (unsigned long long b200_g = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; b200_g < " << total
        << "ull; b200_g += (unsigned long long)gridDim.x * blockDim.x) {\n" << body.str() << "  }\n}\n\n";
    if (folded < 0) {
      code.stages.push_back(st);
      return;
    }
    st.note += " (" + code.prog.tn(todo[(size_t)folded]->tn).label + " where it is made)";
    st.writes = code.stages[at_stage].writes;
    st.origins = code.stages[at_stage].origins;
    st.origins.push_back(cur_origin);
    for (auto* op : todo) packed[op->key()].second = at_stage;
    code.stages[at_stage] = st;
    pieces.erase(at_stage);
  }
  // The stage that makes the operand's node by evaluating one expression per element, if it is the last to write it, the
  // operand takes every element of the node once, and nothing that the expression reads has changed since.  -1: none.
  int pointwise_maker(const PackOp& op) {
    const Tnode& t = code.prog.tn(op.tn);
    std::vector<PackOp::Axis> axes;
    for (auto* v : {&op.batch, &op.mn, &op.k})
      for (auto& a : *v)
        if (a.extent > 1) axes.push_back(a);
    std::sort(axes.begin(), axes.end(), [](const PackOp::Axis& a, const PackOp::Axis& b) { return a.stride < b.stride; });
    int64_t elems = 1;
    for (auto& a : axes) {
      if (a.stride != elems) return -1;
      elems *= a.extent;
    }
    if (op.off != 0 || elems != t.num_elems()) return -1;
    int j = -1;
    for (size_t i = code.stages.size(); i-- > 0 && j < 0;) {
      const Stage& st = code.stages[i];
      if (st.kind == Stage::Memset ? st.memset_tn == op.tn : std::count(st.writes.begin(), st.writes.end(), op.tn) > 0) j = (int)i;
    }
    if (j < 0 || code.stages[(size_t)j].kind != Stage::Generic || !pieces.count((size_t)j)) return -1;
    const Piece& pc = pieces[(size_t)j];
    if (code.stages[(size_t)j].total <= 0) return -1;   // (a loop of no iterations: nothing is assigned)
    if (!pc.any_body || pc.any_body->kind != Stmt::Set || pc.any_body->tn != op.tn || pc.coop != 0 || pc.ser_work != 1 || pc.uses_merge || pc.sum ||
        !pc.whole.empty() || !pc.staged.empty() || pc.written.size() != 1 || !covers_node(*pc.any_body, pc.par))
      return -1;
    bool plain = true;
    std::set<int> reads;
    auto position = [&](const Index& ix) {   // the gathering kernel has no static indices
      for (auto& sy : code.prog.statics)
        if (ix.uses(sy.sym)) plain = false;
    };
    walk_scalar(*pc.any_body->value, [&](const Scalar& e) {
      if (e.kind == Scalar::LocalScope || e.kind == Scalar::GetLocal || e.kind == Scalar::GetMerge) plain = false;
      if (e.kind == Scalar::EmbedIdx) position(e.idx);
      if (e.kind == Scalar::Get || e.kind == Scalar::GetDyn) {
        if (e.tn == op.tn) plain = false;
        reads.insert(e.tn);
        for (auto& ix : e.idcs) position(ix);
      }
    }, [](const Stmt&) {});
    for (size_t i = (size_t)j + 1; i < code.stages.size(); ++i) {
      const Stage& st = code.stages[i];
      for (int n : st.writes) plain = plain && !reads.count(n);
      if (st.kind == Stage::Memset) plain = plain && !reads.count(st.memset_tn);
    }
    return plain ? j : -1;
  }
  std::string pack_body(const PackOp& op, const std::string& dst, int64_t first, const Emitter::Res* made = nullptr, size_t maker = 0) {
    const std::string src_name = code.prog.tn(op.tn).ident;
    // A thread takes 16 bytes of a packed row; where it also makes the values, 4: a chain of one or two evaluations.  (Of
    // eight, 1919 rows of a 90-240-27 character model in bf16 took 15.7 us instead of 14.1.)
    const int eb = prec_bytes(op.prec), V = (made ? 4 : 16) / eb;
    // groups per row of one part
    const int64_t groups = op.ld / V / (op.split && op.kmajor ? 2 : 1);
    std::ostringstream o;
    // 32-bit arithmetic throughout where the packed copy has fewer than 2^31 groups and the node fewer elements
    const bool narrow = first + op.rows() * (op.ld / V) < (1ll << 31) && code.prog.tn(op.tn).num_elems() < (1ll << 31);
    const std::string IT = narrow ? "unsigned int" : "unsigned long long", S = narrow ? "u" : "ull";
    auto num = [&](int64_t v) { return std::to_string(v) + S; };
    o << "      const " << IT << " b200_i = (" << IT << ")(b200_g - " << first << "ull);\n"
      << "      const " << IT << " b200_grp = b200_i % " << num(groups) << ", b200_row = b200_i / " << num(groups) << ";\n";
    // `at`: adds the position `var` along the axes to the variable `acc`
    int tmp = 0;
    auto at = [&](const std::vector<PackOp::Axis>& axes, std::string var, const std::string& acc, const std::string& pad) {
      std::string t;
      for (size_t a = axes.size(); a-- > 0;) {
        if (a == 0) {
          t += pad + acc + " += (" + var + ") * " + num(axes[a].stride) + ";\n";
        } else {
          const std::string q = "b200_q" + std::to_string(tmp++);
          t += pad + acc + " += ((" + var + ") % " + num(axes[a].extent) + ") * " + num(axes[a].stride) + ";\n" + pad + "const " + IT + " " + q + " = (" + var +
               ") / " + num(axes[a].extent) + ";\n";
          var = q;
        }
      }
      return t;
    };
    auto extent = [](const std::vector<PackOp::Axis>& axes) {
      int64_t e = 1;
      for (auto& a : axes) e *= a.extent;
      return e;
    };
    const int64_t K = extent(op.k), MN = extent(op.mn);
    const std::vector<PackOp::Axis>& inner = op.kmajor ? op.k : op.mn;
    const int64_t outer_rows = op.kmajor ? MN : op.seg;
    o << "      " << IT << " b200_base = " << num(op.off) << ";\n";
    if (!op.batch.empty()) o << "      const " << IT << " b200_bt = b200_row / " << num(outer_rows) << ", b200_rr = b200_row % " << num(outer_rows) << ";\n" << at(op.batch, "b200_bt", "b200_base", "      ");
    else o << "      const " << IT << " b200_rr = b200_row;\n";
    const int64_t inner_real = op.kmajor ? K : MN;
    std::string seg_of, in0;
    o << "      const " << IT << " b200_j0 = b200_grp * " << V << S << ";\n";
    if (op.kmajor) {
      o << at(op.mn, "b200_rr", "b200_base", "      ");
      o << "      const bool b200_row_ok = true;\n";
    } else {
      o << "      const " << IT << " b200_kk = b200_rr;\n";
      o << "      const bool b200_row_ok = b200_kk < " << num(K) << ";\n" << at(op.k, "b200_kk", "b200_base", "      ");
    }
    const std::string T = Emitter::ctype(op.prec);
    // the group's elements: the first position is taken apart with divisions, the others by counting on
    o << "      " << T << " b200_v[" << V << "];\n      " << IT << " b200_p = b200_base;\n";
    std::string rest = "b200_j0";
    for (size_t a = inner.size(); a-- > 0;) {
      const std::string c = "b200_c" + std::to_string(a);
      if (a == 0) {
        o << "      b200_p += (" << rest << ") * " << num(inner[a].stride) << ";\n";
      } else {
        o << "      " << IT << " " << c << " = (" << rest << ") % " << num(inner[a].extent) << ";\n      b200_p += " << c << " * " << num(inner[a].stride) << ";\n"
          << "      const " << IT << " b200_r" << a << " = (" << rest << ") / " << num(inner[a].extent) << ";\n";
        rest = "b200_r" + std::to_string(a);
      }
    }
    // A whole group of neighbours that lies on a 16-byte boundary is one load, where the strides put either every group on
    // such a boundary or none: the node itself may lie anywhere, but lanes that disagree would wait for both ways (rows
    // of 30 floats: 0.3 us longer).
    bool neighbours = !made && inner.size() == 1 && inner[0].stride == 1 && op.off % V == 0;
    for (auto* axes : {&op.batch, op.kmajor ? &op.mn : &op.k})
      for (auto& a : *axes) neighbours = neighbours && a.stride % V == 0;
    if (neighbours) {
      o << "      if (b200_row_ok && b200_j0 + " << V << S << " <= " << num(inner_real) << " && ((unsigned long long)(" << src_name << " + b200_p) & 15ull) == 0ull) {\n"
        << "        const uint4 b200_q = *(const uint4*)(" << src_name << " + b200_p);\n";
      for (int w = 0; w < 4; ++w) {
        const std::string word = std::string("b200_q.") + "xyzw"[w];
        if (eb == 4) o << "        b200_v[" << w << "] = __uint_as_float(" << word << ");\n";
        else o << "        b200_v[" << 2 * w << "] = (" << T << ")" << word << "; b200_v[" << 2 * w + 1 << "] = (" << T << ")(" << word << " >> 16);\n";
      }
      o << "      } else\n";
    }
    std::string value = src_name + "[b200_p]";
    o << "#pragma unroll\n      for (unsigned int b200_e = 0; b200_e < " << V << "u; ++b200_e) {\n";
    if (made) {
      // the place in the node gives the maker's loops
      const Tnode& t = code.prog.tn(op.tn);
      const Stmt& set = *pieces[maker].any_body;
      o << "        " << T << " b200_m = (" << T << ")0;\n        if (b200_row_ok && b200_j0 + b200_e < " << num(inner_real) << ") {\n          " << IT << " b200_w = b200_p;\n";
      for (auto& d : code.stages[maker].ser)   // (loops of one iteration that the node does not carry)
        o << "          const unsigned int " << d.sym << " = " << d.from << "u;\n";
      for (size_t a = t.dims.size(); a-- > 0;) {
        if (set.idcs[a].kind == Index::Iter) o << "          const unsigned int " << set.idcs[a].sym << " = (unsigned int)(" << (a ? "b200_w % " + num(t.dims[a]) : std::string("b200_w")) << ");\n";
        if (a) o << "          b200_w /= " << num(t.dims[a]) << ";\n";
      }
      o << "          b200_m = " << Emitter::store_wrap(t.prec, made->expr) << ";\n          " << src_name << "[b200_p] = b200_m;\n        }\n";
      value = "b200_m";
    }
    o << "        b200_v[b200_e] = b200_row_ok && b200_j0 + b200_e < " << num(inner_real) << " ? " << value << " : (" << T << ")0;\n        b200_p += " << num(inner.back().stride) << ";\n";
    for (size_t a = inner.size(); a-- > 1;) {
      const std::string c = "b200_c" + std::to_string(a);
      // carry: this axis starts over, the one outside moves on (strides are unsigned and wrap around)
      o << "        if (++" << c << " == " << num(inner[a].extent) << ") {\n        " << c << " = 0;\n        b200_p += " << num(inner[a - 1].stride) << " - "
        << num(inner[a].extent * inner[a].stride) << ";\n";
    }
    for (size_t a = 1; a < inner.size(); ++a) o << "        }\n";
    o << "      }\n";
    if (op.split) {
      // where the group goes among the rows of both parts, and how far behind it its other part lies
      const int64_t apart = op.kmajor ? groups : op.seg * groups;
      const std::string row_at = op.kmajor ? "b200_row * " + num(2 * groups)
                                 : op.batch.empty() ? "b200_rr * " + num(groups) : "(b200_bt * " + num(2 * op.seg) + " + b200_rr) * " + num(groups);
      o << "      const " << IT << " b200_to = " << row_at << " + b200_grp;\n";
      if (made)
        o << "      ((float*)" << dst << ")[b200_to] = b200_tf32_extreme(b200_v[0], false);\n      ((float*)" << dst << ")[b200_to + " << num(apart)
          << "] = b200_tf32_extreme(b200_v[0], true);\n";
      else
        o << "      " << dst << "[b200_to] = b200_tf32_parts(b200_v, false);\n      " << dst << "[b200_to + " << num(apart) << "] = b200_tf32_parts(b200_v, true);\n";
    } else if (made) {
      o << "      ((b200_u32*)" << dst << ")[b200_i] = " << (eb == 4 ? "__float_as_uint(b200_v[0])" : "(b200_u32)b200_v[0] | ((b200_u32)b200_v[1] << 16)") << ";\n";
    } else if (eb == 4) {
      o << "      " << dst << "[b200_i] = make_uint4(__float_as_uint(b200_v[0]), __float_as_uint(b200_v[1]), __float_as_uint(b200_v[2]), __float_as_uint(b200_v[3]));\n";
    } else {
      o << "      " << dst << "[b200_i] = make_uint4((b200_u32)b200_v[0] | ((b200_u32)b200_v[1] << 16), (b200_u32)b200_v[2] | ((b200_u32)b200_v[3] << 16), "
        << "(b200_u32)b200_v[4] | ((b200_u32)b200_v[5] << 16), (b200_u32)b200_v[6] | ((b200_u32)b200_v[7] << 16));\n";
    }
    return o.str();
  }
  // Places the slots in the routine's scratch: a slot lives from the stage that fills it to the last
  // contraction that reads it, and takes the lowest place no slot alive at the same time occupies (what
  // was just read is then overwritten while it is still in L2).
  void place_packs() {
    const size_t n = code.pack_bytes.size();
    std::vector<size_t> from(n, 0), to(n, 0);
    for (size_t i = 0; i < code.stages.size(); ++i) {
      for (int s : code.stages[i].pack_writes) from[(size_t)s] = to[(size_t)s] = i;
      for (int s : {code.stages[i].gemm.a_slot, code.stages[i].gemm.b_slot})
        if (s >= 0) to[(size_t)s] = i;
    }
    code.pack_offsets.assign(n, 0);
    for (size_t s = 0; s < n; ++s) {
      const size_t bytes = (code.pack_bytes[s] + 255) & ~(size_t)255;
      std::vector<std::pair<size_t, size_t>> taken;
      for (size_t q = 0; q < s; ++q)
        if (from[q] <= to[s] && from[s] <= to[q]) taken.push_back({code.pack_offsets[q], code.pack_offsets[q] + ((code.pack_bytes[q] + 255) & ~(size_t)255)});
      std::sort(taken.begin(), taken.end());
      size_t off = 0;
      for (auto& t : taken) {
        if (off + bytes <= t.first) break;
        off = std::max(off, t.second);
      }
      code.pack_offsets[s] = off;
      code.pack_scratch_bytes = std::max(code.pack_scratch_bytes, off + bytes);
    }
  }

  // A scatter accumulation that is a contraction per written window: the input gradient of a convolution,
  //   for b, oh, ow, co, kh, kw, ci:  gx[b, s oh + kh, s ow + kw, ci] += w[co, kh, kw, ci] * dz[b, oh, ow, co].
  // The products summed over the loops that do not move the position (co) form a dense contraction
  // [b oh ow] x [kh kw ci] on the tensor cores, into scratch; a second kernel gives every element of the
  // node a thread that gathers the windows covering it.  One atomic add per product sum became one read
  // (48 x 48 x 5 images, 5 x 5 kernels, 37 of them: 171 us of atomic adds).
  bool scatter_contraction(const std::vector<LoopDim>& nest, const StmtP& body, bool was_zero) {
    const Stmt& set = *body;
    if (set.kind != Stmt::Set || set.vec_len > 0 || !accumulates_into_self(set) || !opt.enable_coop) return false;
    const Scalar& v = *set.value;
    if (v.kind != Scalar::Tern || v.op != "fma") return false;
    if (code.prog.tn(set.tn).prec != Prec::Single) return false;
    const Scalar &x = *v.args[0].s, &y = *v.args[1].s;
    if (x.kind != Scalar::Get || y.kind != Scalar::Get) return false;
    std::map<std::string, int64_t> extent;
    for (auto& d : nest) {
      if (d.from != 0 || d.extent() <= 0) return false;
      extent[d.sym] = d.extent();
    }
    // written position: loops by themselves, or c1 * i + c2 * j (+ fixed) with both coefficients positive
    bool any_affine = false;
    std::map<std::string, int> seen;
    for (auto& ix : set.idcs) {
      if (ix.kind == Index::Fixed) continue;
      if (ix.kind == Index::Iter) { if (++seen[ix.sym] > 1 || !extent.count(ix.sym)) return false; continue; }
      if (ix.kind != Index::Affine || ix.terms.empty() || ix.terms.size() > 2) return false;
      for (auto& t : ix.terms)
        if (t.first <= 0 || !extent.count(t.second) || ++seen[t.second] > 1) return false;
      any_affine = any_affine || ix.terms.size() == 2;
    }
    if (!any_affine) return false;
    auto uses = [](const Indices& idcs, const std::string& sy) {
      for (auto& ix : idcs)
        if (ix.uses(sy)) return true;
      return false;
    };
    // loops of the scratch node: those of one factor, then those of the other (which holds the last axis)
    std::vector<LoopDim> first, second, red;
    const Index& last = set.idcs.back();
    const std::string last_sym = last.kind == Index::Iter ? last.sym : (last.kind == Index::Affine ? last.terms.back().second : std::string());
    const bool last_in_x = uses(x.idcs, last_sym);
    int64_t elems = 1;
    for (auto& d : nest) {
      const bool ix = uses(x.idcs, d.sym), iy = uses(y.idcs, d.sym);
      if (!seen.count(d.sym)) {
        if (!ix || !iy) return false;
        red.push_back(d);
        continue;
      }
      if (ix == iy) return false;
      (ix == last_in_x ? second : first).push_back(d);
      elems *= d.extent();
    }
    if (first.empty() || second.empty() || red.empty() || elems * 4 > (std::min<int64_t>(opt.gather_mb, 1024) << 20) || elems >= (1ll << 31)) return false;
    // a few hundred multiplications per gathered row do not pay for the gathering (see the convolutions' windows in
    // match_gemm): 8 outputs of 3 x 3 on one channel, 262144 positions: 9 us as scattered additions, 49 us as this
    {
      int64_t e[3] = {1, 1, 1};
      for (auto& d : first) e[0] *= d.extent();
      for (auto& d : second) e[1] *= d.extent();
      for (auto& d : red) e[2] *= d.extent();
      if (e[0] * e[1] * e[2] / std::max({e[0], e[1], e[2]}) < 256) return false;
    }
    const std::string t_ident = code.prog.tn(set.tn).ident;
    const std::vector<int64_t> t_dims = code.prog.tn(set.tn).dims;
    const int64_t t_elems = code.prog.tn(set.tn).num_elems();
    if (t_elems >= (1ll << 31)) return false;
    // the contraction as a statement of its own:  P[first.., second..] := sum over red of x * y
    int next_id = 0;
    for (auto& t : code.prog.tnodes) next_id = std::max(next_id, t.id + 1);
    Tnode acc, P;
    acc.id = next_id;
    acc.ident = "b200_acc" + std::to_string(acc.id);
    acc.dims = {1};
    acc.mode = Mode::Virtual;
    P.id = next_id + 1;
    P.ident = "b200_windows" + std::to_string(P.id);
    P.mode = Mode::Local;
    std::vector<LoopDim> free_loops = first;
    free_loops.insert(free_loops.end(), second.begin(), second.end());
    Indices at;
    for (auto& d : free_loops) {
      P.dims.push_back(d.extent());
      Index ix;
      ix.kind = Index::Iter;
      ix.sym = d.sym;
      at.push_back(ix);
    }
    auto stmt = [](Stmt::Kind k) { auto p = std::make_shared<Stmt>(); p->kind = k; return p; };
    auto scal = [](Scalar::Kind k) { auto p = std::make_shared<Scalar>(); p->kind = k; return p; };
    const int sid = -1000 - acc.id;
    auto zero = scal(Scalar::Const);
    auto init = stmt(Stmt::SetLocal);
    init->scope_id = sid; init->tn = acc.id; init->value = zero;
    auto get = scal(Scalar::GetLocal);
    get->scope_id = sid; get->tn = acc.id;
    auto mac = scal(Scalar::Tern);
    mac->op = "fma";
    mac->args = {v.args[0], v.args[1], {get, Prec::Single}};
    StmtP loop = stmt(Stmt::SetLocal);
    loop->scope_id = sid; loop->tn = acc.id; loop->value = mac;
    for (size_t i = red.size(); i-- > 0;) {
      auto f = stmt(Stmt::For);
      f->index = red[i].sym; f->from = 0; f->to = red[i].to; f->body = loop;
      loop = f;
    }
    auto seq = stmt(Stmt::Seq);
    seq->items = {init, loop};
    auto scope = scal(Scalar::LocalScope);
    scope->scope_id = sid; scope->tn = acc.id; scope->body = seq; scope->idcs = at;
    auto product = stmt(Stmt::Set);
    product->tn = P.id; product->idcs = at; product->value = scope;
    const size_t had = code.prog.tnodes.size();
    for (auto* t : {&acc, &P}) {
      code.prog.tn_index[t->id] = code.prog.tnodes.size();
      code.prog.tnodes.push_back(*t);
    }
    Stage g;
    int n_fused = 0;
    CompileOptions exact = opt;
    exact.exact_single = true;    // single-precision products were exact here, and stay so
    if (!match_gemm(code.prog, free_loops, *product, false, exact, {}, &n_fused, &g)) {
      code.prog.tn_index.erase(acc.id);
      code.prog.tn_index.erase(P.id);
      code.prog.tnodes.resize(had);
      return false;
    }
    kept_stmts.push_back(product);
    pack_stage(g);
    g.copies = true;
    g.kernel = kernel_name();
    g.gemm_source = gemm_translation_unit(code.prog, g, g.kernel, opt);
    code.stages.push_back(g);
    // the gathering kernel: one thread per element of the node
    Stage st;
    st.kind = Stage::Generic;
    st.kernel = kernel_name();
    st.block = 256;
    st.total = t_elems;
    st.args = {{KArg::Node, set.tn}, {KArg::Node, P.id}};
    st.writes = {set.tn};
    std::ostringstream b;
    std::string rem = "b200_g";
    std::vector<std::string> pos(t_dims.size());
    for (size_t a = t_dims.size(); a-- > 0;) {
      pos[a] = "b200_p" + std::to_string(a);
      b << "    const unsigned int " << pos[a] << " = " << (a == 0 ? rem : rem + " % " + std::to_string(t_dims[a]) + "u") << ";\n";
      if (a) {
        b << "    const unsigned int b200_r" << a << " = " << rem << " / " << t_dims[a] << "u;\n";
        rem = "b200_r" + std::to_string(a);
      }
    }
    b << "    float b200_sum = 0.0f;\n";
    std::string pad = "    ", close;
    for (size_t a = 0; a < set.idcs.size(); ++a) {
      const Index& ix = set.idcs[a];
      if (ix.kind == Index::Fixed) {
        b << pad << "if (" << pos[a] << " == " << ix.fixed << "u) {\n";
      } else if (ix.kind == Index::Iter) {
        b << pad << "const unsigned int " << ix.sym << " = " << pos[a] << ";\n" << pad << "if (" << ix.sym << " < " << extent[ix.sym] << "u) {\n";
      } else {
        // the inner loop (the kernel position) runs, the outer one follows from what is left
        const auto& o = ix.terms.size() == 2 ? (extent[ix.terms[0].second] >= extent[ix.terms[1].second] ? ix.terms[0] : ix.terms[1]) : ix.terms[0];
        if (ix.terms.size() == 2) {
          const auto& k = &o == &ix.terms[0] ? ix.terms[1] : ix.terms[0];
          b << "#pragma unroll\n" << pad << "for (unsigned int " << k.second << " = 0; " << k.second << " < " << extent[k.second] << "u; ++" << k.second << ") {\n";
          pad += "  ";
          close = pad.substr(2) + "}\n" + close;
          b << pad << "const unsigned int b200_d" << a << " = " << pos[a] << " - " << ix.fixed << "u - " << k.second << " * " << k.first << "u;\n";
        } else {
          b << pad << "const unsigned int b200_d" << a << " = " << pos[a] << " - " << ix.fixed << "u;\n";
        }
        // (a difference below zero wraps around and fails the comparison)
        b << pad << "const unsigned int " << o.second << " = b200_d" << a << (o.first > 1 ? " / " + std::to_string(o.first) + "u" : std::string()) << ";\n"
          << pad << "if (" << o.second << " < " << extent[o.second] << "u" << (o.first > 1 ? " && b200_d" + std::to_string(a) + " % " + std::to_string(o.first) + "u == 0u" : std::string()) << ") {\n";
      }
      close = pad + "}\n" + close;
      pad += "  ";
    }
    Emitter em(code.prog);
    b << pad << "b200_sum += " << P.ident << "[" << em.offset(at, P.dims) << "];\n" << close
      << "    " << t_ident << "[b200_g] = " << (was_zero ? "b200_sum" : t_ident + "[b200_g] + b200_sum") << ";\n";
    src << "extern \"C\" __global__ void __launch_bounds__(256) " << st.kernel << "(float* " << t_ident << ", const float* __restrict__ " << P.ident << ") {\n" << kGridEntry
        << "  for (unsigned int b200_g = blockIdx.x * 256u + threadIdx.x; b200_g < " << t_elems << "u; b200_g += gridDim.x * 256u) {\n"
        << b.str() << "  }\n}\n\n";
    st.note = "gathers the windows that cover an element (accumulation with moving positions)";
    code.stages.push_back(st);
    return true;
  }
  std::vector<StmtP> kept_stmts;   // statements made here whose indices stages may refer to

  // an epilogue that ends in a grid-wide sum keeps its per-warp partials and its ticket in the
  // routine's reduction scratch (zeroed at link; the kernel resets its ticket itself)
  void assign_epilogue_scratch(Stage& g) {
    if (!g.epi_scratch_bytes) return;
    for (auto& a : g.args)
      if (a.kind == KArg::Scratch) a.tn = (int)code.reduce_scratch_bytes;
    code.reduce_scratch_bytes += g.epi_scratch_bytes;
    code.reduce_scratch_bytes = (code.reduce_scratch_bytes + 255) & ~(size_t)255;
  }

  // A routine of one kernel takes its static indices as a kernel argument instead of through the device
  // table: such a routine is never captured in a graph (`direct` in b200_routine::link follows from the argument),
  // and the table would cost a copy ahead of the kernel every time an index moves -- the next minibatch of a
  // training step.
  void statics_by_value() {
    if (code.stages.size() != 1 || code.stages[0].kind != Stage::Generic || opt.bounds) return;
    for (auto& a : code.stages[0].args)
      if (a.kind == KArg::Statics) a.kind = KArg::StaticValues;
      else continue;
    const std::string was = "const unsigned int* __restrict__ b200_statics";
    const size_t at = code.source.find(was);
    if (at == std::string::npos) return;
    code.source.replace(at, was.size(), "const b200_static_values b200_statics");
    const size_t k = code.source.rfind("extern \"C\" __global__", at);
    code.source.insert(k, "struct b200_static_values {\n  unsigned int v[" + std::to_string(code.prog.statics.size()) +
                              "];\n  __device__ __forceinline__ unsigned int operator[](int i) const { return v[i]; }\n};\n");
  }

  // Range-checked build.  Every generic kernel's node pointers are renamed and shadowed by a
  // b200_checked proxy of the node's size (kernels/numerics.cuh), so that each `node[offset]` the
  // emitters wrote is compared with the number of elements the node has; the kernels get the device
  // status word as a last parameter.
  void apply_bounds() {
    std::string text = code.source;
    for (auto& st : code.stages) {
      if (st.kind != Stage::Generic || st.kernel.empty()) continue;
      const std::string head = " " + st.kernel + "(";
      size_t h = text.find(head);
      if (h == std::string::npos) continue;
      const size_t p0 = h + head.size();
      const size_t p1 = text.find(") {\n", p0);
      if (p1 == std::string::npos) continue;
      std::string params = text.substr(p0, p1 - p0), proxies;
      for (auto& t : code.prog.tnodes) {
        if (t.mode == Mode::Virtual) continue;
        // "<type>* [__restrict__ ]ident" followed by ',' or the end
        for (const std::string& sep : {std::string("* __restrict__ "), std::string("* ")}) {
          const std::string needle = sep + t.ident;
          size_t q = 0;
          while ((q = params.find(needle, q)) != std::string::npos) {
            const size_t end = q + needle.size();
            if (end != params.size() && params[end] != ',') { q = end; continue; }
            size_t b = params.rfind(',', q);
            b = b == std::string::npos ? 0 : b + 1;
            while (b < q && params[b] == ' ') ++b;
            const std::string type = params.substr(b, q - b);
            params.insert(end, "__p");
            proxies += "  const b200_checked<" + type + "> " + t.ident + " = {" + t.ident + "__p, " + std::to_string(t.num_elems()) +
                       "ull, b200_status, " + std::to_string(t.id) + "u};\n";
            q = end + 3;
          }
        }
      }
      params += (params.empty() ? "" : ", ") + std::string("unsigned int* b200_status");
      text.replace(p0, p1 - p0, params);
      const size_t body = text.find(") {\n", p0) + 4;
      text.insert(body, proxies);
      st.args.push_back({KArg::Status, -1});
    }
    code.source = text;
  }

  void memset_stage(int tn) {
    Stage st;
    st.kind = Stage::Memset;
    st.memset_tn = tn;
    st.note = "zero_out";
    st.writes = {tn};
    code.stages.push_back(st);
  }

  void top_level(const StmtP& s, std::vector<StmtP>& flat) {
    if (s->kind == Stmt::Seq)
      for (auto& x : s->items) top_level(x, flat);
    else if (s->kind != Stmt::Noop && s->kind != Stmt::Comment)
      flat.push_back(s);
  }

  // the perfect-nest pointwise assignments that directly follow position `from`
  std::vector<Follower> followers_after(const std::vector<StmtP>& flat, size_t from) {
    std::vector<Follower> out;
    for (size_t k = from; k < flat.size() && out.size() < 8; ++k) {
      Follower f;
      const Stmt* b = flat[k].get();
      while (b->kind == Stmt::For) {
        f.nest.push_back({b->index, b->from, b->to});
        b = b->body.get();
      }
      if (b->kind != Stmt::Set) break;
      f.set = b;
      out.push_back(f);
    }
    return out;
  }

  // Function-scope scalar locals.  `hoist_cross_statement_cse` (arrayjit/lib/low_level.ml:2039-2135)
  // turns a Local_scope shared by sibling assignments into `Declare_local id; <the scope's body>`
  // before the first user, the users reading `Get_local id`; the cc backend prints a function-scope
  // variable (arrayjit/lib/c_syntax.ml:695-704,730-734).  Siblings inside one loop body stay inside
  // one kernel and need nothing.  At the top level of the routine the users become different
  // kernels, so the local becomes a one-element routine-local node: declaration and body turn back
  // into `t[0] := scope { body }` (which the reduction paths recognise) and every later
  // `Get_local id` into `t[0]`.  The value makes one round trip through memory in its own precision.
  void unhoist_function_locals(std::vector<StmtP>& flat) {
    std::map<int, int> hoisted;   // scope id -> synthetic node id
    auto writes_scope = [](const Stmt& s, int sid) {
      bool w = false;
      walk_stmt(s, [](const Scalar&) {}, [&](const Stmt& x) { if (x.kind == Stmt::SetLocal && x.scope_id == sid) w = true; });
      return w;
    };
    int next_id = 0;
    for (auto& t : code.prog.tnodes) next_id = std::max(next_id, t.id + 1);
    std::vector<StmtP> out;
    for (size_t i = 0; i < flat.size(); ++i) {
      const StmtP& s = flat[i];
      if (s->kind != Stmt::DeclareLocal) { out.push_back(s); continue; }
      const Tnode& st = code.prog.tn(s->tn);
      Tnode syn;
      syn.id = next_id++;
      syn.ident = "b200_local" + std::to_string(s->scope_id) + "_" + st.ident;
      syn.prec = st.prec;
      syn.dims = {1};
      syn.mode = Mode::Local;
      syn.zero_init = s->needs_init;
      auto body = std::make_shared<Stmt>();
      body->kind = Stmt::Seq;
      size_t j = i + 1;
      while (j < flat.size() && writes_scope(*flat[j], s->scope_id)) body->items.push_back(flat[j++]);
      hoisted[s->scope_id] = syn.id;
      code.prog.tn_index[syn.id] = code.prog.tnodes.size();
      code.prog.tnodes.push_back(syn);
      if (!body->items.empty()) {
        auto scope = std::make_shared<Scalar>();
        scope->kind = Scalar::LocalScope;
        scope->scope_id = s->scope_id;
        scope->tn = s->tn;
        scope->body = body;
        auto set = std::make_shared<Stmt>();
        set->kind = Stmt::Set;
        set->tn = syn.id;
        Index zero;
        set->idcs = {zero};
        set->value = scope;
        out.push_back(set);
      }
      i = j - 1;
    }
    if (hoisted.empty()) return;
    // every remaining mention of a hoisted scope reads the node
    std::function<ScalarP(const ScalarP&, int)> fix_scalar;
    std::function<StmtP(const StmtP&, int)> fix_stmt = [&](const StmtP& s, int inside) -> StmtP {
      auto c = std::make_shared<Stmt>(*s);
      for (auto& x : c->items) x = fix_stmt(x, inside);
      if (c->body) c->body = fix_stmt(c->body, inside);
      if (c->value) c->value = fix_scalar(c->value, inside);
      if (c->kind == Stmt::SetLocal && c->scope_id != inside && hoisted.count(c->scope_id))
        throw Error(-4, "a function-scope local is assigned after its defining statements");
      return c;
    };
    fix_scalar = [&](const ScalarP& e, int inside) -> ScalarP {
      if (e->kind == Scalar::GetLocal && e->scope_id != inside && hoisted.count(e->scope_id)) {
        auto g = std::make_shared<Scalar>();
        g->kind = Scalar::Get;
        g->tn = hoisted[e->scope_id];
        Index zero;
        g->idcs = {zero};
        return g;
      }
      auto c = std::make_shared<Scalar>(*e);
      // inside the re-wrapped body the scope's own id keeps meaning the local variable
      const int in = (c->kind == Scalar::LocalScope && hoisted.count(c->scope_id)) ? c->scope_id : inside;
      if (c->body) c->body = fix_stmt(c->body, in);
      for (auto& a : c->args) a.s = fix_scalar(a.s, in);
      return c;
    };
    for (auto& s : out) s = fix_stmt(s, -1);
    flat.swap(out);
  }

  void run() {
    std::vector<StmtP> flat;
    top_level(code.prog.body, flat);
    unhoist_function_locals(flat);
    src << kNumericsSource << "\n";
    std::set<int> zeroed;  // nodes zeroed by the previous stage (for beta = 0 contractions)
    std::map<int, size_t> zero_stage;  // ... and the index of the stage that zeroes them
    std::set<int> zero_read;           // zeroed nodes some later stage has read as zeros
    auto drop_zero_out = [&](int tn) {
      // the node is about to be overwritten completely by a stage that does not read it
      auto it = zero_stage.find(tn);
      if (it == zero_stage.end() || zero_read.count(tn)) return;
      code.stages[it->second].memset_tn = -1;   // filtered out in emit_kernels
      zero_stage.erase(it);
    };
    // plans the statement at flat[i]; advances i past the statements it absorbed
    auto plan_one = [&](size_t& i) {
      const StmtP& s = flat[i];
      if (s->kind == Stmt::DeclareLocal || s->kind == Stmt::SetLocal)
        throw Error(-4, "a function-scope scalar local is assigned away from its declaration");
      if (s->kind == Stmt::ZeroOut) {
        const Tnode& t = code.prog.tn(s->tn);
        if (t.mode == Mode::Virtual) return;
        // a zero_out that a following contraction absorbs (beta = 0) is dropped below
        bool absorbed = false;
        if (gemm_at(i + 1) && i + 1 < flat.size() && flat[i + 1]->kind == Stmt::For) {
          std::vector<LoopDim> nest;
          StmtP body = flat[i + 1];
          while (body->kind == Stmt::For) {
            nest.push_back({body->index, body->from, body->to});
            body = body->body;
          }
          Stage g;
          int n_fused = 0;
          if (body->kind == Stmt::Set && body->tn == s->tn &&
              match_gemm(code.prog, nest, *body, true, opt, followers_after(flat, i + 2), &n_fused, &g)) {
            if (g.gemm.split_k > 1) memset_stage(s->tn);   // partial tiles are added to the zeroed node
            pack_stage(g);
            assign_epilogue_scratch(g);
            g.kernel = kernel_name();
            g.gemm_source = gemm_translation_unit(code.prog, g, g.kernel, opt);
            code.stages.push_back(g);
            absorbed = true;
            i += 1 + (size_t)n_fused;
          }
        }
        if (!absorbed) {
          zero_stage[s->tn] = code.stages.size();
          zero_read.erase(s->tn);
          memset_stage(s->tn);
          zeroed.insert(s->tn);  // still all zero until some stage writes it
        }
        return;
      }
      // peel the perfect loop nest
      std::vector<LoopDim> nest;
      StmtP body = s;
      while (body->kind == Stmt::For) {
        nest.push_back({body->index, body->from, body->to});
        body = body->body;
      }
      if (!body_has_set(*body)) return;
      {
        std::set<std::pair<int, int>> declared, used;
        collect_scopes(*body, declared, used);
        for (auto& u : used)
          if (!declared.count(u))
            throw Error(-4, "a scalar local is read outside the statement that defines it");
      }
      // a node zeroed earlier and untouched since lets a contraction skip reading it (beta = 0)
      std::set<int> writes_now;
      walk_stmt(*body, [](const Scalar&) {}, [&](const Stmt& w) {
        if (w.kind == Stmt::Set || w.kind == Stmt::ZeroOut) writes_now.insert(w.tn);
      });
      const bool was_zero = body->kind == Stmt::Set && zeroed.count(body->tn) > 0;
      walk_stmt(*body, [&](const Scalar& e) {
        if ((e.kind == Scalar::Get || e.kind == Scalar::GetDyn) && zeroed.count(e.tn) && !(body->kind == Stmt::Set && e.tn == body->tn))
          zero_read.insert(e.tn);
      }, [](const Stmt&) {});
      for (int w : writes_now) zeroed.erase(w);
      if (opt.enable_attn && gemm_at(i) && body->kind == Stmt::Set && i + 6 <= flat.size()) {
        // scores, softmax and weights . values as one kernel
        bool allowed = true;
        for (size_t k = i; k < i + 6; ++k) allowed = allowed && gemm_at(k);
        Stage a;
        int n_abs = 0;
        if (allowed && match_attention(code.prog, flat, i, opt, &n_abs, &a)) {
          for (int w : a.writes) zeroed.erase(w);
          // masks as bits: one packing stage per mask node (shared when the node is read-only)
          {
            size_t k = 0;
            for (auto& arg : a.args)
              if (arg.kind == KArg::Scratch) arg.tn = (int)pack_bits_stage(a.attn.cond_tns.at(k++));
          }
          a.kernel = kernel_name();
          a.gemm_source = attn_translation_unit(code.prog, a, a.kernel);
          code.stages.push_back(a);
          i += (size_t)n_abs - 1;
          return;
        }
      }
      if (gemm_at(i) && table_stage(nest, body)) return;
      if (gemm_at(i) && body->kind == Stmt::Set) {
        Stage g;
        int n_fused = 0;
        const std::vector<Follower> fol = followers_after(flat, i + 1);
        if (match_gemm(code.prog, nest, *body, was_zero, opt, fol, &n_fused, &g)) {
          for (int f = 0; f < n_fused; ++f) zeroed.erase(fol[(size_t)f].set->tn);
          // beta = 0 over the whole node: the zero_out before it has no reader left
          if (was_zero && !g.gemm.accumulate && g.gemm.split_k == 1 && covers_node(*body, nest)) drop_zero_out(body->tn);
          pack_stage(g);
          assign_epilogue_scratch(g);
          g.kernel = kernel_name();
          g.gemm_source = gemm_translation_unit(code.prog, g, g.kernel, opt);
          code.stages.push_back(g);
          i += (size_t)n_fused;
          return;
        }
      }
      if (gemm_at(i) && scatter_contraction(nest, body, was_zero)) {
        if (was_zero) drop_zero_out(body->tn);   // every element of the node is stored
        return;
      }
      if (generic_stage(nest, body, was_zero)) drop_zero_out(body->tn);
    };
    for (size_t i = 0; i < flat.size(); ++i) {
      const size_t before = code.stages.size(), first = i;
      cur_origin = (int)i;
      plan_one(i);
      for (size_t k = before; k < code.stages.size(); ++k)
        for (size_t o = first; o <= i; ++o) code.stages[k].origins.push_back((int)o);
    }
    emit_kernels();
    place_packs();
    if (opt.enable_fuse) group_contractions(code, opt);
    code.source = src.str();
    statics_by_value();
    if (opt.bounds) apply_bounds();
    // routine-local nodes that some stage touches get scratch (a node whose every use was fused
    // away, such as the score matrix of a fused attention stage, needs none)
    std::set<int> touched;
    for (auto& st : code.stages) {
      if (st.kind == Stage::Memset) touched.insert(st.memset_tn);
      for (auto& a : st.args)
        if (a.kind == KArg::Node) touched.insert(a.tn);
      if (st.kind == Stage::Gemm) { touched.insert(st.gemm.a_tn); touched.insert(st.gemm.b_tn); touched.insert(st.gemm.d_tn); }
      if (st.kind == Stage::Attn) { touched.insert(st.attn.q_tn); touched.insert(st.attn.k_tn); touched.insert(st.attn.v_tn); }
    }
    for (auto& t : code.prog.tnodes)
      if (t.mode == Mode::Local && touched.count(t.id)) code.local_nodes.push_back(t.id);
  }
};

}  // namespace

// Kernel pointers carry the nodes' own names, and generated code keeps to names that begin with b200_.  The
// hand-written kernels around a generated epilogue, and the functions of the attention stages, use shorter ones: a node
// called like one of them (a bias `acc`, a row sum `sum`) gets its number as a suffix.
static void avoid_kernel_names(Program& prog) {
  static const std::set<std::string> taken = [] {
    std::set<std::string> words;
    for (const char* text : {kTcSource, kGemmSource, kAttnSource, kAttnRowsSource}) {
      std::string word;
      for (const char* c = text; ; ++c) {
        if (*c && (isalnum((unsigned char)*c) || *c == '_')) { word += *c; continue; }
        if (!word.empty()) words.insert(word);
        word.clear();
        if (!*c) break;
      }
    }
    return words;
  }();
  for (auto& t : prog.tnodes)
    if (taken.count(t.ident)) t.ident += "_n" + std::to_string(t.id);
}

Code compile_program(Program prog, const CompileOptions& opt) {
  Code code;
  code.prog = std::move(prog);
  if (opt.enable_gemm || opt.enable_attn) avoid_kernel_names(code.prog);
  code.prog.deciding = find_deciding(code.prog);
  Builder b{code, opt};
  b.run();
  return code;
}

}  // namespace b200
