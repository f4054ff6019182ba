// planner.cpp — gate validation, lowering to device ops, and pass planning.
//
// Validation follows NaiveSvBackend::apply_gate (crates/aleph-sv/src/backend.rs:74-152)
// in the same order, with the same error variants: arity, then range and
// duplicates over qubits followed by controls, UnitaryKq validation
// (crates/aleph-sv/src/validation.rs:113-155), matrix materialisation
// (Gate::matrix, crates/aleph-core/src/gate/kinds.rs:213-400) and the
// unitarity check (validation.rs:25-51, AMPLITUDE_TOL = 1e-10).
//
// Planning: the gate list is cut into HBM passes. First it is rewritten: gate
// sequences on a few qubits that multiply out to a diagonal become corner phases
// (diagonal_cores), phases on the same qubits join and cancel (cancel_phases), and the
// gates on a pair of qubits become one 4x4 (fuse_pairs). Then passes take gates:
// * wide-tile passes (the default from n = 12): qubits 0..3 and eight more, in phases
//   of five register qubits;
// * warp-tile passes (short lists that they run faster, changed tuning keys, smaller
//   states): qubits 0..4 plus R register qubits;
// * tensor-core blocks (TC32): six qubits, one dense 64x64 matrix.
// Each walks the pending gates in order and takes every gate that (a) commutes past
// all gates it defers and (b) acts non-diagonally only on its qubits; diagonal
// gates (CZ, phases, DiagonalPhase) and controls may sit on any qubit. This is the
// greedy open-block idea of FuseKq (crates/aleph-ir/src/passes/fuse_kq.rs:144-400)
// applied to tiles instead of matrices. A state of at most 12 qubits is one
// shared-memory pass.

#include <algorithm>
#include <deque>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <thread>
#include <unordered_map>

#include "engine.h"

namespace ab {

namespace {

struct Cx {
  double re, im;
};
inline Cx mul(Cx a, Cx b) { return {a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re}; }
inline Cx add(Cx a, Cx b) { return {a.re + b.re, a.im + b.im}; }
inline Cx sub(Cx a, Cx b) { return {a.re - b.re, a.im - b.im}; }
inline Cx conj(Cx a) { return {a.re, -a.im}; }
inline Cx neg(Cx a) { return {-a.re, -a.im}; }

constexpr double kTol = 1e-10;  // AMPLITUDE_TOL, crates/aleph-core/src/lib.rs:53

void set_kind(aleph_b200_error_info* e, const char* k) { std::snprintf(e->kind, sizeof(e->kind), "%s", k); }
int fail(aleph_b200_error_info* e, int s) {
  e->status = s;
  return s;
}

int arity(const aleph_b200_instr& g) {
  switch (g.kind) {
    case ALEPH_GATE_CNOT: case ALEPH_GATE_CZ: case ALEPH_GATE_SWAP: case ALEPH_GATE_ISWAP:
    case ALEPH_GATE_ISWAPDG: case ALEPH_GATE_CRX: case ALEPH_GATE_CRY: case ALEPH_GATE_CRZ:
    case ALEPH_GATE_UNITARY2Q: case ALEPH_GATE_UNITARY2QDIAG:
      return 2;
    case ALEPH_GATE_TOFFOLI: case ALEPH_GATE_CCZ:
      return 3;
    case ALEPH_GATE_UNITARYKQ:
      return (int)g.aux;
    default:
      return g.kind < 28 ? 1 : -1;
  }
}

// Gate::matrix (kinds.rs:213-400). Returns dim or 0 (error set).
int matrix_of(const aleph_b200_instr& g, const double* pool, uint64_t pool_len, Cx m[8][8],
              aleph_b200_error_info* e) {
  const Cx z{0, 0}, o{1, 0};
  for (int i = 0; i < 8; ++i)
    for (int j = 0; j < 8; ++j) m[i][j] = z;
  for (int i = 0; i < 3; ++i) {
    const bool used = (g.kind >= ALEPH_GATE_RX && g.kind <= ALEPH_GATE_PHASE && i == 0) ||
                      (g.kind == ALEPH_GATE_U3) ||
                      ((g.kind == ALEPH_GATE_CRX || g.kind == ALEPH_GATE_CRY || g.kind == ALEPH_GATE_CRZ) && i == 0);
    if (used && !std::isfinite(g.params[i])) {
      set_kind(e, gate_name(g.kind));
      return fail(e, ALEPH_B200_NON_FINITE_PARAM), 0;
    }
  }
  const double s2 = 0.70710678118654752440, pi4 = 0.78539816339744830962;
  auto from_pool = [&](uint64_t len) -> const double* {
    if (!pool || g.data_len != len || g.data_offset + len > pool_len) {
      set_kind(e, "matrix pool");
      fail(e, ALEPH_B200_INVALID_ARGUMENT);
      return nullptr;
    }
    return pool + 2 * g.data_offset;
  };
  const double t = g.params[0];
  switch (g.kind) {
    case ALEPH_GATE_H: m[0][0] = m[0][1] = m[1][0] = Cx{s2, 0}; m[1][1] = Cx{-s2, 0}; return 2;
    case ALEPH_GATE_X: m[0][1] = m[1][0] = o; return 2;
    case ALEPH_GATE_Y: m[0][1] = Cx{0, -1}; m[1][0] = Cx{0, 1}; return 2;
    case ALEPH_GATE_Z: m[0][0] = o; m[1][1] = neg(o); return 2;
    case ALEPH_GATE_S: m[0][0] = o; m[1][1] = Cx{0, 1}; return 2;
    case ALEPH_GATE_SDG: m[0][0] = o; m[1][1] = Cx{0, -1}; return 2;
    case ALEPH_GATE_T: m[0][0] = o; m[1][1] = Cx{std::cos(pi4), std::sin(pi4)}; return 2;
    case ALEPH_GATE_TDG: m[0][0] = o; m[1][1] = Cx{std::cos(pi4), -std::sin(pi4)}; return 2;
    case ALEPH_GATE_RX:
      m[0][0] = m[1][1] = Cx{std::cos(t / 2), 0};
      m[0][1] = m[1][0] = Cx{0, -std::sin(t / 2)};
      return 2;
    case ALEPH_GATE_RY:
      m[0][0] = m[1][1] = Cx{std::cos(t / 2), 0};
      m[0][1] = Cx{-std::sin(t / 2), 0};
      m[1][0] = Cx{std::sin(t / 2), 0};
      return 2;
    case ALEPH_GATE_RZ:
      m[0][0] = Cx{std::cos(t / 2), -std::sin(t / 2)};
      m[1][1] = Cx{std::cos(t / 2), std::sin(t / 2)};
      return 2;
    case ALEPH_GATE_PHASE: m[0][0] = o; m[1][1] = Cx{std::cos(t), std::sin(t)}; return 2;
    case ALEPH_GATE_U3: {
      const double f = g.params[1], l = g.params[2];
      const Cx c{std::cos(t / 2), 0}, s{std::sin(t / 2), 0};
      m[0][0] = c;
      m[0][1] = neg(mul(Cx{std::cos(l), std::sin(l)}, s));
      m[1][0] = mul(Cx{std::cos(f), std::sin(f)}, s);
      m[1][1] = mul(Cx{std::cos(f + l), std::sin(f + l)}, c);
      return 2;
    }
    case ALEPH_GATE_CNOT: m[0][0] = m[1][1] = m[2][3] = m[3][2] = o; return 4;
    case ALEPH_GATE_CZ: m[0][0] = m[1][1] = m[2][2] = o; m[3][3] = neg(o); return 4;
    case ALEPH_GATE_SWAP: m[0][0] = m[1][2] = m[2][1] = m[3][3] = o; return 4;
    case ALEPH_GATE_ISWAP: m[0][0] = m[3][3] = o; m[1][2] = m[2][1] = Cx{0, 1}; return 4;
    case ALEPH_GATE_ISWAPDG: m[0][0] = m[3][3] = o; m[1][2] = m[2][1] = Cx{0, -1}; return 4;
    case ALEPH_GATE_CRX:
      m[0][0] = m[1][1] = o;
      m[2][2] = m[3][3] = Cx{std::cos(t / 2), 0};
      m[2][3] = m[3][2] = Cx{0, -std::sin(t / 2)};
      return 4;
    case ALEPH_GATE_CRY:
      m[0][0] = m[1][1] = o;
      m[2][2] = m[3][3] = Cx{std::cos(t / 2), 0};
      m[2][3] = Cx{-std::sin(t / 2), 0};
      m[3][2] = Cx{std::sin(t / 2), 0};
      return 4;
    case ALEPH_GATE_CRZ:
      m[0][0] = m[1][1] = o;
      m[2][2] = Cx{std::cos(t / 2), -std::sin(t / 2)};
      m[3][3] = Cx{std::cos(t / 2), std::sin(t / 2)};
      return 4;
    case ALEPH_GATE_TOFFOLI:
      for (int i = 0; i < 6; ++i) m[i][i] = o;
      m[6][7] = m[7][6] = o;
      return 8;
    case ALEPH_GATE_CCZ:
      for (int i = 0; i < 7; ++i) m[i][i] = o;
      m[7][7] = neg(o);
      return 8;
    case ALEPH_GATE_UNITARY1Q: {
      const double* p = from_pool(4);
      if (!p) return 0;
      for (int i = 0; i < 4; ++i) m[i / 2][i % 2] = Cx{p[2 * i], p[2 * i + 1]};
      return 2;
    }
    case ALEPH_GATE_UNITARY2Q: {
      const double* p = from_pool(16);
      if (!p) return 0;
      for (int i = 0; i < 16; ++i) m[i / 4][i % 4] = Cx{p[2 * i], p[2 * i + 1]};
      return 4;
    }
    case ALEPH_GATE_UNITARY1QDIAG: {
      const double* p = from_pool(2);
      if (!p) return 0;
      m[0][0] = Cx{p[0], p[1]};
      m[1][1] = Cx{p[2], p[3]};
      return 2;
    }
    case ALEPH_GATE_UNITARY2QDIAG: {
      const double* p = from_pool(4);
      if (!p) return 0;
      for (int i = 0; i < 4; ++i) m[i][i] = Cx{p[2 * i], p[2 * i + 1]};
      return 4;
    }
  }
  set_kind(e, gate_name(g.kind));
  fail(e, ALEPH_B200_UNSUPPORTED_GATE);
  return 0;
}

double unitarity_deviation(const Cx* m, int dim) {
  double worst = 0.0;
  for (int i = 0; i < dim; ++i)
    for (int j = 0; j < dim; ++j) {
      Cx acc{0, 0};
      for (int c = 0; c < dim; ++c) acc = add(acc, mul(m[i * dim + c], conj(m[j * dim + c])));
      const Cx d = sub(acc, Cx{i == j ? 1.0 : 0.0, 0});
      const double dev = std::hypot(d.re, d.im);
      if (std::isnan(dev)) return NAN;
      if (dev > worst) worst = dev;
    }
  return worst;
}

bool is_zero(Cx a) { return a.re == 0.0 && a.im == 0.0; }
bool is_one(Cx a) { return a.re == 1.0 && a.im == 0.0; }
bool is_minus_one(Cx a) { return a.re == -1.0 && a.im == 0.0; }  // re alone rounds to -1 up to 1e-8 away from it

void push_coef(Lowered* L, const Cx* c, int count) {
  const double* d = reinterpret_cast<const double*>(c);
  L->coef.insert(L->coef.end(), d, d + 2 * count);
}

// Lower a validated dense matrix with MSB-first targets to the cheapest op.
void lower_matrix(const Cx* m, int dim, const uint32_t* tq, uint64_t ctrl, Lowered* L) {
  Op& op = L->op;
  std::memset(&op, 0, sizeof(op));
  op.ctrl = ctrl;
  const int k = dim == 2 ? 1 : dim == 4 ? 2 : dim == 8 ? 3 : dim == 16 ? 4 : 5;
  uint64_t tmask = 0;
  for (int i = 0; i < k; ++i) tmask |= 1ull << tq[i];
  bool diag = true;
  for (int i = 0; i < dim && diag; ++i)
    for (int j = 0; j < dim; ++j)
      if (i != j && !is_zero(m[i * dim + j])) {
        diag = false;
        break;
      }
  if (diag) {
    // diag(1, ..., 1, c): phase on the all-ones corner
    bool corner = true;
    for (int i = 0; i + 1 < dim; ++i)
      if (!is_one(m[i * dim + i])) corner = false;
    const Cx c = m[dim * dim - 1];
    L->nondiag = 0;
    L->diag = tmask | ctrl;
    if (corner) {
      op.mask = tmask | ctrl;
      op.ctrl = 0;
      if (is_minus_one(c)) {
        op.type = OP_NEG;
      } else {
        op.type = OP_CPHASE;
        push_coef(L, &c, 1);
      }
      return;
    }
    if (k <= 3) {
      op.type = OP_DIAG;
      op.nq = (uint8_t)k;
      for (int i = 0; i < k; ++i) op.q[i] = (uint8_t)tq[i];
      Cx d[8];
      for (int i = 0; i < dim; ++i) d[i] = m[i * dim + i];
      push_coef(L, d, dim);
      return;
    }
  }
  // controlled blocks: a 2q matrix I (+) U with the MSB as control -> 1q with control
  if (dim == 4 && is_one(m[0]) && is_zero(m[1]) && is_zero(m[2]) && is_zero(m[3]) && is_zero(m[4]) &&
      is_one(m[5]) && is_zero(m[6]) && is_zero(m[7]) && is_zero(m[8]) && is_zero(m[9]) && is_zero(m[12]) &&
      is_zero(m[13])) {
    const Cx u[4] = {m[10], m[11], m[14], m[15]};
    uint32_t t1 = tq[1];
    lower_matrix(u, 2, &t1, ctrl | (1ull << tq[0]), L);
    return;
  }
  // Toffoli / controlled-controlled-U pattern (8x8 identity except the last 2x2 block)
  if (dim == 8) {
    bool cc = true;
    for (int i = 0; i < 8 && cc; ++i)
      for (int j = 0; j < 8; ++j) {
        if (i >= 6 && j >= 6) continue;
        const Cx v = m[i * 8 + j];
        if (i == j ? !is_one(v) : !is_zero(v)) {
          cc = false;
          break;
        }
      }
    if (cc) {
      const Cx u[4] = {m[54], m[55], m[62], m[63]};
      uint32_t t2 = tq[2];
      lower_matrix(u, 2, &t2, ctrl | (1ull << tq[0]) | (1ull << tq[1]), L);
      return;
    }
  }
  L->nondiag = tmask;
  L->diag = ctrl;
  if (dim == 2) {
    op.nq = 1;
    op.q[0] = (uint8_t)tq[0];
    if (is_zero(m[0]) && is_one(m[1]) && is_one(m[2]) && is_zero(m[3])) {
      op.type = OP_X;
      return;
    }
    op.type = OP_1Q;
    push_coef(L, m, 4);
    return;
  }
  if (dim == 4) {
    op.type = OP_2Q;
    op.nq = 2;
    op.q[0] = (uint8_t)tq[0];
    op.q[1] = (uint8_t)tq[1];
    push_coef(L, m, 16);
    return;
  }
  op.type = OP_KQ;
  op.nq = (uint8_t)k;
  for (int i = 0; i < k; ++i) op.q[i] = (uint8_t)tq[i];
  push_coef(L, m, dim * dim);
}

}  // namespace

int gate_matrix_dense(const aleph_b200_instr& g, const double* pool, uint64_t pool_len, double* out, int* dim,
                      aleph_b200_error_info* e) {
  Cx m[8][8];
  const int d = matrix_of(g, pool, pool_len, m, e);
  if (d == 0) return e->status ? e->status : ALEPH_B200_UNSUPPORTED_GATE;
  for (int i = 0; i < d; ++i)
    for (int j = 0; j < d; ++j) {
      out[2 * (i * d + j)] = m[i][j].re;
      out[2 * (i * d + j) + 1] = m[i][j].im;
    }
  *dim = d;
  return ALEPH_B200_OK;
}

const char* gate_name(uint32_t kind) {
  static const char* names[] = {"H",   "X",   "Y",   "Z",   "S",     "Sdg",     "T",       "Tdg",
                                "Rx",  "Ry",  "Rz",  "Phase", "U3",  "Cnot",    "Cz",      "Swap",
                                "Iswap", "IswapDg", "CRx", "CRy", "CRz", "Toffoli", "Ccz", "Unitary1q",
                                "Unitary2q", "UnitaryKq", "Unitary1qDiag", "Unitary2qDiag"};
  if (kind < 28) return names[kind];
  switch (kind) {
    case ALEPH_INSTR_MEASURE: return "measure";
    case ALEPH_INSTR_RESET: return "reset";
    case ALEPH_INSTR_BARRIER: return "barrier";
    case ALEPH_INSTR_DIAGONAL_PHASE: return "diagonal_phase";
    case ALEPH_INSTR_TILED_BLOCK: return "tiled_block";
  }
  return "unknown";
}

int lower_gate(const aleph_b200_instr& g, uint32_t n, const double* pool, uint64_t pool_len, Lowered* L,
               aleph_b200_error_info* e, bool tiled) {
  const int expected = arity(g);
  if (expected < 0) {
    set_kind(e, gate_name(g.kind));
    return fail(e, ALEPH_B200_UNSUPPORTED_GATE);
  }
  if ((uint32_t)expected != g.num_qubits) {
    set_kind(e, gate_name(g.kind));
    e->expected = (uint32_t)expected;
    e->got = g.num_qubits;
    return fail(e, ALEPH_B200_ARITY_MISMATCH);
  }
  if (g.num_qubits > 8 || g.num_controls > 8) {
    set_kind(e, "record");
    return fail(e, ALEPH_B200_INVALID_ARGUMENT);
  }
  uint32_t seen[16];
  uint32_t ns = 0;
  uint64_t ctrl = 0;
  for (uint32_t i = 0; i < g.num_qubits + g.num_controls; ++i) {
    const uint32_t q = i < g.num_qubits ? g.qubits[i] : g.controls[i - g.num_qubits];
    if (q >= n) {
      e->qubit = q;
      e->num_qubits = n;
      return fail(e, ALEPH_B200_QUBIT_OUT_OF_RANGE);
    }
    for (uint32_t j = 0; j < ns; ++j)
      if (seen[j] == q) {
        e->qubit = q;
        return fail(e, ALEPH_B200_DUPLICATE_QUBIT);
      }
    seen[ns++] = q;
    if (i >= g.num_qubits) ctrl |= 1ull << q;
  }
  if (tiled && g.kind == ALEPH_GATE_UNITARYKQ) {
    // a gate of a TiledBlock goes through Gate::matrix() only
    // (dispatch_tile_kernel, crates/aleph-sv/src/backend.rs:265-299), and a
    // UnitaryKq has no fixed-size matrix there: UnsupportedGate
    set_kind(e, gate_name(g.kind));
    return fail(e, ALEPH_B200_UNSUPPORTED_GATE);
  }
  L->given = g.kind >= ALEPH_GATE_UNITARY1Q && g.kind <= ALEPH_GATE_UNITARY2QDIAG;
  if (g.kind == ALEPH_GATE_UNITARYKQ) {
    // validate_unitary_kq, crates/aleph-sv/src/validation.rs:113-155
    const uint32_t k = g.aux;
    if (k < 2 || k > 5) {
      set_kind(e, "UnitaryKq width");
      return fail(e, ALEPH_B200_INVALID_STATE);
    }
    if (g.num_controls) {
      set_kind(e, "controlled UnitaryKq");
      return fail(e, ALEPH_B200_UNSUPPORTED_GATE);
    }
    const uint64_t w = 1ull << k;
    if (g.data_len != w * w) {
      set_kind(e, "UnitaryKq length");
      return fail(e, ALEPH_B200_INVALID_STATE);
    }
    if (!pool || g.data_offset + g.data_len > pool_len) {
      set_kind(e, "matrix pool");
      return fail(e, ALEPH_B200_INVALID_ARGUMENT);
    }
    const Cx* d = reinterpret_cast<const Cx*>(pool + 2 * g.data_offset);
    for (uint64_t i = 0; i < w * w; ++i)
      if (!std::isfinite(d[i].re) || !std::isfinite(d[i].im)) {
        set_kind(e, "UnitaryKq");
        return fail(e, ALEPH_B200_NON_FINITE_PARAM);
      }
    double dev2 = 0.0;
    for (uint64_t i = 0; i < w; ++i)
      for (uint64_t j = 0; j <= i; ++j) {
        Cx s{0, 0};
        for (uint64_t c = 0; c < w; ++c) s = add(s, mul(d[i * w + c], conj(d[j * w + c])));
        const Cx df = sub(s, Cx{i == j ? 1.0 : 0.0, 0});
        const double er = df.re * df.re + df.im * df.im;
        if (!std::isfinite(er)) {
          e->value = er;
          return fail(e, ALEPH_B200_NON_UNITARY_MATRIX);
        }
        dev2 = std::max(dev2, er);
      }
    if (dev2 > kTol * kTol) {
      e->value = std::sqrt(dev2);
      return fail(e, ALEPH_B200_NON_UNITARY_MATRIX);
    }
    L->record = 0;
    lower_matrix(d, (int)w, g.qubits, 0, L);
    return ALEPH_B200_OK;
  }
  Cx m[8][8];
  const int dim = matrix_of(g, pool, pool_len, m, e);
  if (dim == 0) return e->status;
  Cx flat[64];
  for (int i = 0; i < dim; ++i)
    for (int j = 0; j < dim; ++j) flat[i * dim + j] = m[i][j];
  if (tiled) {
    // TiledBlock gates: the tile kernels take 2x2 and 4x4 matrices; an 8x8
    // is UnsupportedGate, and no unitarity check is made (backend.rs:265-299)
    if (dim > 4) {
      set_kind(e, gate_name(g.kind));
      return fail(e, ALEPH_B200_UNSUPPORTED_GATE);
    }
    lower_matrix(flat, dim, g.qubits, ctrl, L);
    return ALEPH_B200_OK;
  }
  const double dev = unitarity_deviation(flat, dim);
  if (!std::isfinite(dev) || dev > kTol) {
    e->value = dev;
    return fail(e, ALEPH_B200_NON_UNITARY_MATRIX);
  }
  lower_matrix(flat, dim, g.qubits, ctrl, L);
  return ALEPH_B200_OK;
}

int lower_diagonal_phase(const aleph_b200_phase_term* terms, uint64_t n_terms, const uint64_t* conds, uint64_t n_conds,
                         Lowered* L, aleph_b200_error_info* e) {
  std::memset(&L->op, 0, sizeof(L->op));
  L->op.type = OP_POLY;
  L->op.aux = (uint32_t)n_terms;
  uint64_t support = 0;
  for (uint64_t t = 0; t < n_terms; ++t) {
    if ((uint64_t)terms[t].cond_offset + terms[t].cond_count > n_conds || (!conds && terms[t].cond_count)) {
      set_kind(e, "diagonal phase conds");
      return fail(e, ALEPH_B200_INVALID_ARGUMENT);
    }
    L->poly_angle.push_back(terms[t].angle);
    L->poly_cnt.push_back(terms[t].cond_count);
    for (uint32_t c = 0; c < terms[t].cond_count; ++c) {
      L->poly_conds.push_back(conds[terms[t].cond_offset + c]);
      support |= conds[terms[t].cond_offset + c];
    }
  }
  L->nondiag = 0;
  L->diag = support;
  return ALEPH_B200_OK;
}

// ---------------------------------------------------------------------------
// planning
// ---------------------------------------------------------------------------
namespace {

uint32_t append_op(Plan* P, const Lowered& L, Op op) {
  op.coef = (uint32_t)(P->coef.size() / 2);
  P->coef.insert(P->coef.end(), L.coef.begin(), L.coef.end());
  if (op.type == OP_POLY) {
    op.mask = P->poly_angle.size();
    uint32_t off = 0;
    for (size_t t = 0; t < L.poly_angle.size(); ++t) {
      P->poly_angle.push_back(L.poly_angle[t]);
      P->poly_off.push_back((uint32_t)P->poly_conds.size());
      P->poly_cnt.push_back(L.poly_cnt[t]);
      for (uint32_t c = 0; c < L.poly_cnt[t]; ++c) P->poly_conds.push_back(L.poly_conds[off + c]);
      off += L.poly_cnt[t];
    }
  }
  P->ops.push_back(op);
  return (uint32_t)(P->ops.size() - 1);
}

// Cost-model features of a pass from the ops it applies.
void count_ops(const std::vector<const Lowered*>& ops, Pass* ps) {
  for (const Lowered* L : ops) {
    switch (L->op.type) {  // a complex multiply-add is 4 real ones
      case OP_1Q: ps->fma_per_amp += 8; break;
      case OP_2Q: ps->fma_per_amp += 16; break;
      case OP_KQ: ps->fma_per_amp += 4u << L->op.nq; break;
      case OP_CPHASE: case OP_DIAG: case OP_POLY: ps->fma_per_amp += 4; break;
      default: break;  // X and sign flips move or negate
    }
    if (L->nondiag) {
      ++ps->dense_ops;
      if (L->nondiag & 0x1Full) ++ps->lane_ops;
    } else {
      ++ps->diag_ops;
    }
  }
}

// Swap the operand order of a 4x4 matrix (MSB <-> LSB).
void swap_2q_operands(std::vector<double>& c) {
  std::vector<double> out(c.size());
  auto sw = [](int k) { return ((k & 1) << 1) | (k >> 1); };
  for (int r = 0; r < 4; ++r)
    for (int cc = 0; cc < 4; ++cc) {
      const int src = 2 * (4 * r + cc), dst = 2 * (4 * sw(r) + sw(cc));
      out[dst] = c[src];
      out[dst + 1] = c[src + 1];
    }
  c = out;
}

// ---- pair fusion (warp-tile passes) ------------------------------------------
// A tile pass applies its gates one at a time in registers, so its arithmetic
// is the sum of the gates': 8 FP64 multiply-adds per amplitude for a dense
// one-qubit gate, 16 for a dense two-qubit one, one or two for a diagonal.
// In FP64 the pass is bound by that arithmetic. A two-qubit gate together
// with the one-qubit gates around it on its two qubits is one 4x4 (16 per
// amplitude): in a brickwall, the one-qubit layers on both sides of a CZ,
// four dense gates (32) for one 4x4 (16).
//
// The rule, in gate order: one-qubit gates wait on their qubit. A gate on
// exactly two qubits a, b opens a block that takes the waiting one-qubit
// gates of a and b, itself, then every later gate on a and/or b alone, until
// a gate touches a or b together with another qubit. The block is then
// emitted as one 4x4 when its gates cost at least 24 per amplitude; otherwise
// its gates are emitted unchanged and the one-qubit gates at its end wait
// again on their qubits (so a CZ between two already-absorbed layers leaves
// the next layer to the next block). This is the idea of Fuse2q
// (crates/aleph-ir/src/passes/fuse_2q.rs) with a cost rule for register tiles.
namespace {

int tile_cost(const Lowered& L) {
  switch (L.op.type) {
    case OP_1Q: return 8;
    case OP_2Q: return 16;
    case OP_X: case OP_NEG: return 1;
    case OP_CPHASE: case OP_DIAG: return 2;
    default: return 32;
  }
}

constexpr int kFuseMinCost = 24;

// Every coefficient's imaginary part is exactly zero.
bool real_matrix(const Lowered& L) {
  for (size_t c = 1; c < L.coef.size(); c += 2)
    if (L.coef[c] != 0.0) return false;
  return true;
}

// |c| = 1 to rounding. A TiledBlock's matrices are taken as they are, so a
// diagonal's entries need not be phases.
bool unimodular(Cx c) { return std::fabs(std::hypot(c.re, c.im) - 1.0) <= 1e-15; }

// A phase, exactly +-1 or +-i where it lies within `tol` of that. tol is what the
// rounding of the phase's own product can have moved it by, so that no angle is
// dropped that its gates had.
Cx snapped(Cx c, double tol) {
  if (std::fabs(c.im) <= tol) return Cx{c.re > 0 ? 1.0 : -1.0, 0.0};
  if (std::fabs(c.re) <= tol) return Cx{0.0, c.im > 0 ? 1.0 : -1.0};
  return c;
}

// Source gates that an op stands for.
uint32_t gates_of(const Lowered& L) { return L.absorbed ? 0 : L.gates ? L.gates : 1; }

// The 4x4 of an op on qubits {a (matrix MSB), b (LSB)}, left-multiplied into m:
// m := op * m. At most 64 complex products; the plan of a state that fits one SM
// is made of these, and it is made again for every new set of angles.
void fold_into_4x4(const Lowered& L, uint32_t a, uint32_t b, Cx* m) {
  const Op& op = L.op;
  const Cx* c = reinterpret_cast<const Cx*>(L.coef.data());
  auto rows = [&](uint64_t q) { return (uint32_t)(((q >> b) & 1) | (((q >> a) & 1) << 1)); };  // qubit mask -> row bits
  switch (op.type) {
    case OP_NEG:
    case OP_CPHASE: {
      const uint32_t mask = rows(op.mask);
      const Cx f = op.type == OP_NEG ? Cx{-1, 0} : c[0];
      for (uint32_t r = 0; r < 4; ++r)
        if ((r & mask) == mask)
          for (uint32_t k = 0; k < 4; ++k) m[r * 4 + k] = mul(f, m[r * 4 + k]);
      return;
    }
    case OP_DIAG: {
      const uint32_t ctrl = rows(op.ctrl);
      for (uint32_t r = 0; r < 4; ++r) {
        if ((r & ctrl) != ctrl) continue;
        uint32_t idx = 0;
        for (int i = 0; i < op.nq; ++i) idx = (idx << 1) | (op.q[i] == a ? r >> 1 : r & 1);
        for (uint32_t k = 0; k < 4; ++k) m[r * 4 + k] = mul(c[idx], m[r * 4 + k]);
      }
      return;
    }
    case OP_X:
    case OP_1Q: {
      const uint32_t bit = rows(1ull << op.q[0]), ctrl = rows(op.ctrl);
      for (uint32_t r = 0; r < 4; ++r) {
        if ((r & bit) || (r & ctrl) != ctrl) continue;
        Cx *x = m + r * 4, *y = m + (r | bit) * 4;
        for (uint32_t k = 0; k < 4; ++k) {
          const Cx u = x[k], v = y[k];
          x[k] = op.type == OP_X ? v : add(mul(c[0], u), mul(c[1], v));
          y[k] = op.type == OP_X ? u : add(mul(c[2], u), mul(c[3], v));
        }
      }
      return;
    }
    default: {  // OP_2Q, operands in either order
      const uint32_t hi = rows(1ull << op.q[0]), lo = rows(1ull << op.q[1]);
      const uint32_t at[4] = {0, lo, hi, hi | lo};
      Cx out[16];
      for (uint32_t r = 0; r < 4; ++r)
        for (uint32_t k = 0; k < 4; ++k) {
          Cx acc = mul(c[r * 4], m[at[0] * 4 + k]);
          for (uint32_t t = 1; t < 4; ++t) acc = add(acc, mul(c[r * 4 + t], m[at[t] * 4 + k]));
          out[at[r] * 4 + k] = acc;
        }
      for (int i = 0; i < 16; ++i) m[i] = out[i];
      return;
    }
  }
}

// A product of named gates gets rows of length 1 again, where the rounding of
// `gates` factors moved them. That rounding is the same wherever the gates are (an
// H has a squared norm of 1 + 1.4e-16, the rounded product of two 1 + 4.4e-16), so
// it adds up over a circuit: FP64 Grover, n = 10, depth 4, was 1.7e-14 from the
// exact state (1.1e-14 gate by gate) and is 3.9e-15. Not for a matrix that the
// caller gave: its entries are exact as they are.
void unit_rows(Cx* m, int dim, uint32_t gates) {
  long double len2[4];
  for (int r = 0; r < dim; ++r) {
    len2[r] = 0;
    for (int k = 0; k < dim; ++k) {
      const long double x = m[r * dim + k].re, y = m[r * dim + k].im;
      len2[r] += x * x + y * y;
    }
    if (!(std::fabs((double)(len2[r] - 1)) <= 0x1p-50 * gates)) return;
  }
  for (int r = 0; r < dim; ++r) {
    const long double f = 1 / std::sqrt(len2[r]);
    for (int k = 0; k < dim; ++k) {
      Cx& c = m[r * dim + k];
      c = Cx{(double)(c.re * f), (double)(c.im * f)};
    }
  }
}

bool fusable_type(const Lowered& L) {
  return !L.is_measure && !L.is_permute && L.op.type != OP_POLY && L.op.type != OP_KQ;
}

}  // namespace

// ---- diagonal cores -------------------------------------------------------------------------------
// Gate sequences on two or three qubits often multiply out to a diagonal: the
// CX Rz CX of a ZZ rotation, a Toffoli in CX + T without the H around it. As
// written they move amplitudes and tie their qubits to a pass; as a diagonal
// they are sign flips and corner phases, which act on any qubit and are grouped.
//
// Gates are gathered greedily into blocks of at most three qubits (a block
// owns its qubits until a gate joins them to others). Of a closed block, the core
// runs from each qubit's first to its last gate on several qubits; the
// one-qubit gates outside it stay. A core of X-like and diagonal gates whose moves
// cancel is replaced by its corner phases when those cost less than its gates,
// an amplitude-moving gate counted as 8. The phases of all cores on no qubit are one op
// at the end.
//
// In shared-memory passes (`smem`) a run of gates on one pair of qubits costs one 4x4,
// about what two phases cost there, so only cores cheaper than their runs at that
// price are taken: the CCZ of a Toffoli (six runs, one sign flip) is, a ZZ rotation (one
// run, three phases) is not (n = 8 FP32 QAOA, p = 2: 48 us with it, 38 without).
std::vector<const Lowered*> diagonal_cores(const std::vector<const Lowered*>& seg, std::deque<Lowered>& store,
                                           bool smem = false) {
  struct Block {
    uint64_t qubits = 0;
    std::vector<size_t> members;  // indices in seg, ascending; empty: no block
  };
  // Ops with the place they go to (sorted at the end, so that gates that stay keep
  // their order): a gate's own index in seg; for corner phases, the last of the
  // first core gates on their qubits, which is behind all that earlier blocks did there.
  std::vector<std::pair<size_t, const Lowered*>> out;
  out.reserve(seg.size());
  std::vector<Block> blocks;         // open ones; each owns its qubits
  int owner[64];                     // per qubit: its block, or -1
  std::fill(owner, owner + 64, -1);
  bool changed = false;  // some op goes out in another form or place than it came
  Cx global{1.0, 0.0};
  uint32_t last_record = 0;
  auto width = [](const Lowered& L) { return __builtin_popcountll(L.nondiag | L.diag); };
  auto corner = [&](size_t at, uint64_t mask, Cx c, uint32_t record, uint32_t gates) {
    changed = true;
    store.emplace_back();
    Lowered& F = store.back();
    std::memset(&F.op, 0, sizeof(Op));
    F.op.mask = mask;
    F.nondiag = 0;
    F.diag = mask;
    F.record = record;
    F.gates = gates;
    F.absorbed = gates == 0;
    if (is_minus_one(c)) {
      F.op.type = OP_NEG;
    } else {
      F.op.type = OP_CPHASE;
      push_coef(&F, &c, 1);
    }
    out.emplace_back(at, &F);
  };
  // A gate that stays, at `at`. A table diagonal on one qubit (with up to two
  // controls) becomes its corner phases too: the one on the qubits' ones and the
  // one on the controls alone, which without controls joins the global phase.
  auto keep = [&](size_t at, size_t m) {
    const Lowered& L = *seg[m];
    if (L.op.type != OP_DIAG || L.op.nq != 1) {
      out.emplace_back(at, &L);
      return;
    }
    const Cx* d = reinterpret_cast<const Cx*>(L.coef.data());
    if (!unimodular(d[0]) || !unimodular(d[1])) {  // keep the table
      out.emplace_back(at, &L);
      return;
    }
    corner(at, L.op.ctrl | 1ull << L.op.q[0], mul(d[1], conj(d[0])), L.record, gates_of(L));
    if (L.op.ctrl) {
      if (!is_one(d[0])) corner(at, L.op.ctrl, d[0], L.record, 0);
    } else {
      global = mul(global, d[0]);
      last_record = L.record;
    }
  };
  std::vector<size_t> before, after;
  std::vector<const Lowered*> core;
  auto emit = [&](const Block& B) {
    uint32_t bq[3] = {0, 0, 0}, nb = 0;
    for (uint64_t t = B.qubits; t; t &= t - 1) bq[nb++] = (uint32_t)__builtin_ctzll(t);
    const uint32_t dim = 1u << nb;
    auto local = [&](uint64_t m) {  // qubit mask -> bits of the block's index
      uint32_t r = 0;
      for (uint32_t b = 0; b < nb; ++b) r |= (uint32_t)((m >> bq[b]) & 1) << b;
      return r;
    };
    size_t first[3] = {SIZE_MAX, SIZE_MAX, SIZE_MAX}, last[3] = {0, 0, 0};  // per qubit: its gates on several qubits
    uint32_t multi = 0;
    for (size_t k = 0; k < B.members.size(); ++k) {
      const Lowered& L = *seg[B.members[k]];
      if (width(L) < 2) continue;
      ++multi;
      const uint32_t on = local(L.nondiag | L.diag);
      for (uint32_t b = 0; b < nb; ++b)
        if ((on >> b) & 1) {
          first[b] = std::min(first[b], k);
          last[b] = k;
        }
    }
    auto plain = [&] {
      for (size_t m : B.members) keep(m, m);
    };
    if (multi < 2) return plain();
    before.clear();
    after.clear();
    core.clear();
    size_t place = 0;  // behind everything that came before the block on any of the core's qubits
    for (uint32_t b = 0; b < nb; ++b)
      if (first[b] != SIZE_MAX) place = std::max(place, B.members[first[b]]);
    int cost = 0;
    uint32_t gates = 0;
    bool monomial = true;  // a core with a dense member is left alone
    for (size_t k = 0; k < B.members.size(); ++k) {
      const Lowered* L = seg[B.members[k]];
      if (width(*L) < 2) {
        const int b = __builtin_ctz(local(L->nondiag | L->diag));
        if (first[b] == SIZE_MAX || k < first[b] || k > last[b]) {
          // a qubit without multi-qubit gates keeps its order: everything on it comes first
          (first[b] == SIZE_MAX || k < first[b] ? before : after).push_back(B.members[k]);
          continue;
        }
      }
      if (L->op.type != OP_X && L->nondiag) {
        monomial = false;
        break;
      }
      core.push_back(L);
      cost += L->nondiag ? std::max(8, tile_cost(*L)) : tile_cost(*L);
      gates += gates_of(*L);
    }
    if (!monomial) return plain();
    // The core as a map of basis states with phases: its members are X-like or diagonal.
    const double tol = 1e-15 * (double)(core.size() + 2);
    uint32_t to[8];
    Cx d[8];
    for (uint32_t c = 0; c < dim; ++c) {
      to[c] = c;
      d[c] = Cx{1.0, 0.0};
    }
    uint32_t phases = 0;  // members whose products round
    for (const Lowered* L : core) {
      const Op& op = L->op;
      phases += op.type == OP_CPHASE || op.type == OP_DIAG;
      const Cx* k = reinterpret_cast<const Cx*>(L->coef.data());
      const uint32_t ctrl = local(op.ctrl), mask = local(op.mask), bit = local(1ull << op.q[0]);
      for (uint32_t c = 0; c < dim; ++c) {
        const uint32_t x = to[c];
        if (op.type == OP_X) {
          if ((x & ctrl) == ctrl) to[c] = x ^ bit;
        } else if (op.type == OP_DIAG) {
          if ((x & ctrl) != ctrl) continue;
          uint32_t idx = 0;
          for (int i = 0; i < op.nq; ++i) idx = (idx << 1) | ((x & local(1ull << op.q[i])) ? 1u : 0u);
          d[c] = mul(k[idx], d[c]);
        } else if ((x & mask) == mask) {
          d[c] = op.type == OP_NEG ? neg(d[c]) : mul(k[0], d[c]);
        }
      }
    }
    for (uint32_t c = 0; c < dim; ++c) {
      const double len = std::hypot(d[c].re, d[c].im);
      if (to[c] != c || std::fabs(len - 1.0) > tol) return plain();
      d[c] = Cx{d[c].re / len, d[c].im / len};
    }
    // corner phases: c_S = prod over T in S of d_T^(+-1), sign by the parity of |S| - |T|
    Cx cs[8];
    bool used[8];
    int price = 0;
    for (uint32_t S = 0; S < dim; ++S) {
      Cx c{1.0, 0.0};
      for (uint32_t T = 0; T < dim; ++T)
        if ((T & S) == T) c = mul(c, (__builtin_popcount(S ^ T) & 1) ? conj(d[T]) : d[T]);
      cs[S] = c = snapped(c, std::min(0x1p-49, 0x1p-52 * (double)(2 + phases)));
      used[S] = S != 0 && !is_one(c);
      if (used[S]) price += is_minus_one(c) ? 1 : 2;
    }
    if (smem) {
      int runs = 0;
      uint64_t pair = 0;
      for (const Lowered* L : core) {
        const uint64_t q = L->nondiag | L->diag;
        if (runs == 0 || __builtin_popcountll(pair | q) > 2) {
          ++runs;
          pair = q;
        } else {
          pair |= q;
        }
      }
      cost = 2 * runs;
    }
    if (price >= cost) return plain();
    for (size_t m : before) keep(m, m);
    const uint32_t record = core.front()->record;
    bool any = false;
    for (uint32_t S = 1; S < dim; ++S) {
      if (!used[S]) continue;
      uint64_t mask = 0;
      for (uint32_t b = 0; b < nb; ++b)
        if ((S >> b) & 1) mask |= 1ull << bq[b];
      corner(place, mask, cs[S], record, any ? 0 : gates);
      any = true;
    }
    if (!any) corner(place, 0, Cx{1.0, 0.0}, record, gates);  // the identity, kept for its gate count
    global = mul(global, cs[0]);
    last_record = record;
    for (size_t m : after) keep(std::max(m, place), m);
  };
  auto release = [&](Block& B) {
    for (uint64_t t = B.qubits; t; t &= t - 1) owner[__builtin_ctzll(t)] = -1;
    B.qubits = 0;
    B.members.clear();
  };
  auto close = [&](int k) {
    emit(blocks[(size_t)k]);
    release(blocks[(size_t)k]);
  };
  std::vector<size_t> merged;
  for (size_t i = 0; i < seg.size(); ++i) {
    const Lowered& L = *seg[i];
    const uint64_t touched = L.nondiag | L.diag;
    const bool small = fusable_type(L) && touched && __builtin_popcountll(touched) <= 3;
    // close touched blocks, the widest first (the older of two), until the rest and this gate fit three qubits
    int mine = -1;  // the touched block that stays open and is widened
    for (;;) {
      uint64_t all = touched;
      int widest = -1;
      for (uint64_t t = touched; t; t &= t - 1) {
        const int k = owner[__builtin_ctzll(t)];
        if (k < 0 || k == widest) continue;
        const Block& B = blocks[(size_t)k];
        all |= B.qubits;
        if (widest >= 0) {
          const Block& W = blocks[(size_t)widest];
          const int wide = __builtin_popcountll(B.qubits), most = __builtin_popcountll(W.qubits);
          if (wide < most || (wide == most && B.members.back() >= W.members.back())) continue;
        }
        widest = k;
      }
      mine = widest;
      if (widest < 0 || (small && __builtin_popcountll(all) <= 3)) break;
      close(widest);
    }
    if (!small) {
      keep(i, i);
      continue;
    }
    if (mine < 0) {
      for (mine = 0; mine < (int)blocks.size() && !blocks[(size_t)mine].members.empty();) ++mine;
      if (mine == (int)blocks.size()) blocks.emplace_back();
    }
    Block& M = blocks[(size_t)mine];
    for (uint64_t t = touched; t; t &= t - 1) {
      const int k = owner[__builtin_ctzll(t)];
      if (k >= 0 && k != mine) {  // join it: at most twice in a block's life
        Block& B = blocks[(size_t)k];
        merged.resize(M.members.size() + B.members.size());
        std::merge(M.members.begin(), M.members.end(), B.members.begin(), B.members.end(), merged.begin());
        M.members.swap(merged);
        const uint64_t q = B.qubits;
        release(B);
        M.qubits |= q;
      }
    }
    M.qubits |= touched;
    for (uint64_t t = M.qubits; t; t &= t - 1) owner[__builtin_ctzll(t)] = mine;
    M.members.push_back(i);
  }
  std::sort(blocks.begin(), blocks.end(), [](const Block& x, const Block& y) {  // by their last gates
    return (x.members.empty() ? 0 : x.members.back()) < (y.members.empty() ? 0 : y.members.back());
  });
  for (const Block& B : blocks)
    if (!B.members.empty()) emit(B);
  if (!changed) return seg;
  if (!is_one(global)) corner(SIZE_MAX, 0, global, last_record, 0);
  std::stable_sort(out.begin(), out.end(), [](const auto& x, const auto& y) { return x.first < y.first; });
  std::vector<const Lowered*> ops;
  ops.reserve(out.size());
  for (const auto& o : out) ops.push_back(o.second);
  return ops;
}

// After the cores: phases on the same qubits with nothing between that moves
// one of them become one (T and Tdg cancel), and H, a sign flip on t and others,
// H on t become an X on t controlled by the others. A CX + T Toffoli is then one
// exact move instead of two roundings by sqrt(1/2) and some phases, each of which
// shortens an FP32 state a little in the same direction.
// Measured: n = 22 FP32 Grover 1697 -> 1060 us (19 -> 14 passes), its error against
// 64 bits 1.3e-5 -> 2.4e-6.
std::vector<const Lowered*> cancel_phases(const std::vector<const Lowered*>& seg, std::deque<Lowered>& store) {
  // A mask's last phase op can still be joined while no op behind it moves one of
  // the mask's qubits.
  std::unordered_map<uint64_t, size_t> phase;  // mask -> its last phase op, counted from 1
  size_t moved[64] = {};                       // per qubit: the last op that moves it, counted from 1
  size_t h[64];                                // per qubit: an H with only phases since; SIZE_MAX: none
  std::vector<size_t> since[64];               // those phases
  std::fill(h, h + 64, SIZE_MAX);
  auto is_phase = [](const Lowered& L) {
    return fusable_type(L) && (L.op.type == OP_NEG || L.op.type == OP_CPHASE) && !L.nondiag && L.op.mask && L.diag == L.op.mask;
  };
  auto is_h = [](const Lowered& L) {
    if (!fusable_type(L) || L.op.type != OP_1Q || L.op.ctrl || L.coef.size() < 4 * sizeof(Cx) / sizeof(L.coef[0])) return false;
    const Cx* m = reinterpret_cast<const Cx*>(L.coef.data());
    const double s = std::sqrt(0.5);
    for (int k = 0; k < 4; ++k)
      if (m[k].im != 0.0 || std::fabs(m[k].re - (k == 3 ? -s : s)) > 1e-15) return false;
    return true;
  };
  auto coef = [](const Lowered& L) { return L.op.type == OP_NEG ? Cx{-1.0, 0.0} : *reinterpret_cast<const Cx*>(L.coef.data()); };
  if (std::none_of(seg.begin(), seg.end(), [&](const Lowered* L) { return is_phase(*L); })) return seg;
  std::vector<const Lowered*> ops = seg;
  for (size_t i = 0; i < ops.size(); ++i) {
    const Lowered& L = *ops[i];
    const uint64_t touched = L.nondiag | L.diag;
    if (is_phase(L)) {
      size_t& last = phase[L.op.mask];
      for (uint64_t t = L.op.mask; t; t &= t - 1)
        if (last <= moved[__builtin_ctzll(t)]) last = 0;
      if (last && unimodular(coef(*ops[last - 1])) && unimodular(coef(L))) {  // join the earlier one, here
        const size_t e = last - 1;
        const Lowered& E = *ops[e];
        Cx c = mul(coef(E), coef(L));
        const double len = std::hypot(c.re, c.im);
        c = snapped(Cx{c.re / len, c.im / len}, 0x1p-52);  // one product
        store.emplace_back();
        Lowered& F = store.back();
        std::memset(&F.op, 0, sizeof(Op));
        F.record = L.record;
        F.gates = gates_of(E) + gates_of(L);
        F.absorbed = F.gates == 0;
        F.op.mask = F.diag = L.op.mask;
        F.nondiag = 0;
        if (is_minus_one(c)) {
          F.op.type = OP_NEG;
        } else {
          F.op.type = OP_CPHASE;
          push_coef(&F, &c, 1);
        }
        const bool gone = is_one(c);
        if (gone) F.op.mask = F.diag = 0;  // the identity, kept for its gate count
        // an H before the earlier phase sees the joined one instead
        for (uint64_t t = L.op.mask; t; t &= t - 1) {
          const int q = __builtin_ctzll(t);
          if (h[q] == SIZE_MAX) continue;
          auto& list = since[q];
          list.erase(std::remove(list.begin(), list.end(), e), list.end());
          if (!gone) list.push_back(i);
        }
        ops[e] = nullptr;
        ops[i] = &F;
        last = gone ? 0 : i + 1;
        continue;
      }
      last = i + 1;
      for (uint64_t t = L.op.mask; t; t &= t - 1)
        if (h[__builtin_ctzll(t)] != SIZE_MAX) since[__builtin_ctzll(t)].push_back(i);
      continue;
    }
    const int q = touched ? __builtin_ctzll(touched) : 0;
    if (is_h(L) && h[q] != SIZE_MAX && since[q].size() == 1 && ops[since[q][0]]->op.type == OP_NEG &&
        ops[since[q][0]]->op.mask != touched) {
      const size_t at = since[q][0];
      const Lowered& N = *ops[at];
      const uint64_t others = N.op.mask & ~touched;
      store.emplace_back();
      Lowered& F = store.back();
      std::memset(&F.op, 0, sizeof(Op));
      F.record = N.record;
      F.gates = gates_of(*ops[h[q]]) + gates_of(N) + gates_of(L);
      F.absorbed = F.gates == 0;
      F.op.type = OP_X;
      F.op.nq = 1;
      F.op.q[0] = (uint8_t)q;
      F.op.ctrl = F.diag = others;
      F.nondiag = touched;
      ops[h[q]] = ops[i] = nullptr;
      for (uint64_t t = others; t; t &= t - 1) h[__builtin_ctzll(t)] = SIZE_MAX;  // the flip is gone from their runs
      ops[at] = &F;
      h[q] = SIZE_MAX;
    } else {
      for (uint64_t t = touched; t; t &= t - 1) h[__builtin_ctzll(t)] = SIZE_MAX;
      if (is_h(L)) {
        h[q] = i;
        since[q].clear();
      }
    }
    for (uint64_t t = L.nondiag; t; t &= t - 1) moved[__builtin_ctzll(t)] = i + 1;
  }
  ops.erase(std::remove(ops.begin(), ops.end(), nullptr), ops.end());
  return ops;
}

// barrier_cost: what an op that moves amplitudes costs beside its arithmetic
// (shared-memory passes: a barrier and its latency); 0 in tile passes.
std::vector<const Lowered*> fuse_pairs(const std::vector<const Lowered*>& seg, std::deque<Lowered>& store,
                                       int barrier_cost = 0) {
  const int min_cost = barrier_cost ? 17 + barrier_cost : kFuseMinCost;
  auto gate_cost = [&](const Lowered& L) { return tile_cost(L) + (L.nondiag ? barrier_cost : 0); };
  // Lists (a block's members, the gates waiting on a qubit) are links in one
  // array: no allocation for each.
  struct Link {
    size_t at;  // an index in seg (members) or in out (waiting)
    int next;
  };
  struct List {
    int head = -1, tail = -1;
  };
  std::vector<Link> links;
  links.reserve(2 * seg.size());
  auto append = [&](List& l, size_t at) {
    links.push_back(Link{at, -1});
    const int k = (int)links.size() - 1;
    if (l.tail >= 0) links[(size_t)l.tail].next = k;
    else l.head = k;
    l.tail = k;
  };
  struct Block {
    uint32_t a, b;
    Cx m[16];
    List members;
    int cost = 0;
    uint32_t record = 0, gates = 0;
    bool given = false;
  };
  std::vector<const Lowered*> out;
  out.reserve(seg.size());
  List waiting[kMaxQubits];  // one-qubit gates waiting per qubit
  int open[kMaxQubits];
  std::fill(open, open + kMaxQubits, -1);
  std::vector<Block> blocks;
  blocks.reserve(seg.size() / 3 + 1);
  auto member = [&](Block& B, const Lowered* L, size_t at) {
    fold_into_4x4(*L, B.a, B.b, B.m);
    append(B.members, at);
    B.cost += gate_cost(*L);
    B.gates += gates_of(*L);
    B.given = B.given || L->given;
  };
  std::vector<size_t> source;  // per op of out: its index in seg
  source.reserve(seg.size());
  auto emit = [&](const Lowered* L, size_t at) {
    out.push_back(L);
    source.push_back(at);
  };
  auto close = [&](uint32_t q) {
    const int k = open[q];
    if (k < 0) return;
    Block& B = blocks[(size_t)k];
    open[B.a] = open[B.b] = -1;
    waiting[B.a] = waiting[B.b] = List();
    if (B.cost >= min_cost) {
      store.emplace_back();
      Lowered& F = store.back();
      std::memset(&F.op, 0, sizeof(Op));
      F.op.type = OP_2Q;
      F.op.nq = 2;
      F.op.q[0] = (uint8_t)B.a;
      F.op.q[1] = (uint8_t)B.b;
      F.given = B.given;
      if (!F.given) unit_rows(B.m, 4, B.gates);
      push_coef(&F, B.m, 16);
      F.nondiag = (1ull << B.a) | (1ull << B.b);
      F.diag = 0;
      F.record = B.record;
      F.gates = B.gates;
      emit(&F, 0);
      return;
    }
    // not worth a 4x4: the gates go out as they came; the one-qubit gates
    // after the block's last two-qubit gate wait again on their qubits
    int last2 = -1;
    for (int i = B.members.head; i >= 0; i = links[(size_t)i].next) {
      const Lowered* L = seg[links[(size_t)i].at];
      if (__builtin_popcountll(L->nondiag | L->diag) == 2) last2 = i;
    }
    bool behind = false;
    for (int i = B.members.head; i >= 0; i = links[(size_t)i].next) {
      const size_t at = links[(size_t)i].at;
      emit(seg[at], at);
      if (behind) append(waiting[__builtin_ctzll(seg[at]->nondiag | seg[at]->diag)], out.size() - 1);
      behind = behind || i == last2;
    }
  };
  for (size_t at = 0; at < seg.size(); ++at) {
    const Lowered* L = seg[at];
    const uint64_t touched = L->nondiag | L->diag;
    const int width = __builtin_popcountll(touched);
    if (fusable_type(*L) && width == 1) {
      const uint32_t q = (uint32_t)__builtin_ctzll(touched);
      if (open[q] >= 0) {
        member(blocks[(size_t)open[q]], L, at);
      } else {
        emit(L, at);
        append(waiting[q], out.size() - 1);
      }
      continue;
    }
    if (fusable_type(*L) && width == 2) {
      const uint32_t lo = (uint32_t)__builtin_ctzll(touched), hi = 63u - (uint32_t)__builtin_clzll(touched);
      if (open[lo] >= 0 && open[lo] == open[hi]) {  // another gate on the same pair
        member(blocks[(size_t)open[lo]], L, at);
        continue;
      }
      close(lo);
      close(hi);
      blocks.emplace_back();
      Block& B = blocks.back();
      B.a = hi;
      B.b = lo;
      for (int i = 0; i < 16; ++i) B.m[i] = Cx{(i % 5) == 0 ? 1.0 : 0.0, 0.0};
      B.record = L->record;
      for (uint32_t q : {hi, lo}) {
        for (int i = waiting[q].head; i >= 0; i = links[(size_t)i].next) {
          const size_t o = links[(size_t)i].at;
          member(B, out[o], source[o]);
          out[o] = nullptr;
        }
        waiting[q] = List();
      }
      member(B, L, at);
      open[hi] = open[lo] = (int)blocks.size() - 1;
      continue;
    }
    for (uint64_t t = touched; t; t &= t - 1) {
      const uint32_t q = (uint32_t)__builtin_ctzll(t);
      close(q);
      waiting[q] = List();
    }
    emit(L, at);
  }
  for (uint32_t q = 0; q < kMaxQubits; ++q) close(q);
  out.erase(std::remove(out.begin(), out.end(), nullptr), out.end());
  return out;
}

// Shared-memory passes: after pair fusion, two dense one-qubit gates in a row
// become one op, their product on one qubit or their 4x4 on two (one barrier
// for two).
constexpr int kBarrierCost = 16;
std::vector<const Lowered*> fuse_for_smem(const std::vector<const Lowered*>& seg, std::deque<Lowered>& store) {
  const std::vector<const Lowered*> in = fuse_pairs(seg, store, kBarrierCost);
  auto plain_1q = [](const Lowered* L) { return L->op.type == OP_1Q && L->op.ctrl == 0; };
  std::vector<const Lowered*> out;
  out.reserve(in.size());
  for (const Lowered* L : in) {
    if (out.empty() || !plain_1q(L) || !plain_1q(out.back())) {
      out.push_back(L);
      continue;
    }
    const Lowered* W = out.back();
    const uint32_t a = W->op.q[0], b = L->op.q[0];
    store.emplace_back();
    Lowered& F = store.back();
    std::memset(&F.op, 0, sizeof(Op));
    F.record = W->record;
    F.gates = gates_of(*W) + gates_of(*L);
    F.given = W->given || L->given;
    F.diag = 0;
    F.nondiag = (1ull << a) | (1ull << b);
    if (a == b) {
      const Cx* u = reinterpret_cast<const Cx*>(W->coef.data());
      const Cx* v = reinterpret_cast<const Cx*>(L->coef.data());
      Cx m[4];
      for (int r = 0; r < 2; ++r)
        for (int c = 0; c < 2; ++c) m[2 * r + c] = add(mul(v[2 * r], u[c]), mul(v[2 * r + 1], u[2 + c]));
      F.op.type = OP_1Q;
      F.op.nq = 1;
      F.op.q[0] = (uint8_t)a;
      if (!F.given) unit_rows(m, 2, F.gates);
      push_coef(&F, m, 4);
    } else {
      Cx m[16];
      for (int i = 0; i < 16; ++i) m[i] = Cx{(i % 5) == 0 ? 1.0 : 0.0, 0.0};
      fold_into_4x4(*W, a, b, m);
      fold_into_4x4(*L, a, b, m);
      F.op.type = OP_2Q;
      F.op.nq = 2;
      F.op.q[0] = (uint8_t)a;
      F.op.q[1] = (uint8_t)b;
      if (!F.given) unit_rows(m, 4, F.gates);
      push_coef(&F, m, 16);
    }
    out.back() = &F;
  }
  return out;
}

int plan_segment_tiles(const std::vector<const Lowered*>& seg, uint32_t n, uint32_t R, Plan* P) {
  std::vector<const Lowered*> pending = seg;
  while (!pending.empty()) {
    const Lowered* head = pending.front();
    if (head->op.type == OP_KQ) {
      Pass ps{};
      ps.kind = PASS_KQ;
      ps.tile.n = n;
      ps.tile.op_begin = append_op(P, *head, head->op);
      ps.tile.op_count = 1;
      ps.record = head->record;
      ps.gates = 1;
      ps.dense_ops = 1;
      P->passes.push_back(ps);
      pending.erase(pending.begin());
      continue;
    }
    uint64_t hi = 0;          // register qubits chosen so far
    uint32_t nhi = 0;
    uint64_t blocked_full = 0, blocked_diag = 0;
    std::vector<const Lowered*> take, rest;
    for (const Lowered* L : pending) {
      bool ok = !(L->nondiag & (blocked_full | blocked_diag)) && !(L->diag & blocked_full);
      uint64_t need = 0;
      if (ok && L->op.type == OP_KQ) ok = false;
      if (ok && L->nondiag) {
        need = (L->nondiag >> 5 << 5) & ~hi;
        if (nhi + (uint32_t)__builtin_popcountll(need) > R) ok = false;
      }
      if (ok) {
        hi |= need;
        nhi += (uint32_t)__builtin_popcountll(need);
        take.push_back(L);
      } else {
        blocked_full |= L->nondiag;
        blocked_diag |= L->diag;
        rest.push_back(L);
      }
    }
    // register qubits: the chosen ones, padded with the lowest unused qubits >= 5
    TilePass tp{};
    tp.n = n;
    tp.R = R;
    uint32_t j = 0;
    for (uint32_t q = 5; q < n && j < R; ++q)
      if ((hi >> q) & 1) tp.hq[j++] = q;
    for (uint32_t q = 5; q < n && j < R; ++q)
      if (!((hi >> q) & 1)) {
        tp.hq[j++] = q;
        hi |= 1ull << q;
      }
    auto slot = [&](uint32_t q) -> uint8_t {
      if (q < 5) return (uint8_t)q;
      for (uint32_t i = 0; i < R; ++i)
        if (tp.hq[i] == q) return (uint8_t)(5 + i);
      return 255;
    };
    tp.op_begin = (uint32_t)P->ops.size();
    // Split a global qubit mask into the bits outside the register qubits and
    // an R-bit mask over the register slots (tested per element in the kernel).
    auto split = [&](uint64_t m, uint64_t* rest, uint8_t* creg) {
      *rest = m;
      *creg = 0;
      for (uint32_t j = 0; j < R; ++j)
        if ((m >> tp.hq[j]) & 1) {
          *creg |= (uint8_t)(1u << j);
          *rest &= ~(1ull << tp.hq[j]);
        }
    };
    for (const Lowered* L : take) {
      Op op = L->op;
      if (op.type == OP_NEG || op.type == OP_CPHASE) {
        split(op.mask, &op.mask, &op.creg);
        op.ctrl = 0;
      } else if (op.type != OP_POLY) {
        split(op.ctrl, &op.ctrl, &op.creg);
      }
      if (op.type == OP_DIAG) {
        op.dsrc = 0;
        for (int i = 0; i < op.nq; ++i) {
          const uint8_t s = slot(op.q[i]);
          if (s >= 5 && s != 255) {
            op.dsrc |= (uint8_t)(1u << i);
            op.q[3 + i] = (uint8_t)(s - 5);
          }
        }
      }
      if (op.type == OP_1Q || op.type == OP_X) {
        op.a = slot(op.q[0]);
        append_op(P, *L, op);
      } else if (op.type == OP_2Q) {
        uint8_t sa = slot(op.q[0]), sb = slot(op.q[1]);
        if (sa < sb) {
          Lowered tmp = *L;
          swap_2q_operands(tmp.coef);
          std::swap(op.q[0], op.q[1]);
          op.a = sb;
          op.b = sa;
          append_op(P, tmp, op);
        } else {
          op.a = sa;
          op.b = sb;
          append_op(P, *L, op);
        }
      } else {
        append_op(P, *L, op);
      }
    }
    tp.op_count = (uint32_t)P->ops.size() - tp.op_begin;
    if (take.empty()) return ALEPH_B200_OPTIMIZATION;  // no progress: the head op fits no tile
    Pass ps{};
    ps.kind = PASS_TILE;
    ps.tile = tp;
    ps.record = take.empty() ? 0 : take.front()->record;
    ps.gates = 0;
    for (const Lowered* L : take) ps.gates += gates_of(*L);
    count_ops(take, &ps);
    P->passes.push_back(ps);
    pending.swap(rest);
  }
  return ALEPH_B200_OK;
}

// ---- wide tile passes ------------------------------------------------------------
// The ops of `pending` that fit one pass (or one phase of it), in order: an op
// joins if it commutes past every op left behind and acts non-diagonally only on
// qubits of the set. The set is `have` plus up to `room` qubits taken first come.
struct WideTake {
  uint64_t set = 0;
  std::vector<const Lowered*> take, rest;
};

double wide_weight(const Lowered& L) {  // arithmetic, and a little for every op's own overhead
  return 2.0 + tile_cost(L);
}

// What the choice of a set needs of an op.
struct WideOp {
  uint64_t nondiag, diag;
  double score;  // arithmetic, older ops counting more (see BlockTake); 0 for diagonal ops
  bool joins;    // not a k-qubit unitary, which has a pass of its own
};

// The score and the set of one choice. `all`: the qubits of the ops; once every one
// of them is blocked no further op can score.
double wide_score(const std::vector<WideOp>& ops, uint64_t have, uint32_t room, uint64_t all, uint64_t* out) {
  uint64_t set = have, blocked_full = 0, blocked_diag = 0;
  double score = 0.0;
  for (const WideOp& o : ops) {
    const uint64_t need = o.nondiag & ~set;
    if (o.joins && !(o.nondiag & (blocked_full | blocked_diag)) && !(o.diag & blocked_full) &&
        (!need || (uint32_t)__builtin_popcountll(need) <= room)) {
      set |= need;
      room -= (uint32_t)__builtin_popcountll(need);
      score += o.score;
    } else {
      blocked_full |= o.nondiag;
      blocked_diag |= o.diag;
      if (blocked_full == all) break;
    }
  }
  *out = set;
  return score;
}

// The best of the first-come set and of every window of consecutive qubits
// (on a brickwall the windows follow the light cone).
WideTake wide_best(const std::vector<const Lowered*>& pending, uint64_t have, uint32_t room, const uint8_t* qubits,
                   uint32_t nq, std::vector<WideOp>& ops) {
  const uint32_t base = pending.front()->record;
  uint64_t all = 0;
  ops.clear();
  for (const Lowered* L : pending) {
    const double age = L->record > base ? (double)(L->record - base) : 0.0;
    ops.push_back(WideOp{L->nondiag, L->diag, L->nondiag ? wide_weight(*L) / (1.0 + age / 256.0) : 0.0,
                         L->op.type != OP_KQ});
    all |= L->nondiag | L->diag;
  }
  uint64_t set = 0;
  double best = wide_score(ops, have, room, all, &set);
  for (uint32_t a = 0; a + room <= nq; ++a) {
    uint64_t window = have, s;
    for (uint32_t k = 0; k < room; ++k) window |= 1ull << qubits[a + k];
    const double score = wide_score(ops, window, 0, all, &s);
    if (score > best) {
      best = score;
      set = s;
    }
  }
  WideTake T;
  T.set = set;
  uint64_t blocked_full = 0, blocked_diag = 0;
  for (const Lowered* L : pending) {
    if (L->op.type != OP_KQ && !(L->nondiag & (blocked_full | blocked_diag)) && !(L->diag & blocked_full) &&
        !(L->nondiag & ~set)) {
      T.take.push_back(L);
    } else {
      blocked_full |= L->nondiag;
      blocked_diag |= L->diag;
      T.rest.push_back(L);
    }
  }
  return T;
}

// Appends the ops of one phase, `reg_of[q]` the register bit of qubit q (255:
// none). Sign flips and corner phases with at most one register qubit are
// collected into groups: such an op joins the last group if it commutes with the
// dense ops after it. A group costs one sweep over the registers per class however
// many ops it holds (the QFT's passes hold some 20 phases per dense gate; one at
// a time, each cost half a sweep and its predicates).
void emit_wide_phase(const std::vector<const Lowered*>& ops, const uint8_t* reg_of, uint32_t n, bool f64, Plan* P) {
  struct Group {
    std::vector<const Lowered*> signs, phases[6];
    bool empty() const {
      for (const auto& c : phases)
        if (!c.empty()) return false;
      return signs.empty();
    }
  };
  struct Item {
    const Lowered* op = nullptr;  // null: group `group`
    size_t group = 0;
  };
  std::vector<Group> groups;
  std::vector<Item> items;
  uint64_t after = 0;  // qubits acted on non-diagonally after the last group
  uint64_t in_regs = 0;
  for (uint32_t q = 0; q < n; ++q)
    if (reg_of[q] != 255) in_regs |= 1ull << q;
  auto split = [&](uint64_t m, uint64_t* rest, uint32_t* regs) {
    *rest = m & ~in_regs;
    *regs = 0;
    for (uint64_t t = m & in_regs; t; t &= t - 1) *regs |= 1u << reg_of[__builtin_ctzll(t)];
  };
  for (const Lowered* L : ops) {
    uint64_t rest = 0;
    uint32_t regs = 0;
    if (L->op.type == OP_NEG || L->op.type == OP_CPHASE) split(L->op.mask, &rest, &regs);
    const bool sign = L->op.type == OP_NEG;
    const bool phase = L->op.type == OP_CPHASE && __builtin_popcount(regs) <= 1;
    if (!sign && !phase) {
      items.push_back(Item{L, 0});
      if (L->nondiag) after |= L->nondiag;
      continue;
    }
    if (groups.empty() || (L->diag & after)) {
      groups.emplace_back();
      items.push_back(Item{nullptr, groups.size() - 1});
      after = 0;
    }
    Group& G = groups.back();
    if (sign) G.signs.push_back(L);
    else G.phases[regs ? (uint32_t)__builtin_ctz(regs) : 5u].push_back(L);
  }
  auto group_op = [&](uint8_t type, uint8_t cls, size_t count) {
    Op op;
    std::memset(&op, 0, sizeof(Op));
    op.type = type;
    op.a = cls;
    op.aux = (uint32_t)count;
    op.coef = (uint32_t)(P->coef.size() / 2);
    P->ops.push_back(op);
  };
  for (const Item& it : items) {
    if (!it.op) {
      const Group& G = groups[it.group];
      if (!G.signs.empty()) {
        group_op(OP_SIGNS, 0, G.signs.size());
        for (const Lowered* L : G.signs) {
          Op op = L->op;
          uint32_t regs = 0, flips = 0;
          split(L->op.mask, &op.mask, &regs);
          for (uint32_t r = 0; r < 32; ++r)
            if ((r & regs) == regs) flips |= 1u << r;
          append_op(P, *L, op);
          P->ops.back().aux = flips;
        }
      }
      for (uint32_t c = 0; c < 6; ++c) {
        if (G.phases[c].empty()) continue;
        group_op(OP_PHASES, (uint8_t)c, G.phases[c].size());
        for (const Lowered* L : G.phases[c]) {
          Op op = L->op;
          uint32_t regs = 0;
          split(L->op.mask, &op.mask, &regs);
          append_op(P, *L, op);
        }
      }
      continue;
    }
    const Lowered* L = it.op;
    Op op = L->op;
    uint32_t regs = 0;
    if (op.type == OP_CPHASE) {
      split(op.mask, &op.mask, &regs);
      op.creg = (uint8_t)regs;
      op.ctrl = 0;
    } else if (op.type != OP_POLY) {
      split(op.ctrl, &op.ctrl, &regs);
      op.creg = (uint8_t)regs;
    }
    if (op.type == OP_DIAG) {
      op.dsrc = 0;
      for (int i = 0; i < op.nq; ++i)
        if (reg_of[op.q[i]] != 255) {
          op.dsrc |= (uint8_t)(1u << i);
          op.q[3 + i] = reg_of[op.q[i]];
        }
    }
    if (op.type == OP_X) op.a = (uint8_t)(5 + reg_of[op.q[0]]);
    if (op.type == OP_1Q || op.type == OP_2Q) {
      Lowered M = *L;
      op.a = (uint8_t)(5 + reg_of[op.q[0]]);
      if (op.type == OP_2Q) {
        op.b = (uint8_t)(5 + reg_of[op.q[1]]);
        if (op.a < op.b) {
          swap_2q_operands(M.coef);
          std::swap(op.q[0], op.q[1]);
          std::swap(op.a, op.b);
        }
      }
      if (L->op.ctrl == 0) {
        const bool real = real_matrix(M);
        op.dsrc = real ? WIDE_REAL : f64 ? 0 : WIDE_PAIRED;
        if (!f64) {  // duplicated for paired arithmetic
          std::vector<double> dup;
          for (size_t c = 0; c < M.coef.size(); c += 2) {
            dup.insert(dup.end(), 2, M.coef[c]);
            if (!real) dup.insert(dup.end(), 2, M.coef[c + 1]);
          }
          M.coef = std::move(dup);
        }
      }
      append_op(P, M, op);
      continue;
    }
    append_op(P, *L, op);
  }
}

// R: register qubits of a phase, 4 or 5.
int plan_segment_wide(const std::vector<const Lowered*>& seg, uint32_t n, bool f64, uint32_t tile_r, uint32_t R, Plan* P) {
  std::vector<const Lowered*> pending = seg;
  std::vector<WideOp> scored;  // wide_best's, kept between its calls
  uint8_t all[kMaxQubits];
  for (uint32_t q = 0; q < n; ++q) all[q] = (uint8_t)q;
  while (!pending.empty()) {
    if (pending.front()->op.type == OP_KQ) {
      const std::vector<const Lowered*> one{pending.front()};
      if (int s = plan_segment_tiles(one, n, tile_r, P)) return s;
      pending.erase(pending.begin());
      continue;
    }
    WideTake T = wide_best(pending, 0xFull, kWideBits - 4, all + 4, n - 4, scored);
    if (T.take.empty()) return ALEPH_B200_OPTIMIZATION;
    // the tile: the chosen qubits, padded with the lowest unused ones
    uint64_t set = T.set;
    for (uint32_t q = 4; q < n && __builtin_popcountll(set) < (int)kWideBits; ++q) set |= 1ull << q;
    Pass ps{};
    ps.kind = PASS_WIDE;
    WidePass& W = ps.wide;
    W.n = n;
    W.R = R;
    uint8_t tile[kWideBits];
    uint32_t k = 0;
    for (uint32_t q = 0; q < n; ++q) {
      if ((set >> q) & 1) {
        if (k >= 4) W.free_q[k - 4] = q;
        tile[k++] = (uint8_t)q;
      }
    }
    for (uint32_t q = 0, src = 0; q < n;) {
      if ((set >> q) & 1) {
        ++q;
        continue;
      }
      uint32_t len = 0;
      while (q + len < n && !((set >> (q + len)) & 1)) ++len;
      W.dep_src[W.n_dep] = src;
      W.dep_mask[W.n_dep] = (1u << len) - 1;  // len <= 28
      W.dep_dst[W.n_dep] = q;
      ++W.n_dep;
      src += len;
      q += len;
    }
    // phases: sets of R tile qubits, until the pass's ops are spent
    W.phase_begin = (uint32_t)P->phases.size();
    W.op_begin = (uint32_t)P->ops.size();
    std::vector<const Lowered*> left = T.take;
    auto add_phase = [&](uint32_t regs, bool io, const std::vector<const Lowered*>& ops) {
      WidePhase ph{};
      wide_layout(tile, W.R, regs, io, f64, &ph);
      uint8_t reg_of[kMaxQubits];
      std::memset(reg_of, 255, sizeof(reg_of));
      for (uint32_t j = 0; j < W.R; ++j) reg_of[ph.rq[j]] = (uint8_t)j;
      ph.op_begin = (uint32_t)P->ops.size();
      emit_wide_phase(ops, reg_of, n, f64, P);
      ph.op_count = (uint32_t)P->ops.size() - ph.op_begin;
      P->phases.push_back(ph);
    };
    const uint32_t kIoRegs = ((1u << W.R) - 1) << (kWideBits - W.R);  // the top tile bits: lanes take bits 0..4
    bool first = true;
    while (!left.empty()) {
      WideTake F = wide_best(left, 0, W.R, tile, kWideBits, scored);
      if (F.take.empty()) return ALEPH_B200_OPTIMIZATION;
      uint32_t regs = 0;
      for (uint32_t b = 0; b < kWideBits; ++b)
        if ((F.set >> tile[b]) & 1) regs |= 1u << b;
      for (int b = (int)kWideBits - 1; b >= 0 && __builtin_popcount(regs) < (int)W.R; --b) regs |= 1u << b;
      const bool low = (regs & 0xFu) != 0, last = F.rest.empty();
      if (first && low) add_phase(kIoRegs, true, {});
      add_phase(regs, !low && (first || last), F.take);
      if (last && low) add_phase(kIoRegs, true, {});
      first = false;
      left.swap(F.rest);
    }
    W.phase_count = (uint32_t)P->phases.size() - W.phase_begin;
    W.op_count = (uint32_t)P->ops.size() - W.op_begin;
    W.full = 0;
    for (uint32_t i = W.op_begin; i < W.op_begin + W.op_count; ++i) {
      const Op& op = P->ops[i];
      if (op.type == OP_SIGNS) {  // its records follow
        i += op.aux;
        continue;
      }
      const bool dense = op.type == OP_1Q || op.type == OP_2Q;
      if (dense ? op.dsrc == WIDE_REAL : op.type != OP_X) W.full = 1;
    }
    ps.record = T.take.front()->record;
    for (const Lowered* L : T.take) ps.gates += gates_of(*L);
    count_ops(T.take, &ps);
    P->passes.push_back(ps);
    pending.swap(T.rest);
  }
  return ALEPH_B200_OK;
}

// ---- warp or wide tiles for a short list ----------------------------------------------
// A list of a few gates often fits one pass of either kind, and then a wide tile
// has nothing to save: it pays an exchange for every further set of register
// qubits (two for one gate on a low qubit), a warp tile pays shuffles on the lane
// qubits only. Both are planned and the cheaper one by this table is taken.
// The table: milliseconds per 2^27 amplitudes, least squares over 1700 measured
// passes (single families of 1 to 40 gates, n = 16..27; 5 to 10% rms). Up to
// n = 21 a pass is one wave or less and its latency counts, above that its
// throughput. Measured with the choice against wide tiles alone: FP64 n = 24, one H
// on qubit 0 161 -> 118 us, 4 U3 163 -> 121 us; n = 27, 4 H 1.13 -> 0.85 ms; FP32
// n = 24, 4 controlled rotations and Toffolis 0.78 of the time.
// Gates: in FP32 longer lists save passes with wide tiles; in FP64 lists of one-qubit gates
// alone may not (n = 27, 120 U3: 0.93 of the speed), and beyond its limit planning
// twice costs more than the choice gives.
constexpr size_t kShortList[2] = {64, 512};
constexpr double kWideLead = 1.06;  // wide tiles are taken where the table has them ahead by its error
struct TileCosts {
  double pass, x, x_lane, one, one_real, one_lane, two, two_real, two_lane, two_lanes, controlled, sign, phase, group,
      member, table, exchange;
};
double tiles_ms(const Plan& P, size_t pass0, bool f64, uint32_t n) {
  static const TileCosts costs[2][2][2] = {
      // FP32: n < 22 (warp, wide), n >= 22
      {{{1.05, .060, .100, .115, .115, .135, .335, .335, .380, .470, .070, .040, .200, .0, .0, .400, .0},
        {1.05, .050, .0, .086, .071, .0, .152, .100, .0, .0, .055, .040, .200, .250, .05, .390, .140}},
       {{.310, .026, .044, .047, .047, .068, .140, .140, .190, .200, .010, .020, .080, .0, .0, .212, .0},
        {.285, .026, .0, .034, .023, .0, .098, .050, .0, .0, .027, .020, .080, .095, .015, .196, .076}}},
      // FP64
      {{{1.30, .070, .110, .130, .130, .170, .290, .290, .460, .780, .150, .050, .265, .0, .0, .400, .0},
        {1.30, .068, .0, .146, .086, .0, .218, .120, .0, .0, .030, .050, .265, .280, .05, .405, .150}},
       {{.600, .044, .071, .070, .070, .150, .140, .140, .320, .530, .030, .030, .115, .0, .0, .310, .0},
        {.600, .044, .0, .088, .073, .0, .155, .090, .0, .0, .017, .030, .115, .190, .02, .312, .136}}}};
  double ms = 0.0;
  // a wide pass's launch takes the host some 2 us longer
  if (pass0 < P.passes.size() && P.passes[pass0].kind == PASS_WIDE) ms += .002 * (double)(1u << (27 - std::min(27u, std::max(n, 20u))));
  for (size_t k = pass0; k < P.passes.size(); ++k) {
    const Pass& ps = P.passes[k];
    if (ps.kind != PASS_TILE && ps.kind != PASS_WIDE) continue;  // k-qubit unitaries: the same in both
    const bool wide = ps.kind == PASS_WIDE;
    const TileCosts& c = costs[f64][n >= 22][wide];
    ms += c.pass + (wide ? (ps.wide.phase_count - 1) * c.exchange : 0.0);
    const uint32_t begin = wide ? ps.wide.op_begin : ps.tile.op_begin, count = wide ? ps.wide.op_count : ps.tile.op_count;
    for (uint32_t i = begin; i < begin + count; ++i) {
      const Op& op = P.ops[i];
      const int lanes = wide ? 0 : (op.a < 5) + (op.type == OP_2Q && op.b < 5);
      const bool real = wide && op.dsrc == WIDE_REAL;
      switch (op.type) {
        case OP_X: ms += lanes ? c.x_lane : c.x; break;
        case OP_1Q: ms += (lanes ? c.one_lane : real ? c.one_real : c.one) + (op.ctrl || op.creg ? c.controlled : 0.0); break;
        case OP_2Q: ms += lanes == 2 ? c.two_lanes : lanes ? c.two_lane : real ? c.two_real : c.two; break;
        case OP_NEG: ms += c.sign; break;
        case OP_SIGNS:
          ms += c.sign;
          i += op.aux;
          break;
        case OP_CPHASE: ms += c.phase; break;
        case OP_PHASES:
          ms += c.group + op.aux * c.member;
          i += op.aux;
          break;
        default: ms += c.table; break;
      }
    }
  }
  return ms;
}

// ---- tensor-core dense blocks ------------------------------------------------
// Apply a lowered op to a vector over the block qubits bq[0..6) (index bit b
// <-> qubit bq[b]); the op's qubits must all be block qubits, except for the
// diagonal-polynomial case where only the support matters.
void apply_local(const Lowered& L, const uint32_t* bq, Cx* s) {
  auto lbit = [&](uint32_t q) -> uint32_t {
    for (uint32_t b = 0; b < 6; ++b)
      if (bq[b] == q) return b;
    return 63;
  };
  auto lmask = [&](uint64_t m) -> uint32_t {
    uint32_t r = 0;
    for (; m; m &= m - 1) r |= 1u << lbit((uint32_t)__builtin_ctzll(m));
    return r;
  };
  auto gidx = [&](uint32_t x) -> uint64_t {
    uint64_t g = 0;
    for (uint32_t b = 0; b < 6; ++b)
      if ((x >> b) & 1) g |= 1ull << bq[b];
    return g;
  };
  const Op& op = L.op;
  const Cx* c = reinterpret_cast<const Cx*>(L.coef.data());
  switch (op.type) {
    case OP_NEG:
    case OP_CPHASE: {
      const uint32_t m = lmask(op.mask);
      const Cx f = op.type == OP_NEG ? Cx{-1, 0} : c[0];
      for (uint32_t x = 0; x < 64; ++x)
        if ((x & m) == m) s[x] = mul(f, s[x]);
      return;
    }
    case OP_DIAG: {
      const uint32_t cm = lmask(op.ctrl);
      for (uint32_t x = 0; x < 64; ++x) {
        if ((x & cm) != cm) continue;
        uint32_t idx = 0;
        for (int i = 0; i < op.nq; ++i) idx = (idx << 1) | ((x >> lbit(op.q[i])) & 1);
        s[x] = mul(c[idx], s[x]);
      }
      return;
    }
    case OP_POLY: {
      for (uint32_t x = 0; x < 64; ++x) {
        const uint64_t g = gidx(x);
        double phi = 0.0;
        size_t off = 0;
        for (size_t t = 0; t < L.poly_angle.size(); ++t) {
          bool all = true;
          for (uint32_t k = 0; k < L.poly_cnt[t]; ++k)
            if ((__builtin_popcountll(L.poly_conds[off + k] & g) & 1) == 0) all = false;
          off += L.poly_cnt[t];
          if (all) phi += L.poly_angle[t];
        }
        s[x] = mul(Cx{std::cos(phi), std::sin(phi)}, s[x]);
      }
      return;
    }
    default: break;
  }
  // dense: k targets MSB-first, controls
  const int k = op.type == OP_2Q ? 2 : op.type == OP_KQ ? op.nq : 1;
  const uint32_t dim = 1u << k;
  const uint32_t cm = lmask(op.ctrl);
  uint32_t tmask = 0, off[32];
  for (int i = 0; i < k; ++i) tmask |= 1u << lbit(op.q[i]);
  for (uint32_t r = 0; r < dim; ++r) {
    uint32_t o = 0;
    for (int p = 0; p < k; ++p)
      if ((r >> p) & 1) o |= 1u << lbit(op.q[k - 1 - p]);
    off[r] = o;
  }
  for (uint32_t base = 0; base < 64; ++base) {
    if ((base & tmask) || (base & cm) != cm) continue;
    Cx v[32], w[32];
    for (uint32_t r = 0; r < dim; ++r) v[r] = s[base | off[r]];
    for (uint32_t r = 0; r < dim; ++r) {
      if (op.type == OP_X) {
        w[r] = v[r ^ 1];
        continue;
      }
      Cx acc{0, 0};
      for (uint32_t cc = 0; cc < dim; ++cc) acc = add(acc, mul(c[r * dim + cc], v[cc]));
      w[r] = acc;
    }
    for (uint32_t r = 0; r < dim; ++r) s[base | off[r]] = w[r];
  }
}

// One block pass drawn from the pending ops: the ops fused into the block
// (`take`), the diagonal ops applied after it in the epilogue (`post`) and the
// ops left for later passes (`rest`, in order). With `fixed`, the block
// qubits are `fixedB`; otherwise they grow first-come up to 6 qubits. An op
// joins only if it commutes past every op deferred before it.
struct BlockTake {
  uint64_t B = 0;
  std::vector<const Lowered*> take, post, rest;
  // Ops consumed, each weighted by its age: 1 / (1 + (record - base) / 64),
  // base = the oldest pending record. Preferring old ops keeps the frontier
  // level; on the n=32 depth-40 brickwall it plans 67 passes where a plain
  // count plans 70 (a planner model swept the scale: 64-128 best).
  double score(uint32_t base) const {
    if (take.empty()) return 0.0;
    double s = 0.0;
    auto weight = [&](const Lowered* L) { return 1.0 / (1.0 + (L->record > base ? (double)(L->record - base) : 0.0) / 64.0); };
    for (const Lowered* L : take) s += weight(L);
    for (const Lowered* L : post) s += weight(L);
    return s;
  }
};

void block_take(const std::vector<const Lowered*>& pending, uint64_t fixedB, bool fixed, BlockTake* out) {
  uint64_t B = fixed ? fixedB : 0, bf = 0, bd = 0, post_lock = 0;
  auto fits = [&](uint64_t supp) {
    return fixed ? (supp & ~fixedB) == 0 : __builtin_popcountll(B | supp) <= 6;
  };
  for (const Lowered* L : pending) {
    const uint64_t supp = L->nondiag | L->diag;
    if (L->nondiag) {
      if (!(L->nondiag & (bf | bd | post_lock)) && !(L->diag & bf) && fits(supp)) {
        B |= supp;
        out->take.push_back(L);
        continue;
      }
    } else if (!(L->diag & bf)) {
      if (fits(supp)) {
        B |= supp;
        out->take.push_back(L);
        continue;
      }
      if (B != 0 && out->post.size() < 48) {  // the block kernel caches up to 48 post ops
        out->post.push_back(L);
        post_lock |= supp;
        continue;
      }
    }
    bf |= L->nondiag;
    bd |= L->diag;
    out->rest.push_back(L);
  }
  out->B = B;
}

// One block pass's fused unitary, still to be built: its ops, its qubits and
// the byte offset of its image in the plan.
struct BlockJob {
  std::vector<const Lowered*> take;
  uint32_t bq[6];
  uint32_t mat;
};

// Fuse each job's ops into a 64x64 unitary (columns = images of the basis
// vectors, in FP64), lay it out as W = [[Re U, -Im U], [Im U, Re U]] and write
// the split-BF16 image. The jobs are independent: they run on host threads.
void build_block_images(const std::vector<BlockJob>& jobs, Plan* P) {
  if (jobs.empty()) return;
  P->block_images.resize(P->block_images.size() + jobs.size() * kBlockImageBytes);
  auto build = [&](size_t k) {
    const BlockJob& J = jobs[k];
    std::vector<Cx> U(64 * 64);
    for (uint32_t col = 0; col < 64; ++col) {
      Cx s[64];
      for (uint32_t x = 0; x < 64; ++x) s[x] = Cx{x == col ? 1.0 : 0.0, 0.0};
      for (const Lowered* L : J.take) apply_local(*L, J.bq, s);
      for (uint32_t x = 0; x < 64; ++x) U[x * 64 + col] = s[x];
    }
    std::vector<double> W(128 * 128);
    for (uint32_t r = 0; r < 64; ++r)
      for (uint32_t c = 0; c < 64; ++c) {
        const Cx u = U[r * 64 + c];
        W[r * 128 + c] = u.re;
        W[r * 128 + 64 + c] = -u.im;
        W[(64 + r) * 128 + c] = u.im;
        W[(64 + r) * 128 + 64 + c] = u.re;
      }
    build_block_image(W.data(), P->block_images.data() + J.mat);
  };
  const unsigned hw = std::thread::hardware_concurrency();
  const size_t nt = std::min<size_t>(jobs.size(), hw ? std::min(hw, 16u) : 1u);
  if (nt <= 1) {
    for (size_t k = 0; k < jobs.size(); ++k) build(k);
    return;
  }
  std::vector<std::thread> ws;
  for (size_t t = 0; t < nt; ++t)
    ws.emplace_back([&, t] {
      for (size_t k = t; k < jobs.size(); k += nt) build(k);
    });
  for (auto& w : ws) w.join();
}

int plan_segment_blocks(const std::vector<const Lowered*>& seg, uint32_t n, uint32_t R, bool window_search,
                        Plan* P) {
  std::vector<const Lowered*> pending = seg;
  std::vector<BlockJob> jobs;
  while (!pending.empty()) {
    // Candidates: the first-come block, and (window_search) every window of 6
    // consecutive qubits; the one with the highest age-weighted op count wins
    // (ties keep the earlier candidate). On a brickwall the windows follow
    // the light cone, which first-come growth does not.
    const uint32_t base = pending.front()->record;
    BlockTake best;
    block_take(pending, 0, false, &best);
    double best_score = best.score(base);
    if (window_search)
      for (uint32_t a = 0; a + 6 <= n; ++a) {
        BlockTake c;
        block_take(pending, 0x3Full << a, true, &c);
        const double s = c.score(base);
        if (s > best_score) {
          best = std::move(c);
          best_score = s;
        }
      }
    uint64_t B = best.B;
    std::vector<const Lowered*>& take = best.take;
    std::vector<const Lowered*>& post = best.post;
    std::vector<const Lowered*>& rest = best.rest;
    if (take.empty()) {
      // the head op does not fit a 6-qubit block: run it on the CUDA cores
      std::vector<const Lowered*> one{pending.front()};
      if (int s = plan_segment_tiles(one, n, R, P)) return s;
      pending.erase(pending.begin());
      continue;
    }
    // pad the block to 6 qubits with the lowest unused qubits
    for (uint32_t q = 0; q < n && __builtin_popcountll(B) < 6; ++q) B |= 1ull << q;
    uint32_t bq[6], nb = 0;
    for (uint32_t q = 0; q < n; ++q)
      if ((B >> q) & 1) bq[nb++] = q;
    Pass ps{};
    ps.kind = PASS_BLOCK;
    ps.block.n = n;
    for (int j = 0; j < 6; ++j) ps.block.bq[j] = bq[j];
    ps.block.mat = (uint32_t)(P->block_images.size() + jobs.size() * kBlockImageBytes);
    jobs.push_back(BlockJob{take, {bq[0], bq[1], bq[2], bq[3], bq[4], bq[5]}, ps.block.mat});
    ps.block.post_begin = (uint32_t)P->ops.size();
    for (const Lowered* L : post) append_op(P, *L, L->op);
    ps.block.post_count = (uint32_t)P->ops.size() - ps.block.post_begin;
    ps.block.fold = 0;
    for (const Lowered* L : post) {
      const Op& op = L->op;
      if ((op.type == OP_CPHASE && __builtin_popcountll(op.mask & B) <= 1) ||
          (op.type == OP_DIAG && op.nq == 1 && !((B >> op.q[0]) & 1) && !(op.ctrl & B)))
        ps.block.fold = 1;
    }
    ps.record = take.front()->record;
    for (const Lowered* L : take) ps.gates += gates_of(*L);
    for (const Lowered* L : post) ps.gates += gates_of(*L);
    count_ops(take, &ps);
    ps.lane_ops = 0;  // a block has no lane shuffles
    ps.diag_ops += (uint32_t)post.size();
    P->passes.push_back(ps);
    pending.swap(rest);
  }
  build_block_images(jobs, P);
  return ALEPH_B200_OK;
}

}  // namespace

// A cycle c_0 -> c_1 -> ... -> c_{m-1} -> c_0 of pi is alpha o beta with the
// reflections beta(c_i) = c_{-i} and alpha(c_i) = c_{1-i} (indices mod m), both
// involutions; alpha is applied first (P_beta P_alpha psi = psi o alpha o beta).
std::vector<std::vector<uint8_t>> split_into_involutions(const std::vector<uint32_t>& pi) {
  const uint32_t n = (uint32_t)pi.size();
  std::vector<uint8_t> alpha(n), beta(n);
  std::vector<bool> seen(n, false);
  bool alpha_id = true, beta_id = true;
  for (uint32_t s = 0; s < n; ++s) {
    if (seen[s]) continue;
    std::vector<uint32_t> cyc;
    for (uint32_t q = s; !seen[q]; q = pi[q]) {
      seen[q] = true;
      cyc.push_back(q);
    }
    const uint32_t m = (uint32_t)cyc.size();
    for (uint32_t i = 0; i < m; ++i) {
      beta[cyc[i]] = (uint8_t)cyc[(m - i) % m];
      alpha[cyc[i]] = (uint8_t)cyc[(m + 1 - i) % m];
      beta_id &= beta[cyc[i]] == cyc[i];
      alpha_id &= alpha[cyc[i]] == cyc[i];
    }
  }
  std::vector<std::vector<uint8_t>> out;
  if (!alpha_id) out.push_back(alpha);
  if (!beta_id) out.push_back(beta);
  return out;
}

int build_plan(const std::vector<Lowered>& ops, uint32_t n, bool f64, const PlanOptions& o, Plan* P) {
  P->renormalize = o.renormalize;
  std::vector<const Lowered*> seg;
  int status = ALEPH_B200_OK;
  auto flush = [&]() {
    if (seg.empty() || status) return;
    if (n <= o.smem_max_n || n < 6) {
      Pass ps{};
      ps.kind = PASS_SMEM;
      ps.tile.n = n;
      ps.tile.op_begin = (uint32_t)P->ops.size();
      std::deque<Lowered> fused;
      const std::vector<const Lowered*> list = o.pair_fusion && seg.size() > 1 ? fuse_for_smem(diagonal_cores(seg, fused, true), fused) : seg;
      for (const Lowered* L : list) {
        Op op = L->op;
        if ((op.type == OP_1Q || op.type == OP_2Q) && real_matrix(*L)) op.dsrc = WIDE_REAL;
        ps.has_poly = ps.has_poly || op.type == OP_POLY;
        append_op(P, *L, op);
      }
      ps.tile.op_count = (uint32_t)P->ops.size() - ps.tile.op_begin;
      ps.record = seg.front()->record;
      ps.gates = (uint32_t)seg.size();
      count_ops(list, &ps);
      P->passes.push_back(ps);
    } else {
      // a 2-qubit gate may need two register qubits: R >= 2 unless only one high qubit exists
      const uint32_t R = std::min<uint32_t>(std::max<uint32_t>(o.tile_r, 2), std::min<uint32_t>(5, n - 5));
      if (o.tensor_blocks && !f64 && n >= 13) {  // blocks act on FP32 states
        // diagonal cores follow a block as its post ops instead of ending it
        std::deque<Lowered> fused;
        status = plan_segment_blocks(o.pair_fusion ? diagonal_cores(seg, fused) : seg, n, R, o.block_window_search, P);
      } else if (o.pair_fusion) {
        std::deque<Lowered> fused;
        // Wide tiles in the default configuration (five register qubits), and with four
        // for tile_r = 4, which the learned planner may choose: FP64 measured at n = 25
        // and 26, QFT passes 1.0 to 1.2 times faster, brickwall 1.35 times slower, FP32
        // 1.2 times slower; other values of the warp-tile keys (and pair_fusion or
        // relabel_swaps off) compare the parts of the warp-tile planner, and a state
        // smaller than one wide tile has no choice.
        const bool wide = n >= kWideBits && o.relabel_swaps && ((o.tile_r == 5 && o.tile_occupancy == 0) || o.tile_r == 4);
        auto plan_wide = [&](Plan* to) {
          return plan_segment_wide(fuse_pairs(cancel_phases(diagonal_cores(seg, fused), fused), fused), n, f64, R,
                                   o.tile_r == 4 ? 4 : 5, to);
        };
        auto plan_warp = [&](Plan* to) { return plan_segment_tiles(fuse_pairs(seg, fused), n, R, to); };
        if (wide && o.tile_r == 5 && seg.size() == 1 && seg[0]->op.type != OP_2Q) {
          status = plan_warp(P);  // the table's answer, without the second plan
        } else if (wide && o.tile_r == 5 && seg.size() <= kShortList[f64]) {
          Plan W, T;
          W.renormalize = T.renormalize = P->renormalize;
          status = plan_wide(&W);
          if (!status) status = plan_warp(&T);
          if (!status) {
            const bool warp = tiles_ms(T, 0, f64, n) <= kWideLead * tiles_ms(W, 0, f64, n);
            if (P->passes.empty()) *P = std::move(warp ? T : W);
            else status = warp ? plan_warp(P) : plan_wide(P);
          }
        } else {
          status = wide ? plan_wide(P) : plan_warp(P);
        }
      } else {
        status = plan_segment_tiles(seg, n, R, P);
      }
    }
    seg.clear();
  };
  for (const Lowered& L : ops) {
    if (L.is_measure) {
      flush();
      Pass ps{};
      ps.kind = PASS_MEASURE;
      ps.qubit = L.measure_qubit;
      ps.record = L.record;
      P->passes.push_back(ps);
      ++P->n_measures;
    } else if (L.is_permute) {
      flush();
      Pass ps{};
      ps.kind = PASS_PERMUTE;
      for (uint32_t q = 0; q < n && q < kMaxQubits; ++q) ps.sigma[q] = L.sigma[q];
      ps.record = L.record;
      ps.gates = L.gates;
      P->passes.push_back(ps);
    } else {
      seg.push_back(&L);
    }
  }
  flush();
  for (Pass& ps : P->passes)
    if (ps.kind == PASS_TILE) ps.tile.occupancy = o.tile_occupancy;
  return status;
}

}  // namespace ab
