// kernels_tile.cu — the warp-tile gate pass of the B200 state-vector engine.
//
// One warp owns a tile of 2^(5+R) amplitudes: the lane index supplies qubits
// 0..4, so every load/store instruction of a warp moves 32 consecutive
// amplitudes (512 B in FP64, 256 B in FP32, fully coalesced 16-/8-byte
// accesses), and each thread keeps 2^R amplitudes in registers spanning the R
// "register" qubits hq[0..R) of the pass. An ordered op list is applied in
// registers: gates on register qubits are register arithmetic, gates on
// qubits 0..4 use warp shuffles, diagonal ops (CZ, phases, DiagonalPhase) act
// on any qubit, and controls may sit on any qubit. One HBM read and one write
// per pass, however many gates it applies.
//
// Per-element predicates (controls, CZ masks, diagonal table indices) are
// split by the planner into a thread-constant part (bits of the lane and of
// the tile base) and a register part (an R-bit mask tested against the
// compile-time register index), so the inner loops do 32-bit tests only.
//
// Semantics follow the reference kernels: pair/quartet butterflies
// (crates/aleph-sv/src/kernels/aos.rs:192-223, :1335-1394), MSB-first operand
// order (crates/aleph-sv/src/kernels/unitary_kq.rs:66-96), controls as an AND
// mask over the basis index (aos.rs:198-205).

#include "tile_ops.cuh"

namespace ab {

// ---- lane-qubit ops (qubits 0..4, warp shuffles) ----------------------------
template <typename Real, int R>
__device__ __forceinline__ void lane_1q(V2<Real> (&v)[1 << R], int s, const V2<Real>* m, bool thr, uint32_t creg) {
  const int lane = threadIdx.x & 31;
  const bool hi = (lane >> s) & 1;
  const V2<Real> cs = ld_coef<Real>(m + (hi ? 3 : 0));  // coefficient on own amplitude
  const V2<Real> co = ld_coef<Real>(m + (hi ? 2 : 1));  // coefficient on partner amplitude
  if (thr && creg == 0) {  // no register-part controls
#pragma unroll
    for (int r = 0; r < (1 << R); ++r) {
      const V2<Real> o = shfl_xor<Real>(v[r], 1 << s);
      v[r] = cmul2<Real>(cs, v[r], co, o);
    }
    return;
  }
#pragma unroll
  for (int r = 0; r < (1 << R); ++r) {
    const V2<Real> o = shfl_xor<Real>(v[r], 1 << s);
    const V2<Real> nv = cmul2<Real>(cs, v[r], co, o);
    if (AB_ON(r)) v[r] = nv;
  }
}

template <typename Real, int R>
__device__ __forceinline__ void lane_x(V2<Real> (&v)[1 << R], int s, bool thr, uint32_t creg) {
#pragma unroll
  for (int r = 0; r < (1 << R); ++r) {
    const V2<Real> o = shfl_xor<Real>(v[r], 1 << s);
    if (AB_ON(r)) v[r] = o;
  }
}

// 4x4 with matrix MSB on register bit JA and LSB on lane bit s.
template <typename Real, int R, int JA>
__device__ __forceinline__ void regl_2q(V2<Real> (&v)[1 << R], int s, const V2<Real>* m, bool thr, uint32_t creg) {
  const int lane = threadIdx.x & 31;
  const int l = (lane >> s) & 1;
  V2<Real> r0[4], r1[4];  // own rows: k = l and k = 2 + l
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    r0[c] = ld_coef<Real>(m + 4 * l + c);
    r1[c] = ld_coef<Real>(m + 4 * (2 + l) + c);
  }
#pragma unroll
  for (int r = 0; r < (1 << R); ++r) {
    if (r & (1 << JA)) continue;
    const int ra = r | (1 << JA);
    const V2<Real> A0 = v[r], A1 = v[ra];
    const V2<Real> P0 = shfl_xor<Real>(A0, 1 << s), P1 = shfl_xor<Real>(A1, 1 << s);
    if (!AB_ON(r)) continue;
    const V2<Real> x0 = l ? P0 : A0, x1 = l ? A0 : P0, x2 = l ? P1 : A1, x3 = l ? A1 : P1;
    v[r] = cadd<Real>(cmul2<Real>(r0[0], x0, r0[1], x1), cmul2<Real>(r0[2], x2, r0[3], x3));
    v[ra] = cadd<Real>(cmul2<Real>(r1[0], x0, r1[1], x1), cmul2<Real>(r1[2], x2, r1[3], x3));
  }
}

// 4x4 with matrix MSB on lane bit sa and LSB on lane bit sb.
template <typename Real, int R>
__device__ __forceinline__ void lane_2q(V2<Real> (&v)[1 << R], int sa, int sb, const V2<Real>* m, bool thr,
                                        uint32_t creg) {
  const int lane = threadIdx.x & 31;
  const int k0 = (((lane >> sa) & 1) << 1) | ((lane >> sb) & 1);
  const V2<Real> c0 = ld_coef<Real>(m + 4 * k0 + k0), c1 = ld_coef<Real>(m + 4 * k0 + (k0 ^ 1)),
                 c2 = ld_coef<Real>(m + 4 * k0 + (k0 ^ 2)), c3 = ld_coef<Real>(m + 4 * k0 + (k0 ^ 3));
  const int mb = 1 << sb, ma = 1 << sa;
#pragma unroll
  for (int r = 0; r < (1 << R); ++r) {
    const V2<Real> own = v[r];
    const V2<Real> p1 = shfl_xor<Real>(own, mb), p2 = shfl_xor<Real>(own, ma), p3 = shfl_xor<Real>(own, ma | mb);
    const V2<Real> nv = cadd<Real>(cmul2<Real>(c0, own, c1, p1), cmul2<Real>(c2, p2, c3, p3));
    if (AB_ON(r)) v[r] = nv;
  }
}

template <typename Real, int R, int QB>
__device__ __forceinline__ void dispatch_2q(const Op& op, V2<Real> (&v)[1 << R], const V2<Real>* m, bool thr) {
  const uint32_t creg = op.creg;
  if (op.b < 5) {
    if (op.a < 5) {
      lane_2q<Real, R>(v, op.a, op.b, m, thr, creg);
      return;
    }
    switch (op.a - 5) {
      case 0: if constexpr (R > 0) regl_2q<Real, R, 0>(v, op.b, m, thr, creg); break;
      case 1: if constexpr (R > 1) regl_2q<Real, R, 1>(v, op.b, m, thr, creg); break;
      case 2: if constexpr (R > 2) regl_2q<Real, R, 2>(v, op.b, m, thr, creg); break;
      case 3: if constexpr (R > 3) regl_2q<Real, R, 3>(v, op.b, m, thr, creg); break;
      case 4: if constexpr (R > 4) regl_2q<Real, R, 4>(v, op.b, m, thr, creg); break;
    }
    return;
  }
  dispatch_reg_2q<Real, R, QB>(op.a - 5, op.b - 5, v, m, thr, creg);
}

// ---- the warp-tile pass -----------------------------------------------------
// OCC: the resident 128-thread blocks per SM the variant is compiled for
// (register budget 65536 / (128 * OCC)); more resident warps hide more
// latency, fewer registers per thread cost spills at large R.
template <typename Real, int R, int OCC>
__global__ void __launch_bounds__(128, OCC) tile_kernel(V2<Real>* __restrict__ amps, const TilePass p,
                                                        const Op* __restrict__ ops, const V2<Real>* __restrict__ coef,
                                                        const PolyTables poly) {
  constexpr int NR = 1 << R;
  // quartets of a 4x4 per coefficient load: what the register budget
  // (65536 / (128 * OCC), at most 255) leaves beside the tile's amplitudes
  // for QB x 4 outputs and a row of coefficients
  constexpr int kRegBudget = 65536 / (128 * OCC) > 255 ? 255 : 65536 / (128 * OCC);
  constexpr int kRegData = (1 << R) * 2 * (int)sizeof(Real) / 4;
  constexpr int kCplx = 2 * (int)sizeof(Real) / 4;  // registers per complex value
  constexpr int kQuartetBlock = kRegBudget - kRegData >= (16 + 4) * kCplx + 40   ? 4
                                : kRegBudget - kRegData >= (8 + 4) * kCplx + 56 ? 2
                                                                                 : 1;
  const int lane = threadIdx.x & 31;
  const uint64_t warp = (uint64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (warp >= (1ull << (p.n - 5 - R))) return;

  uint64_t hb[5] = {0, 0, 0, 0, 0};
  uint64_t tilemask = 0x1Full;
#pragma unroll
  for (int j = 0; j < R; ++j) {
    hb[j] = 1ull << p.hq[j];
    tilemask |= hb[j];
  }
  // Deposit the warp index into the non-tile qubits (ascending).
  uint64_t base = 0, w = warp;
  for (uint32_t pos = 5; w != 0 && pos < p.n; ++pos) {
    if ((tilemask >> pos) & 1) continue;
    base |= (w & 1ull) << pos;
    w >>= 1;
  }
  const uint64_t gl = base | (uint64_t)lane;

  V2<Real> v[NR];
#pragma unroll
  for (int r = 0; r < NR; ++r) v[r] = ld_amp<Real>(amps + (gl | roff<R>(r, hb)));

  for (uint32_t i = 0; i < p.op_count; ++i) {
    const Op op = ops[p.op_begin + i];
    const V2<Real>* m = coef + op.coef;
    const bool thr = (gl & op.ctrl) == op.ctrl;
    switch (op.type) {
      case OP_1Q: {
        if (op.a < 5) {
          lane_1q<Real, R>(v, op.a, m, thr, op.creg);
          break;
        }
        // gate pairs need the coefficients of both gates and a quartet of
        // temporaries live: only in the variants whose register budget
        // (65536 / (128 * OCC), at most 255) leaves room for them beside the
        // tile's amplitudes
        constexpr int kBudget = 65536 / (128 * OCC) > 255 ? 255 : 65536 / (128 * OCC);
        constexpr int kData = (1 << R) * 2 * (int)sizeof(Real) / 4;
        constexpr bool kPairs = R >= 2 && kBudget - kData >= 96;
        if (kPairs && op.ctrl == 0 && op.creg == 0 && i + 1 < p.op_count) {
          const Op nx = ops[p.op_begin + i + 1];
          if (nx.type == OP_1Q && nx.a >= 5 && nx.a != op.a && nx.ctrl == 0 && nx.creg == 0) {
            dispatch_pair<Real, R>(op.a - 5, nx.a - 5, v, m, coef + nx.coef);
            ++i;
            break;
          }
        }
        dispatch_reg<Real, R>(op, v, m, thr);
        break;
      }
      case OP_X:
        if (op.a < 5) lane_x<Real, R>(v, op.a, thr, op.creg);
        else dispatch_reg<Real, R>(op, v, m, thr);
        break;
      case OP_2Q:
        dispatch_2q<Real, R, kQuartetBlock>(op, v, m, thr);
        break;
      default:
        diag_ops<Real, R>(op, v, gl, hb, coef, poly);
        break;
    }
  }

#pragma unroll
  for (int r = 0; r < NR; ++r) st_amp<Real>(amps + (gl | roff<R>(r, hb)), v[r]);
}

template <typename Real, int R, int OCC>
static cudaError_t launch_tile_t(void* amps, const TilePass& p, const Op* ops, const void* coef, PolyTables poly,
                                 cudaStream_t s) {
  const uint64_t warps = 1ull << (p.n - 5 - R);
  const uint32_t wpb = 4;
  const uint64_t blocks = (warps + wpb - 1) / wpb;
  tile_kernel<Real, R, OCC>
      <<<(unsigned)blocks, 32 * wpb, 0, s>>>((V2<Real>*)amps, p, ops, (const V2<Real>*)coef, poly);
  return cudaGetLastError();
}

template <typename Real, int R>
static cudaError_t launch_tile_occ(void* amps, const TilePass& p, const Op* ops, const void* coef, PolyTables poly,
                                   cudaStream_t s) {
  // default: FP32 tiles run best at 4 blocks per SM, FP64 at 2 (measured on
  // the n=30 depth-40 brickwall: FP32 R=5 occ 2/3/4 = 1.22/1.00/0.94 s, FP64
  // R=5 occ 2/3 = 1.57/1.63 s)
  const uint32_t occ = p.occupancy ? p.occupancy : (sizeof(Real) == 4 ? 4u : 2u);
  switch (occ) {
    case 3: return launch_tile_t<Real, R, 3>(amps, p, ops, coef, poly, s);
    case 4: return launch_tile_t<Real, R, 4>(amps, p, ops, coef, poly, s);
    default: return launch_tile_t<Real, R, 2>(amps, p, ops, coef, poly, s);
  }
}

cudaError_t launch_tile_pass(void* amps, int precision, const TilePass& p, const Op* ops, const void* coef,
                             PolyTables poly, int* /*dev_error: no waits in this kernel*/, int /*sm_count*/,
                             cudaStream_t s) {
  if (p.R < 1 || p.R > 5 || p.n < 5 + p.R) return cudaErrorInvalidValue;
  const bool f64 = precision == ALEPH_B200_F64;
  switch (p.R) {
#define AB_TILE_CASE(RR)                                                        \
  case RR:                                                                      \
    return f64 ? launch_tile_occ<double, RR>(amps, p, ops, coef, poly, s)       \
               : launch_tile_occ<float, RR>(amps, p, ops, coef, poly, s);
    AB_TILE_CASE(1)
    AB_TILE_CASE(2)
    AB_TILE_CASE(3)
    AB_TILE_CASE(4)
    AB_TILE_CASE(5)
#undef AB_TILE_CASE
  }
  return cudaErrorInvalidValue;
}

}  // namespace ab
