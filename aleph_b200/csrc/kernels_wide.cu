// kernels_wide.cu — the wide-tile gate pass: a CTA owns a tile of 2^12 amplitudes
// (qubits 0..3 and eight more) and applies an ordered op list in phases.
//
// In a phase every thread holds 32 amplitudes over five of the twelve tile
// qubits, and all dense gates of the phase act on those five: register
// arithmetic, no shuffles. Between phases the tile goes through shared memory
// (each amplitude is written and read once) and comes back with another
// choice of register qubits. Diagonal ops and controls may sit on any qubit.
//
// What bounds it, and why this split: a pass costs one read and one write of the
// state whatever it applies, so the gates per pass decide (8 free qubits take
// two to three times the gates of the warp tile's 5), and within it the FP64
// (or FP32) pipe. A warp tile instead keeps qubits 0..4 on lanes and pays up to
// twelve shuffles per amplitude for a 4x4 there: on the n = 27 depth-20
// brickwall its passes with lane gates took 3.4-5.7 ms, the others 1.2 ms. An
// exchange costs 64 shared-memory instructions per thread, about one 4x4's time
// on that pipe, and carries several gates. Twelve qubits: 64 KiB in FP64, so
// that two CTAs share an SM and one computes while the other moves its tile.
// At those two warps per scheduler a pass of 4x4s is bound by latency (n = 27 FP64:
// FP64 pipe 43%, issue 37%). Measured against warp tiles: n = 27 depth-20 FP64
// brickwall 44.5 -> 36.5 ms, n = 25 FP64 QFT 8.0 -> 4.6 ms, n = 22 FP32 Grover
// 4.06 -> 1.06 ms (the last two with grouped phases and diagonal cores).
//
// Bank conflicts: amplitude i of the tile sits at slot i ^ f(i >> 3) (FP64; i >> 4
// in FP32) with f linear over bits; the host orders a phase's lane qubits so
// that the lanes of one shared-memory wavefront fall on distinct banks.

#include <algorithm>

#include "tile_ops.cuh"

namespace ab {

namespace wide {

// Every register's slot offset is an XOR of the phase's five register-bit
// offsets; walked in Gray-code order it takes one XOR per register.
template <typename Real, int R, bool STORE>
__device__ __forceinline__ void exchange(V2<Real> (&v)[1 << R], V2<Real>* sm, uint32_t slot, const uint16_t (&rs)[R]) {
#pragma unroll
  for (int g = 0; g < (1 << R); ++g) {
    const int r = g ^ (g >> 1);
    if (g) {
      const int flip = (g & 1) ? 0 : (g & 2) ? 1 : (g & 4) ? 2 : (g & 8) ? 3 : R - 1;  // the bit Gray code changes
      slot ^= rs[flip];
    }
    if constexpr (STORE) sm[slot] = v[r];
    else v[r] = sm[slot];
  }
}

// Sign flips of the registers whose bit is set in `flips`.
__device__ __forceinline__ double flip_sign(double x, uint32_t sign) {
  return __hiloint2double(__double2hiint(x) ^ (int)sign, __double2loint(x));
}
__device__ __forceinline__ float flip_sign(float x, uint32_t sign) {
  return __uint_as_float(__float_as_uint(x) ^ sign);
}

// v[r] *= f for the registers with bit J set (J < 0: all of them).
template <typename Real, int R, int J>
__device__ __forceinline__ void scale_class(V2<Real> (&v)[1 << R], V2<Real> f) {
#pragma unroll
  for (int r = 0; r < (1 << R); ++r)
    if (J < 0 || ((r >> (J < 0 ? 0 : J)) & 1)) v[r] = cmul<Real>(f, v[r]);
}

// v[r] *= f for the registers with bits J and K set.
template <typename Real, int R, int J, int K>
__device__ __forceinline__ void scale_pair(V2<Real> (&v)[1 << R], V2<Real> f) {
  if constexpr (J < R && K < R) {
#pragma unroll
    for (int r = 0; r < (1 << R); ++r)
      if (((r >> J) & 1) && ((r >> K) & 1)) v[r] = cmul<Real>(f, v[r]);
  }
}
// The same for a two-bit register mask known at run time; false for any other mask.
template <typename Real, int R>
__device__ __forceinline__ bool dispatch_pair_phase(V2<Real> (&v)[1 << R], uint32_t creg, V2<Real> f) {
  switch (creg) {
    case 0x03: scale_pair<Real, R, 0, 1>(v, f); return true;
    case 0x05: scale_pair<Real, R, 0, 2>(v, f); return true;
    case 0x06: scale_pair<Real, R, 1, 2>(v, f); return true;
    case 0x09: scale_pair<Real, R, 0, 3>(v, f); return true;
    case 0x0a: scale_pair<Real, R, 1, 3>(v, f); return true;
    case 0x0c: scale_pair<Real, R, 2, 3>(v, f); return true;
    case 0x11: scale_pair<Real, R, 0, 4>(v, f); return true;
    case 0x12: scale_pair<Real, R, 1, 4>(v, f); return true;
    case 0x14: scale_pair<Real, R, 2, 4>(v, f); return true;
    case 0x18: scale_pair<Real, R, 3, 4>(v, f); return true;
  }
  return false;
}

// R = 5: 32 amplitudes per thread, so that a row of a 4x4's coefficients serves
// several quartets. R = 4: 16, at twice the warps, which hide more latency in FP64
// passes with few 4x4s (see the planner). OCC: resident CTAs per SM the
// registers are budgeted for.
// FULL: the variant with phases, tables and real matrices; passes of complex dense
// gates, permutations and sign flips run without them (the smaller kernel is 4%
// faster on the n = 27 brickwall: fewer instruction-cache misses).
template <typename Real, int R, int OCC, bool FULL>
__global__ void __launch_bounds__((1 << kWideBits) >> R, OCC)
    wide_kernel(V2<Real>* __restrict__ amps, const WidePass p, const WidePhase* __restrict__ phases,
                const Op* __restrict__ ops, const V2<Real>* __restrict__ coef, const PolyTables poly) {
  constexpr int NR = 1 << R;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  V2<Real>* sm = reinterpret_cast<V2<Real>*>(smem_raw);
  // quartets per coefficient row: what the registers leave room for
  constexpr int kQB = R == 4 ? 1 : 4;
  uint64_t base = 0;  // the tile's place: its index over the runs of the other qubits
  for (uint32_t k = 0; k < p.n_dep; ++k)
    base |= (uint64_t)((blockIdx.x >> p.dep_src[k]) & p.dep_mask[k]) << p.dep_dst[k];

  grid_launch_next();
  grid_wait_previous();
  V2<Real> v[NR];
  for (uint32_t ph = 0; ph < p.phase_count; ++ph) {
    const WidePhase& P = phases[p.phase_begin + ph];
    uint64_t gl = base;  // this thread's global index, register bits zero
    uint32_t slot = 0;
#pragma unroll
    for (int b = 0; b < (int)kWideBits - R; ++b)
      if ((threadIdx.x >> b) & 1) {
        gl |= 1ull << P.tq[b];
        slot ^= P.ts[b];
      }
    uint64_t hb[5] = {0, 0, 0, 0, 0};
    uint16_t rs[R];
#pragma unroll
    for (int j = 0; j < R; ++j) {
      hb[j] = 1ull << P.rq[j];
      rs[j] = P.rs[j];
    }
    if (ph == 0) {
#pragma unroll
      for (int r = 0; r < NR; ++r) v[r] = ld_amp<Real>(amps + (gl | roff<R>(r, hb)));
    } else {
      exchange<Real, R, false>(v, sm, slot, rs);
    }
    const uint32_t end = P.op_begin + P.op_count;
    for (uint32_t i = P.op_begin; i < end; ++i) {
      const Op op = ops[i];
      const V2<Real>* m = coef + op.coef;
      switch (op.type) {
        case OP_1Q: {
          if constexpr (sizeof(Real) == 4) {
            if (FULL && op.dsrc == WIDE_REAL) dispatch_1q_f32x2<R, true>(op.a - 5, v, m);
            if (op.dsrc == WIDE_PAIRED) dispatch_1q_f32x2<R, false>(op.a - 5, v, m);
            if (op.dsrc) break;
          } else if (FULL && op.dsrc == WIDE_REAL) {
            dispatch_reg_real<Real, R>(op.a - 5, v, m);
            break;
          }
          if (sizeof(Real) == 8 && R == 5 && op.ctrl == 0 && op.creg == 0 && i + 1 < end) {
            const Op nx = ops[i + 1];
            if (nx.type == OP_1Q && nx.a != op.a && nx.ctrl == 0 && nx.creg == 0 && !nx.dsrc) {
              dispatch_pair<Real, R>(op.a - 5, nx.a - 5, v, m, coef + nx.coef);
              ++i;
              break;
            }
          }
          dispatch_reg<Real, R>(op, v, m, (gl & op.ctrl) == op.ctrl);
          break;
        }
        case OP_X:
          dispatch_reg<Real, R>(op, v, m, (gl & op.ctrl) == op.ctrl);
          break;
        case OP_2Q:
          if constexpr (sizeof(Real) == 4) {
            if (FULL && op.dsrc == WIDE_REAL) dispatch_2q_f32x2<R, kQB, true>(op.a - 5, op.b - 5, v, m);
            if (op.dsrc == WIDE_PAIRED) dispatch_2q_f32x2<R, kQB, false>(op.a - 5, op.b - 5, v, m);
            if (op.dsrc) break;
          } else if (FULL && op.dsrc == WIDE_REAL) {
            dispatch_reg_2q_real<Real, R, kQB>(op.a - 5, op.b - 5, v, m);
            break;
          }
          // FP32: only controlled ones come here, quartet by quartet
          dispatch_reg_2q<Real, R, sizeof(Real) == 8 ? kQB : 1>(op.a - 5, op.b - 5, v, m, (gl & op.ctrl) == op.ctrl, op.creg);
          break;
        case OP_SIGNS: {  // aux sign flips follow: thread condition `mask`, registers `aux`
          uint32_t flips = 0;
          for (uint32_t e = i + 1; e <= i + op.aux; ++e) {
            const uint64_t mask = ops[e].mask;
            const uint32_t regs = ops[e].aux;
            if ((gl & mask) == mask) flips ^= regs;
          }
          i += op.aux;
          if (__any_sync(0xffffffffu, flips != 0)) {
#pragma unroll
            for (int r = 0; r < NR; ++r) {
              const uint32_t sign = (flips << (31 - r)) & 0x80000000u;
              v[r] = mk<Real>(flip_sign(v[r].x, sign), flip_sign(v[r].y, sign));
            }
          }
          break;
        }
        case OP_PHASES: if constexpr (FULL) {  // aux phases follow: thread condition `mask`; their product scales one class of registers
          V2<Real> f0 = mk<Real>(1, 0), f1 = f0;  // two chains of products
          bool any = false;
#pragma unroll 4
          for (uint32_t e = 0; e < op.aux; ++e) {  // their coefficients are contiguous
            const uint64_t mask = ops[i + 1 + e].mask;
            const V2<Real> c = ld_coef<Real>(m + e);
            if ((gl & mask) == mask) {
              if (e & 1) f1 = cmul<Real>(f1, c);
              else f0 = cmul<Real>(f0, c);
              any = true;
            }
          }
          i += op.aux;
          if (__any_sync(0xffffffffu, any)) {
            const V2<Real> f = cmul<Real>(f0, f1);
            switch (op.a) {
              case 0: scale_class<Real, R, 0>(v, f); break;
              case 1: scale_class<Real, R, 1>(v, f); break;
              case 2: scale_class<Real, R, 2>(v, f); break;
              case 3: scale_class<Real, R, 3>(v, f); break;
              case 4: if constexpr (R > 4) scale_class<Real, R, R - 1>(v, f); break;
              default: scale_class<Real, R, -1>(v, f); break;
            }
          }
          break;
        }
        case OP_CPHASE: if constexpr (FULL) {  // two or more register qubits
          const V2<Real> c = ld_coef<Real>(m);
          const bool on = (gl & op.mask) == op.mask;
          if (__any_sync(0xffffffffu, on) && !dispatch_pair_phase<Real, R>(v, op.creg, on ? c : mk<Real>(1, 0)))
            diag_ops<Real, R>(op, v, gl, hb, coef, poly);
          break;
        }
        default:
          if constexpr (FULL) diag_ops<Real, R>(op, v, gl, hb, coef, poly);
          break;
      }
    }
    if (ph + 1 < p.phase_count) {
      if (ph) __syncthreads();  // every thread has read this phase's tile
      exchange<Real, R, true>(v, sm, slot, rs);
      __syncthreads();
    } else {
#pragma unroll
      for (int r = 0; r < NR; ++r) st_amp<Real>(amps + (gl | roff<R>(r, hb)), v[r]);
    }
  }
}

template <typename Real, int R, int OCC, bool FULL>
static cudaError_t launch_t(void* amps, const WidePass& p, const WidePhase* phases, const Op* ops, const void* coef,
                          PolyTables poly, cudaStream_t s) {
  constexpr int bytes = (int)(sizeof(V2<Real>) << kWideBits);
  auto kern = wide_kernel<Real, R, OCC, FULL>;
  static uint64_t ready = 0;  // devices with the shared-memory opt-in
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev >= 64 || !((ready >> dev) & 1)) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return e;
    if (dev < 64) ready |= 1ull << dev;
  }
  return launch_overlapped(kern, 1u << (p.n - kWideBits), (1u << kWideBits) >> R, bytes, s, (V2<Real>*)amps, p, phases, ops,
                           (const V2<Real>*)coef, poly);
}

template <typename Real, int R, int OCC>
static cudaError_t launch(void* amps, const WidePass& p, const WidePhase* phases, const Op* ops, const void* coef,
                          PolyTables poly, cudaStream_t s) {
  return p.full ? launch_t<Real, R, OCC, true>(amps, p, phases, ops, coef, poly, s)
                : launch_t<Real, R, OCC, false>(amps, p, phases, ops, coef, poly, s);
}

}  // namespace wide

cudaError_t launch_wide_pass(void* amps, int precision, const WidePass& p, const WidePhase* phases, const Op* ops,
                             const void* coef, PolyTables poly, cudaStream_t s) {
  if (p.n < kWideBits || p.phase_count == 0) return cudaErrorInvalidValue;
  const bool f64 = precision == ALEPH_B200_F64;
  if (p.R == 4)
    return f64 ? wide::launch<double, 4, 2>(amps, p, phases, ops, coef, poly, s)
               : wide::launch<float, 4, 3>(amps, p, phases, ops, coef, poly, s);
  if (p.R != 5) return cudaErrorInvalidValue;
  return f64 ? wide::launch<double, 5, 2>(amps, p, phases, ops, coef, poly, s)
             : wide::launch<float, 5, 4>(amps, p, phases, ops, coef, poly, s);
}

// Layout of a phase: `regs` (R tile bits) go to registers; the others
// to lanes and warps, the lanes of one shared-memory wavefront first on bits whose
// slot vectors are independent. `io`: the phase loads or stores the state, so
// tile bits 0..3 (and 4 if it is free) take the lanes in order: runs of 16 or more
// contiguous amplitudes.
void wide_layout(const uint8_t* tile_qubits, uint32_t R, uint32_t regs, bool io, bool f64, WidePhase* P) {
  static const uint8_t vec64[kWideBits] = {1, 2, 4, 3, 5, 6, 7, 1, 2, 4, 3, 5};
  static const uint8_t vec32[kWideBits] = {1, 2, 4, 8, 3, 6, 12, 11, 5, 10, 7, 14};
  const uint8_t* vec = f64 ? vec64 : vec32;
  const uint32_t low = f64 ? 3 : 4;  // index bits that are bank bits by themselves
  auto slot_of = [&](uint32_t b) -> uint16_t { return (uint16_t)((1u << b) ^ (b >= low ? vec[b] : 0u)); };
  const uint32_t T = kWideBits - R;
  uint8_t rest[8], nr = 0, reg[5], ng = 0;
  for (uint8_t b = 0; b < kWideBits; ++b) {
    if ((regs >> b) & 1) reg[ng++] = b;
    else rest[nr++] = b;
  }
  if (!io) {
    // the first `low` lanes: a set of tile bits with independent bank vectors
    const uint32_t want = low;
    uint32_t best = 0;
    for (uint32_t set = 0; set < (1u << T) && !best; ++set) {
      if ((uint32_t)__builtin_popcount(set) != want) continue;
      uint32_t basis[4] = {0, 0, 0, 0}, rank = 0;
      for (uint32_t k = 0; k < T; ++k) {
        if (!((set >> k) & 1)) continue;
        uint32_t x = vec[rest[k]];
        for (uint32_t t = 0; t < rank; ++t) x = std::min(x, x ^ basis[t]);
        if (x) basis[rank++] = x;
      }
      if (rank == want) best = set;
    }
    uint8_t first[8], nf = 0;
    for (uint32_t pass = 0; pass < 2; ++pass)
      for (uint32_t k = 0; k < T; ++k)
        if ((((best >> k) & 1) != 0) == (pass == 0)) first[nf++] = rest[k];
    std::copy(first, first + T, rest);
  }
  for (uint32_t k = 0; k < T; ++k) {
    P->tq[k] = tile_qubits[rest[k]];
    P->ts[k] = slot_of(rest[k]);
  }
  for (uint32_t k = 0; k < R; ++k) {
    P->rq[k] = tile_qubits[reg[k]];
    P->rs[k] = slot_of(reg[k]);
  }
}

}  // namespace ab
