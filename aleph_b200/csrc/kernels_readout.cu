// kernels_readout.cu — on-device FP64 readout: norm, measurement
// (reduce + decide + collapse, no host round trip), Pauli expectation and
// marginal probabilities. All reductions accumulate in FP64 (also for FP32
// states) and are deterministic: fixed per-block partials, then one block
// sums the partials in index order.
//
// Semantics: validate_state (crates/aleph-sv/src/measure.rs:23-33,
// crates/aleph-sv/src/sampling.rs:36-57), measure_impl (measure.rs:41-102),
// expectation_value_impl (measure.rs:155-233), probabilities_impl
// (measure.rs:239-273).

#include <cmath>

#include "common.cuh"

namespace ab {

constexpr int RB = 256;  // threads per reduction block

uint32_t reduce_blocks(uint32_t n, int sm_count) {
  const uint64_t len = 1ull << n;
  uint64_t b = (len + RB * 8 - 1) / (RB * 8);
  const uint64_t cap = (uint64_t)sm_count * 8;
  if (b > cap) b = cap;
  return (uint32_t)(b ? b : 1);
}

template <int NV>
__device__ __forceinline__ void block_reduce_store(double (&v)[NV], double* out) {
  __shared__ double red[NV][RB / 32];
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    double x = v[k];
    for (int o = 16; o; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if ((threadIdx.x & 31) == 0) red[k][threadIdx.x >> 5] = x;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      double s = 0.0;
      for (int w = 0; w < RB / 32; ++w) s += red[k][w];
      out[k] = s;
    }
  }
}

// Sum over the blocks of one of NV partials by a warp: every lane adds a
// strided share (four loads in flight), then a shuffle tree; the order is fixed.
// (One thread adding 1184 partials in order took 65 us, as long as a sweep
// over 2^25 complex64 amplitudes.)
template <int NV>
__device__ __forceinline__ double sum_partials(const double* __restrict__ partials, uint32_t nblocks, int k) {
  double s[4] = {0.0, 0.0, 0.0, 0.0};
  uint32_t b = threadIdx.x & 31;
  for (; b + 96 < nblocks; b += 128) {
#pragma unroll
    for (int u = 0; u < 4; ++u) s[u] += __ldcg(partials + (size_t)(b + 32 * u) * NV + k);
  }
  for (; b < nblocks; b += 32) s[0] += __ldcg(partials + (size_t)b * NV + k);
  double x = (s[0] + s[1]) + (s[2] + s[3]);
  for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// Stores this block's sums; the block that finishes last then adds all blocks'
// and returns true with the totals in tot (valid for every thread). The
// ticket returns to zero by itself. A kernel of its own for the totals cost
// 4 us and a launch after every sweep.
template <int NV>
__device__ __forceinline__ bool reduce_grid(double (&v)[NV], double* partials, double (&tot)[NV]) {
  __shared__ double all[NV];
  __shared__ bool last;
  block_reduce_store<NV>(v, partials + NV * (size_t)blockIdx.x);
  if (threadIdx.x == 0) {
    __threadfence();
    uint32_t* ticket = reinterpret_cast<uint32_t*>(reinterpret_cast<char*>(partials) - kReduceHeader);
    last = atomicInc(ticket, gridDim.x - 1) == gridDim.x - 1;
    __threadfence();
  }
  __syncthreads();
  if (!last) return false;
  for (int k = threadIdx.x >> 5; k < NV; k += RB / 32) {
    const double s = sum_partials<NV>(partials, gridDim.x, k);
    if ((threadIdx.x & 31) == 0) all[k] = s;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < NV; ++k) tot[k] = all[k];
  return true;
}
template <int NV>
__device__ __forceinline__ void reduce_grid_to(double (&v)[NV], double* partials, double* out) {
  double tot[NV];
  if (reduce_grid<NV>(v, partials, tot) && threadIdx.x == 0)
#pragma unroll
    for (int k = 0; k < NV; ++k) out[k] = tot[k];
}

template <typename Real>
__device__ __forceinline__ double abs2(V2<Real> a) {
  const double x = a.x, y = a.y;
  return x * x + y * y;
}

// ---- norm: [sum |a|^2, non-finite count] ------------------------------------
template <typename Real>
__global__ void __launch_bounds__(RB) norm_kernel(const V2<Real>* __restrict__ amps, uint64_t len,
                                                  double* partials, double* __restrict__ out2) {
  double v[2] = {0.0, 0.0};
  // four independent loads per step keep enough bytes in flight for the
  // 8-byte complex64 amplitudes (one load per step left the pass latency-bound)
  const uint64_t stride = (uint64_t)gridDim.x * RB;
  uint64_t i = (uint64_t)blockIdx.x * RB + threadIdx.x;
  for (; i + 3 * stride < len; i += 4 * stride) {
    V2<Real> a[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) a[k] = ld_amp<Real>(amps + i + k * stride);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const double p = abs2<Real>(a[k]);
      if (isfinite(p)) v[0] += p;
      else v[1] += 1.0;
    }
  }
  for (; i < len; i += stride) {
    const double p = abs2<Real>(ld_amp<Real>(amps + i));
    if (isfinite(p)) v[0] += p;
    else v[1] += 1.0;
  }
  reduce_grid_to<2>(v, partials, out2);
}

cudaError_t launch_norm(const void* amps, int precision, uint32_t n, double* partials, uint32_t nblocks, double* out2,
                        cudaStream_t s) {
  const uint64_t len = 1ull << n;
  if (precision == ALEPH_B200_F64) norm_kernel<double><<<nblocks, RB, 0, s>>>((const double2*)amps, len, partials, out2);
  else norm_kernel<float><<<nblocks, RB, 0, s>>>((const float2*)amps, len, partials, out2);
  return cudaGetLastError();
}

// ---- measurement ---------------------------------------------------------------
// What a measurement's decision needs and writes.
struct Decision {
  uint32_t qubit, n_uniforms;
  const double* uniforms;
  int32_t* status;
  double* dec;
  uint8_t* outcome_slot;
  double tol;
};
__device__ void measure_decide(const double* sums, const Decision& d);

// [p0, p1, non-finite count], and the decision by the last block.
template <typename Real>
__global__ void __launch_bounds__(RB) branch_kernel(const V2<Real>* __restrict__ amps, uint64_t len, uint64_t qb,
                                                    double* partials, const Decision d) {
  double v[3] = {0.0, 0.0, 0.0};
  auto add = [&](uint64_t i, double p) {
    if (!isfinite(p)) v[2] += 1.0;
    else if (i & qb) v[1] += p;
    else v[0] += p;
  };
  const uint64_t stride = (uint64_t)gridDim.x * RB;
  uint64_t i = (uint64_t)blockIdx.x * RB + threadIdx.x;
  for (; i + 3 * stride < len; i += 4 * stride) {  // four loads in flight per step (see norm_kernel)
    V2<Real> a[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) a[k] = ld_amp<Real>(amps + i + k * stride);
#pragma unroll
    for (int k = 0; k < 4; ++k) add(i + k * stride, abs2<Real>(a[k]));
  }
  for (; i < len; i += stride) add(i, abs2<Real>(ld_amp<Real>(amps + i)));
  double tot[3];
  if (reduce_grid<3>(v, partials, tot) && threadIdx.x == 0) measure_decide(tot, d);
}

// status[0]: error code (0 ok), status[1]: uniforms consumed, status[2]: failing qubit;
// dec[0] = outcome (0/1), dec[1] = 1/norm scale; dval[0] = reported probability.
__device__ void measure_decide(const double* sums, const Decision& d) {
  double* dec = d.dec;
  int32_t* status = d.status;
  const uint32_t qubit = d.qubit;
  dec[0] = -1.0;  // "skip collapse" unless a decision is made below
  if (status[0] != 0) return;  // an earlier instruction failed: do nothing further
  const double p0r = sums[0], p1r = sums[1], bad = sums[2];
  const double total = p0r + p1r;
  if (bad > 0.0 || !isfinite(total) || fabs(total - 1.0) > d.tol) {
    status[0] = ALEPH_B200_INVALID_STATE;
    status[2] = (int32_t)qubit;
    return;
  }
  const double p0 = fmin(fmax(p0r, 0.0), 1.0), p1 = fmin(fmax(p1r, 0.0), 1.0);
  const bool one_degen = p1 < 1e-300, zero_degen = p0 < 1e-300;
  bool outcome;
  double p;
  if (zero_degen && one_degen) {
    status[0] = ALEPH_B200_DEGENERATE_MEASUREMENT;
    status[2] = (int32_t)qubit;
    dec[2] = fmax(p1, p0);
    return;
  } else if (zero_degen) {
    outcome = true;
    p = p1;
  } else if (one_degen) {
    outcome = false;
    p = p0;
  } else {
    const uint32_t used = (uint32_t)status[1];
    if (used >= d.n_uniforms) {
      status[0] = ALEPH_B200_INVALID_ARGUMENT;
      status[2] = (int32_t)qubit;
      return;
    }
    outcome = d.uniforms[used] < p1;
    status[1] = (int32_t)(used + 1);
    p = outcome ? p1 : p0;
  }
  dec[0] = outcome ? 1.0 : 0.0;
  dec[1] = sqrt(p);
  if (d.outcome_slot) *d.outcome_slot = outcome ? 1 : 0;
}

// The kept half is read, divided and written; the other half is only written.
// A thread takes pairs (bit 0, bit 1) of the measured qubit, four per step, so
// that four loads are in flight and the discarded amplitudes are never loaded.
template <typename Real>
__global__ void __launch_bounds__(256) collapse_kernel(V2<Real>* __restrict__ amps, uint64_t pairs, uint32_t qubit,
                                                       const double* __restrict__ dec) {
  const double o = dec[0];
  if (o < 0.0) return;
  const uint64_t qb = 1ull << qubit, keep = o > 0.5 ? qb : 0, drop = qb ^ keep;
  const double norm = dec[1];
  const double d = norm * norm;
  // num-complex division by Complex::new(norm, 0.0), as the reference's `*a /= ...`
  auto scaled = [&](V2<Real> a) { return mk<Real>((Real)(((double)a.x * norm) / d), (Real)(((double)a.y * norm) / d)); };
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  for (; p + 3 * stride < pairs; p += 4 * stride) {
    V2<Real> a[4];
    uint64_t at[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      at[k] = insert_zero(p + k * stride, qubit);
      a[k] = ld_amp<Real>(amps + (at[k] | keep));
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      st_amp<Real>(amps + (at[k] | keep), scaled(a[k]));
      st_amp<Real>(amps + (at[k] | drop), mk<Real>(0, 0));
    }
  }
  for (; p < pairs; p += stride) {
    const uint64_t i = insert_zero(p, qubit);
    st_amp<Real>(amps + (i | keep), scaled(ld_amp<Real>(amps + (i | keep))));
    st_amp<Real>(amps + (i | drop), mk<Real>(0, 0));
  }
}

cudaError_t launch_measure_pass(void* amps, int precision, uint32_t n, uint32_t qubit, double* partials,
                                uint32_t nblocks, const double* uniforms, uint32_t n_uniforms, int32_t* status,
                                uint8_t* outcome_slot, cudaStream_t s) {
  const uint64_t len = 1ull << n;
  const uint64_t qb = 1ull << qubit;
  double* dec = partials + 3 * (size_t)nblocks;
  const Decision d{qubit, n_uniforms, uniforms, status, dec, outcome_slot, norm_tolerance(len, precision)};
  if (precision == ALEPH_B200_F64)
    branch_kernel<double><<<nblocks, RB, 0, s>>>((const double2*)amps, len, qb, partials, d);
  else
    branch_kernel<float><<<nblocks, RB, 0, s>>>((const float2*)amps, len, qb, partials, d);
  const uint64_t pairs = len / 2, b = (pairs + 255) / 256;
  const unsigned blocks = (unsigned)(b > 148ull * 32 ? 148ull * 32 : b);
  if (precision == ALEPH_B200_F64) collapse_kernel<double><<<blocks, 256, 0, s>>>((double2*)amps, pairs, qubit, dec);
  else collapse_kernel<float><<<blocks, 256, 0, s>>>((float2*)amps, pairs, qubit, dec);
  return cudaGetLastError();
}

// ---- Pauli sum: up to 16 terms that share one X/Y (flip) mask, one sweep ----------
// P = (x) Paulis with X/Y positions `xmask` (flip), Z/Y positions `zmask`
// (sign), ny = number of Y factors. (P psi)_i = i^ny (-1)^{popc(zmask & j)} psi_j
// with j = i ^ xmask: Y = i X Z, X flips, Z signs the pre-image bit. The terms of
// a group differ only in the sign and in i^ny, so conj(a_i) a_j is formed once
// per pair and shared. i and j contribute the same real part (P is Hermitian:
// the two products are conjugate to each other), so with a flip a thread takes
// the pair once, at the member with the mask's highest bit clear: every
// amplitude is read once and the products are formed once. (One thread per
// member read everything twice: 93 us a group at n = 23 FP64 against 28 us
// now, with the terms unrolled to the group's size and not to 16.)
// partials per block: [sum |a|^2, non-finite count, term 0 .. NT-1].
//
// Signs: an index is a warp-uniform part plus a lane part on disjoint bits, so the
// parity of a term's mask splits the same way. Each lane forms one term's uniform
// parity and a ballot hands all of them to the warp as one word.
template <typename Real, bool DIAG, int NT>
__global__ void __launch_bounds__(RB) pauli_group_kernel(const V2<Real>* __restrict__ amps, uint64_t count,
                                                         const PauliGroup g, uint32_t pivot, double* partials,
                                                         double* __restrict__ out) {
  constexpr int NV = 2 + NT, U = 4;
  double v[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) v[k] = 0.0;
  const uint64_t stride = (uint64_t)gridDim.x * RB;
  const uint32_t lane = threadIdx.x & 31;
  auto index = [&](uint64_t p) { return DIAG ? p : insert_zero(p, pivot); };
  uint64_t my_z = 0;  // this lane's term
  uint32_t lane_word = 0, swap = 0;  // per term: parity of the lane part; i^ny takes the imaginary part
#pragma unroll
  for (int k = 0; k < NT; ++k) {
    if (k >= (int)g.count) break;
    if ((int)lane == k) my_z = g.zmask[k];
    const uint32_t y = DIAG ? 0u : g.ny[k] & 3;
    // i^ny: ny & 3 = 0, 1, 2, 3 keeps re, -im, -re, im; the sign mask applies to j = i ^ xmask
    const uint32_t flip = (y == 1 || y == 2) ^ (__popcll(g.zmask[k] & g.xmask) & 1);
    lane_word |= ((__popcll(g.zmask[k] & index(lane)) & 1) ^ flip) << k;
    swap |= (y & 1) << k;
  }
  auto add = [&](uint32_t word, V2<Real> a, V2<Real> b) {
    const double p = abs2<Real>(a), q = DIAG ? 0.0 : abs2<Real>(b);
    if (!isfinite(p) || !isfinite(q)) {
      v[1] += 1.0;
      return;
    }
    v[0] += p + q;
    const double re = DIAG ? p : (double)a.x * b.x + (double)a.y * b.y;  // conj(a) * b
    const double im = DIAG ? 0.0 : (double)a.x * b.y - (double)a.y * b.x;
#pragma unroll
    for (int k = 0; k < NT; ++k)
      if (k < (int)g.count) {
        const double t = !DIAG && ((swap >> k) & 1) ? im : re;
        v[2 + k] += __hiloint2double(__double2hiint(t) ^ (int)((word << (31 - k)) & 0x80000000u), __double2loint(t));
      }
  };
  // the word of a warp whose first index is p: count and stride are multiples of 32, or there is one warp
  auto word_at = [&](uint64_t p) {
    return __ballot_sync(0xffffffffu, __popcll(my_z & index(p)) & 1) ^ lane_word;
  };
  uint64_t p0 = (uint64_t)blockIdx.x * RB + (threadIdx.x & ~31u);  // the warp's first
  for (; p0 + (U - 1) * stride + 31 < count; p0 += U * stride) {  // loads in flight (see norm_kernel)
    V2<Real> a[U], b[U];
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const uint64_t i = index(p0 + k * stride) | index(lane);
      a[k] = ld_amp<Real>(amps + i);
      if constexpr (!DIAG) b[k] = ld_amp<Real>(amps + (i ^ g.xmask));
    }
#pragma unroll
    for (int k = 0; k < U; ++k) add(word_at(p0 + k * stride), a[k], DIAG ? a[k] : b[k]);
  }
  for (; p0 < count; p0 += stride) {
    const uint32_t word = word_at(p0);
    if (p0 + lane >= count) continue;
    const uint64_t i = index(p0) | index(lane);
    const V2<Real> a = ld_amp<Real>(amps + i);
    add(word, a, DIAG ? a : ld_amp<Real>(amps + (i ^ g.xmask)));
  }
  if constexpr (!DIAG) {  // both members of each pair
#pragma unroll
    for (int k = 0; k < NT; ++k) v[2 + k] *= 2.0;
  }
  reduce_grid_to<NV>(v, partials, out);
}

template <typename Real, int NT>
static cudaError_t launch_pauli_t(const V2<Real>* amps, uint32_t n, const PauliGroup& g, double* partials,
                                  uint32_t nblocks, double* out, cudaStream_t s) {
  const uint64_t len = 1ull << n;
  if (g.xmask == 0)
    pauli_group_kernel<Real, true, NT><<<nblocks, RB, 0, s>>>(amps, len, g, 0, partials, out);
  else
    pauli_group_kernel<Real, false, NT>
        <<<nblocks, RB, 0, s>>>(amps, len / 2, g, 63u - (uint32_t)__builtin_clzll(g.xmask), partials, out);
  return cudaGetLastError();
}

cudaError_t launch_pauli_group(const void* amps, int precision, uint32_t n, const PauliGroup& g, double* partials,
                               uint32_t nblocks, double* out, cudaStream_t s) {
  if (g.count == 0 || g.count > (uint32_t)PauliGroup::MAX_TERMS) return cudaErrorInvalidValue;
  // accumulators for 1, 2, 4, 8 or 16 terms
  uint32_t slots = 1;
  while (slots < g.count) slots *= 2;
  const bool f64 = precision == ALEPH_B200_F64;
  switch (slots) {
#define AB_PAULI(nt)                                                                                    \
  case nt:                                                                                              \
    return f64 ? launch_pauli_t<double, nt>((const double2*)amps, n, g, partials, nblocks, out, s)      \
               : launch_pauli_t<float, nt>((const float2*)amps, n, g, partials, nblocks, out, s);
    AB_PAULI(1)
    AB_PAULI(2)
    AB_PAULI(4)
    AB_PAULI(8)
    AB_PAULI(16)
#undef AB_PAULI
  }
  return cudaErrorInvalidValue;
}

// One Pauli string: [sum |a|^2, non-finite count, Re <psi|P|psi>].
cudaError_t launch_expectation(const void* amps, int precision, uint32_t n, uint64_t xmask, uint64_t zmask,
                               uint32_t ny, double* partials, uint32_t nblocks, double* out3, cudaStream_t s) {
  PauliGroup g{};
  g.xmask = xmask;
  g.count = 1;
  g.zmask[0] = zmask;
  g.ny[0] = ny;
  return launch_pauli_group(amps, precision, n, g, partials, nblocks, out3, s);
}

// ---- marginal probabilities ------------------------------------------------------
// out[o] = sum of |a_i|^2 over the basis states i whose selected qubits spell
// o. Lanes are qubits 0..4, so every load is one run of 32 amplitudes. A warp
// fixes the selected qubits above 4 (a pattern) and adds over the unselected
// ones above 4 in its own registers; at the end a shuffle tree adds over the
// unselected lane qubits. Where the patterns alone would leave the chip idle, the
// unselected qubits' top `split_bits` are split over warps: 8 of a CTA meet in
// shared memory, and a second kernel adds the CTAs' partial tables. No atomics,
// one read of the state, and the norm comes with it. (At n = 23 FP64 a histogram
// of shared-memory atomics took 150 us for 6 qubits and a thread per output 2.8 ms
// for 12; both take 24 us now.)
struct Marginal {
  uint32_t k, lane_sel;  // selected count; mask of the selected lane qubits
  uint32_t lanes;        // active lanes (32, or 2^n below 5 qubits)
  uint32_t pat_bits, split_bits;
  uint64_t split_mask, loop_mask;  // qubits above 4: split / added in the loop
  uint64_t loops;
  // Index bits move in runs of consecutive ones (bit by bit, the moves of a marginal
  // over all qubits took longer than its loads): pattern -> selected qubits above 4, and
  // those qubits -> the outcome's bits.
  struct Runs {
    uint32_t count;
    uint8_t from[40], to[40];
    uint64_t mask[40];
    __device__ __forceinline__ uint64_t operator()(uint64_t x) const {
      uint64_t r = 0;
      for (uint32_t k = 0; k < count; ++k) r |= ((x >> from[k]) & mask[k]) << to[k];
      return r;
    }
    void add(uint32_t a, uint32_t b) {  // bit a goes to bit b; extends the last run where it can
      if (count) {
        const uint32_t len = (uint32_t)__builtin_popcountll(mask[count - 1]);
        if (from[count - 1] + len == a && to[count - 1] + len == b) {
          mask[count - 1] = mask[count - 1] << 1 | 1;
          return;
        }
      }
      from[count] = (uint8_t)a;
      to[count] = (uint8_t)b;
      mask[count++] = 1;
    }
  } place, outcome;
  uint8_t qubits[64];
};

__device__ __forceinline__ uint64_t deposit(uint64_t x, uint64_t mask) {  // bits of x into the set bits of mask
  uint64_t r = 0;
  while (mask && x) {
    const uint64_t low = mask & (~mask + 1);
    if (x & 1) r |= low;
    x >>= 1;
    mask ^= low;
  }
  return r;
}

template <typename Real>
__global__ void __launch_bounds__(RB) marginal_kernel(const V2<Real>* __restrict__ amps, const Marginal m,
                                                      uint64_t items, double* __restrict__ tables,
                                                      double* norm_partials, double* __restrict__ norm_out) {
  __shared__ double red[RB / 32][32];
  const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const bool meet = m.split_bits >= 3;  // the CTA's warps are eight splits of one pattern
  const bool on = lane < m.lanes;
  uint32_t o_lane = 0;
  for (uint32_t t = 0; t < m.k; ++t)
    if (m.qubits[t] < 5) o_lane |= ((lane >> m.qubits[t]) & 1) << t;
  double v[2] = {0.0, 0.0};
  const uint64_t warps = 1ull << (m.pat_bits + m.split_bits);
  for (uint64_t item = blockIdx.x; item < items; item += gridDim.x) {
    const uint64_t id = item * (RB / 32) + w;
    double s = 0.0;
    const uint64_t pat = id >> m.split_bits, split = id & ((1ull << m.split_bits) - 1);
    const uint64_t fixed = m.place(pat);
    if (id < warps && on) {
      const V2<Real>* base = amps + (fixed | deposit(split, m.split_mask) | lane);
      uint64_t x = 0;
      auto next = [&] { x = ((x | ~m.loop_mask) + 1) & m.loop_mask; };
      double bad = 0.0;
      auto add = [&](double p) {
        if (isfinite(p)) s += p;
        else bad += 1.0;
      };
      uint64_t r = 0;
      for (; r + 4 <= m.loops; r += 4) {  // four loads in flight (see norm_kernel)
        V2<Real> a[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          a[k] = ld_amp<Real>(base + x);
          next();
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) add(abs2<Real>(a[k]));
      }
      for (; r < m.loops; ++r) {
        add(abs2<Real>(ld_amp<Real>(base + x)));
        next();
      }
      v[0] += s;
      v[1] += bad;
    }
#pragma unroll
    for (int b = 0; b < 5; ++b) {
      const double other = __shfl_xor_sync(0xffffffffu, s, 1 << b);
      if (!((m.lane_sel >> b) & 1)) s += other;
    }
    bool writes = id < warps && on && (lane & ~m.lane_sel) == 0;
    uint64_t table = split;
    if (meet) {
      __syncthreads();  // the previous item's sums have been read
      red[w][lane] = s;
      __syncthreads();
      s = 0.0;
#pragma unroll
      for (int x = 0; x < RB / 32; ++x) s += red[x][lane];
      writes = writes && w == 0;
      table = split >> 3;
    }
    if (writes) {
      tables[(table << m.k) + (o_lane | m.outcome(fixed))] = s;
    }
  }
  __syncthreads();
  reduce_grid_to<2>(v, norm_partials, norm_out);
}

// out[o] = sum over the tables, a warp per output in a fixed order.
__global__ void __launch_bounds__(256) marginal_sum_kernel(const double* __restrict__ tables, uint32_t ntables,
                                                           uint64_t dim, double* __restrict__ out) {
  const uint32_t lane = threadIdx.x & 31;
  for (uint64_t o = (uint64_t)blockIdx.x * 8 + (threadIdx.x >> 5); o < dim; o += (uint64_t)gridDim.x * 8) {
    double s = 0.0;
    for (uint32_t t = lane; t < ntables; t += 32) s += tables[(uint64_t)t * dim + o];
    for (int x = 16; x; x >>= 1) s += __shfl_xor_sync(0xffffffffu, s, x);
    if (lane == 0) out[o] = s;
  }
}

namespace {
struct MarginalPlan {
  Marginal m;
  uint64_t items;
  uint32_t blocks, tables;
};
MarginalPlan plan_marginal(uint32_t n, const uint32_t* qubits, uint32_t k, int sm_count) {
  MarginalPlan P{};
  Marginal& m = P.m;
  m.k = k;
  m.lanes = n < 5 ? 1u << n : 32u;
  uint64_t sel = 0;
  for (uint32_t t = 0; t < k; ++t) {
    sel |= 1ull << qubits[t];
    m.qubits[t] = (uint8_t)qubits[t];
  }
  m.lane_sel = (uint32_t)(sel & 31u) | (n < 5 ? 31u & ~((1u << n) - 1) : 0u);  // absent lane qubits: nothing to add
  const uint64_t high = n > 5 ? ((1ull << n) - 1) & ~31ull : 0ull;
  for (uint32_t q = 5; q < n; ++q)
    if ((sel >> q) & 1) m.place.add(m.pat_bits++, q);
  for (uint32_t t = 0; t < k; ++t)
    if (qubits[t] >= 5) m.outcome.add(qubits[t], t);
  uint64_t rest = high & ~sel;
  const uint32_t rest_bits = (uint32_t)__builtin_popcountll(rest);
  // about 2^13 warps: 55 per SM, a little under what an SM holds
  m.split_bits = m.pat_bits < 13 ? (rest_bits < 13 - m.pat_bits ? rest_bits : 13 - m.pat_bits) : 0;
  for (uint32_t b = 0; b < m.split_bits; ++b) {
    const uint64_t top = 1ull << (63 - __builtin_clzll(rest));
    m.split_mask |= top;
    rest ^= top;
  }
  m.loop_mask = rest;
  m.loops = 1ull << (rest_bits - m.split_bits);
  const uint64_t warps = 1ull << (m.pat_bits + m.split_bits);
  P.items = (warps + RB / 32 - 1) / (RB / 32);
  P.blocks = (uint32_t)(P.items < (uint64_t)sm_count * 8 ? P.items : (uint64_t)sm_count * 8);
  P.tables = m.split_bits >= 3 ? 1u << (m.split_bits - 3) : 1u << m.split_bits;
  return P;
}
}  // namespace

size_t probabilities_scratch_bytes(uint32_t n, const uint32_t* qubits, uint32_t k, int sm_count) {
  const MarginalPlan P = plan_marginal(n, qubits, k, sm_count);
  return ((size_t)2 * P.blocks + (P.tables > 1 ? (size_t)P.tables << k : 0)) * 8;
}

cudaError_t launch_probabilities(const void* amps, int precision, uint32_t n, const uint32_t* qubits, uint32_t k,
                                 double* scratch, double* out, double* norm_out, int sm_count, cudaStream_t s) {
  const MarginalPlan P = plan_marginal(n, qubits, k, sm_count);
  double* partials = scratch;
  double* tables = P.tables > 1 ? scratch + 2 * (size_t)P.blocks : out;
  if (precision == ALEPH_B200_F64)
    marginal_kernel<double><<<P.blocks, RB, 0, s>>>((const double2*)amps, P.m, P.items, tables, partials, norm_out);
  else
    marginal_kernel<float><<<P.blocks, RB, 0, s>>>((const float2*)amps, P.m, P.items, tables, partials, norm_out);
  if (P.tables > 1) {
    const uint64_t dim = 1ull << k, b = (dim + 7) / 8;
    marginal_sum_kernel<<<(unsigned)(b < 4096 ? b : 4096), 256, 0, s>>>(tables, P.tables, dim, out);
  }
  return cudaGetLastError();
}

}  // namespace ab
