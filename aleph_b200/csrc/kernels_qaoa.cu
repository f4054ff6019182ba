// kernels_qaoa.cu — batched QAOA Max-Cut sweep: many parameter sets with
// ragged qubit counts in one persistent launch.
//
// Circuit of one set (build_qaoa, crates/aleph-ir/src/ansatz.rs:71-98): H on
// every qubit, then p layers of [CNOT(i,j) Rz(2 gamma)_j CNOT(i,j) per edge,
// Rx(2 beta) on every qubit]. On a basis state z the edge gadget is the phase
// exp(-i gamma (1 - 2 [z_i != z_j])), so a cost layer is the diagonal
// exp(-i gamma (m - 2 cut(z))) with m edges; a mixer layer is Rx(2 beta) on
// every qubit. The output is <C> = sum_z |psi_z|^2 cut(z), the expectation of
// H_C = sum_edges 1/2 (I - Z_i Z_j) (ansatz.rs:100-117), reduced in FP64.
//
// A state of at most SMEM_N qubits lives in one CTA's shared memory for the
// whole circuit. A larger one is streamed in tiles of 2^13 amplitudes, and its
// tiles are spread over all CTAs: a set's passes are work items in one queue.
//
// Passes. The mixer of a layer is a product of Rx on every qubit, so its parts
// on the low qubits 0..12 (A) and on the high ones 13..n-1 (B) commute; a cost
// layer is diagonal and needs whole amplitudes only. So the layers alternate which
// part they start with, and two halves meet in one pass:
//     A: cost 1, low 1 | B: high 1, cost 2, high 2 | A: low 2, cost 3, low 3 | ...
// p + 1 passes over the state for p layers, where one pass per part takes 2p. The
// first pass generates |+>^n, the last one accumulates <C> and writes nothing. An
// A tile is a contiguous chunk; a B tile spans the high qubits and the lowest
// c = 26 - n ones.
//
// In a tile, the top bits are mixed in registers and bits 0..4 by lane shuffles
// (layout 1), one trip through shared memory brings the bits between (5..7 in FP32,
// 5..8 in FP64) into registers (layout 2), where the cost phase is applied and the
// next layer's part starts, and a second trip brings the top bits back. The first
// pass goes the same way from a constant tile with nothing to finish.
//
// cut(z) of a tile amplitude i: T[i] (edges inside the tile's qubits, a table per
// set and tile kind, built once by prep_kernel) + edges among the tile's fixed
// qubits (a constant) + X0[i & 127] + X1[i >> 7] (edges between the two, rebuilt
// per tile from neighbour masks). Multiple edges between the same pair count
// once each, as the repeated gadgets do (the masks come in bit planes).
//
// Queue. Items are handed out in order: wave by wave, pass by pass, set by set. The
// sets of a wave share one half of the state buffer; a wave starts once the wave
// before the last has finished with that half, and a pass of a set once the
// set's previous pass has. An item waits only for items before it in the queue, and
// those are held by CTAs that already run, so the queue cannot lock up; every
// wait is bounded all the same.
//
// Measured (n = 12..22, p = 4): one CTA per set with 2p passes took 39 ms for 384
// FP32 sets, most of it the last n = 22 sets on one CTA each; the queue with p + 1
// passes takes 10.9 ms, host staging included. FP64: 35.6 and 19.4 ms. 1024 FP64 sets
// of n = 12..24, which kept the former kernel busy to the end: 177 ms; 207 with the
// queue on 8 warps, 195 with 16, 189 with the next tile fetched ahead, 160 with the
// first pass on the common way (its own form held both results of every register and
// spilled; a third of the shared-memory pipe's work was spills). That pipe is what
// bounds FP64 then: shuffles of 16-byte amplitudes and two trips per tile.

#include "common.cuh"

namespace ab {

namespace qaoa {

constexpr int PREP_THREADS = 256;
constexpr int TILE_BITS = 13;
constexpr uint32_t TILE = 1u << TILE_BITS;
constexpr int MAX_EDGES = 128;
template <typename Real>
struct Cfg {
  static constexpr int SMEM_N = 13;  // states kept in shared memory (the tile size)
  // FP32 tiles (64 KiB) leave room for two CTAs per SM, which overlap one
  // CTA's tile loads with the other's arithmetic
  static constexpr int CTAS_PER_SM = sizeof(Real) == 4 ? 2 : 1;
  // FP64: 16 warps on the one 128 KiB tile, 16 amplitudes a thread
  static constexpr int WARP_BITS = sizeof(Real) == 4 ? 3 : 4;
  static constexpr int THREADS = 32 << WARP_BITS;
};

// Per streamed set and tile kind (0: A, 1: B): the neighbour masks in bit planes.
constexpr int PLANES = 8;  // multiplicities up to 128 edges
struct Masks {
  uint16_t cross[TILE_BITS][PLANES];  // tile bit -> neighbours among the fixed qubits
  uint16_t fixed[TILE_BITS][PLANES];  // fixed qubit -> neighbours among the fixed qubits
  uint32_t planes;                    // planes in use
  uint32_t pad;
};

struct Args {
  const aleph_b200_qaoa_set* sets;
  const uint32_t* edges;   // (u, v) pairs
  const double* angles;    // per set: gamma[0..p), beta[0..p)
  const QaoaGroup* groups; // the queue, in order
  uint32_t* counters;      // [0] next item, [1] abort, then the groups' counters
  double* out;
  void* scratch;           // the two state halves (V2<Real>)
  uint8_t* tables;         // per streamed set: T of kind 0, T of kind 1
  Masks* masks;            // per streamed set: kind 0, kind 1
  void* phases;            // per streamed set and layer: exp(-i gamma (m - 2k)), k = 0..m
  double* partials;        // last-pass items
  uint32_t n_groups, n_items, p;
  int* error;
};

// Rx(2 beta) on tile-local bit k of every pair in S[0..len): (a, b) -> (c a - i s b, c b - i s a).
template <typename Real>
__device__ __forceinline__ void mixer_bit(V2<Real>* S, uint32_t len, uint32_t k, Real c, Real s) {
  for (uint32_t i = threadIdx.x; i < len / 2; i += Cfg<Real>::THREADS) {
    const uint32_t j0 = (uint32_t)insert_zero(i, k), j1 = j0 | (1u << k);
    const V2<Real> a = S[j0], b = S[j1];
    S[j0] = mk<Real>(c * a.x + s * b.y, c * a.y - s * b.x);
    S[j1] = mk<Real>(c * b.x + s * a.y, c * b.y - s * a.x);
  }
}

// Rx(2 beta) on tile-local bits k0 < k1 of every quartet: one shared-memory
// sweep for two qubits (the four amplitudes of a quartet in registers).
template <typename Real>
__device__ __forceinline__ void mixer_bits2(V2<Real>* S, uint32_t len, uint32_t k0, uint32_t k1, Real c, Real s) {
  auto rx = [&](V2<Real>& a, V2<Real>& b) {
    const V2<Real> x = a, y = b;
    a = mk<Real>(c * x.x + s * y.y, c * x.y - s * y.x);
    b = mk<Real>(c * y.x + s * x.y, c * y.y - s * x.x);
  };
  for (uint32_t i = threadIdx.x; i < len / 4; i += Cfg<Real>::THREADS) {
    const uint32_t e00 = (uint32_t)insert_zero(insert_zero(i, k0), k1);
    const uint32_t e01 = e00 | (1u << k0), e10 = e00 | (1u << k1), e11 = e01 | (1u << k1);
    V2<Real> a00 = S[e00], a01 = S[e01], a10 = S[e10], a11 = S[e11];
    rx(a00, a01);
    rx(a10, a11);
    rx(a00, a10);
    rx(a01, a11);
    S[e00] = a00;
    S[e01] = a01;
    S[e10] = a10;
    S[e11] = a11;
  }
}

// Rx on the tile-local bits first, first+1, ..., first+count-1: two per sweep.
template <typename Real>
__device__ __forceinline__ void mixer_range(V2<Real>* S, uint32_t len, uint32_t first, uint32_t count, Real c, Real s) {
  uint32_t k = 0;
  for (; k + 1 < count; k += 2) {
    __syncthreads();
    mixer_bits2<Real>(S, len, first + k, first + k + 1, c, s);
  }
  if (k < count) {
    __syncthreads();
    mixer_bit<Real>(S, len, first + k, c, s);
  }
  __syncthreads();
}

// Streamed tiles are swept in registers. Register layout: tile index
// i = tid | r << (5 + w) for 2^w warps (lane = tile bits 0..4, warp = the next w,
// register r = the rest), so one thread issues all of its loads before it uses one.

template <typename Real>
__device__ __forceinline__ void rx_pair(V2<Real>& a, V2<Real>& b, Real c, Real s) {
  const V2<Real> x = a, y = b;
  a = mk<Real>(c * x.x + s * y.y, c * x.y - s * y.x);
  b = mk<Real>(c * y.x + s * x.y, c * y.y - s * x.x);
}

// Rx(2 beta) on register bit k of v for every k set in mask.
template <typename Real, int NR>
__device__ __forceinline__ void rx_regs(V2<Real> (&v)[NR], uint32_t mask, Real c, Real s) {
#pragma unroll
  for (int k = 0; (1 << k) < NR; ++k) {
    if (!((mask >> k) & 1u)) continue;
#pragma unroll
    for (int r = 0; r < NR; ++r)
      if (!(r & (1 << k))) rx_pair<Real>(v[r], v[r | (1 << k)], c, s);
  }
}

// Rx(2 beta) on lane bit k for every k set in mask (uniform across the warp):
// the partner amplitude comes from lane ^ (1 << k), and both halves of a pair
// take the same form x' = c x - i s y.
template <typename Real, int NR>
__device__ __forceinline__ void rx_lanes(V2<Real> (&v)[NR], uint32_t mask, Real c, Real s) {
  // The lane bit is a runtime shuffle mask, so a rolled loop keeps one copy of the
  // body (unrolled, the FP32 sweeps stall on instruction fetch, and ran 4% slower;
  // the FP64 ones spill 2.4 KiB a thread).
#pragma unroll 1
  for (int k = 0; k < 5; ++k) {
    if (!((mask >> k) & 1u)) continue;
#pragma unroll
    for (int r = 0; r < NR; ++r) {
      const Real yx = __shfl_xor_sync(0xffffffffu, v[r].x, 1 << k);
      const Real yy = __shfl_xor_sync(0xffffffffu, v[r].y, 1 << k);
      v[r] = mk<Real>(c * v[r].x + s * yy, c * v[r].y - s * yx);
    }
  }
}

template <int WARPS>
__device__ __forceinline__ double block_sum(double v, double* red) {
  for (int o = 16; o; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double s = 0.0;
  if (threadIdx.x == 0)
    for (int w = 0; w < WARPS; ++w) s += red[w];
  __syncthreads();
  return s;
}

// 16 bytes global -> shared, asynchronously (L2 only).
__device__ __forceinline__ void copy16_async(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Tile bit of qubit q for tile kind B (c lowest qubits, then 13..n-1), or 16 + its fixed index.
__device__ __forceinline__ uint32_t place(uint32_t kind, uint32_t n, uint32_t q) {
  const uint32_t c = 2 * TILE_BITS - n;
  if (kind == 0) return q < TILE_BITS ? q : 16 + (q - TILE_BITS);
  return q < c ? q : q < TILE_BITS ? 16 + (q - c) : q - TILE_BITS + c;
}

// One CTA per streamed set and tile kind: masks, the table T, and (kind 0) the layers' phases.
template <typename Real>
__global__ void __launch_bounds__(PREP_THREADS) prep_kernel(Args a, const uint32_t* __restrict__ streamed) {
  __shared__ uint32_t mult[2 * TILE_BITS][2 * TILE_BITS];  // edge multiplicities: tile bits, then fixed qubits
  __shared__ uint16_t tt[TILE_BITS][PLANES];
  __shared__ uint32_t used;
  const uint32_t slot = blockIdx.x >> 1, kind = blockIdx.x & 1, tid = threadIdx.x;
  const aleph_b200_qaoa_set cs = a.sets[streamed[slot]];
  const uint32_t n = cs.num_qubits, m = cs.num_edges;
  for (uint32_t i = tid; i < 4 * TILE_BITS * TILE_BITS; i += PREP_THREADS) (&mult[0][0])[i] = 0;
  if (tid == 0) used = 1;
  __syncthreads();
  for (uint32_t e = tid; e < m; e += PREP_THREADS) {
    uint32_t u = place(kind, n, a.edges[2 * (cs.edge_offset + e)]), v = place(kind, n, a.edges[2 * (cs.edge_offset + e) + 1]);
    u = u < 16 ? u : u - 16 + TILE_BITS;
    v = v < 16 ? v : v - 16 + TILE_BITS;
    atomicAdd(&mult[u][v], 1u);
    atomicAdd(&mult[v][u], 1u);
  }
  __syncthreads();
  Masks& M = a.masks[2 * slot + kind];
  for (uint32_t i = tid; i < TILE_BITS * PLANES; i += PREP_THREADS) {
    const uint32_t q = i / PLANES, b = i % PLANES;
    uint32_t x = 0, y = 0, z = 0;
    for (uint32_t f = 0; f < TILE_BITS; ++f) {
      x |= ((mult[q][TILE_BITS + f] >> b) & 1u) << f;
      y |= ((mult[TILE_BITS + q][TILE_BITS + f] >> b) & 1u) << f;
      z |= ((mult[q][f] >> b) & 1u) << f;
    }
    M.cross[q][b] = (uint16_t)x;
    M.fixed[q][b] = (uint16_t)y;
    tt[q][b] = (uint16_t)z;
    if (x | y | z) atomicMax(&used, b + 1);
  }
  __syncthreads();
  const uint32_t np = used;
  if (tid == 0) M.planes = np;
  uint8_t* T = a.tables + (2 * (size_t)slot + kind) * TILE;
  for (uint32_t z = tid; z < TILE; z += PREP_THREADS) {
    uint32_t c = 0;
    for (uint32_t b = 0; b < np; ++b)
#pragma unroll
      for (uint32_t q = 0; q < TILE_BITS; ++q)
        if ((z >> q) & 1u) c += (uint32_t)__popc(tt[q][b] & ~z) << b;
    T[z] = (uint8_t)c;
  }
  if (kind == 0) {
    const double* gam = a.angles + (size_t)streamed[slot] * 2 * a.p;
    V2<Real>* ph = (V2<Real>*)a.phases + (size_t)slot * a.p * (MAX_EDGES + 1);
    for (uint32_t i = tid; i < a.p * (m + 1); i += PREP_THREADS) {
      const uint32_t l = i / (m + 1), k = i % (m + 1);
      double sn, cn;
      sincos(-gam[l] * ((double)m - 2.0 * (double)k), &sn, &cn);
      ph[(size_t)l * (MAX_EDGES + 1) + k] = mk<Real>((Real)cn, (Real)sn);
    }
  }
}

// <C> of the streamed sets: their last pass's partial sums, in item order.
__global__ void __launch_bounds__(32) total_kernel(Args a) {
  const QaoaGroup g = a.groups[blockIdx.x];
  if (g.pass != a.p) return;  // small sets (kQaoaSmall) write their result themselves
  double s = 0.0;
  const uint32_t items = (g.ntiles + g.tiles_per_item - 1) / g.tiles_per_item;
  for (uint32_t i = threadIdx.x; i < items; i += 32) s += a.partials[g.part0 + i];
  for (int o = 16; o; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if (threadIdx.x == 0) a.out[g.set] = s;
}

template <typename Real>
struct Shared {
  V2<Real> S[TILE];
  V2<Real> ph[MAX_EDGES + 1];  // cost-layer phase by cut value
  double red[Cfg<Real>::THREADS / 32];
  Real rot[4];
  alignas(16) uint8_t cutT[TILE];  // filled by 16-byte copies
  uint8_t X0[2][128], X1[2][64];
  uint32_t ch[2];
  Masks masks;
  uint8_t eu[MAX_EDGES], ev[MAX_EDGES];
  uint32_t item[2], group[2];
  int ok;
};

template <typename Real>
__global__ void __launch_bounds__(Cfg<Real>::THREADS, Cfg<Real>::CTAS_PER_SM) sweep_kernel(Args a) {
  constexpr int THREADS = Cfg<Real>::THREADS, WB = Cfg<Real>::WARP_BITS;
  constexpr bool AHEAD = sizeof(Real) == 8;
  constexpr int R1 = 5 + WB, REGS = TILE / THREADS;           // layout 1: registers from bit R1
  constexpr int G2 = 1 << WB, LOOPS = TILE / (32 * G2) >> WB;  // layout 2: registers from bit 5, LOOPS groups a warp
  extern __shared__ __align__(16) uint8_t qsm[];
  Shared<Real>& sh = *(Shared<Real>*)qsm;
  V2<Real>* S = sh.S;
  const uint32_t tid = threadIdx.x, lane = tid & 31u, w = tid >> 5;

  // warp 0: the next item and its group (the last one whose first item is not past it)
  auto fetch = [&](int at) {
    uint32_t idx = 0;
    if (lane == 0) idx = atomicAdd(a.counters, 1u);
    idx = __shfl_sync(0xffffffffu, idx, 0);
    uint32_t lo = 0, hi = a.n_groups;  // groups[lo].first_item <= idx < groups[hi].first_item
    if (idx < a.n_items)
      while (hi - lo > 1) {
        const uint32_t step = (hi - lo + 31) / 32;
        const uint32_t g = lo + step * (lane + 1);
        const bool past = g >= hi || a.groups[g].first_item > idx;
        const uint32_t first = __ffs(__ballot_sync(0xffffffffu, past)) - 1;  // lane 31 is always past
        hi = min(hi, lo + step * (first + 1));
        lo += step * first;
      }
    if (lane == 0) {
      sh.item[at] = idx;
      sh.group[at] = lo;
    }
  };
  if (w == 0) fetch(0);
  for (int at = 0;; at ^= 1) {
    __syncthreads();
    const uint32_t idx = sh.item[at];
    if (idx >= a.n_items) break;
    const QaoaGroup g = a.groups[sh.group[at]];
    const aleph_b200_qaoa_set cs = a.sets[g.set];
    const uint32_t n = cs.num_qubits, m = cs.num_edges;
    const double* bet = a.angles + (size_t)g.set * 2 * a.p + a.p;
    const Real amp0 = (Real)rsqrt((double)(1ull << n));  // |+>^n
    double acc = 0.0;

    if (g.pass == kQaoaSmall) {
      // ---- whole state in shared memory ----
      if (w == 0) fetch(at ^ 1);
      const double* gam = bet - a.p;
      for (uint32_t e = tid; e < m; e += THREADS) {
        sh.eu[e] = (uint8_t)a.edges[2 * (cs.edge_offset + e)];
        sh.ev[e] = (uint8_t)a.edges[2 * (cs.edge_offset + e) + 1];
      }
      __syncthreads();
      const uint32_t L = 1u << n;
      for (uint32_t z = tid; z < L; z += THREADS) {
        uint32_t c = 0;
        for (uint32_t e = 0; e < m; ++e) c += ((z >> sh.eu[e]) ^ (z >> sh.ev[e])) & 1u;
        sh.cutT[z] = (uint8_t)c;
      }
      for (uint32_t i = tid; i < L; i += THREADS) S[i] = mk<Real>(amp0, (Real)0);
      for (uint32_t l = 0; l < a.p; ++l) {
        __syncthreads();
        for (uint32_t k = tid; k <= m; k += THREADS) {  // ph[k] = exp(-i gamma (m - 2k))
          double sn, cn;
          sincos(-gam[l] * ((double)m - 2.0 * (double)k), &sn, &cn);
          sh.ph[k] = mk<Real>((Real)cn, (Real)sn);
        }
        __syncthreads();
        for (uint32_t i = tid; i < L; i += THREADS) S[i] = cmul<Real>(sh.ph[sh.cutT[i]], S[i]);
        double sb, cb;
        sincos(bet[l], &sb, &cb);
        mixer_range<Real>(S, L, 0, n, (Real)cb, (Real)sb);
      }
      for (uint32_t i = tid; i < L; i += THREADS) {
        const double x = (double)S[i].x, y = (double)S[i].y;
        acc += (x * x + y * y) * (double)sh.cutT[i];
      }
      const double tot = block_sum<THREADS / 32>(acc, sh.red);
      if (tid == 0) a.out[g.set] = tot;
      continue;
    }

    // ---- tiles [t0, t1) of one pass of a streamed set ----
    const uint32_t kind = g.pass & 1u, k = g.pass;
    const uint32_t chunk = idx - g.first_item;
    const uint32_t t0 = chunk * g.tiles_per_item, t1 = min(g.ntiles, t0 + g.tiles_per_item);
    const bool pre = k > 0, last = k == a.p;
    const uint32_t c = 2 * TILE_BITS - n, lowm = (1u << c) - 1;
    const uint32_t mix = kind == 0 ? TILE - 1 : (TILE - 1) & ~lowm;  // tile bits mixed by this pass
    const uint32_t ends = pre ? mix : 0;                             // ... for the layer that ends in it
    V2<Real>* X = (V2<Real>*)a.scratch + g.state_off;
    // state offset of tile amplitude i (offsets fit in 32 bits: n <= 26)
    auto at_tile = [&](uint32_t t, uint32_t i) -> uint32_t {
      return kind == 0 ? (t << TILE_BITS) | i : (i & lowm) | t << c | (i >> c) << TILE_BITS;
    };
    // offset of register bit j of layout 1; the offsets of a thread's registers are
    // walked in Gray-code order (16 or 32 of them kept were spilled)
    static_assert(REGS == 1 << (8 - WB), "layout 1 has the bits from R1 up in registers");
    uint32_t step[8 - WB];
#pragma unroll
    for (int j = 0; j < 8 - WB; ++j) step[j] = at_tile(0, 1u << (R1 + j));
    auto each_register = [&](uint32_t t, auto&& f) {  // f(r, its state offset)
      uint32_t off = at_tile(t, tid);
#pragma unroll
      for (int q = 0; q < REGS; ++q) {
        if (q) off ^= step[(q & 1) ? 0 : (q & 2) ? 1 : (q & 4) ? 2 : (q & 8) ? 3 : 7 - WB];
        f(q ^ (q >> 1), off);
      }
    };
    if (tid == 0) {  // Rx of the finishing and of the starting layer (in shared memory: registers are short)
      double sn, cn;
      if (pre) {
        sincos(bet[k - 1], &sn, &cn);
        sh.rot[0] = (Real)cn;
        sh.rot[1] = (Real)sn;
      }
      if (!last) {
        sincos(bet[k], &sn, &cn);
        sh.rot[2] = (Real)cn;
        sh.rot[3] = (Real)sn;
      }
    }
    {
      const uint4* T = (const uint4*)(a.tables + (2 * (size_t)g.slot + kind) * TILE);
      for (uint32_t i = tid; i < TILE / 16; i += THREADS) ((uint4*)sh.cutT)[i] = T[i];
      const uint32_t* M = (const uint32_t*)(a.masks + 2 * (size_t)g.slot + kind);
      for (uint32_t i = tid; i < sizeof(Masks) / 4; i += THREADS) ((uint32_t*)&sh.masks)[i] = M[i];
      if (!last) {
        const V2<Real>* ph = (const V2<Real>*)a.phases + ((size_t)g.slot * a.p + k) * (MAX_EDGES + 1);
        for (uint32_t i = tid; i <= m; i += THREADS) sh.ph[i] = ph[i];
      }
    }
    if (tid == 0) {  // what this item reads (or overwrites) is complete
      sh.ok = 1;
      volatile uint32_t* cnt = a.counters + g.wait_idx;
      if (g.wait_val && *cnt < g.wait_val) {
        const uint64_t start = globaltimer_ns();
        for (uint32_t spin = 1; *cnt < g.wait_val; ++spin) {
          __nanosleep(64);
          if ((spin & 63) == 0 && (*(volatile uint32_t*)(a.counters + 1) || globaltimer_ns() - start > 10 * kWaitDeadlineNs)) {
            sh.ok = 0;
            break;
          }
        }
      }
      __threadfence();
    }
    __syncthreads();
    if (!sh.ok) {
      if (tid == 0) {
        atomicExch(a.counters + 1, 1u);
        atomicExch(a.error, ALEPH_B200_DEVICE_FAILURE);
      }
      return;
    }
    if (w == 0) fetch(at ^ 1);
    // the cut contributions of a tile's fixed qubits (bits of t)
    auto tile_tables = [&](uint32_t t, int b) {
      const uint32_t np = sh.masks.planes;
      if (tid < 192) {
        const uint32_t first = tid < 128 ? 0u : 7u, v = tid < 128 ? tid : tid - 128, bits = tid < 128 ? 7u : 6u;
        uint32_t x = 0;
        for (uint32_t pl = 0; pl < np; ++pl)
          for (uint32_t q = 0; q < bits; ++q) {
            const uint32_t f = sh.masks.cross[first + q][pl];
            x += (uint32_t)__popc(f & (((v >> q) & 1u) ? ~t : t)) << pl;
          }
        if (tid < 128) sh.X0[b][v] = (uint8_t)x;
        else sh.X1[b][v] = (uint8_t)x;
      } else if (tid == 192) {
        uint32_t x = 0;
        for (uint32_t pl = 0; pl < np; ++pl)
          for (uint32_t f = 0; f < TILE_BITS; ++f)
            if ((t >> f) & 1u) x += (uint32_t)__popc(sh.masks.fixed[f][pl] & ~t) << pl;
        sh.ch[b] = x;
      }
    };
    V2<Real> v[REGS];
    // AHEAD (FP64, one CTA per SM: nothing else hides the loads): the next tile's
    // amplitudes come straight into shared memory. In layout 1 a thread has slots of its
    // own there, free as soon as it has read them.
    auto fetch_tile = [&](uint32_t t) {
      each_register(t, [&](int r, uint32_t off) { copy16_async(S + (tid | (uint32_t)r << R1), X + off); });
    };
    if (AHEAD && pre) fetch_tile(t0);
    for (uint32_t t = t0; t < t1; ++t) {
      const int b = t & 1;
      tile_tables(t, b);
      if (!pre) {
#pragma unroll
        for (int r = 0; r < REGS; ++r) v[r] = mk<Real>(amp0, (Real)0);
      } else if constexpr (AHEAD) {
        copies_wait();
#pragma unroll
        for (int r = 0; r < REGS; ++r) v[r] = S[tid | (uint32_t)r << R1];
      } else {
        each_register(t, [&](int r, uint32_t off) { v[r] = ld_amp<Real>(X + off); });
      }
      rx_regs<Real, REGS>(v, ends >> R1, sh.rot[0], sh.rot[1]);
      rx_lanes<Real, REGS>(v, ends & 0x1fu, sh.rot[0], sh.rot[1]);
      if (!AHEAD) __syncthreads();  // the previous tile's reads are done
#pragma unroll
      for (int r = 0; r < REGS; ++r) S[tid | (uint32_t)r << R1] = v[r];
      __syncthreads();  // the tile and its tables are visible
      // layout 2: lane = tile bits 0..4, register = the next WB, warp and loop = the rest
      const uint32_t ch = sh.ch[b];
#pragma unroll
      for (int j = 0; j < LOOPS; ++j) {
        const uint32_t hi = (w | (uint32_t)j << WB) << R1;
        V2<Real> u[G2];
#pragma unroll
        for (int r = 0; r < G2; ++r) u[r] = S[hi | (uint32_t)r << 5 | lane];
        static_assert(!AHEAD || LOOPS == 1, "a tile read ahead takes the place of one that is in registers");
        if (AHEAD && last) {
          __syncthreads();
          if (t + 1 < t1) fetch_tile(t + 1);
        }
        rx_regs<Real, G2>(u, (ends >> 5) & (G2 - 1), sh.rot[0], sh.rot[1]);
        auto cut = [&](int r) -> uint32_t {
          const uint32_t i = hi | (uint32_t)r << 5 | lane;
          return sh.cutT[i] + ch + sh.X0[b][i & 127] + sh.X1[b][i >> 7];
        };
        if (last) {
#pragma unroll
          for (int r = 0; r < G2; ++r) {
            const double x = (double)u[r].x, y = (double)u[r].y;
            acc += (x * x + y * y) * (double)cut(r);
          }
        } else {
#pragma unroll
          for (int r = 0; r < G2; ++r) {
            const V2<Real> f = sh.ph[cut(r)];
            u[r] = cmul<Real>(f, u[r]);
          }
          rx_regs<Real, G2>(u, (mix >> 5) & (G2 - 1), sh.rot[2], sh.rot[3]);
          rx_lanes<Real, G2>(u, mix & 0x1fu, sh.rot[2], sh.rot[3]);
#pragma unroll
          for (int r = 0; r < G2; ++r) S[hi | (uint32_t)r << 5 | lane] = u[r];
        }
      }
      if (!last) {
        __syncthreads();
#pragma unroll
        for (int r = 0; r < REGS; ++r) v[r] = S[tid | (uint32_t)r << R1];
        if (AHEAD && pre && t + 1 < t1) {
          __syncwarp();  // the reads above come first
          fetch_tile(t + 1);
        }
        rx_regs<Real, REGS>(v, mix >> R1, sh.rot[2], sh.rot[3]);
        each_register(t, [&](int r, uint32_t off) { st_amp<Real>(X + off, v[r]); });
      }
    }
    if (last) {
      const double tot = block_sum<THREADS / 32>(acc, sh.red);
      if (tid == 0) a.partials[g.part0 + chunk] = tot;
    }
    __syncthreads();
    if (tid == 0) {
      __threadfence();
      atomicAdd(a.counters + g.done_idx, 1u);
      if (last) atomicAdd(a.counters + g.wave_idx, 1u);
    }
  }
}

}  // namespace qaoa

uint32_t qaoa_smem_max_n(int precision) {
  return precision == ALEPH_B200_F64 ? (uint32_t)qaoa::Cfg<double>::SMEM_N : (uint32_t)qaoa::Cfg<float>::SMEM_N;
}

int qaoa_ctas_per_sm(int precision) {
  return precision == ALEPH_B200_F64 ? qaoa::Cfg<double>::CTAS_PER_SM : qaoa::Cfg<float>::CTAS_PER_SM;
}

QaoaSizes qaoa_sizes(int precision, uint32_t n_streamed, uint32_t p) {
  const size_t amp = precision == ALEPH_B200_F64 ? sizeof(double2) : sizeof(float2);
  QaoaSizes z;
  z.tables = (size_t)n_streamed * 2 * qaoa::TILE;
  z.masks = (size_t)n_streamed * 2 * sizeof(qaoa::Masks);
  z.phases = (size_t)n_streamed * p * (qaoa::MAX_EDGES + 1) * amp;
  return z;
}

template <typename Real>
static cudaError_t launch_qaoa_t(const qaoa::Args& a, const uint32_t* streamed, uint32_t n_streamed, int grid,
                                 cudaStream_t s) {
  constexpr int bytes = (int)sizeof(qaoa::Shared<Real>);
  static uint64_t attr_devices = 0;  // devices with the shared-memory opt-in
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev >= 64 || !((attr_devices >> dev) & 1)) {
    e = cudaFuncSetAttribute(qaoa::sweep_kernel<Real>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return e;
    if (dev < 64) attr_devices |= 1ull << dev;
  }
  if (n_streamed) qaoa::prep_kernel<Real><<<2 * n_streamed, qaoa::PREP_THREADS, 0, s>>>(a, streamed);
  qaoa::sweep_kernel<Real><<<grid, qaoa::Cfg<Real>::THREADS, bytes, s>>>(a);
  if (n_streamed) qaoa::total_kernel<<<a.n_groups, 32, 0, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_qaoa_sweep(int precision, const QaoaLaunch& q, int grid, cudaStream_t s) {
  qaoa::Args a;
  a.sets = q.sets;
  a.edges = q.edges;
  a.angles = q.angles;
  a.groups = q.groups;
  a.counters = q.counters;
  a.out = q.out;
  a.scratch = q.state;
  a.tables = (uint8_t*)q.tables;
  a.masks = (qaoa::Masks*)q.masks;
  a.phases = q.phases;
  a.partials = q.partials;
  a.n_groups = q.n_groups;
  a.n_items = q.n_items;
  a.p = q.p;
  a.error = q.error;
  return precision == ALEPH_B200_F64 ? launch_qaoa_t<double>(a, q.streamed, q.n_streamed, grid, s)
                                     : launch_qaoa_t<float>(a, q.streamed, q.n_streamed, grid, s);
}

}  // namespace ab
