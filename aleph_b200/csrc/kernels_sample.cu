// kernels_sample.cu — on-device shot sampling with the reference's exact
// seed-to-outcome mappings, given the same variates.
//
// ALIAS (the reference's shots >= 2 path, crates/aleph-sv/src/measure.rs:109-124):
//   probabilities p_i = re*re + im*im rounded exactly like the CPU (no FMA),
//   Vose's table built by AliasTable::build (crates/aleph-sv/src/sampling.rs:104-167)
//   with the same LIFO stack discipline and the same floating-point operation
//   order, so the table is bit-identical. The build's chain of dependent
//   additions is evaluated in parallel chunks, exactly (see ALIAS below).
//   Draw: index = (word >> 32) & (N-1), u = (u32)word * 2^-32,
//   u < prob[i] ? i : alias[i] (sampling.rs:179-197).
// CUMULATIVE (the reference's shots <= 1 path, sampling.rs:59-91): the
//   inverse CDF of the sequential left-to-right prefix sum with strict
//   `target < cumulative`, zero bins skipped, last positive bin as fallback.
//   Shots are resolved by a warp each on a two-level prefix (tree block sums,
//   then the block added in order); a shot whose target lies within the
//   rounding bound of a bin boundary is re-resolved against the exact
//   sequential running sum (for n <= 28), so the outcome equals the
//   sequential CPU result. The running sum, too, is evaluated in parallel.
//
// Measured on B200: alias table and 1024 shots of a scrambled n = 22 FP64 state 0.71
// ms (234 ms with the chain on one lane); 4096 cumulative shots at n = 26 FP32 0.76
// ms (458 ms with the sum on one lane). Parts of the alias chain that no chunk covers
// run step by step, at 48 ns a step: product states (wide jumps of V) take 12 ms at
// n = 22, and states with half of the basis at one probability (every sum on a
// binade's edge) run wholly so, 0.2 s at n = 22.

#include <cmath>

#include "common.cuh"

namespace ab {

constexpr uint32_t CUM_BLOCK = 2048;  // amplitudes per level-1 CDF block
constexpr uint32_t EXACT_MAX_N = kExactCumulativeMaxN;  // exact re-resolution of ambiguous shots up to this n

template <typename Real>
__device__ __forceinline__ double prob_exact(const V2<Real>* amps, uint64_t i) {
  const V2<Real> a = ld_amp<Real>(amps + i);
  const double x = (double)a.x, y = (double)a.y;
  return __dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y));
}

// ------------------------------------------------------------------ ALIAS ----
// Vose's loop (AliasTable::build) is one chain of dependent FP64 steps. With
// LIFO stacks the element pushed in one step is popped in the next, so the
// chain has a single state V, the value of the element in hand, and a fixed
// operand order per stack: smalls a_0, a_1, ... and larges b_0, b_1, ... from
// the stack tops. V starts as b_0; a step is
//     V >= 1: pop a_i,  alias[a_i] = current large,          V = fl(V + a_i) - 1
//     V <  1: pop b_j+1, alias[b_j] = b_j+1, threshold V,    V = fl(V + b_j+1) - 1
// One lane needs about 57 ns a step (two dependent FP64 adds, a compare and
// selects): 234 ms for a scrambled n = 22 state. The table must match it bit
// for bit, and it is built in parallel as follows.
//
// * Order. In exact arithmetic V = 1 + E_j - D_i with D_i = sum of the deficits
//   1 - a of the smalls popped before a_i and E_j = sum of the surpluses b - 1 up
//   to b_j, so the pops are the merge of the two sorted sequences D and E (small
//   first on ties). D and E are prefix sums in 64.64 fixed point; the merge is
//   cut into chunks of about CH steps by binary search (merge path).
// * Rounding. fl(V + v) - 1 depends on V only through its binade and its low
//   bits: with S = fl(V + v) in [2^b, 2^(b+1)), moving V by a multiple D of
//   2^(b+1) units (unit = 2^-52) moves S by exactly D (ties to even included),
//   as long as S stays in the binade. S >= 2 is also the decision V' >= 1. So a
//   chunk is run once for each of 32 residues of its start value, one per lane,
//   around the value that the prefix sums predict; the true start (which differs
//   by the accumulated rounding, some 1e3 units) has one of these residues, and
//   the chunk's true end is that lane's end plus the difference, provided the
//   difference is smaller than the least distance of any S to a binade
//   boundary (the chunk's margin). Chunks start where V is large (its grid is
//   coarse there), so that 32 residues cover the binades of the whole chunk.
// * Composition. 64 chunks compose to one of the same form; one warp then steps
//   from group to group, checking each condition, and runs what fails one (about
//   one chunk in 1e8 for a scrambled state, chunks in which V jumps by more than
//   five binades, and the chain's end) step by step.
// * A last kernel replays every chunk from its true start and writes the table.
using u128 = unsigned __int128;

struct AliasScratch {
  double* prob;       // N: scaled probabilities, then the table thresholds
  uint32_t* alias;    // N
  uint32_t* idx;      // N: basis states in pop order, the m smalls, then the k larges
  double* val;        // N: their scaled values (null: step by step only, see sample_scratch_bytes)
  u128* pre;          // N: D_i of small i (deficits before it), E_j of large j (surpluses up to it)
  // per partition block: smalls, deficits, surpluses (then what pops before the block), norm partials
  uint32_t* bcount;
  u128* bdef;
  u128* bsur;
  double* normsum;    // 2 per block: [sum p, non-finite]
  uint32_t* totals;   // smalls m, larges k, smalls popped, index of the last current large
  // chunks of the merged order (nc + 1 cuts)
  uint32_t *ci, *cj;  // smalls popped and current large at the cut
  double *cbase, *cunit;  // lane r starts at base + r * unit
  long long* cmargin;     // least distance to a binade boundary, units of 2^-52 (<= 0: not usable)
  int* cmax;              // exponent of the largest S
  double* cend;           // 32 per chunk: end values
  double* cstart;         // true start value
  uint8_t* cflag;         // 1: replay from cstart (0: its steps were run one by one)
  // groups of CGROUP chunks, the same form
  long long* gmargin;
  double* gend;
  double* gstart;
  uint8_t* gflag;
};

constexpr uint32_t PART_B = 1024;  // elements per partition block
constexpr uint32_t CH = 256;       // merged steps per chunk: a cut lies within the next 32 steps
constexpr uint32_t CH_MAX = CH + 31;
constexpr uint32_t CGROUP = 64;    // chunks per group
constexpr double kUnits = 4503599627370496.0;  // 2^52

// Chunks of a chain over n elements: the last two chunks' worth of steps stay
// with the step-by-step walk, which ends where a stack runs empty.
static inline uint32_t alias_chunks(uint64_t len) { return len > 4 * CH ? (uint32_t)((len - 1 - 2 * CH) / CH) : 0u; }

__device__ __forceinline__ u128 fx_deficit(double a) {  // 1 - a for a in [0, 1), 64 fraction bits
  return ((u128)1 << 64) - (u128)__double2ull_rd(a * 18446744073709551616.0);
}
__device__ __forceinline__ u128 fx_surplus(double b) {  // b - 1 for b >= 1
  const double x = b - 1.0, f = floor(x);
  return ((u128)__double2ull_rd(f) << 64) + (u128)__double2ull_rd((x - f) * 18446744073709551616.0);
}
__device__ __forceinline__ u128 shfl_up_u128(u128 v, int o) {
  const unsigned long long lo = __shfl_up_sync(0xffffffffu, (unsigned long long)v, o);
  const unsigned long long hi = __shfl_up_sync(0xffffffffu, (unsigned long long)(v >> 64), o);
  return ((u128)hi << 64) | lo;
}
// Inclusive prefix over a block of 1024 threads (warp_tot: 32 slots of shared memory).
template <typename T, typename Up>
__device__ __forceinline__ T block_scan_1024(T v, T* warp_tot, Up&& up) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const T x = up(v, o);
    if (lane >= o) v += x;
  }
  if (lane == 31) warp_tot[w] = v;
  __syncthreads();
  if (w == 0) {
    T t = warp_tot[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const T x = up(t, o);
      if (lane >= o) t += x;
    }
    warp_tot[lane] = t;
  }
  __syncthreads();
  if (w) v += warp_tot[w - 1];
  return v;
}
__device__ __forceinline__ u128 block_scan_u128(u128 v, u128* tot) {
  return block_scan_1024<u128>(v, tot, [](u128 x, int o) { return shfl_up_u128(x, o); });
}
__device__ __forceinline__ uint32_t block_scan_u32(uint32_t v, uint32_t* tot) {
  return block_scan_1024<uint32_t>(v, tot, [](uint32_t x, int o) { return __shfl_up_sync(0xffffffffu, x, o); });
}

// Norm check of validate_state (sampling.rs:36-57): sets status on failure.
__device__ __forceinline__ void check_norm(double total, double bad, double tol, int32_t* status) {
  if (bad > 0.0 || !isfinite(total) || fabs(total - 1.0) > tol) status[0] = ALEPH_B200_INVALID_STATE;
}

// Thread t of block b takes element b * PART_B + (PART_B - 1 - t): ascending
// threads are the pop order (stacks are filled in ascending index order).
__device__ __forceinline__ uint64_t part_element() { return (uint64_t)blockIdx.x * PART_B + (PART_B - 1 - threadIdx.x); }

// Scaled values, per-block small counts, deficit / surplus sums and norm partials.
template <typename Real>
__global__ void __launch_bounds__(PART_B) alias_scale_kernel(const V2<Real>* __restrict__ amps, uint64_t len,
                                                             AliasScratch s) {
  __shared__ uint32_t cs[32];
  __shared__ u128 sd[32], se[32];
  __shared__ double ns[32], nb[32];
  const double nf = (double)len;
  const uint64_t i = part_element();
  bool small = false;
  u128 d = 0, e = 0;
  double psum = 0.0, bad = 0.0;
  if (i < len) {
    const double p = prob_exact<Real>(amps, i);
    if (!isfinite(p)) bad = 1.0;
    else psum = p;
    const double sc = __dmul_rn(nf, p);
    s.prob[i] = sc;
    small = sc < 1.0;
    if (small) d = fx_deficit(sc);
    else e = fx_surplus(sc);
  }
  const unsigned bs = __ballot_sync(0xffffffffu, small);
  for (int o = 16; o; o >>= 1) {
    psum += __shfl_down_sync(0xffffffffu, psum, o);
    bad += __shfl_down_sync(0xffffffffu, bad, o);
    d += ((u128)__shfl_down_sync(0xffffffffu, (unsigned long long)(d >> 64), o) << 64) +
         (u128)__shfl_down_sync(0xffffffffu, (unsigned long long)d, o);
    e += ((u128)__shfl_down_sync(0xffffffffu, (unsigned long long)(e >> 64), o) << 64) +
         (u128)__shfl_down_sync(0xffffffffu, (unsigned long long)e, o);
  }
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) {
    cs[w] = __popc(bs);
    ns[w] = psum;
    nb[w] = bad;
    sd[w] = d;
    se[w] = e;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t a = 0;
    double x = 0.0, y = 0.0;
    u128 dd = 0, ee = 0;
    for (int k = (int)(PART_B / 32) - 1; k >= 0; --k) {  // ascending element order
      a += cs[k];
      x += ns[k];
      y += nb[k];
      dd += sd[k];
      ee += se[k];
    }
    s.bcount[blockIdx.x] = a;
    s.bdef[blockIdx.x] = dd;
    s.bsur[blockIdx.x] = ee;
    s.normsum[2 * blockIdx.x] = x;
    s.normsum[2 * blockIdx.x + 1] = y;
  }
}

// What pops before each block (blocks pop from the last to the first): counts
// of smalls, deficits and surpluses; the totals and the norm with its check. One
// CTA; a thread takes a contiguous range of blocks. (One thread for all of them was
// 0.7 ms at n = 22.)
__global__ void __launch_bounds__(1024) alias_offsets_kernel(AliasScratch s, uint64_t len, uint32_t nblocks,
                                                             double tol, int32_t* status) {
  __shared__ u128 tot[32];
  __shared__ uint32_t tot32[32];
  __shared__ double red[2][32];
  const uint32_t per = (nblocks + 1023) / 1024;
  const uint32_t q0 = min(nblocks, threadIdx.x * per), q1 = min(nblocks, q0 + per);
  uint32_t c = 0;
  u128 d = 0, e = 0;
  double x = 0.0, y = 0.0;
  for (uint32_t q = q0; q < q1; ++q) {
    const uint32_t b = nblocks - 1 - q;
    c += s.bcount[b];
    d += s.bdef[b];
    e += s.bsur[b];
    x += s.normsum[2 * b];
    y += s.normsum[2 * b + 1];
  }
  const uint32_t ci = block_scan_u32(c, tot32);
  const u128 di = block_scan_u128(d, tot);
  __syncthreads();  // tot is reused
  const u128 ei = block_scan_u128(e, tot);
  uint32_t rc = ci - c;
  u128 rd = di - d, re = ei - e;
  for (uint32_t q = q0; q < q1; ++q) {
    const uint32_t b = nblocks - 1 - q;
    const uint32_t cb = s.bcount[b];
    const u128 db = s.bdef[b], eb = s.bsur[b];
    s.bcount[b] = rc;
    s.bdef[b] = rd;
    s.bsur[b] = re;
    rc += cb;
    rd += db;
    re += eb;
  }
  for (int o = 16; o; o >>= 1) {
    x += __shfl_down_sync(0xffffffffu, x, o);
    y += __shfl_down_sync(0xffffffffu, y, o);
  }
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = x;
    red[1][threadIdx.x >> 5] = y;
  }
  if (threadIdx.x == 1023) {
    s.totals[0] = ci;
    s.totals[1] = (uint32_t)(len - ci);
    s.totals[2] = 0;
    s.totals[3] = 0;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0.0, b = 0.0;
    for (int w = 0; w < 32; ++w) {
      a += red[0][w];
      b += red[1][w];
    }
    check_norm(a, b, tol, status);
  }
}

// Values, basis states and prefix sums in pop order.
__global__ void __launch_bounds__(PART_B) alias_partition_kernel(uint64_t len, AliasScratch s, const int32_t* status) {
  __shared__ u128 tot[32];
  __shared__ uint32_t tot32[32];
  if (status[0] != 0) return;  // not a normalised state: uniform over the grid
  const uint64_t i = part_element();
  const bool valid = i < len;
  const double sc = valid ? s.prob[i] : 0.0;
  const bool small = valid && sc < 1.0;
  const u128 d = small ? fx_deficit(sc) : 0, e = valid && !small ? fx_surplus(sc) : 0;
  const uint32_t rank = block_scan_u32(small ? 1u : 0u, tot32);  // smalls up to this element, in pop order
  const u128 di = block_scan_u128(d, tot);
  __syncthreads();
  const u128 ei = block_scan_u128(e, tot);
  if (!valid) return;
  // elements of this block that pop before this one: threadIdx.x less the padding of the last block
  const uint64_t top = ((uint64_t)blockIdx.x + 1) * PART_B;
  const uint32_t pad = top > len ? (uint32_t)(top - len) : 0u;
  const uint32_t m = s.totals[0], sb = s.bcount[blockIdx.x];
  const uint64_t popped = len > top ? len - top : 0;  // elements of later blocks
  uint64_t at;
  if (small) at = sb + rank - 1;
  else at = m + (popped - sb) + (threadIdx.x - pad - rank);
  s.idx[at] = (uint32_t)i;
  if (!s.val) return;
  s.val[at] = sc;
  s.pre[at] = small ? s.bdef[blockIdx.x] + di - d : s.bsur[blockIdx.x] + ei;
}

// Smalls among the first t pops of the merged order; lo..hi brackets the answer.
__device__ __forceinline__ uint32_t merge_smalls(const AliasScratch& s, uint32_t m, uint32_t t, uint32_t lo, uint32_t hi) {
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    // small mid against large t - mid, whose key is E of the large before it
    if (s.pre[mid] <= s.pre[(uint64_t)m + (t - 1 - mid)]) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// The exponent of x >= 2^-1022 (unbiased).
__device__ __forceinline__ int exponent_of(double x) {
  return (int)((__double_as_longlong(x) >> 52) & 0x7ff) - 1023;
}
__device__ __forceinline__ double pow2(int e) { return __longlong_as_double((long long)(e + 1023) << 52); }

// Cut c lies within 32 steps from c * CH, where the predicted V is largest.
// One warp per cut, a lane per candidate.
__global__ void __launch_bounds__(128) alias_cuts_kernel(AliasScratch s, uint32_t nc, const int32_t* status) {
  const uint32_t c = blockIdx.x * 4 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  const uint32_t m = s.totals[0], k = s.totals[1];
  if (c > nc || status[0] != 0 || m == 0 || k == 0) return;
  const uint32_t t0 = c * CH, nl = k - 1;
  uint32_t i0 = 0;
  if (lane == 0) i0 = merge_smalls(s, m, t0, t0 > nl ? t0 - nl : 0u, min(t0, m));
  i0 = __shfl_sync(0xffffffffu, i0, 0);
  const uint32_t t = c == 0 ? 0u : t0 + lane;
  const uint32_t i = merge_smalls(s, m, t, max(i0, t > nl ? t - nl : 0u), min(min(t, m), i0 + (t - t0)));
  const uint32_t j = t - i;
  // V = 1 + E_j - D_i (D of one small past the last: the running total; such cuts are never used)
  const __int128 x = (__int128)s.pre[(uint64_t)m + j] - (__int128)(i < m ? s.pre[i] : s.pre[m - 1]);
  double V = 1.0 + ((double)(long long)(x >> 64) + (double)(unsigned long long)x * 0x1p-64);
  if (!(V > 0.0)) V = 0.0;
  double best = V;
  for (int o = 16; o; o >>= 1) best = fmax(best, __shfl_xor_sync(0xffffffffu, best, o));
  const unsigned who = __ballot_sync(0xffffffffu, V == best);
  if (lane != __ffs(who) - 1) return;
  int g = exponent_of(V + 1.0);  // V is a multiple of ulp(V + 1) after a step
  if (c == 0) {
    V = s.val[m];  // the first large itself
    g = exponent_of(V);
  }
  const double unit = pow2(g - 52);
  s.ci[c] = i;
  s.cj[c] = j;
  s.cbase[c] = floor(V / (32.0 * unit)) * (32.0 * unit);
  s.cunit[c] = unit;
  s.cflag[c] = 0;
}

// A chunk's operands in shared memory: its smalls, and the larges after its first one.
struct ChunkOps {
  double a[CH_MAX + 1], b[CH_MAX + 1];
};
__device__ __forceinline__ void stage_chunk(const AliasScratch& s, uint32_t m, uint32_t i0, uint32_t j0, uint32_t ns,
                                            uint32_t nl, ChunkOps& o) {
  const int lane = threadIdx.x & 31;
  for (uint32_t x = lane; x < ns; x += 32) o.a[x] = s.val[i0 + x];
  for (uint32_t x = lane; x < nl; x += 32) o.b[x] = s.val[(uint64_t)m + j0 + 1 + x];
  __syncwarp();
}

// One warp per chunk, one start residue per lane.
__global__ void __launch_bounds__(128) alias_spec_kernel(AliasScratch s, uint32_t nc, const int32_t* status) {
  __shared__ ChunkOps ops[4];
  const uint32_t c = blockIdx.x * 4 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  const uint32_t m = s.totals[0], k = s.totals[1];
  if (c >= nc || status[0] != 0 || m == 0 || k == 0) return;
  ChunkOps& o = ops[threadIdx.x >> 5];
  const uint32_t i0 = s.ci[c], j0 = s.cj[c];
  const uint32_t ns = s.ci[c + 1] - i0, nl = s.cj[c + 1] - j0, len = ns + nl;  // len <= CH_MAX
  stage_chunk(s, m, i0, j0, ns, nl, o);
  const double unit = s.cunit[c];
  double V = s.cbase[c] + (double)lane * unit;
  const double start = fmin(fabs(V - 1.0) * kUnits, 0x1p60);
  uint32_t near = 0xffffffffu;  // least distance of an S to its binade's ends, units of 2^-32 of the binade
  int smax = 0;
  uint32_t is = 0, il = 0;
  double va = o.a[0], vb = o.b[0];
  for (uint32_t t = 0; t < len; ++t) {
    const bool small = V >= 1.0;
    const double S = __dadd_rn(V, small ? va : vb);
    is += small ? 1u : 0u;
    il += small ? 0u : 1u;
    va = o.a[is];  // is, il <= len <= CH_MAX: inside the arrays whatever this lane decided
    vb = o.b[il];
    // the top 32 mantissa bits: S is at least that far above its binade's lower end
    // (which binds from 2 up; S >= 1 always) and at least the complement below the upper one
    const int hi = __double2hiint(S);
    const uint32_t top = __funnelshift_l((uint32_t)__double2loint(S), (uint32_t)hi, 12);
    near = min(near, hi >= 0x40000000 ? min(top, ~top) : ~top);
    smax = max(smax, hi);
    V = __dsub_rn(S, 1.0);
  }
  const bool ok = is == ns && il == nl;  // this lane popped what the prefix sums predicted
  // in units of 2^-52, rounded down: a binade spans 2^52 units or more
  long long margin = min((long long)start, (long long)near << 20);
  for (int x = 16; x; x >>= 1) {
    margin = min(margin, __shfl_xor_sync(0xffffffffu, margin, x));
    smax = max(smax, __shfl_xor_sync(0xffffffffu, smax, x));
  }
  const int g = (smax >> 20) - 1023;
  const bool all = __all_sync(0xffffffffu, ok);
  s.cend[(size_t)c * 32 + lane] = V;
  if (lane == 0) {
    // 32 residues of `unit` fix every rounding up to binade exponent_of(unit) + 52 + 4
    s.cmargin[c] = all && g <= exponent_of(unit) + 56 ? margin : 0;
    s.cmax[c] = g;
  }
}

// Where the true value V enters a chunk: the lane with its residue and the
// distance to that lane's start. False when the chunk does not cover V.
struct Entry {
  int lane;
  double shift;
};
// A group's chunks are entered within 2^28 units of their lanes, and so is the
// group itself, so that no chunk of a walked group is further than 2^30 off.
constexpr long long kMoved = 1ll << 28;
__device__ __forceinline__ bool enter_chunk(double V, double base, double unit, long long margin, long long max_moved,
                                            Entry* e, long long* left) {
  const int g = exponent_of(unit) + 52;
  if (g < 0 || g > 30) return false;
  const double q = (V - base) * pow2(52 - g);  // over unit, a power of two: exact, with V close to base on its grid
  if (!(fabs(q) < 0x1p30)) return false;
  const long long qi = (long long)q;
  if ((double)qi != q) return false;  // not on this chunk's grid
  const int r = (int)(qi & 31);
  const long long D = qi - r;
  const long long moved = (D < 0 ? -D : D) << g;  // units of 2^-52
  *left = margin - moved;
  if (*left <= 0 || moved > max_moved) return false;
  e->lane = r;
  e->shift = (double)D * unit;
  return true;
}

// One warp per group: lane r follows its chunk-0 start through the group's chunks.
__global__ void __launch_bounds__(128) alias_compose_kernel(AliasScratch s, uint32_t nc, uint32_t ng,
                                                            const int32_t* status) {
  const uint32_t q = blockIdx.x * 4 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (q >= ng || status[0] != 0 || s.totals[0] == 0 || s.totals[1] == 0) return;
  const uint32_t c0 = q * CGROUP, c1 = min(nc, c0 + CGROUP);
  const double unit0 = s.cunit[c0];
  double V = s.cbase[c0] + (double)lane * unit0;
  long long margin = 1ll << 60;
  int g = 0;
  bool ok = true;
#pragma unroll 4
  for (uint32_t c = c0; c < c1; ++c) {
    const double end = s.cend[(size_t)c * 32 + lane], base = s.cbase[c], unit = s.cunit[c];
    const long long cm = s.cmargin[c];
    g = max(g, s.cmax[c]);
    Entry e{0, 0.0};
    long long left = 0;
    if (!enter_chunk(V, base, unit, cm, kMoved, &e, &left)) ok = false;
    // a start that is D off takes the lane of another residue when D is no
    // multiple of this chunk's 32 units: up to 31 units further off
    margin = min(margin, left - (long long)(32.0 * unit * kUnits));
    V = __shfl_sync(0xffffffffu, end, e.lane) + e.shift;
  }
  for (int x = 16; x; x >>= 1) margin = min(margin, __shfl_xor_sync(0xffffffffu, margin, x));
  const bool all = __all_sync(0xffffffffu, ok);
  s.gend[(size_t)q * 32 + lane] = V;
  if (lane == 0) {
    s.gmargin[q] = all && g <= exponent_of(unit0) + 56 ? margin : 0;
    s.gflag[q] = 0;
  }
}

// The chain one step at a time (lane 0 out of shared memory; the warp stages
// operands and scatters the records): at most `steps` steps from (V, i, j).
// Returns false when the chain has ended: the stack it needs is empty.
// A step keeps V and one bit, which stack it popped; the indices of all steps
// follow from the bits. Each step pops one element, so as many steps as both
// buffers still hold need no bounds, and the operand behind a consumed one is in a
// register already. 48 ns a step (72 with indices and bounds kept per step; the
// two-stack loop in the reference's form takes 57).
constexpr uint32_t RAW = 1024;
struct RawShared {
  double a[RAW + 2], b[RAW + 2], v[RAW];
  uint32_t bits[RAW / 32];  // step n popped a small
};
__device__ bool raw_steps(const AliasScratch& s, uint32_t m, uint32_t k, RawShared& sh, double& V, uint32_t& i,
                          uint32_t& j, uint64_t steps) {
  const int lane = threadIdx.x & 31;
  for (;;) {
    if (V >= 1.0 ? i >= m : j + 1 >= k) return false;
    if (steps == 0) return true;
    const uint32_t ns = min(RAW, m - i), nl = min(RAW, k - 1 - j);
    if (s.val) {
      for (uint32_t x = lane; x < ns; x += 32) sh.a[x] = s.val[i + x];
      for (uint32_t x = lane; x < nl; x += 32) sh.b[x] = s.val[(uint64_t)m + j + 1 + x];
    } else {  // no values in pop order: what has not been popped still has its value in the table
      for (uint32_t x = lane; x < ns; x += 32) sh.a[x] = s.prob[s.idx[i + x]];
      for (uint32_t x = lane; x < nl; x += 32) sh.b[x] = s.prob[s.idx[(uint64_t)m + j + 1 + x]];
    }
    __syncwarp();
    uint32_t is = 0, n = 0;
    if (lane == 0) {
      const uint32_t lim = steps < RAW ? (uint32_t)steps : RAW;
      uint32_t word = 0;
      double va = sh.a[0], vb = sh.b[0], va1 = sh.a[1], vb1 = sh.b[1];
      while (n < lim) {
        uint32_t end = n + min(lim - n, min(ns - is, nl - (n - is)));
        if (end == n) {  // one buffer is spent: a step that pops the other
          if (V >= 1.0 ? is >= ns : n - is >= nl) break;
          end = n + 1;
        }
        end = min(end, (n | 31u) + 1);  // a word of bits at a time
#pragma unroll 4
        for (; n < end; ++n) {
          const bool t = V >= 1.0;
          sh.v[n] = V;
          word |= (t ? 1u : 0u) << (n & 31);
          V = __dsub_rn(__dadd_rn(V, t ? va : vb), 1.0);
          is += t ? 1u : 0u;
          va = t ? va1 : va;
          vb = t ? vb : vb1;
          va1 = sh.a[is + 1];
          vb1 = sh.b[n + 2 - is];
        }
        sh.bits[(n - 1) >> 5] = word;
        if ((n & 31) == 0) word = 0;
      }
    }
    n = __shfl_sync(0xffffffffu, n, 0);
    is = __shfl_sync(0xffffffffu, is, 0);
    V = __shfl_sync(0xffffffffu, V, 0);
    __syncwarp();
    uint32_t before = 0;  // smalls popped before this word's steps
    for (uint32_t x0 = 0; x0 < n; x0 += 32) {
      const uint32_t word = sh.bits[x0 >> 5], x = x0 + lane;
      if (x < n) {
        const uint32_t a = before + __popc(word & ((1u << lane) - 1u)), b = x - a;
        const uint32_t l = s.idx[(uint64_t)m + j + b];
        if ((word >> lane) & 1) {
          s.alias[s.idx[i + a]] = l;
        } else {  // the current large fell below 1: it gets the next large
          s.alias[l] = s.idx[(uint64_t)m + j + b + 1];
          s.prob[l] = sh.v[x];
        }
      }
      before += __popc(word);
    }
    __syncwarp();
    i += is;
    j += n - is;
    steps -= n;
  }
}

// One warp walks the groups with the true value, and what they do not cover
// chunk by chunk or step by step; then the chain's end.
constexpr uint32_t WALK = 16;  // records staged at a time
__global__ void __launch_bounds__(32) alias_walk_kernel(AliasScratch s, uint32_t nc, uint32_t ng, const int32_t* status) {
  __shared__ RawShared raw;
  __shared__ double send[WALK][32], sbase[WALK], sunit[WALK];
  __shared__ long long smargin[WALK];
  __shared__ uint32_t si[WALK + 1], sj[WALK + 1];
  const int lane = threadIdx.x;
  const uint32_t m = s.totals[0], k = s.totals[1];
  if (status[0] != 0 || m == 0 || k == 0) return;
  double V = s.val ? s.val[m] : s.prob[s.idx[m]];
  uint32_t i = 0, j = 0;
  bool more = true;
  // records [r0, r1) of chunks (per = 1) or groups (per = CGROUP): staged in shared memory
  auto stage = [&](uint32_t r0, uint32_t n, uint32_t per, const long long* margin, const double* end) {
    __syncwarp();
    for (uint32_t x = lane; x <= n; x += 32) {
      const uint32_t c = min(nc, (r0 + x) * per);
      si[x] = s.ci[c];
      sj[x] = s.cj[c];
      if (x < n) {
        sbase[x] = s.cbase[c];
        sunit[x] = s.cunit[c];
        smargin[x] = margin[r0 + x];
      }
    }
    for (uint32_t x = 0; x < n; ++x) send[x][lane] = end[(size_t)(r0 + x) * 32 + lane];
    __syncwarp();
  };
  uint32_t w0 = 0, wn = 0;  // staged groups
  for (uint32_t g = 0; g < ng && more; ++g) {
    if (g >= w0 + wn) {
      w0 = g;
      wn = min(WALK, ng - g);
      stage(w0, wn, CGROUP, s.gmargin, s.gend);
    }
    const uint32_t x = g - w0;
    Entry e;
    long long left;
    if (i == si[x] && j == sj[x] && enter_chunk(V, sbase[x], sunit[x], smargin[x], kMoved, &e, &left)) {
      if (lane == 0) {
        s.gstart[g] = V;
        s.gflag[g] = 1;
      }
      V = send[x][e.lane] + e.shift;
      i = si[x + 1];
      j = sj[x + 1];
      continue;
    }
    const uint32_t c1 = min(nc, (g + 1) * CGROUP);
    for (uint32_t c0 = g * CGROUP; c0 < c1 && more; c0 += WALK) {
      const uint32_t n = min(WALK, c1 - c0);
      stage(c0, n, 1, s.cmargin, s.cend);
      for (uint32_t y = 0; y < n && more; ++y) {
        if (i == si[y] && j == sj[y] && enter_chunk(V, sbase[y], sunit[y], smargin[y], 1ll << 60, &e, &left)) {
          if (lane == 0) {
            s.cstart[c0 + y] = V;
            s.cflag[c0 + y] = 1;
          }
          V = send[y][e.lane] + e.shift;
          i = si[y + 1];
          j = sj[y + 1];
        } else {
          const uint64_t to = (uint64_t)si[y + 1] + sj[y + 1], at = (uint64_t)i + j;
          if (to > at) more = raw_steps(s, m, k, raw, V, i, j, to - at);
        }
      }
    }
    wn = 0;  // the chunk records took the place of the group records
  }
  while (more) more = raw_steps(s, m, k, raw, V, i, j, ~0ull);
  if (lane == 0) {
    s.totals[2] = i;
    s.totals[3] = j;
  }
}

// One warp per walked group: the true start of each of its chunks.
__global__ void __launch_bounds__(128) alias_expand_kernel(AliasScratch s, uint32_t nc, uint32_t ng,
                                                           int32_t* status) {
  const uint32_t q = blockIdx.x * 4 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (q >= ng || status[0] != 0 || s.totals[0] == 0 || s.totals[1] == 0 || !s.gflag[q]) return;
  const uint32_t c0 = q * CGROUP, c1 = min(nc, c0 + CGROUP);
  double V = s.gstart[q];
#pragma unroll 4
  for (uint32_t c = c0; c < c1; ++c) {
    const double end = s.cend[(size_t)c * 32 + lane];
    Entry e{0, 0.0};
    long long left;
    const bool in = enter_chunk(V, s.cbase[c], s.cunit[c], s.cmargin[c], 1ll << 60, &e, &left);
    if (lane == 0) {
      if (!in) status[0] = ALEPH_B200_DEVICE_FAILURE;  // never: the group's margin covers its chunks
      s.cstart[c] = V;
      s.cflag[c] = 1;
    }
    V = __shfl_sync(0xffffffffu, end, e.lane) + e.shift;
  }
}

// One warp per chunk: replay from the true start, then write its table entries.
__global__ void __launch_bounds__(128) alias_emit_kernel(AliasScratch s, uint32_t nc, const int32_t* status) {
  __shared__ ChunkOps ops[4];
  __shared__ uint16_t cur[4][CH_MAX + 1];
  const uint32_t c = blockIdx.x * 4 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  const uint32_t m = s.totals[0], k = s.totals[1];
  if (c >= nc || status[0] != 0 || m == 0 || k == 0 || !s.cflag[c]) return;
  ChunkOps& o = ops[threadIdx.x >> 5];
  uint16_t* cl = cur[threadIdx.x >> 5];  // per small: local index of its large
  const uint32_t i0 = s.ci[c], j0 = s.cj[c];
  const uint32_t ns = s.ci[c + 1] - i0, nl = s.cj[c + 1] - j0, len = ns + nl;
  stage_chunk(s, m, i0, j0, ns, nl, o);
  if (lane == 0) {
    double V = s.cstart[c];
    uint32_t is = 0, il = 0;
    double va = o.a[0], vb = o.b[0];
    for (uint32_t t = 0; t < len; ++t) {
      const bool small = V >= 1.0;
      const double v = small ? va : vb;
      if (small) cl[is] = (uint16_t)il;
      else o.b[il] = V;  // the threshold of large il takes the place of its successor's value, already read
      is += small ? 1u : 0u;
      il += small ? 0u : 1u;
      va = o.a[is];
      vb = o.b[il];
      V = __dsub_rn(__dadd_rn(V, v), 1.0);
    }
  }
  __syncwarp();
  for (uint32_t x = lane; x < ns; x += 32) s.alias[s.idx[i0 + x]] = s.idx[(uint64_t)m + j0 + cl[x]];
  for (uint32_t x = lane; x < nl; x += 32) {
    const uint32_t l = s.idx[(uint64_t)m + j0 + x];
    s.alias[l] = s.idx[(uint64_t)m + j0 + x + 1];
    s.prob[l] = o.b[x];
  }
}

// What was never popped keeps itself with threshold 1, and so does the large in hand.
__global__ void alias_drain_kernel(AliasScratch s, const int32_t* status) {
  if (status[0] != 0) return;
  const uint32_t m = s.totals[0], k = s.totals[1], i0 = s.totals[2], j0 = s.totals[3];
  const uint64_t n = (uint64_t)(m - i0) + (k - j0);
  for (uint64_t x = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; x < n; x += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t i = s.idx[x < m - i0 ? i0 + x : (uint64_t)m + j0 + (x - (m - i0))];
    s.prob[i] = 1.0;
    s.alias[i] = i;
  }
}

__global__ void alias_draw_kernel(AliasScratch s, uint64_t mask, const uint64_t* __restrict__ words, uint32_t shots,
                                  uint64_t* __restrict__ out, const int32_t* status) {
  if (status[0] != 0) return;
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < shots; k += gridDim.x * blockDim.x) {
    const uint64_t bits = words[k];
    const uint64_t i = (bits >> 32) & mask;
    const double u = (double)(uint32_t)bits * (1.0 / 4294967296.0);
    out[k] = u < s.prob[i] ? i : (uint64_t)s.alias[i];
  }
}

// States of at most PART_B amplitudes: the whole build and the draws in one kernel, the
// table in shared memory. The chain is short (some 40 ns a step), and the launches
// of the parallel build alone cost more. Each CTA builds the table for its share of the shots.
template <typename Real>
__global__ void __launch_bounds__(PART_B) alias_small_kernel(const V2<Real>* __restrict__ amps, uint32_t len,
                                                             const uint64_t* __restrict__ words, uint32_t shots,
                                                             uint64_t* __restrict__ out, double tol, int32_t* status) {
  __shared__ double prob[PART_B], sv[PART_B + 2], lv[PART_B + 2];
  __shared__ uint16_t alias[PART_B], si[PART_B + 2], li[PART_B + 2];
  __shared__ uint32_t smalls[32];
  __shared__ double red[2][32];
  __shared__ uint32_t m_sh, ok_sh;
  const uint32_t tid = threadIdx.x, lane = tid & 31, w = tid >> 5, warps = blockDim.x >> 5;
  const bool valid = tid < len;
  const uint32_t i0 = valid ? len - 1 - tid : 0;  // pop order: descending basis states
  double sc = 0.0, psum = 0.0, bad = 0.0;
  if (valid) {
    const double p = prob_exact<Real>(amps, i0);
    if (isfinite(p)) psum = p;
    else bad = 1.0;
    sc = __dmul_rn((double)len, p);
    prob[i0] = 1.0;  // what is never popped keeps itself
    alias[i0] = (uint16_t)i0;
  }
  const unsigned bs = __ballot_sync(0xffffffffu, valid && sc < 1.0);
  for (int o = 16; o; o >>= 1) {
    psum += __shfl_down_sync(0xffffffffu, psum, o);
    bad += __shfl_down_sync(0xffffffffu, bad, o);
  }
  if (lane == 0) {
    smalls[w] = __popc(bs);
    red[0][w] = psum;
    red[1][w] = bad;
  }
  __syncthreads();
  if (tid == 0) {
    uint32_t m = 0;
    double a = 0.0, b = 0.0;
    for (uint32_t x = 0; x < warps; ++x) {
      const uint32_t c = smalls[x];
      smalls[x] = m;
      m += c;
      a += red[0][x];
      b += red[1][x];
    }
    m_sh = m;
    ok_sh = !(b > 0.0) && isfinite(a) && fabs(a - 1.0) <= tol;
    check_norm(a, b, tol, status);
  }
  __syncthreads();
  if (!ok_sh) return;
  if (valid) {
    const uint32_t before = smalls[w] + __popc(bs & ((1u << lane) - 1u));  // smalls popped before this element
    if (sc < 1.0) {
      sv[before] = sc;
      si[before] = (uint16_t)i0;
    } else {
      lv[tid - before] = sc;
      li[tid - before] = (uint16_t)i0;
    }
  }
  __syncthreads();
  const uint32_t m = m_sh, k = len - m;
  if (tid == 0 && m && k) {  // see raw_steps
    uint32_t i = 0, j = 0, cs = si[0], cs1 = si[1], cl = li[0], cl1 = li[1], cl2 = li[2];
    double V = lv[0], va = sv[0], va1 = sv[1], vb = lv[1], vb1 = lv[2];
    for (;;) {
      const bool t = V >= 1.0;
      if (t ? i >= m : j + 1 >= k) break;
      const double Sa = __dadd_rn(V, va), Sb = __dadd_rn(V, vb);
      const uint32_t at = t ? cs : cl;
      prob[at] = t ? va : V;
      alias[at] = (uint16_t)(t ? cl : cl1);
      i += t ? 1u : 0u;
      j += t ? 0u : 1u;
      va = t ? va1 : va;
      cs = t ? cs1 : cs;
      vb = t ? vb : vb1;
      cl = t ? cl : cl1;
      cl1 = t ? cl1 : cl2;
      va1 = sv[i + 1];  // i <= m, j < k: inside the arrays
      cs1 = si[i + 1];
      vb1 = lv[j + 2];
      cl2 = li[j + 2];
      V = __dsub_rn(t ? Sa : Sb, 1.0);
    }
  }
  __syncthreads();
  for (uint64_t x = (uint64_t)blockIdx.x * blockDim.x + tid; x < shots; x += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t bits = words[x];
    const uint32_t i = (uint32_t)(bits >> 32) & (len - 1);
    const double u = (double)(uint32_t)bits * (1.0 / 4294967296.0);
    out[x] = u < prob[i] ? i : alias[i];
  }
}

// ------------------------------------------------------------- CUMULATIVE ----
// A run of S <- fl(S + p) with S in one binade [2^e, 2^(e+1)) adds to S, in
// units of 2^(e-52), the integer nearest to p; only an exact tie depends on S,
// through its parity. So a run of additions is a function of the start's
// parity, two integers, and runs compose: the reference's left-to-right sum is
// evaluated in parallel, bit for bit, binade by binade. (One lane adding in
// order took 6.8 ns an element, 459 ms at n = 26.)
struct SeqFn {
  long long o0, o1;  // units added to an even / odd start
};
__device__ __forceinline__ SeqFn seq_then(const SeqFn& a, const SeqFn& b) {
  SeqFn r;
  r.o0 = a.o0 + ((a.o0 & 1) ? b.o1 : b.o0);
  r.o1 = a.o1 + ((a.o1 & 1) ? b.o0 : b.o1);
  return r;
}
constexpr long long kSeqOver = 1ll << 53;  // at least this many units leave the binade
// One addition of p >= 0; scale = 2^(52-e). *tie is set when the rounding depends on the parity.
__device__ __forceinline__ SeqFn seq_fn(double p, double scale, bool* tie) {
  const double x = p * scale;  // exact: a power of two, and the result is normal or zero (e >= -500)
  if (!(x < 0x1p53)) return SeqFn{kSeqOver, kSeqOver};
  const double f = floor(x), d = x - f;
  const long long fi = (long long)f;
  if (d != 0.5) {
    const long long r = d > 0.5 ? fi + 1 : fi;
    return SeqFn{r, r};
  }
  *tie = true;
  return SeqFn{fi + (fi & 1), fi + ((fi + 1) & 1)};
}
// S + off units of 2^(e-52), for a sum inside the binade (exact).
__device__ __forceinline__ double seq_add(double S, long long off, double unit) { return S + (double)off * unit; }
constexpr double kSeqMin = 0x1p-500;  // smaller sums (zero among them) are added one by one

struct CumScratch {
  double* bsum;      // nb + 1: block sums, then exclusive block prefix (bsum[nb] = total)
  double* norm;      // 2: [unused, non-finite count]
  uint32_t* namb;    // ambiguous shot count
  uint32_t* amb;     // shots: ambiguous shot ids
  double* ck;        // exact mode: sequential sum at the end of every SEQ_CH chunk
  double* seq;       // exact mode: [sequential total, last positive index (bits)]
  double* part;      // PREFIX_T range totals of the block prefix
  // exact mode: the chunks in up to PREFIX_T segments: function, binade, start (< 0: not walked whole)
  SeqFn* sfn;
  int* sfe;
  double* sstart;
  SeqFn* fn;         // exact mode: the chunk as a function of the start's parity
  int* fe;           // exact mode: its binade (kNoBinade: crosses one; kAnyBinade: adds nothing)
};
constexpr int kNoBinade = -100000, kAnyBinade = 100000;

template <typename Real>
__global__ void cum_blocks_kernel(const V2<Real>* __restrict__ amps, uint64_t len, CumScratch c) {
  __shared__ double red[2][8];
  const uint64_t b0 = (uint64_t)blockIdx.x * CUM_BLOCK;
  double x = 0.0, bad = 0.0;
  for (uint32_t j = threadIdx.x; j < CUM_BLOCK && b0 + j < len; j += blockDim.x) {
    const double p = prob_exact<Real>(amps, b0 + j);
    if (isfinite(p)) x += p;
    else bad += 1.0;
  }
  for (int o = 16; o; o >>= 1) {
    x += __shfl_down_sync(0xffffffffu, x, o);
    bad += __shfl_down_sync(0xffffffffu, bad, o);
  }
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = x;
    red[1][threadIdx.x >> 5] = bad;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0, b = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
      s += red[0][w];
      b += red[1][w];
    }
    c.bsum[blockIdx.x] = s;
    if (b > 0.0) atomicAdd(&c.norm[1], b);
  }
}

// Exclusive prefix of the block sums: PREFIX_T contiguous ranges are added in
// order, their totals are scanned, and each range's prefixes are written in
// order. The draws treat this prefix as an approximation (guard band E below), so
// its rounding order is free, but it is kept. The ranges are spread over CTAs
// of one warp: on one SM the strided reads alone took 50 us at n = 26.
constexpr uint32_t PREFIX_T = 1024;
constexpr uint32_t RANGE_T = 32;  // threads per CTA of the range kernels
__device__ __forceinline__ void range_of(uint32_t n, uint32_t t, uint32_t* b0, uint32_t* b1) {
  const uint32_t per = (n + PREFIX_T - 1) / PREFIX_T;
  *b0 = min(n, t * per);
  *b1 = min(n, *b0 + per);
}
__global__ void __launch_bounds__(RANGE_T) cum_range_kernel(CumScratch c, uint32_t nb) {
  const uint32_t t = blockIdx.x * RANGE_T + threadIdx.x;
  uint32_t b0, b1;
  range_of(nb, t, &b0, &b1);
  double s = 0.0;
  for (uint32_t b = b0; b < b1; ++b) s += c.bsum[b];
  c.part[t] = s;
}
// ONE: up to PREFIX_T blocks, a block per range: this kernel alone does it (three
// kernels took 8 us more from small states).
template <bool ONE>
__global__ void __launch_bounds__(PREFIX_T) cum_prefix_kernel(CumScratch c, uint32_t nb, double tol, int32_t* status) {
  __shared__ double part[PREFIX_T];
  const uint32_t t = threadIdx.x;
  part[t] = !ONE ? c.part[t] : t < nb ? c.bsum[t] : 0.0;
  __syncthreads();
  for (uint32_t off = 1; off < blockDim.x; off <<= 1) {  // inclusive Hillis-Steele scan
    const double v = t >= off ? part[t - off] : 0.0;
    __syncthreads();
    part[t] += v;
    __syncthreads();
  }
  if (!ONE) c.part[t] = part[t];
  else if (t < nb) c.bsum[t] = t ? part[t - 1] : 0.0;
  if (t == blockDim.x - 1) {
    c.bsum[nb] = part[t];
    check_norm(part[t], c.norm[1], tol, status);
  }
}
__global__ void __launch_bounds__(RANGE_T) cum_spread_kernel(CumScratch c, uint32_t nb) {
  const uint32_t t = blockIdx.x * RANGE_T + threadIdx.x;
  uint32_t b0, b1;
  range_of(nb, t, &b0, &b1);
  double run = t ? c.part[t - 1] : 0.0;
  for (uint32_t b = b0; b < b1; ++b) {
    const double x = c.bsum[b];
    c.bsum[b] = run;
    run += x;
  }
}

// One warp adds amplitudes [b, e) to S in order and stops at the first index i
// with target < S_i: *before = S_i-1, *at = S_i; *last_pos is the last positive
// bin seen. Returns -1 when there is none. Every S is the sequential sum.
template <typename Real>
__device__ int64_t seq_search(const V2<Real>* __restrict__ amps, uint64_t b, uint64_t e, double S, double target,
                              double* before, double* at, int64_t* last_pos) {
  const int lane = threadIdx.x & 31;
  for (uint64_t r0 = b; r0 < e; r0 += 32) {
    const double p = r0 + lane < e ? prob_exact<Real>(amps, r0 + lane) : 0.0;
    const unsigned pos = __ballot_sync(0xffffffffu, p > 0.0);
    if (pos == 0) continue;
    double mine;
    bool in_binade = false;
    if (S >= kSeqMin) {
      const int ex = (int)((__double_as_longlong(S) >> 52) & 0x7ff) - 1023;
      const double unit = __longlong_as_double((long long)(ex - 52 + 1023) << 52);
      const double scale = __longlong_as_double((long long)(52 - ex + 1023) << 52);
      bool tie = false;
      SeqFn f = seq_fn(p, scale, &tie);
      long long off;
      if (__any_sync(0xffffffffu, tie)) {
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          SeqFn g;
          g.o0 = __shfl_up_sync(0xffffffffu, f.o0, o);
          g.o1 = __shfl_up_sync(0xffffffffu, f.o1, o);
          if (lane >= o) f = seq_then(g, f);
        }
        off = (__double_as_longlong(S) & 1) ? f.o1 : f.o0;
      } else {
        off = f.o0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const long long g = __shfl_up_sync(0xffffffffu, off, o);
          if (lane >= o) off += g;
        }
      }
      const long long mant = (__double_as_longlong(S) & ((1ll << 52) - 1)) | (1ll << 52);
      in_binade = __all_sync(0xffffffffu, mant + off < kSeqOver);  // offsets ascend: at most 32 * 2^53
      mine = seq_add(S, off, unit);
    }
    if (!in_binade) {  // a binade boundary in these 32 (or a sum near zero): one by one
      double run = S;
      mine = S;
#pragma unroll
      for (int q = 0; q < 32; ++q) {
        run = __dadd_rn(run, __shfl_sync(0xffffffffu, p, q));
        if (lane == q) mine = run;
      }
    }
    const unsigned hit = __ballot_sync(0xffffffffu, p > 0.0 && target < mine);
    double prev = __shfl_up_sync(0xffffffffu, mine, 1);
    if (lane == 0) prev = S;
    if (hit) {
      const int w = __ffs(hit) - 1;
      *before = __shfl_sync(0xffffffffu, prev, w);
      *at = __shfl_sync(0xffffffffu, mine, w);
      return (int64_t)(r0 + w);
    }
    *last_pos = (int64_t)(r0 + (31 - __clz(pos)));
    S = __shfl_sync(0xffffffffu, mine, 31);
  }
  return -1;
}

// One warp per shot: the block by binary search over the prefix, the bin by
// adding the block in order.
template <typename Real>
__global__ void __launch_bounds__(128) cum_draw_kernel(const V2<Real>* __restrict__ amps, uint64_t len, uint32_t nb,
                                                       CumScratch c, const double* __restrict__ uniforms,
                                                       uint32_t shots, uint64_t* __restrict__ out) {
  const uint32_t k = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (k >= shots) return;
  const double total = c.bsum[nb];
  // Bound on |sequential - two-level| for prefixes and for u * total.
  const double E = 8.0 * ((double)len + 64.0) * 1.1102230246251565e-16 * total;
  const double target = uniforms[k] * total;
  // last block whose exclusive prefix <= target
  uint32_t lo = 0, hi = nb;  // invariant: prefix[lo] <= target (prefix[0] = 0)
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (c.bsum[mid] <= target) lo = mid;
    else hi = mid;
  }
  double before = 0.0, at = 0.0;
  int64_t last_pos = -1;
  int64_t found = seq_search<Real>(amps, (uint64_t)lo * CUM_BLOCK, len, c.bsum[lo], target, &before, &at, &last_pos);
  // the sums ascend, so the boundary next to the target is the nearest one
  double margin = fmin(fabs(target - before), fabs(at - target));
  if (found < 0) {
    // ran off the end: the last positive bin at or after the start block,
    // or, if none, any earlier positive bin (resolved exactly below)
    found = last_pos;
    margin = 0.0;
  }
  if ((threadIdx.x & 31) == 0) {
    out[k] = (uint64_t)(found < 0 ? 0 : found);
    if (margin <= E) {
      const uint32_t slot = atomicAdd(c.namb, 1u);
      c.amb[slot] = k;
    }
  }
}

// Exact resolution of the ambiguous shots, in three kernels.
//
// cum_fn_kernel: every SEQ_CH-element chunk as a function of its start's parity
// (SeqFn), in the binade that the approximate prefix predicts, and the last
// positive index.
// cum_walk_kernel: the reference's sequential left-to-right sum (validate_norm's
// total and cumulative_index's running sum are the same sequence
// S_i = fl(S_{i-1} + p_i)) through the chunks: exact checkpoints at the end of
// every chunk and the total. One CTA: 1024 segments of chunks compose, one
// lane steps through the segments, and the chunks that cross a binade (some
// log2(chunks) of them) are scanned by the whole CTA.
// cum_exact_kernel: per ambiguous shot, the first chunk whose checkpoint
// exceeds the target, added again in order from the previous checkpoint,
// so every outcome equals the sequential CPU scan's.
constexpr uint32_t SEQ_CH = 2048;
static_assert(SEQ_CH == CUM_BLOCK, "the chunks' binades come from the block prefix");

template <typename Real>
__global__ void __launch_bounds__(256) cum_fn_kernel(const V2<Real>* __restrict__ amps, uint64_t len, CumScratch c) {
  __shared__ long long red[8];
  __shared__ SeqFn fr[8];
  __shared__ uint32_t lastp;
  if (*c.namb == 0) return;  // uniform: no ambiguous shot, nothing to resolve
  const uint32_t ch = blockIdx.x, tid = threadIdx.x;
  const uint64_t b0 = (uint64_t)ch * SEQ_CH;
  const double s0 = c.bsum[ch], s1 = c.bsum[ch + 1];
  const int e = (int)((__double_as_longlong(s0) >> 52) & 0x7ff) - 1023;
  const bool one = s0 >= kSeqMin && (int)((__double_as_longlong(s1) >> 52) & 0x7ff) - 1023 == e;
  const double scale = one ? __longlong_as_double((long long)(52 - e + 1023) << 52) : 1.0;
  if (tid == 0) lastp = 0;
  __syncthreads();
  double p[SEQ_CH / 256];
#pragma unroll
  for (int r = 0; r < (int)(SEQ_CH / 256); ++r) {
    const uint64_t i = b0 + r * 256 + tid;
    p[r] = i < len ? prob_exact<Real>(amps, i) : 0.0;
  }
  long long sum = 0;
  bool tie = false;
  uint32_t last = 0;  // 1 + last positive element of the chunk
#pragma unroll
  for (int r = 0; r < (int)(SEQ_CH / 256); ++r) {
    if (p[r] > 0.0) last = r * 256 + tid + 1;
    sum += seq_fn(p[r], scale, &tie).o0;
  }
  last = __reduce_max_sync(0xffffffffu, last);
  if ((tid & 31) == 0 && last) atomicMax(&lastp, last);
  const bool ties = __syncthreads_or(tie ? 1 : 0) != 0;
  if (lastp == 0) {
    if (tid == 0) c.fe[ch] = kAnyBinade;
    return;
  }
  if (tid == 0) atomicMax((unsigned long long*)&c.seq[1], (unsigned long long)(b0 + lastp));  // 1 + index
  if (!one) {
    if (tid == 0) c.fe[ch] = kNoBinade;
    return;
  }
  if (!ties) {
    for (int o = 16; o; o >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, o);
    if ((tid & 31) == 0) red[tid >> 5] = sum;
    __syncthreads();
    if (tid == 0) {
      long long t = 0;
      for (int w = 0; w < 8; ++w) t += red[w];
      c.fn[ch] = SeqFn{t, t};
      c.fe[ch] = e;
    }
    return;
  }
  // ties: the order matters, so each thread composes 8 consecutive elements
  SeqFn f{0, 0};
  for (int r = 0; r < (int)(SEQ_CH / 256); ++r) {
    const uint64_t i = b0 + (uint64_t)tid * (SEQ_CH / 256) + r;
    bool t = false;
    f = seq_then(f, seq_fn(i < len ? prob_exact<Real>(amps, i) : 0.0, scale, &t));
  }
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    SeqFn g;
    g.o0 = __shfl_down_sync(0xffffffffu, f.o0, o);
    g.o1 = __shfl_down_sync(0xffffffffu, f.o1, o);
    f = seq_then(f, g);  // lane 0's is the warp's, in order
  }
  if ((tid & 31) == 0) fr[tid >> 5] = f;
  __syncthreads();
  if (tid == 0) {
    SeqFn t = fr[0];
    for (int w = 1; w < 8; ++w) t = seq_then(t, fr[w]);
    c.fn[ch] = t;
    c.fe[ch] = e;
  }
}

// A sum as its mantissa (units of 2^(e-52)) and binade.
struct SeqSum {
  long long mant;
  int e;
};
__device__ __forceinline__ SeqSum seq_sum(double S) {
  const long long bits = __double_as_longlong(S);
  return SeqSum{(bits & ((1ll << 52) - 1)) | (1ll << 52), (int)((bits >> 52) & 0x7ff) - 1023};
}
__device__ __forceinline__ double seq_value(const SeqSum& s) {
  return __longlong_as_double(((long long)(s.e + 1023) << 52) | (s.mant & ((1ll << 52) - 1)));
}
// Applies a chunk's (or segment's) function; false when the sum does not stay in its binade.
__device__ __forceinline__ bool seq_step(SeqSum* s, int e, const SeqFn& f) {
  if (e == kAnyBinade) return true;
  if (e != s->e) return false;
  const long long m = s->mant + ((s->mant & 1) ? f.o1 : f.o0);
  if (m >= kSeqOver) return false;
  s->mant = m;
  return true;
}

// The chunks of each segment composed: one binade, or kNoBinade.
__global__ void __launch_bounds__(RANGE_T) cum_compose_kernel(CumScratch c, uint32_t nch) {
  if (*c.namb == 0) return;
  const uint32_t t = blockIdx.x * RANGE_T + threadIdx.x;
  uint32_t c0, c1;
  range_of(nch, t, &c0, &c1);
  SeqFn f{0, 0};
  int e = kAnyBinade;
  for (uint32_t k = c0; k < c1; ++k) {
    const int ek = c.fe[k];
    const SeqFn fk = c.fn[k];
    if (ek == kAnyBinade) continue;
    if (e == kAnyBinade) {
      e = ek;
      f = fk;
    } else if (ek == e && e != kNoBinade) {
      f = seq_then(f, fk);
    } else {
      e = kNoBinade;
    }
  }
  c.sfn[t] = f;
  c.sfe[t] = e;
  c.sstart[t] = -1.0;
}

constexpr uint32_t WALK_T = 1024;
static_assert(WALK_T == PREFIX_T && 2 * WALK_T == SEQ_CH, "a thread per segment, and two elements of a crossing chunk");
// chunks per segment at most (n = kExactCumulativeMaxN)
constexpr uint32_t kWalkChunks = (uint32_t)(((uint64_t)1 << kExactCumulativeMaxN) / SEQ_CH / WALK_T);
template <typename Real>
__global__ void __launch_bounds__(WALK_T) cum_walk_kernel(const V2<Real>* __restrict__ amps, uint64_t len,
                                                          uint32_t nch, CumScratch c) {
  __shared__ SeqFn sfn[WALK_T];
  __shared__ int se[WALK_T];
  __shared__ SeqFn wtot[32];
  __shared__ SeqFn cfn[kWalkChunks];  // the chunks of the segment at hand
  __shared__ int cfe[kWalkChunks];
  __shared__ double S_sh;
  __shared__ uint32_t seg_sh, ch_sh, first_sh;
  if (*c.namb == 0) return;
  const uint32_t t = threadIdx.x, lane = t & 31, w = t >> 5;
  const uint32_t per = (nch + WALK_T - 1) / WALK_T;
  if (nch == 1) {  // one chunk, scanned by the whole CTA: no functions were formed
    if (t == 0) c.fe[0] = kNoBinade;
    const uint64_t i = 2 * t;
    const bool p0 = i < len && prob_exact<Real>(amps, i) > 0.0, p1 = i + 1 < len && prob_exact<Real>(amps, i + 1) > 0.0;
    if (p0 || p1) atomicMax((unsigned long long*)&c.seq[1], (unsigned long long)(i + (p1 ? 2 : 1)));  // 1 + index
    se[t] = kNoBinade;
  } else if (per == 1) {  // a chunk per segment: nothing was composed
    if (t < nch) {
      sfn[t] = c.fn[t];
      se[t] = c.fe[t];
    }
  } else {
    sfn[t] = c.sfn[t];
    se[t] = c.sfe[t];
  }
  if (t == 0) {
    S_sh = 0.0;
    seg_sh = 0;
  }
  __syncthreads();
  const uint32_t nseg = (nch + per - 1) / per;
  for (;;) {
    if (t == 0) {  // as many whole segments as hold
      SeqSum S = seq_sum(S_sh);
      uint32_t g = seg_sh;
      for (; g < nseg; ++g) {
        const SeqSum at = S;
        if (!seq_step(&S, se[g], sfn[g])) break;
        if (per == 1) c.ck[g] = S_sh > 0.0 ? seq_value(S) : 0.0;
        else c.sstart[g] = S_sh > 0.0 ? seq_value(at) : 0.0;
      }
      if (S_sh > 0.0) S_sh = seq_value(S);
      seg_sh = g;
      ch_sh = g * per;
    }
    __syncthreads();
    const uint32_t g = seg_sh;
    if (g >= nseg) break;
    const uint32_t first = g * per, end = min(nch, first + per);
    for (uint32_t k = first + t; k < end; k += WALK_T) {
      cfe[k - first] = c.fe[k];
      cfn[k - first] = c.fn[k];
    }
    for (;;) {  // its chunks one by one
      __syncthreads();
      if (t == 0) {
        SeqSum S = seq_sum(S_sh);
        const bool zero = !(S_sh > 0.0);
        uint32_t k = ch_sh;
        for (; k < end; ++k) {
          if (!seq_step(&S, cfe[k - first], cfn[k - first])) break;
          c.ck[k] = zero ? 0.0 : seq_value(S);
        }
        if (!zero) S_sh = seq_value(S);
        ch_sh = k;
      }
      __syncthreads();
      const uint32_t k = ch_sh;
      if (k >= end) break;
      // a chunk that crosses a binade: two elements a thread, scanned once per binade
      const uint64_t b0 = (uint64_t)k * SEQ_CH + 2 * t;
      const double p0 = b0 < len ? prob_exact<Real>(amps, b0) : 0.0;
      const double p1 = b0 + 1 < len ? prob_exact<Real>(amps, b0 + 1) : 0.0;
      uint32_t pos = 0;  // elements before pos are in S
      while (pos < SEQ_CH) {
        const double S = S_sh;
        const bool a0 = 2 * t >= pos, a1 = 2 * t + 1 >= pos;
        double before = S;  // the sum before the element where the scan stops
        uint32_t stop = SEQ_CH;
        if (t == 0) first_sh = SEQ_CH;
        __syncthreads();
        if (S < kSeqMin) {  // near zero: the next positive element by itself
          if (a0 && p0 > 0.0) stop = 2 * t;
          else if (a1 && p1 > 0.0) stop = 2 * t + 1;
          if (stop < SEQ_CH) atomicMin(&first_sh, stop);
          __syncthreads();
          if (first_sh == SEQ_CH) break;
        } else {
          const SeqSum q = seq_sum(S);
          const double scale = __longlong_as_double((long long)(52 - q.e + 1023) << 52);
          bool tie = false;
          const SeqFn f0 = a0 ? seq_fn(p0, scale, &tie) : SeqFn{0, 0}, f1 = a1 ? seq_fn(p1, scale, &tie) : SeqFn{0, 0};
          SeqFn inc = seq_then(f0, f1);
          auto scan = [&](SeqFn x) {  // inclusive over the warp, in order
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
              SeqFn y;
              y.o0 = __shfl_up_sync(0xffffffffu, x.o0, o);
              y.o1 = __shfl_up_sync(0xffffffffu, x.o1, o);
              if (lane >= (uint32_t)o) x = seq_then(y, x);
            }
            return x;
          };
          inc = scan(inc);
          if (lane == 31) wtot[w] = inc;
          SeqFn ex;  // exclusive within the warp
          ex.o0 = __shfl_up_sync(0xffffffffu, inc.o0, 1);
          ex.o1 = __shfl_up_sync(0xffffffffu, inc.o1, 1);
          if (lane == 0) ex = SeqFn{0, 0};
          __syncthreads();
          if (w == 0) wtot[lane] = scan(wtot[lane]);
          __syncthreads();
          const SeqFn pre = seq_then(w ? wtot[w - 1] : SeqFn{0, 0}, ex);
          // at the first element that leaves the binade all sums before it are below 2^53
          const long long m0 = q.mant + ((q.mant & 1) ? pre.o1 : pre.o0);
          const long long m1 = m0 + ((m0 & 1) ? f0.o1 : f0.o0);
          const long long m2 = m1 + ((m1 & 1) ? f1.o1 : f1.o0);
          if (a0 && m1 >= kSeqOver) {
            stop = 2 * t;
            before = seq_value(SeqSum{m0, q.e});
          } else if (a1 && m2 >= kSeqOver) {
            stop = 2 * t + 1;
            before = seq_value(SeqSum{m1, q.e});
          }
          if (stop < SEQ_CH) atomicMin(&first_sh, stop);
          __syncthreads();
          if (first_sh == SEQ_CH) {  // the rest stays in the binade
            if (t == WALK_T - 1) S_sh = seq_value(SeqSum{m2, q.e});
            break;
          }
        }
        if (stop == first_sh) S_sh = __dadd_rn(before, (stop & 1) ? p1 : p0);
        pos = first_sh + 1;
        __syncthreads();
      }
      __syncthreads();
      if (t == 0) {
        c.ck[k] = S_sh;
        ch_sh = k + 1;
      }
      __syncthreads();
    }
    if (t == 0) seg_sh = g + 1;
    __syncthreads();
  }
  if (t == 0) c.seq[0] = S_sh;
}

// The checkpoints inside the segments that were walked whole.
__global__ void __launch_bounds__(RANGE_T) cum_expand_kernel(CumScratch c, uint32_t nch) {
  if (*c.namb == 0) return;
  const uint32_t t = blockIdx.x * RANGE_T + threadIdx.x;
  uint32_t c0, c1;
  range_of(nch, t, &c0, &c1);
  const double start = c.sstart[t];
  if (start < 0.0) return;
  SeqSum S = seq_sum(start);
  for (uint32_t k = c0; k < c1; ++k) {
    seq_step(&S, c.fe[k], c.fn[k]);
    c.ck[k] = start > 0.0 ? seq_value(S) : 0.0;
  }
}

// One warp per ambiguous shot.
template <typename Real>
__global__ void __launch_bounds__(128) cum_exact_kernel(const V2<Real>* __restrict__ amps, uint64_t len, CumScratch c,
                                                        const double* __restrict__ uniforms,
                                                        uint64_t* __restrict__ out, int32_t* status) {
  const uint32_t na = *c.namb;
  const uint32_t a = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (a >= na) return;
  const uint64_t nch = (len + SEQ_CH - 1) / SEQ_CH;
  const double total = c.seq[0];
  const int64_t last_pos = __double_as_longlong(c.seq[1]) - 1;  // -1: none
  const uint32_t k = c.amb[a];
  const double target = uniforms[k] * total;
  // first chunk whose inclusive checkpoint exceeds the target
  uint64_t lo = 0, hi = nch;
  while (lo < hi) {
    const uint64_t mid = (lo + hi) >> 1;
    if (target < c.ck[mid]) hi = mid;
    else lo = mid + 1;
  }
  int64_t found = last_pos;  // target >= total: the last positive bin
  if (lo < nch) {
    const uint64_t e = (lo + 1) * SEQ_CH < len ? (lo + 1) * SEQ_CH : len;
    double before, at;
    int64_t seen = -1;
    found = seq_search<Real>(amps, lo * SEQ_CH, e, lo ? c.ck[lo - 1] : 0.0, target, &before, &at, &seen);
    if (found < 0) return;  // never: the checkpoint exceeds the target
  }
  if ((threadIdx.x & 31) == 0) {
    if (found < 0) status[0] = ALEPH_B200_INVALID_STATE;
    else out[k] = (uint64_t)found;
  }
}

// The chunk functions of the exact resolution (SeqFn and binade per chunk).
size_t sample_chunk_fn_bytes(uint32_t n) {
  const uint64_t len = 1ull << n;
  const uint64_t nch = n <= EXACT_MAX_N ? (len + SEQ_CH - 1) / SEQ_CH : 0;
  return nch * (sizeof(SeqFn) + 4) + PREFIX_T * (8 + sizeof(SeqFn) + 4 + 8) + 128;
}

namespace {
// Lays fields out one after the other, 16-byte aligned; with a null base it only counts bytes.
struct Carver {
  char* base;
  size_t off = 0;
  template <typename T>
  T* take(uint64_t count) {
    off = (off + 15) & ~(size_t)15;
    T* p = base ? (T*)(base + off) : nullptr;
    off += count * sizeof(T);
    return p;
  }
};

// The alias table's scratch: 41.3 bytes per amplitude, or 16 without the values,
// prefixes and chunks of the parallel build (the chain then runs step by step).
AliasScratch alias_scratch(Carver& c, uint32_t n, bool parallel) {
  const uint64_t len = 1ull << n;
  const uint64_t nb = (len + PART_B - 1) / PART_B;
  const uint64_t nc = alias_chunks(len), ng = (nc + CGROUP - 1) / CGROUP;
  AliasScratch s{};
  s.prob = c.take<double>(len);
  s.alias = c.take<uint32_t>(len);
  s.idx = c.take<uint32_t>(len);
  s.bcount = c.take<uint32_t>(nb);
  s.bdef = c.take<u128>(nb);
  s.bsur = c.take<u128>(nb);
  s.normsum = c.take<double>(2 * nb);
  s.totals = c.take<uint32_t>(4);
  if (!parallel) return s;
  s.val = c.take<double>(len);
  s.pre = c.take<u128>(len);
  s.ci = c.take<uint32_t>(nc + 1);
  s.cj = c.take<uint32_t>(nc + 1);
  s.cbase = c.take<double>(nc + 1);
  s.cunit = c.take<double>(nc + 1);
  s.cmargin = c.take<long long>(nc);
  s.cmax = c.take<int>(nc);
  s.cend = c.take<double>(nc * 32);
  s.cstart = c.take<double>(nc);
  s.cflag = c.take<uint8_t>(nc + 1);
  s.gmargin = c.take<long long>(ng);
  s.gend = c.take<double>(ng * 32);
  s.gstart = c.take<double>(ng);
  s.gflag = c.take<uint8_t>(ng);
  return s;
}
}  // namespace

size_t sample_scratch_bytes(uint32_t n, int mode, uint32_t shots, bool least) {
  const uint64_t len = 1ull << n;
  if (mode == ALEPH_B200_SAMPLE_ALIAS) {
    if (len <= PART_B) return 256;
    Carver c{nullptr};
    alias_scratch(c, n, !least);
    return c.off + 256;
  }
  const uint64_t nb = (len + CUM_BLOCK - 1) / CUM_BLOCK;
  const uint64_t nch = n <= EXACT_MAX_N ? (len + SEQ_CH - 1) / SEQ_CH : 0;  // exact-mode checkpoints
  return (nb + 1) * 8 + 64 + 256 + (size_t)shots * 4 + 16 + nch * 8 + 32 + sample_chunk_fn_bytes(n);
}

static inline char* align_up(char* p, size_t a) {
  return (char*)(((uintptr_t)p + a - 1) & ~(uintptr_t)(a - 1));
}

cudaError_t launch_sample(const void* amps, int precision, uint32_t n, uint32_t shots, int mode, const void* variates,
                          uint64_t* out, void* scratch, size_t scratch_bytes, int32_t* status, int sm_count,
                          uint32_t* launches, cudaStream_t st) {
  const uint64_t len = 1ull << n;
  const bool f64 = precision == ALEPH_B200_F64;
  const double tol = norm_tolerance(len, precision);
  if (mode == ALEPH_B200_SAMPLE_ALIAS && len <= PART_B) {
    const unsigned threads = len < 32 ? 32u : (unsigned)len;
    const unsigned want = shots / 4096 + 1, grid = want < (unsigned)sm_count ? want : (unsigned)sm_count;
    const uint64_t* words = (const uint64_t*)variates;
    if (f64)
      alias_small_kernel<double><<<grid, threads, 0, st>>>((const double2*)amps, (uint32_t)len, words, shots, out, tol, status);
    else
      alias_small_kernel<float><<<grid, threads, 0, st>>>((const float2*)amps, (uint32_t)len, words, shots, out, tol, status);
    *launches = 1;
    return cudaGetLastError();
  }
  if (mode == ALEPH_B200_SAMPLE_ALIAS) {
    const uint32_t nb = (uint32_t)((len + PART_B - 1) / PART_B);
    const bool parallel = scratch_bytes >= sample_scratch_bytes(n, mode, shots, false);
    const uint32_t nc = parallel ? alias_chunks(len) : 0, ng = (nc + CGROUP - 1) / CGROUP;
    Carver c{(char*)scratch};
    const AliasScratch s = alias_scratch(c, n, parallel);
    if (c.off > scratch_bytes) return cudaErrorInvalidValue;
    if (f64) alias_scale_kernel<double><<<nb, PART_B, 0, st>>>((const double2*)amps, len, s);
    else alias_scale_kernel<float><<<nb, PART_B, 0, st>>>((const float2*)amps, len, s);
    alias_offsets_kernel<<<1, 1024, 0, st>>>(s, len, nb, tol, status);
    alias_partition_kernel<<<nb, PART_B, 0, st>>>(len, s, status);
    if (nc) {
      alias_cuts_kernel<<<nc / 4 + 1, 128, 0, st>>>(s, nc, status);
      alias_spec_kernel<<<(nc + 3) / 4, 128, 0, st>>>(s, nc, status);
      alias_compose_kernel<<<(ng + 3) / 4, 128, 0, st>>>(s, nc, ng, status);
    }
    alias_walk_kernel<<<1, 32, 0, st>>>(s, nc, ng, status);
    if (nc) {
      alias_expand_kernel<<<(ng + 3) / 4, 128, 0, st>>>(s, nc, ng, status);
      alias_emit_kernel<<<(nc + 3) / 4, 128, 0, st>>>(s, nc, status);
    }
    alias_drain_kernel<<<(unsigned)sm_count * 4, 256, 0, st>>>(s, status);
    if (shots)
      alias_draw_kernel<<<(shots + 255) / 256, 256, 0, st>>>(s, len - 1, (const uint64_t*)variates, shots, out, status);
    *launches = (nc ? 10 : 5) + (shots ? 1 : 0);
    return cudaGetLastError();
  }
  char* p = (char*)scratch;
  const uint32_t nb = (uint32_t)((len + CUM_BLOCK - 1) / CUM_BLOCK);
  CumScratch c;
  c.bsum = (double*)p; p += ((size_t)nb + 1) * 8;
  p = align_up(p, 16);
  c.norm = (double*)p; p += 16;
  c.namb = (uint32_t*)p; p += 16;
  c.seq = (double*)p; p += 16;
  c.amb = (uint32_t*)p;
  p = align_up((char*)(c.amb + shots), 16);
  const uint32_t nch = n <= EXACT_MAX_N ? (uint32_t)((len + SEQ_CH - 1) / SEQ_CH) : 0u;
  c.ck = (double*)p; p += (size_t)nch * 8;
  c.fn = (SeqFn*)align_up(p, 16); p = (char*)(c.fn + nch);
  c.fe = (int*)p; p += (size_t)nch * 4;
  c.part = (double*)align_up(p, 16); p = (char*)(c.part + PREFIX_T);
  c.sfn = (SeqFn*)align_up(p, 16); p = (char*)(c.sfn + PREFIX_T);
  c.sstart = (double*)p; p += PREFIX_T * 8;
  c.sfe = (int*)p; p += PREFIX_T * 4;
  if ((size_t)(p - (char*)scratch) > scratch_bytes) return cudaErrorInvalidValue;
  cudaMemsetAsync(c.norm, 0, 48, st);  // norm, namb, seq
  if (f64) cum_blocks_kernel<double><<<nb, 256, 0, st>>>((const double2*)amps, len, c);
  else cum_blocks_kernel<float><<<nb, 256, 0, st>>>((const float2*)amps, len, c);
  if (nb <= PREFIX_T) {
    uint32_t threads = 32;
    while (threads < nb) threads *= 2;
    cum_prefix_kernel<true><<<1, threads, 0, st>>>(c, nb, tol, status);
    *launches = 2;
  } else {
    cum_range_kernel<<<PREFIX_T / RANGE_T, RANGE_T, 0, st>>>(c, nb);
    cum_prefix_kernel<false><<<1, PREFIX_T, 0, st>>>(c, nb, tol, status);
    cum_spread_kernel<<<PREFIX_T / RANGE_T, RANGE_T, 0, st>>>(c, nb);
    *launches = 4;
  }
  if (shots) {
    const unsigned wb = (shots + 3) / 4;  // a warp per shot
    const double* u = (const double*)variates;
    if (f64) cum_draw_kernel<double><<<wb, 128, 0, st>>>((const double2*)amps, len, nb, c, u, shots, out);
    else cum_draw_kernel<float><<<wb, 128, 0, st>>>((const float2*)amps, len, nb, c, u, shots, out);
    // status[2]: the shots inside the guard band (re-resolved below when n <= EXACT_MAX_N)
    cudaMemcpyAsync(status + 2, c.namb, 4, cudaMemcpyDeviceToDevice, st);
    *launches += 1;
    if (n <= EXACT_MAX_N) {
      // one chunk needs no function, and up to a segment each need no composition
      const bool fn = nch > 1, compose = nch > PREFIX_T;
      if (fn && f64) cum_fn_kernel<double><<<nch, 256, 0, st>>>((const double2*)amps, len, c);
      else if (fn) cum_fn_kernel<float><<<nch, 256, 0, st>>>((const float2*)amps, len, c);
      if (compose) cum_compose_kernel<<<PREFIX_T / RANGE_T, RANGE_T, 0, st>>>(c, nch);
      if (f64) cum_walk_kernel<double><<<1, WALK_T, 0, st>>>((const double2*)amps, len, nch, c);
      else cum_walk_kernel<float><<<1, WALK_T, 0, st>>>((const float2*)amps, len, nch, c);
      if (compose) cum_expand_kernel<<<PREFIX_T / RANGE_T, RANGE_T, 0, st>>>(c, nch);
      if (f64) cum_exact_kernel<double><<<wb, 128, 0, st>>>((const double2*)amps, len, c, u, out, status);
      else cum_exact_kernel<float><<<wb, 128, 0, st>>>((const float2*)amps, len, c, u, out, status);
      *launches += 2 + (fn ? 1 : 0) + (compose ? 2 : 0);
    }
  }
  return cudaGetLastError();
}

// ---- fixed scratch of aleph_b200_sample_cumulative_noalloc ----------------------
// Reserved when this module is loaded on a device, so the entry point that
// uses it never allocates. One copy per device; calls that overlap on one
// device share it.
static __device__ __align__(256) unsigned char g_fixed_sample_scratch[kFixedSampleScratchBytes + kFixedChunkFnBytes];

cudaError_t fixed_sample_scratch_address(void** out) {
  return cudaGetSymbolAddress(out, g_fixed_sample_scratch);
}

}  // namespace ab
