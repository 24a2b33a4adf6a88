// Persistent block-Jacobi PCG with one tagged grid reduction per iteration (sm_103a).
//
// What bounds the other persistent form (cg_persistent.cu) is not the matrix stream but the two grid barriers of an
// iteration, each a chain of five L2 round trips (partial, fence, arrival, poll, partials), the gathers of two vectors
// per neighbour, and -- below a few thousand rows -- that a row is one thread's serial work on a handful of SMs.  Here:
//   * rows are split evenly and contiguously over one CTA per SM.  A CTA keeps p of its own rows and of every row its
//     blocks refer to (its halo, listed once per pattern by halo_plan_kernel) in shared memory and addresses it with 16-bit
//     local indices, so a neighbour costs one shared-memory read per block and one L2 read per CTA;
//   * data carries its own arrival: a published row of p, and each published CTA sum, is a 128-bit word with the
//     iteration number inside, written and polled as one access.  No fence, no counter, no second read;
//   * an iteration has one reduction.  q = K p and w = M^-1 q give p.q, z.q, q.w, r.z and r.r together; then
//       alpha = rz / pq,  r'z' = rz - 2 alpha zq + alpha^2 qw,  beta = r'z' / rz
//     (r.z and r.r are formed from the vectors in every iteration, so nothing drifts; r, z, p and x follow the same
//     recurrences as the other forms).  r.r tells of the previous update: a solve ends one product later;
//   * the blocks of a CTA are contiguous in the sliced-ELL values; its warps take equal runs of block columns whatever
//     the slice boundaries, and a slice's partial products meet in shared memory in warp order.  As many block columns
//     as fit stay in shared memory for the whole solve, the rest are streamed by per-warp bulk copies;
//   * small systems cut slices into chunks of 4, 8 or 16 rows (one per CTA, everything resident), the lanes of a warp
//     taking several blocks of a row;
//   * sums are formed as aligned 64-bit integers with redux: GB300 retires two FP64 operations per clock and SM, and
//     a butterfly of doubles over 16 warps costs more than the products of a mid-sized system.  The alignment keeps
//     every summand to 2^-56 of the largest of its warp, 2^-53 of the largest warp sum and of the largest CTA sum, so a
//     total is as good as one of doubles; it does not depend on an order.
// Measured, microseconds per iteration, the best of the two-barrier forms -> this kernel:
//   rows        44            425           2 673         18 785        35 721        140 481
//   FP32    6.6 ->  3.7  13.6 ->  4.1  13.5 ->  4.5  14.1 ->  6.3  14.3 ->  8.1  29.1 -> 23.6
//   FP64   17.0 ->  4.9  36.4 ->  5.7  38.9 ->  6.8  39.7 -> 15.0  39.5 -> 24.4   127 ->   78
// Node numberings cost it less than the two-barrier forms (nodes shuffled throughout, 18 785 rows FP32 22.1 -> 7.2, FP64
// 41.2 -> 18.7; 35 721 rows 23.1 -> 14.5 and 41.2 -> 36.3, the closest of 50 combinations of size, numbering and
// precision; 80 625 rows shuffled within 512 nodes 27.1 -> 17.0 and 82 -> 53.5).
// The small sizes are bound by two trips through L2 (p to the neighbours, the sums to everyone) and the chains between
// them, FP64 from 18 785 rows on by the FP64 pipe (nine multiply-adds per block: 8, 15 and 54 us of the last three), FP32
// at 140 481 rows by the 118 MB of blocks streamed through L2, 72 MB of them from DRAM (45 % of the copy bandwidth); the
// other fifth of the matrix stays in shared memory.
// GROUPS: the same for many independent instances, a group of CTAs each (plan_halo in batched_host.cpp).  A load step
// of 128 instances in mixed precision (mean of four) 241 -> 131 ms, of 300 472 -> 291 ms, of 100 in FP64 (two) 789 -> 269 ms
// against the kernels of batched.cu.
// The launch is cooperative (all CTAs co-resident) and every wait is bounded: one that gives up ends the CTA with
// scal[kDone] = 6 after its copies in flight have been drained, and with it the waits of the others.
#include <algorithm>
#include <mutex>

#include "cg_grid.cuh"

namespace ikr {

namespace {

using namespace cg;

constexpr int kSums = 5;       // p.q, z.q, q.w, r.z, r.r
constexpr int kMaxCtas = 160;  // five partials per lane of the summing warps
// Every CTA polls every CTA's words: kept once, 152 readers queue at the few L2 lines that hold them (and the writers
// behind them: at 18 785 rows FP32 a poll phase of 4 800 cycles fell to 1 600).  A word is written kCopies times, one per
// lane, and a CTA reads one copy.
constexpr int kCopies = 8;
constexpr int kSmemBudget = 224 * 1024;
// A word travels to L2 and back in about 950 cycles, and a poll that finds it missing costs as much again: the first poll
// waits this many cycles after the own publication.  Microseconds per iteration with 0 / 300 / 450 / 600 cycles: 44 rows
// FP32 3.37 / 3.54 / 3.61 / 3.70 (eleven CTAs, hardly any skew), 425 rows 4.62 / 4.41 / 4.29 / 4.22, 18 785 rows 6.36 /
// 6.28 / 6.22 / 6.20, 140 481 rows 25.9 / 26.0 / 26.0 / 26.1.
constexpr int kPollDelay = 450;
constexpr int kMaxRing = 2;  // stages of streamed block columns per warp
template <typename T>
constexpr int unit_bytes() {
  return 288 * (int)sizeof(T) + 64;  // nine entries and a 16-bit local column of 32 lanes
}

// ---- 128-bit words with their arrival tag -----------------------------------------------------------------------
__device__ __forceinline__ void st_word(void* p, uint64_t lo, uint64_t hi) {
  asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p), "l"(lo),
               "l"(hi)
               : "memory");
}
__device__ __forceinline__ void ld_word(const void* p, uint64_t& lo, uint64_t& hi) {
  asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
               : "=l"(lo), "=l"(hi)
               : "l"(p)
               : "memory");
}
__device__ __forceinline__ uint64_t pack32(uint32_t lo, uint32_t hi) { return (uint64_t)lo | ((uint64_t)hi << 32); }

__device__ __forceinline__ void wait_cycles(int n) {
  const long long t = clock64();
  while (clock64() - t < n) {
  }
}

// a row of p: FP32 one word {x, y, z, tag}; FP64 two words {x, y low half, tag} and {z, y high half, tag}
__device__ __forceinline__ void publish_row(float* v, int row, float x, float y, float z, uint32_t tag) {
  st_word(v + 4 * (int64_t)row, pack32(__float_as_uint(x), __float_as_uint(y)), pack32(__float_as_uint(z), tag));
}
__device__ __forceinline__ void publish_row(double* v, int row, double x, double y, double z, uint32_t tag) {
  const uint64_t yb = (uint64_t)__double_as_longlong(y);
  st_word(v + 4 * (int64_t)row, (uint64_t)__double_as_longlong(x), pack32((uint32_t)yb, tag));
  st_word(v + 4 * (int64_t)row + 2, (uint64_t)__double_as_longlong(z), pack32((uint32_t)(yb >> 32), tag));
}
__device__ __forceinline__ bool fetch_row(const float* v, int row, uint32_t tag, float& x, float& y, float& z) {
  uint64_t lo, hi;
  ld_word(v + 4 * (int64_t)row, lo, hi);
  x = __uint_as_float((uint32_t)lo), y = __uint_as_float((uint32_t)(lo >> 32)), z = __uint_as_float((uint32_t)hi);
  return (uint32_t)(hi >> 32) == tag;
}
__device__ __forceinline__ bool fetch_row(const double* v, int row, uint32_t tag, double& x, double& y, double& z) {
  uint64_t a, b, c, d;
  ld_word(v + 4 * (int64_t)row, a, b);
  ld_word(v + 4 * (int64_t)row + 2, c, d);
  x = __longlong_as_double((long long)a), z = __longlong_as_double((long long)c);
  y = __longlong_as_double((long long)pack32((uint32_t)b, (uint32_t)d));
  return (uint32_t)(b >> 32) == tag && (uint32_t)(d >> 32) == tag;
}

// ---- sums as aligned integers -----------------------------------------------------------------------------------
// A number S * 2^x; normalised |S| in [2^60, 2^61).  Zero has the exponent kZeroExp, an infinity or NaN kBadExp.
struct Num {
  long long S;
  int x;
};
constexpr int kZeroExp = -20000, kBadExp = 20000;

// mantissa of 53 bits (a float's 24 bits at the top of them) and its exponent
__device__ __forceinline__ Num num_of(double v) {
  const long long b = __double_as_longlong(v);
  const int e = (int)((b >> 52) & 2047);
  long long m = (b & 0xfffffffffffffll) | (e ? 1ll << 52 : 0);
  if (b < 0) m = -m;
  return {m, e == 2047 ? kBadExp : m == 0 ? kZeroExp : (e ? e : 1) - 1075};
}
__device__ __forceinline__ Num num_of(float v) {
  const uint32_t b = __float_as_uint(v);
  const int e = (int)((b >> 23) & 255u);
  const uint32_t f = (b & 0x7fffffu) | (e ? 1u << 23 : 0u);
  long long m = (long long)f << 29;
  if ((int32_t)b < 0) m = -m;
  return {m, e == 255 ? kBadExp : f == 0 ? kZeroExp : (e ? e : 1) - 179};
}
__device__ __forceinline__ long long shift_right(long long m, int sh) { return m >> (sh < 63 ? sh : 63); }
// Sum over the lanes of m * 2^x, in every lane, normalised.  |m| < 2^58: of 32 summands 2^63 is the bound.  One copy of
// this code serves the eight sums of an iteration: the loop body has to stay in the instruction cache (inlined, the
// kernel took 56 KB and every phase run by one warp waited for its instructions).
__device__ __noinline__ Num warp_sum(long long m, int x) {
  __syncwarp();
  const int X = __reduce_max_sync(0xffffffffu, x);
  const long long a = shift_right(m, X - x);
  // 27 + 27 bits and the signed rest
  const uint32_t lo = __reduce_add_sync(0xffffffffu, (uint32_t)a & 0x7ffffffu);
  const uint32_t mid = __reduce_add_sync(0xffffffffu, (uint32_t)(a >> 27) & 0x7ffffffu);
  const int hi = __reduce_add_sync(0xffffffffu, (int)(a >> 54));
  const long long S = (long long)lo + ((long long)mid << 27) + ((long long)hi << 54);
  if (X == kBadExp || S == 0) return {0, X == kBadExp ? kBadExp : kZeroExp};
  const int k = __clzll(S < 0 ? ~S : S) - 3;  // the highest bit goes to bit 60
  return {k >= 0 ? S << k : S >> 1, X - (k >= 0 ? k : -1)};
}
// S / 16 * 2^x, |S| < 2^58: what the warp sums take
struct Num16 {
  long long S;
  int x;
};
template <typename T>
__device__ __forceinline__ Num16 num16_of(T v) {
  const Num u = num_of(v);
  return {u.S * 16, u.x};
}
__device__ __forceinline__ Num16 num16_of(Num16 v) { return v; }
// Exact squares of floats, summed to 56 bits of the largest: at most 16 squares of 48 bits, ten bits up.  (Two floats, the
// square and its rounding error, underflow below 1e-19 and have 48 bits; a conversion and an addition in FP64 per square
// load GB300's narrow FP64 pipe.)
struct SquareSum {
  long long S = 0;
  int x = kZeroExp;
  __device__ __forceinline__ void add(float v) {
    const uint32_t b = __float_as_uint(v);
    const int e = (int)((b >> 23) & 255u);
    const uint32_t f = (b & 0x7fffffu) | (e ? 1u << 23 : 0u);
    const int xv = e == 255 ? kBadExp : f == 0 ? kZeroExp : 2 * (e ? e : 1) - 310, X = x > xv ? x : xv;
    S = shift_right(S, X - x) + shift_right((long long)((uint64_t)f * f << 10), X - xv);
    x = X;
  }
  __device__ __forceinline__ Num16 num16() const {
    if (x == kBadExp || S == 0) return {0, x};
    const int k = __clzll(S) - 6;  // the highest bit goes to bit 57
    return {k >= 0 ? S << k : S >> -k, x + 4 - k};
  }
};
// Warp sums of three values at once (the redux chains overlap), as S * 2^x with |S| < 2^62, to slot `warp` of the CTA's
// lists S[k * stride], x[k * stride].  The second may be a SquareSum's.
template <typename T, typename U>
__device__ __noinline__ void warp_parts(T v0, U v1, T v2, long long* S, int* x, int stride) {
  __syncwarp();
  const Num16 u[3] = {num16_of(v0), num16_of(v1), num16_of(v2)};
  int X[3];
  uint32_t lo[3], mid[3];
  int hi[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) X[k] = __reduce_max_sync(0xffffffffu, u[k].x);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const long long a = shift_right(u[k].S, X[k] - u[k].x);
    lo[k] = __reduce_add_sync(0xffffffffu, (uint32_t)a & 0x7ffffffu);
    mid[k] = __reduce_add_sync(0xffffffffu, (uint32_t)(a >> 27) & 0x7ffffffu);
    hi[k] = __reduce_add_sync(0xffffffffu, (int)(a >> 54));
  }
  if ((threadIdx.x & 31) == 0) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      S[k * stride] = (long long)lo[k] + ((long long)mid[k] << 27) + ((long long)hi[k] << 54);
      x[k * stride] = X[k];  // of the values; S carries four more bits
    }
  }
  __syncwarp();
}
__device__ __forceinline__ double to_double(const Num& u) {
  if (u.x == kBadExp) return __longlong_as_double(0x7ff8000000000000ll);
  if (u.S == 0) return 0.0;
  const long long b = __double_as_longlong(__ll2double_rn(u.S));
  const int e = (int)((b >> 52) & 2047) + u.x;
  if (e <= 0) return 0.0;
  if (e >= 2047) return __longlong_as_double((b & (1ll << 63)) | 0x7ff0000000000000ll);
  return __longlong_as_double((b & 0x800fffffffffffffll) | ((long long)e << 52));
}

// Independent instances of one element set, a group of CTAs each (the GROUPS form of the kernel): CTA b is number
// b - first[b] of the size[b] that serve instance inst[b], whose rows are [node_off[inst], node_off[inst + 1]).  The slices
// an instance's rows touch are split evenly over its group; lanes of other instances' rows compute along unseen.
struct HaloGroups {
  const int32_t *inst, *first, *size, *node_off;
  const double* rtol;  // per instance
  int max_iter, chunk;  // an instance's iterations in all and in one launch
  void* p;              // p between the launches of a solve (node-padded)
  double* st;           // four per instance, the third b.b
  int32_t *its, *flag;
  double *relres, *x_out;
};
struct GroupRows {
  int s0, ns, lo, hi;  // slices and rows [lo, hi) of a CTA
};
__device__ __forceinline__ GroupRows group_rows(const HaloGroups& g, int b) {
  const int i = g.inst[b], r0 = g.node_off[i], r1 = g.node_off[i + 1], sa = r0 >> 5, n = ((r1 - 1) >> 5) - sa + 1;
  const int k = b - g.first[b], m = g.size[b];
  const int a = sa + (int)((int64_t)k * n / m), e = sa + (int)((int64_t)(k + 1) * n / m);
  return {a, e - a, max(r0, 32 * a), min(r1, 32 * e)};
}

template <typename T>
struct HaloArgs {
  HaloPlan P;
  Bsr A;
  const T* val;
  const T* minv;
  T* x;
  const T* r;
  const T* z;
  T* p;          // published rows, zeroed by the init kernel
  double* part;  // 2 parities x kSums x kCopies x kMaxCtas words, zeroed by the init kernel
  double* scal;
  int64_t keep_g;
  WaitCtl wc;
  // shared memory: elements of a p component and of a component of the partial products, resident block columns per
  // warp, stages of the stream per warp
  int np, qstride, resident, ring;
  HaloGroups g;
};

// Who owns a row in the vector part of an iteration.  Small systems (CB = 0): warps in tens of rows, lane 3 k + c holding
// component c of row k (lanes 30 and 31 idle), so that the dependent FP64 instructions, about 60 cycles each, are a third
// as many.  Streamed ones: a lane per row, which takes fewer instructions.  MAXP: passes of WARPS x 10 or 32 rows.
constexpr int rows_per_warp(bool streamed) { return streamed ? 32 : 10; }

// CB: streamed block columns per stage; 0: everything is resident and the code of the stream is left out, which keeps
// the loop body of the latency-bound sizes small.
template <typename T, int WARPS, int MAXP, int CB, bool GROUPS>
__global__ void __launch_bounds__(WARPS * 32, 1) pcg_halo_kernel(const __grid_constant__ HaloArgs<T> H) {
  constexpr int kThreads = WARPS * 32;
  constexpr int kValBytes = 288 * (int)sizeof(T), kColBytes = 64, kUnitBytes = unit_bytes<T>();
  constexpr bool STREAM = CB > 0;
  constexpr int kUnits = STREAM ? CB : 1;
  constexpr int NC = STREAM ? 3 : 1;  // components of a row that a lane holds
  constexpr int kRowsPerWarp = rows_per_warp(STREAM);
  // the inverse blocks of a lane's rows in registers where the register file allows it
  constexpr bool kRegM = MAXP * NC * sizeof(T) <= 24;
  constexpr int kBatch = STREAM ? 4 : 2;  // halo rows a thread fetches at a time (6: 1.4 us slower at 140 481 rows)
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ __align__(8) uint64_t bars[WARPS][STREAM ? kMaxRing : 1];
  __shared__ long long swS[kSums + 1][WARPS];  // the warps' sums
  __shared__ int swx[kSums + 1][WARPS];
  __shared__ double ssum[kSums], srec[2];  // the grid's sums; 1 / p.q and 1 / r.z
  __shared__ T s_ab[2];
  __shared__ int s_done;
  __shared__ int s_fail;

  const HaloPlan& P = H.P;
  const Bsr& A = H.A;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int G = GROUPS ? H.g.size[blockIdx.x] : gridDim.x, cta = GROUPS ? blockIdx.x - H.g.first[blockIdx.x] : blockIdx.x;
  const int ch = GROUPS ? 32 : P.chunk;
  double* part = GROUPS ? H.part + 2 * H.g.first[blockIdx.x] : H.part;

  // layout: units (resident, then the ring), p components, partial products, halo rows, slice offsets
  const int resident = H.resident;
  const int nring = STREAM ? H.ring : 0;  // stages per warp
  const int warp_units = resident + nring * kUnits;
  unsigned char* wunit = smem + (size_t)warp * warp_units * kUnitBytes;
  T* px = reinterpret_cast<T*>(smem + (size_t)WARPS * warp_units * kUnitBytes);
  T* py = px + H.np;
  T* pz = py + H.np;
  T* qp = pz + H.np;
  const int qstride = H.qstride;
  int* hl = reinterpret_cast<int*>(qp + 3 * qstride);
  int* soff = hl + P.max_halo;

  // own rows [row0, row0 + m), slices [s0, s0 + ns), units (block columns, or chunks of them) [0, ng)
  // (GROUPS: the rows start at row0 + off, and local rows below off are another CTA's)
  int row0, m, s0, ns, ng, off = 0;
  if constexpr (GROUPS) {
    const GroupRows q = group_rows(H.g, blockIdx.x);
    s0 = q.s0, ns = q.ns, row0 = 32 * s0, off = q.lo - row0, m = q.hi - row0;
#pragma unroll 1
    for (int i = tid; i <= ns; i += kThreads) soff[i] = A.slice_off[s0 + i] - A.slice_off[s0];
    ng = A.slice_off[s0 + ns] - A.slice_off[s0];
  } else if (ch == 32) {
    s0 = P.slice0[cta];
    ns = P.slice0[cta + 1] - s0;
    row0 = 32 * s0;
    m = min(32 * ns, A.n_rows - row0);
#pragma unroll 1
    for (int i = tid; i <= ns; i += kThreads) soff[i] = A.slice_off[s0 + i] - A.slice_off[s0];
    ng = A.slice_off[s0 + ns] - A.slice_off[s0];
  } else {
    row0 = cta * ch;
    s0 = row0 >> 5;
    ns = 1;
    m = min(ch, A.n_rows - row0);
    ng = ((A.slice_off[s0 + 1] - A.slice_off[s0]) * ch + 31) / 32;
    if (tid == 0) soff[0] = 0, soff[1] = ng;
  }
  const int64_t g0 = A.slice_off[s0];  // first block column (chunk 32)
  const int nh = P.halo_cnt[blockIdx.x];
#pragma unroll 1
  for (int i = tid; i < nh; i += kThreads) hl[i] = P.halo[(int64_t)blockIdx.x * P.halo_cap + i];
  const int per = (ng + WARPS - 1) / WARPS;
  const int ub = min(ng, warp * per), ue = min(ng, ub + per);  // this warp's units
  const int ures = min(ue, ub + resident);                     // [ub, ures) resident, [ures, ue) streamed
  const int nwr = min(WARPS, (m + kRowsPerWarp - 1) / kRowsPerWarp);  // warps with rows

  // resident units
#pragma unroll 1
  for (int u = ub; u < ures; ++u) {
    T* dv = reinterpret_cast<T*>(wunit + (size_t)(u - ub) * kUnitBytes);
    uint16_t* dc = reinterpret_cast<uint16_t*>(wunit + (size_t)(u - ub) * kUnitBytes + kValBytes);
    if (ch == 32) {
      const T* sv = H.val + (g0 + u) * 288;
#pragma unroll
      for (int e = 0; e < 9; ++e) dv[32 * e + lane] = __ldg(sv + 32 * e + lane);
      dc[lane] = P.col16[(g0 + u) * 32 + lane];
    } else {
      const int row = row0 + (lane & (ch - 1)), k = u * (32 / ch) + lane / ch;
      const bool in = row < A.n_rows && k < A.slice_off[s0 + 1] - (int)g0;
      const int64_t b = (g0 + k) * 32 + (row & 31);
#pragma unroll
      for (int e = 0; e < 9; ++e) dv[32 * e + lane] = in ? __ldg(H.val + block_entry(b, e)) : T(0);
      dc[lane] = in ? P.col16[b] : uint16_t(0);
    }
  }
  __syncthreads();  // soff

  // CG state of this lane's components of its rows
  const int rl = STREAM ? lane : lane / 3, comp = STREAM ? 0 : lane - 3 * rl;
  auto row_of = [&](int j) { return (j * WARPS + warp) * kRowsPerWarp + rl; };
  auto owns = [&](int j) { return (STREAM || lane < 30) && row_of(j) < m && (!GROUPS || row_of(j) >= off); };
  T xr[MAXP][NC], rr[MAXP][NC], zr[MAXP][NC], pr[MAXP][NC], qr[MAXP][NC];
  T mi[kRegM ? MAXP : 1][3 * NC];
  int qfrom[MAXP];  // first partial product of the row (index into qp) and, above bit 20, their number
#pragma unroll
  for (int j = 0; j < MAXP; ++j) {
    const int i = row_of(j);
    const bool own = owns(j);
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      rr[j][c] = own ? H.r[4 * (int64_t)(row0 + i) + comp + c] : T(0);
      zr[j][c] = pr[j][c] = own ? H.z[4 * (int64_t)(row0 + i) + comp + c] : T(0);
      xr[j][c] = qr[j][c] = T(0);
      if (GROUPS && own) {
        pr[j][c] = static_cast<const T*>(H.g.p)[4 * (int64_t)(row0 + i) + comp + c];
        xr[j][c] = H.x[4 * (int64_t)(row0 + i) + comp + c];
      }
    }
    if constexpr (kRegM) {
#pragma unroll
      for (int k = 0; k < 3 * NC; ++k) mi[j][k] = own ? __ldg(H.minv + 9 * (int64_t)(row0 + i) + 3 * comp + k) : T(0);
    }
    qfrom[j] = 0;
    if (own) {
      const int s = ch == 32 ? i >> 5 : 0;
      const int wf = soff[s] / per, wl = (soff[s + 1] - 1) / per;
      qfrom[j] = ((wf + s) * 32 + (i & 31)) | ((soff[s + 1] > soff[s] ? wl - wf + 1 : 0) << 20);
    }
  }
  // this lane's components of M^-1 v; zero where the lane owns nothing
  auto precond = [&](int j, const T (&v)[NC], T (&y)[NC]) {
    T u[3];
    if constexpr (STREAM) {
#pragma unroll
      for (int c = 0; c < 3; ++c) u[c] = v[c];
    } else {
#pragma unroll
      for (int c = 0; c < 3; ++c) u[c] = __shfl_sync(0xffffffffu, v[0], lane - comp + c);
    }
    const T* q = H.minv + 9 * (int64_t)(row0 + (owns(j) ? row_of(j) : 0)) + 3 * comp;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      if constexpr (kRegM) {
        y[c] = mi[j][3 * c] * u[0] + mi[j][3 * c + 1] * u[1] + mi[j][3 * c + 2] * u[2];
      } else {
        y[c] = __ldg(q + 3 * c) * u[0] + __ldg(q + 3 * c + 1) * u[1] + __ldg(q + 3 * c + 2) * u[2];
        if (!owns(j)) y[c] = T(0);
      }
    }
  };
  double tol2, rrs = 0.0, rz = 0.0, beta = 0.0;  // thread 0's
  int maxit, it, done, it_end = 0;
  if constexpr (GROUPS) {
    const int i = H.g.inst[blockIdx.x];
    tol2 = H.g.rtol[i] * H.g.rtol[i] * H.g.st[4 * i + 2];
    maxit = H.g.max_iter;
    it = H.g.its[i];
    it_end = it + H.g.chunk;
    done = 0;
  } else {
    tol2 = H.scal[kTol2];
    maxit = (int)H.scal[kMaxIt];
    rrs = H.scal[kRR], rz = H.scal[kRz];
    it = (int)H.scal[kIters];
    done = (int)H.scal[kDone];
  }
  if (tid == 0) s_fail = 0;

  T* pown = comp == 0 ? px : comp == 1 ? py : pz;  // (a lane per component)
  // the words of sum k for iteration `tag` - 1 in copy c, and one warp forming the CTA's sum from the warps' and
  // writing its word to every copy
  auto sum_words = [&](int k, uint32_t tag, int c) {
    return part + 2 * ((((tag - 1u) & 1u) * kSums + k) * kCopies + c) * kMaxCtas;
  };
  auto publish_sum = [&](int k, uint32_t tag) {
    // (selects, no branch: a warp that enters the sum diverged takes two thousand cycles for it)
    const int l = lane < nwr ? lane : 0;
    const Num t = warp_sum(lane < nwr ? swS[k][l] >> 4 : 0, lane < nwr ? swx[k][l] : kZeroExp);
    if (lane < kCopies && (GROUPS || !(H.wc.withhold_first && cta == 0 && tag == 1u)))
      st_word(sum_words(k, tag, lane) + 2 * cta, (uint64_t)t.S, pack32((uint32_t)t.x, tag));
  };

  // streamed units: copies of this warp's cyclic sequence, nring stages ahead
  unsigned char* ring = wunit + (size_t)resident * kUnitBytes;
  const bool streams = STREAM && ures < ue;
  if (STREAM && lane == 0) {
#pragma unroll 1
    for (int st = 0; st < nring; ++st) mbar_init(smem_addr(&bars[warp][st]), 1);
    mbar_init_fence();
  }
  __syncwarp();
  const uint32_t keep16 = (uint32_t)(65536.0 * 32.0 * (double)H.keep_g / (double)A.n_padded);
  auto issue = [&](int st, int u) {
    if (lane == 0) {
      const int64_t g = g0 + u;
      const uint32_t b = smem_addr(&bars[warp][st]);
      const uint32_t nb = min(kUnits, ue - u);
      unsigned char* d = ring + (size_t)st * kUnits * kUnitBytes;
      // the stages kept in L2 are spread over the run (a low-discrepancy sequence), so that reads from DRAM and from L2
      // overlap: with the kept ones first, an iteration at 140 481 rows FP32 took 25.3 us, so 23.3
      const uint64_t pol = l2_policy((((uint32_t)((u - ures) / kUnits) * 2654435769u) >> 16) < keep16);
      mbar_expect_tx(b, nb * kUnitBytes);
      bulk_g2s(smem_addr(d), H.val + g * 288, nb * kValBytes, b, pol);
      bulk_g2s(smem_addr(d + kUnits * kValBytes), P.col16 + g * 32, nb * kColBytes, b, pol);
    }
  };
  int unext = ures, st = 0;
  uint32_t phase = 0;
  const bool started = done == 0;
  if (streams && started)
#pragma unroll 1
    for (int k = 0; k < nring; ++k) {
      issue(k, unext);
      unext = unext + kUnits >= ue ? ures : unext + kUnits;
    }

  // slice of the warp's first unit and the end of that slice
  int sfirst = 0;
  while (ub < ue && soff[sfirst + 1] <= ub) ++sfirst;
  const int sfirst_end = ub < ue ? soff[sfirst + 1] : 0;

  bool failed = false;

  while (done == 0) {
    const uint32_t tag = (uint32_t)it + 1u;
    // ---- p of the own rows first: the neighbours wait for it
#pragma unroll
    for (int j = 0; j < MAXP; ++j) {
      if (MAXP > 1 && j * WARPS * kRowsPerWarp >= m) break;
      if constexpr (STREAM) {
        if (owns(j)) {
          const int i = row_of(j);
          publish_row(H.p, row0 + i, pr[j][0], pr[j][1], pr[j][2], tag);
          px[i] = pr[j][0], py[i] = pr[j][1], pz[i] = pr[j][2];
        }
      } else {
        const T v1 = __shfl_down_sync(0xffffffffu, pr[j][0], 1), v2 = __shfl_down_sync(0xffffffffu, pr[j][0], 2);
        if (owns(j)) {
          if (comp == 0) publish_row(H.p, row0 + row_of(j), pr[j][0], v1, v2, tag);
          pown[row_of(j)] = pr[j][0];
        }
      }
    }
    // ---- halo: every row once, polled until it carries this iteration's tag; without a stream (registers) the first
    // batch's reads travel while the sums are formed
    T vx[kBatch], vy[kBatch], vz[kBatch];
    unsigned pend = 0;
    auto fetch = [&](int i0) {
#pragma unroll
      for (int j = 0; j < kBatch; ++j)
        if ((pend >> j) & 1u)
          if (fetch_row(H.p, hl[i0 + j * kThreads], tag, vx[j], vy[j], vz[j])) pend &= ~(1u << j);
    };
    auto wanted = [&](int i0) {
#pragma unroll
      for (int j = 0; j < kBatch; ++j)
        if (i0 + j * kThreads < nh) pend |= 1u << j;
    };
    wait_cycles(kPollDelay);
    wanted(tid);
    bool got[kBatch];
#pragma unroll
    for (int j = 0; j < kBatch; ++j) {
      got[j] = false;
      if (!STREAM && ((pend >> j) & 1u)) got[j] = fetch_row(H.p, hl[tid + j * kThreads], tag, vx[j], vy[j], vz[j]);
    }
    if (warp < nwr) {
      // GROUPS in FP32: r.r of exact squares, to more than FP64's bits and in a wider range than FP32's (the instances'
      // tolerances go down to where 24 bits of a lane's squares would show)
      constexpr bool kExact = GROUPS && sizeof(T) == 4;
      static_assert(MAXP * NC <= 16, "squares of a lane");
      T srz = T(0), srr = T(0);
      SquareSum sq;
#pragma unroll
      for (int j = 0; j < MAXP; ++j)  // zero where the lane owns nothing
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          srz += rr[j][c] * zr[j][c];
          if constexpr (kExact) sq.add(rr[j][c]);
          else srr += rr[j][c] * rr[j][c];
        }
      if constexpr (kExact) warp_parts<T>(srz, sq.num16(), T(0), &swS[3][warp], &swx[3][warp], WARPS);
      else warp_parts<T>(srz, srr, T(0), &swS[3][warp], &swx[3][warp], WARPS);
    }
#pragma unroll
    for (int j = 0; j < kBatch; ++j)
      if (got[j]) pend &= ~(1u << j);
#pragma unroll 1
    for (int i0 = tid; i0 < nh; i0 += kBatch * kThreads) {
      if (i0 != tid) wanted(i0);
#pragma unroll 1
      for (int k = 0; pend && k < H.wc.polls; ++k) {
        if (k > 64) __nanosleep(16);
        fetch(i0);
      }
      if (pend) failed = true;
      pend = 0;
#pragma unroll
      for (int j = 0; j < kBatch; ++j) {
        const int i = i0 + j * kThreads;
        if (i < nh) px[m + i] = vx[j], py[m + i] = vy[j], pz[m + i] = vz[j];
      }
    }
    if (__syncthreads_or(failed)) {
      failed = true;
      break;
    }
    // r.z and r.r are known before the product: their words travel while it runs
    if (warp >= WARPS - 2) publish_sum(3 + warp - (WARPS - 2), tag);
    // ---- q = K p: this warp's units, partial products per (warp, slice)
    if (ub < ue) {
      int s = sfirst, snext = sfirst_end;
      T a0 = T(0), a1 = T(0), a2 = T(0);
      auto product = [&](const unsigned char* vals, const unsigned char* cols) {
        const T* v = reinterpret_cast<const T*>(vals) + lane;
        int c = reinterpret_cast<const uint16_t*>(cols)[lane];
        if (GROUPS) c = min(c, H.np - 1);  // another CTA's row of a shared slice: its column means nothing here
        const T x0 = px[c], x1 = py[c], x2 = pz[c];
        // one multiply-add per entry: as a sum of three products the row would cost a fourth instruction, and nine FP64
        // instructions per block are what bounds the FP64 form
        a0 = fma(v[0], x0, a0), a1 = fma(v[96], x0, a1), a2 = fma(v[192], x0, a2);
        a0 = fma(v[32], x1, a0), a1 = fma(v[128], x1, a1), a2 = fma(v[224], x1, a2);
        a0 = fma(v[64], x2, a0), a1 = fma(v[160], x2, a1), a2 = fma(v[256], x2, a2);
      };
      auto flush = [&]() {
        T* d = qp + (warp + s) * 32 + lane;
        d[0] = a0, d[qstride] = a1, d[2 * qstride] = a2;
        a0 = a1 = a2 = T(0);
      };
      auto next = [&](int u) {  // after unit u
        while (u + 1 == snext && u + 1 < ue) {
          flush();
          ++s;
          snext = soff[s + 1];
        }
      };
#pragma unroll 2
      for (int u = ub; u < ures; ++u) {
        const unsigned char* d = wunit + (size_t)(u - ub) * kUnitBytes;
        product(d, d + kValBytes);
        next(u);
      }
#pragma unroll 1
      for (int u = ures; STREAM && u < ue; u += kUnits) {
        if (!__all_sync(0xffffffffu, mbar_wait_bounded(smem_addr(&bars[warp][st]), (phase >> st) & 1u))) {
          failed = true;
          break;
        }
        phase ^= 1u << st;
        const unsigned char* d = ring + (size_t)st * kUnits * kUnitBytes;
#pragma unroll
        for (int k = 0; k < kUnits; ++k)
          if (u + k < ue) {
            product(d + k * kValBytes, d + kUnits * kValBytes + k * kColBytes);
            next(u + k);
          }
        __syncwarp();  // the stage is consumed before it is refilled
        issue(st, unext);
        unext = unext + kUnits >= ue ? ures : unext + kUnits;
        st = st + 1 == nring ? 0 : st + 1;
      }
      if (ch < 32) {  // lanes of one row
#pragma unroll 1
        for (int o = ch; o < 32; o <<= 1) {
          a0 += __shfl_xor_sync(0xffffffffu, a0, o);
          a1 += __shfl_xor_sync(0xffffffffu, a1, o);
          a2 += __shfl_xor_sync(0xffffffffu, a2, o);
        }
      }
      flush();
    }
    if (__syncthreads_or(failed)) {
      failed = true;
      break;
    }
    // ---- rows: q, w = M^-1 q, and p.q, z.q and q.w
    if (warp < nwr) {
      T spq = T(0), szq = T(0), sqw = T(0);
#pragma unroll
      for (int j = 0; j < MAXP; ++j) {
        if (MAXP > 1 && j * WARPS * kRowsPerWarp >= m) break;
        const T* d = qp + (qfrom[j] & 0xfffff) + comp * qstride;
        const int n = qfrom[j] >> 20;
        T w[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c) {  // a slice of a large system has one or two
          qr[j][c] = n > 0 ? d[c * qstride] : T(0);
          if (n > 1) qr[j][c] += d[c * qstride + 32];
        }
#pragma unroll 1
        for (int k = 2; k < n; ++k)
#pragma unroll
          for (int c = 0; c < NC; ++c) qr[j][c] += d[c * qstride + 32 * k];
        precond(j, qr[j], w);
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          spq += pr[j][c] * qr[j][c];
          szq += zr[j][c] * qr[j][c];
          sqw += qr[j][c] * w[c];
        }
      }
      warp_parts<T>(spq, szq, sqw, &swS[0][warp], &swx[0][warp], WARPS);
    }
    __syncthreads();
    // ---- grid sums: warps 0 .. 2 publish this CTA's, warps 0 .. 4 collect everyone's
    if (warp < kSums) {
      if (warp < 3) {
        publish_sum(warp, tag);
        wait_cycles(kPollDelay);
      }
      const double* words = sum_words(warp, tag, cta & (kCopies - 1));
      Num t[kMaxCtas / 32];
      unsigned pend = 0;
#pragma unroll
      for (int j = 0; j < kMaxCtas / 32; ++j) {
        t[j] = {0, kZeroExp};
        if (lane + 32 * j < G) pend |= 1u << j;
      }
#pragma unroll 1
      for (int k = 0; pend && k < H.wc.polls; ++k) {
        if (k > 64) __nanosleep(16);
        uint64_t lo[kMaxCtas / 32], hi[kMaxCtas / 32];
#pragma unroll
        for (int j = 0; j < kMaxCtas / 32; ++j)
          if ((pend >> j) & 1u) ld_word(words + 2 * (lane + 32 * j), lo[j], hi[j]);
#pragma unroll
        for (int j = 0; j < kMaxCtas / 32; ++j)
          if (((pend >> j) & 1u) && (uint32_t)(hi[j] >> 32) == tag) {
            t[j] = {(long long)lo[j], (int)(uint32_t)hi[j]};
            pend &= ~(1u << j);
          }
      }
      if (__any_sync(0xffffffffu, pend != 0) && lane == 0) s_fail = 1;
      __syncwarp();
      // five normalised numbers below 2^61 per lane, a sixty-fourth of each: below 2^57.4, inside warp_sum's bound
      int X = kZeroExp;
#pragma unroll
      for (int j = 0; j < kMaxCtas / 32; ++j) X = max(X, t[j].x);
      long long a = 0;
#pragma unroll
      for (int j = 0; j < kMaxCtas / 32; ++j) a += shift_right(t[j].S >> 6, X - t[j].x);
      const Num g = warp_sum(a, X == kBadExp ? kBadExp : X + 6);
      if (lane == 0) {
        const double v = to_double(g);
        ssum[warp] = v;
        if (warp == 0) srec[0] = 1.0 / v;
        if (warp == 3) srec[1] = 1.0 / v;  // off the critical path: r.z is here before p.q
      }
      asm volatile("bar.sync 1, %0;" ::"n"(kSums * 32) : "memory");
      if (tid == 0) {
        const double pq = ssum[0], zq = ssum[1], qw = ssum[2];
        auto exponent = [](double v) { return (int)((__double_as_longlong(v) >> 52) & 2047); };
        const int ex = exponent(pq);
        rz = ssum[3];
        rrs = ssum[4];
        int d = 0;
        double alpha = 0.0;
        // rrs and tol2 are not negative: their order is that of their bits (a NaN is above every number)
        if ((GROUPS || it > 0) && __double_as_longlong(rrs) <= __double_as_longlong(tol2)) d = 1;
        else if ((GROUPS || it > 0) && it >= maxit) d = GROUPS ? 1 : 2;
        else if ((__double_as_longlong(pq) << 1) == 0 || ex == 2047) d = GROUPS ? 2 : 3;  // negative curvature alone does not stop CG
        else if (const int ez = exponent(rz); ex >= 64 && ex <= 1980 && ez >= 64 && ez <= 1980) {
          // in FP64 alpha's last bit is corrected beside beta.  (beta for the alpha that FP32 vectors are updated with, rounded,
          // costs 0.1 us and makes the solutions no more accurate: errors of 40 right-hand sides on 208 rows, root mean square,
          // 8.6e-5 with it, 8.7e-5 without, 8.3e-5 with beta as a quotient of two r.z in the two-barrier kernels)
          alpha = rz * srec[0];
          beta = fma(alpha * srec[1], fma(alpha, qw, -2.0 * zq), 1.0);
          if (sizeof(T) == 8) alpha = fma(fma(-alpha, pq, rz), srec[0], alpha);
        } else {  // sums near the ends of the range
          alpha = rz / pq;
          beta = 1.0 + (alpha * qw - 2.0 * zq) / pq;
        }
        s_ab[0] = T(alpha);
        s_ab[1] = T(beta);
        s_done = d;
      }
    }
    __syncthreads();
    if (s_fail) {
      failed = true;
      break;
    }
    done = s_done;
    if (done != 0) break;
    // ---- update of the own rows
    const T al = s_ab[0], be = s_ab[1];
    if (warp < nwr) {
#pragma unroll
      for (int j = 0; j < MAXP; ++j) {
        if (MAXP > 1 && j * WARPS * kRowsPerWarp >= m) break;
#pragma unroll
        for (int c = 0; c < NC; ++c) rr[j][c] -= al * qr[j][c];
        precond(j, rr[j], zr[j]);
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          xr[j][c] += al * pr[j][c];
          pr[j][c] = zr[j][c] + be * pr[j][c];
        }
      }
    }
    ++it;
    if (GROUPS && it == it_end) break;
  }

  // drain the copies in flight (the cyclic stream runs ahead of the last iteration)
  if (streams && started) {
#pragma unroll 1
    for (int k = 0; k < nring; ++k) {
      mbar_wait_bounded(smem_addr(&bars[warp][st]), (phase >> st) & 1u);
      phase ^= 1u << st;
      st = st + 1 == nring ? 0 : st + 1;
    }
  }
  if constexpr (GROUPS) {
    const int inst = H.g.inst[blockIdx.x];
    if (!failed) {
#pragma unroll
      for (int j = 0; j < MAXP; ++j)
        if (owns(j)) {
#pragma unroll
          for (int c = 0; c < NC; ++c) {
            const int64_t row = row0 + row_of(j), i = 4 * row + comp + c;
            if (done != 0) {
              H.g.x_out[3 * row + comp + c] = double(xr[j][c]);
            } else {  // continued by the next launch
              H.x[i] = xr[j][c];
              const_cast<T*>(H.r)[i] = rr[j][c];
              const_cast<T*>(H.z)[i] = zr[j][c];
              static_cast<T*>(H.g.p)[i] = pr[j][c];
            }
          }
        }
    }
    if (tid == 0 && (cta == 0 || failed)) {
      if (cta == 0 && !failed) {
        const double bb = H.g.st[4 * inst + 2];
        H.g.its[inst] = it;
        H.g.relres[inst] = bb > 0.0 ? sqrt(rrs / bb) : 0.0;
      }
      atomicMin(&H.g.flag[inst], failed ? -1 : done);  // the host sets it above every value before the launch
    }
    return;
  }
#pragma unroll
  for (int j = 0; j < MAXP; ++j)
    if (owns(j)) {
#pragma unroll
      for (int c = 0; c < NC; ++c) H.x[4 * (int64_t)(row0 + row_of(j)) + comp + c] = xr[j][c];
    }
  if (tid == 0 && (cta == 0 || failed)) {
    // a CTA that gave up says so itself, and CTA 0 may have finished before or after it: the largest status stays (as bits,
    // statuses are not negative)
    if (cta == 0) {
      H.scal[kIters] = (double)it;
      H.scal[kRR] = rrs;
      H.scal[kRz] = rz;
      H.scal[kBeta] = beta;
    }
    atomicMax(reinterpret_cast<long long*>(H.scal + kDone), __double_as_longlong(failed ? kDoneDeviceTimeout : (double)done));
  }
}

// ---- the pattern's plan: halo rows and 16-bit local columns, one CTA per CG CTA ---------------------------------
// own row r is local r - row0; a row outside is m + its rank among the CTA's halo rows (ascending): a bitmap of the
// referenced rows and the running count of its words give the rank
// (GROUPS: per CTA of an instance's group, among the instance's rows; a block of another CTA's row is left alone)
template <bool GROUPS>
__global__ void __launch_bounds__(1024) halo_plan_kernel(Bsr A, HaloPlan P, HaloGroups g, int32_t* slice0, int32_t* cnt,
                                                         int32_t* halo, uint16_t* col16) {
  extern __shared__ uint32_t sm[];
  __shared__ int wtot[32];
  __shared__ int carry;
  const int tid = threadIdx.x, cta = blockIdx.x, ch = P.chunk;
  const int r0 = GROUPS ? g.node_off[g.inst[cta]] : 0, r1 = GROUPS ? g.node_off[g.inst[cta] + 1] : A.n_rows;
  const int words = (r1 - r0 + 31) / 32;
  uint32_t* bits = sm;
  int* rank = reinterpret_cast<int*>(sm + words);
  int row0, m, off = 0;  // local rows [off, m)
  if constexpr (GROUPS) {
    const GroupRows q = group_rows(g, cta);
    row0 = 32 * q.s0, off = q.lo - row0, m = q.hi - row0;
  } else if (ch == 32) {
    const int sa = (int)((int64_t)cta * A.n_slices / P.n_cta), sb = (int)((int64_t)(cta + 1) * A.n_slices / P.n_cta);
    row0 = 32 * sa;
    m = min(32 * (sb - sa), A.n_rows - row0);
    if (tid == 0) slice0[cta] = sa;
    if (tid == 0 && cta == P.n_cta - 1) slice0[P.n_cta] = sb;
  } else {
    row0 = cta * ch;
    m = min(ch, A.n_rows - row0);
  }
  for (int i = tid; i < words; i += blockDim.x) bits[i] = 0u;
  if (tid == 0) carry = 0;
  __syncthreads();
  for (int i = off + tid; i < m; i += blockDim.x) {
    const int row = row0 + i;
    for (int k = A.row_ptr[row]; k < A.row_ptr[row + 1]; ++k) {
      const int c = A.col[k], d = c - r0;
      if (c < row0 + off || c >= row0 + m) atomicOr(&bits[d >> 5], 1u << (d & 31));
    }
  }
  __syncthreads();
  for (int w0 = 0; w0 < words; w0 += blockDim.x) {  // exclusive running count of the words' bits
    const int i = w0 + tid, lane = tid & 31, warp = tid >> 5;
    const int own = i < words ? __popc(bits[i]) : 0;
    int inc = own;
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += t;
    }
    if (lane == 31) wtot[warp] = inc;
    __syncthreads();
    int base = carry;
    for (int w = 0; w < warp; ++w) base += wtot[w];
    if (i < words) rank[i] = base + inc - own;
    __syncthreads();
    if (tid == (int)blockDim.x - 1) carry = base + inc;
    __syncthreads();
  }
  if (tid == 0) cnt[cta] = carry;
  if (carry > P.halo_cap) return;  // the host sees the count and does not use the plan
  for (int i = tid; i < words; i += blockDim.x) {
    int k = rank[i];
    for (uint32_t b = bits[i]; b; b &= b - 1) halo[(int64_t)cta * P.halo_cap + k++] = r0 + 32 * i + __ffs(b) - 1;
  }
  const int mp = !GROUPS && ch == 32 ? (m + 31) / 32 * 32 : m;  // lanes without a row get the column 0
  for (int i = off + tid; i < mp; i += blockDim.x) {
    const int row = row0 + i, s = row >> 5;
    for (int g = A.slice_off[s]; g < A.slice_off[s + 1]; ++g) {
      const int64_t b = (int64_t)g * 32 + (row & 31);
      int l = 0;
      if (row < A.n_rows) {
        const int c = A.col_sell[b], d = c - r0;
        l = c >= row0 + off && c < row0 + m ? c - row0 : m + rank[d >> 5] + __popc(bits[d >> 5] & ((1u << (d & 31)) - 1u));
      }
      col16[b] = (uint16_t)l;
    }
  }
}

// GROUPS: start of a solve on b.  One CTA per instance: x = 0, r = b, z = M^-1 r, p = z, no published rows, b.b.
template <typename T>
__global__ void __launch_bounds__(512) halo_groups_init_kernel(HaloGroups g, const double* __restrict__ b,
                                                               const T* __restrict__ minv, T* x, T* r, T* z, T* published) {
  __shared__ double sh[512];
  if (g.first[blockIdx.x] != (int)blockIdx.x) return;
  const int inst = g.inst[blockIdx.x];
  double bb[1] = {0.0};
  for (int64_t i = g.node_off[inst] + threadIdx.x; i < g.node_off[inst + 1]; i += blockDim.x) {
    const T v[3] = {T(b[3 * i]), T(b[3 * i + 1]), T(b[3 * i + 2])};
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const T* q = minv + 9 * i + 3 * c;
      x[4 * i + c] = T(0);
      r[4 * i + c] = v[c];
      z[4 * i + c] = static_cast<T*>(g.p)[4 * i + c] = q[0] * v[0] + q[1] * v[1] + q[2] * v[2];
      bb[0] += double(v[c]) * double(v[c]);
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) published[4 * i + c] = T(0);
  }
  cta_reduce_smem<1>(bb, sh);
  if (threadIdx.x == 0) {
    g.st[4 * inst + 2] = bb[0];
    g.its[inst] = 0;
  }
}

// GROUPS: from the state that the kernels of batched.cu leave between launches (p_old in p0 or p1 by the parity of the
// iteration, beta in st) to this form's: p = z + beta p_old, no published rows.  One CTA per instance.
template <typename T>
__global__ void __launch_bounds__(512) halo_groups_take_over_kernel(HaloGroups g, const T* __restrict__ z, T* published) {
  if (g.first[blockIdx.x] != (int)blockIdx.x) return;
  const int inst = g.inst[blockIdx.x];
  T* p = static_cast<T*>(g.p);
  const T beta = T(g.st[4 * inst + 3]);
  const bool in_p = g.its[inst] & 1;
  for (int64_t i = g.node_off[inst] + threadIdx.x; i < g.node_off[inst + 1]; i += blockDim.x)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const T old = in_p ? p[4 * i + c] : published[4 * i + c];
      if (c < 3) p[4 * i + c] = z[4 * i + c] + beta * old;
      published[4 * i + c] = T(0);
    }
}

// Shared-memory layout and eligibility of a variant on a system.  Rows per thread and the shared memory of p, the
// partial products and the halo list bound the size: about 250 k rows of a structured mesh in FP32, 150 k in FP64.
struct Layout {
  int np = 0, qstride = 0, resident = 0, ring = 0, units = 0, passes = 0, bytes = 0;
  bool ok = false;
};
template <typename T>
Layout layout_of(const HaloPlan& P, int warps) {
  Layout L;
  if (!P.n_cta || P.n_cta > kMaxCtas) return L;
  const int rows = P.chunk == 32 ? 32 * P.max_ns : P.chunk;
  // a warp reads three components of ten consecutive rows of the partial products: 11 words apart in the banks
  const int np = (rows + P.max_halo + 3) / 4 * 4, qstride = (warps + P.max_ns) * 32 + 11;
  const int64_t fixed = 3LL * np * sizeof(T) + 3LL * qstride * sizeof(T) + 4LL * (P.max_halo + P.max_ns + 1);
  const int units = (int)((kSmemBudget - fixed) / ((int64_t)warps * unit_bytes<T>()));
  const int per = (P.max_units + warps - 1) / warps;
  if (fixed > kSmemBudget || rows + P.max_halo > 65535) return L;
  auto passes = [&](bool streamed) { return (rows + warps * rows_per_warp(streamed) - 1) / (warps * rows_per_warp(streamed)); };
  if (units >= per && passes(false) <= 2) {
    L.resident = per;
    L.passes = passes(false);
  } else {
    // two stages in flight first, as the bandwidth of the stream comes from them: four block columns each in FP32 (two:
    // 13.2 instead of 10.0 us per iteration at 60 625 rows, although more columns stay resident), two in FP64 (one: 26.1
    // instead of 24.8 us at 35 721 rows), less where the vectors leave no room
    L.passes = passes(true);
    if (P.chunk < 32 || L.passes > 4) return L;
    L.units = sizeof(T) == 8 ? (units >= 4 ? 2 : 1) : units >= 8 && L.passes <= 2 ? 4 : 2;
    L.ring = 2;
    if (L.ring * L.units > units) return L;
    L.resident = std::min(units - L.ring * L.units, per);
  }
  L.np = np, L.qstride = qstride;
  L.bytes = (int)(fixed + (int64_t)warps * (L.resident + L.ring * L.units) * unit_bytes<T>());
  L.ok = true;
  return L;
}

template <typename T, int WARPS, int MAXP, int CB, bool GROUPS = false>
cudaError_t launch_variant(const Bsr& A, PcgWork& w, const Layout& L, cudaStream_t s, const HaloPlan& P,
                           const HaloGroups& g = HaloGroups{}) {
  auto kern = pcg_halo_kernel<T, WARPS, MAXP, CB, GROUPS>;
  static std::mutex mu;
  static bool set[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  {
    std::lock_guard<std::mutex> lk(mu);
    if (dev >= 64 || !set[dev]) {
      cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBudget);
      if (e != cudaSuccess) return e;
      if (dev < 64) set[dev] = true;
    }
  }
  HaloArgs<T> H;
  H.P = P;
  H.g = g;
  H.A = A;
  H.val = (const T*)A.val;
  H.minv = (const T*)w.minv;
  H.x = (T*)w.x;
  H.r = (const T*)w.r;
  H.z = (const T*)w.z;
  H.p = (T*)w.p1;
  H.part = w.part_c;
  H.scal = w.scal;
  H.keep_g = w.keep_g;
  H.wc = WaitCtl{w.barrier_polls > 0 ? w.barrier_polls : kBarrierSpinLimit, w.withhold_first_arrival};
  H.np = L.np, H.qstride = L.qstride, H.resident = L.resident, H.ring = L.ring;
  void* args[] = {&H};
  return cudaLaunchCooperativeKernel((const void*)kern, dim3(H.P.n_cta), dim3(WARPS * 32), args, L.bytes, s);
}

// warps per CTA of a variant; the tuner times both where both exist.  FP32 16 (8: 0.1 us faster per iteration below 5 000
// rows, 0.3 us slower at 18 785 and not built for streams), FP64 8 (16: slower below 20 000 rows, 3 % faster at 35 721,
// 9 % at 60 625)
constexpr int warps_of(bool fp32, int variant) { return fp32 == (variant == 0) ? 16 : 8; }

cudaError_t launch(const Bsr& A, PcgWork& w, int variant, cudaStream_t s) {
  if (w.fp32) {
    const Layout L = layout_of<float>(*w.halo, warps_of(true, variant));
    if (!L.ok) return cudaErrorInvalidConfiguration;
    if (variant == 1)
      return L.passes <= 1 ? launch_variant<float, 8, 1, 0>(A, w, L, s, *w.halo) : launch_variant<float, 8, 2, 0>(A, w, L, s, *w.halo);
    if (!L.ring) return L.passes <= 1 ? launch_variant<float, 16, 1, 0>(A, w, L, s, *w.halo) : launch_variant<float, 16, 2, 0>(A, w, L, s, *w.halo);
    if (L.units == 2) return launch_variant<float, 16, 4, 2>(A, w, L, s, *w.halo);
    return L.passes <= 1 ? launch_variant<float, 16, 1, 4>(A, w, L, s, *w.halo) : launch_variant<float, 16, 2, 4>(A, w, L, s, *w.halo);
  }
  const Layout L = layout_of<double>(*w.halo, warps_of(false, variant));
  if (!L.ok) return cudaErrorInvalidConfiguration;
  if (variant == 1) {
    if (!L.ring) return launch_variant<double, 16, 2, 0>(A, w, L, s, *w.halo);
    if (L.units == 1) return launch_variant<double, 16, 2, 1>(A, w, L, s, *w.halo);
    return L.passes <= 1 ? launch_variant<double, 16, 1, 2>(A, w, L, s, *w.halo) : launch_variant<double, 16, 2, 2>(A, w, L, s, *w.halo);
  }
  if (!L.ring) return L.passes <= 1 ? launch_variant<double, 8, 1, 0>(A, w, L, s, *w.halo) : launch_variant<double, 8, 2, 0>(A, w, L, s, *w.halo);
  if (L.units == 1) return launch_variant<double, 8, 4, 1>(A, w, L, s, *w.halo);
  if (L.passes <= 1) return launch_variant<double, 8, 1, 2>(A, w, L, s, *w.halo);
  return L.passes <= 2 ? launch_variant<double, 8, 2, 2>(A, w, L, s, *w.halo) : launch_variant<double, 8, 4, 2>(A, w, L, s, *w.halo);
}
// The GROUPS form is built with the warps of variant 0.
template <typename T, int WARPS>
cudaError_t launch_groups(const Bsr& A, PcgWork& w, const Layout& L, cudaStream_t s, const HaloPlan& P,
                          const HaloGroups& g) {
  constexpr int U = sizeof(T) == 8 ? 2 : 4;
  if (!L.ring)
    return L.passes <= 1 ? launch_variant<T, WARPS, 1, 0, true>(A, w, L, s, P, g)
                         : launch_variant<T, WARPS, 2, 0, true>(A, w, L, s, P, g);
  if (L.units < U) return launch_variant<T, WARPS, 4, U / 2, true>(A, w, L, s, P, g);
  if (L.passes <= 1) return launch_variant<T, WARPS, 1, U, true>(A, w, L, s, P, g);
  if (L.passes <= 2) return launch_variant<T, WARPS, 2, U, true>(A, w, L, s, P, g);
  return launch_variant<T, WARPS, 4, U / (sizeof(T) == 4 ? 2 : 1), true>(A, w, L, s, P, g);
}
// variant 1 exists where it can be faster: FP32 without a stream, FP64 up to two passes
Layout usable(const PcgWork& w, int variant) {
  Layout L = w.fp32 ? layout_of<float>(*w.halo, warps_of(true, variant)) : layout_of<double>(*w.halo, warps_of(false, variant));
  if (variant == 1 && (w.fp32 ? L.ring > 0 : L.passes > 2)) L.ok = false;
  return L;
}

}  // namespace

// Chunk: with at least 32 rows per SM whole slices; below that the smallest power of two that spreads the rows over
// the SMs, so that a row's blocks are shared by 32 / chunk lanes of a warp and the FP64 products of a small system do
// not queue on a few SMs.
int halo_chunk(int n_rows, int sms) {
  for (int c = 4; c < 32; c *= 2)
    if (n_rows <= (int64_t)c * sms) return c;
  return 32;
}
int halo_ctas(int n_rows, int sms) {
  sms = sms < kMaxCtas ? sms : kMaxCtas;
  const int c = halo_chunk(n_rows, sms), n = (n_rows + c - 1) / c;
  return n < sms ? n : sms;
}
// the bitmap and its ranks: eight bytes per 32 rows of shared memory
int halo_max_rows() { return kSmemBudget / 8 * 32; }

cudaError_t launch_halo_plan(const Bsr& A, const HaloPlan& P, int32_t* slice0, int32_t* cnt, int32_t* halo,
                             uint16_t* col16, cudaStream_t s) {
  const int bytes = (A.n_rows + 31) / 32 * 8;
  cudaError_t e = cudaFuncSetAttribute(halo_plan_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBudget);
  if (e != cudaSuccess) return e;
  halo_plan_kernel<false><<<P.n_cta, 1024, bytes, s>>>(A, P, HaloGroups{}, slice0, cnt, halo, col16);
  return cudaGetLastError();
}

bool pcg_halo_eligible(const PcgWork& w, int variant) {
  if (!w.halo || variant < 0 || variant >= kHaloVariants) return false;
  int dev = 0, coop = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
  return coop && usable(w, variant).ok;
}
bool pcg_halo_streams(const PcgWork& w, int variant) { return usable(w, variant).ring > 0; }

static_assert(kHaloWords == 2 * kSums * kCopies * kMaxCtas * 2, "the words' share of the work array");

bool batched_halo_fits(const HaloPlan& P, bool fp32) {
  return (fp32 ? layout_of<float>(P, warps_of(true, 0)) : layout_of<double>(P, warps_of(false, 0))).ok;
}
cudaError_t launch_batched_halo(const Bsr& A, const PcgWork& work, const HaloPlan& P, int32_t* cnt, int32_t* halo,
                                uint16_t* col16, int max_rows, const double* b, double* x_out, const int32_t* node_off,
                                const int32_t* cta_inst, const int32_t* cta_first, const int32_t* cta_size,
                                const double* rtol, int max_iter, int chunk, HaloStart start, double* st, int32_t* its,
                                int32_t* flag, double* relres, cudaStream_t s) {
  const Layout L = work.fp32 ? layout_of<float>(P, warps_of(true, 0)) : layout_of<double>(P, warps_of(false, 0));
  if (!L.ok) return cudaErrorInvalidConfiguration;
  PcgWork w = work;
  // the streamed blocks stay in L2 as far as 90 of its 129 MB go
  const int64_t groups = A.n_padded / 32, kept = (90ll << 20) / (w.fp32 ? unit_bytes<float>() : unit_bytes<double>());
  w.keep_g = groups < kept ? groups : kept;
  const HaloGroups g{cta_inst, cta_first, cta_size, node_off, rtol, max_iter, chunk, w.p0, st, its, flag, relres, x_out};
  cudaError_t e = cudaMemsetAsync(w.part_c, 0, sizeof(double) * kHaloWords, s);
  if (e != cudaSuccess) return e;
  halo_plan_kernel<true><<<P.n_cta, 1024, (max_rows + 31) / 32 * 8, s>>>(A, P, g, nullptr, cnt, halo, col16);
  if (start == HaloStart::kTakeOver && w.fp32)
    halo_groups_take_over_kernel<float><<<P.n_cta, 512, 0, s>>>(g, (const float*)w.z, (float*)w.p1);
  else if (start == HaloStart::kTakeOver)
    halo_groups_take_over_kernel<double><<<P.n_cta, 512, 0, s>>>(g, (const double*)w.z, (double*)w.p1);
  else if (start == HaloStart::kFirst && w.fp32)
    halo_groups_init_kernel<float><<<P.n_cta, 512, 0, s>>>(g, b, (const float*)w.minv, (float*)w.x, (float*)w.r,
                                                          (float*)w.z, (float*)w.p1);
  else if (start == HaloStart::kFirst)
    halo_groups_init_kernel<double><<<P.n_cta, 512, 0, s>>>(g, b, (const double*)w.minv, (double*)w.x, (double*)w.r,
                                                           (double*)w.z, (double*)w.p1);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  return w.fp32 ? launch_groups<float, 16>(A, w, L, s, P, g) : launch_groups<double, 8>(A, w, L, s, P, g);
}

cudaError_t launch_pcg_halo(const Bsr& A, PcgWork& w, int variant, cudaStream_t s) {
  return usable(w, variant).ok ? launch(A, w, variant, s) : cudaErrorInvalidConfiguration;
}

}  // namespace ikr
