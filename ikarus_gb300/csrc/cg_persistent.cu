// Persistent block-Jacobi PCG: a whole CG solve in one cooperative launch (sm_103a).
//
// Same iteration as the two-kernel CG of solver.cu / spmv_staged.cu (p_new = z + beta p_old formed on the fly
// for every gathered neighbour, q = K p_new, alpha = rz / p.q, x += alpha p, r -= alpha q, z = M^{-1} r,
// beta = rz_new / rz), but every CTA stays resident for all iterations and the two global reductions of an
// iteration are grid barriers:
//   * each warp owns up to MAXS slices (32 block rows each) and keeps x, r, z, p and q of its rows in registers,
//     so the update phase touches global memory only to publish z (and p_new in the product phase), which the
//     neighbours' gathers need;
//   * the matrix is streamed with the same per-warp bulk-copy pipeline as the staged SpMV; the stream of a
//     warp's chunks is cyclic over iterations, so the copies of the next iteration's first chunks are in flight
//     while the CTA waits at the barriers;
//   * a grid barrier publishes one partial per CTA (double-buffered by iteration parity), arrives on a counter
//     and waits until every CTA has arrived; every CTA then sums all partials in CTA order, so alpha, beta and
//     the convergence decision are bit-identical in all CTAs and from run to run.
// The launch is cooperative (all CTAs co-resident).  Every wait is bounded: a grid barrier or stage wait that
// gives up sets scal[kDone] = 6, the kernel drains its copies in flight (bounded) and returns.
#include <mutex>

#include "cg_grid.cuh"

namespace ikr {

namespace {

using namespace cg;

// The block-Jacobi inverses of a CTA's rows in shared memory for the whole solve (they do not change within it), so
// that the update phase after the first grid barrier of an iteration reads them without an L2 round trip -- where
// they fit beside the staging buffers.
template <typename T, int CB, int NST, int WARPS, int MAXS>
struct MinvShared {
  static constexpr int kBytes = WARPS * MAXS * 32 * 9 * (int)sizeof(T);
  static constexpr bool kOn = PersistentCfg<T, CB, NST, WARPS>::kSmemBytes + kBytes <= 200 * 1024;
  static constexpr int kDynBytes = PersistentCfg<T, CB, NST, WARPS>::kSmemBytes + (kOn ? kBytes : 0);
};

// the right-hand sides one launch solves together: per RHS its solution, residual, preconditioned residual, the
// two search-direction buffers (alternating by iteration parity) and its scalar block
template <typename T, int NR>
struct RhsSet {
  T* x[NR];
  const T* r[NR];
  T* z[NR];
  T* p0[NR];
  T* p1[NR];
  double* scal[NR];
};

// NR right-hand sides with the same matrix: every chunk of the matrix stream is staged once and multiplied
// against each unfinished RHS, so two solves cost one matrix stream per iteration instead of two.  Each RHS
// keeps its own CG scalars, iteration count and stop decision; the grid reductions carry the NR values together.
template <typename T, int CB, int NST, int WARPS, int MAXS, int MINB, int NR>
__global__ void __launch_bounds__(WARPS * 32, MINB)
    pcg_persistent_kernel(Bsr A, const T* __restrict__ val, const T* __restrict__ minv, RhsSet<T, NR> V,
                          double* part_a, double* part_b, int64_t keep_g, WaitCtl wc) {
  using C = PersistentCfg<T, CB, NST, WARPS>;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ __align__(8) uint64_t bars[WARPS][NST];
  __shared__ double sv[2 * NR];
  __shared__ T s_alpha[NR], s_tb[NR];
  __shared__ int s_dn[NR];
  __shared__ double sfull[2 * NR * WARPS * 32];
  __shared__ bool ok_sh;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int G = gridDim.x;
  const int nw = G * WARPS;
  const int gw = blockIdx.x * WARPS + warp;
  const int n_slices = A.n_slices;
  unsigned int* bar_count = &tickets(V.scal[0])[3];
  unsigned char* wbase = smem + (size_t)warp * NST * C::kStageBytes;

  // owned slices and their block ranges
  int ns = 0;
  int s_first[MAXS], s_end[MAXS];
#pragma unroll
  for (int j = 0; j < MAXS; ++j) {
    const int sj = gw + j * nw;
    s_first[j] = 0, s_end[j] = 0;
    if (sj < n_slices) {
      s_first[j] = A.slice_off[sj];
      s_end[j] = A.slice_off[sj + 1];
      ns = j + 1;
    }
  }
  // CG state of the owned rows, per RHS.  With one RHS x, r, z, p and q of the owned rows live in registers;
  // with several (kLean) only r and q do, and x, z, p of the owned rows are re-read from the global vectors
  // (which the gathers need anyway; own-row reads hit L2) to keep the register count without spills.
  constexpr bool kLean = NR > 1;
  constexpr int XS = kLean ? 1 : MAXS;
  T xr[NR][XS][3], rr_[NR][MAXS][3], zr[NR][XS][3], pr[NR][XS][3], qr[NR][MAXS][3];
  // The CG scalars are FP64 and thread 0 alone updates them (rz, r.r, beta, the stop decision); the other threads
  // get the state code, alpha and beta in the CG's type through shared memory (GB300's FP64 pipe is narrow: 512
  // threads repeating the divisions, comparisons and conversions cost microseconds per iteration)
  double rz[NR], tol2[NR], rrs[NR], beta[NR];
  int maxit[NR], it[NR], dn[NR];  // dn: 0 running, 1 converged, 2 iteration cap, 3 breakdown (as scal[kDone])
  T tbv[NR];
  bool all_done = true;
#pragma unroll
  for (int q = 0; q < NR; ++q) {
#pragma unroll
    for (int j = 0; j < MAXS; ++j) {
      const int row = 32 * (gw + j * nw) + lane;
      const bool own = j < ns && row < A.n_rows;
      V3<T> r0 = {T(0), T(0), T(0)}, z0 = {T(0), T(0), T(0)};
      if (own) r0 = load3rw(V.r[q], row), z0 = load3rw(V.z[q], row);
#pragma unroll
      for (int c = 0; c < 3; ++c) qr[q][j][c] = T(0);
      rr_[q][j][0] = r0.x, rr_[q][j][1] = r0.y, rr_[q][j][2] = r0.z;
      if constexpr (!kLean) {
#pragma unroll
        for (int c = 0; c < 3; ++c) xr[q][j][c] = pr[q][j][c] = T(0);
        zr[q][j][0] = z0.x, zr[q][j][1] = z0.y, zr[q][j][2] = z0.z;
      }
    }
    const double* sc = V.scal[q];
    rz[q] = sc[kRz];
    tol2[q] = sc[kTol2];
    maxit[q] = (int)sc[kMaxIt];
    rrs[q] = sc[kRR];
    dn[q] = (int)sc[kDone];
    it[q] = (int)sc[kIters];
    beta[q] = 0.0;
    tbv[q] = T(0);
    all_done = all_done && dn[q] != 0;
  }

  using MS = MinvShared<T, CB, NST, WARPS, MAXS>;
  T* msh = reinterpret_cast<T*>(smem + C::kSmemBytes);  // used when MS::kOn
  if constexpr (MS::kOn) {
#pragma unroll
    for (int j = 0; j < MAXS; ++j) {
      const int row = 32 * (gw + j * nw) + lane;
      T* d = msh + ((size_t)(warp * MAXS + j) * 32 + lane) * 9;
#pragma unroll
      for (int k = 0; k < 9; ++k) d[k] = (j < ns && row < A.n_rows) ? __ldg(minv + 9 * (int64_t)row + k) : T(0);
    }
  }
  auto minv_of = [&](int j, int row) -> const T* {
    if constexpr (MS::kOn) return msh + ((size_t)(warp * MAXS + j) * 32 + lane) * 9;
    return minv + 9 * (int64_t)row;
  };

  if (lane == 0) {
    for (int st = 0; st < NST; ++st) mbar_init(smem_addr(&bars[warp][st]), 1);
    mbar_init_fence();
  }
  __syncwarp();

  auto issue = [&](int st, const CyclicPos& P) {
    if (lane == 0) {
      const int nb = min(CB, P.gend - P.g);
      const uint32_t vb = nb * 288 * (uint32_t)sizeof(T), cb = nb * 128;
      const uint32_t b = smem_addr(&bars[warp][st]);
      unsigned char* stage = wbase + (size_t)st * C::kStageBytes;
      const uint64_t pol = l2_policy(P.g < keep_g);
      mbar_expect_tx(b, vb + cb);
      bulk_g2s(smem_addr(stage), val + (int64_t)P.g * 288, vb, b, pol);
      bulk_g2s(smem_addr(stage + C::kValBytes), A.col_sell + (int64_t)P.g * 32, cb, b, pol);
    }
  };
  auto advance = [&](CyclicPos& P) {
    P.g += CB;
    if (P.g >= P.gend) {
      P.j = (P.j + 1 == ns) ? 0 : P.j + 1;
      // s_first / s_end are indexed with a runtime j here: pick through an unrolled select
#pragma unroll
      for (int j = 0; j < MAXS; ++j)
        if (j == P.j) P.g = s_first[j], P.gend = s_end[j];
    }
  };

  CyclicPos P{0, s_first[0], s_end[0]};
  int inflight = 0;
  if (ns > 0 && !all_done) {
    for (int st = 0; st < NST; ++st) {
      issue(st, P);
      ++inflight;
      advance(P);
    }
  }
  uint32_t phase = 0;
  int st = 0;
  bool failed = false;
  unsigned int barrier_no = 0;
  int loop = 0;  // parity of the partial buffers

  while (!all_done) {
    T tb[NR];
    const T* pold[NR];
    T* pnew[NR];
    bool act[NR];
    double pq[NR];
    T pql[NR];  // a lane's p.q in the CG's type, converted once
#pragma unroll
    for (int q = 0; q < NR; ++q) {
      act[q] = dn[q] == 0;
      tb[q] = tbv[q];
      pold[q] = (it[q] & 1) ? V.p0[q] : V.p1[q];
      pnew[q] = (it[q] & 1) ? V.p1[q] : V.p0[q];
      pq[q] = 0.0;
      pql[q] = T(0);
    }
    // ---- product phase: q = K p_new over the owned slices, every active RHS from the same staged chunk
#pragma unroll
    for (int j = 0; j < MAXS; ++j) {
      if (j < ns && !failed) {
        T acc[NR][3];
#pragma unroll
        for (int q = 0; q < NR; ++q) acc[q][0] = acc[q][1] = acc[q][2] = T(0);
        for (int g = s_first[j]; g < s_end[j]; g += CB) {
          const bool okw = __all_sync(0xffffffffu, mbar_wait_bounded(smem_addr(&bars[warp][st]), (phase >> st) & 1u));
          if (!okw) {
            failed = true;
            break;
          }
          phase ^= 1u << st;
          --inflight;
          const T* sval = reinterpret_cast<const T*>(wbase + (size_t)st * C::kStageBytes);
          const int32_t* scol = reinterpret_cast<const int32_t*>(wbase + (size_t)st * C::kStageBytes + C::kValBytes);
          const int nb = min(CB, s_end[j] - g);
          int cols[CB];
#pragma unroll
          for (int k = 0; k < CB; ++k) cols[k] = k < nb ? scol[32 * k + lane] : 0;
#pragma unroll
          for (int q = 0; q < NR; ++q) {
            if (!act[q]) continue;
            V3<T> zc[CB], pc[CB];
#pragma unroll
            for (int k = 0; k < CB; ++k) {
              zc[k] = load3rw(V.z[q], cols[k]);
              pc[k] = load3rw(pold[q], cols[k]);
            }
#pragma unroll
            for (int k = 0; k < CB; ++k) {
              if (k < nb) {
                const T x0 = zc[k].x + tb[q] * pc[k].x, x1 = zc[k].y + tb[q] * pc[k].y,
                        x2 = zc[k].z + tb[q] * pc[k].z;
                const T* v = sval + 288 * k + lane;
                acc[q][0] += v[0] * x0 + v[32] * x1 + v[64] * x2;
                acc[q][1] += v[96] * x0 + v[128] * x1 + v[160] * x2;
                acc[q][2] += v[192] * x0 + v[224] * x1 + v[256] * x2;
              }
            }
          }
          __syncwarp();  // the stage is consumed before it is refilled
          issue(st, P);
          ++inflight;
          advance(P);
          st = (st + 1 == NST) ? 0 : st + 1;
        }
        const int row = 32 * (gw + j * nw) + lane;
#pragma unroll
        for (int q = 0; q < NR; ++q) {
          if (!act[q]) continue;
          V3<T> zo, po;
          if constexpr (kLean) {
            zo = {T(0), T(0), T(0)}, po = {T(0), T(0), T(0)};
            if (row < A.n_rows) zo = load3rw(V.z[q], row), po = load3rw(pold[q], row);
          } else {
            zo = {zr[q][j][0], zr[q][j][1], zr[q][j][2]};
            po = {pr[q][j][0], pr[q][j][1], pr[q][j][2]};
          }
          const T n0 = zo.x + tb[q] * po.x, n1 = zo.y + tb[q] * po.y, n2 = zo.z + tb[q] * po.z;
          if constexpr (!kLean) pr[q][j][0] = n0, pr[q][j][1] = n1, pr[q][j][2] = n2;
          qr[q][j][0] = acc[q][0], qr[q][j][1] = acc[q][1], qr[q][j][2] = acc[q][2];
          if (row < A.n_rows) {
            store3(pnew[q], row, n0, n1, n2);
            pql[q] += n0 * acc[q][0] + n1 * acc[q][1] + n2 * acc[q][2];
          }
        }
      }
    }
    // ---- grid reduction of p.q (all RHS together)
    const int par = loop & 1;
    failed = __syncthreads_or(failed);
    if (failed) break;
#pragma unroll
    for (int q = 0; q < NR; ++q) pq[q] = double(pql[q]);
    cta_reduce_smem<NR>(pq, sfull);
    ++barrier_no;
    if (!grid_allreduce<NR>(pq, part_a + par * NR * G, bar_count, barrier_no * (unsigned)G, sv, &ok_sh, wc)) {
      failed = true;
      break;
    }
    if (threadIdx.x == 0) {
#pragma unroll
      for (int q = 0; q < NR; ++q) {
        T a = T(0);
        if (dn[q] == 0) {
          if (!(fabs(pq[q]) > 0.0) || !isfinite(pq[q])) dn[q] = 3;  // breakdown (negative curvature alone does not stop CG)
          else a = T(rz[q] / pq[q]);
        }
        s_alpha[q] = a;
        s_dn[q] = dn[q];
      }
    }
    __syncthreads();
    T alpha[NR];
#pragma unroll
    for (int q = 0; q < NR; ++q) {
      alpha[q] = s_alpha[q];
      dn[q] = s_dn[q];
      act[q] = dn[q] == 0;
    }
    // ---- update phase on the owned rows
    double red2[2 * NR];
#pragma unroll
    for (int q = 0; q < NR; ++q) {
      // a lane's rows are summed in the CG's type and converted once (FP64 additions and conversions per row would
      // load GB300's narrow FP64 pipe); the CTA and grid sums above them are FP64
      T lrz = T(0), lrr = T(0);
      if (act[q]) {
        const T a = alpha[q];
#pragma unroll
        for (int j = 0; j < MAXS; ++j) {
          const int row = 32 * (gw + j * nw) + lane;
          if (j < ns && row < A.n_rows) {
            T r1[3];
            if constexpr (kLean) {
              const V3<T> pv = load3rw(pnew[q], row);
              const V3<T> xv = load3rw(V.x[q], row);
              store3(V.x[q], row, xv.x + a * pv.x, xv.y + a * pv.y, xv.z + a * pv.z);
            } else {
#pragma unroll
              for (int c = 0; c < 3; ++c) xr[q][j][c] += a * pr[q][j][c];
            }
#pragma unroll
            for (int c = 0; c < 3; ++c) {
              r1[c] = rr_[q][j][c] - a * qr[q][j][c];
              rr_[q][j][c] = r1[c];
            }
            const T* m = minv_of(j, row);
            T zv[3];
#pragma unroll
            for (int b = 0; b < 3; ++b) {
              zv[b] = m[3 * b] * r1[0] + m[3 * b + 1] * r1[1] + m[3 * b + 2] * r1[2];
              if constexpr (!kLean) zr[q][j][b] = zv[b];
            }
            store3(V.z[q], row, zv[0], zv[1], zv[2]);
            T trz = T(0), trr = T(0);
#pragma unroll
            for (int b = 0; b < 3; ++b) {
              trz += r1[b] * zv[b];
              trr += r1[b] * r1[b];
            }
            lrz += trz;
            lrr += trr;
          }
        }
      }
      red2[2 * q] = double(lrz);
      red2[2 * q + 1] = double(lrr);
    }
    cta_reduce_smem<2 * NR>(red2, sfull);
    ++barrier_no;
    if (!grid_allreduce<2 * NR>(red2, part_b + par * 2 * NR * G, bar_count, barrier_no * (unsigned)G, sv, &ok_sh,
                                wc)) {
      failed = true;
      break;
    }
    if (threadIdx.x == 0) {
#pragma unroll
      for (int q = 0; q < NR; ++q) {
        if (act[q]) {
          const double rzs = red2[2 * q];
          rrs[q] = red2[2 * q + 1];
          beta[q] = rzs / rz[q];
          rz[q] = rzs;
          if (rrs[q] <= tol2[q]) dn[q] = 1;
          else if (it[q] + 1 >= maxit[q]) dn[q] = 2;
        }
        s_tb[q] = T(beta[q]);
        s_dn[q] = dn[q];
      }
    }
    __syncthreads();
    all_done = true;
#pragma unroll
    for (int q = 0; q < NR; ++q) {
      if (act[q]) ++it[q];
      dn[q] = s_dn[q];
      tbv[q] = s_tb[q];
      all_done = all_done && dn[q] != 0;
    }
    ++loop;
  }
  // drain the copies still in flight (the cyclic stream runs ahead of the last iteration)
  for (int k = 0; k < inflight; ++k) {
    mbar_wait_bounded(smem_addr(&bars[warp][st]), (phase >> st) & 1u);
    phase ^= 1u << st;
    st = (st + 1 == NST) ? 0 : st + 1;
  }
  // solutions of the owned rows; the final scalars from CTA 0 (identical in every CTA)
#pragma unroll
  for (int q = 0; q < NR; ++q) {
    if constexpr (!kLean) {
#pragma unroll
      for (int j = 0; j < MAXS; ++j) {
        const int row = 32 * (gw + j * nw) + lane;
        if (j < ns && row < A.n_rows) store3(V.x[q], row, xr[q][j][0], xr[q][j][1], xr[q][j][2]);
      }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      double* sc = V.scal[q];
      sc[kIters] = (double)it[q];
      sc[kRR] = rrs[q];
      sc[kRz] = rz[q];
      sc[kBeta] = beta[q];
      sc[kDone] = failed ? kDoneDeviceTimeout : (double)dn[q];
    }
    if (failed && threadIdx.x == 0) V.scal[q][kDone] = kDoneDeviceTimeout;
  }
}

template <typename T, int CB, int NST, int WARPS, int MAXS, int MINB, int NR>
cudaError_t launch_persistent(const Bsr& A, PcgWork* const* ws, double* part_a, double* part_b, cudaStream_t s,
                              bool query_only, bool* eligible) {
  using C = PersistentCfg<T, CB, NST, WARPS>;
  constexpr int kDyn = MinvShared<T, CB, NST, WARPS, MAXS>::kDynBytes;
  auto kern = pcg_persistent_kernel<T, CB, NST, WARPS, MAXS, MINB, NR>;
  static std::mutex mu;
  static int blocks_per_sm[64] = {0};
  PcgWork& w = *ws[0];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 64) dev = 63;
  int bps;
  {
    std::lock_guard<std::mutex> lk(mu);
    if (!blocks_per_sm[dev]) {
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kDyn);
      int b = 0;
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kern, C::kThreads, kDyn);
      blocks_per_sm[dev] = b > 0 ? b : -1;
    }
    bps = blocks_per_sm[dev];
  }
  int coop = 0;
  cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
  // one wave of co-resident CTAs; the partial buffers hold 2 NR w.grid (part_a) and 4 NR w.grid (part_b) values,
  // 2 NR and 4 NR per CTA here
  int grid = bps > 0 ? w.sms * bps : 0;
  if (grid > w.grid) grid = w.grid;
  const int nw = grid * WARPS;
  *eligible = coop && grid > 0 && (int64_t)nw * MAXS >= A.n_slices;
  if (query_only || !*eligible) return cudaSuccess;
  const T* val = (const T*)A.val;
  const T* minv = (const T*)w.minv;
  RhsSet<T, NR> V;
  for (int q = 0; q < NR; ++q) {
    V.x[q] = (T*)ws[q]->x;
    V.r[q] = (const T*)ws[q]->r;
    V.z[q] = (T*)ws[q]->z;
    V.p0[q] = (T*)ws[q]->p0;
    V.p1[q] = (T*)ws[q]->p1;
    V.scal[q] = ws[q]->scal;
  }
  Bsr Acopy = A;
  int64_t keep = w.keep_g;
  WaitCtl wc{w.barrier_polls > 0 ? w.barrier_polls : kBarrierSpinLimit, w.withhold_first_arrival};
  void* args[] = {&Acopy, &val, &minv, &V, &part_a, &part_b, &keep, &wc};
  return cudaLaunchCooperativeKernel((const void*)kern, dim3(grid), dim3(C::kThreads), args, kDyn, s);
}

template <typename T, int NR>
cudaError_t dispatch(int variant, const Bsr& A, PcgWork* const* ws, double* pa, double* pb, cudaStream_t s,
                     bool query, bool* eligible) {
  if constexpr (sizeof(T) == 4) {
    if (variant == 0) return launch_persistent<float, 8, 2, 8, 4, 1, NR>(A, ws, pa, pb, s, query, eligible);
    if (variant == 1) return launch_persistent<float, 4, 3, 8, 8, 1, NR>(A, ws, pa, pb, s, query, eligible);
    if (variant == 2) return launch_persistent<float, 4, 2, 8, 2, 2, NR>(A, ws, pa, pb, s, query, eligible);
    if (variant == 3) return launch_persistent<float, 2, 3, 8, 2, 3, NR>(A, ws, pa, pb, s, query, eligible);
    if (variant == 4) return launch_persistent<float, 4, 2, 16, 2, 1, NR>(A, ws, pa, pb, s, query, eligible);
    if (variant == 5) return launch_persistent<float, 4, 2, 12, 3, 1, NR>(A, ws, pa, pb, s, query, eligible);
    return launch_persistent<float, 5, 2, 16, 2, 1, NR>(A, ws, pa, pb, s, query, eligible);
  } else {
    if (variant == 0) return launch_persistent<double, 4, 2, 8, 4, 1, NR>(A, ws, pa, pb, s, query, eligible);
    if (variant == 1) return launch_persistent<double, 2, 3, 8, 4, 1, NR>(A, ws, pa, pb, s, query, eligible);
    if (variant == 2) return launch_persistent<double, 2, 2, 8, 2, 2, NR>(A, ws, pa, pb, s, query, eligible);
    if (variant == 3) return launch_persistent<double, 1, 3, 8, 2, 2, NR>(A, ws, pa, pb, s, query, eligible);
    if (variant == 4) return launch_persistent<double, 2, 2, 16, 2, 1, NR>(A, ws, pa, pb, s, query, eligible);
    if (variant == 5) return launch_persistent<double, 2, 2, 12, 3, 1, NR>(A, ws, pa, pb, s, query, eligible);
    return launch_persistent<double, 1, 3, 16, 2, 1, NR>(A, ws, pa, pb, s, query, eligible);
  }
}


constexpr int kClassicVariants = 7;

// the last kHaloVariants variants: cg_halo.cu, or -- on a system without a split that fits -- the variant of this file
// with the same capacity
constexpr int kWithoutHalo[kHaloVariants] = {2, 0};

}  // namespace

int pcg_persistent_variants() { return kClassicVariants + kHaloVariants; }

bool pcg_persistent_eligible(const Bsr& A, PcgWork& w, int variant) {
  bool ok = false;
  if (variant >= kClassicVariants) {
    if (pcg_halo_eligible(w, variant - kClassicVariants)) return true;
    variant = kWithoutHalo[variant - kClassicVariants];
  }
  PcgWork* ws[1] = {&w};
  if (w.fp32) dispatch<float, 1>(variant, A, ws, w.part_a, w.part_b, nullptr, true, &ok);
  else dispatch<double, 1>(variant, A, ws, w.part_a, w.part_b, nullptr, true, &ok);
  return ok;
}

cudaError_t launch_pcg_persistent(const Bsr& A, PcgWork& w, int variant, cudaStream_t s) {
  bool ok = false;
  if (variant >= kClassicVariants) {
    if (pcg_halo_eligible(w, variant - kClassicVariants)) return launch_pcg_halo(A, w, variant - kClassicVariants, s);
    variant = kWithoutHalo[variant - kClassicVariants];
  }
  PcgWork* ws[1] = {&w};
  const cudaError_t e = w.fp32 ? dispatch<float, 1>(variant, A, ws, w.part_a, w.part_b, s, false, &ok)
                               : dispatch<double, 1>(variant, A, ws, w.part_a, w.part_b, s, false, &ok);
  if (e == cudaSuccess && !ok) return cudaErrorInvalidConfiguration;
  return e;
}

bool pcg_persistent2_eligible(const Bsr& A, PcgWork& w0, PcgWork& w1, int variant) {
  if (variant >= kClassicVariants) return false;  // the one-reduction kernel runs one right-hand side
  bool ok = false;
  PcgWork* ws[2] = {&w0, &w1};
  if (w0.fp32) dispatch<float, 2>(variant, A, ws, nullptr, nullptr, nullptr, true, &ok);
  else dispatch<double, 2>(variant, A, ws, nullptr, nullptr, nullptr, true, &ok);
  return ok;
}

cudaError_t launch_pcg_persistent2(const Bsr& A, PcgWork& w0, PcgWork& w1, int variant, double* part_a,
                                   double* part_b, cudaStream_t s) {
  if (variant >= kClassicVariants) return cudaErrorInvalidConfiguration;
  bool ok = false;
  PcgWork* ws[2] = {&w0, &w1};
  cudaError_t e = w0.fp32 ? dispatch<float, 2>(variant, A, ws, part_a, part_b, s, false, &ok)
                          : dispatch<double, 2>(variant, A, ws, part_a, part_b, s, false, &ok);
  if (e == cudaSuccess && !ok) return cudaErrorInvalidConfiguration;
  return e;
}

}  // namespace ikr
