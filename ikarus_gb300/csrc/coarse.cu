// Coarse correction of the block-Jacobi CG: an additive two-level preconditioner (sm_103a).
//
//   M^-1 r = D^-1 r + P A_c^-1 P^T r,   A_c = P^T K P
//
// D is the 3x3 block diagonal of the tangent K (the CG's block-Jacobi preconditioner).  P has six columns per
// aggregate of nodes, the rigid-body modes of that aggregate: translations e_k and rotations e_k x y about its
// centroid (y = node position - centroid), zero at constrained dofs.  With slab aggregates along a slender
// body's long axis the coarse space carries the beam-like bending and torsion modes that make block-Jacobi CG
// slow there.  M is symmetric positive definite (D^-1 SPD, P A_c^-1 P^T semi-definite), so CG stays CG.
//
// Per CG iteration, after the update kernel (which leaves z = D^-1 r and the partial r.D^-1 r in kRzF), two
// kernels:
//   restrict and solve: one CTA per chunk (up to 2048 nodes of one aggregate) writes the chunk's six sums of
//             P^T r; the CTA that finishes last sums the chunks of every aggregate in a fixed order (r_c), forms
//             e = A_c^-1 r_c with the dense inverse, r.z = r.D^-1 r + r_c.e, and beta (or the initial r.z);
//   prolong:  z += P e.
// Setup per tangent (A_c): one pass over the matrix.  A block K_IJ of rows in aggregate b and columns in aggregate b + d
// (|d| <= reach) adds P_I^T K_IJ P_J to A_c(b, b + d); a thread sums W = sum_J K_IJ P_J of its row per d (27 FP64
// instructions per block, the translations being additions), then P_I^T W, a CTA its 256 rows, and a second kernel the
// CTAs of an aggregate in order.  The host symmetrises A_c and inverts it (ikr_ls_s in host_internal.h).  All sums are
// fixed-order: results are bit-identical run to run.  Measured at 140 481 rows, three distances: 18 probe products
// K V_m (164 us each, the matrix read 18 times) and their restrictions took 3.3 ms, this pass 0.47 ms.
#include "cg_common.cuh"

namespace ikr {

namespace {

using namespace cg;
constexpr int kThreads = 1024;       // CTA of the restrict-and-solve kernel (a chunk is up to 2048 nodes)
static_assert(kCoarseMaxDofs <= kThreads, "the coarse solve splits the coarse dofs over the threads of one CTA");
constexpr int kCoarseTicket = 4;     // ticket slot of its last-block reduction (scalar slot 14)

// node data: offset from the aggregate centroid (x, y, z) and, in the fourth lane as integer bits, the
// aggregate id (bits 0-23) and the free-dof mask (bits 24-26)
struct NodeP {
  float y[3];
  int agg;
  int mask;
};
__device__ __forceinline__ NodeP node_p(const float4* __restrict__ y4, int node) {
  const float4 v = __ldg(y4 + node);
  const int bits = __float_as_int(v.w);
  return {{v.x, v.y, v.z}, bits & 0xFFFFFF, (bits >> 24) & 7};
}

// the six mode columns of P at a node (3 x 6), masked: P[c][m]
__device__ __forceinline__ void p_cols(const NodeP& n, double P[3][6]) {
  const double yx = n.y[0], yy = n.y[1], yz = n.y[2];
  const double cols[3][6] = {{1, 0, 0, 0.0, yz, -yy}, {0, 1, 0, -yz, 0.0, yx}, {0, 0, 1, yy, -yx, 0.0}};
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const double on = ((n.mask >> c) & 1) ? 1.0 : 0.0;
#pragma unroll
    for (int m = 0; m < 6; ++m) P[c][m] = on * cols[c][m];
  }
}

// P^T r per chunk; the CTA that finishes last sums the chunks of every aggregate in a fixed order (r_c), forms
// e = A_c^-1 r_c with the dense inverse, r.z = r.D^-1 r + r_c.e and beta (or the initial r.z)
template <typename T>
__global__ void __launch_bounds__(kThreads) coarse_restrict_solve_kernel(Coarse C, const T* __restrict__ r,
                                                                         double* scal, int init) {
  __shared__ double sh[32];
  __shared__ double rc[kCoarseMaxDofs];
  __shared__ double red[kThreads];
  __shared__ bool last;
  if (scal[kDone] != 0.0) return;
  const int k = blockIdx.x;
  double s[6] = {0, 0, 0, 0, 0, 0};
  for (int i = C.chunk_off[k] + threadIdx.x; i < C.chunk_off[k + 1]; i += blockDim.x) {
    const int node = __ldg(C.nodes + i);
    const NodeP n = node_p(C.y4, node);
    const V3<T> rv = load3(r, node);
    double P[3][6];
    p_cols(n, P);
#pragma unroll
    for (int m = 0; m < 6; ++m) s[m] += P[0][m] * double(rv.x) + P[1][m] * double(rv.y) + P[2][m] * double(rv.z);
  }
#pragma unroll
  for (int m = 0; m < 6; ++m) {
    const double t = block_sum_all(s[m], sh);
    if (threadIdx.x == 0) C.rpart[6 * k + m] = t;
  }
  if (!publish_and_check_last(&tickets(scal)[kCoarseTicket], &last)) return;
  const int nc = C.n_c;
  for (int j = threadIdx.x; j < nc; j += blockDim.x) {
    const int a = j / 6, m = j - 6 * a;
    double t = 0.0;
    for (int q = C.agg_chunk[a]; q < C.agg_chunk[a + 1]; ++q) t += __ldcg(C.rpart + 6 * q + m);
    rc[j] = t;
  }
  __syncthreads();
  // e = A_c^-1 r_c: thread t forms the part of entry i = t mod n_c over segment t / n_c of the columns (A_c^-1
  // is symmetric: column-major reads, coalesced along i; all loads of a thread independent), then the segments
  // are added in order
  const T* ainv = static_cast<const T*>(C.ainv);
  const int t = threadIdx.x, nseg = blockDim.x / nc, seg_len = (nc + nseg - 1) / nseg;
  const int i = t % nc, seg = t / nc;
  double acc = 0.0;
  if (seg < nseg) {
    const int j1 = min(nc, (seg + 1) * seg_len);
#pragma unroll 8
    for (int j = seg * seg_len; j < j1; ++j) acc += double(__ldg(ainv + (size_t)j * nc + i)) * rc[j];
  }
  red[t] = acc;
  __syncthreads();
  double qc = 0.0;
  if (t < nc) {
    double ev = 0.0;
    for (int g = 0; g < nseg; ++g) ev += red[g * nc + t];
    const T ei = T(ev);
    static_cast<T*>(C.e)[t] = ei;
    qc = rc[t] * double(ei);
  }
  qc = block_sum_all(qc, sh);
  if (threadIdx.x == 0) {
    const double rz = scal[kRzF] + qc;
    if (init) {
      scal[kRz] = rz;
      scal[kBeta] = 0.0;
    } else {
      scal[kBeta] = rz / scal[kRz];
      scal[kRz] = rz;
    }
    tickets(scal)[kCoarseTicket] = 0u;
  }
}

template <typename T>
__global__ void __launch_bounds__(256) coarse_prolong_kernel(Coarse C, T* z, const double* __restrict__ scal) {
  __shared__ T e[kCoarseMaxDofs];
  if (scal[kDone] != 0.0) return;
  for (int j = threadIdx.x; j < C.n_c; j += blockDim.x) e[j] = static_cast<const T*>(C.e)[j];
  __syncthreads();
  for (int node = blockIdx.x * blockDim.x + threadIdx.x; node < C.n_rows; node += gridDim.x * blockDim.x) {
    const NodeP n = node_p(C.y4, node);
    const T* ea = e + 6 * n.agg;
    const T yx = T(n.y[0]), yy = T(n.y[1]), yz = T(n.y[2]);
    // t + w x y with t = e[0..2], w = e[3..5]
    T d0 = ea[0] + ea[4] * yz - ea[5] * yy;
    T d1 = ea[1] + ea[5] * yx - ea[3] * yz;
    T d2 = ea[2] + ea[3] * yy - ea[4] * yx;
    if (!(n.mask & 1)) d0 = T(0);
    if (!(n.mask & 2)) d1 = T(0);
    if (!(n.mask & 4)) d2 = T(0);
    const V3<T> zv = load3rw(z, node);
    store3(z, node, zv.x + d0, zv.y + d1, zv.z + d2);
  }
}

// Lane sums of the 36 entries in v: halves are exchanged, so the butterfly takes 37 additions instead of 180.  The lane ends
// with the sums of entries first .. first + n - 1 (n <= 2) in v[0], v[1].
template <int SIZE, int M>
__device__ __forceinline__ void reduce_step(double (&v)[36], int lane, int& first, int& n) {
  constexpr int kHalf = (SIZE + 1) / 2;
  const bool up = lane & M;
#pragma unroll
  for (int k = 0; k < kHalf; ++k) {
    const double hi = kHalf + k < SIZE ? v[kHalf + k] : 0.0;
    v[k] = (up ? hi : v[k]) + __shfl_xor_sync(0xffffffffu, up ? v[k] : hi, M);
  }
  first += up ? kHalf : 0;
  n = up ? n - kHalf : min(n, kHalf);
  if constexpr (M > 1) reduce_step<kHalf, M / 2>(v, lane, first, n);
}
__device__ __forceinline__ void reduce_36(double (&v)[36], int lane, int& first, int& n) {
  first = 0, n = 36;
  reduce_step<36, 16>(v, lane, first, n);
}

// float to double of zeros and normal numbers on the integer pipe (a conversion instruction is as slow as the FP64 ones)
__device__ __forceinline__ bool widens(float f) {
  const uint32_t m = __float_as_uint(f) & 0x7fffffffu;
  return m == 0 || m - 0x800000u < 0x7f000000u;
}
__device__ __forceinline__ double widened(float f) {
  const uint32_t b = __float_as_uint(f), m = b & 0x7fffffffu;
  return __hiloint2double((int)((b & 0x80000000u) | (m ? (m >> 3) + (896u << 20) : 0u)), (int)(b << 29));
}
__device__ __forceinline__ bool widens(double) { return true; }
__device__ __forceinline__ double widened(double v) { return v; }

// part[((d + reach) * n_parts + part) * 36 + 6 r + m], one CTA per run of kGalerkinRows nodes of a chunk: a thread forms
// W = sum_j K_ij P_j of its row i over the columns of aggregate b + d, the CTA sums P_i^T W.  Bound by the FP64 pipe (27
// operations per block and, before, twelve conversions), so only the distances that a row of the CTA has are walked, P_i^T W
// takes its 36 operations and the sums share the butterfly.  140 481 rows of 27 blocks, 16 slabs, FP32: 0.83 -> 0.47 ms (0.66
// with conversion instructions).  Where nodes are numbered along the slabs' axis, every warp has rows of all three distances
// and walks 45 blocks instead of 27.
constexpr int kGalerkinRows = 256;
template <typename T>
__global__ void __launch_bounds__(kGalerkinRows) coarse_galerkin_kernel(Coarse C, Bsr A, const T* __restrict__ val,
                                                                        int reach, int runs, double* __restrict__ part) {
  __shared__ double sh[kGalerkinRows / 32][36];
  const int chunk = blockIdx.x / runs, run = blockIdx.x - chunk * runs, lane = threadIdx.x & 31;
  const int i = C.chunk_off[chunk] + run * kGalerkinRows + threadIdx.x;
  const bool active = i < C.chunk_off[chunk + 1];
  const int node = active ? __ldg(C.nodes + i) : 0;
  const NodeP n = node_p(C.y4, node);
  const int g0 = A.slice_off[node >> 5], width = active ? A.slice_off[(node >> 5) + 1] - g0 : 0, l = node & 31;
  unsigned mine = 0;  // bit d + reach: the row has a column in aggregate b + d
#pragma unroll 4
  for (int k = 0; k < width; ++k) {
    const int J = __ldg(A.col_sell + 32 * (int64_t)(g0 + k) + l);
    mine |= 1u << (node_p(C.y4, J).agg - n.agg + reach);
  }
  for (int d = -reach; d <= reach; ++d) {
    const bool any = (mine >> (d + reach)) & 1u;
    double* out = part + ((size_t)(d + reach) * gridDim.x + blockIdx.x) * 36;
    if (!__syncthreads_or(any)) {  // no row of this run couples with aggregate b + d
      if (threadIdx.x < 36) out[threadIdx.x] = 0.0;
      continue;
    }
    double W[3][6] = {};
    for (int k = 0; any && k < width; ++k) {
      const int J = __ldg(A.col_sell + 32 * (int64_t)(g0 + k) + l);
      const NodeP nj = node_p(C.y4, J);
      if (nj.agg != n.agg + d) continue;
      const T* v = val + (int64_t)(g0 + k) * 288 + l;
      T t[3][3];
      bool normal = widens(nj.y[0]) && widens(nj.y[1]) && widens(nj.y[2]);
#pragma unroll
      for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          t[c][q] = (nj.mask >> q) & 1 ? __ldg(v + 96 * c + 32 * q) : T(0);
          normal = normal && widens(t[c][q]);
        }
      double y0 = widened(nj.y[0]), y1 = widened(nj.y[1]), y2 = widened(nj.y[2]), a[3][3];
#pragma unroll
      for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int q = 0; q < 3; ++q) a[c][q] = widened(t[c][q]);
      if (!normal) {
        asm volatile("");  // a branch: as selects the conversions would run for every block
        y0 = nj.y[0], y1 = nj.y[1], y2 = nj.y[2];
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
          for (int q = 0; q < 3; ++q) a[c][q] = t[c][q];
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const double a0 = a[c][0], a1 = a[c][1], a2 = a[c][2];
        W[c][0] += a0, W[c][1] += a1, W[c][2] += a2;
        W[c][3] = fma(a2, y1, fma(-a1, y2, W[c][3]));  // e_k x y
        W[c][4] = fma(a0, y2, fma(-a2, y0, W[c][4]));
        W[c][5] = fma(a1, y0, fma(-a0, y1, W[c][5]));
      }
    }
    double v[36];  // P_i^T W: the free components, and y_i x them
    const double y0 = n.y[0], y1 = n.y[1], y2 = n.y[2];
#pragma unroll
    for (int m = 0; m < 6; ++m) {
      const double w0 = (n.mask & 1) ? W[0][m] : 0.0, w1 = (n.mask & 2) ? W[1][m] : 0.0, w2 = (n.mask & 4) ? W[2][m] : 0.0;
      v[m] = w0, v[6 + m] = w1, v[12 + m] = w2;
      v[18 + m] = fma(y1, w2, -y2 * w1);
      v[24 + m] = fma(y2, w0, -y0 * w2);
      v[30 + m] = fma(y0, w1, -y1 * w0);
    }
    int first, cnt;
    reduce_36(v, lane, first, cnt);
    if (cnt > 0) sh[threadIdx.x >> 5][first] = v[0];
    if (cnt > 1) sh[threadIdx.x >> 5][first + 1] = v[1];
    __syncthreads();
    if (threadIdx.x < 36) {
      double t = 0.0;
#pragma unroll
      for (int w = 0; w < kGalerkinRows / 32; ++w) t += sh[w][threadIdx.x];
      out[threadIdx.x] = t;
    }
    __syncthreads();
  }
}
// blk[((d + reach) * n_agg + b) * 36 + q]: the runs of aggregate b in order
__global__ void coarse_blocks_kernel(Coarse C, int nd, int runs, const double* __restrict__ part,
                                     double* __restrict__ blk) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nd * C.n_agg * 36) return;
  const int q = t % 36, b = t / 36 % C.n_agg, d = t / 36 / C.n_agg;
  double s = 0.0;
  const size_t n_parts = (size_t)C.n_chunks * runs;
  for (int k = C.agg_chunk[b] * runs; k < C.agg_chunk[b + 1] * runs; ++k) s += part[(d * n_parts + k) * 36 + q];
  blk[t] = s;
}

int grid_for(int n, int bs, int cap) {
  int b = (n + bs - 1) / bs;
  return b < 1 ? 1 : (b > cap ? cap : b);
}

}  // namespace

void launch_coarse_correction(const Coarse& C, const PcgWork& w, bool init, cudaStream_t s) {
  if (w.fp32) {
    coarse_restrict_solve_kernel<float><<<C.n_chunks, kThreads, 0, s>>>(C, (const float*)w.r, w.scal, init ? 1 : 0);
    coarse_prolong_kernel<float><<<w.grid, 256, 0, s>>>(C, (float*)w.z, w.scal);
  } else {
    coarse_restrict_solve_kernel<double><<<C.n_chunks, kThreads, 0, s>>>(C, (const double*)w.r, w.scal, init ? 1 : 0);
    coarse_prolong_kernel<double><<<w.grid, 256, 0, s>>>(C, (double*)w.z, w.scal);
  }
}
int coarse_galerkin_runs(int chunk_rows) { return (chunk_rows + kGalerkinRows - 1) / kGalerkinRows; }
void launch_coarse_galerkin(const Coarse& C, const Bsr& A, bool fp32, int reach, int runs, double* part, double* blk,
                            cudaStream_t s) {
  const int grid = C.n_chunks * runs;
  if (fp32) coarse_galerkin_kernel<float><<<grid, kGalerkinRows, 0, s>>>(C, A, (const float*)A.val, reach, runs, part);
  else coarse_galerkin_kernel<double><<<grid, kGalerkinRows, 0, s>>>(C, A, (const double*)A.val, reach, runs, part);
  const int nd = 2 * reach + 1;
  coarse_blocks_kernel<<<(nd * C.n_agg * 36 + 127) / 128, 128, 0, s>>>(C, nd, runs, part, blk);
}

}  // namespace ikr
