// vlba_pcg_small.cu -- block-Jacobi PCG on the reduced systems of small
// problems (at most kSmallPcgRows tile rows, 128 cameras), one thread-block
// cluster per problem.
//
// The persistent k_pcg (vlba_kernels.cu) streams tiles of S and crosses two
// grid barriers in each iteration: 5-6 us for a 20-keyframe window whatever
// its size, nearly all of it waiting.  Here S lives in registers for the whole
// solve and an iteration crosses two barriers of one cluster (of one block
// for up to 16 cameras), the same recurrence and stopping rule:
//
//   one warp per camera (two of 17 to 32 cameras): lane l holds columns l,
//   l + 32, ... of the camera's six rows of S, and its own copy of those
//   entries of p;
//   q = S p      each lane's partial products, then a reduce-scatter butterfly
//   -- barrier: every warp's p.q
//   x, r, z of the camera on lanes 0-5; z pushed to every block of the
//   cluster through distributed shared memory
//   -- barrier: z, and every warp's r.z and r.r
//   p = z + beta p, on every lane for its columns.
//
// What bounds it is the chain of one iteration (LDS, FMA, shuffles, barrier),
// so the cluster is as small as the registers allow (a cluster's barrier takes
// 330 cycles and more, a block's 20): one block of 16 warps up to 16 cameras (3
// columns per lane) and up to 32 (6 columns, two cameras a warp), four blocks
// up to 64 (12 columns, 72 registers of S per thread) and sixteen blocks of 8
// warps up to 128 (24 columns, 144 registers).  Measured on B200 for one LM
// iteration's solve, k_pcg against this kernel: 18 cameras and 29 PCG
// iterations 300 -> 43 us, 48 cameras and 25 iterations 280 -> 62 us, a batch
// of 48 windows of up to 36 cameras 554 -> 173 us over its three classes.
//
// Every sum runs in an order fixed by the problem's own size, so a problem
// solves the same alone and in any batch.  The cluster's blocks compute the
// same scalars from the same slots and leave the loop together.

#include <cuda_runtime.h>

#include <cstdint>

#include "vlba_common.cuh"
#include "vlba_kernels.cuh"

namespace vlba {
namespace {

// Sum over lanes 0-7 (lanes 6 and 7 hold zero), in lane 0 and its group.
__device__ __forceinline__ double group_sum(double v) {
#pragma unroll
  for (int off = 4; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}

// Address of `p` (in this block's shared memory) in block `rank` of the cluster.
__device__ __forceinline__ uint32_t peer_addr(const void* p, uint32_t rank) {
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;"
      : "=r"(a)
      : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
  return a;
}
__device__ __forceinline__ void st_peer(uint32_t a, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
__device__ __forceinline__ void st_peer(uint32_t a, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}

// Barrier over the problem's blocks: the stores before it (also those into
// other blocks' shared memory) are visible after it.
template <int C>
__device__ __forceinline__ void team_barrier() {
  if (C == 1) {
    __syncthreads();
  } else {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
}

// C blocks of W warps, N cameras per warp; CPL columns of S per lane
// (32 CPL = 6 C W N).
template <int C, int W, int CPL, int N>
__global__ void __launch_bounds__(32 * W, 1) k_pcg_small(Dev d, const uint32_t* list) {
  constexpr int kNodes = C * W * N, kRows = kNodes / 8;
  // Dot slots of a camera: its six products (a warp then sums them all, three
  // butterfly levels fewer in the chain), or one sum where six would be more
  // to push to every block than that saves (four blocks: 91 us a solve of 40
  // cameras with sums, 106 with products).
  constexpr int kPer = C == 1 ? 6 : 1, kDots = kPer * kNodes;
  static_assert(C == 1 || N == 1, "a camera a warp where blocks exchange");
  static_assert(32 * CPL == 6 * kNodes, "a lane's columns cover the system");
  __shared__ float zs[32 * CPL];
  __shared__ double s_pq[kDots], s_rz[kDots], s_rr[kDots];
  __shared__ double s_sum[2];
  __shared__ uint32_t tmap[kRows * kRows];  // tile of (I, J), J <= I
  const uint32_t P = list[blockIdx.x / C];
  if (d.ctrl[P].done) return;  // the same for every block of the cluster
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t rank = C == 1 ? 0u : blockIdx.x % C;
  const uint32_t node = (rank * W + warp) * N;  // the warp's first camera
  const uint32_t tr0 = d.prob_tr_begin[P], rows = d.prob_tr_begin[P + 1] - tr0;
  const uint32_t nodes = rows * 8u;  // padded slots have zero rows and rhs

  for (uint32_t i = threadIdx.x; i < (uint32_t)(kRows * kRows); i += 32 * W) tmap[i] = kNone;
  __syncthreads();
  for (uint32_t t = d.prob_tile_begin[P] + threadIdx.x; t < d.prob_tile_begin[P + 1]; t += 32 * W) {
    const uint32_t ij = d.tile_ij[t];
    tmap[((ij >> 16) - tr0) * kRows + ((ij & 0xFFFFu) - tr0)] = t;
  }
  __syncthreads();

  // The cameras' rows of S: from the tile right of (or on) the diagonal of
  // its tile row, else the mirrored block of the lower tile.
  float S[N][6][CPL], p[CPL];
#pragma unroll
  for (int j = 0; j < CPL; ++j) {
    const uint32_t col = lane + 32u * j, cn = col / 6u, c = col % 6u;
    p[j] = 0.0f;
#pragma unroll
    for (int u = 0; u < N; ++u) {
#pragma unroll
      for (int r = 0; r < 6; ++r) S[u][r][j] = 0.0f;
      const uint32_t n = node + u;
      if (n < nodes && cn < nodes) {
        const uint32_t I = n >> 3, J = cn >> 3;
        const bool lower = I >= J;
        const uint32_t t = lower ? tmap[I * kRows + J] : tmap[J * kRows + I];
        if (t != kNone) {
          const float* tile = d.tiles + (size_t)t * (64 * kBlock);
          if (lower) {
            const float* b = tile + ((n & 7u) * 8u + (cn & 7u)) * kBlock + c;
#pragma unroll
            for (int r = 0; r < 6; ++r) S[u][r][j] = b[6 * r];
          } else {
            const float2* b =
                reinterpret_cast<const float2*>(tile + ((cn & 7u) * 8u + (n & 7u)) * kBlock + c * 6u);
#pragma unroll
            for (int r = 0; r < 3; ++r) {
              const float2 v = b[r];
              S[u][2 * r][j] = v.x;
              S[u][2 * r + 1][j] = v.y;
            }
          }
        }
      }
    }
  }

  // The cameras' vector entries on lanes 0 to 6 N - 1 (zero on the others):
  // entry a of the warp's camera `sub`.
  const uint32_t sub = lane < 6u * N ? lane / 6u : 0u, a = lane < 6u * N ? lane % 6u : 0u;
  const bool own = node + sub < nodes && lane < 6u * N;
  const size_t at = (size_t)6 * (8u * tr0 + node + sub) + a;
  float m[6];
#pragma unroll
  for (int b = 0; b < 6; ++b) m[b] = own ? d.minv[6 * at + b] : 0.0f;
  float x = 0.0f, r = own ? d.rhs[at] : 0.0f, z, po = 0.0f;
  auto precondition = [&]() {
    z = 0.0f;
#pragma unroll
    for (int b = 0; b < 6; ++b) z += m[b] * __shfl_sync(0xffffffffu, r, 6u * sub + b);
  };
  // The camera's products v (lanes 0-5) into its slots of every block.
  auto push = [&](double* slots, double v) {
    if (kPer == 1) v = group_sum(v);
    if (C == 1) {
      if (lane < (uint32_t)(kPer * N)) slots[kPer * node + lane] = v;
    } else {
#pragma unroll
      for (int i = 0; i < kPer * C; i += 32) {
        const uint32_t e = lane + i, peer = e / (uint32_t)kPer, q = e % (uint32_t)kPer;
        const double w = __shfl_sync(0xffffffffu, v, q);
        if (e < (uint32_t)(kPer * C)) st_peer(peer_addr(&slots[kPer * node + q], peer), w);
      }
    }
  };
  // z and the products of r.z and r.r into every block of the cluster.
  auto publish = [&]() {
    if (C == 1) {
      if (lane < 6u * N) zs[6 * node + lane] = z;
    } else {
#pragma unroll
      for (int i = 0; i < 6 * C; i += 32) {
        const uint32_t e = lane + i, peer = e / 6u, q = e % 6u;
        const float v = __shfl_sync(0xffffffffu, z, q);
        if (e < 6u * C) st_peer(peer_addr(&zs[6 * node + q], peer), v);
      }
    }
    push(s_rz, (double)r * (double)z);
    push(s_rr, (double)r * (double)r);
  };
  // A lane's slots by a tree, then a butterfly over the lanes.
  auto sum = [&](const double* s) {
    constexpr int kLane = (kDots + 31) / 32;
    double v[kLane];
#pragma unroll
    for (int i = 0; i < kLane; ++i) v[i] = lane + 32 * i < (uint32_t)kDots ? s[lane + 32 * i] : 0.0;
#pragma unroll
    for (int n = kLane; n > 1; n = (n + 1) / 2)
#pragma unroll
      for (int i = 0; i < n / 2; ++i) v[i] += v[n - 1 - i];
    return warp_sum(v[0]);
  };
  // The sums every thread of the block needs, each by one warp: with all
  // sixteen summing for themselves the shuffle unit was the bound.
  auto totals = [&](const double* s0, const double* s1) {
    if (warp < 2 && (warp == 0 || s1)) {
      const double v = sum(warp == 0 ? s0 : s1);
      if (lane == 0) s_sum[warp] = v;
    }
    __syncthreads();
    return make_double2(s_sum[0], s_sum[1]);
  };

  precondition();
  if (C > 1) team_barrier<C>();  // every block runs before its memory is written
  publish();
  team_barrier<C>();
  const double2 first = totals(s_rz, s_rr);
  double rz = first.x, rr = first.y;
  const LmParams& lp = d.params[P];
  const double bnorm = sqrt(rr);
  // |r| <= stop without the root: on squares; a negative tolerance is never met.
  const double stop = lp.pcg_relative_tolerance * bnorm, stop2 = stop >= 0.0 ? stop * stop : -1.0;
  const uint32_t cap = lp.max_pcg_iterations;
  uint32_t iters = 0, status = 0;
  // pcg_init (ba.wgsl:420-439): done when |b| = 0 or r.z <= 0.
  if (rr > 0.0 && rz > 0.0 && cap != 0u) {
    float beta = 0.0f;
    for (;;) {
      const double inv_rz = 1.0 / rz;  // for beta, off the chain of the sums
      float acc[N][6];
#pragma unroll
      for (int u = 0; u < N; ++u)
#pragma unroll
        for (int q = 0; q < 6; ++q) acc[u][q] = 0.0f;
#pragma unroll
      for (int j = 0; j < CPL; ++j) {
        p[j] = __fmaf_rn(beta, p[j], zs[lane + 32 * j]);
#pragma unroll
        for (int u = 0; u < N; ++u)
#pragma unroll
          for (int q = 0; q < 6; ++q) acc[u][q] = __fmaf_rn(S[u][q][j], p[j], acc[u][q]);
      }
      po = __fmaf_rn(beta, po, z);
      // The row sums over the lanes, row a back to its lane.
      const uint32_t part = a >= 3u ? a - 3u : a;
      const uint32_t src = (a >= 3u ? 16u : 0u) + (part == 2u ? 8u : 0u);
      float qa = 0.0f;
#pragma unroll
      for (int w = 0; w < N; ++w) {
        float u, v;
        row_sums(acc[w], lane, u, v);
        const float qu = __shfl_sync(0xffffffffu, u, src), qv = __shfl_sync(0xffffffffu, v, src);
        if (sub == (uint32_t)w) qa = part == 1u ? qv : qu;
      }
      if (!own) qa = 0.0f;
      push(s_pq, (double)po * (double)qa);
      team_barrier<C>();
      const double pq = totals(s_pq, nullptr).x;
      if (!(pq > 0.0) || !isfinite(pq)) {
        status = 2;  // non-positive curvature: x unchanged
        break;
      }
      const float alpha = (float)(rz / pq);
      x = x + alpha * po;
      r = r - alpha * qa;
      precondition();
      publish();
      team_barrier<C>();
      const double2 now = totals(s_rz, s_rr);
      const double rz_new = now.x;
      rr = now.y;
      ++iters;
      const double rz_inv = inv_rz;
      rz = rz_new;
      if (rr <= stop2 || !(rz_new > 0.0)) break;
      if (iters >= cap) {
        status = 1;
        break;
      }
      beta = (float)(rz_new * rz_inv);
    }
  }
  if (own) d.x[at] = x;
  if (rank == 0 && threadIdx.x == 0) {
    PcgState& st = d.pcg[P];
    st.iters = iters;
    st.status = status;
    st.bnorm = bnorm;
    st.rnorm = sqrt(rr);
    st.rz = rz;
    st.active = 0u;
  }
}

// The launch of a class's kernel on `problems` clusters of C blocks.
template <int C, int W, int CPL, int N>
struct ClassLaunch {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  cudaError_t error = cudaSuccess;
  ClassLaunch(uint32_t problems, cudaStream_t s) {
    if (C > 8)  // beyond the portable cluster size
      error = cudaFuncSetAttribute(k_pcg_small<C, W, CPL, N>,
                                   cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    cfg.gridDim = dim3(C * problems);
    cfg.blockDim = dim3(32 * W);
    cfg.stream = s;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = C;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = C > 1 ? 1 : 0;
  }
};

template <int C, int W, int CPL, int N>
cudaError_t launch_class(const Dev& d, uint32_t begin, uint32_t end, cudaStream_t s) {
  if (begin == end) return cudaSuccess;
  const ClassLaunch<C, W, CPL, N> l(end - begin, s);
  if (l.error != cudaSuccess) return l.error;
  return cudaLaunchKernelEx(&l.cfg, k_pcg_small<C, W, CPL, N>, d, d.small_list + begin);
}

// Whether the device can place one of the class's clusters (a partition of it
// may have no 16 SMs in one GPC).
template <int C, int W, int CPL, int N>
bool class_fits() {
  const ClassLaunch<C, W, CPL, N> l(1, nullptr);
  int clusters = 0;
  const bool ok = l.error == cudaSuccess &&
                  cudaOccupancyMaxActiveClusters(&clusters, k_pcg_small<C, W, CPL, N>, &l.cfg) ==
                      cudaSuccess;
  cudaGetLastError();
  return ok && clusters > 0;
}

}  // namespace

int small_pcg_class(uint32_t rows) {
  if (rows <= 2) return 0;
  if (rows <= 4) return 1;
  if (rows <= 8) return 2;
  if (rows <= kSmallPcgRows) return 3;
  return -1;
}

uint32_t small_pcg_rows(uint32_t max_cluster) {
  if (max_cluster < 4 || !class_fits<4, 16, 12, 1>()) return 4;
  return max_cluster < 16 || !class_fits<16, 8, 24, 1>() ? 8 : kSmallPcgRows;
}

cudaError_t launch_pcg_small(const Dev& d, cudaStream_t s) {
  cudaError_t e = launch_class<1, 16, 3, 1>(d, d.small_off[0], d.small_off[1], s);
  if (e == cudaSuccess) e = launch_class<1, 16, 6, 2>(d, d.small_off[1], d.small_off[2], s);
  if (e == cudaSuccess) e = launch_class<4, 16, 12, 1>(d, d.small_off[2], d.small_off[3], s);
  if (e == cudaSuccess) e = launch_class<16, 8, 24, 1>(d, d.small_off[3], d.small_off[4], s);
  return e;
}

}  // namespace vlba
