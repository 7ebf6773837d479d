// vlba_pcg_team.cu -- block-Jacobi PCG on reduced systems that fit the
// registers and shared memory of a team of SMs (past the cluster kernels' 128
// cameras, up to 576 cameras of a dense system, and 4,736, 2,808 or 1,328 of a
// street whose tile rows reach 2, 6 or 12 rows to each side).
//
// The persistent k_pcg (vlba_kernels.cu) reads S again in every iteration,
// sums partials of both triangles through global memory and crosses two grid
// barriers: 20 us an iteration for 1,400 street cameras, whose S of 5 MB needs
// none of that.  Here a problem has a team of blocks, one per SM; a block owns
// consecutive cameras and keeps their rows of S (both triangles, the columns
// of the tile rows they touch) on the chip for the whole solve, so each
// row of q = S p is summed where it is used and only z and three dots cross
// blocks.  The same recurrence and stopping rule as k_pcg; two exchanges an
// iteration, three waits in a row:
//
//   q = S p for the block's rows, p.q           -> slot; all slots awaited
//   x, r, z for the block's rows, r.z, r.r      -> z words and slot; all slots
//                                                  awaited, then the z words
//   p = z + beta p for the columns the block reads
//
// An exchange has no barrier, flag or fence: every word published carries the
// exchange's number beside its 32 bits of value (one 64-bit store, single-copy
// atomic), so a reader that finds the number has the value.  A word is written
// again only after its writer has seen every block's slot of the exchange in
// between, which each block publishes after its own reads.  The numbers go on
// from one solve to the next (team_epoch), so what an earlier solve left is never
// taken for news (after a wait that gave up, whose blocks may have stopped at
// different numbers, the host clears words and numbers).  A slot, and a block's
// z, has its 128-byte lines to itself: with eight slots a line, polled by a
// hundred blocks while eight write, an exchange took 3,800 cycles of 148 blocks,
// alone in a line 1,800 (a counter barrier with loads behind it: 3,000; a kernel
// of exchanges and nothing else on B200).
//
// What bounds an iteration is the trips through L2 (a store, then loads that find
// it) and the chain of sums between them; the team is the smallest whose blocks
// hold their rows in registers (polls lengthen with the team), else all of the
// device with up to kExtra more parts a block.  Measured on B200, k_pcg and this
// kernel, us per PCG iteration of 60, the load of S in it: dense systems of 132
// cameras 13.3 and 4.7, 300 10.2 and 5.3, 400 10.8 and 6.8, 500 11.2 and 7.9, 576
// 12.0 and 8.8; streets of 300 cameras 14.2 and 4.7, 1,400 21.0 and 6.0, 2,800
// 14.5 and 8.8: the line lies where the rows no longer fit.  A problem's team,
// its blocks' rows and every sum's order follow from the problem alone; teams of
// several problems run beside each other in rounds that fit the device, a launch
// each, so a problem solves the same alone and in any batch.  Every wait is
// bounded.

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <vector>

#include "vlba_common.cuh"
#include "vlba_kernels.cuh"

namespace vlba {
namespace {

constexpr int kTeamThreads = 256, kTeamWarps = kTeamThreads / 32;
constexpr int kHeld = 2;                              // parts a warp holds in registers
constexpr uint32_t kRegParts = kHeld * kTeamWarps;
constexpr uint32_t kTeamMaxNodes = kTeamThreads / 8;  // eight threads a camera
constexpr uint32_t kTeamBlocks = 148;                // blocks in a team at most
constexpr uint32_t kTeamMaxCols = 192;                // tile columns a block reads
constexpr int kTeamPolls = (kTeamBlocks + 31) / 32;  // warps that await the slots
constexpr int kInFlight = 4;                          // pairs of z words in flight per thread
constexpr uint32_t kSegTiles = 8, kSegment = 48 * kSegTiles;  // columns of a part: a camera's
                                                      // six rows over one segment
constexpr int kSegVec = kSegment / 128;               // float4 per lane and row
constexpr uint32_t kPartFloats = 6 * kSegment;
constexpr uint32_t kExtra = 22;                       // parts kept in shared memory
// Dynamic shared memory a block may take: sm_100's 227 KB less the static
// arrays.  The launch attribute is always set to it, whatever a plan needs: it
// belongs to the kernel, and another thread's smaller plan set it below what
// this one was about to launch with.
constexpr size_t kTeamMaxSmem = (227 - 1) * 1024;

__device__ __forceinline__ void put_word(unsigned long long* a, uint32_t value, uint32_t epoch) {
  const unsigned long long w = ((unsigned long long)epoch << 32) | value;
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(a), "l"(w) : "memory");
}
// Two words with one request (each single-copy atomic).
__device__ __forceinline__ void get_words(const unsigned long long* a, unsigned long long& w0,
                                          unsigned long long& w1) {
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(w0), "=l"(w1) : "l"(a) : "memory");
}
__device__ __forceinline__ bool fresh(unsigned long long w, uint32_t epoch) {
  return (uint32_t)(w >> 32) == epoch;
}
__device__ __forceinline__ double join(unsigned long long lo, unsigned long long hi) {
  return __hiloint2double((int)(uint32_t)hi, (int)(uint32_t)lo);
}

// Bounded polling: true while the deadline is ahead (the timer, slow to read,
// only every 256 misses).
struct Deadline {
  unsigned long long limit_ns;
  unsigned long long t_end = 0;
  uint32_t misses = 0;
  __device__ __forceinline__ bool wait() {
    if ((++misses & 255u) != 0u) return true;
    const unsigned long long t = now_ns();
    if (t_end == 0) t_end = t + limit_ns;
    return t <= t_end;
  }
};

// Sum of this warp's 32 of the team's slots of V doubles each, awaited, in a
// fixed order; false when a slot never came.
template <int V>
__device__ __forceinline__ bool gather_slots(const unsigned long long* slots, uint32_t size,
                                             uint32_t epoch, unsigned long long limit_ns,
                                             double (&sum)[V]) {
  const uint32_t g = threadIdx.x;  // warp w has slots 32 w to 32 w + 31
  unsigned long long w[2 * V];
  bool ok = true;
#pragma unroll
  for (int v = 0; v < 2 * V; ++v) w[v] = (unsigned long long)epoch << 32;
  if (g < size) {
    Deadline dl{limit_ns};
    for (;;) {
      bool miss = false;
#pragma unroll
      for (int v = 0; v < 2 * V; v += 2) get_words(slots + kLineWords * (size_t)g + v, w[v], w[v + 1]);
#pragma unroll
      for (int v = 0; v < 2 * V; ++v) miss = miss || !fresh(w[v], epoch);
      if (!miss) break;
      if (!dl.wait()) {
        ok = false;
        break;
      }
    }
  }
  ok = __all_sync(0xffffffffu, ok);
#pragma unroll
  for (int v = 0; v < V; ++v) sum[v] = warp_sum(join(w[2 * v], w[2 * v + 1]));
  return ok;
}

// Block `absent` (kNone: none) stays out, for the test of the waits.
__global__ void __launch_bounds__(kTeamThreads, 1) k_pcg_team(Dev d, uint32_t first, uint32_t absent,
                                                              unsigned long long limit_ns) {
  extern __shared__ __align__(16) float smem[];
  __shared__ double s_a[kTeamWarps], s_b[kTeamWarps], s_rz[kTeamPolls], s_rr[kTeamPolls],
      s_pq[kTeamPolls];
  __shared__ int s_fail;
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  if (tid == 0) s_fail = 0;
  const TeamCta T = d.team_cta[first + blockIdx.x];
  const uint32_t P = T.prob;
  if (d.ctrl[P].done) return;  // the same for the whole team
  if (blockIdx.x == absent) return;
  const uint32_t nn = T.node1 - T.node0, L = 48u * T.ncols, nseg = (T.ncols + kSegTiles - 1) / kSegTiles;
  const uint32_t parts = nn * nseg, Lp = nseg * kSegment;
  const uint32_t tr0 = d.prob_tr_begin[P], slot0 = 8u * tr0;
  const uint32_t* cols = d.team_cols + T.col_begin;  // tile rows (of the problem), ascending
  const uint32_t staged = max(min(parts, kRegParts), parts > kRegParts ? parts - kRegParts : 0u);
  float* const S = smem;                                  // [staged] parts of [6][kSegment]
  float* const p = S + (size_t)staged * kPartFloats;      // [Lp], zero past L
  float* const z_in = p + Lp;                             // [L]
  float* const part = z_in + Lp;                          // [nseg][6 nn] products
  // Where each pair of the block's columns finds its z.
  uint32_t* const z_at = reinterpret_cast<uint32_t*>(part + (size_t)nseg * 6 * nn);  // [L / 2]
  const unsigned long long* const zw = d.team_z + T.z_team;
  unsigned long long* const z_mine = d.team_z + T.z_team + T.z_own;
  unsigned long long* const pq_slots = d.team_slots + kLineWords * (size_t)T.slot_base;
  unsigned long long* const rz_slots = pq_slots + kLineWords * (size_t)d.team_slots_total;

  // Part q (camera q % nn, segment q / nn) of the block's rows of S: parts
  // [q0, q1) into shared memory, a camera and tile column per warp at a time.
  auto stage = [&](uint32_t q0, uint32_t q1) {
    for (uint32_t it = warp; it < (q1 - q0) * kSegTiles; it += kTeamWarps) {
      const uint32_t q = q0 + it / kSegTiles, kk = it % kSegTiles;
      const uint32_t node = T.node0 + q % nn, k = q / nn * kSegTiles + kk;
      const uint32_t I = node >> 3, li = node & 7u, J = k < T.ncols ? cols[k] : 0u;
      const uint32_t t = k < T.ncols ? d.team_ents[T.ent_begin + (I - (T.node0 >> 3)) * T.ncols + k]
                                     : kNone;
      float* dst = S + (size_t)(q - q0) * kPartFloats + 48u * kk;
      const float* src = d.tiles + (size_t)t * (64 * kBlock) + (I >= J ? li * 288u : li * 36u);
#pragma unroll
      for (int i = 0; i < 9; ++i) {
        const uint32_t e = lane + 32u * i, lj = e / 36u, w = e % 36u;
        // Below or on the diagonal: block (li, lj) row by row; above it: the
        // mirrored block (lj, li) column by column.
        const float v = t == kNone ? 0.0f : (I >= J ? src[e] : src[lj * 288u + w]);
        const uint32_t a = I >= J ? w / 6u : w % 6u, c = I >= J ? w % 6u : w / 6u;
        dst[a * kSegment + lj * 6u + c] = v;
      }
    }
  };
  float4 Sr[kHeld][6][kSegVec];  // this warp's parts: warp, warp + kTeamWarps
  stage(0, min(parts, kRegParts));
  __syncthreads();
#pragma unroll
  for (int u = 0; u < kHeld; ++u) {
    const uint32_t it = warp + u * kTeamWarps;
    const float4* s4 = reinterpret_cast<const float4*>(S + (size_t)it * kPartFloats);
#pragma unroll
    for (int q = 0; q < 6; ++q)
#pragma unroll
      for (int j = 0; j < kSegVec; ++j)
        Sr[u][q][j] = it < parts ? s4[q * (kSegment / 4) + lane + 32 * j]
                                 : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  }
  if (parts > kRegParts) {
    __syncthreads();
    stage(kRegParts, parts);
  }
  uint32_t node_held[kHeld], seg_held[kHeld];
#pragma unroll
  for (int u = 0; u < kHeld; ++u) {
    const uint32_t it = min(warp + u * kTeamWarps, parts - 1u);
    node_held[u] = it % nn;
    seg_held[u] = it / nn;
  }
  for (uint32_t e = tid; e < Lp; e += kTeamThreads) p[e] = 0.0f;
  for (uint32_t e = 2u * tid; e < L; e += 2u * kTeamThreads) {
    // The owner of a camera: the last block whose first camera is not past it.
    const uint32_t entry = 48u * cols[e / 48u] + e % 48u, node = entry / 6u;
    uint32_t g = (uint32_t)((uint64_t)node * T.size / (8u * (d.prob_tr_begin[P + 1] - tr0)));
    const TeamCta* team = d.team_cta + T.slot_base;
    while (g + 1 < T.size && team[g + 1].node0 <= node) ++g;
    while (team[g].node0 > node) --g;
    z_at[e / 2u] = team[g].z_own + entry - 6u * team[g].node0;
  }

  // Eight threads a camera: vector entry a of camera gi.
  const uint32_t gi = tid >> 3, a = tid & 7u;
  const bool own = gi < nn && a < 6u;
  const uint32_t nwarp = (nn + 3) / 4;  // warps that own cameras
  const size_t at = (size_t)6 * (slot0 + T.node0 + gi) + a;
  float m[6];
#pragma unroll
  for (int b = 0; b < 6; ++b) m[b] = own ? d.minv[6 * at + b] : 0.0f;
  float x = 0.0f, r = own ? d.rhs[at] : 0.0f, z = 0.0f, po = 0.0f;
  const uint32_t epoch0 = d.team_epoch[P];
  uint32_t epoch = epoch0;

  // The team's total from the polling warps' sums, in order.
  auto total = [&](const double* s) {
    double v = 0.0;
#pragma unroll
    for (int i = 0; i < kTeamPolls; ++i) v += 32u * i < T.size ? s[i] : 0.0;
    return v;
  };
  bool ok = true;
  // z = M^-1 r, published with the block's r.z and r.r; waits for the
  // team's slots (their sums in s_rz and s_rr) and the z of the block's
  // columns.
  auto exchange_z = [&]() {
    ++epoch;
    z = 0.0f;
#pragma unroll
    for (int b = 0; b < 6; ++b) z += m[b] * __shfl_sync(0xffffffffu, r, b, 8);
    if (own) put_word(z_mine + 6 * gi + a, __float_as_uint(z), epoch);
    double rz = 0.0, rr = 0.0;
    if (warp < nwarp) {
      rz = warp_sum((double)r * (double)z);
      rr = warp_sum((double)r * (double)r);
      if (lane == 0) {
        s_a[warp] = rz;
        s_b[warp] = rr;
      }
    }
    if (nwarp > 1) __syncthreads();
    if (warp == 0) {
      for (uint32_t w = 1; w < nwarp; ++w) {
        rz += s_a[w];
        rr += s_b[w];
      }
      if (lane < 4u) {
        const double s = lane < 2u ? rz : rr;
        put_word(rz_slots + kLineWords * T.rank + lane,
                 (uint32_t)((lane & 1u) ? __double2hiint(s) : __double2loint(s)), epoch);
      }
    }
    if (32u * warp < T.size) {
      double sum[2];
      const bool got = gather_slots<2>(rz_slots, T.size, epoch, limit_ns, sum);
      if (lane == 0) {
        s_rz[warp] = sum[0];
        s_rr[warp] = sum[1];
        if (!got) s_fail = 1;
      }
    }
    __syncthreads();
    // A wait that gives up has lasted limit_ns: no thread sets s_fail
    // while another is still on its way here.  One that gives up below is
    // seen at the next check.
    ok = s_fail == 0;
    if (!ok) return;
    // The team's z is there or about to be (each block stored it before its
    // slot): read only now, so that early polls do not crowd the stores.
    for (uint32_t e0 = 2u * tid; e0 < L; e0 += 2u * kInFlight * kTeamThreads) {
      unsigned long long v[kInFlight][2];
      const unsigned long long* w[kInFlight];
#pragma unroll
      for (int i = 0; i < kInFlight; ++i) {
        const uint32_t e = min(e0 + i * 2u * kTeamThreads, L - 2u);
        w[i] = zw + z_at[e / 2u];
        get_words(w[i], v[i][0], v[i][1]);
      }
      Deadline dl{limit_ns};
#pragma unroll
      for (int i = 0; i < kInFlight; ++i) {
        while (!fresh(v[i][0], epoch) || !fresh(v[i][1], epoch)) {
          if (!dl.wait()) {
            s_fail = 1;
            break;
          }
          get_words(w[i], v[i][0], v[i][1]);
        }
        const uint32_t e = e0 + i * 2u * kTeamThreads;
        if (e < L)
          *reinterpret_cast<float2*>(z_in + e) =
              make_float2(__uint_as_float((uint32_t)v[i][0]), __uint_as_float((uint32_t)v[i][1]));
      }
    }
    // Each thread updates the entries of p that it read: the next barrier
    // is the one before the product.
  };

  exchange_z();
  double rz = total(s_rz), rr = total(s_rr);
  const LmParams& lp = d.params[P];
  const double bnorm = sqrt(rr), stop = lp.pcg_relative_tolerance * bnorm;
  // |r| <= stop without the root: on squares; a negative tolerance is never met.
  const double stop2 = stop >= 0.0 ? stop * stop : -1.0;
  const uint32_t cap = lp.max_pcg_iterations;
  uint32_t iters = 0, status = 0;
  // pcg_init (ba.wgsl:420-439): done when |b| = 0 or r.z <= 0.
  if (ok && rr > 0.0 && rz > 0.0 && cap != 0u) {
    float beta = 0.0f;
    for (;;) {
      const double inv_rz = 1.0 / rz;  // for beta, off the chain of the sums
      for (uint32_t e = 2u * tid; e < L; e += 2u * kTeamThreads) {
        const float2 zv = *reinterpret_cast<const float2*>(z_in + e);
        float2 pv = *reinterpret_cast<const float2*>(p + e);
        pv.x = __fmaf_rn(beta, pv.x, zv.x);
        pv.y = __fmaf_rn(beta, pv.y, zv.y);
        *reinterpret_cast<float2*>(p + e) = pv;
      }
      po = __fmaf_rn(beta, po, z);
      __syncthreads();
      // Row sums of a part.
      auto reduce = [&](const float (&acc)[6], uint32_t node, uint32_t seg, bool store) {
        float u, v;
        row_sums(acc, lane, u, v);
        const bool b4 = (lane >> 4) & 1u, b3 = (lane >> 3) & 1u;
        float* out = part + (size_t)seg * 6 * nn + 6 * node + (b4 ? 3 : 0);
        if (store && (lane & 7u) == 0) out[b3 ? 2 : 0] = u;
        if (store && (lane & 15u) == 1) out[1] = v;
      };
      auto madd = [](float4 s, float4 v, float& acc) {
        acc = __fmaf_rn(s.x, v.x, acc);
        acc = __fmaf_rn(s.y, v.y, acc);
        acc = __fmaf_rn(s.z, v.z, acc);
        acc = __fmaf_rn(s.w, v.w, acc);
      };
      const float4* p4 = reinterpret_cast<const float4*>(p);
      // The held parts' products, then their reductions side by side (a
      // part past the last holds zeros and stores nothing).
      float held[kHeld][6];
#pragma unroll
      for (int u = 0; u < kHeld; ++u) {
#pragma unroll
        for (int q = 0; q < 6; ++q) held[u][q] = 0.0f;
#pragma unroll
        for (int j = 0; j < kSegVec; ++j) {
          const float4 pv = p4[seg_held[u] * (kSegment / 4) + lane + 32 * j];
#pragma unroll
          for (int q = 0; q < 6; ++q) madd(Sr[u][q][j], pv, held[u][q]);
        }
      }
#pragma unroll
      for (int u = 0; u < kHeld; ++u)
        reduce(held[u], node_held[u], seg_held[u], warp + u * kTeamWarps < parts);
      for (uint32_t it = kRegParts + warp; it < parts; it += kTeamWarps) {
        const uint32_t node = it % nn, seg = it / nn;
        const float4* s4 = reinterpret_cast<const float4*>(S + (size_t)(it - kRegParts) * kPartFloats);
        float acc[6] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 1
        for (int j = 0; j < kSegVec; ++j) {
          const float4 pv = p4[seg * (kSegment / 4) + lane + 32 * j];
#pragma unroll
          for (int q = 0; q < 6; ++q) madd(s4[q * (kSegment / 4) + lane + 32 * j], pv, acc[q]);
        }
        reduce(acc, node, seg, true);
      }
      __syncthreads();
      float qa = 0.0f;
      if (own)
        for (uint32_t s = 0; s < nseg; ++s) qa += part[(size_t)s * 6 * nn + 6 * gi + a];
      ++epoch;
      double pq_own = 0.0;
      if (warp < nwarp) {
        pq_own = warp_sum((double)po * (double)qa);
        if (lane == 0) s_a[warp] = pq_own;
      }
      if (nwarp > 1) __syncthreads();
      if (warp == 0) {
        for (uint32_t w = 1; w < nwarp; ++w) pq_own += s_a[w];
        if (lane < 2u)
          put_word(pq_slots + kLineWords * T.rank + lane,
                   (uint32_t)(lane ? __double2hiint(pq_own) : __double2loint(pq_own)), epoch);
      }
      if (32u * warp < T.size) {
        double sum[1];
        const bool got = gather_slots<1>(pq_slots, T.size, epoch, limit_ns, sum);
        if (lane == 0) {
          s_pq[warp] = sum[0];
          if (!got) s_fail = 1;
        }
      }
      __syncthreads();
      const double pq = total(s_pq);
      ok = s_fail == 0;
      if (!ok) break;
      if (!(pq > 0.0) || !isfinite(pq)) {
        status = 2;  // non-positive curvature: x unchanged
        break;
      }
      const float alpha = (float)(rz / pq);
      x = x + alpha * po;
      r = r - alpha * qa;
      exchange_z();
      if (!ok) break;
      const double rz_new = total(s_rz);
      rr = total(s_rr);
      ++iters;
      rz = rz_new;
      if (rr <= stop2 || !(rz_new > 0.0)) break;
      if (iters >= cap) {
        status = 1;
        break;
      }
      beta = (float)(rz_new * inv_rz);
    }
  }
  if (own) d.x[at] = x;
  if (T.rank == 0 && tid == 0) {
    PcgState& st = d.pcg[P];
    st.iters = iters;
    st.status = status;
    st.bnorm = bnorm;
    st.rnorm = sqrt(rr);
    st.rz = rz;
    st.active = 0u;
    // Every block has read epoch0: this one has seen all their slots.  (A
    // block that gave up is at most one exchange ahead of another.)
    d.team_epoch[P] = epoch + 2u;
  }
  __syncthreads();
  if (s_fail && tid == 0) atomicOr(d.error, (unsigned int)kErrBarrierTimeout);
}

uint32_t team_parts(uint32_t nodes, uint32_t ncols) {
  return nodes * ((ncols + kSegTiles - 1) / kSegTiles);
}
size_t team_smem(uint32_t nodes, uint32_t ncols) {
  const uint32_t parts = team_parts(nodes, ncols), nseg = parts / nodes;
  const uint32_t staged = std::max(std::min(parts, kRegParts), parts > kRegParts ? parts - kRegParts : 0u);
  return 4 * ((size_t)staged * kPartFloats + 2 * (size_t)nseg * kSegment + (size_t)nseg * 6 * nodes +
              24 * (size_t)ncols);
}

}  // namespace

namespace {
// The tile columns of each tile row (both triangles), a bit each.
struct Near {
  uint32_t rows, words;
  std::vector<uint64_t> bits;
  explicit Near(uint32_t r) : rows(r), words((r + 63) / 64), bits((size_t)r * words) {}
  void set(uint32_t i, uint32_t j) { bits[(size_t)i * words + j / 64] |= 1ull << (j % 64); }
};
}  // namespace

// Blocks of one problem for a team of `size`, whose largest needs *smem bytes;
// false when a block would own or read too many cameras, have more than
// `most` parts or not fit its shared memory.
static bool split_team(const Near& near, uint32_t size, uint32_t most, std::vector<TeamCta>* out,
                       std::vector<uint32_t>* cols, size_t* smem) {
  const uint32_t nodes = 8 * near.rows;
  std::vector<uint64_t> u(near.words);
  for (uint32_t g = 0; g < size; ++g) {
    TeamCta T{};
    T.rank = g;
    T.size = size;
    T.node0 = (uint32_t)((uint64_t)nodes * g / size);
    T.node1 = (uint32_t)((uint64_t)nodes * (g + 1) / size);
    if (T.node1 == T.node0 || T.node1 - T.node0 > kTeamMaxNodes) return false;
    std::fill(u.begin(), u.end(), 0ull);
    for (uint32_t I = T.node0 / 8; I <= (T.node1 - 1) / 8; ++I)
      for (uint32_t w = 0; w < near.words; ++w) u[w] |= near.bits[(size_t)I * near.words + w];
    for (uint64_t w : u) T.ncols += (uint32_t)__builtin_popcountll(w);
    if (T.ncols > kTeamMaxCols || team_parts(T.node1 - T.node0, T.ncols) > most) return false;
    const size_t bytes = team_smem(T.node1 - T.node0, T.ncols);
    if (bytes > kTeamMaxSmem) return false;
    *smem = std::max(*smem, bytes);
    if (!out) continue;
    T.col_begin = (uint32_t)cols->size();
    for (uint32_t w = 0; w < near.words; ++w)
      for (uint64_t b = u[w]; b; b &= b - 1) cols->push_back(64 * w + (uint32_t)__builtin_ctzll(b));
    out->push_back(T);
  }
  return true;
}

TeamPlan build_team_plan(const uint32_t* prob_tr_begin, uint32_t num_problems,
                         const std::vector<uint32_t>& tile_ij,
                         const std::vector<uint32_t>& tile_begin, uint32_t small_rows,
                         uint32_t max_blocks) {
  TeamPlan tp;
  tp.in_team.assign(num_problems, 0);
  max_blocks = std::min(max_blocks, kTeamBlocks);
  struct Team {
    uint32_t first, size;
  };
  std::vector<Team> teams;
  for (uint32_t p = 0; p < num_problems; ++p) {
    const uint32_t tr0 = prob_tr_begin[p], R = prob_tr_begin[p + 1] - tr0;
    if (R <= small_rows) continue;
    const uint32_t most = kRegParts + kExtra;
    const uint64_t tiles = tile_begin[p + 1] - tile_begin[p];
    // What cannot fit: the parts or the cameras of all blocks.
    if ((2 * tiles - R) * 8 / kSegTiles > (uint64_t)max_blocks * most ||
        8 * (uint64_t)R > (uint64_t)max_blocks * kTeamMaxNodes)
      continue;
    Near near(R);
    for (uint32_t t = tile_begin[p]; t < tile_begin[p + 1]; ++t) {
      const uint32_t I = (tile_ij[t] >> 16) - tr0, J = (tile_ij[t] & 0xFFFFu) - tr0;
      near.set(I, J);
      near.set(J, I);
    }
    uint32_t size = 0;
    for (uint32_t s : {16u, 24u, 32u, 48u, 64u, 80u, 96u, 112u, 128u, 148u}) {
      s = std::min(s, max_blocks);
      size_t bytes = 0;
      if (split_team(near, s, s == max_blocks ? most : kRegParts, nullptr, nullptr, &bytes)) size = s;
      if (size || s == max_blocks) break;
    }
    if (!size) continue;
    const uint32_t first = (uint32_t)tp.cta.size();
    split_team(near, size, most, &tp.cta, &tp.cols, &tp.smem);
    // The tile of each (tile row, column) the block reads.
    std::vector<uint32_t> id((size_t)R * R, kNone);
    for (uint32_t t = tile_begin[p]; t < tile_begin[p + 1]; ++t) {
      const uint32_t I = (tile_ij[t] >> 16) - tr0, J = (tile_ij[t] & 0xFFFFu) - tr0;
      id[(size_t)I * R + J] = id[(size_t)J * R + I] = t;
    }
    const uint64_t team_words = tp.z_words;
    uint32_t own_words = 0;
    for (uint32_t c = first; c < tp.cta.size(); ++c) {
      TeamCta& T = tp.cta[c];
      T.prob = p;
      T.slot_base = first;
      T.z_team = team_words;
      T.z_own = own_words;
      own_words += (6 * (T.node1 - T.node0) + kLineWords - 1) / kLineWords * kLineWords;
      T.ent_begin = (uint32_t)tp.ents.size();
      const uint32_t I0 = T.node0 / 8, I1 = (T.node1 - 1) / 8 + 1;
      tp.ents.resize(tp.ents.size() + (size_t)(I1 - I0) * T.ncols);
      uint32_t* e = tp.ents.data() + T.ent_begin;
      for (uint32_t I = I0; I < I1; ++I)
        for (uint32_t k = 0; k < T.ncols; ++k) *e++ = id[(size_t)I * R + tp.cols[T.col_begin + k]];
    }
    tp.z_words += own_words;
    tp.in_team[p] = 1;
    teams.push_back(Team{first, size});
  }
  // Rounds of teams that fit the device together, in problem order.
  uint32_t used = 0;
  for (const Team& t : teams) {
    if (tp.round_begin.empty() || used + t.size > max_blocks) {
      tp.round_begin.push_back(t.first);
      used = 0;
    }
    used += t.size;
  }
  if (!teams.empty()) tp.round_begin.push_back((uint32_t)tp.cta.size());
  return tp;
}

static cudaError_t launch_round(const Dev& d, uint32_t round, uint32_t absent,
                                unsigned long long limit_ns, cudaStream_t s) {
  const cudaError_t e = cudaFuncSetAttribute(
      k_pcg_team, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTeamMaxSmem);
  if (e != cudaSuccess) return e;
  uint32_t first = d.team_round_begin[round];
  void* args[] = {const_cast<Dev*>(&d), &first, &absent, &limit_ns};
  return cudaLaunchCooperativeKernel((const void*)k_pcg_team, d.team_round_begin[round + 1] - first,
                                     kTeamThreads, args, d.team_smem, s);
}

cudaError_t launch_pcg_team(const Dev& d, cudaStream_t s) {
  // A launch a round: in one launch over all of them a block waited for the
  // teammates of its next round while they still solved the last one, as long
  // as that solve took, under the limit of a wait.
  cudaError_t e = cudaSuccess;
  for (uint32_t r = 0; r < d.team_rounds && e == cudaSuccess; ++r)
    e = launch_round(d, r, kNone, kWaitLimitNs, s);
  return e;
}

cudaError_t launch_team_probe(const Dev& d, unsigned long long limit_ns, cudaStream_t s) {
  return launch_round(d, 0, 0u, limit_ns, s);
}

cudaError_t clear_team_words(const Dev& d, cudaStream_t s) {
  if (d.team_rounds == 0) return cudaSuccess;
  // The slots follow the z words.
  const size_t words = (size_t)(d.team_slots - d.team_z) + 2 * kLineWords * (size_t)d.team_slots_total;
  const cudaError_t e = cudaMemsetAsync(d.team_z, 0, 8 * words, s);
  return e != cudaSuccess ? e : cudaMemsetAsync(d.team_epoch, 0, 4 * (size_t)d.num_problems, s);
}

}  // namespace vlba
