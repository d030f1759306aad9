// project.cu -- project! for Stabilizer, MixedStabilizer, Destabilizer and
// MixedDestabilizer tableaux (src/project_trace_reset.jl:231-439).
//
// Runs of 32 Paulis and more go by panels over the whole GPU (below).  Else
// one thread-block cluster projects a list of Paulis in order on one state.
// The tableau stays in global memory (it is L2 resident at these sizes).  Per
// Pauli:
//   1. every CTA computes comm(pauli, row) for its share of the rows (warp per
//      row, parity of popcounts) into a flag array, and the first
//      anticommuting row of each range the reference scans;
//   2. after a cluster barrier every CTA reads all CTAs' minima through
//      distributed shared memory, so all take the same branch;
//   3. the row swaps of the MixedDestabilizer logical branch are done by CTA 0
//      (flags swapped with the rows), then every CTA left-multiplies its
//      anticommuting rows by the pivot row exactly as anticomm_update_rows
//      (:319-335) does (comm is evaluated on the rows before any update, and
//      the pivot row is never updated, so the row updates are independent);
//   4. CTA 0 does the row copies, rank update and the result.
// The commuting branch of Stabilizer / MixedStabilizer needs canonicalize! +
// generate!; the kernel stops there and the host runs those kernels before
// resuming with the next Pauli.
#include <cooperative_groups.h>

#include <algorithm>
#include <memory>

#include "panel.cuh"
#include "qcb_internal.h"

namespace cg = cooperative_groups;

namespace qcb {

int canonicalize_view(uint64_t* xzs, uint8_t* ph, uint32_t rows, uint32_t n, uint32_t W, int phases,
                      int32_t* d_out, cudaStream_t st, bool waits);
int generate_dev(uint64_t* pauli, uint8_t* pph, const uint64_t* xzs, const uint8_t* ph, uint32_t rows,
                 uint32_t W, int phases, int32_t* d_ok, int32_t* d_used, uint32_t cap, uint32_t* d_nused,
                 cudaStream_t st);

__device__ __forceinline__ void mul_step_p(uint64_t x1, uint64_t z1, uint64_t& x2, uint64_t& z2,
                                           uint64_t& c1, uint64_t& c2) {
  const uint64_t nx = x1 ^ x2, nz = z1 ^ z2;
  const uint64_t x1z2 = x1 & z2;
  const uint64_t anti = (x2 & z1) ^ x1z2;
  c2 ^= (c1 ^ nx ^ nz ^ x1z2) & anti;
  c1 ^= anti;
  x2 = nx;
  z2 = nz;
}

enum : int32_t { PST_OK = 0, PST_NEED_CANON = 1, PST_BADSTRUCT = 2 };

struct ProjArgs {
  uint64_t* xzs;
  uint8_t* ph;
  uint32_t rows, n, W;
  int kind;
  int32_t* rank;         // device rank (mixed kinds)
  const uint64_t* paulis;
  const uint8_t* pph;
  uint32_t j0, k;        // project Paulis [j0, k)
  int keep_result, phases;
  int32_t* anticom;
  int32_t* result;
  int32_t* status;       // [0] = status, [1] = index reached
  uint8_t* flags;        // rows
  const uint32_t* qubits;  // projectX!/Y!/Z!: Pauli j is the single-qubit Pauli on qubits[j] (0-based), or null
  uint32_t basis;          // with qubits: bit 0 = X component, bit 1 = Z component
  const uint8_t* rand_ph;  // projectrand!: phase (0 or 2) given to the new stabilizer row of Pauli j, or null
  // a trial by panels from j0 on, launched before: [0] ended, [1] the next
  // Pauli; unless it ended within PROJ_PANEL_SHORT Paulis this launch does
  // nothing (null: always)
  const int32_t* trial;
};

constexpr uint32_t PROJ_THREADS = 1024;

// Steps of a run's first panel that are not worth the launches which bring the
// rows up to date (about 30 us, 3 to 5 us a Pauli by the other kernels).
constexpr uint32_t PROJ_PANEL_SHORT = 8;
__host__ __device__ inline bool short_trial(const int32_t* state, uint32_t j0) {
  return state[0] && (uint32_t)state[1] - j0 < PROJ_PANEL_SHORT;
}

// row m <- row i * row m (mul_left!(tab, m, i)), warp-cooperative.
__device__ __forceinline__ void warp_rowmul(uint64_t* xzs, uint8_t* ph, uint32_t W, uint32_t m,
                                            const uint64_t* piv, uint32_t pph, bool phases,
                                            uint32_t lane) {
  const uint32_t len = W / 2;
  uint64_t* row = xzs + (size_t)m * W;
  uint64_t c1 = 0, c2 = 0;
  for (uint32_t w = lane; w < len; w += 32) {
    uint64_t x2 = row[w], z2 = row[len + w];
    mul_step_p(piv[w], piv[len + w], x2, z2, c1, c2);
    row[w] = x2;
    row[len + w] = z2;
  }
  if (phases) {
    const uint32_t s =
        __reduce_add_sync(0xFFFFFFFFu, (uint32_t)(__popcll(c1) + 2 * __popcll(c2)) & 3u) & 3u;
    if (lane == 0) ph[m] = (uint8_t)((s + ph[m] + pph) & 3u);
  }
}

__global__ void __launch_bounds__(PROJ_THREADS) project_kernel(const ProjArgs a) {
  if (a.trial && !short_trial(a.trial, a.j0)) return;
  cg::cluster_group cl = cg::this_cluster();
  const uint32_t me = cl.block_rank(), CS = cl.num_blocks();
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
  const uint32_t gw = me * nwarps + warp, NW = CS * nwarps;
  const uint32_t W = a.W, len = W / 2;
  extern __shared__ __align__(16) uint64_t smem[];
  uint64_t* P = smem;            // W words: the Pauli
  uint64_t* piv = smem + W;      // W words: the pivot row
  __shared__ uint32_t mins[3];   // first anticommuting: stab range, logical X, logical Z
  __shared__ int32_t dec[8];     // decision broadcast

  const uint32_t rows = a.rows;
  for (uint32_t j = a.j0; j < a.k; j++) {
    const bool single = a.qubits != nullptr;
    uint32_t wq = 0;
    uint64_t bq = 0;
    if (single) {
      wq = a.qubits[j] >> 6;
      bq = 1ull << (a.qubits[j] & 63);
      for (uint32_t w = tid; w < W; w += blockDim.x)
        P[w] = (((a.basis & 1u) && w == wq) ? bq : 0ull) | (((a.basis & 2u) && w == len + wq) ? bq : 0ull);
    } else {
      const uint64_t* pj = a.paulis + (size_t)j * W;
      for (uint32_t w = tid; w < W; w += blockDim.x) P[w] = pj[w];
    }
    if (tid < 3) mins[tid] = 0xFFFFFFFFu;
    const uint32_t pphase = single ? 0u : a.pph[j];
    int32_t r = a.kind == QCB_STABILIZER ? (int32_t)rows : (a.kind == QCB_DESTABILIZER ? (int32_t)(rows / 2) : *a.rank);
    __syncthreads();
    const uint32_t nn = (a.kind == QCB_DESTABILIZER || a.kind == QCB_MIXED_DESTABILIZER) ? rows / 2 : rows;
    // 1. comm flags for every row and the first anticommuting rows
    auto note = [&](uint32_t m, uint32_t c) {
      a.flags[m] = (uint8_t)c;
      if (c) {
        if (a.kind == QCB_STABILIZER || a.kind == QCB_MIXED_STABILIZER) {
          if (m < (uint32_t)r) atomicMin(&mins[0], m);
        } else {
          if (m >= nn && m < nn + (uint32_t)r) atomicMin(&mins[0], m - nn);
          if (a.kind == QCB_MIXED_DESTABILIZER) {
            if (m >= (uint32_t)r && m < nn) atomicMin(&mins[1], m);
            if (m >= nn + (uint32_t)r) atomicMin(&mins[2], m);
          }
        }
      }
    };
    if (single) {
      // comm with a single-qubit Pauli is one bit of the row (the isX / isZ /
      // isXorZ tests of project_cond!, src/project_trace_reset.jl:476-479)
      for (uint32_t m = me * blockDim.x + tid; m < rows; m += CS * blockDim.x) {
        const uint64_t* row = a.xzs + (size_t)m * W;
        uint32_t c = 0;
        if (a.basis & 1u) c ^= (uint32_t)((row[len + wq] & bq) != 0);
        if (a.basis & 2u) c ^= (uint32_t)((row[wq] & bq) != 0);
        note(m, c);
      }
    } else {
      for (uint32_t m = gw; m < rows; m += NW) {
        const uint64_t* row = a.xzs + (size_t)m * W;
        uint64_t acc = 0;
        for (uint32_t w = lane; w < len; w += 32) acc ^= (P[len + w] & row[w]) ^ (P[w] & row[len + w]);
        const uint32_t c = __reduce_add_sync(0xFFFFFFFFu, (uint32_t)__popcll(acc)) & 1u;
        if (lane == 0) note(m, c);
      }
    }
    __syncthreads();
    cl.sync();
    // 2. uniform decision
    if (tid == 0) {
      uint32_t m0 = 0xFFFFFFFFu, m1 = 0xFFFFFFFFu, m2 = 0xFFFFFFFFu;
      for (uint32_t q = 0; q < CS; q++) {
        uint32_t* rm = cl.map_shared_rank(mins, q);
        m0 = min(m0, rm[0]); m1 = min(m1, rm[1]); m2 = min(m2, rm[2]);
      }
      // dec: [0] branch, [1] pivot row, [2] anticom (1-based), [3] update r, [4] update anticommutes
      int32_t branch = 0, pivrow = -1, anticom = 0;
      if (m0 != 0xFFFFFFFFu) {
        branch = 1;  // anticommutes with a stabilizer row
        anticom = (int32_t)m0 + 1;
      } else if (a.kind == QCB_MIXED_DESTABILIZER && (m1 != 0xFFFFFFFFu || m2 != 0xFFFFFFFFu)) {
        branch = 2;  // anticommutes with a logical operator
        anticom = (int32_t)(m1 != 0xFFFFFFFFu ? m1 : m2) + 1;  // 1-based anticomlog
      } else {
        branch = 0;
      }
      if (branch == 1) {
        pivrow = (a.kind == QCB_STABILIZER || a.kind == QCB_MIXED_STABILIZER) ? anticom - 1 : (int32_t)nn + anticom - 1;
      } else if (branch == 2) {
        pivrow = (int32_t)nn + r;  // row n+r+1 (1-based) after the swaps
      }
      dec[0] = branch; dec[1] = pivrow; dec[2] = anticom;
    }
    __syncthreads();
    const int32_t branch = dec[0];
    if (branch == 0) {
      // commutes with every stabilizer row
      bool stop = false;
      if (a.kind == QCB_STABILIZER || a.kind == QCB_MIXED_STABILIZER) {
        if (a.keep_result || a.kind == QCB_MIXED_STABILIZER) stop = true;
        else if (me == 0 && tid == 0) { a.anticom[j] = 0; a.result[j] = -1; }
      } else if (a.kind == QCB_DESTABILIZER && nn != a.n) {
        if (me == 0 && tid == 0) { a.status[0] = PST_BADSTRUCT; a.status[1] = (int32_t)j; }
        cl.sync();
        return;
      } else if (me == 0 && warp == 0) {
        int32_t res = -1;
        if (a.keep_result) {
          // new_pauli = product of the stabilizer rows whose destabilizer
          // anticommutes with the Pauli, phase starting from the Pauli's
          uint64_t c1 = 0, c2 = 0;
          uint32_t extra = pphase;
          uint64_t* buf = piv;  // the pivot buffer is free in this branch
          for (uint32_t w = lane; w < W; w += 32) buf[w] = 0;
          __syncwarp();
          for (uint32_t i = 0; i < (uint32_t)r; i++) {
            if (!a.flags[i]) continue;  // comm(pauli, destabilizer row i)
            const uint64_t* srow = a.xzs + (size_t)(nn + i) * W;
            for (uint32_t w = lane; w < len; w += 32) {
              uint64_t x2 = buf[w], z2 = buf[len + w];
              mul_step_p(srow[w], srow[len + w], x2, z2, c1, c2);
              buf[w] = x2;
              buf[len + w] = z2;
            }
            __syncwarp();
            extra += a.ph[nn + i];
          }
          const uint32_t s =
              __reduce_add_sync(0xFFFFFFFFu, (uint32_t)(__popcll(c1) + 2 * __popcll(c2)) & 3u) & 3u;
          res = a.phases ? (int32_t)((s + extra) & 3u) : (int32_t)(pphase & 3u);
        }
        if (lane == 0) { a.anticom[j] = 0; a.result[j] = res; }
      }
      if (stop) {
        if (me == 0 && tid == 0) { a.status[0] = PST_NEED_CANON; a.status[1] = (int32_t)j; }
        cl.sync();
        return;
      }
      cl.sync();
      continue;
    }
    // 3. swaps (MixedDestabilizer logical branch), done by CTA 0
    if (branch == 2) {
      if (me == 0) {
        const uint32_t al = (uint32_t)dec[2];  // 1-based anticomlog
        auto swaprow = [&](uint32_t u, uint32_t v) {  // 0-based
          if (u == v) return;
          uint64_t* ru = a.xzs + (size_t)u * W;
          uint64_t* rv = a.xzs + (size_t)v * W;
          for (uint32_t w = tid; w < W; w += blockDim.x) { uint64_t t = ru[w]; ru[w] = rv[w]; rv[w] = t; }
          if (tid == 0) {
            uint8_t t = a.ph[u]; a.ph[u] = a.ph[v]; a.ph[v] = t;
            uint8_t f = a.flags[u]; a.flags[u] = a.flags[v]; a.flags[v] = f;
          }
          __syncthreads();
        };
        const uint32_t ru = (uint32_t)r;
        if (al <= nn) {
          swaprow(ru + nn, al - 1);
          if (nn != ru + 1 && al != ru + 1) swaprow(ru, al + nn - 1);
        } else {
          swaprow(ru, al - nn - 1);
          swaprow(ru + nn, al - 1);
        }
      }
      cl.sync();
    }
    // 4. row updates (anticomm_update_rows or the Stabilizer loop)
    const uint32_t pivrow = (uint32_t)dec[1];
    for (uint32_t w = tid; w < W; w += blockDim.x) piv[w] = a.xzs[(size_t)pivrow * W + w];
    __syncthreads();
    const uint32_t pph = a.ph[pivrow];
    if (a.kind == QCB_STABILIZER || a.kind == QCB_MIXED_STABILIZER) {
      const uint32_t ac = (uint32_t)dec[2];
      for (uint32_t m = ac + gw; m < (uint32_t)r; m += NW)
        if (a.flags[m]) warp_rowmul(a.xzs, a.ph, W, m, piv, pph, a.phases != 0, lane);
    } else {
      const uint32_t ru = branch == 2 ? (uint32_t)r + 1 : (uint32_t)r;
      const uint32_t ac = branch == 2 ? (uint32_t)r + 1 : (uint32_t)dec[2];
      for (uint32_t m = gw; m < 2 * nn; m += NW) {
        if (!a.flags[m] || m == pivrow) continue;
        if (m >= ru && m < nn) warp_rowmul(a.xzs, a.ph, W, m, piv, pph, a.phases != 0, lane);
        else if (m >= nn + ac && m < 2 * nn) warp_rowmul(a.xzs, a.ph, W, m, piv, pph, a.phases != 0, lane);
        else if (m < ru && m != ac - 1) warp_rowmul(a.xzs, a.ph, W, m, piv, pph, false, lane);
      }
    }
    cl.sync();
    // 5. row copies, rank, outputs (CTA 0)
    if (me == 0) {
      if (a.kind == QCB_STABILIZER || a.kind == QCB_MIXED_STABILIZER) {
        const uint32_t ac = (uint32_t)dec[2];
        for (uint32_t w = tid; w < W; w += blockDim.x) a.xzs[(size_t)(ac - 1) * W + w] = P[w];
        if (tid == 0) {
          // projectrand!: the undetermined outcome gets a random sign
          const int32_t rp = a.rand_ph ? (int32_t)a.rand_ph[j] : -1;
          a.ph[ac - 1] = (uint8_t)(rp >= 0 ? rp : (int32_t)pphase);
          a.anticom[j] = (int32_t)ac;
          a.result[j] = rp;
        }
      } else {
        const uint32_t ac = branch == 2 ? (uint32_t)r + 1 : (uint32_t)dec[2];
        // destabilizer[ac] = stabilizer[ac]; stabilizer[ac] = pauli
        for (uint32_t w = tid; w < W; w += blockDim.x) {
          a.xzs[(size_t)(ac - 1) * W + w] = a.xzs[(size_t)(nn + ac - 1) * W + w];
        }
        __syncthreads();
        for (uint32_t w = tid; w < W; w += blockDim.x) a.xzs[(size_t)(nn + ac - 1) * W + w] = P[w];
        if (tid == 0) {
          const int32_t rp = a.rand_ph ? (int32_t)a.rand_ph[j] : -1;
          a.ph[ac - 1] = a.ph[nn + ac - 1];
          a.ph[nn + ac - 1] = (uint8_t)(rp >= 0 ? rp : (int32_t)pphase);
          if (branch == 2) *a.rank = r + 1;
          a.anticom[j] = (int32_t)(branch == 2 ? r + 1 : (int32_t)ac);
          a.result[j] = rp;
        }
      }
    }
    cl.sync();
  }
  if (me == 0 && tid == 0) { a.status[0] = PST_OK; a.status[1] = (int32_t)a.k; }
}

// ---------------------------------------------------------------------------
// project_smem_kernel: the same projections with the whole tableau held in
// the cluster's shared memory (CTA c owns rows [c*RB, c*RB + RB), row stride
// W+1 words).  Per Pauli there are two cluster barriers: one after every CTA
// has published the first anticommuting row of each range it owns (every CTA
// then reads all of them through distributed shared memory and takes the
// same decision), one after every CTA has fetched the pivot row.  The row
// products then run on local rows only, and the row copies are done by the
// rows' owners from their local copies of the pivot and the Pauli (neither
// row is among the updated ones).  Rows are read from and written back to
// global memory once per launch.
struct ProjSmemArgs {
  ProjArgs a;
  uint32_t RB;
};

// Lanes per row: the smallest power of two >= the words of one half, at most 32.
__device__ __forceinline__ uint32_t group_lanes(uint32_t len) {
  uint32_t g = 1;
  while (g < len && g < 32) g <<= 1;
  return g;
}

__global__ void __launch_bounds__(PROJ_THREADS) project_smem_kernel(const ProjSmemArgs pa) {
  const ProjArgs& a = pa.a;
  if (a.trial && !short_trial(a.trial, a.j0)) return;
  cg::cluster_group cl = cg::this_cluster();
  const uint32_t me = cl.block_rank(), CS = cl.num_blocks();
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
  const uint32_t W = a.W, len = W / 2, WS = W + 1, RB = pa.RB;
  const uint32_t rows = a.rows;
  const uint32_t r0 = me * RB;
  const uint32_t nloc = r0 < rows ? min(RB, rows - r0) : 0u;
  const uint32_t G = group_lanes(len), GPW = 32 / G;  // lanes per row, rows per warp pass
  const uint32_t gl = lane % G, gi = lane / G;

  extern __shared__ __align__(16) uint64_t smem[];
  uint64_t* P = smem;                       // W: the Pauli
  uint64_t* piv = P + W;                    // W: the pivot row / partial product
  uint64_t* R = piv + W + 1;                // RB * WS: the rows
  uint8_t* ph = (uint8_t*)(R + (size_t)RB * WS);  // RB
  uint8_t* fl = ph + RB;                    // RB: comm flags
  uint32_t* slot = (uint32_t*)(((uintptr_t)(fl + RB) + 15) & ~(uintptr_t)15);  // [2][4]
  uint32_t* mins = slot + 8;                // 3
  int32_t* dec = (int32_t*)(mins + 4);      // 8

  auto ROW = [&](uint32_t lr) -> uint64_t* { return R + (size_t)lr * WS; };
  // (owner CTA, local row) of a global row
  auto owner_of = [&](uint32_t m) -> uint32_t { return m / RB; };

  for (uint32_t lr = warp; lr < nloc; lr += nwarps)
    for (uint32_t w = lane; w < W; w += 32) ROW(lr)[w] = a.xzs[(size_t)(r0 + lr) * W + w];
  for (uint32_t lr = tid; lr < nloc; lr += blockDim.x) ph[lr] = a.ph[r0 + lr];
  const bool destab = a.kind == QCB_DESTABILIZER || a.kind == QCB_MIXED_DESTABILIZER;
  const uint32_t nn = destab ? rows / 2 : rows;
  int32_t r = a.kind == QCB_STABILIZER ? (int32_t)rows : (a.kind == QCB_DESTABILIZER ? (int32_t)(rows / 2) : *a.rank);
  __syncthreads();
  cl.sync();

  uint32_t status = PST_OK, jstop = a.k;
  for (uint32_t j = a.j0; j < a.k; j++) {
    const uint32_t par = j & 1;
    const bool single = a.qubits != nullptr;
    uint32_t wq = 0;
    uint64_t bq = 0;
    if (single) {
      wq = a.qubits[j] >> 6;
      bq = 1ull << (a.qubits[j] & 63);
      for (uint32_t w = tid; w < W; w += blockDim.x)
        P[w] = (((a.basis & 1u) && w == wq) ? bq : 0ull) | (((a.basis & 2u) && w == len + wq) ? bq : 0ull);
    } else {
      const uint64_t* pj = a.paulis + (size_t)j * W;
      for (uint32_t w = tid; w < W; w += blockDim.x) P[w] = pj[w];
    }
    if (tid < 3) mins[tid] = 0xFFFFFFFFu;
    const uint32_t pphase = single ? 0u : a.pph[j];
    __syncthreads();
    // 1. comm flags of the local rows and the first anticommuting row of each range
    auto note = [&](uint32_t m, uint32_t c) {
      if (!c) return;
      if (!destab) {
        if (m < (uint32_t)r) atomicMin(&mins[0], m);
      } else {
        if (m >= nn && m < nn + (uint32_t)r) atomicMin(&mins[0], m - nn);
        if (a.kind == QCB_MIXED_DESTABILIZER) {
          if (m >= (uint32_t)r && m < nn) atomicMin(&mins[1], m);
          if (m >= nn + (uint32_t)r) atomicMin(&mins[2], m);
        }
      }
    };
    if (single) {
      for (uint32_t lr = tid; lr < nloc; lr += blockDim.x) {
        const uint64_t* row = ROW(lr);
        uint32_t c = 0;
        if (a.basis & 1u) c ^= (uint32_t)((row[len + wq] & bq) != 0);
        if (a.basis & 2u) c ^= (uint32_t)((row[wq] & bq) != 0);
        fl[lr] = (uint8_t)c;
        note(r0 + lr, c);
      }
    } else {
      for (uint32_t base = warp * GPW; base < nloc; base += nwarps * GPW) {
        const uint32_t lr = base + gi;
        uint64_t acc = 0;
        if (lr < nloc) {
          const uint64_t* row = ROW(lr);
          for (uint32_t w = gl; w < len; w += G) acc ^= (P[len + w] & row[w]) ^ (P[w] & row[len + w]);
        }
        uint32_t c = (uint32_t)__popcll(acc);
        for (uint32_t off = G >> 1; off; off >>= 1) c += __shfl_xor_sync(0xFFFFFFFFu, c, off);
        c &= 1u;
        if (gl == 0 && lr < nloc) {
          fl[lr] = (uint8_t)c;
          note(r0 + lr, c);
        }
      }
    }
    __syncthreads();
    if (tid < 3) slot[par * 4 + tid] = mins[tid];
    cl.sync();
    // 2. the same decision in every CTA
    if (warp == 0) {
      uint32_t m0 = 0xFFFFFFFFu, m1 = 0xFFFFFFFFu, m2 = 0xFFFFFFFFu;
      if (lane < CS) {
        const uint32_t* rs = cl.map_shared_rank(slot + par * 4, lane);
        m0 = rs[0]; m1 = rs[1]; m2 = rs[2];
      }
      m0 = __reduce_min_sync(0xFFFFFFFFu, m0);
      m1 = __reduce_min_sync(0xFFFFFFFFu, m1);
      m2 = __reduce_min_sync(0xFFFFFFFFu, m2);
      if (lane == 0) {
        int32_t branch = 0, pivrow = -1, anticom = 0;
        if (m0 != 0xFFFFFFFFu) {
          branch = 1;
          anticom = (int32_t)m0 + 1;
          pivrow = destab ? (int32_t)nn + anticom - 1 : anticom - 1;
        } else if (a.kind == QCB_MIXED_DESTABILIZER && (m1 != 0xFFFFFFFFu || m2 != 0xFFFFFFFFu)) {
          branch = 2;
          anticom = (int32_t)(m1 != 0xFFFFFFFFu ? m1 : m2) + 1;  // 1-based anticomlog
          pivrow = (int32_t)nn + r;
        }
        dec[0] = branch; dec[1] = pivrow; dec[2] = anticom;
      }
    }
    __syncthreads();
    const int32_t branch = dec[0];
    if (branch == 0) {
      if (!destab) {
        if (a.keep_result || a.kind == QCB_MIXED_STABILIZER) { status = PST_NEED_CANON; jstop = j; break; }
        if (me == 0 && tid == 0) { a.anticom[j] = 0; a.result[j] = -1; }
        continue;
      }
      if (a.kind == QCB_DESTABILIZER && nn != a.n) { status = PST_BADSTRUCT; jstop = j; break; }
      if (!a.keep_result) {
        if (me == 0 && tid == 0) { a.anticom[j] = 0; a.result[j] = -1; }
        continue;
      }
      // result: the product of the stabilizer rows i < r whose destabilizer
      // row anticommutes with the Pauli (the stabilizer rows commute, so the
      // per-CTA partial products can be combined in any order with the exact
      // phase).  Warp 0 of each CTA multiplies its own stabilizer rows.
      if (warp == 0) {
        uint64_t c1 = 0, c2 = 0;
        uint32_t extra = 0;
        for (uint32_t w = lane; w < W; w += 32) piv[w] = 0;
        __syncwarp();
        for (uint32_t lr = 0; lr < nloc; lr++) {
          const uint32_t m = r0 + lr;
          if (m < nn || m >= nn + (uint32_t)r) continue;
          const uint32_t i = m - nn;  // destabilizer partner row i
          const uint32_t o = owner_of(i);
          const uint8_t f = o == me ? fl[i - r0] : *cl.map_shared_rank(fl + (i - o * RB), o);
          if (!f) continue;
          const uint64_t* srow = ROW(lr);
          for (uint32_t w = lane; w < len; w += 32) {
            uint64_t x2 = piv[w], z2 = piv[len + w];
            mul_step_p(srow[w], srow[len + w], x2, z2, c1, c2);
            piv[w] = x2;
            piv[len + w] = z2;
          }
          __syncwarp();
          extra += ph[lr];
        }
        const uint32_t s = __reduce_add_sync(0xFFFFFFFFu, (uint32_t)(__popcll(c1) + 2 * __popcll(c2)) & 3u) & 3u;
        if (lane == 0) piv[W] = (uint64_t)((s + extra) & 3u);
      }
      cl.sync();
      if (me == 0 && warp == 0) {
        // combine the CTAs' partial products in CTA order into P's buffer
        uint64_t c1 = 0, c2 = 0;
        uint32_t extra = pphase;
        for (uint32_t w = lane; w < W; w += 32) P[w] = 0;
        __syncwarp();
        for (uint32_t q = 0; q < CS; q++) {
          const uint64_t* pq = q == 0 ? piv : cl.map_shared_rank(piv, q);
          for (uint32_t w = lane; w < len; w += 32) {
            uint64_t x2 = P[w], z2 = P[len + w];
            mul_step_p(pq[w], pq[len + w], x2, z2, c1, c2);
            P[w] = x2;
            P[len + w] = z2;
          }
          __syncwarp();
          extra += (uint32_t)pq[W];
        }
        const uint32_t s = __reduce_add_sync(0xFFFFFFFFu, (uint32_t)(__popcll(c1) + 2 * __popcll(c2)) & 3u) & 3u;
        if (lane == 0) {
          a.anticom[j] = 0;
          a.result[j] = a.phases ? (int32_t)((s + extra) & 3u) : (int32_t)(pphase & 3u);
        }
      }
      // CTA 0's other warps fill P for the next Pauli only now; the other CTAs
      // reuse their partial products after its first cluster barrier, which
      // CTA 0 enters when it has read them
      __syncthreads();
      continue;
    }
    // 3. MixedDestabilizer logical branch: the row swaps (rare), by CTA 0
    //    through distributed shared memory
    if (branch == 2) {
      if (me == 0) {
        const uint32_t al = (uint32_t)dec[2];
        auto swaprow = [&](uint32_t u, uint32_t v) {
          if (u == v) return;
          const uint32_t ou = owner_of(u), ov = owner_of(v);
          uint64_t* ru = cl.map_shared_rank(R + (size_t)(u - ou * RB) * WS, ou);
          uint64_t* rv = cl.map_shared_rank(R + (size_t)(v - ov * RB) * WS, ov);
          for (uint32_t w = tid; w < W; w += blockDim.x) { const uint64_t t = ru[w]; ru[w] = rv[w]; rv[w] = t; }
          if (tid == 0) {
            uint8_t* pu = cl.map_shared_rank(ph + (u - ou * RB), ou);
            uint8_t* pv = cl.map_shared_rank(ph + (v - ov * RB), ov);
            uint8_t t = *pu; *pu = *pv; *pv = t;
            uint8_t* fu = cl.map_shared_rank(fl + (u - ou * RB), ou);
            uint8_t* fv = cl.map_shared_rank(fl + (v - ov * RB), ov);
            t = *fu; *fu = *fv; *fv = t;
          }
          __syncthreads();
        };
        const uint32_t ru = (uint32_t)r;
        if (al <= nn) {
          swaprow(ru + nn, al - 1);
          if (nn != ru + 1 && al != ru + 1) swaprow(ru, al + nn - 1);
        } else {
          swaprow(ru, al - nn - 1);
          swaprow(ru + nn, al - 1);
        }
      }
      cl.sync();
    }
    // 4. every CTA fetches the pivot row, then a barrier before its owner may
    //    overwrite it
    const uint32_t pivrow = (uint32_t)dec[1];
    {
      const uint32_t o = owner_of(pivrow), lr = pivrow - o * RB;
      const uint64_t* src = o == me ? ROW(lr) : cl.map_shared_rank(R + (size_t)lr * WS, o);
      for (uint32_t w = tid; w < W; w += blockDim.x) piv[w] = src[w];
      if (tid == 0) piv[W] = o == me ? ph[lr] : *cl.map_shared_rank(ph + lr, o);
    }
    cl.sync();
    const uint32_t pph = (uint32_t)piv[W];
    // 5. row products on local rows (anticomm_update_rows or the Stabilizer loop)
    const uint32_t ac = branch == 2 ? (uint32_t)r + 1 : (uint32_t)dec[2];
    const uint32_t ru = branch == 2 ? (uint32_t)r + 1 : (uint32_t)r;
    for (uint32_t base = warp * GPW; base < nloc; base += nwarps * GPW) {
      const uint32_t lr = base + gi;
      const uint32_t m = r0 + lr;
      int mode = 0;  // 0: skip, 1: with phase, 2: without phase
      if (lr < nloc && fl[lr] && m != pivrow) {
        if (!destab) mode = (m >= ac && m < (uint32_t)r) ? 1 : 0;
        else if (m >= ru && m < nn) mode = 1;
        else if (m >= nn + ac && m < 2 * nn) mode = 1;
        else if (m < ru && m != ac - 1) mode = 2;
      }
      uint64_t c1 = 0, c2 = 0;
      if (mode) {
        uint64_t* row = ROW(lr);
        for (uint32_t w = gl; w < len; w += G) {
          uint64_t x2 = row[w], z2 = row[len + w];
          mul_step_p(piv[w], piv[len + w], x2, z2, c1, c2);
          row[w] = x2;
          row[len + w] = z2;
        }
      }
      uint32_t sc = (uint32_t)(__popcll(c1) + 2 * __popcll(c2));
      for (uint32_t off = G >> 1; off; off >>= 1) sc += __shfl_xor_sync(0xFFFFFFFFu, sc, off);
      if (gl == 0 && mode == 1 && a.phases) ph[lr] = (uint8_t)((sc + ph[lr] + pph) & 3u);
    }
    // 6. row copies by the owners, outputs by CTA 0
    const int32_t rp = a.rand_ph ? (int32_t)a.rand_ph[j] : -1;
    if (!destab) {
      const uint32_t dst = ac - 1;
      if (owner_of(dst) == me) {
        const uint32_t lr = dst - r0;
        for (uint32_t w = tid; w < W; w += blockDim.x) ROW(lr)[w] = P[w];
        if (tid == 0) ph[lr] = (uint8_t)(rp >= 0 ? rp : (int32_t)pphase);
      }
    } else {
      // destabilizer[ac] = stabilizer[ac] (the pivot row); stabilizer[ac] = pauli
      const uint32_t dd = ac - 1, ds = nn + ac - 1;
      if (owner_of(dd) == me) {
        const uint32_t lr = dd - r0;
        for (uint32_t w = tid; w < W; w += blockDim.x) ROW(lr)[w] = piv[w];
        if (tid == 0) ph[lr] = (uint8_t)pph;
      }
      if (owner_of(ds) == me) {
        const uint32_t lr = ds - r0;
        for (uint32_t w = tid; w < W; w += blockDim.x) ROW(lr)[w] = P[w];
        if (tid == 0) ph[lr] = (uint8_t)(rp >= 0 ? rp : (int32_t)pphase);
      }
      if (branch == 2) r += 1;
    }
    if (me == 0 && tid == 0) {
      a.anticom[j] = (int32_t)ac;
      a.result[j] = rp;
    }
    __syncthreads();
  }
  // write the rows back; every CTA is done with remote shared memory first
  cl.sync();
  for (uint32_t lr = warp; lr < nloc; lr += nwarps)
    for (uint32_t w = lane; w < W; w += 32) a.xzs[(size_t)(r0 + lr) * W + w] = ROW(lr)[w];
  for (uint32_t lr = tid; lr < nloc; lr += blockDim.x) a.ph[r0 + lr] = ph[lr];
  if (me == 0 && tid == 0) {
    if (a.kind == QCB_MIXED_STABILIZER || a.kind == QCB_MIXED_DESTABILIZER) *a.rank = r;
    a.status[0] = (int32_t)status;
    a.status[1] = (int32_t)jstop;
  }
}

static size_t proj_smem_bytes(uint32_t RB, uint32_t W) {
  return ((size_t)2 * W + 1 + (size_t)RB * (W + 1)) * 8 + 2 * (size_t)RB + 16 + 32 + 16 + 32 + 16;
}

// ---------------------------------------------------------------- the whole GPU
// project! of a Stabilizer / MixedStabilizer tableau too tall for one
// cluster's shared memory, on every SM: a cooperative grid (one CTA per SM,
// all resident) with two grid barriers per Pauli.  Phase 1: comm(pauli, row)
// for every row (warp per row) and the first anticommuting stabilizer row by
// a global atomicMin; barrier; phase 2: the same decision in every CTA, then
// row m <- pivot * row m for the anticommuting rows after the pivot (the
// loop of src/project_trace_reset.jl:296-305); barrier.  Writing the Pauli
// into the pivot row is deferred to the next Pauli's phase 1 (CTA 0), whose
// comm test takes that row from the Pauli kept in shared memory, so no third
// barrier is needed.  Every wait at a grid barrier is bounded: on expiry the
// CTA records QCB_ETIMEOUT and returns, and the others give up at their next
// barrier.
struct ProjGridArgs {
  ProjArgs a;
  uint32_t* bar;   // [0] arrivals, [1] generation
  uint32_t* gmin;  // [3]: the first anticommuting row of Pauli j at gmin[j % 3]
  int32_t* err;    // QCB_ETIMEOUT when a grid barrier wait gave up
  // test knob: CTA 1 leaves before the first barrier, so the others' waits
  // run out (0: off)
  uint32_t withhold;
};

// Bounded grid barrier; false when this CTA gave up waiting.
__device__ bool grid_barrier(uint32_t* bar, uint32_t nblocks, int32_t* err) {
  __shared__ int ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    volatile uint32_t* gen = bar + 1;
    const uint32_t g0 = *gen;
    __threadfence();
    ok = 1;
    if (atomicAdd(bar, 1u) == nblocks - 1) {
      atomicExch(bar, 0u);
      __threadfence();
      atomicAdd(bar + 1, 1u);
    } else {
      uint32_t it = 0;
      while (*gen == g0) {
        if (++it > (1u << 24)) {  // about a second
          ok = 0;
          atomicExch(err, QCB_ETIMEOUT);
          break;
        }
        __nanosleep(64);
      }
    }
    __threadfence();
  }
  __syncthreads();
  return ok != 0;
}

__global__ void __launch_bounds__(PROJ_THREADS) project_grid_kernel(const ProjGridArgs g) {
  const ProjArgs& a = g.a;
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
  const uint32_t G = gridDim.x, gw = blockIdx.x * nwarps + warp, NW = G * nwarps;
  const uint32_t W = a.W, len = W / 2, rows = a.rows;
  const bool lead = blockIdx.x == 0;
  extern __shared__ __align__(16) uint64_t smem[];
  uint64_t* Pb[2] = {smem, smem + W};  // the Pauli of projection j in Pb[j & 1]
  uint64_t* piv = smem + 2 * W;
  const uint32_t r = a.kind == QCB_STABILIZER ? rows : (uint32_t)*a.rank;
  uint32_t pprev = 0xFFFFFFFFu;  // the last pivot row, whose Pauli is not written yet
  uint8_t phprev = 0;
  uint32_t j = a.j0;
  for (; j < a.k; j++) {
    uint64_t* P = Pb[j & 1];
    const uint64_t* Pp = Pb[(j + 1) & 1];  // the previous Pauli
    const uint64_t* pj = a.paulis + (size_t)j * W;
    for (uint32_t w = tid; w < W; w += blockDim.x) P[w] = pj[w];
    __syncthreads();
    if (lead && pprev != 0xFFFFFFFFu) {
      for (uint32_t w = tid; w < W; w += blockDim.x) a.xzs[(size_t)pprev * W + w] = Pp[w];
      if (tid == 0) a.ph[pprev] = phprev;
    }
    if (lead && tid == 0) g.gmin[(j + 1) % 3] = 0xFFFFFFFFu;  // the slot of Pauli j + 1 (last used by j - 2)
    // 1. comm flags and the first anticommuting stabilizer row
    for (uint32_t m = gw; m < rows; m += NW) {
      const uint64_t* row = m == pprev ? Pp : a.xzs + (size_t)m * W;
      uint64_t acc = 0;
      for (uint32_t w = lane; w < len; w += 32) acc ^= (P[len + w] & row[w]) ^ (P[w] & row[len + w]);
      const uint32_t c = __reduce_add_sync(0xFFFFFFFFu, (uint32_t)__popcll(acc)) & 1u;
      if (lane == 0) {
        a.flags[m] = (uint8_t)c;
        if (c && m < r) atomicMin(&g.gmin[j % 3], m);
      }
    }
    if (g.withhold && blockIdx.x == 1) return;
    if (!grid_barrier(g.bar, G, g.err)) return;
    // 2. the decision, the same in every CTA
    const uint32_t p = *(volatile uint32_t*)&g.gmin[j % 3];
    const int32_t rp = a.rand_ph ? (int32_t)a.rand_ph[j] : -1;
    if (p == 0xFFFFFFFFu) {
      // commutes with every stabilizer row
      pprev = 0xFFFFFFFFu;  // written in this Pauli's phase 1
      if (a.kind == QCB_STABILIZER && !a.keep_result) {
        if (lead && tid == 0) { a.anticom[j] = 0; a.result[j] = -1; }
        continue;  // phase 2 wrote nothing: no barrier needed
      }
      if (lead && tid == 0) { a.status[0] = PST_NEED_CANON; a.status[1] = (int32_t)j; }
      return;
    }
    for (uint32_t w = tid; w < W; w += blockDim.x) piv[w] = a.xzs[(size_t)p * W + w];
    __syncthreads();
    const uint32_t pph = a.ph[p];
    for (uint32_t m = p + 1 + gw; m < r; m += NW)
      if (a.flags[m]) warp_rowmul(a.xzs, a.ph, W, m, piv, pph, a.phases != 0, lane);
    if (lead && tid == 0) { a.anticom[j] = (int32_t)p + 1; a.result[j] = rp; }
    phprev = (uint8_t)(rp >= 0 ? rp : (int32_t)a.pph[j]);
    pprev = p;
    if (!grid_barrier(g.bar, G, g.err)) return;
  }
  if (lead && pprev != 0xFFFFFFFFu) {
    const uint64_t* Pp = Pb[(j + 1) & 1];
    for (uint32_t w = tid; w < W; w += blockDim.x) a.xzs[(size_t)pprev * W + w] = Pp[w];
    if (tid == 0) a.ph[pprev] = phprev;
  }
  if (lead && tid == 0) { a.status[0] = PST_OK; a.status[1] = (int32_t)a.k; }
}

// ---------------------------------------------------------------- by panels
// Runs of projections by panels of up to 64 Paulis over the whole GPU
// (panel.cuh).  Projection j multiplies every row that anticommutes with P_j
// by the first such stabilizer row (the pivot), copies the pivot into its
// destabilizer row and puts P_j in its place.  Whether a row anticommutes with
// the panel's Paulis is one word per row, and products act on these words as
// on the rows, so the panel's steps run on them alone.  A row's start words
// are its own, those of the last Pauli put into it (word CP[j], its
// commutation bits with the other Paulis of the panel), or none (a copied
// pivot: the set U is that step alone).  Per panel k two launches:
//   SA(k)  CTA 0 (S): panel k's steps on the words; the other CTAs (AF): panel
//          k - 1 applied, a CTA per tile and range of rows, and on the new
//          words the tile's share of the rows' commutation words with panel k +
//          1's Paulis (32 byte lookups in tables over them); a few CTAs the
//          rows' q;
//   M(k)   a CTA per tile: the reduced pivots and the tile's share of the phase
//          data; CTAs over the rows: their sets U and start words, and their
//          words of panel k + 1: the word AF(k - 1) found and the reduced
//          pivots' for the steps in U.
// So the apply is off the chain S, M of a panel.
// A Pauli that commutes with the stabilizer (its result needs the rows), or
// anticommutes with a logical row only, ends the run after the steps before
// it; the host handles that one with the kernels above and goes on.
// Bound by that chain: SA 10.4 + M 8.7 us a panel (n = 1000; 15.0 + 8.3 at
// 4000, where the lookups set SA's length) and 1.6 us a launch.  1000 random
// Paulis, us each with the call: Stabilizer n = 1000 / 4000 4.9 / 12.4 -> 0.48 /
// 0.59, Destabilizer n = 1000 / 2000 5.4 / 11.3 -> 0.48 / 0.53 (one Pauli at a
// time, two cluster or grid barriers each, before; with S, M and the apply as
// three launches in turn 0.54 / 0.64, 0.53 / 0.58).
struct ProjPanelArgs {
  PanelTiles p;
  uint64_t* xzs;
  uint8_t* ph;
  uint32_t nn;         // tableau row of the first stabilizer row; 0 without destabilizer rows
  uint32_t rank;       // stabilizer rows
  uint32_t plain;      // rows below it keep their phase in products (destabilizer rows)
  int skip;            // a commuting Pauli does nothing (Stabilizer without a result)
  const uint64_t* paulis;
  const uint8_t* pph;
  const uint8_t* rand_ph;
  uint32_t j0, cnt;    // this panel's Paulis
  uint32_t jn, cntn;   // the next panel's
  uint32_t jp;         // the first of the previous panel's
  PanelRecord *rec, *prev;  // of this panel and the previous one
  int32_t* state;      // [0] stopped, [1] the next Pauli
  int32_t* anticom;
  int32_t* result;
  uint64_t *word, *wordn;   // [rows] commutation words of this and the next panel
  // [rows] words with the next panel's Paulis before this panel (AF writes,
  // M reads), and the buffer of the SA after the next one, which M clears;
  // likewise [PSTEPS] this panel's Paulis with the next panel's
  unsigned long long *F, *Fz, *CPX, *CPXz;
  unsigned long long *CP, *CPn, *CPz;  // [PSTEPS] the Paulis' own words
  uint32_t *pq, *pqn, *pqz, *pqp;      // [PSTEPS] the Paulis' q; pqp: the previous panel's
  uint8_t* base;       // [rows] start words: BASE_ROW, BASE_NONE or the Pauli's index in the panel
  // up to the first panel's steps: set by the load when the run's first Pauli
  // anticommutes with a stabilizer row; while it is not, these launches do
  // nothing and the run ends before its first Pauli (null: always live)
  uint32_t* live;
  uint32_t first;      // the run's first Pauli
  uint32_t steps, apply, nq, groups, per;
};
constexpr uint32_t BASE_ROW = 255, BASE_NONE = 254;
constexpr uint32_t PP_SLOTS = 3, PP_WINDOW = 32 * PP_SLOTS, PP_REST = 31 * 32;

// S: as canonicalize!'s steps, with the stabilizer rows in their fixed order.
template <uint32_t RPT>
__device__ __forceinline__ void project_steps(const ProjPanelArgs& a) {
  constexpr uint32_t NONE = 0xFFFFFFFFu, KW = PP_SLOTS;
  __shared__ uint4 recA[PSTEPS];  // pivot t: (word, mask)
  __shared__ uint4 recB[PSTEPS];  // (stabilizer row, Pauli, src)
  __shared__ uint2 sCP[PSTEPS];
  __shared__ uint64_t rw[32], ra[32];
  __shared__ uint32_t rs[32], rpos[32], shT, shB, rb, rT;
  PanelRecord& g = *a.rec;
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, R = a.rank;
  if (tid < PSTEPS) {
    g.G[tid] = 0;
    g.q0[tid] = 0;
    g.s[tid] = 0;
    const uint64_t c = a.CP[tid];
    sCP[tid] = make_uint2((uint32_t)c, (uint32_t)(c >> 32));
  }
  if (a.state[0] || (a.live && !*a.live)) {
    if (tid == 0) {
      g.T = 0;
      g.done = 1;
      a.state[0] = 1;
    }
    return;
  }
  const uint64_t* word = a.word + a.nn;
  uint32_t wd[KW][4], src[KW];
  uint64_t w[RPT], A[RPT];
  uint32_t ws[RPT];
  if (warp == 0) {
#pragma unroll
    for (uint32_t k = 0; k < KW; k++) {
      const uint32_t r = 32 * k + lane;
      const uint64_t v = r < R ? word[r] : 0ull;
      wd[k][0] = (uint32_t)v;
      wd[k][1] = (uint32_t)(v >> 32);
      wd[k][2] = wd[k][3] = 0;
      src[k] = PSTEPS;
    }
  } else {
#pragma unroll
    for (uint32_t k = 0; k < RPT; k++) {
      const uint32_t r = PP_WINDOW + PP_REST * k + tid - 32;
      w[k] = r < R ? word[r] : 0ull;
      A[k] = 0;
      ws[k] = PSTEPS;
    }
  }
  __syncthreads();
  const uint32_t nrest = R > PP_WINDOW ? R - PP_WINDOW : 0u, nbw = min(31u, (nrest + 31) / 32), nbar = 32 * (nbw + 1);
  if (warp == 0) {
    uint32_t T = 0, t0 = 1, t1 = 0, stop = a.cnt;  // t1:t0: bit T
    uint32_t ad = (uint32_t)__cvta_generic_to_shared(recA);
    const uint32_t bd = (uint32_t)__cvta_generic_to_shared(recB) - ad;
    const uint32_t cd = (uint32_t)__cvta_generic_to_shared(sCP);
#pragma unroll
    for (uint32_t h = 0; h < 2; h++) {
      const uint32_t ce = a.cnt > 32 * h ? min(32u, a.cnt - 32 * h) : 0u;
      for (uint32_t c = 0; c < ce && stop == a.cnt; c++) {
        bool miss = false;
        uint32_t cm = 1u << c;
        // Paulis whose pivot is in the window
#pragma unroll 1
        for (; c < ce; c++, cm <<= 1) {
          const uint32_t c0 = (wd[0][h] & cm) ? lane : NONE, c1 = (wd[1][h] & cm) ? 32 + lane : NONE,
                         c2 = (wd[2][h] & cm) ? 64 + lane : NONE;
          const uint32_t best = min(min(c0, c1), c2), m = __reduce_min_sync(0xFFFFFFFFu, best);
          if (m == NONE) { miss = true; break; }
          const bool y1 = c1 == best, y2 = c2 == best;
          uint32_t s[4];
#pragma unroll
          for (uint32_t q = 0; q < 4; q++) s[q] = y2 ? wd[2][q] : (y1 ? wd[1][q] : wd[0][q]);
          const uint32_t sr = y2 ? src[2] : (y1 ? src[1] : src[0]);
          asm volatile("{.reg .pred p; setp.eq.u32 p, %0, %1; @p st.shared.v4.u32 [%2], {%3, %4, %5, %6};"
                       "@p st.shared.v4.u32 [%7], {%1, %8, %9, %9};}" ::"r"(best), "r"(m), "r"(ad), "r"(s[0]), "r"(s[1]),
                       "r"(s[2] | t0), "r"(s[3] | t1), "r"(ad + bd), "r"(32 * h + c), "r"(sr)
                       : "memory");
          __syncwarp();
          uint32_t p[4], n0, n1;
          asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(p[0]), "=r"(p[1]), "=r"(p[2]), "=r"(p[3]) : "r"(ad) : "memory");
          asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(n0), "=r"(n1) : "r"(cd + 8 * (32 * h + c)) : "memory");
          ad += 16;
#pragma unroll
          for (uint32_t k = 0; k < KW; k++) {
            xor_if(wd[k], wd[k][h], cm, p);
            if (32 * k + lane == m) {  // the Pauli takes the pivot's place
              wd[k][0] = n0;
              wd[k][1] = n1;
              wd[k][2] = wd[k][3] = 0;
              src[k] = T;
            }
          }
          T++;
          t1 = (t1 << 1) | (t0 >> 31);
          t0 <<= 1;
        }
        if (!miss) break;
        uint32_t m = NONE;
        if (nrest) {
          if (lane == 0) { rb = 32 * h + c; rT = T; }
          __syncwarp();
          asm volatile("bar.sync 1, %0;" ::"r"(nbar) : "memory");
          asm volatile("bar.sync 2, %0;" ::"r"(nbar) : "memory");
          const uint32_t v = lane >= 1 && lane <= nbw ? rpos[lane] : NONE;
          m = __reduce_min_sync(0xFFFFFFFFu, v);
          if (m != NONE && v == m) {
            recA[T] = make_uint4((uint32_t)rw[lane], (uint32_t)(rw[lane] >> 32), (uint32_t)ra[lane] | t0,
                                 (uint32_t)(ra[lane] >> 32) | t1);
            recB[T] = make_uint4(m, 32 * h + c, rs[lane], 0);
          }
        }
        if (m == NONE) {  // commutes with every stabilizer row
          if (!a.skip) stop = 32 * h + c;
          continue;
        }
        __syncwarp();  // no row of the window has the bit
        ad += 16;
        T++;
        t1 = (t1 << 1) | (t0 >> 31);
        t0 <<= 1;
      }
    }
    if (lane == 0) { shT = T; shB = stop; rb = NONE; }
    __syncwarp();
    if (nrest) asm volatile("bar.sync 1, %0;" ::"r"(nbar) : "memory");
  } else if (warp <= nbw) {
    const uint32_t r0 = PP_WINDOW + tid - 32;
    uint32_t t = 0;
    while (true) {
      asm volatile("bar.sync 1, %0;" ::"r"(nbar) : "memory");
      const uint32_t b = rb, T = rT;
      if (b == NONE) break;
      for (; t < T; t++) {
        const uint4 e = recA[t], f = recB[t];
        const uint64_t pw = (uint64_t)e.x | ((uint64_t)e.y << 32), pA = (uint64_t)e.z | ((uint64_t)e.w << 32);
        const uint2 n = sCP[f.y];
#pragma unroll
        for (uint32_t k = 0; k < RPT; k++) {
          if (k && k * PP_REST >= nrest) break;
          const uint64_t y = bitmask64(w[k], f.y);
          w[k] ^= pw & y;
          A[k] ^= pA & y;
          if (f.x == r0 + k * PP_REST) {
            w[k] = (uint64_t)n.x | ((uint64_t)n.y << 32);
            A[k] = 0;
            ws[k] = t;
          }
        }
      }
      uint32_t bp = NONE, bs = 0;
      uint64_t bw = 0, bA = 0;
#pragma unroll
      for (uint32_t k = RPT; k-- > 0;)
        if ((w[k] >> b) & 1ull) {
          bp = r0 + k * PP_REST;
          bw = w[k];
          bA = A[k];
          bs = ws[k];
        }
      const uint32_t m = __reduce_min_sync(0xFFFFFFFFu, bp);
      if (lane == 0) rpos[warp] = m;
      if (bp == m && m != NONE) { rw[warp] = bw; ra[warp] = bA; rs[warp] = bs; }
      asm volatile("bar.sync 2, %0;" ::"r"(nbar) : "memory");
    }
  }
  __syncthreads();
  const uint32_t T = shT, done = shB;
  if (tid < T) {
    const uint4 e = recA[tid], f = recB[tid];
    g.stp[tid] = a.nn + f.x;
    g.bt[tid] = f.y;
    g.src[tid] = f.z;
    g.sbt[tid] = f.z < PSTEPS ? recB[f.z].y : PSTEPS;
    g.A[tid] = (uint64_t)e.z | ((uint64_t)e.w << 32);
    g.PW[tid] = (uint64_t)e.x | ((uint64_t)e.y << 32);
    a.anticom[a.j0 + f.y] = (int32_t)f.x + 1;
    a.result[a.j0 + f.y] = a.rand_ph ? (int32_t)a.rand_ph[a.j0 + f.y] : -1;
  }
  if (tid == 0) {
    g.T = T;
    g.done = done < a.cnt;
    a.state[0] = done < a.cnt;
    a.state[1] = (int32_t)(a.j0 + done);
  }
}

// q of the stabilizer row that Pauli b of the panel from j0 on becomes.
__device__ __forceinline__ uint32_t new_row_q(const ProjPanelArgs& a, const uint32_t* pq, uint32_t j0, uint32_t b) {
  return (__ldcg(pq + b) + (a.rand_ph ? __ldcg(a.rand_ph + j0 + b) - __ldcg(a.pph + j0 + b) : 0u)) & 3u;
}

// M: blocks 0 .. ntile - 1 a tile each, block ntile the pivots' own sets, the
// others MID_THREADS rows each.
__global__ void __launch_bounds__(MID_THREADS) project_mid_kernel(const ProjPanelArgs a) {
  __shared__ union {
    TileSmem t;
    struct {
      ulonglong2 P[PSTEPS];   // (pivot's word, the Pauli's word)
      ulonglong2 N[PSTEPS];   // the same with the next panel's Paulis
      ulonglong2 C[PSTEPS];   // the Paulis' words with this panel's and the next one's
      uint64_t start[PSTEPS];  // the pivots' start rows' words with the next one's
      uint2 sb[PSTEPS];       // (pivot row, 31 - bit within its half word | Pauli << 8)
      uint32_t bt[PSTEPS];
    } r;
  } s;
  const PanelTiles& p = a.p;
  const uint32_t tid = threadIdx.x, blk = blockIdx.x;
  // While SA runs: the Paulis' words of the tile as the tiles keep them, or the
  // rows' panel words.  SA waited for the launch that wrote them before it let
  // this kernel start, so they are in L2; loads before the wait pass L1 by.
  __shared__ ulonglong2 pw[PSTEPS][2];
  __shared__ uint32_t sq[PSTEPS];  // tile 0: q of the rows the Paulis become
  const uint32_t r = blk > p.ntile ? (blk - p.ntile - 1) * MID_THREADS + tid : p.rows;
  uint64_t w = 0;
  if (blk == 0 && tid < a.cnt) sq[tid] = new_row_q(a, a.pq, a.j0, tid);
  if (blk < p.ntile) {
    const uint32_t b = tid >> 2, c = 2 * blk + (tid & 1);
    ((uint64_t*)pw[b])[tid & 3] =
        b < a.cnt && c < p.len ? __ldcg(a.paulis + (size_t)(a.j0 + b) * p.W + (tid & 2 ? p.len : 0) + c) : 0ull;
  } else if (r < p.rows) {
    w = __ldcg(a.word + r);
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;");
  PanelRecord& g = *a.rec;
  const uint32_t T = g.T;
  if (blk < p.ntile) {
    __syncthreads();
    tile_reduce(
        p, g, blk, s.t,
        [&](uint32_t t, uint32_t r) -> const ulonglong2* {
          const uint32_t b = g.sbt[t];  // of the record's T steps, or stale
          return b < PSTEPS ? pw[b] : p.t + ((size_t)blk * p.rows + r) * 2;
        },
        [&](uint32_t t, uint32_t r) -> uint32_t {
          const uint32_t b = g.sbt[t];
          if (b < PSTEPS) return blk == 0 ? sq[b] : 0u;
          return 2u * p.par[(size_t)blk * p.rows + r] + (blk == 0 ? p.q[r] : 0u);
        },
        [&](uint32_t t, const uint64_t* v) {
          const uint32_t c = (uint32_t)(__popcll(v[0] & v[2]) + __popcll(v[1] & v[3]));
          if (c) atomicAdd(&g.s[t], c);
        });
    return;
  }
  // The record's fields beyond its T steps are stale but readable (zero at the
  // start): nothing here waits for T, or for an index, before loading what it can.
  const bool next = a.cntn != 0;
  const uint32_t t4 = tid >> 2, x0 = (tid & 3) * 16;
  const uint64_t A = g.A[t4] >> x0;
  uint32_t b = 0, sp = 0, sr = PSTEPS, sbt = PSTEPS;
  uint64_t PW = 0, F = 0, v = 0, w_own = 0;
  if (tid < PSTEPS) {
    b = g.bt[tid];
    sp = g.stp[tid];
    sr = g.src[tid];
    sbt = g.sbt[tid];
    PW = g.PW[tid];
    s.r.bt[tid] = b;
    if (blk == p.ntile && sr >= PSTEPS) w_own = a.word[sp];
    s.r.C[tid] = make_ulonglong2(a.CP[tid], next ? a.CPX[tid] : 0ull);
    if (next) F = a.F[sp];
  }
  if (r < p.rows) {
    a.Fz[r] = 0;
    if (next) v = a.F[r];
  }
  const uint32_t T0 = __syncthreads_count(tid < T && b < 32);  // steps in the words' low halves
  if (tid < PSTEPS) {
    const ulonglong2 c = s.r.C[b];
    const bool in = tid < T;
    s.r.P[tid] = make_ulonglong2(PW, c.x);
    s.r.N[tid].y = c.y;
    s.r.sb[tid] = make_uint2(sp, (31u - (b & 31u)) | b << 8);
    s.r.start[tid] = !in ? 0ull : sbt < PSTEPS ? s.r.C[sbt].y : F;
  }
  __syncthreads();
  {  // the reduced pivots' next words: a thread per pivot and 16 start rows
    uint64_t n = 0;
#pragma unroll
    for (uint32_t x = 0; x < 16; x++) n ^= s.r.start[x0 + x] & bitmask64(A, x);
    n ^= __shfl_xor_sync(0xFFFFFFFFu, n, 1);
    n ^= __shfl_xor_sync(0xFFFFFFFFu, n, 2);
    if ((tid & 3) == 0) s.r.N[t4].x = n;
  }
  __syncthreads();
  if (blk == p.ntile) {
    if (tid < PSTEPS) { a.CPz[tid] = 0; a.pqz[tid] = 0; a.CPXz[tid] = 0; }
    // pivot t's start word replayed up to its step
    if (tid < T) {
      uint64_t w = sr < PSTEPS ? s.r.P[sr].y : w_own, U = 0;
      for (uint32_t t = sr < PSTEPS ? sr + 1 : 0; t < tid; t++) {
        const uint64_t y = bitmask64(w, s.r.bt[t]);
        w ^= s.r.P[t].x & y;
        U |= (1ull << t) & y;
      }
      g.own[tid] = U;
    }
    return;
  }
  if (r >= p.rows) return;
  uint32_t p0 = (uint32_t)w, p1 = (uint32_t)(w >> 32), v0 = (uint32_t)v, v1 = (uint32_t)(v >> 32), u0 = 0, u1 = 0;
  uint32_t base = BASE_ROW;
  const uint32_t partner = r < a.nn ? r + a.nn : 0xFFFFFFFEu;  // its stabilizer row
  auto replay = [&](uint32_t t, uint32_t& half) {
    const ulonglong2 P = s.r.P[t], N = s.r.N[t];
    const uint2 sb = s.r.sb[t];
    const uint32_t m = (uint32_t)((int32_t)__funnelshift_l(0u, half, sb.y) >> 31);  // by 31 - bit
    const uint32_t tb = 1u << (t & 31), b0 = t < 32 ? tb : 0u, b1 = t < 32 ? 0u : tb;
    p0 ^= (uint32_t)P.x & m;
    p1 ^= (uint32_t)(P.x >> 32) & m;
    v0 ^= (uint32_t)N.x & m;
    v1 ^= (uint32_t)(N.x >> 32) & m;
    u0 |= b0 & m;
    u1 |= b1 & m;
    const bool pivot = sb.x == r;
    if (pivot || sb.x == partner) {  // the Pauli takes its place; a copy of the pivot
      const uint64_t nw = pivot ? P.y : P.x, nv = pivot ? N.y : N.x;
      p0 = (uint32_t)nw;
      p1 = (uint32_t)(nw >> 32);
      v0 = (uint32_t)nv;
      v1 = (uint32_t)(nv >> 32);
      u0 = pivot ? 0u : b0;
      u1 = pivot ? 0u : b1;
      base = pivot ? sb.y >> 8 : BASE_NONE;
    }
  };
#pragma unroll 4
  for (uint32_t t = 0; t < T0; t++) replay(t, p0);
#pragma unroll 4
  for (uint32_t t = T0; t < T; t++) replay(t, p1);
  a.wordn[r] = (uint64_t)v0 | ((uint64_t)v1 << 32);
  p.U[r] = (uint64_t)u0 | ((uint64_t)u1 << 32);
  a.base[r] = (uint8_t)base;
}

// The byte tables of the next panel's Paulis on one tile: tab[b][v] is the
// XOR, over the bits of v, of the Paulis that anticommute with that bit of
// byte b of a row's words (x, x, z, z).
struct FlagSmem {
  uint64_t col[256];
  uint64_t tab4[64][16];
  uint64_t tab[32][256];
};

__device__ __forceinline__ void flag_tables(const ProjPanelArgs& a, uint32_t tile, FlagSmem& s) {
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const PanelTiles& p = a.p;
  {  // word k of the row (x0, x1, z0, z1) against word k ^ 2 of the Paulis; 32 warps, 8 bits each
    const uint32_t k = warp >> 3, q = k ^ 2, c = 2 * tile + (q & 1);
    const bool in = c < p.len;
    const uint64_t* P = a.paulis + (size_t)a.jn * p.W + (q >= 2 ? p.len : 0) + c;
    const uint64_t v0 = in && lane < a.cntn ? __ldcg(P + (size_t)lane * p.W) : 0ull;
    const uint64_t v1 = in && lane + 32 < a.cntn ? __ldcg(P + (size_t)(lane + 32) * p.W) : 0ull;
    for (uint32_t b = 8 * (warp & 7), e = b + 8; b < e; b++) {
      const uint32_t lo = __ballot_sync(0xFFFFFFFFu, (v0 >> b) & 1ull), hi = __ballot_sync(0xFFFFFFFFu, (v1 >> b) & 1ull);
      if (lane == 0) s.col[64 * k + b] = (uint64_t)lo | ((uint64_t)hi << 32);
    }
  }
  __syncthreads();
  {
    const uint32_t k = tid >> 4, v = tid & 15;
    uint64_t x = 0;
#pragma unroll
    for (uint32_t b = 0; b < 4; b++) x ^= s.col[4 * k + b] & bitmask64(v, b);
    s.tab4[k][v] = x;
  }
  __syncthreads();
#pragma unroll 4
  for (uint32_t e = tid; e < 8192; e += 1024) {
    const uint32_t k = e >> 8, v = e & 255;
    s.tab[k][v] = s.tab4[2 * k][v & 15] ^ s.tab4[2 * k + 1][v >> 4];
  }
  __syncthreads();
}

__device__ __forceinline__ uint64_t flag_lookup(const FlagSmem& s, ulonglong2 x, ulonglong2 z) {
  const uint64_t v[4] = {x.x, x.y, z.x, z.y};
  uint64_t f = 0;
#pragma unroll
  for (uint32_t k = 0; k < 4; k++)
#pragma unroll
    for (uint32_t b = 0; b < 8; b++) f ^= s.tab[8 * k + b][(uint32_t)(v[k] >> (8 * b)) & 255u];
  return f;
}

struct ApplyFlagSmem {
  ApplySmem a;
  FlagSmem f;
};

// SA.
template <uint32_t RPT>
__global__ void __launch_bounds__(1024) project_steps_apply_kernel(const ProjPanelArgs a) {
  extern __shared__ __align__(16) uint8_t dsm[];
  if (blockIdx.x == 0) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;");
    if (a.steps) project_steps<RPT>(a);
    return;
  }
  const PanelRecord& g = *a.prev;
  const PanelTiles& p = a.p;
  const uint32_t tid = threadIdx.x, blk = blockIdx.x - 1;
  // While M runs: the next Paulis' tables, and the thread's first row (the
  // previous apply wrote it, and M waited for that; loads past L1 as in M).
  const uint32_t u = blk < a.nq ? 0u : blk - a.nq, tile = u / a.groups, grp = u - tile * a.groups;
  const uint32_t r0 = grp * a.per + tid, r1 = min(p.rows, (grp + 1) * a.per);
  ApplyFlagSmem& s = *(ApplyFlagSmem*)dsm;
  ulonglong2 x0 = make_ulonglong2(0, 0), z0 = x0;
  if (blk >= a.nq) {
    if (a.apply && r0 < r1) {
      const ulonglong2* d = p.t + ((size_t)tile * p.rows + r0) * 2;
      x0 = __ldcg(d);
      z0 = __ldcg(d + 1);
    }
    if (a.cntn) flag_tables(a, tile, s.f);
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;");
  if (a.live && !*a.live) return;
  const uint32_t T = a.apply ? g.T : 0u;
  if (blk < a.nq) {  // q of every row
    if (!T) return;
    PhaseSmem& s = *(PhaseSmem*)dsm;
    phase_data(g, s, [&](uint32_t t) { return g.own[t]; });
    for (uint32_t r = blk * blockDim.x + tid; r < p.rows; r += a.nq * blockDim.x) {
      const uint64_t U = p.U[r];
      const uint32_t base = a.base[r];
      if (r < a.plain) {
        // a destabilizer row: products keep its phase, a copy brings the pivot's
        if (base == BASE_NONE) {
          const uint32_t t = __ffsll((long long)U) - 1;
          p.q[r] = (uint8_t)(((uint32_t)((s.Q1 >> t) & 1ull) + 2u * (uint32_t)((s.Q2 >> t) & 1ull) - g.s[t]) & 3u);
        }
      } else if (base != BASE_ROW || U) {
        const uint32_t q = base != BASE_ROW ? new_row_q(a, a.pqp, a.jp, base) : p.q[r];
        p.q[r] = (uint8_t)((q + phase_of(s, U)) & 3u);
      }
    }
    return;
  }
  const bool next = a.cntn && !(a.apply && g.done);
  if (!T && !next) return;
  if (T) apply_tables(p, tile, s.a);
  const bool two = 2 * tile + 1 < p.len;
  auto pauli = [&](uint32_t j, ulonglong2& x, ulonglong2& z) {
    const uint64_t* P = a.paulis + (size_t)j * p.W + 2 * tile;
    x = make_ulonglong2(P[0], two ? P[1] : 0ull);
    z = make_ulonglong2(P[p.len], two ? P[p.len + 1] : 0ull);
  };
  for (uint32_t r = r0; r < r1; r += blockDim.x) {
    ulonglong2* d = p.t + ((size_t)tile * p.rows + r) * 2;
    const bool have = a.apply && r == r0;
    ulonglong2 x = have ? x0 : d[0], z = have ? z0 : d[1];
    if (T) {
      const uint64_t U = p.U[r];
      const uint32_t base = a.base[r];
      if (base == BASE_NONE) x = z = make_ulonglong2(0, 0);
      else if (base != BASE_ROW) pauli(a.jp + base, x, z);
      if (U || base != BASE_ROW) {
        ulonglong2 mx, mz;
        apply_lookup(s.a, U, mx, mz);
        const uint32_t odd = parity64((mz.x & x.x) ^ (mz.y & x.y));
        x = xor128(x, mx);
        z = xor128(z, mz);
        d[0] = x;
        d[1] = z;
        if (r >= a.plain) {
          uint8_t* par = p.par + (size_t)tile * p.rows + r;
          if (base != BASE_ROW) *par = (uint8_t)odd;
          else if (odd) *par ^= 1u;
        }
      }
    }
    if (next) {
      const uint64_t f = flag_lookup(s.f, x, z);
      if (f) atomicXor(a.F + r, (unsigned long long)f);
    }
  }
  if (next && grp == 0 && tid < a.cntn) {  // the next Paulis' own words and q
    ulonglong2 x, z;
    pauli(a.jn + tid, x, z);
    const uint64_t f = flag_lookup(s.f, x, z);
    if (f) atomicXor(a.CPn + tid, (unsigned long long)f);
    const uint32_t q = (uint32_t)(__popcll(x.x & z.x) + __popcll(x.y & z.y)) + (tile == 0 ? a.pph[a.jn + tid] : 0u);
    if (q) atomicAdd(a.pqn + tid, q);
  }
  if (next && grp == 0 && tid >= 512 && tid - 512 < a.cnt) {  // this panel's Paulis with them
    ulonglong2 x, z;
    pauli(a.j0 + tid - 512, x, z);
    const uint64_t f = flag_lookup(s.f, x, z);
    if (f) atomicXor(a.CPX + tid - 512, (unsigned long long)f);
  }
}

// The rows into the tiles, and back (a warp a row).
__global__ void __launch_bounds__(256) project_load_kernel(const ProjPanelArgs a) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;");
  const uint32_t r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (blockIdx.x == 0) {
    // both records, and the Paulis' words and q of three panels
    for (uint32_t k = threadIdx.x; k < 2 * sizeof(PanelRecord) / 4; k += blockDim.x) ((uint32_t*)a.rec)[k] = 0;
    for (uint32_t k = threadIdx.x; k < 3 * PSTEPS; k += blockDim.x) { a.CP[k] = 0; a.pq[k] = 0; }
    for (uint32_t k = threadIdx.x; k < 2 * PSTEPS; k += blockDim.x) a.CPX[k] = 0;
    if (threadIdx.x == 0) { a.state[0] = 0; a.state[1] = (int32_t)a.j0; }
  }
  if (r >= a.p.rows) return;
  const uint32_t ph = a.ph[r];
  const uint64_t* row = a.xzs + (size_t)r * a.p.W;
  tiles_load_row(a.p, row, r, ph, lane);
  if (a.live && r >= a.nn && r < a.nn + a.rank) {
    const uint64_t* P = a.paulis + (size_t)a.j0 * a.p.W;
    uint64_t c = 0;
    for (uint32_t k = lane; k < a.p.len; k += 32) c ^= (row[k] & P[a.p.len + k]) ^ (row[a.p.len + k] & P[k]);
    const uint32_t odd = __reduce_xor_sync(0xFFFFFFFFu, parity64(c));
    if (lane == 0 && odd) *a.live = 1;
  }
  if (lane == 0) {
    a.word[r] = 0;
    a.F[r] = a.Fz[r] = 0;
    if (r < a.plain) a.p.q[r] = (uint8_t)ph;
  }
}

__global__ void __launch_bounds__(256) project_store_kernel(const ProjPanelArgs a) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;");
  const uint32_t r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (r >= a.p.rows || short_trial(a.state, a.first)) return;
  const uint32_t ph = tiles_store_row(a.p, a.xzs + (size_t)r * a.p.W, r, lane);
  if (lane == 0) a.ph[r] = r < a.plain ? a.p.q[r] : (uint8_t)ph;
}

// A launch as a programmatic dependent of the one before it on the stream.
static cudaError_t launch_pp(void (*k)(const ProjPanelArgs), uint32_t grid, uint32_t block, size_t smem, cudaStream_t st,
                             const ProjPanelArgs& a) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return cudaLaunchKernelEx(&cfg, k, a);
}

// Runs worth a panel (32 random Paulis on 100 / 1000 / 4000 qubits 186 / 244 / 486
// -> 112 / 114 / 142 us with the call), the most stabilizer rows its search holds in
// registers, the steps a run has to make before the next is tried at once, the
// Paulis before the next trial after a first failed one and those that have to be
// left for it (a trial costs 20 to 40 us), and the panels queued before anything is
// waited for.
constexpr uint32_t PROJ_PANEL_MIN = 32, PROJ_PANEL_ROWS = PP_WINDOW + 9 * PP_REST, PROJ_PANEL_GOOD = 32,
                   PROJ_PANEL_BACKOFF = 64, PROJ_PANEL_AGAIN = 128,
                   PROJ_TRIAL_PANELS = 4;

// Projections [first, k) by panels until one that commutes with the stabilizer
// (or all are done): begin(), queue() of the panels, store().  A run that ends
// within PROJ_PANEL_SHORT Paulis (short_trial of `state`) is a failed trial: its
// store() leaves the tableau as it was, for the other kernels.  Panels queued
// past a run's end do nothing.  `live` is zero before.
struct PanelRun {
  Scratch scratch;
  cudaStream_t st;
  ProjPanelArgs a{};
  uint32_t R = 0, k = 0, grid = 0, row_blocks = 0, next = 0;  // next: the panel to queue
  uint64_t* word = nullptr;
  unsigned long long *F = nullptr, *CP = nullptr;
  uint32_t* pq = nullptr;
  PanelRecord* rec = nullptr;
  void (*sa)(const ProjPanelArgs) = nullptr;
  static constexpr size_t SMEM = std::max(sizeof(ApplyFlagSmem), sizeof(PhaseSmem));

  explicit PanelRun(cudaStream_t s) : scratch(s), st(s) {}

  void buffers(uint32_t b) {  // of panel b
    const uint32_t e = b & 1, o = e ^ 1, i0 = b % 3, i1 = (b + 1) % 3, i2 = (b + 2) % 3;
    a.rec = rec + e; a.prev = rec + o;
    a.word = word + (size_t)e * R; a.wordn = word + (size_t)o * R;
    a.F = F + (size_t)o * R; a.Fz = F + (size_t)e * R;
    a.CP = CP + i0 * PSTEPS; a.CPn = CP + i1 * PSTEPS; a.CPz = CP + i2 * PSTEPS;
    a.pq = pq + i0 * PSTEPS; a.pqn = pq + i1 * PSTEPS; a.pqz = a.pqp = pq + i2 * PSTEPS;
    a.CPX = CP + (3 + e) * PSTEPS; a.CPXz = CP + (3 + o) * PSTEPS;
  }
  uint32_t panels() const { return (k - a.first + PSTEPS - 1) / PSTEPS; }
  uint32_t span(uint32_t b) const { return b < panels() ? std::min(PSTEPS, k - a.first - b * PSTEPS) : 0u; }

  // Launch SA of panel b.
  int steps(uint32_t b) {
    buffers(b);
    a.jp = a.j0;
    a.j0 = a.first + b * PSTEPS; a.cnt = span(b);
    a.jn = a.j0 + a.cnt; a.cntn = span(b + 1);
    a.steps = b < panels(); a.apply = b > 0;
    QCB_CUDA(launch_pp(sa, a.apply || a.cntn ? grid : 1u, 1024, SMEM, st, a));
    return QCB_OK;
  }

  // *none: no room for a copy of the rows, nothing launched.
  int begin(const qcb_tableau* t, int kind, uint32_t rank, const uint64_t* pxzs, const uint8_t* pph,
            const uint8_t* d_rand, uint32_t j0, uint32_t end, int skip, int32_t* d_anti, int32_t* d_res, uint32_t* live,
            bool* none) {
    const bool destab = kind == QCB_DESTABILIZER || kind == QCB_MIXED_DESTABILIZER;
    const uint32_t W = t->W, len = W / 2, ntile = (len + 1) / 2;
    R = destab ? t->rows : rank;
    a.first = j0;
    k = end;
    size_t bytes = 0;
    auto place = [&](size_t n) { const size_t o = bytes; bytes += (n + 127) / 128 * 128; return o; };
    const size_t o_t = place((size_t)ntile * R * 32), o_po = place((size_t)ntile * PSTEPS * 32),
                 o_w = place((size_t)4 * R * 8), o_u = place((size_t)R * 8), o_q = place(R), o_b = place(R),
                 o_par = place((size_t)ntile * R), o_rec = place(2 * sizeof(PanelRecord)), o_cp = place(5 * PSTEPS * 8),
                 o_pq = place(3 * PSTEPS * 4), o_st = place(8);
    const cudaError_t e = scratch.alloc(bytes);
    *none = e == cudaErrorMemoryAllocation;
    if (*none) return QCB_OK;
    QCB_CUDA(e);
    uint8_t* m = scratch.p;
    a.p = PanelTiles{R, W, len, ntile, 1, (ulonglong2*)(m + o_t), (ulonglong2*)(m + o_po), nullptr, (uint64_t*)(m + o_u),
                     m + o_q, m + o_par};
    a.xzs = t->xzs; a.ph = t->phases; a.nn = destab ? t->rows / 2 : 0; a.rank = rank; a.plain = destab ? rank : 0;
    a.skip = skip; a.paulis = pxzs; a.pph = pph; a.rand_ph = d_rand;
    a.state = (int32_t*)(m + o_st); a.anticom = d_anti; a.result = d_res; a.base = m + o_b;
    word = (uint64_t*)(m + o_w);
    F = (unsigned long long*)word + (size_t)2 * R;
    CP = (unsigned long long*)(m + o_cp);
    pq = (uint32_t*)(m + o_pq);
    rec = (PanelRecord*)(m + o_rec);
    const uint32_t rest = rank > PP_WINDOW ? rank - PP_WINDOW : 0;
    sa = rest <= PP_REST ? project_steps_apply_kernel<1>
       : rest <= 2 * PP_REST ? project_steps_apply_kernel<2>
       : rest <= 5 * PP_REST ? project_steps_apply_kernel<5> : project_steps_apply_kernel<9>;
    QCB_CUDA(cudaFuncSetAttribute(sa, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM));
    const uint32_t nsm = (uint32_t)std::max(device_sm_count(), 1);
    a.nq = (R + 1023) / 1024;
    a.groups = std::max<uint32_t>(1, std::min<uint32_t>((nsm > a.nq + 1 ? nsm - 1 - a.nq : 1) / ntile, (R + 255) / 256));
    a.per = (R + a.groups - 1) / a.groups;
    grid = 1 + a.nq + ntile * a.groups;
    row_blocks = (R + 7) / 8;
    buffers(0);
    a.j0 = a.first;
    a.live = skip ? nullptr : live;  // skipped Paulis do not end the run
    QCB_CUDA(launch_pp(project_load_kernel, row_blocks, 256, 0, st, a));
    // panel 0's words, as the next words of a panel before it without steps
    a.jn = a.first; a.cntn = span(0);
    a.F = (unsigned long long*)a.word; a.CPn = a.CP; a.pqn = a.pq;
    QCB_CUDA(launch_pp(sa, grid, 1024, SMEM, st, a));
    if (int s = steps(0)) return s;
    a.live = nullptr;
    return QCB_OK;
  }

  // Launches up to and with the apply of panel `upto` - 1.
  int queue(uint32_t upto) {
    for (; next < upto; next++) {
      QCB_CUDA(launch_pp(project_mid_kernel, a.p.ntile + 1 + (R + MID_THREADS - 1) / MID_THREADS, MID_THREADS, 0, st, a));
      if (int s = steps(next + 1)) return s;
    }
    return QCB_OK;
  }
  int store() {
    QCB_CUDA(launch_pp(project_store_kernel, row_blocks, 256, 0, st, a));
    return QCB_OK;
  }
};

static uint32_t g_proj_cs = 0;  // tuner override (0 = automatic)
static uint32_t g_proj_grid = 0;  // the whole-GPU kernel: 0 automatic, 1 always (where it applies), 2 never
static uint32_t g_proj_withhold = 0;  // test knob, see ProjGridArgs::withhold

}  // namespace qcb

using namespace qcb;

extern "C" {

// The k projections of one call: Paulis from a device tableau (pxzs, pph),
// or single-qubit Paulis (qubits: 1-based host array, basis bit 0 = X,
// bit 1 = Z); rand_host (host, 0 or 2 per projection) turns them into
// projectrand!.
static int project_impl(qcb_tableau* t, int kind, int32_t* rank_io, const uint64_t* pxzs, const uint8_t* pph,
                        const uint32_t* qubits, uint32_t basis, uint32_t k, int keep_result, int phases,
                        const uint8_t* rand_host, int32_t* anticom, int32_t* result, uint32_t* n_done, void* stream) {
  if (!t || !anticom || !result) return fail(QCB_EARG, "null argument");
  if (kind < 0 || kind > 3) return fail(QCB_EARG, "project!: bad state kind");
  const bool mixed = kind == QCB_MIXED_STABILIZER || kind == QCB_MIXED_DESTABILIZER;
  if (mixed && !rank_io) return fail(QCB_EARG, "project!: rank required for mixed states");
  if ((kind == QCB_DESTABILIZER || kind == QCB_MIXED_DESTABILIZER) && (t->rows % 2))
    return fail(QCB_EDIM, "project!: destabilizer tableaux have an even number of rows");
  if (kind == QCB_MIXED_DESTABILIZER && t->rows != 2 * t->nqubits)
    return fail(QCB_EDIM, "project!: MixedDestabilizer tableaux have 2n rows");
  if (mixed && (*rank_io < 0 || (uint32_t)*rank_io > (kind == QCB_MIXED_STABILIZER ? t->rows : t->rows / 2)))
    return fail(QCB_EBOUNDS, "project!: rank out of range");
  cudaStream_t st = S(stream);
  if (n_done) *n_done = 0;
  if (!k) return QCB_OK;
  const uint32_t W = t->W, len = W / 2;
  std::vector<uint32_t> q0;
  if (qubits) {
    q0.resize(k);
    for (uint32_t j = 0; j < k; j++) {
      if (qubits[j] == 0) return fail(QCB_EZEROQUBIT, "qubit indices start at 1 (NoZeroQubit)");
      if (qubits[j] > t->nqubits) return fail(QCB_EBOUNDS, "project: qubit index exceeds the state's qubits");
      q0[j] = qubits[j] - 1;
    }
  }
  // the Pauli of projection j in host memory (single-qubit mode)
  auto single_pauli = [&](uint32_t j) {
    std::vector<uint64_t> hp(W, 0);
    if (basis & 1u) hp[q0[j] >> 6] |= 1ull << (q0[j] & 63);
    if (basis & 2u) hp[len + (q0[j] >> 6)] |= 1ull << (q0[j] & 63);
    return hp;
  };
  uint32_t* d_q = nullptr;
  uint8_t* d_rand = nullptr;
  int32_t *d_anti = nullptr, *d_res = nullptr, *d_stat = nullptr, *d_rank = nullptr, *d_cout = nullptr;
  uint8_t* d_flags = nullptr;
  uint64_t* d_tmp = nullptr;
  uint8_t* d_tmpph = nullptr;
  const uint32_t tries = k / PROJ_PANEL_MIN + 1;  // by panels: each takes at least PROJ_PANEL_MIN Paulis of the run
  QCB_CUDA(cudaMallocAsync(&d_anti, ((size_t)k + tries) * 4, st));
  QCB_CUDA(cudaMallocAsync(&d_res, (size_t)k * 4, st));
  QCB_CUDA(cudaMallocAsync(&d_stat, 64, st));
  QCB_CUDA(cudaMallocAsync(&d_rank, 4, st));
  QCB_CUDA(cudaMallocAsync(&d_cout, 16, st));
  QCB_CUDA(cudaMallocAsync(&d_flags, std::max<uint32_t>(t->rows, 1), st));
  QCB_CUDA(cudaMallocAsync(&d_tmp, (size_t)t->W * 8 + 16, st));
  QCB_CUDA(cudaMallocAsync(&d_tmpph, 16, st));
  if (qubits) {
    QCB_CUDA(cudaMallocAsync(&d_q, (size_t)k * 4, st));
    QCB_CUDA(cudaMemcpyAsync(d_q, q0.data(), (size_t)k * 4, cudaMemcpyHostToDevice, st));
  }
  if (rand_host) {
    QCB_CUDA(cudaMallocAsync(&d_rand, k, st));
    QCB_CUDA(cudaMemcpyAsync(d_rand, rand_host, k, cudaMemcpyHostToDevice, st));
  }
  int32_t rank = mixed ? *rank_io : 0;
  QCB_CUDA(cudaMemcpyAsync(d_rank, &rank, 4, cudaMemcpyHostToDevice, st));

  // launch shape: the tableau in the cluster's shared memory when it fits
  // (the smallest cluster with at most 128 rows per CTA, or the tuned size),
  // else the rows stay in global memory
  const size_t maxsm = (size_t)device_max_smem_optin();
  uint32_t cs = 0, RB = 0;
  bool use_smem = false;
  for (uint32_t c = 1; c <= 16; c <<= 1) {
    if (g_proj_cs && c != g_proj_cs) continue;
    const uint32_t rb = (t->rows + c - 1) / c;
    if (proj_smem_bytes(rb, W) > maxsm) continue;
    cs = c; RB = rb; use_smem = true;
    if (g_proj_cs || rb <= 128) break;
  }
  const size_t sm = use_smem ? proj_smem_bytes(RB, W) : std::max<size_t>((size_t)2 * W * 8, 1024);
  if (!use_smem) cs = g_proj_cs ? g_proj_cs : 8;
  if (use_smem) {
    QCB_CUDA(cudaFuncSetAttribute(project_smem_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, device_max_smem_optin()));
    if (cs > 8) QCB_CUDA(cudaFuncSetAttribute(project_smem_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  } else {
    QCB_CUDA(cudaFuncSetAttribute(project_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, device_max_smem_optin() - 1024));  // it has static shared memory too
    if (cs > 8) QCB_CUDA(cudaFuncSetAttribute(project_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  }
  // generic Paulis on a Stabilizer / MixedStabilizer tableau that does not
  // fit one cluster's shared memory: the whole GPU (project_grid_kernel)
  const size_t gsm = (size_t)3 * W * 8;
  const bool grid = g_proj_grid != 2 && !qubits && (kind == QCB_STABILIZER || kind == QCB_MIXED_STABILIZER) &&
                    (g_proj_grid == 1 || !use_smem) && gsm <= maxsm;
  uint32_t G = 0;
  uint32_t* d_bar = nullptr;  // [0..1] barrier, [2..4] first anticommuting rows, [5] timeout flag
  if (grid) {
    if (gsm > 48 * 1024)
      QCB_CUDA(allow_max_smem(project_grid_kernel));
    int nb = 0;
    QCB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, project_grid_kernel, PROJ_THREADS, gsm));
    G = (uint32_t)std::max(1, nb) * (uint32_t)std::max(device_sm_count(), 1);
    QCB_CUDA(cudaMallocAsync(&d_bar, 32, st));
  }
  int status = QCB_OK;
  uint32_t j0 = 0;
  std::vector<int32_t> h_anti(k, 0), h_res(k, -1);
  // runs of generic Paulis go by panels (the tuner's choices of the other
  // kernels turn them off).  The first panel's steps are a trial: the other
  // kernels are launched behind it and take the run where it ends at once (a
  // Pauli that commutes with the state), for more Paulis each time before the
  // next trial
  const bool destab = kind == QCB_DESTABILIZER || kind == QCB_MIXED_DESTABILIZER;
  const bool panels = !qubits && phases && len && !g_proj_grid && !g_proj_cs;
  const int skip = !keep_result && (kind == QCB_STABILIZER || (kind == QCB_DESTABILIZER && t->rows / 2 == t->nqubits));
  uint32_t next_try = 0, backoff = PROJ_PANEL_BACKOFF, tried = 0;
  auto after = [&](uint32_t j) {  // the next trial behind a failed one at j, or none
    return k - j >= backoff + PROJ_PANEL_AGAIN ? j + backoff : k;
  };
  if (panels) {
    QCB_CUDA(cudaMemsetAsync(d_anti, 0, ((size_t)k + tries) * 4, st));
    QCB_CUDA(cudaMemsetAsync(d_res, 0xFF, (size_t)k * 4, st));
  }
  while (j0 < k) {
    uint32_t kend = k;
    std::unique_ptr<PanelRun> trial;
    if (panels && k - j0 >= PROJ_PANEL_MIN && j0 >= next_try) {
      int32_t r_now = rank;
      if (mixed && j0) {
        QCB_CUDA(cudaMemcpyAsync(&r_now, d_rank, 4, cudaMemcpyDeviceToHost, st));
        QCB_CUDA(cudaStreamSynchronize(st));
      }
      const uint32_t nr = kind == QCB_STABILIZER ? t->rows : kind == QCB_DESTABILIZER ? t->rows / 2 : (uint32_t)r_now;
      if (nr && nr <= PROJ_PANEL_ROWS) {
        uint32_t* live = (uint32_t*)d_anti + k + std::min(tried++, tries - 1);
        trial = std::make_unique<PanelRun>(st);
        bool none = false;
        if ((status = trial->begin(t, kind, nr, pxzs, pph, d_rand, j0, k, skip, d_anti, d_res, live, &none))) break;
        if (none) trial.reset();
        next_try = after(j0);
        kend = next_try;
      }
    } else if (panels && next_try > j0 && (destab || next_try > j0 + 1)) {
      kend = std::min(k, next_try);
    }
    // The first panels are queued at once.  A run of no more is stored, and the
    // other kernels launched behind it for the case that it fails, with one
    // wait for all; a longer one goes on when its first panels are known.
    int32_t at[2] = {0, 0};  // the trial's state
    auto read_trial = [&]() -> int {
      QCB_CUDA(cudaMemcpyAsync(at, trial->a.state, 8, cudaMemcpyDeviceToHost, st));
      return QCB_OK;
    };
    auto advance = [&]() {  // behind a run that did not fail; where the next may start
      const uint32_t from = j0;
      j0 = (uint32_t)at[1];
      if (j0 - from >= PROJ_PANEL_GOOD) {
        backoff = PROJ_PANEL_BACKOFF;
        next_try = j0 + 1;
      } else {
        next_try = after(j0);
        backoff = std::min<uint32_t>(backoff * 4, 1u << 20);
      }
    };
    const bool whole = trial && !grid && trial->panels() <= PROJ_TRIAL_PANELS;
    if (trial) {
      const uint32_t np = trial->panels();
      if ((status = trial->queue(std::min(np, PROJ_TRIAL_PANELS)))) break;
      if (whole) {
        if ((status = trial->store())) break;
      } else {
        if ((status = read_trial())) break;
        QCB_CUDA(cudaStreamSynchronize(st));
        if (!short_trial(at, j0)) {
          // ended: the steps of the panel after the queued ones are still to be applied
          if ((status = trial->queue(at[0] ? std::min(np, trial->next + 1) : np))) break;
          if ((status = trial->store()) || (status = read_trial())) break;
          QCB_CUDA(cudaStreamSynchronize(st));
          advance();
          continue;
        }
        backoff = std::min<uint32_t>(backoff * 4, 1u << 20);
      }
    }
    ProjArgs a{};
    a.xzs = t->xzs; a.ph = t->phases; a.rows = t->rows; a.n = t->nqubits; a.W = t->W;
    a.kind = kind; a.rank = d_rank; a.paulis = pxzs; a.pph = pph;
    a.j0 = j0; a.k = kend; a.keep_result = keep_result; a.phases = phases;
    a.anticom = d_anti; a.result = d_res; a.status = d_stat; a.flags = d_flags;
    a.qubits = d_q; a.basis = basis; a.rand_ph = d_rand;
    a.trial = whole ? trial->a.state : nullptr;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(cs);
    cfg.blockDim = dim3(PROJ_THREADS);
    cfg.dynamicSmemBytes = sm;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cs;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int32_t htimeout = 0;
    if (grid) {
      QCB_CUDA(cudaMemsetAsync(d_bar, 0, 8, st));
      QCB_CUDA(cudaMemsetAsync(d_bar + 2, 0xFF, 12, st));
      QCB_CUDA(cudaMemsetAsync(d_bar + 5, 0, 4, st));
      QCB_CUDA(cudaMemsetAsync(d_stat, 0xFF, 8, st));
      ProjGridArgs ga{a, d_bar, d_bar + 2, (int32_t*)(d_bar + 5), G > 1 ? g_proj_withhold : 0u};
      void* args[] = {&ga};
      QCB_CUDA(cudaLaunchCooperativeKernel((const void*)project_grid_kernel, dim3(G), dim3(PROJ_THREADS), args, gsm,
                                           st));
    } else if (use_smem) {
      ProjSmemArgs pa{a, RB};
      QCB_CUDA(cudaLaunchKernelEx(&cfg, project_smem_kernel, pa));
    } else {
      QCB_CUDA(cudaLaunchKernelEx(&cfg, project_kernel, a));
    }
    QCB_LAUNCHED();
    int32_t hs[2];
    QCB_CUDA(cudaMemcpyAsync(hs, d_stat, 8, cudaMemcpyDeviceToHost, st));
    if (grid) QCB_CUDA(cudaMemcpyAsync(&htimeout, d_bar + 5, 4, cudaMemcpyDeviceToHost, st));
    if (whole && (status = read_trial())) break;
    QCB_CUDA(cudaStreamSynchronize(st));
    if (whole) {
      if (!short_trial(at, j0)) {
        advance();
        continue;
      }
      backoff = std::min<uint32_t>(backoff * 4, 1u << 20);
    }
    if (htimeout) {
      status = fail(QCB_ETIMEOUT, "project!: a grid barrier wait of the whole-GPU kernel expired");
      break;
    }
    if (hs[0] == PST_OK) {
      j0 = kend;
      continue;
    }
    const uint32_t j = (uint32_t)hs[1];
    if (hs[0] == PST_BADSTRUCT) {
      status = fail(QCB_EBADSTRUCT,
                    "`Destabilizer` can not efficiently (faster than n^3) detect whether you are projecting on a "
                    "stabilized or a logical operator. Switch to one of the `Mixed*` data structures.");
      if (n_done) *n_done = j;
      j0 = k;
      break;
    }
    // PST_NEED_CANON: canonicalize the stabilizer view, then generate!
    int32_t r_now = rank;
    if (kind == QCB_MIXED_STABILIZER) QCB_CUDA(cudaMemcpy(&r_now, d_rank, 4, cudaMemcpyDeviceToHost));
    const uint32_t nr = kind == QCB_STABILIZER ? t->rows : (uint32_t)r_now;
    if (int s = canonicalize_view(t->xzs, t->phases, nr, t->nqubits, t->W, phases, d_cout, st, true)) { status = s; break; }
    std::vector<uint64_t> hp;
    const uint8_t zero = 0;
    if (qubits) {
      hp = single_pauli(j);
      QCB_CUDA(cudaMemcpyAsync(d_tmp, hp.data(), (size_t)W * 8, cudaMemcpyHostToDevice, st));
      QCB_CUDA(cudaMemcpyAsync(d_tmpph, &zero, 1, cudaMemcpyHostToDevice, st));
    } else {
      QCB_CUDA(cudaMemcpyAsync(d_tmp, pxzs + (size_t)j * W, (size_t)W * 8, cudaMemcpyDeviceToDevice, st));
      QCB_CUDA(cudaMemcpyAsync(d_tmpph, pph + j, 1, cudaMemcpyDeviceToDevice, st));
    }
    if (int s = generate_dev(d_tmp, d_tmpph, t->xzs, t->phases, nr, t->W, phases, d_cout + 2, nullptr, 0,
                             (uint32_t*)(d_cout + 3), st)) { status = s; break; }
    int32_t cout[4];
    uint8_t gph = 0;
    QCB_CUDA(cudaMemcpyAsync(cout, d_cout, 16, cudaMemcpyDeviceToHost, st));
    QCB_CUDA(cudaMemcpyAsync(&gph, d_tmpph, 1, cudaMemcpyDeviceToHost, st));
    QCB_CUDA(cudaStreamSynchronize(st));
    int32_t anti = 0, res = -1;
    if (cout[2]) {
      res = gph;
    } else {
      anti = cout[1] + 1;
      if (kind == QCB_MIXED_STABILIZER && anti == r_now + 1) {
        // ms.tab[rank+1] = pauli; rank += 1  (src/project_trace_reset.jl:310-317)
        if ((uint32_t)r_now >= t->rows) { status = fail(QCB_EBOUNDS, "MixedStabilizer tableau is full"); break; }
        if (qubits) {
          QCB_CUDA(cudaMemcpyAsync(t->xzs + (size_t)r_now * W, hp.data(), (size_t)W * 8, cudaMemcpyHostToDevice, st));
          QCB_CUDA(cudaMemcpyAsync(t->phases + r_now, &zero, 1, cudaMemcpyHostToDevice, st));
        } else {
          QCB_CUDA(cudaMemcpyAsync(t->xzs + (size_t)r_now * W, pxzs + (size_t)j * W, (size_t)W * 8,
                                   cudaMemcpyDeviceToDevice, st));
          QCB_CUDA(cudaMemcpyAsync(t->phases + r_now, pph + j, 1, cudaMemcpyDeviceToDevice, st));
        }
        r_now += 1;
        QCB_CUDA(cudaMemcpyAsync(d_rank, &r_now, 4, cudaMemcpyHostToDevice, st));
      }
      if (rand_host && anti > 0) {
        // projectrand!: the new stabilizer row anti gets a random sign
        if ((uint32_t)anti > t->rows) { status = fail(QCB_EBOUNDS, "projectrand!: no stabilizer row to randomize"); break; }
        QCB_CUDA(cudaMemcpyAsync(t->phases + (anti - 1), rand_host + j, 1, cudaMemcpyHostToDevice, st));
        res = rand_host[j];
      }
    }
    QCB_CUDA(cudaMemcpyAsync(d_anti + j, &anti, 4, cudaMemcpyHostToDevice, st));
    QCB_CUDA(cudaMemcpyAsync(d_res + j, &res, 4, cudaMemcpyHostToDevice, st));
    QCB_CUDA(cudaStreamSynchronize(st));
    j0 = j + 1;
  }
  if (status == QCB_OK || status == QCB_EBADSTRUCT) {
    QCB_CUDA(cudaMemcpyAsync(h_anti.data(), d_anti, (size_t)k * 4, cudaMemcpyDeviceToHost, st));
    QCB_CUDA(cudaMemcpyAsync(h_res.data(), d_res, (size_t)k * 4, cudaMemcpyDeviceToHost, st));
    if (mixed) QCB_CUDA(cudaMemcpyAsync(&rank, d_rank, 4, cudaMemcpyDeviceToHost, st));
    QCB_CUDA(cudaStreamSynchronize(st));
    std::copy(h_anti.begin(), h_anti.end(), anticom);
    std::copy(h_res.begin(), h_res.end(), result);
    if (mixed) *rank_io = rank;
    if (status == QCB_OK && n_done) *n_done = k;
  }
  cudaFreeAsync(d_anti, st); cudaFreeAsync(d_res, st); cudaFreeAsync(d_stat, st);
  cudaFreeAsync(d_rank, st); cudaFreeAsync(d_cout, st); cudaFreeAsync(d_flags, st);
  cudaFreeAsync(d_tmp, st); cudaFreeAsync(d_tmpph, st);
  if (d_q) cudaFreeAsync(d_q, st);
  if (d_rand) cudaFreeAsync(d_rand, st);
  if (d_bar) cudaFreeAsync(d_bar, st);
  cudaStreamSynchronize(st);
  return status;
}

int qcb_project(qcb_tableau* t, int kind, int32_t* rank_io, const qcb_tableau* paulis, int keep_result,
                int phases, int32_t* anticom, int32_t* result, uint32_t* n_done, void* stream) {
  if (!t || !paulis) return fail(QCB_EARG, "null argument");
  if (paulis->nqubits != t->nqubits) return fail(QCB_EDIM, "project!: the Pauli and the state act on different numbers of qubits");
  return project_impl(t, kind, rank_io, paulis->xzs, paulis->phases, nullptr, 0, paulis->rows, keep_result, phases,
                      nullptr, anticom, result, n_done, stream);
}

int qcb_project_qubit(qcb_tableau* t, int kind, int32_t* rank_io, uint32_t basis, const uint32_t* qubits, size_t k,
                      int keep_result, int phases, int32_t* anticom, int32_t* result, uint32_t* n_done,
                      void* stream) {
  if (basis < 1 || basis > 3) return fail(QCB_EARG, "project: basis is 1 (X), 2 (Z) or 3 (Y)");
  if (k && !qubits) return fail(QCB_EARG, "null argument");
  if (k > 0xFFFFFFFFull) return fail(QCB_EARG, "too many projections");
  return project_impl(t, kind, rank_io, nullptr, nullptr, qubits, basis, (uint32_t)k, keep_result, phases, nullptr,
                      anticom, result, n_done, stream);
}

int qcb_projectrand(qcb_tableau* t, int kind, int32_t* rank_io, const qcb_tableau* paulis, uint32_t basis,
                    const uint32_t* qubits, size_t k, const uint8_t* rand_phases, int32_t* anticom, int32_t* result,
                    uint32_t* n_done, void* stream) {
  if (!rand_phases) return fail(QCB_EARG, "null argument");
  if (paulis) {
    if (paulis->nqubits != t->nqubits) return fail(QCB_EDIM, "project!: the Pauli and the state act on different numbers of qubits");
    for (uint32_t j = 0; j < paulis->rows; j++)
      if (rand_phases[j] != 0 && rand_phases[j] != 2) return fail(QCB_EARG, "projectrand!: random phases are 0 or 2");
    return project_impl(t, kind, rank_io, paulis->xzs, paulis->phases, nullptr, 0, paulis->rows, 1, 1, rand_phases,
                        anticom, result, n_done, stream);
  }
  if (basis < 1 || basis > 3) return fail(QCB_EARG, "project: basis is 1 (X), 2 (Z) or 3 (Y)");
  if (k && !qubits) return fail(QCB_EARG, "null argument");
  for (size_t j = 0; j < k; j++)
    if (rand_phases[j] != 0 && rand_phases[j] != 2) return fail(QCB_EARG, "projectrand!: random phases are 0 or 2");
  return project_impl(t, kind, rank_io, nullptr, nullptr, qubits, basis, (uint32_t)k, 1, 1, rand_phases, anticom,
                      result, n_done, stream);
}

}  // extern "C"

namespace qcb {
void set_project_cluster(uint32_t cs) { g_proj_cs = cs; }
void set_project_grid(uint32_t v) { g_proj_grid = v; }
void set_project_withhold(uint32_t v) { g_proj_withhold = v; }
}
