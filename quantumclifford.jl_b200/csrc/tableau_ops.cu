// tableau_ops.cu -- row algebra on device tableaux.
//
//  mul_left!  (src/mul_leftright.jl:75-142, 171-229): r <- l * r with the
//             phase of the product.  The phase is the sum over bit lanes of
//             independent mod-4 counters (cnt1 = low bit, cnt2 = high bit),
//             so any partition of the words into threads sums exactly:
//             phase = (sum popc(cnt1) + 2 * sum popc(cnt2)) mod 4.
//  prodphase / comm (src/QuantumClifford.jl:723-859).
//  symbolic gates with phases (src/symbolic_cliffords.jl:62-74, 293-316).
//  dense apply! (src/dense_cliffords.jl:135-169).
#include <algorithm>
#include <mutex>

#include "qcb_internal.h"

namespace qcb {

// Stim phase-counter step on one word pair (src/mul_leftright.jl:90-96).
template <class T>
__device__ __forceinline__ void mul_step(T x1, T z1, T& x2, T& z2, uint64_t& c1, uint64_t& c2) {
  const uint64_t nx = x1 ^ x2, nz = z1 ^ z2;
  const uint64_t x1z2 = (uint64_t)x1 & (uint64_t)z2;
  const uint64_t anti = ((uint64_t)x2 & (uint64_t)z1) ^ x1z2;
  c2 ^= (c1 ^ nx ^ nz ^ x1z2) & anti;
  c1 ^= anti;
  x2 = (T)nx;
  z2 = (T)nz;
}

__device__ __forceinline__ uint32_t cnt_phase(uint64_t c1, uint64_t c2) {
  return (uint32_t)(__popcll(c1) + 2 * __popcll(c2));
}

// mul_right!(l, r) runs the word steps of mul_left!(l <- r * l) and adds
// twice the anticommutation count (src/mul_leftright.jl:128-131): phase
// (rcnt1 + 2 rcnt2) + 2 rcnt1, i.e. 3 popc(cnt1) + 2 popc(cnt2) per lane.
template <bool RIGHT>
__device__ __forceinline__ uint32_t lane_phase(uint64_t c1, uint64_t c2) {
  return RIGHT ? (uint32_t)(3 * __popcll(c1) + 2 * __popcll(c2)) : cnt_phase(c1, c2);
}

// Grid-stride mul_left! over two long Paulis.  VEC = 2 uses 128-bit loads
// (needs len even and 16-byte aligned halves).  Each block adds its phase
// sum (mod 4) into acc[0] and counts itself done in acc[1]; the last block
// to finish writes r.phase <- (s + r.phase + l.phase) & 3
// (src/mul_leftright.jl:140) and clears both, so one launch does the call.
template <int VEC, bool PH, bool RIGHT = false>
__global__ void __launch_bounds__(256) mul_left_long_kernel(uint64_t* __restrict__ r,
                                                            const uint64_t* __restrict__ l,
                                                            uint64_t len, uint32_t* acc,
                                                            uint8_t* r_phase, const uint8_t* l_phase) {
  uint64_t c1a = 0, c2a = 0, c1b = 0, c2b = 0;
  const uint64_t nvec = len / VEC;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nvec; i += stride) {
    if (VEC == 2) {
      const ulonglong2 lx = __ldcs((const ulonglong2*)l + i);
      const ulonglong2 lz = __ldcs((const ulonglong2*)(l + len) + i);
      ulonglong2 rx = __ldcs((const ulonglong2*)r + i);
      ulonglong2 rz = __ldcs((const ulonglong2*)(r + len) + i);
      if (PH) {
        mul_step(lx.x, lz.x, rx.x, rz.x, c1a, c2a);
        mul_step(lx.y, lz.y, rx.y, rz.y, c1b, c2b);
      } else {
        rx.x ^= lx.x; rx.y ^= lx.y; rz.x ^= lz.x; rz.y ^= lz.y;
      }
      __stcs((ulonglong2*)r + i, rx);
      __stcs((ulonglong2*)(r + len) + i, rz);
    } else {
      const uint64_t lx = __ldcs(l + i), lz = __ldcs(l + len + i);
      uint64_t rx = __ldcs(r + i), rz = __ldcs(r + len + i);
      if (PH) mul_step(lx, lz, rx, rz, c1a, c2a);
      else { rx ^= lx; rz ^= lz; }
      __stcs(r + i, rx);
      __stcs(r + len + i, rz);
    }
  }
  if (!PH) return;
  uint32_t v = (lane_phase<RIGHT>(c1a, c2a) + lane_phase<RIGHT>(c1b, c2b)) & 3u;
  v = __reduce_add_sync(0xFFFFFFFFu, v) & 3u;
  __shared__ uint32_t wsum[32];
  const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) wsum[wid] = v;
  __syncthreads();
  if (wid == 0) {
    uint32_t s = lane < (blockDim.x >> 5) ? wsum[lane] : 0u;
    s = __reduce_add_sync(0xFFFFFFFFu, s) & 3u;
    if (lane == 0) {
      if (s) atomicAdd(acc, s);
      __threadfence();
      if (atomicAdd(acc + 1, 1u) == gridDim.x - 1) {  // the last block
        __threadfence();
        const uint32_t tot = atomicExch(acc, 0u) & 3u;
        atomicExch(acc + 1, 0u);
        r_phase[0] = (uint8_t)((tot + r_phase[0] + l_phase[0]) & 3u);
      }
    }
  }
}

// r.phase <- (s + r.phase + l.phase) & 3 (src/mul_leftright.jl:140); clears acc.
__global__ void mul_left_finish_kernel(uint8_t* r_phase, const uint8_t* l_phase, uint32_t* acc,
                                       int phases) {
  const uint32_t s = acc[0] & 3u;
  if (phases) r_phase[0] = (uint8_t)((s + r_phase[0] + l_phase[0]) & 3u);
  acc[0] = 0;
}

// Row-level ops: one warp per target row; lanes stride over the words.
template <bool PH>
__device__ __forceinline__ uint32_t warp_mul_left_row(uint64_t* r, const uint64_t* l, uint32_t len,
                                                      uint32_t lane) {
  uint64_t c1 = 0, c2 = 0;
  for (uint32_t w = lane; w < len; w += 32) {
    uint64_t rx = r[w], rz = r[len + w];
    const uint64_t lx = l[w], lz = l[len + w];
    if (PH) mul_step(lx, lz, rx, rz, c1, c2);
    else { rx ^= lx; rz ^= lz; }
    r[w] = rx;
    r[len + w] = rz;
  }
  if (!PH) return 0;
  return __reduce_add_sync(0xFFFFFFFFu, cnt_phase(c1, c2) & 3u) & 3u;
}

// mul_left!(s::Tableau, p::PauliOperator) (src/mul_leftright.jl:221-227).
__global__ void mul_left_tab_pauli_kernel(uint64_t* xzs, uint8_t* ph, uint32_t rows, uint32_t W,
                                          const uint64_t* p, const uint8_t* pph, int phases) {
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= rows) return;
  uint64_t* r = xzs + (uint64_t)warp * W;
  if (phases) {
    const uint32_t s = warp_mul_left_row<true>(r, p, W / 2, lane);
    if (lane == 0) ph[warp] = (uint8_t)((s + ph[warp] + pph[0]) & 3u);
  } else {
    warp_mul_left_row<false>(r, p, W / 2, lane);
  }
}

// mul_left!(s::Tableau, m, i) (src/mul_leftright.jl:177-181), 0-based rows.
__global__ void mul_left_row_kernel(uint64_t* xzs, uint8_t* ph, uint32_t W, uint32_t m, uint32_t i,
                                    int phases) {
  const uint32_t lane = threadIdx.x & 31;
  if (threadIdx.x >= 32) return;
  uint64_t* r = xzs + (uint64_t)m * W;
  const uint64_t* l = xzs + (uint64_t)i * W;
  if (phases) {
    const uint32_t s = warp_mul_left_row<true>(r, l, W / 2, lane);
    if (lane == 0) ph[m] = (uint8_t)((s + ph[m] + ph[i]) & 3u);
  } else {
    warp_mul_left_row<false>(r, l, W / 2, lane);
  }
}

// The mul_left!/mul_right! family on rows (src/mul_leftright.jl:137-245,
// ext/QuantumCliffordKAExt/mul_leftright.jl:101-460): one warp per target row
// a = s_row + k, source row b = t_row + k * t_step; the added phase is
// add_ph[b] (t's phases, or s's for the reference's cross-tableau methods).
template <bool RIGHT, bool PH>
__global__ void __launch_bounds__(256) mul_rows_kernel(uint64_t* s_xz, uint8_t* s_ph, uint32_t s_row,
                                                       uint32_t count, const uint64_t* t_xz, uint32_t t_row,
                                                       uint32_t t_step, uint32_t W, const uint8_t* add_ph) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  const uint32_t len = W / 2;
  for (uint32_t k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; k < count; k += nwarps) {
    const uint32_t a = s_row + k, b = t_row + k * t_step;
    uint64_t* r = s_xz + (uint64_t)a * W;
    const uint64_t* l = t_xz + (uint64_t)b * W;
    uint64_t c1 = 0, c2 = 0;
    for (uint32_t w = lane; w < len; w += 32) {
      uint64_t rx = r[w], rz = r[len + w];
      const uint64_t lx = l[w], lz = l[len + w];
      if (PH) mul_step(lx, lz, rx, rz, c1, c2);
      else { rx ^= lx; rz ^= lz; }
      r[w] = rx;
      r[len + w] = rz;
    }
    if (PH) {
      const uint32_t v = __reduce_add_sync(0xFFFFFFFFu, lane_phase<RIGHT>(c1, c2) & 3u) & 3u;
      if (lane == 0) s_ph[a] = (uint8_t)((v + s_ph[a] + add_ph[b]) & 3u);
    }
  }
}

// prodphase (src/QuantumClifford.jl:723-733) and comm (:791-798) of two rows.
__global__ void prodphase_comm_kernel(const uint64_t* l, uint8_t lph, const uint64_t* r, uint8_t rph,
                                      uint32_t len, int what, uint8_t* out) {
  const uint32_t lane = threadIdx.x & 31;
  if (threadIdx.x >= 32) return;
  int32_t acc = 0;
  uint64_t cm = 0;
  for (uint32_t w = lane; w < len; w += 32) {
    const uint64_t x1 = l[w], x2 = r[w], z1 = l[len + w], z2 = r[len + w];
    acc += __popcll((~z2 & x2 & ~x1 & z1) | (z2 & ~x2 & x1 & z1) | (z2 & x2 & x1 & ~z1));
    acc -= __popcll((z2 & x2 & ~x1 & z1) | (~z2 & x2 & x1 & z1) | (z2 & ~x2 & x1 & ~z1));
    cm ^= (z1 & x2) ^ (x1 & z2);
  }
  const int32_t tot = __reduce_add_sync(0xFFFFFFFFu, acc);
  const uint32_t par = __reduce_add_sync(0xFFFFFFFFu, (uint32_t)__popcll(cm)) & 1u;
  if (lane == 0) {
    if (what == 0) out[0] = (uint8_t)(((uint32_t)tot + lph + rph) & 3u);
    else out[0] = (uint8_t)par;
  }
}

// ---------------------------------------------------------- symbolic gates
// Bit-sliced truth tables with the phase flag (src/symbolic_cliffords.jl
// :105-118 and :358-395).
template <class T>
__device__ __forceinline__ T g1(uint32_t op, T& x, T& z) {
  const T X = x, Z = z;
  if ((op & 0xFFu) == QCB_OP_SQO) {
    // SingleQubitOperator (src/symbolic_cliffords.jl:178-206), flags in bits
    // 8..13: +2 for px & x, for pz & z, and for x & z when the map sends Y to
    // minus the product of the images of X and Z
    const uint32_t f = op >> 8;
    const bool bxx = f & 1u, bxz = f & 2u, bzx = f & 4u, bzz = f & 8u;
    const T xx = (T)0 - (T)bxx, xz = (T)0 - (T)bxz;
    const T zx = (T)0 - (T)bzx, zz = (T)0 - (T)bzz;
    const bool anticom = (!bzz && bxz && !bxx && bzx) || (bzz && !bxz && bxx && bzx) || (bzz && bxz && bxx && !bzx);
    x = (X & xx) ^ (Z & zx);
    z = (X & xz) ^ (Z & zz);
    return ((f & 16u) ? X : (T)0) ^ ((f & 32u) ? Z : (T)0) ^ (anticom ? (X & Z) : (T)0);
  }
  switch (op) {
    case QCB_OP_H: x = Z; z = X; return X & Z;
    case QCB_OP_HXY: z = X ^ Z; return ~X & Z;
    case QCB_OP_HYZ: x = X ^ Z; return X & ~Z;
    case QCB_OP_S: z = X ^ Z; return X & Z;
    case QCB_OP_SDAG: z = X ^ Z; return X & ~Z;
    case QCB_OP_X: return Z;
    case QCB_OP_Y: return X ^ Z;
    case QCB_OP_Z: return X;
    case QCB_OP_SQRTX: x = X ^ Z; return ~X & Z;
    case QCB_OP_INVSQRTX: x = X ^ Z; return X & Z;
    case QCB_OP_SQRTY: x = Z; z = X; return X & ~Z;
    case QCB_OP_INVSQRTY: x = Z; z = X; return Z & ~X;
    case QCB_OP_CXYZ: x = X ^ Z; z = X; return 0;
    case QCB_OP_CZYX: x = Z; z = X ^ Z; return 0;
    default: return 0;
  }
}

template <class T>
__device__ __forceinline__ T g2(uint32_t op, T& x1, T& z1, T& x2, T& z2) {
  const T a = x1, b = z1, c = x2, d = z2;
  switch (op) {
    case QCB_OP_SWAP: x1 = c; z1 = d; x2 = a; z2 = b; return 0;
    case QCB_OP_CNOT: z1 = b ^ d; x2 = c ^ a; return (a & b & c & d) | (a & d & ~(b | c));
    case QCB_OP_CPHASE: z1 = b ^ c; z2 = d ^ a; return (a & b & c & ~d) | (a & ~b & c & d);
    case QCB_OP_ZCX: z1 = b ^ d; x2 = c ^ a; return (a & d) & ~(b ^ c);
    case QCB_OP_ZCY: z1 = c ^ b ^ d; x2 = c ^ a; z2 = d ^ a; return a & (c ^ b) & (c ^ d);
    case QCB_OP_ZCZ: z1 = b ^ c; z2 = d ^ a; return (b ^ d) & (a & c);
    case QCB_OP_XCX: x1 = d ^ a; x2 = c ^ b; return (b & d) & (a ^ c);
    case QCB_OP_XCY: x1 = a ^ c ^ d; x2 = b ^ c; z2 = d ^ b; return b & (c ^ d) & ~(c ^ a);
    case QCB_OP_XCZ: x1 = a ^ c; z2 = d ^ b; return (c & b) & ~(a ^ d);
    case QCB_OP_YCX: x1 = a ^ d; z1 = d ^ b; x2 = a ^ b ^ c; return d & (a ^ b) & ~(c ^ a);
    case QCB_OP_YCY:
      x1 = a ^ d ^ c; z1 = b ^ c ^ d; x2 = a ^ c ^ b; z2 = a ^ b ^ d;
      return (a & ~b & ~c & d) | (~a & b & c & ~d);
    case QCB_OP_YCZ: x1 = a ^ c; z1 = c ^ b; z2 = d ^ a ^ b; return c & (a ^ b) & (d ^ a);
    case QCB_OP_SWAPCX:
      x1 = c; z1 = d ^ b; x2 = c ^ a; z2 = b;
      return (a & b & c & d) | (~a & b & c & ~d);
    case QCB_OP_INVSWAPCX:
      x1 = c ^ a; z1 = d; x2 = a; z2 = d ^ b;
      return (a & b & c & d) | (a & ~b & ~c & d);
    case QCB_OP_ISWAP:
      x1 = c; z1 = a ^ d ^ c; x2 = a; z2 = a ^ c ^ b;
      return (a & b & ~c) | (~a & c & d);
    case QCB_OP_INVISWAP:
      x1 = c; z1 = a ^ d ^ c; x2 = a; z2 = a ^ c ^ b;
      return (a & ~b & ~c) | (~a & c & ~d);
    case QCB_OP_CZSWAP:
      x1 = c; z1 = d ^ a; x2 = a; z2 = c ^ b;
      return (a & ~b & c & d) | (a & b & c & ~d);
    case QCB_OP_CXSWAP:
      x1 = c ^ a; z1 = d; x2 = a; z2 = d ^ b;
      return (a & ~b & ~c & d) | (a & b & c & d);
    case QCB_OP_ZCRY:
      z1 = a ^ b ^ c ^ d; x2 = a ^ c; z2 = a ^ d;
      return (a & ~b & c) | (a & ~b & ~d) | (a & c & ~d);
    case QCB_OP_INVZCRY:
      z1 = a ^ b ^ c ^ d; x2 = a ^ c; z2 = a ^ d;
      return (a & b & ~c) | (a & b & d) | (a & ~c & d);
    case QCB_OP_SQRTZZ:
      z1 = a ^ c ^ b; z2 = a ^ d ^ c;
      return (a & b & ~c) | (~a & c & d);
    case QCB_OP_INVSQRTZZ:
      z1 = a ^ c ^ b; z2 = a ^ d ^ c;
      return (a & ~b & ~c) | (~a & c & ~d);
    case QCB_OP_SQRTXX:
      x1 = b ^ d ^ a; x2 = b ^ c ^ d;
      return (~a & b & ~d) | (~b & ~c & d);
    case QCB_OP_INVSQRTXX:
      x1 = b ^ d ^ a; x2 = b ^ c ^ d;
      return (a & b & ~d) | (~b & c & d);
    case QCB_OP_SQRTYY:
      x1 = b ^ c ^ d; z1 = a ^ d ^ c; x2 = a ^ b ^ d; z2 = a ^ c ^ b;
      return (~a & ~b & c & ~d) | (a & ~b & ~c & ~d) | (a & ~b & c & d) | (a & b & c & ~d);
    case QCB_OP_INVSQRTYY:
      x1 = b ^ c ^ d; z1 = a ^ d ^ c; x2 = a ^ b ^ d; z2 = a ^ c ^ b;
      return (a & b & ~c & d) | (~a & b & c & d) | (~a & b & ~c & ~d) | (~a & ~b & ~c & d);
    default: return 0;
  }
}

struct GateOp {
  uint32_t op, q1, q2, pad;
};
// Gates passed to one launch by value (kernel parameter space, 2 KB), so a
// gate list needs no device allocation, no copy and no synchronisation.
constexpr uint32_t GATE_BATCH = 128;
struct GateBatch {
  GateOp op[GATE_BATCH];
};

// Thread per row; the batch's gates are applied to that row in order.  The
// launch may be a programmatic dependent of the launch before it on the
// stream: the dependents of this one are released at once, and the rows are
// touched only after griddepcontrol.wait (the predecessor has completed and
// its writes are visible; a no-op for a plain launch).
__global__ void apply_gates_kernel(uint64_t* xzs, uint8_t* ph, uint32_t rows, uint32_t W,
                                   const __grid_constant__ GateBatch ops, uint32_t nops, int phases) {
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= rows) return;
  uint64_t* row = xzs + (uint64_t)r * W;
  const uint32_t len = W / 2;
  uint32_t p = ph[r];
  for (uint32_t k = 0; k < nops; k++) {
    const GateOp g = ops.op[k];
    if ((g.op & 0xFFu) < QCB_OP_CNOT) {  // SingleQubitOperator carries flags above bit 8
      const uint32_t q = g.q1, w = q >> 6, s = q & 63;
      uint64_t x = (row[w] >> s) & 1, z = (row[len + w] >> s) & 1;
      const uint64_t f = g1(g.op, x, z) & 1;
      row[w] = (row[w] & ~(1ull << s)) | ((x & 1) << s);
      row[len + w] = (row[len + w] & ~(1ull << s)) | ((z & 1) << s);
      if (phases && f) p = (p + 2) & 3;
    } else {
      const uint32_t w1 = g.q1 >> 6, s1 = g.q1 & 63, w2 = g.q2 >> 6, s2 = g.q2 & 63;
      uint64_t x1 = (row[w1] >> s1) & 1, z1 = (row[len + w1] >> s1) & 1;
      uint64_t x2 = (row[w2] >> s2) & 1, z2 = (row[len + w2] >> s2) & 1;
      const uint64_t f = g2(g.op, x1, z1, x2, z2) & 1;
      row[w1] = (row[w1] & ~(1ull << s1)) | ((x1 & 1) << s1);
      row[len + w1] = (row[len + w1] & ~(1ull << s1)) | ((z1 & 1) << s1);
      row[w2] = (row[w2] & ~(1ull << s2)) | ((x2 & 1) << s2);
      row[len + w2] = (row[len + w2] & ~(1ull << s2)) | ((z2 & 1) << s2);
      if (phases && f) p = (p + 2) & 3;
    }
  }
  ph[r] = (uint8_t)p;
}

// Gate lists bit-sliced over rows (apply_layers_kernel).  A CTA takes 32 rows
// and keeps them transposed in shared memory: one word holds the x bits of a
// qubit in those rows, one its z bits, so a gate is a few 32-bit operations, gates on different qubits run on different threads, and a phase
// flip is the XOR of the gates' flag words in any order.  The host sorts the
// list into levels (a gate's level is one past the last level of a gate before
// it on one of its qubits: levels hold disjoint qubits, and every qubit sees
// its gates in list order); one barrier orders two levels.  The list comes by
// value (kernel parameters, up to 32 KB): no allocation, no copy, nothing that
// a graph capture of the call would have to keep alive.  Bound by a level's
// latency (the parameter reads, the words, a barrier: 0.3-0.5 us) and, for few
// gates, by the transposes.  400 gates on a 2000 x 1000-qubit tableau: 7.1 us;
// a circuit of 2300 gates on 1000 x 500 qubits 11 us, with one row per thread
// (every gate a read and a write of global words) 1.5 ms.
//  list: per level a header (the level's gate count), then its gates
//  (opcode and flags | q1 << 16 | q2 << 40, 0-based qubits below 2^24).
template <uint32_t CAP>
struct LayerList {
  uint64_t e[CAP];
};
constexpr uint32_t LAYER_CAP_S = 480, LAYER_CAP_L = 4032;  // entries of a launch: 4 KB and 32 KB of parameters
constexpr uint32_t LAYER_SLICE = 32;                       // rows of a CTA

// 32 x 32 bits, lane i holding row i: afterwards lane i holds column i.  Round
// j swaps the off-diagonal j x j blocks with the lane j away: keep the words'
// own blocks (mask) and take the partner's, rotated into place.
struct WarpTranspose {
  uint32_t keep[5], rot[5];
  __device__ __forceinline__ explicit WarpTranspose(uint32_t lane) {
    const uint32_t m[5] = {0x0000FFFFu, 0x00FF00FFu, 0x0F0F0F0Fu, 0x33333333u, 0x55555555u};
#pragma unroll
    for (uint32_t k = 0; k < 5; k++) {
      const bool up = lane & (16u >> k);
      keep[k] = up ? ~m[k] : m[k];
      rot[k] = up ? 32u - (16u >> k) : 16u >> k;
    }
  }
  __device__ __forceinline__ uint32_t operator()(uint32_t v) const {
#pragma unroll
    for (uint32_t k = 0; k < 5; k++) {
      const uint32_t o = __shfl_xor_sync(0xFFFFFFFFu, v, 16u >> k);
      v = (v & keep[k]) | (__funnelshift_l(o, o, rot[k]) & ~keep[k]);
    }
    return v;
  }
};

// The slice [32 rows][2 W words of 32 bits] at an odd row stride; a column of
// words (word w of the 32 rows) is transposed in place, which leaves qubit q's
// x word at row q % 32, word q / 32, and its z word W further on.
template <uint32_t CAP>
__global__ void __launch_bounds__(512) apply_layers_kernel(uint64_t* xzs, uint8_t* ph, uint32_t rows, uint32_t W,
                                                           const __grid_constant__ LayerList<CAP> list,
                                                           uint32_t nent, int phases) {
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  extern __shared__ __align__(16) uint32_t sl[];
  __shared__ uint32_t flip;
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
  const uint32_t r0 = blockIdx.x * LAYER_SLICE, nr = min(LAYER_SLICE, rows - r0);
  const uint32_t words = 2 * W, ST = words + 1;  // 32-bit words of a row, their stride
  uint32_t* base = (uint32_t*)(xzs + (uint64_t)r0 * W);
  const WarpTranspose transpose(lane);
  if (tid == 0) flip = 0;
  for (uint32_t r = warp; r < LAYER_SLICE; r += nw)
#pragma unroll 4
    for (uint32_t w = lane; w < words; w += 32) sl[r * ST + w] = r < nr ? base[(uint64_t)r * words + w] : 0u;
  __syncthreads();
#pragma unroll 2
  for (uint32_t w = warp; w < words; w += nw) sl[lane * ST + w] = transpose(sl[lane * ST + w]);
  __syncthreads();
  uint32_t f = 0;
#pragma unroll 1
  for (uint32_t k = 0; k < nent;) {
    const uint32_t cnt = (uint32_t)list.e[k++];
#pragma unroll 1
    for (uint32_t g = tid; g < cnt; g += blockDim.x) {
      const uint64_t e = list.e[k + g];
      const uint32_t op = (uint32_t)e & 0xFFFFu, q1 = (uint32_t)(e >> 16) & 0xFFFFFFu, q2 = (uint32_t)(e >> 40);
      uint32_t* a = sl + (q1 & 31) * ST + (q1 >> 5);
      uint32_t x1 = a[0], z1 = a[W];
      if ((op & 0xFFu) < QCB_OP_CNOT) {
        f ^= g1<uint32_t>(op, x1, z1);
      } else {
        uint32_t* b = sl + (q2 & 31) * ST + (q2 >> 5);
        uint32_t x2 = b[0], z2 = b[W];
        f ^= g2<uint32_t>(op, x1, z1, x2, z2);
        b[0] = x2;
        b[W] = z2;
      }
      a[0] = x1;
      a[W] = z1;
    }
    k += cnt;
    __syncthreads();
  }
  f = __reduce_xor_sync(0xFFFFFFFFu, f);
  if (lane == 0 && f) atomicXor(&flip, f);
#pragma unroll 2
  for (uint32_t w = warp; w < words; w += nw) sl[lane * ST + w] = transpose(sl[lane * ST + w]);
  __syncthreads();
  for (uint32_t r = warp; r < nr; r += nw)
    for (uint32_t w = lane; w < words; w += 32) base[(uint64_t)r * words + w] = sl[r * ST + w];
  if (phases && warp == 0 && lane < nr && ((flip >> lane) & 1u)) ph[r0 + lane] = (uint8_t)((ph[r0 + lane] + 2u) & 3u);
}

// ---------------------------------------------------------- dense apply!
// Tableaux of few qubits (one word per half, see dense_tables_pay), a warp
// per state row: the ordered product over qubits of the Clifford's images
// (src/dense_cliffords.jl:152-169) in registers; the phase counters run across
// all the multiplications (each adds +-1 per anticommuting lane, independent
// of the current counter value), so one reduction gives the exact total.
__global__ void __launch_bounds__(256) apply_dense_kernel(uint64_t* xzs, uint8_t* ph, uint32_t rows, uint32_t W,
                                                          uint32_t n, const uint64_t* __restrict__ c,
                                                          const uint8_t* __restrict__ cph, int phases) {
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= rows) return;
  uint64_t bx = 0, bz = 0, c1 = 0, c2 = 0;
  uint64_t* row = xzs + (uint64_t)warp * W;
  const uint64_t xw = W ? row[0] : 0ull, zw = W ? row[1] : 0ull;  // broadcast loads
  uint32_t extra = 0;  // sum of Clifford-row phases and -1 corrections (mod 4)
  uint64_t both = xw | zw;
  while (both) {
    const uint32_t q = __ffsll((long long)both) - 1;
    both &= both - 1;
    if (q >= n) break;
    const bool x = (xw >> q) & 1, z = (zw >> q) & 1;
    if (x && z) extra += 3;  // phase -= 1
    if (x) {
      const uint64_t* cr = c + (uint64_t)q * W;
      mul_step<uint64_t>(__ldg(cr), __ldg(cr + 1), bx, bz, c1, c2);
      extra += cph[q];
    }
    if (z) {
      const uint64_t* cr = c + (uint64_t)(q + n) * W;
      mul_step<uint64_t>(__ldg(cr), __ldg(cr + 1), bx, bz, c1, c2);
      extra += cph[q + n];
    }
  }
  __syncwarp();
  if (lane == 0) {
    if (W) { row[0] = bx; row[1] = bz; }
    ph[warp] = phases ? (uint8_t)((cnt_phase(c1, c2) + extra + ph[warp]) & 3u) : (uint8_t)0;
  }
}

// The same for any width where the tables' scratch is not there: lane l holds
// words l, l + 32, ... of the product.
template <int PER>
__global__ void __launch_bounds__(256) apply_dense_rows_kernel(uint64_t* xzs, uint8_t* ph, uint32_t rows, uint32_t W,
                                                               uint32_t n, const uint64_t* __restrict__ c,
                                                               const uint8_t* __restrict__ cph, int phases) {
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31, len = W / 2;
  if (warp >= rows) return;
  uint64_t* row = xzs + (uint64_t)warp * W;
  uint64_t bx[PER], bz[PER], c1[PER], c2[PER];
#pragma unroll
  for (int k = 0; k < PER; k++) bx[k] = bz[k] = c1[k] = c2[k] = 0;
  uint32_t extra = 0;  // sum of Clifford-row phases and -1 corrections (mod 4)
  auto image = [&](uint32_t r) {
    const uint64_t* cr = c + (uint64_t)r * W;
#pragma unroll
    for (int k = 0; k < PER; k++) {
      const uint32_t w = lane + 32 * k;
      if (w < len) mul_step<uint64_t>(__ldg(cr + w), __ldg(cr + len + w), bx[k], bz[k], c1[k], c2[k]);
    }
    extra += cph[r];
  };
  for (uint32_t wq = 0; wq < len; wq++) {
    const uint64_t xw = row[wq], zw = row[len + wq];  // broadcast loads
    uint64_t both = xw | zw;
    while (both) {
      const uint32_t b = __ffsll((long long)both) - 1, q = wq * 64 + b;
      both &= both - 1;
      if (q >= n) break;
      const bool x = (xw >> b) & 1, z = (zw >> b) & 1;
      if (x && z) extra += 3;  // phase -= 1
      if (x) image(q);
      if (z) image(q + n);
    }
  }
  uint32_t s = 0;
#pragma unroll
  for (int k = 0; k < PER; k++) s += cnt_phase(c1[k], c2[k]);
  s = __reduce_add_sync(0xFFFFFFFFu, s & 3u);
  __syncwarp();
#pragma unroll
  for (int k = 0; k < PER; k++) {
    const uint32_t w = lane + 32 * k;
    if (w < len) { row[w] = bx[k]; row[len + w] = bz[k]; }
  }
  if (lane == 0) ph[warp] = phases ? (uint8_t)((s + extra + ph[warp]) & 3u) : (uint8_t)0;
}

// Dense apply! by tables.  A state row selects up to four of the Clifford rows
// of two qubits (x_q, z_q, x_q+1, z_q+1, in this order): 16 ordered products,
// kept in shared memory for a run of qubits, so a row takes one table entry per
// two qubits instead of up to four images.  Lanes hold the words of a row, so
// an entry is read without bank conflicts.  With q = phase + |x & z| a product
// L . R has q_L + q_R + 2 (z_L . x_R): the crossings of the entries with the
// product so far are XOR-accumulated over all of them and counted once, and
// the entries' own q (phases, crossings within an entry, -1 for each Y) are a
// table of the Clifford alone (dense_q_kernel), summed over the row's entries
// at the end.  The qubits are split into KG runs over CTAs; their partial
// products are multiplied in order by dense_join_kernel.
// Bound by shared memory (an entry is len x 16 bytes; about half its rate) and
// by the instructions around each read.  Rows x qubits, us, against a product
// of one image at a time with eight warps per row: 500 x 500 36 -> 17.5, 1000 x
// 1000 122 -> 19.7, 2000 x 2000 392 -> 93, 4000 x 4000 2150 -> 385, 8000 x 8000
// 12645 -> 5365, 20000 x 100 190 -> 53.  (The tables waiting for dense_q_kernel,
// loads through L1, the join's loads four at a time: 1000 22, 4000 759.)
constexpr uint32_t DENSE_RUNS = 16;
// Shared memory of the tables at most: the limit of every launch of a form, so
// that calls of other sizes on other threads never lower it in between.
constexpr size_t DENSE_TABLE_SMEM = 200 * 1024;
constexpr size_t DENSE_SCRATCH = 256ull << 20;  // of partial products at most
struct DenseArgs {
  uint64_t* xzs;
  uint8_t* ph;
  uint32_t rows, W, n;
  const uint64_t* c;
  const uint8_t* cph;
  uint8_t* qt;         // [32 len][16] q of the entries of every two qubits
  ulonglong2* part;    // [KG][rows][len] partial products (x, z)
  uint8_t* odd;        // [KG][rows] parity of their crossings
  uint32_t KG, wpg;    // runs (at most DENSE_RUNS), qubit words per run
  uint32_t NT;         // tables in shared memory at a time
  uint32_t beside;     // the tables run beside dense_q_kernel
  int phases;
};

// The Clifford row of bit b of an entry (b & 1: second qubit, b & 2: z), or
// null past the qubits.
__device__ __forceinline__ const uint64_t* dense_image(const DenseArgs& a, uint32_t pair, uint32_t b, uint32_t& row) {
  const uint32_t q = 2 * pair + (b & 1);
  row = q + ((b & 2) ? a.n : 0);
  return q < a.n ? a.c + (uint64_t)row * a.W : nullptr;
}

// A warp per two qubits: the q of their 16 entries.
__global__ void __launch_bounds__(256) dense_q_kernel(const DenseArgs a) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;");
  const uint32_t pair = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31, len = a.W / 2;
  if (pair >= 32 * len) return;
  const uint32_t order[4] = {0, 2, 1, 3};  // entry bits in the order of the product
  const uint64_t* row[4];
  uint32_t q[4];
#pragma unroll
  for (uint32_t i = 0; i < 4; i++) {
    uint32_t r;
    row[i] = dense_image(a, pair, order[i], r);
    q[i] = lane == 0 && row[i] ? a.cph[r] : 0u;
  }
  uint64_t cr[6] = {0, 0, 0, 0, 0, 0};
  for (uint32_t w = lane; w < len; w += 32) {
    uint64_t x[4], z[4];
#pragma unroll
    for (uint32_t i = 0; i < 4; i++) {
      x[i] = row[i] ? __ldg(row[i] + w) : 0ull;
      z[i] = row[i] ? __ldg(row[i] + len + w) : 0ull;
      q[i] += __popcll(x[i] & z[i]);
    }
    uint32_t k = 0;
#pragma unroll
    for (uint32_t i = 1; i < 4; i++)
#pragma unroll
      for (uint32_t j = 0; j < i; j++) cr[k++] ^= z[i] & x[j];
  }
  uint32_t odd = 0;
#pragma unroll
  for (uint32_t k = 0; k < 6; k++) odd |= ((uint32_t)__popcll(cr[k]) & 1u) << k;
  odd = __reduce_xor_sync(0xFFFFFFFFu, odd);
  uint32_t s = 0;
#pragma unroll
  for (uint32_t i = 0; i < 4; i++) {
    q[i] = __reduce_add_sync(0xFFFFFFFFu, q[i]);
    if ((lane >> order[i]) & 1u) s += q[i];
  }
  uint32_t k = 0;
#pragma unroll
  for (uint32_t i = 1; i < 4; i++)
#pragma unroll
    for (uint32_t j = 0; j < i; j++, k++)
      if (((lane >> order[i]) & 1u) && ((lane >> order[j]) & 1u)) s += 2u * ((odd >> k) & 1u);
  if ((lane & 5) == 5 && row[0]) s += 3;  // Y on the first / second qubit
  if ((lane & 10) == 10 && row[2]) s += 3;
  if (lane < 16) a.qt[(size_t)pair * 16 + lane] = (uint8_t)(s & 3u);
}

// THREADS / 32 warps with 32 / LPR row slots each (LPR lanes), KPL words per
// lane, RPW rows per slot (their products stay in registers while the tables
// change).  NT divides 16, so a set of tables lies within half a qubit word;
// a thread makes the 16 entries of at most one (table, word), its images
// loaded while the rows take the previous tables.
template <int THREADS, int LPR, int KPL, int RPW>
__global__ void __launch_bounds__(THREADS, 1) dense_tables_kernel(const DenseArgs a) {
  extern __shared__ __align__(16) ulonglong2 tab[];  // [NT][16][len]
  // Behind dense_q_kernel, which waited for all before it, this kernel runs
  // beside it and waits at its end (the join needs both); its loads pass L1 by.
  if (!a.beside) asm volatile("griddepcontrol.wait;" ::: "memory");
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, len = a.W / 2;
  const uint32_t kg = blockIdx.x, w0 = kg * a.wpg, w1 = min(len, w0 + a.wpg);
  const uint32_t sl = lane & (LPR - 1);
  const uint32_t r0 = ((blockIdx.y * (THREADS / 32) + warp) * (32 / LPR) + lane / LPR) * RPW;
  const uint32_t mt = tid / len, mw = tid - mt * len;  // the thread's table and word
  ulonglong2 v[4];
  auto load = [&](uint32_t p0) {
#pragma unroll
    for (uint32_t b = 0; b < 4; b++) {
      uint32_t r;
      const uint64_t* im = mt < a.NT ? dense_image(a, p0 + mt, b, r) : nullptr;
      v[b] = im ? make_ulonglong2(__ldcg(im + mw), __ldcg(im + len + mw)) : make_ulonglong2(0, 0);
    }
  };
  uint64_t x[RPW][KPL], z[RPW][KPL], P[RPW];
#pragma unroll
  for (int i = 0; i < RPW; i++) {
    P[i] = 0;
#pragma unroll
    for (int k = 0; k < KPL; k++) x[i][k] = z[i][k] = 0;
  }
  load(32 * w0);
  for (uint32_t p0 = 32 * w0; p0 < 32 * w1; p0 += a.NT) {
    // the rows' selector bits: two of the x word and two of the z word per entry
    uint32_t xs[RPW], zs[RPW];
#pragma unroll
    for (int i = 0; i < RPW; i++) {
      const uint64_t* row = a.xzs + (uint64_t)min(r0 + i, a.rows - 1) * a.W + (p0 >> 5);
      xs[i] = (uint32_t)(__ldcg(row) >> (2 * (p0 & 31)));
      zs[i] = (uint32_t)(__ldcg(row + len) >> (2 * (p0 & 31)));
    }
    __syncthreads();  // the previous tables are read until here
    if (mt < a.NT) {
      ulonglong2* d = tab + (size_t)mt * 16 * len + mw;
#pragma unroll
      for (uint32_t m = 0; m < 16; m++) {
        ulonglong2 o = make_ulonglong2(0, 0);
#pragma unroll
        for (uint32_t b = 0; b < 4; b++)
          if ((m >> b) & 1u) { o.x ^= v[b].x; o.y ^= v[b].y; }
        d[m * len] = o;
      }
    }
    __syncthreads();
    if (p0 + a.NT < 32 * w1) load(p0 + a.NT);
    if (r0 < a.rows) {
#pragma unroll 1
      for (uint32_t t = 0; t < a.NT; t++) {
        const ulonglong2* tt = tab + (size_t)t * 16 * len + sl;
#pragma unroll
        for (int i = 0; i < RPW; i++) {
          const uint32_t e = (xs[i] & 3u) | ((zs[i] & 3u) << 2);
          xs[i] >>= 2;
          zs[i] >>= 2;
#pragma unroll
          for (int k = 0; k < KPL; k++) {
            if (sl + LPR * k < len) {
              const ulonglong2 o = tt[e * len + LPR * k];
              P[i] ^= o.y & x[i][k];
              x[i][k] ^= o.x;
              z[i][k] ^= o.y;
            }
          }
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < RPW; i++) {
    uint32_t odd = (uint32_t)__popcll(P[i]);
#pragma unroll
    for (int d = LPR / 2; d; d >>= 1) odd += __shfl_xor_sync(0xFFFFFFFFu, odd, d);
    if (r0 + i >= a.rows) continue;
    ulonglong2* d = a.part + ((size_t)kg * a.rows + r0 + i) * len;
#pragma unroll
    for (int k = 0; k < KPL; k++) {
      const uint32_t w = sl + LPR * k;
      if (w < len) d[w] = make_ulonglong2(x[i][k], z[i][k]);
    }
    if (sl == 0) a.odd[(size_t)kg * a.rows + r0 + i] = (uint8_t)(odd & 1u);
  }
  if (a.beside) asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;");
}

// A warp per row: the runs' products multiplied in order, the row's phase.
__global__ void __launch_bounds__(256) dense_join_kernel(const DenseArgs a) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;");
  const uint32_t r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31, len = a.W / 2;
  if (r >= a.rows) return;
  uint64_t* row = a.xzs + (uint64_t)r * a.W;
  uint32_t q = 0;
  if (a.phases) {
    // the entries' q: lane = two qubits of each word, eight words' loads in flight
    for (uint32_t w0 = 0; w0 < len; w0 += 8) {
      uint32_t e[8];
#pragma unroll
      for (uint32_t i = 0; i < 8; i++) {
        const uint32_t w = min(w0 + i, len - 1);
        e[i] = ((uint32_t)(row[w] >> (2 * lane)) & 3u) | (((uint32_t)(row[len + w] >> (2 * lane)) & 3u) << 2);
      }
#pragma unroll
      for (uint32_t i = 0; i < 8; i++)
        if (w0 + i < len) q += a.qt[((size_t)(w0 + i) * 32 + lane) * 16 + e[i]];
    }
    for (uint32_t g = lane; g < a.KG; g += 32) q += 2u * a.odd[(size_t)g * a.rows + r];
  }
  __syncwarp();
  uint64_t P = 0;
  for (uint32_t w = lane; w < len; w += 32) {
    ulonglong2 v[DENSE_RUNS];
#pragma unroll
    for (uint32_t g = 0; g < DENSE_RUNS; g++)
      v[g] = g < a.KG ? a.part[((size_t)g * a.rows + r) * len + w] : make_ulonglong2(0, 0);
    uint64_t x = 0, z = 0;
#pragma unroll
    for (uint32_t g = 0; g < DENSE_RUNS; g++) {
      P ^= v[g].y & x;
      x ^= v[g].x;
      z ^= v[g].y;
    }
    row[w] = x;
    row[len + w] = z;
    q -= (uint32_t)__popcll(x & z);
  }
  q += 2u * ((uint32_t)__popcll(P) & 1u);
  q = __reduce_add_sync(0xFFFFFFFFu, q);
  if (lane == 0) a.ph[r] = a.phases ? (uint8_t)((q + a.ph[r]) & 3u) : (uint8_t)0;
}

// rowswap!(state, i, j; phases) (src/QuantumClifford.jl:899-927): rows i and
// j of the view (and their destabilizer rows for the Destabilizer kinds), the
// phases only when `phases`.  One thread per word.
__global__ void rowswap_kernel(uint64_t* xzs, uint8_t* ph, uint32_t W, uint32_t i, uint32_t j, uint32_t di,
                               uint32_t dj, int destab, int phases) {
  const uint32_t w = blockIdx.x * blockDim.x + threadIdx.x;
  if (w < W) {
    uint64_t t = xzs[(size_t)i * W + w]; xzs[(size_t)i * W + w] = xzs[(size_t)j * W + w]; xzs[(size_t)j * W + w] = t;
    if (destab) { t = xzs[(size_t)di * W + w]; xzs[(size_t)di * W + w] = xzs[(size_t)dj * W + w]; xzs[(size_t)dj * W + w] = t; }
  }
  if (w == 0 && phases) {
    uint8_t p = ph[i]; ph[i] = ph[j]; ph[j] = p;
    if (destab) { p = ph[di]; ph[di] = ph[dj]; ph[dj] = p; }
  }
}

// ---------------------------------------------------------------- no-alloc batch
// Phase accumulators of qcb_mul_left_pauli_batch_noalloc, one per pair.  Zero
// between calls: the finish kernel clears what it read.
static __device__ __align__(256) uint32_t g_noalloc_acc[QCB_NOALLOC_MAX_PAIRS];

// Pair blockIdx.y of a batch: the grid-stride loop of mul_left_long_kernel
// over that pair's words, the phase sum added into acc[pair].
template <int VEC, bool PH>
__global__ void __launch_bounds__(256) mul_left_batch_kernel(uint64_t* __restrict__ r,
                                                             const uint64_t* __restrict__ l,
                                                             uint64_t len, uint32_t* acc) {
  const uint32_t pair = blockIdx.y;
  r += (uint64_t)pair * 2 * len;
  l += (uint64_t)pair * 2 * len;
  uint64_t c1a = 0, c2a = 0, c1b = 0, c2b = 0;
  const uint64_t nvec = len / VEC;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nvec; i += stride) {
    if (VEC == 2) {
      const ulonglong2 lx = __ldcs((const ulonglong2*)l + i);
      const ulonglong2 lz = __ldcs((const ulonglong2*)(l + len) + i);
      ulonglong2 rx = __ldcs((const ulonglong2*)r + i);
      ulonglong2 rz = __ldcs((const ulonglong2*)(r + len) + i);
      if (PH) {
        mul_step(lx.x, lz.x, rx.x, rz.x, c1a, c2a);
        mul_step(lx.y, lz.y, rx.y, rz.y, c1b, c2b);
      } else {
        rx.x ^= lx.x; rx.y ^= lx.y; rz.x ^= lz.x; rz.y ^= lz.y;
      }
      __stcs((ulonglong2*)r + i, rx);
      __stcs((ulonglong2*)(r + len) + i, rz);
    } else {
      const uint64_t lx = __ldcs(l + i), lz = __ldcs(l + len + i);
      uint64_t rx = __ldcs(r + i), rz = __ldcs(r + len + i);
      if (PH) mul_step(lx, lz, rx, rz, c1a, c2a);
      else { rx ^= lx; rz ^= lz; }
      __stcs(r + i, rx);
      __stcs(r + len + i, rz);
    }
  }
  if (!PH) return;
  uint32_t v = (cnt_phase(c1a, c2a) + cnt_phase(c1b, c2b)) & 3u;
  v = __reduce_add_sync(0xFFFFFFFFu, v) & 3u;
  __shared__ uint32_t wsum[32];
  const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) wsum[wid] = v;
  __syncthreads();
  if (wid == 0) {
    uint32_t s = lane < (blockDim.x >> 5) ? wsum[lane] : 0u;
    s = __reduce_add_sync(0xFFFFFFFFu, s) & 3u;
    if (lane == 0 && s) atomicAdd(acc + pair, s);
  }
}

// r_phase[i] <- (s_i + r_phase[i] + l_phase[i]) & 3 (src/mul_leftright.jl:140)
// when phases; clears acc[i] either way.
__global__ void mul_left_batch_finish_kernel(uint8_t* r_phase, const uint8_t* l_phase, uint32_t* acc,
                                             uint32_t count, int phases) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  if (phases) r_phase[i] = (uint8_t)(((acc[i] & 3u) + r_phase[i] + l_phase[i]) & 3u);
  acc[i] = 0;
}

static uint32_t g_gates_pdl = 1;  // symbolic gate launches as programmatic dependents (0: plain)
void set_gates_pdl(uint32_t v) { g_gates_pdl = v; }

// A gate launch: a programmatic dependent of the previous launch on the
// stream, so that in a stream of single-gate calls each launch is scheduled
// while the one before it runs, instead of after it drains.
template <class... P, class... A>
static cudaError_t launch_gates(void (*k)(P...), uint32_t grid, uint32_t block, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = g_gates_pdl ? 1 : 0;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k, args...);
}

// Shortest gate list that runs bit-sliced.  The row-per-thread kernel takes 4 us
// a call in a stream up to 10 gates, then 0.3 to 1 us a gate; the slices cost a
// read, two transposes and a write of the tableau whatever the gates: 4.5 us up
// to 2000 qubits, where 8 gates are as fast either way, then a CTA's 32 rows of
// all qubits take 1.9 us per 1000 qubits (20 rows or 1000; us, slices / rows of 12
// gates: 5000 qubits 11 / 9.5, 10000 22 / 9.8, 20000 39 / 10.7; the lines cross at
// 15, 29 and 50 gates), and many slices the tableau's traffic (a gate per MB).
static size_t layer_min_gates(const qcb_tableau* t) {
  const size_t mb = ((size_t)t->rows * t->W * 8) >> 20;
  const size_t least = t->rows < 64 || t->W <= 2 ? 12 : 8;  // the sorting into levels, 0.8 us on the host
  return std::max(least + mb, t->W / 12 + (t->rows > 4096 ? mb : 0));
}

static size_t layer_smem(const qcb_tableau* t) { return (size_t)LAYER_SLICE * (2 * t->W + 1) * 4; }

// The most a slice may take, and the limit of every launch above the default
// one: a call on a smaller tableau on another thread does not lower it.
static size_t layer_smem_max() { return (size_t)device_max_smem_optin() - 1024; }

template <uint32_t CAP>
static int launch_layers(const qcb_tableau* t, const std::vector<uint64_t>& list, uint32_t threads, int phases,
                         cudaStream_t st) {
  LayerList<CAP> l;
  std::copy(list.begin(), list.end(), l.e);
  const size_t sm = layer_smem(t);
  if (sm > 40 * 1024)
    QCB_CUDA(cudaFuncSetAttribute(apply_layers_kernel<CAP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)layer_smem_max()));
  QCB_CUDA(launch_gates(apply_layers_kernel<CAP>, (t->rows + LAYER_SLICE - 1) / LAYER_SLICE, threads, sm, st, t->xzs,
                        t->phases, t->rows, t->W, (const LayerList<CAP>&)l, (uint32_t)list.size(), phases));
  QCB_LAUNCHED();
  return QCB_OK;
}

// The list as levels of disjoint gates, launch by launch.
static int apply_layers(const qcb_tableau* t, const std::vector<GateOp>& g, int phases, cudaStream_t st) {
  std::vector<uint32_t> qlev(t->nqubits), lev, start, at;
  std::vector<uint64_t> list;
  for (size_t k0 = 0; k0 < g.size();) {
    // as many gates as fit with their level headers
    std::fill(qlev.begin(), qlev.end(), 0u);
    lev.clear();
    uint32_t depth = 0;
    size_t k = k0;
    for (; k < g.size(); k++) {
      const bool two = (g[k].op & 0xFFu) >= QCB_OP_CNOT;
      const uint32_t l = std::max(qlev[g[k].q1], two ? qlev[g[k].q2] : 0u);
      if (k - k0 + 1 + std::max(depth, l + 1) > LAYER_CAP_L) break;
      depth = std::max(depth, l + 1);
      qlev[g[k].q1] = l + 1;
      if (two) qlev[g[k].q2] = l + 1;
      lev.push_back(l);
    }
    // by opcode (a warp then runs one branch of the gate table), then by level
    const size_t n = k - k0;
    start.assign(257, 0);
    for (size_t i = 0; i < n; i++) start[(g[k0 + i].op & 0xFFu) + 1]++;
    for (uint32_t i = 0; i < 256; i++) start[i + 1] += start[i];
    at.resize(n);
    for (size_t i = 0; i < n; i++) at[start[g[k0 + i].op & 0xFFu]++] = (uint32_t)i;
    start.assign(depth + 1, 0);
    for (size_t i = 0; i < n; i++) start[lev[i] + 1]++;
    uint32_t most = 0;
    for (uint32_t i = 0; i < depth; i++) {
      most = std::max(most, start[i + 1]);
      start[i + 1] += start[i];
    }
    list.resize(n + depth);
    for (uint32_t i = 0; i < depth; i++) list[start[i] + i] = start[i + 1] - start[i];
    for (size_t i = 0; i < n; i++) {
      const GateOp& o = g[k0 + at[i]];
      const uint32_t l = lev[at[i]];
      list[start[l]++ + l + 1] = (uint64_t)o.op | ((uint64_t)o.q1 << 16) | ((uint64_t)o.q2 << 40);
    }
    // threads for the widest level and a warp per two transposes, at least 256:
    // the slice's loads and stores take a warp a row (64 threads up to 64 qubits,
    // us a call in a stream: 8 gates, 100 x 10 8.4 -> 4.4, 1000 x 64 8.8 -> 4.4; 128
    // up to 128 qubits, 1000 x 100 6.7 -> 4.4)
    const uint32_t threads = std::min<uint32_t>(512, std::max<uint32_t>(256, std::max((most + 31) / 32 * 32, 32 * t->W)));
    if (int s = list.size() <= LAYER_CAP_S ? launch_layers<LAYER_CAP_S>(t, list, threads, phases, st)
                                           : launch_layers<LAYER_CAP_L>(t, list, threads, phases, st))
      return s;
    k0 = k;
  }
  return QCB_OK;
}

// Whether dense apply! goes by tables: its three launches take 11 to 16 us in a
// stream of calls and 25 to 29 us alone for any small tableau, a warp per row 8 us
// (16 alone) and 0.17 us a qubit.  us in a stream / alone, tables against warps:
// 48 qubits x 1 row 11.6 / 25.6 and 16.7 / 24.8, x 200 rows 16.1 / 29.1 and 14.5 /
// 23.1, x 4000 19.4 / 32.1 and 28.7 / 36.2; 56 x 200 16.1 / 28.9 and 16.6 / 25.0;
// 64 x 200 16.1 / 29.1 and 18.6 / 26.8.  Many rows cross earlier (20000 rows: 16
// qubits 42 / 55 and 36 / 44, 32 42 / 56 and 66 / 74).
static bool dense_tables_pay(uint32_t rows, uint32_t n) {
  if (rows >= 16384) return n >= 24;
  return n >= (rows < 128 || rows >= 2048 ? 48u : 56u);
}

template <class... P, class... A>
static cudaError_t launch_dependent(void (*k)(P...), dim3 grid, uint32_t block, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return cudaLaunchKernelEx(&cfg, k, args...);
}

// *none: no room for the partial products of one row group, nothing done.
static int apply_dense_tables(qcb_tableau* t, const qcb_tableau* c, int phases, cudaStream_t st, bool* none) {
  const uint32_t R = t->rows, len = t->W / 2;
  // threads; lanes per row (half a warp up to 16 words), words per lane and
  // rows per slot, whose products fill the registers
  struct Form { void (*k)(const DenseArgs); uint32_t threads, rows; };
  const Form f = len <= 16 ? Form{dense_tables_kernel<1024, 16, 1, 2>, 1024, 128}
               : len <= 32 ? Form{dense_tables_kernel<1024, 32, 1, 4>, 1024, 128}
               : len <= 64 ? Form{dense_tables_kernel<512, 32, 2, 6>, 512, 96}
                           : Form{dense_tables_kernel<512, 32, 4, 4>, 512, 64};
  DenseArgs a{};
  a.W = t->W; a.n = t->nqubits; a.c = c->xzs; a.cph = c->phases; a.phases = phases;
  const size_t table = (size_t)16 * len * sizeof(ulonglong2);
  a.NT = 16;
  while (a.NT * len > f.threads || a.NT * table > DENSE_TABLE_SMEM) a.NT /= 2;
  const size_t smem = a.NT * table;
  // Runs of whole qubit words and rows at a time (a slab): the least waves x
  // (words of a run x the time of a word's tables, with 3 us for a CTA) and the
  // partial products' traffic, among those whose partial products (16 len bytes
  // a row and run) take at most `cap`.  As many runs as fill one wave leaves
  // large ones a half-empty last wave (rows x qubits, us: 20000 x 2000 1304 ->
  // 779, 8000 x 4000 1269 -> 752, 4000 x 4000 441 -> 385, 8000 x 8000 6148 -> 5365).
  const uint32_t nsm = (uint32_t)std::max(device_sm_count(), 1);
  uint32_t slab = 0;
  auto split = [&](size_t cap) {
    auto time = [&](uint32_t rows, uint32_t kg, uint32_t wpg) {
      const uint32_t RG = (rows + f.rows - 1) / f.rows;
      const double word_us = 0.005 * f.rows * len, run_us = (double)rows * len * 32 / 5e6;
      return (RG * kg + nsm - 1) / nsm * (wpg * word_us + 3.0) + kg * run_us;
    };
    double best = 0;
    slab = 0;
    for (uint32_t g = 1; g <= std::min(len, DENSE_RUNS); g++) {
      const uint32_t wpg = (len + g - 1) / g, kg = (len + wpg - 1) / wpg;
      size_t fit = std::min<size_t>(R, cap / ((size_t)kg * (16 * len + 1)) / f.rows * f.rows);
      if (!fit && kg == 1) fit = std::min(R, f.rows);  // the least
      if (!fit) continue;
      const uint32_t full = R / (uint32_t)fit, rest = R % (uint32_t)fit;
      const double us = full * time((uint32_t)fit, kg, wpg) + (rest ? time(rest, kg, wpg) : 0.0);
      if (!slab || us < best) { best = us; slab = (uint32_t)fit; a.KG = kg; a.wpg = wpg; }
    }
  };
  Scratch scratch(st);
  size_t o_part = 0, o_odd = 0;
  for (size_t cap = DENSE_SCRATCH;; cap /= 2) {  // less where that much memory is not there
    split(cap);
    size_t bytes = 0;
    auto place = [&](size_t n) { const size_t o = bytes; bytes += (n + 127) / 128 * 128; return o; };
    place((size_t)32 * len * 16);
    o_part = place((size_t)a.KG * slab * len * 16);
    o_odd = place((size_t)a.KG * slab);
    const cudaError_t e = scratch.alloc(bytes);
    if (e == cudaSuccess) break;
    if (e != cudaErrorMemoryAllocation) return cuda_fail(e, "qcb_apply_dense scratch");
    *none = a.KG == 1 && slab <= f.rows;
    if (*none) return QCB_OK;
  }
  uint8_t* m = scratch.p;
  a.qt = m; a.part = (ulonglong2*)(m + o_part); a.odd = m + o_odd;
  QCB_CUDA(cudaFuncSetAttribute(f.k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DENSE_TABLE_SMEM));
  if (phases) QCB_CUDA(launch_dependent(dense_q_kernel, dim3((32 * len + 7) / 8), 256, 0, st, a));
  for (uint32_t r0 = 0; r0 < R; r0 += slab) {
    a.xzs = t->xzs + (size_t)r0 * t->W;
    a.ph = t->phases + r0;
    a.rows = std::min(slab, R - r0);
    a.beside = phases && r0 == 0;  // later slabs wait for the join before them
    QCB_CUDA(launch_dependent(f.k, dim3(a.KG, (a.rows + f.rows - 1) / f.rows), f.threads, smem, st, a));
    QCB_CUDA(launch_dependent(dense_join_kernel, dim3((a.rows + 7) / 8), 256, 0, st, a));
  }
  return QCB_OK;
}

}  // namespace qcb

using namespace qcb;

extern "C" {

int qcb_mul_left_pauli(qcb_tableau* r, const qcb_tableau* l, int phases, uint8_t* phase_out,
                       void* stream) {
  if (!r || !l) return fail(QCB_EARG, "null argument");
  if (r->nqubits != l->nqubits)
    return fail(QCB_EDIM, "The two Pauli operators should have the same length!");
  if (r->rows < 1 || l->rows < 1) return fail(QCB_EDIM, "empty Pauli");
  const uint64_t len = r->W / 2;
  cudaStream_t st = S(stream);
  const int sms = device_sm_count();
  const bool vec = (len % 2 == 0);
  const uint64_t work = vec ? len / 2 : len;
  // one wave of resident blocks (no tail wave for the grid-stride loop)
  void (*k)(uint64_t*, const uint64_t*, uint64_t, uint32_t*, uint8_t*, const uint8_t*) =
      vec ? (phases ? mul_left_long_kernel<2, true> : mul_left_long_kernel<2, false>)
          : (phases ? mul_left_long_kernel<1, true> : mul_left_long_kernel<1, false>);
  int per_sm = 0;
  QCB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, 256, 0));
  uint32_t blocks = (uint32_t)std::min<uint64_t>((work + 255) / 256, (uint64_t)sms * std::max(per_sm, 1));
  if (blocks == 0) blocks = 1;
  if (len) {
    k<<<blocks, 256, 0, st>>>(r->xzs, l->xzs, len, r->scratch, r->phases, l->phases);
    QCB_LAUNCHED();
  } else if (phases) {
    mul_left_finish_kernel<<<1, 1, 0, st>>>(r->phases, l->phases, r->scratch, phases);
    QCB_LAUNCHED();
  }
  if (phase_out) {
    QCB_CUDA(cudaMemcpyAsync(phase_out, r->phases, 1, cudaMemcpyDeviceToHost, st));
    QCB_CUDA(cudaStreamSynchronize(st));
  }
  return QCB_OK;
}

int qcb_rowswap(qcb_tableau* t, int kind, uint32_t i, uint32_t j, int phases, void* stream) {
  if (!t) return fail(QCB_EARG, "null tableau");
  if (i == 0 || j == 0) return fail(QCB_EBOUNDS, "rows are 1-based");
  const bool destab = kind == QCB_DESTABILIZER || kind == QCB_MIXED_DESTABILIZER;
  if (kind < 0 || kind > 3) return fail(QCB_EARG, "rowswap!: bad state kind");
  if (destab && t->rows % 2) return fail(QCB_EDIM, "destabilizer tableaux have an even number of rows");
  const uint32_t nn = destab ? t->rows / 2 : t->rows;
  if (i > nn || j > nn) return fail(QCB_EBOUNDS, "rowswap!: row out of range");
  if (i == j) return QCB_OK;
  const uint32_t off = destab ? nn : 0;
  rowswap_kernel<<<(t->W + 127) / 128, 128, 0, S(stream)>>>(t->xzs, t->phases, t->W, off + i - 1, off + j - 1, i - 1,
                                                           j - 1, destab ? 1 : 0, phases);
  QCB_LAUNCHED();
  return QCB_OK;
}

int qcb_mul_rows(qcb_tableau* s, uint32_t s_row, uint32_t count, const qcb_tableau* t, uint32_t t_row,
                 uint32_t t_step, int right, int phase_src, int phases, uint8_t* phase_out, void* stream) {
  if (!s || !t) return fail(QCB_EARG, "null tableau");
  if (s->nqubits != t->nqubits) return fail(QCB_EDIM, "The two Pauli operators should have the same length!");
  if (!count) return QCB_OK;
  const uint64_t last_b = (uint64_t)t_row + (uint64_t)(count - 1) * t_step;
  if (s_row < 1 || t_row < 1 || (uint64_t)s_row + count - 1 > s->rows || last_b > t->rows)
    return fail(QCB_EBOUNDS, "row index out of bounds");
  if (phase_src && last_b > s->rows) return fail(QCB_EBOUNDS, "row index out of bounds (phase taken from s)");
  if (s == t && count > 1) {  // rows read by one warp must not be written by another
    const bool same = (t_row == s_row && t_step == 1);
    const uint64_t b_lo = t_row, b_hi = last_b;
    const bool disjoint = (b_hi < s_row || b_lo >= (uint64_t)s_row + count);
    if (!same && !disjoint)
      return fail(QCB_EARG, "source rows overlap the target rows of the same tableau");
  }
  cudaStream_t st = S(stream);
  const uint8_t* add = phase_src ? s->phases : t->phases;
  const uint32_t a0 = s_row - 1, b0 = t_row - 1;
  const uint64_t len = s->W / 2;
  if (count == 1 && len >= (1u << 15)) {
    // one long row: the grid-stride kernel of mul_left!(::PauliOperator, ...)
    const bool vec = (len % 2 == 0);
    uint64_t* r = s->xzs + (uint64_t)a0 * s->W;
    const uint64_t* l = t->xzs + (uint64_t)b0 * t->W;
    const bool aligned = ((uintptr_t)r % 16 == 0) && ((uintptr_t)l % 16 == 0);
    void (*k)(uint64_t*, const uint64_t*, uint64_t, uint32_t*, uint8_t*, const uint8_t*);
    if (vec && aligned)
      k = right ? (phases ? mul_left_long_kernel<2, true, true> : mul_left_long_kernel<2, false, true>)
                : (phases ? mul_left_long_kernel<2, true> : mul_left_long_kernel<2, false>);
    else
      k = right ? (phases ? mul_left_long_kernel<1, true, true> : mul_left_long_kernel<1, false, true>)
                : (phases ? mul_left_long_kernel<1, true> : mul_left_long_kernel<1, false>);
    int per_sm = 0;
    QCB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, 256, 0));
    const uint64_t work = (vec && aligned) ? len / 2 : len;
    uint32_t blocks = (uint32_t)std::min<uint64_t>((work + 255) / 256,
                                                   (uint64_t)device_sm_count() * std::max(per_sm, 1));
    k<<<std::max(blocks, 1u), 256, 0, st>>>(r, l, len, s->scratch, s->phases + a0, add + b0);
    QCB_LAUNCHED();
  } else {
    const uint32_t warps_per_block = 8;
    const uint32_t blocks = (uint32_t)std::min<uint64_t>((count + warps_per_block - 1) / warps_per_block,
                                                         (uint64_t)device_sm_count() * 16);
    void (*k)(uint64_t*, uint8_t*, uint32_t, uint32_t, const uint64_t*, uint32_t, uint32_t, uint32_t,
              const uint8_t*) = right ? (phases ? mul_rows_kernel<true, true> : mul_rows_kernel<true, false>)
                                      : (phases ? mul_rows_kernel<false, true> : mul_rows_kernel<false, false>);
    k<<<blocks, 256, 0, st>>>(s->xzs, s->phases, a0, count, t->xzs, b0, t_step, s->W, add);
    QCB_LAUNCHED();
  }
  if (phase_out) {
    QCB_CUDA(cudaMemcpyAsync(phase_out, s->phases + a0, 1, cudaMemcpyDeviceToHost, st));
    QCB_CUDA(cudaStreamSynchronize(st));
  }
  return QCB_OK;
}

int qcb_mul_left_state(qcb_tableau* s, int kind, uint32_t i, uint32_t j, int phases, void* stream) {
  if (!s) return fail(QCB_EARG, "null tableau");
  if (kind == QCB_DESTABILIZER || kind == QCB_MIXED_DESTABILIZER) {
    // src/mul_leftright.jl:200-219: destabilizer j <- destabilizer i * j
    // without phases (indices flipped), then stabilizer i <- stabilizer j * i
    if (s->rows % 2) return fail(QCB_EDIM, "a Destabilizer tableau has 2n rows");
    const uint32_t n = s->rows / 2;
    if (i < 1 || j < 1 || i > n || j > n) return fail(QCB_EBOUNDS, "row index out of bounds");
    if (int st = qcb_mul_rows(s, j, 1, s, i, 0, 0, 0, 0, nullptr, stream)) return st;
    return qcb_mul_rows(s, i + n, 1, s, j + n, 0, 0, 0, phases, nullptr, stream);
  }
  if (kind != QCB_STABILIZER && kind != QCB_MIXED_STABILIZER) return fail(QCB_EARG, "unknown state kind");
  // src/mul_leftright.jl:194-198, 207-211: rows of the tableau
  return qcb_mul_rows(s, i, 1, s, j, 0, 0, 0, phases, nullptr, stream);
}

int qcb_mul_left_row(qcb_tableau* s, uint32_t m, uint32_t i, int phases, void* stream) {
  if (!s) return fail(QCB_EARG, "null tableau");
  if (m < 1 || i < 1 || m > s->rows || i > s->rows) return fail(QCB_EBOUNDS, "row index out of bounds");
  mul_left_row_kernel<<<1, 32, 0, S(stream)>>>(s->xzs, s->phases, s->W, m - 1, i - 1, phases);
  QCB_LAUNCHED();
  return QCB_OK;
}

int qcb_mul_left_tableau_pauli(qcb_tableau* s, const qcb_tableau* p, int phases, void* stream) {
  if (!s || !p) return fail(QCB_EARG, "null argument");
  if (s->nqubits != p->nqubits) return fail(QCB_EDIM, "The tableau and the Pauli operator must have the same number of qubits");
  if (!s->rows) return QCB_OK;
  const uint32_t threads = 256, blocks = (s->rows * 32 + threads - 1) / threads;
  mul_left_tab_pauli_kernel<<<blocks, threads, 0, S(stream)>>>(s->xzs, s->phases, s->rows, s->W,
                                                               p->xzs, p->phases, phases);
  QCB_LAUNCHED();
  return QCB_OK;
}

static int pc_common(const qcb_tableau* l, uint32_t i, const qcb_tableau* r, uint32_t j, uint8_t* out,
                     void* stream, int what) {
  if (!l || !r || !out) return fail(QCB_EARG, "null argument");
  if (l->nqubits != r->nqubits) return fail(QCB_EDIM, "operands must have the same number of qubits");
  if (i < 1 || i > l->rows || j < 1 || j > r->rows) return fail(QCB_EBOUNDS, "row index out of bounds");
  cudaStream_t st = S(stream);
  uint8_t lph = 0, rph = 0;
  QCB_CUDA(cudaMemcpyAsync(&lph, l->phases + (i - 1), 1, cudaMemcpyDeviceToHost, st));
  QCB_CUDA(cudaMemcpyAsync(&rph, r->phases + (j - 1), 1, cudaMemcpyDeviceToHost, st));
  QCB_CUDA(cudaStreamSynchronize(st));
  uint8_t* d = (uint8_t*)l->scratch + 64;
  prodphase_comm_kernel<<<1, 32, 0, st>>>(l->xzs + (uint64_t)(i - 1) * l->W, lph,
                                          r->xzs + (uint64_t)(j - 1) * r->W, rph, l->W / 2, what, d);
  QCB_LAUNCHED();
  QCB_CUDA(cudaMemcpyAsync(out, d, 1, cudaMemcpyDeviceToHost, st));
  QCB_CUDA(cudaStreamSynchronize(st));
  return QCB_OK;
}

int qcb_prodphase(const qcb_tableau* l, uint32_t i, const qcb_tableau* r, uint32_t j, uint8_t* out,
                  void* stream) {
  return pc_common(l, i, r, j, out, stream, 0);
}

int qcb_comm(const qcb_tableau* l, uint32_t i, const qcb_tableau* r, uint32_t j, uint8_t* out,
             void* stream) {
  return pc_common(l, i, r, j, out, stream, 1);
}

int qcb_apply_gates(qcb_tableau* t, const qcb_op* ops, size_t n_ops, int phases, void* stream) {
  if (!t) return fail(QCB_EARG, "null tableau");
  std::vector<GateOp> g;
  g.reserve(n_ops);
  for (size_t k = 0; k < n_ops; k++) {
    const qcb_op& o = ops[k];
    const bool one = o.opcode >= QCB_OP_I && o.opcode <= QCB_OP_SQO;
    const bool two = o.opcode >= QCB_OP_CNOT && o.opcode <= QCB_OP_LAST2Q;
    if (!one && !two) return fail(QCB_EUNSUPPORTED, "qcb_apply_gates: op " + std::to_string(k) + " is not a symbolic Clifford gate");
    if (o.q1 == 0 || (two && o.q2 == 0)) return fail(QCB_EZEROQUBIT, "qubit indices start at 1 (NoZeroQubit)");
    if (two && o.q1 == o.q2) return fail(QCB_EARG, "Failed to create a two qubit gate because the two qubits it acts on have the same index. The qubit indices have to be different.");
    if (o.q1 > t->nqubits || (two && o.q2 > t->nqubits)) return fail(QCB_EBOUNDS, "gate qubit index exceeds the tableau's qubits");
    const uint32_t code = o.opcode == QCB_OP_SQO ? o.opcode | ((o.q2 & 63u) << 8) : o.opcode;
    g.push_back({code, o.q1 - 1, two ? o.q2 - 1 : 0, 0});
  }
  if (g.empty() || !t->rows) return QCB_OK;
  cudaStream_t st = S(stream);
  if (g.size() >= layer_min_gates(t) && layer_smem(t) <= layer_smem_max())
    return apply_layers(t, g, phases, st);
  for (size_t k0 = 0; k0 < g.size(); k0 += GATE_BATCH) {
    const uint32_t n = (uint32_t)std::min<size_t>(GATE_BATCH, g.size() - k0);
    GateBatch b{};
    std::copy(g.begin() + k0, g.begin() + k0 + n, b.op);
    QCB_CUDA(launch_gates(apply_gates_kernel, (t->rows + 127) / 128, 128, 0, st, t->xzs, t->phases, t->rows, t->W,
                          (const GateBatch)b, n, phases));
    QCB_LAUNCHED();
  }
  return QCB_OK;
}

int qcb_apply_dense(qcb_tableau* t, const qcb_tableau* c, int phases, void* stream) {
  if (!t || !c) return fail(QCB_EARG, "null argument");
  if (t->nqubits != c->nqubits || c->rows != 2 * c->nqubits)
    return fail(QCB_EDIM, "The tableau and the Clifford operator need to act on the same number of qubits.");
  if (!t->rows) return QCB_OK;
  cudaStream_t st = S(stream);
  const uint32_t W = t->W;
  if (W > 256) return fail(QCB_EUNSUPPORTED, "qcb_apply_dense: at most 8192 qubits");
  if (dense_tables_pay(t->rows, t->nqubits)) {
    bool none = false;
    const int s = apply_dense_tables(t, c, phases, st, &none);
    if (!none) return s;
  }
  const uint32_t threads = 256, blocks = (uint32_t)(((uint64_t)t->rows * 32 + threads - 1) / threads);
  auto kern = W <= 2 ? apply_dense_kernel : W <= 64 ? apply_dense_rows_kernel<1> : apply_dense_rows_kernel<4>;
  kern<<<blocks, threads, 0, st>>>(t->xzs, t->phases, t->rows, W, t->nqubits, c->xzs, c->phases, phases);
  QCB_LAUNCHED();
  return QCB_OK;
}

// The no-alloc scratch of the current device: looked up once per device with
// that device current, cleared once, then reused by every call.
static std::mutex g_noalloc_mu;
static uint32_t* g_noalloc_ptr[64] = {};

static int noalloc_scratch(uint32_t** out) {
  int dev = 0;
  QCB_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return fail(QCB_EARG, "device ordinal out of range for the no-alloc scratch");
  std::lock_guard<std::mutex> lock(g_noalloc_mu);
  if (!g_noalloc_ptr[dev]) {
    uint32_t* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress((void**)&p, g_noalloc_acc);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(no-alloc scratch)");
    e = cudaMemset(p, 0, sizeof(uint32_t) * QCB_NOALLOC_MAX_PAIRS);
    if (e != cudaSuccess) return cuda_fail(e, "clearing the no-alloc scratch");
    e = cudaDeviceSynchronize();
    if (e != cudaSuccess) return cuda_fail(e, "clearing the no-alloc scratch");
    g_noalloc_ptr[dev] = p;
  }
  *out = g_noalloc_ptr[dev];
  return QCB_OK;
}

int qcb_mul_left_pauli_batch_noalloc(uint64_t* r_xz, uint8_t* r_phases, const uint64_t* l_xz,
                                     const uint8_t* l_phases, uint32_t nqubits, uint32_t count,
                                     int phases, void* stream) {
  if (count == 0) return QCB_OK;
  if (count > QCB_NOALLOC_MAX_PAIRS)
    return fail(QCB_EARG, "qcb_mul_left_pauli_batch_noalloc: count " + std::to_string(count) +
                              " exceeds the no-alloc scratch of " + std::to_string(QCB_NOALLOC_MAX_PAIRS) +
                              " pairs; split the batch");
  if (!r_xz || !l_xz) return fail(QCB_EARG, "qcb_mul_left_pauli_batch_noalloc: null Pauli words");
  if (phases && (!r_phases || !l_phases)) return fail(QCB_EARG, "qcb_mul_left_pauli_batch_noalloc: null phases");
  uint32_t* acc = nullptr;
  if (int st = noalloc_scratch(&acc)) return st;
  const uint64_t len = ((uint64_t)nqubits + 63) / 64;
  cudaStream_t st = S(stream);
  const bool vec = len % 2 == 0 && (((uintptr_t)r_xz | (uintptr_t)l_xz) & 15u) == 0;
  const uint64_t work = vec ? len / 2 : len;
  const uint32_t bx = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>((work + 255) / 256, (uint64_t)device_sm_count() * 8));
  if (len) {
    const dim3 grid(bx, count);
    if (vec) {
      if (phases) mul_left_batch_kernel<2, true><<<grid, 256, 0, st>>>(r_xz, l_xz, len, acc);
      else mul_left_batch_kernel<2, false><<<grid, 256, 0, st>>>(r_xz, l_xz, len, acc);
    } else {
      if (phases) mul_left_batch_kernel<1, true><<<grid, 256, 0, st>>>(r_xz, l_xz, len, acc);
      else mul_left_batch_kernel<1, false><<<grid, 256, 0, st>>>(r_xz, l_xz, len, acc);
    }
    QCB_LAUNCHED();
  }
  mul_left_batch_finish_kernel<<<(count + 255) / 256, 256, 0, st>>>(r_phases, l_phases, acc, count, phases);
  QCB_LAUNCHED();
  return QCB_OK;
}

}  // extern "C"
