// panel.cuh -- eliminations by panels of up to 64 pivot steps.
//
// canonicalize! and a run of project! steps share one structure: a step picks
// a pivot row and left-multiplies every other row that has the step's bit (a
// column of the tableau, or the commutation bit with a Pauli) by it.  The
// steps of a panel need one 64-bit word per row (the panel's bits), so they
// run on those words alone, and the rows are brought up to date once per
// panel.
//
//   U(r)   the set of steps of the panel that multiplied row r, found by
//          replaying the recorded steps on the row's word;
//   P_t    the pivot row as it was at step t ("reduced"): the XOR of the
//          pivots' start rows selected by A_t, A = (I + U)^-1 over the
//          pivots' own sets U_t (lower triangular);
//   row r  becomes M . row r with M the ordered product of the P_t, t in U(r).
//
// Phases.  With q = phase + |x & z| (mod 4) a product L . R has q = q_L + q_R
// + 2 (z_L . x_R).  So q grows by q_M + 2 (z_M . x_r), and q_M = sum q(P_t) +
// 2 sum over t > s in U of G[t][s], G[t][s] = z_{P_t} . x_{P_s}: one 64 x 64
// bit matrix per panel and one dot product per row, whatever the number of
// steps.  q(P_t) solves a triangular system mod 4, which A inverts bit by bit.
// The products equal the reference's mul_left! sequence for any rows,
// commuting or not.
//
// Layout.  The rows live in a scratch copy by tiles of two word columns:
// t[tile][row] = (x words 2 tile, 2 tile + 1), (z words), 32 bytes.  A CTA of
// the apply takes one tile of a range of rows and forms M's words with eight
// table lookups, a table per byte of U (256 combinations of 8 reduced pivots).
// The parity z_M . x_r is a sum over the tiles: each tile keeps its own bit
// per row (par[tile][row]), folded in when a row's q is read.
#pragma once
#include "qcb_internal.h"

namespace qcb {

constexpr uint32_t PSTEPS = 64;   // steps of a panel at most

struct PanelRecord {
  uint32_t T;                 // steps taken
  uint32_t i0, i;             // canonicalize!: next pivot position before and after the panel
  uint32_t rx;                // pivots of the X stage
  uint32_t done;              // no later panel does anything
  uint32_t stp[PSTEPS];       // pivot row of step t
  uint32_t bt[PSTEPS];        // its bit of the panel word
  uint32_t m[PSTEPS];         // canonicalize!: its position before the step
  uint64_t A[PSTEPS];         // start rows in the reduced pivot t
  uint64_t PW[PSTEPS];        // the pivot's panel word at its step
  uint32_t src[PSTEPS];       // project!: the step whose Pauli is pivot t's start row (PSTEPS: row stp)
  uint32_t sbt[PSTEPS];       // project!: that Pauli (PSTEPS: none)
  uint64_t own[PSTEPS];       // project!: the steps that multiplied pivot t before its own
  uint32_t s[PSTEPS];         // project!: |x & z| of the reduced pivot, summed over the tiles
  unsigned long long G[PSTEPS];  // z_{P_t} . x_{P_s} (bit s), summed over the tiles
  uint32_t q0[PSTEPS];        // q of the pivot's start row, summed over the tiles
};

struct PanelTiles {
  uint32_t rows, W, len, ntile;
  int phases;
  ulonglong2* t;      // [ntile][rows][2]
  ulonglong2* po;     // [ntile][PSTEPS][2] reduced pivots
  uint64_t* word;     // [rows] the panel's word at the panel start
  uint64_t* U;        // [rows]
  uint8_t* q;         // [rows] q without the tiles' parities
  uint8_t* par;       // [ntile][rows]
};

// (word, mask) ^= p where `test` has the bit.
__device__ __forceinline__ void xor_if(uint32_t (&v)[4], uint32_t test, uint32_t bit, const uint32_t (&p)[4]) {
  asm("{.reg .pred y; .reg .u32 x; and.b32 x, %4, %5; setp.ne.u32 y, x, 0;"
      "@y xor.b32 %0, %0, %6; @y xor.b32 %1, %1, %7; @y xor.b32 %2, %2, %8; @y xor.b32 %3, %3, %9;}"
      : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3])
      : "r"(test), "r"(bit), "r"(p[0]), "r"(p[1]), "r"(p[2]), "r"(p[3]));
}

__device__ __forceinline__ ulonglong2 xor128(ulonglong2 a, ulonglong2 b) { return make_ulonglong2(a.x ^ b.x, a.y ^ b.y); }
__device__ __forceinline__ uint32_t parity64(uint64_t v) { return __popc((uint32_t)v ^ (uint32_t)(v >> 32)) & 1u; }
__device__ __forceinline__ uint64_t bitmask64(uint64_t v, uint32_t b) { return 0ull - ((v >> b) & 1ull); }

// One word of one row of the tiles: word w of the row layout (X words, then Z).
__device__ __forceinline__ uint64_t tile_word(const PanelTiles& p, uint32_t row, uint32_t w) {
  const uint32_t z = w >= p.len, k = w - z * p.len;
  const uint64_t* e = (const uint64_t*)(p.t + ((size_t)(k >> 1) * p.rows + row) * 2);
  return e[2 * z + (k & 1)];
}

// Row r (a warp) from the row layout into the tiles; its q.
__device__ __forceinline__ void tiles_load_row(const PanelTiles& p, const uint64_t* row, uint32_t r, uint32_t ph,
                                               uint32_t lane) {
  uint32_t s = 0;
  for (uint32_t k = lane; k < p.ntile; k += 32) {
    const bool two = 2 * k + 1 < p.len;
    ulonglong2 x = make_ulonglong2(row[2 * k], two ? row[2 * k + 1] : 0ull);
    ulonglong2 z = make_ulonglong2(row[p.len + 2 * k], two ? row[p.len + 2 * k + 1] : 0ull);
    ulonglong2* d = p.t + ((size_t)k * p.rows + r) * 2;
    d[0] = x;
    d[1] = z;
    s += __popcll(x.x & z.x) + __popcll(x.y & z.y);
    p.par[(size_t)k * p.rows + r] = 0;
  }
  s = __reduce_add_sync(0xFFFFFFFFu, s);
  if (lane == 0) p.q[r] = (uint8_t)((ph + s) & 3u);
}

// Row r (a warp) back into the row layout; returns its phase (all lanes).
__device__ __forceinline__ uint32_t tiles_store_row(const PanelTiles& p, uint64_t* row, uint32_t r, uint32_t lane) {
  uint32_t s = 0, par = 0;
  for (uint32_t k = lane; k < p.ntile; k += 32) {
    const bool two = 2 * k + 1 < p.len;
    const ulonglong2* d = p.t + ((size_t)k * p.rows + r) * 2;
    const ulonglong2 x = d[0], z = d[1];
    row[2 * k] = x.x;
    row[p.len + 2 * k] = z.x;
    if (two) {
      row[2 * k + 1] = x.y;
      row[p.len + 2 * k + 1] = z.y;
    }
    s += __popcll(x.x & z.x) + __popcll(x.y & z.y);
    par ^= p.par[(size_t)k * p.rows + r];
  }
  s = __reduce_add_sync(0xFFFFFFFFu, s);
  par = __reduce_xor_sync(0xFFFFFFFFu, par);
  return (p.q[r] + 2u * par - s) & 3u;
}

// ---------------------------------------------------------------- reduced pivots
// A CTA of 256 threads on one tile: the pivots' start rows reduced by A into
// po, and the tile's share of G and of the start rows' q.  base(t, r) are the
// start words of pivot t, row r, on the tile (two ulonglong2, readable for
// stale records too), q0(t, r) its share of q; red(t) sees the reduced pivot.
constexpr uint32_t MID_THREADS = 256;

struct __align__(16) TileSmem {
  uint64_t start[PSTEPS][4], red[PSTEPS][4];
};

template <class Base, class Q0, class Red>
__device__ __forceinline__ void tile_reduce(const PanelTiles& p, PanelRecord& g, uint32_t tile, TileSmem& s, Base base,
                                            Q0 q0, Red red) {
  // fields beyond the record's T steps are stale but readable
  const uint32_t tid = threadIdx.x, T = g.T;
  const uint32_t t = tid >> 2, w = tid & 3;
  const uint32_t r = g.stp[t];
  const uint64_t A0 = g.A[t], st = ((const uint64_t*)base(t, r))[w];
  if (T == 0) return;
  uint64_t A = t < T ? A0 : 0ull;
  s.start[t][w] = t < T ? st : 0ull;
  __syncthreads();
  uint64_t v = 0;
#pragma unroll 16
  for (uint32_t x = 0; x < PSTEPS; x++) {
    v ^= s.start[x][w] & bitmask64(A, 0);
    A >>= 1;
  }
  s.red[t][w] = v;
  ((uint64_t*)(p.po + ((size_t)tile * PSTEPS + t) * 2))[w] = v;
  if (!p.phases) return;
  const uint32_t q = w == 0 && t < T ? q0(t, r) : 0u;
  __syncthreads();
  if (w == 1 && t < T) red(t, s.red[t]);
  // G[t] bits 16 w .. 16 w + 15
  const uint64_t z0 = s.red[t][2], z1 = s.red[t][3];
  uint32_t bits = 0;
#pragma unroll 8
  for (uint32_t k = 0; k < 16; k++) {
    const ulonglong2 x = *(const ulonglong2*)s.red[16 * w + k];
    const uint64_t y = (z0 & x.x) ^ (z1 & x.y);
    bits |= (__popc((uint32_t)y ^ (uint32_t)(y >> 32)) & 1u) << k;
  }
  uint64_t all = (uint64_t)bits << (16 * w);
  all |= __shfl_xor_sync(0xFFFFFFFFu, all, 1);
  all |= __shfl_xor_sync(0xFFFFFFFFu, all, 2);
  if (w == 0 && t < T) {
    if (all) atomicXor(&g.G[t], (unsigned long long)all);
    if (q) atomicAdd(&g.q0[t], q);
  }
}

// ---------------------------------------------------------------- phase data
// The pivots' q and the lower triangle of G of one record, by a whole CTA;
// own(t): the steps that multiplied pivot t before its own.
struct PhaseSmem {
  uint64_t U[PSTEPS], A[PSTEPS], G[PSTEPS], GL[PSTEPS];
  uint32_t bal[8];
  uint64_t Q1, Q2;          // bit t: low / high bit of q(P_t)
  uint64_t tab4[16][16], tab[8][256];  // XOR of the GL_t of a nibble's / byte's set
};

__device__ __forceinline__ uint64_t vote64(PhaseSmem& s, uint32_t slot, bool b) {
  const uint32_t m = __ballot_sync(0xFFFFFFFFu, b);
  if ((threadIdx.x & 31) == 0 && threadIdx.x < 64) s.bal[2 * slot + (threadIdx.x >> 5)] = m;
  __syncthreads();
  return (uint64_t)s.bal[2 * slot] | ((uint64_t)s.bal[2 * slot + 1] << 32);
}

template <class Own>
__device__ __forceinline__ void phase_data(const PanelRecord& g, PhaseSmem& s, Own own) {
  const uint32_t tid = threadIdx.x, T = g.T;
  uint32_t q0 = 0;
  if (tid < PSTEPS) {
    const bool in = tid < T;
    s.U[tid] = in ? own(tid) : 0ull;
    s.A[tid] = in ? g.A[tid] : 0ull;
    s.G[tid] = in ? g.G[tid] : 0ull;
    s.GL[tid] = s.G[tid] & ((1ull << tid) - 1ull);
    q0 = in ? g.q0[tid] : 0u;
  }
  __syncthreads();
  // c_t: q0 plus twice the crossings of the pivot's own products
  uint32_t c = 0;
  uint64_t U = 0;
  if (tid < PSTEPS) {
    U = s.U[tid];
    uint64_t vg = 0, vl = 0;
#pragma unroll 8
    for (uint32_t x = 0; x < PSTEPS; x++) {
      const uint64_t m = bitmask64(U, x);
      vg ^= s.G[x] & m;
      vl ^= s.GL[x] & m;
    }
    c = q0 + 2u * (parity64(vg & (U | (1ull << tid))) + parity64(vl & U));
  }
  const uint64_t A = tid < PSTEPS ? s.A[tid] : 0ull;
  const uint64_t c1 = vote64(s, 0, tid < PSTEPS && (c & 1u));
  const uint64_t Q1 = vote64(s, 1, tid < PSTEPS && parity64(A & c1));
  const uint32_t carry = ((uint32_t)__popcll(U & Q1) + (c & 1u)) >> 1;
  const uint64_t ch = vote64(s, 2, tid < PSTEPS && (((c >> 1) ^ carry) & 1u));
  const uint64_t Q2 = vote64(s, 3, tid < PSTEPS && parity64(A & ch));
  if (tid == 0) { s.Q1 = Q1; s.Q2 = Q2; }
  for (uint32_t e = tid; e < 256; e += blockDim.x) {
    uint64_t v = 0;
    for (uint32_t b = 0; b < 4; b++) v ^= s.GL[4 * (e >> 4) + b] & bitmask64(e, b);
    s.tab4[e >> 4][e & 15] = v;
  }
  __syncthreads();
  for (uint32_t e = tid; e < 2048; e += blockDim.x) {
    const uint32_t k = e >> 8;
    s.tab[k][e & 255] = s.tab4[2 * k][e & 15] ^ s.tab4[2 * k + 1][(e >> 4) & 15];
  }
  __syncthreads();
}

// q_M of the set U.
__device__ __forceinline__ uint32_t phase_of(const PhaseSmem& s, uint64_t U) {
  uint64_t v = 0;
#pragma unroll
  for (uint32_t k = 0; k < 8; k++) v ^= s.tab[k][(U >> (8 * k)) & 255];
  return (uint32_t)__popcll(U & s.Q1) + 2u * ((uint32_t)__popcll(U & s.Q2) + parity64(v & U));
}

// ---------------------------------------------------------------- apply
// The byte tables of one tile's reduced pivots: tab[k][e] = XOR of the pivots
// 8 k + b, b in e.  64 KB, and 8 KB for the nibble tables they come from.
struct ApplySmem {
  ulonglong2 tab4[16][16][2];
  ulonglong2 tab[8][256][2];
};

__device__ __forceinline__ void apply_tables(const PanelTiles& p, uint32_t tile, ApplySmem& s) {
  const ulonglong2* P = p.po + (size_t)tile * PSTEPS * 2;
  for (uint32_t e = threadIdx.x; e < 512; e += blockDim.x) {
    const uint32_t h = e & 1, v = (e >> 1) & 15, k = e >> 5;
    ulonglong2 a = make_ulonglong2(0, 0);
#pragma unroll
    for (uint32_t b = 0; b < 4; b++)
      if ((v >> b) & 1u) a = xor128(a, P[(4 * k + b) * 2 + h]);
    s.tab4[k][v][h] = a;
  }
  __syncthreads();
  for (uint32_t e = threadIdx.x; e < 4096; e += blockDim.x) {
    const uint32_t h = e & 1, v = (e >> 1) & 255, k = e >> 9;
    s.tab[k][v][h] = xor128(s.tab4[2 * k][v & 15][h], s.tab4[2 * k + 1][v >> 4][h]);
  }
  __syncthreads();
}

// M's words of this tile for the set U.
__device__ __forceinline__ void apply_lookup(const ApplySmem& s, uint64_t U, ulonglong2& mx, ulonglong2& mz) {
  mx = mz = make_ulonglong2(0, 0);
#pragma unroll
  for (uint32_t k = 0; k < 8; k++) {
    const uint32_t e = (uint32_t)(U >> (8 * k)) & 255u;
    mx = xor128(mx, s.tab[k][e][0]);
    mz = xor128(mz, s.tab[k][e][1]);
  }
}

}  // namespace qcb
