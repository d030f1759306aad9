// decode.cu -- the decoder hand-off of a sampled frame
// (src/ecc/decoder_pipeline.jl:163-193): the syndrome and fault columns of
// the record, the syndrome matrix a decoder consumes, and evaluate_guesses.
//
// The record lives as shot-packed bit planes (row b = record bit b, word c =
// shots 32c..32c+31).  A decoder wants it shot-major: per shot the selected
// bits in order.  `syndrome_rows_kernel` transposes 32 x 32 bit blocks in the
// registers of one thread, stages them in shared memory and writes each
// shot's words out contiguously.  `evaluate_guesses_kernel` works on
// planes: per 32 shots, the parity of the guessed faults selected by each
// row of the faults matrix against the measured logical row, a miss on any
// row failing the shot, then a popcount.
#include <algorithm>
#include <vector>

#include "qcb_internal.h"

namespace qcb {

// out[s, k] (column-major Bool, S x nsel) = record[rows[k], s] ^ flip[k].
__global__ void record_columns_kernel(const uint32_t* rec, uint64_t pitch, uint64_t S, const uint32_t* rows,
                                      const uint8_t* flip, uint32_t nsel, uint8_t* out) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;  // 4 shots per thread
  const uint32_t k = blockIdx.y;
  const uint64_t f = i * 4;
  if (f >= S || k >= nsel) return;
  const uint32_t word = __ldg(rec + (uint64_t)rows[k] * pitch + (f >> 5));
  const uint32_t sh = (uint32_t)(f & 31);
  const uint8_t x = flip ? (flip[k] & 1u) : 0u;
  uint8_t* dst = out + (uint64_t)k * S + f;
  for (uint32_t j = 0; j < 4 && f + j < S; j++) dst[j] = (uint8_t)(((word >> (sh + j)) & 1u) ^ x);
}

template <uint32_t J>
__device__ __forceinline__ void swap_bits(uint32_t v[32], uint32_t m) {
#pragma unroll
  for (uint32_t i = 0; i < 32; i++) {
    if (i & J) continue;
    // two shifts and two selects; the exchange by XORs takes five
    const uint32_t a = v[i], b = v[i + J];
    v[i] = (a & m) | ((b << J) & ~m);
    v[i + J] = ((a >> J) & m) | (b & ~m);
  }
}

// The 32 x 32 bit matrix in v (v[i] bit s) transposed in place (v[s] bit i),
// by one thread in its registers: five rounds of masked swaps of halves.
__device__ __forceinline__ void transpose32(uint32_t v[32]) {
#pragma unroll
  for (uint32_t i = 0; i < 16; i++) {  // halves of 16 and 8 bits are byte moves
    const uint32_t a = v[i], b = v[i + 16];
    v[i] = __byte_perm(a, b, 0x5410);
    v[i + 16] = __byte_perm(a, b, 0x7632);
  }
#pragma unroll
  for (uint32_t i = 0; i < 32; i++) {
    if (i & 8u) continue;
    const uint32_t a = v[i], b = v[i + 8];
    v[i] = __byte_perm(a, b, 0x6240);
    v[i + 8] = __byte_perm(a, b, 0x7351);
  }
  swap_bits<4>(v, 0x0F0F0F0Fu);
  swap_bits<2>(v, 0x33333333u);
  swap_bits<1>(v, 0x55555555u);
}

// Shot-major syndrome matrix: out[s * Wsyn + w] bit b = record[rows[64w + b], s]
// (bits past nsel are zero; without LIST: record row rows[0] + k for bit k).
// The rows come by value, up to SYN_LIST to a launch: nothing is allocated or
// copied, and the call need not wait.
// A CTA takes SYN_COLS word columns (512 shots) and a block of `pairs` output
// words (blockIdx.x; 64 record rows each).  Half-warp h of warp w loads the 32
// rows of 32-bit group 2w + h, a lane per column (64 contiguous bytes a row),
// and each lane transposes its 32 x 32 bits in registers; the CTA's words are
// staged in shared memory, a column's shots at a stride of 2 mod 32 words (the
// stores of a warp then hit 32 banks and the 64-bit loads are aligned), and
// leave as contiguous runs of `pairs` words per shot, a column of 32 shots per
// step of the CTA.  Bound by DRAM (the record in, the matrix out).
// 1e6 shots x 1441 bits 85 us (364 MB, 4.3 TB/s), 150001 x 9681 73 us (5.0);
// output steps of two shots a warp with an odd column stride, and exchanges by
// five instructions: 92 and 93 us.  A persistent CTA with the next tile's
// loads on their way while one leaves spills at 64 registers: 110 us.
// With a column per CTA (4-byte reads a plane apart, 32 ballots per 32 x 32
// block) 519 us, with the loads behind branches instead of predicates (one in
// flight at a time) 262 us.
constexpr uint32_t SYN_COLS = 16;
constexpr uint32_t SYN_PAIRS = 16;  // output words of a CTA at most (512 threads)

constexpr uint32_t SYN_LIST = 4096;  // 16 KB of parameters

template <bool LIST>
struct SynRows {
  uint32_t row[LIST ? SYN_LIST : 1];
};

template <bool LIST>
__global__ void __launch_bounds__(32 * SYN_PAIRS, 2)
syndrome_rows_kernel(const uint32_t* __restrict__ rec, uint64_t pitch, uint64_t ncols, uint64_t S,
                     const __grid_constant__ SynRows<LIST> rows, uint32_t nsel, uint32_t nwords, uint32_t Wsyn,
                     uint32_t pairs, uint64_t* __restrict__ out) {
  extern __shared__ __align__(16) uint32_t tile[];  // [SYN_COLS][32 * RS + 2]
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;");
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;  // `pairs` warps
  const uint32_t RS = 2 * pairs, CS = 32 * RS + 2;  // words of a shot, of a column
  const uint32_t w0 = blockIdx.x * pairs;           // the CTA's first output word
  const uint32_t words = min(pairs, nwords - w0);
  const uint64_t c0 = (uint64_t)blockIdx.y * SYN_COLS;
  const uint32_t cl = lane & (SYN_COLS - 1), h = lane / SYN_COLS;
  const uint64_t c = c0 + cl;
  if (warp < words) {
    const uint32_t k0 = (w0 + warp) * 64 + h * 32;  // first selected bit of the group
    // all 32 loads in flight: predicates, no branches
    const uint32_t lim = c < ncols ? min(32u, nsel - min(nsel, k0)) : 0u;
    uint32_t v[32];
    if (LIST) {
#pragma unroll
      for (uint32_t i = 0; i < 32; i++) v[i] = i < lim ? rows.row[k0 + i] : 0u;
#pragma unroll
      for (uint32_t i = 0; i < 32; i++) v[i] = i < lim ? __ldcs(rec + (uint64_t)v[i] * pitch + c) : 0u;
    } else {
      const uint32_t* src = rec + (uint64_t)(rows.row[0] + k0) * pitch + c;  // read below lim only
#pragma unroll
      for (uint32_t i = 0; i < 32; i++, src += pitch) v[i] = i < lim ? __ldcs(src) : 0u;
    }
    transpose32(v);
    uint32_t* t = tile + (size_t)cl * CS + 2 * warp + h;
#pragma unroll
    for (uint32_t s = 0; s < 32; s++) t[s * RS] = v[s];
  }
  __syncthreads();
  // 32 * pairs threads: word wl of shot r of each column in turn
  const uint32_t r = threadIdx.x / pairs, wl = threadIdx.x - r * pairs;
  if (wl >= words) return;
  const uint32_t* t = tile + r * RS + 2 * wl;
  uint64_t* o = out + (c0 * 32 + r) * Wsyn + w0 + wl;
  const uint64_t step = (uint64_t)32 * Wsyn, left = S - c0 * 32;  // c0 < ncols: at least one shot
#pragma unroll
  for (uint32_t k = 0; k < SYN_COLS; k++, t += CS, o += step)
    if (k * 32 + r < left) *o = *(const uint64_t*)t;
}

// guesses (column-major Bool S x k) -> planes [k][ncols] u32.
__global__ void bools_to_planes_kernel(const uint8_t* g, uint64_t S, uint32_t k, uint64_t ncols, uint32_t* planes) {
  const uint64_t c = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t col = blockIdx.y;
  if (c >= ncols || col >= k) return;
  const uint8_t* src = g + (uint64_t)col * S + c * 32;
  uint32_t w = 0;
  const uint32_t n = (uint32_t)(S - c * 32 < 32 ? S - c * 32 : 32);
  for (uint32_t b = 0; b < n; b++) w |= (uint32_t)(src[b] & 1u) << b;
  planes[(uint64_t)col * ncols + c] = w;
}

// evaluate_guesses (src/ecc/decoder_pipeline.jl:172-190) over 32 shots per
// thread: shot s fails when some row j of the faults matrix gives
// parity(F[j,:] . guess_s) != measured fault j of shot s.  F is nlog rows of
// Fw 32-bit words in shared memory.
__global__ void evaluate_guesses_kernel(const uint32_t* rec, uint64_t pitch, uint64_t S, const uint32_t* log_rows,
                                        uint32_t nlog, const uint32_t* gplanes, uint32_t k, uint64_t ncols,
                                        const uint32_t* F, uint32_t Fw, unsigned long long* fails) {
  extern __shared__ uint32_t Fs[];
  for (uint32_t t = threadIdx.x; t < nlog * Fw; t += blockDim.x) Fs[t] = F[t];
  __syncthreads();
  uint32_t cnt = 0;
  for (uint64_t c = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; c < ncols; c += (uint64_t)gridDim.x * blockDim.x) {
    uint32_t bad = 0;
    for (uint32_t j = 0; j < nlog; j++) {
      uint32_t par = __ldg(rec + (uint64_t)log_rows[j] * pitch + c);
      for (uint32_t fw = 0; fw < Fw; fw++) {
        uint32_t m = Fs[j * Fw + fw];
        while (m) {
          const uint32_t b = __ffs(m) - 1;
          m &= m - 1;
          par ^= __ldg(gplanes + (uint64_t)(fw * 32 + b) * ncols + c);
        }
      }
      bad |= par;
    }
    const uint64_t base = c * 32;
    if (S - base < 32) bad &= (1u << (uint32_t)(S - base)) - 1u;
    cnt += __popc(bad);
  }
  cnt = __reduce_add_sync(0xFFFFFFFFu, cnt);
  if ((threadIdx.x & 31) == 0 && cnt) atomicAdd(fails, (unsigned long long)cnt);
}

// The syndrome words of nsel selected bits: words out[s * Wsyn ..] of every shot s.
template <bool LIST>
static int launch_syndrome(const qcb_frame* f, const SynRows<LIST>& rows, uint32_t nsel, uint32_t Wsyn, uint64_t* out,
                           cudaStream_t st) {
  const uint32_t nwords = (nsel + 63) / 64;
  // words per CTA: the blocks of a shot's words as even as they divide; 8 where
  // the runs then start and end on 64 bytes of the output (150001 x 9681 73 us
  // against 78 with 16, 2^20 x 2048 104 against 110; with Wsyn = 23 or 21
  // shorter runs lose, 1e6 x 1320 89 against 81)
  const uint32_t most = Wsyn % 8 ? SYN_PAIRS : 8;
  const uint32_t blocks = (nwords + most - 1) / most, pairs = (nwords + blocks - 1) / blocks;
  const size_t sm = (size_t)SYN_COLS * (64 * pairs + 2) * 4;
  auto kern = syndrome_rows_kernel<LIST>;
  QCB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)(SYN_COLS * (64 * SYN_PAIRS + 2) * 4)));
  // column blocks in slices of the grid's y limit (33.5e6 shots each)
  const uint64_t nblk = (f->ncols + SYN_COLS - 1) / SYN_COLS;
  for (uint64_t b0 = 0; b0 < nblk; b0 += 65535) {
    const uint32_t nb = (uint32_t)std::min<uint64_t>(65535, nblk - b0);
    const uint64_t cb = b0 * SYN_COLS;
    // a programmatic dependent of the launch before it, so that a row of these
    // (the jobs of a batch) and the walk before them leave no launch gaps: 24
    // jobs with their walk 811 -> 778 us
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(blocks, nb);
    cfg.blockDim = dim3(32 * pairs);
    cfg.dynamicSmemBytes = sm;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    QCB_CUDA(cudaLaunchKernelEx(&cfg, kern, (const uint32_t*)(f->record + cb), f->pitch, f->ncols - cb,
                                f->frames - cb * 32, rows, nsel, nwords, Wsyn, pairs, out + cb * 32 * Wsyn));
    QCB_LAUNCHED();
  }
  return QCB_OK;
}

}  // namespace qcb

using namespace qcb;

// Validated 0-based record rows of 1-based bits.
static int record_rows(const qcb_frame* f, const uint32_t* bits, size_t n, std::vector<uint32_t>& rows) {
  rows.resize(n);
  for (size_t k = 0; k < n; k++) {
    if (bits[k] == 0) return fail(QCB_EZEROQUBIT, "record bits start at 1");
    if (bits[k] > f->nbits) return fail(QCB_EBOUNDS, "record bit exceeds the frame's measurements");
    rows[k] = bits[k] - 1;
  }
  return QCB_OK;
}

extern "C" {

int qcb_frame_measurement_columns(const qcb_frame* f, const uint32_t* bits, size_t nsel, const uint8_t* reference,
                                  uint8_t* bools, void* stream) {
  if (!f || (nsel && (!bits || !bools))) return fail(QCB_EARG, "null argument");
  std::vector<uint32_t> rows;
  if (int s = record_rows(f, bits, nsel, rows)) return s;
  if (!nsel || !f->frames) return QCB_OK;
  if (nsel > 65535) return fail(QCB_EARG, "at most 65535 columns per call");
  cudaStream_t st = S(stream);
  uint32_t* d_rows = nullptr;
  uint8_t *d_flip = nullptr, *d_out = nullptr;
  const size_t bytes = (size_t)f->frames * nsel;
  QCB_CUDA(cudaMallocAsync(&d_rows, nsel * 4, st));
  QCB_CUDA(cudaMallocAsync(&d_out, bytes, st));
  QCB_CUDA(cudaMemcpyAsync(d_rows, rows.data(), nsel * 4, cudaMemcpyHostToDevice, st));
  std::vector<uint8_t> flip;
  if (reference) {
    // measurements(register, frame): the Register's reference bits XORed in
    flip.resize(nsel);
    for (size_t k = 0; k < nsel; k++) flip[k] = reference[rows[k]] & 1u;
    QCB_CUDA(cudaMallocAsync(&d_flip, nsel, st));
    QCB_CUDA(cudaMemcpyAsync(d_flip, flip.data(), nsel, cudaMemcpyHostToDevice, st));
  }
  dim3 grid((unsigned)(((f->frames + 3) / 4 + 255) / 256), (unsigned)nsel);
  record_columns_kernel<<<grid, 256, 0, st>>>(f->record, f->pitch, f->frames, d_rows, d_flip, (uint32_t)nsel, d_out);
  QCB_LAUNCHED();
  QCB_CUDA(cudaMemcpyAsync(bools, d_out, bytes, cudaMemcpyDeviceToHost, st));
  cudaFreeAsync(d_rows, st);
  cudaFreeAsync(d_out, st);
  if (d_flip) cudaFreeAsync(d_flip, st);
  QCB_CUDA(cudaStreamSynchronize(st));
  return QCB_OK;
}

int qcb_frame_syndrome_rows(const qcb_frame* f, const uint32_t* bits, size_t nsel, uint64_t* out, int out_on_device,
                            void* stream) {
  if (!f || (nsel && (!bits || !out))) return fail(QCB_EARG, "null argument");
  std::vector<uint32_t> rows;
  if (int s = record_rows(f, bits, nsel, rows)) return s;
  if (!nsel || !f->frames) return QCB_OK;
  cudaStream_t st = S(stream);
  const uint32_t Wsyn = (uint32_t)((nsel + 63) / 64);
  const size_t out_bytes = (size_t)f->frames * Wsyn * 8;
  Scratch host_out(st);
  uint64_t* d_out = out;
  if (!out_on_device) {
    QCB_CUDA(host_out.alloc(out_bytes, false));
    d_out = (uint64_t*)host_out.p;
  }
  // a run of consecutive record bits (the whole record, the syndrome of a
  // round) in one launch, other selections SYN_LIST bits to a launch
  bool run = true;
  for (size_t k = 1; k < nsel && run; k++) run = rows[k] == rows[0] + k;
  if (run) {
    SynRows<false> r{{rows[0]}};
    if (int s = launch_syndrome(f, r, (uint32_t)nsel, Wsyn, d_out, st)) return s;
  } else {
    for (size_t k = 0; k < nsel; k += SYN_LIST) {
      SynRows<true> r;
      const uint32_t n = (uint32_t)std::min<size_t>(SYN_LIST, nsel - k);
      std::copy(rows.begin() + k, rows.begin() + k + n, r.row);
      if (int s = launch_syndrome(f, r, n, Wsyn, d_out + k / 64, st)) return s;
    }
  }
  if (!out_on_device) {
    QCB_CUDA(cudaMemcpyAsync(out, d_out, out_bytes, cudaMemcpyDeviceToHost, st));
    QCB_CUDA(cudaStreamSynchronize(st));
  }
  return QCB_OK;
}

int qcb_evaluate_guesses(const qcb_frame* f, const uint32_t* logical_bits, size_t nlog, const uint8_t* guesses,
                         size_t k, const uint8_t* faults, uint64_t* fails, void* stream) {
  if (!f || !fails || (nlog && !logical_bits) || (k && (!guesses || !faults))) return fail(QCB_EARG, "null argument");
  std::vector<uint32_t> rows;
  if (int s = record_rows(f, logical_bits, nlog, rows)) return s;
  *fails = 0;
  if (!nlog || !f->frames) return QCB_OK;
  if (k > 65535) return fail(QCB_EARG, "at most 65535 guess columns");
  cudaStream_t st = S(stream);
  // faults: nlog x k Bool, column-major (Julia Matrix layout) -> bit rows
  const uint32_t Fw = (uint32_t)((k + 31) / 32);
  std::vector<uint32_t> F((size_t)nlog * std::max<uint32_t>(Fw, 1), 0);
  for (size_t j = 0; j < nlog; j++)
    for (size_t c = 0; c < k; c++)
      if (faults[c * nlog + j] & 1u) F[j * Fw + c / 32] |= 1u << (c % 32);
  const size_t smF = F.size() * 4;
  if (smF > 200 * 1024) return fail(QCB_EARG, "faults matrix too large for one call");
  uint32_t *d_rows = nullptr, *d_F = nullptr, *d_planes = nullptr;
  uint8_t* d_g = nullptr;
  unsigned long long* d_fails = nullptr;
  QCB_CUDA(cudaMallocAsync(&d_rows, nlog * 4, st));
  QCB_CUDA(cudaMallocAsync(&d_F, smF, st));
  QCB_CUDA(cudaMallocAsync(&d_fails, 8, st));
  QCB_CUDA(cudaMemcpyAsync(d_rows, rows.data(), nlog * 4, cudaMemcpyHostToDevice, st));
  QCB_CUDA(cudaMemcpyAsync(d_F, F.data(), smF, cudaMemcpyHostToDevice, st));
  QCB_CUDA(cudaMemsetAsync(d_fails, 0, 8, st));
  if (k) {
    QCB_CUDA(cudaMallocAsync(&d_g, (size_t)f->frames * k, st));
    QCB_CUDA(cudaMallocAsync(&d_planes, (size_t)k * f->ncols * 4, st));
    QCB_CUDA(cudaMemcpyAsync(d_g, guesses, (size_t)f->frames * k, cudaMemcpyHostToDevice, st));
    dim3 g1((unsigned)((f->ncols + 255) / 256), (unsigned)k);
    bools_to_planes_kernel<<<g1, 256, 0, st>>>(d_g, f->frames, (uint32_t)k, f->ncols, d_planes);
    QCB_LAUNCHED();
  }
  if (smF > 48 * 1024)
    QCB_CUDA(allow_max_smem(evaluate_guesses_kernel));
  const uint32_t blocks = (uint32_t)std::min<uint64_t>((f->ncols + 255) / 256, 4ull * device_sm_count());
  evaluate_guesses_kernel<<<std::max<uint32_t>(blocks, 1), 256, smF, st>>>(
      f->record, f->pitch, f->frames, d_rows, (uint32_t)nlog, d_planes, (uint32_t)k, f->ncols, d_F, Fw, d_fails);
  QCB_LAUNCHED();
  unsigned long long h = 0;
  QCB_CUDA(cudaMemcpyAsync(&h, d_fails, 8, cudaMemcpyDeviceToHost, st));
  cudaFreeAsync(d_rows, st);
  cudaFreeAsync(d_F, st);
  cudaFreeAsync(d_fails, st);
  if (d_g) cudaFreeAsync(d_g, st);
  if (d_planes) cudaFreeAsync(d_planes, st);
  QCB_CUDA(cudaStreamSynchronize(st));
  *fails = h;
  return QCB_OK;
}

}  // extern "C"
