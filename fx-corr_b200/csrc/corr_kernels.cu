// corr_kernels.cu — what surrounds the correlation kernels, for sm_100a.
//
// frame_info_kernel evaluates the FP64 per-frame delay model
// (src/main.rs:184-241) for every frame of a sector, one thread per frame, into
// 48-byte FrameInfo records; batch_frame_info_kernel does so for every sector of
// a batch.
//
// spectra_kernel is the spectra stage's kernel (FFT <= 8192): both stations'
// spectra of every frame, by a decode of its own.  One CTA
// processes a contiguous run of frame pairs: FrameInfo and packed words arrive
// by cp.async.bulk tracked by an mbarrier, two stages deep; 32-bit word shuffle,
// b-bit codes -> f32 levels, LSB->USB flip of odd samples (src/utils.rs:215-376),
// integer shift with zero fill (src/utils.rs:126-145), one complex FFT for both
// stations, two-for-one split (src/utils.rs:47-59).  The correlation itself is in
// corr_small.cu (FFT 1024..4096), corr_fold.cu (8192, 16384) and the kernels of
// larger FFTs.
//
// reduce_partials_kernel and its wide and batched forms sum the per-CTA partials
// in a fixed order.
#include <cuda_runtime.h>
#include <stdint.h>

#include "fxc_device.cuh"
#include "fxc_kernels.h"

namespace fxc {

// Per-CTA setup of spectra_kernel: mbarriers, error flag, twiddle chains.
template <int N, int FPC>
__device__ __forceinline__ void corr_cta_init(const SmemLayout& L, uint8_t* smem, Twiddles<N>& tw) {
  constexpr int T1 = N / 16;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L.off_bar);
  int* flag = reinterpret_cast<int*>(smem + L.off_flag);
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) mbar_init(&bars[s], 1);
    *flag = 0;
    fence_proxy_async();
  }
  tw.init(threadIdx.x % T1);
}

__device__ __forceinline__ void corr_cta_drain(const SmemLayout& L, uint8_t* smem) {
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L.off_bar);
  const int* flag = reinterpret_cast<const int*>(smem + L.off_flag);
  // never leave a bulk copy in flight into a finished CTA's shared memory
  if (threadIdx.x == 0 && *flag) {
    for (int s = 0; s < kStages; ++s) mbar_wait(&bars[s], 0, kWaitPolls);
  }
}

// Iterations [it0, it1) (FPC frame pairs each) of the sector described by p into
// p.out_a, p.out_b.
template <int N, int FPC>
__device__ __forceinline__ void stage_span(const CorrParams& p, uint64_t it0, uint64_t it1,
                                           uint8_t* smem, const SmemLayout& L,
                                           const Twiddles<N>& tw) {
  constexpr int T1 = N / 16;
  constexpr int T = FPC * T1;
  constexpr int H = N / 2 + 1;

  float2* bufA = reinterpret_cast<float2*>(smem + L.off_a);
  float2* bufB = reinterpret_cast<float2*>(smem + L.off_b);
  uint8_t* stage = smem + L.off_stage;
  uint32_t* lut = reinterpret_cast<uint32_t*>(smem + L.off_lut);
  float* lv = reinterpret_cast<float*>(smem + L.off_lv);
  FrameInfo* finfo = reinterpret_cast<FrameInfo*>(smem + L.off_fi);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L.off_bar);
  int* flag = reinterpret_cast<int*>(smem + L.off_flag);

  const int tid = threadIdx.x;
  const int g = tid / T1;  // frame slot of this thread in an iteration
  const int t = tid % T1;  // thread index within its frame pair

  const uint32_t bpf1 = p.st[0].bpf, bpf2 = p.st[1].bpf;
  const uint8_t* raw1 = p.st[0].raw;
  const uint8_t* raw2 = p.st[1].raw;
  const FrameInfo* gfi = p.finfo;
  constexpr uint32_t kRaw1 = FPC * kFiBytes;  // offset of station 1 bytes in a slot

  auto issue = [&](uint64_t it) {
    const int slot = (int)((uint32_t)(it - it0) % kStages);
    const uint64_t f0 = it * FPC;
    const uint64_t nvalid = (p.nf - f0) < (uint64_t)FPC ? (p.nf - f0) : (uint64_t)FPC;
    const uint32_t bf = (uint32_t)(nvalid * kFiBytes);
    const uint32_t b1 = (uint32_t)(nvalid * bpf1), b2 = (uint32_t)(nvalid * bpf2);
    uint8_t* dst = stage + slot * L.stage_stride;
    mbar_expect_tx(&bars[slot], bf + b1 + b2);
    bulk_g2s(dst, gfi + f0, bf, &bars[slot]);
    bulk_g2s(dst + kRaw1, raw1 + f0 * bpf1, b1, &bars[slot]);
    bulk_g2s(dst + kRaw1 + FPC * bpf1, raw2 + f0 * bpf2, b2, &bars[slot]);
  };
  // The first iterations' copies go out first, the tables are built meanwhile.
  __syncthreads();
  if (tid == 0) {
    fence_proxy_async();
    for (uint64_t it = it0; it < it1 && it < it0 + kStages; ++it) issue(it);
  }
  for (int i = tid; i < 512; i += T) lv[i] = p.st[i >> 8].levels[i & 255] * p.st[i >> 8].scale;
  for (int s = 0; s < 2; ++s)
    if (p.st[s].shkind == SH_GENERIC)
      for (int i = tid; i < 1024; i += T) lut[s * 1024 + i] = p.st[s].shlut[i];
  __syncthreads();

  for (uint64_t it = it0; it < it1; ++it) {
    const uint32_t q_it = (uint32_t)(it - it0);
    const int slot = (int)(q_it % kStages);
    const uint32_t parity = (q_it / kStages) & 1u;
    const uint64_t frame_local = it * FPC + g;
    const bool valid = frame_local < p.nf;

    if (!mbar_wait(&bars[slot], parity, kWaitPolls)) {
      atomicOr(flag, 1);
      atomicOr(p.err, ERR_WAIT_TIMEOUT);
    }
    uint8_t* st = stage + slot * L.stage_stride;
    uint32_t* w1 = reinterpret_cast<uint32_t*>(st + kRaw1);
    uint32_t* w2 = reinterpret_cast<uint32_t*>(st + kRaw1 + FPC * bpf1);
    // non-identity 32-bit shuffles are applied once, in place, to the staged words
    preshuffle_slot(w1, FPC * bpf1 / 4, p.st[0].shkind, lut, w2, FPC * bpf2 / 4, p.st[1].shkind,
                    lut + 1024, tid, T);
    if (t == 0 && valid) finfo[g] = reinterpret_cast<const FrameInfo*>(st)[g];
    __syncthreads();
    if (*flag) break;
    const int s1 = valid ? finfo[g].s1 : 0;
    const int s2 = valid ? finfo[g].s2 : 0;
    const PackedStation pa{w1 + g * (bpf1 / 4), lv, (uint32_t)p.st[0].bits,
                           (1u << p.st[0].bits) - 1u, p.st[0].lsb ? 1 : 0, s1};
    const PackedStation pb{w2 + g * (bpf2 / 4), lv + 256, (uint32_t)p.st[1].bits,
                           (1u << p.st[1].bits) - 1u, p.st[1].lsb ? 1 : 0, s2};

    float2* za = bufA + g * Geom<N>::CSTRIDE;
    float2* zb = bufB + g * Geom<N>::CSTRIDE;
    first_pass_packed<N>(pa, pb, za, t);
    float2* Z0 = fft_rest<N>(za, zb, t, tw);
    // fft_rest opened with a barrier after the fused first pass: the staging
    // slot is consumed, refill it with iteration it + kStages
    if (tid == 0 && it + kStages < it1) {
      fence_proxy_async();
      issue(it + kStages);
    }
    __syncthreads();

    if (valid) {
      float2* o1 = reinterpret_cast<float2*>(p.out_a) + frame_local * H;
      float2* o2 = reinterpret_cast<float2*>(p.out_b) + frame_local * H;
      const float u1 = 0.5f / p.st[0].scale, u2 = 0.5f / p.st[1].scale;  // exact
      for (int k = t; k < H; k += T1) {
        const float2 a = Z0[k], b = Z0[(N - k) & (N - 1)];
        o1[k] = make_float2(u1 * (a.x + b.x), u1 * (a.y - b.y));
        o2[k] = make_float2(u2 * (a.y + b.y), -u2 * (a.x - b.x));
      }
    }
    __syncthreads();
  }
}

template <int N, int FPC>
__global__ void __launch_bounds__(FPC * N / 16, (N >= 8192 ? 1 : 2))
spectra_kernel(const CorrParams p) {
  extern __shared__ __align__(128) uint8_t smem[];
  const SmemLayout L = smem_layout<N, FPC>(p.stage_bytes);
  Twiddles<N> tw;
  corr_cta_init<N, FPC>(L, smem, tw);
  // ---- this CTA's iterations (FPC frame pairs each)
  const uint64_t iters = (p.nf + FPC - 1) / FPC;
  const uint64_t it0 = (blockIdx.x * iters) / gridDim.x;
  const uint64_t it1 = ((blockIdx.x + 1) * iters) / gridDim.x;
  stage_span<N, FPC>(p, it0, it1, smem, L, tw);
  corr_cta_drain(L, smem);
}

// Fixed-order sum of the per-CTA partials.  The multipliers (exact powers of
// two) undo the two-for-one 2x factor of each spectrum and the per-station
// level scaling.  Writes acf11, acf22, xcf (re,im) and zeroes the phased slot.
// A block covers 32 bins: each of its warps sums a contiguous share of the
// slots in slot order (coalesced 256-byte rows), then the warp sums are added
// in warp order; the order depends only on nblk, so the result is
// deterministic.  Bound by the latency of the slots' loads, a serial chain per
// warp: many slots take 32 warps and a block per column, so that a warp has all
// its loads (ten of 296 slots) in flight at once.  8 warps with all four
// columns took 40 us at the 296 slots of FFT 1024..4096 and 21 us at the 148 of
// FFT 8192; 32 warps take 7.4 and 10.1 us.  At the 33 slots of FFT 65536 it is
// the other way round: 9.4 us with 8 warps, 15 us with a block per column.
constexpr int kRedBins = 32;
constexpr int kRedWideSlots = 64;

// The sum of this thread's column and bin; in warp 0 only.
template <int WARPS>
__device__ __forceinline__ double reduce_column(const double* __restrict__ part, int nblk,
                                                size_t stride, int k, bool in,
                                                double (&sm)[WARPS][kRedBins]) {
  const int lane = threadIdx.x & 31, grp = threadIdx.x >> 5;
  const int b0 = (nblk * grp) / WARPS, b1 = (nblk * (grp + 1)) / WARPS;
  double s = 0.0;
  if (in) {
    const double* q = part + (size_t)b0 * stride + k;
#pragma unroll 10
    for (int b = b0; b < b1; ++b, q += stride) s += *q;
  }
  sm[grp][lane] = s;
  __syncthreads();
  double t = 0.0;
  if (grp == 0) {
#pragma unroll
    for (int g = 0; g < WARPS; ++g) t += sm[g][lane];
  }
  return t;
}

__device__ __forceinline__ void reduce_store(int v, int k, int h, double t, double m11, double m22,
                                             double m12, double* __restrict__ out) {
  if (v < 2) out[(size_t)v * h + k] = (v ? m22 : m11) * t;
  else out[2 * (size_t)h + 2 * k + (v - 2)] = m12 * t;
  if (v == 0) out[4 * (size_t)h + k] = 0.0;
}

// One column per block (blockIdx.y), 32 warps.
__global__ void __launch_bounds__(kRedBins * 32)
reduce_partials_wide_kernel(const double* __restrict__ part, int nblk, int h, double m11,
                            double m22, double m12, double* __restrict__ out) {
  __shared__ double sm[32][kRedBins];
  const int k = blockIdx.x * kRedBins + (threadIdx.x & 31), v = blockIdx.y;
  grid_wait();
  const double t = reduce_column<32>(part + (size_t)v * h, nblk, (size_t)4 * h, k, k < h, sm);
  if (threadIdx.x < kRedBins && k < h) reduce_store(v, k, h, t, m11, m22, m12, out);
}

// All four columns per block, 8 warps.
__global__ void __launch_bounds__(kRedBins * 8)
reduce_partials_kernel(const double* __restrict__ part, int nblk, int h, double m11, double m22,
                       double m12, double* __restrict__ out) {
  __shared__ double sm[8][4][kRedBins];
  const int lane = threadIdx.x & 31, grp = threadIdx.x >> 5;
  const int k = blockIdx.x * kRedBins + lane;
  const int b0 = (nblk * grp) / 8, b1 = (nblk * (grp + 1)) / 8;
  double s[4] = {0, 0, 0, 0};
  grid_wait();
  if (k < h) {
    for (int b = b0; b < b1; ++b) {
      const double* q = part + (size_t)b * 4 * h + k;
#pragma unroll
      for (int v = 0; v < 4; ++v) s[v] += q[(size_t)v * h];
    }
  }
#pragma unroll
  for (int v = 0; v < 4; ++v) sm[grp][v][lane] = s[v];
  __syncthreads();
  if (grp != 0 || k >= h) return;
#pragma unroll
  for (int v = 0; v < 4; ++v) {
    double t = 0.0;
#pragma unroll
    for (int g = 0; g < 8; ++g) t += sm[g][v][lane];
    reduce_store(v, k, h, t, m11, m22, m12, out);
  }
}

// Fixed-order sum of the per-CTA phased partials into acc[4H, 5H).
template <int WARPS>
__global__ void __launch_bounds__(kRedBins * WARPS)
reduce_phased_kernel(const double* __restrict__ part, int nblk, int h, int zero,
                     double* __restrict__ out) {
  __shared__ double sm[WARPS][kRedBins];
  const int k = blockIdx.x * kRedBins + (threadIdx.x & 31);
  grid_wait();
  const double t = reduce_column<WARPS>(part, nblk, (size_t)h, k, k < h, sm);
  if (threadIdx.x >= kRedBins || k >= h) return;
  out[4 * (size_t)h + k] = t;
  if (zero) {
    out[k] = out[(size_t)h + k] = 0.0;
    out[2 * (size_t)h + 2 * k] = out[2 * (size_t)h + 2 * k + 1] = 0.0;
  }
}

__global__ void delay_entries_kernel(const DelayParams p, uint64_t first, uint64_t nf,
                                     fxc_frame_delay_dev* out) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nf) return;
  int64_t i1, i2;
  double f1, f2;
  float2 l1, l2;
  frame_delay(p, first + i, &i1, &i2, &f1, &f2, &l1, &l2);
  fxc_frame_delay_dev d;
  d.int1 = i1;
  d.int2 = i2;
  d.frac1 = f1;
  d.frac2 = f2;
  d.fr_lo1[0] = l1.x;
  d.fr_lo1[1] = l1.y;
  d.fr_lo2[0] = l2.x;
  d.fr_lo2[1] = l2.y;
  out[i] = d;
}

__global__ void frame_info_kernel(const DelayParams p, uint64_t first, uint64_t nf, int n,
                                  double df_hz, int a1s, int a2s, FrameInfo* out) {
  grid_dependents();
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nf) return;
  FrameInfo fi;
  frame_info(p, first + i, n, df_hz, a1s, a2s, &fi);
  out[i] = fi;
}

// Last sector of the batch whose first frame (bins = false) or first bin
// (bins = true) is <= x; sectors are numbered in ascending order of both.
__device__ __forceinline__ uint32_t batch_find(const BatchScan* sc, uint32_t n, uint64_t x,
                                               bool bins) {
  uint32_t lo = 0, hi = n;
  while (hi - lo > 1) {
    const uint32_t m = (lo + hi) >> 1;
    const uint64_t st = bins ? sc[m].bin0 : sc[m].fi0;
    if (st <= x) lo = m;
    else hi = m;
  }
  return lo;
}

// Frame records of every sector of a batch (grid-stride over all frames);
// also rearms the groups' tickets for the launches that follow.
__global__ void batch_frame_info_kernel(const BatchArgs a) {
  const uint32_t ns = a.hdr->nscans;
  const uint64_t total = a.hdr->nframes;
  if (blockIdx.x == 0 && threadIdx.x < kBatchGroups) a.hdr->ticket[threadIdx.x] = 0;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t x = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; x < total; x += stride) {
    const BatchScan& b = a.hdr->scans[batch_find(a.hdr->scans, ns, x, false)];
    const uint64_t i = x - b.fi0;
    FrameInfo fi;
    frame_info(b.p.dl, b.p.first_frame + i, (int)b.n, b.p.df_hz, b.p.a1s, b.p.a2s, &fi);
    const_cast<FrameInfo*>(b.p.finfo)[i] = fi;
  }
}

// Fixed-order sum of each sector's item partials (grid-stride over all columns
// and bins of the batch, one thread each: a serial chain of loads per thread,
// so the more threads the better), with the same multipliers and output layout
// as reduce_partials_kernel (a phased sector: its power in [4H, 5H), the
// correlation columns zero, as reduce_phased_kernel after a zeroed block).
__global__ void batch_reduce_kernel(const BatchArgs a) {
  const uint32_t ns = a.hdr->nscans;
  const uint64_t total = 4 * a.hdr->nbins;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t x = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; x < total; x += stride) {
    const BatchScan& b = a.hdr->scans[batch_find(a.hdr->scans, ns, x >> 2, true)];
    const uint32_t h = b.h, r = (uint32_t)(x - 4 * b.bin0);
    const uint32_t v = r / h, k = r % h;
    double* out = b.acc;
    const size_t slot = b.phased ? h : 4 * (size_t)h;
    const double* q = a.partials + b.part + (b.phased ? k : r);
    double t = 0.0;
    if (!b.phased || v == 0) {
#pragma unroll 8
      for (uint32_t i = 0; i < b.nparts; ++i, q += slot) t += *q;
    }
    if (b.phased) {
      // phased power: H partials per item
      if (v == 0) out[4 * (size_t)h + k] = t;
      else if (v == 1) out[k] = out[h + k] = 0.0;
      else if (v == 2) out[2 * (size_t)h + 2 * k] = out[2 * (size_t)h + 2 * k + 1] = 0.0;
    } else {
      reduce_store((int)v, (int)k, (int)h, t, b.m11, b.m22, b.m12, out);
    }
  }
}

// ------------------------------------------------------------- launchers

template <int N, int FPC>
static cudaError_t launch_one(const CorrParams& p, int grid, cudaStream_t stream) {
  const SmemLayout L = smem_layout<N, FPC>(p.stage_bytes);
  auto kern = spectra_kernel<N, FPC>;
  // the limit is shared by every host thread: always the largest layout
  // (8-bit stations), never lowered under a concurrent launch
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)smem_layout<N, FPC>(2u * FPC * N).total);
  if (e != cudaSuccess) return e;
  kern<<<grid, FPC * N / 16, L.total, stream>>>(p);
  return cudaGetLastError();
}

int corr_frames_per_cta_iter(uint32_t n) {
  return n == 1024 ? 4 : (n == 2048 ? 2 : 1);
}

int corr_ctas_per_sm(uint32_t n) { return n >= 8192 ? 1 : 2; }

cudaError_t launch_corr(uint32_t n, const CorrParams& p, int grid, cudaStream_t s) {
  // FFT 16384 as two 8192-point rows; odd band shifts take other kernels
  if (n == 8192) return launch_corr_fold(p, grid, s);
  if (n == 16384) return launch_corr_fold2(p, grid, s);
  return launch_corr_small(n, p, grid, s);
}

cudaError_t launch_spectra(uint32_t n, const CorrParams& p, int grid, cudaStream_t s) {
  switch (n) {
    case 1024: return launch_one<1024, 4>(p, grid, s);
    case 2048: return launch_one<2048, 2>(p, grid, s);
    case 4096: return launch_one<4096, 1>(p, grid, s);
    case 8192: return launch_one<8192, 1>(p, grid, s);
    default: return cudaErrorInvalidValue;  // the four-step path
  }
}

// ------------------------------------------------------- batched launchers

uint32_t fold_batch_smem_bytes(int rows);
cudaError_t prepare_fold_batch(int rows);
cudaError_t launch_fold_batch(int rows, const BatchArgs& a, int grp, int grid, cudaStream_t s);
int fold_batch_ctas_per_sm(int rows);

cudaError_t batch_prepare(int g, int fpc) {
  if (g == BG_8192 || g == BG_16384) return prepare_fold_batch(g == BG_8192 ? 1 : 2);
  return small_batch_prepare(g, fpc);
}

int batch_group_ctas_per_sm(int g, int fpc) {
  if (g == BG_8192 || g == BG_16384) return fold_batch_ctas_per_sm(g == BG_8192 ? 1 : 2);
  return small_batch_ctas_per_sm(g, fpc);
}

cudaError_t launch_batch_group(int g, int fpc, const BatchArgs& a, int grid, cudaStream_t s) {
  if (grid <= 0) return cudaErrorInvalidValue;
  if (g == BG_8192 || g == BG_16384) return launch_fold_batch(g == BG_8192 ? 1 : 2, a, g, grid, s);
  return launch_small_batch(g, fpc, a, grid, s);
}

cudaError_t launch_batch_frame_info(const BatchArgs& a, int grid, cudaStream_t s) {
  batch_frame_info_kernel<<<grid, 128, 0, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_batch_reduce(const BatchArgs& a, int grid, cudaStream_t s) {
  batch_reduce_kernel<<<grid, 256, 0, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_reduce(const double* part, int nblk, int h, double m11, double m22, double m12,
                          double* out, cudaStream_t s) {
  const int grid = (h + kRedBins - 1) / kRedBins;
  if (nblk >= kRedWideSlots)
    return launch_dependent(reduce_partials_wide_kernel, dim3(grid, 4), kRedBins * 32, 0, s, part,
                            nblk, h, m11, m22, m12, out);
  return launch_dependent(reduce_partials_kernel, dim3(grid), kRedBins * 8, 0, s, part, nblk, h, m11,
                          m22, m12, out);
}

cudaError_t launch_reduce_phased(const double* part, int nblk, int h, bool zero, double* out,
                                 cudaStream_t s) {
  const dim3 grid((h + kRedBins - 1) / kRedBins);
  const int z = zero ? 1 : 0;
  if (nblk >= kRedWideSlots)
    return launch_dependent(reduce_phased_kernel<32>, grid, kRedBins * 32, 0, s, part, nblk, h, z, out);
  return launch_dependent(reduce_phased_kernel<8>, grid, kRedBins * 8, 0, s, part, nblk, h, z, out);
}

cudaError_t launch_delay_entries(const DelayParams& p, uint64_t first, uint64_t nf,
                                 fxc_frame_delay_dev* out, cudaStream_t s) {
  if (nf == 0) return cudaSuccess;
  delay_entries_kernel<<<(unsigned)((nf + 255) / 256), 256, 0, s>>>(p, first, nf, out);
  return cudaGetLastError();
}

cudaError_t launch_frame_info(const DelayParams& p, uint64_t first, uint64_t nf, int n,
                              double df_hz, int a1s, int a2s, FrameInfo* out, cudaStream_t s) {
  if (nf == 0) return cudaSuccess;
  frame_info_kernel<<<(unsigned)((nf + 127) / 128), 128, 0, s>>>(p, first, nf, n, df_hz, a1s,
                                                                   a2s, out);
  return cudaGetLastError();
}

}  // namespace fxc
