// corr_small.cu — the correlation kernels of FFT 1024, 2048 and 4096
// (src/main.rs:2491-2568 per frame pair), single-sector and batched.
//
// A CTA runs FPC frame pairs at a time, N/16 threads each, both stations of a
// pair in one complex FFT.  The station whose bin grid the products are indexed
// on (the primary: station 1 for grid 0, station 2 for grid 1) is the real part,
// so the accumulation has no grid selects.  Per iteration:
//   1. the frames' records and packed words arrive by cp.async.bulk, two stages
//      deep, tracked by mbarriers;
//   2. a thread's 16 first-pass inputs of a station sit at one bit position of
//      16 words (fold_decode.cuh): word load, rotate, masked merge into a byte
//      offset of the level table; the LSB flip selects a negated copy.  Shuffles
//      of 1- and 2-bit stations and of whole samples are part of the rotate, those
//      that tear wider samples apart are applied in place by byte LUTs first;
//   3. radix-16 Stockham passes and the trailing radix-4 or -8 pass in padded
//      shared memory.  The three passes end in the buffer they began in, so the
//      next iteration begins in the other one and no barrier closes an iteration:
//      three barriers in all;
//   4. two-for-one split at the bin and at the band-shifted bin, |P|^2, |S|^2 and
//      P conj(S) times the phase ramp into f32 registers, flushed every 32 frames
//      (p.flush_every iterations) to f64 partials.  All sums run unconditionally:
//      out of the overlap the secondary spectrum is zero, and the flush leaves out
//      those bins and what was not asked for.
// Bound by instruction issue (66 % of the slots with 16 warps per SM; 1000 of 1660
// instructions per thread and frame pair of FFT 4096 are the FFT's and the sums'
// FP32).  Against the general form it replaced (words rewritten by LUT for every
// shuffle, a check and a sign per sample, grid selects and product predicates per
// bin, five barriers, partials loaded to add to them), sector calls of 31250 frame
// pairs, 2-bit, no band shift: FFT 1024 173 -> 141 us, 2048 291 -> 248, 4096 566 -> 488;
// 8-bit auto-spectra of FFT 2048 (20011), pairs of bits swapped, 204 -> 164; 4-bit
// against 2-bit cross-spectra of FFT 4096 (12207), LSB, shifted band 256 -> 228 us.
#include <cuda_runtime.h>
#include <stdint.h>

#include "decode_tables.cuh"
#include "fold_decode.cuh"
#include "fxc_device.cuh"
#include "fxc_kernels.h"

namespace fxc {
namespace {

// Shared memory: decode tables [0, 4352), frame records (double-buffered), mbarriers,
// flag and batch ticket, byte LUTs, the two buffers, the stages.
template <int N, int FPC>
struct SmallLayout {
  static constexpr uint32_t FI = kTabPos + 256;  // 2 FPC records
  static constexpr uint32_t BAR = FI + 2 * FPC * kFiBytes;
  static constexpr uint32_t FLAG = BAR + kStages * 8;
  static constexpr uint32_t TICKET = FLAG + 4;
  static constexpr uint32_t LUT = (FLAG + 8 + 15) / 16 * 16;
  static constexpr uint32_t BUF = (LUT + 8192 + 127) / 128 * 128;
  static constexpr uint32_t BUF_BYTES = FPC * Geom<N>::CSTRIDE * 8;
  static constexpr uint32_t STAGE = (BUF + 2 * BUF_BYTES + 127) / 128 * 128;
  __host__ __device__ static constexpr uint32_t stride(uint32_t raw) {
    return (FPC * kFiBytes + raw + 127u) & ~127u;
  }
  __host__ __device__ static constexpr uint32_t total(uint32_t raw) {
    return STAGE + kStages * stride(raw);
  }
};

// Per-CTA state that does not depend on the scan.
template <int N>
struct SmallCta {
  Twiddles<N> tw;
  uint32_t seq;  // staging iterations so far (mbarrier slot and phase, start buffer)
};

template <int N, int FPC>
__device__ __forceinline__ void small_cta_init(uint8_t* smem, SmallCta<N>& c) {
  using L = SmallLayout<N, FPC>;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BAR);
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) mbar_init(&bars[s], 1);
    *reinterpret_cast<int*>(smem + L::FLAG) = 0;
    fence_proxy_async();
  }
  c.tw.init(threadIdx.x % (N / 16));
  c.seq = 0;
}

// Never leave a bulk copy in flight into a finished CTA's shared memory.
template <int N, int FPC>
__device__ __forceinline__ void small_cta_drain(uint8_t* smem) {
  using L = SmallLayout<N, FPC>;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BAR);
  if (threadIdx.x == 0 && *reinterpret_cast<const int*>(smem + L::FLAG))
    for (int s = 0; s < kStages; ++s) mbar_wait(&bars[s], 0, kWaitPolls);
}

// Iterations [it0, it1) (FPC frame pairs each, frames below fend) of the sector
// described by p, into the f64 partials at part ([4][H]; slots: one for every flush).
// Returns false when a bounded wait gave up (the CTA must stop).
template <int N, int FPC>
__device__ __forceinline__ bool small_span(const CorrParams& p, uint64_t it0, uint64_t it1,
                                           uint64_t fend, double* part, bool slots, uint8_t* smem,
                                           uint32_t raw_bytes, SmallCta<N>& c) {
  using L = SmallLayout<N, FPC>;
  constexpr int T1 = N / 16;
  constexpr int T = FPC * T1;
  constexpr int H = N / 2 + 1;
  constexpr int BPT = (N / 2) / T;
  static_assert(BPT * T == N / 2 && BPT >= 2, "bins per thread");
  static_assert(Geom<N>::NPASS == 3, "the transform ends in the buffer it began in");
  FrameInfo* finfo = reinterpret_cast<FrameInfo*>(smem + L::FI);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BAR);
  int* flag = reinterpret_cast<int*>(smem + L::FLAG);
  uint32_t* lut = reinterpret_cast<uint32_t*>(smem + L::LUT);
  const uint32_t* pos = reinterpret_cast<const uint32_t*>(smem + kTabPos);
  float2* buf0 = reinterpret_cast<float2*>(smem + L::BUF);
  uint8_t* stage = smem + L::STAGE;
  const uint32_t stride = L::stride(raw_bytes);
  const int tid = threadIdx.x;
  const int g = tid / T1;  // frame slot of this thread in an iteration
  const int t = tid % T1;  // thread index within its frame pair
  const uint32_t seq0 = c.seq;

  const bool g0 = p.grid == 0;
  const StationParams& sp = p.st[g0 ? 0 : 1];
  const StationParams& ss = p.st[g0 ? 1 : 0];
  const bool preP = rewritten(sp);
  const bool preS = rewritten(ss);

  // slot: [FPC FrameInfo][FPC primary frames][FPC secondary frames]
  auto issue = [&](uint64_t it) {
    const uint32_t bP = sp.bpf, bS = ss.bpf;
    const int slot = (int)((seq0 + (uint32_t)(it - it0)) % kStages);
    const uint64_t f0 = it * FPC;
    const uint32_t nv = (fend - f0) < (uint64_t)FPC ? (uint32_t)(fend - f0) : (uint32_t)FPC;
    uint8_t* dst = stage + slot * stride;
    mbar_expect_tx(&bars[slot], nv * (kFiBytes + bP + bS));
    bulk_g2s(dst, p.finfo + f0, nv * kFiBytes, &bars[slot]);
    bulk_g2s(dst + FPC * kFiBytes, sp.raw + f0 * bP, nv * bP, &bars[slot]);
    bulk_g2s(dst + FPC * (kFiBytes + bP), ss.raw + f0 * bS, nv * bS, &bars[slot]);
  };
  // The previous span, if any, is past its last decode; its last spectra may
  // still be read, from the buffer that this span does not begin in.  The first
  // iterations' copies go out first, the tables are built meanwhile.
  __syncthreads();
  if (tid == 0) {
    fence_proxy_async();
    for (uint64_t it = it0; it < it1 && it < it0 + kStages; ++it) issue(it);
  }
  build_decode_tables_at<true>(sp, ss, preP, preS, smem, lut, tid, T);
  const bool splitP = split_2bit<true>(sp), splitS = split_2bit<true>(ss);
  __syncthreads();

  // Sums of bins tid + T i (and N/2 by thread 0): primary ACF, secondary ACF at
  // the primary's bin, XCF re, im.
  float acc[BPT + 1][4];
#pragma unroll
  for (int i = 0; i <= BPT; ++i)
#pragma unroll
    for (int v = 0; v < 4; ++v) acc[i][v] = 0.f;
  const int ov = p.a1e - p.a1s;
  const int ovs = g0 ? p.a1s : p.a2s;                   // overlap on the primary grid
  const int qoff = g0 ? p.a2s - p.a1s : p.a1s - p.a2s;  // secondary bin = primary bin + qoff
  uint32_t inov = 0;
#pragma unroll
  for (int i = 0; i <= BPT; ++i)
    if ((unsigned)((i < BPT ? tid + T * i : N / 2) - ovs) < (unsigned)ov) inov |= 1u << i;
  // every bin of the warp in the overlap (bin N/2 apart)
  const bool whole = __all_sync(0xFFFFFFFFu, (inov & ((1u << BPT) - 1u)) == (1u << BPT) - 1u);
  const bool want_xcf = (p.products & 2u) != 0;
  const uint32_t flush_every = p.flush_every;
  bool first_flush = true;
  uint32_t since_flush = 0;

  // Each address is this thread's alone: the atomics are additions that nothing
  // waits for, in order (corr_fold.cu).
  auto flush = [&]() {
    const bool want_acf = (p.products & 1u) != 0, ov_only = (p.products & 16u) != 0;
    const int colP = g0 ? 0 : 1, colS = g0 ? 1 : 0;  // output columns of the two ACFs
#pragma unroll
    for (int i = 0; i <= BPT; ++i) {
      if (i == BPT && tid != 0) continue;
      const int bin = (i < BPT) ? (tid + T * i) : N / 2;
      const bool in = (inov >> i) & 1u;
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        float x = acc[i][v];
        // (a zero secondary spectrum times an infinite or NaN primary bin is NaN)
        if (!(v < 2 ? want_acf : want_xcf) || (!in && (v > 0 || ov_only))) x = 0.f;
        if (v == 3 && !g0) x = -x;  // grid 1: the conjugate was summed
        double* q = part + (size_t)(v == 0 ? colP : (v == 1 ? colS : v)) * H + bin;
        if (first_flush || slots) *q = 0.0 + (double)x;
        else atomicAdd(q, (double)x);
        acc[i][v] = 0.f;
      }
    }
    first_flush = false;
    since_flush = 0;
    if (slots) part += 4 * H;
  };

  bool ok = true;
  for (uint64_t it = it0; it < it1; ++it) {
    const uint32_t q_it = seq0 + (uint32_t)(it - it0);
    const int slot = (int)(q_it % kStages);
    const uint64_t frame = it * FPC + g;
    if (!mbar_wait(&bars[slot], (q_it / kStages) & 1u, kWaitPolls)) {
      atomicOr(flag, 1);
      atomicOr(p.err, ERR_WAIT_TIMEOUT);
    }
    uint8_t* st = stage + slot * stride;
    const FrameInfo* fs = reinterpret_cast<const FrameInfo*>(st) + g;
    uint32_t* wP = reinterpret_cast<uint32_t*>(st + FPC * kFiBytes);
    uint32_t* wS = reinterpret_cast<uint32_t*>(st + FPC * (kFiBytes + sp.bpf));
    FrameInfo* fi = finfo + (q_it & 1u) * FPC;
    if (preP || preS) {  // CTA-uniform
      preshuffle_slot(wP, FPC * sp.bpf / 4, preP ? sp.shkind : SH_IDENTITY, lut, wS,
                      FPC * ss.bpf / 4, preS ? ss.shkind : SH_IDENTITY, lut + 1024, tid, T);
      __syncthreads();
    }
    float2* za = buf0 + ((q_it & 1u) * FPC + g) * Geom<N>::CSTRIDE;
    float2* zb = buf0 + (((q_it & 1u) ^ 1u) * FPC + g) * Geom<N>::CSTRIDE;
    if (frame < fend) {  // warp-uniform
      float2 v[16];
      const int sP = g0 ? fs->s1 : fs->s2, sS = g0 ? fs->s2 : fs->s1;
      const int mP = t - sP, mS = t - sS;
      const uint32_t tbP = (uint32_t)((mP & (sp.lsb ? 1 : 0)) << (sp.bits + 2));
      // The secondary station enters odd frames negated, undone in the ramp:
      // the shared FFT's cross-station rounding leak then alternates in sign and
      // cancels over frames instead of biasing the XCF.
      const uint32_t tbS = 2048u + ((((uint32_t)mS & (ss.lsb ? 1u : 0u)) ^ (uint32_t)(frame & 1u))
                                    << (ss.bits + 2));
      fold::row_station<N, false>(sp.bits, splitP, wP + g * (sp.bpf / 4), smem, sP,
                                  pos[mP & ((32 / sp.bits) - 1)], tbP, v, t);
      fold::row_station<N, true>(ss.bits, splitS, wS + g * (ss.bpf / 4), smem, sS,
                                 pos[32 + (mS & ((32 / ss.bits) - 1))], tbS, v, t);
      if (t == 0) fi[g] = *fs;
      dft16(v);
      float2* dst = za + 17 * t;  // cpad(16 t + r) = 17 t + r
#pragma unroll
      for (int r = 0; r < 16; ++r) dst[r] = v[out_pos<16>(r)];
    }
    const float2* Z0 = fft_rest<N>(za, zb, t, c.tw);
    // fft_rest opened with a barrier after the first pass: the staging slot is
    // consumed, refill it.  Not after a wait gave up (flagged before it).
    if (tid == 0 && it + kStages < it1 && !*flag) {
      fence_proxy_async();
      issue(it + kStages);
    }
    // Z[N] = Z[0], so that the mirror index N - k needs no mask
    if (t == 0) const_cast<float2*>(Z0)[N] = Z0[0];
    const bool stop = *flag != 0;  // not written between the first and the last barrier
    __syncthreads();
    if (stop) {
      ok = false;
      break;
    }

    // ---- accumulate every valid frame of the iteration
    const float2* Zi = buf0 + (q_it & 1u) * FPC * Geom<N>::CSTRIDE;
#pragma unroll
    for (int f = 0; f < FPC; ++f) {
      if (it * FPC + f >= fend) break;
      const float2* Z = Zi + f * Geom<N>::CSTRIDE;
      const float2* U = Z + tid;             // Z[k]
      const float2* W = Z + (N - tid);       // Z[N - k]
      const float2* C = U + qoff;            // Z[k + qoff]
      const float2* D = W - qoff;            // Z[N - k - qoff]
      const FrameInfo& F = fi[f];
      const float sg = ((it * FPC + f) & 1u) ? -1.0f : 1.0f;  // secondary's sign in this frame
      // Ramp of owned bin tid + T i: SFU sin/cos (|angle| <= ~pi, absolute error
      // < 4e-7) at i = 0 and BPT / 2, short recurrences between.  XCF = S1
      // conj(S2): P conj(S) times the ramp for grid 0; for grid 1 its conjugate
      // is summed, P conj(S) times the ramp's conjugate.
      const float cj = g0 ? 1.0f : -1.0f;
      const float dphi = cj * F.dphi, phi0 = cj * F.phi0;
      const float2 mix = make_float2(sg * F.fr_mix.x, sg * cj * F.fr_mix.y);
      auto ramp = [&](int bin) -> float2 {
        float sn, cs;
        __sincosf(fmaf((float)(bin - ovs), dphi, phi0), &sn, &cs);
        return cmul(mix, make_float2(cs, sn));
      };
      auto bin_acc = [&](float2 u, float2 w, float2 s, float2 r, float* a) {
        const float2 pv = make_float2(u.x + w.x, u.y - w.y);  // 2 P[k]
        a[0] = fmaf(pv.x, pv.x, fmaf(pv.y, pv.y, a[0]));
        a[1] = fmaf(s.x, s.x, fmaf(s.y, s.y, a[1]));
        if (want_xcf) {
          const float2 x = cmulc(pv, s);
          a[2] = fmaf(x.x, r.x, fmaf(-x.y, r.y, a[2]));
          a[3] = fmaf(x.x, r.y, fmaf(x.y, r.x, a[3]));
        }
      };
      auto second = [](float2 cc, float2 d) -> float2 {  // 2 S[k + qoff]
        return make_float2(cc.y + d.y, d.x - cc.x);
      };
      float2 rot = make_float2(0.f, 0.f), rstep = rot, half = rot;
      if (want_xcf) {
        float sn, cs;
        rot = ramp(tid);
        half = ramp(tid + T * (BPT / 2));
        if (BPT > 2) {
          __sincosf((float)T * dphi, &sn, &cs);
          rstep = make_float2(cs, sn);
        }
      }
      if (BPT > 2 && qoff == 0) {  // no band shift: the secondary is at the same bin
#pragma unroll
        for (int i = 0; i < BPT; ++i) {
          if (i == BPT / 2) rot = half;
          const float2 u = U[T * i], w = W[-T * i];
          float2 s = second(u, w);
          if (!((inov >> i) & 1u)) s = make_float2(0.f, 0.f);
          bin_acc(u, w, s, rot, acc[i]);
          if (want_xcf && i + 1 < BPT && i + 1 != BPT / 2) rot = cmul(rot, rstep);
        }
      } else if (whole) {
#pragma unroll
        for (int i = 0; i < BPT; ++i) {
          if (i == BPT / 2) rot = half;
          bin_acc(U[T * i], W[-T * i], second(C[T * i], D[-T * i]), rot, acc[i]);
          if (want_xcf && i + 1 < BPT && i + 1 != BPT / 2) rot = cmul(rot, rstep);
        }
      } else {
#pragma unroll
        for (int i = 0; i < BPT; ++i) {
          if (i == BPT / 2) rot = half;
          float2 s = make_float2(0.f, 0.f);
          if ((inov >> i) & 1u) s = second(C[T * i], D[-T * i]);
          bin_acc(U[T * i], W[-T * i], s, rot, acc[i]);
          if (want_xcf && i + 1 < BPT && i + 1 != BPT / 2) rot = cmul(rot, rstep);
        }
      }
      if (tid == 0) {
        float2 s = make_float2(0.f, 0.f);
        if ((inov >> BPT) & 1u) s = second(Z[N / 2 + qoff], Z[N / 2 - qoff]);
        bin_acc(Z[N / 2], Z[N / 2], s, ramp(N / 2), acc[BPT]);
      }
    }
    if (++since_flush >= flush_every) flush();
  }
  if (ok && (since_flush > 0 || first_flush)) flush();
  c.seq = seq0 + (uint32_t)(it1 - it0);
  return ok;
}

}  // namespace

template <int N, int FPC>
__global__ void __launch_bounds__(FPC * N / 16, 2)
corr_small_kernel(const __grid_constant__ CorrParams p) {
  constexpr int H = N / 2 + 1;
  extern __shared__ __align__(128) uint8_t smem[];
  SmallCta<N> c;
  grid_dependents();
  small_cta_init<N, FPC>(smem, c);
  grid_wait();  // the frame records
  const uint64_t iters = (p.nf + FPC - 1) / FPC;
  const uint64_t it0 = (blockIdx.x * iters) / gridDim.x;
  const uint64_t it1 = ((blockIdx.x + 1) * iters) / gridDim.x;
  small_span<N, FPC>(p, it0, it1, p.nf, p.partials + (size_t)blockIdx.x * 4 * H, false,
                     smem, p.stage_bytes, c);
  small_cta_drain<N, FPC>(smem);
}

// Batched: a persistent grid takes the items of batch group `grp` by ticket;
// every item is a frame range of one scan's sector (frames aligned to FPC)
// with its own partials.  The layout is sized for the largest stage (8-bit
// stations), so one launch serves every bit depth.
template <int N, int FPC, int MINB>
__global__ void __launch_bounds__(FPC * N / 16, MINB)
corr_small_batch_kernel(const BatchArgs a, int grp) {
  extern __shared__ __align__(128) uint8_t smem[];
  if (blockIdx.x >= a.hdr->nitems[grp]) return;  // a graph launches the full grid
  uint32_t* ticket = reinterpret_cast<uint32_t*>(smem + SmallLayout<N, FPC>::TICKET);
  SmallCta<N> c;
  small_cta_init<N, FPC>(smem, c);
  const uint32_t n_items = a.hdr->nitems[grp];
  const BatchItem* items = a.hdr->items + a.hdr->item0[grp];
  const BatchScan* scans = a.hdr->scans;
  for (;;) {
    if (threadIdx.x == 0) *ticket = atomicAdd(&a.hdr->ticket[grp], 1u);
    __syncthreads();
    const uint32_t k = *ticket;  // small_span opens with a barrier before the next write
    if (k >= n_items) break;
    const BatchItem w = items[k];
    if (!small_span<N, FPC>(scans[w.scan].p, w.f0 / FPC, (w.f1 + FPC - 1) / FPC, w.f1,
                            a.partials + w.part, w.slots != 0, smem, 2u * FPC * N, c))
      break;
  }
  small_cta_drain<N, FPC>(smem);
}

// Decode + integer shift of FPC frame pairs a CTA iteration, by the correlation and
// phased kernels' own tables and inputs (fold::row_station), written out as f32
// samples (src/utils.rs:126-376).
template <int N, int FPC>
__global__ void __launch_bounds__(FPC * N / 16) row_decode_kernel(const CorrParams p) {
  constexpr int T1 = N / 16, T = FPC * T1;
  extern __shared__ __align__(128) uint8_t smem[];
  const int tid = threadIdx.x, g = tid / T1, t = tid % T1;
  const bool g0 = p.grid == 0;
  const StationParams& sp = p.st[g0 ? 0 : 1];
  const StationParams& ss = p.st[g0 ? 1 : 0];
  const bool preP = rewritten(sp), preS = rewritten(ss);
  const uint32_t* pos = reinterpret_cast<const uint32_t*>(smem + kTabPos);
  uint32_t* lut = reinterpret_cast<uint32_t*>(smem + kTabLut);
  uint32_t* wP = reinterpret_cast<uint32_t*>(smem + kTabEnd);
  uint32_t* wS = wP + FPC * (sp.bpf / 4);
  build_decode_tables_at<true>(sp, ss, preP, preS, smem, lut, tid, T);
  const bool splitP = split_2bit<true>(sp), splitS = split_2bit<true>(ss);
  float* outP = g0 ? p.out_a : p.out_b;
  float* outS = g0 ? p.out_b : p.out_a;
  const float uP = 1.0f / sp.scale, uS = 1.0f / ss.scale;  // powers of two: exact
  for (uint64_t f0 = (uint64_t)blockIdx.x * FPC; f0 < p.nf; f0 += (uint64_t)gridDim.x * FPC) {
    const uint32_t nv = (uint32_t)(p.nf - f0 < (uint64_t)FPC ? p.nf - f0 : (uint64_t)FPC);
    __syncthreads();  // tables built / previous frames' words consumed
    const uint4* gP = reinterpret_cast<const uint4*>(sp.raw + f0 * sp.bpf);
    const uint4* gS = reinterpret_cast<const uint4*>(ss.raw + f0 * ss.bpf);
    for (uint32_t i = tid; i < nv * sp.bpf / 16; i += T) reinterpret_cast<uint4*>(wP)[i] = gP[i];
    for (uint32_t i = tid; i < nv * ss.bpf / 16; i += T) reinterpret_cast<uint4*>(wS)[i] = gS[i];
    __syncthreads();
    if (preP || preS) {
      preshuffle_slot(wP, nv * sp.bpf / 4, preP ? sp.shkind : SH_IDENTITY, lut, wS, nv * ss.bpf / 4,
                      preS ? ss.shkind : SH_IDENTITY, lut + 1024, tid, T);
      __syncthreads();
    }
    if (g >= (int)nv) continue;
    const FrameInfo fi = p.finfo[f0 + g];
    const int sP = g0 ? fi.s1 : fi.s2, sS = g0 ? fi.s2 : fi.s1;
    const int mP = t - sP, mS = t - sS;
    const uint32_t tbP = (uint32_t)((mP & (sp.lsb ? 1 : 0)) << (sp.bits + 2));
    const uint32_t tbS = 2048u + (uint32_t)((mS & (ss.lsb ? 1 : 0)) << (ss.bits + 2));
    float2 v[16];
    fold::row_station<N, false>(sp.bits, splitP, wP + g * (sp.bpf / 4), smem, sP,
                                pos[mP & ((32 / sp.bits) - 1)], tbP, v, t);
    fold::row_station<N, true>(ss.bits, splitS, wS + g * (ss.bpf / 4), smem, sS,
                               pos[32 + (mS & ((32 / ss.bits) - 1))], tbS, v, t);
    float* oP = outP + (f0 + g) * N + t;
    float* oS = outS + (f0 + g) * N + t;
#pragma unroll
    for (int r = 0; r < 16; ++r) {
      oP[r * T1] = v[r].x * uP;
      oS[r * T1] = v[r].y * uS;
    }
  }
}

namespace {

template <int N, int FPC>
cudaError_t decode_one(const CorrParams& p, int sms, cudaStream_t s) {
  const uint64_t iters = (p.nf + FPC - 1) / FPC;
  const int grid = (int)(iters < (uint64_t)sms * 6 ? iters : (uint64_t)sms * 6);
  row_decode_kernel<N, FPC><<<grid, FPC * N / 16, kTabEnd + 2u * FPC * N, s>>>(p);
  return cudaGetLastError();
}

template <int N, int FPC>
cudaError_t launch_one(const CorrParams& p, int grid, cudaStream_t s) {
  // the limit is shared by every host thread: always the largest layout
  // (8-bit stations), never lowered under a concurrent launch
  cudaError_t e = cudaFuncSetAttribute(corr_small_kernel<N, FPC>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)SmallLayout<N, FPC>::total(2u * FPC * N));
  if (e != cudaSuccess) return e;
  return launch_dependent(corr_small_kernel<N, FPC>, dim3(grid), FPC * N / 16,
                          SmallLayout<N, FPC>::total(p.stage_bytes), s, p);
}

// Variants of the batched kernels: FFT length, frames per CTA iteration and
// resident CTAs per SM (shared memory with 8-bit staging: FPC*N = 1024 ->
// 34 KB, 2048 -> 56 KB, 4096 -> 99 KB, 8192 -> 185 KB).
template <int N, int FPC>
constexpr int batch_minb() {
  return FPC * N <= 1024 ? 6 : (FPC * N <= 2048 ? 4 : (FPC * N <= 4096 ? 2 : 1));
}
template <int N, int FPC>
uint32_t batch_smem() {
  return SmallLayout<N, FPC>::total(2u * FPC * N);
}
template <int N, int FPC>
cudaError_t batch_prepare_one() {
  return cudaFuncSetAttribute(corr_small_batch_kernel<N, FPC, batch_minb<N, FPC>()>,
                              cudaFuncAttributeMaxDynamicSharedMemorySize, (int)batch_smem<N, FPC>());
}
template <int N, int FPC>
int batch_ctas_one() {
  int nb = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(
          &nb, corr_small_batch_kernel<N, FPC, batch_minb<N, FPC>()>, FPC * N / 16,
          batch_smem<N, FPC>()) != cudaSuccess)
    return 0;
  return nb;
}
template <int N, int FPC>
cudaError_t batch_launch_one(const BatchArgs& a, int grp, int grid, cudaStream_t s) {
  corr_small_batch_kernel<N, FPC, batch_minb<N, FPC>()>
      <<<grid, FPC * N / 16, batch_smem<N, FPC>(), s>>>(a, grp);
  return cudaGetLastError();
}

// Returns CALL(N, FPC) for the variant (g, fpc) if there is one.
#define FXC_BATCH_VARIANTS(g, fpc, CALL)              \
  switch ((g) * 16 + (fpc)) {                         \
    case BG_1024 * 16 + 1: return CALL(1024, 1);      \
    case BG_1024 * 16 + 2: return CALL(1024, 2);      \
    case BG_1024 * 16 + 4: return CALL(1024, 4);      \
    case BG_2048 * 16 + 1: return CALL(2048, 1);      \
    case BG_2048 * 16 + 2: return CALL(2048, 2);      \
    case BG_2048 * 16 + 4: return CALL(2048, 4);      \
    case BG_4096 * 16 + 1: return CALL(4096, 1);      \
    case BG_4096 * 16 + 2: return CALL(4096, 2);      \
    default: break;                                   \
  }

}  // namespace

cudaError_t launch_corr_small(uint32_t n, const CorrParams& p, int grid, cudaStream_t s) {
  switch (n) {
    case 1024: return launch_one<1024, 4>(p, grid, s);
    case 2048: return launch_one<2048, 2>(p, grid, s);
    case 4096: return launch_one<4096, 1>(p, grid, s);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_row_decode(uint32_t n, const CorrParams& p, int sms, cudaStream_t s) {
  switch (n) {
    case 1024: return decode_one<1024, 4>(p, sms, s);
    case 2048: return decode_one<2048, 2>(p, sms, s);
    case 4096: return decode_one<4096, 1>(p, sms, s);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t small_batch_prepare(int g, int fpc) {
#define FXC_PREP(N, F) batch_prepare_one<N, F>()
  FXC_BATCH_VARIANTS(g, fpc, FXC_PREP)
#undef FXC_PREP
  return cudaErrorInvalidValue;
}

int small_batch_ctas_per_sm(int g, int fpc) {
#define FXC_CTAS(N, F) batch_ctas_one<N, F>()
  FXC_BATCH_VARIANTS(g, fpc, FXC_CTAS)
#undef FXC_CTAS
  return 0;
}

cudaError_t launch_small_batch(int g, int fpc, const BatchArgs& a, int grid, cudaStream_t s) {
#define FXC_LAUNCH(N, F) batch_launch_one<N, F>(a, g, grid, s)
  FXC_BATCH_VARIANTS(g, fpc, FXC_LAUNCH)
#undef FXC_LAUNCH
  return cudaErrorInvalidValue;
}

}  // namespace fxc
