// phased_kernels.cu — phased-array synthesis for sm_100a (yi-phasedarray,
// src/main.rs:2222-2412).
//
// Per frame pair, after the same staging / decode / shift / shared two-for-one
// FFT front end as the correlation kernel:
//   1. S1, S2 from the shared spectrum, each rotated by its own fractional
//      delay exp(-2 pi i k df frac_i) with the Nyquist imaginary part zeroed
//      (apply_delay_and_rate_regular_bins, src/utils.rs:69-124);
//   2. fringe phasors fr_lo1 / fr_lo2, band alignment onto the output grid
//      and the weighted sum cb = w1 S1 + w2 S2 (src/main.rs:2264-2280);
//   3. |cb|^2 accumulated per bin (f32 registers, f64 flushes);
//   4. for the .raw product: cb[0].im = cb[N/2].im = 0, the inverse real FFT
//      computed as the forward FFT of the Hermitian-extended conj(cb) scaled by
//      1/N (src/utils.rs:60-66), odd samples negated when both inputs are LSB,
//      nearest-level re-quantisation with ant1's levels and packing with ant1's
//      shuffle (quantise_frame, src/utils.rs:378-410).
//
// Bound by instruction issue (59 % of the slots, 16 warps per SM): two FFTs, the
// synthesis and the re-quantiser are 34.2k warp instructions per frame pair of
// FFT 4096 with a search of the levels for every sample and the spectrum written
// as two planes of the Hermitian extension.  With the spectrum kept by bin (one
// 8-byte store; the inverse's first pass mirrors as it reads), thresholds
// instead of the search, and 1- and 2-bit samples quantised in the registers of
// the last pass (votes, no exchange): FFT 1024, 50001 frame pairs 620 -> 471 us,
// 2048 1208 -> 908, 4096 (20000) 1004 -> 745, 8192 (12503) 1348 -> 1015 us; 8-bit
// FFT 8192 2097 -> 1322 us; the .raw bytes are the same.  Decoding from the raw words
// as the correlation kernels do (one barrier and a rewrite of every shuffled word
// less): 462 -> 431 us, 4096 733 -> 681, 8192 1011 -> 972, 4-bit FFT 1024 584 -> 547 us.
#include <cuda_runtime.h>
#include <stdint.h>

#include "decode_tables.cuh"
#include "fold_decode.cuh"
#include "fxc_device.cuh"
#include "fxc_kernels.h"

namespace fxc {

constexpr uint32_t kQuantBytes = (kQuantFloats * 4 + 15) / 16 * 16;

// Shared memory: decode tables (levels and rotate amounts, decode_tables.cuh),
// frame records, mbarriers, flag and ticket, byte LUTs of 4- and 8-bit generic
// shuffles, quantiser and encode tables, the two buffers, the staging slots
// [FPC FrameInfo][FPC frames of station 1][FPC frames of station 2].
template <int N, int FPC>
struct PhasedLayout {
  static constexpr uint32_t FI = kTabPos + 256;
  static constexpr uint32_t BAR = FI + FPC * kFiBytes;
  static constexpr uint32_t FLAG = BAR + kStages * 8;
  static constexpr uint32_t TICKET = FLAG + 4;
  static constexpr uint32_t LUT = (FLAG + 8 + 15) / 16 * 16;
  static constexpr uint32_t QL = LUT + 8192;
  static constexpr uint32_t ENC = QL + kQuantBytes;
  static constexpr uint32_t A = (ENC + 4096 + 127) / 128 * 128;
  static constexpr uint32_t B = A + FPC * Geom<N>::CSTRIDE * 8;
  static constexpr uint32_t STAGE = (B + FPC * Geom<N>::CSTRIDE * 8 + 127) / 128 * 128;
  __host__ __device__ static constexpr uint32_t stride(uint32_t raw) {
    return (FPC * kFiBytes + raw + 127u) & ~127u;
  }
  __host__ __device__ static constexpr uint32_t total(uint32_t raw) {
    return STAGE + kStages * stride(raw);
  }
};

// Per-CTA state that outlives one sector: the twiddle bases and the number of
// staging iterations consumed so far (it sets the mbarrier slot and phase, so
// a persistent CTA can run spans of several scans back to back).
template <int N>
struct PhasedCta {
  Twiddles<N> tw;
  uint32_t seq;
};

template <int N, int FPC>
__device__ __forceinline__ void phased_cta_init(uint8_t* smem, PhasedCta<N>& c) {
  using L = PhasedLayout<N, FPC>;
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
__device__ __forceinline__ void phased_cta_drain(uint8_t* smem) {
  using L = PhasedLayout<N, FPC>;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BAR);
  if (threadIdx.x == 0 && *reinterpret_cast<const int*>(smem + L::FLAG))
    for (int s = 0; s < kStages; ++s) mbar_wait(&bars[s], 0, kWaitPolls);
}

// CTA iterations [it0, it1) (FPC frame pairs each) of the sector p: phased
// power per bin into part[H] (f32 registers, f64 flushes) and, with
// p.want_raw, the re-quantised frames at p.raw_out.  Returns false when a
// bounded wait gave up (the CTA must stop).  Compiled once (not inlined) and
// called by both the single-scan and the batched kernel, so that a frame's
// .raw bytes do not depend on which of them computed it: two inlined copies
// may contract or schedule the floating-point operations differently, which
// moves samples that sit on a quantiser decision boundary.
template <int N, int FPC>
__device__ __noinline__ bool phased_span(const PhasedParams& p, uint64_t it0, uint64_t it1,
                                            double* part, uint8_t* smem, uint32_t raw_bytes,
                                            PhasedCta<N>& c) {
  using L = PhasedLayout<N, FPC>;
  constexpr int T1 = N / 16;
  constexpr int T = FPC * T1;
  constexpr int BPT = (N / 2) / T;
  static_assert(BPT * T == N / 2 && BPT >= 2, "bins per thread");

  float2* bufA = reinterpret_cast<float2*>(smem + L::A);
  float2* bufB = reinterpret_cast<float2*>(smem + L::B);
  uint8_t* stage = smem + L::STAGE;
  const uint32_t stride = L::stride(raw_bytes);
  uint32_t* lut = reinterpret_cast<uint32_t*>(smem + L::LUT);
  const uint32_t* pos = reinterpret_cast<const uint32_t*>(smem + kTabPos);
  FrameInfo* finfo = reinterpret_cast<FrameInfo*>(smem + L::FI);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BAR);
  int* flag = reinterpret_cast<int*>(smem + L::FLAG);
  float* ql = reinterpret_cast<float*>(smem + L::QL);  // levels and thresholds
  uint32_t* elut = reinterpret_cast<uint32_t*>(smem + L::ENC);  // [4][256] encode LUT

  const int tid = threadIdx.x;
  const int g = tid / T1;
  const int t = tid % T1;
  const Twiddles<N>& tw = c.tw;
  const uint32_t seq0 = c.seq;

  const uint32_t bpf1 = p.st[0].bpf, bpf2 = p.st[1].bpf;
  constexpr uint32_t kRaw1 = FPC * kFiBytes;

  auto issue = [&](uint64_t it) {
    const int slot = (int)((seq0 + (uint32_t)(it - it0)) % kStages);
    const uint64_t f0 = it * FPC;
    const uint64_t nvalid = (p.nf - f0) < (uint64_t)FPC ? (p.nf - f0) : (uint64_t)FPC;
    const uint32_t bf = (uint32_t)(nvalid * kFiBytes);
    const uint32_t b1 = (uint32_t)(nvalid * bpf1), b2 = (uint32_t)(nvalid * bpf2);
    uint8_t* dst = stage + slot * stride;
    mbar_expect_tx(&bars[slot], bf + b1 + b2);
    bulk_g2s(dst, p.finfo + f0, bf, &bars[slot]);
    bulk_g2s(dst + kRaw1, p.st[0].raw + f0 * bpf1, b1, &bars[slot]);
    bulk_g2s(dst + kRaw1 + FPC * bpf1, p.st[1].raw + f0 * bpf2, b2, &bars[slot]);
  };
  // The previous span, if any, is past its last reads of the staging ring and
  // the tables: the first frames' copies go out, the tables are built while
  // they are in flight.
  __syncthreads();
  if (tid == 0) {
    fence_proxy_async();
    for (uint64_t it = it0; it < it1 && it < it0 + kStages; ++it) issue(it);
  }
  // 4- and 8-bit stations whose shuffle tears samples apart are rewritten in place
  // (byte LUTs), all others decoded from the raw words
  const bool pre1 = rewritten(p.st[0]);
  const bool pre2 = rewritten(p.st[1]);
  build_decode_tables_at<true>(p.st[0], p.st[1], pre1, pre2, smem, lut, tid, T);
  const bool split1 = split_2bit<true>(p.st[0]), split2 = split_2bit<true>(p.st[1]);
  for (int i = tid; i < kQuantFloats; i += T) ql[i] = p.qlevels[i];
  for (int i = tid; i < 1024; i += T) elut[i] = p.enc_lut[i];
  __syncthreads();

  float acc[BPT + 1];
#pragma unroll
  for (int i = 0; i <= BPT; ++i) acc[i] = 0.f;
  const int a1s = p.a1s, a1e = p.a1e, a2s = p.a2s;
  const int ov = a1e - a1s;
  const int sb = a2s - a1s;
  // undo the two-for-one factor 2 and the exact per-station level scaling
  const float u1 = 0.5f / p.st[0].scale, u2 = 0.5f / p.st[1].scale;
  bool first_flush = true;
  uint32_t since_flush = 0;
  const uint32_t spw = 32u / p.bits_out;           // samples per packed word
  const uint32_t wpf = (uint32_t)N / spw;          // words per output frame
  const uint32_t qmask = (p.bits_out >= 32) ? 0xFFFFFFFFu : ((1u << p.bits_out) - 1u);

  auto flush = [&]() {
#pragma unroll
    for (int i = 0; i <= BPT; ++i) {
      if (i == BPT && tid != 0) continue;
      const int bin = (i < BPT) ? (tid + T * i) : N / 2;
      double* q = part + bin;
      *q = (first_flush ? 0.0 : *q) + (double)acc[i];
      acc[i] = 0.f;
    }
    first_flush = false;
    since_flush = 0;
  };

  bool ok = true;
  for (uint64_t it = it0; it < it1; ++it) {
    const uint32_t q_it = seq0 + (uint32_t)(it - it0);
    const int slot = (int)(q_it % kStages);
    const uint32_t parity = (q_it / kStages) & 1u;
    const uint64_t frame_local = it * FPC + g;
    const bool valid = frame_local < p.nf;

    if (!mbar_wait(&bars[slot], parity, kWaitPolls)) {
      atomicOr(flag, 1);
      atomicOr(p.err, ERR_WAIT_TIMEOUT);
    }
    uint8_t* st = stage + slot * stride;
    uint32_t* w1 = reinterpret_cast<uint32_t*>(st + kRaw1);
    uint32_t* w2 = reinterpret_cast<uint32_t*>(st + kRaw1 + FPC * bpf1);
    if (pre1 || pre2) {  // CTA-uniform
      preshuffle_slot(w1, FPC * bpf1 / 4, pre1 ? p.st[0].shkind : SH_IDENTITY, lut, w2,
                      FPC * bpf2 / 4, pre2 ? p.st[1].shkind : SH_IDENTITY, lut + 1024, tid, T);
      __syncthreads();
    }
    float2* za = bufA + g * Geom<N>::CSTRIDE;
    float2* zb = bufB + g * Geom<N>::CSTRIDE;
    if (valid) {  // warp-uniform
      const FrameInfo* fs = reinterpret_cast<const FrameInfo*>(st) + g;
      const int b1 = p.st[0].bits, b2 = p.st[1].bits;
      const int s1 = fs->s1, s2 = fs->s2;
      const int m1 = t - s1, m2 = t - s2;
      const uint32_t tb1 = (uint32_t)((m1 & (p.st[0].lsb ? 1 : 0)) << (b1 + 2));
      const uint32_t tb2 = 2048u + (uint32_t)((m2 & (p.st[1].lsb ? 1 : 0)) << (b2 + 2));
      float2 v[16];
      fold::row_station<N, false>(b1, split1, w1 + g * (bpf1 / 4), smem, s1,
                                  pos[m1 & ((32 / b1) - 1)], tb1, v, t);
      fold::row_station<N, true>(b2, split2, w2 + g * (bpf2 / 4), smem, s2,
                                 pos[32 + (m2 & ((32 / b2) - 1))], tb2, v, t);
      if (t == 0) finfo[g] = *fs;
      dft16(v);
      float2* dst = za + 17 * t;  // cpad(16 t + r) = 17 t + r
#pragma unroll
      for (int r = 0; r < 16; ++r) dst[r] = v[out_pos<16>(r)];
    }
    float2* Z0 = fft_rest<N>(za, zb, t, tw);
    // fft_rest opened with a barrier after the first pass: the staging slot is
    // consumed, refill it.  Not after a wait gave up (flagged before it).
    if (tid == 0 && it + kStages < it1 && !*flag) {
      fence_proxy_async();
      issue(it + kStages);
    }
    const bool fin_b = Z0 != za;
    const bool stop = *flag != 0;  // not written between the first barrier and the next frame
    __syncthreads();
    if (stop) {
      ok = false;
      break;
    }

    // ---- per-bin synthesis over every valid frame of the iteration; cb goes
    // by bin to the buffer that does not hold Z
#pragma unroll 1
    for (int f = 0; f < FPC; ++f) {
      if (it * FPC + f >= p.nf) break;
      const float2* Z = (fin_b ? bufB : bufA) + f * Geom<N>::CSTRIDE;
      float2* cbs = (fin_b ? bufA : bufB) + f * Geom<N>::CSTRIDE;
      const FrameInfo& F = finfo[f];
      // spectrum of station s at its own bin k: unscaled, rotated by the
      // station's fractional delay, Nyquist imaginary part zeroed, times fr_lo
      auto station_bin = [&](int s, int k) -> float2 {
        const float2 a = Z[k], b = Z[(N - k) & (N - 1)];
        float2 v = s == 0 ? make_float2(u1 * (a.x + b.x), u1 * (a.y - b.y))
                          : make_float2(u2 * (a.y + b.y), u2 * (b.x - a.x));
        float sn, cs;
        __sincosf((float)k * (s == 0 ? F.st1 : F.st2), &sn, &cs);
        v = cmul(v, make_float2(cs, sn));
        if (k == N / 2) v.y = 0.f;
        return cmul(v, s == 0 ? F.fr_lo1 : F.fr_lo2);
      };
      auto bin_cb = [&](int k) -> float2 {
        float2 a1 = make_float2(0.f, 0.f), a2 = make_float2(0.f, 0.f);
        if (p.grid == 0) {
          a1 = station_bin(0, k);
          if (k >= a1s && k < a1e) a2 = station_bin(1, k + sb);
        } else {
          a2 = station_bin(1, k);
          if (k >= a2s && k < a2s + ov) a1 = station_bin(0, k - sb);
        }
        return make_float2(a1.x * p.w1 + a2.x * p.w2, a1.y * p.w1 + a2.y * p.w2);
      };
      auto emit = [&](int k, float2 cb) {
        if (k == 0 || k == N / 2) cb.y = 0.f;
        cbs[k] = cb;
      };
#pragma unroll
      for (int i = 0; i < BPT; ++i) {
        const int k = tid + T * i;
        const float2 cb = bin_cb(k);
        acc[i] += cnorm2(cb);
        if (p.want_raw) emit(k, cb);
      }
      if (tid == 0) {
        const float2 cb = bin_cb(N / 2);
        acc[BPT] += cnorm2(cb);
        if (p.want_raw) emit(N / 2, cb);
      }
    }
    if (++since_flush >= p.flush_every) flush();

    if (p.want_raw) {
      __syncthreads();
      // inverse real FFT of frame slot g: forward FFT of the Hermitian extension
      // of conj(cb), real part / N.  First pass: x[n] = conj(cb[n]) for n <= N/2,
      // cb[N - n] above.
      float2* qa = (fin_b ? bufB : bufA) + g * Geom<N>::CSTRIDE;  // free: Z consumed
      float2* qb = (fin_b ? bufA : bufB) + g * Geom<N>::CSTRIDE;
      float2 v[16];
#pragma unroll
      for (int r = 0; r < 16; ++r) {
        const int n = t + r * T1;
        const float2 cb = qb[r < 8 || n == N / 2 ? n : N - n];
        v[r] = make_float2(cb.x, r < 8 || n == N / 2 ? -cb.y : cb.y);
      }
      dft16(v);
      {
        float2* dst = qa + 17 * t;  // cpad(16 t + r) = 17 t + r
#pragma unroll
        for (int r = 0; r < 16; ++r) dst[r] = v[out_pos<16>(r)];
      }
      const float inv_n = 1.0f / (float)N;
      uint32_t* out = reinterpret_cast<uint32_t*>(p.raw_out + frame_local * p.bpf_out);
      const Quantiser quant{ql, (int)p.nqlevels, p.qmonotonic, p.qkind, p.qhi, p.qstep, p.qoffset};
      auto encode = [&](uint32_t word) -> uint32_t {  // ant1's shuffle
        return elut[word & 255u] | elut[256 + ((word >> 8) & 255u)] |
               elut[512 + ((word >> 16) & 255u)] | elut[768 + (word >> 24)];
      };
      constexpr int R = fft_last_radix<N>;
      fft_rest_values<N>(qa, qb, t, tw, v);
      if (p.bits_out <= 2 && p.qkind == QUANT_COMPARE) {
        // 1- and 2-bit output: a warp holds 32 consecutive samples in each of
        // its 16 output registers; the comparisons with the thresholds are
        // collected by votes, 32 codes at a time, and lane q of each half
        // keeps row q.  (Codes by way of shared memory, as below: 2-bit FFT 8192
        // 972 us against 959, FFT 1024 444 against 433, 1-bit 432 against 413.)
        if (valid) {
          const uint32_t lane = (uint32_t)t & 31u;
          const uint32_t flip = p.out_lsb ? lane << 31 : 0u;  // odd samples negated
          float top = 0.f;
#pragma unroll
          for (int q = 0; q < 16; ++q) {
            v[q].x = __uint_as_float(__float_as_uint(v[q].x * inv_n) ^ flip);
            top = fmaxf(top, fabsf(v[q].x));
          }
          const float t1 = ql[257], t2 = ql[258], t3 = ql[259];
          uint32_t lo = 0, hi = 0;
          if (__all_sync(0xFFFFFFFFu, top <= p.qhi)) {
#pragma unroll
            for (int q = 0; q < 16; ++q) {
              const float x = v[q / R * R + out_pos<R>(q % R)].x;
              const uint32_t b1 = __ballot_sync(0xFFFFFFFFu, x >= t1);
              const uint32_t b2 = __ballot_sync(0xFFFFFFFFu, x >= t2);
              const uint32_t b3 = __ballot_sync(0xFFFFFFFFu, x >= t3);
              if ((lane & 15u) == (uint32_t)q) {
                lo = b1 ^ b2 ^ b3;
                hi = b2;
              }
            }
          } else {
#pragma unroll 1
            for (int q = 0; q < 16; ++q) {
              float x = 0.f;  // a runtime index would move v to local memory
#pragma unroll
              for (int k = 0; k < 16; ++k)
                if (k == q) x = v[k / R * R + out_pos<R>(k % R)].x;
              const uint32_t c = nearest_level(x, ql, (int)p.nqlevels, p.qmonotonic);
              const uint32_t b0 = __ballot_sync(0xFFFFFFFFu, (c & 1u) != 0);
              const uint32_t b1 = __ballot_sync(0xFFFFFFFFu, (c & 2u) != 0);
              if ((lane & 15u) == (uint32_t)q) {
                lo = b0;
                hi = b1;
              }
            }
          }
          // row q: samples n0 + 0..31
          const uint32_t q = lane & 15u;
          const uint32_t n0 = ((uint32_t)t & ~31u) + T1 * (q / R) + (N / R) * (q % R);
          if (p.bits_out == 1) {
            if (lane < 16u) out[n0 / 32u] = encode(lo);
          } else {
            auto spread = [](uint32_t x) -> uint32_t {  // bit i to bit 2 i
              x = (x | (x << 8)) & 0x00FF00FFu;
              x = (x | (x << 4)) & 0x0F0F0F0Fu;
              x = (x | (x << 2)) & 0x33333333u;
              return (x | (x << 1)) & 0x55555555u;
            };
            const uint32_t sh = lane & 16u;
            const uint32_t word = spread((lo >> sh) & 0xFFFFu) | (spread((hi >> sh) & 0xFFFFu) << 1);
            out[n0 / 16u + (lane >> 4)] = encode(word);
          }
        }
      } else {
        // wider output (or a table without thresholds): the codes of the last
        // pass's samples, one byte each, go into the buffer that pass does not read
        // and are packed after a barrier.  Against samples written there and
        // gathered by word, an inlined search each: 4-bit stations at FFT 8192
        // (12503 frame pairs) 1222 -> 1048 us, at FFT 1024 (50001) 546 -> 481 us.
        uint8_t* codes = reinterpret_cast<uint8_t*>(fft_last_reads_b<N> ? qa : qb);
        const float3 thr = make_float3(ql[257], ql[258], ql[259]);
        const float in = p.out_lsb && (t & 1) ? -inv_n : inv_n;  // odd samples negated
#pragma unroll
        for (int q0 = 0; q0 < 16; q0 += 4) {
          float x[4];
          uint32_t c[4];
#pragma unroll
          for (int k = 0; k < 4; ++k)
            x[k] = v[(q0 + k) / R * R + out_pos<R>((q0 + k) % R)].x * in;
          quantise_many<false, true>(x, quant, ql + 256, thr, c);
#pragma unroll
          for (int k = 0; k < 4; ++k)
            codes[t + T1 * ((q0 + k) / R) + (N / R) * ((q0 + k) % R)] = (uint8_t)(c[k] & qmask);
        }
        __syncthreads();
        if (valid) {
          for (uint32_t w = (uint32_t)t; w < wpf; w += T1) {
            const uint32_t word = pack_codes(reinterpret_cast<const uint32_t*>(codes + w * spw),
                                             spw / 4, p.bits_out);
            out[w] = encode(word);
          }
        }
      }
    }
    __syncthreads();
  }
  if (since_flush > 0 || first_flush) flush();
  c.seq = seq0 + (uint32_t)(it1 - it0);
  return ok;
}

template <int N, int FPC>
__global__ void __launch_bounds__(FPC * N / 16, (N >= 8192 ? 1 : 2))
phased_kernel(const __grid_constant__ PhasedParams p) {
  constexpr int H = N / 2 + 1;
  extern __shared__ __align__(128) uint8_t smem[];
  PhasedCta<N> c;
  grid_dependents();
  phased_cta_init<N, FPC>(smem, c);
  grid_wait();  // the frame records
  const uint64_t iters = (p.nf + FPC - 1) / FPC;
  const uint64_t it0 = (blockIdx.x * iters) / gridDim.x;
  const uint64_t it1 = ((blockIdx.x + 1) * iters) / gridDim.x;
  phased_span<N, FPC>(p, it0, it1, p.partials + (size_t)blockIdx.x * H, smem, p.stage_bytes, c);
  phased_cta_drain<N, FPC>(smem);
}

// Batched: a persistent grid takes the items of batch group `grp` by ticket;
// an item is a frame range of one scan's phased sector (its own tables, frame
// records, raw words and .raw output) with its own H partials.  The layout is
// sized for 8-bit stations, so one launch serves every bit depth, and every
// frame is computed exactly as by phased_kernel.
template <int N, int FPC>
__global__ void __launch_bounds__(FPC * N / 16, (N >= 8192 ? 1 : 2))
phased_batch_kernel(const BatchArgs a, int grp) {
  extern __shared__ __align__(128) uint8_t smem[];
  if (blockIdx.x >= a.hdr->nitems[grp]) return;  // a graph launches the full grid
  uint32_t* ticket = reinterpret_cast<uint32_t*>(smem + PhasedLayout<N, FPC>::TICKET);
  PhasedCta<N> c;
  phased_cta_init<N, FPC>(smem, c);
  const uint32_t n_items = a.hdr->nitems[grp];
  const BatchItem* items = a.hdr->items + a.hdr->item0[grp];
  const BatchScan* scans = a.hdr->scans;
  for (;;) {
    if (threadIdx.x == 0) *ticket = atomicAdd(&a.hdr->ticket[grp], 1u);
    __syncthreads();
    const uint32_t k = *ticket;  // phased_span opens with a barrier before the next write
    if (k >= n_items) break;
    const BatchItem w = items[k];
    const uint64_t it0 = w.f0 / FPC, it1 = (w.f1 + FPC - 1) / FPC;
    if (!phased_span<N, FPC>(scans[w.scan].pp, it0, it1, a.partials + w.part, smem, 2u * FPC * N, c))
      break;
  }
  phased_cta_drain<N, FPC>(smem);
}

template <int N, int FPC>
static cudaError_t launch_phased_one(const PhasedParams& p, int grid, cudaStream_t stream) {
  const uint32_t smem = PhasedLayout<N, FPC>::total(p.stage_bytes);
  auto kern = phased_kernel<N, FPC>;
  // the limit is shared by every host thread: always the largest layout
  // (8-bit stations), never lowered under a concurrent launch
  cudaError_t e = cudaFuncSetAttribute(
      kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
      (int)(PhasedLayout<N, FPC>::total(2u * FPC * N)));
  if (e != cudaSuccess) return e;
  return launch_dependent(kern, dim3(grid), FPC * N / 16, smem, stream, p);
}

cudaError_t launch_phased(uint32_t n, const PhasedParams& p, int grid, cudaStream_t s) {
  switch (n) {
    case 1024: return launch_phased_one<1024, 4>(p, grid, s);
    case 2048: return launch_phased_one<2048, 2>(p, grid, s);
    case 4096: return launch_phased_one<4096, 1>(p, grid, s);
    case 8192: return launch_phased_one<8192, 1>(p, grid, s);
    default: return cudaErrorInvalidValue;
  }
}

namespace {
template <int N, int FPC>
uint32_t phased_batch_smem() {
  return PhasedLayout<N, FPC>::total(2u * FPC * N);
}
}  // namespace

// Batch groups of the phased kernels: FFT 1024 / 2048 / 4096 / 8192 with the
// single-scan kernels' frames per CTA iteration (4 / 2 / 1 / 1); FFT 16384
// is the two-row kernel's group (phased_pair.cu).
cudaError_t phased_batch_prepare(uint32_t n) {
  switch (n) {
    case 16384: return phased_pair_batch_prepare();
    case 1024: return cudaFuncSetAttribute(phased_batch_kernel<1024, 4>,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)phased_batch_smem<1024, 4>());
    case 2048: return cudaFuncSetAttribute(phased_batch_kernel<2048, 2>,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)phased_batch_smem<2048, 2>());
    case 4096: return cudaFuncSetAttribute(phased_batch_kernel<4096, 1>,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)phased_batch_smem<4096, 1>());
    case 8192: return cudaFuncSetAttribute(phased_batch_kernel<8192, 1>,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)phased_batch_smem<8192, 1>());
    default: return cudaErrorInvalidValue;
  }
}

int phased_batch_ctas_per_sm(uint32_t n) {
  int nb = 0;
  cudaError_t e = cudaErrorInvalidValue;
  switch (n) {
    case 1024: e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, phased_batch_kernel<1024, 4>,
                                                                 256, phased_batch_smem<1024, 4>());
      break;
    case 2048: e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, phased_batch_kernel<2048, 2>,
                                                                 256, phased_batch_smem<2048, 2>());
      break;
    case 4096: e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, phased_batch_kernel<4096, 1>,
                                                                 256, phased_batch_smem<4096, 1>());
      break;
    case 8192: e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, phased_batch_kernel<8192, 1>,
                                                                 512, phased_batch_smem<8192, 1>());
      break;
    case 16384: return phased_pair_batch_ctas_per_sm();
    default: break;
  }
  return e == cudaSuccess ? nb : 0;
}

int phased_frames_per_cta_iter(uint32_t n) { return n == 1024 ? 4 : (n == 2048 ? 2 : 1); }

cudaError_t launch_phased_batch(uint32_t n, const BatchArgs& a, int grp, int grid, cudaStream_t s) {
  switch (n) {
    case 1024: phased_batch_kernel<1024, 4><<<grid, 256, phased_batch_smem<1024, 4>(), s>>>(a, grp); break;
    case 2048: phased_batch_kernel<2048, 2><<<grid, 256, phased_batch_smem<2048, 2>(), s>>>(a, grp); break;
    case 4096: phased_batch_kernel<4096, 1><<<grid, 256, phased_batch_smem<4096, 1>(), s>>>(a, grp); break;
    case 8192: phased_batch_kernel<8192, 1><<<grid, 512, phased_batch_smem<8192, 1>(), s>>>(a, grp); break;
    case 16384: return launch_phased_pair_batch(a, grp, grid, s);
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

}  // namespace fxc
