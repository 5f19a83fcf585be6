// NVFP4 quantizer kernels for sm_100a: per-tensor amax, 1x16 row quantizer, transposed
// RHT16 quantizer, 16x16 weight quantizer (W and W^T), scale re-swizzle.  All HBM-bound:
// 128-bit coalesced loads, register-resident blocks, warp shuffles for exchanges/reductions.
#include <stdlib.h>

#include <mutex>
#include <unordered_map>
#include <vector>

#include "common.cuh"

namespace nvfp4 {

__device__ __forceinline__ void unpack8(const uint4& q, float* f) {
  const u32 w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
  for (int i = 0; i < 4; i++) {
    f[2 * i] = __uint_as_float(w[i] << 16);
    f[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
  }
}

__device__ __forceinline__ uint4 ldg128(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

// ------------------------------------------------------------------------------------------ amax
__device__ __forceinline__ uint4 ld_cg_128(const uint4* p) {
  uint4 v;
  asm volatile("ld.global.cg.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

// Meeting point of the blocks of one launch: running maximum and number of blocks done, both zero between launches.
struct AmaxSlot { u32 bits, done; };
constexpr int kAmaxSlots = 1024;
__device__ AmaxSlot g_amax_slots[kAmaxSlots];
struct AmaxWords { float v[8]; };
__device__ AmaxWords g_amax_words[kAmaxSlots];      // see nvfp4_amax_bf16_word

// Running maximum of |x| as integer bit patterns (non-negative floats order like unsigned ints): bf16 values in both
// halves of a word, FP32 values whole.
template <bool F32>
__device__ __forceinline__ u32 amax_take(u32 m, const uint4& v) {
  if (F32) return max(max(m, v.x & 0x7FFFFFFFu), max(max(v.y & 0x7FFFFFFFu, v.z & 0x7FFFFFFFu), v.w & 0x7FFFFFFFu));
  m = __vmaxu2(m, v.x & 0x7FFF7FFFu); m = __vmaxu2(m, v.y & 0x7FFF7FFFu);
  m = __vmaxu2(m, v.z & 0x7FFF7FFFu);
  return __vmaxu2(m, v.w & 0x7FFF7FFFu);
}

// HBM-bound: 5.0 to 5.2 TB/s on tensors of 134 to 403 MB, 7.1 at 2 GB, where the first loads and the uneven last round no
// longer count.  A thread keeps four loads in flight all the time (the oldest is
// consumed and replaced): batches of four with a wait in between left the memory idle once per batch, which on a tensor
// of two or three batches is a fifth of the time (46 MB: 11.0 -> 8.7 us; 33 MB from L2: 4.6 -> 3.8 us).
// Where the result goes:
//   slot null    raise *out, which is zero or a running maximum; `next`, if any, is a word to clear for a later launch
//   slot given   *out needs no clearing: every block raises the slot, the last one to arrive moves the result to *out and
//                leaves the slot zero (1.8 us for the two dependent atomics and fences; a memset in front is 1.4 us, a
//                launch, and no programmatic launch across it)
template <bool F32>
__global__ void __launch_bounds__(256) amax_kernel(const uint4* __restrict__ x, long long nv, float* out, float* next, AmaxSlot* slot) {
  pdl_trigger();
  pdl_wait();
  u32 m = 0u;
  const long long stride = (long long)gridDim.x * blockDim.x, last = nv - 1;
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (next && i == 0) *next = 0.f;
  uint4 v[4];
#pragma unroll
  for (int j = 0; j < 4; j++) v[j] = ld_cg_128(x + min(i + j * stride, last));      // a maximum does not mind reading the last one again
  for (i += 4 * stride; i - 4 * stride < nv;) {
#pragma unroll
    for (int j = 0; j < 4; j++) {
      m = amax_take<F32>(m, v[j]);
      if (i < nv) v[j] = ld_cg_128(x + i);
      i += stride;
    }
  }
  // bf16: NaN patterns (> 0x7F80) count as +inf;  FP32: a NaN is larger than every number and stays
  u32 mm = F32 ? m : min(max(m & 0xFFFFu, m >> 16), 0x7F80u) << 16;
  mm = __reduce_max_sync(0xffffffffu, mm);
  __shared__ u32 sm[8];
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = mm;
  __syncthreads();
  if (threadIdx.x < 32) {
    mm = __reduce_max_sync(0xffffffffu, sm[threadIdx.x & 7]);
    if (threadIdx.x == 0) {
      if (!slot) {
        if (mm) atomicMax(reinterpret_cast<unsigned*>(out), mm);
      } else if (gridDim.x == 1) {
        *out = __uint_as_float(mm);
      } else {
        if (mm) atomicMax(&slot->bits, mm);
        __threadfence();
        if (atomicAdd(&slot->done, 1u) == gridDim.x - 1) {
          __threadfence();
          *out = __uint_as_float(atomicExch(&slot->bits, 0u));
          atomicExch(&slot->done, 0u);
        }
      }
    }
  }
}

// ------------------------------------------------------------------------------------------ rows
template <bool WIDE>
__device__ __forceinline__ Block32 load_block(const __nv_bfloat16* p) {
  Block32 r;
  if (WIDE) {
    asm volatile("ld.global.nc.L1::no_allocate.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r.w[0]), "=r"(r.w[1]), "=r"(r.w[2]), "=r"(r.w[3]), "=r"(r.w[4]), "=r"(r.w[5]), "=r"(r.w[6]), "=r"(r.w[7])
                 : "l"(p));
  } else {
    const uint4 a = ldg128(p), b = ldg128(p + 8);
    r.w[0] = a.x; r.w[1] = a.y; r.w[2] = a.z; r.w[3] = a.w; r.w[4] = b.x; r.w[5] = b.y; r.w[6] = b.z; r.w[7] = b.w;
  }
  return r;
}

// One warp per (row, 512-column segment); a lane owns one 16-block (32 contiguous bytes, one
// 256-bit load when rows are 32-byte aligned), so the warp reads 1 KB contiguous and needs no
// exchange.  The next item's load is issued before the current one is processed.
template <int ROUNDING, bool WIDE>
__global__ void __launch_bounds__(256, 4) quant_rows_kernel(const __nv_bfloat16* __restrict__ x, long long ldx,
                                                          uint2* __restrict__ codes, unsigned char* __restrict__ scales,
                                                          const float* __restrict__ amax, int R, int C, int layout,
                                                          u32 seed, const u32* __restrict__ seed_dev,
                                                          float* __restrict__ gs_out) {
  if (ROUNDING != NVFP4_ROUND_NEAREST && seed_dev) seed = __ldg(seed_dev);
  const int lane = threadIdx.x & 31;
  const int nblk = C >> 4;
  unsigned char* scales_sw = layout == NVFP4_SCALES_BOTH ? scales + (long long)R * nblk : scales;
  const int nseg = (nblk + 31) >> 5;
  // walk (row, segment) pairs with a fixed warp stride, without a division per item
  const unsigned nwarps = gridDim.x * (blockDim.x >> 5);
  const unsigned w0 = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int dr = (int)(nwarps / (unsigned)nseg), ds = (int)(nwarps % (unsigned)nseg);
  int r = (int)(w0 / (unsigned)nseg), seg = (int)(w0 % (unsigned)nseg);
  Block32 cur = {};
  if (r < R && seg * 32 + lane < nblk) cur = load_block<WIDE>(x + (long long)r * ldx + (seg * 32 + lane) * 16);
  // (the first load is under way while the tables are built)
  __shared__ __align__(8) float lut[kLutFloats];
  const TensorScale ts = make_tensor_scale<ROUNDING>(__ldg(amax), 1.f, lut,
                                                     (blockIdx.x == 0 && threadIdx.x == 0) ? gs_out : nullptr);
  while (r < R) {
    int rn = r + dr, sn = seg + ds;
    if (sn >= nseg) { sn -= nseg; rn++; }
    Block32 nxt = {};
    if (rn < R && sn * 32 + lane < nblk) nxt = load_block<WIDE>(x + (long long)rn * ldx + (sn * 32 + lane) * 16);
    const int blk = seg * 32 + lane;
    if (blk < nblk) {
      u64 P[8];
#pragma unroll
      for (int i = 0; i < 8; i++) P[i] = f2_from_bf16x2(cur.w[i]);
      const u32 sb = block_scale_byte(absmax16(P), ts);
      const long long b = (long long)r * nblk + blk;
      codes[b] = quant_block16<ROUNDING>(P, sb, ts, seed, (u32)b, (u32)(b * 16));
      if (layout != NVFP4_SCALES_SWIZZLED) scales[b] = (unsigned char)sb;
      if (layout != NVFP4_SCALES_LINEAR) scales_sw[sw_off(r, blk, nblk >> 2)] = (unsigned char)sb;
    }
    r = rn; seg = sn; cur = nxt;
  }
}

// ------------------------------------------------------------------------------------------ cols + RHT16
// CTA tile: 64 columns x 256 tokens.  A thread loads 16 tokens x 4 columns with 16 64-bit loads (half-warp = 128
// contiguous bytes of one token row), under way while the tables are built, so each 16-token column block lives in its
// registers: sign flip, 4 butterfly stages, x0.25 and quantization need no shared memory.  The outputs do: 8 bytes of
// codes and a scale byte per (column, token block) would be stored 16 columns at a time, M / 2 bytes apart; staged, a
// half-warp writes 128 contiguous bytes of a column.  Issue-bound.  Against a tile of 128 columns, 8 per thread, stored
// directly: [2048, 1024] 7.2 -> 3.7 us, [16000, 5904] 78 -> 70, with the dither [5008, 1552] 12.4 -> 11.8.
template <int ROUNDING>
__global__ void __launch_bounds__(256, 3) quant_cols_rht_kernel(const __nv_bfloat16* __restrict__ x,
                                                              unsigned char* __restrict__ codes,
                                                              unsigned char* __restrict__ scales,
                                                              const float* __restrict__ amax, int M, int C, int layout,
                                                              u32 signs, u32 seed, const u32* __restrict__ seed_dev,
                                                              float* __restrict__ gs_out) {
  constexpr int kCols = 64, kMb = 16;                          // of a CTA tile: columns, 16-token blocks
  if (ROUNDING != NVFP4_ROUND_NEAREST && seed_dev) seed = __ldg(seed_dev);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c0 = blockIdx.x * kCols, mb0 = blockIdx.y * kMb;
  const int tc = (lane & 15) * 4, tm = warp * 2 + (lane >> 4); // this thread's first column and token block in the tile
  const int nmb = M >> 4;
  const bool in = c0 + tc < C && mb0 + tm < nmb;
  __shared__ __align__(8) float lut[kLutFloats];
  // codes of (column, block) at column * 128 + (block ^ (column / 4 % 16)) * 8: neither side meets a bank conflict
  __shared__ __align__(16) uint2 stage_codes[kCols * kMb];
  __shared__ __align__(16) unsigned char stage_scales[kCols * kMb];
  uint2 raw[16];
  const __nv_bfloat16* p = x + (long long)(mb0 + tm) * 16 * C + c0 + tc;
#pragma unroll
  for (int i = 0; i < 16; i++) {
    raw[i] = make_uint2(0u, 0u);
    if (in) asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0,%1}, [%2];" : "=r"(raw[i].x), "=r"(raw[i].y) : "l"(p + (long long)i * C));
  }
  // the x0.25 that follows the butterflies is folded into the tensor scale (a power of two)
  const TensorScale ts = make_tensor_scale<ROUNDING>(__ldg(amax), 4.f, lut,
      (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) ? gs_out : nullptr, 0.25f);
  if (in) {
    // apply the sign vector on the packed bf16 words: token i is negated when bit i of signs is set
#pragma unroll
    for (int i = 0; i < 16; i++) {
      const u32 f = ((signs >> i) & 1u) ? 0x80008000u : 0u;
      raw[i].x ^= f; raw[i].y ^= f;
    }
    // two rounds of two columns (one packed word per token): the loop body exists once in the instruction stream.  The
    // two columns ride in the two halves of packed FP32 pairs through the butterflies and the scaling.
#pragma unroll 1
    for (int jw = 0; jw < 2; jw++) {
      u64 P[16];
#pragma unroll
      for (int i = 0; i < 16; i++) P[i] = f2_from_bf16x2(raw[i].x);
#pragma unroll
      for (int h = 1; h < 16; h <<= 1)
#pragma unroll
        for (int i = 0; i < 16; i++)
          if (!(i & h)) { const u64 a = P[i], b = P[i + h]; P[i] = f2_add(a, b); P[i + h] = f2_sub(a, b); }
      const int c = tc + jw * 2;
      const long long b0 = (long long)(c0 + c) * nmb + mb0 + tm, b1 = b0 + nmb;
      uint2 o0, o1; u32 sb0, sb1;
      quant_block16x2<ROUNDING>(P, ts, seed, (u32)b0, (u32)b1, block_key<ROUNDING>(seed, (u32)b0), block_key<ROUNDING>(seed, (u32)b1),
                                o0, o1, sb0, sb1);
      const int slot = tm ^ (lane & 15);
      stage_codes[c * kMb + slot] = o0;
      stage_codes[(c + 1) * kMb + slot] = o1;
      stage_scales[c * kMb + tm] = (unsigned char)sb0;
      stage_scales[(c + 1) * kMb + tm] = (unsigned char)sb1;
#pragma unroll
      for (int i = 0; i < 16; i++) raw[i].x = raw[i].y;
    }
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kCols * kMb / 256; k++) {
    const int at = k * 256 + (int)threadIdx.x, c = at >> 4, mb = (at & 15) ^ ((c >> 2) & 15);
    if (c0 + c < C && mb0 + mb < nmb) *reinterpret_cast<uint2*>(codes + ((long long)(c0 + c) * nmb + mb0 + mb) * 8) = stage_codes[at];
  }
  const bool linear = layout != NVFP4_SCALES_SWIZZLED, swizzled = layout != NVFP4_SCALES_LINEAR;
  unsigned char* scales_sw = layout == NVFP4_SCALES_BOTH ? scales + (long long)C * nmb : scales;
  if (!(nmb & 3) && !(reinterpret_cast<uintptr_t>(scales) & 3u)) {
    // four scale bytes of a column are neighbours in both layouts (swizzled: M is a multiple of 64)
    const int c = (int)threadIdx.x >> 2, mb = ((int)threadIdx.x & 3) * 4;
    if (c0 + c < C && mb0 + mb < nmb) {
      const u32 v = reinterpret_cast<const u32*>(stage_scales)[threadIdx.x];
      if (linear) *reinterpret_cast<u32*>(scales + (long long)(c0 + c) * nmb + mb0 + mb) = v;
      if (swizzled) *reinterpret_cast<u32*>(scales_sw + sw_off(c0 + c, mb0 + mb, nmb >> 2)) = v;
    }
  } else {
#pragma unroll
    for (int k = 0; k < kCols * kMb / 256; k++) {
      const int at = k * 256 + (int)threadIdx.x, c = at >> 4, mb = at & 15;
      if (c0 + c < C && mb0 + mb < nmb) {
        if (linear) scales[(long long)(c0 + c) * nmb + mb0 + mb] = stage_scales[at];
        if (swizzled) scales_sw[sw_off(c0 + c, mb0 + mb, nmb >> 2)] = stage_scales[at];
      }
    }
  }
}

// ------------------------------------------------------------------------------------------ 16x16 weights
// Any N and K that are multiples of 16 (weights in whole 128 x 128 tiles take the TMA-fed kernel of quant_w2d.cu).
// Persistent CTAs; one warp per group of four 16x16 blocks that are neighbours along N (same K
// block): lane = (row, 8-column half) of each block, four independent 16-byte loads in flight per
// lane.  Block max by warp shuffles, codes for W written as one word per lane and block, codes for
// W^T gathered with shuffles (lane = (k row, 8-row half)) and, after one exchange inside each lane
// pair, stored as 16 contiguous bytes per lane: a k row's 32 bytes for the four blocks leave together.
// L1-bound: the lanes of a load or store are on 16 rows.  A half-warp per patch of 4 x 2 blocks, a lane
// on whole 16-value rows, leaves too few warps and puts 32 rows into each load (us, that one / this one:
// FP32 [9616, 336] 32.3 / 10.3, [5008, 1552] 46.0 / 20.5, [20000, 5904] 326 / 222, bf16 [2064, 2064] 30.5 / 14.4).
template <typename T>
__global__ void __launch_bounds__(256) quant_w2d_kernel(const T* __restrict__ w, u32* __restrict__ q,
                                                         unsigned char* __restrict__ s, u32* __restrict__ qt,
                                                         unsigned char* __restrict__ st, const float* __restrict__ amax,
                                                         int N, int K, int layout, float* __restrict__ gs_out) {
  const int lane = threadIdx.x & 31;
  const int nb = N >> 4, kb = K >> 4;
  const int ngrp = (nb + 3) >> 2;
  const bool linear = layout != NVFP4_SCALES_SWIZZLED, swizzled = layout != NVFP4_SCALES_LINEAR;
  unsigned char* s_sw = layout == NVFP4_SCALES_BOTH ? s + (long long)N * kb : s;
  unsigned char* st_sw = layout == NVFP4_SCALES_BOTH ? st + (long long)K * nb : st;
  __shared__ __align__(8) float lut[kLutFloats];
  const TensorScale ts = make_tensor_scale<NVFP4_ROUND_NEAREST>(__ldg(amax), 1.f, lut,
                                                               (blockIdx.x == 0 && threadIdx.x == 0) ? gs_out : nullptr);
  const u64 G = f2_pack(ts.gs, ts.gs), NRG = f2_pack(ts.nrgs, ts.nrgs);
  const int r = lane >> 1, c0 = (lane & 1) * 8;
  const bool wide_t = !(N & 31) && !(reinterpret_cast<uintptr_t>(qt) & 15u);   // 16-byte stores of W^T codes possible
  const long long nitems = (long long)ngrp * kb;
  const long long wstride = (long long)gridDim.x * (blockDim.x >> 5);
  for (long long item = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); item < nitems; item += wstride) {
    // consecutive warps walk K: the loads of a CTA are contiguous along each row
    const int grp = (int)(item / kb), bk = (int)(item - (long long)grp * kb);
    float v[4][8];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int bn = grp * 4 + j;
      if (bn < nb) {
        const T* src = w + (long long)(bn * 16 + r) * K + bk * 16 + c0;
        if constexpr (sizeof(T) == 2) {
          unpack8(ldg128(src), v[j]);
        } else {
          const float4 a = __ldg(reinterpret_cast<const float4*>(src)), b = __ldg(reinterpret_cast<const float4*>(src) + 1);
          v[j][0] = a.x; v[j][1] = a.y; v[j][2] = a.z; v[j][3] = a.w; v[j][4] = b.x; v[j][5] = b.y; v[j][6] = b.z; v[j][7] = b.w;
        }
      } else {
#pragma unroll
        for (int i = 0; i < 8; i++) v[j][i] = 0.f;
      }
    }
    u32 wt[4], sbs[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int bn = grp * 4 + j;
      float bmax = absmax3(v[j][0], v[j][1], v[j][2]);
      bmax = absmax3(bmax, v[j][3], v[j][4]);
      bmax = absmax3(bmax, v[j][5], v[j][6]);
      bmax = absmax3(bmax, v[j][7], bmax);
#pragma unroll
      for (int o = 16; o; o >>= 1) bmax = fmaxf(bmax, __shfl_xor_sync(0xffffffffu, bmax, o));
      const u32 sb = block_scale_byte(bmax, ts);
      sbs[j] = sb;
      const float2 kf = lut_entry(ts, sb);
      const u64 NRH = f2_pack(kf.x, kf.x), NRL = f2_pack(kf.y, kf.y);
      float y[8];
#pragma unroll
      for (int i = 0; i < 8; i += 2) {
        const u64 t = f2_div_bs(f2_ndiv(f2_pack(v[j][i], v[j][i + 1]), G, NRG), NRH, NRL);
        y[i] = f2_lo(t); y[i + 1] = f2_hi(t);
      }
      const u32 word = e2m1x8_rn(y);
      if (q && bn < nb) {
        q[((long long)(bn * 16 + r) * K + bk * 16 + c0) >> 3] = word;
        if (!(lane & 1) && linear) s[(long long)(bn * 16 + r) * kb + bk] = (unsigned char)sb;
        if (!(lane & 1) && swizzled) s_sw[sw_off(bn * 16 + r, bk, kb >> 2)] = (unsigned char)sb;
      }
      // transposed block: this lane builds k-row kk = lane>>1, n values (lane&1)*8 .. +7
      const int kk = lane >> 1;
      u32 t = 0u;
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const u32 ww = __shfl_sync(0xffffffffu, word, 2 * (c0 + i) + (kk >> 3));
        t |= ((ww >> (4 * (kk & 7))) & 15u) << (4 * i);
      }
      wt[j] = t;
    }
    if (qt) {
      const int kk = lane >> 1;
      const long long krow = (long long)bk * 16 + kk;
      if (grp * 4 + 3 < nb && wide_t) {
        // even lane keeps blocks 0,1 (both 8-row halves), odd lane blocks 2,3: 16 contiguous bytes each
        const bool odd = lane & 1;
        const u32 give0 = odd ? wt[0] : wt[2], give1 = odd ? wt[1] : wt[3];
        const u32 got0 = __shfl_xor_sync(0xffffffffu, give0, 1), got1 = __shfl_xor_sync(0xffffffffu, give1, 1);
        const uint4 o = odd ? make_uint4(got0, wt[2], got1, wt[3]) : make_uint4(wt[0], got0, wt[1], got1);
        *reinterpret_cast<uint4*>(reinterpret_cast<unsigned char*>(qt) + krow * (N >> 1) + grp * 32 + (odd ? 16 : 0)) = o;
      } else {
#pragma unroll
        for (int j = 0; j < 4; j++)
          if (grp * 4 + j < nb) qt[(krow * N + (grp * 4 + j) * 16 + c0) >> 3] = wt[j];
      }
      if (!(lane & 1)) {
        if (grp * 4 + 3 < nb && !(nb & 3)) {
          // the four blocks' scale bytes are neighbours in both layouts (swizzled: nb is a multiple of 8)
          const u32 four = sbs[0] | (sbs[1] << 8) | (sbs[2] << 16) | (sbs[3] << 24);
          if (linear) *reinterpret_cast<u32*>(st + krow * nb + grp * 4) = four;
          if (swizzled) *reinterpret_cast<u32*>(st_sw + sw_off(krow, grp * 4, nb >> 2)) = four;
        } else {
#pragma unroll
          for (int j = 0; j < 4; j++)
            if (grp * 4 + j < nb) st[krow * nb + grp * 4 + j] = (unsigned char)sbs[j];
        }
      }
    }
  }
}

// ------------------------------------------------------------------------------------------ scale re-swizzle
__global__ void __launch_bounds__(256) swizzle_scales_kernel(const unsigned char* __restrict__ src, long long lds,
                                                              int R, int C16, unsigned char* __restrict__ dst) {
  const int ncb = C16 >> 2;
  const long long total = (long long)R * ncb;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    // consecutive threads walk the destination so stores coalesce
    const long long tile = i >> 7;           // (row block, column tile)
    const int in = (int)(i & 127);           // (r%32)*4 + (r%128)/32
    const long long rb = tile / ncb; const int cb = (int)(tile - rb * ncb);
    const long long r = rb * 128 + (in & 3) * 32 + (in >> 2);
    const unsigned char* p = src + r * lds + cb * 4;
    const u32 v = (u32)p[0] | ((u32)p[1] << 8) | ((u32)p[2] << 16) | ((u32)p[3] << 24);
    *reinterpret_cast<u32*>(dst + i * 4) = v;
  }
}

// ------------------------------------------------------------------------------------------ raw SR convert
__global__ void __launch_bounds__(256) e2m1x4_sr_kernel(const float4* __restrict__ y, const u32* __restrict__ rbits,
                                                         unsigned short* __restrict__ out, long long n4) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n4) return;
  const float4 v = y[i];
  out[i] = (unsigned short)e2m1x4_rs(v.x, v.y, v.z, v.w, rbits[i]);
}

static int sm_count() {
  static int cached[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 148;
  if (dev < 0 || dev >= 64) return 148;
  if (!cached[dev]) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    cached[dev] = n;
  }
  return cached[dev];
}

}  // namespace nvfp4

using namespace nvfp4;

// -1: not decided yet (environment variable NVFP4_PDL, else 2), else as nvfp4_set_pdl.  2: short launches only, us per
// pass off -> on: forward [256, 5632, 2048] 20.5 -> 15.6, weight refresh of a block 77 -> 67, layer [4096, 2048, 3072]
// 131 -> 125.  With every launch in it the long ones lose (weight gradient of 16384 tokens 204 -> 218): a staged grid
// crowds onto the SMs that come free first.
static int g_pdl = -1;
bool nvfp4_pdl_enabled(bool brief) {
  if (g_pdl < 0) {
    const char* e = getenv("NVFP4_PDL");
    g_pdl = !e || !e[0] ? 2 : e[0] == '1' ? 1 : e[0] == '2' ? 2 : 0;
  }
  return g_pdl == 1 || (g_pdl == 2 && brief);
}
extern "C" int nvfp4_set_pdl(int on) {
  g_pdl = on == 2 ? 2 : on ? 1 : 0;
  return NVFP4_OK;
}

static inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// (device, unique id) of a stream outside a capture; false where there is none to be had.  Launches of one stream never
// overlap (a programmatically dependent one waits before it touches memory), so memory that belongs to a stream is
// free for its next launch.  Not inside a capture: a graph may be replayed on another stream beside later work of
// this one.  Ids are never given out twice.
static bool stream_id(cudaStream_t st, int& dev, unsigned long long& id) {
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (st == cudaStreamPerThread) return false;              // one handle, a stream per thread
  if (cudaStreamIsCapturing(st, &cap) != cudaSuccess) {
    (void)cudaGetLastError();
    return false;
  }
  if (cap != cudaStreamCaptureStatusNone) return false;     // asking a capturing stream for its id would end the capture
  if (cudaStreamGetId(st, &id) != cudaSuccess || cudaGetDevice(&dev) != cudaSuccess) {
    (void)cudaGetLastError();
    return false;
  }
  return dev >= 0 && dev < 64;
}

template <typename T>
static T* symbol_base(const T (&sym)[kAmaxSlots], int dev) {
  static T* base[64];
  if (!base[dev]) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, sym) != cudaSuccess) { (void)cudaGetLastError(); return nullptr; }
    base[dev] = static_cast<T*>(p);
  }
  return base[dev];
}

// The slot of a stream; null (the caller then clears with a memset) inside captures and for streams beyond the table.
static AmaxSlot* amax_slot(cudaStream_t st) {
  int dev;
  unsigned long long id;
  if (!stream_id(st, dev, id)) return nullptr;
  static std::mutex lock;
  static std::unordered_map<unsigned long long, int>* index = new std::unordered_map<unsigned long long, int>[64];
  std::lock_guard<std::mutex> hold(lock);
  AmaxSlot* base = symbol_base(g_amax_slots, dev);
  if (!base) return nullptr;
  const auto it = index[dev].find(id);
  if (it != index[dev].end()) return base + it->second;
  const int n = (int)index[dev].size();
  if (n >= kAmaxSlots) return nullptr;
  index[dev].emplace(id, n);
  return base + n;
}

// Result words for an amax whose consumers this thread launches next on the same stream: a ring of eight per (thread,
// stream).  The launch that fills one word clears the next, so none needs a memset or a meeting point of blocks, and a
// word is not touched again before the thread's seventh later call on that stream.  A ring per thread, because two
// threads that share a stream could slip any number of calls between one's amax and its consumer.  The rings are fixed
// memory of the library; a thread's are handed on, per stream, when it ends; calls beyond the table get null.
struct WordRing { unsigned long long id; int dev, slot; unsigned at; };
struct WordRings {
  static std::mutex& lock() { static std::mutex* m = new std::mutex; return *m; }
  static std::vector<WordRing>& spare() { static auto* v = new std::vector<WordRing>; return *v; }
  static int* taken() { static int n[64]; return n; }
  std::vector<WordRing> mine;
  ~WordRings() {
    std::lock_guard<std::mutex> hold(lock());
    spare().insert(spare().end(), mine.begin(), mine.end());
  }
  WordRing* find(int dev, unsigned long long id) {
    for (WordRing& r : mine)
      if (r.id == id && r.dev == dev) return &r;
    std::lock_guard<std::mutex> hold(lock());
    for (size_t k = 0; k < spare().size(); k++)
      if (spare()[k].id == id && spare()[k].dev == dev) {
        mine.push_back(spare()[k]);
        spare().erase(spare().begin() + k);
        return &mine.back();
      }
    if (taken()[dev] >= kAmaxSlots) return nullptr;
    mine.push_back(WordRing{id, dev, taken()[dev]++, 0u});
    return &mine.back();
  }
};

template <bool F32>
static cudaError_t amax_start(const void* x, long long nv, float* out, float* next, AmaxSlot* slot, cudaStream_t st) {
  // four loads per thread and four CTAs per SM (or as many as there is work for)
  long long blocks = (nv + 256 * 4 - 1) / (256 * 4);
  const long long cap = (long long)sm_count() * 4;
  if (blocks > cap) blocks = cap;
  const cudaError_t rc = nvfp4_launch_kernel(amax_kernel<F32>, nvfp4_brief(nv * 16), dim3((unsigned)blocks), dim3(256), 0, st, static_cast<const uint4*>(x), nv, out, next, slot);
  if (rc != cudaSuccess) (void)cudaGetLastError();
  return rc;
}

// `n` values, 16 / sizeof of them per load
template <bool F32>
static int amax_launch(const void* x, long long n, float* out, bool clear, void* stream) {
  constexpr int kPer = F32 ? 4 : 8;
  if (!out || (!x && n > 0)) return NVFP4_ERR_NULL;
  if (n < 0 || n % kPer) return NVFP4_ERR_SHAPE;
  if (!aligned16(x)) return NVFP4_ERR_ALIGN;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  AmaxSlot* slot = clear && n > 0 ? amax_slot(st) : nullptr;
  if (clear && !slot && cudaMemsetAsync(out, 0, sizeof(float), st) != cudaSuccess) return NVFP4_ERR_CUDA;
  if (n == 0) return NVFP4_OK;
  return amax_start<F32>(x, n / kPer, out, nullptr, slot, st) == cudaSuccess ? NVFP4_OK : NVFP4_ERR_CUDA;
}

extern "C" int nvfp4_amax_bf16_word(const void* x, long long n, float* fallback, const float** word, void* stream) {
  if (!word || !x) return NVFP4_ERR_NULL;
  if (n <= 0 || (n & 7)) return NVFP4_ERR_SHAPE;
  if (!aligned16(x)) return NVFP4_ERR_ALIGN;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  static thread_local WordRings rings;
  int dev;
  unsigned long long id;
  WordRing* ring = stream_id(st, dev, id) ? rings.find(dev, id) : nullptr;
  AmaxWords* base = ring ? symbol_base(g_amax_words, dev) : nullptr;
  if (!base) {
    *word = fallback;
    return fallback ? nvfp4_amax_bf16(x, n, fallback, stream) : NVFP4_OK;
  }
  AmaxWords& w = base[ring->slot];
  float* out = &w.v[ring->at & 7u];
  if (amax_start<false>(x, n >> 3, out, &w.v[(ring->at + 1u) & 7u], nullptr, st) != cudaSuccess) return NVFP4_ERR_CUDA;
  ring->at++;
  *word = out;
  return NVFP4_OK;
}

extern "C" int nvfp4_amax_bf16(const void* x, long long n, float* out, void* stream) {
  return amax_launch<false>(x, n, out, true, stream);
}

extern "C" int nvfp4_amax_bf16_update(const void* x, long long n, float* out, void* stream) {
  return amax_launch<false>(x, n, out, false, stream);
}

extern "C" int nvfp4_amax_f32(const float* x, long long n, float* out, void* stream) {
  return amax_launch<true>(x, n, out, true, stream);
}

extern "C" int nvfp4_quant_rows(const void* x, long long ldx, int R, int C, void* codes, void* scales,
                                int scale_layout, const float* amax, float* gs_out, int rounding, unsigned seed,
                                const unsigned* seed_dev, void* stream) {
  if (!x || !codes || !scales || !amax) return NVFP4_ERR_NULL;
  if (scale_layout < NVFP4_SCALES_SWIZZLED || scale_layout > NVFP4_SCALES_BOTH) return NVFP4_ERR_ENUM;
  if (rounding < NVFP4_ROUND_NEAREST || rounding > NVFP4_ROUND_SR_HW) return NVFP4_ERR_ENUM;
  if (R < 0 || C < 0 || (C & 15) || ldx < C) return NVFP4_ERR_SHAPE;
  if (scale_layout != NVFP4_SCALES_LINEAR && ((R & 127) || (C & 63))) return NVFP4_ERR_SHAPE;
  if (!aligned16(x) || (ldx & 7) || (reinterpret_cast<uintptr_t>(codes) & 7u)) return NVFP4_ERR_ALIGN;
  if (R == 0 || C == 0) return NVFP4_OK;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // Contiguous rows with row-major scales are one long row: no lane idles at a row's end ([5008, 1552]: 97 blocks a row
  // in segments of 32 leave a quarter of the lanes without work: 9.2 -> 6.8 us)
  if (ldx == C && scale_layout == NVFP4_SCALES_LINEAR && (long long)R * C <= 0x7FFFF000ll) {
    C *= R;
    ldx = C;
    R = 1;
  }
  const long long nitems = (long long)R * (((C >> 3) + 63) >> 6);
  long long blocks = (nitems + 7) / 8;
  const long long cap = (long long)sm_count() * 16;
  if (blocks > cap) blocks = cap;
  const __nv_bfloat16* xp = static_cast<const __nv_bfloat16*>(x);
  uint2* cp = static_cast<uint2*>(codes);
  unsigned char* sp = static_cast<unsigned char*>(scales);
  // 256-bit loads need 32-byte aligned rows
  const bool wide = (reinterpret_cast<uintptr_t>(x) & 31u) == 0 && (ldx & 15) == 0;
#define NVFP4_ROWS(RND)                                                                                              \
  do {                                                                                                               \
    if (wide) quant_rows_kernel<RND, true><<<(unsigned)blocks, 256, 0, st>>>(xp, ldx, cp, sp, amax, R, C, scale_layout, seed, seed_dev, gs_out); \
    else quant_rows_kernel<RND, false><<<(unsigned)blocks, 256, 0, st>>>(xp, ldx, cp, sp, amax, R, C, scale_layout, seed, seed_dev, gs_out);     \
  } while (0)
  switch (rounding) {
    case NVFP4_ROUND_NEAREST: NVFP4_ROWS(NVFP4_ROUND_NEAREST); break;
    case NVFP4_ROUND_SR_DITHER: NVFP4_ROWS(NVFP4_ROUND_SR_DITHER); break;
    case NVFP4_ROUND_SR_DITHER_K: NVFP4_ROWS(NVFP4_ROUND_SR_DITHER_K); break;
    default: NVFP4_ROWS(NVFP4_ROUND_SR_HW); break;
  }
#undef NVFP4_ROWS
  NVFP4_LAUNCH_CHECK();
  return NVFP4_OK;
}

extern "C" int nvfp4_quant_cols_rht(const void* x, int M, int C, void* codes, void* scales, int scale_layout,
                                    const float* amax, float* gs_out, unsigned signs, int rounding, unsigned seed,
                                    const unsigned* seed_dev, void* stream) {
  if (!x || !codes || !scales || !amax) return NVFP4_ERR_NULL;
  if (scale_layout < NVFP4_SCALES_SWIZZLED || scale_layout > NVFP4_SCALES_BOTH) return NVFP4_ERR_ENUM;
  if (rounding < NVFP4_ROUND_NEAREST || rounding > NVFP4_ROUND_SR_HW) return NVFP4_ERR_ENUM;
  if (M < 0 || C < 0 || (M & 15) || (C & 7)) return NVFP4_ERR_SHAPE;
  if (scale_layout != NVFP4_SCALES_LINEAR && ((C & 127) || (M & 63))) return NVFP4_ERR_SHAPE;
  if (!aligned16(x) || (reinterpret_cast<uintptr_t>(codes) & 7u)) return NVFP4_ERR_ALIGN;
  if (M == 0 || C == 0) return NVFP4_OK;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  dim3 grid((unsigned)((C + 63) / 64), (unsigned)((M + 255) / 256));
  if (grid.y > 65535u) return NVFP4_ERR_TOO_LARGE;
  const __nv_bfloat16* xp = static_cast<const __nv_bfloat16*>(x);
  unsigned char* cp = static_cast<unsigned char*>(codes);
  unsigned char* sp = static_cast<unsigned char*>(scales);
  signs &= 0xFFFFu;
  switch (rounding) {
    case NVFP4_ROUND_NEAREST:
      quant_cols_rht_kernel<NVFP4_ROUND_NEAREST><<<grid, 256, 0, st>>>(xp, cp, sp, amax, M, C, scale_layout, signs, seed, seed_dev, gs_out); break;
    case NVFP4_ROUND_SR_DITHER:
      quant_cols_rht_kernel<NVFP4_ROUND_SR_DITHER><<<grid, 256, 0, st>>>(xp, cp, sp, amax, M, C, scale_layout, signs, seed, seed_dev, gs_out); break;
    case NVFP4_ROUND_SR_DITHER_K:
      quant_cols_rht_kernel<NVFP4_ROUND_SR_DITHER_K><<<grid, 256, 0, st>>>(xp, cp, sp, amax, M, C, scale_layout, signs, seed, seed_dev, gs_out); break;
    default:
      quant_cols_rht_kernel<NVFP4_ROUND_SR_HW><<<grid, 256, 0, st>>>(xp, cp, sp, amax, M, C, scale_layout, signs, seed, seed_dev, gs_out); break;
  }
  NVFP4_LAUNCH_CHECK();
  return NVFP4_OK;
}

// the TMA-fed kernel (quant_w2d.cu)
bool nvfp4_quant_w2d_tile_accepts(const void* w, int N, int K, const void* q, const void* s, const void* qt, const void* st);
int nvfp4_quant_w2d_tile_launch(const void* w, int w_dtype, int N, int K, void* q, void* s, void* qt, void* st, int scale_layout,
                                const float* amax, float* gs_out, void* stream);

extern "C" int nvfp4_quant_w2d(const void* w, int w_dtype, int N, int K, void* q, void* s, void* qt, void* st_,
                               int scale_layout, const float* amax, float* gs_out, void* stream) {
  if (!w || !amax || (!q && !qt) || (q && !s) || (qt && !st_)) return NVFP4_ERR_NULL;
  if (scale_layout < NVFP4_SCALES_SWIZZLED || scale_layout > NVFP4_SCALES_BOTH) return NVFP4_ERR_ENUM;
  if (w_dtype != NVFP4_DTYPE_BF16 && w_dtype != NVFP4_DTYPE_FP32) return NVFP4_ERR_ENUM;
  if (N < 0 || K < 0 || (N & 15) || (K & 15)) return NVFP4_ERR_SHAPE;
  if (scale_layout != NVFP4_SCALES_LINEAR && ((N & 127) || (K & 127))) return NVFP4_ERR_SHAPE;
  if (!aligned16(w) || (q && (reinterpret_cast<uintptr_t>(q) & 3u)) || (qt && ((reinterpret_cast<uintptr_t>(qt) | reinterpret_cast<uintptr_t>(st_)) & 3u)))
    return NVFP4_ERR_ALIGN;
  if (N == 0 || K == 0) return NVFP4_OK;
  cudaStream_t stm = static_cast<cudaStream_t>(stream);
  if (nvfp4_quant_w2d_tile_accepts(w, N, K, q, s, qt, st_))
    return nvfp4_quant_w2d_tile_launch(w, w_dtype, N, K, q, s, qt, st_, scale_layout, amax, gs_out, stream);
  const long long nwarps = (long long)(((N >> 4) + 3) >> 2) * (K >> 4);
  long long blocks = (nwarps + 7) / 8;
  const long long cap = (long long)sm_count() * 8;
  if (blocks > cap) blocks = cap;
#define NVFP4_W2D(T)                                                                                                     \
  quant_w2d_kernel<T><<<(unsigned)blocks, 256, 0, stm>>>(static_cast<const T*>(w), static_cast<u32*>(q), static_cast<unsigned char*>(s), \
      static_cast<u32*>(qt), static_cast<unsigned char*>(st_), amax, N, K, scale_layout, gs_out)
  if (w_dtype == NVFP4_DTYPE_BF16) NVFP4_W2D(__nv_bfloat16);
  else NVFP4_W2D(float);
#undef NVFP4_W2D
  NVFP4_LAUNCH_CHECK();
  return NVFP4_OK;
}

extern "C" int nvfp4_swizzle_scales(const void* s_linear, long long lds, int R, int C16, void* s_swizzled, void* stream) {
  if (!s_linear || !s_swizzled) return NVFP4_ERR_NULL;
  if (R < 0 || C16 < 0 || (R & 127) || (C16 & 3) || lds < C16) return NVFP4_ERR_SHAPE;
  if (reinterpret_cast<uintptr_t>(s_swizzled) & 3u) return NVFP4_ERR_ALIGN;
  if (R == 0 || C16 == 0) return NVFP4_OK;
  const long long total = (long long)R * (C16 >> 2);
  long long blocks = (total + 255) / 256;
  const long long cap = (long long)sm_count() * 8;
  if (blocks > cap) blocks = cap;
  swizzle_scales_kernel<<<(unsigned)blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const unsigned char*>(s_linear), lds, R, C16, static_cast<unsigned char*>(s_swizzled));
  NVFP4_LAUNCH_CHECK();
  return NVFP4_OK;
}

extern "C" int nvfp4_e2m1x4_sr(const float* y, const unsigned* rbits, void* codes, long long n4, void* stream) {
  if (!y || !rbits || !codes) return NVFP4_ERR_NULL;
  if (n4 < 0) return NVFP4_ERR_SHAPE;
  if (!aligned16(y) || (reinterpret_cast<uintptr_t>(rbits) & 3u) || (reinterpret_cast<uintptr_t>(codes) & 1u)) return NVFP4_ERR_ALIGN;
  if (n4 == 0) return NVFP4_OK;
  const long long blocks = (n4 + 255) / 256;
  if (blocks > 0x7FFFFFFFLL) return NVFP4_ERR_TOO_LARGE;
  e2m1x4_sr_kernel<<<(unsigned)blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<const float4*>(y), rbits, static_cast<unsigned short*>(codes), n4);
  NVFP4_LAUNCH_CHECK();
  return NVFP4_OK;
}
