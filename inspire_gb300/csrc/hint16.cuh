// ComputeHintMatrix (crypto/hint_computation.cc:78-160) for d = 2048..8192 with
// the radix-16 register transforms: out[row] = sum_k DB[row][k] v_k mod 2^w for
// the inverted a-components v_k (v[0] = a[0], v[j] = -a[d - j]).
//
// The a-components are split into two halves of w / 2 bits, so that the sums
// are small: two 27-bit primes hold a u16 database over Z_2^32 up to n d =
// 2^20 where whole words took three, and a third prime is cheaper than a
// fourth over Z_2^64. A database block is transformed once per prime and
// multiplied with both halves; each half has one inverse transform per prime
// and row. The multiplier bounds the kernel (a butterfly takes four of the 64
// slots a cycle, a 64-bit multiply-add three): n = 8 blocks of 4096 over Z_2^32
// come to 37 thousand cycles per row, 3.9 ms for 32768 rows; the kernel takes
// 7.1 ms (issue 57 % of cycles, 68-92 bytes of spills at 128 registers; 228-268 at
// d = 2048, 128-144 at d = 8192), three primes with whole words and a separate
// reconstruction took 13.
#pragma once
#include <cstdint>

#include "answer_poly.cuh"

namespace inspire {

constexpr int kHintParts = 2;

#ifdef __CUDACC__
// Transforms of the a-component halves, in the order the row kernel reads
// them: slot 16 tid + 4 v + i of (component k, half h, prime pi) at
// ((k r + pi) 2 + h) d + (v d / 16 + tid) 4 + i. grid = (2 n, r).
template <typename T, int LOGD>
__global__ void __launch_bounds__(Ntt16<LOGD>::kThreads)
hint_parts16_kernel(const T* __restrict__ a, uint32_t* __restrict__ out, NttCtx c) {
  constexpr int d = Ntt16<LOGD>::kD;
  constexpr int NT = Ntt16<LOGD>::kThreads;
  constexpr int kHalf = 4 * sizeof(T);
  __shared__ uint32_t xs[d];
  const int tid = threadIdx.x;
  const int k = blockIdx.x / kHintParts, h = blockIdx.x % kHintParts, pi = blockIdx.y;
  const T* ak = a + static_cast<int64_t>(k) * d;
  uint32_t x[16];
#pragma unroll
  for (int m = 0; m < 16; ++m) {
    const int j = tid + NT * m;
    const T v = j == 0 ? ak[0] : static_cast<T>(T{0} - ak[d - j]);
    const T part = h == 0 ? static_cast<T>(v & ((T{1} << kHalf) - 1)) : static_cast<T>(v >> kHalf);
    x[m] = reduce_word(static_cast<uint32_t>(part), c, pi);
  }
  ntt16_forward<LOGD, false, true, true>(x, xs, c.tables16 + static_cast<size_t>(pi) * 2 * d,
                                         c.p[pi], c.one_s[pi], tid);
  uint4* o = reinterpret_cast<uint4*>(
      out + (static_cast<int64_t>(k * c.r + pi) * kHintParts + h) * d) + tid;
#pragma unroll
  for (int v = 0; v < 4; ++v) {
    o[v * NT] = make_uint4(x[4 * v], x[4 * v + 1], x[4 * v + 2], x[4 * v + 3]);
  }
}

// Bytes of dynamic shared memory: the exchange buffer, and per coefficient
// the word and the two halves' fractions summed over the primes so far.
template <typename T, int LOGD>
constexpr size_t HintRowsSmem() {
  return static_cast<size_t>(Ntt16<LOGD>::kD) * (4 + sizeof(T) + 4 * kHintParts);
}

// One row per block, all primes in turn. V: hint_parts16_kernel's output.
// Two blocks of d = 4096 per SM: the 64-bit sums of both halves take 64
// registers. grid = rows, d / 16 threads.
template <typename T, typename S, int LOGD>
__global__ void __launch_bounds__(Ntt16<LOGD>::kThreads, 512 / Ntt16<LOGD>::kThreads)
hint_rows16_kernel(const S* __restrict__ db, int64_t cols, int n,
                   const uint32_t* __restrict__ V, T* __restrict__ out,
                   const __grid_constant__ NttCtx c, const __grid_constant__ CrtArgs crt) {
  extern __shared__ __align__(16) unsigned char hint_smem[];
  constexpr int d = Ntt16<LOGD>::kD;
  constexpr int NT = Ntt16<LOGD>::kThreads;
  constexpr int kHalf = 4 * sizeof(T);
  constexpr int kFold = 24;  // products below 2^59 in a 64-bit sum
  T* word = reinterpret_cast<T*>(hint_smem);
  uint32_t* xs = reinterpret_cast<uint32_t*>(word + d);
  uint32_t* frac = xs + d;  // [half][d]
  const int tid = threadIdx.x;
  const S* src = db + static_cast<int64_t>(blockIdx.x) * cols + tid;
  for (int pi = 0; pi < c.r; ++pi) {
    const uint32_t p = c.p[pi], pinv = c.pinv[pi], one_s = c.one_s[pi];
    const uint2* tw = c.tables16 + static_cast<size_t>(pi) * 2 * d;
    uint64_t sum[kHintParts][16];
#pragma unroll
    for (int h = 0; h < kHintParts; ++h) {
#pragma unroll
      for (int m = 0; m < 16; ++m) sum[h][m] = 0;
    }
    uint32_t x[16];
#pragma unroll 1
    for (int k = 0; k < n; ++k) {
      const S* rk = src + static_cast<int64_t>(k) * d;
      const uint4* vk = reinterpret_cast<const uint4*>(
          V + static_cast<int64_t>(k * c.r + pi) * kHintParts * d) + tid;
      // 128 bytes per thread: this block's factors and the next block's
      // entries, on their way while this block is transformed.
      asm volatile("prefetch.global.L1 [%0];" ::"l"(vk + 7 * tid));
      if (tid * 128 < d * static_cast<int>(sizeof(S)) && k + 1 < n) {
        asm volatile("prefetch.global.L1 [%0];" ::"l"(
            reinterpret_cast<const char*>(rk - tid + d) + 128 * tid));
      }
#pragma unroll
      for (int m = 0; m < 16; ++m) {
        // Entries of up to 16 bits are residues as they are.
        const uint32_t v = static_cast<uint32_t>(__ldg(rk + NT * m));
        x[m] = sizeof(S) <= 2 ? v : reduce_word(v, c, pi);
      }
      ntt16_forward<LOGD>(x, xs, tw, p, one_s, tid);
#pragma unroll
      for (int h = 0; h < kHintParts; ++h) {
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          const uint4 w = __ldg(vk + h * (d / 4) + v * NT);
          const uint32_t wv[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            sum[h][4 * v + i] += static_cast<uint64_t>(x[4 * v + i]) * wv[i];
          }
        }
      }
      if (k % kFold == kFold - 1) {
#pragma unroll
        for (int h = 0; h < kHintParts; ++h) {
#pragma unroll
          for (int m = 0; m < 16; ++m) sum[h][m] = reduce_word(sum[h][m], c, pi);
        }
      }
    }
#pragma unroll 1
    for (int h = 0; h < kHintParts; ++h) {
#pragma unroll
      for (int m = 0; m < 16; ++m) {
        x[m] = reduce_sum(h == 0 ? sum[0][m] : sum[1][m], p, pinv, one_s);
      }
      ntt16_inverse<LOGD>(x, xs, tw + d, p, one_s, tid);
#pragma unroll
      for (int m = 0; m < 16; ++m) {
        // The thread's own places: no barrier.
        const int j = tid + NT * m;
        const uint32_t y = shoup_mul(x[m], crt.scale[pi], crt.scale_s[pi], p);
        const T part = static_cast<T>(static_cast<T>(y) * static_cast<T>(crt.part[pi]))
                       << (h * kHalf);
        word[j] = pi == 0 && h == 0 ? part : static_cast<T>(word[j] + part);
        frac[h * d + j] =
            (pi == 0 ? 1u << 25 : frac[h * d + j]) + __umulhi(y, crt.frac[pi]);
      }
    }
  }
  T* o = out + static_cast<int64_t>(blockIdx.x) * d;
#pragma unroll
  for (int m = 0; m < 16; ++m) {
    const int j = tid + NT * m;
    T v = word[j];
#pragma unroll
    for (int h = 0; h < kHintParts; ++h) {
      v -= static_cast<T>(static_cast<T>(frac[h * d + j] >> 26) * static_cast<T>(crt.m))
           << (h * kHalf);
    }
    o[j] = v;
  }
}
#endif

}  // namespace inspire
