// The reduction chains of PreprocessPack (crypto/lwes_to_rlwe.cc:310-344) for
// d = 2048 and 4096, and d = 8192 over Z_2^32, a cluster of one CTA per prime
// for each (chain, slice).
//
// A chain is d/2 - 1 dependent links: signed digits of the running word
// vector, their products with the key parts read through an automorphism, an
// add. Latency is all that counts (two chains a slice keep few SMs busy), so
// a link touches global memory only for the word vector it adds, loaded
// ahead, and for the digits it leaves behind: twiddles, the prime's key-part
// transforms and the digit planes stay in shared memory, the residues go
// through distributed shared memory, and the code is one transform body each
// way. The one-block form (all primes side by side, twiddles and permuted key
// words from L2, 75 KB of code) took 20 us a link at d = 2048 over Z_2^64, this
// one 5.5 (chains of 8 slices 23.7 -> 5.65 ms). At d = 8192 twiddles and key-part
// transforms do not fit beside the rest and stay in L2.
#pragma once
#include <cstdint>

#include "answer_poly.cuh"
#include "preprocess_kernels.cuh"

namespace inspire {

// Digits transformed side by side at most; blocks of G groups of d / 16 threads
// (the other groups help with the products and the reconstruction).
constexpr int kChainSide = 2;

// Bytes of shared memory with `side` digits side by side: twiddle pairs,
// key-part transforms, exchange buffers, residues, digit planes. Two where
// they fit (up to three digits at d = 4096, ten at d = 2048), else one: a
// block per chain takes longer by more (four digits at d = 4096 over Z_2^32:
// 83 ms a slice).
template <int LOGD>
constexpr size_t Chain16Smem(int k, int side) {
  return static_cast<size_t>(Ntt16<LOGD>::kD) * 4 *
         ((LOGD <= 12 ? 4 + k : 0) + side + 1 + k);
}

#ifdef __CUDACC__
// grid = (2 R, slices), clusters of R, G d / 16 threads, SIDE digits side by
// side (compiled in: as an argument it cost the links of d = 2048 2 %). Needs
// log_digit <= 27 and at most 30 digits. Outputs as pp_chain_kernel's.
template <typename T, int LOGD, int G, int R, int SIDE>
__global__ void __launch_bounds__(G * Ntt16<LOGD>::kThreads, 1)
chain16_cluster_kernel(const T* __restrict__ ev, const __grid_constant__ ChainArgs a,
                       const __grid_constant__ NttCtx c, const __grid_constant__ CrtArgs crt,
                       T* __restrict__ tg, T* __restrict__ tgh, T* __restrict__ fin) {
  extern __shared__ __align__(16) uint32_t smem[];
  constexpr int d = Ntt16<LOGD>::kD;
  constexpr int NT = Ntt16<LOGD>::kThreads;
  constexpr int kThreads = G * NT;
  constexpr int kQuads = (d / 4 + kThreads - 1) / kThreads;
  constexpr int kWords = (d + kThreads - 1) / kThreads;
  constexpr bool kLocal = LOGD <= 12;  // twiddles and key parts in shared memory
  static_assert(SIDE <= kChainSide && G >= SIDE, "a group per digit");
  using S = typename std::make_signed<T>::type;
  const int tid = threadIdx.x;
  const int grp = tid / NT;
  const int lt = tid & (NT - 1);
  const int bar = 1 + grp;
  const int pi = blockIdx.x % R;
  const int chain = blockIdx.x / R;
  const int s = blockIdx.y;
  const int k = a.k;
  const uint32_t p = c.p[pi], pinv = c.pinv[pi], one_s = c.one_s[pi];
  const uint2* tables = c.tables16 + static_cast<size_t>(pi) * 2 * d;
  const uint2* tw = kLocal ? reinterpret_cast<const uint2*>(smem) : tables;
  const uint2* itw = tw + d;
  uint32_t* W = smem + 4 * d;                                       // [k][d] if kLocal
  uint32_t* regions = kLocal ? W + static_cast<int64_t>(k) * d : smem;  // [SIDE][d]
  uint32_t* region = regions + grp * d;
  uint32_t* res = regions + SIDE * d;
  int32_t* dig = reinterpret_cast<int32_t*>(res + d);      // [k][d]
  if constexpr (kLocal) {
    const uint4* src = reinterpret_cast<const uint4*>(tables);
    uint4* dst = reinterpret_cast<uint4*>(smem);
    for (int i = tid; i < d; i += kThreads) dst[i] = __ldg(src + i);
    uint4* wd = reinterpret_cast<uint4*>(W);
    for (int i = tid; i < k * (d / 4); i += kThreads) {
      const int l = i / (d / 4);
      wd[i] = __ldg(reinterpret_cast<const uint4*>(
                        a.Wg + (static_cast<int64_t>(l) * R + pi) * d) + i % (d / 4));
    }
  }
  const T* evs = ev + static_cast<int64_t>(s) * d * d;
  T* out = (chain == 0 ? tg : tgh) + s * a.chain_stride;
  // The digits of word j of the running vector: to shared memory, and out
  // for the matrix (each CTA writes its share).
  auto put_digits = [&](int j, T x, T* to, bool mine) {
    constexpr int kW = 8 * sizeof(T);
    const int lq = a.log_q == 0 ? kW : a.log_q;
    T cur = pp_low<T>(x, a.log_q);
    const int to_shift = lq - k * a.log_digit;
    if (to_shift > 0) {
      const T half = T{1} << (to_shift - 1);
      const T sum = static_cast<T>(cur + half);
      const T carry = sum < cur ? T{1} : T{0};
      cur = static_cast<T>((sum >> to_shift) | (carry << (kW - to_shift)));
    }
    const uint32_t mask = (1u << a.log_digit) - 1, half = 1u << (a.log_digit - 1);
#pragma unroll 1
    for (int l = 0; l < k; ++l) {
      const uint32_t lower = static_cast<uint32_t>(cur) & mask;
      const bool up = lower >= half;
      const int32_t v = static_cast<int32_t>(lower) - (up ? static_cast<int32_t>(mask) + 1 : 0);
      cur = static_cast<T>((cur >> a.log_digit) + (up ? 1 : 0));
      dig[l * d + j] = v;
      if (mine) to[static_cast<int64_t>(l) * d + j] = static_cast<T>(static_cast<S>(v));
    }
  };
  {
    const T* start =
        evs + static_cast<int64_t>(__ldg(a.hat_row + (chain == 0 ? d / 2 - 1 : d - 1))) * d;
    T* to = out + static_cast<int64_t>(d / 2 - 2) * k * d;
    for (int n = 0; n < kWords; ++n) {
      const int j = tid + n * kThreads;
      if (j < d) put_digits(j, start[j], to, n % R == pi);
    }
  }
  __syncthreads();
  const uint32_t la = static_cast<uint32_t>(__cvta_generic_to_shared(res));
  uint32_t peer[R];
#pragma unroll
  for (int q = 0; q < R; ++q) peer[q] = cluster_map(la, q);

#pragma unroll 1
  for (int i = d / 2 - 2; i >= 0; --i) {
    const int p5 = __ldg(a.pow5 + i);
    const int power = chain == 0 ? p5 : (p5 * (2 * d - 1)) & (2 * d - 1);
    const T* add = evs + static_cast<int64_t>(__ldg(a.hat_row + (chain == 0 ? i : d / 2 + i))) * d;
    uint64_t sum[kQuads][4];
#pragma unroll
    for (int u = 0; u < kQuads; ++u) {
#pragma unroll
      for (int m = 0; m < 4; ++m) sum[u][m] = 0;
    }
    uint32_t x[16];
#pragma unroll 1
    for (int l0 = 0; l0 < k; l0 += SIDE) {
      if (grp < SIDE && l0 + grp < k) {
        const int32_t* src = dig + (l0 + grp) * d + lt;
#pragma unroll
        for (int m = 0; m < 16; ++m) {
          const int32_t v = src[NT * m];
          x[m] = static_cast<uint32_t>(v) + (v < 0 ? p : 0u);
        }
        ntt16_forward<LOGD, kLocal, !kLocal>(x, region, tw, p, one_s, lt, bar);
        ntt16_store_slots<LOGD>(x, region, lt);
      }
      __syncthreads();
#pragma unroll
      for (int u = 0; u < kQuads; ++u) {
        const int e = 4 * (tid + u * kThreads);
        if (e < d) {
#pragma unroll
          for (int m = 0; m < 4; ++m) {
            // Slot e + m times the key part read through X -> X^power
            // (pp_link's permutation).
            const int odd = 2 * pp_bitrev(e + m, LOGD) + 1;
            const int from = pp_bitrev(((power * odd) & (2 * d - 1)) >> 1, LOGD);
            const int at = ntt16_pos<LOGD>(e + m);
#pragma unroll
            for (int o = 0; o < SIDE; ++o) {
              if (l0 + o < k) {
                uint32_t w;
                if constexpr (kLocal) {
                  w = W[(l0 + o) * d + from];
                } else {
                  w = __ldg(a.Wg + ((l0 + o) * R + pi) * d + from);
                }
                sum[u][m] += static_cast<uint64_t>(regions[o * d + at]) * w;
              }
            }
          }
        }
      }
      if (l0 + SIDE < k) __syncthreads();
    }
#pragma unroll
    for (int u = 0; u < kQuads; ++u) {
      const int e = 4 * (tid + u * kThreads);
      if (e < d) {
#pragma unroll
        for (int m = 0; m < 4; ++m) {
          regions[ntt16_pos<LOGD>(e + m)] = reduce_sum(sum[u][m], p, pinv, one_s);
        }
      }
    }
    if (i != d / 2 - 2) cluster_wait();  // the last link's residues have been read
    __syncthreads();
    if (grp == 0) {
      ntt16_load_slots<LOGD>(x, region, lt);
      ntt16_inverse<LOGD, kLocal, !kLocal>(x, region, itw, p, one_s, lt, bar);
#pragma unroll
      for (int m = 0; m < 16; ++m) {
        res[lt + NT * m] = shoup_mul(x[m], crt.scale[pi], crt.scale_s[pi], p);
      }
    }
    T own[kWords];
#pragma unroll
    for (int n = 0; n < kWords; ++n) {
      const int j = tid + n * kThreads;
      own[n] = j < d ? __ldg(add + j) : T{0};
    }
    cluster_arrive();
    cluster_wait();
    T* to = out + static_cast<int64_t>(i - 1) * k * d;
    T* f = fin + (static_cast<int64_t>(s) * 2 + chain) * d;
#pragma unroll
    for (int n = 0; n < kWords; ++n) {
      const int j = tid + n * kThreads;
      if (j >= d) break;
      T acc = own[n];
      uint32_t frac = 1u << 25;
#pragma unroll
      for (int q = 0; q < R; ++q) {
        const uint32_t y = cluster_load(peer[q] + 4 * j);
        acc += static_cast<T>(y) * static_cast<T>(crt.part[q]);
        frac += __umulhi(y, crt.frac[q]);
      }
      acc -= static_cast<T>(static_cast<T>(frac >> 26) * static_cast<T>(crt.m));
      if (i > 0) {
        put_digits(j, acc, to, n % R == pi);
      } else if (n % R == pi) {
        f[j] = acc;
      }
    }
    cluster_arrive();  // the residues are read
    __syncthreads();
  }
  cluster_wait();
}
#endif

}  // namespace inspire
