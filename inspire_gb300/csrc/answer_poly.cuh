// The whole polynomial stage of an answer in one launch, for d = 2048 and
// 4096: FinalizeMatrixPack of every slice, the t - 1 external products of
// EvalPoly and the modulus switch (crypto/lwes_to_rlwe.cc:448-479,
// crypto/pir/server/pir_server.cc:128-150, 283-297).
//
// A cluster of r CTAs answers one (shard, request), one CTA per prime. Each
// keeps its prime's twiddle pairs in shared memory for the whole chain, and
// the product residues go to the other CTAs through distributed shared
// memory, so a Horner step costs two cluster barriers instead of a launch,
// and its transforms no longer wait on L2 for twiddles stage by stage (at
// one request or forty-five, a launch per step took 24-35 us of which the
// arithmetic was a few). The inner product <t_vec_h, y_vec_h> of slice i joins
// the external product before its inverse transform: integers add, so the
// slice needs no transform of its own. Only the first slice (no external
// product yet) and, when q < 2^w, the last one (its packed value is reduced
// mod q before the full word is rescaled) are inverted separately.
//
// Every block runs its code once per step, so the code is kept small enough
// for the instruction cache: one call site per transform, the prime count
// known at compile time. With both transforms inlined at every use and the
// general Garner reconstruction it came to 160 KB, and every phase waited on
// instruction fetch (26 us a step at d = 4096; 15 us now, 30 thousand cycles by
// clock64 stamps: transforms 10.5, products 5, inverse 6.4, barrier 1.8, words
// 4.5). Over Z_2^64 at d = 4096 it spills 200 bytes at 80 registers.
//
// G groups of d / 16 threads transform a gadget digit each (as many rounds as
// the live digits need); then every thread takes four slots of all digits and
// both outputs: the products are summed in 64 bits (three multiplier slots
// each instead of a Montgomery product's six) and reduced once. Groups 0 and
// 1 invert a' and b', group 2 a separate inner product.
#pragma once
#include <cstdint>

#include "poly_kernels.cuh"

namespace inspire {

// Reconstruction constants: with y_i = x_i (M / p_i)^-1 mod p_i (the inverse
// folded into the transform's scaling) the integer is sum_i y_i (M / p_i) - k M
// with k the nearest integer to sum_i y_i / p_i, taken from 26-bit fractions:
// they are off by less than 2^-23 in sum, and the products stay at least
// 2^-9 M away from the ends of (-M / 2, M / 2) (PrimesFor's margin). Per word
// and prime a multiply-add and a high product, where Garner's digits take a
// Montgomery product for every pair of primes.
struct CrtArgs {
  uint32_t scale[kMaxPrimes], scale_s[kMaxPrimes];  // d^-1 2^32 (M / p_i)^-1
  uint32_t frac[kMaxPrimes];                        // floor(2^58 / p_i)
  uint64_t part[kMaxPrimes];                        // M / p_i mod 2^64
  uint64_t m;                                       // M mod 2^64
};

template <typename T>
struct AnswerPolyArgs {
  const uint32_t* th;     // [l t][k][r][d] transforms of t_vec_h
  const uint32_t* yh;     // [batch][k][r][d] transforms of y_vec_h
  const T* gemv;          // [batch][l t d] stage-1 words
  const T* a_tilde;       // [l t][d]
  const uint32_t* rgswa;  // [2 ne][r][d]
  const uint32_t* rgswb;  // [batch][2 ne][r][d]
  T* resp;                // [batch][l][2][d]
  int k, t, log_q1, log_q2;
  ExtArgs e;
  CrtArgs crt;
  NttCtx c;
};

// Primes (27 bits each): three hold every Z_2^32 product of digits of up to 31
// bits, four the Z_2^64 products of digits of up to 27 bits.
template <typename T>
constexpr int AnswerPolyPrimes() {
  return sizeof(T) == 4 ? 3 : 4;
}

#ifdef __CUDACC__
__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Shared-memory address `local` of this CTA in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t cluster_map(uint32_t local, int rank) {
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(local), "r"(rank));
  return a;
}
__device__ __forceinline__ uint32_t cluster_load(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}

// Bytes of dynamic shared memory: the twiddle pairs (4 d words), a d-word
// buffer per group, three residue vectors, the state (a, b).
template <typename T, int LOGD, int G>
constexpr size_t AnswerPolySmem() {
  return static_cast<size_t>(Ntt16<LOGD>::kD) * (16 + 4 * G + 12 + 2 * sizeof(T));
}

// A sum of products x w (w < p, the x below 2^32) in Montgomery form: the sum
// times 2^-32, below n p for n products plus 2 p, then below 2 p.
__device__ __forceinline__ uint32_t reduce_sum(uint64_t s, uint32_t p, uint32_t pinv,
                                               uint32_t one_s) {
  const uint32_t m = static_cast<uint32_t>(s) * pinv;
  return barrett_lazy(static_cast<uint32_t>(s >> 32) - __umulhi(m, p) + p, one_s, p);
}

// A LowBits'd coefficient after GadgetInv's rounding shift (gadget_digit's
// `cur`): digit i is its bits from i log_digit on.
template <typename T>
__device__ __forceinline__ T gadget_word(T c, const ExtArgs& e) {
  const int to_shift = e.log_q - e.num_digits * e.log_digit;
  return to_shift > 0 ? (c >> to_shift) + ((c >> (to_shift - 1)) & T{1}) : c;
}

// grid = (r l, batch), clusters of r = R, G d / 16 threads.
template <typename T, int LOGD, int G, int R>
__global__ void __launch_bounds__(G * Ntt16<LOGD>::kThreads,
                                  G * Ntt16<LOGD>::kThreads <= 512 ? 2 : 1)
answer_poly_kernel(const __grid_constant__ AnswerPolyArgs<T> a) {
  extern __shared__ __align__(16) uint32_t smem[];
  constexpr int d = Ntt16<LOGD>::kD;
  constexpr int NT = Ntt16<LOGD>::kThreads;
  constexpr int kThreads = G * NT;
  constexpr int kQuads = (d / 4 + kThreads - 1) / kThreads;  // slot quads per thread
  static_assert(G >= 3, "a group per inverse transform");
  const NttCtx& c = a.c;
  constexpr int r = R;
  const int tid = threadIdx.x;
  const int grp = tid / NT;
  const int lt = tid & (NT - 1);
  const int bar = 1 + grp;
  const int pi = blockIdx.x % r;  // rank in the cluster
  const int shard = blockIdx.x / r;
  const int l = gridDim.x / r;
  const int q = blockIdx.y;
  const uint32_t p = c.p[pi];
  const uint32_t pinv = c.pinv[pi];
  const uint32_t one_s = c.one_s[pi];

  const uint2* tw = reinterpret_cast<const uint2*>(smem);
  const uint2* itw = tw + d;
  uint32_t* regions = smem + 4 * d;
  uint32_t* region = regions + grp * d;
  uint32_t* res = regions + G * d;  // a', b', separate inner product
  T* st = reinterpret_cast<T*>(res + 3 * d);  // gadget words of a, then of b
  {
    const uint4* src = reinterpret_cast<const uint4*>(c.tables16 + static_cast<size_t>(pi) * 2 * d);
    uint4* dst = reinterpret_cast<uint4*>(smem);
    for (int i = tid; i < d; i += kThreads) dst[i] = __ldg(src + i);
  }
  __syncthreads();

  const int ng = 2 * a.e.num_digits;
  const int n_live = 2 * a.e.live_digits;
  const bool small_digits = a.e.log_digit <= 27;
  const T digit_mask = low_bits<T>(static_cast<T>(a.e.umask), a.e.log_digit);
  const int64_t step = static_cast<int64_t>(r) * d;  // one polynomial's residues
  const uint32_t* rgswa = a.rgswa + static_cast<int64_t>(pi) * d;
  const uint32_t* rgswb = a.rgswb + (static_cast<int64_t>(q) * ng * r + pi) * d;
  const uint32_t* yh = a.yh + (static_cast<int64_t>(q) * a.k * r + pi) * d;
  auto row_of = [&](int ti) {  // digit ti (those of a, then of b) in the RGSW ciphertext
    return ti < a.e.live_digits ? ti : ti - a.e.live_digits + a.e.num_digits;
  };

  for (int i = a.t - 1; i >= 0; --i) {
    const bool first = i == a.t - 1;
    const bool sep = first || (i == 0 && a.e.log_q < Bits<T>::value);
    uint64_t sum_a[kQuads][4], sum_b[kQuads][4], sum_c[kQuads][4];
#pragma unroll
    for (int u = 0; u < kQuads; ++u) {
#pragma unroll
      for (int m = 0; m < 4; ++m) sum_a[u][m] = sum_b[u][m] = sum_c[u][m] = 0;
    }
    uint32_t x[16];
#pragma unroll 1
    for (int t0 = 0; t0 == 0 || t0 < n_live; t0 += G) {
      if (!first && t0 + grp < n_live) {
        const int row = row_of(t0 + grp);
        const int poly = row < a.e.num_digits ? 0 : 1;
        const T* src = st + poly * d + lt;
        const int sh = (row - poly * a.e.num_digits) * a.e.log_digit;
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          const T dig = (src[NT * k] >> sh) & digit_mask;
          x[k] = small_digits ? static_cast<uint32_t>(dig) : reduce_word(dig, c, pi);
        }
        ntt16_forward<LOGD, true>(x, region, tw, p, one_s, lt, bar);
        ntt16_store_slots<LOGD>(x, region, lt);
      }
      if (t0 == 0) {
        // The slice's inner product, while other groups still transform.
#pragma unroll
        for (int u = 0; u < kQuads; ++u) {
          const int e = 4 * (tid + u * kThreads);
          if (e < d) {
            const uint32_t* th =
                a.th + (static_cast<int64_t>(shard * a.t + i) * a.k * r + pi) * d + e;
#pragma unroll 2
            for (int j = 0; j < a.k; ++j) {
              const uint4 y = __ldg(reinterpret_cast<const uint4*>(yh + j * step + e));
              const uint4 h = __ldg(reinterpret_cast<const uint4*>(th + j * step));
              sum_c[u][0] += static_cast<uint64_t>(h.x) * y.x;
              sum_c[u][1] += static_cast<uint64_t>(h.y) * y.y;
              sum_c[u][2] += static_cast<uint64_t>(h.z) * y.z;
              sum_c[u][3] += static_cast<uint64_t>(h.w) * y.w;
            }
          }
        }
        if (first) break;
      }
      __syncthreads();
#pragma unroll
      for (int u = 0; u < kQuads; ++u) {
        const int e = 4 * (tid + u * kThreads);
        if (e < d) {
          int pos[4];
#pragma unroll
          for (int m = 0; m < 4; ++m) pos[m] = ntt16_pos<LOGD>(e + m);
#pragma unroll
          for (int o = 0; o < G; ++o) {
            if (t0 + o < n_live) {
              const int64_t at = row_of(t0 + o) * step + e;
              const uint4 va = __ldg(reinterpret_cast<const uint4*>(rgswa + at));
              const uint4 vb = __ldg(reinterpret_cast<const uint4*>(rgswb + at));
              const uint32_t wa[4] = {va.x, va.y, va.z, va.w};
              const uint32_t wb[4] = {vb.x, vb.y, vb.z, vb.w};
#pragma unroll
              for (int m = 0; m < 4; ++m) {
                const uint64_t v = regions[o * d + pos[m]];
                sum_a[u][m] += v * wa[m];
                sum_b[u][m] += v * wb[m];
              }
            }
          }
        }
      }
      if (t0 + G < n_live) __syncthreads();  // the next round overwrites the digits
    }
    // a', b' and c to the groups that invert them.
#pragma unroll
    for (int u = 0; u < kQuads; ++u) {
      const int e = 4 * (tid + u * kThreads);
      if (e < d) {
#pragma unroll
        for (int m = 0; m < 4; ++m) {
          const int at = ntt16_pos<LOGD>(e + m);
          if (!first) {
            regions[at] = reduce_sum(sum_a[u][m], p, pinv, one_s);
            regions[d + at] =
                reduce_sum(sum_b[u][m] + (sep ? 0 : sum_c[u][m]), p, pinv, one_s);
          }
          if (sep) regions[2 * d + at] = reduce_sum(sum_c[u][m], p, pinv, one_s);
        }
      }
    }
    if (!first) cluster_wait();  // the last step's residues have been read
    __syncthreads();
    if (grp < 2 ? !first : (grp == 2 && sep)) {
      ntt16_load_slots<LOGD>(x, region, lt);
      ntt16_inverse<LOGD, true>(x, region, itw, p, one_s, lt, bar);
#pragma unroll
      for (int m = 0; m < 16; ++m) {
        res[grp * d + lt + NT * m] = shoup_mul(x[m], a.crt.scale[pi], a.crt.scale_s[pi], p);
      }
    }
    cluster_arrive();
    // The state of every coefficient (each CTA needs all of them) or, at the
    // last slice, the response (each CTA writes its share). The slice's own
    // words come in before the other CTAs' residues do.
    const int j0 = i > 0 ? tid : tid + pi * kThreads;
    const int dj = i > 0 ? kThreads : r * kThreads;
    const T* ca = a.a_tilde + (static_cast<int64_t>(shard) * a.t + i) * d;
    const T* cg = a.gemv + (static_cast<int64_t>(q) * l * a.t + shard * a.t + i) * d;
    constexpr int kWords = (d + kThreads - 1) / kThreads;
    constexpr int kAhead = kWords <= 4 ? kWords : 1;  // as many as registers allow
    T wa[kAhead], wg[kAhead];
    auto own = [&](int n) {
      const int j = j0 + n * dj;
      wa[n % kAhead] = j < d ? __ldg(ca + j) : T{0};
      wg[n % kAhead] = j < d ? cg[j] : T{0};
    };
#pragma unroll
    for (int n = 0; n < kAhead; ++n) own(n);
    cluster_wait();
    const uint32_t la = static_cast<uint32_t>(__cvta_generic_to_shared(res));
    uint32_t peer[R];
#pragma unroll
    for (int s = 0; s < R; ++s) peer[s] = cluster_map(la, s);
    auto word = [&](int j, uint32_t off) {
      T acc = 0;
      uint32_t k = 1u << 25;
#pragma unroll
      for (int s = 0; s < R; ++s) {
        const uint32_t y = cluster_load(peer[s] + off + 4 * j);
        acc += static_cast<T>(y) * static_cast<T>(a.crt.part[s]);
        k += __umulhi(y, a.crt.frac[s]);
      }
      return static_cast<T>(acc - static_cast<T>(k >> 26) * static_cast<T>(a.crt.m));
    };
    T* oa = a.resp + (static_cast<int64_t>(q) * l + shard) * 2 * d;
#pragma unroll kAhead
    for (int n = 0; n < kWords; ++n) {
      const int j = j0 + n * dj;
      if (j >= d) break;
      T ra = wa[n % kAhead], rb = wg[n % kAhead];
      if (n + kAhead < kWords) own(n + kAhead);
      if (sep) rb = low_bits<T>(static_cast<T>(rb + word(j, 8 * d)), a.e.log_q);
      if (!first) {
        ra += word(j, 0);
        rb += word(j, 4 * d);
      }
      if (i > 0) {
        // What GadgetInv takes its digits from.
        st[j] = gadget_word<T>(low_bits<T>(ra, a.e.log_q), a.e);
        st[d + j] = gadget_word<T>(low_bits<T>(rb, a.e.log_q), a.e);
      } else {
        oa[j] = rescale_word<T>(ra, a.e.log_q, a.log_q1);
        oa[d + j] = rescale_word<T>(rb, a.e.log_q, a.log_q2);
      }
    }
    // The residues are read: they are overwritten (and the CTA left) only
    // after every CTA of the cluster has got here.
    cluster_arrive();
    __syncthreads();
  }
  cluster_wait();
}
#endif

}  // namespace inspire
