// ExternalProduct (crypto/external_product.cc:35-114) of a batch of ciphertexts,
// each with its own RGSW ciphertext, in one launch for d = 2048 and 4096: a
// cluster of one CTA per prime for each ciphertext.
//
// Every RGSW row is used once, so its transform never leaves the registers:
// group g transforms digit g, then the row's a and b polynomials, and
// multiplies slot by slot in the layout the transforms leave. Rows of digits
// that are always zero are not read. The launches this replaces (two
// transforms of all rows, the product, the reconstruction) wrote and read
// every row's residues and took 152 us for 256 ciphertexts at d = 2048 over
// Z_2^32 (the packing workload around them: 250 -> 183 us).
#pragma once
#include <cstdint>

#include "answer_poly.cuh"

namespace inspire {

template <typename T>
struct ExtProductArgs {
  const T* ct;    // [batch][2][d]
  const T* rgsw;  // [batch][2 ne][2][d]
  T* out;         // [batch][2][d]
  T vmask;        // bits of an RGSW word the chunk rule reads
  ExtArgs e;
  CrtArgs crt;
  NttCtx c;
};

// Bytes of shared memory: twiddle pairs, a buffer per group, two residue
// vectors, the ciphertext's gadget words.
template <typename T, int LOGD, int G>
constexpr size_t ExtProductSmem() {
  return static_cast<size_t>(Ntt16<LOGD>::kD) * (16 + 4 * G + 8 + 2 * sizeof(T));
}

#ifdef __CUDACC__
// grid = (R, batch), clusters of R, G d / 16 threads. kOne: a digit per group
// at most (the products go straight to shared memory, 64 registers).
template <typename T, int LOGD, int G, bool kOne, int R>
__global__ void __launch_bounds__(G * Ntt16<LOGD>::kThreads,
                                  kOne && G * Ntt16<LOGD>::kThreads <= 512 ? 2 : 1)
ext_product_kernel(const __grid_constant__ ExtProductArgs<T> a) {
  extern __shared__ __align__(16) uint32_t smem[];
  constexpr int d = Ntt16<LOGD>::kD;
  constexpr int NT = Ntt16<LOGD>::kThreads;
  constexpr int kThreads = G * NT;
  static_assert(G >= 2 && G <= 8, "sum of the partials");
  const NttCtx& c = a.c;
  const int tid = threadIdx.x;
  const int grp = tid / NT;
  const int lt = tid & (NT - 1);
  const int bar = 1 + grp;
  const int pi = blockIdx.x;
  const int q = blockIdx.y;
  const uint32_t p = c.p[pi], pinv = c.pinv[pi], one_s = c.one_s[pi];
  const uint2* tw = reinterpret_cast<const uint2*>(smem);
  const uint2* itw = tw + d;
  uint32_t* regions = smem + 4 * d;
  uint32_t* region = regions + grp * d;
  uint32_t* res = regions + G * d;
  T* st = reinterpret_cast<T*>(res + 2 * d);
  {
    const uint4* src =
        reinterpret_cast<const uint4*>(c.tables16 + static_cast<size_t>(pi) * 2 * d);
    uint4* dst = reinterpret_cast<uint4*>(smem);
    for (int i = tid; i < d; i += kThreads) dst[i] = __ldg(src + i);
    const T* ct = a.ct + static_cast<int64_t>(q) * 2 * d;
    for (int i = tid; i < 2 * d; i += kThreads) {
      st[i] = gadget_word<T>(low_bits<T>(ct[i], a.e.log_q), a.e);
    }
  }
  __syncthreads();
  const int n_live = 2 * a.e.live_digits;
  const bool small_digits = a.e.log_digit <= 27;
  const T digit_mask = low_bits<T>(static_cast<T>(a.e.umask), a.e.log_digit);
  // One polynomial of the RGSW row, transformed (below 2p, as Montgomery
  // products with an unreduced factor need).
  auto row_poly = [&](uint32_t (&y)[16], const T* poly) {
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      y[k] = reduce_word(static_cast<T>(poly[lt + NT * k] & a.vmask), c, pi);
    }
    ntt16_forward<LOGD, true>(y, region, tw, p, one_s, lt, bar);
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      const uint32_t r = barrett_lazy(y[k], one_s, p);
      y[k] = umin32(r, r - p);
    }
  };
  auto digit = [&](uint32_t (&x)[16], int poly, int dg) {
    const T* src = st + poly * d + lt;
    const int sh = dg * a.e.log_digit;
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      const T v = (src[NT * k] >> sh) & digit_mask;
      x[k] = small_digits ? static_cast<uint32_t>(v) : reduce_word(v, c, pi);
    }
  };
  auto poly_of = [&](int ti) { return ti < a.e.live_digits ? 0 : 1; };
  auto row_of = [&](int ti) {
    const int poly = poly_of(ti);
    return a.rgsw + (static_cast<int64_t>(q) * 2 * a.e.num_digits +
                     poly * a.e.num_digits + ti - poly * a.e.live_digits) * 2 * d;
  };
  uint32_t x[16], y[16];
  // Partial sums of a' and b' per group, in slot layout.
  uint32_t* parts_a = res;
  if constexpr (kOne) {
    // The a' parts go where nothing is kept any more once the digits are in
    // registers: the residue vectors and the gadget words behind them.
    static_assert(G <= 4, "room for the parts");
    const bool live = grp < n_live;
    if (live) digit(x, poly_of(grp), grp - poly_of(grp) * a.e.live_digits);
    __syncthreads();
    const T* row = live ? row_of(grp) : nullptr;
    if (live) ntt16_forward<LOGD, true>(x, region, tw, p, one_s, lt, bar);
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
      if (live) {
        row_poly(y, row + h * d);
#pragma unroll
        for (int k = 0; k < 16; ++k) y[k] = mont_mul_lazy(x[k], y[k], p, pinv);
      } else {
#pragma unroll
        for (int k = 0; k < 16; ++k) y[k] = 0;
      }
      ntt16_store_slots<LOGD>(y, h == 0 ? parts_a + grp * d : region, lt);
    }
  } else {
    uint32_t part_a[16], part_b[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) part_a[k] = part_b[k] = 0;
#pragma unroll 1
    for (int ti = grp; ti < n_live; ti += G) {
      const T* row = row_of(ti);
      digit(x, poly_of(ti), ti - poly_of(ti) * a.e.live_digits);
      ntt16_forward<LOGD, true>(x, region, tw, p, one_s, lt, bar);
#pragma unroll 1
      for (int h = 0; h < 2; ++h) {
        row_poly(y, row + h * d);
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          const uint32_t m = mont_mul_lazy(x[k], y[k], p, pinv);
          const uint32_t sa = part_a[k] + m, sb = part_b[k] + m;
          part_a[k] = h == 0 ? umin32(sa, sa - 2 * p) : part_a[k];
          part_b[k] = h == 0 ? part_b[k] : umin32(sb, sb - 2 * p);
        }
      }
    }
    // a' through the groups' buffers, then b'.
    ntt16_store_slots<LOGD>(part_a, region, lt);
    __syncthreads();
    if (grp == 0) {
#pragma unroll
      for (int k = 0; k < 16; ++k) x[k] = 0;
#pragma unroll 1
      for (int o = 0; o < G; ++o) {
        ntt16_load_slots<LOGD>(y, regions + o * d, lt);
#pragma unroll
        for (int k = 0; k < 16; ++k) x[k] += y[k];
      }
    }
    __syncthreads();
    ntt16_store_slots<LOGD>(part_b, region, lt);
  }
  // Group 0 sums and inverts a', group 1 b'.
  __syncthreads();
  if (grp == 1 || (kOne && grp == 0)) {
    const uint32_t* parts = grp == 1 ? regions : parts_a;
#pragma unroll
    for (int k = 0; k < 16; ++k) x[k] = 0;
#pragma unroll 1
    for (int o = 0; o < G; ++o) {
      ntt16_load_slots<LOGD>(y, parts + o * d, lt);
#pragma unroll
      for (int k = 0; k < 16; ++k) x[k] += y[k];
    }
  }
  __syncthreads();
  if (grp < 2) {
#pragma unroll
    for (int k = 0; k < 16; ++k) x[k] = barrett_lazy(x[k], one_s, p);
    ntt16_inverse<LOGD, true>(x, region, itw, p, one_s, lt, bar);
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      res[grp * d + lt + NT * k] = shoup_mul(x[k], a.crt.scale[pi], a.crt.scale_s[pi], p);
    }
  }
  cluster_arrive();
  cluster_wait();
  const uint32_t la = static_cast<uint32_t>(__cvta_generic_to_shared(res));
  uint32_t peer[R];
#pragma unroll
  for (int s = 0; s < R; ++s) peer[s] = cluster_map(la, s);
  T* out = a.out + static_cast<int64_t>(q) * 2 * d;
#pragma unroll 2
  for (int j = tid + pi * kThreads; j < 2 * d; j += R * kThreads) {
    T acc = 0;
    uint32_t k = 1u << 25;
#pragma unroll
    for (int s = 0; s < R; ++s) {
      const uint32_t v = cluster_load(peer[s] + 4 * j);
      acc += static_cast<T>(v) * static_cast<T>(a.crt.part[s]);
      k += __umulhi(v, a.crt.frac[s]);
    }
    out[j] = static_cast<T>(acc - static_cast<T>(k >> 26) * static_cast<T>(a.crt.m));
  }
  cluster_arrive();  // no CTA leaves while another reads its residues
  cluster_wait();
}
#endif

}  // namespace inspire
