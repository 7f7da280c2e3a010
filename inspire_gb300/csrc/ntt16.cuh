// Register-resident negacyclic NTT for d = 2^LOGD (LOGD = 11, 12, 13) with
// d / 16 threads: passes of up to four stages on 16 coefficients per
// thread, exchanges through shared memory in between.
//
// The transform is the one of ntt.cuh (Cooley-Tukey forward with the
// psi-twisted twiddles, natural order in and bit-reversed order out;
// Gentleman-Sande inverse), so both give the same residues. Only the
// grouping of the stages differs. Stage j (m = 2^j groups, distance
// t = d / 2m) takes the pair (e, e + t) of group i = e / 2t with twiddle
// W[m + i]. A pass is a window of four stages sp .. sp + 3, of which the
// first `skip` are left out: (0, 0), (4, 0), (8, 0), ... and, when LOGD is
// not a multiple of 4, a last window (LOGD - 4, 4 - LOGD % 4). With
// m0 = 2^sp and t0 = d / (2 m0), a thread holds the 16 coefficients
// e_k = 2 g t0 + o + k t0 / 8 of group g = tid / (t0 / 8) and offset
// o = tid % (t0 / 8). The first pass reads e_k = tid + (d / 16) k (natural
// order, coalesced), the last one e_k = 16 tid + k. Stage s of a window
// pairs k with k + 8 / 2^s and takes W[m0 2^s + g 2^s + (k >> (4 - s))].
//
// Twiddles are read as (value, Shoup constant) pairs from a permuted copy of
// the tables (ntt_tables_kernel): window w, stage s, sub-block x, group g at
// base_w + m0 (2^s - 2^skip) + x m0 + g, so the threads of a warp read one
// pair, a few pairs or consecutive pairs.
//
// The primes are below 2^27, so 32 p < 2^32 and the butterflies reduce
// nothing (after Harvey, "Faster arithmetic for number-theoretic transforms",
// 2014, whose [0, 4p) this stretches): a forward butterfly is Shoup's product
// without its correction (three multiplier instructions, four of the 64
// lanes per cycle that a multiplier takes, since the high product counts
// twice), u + v and u - v + 2p, and a value grows by at most 2p per stage.
// An inverse butterfly doubles the bound of its sum, so every window of four
// stages ends with one reduction of the values above 2p. With 31-bit primes
// the same butterfly took four more instructions and the transforms were
// bound by issue; the multiplier is the bound now.
//
// Shared memory holds coefficient e at e ^ swz(e >> 5), with a swz per size
// that keeps every pass's access pattern free of bank conflicts (the
// patterns and the swz were checked exhaustively on the host).
#pragma once
#include <cstdint>

#include "arith.cuh"

namespace inspire {

constexpr int kNtt16MinLogD = 11;
constexpr int kNtt16MaxLogD = 13;

template <int LOGD>
struct Ntt16 {
  static_assert(LOGD >= kNtt16MinLogD && LOGD <= kNtt16MaxLogD, "ring degree");
  static constexpr int kD = 1 << LOGD;
  static constexpr int kThreads = kD / 16;
  static constexpr int kPasses = (LOGD + 3) / 4;
  __host__ __device__ static constexpr int Start(int w) {
    return (w < kPasses - 1 || LOGD % 4 == 0) ? 4 * w : LOGD - 4;
  }
  __host__ __device__ static constexpr int Skip(int w) {
    return (w == kPasses - 1 && LOGD % 4 != 0) ? 4 - LOGD % 4 : 0;
  }
  // First slot of window w: the full windows before it hold 15 m0 each.
  __host__ __device__ static constexpr int Base(int w) {
    int b = 0;
    for (int i = 0; i < w; ++i) b += 15 << (4 * i);
    return b;
  }
};

#ifdef __CUDACC__
template <int LOGD>
__device__ __forceinline__ int ntt16_pos(int e) {
  const int r = e >> 5;
  if constexpr (LOGD == 11) {
    return e ^ ((r & 7) | ((((r >> 3) ^ (r >> 2)) & 1) << 3) | (((r >> 3) & 1) << 4));
  } else if constexpr (LOGD == 12) {
    return e ^ ((r & 15) | (((r >> 3) & 1) << 4));
  } else {
    return e ^ ((r & 15) ^ ((r & 15) << 1));
  }
}

// Geometry of window w for thread tid: coefficient e_k = base + stride * k,
// group g.
template <int LOGD>
__device__ __forceinline__ void ntt16_geometry(int w, int tid, int& base, int& stride,
                                               int& g) {
  const int m0 = 1 << Ntt16<LOGD>::Start(w);
  const int t0 = Ntt16<LOGD>::kD / (2 * m0);
  stride = t0 / 8;
  g = tid / stride;
  base = 2 * g * t0 + tid % stride;
}

// Barrier of the threads running one transform: the whole block (bar == 0)
// or named barrier `bar` when several groups of threads run transforms of
// their own.
template <int LOGD>
__device__ __forceinline__ void ntt16_sync(int bar) {
  if (bar == 0) {
    __syncthreads();
  } else {
    asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(Ntt16<LOGD>::kThreads) : "memory");
  }
}

// A twiddle pair: read-only global memory (kSmem = false) or a copy of the
// tables in shared memory.
template <bool kSmem>
__device__ __forceinline__ uint2 ntt16_tw(const uint2* t, int i) {
  if constexpr (kSmem) {
    return t[i];
  } else {
    return __ldg(t + i);
  }
}

// Before the inverse stage of half-length h = 2^L (stages 1, 2, .. 2^(L-1)
// done on values below 2p), coefficient k holds less than 2p << grow(k, L):
// its bound doubled in each stage since it last came out of a product.
__host__ __device__ constexpr int ntt16_grow(int k, int L) {
  const int i = k & ((1 << L) - 1);
  if (i == 0) return L;
  int hb = 0;
  while ((i >> (hb + 1)) != 0) ++hb;
  return L - 1 - hb;
}

// The stages of window w on the thread's 16 coefficients, forward (Cooley-
// Tukey, stages skip .. 3) or inverse (Gentleman-Sande, 3 .. skip). With a
// compile-time window every index folds; the compact transforms pass a
// run-time one and the same instructions serve every window. Forward: adds
// less than 2p per stage to values of any size below 2^32. Inverse: from
// values below 2p to values below 32p.
template <int LOGD, bool kSmem, bool kInverse>
__device__ __forceinline__ void ntt16_window(uint32_t (&x)[16], const uint2* __restrict__ tw,
                                             uint32_t p, int w, int g) {
  const int m0 = 1 << Ntt16<LOGD>::Start(w);
  const int skip = Ntt16<LOGD>::Skip(w);
  const int base = Ntt16<LOGD>::Base(w) + g - m0 * (1 << skip);
  const uint32_t p2 = 2 * p;
#pragma unroll
  for (int si = 0; si < 4; ++si) {
    const int s = kInverse ? 3 - si : si;
    if (s < skip) continue;
    const int half = 8 >> s;
    uint2 wv[8];
#pragma unroll
    for (int b = 0; b < (1 << s); ++b) wv[b] = ntt16_tw<kSmem>(tw, base + m0 * ((1 << s) + b));
#pragma unroll
    for (int b = 0; b < (1 << s); ++b) {
#pragma unroll
      for (int i = 0; i < half; ++i) {
        const int k = b * 2 * half + i;
        const uint32_t u = x[k], v = x[k + half];
        if (kInverse) {
          x[k] = u + v;
          x[k + half] =
              shoup_mul_lazy(u - v + (p2 << ntt16_grow(i, 3 - s)), wv[b].x, wv[b].y, p);
        } else {
          const uint32_t y = shoup_mul_lazy(v, wv[b].x, wv[b].y, p);
          x[k] = u + y;
          x[k + half] = u - y + p2;
        }
      }
    }
  }
}

// How far coefficient k of window w's inverse result may be above 2p (below
// 2p << n); with w < 0 the largest over the windows that another one follows.
template <int LOGD>
__host__ __device__ constexpr int ntt16_excess(int k, int w) {
  if (w >= 0) return ntt16_grow(k, 4 - Ntt16<LOGD>::Skip(w));
  int n = 0;
  for (int v = 1; v < Ntt16<LOGD>::kPasses; ++v) {
    const int e = ntt16_grow(k, 4 - Ntt16<LOGD>::Skip(v));
    n = e > n ? e : n;
  }
  return n;
}

// Between two inverse windows: back below 2p.
template <int LOGD>
__device__ __forceinline__ void ntt16_settle(uint32_t (&x)[16], uint32_t p, uint32_t one_s,
                                             int w) {
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    const int n = ntt16_excess<LOGD>(k, w);
    if (n >= 2) {
      x[k] = barrett_lazy(x[k], one_s, p);
    } else if (n == 1) {
      x[k] = umin32(x[k], x[k] - 2 * p);
    }
  }
}

// Byte offset in a d-word buffer of the thread's coefficient k of window w.
// The swizzle is linear over GF(2) and the bits of stride * k are apart from
// those of the base, so the 16 offsets are one base XOR sums of four words:
// a few instructions where a general position took eight per coefficient,
// most of a compact pass's code.
template <int LOGD>
struct Ntt16Slots {
  uint32_t base, bit[4];
  __device__ __forceinline__ Ntt16Slots(int w, int tid) {
    int e, stride, g;
    ntt16_geometry<LOGD>(w, tid, e, stride, g);
    base = 4u * ntt16_pos<LOGD>(e);
#pragma unroll
    for (int i = 0; i < 4; ++i) bit[i] = 4u * ntt16_pos<LOGD>(stride << i);
  }
  __device__ __forceinline__ uint32_t operator()(int k) const {
    return base ^ ((k & 1) ? bit[0] : 0u) ^ ((k & 2) ? bit[1] : 0u) ^ ((k & 4) ? bit[2] : 0u) ^
           ((k & 8) ? bit[3] : 0u);
  }
};

template <int LOGD>
__device__ __forceinline__ void ntt16_store(const uint32_t (&x)[16], uint32_t* xs, int w,
                                            int tid) {
  const Ntt16Slots<LOGD> at(w, tid);
  char* b = reinterpret_cast<char*>(xs);
#pragma unroll
  for (int k = 0; k < 16; ++k) *reinterpret_cast<uint32_t*>(b + at(k)) = x[k];
}

template <int LOGD>
__device__ __forceinline__ void ntt16_load(uint32_t (&x)[16], const uint32_t* xs, int w,
                                           int tid) {
  const Ntt16Slots<LOGD> at(w, tid);
  const char* b = reinterpret_cast<const char*>(xs);
#pragma unroll
  for (int k = 0; k < 16; ++k) x[k] = *reinterpret_cast<const uint32_t*>(b + at(k));
}

// Forward transform. In: x[k] = coefficient tid + (d / 16) k, any value
// below 6p. Out: x[k] = NTT slot 16 tid + k (the bit-reversed output array of
// ntt_forward) below 32p, fit for a Montgomery product with a factor below p;
// reduced to [0, p) with kReduce. `xs` is a d-word shared buffer, free again
// when this returns. tw = the prime's forward pairs. tid in [0, d / 16) within
// the group that synchronises on `bar`. kSmem: the pairs were copied to
// shared memory. kCompact: one window body for all windows (a third of the
// code, for launches whose blocks each run once per SM, where fetching
// unrolled code sets the time).
template <int LOGD, bool kSmem = false, bool kCompact = false, bool kReduce = false>
__device__ __forceinline__ void ntt16_forward(uint32_t (&x)[16], uint32_t* xs,
                                              const uint2* __restrict__ tw, uint32_t p,
                                              uint32_t one_s, int tid, int bar = 0) {
  using N = Ntt16<LOGD>;
  auto pass = [&](int w) {
    int base, stride, g;
    ntt16_geometry<LOGD>(w, tid, base, stride, g);
    if (w > 0) ntt16_load<LOGD>(x, xs, w, tid);
    ntt16_window<LOGD, kSmem, false>(x, tw, p, w, g);
    // The store goes to the words this thread read (no barrier between).
    if (w < N::kPasses - 1) ntt16_store<LOGD>(x, xs, w, tid);
    ntt16_sync<LOGD>(bar);
  };
  if constexpr (kCompact) {
#pragma unroll 1
    for (int w = 0; w < N::kPasses; ++w) pass(w);
  } else {
#pragma unroll
    for (int w = 0; w < N::kPasses; ++w) pass(w);
  }
  if constexpr (kReduce) {
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      const uint32_t r = barrett_lazy(x[k], one_s, p);
      x[k] = umin32(r, r - p);
    }
  }
}

// Inverse transform without the 1/d scaling. In: x[k] = slot 16 tid + k below
// 2p. Out: x[k] = coefficient tid + (d / 16) k below 32p (the scaling's Shoup
// product takes any word). itw = the prime's inverse pairs.
template <int LOGD, bool kSmem = false, bool kCompact = false>
__device__ __forceinline__ void ntt16_inverse(uint32_t (&x)[16], uint32_t* xs,
                                              const uint2* __restrict__ itw, uint32_t p,
                                              uint32_t one_s, int tid, int bar = 0) {
  using N = Ntt16<LOGD>;
  auto pass = [&](int w) {
    int base, stride, g;
    ntt16_geometry<LOGD>(w, tid, base, stride, g);
    if (w < N::kPasses - 1) ntt16_load<LOGD>(x, xs, w, tid);
    ntt16_window<LOGD, kSmem, true>(x, itw, p, w, g);
    if (w > 0) {
      ntt16_settle<LOGD>(x, p, one_s, kCompact ? -1 : w);
      ntt16_store<LOGD>(x, xs, w, tid);
    }
    ntt16_sync<LOGD>(bar);
  };
  if constexpr (kCompact) {
#pragma unroll 1
    for (int w = N::kPasses - 1; w >= 0; --w) pass(w);
  } else {
#pragma unroll
    for (int w = N::kPasses - 1; w >= 0; --w) pass(w);
  }
}

// The slot layout the forward transform leaves (x[k] = slot 16 tid + k) in
// and out of the d-word buffer `xs`, conflict-free.
template <int LOGD>
__device__ __forceinline__ void ntt16_store_slots(const uint32_t (&x)[16], uint32_t* xs,
                                                  int tid) {
  ntt16_store<LOGD>(x, xs, Ntt16<LOGD>::kPasses - 1, tid);
}

template <int LOGD>
__device__ __forceinline__ void ntt16_load_slots(uint32_t (&x)[16], const uint32_t* xs,
                                                 int tid) {
  ntt16_load<LOGD>(x, xs, Ntt16<LOGD>::kPasses - 1, tid);
}
#endif

}  // namespace inspire
