// Kernels of a batched PIR client (query generation and response
// decryption) for load generation and end-to-end tests.
//
// Reference: PirClient::CreateRequest / CreateFirstDimensionQuery /
// CreateSecondDimensionQuery / CreatePackingKey / ProcessResponse
// (crypto/pir/client/pir_client.cc:61-272) over GenerateRlweSamples,
// EncryptFromRlweSample, EncryptGadgetCiphertextFromRlweSamples,
// EncryptRgswCiphertextFromRlweSamples and DecryptAfterModulusSwitch
// (crypto/encryption.cc:150-518).
//
// Every RLWE sample is b = e - a s mod q for a public a-component a (the same
// ones the server preprocessed) and the client's ternary key s; a s is an
// exact multi-prime NTT product. The error e is a centred binomial of the
// parameters' variance drawn from a counter-based hash (the SplitMix64
// finaliser) of (seed, client, row, coefficient): reproducible and fast, NOT
// a cryptographic generator; the reference's clients use ChaCha.
#pragma once
#include <cstdint>

#include "hint16.cuh"

namespace inspire {

// SplitMix64 finaliser (Steele, Lea, Flood 2014).
__device__ __forceinline__ uint64_t cl_mix(uint64_t z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

// Centred binomial of variance var: popcount of 2 var bits minus popcount of
// 2 var further bits of the stream of hash words. Which bits of a word count
// with which sign depends on its number alone, so a word is two masked
// popcounts.
__device__ __forceinline__ int cl_error(uint64_t seed, uint64_t ctr, int var) {
  const int n = 2 * var;
  int acc = 0;
  for (int lo = 0, word = 0; lo < 2 * n; lo += 64, ++word) {
    const uint64_t bits = cl_mix(seed ^ cl_mix((ctr << 6) + word));
    auto low = [&](int count) {
      return count >= 64 ? ~0ull : count <= 0 ? 0ull : (1ull << count) - 1;
    };
    const uint64_t plus = low(n - lo);
    acc += __popcll(bits & plus) - __popcll(bits & low(2 * n - lo) & ~plus);
  }
  return acc;
}

struct ClientArgs {
  int d, log_d, log_q, k_pack, ne, ns;   // ns first-dimension samples
  int t;                                 // interpolation degree
  int64_t fd_len;                        // first-dimension query words
  int pack_log_digit, eval_log_digit;
  int var;
  uint64_t seed;
  uint64_t plaintext_modulus;
  const int8_t* keys;                    // [batch][d] ternary secret keys
  const int64_t* index;                  // [batch]
};

template <typename T>
__device__ __forceinline__ T cl_qmask(int log_q) {
  return log_q >= static_cast<int>(8 * sizeof(T)) ? ~T{0} : ((T{1} << log_q) - 1);
}

// Coefficient j of X^e * s (0 <= e < 2d) for a ternary s, as a word.
template <typename T>
__device__ __forceinline__ T cl_shift_key(const int8_t* s, int d, int e, int j) {
  bool neg = e >= d;
  if (neg) e -= d;
  int i = j - e;
  if (i < 0) {
    i += d;
    neg = !neg;
  }
  const int v = neg ? -s[i] : s[i];
  return static_cast<T>(static_cast<int64_t>(v));
}

// Coefficient j of s(X^p) (Polynomial::Automorph) for odd p: the i with
// i p = j (or j + d, negated) mod 2d; pinv = p^-1 mod 2d.
template <typename T>
__device__ __forceinline__ T cl_aut_key(const int8_t* s, int d, int pinv, int j) {
  const int e = static_cast<int>(static_cast<int64_t>(j) * pinv & (2 * d - 1));
  const int v = e < d ? s[e] : -s[e - d];
  return static_cast<T>(static_cast<int64_t>(v));
}

// Forward NTTs of the ternary keys: out[b][pi][d]. grid = (r, batch).
template <int ITERS>
__global__ void __launch_bounds__(1024)
cl_key_ntt_kernel(const int8_t* __restrict__ keys, NttCtx c, uint32_t* __restrict__ out) {
  extern __shared__ uint32_t cl_smem[];
  const int d = 1 << c.logd;
  const int pi = blockIdx.x, b = blockIdx.y;
  const uint32_t p = c.p[pi];
  for (int j = threadIdx.x; j < d; j += blockDim.x) {
    const int v = keys[static_cast<int64_t>(b) * d + j];
    cl_smem[j] = v >= 0 ? static_cast<uint32_t>(v) : p - static_cast<uint32_t>(-v);
  }
  ntt_forward_t<ITERS>(cl_smem, c, pi);
  uint32_t* o = out + (static_cast<int64_t>(b) * c.r + pi) * d;
  for (int j = threadIdx.x; j < d; j += blockDim.x) o[j] = cl_smem[j];
}

// a s for one a (T words) and one key transform: leaves the r residue
// vectors of the product in sm (r * d words), read back by cl_crt.
template <typename T, int ITERS>
__device__ __forceinline__ void cl_times_key(const T* a, const uint32_t* s_hat, uint32_t* sm,
                                             const NttCtx& c, int d) {
  for (int pi = 0; pi < c.r; ++pi) {
    uint32_t* x = sm + static_cast<int64_t>(pi) * d;
    const uint32_t p = c.p[pi];
    for (int j = threadIdx.x; j < d; j += blockDim.x) {
      x[j] = reduce_word(a[j], c, pi);
    }
    ntt_forward_t<ITERS>(x, c, pi);
    const uint32_t* sh = s_hat + static_cast<int64_t>(pi) * d;
    for (int j = threadIdx.x; j < d; j += blockDim.x) {
      x[j] = mont_mul(x[j], __ldg(sh + j), p, c.pinv[pi]);
    }
    ntt_inverse_t<ITERS>(x, c, pi);
  }
}

template <typename T>
__device__ __forceinline__ T cl_crt(const uint32_t* sm, const NttCtx& c, int d, int j) {
  uint32_t x[kMaxPrimes] = {0, 0, 0, 0, 0};
#pragma unroll
  for (int pi = 0; pi < kMaxPrimes; ++pi) {
    if (pi < c.r) {
      x[pi] = shoup_mul(sm[static_cast<int64_t>(pi) * d + j], c.scale[pi], c.scale_s[pi],
                        c.p[pi]);
    }
  }
  return crt_reconstruct<T>(x, c);
}

// One request row per block: rows [0, ns) are the first-dimension samples
// (Enc(one-hot)), then 2 ne second-dimension gadget rows (u: m s, v: m, the
// monomial X^{(2d/t) col}), then 2 k packing-key rows (gadget encryptions of
// s(X^5) and s(X^{2d-1})). What a block needs of its row and client:
template <typename T>
struct ClientRow {
  const int8_t* s;
  uint64_t ctr;       // of coefficient 0's error
  int row, hot;       // hot: the coefficient of the one-hot message, or -1
  int shift, digit_shift, kind, pinv;
  T* out;             // of coefficient 0
  int64_t len;        // coefficients kept

  __device__ __forceinline__ ClientRow(const ClientArgs& a, int row_, int rows, int b, T* fd,
                                       T* sd, T* pk)
      : row(row_) {
    const int d = a.d;
    s = a.keys + static_cast<int64_t>(b) * d;
    ctr = (static_cast<uint64_t>(b) * rows + row) * d;
    const int64_t index = a.index[b];
    const int row_index = static_cast<int>(index / a.t);
    shift = (2 * d / a.t) * static_cast<int>(index % a.t);
    hot = -1;
    kind = 0;
    digit_shift = 0;
    pinv = 2 * d - 1;
    len = d;
    if (row < a.ns) {
      if (row == row_index / d) hot = row_index % d;
      out = fd + static_cast<int64_t>(b) * a.fd_len + static_cast<int64_t>(row) * d;
      len = a.fd_len - static_cast<int64_t>(row) * d;
      return;
    }
    int g = row - a.ns, nd, log_digit, digit;
    if (g < 2 * a.ne) {
      nd = a.ne;
      log_digit = a.eval_log_digit;
      digit = g < a.ne ? g : g - a.ne;
      kind = g < a.ne ? 1 : 2;
      out = sd + (static_cast<int64_t>(b) * 2 * a.ne + g) * d;
    } else {
      g -= 2 * a.ne;
      nd = a.k_pack;
      log_digit = a.pack_log_digit;
      digit = g < a.k_pack ? g : g - a.k_pack;
      kind = 3;
      // s(X^5) or s(X^{2d-1}); inverses of 5 and 2d-1 mod 2d.
      if (g < a.k_pack) {
        // 5^-1 mod 2d by Newton iteration (2d is a power of two).
        uint32_t x = 5;
        for (int it = 0; it < 5; ++it) x *= 2 - 5 * x;
        pinv = static_cast<int>(x & static_cast<uint32_t>(2 * d - 1));
      }
      out = pk + (static_cast<int64_t>(b) * 2 * a.k_pack + g) * d;
    }
    // EncryptGadgetCiphertextFromRlweSamples: y = b + (target << (i l + off)).
    digit_shift = digit * log_digit + max(0, a.log_q - nd * log_digit);
  }

  // Coefficient j of the row from that of a s.
  __device__ __forceinline__ void put(const ClientArgs& a, int j, T as) const {
    constexpr int kW = 8 * sizeof(T);
    const T qm = cl_qmask<T>(a.log_q);
    const int e = cl_error(a.seed, ctr + j, a.var);
    T v = static_cast<T>(static_cast<T>(static_cast<int64_t>(e)) - as) & qm;
    if (kind == 0) {
      // EncryptFromRlweSample of the one-hot message: + round(m q / p).
      if (j == hot) {
        const unsigned __int128 q = static_cast<unsigned __int128>(1) << a.log_q;
        const unsigned __int128 p = a.plaintext_modulus;
        v = static_cast<T>(v + static_cast<T>((q + p / 2) / p)) & qm;
      }
      if (j < len) out[j] = v;
      return;
    }
    T target;
    if (kind == 1) {
      target = cl_shift_key<T>(s, a.d, shift, j);
    } else if (kind == 2) {
      // The monomial: X^shift, or -X^(shift - d) written as q - 1.
      const bool neg = shift >= a.d;
      target = j == (neg ? shift - a.d : shift) ? (neg ? qm : T{1}) : T{0};
    } else {
      target = cl_aut_key<T>(s, a.d, pinv, j);
    }
    if (digit_shift < kW) v = static_cast<T>(v + static_cast<T>(target << digit_shift)) & qm;
    out[j] = v;
  }
};

// grid = (rows, batch). Outputs: fd[b][fd_len], sd[b][2 ne][d], pk[b][2 k][d].
template <typename T, int ITERS>
__global__ void __launch_bounds__(1024)
cl_request_kernel(const T* __restrict__ a_rows, const uint32_t* __restrict__ s_hat,
                  ClientArgs a, NttCtx c, T* __restrict__ fd, T* __restrict__ sd,
                  T* __restrict__ pk) {
  extern __shared__ uint32_t cl_smem[];
  const int d = a.d;
  const int row = blockIdx.x, b = blockIdx.y;
  cl_times_key<T, ITERS>(a_rows + static_cast<int64_t>(row) * d,
                         s_hat + static_cast<int64_t>(b) * c.r * d, cl_smem, c, d);
  const ClientRow<T> out(a, row, gridDim.x, b, fd, sd, pk);
  for (int j = threadIdx.x; j < d; j += blockDim.x) out.put(a, j, cl_crt<T>(cl_smem, c, d, j));
}

// Decrypted coefficient: (a s) mod q1 rescaled to q2, plus b mod q2, then
// round(x p / q2) mod p. q2 is a power of two and x < q2, so the rounded
// quotient is a shift and at most p.
template <typename T>
__device__ __forceinline__ T cl_plain(T as, T cb, int log_q1, int log_q2,
                                      uint64_t plaintext_modulus) {
  as = rescale_word<T>(as & cl_qmask<T>(log_q1), log_q1, log_q2);
  const T v = static_cast<T>(cb + as) & cl_qmask<T>(log_q2);
  const unsigned __int128 p = plaintext_modulus;
  const unsigned __int128 x =
      (static_cast<unsigned __int128>(v) * p +
       ((static_cast<unsigned __int128>(1) << log_q2) >> 1)) >> log_q2;
  return static_cast<T>(x >= p ? x - p : x);
}

// DecryptAfterModulusSwitch per (client, shard): a s mod q1, rescaled to
// q2, + b mod q2, then round(x p / q2) mod p. grid = (l, batch).
template <typename T, int ITERS>
__global__ void __launch_bounds__(1024)
cl_decrypt_kernel(const T* __restrict__ resp, const uint32_t* __restrict__ s_hat, int l,
                  int log_q1, int log_q2, uint64_t plaintext_modulus, NttCtx c,
                  T* __restrict__ out) {
  extern __shared__ uint32_t cl_smem[];
  const int d = 1 << c.logd;
  const int k = blockIdx.x, b = blockIdx.y;
  const T* ct = resp + (static_cast<int64_t>(b) * l + k) * 2 * d;
  cl_times_key<T, ITERS>(ct, s_hat + static_cast<int64_t>(b) * c.r * d, cl_smem, c, d);
  for (int j = threadIdx.x; j < d; j += blockDim.x) {
    out[(static_cast<int64_t>(b) * l + k) * d + j] =
        cl_plain<T>(cl_crt<T>(cl_smem, c, d, j), ct[d + j], log_q1, log_q2, plaintext_modulus);
  }
}

// d = 2048..8192: the radix-16 register transforms on 27-bit primes. The
// a-components are transformed once, not once per client, and a row is one
// inverse transform per prime with the words rebuilt in registers: half of
// what is left is the error sampling (a 64-bit hash word per 64 of the 4 var
// bits, two hashes of two 64-bit products each).
//
// Transforms of the rows' a-components (blocks below rows: a_hat[row][r][d])
// and of the ternary keys (s_hat[b][r][d]). grid = (rows + batch, r).
template <typename T, int LOGD>
__global__ void __launch_bounds__(Ntt16<LOGD>::kThreads)
cl_transforms16_kernel(const T* __restrict__ a_rows, const int8_t* __restrict__ keys, int rows,
                       uint32_t* __restrict__ a_hat, uint32_t* __restrict__ s_hat, NttCtx c) {
  constexpr int d = Ntt16<LOGD>::kD;
  constexpr int NT = Ntt16<LOGD>::kThreads;
  __shared__ uint32_t xs[d];
  const int tid = threadIdx.x, pi = blockIdx.y;
  const uint32_t p = c.p[pi];
  const int row = blockIdx.x, b = row - rows;
  uint32_t x[16];
#pragma unroll
  for (int m = 0; m < 16; ++m) {
    const int j = tid + NT * m;
    if (b < 0) {
      x[m] = reduce_word(a_rows[static_cast<int64_t>(row) * d + j], c, pi);
    } else {
      const int v = keys[static_cast<int64_t>(b) * d + j];
      x[m] = v >= 0 ? static_cast<uint32_t>(v) : p - static_cast<uint32_t>(-v);
    }
  }
  ntt16_forward<LOGD, false, true, true>(x, xs, c.tables16 + static_cast<size_t>(pi) * 2 * d, p,
                                         c.one_s[pi], tid);
  uint32_t* o = (b < 0 ? a_hat + static_cast<int64_t>(row) * c.r * d
                       : s_hat + static_cast<int64_t>(b) * c.r * d) +
                static_cast<int64_t>(pi) * d;
#pragma unroll
  for (int v = 0; v < 4; ++v) {
    reinterpret_cast<uint4*>(o + 16 * tid)[v] =
        make_uint4(x[4 * v], x[4 * v + 1], x[4 * v + 2], x[4 * v + 3]);
  }
}

// cl_request_kernel from the transforms. The words go through shared memory
// (each thread's own places) so that the sampling is one loop: unrolled over
// the registers the kernel came to 140 KB of code. grid = (rows, batch), d / 16
// threads, d words of T of shared memory.
template <typename T, int LOGD>
__global__ void __launch_bounds__(Ntt16<LOGD>::kThreads, 512 / Ntt16<LOGD>::kThreads)
cl_request16_kernel(const uint32_t* __restrict__ a_hat, const uint32_t* __restrict__ s_hat,
                    const __grid_constant__ ClientArgs a, const __grid_constant__ NttCtx c,
                    const __grid_constant__ CrtArgs crt, T* __restrict__ fd,
                    T* __restrict__ sd, T* __restrict__ pk) {
  constexpr int d = Ntt16<LOGD>::kD;
  constexpr int NT = Ntt16<LOGD>::kThreads;
  extern __shared__ uint32_t cl_smem[];
  uint32_t* xs = cl_smem;
  const int tid = threadIdx.x;
  const int row = blockIdx.x, b = blockIdx.y;
  T word[16];
  uint32_t frac[16];
#pragma unroll
  for (int m = 0; m < 16; ++m) {
    word[m] = 0;
    frac[m] = 1u << 25;
  }
#pragma unroll 1
  for (int pi = 0; pi < c.r; ++pi) {
    const uint32_t p = c.p[pi], pinv = c.pinv[pi];
    const uint4* ah = reinterpret_cast<const uint4*>(
        a_hat + (static_cast<int64_t>(row) * c.r + pi) * d + 16 * tid);
    const uint4* sh = reinterpret_cast<const uint4*>(
        s_hat + (static_cast<int64_t>(b) * c.r + pi) * d + 16 * tid);
    uint32_t x[16];
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const uint4 u = __ldg(ah + v), w = __ldg(sh + v);
      x[4 * v] = mont_mul_lazy(u.x, w.x, p, pinv);
      x[4 * v + 1] = mont_mul_lazy(u.y, w.y, p, pinv);
      x[4 * v + 2] = mont_mul_lazy(u.z, w.z, p, pinv);
      x[4 * v + 3] = mont_mul_lazy(u.w, w.w, p, pinv);
    }
    ntt16_inverse<LOGD>(x, xs, c.tables16 + static_cast<size_t>(2 * pi + 1) * d, p,
                        c.one_s[pi], tid);
#pragma unroll
    for (int m = 0; m < 16; ++m) {
      const uint32_t y = shoup_mul(x[m], crt.scale[pi], crt.scale_s[pi], p);
      word[m] += static_cast<T>(y) * static_cast<T>(crt.part[pi]);
      frac[m] += __umulhi(y, crt.frac[pi]);
    }
  }
  T* words = reinterpret_cast<T*>(cl_smem);  // the exchange buffer is free
#pragma unroll
  for (int m = 0; m < 16; ++m) {
    words[tid + NT * m] =
        static_cast<T>(word[m] - static_cast<T>(frac[m] >> 26) * static_cast<T>(crt.m));
  }
  const ClientRow<T> out(a, row, gridDim.x, b, fd, sd, pk);
#pragma unroll 2
  for (int m = 0; m < 16; ++m) out.put(a, tid + NT * m, words[tid + NT * m]);
}

// cl_decrypt_kernel with two groups of d / 16 threads that take the primes in
// turns (one group at d = 8192), each transforming the key and the ciphertext's
// a itself: with a block per ciphertext the launch is a chain of transforms,
// and a launch for the keys would only lengthen it. grid = (l, batch), (r + G)
// d words of shared memory.
template <typename T, int LOGD, int G>
__global__ void __launch_bounds__(G * Ntt16<LOGD>::kThreads)
cl_decrypt16_kernel(const T* __restrict__ resp, const int8_t* __restrict__ keys, int l,
                    int log_q1, int log_q2, uint64_t plaintext_modulus,
                    const __grid_constant__ NttCtx c, const __grid_constant__ CrtArgs crt,
                    T* __restrict__ out) {
  extern __shared__ uint32_t cl_smem[];
  constexpr int d = Ntt16<LOGD>::kD;
  constexpr int NT = Ntt16<LOGD>::kThreads;
  const int grp = threadIdx.x / NT, lt = threadIdx.x & (NT - 1), bar = 1 + grp;
  uint32_t* xs = cl_smem + grp * d;
  uint32_t* ys = cl_smem + G * d;  // [r][d]
  const int k = blockIdx.x, b = blockIdx.y;
  const T* ct = resp + (static_cast<int64_t>(b) * l + k) * 2 * d;
#pragma unroll 1
  for (int pi = grp; pi < c.r; pi += G) {
    const uint32_t p = c.p[pi], pinv = c.pinv[pi];
    const uint2* tw = c.tables16 + static_cast<size_t>(pi) * 2 * d;
    uint32_t x[16], s[16];
#pragma unroll
    for (int m = 0; m < 16; ++m) {
      const int j = lt + NT * m;
      const int v = keys[static_cast<int64_t>(b) * d + j];
      s[m] = v >= 0 ? static_cast<uint32_t>(v) : p - static_cast<uint32_t>(-v);
      x[m] = reduce_word(ct[j], c, pi);
    }
    ntt16_forward<LOGD, false, true, true>(s, xs, tw, p, c.one_s[pi], lt, bar);
    ntt16_forward<LOGD, false, true>(x, xs, tw, p, c.one_s[pi], lt, bar);
#pragma unroll
    for (int m = 0; m < 16; ++m) x[m] = mont_mul_lazy(x[m], s[m], p, pinv);
    ntt16_inverse<LOGD, false, true>(x, xs, tw + d, p, c.one_s[pi], lt, bar);
#pragma unroll
    for (int m = 0; m < 16; ++m) {
      ys[pi * d + lt + NT * m] = shoup_mul(x[m], crt.scale[pi], crt.scale_s[pi], p);
    }
  }
  __syncthreads();
  T* o = out + (static_cast<int64_t>(b) * l + k) * d;
  for (int j = threadIdx.x; j < d; j += G * NT) {
    T word = 0;
    uint32_t frac = 1u << 25;
    for (int pi = 0; pi < c.r; ++pi) {
      const uint32_t y = ys[pi * d + j];
      word += static_cast<T>(y) * static_cast<T>(crt.part[pi]);
      frac += __umulhi(y, crt.frac[pi]);
    }
    word -= static_cast<T>(static_cast<T>(frac >> 26) * static_cast<T>(crt.m));
    o[j] = cl_plain<T>(word, ct[d + j], log_q1, log_q2, plaintext_modulus);
  }
}

}  // namespace inspire
