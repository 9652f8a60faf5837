// Register-blocked NTT passes in shared memory (sm_100a, CUDA cores).
//
// A transform of N = 2^lgN points is done in passes of up to L = 3 stages.
// In a pass covering stages s0 .. s0+L-1 a "group" is the 2^L points
//     x = hi * 2 t_max + q * t_min + lo,   q = 0 .. 2^L - 1,
// with t_max = N >> (s0+1), t_min = N >> (s0+L), lo < t_min, hi < 2^s0; all
// butterflies of the pass stay inside a group, so one thread loads its group
// into registers, runs the L stages there and stores it back: one shared
// memory round trip and one barrier per pass instead of per stage.
//
// Forward stages are Cooley-Tukey (natural order in, bit-reversed order out)
// with twiddle T[m + i] = w_{2m}^{brev(i)}, m = 2^s, i = x / (2t); the
// inverse runs the same butterflies backwards (Gentleman-Sande) with T^{-1}.
// Values are lazy (Harvey, "Faster arithmetic for number-theoretic
// transforms", JSC 2014): in [0, 4p) between forward stages, [0, 2p)
// between inverse stages; p < 2^30 keeps 4p below 2^32.
#pragma once

#include <cstdint>

namespace mpzmm {

// shared-memory index with one pad word per 32 (spreads power-of-two strides
// over the banks)
__device__ __forceinline__ int smi(int x) { return x + (x >> 5); }

// x * w mod p in [0, 2p) for any 32-bit x (Shoup, no final correction)
__device__ __forceinline__ uint32_t mul_shoup_lazy(uint32_t x, uint32_t w, uint32_t wq,
                                                   uint32_t p) {
  const uint32_t q = __umulhi(x, wq);
  return x * w - q * p;
}

__device__ __forceinline__ uint32_t reduce_2p(uint32_t x, uint32_t p2) {
  const uint32_t y = x - p2;
  return y < x ? y : x;  // x >= 2p ? x - 2p : x (unsigned min)
}

// Forward: L stages starting at s0 on the 2^L registers a[] of one group.
// hi is the group's high index; twiddles from tw (the prime's table).
template <int L, int LSTART = 0>
__device__ __forceinline__ void fwd_group(uint32_t (&a)[1 << L], int s0, int hi,
                                          const uint2* __restrict__ tw, uint32_t p) {
  const uint32_t p2 = 2 * p;
#pragma unroll
  for (int l = LSTART; l < L; ++l) {
    const int span = 1 << (L - 1 - l);
    const int m = 1 << (s0 + l);
#pragma unroll
    for (int q = 0; q < (1 << L); ++q) {
      if (q & span) continue;
      const int i = (hi << l) + (q >> (L - l));
      const uint2 S = __ldg(tw + m + i);
      const uint32_t U = reduce_2p(a[q], p2);
      const uint32_t V = mul_shoup_lazy(a[q + span], S.x, S.y, p);
      a[q] = U + V;
      a[q + span] = U - V + p2;
    }
  }
}

// First forward stage of a group whose upper half (points a[2^(L-1) ..])
// is zero: every butterfly's product is 0, so it only copies -- the same
// values the general butterfly gives (U and U + 2p).
template <int L>
__device__ __forceinline__ void fwd_stage0_upper_zero(uint32_t (&a)[1 << L], uint32_t p) {
  const uint32_t p2 = 2 * p;
#pragma unroll
  for (int q = 0; q < (1 << (L - 1)); ++q) {
    const uint32_t U = reduce_2p(a[q], p2);
    a[q] = U;
    a[q + (1 << (L - 1))] = U + p2;
  }
}

// Inverse: the same L stages in reverse order (Gentleman-Sande).
template <int L>
__device__ __forceinline__ void inv_group(uint32_t (&a)[1 << L], int s0, int hi,
                                          const uint2* __restrict__ tw, uint32_t p) {
  const uint32_t p2 = 2 * p;
#pragma unroll
  for (int l = L - 1; l >= 0; --l) {
    const int span = 1 << (L - 1 - l);
    const int m = 1 << (s0 + l);
#pragma unroll
    for (int q = 0; q < (1 << L); ++q) {
      if (q & span) continue;
      const int i = (hi << l) + (q >> (L - l));
      const uint2 S = __ldg(tw + m + i);
      const uint32_t X = a[q];
      const uint32_t Y = a[q + span];
      a[q] = reduce_2p(X + Y, p2);
      a[q + span] = mul_shoup_lazy(X - Y + p2, S.x, S.y, p);
    }
  }
}

// ---------------------------------------------------------------------------
// Whole transforms of a compile-time length N = 2^LGN (3 <= LGN <= 15), eight
// points a thread (or several times eight): passes of three stages from the
// top, the last one of LP = 1 to 3 on eight consecutive points.  With the
// length known every shared-memory address is a base computed once a pass
// plus immediate offsets, and a group's seven twiddles, which lie in three
// runs of the table, load as one 8-byte and three 16-byte words.
//
// Shared memory holds four pad words per 32: the strided groups of every pass
// then spread over the banks (two-way conflicts remain where LP = 1) and
// eight consecutive points stay two aligned 16-byte words.  After the pass
// from stage S the exchange stays inside blocks of N >> S points, (N >> S) / 8
// threads: up to 256 points that is one warp, and __syncwarp is enough.
// ---------------------------------------------------------------------------
__host__ __device__ constexpr int pad4(int x) { return x + ((x >> 5) << 2); }

template <int LGN>
struct NttShape {
  static constexpr int N = 1 << LGN;
  static constexpr int NG = N >> 3;                  // groups of eight points
  static constexpr int LAST = ((LGN - 1) / 3) * 3;   // first stage of the last pass
  static constexpr int LP = LGN - LAST;              // its stages
  static constexpr int WORDS = pad4(N);              // in shared memory
};

// group g of the pass from stage S0 (three stages, S0 < LAST): its first
// point's word, the offset of its point q, its high index
template <int LGN, int S0>
struct NttPass {
  static constexpr int LT = LGN - S0 - 3;  // log2 of the distance of its points
  __device__ __forceinline__ static int base(int g) {
    return pad4(((g >> LT) << (LT + 3)) + (g & ((1 << LT) - 1)));
  }
  __host__ __device__ static constexpr int off(int q) { return pad4(q << LT); }
  __device__ __forceinline__ static int high(int g) { return g >> LT; }
};

// the twiddles of a group of three stages whose first is T[b]
struct Tw8 {
  uint2 w1, w2[2], w4[4];
  __device__ __forceinline__ Tw8(const uint2* __restrict__ tw, int b) {
    w1 = __ldg(tw + b);
    const uint4 u = __ldg(reinterpret_cast<const uint4*>(tw + 2 * b));
    const uint4 v = __ldg(reinterpret_cast<const uint4*>(tw + 4 * b));
    const uint4 x = __ldg(reinterpret_cast<const uint4*>(tw + 4 * b + 2));
    w2[0] = make_uint2(u.x, u.y);
    w2[1] = make_uint2(u.z, u.w);
    w4[0] = make_uint2(v.x, v.y);
    w4[1] = make_uint2(v.z, v.w);
    w4[2] = make_uint2(x.x, x.y);
    w4[3] = make_uint2(x.z, x.w);
  }
};

__device__ __forceinline__ void bf_fwd(uint32_t& a, uint32_t& b, uint2 S, uint32_t p,
                                       uint32_t p2) {
  const uint32_t U = reduce_2p(a, p2);
  const uint32_t V = mul_shoup_lazy(b, S.x, S.y, p);
  a = U + V;
  b = U - V + p2;
}
__device__ __forceinline__ void bf_inv(uint32_t& a, uint32_t& b, uint2 S, uint32_t p,
                                       uint32_t p2) {
  const uint32_t X = a, Y = b;
  a = reduce_2p(X + Y, p2);
  b = mul_shoup_lazy(X - Y + p2, S.x, S.y, p);
}

// three forward stages
__device__ __forceinline__ void fwd8(uint32_t (&a)[8], const Tw8& t, uint32_t p) {
  const uint32_t p2 = 2 * p;
#pragma unroll
  for (int q = 0; q < 4; ++q) bf_fwd(a[q], a[q + 4], t.w1, p, p2);
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    bf_fwd(a[q], a[q + 2], t.w2[0], p, p2);
    bf_fwd(a[q + 4], a[q + 6], t.w2[1], p, p2);
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) bf_fwd(a[2 * q], a[2 * q + 1], t.w4[q], p, p2);
}
__device__ __forceinline__ void inv8(uint32_t (&a)[8], const Tw8& t, uint32_t p) {
  const uint32_t p2 = 2 * p;
#pragma unroll
  for (int q = 0; q < 4; ++q) bf_inv(a[2 * q], a[2 * q + 1], t.w4[q], p, p2);
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    bf_inv(a[q], a[q + 2], t.w2[0], p, p2);
    bf_inv(a[q + 4], a[q + 6], t.w2[1], p, p2);
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) bf_inv(a[q], a[q + 4], t.w1, p, p2);
}

// The first pass has one group shape: its twiddles are T[1 .. 7], of which
// T[1], T[2] and T[4] are 1 (the first block of every stage), so seven of its
// twelve butterflies need no product -- the forward and inverse multiply pipes
// are as busy as the issue slots.
__device__ __forceinline__ void bf_one(uint32_t& a, uint32_t& b, uint32_t p2) {
  const uint32_t U = reduce_2p(a, p2), V = reduce_2p(b, p2);
  a = U + V;
  b = U - V + p2;
}
__device__ __forceinline__ void fwd8_first(uint32_t (&a)[8], const Tw8& t, uint32_t p) {
  const uint32_t p2 = 2 * p;
#pragma unroll
  for (int q = 0; q < 4; ++q) bf_one(a[q], a[q + 4], p2);
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    bf_one(a[q], a[q + 2], p2);
    bf_fwd(a[q + 4], a[q + 6], t.w2[1], p, p2);
  }
  bf_one(a[0], a[1], p2);
#pragma unroll
  for (int q = 1; q < 4; ++q) bf_fwd(a[2 * q], a[2 * q + 1], t.w4[q], p, p2);
}
// the same where points 4 .. 7 are zero: stage 0 only copies
__device__ __forceinline__ void fwd8_first_half(uint32_t (&a)[8], const Tw8& t, uint32_t p) {
  const uint32_t p2 = 2 * p;
#pragma unroll
  for (int q = 0; q < 4; ++q) a[q] = a[q + 4] = reduce_2p(a[q], p2);
#pragma unroll
  for (int q = 0; q < 2; ++q) {  // both inputs below 2p already
    const uint32_t U = a[q], V = a[q + 2];
    a[q] = U + V;
    a[q + 2] = U - V + p2;
    const uint32_t W = mul_shoup_lazy(a[q + 6], t.w2[1].x, t.w2[1].y, p);
    a[q + 6] = a[q + 4] - W + p2;
    a[q + 4] += W;
  }
  bf_one(a[0], a[1], p2);
#pragma unroll
  for (int q = 1; q < 4; ++q) bf_fwd(a[2 * q], a[2 * q + 1], t.w4[q], p, p2);
}
__device__ __forceinline__ void inv8_first(uint32_t (&a)[8], const Tw8& t, uint32_t p) {
  const uint32_t p2 = 2 * p;
  auto one = [p2](uint32_t& x, uint32_t& y) {
    const uint32_t X = x, Y = y;
    x = reduce_2p(X + Y, p2);
    y = reduce_2p(X - Y + p2, p2);
  };
  one(a[0], a[1]);
#pragma unroll
  for (int q = 1; q < 4; ++q) bf_inv(a[2 * q], a[2 * q + 1], t.w4[q], p, p2);
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    one(a[q], a[q + 2]);
    bf_inv(a[q + 4], a[q + 6], t.w2[1], p, p2);
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) one(a[q], a[q + 4]);
}

// the last pass's LP stages on eight consecutive points 8g ..
template <int LGN>
__device__ __forceinline__ void fwd_tail(uint32_t (&a)[8], int g, const uint2* __restrict__ tw,
                                         uint32_t p) {
  constexpr int LP = NttShape<LGN>::LP, M = 1 << NttShape<LGN>::LAST;
  const uint32_t p2 = 2 * p;
  if constexpr (LP == 3) {
    fwd8(a, Tw8(tw, M + g), p);
  } else if constexpr (LP == 2) {
    const uint4 u = __ldg(reinterpret_cast<const uint4*>(tw + M + 2 * g));
    const uint4 v = __ldg(reinterpret_cast<const uint4*>(tw + 2 * M + 4 * g));
    const uint4 x = __ldg(reinterpret_cast<const uint4*>(tw + 2 * M + 4 * g + 2));
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      bf_fwd(a[q], a[q + 2], make_uint2(u.x, u.y), p, p2);
      bf_fwd(a[q + 4], a[q + 6], make_uint2(u.z, u.w), p, p2);
    }
    bf_fwd(a[0], a[1], make_uint2(v.x, v.y), p, p2);
    bf_fwd(a[2], a[3], make_uint2(v.z, v.w), p, p2);
    bf_fwd(a[4], a[5], make_uint2(x.x, x.y), p, p2);
    bf_fwd(a[6], a[7], make_uint2(x.z, x.w), p, p2);
  } else {
    const uint4 v = __ldg(reinterpret_cast<const uint4*>(tw + M + 4 * g));
    const uint4 x = __ldg(reinterpret_cast<const uint4*>(tw + M + 4 * g + 2));
    bf_fwd(a[0], a[1], make_uint2(v.x, v.y), p, p2);
    bf_fwd(a[2], a[3], make_uint2(v.z, v.w), p, p2);
    bf_fwd(a[4], a[5], make_uint2(x.x, x.y), p, p2);
    bf_fwd(a[6], a[7], make_uint2(x.z, x.w), p, p2);
  }
}
template <int LGN>
__device__ __forceinline__ void inv_tail(uint32_t (&a)[8], int g, const uint2* __restrict__ tw,
                                         uint32_t p) {
  constexpr int LP = NttShape<LGN>::LP, M = 1 << NttShape<LGN>::LAST;
  const uint32_t p2 = 2 * p;
  if constexpr (LP == 3) {
    inv8(a, Tw8(tw, M + g), p);
  } else {
    constexpr int E = LP == 2 ? 2 * M : M;  // the last stage's twiddles
    const uint4 v = __ldg(reinterpret_cast<const uint4*>(tw + E + 4 * g));
    const uint4 x = __ldg(reinterpret_cast<const uint4*>(tw + E + 4 * g + 2));
    bf_inv(a[0], a[1], make_uint2(v.x, v.y), p, p2);
    bf_inv(a[2], a[3], make_uint2(v.z, v.w), p, p2);
    bf_inv(a[4], a[5], make_uint2(x.x, x.y), p, p2);
    bf_inv(a[6], a[7], make_uint2(x.z, x.w), p, p2);
    if constexpr (LP == 2) {
      const uint4 u = __ldg(reinterpret_cast<const uint4*>(tw + M + 2 * g));
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        bf_inv(a[q], a[q + 2], make_uint2(u.x, u.y), p, p2);
        bf_inv(a[q + 4], a[q + 6], make_uint2(u.z, u.w), p, p2);
      }
    }
  }
}

template <int LGN, int S0>
__device__ __forceinline__ void load_group(const uint32_t* s, int g, uint32_t (&a)[8]) {
  const uint32_t* b = s + NttPass<LGN, S0>::base(g);
#pragma unroll
  for (int q = 0; q < 8; ++q) a[q] = b[NttPass<LGN, S0>::off(q)];
}
template <int LGN, int S0>
__device__ __forceinline__ void store_group(uint32_t* s, int g, const uint32_t (&a)[8]) {
  uint32_t* b = s + NttPass<LGN, S0>::base(g);
#pragma unroll
  for (int q = 0; q < 8; ++q) b[NttPass<LGN, S0>::off(q)] = a[q];
}
__device__ __forceinline__ void load_run(const uint32_t* s, int g, uint32_t (&a)[8]) {
  const uint4* b = reinterpret_cast<const uint4*>(s + pad4(8 * g));
  const uint4 u = b[0], v = b[1];
  a[0] = u.x; a[1] = u.y; a[2] = u.z; a[3] = u.w;
  a[4] = v.x; a[5] = v.y; a[6] = v.z; a[7] = v.w;
}
__device__ __forceinline__ void store_run(uint32_t* s, int g, const uint32_t (&a)[8]) {
  uint4* b = reinterpret_cast<uint4*>(s + pad4(8 * g));
  b[0] = make_uint4(a[0], a[1], a[2], a[3]);
  b[1] = make_uint4(a[4], a[5], a[6], a[7]);
}

// groups tt, tt + TS, .. of a transform (just tt where there are TS)
template <int LGN, int TS, class F>
__device__ __forceinline__ void each_group(int tt, F f) {
  if constexpr (NttShape<LGN>::NG <= TS) {
    f(tt);
  } else {
#pragma unroll 1
    for (int g = tt; g < NttShape<LGN>::NG; g += TS) f(g);
  }
}

// the barrier after (forward) or before (inverse) the exchange of the pass
// from stage S0
template <int LGN, int S0>
__device__ __forceinline__ void pass_sync() {
  if constexpr (((1 << LGN) >> S0) / 8 > 32)
    __syncthreads();
  else
    __syncwarp();
}

// Forward passes S0 .. LAST - 3 of `count` transforms (words WORDS apart,
// primes j, j + 1, ..) by threads tt, tt + TS, ..: the groups of the first
// pass are in shared memory and synchronised.
template <int LGN, int S0, int TS, class Tables>
__device__ __forceinline__ void fwd_middle(uint32_t* s, int count, int j, int tt,
                                           const Tables& tables) {
  if constexpr (S0 < NttShape<LGN>::LAST) {
    for (int c = 0; c < count; ++c) {
      const uint32_t p = tables.p(j + c);
      const uint2* tw = tables.tw(j + c);
      uint32_t* sc = s + c * NttShape<LGN>::WORDS;
      each_group<LGN, TS>(tt, [&](int g) {
        uint32_t a[8];
        load_group<LGN, S0>(sc, g, a);
        fwd8(a, Tw8(tw, (1 << S0) + NttPass<LGN, S0>::high(g)), p);
        store_group<LGN, S0>(sc, g, a);
      });
    }
    pass_sync<LGN, S0>();
    fwd_middle<LGN, S0 + 3, TS>(s, count, j, tt, tables);
  }
}
// Inverse passes S0 .. 3 (downwards) of one transform; the last pass's
// results are in shared memory, not yet synchronised.
template <int LGN, int S0, int TS, class Tables>
__device__ __forceinline__ void inv_middle(uint32_t* s, int j, int tt, const Tables& tables) {
  pass_sync<LGN, S0>();
  if constexpr (S0 >= 3) {
    const uint32_t p = tables.p(j);
    const uint2* tw = tables.tw(j);
    each_group<LGN, TS>(tt, [&](int g) {
      uint32_t a[8];
      load_group<LGN, S0>(s, g, a);
      inv8(a, Tw8(tw, (1 << S0) + NttPass<LGN, S0>::high(g)), p);
      store_group<LGN, S0>(s, g, a);
    });
    inv_middle<LGN, S0 - 3, TS>(s, j, tt, tables);
  }
}

}  // namespace mpzmm
