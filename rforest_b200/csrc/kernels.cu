// sm_100a kernels of the exact matrix-product pipeline.
//
//   k_fwd_team, k_fwd_cta
//                    limbs -> r-bit coefficients -> 30-bit digits ->
//                    residues mod p -> forward NTT, register-blocked passes
//                    (several small transforms or one large one per CTA)
//   k_split_fwd      the same, radix 2, one CTA per (entry, prime): tiny
//                    transforms (2^2 points)
//   k_contract       per frequency h and prime: C[h] = A[h] B[h] mod p on
//                    CUDA cores (64-bit lazy accumulation, Montgomery fold)
//   k_contract_tc    the same on tensor cores (tcgen05 kind::i8, exact
//                    byte split; contract_tc.cuh)
//   k_inv_team, k_inv_cta
//                    inverse NTT, register-blocked; k_inv_ntt radix 2
//   k_crt_mixed      explicit CRT to signed multi-word coefficients, then
//                    sum_i c_i 2^(i r) with carries resolved by a
//                    carry-lookahead prefix scan over 32-bit output words,
//                    sign + negation + normalisation (one warp per entry
//                    or, of few long entries, per segment; every prime
//                    count of a range in one launch); k_crt_finish closes
//                    the entries in segments
//
// Reference counterparts: split/reduce src/lib/split_reduce.c:15-66,
// NTTs src/lib/mpnfft.c:354-432, contraction src/lib/mpnfft.c:559-651,
// CRT src/lib/crt.c:11-94, recompose src/lib/recompose.c:11-107 and
// src/lib/crt_recompose.c:15-156, sign/normalise src/lib/hwmpz.c:116-122.

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstdlib>
#include <vector>

#include "kernels.h"
#include "modarith.cuh"
#include "mpzmm_internal.h"
#include "ntt_fast.cuh"
#include "contract_tc.cuh"

namespace mpzmm {

__constant__ PrimeConst c_primes[kMaxPrimes];
__constant__ CrtConst c_crt;

constexpr int kTwStride = 1 << kTwiddleLg;  // twiddle entries per prime

// The stages of a single product follow one another as small grids, so each
// lets the next one's blocks come up while it runs and waits for its
// predecessor's results here (no effect unless the launch asks for it:
// launch_next).  5 x 7 x 3 of 20011 bits on device buffers 31.7 us, 40.2 with
// each launch after the end of the one in front; a chain of 15 products 3.00
// ms, 3.10.
__device__ __forceinline__ void stage_begin() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// A load of what the kernel in front writes, in a kernel that starts with
// stage_begin(): its grid may live while the writer does, and the read-only
// path (__ldg, const __restrict__) is defined only for memory that nothing
// writes as long as the grid lives.  The wait orders ordinary loads.
template <class T>
__device__ __forceinline__ T stage_load(const T* p) {
  return __ldca(p);
}

// A launch that may come up before the kernel in front of it in the stream
// has ended; the kernel must start with stage_begin().
template <class... P, class... A>
static cudaError_t launch_next(void (*kernel)(P...), int grid, int threads, size_t smem,
                               cudaStream_t st, A... args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = dim3((unsigned)grid);
  c.blockDim = dim3((unsigned)threads);
  c.dynamicSmemBytes = smem;
  c.stream = st;
  c.attrs = &at;
  c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
}

// ---------------------------------------------------------------------------
// NTT building blocks (shared memory, radix-2)
//
// Forward (Cooley-Tukey, natural order in, bit-reversed order out): for
// m = 1, 2, ..., N/2 and t = N/(2m), block i of 2t values is split with the
// twiddle T[m + i] = w_{2m}^{brev(i)}, a primitive-root power that does not
// depend on N, so one table of 2^kTwiddleLg entries per prime serves every N.
// Inverse (Gentleman-Sande) runs the same (m, i) pairs in reverse order with
// T^{-1}; it returns N times the input, the factor is removed before CRT.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void ntt_fwd_smem(uint32_t* a, int lgN, const uint2* tw,
                                             uint32_t p) {
  const int half = 1 << (lgN - 1);
  for (int lgm = 0; lgm < lgN; ++lgm) {
    const int lgt = lgN - 1 - lgm;
    const int t = 1 << lgt;
    const int m = 1 << lgm;
    for (int b = threadIdx.x; b < half; b += blockDim.x) {
      const int i = b >> lgt;
      const int j = (i << (lgt + 1)) + (b & (t - 1));
      const uint2 S = tw[m + i];
      const uint32_t U = a[j];
      const uint32_t V = mul_shoup(a[j + t], S.x, S.y, p);
      a[j] = add_mod(U, V, p);
      a[j + t] = sub_mod(U, V, p);
    }
    __syncthreads();
  }
}

__device__ __forceinline__ void ntt_inv_smem(uint32_t* a, int lgN, const uint2* tw,
                                             uint32_t p) {
  const int half = 1 << (lgN - 1);
  for (int lgm = lgN - 1; lgm >= 0; --lgm) {
    const int lgt = lgN - 1 - lgm;
    const int t = 1 << lgt;
    const int m = 1 << lgm;
    for (int b = threadIdx.x; b < half; b += blockDim.x) {
      const int i = b >> lgt;
      const int j = (i << (lgt + 1)) + (b & (t - 1));
      const uint2 S = tw[m + i];
      const uint32_t X = a[j];
      const uint32_t Y = a[j + t];
      a[j] = add_mod(X, Y, p);
      a[j + t] = mul_shoup(sub_mod(X, Y, p), S.x, S.y, p);
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Split + reduce + forward NTT.  grid = (entries of this class, P).
// Coefficient i of an entry is bits [i r, (i+1) r) of its magnitude; its
// residue is taken by Horner over 32-bit words (Shoup multiply by 2^32 mod p)
// and negated for a negative entry, which is how the reference folds the
// sign into the split (src/lib/split_reduce.c:27-38).
// ---------------------------------------------------------------------------
__global__ void k_split_fwd(const FwdDesc* __restrict__ descs,
                            const uint32_t* __restrict__ idx,
                            const uint64_t* __restrict__ limbs,
                            uint32_t* __restrict__ res,
                            const uint2* __restrict__ twf) {
  extern __shared__ uint32_t sm[];
  const FwdDesc d = descs[idx ? idx[blockIdx.x] : blockIdx.x];
  const int j = blockIdx.y;
  const uint32_t p = c_primes[j].p;
  const uint32_t mu = c_primes[j].mu;
  const uint32_t b32 = c_primes[j].b32;
  const uint32_t b32q = c_primes[j].b32q;
  const int N = 1 << d.lgN;
  const uint32_t nl = (uint32_t)(d.size < 0 ? -d.size : d.size);
  const uint32_t nw = 2 * nl;
  const uint32_t* __restrict__ w32 = reinterpret_cast<const uint32_t*>(limbs + d.limb_off);
  const uint32_t r = d.r;
  const int ncw = (int)((r + 31) >> 5);
  const uint32_t topbits = r - 32u * (uint32_t)(ncw - 1);
  const uint32_t topmask = topbits >= 32 ? 0xffffffffu : ((1u << topbits) - 1u);
  const bool neg = d.size < 0;

  for (int i = threadIdx.x; i < N; i += blockDim.x) {
    uint32_t v = 0;
    if ((uint32_t)i < d.ncoef) {
      const uint64_t bit = (uint64_t)i * r;
      const uint64_t wi = bit >> 5;
      const uint32_t sh = (uint32_t)(bit & 31);
      uint32_t acc = 0;
      for (int q = ncw - 1; q >= 0; --q) {
        const uint64_t a0 = wi + (uint64_t)q;
        const uint32_t lo = a0 < nw ? w32[a0] : 0u;
        const uint32_t hi = a0 + 1 < nw ? w32[a0 + 1] : 0u;
        uint32_t c = __funnelshift_r(lo, hi, sh);
        if (q == ncw - 1) c &= topmask;
        acc = add_mod(mul_shoup(acc, b32, b32q, p), mod32(c, p, mu), p);
      }
      v = (neg && acc) ? p - acc : acc;
    }
    sm[i] = v;
  }
  __syncthreads();
  ntt_fwd_smem(sm, d.lgN, twf + (size_t)j * kTwStride, p);
  uint32_t* out = res + d.res_off + (uint64_t)j * (uint64_t)N;
  for (int i = threadIdx.x; i < N; i += blockDim.x) out[i] = sm[i];
}

// ---------------------------------------------------------------------------
// Inverse NTT.  grid = (entries of this class, P).
// ---------------------------------------------------------------------------
__global__ void k_inv_ntt(const InvDesc* __restrict__ descs,
                          const uint32_t* __restrict__ idx, uint32_t* __restrict__ res,
                          const uint2* __restrict__ twi) {
  extern __shared__ uint32_t sm[];
  const InvDesc d = descs[idx ? idx[blockIdx.x] : blockIdx.x];
  const int j = blockIdx.y;
  const uint32_t p = c_primes[j].p;
  const int N = 1 << d.lgN;
  uint32_t* io = res + d.res_off + (uint64_t)j * (uint64_t)N;
  // the contraction leaves values in [0, 2p); these butterflies want [0, p)
  for (int i = threadIdx.x; i < N; i += blockDim.x) sm[i] = min(io[i], io[i] - p);
  __syncthreads();
  ntt_inv_smem(sm, d.lgN, twi + (size_t)j * kTwStride, p);
  for (int i = threadIdx.x; i < N; i += blockDim.x) io[i] = sm[i];
}

// ---------------------------------------------------------------------------
// Contraction on CUDA cores.  One thread per residue position x of a
// polynomial (prime x >> lgN, frequency x mod N: the primes' residues follow
// one another, so a block takes 128 positions whatever the transform's
// length); it walks its share of the m x n outputs in register tiles of
// TI x TJ (1 to 4 each, chosen per product and stored in ProdDesc::pad),
// loading TI + TJ residues per TI * TJ products.
// Edge tiles clamp their row/column to the last one (in-bounds duplicate
// work, results discarded).  Products of residues < p < 2^30 are at most
// 2^60 - 2^31, so sixteen of them accumulate exactly in 64 bits (the
// reference reduces every 16 terms for the same reason with 128-bit
// accumulators, src/lib/mpnfft.c:621-627); then the high word is folded down
// and twelve more fit.  Outputs carry a factor 2^-32 that the CRT stage
// removes.
// The tiles of a block of positions are split over several CTAs where whole
// ones would not fill the GPU: a 2000 x 1 by 1 x 1 product of 10^4-bit
// integers (1408 positions) took 295 us in 11 CTAs, 16 split.
// Bound by its loads (operands straight from L2, DRAM at about 40 % of its
// rate): up to four terms' loads go out together, and 80 registers leave
// six CTAs an SM.  1314 us for the first 512 products of the default batch,
// 1400 before the terms past a multiple of four were loaded together and
// the folds cut to one multiply-add; 1360 at 128 registers, 1470 at 64.
// Staging a block's operands in shared memory (cp.async, two buffers)
// measured 1850: too little work a CTA for its two waits.
// ---------------------------------------------------------------------------
constexpr int kContractThreads = 128;

constexpr int kContractFirst = 16;  // products a fresh accumulator holds
constexpr int kContractMore = 12;   // further ones after a fold

// The high word folded down: lo + hi (2^32 mod p), below 2^62 + 2^32.
__device__ __forceinline__ uint64_t fold64(uint64_t x, uint32_t b32) {
  return (uint64_t)(uint32_t)(x >> 32) * b32 + (uint32_t)x;
}

// R terms (1 to 4) of a tile, their loads issued together.
template <int TI, int TJ, int R>
__device__ __forceinline__ void contract_terms(uint64_t (&acc)[TI][TJ],
                                               const uint32_t* A, const uint32_t* B,
                                               const uint32_t (&ao)[TI], const uint32_t (&bo)[TJ],
                                               uint32_t stride, uint32_t bstep, uint32_t b32,
                                               int& room) {
  uint32_t av[R][TI], bv[R][TJ];
#pragma unroll
  for (int u = 0; u < R; ++u) {
#pragma unroll
    for (int x = 0; x < TI; ++x) av[u][x] = stage_load(A + ao[x] + (uint32_t)u * stride);
#pragma unroll
    for (int y = 0; y < TJ; ++y) bv[u][y] = stage_load(B + bo[y] + (uint32_t)u * bstep);
  }
  if (room < R) {
#pragma unroll
    for (int x = 0; x < TI; ++x)
#pragma unroll
      for (int y = 0; y < TJ; ++y) acc[x][y] = fold64(acc[x][y], b32);
    room = kContractMore;
  }
  room -= R;
#pragma unroll
  for (int u = 0; u < R; ++u)
#pragma unroll
    for (int x = 0; x < TI; ++x)
#pragma unroll
      for (int y = 0; y < TJ; ++y) acc[x][y] += (uint64_t)av[u][x] * bv[u][y];
}

template <int TI, int TJ>
__device__ __forceinline__ void contract_tiles(const ProdDesc& d, const ContractItem& it,
                                               uint32_t pos, uint32_t* __restrict__ res) {
  const int j = (int)(pos >> d.lgN);
  const uint32_t p = c_primes[j].p;
  const uint32_t pinv = c_primes[j].pinv;
  const uint32_t b32 = c_primes[j].b32;
  const uint32_t stride = (uint32_t)d.P << d.lgN;  // words between polynomials
  const uint32_t* A = res + d.a_res + pos;
  const uint32_t* B = res + d.b_res + pos;
  uint32_t* C = res + d.c_res + pos;
  const int m = d.m, k = d.k, n = d.n;
  const uint32_t bstep = (uint32_t)n * stride;
  const uint32_t tn = (uint32_t)(n + TJ - 1) / TJ;  // tiles of a row of them
  int i0 = (int)(it.t0 / tn) * TI, l0 = (int)(it.t0 % tn) * TJ;
  for (uint32_t t = 0; t < it.nt; ++t) {
    uint32_t ao[TI], bo[TJ];  // word offsets of the tile's rows / columns
#pragma unroll
    for (int x = 0; x < TI; ++x) {
      const int ii = (i0 + x) < m ? (i0 + x) : (m - 1);
      ao[x] = (uint32_t)ii * (uint32_t)k * stride;
    }
#pragma unroll
    for (int y = 0; y < TJ; ++y) {
      const int ll = (l0 + y) < n ? (l0 + y) : (n - 1);
      bo[y] = (uint32_t)ll * stride;
    }
    uint64_t acc[TI][TJ];
#pragma unroll
    for (int x = 0; x < TI; ++x)
#pragma unroll
      for (int y = 0; y < TJ; ++y) acc[x][y] = 0;
    int room = kContractFirst;
    const uint32_t* Aq = A;
    const uint32_t* Bq = B;
    for (int q = k; q >= 4; q -= 4) {
      contract_terms<TI, TJ, 4>(acc, Aq, Bq, ao, bo, stride, bstep, b32, room);
      Aq += 4 * (uint64_t)stride;
      Bq += 4 * (uint64_t)bstep;
    }
    switch (k & 3) {
      case 3: contract_terms<TI, TJ, 3>(acc, Aq, Bq, ao, bo, stride, bstep, b32, room); break;
      case 2: contract_terms<TI, TJ, 2>(acc, Aq, Bq, ao, bo, stride, bstep, b32, room); break;
      case 1: contract_terms<TI, TJ, 1>(acc, Aq, Bq, ao, bo, stride, bstep, b32, room); break;
    }
#pragma unroll
    for (int x = 0; x < TI; ++x) {
      if (i0 + x >= m) continue;
#pragma unroll
      for (int y = 0; y < TJ; ++y) {
        if (l0 + y >= n) continue;
        // the value times 2^-32 (the Montgomery factor the CRT removes), in
        // [0, 2p): the fold leaves T < 2^62 + 2^32, its REDC is at most
        // p + 2^30 + 1, and p is above 2^29
        const uint64_t T = fold64(acc[x][y], b32);
        const uint32_t v = (uint32_t)((T + (uint64_t)((uint32_t)T * pinv) * p) >> 32);
        C[(uint32_t)((i0 + x) * n + (l0 + y)) * stride] = min(v, v - p);
      }
    }
    l0 += TJ;
    if (l0 >= n) {
      l0 = 0;
      i0 += TI;
    }
  }
}

// items == nullptr: product 0 alone, its blocks of positions and groups of
// u.per tiles in grid order
__global__ void __launch_bounds__(kContractThreads, 6)
k_contract(const ProdDesc* __restrict__ prods, const ContractItem* __restrict__ items,
           ContractUniform u, uint32_t* __restrict__ res) {
  stage_begin();
  ContractItem it;
  if (items) {
    it = items[blockIdx.x];
  } else {
    const uint32_t g = blockIdx.x / u.blocks;
    it.prod = 0;
    it.x0 = (blockIdx.x - g * u.blocks) * (uint32_t)kContractThreads;
    it.t0 = g * u.per;
    it.nt = min(u.per, u.tiles - it.t0);
  }
  const ProdDesc d = prods[it.prod];
  const uint32_t pos = it.x0 + threadIdx.x;
  if (pos >= ((uint32_t)d.P << d.lgN)) return;
  switch (d.pad) {  // tile shape 4 (TI - 1) + (TJ - 1), uniform over the CTA
#define MPZMM_TILE(TI, TJ) \
  case 4 * (TI - 1) + (TJ - 1): contract_tiles<TI, TJ>(d, it, pos, res); break;
    MPZMM_TILE(4, 4) MPZMM_TILE(4, 3) MPZMM_TILE(4, 2) MPZMM_TILE(4, 1)
    MPZMM_TILE(3, 4) MPZMM_TILE(3, 3) MPZMM_TILE(3, 2) MPZMM_TILE(3, 1)
    MPZMM_TILE(2, 4) MPZMM_TILE(2, 3) MPZMM_TILE(2, 2) MPZMM_TILE(2, 1)
    MPZMM_TILE(1, 4) MPZMM_TILE(1, 3) MPZMM_TILE(1, 2) MPZMM_TILE(1, 1)
#undef MPZMM_TILE
  }
}

// ---------------------------------------------------------------------------
// CRT + recompose + sign + normalise: shared pieces.
//
// Coefficient i of an output entry is recovered as the symmetric residue
// X_i in (-M/4, M/4), M = p_0...p_{P-1}, written as X_i = U_i - s_i 2^(32P)
// with U_i the P-word two's complement and s_i its sign bit.  The entry is
// sum_i X_i 2^(i r) mod 2^(32 W).  Output word w gathers its local sum
//      s_w = sum_i slice_w(U_i 2^(i r)) - sum_i s_i [borrow of i lands in w]
// (a small signed 64-bit value), then s_w = lo_w + 2^32 hi_w is rewritten as
// words y_w with carries g_w in {-1,0,1}; the remaining carry ripple is a
// prefix scan whose element is the word's transfer function
// {-1,0,1} -> {-1,0,1}, composed associatively.  This is the parallel form
// of the reference's serial borrow chain (src/lib/recompose.c:43-87) and of
// its chunk fix-up (src/lib/crt_recompose.c:101-153); the reference's CRT is
// Garner's (src/lib/crt.c:11-94), the explicit form here needs O(P) modular
// products instead of O(P^2).
// ---------------------------------------------------------------------------

__device__ __forceinline__ int apply_tf(uint32_t f, int c) {
  return (int)((f >> (2 * (c + 1))) & 3u) - 1;
}
// g after f
__device__ __forceinline__ uint32_t compose_tf(uint32_t g, uint32_t f) {
  uint32_t out = 0;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const uint32_t fc = (f >> (2 * c)) & 3u;
    out |= ((g >> (2 * fc)) & 3u) << (2 * c);
  }
  return out;
}
constexpr uint32_t kTfIdentity = (0u) | (1u << 2) | (2u << 4);

__device__ __forceinline__ uint32_t word_tf(uint32_t y, int g) {
  uint32_t f = 0;
#pragma unroll
  for (int c = -1; c <= 1; ++c) {
    int delta = 0;
    if (c == 1 && y == 0xffffffffu) delta = 1;
    if (c == -1 && y == 0u) delta = -1;
    f |= (uint32_t)(g + delta + 1) << (2 * (c + 1));
  }
  return f;
}

// ---------------------------------------------------------------------------
// Split + forward NTT, register-blocked (lgN >= 3, ntt_fast.cuh).
//
// Team CTAs (N <= 2048): 256 threads, 2048 / N entries; a team of N / 8
// threads owns one entry and each thread the 8 points x = q N/8 + t of the
// first pass, whose 30-bit coefficient digits it extracts once and keeps in
// registers for all its primes.  A residue is
//     c mod p = REDC( sum_q d_q * (2^(30 q + 32) mod p) )
// (D products of 30-bit by 30-bit numbers, exact in 64 bits for D <= 8), so
// each prime costs D wide multiply-adds and one Montgomery reduction instead
// of a Horner chain.  Larger transforms take a whole CTA of 512 or 1024
// threads, which extracts a coefficient's digits once for cta_primes() primes
// whose transforms sit in shared memory together.
//
// Bound by integer issue: about 58 instructions a residue (2^9 .. 2^11
// points, 5 digits), the multiply pipe as busy as the issue slots.  With the
// length a template parameter (addresses and twiddle runs, ntt_fast.cuh),
// exchanges inside a warp past the first pass and two buffers, a team has one
// barrier a prime; 64 registers leave four CTAs an SM.  The first 512
// products of the default batch: 1937 us, 2675 with lengths at run time, a
// barrier a pass and three CTAs an SM (86 instructions a residue); 1980 at
// 80 registers.  Few CTAs are cut by primes (prime_chunks): 4 x 4 of
// 4096-bit entries 10.8 us, 19 with all nine primes in one CTA.
// ---------------------------------------------------------------------------
constexpr int kFwdThreads = 256;
constexpr int kTeamWords = pad4(8 * kFwdThreads);  // one buffer of a team CTA

// Digits of the coefficient starting at bit bit0 (r bits of the entry's nw
// 32-bit words; bits past the entry read as 0).  Bit positions fit 32 bits:
// a transform has at most 2^15 coefficients of at most 210 bits.
template <int D>
__device__ __forceinline__ void coeff_digits(const uint32_t* __restrict__ w32, uint32_t nw,
                                             uint32_t bit0, uint32_t r, bool live,
                                             uint32_t (&dg)[D]) {
  // every word the D digits touch lies inside the entry (the usual case)
  const bool inside = live && ((bit0 + 30u * (D - 1)) >> 5) + 2u <= nw;
#pragma unroll
  for (int q = 0; q < D; ++q) {
    const uint32_t b = bit0 + 30u * q;
    const uint32_t wi = b >> 5;
    uint32_t lo, hi;
    if (inside) {
      lo = __ldg(w32 + wi);
      hi = __ldg(w32 + wi + 1);
    } else {
      lo = (live && wi < nw) ? __ldg(w32 + wi) : 0u;
      hi = (live && wi + 1 < nw) ? __ldg(w32 + wi + 1) : 0u;
    }
    uint32_t v = __funnelshift_r(lo, hi, b & 31u) & 0x3fffffffu;
    const int rem = (int)r - 30 * q;  // bits of the coefficient left for this digit
    if (rem < 30) v = rem <= 0 ? 0u : (v & ((1u << rem) - 1u));
    dg[q] = v;
  }
}

// The residue of a coefficient from its digits, lazily reduced: the REDC
// of S = sum_q d_q (2^(30q+32) mod p) < D 2^30 p is below (D/4 + 1) p < 3p
// for D <= 7, and a negative entry's residue is taken as 3p - v, in (0, 3p]:
// both below 4p, the forward transform's input range.
template <int D>
__device__ __forceinline__ uint32_t digits_residue(const uint32_t (&dg)[D], int j, bool neg) {
  const uint32_t p = c_primes[j].p;
  uint64_t S = 0;
#pragma unroll
  for (int q = 0; q < D; ++q) S += (uint64_t)dg[q] * c_primes[j].dig[q];
  const uint32_t m = (uint32_t)S * c_primes[j].pinv;
  const uint32_t v = (uint32_t)((S + (uint64_t)m * p) >> 32);
  return neg ? 3u * p - v : v;
}

// Where the forward transform leaves eight points 8 g .. of prime j of an
// entry: the plain frequency-contiguous layout (base + j N + 8 g), or, for an
// operand of a tensor-core product, blocked by kTcTile = 8 frequencies (a
// 32-byte sector) across the operand's np entries (base + ((j N / 8 + g) np +
// e) 8).  Either way run number j N / 8 + g times one stride.
struct FwdOut {
  uint32_t* base;
  uint32_t stride;
  __device__ __forceinline__ FwdOut(uint32_t* res, const FwdDesc& d)
      : base(res + d.res_off + kTcTile * (uint64_t)d.tile_e),
        stride(d.tile_np ? kTcTile * d.tile_np : kTcTile) {}
  // reduced from [0, 4p) to [0, p), vector stores
  __device__ __forceinline__ void store(uint32_t run, uint32_t (&a)[8], uint32_t p) const {
    static_assert(kTcTile == 8, "a run is one block");
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const uint32_t v = reduce_2p(a[q], 2 * p);
      a[q] = min(v, v - p);
    }
    uint4* o = reinterpret_cast<uint4*>(base + (uint64_t)run * stride);
    o[0] = make_uint4(a[0], a[1], a[2], a[3]);
    o[1] = make_uint4(a[4], a[5], a[6], a[7]);
  }
};

struct NttTables {
  const uint2* t;
  __device__ __forceinline__ uint32_t p(int j) const { return c_primes[j].p; }
  __device__ __forceinline__ const uint2* tw(int j) const { return t + (size_t)j * kTwStride; }
};

// One entry's coefficients in shared use by the first pass: HZ (at most N/2
// of them, the usual case: both factors of a product fit in N together): the
// upper four points of every group are zero, so their digits and residues
// are skipped and stage 0 only copies.
struct Coeffs {
  const uint32_t* w32;
  uint32_t nw, r, ncoef;
  bool neg;
  __device__ __forceinline__ Coeffs(const FwdDesc& d, const uint64_t* __restrict__ limbs) {
    const uint32_t nl = (uint32_t)(d.size < 0 ? -d.size : d.size);
    nw = nl < 0x40000000u ? 2u * nl : 0x80000000u;
    w32 = reinterpret_cast<const uint32_t*>(limbs + d.limb_off);
    r = d.r;
    ncoef = d.ncoef;
    neg = d.size < 0;
  }
  template <int D>
  __device__ __forceinline__ void digits(int x, uint32_t (&dg)[D]) const {
    coeff_digits<D>(w32, nw, (uint32_t)x * r, r, (uint32_t)x < ncoef, dg);
  }
};

// The same value, computed anew as far as the compiler knows: the addresses
// that follow from it are worth an instruction or two a prime, not a
// register each across the loop over the primes.
__device__ __forceinline__ int fresh(int x) {
  asm volatile("" : "+r"(x));
  return x;
}

// The coefficients of a first-pass group: their digits held in registers for
// all primes (HZ), or extracted again for every prime (long operands: eight
// points' digits are too many registers).
template <int LGN, int D, bool HZ>
struct FirstGroup {
  uint32_t dg[HZ ? 4 : 1][D];
  __device__ __forceinline__ FirstGroup(const Coeffs& co, int g) {
    if (HZ) {
#pragma unroll
      for (int q = 0; q < 4; ++q) co.digits<D>(q * NttShape<LGN>::NG + g, dg[q]);
    }
  }
  // the group's residues mod prime j through the first pass
  __device__ __forceinline__ void run(const Coeffs& co, int g, int j,
                                      const uint2* __restrict__ tw, uint32_t (&a)[8]) {
    const uint32_t p = c_primes[j].p;
    if (HZ) {
#pragma unroll
      for (int q = 0; q < 4; ++q) a[q] = digits_residue<D>(dg[q], j, co.neg);
    } else {
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        co.digits<D>(q * NttShape<LGN>::NG + g, dg[0]);
        a[q] = digits_residue<D>(dg[0], j, co.neg);
      }
    }
    if (HZ)
      fwd8_first_half(a, Tw8(tw, 1), p);
    else
      fwd8_first(a, Tw8(tw, 1), p);
  }
};

template <int LGN, int D, bool HZ>
__device__ __forceinline__ void fwd_team(const FwdDesc& d, bool valid, uint32_t* sm, int team,
                                         int tt, int j0, int j1,
                                         const uint64_t* __restrict__ limbs,
                                         uint32_t* __restrict__ res, NttTables tables) {
  using S = NttShape<LGN>;
  const Coeffs co(d, limbs);
  const FwdOut out(res, d);
  FirstGroup<LGN, D, HZ> first(co, tt);
#pragma unroll 1
  for (int j = j0; j < j1; ++j) {
    tt = fresh(tt);
    const uint32_t p = c_primes[j].p;
    const uint2* tw = tables.tw(j);
    // primes alternate between two buffers: a buffer is written again only
    // after the next prime's barrier, past every thread's last read of it
    uint32_t* s = sm + pad4(team << LGN) + (j & 1) * kTeamWords;
    uint32_t a[8];
    first.run(co, tt, j, tw, a);
    if constexpr (S::LAST > 0) {
      store_group<LGN, 0>(s, tt, a);
      pass_sync<LGN, 0>();
      fwd_middle<LGN, 3, S::NG>(s, 1, j, tt, tables);
      load_run(s, tt, a);
      fwd_tail<LGN>(a, tt, tw, p);
    }
    if (valid) out.store((uint32_t)(j * S::NG + tt), a, p);
  }
}

// the entry of a team or CTA: items == nullptr: entries 0, 1, .. all alike (u)
__device__ __forceinline__ CtaItem cta_item(const CtaItem* __restrict__ items,
                                            const CtaUniform& u) {
  if (items) return items[blockIdx.x];
  CtaItem it;
  const uint32_t g = blockIdx.x / u.chunks, c = blockIdx.x - g * u.chunks;
  it.first = g * u.per;
  it.count = (uint16_t)min(u.per, u.total - it.first);
  it.lgN = (uint8_t)u.lgN;
  it.j0 = (uint8_t)(u.P * c / u.chunks);
  it.j1 = (uint8_t)(u.P * (c + 1) / u.chunks);
  return it;
}

#define MPZMM_TEAM_SIZES(X) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(11)

template <int D>
__global__ void __launch_bounds__(kFwdThreads, 4)
k_fwd_team(const FwdDesc* __restrict__ descs, const uint32_t* __restrict__ idx,
           const CtaItem* __restrict__ items, CtaUniform u, const uint64_t* __restrict__ limbs,
           uint32_t* __restrict__ res, const uint2* __restrict__ twf) {
  stage_begin();
  __shared__ __align__(16) uint32_t buf[2 * kTeamWords];
  const CtaItem item = cta_item(items, u);
  const int lgN = item.lgN;
  const int team = (int)threadIdx.x >> (lgN - 3);
  const int tt = (int)threadIdx.x & ((1 << (lgN - 3)) - 1);
  const bool valid = team < (int)item.count;
  FwdDesc d{};
  d.r = 1;
  if (valid) d = descs[idx ? idx[item.first + team] : item.first + team];
  // one form for the whole CTA (its barriers must be the same code)
  const bool hz = __syncthreads_and(d.ncoef <= (1u << lgN >> 1));
  switch (lgN) {
#define MPZMM_CASE(L)                                                                         \
  case L:                                                                                     \
    if (hz)                                                                                   \
      fwd_team<L, D, true>(d, valid, buf, team, tt, item.j0, item.j1, limbs, res,             \
                           NttTables{twf});                                                   \
    else                                                                                      \
      fwd_team<L, D, false>(d, valid, buf, team, tt, item.j0, item.j1, limbs, res,            \
                            NttTables{twf});                                                  \
    break;
    MPZMM_TEAM_SIZES(MPZMM_CASE)
#undef MPZMM_CASE
  }
}

// Whole-CTA transforms: threads, and primes whose transforms share the
// shared memory (their coefficients' digits are extracted once for all).
__host__ __device__ constexpr int cta_threads(int lgN) { return lgN <= 12 ? 512 : 1024; }
__host__ __device__ constexpr int cta_primes(int lgN) {
  return lgN <= 13 ? 5 : (lgN == 14 ? 3 : 1);
}

// the first pass of primes jb .. jb + nb - 1, into their buffers
template <int LGN, int D, bool HZ>
__device__ __forceinline__ void fwd_cta_first(const Coeffs& co, uint32_t* sm, int jb, int nb,
                                              NttTables tables) {
  each_group<LGN, cta_threads(LGN)>((int)threadIdx.x, [&](int g) {
    FirstGroup<LGN, D, HZ> first(co, g);
#pragma unroll 1
    for (int c = 0; c < nb; ++c) {
      const int gc = fresh(g);
      uint32_t a[8];
      first.run(co, gc, jb + c, tables.tw(jb + c), a);
      store_group<LGN, 0>(sm + c * NttShape<LGN>::WORDS, gc, a);
    }
  });
}

template <int LGN, int D>
__global__ void __launch_bounds__(cta_threads(LGN), 1024 / cta_threads(LGN))
k_fwd_cta(const FwdDesc* __restrict__ descs, const uint32_t* __restrict__ idx,
          const CtaItem* __restrict__ items, CtaUniform u, const uint64_t* __restrict__ limbs,
          uint32_t* __restrict__ res, const uint2* __restrict__ twf) {
  stage_begin();
  extern __shared__ __align__(16) uint32_t sm[];
  using S = NttShape<LGN>;
  constexpr int NT = cta_threads(LGN);
  const CtaItem item = cta_item(items, u);
  const FwdDesc d = descs[idx ? idx[item.first] : item.first];
  const Coeffs co(d, limbs);
  const FwdOut out(res, d);
  const NttTables tables{twf};
  const bool hz = d.ncoef <= (uint32_t)(S::N >> 1);
  const int tid = threadIdx.x, j1 = item.j1;
  for (int jb = item.j0; jb < j1; jb += cta_primes(LGN)) {
    const int nb = min(cta_primes(LGN), j1 - jb);
    if (jb > (int)item.j0) __syncthreads();  // every read of the buffers is done
    if (hz)
      fwd_cta_first<LGN, D, true>(co, sm, jb, nb, tables);
    else
      fwd_cta_first<LGN, D, false>(co, sm, jb, nb, tables);
    pass_sync<LGN, 0>();
    fwd_middle<LGN, 3, NT>(sm, nb, jb, tid, tables);
    for (int c = 0; c < nb; ++c)
      each_group<LGN, NT>(tid, [&](int g) {
        uint32_t a[8];
        load_run(sm + c * S::WORDS, g, a);
        fwd_tail<LGN>(a, g, tables.tw(jb + c), c_primes[jb + c].p);
        out.store((uint32_t)((jb + c) * S::NG + g), a, c_primes[jb + c].p);
      });
  }
}

// ---------------------------------------------------------------------------
// Inverse NTT, register-blocked (lgN >= 3): the forward passes backwards.
// Every thread reads its eight consecutive points of the last forward pass
// straight from global memory with vector loads, and the next prime's are
// loaded before the current prime's passes run (where a thread has one
// group), so the loads overlap the arithmetic.  The first forward pass
// inverted writes straight to global memory, values in [0, 2p).  Bound as the
// forward: 794 us for the first 512 products of the default batch (40
// registers, six CTAs an SM), 1137 in the earlier form; a chain step of 64
// entries of 2^14 points 32 us, 157 before its primes went to CTAs of their
// own.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void load_points(const uint32_t* src, uint32_t (&a)[8]) {
  const uint4 u = reinterpret_cast<const uint4*>(src)[0];
  const uint4 v = reinterpret_cast<const uint4*>(src)[1];
  a[0] = u.x; a[1] = u.y; a[2] = u.z; a[3] = u.w;
  a[4] = v.x; a[5] = v.y; a[6] = v.z; a[7] = v.w;
}

// TS threads of one transform (tt among them); primes alternate between two
// buffers `next` words apart (0: one buffer, a barrier more).
template <int LGN, int TS>
__device__ __forceinline__ void inv_run(uint32_t* __restrict__ io, bool valid, uint32_t* sm,
                                        int next, int tt, int j0, int j1, NttTables tables) {
  using S = NttShape<LGN>;
  constexpr bool ONE = S::NG <= TS;  // a group a thread
  io += (uint64_t)j0 << LGN;
  uint32_t nx[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) nx[q] = 0u;
  if (ONE && valid) load_points(io + 8 * tt, nx);
#pragma unroll 1
  for (int j = j0; j < j1; ++j, io += S::N) {
    const uint32_t p = c_primes[j].p;
    const uint2* tw = tables.tw(j);
    uint32_t* s = sm + (j & 1) * next;
    if constexpr (S::LAST == 0) {  // one pass, global -> registers -> global
      uint32_t a[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) a[q] = nx[q];
      if (valid && j + 1 < j1) load_points(io + S::N, nx);
      inv_tail<LGN>(a, 0, tw, p);
      if (valid) {
        uint4* o = reinterpret_cast<uint4*>(io);
        o[0] = make_uint4(a[0], a[1], a[2], a[3]);
        o[1] = make_uint4(a[4], a[5], a[6], a[7]);
      }
    } else {
      each_group<LGN, TS>(tt, [&](int g) {
        uint32_t a[8];
        if constexpr (ONE) {
#pragma unroll
          for (int q = 0; q < 8; ++q) a[q] = nx[q];
          if (valid && j + 1 < j1) load_points(io + S::N + 8 * g, nx);
        } else {
          load_points(io + 8 * g, a);
        }
        inv_tail<LGN>(a, g, tw, p);
        store_run(s, g, a);
      });
      inv_middle<LGN, S::LAST - 3, TS>(s, j, tt, tables);
      const Tw8 t(tw, 1);
      each_group<LGN, TS>(tt, [&](int g) {
        uint32_t a[8];
        load_group<LGN, 0>(s, g, a);
        inv8_first(a, t, p);
        if (valid) {
#pragma unroll
          for (int q = 0; q < 8; ++q) io[q * S::NG + g] = a[q];
        }
      });
      if (next == 0) __syncthreads();
    }
  }
}

__global__ void __launch_bounds__(kFwdThreads, 6)
k_inv_team(const InvDesc* __restrict__ descs, const uint32_t* __restrict__ idx,
           const CtaItem* __restrict__ items, CtaUniform u, uint32_t* __restrict__ res,
           const uint2* __restrict__ twi) {
  stage_begin();
  __shared__ __align__(16) uint32_t buf[2 * kTeamWords];
  const CtaItem item = cta_item(items, u);
  const int lgN = item.lgN;
  const int team = (int)threadIdx.x >> (lgN - 3);
  const int tt = (int)threadIdx.x & ((1 << (lgN - 3)) - 1);
  const bool valid = team < (int)item.count;
  uint32_t* io = res + (valid ? descs[idx ? idx[item.first + team] : item.first + team].res_off : 0);
  switch (lgN) {
#define MPZMM_CASE(L)                                                                      \
  case L:                                                                                  \
    inv_run<L, (1 << L) / 8>(io, valid, buf + pad4(team << L), kTeamWords, tt, item.j0,    \
                             item.j1, NttTables{twi});                                     \
    break;
    MPZMM_TEAM_SIZES(MPZMM_CASE)
#undef MPZMM_CASE
  }
}

template <int LGN>
__global__ void __launch_bounds__(cta_threads(LGN), 1024 / cta_threads(LGN))
k_inv_cta(const InvDesc* __restrict__ descs, const uint32_t* __restrict__ idx,
          const CtaItem* __restrict__ items, CtaUniform u, uint32_t* __restrict__ res,
          const uint2* __restrict__ twi) {
  stage_begin();
  extern __shared__ __align__(16) uint32_t sm[];
  const CtaItem item = cta_item(items, u);
  uint32_t* io = res + descs[idx ? idx[item.first] : item.first].res_off;
  inv_run<LGN, cta_threads(LGN)>(io, true, sm, LGN == 15 ? 0 : NttShape<LGN>::WORDS,
                                 (int)threadIdx.x, item.j0, item.j1, NttTables{twi});
}

// ---------------------------------------------------------------------------
// Transforms longer than one CTA holds (2^16 .. 2^20 points): four steps on
// the same tree.
//
// The forward tree's first lgR stages only combine points x = q C + lo with
// the same lo (C = 2^kLargeLgC, R = N / C), and their twiddles T[m + i] do
// not depend on N: for each of the C columns they are an ordinary R-point
// forward transform.  Afterwards block b = [b C, (b + 1) C) (b = the row
// position, already bit-reversed) holds a(X) mod (X^C - psi_b^C) with
// psi_b = w_N^brev(b), and the remaining stages on the block equal the
// twist y -> psi_b^y a_y followed by an ordinary C-point transform.  So:
//   k_fwd_cols           split + column transforms + twist, on tiles of
//                        R rows x W columns (R W = 2048 points: one group of
//                        eight a thread, its digits kept in registers for all
//                        P primes)
//   k_ntt_blocks<true>   C-point transforms of the blocks (vector loads)
// and the inverse the other way round:
//   k_ntt_blocks<false>  inverse C-point transforms, untwist by psi_b^-y
//   k_inv_cols           inverse column transforms, natural order out
// The result is the same canonical evaluation at the same position as the
// one-CTA transform, and the inverse again returns N times its input.
// Twist factors W^E, W a primitive 2^20-th root with W^32 the 2^15 table's
// root and E = brev(b) y 2^(20 - lgN), take one Shoup product of two table
// entries (TwistTab) and one Montgomery product.
// ---------------------------------------------------------------------------
constexpr int kColPoints = 2048;  // points of a column tile (R x W)
constexpr int kLgColPoints = 11;

// x W^E mod p in [0, p) for x < 4p, E < 2^20 (tables of one prime)
__device__ __forceinline__ uint32_t twist_mul(uint32_t x, uint32_t E,
                                              const uint2* __restrict__ hi,
                                              const uint32_t* __restrict__ lo, uint32_t p,
                                              uint32_t pinv) {
  const uint2 h = __ldg(hi + (E >> 10));
  const uint32_t f = mul_shoup(__ldg(lo + (E & 1023u)), h.x, h.y, p);  // W^E 2^32 mod p
  return redc((uint64_t)x * f, p, pinv);  // x f < 4 p^2 < p 2^32
}

// element (row q, column c) of a column tile with 2^lgW columns
__device__ __forceinline__ int cti(int q, int c, int lgW) { return smi((q << lgW) + c); }

// one pass of three stages (s0 .. s0 + 2) over every column of the tile
template <bool FWD>
__device__ __forceinline__ void col_pass3(uint32_t* s, int lgR, int lgW, int s0,
                                          const uint2* __restrict__ tw, uint32_t p) {
  const int lg_tmin = lgR - s0 - 3;
  const int groups = (1 << (lgR - 3)) << lgW;
  for (int gi = threadIdx.x; gi < groups; gi += blockDim.x) {
    const int c = gi & ((1 << lgW) - 1);
    const int g = gi >> lgW;
    const int lo = g & ((1 << lg_tmin) - 1);
    const int hi = g >> lg_tmin;
    const int base = (hi << (lg_tmin + 3)) + lo;
    uint32_t a[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) a[q] = s[cti(base + (q << lg_tmin), c, lgW)];
    if (FWD)
      fwd_group<3>(a, s0, hi, tw, p);
    else
      inv_group<3>(a, s0, hi, tw, p);
#pragma unroll
    for (int q = 0; q < 8; ++q) s[cti(base + (q << lg_tmin), c, lgW)] = a[q];
  }
}

// the last forward column pass (LP stages from last_s0, groups of 2^LP
// consecutive rows), twisted and stored to the polynomial `out`
template <int LP>
__device__ __forceinline__ void col_last_fwd(const uint32_t* s, uint32_t* __restrict__ out,
                                             int lgR, int lgW, int lgN, int lo0, int last_s0,
                                             const uint2* __restrict__ tw,
                                             const uint2* __restrict__ th,
                                             const uint32_t* __restrict__ tl, uint32_t p,
                                             uint32_t pinv) {
  const int groups = (1 << (lgR - LP)) << lgW;
  for (int gi = threadIdx.x; gi < groups; gi += blockDim.x) {
    const int c = gi & ((1 << lgW) - 1);
    const int hi = gi >> lgW;
    uint32_t a[1 << LP];
#pragma unroll
    for (int q = 0; q < (1 << LP); ++q) a[q] = s[cti((hi << LP) + q, c, lgW)];
    fwd_group<LP>(a, last_s0, hi, tw, p);
    const uint32_t y = (uint32_t)(lo0 + c);
#pragma unroll
    for (int q = 0; q < (1 << LP); ++q) {
      const uint32_t row = (uint32_t)((hi << LP) + q);
      const uint32_t E = ((__brev(row) >> (32 - lgR)) * y) << (20 - lgN);
      out[((uint64_t)row << kLargeLgC) + y] = twist_mul(a[q], E, th, tl, p, pinv);
    }
  }
}

// the last forward column pass inverted: groups of 2^LP consecutive rows
// from the polynomial `in`, into the tile
template <int LP>
__device__ __forceinline__ void col_last_inv(uint32_t* s, const uint32_t* __restrict__ in,
                                             int lgR, int lgW, int lo0, int last_s0,
                                             const uint2* __restrict__ tw, uint32_t p) {
  const int groups = (1 << (lgR - LP)) << lgW;
  for (int gi = threadIdx.x; gi < groups; gi += blockDim.x) {
    const int c = gi & ((1 << lgW) - 1);
    const int hi = gi >> lgW;
    uint32_t a[1 << LP];
#pragma unroll
    for (int q = 0; q < (1 << LP); ++q)
      a[q] = in[((uint64_t)((hi << LP) + q) << kLargeLgC) + (uint32_t)(lo0 + c)];
    inv_group<LP>(a, last_s0, hi, tw, p);
#pragma unroll
    for (int q = 0; q < (1 << LP); ++q) s[cti((hi << LP) + q, c, lgW)] = a[q];
  }
}

// primes [P y / Y, P (y + 1) / Y) of grid row y of Y
__device__ __forceinline__ void chunk_primes(int P, int* j0, int* j1) {
  *j0 = (int)(P * blockIdx.y / gridDim.y);
  *j1 = (int)(P * (blockIdx.y + 1) / gridDim.y);
}

// Split + column transforms + twist.  grid = (entries x tiles, chunks of
// primes) (2 R tiles of W = 2048 / R columns per entry); every entry of a
// launch has 2^lgN points.
template <int D>
__global__ void __launch_bounds__(kFwdThreads, 3)
k_fwd_cols(const FwdDesc* __restrict__ descs, const uint32_t* __restrict__ idx, int tiles,
           const uint64_t* __restrict__ limbs, uint32_t* __restrict__ res,
           const uint2* __restrict__ twf, TwistTab tt) {
  extern __shared__ uint32_t sm[];
  const int e = blockIdx.x / tiles;
  const int tile = blockIdx.x - e * tiles;
  const FwdDesc d = descs[idx ? idx[e] : e];
  const int lgN = d.lgN;
  const int lgR = lgN - kLargeLgC;
  const int lgW = kLgColPoints - lgR;
  const int lo0 = tile << lgW;
  const uint64_t N = (uint64_t)1 << lgN;
  const uint32_t nl = (uint32_t)(d.size < 0 ? -d.size : d.size);
  const uint32_t nw = nl < 0x40000000u ? 2u * nl : 0x80000000u;
  const uint32_t* __restrict__ w32 = reinterpret_cast<const uint32_t*>(limbs + d.limb_off);
  const bool neg = d.size < 0;
  // first-pass group of this thread: rows k R/8 + g of column c
  const int c = (int)threadIdx.x & ((1 << lgW) - 1);
  const int g = (int)threadIdx.x >> lgW;
  const int lgR8 = lgR - 3;
  // no coefficient in the upper half of the transform: rows k >= 4 of every
  // first-pass group are zero (uniform: one entry per CTA)
  const bool hz = d.ncoef <= (uint32_t)(N >> 1);
  uint32_t dg[8][D];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const uint32_t x = ((uint32_t)((k << lgR8) + g) << kLargeLgC) + (uint32_t)(lo0 + c);
    coeff_digits<D>(w32, nw, x * d.r, d.r, x < d.ncoef && !(hz && k >= 4), dg[k]);
  }
  const int last_s0 = ((lgR - 1) / 3) * 3;
  int j0, j1;
  chunk_primes(d.P, &j0, &j1);
  for (int j = j0; j < j1; ++j) {
    const uint32_t p = c_primes[j].p;
    const uint2* tw = twf + (size_t)j * kTwStride;
    uint32_t a[8];
    if (hz) {
#pragma unroll
      for (int k = 0; k < 4; ++k) a[k] = digits_residue<D>(dg[k], j, neg);
      fwd_stage0_upper_zero<3>(a, p);
      fwd_group<3, 1>(a, 0, 0, tw, p);
    } else {
#pragma unroll
      for (int k = 0; k < 8; ++k) a[k] = digits_residue<D>(dg[k], j, neg);
      fwd_group<3>(a, 0, 0, tw, p);
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) sm[cti((k << lgR8) + g, c, lgW)] = a[k];
    __syncthreads();
    for (int s0 = 3; s0 < last_s0; s0 += 3) {
      col_pass3<true>(sm, lgR, lgW, s0, tw, p);
      __syncthreads();
    }
    uint32_t* out = res + d.res_off + (uint64_t)j * N;
    const uint2* th = tt.hi + (size_t)j * kTwistEntries;
    const uint32_t* tl = tt.lo + (size_t)j * kTwistEntries;
    const uint32_t pinv = c_primes[j].pinv;
    switch (lgR - last_s0) {
      case 1: col_last_fwd<1>(sm, out, lgR, lgW, lgN, lo0, last_s0, tw, th, tl, p, pinv); break;
      case 2: col_last_fwd<2>(sm, out, lgR, lgW, lgN, lo0, last_s0, tw, th, tl, p, pinv); break;
      default: col_last_fwd<3>(sm, out, lgR, lgW, lgN, lo0, last_s0, tw, th, tl, p, pinv); break;
    }
    __syncthreads();  // before the next prime overwrites the tile
  }
}

// C-point transforms of the blocks.  grid = (entries x R blocks, chunks of
// primes).  Forward: ordinary forward transform of each (twisted) block.
// Inverse: ordinary inverse transform, then the untwist psi_b^-y (tt holds
// the inverse twist tables).  Descriptors: fdescs (forward) or idescs
// (inverse).  Two buffers in turn, as the team kernels.
constexpr int kBlockThreads = 1 << (kLargeLgC - 3);  // a group of eight a thread

template <bool FWD>
__global__ void __launch_bounds__(kBlockThreads, 2)
k_ntt_blocks(const FwdDesc* __restrict__ fdescs, const InvDesc* __restrict__ idescs,
             const uint32_t* __restrict__ idx, int blocks, uint32_t* __restrict__ res,
             const uint2* __restrict__ tws, TwistTab tt) {
  constexpr int lgC = kLargeLgC;
  using S = NttShape<lgC>;
  __shared__ __align__(16) uint32_t buf[2 * S::WORDS];
  const int e = blockIdx.x / blocks;
  const int b = blockIdx.x - e * blocks;
  uint64_t off;
  int lgN, P;
  if (FWD) {
    const FwdDesc& d = fdescs[idx ? idx[e] : e];
    off = d.res_off;
    lgN = d.lgN;
    P = d.P;
  } else {
    const InvDesc& d = idescs[idx ? idx[e] : e];
    off = d.res_off;
    lgN = d.lgN;
    P = d.P;
  }
  const int lgR = lgN - lgC;
  const uint64_t N = (uint64_t)1 << lgN;
  const int tid = threadIdx.x;
  const uint32_t bb = __brev((uint32_t)b) >> (32 - lgR);
  const NttTables tables{tws};
  int j0, j1;
  chunk_primes(P, &j0, &j1);
#pragma unroll 1
  for (int j = j0; j < j1; ++j) {
    const uint32_t p = c_primes[j].p;
    const uint2* tw = tables.tw(j);
    uint32_t* io = res + off + (uint64_t)j * N + ((uint64_t)b << lgC);
    uint32_t* s = buf + (j & 1) * S::WORDS;
    uint32_t a[8];
    if (FWD) {
#pragma unroll
      for (int q = 0; q < 8; ++q) a[q] = io[q * S::NG + tid];
      fwd8_first(a, Tw8(tw, 1), p);
      store_group<lgC, 0>(s, tid, a);
      pass_sync<lgC, 0>();
      fwd_middle<lgC, 3, kBlockThreads>(s, 1, j, tid, tables);
      load_run(s, tid, a);
      fwd_tail<lgC>(a, tid, tw, p);
      FwdDesc d{};
      d.res_off = off + (uint64_t)j * N + ((uint64_t)b << lgC);
      FwdOut(res, d).store((uint32_t)tid, a, p);
    } else {
      load_points(io + 8 * tid, a);
      inv_tail<lgC>(a, tid, tw, p);
      store_run(s, tid, a);
      inv_middle<lgC, S::LAST - 3, kBlockThreads>(s, j, tid, tables);
      load_group<lgC, 0>(s, tid, a);
      inv8_first(a, Tw8(tw, 1), p);
      const uint2* th = tt.hi + (size_t)j * kTwistEntries;
      const uint32_t* tl = tt.lo + (size_t)j * kTwistEntries;
      const uint32_t pinv = c_primes[j].pinv;
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const uint32_t y = (uint32_t)(q * S::NG + tid);
        io[y] = twist_mul(a[q], (bb * y) << (20 - lgN), th, tl, p, pinv);
      }
    }
  }
}

// Inverse column transforms, natural coefficient order out (values in
// [0, 2p), as the CRT expects).  grid as k_fwd_cols.
__global__ void __launch_bounds__(kFwdThreads)
k_inv_cols(const InvDesc* __restrict__ descs, const uint32_t* __restrict__ idx, int tiles,
           uint32_t* __restrict__ res, const uint2* __restrict__ twi) {
  extern __shared__ uint32_t sm[];
  const int e = blockIdx.x / tiles;
  const int tile = blockIdx.x - e * tiles;
  const InvDesc d = descs[idx ? idx[e] : e];
  const int lgN = d.lgN;
  const int lgR = lgN - kLargeLgC;
  const int lgW = kLgColPoints - lgR;
  const int lo0 = tile << lgW;
  const uint64_t N = (uint64_t)1 << lgN;
  const int c = (int)threadIdx.x & ((1 << lgW) - 1);
  const int g = (int)threadIdx.x >> lgW;
  const int lgR8 = lgR - 3;
  const int last_s0 = ((lgR - 1) / 3) * 3;
  int j0, j1;
  chunk_primes(d.P, &j0, &j1);
  for (int j = j0; j < j1; ++j) {
    const uint32_t p = c_primes[j].p;
    const uint2* tw = twi + (size_t)j * kTwStride;
    uint32_t* io = res + d.res_off + (uint64_t)j * N;
    switch (lgR - last_s0) {
      case 1: col_last_inv<1>(sm, io, lgR, lgW, lo0, last_s0, tw, p); break;
      case 2: col_last_inv<2>(sm, io, lgR, lgW, lo0, last_s0, tw, p); break;
      default: col_last_inv<3>(sm, io, lgR, lgW, lo0, last_s0, tw, p); break;
    }
    __syncthreads();
    for (int s0 = last_s0 - 3; s0 >= 3; s0 -= 3) {
      col_pass3<false>(sm, lgR, lgW, s0, tw, p);
      __syncthreads();
    }
    uint32_t a[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) a[k] = sm[cti((k << lgR8) + g, c, lgW)];
    inv_group<3>(a, 0, 0, tw, p);
#pragma unroll
    for (int k = 0; k < 8; ++k)
      io[((uint64_t)((k << lgR8) + g) << kLargeLgC) + (uint32_t)(lo0 + c)] = a[k];
    __syncthreads();  // before the next prime overwrites the tile
  }
}


// ---------------------------------------------------------------------------
// CRT + recompose, one warp per output entry or segment of one (no block
// barriers).
//
// Explicit CRT (crt_coeff) to the symmetric P-word value U_i - s_i 2^(32P)
// of each coefficient (s_i = top bit of U_i), per-word gathered sums, carries
// normalised into {-1, 0, 1}.  The ripple is resolved per 32-word step: when
// no word of the step is 0 or all-ones (a carry can only pass through such a
// word), word w's incoming carry is just the generated carry g_{w-1}; only
// otherwise does the warp run the prefix scan of transfer functions.
// ---------------------------------------------------------------------------
constexpr int kCrtWarps = 4;       // entries per CTA
constexpr int kCrtSteps = 8;       // 32-word steps per tile
constexpr int kCrtTileWords = 32 * kCrtSteps;
constexpr size_t kCrtSmemLimit = 200 * 1024;
// scratch words of a coefficient: P + 1 of them used, an odd number apart
// (the lanes' stores spread over the banks)
template <int P>
constexpr int kCrtStride = (P + 1) | 1;

// Explicit CRT of one coefficient (constants in CrtConst): the symmetric
// residue X in (-M_P/4, M_P/4) as P words of two's complement.
template <int P>
__device__ __forceinline__ void crt_coeff(const uint32_t* src, uint32_t N, int lgN,
                                          uint32_t (&X)[P]) {
  int32_t y[P];
  uint64_t frac = 0;
#pragma unroll
  for (int j = 0; j < P; ++j) {
    const uint32_t p = c_primes[j].p;
    const uint64_t T = (uint64_t)stage_load(src) * c_crt.cm[P][lgN][j];  // [0, 2p) times [0, p)
    src += N;
    const uint32_t m = (uint32_t)T * c_primes[j].pinv;
    uint32_t v = (uint32_t)((T + (uint64_t)m * p) >> 32);  // [0, 2p)
    // beyond eight primes the columns below have room for [0, p) only
    if (P > 8) v = min(v, v - p);
    y[j] = (int32_t)v;
    frac += (uint64_t)v * c_crt.fq[j];
  }
  const int32_t q = (int32_t)((frac + (1ull << 57)) >> 58);  // nearest integer
  // sum_j y_j (M_P / p_j) - q M_P in balanced base-2^30 columns, no carries
  // inside the sums
  int64_t acc[P];
#pragma unroll
  for (int w = 0; w < P; ++w) acc[w] = -(int64_t)q * c_crt.M30[P][w];
#pragma unroll
  for (int j = 0; j < P; ++j)
#pragma unroll
    for (int w = 0; w < P; ++w) acc[w] += (int64_t)y[j] * c_crt.mop30[P][j][w];
  // one signed carry pass to digits in [0, 2^30); what is left over is 0 for
  // X >= 0 and -1 for X < 0.  The 30P bits go to P 32-bit words on the way.
  int64_t cy = 0;
  uint64_t buf = 0;
  int bits = 0, wi = 0;
#pragma unroll
  for (int w = 0; w < P; ++w) {
    const int64_t t = acc[w] + cy;
    buf |= (uint64_t)((uint32_t)t & 0x3fffffffu) << bits;
    cy = t >> 30;  // arithmetic: floor division
    bits += 30;
    if (bits >= 32) {
      X[wi++] = (uint32_t)buf;
      buf >>= 32;
      bits -= 32;
    }
  }
  const uint32_t fill = cy < 0 ? 0xffffffffu : 0u;
#pragma unroll
  for (int w = 0; w < P; ++w) {
    if (w < wi) continue;
    X[w] = (w == wi) ? ((uint32_t)buf | (fill << bits)) : fill;
  }
}

// floor(x / d) for x < 2^31: a multiply-high by floor((2^32 - 1) / d) is at
// most 2 below the quotient, then at most two corrections
struct FastDiv {
  uint32_t d, m;
  __device__ explicit FastDiv(uint32_t d_) : d(d_), m(0xffffffffu / d_) {}
  __device__ __forceinline__ uint32_t operator()(uint32_t x) const {
    uint32_t q = __umulhi(x, m);
    if ((q + 1) * d <= x) ++q;
    if ((q + 1) * d <= x) ++q;
    return q;
  }
};

// The carry into word `wbeg` of a segment, from a look at the 32 words below
// it (lane l holds word wbeg - 32 + l; lane 0 lacks the word below it, so
// its own carry stays open): kCarryUnknown when every word of 1..31 lets a
// carry pass.
constexpr int kCarryUnknown = 2;
__device__ __forceinline__ bool tf_const(uint32_t f) {
  return ((f ^ (f >> 2)) & 15u) == 0u;
}
__device__ __forceinline__ int lookback_carry(uint32_t y, int g, bool prop, int lane) {
  const unsigned FULL = 0xffffffffu;
  const unsigned pm = __ballot_sync(FULL, prop);
  if (!(pm >> 31)) return __shfl_sync(FULL, g, 31);  // word wbeg - 1 settles it
  uint32_t inc = lane == 0 ? kTfIdentity : word_tf(y, g);
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t u = __shfl_up_sync(FULL, inc, off);
    if (lane >= off) inc = compose_tf(inc, u);
  }
  inc = __shfl_sync(FULL, inc, 31);
  return tf_const(inc) ? apply_tf(inc, 0) : kCarryUnknown;
}

// Words [wbeg, wend) of one output entry by one warp: CRT of its
// coefficients tile by tile into the warp's scratch sV, each coefficient
// pre-shifted to its place in the output words (P + 1 words of tile
// coefficient c at [c kCrtStride<P>]), the words' sums, the carry ripple.
//
// SEG false: the whole entry (wbeg = 0, wend = out_words), with its sign,
// negation and size.  SEG true: one segment of an entry that several warps
// share (wbeg a multiple of 32): the carry into the segment comes from
// the 32 words below it, which the first tile computes again without
// storing them; the words are written in two's complement and the record
// tells k_crt_finish what it needs of the segment.  While the carry in is
// unknown (the words below are all 0 or all ones: structured operands, or
// the sign fill above a short result) the words are written for a carry of
// 0 and the record keeps the three possible outcomes.
//
// One warp an entry, whatever its length, left the GPU idle on few long
// entries: a 2 x 2 product of 10^7-bit integers spent 12.9 of its 13.3 ms on
// four warps here, an 8 x 8 one of 2^16-bit integers 103 of 150 us of
// kernels on 64.  (Two kernels, because the segment's state costs whole
// entries 8 registers and a CTA less an SM: 9 % of the stage's time.)
template <int P, bool SEG>
__device__ __forceinline__ void crt_range(const InvDesc& d, const uint32_t* res,
                                          uint32_t* __restrict__ out,
                                          int32_t* __restrict__ out_sizes, uint32_t* sV,
                                          int wbeg, int wend, CrtRec* __restrict__ rec,
                                          int lane) {
  const unsigned FULL = 0xffffffffu;
  // bit positions fit 31 bits (an entry's words times 32 stays below 2^31),
  // so index arithmetic is 32-bit and the divisions by r are multiply-highs
  const int r = (int)d.r;
  const FastDiv divr((uint32_t)r);
  const uint32_t half_r = 0x80000000u / (uint32_t)r;  // see the division by r below
  const int reach = (32 * P + 31) / r + 1;  // most coefficients that meet in a word
  const int ncoef = (int)d.ncoef;
  const uint32_t* src = res + d.res_off;
  const uint32_t N = 1u << d.lgN;
  uint32_t* o = out + d.out_word;

  int hi_prev = 0, carry = 0;
  int first_nz = 0x7fffffff, last_nz = -1, last_no = -1;
  uint32_t topval = 0;
  bool unknown = false;           // the carry into the segment is still open
  bool open = false, top_open = false;  // it was at the start / at the last step
  uint32_t cf = kTfIdentity;      // from that carry to the current one
  for (int w0 = SEG && wbeg > 0 ? wbeg - 32 : 0; w0 < wend; w0 += kCrtTileWords) {
    const int wt = w0 + kCrtTileWords < wend ? w0 + kCrtTileWords : wend;
    int lo_i = 0;
    if (32 * w0 > 32 * P) lo_i = (int)divr((uint32_t)(32 * w0 - 32 * P + r - 1));
    int hi_i = (int)divr((uint32_t)(32 * wt - 1));
    if (hi_i > ncoef - 1) hi_i = ncoef - 1;
    const int ncf = hi_i >= lo_i ? hi_i - lo_i + 1 : 0;
    // coefficient i = lo_i + c as X_i 2^(i r mod 32): P + 1 words, the top
    // one signed (it carries the sign's borrow), so output word w adds word
    // w - floor(i r / 32) of every coefficient that reaches it
#pragma unroll 1
    for (int c = lane; c < ncf; c += 32) {
      uint32_t X[P];
      crt_coeff<P>(src + lo_i + c, N, d.lgN, X);
      const uint32_t sh = (uint32_t)((lo_i + c) * r) & 31u;
      uint32_t* v = sV + c * kCrtStride<P>;
      v[0] = X[0] << sh;
#pragma unroll
      for (int q = 1; q < P; ++q) v[q] = __funnelshift_l(X[q - 1], X[q], sh);
      v[P] = __funnelshift_l(X[P - 1], (uint32_t)((int32_t)X[P - 1] >> 31), sh);
    }
    __syncwarp();
    const int bit0 = lo_i * r;  // where the tile's first coefficient starts
#pragma unroll 1
    for (int st = 0; st < kCrtSteps; ++st) {
      const int ws = w0 + 32 * st;
      if (ws >= wt) break;
      const int w = ws + lane;
      const bool active = w < wend;
      int64_t sw = 0;
      if (active) {
        // the last coefficient that reaches word w starts at or before its
        // top bit x = 32 w + 31 - bit0 (below 2^14): floor(x / r) as the
        // multiply-high of 2x + 1 by floor(2^31 / r), which errs by less than
        // 2^-17 below (2x + 1) / (2r), at least 1 / (2r) above an integer
        int b = 32 * w + 31 - bit0;
        int c = (int)__umulhi(2u * (uint32_t)b + 1u, half_r);
        if (c > ncf - 1) c = ncf - 1;
        b -= c * r;
        // b: from the coefficient's first bit up to the word's top bit, so
        // the word takes word b / 32 of it; earlier ones lie r bits further
        const uint32_t* v = sV + c * kCrtStride<P>;
#pragma unroll 1
        for (int t = 0; t < reach; ++t) {
          const int q = b >> 5;
          if (c >= 0 && q <= P) {
            const uint32_t x = v[q];
            sw += q == P ? (int64_t)(int32_t)x : (int64_t)x;
          }
          --c;
          v -= kCrtStride<P>;
          b += r;
        }
      }
      const int hi = active ? (int)(sw >> 32) : 0;
      int hprev = __shfl_up_sync(FULL, hi, 1);
      if (lane == 0) hprev = hi_prev;
      hi_prev = __shfl_sync(FULL, hi, 31);
      const int64_t z = (int64_t)(uint32_t)sw + hprev;
      const uint32_t y = (uint32_t)z;
      const int g = active ? (int)(z >> 32) : 0;
      const bool prop = active && (y == 0u || y == 0xffffffffu);
      if (SEG && ws < wbeg) {  // the look at the words below the segment
        carry = lookback_carry(y, g, prop, lane);
        if (carry == kCarryUnknown) {
          unknown = open = true;
          carry = 0;
          if (lane == 0)
            for (int c = 0; c < 3; ++c) {
              rec->first_nz[c] = 0x7fffffff;
              rec->last_nz[c] = rec->last_no[c] = -1;
            }
        }
        continue;
      }
      int cin, cout;
      if (__any_sync(FULL, prop) || (SEG && unknown)) {
        const uint32_t f = active ? word_tf(y, g) : kTfIdentity;
        uint32_t inc = f;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
          const uint32_t u = __shfl_up_sync(FULL, inc, off);
          if (lane >= off) inc = compose_tf(inc, u);
        }
        uint32_t exc = __shfl_up_sync(FULL, inc, 1);
        if (lane == 0) exc = kTfIdentity;
        const uint32_t all = __shfl_sync(FULL, inc, 31);
        if (SEG && unknown) {  // this step's outcomes for each carry into the segment
          for (int c = 0; c < 3; ++c) {
            const uint32_t F = y + (uint32_t)apply_tf(compose_tf(exc, cf), c - 1);
            const unsigned nz = __ballot_sync(FULL, active && F != 0u);
            const unsigned no = __ballot_sync(FULL, active && F != 0xffffffffu);
            const unsigned top = __ballot_sync(FULL, w == wend - 1 && (F >> 31));
            if (lane == 0) {
              if (nz && rec->first_nz[c] == 0x7fffffff) rec->first_nz[c] = ws + __ffs(nz) - 1;
              if (nz) rec->last_nz[c] = ws + 31 - __clz(nz);
              if (no) rec->last_no[c] = ws + 31 - __clz(no);
              rec->top[c] = top != 0;
            }
          }
          cf = compose_tf(all, cf);
        }
        cin = apply_tf(exc, carry);
        cout = apply_tf(all, carry);
      } else {
        cin = __shfl_up_sync(FULL, g, 1);
        if (lane == 0) cin = carry;
        cout = __shfl_sync(FULL, g, 31);
      }
      if (active) {
        const uint32_t F = y + (uint32_t)cin;
        o[w] = F;
        if (!SEG || !unknown) {
          if (F != 0u) {
            first_nz = min(first_nz, w);
            last_nz = w;
          }
          if (F != 0xffffffffu) last_no = w;
          if (w == wend - 1) topval = F;
        }
      }
      carry = cout;
      if (SEG) {
        top_open = unknown;
        if (unknown && tf_const(cf)) unknown = false;  // settled from the next word on
      }
    }
    __syncwarp();
  }
  first_nz = __reduce_min_sync(FULL, first_nz);
  last_nz = __reduce_max_sync(FULL, last_nz);
  last_no = __reduce_max_sync(FULL, last_no);
  topval = __reduce_or_sync(FULL, topval);
  if (SEG) {
    if (lane != 0) return;
    for (int c = 0; c < 3; ++c) {
      if (!open) {
        rec->first_nz[c] = first_nz;
        rec->last_nz[c] = last_nz;
        rec->last_no[c] = last_no;
      } else {
        rec->first_nz[c] = min(rec->first_nz[c], first_nz);
        rec->last_nz[c] = max(rec->last_nz[c], last_nz);
        rec->last_no[c] = max(rec->last_no[c], last_no);
      }
      if (!top_open) rec->top[c] = (int32_t)(topval >> 31);
    }
    rec->tf = unknown ? cf : 0x15u * (uint32_t)(carry + 1);
    rec->open = open;
    return;
  }
  const bool negative = wend > 0 && (topval >> 31);
  int top;
  if (negative) {
    const int zf = first_nz;
    for (int w = zf + lane; w < wend; w += 32) {
      const uint32_t F = o[w];
      o[w] = (w == zf) ? (0u - F) : ~F;
    }
    top = last_no > zf ? last_no : zf;
  } else {
    top = last_nz;
  }
  if (lane == 0) {
    const int limbs = top >= 0 ? top / 2 + 1 : 0;
    out_sizes[d.entry] = negative ? -limbs : limbs;
  }
}

// item `slot` of a launch whose entries 0, 1, ... are all alike
__device__ __forceinline__ CrtItem uniform_item(const CrtUniform& u, uint32_t slot) {
  CrtItem it;
  it.inv = slot / u.nseg;
  it.seg = slot - it.inv * u.nseg;
  it.nseg = u.nseg;
  it.rec = it.inv * u.nseg;
  it.w0 = it.seg * u.step;
  it.w1 = it.seg + 1 < u.nseg ? it.w0 + u.step : u.words;
  return it;
}

template <int P, int PHI, bool SEG>
__device__ __forceinline__ void crt_dispatch(const InvDesc& d, const CrtItem& it,
                                             const uint32_t* res, uint32_t* __restrict__ out,
                                             int32_t* __restrict__ out_sizes, uint32_t* sU,
                                             CrtRec* __restrict__ rec, int lane) {
  if (d.P == P) {
    crt_range<P, SEG>(d, res, out, out_sizes, sU, (int)it.w0, (int)it.w1, rec, lane);
  } else {
    if constexpr (P < PHI)
      crt_dispatch<P + 1, PHI, SEG>(d, it, res, out, out_sizes, sU, rec, lane);
  }
}

// Prime counts PLO..PHI in one launch (one tail instead of one per count), one
// warp an item: segments (SEG; segs, or u where all entries are alike), or
// whole entries (idx, or entries 0, 1, ...).  Each warp's scratch holds
// warp_words words.
//
// Bound by integer issue and, over mixed prime counts, by instruction fetch:
// each count is code of its own, so loops stay rolled and the lists are in
// prime count order.  64 x 64 entries of 65538 words (10 primes) 3190 us,
// 3650 with the columns' carries, the subtraction of q M and the repacking in
// passes of their own and two checked divisions a word; 512 mixed products
// 1763 us, 1995 before.
template <int PLO, int PHI, bool SEG>
__global__ void __launch_bounds__(32 * kCrtWarps, PLO > 2 ? 6 : 7)
k_crt_mixed(const InvDesc* __restrict__ descs, const CrtItem* __restrict__ segs,
            const uint32_t* __restrict__ idx, int count, CrtUniform u,
            const uint32_t* res, uint32_t* __restrict__ out, int32_t* __restrict__ out_sizes,
            CrtRec* __restrict__ recs, int warp_words) {
  stage_begin();
  extern __shared__ uint32_t sm[];
  const int warp = threadIdx.x >> 5;
  const int slot = blockIdx.x * kCrtWarps + warp;
  if (slot >= count) return;  // whole warp; no block-wide barrier below
  CrtItem it;
  if (SEG) {
    it = segs ? segs[slot] : uniform_item(u, (uint32_t)slot);
  } else {
    it.inv = idx ? idx[slot] : (uint32_t)slot;
    it.w0 = it.rec = it.seg = 0;
    it.w1 = descs[it.inv].out_words;
  }
  const InvDesc d = descs[it.inv];
  crt_dispatch<PLO, PHI, SEG>(d, it, res, out, out_sizes, sm + warp * warp_words,
                              SEG ? recs + it.rec + it.seg : nullptr, threadIdx.x & 31);
}

// The sign, negation and size of entries in segments, one warp a segment:
// settles the carry into segments whose own look left it open, complements
// the words of negative entries and (the top segment's warp) writes the
// size.  Mostly three records tell everything: this segment's carry is
// known, the one below holds a nonzero word, the top one knows its sign.
// Otherwise (zeros, powers of two, sign fill above a short result) the warp
// runs over the entry's records once, 32 a step.
__global__ void __launch_bounds__(32 * kCrtWarps)
k_crt_finish(const InvDesc* __restrict__ descs, const CrtItem* __restrict__ segs, int count,
             CrtUniform un, const CrtRec* recs, uint32_t* __restrict__ out,
             int32_t* __restrict__ out_sizes) {
  stage_begin();
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int slot = blockIdx.x * kCrtWarps + (threadIdx.x >> 5);
  if (slot >= count) return;  // whole warp
  const CrtItem it = segs ? segs[slot] : uniform_item(un, (uint32_t)slot);
  const InvDesc& d = descs[it.inv];
  const CrtRec* R = recs + it.rec;
  const int s = (int)it.seg, S = (int)it.nseg;
  const CrtRec& me = R[s];
  uint32_t* o = out + d.out_word;
  const bool open = stage_load(&me.open) != 0;
  int cs = 1;        // the carry into this segment, plus one
  bool negative, below;  // the entry's sign; a nonzero word below this segment
  int top;           // (top segment) last word of the magnitude that is not zero
  if (!open && !stage_load(&R[S - 1].open) &&
      (s == 0 || (!stage_load(&R[s - 1].open) && stage_load(&R[s - 1].last_nz[1]) >= 0)) &&
      (s != S - 1 || (stage_load(&me.last_nz[1]) >= 0 && stage_load(&me.last_no[1]) >= 0))) {
    negative = stage_load(&R[S - 1].top[1]) != 0;
    below = s > 0;
    top = stage_load(negative ? &me.last_no[1] : &me.last_nz[1]);
  } else {
    int c = 1, zf = 0x7fffffff, zb = 0x7fffffff, lz = -1, lo = -1, neg = 0;
    for (int t0 = 0; t0 < S; t0 += 32) {
      const int t = t0 + lane;
      const bool live = t < S;
      const uint32_t tf = live ? stage_load(&R[t].tf) : kTfIdentity;
      int mc = 1;
#pragma unroll
      for (int u = 0; u < 32; ++u) {
        if (lane == u) mc = c;
        c = (int)((__shfl_sync(FULL, tf, u) >> (2 * c)) & 3u);
      }
      const int fn = live ? stage_load(&R[t].first_nz[mc]) : 0x7fffffff;
      zf = min(zf, __reduce_min_sync(FULL, fn));
      zb = min(zb, __reduce_min_sync(FULL, t < s ? fn : 0x7fffffff));
      lz = max(lz, __reduce_max_sync(FULL, live ? stage_load(&R[t].last_nz[mc]) : -1));
      lo = max(lo, __reduce_max_sync(FULL, live ? stage_load(&R[t].last_no[mc]) : -1));
      neg |= __reduce_max_sync(FULL, t == S - 1 ? stage_load(&R[t].top[mc]) : 0);
      if (s >= t0 && s < t0 + 32) cs = __shfl_sync(FULL, mc, s - t0);
    }
    negative = neg != 0;
    below = zb != 0x7fffffff;
    top = negative ? (lo > zf ? lo : zf) : lz;
  }
  const int w0 = (int)it.w0, w1 = (int)it.w1;
  if (open && cs != 1) {  // written for a carry of 0: add it to the segment
    const uint32_t pass = cs == 2 ? 0xffffffffu : 0u;
    for (int ws = w0; ws < w1; ws += 32) {
      const int w = ws + lane;
      const uint32_t F = w < w1 ? o[w] : pass;
      const unsigned stop = __ballot_sync(FULL, F != pass);
      const int k = stop ? __ffs(stop) - 1 : 32;
      if (w < w1 && lane <= k) o[w] = F + (uint32_t)(cs - 1);
      if (stop) break;
    }
  }
  if (negative) {
    const int zf = below ? -1 : stage_load(&me.first_nz[cs]);
    for (int w = w0 + lane; w < w1; w += 32) {
      const uint32_t F = o[w];
      if (w >= zf) o[w] = w == zf ? 0u - F : ~F;
    }
  }
  if (s == S - 1 && lane == 0) {
    const int limbs = top >= 0 ? top / 2 + 1 : 0;
    out_sizes[d.entry] = negative ? -limbs : limbs;
  }
}


// ---------------------------------------------------------------------------
// Tensor-core contraction (byte-plane scheme: contract_tc.cuh).
// ---------------------------------------------------------------------------
__device__ __forceinline__ void tc_mma(uint32_t d, uint64_t ad, uint64_t bd, uint32_t idesc,
                                       uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n"
      :: "r"(d), "l"(ad), "l"(bd), "r"(idesc), "r"(acc), "r"(0u), "r"(0u), "r"(0u), "r"(0u)
      : "memory");
}

__device__ __forceinline__ void tc_commit(uint32_t barp) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
               :: "r"(barp) : "memory");
}

// The MMAs of group gu / nunits of the staged block, output columns
// npl (gu mod nunits) .., into the accumulator at TMEM column dcol: one M
// tile of 128 A' rows at a time, K' in steps of 32 bytes.
__device__ __forceinline__ void tc_issue_unit(const tc::Shape& sh, uint32_t a_base,
                                              uint32_t b_base, int gu, uint32_t dcol) {
  const int g = gu / sh.nunits;
  const int uu = gu - g * sh.nunits;
  const uint32_t kp = (uint32_t)sh.kp;
  const uint32_t a0 = a_base + (uint32_t)(g * sh.a_bytes);
  // B' row 4 npl uu (a multiple of 8: npl = 32 when there are several units)
  const uint32_t b0 = b_base + (uint32_t)(g * sh.b_bytes) + (uint32_t)(4 * sh.npl * uu) * kp;
  const uint32_t idesc = tc::idesc_u8((uint32_t)sh.ncol);
  for (int q = 0; q < sh.mt; ++q)
    for (uint32_t ks = 0; ks < kp / 32; ++ks)
      tc_mma(dcol + (uint32_t)(q * sh.ncol),
             tc::smem_desc(a0 + 128u * (uint32_t)q * kp + 256u * ks, kp),
             tc::smem_desc(b0 + 256u * ks, kp), idesc, ks > 0 ? 1u : 0u);
}

__device__ __forceinline__ void tmem_ld16(uint32_t addr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
        "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]),
        "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(addr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// F consecutive residues (frequencies hs .. hs + F - 1) of entry e of an
// operand stored in the blocked layout (FwdOut): blk is the operand block, np
// its entries, tile the block of frequency hs (prime j included: j N/8 +
// hs/8) and sub = hs mod 8.  Only nf of them exist when the transform is
// shorter than the CTA's frequencies.  Lanes take consecutive entries, so a
// warp's loads are one contiguous run per block.
template <int F>
__device__ __forceinline__ void load_freqs(const uint32_t* __restrict__ blk, uint64_t np,
                                           uint64_t e, uint64_t tile, uint32_t sub, bool ok,
                                           int nf, uint32_t (&x)[F]) {
  if (ok && nf == F && F >= 4) {  // sub is a multiple of 4: 16-byte pieces of blocks
#pragma unroll
    for (int c = 0; c < F / 4; ++c) {
      const uint32_t h = sub + 4u * (uint32_t)c;
      const uint4 u = __ldg(reinterpret_cast<const uint4*>(
          blk + ((tile + (h >> kTcTileLg)) * np + e) * kTcTile + (h & (kTcTile - 1u))));
      x[4 * c] = u.x;
      x[4 * c + 1] = u.y;
      x[4 * c + 2] = u.z;
      x[4 * c + 3] = u.w;
    }
  } else {
#pragma unroll
    for (int f = 0; f < F; ++f) {
      const uint32_t h = sub + (uint32_t)f;
      x[f] = (ok && f < nf) ? __ldg(blk + ((tile + (h >> kTcTileLg)) * np + e) * kTcTile +
                                    (h & (kTcTile - 1u)))
                            : 0u;
    }
  }
}

// Stages the nf frequencies of a packed product (phi > 1): a warp task is 8
// rows (i of A, l of B) by 16 terms of a slot; a thread gathers four terms'
// residues of one row for every frequency and writes their byte planes.
// Small F keeps TU tasks' loads in flight at once.
template <int F, int NT>
__device__ __forceinline__ void tc_stage_packed(const ProdDesc& d, const tc::Shape& sh, int m,
                                                int n, int i_base, int l_base, uint64_t tile0,
                                                uint32_t sub0, int nf,
                                                const uint32_t* __restrict__ res, uint8_t* As,
                                                uint8_t* Bs) {
  const int warp = (int)threadIdx.x >> 5, lane = (int)threadIdx.x & 31;
  const int k = d.k, lgphi = sh.phi == 4 ? 2 : 1;
  const int kbn = (sh.kq + 15) / 16;
  const int a_tasks = ((m + 7) / 8) * kbn;
  const int tasks = a_tasks + ((n + 7) / 8) * kbn;
  constexpr int TU = F <= 4 ? 2 : 1;
  constexpr int kWarps = NT / 32;
  for (int task0 = warp; task0 < tasks; task0 += TU * kWarps) {
    uint32_t x[TU][4][F];
    int rr[TU], kq[TU];
    bool isa[TU];
#pragma unroll
    for (int w2 = 0; w2 < TU; ++w2) {
      const int task = task0 + w2 * kWarps;
      const bool live = task < tasks;
      const bool isA = task < a_tasks;
      const int tt = isA ? task : task - a_tasks;
      const int rb = tt / kbn;
      const int kb = tt - rb * kbn;
      const int kk0 = 16 * kb + 4 * (lane & 3);
      // lane -> (row i of A or column l of B mod 8, term quad)
      const int r = 8 * rb + (lane >> 2);
      rr[w2] = r;
      kq[w2] = kk0;
      isa[w2] = isA;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int kk = kk0 + c;
        const bool ok = live && kk < k && r < (isA ? m : n);
        const uint64_t poly =
            ok ? (isA ? (uint64_t)((i_base + r) * k + kk) : (uint64_t)(kk * d.n + l_base + r))
               : 0;
        load_freqs<F>(res + (isA ? d.a_res : d.b_res),
                      isA ? (uint64_t)d.m * k : (uint64_t)k * d.n, poly, tile0, sub0, ok, nf,
                      x[w2][c]);
      }
    }
#pragma unroll
    for (int w2 = 0; w2 < TU; ++w2) {
      if (task0 + w2 * kWarps >= tasks) break;  // uniform over the warp
      const int r = rr[w2], kk0 = kq[w2];
      if (kk0 >= sh.kq) continue;  // past the slot (a packed slot of 8 or 24 bytes)
#pragma unroll
      for (int f = 0; f < F; ++f) {
        if (f >= nf) break;
        // frequency f: group f / phi, slot f mod phi
        const int g = f >> lgphi, sl = f - (g << lgphi);
        uint32_t pl[4];
        tc::byte_planes(x[w2][0][f], x[w2][1][f], x[w2][2][f], x[w2][3][f], pl);
        // plane s of row i of A (column l of B): row 4 mp sl + 4 r + s of
        // A' (4 r + s of B'), bytes sl kq + kk; the store order rotates
        // with bits 3-4 of the lane so every store covers all 32 banks
        uint8_t* t = isa[w2] ? As + g * sh.a_bytes : Bs + g * sh.b_bytes;
        const uint32_t row0 = isa[w2] ? (uint32_t)(4 * sh.mp * sl + 4 * r) : (uint32_t)(4 * r);
        const uint32_t kb = (uint32_t)(sl * sh.kq + kk0);
        const int gq = (lane >> 3) & 3;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int tp = (q + gq) & 3;
          const uint32_t v = tp == 0 ? pl[0] : (tp == 1 ? pl[1] : (tp == 2 ? pl[2] : pl[3]));
          *reinterpret_cast<uint32_t*>(t + tc::tile_off(row0 + (uint32_t)tp, kb,
                                                        (uint32_t)sh.kp)) = v;
        }
      }
    }
  }
}

// Stages the nf frequencies of a product with one frequency a group (phi =
// 1): a warp task is the block's rows of A (or columns of B), a lane each, by
// 16 terms.  The lane's sixteen loads go out together, and of every
// frequency it writes four 16-byte rows of a core matrix, plane (q + r / 2)
// mod 4 in turn q, so that eight lanes' stores cover all banks (rows r and r
// + 2 lie a multiple of 128 bytes apart).  About 5 instructions a residue;
// four terms a thread, each plane a 4-byte store at an address of its own,
// took 67, three quarters of the kernel's: a 64 x 64 x 64 product of 2^20-bit
// entries contracted in 13.7 ms, in 8.4 now (with the epilogue's weights in
// pairs; 9.1 without).
template <int F, int NT>
__device__ __forceinline__ void tc_stage_rows(const ProdDesc& d, const tc::Shape& sh, int m, int n,
                                              int i_base, int l_base, uint64_t tile0,
                                              uint32_t sub0, int nf,
                                              const uint32_t* __restrict__ res, uint8_t* As,
                                              uint8_t* Bs) {
  const int warp = (int)threadIdx.x >> 5, r = (int)threadIdx.x & 31;
  const int k = d.k;
  const int chunks = sh.kq / 16;
  constexpr int FS = F < 4 ? F : 4;  // frequencies in registers at a time
  for (int task = warp; task < 2 * chunks; task += NT / 32) {
    const bool isa = task < chunks;
    const int ch = isa ? task : task - chunks, kk = 16 * ch;
    if (r >= (isa ? m : n)) continue;  // rows past the block: their results are not read
    const uint32_t np = (uint32_t)(isa ? d.m * k : k * d.n);
    const uint32_t step = (isa ? 1u : (uint32_t)d.n) * kTcTile;  // words a term
    const uint32_t e0 = isa ? (uint32_t)((i_base + r) * k + kk) : (uint32_t)(kk * d.n + l_base + r);
    const uint32_t* __restrict__ blk = res + (isa ? d.a_res : d.b_res) + (uint64_t)e0 * kTcTile;
    uint8_t* dst = (isa ? As : Bs) + tc::tile_off(4u * (uint32_t)r, (uint32_t)kk, (uint32_t)sh.kp);
    const int bytes = isa ? sh.a_bytes : sh.b_bytes;
#pragma unroll 1
    for (int fs = 0; fs < F; fs += FS) {
      const uint32_t h = sub0 + (uint32_t)fs;
      const uint32_t* __restrict__ src =
          blk + (tile0 + (h >> kTcTileLg)) * np * (uint64_t)kTcTile + (h & (kTcTile - 1u));
      uint32_t x[16][FS];
#pragma unroll
      for (int t = 0; t < 16; ++t) {
        const bool ok = kk + t < k;
        if (FS == 4 && nf == F) {  // h is a multiple of 4
          const uint4 u = ok ? __ldg(reinterpret_cast<const uint4*>(src + (uint32_t)t * step))
                             : make_uint4(0u, 0u, 0u, 0u);
          x[t][0] = u.x;
          x[t][1 % FS] = u.y;
          x[t][2 % FS] = u.z;
          x[t][3 % FS] = u.w;
        } else {
#pragma unroll
          for (int f = 0; f < FS; ++f) {
            const uint32_t hf = h + (uint32_t)f;
            x[t][f] = ok && fs + f < nf
                          ? __ldg(blk + (tile0 + (hf >> kTcTileLg)) * np * (uint64_t)kTcTile +
                                  (hf & (kTcTile - 1u)) + (uint32_t)t * step)
                          : 0u;
          }
        }
      }
#pragma unroll
      for (int f = 0; f < FS; ++f) {
        if (fs + f >= nf) break;
        uint8_t* o = dst + (fs + f) * bytes;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const uint32_t s = (uint32_t)(q + (r >> 1)) & 3u;
          const uint32_t sel = s | ((4u + s) << 4);  // byte s of either word
          uint32_t w[4];
#pragma unroll
          for (int c = 0; c < 4; ++c)
            w[c] = __byte_perm(__byte_perm(x[4 * c][f], x[4 * c + 1][f], sel),
                               __byte_perm(x[4 * c + 2][f], x[4 * c + 3][f], sel), 0x5410);
          *reinterpret_cast<uint4*>(o + 16u * s) = make_uint4(w[0], w[1], w[2], w[3]);
        }
      }
    }
  }
}

// NT threads: 128 where four CTAs share an SM (one warp a TMEM lane
// quadrant), 256 where two do, 512 where one CTA has it to itself.
template <int F, int NT>
__global__ void __launch_bounds__(NT, 512 / NT)
k_contract_tc(const ProdDesc* __restrict__ prods, const TcItem* __restrict__ items,
              uint32_t* __restrict__ res, int bufcols, int* __restrict__ status, int stall) {
  extern __shared__ __align__(1024) uint8_t tsm[];
  __shared__ __align__(8) uint64_t bars[2];
  __shared__ uint32_t tmem_slot;
  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;
  const TcItem it = items[blockIdx.x];
  const ProdDesc d = prods[it.prod];
  // the item's block of C: rows i_base .. + m, columns l_base .. + n (at
  // most kBlock each); m, n below are the block's, d.m, d.n the product's
  const int i_base = (int)(it.pad >> 8) * tc::kBlock, l_base = (int)(it.pad & 0xffu) * tc::kBlock;
  const int m = d.m - i_base < tc::kBlock ? d.m - i_base : tc::kBlock;
  const int n = d.n - l_base < tc::kBlock ? d.n - l_base : tc::kBlock;
  const int k = d.k;
  const int N = 1 << d.lgN;
  const int j = it.prime;
  const uint32_t p = c_primes[j].p;
  const uint32_t pinv = c_primes[j].pinv;
  const uint64_t stride = (uint64_t)d.P * (uint64_t)N;
  const tc::Shape sh = tc::shape_of(m, k, n, F);
  const int phi = sh.phi;
  const int G = F / phi;  // groups of a staged block
  const bool dbl = tc::double_buffered(bufcols);
  const int tmem_cols = dbl ? 2 * bufcols : bufcols;
  const uint32_t ucols = (uint32_t)tc::unit_cols(sh);
  // groups per unit: products with one column range put several groups'
  // accumulators side by side in a TMEM buffer
  const int gf = tc::group_freqs(sh, F, bufcols);
  uint8_t* As = tsm;
  uint8_t* Bs = As + G * sh.a_bytes;
  // results of the staged frequencies, F + 1 words an output entry (odd
  // stride: the epilogue's scattered stores spread over the banks)
  uint32_t* outs = reinterpret_cast<uint32_t*>(Bs + G * sh.b_bytes);
  // this lane's byte plane s of A (rows 4 i + s): its weights 2^(8(s+t)) mod p
  // for planes t = 0 and 2 of B
  const uint32_t wt01 = c_primes[j].w8[lane & 3], wt23 = c_primes[j].w8[(lane & 3) + 2];
  const uint32_t a_base = tc::smem_u32(As), b_base = tc::smem_u32(Bs);
  const uint32_t barp[2] = {tc::smem_u32(&bars[0]), tc::smem_u32(&bars[1])};

  // packed groups: A' is zero outside each slot's K' bytes; the staging
  // writes only inside the slots, so the zeros stay for the whole CTA
  if (phi > 1)
    for (int x = tid; x < G * sh.a_bytes / 16; x += NT)
      reinterpret_cast<uint4*>(As)[x] = make_uint4(0u, 0u, 0u, 0u);
  if (warp == 0) {
    const uint32_t slot = tc::smem_u32(&tmem_slot);
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 :: "r"(slot), "r"((uint32_t)tmem_cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(barp[0]) : "memory");
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(barp[1]) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_slot;
  // commits issued and not yet waited for, and the parity to wait for, per
  // accumulator (the same on every thread)
  uint32_t phase[2] = {0u, 0u};
  int pending[2] = {0, 0};
  bool failed = false;
  const int issue_mma = stall ? 0 : 1;  // stall (failure-path tests only): no MMA, no commit
  // this warp's TMEM lanes 32 qd + lane of every M tile: packed slot fl and
  // first row i (ib0 + 32 q; lane / 4 is added)
  const int qd = warp & 3;
  const int fl = phi > 1 ? (32 * qd) / (4 * sh.mp) : 0;
  const int ib0 = phi > 1 ? ((32 * qd) % (4 * sh.mp)) / 4 : 8 * qd;

  for (int fb0 = 0; fb0 < tc::kFreqs; fb0 += F) {
    const uint32_t hs = it.h0 + (uint32_t)fb0;
    if (hs >= (uint32_t)N) break;  // uniform over the CTA
    const int nf = (int)((uint32_t)N - hs < (uint32_t)F ? (uint32_t)N - hs : (uint32_t)F);
    const uint64_t base = (uint64_t)j * (uint64_t)N + hs;
    // the operands' blocked layout: frequency block of hs, offset inside it
    const uint64_t tile0 = ((uint64_t)j << (d.lgN - kTcTileLg)) + (hs >> kTcTileLg);
    const uint32_t sub0 = hs & (kTcTile - 1u);

    // ---- stage A' and B' of the nf frequencies ----
    if (phi == 1)
      tc_stage_rows<F, NT>(d, sh, m, n, i_base, l_base, tile0, sub0, nf, res, As, Bs);
    else
      tc_stage_packed<F, NT>(d, sh, m, n, i_base, l_base, tile0, sub0, nf, res, As, Bs);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();

    // ---- units: MMAs, then the epilogue of each.  A unit is gf groups
    // (products with one column range) or one frequency's column range uu;
    // its accumulators are consecutive in TMEM ----
    const int ng = (nf + phi - 1) / phi;  // groups holding staged frequencies
    const int U = sh.nunits == 1 ? (ng + gf - 1) / gf : nf * sh.nunits;
    auto unit_groups = [&](int u, int* g0, int* ngu, int* uu) {
      if (sh.nunits == 1) {
        *g0 = u * gf;
        *ngu = (ng - *g0) < gf ? (ng - *g0) : gf;
        *uu = 0;
      } else {
        *g0 = u / sh.nunits;
        *ngu = 1;
        *uu = u - *g0 * sh.nunits;
      }
    };
    auto issue = [&](int u, uint32_t dcol) {
      int g0, ngu, uu;
      unit_groups(u, &g0, &ngu, &uu);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      for (int gi = 0; gi < ngu; ++gi)
        tc_issue_unit(sh, a_base, b_base, (g0 + gi) * sh.nunits + uu,
                      dcol + (uint32_t)gi * ucols);
    };
    // both buffers are free at a block's start (every warp passed the last
    // block's barriers after draining them): units 0 and 1 go at once
    const bool two = dbl && U > 1;
    if (tid == 0 && issue_mma) {
      issue(0, tmem);
      tc_commit(barp[0]);
      if (two) {
        issue(1, tmem + (uint32_t)bufcols);
        tc_commit(barp[1]);
      }
    }
    pending[0] += issue_mma;
    if (two) pending[1] += issue_mma;
    for (int u = 0; u < U; ++u) {
      const int buf = dbl ? (u & 1) : 0;
      // one warp waits for the unit's MMAs; the barrier releases the others
      // and, with two buffers, tells that every warp has drained unit u - 1
      const bool ok = warp == 0 ? tc::mbar_wait(barp[buf], phase[buf]) : true;
      if (__syncthreads_or(!ok)) {  // every thread takes the same branch
        failed = true;
        break;
      }
      phase[buf] ^= 1u;
      pending[buf] -= 1;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (dbl && u >= 1 && u + 1 < U) {  // into unit u - 1's buffer: overlaps this epilogue
        const int nb = (u + 1) & 1;
        if (tid == 0 && issue_mma) {
          issue(u + 1, tmem + (uint32_t)(nb * bufcols));
          tc_commit(barp[nb]);
        }
        pending[nb] += issue_mma;
      }
      int g0, ngu, uu;
      unit_groups(u, &g0, &ngu, &uu);
      const int l0 = uu * sh.npl;
      const int nl = (n - l0) < sh.npl ? (n - l0) : sh.npl;
      const int nch = (nl + 3) / 4;
      const uint32_t laddr = tmem + ((uint32_t)(32 * qd) << 16) + (uint32_t)(buf * bufcols);
      // the warps of quadrant qd share its (group, M tile, 16-column chunk)
      // items; rows i of the quadrant in tile q: ib0 + 32 q + lane / 4
      int gi = 0, q = 0, ch = warp >> 2;
      auto carry = [&] {
        while (ch >= nch) {
          ch -= nch;
          if (++q == sh.mt) {
            q = 0;
            ++gi;
          }
        }
      };
      for (carry(); gi < ngu; ch += NT / 128, carry()) {
        const int f = (g0 + gi) * phi + fl;  // phi = 1 when nunits > 1
        const int ib = ib0 + 32 * q;
        if (fl >= phi || f >= nf || ib >= m) continue;  // warp-uniform: no row here
        uint32_t v[16];
        tmem_ld16(laddr + (uint32_t)(gi * (int)ucols + q * sh.ncol + 16 * ch), v);
        // columns 4 c + t of the chunk: output l0 + 4 ch + c, B plane t
        uint64_t part[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          // planes t in pairs: v < 2^22 (k <= 64), so v_t + 2^8 v_t+1 fits 32 bits
          const uint32_t t01 = v[4 * c] + (v[4 * c + 1] << 8);
          const uint32_t t23 = v[4 * c + 2] + (v[4 * c + 3] << 8);
          part[c] = (uint64_t)t01 * wt01 + (uint64_t)t23 * wt23;
        }
        // add over the four lanes of row i (planes s), lane s ending with
        // output c = s: swap halves across lane bit 1, then across bit 0
        const bool h1 = (lane & 2) != 0, h0 = (lane & 1) != 0;
        uint64_t k0 = h1 ? part[2] : part[0], k1 = h1 ? part[3] : part[1];
        k0 += __shfl_xor_sync(0xffffffffu, h1 ? part[0] : part[2], 2);
        k1 += __shfl_xor_sync(0xffffffffu, h1 ? part[1] : part[3], 2);
        uint64_t z = h0 ? k1 : k0;
        z += __shfl_xor_sync(0xffffffffu, h0 ? k0 : k1, 1);
        const int i = ib + (lane >> 2);
        const int l = 4 * ch + (lane & 3);
        // z 2^-32 mod p in [0, 2p): only the weights 2^32 and 2^40 mod p
        // reach 30 bits, so z < 2^61 + 2^56 < p 2^32; the inverse transform
        // takes values below 2p
        if (i < m && l < nl)
          outs[(i * n + l0 + l) * (F + 1) + f] =
              (uint32_t)((z + (uint64_t)((uint32_t)z * pinv) * p) >> 32);
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      if (!dbl && u + 1 < U) {  // one buffer: the next MMAs wait for every warp
        __syncthreads();
        if (tid == 0 && issue_mma) {
          issue(u + 1, tmem);
          tc_commit(barp[0]);
        }
        pending[0] += issue_mma;
      }
    }
    if (failed) break;
    __syncthreads();  // every epilogue store of the block is in outs
    // ---- the nf frequencies of every output, F residues a vector store.
    // The next block's staging may start at once: this block's MMAs have
    // all completed, and its epilogue writes outs only after its own barrier.
    for (int e = tid; e < m * n; e += NT) {
      const int ei = e / n, el = e - ei * n;  // the block's row and column
      const uint64_t ge = (uint64_t)(i_base + ei) * (uint64_t)d.n + (uint64_t)(l_base + el);
      uint32_t* dst = res + d.c_res + ge * stride + base;
      const uint32_t* sv = outs + e * (F + 1);
      if (nf == F && F >= 4) {
#pragma unroll
        for (int c = 0; c < F / 4; ++c)
          reinterpret_cast<uint4*>(dst)[c] =
              make_uint4(sv[4 * c], sv[4 * c + 1], sv[4 * c + 2], sv[4 * c + 3]);
      } else {
        for (int f = 0; f < nf; ++f) dst[f] = sv[f];
      }
    }
  }
  if (failed) {
    if (tid == 0) atomicExch(status, 1);
    // MMAs already issued must finish before their TMEM is freed
    for (int b = 0; b < 2; ++b)
      while (pending[b] > 0) {
        if (!tc::mbar_wait(barp[b], phase[b])) break;
        phase[b] ^= 1u;
        pending[b] -= 1;
      }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;"
                 :: "r"(tmem), "r"((uint32_t)tmem_cols) : "memory");
}

// ---------------------------------------------------------------------------
// Sizes of operands that live in device memory (results of an earlier plan):
// the planner sized their transforms for a bound; the true signed size and
// coefficient count go into the forward descriptors before the transforms.
// ---------------------------------------------------------------------------
__global__ void k_fix_sizes(FwdDesc* __restrict__ descs, int count,
                            const int32_t* __restrict__ sizes) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  FwdDesc d = descs[i];
  const int32_t sz = sizes[i];
  const uint64_t nl = (uint64_t)(sz < 0 ? -(int64_t)sz : sz);
  const uint64_t nc = (nl * 64 + d.r - 1) / d.r;
  const uint64_t N = (uint64_t)1 << d.lgN;
  descs[i].size = sz;
  descs[i].ncoef = (uint32_t)(nc < N ? nc : N);
}

cudaError_t launch_fix_sizes(FwdDesc* descs, int count, const int32_t* sizes, cudaStream_t st) {
  if (count <= 0) return cudaSuccess;
  k_fix_sizes<<<(count + 255) / 256, 256, 0, st>>>(descs, count, sizes);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Modular reduction r = x mod d (Barrett, HAC 14.42 with B = 2^64): the two
// big products run on the multiplication engine; these kernels shift sizes
// between them and finish each x with one warp.
// ---------------------------------------------------------------------------
// out[i] = max(0, |in[i]| - shift): sizes of operands viewed `shift` limbs up
__global__ void k_shift_sizes(const int32_t* __restrict__ in, int32_t* __restrict__ out,
                              int count, int shift) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const int32_t s = in[i];
  const int32_t a = s < 0 ? -s : s;
  out[i] = a > shift ? a - shift : 0;
}

cudaError_t launch_shift_sizes(const int32_t* in, int32_t* out, int count, int shift,
                               cudaStream_t st) {
  if (count <= 0) return cudaSuccess;
  k_shift_sizes<<<(count + 255) / 256, 256, 0, st>>>(in, out, count, shift);
  return cudaGetLastError();
}

namespace {
// One 32-limb step of a - b - bin over the warp (limb `lane`): returns the
// difference limb; *bstep carries the borrow into the next step.
__device__ __forceinline__ uint64_t warp_sub_step(uint64_t a, uint64_t b, uint32_t* bstep) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  // borrow transfer per limb: out = g | (p & in)
  uint32_t g = a < b ? 1u : 0u, pp = a == b ? 1u : 0u;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t gu = __shfl_up_sync(FULL, g, off), pu = __shfl_up_sync(FULL, pp, off);
    if (lane >= off) {
      g = g | (pp & gu);
      pp = pp & pu;
    }
  }
  const uint32_t out = g | (pp & *bstep);  // borrow out of this limb
  uint32_t in = __shfl_up_sync(FULL, out, 1);
  if (lane == 0) in = *bstep;
  *bstep = __shfl_sync(FULL, out, 31);
  return a - b - (uint64_t)in;
}

// r >= d over limbs [0, nl) (d is zero from limb nd on), warp-wide
__device__ __forceinline__ bool warp_geq(const uint64_t* r, const uint64_t* d, int nl, int nd) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  for (int j0 = ((nl - 1) >> 5) << 5; j0 >= 0; j0 -= 32) {
    const int j = j0 + lane;
    const uint64_t a = j < nl ? r[j] : 0, b = j < nd ? d[j] : 0;
    const unsigned diff = __ballot_sync(FULL, a != b);
    if (diff) {
      const int top = 31 - __clz(diff);
      return __shfl_sync(FULL, a > b ? 1 : 0, top) != 0;
    }
  }
  return true;  // equal
}
}  // namespace

// r_i = x_i mod d in [0, d): r = (|x| - s) mod B^(n+1) with s = q d and q at
// most 2 below floor(|x| / d), then up to two subtractions of d, then d - r
// for a negative x with r != 0.  One warp per x; rbuf holds n + 1 limbs per x.
__global__ void __launch_bounds__(128)
k_mod_finish(int count, int n, const uint64_t* __restrict__ xl, const int64_t* __restrict__ xo,
             const int32_t* __restrict__ xs, const uint64_t* __restrict__ sl, int64_t s_stride,
             const int32_t* __restrict__ ss, const uint64_t* __restrict__ d,
             uint64_t* __restrict__ rbuf, int32_t* __restrict__ rs) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (i >= count) return;  // whole warp
  const int nl = n + 1;
  const int32_t xsz = xs[i];
  const bool neg = xsz < 0;
  const int xa = neg ? -xsz : xsz;
  const int sa = ss[i] < 0 ? -ss[i] : ss[i];
  const uint64_t* x = xl + xo[i];
  const uint64_t* s = sl + (int64_t)i * s_stride;
  uint64_t* r = rbuf + (int64_t)i * nl;
  uint32_t b = 0;
  for (int j0 = 0; j0 < nl; j0 += 32) {  // r = |x| - s mod B^(n+1)
    const int j = j0 + lane;
    const uint64_t a = (j < xa && j < nl) ? x[j] : 0, c = (j < sa && j < nl) ? s[j] : 0;
    const uint64_t v = warp_sub_step(a, c, &b);
    if (j < nl) r[j] = v;
  }
  __syncwarp();
  for (int rep = 0; rep < 2; ++rep) {  // r < 3d: at most two subtractions
    if (!warp_geq(r, d, nl, n)) break;
    b = 0;
    for (int j0 = 0; j0 < nl; j0 += 32) {
      const int j = j0 + lane;
      const uint64_t a = j < nl ? r[j] : 0, c = j < n ? d[j] : 0;
      const uint64_t v = warp_sub_step(a, c, &b);
      if (j < nl) r[j] = v;
    }
    __syncwarp();
  }
  // size, and d - r for a negative x with r != 0
  int top = -1;
  for (int j0 = 0; j0 < nl; j0 += 32) {
    const int j = j0 + lane;
    const unsigned nz = __ballot_sync(FULL, j < nl && r[j] != 0);
    if (nz) top = j0 + 31 - __clz(nz);
  }
  if (neg && top >= 0) {
    b = 0;
    top = -1;
    for (int j0 = 0; j0 < nl; j0 += 32) {
      const int j = j0 + lane;
      const uint64_t a = j < n ? d[j] : 0, c = j < nl ? r[j] : 0;
      const uint64_t v = warp_sub_step(a, c, &b);
      if (j < nl) r[j] = v;
      const unsigned nz = __ballot_sync(FULL, j < nl && v != 0);
      if (nz) top = j0 + 31 - __clz(nz);
    }
  }
  if (lane == 0) rs[i] = top + 1;
}

cudaError_t launch_mod_finish(int count, int n, const uint64_t* xl, const int64_t* xo,
                              const int32_t* xs, const uint64_t* sl, int64_t s_stride,
                              const int32_t* ss, const uint64_t* d, uint64_t* rbuf, int32_t* rs,
                              cudaStream_t st) {
  if (count <= 0) return cudaSuccess;
  k_mod_finish<<<(count + 3) / 4, 128, 0, st>>>(count, n, xl, xo, xs, sl, s_stride, ss, d, rbuf,
                                                rs);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Host launchers
// ---------------------------------------------------------------------------
cudaError_t upload_constants(const PrimeConst* primes, const CrtConst* crt) {
  cudaError_t e = cudaMemcpyToSymbol(c_primes, primes, sizeof(PrimeConst) * kMaxPrimes);
  if (e != cudaSuccess) return e;
  return cudaMemcpyToSymbol(c_crt, crt, sizeof(CrtConst));
}

static int ntt_threads(int lgN) {
  const int half = 1 << (lgN - 1);
  return half < 32 ? 32 : (half > 1024 ? 1024 : half);
}

int fwd_team_points() { return 8 * kFwdThreads; }

#define MPZMM_CTA_SIZES(X) X(12) X(13) X(14) X(15)
#define MPZMM_DIGITS(X) X(1) X(2) X(3) X(4) X(5) X(6) X(7)

// dynamic shared memory of a whole-CTA launch whose CTAs have up to `primes`
static size_t fwd_cta_bytes(int lgN, int primes) {
  return sizeof(uint32_t) * (size_t)pad4(1 << lgN) * (size_t)std::min(primes, cta_primes(lgN));
}
static size_t inv_cta_bytes(int lgN) {
  return sizeof(uint32_t) * (size_t)pad4(1 << lgN) * (lgN == 15 ? 1 : 2);
}

template <int D>
static cudaError_t launch_fwd_d(const FwdDesc* descs, const uint32_t* idx, const CtaItem* items,
                                int nitems, CtaUniform u, int lgN, int primes,
                                const uint64_t* limbs, uint32_t* res, const uint2* twf,
                                cudaStream_t st) {
  switch (lgN) {
#define MPZMM_CASE(L)                                                                           \
  case L:                                                                                       \
    k_fwd_cta<L, D><<<nitems, cta_threads(L), fwd_cta_bytes(L, primes), st>>>(descs, idx,       \
                                                                              items, u, limbs,  \
                                                                              res, twf);        \
    break;
    MPZMM_CTA_SIZES(MPZMM_CASE)
#undef MPZMM_CASE
    default:
      k_fwd_team<D><<<nitems, kFwdThreads, 0, st>>>(descs, idx, items, u, limbs, res, twf);
  }
  return cudaGetLastError();
}

static cudaError_t launch_fwd(const FwdDesc* descs, const uint32_t* idx, const CtaItem* items,
                              int nitems, CtaUniform u, int D, int lgN, int primes,
                              const uint64_t* limbs, uint32_t* res, const uint2* twf,
                              cudaStream_t st) {
  if (nitems == 0) return cudaSuccess;
  switch (D) {
#define MPZMM_CASE(DD) \
  case DD:             \
    return launch_fwd_d<DD>(descs, idx, items, nitems, u, lgN, primes, limbs, res, twf, st);
    MPZMM_DIGITS(MPZMM_CASE)
#undef MPZMM_CASE
    default:
      return cudaErrorInvalidValue;
  }
}

static cudaError_t launch_inv(const InvDesc* descs, const uint32_t* idx, const CtaItem* items,
                              int nitems, CtaUniform u, int lgN, uint32_t* res,
                              const uint2* twi, cudaStream_t st) {
  if (nitems == 0) return cudaSuccess;
  switch (lgN) {
#define MPZMM_CASE(L)                                                                      \
  case L:                                                                                  \
    if (!items)                                                                            \
      return launch_next(k_inv_cta<L>, nitems, cta_threads(L), inv_cta_bytes(L), st, descs, \
                         idx, items, u, res, twi);                                         \
    k_inv_cta<L><<<nitems, cta_threads(L), inv_cta_bytes(L), st>>>(descs, idx, items, u, res, \
                                                                   twi);                   \
    break;
    MPZMM_CTA_SIZES(MPZMM_CASE)
#undef MPZMM_CASE
    default:
      if (!items)
        return launch_next(k_inv_team, nitems, kFwdThreads, 0, st, descs, idx, items, u, res, twi);
      k_inv_team<<<nitems, kFwdThreads, 0, st>>>(descs, idx, items, u, res, twi);
  }
  return cudaGetLastError();
}

cudaError_t launch_fwd_items(const FwdDesc* descs, const uint32_t* idx, const CtaItem* items,
                             int nitems, int D, bool team, int max_lgN, int primes,
                             const uint64_t* limbs, uint32_t* res, const uint2* twf,
                             cudaStream_t st) {
  return launch_fwd(descs, idx, items, nitems, CtaUniform{}, D, team ? 0 : max_lgN, primes, limbs,
                    res, twf, st);
}

cudaError_t launch_inv_items(const InvDesc* descs, const uint32_t* idx, const CtaItem* items,
                             int nitems, bool team, int max_lgN, uint32_t* res,
                             const uint2* twi, cudaStream_t st) {
  return launch_inv(descs, idx, items, nitems, CtaUniform{}, team ? 0 : max_lgN, res, twi, st);
}

// Chunks of primes a transform's CTAs take each, when there are `ctas`
// whole ones: one while those give every SM two, else as many as do.
int prime_chunks(uint64_t ctas, int P, int sms) {
  const uint64_t want = 2 * (uint64_t)(sms > 0 ? sms : 1);
  if (ctas == 0 || ctas >= want) return 1;
  return (int)std::min<uint64_t>((uint64_t)P, (want + ctas - 1) / ctas);
}

// entries 0 .. total - 1 alike: CTAs of `per`, their primes in chunks
static CtaUniform cta_uniform(uint32_t total, int lgN, int P, int sms, int* nitems, int* primes) {
  CtaUniform u;
  u.total = total;
  u.per = (uint32_t)std::max(1, fwd_team_points() >> lgN);
  u.lgN = lgN;
  u.P = P;
  const uint32_t ctas = (total + u.per - 1) / u.per;
  u.chunks = (uint32_t)prime_chunks(ctas, P, sms);
  *nitems = (int)(ctas * u.chunks);
  *primes = (P + (int)u.chunks - 1) / (int)u.chunks;
  return u;
}

cudaError_t launch_fwd_uniform(const FwdDesc* descs, uint32_t total, int lgN, int P, int D,
                               int sms, const uint64_t* limbs, uint32_t* res, const uint2* twf,
                               cudaStream_t st) {
  if (total == 0) return cudaSuccess;
  if (lgN < 3) return launch_split_fwd(descs, nullptr, (int)total, P, lgN, limbs, res, twf, st);
  int nitems, primes;
  const CtaUniform u = cta_uniform(total, lgN, P, sms, &nitems, &primes);
  return launch_fwd(descs, nullptr, nullptr, nitems, u, D, lgN, primes, limbs, res, twf, st);
}

cudaError_t launch_inv_uniform(const InvDesc* descs, uint32_t total, int lgN, int P, int sms,
                               uint32_t* res, const uint2* twi, cudaStream_t st) {
  if (total == 0) return cudaSuccess;
  if (lgN < 3) return launch_inv_ntt(descs, nullptr, (int)total, P, lgN, res, twi, st);
  int nitems, primes;
  const CtaUniform u = cta_uniform(total, lgN, P, sms, &nitems, &primes);
  return launch_inv(descs, nullptr, nullptr, nitems, u, lgN, res, twi, st);
}

// shared memory of a column tile of the four-step kernels
static size_t col_tile_bytes() { return sizeof(uint32_t) * (size_t)(kColPoints + (kColPoints >> 5)); }

template <int D>
static void launch_fwd_cols_d(dim3 grid, cudaStream_t st, const FwdDesc* descs, const uint32_t* idx,
                              int tiles, const uint64_t* limbs, uint32_t* res, const uint2* twf,
                              const TwistTab& tt) {
  k_fwd_cols<D><<<grid, kFwdThreads, col_tile_bytes(), st>>>(descs, idx, tiles, limbs, res, twf,
                                                             tt);
}

int large_tiles(int lgN) { return 1 << (lgN - kLargeLgC + 1); }

cudaError_t launch_large_fwd(const FwdDesc* descs, const uint32_t* idx, int count, int lgN, int P,
                             int D, int sms, const uint64_t* limbs, uint32_t* res, const uint2* twf,
                             const TwistTab& tt, cudaStream_t st) {
  if (count == 0) return cudaSuccess;
  if (lgN <= kMaxLgNOneCta || lgN > kMaxLgN) return cudaErrorInvalidValue;
  const int tiles = large_tiles(lgN);
  const int blocks = 1 << (lgN - kLargeLgC);
  const dim3 grid(count * tiles, prime_chunks((uint64_t)count * tiles, P, sms));
  switch (D) {
    case 1: launch_fwd_cols_d<1>(grid, st, descs, idx, tiles, limbs, res, twf, tt); break;
    case 2: launch_fwd_cols_d<2>(grid, st, descs, idx, tiles, limbs, res, twf, tt); break;
    case 3: launch_fwd_cols_d<3>(grid, st, descs, idx, tiles, limbs, res, twf, tt); break;
    case 4: launch_fwd_cols_d<4>(grid, st, descs, idx, tiles, limbs, res, twf, tt); break;
    case 5: launch_fwd_cols_d<5>(grid, st, descs, idx, tiles, limbs, res, twf, tt); break;
    case 6: launch_fwd_cols_d<6>(grid, st, descs, idx, tiles, limbs, res, twf, tt); break;
    case 7: launch_fwd_cols_d<7>(grid, st, descs, idx, tiles, limbs, res, twf, tt); break;
    default: return cudaErrorInvalidValue;
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  const dim3 bgrid(count * blocks, prime_chunks((uint64_t)count * blocks, P, sms));
  k_ntt_blocks<true><<<bgrid, kBlockThreads, 0, st>>>(descs, nullptr, idx, blocks, res, twf, tt);
  return cudaGetLastError();
}

cudaError_t launch_large_inv(const InvDesc* descs, const uint32_t* idx, int count, int lgN, int P,
                             int sms, uint32_t* res, const uint2* twi, const TwistTab& tt,
                             cudaStream_t st) {
  if (count == 0) return cudaSuccess;
  if (lgN <= kMaxLgNOneCta || lgN > kMaxLgN) return cudaErrorInvalidValue;
  const int tiles = large_tiles(lgN);
  const int blocks = 1 << (lgN - kLargeLgC);
  const dim3 bgrid(count * blocks, prime_chunks((uint64_t)count * blocks, P, sms));
  k_ntt_blocks<false><<<bgrid, kBlockThreads, 0, st>>>(nullptr, descs, idx, blocks, res, twi, tt);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  const dim3 grid(count * tiles, prime_chunks((uint64_t)count * tiles, P, sms));
  k_inv_cols<<<grid, kFwdThreads, col_tile_bytes(), st>>>(descs, idx, tiles, res, twi);
  return cudaGetLastError();
}

cudaError_t launch_split_fwd(const FwdDesc* descs, const uint32_t* idx, int count, int P,
                             int lgN, const uint64_t* limbs, uint32_t* res,
                             const uint2* twf, cudaStream_t st) {
  if (count == 0) return cudaSuccess;
  const size_t smem = sizeof(uint32_t) << lgN;
  dim3 grid(count, P);
  k_split_fwd<<<grid, ntt_threads(lgN), smem, st>>>(descs, idx, limbs, res, twf);
  return cudaGetLastError();
}

cudaError_t launch_inv_ntt(const InvDesc* descs, const uint32_t* idx, int count, int P,
                           int lgN, uint32_t* res, const uint2* twi, cudaStream_t st) {
  if (count == 0) return cudaSuccess;
  const size_t smem = sizeof(uint32_t) << lgN;
  dim3 grid(count, P);
  k_inv_ntt<<<grid, ntt_threads(lgN), smem, st>>>(descs, idx, res, twi);
  return cudaGetLastError();
}

cudaError_t launch_contract(const ProdDesc* prods, const ContractItem* items, int count,
                            uint32_t* res, cudaStream_t st) {
  if (count == 0) return cudaSuccess;
  k_contract<<<count, kContractThreads, 0, st>>>(prods, items, ContractUniform{}, res);
  return cudaGetLastError();
}

// Tiles of product d, and the blocks of positions of its polynomials.
static uint32_t contract_tiles_of(const ProdDesc& d) {
  const uint32_t ti = d.pad / 4 + 1u, tj = d.pad % 4 + 1u;
  return ((d.m + ti - 1) / ti) * ((d.n + tj - 1) / tj);
}
static uint32_t contract_blocks_of(const ProdDesc& d) {
  return (((uint32_t)d.P << d.lgN) + kContractThreads - 1) / kContractThreads;
}

// Tiles a CTA takes where the launches that run beside one another have
// `work` tiles (over all blocks of positions): one while that is below eight
// times the CTAs that run at once (six an SM), more as it grows.
static uint32_t contract_per(uint64_t work, int sms) {
  const uint64_t per = work / ((uint64_t)(sms > 0 ? sms : 1) * 24);
  return per < 1 ? 1u : (uint32_t)std::min<uint64_t>(per, 0xffffffffu);
}

void contract_items(const ProdDesc* prods, const std::vector<uint32_t>& which, int sms,
                    double beside, std::vector<ContractItem>* items) {
  uint64_t work = 0;
  for (const uint32_t q : which)
    work += (uint64_t)contract_tiles_of(prods[q]) * contract_blocks_of(prods[q]);
  const uint32_t per = contract_per((uint64_t)((double)work * beside), sms);
  for (const uint32_t q : which) {
    const uint32_t tiles = contract_tiles_of(prods[q]), nb = contract_blocks_of(prods[q]);
    // equal groups: no short one at the end
    const uint32_t groups = (tiles + per - 1) / per, each = (tiles + groups - 1) / groups;
    for (uint32_t b = 0; b < nb; ++b)
      for (uint32_t t = 0; t < tiles; t += each)
        items->push_back(ContractItem{q, b * (uint32_t)kContractThreads, t,
                                      std::min(each, tiles - t)});
  }
}

cudaError_t launch_contract_one(const ProdDesc* prod, const ProdDesc& d, int sms, uint32_t* res,
                                cudaStream_t st) {
  ContractUniform u;
  u.blocks = contract_blocks_of(d);
  u.tiles = contract_tiles_of(d);
  u.per = std::min(u.tiles, contract_per((uint64_t)u.tiles * u.blocks, sms));
  const uint32_t groups = (u.tiles + u.per - 1) / u.per;
  return launch_next(k_contract, (int)(groups * u.blocks), kContractThreads, 0, st, prod,
                     (const ContractItem*)nullptr, u, res);
}

__device__ __forceinline__ bool fwd_in_bounds(const FwdDesc& f, const BoundsCaps& c) {
  if (f.lgN > kMaxLgN || f.P > kMaxPrimes) return false;
  const uint64_t nl = f.size < 0 ? (uint64_t)(-(int64_t)f.size) : (uint64_t)f.size;
  if (f.limb_off + nl > c.limbs) return false;
  if (f.tile_np && f.tile_e >= f.tile_np) return false;
  // the plain layout: P polynomials of N words; blocked: the operand's block
  const uint64_t words = ((uint64_t)f.P << f.lgN) * (f.tile_np ? f.tile_np : 1u);
  return f.res_off + words <= c.res;
}

__device__ __forceinline__ bool inv_in_bounds(const InvDesc& v, const BoundsCaps& c) {
  if (v.lgN > kMaxLgN || v.P > kMaxPrimes) return false;
  return v.res_off + ((uint64_t)v.P << v.lgN) <= c.res &&
         v.out_word + v.out_words <= c.out_words && v.entry < c.sizes;
}

__device__ __forceinline__ bool prod_in_bounds(const ProdDesc& d, const BoundsCaps& c) {
  if (d.lgN > kMaxLgN || d.P > kMaxPrimes) return false;
  const uint64_t poly = (uint64_t)d.P << d.lgN;
  return d.a_res + (uint64_t)d.m * d.k * poly <= c.res &&
         d.b_res + (uint64_t)d.k * d.n * poly <= c.res &&
         d.c_res + (uint64_t)d.m * d.n * poly <= c.res;
}

__global__ void k_check_bounds(const FwdDesc* __restrict__ fwd, int nfwd,
                               const InvDesc* __restrict__ inv, int ninv,
                               const ProdDesc* __restrict__ prods, int nprods, BoundsCaps caps,
                               int* __restrict__ status) {
  const int total = nfwd + ninv + nprods;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const bool ok = i < nfwd          ? fwd_in_bounds(fwd[i], caps)
                    : i < nfwd + ninv ? inv_in_bounds(inv[i - nfwd], caps)
                                      : prod_in_bounds(prods[i - nfwd - ninv], caps);
    if (!ok) atomicExch(status, 2);
  }
}

cudaError_t launch_check_bounds(const FwdDesc* fwd, int nfwd, const InvDesc* inv, int ninv,
                                const ProdDesc* prods, int nprods, BoundsCaps caps, int* status,
                                cudaStream_t st) {
  const int total = nfwd + ninv + nprods;
  if (total <= 0) return cudaSuccess;
  const int blocks = (total + 255) / 256 < 1184 ? (total + 255) / 256 : 1184;
  k_check_bounds<<<blocks, 256, 0, st>>>(fwd, nfwd, inv, ninv, prods, nprods, caps, status);
  return cudaGetLastError();
}

bool contract_tc_eligible(int m, int k, int n) {
  return m >= 1 && m <= tc::kMaxM && k >= 1 && k <= tc::kMaxK && n >= 1 && n <= tc::kMaxN;
}

// Dynamic shared memory of one product's CTA with F frequencies staged: the
// byte tiles of A' and B' and the results of the F frequencies.
int tc_smem_bytes(int m, int k, int n, int F) {
  const tc::Shape sh = tc::shape_of(m, k, n, F);
  return (F / sh.phi) * (sh.a_bytes + sh.b_bytes) + ((m * n * (F + 1) * 4 + 15) & ~15);
}

// Accumulator buffer width, frequencies staged at once (F), dynamic shared
// memory and threads of a launch over products of the given shapes.  The
// buffer is the widest accumulator rounded up to a power of two, at least
// the floor below; CTAs share an SM as far as TMEM allows (four of 128
// threads, two of 256, or one of 512), and F is the largest whose shared
// memory lets them, else the launch takes fewer CTAs an SM.
static bool tc_launch_config(const int* shapes, int nshapes, int* bufcols, int* F, int* smem,
                             int* threads) {
  int widest = 0;
  for (int i = 0; i < nshapes; ++i) {
    // the accumulator width does not depend on F
    const int c =
        tc::unit_cols(tc::shape_of(shapes[3 * i], shapes[3 * i + 1], shapes[3 * i + 2], 1));
    if (c > widest) widest = c;
  }
  // The narrowest buffer is 64 columns, so four double-buffered CTAs of
  // 128 threads share an SM and overlap one another's staging, MMA round
  // trips and barriers: 4096 products of 2..16 rows and columns forced onto
  // the tensor cores contracted in 74 ms that way, 107 ms with 128 columns
  // (two CTAs of 256 threads an SM).  MPZMM_TC_BUFCOLS (a power of two from
  // 32 to 256) replaces that floor for tuning.
  static const int b_floor = [] {
    const char* e = std::getenv("MPZMM_TC_BUFCOLS");
    const int v = e ? std::atoi(e) : 0;
    return (v >= 32 && v <= 256 && (v & (v - 1)) == 0) ? v : 64;
  }();
  int b = b_floor;
  while (b < widest) b <<= 1;
  *bufcols = b;
  const int tcols = tc::double_buffered(b) ? 2 * b : b;
  const int per_sm = 512 / tcols >= 4 ? 4 : (512 / tcols >= 2 ? 2 : 1);
  for (int target = per_sm; target >= 1; target >>= 1) {
    const int limit = target == 1 ? tc::kDynSmemLimit
                                  : (tc::kSmemLimit / target) - tc::kStaticSmem - 1024;
    for (int f = 16; f >= 1; f >>= 1) {
      int bytes = 0;
      for (int i = 0; i < nshapes; ++i) {
        const int sb = tc_smem_bytes(shapes[3 * i], shapes[3 * i + 1], shapes[3 * i + 2], f);
        if (sb > bytes) bytes = sb;
      }
      // below four staged frequencies a shared SM is not worth the loss
      if (bytes <= limit && (target == 1 || f >= 4)) {
        *F = f;
        *smem = bytes;
        *threads = 512 / target;  // as many threads an SM either way
        return true;
      }
    }
  }
  return false;
}

template <int F>
static void launch_tc_f(int count, int smem, int threads, cudaStream_t st,
                        const ProdDesc* prods, const TcItem* items, uint32_t* res,
                        int bufcols, int* status, int stall) {
  if (threads == 512)
    k_contract_tc<F, 512><<<count, 512, smem, st>>>(prods, items, res, bufcols, status, stall);
  else if (threads == 256)
    k_contract_tc<F, 256><<<count, 256, smem, st>>>(prods, items, res, bufcols, status, stall);
  else
    k_contract_tc<F, 128><<<count, 128, smem, st>>>(prods, items, res, bufcols, status, stall);
}

cudaError_t launch_contract_tc(const ProdDesc* prods, const TcItem* items, int count,
                               uint32_t* res, const int* shapes, int nshapes, int* status,
                               cudaStream_t st, int stall) {
  if (count == 0) return cudaSuccess;
  for (int i = 0; i < nshapes; ++i)
    if (!contract_tc_eligible(shapes[3 * i], shapes[3 * i + 1], shapes[3 * i + 2]))
      return cudaErrorInvalidValue;
  int F = 0, smem = 0, bufcols = 0, threads = 0;
  if (!tc_launch_config(shapes, nshapes, &bufcols, &F, &smem, &threads))
    return cudaErrorInvalidValue;
  switch (F) {
    case 16: launch_tc_f<16>(count, smem, threads, st, prods, items, res, bufcols, status, stall); break;
    case 8: launch_tc_f<8>(count, smem, threads, st, prods, items, res, bufcols, status, stall); break;
    case 4: launch_tc_f<4>(count, smem, threads, st, prods, items, res, bufcols, status, stall); break;
    case 2: launch_tc_f<2>(count, smem, threads, st, prods, items, res, bufcols, status, stall); break;
    default: launch_tc_f<1>(count, smem, threads, st, prods, items, res, bufcols, status, stall); break;
  }
  return cudaGetLastError();
}

static_assert(kTcFreqs == tc::kFreqs, "work items are cut to the kernel's blocks");

// coefficients a CRT tile can touch for coefficient width rmin
static int crt_cmax(int P, int rmin) {
  return (int)((32 * (int64_t)kCrtTileWords + 32 * P) / rmin + 3);
}

// Words a warp takes of an entry when a launch writes total_words words: as
// many as leave every SM kCrtSegWarps warps (a few waves of them, so that no
// long entry is the launch's tail), in whole tiles less the 32 words of the
// look below a segment.
constexpr int kCrtSegWarps = 128;
static int crt_segment_words(uint64_t total_words, int sms) {
  const uint64_t t = total_words / ((uint64_t)(sms > 0 ? sms : 1) * kCrtSegWarps);
  const uint64_t tiles = (t + 32 + kCrtTileWords - 1) / kCrtTileWords;
  return (int)((tiles < 1 ? 1 : tiles) * kCrtTileWords) - 32;
}

// Segments of an entry of W words, each *step words but the last.  The look
// and the second launch cost a segment about 40 words' time, so an entry of
// up to two segments stays whole, and where a warp an entry fills the SMs
// only entries well above the others are split (4096 entries of 2050 words
// took 121 us whole, 140 in five segments; 2000 of 630 words 33 and 38; 256
// mixed products 940 us with the long entries split, 1030 without; 512 of
// them 1763 whole, 1835 with entries above four segments split).
//
// Both questions are about what is on the GPU, not about one launch: the
// chunks of a batch overlap one another, so their entries are counted
// together.  Asked of each chunk alone, 19 of the 33 launches of 512 mixed
// products in 17 chunks were few and cut 350,000 segments, whose lists the
// host built and the link carried: 11 ms of planning and 559.4 MB to the
// device, against 7 ms and 550.0 MB.
//
// But a chunk waits for its longest entry: one of kCrtLong words takes a warp
// 0.6 ms, as long as a chunk of 32 MB takes on the link, and few chunks are
// in flight.  Longer ones are judged by at most kCrtBeside chunks' work: 1000
// 2 x 2 x 2 products of 2^20 bits host to host 30.8 ms so, 37.2 by the whole
// batch, 31.3 by each chunk; 512 mixed products 15.4 by the batch, 15.7 by
// four chunks' work, 16.1 by each chunk.
constexpr uint32_t kCrtShort = 16 * kCrtTileWords;
constexpr uint32_t kCrtLong = 28 * 1024;
constexpr double kCrtBeside = 8.0;
static uint32_t crt_split(uint32_t W, uint32_t seg, bool few, uint32_t* step) {
  const bool split = few ? W > 2 * seg : W > kCrtShort && W > 6 * seg;
  uint32_t ns = split ? (W + seg - 1) / seg : 1u;
  *step = (((W + ns - 1) / ns) + 31) & ~31u;
  return ns > 1 ? (W + *step - 1) / *step : 1u;
}
static bool crt_few(uint64_t count, int sms) { return count < 8 * (uint64_t)sms; }

CrtUniform crt_uniform(uint32_t words, uint32_t count, int sms, uint64_t max_recs) {
  CrtUniform u;
  u.words = words;
  u.nseg = crt_split(words, (uint32_t)crt_segment_words((uint64_t)words * count, sms),
                     crt_few(count, sms), &u.step);
  if ((uint64_t)u.nseg * count > max_recs) u.nseg = 1;
  return u;
}

void crt_items(const InvDesc* descs, std::vector<uint32_t>* idx, int sms, double beside,
               uint32_t* nrecs, std::vector<CrtItem>* segs) {
  // by prime count, most first (each count is code of its own, and warps that
  // run side by side share the instruction cache: 1870 -> 1800 us for the
  // first 512 products of the default batch), then longest first (the warp
  // that gets one works longest), ties in entry order: one sort of packed
  // integers, which the entries of a single product need not
  std::vector<uint64_t> keys(idx->size());
  uint64_t total = 0;
  for (size_t i = 0; i < keys.size(); ++i) {
    const uint32_t W = descs[(*idx)[i]].out_words;
    total += W;
    keys[i] = ((uint64_t)(kMaxPrimes - descs[(*idx)[i]].P) << 59) | ((uint64_t)(0x7ffffffu - W) << 32) |
              (*idx)[i];
  }
  if (!std::is_sorted(keys.begin(), keys.end())) std::sort(keys.begin(), keys.end());
  const auto segment = [&](double times) {
    return (uint32_t)crt_segment_words((uint64_t)((double)total * times), sms);
  };
  const auto are_few = [&](double times) {
    return crt_few((uint64_t)((double)keys.size() * times), sms);
  };
  const double flight = std::min(beside, kCrtBeside);
  const uint32_t seg = segment(beside), seg_long = segment(flight);
  const bool few = are_few(beside), few_long = are_few(flight);
  idx->clear();
  for (const uint64_t key : keys) {
    const uint32_t e = (uint32_t)key, W = descs[e].out_words;
    uint32_t step;
    const uint32_t ns = W > kCrtLong ? crt_split(W, seg_long, few_long, &step)
                                     : crt_split(W, seg, few, &step);
    if (ns == 1) {
      idx->push_back(e);
      continue;
    }
    for (uint32_t s = 0; s < ns; ++s)
      segs->push_back(CrtItem{e, s * step, s + 1 < ns ? (s + 1) * step : W, *nrecs, s, ns});
    *nrecs += ns;
  }
}

// The product alone: every list is cut finest there, since each rule takes
// larger pieces as the launches' work grows.
int64_t cut_list_bytes(const ProdDesc& d, uint32_t words, int sms) {
  const int64_t entries = (int64_t)d.m * d.n, operands = (int64_t)(d.m + d.n) * d.k;
  uint32_t step;
  const uint32_t ns =
      crt_split(words, (uint32_t)crt_segment_words((uint64_t)words * entries, sms),
                crt_few((uint64_t)entries, sms), &step);
  int64_t bytes = ns > 1 ? entries * ns * (int64_t)(sizeof(CrtRec) + sizeof(CrtItem)) : 0;
  const uint32_t tiles = contract_tiles_of(d), nb = contract_blocks_of(d);
  const uint32_t per = contract_per((uint64_t)tiles * nb, sms);
  int64_t contract = (int64_t)((tiles + per - 1) / per) * nb * (int64_t)sizeof(ContractItem);
  if (contract_tc_eligible(d.m, d.k, d.n)) {
    const int64_t blocks = (int64_t)((d.m + tc::kBlock - 1) / tc::kBlock) *
                           ((d.n + tc::kBlock - 1) / tc::kBlock);
    const int64_t freqs = ((int64_t)1 << d.lgN) / tc::kFreqs + 1;
    contract = std::max(contract, blocks * freqs * d.P * (int64_t)sizeof(TcItem));
  }
  bytes += contract;
  if (d.lgN > kMaxLgNOneCta) return bytes;
  const int64_t per_cta = std::max(1, fwd_team_points() >> d.lgN);
  for (const int64_t n : {operands, entries}) {
    const int64_t ctas = (n + per_cta - 1) / per_cta;
    bytes += ctas * prime_chunks((uint64_t)ctas, d.P, sms) * (int64_t)sizeof(CtaItem);
  }
  return bytes;
}

template <int PLO, int PHI>
static cudaError_t launch_crt(const InvDesc* descs, const CrtItem* segs, int nsegs,
                              const uint32_t* idx, int count, CrtUniform u, int warp_words,
                              const uint32_t* res, uint32_t* out, int32_t* sizes, CrtRec* recs,
                              cudaStream_t st) {
  const size_t smem = sizeof(uint32_t) * (size_t)warp_words * kCrtWarps;
  if (smem == 0 || smem > kCrtSmemLimit) return cudaErrorInvalidValue;
  constexpr int NT = 32 * kCrtWarps;
  const int gs = (nsegs + kCrtWarps - 1) / kCrtWarps, gw = (count + kCrtWarps - 1) / kCrtWarps;
  if (!segs && !idx) {  // entries all alike
    const CrtItem* no_items = nullptr;
    if (nsegs == 0)
      return launch_next(k_crt_mixed<PLO, PHI, false>, gw, NT, smem, st, descs, no_items, idx,
                         count, u, res, out, sizes, recs, warp_words);
    const cudaError_t e = launch_next(k_crt_mixed<PLO, PHI, true>, gs, NT, smem, st, descs,
                                      no_items, idx, nsegs, u, res, out, sizes, recs, warp_words);
    if (e != cudaSuccess) return e;
    return launch_next(k_crt_finish, gs, NT, 0, st, descs, no_items, nsegs, u, recs, out, sizes);
  }
  if (nsegs > 0) {
    k_crt_mixed<PLO, PHI, true><<<gs, NT, smem, st>>>(descs, segs, nullptr, nsegs, u, res, out,
                                                      sizes, recs, warp_words);
    k_crt_finish<<<gs, NT, 0, st>>>(descs, segs, nsegs, u, recs, out, sizes);
  }
  if (count > 0)
    k_crt_mixed<PLO, PHI, false><<<gw, NT, smem, st>>>(descs, nullptr, idx, count, u, res, out,
                                                       sizes, recs, warp_words);
  return cudaGetLastError();
}

cudaError_t launch_crt_mixed(const InvDesc* descs, const CrtItem* segs, int nsegs,
                             const uint32_t* idx, int count, bool high, const int* rmin,
                             const uint32_t* res, uint32_t* out, int32_t* sizes, CrtRec* recs,
                             cudaStream_t st) {
  const int plo = high ? kCrtMixedSplit + 1 : 2, phi = high ? kMaxPrimes : kCrtMixedSplit;
  int words = 0;
  for (int P = plo; P <= phi; ++P)
    if (rmin[P] > 0) words = std::max(words, crt_cmax(P, rmin[P]) * ((P + 1) | 1));
  const auto fn = high ? launch_crt<kCrtMixedSplit + 1, kMaxPrimes> : launch_crt<2, kCrtMixedSplit>;
  return fn(descs, segs, nsegs, idx, count, CrtUniform{}, words, res, out, sizes, recs, st);
}

cudaError_t launch_crt_uniform(const InvDesc* descs, int count, CrtUniform u, int P, int r,
                               const uint32_t* res, uint32_t* out, int32_t* sizes, CrtRec* recs,
                               cudaStream_t st) {
  const bool seg = u.nseg > 1;
  const auto fn = P > kCrtMixedSplit ? launch_crt<kCrtMixedSplit + 1, kMaxPrimes>
                                     : launch_crt<2, kCrtMixedSplit>;
  return fn(descs, nullptr, seg ? count * (int)u.nseg : 0, nullptr, seg ? 0 : count, u,
            crt_cmax(P, r) * ((P + 1) | 1), res, out, sizes, recs, st);
}

// Dynamic shared memory limits of every kernel, set once per device at
// set-up (so that launches, including those captured into a CUDA graph,
// issue nothing but stream work).
template <class K>
static cudaError_t allow_smem(K kernel, size_t bytes) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

cudaError_t init_kernel_attributes() {
  cudaError_t e;
  if ((e = allow_smem(k_split_fwd, sizeof(uint32_t) << kMaxLgNOneCta)) != cudaSuccess ||
      (e = allow_smem(k_inv_ntt, sizeof(uint32_t) << kMaxLgNOneCta)) != cudaSuccess)
    return e;
#define MPZMM_FWD(L, D) \
  if ((e = allow_smem(k_fwd_cta<L, D>, fwd_cta_bytes(L, kMaxPrimes))) != cudaSuccess) return e;
#define MPZMM_CASE(L)                                                                 \
  if ((e = allow_smem(k_inv_cta<L>, inv_cta_bytes(L))) != cudaSuccess) return e;      \
  MPZMM_FWD(L, 1) MPZMM_FWD(L, 2) MPZMM_FWD(L, 3) MPZMM_FWD(L, 4) MPZMM_FWD(L, 5)     \
  MPZMM_FWD(L, 6) MPZMM_FWD(L, 7)
  MPZMM_CTA_SIZES(MPZMM_CASE)
#undef MPZMM_CASE
#undef MPZMM_FWD
  for (auto fn : {k_crt_mixed<2, kCrtMixedSplit, false>, k_crt_mixed<2, kCrtMixedSplit, true>,
                  k_crt_mixed<kCrtMixedSplit + 1, kMaxPrimes, false>,
                  k_crt_mixed<kCrtMixedSplit + 1, kMaxPrimes, true>})
    if ((e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)kCrtSmemLimit)) != cudaSuccess)
      return e;
  for (auto fn : {k_contract_tc<16, 128>, k_contract_tc<8, 128>, k_contract_tc<4, 128>,
                  k_contract_tc<2, 128>, k_contract_tc<1, 128>, k_contract_tc<16, 256>,
                  k_contract_tc<8, 256>, k_contract_tc<4, 256>, k_contract_tc<2, 256>,
                  k_contract_tc<1, 256>, k_contract_tc<16, 512>, k_contract_tc<8, 512>,
                  k_contract_tc<4, 512>, k_contract_tc<2, 512>, k_contract_tc<1, 512>})
    if ((e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  tc::kDynSmemLimit)) != cudaSuccess)
      return e;
  return cudaSuccess;
}

}  // namespace mpzmm
