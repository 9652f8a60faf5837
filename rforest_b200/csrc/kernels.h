// Host-side launchers of the sm_100a kernels (kernels.cu).
#pragma once

#include <cuda_runtime.h>

#include <vector>

#include "mpzmm_internal.h"

namespace mpzmm {

cudaError_t upload_constants(const PrimeConst* primes, const CrtConst* crt);
// Sets every kernel's dynamic shared-memory limit on the current device.
cudaError_t init_kernel_attributes();

// Radix-2 split + forward NTT / inverse NTT, one CTA per (entry, prime),
// for `count` entries of one class (any lgN >= 1; used for lgN < 3); idx ==
// nullptr: entries 0, 1, ...
cudaError_t launch_split_fwd(const FwdDesc* descs, const uint32_t* idx, int count, int P,
                             int lgN, const uint64_t* limbs, uint32_t* res,
                             const uint2* twf, cudaStream_t st);
cudaError_t launch_inv_ntt(const InvDesc* descs, const uint32_t* idx, int count, int P,
                           int lgN, uint32_t* res, const uint2* twi, cudaStream_t st);

// Register-blocked transforms (lgN >= 3) over CTA work items of mixed size
// classes in ONE launch.  team: every item has 2^lgN <= fwd_team_points()
// (several entries per CTA); otherwise one entry of 2^max_lgN points per CTA,
// with up to `primes` primes.  D = digits of 30 bits of the widest
// coefficient.  Operands of tensor-core products (FwdDesc::tile_np) are
// written in the frequency-blocked layout, others in the plain one.
int fwd_team_points();
cudaError_t launch_fwd_items(const FwdDesc* descs, const uint32_t* idx, const CtaItem* items,
                             int nitems, int D, bool team, int max_lgN, int primes,
                             const uint64_t* limbs, uint32_t* res, const uint2* twf,
                             cudaStream_t st);
cudaError_t launch_inv_items(const InvDesc* descs, const uint32_t* idx, const CtaItem* items,
                             int nitems, bool team, int max_lgN, uint32_t* res,
                             const uint2* twi, cudaStream_t st);
// The same over entries 0 .. total - 1 that are all alike, without lists (any
// lgN up to one CTA's).
cudaError_t launch_fwd_uniform(const FwdDesc* descs, uint32_t total, int lgN, int P, int D,
                               int sms, const uint64_t* limbs, uint32_t* res, const uint2* twf,
                               cudaStream_t st);
cudaError_t launch_inv_uniform(const InvDesc* descs, uint32_t total, int lgN, int P, int sms,
                               uint32_t* res, const uint2* twi, cudaStream_t st);
// Chunks a launch of `ctas` transform CTAs cuts its P primes into.
int prime_chunks(uint64_t ctas, int P, int sms);

// Transforms of 2^16 .. 2^20 points (four-step: column transforms, twist,
// block transforms), `count` entries of one length 2^lgN in one group (idx
// lists their descriptors; nullptr: 0, 1, ...).  Forward: split of D-digit coefficients + the
// transform; inverse: the transform back to natural order, ready for the
// CRT.  Two launches each (P primes, cut into chunks where the CTAs are
// few).  tt: the twist tables of the direction.
cudaError_t launch_large_fwd(const FwdDesc* descs, const uint32_t* idx, int count, int lgN, int P,
                             int D, int sms, const uint64_t* limbs, uint32_t* res, const uint2* twf,
                             const TwistTab& tt, cudaStream_t st);
cudaError_t launch_large_inv(const InvDesc* descs, const uint32_t* idx, int count, int lgN, int P,
                             int sms, uint32_t* res, const uint2* twi, const TwistTab& tt,
                             cudaStream_t st);
constexpr int kLargeLaunches = 2;  // kernel launches per direction of a four-step group

// CUDA-core contraction over `count` work items.
cudaError_t launch_contract(const ProdDesc* prods, const ContractItem* items, int count,
                            uint32_t* res, cudaStream_t st);
// The work of the products `which` (indices into prods), appended to items;
// launches that run beside this one make the work `beside` times as much.
void contract_items(const ProdDesc* prods, const std::vector<uint32_t>& which, int sms,
                    double beside, std::vector<ContractItem>* items);
// One product alone (its descriptor on the device and here), without a list.
cudaError_t launch_contract_one(const ProdDesc* prod, const ProdDesc& d, int sms, uint32_t* res,
                                cudaStream_t st);
// writes the device-held signed sizes (and coefficient counts) of `count`
// forward descriptors
cudaError_t launch_fix_sizes(FwdDesc* descs, int count, const int32_t* sizes, cudaStream_t st);
// modular reduction helpers: sizes of operands viewed `shift` limbs up, and
// the final step of x mod d (see mod.cpp)
cudaError_t launch_shift_sizes(const int32_t* in, int32_t* out, int count, int shift,
                               cudaStream_t st);
cudaError_t launch_mod_finish(int count, int n, const uint64_t* xl, const int64_t* xo,
                              const int32_t* xs, const uint64_t* sl, int64_t s_stride,
                              const int32_t* ss, const uint64_t* d, uint64_t* rbuf, int32_t* rs,
                              cudaStream_t st);

// Debug check (MPZMM_OPT_CHECK_BOUNDS): every forward, inverse and product
// descriptor's extents against the workspace capacities (limbs, residue
// words, output words, result sizes); a thread that finds one outside sets
// *status to 2 and touches nothing else.
struct BoundsCaps {
  uint64_t limbs, res, out_words, sizes;
};
cudaError_t launch_check_bounds(const FwdDesc* fwd, int nfwd, const InvDesc* inv, int ninv,
                                const ProdDesc* prods, int nprods, BoundsCaps caps, int* status,
                                cudaStream_t st);
// Tensor-core contraction (tcgen05 kind::i8) for products with m, n <= 1024
// and k <= 64 (contract_tc_eligible); each work item covers kTcFreqs
// consecutive frequencies of one block of at most kTcBlock rows and columns
// of C; shapes: the launch's distinct blocks (rows, k, columns), nshapes
// triples (they size its shared memory).  *status is set to 1 if a bounded
// wait gave up.  stall != 0 (failure-path tests only) issues no tensor work,
// so every CTA's wait runs out.
bool contract_tc_eligible(int m, int k, int n);
int tc_smem_bytes(int m, int k, int n, int F);
cudaError_t launch_contract_tc(const ProdDesc* prods, const TcItem* items, int count,
                               uint32_t* res, const int* shapes, int nshapes, int* status,
                               cudaStream_t st, int stall = 0);

// CRT + recompose + sign.  crt_items takes the output entries idx and leaves
// in it those that a warp each recomposes whole, by prime count and then
// longest first; entries so long that one warp each would leave the GPU (of
// `sms` SMs) idle go to segs, their records numbered from *nrecs (advanced);
// launches that run beside this one make its entries `beside` times as many.
// launch_crt_mixed runs both lists over several prime counts: high = false
// takes entries with 2..kCrtMixedSplit primes, high = true those with more;
// rmin[P] is the narrowest coefficient width among the entries with P primes
// (0: none; it sizes the scratch).  One kernel for the whole entries, two
// for the segments.
constexpr int kCrtMixedSplit = 10;
void crt_items(const InvDesc* descs, std::vector<uint32_t>* idx, int sms, double beside,
               uint32_t* nrecs, std::vector<CrtItem>* segs);
constexpr int kCrtSegLaunches = 2;
// Most device bytes that the segment records and the work lists of product d
// (out_words words a result) take in any plan.
int64_t cut_list_bytes(const ProdDesc& d, uint32_t out_words, int sms);
cudaError_t launch_crt_mixed(const InvDesc* descs, const CrtItem* segs, int nsegs,
                             const uint32_t* idx, int count, bool high, const int* rmin,
                             const uint32_t* res, uint32_t* out, int32_t* sizes, CrtRec* recs,
                             cudaStream_t st);
// The same over entries 0 .. count - 1 that are all alike (`words` words, P
// primes, r bits a coefficient), without a list: crt_uniform splits them
// (into at most max_recs segments in all).
CrtUniform crt_uniform(uint32_t words, uint32_t count, int sms, uint64_t max_recs);
cudaError_t launch_crt_uniform(const InvDesc* descs, int count, CrtUniform u, int P, int r,
                               const uint32_t* res, uint32_t* out, int32_t* sizes, CrtRec* recs,
                               cudaStream_t st);

}  // namespace mpzmm
