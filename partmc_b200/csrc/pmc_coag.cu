// pmc_coag.cu -- host orchestration and C ABI of the B200 coagulation step.
//
// The C ABI (include/pmc_coag_gpu.h) is the drop-in for mc_coag
// (coagulation.F90:43-96).  A context owns one or more particle
// populations resident in HBM; a step runs the rounds described in
// pmc_kernels.cuh over all populations at once.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <climits>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <memory>
#include <string>
#include <vector>
#include <condition_variable>
#include <functional>
#include <mutex>
#include <thread>
#include <type_traits>

#include "../../include/pmc_coag_gpu.h"
#include "pmc_kernels.cuh"
#include "pmc_merge.cuh"
#include "pmc_replay.cuh"
#include "pmc_sample.cuh"

using namespace pmc;

namespace {

inline void note_launch();

// ---------------------------------------------------------------------------
// exclusive scan of n values into out[0..n] (out[n] = total): one
// single-pass launch with decoupled look-back, for up to kScanMaxJobs arrays
// of the same element type at once (blockIdx.y selects the array)
constexpr int kScanThreads = 512;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;
constexpr int kScanMaxJobs = 4;
constexpr int kScanSpinLimit = 1 << 20;  // bounded wait on a predecessor tile

// the element count is n, or *nd when nd is given (a count that only the
// device knows; n is then its upper bound)
__device__ __forceinline__ long long scan_n(long long n, const long long* nd) {
  if (!nd) return n;
  long long m = *nd;
  return m < n ? m : n;
}

__device__ long long block_excl_scan_ll(long long v, long long* total) {
  __shared__ long long ws[32];
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  long long x = v;
  for (int o = 1; o < 32; o <<= 1) {
    long long y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) ws[wid] = x;
  __syncthreads();
  int nw = (blockDim.x + 31) >> 5;
  if (wid == 0) {
    long long s = lane < nw ? ws[lane] : 0;
    for (int o = 1; o < 32; o <<= 1) {
      long long y = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += y;
    }
    ws[lane] = s;
  }
  __syncthreads();
  long long pre = (wid > 0 ? ws[wid - 1] : 0) + x - v;
  if (total) *total = ws[nw - 1];
  __syncthreads();
  return pre;
}

struct ScanJob {
  const void* in;
  long long* out;
  long long n_max;
  const long long* nd;
  long long* total_out;  // optional second copy of the total at a fixed address
};
struct ScanJobs {
  ScanJob j[kScanMaxJobs];
};

// tile status word: flag (2 bits: 1 aggregate, 2 inclusive prefix) | value
// (62 bits); 0 = not published.  The last block of a launch to finish
// clears the launch's words, so the array is all zero between launches and
// a launch can be replayed (CUDA graphs) without host bookkeeping.
__device__ __forceinline__ unsigned long long scan_word(unsigned flag, long long v) {
  return ((unsigned long long)flag << 62) | ((unsigned long long)v & ((1ULL << 62) - 1));
}

template <class T>
__global__ void __launch_bounds__(kScanThreads) k_scan_lb(ScanJobs jobs, unsigned long long* status,
                                                          int status_stride, unsigned* tile_ctr,
                                                          unsigned* done_ctr, unsigned long long* err) {
  chain_wait();
  const ScanJob J = jobs.j[blockIdx.y];
  __shared__ unsigned tile_sh;
  __shared__ long long carry_sh;
  unsigned long long* st = status + (size_t)blockIdx.y * status_stride;
  if (threadIdx.x == 0) {
    // tiles in the order blocks start, so a tile only waits on running blocks
    unsigned t = atomicAdd(&tile_ctr[blockIdx.y], 1u);
    if (t == gridDim.x - 1) tile_ctr[blockIdx.y] = 0;  // the last claimant re-arms the counter
    tile_sh = t;
  }
  __syncthreads();
  long long tile = tile_sh;
  long long n = scan_n(J.n_max, J.nd);
  long long nb = (n + kScanTile - 1) / kScanTile;
  if (n <= 0) {
    if (tile == 0 && threadIdx.x == 0) {
      J.out[0] = 0;
      if (J.total_out) *J.total_out = 0;
    }
  } else if (tile < nb) {
    const T* in = (const T*)J.in;
    long long base = tile * kScanTile + (long long)threadIdx.x * kScanItems;
    long long v[kScanItems];
    long long s = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
      long long i = base + k;
      v[k] = i < n ? (long long)in[i] : 0;
      s += v[k];
    }
    long long agg;
    long long pre = block_excl_scan_ll(s, &agg);
    if (threadIdx.x == 0) {
      long long excl = 0;
      if (tile == 0) {
        atomicExch(&st[0], scan_word(2u, agg));
      } else {
        atomicExch(&st[tile], scan_word(1u, agg));
        long long look = tile - 1;
        int spins = 0;
        while (look >= 0) {
          unsigned long long w = *(volatile unsigned long long*)&st[look];
          unsigned flag = (unsigned)(w >> 62);
          if (flag == 0) {
            if (++spins > kScanSpinLimit) {
              atomicAdd(err, 1ULL);
              break;
            }
            __nanosleep(32);
            continue;
          }
          excl += (long long)(w & ((1ULL << 62) - 1));
          if (flag == 2u) break;
          look--;
        }
        atomicExch(&st[tile], scan_word(2u, excl + agg));
      }
      carry_sh = excl;
    }
    __syncthreads();
    long long off = carry_sh + pre;
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
      long long i = base + k;
      if (i < n) J.out[i] = off;
      off += v[k];
    }
    if (tile == nb - 1 && threadIdx.x == 0) {
      J.out[n] = carry_sh + agg;
      if (J.total_out) *J.total_out = carry_sh + agg;
    }
  }
  // the last block of this job to finish clears the job's status words
  if (threadIdx.x == 0) {
    __threadfence();
    unsigned d = atomicAdd(&done_ctr[blockIdx.y], 1u);
    if (d == gridDim.x - 1) {
      for (unsigned k = 0; k < gridDim.x; k++) st[k] = 0ULL;
      done_ctr[blockIdx.y] = 0;
      __threadfence();
    }
  }
}

// ---------------------------------------------------------------------------
// small helper kernels


// The exclusive prefix of a tile's sum (62 bits) over the tiles before it, by
// the block's first warp (decoupled look-back, 32 predecessors at a time; see
// k_scan_lb for the status words).  Tiles are numbered in the order blocks
// start, so a tile only waits on running blocks.
__device__ unsigned long long tile_prefix(unsigned long long* st, long long tile, unsigned long long agg,
                                          unsigned long long* err) {
  constexpr unsigned kFull = 0xffffffffu;
  constexpr unsigned long long kMask = (1ULL << 62) - 1;
  const int lane = threadIdx.x & 31;
  if (tile == 0) {
    if (lane == 0) atomicExch(&st[0], scan_word(2u, (long long)agg));
    return 0ULL;
  }
  if (lane == 0) atomicExch(&st[tile], scan_word(1u, (long long)agg));
  unsigned long long excl = 0ULL;
  int spins = 0;
  for (long long base = tile - 1; base >= 0;) {
    const long long i = base - lane;
    const unsigned long long w = i >= 0 ? *(volatile unsigned long long*)&st[i] : (2ULL << 62);
    const unsigned flag = (unsigned)(w >> 62);
    const unsigned m2 = __ballot_sync(kFull, flag == 2u), m0 = __ballot_sync(kFull, flag == 0u);
    const unsigned upto = m2 ? (m2 & (0u - m2)) * 2u - 1u : kFull;  // lanes to the nearest inclusive prefix
    if (m0 & upto) {
      if (++spins > kScanSpinLimit) {
        if (lane == 0) atomicAdd(err, 1ULL);
        break;
      }
      __nanosleep(20);
      continue;
    }
    unsigned long long v = ((upto >> lane) & 1u) ? (w & kMask) : 0ULL;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
    excl += v;
    if (m2) break;
    base -= 32;
  }
  if (lane == 0) atomicExch(&st[tile], scan_word(2u, (long long)((excl + agg) & kMask)));
  return excl;
}

// what a tiled kernel shares between its blocks: status words (zero between
// launches), tile and finished-block counters, give-ups
struct TileCtl {
  unsigned long long* status;
  unsigned *tile_ctr, *done_ctr;
  unsigned long long* err;
};

// the block's tile, in the order blocks start
__device__ __forceinline__ long long take_tile(const TileCtl& T) {
  __shared__ unsigned tile_sh;
  if (threadIdx.x == 0) {
    const unsigned t = atomicAdd(T.tile_ctr, 1u);
    if (t == gridDim.x - 1) *T.tile_ctr = 0;  // the last claimant re-arms the counter
    tile_sh = t;
  }
  __syncthreads();
  return tile_sh;
}

// true in the last block to come here, which then sees what the others wrote
// and has cleared the status words for the next launch
__device__ __forceinline__ bool last_block(const TileCtl& T) {
  __shared__ bool last_sh;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last_sh = atomicAdd(T.done_ctr, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last_sh) return false;
  __threadfence();
  for (unsigned k = threadIdx.x; k < gridDim.x; k += blockDim.x) T.status[k] = 0ULL;
  if (threadIdx.x == 0) *T.done_ctr = 0;
  return true;
}

// The events of a round in order, from the flagged samples (round 0) or items:
// flags are counted, ranked and their events written in one launch.  A tile is
// small so that a round of a few thousand events still spreads over the chip.
constexpr int kCompactThreads = 256;
constexpr int kCompactTile = 4 * kCompactThreads;

struct CompactArgs {
  const uint8_t* flag;
  const long long* n;  // flags
  long long* n_events;
  TileCtl ctl;
  // the events
  unsigned long long* ev_key;
  int2* ev_c;
  int* gp_c;
  float* ev_pos;
  int* ev_len;
  int4* ev_term;
  uint32_t* dec;
};

// flags i..i+3 of n, as the bits 0..3
__device__ __forceinline__ unsigned flags_of(const uint8_t* flag, long long i, long long n) {
  if (i + 4 <= n) {
    const uchar4 f = *reinterpret_cast<const uchar4*>(flag + i);
    return (f.x ? 1u : 0u) | (f.y ? 2u : 0u) | (f.z ? 4u : 0u) | (f.w ? 8u : 0u);
  }
  unsigned m = 0u;
  for (int k = 0; k < 4; k++)
    if (i + k < n && flag[i + k]) m |= 1u << k;
  return m;
}
// the same of entries that hold a population (-1: none)
__device__ __forceinline__ unsigned flags_of(const int* pop, long long i, long long n) {
  unsigned m = 0u;
  for (int k = 0; k < 4; k++)
    if (i + k < n && pop[i + k] >= 0) m |= 1u << k;
  return m;
}

// places of the tile's flagged entries of n: sh_idx[r] is the tile's r-th, and
// the place of the tile's first among all is returned; *n_out gets their count
template <class T>
__device__ long long compact_tile(const T* flag, long long n, long long* n_out, const TileCtl& ctl, int* sh_idx,
                                  int* count) {
  __shared__ unsigned long long excl_sh;
  const long long n_tiles = (n + kCompactTile - 1) / kCompactTile;
  const long long tile = take_tile(ctl);
  if (tile >= n_tiles) {
    if (n_tiles == 0 && tile == 0 && threadIdx.x == 0) *n_out = 0;
    *count = 0;
    return 0;
  }
  const unsigned f = flags_of(flag, tile * kCompactTile + 4 * threadIdx.x, n);
  int tot;
  int r = block_excl_scan(__popc(f), &tot);
  for (int k = 0; k < 4; k++)
    if ((f >> k) & 1u) sh_idx[r++] = (int)(tile * kCompactTile) + 4 * (int)threadIdx.x + k;
  if (threadIdx.x < 32) {
    const unsigned long long e = tile_prefix(ctl.status, tile, (unsigned long long)tot, ctl.err);
    if (threadIdx.x == 0) {
      excl_sh = e;
      if (tile == n_tiles - 1) *n_out = (long long)e + tot;
    }
  }
  __syncthreads();
  *count = tot;
  return (long long)excl_sh;
}

// Round 0: accepted samples in sample order.  Event e gets its key (pair,
// sample), its two slots, its global pair and its position in the pair's test
// sequence ((s + 1) / n_samp: the part of the pair done after it), its merge
// decision (coagulate_weighting, coagulation.F90:810-922) from the sample's
// own stream (merge_rng of its key), and the claims on its two slots by it: a
// write claim on a slot the merge removes or rewrites, a read claim on one it
// keeps.  One launch for what were three (scan, compaction, decisions).
__global__ void __launch_bounds__(kCompactThreads) k_compact_samples(CompactArgs A, const PopDev* pops,
                                                                     const int* gpair_pop, const int* gpair_local,
                                                                     const int2* ev, const int* ev_gp,
                                                                     const long long* work_off) {
  chain_wait();
  __shared__ int sh_idx[kCompactTile];
  int count;
  const long long e0 = compact_tile(A.flag, *A.n, A.n_events, A.ctl, sh_idx, &count);
  for (int r = threadIdx.x; r < count; r += kCompactThreads) {
    const long long i = sh_idx[r], e = e0 + r;
    const int gp = ev_gp[i];
    const int2 sl = ev[i];
    const long long w0 = work_off[gp];
    const long long s = i - w0, ns = work_off[gp + 1] - w0;
    const int p = gpair_local[gp];
    const PopDev& P = pops[gpair_pop[gp]];
    const unsigned long long key = make_key((uint32_t)p, 0u, (uint32_t)s);
    A.ev_key[e] = key;
    A.ev_c[e] = sl;
    A.gp_c[e] = gp;
    A.ev_pos[e] = (float)((double)(s + 1) / (double)ns);
    A.ev_len[e] = 0;
    A.ev_term[e] = no_term();
    const PairState& S = P.pair[p];
    const PairDesc d = P.pair_desc[p];
    Rng gm = merge_rng(P, key);
    const MergeDecision m = merge_decide(P, gm, sl.x, sl.y, d.c1, d.c2, S.cc);
    if (m.new_group == 0) set_status(P.ctr, kErrTimeout);
    A.dec[e] = pack_decision(m, gm.used());
    const unsigned long long ck = claim_key(P, key);
    claim_slot(P, sl.x, ck, m.rm1);
    claim_slot(P, sl.y, ck, m.rm2);
  }
  last_block(A.ctl);
}

// Later rounds: the events the items made, in item order (grouped: at the
// places group_by_pop gave them)
__global__ void __launch_bounds__(kCompactThreads) k_compact_items(CompactArgs A, const unsigned long long* it_key,
                                                                   const int2* it_c, const int* it_gp,
                                                                   const float* it_pos, const int* it_len,
                                                                   const int* it_head, const uint8_t* it_done,
                                                                   const uint32_t* it_dec, const int4* it_term,
                                                                   int* ev_head, uint8_t* ev_done,
                                                                   const long long* grouped) {
  chain_wait();
  __shared__ int sh_idx[kCompactTile];
  int count;
  const long long e0 = compact_tile(A.flag, *A.n, A.n_events, A.ctl, sh_idx, &count);
  for (int r = threadIdx.x; r < count; r += kCompactThreads) {
    const long long i = sh_idx[r], e = grouped ? grouped[i] : e0 + r;
    if (e < 0) continue;
    A.ev_key[e] = it_key[i];
    A.ev_c[e] = it_c[i];
    A.gp_c[e] = it_gp[i];
    A.ev_pos[e] = it_pos[i];
    A.ev_len[e] = it_len[i];
    ev_head[e] = it_head[i];
    ev_done[e] = it_done[i];
    A.dec[e] = it_dec[i];
    A.ev_term[e] = it_term[i];
  }
  last_block(A.ctl);
}

// target operations of round 0 (the first cap of them), in the reference's
// backwards target order (coagulation.F90:220-237)
__global__ void k_build_ops(const PopDev* pops, const int* gpair_pop, const int* gpair_local,
                            const long long* pp_off, int n_gpairs, long long cap, int* op_pop, int* op_pair,
                            int* op_slot, int* op_k, unsigned long long* op_key) {
  int gp = blockIdx.x;
  if (gp >= n_gpairs) return;
  long long n = pp_off[gp + 1] - pp_off[gp];
  if (n == 0) return;
  int pop = gpair_pop[gp];
  const PopDev& P = pops[pop];
  int p = gpair_local[gp];
  const PairState& S = P.pair[p];
  int tcell = S.bt + P.grid->n_bin * S.ct;
  int start = P.cell_start[tcell];
  for (long long k = threadIdx.x; k < n; k += blockDim.x) {
    long long q = pp_off[gp] + k;
    if (q >= cap) break;  // more than a step graph has room for: k_step_check stops it
    op_pop[q] = pop;
    op_pair[q] = p;
    op_slot[q] = P.list[start + (int)(n - 1 - k)];
    op_k[q] = (int)k;
    op_key[q] = make_key((uint32_t)p, 0u, (uint32_t)k);
  }
}

// redo list of lost target operations (order of q kept); a redo keeps its
// place in the loop order (its key)
__global__ void k_build_redo(const PopDev* pops, const int* op_pop, const int* op_pair, const int* op_slot,
                             const int* op_k, const unsigned long long* op_key, const int* lost,
                             const long long* lost_off, const long long* n_ops, int* r_pop, int* r_pair, int* r_slot,
                             int* r_k, unsigned long long* r_key, uint32_t begun) {
  const long long Q = *n_ops;
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < Q;
       q += (long long)gridDim.x * blockDim.x) {
    if (!lost[q]) continue;
    long long j = lost_off[q];
    const PopDev& P = pops[op_pop[q]];
    const int t = op_slot[q];
    r_pop[j] = op_pop[q];
    r_pair[j] = op_pair[q];
    // a target that an earlier operation or event of the round consumed
    // (removed or rewrote) walks on from there instead: its redo is void.  A
    // slot is stamped with that round's generation, the one before a round
    // that has begun
    const bool consumed = t < 0 || t >= P.cap || !P.alive[t] || P.touched[t] == *P.gen_p - begun;
    r_slot[j] = consumed ? -1 : t;
    r_k[j] = op_k[q] + (1 << 24);  // fresh random stream for the redo
    r_key[j] = op_key[q];
  }
}

// first event of population k (events are ordered by population)
__device__ long long first_event_of(int k, long long E, const int* ev_gp, const int* gpair_pop) {
  long long lo = 0, hi = E;
  while (lo < hi) {
    long long mid = (lo + hi) >> 1;
    if (gpair_pop[ev_gp[mid]] < k) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// Per-population bases of the allocations of one round.  Events and target
// operations are ordered by population, so a global exclusive rank minus the
// count of earlier populations is the rank inside the population.  Per-set
// counts come from the rank scans at the population boundaries (and are
// stored in per_pop for the host); per-particle counts were summed into
// per_pop by k_pp_resolve.  The slot and ID counters of each population
// advance here by the round's allocations: the apply kernels read only the
// bases.  By one block; populations in tiles of blockDim.x.
__device__ void alloc_bases(const PopDev* pops, int n_pop, long long E, const int* ev_gp, const int* gpair_pop,
                            const long long* rank_slot_set, const long long* rank_id_set, int* per_pop,
                            int* set_slot_base, long long* set_id_base, int* pp_slot_base, long long* pp_id_base) {
  long long carry[4] = {0, 0, 0, 0};
  for (int base = 0; base < n_pop; base += blockDim.x) {
    int k = base + threadIdx.x;
    long long cnt[4] = {0, 0, 0, 0};
    if (k < n_pop) {
      if (E > 0) {
        long long e_lo = n_pop == 1 ? 0 : first_event_of(k, E, ev_gp, gpair_pop);
        long long e_hi = n_pop == 1 ? E : first_event_of(k + 1, E, ev_gp, gpair_pop);
        cnt[0] = rank_slot_set[e_hi] - rank_slot_set[e_lo];
        cnt[1] = rank_id_set[e_hi] - rank_id_set[e_lo];
      }
      per_pop[k] = (int)cnt[0];
      per_pop[n_pop + k] = (int)cnt[1];
      cnt[2] = per_pop[2 * n_pop + k];
      cnt[3] = per_pop[3 * n_pop + k];
    }
    long long pre[4], tot[4];
    for (int j = 0; j < 4; j++) pre[j] = block_excl_scan_ll(cnt[j], &tot[j]);
    if (k < n_pop) {
      PopCtr* c = pops[k].ctr;
      long long cs = carry[0] + pre[0], ci = carry[1] + pre[1], ps = carry[2] + pre[2], pi = carry[3] + pre[3];
      set_slot_base[k] = c->n_slots - (int)cs;
      set_id_base[k] = c->next_id - ci;
      pp_slot_base[k] = c->n_slots + (int)cnt[0] - (int)ps;
      pp_id_base[k] = c->next_id + cnt[1] - pi;
      c->n_slots += (int)(cnt[0] + cnt[2]);
      c->next_id += cnt[1] + cnt[3];
    }
    for (int j = 0; j < 4; j++) carry[j] += tot[j];
  }
}

// Resolve the events of a round: winner test, slot/id needs.  Event e has
// key ev_key[e], slots ev[e], global pair ev_gp[e] and merge decision dec[e]
// (drawn when the event was formed); the events are ordered by population.
// A winning chain (ev_len[e] > 0) gets win 2 and the number of its events
// whose claims hold (ev_app[e]).  The same launch ranks the winners' new slots
// and IDs (31 bits of a status word each) and, in its last block, sets the
// populations' bases (alloc_bases): three launches in one.
constexpr int kResolveMin = 64;  // smallest block of k_resolve

struct ResolveArgs {
  const PopDev* pops;
  const int* gpair_pop;
  const long long* n_events;  // null: the round has no events, only bases to set
  const unsigned long long* ev_key;
  const int2* ev;
  const int* ev_gp;
  uint8_t* win;
  const uint32_t* dec;
  long long* n_losers;
  const int *ev_len, *ev_head;
  int* ev_app;
  ChainPool pool;
  int* chain_list;
  long long* n_chain;
  long long *rank_slot, *rank_id;
  TileCtl ctl;
  int n_pop;
  int *per_pop, *set_slot_base, *pp_slot_base;
  long long *set_id_base, *pp_id_base;
};

// 1 if event e wins (2: a chain), with its needs
__device__ __forceinline__ int resolve_event(const ResolveArgs& A, long long e, int* need_slot, int* need_id) {
  *need_slot = *need_id = 0;
  const int gp = A.ev_gp[e];
  const PopDev& P = A.pops[A.gpair_pop[gp]];
  const unsigned long long key = A.ev_key[e];
  const int p = (int)key_pair(key);
  const int2 sl = A.ev[e];
  const int len = A.ev_len[e];
  uint32_t used;
  const MergeDecision m = unpack_decision(A.dec[e], &used);
  if (sl.x < 0 || sl.x >= P.cap || sl.y < 0 || sl.y >= P.cap || p >= P.n_pairs) {
    bad_index(P.ctr, kBadEventSlot, sl.x < 0 || sl.x >= P.cap ? sl.x : sl.y);
    return 0;
  }
  const unsigned long long ck = claim_key(P, key);
  if (!(holds_slot(P, sl.x, ck, m.rm1) && holds_slot(P, sl.y, ck, m.rm2))) {
    add_ll_warp(A.n_losers, 1);
    return 0;
  }
  if (len > 0) {
    // a chain: its events apply as far as each partner's claim holds (the
    // walking particle's is the first event's)
    ChainReader rd(A.ev_head[e]);
    const uint32_t x = key_idx(key);
    int app = 0;
    for (int i = 0; i < len; i++) {
      const long long ix = rd.next(A.pool);
      if (ix < 0) break;
      const int y = A.pool.y[ix], qw = A.pool.q[ix];
      const int q = qw & kChainPairMask;
      if (y < 0 || y >= P.cap || q < 0 || q >= P.n_pairs) break;
      if (!holds_slot(P, y, claim_key(P, make_key((uint32_t)q, 1u, x)), (qw & kChainRemoves) != 0)) break;
      app++;
    }
    A.ev_app[e] = app;
    A.chain_list[inc_warp((unsigned long long*)A.n_chain)] = (int)e;
    return 2;
  }
  if (m.create) {
    *need_slot = (!m.rm1 && !m.rm2) ? 1 : 0;
    const bool keep1 = m.rm1 && !m.lost1, keep2 = m.rm2 && !m.lost2;
    *need_id = (!keep1 && !keep2) ? 1 : 0;
  }
  return 1;
}

__global__ void __launch_bounds__(256) k_resolve(ResolveArgs A) {
  chain_wait();
  __shared__ unsigned long long excl_sh;
  const long long E = A.n_events ? *A.n_events : 0;
  const int tb = blockDim.x;  // events of a tile
  const long long n_tiles = (E + tb - 1) / tb;
  const long long tile = take_tile(A.ctl);
  if (tile < n_tiles) {
    const long long e = tile * tb + threadIdx.x;
    int ns = 0, ni = 0;
    if (e < E) A.win[e] = (uint8_t)resolve_event(A, e, &ns, &ni);
    // at most 256 of each in a tile: one scan of both
    int tot;
    const int pre = block_excl_scan(ns | (ni << 16), &tot);
    if (threadIdx.x < 32) {
      const unsigned long long agg = (unsigned long long)(tot & 0xffff) | ((unsigned long long)(tot >> 16) << 31);
      const unsigned long long x = tile_prefix(A.ctl.status, tile, agg, A.ctl.err);
      if (threadIdx.x == 0) excl_sh = x;
    }
    __syncthreads();
    const long long s0 = (long long)(excl_sh & 0x7fffffffULL), i0 = (long long)(excl_sh >> 31);
    if (e < E) {
      A.rank_slot[e] = s0 + (pre & 0xffff);
      A.rank_id[e] = i0 + (pre >> 16);
    }
    if (tile == n_tiles - 1 && threadIdx.x == 0) {
      A.rank_slot[E] = s0 + (tot & 0xffff);
      A.rank_id[E] = i0 + (tot >> 16);
    }
  }
  if (last_block(A.ctl))
    alloc_bases(A.pops, A.n_pop, E, A.ev_gp, A.gpair_pop, A.rank_slot, A.rank_id, A.per_pop, A.set_slot_base,
                A.set_id_base, A.pp_slot_base, A.pp_id_base);
}

// The bound on each target operation's removals (pp_remove_bound), scanned into
// its place in the removal pool; their total to *total.  At most cap operations
// are counted (a step graph's bound; the step does not run beyond it).
__global__ void __launch_bounds__(256) k_pp_count(const PopDev* pops, const int* op_pop, const int* op_pair,
                                                  const int* op_slot, const int* op_k, const long long* n_ops,
                                                  long long cap, long long* rm_off, long long* total, TileCtl ctl) {
  chain_wait();
  __shared__ unsigned long long excl_sh;
  const long long Q = *n_ops < cap ? *n_ops : cap, n_tiles = (Q + 255) / 256;
  const long long tile = take_tile(ctl);
  if (tile < n_tiles) {
    const long long q = tile * 256 + threadIdx.x;
    int n = 0;
    if (q < Q) {
      Rng g(0, 0, 0, 0);
      int n_extra = 0;
      double prm = 0.0;
      n = pp_remove_bound(pops[op_pop[q]], op_pair[q], op_slot[q], op_k[q], &g, &n_extra, &prm);
      if (n < 0) n = 0;
    }
    long long tot;
    const long long pre = block_excl_scan_ll(n, &tot);
    if (threadIdx.x < 32) {
      const unsigned long long x = tile_prefix(ctl.status, tile, (unsigned long long)tot, ctl.err);
      if (threadIdx.x == 0) excl_sh = x;
    }
    __syncthreads();
    if (q < Q) rm_off[q] = (long long)excl_sh + pre;
    if (tile == n_tiles - 1 && threadIdx.x == 0) *total = (long long)excl_sh + tot;
  } else if (n_tiles == 0 && tile == 0 && threadIdx.x == 0) {
    *total = 0;
  }
  last_block(ctl);
}

// Winners of the round's target operations, the ranks of the slots (and IDs:
// as many) that their copies need, the needs per population, and the places of
// the operations that lost, whose count goes to *n_lost: one launch for what
// were five.
__global__ void __launch_bounds__(256) k_pp_resolve(const PopDev* pops, int n_pop, const int* op_pop,
                                                    const unsigned long long* op_key, const long long* n_ops,
                                                    const PPResult* res, const int* rm_pool, uint8_t* win,
                                                    long long* rank, int* per_pop, int* lost, long long* lost_off,
                                                    long long* n_lost, TileCtl ctl) {
  chain_wait();
  __shared__ unsigned long long excl_sh;
  const long long Q = *n_ops, n_tiles = (Q + 255) / 256;
  const long long tile = take_tile(ctl);
  if (tile < n_tiles) {
    const long long q = tile * 256 + threadIdx.x;
    bool ok = true;
    int extra = 0;
    if (q < Q) {
      const int pop = op_pop[q];
      const PopDev& P = pops[pop];
      const PPResult& R = res[q];
      const unsigned long long ck = claim_key(P, op_key[q]);
      ok = !R.nofit;
      if (R.merged) ok = ok && holds_slot(P, R.target, ck, true);
      for (int z = 0; z < R.n_rm && ok; z++) ok = holds_slot(P, rm_pool[R.rm_off + z], ck, true);
      win[q] = ok ? 1 : 0;
      lost[q] = ok ? 0 : 1;
      extra = (ok && R.merged && R.n_copies > 1) ? R.n_copies - 1 : 0;
      if (extra) {
        atomicAdd(&per_pop[2 * n_pop + pop], extra);
        atomicAdd(&per_pop[3 * n_pop + pop], extra);
      }
    }
    // at most 7 x 256 copies and 256 losers in a tile: one scan of both
    int tot;
    const int pre = block_excl_scan(extra | (ok ? 0 : 1 << 16), &tot);
    if (threadIdx.x < 32) {
      const unsigned long long agg = (unsigned long long)(tot & 0xffff) | ((unsigned long long)(tot >> 16) << 31);
      const unsigned long long x = tile_prefix(ctl.status, tile, agg, ctl.err);
      if (threadIdx.x == 0) excl_sh = x;
    }
    __syncthreads();
    const long long s0 = (long long)(excl_sh & 0x7fffffffULL), l0 = (long long)(excl_sh >> 31);
    if (q < Q) {
      rank[q] = s0 + (pre & 0xffff);
      lost_off[q] = l0 + (pre >> 16);
    }
    if (tile == n_tiles - 1 && threadIdx.x == 0) *n_lost = l0 + (tot >> 16);
  } else if (n_tiles == 0 && tile == 0 && threadIdx.x == 0) {
    *n_lost = 0;
  }
  last_block(ctl);
}

// walker places of the round's operations (kMaxCopies each), compacted in order
__global__ void __launch_bounds__(kCompactThreads) k_compact_walkers(const uint8_t* flag, const long long* n_ops,
                                                                     long long* n_walkers, TileCtl ctl,
                                                                     const int* wk_slot, const int* wk_gp,
                                                                     int* ppw_slot, int* ppw_gp) {
  chain_wait();
  __shared__ int sh_idx[kCompactTile];
  int count;
  const long long e0 = compact_tile(flag, *n_ops * kMaxCopies, n_walkers, ctl, sh_idx, &count);
  for (int r = threadIdx.x; r < count; r += kCompactThreads) {
    ppw_slot[e0 + r] = wk_slot[sh_idx[r]];
    ppw_gp[e0 + r] = wk_gp[sh_idx[r]];
  }
  last_block(ctl);
}

// A later round's target operations of one population from the staging list,
// in order, without the places that hold none
__global__ void __launch_bounds__(kCompactThreads) k_compact_ops(const long long* n_staged, long long* n_ops,
                                                                 TileCtl ctl, const int* pop, const int* pair,
                                                                 const int* slot, const int* k,
                                                                 const unsigned long long* key, int* pop_o,
                                                                 int* pair_o, int* slot_o, int* k_o,
                                                                 unsigned long long* key_o) {
  chain_wait();
  __shared__ int sh_idx[kCompactTile];
  int count;
  const long long e0 = compact_tile(pop, *n_staged, n_ops, ctl, sh_idx, &count);
  for (int r = threadIdx.x; r < count; r += kCompactThreads) {
    const int i = sh_idx[r];
    const long long e = e0 + r;
    pop_o[e] = pop[i];
    pair_o[e] = pair[i];
    slot_o[e] = slot[i];
    k_o[e] = k[i];
    key_o[e] = key[i];
  }
  last_block(ctl);
}

// particle upload: the caller's arrays were copied straight into slots
// 0..n-1 (same particle-major layout); fill the caches and the fields the
// caller did not give
__global__ void k_upload(PopDev P, int n, int have_grp, int have_cls, int have_id, int have_nprim,
                         long long id0, int* bad, unsigned long long* max_id) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    // the caller's groups and classes are checked here, on the device
    if (have_grp && (P.grp[i] < 1 || P.grp[i] > P.n_group)) atomicOr(bad, 1);
    if (have_cls && (P.cls[i] < 1 || P.cls[i] > P.n_class)) atomicOr(bad, 2);
    if (have_id && P.id[i] >= 0) atomicMax(max_id, (unsigned long long)P.id[i]);
    P.changed[i] = 0;
    double vt = 0.0, ms = 0.0;
    for (int s = 0; s < P.n_spec; s++) vt = vt + P.vol[vol_at(P, i, s)];
    for (int s = 0; s < P.n_spec; s++) ms = ms + P.vol[vol_at(P, i, s)] * P.density[s];
    P.vtot[i] = vt;
    P.mass[i] = ms;
    if (!have_grp) P.grp[i] = 1;
    if (!have_cls) P.cls[i] = 1;
    if (!have_id) P.id[i] = id0 + i;
    if (!have_nprim) P.nprim[i] = 1;
    P.ncomp[i] = 1;
    P.csrc[comp_at(i, 0)] = 1;
    P.ctime[comp_at(i, 0)] = 0.0;
    P.lct[i] = 0.0;
    P.gct[i] = 0.0;
    P.imf[i] = 0.0;
    P.den_ice[i] = __longlong_as_double(0x7ff8000000000000LL);
    P.phi[i] = __longlong_as_double(0x7ff8000000000000LL);
    P.hyst[i] = 0;
    P.frozen[i] = 0;
    P.alive[i] = 1;
    P.cell[i] = -1;  // set by the first refresh after the grid decision
  }
}

// live slots gathered in order into the caller's layout, only the fields asked
// for (non-null outputs).  A warp takes 32 slots: a lane each for the scalars,
// then the slots' species and components in memory order across the lanes (a
// thread per slot moved them at its own stride: 140 us for 1e6 slots of 20
// species, now 70)
__global__ void __launch_bounds__(256) k_download(PopDev P, const long long* live_off, int n_slots, double* vol_pm,
                                                  int* grp, int* cls, long long* id, int* nprim, int* ncomp,
                                                  int* csrc, double* ctime) {
  constexpr unsigned kFull = 0xffffffffu;
  const int lane = threadIdx.x & 31, ns = P.n_spec;
  const int warps = (gridDim.x * blockDim.x) >> 5;
  for (int base = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 32; base < n_slots; base += warps * 32) {
    const int i = base + lane;
    const bool on = i < n_slots && P.alive[i];
    const long long j = on ? live_off[i] : -1;
    int nc = 0;
    if (on) {
      if (grp) grp[j] = P.grp[i];
      if (cls) cls[j] = P.cls[i];
      if (id) id[j] = P.id[i];
      if (nprim) nprim[j] = P.nprim[i];
      if (ncomp || csrc || ctime) nc = P.ncomp[i];
      if (ncomp) ncomp[j] = nc;
    }
    if (vol_pm) {
      int part = lane / ns, sp = lane % ns;
      for (int k = 0; k < ns; k++) {  // 32 ns words
        const long long jp = __shfl_sync(kFull, j, part);
        if (jp >= 0) vol_pm[jp * ns + sp] = P.vol[vol_at(P, base + part, sp)];
        sp += 32;
        while (sp >= ns) {
          sp -= ns;
          part++;
        }
        part &= 31;  // past the last word only
      }
    }
    if (csrc || ctime) {
      int part = lane / kMaxComponent, q = lane % kMaxComponent;
      for (int k = 0; k < kMaxComponent; k++) {
        const long long jp = __shfl_sync(kFull, j, part);
        const int np = __shfl_sync(kFull, nc, part);
        if (jp >= 0) {
          if (csrc) csrc[jp * kMaxComponent + q] = q < np ? P.csrc[comp_at(base + part, q)] : 0;
          if (ctime) ctime[jp * kMaxComponent + q] = q < np ? P.ctime[comp_at(base + part, q)] : 0.0;
        }
        q += 32;
        while (q >= kMaxComponent) {
          q -= kMaxComponent;
          part++;
        }
        part &= 31;
      }
    }
  }
}

// Changed slots of [lo, hi) packed for the host copy, one record of
// rec_bytes = kSyncHead + 8 n_spec bytes rounded up to a multiple of 16:
// {slot, alive, group, class, n_primary, 0, id (8 bytes)} then the species
// volumes.  Each warp takes 32 slots and reserves places for its changed
// ones with one atomic; it assembles their records in shared memory (one
// lane per species for the volumes) and writes them out as consecutive
// 16-byte words, so that a write into host memory goes over the bus in full
// lines.  Record order is arbitrary (the host scatters by slot).  Clears the
// changed flags.
constexpr int kSyncHead = 32;
__global__ void k_pack_changed(PopDev P, int lo, int hi, unsigned long long* count, unsigned char* out,
                               int rec_bytes) {
  extern __shared__ int4 pack_stage[];  // [warps of the block][32 records]
  const int lane = threadIdx.x & 31;
  unsigned char* my = (unsigned char*)pack_stage + (size_t)(threadIdx.x >> 5) * 32 * rec_bytes;
  const int warps = (gridDim.x * blockDim.x) >> 5;
  for (int base = lo + ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 32; base < hi; base += warps * 32) {
    const int i = base + lane;
    const bool ch = i < hi && P.changed[i];
    const unsigned m = __ballot_sync(0xffffffffu, ch);
    if (!m) continue;
    unsigned long long b = 0;
    if (lane == 0) b = atomicAdd(count, (unsigned long long)__popc(m));
    b = __shfl_sync(0xffffffffu, b, 0);
    if (ch) {
      unsigned char* r = my + (size_t)__popc(m & ((1u << lane) - 1u)) * rec_bytes;
      const int a = P.alive[i];
      *(int4*)r = make_int4(i, a, a ? P.grp[i] : 0, a ? P.cls[i] : 0);
      *(int2*)(r + 16) = make_int2(a ? P.nprim[i] : 0, 0);
      *(long long*)(r + 24) = a ? P.id[i] : 0;
      P.changed[i] = 0;
    }
    for (unsigned mm = m; mm; mm &= mm - 1) {
      const int src = __ffs(mm) - 1;
      const int si = base + src;
      if (!P.alive[si]) continue;
      double* v = (double*)(my + (size_t)__popc(m & ((1u << src) - 1u)) * rec_bytes + kSyncHead);
      for (int sp = lane; sp < P.n_spec; sp += 32) v[sp] = P.vol[vol_at(P, si, sp)];
    }
    __syncwarp();
    const int n16 = __popc(m) * (rec_bytes / 16);
    int4* d = (int4*)(out + (size_t)b * rec_bytes);
    const int4* sm = (const int4*)my;
    for (int k = lane; k < n16; k += 32) d[k] = sm[k];
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------
// aero_state_rebalance (aero_state.F90:1722-1852) on the device

// live particles per (group, class): counts[(g-1) + n_group*(c-1)]
__global__ void k_count_group_class(PopDev P, int* counts) {
  int n = P.ctr->n_slots;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    if (!P.alive[i]) continue;
    int g = P.grp[i], c = P.cls[i];
    if (g >= 1 && g <= P.n_group && c >= 1 && c <= P.n_class) atomicAdd(&counts[(g - 1) + P.n_group * (c - 1)], 1);
  }
}

// members of (g, c) among slots 0..n-1
__global__ void k_flag_group_class(PopDev P, int n, int g, int c, uint8_t* flag) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    flag[i] = (P.alive[i] && P.grp[i] == g && P.cls[i] == c) ? 1 : 0;
}

// aero_state_double: member j (in slot order) is copied to slot n + j with
// ID id0 + j (aero_particle_new_id); every field is copied, caches included
__global__ void k_double(PopDev P, int n, const uint8_t* flag, const long long* off, long long id0) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    if (!flag[i]) continue;
    int d = n + (int)off[i];
    if (d >= P.cap) {
      cap_fail(P.ctr, kCapDupSlot);
      continue;
    }
    copy_particle(P, i, d, id0 + off[i]);
  }
}

// aero_state_halve: each member removed with probability 1/2; the draw of
// slot i is keyed by the population's seed and step, the rebalance call and i
__global__ void k_halve(PopDev P, int g, int c, uint32_t call) {
  int n = P.ctr->n_slots;
  int removed = 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    if (!(P.alive[i] && P.grp[i] == g && P.cls[i] == c)) continue;
    U4 r = philox4x32_10(U4{P.step, (call << 4) | kStreamHalve, (uint32_t)i, 0u}, (uint32_t)P.seed,
                         (uint32_t)(P.seed >> 32));
    if (u53(r.x, r.y) < 0.5) {
      log_removal(P, P.id[i], kInfoHalved, 0);  // aero_state_halve records it (aero_state.F90:1768-1781)
      kill_slot(P, i);
      removed++;
    }
  }
  if (removed) add_ll(&P.ctr->n_live, -(long long)removed);
}

// ---------------------------------------------------------------------------
// size distributions (extract_aero_size.F90:132-138 with
// bin_grid_histogram_1d, bin_grid.F90:225-248): diameters on a log grid of
// n_bin bins from d_min to d_max, each particle weighted by its number
// concentration (aero_state_num_concs), per unit log diameter.  out holds
// n_bin number values, then n_bin x n_spec species masses (kg m^-3).
// A block takes TILE slots at a time and orders them by bin (counts and
// ranks in shared memory).  A warp then goes over 64 of the ordered particles
// with a lane per species (a particle's volumes are consecutive; HI: over 32
// species, two a lane), eight particles' loads in flight, and sums a run of
// one bin in registers; a run ends in one add to the block's sums.  Then one
// atomic per bin and block, each block starting at another bin.
// One thread per particle read each volume at its own stride and made
// 1 + n_spec FP64 atomics (a compare-and-swap loop each) on shared words that
// its neighbours also hit: 175 us for 1e6 particles of 20 species on 160 bins,
// now 87.  (Sums of its own for every warp need no atomics, but leave room for
// 8 warps an SM, too few to hide the loads: 290 us.  Adding the sums up over a
// cluster first: 150 us, the blocks of a cluster wait for their slowest.)
constexpr int kDistThreads = 512;
constexpr int kDistTile = 2 * kDistThreads;
constexpr int kDistFewSpec = 8;

// With at most kDistFewSpec species a thread per particle and its 1 + n_spec
// atomics are the shorter way: 1e6 slots of 1 and 7 species take 84 and 105 us
// a call, 123 and 128 in order of bins with a lane per species (most lanes
// idle); 20 species 226 and 145.
__global__ void __launch_bounds__(256) k_size_dist_few(PopDev P, int n_bin, double log_lo, double log_hi,
                                                       double inv_width, double* out) {
  extern __shared__ double hs[];  // [n_bin * (1 + n_spec)]
  const int nv = n_bin * (1 + P.n_spec);
  for (int k = threadIdx.x; k < nv; k += blockDim.x) hs[k] = 0.0;
  __syncthreads();
  const int n = P.ctr->n_slots;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    if (!P.alive[i]) continue;
    const double r = vol2rad(P.benv.frac, P.vtot[i]);  // aero_particle_radius (fractal_vol2rad)
    const int b = bin_find(n_bin, log_lo, log_hi, 2.0 * r);
    if (b < 1 || b > n_bin) continue;
    const double nc = num_conc_at_radius<double>(P.w, P.cls[i] - 1, r) * inv_width;
    atomicAdd(&hs[b - 1], nc);
    for (int s = 0; s < P.n_spec; s++)
      atomicAdd(&hs[n_bin + (b - 1) * P.n_spec + s], nc * P.vol[vol_at(P, i, s)] * P.density[s]);
  }
  __syncthreads();
  for (int k = threadIdx.x; k < nv; k += blockDim.x)
    if (hs[k] != 0.0) atomicAdd(&out[k], hs[k]);
}

template <bool HI, int TILE>
__global__ void __launch_bounds__(kDistThreads) k_size_dist(PopDev P, int n_bin, double log_lo, double log_hi,
                                                            double inv_width, double* out) {
  constexpr int kPer = TILE / kDistThreads;
  extern __shared__ double hs[];  // [n_bin * (1 + n_spec)] sums, then the ordered slots
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, ns = P.n_spec;
  const int nv = n_bin * (1 + ns);
  double* s_nc = hs + nv;                  // [TILE] number concentration, in bin order
  int* s_slot = (int*)(s_nc + TILE);  // [TILE]
  int* s_bin = s_slot + TILE;         // [TILE]
  int* cnt = s_bin + TILE;            // [n_bin]
  for (int k = threadIdx.x; k < nv; k += blockDim.x) hs[k] = 0.0;
  const double den0 = lane < ns ? P.density[lane] : 0.0, den1 = HI && lane + 32 < ns ? P.density[lane + 32] : 0.0;
  const int n = P.ctr->n_slots;
  const int per = (n_bin + kDistThreads - 1) / kDistThreads;  // bins a thread scans
  for (long long base = blockIdx.x * (long long)TILE; base < n; base += (long long)gridDim.x * TILE) {
    for (int k = threadIdx.x; k < n_bin; k += blockDim.x) cnt[k] = 0;
    __syncthreads();
    int b[kPer] = {}, rank[kPer];
    double nc[kPer];
#pragma unroll
    for (int u = 0; u < kPer; u++) {
      const long long i = base + u * kDistThreads + threadIdx.x;
      if (!(i < n && P.alive[i])) continue;
      const double r = vol2rad(P.benv.frac, P.vtot[i]);  // aero_particle_radius (fractal_vol2rad)
      const int bi = bin_find(n_bin, log_lo, log_hi, 2.0 * r);
      if (bi < 1 || bi > n_bin) continue;
      b[u] = bi;
      nc[u] = num_conc_at_radius<double>(P.w, P.cls[i] - 1, r) * inv_width;
      rank[u] = atomicAdd(&cnt[bi - 1], 1);
    }
    __syncthreads();
    // starts of the bins
    int mine = 0;
    for (int k = 0; k < per; k++) {
      const int c = (int)threadIdx.x * per + k;
      if (c < n_bin) mine += cnt[c];
    }
    int total;
    int at = block_excl_scan(mine, &total);
    for (int k = 0; k < per; k++) {
      const int c = (int)threadIdx.x * per + k;
      if (c < n_bin) {
        const int x = cnt[c];
        cnt[c] = at;
        at += x;
      }
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kPer; u++)
      if (b[u] > 0) {
        const int pos = cnt[b[u] - 1] + rank[u];
        s_slot[pos] = (int)base + u * kDistThreads + (int)threadIdx.x;
        s_bin[pos] = b[u] - 1;
        s_nc[pos] = nc[u];
      }
    __syncthreads();
    // the live particles shared out evenly over the warps
    const int share = (total + kDistThreads / 32 - 1) / (kDistThreads / 32);
    const int q0 = min(total, share * w), q1 = min(total, share * (w + 1));
    int cur = -1;
    double a0 = 0.0, a1 = 0.0, an = 0.0;
    auto flush = [&]() {
      if (cur < 0) return;
      double* hm = hs + n_bin + (size_t)cur * ns;
      if (lane < ns) atomicAdd(&hm[lane], a0);
      if (HI && lane + 32 < ns) atomicAdd(&hm[lane + 32], a1);
      if (lane == 31) atomicAdd(&hs[cur], an);
    };
    constexpr int kIn = HI ? 4 : 8;
    for (int p0 = q0; p0 < q1; p0 += kIn) {
      double v0[kIn], v1[HI ? kIn : 1];
#pragma unroll
      for (int u = 0; u < kIn; u++) {
        const int p = p0 + u < q1 ? p0 + u : q1 - 1;
        const double* v = P.vol + vol_at(P, s_slot[p], 0);
        v0[u] = lane < ns ? v[lane] : 0.0;
        if constexpr (HI) v1[u] = lane + 32 < ns ? v[lane + 32] : 0.0;
      }
#pragma unroll
      for (int u = 0; u < kIn; u++) {
        if (p0 + u >= q1) break;
        const int bp = s_bin[p0 + u];
        const double np = s_nc[p0 + u];
        if (bp != cur) {
          flush();
          cur = bp;
          a0 = a1 = an = 0.0;
        }
        a0 += np * v0[u] * den0;
        if constexpr (HI) a1 += np * v1[u] * den1;
        an += np;
      }
    }
    flush();
    __syncthreads();
  }
  __syncthreads();
  const int k0 = (int)(((long long)blockIdx.x * nv) / gridDim.x);
  for (int k = threadIdx.x; k < nv; k += blockDim.x) {
    const int j = k0 + k < nv ? k0 + k : k0 + k - nv;
    if (hs[j] != 0.0) atomicAdd(&out[j], hs[j]);
  }
}

// move live slots of src into dst compactly (relayout)
__global__ void k_relayout(PopDev S, PopDev D, const long long* live_off, int n_slots,
                           int compact) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_slots; i += gridDim.x * blockDim.x) {
    if (compact && !S.alive[i]) continue;
    int j = compact ? (int)live_off[i] : i;
    for (int s = 0; s < S.n_spec; s++) D.vol[vol_at(D, j, s)] = S.vol[vol_at(S, i, s)];
    D.vtot[j] = S.vtot[i];
    D.mass[j] = S.mass[i];
    D.rad[j] = S.rad[i];
    D.grp[j] = S.grp[i];
    D.cls[j] = S.cls[i];
    D.id[j] = S.id[i];
    D.nprim[j] = S.nprim[i];
    D.ncomp[j] = S.ncomp[i];
    for (int k = 0; k < S.ncomp[i]; k++) {
      D.csrc[comp_at(j, k)] = S.csrc[comp_at(i, k)];
      D.ctime[comp_at(j, k)] = S.ctime[comp_at(i, k)];
    }
    D.lct[j] = S.lct[i];
    D.gct[j] = S.gct[i];
    D.imf[j] = S.imf[i];
    D.den_ice[j] = S.den_ice[i];
    D.phi[j] = S.phi[i];
    D.hyst[j] = S.hyst[i];
    D.frozen[j] = S.frozen[i];
    D.alive[j] = S.alive[i];
    D.changed[j] = S.changed[i];
    D.cell[j] = S.cell[i];
    D.claim[j] = S.claim[i];
    D.rclaim[j] = S.rclaim[i];
    D.touched[j] = S.touched[i];
    D.recd[j] = S.recd[i];
    D.recf[j] = S.recf[i];
  }
  // growth keeps slot numbers, so the current cell list (positions below
  // n_slots) stays valid and is carried over; compaction renumbers slots
  // and the next sort rebuilds the list
  if (!compact)
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_slots; i += gridDim.x * blockDim.x)
      D.list[i] = S.list[i];
}

__global__ void k_eval_kernel(PopDev P, int n, const double* v1, const int* c1, const double* v2,
                              const int* c2, const int* cij, double* out, int precision) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  // records of the two particles, built as the sort pass builds them
  double vt1 = 0.0, vt2 = 0.0, m1 = 0.0, m2 = 0.0;
  for (int s = 0; s < P.n_spec; s++) {
    vt1 = vt1 + v1[(size_t)i * P.n_spec + s];
    vt2 = vt2 + v2[(size_t)i * P.n_spec + s];
  }
  for (int s = 0; s < P.n_spec; s++) {
    m1 = m1 + v1[(size_t)i * P.n_spec + s] * P.density[s];
    m2 = m2 + v2[(size_t)i * P.n_spec + s] * P.density[s];
  }
  RecD q[2];
  double vt[2] = {vt1, vt2}, ms[2] = {m1, m2};
  int cl[2] = {c1[i] - 1, c2[i] - 1};
  for (int k = 0; k < 2; k++) q[k] = make_rec_v(P, vol2rad(P.benv.frac, vt[k]), vt[k], ms[k], cl[k] + 1);
  int cc = cij[i] - 1;
  double k;
  if (precision == 0) {
    const double* a = (const double*)&q[0];
    const double* b = (const double*)&q[1];
    switch (P.kernel_type) {
      case kKernelAdditive: k = pair_kernel<kKernelAdditive, double, false>(P, a, b, cl[0], cl[1], cc, 0.0, P.coeff); break;
      case kKernelConstant: k = pair_kernel<kKernelConstant, double, false>(P, a, b, cl[0], cl[1], cc, 0.0, P.coeff); break;
      case kKernelBrown: k = pair_kernel<kKernelBrown, double, false>(P, a, b, cl[0], cl[1], cc, 0.0, P.coeff); break;
      case kKernelSedi: k = pair_kernel<kKernelSedi, double, false>(P, a, b, cl[0], cl[1], cc, 0.0, P.coeff); break;
      case kKernelBrownFree: k = pair_kernel<kKernelBrownFree, double, false>(P, a, b, cl[0], cl[1], cc, 0.0, P.coeff); break;
      case kKernelBrownCont: k = pair_kernel<kKernelBrownCont, double, false>(P, a, b, cl[0], cl[1], cc, 0.0, P.coeff); break;
      default: k = 0.0;
    }
  } else {
    float a[6], b[6];
    const double* qa = (const double*)&q[0];
    const double* qb = (const double*)&q[1];
    for (int j = 0; j < 6; j++) {
      a[j] = (float)qa[j];
      b[j] = (float)qb[j];
    }
    float kf;
    switch (P.kernel_type) {
      case kKernelAdditive: kf = pair_kernel<kKernelAdditive, float, false>(P, a, b, cl[0], cl[1], cc, 0.f, (float)P.coeff); break;
      case kKernelConstant: kf = pair_kernel<kKernelConstant, float, false>(P, a, b, cl[0], cl[1], cc, 0.f, (float)P.coeff); break;
      case kKernelBrown: kf = pair_kernel<kKernelBrown, float, false>(P, a, b, cl[0], cl[1], cc, 0.f, (float)P.coeff); break;
      case kKernelSedi: kf = pair_kernel<kKernelSedi, float, false>(P, a, b, cl[0], cl[1], cc, 0.f, (float)P.coeff); break;
      case kKernelBrownFree: kf = pair_kernel<kKernelBrownFree, float, false>(P, a, b, cl[0], cl[1], cc, 0.f, (float)P.coeff); break;
      case kKernelBrownCont: kf = pair_kernel<kKernelBrownCont, float, false>(P, a, b, cl[0], cl[1], cc, 0.f, (float)P.coeff); break;
      default: kf = 0.f;
    }
    k = kf;
  }
  out[i] = k;
}

// ---------------------------------------------------------------------------
// host side

#define CK(x)                                                          \
  do {                                                                 \
    cudaError_t e_ = (x);                                              \
    if (e_ != cudaSuccess) {                                           \
      snprintf(g_last_error, sizeof(g_last_error), "%s: %s (%s:%d)", #x, \
               cudaGetErrorString(e_), __FILE__, __LINE__);            \
      throw Fail(PMC_ERR_CUDA);                                        \
    }                                                                  \
  } while (0)

char g_last_error[512];
char g_last_assert[256];  // site and index of the last failed device bounds check
char g_last_capacity[256];  // which limit the last PMC_ERR_CAPACITY hit
[[noreturn]] void cap_throw(const char* why);
// kernel launches issued by this library (for the benchmark's launch count)
long long g_launches = 0;
inline void note_launch() { ++g_launches; }

struct Fail {
  int code;
  explicit Fail(int c) : code(c) {}
};

void cap_throw(const char* why) {
  cudaGetLastError();  // a failed allocation leaves an error behind
  snprintf(g_last_capacity, sizeof(g_last_capacity), "capacity exceeded: %s", why);
  throw Fail(PMC_ERR_CAPACITY);
}

template <class T>
struct DevBuf {
  T* p = nullptr;
  size_t n = 0;
  void reserve(size_t m) {
    if (m <= n) return;
    if (p) cudaFree(p);
    p = nullptr;
    // geometric growth: sizes that creep up step by step (slot counts,
    // sample counts) reallocate rarely
    size_t want = std::max<size_t>(std::max<size_t>(m, n + n / 2), 1024);
    n = 0;
    if (cudaMalloc(&p, want * sizeof(T)) != cudaSuccess) {
      p = nullptr;
      cap_throw("device memory: an allocation failed");
    }
    n = want;
  }
  void release() {
    if (p) cudaFree(p);
    p = nullptr;
    n = 0;
  }
};

// page-locked host staging (cudaHostAlloc), grown on demand
struct PinnedBuf {
  void* p = nullptr;
  size_t bytes = 0;
  void reserve(size_t b) {
    if (b <= bytes) return;
    if (p) cudaFreeHost(p);
    p = nullptr;
    bytes = 0;
    size_t want = std::max<size_t>(b + b / 4, 1 << 20);
    if (cudaHostAlloc(&p, want, cudaHostAllocDefault) != cudaSuccess) {
      p = nullptr;
      cap_throw("page-locked host memory: an allocation failed");
    }
    bytes = want;
  }
  void release() {
    if (p) cudaFreeHost(p);
    p = nullptr;
    bytes = 0;
  }
};

// page-locked host memory that the device writes directly (mapped into the
// device's address space), grown on demand
struct MappedBuf {
  void* p = nullptr;    // host address
  void* dev = nullptr;  // device address of the same memory
  size_t bytes = 0;
  void reserve(size_t b) {
    if (b <= bytes) return;
    release();
    size_t want = b + b / 4;
    if (cudaHostAlloc(&p, want, cudaHostAllocMapped) != cudaSuccess ||
        cudaHostGetDevicePointer(&dev, p, 0) != cudaSuccess) {
      cudaGetLastError();
      release();
      cap_throw("mapped host memory: an allocation failed");
    }
    bytes = want;
  }
  void release() {
    if (p) cudaFreeHost(p);
    p = dev = nullptr;
    bytes = 0;
  }
};

// Persistent host workers for the scatter of pmc_coag_gpu_sync_host: run(n,
// f) calls f(q, n) for q = 0..n-1 on n threads (the caller's among them) and
// returns when all are done.
class HostPool {
 public:
  ~HostPool() {
    {
      std::lock_guard<std::mutex> l(mu_);
      stop_ = true;
    }
    cv_.notify_all();
    for (auto& t : th_) t.join();
  }
  void run(int n, const std::function<void(int, int)>& f) {
    if (n <= 1) {
      f(0, 1);
      return;
    }
    while ((int)th_.size() < n - 1) {
      int q = (int)th_.size() + 1;
      th_.emplace_back([this, q] { loop(q); });
    }
    {
      std::lock_guard<std::mutex> l(mu_);
      job_ = &f;
      n_ = n;
      left_ = n - 1;
      gen_++;
    }
    cv_.notify_all();
    f(0, n);
    std::unique_lock<std::mutex> l(mu_);
    done_.wait(l, [this] { return left_ == 0; });
    job_ = nullptr;
  }

 private:
  void loop(int q) {
    unsigned long long seen = 0;
    for (;;) {
      const std::function<void(int, int)>* f;
      int n;
      {
        std::unique_lock<std::mutex> l(mu_);
        cv_.wait(l, [&] { return stop_ || gen_ != seen; });
        if (stop_) return;
        seen = gen_;
        f = job_;
        n = n_;
      }
      if (q < n) (*f)(q, n);
      std::lock_guard<std::mutex> l(mu_);
      if (q < n && --left_ == 0) done_.notify_one();
    }
  }
  std::vector<std::thread> th_;
  std::mutex mu_;
  std::condition_variable cv_, done_;
  const std::function<void(int, int)>* job_ = nullptr;
  int n_ = 0, left_ = 0;
  unsigned long long gen_ = 0;
  bool stop_ = false;
};

struct PopHost {
  PopDev h{};
  bool valid_sort = false;
  int n_bin = 0;
  std::vector<double> edges, centers;
  // owned allocations (freed on relayout / destroy)
  std::vector<void*> slot_allocs;
  std::vector<void*> sort_allocs;
  std::vector<void*> fixed_allocs;
  PopDev none{};  // its sort structures, those of no bins, stay for good (fixed_allocs)
  uint64_t seed = 1;
  uint32_t step = 0;
  uint32_t dev_step = 0;  // the step count of the device's copy of h
  int kmax_kt = 0;  // kernel type of the current k_max table
  bool own_w = false;  // weights set for this population alone
  // host copy kept slot by slot (pmc_coag_gpu_sync_host): refreshed in full
  // after an upload or a compaction, else by the slots written since
  bool mirror_full = true;
  int mirror_slots = 0;
  uint32_t rebalance_calls = 0;  // halving draws: one stream per call
  uint32_t sample_calls = 0;     // initial-condition samples: one stream per call
  Weights w{};
  int chunk_hist_cap = 0;
  // per-slot radius/bin/record caches are valid for this grid, kernel,
  // environment and weights
  bool caches_valid = false;
  int key_kt = 0, key_wver = -1;
  int wver = 0;  // bumped when this population's weights change
  double key_temp = 0, key_press = 0, key_coeff = 0;
  long long rm_count = 0;  // removal records on the device at the last counter read
};

// Launch shapes of the step that the autotuner chooses: threads per block
// at five launch sites.  Every kernel there walks its work with a
// grid-stride loop and keeps no per-block state, every draw is keyed by
// index and every counter is a sum, so the particles do not depend on these
// shapes, and tuning runs on the caller's own steps.
enum TuneSite : int { kTuneTest, kTuneResolve, kTuneItems, kTuneChain, kTuneApply, kTuneSites };
constexpr int kTuneCands = 3;
// candidates per site (within each kernel's __launch_bounds__)
constexpr int kTuneCand[kTuneSites][kTuneCands] = {
    {64, 128, 256},  // k_test: one pair test per thread
    {64, 128, 256},  // k_resolve: one event per thread
    {64, 128, 256},  // k_items: one walk per thread
    {32, 64, 128},   // k_chain: one chain per thread
    {64, 128, 256},  // k_apply: one event per thread
};
constexpr int kTuneReps = 3;  // steps per candidate
struct Tune {
  int threads[kTuneSites] = {256, 256, 256, 128, 256};
};
// Coordinate search, one site at a time.  While it runs the later rounds
// are launched from the host loop (the same particles as the graph), so
// that every launch of the site being searched can be bracketed by CUDA
// events.  A candidate's score is the device time of the site's launches
// over its kTuneReps steps divided by those steps' pair tests: the site's
// cost per unit of work, which does not drift with the state as the whole
// step's time does.  The site keeps its best candidate before the next site
// is searched.
struct Tuner {
  bool on = false;
  int site = 0, cand = 0, rep = 0, best = 0;
  float best_ms = 0.f;           // best score (ms per million pair tests)
  double cand_ms = 0.0;          // the candidate's site time so far (ms)
  long long cand_tests = 0;      // and its steps' pair tests
  float site_ms[kTuneSites][kTuneCands] = {};
  std::vector<std::pair<cudaEvent_t, cudaEvent_t>> pending;  // this step's launches of the site
  std::vector<cudaEvent_t> spare;
};

void pool_release(int dev);
struct PoolRef {  // a context's hold on its device's memory pool
  int dev = -1;
  ~PoolRef() {
    if (dev >= 0) pool_release(dev);
  }
};

struct Ctx {
  int n_pop = 1, n_spec = 1, n_group = 1, n_class = 1, i_water = 0;
  std::vector<double> density;
  Weights w{};
  int wver = 0;  // bumped on every weight change
  int mode = PMC_MODE_FP64;
  std::vector<PopHost> pops;
  PopDev* d_pops = nullptr;
  PopCtr* d_ctrs = nullptr;  // one counter block per population
  uint32_t* d_round = nullptr;  // [round of the current step, claim generation], read by the kernels
  uint32_t claim_gen = 0;
  bool dirty = true;            // host PopDev copies changed since the last push
  std::vector<PopCtr> h_ctrs;
  MappedBuf report;                // the step graph's report and counters, then its sequence number
  DevBuf<unsigned> report_seq;
  unsigned report_count = 0;
  cudaStream_t stream = nullptr;
  int max_rounds = 200;  // below 256: the round is 8 bits of the random streams' counters
  int n_sm = 148;        // multiprocessors of the device
  // later rounds as a CUDA graph
  bool use_graph = true;
  cudaStream_t cap_stream = nullptr;  // capture stream
  cudaMemPool_t mem = nullptr;        // the populations' arrays (dalloc)
  PoolRef mem_ref;
  cudaStream_t side_stream = nullptr;  // a branch of a captured step
  cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
  bool fork = false;                   // capturing: independent launches go to branches
  bool chained = false;                // capturing a step: launch_chained
  cudaGraph_t rg_graph = nullptr;
  cudaGraphExec_t rg_exec = nullptr;
  std::vector<long long> rg_key;
  std::vector<long long> rg_seen;  // the key of the previous step's later rounds
  int rg_held = 0;                 // steps in a row that had it
  long long rg_nodes = 0, rg_builds = 0;
  DevBuf<long long> graph_stats;
  // the whole step as one graph (run_step_graph)
  cudaGraph_t sg_graph = nullptr;
  cudaGraphExec_t sg_exec = nullptr;
  std::vector<long long> sg_key, sg_seen;
  int sg_pause = 0;                  // steps left that go the long way (kGraphPause)
  long long sg_w = 0, sg_e = 0;      // samples and items it holds room for
  long long sg_q = 0, sg_qb = 0;     // target operations of round 0 and of a later round
  long long sg_nodes0 = 0, sg_nodes = 0;  // launches of its round 0 and of one later round
  cudaEvent_t sg_ev[6] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};  // when profiling: sort, tests, later rounds
  long long* d_stat = nullptr;       // kStatWords words before the counter blocks, read back with them
  // the last step's samples, largest items and target operations of a later
  // round, target operations of round 0 and largest removal bound
  long long last_w = -1, last_e0 = 0, last_qb = 0, last_q = 0, last_rm = 0;
  bool ctrs_fresh = false;           // h_ctrs and n_slots_host are the device's counters
  Tune tune;
  Tuner tuner;
  // removal pool of the round's target operations
  DevBuf<int> pp_rm_pool;
  DevBuf<uint8_t> pop_on;  // the populations a refresh covers
  // a batched round's lists grouped by population (group_by_pop)
  DevBuf<int> grp_hist, item_pop;
  DevBuf<long long> grp_off, grp_dest;
  // walkers of the round's operations, one place per operation and copy
  DevBuf<int> wk_slot, wk_gp;
  DevBuf<uint8_t> wk_flag;
  DevBuf<long long> pp_rm_off, pp_rm_tot;
  // initial-condition sampler: staging of the modes, copy counts, radix select
  DevBuf<double> sample_buf;
  DevBuf<int> dup_n;
  DevBuf<unsigned char> select_buf;
  size_t sort_smem = 0;  // dynamic shared memory the sort grid was sized for
  int sort_blocks = 0;   // co-resident sort blocks at that size
  // per-round buffers
  DevBuf<int> gpair_pop, gpair_local;
  DevBuf<long long> pop_pair_base;
  DevBuf<long long> nwork_set, nwork_pp, work_off, pp_off;
  DevBuf<uint8_t> flag, win_set, win_pp;
  DevBuf<uint32_t> dec_set;  // merge decision of each event (drawn when the event is formed)
  DevBuf<int> ev_gp, gp_c;   // global pair of each accepted sample / event
  DevBuf<int2> ev_c;         // slots of each event
  DevBuf<unsigned long long> ev_key;  // key of each event (make_key)
  DevBuf<float> ev_pos;      // position of each event in its pair's test sequence
  DevBuf<int> ev_dest;       // slot of the particle each event made (-1: none)
  DevBuf<int> ev_len, ev_head, ev_app;  // chains: events, first chunk, events applied
  DevBuf<uint8_t> ev_done;   // chains: the walk ran to the end
  DevBuf<int> chain_list;    // the round's winning chains (round_dev[4] of them)
  DevBuf<int2> ev;
  // a later round's items (one per event of the round before) and what they made
  DevBuf<uint8_t> it_flag, it_done;
  DevBuf<unsigned long long> it_key;
  DevBuf<int2> it_c;
  DevBuf<int> it_gp, it_len, it_head, it_start;
  DevBuf<float> it_pos;
  DevBuf<uint32_t> it_dec, it_gused;
  DevBuf<int4> it_term, ev_term;  // pending tests where chains stopped (kPendingTerm)
  // walkers made by target operations (slot, global pair), read by the next
  // round's k_items; their count is round_dev[5]
  DevBuf<int> ppw_slot, ppw_gp;  // read by a round's k_items, then written by its k_compact_walkers
  long long op_cap = 0;   // room in the target-operation arrays this round
  bool pp_step = false;   // the step has target operations (per-particle path), or one of the last kPPIdle had
  int pp_idle = 0;        // graph steps since one that had
  // chain events of a round (ChainPool), in chunks
  DevBuf<int> ch_y, ch_q;
  DevBuf<float> ch_pos;
  long long ch_chunks = 0;
  DevBuf<int> lost_pp;
  DevBuf<long long> rank_slot_set, rank_id_set, rank_slot_pp, lost_off;
  DevBuf<int> op_pop, op_pair, op_slot, op_k, r_pop, r_pair, r_slot, r_k;
  DevBuf<unsigned long long> op_key, r_key;
  DevBuf<PPResult> pp_res;
  DevBuf<double> pp_vol;
  DevBuf<int> per_pop_i;  // 4 x n_pop counters
  DevBuf<int> slot_base_set, slot_base_pp;
  DevBuf<long long> id_base_set, id_base_pp;
  DevBuf<unsigned long long> scan_status;  // look-back tile words
  size_t scan_status_n = 0;                // words cleared so far
  DevBuf<unsigned> scan_ctr;               // per-job tile and finished-block counters (re-armed by the kernel)
  DevBuf<unsigned long long> scan_err;     // look-backs that gave up
  DevBuf<long long> n_dev;  // device scalars
  // staging for upload / download (shared by all populations; every call
  // synchronises before it returns)
  DevBuf<double> st_d;
  DevBuf<int> st_i;
  DevBuf<long long> st_l;
  PinnedBuf pin;  // host staging of the changed slots
  MappedBuf map;  // packed changed slots, written by the device into host memory
  cudaEvent_t sync_ev[4] = {nullptr, nullptr, nullptr, nullptr};  // chunks of a host sync
  DevBuf<unsigned long long> st_cnt;        // their count
  std::unique_ptr<HostPool> pool;           // scatter workers
  long long h_total = 0;
  // stats of the last step
  long long last_redraws = 0, last_rounds = 0, last_kmax_warn = 0, exact_tests = 0;
  long long last_set_losers = 0, last_pp_lost = 0, last_events = 0, last_ops = 0;
  // optional per-kernel timing with CUDA events on the library's stream:
  // 0 pair tests, 1 sorts (k_sort_all), 2 later-round graph launches,
  // 3 whole steps
  bool prof = false;
  struct ProfPair {
    int id;
    long long units;
    cudaEvent_t e0, e1;
  };
  std::vector<ProfPair> prof_pending;
  std::vector<cudaEvent_t> prof_free;
  // host copy of each population's slot count, kept current after every
  // round so the sort can size itself without reading the device
  std::vector<int> n_slots_host;
  // device scalars of a round: [0] events that lost a claim, [1] events,
  // [2] items (the events of the round before), [3] chain chunks handed out,
  // [4] winning chains of the round
  DevBuf<long long> round_dev;
  std::vector<long long> base_cached;  // pair-list layout last uploaded
  double prof_ms[4] = {0, 0, 0, 0};
  long long prof_launch[4] = {0, 0, 0, 0}, prof_units[4] = {0, 0, 0, 0};
  // replay
  DevBuf<double> replay_u;
  long long replay_n = 0, replay_used = 0;
  ReplayBuffers replay;
  // particle shape of aero_data (fractal_t); spherical unless set
  Fractal frac = fractal_spherical();
};

// Population arrays come from a memory pool, in the order of the context's
// stream: a server's slot is emptied and filled again for every job, and
// the 76 cudaMalloc and cudaFree calls of that (each a device
// synchronisation) made emptying and uploading take 19.2 ms at 1e6 particles
// of 20 species, 3.0 ms of it the copy, and 3.2 ms a population in a context
// of 256; from the pool 3.3 and 0.4 ms.
// One pool per device, shared by its contexts (the driver orders memory that
// moves between their streams; a pool per context took 1 ms to create); it
// keeps at most kPoolKeep bytes that are not in use past a synchronisation
// (a cudaMalloc of the process that would fail gets them: measured with 1 GiB
// on a device with 49 MiB free), and the last context to go gives back all but
// kPoolIdle.  For the process stay the pool itself with its first block (its
// unit is 32 MiB), and one page of page-locked memory: the first such
// allocation of a process maps a block that later small ones share (1 to 3 ms,
// then 5 us each), and freeing the last unmaps it.  A program that makes a
// context for each job paid for both every time: 6.8 ms for a context that
// takes 1000 particles through 3 steps, now 3.6 (4.1 with nothing kept of the
// pool; 3.5 with cudaMalloc and cudaFree).
constexpr uint64_t kPoolKeep = 4ULL << 30, kPoolIdle = 32ULL << 20;

struct DevicePools {
  std::mutex mu;
  std::vector<std::pair<cudaMemPool_t, int>> by_dev;  // pool, contexts
  void* page = nullptr;  // page-locked
};
DevicePools& device_pools() {
  static DevicePools* p = new DevicePools();  // lives until the process ends: contexts may be destroyed at exit
  return *p;
}

cudaMemPool_t pool_acquire(int dev) {
  DevicePools& d = device_pools();
  std::lock_guard<std::mutex> l(d.mu);
  if ((int)d.by_dev.size() <= dev) d.by_dev.resize(dev + 1, {nullptr, 0});
  if (!d.page && cudaHostAlloc(&d.page, 4096, cudaHostAllocMapped) != cudaSuccess) {
    cudaGetLastError();  // a saving only
    d.page = nullptr;
  }
  auto& e = d.by_dev[dev];
  if (!e.first) {
    cudaMemPoolProps mp = {};
    mp.allocType = cudaMemAllocationTypePinned;
    mp.handleTypes = cudaMemHandleTypeNone;
    mp.location.type = cudaMemLocationTypeDevice;
    mp.location.id = dev;
    CK(cudaMemPoolCreate(&e.first, &mp));
    uint64_t keep = kPoolKeep;
    CK(cudaMemPoolSetAttribute(e.first, cudaMemPoolAttrReleaseThreshold, &keep));
  }
  e.second++;
  return e.first;
}

void pool_release(int dev) {
  DevicePools& d = device_pools();
  std::lock_guard<std::mutex> l(d.mu);
  auto& e = d.by_dev[dev];
  if (--e.second == 0) cudaMemPoolTrimTo(e.first, kPoolIdle);
}

void free_list(Ctx& c, std::vector<void*>& v) {
  for (void* p : v) cudaFreeAsync(p, c.stream);
  v.clear();
}

template <class T>
T* dalloc(Ctx& c, std::vector<void*>& owner, size_t n) {
  void* p = nullptr;
  const size_t bytes = std::max<size_t>(n, 1) * sizeof(T);
  if (cudaMallocFromPoolAsync(&p, bytes, c.mem, c.stream) != cudaSuccess) {
    // what the pool holds unused may be in other sizes: give it back first
    cudaGetLastError();
    cudaStreamSynchronize(c.stream);
    cudaMemPoolTrimTo(c.mem, 0);
    if (cudaMallocFromPoolAsync(&p, bytes, c.mem, c.stream) != cudaSuccess)
      cap_throw("device memory: an allocation failed");
  }
  owner.push_back(p);
  return (T*)p;
}

// Launch k on st.  In a captured step (c.chained) it starts while the kernel
// before it in the stream ends (programmatic dependent launch): every kernel
// launched this way begins with chain_wait(), which waits for that kernel and
// its writes, so only the launch itself overlaps, 1 to 1.5 us of a step's 20
// to 25 kernels that mostly run 3 to 10 us.
template <class... KA, class... A>
void launch_chained(Ctx& c, void (*k)(KA...), dim3 g, dim3 b, size_t smem, cudaStream_t st, A... a) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = g;
  cfg.blockDim = b;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = c.chained ? 1 : 0;
  CK(cudaLaunchKernelEx(&cfg, k, KA(a)...));
  note_launch();
}

int grid_for(long long n, int threads) {
  long long b = (n + threads - 1) / threads;
  if (b < 1) b = 1;
  if (b > 148 * 16) b = 148 * 16;
  return (int)b;
}

// k_kmax_table over every population whose table is not current, with room in
// shared memory for the Brownian kernel's halves of the largest; a block goes
// over at least 16 sets of pairs, so that filling that table is the smaller
// part
void launch_kmax(Ctx& c) {
  int nb = 1, nb_brown = 0;
  for (const PopHost& ph : c.pops) {
    nb = std::max(nb, ph.n_bin);
    if (ph.h.kernel_type == kKernelBrown) nb_brown = std::max(nb_brown, ph.n_bin);
  }
  const int max_part = 9 * nb_brown;
  const size_t smem = sizeof(BrownPart) * (size_t)max_part;
  if (smem > 48 * 1024)
    CK(cudaFuncSetAttribute(k_kmax_table, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int sets = (nb * nb + kKmaxPairs - 1) / kKmaxPairs;
  const int blocks = std::max(std::min(sets, std::max(1, c.n_sm / c.n_pop)), (sets + 15) / 16);
  k_kmax_table<<<dim3((unsigned)blocks, (unsigned)c.n_pop), kKmaxThreads, smem, c.stream>>>(c.d_pops, max_part);
  note_launch();
}

// Times the launches issued inside its scope when profiling is on: a pair
// of CUDA events on the library's stream, read back only when the totals
// are asked for, so timing adds no synchronisation to the step.
struct ProfScope {
  Ctx& c;
  int id;
  long long units;
  cudaEvent_t e0 = nullptr;
  ProfScope(Ctx& c_, int id_, long long units_) : c(c_), id(id_), units(units_) {
    if (!c.prof) return;
    e0 = prof_event(c);
    cudaEventRecord(e0, c.stream);
  }
  ~ProfScope() {
    if (!c.prof || !e0) return;
    cudaEvent_t e1 = prof_event(c);
    cudaEventRecord(e1, c.stream);
    c.prof_pending.push_back({id, units, e0, e1});
  }
  static cudaEvent_t prof_event(Ctx& c) {
    if (!c.prof_free.empty()) {
      cudaEvent_t e = c.prof_free.back();
      c.prof_free.pop_back();
      return e;
    }
    cudaEvent_t e = nullptr;
    cudaEventCreate(&e);
    return e;
  }
};

// fold the recorded event pairs into the per-kernel totals
void prof_collect(Ctx& c) {
  if (c.prof_pending.empty()) return;
  cudaStreamSynchronize(c.stream);
  for (auto& p : c.prof_pending) {
    float ms = 0.f;
    cudaEventElapsedTime(&ms, p.e0, p.e1);
    c.prof_ms[p.id] += ms;
    c.prof_launch[p.id] += 1;
    c.prof_units[p.id] += p.units;
    c.prof_free.push_back(p.e0);
    c.prof_free.push_back(p.e1);
  }
  c.prof_pending.clear();
}

// exclusive scans of in[0..n) into out[0..n] (out[n] = total), up to
// kScanMaxJobs arrays of one element type in one launch.  With nd, a job's
// count is *nd (device memory) and n only bounds it.
template <class T>
struct ScanArg {
  const T* in;
  long long n;
  const long long* nd;
  long long* out;
  long long* total_out = nullptr;
};

// room for n look-back words; fresh memory is cleared once
void reserve_scan_status(Ctx& c, size_t n, cudaStream_t st) {
  if (n > c.scan_status.n) c.scan_status_n = 0;  // also if this fails
  c.scan_status.reserve(n);
  if (c.scan_status.n > c.scan_status_n) {
    CK(cudaMemsetAsync(c.scan_status.p, 0, sizeof(unsigned long long) * c.scan_status.n, st));
    c.scan_status_n = c.scan_status.n;
  }
}

template <class T>
void scan_multi(Ctx& c, std::initializer_list<ScanArg<T>> args, cudaStream_t st = nullptr) {
  if (!st) st = c.stream;
  ScanJobs jobs{};
  int k = 0;
  long long nb = 1;
  for (const auto& a : args) {
    jobs.j[k].in = a.in;
    jobs.j[k].out = a.out;
    jobs.j[k].n_max = a.n;
    jobs.j[k].nd = a.nd;
    jobs.j[k].total_out = a.total_out;
    nb = std::max(nb, (a.n + kScanTile - 1) / kScanTile);
    k++;
  }
  if (k == 0) return;
  if (nb > (1LL << 30)) cap_throw("scan longer than its tile limit");
  reserve_scan_status(c, (size_t)kScanMaxJobs * nb, st);
  dim3 g((unsigned)nb, (unsigned)k);
  launch_chained(c, k_scan_lb<T>, g, dim3(kScanThreads), 0, st, jobs, c.scan_status.p, (int)nb, c.scan_ctr.p,
                 c.scan_ctr.p + kScanMaxJobs, c.scan_err.p);
}

long long compact_tiles(long long n) { return std::max<long long>(1, (n + kCompactTile - 1) / kCompactTile); }

// shared words of a tiled launch of at most `tiles` blocks
TileCtl tile_ctl(Ctx& c, long long tiles, cudaStream_t st) {
  if (tiles > (1LL << 30)) cap_throw("scan longer than its tile limit");
  reserve_scan_status(c, (size_t)std::max<long long>(tiles, 1), st);
  return TileCtl{c.scan_status.p, c.scan_ctr.p, c.scan_ctr.p + kScanMaxJobs, c.scan_err.p};
}

template <class T>
void scan_dev(Ctx& c, const T* in, long long n, const long long* nd, long long* out) {
  scan_multi<T>(c, {ScanArg<T>{in, n, nd, out}});
}

// a look-back that gave up is reported as a timed-out step
void check_scan_err(Ctx& c) {
  unsigned long long e = 0;
  CK(cudaMemcpyAsync(&e, c.scan_err.p, sizeof(e), cudaMemcpyDeviceToHost, c.stream));
  CK(cudaStreamSynchronize(c.stream));
  if (e) {
    CK(cudaMemsetAsync(c.scan_err.p, 0, sizeof(e), c.stream));
    throw Fail(PMC_ERR_TIMEOUT);
  }
}

template <class T>
long long scan(Ctx& c, const T* in, long long n, long long* out, bool read_total) {
  scan_dev(c, in, n, (const long long*)nullptr, out);
  if (!read_total) return -1;
  long long t = 0;
  CK(cudaMemcpyAsync(&t, out + n, sizeof(long long), cudaMemcpyDeviceToHost, c.stream));
  CK(cudaStreamSynchronize(c.stream));
  check_scan_err(c);
  return t;
}

void push_pops(Ctx& c) {
  std::vector<PopDev> v(c.n_pop);
  for (int k = 0; k < c.n_pop; k++) {
    v[k] = c.pops[k].h;
    v[k].round_p = c.d_round;
    v[k].gen_p = c.d_round + 1;
    c.pops[k].dev_step = v[k].step;
  }
  CK(cudaMemcpyAsync(c.d_pops, v.data(), sizeof(PopDev) * c.n_pop, cudaMemcpyHostToDevice, c.stream));
  c.dirty = false;
}

// words of the step graph's report, in front of the counter blocks:
// [0..3] and [6..11] as k_round_end's stats, [4] why round 0 was not run
// (kNoGo*, 0: it was), [5] samples, [12] target operations of round 0
constexpr int kStatWords = 16;

// counters of every population in one copy
std::vector<PopCtr>& read_ctrs(Ctx& c) {
  c.h_ctrs.resize(c.n_pop);
  CK(cudaMemcpyAsync(c.h_ctrs.data(), c.d_ctrs, sizeof(PopCtr) * c.n_pop, cudaMemcpyDeviceToHost, c.stream));
  CK(cudaStreamSynchronize(c.stream));
  return c.h_ctrs;
}

void write_ctrs(Ctx& c) {
  c.ctrs_fresh = false;
  CK(cudaMemcpyAsync(c.d_ctrs, c.h_ctrs.data(), sizeof(PopCtr) * c.n_pop, cudaMemcpyHostToDevice, c.stream));
  CK(cudaStreamSynchronize(c.stream));
}

PopCtr read_ctr(Ctx& c, int k) { return read_ctrs(c)[k]; }

void write_ctr(Ctx& c, int k, const PopCtr& r) {
  c.ctrs_fresh = false;
  CK(cudaMemcpyAsync(c.d_ctrs + k, &r, sizeof(PopCtr), cudaMemcpyHostToDevice, c.stream));
  CK(cudaStreamSynchronize(c.stream));
}

// allocate slot arrays of capacity cap into h, owned by o: all of them, or an
// error and none
void alloc_slots(Ctx& c, PopDev& h, std::vector<void*>& o, int cap) try {
  h.cap = cap;
  h.vol = dalloc<double>(c, o, (size_t)cap * c.n_spec);
  h.vtot = dalloc<double>(c, o, cap);
  h.mass = dalloc<double>(c, o, cap);
  h.rad = dalloc<double>(c, o, cap);
  h.grp = dalloc<int>(c, o, cap);
  h.cls = dalloc<int>(c, o, cap);
  h.id = dalloc<long long>(c, o, cap);
  h.nprim = dalloc<int>(c, o, cap);
  h.ncomp = dalloc<int>(c, o, cap);
  h.csrc = dalloc<int>(c, o, (size_t)cap * kMaxComponent);
  h.ctime = dalloc<double>(c, o, (size_t)cap * kMaxComponent);
  h.lct = dalloc<double>(c, o, cap);
  h.gct = dalloc<double>(c, o, cap);
  h.imf = dalloc<double>(c, o, cap);
  h.den_ice = dalloc<double>(c, o, cap);
  h.phi = dalloc<double>(c, o, cap);
  h.hyst = dalloc<int>(c, o, cap);
  h.frozen = dalloc<int>(c, o, cap);
  h.alive = dalloc<uint8_t>(c, o, cap);
  h.changed = dalloc<uint8_t>(c, o, cap);
  h.cell = dalloc<int>(c, o, cap);
  h.list = dalloc<int>(c, o, cap);
  h.recd = dalloc<RecD>(c, o, cap);
  h.recf = dalloc<RecF>(c, o, cap);
  h.claim = dalloc<unsigned long long>(c, o, cap);
  h.rclaim = dalloc<unsigned long long>(c, o, cap);
  h.touched = dalloc<uint32_t>(c, o, cap);
  CK(cudaMemsetAsync(h.alive, 0, cap, c.stream));
  CK(cudaMemsetAsync(h.changed, 0, cap, c.stream));
  CK(cudaMemsetAsync(h.claim, 0xff, sizeof(unsigned long long) * cap, c.stream));  // no claim
  CK(cudaMemsetAsync(h.rclaim, 0xff, sizeof(unsigned long long) * cap, c.stream));
  CK(cudaMemsetAsync(h.touched, 0xff, sizeof(uint32_t) * cap, c.stream));        // no generation
  c.dirty = true;
} catch (...) {
  free_list(c, o);
  throw;
}

// sort structures of a grid of n_bin bins into h, owned by o
void fill_sort(Ctx& c, PopDev& h, std::vector<void*>& o, int n_bin) {
  int nb = std::max(n_bin, 1);
  h.n_cells = nb * c.n_class;
  h.chunk_hist = nullptr;  // allocated by the sort when needed
  h.chunk_hist_len = 0;
  h.cell_count = dalloc<int>(c, o, h.n_cells);
  h.cell_start = dalloc<int>(c, o, h.n_cells + 1);
  h.kmax_tab = dalloc<double>(c, o, (size_t)nb * nb);
  // pairs in the reference's loop order (coagulation.F90:74-94)
  std::vector<PairDesc> pair_desc;
  for (int c1 = 0; c1 < c.n_class; c1++)
    for (int c2 = 0; c2 <= c1; c2++)
      for (int b1 = 0; b1 < n_bin; b1++)
        for (int b2 = (c1 == c2 ? b1 : 0); b2 < n_bin; b2++) {
          PairDesc d;
          d.b1 = (int16_t)b1;
          d.b2 = (int16_t)b2;
          d.c1 = (int8_t)c1;
          d.c2 = (int8_t)c2;
          d.pad0 = d.pad1 = 0;
          pair_desc.push_back(d);
        }
  h.n_pairs = (int)pair_desc.size();
  if (h.n_pairs >= (1 << 20)) cap_throw("more than 2^20 bin pairs");  // pair numbers in keys and random streams
  // the pairs of each cell in loop order, for walks
  {
    std::vector<int> off(h.n_cells + 1, 0), list;
    for (const PairDesc& d : pair_desc) {
      off[d.b1 + nb * d.c1 + 1]++;
      if (d.b2 + nb * d.c2 != d.b1 + nb * d.c1) off[d.b2 + nb * d.c2 + 1]++;
    }
    for (int k = 0; k < h.n_cells; k++) off[k + 1] += off[k];
    list.assign(std::max(off[h.n_cells], 1), 0);
    std::vector<int> fill(off.begin(), off.end() - 1);
    for (int p = 0; p < h.n_pairs; p++) {
      const PairDesc& d = pair_desc[p];
      int a = d.b1 + nb * d.c1, b = d.b2 + nb * d.c2;
      list[fill[a]++] = p;
      if (b != a) list[fill[b]++] = p;
    }
    int max_len = 1;
    for (int k = 0; k < h.n_cells; k++) max_len = std::max(max_len, off[k + 1] - off[k]);
    const int n_coarse = ((max_len + 15) / 16 + 3) / 4 * 4;
    std::vector<int> coarse((size_t)h.n_cells * n_coarse, INT_MAX);
    for (int k = 0; k < h.n_cells; k++)
      for (int j = off[k], i = 0; j < off[k + 1]; j += 16, i++) coarse[(size_t)k * n_coarse + i] = list[j];
    int* d_coarse = dalloc<int>(c, o, coarse.size());
    CK(cudaMemcpyAsync(d_coarse, coarse.data(), sizeof(int) * coarse.size(), cudaMemcpyHostToDevice, c.stream));
    h.cp_coarse = d_coarse;
    h.n_coarse = n_coarse;
    int* d_off = dalloc<int>(c, o, off.size());
    int* d_list = dalloc<int>(c, o, list.size());
    h.cp_cum = dalloc<double>(c, o, (size_t)off[h.n_cells] + h.n_cells);
    h.cp_ent = dalloc<int4>(c, o, std::max(off[h.n_cells], 1));
    h.cp_nstop = dalloc<int>(c, o, std::max(off[h.n_cells], 1));
    h.cp_tab = dalloc<int>(c, o, (size_t)h.n_cells * kWalkTab);
    CK(cudaMemcpyAsync(d_off, off.data(), sizeof(int) * off.size(), cudaMemcpyHostToDevice, c.stream));
    CK(cudaMemcpyAsync(d_list, list.data(), sizeof(int) * list.size(), cudaMemcpyHostToDevice, c.stream));
    // copies from pageable memory are staged before they return, so the host
    // vectors may go
    h.cp_off = d_off;
    h.cp_list = d_list;
  }
  PairDesc* pd = dalloc<PairDesc>(c, o, std::max<size_t>(pair_desc.size(), 1));
  if (!pair_desc.empty())
    CK(cudaMemcpyAsync(pd, pair_desc.data(), sizeof(PairDesc) * pair_desc.size(),
                       cudaMemcpyHostToDevice, c.stream));
  h.pair_desc = pd;
  h.pair = dalloc<PairState>(c, o, std::max<size_t>(pair_desc.size(), 1));
  h.kmax_valid = 0;
  h.pair_setup_valid = 0;
}

// the sort structures of src (fill_sort) as dst's
void take_sort(PopDev& dst, const PopDev& src) {
  dst.n_cells = src.n_cells;
  dst.chunk_hist = src.chunk_hist;
  dst.chunk_hist_len = src.chunk_hist_len;
  dst.cell_count = src.cell_count;
  dst.cell_start = src.cell_start;
  dst.kmax_tab = src.kmax_tab;
  dst.n_pairs = src.n_pairs;
  dst.cp_off = src.cp_off;
  dst.cp_list = src.cp_list;
  dst.cp_cum = src.cp_cum;
  dst.cp_ent = src.cp_ent;
  dst.cp_nstop = src.cp_nstop;
  dst.cp_tab = src.cp_tab;
  dst.cp_coarse = src.cp_coarse;
  dst.n_coarse = src.n_coarse;
  dst.pair_desc = src.pair_desc;
  dst.pair = src.pair;
  dst.kmax_valid = 0;
  dst.pair_setup_valid = 0;
}

// no grid, with the sort structures that stay
void no_grid(Ctx& c, PopHost& ph) {
  free_list(c, ph.sort_allocs);
  take_sort(ph.h, ph.none);
  ph.n_bin = 0;
  ph.chunk_hist_cap = 0;
  c.dirty = true;
  GridDev g{};
  CK(cudaMemcpyAsync(ph.h.grid, &g, sizeof(GridDev), cudaMemcpyHostToDevice, c.stream));  // staged before it returns
}

// the population's sort structures for n_bin bins, or an error and no grid
// (the old ones go first: the pool then hands out the same blocks; new ones
// first made an upload and an emptying of one of 256 populations 15 us longer)
void alloc_sort(Ctx& c, PopHost& ph, int n_bin) {
  no_grid(c, ph);
  if (n_bin == 0) return;
  PopDev h = ph.h;
  std::vector<void*> o;
  try {
    fill_sort(c, h, o, n_bin);
  } catch (...) {
    free_list(c, o);
    ph.valid_sort = ph.caches_valid = false;
    throw;
  }
  take_sort(ph.h, h);
  ph.sort_allocs = o;
  ph.n_bin = n_bin;
}

// bin_grid_make (log) on the host, with glibc's log/exp like the reference
void make_grid(Ctx& c, PopHost& ph, int n_bin, double rmin, double rmax) {
  alloc_sort(c, ph, n_bin);
  ph.edges.assign(n_bin + 1, 0.0);
  ph.centers.assign(std::max(n_bin, 1), 0.0);
  if (n_bin > 0) {
    auto linspace = [](double a, double b, int n, double* out) {
      for (int i = 2; i <= n - 1; i++) {
        double t = (double)(i - 1) / (double)(n - 1);
        out[i - 1] = (1.0 - t) * a + t * b;
      }
      if (n > 0) {
        out[0] = a;
        out[n - 1] = b;
      }
    };
    auto logspace = [&](double a, double b, int n, double* out) {
      if (n == 0) return;
      linspace(log(a), log(b), n, out);
      for (int i = 0; i < n; i++) out[i] = exp(out[i]);
      out[0] = a;
      out[n - 1] = b;
    };
    logspace(rmin, rmax, n_bin + 1, ph.edges.data());
    double c1 = exp(interp_linear_disc(log(rmin), log(rmax), 2 * n_bin + 1, 2));
    double c2 = exp(interp_linear_disc(log(rmin), log(rmax), 2 * n_bin + 1, 2 * n_bin));
    logspace(c1, c2, n_bin, ph.centers.data());
  }
  GridDev g{};
  g.n_bin = n_bin;
  if (n_bin > 0) {
    g.log_lo = log(ph.edges[0]);
    g.log_hi = log(ph.edges[n_bin]);
    for (int i = 0; i <= n_bin; i++) g.edges[i] = ph.edges[i];
    for (int i = 0; i < n_bin; i++) g.centers[i] = ph.centers[i];
  }
  CK(cudaMemcpyAsync(ph.h.grid, &g, sizeof(GridDev), cudaMemcpyHostToDevice, c.stream));  // staged before it returns
}

void set_params(Ctx& c, PopHost& ph) {
  PopDev& h = ph.h;
  h.n_spec = c.n_spec;
  h.n_group = c.n_group;
  h.n_class = c.n_class;
  h.i_water = c.i_water;
  h.w = ph.own_w ? ph.w : c.w;
  h.flat = weights_flat(h.w);
  bool inc, dec;
  weight_monotonicity(h.w, &inc, &dec);
  h.mono_dec = dec;
  h.dmin = *std::min_element(c.density.begin(), c.density.end());
  h.dmax = *std::max_element(c.density.begin(), c.density.end());
  h.seed = ph.seed;
  h.pair_setup_valid = 0;  // the per-pair weight factors depend on the weights
  // radii follow the particle shape from the first sort on, before any step
  // sets the environment
  h.benv.frac = c.frac;
  c.dirty = true;
}

void init_pop(Ctx& c, PopHost& ph, int cap) {
  std::vector<void*>& o = ph.fixed_allocs;
  ph.h.ctr = c.d_ctrs + (&ph - c.pops.data());
  ph.h.grid = dalloc<GridDev>(c, o, 1);
  double* dens = dalloc<double>(c, o, c.n_spec);
  CK(cudaMemcpyAsync(dens, c.density.data(), sizeof(double) * c.n_spec, cudaMemcpyHostToDevice, c.stream));
  ph.h.density = dens;
  set_params(c, ph);
  alloc_slots(c, ph.h, ph.slot_allocs, cap);
  PopCtr z{};
  ph.rm_count = 0;  // the population's removal records start empty
  z.next_id = 1;
  z.bmin = 1 << 30;
  z.bmax = -1;
  write_ctr(c, (int)(&ph - c.pops.data()), z);
  ph.none = ph.h;
  fill_sort(c, ph.none, o, 0);
  no_grid(c, ph);
}

// grow (compact = false, slot numbers kept) or compact (slot order kept); on an
// error the population keeps its arrays
void relayout(Ctx& c, int k, int new_cap, bool compact) {
  PopHost& ph = c.pops[k];
  PopCtr r = read_ctr(c, k);
  PopDev h = ph.h;
  std::vector<void*> allocs, tmp;
  long long n_live = r.n_slots;
  try {
    alloc_slots(c, h, allocs, new_cap);
    long long* off = dalloc<long long>(c, tmp, (size_t)r.n_slots + 1);
    if (compact) n_live = scan(c, ph.h.alive, r.n_slots, off, true);
    if (r.n_slots > 0) {
      k_relayout<<<grid_for(r.n_slots, 256), 256, 0, c.stream>>>(ph.h, h, off, r.n_slots, compact ? 1 : 0);
      note_launch();
    }
  } catch (...) {
    free_list(c, tmp);
    free_list(c, allocs);
    throw;
  }
  ph.h = h;
  allocs.swap(ph.slot_allocs);
  free_list(c, tmp);
  free_list(c, allocs);
  if (compact) {
    r.n_slots = (int)n_live;
    ph.mirror_full = true;  // slots renumbered
  }
  write_ctr(c, k, r);
  push_pops(c);
  CK(cudaStreamSynchronize(c.stream));
}

// ---------------------------------------------------------------------------
// sort, with the grid decision of aero_sorted_remake_if_needed
// (aero_sorted.F90:214-373)

__global__ void k_radius_reset(PopCtr* ctrs, int n_pop, const uint8_t* on) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n_pop || !on[k]) return;
  ctrs[k].rmin_bits = 0x7ff0000000000000ULL;
  ctrs[k].rmax_bits = 0;
}

__global__ void k_radius_minmax_masked(const PopDev* pops, const uint8_t* on) {
  if (!on[blockIdx.y]) return;
  const PopDev& P = pops[blockIdx.y];
  int n = P.ctr->n_slots;
  // positive doubles order like their bit patterns: reduce the bits in the
  // block, then one atomic per block
  unsigned long long lo = ~0ULL, hi = 0ULL;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    if (!P.alive[i]) continue;
    unsigned long long b = (unsigned long long)__double_as_longlong(vol2rad(P.benv.frac, P.vtot[i]));
    lo = b < lo ? b : lo;
    hi = b > hi ? b : hi;
  }
  for (int o = 16; o > 0; o >>= 1) {
    unsigned long long l2 = __shfl_down_sync(0xffffffffu, lo, o);
    unsigned long long h2 = __shfl_down_sync(0xffffffffu, hi, o);
    lo = l2 < lo ? l2 : lo;
    hi = h2 > hi ? h2 : hi;
  }
  __shared__ unsigned long long slo[32], shi[32];
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) {
    slo[wid] = lo;
    shi[wid] = hi;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < (int)(blockDim.x >> 5); k++) {
      lo = slo[k] < lo ? slo[k] : lo;
      hi = shi[k] > hi ? shi[k] : hi;
    }
    if (hi > 0ULL) {
      atomicMin(&P.ctr->rmin_bits, lo);
      atomicMax(&P.ctr->rmax_bits, hi);
    }
  }
}


// chunk counts and histograms for the host's copy of the slot counts plus extra
// slots per population (the growth a device-driven loop may add before the
// host looks)
void prepare_chunks(Ctx& c, long long extra = 0) {
  for (int k = 0; k < c.n_pop; k++) {
    PopHost& ph = c.pops[k];
    ph.h.n_chunks = (int)((c.n_slots_host[k] + extra + kChunk - 1) / kChunk);
    int need = std::max(ph.h.n_chunks, 1) * ph.h.n_cells;
    if (need > ph.chunk_hist_cap) {
      int want = std::max(need * 2, 1024);  // headroom: slots grow inside a step
      ph.h.chunk_hist = dalloc<int>(c, ph.sort_allocs, want);
      ph.h.chunk_hist_len = want;
      ph.chunk_hist_cap = want;
      c.dirty = true;
    }
  }
}

// co-resident blocks of the sort for max_cells cells, and its shared memory
size_t size_sort(Ctx& c, int max_cells) {
  size_t smem = sizeof(int) * ((kSortWarps + 1) * (size_t)max_cells + (c.n_pop <= kSortMapPops ? c.n_pop + 1 : 0));
  if (smem != c.sort_smem) {
    int per_sm = 0;
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_sort_all, kSortThreads, smem));
    if (per_sm < 1) cap_throw("the sort does not fit one block per multiprocessor");
    c.sort_blocks = per_sm * c.n_sm;
    c.sort_smem = smem;
  }
  return smem;
}

// one cooperative launch of k_sort_all on a persistent grid of co-resident
// blocks, for chunk and cell counts up to max_chunks and max_cells
void launch_sort(Ctx& c, cudaStream_t st, int max_chunks, int max_cells, const StepBegin& begin = StepBegin{}) {
  size_t smem = size_sort(c, max_cells);
  long long items = (long long)c.n_pop * max_chunks;
  int blocks = (int)std::min<long long>(c.sort_blocks, std::max<long long>(items, 1));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(kSortThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const PopDev* pops = c.d_pops;
  CK(cudaLaunchKernelEx(&cfg, k_sort_all, pops, c.n_pop, max_chunks, max_cells, begin));
  note_launch();
}

int max_cells_of(const Ctx& c) {
  int m = 1;
  for (int k = 0; k < c.n_pop; k++) m = std::max(m, c.pops[k].h.n_cells);
  return m;
}

// the full sort of every population with its current grid
void run_sort(Ctx& c) {
  prepare_chunks(c);
  if (c.dirty) push_pops(c);
  int max_chunks = 1;
  long long units = 0;
  for (int k = 0; k < c.n_pop; k++) {
    max_chunks = std::max(max_chunks, c.pops[k].h.n_chunks);
    units += (long long)c.n_slots_host[k];
  }
  ProfScope ps(c, 1, units);
  launch_sort(c, c.stream, max_chunks, max_cells_of(c));
}

bool caches_current(const Ctx& c, const PopHost& ph) {
  return ph.caches_valid && ph.key_kt == ph.h.kernel_type && ph.key_temp == ph.h.temp &&
         ph.key_press == ph.h.pressure && ph.key_coeff == ph.h.coeff && ph.key_wver == ph.wver;
}

// recompute radius, bin and records of every live slot of the marked
// populations (after a grid, environment, kernel or weight change)
void refresh_caches(Ctx& c, const std::vector<uint8_t>& on) {
  bool any = false;
  for (int k = 0; k < c.n_pop; k++) any = any || on[k];
  if (!any) return;  // no read-back (a stream sync) in the common case
  int max_slots = 1;
  for (int k = 0; k < c.n_pop; k++)
    if (on[k]) max_slots = std::max(max_slots, c.n_slots_host[k]);  // sort_pops has just read them
  push_pops(c);
  c.pop_on.reserve(c.n_pop);
  CK(cudaMemcpyAsync(c.pop_on.p, on.data(), c.n_pop, cudaMemcpyHostToDevice, c.stream));
  dim3 g(grid_for(max_slots, 256), c.n_pop);
  k_refresh_all<<<g, 256, 0, c.stream>>>(c.d_pops, c.pop_on.p);
  note_launch();
  for (int k = 0; k < c.n_pop; k++)
    if (on[k]) {
      PopHost& ph = c.pops[k];
      ph.caches_valid = true;
      ph.key_kt = ph.h.kernel_type;
      ph.key_temp = ph.h.temp;
      ph.key_press = ph.h.pressure;
      ph.key_coeff = ph.h.coeff;
      ph.key_wver = ph.wver;
    }
}

// aero_state_sort: grid decision (remake_if_needed) then the sort itself
void sort_pops(Ctx& c, bool decide_grid) {
  bool hist_current = false;
  if (decide_grid) {
    std::vector<PopCtr>& r0 = read_ctrs(c);
    c.n_slots_host.resize(c.n_pop);
    for (int k = 0; k < c.n_pop; k++) c.n_slots_host[k] = r0[k].n_slots;
    // radius range of populations without a valid sort
    std::vector<uint8_t> on(c.n_pop, 0), fresh(c.n_pop, 0);
    bool any = false, any_valid = false;
    int max_slots = 1;
    for (int k = 0; k < c.n_pop; k++) {
      any_valid = any_valid || c.pops[k].valid_sort;
      if (!c.pops[k].valid_sort) {
        on[k] = 1;
        any = true;
        max_slots = std::max(max_slots, r0[k].n_slots);
      } else if (!caches_current(c, c.pops[k])) {
        fresh[k] = 1;  // current grid, stale caches
      }
    }
    if (any) {
      c.pop_on.reserve(c.n_pop);
      CK(cudaMemcpyAsync(c.pop_on.p, on.data(), c.n_pop, cudaMemcpyHostToDevice, c.stream));
      k_radius_reset<<<(c.n_pop + 127) / 128, 128, 0, c.stream>>>(c.d_ctrs, c.n_pop, c.pop_on.p);
      note_launch();
      dim3 g(grid_for(max_slots, 256), c.n_pop);
      k_radius_minmax_masked<<<g, 256, 0, c.stream>>>(c.d_pops, c.pop_on.p);
      note_launch();
    }
    refresh_caches(c, fresh);
    // sort with the current grid; the occupied bin range decides whether the
    // grid is kept.  (Where no population has a grid yet there is nothing to
    // sort by.)
    if (any_valid) {
      run_sort(c);
      hist_current = true;
    }
    std::vector<PopCtr>& q = read_ctrs(c);
    std::vector<uint8_t> regrid(c.n_pop, 0);
    for (int k = 0; k < c.n_pop; k++) {
      PopHost& ph = c.pops[k];
      double rmin = 0.0, rmax = 0.0;
      if (!ph.valid_sort) {
        if (q[k].n_live > 0) {
          memcpy(&rmin, &q[k].rmin_bits, 8);
          memcpy(&rmax, &q[k].rmax_bits, 8);
        }
      } else if (q[k].bmax < 0) {
        if (ph.n_bin > 0) {
          rmin = ph.edges[ph.n_bin];
          rmax = ph.edges[0];
        }
      } else {
        rmin = ph.edges[q[k].bmin];
        rmax = ph.edges[q[k].bmax + 1];
      }
      bool need = false;
      if (rmax == 0.0) {
        if (!ph.valid_sort && ph.n_bin != 0) make_grid(c, ph, 0, 0.0, 0.0);
      } else if (ph.n_bin < 1) {
        need = true;
      } else {
        double gmin = ph.edges[0], gmax = ph.edges[ph.n_bin];
        if (rmin / gmin < 3.0 || gmax / rmax < 3.0) need = true;
      }
      if (need) {
        double gmin = rmin / 10.0, gmax = rmax * 10.0;
        int n_bin = (int)ceil((log10(gmax) - log10(gmin)) * 10.0);
        if (n_bin > kMaxBin) cap_throw("more than 256 bins");
        make_grid(c, ph, n_bin, gmin, gmax);
      }
      // a new grid or a population without a valid sort: all bins change
      if (need || !ph.valid_sort) {
        regrid[k] = 1;
        ph.caches_valid = false;
        hist_current = false;
      }
      ph.valid_sort = true;
    }
    refresh_caches(c, regrid);
  }
  if (!hist_current) run_sort(c);
}

// ---------------------------------------------------------------------------
// one step over all populations

// call f(std::integral_constant<int, KT>, T{}) with the kernel type kt and the
// pair-test arithmetic of the mode (FP32 in MIXED, else FP64)
template <class F>
void with_kt(const Ctx& c, int kt, F&& f) {
  bool f32 = c.mode == PMC_MODE_MIXED;
  auto go = [&](auto ktc) {
    if (f32) f(ktc, float{});
    else f(ktc, double{});
  };
  switch (kt) {
    case kKernelAdditive: go(std::integral_constant<int, kKernelAdditive>{}); break;
    case kKernelConstant: go(std::integral_constant<int, kKernelConstant>{}); break;
    case kKernelBrown: go(std::integral_constant<int, kKernelBrown>{}); break;
    case kKernelSedi: go(std::integral_constant<int, kKernelSedi>{}); break;
    case kKernelBrownFree: go(std::integral_constant<int, kKernelBrownFree>{}); break;
    case kKernelBrownCont: go(std::integral_constant<int, kKernelBrownCont>{}); break;
    default: f(std::integral_constant<int, kKernelZero>{}, double{});
  }
}

// Brackets the launches of one tunable site with CUDA events while the
// autotuner searches that site; otherwise does nothing.
struct TuneScope {
  Ctx& c;
  cudaEvent_t e0 = nullptr;
  cudaStream_t st;
  static cudaEvent_t event(Ctx& c) {
    if (!c.tuner.spare.empty()) {
      cudaEvent_t e = c.tuner.spare.back();
      c.tuner.spare.pop_back();
      return e;
    }
    cudaEvent_t e = nullptr;
    CK(cudaEventCreate(&e));
    return e;
  }
  TuneScope(Ctx& c_, int site, cudaStream_t st_) : c(c_), st(st_) {
    if (!c.tuner.on || c.tuner.site != site) return;
    e0 = event(c);
    CK(cudaEventRecord(e0, st));
  }
  ~TuneScope() {
    if (!e0) return;
    cudaEvent_t e1 = event(c);
    cudaEventRecord(e1, st);
    c.tuner.pending.push_back({e0, e1});
  }
};

void launch_test_kt(Ctx& c, int kt, bool flat, int n_gpairs, long long W, cudaStream_t st) {
  TuneScope ts(c, kTuneTest, st);
  // sized from the round's sample count, at most 8 x 256 threads per SM
  const int tb = c.tune.threads[kTuneTest];
  int blocks = (int)std::min<long long>((long long)c.n_sm * 8 * 256 / tb, std::max<long long>(1, (W + tb - 1) / tb));
  with_kt(c, kt, [&](auto ktc, auto tt) {
    constexpr int KT = decltype(ktc)::value;
    using T = decltype(tt);
    if (flat)
      launch_chained(c, k_test<KT, T, true>, dim3(blocks), dim3(tb), 0, st, c.d_pops, c.gpair_pop.p, c.gpair_local.p, c.work_off.p, n_gpairs,
                                                 c.work_off.p + n_gpairs, c.flag.p, c.ev.p, c.ev_gp.p);
    else
      launch_chained(c, k_test<KT, T, false>, dim3(blocks), dim3(tb), 0, st, c.d_pops, c.gpair_pop.p, c.gpair_local.p, c.work_off.p, n_gpairs,
                                                  c.work_off.p + n_gpairs, c.flag.p, c.ev.p, c.ev_gp.p);
  });
}

ChainPool chain_pool(Ctx& c) {
  ChainPool pool;
  pool.y = c.ch_y.p;
  pool.q = c.ch_q.p;
  pool.pos = c.ch_pos.p;
  pool.ctr = c.round_dev.p + 3;
  pool.n_chunks = c.ch_chunks;
  return pool;
}

// blocks of tb threads for a warp per item of a later round, at most 2 x 256
// threads per SM, which is what its registers let it hold (the kernels fall
// back to a thread per item beyond that)
int grid_warps(const Ctx& c, long long W, int tb) {
  return (int)std::min<long long>((long long)c.n_sm * 2 * 256 / tb, std::max<long long>(1, (32 * W + tb - 1) / tb));
}

// a later round's items: the events of the round before, n_items =
// round_dev[2] on the device, W bounds it
void launch_items_kt(Ctx& c, int kt, bool flat, int n_gpairs, long long W, cudaStream_t st) {
  const int ti = c.tune.threads[kTuneItems], tc = c.tune.threads[kTuneChain];
  ChainPool pool = chain_pool(c);
  ItemArgs A;
  A.pops = c.d_pops;
  A.gpair_pop = c.gpair_pop.p;
  A.gpair_local = c.gpair_local.p;
  A.pop_pair_base = c.pop_pair_base.p;
  A.n_gpairs = n_gpairs;
  A.n_items = c.round_dev.p + 2;
  A.n_items_ev = c.round_dev.p + 6;
  A.ppw_slot = c.ppw_slot.p;
  A.ppw_gp = c.ppw_gp.p;
  A.op_pop = c.r_pop.p;
  A.op_pair = c.r_pair.p;
  A.op_slot = c.r_slot.p;
  A.op_k = c.r_k.p;
  A.op_key = c.r_key.p;
  A.n_ops = c.n_dev.p;
  A.op_cap = c.op_cap;
  A.win = c.win_set.p;
  A.dest = c.ev_dest.p;
  A.ev_key = c.ev_key.p;
  A.ev_c = c.ev_c.p;
  A.gp_c = c.gp_c.p;
  A.ev_pos = c.ev_pos.p;
  A.dec = c.dec_set.p;
  A.it_flag = c.it_flag.p;
  A.it_key = c.it_key.p;
  A.it_c = c.it_c.p;
  A.it_gp = c.it_gp.p;
  A.it_pos = c.it_pos.p;
  A.it_len = c.it_len.p;
  A.it_head = c.it_head.p;
  A.it_done = c.it_done.p;
  A.it_dec = c.it_dec.p;
  A.it_gused = c.it_gused.p;
  A.it_term = c.it_term.p;
  A.start_list = c.it_start.p;
  A.n_start = c.round_dev.p + 10;
  with_kt(c, kt, [&](auto ktc, auto tt) {
    constexpr int KT = decltype(ktc)::value;
    using T = decltype(tt);
    auto k = flat ? k_items<KT, T, true> : k_items<KT, T, false>;
    {
      TuneScope ts_items(c, kTuneItems, st);
      launch_chained(c, k, dim3(grid_warps(c, W, ti)), dim3(ti), 0, st, A);
    }
    auto kc = flat ? k_chain<KT, T, true> : k_chain<KT, T, false>;
    {
      TuneScope ts_chain(c, kTuneChain, st);
      launch_chained(c, kc, dim3(grid_warps(c, W, tc)), dim3(tc), 0, st, A, pool);
    }
  });
}

// Stable grouping by population of a batched context's per-round lists.
// Slot and ID ranks come from one scan over a list, and the per-population
// bases of alloc_bases assume that each population's entries lie together
// and in population order.  Round 0's samples and target operations are
// built that way; later rounds add entries from every population at the end
// (the walkers of target operations, and the target operations that walks
// add).  Entry i with population pop_of[i] >= 0 (negative: not kept) goes to
// dest[i]: all of population 0 first, then 1, ..., each in list order.
// Tiles of kGrpTile entries: per tile and population a count (hist, laid
// out population-major so that one scan gives every (population, tile) its
// start), then each entry's rank within its tile.
constexpr int kGrpTile = 256;

__global__ void __launch_bounds__(kGrpTile) k_grp_hist(const long long* n, const int* pop_of, int n_pop, int n_tiles,
                                                       int* hist, PopCtr* ctr0) {
  const long long N = *n;
  const long long i = blockIdx.x * (long long)kGrpTile + threadIdx.x;
  if (i >= N) return;
  const int p = pop_of[i];
  if (p < 0) return;
  if (p >= n_pop || blockIdx.x >= (unsigned)n_tiles) {
    bad_index(ctr0, kBadEventSlot, p);
    return;
  }
  atomicAdd(&hist[(size_t)p * n_tiles + blockIdx.x], 1);
}

__global__ void __launch_bounds__(kGrpTile) k_grp_rank(const long long* n, const int* pop_of, int n_tiles,
                                                       const long long* off, long long* dest) {
  chain_wait();
  __shared__ int wpop[kGrpTile / 32][32], wcnt[kGrpTile / 32][32];
  const long long N = *n;
  const long long i = blockIdx.x * (long long)kGrpTile + threadIdx.x;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int p = i < N ? pop_of[i] : -1;
  const unsigned same = __match_any_sync(0xffffffffu, p);
  const int rank = __popc(same & ((1u << lane) - 1u));
  // one entry per distinct population of the warp: its count there
  wpop[w][lane] = -1;
  wcnt[w][lane] = 0;
  __syncthreads();
  // the lowest lane of each group writes at its own lane index
  if (rank == 0) {
    wpop[w][lane] = p;
    wcnt[w][lane] = __popc(same);
  }
  __syncthreads();
  if (p < 0) {
    if (i < N) dest[i] = -1;  // not kept
    return;
  }
  int before = 0;
  for (int v = 0; v < w; v++)
    for (int l = 0; l < 32; l++)
      if (wpop[v][l] == p) before += wcnt[v][l];
  dest[i] = off[(size_t)p * n_tiles + blockIdx.x] + before + rank;
}

__global__ void k_scatter_ops(const long long* n_ops, const long long* dest, const int* pop, const int* pair,
                              const int* slot, const int* k, const unsigned long long* key, int* pop_o, int* pair_o,
                              int* slot_o, int* k_o, unsigned long long* key_o) {
  chain_wait();
  const long long Q = *n_ops;
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < Q; q += (long long)gridDim.x * blockDim.x) {
    const long long d = dest[q];
    if (d < 0) continue;  // a place without an operation: dropped
    pop_o[d] = pop[q];
    pair_o[d] = pair[q];
    slot_o[d] = slot[q];
    k_o[d] = k[q];
    key_o[d] = key[q];
  }
}

// the population of each kept item of a later round (-1 for an item that
// made no event)
__global__ void k_item_pops(const long long* n_items, const uint8_t* it_flag, const int* it_gp, const int* gpair_pop,
                            int n_gpairs, int* pop_of) {
  chain_wait();
  const long long n = *n_items;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const int gp = it_gp[i];
    pop_of[i] = (it_flag[i] && gp >= 0 && gp < n_gpairs) ? gpair_pop[gp] : -1;
  }
}

// dest for the entries of a list of at most bound entries (count *n on the
// device), grouped by population (k_grp_hist, k_grp_rank)
void group_by_pop(Ctx& c, const long long* n, long long bound, const int* pop_of, long long* dest, cudaStream_t st,
                  long long* kept = nullptr) {
  const int n_tiles = (int)std::max<long long>(1, (bound + kGrpTile - 1) / kGrpTile);
  const long long nh = (long long)n_tiles * c.n_pop;
  c.grp_hist.reserve((size_t)nh);
  c.grp_off.reserve((size_t)nh + 1);
  CK(cudaMemsetAsync(c.grp_hist.p, 0, sizeof(int) * (size_t)nh, st));
  k_grp_hist<<<n_tiles, kGrpTile, 0, st>>>(n, pop_of, c.n_pop, n_tiles, c.grp_hist.p, c.d_ctrs);
  note_launch();
  scan_multi<int>(c, {ScanArg<int>{c.grp_hist.p, nh, nullptr, c.grp_off.p, kept}}, st);
  launch_chained(c, k_grp_rank, dim3(n_tiles), dim3(kGrpTile), 0, st, n, pop_of, n_tiles, c.grp_off.p, dest);
}

// Buffers of a round's at most Q target operations that carry nothing from
// the round before
void reserve_ops(Ctx& c, long long Q) {
  const size_t q = (size_t)Q;
  c.op_pop.reserve(q); c.op_pair.reserve(q); c.op_slot.reserve(q); c.op_k.reserve(q); c.op_key.reserve(q);
  c.pp_res.reserve(q);
  c.pp_vol.reserve(q * c.n_spec);
  c.pp_rm_off.reserve(q + 2);
  c.pp_rm_tot.reserve(1);
  c.win_pp.reserve(q + 1); c.lost_pp.reserve(q + 1);
  c.lost_off.reserve(q + 2); c.rank_slot_pp.reserve(q + 2);
  c.grp_dest.reserve(q + 1);
  const size_t nw = q * kMaxCopies;
  c.wk_slot.reserve(nw); c.wk_gp.reserve(nw); c.wk_flag.reserve(nw);
  const size_t nh = std::max<size_t>(1, (q + kGrpTile - 1) / kGrpTile) * c.n_pop;
  c.grp_hist.reserve(nh);
  c.grp_off.reserve(nh + 1);
}

// staging list of a later round's target operations (redone and added ones)
void reserve_redo(Ctx& c, long long Q) {
  const size_t q = (size_t)Q;
  c.r_pop.reserve(q); c.r_pair.reserve(q); c.r_slot.reserve(q); c.r_k.reserve(q); c.r_key.reserve(q);
}

// A later round's target operations (at most Q staged in r_*, n_dev[2] of
// them): the redone ones, then one place per item (population -1 where the
// item made none).  Grouped by population into op_*, which also drops the
// empty places; n_dev[1] counts the operations kept.
void launch_pp_group(Ctx& c, long long Q, cudaStream_t st) {
  if (c.n_pop == 1) {  // one population: only the empty places go
    launch_chained(c, k_compact_ops, dim3((unsigned)compact_tiles(Q)), dim3(kCompactThreads), 0, st, c.n_dev.p + 2,
                   c.n_dev.p + 1, tile_ctl(c, compact_tiles(Q), st), c.r_pop.p, c.r_pair.p, c.r_slot.p, c.r_k.p,
                   c.r_key.p, c.op_pop.p, c.op_pair.p, c.op_slot.p, c.op_k.p, c.op_key.p);
    return;
  }
  group_by_pop(c, c.n_dev.p + 2, Q, c.r_pop.p, c.grp_dest.p, st, c.n_dev.p + 1);
  launch_chained(c, k_scatter_ops, dim3(grid_for(Q, 256)), dim3(256), 0, st, c.n_dev.p + 2, c.grp_dest.p, c.r_pop.p,
                 c.r_pair.p, c.r_slot.p, c.r_k.p, c.r_key.p, c.op_pop.p, c.op_pair.p, c.op_slot.p, c.op_k.p,
                 c.op_key.p);
}

// the bound on each target operation's removals, scanned into its place in
// the removal pool (their total in pp_rm_tot); n_ops: their count
void launch_pp_count(Ctx& c, long long Q, const long long* n_ops, cudaStream_t st) {
  const long long tiles = std::max<long long>(1, (Q + 255) / 256);
  launch_chained(c, k_pp_count, dim3((unsigned)tiles), dim3(256), 0, st, c.d_pops, c.op_pop.p, c.op_pair.p,
                 c.op_slot.p, c.op_k.p, n_ops, Q, c.pp_rm_off.p, c.pp_rm_tot.p, tile_ctl(c, tiles, st));
}

// Every operation's removals fit the pool: one that did not would lose
// and draw anew a round later, so the pool's size (in a batch, the other
// populations' removals) would decide the particles.  One read-back; in a
// step graph the device checks it (k_step_check, k_pp_fits).
void fit_rm_pool(Ctx& c) {
  long long rm_tot = 0;
  unsigned long long scan_err = 0;
  CK(cudaMemcpyAsync(&rm_tot, c.pp_rm_tot.p, sizeof(rm_tot), cudaMemcpyDeviceToHost, c.stream));
  CK(cudaMemcpyAsync(&scan_err, c.scan_err.p, sizeof(scan_err), cudaMemcpyDeviceToHost, c.stream));
  CK(cudaStreamSynchronize(c.stream));
  if (scan_err) {
    CK(cudaMemsetAsync(c.scan_err.p, 0, sizeof(scan_err), c.stream));
    throw Fail(PMC_ERR_TIMEOUT);
  }
  if (rm_tot < 0 || rm_tot >= (1LL << 31)) cap_throw("more than 2^31 removals in one round");
  if (rm_tot + 1 > (long long)c.pp_rm_pool.n) c.pp_rm_pool.reserve((size_t)(rm_tot + rm_tot / 2 + 1024));
  c.last_rm = std::max(c.last_rm, rm_tot);
}

// the round's target operations (n_dev[1], at most Q)
void launch_pp_ops(Ctx& c, int kt, long long Q, cudaStream_t st) {
  with_kt(c, kt, [&](auto ktc, auto) {
    constexpr int KT = decltype(ktc)::value;
    launch_chained(c, k_pp_ops<KT>, dim3(grid_for(32 * Q, 32 * kPPWarps)), dim3(32 * kPPWarps), 0, st, c.d_pops, c.op_pop.p, c.op_pair.p, c.op_slot.p, c.op_k.p, c.op_key.p, c.n_dev.p + 1, c.pp_res.p, c.pp_vol.p,
        c.pp_rm_off.p, c.pp_rm_pool.p, (long long)c.pp_rm_pool.n);
  });
}

// One mc_coag call in replay mode: the grid decision of
// aero_sorted_remake_if_needed on the host (glibc log/exp, as the reference),
// then one device thread runs the reference's loop on the persisted inverse
// maps.  One population only.
int replay_step_host(Ctx& c, long long* s_out, long long* k_out) {
  if (c.n_pop != 1) return PMC_ERR_INVALID_ARG;
  PopHost& ph = c.pops[0];
  ReplayBuffers& rb = c.replay;
  PopCtr r = read_ctr(c, 0);
  if (r.n_live != r.n_slots) {
    relayout(c, 0, ph.h.cap, true);  // dense slots, order kept
    r = read_ctr(c, 0);
    rb.valid = false;
  }
  if (ph.h.cap < 2 * r.n_slots + 1024) {
    relayout(c, 0, 2 * r.n_slots + 1024, false);
    rb.valid = false;
  }
  // radius range: from the inverse maps while they are valid, else from the
  // particles (aero_sorted.F90:263-306)
  double rmin = 0.0, rmax = 0.0;
  if (!rb.valid || ph.n_bin < 1) {
    r.rmin_bits = 0x7ff0000000000000ULL;
    r.rmax_bits = 0;
    write_ctr(c, 0, r);
    push_pops(c);
    DevBuf<uint8_t> on;
    on.reserve(1);
    uint8_t one = 1;
    CK(cudaMemcpyAsync(on.p, &one, 1, cudaMemcpyHostToDevice, c.stream));
    dim3 g(grid_for(std::max(r.n_slots, 1), 256), 1);
    k_radius_minmax_masked<<<g, 256, 0, c.stream>>>(c.d_pops, on.p);
    note_launch();
    PopCtr q = read_ctr(c, 0);
    on.release();
    if (q.n_live > 0) {
      memcpy(&rmin, &q.rmin_bits, 8);
      memcpy(&rmax, &q.rmax_bits, 8);
    }
  } else {
    std::vector<int> cnt(ph.n_bin * c.n_class);
    DevBuf<int> d;
    d.reserve(cnt.size());
    replay_cell_counts(rb.dev, d.p, c.stream);
    note_launch();
    CK(cudaMemcpyAsync(cnt.data(), d.p, sizeof(int) * cnt.size(), cudaMemcpyDeviceToHost, c.stream));
    CK(cudaStreamSynchronize(c.stream));
    d.release();
    int bmin = 0, bmax = 0;
    for (int b = 1; b <= ph.n_bin; b++) {
      int s = 0;
      for (int cl = 0; cl < c.n_class; cl++) s += cnt[(b - 1) + ph.n_bin * cl];
      if (s > 0) {
        if (bmin == 0) bmin = b;
        bmax = b;
      }
    }
    if (bmin == 0) {
      rmin = ph.edges[ph.n_bin];
      rmax = ph.edges[0];
    } else {
      rmin = ph.edges[bmin - 1];
      rmax = ph.edges[bmax];
    }
  }
  bool rebuild = !rb.valid;
  if (rmax == 0.0) {
    if (!rb.valid) make_grid(c, ph, 0, 0.0, 0.0);
  } else {
    bool need = ph.n_bin < 1;
    if (!need) {
      double gmin = ph.edges[0], gmax = ph.edges[ph.n_bin];
      need = rmin / gmin < 3.0 || gmax / rmax < 3.0;
    }
    if (need) {
      double gmin = rmin / 10.0, gmax = rmax * 10.0;
      int n_bin = (int)ceil((log10(gmax) - log10(gmin)) * 10.0);
      if (n_bin > kMaxBin) return PMC_ERR_CAPACITY;
      make_grid(c, ph, n_bin, gmin, gmax);
      rebuild = true;
    }
  }
  ph.valid_sort = true;
  int nb = std::max(ph.n_bin, 1);
  if (!replay_reserve(rb, ph.h.cap, nb * c.n_class, c.n_group * c.n_class, nb, c.n_class, c.n_group, c.stream))
    return PMC_ERR_CAPACITY;
  if (rb.n_cells != nb * c.n_class || !rb.valid) rebuild = true;
  push_pops(c);
  if (!ph.h.kmax_valid && ph.n_bin > 0) {
    launch_kmax(c);
    ph.h.kmax_valid = 1;
    push_pops(c);
  }
  long long hv[4] = {c.replay_used, 0, 0, r.next_id};
  CK(cudaMemcpyAsync(rb.dev.used, hv, sizeof(long long) * 4, cudaMemcpyHostToDevice, c.stream));
  int hi[2] = {0, r.n_slots};
  CK(cudaMemcpyAsync(rb.dev.status, hi, sizeof(int) * 2, cudaMemcpyHostToDevice, c.stream));
  ReplayDev rd = rb.dev;
  rd.u = c.replay_u.p;
  rd.n_u = c.replay_n;
  rd.rebuild = rebuild ? 1 : 0;
  size_t stack = 0;
  cudaDeviceGetLimit(&stack, cudaLimitStackSize);
  if (stack < 16384) CK(cudaDeviceSetLimit(cudaLimitStackSize, 16384));
  replay_launch(c.d_pops, 0, rd, c.stream);
  note_launch();
  CK(cudaGetLastError());
  CK(cudaMemcpyAsync(hv, rb.dev.used, sizeof(long long) * 4, cudaMemcpyDeviceToHost, c.stream));
  CK(cudaMemcpyAsync(hi, rb.dev.status, sizeof(int) * 2, cudaMemcpyDeviceToHost, c.stream));
  CK(cudaStreamSynchronize(c.stream));
  c.replay_used = hv[0];
  *s_out = hv[1];
  *k_out = hv[2];
  r = read_ctr(c, 0);
  r.n_slots = r.n_live = hi[1];
  r.next_id = hv[3];
  r.tot_samp = hv[1];
  r.tot_coag = hv[2];
  write_ctr(c, 0, r);
  rb.valid = hi[0] == 0;
  ph.caches_valid = false;  // the replay rewrote slots without the caches
  static const int map[] = {PMC_OK, PMC_ERR_INVALID_ARG, PMC_ERR_OUT_OF_GRID, PMC_ERR_CAPACITY,
                            PMC_ERR_CUDA, PMC_ERR_TIMEOUT, PMC_ERR_RNG_EXHAUSTED, PMC_ERR_ASSERT};
  return (hi[0] >= 0 && hi[0] <= 7) ? map[hi[0]] : PMC_ERR_ASSERT;
}

__global__ void k_step_reset(PopCtr* ctrs, int n_pop) {
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n_pop) return;
  ctrs[k].tot_samp = ctrs[k].tot_coag = ctrs[k].kmax_warn = ctrs[k].redraws = ctrs[k].walk_tests = 0;
  ctrs[k].status = 0;
  ctrs[k].bad_site = 0;
  ctrs[k].bad_index = 0;
  ctrs[k].cap_site = 0;
}

// every slot, those above n_slots included: a slot that an earlier, larger
// population used keeps its claim word, and a word of an old generation is
// below every word of a restarted one
__global__ void k_fill_claims(const PopDev* pops) {
  const PopDev& P = pops[blockIdx.y];
  if (P.ctr->n_slots > P.cap && blockIdx.x == 0 && threadIdx.x == 0) bad_index(P.ctr, kBadSlotCount, P.ctr->n_slots);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < P.cap; i += gridDim.x * blockDim.x) {
    P.claim[i] = ~0ULL;
    P.rclaim[i] = ~0ULL;
    P.touched[i] = ~0u;
  }
}

// per-population work of a round: samples and target operations
__global__ void k_pop_work(const long long* pop_pair_base, int n_pop, const long long* work_off,
                           const long long* pp_off, long long* out) {
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n_pop) return;
  long long a = pop_pair_base[k], b = pop_pair_base[k + 1];
  out[2 * k] = work_off[b] - work_off[a];
  out[2 * k + 1] = pp_off[b] - pp_off[a];
}

// ---------------------------------------------------------------------------
// Later rounds.  After round 0 every kernel of a round reads its counts from
// the device, and round 0's events bound every later round's items and
// events (each event yields at most one item of the next round, each item at
// most one event or chain).  So the later rounds run as the body of a
// conditional WHILE node of one CUDA graph: k_round_begin advances the round
// and the claim generation and makes the last round's events this round's
// items; the sort brings the cell lists to the round's start, so walks meet
// the particles earlier rounds made; k_round_end adds up the step's
// statistics and sets the loop condition: events in this round, fewer than
// max_rounds rounds, and room in every population for the next round's new
// slots, in the slot arrays and in the sort's chunks.  Without room the
// graph stops and the host loop, which can grow both, carries on.  A step
// graph's rounds take target operations too, their tail an IF node
// (k_pp_fits); in a step that the host begins, rounds with target operations
// run from the host loop.

__device__ void round_begin(uint32_t* d_round, long long* round_dev, int* per_pop, int n_per_pop, long long* n_dev) {
  if (threadIdx.x == 0) {
    d_round[0] += 1u;
    d_round[1] += 1u;
    // this round's items: the events of the round before, then the walkers
    // its target operations made
    round_dev[6] = round_dev[1];
    round_dev[7] = round_dev[5];
    round_dev[2] = round_dev[1] + round_dev[5];
    // the target operations redone in this round, and the places of its
    // staging list: those, then one per item
    n_dev[0] = round_dev[8];
    n_dev[2] = round_dev[8] + round_dev[2];
    round_dev[0] = 0;
    round_dev[1] = 0;
    round_dev[3] = 0;
    round_dev[4] = 0;
    round_dev[5] = 0;
    round_dev[8] = 0;
    round_dev[10] = 0;
  }
  for (int k = threadIdx.x; k < n_per_pop; k += blockDim.x) per_pop[k] = 0;
}
__global__ void k_round_begin(uint32_t* d_round, long long* round_dev, int* per_pop, int n_per_pop, long long* n_dev) {
  round_begin(d_round, round_dev, per_pop, n_per_pop, n_dev);
}

// stats: [0] events that lost a claim, [1] events, [2] rounds, [3] 1 if the
// graph stopped for lack of room (slots, sort chunks, or more items or target
// operations than its later launches are bounded by) with work left (2: in the
// middle of a round, k_pp_fits), [6] scans that gave up, [7] the largest number
// of items of a later round, [8] of its target operations, at most, [9] target
// operations, [10] those that lost a claim, [11] the largest removal bound.
// If the loop goes on, the next round begins here (per_pop null: it begins by
// itself).
__global__ void k_round_end(long long* round_dev, long long* stats, uint32_t* d_round, int max_rounds,
                            const PopDev* pops, PopCtr* ctrs, int n_pop, long long sort_slots, long long max_items,
                            long long max_ops, long long* n_dev, const unsigned long long* scan_err, int* per_pop,
                            cudaGraphConditionalHandle cond) {
  const long long E = round_dev[1], lost = round_dev[8], items = E + round_dev[5];
  // a step with target operations: at most one more per item
  const long long ops = max_ops > 0 ? lost + items : 0;
  bool fits = items <= max_items && ops <= max_ops;
  for (int k = threadIdx.x; k < n_pop; k += blockDim.x) {
    const long long need = (long long)ctrs[k].n_slots + items + (kMaxCopies - 1) * ops;
    if (need > (long long)pops[k].cap || need > sort_slots) fits = false;
  }
  const bool room = __syncthreads_and(fits);
  const bool left = items > 0 || lost > 0;
  const bool more = left && room && (int)d_round[0] + 1 < max_rounds;
  if (left && room && !more)
    for (int k = threadIdx.x; k < n_pop; k += blockDim.x)
      if (ctrs[k].status == 0) ctrs[k].status = kErrTimeout;
  if (threadIdx.x == 0) {
    stats[0] += round_dev[0];
    stats[1] += E;
    stats[2] += 1;
    stats[6] = (long long)*scan_err;
    if (items > stats[7]) stats[7] = items;
    if (ops > stats[8]) stats[8] = ops;
    if (max_ops > 0) {
      stats[9] += n_dev[1];
      stats[10] += lost;
    }
    if (left && !room) stats[3] = 1;
    cudaGraphSetConditional(cond, more ? 1u : 0u);
  }
  if (!more || !per_pop) return;
  __syncthreads();  // the round's counts are read
  round_begin(d_round, round_dev, per_pop, 4 * n_pop, n_dev);
}

// The removals of a later round's target operations fit their pool: the
// round's tail runs.  Otherwise the graph stops here and the host, which can
// grow the pool, runs the tail.
__global__ void k_pp_fits(const long long* rm_tot, long long pool, long long* stats, cudaGraphConditionalHandle tail,
                          cudaGraphConditionalHandle loop) {
  const bool fits = *rm_tot + 1 <= pool;
  if (*rm_tot > stats[11]) stats[11] = *rm_tot;
  if (!fits) {
    stats[3] = 2;
    cudaGraphSetConditional(loop, 0u);
  }
  cudaGraphSetConditional(tail, fits ? 1u : 0u);
}

// ---------------------------------------------------------------------------
// A whole step as one graph: round 0 in stream order, then the later rounds'
// WHILE node.  What round 0 needed the host for is checked on the device
// (k_step_check): the grid is kept (aero_sorted_remake_if_needed's rule on the
// occupied bins), the samples and target operations (none in a graph without
// them) and their removals fit the buffers, every population has room for a
// particle per sample and the copies, and no scan gave up (its offsets would
// be wrong).  If not, the totals are set to zero, so the rest of the graph does
// nothing and the host runs the step the long way, which reports such a scan
// before a particle has changed.  A population's walks stop at per-particle
// pairs if it has target operations in this step; that is set here too, so a
// population whose operations come and go does not send the step the long way.
enum : long long { kNoGoGrid = 1, kNoGoOps = 2, kNoGoSamples = 4, kNoGoSlots = 8, kNoGoPool = 16, kNoGoScan = 32 };

__global__ void k_step_check(PopDev* pops, int n_pop, const long long* pop_pair_base, long long* work_off,
                             long long* pp_off, int n_gp, long long w_cap, long long q_cap, const long long* rm_tot,
                             long long pool, long long sort_slots, long long* n_dev, long long* stat,
                             const unsigned long long* scan_err) {
  chain_wait();
  const long long W = work_off[n_gp], Q = pp_off[n_gp];
  long long why = *scan_err ? kNoGoScan : 0;
  if (Q > q_cap) why |= kNoGoOps;
  if (W > w_cap) why |= kNoGoSamples;
  if (Q > 0 && q_cap > 0 && *rm_tot + 1 > pool) why |= kNoGoPool;
  for (int k = threadIdx.x; k < n_pop; k += blockDim.x) {
    PopDev& P = pops[k];
    const GridDev& G = *P.grid;
    PopCtr& r = *P.ctr;
    if (G.n_bin >= 1) {
      const double gmin = G.edges[0], gmax = G.edges[G.n_bin];
      const double rmin = r.bmax < 0 ? gmax : G.edges[r.bmin], rmax = r.bmax < 0 ? gmin : G.edges[r.bmax + 1];
      if (rmin / gmin < 3.0 || gmax / rmax < 3.0) why |= kNoGoGrid;
    } else if (r.bmax >= 0 || r.n_live > 0) {
      why |= kNoGoGrid;
    }
    const long long a = pop_pair_base[k], b = pop_pair_base[k + 1];
    const long long Wk = work_off[b] - work_off[a], Qk = pp_off[b] - pp_off[a];
    P.walk_stops = r.walk_stops = Qk > 0 ? 1 : 0;
    const long long need = (long long)r.n_slots + Wk + (kMaxCopies - 1) * Qk;
    if (need > (long long)P.cap || (long long)r.n_slots > sort_slots) why |= kNoGoSlots;
  }
  const int all = __syncthreads_or((int)why);
  if (threadIdx.x != 0) return;
  stat[4] = all;
  stat[5] = W;
  stat[12] = Q;
  if (q_cap > 0) stat[11] = *rm_tot;
  n_dev[1] = all ? 0 : Q;
  if (all) work_off[n_gp] = pp_off[n_gp] = 0;
}

// The step graph's last launch: its report and the counter blocks (n16 words of
// 16 bytes from stat on) into page-locked host memory, then the step's sequence
// number, which the host waits for.  A copy and a stream synchronisation in its
// place took 12 us of a step longer (0.131 to 0.119 ms at 1e4 particles).
__global__ void __launch_bounds__(1024) k_step_report(const uint4* stat, int n16, uint4* out, volatile unsigned* flag,
                                                      unsigned* seq) {
  for (int k = threadIdx.x; k < n16; k += blockDim.x) out[k] = stat[k];
  __threadfence_system();
  __syncthreads();
  if (threadIdx.x == 0) *flag = ++*seq;
}

// Resolve and apply the events of a round (E at round_dev[1], at most W) and,
// with Q > 0, its target operations (n_dev[1] of them, at most Q).  chains: the
// round may have chains (every round but the first).
void resolve_apply(Ctx& c, cudaStream_t st, long long W, long long Q, bool chains) {
  long long* Ed = c.round_dev.p + 1;
  ChainPool pool = chain_pool(c);
  // Q bounds the round's target operations; their count is n_dev[1] (the
  // redone ones, then those that walks appended)
  if (Q > 0) {
    const long long tiles = std::max<long long>(1, (Q + 255) / 256);
    launch_chained(c, k_pp_resolve, dim3((unsigned)tiles), dim3(256), 0, st, c.d_pops, c.n_pop, c.op_pop.p, c.op_key.p,
                   c.n_dev.p + 1, c.pp_res.p, c.pp_rm_pool.p, c.win_pp.p, c.rank_slot_pp.p, c.per_pop_i.p, c.lost_pp.p,
                   c.lost_off.p, c.round_dev.p + 8, tile_ctl(c, tiles, st));
  }
  {
    TuneScope ts(c, kTuneResolve, st);
    ResolveArgs A;
    A.pops = c.d_pops;
    A.gpair_pop = c.gpair_pop.p;
    A.n_events = W > 0 ? Ed : nullptr;
    A.ev_key = c.ev_key.p;
    A.ev = c.ev_c.p;
    A.ev_gp = c.gp_c.p;
    A.win = c.win_set.p;
    A.dec = c.dec_set.p;
    A.n_losers = c.round_dev.p;
    A.ev_len = c.ev_len.p;
    A.ev_head = c.ev_head.p;
    A.ev_app = c.ev_app.p;
    A.pool = pool;
    A.chain_list = c.chain_list.p;
    A.n_chain = c.round_dev.p + 4;
    A.rank_slot = c.rank_slot_set.p;
    A.rank_id = c.rank_id_set.p;
    const int tr = c.tune.threads[kTuneResolve];
    const long long tiles = std::max<long long>(1, (W + tr - 1) / tr);
    A.ctl = tile_ctl(c, tiles, st);
    A.n_pop = c.n_pop;
    A.per_pop = c.per_pop_i.p;
    A.set_slot_base = c.slot_base_set.p;
    A.pp_slot_base = c.slot_base_pp.p;
    A.set_id_base = c.id_base_set.p;
    A.pp_id_base = c.id_base_pp.p;
    launch_chained(c, k_resolve, dim3((unsigned)tiles), dim3(tr), 0, st, A);
  }
  if (W > 0) {
    const int ta = c.tune.threads[kTuneApply];
    // chains, one warp each, beside the other events (their claims keep them
    // on different slots): a branch of its own in a captured step
    cudaStream_t sc = st;
    if (chains && c.fork) {
      CK(cudaEventRecord(c.ev_fork, st));
      CK(cudaStreamWaitEvent(c.side_stream, c.ev_fork, 0));
      sc = c.side_stream;
    }
    if (chains) {
      k_apply_chain<<<grid_for(W, 32), 32, 0, sc>>>(c.d_pops, c.gpair_pop.p, c.pop_pair_base.p, c.chain_list.p,
                                                    c.round_dev.p + 4, c.ev_key.p, c.ev_len.p, c.ev_app.p,
                                                    c.ev_head.p, c.ev_done.p, pool, c.gp_c.p, c.ev_pos.p,
                                                    c.ev_dest.p, c.ev_key.p, c.ev_c.p, c.dec_set.p, c.ev_term.p);
      note_launch();
    }
    {
      TuneScope ts(c, kTuneApply, st);
      launch_chained(c, k_apply, dim3(grid_for(W, ta)), dim3(ta), 0, st, c.d_pops, c.gpair_pop.p, Ed, c.win_set.p, c.rank_slot_set.p,
                                              c.rank_id_set.p, c.slot_base_set.p, c.id_base_set.p, c.ev_done.p,
                                              c.ev_dest.p, c.ev_key.p, c.ev_c.p, c.gp_c.p, c.ev_pos.p, c.dec_set.p,
                                              c.ev_term.p, c.pop_pair_base.p);
    }
    if (chains && c.fork) {
      CK(cudaEventRecord(c.ev_join, c.side_stream));
      CK(cudaStreamWaitEvent(st, c.ev_join, 0));
    }
  }
  if (Q > 0) {
    launch_chained(c, k_pp_apply, dim3(grid_for(Q, 128)), dim3(128), 0, st, c.d_pops, c.op_pop.p, c.n_dev.p + 1,
                   c.pp_res.p, c.pp_vol.p, c.pp_rm_pool.p, c.win_pp.p, c.rank_slot_pp.p, c.slot_base_pp.p,
                   c.id_base_pp.p, c.pop_pair_base.p, c.op_k.p, c.wk_slot.p, c.wk_gp.p, c.wk_flag.p);
    const long long tiles = compact_tiles(Q * kMaxCopies);
    launch_chained(c, k_compact_walkers, dim3((unsigned)tiles), dim3(kCompactThreads), 0, st, c.wk_flag.p,
                   c.n_dev.p + 1, c.round_dev.p + 5, tile_ctl(c, tiles, st), c.wk_slot.p, c.wk_gp.p, c.ppw_slot.p,
                   c.ppw_gp.p);
  }
}


CompactArgs compact_args(Ctx& c, const uint8_t* flag, const long long* n, long long bound, cudaStream_t st) {
  CompactArgs A;
  A.flag = flag;
  A.n = n;
  A.n_events = c.round_dev.p + 1;
  A.ctl = tile_ctl(c, compact_tiles(bound), st);
  A.ev_key = c.ev_key.p;
  A.ev_c = c.ev_c.p;
  A.gp_c = c.gp_c.p;
  A.ev_pos = c.ev_pos.p;
  A.ev_len = c.ev_len.p;
  A.ev_term = c.ev_term.p;
  A.dec = c.dec_set.p;
  return A;
}

// round 0's events from the tests' flags (their count *n on the device, at most W)
void launch_compact_samples(Ctx& c, const long long* n, long long W, cudaStream_t st) {
  launch_chained(c, k_compact_samples, dim3((unsigned)compact_tiles(W)), dim3(kCompactThreads), 0, st, 
      compact_args(c, c.flag.p, n, W, st), c.d_pops, c.gpair_pop.p, c.gpair_local.p, c.ev.p, c.ev_gp.p,
      c.work_off.p);
}

// a buffer's growth that keeps what it holds
template <class T>
void grow_keeping(Ctx& c, DevBuf<T>& b, size_t m) {
  if (m <= b.n) return;
  DevBuf<T> nb;
  nb.reserve(std::max(m, b.n + b.n / 2));
  if (b.n) CK(cudaMemcpyAsync(nb.p, b.p, b.n * sizeof(T), cudaMemcpyDeviceToDevice, c.stream));
  CK(cudaStreamSynchronize(c.stream));
  std::swap(nb, b);
  nb.release();
}

// round 0's target operations, at most cap
void launch_build_ops(Ctx& c, int n_gpairs, long long cap, cudaStream_t st) {
  k_build_ops<<<n_gpairs, 128, 0, st>>>(c.d_pops, c.gpair_pop.p, c.gpair_local.p, c.pp_off.p, n_gpairs, cap,
                                        c.op_pop.p, c.op_pair.p, c.op_slot.p, c.op_k.p, c.op_key.p);
  note_launch();
}

struct RoundBounds {
  int kt;
  bool flat;
  int n_gpairs;
  long long W;     // items and events of a round, at most
  int max_chunks;  // sort chunks per population, at most
  int max_cells;
};

// The kernels of one later round on stream st, after k_round_begin, in two
// parts.  The head: the sort, the items and their chains and, with Q > 0 (a
// step with target operations), the round's at most Q target operations: the
// redone ones (k_build_redo staged them, before k_round_begin) and those that
// walks add (at most one per item), with the bound of their removals.  The
// tail, once the removals fit their pool: the operations, which claim
// alongside, the items' events in item order, then resolve and apply.
void enqueue_round_head(Ctx& c, cudaStream_t st, const RoundBounds& b, long long Q) {
  launch_sort(c, st, b.max_chunks, b.max_cells);
  {
    dim3 g(b.max_cells, c.n_pop);
    launch_chained(c, k_walk_rates, dim3(g), dim3(128), 0, st, c.d_pops);
  }
  launch_items_kt(c, b.kt, b.flat, b.n_gpairs, b.W, st);
  if (Q > 0) {
    launch_pp_group(c, Q, st);
    launch_pp_count(c, Q, c.n_dev.p + 1, st);
  }
}

void enqueue_round_tail(Ctx& c, cudaStream_t st, const RoundBounds& b, long long Q) {
  const long long W = b.W;
  if (Q > 0) launch_pp_ops(c, b.kt, Q, st);
  const long long* Id = c.round_dev.p + 2;
  // a batched step with target operations: the walkers they made join the
  // items after the events, from every population, so the events are
  // grouped by population for the allocation (group_by_pop)
  const long long* grouped = nullptr;
  if (Q > 0 && c.n_pop > 1) {
    c.item_pop.reserve((size_t)W + 1);
    c.grp_dest.reserve((size_t)W + 1);
    launch_chained(c, k_item_pops, dim3(grid_for(W, 256)), dim3(256), 0, st, Id, c.it_flag.p, c.it_gp.p, c.gpair_pop.p, b.n_gpairs,
                                                  c.item_pop.p);
    group_by_pop(c, Id, W, c.item_pop.p, c.grp_dest.p, st);
    grouped = c.grp_dest.p;
  }
  launch_chained(c, k_compact_items, dim3((unsigned)compact_tiles(W)), dim3(kCompactThreads), 0, st, 
      compact_args(c, c.it_flag.p, Id, W, st), c.it_key.p, c.it_c.p, c.it_gp.p, c.it_pos.p, c.it_len.p, c.it_head.p,
      c.it_done.p, c.it_dec.p, c.it_term.p, c.ev_head.p, c.ev_done.p, grouped);
  resolve_apply(c, st, W, Q, true);
}

// begun: 1 if the new round has begun already, 0 before k_round_begin
void launch_build_redo(Ctx& c, long long Q, uint32_t begun, cudaStream_t st) {
  k_build_redo<<<grid_for(Q, 256), 256, 0, st>>>(c.d_pops, c.op_pop.p, c.op_pair.p, c.op_slot.p, c.op_k.p, c.op_key.p,
                                                 c.lost_pp.p, c.lost_off.p, c.n_dev.p + 1, c.r_pop.p, c.r_pair.p,
                                                 c.r_slot.p, c.r_k.p, c.r_key.p, begun);
  note_launch();
}

// everything the captured launches depend on: sizes and device addresses
std::vector<long long> round_graph_key(const Ctx& c, const RoundBounds& b) {
  return {c.n_pop, b.kt, b.flat, b.n_gpairs, b.W, b.max_chunks, b.max_cells, c.sort_blocks, (long long)c.sort_smem,
          c.max_rounds, c.mode, c.ch_chunks, c.tune.threads[kTuneItems], c.tune.threads[kTuneChain],
          c.tune.threads[kTuneResolve], c.tune.threads[kTuneApply],
          (long long)c.d_pops, (long long)c.d_round, (long long)c.d_ctrs, (long long)c.round_dev.p,
          (long long)c.per_pop_i.p, (long long)c.pop_pair_base.p, (long long)c.gpair_pop.p,
          (long long)c.gpair_local.p, (long long)c.ev_key.p, (long long)c.ev_c.p, (long long)c.gp_c.p,
          (long long)c.ev_pos.p, (long long)c.ev_dest.p, (long long)c.ev_len.p, (long long)c.ev_head.p,
          (long long)c.ev_app.p, (long long)c.ev_done.p, (long long)c.chain_list.p, (long long)c.it_flag.p, (long long)c.it_key.p,
          (long long)c.it_c.p, (long long)c.it_gp.p, (long long)c.it_pos.p, (long long)c.it_len.p,
          (long long)c.it_head.p, (long long)c.it_start.p, (long long)c.it_done.p, (long long)c.it_dec.p, (long long)c.it_gused.p,
          (long long)c.it_term.p, (long long)c.ev_term.p, (long long)c.ppw_slot.p, (long long)c.ppw_gp.p,
          (long long)c.ch_y.p,
          (long long)c.ch_q.p, (long long)c.ch_pos.p,
          (long long)c.win_set.p, (long long)c.dec_set.p, (long long)c.rank_slot_set.p, (long long)c.rank_id_set.p,
          (long long)c.slot_base_set.p, (long long)c.id_base_set.p, (long long)c.slot_base_pp.p,
          (long long)c.id_base_pp.p, (long long)c.scan_status.p, (long long)c.scan_ctr.p,
          (long long)c.scan_err.p, (long long)c.graph_stats.p};
}

void free_redraw_graph(Ctx& c) {
  if (c.rg_exec) cudaGraphExecDestroy(c.rg_exec);
  if (c.rg_graph) cudaGraphDestroy(c.rg_graph);
  c.rg_exec = nullptr;
  c.rg_graph = nullptr;
  c.rg_key.clear();
}

// the item and event bound of the later rounds' graph for round-0 events
// e0: a power of two, at least 4096, so that it holds from step to step
long long graph_bound(long long e0) {
  long long w = 4096;
  while (w < e0) w *= 2;
  return w;
}

// Event arrays, sized in round 0 for graph_bound(samples), which bounds the
// events of every later round.  Some of them (key, slots, pair, position,
// win, destination) carry a round's events into the next one (k_items reads
// them), so nothing may reallocate them while a step runs.  The chain pool
// gets one chunk per possible chain start and 4096 more for long chains.
void reserve_events(Ctx& c, long long W) {
  size_t w = (size_t)graph_bound(W);
  c.ev_key.reserve(w + 1); c.ev_c.reserve(w + 1); c.gp_c.reserve(w + 1); c.ev_pos.reserve(w + 1);
  c.ev_dest.reserve(w + 1); c.win_set.reserve(w + 1); c.dec_set.reserve(w + 1);
  c.ev_len.reserve(w + 1); c.ev_head.reserve(w + 1); c.ev_app.reserve(w + 1); c.ev_done.reserve(w + 1);
  c.ev_term.reserve(w + 1);
  c.chain_list.reserve(w + 1);
  c.rank_slot_set.reserve(w + 2); c.rank_id_set.reserve(w + 2);
  size_t chunks = w + 4096;
  c.ch_y.reserve(chunks * kChainChunk);
  c.ch_q.reserve(chunks * kChainChunk);
  c.ch_pos.reserve(chunks * kChainChunk);
  c.ch_chunks = (long long)(std::min(std::min(c.ch_y.n, c.ch_q.n), c.ch_pos.n) / kChainChunk);
}

bool events_fit(const Ctx& c, long long W) {
  size_t w = (size_t)W;
  return c.ev_key.n >= w + 1 && c.ev_c.n >= w + 1 && c.gp_c.n >= w + 1 && c.ev_pos.n >= w + 1 &&
         c.ev_dest.n >= w + 1 && c.win_set.n >= w + 1 && c.dec_set.n >= w + 1 && c.ev_len.n >= w + 1 &&
         c.ev_head.n >= w + 1 && c.ev_app.n >= w + 1 && c.ev_done.n >= w + 1 && c.chain_list.n >= w + 1 &&
         c.ev_term.n >= w + 1 &&
         c.rank_slot_set.n >= w + 2 &&
         c.rank_id_set.n >= w + 2;
}

// the item buffers of a later round, sized for W items (they hold nothing
// from one round to the next)
void reserve_round(Ctx& c, long long W) {
  size_t w = (size_t)std::max<long long>(W, 1);
  c.it_flag.reserve(w + 1); c.it_key.reserve(w + 1); c.it_c.reserve(w + 1); c.it_gp.reserve(w + 1);
  c.it_pos.reserve(w + 1); c.it_len.reserve(w + 1); c.it_head.reserve(w + 1); c.it_done.reserve(w + 1); c.it_start.reserve(w + 1);
  c.it_dec.reserve(w + 1); c.it_gused.reserve(w + 1); c.it_term.reserve(w + 1);
}

struct GraphRun {
  long long rounds = -1;  // -1: the caller runs the rounds from the host loop
  long long losers = 0, events = 0;
  bool stopped_for_room = false;
};

// Run the later rounds of this step as the graph (captured again when a
// bound or an address changed and the change held for three steps in a row:
// after two, the next step is a graph as a whole, unless the program's own
// calls between steps keep it from that).
// e0: the events of the round before.
GraphRun run_round_graph(Ctx& c, int kt, bool flat, int n_gpairs, long long e0) {
  GraphRun out;
  RoundBounds b;
  b.kt = kt;
  b.flat = flat;
  b.n_gpairs = n_gpairs;
  // rounded up so that the graph survives ordinary step-to-step changes
  b.W = graph_bound(e0);
  // the event arrays hold the last round's events: they must already be
  // large enough (reserve_events), never reallocated here
  if (!events_fit(c, b.W)) return out;
  // the sort's chunks cover the slots of several rounds' growth; the graph
  // stops before they would not
  long long slots = 0, min_slots = -1;
  for (int k = 0; k < c.n_pop; k++) {
    slots = std::max<long long>(slots, c.n_slots_host[k]);
    min_slots = min_slots < 0 ? c.n_slots_host[k] : std::min<long long>(min_slots, c.n_slots_host[k]);
  }
  b.max_chunks = (int)((slots + 4 * b.W + kChunk - 1) / kChunk);
  b.max_chunks = (b.max_chunks + 15) / 16 * 16;
  b.max_cells = max_cells_of(c);
  prepare_chunks(c, (long long)b.max_chunks * kChunk - min_slots);
  size_sort(c, b.max_cells);
  // every other buffer at its final size before the addresses are taken
  reserve_round(c, b.W);
  c.graph_stats.reserve(kStatWords);
  {
    const long long nb = (b.W + kScanTile - 1) / kScanTile;
    reserve_scan_status(c, (size_t)std::max(kScanMaxJobs * nb, b.W / kResolveMin + 2), c.stream);
  }
  if (c.dirty) push_pops(c);
  std::vector<long long> key = round_graph_key(c, b);
  if (key != c.rg_key) {
    // bounds or addresses new since the last steps: capturing pays only when
    // they hold, so this step's later rounds run from the host loop
    c.rg_held = key == c.rg_seen ? c.rg_held + 1 : 1;
    c.rg_seen = key;
    if (c.rg_held < 3) return out;
  }
  if (key != c.rg_key) {
    free_redraw_graph(c);
    CK(cudaGraphCreate(&c.rg_graph, 0));
    cudaGraphConditionalHandle cond;
    CK(cudaGraphConditionalHandleCreate(&cond, c.rg_graph, 1, cudaGraphCondAssignDefault));
    cudaGraphNodeParams np = {};
    np.type = cudaGraphNodeTypeConditional;
    np.conditional.handle = cond;
    np.conditional.type = cudaGraphCondTypeWhile;
    np.conditional.size = 1;
    cudaGraphNode_t node;
    CK(cudaGraphAddNode(&node, c.rg_graph, nullptr, 0, &np));
    cudaGraph_t body = np.conditional.phGraph_out[0];
    bool prof = c.prof;
    c.prof = false;  // no event records inside the body
    long long n0 = g_launches;
    CK(cudaStreamBeginCaptureToGraph(c.cap_stream, body, nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed));
    try {
      k_round_begin<<<1, 128, 0, c.cap_stream>>>(c.d_round, c.round_dev.p, c.per_pop_i.p, 4 * c.n_pop, c.n_dev.p);
      note_launch();
      enqueue_round_head(c, c.cap_stream, b, 0);
      enqueue_round_tail(c, c.cap_stream, b, 0);
      k_round_end<<<1, 128, 0, c.cap_stream>>>(c.round_dev.p, c.graph_stats.p, c.d_round, c.max_rounds, c.d_pops,
                                               c.d_ctrs, c.n_pop, (long long)b.max_chunks * kChunk, b.W, 0, c.n_dev.p,
                                               c.scan_err.p, nullptr, cond);
      note_launch();
    } catch (...) {
      cudaGraph_t dummy;
      cudaStreamEndCapture(c.cap_stream, &dummy);
      c.prof = prof;
      free_redraw_graph(c);
      throw;
    }
    cudaGraph_t captured = nullptr;
    CK(cudaStreamEndCapture(c.cap_stream, &captured));
    c.prof = prof;
    c.rg_nodes = g_launches - n0;
    g_launches = n0;  // counted when they run
    CK(cudaGraphInstantiate(&c.rg_exec, c.rg_graph, 0));
    c.rg_key = key;
    c.rg_builds++;
  }
  CK(cudaMemsetAsync(c.graph_stats.p, 0, sizeof(long long) * kStatWords, c.stream));
  {
    ProfScope ps(c, 2, 1);
    CK(cudaGraphLaunch(c.rg_exec, c.stream));
  }
  long long st[4] = {0, 0, 0, 0};
  CK(cudaMemcpyAsync(st, c.graph_stats.p, sizeof(st), cudaMemcpyDeviceToHost, c.stream));
  unsigned long long scan_err = 0;
  CK(cudaMemcpyAsync(&scan_err, c.scan_err.p, sizeof(scan_err), cudaMemcpyDeviceToHost, c.stream));
  CK(cudaStreamSynchronize(c.stream));
  if (scan_err) {
    CK(cudaMemsetAsync(c.scan_err.p, 0, sizeof(scan_err), c.stream));
    throw Fail(PMC_ERR_TIMEOUT);
  }
  g_launches += c.rg_nodes * st[2];
  c.claim_gen += (uint32_t)st[2];
  out.rounds = st[2];
  out.losers = st[0];
  out.events = st[1];
  out.stopped_for_room = st[3] != 0;
  return out;
}

// capacity for a round that may add `slots` new slots to every population
void ensure_room(Ctx& c, long long slots) {
  for (int k = 0; k < c.n_pop; k++) {
    long long need = (long long)c.n_slots_host[k] + slots;
    if (need > c.pops[k].h.cap) {
      int nc = (int)std::min<long long>(std::max<long long>(need * 3 / 2, 1024), (1LL << 31) - 1);
      relayout(c, k, nc, false);  // slot numbers kept
    }
  }
}

// the populations' places in the global pair list
std::vector<long long> pair_layout(const Ctx& c) {
  std::vector<long long> base(c.n_pop + 1, 0);
  for (int k = 0; k < c.n_pop; k++) base[k + 1] = base[k] + c.pops[k].h.n_pairs;
  return base;
}

// pairs the step graph is captured for: a multiple of 1024, so that a changed
// grid seldom needs another capture; the places past the last pair are empty
int padded_pairs(long long n) { return (int)((n + 1023) / 1024 * 1024); }

// global pair list, uploaded when its layout changes
void upload_pair_layout(Ctx& c, const std::vector<long long>& base) {
  if (base == c.base_cached) return;
  c.base_cached.clear();  // if a buffer does not fit
  const int n = padded_pairs(base[c.n_pop]);
  std::vector<int> gp_pop(std::max(n, 1), 0), gp_loc(std::max(n, 1), 0);
  for (int k = 0; k < c.n_pop; k++)
    for (int p = 0; p < c.pops[k].h.n_pairs; p++) {
      gp_pop[base[k] + p] = k;
      gp_loc[base[k] + p] = p;
    }
  c.gpair_pop.reserve(gp_pop.size());
  c.gpair_local.reserve(gp_loc.size());
  c.pop_pair_base.reserve(base.size());
  CK(cudaMemcpyAsync(c.gpair_pop.p, gp_pop.data(), sizeof(int) * gp_pop.size(), cudaMemcpyHostToDevice, c.stream));
  CK(cudaMemcpyAsync(c.gpair_local.p, gp_loc.data(), sizeof(int) * gp_loc.size(), cudaMemcpyHostToDevice, c.stream));
  CK(cudaMemcpyAsync(c.pop_pair_base.p, base.data(), sizeof(long long) * base.size(), cudaMemcpyHostToDevice, c.stream));
  c.base_cached = base;
}

void free_step_graph(Ctx& c) {
  if (c.sg_exec) cudaGraphExecDestroy(c.sg_exec);
  if (c.sg_graph) cudaGraphDestroy(c.sg_graph);
  c.sg_exec = nullptr;
  c.sg_graph = nullptr;
  c.sg_key.clear();
}

// 16-byte words of the step graph's report
int report_words(const Ctx& c) {
  return (int)((sizeof(long long) * kStatWords + sizeof(PopCtr) * c.n_pop + 15) / 16);
}

// what the step graph's captured launches depend on, beyond round_graph_key
std::vector<long long> step_graph_key(const Ctx& c, const RoundBounds& b, long long w_cap, int max_pairs,
                                      long long q_cap, long long qb_cap) {
  std::vector<long long> k = round_graph_key(c, b);
  if (q_cap > 0)
    for (long long v :
         {q_cap, qb_cap, (long long)c.op_pop.p, (long long)c.op_pair.p, (long long)c.op_slot.p, (long long)c.op_k.p,
          (long long)c.op_key.p, (long long)c.r_pop.p, (long long)c.r_pair.p, (long long)c.r_slot.p,
          (long long)c.r_k.p, (long long)c.r_key.p, (long long)c.pp_res.p, (long long)c.pp_vol.p,
          (long long)c.pp_rm_off.p, (long long)c.pp_rm_tot.p, (long long)c.pp_rm_pool.p,
          (long long)c.pp_rm_pool.n, (long long)c.win_pp.p,
          (long long)c.lost_pp.p, (long long)c.lost_off.p, (long long)c.rank_slot_pp.p,
          (long long)c.grp_dest.p, (long long)c.grp_hist.p, (long long)c.grp_off.p, (long long)c.item_pop.p,
          (long long)c.wk_slot.p, (long long)c.wk_gp.p, (long long)c.wk_flag.p})
      k.push_back(v);
  for (long long v : {(long long)c.report.dev, (long long)c.report_seq.p, (long long)c.n_dev.p, w_cap, (long long)max_pairs, (long long)c.prof, (long long)c.tune.threads[kTuneTest],
                      (long long)c.nwork_set.p, (long long)c.nwork_pp.p, (long long)c.work_off.p,
                      (long long)c.pp_off.p, (long long)c.flag.p, (long long)c.ev.p, (long long)c.ev_gp.p,
                      (long long)c.d_stat})
    k.push_back(v);
  return k;
}

// The step graph's nodes, captured on c.cap_stream: round 0, then the WHILE
// node over the later rounds.
void capture_step_graph(Ctx& c, const RoundBounds& b, long long w_cap, int max_pairs, long long q_cap, long long qb_cap) {
  CK(cudaGraphCreate(&c.sg_graph, 0));
  cudaGraphConditionalHandle cond;
  CK(cudaGraphConditionalHandleCreate(&cond, c.sg_graph, 0, cudaGraphCondAssignDefault));
  cudaStream_t st = c.cap_stream;
  const long long sort_slots = (long long)b.max_chunks * kChunk;
  const int n_gp = b.n_gpairs;
  auto mark = [&](int k) {
    if (c.prof) CK(cudaEventRecordWithFlags(c.sg_ev[k], st, cudaEventRecordExternal));
  };
  const long long n0 = g_launches;
  c.chained = true;
  CK(cudaStreamBeginCaptureToGraph(st, c.sg_graph, nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed));
  cudaGraph_t done = nullptr;
  try {
    mark(0);
    StepBegin begin;
    begin.pops = c.d_pops;
    begin.ctrs = c.d_ctrs;
    begin.d_round = c.d_round;
    begin.round_dev = c.round_dev.p;
    begin.per_pop = c.per_pop_i.p;
    begin.stat = c.d_stat;
    begin.n_stat = kStatWords;
    begin.pop_pair_base = c.pop_pair_base.p;
    begin.n_gp = n_gp;
    begin.nwork_set = c.nwork_set.p;
    begin.nwork_pp = c.nwork_pp.p;
    launch_sort(c, st, b.max_chunks, b.max_cells, begin);
    mark(1);
    launch_chained(c, k_pairs, dim3(dim3((max_pairs + 127) / 128, c.n_pop)), dim3(128), 0, st, c.d_pops, c.pop_pair_base.p, c.nwork_set.p,
                                                                   c.nwork_pp.p, 1);
    scan_multi<long long>(c, {{c.nwork_set.p, n_gp, nullptr, c.work_off.p}, {c.nwork_pp.p, n_gp, nullptr, c.pp_off.p}},
                          st);
    if (q_cap > 0) {
      launch_build_ops(c, n_gp, q_cap, st);
      launch_pp_count(c, q_cap, c.pp_off.p + n_gp, st);
    }
    launch_chained(c, k_step_check, dim3(1), dim3(256), 0, st, c.d_pops, c.n_pop, c.pop_pair_base.p, c.work_off.p, c.pp_off.p, n_gp, w_cap, q_cap,
                                    c.pp_rm_tot.p, (long long)c.pp_rm_pool.n, sort_slots, c.n_dev.p, c.d_stat, c.scan_err.p);
    if (q_cap > 0) launch_pp_ops(c, b.kt, q_cap, st);
    mark(2);
    launch_test_kt(c, b.kt, b.flat, n_gp, w_cap, st);
    mark(3);
    const long long* Wd = c.work_off.p + n_gp;
    launch_compact_samples(c, Wd, w_cap, st);
    resolve_apply(c, st, w_cap, q_cap, false);
    k_round_end<<<1, 128, 0, st>>>(c.round_dev.p, c.d_stat, c.d_round, c.max_rounds, c.d_pops, c.d_ctrs, c.n_pop,
                                   sort_slots, b.W, qb_cap, c.n_dev.p, c.scan_err.p, c.per_pop_i.p, cond);
    note_launch();
    mark(4);
    c.sg_nodes0 = g_launches - n0;
    // a conditional node follows the launches captured so far, and what the
    // stream captures next follows it
    auto add_conditional = [&](cudaGraphConditionalHandle h, cudaGraphConditionalNodeType type) {
      cudaStreamCaptureStatus cs;
      unsigned long long id = 0;
      cudaGraph_t g = nullptr;
      const cudaGraphNode_t* deps = nullptr;
      size_t n_deps = 0;
      CK(cudaStreamGetCaptureInfo_v2(st, &cs, &id, &g, &deps, &n_deps));
      std::vector<cudaGraphNode_t> dv(deps, deps + n_deps);
      cudaGraphNodeParams np = {};
      np.type = cudaGraphNodeTypeConditional;
      np.conditional.handle = h;
      np.conditional.type = type;
      np.conditional.size = 1;
      cudaGraphNode_t node;
      CK(cudaGraphAddNode(&node, g, dv.data(), dv.size(), &np));
      CK(cudaStreamUpdateCaptureDependencies(st, &node, 1, cudaStreamSetCaptureDependencies));
      return np.conditional.phGraph_out[0];
    };
    cudaGraph_t body = add_conditional(cond, cudaGraphCondTypeWhile);
    mark(5);
    k_step_report<<<1, 1024, 0, st>>>((const uint4*)c.d_stat, report_words(c), (uint4*)c.report.dev,
                                      (unsigned*)((char*)c.report.dev + 16 * (size_t)report_words(c)), c.report_seq.p);
    note_launch();
    CK(cudaStreamEndCapture(st, &done));
    const long long n1 = g_launches;
    CK(cudaStreamBeginCaptureToGraph(st, body, nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed));
    if (qb_cap > 0) launch_build_redo(c, qb_cap, 1, st);  // the round has begun (k_round_end)
    c.fork = true;
    enqueue_round_head(c, st, b, qb_cap);
    if (qb_cap > 0) {
      // the tail runs if the round's removals fit their pool
      cudaGraphConditionalHandle fits;
      CK(cudaGraphConditionalHandleCreate(&fits, body, 0, cudaGraphCondAssignDefault));
      k_pp_fits<<<1, 1, 0, st>>>(c.pp_rm_tot.p, (long long)c.pp_rm_pool.n, c.d_stat, fits, cond);
      note_launch();
      cudaGraph_t tail = add_conditional(fits, cudaGraphCondTypeIf);
      CK(cudaStreamEndCapture(st, &done));
      CK(cudaStreamBeginCaptureToGraph(st, tail, nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed));
    }
    enqueue_round_tail(c, st, b, qb_cap);
    c.fork = false;
    k_round_end<<<1, 128, 0, st>>>(c.round_dev.p, c.d_stat, c.d_round, c.max_rounds, c.d_pops, c.d_ctrs, c.n_pop,
                                   sort_slots, b.W, qb_cap, c.n_dev.p, c.scan_err.p, c.per_pop_i.p, cond);
    note_launch();
    c.sg_nodes = g_launches - n1;
  } catch (...) {
    c.fork = c.chained = false;
    cudaStreamEndCapture(st, &done);
    cudaGetLastError();
    g_launches = n0;
    free_step_graph(c);
    throw;
  }
  c.chained = false;
  CK(cudaStreamEndCapture(st, &done));
  g_launches = n0;  // counted when they run
  CK(cudaGraphInstantiate(&c.sg_exec, c.sg_graph, 0));
}

constexpr int kPPIdle = 8;  // steps
constexpr int kGraphPause = 32;  // steps the long way after bounds that did not fit the device

// a step's buffers that hold nothing between steps
void release_step_buffers(Ctx& c) {
  auto release = [](auto&... b) { (b.release(), ...); };
  release(c.flag, c.ev, c.ev_gp, c.ev_key, c.ev_c, c.gp_c, c.ev_pos, c.ev_dest, c.win_set, c.dec_set, c.ev_len,
          c.ev_head, c.ev_app, c.ev_done, c.ev_term, c.chain_list, c.rank_slot_set, c.rank_id_set, c.ch_y, c.ch_q,
          c.ch_pos);
  release(c.it_flag, c.it_key, c.it_c, c.it_gp, c.it_pos, c.it_len, c.it_head, c.it_done, c.it_start, c.it_dec,
          c.it_gused, c.it_term);
  release(c.op_pop, c.op_pair, c.op_slot, c.op_k, c.op_key, c.r_pop, c.r_pair, c.r_slot, c.r_k, c.r_key, c.pp_res,
          c.pp_vol, c.pp_rm_off, c.pp_rm_pool, c.wk_slot, c.wk_gp, c.wk_flag, c.ppw_slot, c.ppw_gp);
}

struct StepRun {
  bool ran = false;   // round 0 ran on the device
  // 1: work is left, the host loop carries on after `rounds` rounds; 2: also
  // the last round's tail (the removals of its target operations did not fit)
  int stopped = 0;
  long long rounds = 0, losers = 0, events = 0, ops = 0, ops_lost = 0;
  RoundBounds b;
  long long Q = 0;    // bound of a later round's target operations
};

// Run this step as the graph, if what it relies on holds: a valid sort and
// current caches and bounds from the steps before.  d_pops' copies keep their
// step count on the device (the sort's step_begin adds one), so a step whose
// parameters are those of the last one pushes nothing.  Its report comes by
// stores to mapped host memory, without a copy or a synchronisation.  The step
// the long way makes six read-backs, with the copies and launches that wait on
// them: 0.351 ms a step for 1e4 particles under the additive kernel, 0.160 with
// the graph when it came, 0.11 with its kernels as they are now; 0.860, 0.689
// and 0.59 for 1e6 particles of 20 species.
StepRun run_step_graph(Ctx& c, int kt, bool params_same) {
  StepRun out;
  if (!c.use_graph || c.tuner.on || !c.ctrs_fresh || c.last_w < 0) return out;
  if (c.sg_pause > 0) {
    c.sg_pause--;
    return out;
  }
  if (c.claim_gen + 1 + (uint32_t)c.max_rounds + 2u >= kGenLimit) return out;  // the generations restart
  if (c.base_cached.size() != (size_t)c.n_pop + 1) return out;
  RoundBounds b;
  b.kt = kt;
  b.flat = true;
  int max_pairs = 1;
  long long slots = 0, min_slots = -1;
  for (int k = 0; k < c.n_pop; k++) {
    const PopHost& ph = c.pops[k];
    if (!ph.valid_sort || !caches_current(c, ph) || !ph.h.kmax_valid || !ph.h.pair_setup_valid || (ph.h.walk_stops && !c.pp_step) ||
        c.base_cached[k + 1] - c.base_cached[k] != ph.h.n_pairs)
      return out;
    b.flat = b.flat && ph.h.flat;
    max_pairs = std::max(max_pairs, ph.h.n_pairs);
    slots = std::max<long long>(slots, c.n_slots_host[k]);
    min_slots = min_slots < 0 ? c.n_slots_host[k] : std::min<long long>(min_slots, c.n_slots_host[k]);
  }
  // bounds that hold from step to step: powers of two above the last step's
  // counts, lowered only when they are 16 times too large
  const long long w = graph_bound(c.last_w + c.last_w / 4), e = graph_bound(c.last_e0 + c.last_e0 / 4);
  if (w > c.sg_w || 16 * w <= c.sg_w) c.sg_w = w;
  if (e > c.sg_e || 16 * e <= c.sg_e) c.sg_e = e;
  long long q_cap = 0, qb_cap = 0;
  if (c.pp_step) {
    // room for twice as many when they outgrow it
    const long long q = graph_bound(c.last_q + c.last_q / 4), qb = graph_bound(c.last_qb + c.last_qb / 4);
    if (q > c.sg_q || 16 * q <= c.sg_q) c.sg_q = 2 * q;
    if (qb > c.sg_qb || 16 * qb <= c.sg_qb) c.sg_qb = 2 * qb;
    q_cap = c.sg_q;
    qb_cap = c.sg_qb;
  }
  b.W = c.pp_step ? c.sg_e : std::min(c.sg_e, c.sg_w);
  b.n_gpairs = padded_pairs(c.base_cached[c.n_pop]);
  max_pairs = (max_pairs + 511) / 512 * 512;
  b.max_cells = (max_cells_of(c) + 15) / 16 * 16;
  b.max_chunks = (int)((slots + 4 * b.W + kMaxCopies * qb_cap + kChunk - 1) / kChunk);
  b.max_chunks = (b.max_chunks + 15) / 16 * 16;
  auto prepare = [&]() -> bool {
    prepare_chunks(c, (long long)b.max_chunks * kChunk - min_slots);
    size_sort(c, b.max_cells);
    // every buffer at its final size before the addresses are taken
    const size_t ng = (size_t)b.n_gpairs + 1;
    c.nwork_set.reserve(ng);
    c.nwork_pp.reserve(ng);
    c.work_off.reserve(ng);
    c.pp_off.reserve(ng);
    const size_t ws = (size_t)c.sg_w;
    c.flag.reserve(ws + 1); c.ev.reserve(ws + 1); c.ev_gp.reserve(ws + 1);
    reserve_events(c, std::max(c.sg_w + kMaxCopies * q_cap, b.W));
    reserve_round(c, b.W);
    c.pp_rm_tot.reserve(1);
    if (!c.report.p) {
      c.report_seq.reserve(1);
      CK(cudaMemsetAsync(c.report_seq.p, 0, sizeof(unsigned) * c.report_seq.n, c.stream));
      c.report.reserve(16 * (size_t)report_words(c) + 64);
      memset(c.report.p, 0, c.report.bytes);
    }
    if (q_cap > 0) {
      const long long q = std::max(q_cap, qb_cap);
      reserve_ops(c, q);
      reserve_redo(c, q);
      c.ppw_slot.reserve((size_t)(kMaxCopies * (q + 1)));
      c.ppw_gp.reserve((size_t)(kMaxCopies * (q + 1)));
      if (c.n_pop > 1) {
        c.item_pop.reserve((size_t)b.W + 1);
        c.grp_dest.reserve((size_t)b.W + 1);
        const size_t nh = (size_t)((b.W + kGrpTile - 1) / kGrpTile) * c.n_pop;
        c.grp_hist.reserve(nh);
        c.grp_off.reserve(nh + 1);
      }
      // twice the largest bound seen, so that it seldom grows
      if (2 * c.last_rm + 1024 > (long long)c.pp_rm_pool.n) c.pp_rm_pool.reserve((size_t)(4 * c.last_rm + 65536));
    }
    {
      const long long qs = std::max(q_cap, qb_cap), hist = (std::max(qs, q_cap > 0 ? b.W : 0) / kGrpTile + 2) * c.n_pop;
      const long long lists = std::max(std::max(kMaxCopies * qs, hist), (long long)b.n_gpairs);
      const long long nb = std::max((c.sg_w + kScanTile - 1) / kScanTile, (lists + kScanTile - 1) / kScanTile);
      reserve_scan_status(
          c, (size_t)std::max(std::max(kScanMaxJobs * nb, std::max(c.sg_w, b.W) / kResolveMin + 2), qs / 64 + 2), c.stream);
    }
    c.op_cap = qb_cap;
    if (c.prof)
      for (auto& ev : c.sg_ev)
        if (!ev) CK(cudaEventCreate(&ev));
    const std::vector<long long> key = step_graph_key(c, b, c.sg_w, max_pairs, q_cap, qb_cap);
    if (key != c.sg_key) {
      // captured when the bounds and addresses hold for two steps; at once where
      // a step the long way, with its host-driven rounds, costs several captures
      // (0.2 to 0.3 ms each)
      if (key != c.sg_seen && !c.pp_step) {
        c.sg_seen = key;
        return false;
      }
      CK(cudaStreamSynchronize(c.stream));  // a graph's report comes before its end
      free_step_graph(c);
      capture_step_graph(c, b, c.sg_w, max_pairs, q_cap, qb_cap);
      c.sg_key = key;
    }
    return true;
  };
  try {
    if (!prepare()) return out;
  } catch (const Fail&) {
    // the bounds do not fit the device: the long way needs less (an error that
    // stays is its to report)
    cudaGetLastError();
    free_step_graph(c);
    c.sg_seen.clear();
    release_step_buffers(c);
    c.sg_pause = kGraphPause;
    return out;
  }
  // the sort's step_begin advances the device's step counts, which have to be
  // at the step before (a new seed restarts the host's; any call may have
  // copied the population since)
  bool counts = true;
  for (const auto& ph : c.pops) counts = counts && ph.dev_step + 1u == ph.h.step;
  if (c.dirty || !params_same || !counts) {
    for (auto& ph : c.pops) ph.h.step -= 1u;
    push_pops(c);
    for (auto& ph : c.pops) ph.h.step += 1u;
  }
  CK(cudaGraphLaunch(c.sg_exec, c.stream));
  for (auto& ph : c.pops) ph.dev_step++;
  c.report_count++;
  {
    // the report's sequence number; a look at the stream now and then, for an
    // error or a graph that ended without it.  The wait spins, unless the
    // process chose another (cudaSetDeviceFlags), as a stream synchronisation
    // would
    const volatile unsigned* flag = (const volatile unsigned*)((const char*)c.report.p + 16 * (size_t)report_words(c));
    unsigned sched = 0;
    CK(cudaGetDeviceFlags(&sched));
    sched &= cudaDeviceScheduleMask;
    if (sched == cudaDeviceScheduleBlockingSync) CK(cudaStreamSynchronize(c.stream));
    for (long long spins = 1; *flag != c.report_count; spins++) {
      if (sched == cudaDeviceScheduleYield) std::this_thread::yield();
      if (spins % 4096 != 0) continue;
      const cudaError_t e = cudaStreamQuery(c.stream);
      if (e == cudaErrorNotReady) continue;
      CK(e);
      if (*flag != c.report_count) throw Fail(PMC_ERR_CUDA);
    }
    std::atomic_thread_fence(std::memory_order_acquire);
  }
  const unsigned char* report = (const unsigned char*)c.report.p;
  long long stat[kStatWords];
  memcpy(stat, report, sizeof(stat));
  c.last_w = stat[5];
  // target operations may come and go from step to step: their bounds follow
  // a fall by half a step, a rise at once
  c.last_q = std::max(stat[12], c.last_q / 2);
  c.last_rm = std::max(c.last_rm, stat[11]);
  if (stat[4]) {
    c.ctrs_fresh = false;
    return out;  // nothing was tested; the long way starts the step over
  }
  if (stat[6]) {
    CK(cudaMemsetAsync(c.scan_err.p, 0, sizeof(unsigned long long), c.stream));
    throw Fail(PMC_ERR_TIMEOUT);
  }
  memcpy(c.h_ctrs.data(), report + sizeof(stat), sizeof(PopCtr) * c.n_pop);
  for (int k = 0; k < c.n_pop; k++) c.n_slots_host[k] = c.h_ctrs[k].n_slots;
  if (c.prof) {
    const long long units[3] = {slots * c.n_pop, stat[5], 1};
    const int id[3] = {1, 0, 2};
    for (int j = 0; j < 3; j++) {
      float ms = 0.f;
      CK(cudaEventElapsedTime(&ms, c.sg_ev[2 * j], c.sg_ev[2 * j + 1]));
      c.prof_ms[id[j]] += ms;
      c.prof_launch[id[j]] += 1;
      c.prof_units[id[j]] += units[j];
    }
  }
  g_launches += c.sg_nodes0 + c.sg_nodes * (stat[2] - 1);
  c.claim_gen += (uint32_t)(stat[2] + (stat[3] == 2 ? 1 : 0));  // a round left in the middle has begun
  c.last_e0 = stat[7];
  c.last_qb = std::max(stat[8], c.last_qb / 2);
  for (int k = 0; k < c.n_pop; k++) c.pops[k].h.walk_stops = c.h_ctrs[k].walk_stops;
  // without target operations for a while, back to the graph without them
  c.pp_idle = stat[12] > 0 ? 0 : c.pp_idle + 1;
  if (c.pp_idle >= kPPIdle && !stat[3]) c.pp_step = false;
  out.ran = true;
  out.rounds = stat[2];
  out.losers = stat[0];
  out.events = stat[1];
  out.ops = stat[9];
  out.ops_lost = stat[10];
  out.stopped = (int)stat[3];
  out.b = b;
  out.Q = qb_cap;
  return out;
}

void step_rounds(Ctx& c, int kt, bool flat, int n_gpairs, long long Q, int round, bool counted, long long redraws,
                 bool graph_tried);

// params_same: the populations' parameters are those of the last step
void step_parallel(Ctx& c, int kt, bool params_same) {
  {
    const StepRun g = run_step_graph(c, kt, params_same);
    if (g.ran) {
      c.last_set_losers = g.losers;
      c.last_pp_lost = g.ops_lost;
      c.last_ops = g.ops;
      c.last_events = g.events;
      c.last_redraws = g.losers + g.ops_lost;
      c.last_rounds = g.rounds;
      if (!g.stopped) return;
      c.ctrs_fresh = false;
      if (g.stopped == 2) {
        fit_rm_pool(c);
        enqueue_round_tail(c, c.stream, g.b, g.Q);
      }
      step_rounds(c, kt, g.b.flat, (int)c.base_cached[c.n_pop], g.Q, (int)g.rounds, g.stopped != 2, g.losers + g.ops_lost,
                  true);
      return;
    }
  }
  c.ctrs_fresh = false;
  k_step_reset<<<(c.n_pop + 127) / 128, 128, 0, c.stream>>>(c.d_ctrs, c.n_pop);
  note_launch();
  push_pops(c);
  sort_pops(c, true);
  const std::vector<long long> base = pair_layout(c);
  const int n_gpairs = (int)base[c.n_pop];
  const size_t ng = (size_t)n_gpairs + 1;
  upload_pair_layout(c, base);
  c.nwork_set.reserve(ng);
  c.nwork_pp.reserve(ng);
  c.work_off.reserve(ng);
  c.pp_off.reserve(ng);
  c.per_pop_i.reserve(4 * (size_t)c.n_pop);
  c.slot_base_set.reserve(c.n_pop);
  c.slot_base_pp.reserve(c.n_pop);
  c.id_base_set.reserve(c.n_pop);
  c.id_base_pp.reserve(c.n_pop);
  c.n_dev.reserve(4 + 2 * (size_t)c.n_pop);
  // round_dev: [0] losers, [1] events, [2] items, [3] chain chunks, [4] chains,
  // [5] walkers of target operations, [6] items that are events, [7] items
  // that are such walkers, [8] target operations that lost a claim,
  // [10] chains that k_chain carries on
  c.round_dev.reserve(12);
  int max_pairs = 1, nb_max = 1, max_cap = 1;
  for (int k = 0; k < c.n_pop; k++) {
    max_pairs = std::max(max_pairs, c.pops[k].h.n_pairs);
    nb_max = std::max(nb_max, c.pops[k].n_bin);
    max_cap = std::max(max_cap, c.pops[k].h.cap);
  }
  bool flat = true;
  for (int k = 0; k < c.n_pop; k++) flat = flat && c.pops[k].h.flat;
  c.last_set_losers = c.last_pp_lost = c.last_events = c.last_ops = 0;
  std::vector<long long> hw(3 + 2 * (size_t)c.n_pop);

  // ---- round 0: every pair's samples and target operations
  {
    // a new claim generation for every round; they restart (with every
    // claim and touched word cleared) before a step could run out of them
    c.claim_gen++;
    bool wrapped = false;
    if (c.claim_gen + (uint32_t)c.max_rounds + 2u >= kGenLimit) {
      c.claim_gen = 1;
      wrapped = true;
    }
    uint32_t rg[2] = {0u, c.claim_gen};  // staged before the call returns
    CK(cudaMemcpyAsync(c.d_round, rg, sizeof(rg), cudaMemcpyHostToDevice, c.stream));
    if (c.dirty) push_pops(c);
    if (wrapped) {
      dim3 g(grid_for(max_cap, 256), c.n_pop);
      k_fill_claims<<<g, 256, 0, c.stream>>>(c.d_pops);
      note_launch();
    }
  }
  bool need_kmax = false, need_setup = false;
  for (int k = 0; k < c.n_pop; k++) {
    need_kmax = need_kmax || !c.pops[k].h.kmax_valid;
    need_setup = need_setup || !c.pops[k].h.pair_setup_valid;
  }
  if (need_kmax) {
    launch_kmax(c);
  }
  if (need_setup) {
    dim3 g((unsigned)(((long long)max_pairs * 32 + 255) / 256), c.n_pop);
    k_pair_setup<<<g, 256, 0, c.stream>>>(c.d_pops);
    note_launch();
  }
  {
    dim3 gp((max_pairs + 127) / 128, c.n_pop);
    launch_chained(c, k_pairs, dim3(gp), dim3(128), 0, c.stream, c.d_pops, c.pop_pair_base.p, c.nwork_set.p, c.nwork_pp.p, 1);
  }
  // the device copies learn this with the next push
  for (int k = 0; k < c.n_pop; k++) {
    c.pops[k].h.kmax_valid = 1;
    c.pops[k].h.pair_setup_valid = 1;
  }
  c.dirty = true;
  scan_multi<long long>(c, {{c.nwork_set.p, n_gpairs, nullptr, c.work_off.p},
                            {c.nwork_pp.p, n_gpairs, nullptr, c.pp_off.p}});
  long long W, Q;
  {
    long long* popw = c.n_dev.p + 4;
    if (c.n_pop > 1) {
      k_pop_work<<<(c.n_pop + 127) / 128, 128, 0, c.stream>>>(c.pop_pair_base.p, c.n_pop, c.work_off.p, c.pp_off.p,
                                                              popw);
      note_launch();
    }
    // one read-back: totals and per-population work
    CK(cudaMemcpyAsync(&hw[0], c.work_off.p + n_gpairs, sizeof(long long), cudaMemcpyDeviceToHost, c.stream));
    CK(cudaMemcpyAsync(&hw[1], c.pp_off.p + n_gpairs, sizeof(long long), cudaMemcpyDeviceToHost, c.stream));
    if (c.n_pop > 1)
      CK(cudaMemcpyAsync(&hw[3], popw, sizeof(long long) * 2 * c.n_pop, cudaMemcpyDeviceToHost, c.stream));
    unsigned long long pair_scan_err = 0;
    CK(cudaMemcpyAsync(&pair_scan_err, c.scan_err.p, sizeof(pair_scan_err), cudaMemcpyDeviceToHost, c.stream));
    CK(cudaStreamSynchronize(c.stream));
    if (pair_scan_err) {
      CK(cudaMemsetAsync(c.scan_err.p, 0, sizeof(pair_scan_err), c.stream));
      throw Fail(PMC_ERR_TIMEOUT);
    }
    W = hw[0];
    Q = hw[1];
    if (c.n_pop == 1) {
      hw[3] = W;
      hw[4] = Q;
    }
    // in a step with target operations walks that reach a per-particle pair's
    // target cell stop for one; a population's walks stop when it has target
    // operations of its own, so it steps the same alone and in a batch (in a
    // step graph k_step_check sets this)
    c.pp_step = Q > 0;
    c.pp_idle = 0;
    for (int k = 0; k < c.n_pop; k++) {
      const int stops = hw[3 + 2 * k + 1] > 0 ? 1 : 0;
      if (c.pops[k].h.walk_stops != stops) {
        c.pops[k].h.walk_stops = stops;
        c.dirty = true;
      }
    }
    // sample numbers fit in a key's 31 bits below the walk flag of the merge stream
    if (W + Q + 1 >= 0x7fffffffLL) cap_throw("more than 2^31 samples in one step");
  }
  // capacity for the worst case of this round: every sample creates a
  // particle and every target operation makes kMaxCopies - 1 copies
  for (int k = 0; k < c.n_pop; k++) {
    long long need = (long long)c.n_slots_host[k] + hw[3 + 2 * k] + (kMaxCopies - 1) * hw[3 + 2 * k + 1];
    if (need > c.pops[k].h.cap) {
      int nc = (int)std::min<long long>(std::max<long long>(need * 3 / 2, 1024), (1LL << 31) - 1);
      relayout(c, k, nc, false);  // slot numbers kept
    }
  }
  {
    size_t w = (size_t)W;
    c.flag.reserve(w + 1); c.ev.reserve(w + 1); c.ev_gp.reserve(w + 1);
    // the walkers that target operations make (the target and its copies)
    // join a later round's items and events
    reserve_events(c, W + kMaxCopies * Q);
    c.ppw_slot.reserve((size_t)(kMaxCopies * (Q + 1)));
    c.ppw_gp.reserve((size_t)(kMaxCopies * (Q + 1)));
    c.op_cap = Q;
  }
  if (c.dirty) push_pops(c);
  CK(cudaMemsetAsync(c.round_dev.p, 0, sizeof(long long) * 12, c.stream));
  CK(cudaMemsetAsync(c.per_pop_i.p, 0, sizeof(int) * 4 * c.n_pop, c.stream));
  if (W > 0) {
    ProfScope ps(c, 0, W);
    launch_test_kt(c, kt, flat, n_gpairs, W, c.stream);
  }
  if (Q > 0) {
    reserve_ops(c, Q);
    launch_build_ops(c, n_gpairs, Q, c.stream);
    CK(cudaMemcpyAsync(c.n_dev.p + 1, &Q, sizeof(long long), cudaMemcpyHostToDevice, c.stream));
    launch_pp_count(c, Q, c.n_dev.p + 1, c.stream);  // built in population order
    fit_rm_pool(c);
    launch_pp_ops(c, kt, Q, c.stream);
  }
  // accepted samples in sample order; the sample count is work_off[n_gpairs]
  // and the event count E goes to round_dev[1], both on the device
  if (W > 0) {
    const long long* Wd = c.work_off.p + n_gpairs;
    launch_compact_samples(c, Wd, W, c.stream);
  }
  resolve_apply(c, c.stream, W, Q, false);

  c.last_w = W;
  c.last_q = Q;
  c.last_e0 = c.last_qb = 0;
  step_rounds(c, kt, flat, n_gpairs, Q, 0, false, 0, false);
}

// The later rounds: retries, walks and per-particle redo operations, from the
// end of round 0 (round = 0, its Q target operations), or from a round at
// which a graph stopped for lack of room, after `round` rounds (counted: the
// last one's counts are in the statistics already).
void step_rounds(Ctx& c, int kt, bool flat, int n_gpairs, long long Q, int round, bool counted, long long redraws,
                 bool graph_tried) {
  std::vector<int> per_pop(4 * (size_t)c.n_pop);
  long long E = 0, pp_lost = 0;
  long long last_qb = Q;  // bound of the last round's target operations (0: it had none)
  for (;;) {
    // one read-back at the end of each host round
    long long losers = 0, ppw = 0;
    CK(cudaMemcpyAsync(&losers, c.round_dev.p, sizeof(long long), cudaMemcpyDeviceToHost, c.stream));
    CK(cudaMemcpyAsync(&E, c.round_dev.p + 1, sizeof(long long), cudaMemcpyDeviceToHost, c.stream));
    CK(cudaMemcpyAsync(&ppw, c.round_dev.p + 5, sizeof(long long), cudaMemcpyDeviceToHost, c.stream));
    long long Qr = 0;
    pp_lost = 0;
    if (last_qb > 0) {
      CK(cudaMemcpyAsync(&pp_lost, c.round_dev.p + 8, sizeof(long long), cudaMemcpyDeviceToHost, c.stream));
      CK(cudaMemcpyAsync(&Qr, c.n_dev.p + 1, sizeof(long long), cudaMemcpyDeviceToHost, c.stream));
    }
    CK(cudaMemcpyAsync(per_pop.data(), c.per_pop_i.p, sizeof(int) * 4 * c.n_pop, cudaMemcpyDeviceToHost, c.stream));
    unsigned long long scan_err = 0;
    CK(cudaMemcpyAsync(&scan_err, c.scan_err.p, sizeof(scan_err), cudaMemcpyDeviceToHost, c.stream));
    CK(cudaStreamSynchronize(c.stream));
    if (scan_err) {
      CK(cudaMemsetAsync(c.scan_err.p, 0, sizeof(scan_err), c.stream));
      throw Fail(PMC_ERR_TIMEOUT);
    }
    if (!counted) {
      for (int k = 0; k < c.n_pop; k++) c.n_slots_host[k] += per_pop[0 * c.n_pop + k] + per_pop[2 * c.n_pop + k];
      redraws += losers + pp_lost;
      c.last_set_losers += losers;
      c.last_pp_lost += pp_lost;
      c.last_events += E;
      c.last_ops += Qr;
      round++;
    }
    counted = false;
    if (E == 0 && pp_lost == 0 && ppw == 0) break;
    if (round >= c.max_rounds) {
      std::vector<PopCtr>& r = read_ctrs(c);
      for (int k = 0; k < c.n_pop; k++)
        if (r[k].status == 0) r[k].status = PMC_ERR_TIMEOUT;
      write_ctrs(c);
      break;
    }
    // this round's target operations: the redone ones, and with per-particle
    // pairs in the step at most one more per item (a walk that stops there)
    const long long Qb = pp_lost + (c.pp_step ? E + ppw : 0);
    c.last_e0 = std::max(c.last_e0, E + ppw);
    c.last_qb = std::max(c.last_qb, Qb);
    // room for this round's new slots: at most one per item, and
    // kMaxCopies - 1 per target operation
    ensure_room(c, E + ppw + (kMaxCopies - 1) * Qb);
    // a round's items (events and walkers) each make at most one event
    if (!events_fit(c, E + ppw)) cap_throw("a round's events past the event arrays");
    if (!graph_tried && c.use_graph && !c.tuner.on && !c.pp_step && pp_lost == 0 && ppw == 0) {
      graph_tried = true;
      GraphRun g = run_round_graph(c, kt, flat, n_gpairs, E);
      if (g.rounds >= 0) {
        redraws += g.losers;
        c.last_set_losers += g.losers;
        c.last_events += g.events;
        round += (int)g.rounds;
        if (!g.stopped_for_room) break;
        // out of room inside the graph: the host loop grows the slot arrays
        // and carries on from the device's counts
        std::vector<PopCtr>& r = read_ctrs(c);
        for (int k = 0; k < c.n_pop; k++) c.n_slots_host[k] = r[k].n_slots;
        CK(cudaMemcpyAsync(&E, c.round_dev.p + 1, sizeof(long long), cudaMemcpyDeviceToHost, c.stream));
        CK(cudaStreamSynchronize(c.stream));
        if (round >= c.max_rounds) {
          for (int k = 0; k < c.n_pop; k++)
            if (r[k].status == 0) r[k].status = PMC_ERR_TIMEOUT;
          write_ctrs(c);
          break;
        }
        ensure_room(c, E);
      }
    }
    // one host-driven round
    reserve_round(c, E + ppw);
    // the operations that lost are staged for this round before their
    // buffers, which they are read from, may grow
    if (Qb > 0) reserve_redo(c, Qb);
    if (pp_lost > 0) launch_build_redo(c, last_qb, 0, c.stream);
    if (Qb > 0) reserve_ops(c, Qb);
    c.op_cap = Qb;
    // the walkers the last round's operations made are this round's to read
    grow_keeping(c, c.ppw_slot, (size_t)(kMaxCopies * (Qb + 1)));
    grow_keeping(c, c.ppw_gp, (size_t)(kMaxCopies * (Qb + 1)));
    // the round's sort covers the current slots exactly
    prepare_chunks(c);
    int mc = 1;
    for (int k = 0; k < c.n_pop; k++) mc = std::max(mc, c.pops[k].h.n_chunks);
    if (c.dirty) push_pops(c);
    RoundBounds b{kt, flat, n_gpairs, E + ppw, mc, max_cells_of(c)};
    k_round_begin<<<1, 128, 0, c.stream>>>(c.d_round, c.round_dev.p, c.per_pop_i.p, 4 * c.n_pop, c.n_dev.p);
    note_launch();
    c.claim_gen++;  // as k_round_begin on the device
    enqueue_round_head(c, c.stream, b, Qb);
    if (Qb > 0) fit_rm_pool(c);
    enqueue_round_tail(c, c.stream, b, Qb);
    last_qb = Qb;
  }
  c.last_redraws = redraws;
  c.last_rounds = round;
}

}  // namespace

// ---------------------------------------------------------------------------
// C ABI

struct pmc_coag_gpu_ctx {
  Ctx c;
};

extern "C" {

const char* pmc_coag_gpu_status_string(int s) {
  switch (s) {
    case PMC_OK: return "ok";
    case PMC_ERR_INVALID_ARG: return "invalid argument";
    case PMC_ERR_OUT_OF_GRID: return "particle outside of bin_grid: try reducing the timestep del_t";
    case PMC_ERR_CAPACITY: return g_last_capacity[0] ? g_last_capacity : "capacity exceeded";
    case PMC_ERR_CUDA: return g_last_error[0] ? g_last_error : "CUDA error";
    case PMC_ERR_TIMEOUT: return "bounded device loop ran out of iterations";
    case PMC_ERR_RNG_EXHAUSTED: return "replay stream exhausted";
    case PMC_ERR_ASSERT: return g_last_assert[0] ? g_last_assert : "reference assertion failed";
    case PMC_ERR_NO_DEVICE: return "no CUDA device";
  }
  return "unknown status";
}

#define GUARD_BEGIN try {
#define GUARD_END                 \
  }                               \
  catch (Fail & f) {              \
    return f.code;                \
  }                               \
  catch (...) {                   \
    return PMC_ERR_CAPACITY;      \
  }

static int do_init(int n_pop, int n_spec, const double* density, int i_water, int n_group, int n_class,
                   const int* w_type, const double* w_mag, const double* w_exp, const uint64_t* seeds,
                   pmc_coag_gpu_ctx** out) {
  if (!out || n_pop < 1 || n_spec < 1 || n_spec > kMaxSpec || n_group < 1 || n_group > kMaxGroup ||
      n_class < 1 || n_class > kMaxClass || !density || !w_type || !w_mag || !w_exp)
    return PMC_ERR_INVALID_ARG;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev < 1) return PMC_ERR_NO_DEVICE;
  std::unique_ptr<pmc_coag_gpu_ctx> x(new pmc_coag_gpu_ctx());
  Ctx& c = x->c;
  GUARD_BEGIN
  c.n_pop = n_pop;
  c.n_spec = n_spec;
  c.n_group = n_group;
  c.n_class = n_class;
  c.i_water = i_water;
  c.density.assign(density, density + n_spec);
  memset(&c.w, 0, sizeof(c.w));
  c.w.n_group = n_group;
  c.w.n_class = n_class;
  for (int cl = 0; cl < n_class; cl++)
    for (int g = 0; g < n_group; g++) {
      int src = g + n_group * cl;
      int dst = g + kMaxGroup * cl;
      if (w_type[src] < 1 || w_type[src] > 3) return PMC_ERR_INVALID_ARG;
      c.w.type[dst] = w_type[src];
      c.w.mag[dst] = w_mag[src];
      c.w.expo[dst] = w_exp[src];
    }
  CK(cudaStreamCreateWithFlags(&c.stream, cudaStreamNonBlocking));
  CK(cudaStreamCreateWithFlags(&c.cap_stream, cudaStreamNonBlocking));
  CK(cudaStreamCreateWithFlags(&c.side_stream, cudaStreamNonBlocking));
  CK(cudaEventCreateWithFlags(&c.ev_fork, cudaEventDisableTiming));
  CK(cudaEventCreateWithFlags(&c.ev_join, cudaEventDisableTiming));
  {
    int dev = 0;
    CK(cudaGetDevice(&dev));
    c.mem = pool_acquire(dev);
    c.mem_ref.dev = dev;
  }
  {
    int dev = 0, n_sm = 0, coop = 0;
    CK(cudaGetDevice(&dev));
    CK(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev));
    CK(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
    if (!coop) throw Fail(PMC_ERR_NO_DEVICE);  // the sort needs cooperative launches
    c.n_sm = n_sm;
  }
  c.pops.resize(n_pop);
  CK(cudaMalloc(&c.d_pops, sizeof(PopDev) * n_pop));
  CK(cudaMalloc(&c.d_stat, sizeof(long long) * kStatWords + sizeof(PopCtr) * n_pop + 16));  // read in 16-byte words
  c.d_ctrs = (PopCtr*)(c.d_stat + kStatWords);
  CK(cudaMalloc(&c.d_round, 2 * sizeof(uint32_t)));  // round of the step, claim generation
  // cleared in the order of the context's own stream, which does not wait for
  // the default one: a clear queued there behind the caller's work would come
  // after the first uploads
  CK(cudaMemsetAsync(c.d_round, 0, 2 * sizeof(uint32_t), c.stream));
  c.scan_ctr.reserve(2 * kScanMaxJobs);  // tile counters, then finished-block counters
  CK(cudaMemsetAsync(c.scan_ctr.p, 0, sizeof(unsigned) * c.scan_ctr.n, c.stream));
  c.scan_err.reserve(1);
  CK(cudaMemsetAsync(c.scan_err.p, 0, sizeof(unsigned long long) * c.scan_err.n, c.stream));
  CK(cudaMemsetAsync(c.d_ctrs, 0, sizeof(PopCtr) * n_pop, c.stream));
  for (int k = 0; k < n_pop; k++) {
    c.pops[k].seed = seeds ? seeds[k] : (uint64_t)(k + 1);
    init_pop(c, c.pops[k], 1024);
  }
  push_pops(c);
  CK(cudaStreamSynchronize(c.stream));
  *out = x.release();
  return PMC_OK;
  GUARD_END
}

int pmc_coag_gpu_init(int n_spec, const double* density, int i_water, int n_group, int n_class,
                      const int* w_type, const double* w_mag, const double* w_exp, uint64_t seed,
                      pmc_coag_gpu_ctx** ctx) {
  return do_init(1, n_spec, density, i_water, n_group, n_class, w_type, w_mag, w_exp, &seed, ctx);
}

int pmc_coag_gpu_init_batch(int n_pop, int n_spec, const double* density, int i_water, int n_group,
                            int n_class, const int* w_type, const double* w_mag, const double* w_exp,
                            const uint64_t* seeds, pmc_coag_gpu_ctx** ctx) {
  return do_init(n_pop, n_spec, density, i_water, n_group, n_class, w_type, w_mag, w_exp, seeds, ctx);
}

int pmc_coag_gpu_destroy(pmc_coag_gpu_ctx* x) {
  if (!x) return PMC_OK;
  Ctx& c = x->c;
  cudaStreamSynchronize(c.stream);
  for (auto& ph : c.pops) {
    free_list(c, ph.slot_allocs);
    free_list(c, ph.sort_allocs);
    free_list(c, ph.fixed_allocs);
    if (ph.h.rm_log) cudaFree(ph.h.rm_log);
  }
  cudaFree(c.d_pops);
  cudaFree(c.d_stat);
  cudaFree(c.d_round);
  DevBuf<int>* bi[] = {&c.gpair_pop, &c.gpair_local, &c.lost_pp, &c.op_pop, &c.op_pair, &c.op_slot, &c.op_k, &c.r_pop,
                       &c.r_pair, &c.r_slot, &c.r_k, &c.per_pop_i, &c.slot_base_set, &c.slot_base_pp,
                       &c.ev_dest, &c.ev_len, &c.ev_head, &c.ev_app, &c.it_gp, &c.it_len, &c.it_head, &c.it_start,
                       &c.ch_y, &c.ch_q};
  for (auto* b : bi) b->release();
  DevBuf<long long>* bl[] = {&c.pop_pair_base, &c.nwork_set, &c.nwork_pp, &c.work_off, &c.pp_off,
                             &c.rank_slot_set, &c.rank_id_set, &c.rank_slot_pp, &c.lost_off,
                             &c.id_base_set, &c.id_base_pp, &c.n_dev};
  for (auto* b : bl) b->release();
  DevBuf<unsigned long long>* bk[] = {&c.ev_key, &c.it_key, &c.op_key, &c.r_key};
  for (auto* b : bk) b->release();
  c.ev_pos.release();
  c.it_pos.release();
  c.it_dec.release();
  c.it_gused.release();
  c.it_term.release();
  c.ev_term.release();
  c.ch_pos.release();
  c.it_flag.release();
  c.it_done.release();
  c.ev_done.release();
  c.chain_list.release();
  c.it_c.release();
  c.flag.release();
  c.win_set.release();
  c.pop_on.release();
  c.report.release();
  c.report_seq.release();
  c.dec_set.release();
  c.ev_gp.release();
  c.gp_c.release();
  c.ev_c.release();
  c.scan_status.release();
  c.scan_ctr.release();
  c.scan_err.release();
  c.win_pp.release();
  c.ev.release();
  c.pp_res.release();
  c.pp_vol.release();
  c.replay_u.release();
  c.st_d.release();
  c.st_i.release();
  c.st_l.release();
  c.st_cnt.release();
  c.pin.release();
  c.map.release();
  for (auto& ev : c.sync_ev)
    if (ev) cudaEventDestroy(ev);
  replay_free(c.replay);
  free_redraw_graph(c);
  free_step_graph(c);
  for (auto& ev : c.sg_ev)
    if (ev) cudaEventDestroy(ev);
  c.graph_stats.release();
  c.sample_buf.release();
  for (auto* b : {&c.grp_hist, &c.item_pop, &c.ppw_slot, &c.ppw_gp}) b->release();
  c.grp_off.release();
  c.grp_dest.release();
  c.wk_slot.release();
  c.wk_gp.release();
  c.wk_flag.release();
  c.pp_rm_pool.release();
  c.pp_rm_off.release();
  c.pp_rm_tot.release();
  c.dup_n.release();
  c.select_buf.release();
  for (auto& pr : c.tuner.pending) {
    cudaEventDestroy(pr.first);
    cudaEventDestroy(pr.second);
  }
  for (auto e : c.tuner.spare) cudaEventDestroy(e);
  cudaStreamSynchronize(c.stream);  // the arrays are back in the pool
  cudaStreamDestroy(c.cap_stream);
  cudaStreamDestroy(c.side_stream);
  cudaEventDestroy(c.ev_fork);
  cudaEventDestroy(c.ev_join);
  cudaStreamDestroy(c.stream);
  delete x;
  return PMC_OK;
}

int pmc_coag_gpu_upload(pmc_coag_gpu_ctx* x, int pop, int n_part, const double* vol, const int* group,
                        const int* cls, const int64_t* id, const int* n_primary) {
  if (!x || pop < 0 || pop >= x->c.n_pop || n_part < 0 || (n_part > 0 && !vol)) return PMC_ERR_INVALID_ARG;
  Ctx& c = x->c;
  GUARD_BEGIN
  PopHost& ph = c.pops[pop];
  int cap = std::max(1024, n_part + n_part / 2 + 64);
  PopCtr r = read_ctr(c, pop);
  if (cap > ph.h.cap || cap < ph.h.cap / 4) {
    // the old arrays go first: there may not be room for both.  If the new ones
    // do not fit, the population is left empty, without slots
    free_list(c, ph.slot_allocs);
    PopDev h = ph.h;
    ph.h.cap = 0;
    try {
      alloc_slots(c, h, ph.slot_allocs, cap);
    } catch (...) {
      r.n_slots = r.n_live = 0;
      write_ctr(c, pop, r);
      ph.valid_sort = ph.caches_valid = c.replay.valid = false;
      ph.mirror_full = true;
      push_pops(c);
      throw;
    }
    ph.h = h;
  }
  CK(cudaMemsetAsync(ph.h.alive, 0, ph.h.cap, c.stream));
  CK(cudaMemsetAsync(ph.h.changed, 0, ph.h.cap, c.stream));
  ph.mirror_full = true;  // a host copy kept slot by slot must be refreshed in full
  if (n_part > 0) {
    size_t n = (size_t)n_part;
    CK(cudaMemcpyAsync(ph.h.vol, vol, sizeof(double) * n * c.n_spec, cudaMemcpyHostToDevice, c.stream));
    if (group) CK(cudaMemcpyAsync(ph.h.grp, group, sizeof(int) * n, cudaMemcpyHostToDevice, c.stream));
    if (cls) CK(cudaMemcpyAsync(ph.h.cls, cls, sizeof(int) * n, cudaMemcpyHostToDevice, c.stream));
    if (id) CK(cudaMemcpyAsync(ph.h.id, id, sizeof(long long) * n, cudaMemcpyHostToDevice, c.stream));
    if (n_primary) CK(cudaMemcpyAsync(ph.h.nprim, n_primary, sizeof(int) * n, cudaMemcpyHostToDevice, c.stream));
    long long id0 = r.next_id;
    c.st_l.reserve(2);
    CK(cudaMemsetAsync(c.st_l.p, 0, 2 * sizeof(long long), c.stream));
    int* bad = (int*)c.st_l.p;
    unsigned long long* max_id = (unsigned long long*)(c.st_l.p + 1);
    k_upload<<<grid_for(n_part, 256), 256, 0, c.stream>>>(ph.h, n_part, group != nullptr, cls != nullptr,
                                                          id != nullptr, n_primary != nullptr, id0, bad, max_id);
    note_launch();
    long long chk[2] = {0, 0};
    CK(cudaMemcpyAsync(chk, c.st_l.p, sizeof(chk), cudaMemcpyDeviceToHost, c.stream));
    CK(cudaStreamSynchronize(c.stream));
    if ((int)chk[0] != 0) {
      // invalid groups or classes: the population is left empty
      CK(cudaMemsetAsync(ph.h.alive, 0, ph.h.cap, c.stream));
      r.n_slots = r.n_live = 0;
      write_ctr(c, pop, r);
      ph.valid_sort = false;
      ph.caches_valid = false;
      c.replay.valid = false;
      return PMC_ERR_INVALID_ARG;
    }
    if (id) r.next_id = std::max<long long>(r.next_id, chk[1] + 1);
    else r.next_id = id0 + n_part;
  }
  r.n_slots = n_part;
  r.n_live = n_part;
  write_ctr(c, pop, r);
  ph.valid_sort = false;
  ph.caches_valid = false;
  c.replay.valid = false;
  no_grid(c, ph);
  push_pops(c);
  CK(cudaStreamSynchronize(c.stream));
  return PMC_OK;
  GUARD_END
}

int pmc_coag_gpu_upload_components(pmc_coag_gpu_ctx* x, int pop, int n_part, const int* n_comp,
                                   const int* comp_source, const double* comp_create_time) {
  if (!x || pop < 0 || pop >= x->c.n_pop || !n_comp || !comp_source || !comp_create_time)
    return PMC_ERR_INVALID_ARG;
  Ctx& c = x->c;
  GUARD_BEGIN
  PopHost& ph = c.pops[pop];
  PopCtr r = read_ctr(c, pop);
  if (n_part != r.n_slots) return PMC_ERR_INVALID_ARG;
  // the slot arrays hold components particle-major, as the caller passes them
  std::vector<double> lct(n_part), gct(n_part);
  for (int i = 0; i < n_part; i++) {
    if (n_comp[i] < 0 || n_comp[i] > kMaxComponent) return PMC_ERR_INVALID_ARG;
    double lo = 0.0, hi = 0.0;
    for (int k = 0; k < n_comp[i]; k++) {
      double t = comp_create_time[comp_at(i, k)];
      if (k == 0 || t < lo) lo = t;
      if (k == 0 || t > hi) hi = t;
    }
    lct[i] = lo;
    gct[i] = hi;
  }
  size_t nc = (size_t)n_part * kMaxComponent;
  CK(cudaMemcpyAsync(ph.h.ncomp, n_comp, sizeof(int) * n_part, cudaMemcpyHostToDevice, c.stream));
  CK(cudaMemcpyAsync(ph.h.csrc, comp_source, sizeof(int) * nc, cudaMemcpyHostToDevice, c.stream));
  CK(cudaMemcpyAsync(ph.h.ctime, comp_create_time, sizeof(double) * nc, cudaMemcpyHostToDevice, c.stream));
  CK(cudaMemcpyAsync(ph.h.lct, lct.data(), sizeof(double) * n_part, cudaMemcpyHostToDevice, c.stream));
  CK(cudaMemcpyAsync(ph.h.gct, gct.data(), sizeof(double) * n_part, cudaMemcpyHostToDevice, c.stream));
  CK(cudaStreamSynchronize(c.stream));
  return PMC_OK;
  GUARD_END
}

// Removal logs that record: room for the records kept so far plus the most
// one step or rebalance can add (each removal frees a slot, and a step ends
// with at most cap slots; twice that allows for slot growth within the
// step).  Grows a log by copying its records into a larger buffer.
void reserve_removal_logs(Ctx& c) {
  for (auto& ph : c.pops) {
    if (!ph.h.rm_on) continue;
    long long need = ph.rm_count + 2LL * ph.h.cap + 1024;
    if (ph.h.rm_cap >= need) continue;
    long long cap = std::max(need, ph.h.rm_cap + ph.h.rm_cap / 2);
    RemovalRec* p = nullptr;
    if (cudaMalloc(&p, sizeof(RemovalRec) * (size_t)cap) != cudaSuccess) {
      cudaGetLastError();
      throw Fail(PMC_ERR_CAPACITY);
    }
    if (ph.h.rm_log) {
      long long keep = std::min(ph.rm_count, ph.h.rm_cap);
      if (keep > 0)
        CK(cudaMemcpyAsync(p, ph.h.rm_log, sizeof(RemovalRec) * (size_t)keep, cudaMemcpyDeviceToDevice, c.stream));
      CK(cudaStreamSynchronize(c.stream));
      cudaFree(ph.h.rm_log);
    }
    ph.h.rm_log = p;
    ph.h.rm_cap = cap;
    c.dirty = true;
  }
}

static int finish_step(Ctx& c, long long* samp, long long* coag) {
  long long s = 0, k = 0, warn = 0, exact = 0;
  int status = 0;
  // one read-back (a stream sync) for every population; a compaction below
  // changes only its own population's counters
  const std::vector<PopCtr> all = c.ctrs_fresh ? c.h_ctrs : read_ctrs(c);
  c.n_slots_host.resize(c.n_pop);
  for (int p = 0; p < c.n_pop; p++) c.n_slots_host[p] = all[p].n_slots;
  c.ctrs_fresh = true;  // until a call below or a later one writes them
  for (int p = 0; p < c.n_pop; p++) {
    const PopCtr& r = all[p];
    s += r.tot_samp;
    k += r.tot_coag;
    warn += r.kmax_warn;
    exact += r.exact_tests;
    c.pops[p].rm_count = r.n_removed;
    if (c.pops[p].h.rm_on && r.n_removed > c.pops[p].h.rm_cap) {
      snprintf(g_last_assert, sizeof(g_last_assert), "removal log of population %d overflowed", p);
      if (!status) status = PMC_ERR_CAPACITY;
    }
    if (r.status && !status) status = r.status;
    if (r.status == kErrCapacity && r.cap_site) {
      static const char* site[] = {"", "an event's new particle past the slot arrays",
                                   "the round's target-operation list is full",
                                   "a target operation's removals past its share of the pool",
                                   "more dup copies than one target operation holds",
                                   "a target operation's copy past the slot arrays",
                                   "the walker list of target operations is full",
                                   "a sampled particle past the slot arrays",
                                   "a doubled or dup copy past the slot arrays"};
      snprintf(g_last_capacity, sizeof(g_last_capacity), "capacity exceeded: %s (population %d)",
               r.cap_site < 9 ? site[r.cap_site] : "?", p);
    }
    if (r.bad_site) {
      static const char* site[] = {"", "pair test: list position", "pair test: slot", "event: slot",
                                   "sort scatter: list position", "sort: chunk histogram size",
                                   "pair set-up: cell range", "slot count above capacity",
                                   "event: destination slot"};
      snprintf(g_last_assert, sizeof(g_last_assert),
               "device bounds check failed (%s, population %d, index %lld)",
               r.bad_site < 9 ? site[r.bad_site] : "?", p, r.bad_index);
      status = PMC_ERR_ASSERT;
      continue;  // no compaction of a population in this state
    }
    // compact when more than half of the used slots are dead
    if (r.n_slots > 4096 && r.n_live < r.n_slots / 2) relayout(c, p, c.pops[p].h.cap, true);
  }
  c.last_kmax_warn = warn;
  c.exact_tests = exact;
  *samp = s;
  *coag = k;
  return status;
}

// After a step that an error ended: the host does not know how far the device
// came, so the next step reads the counters, copies the populations to the
// device, and restarts the claim generations (a word of a round that the host
// did not count would win against the next step's).
static void step_left(Ctx& c) {
  c.ctrs_fresh = false;
  c.dirty = true;
  c.claim_gen = kGenLimit;
}

// the autotuner around one step: the candidate's shape before it; after it
// (finish_step has synchronised the stream) the device time of the site's
// launches and the step's pair tests
static void tune_before(Ctx& c) {
  Tuner& t = c.tuner;
  c.tune.threads[t.site] = kTuneCand[t.site][t.cand];
}

static void tune_after(Ctx& c, long long tests) {
  Tuner& t = c.tuner;
  for (auto& pr : t.pending) {
    float ms = 0.f;
    CK(cudaEventElapsedTime(&ms, pr.first, pr.second));
    t.cand_ms += ms;
    t.spare.push_back(pr.first);
    t.spare.push_back(pr.second);
  }
  t.pending.clear();
  t.cand_tests += tests;
  if (++t.rep < kTuneReps) return;
  const float score = (float)(t.cand_ms / (double)std::max(t.cand_tests, 1LL) * 1e6);
  t.site_ms[t.site][t.cand] = score;
  if (t.cand == 0 || score < t.best_ms) {
    t.best_ms = score;
    t.best = t.cand;
  }
  t.rep = 0;
  t.cand_ms = 0.0;
  t.cand_tests = 0;
  if (++t.cand < kTuneCands) return;
  c.tune.threads[t.site] = kTuneCand[t.site][t.best];
  t.cand = 0;
  if (++t.site < kTuneSites) return;
  t.on = false;
}

int pmc_coag_gpu_autotune(pmc_coag_gpu_ctx* x, int enable) {
  if (!x) return PMC_ERR_INVALID_ARG;
  Tuner& t = x->c.tuner;
  t.on = enable != 0;
  t.site = t.cand = t.rep = t.best = 0;
  t.best_ms = 0.f;
  t.cand_ms = 0.0;
  t.cand_tests = 0;
  for (auto& pr : t.pending) {
    t.spare.push_back(pr.first);
    t.spare.push_back(pr.second);
  }
  t.pending.clear();
  return PMC_OK;
}

int pmc_coag_gpu_tune_state(pmc_coag_gpu_ctx* x, int* tuning, int* threads, float* ms) {
  if (!x) return PMC_ERR_INVALID_ARG;
  const Ctx& c = x->c;
  if (tuning) *tuning = c.tuner.on ? 1 : 0;
  if (threads)
    for (int k = 0; k < kTuneSites; k++) threads[k] = c.tune.threads[k];
  if (ms)
    for (int k = 0; k < kTuneSites; k++)
      for (int j = 0; j < kTuneCands; j++) ms[k * kTuneCands + j] = c.tuner.site_ms[k][j];
  return PMC_OK;
}

int pmc_coag_gpu_set_tune(pmc_coag_gpu_ctx* x, const int* threads) {
  if (!x || !threads) return PMC_ERR_INVALID_ARG;
  for (int k = 0; k < kTuneSites; k++) {
    bool ok = false;
    for (int j = 0; j < kTuneCands; j++) ok = ok || threads[k] == kTuneCand[k][j];
    if (!ok) return PMC_ERR_INVALID_ARG;
  }
  for (int k = 0; k < kTuneSites; k++) x->c.tune.threads[k] = threads[k];
  x->c.tuner.on = false;
  return PMC_OK;
}

int pmc_coag_gpu_step_batch(pmc_coag_gpu_ctx* x, int kernel_type, const double* temp,
                            const double* pressure, double additive_coeff, double del_t, int n_steps,
                            int64_t* tot_n_samp, int64_t* tot_n_coag) {
  if (!x || kernel_type < 1 || kernel_type > 7 || !temp || !pressure || n_steps < 0)
    return PMC_ERR_INVALID_ARG;
  Ctx& c = x->c;
  GUARD_BEGIN
  long long S = 0, K = 0;
  for (int st = 0; st < n_steps; st++) {
    bool params_same = true;
    for (int k = 0; k < c.n_pop; k++) {
      PopHost& ph = c.pops[k];
      params_same = params_same && ph.h.kernel_type == kernel_type && ph.h.temp == temp[k] &&
                    ph.h.pressure == pressure[k] && ph.h.coeff == additive_coeff && ph.h.del_t == del_t;
      ph.h.kernel_type = kernel_type;
      ph.h.temp = temp[k];
      ph.h.pressure = pressure[k];
      ph.h.coeff = additive_coeff;
      ph.h.del_t = del_t;
      ph.h.benv = brown_env(temp[k], pressure[k], c.frac);
      ph.h.step = ++ph.step;
      // the reference keeps its bounds until the grid changes
      // (coag_kernel_bounds_valid, aero_sorted.F90:55); a new kernel type
      // would make them meaningless, so that case recomputes them
      if (ph.kmax_kt != kernel_type) {
        ph.h.kmax_valid = 0;
        ph.kmax_kt = kernel_type;
      }
    }
    reserve_removal_logs(c);
    long long s = 0, k = 0;
    int status;
    if (c.mode == PMC_MODE_REPLAY) {
      push_pops(c);
      c.ctrs_fresh = false;
      status = replay_step_host(c, &s, &k);
    } else {
      ProfScope ps(c, 3, 1);
      c.replay.valid = false;  // the parallel step reorders and rewrites slots
      if (c.tuner.on) tune_before(c);
      try {
        step_parallel(c, kernel_type, params_same);
        status = finish_step(c, &s, &k);
      } catch (...) {
        step_left(c);
        throw;
      }
      if (c.tuner.on && status == 0) tune_after(c, s);
    }
    S += s;
    K += k;
    if (status) {
      if (tot_n_samp) *tot_n_samp = S;
      if (tot_n_coag) *tot_n_coag = K;
      return status;
    }
  }
  if (tot_n_samp) *tot_n_samp = S;
  if (tot_n_coag) *tot_n_coag = K;
  return PMC_OK;
  GUARD_END
}

int pmc_coag_gpu_step(pmc_coag_gpu_ctx* x, int kernel_type, double temp, double pressure,
                      double additive_coeff, double del_t, int* tot_n_samp, int* tot_n_coag) {
  if (!x) return PMC_ERR_INVALID_ARG;
  std::vector<double> t(x->c.n_pop, temp), p(x->c.n_pop, pressure);
  int64_t s = 0, k = 0;
  int rc = pmc_coag_gpu_step_batch(x, kernel_type, t.data(), p.data(), additive_coeff, del_t, 1, &s, &k);
  if (tot_n_samp) *tot_n_samp = (int)s;
  if (tot_n_coag) *tot_n_coag = (int)k;
  return rc;
}

int pmc_coag_gpu_n_part(pmc_coag_gpu_ctx* x, int pop, int* n_part) {
  if (!x || pop < 0 || pop >= x->c.n_pop || !n_part) return PMC_ERR_INVALID_ARG;
  GUARD_BEGIN
  PopCtr r = read_ctr(x->c, pop);
  *n_part = r.n_live;
  return PMC_OK;
  GUARD_END
}

static int do_download(Ctx& c, int pop, int max_part, double* vol, int* group, int* cls, int64_t* id,
                       int* n_primary, int* n_comp, int* comp_source, double* comp_time, int* n_part) {
  PopHost& ph = c.pops[pop];
  PopCtr r = read_ctr(c, pop);
  if (n_part) *n_part = r.n_live;
  if (r.n_live > max_part) return PMC_ERR_CAPACITY;
  size_t ns = (size_t)r.n_slots + 1;
  size_t n = std::max(r.n_live, 1);
  c.st_l.reserve(ns + n);
  long long* off = c.st_l.p;
  long long nl = scan(c, ph.h.alive, r.n_slots, off, true);
  if (nl != r.n_live) return PMC_ERR_ASSERT;
  if (nl > 0 && nl == r.n_slots && !comp_source && !comp_time) {
    // no dead slots: the slot arrays already hold the particles in order,
    // in the caller's particle-major layout
    if (vol) CK(cudaMemcpyAsync(vol, ph.h.vol, sizeof(double) * nl * c.n_spec, cudaMemcpyDeviceToHost, c.stream));
    if (group) CK(cudaMemcpyAsync(group, ph.h.grp, sizeof(int) * nl, cudaMemcpyDeviceToHost, c.stream));
    if (cls) CK(cudaMemcpyAsync(cls, ph.h.cls, sizeof(int) * nl, cudaMemcpyDeviceToHost, c.stream));
    if (id) CK(cudaMemcpyAsync(id, ph.h.id, sizeof(long long) * nl, cudaMemcpyDeviceToHost, c.stream));
    if (n_primary) CK(cudaMemcpyAsync(n_primary, ph.h.nprim, sizeof(int) * nl, cudaMemcpyDeviceToHost, c.stream));
    if (n_comp) CK(cudaMemcpyAsync(n_comp, ph.h.ncomp, sizeof(int) * nl, cudaMemcpyDeviceToHost, c.stream));
    CK(cudaStreamSynchronize(c.stream));
    return PMC_OK;
  }
  c.st_d.reserve(n * (c.n_spec + kMaxComponent));
  c.st_i.reserve(n * (4 + kMaxComponent));
  long long* di = c.st_l.p + ns;
  double* dv = c.st_d.p;
  double* dct = c.st_d.p + n * c.n_spec;
  int* dg = c.st_i.p;
  int* dc = dg + n;
  int* dn = dc + n;
  int* dnc = dn + n;
  int* dcs = dnc + n;
  if (r.n_slots > 0)
    k_download<<<grid_for(r.n_slots, 256), 256, 0, c.stream>>>(
        ph.h, off, r.n_slots, vol ? dv : nullptr, group ? dg : nullptr, cls ? dc : nullptr, id ? di : nullptr,
        n_primary ? dn : nullptr, n_comp ? dnc : nullptr, comp_source ? dcs : nullptr,
        comp_time ? dct : nullptr);
  note_launch();
  if (nl > 0) {
    if (vol) CK(cudaMemcpyAsync(vol, dv, sizeof(double) * nl * c.n_spec, cudaMemcpyDeviceToHost, c.stream));
    if (group) CK(cudaMemcpyAsync(group, dg, sizeof(int) * nl, cudaMemcpyDeviceToHost, c.stream));
    if (cls) CK(cudaMemcpyAsync(cls, dc, sizeof(int) * nl, cudaMemcpyDeviceToHost, c.stream));
    if (id) CK(cudaMemcpyAsync(id, di, sizeof(long long) * nl, cudaMemcpyDeviceToHost, c.stream));
    if (n_primary) CK(cudaMemcpyAsync(n_primary, dn, sizeof(int) * nl, cudaMemcpyDeviceToHost, c.stream));
    if (n_comp) CK(cudaMemcpyAsync(n_comp, dnc, sizeof(int) * nl, cudaMemcpyDeviceToHost, c.stream));
    if (comp_source) CK(cudaMemcpyAsync(comp_source, dcs, sizeof(int) * nl * kMaxComponent, cudaMemcpyDeviceToHost, c.stream));
    if (comp_time) CK(cudaMemcpyAsync(comp_time, dct, sizeof(double) * nl * kMaxComponent, cudaMemcpyDeviceToHost, c.stream));
  }
  CK(cudaStreamSynchronize(c.stream));
  return PMC_OK;
}

// particles of population k per (group, class)
static std::vector<int> count_group_class(Ctx& c, int k) {
  PopHost& ph = c.pops[k];
  int ngc = c.n_group * c.n_class;
  c.st_i.reserve(ngc);
  CK(cudaMemsetAsync(c.st_i.p, 0, sizeof(int) * ngc, c.stream));
  PopCtr r = read_ctr(c, k);
  if (r.n_slots > 0) {
    k_count_group_class<<<grid_for(r.n_slots, 256), 256, 0, c.stream>>>(ph.h, c.st_i.p);
    note_launch();
  }
  std::vector<int> n(ngc);
  CK(cudaMemcpyAsync(n.data(), c.st_i.p, sizeof(int) * ngc, cudaMemcpyDeviceToHost, c.stream));
  CK(cudaStreamSynchronize(c.stream));
  return n;
}

// scale the weight magnitude of (g, c) of population k (aero_weight_scale);
// the population takes weights of its own
static void scale_weight(Ctx& c, int k, int g, int cl, double f) {
  PopHost& ph = c.pops[k];
  if (!ph.own_w) {
    ph.w = c.w;
    ph.own_w = true;
  }
  ph.w.mag[(g - 1) + kMaxGroup * (cl - 1)] *= f;
  ph.wver++;
  set_params(c, ph);
}

int pmc_coag_gpu_rebalance(pmc_coag_gpu_ctx* x, int pop, const double* n_part_ideal, int allow_doubling,
                           int allow_halving) {
  if (!x || pop < 0 || pop >= x->c.n_pop || !n_part_ideal) return PMC_ERR_INVALID_ARG;
  Ctx& c = x->c;
  GUARD_BEGIN
  PopHost& ph = c.pops[pop];
  bool changed = false;
  if (allow_doubling)
    for (int g = 1; g <= c.n_group; g++)
      for (int cl = 1; cl <= c.n_class; cl++) {
        int idx = (g - 1) + c.n_group * (cl - 1);
        double ideal = n_part_ideal[idx];
        for (int it = 0; it < 64; it++) {
          int cnt = count_group_class(c, pop)[idx];
          if (!((double)cnt < ideal / 2.0 && cnt > 0)) break;
          PopCtr r = read_ctr(c, pop);
          long long need = (long long)r.n_slots + cnt;
          if (need > ph.h.cap)
            relayout(c, pop, (int)std::min<long long>(need * 3 / 2 + 1024, (1LL << 31) - 1), false);
          r = read_ctr(c, pop);
          size_t n = (size_t)r.n_slots;
          c.st_l.reserve(n + 1);
          c.flag.reserve(n + 1);
          if (c.dirty) push_pops(c);
          k_flag_group_class<<<grid_for(n, 256), 256, 0, c.stream>>>(ph.h, r.n_slots, g, cl, c.flag.p);
          note_launch();
          long long members = scan(c, c.flag.p, (long long)n, c.st_l.p, true);
          k_double<<<grid_for(n, 256), 256, 0, c.stream>>>(ph.h, r.n_slots, c.flag.p, c.st_l.p, r.next_id);
          note_launch();
          r.n_slots += (int)members;
          r.n_live += (int)members;
          r.next_id += members;
          write_ctr(c, pop, r);
          scale_weight(c, pop, g, cl, 0.5);
          changed = true;
        }
      }
  if (allow_halving) reserve_removal_logs(c);  // halving records its removals
  if (allow_halving)
    for (int g = 1; g <= c.n_group; g++)
      for (int cl = 1; cl <= c.n_class; cl++) {
        int idx = (g - 1) + c.n_group * (cl - 1);
        double ideal = n_part_ideal[idx];
        for (int it = 0; it < 64; it++) {
          int cnt = count_group_class(c, pop)[idx];
          if (!((double)cnt > ideal * 2.0)) break;
          push_pops(c);
          PopCtr r = read_ctr(c, pop);
          k_halve<<<grid_for(r.n_slots, 256), 256, 0, c.stream>>>(ph.h, g, cl, ph.rebalance_calls++);
          note_launch();
          scale_weight(c, pop, g, cl, 2.0);
          changed = true;
        }
      }
  if (changed) {
    ph.valid_sort = false;  // aero_state_double clears valid_sort; halving removed particles
    c.replay.valid = false;
    push_pops(c);
    CK(cudaStreamSynchronize(c.stream));
    PopCtr r = read_ctr(c, pop);
    ph.rm_count = r.n_removed;
    if (r.status) return r.status;
    if (ph.h.rm_on && r.n_removed > ph.h.rm_cap) return PMC_ERR_CAPACITY;
  }
  return PMC_OK;
  GUARD_END
}

// ---------------------------------------------------------------------------
// aero_state_add_aero_dist_sample (aero_state.F90:758-831) on the device

// One mode of the caller's distribution (aero_mode_t, aero_mode.F90:40-66)
struct HostMode {
  int type = 0;
  double char_radius = 0, log10_std = 0, num_conc = 0;
  int source = 1;
  int n_sample = 0;
  const double* sample_radius = nullptr;  // [n_sample + 1] (host)
  const double* sample_nc = nullptr;      // [n_sample] (host)
  long long r_off = 0;                    // offset of sample_radius in the device copy
};

// aero_mode_weighted_sampled_num_conc (aero_mode.F90:457-491).  Under a
// power weight of exponent 0 the reference's expression is 0/0; its limit,
// the unweighted concentration, is used.
static void weighted_sampled_num_conc(const HostMode& m, int w_type, double expo, std::vector<double>& out) {
  out.resize(m.n_sample);
  for (int i = 0; i < m.n_sample; i++) {
    if (w_type == kWeightNone || expo == 0.0) {
      out[i] = m.sample_nc[i];
      continue;
    }
    double x0 = log(m.sample_radius[i]), x1 = log(m.sample_radius[i + 1]);
    out[i] = m.sample_nc[i] / expo * (exp(-expo * x0) - exp(-expo * x1)) / (x1 - x0);
  }
}

// log10 of the weighted mode's median radius, x_mean_prime
// (aero_mode.F90:510-513, :574-577)
static double x_mean_prime(const HostMode& m, int w_type, double expo) {
  double x = log10(m.char_radius);
  if (w_type == kWeightNone) return x;
  return x - expo * (m.log10_std * m.log10_std) * log(10.0);
}

// aero_mode_number (aero_mode.F90:495-546): the mean number of computational
// particles per unit sample proportion under weight (w_type, mag, expo);
// wnc receives a sampled mode's weighted interval concentrations
static double mode_number(const HostMode& m, int w_type, double mag, double expo, std::vector<double>& wnc) {
  switch (m.type) {
    case kModeLogNormal: {
      if (w_type == kWeightNone) return m.num_conc / mag;
      double x = log10(m.char_radius), xp = x_mean_prime(m, w_type, expo);
      return m.num_conc / mag * exp((xp * xp - x * x) / (2.0 * (m.log10_std * m.log10_std)));
    }
    case kModeExp:
      if (w_type != kWeightNone) throw Fail(PMC_ERR_INVALID_ARG);  // die_msg(822252601)
      return m.num_conc / mag;
    case kModeMono:
      return m.num_conc / (w_type == kWeightNone ? mag : mag * fast_pow<double>(m.char_radius, expo));
    case kModeSampled: {
      weighted_sampled_num_conc(m, w_type, expo, wnc);
      double s = 0.0;
      for (double v : wnc) s = s + v;
      return s / mag;
    }
  }
  throw Fail(PMC_ERR_INVALID_ARG);
}

// aero_state_scale_weight (aero_state.F90:1859-1922) for (g, cl) of
// population k holding n members: returns the members after the call
static long long scale_weight_members(Ctx& c, int k, int g, int cl, long long n, double ratio, bool allow_doubling,
                                      bool allow_halving, Rng& hr, uint32_t call) {
  PopHost& ph = c.pops[k];
  if (ratio > 1.0 && (allow_halving || n == 0)) {
    scale_weight(c, k, g, cl, ratio);
    long long n_remove = prob_round(hr, (double)n * (1.0 - 1.0 / ratio));
    if (n_remove <= 0) return n;
    reserve_removal_logs(c);  // the removals are recorded (AERO_INFO_HALVED)
    if (c.dirty) push_pops(c);
    c.select_buf.reserve(sizeof(SelectState));
    SelectState* S = (SelectState*)c.select_buf.p;
    CK(cudaMemsetAsync(S, 0, sizeof(SelectState), c.stream));
    CK(cudaMemcpyAsync(&S->need, &n_remove, sizeof(long long), cudaMemcpyHostToDevice, c.stream));
    PopCtr r = read_ctr(c, k);
    int grid = grid_for(r.n_slots, 256);
    for (int shift = 48; shift >= 0; shift -= 16) {
      k_select_hist<<<grid, 256, 0, c.stream>>>(ph.h, g, cl, call, S, shift);
      note_launch();
      k_select_pick<<<1, 1024, 0, c.stream>>>(S, shift);
      note_launch();
    }
    k_select_remove<<<grid, 256, 0, c.stream>>>(ph.h, g, cl, call, S);
    note_launch();
    // the records kept so far, for a later growth of the log
    ph.rm_count = read_ctr(c, k).n_removed;
    return n - n_remove;
  }
  if (ratio < 1.0 && (allow_doubling || n == 0)) {
    scale_weight(c, k, g, cl, ratio);
    if (n == 0) return 0;
    if (c.dirty) push_pops(c);
    PopCtr r = read_ctr(c, k);
    size_t ns = (size_t)r.n_slots;
    c.dup_n.reserve(ns + 1);
    c.st_l.reserve(ns + 1);
    k_dup_count<<<grid_for(ns, 256), 256, 0, c.stream>>>(ph.h, r.n_slots, g, cl, 1.0 / ratio, call, c.dup_n.p);
    note_launch();
    long long copies = scan(c, c.dup_n.p, (long long)ns, c.st_l.p, true);
    if (copies > 0) {
      long long need = (long long)r.n_slots + copies;
      if (need > (1LL << 31) - 1) throw Fail(PMC_ERR_CAPACITY);
      if (need > ph.h.cap) {
        relayout(c, k, (int)std::min<long long>(need * 3 / 2 + 1024, (1LL << 31) - 1), false);
        push_pops(c);
      }
      k_dup_write<<<grid_for(ns, 256), 256, 0, c.stream>>>(ph.h, r.n_slots, c.dup_n.p, c.st_l.p, r.next_id);
      note_launch();
      r.n_slots += (int)copies;
      r.n_live += (int)copies;
      r.next_id += copies;
      write_ctr(c, k, r);
    }
    return n + copies;
  }
  return n;
}

int pmc_coag_gpu_add_dist_sample(pmc_coag_gpu_ctx* x, int pop, int n_mode, const int* mode_type,
                                 const double* char_radius, const double* log10_std, const double* num_conc,
                                 const double* vol_frac, const double* vol_frac_std, const int* source,
                                 const int* n_sample, const double* sample_radius, const double* sample_num_conc,
                                 double sample_prop, double characteristic_factor, double create_time,
                                 const double* n_part_ideal, int allow_doubling, int allow_halving,
                                 int64_t* n_part_add) {
  if (n_part_add) *n_part_add = 0;
  if (!x || pop < 0 || pop >= x->c.n_pop || n_mode < 0) return PMC_ERR_INVALID_ARG;
  if (n_mode > 0 && (!mode_type || !char_radius || !num_conc || !vol_frac)) return PMC_ERR_INVALID_ARG;
  if (!(sample_prop >= 0.0) || !(characteristic_factor > 0.0)) return PMC_ERR_INVALID_ARG;
  Ctx& c = x->c;
  // the modes, checked as aero_mode_read and the samplers check them
  std::vector<HostMode> modes(n_mode);
  long long r_tot = 0, nc_tot = 0;
  for (int m = 0; m < n_mode; m++) {
    HostMode& h = modes[m];
    h.type = mode_type[m];
    h.char_radius = char_radius[m];
    h.log10_std = log10_std ? log10_std[m] : 0.0;
    h.num_conc = num_conc[m];
    h.source = source ? source[m] : m + 1;
    if (h.type < kModeLogNormal || h.type > kModeSampled || !(h.num_conc >= 0.0) || h.source < 1)
      return PMC_ERR_INVALID_ARG;
    if (c.n_class > 1 && h.source > c.n_class) return PMC_ERR_INVALID_ARG;  // assert(765048788)
    if (h.type == kModeLogNormal && (!log10_std || !(h.log10_std > 0.0) || !(h.char_radius > 0.0)))
      return PMC_ERR_INVALID_ARG;
    if ((h.type == kModeExp || h.type == kModeMono) && !(h.char_radius > 0.0)) return PMC_ERR_INVALID_ARG;
    if (h.type == kModeSampled) {
      if (!n_sample || !sample_radius || !sample_num_conc || n_sample[m] < 1) return PMC_ERR_INVALID_ARG;
      h.n_sample = n_sample[m];
      h.sample_radius = sample_radius + r_tot;
      h.sample_nc = sample_num_conc + nc_tot;
      h.r_off = r_tot;
      for (int i = 0; i <= h.n_sample; i++)
        if (!(h.sample_radius[i] > 0.0) || (i > 0 && !(h.sample_radius[i] > h.sample_radius[i - 1])))
          return PMC_ERR_INVALID_ARG;
      for (int i = 0; i < h.n_sample; i++)
        if (!(h.sample_nc[i] >= 0.0)) return PMC_ERR_INVALID_ARG;
      r_tot += h.n_sample + 1;
      nc_tot += h.n_sample;
    }
    for (int s = 0; s < c.n_spec; s++) {
      double f = vol_frac[m * c.n_spec + s], sd = vol_frac_std ? vol_frac_std[m * c.n_spec + s] : 0.0;
      if (!(f >= 0.0) || !(sd >= 0.0)) return PMC_ERR_INVALID_ARG;
    }
  }
  GUARD_BEGIN
  PopHost& ph = c.pops[pop];
  const uint32_t call = ph.sample_calls++;
  Rng hr(ph.seed, ph.step, sample_ctr(call, kSubHost), 0u);
  // device copies: fractions and their deviations per mode, the sampled
  // modes' radius edges, one weighted-concentration array per batch
  const int ns = c.n_spec;
  size_t n_vf = (size_t)n_mode * ns;
  std::vector<double> hbuf(2 * n_vf + (size_t)r_tot + (size_t)nc_tot * c.n_group + 1, 0.0);
  for (size_t i = 0; i < n_vf; i++) {
    hbuf[i] = vol_frac[i];
    hbuf[n_vf + i] = vol_frac_std ? vol_frac_std[i] : 0.0;
  }
  if (r_tot) std::memcpy(&hbuf[2 * n_vf], sample_radius, sizeof(double) * (size_t)r_tot);
  c.sample_buf.reserve(hbuf.size());
  double* d_vf = c.sample_buf.p;
  double* d_sr = d_vf + 2 * n_vf;
  double* d_wnc = d_sr + r_tot;
  std::vector<int> cnt = count_group_class(c, pop);
  {
    // room for the whole call at once: the batches' expected counts, with
    // the weight preparation run on expected values, plus a margin of 8
    // standard deviations (a larger draw grows the slots below)
    Weights w = ph.own_w ? ph.w : c.w;
    std::vector<double> est(cnt.begin(), cnt.end());
    double slots = 0.0, var = 0.0;
    std::vector<double> tmp;
    for (int g = 1; g <= c.n_group; g++)
      for (int m = 0; m < n_mode; m++) {
        int cl = c.n_class > 1 ? modes[m].source : 1;
        int kc = (g - 1) + c.n_group * (cl - 1), kw = (g - 1) + kMaxGroup * (cl - 1);
        double n_avg = sample_prop * mode_number(modes[m], w.type[kw], w.mag[kw], w.expo[kw], tmp);
        if (n_part_ideal) {
          double n_new = est[kc] + n_avg, ideal = n_part_ideal[kc];
          if (n_new != 0.0 && (n_new < ideal / 2.0 || n_new > ideal * 2.0)) {
            double ratio = n_new / ideal;
            bool halve = ratio > 1.0 && (allow_halving || est[kc] == 0.0);
            bool dbl = ratio < 1.0 && (allow_doubling || est[kc] == 0.0);
            if (halve || dbl) {
              if (dbl) slots += est[kc] * (1.0 / ratio - 1.0);
              est[kc] /= ratio;
              w.mag[kw] *= ratio;
            }
          }
        }
        if (n_avg == 0.0) continue;
        n_avg = sample_prop * mode_number(modes[m], w.type[kw], w.mag[kw], w.expo[kw], tmp);
        est[kc] += n_avg;
        slots += n_avg;
        var += n_avg;
      }
    PopCtr r = read_ctr(c, pop);
    double need = (double)r.n_slots + slots + 8.0 * std::sqrt(var) + 1024.0;
    if (need > (double)ph.h.cap && need < (double)((1LL << 31) - 1)) relayout(c, pop, (int)need, false);
  }
  long long wnc_used = 0, added = 0;
  uint32_t idx = 0;
  std::vector<double> wnc;
  for (int g = 1; g <= c.n_group; g++)
    for (int m = 0; m < n_mode; m++) {
      const HostMode& h = modes[m];
      int cl = c.n_class > 1 ? h.source : 1;  // aero_state_weight_class_for_source, aero_state.F90:263-282
      int kc = (g - 1) + c.n_group * (cl - 1);
      int kw = (g - 1) + kMaxGroup * (cl - 1);
      const Weights& W0 = ph.own_w ? ph.w : c.w;
      double n_avg = sample_prop * mode_number(h, W0.type[kw], W0.mag[kw], W0.expo[kw], wnc);
      if (n_part_ideal) {
        // aero_state_prepare_weight_for_add (aero_state.F90:704-752)
        double n_new = (double)cnt[kc] + n_avg;
        double ideal = n_part_ideal[kc];
        if (n_new != 0.0 && (n_new < ideal / 2.0 || n_new > ideal * 2.0))
          cnt[kc] = (int)scale_weight_members(c, pop, g, cl, cnt[kc], n_new / ideal, allow_doubling != 0,
                                              allow_halving != 0, hr, call);
      }
      if (n_avg == 0.0) continue;
      const Weights& W = ph.own_w ? ph.w : c.w;
      int wt = W.type[kw];
      double mag = W.mag[kw], expo = W.expo[kw];
      n_avg = sample_prop * mode_number(h, wt, mag, expo, wnc);
      int n = rand_poisson(hr, n_avg);
      if (n < 0) throw Fail(PMC_ERR_CAPACITY);
      double size_factor = std::min(1.0 / (characteristic_factor * n_avg), 0.32);
      added += n;
      if (n == 0) continue;
      PopCtr r = read_ctr(c, pop);
      long long need = (long long)r.n_slots + n;
      if (need > (1LL << 31) - 1) throw Fail(PMC_ERR_CAPACITY);
      if (need > ph.h.cap) relayout(c, pop, (int)std::min<long long>(need * 3 / 2 + 1024, (1LL << 31) - 1), false);
      SampleBatch B{};
      B.n = n;
      B.type = h.type;
      B.group = g;
      B.cls = cl;
      B.w_type = wt;
      B.w_mag = mag;
      B.w_expo = expo;
      B.log10_std = h.log10_std;
      B.x_mean = h.type == kModeLogNormal ? x_mean_prime(h, wt, expo) : 0.0;
      B.threshold = size_factor;
      B.char_radius = h.char_radius;
      B.char_vol = rad2vol(c.frac, h.char_radius);
      B.n_sample = h.n_sample;
      B.sample_radius = d_sr + h.r_off;
      if (h.type == kModeSampled) {
        std::memcpy(&hbuf[2 * n_vf + r_tot + wnc_used], wnc.data(), sizeof(double) * wnc.size());
        B.wnc = d_wnc + wnc_used;
        wnc_used += (long long)wnc.size();
      }
      B.vol_frac = d_vf + (size_t)m * ns;
      B.vol_frac_std = d_vf + n_vf + (size_t)m * ns;
      B.any_std = 0;
      for (int s = 0; s < ns; s++)
        if (hbuf[n_vf + (size_t)m * ns + s] > 0.0) B.any_std = 1;
      B.source = h.source;
      B.create_time = create_time;
      // the whole staging array is copied before every batch: it is small,
      // and the batch's weighted concentrations were just written into it
      CK(cudaMemcpyAsync(c.sample_buf.p, hbuf.data(), sizeof(double) * hbuf.size(), cudaMemcpyHostToDevice,
                         c.stream));
      if (c.dirty) push_pops(c);
      k_sample_batch<<<grid_for(n, 256), 256, 0, c.stream>>>(ph.h, B, r.n_slots, r.next_id, call, idx);
      note_launch();
      idx += (uint32_t)n;
      r.n_slots += n;
      r.n_live += n;
      r.next_id += n;
      write_ctr(c, pop, r);
      cnt[kc] += n;
    }
  ph.valid_sort = false;
  ph.caches_valid = false;
  c.replay.valid = false;
  push_pops(c);
  CK(cudaStreamSynchronize(c.stream));
  PopCtr r = read_ctr(c, pop);
  ph.rm_count = r.n_removed;
  if (n_part_add) *n_part_add = added;
  if (r.status) return r.status;
  if (ph.h.rm_on && r.n_removed > ph.h.rm_cap) return PMC_ERR_CAPACITY;
  return PMC_OK;
  GUARD_END
}

int pmc_coag_gpu_size_dist(pmc_coag_gpu_ctx* x, int pop, int n_bin, double d_min, double d_max, double* num_dist,
                           double* mass_dist) {
  if (!x || pop < 0 || pop >= x->c.n_pop || n_bin < 1 || !(d_min > 0.0) || !(d_max > d_min) || !num_dist)
    return PMC_ERR_INVALID_ARG;
  Ctx& c = x->c;
  size_t nv = (size_t)n_bin * (1 + c.n_spec);
  if (nv * sizeof(double) > 96 * 1024) return PMC_ERR_CAPACITY;  // the per-block histogram lives in shared memory
  GUARD_BEGIN
  PopHost& ph = c.pops[pop];
  c.st_d.reserve(nv);
  CK(cudaMemsetAsync(c.st_d.p, 0, sizeof(double) * nv, c.stream));
  PopCtr r = read_ctr(c, pop);
  if (r.n_slots > 0 && c.n_spec <= kDistFewSpec) {
    const size_t smem = sizeof(double) * nv;
    if (smem > 48 * 1024)
      CK(cudaFuncSetAttribute(k_size_dist_few, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    k_size_dist_few<<<std::min(grid_for(r.n_slots, 256), c.n_sm * 4), 256, smem, c.stream>>>(
        ph.h, n_bin, log(d_min), log(d_max), (double)n_bin / (log(d_max) - log(d_min)), c.st_d.p);
    note_launch();
  } else if (r.n_slots > 0) {
    // half tiles while two blocks an SM take them all: the call takes 63 us for
    // 15,838 slots of 20 species (75 with whole tiles, too few blocks) and 65 for
    // 120,000 (75); from 250,000 slots on, whole tiles are as fast or faster (76
    // against 78; 138 against 150 for 1e6)
    const bool half = r.n_slots <= 2LL * c.n_sm * (kDistTile / 2);
    const int tile = half ? kDistTile / 2 : kDistTile;
    const size_t smem = sizeof(double) * nv + tile * (sizeof(double) + 2 * sizeof(int)) + sizeof(int) * n_bin;
    auto k = c.n_spec > 32 ? (half ? k_size_dist<true, kDistTile / 2> : k_size_dist<true, kDistTile>)
                           : (half ? k_size_dist<false, kDistTile / 2> : k_size_dist<false, kDistTile>);
    if (smem > 48 * 1024) CK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int per_sm = (int)std::max<size_t>(1, std::min<size_t>(4, (220 * 1024) / (smem + 1024)));
    const long long tiles = (r.n_slots + tile - 1) / tile;
    k<<<(unsigned)std::min<long long>(tiles, (long long)c.n_sm * per_sm), kDistThreads, smem, c.stream>>>(
        ph.h, n_bin, log(d_min), log(d_max), (double)n_bin / (log(d_max) - log(d_min)), c.st_d.p);
    note_launch();
  }
  CK(cudaMemcpyAsync(num_dist, c.st_d.p, sizeof(double) * n_bin, cudaMemcpyDeviceToHost, c.stream));
  if (mass_dist)
    CK(cudaMemcpyAsync(mass_dist, c.st_d.p + n_bin, sizeof(double) * n_bin * c.n_spec, cudaMemcpyDeviceToHost,
                       c.stream));
  CK(cudaStreamSynchronize(c.stream));
  return PMC_OK;
  GUARD_END
}

int pmc_coag_gpu_get_weight(pmc_coag_gpu_ctx* x, int pop, double* w_mag) {
  if (!x || pop < 0 || pop >= x->c.n_pop || !w_mag) return PMC_ERR_INVALID_ARG;
  Ctx& c = x->c;
  const Weights& w = c.pops[pop].own_w ? c.pops[pop].w : c.w;
  for (int cl = 0; cl < c.n_class; cl++)
    for (int g = 0; g < c.n_group; g++) w_mag[g + c.n_group * cl] = w.mag[g + kMaxGroup * cl];
  return PMC_OK;
}

int pmc_coag_gpu_sync_host(pmc_coag_gpu_ctx* x, int pop, int cap, double* vol, int* group, int* cls,
                           int64_t* id, int* n_primary, uint8_t* alive, int* n_slots, int* n_changed, int* full) {
  if (!x || pop < 0 || pop >= x->c.n_pop || cap < 0 || !vol || !group || !cls || !id || !n_primary || !alive)
    return PMC_ERR_INVALID_ARG;
  Ctx& c = x->c;
  GUARD_BEGIN
  PopHost& ph = c.pops[pop];
  PopCtr r = read_ctr(c, pop);
  if (n_slots) *n_slots = r.n_slots;
  if (r.n_slots > cap) return PMC_ERR_CAPACITY;
  int ns = c.n_spec;
  if (full && *full) ph.mirror_full = true;  // the caller asks for every slot (new arrays)
  if (ph.mirror_full) {
    // every slot: the slot arrays already have the host layout
    size_t n = (size_t)r.n_slots;
    if (n > 0) {
      CK(cudaMemcpyAsync(vol, ph.h.vol, sizeof(double) * n * ns, cudaMemcpyDeviceToHost, c.stream));
      CK(cudaMemcpyAsync(group, ph.h.grp, sizeof(int) * n, cudaMemcpyDeviceToHost, c.stream));
      CK(cudaMemcpyAsync(cls, ph.h.cls, sizeof(int) * n, cudaMemcpyDeviceToHost, c.stream));
      CK(cudaMemcpyAsync(id, ph.h.id, sizeof(long long) * n, cudaMemcpyDeviceToHost, c.stream));
      CK(cudaMemcpyAsync(n_primary, ph.h.nprim, sizeof(int) * n, cudaMemcpyDeviceToHost, c.stream));
      CK(cudaMemcpyAsync(alive, ph.h.alive, n, cudaMemcpyDeviceToHost, c.stream));
    }
    CK(cudaMemsetAsync(ph.h.changed, 0, ph.h.cap, c.stream));
    CK(cudaStreamSynchronize(c.stream));
    if ((size_t)cap > n) memset(alive + n, 0, (size_t)cap - n);
    ph.mirror_full = false;
    ph.mirror_slots = r.n_slots;
    if (n_changed) *n_changed = r.n_slots;
    if (full) *full = 1;
    return PMC_OK;
  }
  int range = std::max(ph.mirror_slots, r.n_slots);
  if (range > ph.h.cap) range = ph.h.cap;
  long long total = 0;
  if (range > 0) {
    // pack the changed slots into records that the device writes straight
    // into page-locked host memory (room for every slot of the range), so
    // the records cross the bus while the kernel runs.  The range goes in
    // up to four chunks: after each, a copy of the running record count and
    // an event, so the host scatters one chunk's records while the device
    // packs the next
    const int rec = (kSyncHead + 8 * ns + 15) & ~15;  // keeps every record's header 16-byte aligned
    c.map.reserve((size_t)range * rec);
    c.st_cnt.reserve(1);
    c.pin.reserve(64);
    for (auto& ev : c.sync_ev)
      if (!ev) CK(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
    const int n_chunk = range >= (1 << 18) ? 4 : 1;
    const int wpb = std::max(1, std::min(4, (int)(48 * 1024 / (32 * rec))));  // warps per block
    const size_t smem = (size_t)wpb * 32 * rec;
    unsigned long long* h_cnt = (unsigned long long*)c.pin.p;
    const unsigned char* h_rec = (const unsigned char*)c.map.p;
    CK(cudaMemsetAsync(c.st_cnt.p, 0, sizeof(unsigned long long), c.stream));
    for (int k = 0; k < n_chunk; k++) {
      const int lo = (int)((long long)range * k / n_chunk), hi = (int)((long long)range * (k + 1) / n_chunk);
      k_pack_changed<<<grid_for(hi - lo, 32 * wpb), 32 * wpb, smem, c.stream>>>(ph.h, lo, hi, c.st_cnt.p,
                                                                                (unsigned char*)c.map.dev, rec);
      note_launch();
      CK(cudaMemcpyAsync(h_cnt + k, c.st_cnt.p, sizeof(unsigned long long), cudaMemcpyDeviceToHost, c.stream));
      CK(cudaEventRecord(c.sync_ev[k], c.stream));
    }
    // scatter each chunk's records into the caller's slot-indexed arrays
    long long j0 = 0;
    const int n_thr = (int)std::min<unsigned>(16, std::max(1u, std::thread::hardware_concurrency()));
    if (!c.pool) c.pool.reset(new HostPool());
    for (int k = 0; k < n_chunk; k++) {
      CK(cudaEventSynchronize(c.sync_ev[k]));
      const long long j1 = (long long)h_cnt[k];
      const long long nk = j1 - j0;
      const std::function<void(int, int)> work = [&](int q, int nq) {
        const long long a1 = j0 + nk * (q + 1) / nq;
        for (long long j = j0 + nk * q / nq; j < a1; j++) {
          const unsigned char* e = h_rec + (size_t)j * rec;
          const int* hd = (const int*)e;
          const int sl = hd[0];
          alive[sl] = (uint8_t)hd[1];
          if (!hd[1]) continue;
          group[sl] = hd[2];
          cls[sl] = hd[3];
          n_primary[sl] = hd[4];
          memcpy(&id[sl], e + 24, sizeof(long long));
          memcpy(vol + (size_t)sl * ns, e + kSyncHead, sizeof(double) * ns);
        }
      };
      c.pool->run(nk > 4096 ? n_thr : 1, work);
      j0 = j1;
    }
    total = j0;
  }
  ph.mirror_slots = r.n_slots;
  if (n_changed) *n_changed = (int)total;
  if (full) *full = 0;
  return PMC_OK;
  GUARD_END
}

int pmc_coag_gpu_download(pmc_coag_gpu_ctx* x, int pop, int max_part, double* vol, int* group, int* cls,
                          int64_t* id, int* n_primary, int* n_part) {
  if (!x || pop < 0 || pop >= x->c.n_pop) return PMC_ERR_INVALID_ARG;
  GUARD_BEGIN
  return do_download(x->c, pop, max_part, vol, group, cls, id, n_primary, nullptr, nullptr, nullptr, n_part);
  GUARD_END
}

int pmc_coag_gpu_download_components(pmc_coag_gpu_ctx* x, int pop, int max_part, int* n_comp,
                                     int* comp_source, double* comp_create_time) {
  if (!x || pop < 0 || pop >= x->c.n_pop) return PMC_ERR_INVALID_ARG;
  GUARD_BEGIN
  return do_download(x->c, pop, max_part, nullptr, nullptr, nullptr, nullptr, nullptr, n_comp,
                     comp_source, comp_create_time, nullptr);
  GUARD_END
}

int pmc_coag_gpu_set_weight(pmc_coag_gpu_ctx* x, const int* w_type, const double* w_mag,
                            const double* w_exp) {
  if (!x || !w_type || !w_mag || !w_exp) return PMC_ERR_INVALID_ARG;
  Ctx& c = x->c;
  GUARD_BEGIN
  for (int cl = 0; cl < c.n_class; cl++)
    for (int g = 0; g < c.n_group; g++) {
      int src = g + c.n_group * cl, dst = g + kMaxGroup * cl;
      if (w_type[src] < 1 || w_type[src] > 3) return PMC_ERR_INVALID_ARG;
      c.w.type[dst] = w_type[src];
      c.w.mag[dst] = w_mag[src];
      c.w.expo[dst] = w_exp[src];
    }
  c.wver++;
  for (auto& ph : c.pops) {
    if (!ph.own_w) ph.wver++;  // populations with weights of their own keep them
    set_params(c, ph);
    ph.valid_sort = false;  // aero_state_set_weight clears valid_sort
  }
  c.replay.valid = false;
  push_pops(c);
  CK(cudaStreamSynchronize(c.stream));
  return PMC_OK;
  GUARD_END
}

int pmc_coag_gpu_set_fractal(pmc_coag_gpu_ctx* x, double frac_dim, double prime_radius, double vol_fill_factor) {
  // spec_file_read_fractal stops for d_f > 3 (fractal.F90:587); d_f, R0 and
  // f also divide or take roots, so each must be positive
  if (!x || !(frac_dim > 0.0 && frac_dim <= 3.0) || !(prime_radius > 0.0) || !(vol_fill_factor > 0.0))
    return PMC_ERR_INVALID_ARG;
  Ctx& c = x->c;
  GUARD_BEGIN
  c.frac = make_fractal(frac_dim, prime_radius, vol_fill_factor);
  // radii, records, grid and k_max bounds all follow the particle shape
  for (auto& ph : c.pops) {
    ph.h.benv = brown_env(ph.h.temp > 0.0 ? ph.h.temp : 288.0, ph.h.pressure > 0.0 ? ph.h.pressure : 1e5, c.frac);
    ph.wver++;
    ph.valid_sort = false;
    ph.h.kmax_valid = 0;
    ph.h.pair_setup_valid = 0;
  }
  c.replay.valid = false;
  c.dirty = true;
  push_pops(c);
  CK(cudaStreamSynchronize(c.stream));
  return PMC_OK;
  GUARD_END
}

int pmc_coag_gpu_set_weight_pop(pmc_coag_gpu_ctx* x, int pop, const int* w_type, const double* w_mag,
                                const double* w_exp) {
  if (!x || pop < 0 || pop >= x->c.n_pop || !w_type || !w_mag || !w_exp) return PMC_ERR_INVALID_ARG;
  Ctx& c = x->c;
  GUARD_BEGIN
  PopHost& ph = c.pops[pop];
  Weights w = c.w;
  for (int cl = 0; cl < c.n_class; cl++)
    for (int g = 0; g < c.n_group; g++) {
      int src = g + c.n_group * cl, dst = g + kMaxGroup * cl;
      if (w_type[src] < 1 || w_type[src] > 3) return PMC_ERR_INVALID_ARG;
      w.type[dst] = w_type[src];
      w.mag[dst] = w_mag[src];
      w.expo[dst] = w_exp[src];
    }
  ph.w = w;
  ph.own_w = true;
  ph.wver++;  // only this population's caches go stale
  set_params(c, ph);
  ph.valid_sort = false;
  c.replay.valid = false;
  push_pops(c);
  CK(cudaStreamSynchronize(c.stream));
  return PMC_OK;
  GUARD_END
}

int pmc_coag_gpu_set_next_id(pmc_coag_gpu_ctx* x, int pop, int64_t next_id) {
  if (!x || pop < 0 || pop >= x->c.n_pop) return PMC_ERR_INVALID_ARG;
  GUARD_BEGIN
  PopCtr r = read_ctr(x->c, pop);
  r.next_id = next_id;
  write_ctr(x->c, pop, r);
  CK(cudaStreamSynchronize(x->c.stream));
  return PMC_OK;
  GUARD_END
}

int pmc_coag_gpu_get_next_id(pmc_coag_gpu_ctx* x, int pop, int64_t* next_id) {
  if (!x || pop < 0 || pop >= x->c.n_pop || !next_id) return PMC_ERR_INVALID_ARG;
  GUARD_BEGIN
  *next_id = read_ctr(x->c, pop).next_id;
  return PMC_OK;
  GUARD_END
}

int pmc_coag_gpu_set_seed(pmc_coag_gpu_ctx* x, int pop, uint64_t seed) {
  if (!x || pop < 0 || pop >= x->c.n_pop) return PMC_ERR_INVALID_ARG;
  PopHost& ph = x->c.pops[pop];
  ph.seed = seed;
  ph.h.seed = seed;
  ph.step = 0;  // the population's streams start again at step 1
  x->c.dirty = true;
  return PMC_OK;
}

int pmc_coag_gpu_set_graphs(pmc_coag_gpu_ctx* x, int enable) {
  if (!x || (enable != 0 && enable != 1)) return PMC_ERR_INVALID_ARG;
  x->c.use_graph = enable == 1;
  return PMC_OK;
}

// For the tests, not in the header: the next step finds a look-back that gave
// up, as check_scan_err and the step's own checks would after a real one.
int pmc_coag_gpu_test_scan_give_up(pmc_coag_gpu_ctx* x) {
  if (!x) return PMC_ERR_INVALID_ARG;
  Ctx& c = x->c;
  GUARD_BEGIN
  const unsigned long long one = 1ULL;
  CK(cudaMemcpyAsync(c.scan_err.p, &one, sizeof(one), cudaMemcpyHostToDevice, c.stream));
  CK(cudaStreamSynchronize(c.stream));
  return PMC_OK;
  GUARD_END
}

int pmc_coag_gpu_set_mode(pmc_coag_gpu_ctx* x, int mode) {
  if (!x || mode < PMC_MODE_FP64 || mode > PMC_MODE_REPLAY) return PMC_ERR_INVALID_ARG;
  x->c.mode = mode;
  for (auto& ph : x->c.pops) ph.valid_sort = ph.valid_sort && mode != PMC_MODE_REPLAY;
  return PMC_OK;
}

int pmc_coag_gpu_replay_set(pmc_coag_gpu_ctx* x, const double* u, int64_t n) {
  if (!x || (n > 0 && !u) || n < 0) return PMC_ERR_INVALID_ARG;
  Ctx& c = x->c;
  GUARD_BEGIN
  c.replay_u.reserve((size_t)std::max<int64_t>(n, 1));
  if (n > 0) {
    CK(cudaMemcpyAsync(c.replay_u.p, u, sizeof(double) * n, cudaMemcpyHostToDevice, c.stream));
    CK(cudaStreamSynchronize(c.stream));
  }
  c.replay_n = n;
  c.replay_used = 0;
  return PMC_OK;
  GUARD_END
}

int pmc_coag_gpu_replay_open(pmc_coag_gpu_ctx* x, const char* path) {
  if (!x || !path) return PMC_ERR_INVALID_ARG;
  FILE* f = fopen(path, "rb");
  if (!f) return PMC_ERR_INVALID_ARG;
  std::vector<double> u;
  double buf[4096];
  size_t m;
  while ((m = fread(buf, sizeof(double), 4096, f)) > 0) u.insert(u.end(), buf, buf + m);
  fclose(f);
  return pmc_coag_gpu_replay_set(x, u.data(), (int64_t)u.size());
}

int pmc_coag_gpu_replay_used(pmc_coag_gpu_ctx* x, int64_t* n_used) {
  if (!x || !n_used) return PMC_ERR_INVALID_ARG;
  *n_used = x->c.replay_used;
  return PMC_OK;
}

int pmc_coag_gpu_stats(pmc_coag_gpu_ctx* x, int64_t* kmax_violations, int64_t* redraws, int64_t* rounds) {
  if (!x) return PMC_ERR_INVALID_ARG;
  if (kmax_violations) *kmax_violations = x->c.last_kmax_warn;
  if (redraws) *redraws = x->c.last_redraws;
  if (rounds) *rounds = x->c.last_rounds;
  return PMC_OK;
}

int pmc_coag_gpu_exact_tests(pmc_coag_gpu_ctx* x, int64_t* n) {
  if (!x || !n) return PMC_ERR_INVALID_ARG;
  *n = x->c.exact_tests;
  return PMC_OK;
}

int pmc_coag_gpu_set_record_removals(pmc_coag_gpu_ctx* x, int enable) {
  if (!x) return PMC_ERR_INVALID_ARG;
  Ctx& c = x->c;
  GUARD_BEGIN
  for (auto& ph : c.pops) ph.h.rm_on = enable ? 1 : 0;
  reserve_removal_logs(c);
  push_pops(c);
  CK(cudaStreamSynchronize(c.stream));
  return PMC_OK;
  GUARD_END
}

int pmc_coag_gpu_removals(pmc_coag_gpu_ctx* x, int pop, int64_t max_n, int64_t* id, int* action,
                          int64_t* other_id, int64_t* n) {
  if (!x || pop < 0 || pop >= x->c.n_pop || max_n < 0 || !n || (max_n > 0 && (!id || !action || !other_id)))
    return PMC_ERR_INVALID_ARG;
  Ctx& c = x->c;
  GUARD_BEGIN
  PopHost& ph = c.pops[pop];
  PopCtr r = read_ctr(c, pop);
  *n = r.n_removed;
  ph.rm_count = r.n_removed;
  if (r.n_removed > ph.h.rm_cap && ph.h.rm_on) return PMC_ERR_CAPACITY;  // records were dropped
  if (r.n_removed > max_n) return PMC_ERR_CAPACITY;                     // nothing copied or cleared
  if (r.n_removed > 0) {
    std::vector<RemovalRec> h((size_t)r.n_removed);
    CK(cudaMemcpyAsync(h.data(), ph.h.rm_log, sizeof(RemovalRec) * h.size(), cudaMemcpyDeviceToHost, c.stream));
    CK(cudaStreamSynchronize(c.stream));
    for (size_t k = 0; k < h.size(); k++) {
      id[k] = h[k].id;
      action[k] = h[k].action;
      other_id[k] = h[k].other_id;
    }
  }
  r.n_removed = 0;
  write_ctr(c, pop, r);
  ph.rm_count = 0;
  return PMC_OK;
  GUARD_END
}

int pmc_coag_gpu_profile(pmc_coag_gpu_ctx* x, int enable) {
  if (!x) return PMC_ERR_INVALID_ARG;
  Ctx& c = x->c;
  GUARD_BEGIN
  prof_collect(c);
  c.prof = enable != 0;
  for (int i = 0; i < 4; i++) {
    c.prof_ms[i] = 0.0;
    c.prof_launch[i] = c.prof_units[i] = 0;
  }
  return PMC_OK;
  GUARD_END
}

int pmc_coag_gpu_profile_read(pmc_coag_gpu_ctx* x, int which, double* total_ms, int64_t* launches,
                              int64_t* units) {
  if (!x || which < 0 || which > 3) return PMC_ERR_INVALID_ARG;
  prof_collect(x->c);
  if (total_ms) *total_ms = x->c.prof_ms[which];
  if (launches) *launches = x->c.prof_launch[which];
  if (units) *units = x->c.prof_units[which];
  return PMC_OK;
}

int pmc_coag_gpu_launch_count(int64_t* n) {
  if (!n) return PMC_ERR_INVALID_ARG;
  *n = g_launches;
  return PMC_OK;
}

int pmc_coag_gpu_conflicts(pmc_coag_gpu_ctx* x, int64_t* events, int64_t* event_losers,
                           int64_t* target_ops, int64_t* target_op_losers) {
  if (!x) return PMC_ERR_INVALID_ARG;
  if (events) *events = x->c.last_events;
  if (event_losers) *event_losers = x->c.last_set_losers;
  if (target_ops) *target_ops = x->c.last_ops;
  if (target_op_losers) *target_op_losers = x->c.last_pp_lost;
  return PMC_OK;
}

int pmc_coag_gpu_sort(pmc_coag_gpu_ctx* x, int pop, int* n_bin, double* edges, int max_bin, int* counts,
                      int* bins) {
  if (!x || pop < 0 || pop >= x->c.n_pop) return PMC_ERR_INVALID_ARG;
  Ctx& c = x->c;
  GUARD_BEGIN
  sort_pops(c, true);
  CK(cudaStreamSynchronize(c.stream));
  PopHost& ph = c.pops[pop];
  if (n_bin) *n_bin = ph.n_bin;
  if (ph.n_bin > max_bin) return PMC_ERR_CAPACITY;
  if (edges && ph.n_bin > 0) memcpy(edges, ph.edges.data(), sizeof(double) * (ph.n_bin + 1));
  if (counts && ph.n_bin > 0)
    CK(cudaMemcpy(counts, ph.h.cell_count, sizeof(int) * ph.n_bin * c.n_class, cudaMemcpyDeviceToHost));
  if (bins) {
    PopCtr r = read_ctr(c, pop);
    std::vector<int> b(std::max(r.n_slots, 1));
    std::vector<uint8_t> a(std::max(r.n_slots, 1));
    if (r.n_slots > 0) {
      CK(cudaMemcpy(b.data(), ph.h.cell, sizeof(int) * r.n_slots, cudaMemcpyDeviceToHost));
      CK(cudaMemcpy(a.data(), ph.h.alive, r.n_slots, cudaMemcpyDeviceToHost));
    }
    int j = 0;
    for (int i = 0; i < r.n_slots; i++)
      if (a[i]) bins[j++] = (b[i] >= 0 && ph.n_bin > 0) ? b[i] % ph.n_bin + 1 : 0;
  }
  return PMC_OK;
  GUARD_END
}

int pmc_coag_gpu_kmax_table(pmc_coag_gpu_ctx* x, int kernel_type, double temp, double pressure,
                            double additive_coeff, double* kmax, int max_bin) {
  if (!x || !kmax) return PMC_ERR_INVALID_ARG;
  Ctx& c = x->c;
  GUARD_BEGIN
  PopHost& ph = c.pops[0];
  if (ph.n_bin > max_bin) return PMC_ERR_CAPACITY;
  ph.h.kernel_type = kernel_type;
  ph.h.temp = temp;
  ph.h.pressure = pressure;
  ph.h.coeff = additive_coeff;
  ph.h.benv = brown_env(temp, pressure, c.frac);
  ph.h.kmax_valid = 0;
  push_pops(c);
  int nb = std::max(ph.n_bin, 1);
  launch_kmax(c);
  CK(cudaStreamSynchronize(c.stream));
  CK(cudaGetLastError());
  if (ph.n_bin > 0) CK(cudaMemcpy(kmax, ph.h.kmax_tab, sizeof(double) * ph.n_bin * ph.n_bin, cudaMemcpyDeviceToHost));
  ph.h.kmax_valid = 1;
  push_pops(c);
  return PMC_OK;
  GUARD_END
}

int pmc_coag_gpu_eval_kernel(pmc_coag_gpu_ctx* x, int kernel_type, double temp, double pressure,
                             double additive_coeff, int n_pairs, const double* vol1, const int* c1,
                             const double* vol2, const int* c2, const int* c_ij, double* k_out) {
  if (!x || n_pairs < 0 || (n_pairs > 0 && (!vol1 || !vol2 || !c1 || !c2 || !c_ij || !k_out)))
    return PMC_ERR_INVALID_ARG;
  Ctx& c = x->c;
  GUARD_BEGIN
  if (n_pairs == 0) return PMC_OK;
  PopDev P = c.pops[0].h;
  P.kernel_type = kernel_type;
  P.temp = temp;
  P.pressure = pressure;
  P.coeff = additive_coeff;
  P.benv = brown_env(temp, pressure, c.frac);
  std::vector<void*> tmp;
  size_t nv = (size_t)n_pairs * c.n_spec;
  double* d1 = dalloc<double>(c, tmp, nv);
  double* d2 = dalloc<double>(c, tmp, nv);
  int* e1 = dalloc<int>(c, tmp, n_pairs);
  int* e2 = dalloc<int>(c, tmp, n_pairs);
  int* e3 = dalloc<int>(c, tmp, n_pairs);
  double* out = dalloc<double>(c, tmp, n_pairs);
  CK(cudaMemcpyAsync(d1, vol1, sizeof(double) * nv, cudaMemcpyHostToDevice, c.stream));
  CK(cudaMemcpyAsync(d2, vol2, sizeof(double) * nv, cudaMemcpyHostToDevice, c.stream));
  CK(cudaMemcpyAsync(e1, c1, sizeof(int) * n_pairs, cudaMemcpyHostToDevice, c.stream));
  CK(cudaMemcpyAsync(e2, c2, sizeof(int) * n_pairs, cudaMemcpyHostToDevice, c.stream));
  CK(cudaMemcpyAsync(e3, c_ij, sizeof(int) * n_pairs, cudaMemcpyHostToDevice, c.stream));
  k_eval_kernel<<<(n_pairs + 127) / 128, 128, 0, c.stream>>>(P, n_pairs, d1, e1, d2, e2, e3, out,
                                                             c.mode == PMC_MODE_MIXED ? 1 : 0); note_launch();
  CK(cudaStreamSynchronize(c.stream));
  CK(cudaGetLastError());
  CK(cudaMemcpy(k_out, out, sizeof(double) * n_pairs, cudaMemcpyDeviceToHost));
  free_list(c, tmp);
  return PMC_OK;
  GUARD_END
}

}  // extern "C"
