// pmc_merge.cuh -- applying accepted coagulation events on the device.
//
// Per-set events: coagulate_weighting + coagulate (coagulation.F90:810-985).
// Per-particle (accelerated) path: sample_source_particle +
// coag_target_with_source (coagulation.F90:333-582), one warp per target.
// Every write to a particle slot is guarded by the slot's claim word: an
// event or target operation is applied only if it holds the lowest priority
// on every slot it writes or removes; otherwise it is retried (or dropped,
// k_items) in the next round.
#pragma once

#include <type_traits>

#include "pmc_kernels.cuh"
#include "pmc_particle.cuh"

namespace pmc {

// Chains (see the walks below): the events of one walk that absorbs its
// partners one after another, in chunks of kChainChunk entries; entry
// kChainChunk - 1 of a chunk's y holds the index of the next chunk (-1: none)
constexpr int kChainChunk = 32;
constexpr int kChainMaxLen = 1 << 16;  // events of one chain in one round
// q of an entry: the pair, and kChainRemoves if the merge removes the partner
constexpr int kChainPairMask = (1 << 20) - 1;
constexpr int kChainRemoves = 1 << 30;

struct ChainPool {
  int* y;          // [n_chunks * kChainChunk] partner slot; the last entry of a chunk links the next chunk
  int* q;          // pair (local), with kChainRemoves if the merge removes the partner
  float* pos;      // position in the pair's test sequence
  long long* ctr;  // chunks handed out in this round (device)
  long long n_chunks;
};

struct ChainWriter {
  int head = -1, chunk = -1, fill = 0, len = 0;
  __device__ bool append(const ChainPool& C, int y, int q, float pos) {
    if (chunk < 0 || fill == kChainChunk - 1) {
      long long nc = (long long)inc_warp((unsigned long long*)C.ctr);
      if (nc >= C.n_chunks) return false;
      if (chunk >= 0) C.y[(size_t)chunk * kChainChunk + kChainChunk - 1] = (int)nc;
      else head = (int)nc;
      chunk = (int)nc;
      fill = 0;
      C.y[(size_t)chunk * kChainChunk + kChainChunk - 1] = -1;
    }
    size_t i = (size_t)chunk * kChainChunk + fill;
    C.y[i] = y;
    C.q[i] = q;
    C.pos[i] = pos;
    fill++;
    len++;
    return true;
  }
};

struct ChainReader {
  int chunk, k = 0;
  __device__ explicit ChainReader(int head) : chunk(head) {}
  // index of the next entry, -1 past the end of the links
  __device__ long long next(const ChainPool& C) {
    if (chunk < 0 || (long long)chunk >= C.n_chunks) return -1;
    size_t i = (size_t)chunk * kChainChunk + k;
    if (++k == kChainChunk - 1) {
      chunk = C.y[(size_t)chunk * kChainChunk + kChainChunk - 1];
      k = 0;
    }
    return (long long)i;
  }
};

// A chain stops at an accepted test that is no absorb (or that the pool has
// no room for).  That test has happened: dropping it and walking on afresh
// in the next round would redraw its merge decision until an absorb came up,
// which favours absorbs whenever the weights make some decisions keep the
// walking particle (with flat weights every decision absorbs).  So the
// stopping test is carried to the next round as a pending event with its
// decision: its partner, pair (and whether the walker is in the pair's first
// cell), decision and position, packed as {y, q | first << 30, decision,
// position bits}; y = -1 for none.  An event whose dest_out is kPendingTerm
// hands that test to the next round (k_items) instead of a walk.
constexpr int kPendingTerm = -2;
// The same holds for a chain cut short where a partner's claim failed: the
// claim's kind (write or read) follows the event's decision, so the cut
// depends on it, and walking on afresh would redraw that decision.  The
// first event not applied is pending for the next round (kPendingChain),
// its decision recomputed there from the chain's stream (event index in
// the decision word) and the particles' values, which give the decision
// the walk made whenever the partner is unchanged.
constexpr int kPendingChain = -3;
constexpr int kTermFirst = 1 << 30;
__device__ __forceinline__ int4 no_term() { return make_int4(-1, 0, 0, 0); }

__device__ __forceinline__ void kill_slot(const PopDev& P, int i) {
  P.alive[i] = 0;
  P.changed[i] = 1;
  P.cell[i] = -1;
}

// destination slot of a winning event that creates a particle (-1: none)
__device__ __forceinline__ int event_dest(const MergeDecision& m, int s1, int s2, int slot_base,
                                          long long slot_rank) {
  if (!m.create) return -1;
  if (m.rm1) return s1;
  if (m.rm2) return s2;
  return slot_base + (int)slot_rank;
}

constexpr int kMoveBlock = 8;

// The particle of a winning event that creates one, its per-particle vectors:
// the species of the two sources (particle-major, each source a few cache
// lines) are added in blocks of kMoveBlock: a block's loads are all issued
// before its sums are stored, and the destination (which may be a source) is
// written species by species after that species was read.  The components are
// gathered into local arrays before any is written, in the order of the
// random selection (computed from the stream position the test stored).
// Returns the sources' water volumes, read before the destination may be
// overwritten.
__device__ __forceinline__ double2 move_vectors(const PopDev& P, unsigned long long key, int s1, int s2, int dest,
                                                uint32_t used) {
  const int ns = P.n_spec;
  const double* v1 = P.vol + vol_at(P, s1, 0);
  const double* v2 = P.vol + vol_at(P, s2, 0);
  double* vd = P.vol + vol_at(P, dest, 0);
  const double2 ice = P.i_water > 0 ? make_double2(v1[P.i_water - 1], v2[P.i_water - 1]) : make_double2(0.0, 0.0);
  // components: every source entry is read before the first write
  int na = P.ncomp[s1], nb = P.ncomp[s2];
  na = na < kMaxComponent ? na : kMaxComponent;
  nb = nb < kMaxComponent ? nb : kMaxComponent;
  int ca[kMaxComponent], cb[kMaxComponent];
  double ta[kMaxComponent], tb[kMaxComponent];
  for (int k = 0; k < na; k++) {
    ca[k] = P.csrc[comp_at(s1, k)];
    ta[k] = P.ctime[comp_at(s1, k)];
  }
  for (int k = 0; k < nb; k++) {
    cb[k] = P.csrc[comp_at(s2, k)];
    tb[k] = P.ctime[comp_at(s2, k)];
  }
  // totals in the reference's order (species 1..n)
  double vt = 0.0, ms = 0.0;
  for (int s0 = 0; s0 < ns; s0 += kMoveBlock) {
    double x1[kMoveBlock], x2[kMoveBlock];
#pragma unroll
    for (int j = 0; j < kMoveBlock; j++) {
      x1[j] = s0 + j < ns ? v1[s0 + j] : 0.0;
      x2[j] = s0 + j < ns ? v2[s0 + j] : 0.0;
    }
#pragma unroll
    for (int j = 0; j < kMoveBlock; j++) {
      if (s0 + j < ns) {
        double v = x1[j] + x2[j];
        vt = vt + v;
        ms = ms + v * P.density[s0 + j];
        vd[s0 + j] = v;
      }
    }
  }
  int n1_new = na, n2_new = nb;
  if (na + nb > kMaxComponent) {
    int sa[kMaxComponent], sb[kMaxComponent];
    Rng g = merge_rng(P, key);
    g.seek(used);
    coag_components(g, na, P.nprim[s1], nb, P.nprim[s2], &n1_new, &n2_new, sa, sb);
    for (int k = 0; k < n1_new; k++) {
      P.csrc[comp_at(dest, k)] = ca[sa[k] - 1];
      P.ctime[comp_at(dest, k)] = ta[sa[k] - 1];
    }
    for (int k = 0; k < n2_new; k++) {
      P.csrc[comp_at(dest, n1_new + k)] = cb[sb[k] - 1];
      P.ctime[comp_at(dest, n1_new + k)] = tb[sb[k] - 1];
    }
  } else {
    for (int k = 0; k < na; k++) {
      P.csrc[comp_at(dest, k)] = ca[k];
      P.ctime[comp_at(dest, k)] = ta[k];
    }
    for (int k = 0; k < nb; k++) {
      P.csrc[comp_at(dest, na + k)] = cb[k];
      P.ctime[comp_at(dest, na + k)] = tb[k];
    }
  }
  P.vtot[dest] = vt;
  P.mass[dest] = ms;
  P.ncomp[dest] = n1_new + n2_new;
  return ice;
}

// particle fields that coag_scalars reads (component lists excluded)
__device__ __forceinline__ void load_scalars(const PopDev& P, int i, PMeta& m) {
  m.id = P.id[i];
  m.nprim = P.nprim[i];
  m.lct = P.lct[i];
  m.gct = P.gct[i];
  m.imf = P.imf[i];
  m.den_ice = P.den_ice[i];
  m.phi = P.phi[i];
  m.hyst = P.hyst[i];
  m.frozen = P.frozen[i];
}

// Apply winning per-set events (coagulate, coagulation.F90:928-985), one
// thread per event: the coagulated particle's vectors (move_vectors), the
// removals, its scalar fields, its radius, bin and pair-test record.  Among
// the round's winners a slot is written by one event or read by any number, so
// the events need no order among themselves.  Every slot an event removes or
// rewrites is stamped with the round's claim generation, and dest_out[e] gets
// the slot of the particle the event made (-1 if none).  One launch for what
// were two (vectors, then scalars), with the event's words loaded once.
__global__ void __launch_bounds__(256) k_apply(const PopDev* pops, const int* gpair_pop, const long long* n_events,
                                               const uint8_t* win, const long long* slot_rank,
                                               const long long* id_rank, const int* slot_base,
                                               const long long* id_base, const uint8_t* ev_done, int* dest_out,
                                               unsigned long long* ev_key, int2* ev, int* ev_gp, float* ev_pos,
                                               uint32_t* dec, const int4* ev_term, const long long* pop_pair_base) {
  chain_wait();
  long long E = *n_events;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < E;
       e += (long long)gridDim.x * blockDim.x) {
    if (win[e] == 2) continue;  // a chain: k_apply_chain's
    dest_out[e] = -1;
    if (win[e] != 1) continue;
    int gp = ev_gp[e];
    int pop = gpair_pop[gp];
    const PopDev& P = pops[pop];
    const unsigned long long key = ev_key[e];
    int p = (int)key_pair(key);
    int2 sl = ev[e];
    int s1 = sl.x, s2 = sl.y;
    uint32_t gen = *P.gen_p;
    uint32_t used;
    MergeDecision m = unpack_decision(dec[e], &used);
    add_ll_warp(&P.ctr->tot_coag, 1);
    if (m.rm1) P.touched[s1] = gen;
    if (m.rm2) P.touched[s2] = gen;
    if (!m.create) {
      // coagulate (coagulation.F90:928-985) records a removal whose ID is lost
      if (m.rm1 && m.lost1) log_removal(P, P.id[s1], kInfoCoag, 0);
      if (m.rm2 && m.lost2) log_removal(P, P.id[s2], kInfoCoag, 0);
      if (m.rm1) kill_slot(P, s1);
      if (m.rm2) kill_slot(P, s2);
      int dlive = -(int)m.rm1 - (int)m.rm2;
      if (dlive) add_ll_warp(&P.ctr->n_live, dlive);
      continue;
    }
    int dest = event_dest(m, s1, s2, slot_base[pop], m.rm1 || m.rm2 ? 0 : slot_rank[e]);
    if (dest >= P.cap) {
      cap_fail(P.ctr, kCapEventDest);
      continue;
    }
    if (dest < 0) {
      bad_index(P.ctr, kBadDest, dest);
      continue;
    }
    PMeta a, b, c;
    load_scalars(P, s1, a);
    load_scalars(P, s2, b);
    const double2 wi = move_vectors(P, key, s1, s2, dest, used);
    coag_scalars(a, wi.x, b, wi.y, c);
    P.grp[dest] = m.new_group;
    P.cls[dest] = P.pair[p].cc + 1;
    long long new_id;
    if (m.rm1 && !m.lost1) new_id = a.id;
    else if (m.rm2 && !m.lost2) new_id = b.id;
    else new_id = id_base[pop] + id_rank[e];
    P.id[dest] = new_id;
    if (m.rm1 && m.lost1) log_removal(P, a.id, kInfoCoag, new_id);
    if (m.rm2 && m.lost2) log_removal(P, b.id, kInfoCoag, new_id);
    P.nprim[dest] = c.nprim;
    P.lct[dest] = c.lct;
    P.gct[dest] = c.gct;
    P.imf[dest] = c.imf;
    P.den_ice[dest] = c.den_ice;
    P.phi[dest] = c.phi;
    P.hyst[dest] = c.hyst;
    P.frozen[dest] = c.frozen;
    P.alive[dest] = 1;
    P.changed[dest] = 1;
    // the coagulated particle must lie on the grid (aero_state_add_particle
    // with allow_resort=.false., aero_sorted.F90:427-440)
    P.touched[dest] = gen;
    int nbin = refresh_slot(P, dest);
    if (nbin < 1 || nbin > P.grid->n_bin) {
      set_status(P.ctr, kErrOutOfGrid);
    } else if (ev_term[e].x >= 0) {
      // a one-event chain that stopped at a pending test: the coagulated
      // particle (in slot dest) meets that test in the next round
      const int4 t = ev_term[e];
      const int tq = t.y & (kTermFirst - 1);
      const bool tfirst = (t.y & kTermFirst) != 0;
      ev_key[e] = make_key((uint32_t)tq, 1u, (uint32_t)dest);
      ev[e] = tfirst ? make_int2(dest, t.x) : make_int2(t.x, dest);
      ev_gp[e] = (int)(pop_pair_base[pop] + tq);
      ev_pos[e] = __int_as_float(t.w);
      dec[e] = (uint32_t)t.z;
      dest_out[e] = kPendingTerm;
    } else if (!(key_kind(key) == 1u && ev_done[e])) {
      dest_out[e] = dest;  // a walk that ran to its end stops
    }
    if (m.rm1 && dest != s1) kill_slot(P, s1);
    if (m.rm2 && dest != s2) kill_slot(P, s2);
    int dlive = 1 - (int)m.rm1 - (int)m.rm2;
    if (dlive) add_ll_warp(&P.ctr->n_live, dlive);
  }
}

// ---------------------------------------------------------------------------
// Walks.  In the sequential loop a particle that an event creates (or
// changes) at pair p0 takes part in the rest of the step: every later pair
// that contains its cell draws its samples with the particle among the
// cell's members, so it is tested against each member of the pair's other
// cell at rate k_max * del_t (the pair's samples, n1 * n2 * k_max * del_t in
// mean, fall on each of the n1 * n2 possible pairs alike; for one cell with
// itself n (n - 1) / 2 pairs and n - 1 partners).  A walk draws those tests
// as one Poisson process along the pairs that follow p0 in loop order, the
// rest of p0 itself from position pos0 (the fraction of p0's test sequence
// already done).
//
// Partners come from the cell lists of the sort at the round's start, so a
// walk meets every particle that earlier rounds of the step made.  A listed
// slot that is dead, has left the cell since, is the walking particle itself
// or was absorbed earlier in its chain is no member now, and a test that
// falls on it is dropped.  Particles that other walks of the same round
// change are met with the values they had at the round's start.  Pairs on
// the per-particle path are not walked.
//
// Chains.  A walk's accepted test whose merge decision (coagulate_weighting,
// drawn from the stream the event's apply uses) replaces the walking particle
// by the coagulated one is an absorb: the walk goes on at once with the
// coagulated particle's values (volumes summed as the apply sums them,
// radius, record, cell), as the sequential loop would test it next.  Each
// absorbed partner is claimed with its own key; the events are recorded in
// a chain (ChainPool) and applied, as far as their claims hold, by one
// thread in order (k_apply_chain).  A runaway collector that absorbs
// thousands of droplets in one step (the sedimentation kernel) takes one
// round, not one round per droplet.  The chain stops before an accepted
// test that is not an absorb; the walk resumes there in the next round.

// cell of a particle of radius r and class cls (1-based); -1 off the grid
__device__ __forceinline__ int cell_of(const PopDev& P, double r, int cls) {
  const GridDev& G = *P.grid;
  int b = bin_find(G.n_bin, G.log_lo, G.log_hi, r);
  if (b < 1 || b > G.n_bin || cls < 1 || cls > P.n_class) return -1;
  return (b - 1) + G.n_bin * (cls - 1);
}

// the walk's first accepted test, and its chain
struct WalkOut {
  bool found = false;
  int q = 0, y = 0;  // pair and partner of the first event
  float pos = 0.f;
  bool first_cell1 = true;  // the walking particle is in the pair's first cell
  bool done = false;        // the walk ran to the end after its last event
  uint32_t dec = 0;         // merge decision of the first event
  bool cont = false;        // the first event is an absorb: k_chain carries the walk on
  uint32_t g_used = 0;      // index of the walk's next test after the first event
  bool stop = false;        // the walk reached a per-particle pair (q) whose target cell is its cell
};

// true if claim word w is this round's claim of the chain of walker x
__device__ __forceinline__ bool is_walk_claim(const PopDev& P, unsigned long long w, int x) {
  return (w >> 53) == (unsigned long long)(~*P.gen_p & kGenLimit) && ((w >> 32) & 1ULL) &&
         (uint32_t)w == (uint32_t)x;
}

// The uniforms of a walk's test t: one Philox block keyed by the population,
// counted by (step, round, walk stream, walking slot, t).  x, y: the gap to
// the test (u53 -> exponential); z: the partner; w: the accept draw.  Every
// test takes one block whether or not its partner is a member, so a test's
// draws depend on its index alone.
__device__ __forceinline__ U4 walk_draws(const PopDev& P, int x, uint32_t t) {
  return philox4x32_10(U4{P.step, ((*P.round_p & 0xffu) << 4) | kStreamWalk, (uint32_t)x, t}, (uint32_t)P.seed,
                       (uint32_t)(P.seed >> 32));
}

// A walk's place in the stretch of its cell C: the entries lo..end of the
// cell's pair list, cum[j] (indexable by list entry j) the expected tests
// before entry j, at the running position, j the entry that holds it.
struct Stretch {
  const double* cum;
  const int* tab;
  int C, end, j;
  double at, total;
  int stop;  // the stop (cp_nstop) that ends the stretch, or -1: it runs to the cell's last pair
};

// the stretch of cell C from (pair p0, position pos0 in it) on.  The first
// entry of the cell's pair list whose pair is p0 or later: the cell's coarse
// row (every 16th entry, read as int4) counts the coarse entries before p0,
// then the at most 15 entries after the last of them are counted.
__device__ __forceinline__ void walk_stretch(const PopDev& P, int C, int p0, float pos0, Stretch* s) {
  int lo = P.cp_off[C], end = P.cp_off[C + 1];
  const double* cum = P.cp_cum + (lo + C) - lo;
  const int4* cz = reinterpret_cast<const int4*>(P.cp_coarse + (size_t)C * P.n_coarse);
  int k = 0;
#pragma unroll 4
  for (int b = 0; b < P.n_coarse / 4; b++) {
    const int4 v = cz[b];
    k += (v.x < p0) + (v.y < p0) + (v.z < p0) + (v.w < p0);
  }
  int a = k == 0 ? lo : lo + 16 * (k - 1) + 1;
  const int hi = min(lo + 16 * k, end);
  int cnt = 0;
#pragma unroll
  for (int t = 0; t < 15; t++)
    if (a + t < hi) cnt += P.cp_list[a + t] < p0;
  a += cnt;
  double at = cum[a];
  if (a < end && P.cp_list[a] == p0) at += (cum[a + 1] - cum[a]) * (double)pos0;
  // the stretch ends at the first stop after the start; a walk that starts
  // at the end of a pair (its target operation there is done) looks past it
  const int sa = (a < end && P.cp_list[a] == p0 && pos0 >= 1.0f) ? a + 1 : a;
  const int stop = (P.walk_stops && sa < end) ? P.cp_nstop[sa] : end;
  s->cum = cum;
  s->tab = P.cp_tab + (size_t)C * kWalkTab;
  s->C = C;
  s->stop = stop < end ? stop : -1;
  if (stop < end) end = stop;
  s->end = end;
  s->j = a < end ? a : (end > P.cp_off[C] ? end - 1 : end);
  s->at = at;
  s->total = cum[end];
}

// the entry j >= s.j with cum[j] <= at < cum[j + 1] (at < total): the
// cell's bucket table gives a start at or before it, a short scan forward
// usually ends there, a binary search covers the rest
__device__ __forceinline__ int walk_pair(const Stretch& s, double at) {
  const double* cum = s.cum;
  int b = (int)(at / s.total * (double)kWalkTab);
  b = b < 0 ? 0 : (b >= kWalkTab ? kWalkTab - 1 : b);
  int hi = s.end - 1;
  int j = s.tab[b];
  j = j < s.j ? s.j : (j > hi ? hi : j);
  int a, z;
  if (cum[j] > at) {  // rounding put the bucket past at
    a = s.j;
    z = j - 1 < s.j ? s.j : j - 1;
  } else {
    for (int k = 0; k < 4 && j < hi; k++) {
      if (cum[j + 1] > at) return j;
      j++;
    }
    a = j;
    z = hi;
  }
  while (a < z) {
    int mid = (a + z + 1) >> 1;
    if (cum[mid] <= at) a = mid;
    else z = mid - 1;
  }
  return a;
}

// Partner draws of a chain's test t after the first: the walk stream's
// block (x, t + r * 2^26) for the r-th redraw (t stays below 2^26).
constexpr uint32_t kChainRedraws = 64;
constexpr int kRedrawBatch = 4;
__device__ __forceinline__ uint32_t walk_redraw(const PopDev& P, int x, uint32_t t, uint32_t r) {
  return walk_draws(P, x, t | (r << 26)).x;
}

// The first of the redraws r = 1, 2, ... of a test whose partner is no
// absorbed member, -2 if every one is.  A collector that has emptied most of
// a cell redraws tens of times, so the redraws go kRedrawBatch at a time with
// their loads in flight together.
__device__ __noinline__ int redraw_partner(const PopDev& P, int x, uint32_t t, int o_start, int n_o) {
  for (uint32_t r0 = 1; r0 < kChainRedraws; r0 += kRedrawBatch) {
    int y[kRedrawBatch];
    unsigned long long w[kRedrawBatch];
#pragma unroll
    for (int k = 0; k < kRedrawBatch; k++) {
      int i = (int)(u32d(walk_redraw(P, x, t, r0 + k)) * (double)n_o);
      if (i >= n_o) i = n_o - 1;
      y[k] = P.list[o_start + i];
    }
#pragma unroll
    for (int k = 0; k < kRedrawBatch; k++) w[k] = y[k] >= 0 && y[k] < P.cap ? __ldcg(&P.claim[y[k]]) : 0ULL;
#pragma unroll
    for (int k = 0; k < kRedrawBatch; k++) {
      if (r0 + k >= kChainRedraws) break;
      if (!(y[k] >= 0 && y[k] < P.cap && is_walk_claim(P, w[k], x))) return y[k];
    }
  }
  return -2;
}

// One walk test t of particle x (records qxd/qxf) at running position at of
// its stretch, in entry j: the partner drawn from the other cell's members
// and the accept test.  The pair's fields and the partner slot are loaded
// together, then the partner's state.  In a chain, a partner that the chain
// has absorbed already is drawn again: the reference draws a pair's samples
// from the members left when each sample runs, after the earlier samples'
// merges, and exits the pair when a cell is empty (per_set_coag,
// coagulation.F90:628-638); a test whose kChainRedraws draws all land on
// absorbed members counts as that exit.  Returns 0 for no test (no member,
// itself, a dead or moved member, the exit), 1 for a rejected test, 2 for an
// accepted one, -1 for a failed bounds check.  *side gets kSideExact if the
// test was decided in FP64 and kSideWarn if k > k_max: the caller counts them,
// as a test drawn ahead of an accepted one never happens.
constexpr uint32_t kSideExact = 1u, kSideWarn = 2u;
template <int KT, class T, bool FLAT>
__device__ __forceinline__ int walk_test(const PopDev& P, int x, const Stretch& s, int j, double at, uint32_t t,
                                         uint32_t pick, uint32_t accu, const RecD& qxd, const RecF& qxf, bool chain,
                                         int* y_out, float* pos_out, int* q_out, bool* first_out, double* ry_out,
                                         double* vty_out, uint32_t* side) {
  *side = 0u;
  const double c0 = s.cum[j], c1 = s.cum[j + 1];
  const int4 ent = P.cp_ent[j];
  double lam = c1 - c0;
  int n_o = ent.w, o_start = ent.z;
  if (!(lam > 0.0) || n_o < 1) return 0;
  if (o_start < 0 || (long long)o_start + n_o > P.cap || ent.x < 0 || ent.x >= P.n_pairs) {
    bad_index(P.ctr, kBadPairCells, ent.x);
    return -1;
  }
  const int q = ent.x, O = ent.y & ((1 << 30) - 1);
  const bool first = (ent.y >> 30) & 1;
  int i = (int)(u32d(pick) * (double)n_o);
  if (i >= n_o) i = n_o - 1;
  int y = P.list[o_start + i];
  if (chain && y >= 0 && y < P.cap && is_walk_claim(P, __ldcg(&P.claim[y]), x)) {
    y = redraw_partner(P, x, t, o_start, n_o);
    if (y == -2) return 0;
  }
  const PairDesc d = P.pair_desc[q];
  const PairState& S = P.pair[q];
  const double inv_k_max = S.inv_k_max, fflat = S.fflat;
  const int cc = S.cc;
  if (y < 0 || y >= P.cap) {
    bad_index(P.ctr, kBadTestSlot, y);
    return -1;
  }
  const uint8_t alive = P.alive[y];
  const int cell_y = P.cell[y];
  const double ry = P.rad[y], vty = P.vtot[y];  // for the merge decision if the test accepts
  if (y == x || !alive || cell_y != O) return 0;
  const double u = u32d(accu);
  bool acc, warn = false;
  if constexpr (sizeof(T) == 8) {
    const RecD qy = P.recd[y];
    acc = accept_f64_rec<KT, FLAT>(P, first ? qxd : qy, first ? qy : qxd, d, cc, fflat, inv_k_max, u, &warn);
  } else {
    const RecF qy = P.recf[y];
    const float* qw = (const float*)&qxf;
    const float* py = (const float*)&qy;
    const float pf = pair_kernel<KT, float, FLAT>(P, first ? qw : py, first ? py : qw, d.c1, d.c2, cc,
                                                  (float)fflat, (float)P.coeff) *
                     (float)inv_k_max;
    if (f32_decides(pf, u)) {
      acc = u < (double)pf;
    } else {  // decided in FP64 (see f32_decides)
      const RecD qy = P.recd[y];
      acc = accept_f64_rec<KT, FLAT>(P, first ? qxd : qy, first ? qy : qxd, d, cc, fflat, inv_k_max, u, &warn);
      *side = kSideExact;
    }
  }
  if (warn) *side |= kSideWarn;
  *y_out = y;
  *pos_out = (float)((at - c0) / lam);
  *q_out = q;
  *first_out = first;
  *ry_out = ry;
  *vty_out = vty;
  return acc ? 2 : 1;
}

// The next accepted test of walker x from s on, drawing tests t_next,
// t_next + 1, ...: returns 1 with the test's entry in s.j and position in
// s.at, 0 if the walk ran to the end of the stretch, -1 on a failed check or
// the test limit.  n_tests counts the tests with a partner.
template <int KT, class T, bool FLAT>
__device__ __forceinline__ int walk_next(const PopDev& P, int x, Stretch& s, uint32_t& t_next, const RecD& qxd,
                                         const RecF& qxf, bool chain, long long* n_tests, int* y, float* pos,
                                         int* q, bool* first, double* ry, double* vty) {
  for (;;) {
    const uint32_t t = t_next++;
    U4 u = walk_draws(P, x, t);
    double at = s.at - log(u53(u.x, u.y));
    if (!(at < s.total)) {
      s.at = at;
      if (s.stop >= 0) {  // a per-particle pair that takes the particle as a target
        *q = P.cp_list[s.stop];
        return 3;
      }
      return 0;  // no test left in the cell's later pairs
    }
    if (t >= (1u << 26)) {  // far past any mean the step can ask for
      set_status(P.ctr, kErrTimeout);
      return -1;
    }
    int j = walk_pair(s, at);
    s.j = j;
    s.at = at;
    uint32_t side;
    int r = walk_test<KT, T, FLAT>(P, x, s, j, at, t, u.z, u.w, qxd, qxf, chain, y, pos, q, first, ry, vty, &side);
    if (side & kSideExact) add_ll(&P.ctr->exact_tests, 1LL);
    if (side & kSideWarn) add_ll(&P.ctr->kmax_warn, 1LL);
    if (r < 0) return -1;
    if (r == 0) continue;
    (*n_tests)++;
    if (r == 2) return 1;
  }
}

// The next 32 tests of one walker, one a lane (every lane of the warp takes
// the same walker).  What a test reads of the walker's cell, its pair and its
// partner does not depend on the walking particle's size, so a chain that
// stays in its cell goes on with the same tests after an absorb and evaluates
// only their acceptance again.
template <class T>
struct WalkBatch {
  using Rec = typename std::conditional<sizeof(T) == 8, RecD, RecF>::type;
  int n_in;     // tests before the end of the stretch
  double end;   // position after the last of the 32 gaps drawn
  // the lane's test
  uint32_t t;
  double at;    // position and list entry
  int j;
  int state;    // 1: a test, 0: no partner, -1: a failed check
  int y, q, O, o_start, n_o, c1, c2, cc;
  bool first;
  float pos;
  double ry, vty, inv_k_max, fflat, u;
  Rec rec;
};

// the lane's partner B.y: its state and values
template <class T>
__device__ __forceinline__ void batch_partner(const PopDev& P, int x, WalkBatch<T>& B) {
  const int y = B.y;
  if (y < 0 || y >= P.cap) {
    bad_index(P.ctr, kBadTestSlot, y);
    B.state = -1;
    return;
  }
  const uint8_t alive = P.alive[y];
  const int cell_y = P.cell[y];
  B.ry = P.rad[y];
  B.vty = P.vtot[y];
  if constexpr (sizeof(T) == 8) B.rec = P.recd[y];
  else B.rec = P.recf[y];
  B.state = y == x || !alive || cell_y != B.O ? 0 : 1;
}

// a partner that the chain has absorbed is drawn again (see walk_test)
template <class T>
__device__ __forceinline__ void batch_redraw(const PopDev& P, int x, WalkBatch<T>& B) {
  if (!(B.y >= 0 && B.y < P.cap && is_walk_claim(P, __ldcg(&P.claim[B.y]), x))) return;
  B.y = redraw_partner(P, x, B.t, B.o_start, B.n_o);
  if (B.y == -2) B.state = 0;
  else batch_partner(P, x, B);
}

template <class T>
__device__ __forceinline__ void batch_draw(const PopDev& P, int x, const Stretch& s, uint32_t t_next, bool chain,
                                           WalkBatch<T>& B) {
  constexpr unsigned kFull = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  B.t = t_next + (uint32_t)lane;
  const U4 u = walk_draws(P, x, B.t);
  const double gap = -log(u53(u.x, u.y));
  // positions summed in test order
  double acc = s.at;
  B.n_in = 32;
  B.at = 0.0;
#pragma unroll 1
  for (int k0 = 0; k0 < 32 && B.n_in == 32; k0 += 8) {
    double g8[8];
#pragma unroll
    for (int k = 0; k < 8; k++) g8[k] = __shfl_sync(kFull, gap, k0 + k);
#pragma unroll
    for (int k = 0; k < 8; k++)
      if (B.n_in == 32) {
        acc = acc + g8[k];
        if (lane == k0 + k) B.at = acc;
        if (!(acc < s.total)) B.n_in = k0 + k;
      }
  }
  B.end = acc;
  B.j = s.j;
  B.state = 0;
  B.y = -1;
  if (lane >= B.n_in) return;
  if (B.t >= (1u << 26)) {  // far past any mean the step can ask for
    set_status(P.ctr, kErrTimeout);
    B.state = -1;
    return;
  }
  B.j = walk_pair(s, B.at);
  const double c0 = s.cum[B.j], c1 = s.cum[B.j + 1];
  const int4 ent = P.cp_ent[B.j];
  const double lam = c1 - c0;
  B.n_o = ent.w;
  B.o_start = ent.z;
  if (!(lam > 0.0) || B.n_o < 1) return;
  if (B.o_start < 0 || (long long)B.o_start + B.n_o > P.cap || ent.x < 0 || ent.x >= P.n_pairs) {
    bad_index(P.ctr, kBadPairCells, ent.x);
    B.state = -1;
    return;
  }
  B.q = ent.x;
  B.O = ent.y & ((1 << 30) - 1);
  B.first = (ent.y >> 30) & 1;
  B.pos = (float)((B.at - c0) / lam);
  B.u = u32d(u.w);
  int i = (int)(u32d(u.z) * (double)B.n_o);
  if (i >= B.n_o) i = B.n_o - 1;
  B.y = P.list[B.o_start + i];
  const PairDesc d = P.pair_desc[B.q];
  const PairState& S = P.pair[B.q];
  B.c1 = d.c1;
  B.c2 = d.c2;
  B.inv_k_max = S.inv_k_max;
  B.fflat = S.fflat;
  B.cc = S.cc;
  batch_partner(P, x, B);
  if (chain) batch_redraw(P, x, B);
}

// The first accepted test at or after lane `from` for the walking particle
// (records qxd/qxf): its lane, 32 if none is accepted (or -1 - lane for a
// failed check).  *n_tests counts the tests up to it.
template <int KT, class T, bool FLAT>
__device__ __forceinline__ int batch_first(const PopDev& P, const WalkBatch<T>& B, int from, const RecD& qxd,
                                           const RecF& qxf, long long* n_tests) {
  constexpr unsigned kFull = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  bool acc = false, warn = false, exact = false;
  const bool on = lane >= from && lane < B.n_in && B.state == 1;
  if (on) {
    PairDesc d;
    d.c1 = (int8_t)B.c1;
    d.c2 = (int8_t)B.c2;
    if constexpr (sizeof(T) == 8) {
      acc = accept_f64_rec<KT, FLAT>(P, B.first ? qxd : B.rec, B.first ? B.rec : qxd, d, B.cc, B.fflat, B.inv_k_max,
                                     B.u, &warn);
    } else {
      const float* qw = (const float*)&qxf;
      const float* py = (const float*)&B.rec;
      const float pf = pair_kernel<KT, float, FLAT>(P, B.first ? qw : py, B.first ? py : qw, B.c1, B.c2, B.cc,
                                                    (float)B.fflat, (float)P.coeff) *
                       (float)B.inv_k_max;
      if (f32_decides(pf, B.u)) {
        acc = B.u < (double)pf;
      } else {  // decided in FP64 (see f32_decides)
        const RecD qy = P.recd[B.y];
        acc = accept_f64_rec<KT, FLAT>(P, B.first ? qxd : qy, B.first ? qy : qxd, d, B.cc, B.fflat, B.inv_k_max, B.u,
                                       &warn);
        exact = true;
      }
    }
  }
  const unsigned m_end = __ballot_sync(kFull, acc || (lane >= from && lane < B.n_in && B.state < 0));
  const int stop = m_end ? __ffs(m_end) - 1 : 32;
  // the tests after the accepted one have not happened yet
  const unsigned m_cnt = __ballot_sync(kFull, on && lane <= stop);
  const unsigned m_ex = __ballot_sync(kFull, exact && lane <= stop), m_wa = __ballot_sync(kFull, warn && lane <= stop);
  *n_tests += __popc(m_cnt);
  if (lane == 0) {
    if (m_ex) add_ll(&P.ctr->exact_tests, (long long)__popc(m_ex));
    if (m_wa) add_ll(&P.ctr->kmax_warn, (long long)__popc(m_wa));
  }
  if (stop == 32) return 32;
  return __shfl_sync(kFull, B.state, stop) < 0 ? -1 - stop : stop;
}

// walk_next by a warp for one walker: the tests 32 at a time, those up to the
// first accepted one stand.  A test is a chain of about six dependent loads
// and, for some kernels, as much arithmetic (2 to 3 us), and most reject.
template <int KT, class T, bool FLAT>
__device__ __forceinline__ int walk_next_warp(const PopDev& P, int x, Stretch& s, uint32_t& t_next, const RecD& qxd,
                                              const RecF& qxf, long long* n_tests, int* y, float* pos, int* q,
                                              bool* first, double* ry, double* vty) {
  constexpr unsigned kFull = 0xffffffffu;
  for (;;) {
    WalkBatch<T> B;
    batch_draw(P, x, s, t_next, false, B);
    const int at = batch_first<KT, T, FLAT>(P, B, 0, qxd, qxf, n_tests);
    if (at < 0) return -1;
    if (at < 32) {
      t_next += (uint32_t)at + 1u;
      *y = __shfl_sync(kFull, B.y, at);
      *q = __shfl_sync(kFull, B.q, at);
      *pos = __shfl_sync(kFull, B.pos, at);
      *first = __shfl_sync(kFull, B.first ? 1 : 0, at) != 0;
      *ry = __shfl_sync(kFull, B.ry, at);
      *vty = __shfl_sync(kFull, B.vty, at);
      return 1;
    }
    if (B.n_in < 32) {
      if (s.stop >= 0) {  // a per-particle pair that takes the particle as a target
        *q = P.cp_list[s.stop];
        return 3;
      }
      return 0;  // no test left in the cell's later pairs
    }
    s.at = B.end;
    s.j = __shfl_sync(kFull, B.j, 31);
    t_next += 32u;
  }
}

// The first event of walker x from (p0, pos0): the first accepted test,
// claimed by its merge decision; an absorb (the walking particle is replaced
// by the coagulated one) is carried on as a chain by k_chain from the next
// test on.  WARP: by a warp, every lane with the same arguments.
template <int KT, class T, bool FLAT, bool WARP>
__device__ void walk(const PopDev& P, int x, int p0, float pos0, WalkOut* out) {
  const bool lead = !WARP || (threadIdx.x & 31) == 0;
  if (x < 0 || x >= P.cap || !P.alive[x]) return;
  const int C = P.cell[x];
  if (C < 0 || C >= P.n_cells) return;
  Stretch s;
  walk_stretch(P, C, p0, pos0, &s);
  const RecD qxd = P.recd[x];
  const RecF qxf = P.recf[x];
  long long n_tests = 0;
  uint32_t t_next = 0;
  int y, q;
  float pos;
  bool first;
  double ry, vty;
  int r;
  if constexpr (WARP)
    r = walk_next_warp<KT, T, FLAT>(P, x, s, t_next, qxd, qxf, &n_tests, &y, &pos, &q, &first, &ry, &vty);
  else
    r = walk_next<KT, T, FLAT>(P, x, s, t_next, qxd, qxf, false, &n_tests, &y, &pos, &q, &first, &ry, &vty);
  if (r == 0) out->done = true;
  if (r == 3) {
    out->stop = true;
    out->q = q;
  }
  if (r == 1) {
    const PairDesc d = P.pair_desc[q];
    const PairState& S = P.pair[q];
    unsigned long long key = make_key((uint32_t)q, 1u, (uint32_t)x);
    unsigned long long ck = claim_key(P, key);
    Rng gm = merge_rng(P, key);
    double rx = P.rad[x], vtx = P.vtot[x];
    const MergeDecision m = merge_decide_v(P, gm, first ? rx : ry, first ? vtx : vty, first ? ry : rx,
                                           first ? vty : vtx, d.c1, d.c2, S.cc);
    bool rm_x = first ? m.rm1 : m.rm2, rm_y = first ? m.rm2 : m.rm1;
    out->found = true;
    out->q = q;
    out->y = y;
    out->pos = pos;
    out->first_cell1 = first;
    out->dec = pack_decision(m, gm.used());
    if (lead) {
      if (m.new_group == 0) set_status(P.ctr, kErrTimeout);
      claim_slot(P, x, ck, rm_x);
      claim_slot(P, y, ck, rm_y);
    }
    out->cont = m.create && rm_x && m.new_group != 0;
    out->g_used = t_next;
  }
  if (n_tests && lead) {
    add_ll_warp(&P.ctr->tot_samp, (int)n_tests);
    add_ll_warp(&P.ctr->walk_tests, (int)n_tests);
  }
}

// A chain's event i again, for the pending event of a chain cut short: the
// decision the walk made, from the chain's stream and the particles' values
// (0xffffffff for a bad pair index)
__device__ __noinline__ uint32_t chain_event_decision(const PopDev& P, unsigned long long key, int2 sl, int x, int y,
                                                      uint32_t i) {
  const int q = (int)key_pair(key);
  if (q >= P.n_pairs) {
    bad_index(P.ctr, kBadEventSlot, q);
    return 0xffffffffu;
  }
  const PairDesc d = P.pair_desc[q];
  const PairState& S = P.pair[q];
  Rng g = make_rng(P, kStreamChain, i + 1u, (uint32_t)x);
  const int s1 = sl.x == x ? x : y, s2 = sl.x == x ? y : x;
  MergeDecision m = merge_decide_v(P, g, P.rad[s1], P.vtot[s1], P.rad[s2], P.vtot[s2], d.c1, d.c2, S.cc);
  if (m.new_group == 0) set_status(P.ctr, kErrTimeout);
  return pack_decision(m, g.used());
}

// A target operation for particle x at per-particle pair q (its walk reached
// the pair with x in the pair's target cell), at place k of the round's
// operations: after the redone ones, at the item's own index, so that the
// list's order does not depend on scheduling (the places of items without
// one hold population -1 and are dropped when the list is grouped).  It runs
// in this round; its key puts it after the pair's own operations.
__device__ __noinline__ void add_target_op(const PopDev& P, int pop, int q, int x, int* op_pop, int* op_pair,
                                              int* op_slot, int* op_k, unsigned long long* op_key, long long k,
                                              long long op_cap) {
  if (k >= op_cap) {
    cap_fail(P.ctr, kCapTargetOps);
    return;
  }
  op_pop[k] = pop;
  op_pair[k] = q;
  op_slot[k] = x;
  op_k[k] = 0x40000000 | x;  // its own stream: round-0 operations count from 0, redos add 1 << 24
  op_key[k] = make_key((uint32_t)q, 1u, (uint32_t)x);
}

// Walks, or chains, per warp of the launch up to which each takes a warp; with
// more, each takes a thread.  A launch ends with its longest walk, and a
// warp's takes about as long as two tests of a thread's; but a warp each in
// several waves (4 walks a warp: 25 us for the first later round of 1e6
// particles) is slower than 32 walks a warp (22 us).
constexpr int kWarpShare = 1;

// what a later round's kernels read of the round before and write for this one
struct ItemArgs {
  const PopDev* pops;
  const int *gpair_pop, *gpair_local;
  const long long* pop_pair_base;
  int n_gpairs;
  const long long *n_items, *n_items_ev;
  const int *ppw_slot, *ppw_gp;
  int *op_pop, *op_pair, *op_slot, *op_k;
  unsigned long long* op_key;
  const long long* n_ops;
  long long op_cap;
  const uint8_t* win;
  const int* dest;
  const unsigned long long* ev_key;
  const int2* ev_c;
  const int* gp_c;
  const float* ev_pos;
  const uint32_t* dec;
  uint8_t* it_flag;
  unsigned long long* it_key;
  int2* it_c;
  int* it_gp;
  float* it_pos;
  int *it_len, *it_head;
  uint8_t* it_done;
  uint32_t *it_dec, *it_gused;
  int4* it_term;
  int* start_list;      // items whose walk k_chain carries on
  long long* n_start;
};

// The work of a later round, per event e of the round before:
//   - a winner that created or changed a particle (dest[e] >= 0): that
//     particle walks from the event's pair and position (for a chain, its
//     last applied event's);
//   - a loser: consumed = removed or rewritten in the round before
//     (touched), or dead.  A sample (kind 0) is retried with its key if
//     neither particle was consumed, else dropped.  A walk's test (kind 1,
//     a chain's first event): dropped if the walking particle was consumed,
//     the walk resumed after the test if only the partner was, else retried
//     alone.
// Output per e: flag, and key, slots, global pair and position of the new
// event (for a chain its first event) with the chain's length and head; the
// new event holds claims on its slots.
template <int KT, class T, bool FLAT, bool WARP>
__device__ __forceinline__ void do_item(const ItemArgs& A, long long e, long long n_ev, long long op_base) {
  const bool lead = !WARP || (threadIdx.x & 31) == 0;
  if (lead) {
    A.it_flag[e] = 0;
    A.it_term[e] = no_term();
    if (A.op_cap > 0 && op_base + e < A.op_cap) A.op_pop[op_base + e] = -1;
  }
  int gp, walker = -1, p0 = 0;
  float pos0 = 1.0f;
  unsigned long long key = 0;
  int2 sl = make_int2(-1, -1);
  uint32_t dc = 0;
  if (e >= n_ev) {
    // a particle that a target operation of the round before made or
    // changed walks from the end of that operation's pair
    gp = A.ppw_gp[e - n_ev];
    if (gp < 0 || gp >= A.n_gpairs) {
      if (lead) bad_index(A.pops[0].ctr, kBadEventSlot, gp);
      return;
    }
    walker = A.ppw_slot[e - n_ev];
    p0 = A.gpair_local[gp];
  } else {
    gp = A.gp_c[e];
    if (gp < 0 || gp >= A.n_gpairs) {
      if (lead) bad_index(A.pops[0].ctr, kBadEventSlot, gp);
      return;
    }
    const PopDev& P = A.pops[A.gpair_pop[gp]];
    uint32_t pend_dec = 0xffffffffu;  // a pending chain event's recomputed decision
    pos0 = A.ev_pos[e];
    key = A.ev_key[e];
    sl = A.ev_c[e];
    const bool won = A.win[e] != 0;
    const int dst = A.dest[e];
    const bool in = !(sl.x < 0 || sl.x >= P.cap || sl.y < 0 || sl.y >= P.cap);
    if (won && (dst == kPendingTerm || dst == kPendingChain)) {
      // the test where the previous round's chain stopped, with its
      // decision: the walker was rewritten by its own chain, so only its
      // death counts; a partner consumed in that round is no member now,
      // and the walk goes on after the test
      if (!in) {
        if (lead) bad_index(P.ctr, kBadEventSlot, sl.x < 0 || sl.x >= P.cap ? sl.x : sl.y);
        return;
      }
      const int x = (int)key_idx(key), y = x == sl.x ? sl.y : sl.x;
      if (!P.alive[x]) return;
      if (P.touched[y] == *P.gen_p - 1u || !P.alive[y]) {
        walker = x;
        p0 = (int)key_pair(key);
      } else if (dst == kPendingChain) {
        pend_dec = chain_event_decision(P, key, sl, x, y, A.dec[e]);
        if (pend_dec == 0xffffffffu) return;
      }
    } else if (won) {
      walker = dst;
      p0 = A.gpair_local[gp];
      if (walker < 0) return;
    } else {
      if (!in) {
        if (lead) bad_index(P.ctr, kBadEventSlot, sl.x < 0 || sl.x >= P.cap ? sl.x : sl.y);
        return;
      }
      uint32_t gen_prev = *P.gen_p - 1u;
      bool c1 = P.touched[sl.x] == gen_prev || !P.alive[sl.x];
      bool c2 = P.touched[sl.y] == gen_prev || !P.alive[sl.y];
      if (key_kind(key) == 0u) {
        if (c1 || c2) return;
      } else {
        int x = (int)key_idx(key);
        bool cx = x == sl.x ? c1 : c2, cy = x == sl.x ? c2 : c1;
        if (cx) return;
        if (cy) {
          walker = x;
          p0 = (int)key_pair(key);
        }
      }
    }
    dc = pend_dec != 0xffffffffu ? pend_dec : A.dec[e];
  }
  const int pop = A.gpair_pop[gp];
  const PopDev& P = A.pops[pop];
  int len = 0;
  bool done = false;
  if (walker >= 0) {
    WalkOut w;
    walk<KT, T, FLAT, WARP>(P, walker, p0, pos0, &w);
    if (w.stop && lead)
      add_target_op(P, pop, w.q, walker, A.op_pop, A.op_pair, A.op_slot, A.op_k, A.op_key, op_base + e, A.op_cap);
    if (!w.found) return;
    key = make_key((uint32_t)w.q, 1u, (uint32_t)walker);
    sl = w.first_cell1 ? make_int2(walker, w.y) : make_int2(w.y, walker);
    gp = (int)(A.pop_pair_base[pop] + w.q);
    pos0 = w.pos;
    done = w.done;
    dc = w.dec;
    if (w.cont) {
      len = -1;  // k_chain carries the walk on
      if (lead) {
        A.it_gused[e] = w.g_used;
        A.start_list[inc_warp((unsigned long long*)A.n_start)] = (int)e;
      }
    }
  } else if (lead) {
    // a retry keeps its merge decision and claims by it
    uint32_t used;
    MergeDecision m = unpack_decision(dc, &used);
    unsigned long long ck = claim_key(P, key);
    claim_slot(P, sl.x, ck, m.rm1);
    claim_slot(P, sl.y, ck, m.rm2);
  }
  if (lead) {
    A.it_flag[e] = 1;
    A.it_key[e] = key;
    A.it_c[e] = sl;
    A.it_gp[e] = gp;
    A.it_pos[e] = pos0;
    A.it_len[e] = len;
    A.it_head[e] = -1;
    A.it_done[e] = done ? 1 : 0;
    A.it_dec[e] = dc;
  }
}

// A warp per item while the launch has the warps for it, else a thread.  Bound
// by the longest walk's tests, one after another (57 us a launch for 4000
// sedimenting drops in FP64, now 20), and below about 7 us by the item's own
// dependent loads and the kernel's cold instructions.
template <int KT, class T, bool FLAT>
__global__ void __launch_bounds__(256) k_items(ItemArgs A) {
  chain_wait();
  const long long n = *A.n_items, n_ev = *A.n_items_ev;
  const long long op_base = A.op_cap > 0 ? *A.n_ops : 0;  // the redone operations come first
  const long long tid = blockIdx.x * (long long)blockDim.x + threadIdx.x, nt = (long long)gridDim.x * blockDim.x;
  if (n <= kWarpShare * (nt >> 5)) {
    for (long long e = tid >> 5; e < n; e += nt >> 5) do_item<KT, T, FLAT, true>(A, e, n_ev, op_base);
  } else {
    for (long long e = tid; e < n; e += nt) do_item<KT, T, FLAT, false>(A, e, n_ev, op_base);
  }
}

// Chains, after k_items: an item whose first event is an absorb (it_len -1,
// listed) carries its walk on from that event with the coagulated particle,
// drawing the walk's tests on from where k_items stopped.
// The coagulated particle's volumes are summed per species over the events,
// then over the species, as k_apply_chain sums them, so its decisions are
// the apply's.  While the particle stays in the cell it walked, the walk goes
// on in place; a new cell's stretch starts at the event's pair and position.
// The next accepted test is the next event: an absorb extends the chain, any
// other decision ends the chain before it (the walk resumes there in the
// next round).  The chain's events go to the pool, the first one included;
// the item gets the chain's length and head, or length 0 (the first event
// alone) if the pool is full.
template <int KT, class T, bool FLAT>
__device__ __forceinline__ void do_chain(const ItemArgs& A, const ChainPool& pool, long long e) {
  if (!A.it_flag[e] || A.it_len[e] != -1) return;
  const PopDev& P = A.pops[A.gpair_pop[A.it_gp[e]]];
  unsigned long long key = A.it_key[e];
  const int x = (int)key_idx(key);
  int q = (int)key_pair(key);
  int2 sl = A.it_c[e];
  int y = sl.x == x ? sl.y : sl.x;
  uint32_t used;
  MergeDecision m1 = unpack_decision(A.it_dec[e], &used);
  bool rm_y1 = sl.x == x ? m1.rm2 : m1.rm1;
  A.it_len[e] = 0;
  if (x < 0 || x >= P.cap || y < 0 || y >= P.cap || q >= P.n_pairs) return;
  ChainWriter cw;
  float pos = A.it_pos[e];
  if (!cw.append(pool, y, q | (rm_y1 ? kChainRemoves : 0), pos)) return;
  uint32_t t_next = A.it_gused[e];
  long long n_tests = 0;
  bool done = false;
  const int ns = P.n_spec;
  double vcur[kMaxSpec];
  for (int sp = 0; sp < ns; sp++) vcur[sp] = P.vol[vol_at(P, x, sp)];
  int cls = P.pair[q].cc + 1;
  Stretch s;
  s.C = -1;
  for (;;) {
    // absorb y: the coagulated particle's volumes, radius, class, record
    for (int sp = 0; sp < ns; sp++) vcur[sp] = vcur[sp] + P.vol[vol_at(P, y, sp)];
    double s_v = 0.0, s_m = 0.0;
    for (int sp = 0; sp < ns; sp++) s_v = s_v + vcur[sp];
    for (int sp = 0; sp < ns; sp++) s_m = s_m + vcur[sp] * P.density[sp];
    const double vt = s_v, r = vol2rad(P.benv.frac, vt);
    const RecD qxd = make_rec_v(P, r, vt, s_m, cls);
    const RecF qxf = to_f32(qxd);
    const int C = cell_of(P, r, cls);
    if (C < 0 || cw.len >= kChainMaxLen) break;  // off the grid (reported by the apply) or long enough
    if (C != s.C) walk_stretch(P, C, q, pos, &s);
    int yy, qq;
    bool first;
    double ry, vty;
    int rw = walk_next<KT, T, FLAT>(P, x, s, t_next, qxd, qxf, true, &n_tests, &yy, &pos, &qq, &first, &ry, &vty);
    if (rw == 0) done = true;  // every later pair of the cell was walked
    if (rw != 1) break;
    const PairDesc d = P.pair_desc[qq];
    const PairState& S = P.pair[qq];
    unsigned long long k2 = make_key((uint32_t)qq, 1u, (uint32_t)x);
    Rng gm = make_rng(P, kStreamChain, (uint32_t)(cw.len + 1), (uint32_t)x);
    const MergeDecision m = merge_decide_v(P, gm, first ? r : ry, first ? vt : vty, first ? ry : r,
                                           first ? vty : vt, d.c1, d.c2, S.cc);
    bool rm_x = first ? m.rm1 : m.rm2, rm_y = first ? m.rm2 : m.rm1;
    // the chain ends before an event that is no absorb, or when the pool
    // is full; that event is pending for the next round (kPendingTerm)
    if (!(m.create && rm_x && m.new_group != 0) || !cw.append(pool, yy, qq | (rm_y ? kChainRemoves : 0), pos)) {
      if (m.new_group == 0) set_status(P.ctr, kErrTimeout);
      A.it_term[e] = make_int4(yy, qq | (first ? kTermFirst : 0), (int)pack_decision(m, gm.used()),
                               __float_as_int(pos));
      break;
    }
    claim_slot(P, yy, claim_key(P, k2), rm_y);
    y = yy;
    q = qq;
    cls = S.cc + 1;
  }
  // a chain that ended at its first event is that event alone
  A.it_len[e] = cw.len > 1 ? cw.len : 0;
  A.it_head[e] = cw.head;
  A.it_done[e] = done ? 1 : 0;
  if (n_tests) {
    add_ll_warp(&P.ctr->tot_samp, (int)n_tests);
    add_ll_warp(&P.ctr->walk_tests, (int)n_tests);
  }
}

// do_chain by a warp, the same events from the same draws: 32 tests at a time
// (WalkBatch).  What is left in sequence per absorb is the coagulated
// particle's radius, record and cell and the acceptance of the tests already
// drawn; its radius and the decision's are one vol2rad call, on two lanes.
// vs: 2 x kMaxSpec doubles of the warp's shared memory (the walking
// particle's volumes, and those with the partner's added).
template <int KT, class T, bool FLAT>
__device__ __forceinline__ void do_chain_warp(const ItemArgs& A, const ChainPool& pool, long long e, double* vs) {
  constexpr unsigned kFull = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const bool lead = lane == 0;
  if (!A.it_flag[e] || A.it_len[e] != -1) return;
  const PopDev& P = A.pops[A.gpair_pop[A.it_gp[e]]];
  const unsigned long long key = A.it_key[e];
  const int x = (int)key_idx(key);
  int q = (int)key_pair(key);
  const int2 sl = A.it_c[e];
  int y = sl.x == x ? sl.y : sl.x;
  uint32_t used;
  const MergeDecision m1 = unpack_decision(A.it_dec[e], &used);
  const bool rm_y1 = sl.x == x ? m1.rm2 : m1.rm1;
  float pos = A.it_pos[e];
  uint32_t t_next = A.it_gused[e];
  __syncwarp();  // every lane has read the item
  if (lead) A.it_len[e] = 0;
  if (x < 0 || x >= P.cap || y < 0 || y >= P.cap || q >= P.n_pairs) return;
  ChainWriter cw;
  // the lead's append, its result for every lane (len counts on all of them)
  auto append = [&](int yy, int qw, float ps) {
    bool ok = true;
    const int len = cw.len;
    if (lead) ok = cw.append(pool, yy, qw, ps);
    ok = __shfl_sync(kFull, ok ? 1 : 0, 0) != 0;
    cw.len = ok ? len + 1 : len;
    return ok;
  };
  if (!append(y, q | (rm_y1 ? kChainRemoves : 0), pos)) return;
  long long n_tests = 0;
  bool done = false;
  const int ns = P.n_spec;
  const bool flat1 = one_flat_weight(P);
  double* vcur = vs;
  double* vnew = vs + kMaxSpec;
  for (int sp = lane; sp < ns; sp += 32) vcur[sp] = P.vol[vol_at(P, x, sp)] + P.vol[vol_at(P, y, sp)];
  int cls = P.pair[q].cc + 1;
  // total volume and mass of v, in species order
  auto totals = [&](const double* v, double* s_v, double* s_m) {
    __syncwarp();
    double a = 0.0, b = 0.0;
    for (int sp = 0; sp < ns; sp++) {
      const double z = v[sp];
      a = a + z;
      b = b + z * P.density[sp];
    }
    *s_v = a;
    *s_m = b;
  };
  double vt, ms;
  totals(vcur, &vt, &ms);
  double r = vol2rad(P.benv.frac, vt);
  Stretch s;
  s.C = -1;
  WalkBatch<T> B;
  int from = 32;  // lane of the batch's next test (32: none left)
  B.n_in = 32;
  for (;;) {
    const RecD qxd = make_rec_v(P, r, vt, ms, cls);
    const RecF qxf = to_f32(qxd);
    const int C = cell_of(P, r, cls);
    if (C < 0 || cw.len >= kChainMaxLen) break;  // off the grid (reported by the apply) or long enough
    if (C != s.C) {
      walk_stretch(P, C, q, pos, &s);
      from = 32;
      B.n_in = 32;
    }
    // the next accepted test
    int at;
    for (;;) {
      if (from >= 32) {
        batch_draw(P, x, s, t_next, true, B);
        from = 0;
      }
      at = batch_first<KT, T, FLAT>(P, B, from, qxd, qxf, &n_tests);
      if (at != 32 || B.n_in < 32) break;
      s.at = B.end;
      s.j = __shfl_sync(kFull, B.j, 31);
      t_next = __shfl_sync(kFull, B.t, 31) + 1u;
      from = 32;
    }
    if (at == 32) done = s.stop < 0;  // every later pair of the cell was walked
    if (at < 0 || at == 32) break;
    t_next = __shfl_sync(kFull, B.t, at) + 1u;
    s.at = __shfl_sync(kFull, B.at, at);
    s.j = __shfl_sync(kFull, B.j, at);
    from = at + 1;
    const int yy = __shfl_sync(kFull, B.y, at), qq = __shfl_sync(kFull, B.q, at);
    const int c1 = __shfl_sync(kFull, B.c1, at), c2 = __shfl_sync(kFull, B.c2, at);
    const int cc = __shfl_sync(kFull, B.cc, at);
    const bool first = __shfl_sync(kFull, B.first ? 1 : 0, at) != 0;
    const double ry = __shfl_sync(kFull, B.ry, at), vty = __shfl_sync(kFull, B.vty, at);
    pos = __shfl_sync(kFull, B.pos, at);
    for (int sp = lane; sp < ns; sp += 32) vnew[sp] = vcur[sp] + P.vol[vol_at(P, yy, sp)];
    double vt2, ms2;
    totals(vnew, &vt2, &ms2);
    const double r1 = first ? r : ry, r2 = first ? ry : r;
    const double rr = vol2rad(P.benv.frac, lane == 1 && !flat1 ? merge_vol(P, r1, r2) : vt2);
    const double rnew = __shfl_sync(kFull, rr, 0), rc = __shfl_sync(kFull, rr, 1);
    Rng gm = make_rng(P, kStreamChain, (uint32_t)(cw.len + 1), (uint32_t)x);
    const MergeDecision m = merge_decide_rc(P, gm, r1, first ? vt : vty, r2, first ? vty : vt, c1, c2, cc, rc);
    const bool rm_x = first ? m.rm1 : m.rm2, rm_y = first ? m.rm2 : m.rm1;
    // the chain ends before an event that is no absorb, or when the pool
    // is full; that event is pending for the next round (kPendingTerm)
    if (!(m.create && rm_x && m.new_group != 0) || !append(yy, qq | (rm_y ? kChainRemoves : 0), pos)) {
      if (lead) {
        if (m.new_group == 0) set_status(P.ctr, kErrTimeout);
        A.it_term[e] = make_int4(yy, qq | (first ? kTermFirst : 0), (int)pack_decision(m, gm.used()),
                                 __float_as_int(pos));
      }
      break;
    }
    if (lead) claim_slot(P, yy, claim_key(P, make_key((uint32_t)qq, 1u, (uint32_t)x)), rm_y);
    __syncwarp();  // the claim is seen by the other lanes
    if (lane >= from && lane < B.n_in && B.state != -1 && B.y == yy) batch_redraw(P, x, B);
    q = qq;
    cls = cc + 1;
    double* v = vcur;
    vcur = vnew;
    vnew = v;
    vt = vt2;
    ms = ms2;
    r = rnew;
  }
  if (lead) {
    // a chain that ended at its first event is that event alone
    A.it_len[e] = cw.len > 1 ? cw.len : 0;
    A.it_head[e] = cw.head;
    A.it_done[e] = done ? 1 : 0;
    if (n_tests) {
      add_ll(&P.ctr->tot_samp, n_tests);
      add_ll(&P.ctr->walk_tests, n_tests);
    }
  }
}

// Bound by the longest chain: about 5 us an absorb for one thread, its FP64
// pow, log and exp calls one after another; by a warp 1.5 (37,000 sedimenting
// drops: 102 us a launch, now 34; 4000 in FP64: 57 and 33).
constexpr int kChainThreads = 128;
template <int KT, class T, bool FLAT>
__global__ void __launch_bounds__(kChainThreads, 4) k_chain(ItemArgs A, ChainPool pool) {
  chain_wait();
  __shared__ double sh_v[kChainThreads / 32][2 * kMaxSpec];
  const long long n = *A.n_start;
  const long long tid = blockIdx.x * (long long)blockDim.x + threadIdx.x, nt = (long long)gridDim.x * blockDim.x;
  if (n <= kWarpShare * (nt >> 5)) {
    for (long long ci = tid >> 5; ci < n; ci += nt >> 5) {
      do_chain_warp<KT, T, FLAT>(A, pool, A.start_list[ci], sh_v[threadIdx.x >> 5]);
      __syncwarp();
    }
  } else {
    // by item, not by the list: the chains then lie spread over the warps,
    // and few of a warp's threads wait for one another
    const long long n_it = *A.n_items;
    for (long long e = tid; e < n_it; e += nt) do_chain<KT, T, FLAT>(A, pool, e);
  }
}

// Apply the winning chains (win[e] == 2), one warp per chain: the first
// ev_app[e] events in order, each a coagulate (coagulation.F90:928-985) of
// the walking particle with the next partner, with the merge decision
// recomputed from the values and the stream the walk used.  One warp per
// chain of the round's list (chain_list, filled by k_resolve); a chain's entries
// are taken a pool chunk at a time (kBatch events):
//   1. lane k loads event k's partner (slot, pair, radius, scalar fields,
//      species volumes) into shared memory;
//   2. lane s runs species s's sum over the events (the walking particle's
//      volume plus the partners' in order), keeping the sum after each event;
//   3. lane k totals event k's sums over the species (the walk's order, so
//      the values and decisions are the walk's), takes the radius and cell,
//      and draws event k's merge decision from the particle before event k;
//   4. the events' scalar fields and components are merged in order (lanes
//      hold components), and removed partners are killed.
// The coagulated particle stays in the walking particle's slot.  dest[e],
// gp_c[e] and ev_pos[e] are set to where the particle walks on (dest -1 if
// its walk ran to the end).
struct ChainStage {
  int y, q, cell1, cc;
  int c1, c2;
  float pos;
  int pad;
  double ry, vty, ice_y;
  PScal s;
};
constexpr int kApplyBatch = kChainChunk - 1;

__global__ void __launch_bounds__(32) k_apply_chain(const PopDev* pops, const int* gpair_pop,
                                                    const long long* pop_pair_base, const int* chain_list,
                                                    const long long* n_chain, const unsigned long long* ev_key,
                                                    const int* ev_len, const int* ev_app, const int* ev_head,
                                                    const uint8_t* ev_done, ChainPool pool, int* gp_c, float* ev_pos,
                                                    int* dest_out, unsigned long long* ev_key_w, int2* ev_w,
                                                    uint32_t* dec_w, const int4* ev_term) {
  constexpr unsigned kFull = 0xffffffffu;
  constexpr int kBatch = kApplyBatch;
  __shared__ ChainStage stage[kBatch];
  __shared__ double pre[kBatch * kMaxSpec];  // [event][species]
  __shared__ double ubuf[64];                // draws of a component selection
  const long long n_ch = *n_chain;
  const int lane = threadIdx.x;
  for (long long ci = blockIdx.x; ci < n_ch; ci += gridDim.x) {
    {
      const long long e = chain_list[ci];
      int pop = gpair_pop[gp_c[e]];
      const PopDev& P = pops[pop];
      unsigned long long key1 = ev_key[e];
      int x = (int)key_idx(key1);
      int app = ev_app[e];
      if (lane == 0) dest_out[e] = -1;
      if (x < 0 || x >= P.cap) {
        if (lane == 0) bad_index(P.ctr, kBadEventSlot, x);
        continue;
      }
      const int nb = P.grid->n_bin, ns = P.n_spec;
      const int w_ice = P.i_water - 1;  // -1: no water species
      uint32_t gen = *P.gen_p;
      // the walking particle: species (lane, lane + 32), scalars, components (lane)
      double v_lo = lane < ns ? P.vol[vol_at(P, x, lane)] : 0.0;
      double v_hi = lane + 32 < ns ? P.vol[vol_at(P, x, lane + 32)] : 0.0;
      double ice_cur = w_ice >= 0 ? P.vol[vol_at(P, x, w_ice)] : 0.0;
      PScal cur;
      load_scal(P, x, cur);
      int cc_ = 0;
      double ct_ = 0.0;
      if (lane < cur.ncomp && lane < kMaxComponent) {
        cc_ = P.csrc[comp_at(x, lane)];
        ct_ = P.ctime[comp_at(x, lane)];
      }
      double r = P.rad[x], vt = P.vtot[x];
      int C = P.cell[x];
      int chunk = ev_head[e];
      int done_ev = 0, last_q = -1, dlive = 0;
      float last_pos = 0.f;
      bool stop = false;
      for (int base = 0; base < app && !stop; base += kBatch) {
        const int nbatch = app - base < kBatch ? app - base : kBatch;
        // 1. the chunk's partners, one lane each
        const bool chunk_ok = chunk >= 0 && (long long)chunk < pool.n_chunks;  // the same on every lane
        bool bad = !chunk_ok;
        if (chunk_ok && lane < nbatch) {
          size_t ix = (size_t)chunk * kChainChunk + lane;
          int y = pool.y[ix];
          int q = pool.q[ix] & kChainPairMask;
          bad = y < 0 || y >= P.cap || q >= P.n_pairs;
          if (!bad) {
            ChainStage& st = stage[lane];
            const PairDesc d = P.pair_desc[q];
            st.y = y;
            st.q = q;
            st.cell1 = d.b1 + nb * d.c1;
            st.c1 = d.c1;
            st.c2 = d.c2;
            st.cc = P.pair[q].cc;
            st.pos = pool.pos[ix];
            st.ry = P.rad[y];
            st.vty = P.vtot[y];
            st.ice_y = w_ice >= 0 ? P.vol[vol_at(P, y, w_ice)] : 0.0;
            load_scal(P, y, st.s);
            for (int sp = 0; sp < ns; sp++) pre[lane * kMaxSpec + sp] = P.vol[vol_at(P, y, sp)];
          }
        }
        // entries past the first bad one are not applied
        const unsigned bad_mask = __ballot_sync(kFull, bad && lane < nbatch);
        const int n_ok = bad_mask ? __ffs(bad_mask) - 1 : nbatch;
        if (chunk_ok) chunk = pool.y[(size_t)chunk * kChainChunk + kChainChunk - 1];
        __syncwarp();
        // 2. per species, the sums after each event
        const double v_lo0 = v_lo, v_hi0 = v_hi;
        for (int k = 0; k < n_ok; k++) {
          if (lane < ns) {
            v_lo = v_lo + pre[k * kMaxSpec + lane];
            pre[k * kMaxSpec + lane] = v_lo;
          }
          if (lane + 32 < ns) {
            v_hi = v_hi + pre[k * kMaxSpec + lane + 32];
            pre[k * kMaxSpec + lane + 32] = v_hi;
          }
        }
        __syncwarp();
        // 3. per event: total, radius, cell, merge decision
        double vt_k = 0.0, r_k = 0.0;
        int C_k = -1;
        if (lane < n_ok) {
          double s_v = 0.0;
          for (int sp = 0; sp < ns; sp++) s_v = s_v + pre[lane * kMaxSpec + sp];
          vt_k = s_v;
          r_k = vol2rad(P.benv.frac, vt_k);
          C_k = cell_of(P, r_k, stage[lane].cc + 1);
        }
        double r_b = __shfl_up_sync(kFull, r_k, 1), vt_b = __shfl_up_sync(kFull, vt_k, 1);
        int C_b = __shfl_up_sync(kFull, C_k, 1);
        if (lane == 0) {
          r_b = r;
          vt_b = vt;
          C_b = C;
        }
        bool ok = true, first_k = false, rm_y_k = false, lost_x_k = false, lost_y_k = false;
        int group_k = 0;
        uint32_t used_k = 0;
        if (lane < n_ok) {
          const ChainStage& st = stage[lane];
          first_k = C_b == st.cell1;
          const int i = base + lane;
          Rng g = i == 0 ? merge_rng(P, key1) : make_rng(P, kStreamChain, (uint32_t)(i + 1), (uint32_t)x);
          const MergeDecision m = merge_decide_v(P, g, first_k ? r_b : st.ry, first_k ? vt_b : st.vty,
                                                 first_k ? st.ry : r_b, first_k ? st.vty : vt_b, st.c1, st.c2, st.cc);
          bool rm_x = first_k ? m.rm1 : m.rm2;
          rm_y_k = first_k ? m.rm2 : m.rm1;
          lost_x_k = first_k ? m.lost1 : m.lost2;
          bool lost_y = first_k ? m.lost2 : m.lost1;
          lost_y_k = rm_y_k && lost_y;
          ok = m.create && rm_x && m.new_group != 0 && !(lost_x_k && !(rm_y_k && !lost_y));
          group_k = m.new_group;
          used_k = g.used();
        }
        const unsigned bad_dec = __ballot_sync(kFull, lane < n_ok && !ok);
        const int n_app = bad_dec ? __ffs(bad_dec) - 1 : n_ok;
        if (bad_dec) {
          if (lane == 0) set_status(P.ctr, kErrAssert);  // the walk decided an absorb here
          stop = true;
        }
        // 4. scalar fields and components, in order
        int yc = 0;
        double yt = 0.0;
        if (n_app > 0 && lane < stage[0].s.ncomp && lane < kMaxComponent) {
          yc = P.csrc[comp_at(stage[0].y, lane)];
          yt = P.ctime[comp_at(stage[0].y, lane)];
        }
        for (int k = 0; k < n_app; k++) {
          const ChainStage& st = stage[k];
          // the next partner's components, loaded ahead
          int yc_n = 0;
          double yt_n = 0.0;
          if (k + 1 < n_app && lane < stage[k + 1].s.ncomp && lane < kMaxComponent) {
            yc_n = P.csrc[comp_at(stage[k + 1].y, lane)];
            yt_n = P.ctime[comp_at(stage[k + 1].y, lane)];
          }
          const bool first = __shfl_sync(kFull, first_k ? 1 : 0, k) != 0;
          const bool rm_y = __shfl_sync(kFull, rm_y_k ? 1 : 0, k) != 0;
          const bool lost_x = __shfl_sync(kFull, lost_x_k ? 1 : 0, k) != 0;
          const bool lost_y = __shfl_sync(kFull, lost_y_k ? 1 : 0, k) != 0;
          const int new_group = __shfl_sync(kFull, group_k, k);
          const uint32_t used = __shfl_sync(kFull, used_k, k);
          const PScal ys = st.s;
          const double ice_x = k == 0 ? ice_cur : (w_ice >= 0 ? pre[(k - 1) * kMaxSpec + w_ice] : 0.0);
          const double ice_y = st.ice_y;
          // components of aero_particle_coagulate with a = particle 1, b = particle 2
          const PScal& A = first ? cur : ys;
          const PScal& B = first ? ys : cur;
          int ca = first ? cc_ : yc, cb = first ? yc : cc_;
          double ta = first ? ct_ : yt, tb = first ? yt : ct_;
          int na = A.ncomp, nbc = B.ncomp;
          int n1_new = na, n2_new = nbc;
          bool from_a = lane < na;
          int k_src = from_a ? lane : lane - na;
          if (na + nbc > kMaxComponent) {
            const int i = base + k;
            const Rng g = i == 0 ? merge_rng(P, key1) : make_rng(P, kStreamChain, (uint32_t)(i + 1), (uint32_t)x);
            uint32_t at = used;
            warp_coag_components(g, &at, ubuf, na, A.nprim, nbc, B.nprim, &n1_new, &n2_new, &from_a, &k_src);
          }
          k_src &= 31;
          int xa = __shfl_sync(kFull, ca, k_src), xb = __shfl_sync(kFull, cb, k_src);
          double za = __shfl_sync(kFull, ta, k_src), zb = __shfl_sync(kFull, tb, k_src);
          int n_out = n1_new + n2_new;
          PScal nm;
          coag_scalars(A, first ? ice_x : ice_y, B, first ? ice_y : ice_x, nm);
          nm.ncomp = n_out;
          nm.id = !lost_x ? cur.id : ys.id;
          // the removals of this event whose ID is lost (coagulate,
          // coagulation.F90:928-985): the walking particle's is always removed
          if (lane == 0) {
            if (lost_x) log_removal(P, cur.id, kInfoCoag, nm.id);
            if (lost_y) log_removal(P, ys.id, kInfoCoag, nm.id);
          }
          nm.grp = new_group;
          nm.cls = st.cc + 1;
          cc_ = lane < n_out ? (from_a ? xa : xb) : 0;
          ct_ = lane < n_out ? (from_a ? za : zb) : 0.0;
          if (rm_y) {
            if (lane == 0) {
              kill_slot(P, st.y);
              P.touched[st.y] = gen;
            }
            dlive--;
          }
          cur = nm;
          done_ev++;
          last_q = st.q;
          last_pos = st.pos;
          yc = yc_n;
          yt = yt_n;
        }
        // the particle after the batch's last applied event
        if (n_app > 0) {
          r = __shfl_sync(kFull, r_k, n_app - 1);
          vt = __shfl_sync(kFull, vt_k, n_app - 1);
          C = __shfl_sync(kFull, C_k, n_app - 1);
          v_lo = lane < ns ? pre[(n_app - 1) * kMaxSpec + lane] : 0.0;
          v_hi = lane + 32 < ns ? pre[(n_app - 1) * kMaxSpec + lane + 32] : 0.0;
          if (w_ice >= 0) ice_cur = pre[(n_app - 1) * kMaxSpec + w_ice];
        } else {
          v_lo = v_lo0;
          v_hi = v_hi0;
        }
        if (n_ok < nbatch && !stop) {
          if (lane == 0) bad_index(P.ctr, kBadEventSlot, -1);
          stop = true;
        }
        __syncwarp();  // the stage is read before the next chunk overwrites it
      }
      if (done_ev == 0) continue;
    // the coagulated particle in the walking particle's slot
    __syncwarp();
    if (lane < ns) P.vol[vol_at(P, x, lane)] = v_lo;
    if (lane + 32 < ns) P.vol[vol_at(P, x, lane + 32)] = v_hi;
    if (lane < cur.ncomp && lane < kMaxComponent) {
      P.csrc[comp_at(x, lane)] = cc_;
      P.ctime[comp_at(x, lane)] = ct_;
    }
    double ms = 0.0;
    for (int s = 0; s < ns; s++)
      ms = ms + __shfl_sync(kFull, s < 32 ? v_lo : v_hi, s & 31) * P.density[s];
    if (lane == 0) {
      P.vtot[x] = vt;
      P.mass[x] = ms;
      P.grp[x] = cur.grp;
      P.cls[x] = cur.cls;
      P.id[x] = cur.id;
      P.nprim[x] = cur.nprim;
      P.ncomp[x] = cur.ncomp;
      P.lct[x] = cur.lct;
      P.gct[x] = cur.gct;
      P.imf[x] = cur.imf;
      P.den_ice[x] = cur.den_ice;
      P.phi[x] = cur.phi;
      P.hyst[x] = cur.hyst;
      P.frozen[x] = cur.frozen;
      P.alive[x] = 1;
      P.changed[x] = 1;
      P.touched[x] = gen;
      int nbin = refresh_slot(P, x);
      bool on_grid = nbin >= 1 && nbin <= nb;
      if (!on_grid) set_status(P.ctr, kErrOutOfGrid);
      add_ll(&P.ctr->tot_coag, (long long)done_ev);
      if (dlive) add_ll(&P.ctr->n_live, (long long)dlive);
      bool walk_done = ev_done[e] && done_ev == ev_len[e];
      const int4 t = ev_term[e];
      if (on_grid && done_ev == ev_len[e] && t.x >= 0) {
        // every event applied: the test where the chain stopped is pending
        const int tq = t.y & (kTermFirst - 1);
        const bool tfirst = (t.y & kTermFirst) != 0;
        ev_key_w[e] = make_key((uint32_t)tq, 1u, (uint32_t)x);
        ev_w[e] = tfirst ? make_int2(x, t.x) : make_int2(t.x, x);
        gp_c[e] = (int)(pop_pair_base[pop] + tq);
        ev_pos[e] = __int_as_float(t.w);
        dec_w[e] = (uint32_t)t.z;
        dest_out[e] = kPendingTerm;
      } else if (on_grid && !stop && done_ev < ev_len[e]) {
        // cut short where a partner's claim failed: that event is pending
        ChainReader rd(ev_head[e]);
        long long ix = -1;
        for (int i = 0; i <= done_ev; i++) ix = rd.next(pool);
        const int y = ix >= 0 ? pool.y[ix] : -1;
        const int q = ix >= 0 ? (pool.q[ix] & kChainPairMask) : -1;
        if (y >= 0 && y < P.cap && q >= 0 && q < P.n_pairs) {
          const PairDesc d = P.pair_desc[q];
          const bool first = C == d.b1 + nb * d.c1;
          ev_key_w[e] = make_key((uint32_t)q, 1u, (uint32_t)x);
          ev_w[e] = first ? make_int2(x, y) : make_int2(y, x);
          gp_c[e] = (int)(pop_pair_base[pop] + q);
          ev_pos[e] = pool.pos[ix];
          dec_w[e] = (uint32_t)done_ev;
          dest_out[e] = kPendingChain;
        } else {
          bad_index(P.ctr, kBadEventSlot, y);
          dest_out[e] = -1;
        }
      } else {
        // off the grid, or stopped by an error: no walk on
        dest_out[e] = (walk_done || !on_grid || stop) ? -1 : x;
        gp_c[e] = (int)(pop_pair_base[pop] + last_q);
        ev_pos[e] = last_pos;
      }
    }
    }
  }
}

// Walk rates after a round's sort: for every cell, the running sum over its
// pairs (loop order) of k_max * del_t * members of the pair's other cell;
// pairs on the per-particle path add nothing.  One block per cell, its
// threads over the cell's pairs, a block-wide scan in a fixed order.
// P.walk_stops: 1 when the population's round 0 has target operations (the
// step's later rounds then take the operations that walks stop for); with 0,
// its per-particle pairs (whose target cells were all empty at the step's
// start) are walked at the per-set rate like any pair.
__global__ void __launch_bounds__(128) k_walk_rates(const PopDev* pops) {
  chain_wait();
  const PopDev& P = pops[blockIdx.y];
  int c = blockIdx.x;
  if (c >= P.n_cells || P.n_pairs == 0) return;
  const int nb = P.grid->n_bin;
  const int lo = P.cp_off[c], hi = P.cp_off[c + 1];
  double* cum = P.cp_cum + lo + c;
  __shared__ double wsum[4];
  __shared__ double carry;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int stops = P.walk_stops;
  if (threadIdx.x == 0) carry = 0.0;
  __syncthreads();
  for (int base = lo; base < hi; base += blockDim.x) {
    int j = base + threadIdx.x;
    double lam = 0.0;
    if (j < hi) {
      int q = P.cp_list[j];
      const PairState& S = P.pair[q];
      PairDesc d = P.pair_desc[q];
      int cell1 = d.b1 + nb * d.c1, cell2 = d.b2 + nb * d.c2;
      int O = cell1 == c ? cell2 : cell1;
      int n_o = P.cell_count[O];
      P.cp_ent[j] = make_int4(q, O | (cell1 == c ? (1 << 30) : 0), P.cell_start[O], n_o);
      // per-set pairs, and per-particle pairs seen from their source cell: a
      // particle that arrives in the cell meets the other cell's members at
      // the per-set rate.  Seen from its target cell a per-particle pair is a
      // stop (no rate, cp_nstop): a particle that arrives there is one of
      // its targets, and its walk ends at the pair in a target operation
      if (!(stops && S.path == kPathParticle && c == S.bt + nb * S.ct)) {
        double l = S.k_max * P.del_t * (double)n_o;
        if (l > 0.0) lam = l;
      }
    }
    double x = lam;  // inclusive scan within the warp
    for (int o = 1; o < 32; o <<= 1) {
      double y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) wsum[wid] = x;
    __syncthreads();
    double before = carry;
    for (int w = 0; w < wid; w++) before += wsum[w];
    if (j < hi) cum[j - lo] = before + x - lam;
    __syncthreads();
    if (threadIdx.x == 0) carry += wsum[0] + wsum[1] + wsum[2] + wsum[3];
    __syncthreads();
  }
  const double total = carry;
  if (threadIdx.x == 0) cum[hi - lo] = total;
  if (threadIdx.x == 0 && stops) {
    // per entry, the first stop at or after it (hi: none)
    int nxt = hi;
    for (int j = hi - 1; j >= lo; j--) {
      const PairState& S = P.pair[P.cp_list[j]];
      if (stops && S.path == kPathParticle && c == S.bt + nb * S.ct) nxt = j;
      P.cp_nstop[j] = nxt;
    }
  }
  // the bucket table: the last entry whose stretch starts at or before each
  // bucket's start (cum is visible to the block after the barrier above)
  if (threadIdx.x < kWalkTab) {
    double target = total * (double)threadIdx.x / (double)kWalkTab;
    int a = 0, b = hi - lo - 1;
    while (a < b) {
      int mid = (a + b + 1) >> 1;
      if (cum[mid] <= target) a = mid;
      else b = mid - 1;
    }
    P.cp_tab[c * kWalkTab + threadIdx.x] = lo + a;
  }
}

// ---------------------------------------------------------------------------
// Per-particle (accelerated) path, phase 1: run sample_source_particle and
// the target update of coag_target_with_source for one target, store the
// result, and claim the target and every removed source.
constexpr int kMaxCopies = 8;  // dup copies per target operation (the growth limit keeps them at 2 or less)

struct PPResult {
  int target, p;        // target slot, pair (local)
  int n_samp, n_coag;   // counted into tot_n_samp / tot_n_coag when the operation is applied
  int merged;           // n_coag > 0
  int n_copies;         // prob_round(old_nc / new_nc); 0 removes the target
  int n_rm;             // sources it removes: rm_pool[rm_off .. rm_off + n_rm)
  int nofit;            // its removals did not fit the pool (the host sizes it to fit): it loses
  int copy_group[kMaxCopies];
  long long rm_off;
  PMeta meta;           // new target metadata
};

template <int KT>
__device__ double pp_kernel(const PopDev& P, const RecD& qs, const RecD& qt, int cs, int ct) {
  const double* a = (const double*)&qs;
  const double* b = (const double*)&qt;
  return pair_kernel<KT, double, false>(P, a, b, cs, ct, ct, 0.0, P.coeff);
}

// The first draws of a target operation: the number of removal samples,
// which bounds the sources it can remove (sample_source_particle,
// coagulation.F90:397).  k_pp_count scans the bounds, which places every
// operation's removals in one pool, so an operation can remove any number of
// sources.  Returns -1 for an operation that
// draws nothing (void, dead target, empty source cell).
__device__ __forceinline__ int pp_remove_bound(const PopDev& P, int p, int t, int k, Rng* g_out, int* n_extra,
                                               double* prm_out) {
  if (t < 0 || t >= P.cap || !P.alive[t]) return -1;
  const PairState& S = P.pair[p];
  const GridDev& G = *P.grid;
  int nb = G.n_bin;
  int src_cell = S.bs + nb * S.cs;
  if (P.cell_count[src_cell] == 0) return -1;
  double nc_target = P.recd[t].nc;
  double nc_src_min = num_conc_at_radius<double>(P.w, S.cs, G.edges[S.bs]);
  double prm_max = nc_target / nc_src_min;
  if (!(prm_max <= 1.0)) return -2;
  Rng g = make_rng(P, kStreamPart, (uint32_t)p, (uint32_t)k);
  int n_remove = rand_poisson(g, prm_max * S.nspt);
  *n_extra = rand_poisson(g, (1.0 - prm_max) * S.nspt);
  *g_out = g;
  *prm_out = prm_max;
  return n_remove;
}

// uniform number u (counted from 0) of the stream g: Rng::next's values by index
__device__ __forceinline__ double stream_at(const Rng& g, uint32_t u) {
  const U4 b = philox4x32_10(U4{g.c0, g.c1, g.c2, u >> 1}, g.k0, g.k1);
  return (u & 1u) ? u53(b.z, b.w) : u53(b.x, b.y);
}

// sample_source_particle and coag_target_with_source, one warp per target
// operation.  An operation's samples are one random stream, and most of them
// reject: a rejected sample takes two uniforms (the source, the accept draw),
// so the next 32 samples' draws lie at known places while none of them
// accepts.  The lanes test 32 samples ahead; those before the first that
// accepts (or that drew a source this operation removed already) stand, that
// one is carried out with the stream at its place, and the lanes go on after
// it.  The species sums lie with the lanes, the source's metadata in shared
// memory; the closing draws (binomial count, component duplication, the new
// target) are lane 0's.  One thread per operation was bound by its samples'
// dependent loads and FP64 arithmetic: 684 us a launch for the operations of
// 4000 sedimenting drops (about 40 a round, 1000 samples each), now 129 us;
// 61 us to 29 us for 2e4 particles scavenging under the Brownian kernel
// (about 500 operations a round).
constexpr int kPPWarps = 4;

template <int KT>
__global__ void __launch_bounds__(32 * kPPWarps) k_pp_ops(const PopDev* pops, const int* op_pop, const int* op_pair,
                         const int* op_slot, const int* op_k, const unsigned long long* op_key,
                         const long long* n_ops, PPResult* res, double* res_vol, const long long* rm_off,
                         int* rm_pool, long long rm_cap) {
  chain_wait();
  constexpr unsigned kFull = 0xffffffffu;
  __shared__ PMeta sh_src[kPPWarps];
  __shared__ double sh_u[kPPWarps][64];
  const int lane = threadIdx.x & 31;
  PMeta& src = sh_src[threadIdx.x >> 5];
  double* ubuf = sh_u[threadIdx.x >> 5];
  long long Q = *n_ops;
  // every branch up to the closing part depends on the operation alone, so
  // the warp's lanes stay together
  for (long long q = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5; q < Q;
       q += ((long long)gridDim.x * blockDim.x) >> 5) {
    const PopDev& P = pops[op_pop[q]];
    int p = op_pair[q], t = op_slot[q];
    unsigned long long prio = op_key[q];
    PPResult& R = res[q];
    const long long my_off = rm_off[q];
    if (lane == 0) {
      R.target = t;
      R.p = p;
      R.n_samp = 0;
      R.n_coag = 0;
      R.merged = 0;
      R.n_copies = 1;
      R.n_rm = 0;
      R.nofit = 0;
      R.rm_off = my_off;
    }
    if (t < 0 || t >= P.cap || !P.alive[t]) continue;  // t = -1: a redo voided by k_build_redo
    const PairState& S = P.pair[p];
    const GridDev& G = *P.grid;
    int nb = G.n_bin;
    int cs = S.cs, ct = S.ct;
    int src_cell = S.bs + nb * cs;
    int n_src = P.cell_count[src_cell];
    int src_start = P.cell_start[src_cell];
    if (n_src == 0) continue;
    const RecD qt = P.recd[t];
    double nc_target = qt.nc;
    double nc_src_min = num_conc_at_radius<double>(P.w, cs, G.edges[S.bs]);
    double prm_max = nc_target / nc_src_min;
    if (!(prm_max <= 1.0)) {
      if (lane == 0) set_status(P.ctr, kErrAssert);
      continue;
    }
    Rng g = make_rng(P, kStreamPart, (uint32_t)p, (uint32_t)op_k[q]);
    int n_remove = rand_poisson(g, prm_max * S.nspt);
    int n_extra = rand_poisson(g, (1.0 - prm_max) * S.nspt);
    if (n_remove < 0 || n_extra < 0) {
      if (lane == 0) set_status(P.ctr, kErrTimeout);
      continue;
    }
    if (my_off + n_remove > rm_cap) {
      if (lane == 0) R.nofit = 1;  // no draws, no claims; the host sized the pool from the round's total, so a guard only
      continue;
    }
    int n_total = n_remove + n_extra;
    int ns = P.n_spec;
    const double inv_k_max = S.inv_k_max;
    const unsigned long long my_claim = claim_key(P, prio);
    // source volumes of species lane and lane + 32: sums, sums of squares,
    // coefficients of variation
    double acc0 = 0.0, acc1 = 0.0, sq0 = 0.0, sq1 = 0.0, cv0 = 0.0, cv1 = 0.0;
    // the source particle: scalars in every lane, component k in lane k
    PScal cur;
    cur.grp = cur.cls = cur.nprim = cur.ncomp = cur.hyst = cur.frozen = 0;
    cur.id = 0;
    cur.lct = cur.gct = cur.imf = 0.0;
    cur.den_ice = cur.phi = __longlong_as_double(0x7ff8000000000000LL);
    int cur_c = 0;
    double cur_t = 0.0;
    int n_avg = 0, n_samp = 0, n_rm = 0;
    double pc_tot = 0.0;
    uint32_t u = g.used();
    int n_stop = n_total;  // samples to draw: n_remove + 1 once the sources' spread is known well enough
    while (n_samp < n_stop) {
      // sample n_samp + lane, as long as the ones before it reject
      const bool on = n_samp + lane < n_stop;
      int si = -1;
      double pc = 0.0, nc_s = 0.0;
      bool hit = false, again = false;
      if (on) {
        const uint32_t ul = u + 2u * (uint32_t)lane;
        double ua, ub;
        if (ul & 1u) {
          ua = stream_at(g, ul);
          ub = stream_at(g, ul + 1u);
        } else {
          const U4 b = philox4x32_10(U4{g.c0, g.c1, g.c2, ul >> 1}, g.k0, g.k1);
          ua = u53(b.x, b.y);
          ub = u53(b.z, b.w);
        }
        si = P.list[src_start + (int)(ua * (double)n_src) % n_src];
        if (n_rm > 0) again = __ldcg(&P.claim[si]) == my_claim;
        if (!again) {
          const RecD qs = P.recd[si];
          nc_s = qs.nc;
          pc = pp_kernel<KT>(P, qs, qt, cs, ct) * inv_k_max;
          hit = ub < pc;
        }
      }
      const unsigned ev = __ballot_sync(kFull, hit || again);
      const int n_on = n_stop - n_samp < 32 ? n_stop - n_samp : 32;
      const int j = ev ? __ffs(ev) - 1 : n_on;  // the lanes before j rejected
      const bool take = j < n_on;               // sample j stands too
      // the probabilities summed in sample order
      const bool redraw = take && __shfl_sync(kFull, again ? 1 : 0, j & 31) != 0;
      const int n_pc = redraw ? j : (take ? j + 1 : j);
      for (int k = 0; k < n_pc; k++) pc_tot = pc_tot + __shfl_sync(kFull, pc, k);
      n_samp += take ? j + 1 : j;
      u += 2u * (uint32_t)j;
      if (!take) continue;
      bool acc_j;
      if (redraw) {
        // a source this operation removed already has left the bin in the
        // reference, whose later samples draw from the sources left
        // (coagulation.F90:428-430): draw again
        g.seek(u);
        si = P.list[src_start + rand_int(g, n_src) - 1];
        for (int r = 0; r < 64 && __ldcg(&P.claim[si]) == my_claim; r++) si = P.list[src_start + rand_int(g, n_src) - 1];
        const RecD qs = P.recd[si];
        nc_s = qs.nc;
        pc = pp_kernel<KT>(P, qs, qt, cs, ct) * inv_k_max;
        pc_tot = pc_tot + pc;
        acc_j = g.next() < pc;
      } else {
        si = __shfl_sync(kFull, si, j);
        nc_s = __shfl_sync(kFull, nc_s, j);
        g.seek(u + 2u);
        acc_j = true;
      }
      if (acc_j) {
        n_avg++;
        double ice_a = 0.0, ice_b = 0.0;
        if (P.i_water > 0) {
          const int w = P.i_water - 1;
          ice_a = __shfl_sync(kFull, w < 32 ? acc0 : acc1, w & 31);
          ice_b = P.vol[vol_at(P, si, w)];
        }
        // aero_particle_coagulate of the source so far with this one
        PScal ys, nm;
        load_scal(P, si, ys);
        int y_c = 0;
        double y_t = 0.0;
        if (lane < ys.ncomp && lane < kMaxComponent) {
          y_c = P.csrc[comp_at(si, lane)];
          y_t = P.ctime[comp_at(si, lane)];
        }
        u = g.used();
        int n1_new, n2_new, k_src;
        bool from_a;
        warp_coag_components(g, &u, ubuf, cur.ncomp, cur.nprim, ys.ncomp, ys.nprim, &n1_new, &n2_new, &from_a,
                             &k_src);
        k_src &= 31;
        const int xa = __shfl_sync(kFull, cur_c, k_src), xb = __shfl_sync(kFull, y_c, k_src);
        const double za = __shfl_sync(kFull, cur_t, k_src), zb = __shfl_sync(kFull, y_t, k_src);
        coag_scalars(cur, ice_a, ys, ice_b, nm);
        nm.grp = nm.cls = 0;
        nm.id = 0;
        nm.ncomp = n1_new + n2_new;
        cur = nm;
        cur_c = from_a ? xa : xb;
        cur_t = from_a ? za : zb;
        if (lane < ns) {
          const double vi = P.vol[vol_at(P, si, lane)];
          acc0 = acc0 + vi;
          sq0 = sq0 + vi * vi;
        }
        if (lane + 32 < ns) {
          const double vi = P.vol[vol_at(P, si, lane + 32)];
          acc1 = acc1 + vi;
          sq1 = sq1 + vi * vi;
        }
        if (n_samp <= n_remove) {
          double pri = nc_target / nc_s;
          const double ur = stream_at(g, u);
          u++;
          if (ur < pri / prm_max) {
            bool dup = false;
            for (int z = lane; z < n_rm; z += 32) dup = dup || (__ldcg(&rm_pool[my_off + z]) == si);
            if (!__any_sync(kFull, dup)) {
              if (n_rm < n_remove) {  // at most one per removal sample: the pool holds n_remove
                if (lane == 0) {
                  rm_pool[my_off + n_rm] = si;
                  atomicMin(&P.claim[si], my_claim);
                }
                n_rm++;
              } else if (lane == 0) {
                cap_fail(P.ctr, kCapRemovals);
              }
            }
          }
          __syncwarp();
        }
        // stop drawing once past the removal samples and the mean source
        // volume is known to 10% (the largest coefficient of variation)
        if (n_avg >= 2 && n_total > n_remove + 1) {
          if (lane < ns) {
            const double mean = acc0 / (double)n_avg;
            if (mean > 0.0) cv0 = sqrt(sq0 / (double)n_avg - mean * mean) / mean;
          }
          if (lane + 32 < ns) {
            const double mean = acc1 / (double)n_avg;
            if (mean > 0.0) cv1 = sqrt(sq1 / (double)n_avg - mean * mean) / mean;
          }
          double cv = -1.0;  // below every coefficient: none found
          if (lane < ns && !isnan(cv0)) cv = cv0;
          if (lane + 32 < ns && !isnan(cv1) && cv1 > cv) cv = cv1;
          for (int o = 16; o > 0; o >>= 1) {
            const double x = __shfl_xor_sync(kFull, cv, o);
            if (x > cv) cv = x;
          }
          if (cv >= 0.0 && cv / sqrt((double)n_avg) * student_t_95(n_avg) < 0.1)
            n_stop = n_samp > n_remove + 1 ? n_samp : n_remove + 1;
          else
            n_stop = n_total;
        }
      } else {
        u = g.used();
      }
    }
    if (lane == 0) {
      R.n_samp = n_samp;
      R.n_rm = n_rm;
    }
    if (n_avg == 0) continue;
    double pc_mean = pc_tot / (double)n_samp;
    g.seek(u);
    int n_coag = 0;
    if (lane == 0) {
      if (!(pc_mean <= 1.0)) add_ll(&P.ctr->kmax_warn, (long long)(1LL));
      n_coag = rand_binomial(g, n_total, pc_mean);
      R.n_coag = n_coag;
    }
    n_coag = __shfl_sync(kFull, n_coag, 0);
    double scale = (double)n_coag / (double)n_avg;
    double* acc = res_vol + (size_t)q * ns;  // accumulated source volumes, then the new target's
    if (lane < ns) acc[lane] = acc0 * scale;
    if (lane + 32 < ns) acc[lane + 32] = acc1 * scale;
    __syncwarp();
    if (lane < cur.ncomp) {
      src.csrc[lane] = cur_c;
      src.ctime[lane] = cur_t;
    }
    __syncwarp();
    if (lane == 0) {
      src.grp = src.cls = 0;
      src.id = 0;
      src.ncomp = cur.ncomp;
      src.lct = cur.lct;
      src.gct = cur.gct;
      src.imf = cur.imf;
      src.den_ice = cur.den_ice;
      src.phi = cur.phi;
      src.hyst = cur.hyst;
      src.frozen = cur.frozen;
      src.nprim = prob_round(g, (double)cur.nprim * scale);
      {
        int n_comp = src.ncomp;
        int n_new = src.nprim < kMaxComponent ? src.nprim : kMaxComponent;
        int sample[kMaxComponent];
        if (n_new < n_comp) {
          PMeta m = src;
          sample_wo_replacement(g, n_new, n_comp, sample);
          for (int i = 0; i < n_new; i++) {
            m.csrc[i] = src.csrc[sample[i] - 1];
            m.ctime[i] = src.ctime[sample[i] - 1];
          }
          m.ncomp = n_new;
          src = m;
        } else if (n_comp < kMaxComponent && n_comp > 0) {
          PMeta m = src;
          int i_comp = 1;
          while (i_comp <= n_new) {
            if (i_comp + n_comp <= n_new) {
              for (int i = 1; i <= n_comp; i++) {
                m.csrc[i_comp + i - 2] = src.csrc[i - 1];
                m.ctime[i_comp + i - 2] = src.ctime[i - 1];
              }
              i_comp += n_comp;
            } else {
              int size = n_new - i_comp + 1;
              sample_wo_replacement(g, size, n_comp, sample);
              for (int i = 1; i <= size; i++) {
                m.csrc[i_comp + i - 2] = src.csrc[sample[i - 1] - 1];
                m.ctime[i_comp + i - 2] = src.ctime[sample[i - 1] - 1];
              }
              i_comp = n_new + 1;
            }
          }
          m.ncomp = n_new;
          src = m;
        }
      }
      if (n_coag > 0) {
        // coag_target_with_source (coagulation.F90:522-582): new target
        PMeta tm;
        load_meta(P, t, tm);
        double ice_t = 0.0;
        if (P.i_water > 0) ice_t = P.vol[vol_at(P, t, P.i_water - 1)];
        double ice_s = P.i_water > 0 ? acc[P.i_water - 1] : 0.0;
        long long tid = tm.id;
        double old_nc = nc_target;
        PMeta nm;
        coag_meta(g, tm, ice_t, src, ice_s, nm);
        nm.id = tid;
        double vt = 0.0;
        for (int k = 0; k < ns; k++) {
          acc[k] = P.vol[vol_at(P, t, k)] + acc[k];  // now the new target volumes
          vt = vt + acc[k];
        }
        double rnew = vol2rad(P.benv.frac, vt);
        int cc = S.cc;
        nm.grp = rand_group(g, P.w, cc, rnew);
        nm.cls = cc + 1;
        int b = bin_find(nb, G.log_lo, G.log_hi, rnew);
        if (b < 1 || b > nb) set_status(P.ctr, kErrOutOfGrid);
        double new_nc = num_conc_at_radius<double>(P.w, cc, rnew);
        int n_copies = prob_round(g, old_nc / new_nc);
        if (n_copies > kMaxCopies) {
          cap_fail(P.ctr, kCapCopies);
          n_copies = kMaxCopies;
        }
        for (int z = 1; z < n_copies; z++) R.copy_group[z] = rand_group(g, P.w, cc, rnew);
        R.merged = 1;
        R.n_copies = n_copies;
        R.meta = nm;
        atomicMin(&P.claim[t], claim_key(P, prio));
      }
    }
    __syncwarp();  // the shared metadata is free for the warp's next operation
  }
}

// phase 2: apply the winning target operations (k_pp_resolve)
__global__ void __launch_bounds__(128) k_pp_apply(const PopDev* pops, const int* op_pop, const long long* n_ops,
                           const PPResult* res, const double* res_vol, const int* rm_pool, const uint8_t* win,
                           const long long* rank, const int* slot_base, const long long* id_base,
                           const long long* pop_pair_base, const int* op_k, int* wk_slot, int* wk_gp, uint8_t* wk_flag) {
  chain_wait();
  // the walkers an operation makes (its target, then its copies) go to the
  // operation's own kMaxCopies places, compacted afterwards in operation
  // order, so that the next round's items do not depend on scheduling
  long long Q = *n_ops;
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < Q;
       q += (long long)gridDim.x * blockDim.x) {
    for (int z = 0; z < kMaxCopies; z++) wk_flag[q * kMaxCopies + z] = 0;
    if (!win[q]) continue;
    int pop = op_pop[q];
    const PopDev& P = pops[pop];
    const PPResult& R = res[q];
    // an operation that lost a claim is redone from scratch, so only applied
    // operations count their samples and coagulations
    if (R.n_samp) add_ll(&P.ctr->tot_samp, (long long)R.n_samp);
    if (R.n_coag) add_ll(&P.ctr->tot_coag, (long long)R.n_coag);
    uint32_t gen = *P.gen_p;
    int dlive = 0;
    for (int z = 0; z < R.n_rm; z++) {
      // sample_source_particle records each source it removes with the
      // target's ID (coagulation.F90:447-453)
      const int sz = rm_pool[R.rm_off + z];
      log_removal(P, P.id[sz], kInfoCoag, P.id[R.target]);
      kill_slot(P, sz);
      P.touched[sz] = gen;
      dlive--;
    }
    if (R.merged) {
      const double* v = res_vol + (size_t)q * P.n_spec;
      int t = R.target;
      P.touched[t] = gen;
      if (R.n_copies == 0) {
        log_removal(P, P.id[t], kInfoWeight, 0);  // aero_state_dup_particle (aero_state.F90:502-513)
        kill_slot(P, t);
        dlive--;
      } else {
        // the changed target and its copies take part in the rest of the
        // step: they walk from the end of this pair in the next round
        const int wgp = (int)(pop_pair_base[pop] + R.p);
        auto add_walker = [&](int slot, int z) {
          const long long k = q * kMaxCopies + z;
          wk_slot[k] = slot;
          wk_gp[k] = wgp;
          wk_flag[k] = 1;
        };
        store_particle(P, t, v, R.meta);
        refresh_slot(P, t);
        add_walker(t, 0);
        for (int z = 1; z < R.n_copies; z++) {
          int dest = slot_base[pop] + (int)rank[q] + (z - 1);
          if (dest >= P.cap) {
            cap_fail(P.ctr, kCapCopySlot);
            break;
          }
          PMeta cm = R.meta;
          cm.grp = R.copy_group[z];
          cm.id = id_base[pop] + rank[q] + (z - 1);
          store_particle(P, dest, v, cm);
          refresh_slot(P, dest);
          P.touched[dest] = gen;
          add_walker(dest, z);
          dlive++;
        }
      }
    } else if ((op_k[q] & 0x40000000) && R.target >= 0 && R.target < P.cap && P.alive[R.target] &&
               P.touched[R.target] != gen) {
      // a walk that stopped here for this operation, which changed nothing,
      // goes on from the end of the pair: the reference's target stays in
      // its bin for the step's later pairs.  A target that an event of this
      // round rewrote walks on from that event instead (one walker per
      // particle: two would draw the same tests and make the same event)
      const long long k = q * kMaxCopies;
      wk_slot[k] = R.target;
      wk_gp[k] = (int)(pop_pair_base[pop] + R.p);
      wk_flag[k] = 1;
    }
    if (dlive) add_ll(&P.ctr->n_live, (long long)(dlive));
  }
}

}  // namespace pmc
