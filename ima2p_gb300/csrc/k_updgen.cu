// k_updgen.cu -- the genealogy update of the no-migration model on the
// device: updategenealogy (update_gtree.cpp:723-966) with
// slider_nomigration (:79-254), findjointime (:34-77), joinsisdown
// (:375-455) and splitsisdown (:457-534).
//
// A step proposes a new genealogy for one locus of every listed chain.  The
// chains are independent (each draws from generators of its own), so they
// run in parallel, a CTA each; the loci of a chain follow one another, as
// in qupdate -- its proposals because they share its generator, its
// decisions because they share its sums.  But an HKY or stepwise proposal
// depends on no decision (it draws the acceptance uniform itself), and
// neither do the weights and the likelihood of the proposed genealogy.  So
// up to UG_K consecutive loci go through one launch of each kernel:
//   k_ug_propose  a warp per locus stages its nodes, times and labels in
//                 shared memory and keeps the old ones for a rejection; one
//                 thread draws every locus's words (the edge, the slide's
//                 length, the acceptance uniform); a warp per locus takes the
//                 edge out; one thread makes the slides, locus by locus (the
//                 reference's tail recursion as a walk over prepared states);
//                 a warp per locus puts the edge back and writes the
//                 proposed genealogy with its level schedule.
//   weights and likelihoods, as batches (k_treeweight, k_is / k_hky / k_ug_sw)
//   k_ug_decide   a warp per locus loads its weights; then, locus by locus,
//                 the locus's new weights into the chain's sums
//                 (sum_subtract_treeinfo, ginfo.cpp:249-285), the theta
//                 integrals whose count or length changed
//                 (integrate_tree_prob, update_gtree_common.cpp:1945-2055),
//                 one uniform against the ratio -- for three loci at once,
//                 a lane for every parameter after every way the decisions
//                 before can go, so that three decisions take the time of
//                 one; then the warps commit or restore.
// An IS locus goes by itself: its decision draws the uniform only when the
// likelihood does not reject.  The serial part bounds an update: with a
// launch per locus a decision took 43 us (an incomplete gamma function a
// lane, 10 to 20 us, and chains of dependent loads) and a proposal 26, 50 us
// a step with the launches.  Measured (2 sweeps of 50 HKY loci x 32 chains /
// 100 stepwise ones x 64): 5.3 -> 1.5 (1.0 some calls on) and 10.0 -> 2.3
// ms, of which 0.7 and 1.2 ms are set-up; after 300 such calls, when the heated
// chains have lengths that need the gamma functions' series, 6.5 -> 1.6 and
// 21.4 -> 5.6 ms.  A proposal and a
// decision of a launch take 25 to 35 us each, whatever its number of loci.
// The file is compiled with -fmad=false: the reference's adds and
// multiplies round as written; log, exp and sqrt are the device's.
#include "internal.h"

#include <algorithm>
#include <cfloat>
#include <cstddef>

#include "igamma.cuh"
#include "ug_rng.cuh"

namespace {

constexpr double TIMEMAX = 1000000.0;        // imamp.hpp:129
constexpr double SLIDESTDVMAX = 20.0;        // update_gtree.cpp:686
constexpr double ONEOVERSQRT2PI = 0.3989422803;  // utilities.cpp:461, as the reference writes it
constexpr int UG_RNG_WARPS = 3;              // warps of a proposal for the generators
constexpr int UG_BATCH = 4;                  // loads of a lane in flight before their stores
constexpr int UG_WORDS = 8;                  // generator words made ahead per locus (a proposal takes about 4)
constexpr int SLIDE_MAX_STEPS = 1 << 20;     // a slide that long is an error, not a loop

// normdev (utilities.cpp:476-503): the polar method, keeping the second
// deviate for the next call; before it is scaled
__device__ double stdnormal(LocalRng &r)
{
  if (r.iset == 0) {
    while (r.at + 1 < r.ahead) {
      const double d1 = r.v1[r.at], d2 = r.v2[r.at];
      mt_step(r);
      mt_step(r);
      if (d1 == 0.0 && d2 == 0.0) continue;
      r.gset = d1;
      r.iset = 1;
      return d2;
    }
    double v1, v2, rsq;
    do {
      v1 = 2.0 * uniform(r) - 1.0;
      v2 = 2.0 * uniform(r) - 1.0;
      rsq = v1 * v1 + v2 * v2;
    } while (rsq >= 1.0 || rsq == 0.0);
    const double fac = sqrt(-2.0 * log(rsq) / rsq);
    r.gset = v1 * fac;
    r.iset = 1;
    return v2 * fac;
  }
  r.iset = 0;
  return r.gset;
}

__device__ double normprob(double mean, double stdev, double val)
{
  const double z = (val - mean) / stdev;
  const double sq = (z == 0.0) ? 0.0 : z * z;
  return ONEOVERSQRT2PI * exp(-sq / 2) / stdev;
}

__device__ double dmin(double a, double b) { return a < b ? a : b; }

// a < b for values that are not negative (nor -0 or NaN), on the integer
// pipe: an FP64 comparison waits for the FP64 pipe
__device__ __forceinline__ bool lt(double a, double b) { return __double_as_longlong(a) < __double_as_longlong(b); }

// findperiod (update_gtree_common.cpp:1626-1636)
__device__ int findperiod(const double *tv, int nsplit, double t)
{
  int k = 0;
  while (k < nsplit && !lt(t, tv[k])) k++;
  return k;
}

// findjointime (update_gtree.cpp:34-77): when the populations of the sliding
// edge and its sister come together
__device__ double findjointime(const TwModel &M, const double *tv, int nsplit, int slidepop, int sispop,
                               double edgeuptime, double sisuptime)
{
  int ep = findperiod(tv, nsplit, edgeuptime), sp = findperiod(tv, nsplit, sisuptime);
  while (ep < sp) {
    ep++;
    if (slidepop == M.droppops[ep][0] || slidepop == M.droppops[ep][1]) slidepop = M.pop_down[slidepop];
  }
  while (sp < ep) {
    sp++;
    if (sispop == M.droppops[sp][0] || sispop == M.droppops[sp][1]) sispop = M.pop_down[sispop];
  }
  while (slidepop != sispop && ep < nsplit) {
    ep++;
    if (slidepop == M.droppops[ep][0] || slidepop == M.droppops[ep][1]) slidepop = M.pop_down[slidepop];
    if (sispop == M.droppops[ep][0] || sispop == M.droppops[ep][1]) sispop = M.pop_down[sispop];
  }
  return ep == 0 ? 0.0 : tv[ep - 1];
}

// The slide as a walk over states, three per edge k: 3 k up from its lower
// end, 3 k + 1 down from its upper end, 3 k + 2 down from where the sliding
// edge bounced off (its own upper end, or where their populations join).  A
// state knows how far there is to go and the two states that follow, by
// bitran; one that follows without a draw is there twice.  A step is then one
// 16-byte load, one comparison and one subtraction: a slide takes tens of
// steps once a chain has settled, and the loci's slides follow one another.
struct __align__(16) SlideState {
  double room;
  int32_t next[2];
};

// A locus's share of the proposal's shared memory.
struct UgSmem {
  SlideState *ss;
  double *stop;    // where the sliding edge bounces off each edge
  double *t;
  NodeRec *nd;
  int32_t *pop;
  int32_t *h;      // heights, then the level counts (HKY)
  int16_t *sch;
};

// slide states [3][2n-1]; stops, times, nodes and labels [2n-1]; heights [2n-1] then level
// counts [n+2]; the schedule [2n]
__host__ __device__ size_t ug_locus_smem(int maxn)
{
  const size_t maxnl = 2 * (size_t)maxn - 1;
  return (maxnl * (3 * sizeof(SlideState) + 8 + 8 + 8 + 4) + (maxnl + maxn + 2) * 4 + 2 * (size_t)maxn * 2 + 23) / 16 * 16;
}

// the generator's words, twice: the current state and the next
constexpr size_t UG_RNG_SMEM = 2 * 624 * 4;

__device__ UgSmem ug_carve(char *base, int maxn)
{
  const int maxnl = 2 * maxn - 1;
  UgSmem s;
  s.ss = reinterpret_cast<SlideState *>(base);
  s.stop = reinterpret_cast<double *>(s.ss + 3 * maxnl);
  s.t = s.stop + maxnl;
  s.nd = reinterpret_cast<NodeRec *>(s.t + maxnl);
  s.pop = reinterpret_cast<int32_t *>(s.nd + maxnl);
  s.h = s.pop + maxnl;
  s.sch = reinterpret_cast<int16_t *>(s.h + maxnl + maxn + 2);
  return s;
}

__device__ void ug_fail(int32_t *err, int code, int who)
{
  if (atomicCAS(&err[0], 0, code) == 0) atomicExch(&err[1], who);
}

// A CTA per listed chain, a warp per locus of the launch.
__global__ void __launch_bounds__(32 * (UG_K + UG_RNG_WARPS)) k_ug_propose(UgArgs a)
{
  extern __shared__ __align__(16) char smem[];
  __shared__ int s_root[UG_K], s_twists;
  __shared__ ItemDev s_it[UG_K];
  __shared__ TwModel s_M;  // the tables up to pop_down
  __shared__ double s_tv[TW_MAXPOPS];
  __shared__ double s_draws[4 * UG_K * UG_WORDS];
  // per locus: the slide's deviation, its length and where it ended;
  // stepwise: the allele step's log deviate and sign
  __shared__ double s_std[UG_K], s_hold[UG_K], s_tp[UG_K], s_logu[UG_K];
  __shared__ int s_neg[UG_K], s_edges[UG_K][4];  // edge, freed, old and new sister
  const int w = blockIdx.x, tid = threadIdx.x, lane = tid & 31, j = tid >> 5;
  const int ci = a.chains[w];
  const int item = ci * a.nloci + a.locus + min(j, a.k - 1);  // this warp's locus
  const ItemDev it = a.items[item];
  const int n = it.n, nl = 2 * n - 1, maxnl = 2 * a.maxn;
  const size_t base = it.node_off, wj = (size_t)j * a.nch + w;
  const size_t lsm = ug_locus_smem(a.maxn);
  uint32_t *mt = reinterpret_cast<uint32_t *>(smem);
  char *loci = smem + UG_RNG_SMEM;
  const UgSmem s = ug_carve(loci + j * lsm, a.maxn);
  {
    const int32_t *src = reinterpret_cast<const int32_t *>(a.model);
    int32_t *dst = reinterpret_cast<int32_t *>(&s_M);
    for (int k = tid; k < (int)(offsetof(TwModel, toff) + 3) / 4; k += blockDim.x) dst[k] = src[k];
  }
  if (tid < a.nsplit) s_tv[tid] = a.tvals[(size_t)ci * a.nsplit + tid];
  LocalRng g;
  if (j >= a.k) {
    // three warps for the chain's generator
    const int rt = tid - 32 * a.k;
    rng_load(g, a.rng + w, mt, rt, 32 * UG_RNG_WARPS);
    rng_ahead(g, s_draws, a.k * UG_WORDS, rt, 32 * UG_RNG_WARPS);
  } else {
    NodeRec *bkn = a.bk_nodes + wj * maxnl;
    double *bkt = a.bk_t + wj * maxnl;
    int32_t *bkp = a.bk_pop + wj * maxnl;
    int root = -1;
    for (int k0 = lane; k0 < nl; k0 += 32 * UG_BATCH) {
      NodeRec r[UG_BATCH];
      double t[UG_BATCH];
      int32_t p[UG_BATCH];
#pragma unroll
      for (int b = 0; b < UG_BATCH; b++) {
        const int k = k0 + 32 * b;
        if (k >= nl) break;
        r[b] = a.nodes[base + k];
        t[b] = a.t64[base + k];
        p[b] = a.pop[base + k];
      }
#pragma unroll
      for (int b = 0; b < UG_BATCH; b++) {
        const int k = k0 + 32 * b;
        if (k >= nl) break;
        s.nd[k] = bkn[k] = r[b];
        s.t[k] = bkt[k] = t[b];
        s.pop[k] = bkp[k] = p[b];
        if (r[b].down == -1) root = k;
      }
    }
    root = __reduce_max_sync(~0u, root);
    if (root < n) {  // uploads are checked for one internal root; stop rather than read past the genealogy
      if (lane == 0) ug_fail(a.err, UG_E_TREE, w);
      root = nl - 1;
    }
    __syncwarp();
    if (lane == 0) {
      s_it[j] = it;
      s_root[j] = root;
      s_std[j] = dmin(SLIDESTDVMAX, s.t[s.nd[root].up0] / 3);
    }
    if (a.hky) {
      int16_t *bks = a.bk_sched + wj * maxnl;
      for (int k = lane; k < 2 * n; k += 32) bks[k] = a.sched[it.sched_off + k];
    }
    if (a.sw) {  // stepwise: the branch terms too (joinsisdown and splitsisdown zero the new root's)
      const int32_t *A = a.alleles + it.al_off;
      const double *dl = a.dlike + it.dl_off;
      int32_t *bka = a.bk_A + wj * maxnl;
      double *bkd = a.bk_dl + wj * maxnl;
      for (int k0 = lane; k0 < nl; k0 += 32 * UG_BATCH) {
        int32_t al[UG_BATCH];
        double d[UG_BATCH];
#pragma unroll
        for (int b = 0; b < UG_BATCH; b++) {
          const int k = k0 + 32 * b;
          if (k >= nl) break;
          al[b] = A[k];
          d[b] = dl[k];
        }
#pragma unroll
        for (int b = 0; b < UG_BATCH; b++) {
          const int k = k0 + 32 * b;
          if (k >= nl) break;
          bka[k] = al[b];
          bkd[k] = d[b];
        }
      }
    }
    if (lane == 0) {
      a.bk_len[wj] = a.len[item];
      a.bk_nlev[wj] = a.nlev[item];
    }
  }
  __syncthreads();
  // From here on the chain's generators bind the loci together, but only the
  // draws themselves follow one another: first the words of every locus (how
  // many it takes does not depend on the slides), then, after a warp each has
  // taken its edge out, the slides, whose steps take bits of the other
  // register (bitran), from shared memory; a warp each then puts the edge
  // back.
  if (tid == 32 * a.k) {
    for (int jj = 0; jj < a.k; jj++) {
      const NodeRec *nd = ug_carve(loci + jj * lsm, a.maxn).nd;
      const int nl = 2 * s_it[jj].n - 1;
      // pick an edge that is not the root's: floor(uniform() nl), exactly
      // ((y + 1/2) 2^-32 nl has fewer than 53 bits)
      int edge;
      do {
        edge = (int)((2ull * uniform_word(g) + 1) * nl >> 33);
      } while (nd[edge].down == -1);
      s_edges[jj][0] = edge;
      s_hold[jj] = stdnormal(g);
      // stepwise: finishSWupdateA's allele draw (k_ug_sw), its deviate
      if (a.sw) s_logu[jj] = log_uniform(g);
      // the acceptance uniform, next in the stream
      if (a.predraw) a.ustore[(size_t)jj * a.nch + w] = log_uniform(g);
    }
    s_twists = g.twists;
  }
  __syncthreads();
  const bool mine = j < a.k;  // a warp with a locus
  NodeRec *nd = s.nd;
  double *t = s.t;
  double *dl = a.sw ? a.dlike + it.dl_off : nullptr;
  const int edge = mine ? s_edges[j][0] : 0, freed = mine ? nd[edge].down : 0;
  const int oldsis = !mine ? 0 : (nd[freed].up0 == edge) ? nd[freed].up1 : nd[freed].up0;
  int rootmove = 0;
  double roottime = 0.0;  // lane 0, once the root has moved
  __syncwarp();
  if (mine && lane == 0) {
    s_hold[j] = s_hold[j] * s_std[j] + 0.0;
    // joinsisdown: extend the sister over the freed edge
    t[oldsis] = t[freed];
    const int dd = nd[freed].down;
    nd[oldsis].down = (int16_t)dd;
    if (dd != -1) {
      if (nd[dd].up0 == freed) nd[dd].up0 = (int16_t)oldsis;
      else nd[dd].up1 = (int16_t)oldsis;
    } else {
      rootmove = 1;
      roottime = (oldsis < n) ? 0.0 : t[nd[oldsis].up0];
      s_root[j] = oldsis;
      t[oldsis] = TIMEMAX;
      if (dl) dl[oldsis] = 0.0;
    }
    a.prop[2 * wj + 1] = rootmove;  // tmrca
    s_edges[j][2] = oldsis;
  }
  __syncwarp();
  if (mine) {
    const double eup = (edge < n) ? 0.0 : t[nd[edge].up0];
    const int epop = s.pop[edge];
    for (int k = lane; k < nl; k += 32) {
      const NodeRec r = nd[k];
      const double tk = t[k], up = k < n ? 0.0 : t[r.up0];
      const int pop = s.pop[k];
      const double join = pop != epop ? findjointime(s_M, s_tv, a.nsplit, epop, pop, eup, up) : 0.0;
      bool node = lt(eup, up);
      double stop = node ? up : eup;
      if (lt(stop, join)) {
        stop = join;
        node = false;
      }
      SlideState *v = s.ss + 3 * k;
      v[0].room = tk - stop;
      v[0].next[0] = node ? 3 * r.up1 : 3 * k + 2;
      v[0].next[1] = node ? 3 * r.up0 : 3 * k + 2;
      const int d = r.down;
      const int sib = d == -1 ? -1 : nd[d].up0 == k ? nd[d].up1 : nd[d].up0;
      v[1].room = d == -1 ? DBL_MAX : tk - up;
      v[2].room = d == -1 ? DBL_MAX : tk - stop;
      v[1].next[0] = v[2].next[0] = 3 * sib;
      v[1].next[1] = v[2].next[1] = 3 * d + 1;
      s.stop[k] = stop;
    }
  }
  __syncthreads();
  if (tid == 32 * a.k) {
    // slider_nomigration: move each edge's bottom through its genealogy, up
    // where the reference's dist is negative
    for (int jj = 0; jj < a.k; jj++) {
      const UgSmem q = ug_carve(loci + jj * lsm, a.maxn);
      const double hold = s_hold[jj];
      int sis = s_edges[jj][2], steps = 0, state = 3 * sis;
      double tp = q.t[s_edges[jj][0]], dist = fabs(hold);
      bool up = __double2hiint(hold) < 0 && lt(0.0, dist);
      // from the edge's own place to the first node
      double room = DBL_MAX;
      if (up) room = tp - q.stop[sis];
      else if (q.ss[++state].room != DBL_MAX) room = q.t[sis] - tp;
      if (!lt(dist, room)) {
        SlideState S = q.ss[state];
        do {
          dist -= room;
          int next = S.next[0];
          if (next != S.next[1] && bitran(g)) next = S.next[1];
          state = next;
          S = q.ss[state];
          room = S.room;
        } while (!lt(dist, room) && ++steps < SLIDE_MAX_STEPS);
        if (steps >= SLIDE_MAX_STEPS) ug_fail(a.err, UG_E_SLIDE, w);
        sis = state / 3;
        const int kind = state - 3 * sis;
        up = kind == 0;
        tp = up ? q.t[sis] : kind == 2 ? q.stop[sis] : sis < s_it[jj].n ? 0.0 : q.t[q.nd[sis].up0];
      }
      if (up) tp -= dist;
      else tp = lt(tp + dist, TIMEMAX) ? tp + dist : TIMEMAX;
      s_tp[jj] = tp;
      s_edges[jj][3] = sis;
      if (a.sw) s_neg[jj] = bitran(g);  // the allele step's sign
    }
  }
  __syncthreads();
  if (!mine) {
    rng_store(g, a.rng + w, &s_twists, tid - 32 * a.k, 32 * UG_RNG_WARPS);
    return;
  }
  const int newsis = s_edges[j][3];
  if (lane == 0) {
    s_edges[j][1] = freed;
    // splitsisdown: the freed edge becomes the new sister's lower part
    const double curt = s_tp[j];
    t[edge] = curt;
    t[freed] = t[newsis];
    t[newsis] = curt;
    const int dd = nd[newsis].down;
    if (dd != -1) {
      if (nd[dd].up0 == newsis) nd[dd].up0 = (int16_t)freed;
      else nd[dd].up1 = (int16_t)freed;
    } else {
      s_root[j] = freed;
      roottime = curt;
      rootmove = 1;
      if (curt > TIMEMAX) ug_fail(a.err, UG_E_ROOTTIME, w);
      if (dl) dl[freed] = 0.0;
    }
    nd[freed].down = (int16_t)dd;
    int nowpop = s.pop[newsis];
    const int period = findperiod(s_tv, a.nsplit, curt);
    while (s_M.pop_e[nowpop] <= period && s_M.pop_e[nowpop] != -1) nowpop = s_M.pop_down[nowpop];
    s.pop[freed] = nowpop;
    nd[newsis].down = (int16_t)freed;
    nd[edge].down = (int16_t)freed;
    nd[freed].up0 = (int16_t)newsis;
    nd[freed].up1 = (int16_t)edge;
    a.prop[2 * wj] = (oldsis != newsis);
    if (a.hky) {  // the edited edges, as likelihoodHKY takes them
      ReqDev &R = a.req[a.req_of[wj]];
      R.e[0] = edge;
      R.e[1] = freed;
      R.e[2] = oldsis;
      R.e[3] = newsis;
    }
    // the slide's Hastings term, where the root moved
    double sw = 0.0;
    if (rootmove) {
      const double hold = s_hold[j];
      sw = -log(normprob(0.0, s_std[j], hold));
      sw += log(normprob(0.0, dmin(SLIDESTDVMAX, roottime / 3), hold));
    }
    a.slidew[wj] = sw;
  }
  __syncwarp();
  if (lane < 4) a.edges[4 * wj + lane] = s_edges[j][lane];
  if (a.sw && lane == 0) {  // the allele step's deviate, for k_ug_sw
    a.lallele[wj] = s_logu[j];
    a.neg[wj] = s_neg[j];
  }
  if (a.hky) {
    // heights (tips 0, a node one above its higher daughter) by rounds of
    // relaxation over the internal nodes: heights only grow, towards the
    // true ones, and a round that changes nothing ends it (at most n)
    int32_t *h = s.h;
    for (int k = lane; k < nl; k += 32) h[k] = 0;
    __syncwarp();
    bool done = false;
    for (int round = 0; round <= n && !done; round++) {
      bool changed = false;
      for (int k = n + lane; k < nl; k += 32) {
        const int ha = h[s.nd[k].up0], hb = h[s.nd[k].up1];
        const int v = 1 + (ha > hb ? ha : hb);
        if (v != h[k]) {
          h[k] = v;
          changed = true;
        }
      }
      done = !__any_sync(~0u, changed);
    }
    __syncwarp();
    int H = h[s_root[j]];
    if (!done || H < 1 || H > n - 1) {
      if (lane == 0) ug_fail(a.err, UG_E_TREE, w);
      H = 1;
      __syncwarp();
      for (int k = n + lane; k < nl; k += 32) h[k] = 1;
    }
    // the level schedule as the genealogy upload builds it: internal nodes
    // by height, in index order within a level
    int16_t *order = s.sch, *lstart = s.sch + (n - 1);
    int32_t *cnt = h + nl;  // H + 2 <= n + 1 entries past the heights
    for (int k = lane; k <= H + 1; k += 32) cnt[k] = 0;
    __syncwarp();
    for (int k = n + lane; k < nl; k += 32) atomicAdd(&cnt[h[k] + 1], 1);
    __syncwarp();
    if (lane == 0) {
      for (int k = 1; k <= H + 1; k++) {
        cnt[k] += cnt[k - 1];
        lstart[k - 1] = (int16_t)cnt[k];
      }
      a.nlev[item] = H;
    }
    __syncwarp();
    for (int b0 = n; b0 < nl; b0 += 32) {
      const int k = b0 + lane;
      const int hk = k < nl ? h[k] : -1;
      const unsigned peers = __match_any_sync(~0u, hk);
      const int rank = __popc(peers & ((1u << lane) - 1u));
      if (k < nl) order[cnt[hk] + rank] = (int16_t)k;
      __syncwarp();
      if (k < nl && rank == 0) cnt[hk] += __popc(peers);
      __syncwarp();
    }
    __syncwarp();
    for (int k = lane; k < n + H; k += 32) a.sched[it.sched_off + k] = s.sch[k];  // order, then level starts
  }
  for (int k = lane; k < nl; k += 32) {
    a.nodes[base + k] = s.nd[k];
    const double t = s.t[k];
    a.t64[base + k] = t;
    const float hi = (float)t;
    a.tff[base + k] = make_float2(hi, (float)(t - (double)hi));
    a.pop[base + k] = s.pop[k];
  }
  if (lane == 0) a.is_valid[item] = 0;  // the IS site labels follow daughter order, which moved
}

// The decisions of D loci as a binary tree: node 1 is the first one's, node
// 2 v the next one's after v was rejected, 2 v + 1 after it was accepted.
// Seven nodes of up to nine parameters fill two warps, whose FP64 work hides
// behind each other's latency; more parameters take two loci at a time.
constexpr int UG_D = 3, UG_NODES = 1 << UG_D;

// A CTA per listed chain: the Metropolis-Hastings decisions of the launch's
// loci in turn, then commit or restore.
__global__ void __launch_bounds__(32 * UG_K) k_ug_decide(UgArgs a)
{
  __shared__ int32_t s_dc[UG_K][TW_MAXT], s_c0[TW_MAXT];
  __shared__ double s_fold[UG_K][TW_MAXT], s_fnew[UG_K][TW_MAXT], s_hold[UG_K][TW_MAXT], s_hnew[UG_K][TW_MAXT];
  __shared__ double s_f0[TW_MAXT], s_h0[TW_MAXT];
  // per node: the sums as they stand before it (c, f) and with its locus's
  // new weights
  __shared__ int32_t s_cb[UG_NODES][TW_MAXT], s_cn[UG_NODES][TW_MAXT];
  __shared__ double s_fb[UG_NODES][TW_MAXT], s_fn[UG_NODES][TW_MAXT], s_hn[UG_NODES][TW_MAXT];
  __shared__ double s_q0[TW_MAXTH], s_q[UG_NODES][TW_MAXTH];  // integrals: current, with the new weights
  __shared__ int8_t s_keep[UG_NODES][TW_MAXTH], s_st[UG_NODES][TW_MAXTH];
  __shared__ double s_psum[UG_NODES];
  __shared__ double s_u[UG_K], s_dpdg[UG_K], s_pdg[UG_K], s_sw[UG_K], s_at[UG_K];
  __shared__ int s_code[UG_K], s_acc[UG_K], s_fail, s_twists, s_last;
  __shared__ __align__(16) uint32_t s_mt[2 * 624];
  const int w = blockIdx.x, tid = threadIdx.x, lane = tid & 31, j = tid >> 5, nt = blockDim.x;
  const int ci = a.chains[w];
  const TwModel &M = *a.model;
  const int T = M.T, nth = M.nth;
  const int maxnl = 2 * a.maxn;
  const size_t wj = (size_t)j * a.nch + w;
  const int item = ci * a.nloci + a.locus + (j < a.k ? j : 0);  // this warp's locus (j < k)
  const ItemDev it = a.items[item];
  if (j < a.k) {
    for (int q = lane; q < T; q += 32) {
      const size_t ic = (size_t)item * T + q;
      s_dc[j][q] = a.ncc[ic] - a.cc[ic];
      s_fold[j][q] = a.fc[ic];
      s_fnew[j][q] = a.nfc[ic];
      s_hold[j][q] = a.hcc[ic];
      s_hnew[j][q] = a.nhcc[ic];
    }
    if (lane == 0) {
      const int k = a.sw ? 0 : a.req_of[wj];
      const double pdgnew = a.sw ? a.swnew[wj] : a.res[k];
      s_code[j] = a.sw ? IMA_EVAL_OK : a.st[k];
      s_at[j] = a.sw ? a.aterm[wj] : 0.0;
      s_pdg[j] = pdgnew;
      s_dpdg[j] = a.gbeta * (pdgnew - a.pdg[item]);
      s_sw[j] = a.slidew[wj];
      s_u[j] = a.predraw ? a.ustore[wj] : 0.0;
      s_acc[j] = 0;
    }
  }
  for (int q = tid; q < T; q += nt) {
    const size_t gc = (size_t)w * T + q;
    s_c0[q] = a.ag_cc[gc];
    s_f0[q] = a.ag_fc[gc];
    s_h0[q] = a.ag_hcc[gc];
  }
  for (int i = tid; i < nth; i += nt) s_q0[i] = a.qint[(size_t)w * nth + i];
  if (tid == 0) s_fail = a.err[0];
  double probg = a.probg[ci];
  const double beta = a.beta[ci];
  // an IS locus draws its uniform here: the chain's generator staged
  LocalRng g{};
  const bool draw = !a.predraw;
  if (draw) rng_load(g, a.rng + w, s_mt, tid, nt);
  __syncthreads();
  // parameter i's integral as it stands after node v (of depth dep) is accepted
  auto resolve = [&](int v, int dep, int i) {
    double q = s_q0[i];
#pragma unroll
    for (int d = 0; d < UG_D; d++) {
      const int u = d <= dep ? v >> (dep - d) : 0;  // its ancestor there
      const bool accepted = d == dep || (d < dep && ((v >> (dep - 1 - d)) & 1));
      const double x = s_q[u][i];
      if (accepted && !s_keep[u][i]) q = x;
    }
    return q;
  };
  const int step = nth <= 9 ? UG_D : 2;
  for (int j0 = 0; j0 < a.k; j0 += step) {
    const int D = min(step, a.k - j0), nodes = 1 << D;
    if (!a.hky && !a.sw) {  // an IS locus (by itself) that the likelihood rejects or cannot take
      if (s_code[j0] == IMA_EVAL_IS_FAIL && tid == 0) ug_fail(a.err, UG_E_ISFAIL, w);
      if (s_code[j0] == IMA_EVAL_IS_REJECT || s_code[j0] == IMA_EVAL_IS_FAIL) break;
    }
    if (s_fail) break;
    // sum_subtract_treeinfo: the chain's sums plus the new weights minus the
    // old, along every node's path
    for (int x = tid; x < (nodes - 1) * T; x += nt) {
      const int v = 1 + x / T, q = x % T, dep = 31 - __clz(v);
      int c = s_c0[q];
      double f = s_f0[q], hh = s_h0[q];
      for (int d = 0; d <= dep; d++) {
        if (d == dep) {
          s_cb[v][q] = c;
          s_fb[v][q] = f;
        }
        if (d < dep && !((v >> (dep - 1 - d)) & 1)) continue;  // a rejected one
        c += s_dc[j0 + d][q];
        f -= s_fold[j0 + d][q];
        f += s_fnew[j0 + d][q];
        f = (0 > f) ? 0.0 : f;
        hh -= s_hold[j0 + d][q];
        hh += s_hnew[j0 + d][q];
      }
      s_cn[v][q] = c;
      s_fn[v][q] = f;
      s_hn[v][q] = hh;
    }
    __syncthreads();
    // the theta integrals, a lane each: count and length summed over the
    // parameter's cells in order, the last accepted value kept when neither
    // changed (integrate_tree_prob)
    for (int x = tid; x < (nodes - 1) * nth; x += nt) {
      const int v = 1 + x / nth, i = x % nth;
      int c = 0, holdc = 0;
      double f = 0.0, holdf = 0.0, hc = 0.0;
      for (int e = M.th_off[i]; e < M.th_off[i + 1]; e++) {
        const int cell = M.th_idx[e];
        c += s_cn[v][cell];
        holdc += s_cb[v][cell];
        f += s_fn[v][cell];
        holdf += s_fb[v][cell];
        hc += s_hn[v][cell];
      }
      const bool keep = c == holdc && f == holdf;
      Ig ig{{a.logfact, 0}};
      if (!keep) s_q[v][i] = ig.coal(c, f, hc, M.th_max[i], M.th_min[i]);
      s_keep[v][i] = keep;
      s_st[v][i] = (int8_t)ig.st;
    }
    __syncthreads();
    if (j == 0) {
      // a lane per node: its p(G), its ratio; then the path that was taken
      const int v = lane, dep = v > 0 ? 31 - __clz(v) : 0;
      const bool node = v > 0 && v < nodes;
      bool bad = false;
      int last = 0;  // the last accepted node before this one
      if (node) {
        double psum = 0;
#pragma unroll 2
        for (int i = 0; i < nth; i++) {
          psum += resolve(v, dep, i);
          bad |= s_st[v][i] != 0;
        }
        for (int d = 0; d < dep; d++)
          if ((v >> (dep - 1 - d)) & 1) last = v >> (dep - d);
        s_psum[v] = psum;
      }
      __syncwarp();
      bool acc = false;
      // U < min(1, e^mh), as ln U < mh: ln U was taken with the proposal's draws
      double lu = node ? s_u[j0 + dep] : 0.0;
      if (draw && lane == 0) lu = log_uniform(g);
      if (draw) lu = __shfl_sync(~0u, lu, 0);
      if (node) {
        double tpw = -(last ? s_psum[last] : probg);
        tpw += s_psum[v];
        double mh = tpw + s_dpdg[j0 + dep];
        mh = beta * mh + s_sw[j0 + dep] + s_at[j0 + dep];
        acc = lu < mh;
      }
      const unsigned accs = __ballot_sync(~0u, acc), bads = __ballot_sync(~0u, bad);
      int v1 = 1, lastacc = 0;
      for (int d = 0; d < D; d++) {
        if ((bads >> v1) & 1) {
          if (lane == 0) {
            ug_fail(a.err, UG_E_TERM, w);
            s_fail = 1;
          }
          break;
        }
        const int ok = (accs >> v1) & 1;
        if (lane == 0) s_acc[j0 + d] = ok;
        if (ok) lastacc = v1;
        v1 = 2 * v1 + ok;
      }
      if (lane == 0) s_last = lastacc;
    }
    __syncthreads();
    const int last = s_last;
    if (last) {
      const int dep = 31 - __clz(last);
      for (int q = tid; q < T; q += nt) {
        s_c0[q] = s_cn[last][q];
        s_f0[q] = s_fn[last][q];
        s_h0[q] = s_hn[last][q];
      }
      for (int i = tid; i < nth; i += nt) {
        s_q0[i] = resolve(last, dep, i);
      }
      probg = s_psum[last];
    }
    __syncthreads();
  }
  if (draw) {
    if (tid == 0) s_twists = g.twists;
    __syncthreads();
    rng_store(g, a.rng + w, &s_twists, tid, nt);
  }
  for (int q = tid; q < T; q += nt) {
    const size_t gc = (size_t)w * T + q;
    a.ag_cc[gc] = s_c0[q];
    a.ag_fc[gc] = s_f0[q];
    a.ag_hcc[gc] = s_h0[q];
  }
  for (int i = tid; i < nth; i += nt) a.qint[(size_t)w * nth + i] = s_q0[i];
  if (tid == 0) a.probg[ci] = probg;
  if (j >= a.k) return;
  const bool acc = s_acc[j] != 0;
  const int n = it.n, nl = 2 * n - 1;
  const size_t base = it.node_off;
  if (acc) {
    for (int q = lane; q < T; q += 32) {
      const size_t ic = (size_t)item * T + q;
      a.cc[ic] = a.ncc[ic];
      a.fc[ic] = s_fnew[j][q];
      a.hcc[ic] = s_hnew[j][q];
    }
    if (lane == 0) {
      a.pdg[item] = s_pdg[j];
      a.nacc[(size_t)w * a.nloci + a.locus + j]++;
      if (a.prop[2 * wj]) a.ntopo[(size_t)w * a.nloci + a.locus + j]++;
    }
  } else {  // restoreedges, storegenealogystats(..., 1)
    const NodeRec *bkn = a.bk_nodes + wj * maxnl;
    const double *bkt = a.bk_t + wj * maxnl;
    const int32_t *bkp = a.bk_pop + wj * maxnl;
    const int16_t *bks = a.bk_sched + wj * maxnl;
    for (int k0 = lane; k0 < 2 * n; k0 += 32 * UG_BATCH) {
      NodeRec r[UG_BATCH];
      double t[UG_BATCH];
      int32_t p[UG_BATCH];
      int16_t sc[UG_BATCH];
#pragma unroll
      for (int b = 0; b < UG_BATCH; b++) {
        const int k = k0 + 32 * b;
        if (k < nl) {
          r[b] = bkn[k];
          t[b] = bkt[k];
          p[b] = bkp[k];
        }
        if (a.hky && k < 2 * n) sc[b] = bks[k];
      }
#pragma unroll
      for (int b = 0; b < UG_BATCH; b++) {
        const int k = k0 + 32 * b;
        if (k < nl) {
          a.nodes[base + k] = r[b];
          a.t64[base + k] = t[b];
          const float hi = (float)t[b];
          a.tff[base + k] = make_float2(hi, (float)(t[b] - (double)hi));
          a.pop[base + k] = p[b];
        }
        if (a.hky && k < 2 * n) a.sched[it.sched_off + k] = sc[b];
      }
    }
    if (lane == 0) {
      a.len[item] = a.bk_len[wj];
      a.nlev[item] = a.bk_nlev[wj];
      a.is_valid[item] = 0;  // the site labels cached by the evaluation are the proposal's
      if (a.sw) {  // restoreedges: the three moved edges from their copies, the new sister only if nonzero
        const int32_t *eo = a.edges + 4 * wj;
        const int edge = eo[0], freed = eo[1], oldsis = eo[2], newsis = eo[3];
        const int32_t *bka = a.bk_A + wj * maxnl;
        const double *bkd = a.bk_dl + wj * maxnl;
        double *dl = a.dlike + it.dl_off;
        a.alleles[it.al_off + freed] = bka[freed];
        dl[edge] = bkd[edge];
        dl[oldsis] = bkd[oldsis];
        dl[freed] = bkn[freed].down != -1 ? bkd[freed] : 0.0;
        const double hs = a.holdsis[wj];
        if (hs != 0) dl[newsis] = hs;
      }
    }
  }
  if (a.hky)  // copyfraclike / restorescalefactors: the recomputed nodes' slots
    for (int k = lane; k < nl; k += 32) {
      const size_t x = base + k;
      if (a.fresh32[x]) {
        if (acc) a.slot32[x] ^= 1;
        a.fresh32[x] = 0;
      }
      if (a.slot64 && a.fresh64[x]) {
        if (acc) a.slot64[x] ^= 1;
        a.fresh64[x] = 0;
      }
    }
}

}  // namespace

int ug_loci_per_launch(int nloci, int maxn)
{
  // a quarter of the loci at most, so that four launches can be in flight,
  // and what fits in 160 KB of shared memory
  const int fit = (int)((160 * 1024 - UG_RNG_SMEM) / ug_locus_smem(maxn));
  return std::max(1, std::min({UG_K, nloci / 4, fit}));
}

void launch_ug_propose(const UgArgs &a, cudaStream_t st)
{
  const size_t bytes = UG_RNG_SMEM + a.k * ug_locus_smem(a.maxn);
  cudaFuncSetAttribute(k_ug_propose, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
  if (bytes > 36 * 1024)  // (48 KB with the static part)
    cudaFuncSetAttribute(k_ug_propose, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_MAX - 12 * 1024);
  k_ug_propose<<<a.nch, 32 * (a.k + UG_RNG_WARPS), bytes, st>>>(a);
}

void launch_ug_decide(const UgArgs &a, cudaStream_t st)
{
  cudaFuncSetAttribute(k_ug_decide, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
  k_ug_decide<<<a.nch, 32 * std::max(2, a.k), 0, st>>>(a);
}

extern "C" void ima_ug_rng_seed(ima_ug_rng *g, int32_t seed)
{
  if (!g) return;
  ima_mt19937_seed(&g->mt, (uint32_t)seed);
  g->iset = 0;
  g->gset = 0.0;
  g->iseed = 0x7fffffffffffffffull + (uint64_t)(int64_t)seed;
}
