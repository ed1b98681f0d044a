// Delay windows: several LIF steps per pass over the state (included by lif.cu).
//
// A spike of step t arrives at step t + D, so during any K <= D consecutive steps no neuron needs
// what another one does in them. A run of more than one step therefore goes by windows of K steps:
//   update   every item takes its K ring values (all of them final: their spikes were delivered in
//            earlier windows), clears those slots and runs its K steps with its state in registers;
//            the spikes go to the raster rows of the window, as they do in the per-step kernels;
//   deliver  after every item is done, the window's spikes are read back from the raster and their
//            synapses added to the write slots (or the pull kernel delivers them by groups).
// The write slots of steps s .. s + K - 1 are s + D .. s + D + K - 1 mod R >= D + 1, all of them read
// and cleared by now, so nothing pending is touched. The same float operations per item and the
// same integer sums: state, ring, raster and event count equal the per-step kernels' bit for bit.
//
// What it saves: the state is read and written once per window instead of once per step (48-60 of
// the ~68 bytes of an item's step), and a persistent run meets two grid barriers per window
// instead of one per step. The update is then bound by instruction issue (many flies) or by the
// latency of its 18 dependent steps (one fly: ~250 cycles each), the delivery by L2 atomics (or
// the pull's own bound). Measured on 71,618 neurons and 15 M synapses at dense firing: one fly
// 38.7 -> 3.4 us per step; 64 flies, the update alone 55 -> 17 us per step in windows of 8; 2,000
// neurons, one fly: 5.4 -> 0.56 us per step.
#pragma once

namespace flyb {

constexpr int kWindowBlock = 256;
constexpr int kWindowMax = 32;      // steps per window: lane j of a warp keeps the spike word of step j
// Ring values loaded ahead of their steps. A persistent run of few items waits for each of them (6: one
// fly, 2,000 neurons 55.9 us per 100 steps against 57.1 with 4); the update of many items has other
// warps to run and takes 4, with registers bounded for six blocks per SM (64 flies, 71,618 neurons,
// 40 steps: 3040 -> 2918 us).
constexpr int kAheadFew = 6, kAheadMany = 4;
constexpr int kWindowSpikes = 4;    // spikes a thread hands over per delivery round
// Blocks per SM of a delivery launch. At dense firing the atomics of more blocks spread over more of the
// ring than the L2 holds (70,000 neurons, 256 flies in step, 20 steps at a delay of 6: 14.4 ms with 3,
// 15.1 with 4; 8 flies, 8 steps, where 3 leave latency uncovered: 122 us, 107 with 4).
constexpr int kDeliverBlocks = 3;
constexpr int kWindowEdges = 4;     // edges a lane of the delivery keeps in flight

// Steps a window may hold (0: the run does not go by windows). It needs the raster to remember the
// window's spikes; episode counters gate single steps and stay with the per-step kernels. Two rules
// leave them per-step launches that scatter their spikes, where those are the faster:
//  - launches that ask for the staged or the deferred kernel, where a ring slot is larger than a sixth
//    of the L2: the K slots of a window at dense firing then go through DRAM, the one slot of a step
//    less so (20 steps at a delay of 18, all cells bursting, deferred kernel against windows, ms:
//    70,000 neurons, 256 flies, 72 MB 8.8 / 11.6; 40 flies on the fixed ring, 22 MB 2.0 / 2.4; but 64
//    flies, 18 MB 2.9 / 1.9), or where the windows hold two steps only (20,000 neurons, 11 flies,
//    staged, three steps at a delay of 2: 44 us, by windows 56);
//  - depressing runs of two or three steps by windows of two, whose closing pass costs more than the
//    windows save (20,000 neurons, 11 flies, two steps: 31 us, by windows 37).
constexpr long long kWindowSlotBytes = 20ll << 20;

static int window_steps(const LifK& k, int launch, bool staged, int ring_bytes) {
  if (!k.raster || k.nsteps < 2 || k.n_delay < 2 || (k.flags & FLYB_LIF_EPISODES)) return 0;
  int K = k.n_delay < k.nsteps ? k.n_delay : k.nsteps;
  if (k.raster_slots > 0 && K > k.raster_slots) K = k.raster_slots;
  if (K > kWindowMax) K = kWindowMax;
  if (K < 2) return 0;
  if (launch == FLYB_LAUNCH_STEP && !(k.flags & FLYB_LIF_PULL_DELIVERY)) {
    const long long slot_bytes = (long long)k.n * k.batch * ring_bytes;
    if ((staged || k.spike_list) && (K == 2 || slot_bytes > kWindowSlotBytes)) return 0;
    if ((k.flags & FLYB_LIF_STD) && K == 2 && k.nsteps < 4) return 0;
  }
  return K;
}

__device__ __forceinline__ size_t raster_row(const LifK& k, const Clk& clk, int s) {
  return (size_t)(k.raster_slots > 0 ? slot_after(clk.raster_pos, s, k.raster_slots) : s) * k.words;
}

__device__ __forceinline__ float poisson_draw(const LifK& k, const Clk& clk, int s, size_t t, int i, int b) {
  return (k.flags & FLYB_LIF_EXT_UNIFORM)
             ? k.uniforms[(size_t)s * ((size_t)k.n * k.batch) + t]
             : philox_uniform(k.seed, clk.step0 + s, (uint32_t)i, (uint32_t)(k.fly0 + b));
}

// Bit j: Poisson drive forces a spike of this lane's item at step s0 + j. A warp usually holds few
// driven items (one cell in 36): each one's draws of all K <= 32 steps are then made at once, lane
// j making that of step j; with more driven lanes than steps every lane makes its own.
__device__ __forceinline__ unsigned poisson_steps(const LifK& k, const Clk& clk, int s0, int K, long long t, int i, int b,
                                                  float pp) {
  const int lane = threadIdx.x & 31;
  unsigned driven = __ballot_sync(0xffffffffu, pp > 0.0f), forced = 0;
  if (__popc(driven) >= K) {
    if (pp > 0.0f)
      for (int j = 0; j < K; ++j)
        if (poisson_draw(k, clk, s0 + j, (size_t)t, i, b) < pp) forced |= 1u << j;
    return forced;
  }
  for (; driven; driven &= driven - 1) {
    const int src = __ffs(driven) - 1;
    const int si = __shfl_sync(0xffffffffu, i, src), sb = __shfl_sync(0xffffffffu, b, src);
    const float sp = __shfl_sync(0xffffffffu, pp, src);
    const bool hit = lane < K && poisson_draw(k, clk, s0 + lane, (size_t)(t - lane + src), si, sb) < sp;
    const unsigned steps = __ballot_sync(0xffffffffu, hit);
    if (lane == src) forced = steps;
  }
  return forced;
}

// The value of a spike of item t at step s: a Poisson-forced one is 1, any other the cell's `active`.
__device__ __forceinline__ float spike_value(const LifK& k, const Clk& clk, int s, size_t t, int i, int b) {
  const float act = __ldg(&k.active[i]);
  if (act == 1.0f) return 1.0f;
  const float pp = (k.flags & FLYB_LIF_POISSON) ? k.poisson_p[t] : 0.0f;
  return pp > 0.0f && poisson_draw(k, clk, s, t, i, b) < pp ? 1.0f : act;
}

// Steps [s0, s0 + K), K <= kWindowMax, of the block's items [base, base + span). The steps
// are lif_update's operations in its order, without its per-step branches: the loop is bound by
// instruction issue, so what does not depend on the step (the cell's constants, whether a lane of
// the warp has Poisson drive) is decided before it, and lane j keeps the warp's spike word of
// step j until the end, where one store writes the words of all steps. Under depression the
// spikes array keeps the resource at the window's start until the delivery has used it
// (window_finish puts the spikes back).
template <bool FIXED, bool STD, int AHEAD>
__device__ __forceinline__ void window_update(const LifK& k, const Clk& clk, int s0, int K, long long base, int span) {
  using RingT = typename std::conditional<FIXED, long long, int>::type;
  const long long t = base + threadIdx.x;
  const int lane = threadIdx.x & 31;
  if ((int)threadIdx.x >= span || t - lane >= k.t_end) return;   // warp-uniform: span is a multiple of 32
  const bool ok = t < k.t_end;
  const unsigned slot = (unsigned)k.n * (unsigned)k.batch;     // n * batch < 2^31
  const LifP& P = k.P;
  const bool adapt_on = k.flags & FLYB_LIF_ADAPT, counts_on = k.flags & FLYB_LIF_COUNTS;
  const int i = ok ? neuron_of(k, (int)t) : 0, b = ok ? (int)t - i * k.batch : 0;
  RingT* ring = (RingT*)k.ring + t;
  const int first_slot = slot_after(clk.ring_pos, s0, k.R);
  const long long wfirst = (t - lane) >> 5;                    // this warp's raster word
  const auto write_words = [&](unsigned mine) {                // lane j: the word of step s0 + j
    if (lane >= K) return;
    k.raster[raster_row(k, clk, s0 + lane) + wfirst] = mine;
    if (k.pull_bits) k.pull_bits[pull_word_index(k, clk.step0 + s0 + lane, wfirst)] = mine;
  };
  float vv = P.v_rest, gg = 0.0f, ref = 0.0f, ad = 0.0f, rt = 0.0f, dv = 0.0f, pp = 0.0f, cn = 0.0f, rr = 1.0f;
  float act = 0.0f, keep = 1.0f, jump = P.jump;
  if (ok) {
    vv = k.v[t]; gg = k.g[t]; ref = k.refrac[t]; ad = k.adapt[t]; rt = k.rate[t]; dv = k.drive[t];
    if (k.flags & FLYB_LIF_POISSON) pp = k.poisson_p[t];
    if (counts_on) cn = k.counts[t];
    if (STD) { rr = k.res[t]; keep = 1.0f - k.std_u[i]; }
    if (adapt_on && k.adapt_jump) jump = __ldg(&k.adapt_jump[i]);
    act = k.active[i];
  }
  if (k.flags & FLYB_LIF_SKIP_FROZEN) {
    // a warp of frozen cells at rest without input in the window: nothing changes (neural.cu:24-26).
    // A cell that passes the other tests has not spiked in this run, so its spike value is looked at
    // in the first window only: under depression the array then holds the resource.
    bool rest = act == 0.0f && pp == 0.0f && vv == P.v_rest && gg == 0.0f && dv == 0.0f && ad == 0.0f &&
                ref == 0.0f && rt == 0.0f && (!ok || ((s0 > 0 || k.spikes[t] == 0.0f) && k.res[t] == 1.0f));
    if (__all_sync(0xffffffffu, rest)) {
      int slot_of = first_slot;
      for (int j = 0; j < K; ++j) {
        if (ok && ring[(size_t)slot_of * slot]) rest = false;
        slot_of = slot_of + 1 < k.R ? slot_of + 1 : 0;
      }
      if (__all_sync(0xffffffffu, rest)) {
        write_words(0u);
        if (STD && ok) k.spikes[t] = rr;
        return;
      }
    }
  }
  const float res0 = rr;
  // ring values in flight: the value of step j + AHEAD is requested when step j has used its
  // own. Requests beyond the window, and those of lanes without an item, read a word nobody uses:
  // the loop then has no branch around a load.
  RingT due[AHEAD];
  int rs = first_slot, cs = first_slot;                        // slots of the next load and of the step being run
  const RingT* from = (const RingT*)k.ring + (ok ? t : (long long)k.t_end - 1);
  const auto next_value = [&]() {
    const RingT x = from[(size_t)((unsigned long long)(unsigned)rs * slot)];
    rs = rs + 1 < k.R ? rs + 1 : 0;
    return x;
  };
  float spike = 0.0f;
  unsigned my_word = 0;
#pragma unroll
  for (int u = 0; u < AHEAD; ++u) due[u] = next_value();
  const unsigned forced = poisson_steps(k, clk, s0, K, t, i, b, pp);
  for (int j0 = 0; j0 < K; j0 += AHEAD) {
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) {
      const int j = j0 + u;
      if (j >= K) break;
      const RingT c = ok ? due[u] : 0;
      due[u] = next_value();
      // 1. synaptic input due now
      if (c) ring[(size_t)((unsigned long long)(unsigned)cs * slot)] = 0;
      cs = cs + 1 < k.R ? cs + 1 : 0;
      const float in = FIXED ? __double2float_rn((double)c * (1.0 / 4294967296.0)) : P.w_syn * (float)c;
      const float g0 = gg * P.a_s, g1 = c ? g0 + in : g0;
      gg = g1;
      // 2. membrane
      float target = P.v_rest + g1;
      target = target + dv;
      target = target - ad;
      float v1 = vv - target;
      v1 = v1 * P.a_m;
      v1 = target + v1;
      v1 = ref > 0.0f ? P.v_reset : v1;
      float r1 = ref - P.dt;
      r1 = r1 < 0.0f ? 0.0f : r1;
      // 3. threshold x active, Poisson forcing
      spike = (v1 >= P.v_th ? 1.0f : 0.0f) * act;
      spike = (forced >> j) & 1u ? 1.0f : spike;
      const bool fired = spike > 0.0f;
      vv = fired ? P.v_reset : v1;
      ref = fired ? P.t_ref : r1;
      // 4. adaptation, depression, counters, rate
      if (adapt_on) {
        ad = ad * P.a_ad;
        ad = ad + spike * jump;
      }
      if (STD) {
        rr = fired ? rr * keep : rr;
        float dep = 1.0f - rr;
        dep = dep * P.a_std;
        rr = 1.0f - dep;
      }
      cn = cn + spike;
      rt = rt * P.a_r;
      rt = rt + spike * P.rg;
      const unsigned word = __ballot_sync(0xffffffffu, fired);
      my_word = lane == j ? word : my_word;
    }
  }
  write_words(my_word);
  if (!ok) return;
  k.v[t] = vv; k.g[t] = gg; k.refrac[t] = ref; k.rate[t] = rt;
  k.spikes[t] = STD ? res0 : spike;
  if (adapt_on) k.adapt[t] = ad;
  if (counts_on) k.counts[t] = cn;
  if (STD) k.res[t] = rr;
}

// The amount item t transmits with its spike of step s (window start s0, its raster word w, bit):
// the spike value, under depression times the resource replayed from the window's start with
// lif_update's operations.
__device__ __forceinline__ float window_amount(const LifK& k, const Clk& clk, int s0, int s, size_t t, int i, int b,
                                               long long w, int bit) {
  const float spike = spike_value(k, clk, s, t, i, b);
  if (!(k.flags & FLYB_LIF_STD)) return spike;
  float r = k.spikes[t];
  const float keep = 1.0f - __ldg(&k.std_u[i]);
  for (int q = s0; q < s; ++q) {
    if ((k.raster[raster_row(k, clk, q) + w] >> bit) & 1u) r = r * keep;
    float dep = 1.0f - r;
    dep = dep * k.P.a_std;
    r = 1.0f - dep;
  }
  return spike * r;
}

template <bool LISTED>
struct WindowSmem {
  static constexpr int CAP = kWindowBlock * kWindowSpikes;
  int wcnt[kWindowBlock / 32], wdeg[kWindowBlock / 32];
  int wspk[LISTED ? 2 : 1][kWindowBlock / 32];   // spikes per warp of a task's words, alternate tasks
  unsigned short item[LISTED ? CAP : 1];         // the round's spikes: (word of the task) * 32 + bit
  int pre[CAP];            // exclusive prefix of the spikers' out-degrees (all of them positive)
  int start[CAP];          // first outgoing edge
  long long to[CAP];       // ring offset of the fly in the write slot
  float x[CAP];            // transmitted amount (fixed ring)
};

// The last spiker of [lo, hi] whose first edge position is at most q.
__device__ __forceinline__ int spiker_of(const int* pre, int q, int lo, int hi) {
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (pre[mid] <= q) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// Delivery of the window's spikes. A block takes kWindowBlock raster words at a time and hands over their
// spikes in rounds of at most kWindowSpikes per thread. A persistent run of few items is bound by
// latency and fires few cells per word: each thread takes the spikes of its own word. Per-step
// launches list the block's spikes in item order first (LISTED) and share each round alike: where
// many cells fire together a word holds up to 32 spikes, eight rounds of a few busy threads otherwise, and
// the flies of a cell, whose targets share sectors, now go out together. 20 steps by windows of 6,
// bursts under depression, us: 5,000 neurons, 16 flies 289 -> 117; by windows of 18: 20,000 neurons, 11
// flies 170 -> 100; 70,000 neurons, 64 flies 2,240 -> 1,500. Sparse windows of one fly pay 0.5-1 us for
// the list, which the persistent run's six windows of a 10 ms frame would feel (56 -> 63 us).
// The round's edges are cut into `parts` shares, one per block that takes the same words (few words
// then keep as many threads busy), and those into equal shares per warp, whatever the out-degrees
// (10^4 and beyond beside a mean of ~200). A warp walks its share 32 positions at a time, one edge
// per lane: the spikers that start among the 32 positions are marked in a word, and a lane's spiker
// is the one before them plus the marks up to its own position.
template <bool FIXED, bool LISTED>
__device__ void window_deliver(const LifK& k, const Clk& clk, int s0, int K, int parts, WindowSmem<LISTED>& sm) {
  constexpr int NW = kWindowBlock / 32, CAP = WindowSmem<LISTED>::CAP;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned upto = 0xffffffffu >> (31 - lane);            // this lane and those before it
  const size_t slot = (size_t)k.n * k.batch;
  const int w0 = k.t_begin >> 5, nw = ((k.t_end + 31) >> 5) - w0;
  const long long total = (long long)nw * K, tasks = (total + kWindowBlock - 1) / kWindowBlock * parts;
  unsigned long long events = 0;
  int flip = 0;
  for (long long task = blockIdx.x; task < tasks; task += gridDim.x, flip ^= 1) {
    const int part = (int)(task % parts);
    const unsigned u0 = (unsigned)(task / parts) * kWindowBlock, u = u0 + threadIdx.x;   // n * batch * K / 32 < 2^31
    const int j = (int)(u / (unsigned)nw), w = w0 + (int)(u - (unsigned)j * (unsigned)nw), s = s0 + j;
    unsigned bits = u < total ? k.raster[raster_row(k, clk, s) + w] : 0u;
    const size_t ws = (size_t)slot_after(clk.ring_pos, s + k.n_delay, k.R) * slot;
    int rank = 0, spikes = 0;                                  // of the word's first spike in the list, of all words
    if (LISTED) {
      const int mine_spk = __popc(bits), incl = warp_scan(mine_spk);
      if (lane == 31) sm.wspk[flip][warp] = incl;
      __syncthreads();
      rank = incl - mine_spk;
#pragma unroll
      for (int q = 0; q < NW; ++q) {
        if (q < warp) rank += sm.wspk[flip][q];
        spikes += sm.wspk[flip][q];
      }
    }
    for (int r0 = 0; LISTED ? r0 < spikes : __syncthreads_or(bits != 0); r0 += CAP) {   // also: the shared arrays are free
      const int m = spikes - r0 < CAP ? spikes - r0 : CAP, per = (m + kWindowBlock - 1) / kWindowBlock;
      if (LISTED) {
        for (; bits && rank < r0 + m; ++rank, bits &= bits - 1)
          sm.item[rank - r0] = (unsigned short)(threadIdx.x * 32 + __ffs(bits) - 1);
        __syncthreads();
      }
      int cnt = 0, sum = 0;
      int e0[kWindowSpikes], deg[kWindowSpikes], fly[kWindowSpikes];
      size_t at_step[kWindowSpikes];                                  // write slot (LISTED: a list mixes steps)
      float x[kWindowSpikes];
#pragma unroll
      for (int q = 0; q < kWindowSpikes; ++q) {
        deg[q] = 0;
        if (LISTED ? q < per && (int)threadIdx.x * per + q < m : bits != 0) {
          int bit, jq = j, wq = w;
          if (LISTED) {
            const int it = sm.item[threadIdx.x * per + q];
            const unsigned uq = u0 + (it >> 5);
            bit = it & 31;
            jq = (int)(uq / (unsigned)nw);
            wq = w0 + (int)(uq - (unsigned)jq * (unsigned)nw);
            at_step[q] = (size_t)slot_after(clk.ring_pos, s0 + jq + k.n_delay, k.R) * slot;
          } else {
            bit = __ffs(bits) - 1;
            bits &= bits - 1;
          }
          const int t = wq * 32 + bit, i = neuron_of(k, t);
          fly[q] = t - i * k.batch;
          e0[q] = __ldg(&k.out_ptr[i]);
          deg[q] = __ldg(&k.out_ptr[i + 1]) - e0[q];
          if (FIXED) {
            x[q] = window_amount(k, clk, s0, s0 + jq, (size_t)t, i, fly[q], wq, bit);
            if (x[q] == 0.0f) deg[q] = 0;
          }
          cnt += deg[q] > 0;
          sum += deg[q];
        }
      }
      const int icnt = warp_scan(cnt), isum = warp_scan(sum);
      if (lane == 31) { sm.wcnt[warp] = icnt; sm.wdeg[warp] = isum; }
      __syncthreads();
      int pos = icnt - cnt, run = isum - sum, L = 0, E = 0;
#pragma unroll
      for (int q = 0; q < NW; ++q) {
        if (q < warp) { pos += sm.wcnt[q]; run += sm.wdeg[q]; }
        L += sm.wcnt[q];
        E += sm.wdeg[q];
      }
#pragma unroll
      for (int q = 0; q < kWindowSpikes; ++q) {
        if (deg[q] <= 0) continue;
        sm.pre[pos] = run;
        sm.start[pos] = e0[q];
        sm.to[pos] = (long long)((LISTED ? at_step[q] : ws) + fly[q]);
        if (FIXED) sm.x[pos] = x[q];
        run += deg[q];
        ++pos;
      }
      __syncthreads();
      const int mine = ((E + parts - 1) / parts + 31) & ~31, stop = part * mine + mine < E ? part * mine + mine : E;
      const int share = ((mine + NW - 1) / NW + 31) & ~31;
      const int q0 = part * mine + warp * share, end = q0 + share < stop ? q0 + share : stop;
      if (q0 < end) {
        int lo = spiker_of(sm.pre, q0, 0, L - 1);              // of position q0 (warp-uniform)
        for (int qb = q0; qb < end; qb += 32 * kWindowEdges) {
          int2 ed[kWindowEdges];
          int at[kWindowEdges];
#pragma unroll
          for (int v = 0; v < kWindowEdges; ++v) {
            const int q = qb + 32 * v;
            const int next = lo + 1 + lane;
            const unsigned off = next < L ? (unsigned)(sm.pre[next] - q) : 32u;
            const unsigned marks = __reduce_or_sync(0xffffffffu, off < 32u ? 1u << off : 0u);
            at[v] = lo + __popc(marks & upto);
            lo += __popc(marks);
            if (q + lane < end) ed[v] = __ldg(&k.out_edge[sm.start[at[v]] + (q + lane - sm.pre[at[v]])]);
          }
#pragma unroll
          for (int v = 0; v < kWindowEdges; ++v) {
            if (qb + 32 * v + lane >= end) continue;
            const size_t dst = (size_t)sm.to[at[v]] + (size_t)ed[v].x * k.batch;
            if (FIXED) {
              const long long f = __double2ll_rn((double)__int_as_float(ed[v].y) * (double)sm.x[at[v]] * 4294967296.0);
              atomicAdd((unsigned long long*)k.ring + dst, (unsigned long long)f);
            } else {
              atomicAdd((int*)k.ring + dst, ed[v].y);
            }
          }
        }
      }
      if (part == 0) events += (unsigned long long)E;
    }
  }
  if (k.events && threadIdx.x == 0 && events) atomicAdd(k.events, events);
}

// The spikes of the run's last step back into the spikes array (depression only: window_update).
__device__ __forceinline__ void window_finish(const LifK& k, const Clk& clk, long long first, long long stride) {
  const unsigned* __restrict__ row = k.raster + raster_row(k, clk, k.nsteps - 1);
  for (long long t = k.t_begin + first; t < k.t_end; t += stride) {
    const int i = neuron_of(k, (int)t);
    const bool fired = (row[t >> 5] >> (t & 31)) & 1u;
    k.spikes[t] = fired ? spike_value(k, clk, k.nsteps - 1, (size_t)t, i, (int)t - i * k.batch) : 0.0f;
  }
}

// Per-step launches: one update and one delivery launch per window.
template <bool FIXED, bool STD>
__global__ void __launch_bounds__(kWindowBlock, FIXED ? 4 : 6) lif_window_update_kernel(LifK k, int s0, int K) {
  window_update<FIXED, STD, kAheadMany>(k, read_clock(k), s0, K, k.t_begin + (long long)blockIdx.x * kWindowBlock, kWindowBlock);
}

template <bool FIXED>
__global__ void __launch_bounds__(kWindowBlock, kDeliverBlocks) lif_window_deliver_kernel(LifK k, int s0, int K, int parts) {
  __shared__ WindowSmem<true> sm;
  window_deliver<FIXED, true>(k, read_clock(k), s0, K, parts, sm);
}

__global__ void __launch_bounds__(kWindowBlock) lif_window_finish_kernel(LifK k) {
  window_finish(k, read_clock(k), (long long)blockIdx.x * kWindowBlock + threadIdx.x, (long long)gridDim.x * kWindowBlock);
}

// Persistent launch: every window of the run in one cooperative kernel.
template <bool FIXED, bool STD>
__global__ void __launch_bounds__(kWindowBlock, FIXED ? 3 : 4) lif_window_persistent_kernel(LifK k, int kmax, int span, int parts) {
  __shared__ WindowSmem<false> sm;
  const Clk clk = read_clock(k);
  int generation = 0;
  for (int s0 = 0; s0 < k.nsteps; s0 += kmax) {
    const int K = kmax < k.nsteps - s0 ? kmax : k.nsteps - s0;
    const bool last = s0 + K == k.nsteps;
    for (long long base = k.t_begin + (long long)blockIdx.x * span; base < k.t_end; base += (long long)gridDim.x * span)
      window_update<FIXED, STD, kAheadFew>(k, clk, s0, K, base, span);
    if (!grid_barrier(k.sync, k.status, generation, s0)) return;
    if (last && blockIdx.x == 0 && !(k.flags & FLYB_LIF_NO_ADVANCE)) advance_clock(k, clk);   // all have read it
    window_deliver<FIXED, false>(k, clk, s0, K, parts, sm);
    if (last && !STD) return;
    if (!grid_barrier(k.sync, k.status, generation, s0)) return;
  }
  window_finish(k, clk, (long long)blockIdx.x * kWindowBlock + threadIdx.x, (long long)gridDim.x * kWindowBlock);
}

// Blocks that share the edges of the same raster words in the delivery: up to 16 while that gives a
// block of the grid at most two tasks per window.
static int deliver_parts(const LifK& k, int K, long long grid) {
  const long long words = ((long long)k.t_end - k.t_begin + 31) / 32 * K, batches = (words + kWindowBlock - 1) / kWindowBlock;
  int parts = 1;
  while (parts < 16 && batches * parts * 2 <= 2 * grid) parts *= 2;
  return parts;
}

template <bool FIXED, bool STD>
static int run_lif_windows_persistent(const LifK& k, int kmax, int grid_cap, cudaStream_t st) {
  int dev = 0, sms = 0, per_sm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, lif_window_persistent_kernel<FIXED, STD>, kWindowBlock, 0);
  const long long items = (long long)k.t_end - k.t_begin;
  // few items: spread their warps over the SMs, where each has its scheduler to itself
  int span = kWindowBlock;
  while (span > 32 && items <= (long long)sms * (span / 2)) span /= 2;
  const long long chunks = (items + span - 1) / span;
  long long grid = (long long)sms * per_sm;
  int parts = deliver_parts(k, kmax, grid);
  const long long tasks = ((items + 31) / 32 * kmax + kWindowBlock - 1) / kWindowBlock * parts;
  const long long need = chunks > tasks ? chunks : tasks;
  if (grid > need) grid = need;
  if (grid_cap > 0 && grid > grid_cap) grid = grid_cap;
  if (grid < 1) return FLYB_ECOOP;
  cudaError_t e = cudaMemsetAsync(k.sync, 0, 2 * sizeof(int), st);
  if (e != cudaSuccess) return (int)e;
  LifK kk = k;
  void* args[] = {&kk, &kmax, &span, &parts};
  return (int)cudaLaunchCooperativeKernel((void*)lif_window_persistent_kernel<FIXED, STD>, dim3((unsigned)grid),
                                          dim3(kWindowBlock), args, 0, st);
}

// Per-step launches by windows. Under pull delivery a window ends with a delivery group, two groups
// ahead at most (the pull buffer holds two), and its groups are pulled one after the other.
template <bool FIXED, bool STD>
static int run_lif_windows(const LifK& k, int kmax, cudaStream_t st) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const bool pulls = pulls_itself(k);
  const unsigned chunks = (unsigned)(((long long)k.t_end - k.t_begin + kWindowBlock - 1) / kWindowBlock);
  const int L = k.pull_group;
  for (int s0 = 0; s0 < k.nsteps;) {
    int K = kmax < k.nsteps - s0 ? kmax : k.nsteps - s0;
    const int phase = pulls ? (k.pull_phase + s0) % L : 0;
    if (pulls && K > 2 * L - phase) K = 2 * L - phase;
    lif_window_update_kernel<FIXED, STD><<<chunks, kWindowBlock, 0, st>>>(k, s0, K);
    FLYB_CHECK_LAUNCH();
    if (pulls) {
      for (int done = 0; done < K;) {
        const int to_group_end = L - (phase + done) % L, n = K - done < to_group_end ? K - done : to_group_end;
        const int rc = launch_pull(k, n, st);
        if (rc) return rc;
        done += n;
      }
    } else if (!(k.flags & FLYB_LIF_PULL_DELIVERY)) {
      lif_window_deliver_kernel<FIXED><<<sms * kDeliverBlocks, kWindowBlock, 0, st>>>(k, s0, K, deliver_parts(k, K, sms * kDeliverBlocks));
      FLYB_CHECK_LAUNCH();
    }
    s0 += K;
  }
  if (STD) {
    lif_window_finish_kernel<<<sms * 4, kWindowBlock, 0, st>>>(k);
    FLYB_CHECK_LAUNCH();
  }
  if (needs_advance(k)) {
    lif_advance_kernel<<<1, 256, 0, st>>>(k);
    FLYB_CHECK_LAUNCH();
  }
  return 0;
}

template <bool FIXED, bool STD>
static int run_by_windows(const LifK& k, int kmax, int launch, int grid_cap, cudaStream_t st) {
  return launch == FLYB_LAUNCH_STEP ? run_lif_windows<FIXED, STD>(k, kmax, st)
                                    : run_lif_windows_persistent<FIXED, STD>(k, kmax, grid_cap, st);
}

}  // namespace flyb
