// cm_block.cuh -- the resident-steps kernel (included by cm_engine.cu).
//
// k_block holds each block's electrons in shared memory and takes them through many steps per launch.  An
// iteration is one list of tasks of up to 32 electrons each, which the block's warps take one after
// another: the flights, by wave segment (one material and energy band per warp), each with the elastic
// event it ends in, and the inelastic and misc events queued by the iteration before.  What an iteration
// appends is the next one's lists, so a warp runs one kind of work at a time although a thread sees every
// kind, and secondaries start at once in the slots of electrons that ended.
//
// What bounds it: instruction fetch (the warps run different code), the barriers of an iteration, whose pace
// is the longest task's, and in small runs the serial latency of a step (~9 us).  It runs where few electrons
// are left: there the queue kernels take ~55 us an iteration however few electrons they move, and one
// electron per thread through whole steps, which this kernel replaced, left a warp's lanes in different
// events (one B200: 26 M steps of a 3 keV scan with phonons 62 -> 18.7 ms, 10 k primaries of 1 keV in FP64
// 17.3 -> 7.8 ms, the last 256 k electrons of a 500 eV line scan 12.3 -> 6.2 ms).  With the GPU full the queue
// kernels are 2 to 3.6 times faster, so they keep the full waves (whole runs through the queue kernels and
// their tail / through this kernel alone: FP32 line scan 44 / 144 ms, image 209 / 759, deep 120 / 223, FP64
// line scan 32 / 63; 5.5 / 1.7 G electron-steps/s in the first).
//
#pragma once

namespace cm {

// Threads: 512 (128 registers) in FP32, 384 (168) in FP64, where 128 registers spill 430 bytes a step over
// leaf shapes and 168 spill 32 (one B200, 384 against 512 threads: 10 k primaries FP64 7.5 / 8.1 ms, FP64
// line scan 32.9 / 33.4 ms; in FP32 the phonon scan 19.6 / 18.8 ms, the others within 2 %).  Over shape trees
// of depth 2 both still spill about 1450 bytes of stores and 1700 (FP32) or 2200 (FP64) of loads.
#ifndef CM_BLOCK_THREADS
#define CM_BLOCK_THREADS (sizeof(R) == 8 ? 384 : 512)
#endif
#ifndef CM_BLOCK_MINB
#define CM_BLOCK_MINB 1
#endif
#ifndef CM_BLOCK_SLOTS
#define CM_BLOCK_SLOTS 1024
#endif

template <typename R> constexpr int kBlockThreads = CM_BLOCK_THREADS;
constexpr int kBlockSlots = CM_BLOCK_SLOTS;
constexpr int kBlockPerSm = CM_BLOCK_MINB;
// lists a slot can be in: the flights of each wave segment, the inelastic and the misc events, the flights
// that need the full form
constexpr int kListSlow = kSlowSegment, kListOpen = kOpenSegment, kListTab = kWaveSegments, kListMisc = kWaveSegments + 1, kListDead = kWaveSegments + 2;
constexpr int kLists = kWaveSegments + 3;
constexpr int kListNone = kLists;
// The list of a wave segment's electrons.  Over leaf shapes both kinds of full flights share one (a block has
// few of them; two lists: 8 % slower for the quick line scan), over trees, whose walks are long and unlike,
// each has its own (one list: 2 % slower for the FP64 image).
template <int D> __device__ __forceinline__ int block_list(int segment) {
  return D == 0 && segment == kOpenSegment ? kListSlow : segment;
}
// iterations after which a block passes what is left of the wave on to the next one instead of taking it
constexpr int kBlockHardLimit = 4096;

// control words of a block
struct BlockCtl {
  int cnt[2][kLists];  // entries of each list, this iteration's and the next one's
  int nfree;           // free slots (free_slot[0..nfree))
  int taken;           // of which secondaries have taken, from the top
  int task;            // next task of the iteration
  int claim_base, claim_n;
  int exhausted;       // the wave has no electron left to take
};

// The block's electrons: structure of arrays over its slots, in shared memory at fixed offsets (so that
// every access is a shared-memory instruction with an immediate offset).
template <typename R>
struct BlockMem {
  static constexpr int n = kBlockSlots;
  static constexpr int oKey = 24 * n, oR = 32 * n, oW = oR + 8 * n * (int)sizeof(R), oCtl = oW + 16 * n;
  static constexpr int oList = oCtl + ((int)sizeof(BlockCtl) + 15) / 16 * 16;
  static constexpr int oFree = oList + 2 * kLists * n * 2, oBorn = oFree + 2 * n, kBytes = oBorn + n;
  __device__ __forceinline__ static double& p(int a, int i) { return ((double*)cm_stage_smem)[a * n + i]; }
  __device__ __forceinline__ static unsigned long long& key(int i) { return ((unsigned long long*)(cm_stage_smem + oKey))[i]; }
  // direction 0..2, E 3, Ep 4, hit normal 5..7
  __device__ __forceinline__ static R& r(int a, int i) { return ((R*)(cm_stage_smem + oR))[a * n + i]; }
  // region 0, pixel 1, aux 2, step 3
  __device__ __forceinline__ static int& w(int a, int i) { return ((int*)(cm_stage_smem + oW))[a * n + i]; }
  __device__ __forceinline__ static BlockCtl& ctl() { return *(BlockCtl*)(cm_stage_smem + oCtl); }
  __device__ __forceinline__ static unsigned short& list(int par, int l, int i) {
    return ((unsigned short*)(cm_stage_smem + oList))[(par * kLists + l) * n + i];
  }
  __device__ __forceinline__ static unsigned short& free_slot(int i) { return ((unsigned short*)(cm_stage_smem + oFree))[i]; }
  // the slot holds a secondary started in this launch
  __device__ __forceinline__ static unsigned char& born(int i) { return (cm_stage_smem + oBorn)[i]; }

  __device__ __forceinline__ static El<R> load(int i) {
    El<R> e;
    for (int a = 0; a < 3; ++a) {
      e.p[a] = p(a, i);
      e.d[a] = r(a, i);
    }
    e.E = r(3, i);
    e.region = w(0, i); e.pixel = w(1, i);
    e.step = (uint32_t)w(3, i); e.key = key(i);
    return e;
  }
  __device__ __forceinline__ static void store(int i, const El<R>& e) {
    for (int a = 0; a < 3; ++a) {
      p(a, i) = e.p[a];
      r(a, i) = e.d[a];
    }
    r(3, i) = e.E;
    w(0, i) = e.region; w(1, i) = e.pixel;
    w(3, i) = (int)e.step; key(i) = e.key;
  }
  __device__ __forceinline__ static void put(int par, int l, int slot) {
    list(par, l, atomicAdd(&ctl().cnt[par][l], 1)) = (unsigned short)slot;
  }
};

// secondaries take a free slot of the block, or go to the run's pool when there is none
template <typename R, int D>
struct BlockSink : DeviceSink {
  int par;  // parity of the lists being filled
  __device__ __forceinline__ explicit BlockSink(int p) : par(p) {}
  __device__ __forceinline__ bool put_secondary(const RunView<R>& v, const El<R>& se) {
    using B = BlockMem<R>;
    const int k = atomicAdd(&B::ctl().taken, 1), avail = B::ctl().nfree;
    if (k >= avail) return pool_push(v, se, *this);
    const int slot = B::free_slot(avail - 1 - k);
    B::store(slot, se);
    B::born(slot) = 1;
    B::put(par, block_list<D>(wave_segment(v.s, se)), slot);
    return true;
  }
};

// One task: up to 32 electrons of one list through their flight (with the elastic event it ends in) or
// their queued event.  Every lane of the warp calls it; lanes without an electron have slot < 0.
template <typename R, int D>
__device__ __forceinline__ void block_task(const RunView<R>& v, int l, int slot, BlockSink<R, D>& sink, StepCounts& sc) {
  using B = BlockMem<R>;
  int dest = kListNone;
  if (slot >= 0) {
    El<R> e = B::load(slot);
    bool alive;
    dest = kListDead;
    if (l <= kListOpen) {
      const int q = l >= kListSlow ? flight_apply<R, D>(v, e, sink, sc) : flight_fast(v, e, sink, sc, [](El<R>&) {});
      alive = q >= 0;
      if (q == Q_EL) alive = elastic_apply(v, e);
      if (q == Q_SLOW) {
        dest = kListSlow;
      } else if (alive) {
        for (int a = 0; a < 3; ++a) B::p(a, slot) = e.p[a];
        B::r(3, slot) = e.E;
        B::w(0, slot) = e.region;
        B::w(3, slot) = (int)e.step;
        if (q == Q_EL) {
          for (int a = 0; a < 3; ++a) B::r(a, slot) = e.d[a];
        } else {
          B::r(4, slot) = e.Ep;
          B::w(2, slot) = e.aux;
          if (aux_kind(e.aux) == AUX_BARRIER)
            for (int a = 0; a < 3; ++a) B::r(5 + a, slot) = e.h[a];
        }
        // A step without mechanisms that stayed in its region has no event: its next flight, one iteration a
        // step.  (An electron in a vacuum region without a far end flies on to the limit of 10^6 steps: one B200,
        // 5.0 s through the misc list, 3.0 s so.)
        dest = q == Q_EL ? block_list<D>(segment_after(v.s, e))
               : q == Q_TAB ? kListTab
               : aux_kind(e.aux) == AUX_PASS ? block_list<D>(kOpenSegment)
                                             : kListMisc;
      }
    } else {
      e.Ep = B::r(4, slot);
      e.aux = B::w(2, slot);
      if (l == kListTab) {
        alive = inelastic_apply(v, e, sink, sc);
      } else {
        for (int a = 0; a < 3; ++a) e.h[a] = B::r(5 + a, slot);
        alive = misc_apply<R, D>(v, e, sink, sc);
        if (alive) {
          for (int a = 0; a < 3; ++a) B::p(a, slot) = e.p[a];
          B::w(0, slot) = e.region;
        }
      }
      if (alive) {
        for (int a = 0; a < 3; ++a) B::r(a, slot) = e.d[a];
        B::r(3, slot) = e.E;
        dest = block_list<D>(segment_after(v.s, e));
      }
    }
    if (!alive) job_end(v, e.pixel, e.step, sink);
  }
  // append the slots to their lists: one shared-memory atomic per list and warp
  __syncwarp();
  const unsigned same = __match_any_sync(0xffffffffu, dest);
  const int lane = threadIdx.x & 31, leader = __ffs(same) - 1;
  int base = 0;
  if (dest != kListNone && lane == leader) base = atomicAdd(&B::ctl().cnt[sink.par][dest], __popc(same));
  base = __shfl_sync(0xffffffffu, base, leader);
  if (dest != kListNone)
    B::list(sink.par, dest, base + __popc(same & ((1u << lane) - 1))) = (unsigned short)slot;
}

// The tasks of an iteration: 32 entries of one list each, events first (they take longest).  events_only:
// the flights stay in their lists.
template <typename R, int D>
__device__ __forceinline__ void block_stage(const RunView<R>& v, int par, bool events_only, BlockSink<R, D>& sink,
                                            StepCounts& sc) {
  using B = BlockMem<R>;
  // Lane k holds the k-th list in the order they are worked off (the longest tasks first), its entries and the
  // tasks up to its end; a task's list is then one ballot away.
  const int lane = threadIdx.x & 31;
  const int mine = lane == 0 ? kListTab : lane == 1 ? kListMisc : lane == 2 ? kListOpen : lane == 3 ? kListSlow : lane - 4;
  const int n = lane < kSegments + 4 && !(events_only && lane > 1) ? B::ctl().cnt[par][mine] : 0;
  int end = (n + 31) >> 5;
  for (int off = 1; off < 16; off <<= 1) {
    const int up = __shfl_up_sync(0xffffffffu, end, off);
    if (lane >= off) end += up;
  }
  const int begin = end - ((n + 31) >> 5);
  for (;;) {
    int t = 0;
    if (lane == 0) t = atomicAdd(&B::ctl().task, 1);
    t = __shfl_sync(0xffffffffu, t, 0);
    const unsigned after = __ballot_sync(0xffffffffu, t < end && lane < kSegments + 4);
    if (!after) return;
    const int k = __ffs(after) - 1;
    const int l = __shfl_sync(0xffffffffu, mine, k), i = 32 * (t - __shfl_sync(0xffffffffu, begin, k)) + lane;
    const int slot = i < __shfl_sync(0xffffffffu, n, k) ? (int)B::list(par, l, i) : -1;
    block_task<R, D>(v, l, slot, sink, sc);
  }
}

// Electrons of wave `cur` through about `iters` iterations (a flight with its elastic event, or a queued
// event, per electron and iteration), survivors kept in the next wave.  cap: slots a block may use.
template <typename R, int D>
__global__ void __launch_bounds__(kBlockThreads<R>, kBlockPerSm) k_block(const __grid_constant__ RunView<R> v, int cur, int iters, int cap) {
  using B = BlockMem<R>;
  BlockCtl& c = B::ctl();
  const int n = v.c->n[cur];
  const int grid = gridDim.x, tid = threadIdx.x, T = kBlockThreads<R>;
  if (n == 0) return;
  __shared__ int first[kWaveSegments + 1];
  segment_starts(v.c, cur, first);
  // The first share: every block takes the same number of electrons, in runs of `run` from all over the
  // wave, so that the blocks get like mixes of materials and energies
  const int reserve = cap / 8;
  int quota = (n + grid - 1) / grid;
  const int run = quota >= 64 ? 8 : 1;
  quota = (quota + run - 1) / run * run;
  if (quota > cap - reserve) quota = (cap - reserve) / run * run;
  const long long dealt = (long long)quota * grid;
  for (int i = tid; i < cap; i += T) B::free_slot(i) = (unsigned short)(cap - 1 - i);
  for (int i = tid; i < 2 * kLists; i += T) (&c.cnt[0][0])[i] = 0;
  __syncthreads();
  int mine = 0;  // electrons of the share that exist
  {
    // slots [0, quota) of the share; slot j holds electron (j / run * grid + block) * run + j % run
    const int whole = n / (run * grid) * run;
    const int rest = n - n / (run * grid) * (run * grid) - (int)blockIdx.x * run;
    mine = whole + (rest < 0 ? 0 : rest > run ? run : rest);
    if (mine > quota) mine = quota;
  }
  auto take = [&](int i, int slot, int par) {
    const int k = segment_of(first, i);
    const El<R> e = load_live(v.now, k * v.W + (i - first[k]));
    B::store(slot, e);
    B::born(slot) = 0;
    B::put(par, block_list<D>(k), slot);
  };
  for (int j = tid; j < mine; j += T) take((j / run * grid + (int)blockIdx.x) * run + j % run, j, 0);
  if (tid == 0) {
    c.nfree = cap - mine;
    c.taken = 0;
    c.task = 0;
    c.claim_n = 0;
    c.exhausted = dealt >= n;
  }
  __syncthreads();
  StepCounts sc;
  int par = 0, it = 0;
  for (;; ++it) {
    // the last iteration runs the queued events only, so that every electron ends between two steps
    const bool out = c.exhausted != 0;
    const bool last = (c.nfree == cap && out) || (it >= iters && out) || it >= kBlockHardLimit;
    BlockSink<R, D> sink(par ^ 1);
    block_stage<R, D>(v, par, last, sink, sc);
    __syncthreads();
    if (last) break;
    // free slots: those the secondaries took are gone, those of the electrons that ended come back
    const int avail = c.nfree, tk = c.taken < avail ? c.taken : avail, nd = c.cnt[par ^ 1][kListDead];
    for (int i = tid; i < nd; i += T) B::free_slot(avail - tk + i) = B::list(par ^ 1, kListDead, i);
    __syncthreads();
    if (tid < kLists) c.cnt[par][tid] = 0;
    if (tid == 0) {
      const int nf = avail - tk + nd, want = nf - reserve;
      int m = 0;
      if (!out && (want >= 32 || nf == cap)) {
        const long long base = dealt + atomicAdd(&v.c->claim.v, want);
        m = base >= n ? 0 : (n - base < want ? (int)(n - base) : want);
        c.claim_base = (int)base;
        if (base + want >= n) c.exhausted = 1;
      }
      c.claim_n = m;
      c.nfree = nf - m;
      c.taken = 0;
      c.task = 0;
      c.cnt[par ^ 1][kListDead] = 0;
    }
    __syncthreads();
    const int m = c.claim_n;
    if (m > 0) {
      for (int i = tid; i < m; i += T) take(c.claim_base + i, B::free_slot(c.nfree + i), par ^ 1);
      __syncthreads();
    }
    par ^= 1;
  }
  // every electron that is left goes to the next wave (secondaries started here to the pool, whose refill
  // keeps the wave within its bound)
  {
    DeviceSink sink;
    for (int h = 0; h < 2; ++h)
      for (int l = 0; l < kWaveSegments; ++l) {
        const int p = par ^ h, k = c.cnt[p][l];
        for (int i = tid; i < k; i += T) {
          const int slot = B::list(p, l, i);
          const El<R> e = B::load(slot);
          if (B::born(slot)) pool_push(v, e, sink);
          else keep(v, cur ^ 1, e, l, sink);
        }
      }
    // a wave this launch did not get through is passed on as it is
    while (!c.exhausted) {
      __syncthreads();
      if (tid == 0) {
        const long long base = dealt + atomicAdd(&v.c->claim.v, 4096);
        c.claim_n = base >= n ? 0 : (n - base < 4096 ? (int)(n - base) : 4096);
        c.claim_base = (int)base;
        if (base + 4096 >= n) c.exhausted = 1;
      }
      __syncthreads();
      for (int i = tid; i < c.claim_n; i += T) {
        const int w = c.claim_base + i, k = segment_of(first, w);
        keep(v, cur ^ 1, load_live(v.now, k * v.W + (w - first[k])), k, sink);
      }
      __syncthreads();
    }
  }
  flush_counts(v.c, sc);
}

// Slots per block: all of them, or fewer for a small wave, so that the blocks together hold about a wave of
// electrons at most: the secondary pool is sized by the wave, and what the blocks hold may end in it.
static int block_cap(int held, int grid) {
  const int cap = held / grid;
  return cap > kBlockSlots ? kBlockSlots : cap < 1 ? 1 : cap;
}

template <typename R, int D>
static void launch_block_d(const RunView<R>& v, int cur, int nsm, int iters, cudaStream_t s, int held) {
  const int grid = nsm * kBlockPerSm;
  cudaFuncSetAttribute(k_block<R, D>, cudaFuncAttributeMaxDynamicSharedMemorySize, BlockMem<R>::kBytes);
  k_block<R, D><<<grid, kBlockThreads<R>, BlockMem<R>::kBytes, s>>>(v, cur, iters, block_cap(held, grid));
}

// held: electrons the blocks may hold together (0: a wave)
template <typename R>
static void launch_block(const RunView<R>& v, int cur, int nsm, int iters, cudaStream_t s, int held = 0) {
  if (held <= 0) held = v.W;
  if (v.s.depth == 0) launch_block_d<R, 0>(v, cur, nsm, iters, s, held);
  else if (v.s.depth <= 2) launch_block_d<R, 2>(v, cur, nsm, iters, s, held);
  else launch_block_d<R, kMaxShapeDepth>(v, cur, nsm, iters, s, held);
}

}  // namespace cm
