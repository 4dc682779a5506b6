// Grid-wide finish of a max reduction inside one launch, and a bounded grid barrier.
//
// Each block publishes one partial and takes a ticket; the block that draws the last ticket
// reduces all partials.  No output has to be pre-initialised and the workspace is left ready for
// the next launch.  Waiting (only the fused ops wait) is a bounded spin: if what is waited for
// does not come within the limit, the waiter records DTQ_ERR_TIMEOUT in the workspace and the
// block returns, so a launch can never hang the device.
#pragma once

#include "dtq_device.cuh"
#include "dtq_host.h"

namespace dtq {

__device__ __forceinline__ unsigned int ld_acquire(const unsigned int *p) {
  unsigned int v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ float ld_relaxed_f32(const float *p) {
  float v;
  asm volatile("ld.relaxed.gpu.global.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
  return v;
}

// Publishes `block_value` (meaningful in thread 0) and returns, in every thread of the block,
// whether this block arrived last.  `flag` is one int of shared memory.
__device__ __forceinline__ bool publish_and_ticket(Workspace *ws, float block_value, int *flag) {
  if (threadIdx.x == 0) {
    ws->partials[blockIdx.x] = block_value;
    __threadfence();
    const unsigned int ticket = atomicAdd(&ws->arrivals, 1u);
    *flag = (ticket == gridDim.x - 1);
  }
  __syncthreads();
  const bool last = *flag != 0;
  __syncthreads();
  return last;
}

// Run by every thread of the last block: max over all blocks' partials (valid in warp 0).
__device__ __forceinline__ float reduce_partials(const Workspace *ws, float *smem32, float identity) {
  __threadfence();
  float v = identity;
  for (unsigned int i = threadIdx.x; i < gridDim.x; i += blockDim.x) v = fmaxf(v, ld_relaxed_f32(&ws->partials[i]));
  return block_max_nonneg(v, smem32, identity);
}

constexpr unsigned int kSpinLimit = 1u << 20;  // polls, each an L2 round trip plus a short sleep: gives up after about a second

// ---- a grid that meets without having to be resident as a whole -----------------------------------------------------
// Every block of the fused kernel owns a share of the input, adds its share's maximum, and waits until all shares are in.  A
// cooperative launch would make sure that all blocks are there; but in a stream of such launches it costs 2 to 3 us each
// (dsq_fused_kernel has the figures).  Without it some blocks may not have started, because another stream's kernel holds
// their SM, and it may hold it for as long as it likes, or wait in turn for an SM that this grid holds.  So nobody waits for a
// block that has not started: a block claims its share when it starts, a block that has waited for some time takes over
// shares that nobody has claimed, and a block that starts and finds its share taken leaves.  All who are waited for are running.
//
// A share's word counts, in twos, the launches that its owner has come to; the lowest bit says that another block has taken the share over
// in the launch that the owner has not come to yet, and goes when the owner comes.  Every launch counts on in all kMaxShares words,
// so a block knows from its own which launch this is, and of another share's whether its owner has come: nothing is cleared between
// launches, and a block that is late or gives up leaves nothing behind.
//
// A share that was claimed goes in, sooner or later, also when the waiting of others has run out, so the count of shares is
// complete when the launch is over.  Who gives up notes it in the same word, unless the count is complete by then: all who see it complete
// know whether all have met.
constexpr unsigned int kTakenOver = 1, kLaunch = 2;
constexpr unsigned int kOneGaveUp = 1u << 16;  // in shares_in, above the count
static_assert(kMaxShares < kOneGaveUp && int64_t(kMaxShares) * kOneGaveUp <= 0xFFFFFFFFll - kMaxShares, "the halves of shares_in");
constexpr int kGaveUp = 0, kMet = 1, kImpatient = 2, kShareIsGone = 3;
constexpr unsigned int kPatience = 64;  // polls, about 50 us, before a waiting block looks for shares to take over

// Thread 0 of the owner, first thing.  The launch, in twos; with kTakenOver: the share is another block's by now, nothing is left to do.  (The
// block reads it all the same before it looks: a barrier in front of the second tile cost inputs of 16 to 32 MiB 2 to 5 %, and saved 9 % of
// 1 GiB in 1024 blocks, of which 296 fit.)
__device__ __forceinline__ unsigned int come_for_own_share(Workspace *ws) {
  const unsigned int before = atomicAdd(&ws->shares[blockIdx.x], kLaunch);
  if (before & kTakenOver) atomicSub(&ws->shares[blockIdx.x], kTakenOver);
  return before;
}
// All threads: this launch in the words that are no block's.
__device__ __forceinline__ void count_unused_shares(Workspace *ws) {
  for (unsigned int j = blockIdx.x + (threadIdx.x + 1) * gridDim.x; j < kMaxShares; j += blockDim.x * gridDim.x)
    atomicAdd(&ws->shares[j], kLaunch);
}
__device__ __forceinline__ unsigned int parity_of(unsigned int launch) { return launch / kLaunch & 1u; }
__device__ __forceinline__ bool all_in(unsigned int shares_in) { return (shares_in & (kOneGaveUp - 1)) == gridDim.x; }
// What a block knows of the launch from shares_in.
__device__ __forceinline__ int meeting(unsigned int shares_in) {
  return !all_in(shares_in) ? kImpatient : shares_in == gridDim.x ? kMet : kGaveUp;
}
// Thread 0: a share's maximum goes in.  The last one clears the other parity's pair (the previous launch is long over).
__device__ __forceinline__ int add_share(Workspace *ws, unsigned int launch, float value) {
  const unsigned int slot = parity_of(launch);
  atomicMax(&ws->shares_max[slot], __float_as_uint(value));
  __threadfence();
  const unsigned int in = atomicAdd(&ws->shares_in[slot], 1u) + 1u;
  if (!all_in(in)) return kImpatient;
  ws->shares_in[slot ^ 1u] = 0;
  ws->shares_max[slot ^ 1u] = 0;
  __threadfence();  // as the acquiring load of those who wait
  return meeting(in);
}
// Thread 0: waits for all shares, for at most `polls`.
__device__ __forceinline__ int wait_for_shares(const Workspace *ws, unsigned int launch, unsigned int polls) {
  const unsigned int *word = &ws->shares_in[parity_of(launch)];
  int met;
  for (unsigned int spins = 0; (met = meeting(ld_acquire(word))) == kImpatient;) {
    if (++spins > polls) break;
    __nanosleep(20);
  }
  return met;
}
// Thread 0, when it has waited long enough.
__device__ __forceinline__ int give_up_shares(Workspace *ws, unsigned int launch) {
  unsigned int *word = &ws->shares_in[parity_of(launch)];
  for (unsigned int before = ld_acquire(word); !all_in(before);) {  // the word changes at most twice for each block
    const unsigned int now = atomicCAS(word, before, before + kOneGaveUp);
    if (now == before) {
      atomicExch(&ws->status, DTQ_ERR_TIMEOUT);
      return kGaveUp;
    }
    before = now;
  }
  return wait_for_shares(ws, launch, 0);
}
// Thread 0, when all have met: the maximum.
__device__ __forceinline__ float shares_maximum(const Workspace *ws, unsigned int launch) {
  return __uint_as_float(ld_acquire(&ws->shares_max[parity_of(launch)]));
}

// What a block took over (shared memory; a bit per share).
struct TakenShares {
  int candidate;
  int taken;
  unsigned int bits[kMaxShares / 32];
  template <typename F>
  __device__ __forceinline__ void for_each(F f) const {
    for (int w = 0; w < kMaxShares / 32; ++w)
      for (unsigned int left = bits[w]; left; left &= left - 1) f(w * 32 + __ffs(int(left)) - 1);
  }
};
// All threads of a block that has waited in vain: takes over shares until all are in.  share_max(share) is the share's
// maximum as block_max_nonneg returns it.  kMet, or kGaveUp: after kSpinLimit polls without a share to take, or where another gave up.
template <typename ShareMax>
__device__ __forceinline__ int take_over_until_met(Workspace *ws, unsigned int launch, TakenShares &mine, ShareMax share_max) {
  if (threadIdx.x < kMaxShares / 32) mine.bits[threadIdx.x] = 0;
  const unsigned int shortened = *const_cast<const volatile unsigned int *>(&ws->wait_limit_us);
  const unsigned int limit = shortened ? shortened : kSpinLimit;  // a poll takes about a microsecond
  unsigned int spins = 0;
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) mine.candidate = -1;
    __syncthreads();
    // of the shares that nobody has come for, the one farthest behind this block's own: blocks spread out
    int best = -1;
    for (unsigned int j = threadIdx.x; j < gridDim.x; j += blockDim.x)
      if (ld_acquire(&ws->shares[j]) == launch) best = max(best, int((j + gridDim.x - blockIdx.x) % gridDim.x));
    if (best >= 0) atomicMax(&mine.candidate, best);
    __syncthreads();
    if (threadIdx.x == 0) {
      mine.taken = -1;
      if (mine.candidate >= 0) {
        const unsigned int j = (mine.candidate + blockIdx.x) % gridDim.x;
        if (atomicCAS(&ws->shares[j], launch, launch + kTakenOver) == launch) mine.taken = int(j);
      }
    }
    __syncthreads();
    const int j = mine.taken;
    if (j >= 0) {
      const float value = share_max(j);
      if (threadIdx.x == 0) {
        mine.bits[j / 32] |= 1u << (j & 31);
        add_share(ws, launch, value);
      }
    }
    const bool wait = j < 0;  // (after a share taken: only a look)
    if (wait) spins += kPatience;
    if (threadIdx.x == 0) {
      int met = wait_for_shares(ws, launch, wait ? kPatience : 0);
      if (met == kImpatient && wait && spins > limit) met = give_up_shares(ws, launch);
      mine.candidate = met;
    }
    __syncthreads();
    const int met = mine.candidate;
    if (met != kImpatient) return met;
  }
}

// ---- a grid barrier with an exchange across GPUs in its serial section -------------------------
// Every rank (one process per GPU, same launch on each) owns a small exchange buffer that all
// peers can address over NVLink: kPeerParities x kMaxPeers 64-bit slots.  The last block to arrive
// at the local barrier stores {epoch, local maximum} into its slot of EVERY rank's buffer
// (st.release.sys, plain peer stores) and then reads its own buffer until all `world` slots carry
// this launch's epoch (ld.acquire.sys, bounded spin).  The slot parity alternates with the epoch,
// so a fast peer's next launch can never overwrite a value a slow rank has not read yet (a rank
// cannot get two launches ahead: it needs this rank's next value first).  Nothing is ever reset.
constexpr int kMaxPeers = 16;
constexpr int kPeerParities = 2;

struct PeerExchange {
  unsigned long long *buffer[kMaxPeers];  // entry r: rank r's exchange buffer as mapped on this device
  int rank, world;
  unsigned int epoch;       // same on every rank for the same launch, increasing by one per launch
  unsigned int spin_limit;  // polls before a wait gives up
};

__device__ __forceinline__ void st_release_sys(unsigned long long *p, unsigned long long v) {
  asm volatile("st.release.sys.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ void st_relaxed_sys(unsigned long long *p, unsigned long long v) {
  asm volatile("st.relaxed.sys.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned long long ld_relaxed_sys(const unsigned long long *p) {
  unsigned long long v;
  asm volatile("ld.relaxed.sys.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned long long ld_acquire_sys(const unsigned long long *p) {
  unsigned long long v;
  asm volatile("ld.acquire.sys.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

// The exchange alone, for a kernel without a grid barrier: run by all 32 lanes of one warp of one
// block per rank.  Stores {epoch, local_bits} into this rank's slot on every rank and returns the
// maximum of all ranks' values for this epoch (unsigned order); *ok is false if a peer's value did
// not arrive within the spin limit.
__device__ __forceinline__ unsigned int peer_exchange_max(const PeerExchange &px, unsigned int local_bits, bool *ok) {
  const int lane = threadIdx.x & 31;
  const int parity = px.epoch & 1u;
  unsigned int value = 0;
  bool mine_ok = true;
  if (lane < px.world) {
    // The 64-bit word {epoch, value} is the whole message: one store, one load, nothing else to order against it
    // (a release / acquire pair at system scope costs a fence on each side of the link).
    st_relaxed_sys(px.buffer[lane] + parity * kMaxPeers + px.rank,
                   (static_cast<unsigned long long>(px.epoch) << 32) | local_bits);
    const unsigned long long *mine = px.buffer[px.rank] + parity * kMaxPeers + lane;
    unsigned int spins = 0;
    unsigned long long v = ld_relaxed_sys(mine);
    while (static_cast<unsigned int>(v >> 32) != px.epoch) {
      if (++spins > px.spin_limit) {
        mine_ok = false;
        break;
      }
      __nanosleep(40);
      v = ld_relaxed_sys(mine);
    }
    value = static_cast<unsigned int>(v);
  }
  *ok = __all_sync(0xFFFFFFFFu, mine_ok);
  return __reduce_max_sync(0xFFFFFFFFu, value);
}

// For a grid whose blocks are all resident (a cooperative launch): the maximum over all blocks of all ranks.  `gen0` is the generation word as
// read by thread 0 BEFORE the block did anything else.  Returns false on timeout (status word set, nothing may be assumed about
// `*result`).
// Waiting blocks watch the local count reach gridDim.x + 1: the last arriver adds the extra one
// after the exchange, when ws->amax holds the global value.
__device__ __forceinline__ bool grid_max_barrier_exchange(Workspace *ws, unsigned int gen0, float block_value,
                                                          const PeerExchange &px, int *flag, float *shared_result,
                                                          float *result) {
  if (threadIdx.x < 32) {  // warp 0; lane 0 runs the local protocol, lanes < world the exchange
    const unsigned int slot = gen0 & 1u;
    const int lane = threadIdx.x;
    unsigned int ticket = 0;
    if (lane == 0) {
      atomicMax(&ws->bar_max[slot], __float_as_uint(block_value));
      __threadfence();
      ticket = atomicAdd(&ws->bar_count[slot], 1u);
    }
    ticket = __shfl_sync(0xFFFFFFFFu, ticket, 0);
    bool ok = true;
    if (ticket == gridDim.x - 1) {
      unsigned int local_bits = 0;
      if (lane == 0) {
        __threadfence();
        local_bits = ld_acquire(&ws->bar_max[slot]);
      }
      local_bits = __shfl_sync(0xFFFFFFFFu, local_bits, 0);
      const int parity = px.epoch & 1u;
      unsigned int global_bits = 0;
      if (lane < px.world) {
        st_release_sys(px.buffer[lane] + parity * kMaxPeers + px.rank,
                       (static_cast<unsigned long long>(px.epoch) << 32) | local_bits);
        const unsigned long long *mine = px.buffer[px.rank] + parity * kMaxPeers + lane;
        unsigned int spins = 0;
        unsigned long long v = ld_acquire_sys(mine);
        while (static_cast<unsigned int>(v >> 32) != px.epoch) {
          if (++spins > px.spin_limit) {
            ok = false;
            break;
          }
          __nanosleep(40);
          v = ld_acquire_sys(mine);
        }
        global_bits = static_cast<unsigned int>(v);
      }
      ok = __all_sync(0xFFFFFFFFu, ok);
      global_bits = __reduce_max_sync(0xFFFFFFFFu, global_bits);  // non-negative floats order like their bits
      if (lane == 0) {
        if (!ok) atomicExch(&ws->status, DTQ_ERR_TIMEOUT);
        ws->amax = ok ? __uint_as_float(global_bits) : 0.0f;
        ws->bar_count[slot ^ 1u] = 0;
        ws->bar_max[slot ^ 1u] = 0;
        atomicAdd(&ws->generation, 1u);
        __threadfence();
        // release the local waiters; on failure with a count they recognise as "gave up"
        atomicAdd(&ws->bar_count[slot], ok ? 1u : 2u);
      }
    } else if (lane == 0) {
      unsigned int spins = 0;
      unsigned int c = ld_acquire(&ws->bar_count[slot]);
      while (c <= gridDim.x) {
        if (++spins > kSpinLimit + px.spin_limit) {
          atomicExch(&ws->status, DTQ_ERR_TIMEOUT);
          break;
        }
        __nanosleep(20);
        c = ld_acquire(&ws->bar_count[slot]);
      }
      ok = c == gridDim.x + 1;
    }
    if (lane == 0) {
      __threadfence();
      *shared_result = ld_relaxed_f32(&ws->amax);
      *flag = ok;
    }
  }
  __syncthreads();
  *result = *shared_result;
  const bool ok = *flag != 0;
  __syncthreads();
  return ok;
}

}  // namespace dtq
