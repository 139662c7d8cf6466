// MSCCL-IR interpreter for programs whose ranks all live on this GPU (Communicator.emulated).  Same contract as
// exec_kernel.cu - steps of a threadblock in order, the program's protocol, FIFOs, credits, bounds checks, bounded
// waits, bit-identical sums - but laid out for one device:
//
//   * Slices.  Every step works element by element, so a chunk is cut into K slices that never meet: K CTAs run one
//     threadblock, each on its own slice, with its own FIFO slots, counters and progress word.  One CTA per SM (the
//     layout of exec_kernel.cu) leaves the SMs of idle receivers empty and pays every flag round trip in full; four CTAs
//     of 256 threads per SM hide them behind each other.
//   * Roles.  Six data warps move; a control warp polls the flags of the next steps, one flag per lane, and hands
//     the finished job (pointers, sizes) to the data warps; a signal warp fences and publishes what a step finished while
//     the data warps are in the next one.  Jobs are double buffered: control runs up to two steps ahead.
//   * Scope.  All flags are read and written at GPU scope: a system-scope fence costs more and orders nothing extra here.
//   * No drain: the FIFO contents cannot be wanted after the kernel's end, because every receiver is part of it.  No
//     opening handshake for slots that nothing touches before their receive (SF_DIRECT_ALWAYS): every rank's earlier
//     work on this GPU is done when the kernel runs.
//   * The rank table travels in the kernel parameters: no device copy per set of buffers, nothing kept by address.
//
// Bound by L2 / HBM traffic from about 1 MB per chunk on, by the flag round trips (store, fence, poll: about 1.5 us a
// hop) below.
#include <cstdio>

#include "exec_common.cuh"
#include "msccl_device.h"
#include "prims.cuh"

namespace msccl {

namespace {

constexpr int kOgDataWarps = 6;
constexpr int kOgData = kOgDataWarps * 32;      // threads that move
constexpr int kOgThreads = kOgData + 64;        // + control warp + signal warp
constexpr int kOgCtasPerSm = 4;
constexpr int kOgSmemSteps = 128;

enum JobKind : int { JOB_EXIT = 0, JOB_NONE, JOB_MOVE, JOB_BATCH, JOB_SEND, JOB_RECV, JOB_BOTH };

struct __align__(16) Job {
  const char* in;                 // local source / destination slot already holding the data / FIFO packets
  const char* add;                // second operand or null
  char* out0;                     // local destination or null
  char* out1;                     // FIFO slot or the receiver's slot, or null
  long long in_step, add_step, out0_step, out1_step;      // bytes from one chunk of the step to the next
  const char* src[kMaxBatch];     // JOB_BATCH
  long long src_step;
  int kind, cnt, n, nsrc;         // n: accesses (LL128: 8-byte units) per chunk
  unsigned int flag_in, flag_out;
  unsigned long long flag_in128, flag_out128;
  // what the signal warp publishes
  int fence, step, steps, iter;   // first step of the pass and how many (nops in front and batch members included)
  unsigned long long tail, credit, opened, progress;     // 0: nothing to publish
  unsigned long long t0, t1;      // trace
};

struct Shared {
  Job job[2];
  unsigned long long go[2], done[2];     // mbarriers
  int fail;                              // a flag-in-data poll or a wait ran out of time
  int signalled;                         // passes the signal warp has finished with
  DevStep steps[kOgSmemSteps];
};

__device__ __forceinline__ void fence_acq_rel_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
__device__ __forceinline__ unsigned int smem_addr(const void* p) { return static_cast<unsigned int>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void bar_init(unsigned long long* b, unsigned int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_arrive(unsigned long long* b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(b)) : "memory");
}
__device__ __forceinline__ bool bar_try(unsigned long long* b, unsigned int parity) {
  unsigned int ok;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(ok) : "r"(smem_addr(b)), "r"(parity) : "memory");
  return ok != 0;
}
// Bounded: the limit lies a second behind the launch's own, which ends every wait of the control and data warps.
__device__ __forceinline__ bool bar_wait(unsigned long long* b, unsigned int parity, unsigned long long limit) {
  for (unsigned int i = 1;; ++i) {
    if (bar_try(b, parity)) return true;
    if ((i & 255u) == 0 && global_timer_ns() > limit) return false;
  }
}

// out = in0 (+ add1), to one or two places; U loads per operand and thread in flight.  Behind the end the last access is
// loaded again instead of none: no branch between the loads, only the stores are predicated.
template <typename T, int W, int U, bool ADD>
__device__ __forceinline__ void og_move(const char* in0, const char* add1, char* out0, char* out1, int n) {
  using VT = typename Wide<T, W>::V;
#pragma unroll 1
  for (int base = threadIdx.x; base < n; base += kOgData * U) {
    VT val[U];
#pragma unroll
    for (int u = 0; u < U; ++u) val[u] = Access<W>::ld(in0 + static_cast<long long>(min(base + u * kOgData, n - 1)) * W);
    if (ADD) {
      VT other[U];
#pragma unroll
      for (int u = 0; u < U; ++u) other[u] = Access<W>::ld(add1 + static_cast<long long>(min(base + u * kOgData, n - 1)) * W);
#pragma unroll
      for (int u = 0; u < U; ++u) val[u] = Wide<T, W>::add(val[u], other[u]);
    }
    if (out0 != nullptr) {
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (base + u * kOgData < n) Access<W>::st(out0 + static_cast<long long>(base + u * kOgData) * W, val[u]);
    }
    if (out1 != nullptr) {
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (base + u * kOgData < n) Access<W>::st(out1 + static_cast<long long>(base + u * kOgData) * W, val[u]);
    }
  }
}

// dst = ((dst + src_0) + src_1) + ..., rounded after every addition; all operands of an element in flight together
// (operands the step does not have read dst again)
template <typename T, int W>
__device__ __forceinline__ void og_batch(char* dst, const char* const* srcs, long long src_off, int nsrc, int n) {
  using VT = typename Wide<T, W>::V;
#pragma unroll 1
  for (int v = threadIdx.x; v < n; v += kOgData) {
    const long long at = static_cast<long long>(v) * W;
    VT acc = Access<W>::ld(dst + at);
    VT other[kMaxBatch];
#pragma unroll
    for (int k = 0; k < kMaxBatch; ++k) other[k] = Access<W>::ld((k < nsrc ? srcs[k] + src_off : dst) + at);
#pragma unroll
    for (int k = 0; k < kMaxBatch; ++k)
      if (k < nsrc) acc = Wide<T, W>::add(acc, other[k]);
    Access<W>::st(dst + at, acc);
  }
}

// ---- LL packets: U packets per thread polled together (LLPacket<W>::load waits for one after the other) ------------
template <int W> struct Packets;
template <> struct Packets<16> {
  uint4 a, b;
  __device__ __forceinline__ void load(const char* slot, long long v) {
    const uint4* p = reinterpret_cast<const uint4*>(slot) + 2 * v;
    a = ld_volatile_v4(p);
    b = ld_volatile_v4(p + 1);
  }
  __device__ __forceinline__ bool ready(unsigned int f) const { return a.y == f && a.w == f && b.y == f && b.w == f; }
  __device__ __forceinline__ uint4 data() const { return make_uint4(a.x, a.z, b.x, b.z); }
};
template <int W> struct PacketsNarrow {
  uint2 a;
  __device__ __forceinline__ void load(const char* slot, long long v) { a = ld_volatile_v2(reinterpret_cast<const uint2*>(slot) + v); }
  __device__ __forceinline__ bool ready(unsigned int f) const { return a.y == f; }
  __device__ __forceinline__ typename LLPacketNarrow<W>::VT data() const { return static_cast<typename LLPacketNarrow<W>::VT>(a.x); }
};
template <> struct Packets<4> : PacketsNarrow<4> {};
template <> struct Packets<2> : PacketsNarrow<2> {};

template <typename T, int W, bool FIFO_IN, bool FIFO_OUT>
__device__ __forceinline__ void og_move_ll(const char* in, const char* add1, char* out0, char* fifo_out, int n,
                                           unsigned int flag_in, unsigned int flag_out, const Waiter& w, int* fail) {
  using VT = typename Wide<T, W>::V;
  constexpr int U = W == 16 ? 2 : 4;
#pragma unroll 1
  for (int base = threadIdx.x; base < n; base += kOgData * U) {
    VT val[U];
    if (FIFO_IN) {
      Packets<W> pk[U];
      for (unsigned int spins = 1;; ++spins) {
        bool ready = true;
#pragma unroll
        for (int u = 0; u < U; ++u) pk[u].load(in, min(base + u * kOgData, n - 1));
#pragma unroll
        for (int u = 0; u < U; ++u) ready = ready && pk[u].ready(flag_in);
        if (ready) break;
        if ((spins & 127u) == 0 && (*reinterpret_cast<volatile int*>(fail) != 0 || w.expired())) {
          *reinterpret_cast<volatile int*>(fail) = 1;
          break;
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) val[u] = pk[u].data();
    } else {
#pragma unroll
      for (int u = 0; u < U; ++u) val[u] = Access<W>::ld(in + static_cast<long long>(min(base + u * kOgData, n - 1)) * W);
    }
    if (add1 != nullptr) {
      VT other[U];
#pragma unroll
      for (int u = 0; u < U; ++u) other[u] = Access<W>::ld(add1 + static_cast<long long>(min(base + u * kOgData, n - 1)) * W);
#pragma unroll
      for (int u = 0; u < U; ++u) val[u] = Wide<T, W>::add(val[u], other[u]);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (base + u * kOgData < n) {
        if (out0 != nullptr) Access<W>::st(out0 + static_cast<long long>(base + u * kOgData) * W, val[u]);
        if (FIFO_OUT) LLPacket<W>::store(fifo_out, base + u * kOgData, val[u], flag_out);
      }
    }
  }
}

// ---- LL128 lines: eight lanes per line, see exec_common.cuh -------------------------------------------------------
template <typename T, bool FIFO_IN, bool FIFO_OUT>
__device__ __forceinline__ void og_move_ll128(const char* in, const char* add1, char* out0, char* fifo_out, int n8,
                                              unsigned long long flag_in, unsigned long long flag_out, const Waiter& w, int* fail) {
  const int k = threadIdx.x & 7, g = threadIdx.x >> 3;
  constexpr int kGroups = kOgData / 8;
  const int lines = (n8 + 14) / 15;
  const unsigned int in_lo = static_cast<unsigned int>(flag_in), in_hi = static_cast<unsigned int>(flag_in >> 32);
  constexpr int U = 4;
#pragma unroll 1
  for (int l0 = g; l0 < (lines + g); l0 += kGroups * U) {     // the same trip count for every thread
    uint4 val[U];
    if (FIFO_IN) {
      for (unsigned int spins = 1;; ++spins) {
        bool ready = true;
#pragma unroll
        for (int u = 0; u < U; ++u)
          val[u] = ld_volatile_v4(reinterpret_cast<const uint4*>(in + static_cast<long long>(min(l0 + u * kGroups, lines - 1)) * 128 + k * 16));
#pragma unroll
        for (int u = 0; u < U; ++u) ready = ready && (k != 7 || (val[u].z == in_lo && val[u].w == in_hi));
        // the flag vouches for the other seven lanes' part of its line: all look again until every line of the warp is there
        if (__all_sync(kFullWarp, ready)) break;
        if ((spins & 63u) == 0) {
          const bool give_up = (threadIdx.x & 31) == 0 && (*reinterpret_cast<volatile int*>(fail) != 0 || w.expired());
          if (__any_sync(kFullWarp, give_up)) {
            *reinterpret_cast<volatile int*>(fail) = 1;
            break;
          }
        }
      }
    } else {
#pragma unroll
      for (int u = 0; u < U; ++u) val[u] = ld_units(in, static_cast<long long>(min(l0 + u * kGroups, lines - 1)) * 15 + 2 * k, n8, k);
    }
    if (add1 != nullptr) {
      uint4 other[U];
#pragma unroll
      for (int u = 0; u < U; ++u) other[u] = ld_units(add1, static_cast<long long>(min(l0 + u * kGroups, lines - 1)) * 15 + 2 * k, n8, k);
#pragma unroll
      for (int u = 0; u < U; ++u) val[u] = Vec16<T>::add(val[u], other[u]);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int line = l0 + u * kGroups;
      if (line < lines) {
        if (out0 != nullptr) st_units(out0, static_cast<long long>(line) * 15 + 2 * k, n8, k, val[u]);
        if (FIFO_OUT) {
          uint4 v = val[u];
          if (k == 7) {
            v.z = static_cast<unsigned int>(flag_out);
            v.w = static_cast<unsigned int>(flag_out >> 32);
          }
          st_volatile_v4(reinterpret_cast<uint4*>(fifo_out + static_cast<long long>(line) * 128 + k * 16), v);
        }
      }
    }
  }
}

// ------------------------------------------------------------------------------------------------------ the roles
template <typename T, int PROTO, int W>
__device__ __forceinline__ void data_role(Shared& sh, const Waiter& w, unsigned long long limit) {
  for (unsigned int pass = 0;; ++pass) {
    const Job& job = sh.job[pass & 1];
    if (!bar_wait(&sh.go[pass & 1], (pass >> 1) & 1u, limit)) return;
    const int kind = job.kind;
    if (kind >= JOB_MOVE) {
      const int cnt = job.cnt, n = job.n;
      for (int j = 0; j < cnt; ++j) {
        const char* in = job.in + j * job.in_step;
        const char* add = job.add != nullptr ? job.add + j * job.add_step : nullptr;
        char* out0 = job.out0 != nullptr ? job.out0 + j * job.out0_step : nullptr;
        char* out1 = job.out1 != nullptr ? job.out1 + j * job.out1_step : nullptr;
        if (kind == JOB_BATCH) {
          og_batch<T, W>(out0, job.src, j * job.src_step, job.nsrc, n);
        } else if (PROTO == PROTO_SIMPLE || kind == JOB_MOVE) {
          if (add != nullptr) og_move<T, W, 4, true>(in, add, out0, out1, n);
          else og_move<T, W, 8, false>(in, nullptr, out0, out1, n);
        } else if constexpr (PROTO == PROTO_LL) {
          if (kind == JOB_SEND) og_move_ll<T, W, false, true>(in, nullptr, nullptr, out1, n, 0, job.flag_out, w, &sh.fail);
          else if (kind == JOB_RECV) og_move_ll<T, W, true, false>(in, add, out0, nullptr, n, job.flag_in, 0, w, &sh.fail);
          else og_move_ll<T, W, true, true>(in, add, out0, out1, n, job.flag_in, job.flag_out, w, &sh.fail);
        } else if constexpr (PROTO == PROTO_LL128 && W == 16) {
          if (kind == JOB_SEND) og_move_ll128<T, false, true>(in, nullptr, nullptr, out1, 2 * n, 0, job.flag_out128, w, &sh.fail);
          else if (kind == JOB_RECV) og_move_ll128<T, true, false>(in, add, out0, nullptr, 2 * n, job.flag_in128, 0, w, &sh.fail);
          else og_move_ll128<T, true, true>(in, add, out0, out1, 2 * n, job.flag_in128, job.flag_out128, w, &sh.fail);
        }
      }
    }
    __syncwarp();
    if ((threadIdx.x & 31) == 0) bar_arrive(&sh.done[pass & 1]);
    if (kind == JOB_EXIT) return;
  }
}

struct Ends {                       // where this threadblock's flags live
  unsigned long long *tail_out, *credit_out, *open_out, *progress_out;
};

__device__ __forceinline__ void signal_role(Shared& sh, const Ends& e, SyncPage* sync, int rank, int tb, int recv_peer, int chan,
                                            unsigned long long limit, unsigned long long* trace, int trace_steps) {
  for (unsigned int pass = 0;; ++pass) {
    const Job& job = sh.job[pass & 1];
    if (!bar_wait(&sh.done[pass & 1], (pass >> 1) & 1u, limit)) return;
    if (job.kind == JOB_EXIT) return;
    unsigned long long moved = 0;
    if (trace != nullptr) moved = global_timer_ns();
    if (*reinterpret_cast<volatile int*>(&sh.fail) != 0) {
      record_failure(sync, STATUS_TIMEOUT_DATA, rank, tb, job.step, job.iter, recv_peer, chan);   // the first failure recorded wins
    } else {
      // one fence covers everything the step publishes; the credit alone needs none (the data warps have used what they
      // read from the FIFO slot before they came to the barrier)
      if (job.fence) fence_acq_rel_gpu();
      if (job.tail != 0) st_relaxed_gpu(e.tail_out, job.tail);
      if (job.opened != 0) st_relaxed_gpu(e.open_out, job.opened);
      if (job.credit != 0) st_relaxed_gpu(e.credit_out, job.credit);
      if (job.progress != 0) st_relaxed_gpu(e.progress_out, job.progress);
      if (trace != nullptr) {
        const unsigned long long t2 = global_timer_ns();
        for (int s = job.step; s < job.step + job.steps && s < trace_steps; ++s) {
          unsigned long long* rec = trace + static_cast<long long>(s) * 6;
          const bool main_step = s == job.step + job.steps - 1;     // the nops in front of it only waited
          if (job.iter == 0) rec[0] = job.t0;
          rec[1] = main_step ? t2 : job.t1;
          if (main_step) {
            rec[2] += job.t1 - job.t0;
            rec[3] += moved > job.t1 ? moved - job.t1 : 0;
            rec[4] += t2 - moved;
          }
        }
      }
    }
    asm volatile("st.release.cta.shared.s32 [%0], %1;" ::"r"(smem_addr(&sh.signalled)), "r"(static_cast<int>(pass + 1)) : "memory");
  }
}

__device__ __forceinline__ int ld_signalled(const Shared& sh) {
  int v;
  asm volatile("ld.acquire.cta.shared.s32 %0, [%1];" : "=r"(v) : "r"(smem_addr(&sh.signalled)) : "memory");
  return v;
}

template <typename T, int PROTO, int W>
__global__ void __launch_bounds__(kOgThreads, kOgCtasPerSm) exec_one_gpu_kernel(const __grid_constant__ OneGpuArgs a) {
  __shared__ Shared sh;
  const int K = a.slices;
  const int slice = static_cast<int>(blockIdx.x) % K;
  const DevTb& tb = a.tbs[blockIdx.x / K];
  const int my_rank = tb.rank, my_tb = tb.tb_in_rank, nsteps = tb.nsteps;
  const RankCtx& me = a.ranks[my_rank];
  SyncPage* const sync = me.sync;
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const DevStep* sp = a.steps + tb.step_begin;
  if (nsteps <= kOgSmemSteps) {
    const uint4* g = reinterpret_cast<const uint4*>(sp);
    uint4* s = reinterpret_cast<uint4*>(sh.steps);
    for (int i = threadIdx.x; i < nsteps * 2; i += kOgThreads) s[i] = g[i];
    sp = sh.steps;
  }
  if (threadIdx.x == 0) {
    sh.fail = 0;
    sh.signalled = 0;
    for (int i = 0; i < 2; ++i) {
      bar_init(&sh.go[i], 1);
      bar_init(&sh.done[i], kOgDataWarps);
    }
  }
  const unsigned long long epoch = sync->exec_epoch + 1;       // advanced by the rank's last CTA to finish
  Waiter w;
  w.sync = sync;
  w.deadline = global_timer_ns() + a.timeout_ns;
  const unsigned long long limit = w.deadline + 1000000000ull;
  const int send_peer = tb.send_peer, recv_peer = tb.recv_peer, chan = tb.chan;
  const bool has_send = send_peer >= 0, has_recv = recv_peer >= 0;
  // slice s of channel c uses the flags of channel c * K + s
  const int vchan = chan * K + slice;
  const int remote_idx = vchan * kMaxRanks + my_rank;
  const int send_conn = vchan * kMaxRanks + send_peer, recv_conn = vchan * kMaxRanks + recv_peer;
  Ends ends;
  ends.tail_out = has_send ? &a.ranks[send_peer].sync->recv_tail[remote_idx] : nullptr;
  ends.credit_out = has_recv ? &a.ranks[recv_peer].sync->send_head[remote_idx] : nullptr;
  ends.open_out = has_recv ? &a.ranks[recv_peer].sync->recv_posted[remote_idx] : nullptr;
  ends.progress_out = &sync->progress[my_tb * K + slice];
  __syncthreads();

  if (warp < kOgDataWarps) {
    data_role<T, PROTO, W>(sh, w, limit);
  } else if (warp == kOgDataWarps + 1) {
    if (lane == 0) {
      unsigned long long* trace = (a.trace != nullptr && slice == 0) ? a.trace + static_cast<long long>(blockIdx.x / K) * a.trace_steps * 6 : nullptr;
      signal_role(sh, ends, sync, my_rank, my_tb, recv_peer, chan, limit, trace, a.trace_steps);
    }
  } else {
    // ------------------------------------------------------------------------------------------------ control warp
    const long long C = a.chunk_elems;
    const long long lo = min(C, static_cast<long long>(slice) * a.slice_elems), hi = min(C, lo + a.slice_elems);
    const int iterations = static_cast<int>((hi - lo + a.tile_elems - 1) / a.tile_elems);
    const long long slot_bytes = a.slot_bytes;                  // of one slice
    char* const send_fifo = has_send ? a.ranks[send_peer].fifo + tb.send_fifo_off + slice * kFifoSlots * slot_bytes : nullptr;
    const char* const recv_fifo = has_recv ? me.fifo + tb.recv_fifo_off + slice * kFifoSlots * slot_bytes : nullptr;
    unsigned long long sseq = has_send ? sync->send_seq[send_conn] : 0ull;
    unsigned long long rseq = has_recv ? sync->recv_seq[recv_conn] : 0ull;
    const unsigned long long sseq0 = sseq, rseq0 = rseq;
    // LL flags are unique per (launch, tile), as in exec_kernel.cu
    const unsigned int flag_epoch = static_cast<unsigned int>(epoch & 0xfffffull) << 12;
    const unsigned long long flag_epoch128 = epoch << 24;
    const bool opening = PROTO == PROTO_SIMPLE && has_recv && tb.nrecv > 0 && (tb.recv_bufmask & a.direct_mask) != 0 &&
                         tb.opens_at_start != tb.nrecv;
    unsigned long long opened = rseq0;
    unsigned long long head_seen = sseq0, posted_seen = 0;       // all credits of earlier launches have come back
    unsigned int mode_bits = 0;
    unsigned int pass = 0;
    bool stop = false;
    const long long esize = static_cast<long long>(sizeof(T));

    for (int it = 0; it < iterations && !stop; ++it) {
      const long long tile_off = lo + static_cast<long long>(it) * a.tile_elems;
      const long long n = min(a.tile_elems, hi - tile_off);
      const int V = static_cast<int>(n * esize / W);
      const int lines = (2 * V + 14) / 15;
      const long long fifo_chunk = PROTO == PROTO_SIMPLE ? static_cast<long long>(V) * W
                                   : (PROTO == PROTO_LL ? static_cast<long long>(V) * LLPacket<W>::kBytes : static_cast<long long>(lines) * 128);
      if (opening && tb.opens_at_start > 0) {
        opened += tb.opens_at_start;
        if (lane == 0) st_release_gpu(ends.open_out, opened);
      }
      int s = 0;
      while (s < nsteps && !stop) {
        // nops that nobody waits for only add their dependency to the step behind them
        int g = 0;
        while (g < 8 && s + g + 1 < nsteps && sp[s + g].type == ST_NOP && sp[s + g].hasdep == 0) ++g;
        const int ms = s + g;                                    // the step that moves something
        const DevStep st = sp[ms];
        const int nb = st.batch > 1 ? st.batch : 1;
        const int last = ms + nb - 1;
        const bool sends = is_send(st.type), recvs = is_recv(st.type);
        const bool can_direct_send = PROTO == PROTO_SIMPLE && sends && (st.flags & SF_DIRECT_SEND) && ((a.direct_mask >> st.rbuf) & 1);
        const bool can_direct_recv = PROTO == PROTO_SIMPLE && recvs && (st.flags & SF_DIRECT_RECV) && ((a.direct_mask >> st.dstbuf) & 1);
        const bool always = (st.flags & SF_DIRECT_ALWAYS) != 0;
        unsigned long long t0 = 0;
        if (a.trace != nullptr && slice == 0) t0 = global_timer_ns();

        // ---- bounds (as in exec_kernel.cu) ----
        bool in_bounds = true;
        long long worst = 0;
        if (st.type != ST_NOP) {
          const bool reads_src = st.type == ST_SEND || st.type == ST_CPY || st.type == ST_RE;
          const bool uses_dst = st.type != ST_SEND;
          if (reads_src && (static_cast<long long>(st.srcoff) + st.cnt) * C > me.buf_elems[st.srcbuf]) { in_bounds = false; worst = st.srcoff; }
          if (uses_dst && (static_cast<long long>(st.dstoff) + st.cnt) * C > me.buf_elems[st.dstbuf]) { in_bounds = false; worst = st.dstoff; }
          if (can_direct_send && (static_cast<long long>(st.roff) + st.cnt) * C > a.ranks[send_peer].buf_elems[st.rbuf]) { in_bounds = false; worst = st.roff; }
          if ((sends || recvs) && st.cnt * fifo_chunk > slot_bytes) { in_bounds = false; worst = -1; }
        }
        if (nb > 1) {                                            // one batch member per lane
          bool ok = true;
          long long off = 0;
          if (lane >= 1 && lane < nb) {
            const DevStep sk = sp[ms + lane];
            if (sk.type == ST_RE && (static_cast<long long>(sk.srcoff) + sk.cnt) * C > me.buf_elems[sk.srcbuf]) { ok = false; off = sk.srcoff; }
          }
          const unsigned int bad = __ballot_sync(kFullWarp, !ok);
          if (bad != 0 && in_bounds) { in_bounds = false; worst = __shfl_sync(kFullWarp, off, __ffs(bad) - 1); }
        }

        // ---- waits: one flag per lane ----
        // lane 0: a free FIFO slot; lane 1: the tile; lane 2: may this tile go straight into the receiver's slot?;
        // lanes 3..: the dependencies of the pass.  A receive that opens its own slot does so after the dependencies,
        // so it polls the tile in a second round.
        const unsigned long long want_head = sseq + 1 > kFifoSlots ? sseq + 1 - kFifoSlots : 0;
        const bool opens_here = opening && st.opens_before > 0;
        unsigned int failed_lane = 0;
        unsigned long long word = 0;
        const unsigned long long* flag = nullptr;
        unsigned long long want = 0, mask = ~0ull;
        if (lane == 0 && sends && head_seen < want_head) { flag = &sync->send_head[send_conn]; want = want_head; }
        if (lane == 1 && recvs && PROTO == PROTO_SIMPLE && !opens_here) { flag = &sync->recv_tail[recv_conn]; want = rseq + 1; mask = kTailCountMask; }
        if (lane == 2 && can_direct_send && !always && posted_seen < sseq + 1) flag = &sync->recv_posted[send_conn];   // looked at once
        if (lane >= 3 && lane < 3 + g + nb && in_bounds) {
          const DevStep& sk = sp[s + lane - 3];
          if (sk.depid >= 0) { flag = &sync->progress[sk.depid * K + slice]; want = pack_progress(epoch, it, sk.deps + 1); }
        }
        if (!in_bounds) flag = nullptr;
        // the job slot of two passes ago must have been read by the signal warp before it is written below
        const int need_sig = static_cast<int>(pass) - 1;
#pragma unroll 1
        for (int round = 0; round < (opens_here ? 2 : 1) && failed_lane == 0 && in_bounds; ++round) {
          if (round == 1) {
            // the slot may be opened: what came before this step has been signalled, its dependencies have arrived
            for (unsigned int i = 1; ld_signalled(sh) < static_cast<int>(pass) && failed_lane == 0; ++i)
              if ((i & 255u) == 0 && (*reinterpret_cast<volatile int*>(&sh.fail) != 0 || w.expired())) failed_lane = 32;
            failed_lane = __reduce_max_sync(kFullWarp, failed_lane);
            opened += st.opens_before;
            if (lane == 0) st_release_gpu(ends.open_out, opened);
            flag = nullptr;
            if (lane == 1 && recvs) { flag = &sync->recv_tail[recv_conn]; want = rseq + 1; mask = kTailCountMask; }
          }
          bool pending = flag != nullptr;
          unsigned int spins = 0;
          while (__any_sync(kFullWarp, pending)) {
            if (pending) {
              word = ld_acquire_gpu(flag);
              if ((word & mask) >= want) pending = false;
            }
            if ((++spins & 127u) == 0) {
              const bool give_up = lane == 0 && (*reinterpret_cast<volatile int*>(&sh.fail) != 0 || w.expired());
              if (__any_sync(kFullWarp, give_up)) {
                const unsigned int open_lanes = __ballot_sync(kFullWarp, pending);
                if (open_lanes != 0) failed_lane = static_cast<unsigned int>(__ffs(open_lanes));
                break;
              }
            }
          }
        }
        __syncwarp();
        for (unsigned int i = 1; ld_signalled(sh) < need_sig && failed_lane == 0; ++i)
          if ((i & 255u) == 0 && w.expired()) failed_lane = 32;
        failed_lane = __reduce_max_sync(kFullWarp, failed_lane);
        if (sends) head_seen = max(head_seen, __shfl_sync(kFullWarp, word, 0));
        if (can_direct_send && !always && posted_seen < sseq + 1) posted_seen = __shfl_sync(kFullWarp, word, 2);
        const bool direct_send = can_direct_send && (always || posted_seen >= sseq + 1);
        const unsigned long long tail_word = __shfl_sync(kFullWarp, word, 1);
        const bool direct_recv = can_direct_recv && ((tail_word >> (kTailModeShift + static_cast<int>(rseq % kFifoSlots))) & 1ull) != 0;

        if (!in_bounds || failed_lane != 0 || *reinterpret_cast<volatile int*>(&sh.fail) != 0) {
          // a flag-in-data poll that ran out of time is recorded by the signal warp, which knows its step
          if (lane == 0 && *reinterpret_cast<volatile int*>(&sh.fail) == 0) {
            unsigned int code = STATUS_ABORTED, aux0 = 0, aux1 = 0;
            if (!in_bounds) { code = STATUS_BOUNDS; aux0 = st.type; aux1 = static_cast<unsigned int>(worst); }
            else if (failed_lane == 1) { code = STATUS_TIMEOUT_CREDIT; aux0 = send_peer; aux1 = chan; }
            else if (failed_lane == 2) { code = STATUS_TIMEOUT_DATA; aux0 = recv_peer; aux1 = chan; }
            else if (failed_lane > 3 && failed_lane < 32) { code = STATUS_TIMEOUT_DEP; aux0 = sp[s + failed_lane - 4].depid; aux1 = sp[s + failed_lane - 4].deps; }
            record_failure(sync, code, my_rank, my_tb, ms, it, aux0, aux1);
            *reinterpret_cast<volatile int*>(&sh.fail) = 1;
          }
          stop = true;
          break;
        }

        // ---- the job ----
        if (lane == 0) {
          Job& job = sh.job[pass & 1];
          char* const sbase = static_cast<char*>(me.buf[st.srcbuf]) + (static_cast<long long>(st.srcoff) * C + tile_off) * esize;
          char* const dbase = static_cast<char*>(me.buf[st.dstbuf]) + (static_cast<long long>(st.dstoff) * C + tile_off) * esize;
          const char* fifo_in = recvs ? recv_fifo + (rseq % kFifoSlots) * slot_bytes : nullptr;
          char* out1 = nullptr;
          if (sends)
            out1 = direct_send ? static_cast<char*>(a.ranks[send_peer].buf[st.rbuf]) + (static_cast<long long>(st.roff) * C + tile_off) * esize
                               : send_fifo + (sseq % kFifoSlots) * slot_bytes;
          const long long chunk_step = C * esize;
          int kind = JOB_MOVE;
          const char *in = nullptr, *add = nullptr;
          char* out0 = nullptr;
          long long in_step = chunk_step;
          if (recvs && !direct_recv) { in = fifo_in; in_step = fifo_chunk; }
          switch (st.type) {
            case ST_SEND: in = sbase; kind = PROTO == PROTO_SIMPLE ? JOB_MOVE : JOB_SEND; break;
            case ST_RECV:
              out0 = dbase;
              kind = PROTO == PROTO_SIMPLE ? (direct_recv ? JOB_NONE : JOB_MOVE) : JOB_RECV;
              break;
            case ST_RCS:
              if (direct_recv) in = dbase; else out0 = dbase;
              kind = PROTO == PROTO_SIMPLE ? JOB_MOVE : JOB_BOTH;
              break;
            case ST_RRC: add = dbase; out0 = dbase; kind = PROTO == PROTO_SIMPLE ? JOB_MOVE : JOB_RECV; break;
            case ST_RRS: add = dbase; kind = PROTO == PROTO_SIMPLE ? JOB_MOVE : JOB_BOTH; break;
            case ST_RRCS: add = dbase; out0 = dbase; kind = PROTO == PROTO_SIMPLE ? JOB_MOVE : JOB_BOTH; break;
            case ST_CPY: in = sbase; out0 = dbase; break;
            case ST_RE:
              if (nb == 1) { in = dbase; add = sbase; out0 = dbase; }
              else { in = dbase; out0 = dbase; kind = JOB_BATCH; }
              break;
            default: kind = JOB_NONE; break;
          }
          int nsrc = 0;
          unsigned int more = opening ? st.opens_after : 0;
          bool any_dep = st.hasdep != 0;
          for (int k = 0; k < nb; ++k) {
            const DevStep& sk = sp[ms + k];
            if (k > 0) {
              if (opening) more += sk.opens_after;
              any_dep = any_dep || sk.hasdep != 0;
            }
            if (kind == JOB_BATCH && sk.type == ST_RE && nsrc < kMaxBatch)
              job.src[nsrc++] = static_cast<char*>(me.buf[sk.srcbuf]) + (static_cast<long long>(sk.srcoff) * C + tile_off) * esize;
          }
          job.in = in; job.add = add; job.out0 = out0; job.out1 = out1;
          job.in_step = in_step; job.add_step = chunk_step; job.out0_step = chunk_step;
          job.out1_step = direct_send ? chunk_step : fifo_chunk;
          job.src_step = chunk_step;
          job.kind = kind; job.cnt = st.cnt; job.n = V; job.nsrc = nsrc;
          job.flag_in = flag_epoch | (static_cast<unsigned int>((rseq - rseq0) % 4095ull) + 1u);
          job.flag_out = flag_epoch | (static_cast<unsigned int>((sseq - sseq0) % 4095ull) + 1u);
          job.flag_in128 = flag_epoch128 | (rseq - rseq0 + 1);
          job.flag_out128 = flag_epoch128 | (sseq - sseq0 + 1);
          const bool publishes_tile = sends && PROTO == PROTO_SIMPLE;
          if (publishes_tile) {
            const unsigned int bit = 1u << static_cast<int>(sseq % kFifoSlots);
            mode_bits = direct_send ? (mode_bits | bit) : (mode_bits & ~bit);
          }
          job.tail = publishes_tile ? (static_cast<unsigned long long>(mode_bits) << kTailModeShift) | (sseq + 1) : 0ull;
          job.opened = more > 0 ? opened + more : 0ull;
          job.credit = recvs ? rseq + 1 : 0ull;
          job.progress = any_dep ? pack_progress(epoch, it, last + 1) : 0ull;
          job.fence = publishes_tile || more > 0 || any_dep;
          opened += more;
          job.step = s; job.steps = g + nb; job.iter = it;
          if (a.trace != nullptr && slice == 0) { job.t0 = t0; job.t1 = global_timer_ns(); }
          bar_arrive(&sh.go[pass & 1]);
        }
        if (opening) opened = __shfl_sync(kFullWarp, opened, 0);
        ++pass;
        if (sends) ++sseq;
        if (recvs) ++rseq;
        s = last + 1;
      }
    }
    // the last pass: tells data and signal warps to leave
    const int need_sig = static_cast<int>(pass) - 1;
    for (unsigned int i = 1; ld_signalled(sh) < need_sig; ++i)
      if ((i & 255u) == 0 && global_timer_ns() > limit) break;
    __syncwarp();
    if (lane == 0) {
      sh.job[pass & 1].kind = JOB_EXIT;
      bar_arrive(&sh.go[pass & 1]);
      if (has_send) sync->send_seq[send_conn] = sseq;
      if (has_recv) sync->recv_seq[recv_conn] = rseq;
    }
  }
  // every role of this CTA has left: the last CTA of the rank advances its launch epoch
  __syncwarp();
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(&sync->exec_done, 1u) == static_cast<unsigned int>(tb.tbs_in_rank * K) - 1u) {
      sync->exec_done = 0;
      sync->exec_epoch = sync->exec_epoch + 1;
    }
  }
}

template <typename T, int PROTO, int W>
const void* kernel_ptr() { return reinterpret_cast<const void*>(&exec_one_gpu_kernel<T, PROTO, W>); }

template <typename T>
const void* pick_kernel(int proto, int width) {
  constexpr int E = static_cast<int>(sizeof(T));
  if (width == 16) {
    if (proto == PROTO_SIMPLE) return kernel_ptr<T, PROTO_SIMPLE, 16>();
    if (proto == PROTO_LL) return kernel_ptr<T, PROTO_LL, 16>();
    if (proto == PROTO_LL128) return kernel_ptr<T, PROTO_LL128, 16>();
  } else if (width == E) {
    if (proto == PROTO_SIMPLE) return kernel_ptr<T, PROTO_SIMPLE, E>();
    if (proto == PROTO_LL) return kernel_ptr<T, PROTO_LL, E>();
  }
  return nullptr;
}

const void* pick_kernel(int dtype, int proto, int width) {
  switch (dtype) {
    case DT_F32: return pick_kernel<float>(proto, width);
    case DT_BF16: return pick_kernel<__nv_bfloat16>(proto, width);
    case DT_F16: return pick_kernel<__half>(proto, width);
    default: return nullptr;
  }
}

}  // namespace

// `slices` CTAs per threadblock; always cooperative unless the caller vouches for an otherwise idle GPU.
cudaError_t launch_exec_one_gpu(const OneGpuArgs& args, int dtype, int proto, int width, int tbs, cudaStream_t stream, bool cooperative) {
  const void* fn = pick_kernel(dtype, proto, width);
  if (fn == nullptr) return cudaErrorInvalidValue;
  OneGpuArgs copy = args;
  void* params[] = {&copy};
  const dim3 grid(static_cast<unsigned int>(tbs * args.slices)), block(kOgThreads);
  if (cooperative) return cudaLaunchCooperativeKernel(fn, grid, block, params, 0, stream);
  return cudaLaunchKernel(fn, grid, block, params, 0, stream);
}

// CTAs of this kernel that the current device holds at once.
int max_coresident_one_gpu(int dtype, int proto, int width) {
  int per_sm = 0, dev = 0, sms = 0;
  const void* fn = pick_kernel(dtype, proto, width);
  if (fn == nullptr || cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kOgThreads, 0) != cudaSuccess)
    return 0;
  return per_sm * sms;
}

}  // namespace msccl
