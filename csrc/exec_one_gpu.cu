// MSCCL-IR interpreter for programs whose ranks all live on this GPU (Communicator.emulated).  Same contract as
// exec_kernel.cu - steps of a threadblock in order, the program's protocol, FIFOs, credits, bounds checks, bounded
// waits, bit-identical sums - but laid out for one device:
//
//   * Slices.  Every step works element by element, so a chunk is cut into slices that never meet, each with its own FIFO
//     slots, counters and progress words.  K CTAs run one threadblock, and each of them runs P slices: while one slice
//     waits for its tile to come round the ring, another moves.  One CTA per SM (the layout of exec_kernel.cu) leaves the
//     SMs of idle receivers empty and pays every flag round trip in full.
//   * Roles.  Six data warps move; a control warp polls the flags of its slices' next steps, one flag per lane, and hands
//     jobs that are ready (pointers, sizes) to the data warps; a signal warp fences and publishes what a job finished while
//     the data warps are in the next one.  Jobs are double buffered.  Slices share the data warps only under the Simple
//     protocol: there a job never waits once it has been handed over (a flag-in-data job does, and could wait for one
//     queued behind it).
//   * Chunks that are not multiples of 16 bytes still move in 16-byte vectors: stores are aligned, loads are put together
//     from two aligned vectors.
//   * Scope.  All flags are read and written at GPU scope: a system-scope fence costs more and orders nothing extra here.
//   * No drain: the FIFO contents cannot be wanted after the kernel's end, because every receiver is part of it.  No
//     opening handshake for slots that nothing touches before their receive (SF_DIRECT_ALWAYS): every rank's earlier
//     work on this GPU is done when the kernel runs.
//   * The rank table travels in the kernel parameters: no device copy per set of buffers, nothing kept by address.
//
// Bound by L2 / HBM traffic from about 1 MB per chunk on, by the flag round trips (store, fence, poll) below.
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

// A flag-in-data poll that ran out of time leaves its report to the signal warp; whoever in the control warp raises the flag
// reports by itself (and the signal warp, which may see the flag first, must not call that a timeout).
enum FailKind : int { FAIL_REPORTED = 1, FAIL_DATA = 2 };

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
  int fence, traced, step, steps, iter;   // first step of the pass and how many (nops in front and batch members included)
  unsigned long long tail, credit, opened, progress;     // 0: nothing to publish
  unsigned long long *tail_out, *credit_out, *open_out, *progress_out;
  unsigned long long t0, t1;      // trace
};

struct Shared {
  Job job[2];
  unsigned long long go[2], done[2];     // mbarriers
  int fail;                              // FAIL_*: everybody gives up
  int leave;                             // the first data warp waited too long for a job: all leave
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

// ---- chunks that do not start on 16-byte boundaries ------------------------------------------------------------------
// The 16 bytes that start `shift` (a multiple of 2) bytes into the aligned vector `lo` and go on into the next one.
__device__ __forceinline__ uint4 shifted(uint4 lo, uint4 hi, unsigned int shift) {
  unsigned int w[7] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z};
  if (shift & 8u) { w[0] = w[2]; w[1] = w[3]; w[2] = w[4]; w[3] = w[5]; w[4] = w[6]; w[5] = hi.w; }
  if (shift & 4u) { w[0] = w[1]; w[1] = w[2]; w[2] = w[3]; w[3] = w[4]; w[4] = w[5]; }
  if (shift & 2u) return make_uint4(__funnelshift_r(w[0], w[1], 16), __funnelshift_r(w[1], w[2], 16),
                                    __funnelshift_r(w[2], w[3], 16), __funnelshift_r(w[3], w[4], 16));
  return make_uint4(w[0], w[1], w[2], w[3]);
}
__device__ __forceinline__ uint4 shuffle_down(uint4 v) {
  return make_uint4(__shfl_down_sync(kFullWarp, v.x, 1), __shfl_down_sync(kFullWarp, v.y, 1), __shfl_down_sync(kFullWarp, v.z, 1),
                    __shfl_down_sync(kFullWarp, v.w, 1));
}
__device__ __forceinline__ uint4 from_first(uint4 v) {
  return make_uint4(__shfl_sync(kFullWarp, v.x, 0), __shfl_sync(kFullWarp, v.y, 0), __shfl_sync(kFullWarp, v.z, 0),
                    __shfl_sync(kFullWarp, v.w, 0));
}

// out = in (+ add) for element-wide chunks: elements up to the first 16-byte boundary of `out` and behind the last one
// singly, vectors in between.  A warp takes 32 U consecutive vectors; each of its lanes loads the aligned vector in which
// its own starts and gets the next one from its neighbour, so `in` is read once (all-gather of 333333 fp16 elements over 8 ranks:
// 34.6 us a call with two loads per vector and half as many in flight, 28.7 this way).  `add` and a second output must lie like the first output (the
// caller checks).
template <typename T, bool ADD>
__device__ __forceinline__ void og_move_unaligned(const char* in, const char* add, char* out0, char* out1, int n) {
  constexpr int E = static_cast<int>(sizeof(T)), PER = 16 / E;
  constexpr int U = ADD ? 4 : 8;
  const char* out = out0 != nullptr ? out0 : out1;
  const int head = min(n, static_cast<int>((16u - (static_cast<unsigned int>(reinterpret_cast<unsigned long long>(out)) & 15u)) & 15u) / E);
  const int vecs = (n - head) / PER, tail = head + vecs * PER;
  const int singles = head + (n - tail);                     // at most 2 * (PER - 1)
  if (static_cast<int>(threadIdx.x) < singles) {
    const int e = static_cast<int>(threadIdx.x) < head ? threadIdx.x : tail + threadIdx.x - head;
    auto v = Access<E>::ld(in + static_cast<long long>(e) * E);
    if (ADD) v = Wide<T, E>::add(v, Access<E>::ld(add + static_cast<long long>(e) * E));
    if (out0 != nullptr) Access<E>::st(out0 + static_cast<long long>(e) * E, v);
    if (out1 != nullptr) Access<E>::st(out1 + static_cast<long long>(e) * E, v);
  }
  const unsigned long long start = reinterpret_cast<unsigned long long>(in + head * E);
  const unsigned int shift = static_cast<unsigned int>(start) & 15u;
  const uint4* vin = reinterpret_cast<const uint4*>(start & ~15ull);
  // aligned vectors that hold bytes of the `vecs` vectors: one more when they are shifted
  const int last = vecs - 1 + (shift != 0 ? 1 : 0);
  const int lane = threadIdx.x & 31;
#pragma unroll 1
  for (int base = (threadIdx.x >> 5) * (32 * U); base < vecs; base += kOgData * U) {       // the same for the whole warp
    uint4 x[U + 1], y[U];
#pragma unroll
    for (int u = 0; u < U; ++u) x[u] = vin[min(base + u * 32 + lane, last)];
    x[U] = vin[min(base + U * 32, last)];                    // the one behind the warp's last vector
    if (ADD) {
#pragma unroll
      for (int u = 0; u < U; ++u) y[u] = *reinterpret_cast<const uint4*>(add + head * E + static_cast<long long>(min(base + u * 32 + lane, vecs - 1)) * 16);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      uint4 next = shuffle_down(x[u]);
      const uint4 over = from_first(x[u + 1]);
      if (lane == 31) next = over;
      uint4 v = shifted(x[u], next, shift);
      if (ADD) v = Wide<T, 16>::add(v, y[u]);
      const int at = base + u * 32 + lane;
      if (at < vecs) {
        const long long byte = head * E + static_cast<long long>(at) * 16;
        if (out0 != nullptr) *reinterpret_cast<uint4*>(out0 + byte) = v;
        if (out1 != nullptr) *reinterpret_cast<uint4*>(out1 + byte) = v;
      }
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
          *reinterpret_cast<volatile int*>(fail) = FAIL_DATA;
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
            *reinterpret_cast<volatile int*>(fail) = FAIL_DATA;
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
    // the first warp waits for the job, the others for the first warp: a job may read what any warp wrote in the one
    // before, and all warps leave together
    if (threadIdx.x < 32) {
      if (!bar_wait(&sh.go[pass & 1], (pass >> 1) & 1u, limit)) sh.leave = 1;
      __syncwarp();
    }
    asm volatile("barrier.sync 1, %0;" ::"n"(kOgData) : "memory");
    if (*reinterpret_cast<volatile int*>(&sh.leave) != 0) return;
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
          if constexpr (W == 16) {
            if (add != nullptr) {
              og_move<T, W, 4, true>(in, add, out0, out1, n);
            } else {
              og_move<T, W, 8, false>(in, nullptr, out0, out1, n);
            }
          } else {
            const unsigned long long out = reinterpret_cast<unsigned long long>(out0 != nullptr ? out0 : out1);
            unsigned long long apart = out1 != nullptr ? out ^ reinterpret_cast<unsigned long long>(out1) : 0;
            if (add != nullptr) {
              // a sum does not depend on the order of its two operands: the one that lies like the output is read as vectors
              if (((out ^ reinterpret_cast<unsigned long long>(in)) & 15ull) == 0) {
                const char* other = add;
                add = in;
                in = other;
              }
              apart |= out ^ reinterpret_cast<unsigned long long>(add);
            }
            if ((apart & 15ull) != 0) {
              if (add != nullptr) og_move<T, W, 4, true>(in, add, out0, out1, n);
              else og_move<T, W, 8, false>(in, nullptr, out0, out1, n);
            } else if (add != nullptr) {
              og_move_unaligned<T, true>(in, add, out0, out1, n);
            } else {
              og_move_unaligned<T, false>(in, nullptr, out0, out1, n);
            }
          }
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

__device__ __forceinline__ void signal_role(Shared& sh, SyncPage* sync, int rank, int tb, int recv_peer, int chan,
                                            unsigned long long limit, unsigned long long* trace, int trace_steps) {
  for (unsigned int pass = 0;; ++pass) {
    const Job& job = sh.job[pass & 1];
    if (!bar_wait(&sh.done[pass & 1], (pass >> 1) & 1u, limit)) return;
    if (job.kind == JOB_EXIT) return;
    unsigned long long moved = 0;
    if (trace != nullptr) moved = global_timer_ns();
    const int fail = *reinterpret_cast<volatile int*>(&sh.fail);
    if (fail != 0) {
      // the first failure recorded wins
      if (fail == FAIL_DATA) record_failure(sync, STATUS_TIMEOUT_DATA, rank, tb, job.step, job.iter, recv_peer, chan);
    } else {
      // one fence covers everything the step publishes; the credit alone needs none (the data warps have used what they
      // read from the FIFO slot before they came to the barrier)
      if (job.fence) fence_acq_rel_gpu();
      if (job.tail != 0) st_relaxed_gpu(job.tail_out, job.tail);
      if (job.opened != 0) st_relaxed_gpu(job.open_out, job.opened);
      if (job.credit != 0) st_relaxed_gpu(job.credit_out, job.credit);
      if (job.progress != 0) st_relaxed_gpu(job.progress_out, job.progress);
      if (trace != nullptr && job.traced) {
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
  const int K = a.ctas_per_tb, P = a.streams;
  const int tb_index = static_cast<int>(blockIdx.x) / K, part = static_cast<int>(blockIdx.x) % K;
  const DevTb& tb = a.tbs[tb_index];
  const int my_rank = tb.rank, my_tb = tb.tb_in_rank, nsteps = tb.nsteps;
  const OneGpuRank& me = a.ranks[my_rank];
  SyncPage* const sync = me.sync;
  OneGpuFlags* const flags = me.flags;
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
    sh.leave = 0;
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
  __syncthreads();

  if (warp < kOgDataWarps) {
    data_role<T, PROTO, W>(sh, w, limit);
  } else if (warp == kOgDataWarps + 1) {
    if (lane == 0) {
      unsigned long long* trace = (a.trace != nullptr && part == 0) ? a.trace + static_cast<long long>(tb_index) * a.trace_steps * 6 : nullptr;
      signal_role(sh, sync, my_rank, my_tb, recv_peer, chan, limit, trace, a.trace_steps);
    }
  } else {
    // ------------------------------------------------------------------------------------------------ control warp
    // P groups of 32 / P lanes; every lane of a group carries the state of the group's slice
    const int LP = 32 / P, p = lane / LP, gl = lane % LP;
    const unsigned int gmask = (LP == 32 ? ~0u : (1u << LP) - 1u) << (p * LP);
    const bool has_send = send_peer >= 0, has_recv = recv_peer >= 0;
    const int slices = K * P, slice = part * P + p;
    const bool tracing = a.trace != nullptr && slice == 0;
    // slice s of channel c uses the flags of channel c * slices + s, threadblock t the progress word t * slices + s
    const int vchan = chan * slices + slice;
    const int remote_idx = vchan * kMaxRanks + my_rank;
    const int send_conn = vchan * kMaxRanks + send_peer, recv_conn = vchan * kMaxRanks + recv_peer;
    const long long C = a.chunk_elems;
    const long long lo = min(C, static_cast<long long>(slice) * a.slice_elems), hi = min(C, lo + a.slice_elems);
    const int iterations = static_cast<int>((hi - lo + a.tile_elems - 1) / a.tile_elems);
    const long long slot_bytes = a.slot_bytes;                  // of one slice
    char* const send_fifo = has_send ? a.ranks[send_peer].fifo + tb.send_fifo_off + slice * kFifoSlots * slot_bytes : nullptr;
    const char* const recv_fifo = has_recv ? me.fifo + tb.recv_fifo_off + slice * kFifoSlots * slot_bytes : nullptr;
    unsigned long long* const open_out = has_recv ? &a.ranks[recv_peer].flags->posted[remote_idx] : nullptr;
    const unsigned long long sseq0 = has_send ? flags->send_seq[send_conn] : 0ull;
    const unsigned long long rseq0 = has_recv ? flags->recv_seq[recv_conn] : 0ull;
    unsigned long long sseq = sseq0, rseq = rseq0;
    // LL flags are unique per (launch, tile), as in exec_kernel.cu
    const unsigned int flag_epoch = static_cast<unsigned int>(epoch & 0xfffffull) << 12;
    const unsigned long long flag_epoch128 = epoch << 24;
    const bool opening = PROTO == PROTO_SIMPLE && has_recv && tb.nrecv > 0 && (tb.recv_bufmask & a.direct_mask) != 0 &&
                         tb.opens_at_start != tb.nrecv;
    unsigned long long opened = rseq0;
    unsigned long long head_seen = sseq0, posted_seen = 0;       // all credits of earlier launches have come back
    unsigned int mode_bits = 0;
    const long long esize = static_cast<long long>(sizeof(T));
    unsigned int pass = 0;                                       // jobs handed over by this CTA
    int last_pass = -1;                                          // the last one of this slice
    int it = 0, s = 0;
    bool finished = iterations == 0, setup = true, second = false;
    // the step under way, filled in by the setup below
    DevStep st;
    int g = 0, nb = 1, V = 0, dep = 0;
    long long tile_off = 0, fifo_chunk = 0;
    const unsigned long long* flag = nullptr;
    unsigned long long want = 0, word = 0, t0 = 0;
    bool opens_here = false, can_direct_send = false, can_direct_recv = false;
    unsigned int spins = 0;

    // the next dependency of this lane at or behind `dep`
    const auto next_dep = [&]() {
      flag = nullptr;
      for (; dep < g + nb; dep += LP - 3) {
        const DevStep& sk = sp[s + dep];
        if (sk.depid >= 0) {
          flag = &flags->progress[sk.depid * slices + slice];
          want = pack_progress(epoch, it, sk.deps + 1);
          dep += LP - 3;
          return;
        }
      }
    };

    while (true) {
      if (setup && !finished) {
        // ---- the next step of this slice: sizes, bounds, and which flags its lanes look at ----
        setup = false;
        second = false;
        if (s == 0) {
          tile_off = lo + static_cast<long long>(it) * a.tile_elems;
          V = static_cast<int>(min(a.tile_elems, hi - tile_off) * esize / W);
          const int lines = (2 * V + 14) / 15;
          fifo_chunk = PROTO == PROTO_SIMPLE ? static_cast<long long>(V) * W
                       : (PROTO == PROTO_LL ? static_cast<long long>(V) * LLPacket<W>::kBytes : static_cast<long long>(lines) * 128);
          if (opening && tb.opens_at_start > 0) {
            opened += tb.opens_at_start;
            if (gl == 0) st_release_gpu(open_out, opened);
          }
        }
        // nops that nobody waits for only add their dependency to the step behind them
        g = 0;
        while (g < 8 && s + g + 1 < nsteps && sp[s + g].type == ST_NOP && sp[s + g].hasdep == 0) ++g;
        st = sp[s + g];                                          // the step that moves something
        nb = st.batch > 1 ? st.batch : 1;
        const bool sends = is_send(st.type), recvs = is_recv(st.type);
        can_direct_send = PROTO == PROTO_SIMPLE && sends && (st.flags & SF_DIRECT_SEND) && ((a.direct_mask >> st.rbuf) & 1);
        can_direct_recv = PROTO == PROTO_SIMPLE && recvs && (st.flags & SF_DIRECT_RECV) && ((a.direct_mask >> st.dstbuf) & 1);
        opens_here = opening && st.opens_before > 0;
        if (tracing) t0 = global_timer_ns();

        // bounds, as in exec_kernel.cu
        bool in_bounds = true;
        long long worst = 0;
        if (st.type != ST_NOP) {
          const bool reads_src = st.type == ST_SEND || st.type == ST_CPY || st.type == ST_RE;
          const bool uses_dst = st.type != ST_SEND;
          if (reads_src && (static_cast<long long>(st.srcoff) + st.cnt) * C > me.buf_elems[st.srcbuf]) { in_bounds = false; worst = st.srcoff; }
          if (uses_dst && (static_cast<long long>(st.dstoff) + st.cnt) * C > me.buf_elems[st.dstbuf]) { in_bounds = false; worst = st.dstoff; }
          if (can_direct_send && (static_cast<long long>(st.roff) + st.cnt) * C > a.ranks[send_peer].buf_elems[st.rbuf]) { in_bounds = false; worst = st.roff; }
          if ((sends || recvs) && st.cnt * fifo_chunk > slot_bytes) { in_bounds = false; worst = -1; }
          for (int k = 1; k < nb; ++k) {
            const DevStep& sk = sp[s + g + k];
            if (sk.type == ST_RE && (static_cast<long long>(sk.srcoff) + sk.cnt) * C > me.buf_elems[sk.srcbuf]) { in_bounds = false; worst = sk.srcoff; }
          }
        }
        if (!in_bounds) {
          if (gl == 0) record_failure(sync, STATUS_BOUNDS, my_rank, my_tb, s + g, it, st.type, static_cast<unsigned int>(worst));
          *reinterpret_cast<volatile int*>(&sh.fail) = FAIL_REPORTED;
        }

        // lane 0 of the group: a free FIFO slot; 1: the tile; 2: may the tile go straight into the receiver's slot? (looked
        // at once); 3..: the dependencies.  A receive that opens its own slot looks for the tile afterwards.
        const unsigned long long want_head = sseq + 1 > kFifoSlots ? sseq + 1 - kFifoSlots : 0;
        flag = nullptr;
        want = 0;
        word = 0;
        if (gl == 0) {
          if (sends && head_seen < want_head) { flag = &flags->head[send_conn]; want = want_head; }
        } else if (gl == 1) {
          if (recvs && PROTO == PROTO_SIMPLE && !opens_here) { flag = &flags->tail[recv_conn]; want = rseq + 1; }
        } else if (gl == 2) {
          if (can_direct_send && (st.flags & SF_DIRECT_ALWAYS) == 0 && posted_seen < sseq + 1) flag = &flags->posted[send_conn];
        } else {
          dep = gl - 3;
          next_dep();
        }
      }

      // ---- one look at every flag ----
      if (flag != nullptr) {
        word = ld_acquire_gpu(flag);
        if ((gl == 1 ? word & kTailCountMask : word) >= want) {
          flag = nullptr;
          if (gl >= 3) next_dep();
        }
      }
      __syncwarp();
      const int signalled = __shfl_sync(kFullWarp, ld_signalled(sh), 0);
      const unsigned int waiting = __ballot_sync(kFullWarp, flag != nullptr);
      bool ready = !finished && (waiting & gmask) == 0;
      if (ready && opens_here && !second) {
        // the slot may be opened once this slice's last job has been signalled (its dependencies have arrived)
        if (signalled > last_pass) {
          opened += st.opens_before;
          if (gl == 0) st_release_gpu(open_out, opened);
          if (gl == 1) { flag = &flags->tail[recv_conn]; want = rseq + 1; }
          second = true;
        }
        ready = false;
      }
      unsigned int ready_set = __ballot_sync(kFullWarp, ready && gl == 0);
      const bool failed = __any_sync(kFullWarp, *reinterpret_cast<volatile int*>(&sh.fail) != 0);
      if (failed) break;                                         // recorded by whoever raised it
      if (ready_set == 0) {
        if (__all_sync(kFullWarp, finished)) break;
        if ((++spins & 127u) == 0 && __any_sync(kFullWarp, lane == 0 && w.expired())) {
          const unsigned int open_lanes = __ballot_sync(kFullWarp, flag != nullptr);
          const int who = open_lanes != 0 ? __ffs(open_lanes) - 1 : 0;
          if (lane == who) {
            unsigned int code = STATUS_ABORTED, aux0 = 0, aux1 = 0;
            if (open_lanes != 0) {
              if (gl == 0) { code = STATUS_TIMEOUT_CREDIT; aux0 = send_peer; aux1 = chan; }
              else if (gl == 1) { code = STATUS_TIMEOUT_DATA; aux0 = recv_peer; aux1 = chan; }
              else if (gl >= 3) { const DevStep& sk = sp[s + dep - (LP - 3)]; code = STATUS_TIMEOUT_DEP; aux0 = sk.depid; aux1 = sk.deps; }
            }
            record_failure(sync, code, my_rank, my_tb, s + g, it, aux0, aux1);
            *reinterpret_cast<volatile int*>(&sh.fail) = FAIL_REPORTED;
          }
          __syncwarp();
          break;
        }
        continue;
      }

      // ---- hand the jobs that are ready over, one after the other ----
      bool stuck = false;
      while (ready_set != 0) {
        const int q = __ffs(ready_set) - 1;                      // first lane of the group
        ready_set &= ready_set - 1;
        // the job slot of two passes ago must have been read by the signal warp
        for (unsigned int i = 1; ld_signalled(sh) < static_cast<int>(pass) - 1; ++i)
          if ((i & 255u) == 0 && global_timer_ns() > limit) { stuck = true; break; }
        stuck = __any_sync(kFullWarp, stuck);
        if (stuck) break;
        const unsigned long long w_head = __shfl_sync(kFullWarp, word, q), w_tail = __shfl_sync(kFullWarp, word, q + 1),
                                 w_posted = __shfl_sync(kFullWarp, word, q + 2);
        if (p == q / LP) {
          const bool sends = is_send(st.type), recvs = is_recv(st.type), always = (st.flags & SF_DIRECT_ALWAYS) != 0;
          const int last = s + g + nb - 1;
          if (sends) head_seen = max(head_seen, w_head);
          if (can_direct_send && !always) posted_seen = max(posted_seen, w_posted);
          const bool direct_send = can_direct_send && (always || posted_seen >= sseq + 1);
          const bool direct_recv = can_direct_recv && ((w_tail >> (kTailModeShift + static_cast<int>(rseq % kFifoSlots))) & 1ull) != 0;
          const bool publishes_tile = sends && PROTO == PROTO_SIMPLE;
          if (publishes_tile) {
            const unsigned int bit = 1u << static_cast<int>(sseq % kFifoSlots);
            mode_bits = direct_send ? (mode_bits | bit) : (mode_bits & ~bit);
          }
          unsigned int more = opening ? st.opens_after : 0;
          bool any_dep = st.hasdep != 0;
          for (int k = 1; k < nb; ++k) {
            const DevStep& sk = sp[s + g + k];
            if (opening) more += sk.opens_after;
            any_dep = any_dep || sk.hasdep != 0;
          }
          opened += more;
          if (gl == 0) {
            Job& job = sh.job[pass & 1];
            const long long chunk_step = C * esize;
            char* const sbase = static_cast<char*>(me.buf[st.srcbuf]) + (static_cast<long long>(st.srcoff) * C + tile_off) * esize;
            char* const dbase = static_cast<char*>(me.buf[st.dstbuf]) + (static_cast<long long>(st.dstoff) * C + tile_off) * esize;
            char* out1 = nullptr;
            if (sends)
              out1 = direct_send ? static_cast<char*>(a.ranks[send_peer].buf[st.rbuf]) + (static_cast<long long>(st.roff) * C + tile_off) * esize
                                 : send_fifo + (sseq % kFifoSlots) * slot_bytes;
            int kind = JOB_MOVE;
            long long tile_byte = 0;                             // where this threadblock's part of the tile starts
            const char *in = nullptr, *add = nullptr;
            char* out0 = nullptr;
            long long in_step = chunk_step;
            if (recvs && !direct_recv) { in = recv_fifo + (rseq % kFifoSlots) * slot_bytes; in_step = fifo_chunk; }
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
                in = dbase; out0 = dbase;
                if (nb == 1) add = sbase; else kind = JOB_BATCH;
                break;
              default: kind = JOB_NONE; break;
            }
            int nsrc = 0, n = V;
            if (st.part != 0) {
              // one part of every chunk, in whole accesses; the other parts are other threadblocks'
              const int parts = st.part >> 4, part = st.part & 15;
              const int first = static_cast<int>(static_cast<long long>(V) * part / parts);
              n = static_cast<int>(static_cast<long long>(V) * (part + 1) / parts) - first;
              tile_byte = static_cast<long long>(first) * W;
              in += tile_byte;
              out0 += tile_byte;
              if (add != nullptr) add += tile_byte;
              if (n == 0) kind = JOB_NONE;
            }
            if (kind == JOB_BATCH) {
              for (int k = 0; k < nb; ++k) {
                const DevStep& sk = sp[s + g + k];
                if (sk.type == ST_RE && nsrc < kMaxBatch)
                  job.src[nsrc++] = static_cast<char*>(me.buf[sk.srcbuf]) + (static_cast<long long>(sk.srcoff) * C + tile_off) * esize + tile_byte;
              }
            }
            job.in = in; job.add = add; job.out0 = out0; job.out1 = out1;
            job.in_step = in_step; job.add_step = chunk_step; job.out0_step = chunk_step;
            job.out1_step = direct_send ? chunk_step : fifo_chunk;
            job.src_step = chunk_step;
            job.kind = kind; job.cnt = st.cnt; job.n = n; job.nsrc = nsrc;
            if (PROTO != PROTO_SIMPLE) {
              job.flag_in = flag_epoch | (static_cast<unsigned int>((rseq - rseq0) % 4095ull) + 1u);
              job.flag_out = flag_epoch | (static_cast<unsigned int>((sseq - sseq0) % 4095ull) + 1u);
              job.flag_in128 = flag_epoch128 | (rseq - rseq0 + 1);
              job.flag_out128 = flag_epoch128 | (sseq - sseq0 + 1);
            }
            job.tail = publishes_tile ? (static_cast<unsigned long long>(mode_bits) << kTailModeShift) | (sseq + 1) : 0ull;
            job.opened = more > 0 ? opened : 0ull;
            job.credit = recvs ? rseq + 1 : 0ull;
            job.progress = any_dep ? pack_progress(epoch, it, last + 1) : 0ull;
            job.tail_out = has_send ? &a.ranks[send_peer].flags->tail[remote_idx] : nullptr;
            job.credit_out = has_recv ? &a.ranks[recv_peer].flags->head[remote_idx] : nullptr;
            job.open_out = open_out;
            job.progress_out = &flags->progress[my_tb * slices + slice];
            job.fence = publishes_tile || more > 0 || any_dep;
            job.step = s; job.steps = g + nb; job.iter = it; job.traced = tracing;
            if (tracing) { job.t0 = t0; job.t1 = global_timer_ns(); }
            bar_arrive(&sh.go[pass & 1]);
          }
          if (sends) ++sseq;
          if (recvs) ++rseq;
          last_pass = static_cast<int>(pass);
          s = last + 1;
          if (s >= nsteps) { s = 0; finished = ++it >= iterations; }
          setup = true;
        }
        ++pass;
        spins = 0;
        __syncwarp();
      }
      if (stuck) break;
    }
    // the last pass: tells data and signal warps to leave
    for (unsigned int i = 1; ld_signalled(sh) < static_cast<int>(pass) - 1; ++i)
      if ((i & 255u) == 0 && global_timer_ns() > limit) break;
    __syncwarp();
    if (lane == 0) {
      sh.job[pass & 1].kind = JOB_EXIT;
      bar_arrive(&sh.go[pass & 1]);
    }
    if (gl == 0) {
      if (has_send) flags->send_seq[send_conn] = sseq;
      if (has_recv) flags->recv_seq[recv_conn] = rseq;
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

// `args.ctas_per_tb` CTAs per threadblock; cooperative unless the caller vouches for an otherwise idle GPU.
cudaError_t launch_exec_one_gpu(const OneGpuArgs& args, int dtype, int proto, int width, int tbs, cudaStream_t stream, bool cooperative) {
  const void* fn = pick_kernel(dtype, proto, width);
  if (fn == nullptr) return cudaErrorInvalidValue;
  OneGpuArgs copy = args;
  void* params[] = {&copy};
  const dim3 grid(static_cast<unsigned int>(tbs * args.ctas_per_tb)), block(kOgThreads);
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
