// What the two interpreter kernels (exec_kernel.cu: one rank per process; exec_one_gpu.cu: every rank on this GPU) have in
// common: bounded waits, failure records, access widths, and the packet formats of the flag-in-data protocols.
#pragma once
#include <type_traits>

#include "msccl_device.h"
#include "prims.cuh"

namespace msccl {

constexpr unsigned int kFullWarp = 0xffffffffu;

__device__ __forceinline__ unsigned long long pack_progress(unsigned long long epoch, int iter, int step_plus_1) {
  // 32 bits of launch epoch | 20 bits of iteration | 12 bits of step+1 (the host rejects plans beyond these)
  return (epoch << 32) | (static_cast<unsigned long long>(iter & 0xfffff) << 12) |
         static_cast<unsigned long long>(step_plus_1 & 0xfff);
}

struct Waiter {
  SyncPage* sync;
  unsigned long long deadline;

  // Spin until *flag >= want.  Returns false on timeout or when the rank was aborted.
  __device__ bool until_ge(const unsigned long long* flag, unsigned long long want, bool system_scope) const {
    unsigned int spins = 0;
    while (true) {
      unsigned long long v = system_scope ? ld_acquire_sys(flag) : ld_acquire_gpu(flag);
      if (v >= want) return true;
      if ((++spins & 127u) == 0) {
        if (ld_volatile_u32(&sync->abort_flag) != 0) return false;
        if (global_timer_ns() > deadline) return false;
      }
    }
  }
  // The same for a counter that keeps other information above kTailModeShift; the whole word is returned.
  __device__ bool until_count_ge(const unsigned long long* flag, unsigned long long want, unsigned long long* word) const {
    unsigned int spins = 0;
    while (true) {
      const unsigned long long v = ld_acquire_sys(flag);
      if ((v & kTailCountMask) >= want) { *word = v; return true; }
      if ((++spins & 127u) == 0) {
        if (ld_volatile_u32(&sync->abort_flag) != 0) return false;
        if (global_timer_ns() > deadline) return false;
      }
    }
  }
  __device__ bool expired() const {
    return ld_volatile_u32(&sync->abort_flag) != 0 || global_timer_ns() > deadline;
  }
};

__device__ inline void record_failure(SyncPage* sync, unsigned int code, int rank, int tb, int step, int iter,
                               unsigned int aux0, unsigned int aux1) {
  unsigned int already = ld_volatile_u32(&sync->abort_flag);
  if (already != 0 && code != STATUS_ABORTED && code != STATUS_BOUNDS) code = STATUS_ABORTED;
  if (atomicCAS(&sync->status[0], 0u, code) == 0u) {
    sync->status[1] = rank;
    sync->status[2] = tb;
    sync->status[3] = step;
    sync->status[4] = iter;
    sync->status[5] = aux0;
    sync->status[6] = aux1;
  }
  __threadfence();
  atomicExch(&sync->abort_flag, 1u);
}

template <int W> struct Access;
template <> struct Access<16> {
  static __device__ __forceinline__ uint4 ld(const char* p) { return *reinterpret_cast<const uint4*>(p); }
  static __device__ __forceinline__ void st(char* p, uint4 v) { *reinterpret_cast<uint4*>(p) = v; }
};
template <> struct Access<4> {
  static __device__ __forceinline__ unsigned int ld(const char* p) { return *reinterpret_cast<const unsigned int*>(p); }
  static __device__ __forceinline__ void st(char* p, unsigned int v) { *reinterpret_cast<unsigned int*>(p) = v; }
};
template <> struct Access<2> {
  static __device__ __forceinline__ unsigned short ld(const char* p) { return *reinterpret_cast<const unsigned short*>(p); }
  static __device__ __forceinline__ void st(char* p, unsigned short v) { *reinterpret_cast<unsigned short*>(p) = v; }
};

// ---- LL packets -----------------------------------------------------------------------------
// W = 16: two 16-byte packets {data, flag, data, flag} per vector.  W = 4 / 2: one 8-byte packet {data, flag}.
template <int W> struct LLPacket;

template <> struct LLPacket<16> {
  static constexpr int kBytes = 32;
  static __device__ __forceinline__ uint4 load(const char* slot, long long v, unsigned int flag, const Waiter& w, int* fail) {
    const uint4* pk = reinterpret_cast<const uint4*>(slot) + 2 * v;
    uint4 a, b;
    unsigned int spins = 0;
    while (true) {
      a = ld_volatile_v4(pk);
      b = ld_volatile_v4(pk + 1);
      if (a.y == flag && a.w == flag && b.y == flag && b.w == flag) break;
      if ((++spins & 255u) == 0) {
        if (*reinterpret_cast<volatile int*>(fail) != 0 || w.expired()) {
          *reinterpret_cast<volatile int*>(fail) = 1;
          break;
        }
      }
    }
    return make_uint4(a.x, a.z, b.x, b.z);
  }
  static __device__ __forceinline__ void store(char* slot, long long v, uint4 d, unsigned int flag) {
    uint4* pk = reinterpret_cast<uint4*>(slot) + 2 * v;
    st_volatile_v4(pk, make_uint4(d.x, flag, d.y, flag));
    st_volatile_v4(pk + 1, make_uint4(d.z, flag, d.w, flag));
  }
};

template <int W> struct LLPacketNarrow {
  static constexpr int kBytes = 8;
  using VT = typename std::conditional<W == 4, unsigned int, unsigned short>::type;
  static __device__ __forceinline__ VT load(const char* slot, long long v, unsigned int flag, const Waiter& w, int* fail) {
    const uint2* pk = reinterpret_cast<const uint2*>(slot) + v;
    uint2 a;
    unsigned int spins = 0;
    while (true) {
      a = ld_volatile_v2(pk);
      if (a.y == flag) break;
      if ((++spins & 255u) == 0) {
        if (*reinterpret_cast<volatile int*>(fail) != 0 || w.expired()) {
          *reinterpret_cast<volatile int*>(fail) = 1;
          break;
        }
      }
    }
    return static_cast<VT>(a.x);
  }
  static __device__ __forceinline__ void store(char* slot, long long v, VT d, unsigned int flag) {
    st_volatile_v2(reinterpret_cast<uint2*>(slot) + v, make_uint2(static_cast<unsigned int>(d), flag));
  }
};
template <> struct LLPacket<4> : LLPacketNarrow<4> {};
template <> struct LLPacket<2> : LLPacketNarrow<2> {};

// ---- LL128 lines ----------------------------------------------------------------------------
// The payload is counted in 8-byte units; line L carries units [15 L, 15 L + 15).  Lane k of the eight lanes
// that own a line holds units 15 L + 2k and 15 L + 2k + 1; lane 7 holds unit 15 L + 14 and the flag.  The 32
// lanes of a warp store 4 consecutive lines with one 16-byte-per-lane instruction.
__device__ __forceinline__ uint4 ld_units(const char* base, long long u0, long long n8, int k) {
  uint4 r = make_uint4(0, 0, 0, 0);
  if (u0 < n8) {
    const uint2 a = *reinterpret_cast<const uint2*>(base + u0 * 8);
    r.x = a.x; r.y = a.y;
  }
  if (k < 7 && u0 + 1 < n8) {
    const uint2 b = *reinterpret_cast<const uint2*>(base + (u0 + 1) * 8);
    r.z = b.x; r.w = b.y;
  }
  return r;
}
__device__ __forceinline__ void st_units(char* base, long long u0, long long n8, int k, uint4 v) {
  if (u0 < n8) *reinterpret_cast<uint2*>(base + u0 * 8) = make_uint2(v.x, v.y);
  if (k < 7 && u0 + 1 < n8) *reinterpret_cast<uint2*>(base + (u0 + 1) * 8) = make_uint2(v.z, v.w);
}

__device__ __forceinline__ bool is_send(int t) { return t == ST_SEND || t == ST_RCS || t == ST_RRS || t == ST_RRCS; }
__device__ __forceinline__ bool is_recv(int t) {
  return t == ST_RECV || t == ST_RCS || t == ST_RRS || t == ST_RRC || t == ST_RRCS;
}

}  // namespace msccl
