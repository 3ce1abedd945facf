// sm_100a unpack kernels: reassemble scattered rx page fragments on the GPU.
//
// One kernel template covers the four products:
//   K1  unpack_copy            pool fragment -> dst
//   K2  unpack_reduce          dst = acc + pool fragment (bf16 with fp32 add, or fp32)
//   K3  unpack_fanout          K1 + the same fragment stored to every local peer GPU
//   K3r unpack_reduce_fanout   K2 + the reduced fragment stored to every local peer GPU
//
// The reference has no counterpart: with it, NCCL's collective kernels walk the
// scatter list (reference: src/net_tcpx.cc:739-740 declares NCCL_NET_DEVICE_UNPACK;
// src/sock/tcpx.h:136-228 builds the list).  The list format is kept.
//
// Structure.  Persistent grid, one CTA per SM, twelve warps per CTA.  Each warp owns
// a private ring of D shared-memory slots and D mbarriers and walks descriptors
// gw, gw+G, gw+2G, ... (G = warps in the grid).  Per fragment, one elected lane
// issues a bulk-async copy global -> shared (cp.async.bulk, completion counted in
// bytes on the slot's mbarrier); when it lands, the warp optionally adds the
// accumulator tile (also bulk-loaded), and the elected lane issues bulk-async
// stores shared -> global to the local destination and to each peer's mapping.
// D fragments are in flight per warp (4 for the copy, 2 fragment + accumulator
// pairs for the reduce), so an SM keeps 192 KB of loads in the air, which is what
// HBM3e needs to stay busy with 4 KB transfers.  Twelve warps of depth 4 / 2
// measured 2 - 3 % faster on the fused reduce than eight warps of depth 6 / 3.
// Fragments off the 16-byte phase and ragged ends come into the slot as the aligned
// vectors that hold them and are stored by the warp; fragments longer than a slot take
// a warp-cooperative ld/st path.  Long lists and a polling host's short ones go through
// registers instead (unpack_wide_kernel, unpack_few_kernel).
//
// Every wait is bounded: on expiry the kernel records TCPXB_ST_TIMEOUT in the
// status block, stops issuing, waits only for the loads already in flight and
// returns; it never traps and never spins forever.  A launch that recorded any error
// does not publish its fan-out completion flag: the peers then run into their own
// bounded flag wait instead of taking partly written output for complete.
// No load in this file is a cluster-wide one; peers are reached by stores only.
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

#include <mutex>
#include <type_traits>

#include "tcpxb/kernels.h"

namespace {

#ifndef TCPXB_WARPS
#define TCPXB_WARPS 12
#endif
#ifndef TCPXB_DEPTH_COPY
#define TCPXB_DEPTH_COPY 4
#endif
#ifndef TCPXB_DEPTH_REDUCE
#define TCPXB_DEPTH_REDUCE 2
#endif
constexpr int kWarps = TCPXB_WARPS;
constexpr int kThreads = kWarps * 32;
constexpr int kSlot = TCPXB_FRAG_BYTES;
constexpr uint64_t kDefaultWaitNs = 2000000000ull;

enum FanMode { FAN_NONE = 0, FAN_PEER = 1, FAN_NVLS = 2 };

struct UnpackParams {
  const uint8_t* pool;
  uint64_t pool_bytes;
  uint8_t* dst;
  uint64_t dst_bytes;
  const uint8_t* acc;
  uint8_t* mc_dst;
  const tcpxbLoadMeta* descs;
  uint32_t count;
  int npeers;
  uint8_t* peers[TCPXB_MAX_PEERS];
  uint32_t* peer_flags[TCPXB_MAX_PEERS];
  uint32_t flag_value;
  uint32_t* ticket;
  uint32_t* done_flag;
  uint32_t done_value;
  uint32_t* status;
  const uint32_t* ready;
  uint64_t wait_ns;
  uint32_t let_in;  // the next launch may come in once this one is past its own wait; 0: once its work is done
};

struct SlotInfo {
  uint64_t src_off;
  uint64_t dst_off;
  uint32_t len;
  uint32_t bulk;     // bytes moved by the bulk path (multiple of 16, may be 0)
  uint32_t shifted;  // what the bulk path leaves of the fragment is in shared memory too
  uint32_t index;    // record
};

// ---------------------------------------------------------------- PTX wrappers
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ uint32_t mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok;
}
__device__ __forceinline__ void bulk_g2s(uint32_t dst_smem, const void* src, uint32_t bytes,
                                         uint32_t bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
          "r"(dst_smem),
      "l"(__cvta_generic_to_global(src)), "r"(bytes), "r"(bar)
      : "memory");
}
// The same load with an L2 eviction-priority hint: rx pool pages are read exactly once.
__device__ __forceinline__ void bulk_g2s_hint(uint32_t dst_smem, const void* src, uint32_t bytes,
                                              uint32_t bar, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::
          "r"(dst_smem),
      "l"(__cvta_generic_to_global(src)), "r"(bytes), "r"(bar), "l"(policy)
      : "memory");
}
__device__ __forceinline__ uint64_t policy_evict_first() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ void bulk_s2g(void* dst, uint32_t src_smem, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(
                   __cvta_generic_to_global(dst)),
               "r"(src_smem), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void bulk_red_bf16(void* dst, uint32_t src_smem, uint32_t bytes) {
  asm volatile(
      "cp.reduce.async.bulk.global.shared::cta.bulk_group.add.noftz.bf16 [%0], [%1], %2;" ::"l"(
          __cvta_generic_to_global(dst)),
      "r"(src_smem), "r"(bytes)
      : "memory");
}
__device__ __forceinline__ void bulk_red_f32(void* dst, uint32_t src_smem, uint32_t bytes) {
  asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f32 [%0], [%1], %2;" ::"l"(
                   __cvta_generic_to_global(dst)),
               "r"(src_smem), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void bulk_commit() {
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
template <int N>
__device__ __forceinline__ void bulk_wait_read() {
  asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void bulk_wait_all() {
  asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ uint64_t globaltimer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ uint32_t ld_acquire_sys(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint4 ld_volatile_v4(const void* p) {
  uint4 v;
  asm volatile("ld.volatile.global.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p)
               : "memory");
  return v;
}
// Weak and not through the read-only path: with programmatic dependent launch a kernel's lifetime
// begins before its predecessor's writes are visible, so nothing may be assumed constant over it.
__device__ __forceinline__ uint4 ld_v4(const void* p) {
  uint4 v;
  asm volatile("ld.global.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p)
               : "memory");
  return v;
}
__device__ __forceinline__ uint4 ld_v4_hint(const void* p, uint64_t policy) {
  uint4 v;
  asm volatile("ld.global.L1::no_allocate.L2::cache_hint.v4.u32 {%0, %1, %2, %3}, [%4], %5;"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p), "l"(policy)
               : "memory");
  return v;
}
struct Vec32 { uint4 lo, hi; };
__device__ __forceinline__ Vec32 ld_v8(const void* p) {
  Vec32 v;
  asm volatile("ld.global.L1::no_allocate.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(v.lo.x), "=r"(v.lo.y), "=r"(v.lo.z), "=r"(v.lo.w), "=r"(v.hi.x), "=r"(v.hi.y), "=r"(v.hi.z), "=r"(v.hi.w)
               : "l"(p)
               : "memory");
  return v;
}
__device__ __forceinline__ Vec32 ld_v8_evict_first(const void* p) {
  Vec32 v;
  asm volatile("ld.global.L1::no_allocate.L2::evict_first.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(v.lo.x), "=r"(v.lo.y), "=r"(v.lo.z), "=r"(v.lo.w), "=r"(v.hi.x), "=r"(v.hi.y), "=r"(v.hi.z), "=r"(v.hi.w)
               : "l"(p)
               : "memory");
  return v;
}
__device__ __forceinline__ void st_v8(void* p, const Vec32& v) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(v.lo.x), "r"(v.lo.y), "r"(v.lo.z),
               "r"(v.lo.w), "r"(v.hi.x), "r"(v.hi.y), "r"(v.hi.z), "r"(v.hi.w)
               : "memory");
}
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void st_release_sys(uint32_t* p, uint32_t v) {
  asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void multimem_st_v4(void* mc, uint4 v) {
  asm volatile("multimem.st.weak.global.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(mc),
               "f"(__uint_as_float(v.x)), "f"(__uint_as_float(v.y)), "f"(__uint_as_float(v.z)),
               "f"(__uint_as_float(v.w))
               : "memory");
}
__device__ __forceinline__ void multimem_red_bf16x8(void* mc, uint4 v) {
  asm volatile("multimem.red.relaxed.sys.global.add.v4.bf16x2 [%0], {%1, %2, %3, %4};" ::"l"(mc),
               "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
               : "memory");
}
__device__ __forceinline__ void multimem_red_f32x4(void* mc, uint4 v) {
  asm volatile("multimem.red.relaxed.sys.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(mc),
               "f"(__uint_as_float(v.x)), "f"(__uint_as_float(v.y)), "f"(__uint_as_float(v.z)),
               "f"(__uint_as_float(v.w))
               : "memory");
}

__device__ __forceinline__ void report(uint32_t* status, uint32_t code, uint32_t index) {
  if (status == nullptr) return;
  if (atomicCAS(&status[0], 0u, code) == 0u) status[1] = index;
  atomicAdd(&status[2], 1u);
}

// Bounded mbarrier wait: every lane polls, so every lane observes the phase and
// with it the bytes the async proxy wrote.  Returns false when time ran out.
__device__ __forceinline__ bool mbar_wait_bounded(uint32_t bar, uint32_t parity, uint64_t limit_ns) {
  uint64_t t0 = 0;
  for (uint32_t spin = 0;; ++spin) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((spin & 0xff) == 0xff) {
      uint64_t now = globaltimer_ns();
      if (t0 == 0) t0 = now;
      else if (now - t0 > limit_ns) return false;
    }
  }
}

// ------------------------------------------------------------ element helpers
__device__ __forceinline__ uint32_t add_bf16x2(uint32_t a, uint32_t b) {
  // bf16 -> fp32 is a 16-bit shift; add in fp32; round to nearest even once.
  float a0 = __uint_as_float(a << 16), a1 = __uint_as_float(a & 0xffff0000u);
  float b0 = __uint_as_float(b << 16), b1 = __uint_as_float(b & 0xffff0000u);
  __nv_bfloat162 r = __floats2bfloat162_rn(a0 + b0, a1 + b1);
  return *reinterpret_cast<uint32_t*>(&r);
}
template <int RED>
__device__ __forceinline__ uint4 add_vec(uint4 a, uint4 b) {
  uint4 r;
  if (RED == TCPXB_BF16) {
    r.x = add_bf16x2(a.x, b.x); r.y = add_bf16x2(a.y, b.y);
    r.z = add_bf16x2(a.z, b.z); r.w = add_bf16x2(a.w, b.w);
  } else {
    r.x = __float_as_uint(__uint_as_float(a.x) + __uint_as_float(b.x));
    r.y = __float_as_uint(__uint_as_float(a.y) + __uint_as_float(b.y));
    r.z = __float_as_uint(__uint_as_float(a.z) + __uint_as_float(b.z));
    r.w = __float_as_uint(__uint_as_float(a.w) + __uint_as_float(b.w));
  }
  return r;
}

template <typename T>
__device__ __forceinline__ void store_all(uint8_t* dst, const UnpackParams& p, int fan,
                                          uint64_t off, T v) {
  *reinterpret_cast<T*>(dst + off) = v;
  if (fan) {
    for (int i = 0; i < p.npeers; ++i) *reinterpret_cast<T*>(p.peers[i] + off) = v;
  }
}

// Loads in flight per lane in the loops below, spelled out: a load behind a store to what may be the same
// address is not moved before it by the compiler, and one load per trip leaves them bound by latency: 1776 pages off the
// phase, added at the destination, 25.4 -> 9.0 us; 3000 fragments of 9000 bytes on 16 CTAs, bf16 sums, 602 -> 296 us.
constexpr int kBatch = 4;

template <typename T>
__device__ __forceinline__ void copy_units(const uint8_t* src, const UnpackParams& p, int fan,
                                           uint64_t dst_off, uint32_t n_units, int lane) {
  for (uint32_t base = lane; base < n_units; base += 32 * kBatch) {
    T v[kBatch];
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const uint32_t i = base + u * 32;
      if (i < n_units) v[u] = *reinterpret_cast<const T*>(src + (uint64_t)i * sizeof(T));
    }
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const uint32_t i = base + u * 32;
      if (i < n_units) store_all<T>(p.dst, p, fan, dst_off + (uint64_t)i * sizeof(T), v[u]);
    }
  }
}

// Why a record is skipped (TCPXB_ST_OK: it is not).
template <int RED>
__device__ __forceinline__ uint32_t refused(const UnpackParams& p, uint32_t src_off, uint32_t len, uint64_t dst_off) {
  if ((uint64_t)src_off + len > p.pool_bytes || dst_off + len > p.dst_bytes || dst_off + len < dst_off) return TCPXB_ST_BOUNDS;
  if (RED != TCPXB_U8) {
    constexpr uint32_t es = (RED == TCPXB_BF16) ? 2 : 4;
    const uintptr_t a = reinterpret_cast<uintptr_t>(p.pool + src_off) | reinterpret_cast<uintptr_t>(p.dst + dst_off) |
                        reinterpret_cast<uintptr_t>(p.acc + dst_off) | len;
    if ((a & (es - 1)) != 0) return TCPXB_ST_ALIGN;
  }
  return TCPXB_ST_OK;
}

// Warp-cooperative generic path for `n` bytes of any alignment: plain loads and
// stores, widest unit the common alignment of source and destination allows.
template <int RED, bool L2RED, int FAN>
__device__ void warp_generic(const UnpackParams& p, uint64_t src_off, uint64_t dst_off, uint32_t n, int lane) {
  if (n == 0) return;
  const uint8_t* src = p.pool + src_off;
  const int fan = (FAN != FAN_NONE);
  if (RED == TCPXB_U8) {
    uintptr_t s = reinterpret_cast<uintptr_t>(src);
    uintptr_t d = reinterpret_cast<uintptr_t>(p.dst + dst_off);
    if (((s ^ d) & 15) == 0) {
      uint32_t head = static_cast<uint32_t>((16 - (s & 15)) & 15);
      if (head > n) head = n;
      copy_units<uint8_t>(src, p, fan, dst_off, head, lane);
      uint32_t body = (n - head) >> 4;
      copy_units<uint4>(src + head, p, fan, dst_off + head, body, lane);
      uint32_t done = head + (body << 4);
      copy_units<uint8_t>(src + done, p, fan, dst_off + done, n - done, lane);
    } else {
      uint32_t a = static_cast<uint32_t>((s | d) & 15);
      uint32_t w = a & (~a + 1);  // lowest set bit: 1, 2, 4 or 8
      uint32_t units, done;
      if (w == 8) { units = n >> 3; copy_units<uint2>(src, p, fan, dst_off, units, lane); done = units << 3; }
      else if (w == 4) { units = n >> 2; copy_units<uint32_t>(src, p, fan, dst_off, units, lane); done = units << 2; }
      else if (w == 2) { units = n >> 1; copy_units<uint16_t>(src, p, fan, dst_off, units, lane); done = units << 1; }
      else { done = 0; }
      copy_units<uint8_t>(src + done, p, fan, dst_off + done, n - done, lane);
    }
  } else {
    constexpr uint32_t es = (RED == TCPXB_BF16) ? 2 : 4;
    using T = typename std::conditional<RED == TCPXB_BF16, __nv_bfloat16, float>::type;
    const uint32_t elems = n / es;
    for (uint32_t base = lane; base < elems; base += 32 * kBatch) {
      T x[kBatch];
#pragma unroll
      for (int u = 0; u < kBatch; ++u) {
        const uint32_t i = base + u * 32;
        if (i < elems) x[u] = reinterpret_cast<const T*>(src)[i];
      }
      // `to` (and with `all` the peers as well) = `with` + the fragment
      auto add = [&](const uint8_t* with, uint8_t* to, int all) {
        T y[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
          const uint32_t i = base + u * 32;
          if (i < elems) y[u] = reinterpret_cast<const T*>(with + dst_off)[i];
        }
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
          const uint32_t i = base + u * 32;
          if (i < elems) store_all<T>(to, p, all, dst_off + (uint64_t)i * es, static_cast<T>(static_cast<float>(x[u]) + static_cast<float>(y[u])));
        }
      };
      if (L2RED) {
        // reduce-into-all form: each buffer adds the fragment to its own value
        add(p.dst, p.dst, 0);
        if (fan) for (int r = 0; r < p.npeers; ++r) add(p.peers[r], p.peers[r], 0);
      } else {
        add(p.acc, p.dst, fan);
      }
    }
  }
}

// The 16 bytes that start `4 * word + shift / 8` bytes into a:b.
__device__ __forceinline__ uint4 take_vec(const uint4& a, const uint4& b, uint32_t word, uint32_t shift) {
  uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
  if (word & 2) {
#pragma unroll
    for (int i = 0; i < 6; ++i) w[i] = w[i + 2];
  }
  if (word & 1) {
#pragma unroll
    for (int i = 0; i < 5; ++i) w[i] = w[i + 1];
  }
  return make_uint4(__funnelshift_r(w[0], w[1], shift), __funnelshift_r(w[1], w[2], shift), __funnelshift_r(w[2], w[3], shift),
                    __funnelshift_r(w[3], w[4], shift));
}

// 16 bytes of shared memory, `q` bytes into the aligned vector at `v`.
__device__ __forceinline__ uint4 vec_at(const uint8_t* v, uint32_t q) {
  const uint4 a = *reinterpret_cast<const uint4*>(v);
  return q == 0 ? a : take_vec(a, *reinterpret_cast<const uint4*>(v + 16), q >> 2, (q & 3) * 8);
}

// A fragment whose source (and accumulator) lie in shared memory at a phase of their own: `sphase` and `aphase`
// bytes behind the 16-byte aligned `sbase` and `abase`.  The warp writes whole destination vectors; what is before the
// first and behind the last goes one element at a time.  Bound by the stores: with 4-byte ones (128 bytes per
// instruction) 3000 fragments of 1448 bytes to three more buffers took 8.6 us on the whole GPU, and packing 8 MiB of them into host memory
// on 16 CTAs 202 us; with whole vectors 5.1 us and 172.
template <int RED, int FAN>
__device__ __forceinline__ void store_shifted(const UnpackParams& p, const uint8_t* sbase, uint32_t sphase, const uint8_t* abase,
                                              uint32_t aphase, uint64_t dst_off, uint32_t n, int lane) {
  const int fan = (FAN != FAN_NONE);
  uint32_t head = static_cast<uint32_t>((16 - (reinterpret_cast<uintptr_t>(p.dst + dst_off) & 15)) & 15);
  if (head > n) head = n;
  const uint32_t vecs = (n - head) >> 4, sat = sphase + head, aat = aphase + head;
  for (uint32_t i = lane; i < vecs; i += 32) {
    const uint32_t o = i << 4;
    uint4 v = vec_at(sbase + (sat & ~15u) + o, sat & 15);
    if (RED) v = add_vec<RED>(vec_at(abase + (aat & ~15u) + o, aat & 15), v);
    store_all<uint4>(p.dst, p, fan, dst_off + head + o, v);
  }
  // at most 15 bytes on either side: lanes 0.. take the head, lanes 16.. the tail
  constexpr uint32_t es = RED == TCPXB_U8 ? 1 : RED == TCPXB_BF16 ? 2 : 4;
  const uint32_t o = lane < 16 ? lane * es : head + (vecs << 4) + (lane - 16) * es;
  if (lane < 16 ? o < head : o < n) {
    if (RED == TCPXB_U8) {
      store_all<uint8_t>(p.dst, p, fan, dst_off + o, sbase[sphase + o]);
    } else if (RED == TCPXB_BF16) {
      const float x = __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(sbase + sphase + o));
      const float y = __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(abase + aphase + o));
      store_all<__nv_bfloat16>(p.dst, p, fan, dst_off + o, __float2bfloat16_rn(x + y));
    } else {
      store_all<float>(p.dst, p, fan, dst_off + o, *reinterpret_cast<const float*>(abase + aphase + o) + *reinterpret_cast<const float*>(sbase + sphase + o));
    }
  }
}

// ------------------------------------------------------------------ the kernel
template <int RED, bool L2RED, int FAN>
struct Cfg {
  static constexpr bool kAccSlot = (RED != TCPXB_U8) && !L2RED;
  // A slot holds a fragment and the up to 15 bytes on either side that complete its 16-byte vectors.
  static constexpr int kSlotBytes = kSlot + 16;
  static constexpr int kStride = kAccSlot ? 2 * kSlotBytes : kSlotBytes;
  static constexpr int kDepth = kAccSlot ? TCPXB_DEPTH_REDUCE : TCPXB_DEPTH_COPY;
  static constexpr int kDataBytes = kWarps * kDepth * kStride;
  static constexpr int kSmemBytes = kDataBytes + kWarps * kDepth * (8 + (int)sizeof(SlotInfo));
  static_assert(kSmemBytes + 1024 <= 227 * 1024, "slot rings must fit one CTA's shared memory");
};

// At most 80 registers per thread, as for two CTAs per SM, although the slot rings leave room for one: a CTA of another
// kernel has to fit beside one that waits for its producer, 1024 threads of 32 registers included (stage_out_kernel).
template <int RED, bool L2RED, int FAN>
__global__ void __launch_bounds__(kThreads, 2)
unpack_kernel(const __grid_constant__ UnpackParams p) {
  using C = Cfg<RED, L2RED, FAN>;
  extern __shared__ __align__(1024) uint8_t smem[];
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  constexpr uint32_t D = (uint32_t)C::kDepth;
  constexpr uint32_t half = (uint32_t)C::kSlotBytes;  // one slot, or the fragment half of a pair
  constexpr uint32_t stride = (uint32_t)C::kStride;
  uint8_t* wbuf = smem + warp * C::kDepth * C::kStride;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::kDataBytes) + warp * C::kDepth;
  SlotInfo* infos = reinterpret_cast<SlotInfo*>(smem + C::kDataBytes + kWarps * C::kDepth * 8) + warp * C::kDepth;

  // Programmatic dependent launch.  As the later kernel: everything up to the wait below
  // touches only this CTA's shared memory; the wait returns when the previous kernel of the
  // stream has completed and its writes are visible.  As the earlier one: see launchDependent.
  __shared__ uint32_t cta_err;  // any warp of this CTA recorded an error
  if (threadIdx.x == 0) cta_err = 0;
  if (lane < (int)D) mbar_init(smem_u32(&bars[lane]), 1);
  fence_mbar_init();
  __syncthreads();
  pdl_wait();
  if (p.let_in) pdl_launch_dependents();
  auto record = [&](uint32_t code, uint32_t index) {  // one lane calls this
    report(p.status, code, index);
    atomicOr(&cta_err, 1u);
  };

  // Consecutive descriptors go to different SMs first, then to different warps.
  const uint32_t G = gridDim.x * kWarps;
  const uint32_t gw = warp * gridDim.x + blockIdx.x;
  const uint32_t n = (gw < p.count) ? (p.count - gw + G - 1) / G : 0;
  const uint64_t wait_ns = p.wait_ns ? p.wait_ns : kDefaultWaitNs;

  const uint64_t pool_policy = policy_evict_first();
  uint32_t cached_blk = 0xffffffffu;
  uint4 cached = make_uint4(0, 0, 0, 0);
  uint32_t ready_seen = 0;
  uint64_t ready_t0 = 0;
  bool dead = false;  // a bounded wait ran out: stop issuing, drain what is in flight
  uint32_t issued = 0;  // local iterations whose loads were issued

  // Issue the loads of local iteration k into slot k % D.  Warp-uniform.
  auto issue = [&](uint32_t k) {
    const uint32_t slot = k % D;
    const uint32_t idx = gw + k * G;
    issued = k + 1;
    uint32_t so, ln, dlo, dhi;
    if (p.ready != nullptr) {
      // Streaming: descriptor idx exists once the producer's counter passed it.
      if (lane == 0 && ready_seen <= idx) {
        for (uint32_t spin = 0;; ++spin) {
          const uint32_t before = ready_seen;
          ready_seen = ld_acquire_sys(p.ready);
          if (ready_seen != before) ready_t0 = 0;  // the producer moved: the limit bounds its silence, not the launch
          if (ready_seen > idx) break;
          if ((spin & 0x3f) == 0x3f) {
            uint64_t now = globaltimer_ns();
            if (ready_t0 == 0) ready_t0 = now;
            else if (now - ready_t0 > wait_ns) break;
          }
          __nanosleep(200);
        }
      }
      ready_seen = __shfl_sync(0xffffffffu, ready_seen, 0);
      uint4 d = make_uint4(0, 0, 0, 0);
      if (ready_seen <= idx) {
        if (lane == 0) record(TCPXB_ST_TIMEOUT, idx);
        dead = true;
      } else if (lane == 0) {
        d = ld_volatile_v4(&p.descs[idx]);
      }
      so = __shfl_sync(0xffffffffu, d.x, 0);
      ln = __shfl_sync(0xffffffffu, d.y, 0);
      dlo = __shfl_sync(0xffffffffu, d.z, 0);
      dhi = __shfl_sync(0xffffffffu, d.w, 0);
    } else {
      const uint32_t blk = k >> 5;
      if (blk != cached_blk) {
        const uint32_t kk = (blk << 5) + lane;
        if (kk < n) cached = ld_v4(&p.descs[gw + (uint64_t)kk * G]);
        cached_blk = blk;
      }
      so = __shfl_sync(0xffffffffu, cached.x, k & 31);
      ln = __shfl_sync(0xffffffffu, cached.y, k & 31);
      dlo = __shfl_sync(0xffffffffu, cached.z, k & 31);
      dhi = __shfl_sync(0xffffffffu, cached.w, k & 31);
    }
    const uint64_t dof = (static_cast<uint64_t>(dhi) << 32) | dlo;
    if (dead) ln = 0;
    const uint32_t bad = refused<RED>(p, so, ln, dof);
    if (bad != TCPXB_ST_OK) {
      if (lane == 0) record(bad, idx);
      ln = 0;
    }
    const uintptr_t sa = reinterpret_cast<uintptr_t>(p.pool + so);
    const uintptr_t aa = reinterpret_cast<uintptr_t>(p.acc + dof);
    uintptr_t al = sa | reinterpret_cast<uintptr_t>(p.dst + dof);
    if (C::kAccSlot) al |= aa;
    const bool fits = ln <= (uint32_t)kSlot;
    const uint32_t bulk = ((al & 15) == 0 && fits) ? (ln & ~15u) : 0u;
    // off the 16-byte phase, or with a ragged end: that part is stored by the warp out of shared memory
    const bool shifted = !L2RED && ((al | ln) & 15) != 0 && fits && ln != 0;
    if (lane == 0) {
      infos[slot].src_off = so;
      infos[slot].dst_off = dof;
      infos[slot].len = ln;
      infos[slot].bulk = bulk;
      infos[slot].shifted = shifted;
      infos[slot].index = idx;
      const uint32_t bar = smem_u32(&bars[slot]);
      const uint32_t sm = smem_u32(wbuf + slot * stride);
      if (shifted) {
        // the 16-byte vectors that hold the fragment: they reach at most 15 bytes beyond it on either
        // side, inside the same aligned vector and so inside the same allocation
        const uint32_t sbytes = ((uint32_t)(sa & 15) + ln + 15u) & ~15u;
        const uint32_t abytes = C::kAccSlot ? (((uint32_t)(aa & 15) + ln + 15u) & ~15u) : 0u;
        mbar_expect_tx(bar, sbytes + abytes);
        bulk_g2s_hint(sm, reinterpret_cast<const void*>(sa & ~(uintptr_t)15), sbytes, bar, pool_policy);
        if (C::kAccSlot) bulk_g2s(sm + half, reinterpret_cast<const void*>(aa & ~(uintptr_t)15), abytes, bar);
      } else if (bulk) {
        mbar_expect_tx(bar, C::kAccSlot ? 2 * bulk : bulk);
        bulk_g2s_hint(sm, p.pool + so, bulk, bar, pool_policy);
        if (C::kAccSlot) bulk_g2s(sm + half, p.acc + dof, bulk, bar);
      } else {
        mbar_arrive(bar);
      }
    }
    __syncwarp();
  };

  const uint32_t pro = n < D ? n : D;
  for (uint32_t k = 0; k < pro && !dead; ++k) issue(k);  // a wait that ran out is not repeated for the next slot

  for (uint32_t k = 0; k < n; ++k) {
    // After a time-out only the loads already issued are waited for (at most D of
    // them, each with a shortened limit): the drain takes about one wait, not n of them.
    if (dead && k >= issued) break;
    const uint32_t slot = k % D;
    const uint32_t parity = (k / D) & 1;
    const uint32_t bar = smem_u32(&bars[slot]);
    if (!mbar_wait_bounded(bar, parity, dead ? (wait_ns >> 3) + 1 : wait_ns)) {
      if (lane == 0 && !dead) record(TCPXB_ST_TIMEOUT, infos[slot].index);
      dead = true;
    }
    dead = __any_sync(0xffffffffu, dead);
    const SlotInfo info = infos[slot];
    uint8_t* sfrag = wbuf + slot * stride;
    uint8_t* sout = sfrag;
    if (info.bulk && !dead) {
      if (C::kAccSlot) {
        sout = sfrag + half;
        const uint32_t vecs = info.bulk >> 4;
        for (uint32_t i = lane; i < vecs; i += 32) {
          uint4 a = *reinterpret_cast<const uint4*>(sfrag + (i << 4));
          uint4 b = *reinterpret_cast<const uint4*>(sout + (i << 4));
          *reinterpret_cast<uint4*>(sout + (i << 4)) = add_vec<RED>(b, a);
        }
        if (FAN != FAN_NVLS) fence_proxy_async_smem();
        __syncwarp();
      }
      if (FAN == FAN_NVLS) {
        // One multimem instruction per 16 B reaches every GPU of the group,
        // this one included, through the switch.
        const uint32_t vecs = info.bulk >> 4;
        for (uint32_t i = lane; i < vecs; i += 32) {
          uint4 v = *reinterpret_cast<const uint4*>(sout + (i << 4));
          void* mc = p.mc_dst + info.dst_off + (i << 4);
          if (L2RED) {
            if (RED == TCPXB_BF16) multimem_red_bf16x8(mc, v);
            else multimem_red_f32x4(mc, v);
          } else {
            multimem_st_v4(mc, v);
          }
        }
        __syncwarp();
      } else if (lane == 0) {
        const uint32_t s = smem_u32(sout);
        if (L2RED) {
          if (RED == TCPXB_BF16) bulk_red_bf16(p.dst + info.dst_off, s, info.bulk);
          else bulk_red_f32(p.dst + info.dst_off, s, info.bulk);
          if (FAN == FAN_PEER) {
            for (int r = 0; r < p.npeers; ++r) {
              if (RED == TCPXB_BF16) bulk_red_bf16(p.peers[r] + info.dst_off, s, info.bulk);
              else bulk_red_f32(p.peers[r] + info.dst_off, s, info.bulk);
            }
          }
        } else {
          bulk_s2g(p.dst + info.dst_off, s, info.bulk);
          if (FAN == FAN_PEER) {
            for (int r = 0; r < p.npeers; ++r) bulk_s2g(p.peers[r] + info.dst_off, s, info.bulk);
          }
        }
      }
    }
    // An (often empty) group per iteration keeps "all but the newest group" equal
    // to "every store of the iterations before this one".
    if (lane == 0) bulk_commit();
    if (!dead) {
      if (!L2RED && info.shifted) {
        // all of the fragment, or the up to 15 bytes behind its last whole vector
        store_shifted<RED, FAN>(p, sfrag + info.bulk, (uint32_t)(reinterpret_cast<uintptr_t>(p.pool + info.src_off) & 15),
                                sfrag + half + info.bulk, (uint32_t)(reinterpret_cast<uintptr_t>(p.acc + info.dst_off) & 15),
                                info.dst_off + info.bulk, info.len - info.bulk, lane);
        __syncwarp();
      } else if (info.len > info.bulk) {
        warp_generic<RED, L2RED, FAN>(p, info.src_off + info.bulk, info.dst_off + info.bulk, info.len - info.bulk, lane);
      }
    }
    // Refill the slot of the previous iteration: its store has had one iteration
    // to read shared memory, so this wait rarely blocks.
    if (k >= 1 && (k - 1) + D < n && !dead) {
      if (lane == 0) bulk_wait_read<1>();
      __syncwarp();
      issue((k - 1) + D);
    }
  }
  if (lane == 0) bulk_wait_all();
  if (!p.let_in) {
    __syncthreads();  // the first thread to say so speaks for the whole CTA
    pdl_launch_dependents();
  }

  if ((p.flag_value != 0 || p.done_flag != nullptr) && p.ticket != nullptr) {
    // Publish completion once every CTA's stores are done: to the peers (unless there were errors), and to
    // a host that watches a mapped word.
    // The ticket counts CTAs in its low half and CTAs with errors in its high half.
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence_system();
      const uint32_t mine = 1u + (cta_err ? 0x10000u : 0u);
      const uint32_t t = atomicAdd(p.ticket, mine) + mine;
      if ((t & 0xffffu) == gridDim.x) {
        *p.ticket = 0;
        __threadfence_system();
        if (p.flag_value != 0 && (t >> 16) == 0) {
          for (int r = 0; r < TCPXB_MAX_PEERS; ++r) {
            if (p.peer_flags[r] != nullptr) st_release_sys(p.peer_flags[r], p.flag_value);
          }
        }
        if (p.done_flag != nullptr) st_release_sys(p.done_flag, p.done_value);
      }
    }
  }
}

// ------------------------------------------------------------ long scatter lists
// K1 and K2 for lists of more records than the ring kernel has warps (wide_from below): one warp per record, through
// registers, as many CTAs as that takes.  What bounds it is HBM; what it saves against the ring kernel is the
// last, part-filled round of a persistent grid (the hardware hands a finished SM its next CTA) and, for
// fragments off the 16-byte phase, the trip through shared memory: a warp shifts its vectors into the
// destination's phase with lane exchanges.  A whole aligned page goes as 32-byte loads and stores; 4 x 16 bytes
// per lane are in flight per step, which leaves room for 32 warps per SM (24 in the reduce).  Steps of 8 x 16
// bytes are as fast on whole pages, but half of one is wasted on a 1448-byte fragment (10.5 against 7.8 us).
// Measured inside CUDA graphs, ring kernel -> this one: copy of 64 MiB in pages 24.2 -> 23.0 us (0.87 -> 0.91 of the
// measured copy rate), reduce 33.6 -> 31.8 us; 16 MiB in 1448-byte fragments 10.0 -> 7.6 us.
constexpr int kWideThreads = 256;
constexpr int kWideWarps = kWideThreads / 32;
constexpr int kWideUnroll = 4;
template <int RED>
__device__ __forceinline__ void wide_record(const UnpackParams& p, const uint4& d, uint32_t idx, uint64_t pool_policy, int lane) {
  constexpr int U = kWideUnroll;
  constexpr uint32_t es = RED == TCPXB_U8 ? 1 : RED == TCPXB_BF16 ? 2 : 4;
  const uint32_t n = d.y;
  const uint64_t dof = (static_cast<uint64_t>(d.w) << 32) | d.z;
  const uint32_t bad = refused<RED>(p, d.x, n, dof);
  if (bad != TCPXB_ST_OK) {
    if (lane == 0) report(p.status, bad, idx);
    return;
  }
  const uint8_t* s = p.pool + d.x;
  const uint8_t* a = p.acc + dof;
  uint8_t* t = p.dst + dof;
  const uintptr_t phases = reinterpret_cast<uintptr_t>(s) | reinterpret_cast<uintptr_t>(t) | (RED ? reinterpret_cast<uintptr_t>(a) : 0);
  if (n == (uint32_t)kSlot && (phases & 31) == 0) {
#pragma unroll
    for (int h = 0; h < kSlot / (U * 512); ++h) {
      Vec32 v[U / 2], c[U / 2];
      const uint32_t off = h * U * 512 + lane * 32;
#pragma unroll
      for (int u = 0; u < U / 2; ++u) v[u] = ld_v8_evict_first(s + off + u * 1024);
      if (RED) {
#pragma unroll
        for (int u = 0; u < U / 2; ++u) c[u] = ld_v8(a + off + u * 1024);
#pragma unroll
        for (int u = 0; u < U / 2; ++u) {
          v[u].lo = add_vec<RED>(c[u].lo, v[u].lo);
          v[u].hi = add_vec<RED>(c[u].hi, v[u].hi);
        }
      }
#pragma unroll
      for (int u = 0; u < U / 2; ++u) st_v8(t + off + u * 1024, v[u]);
    }
    return;
  }
  if (RED && ((reinterpret_cast<uintptr_t>(a) ^ reinterpret_cast<uintptr_t>(t)) & 15) != 0) {
    warp_generic<RED, false, FAN_NONE>(p, d.x, dof, n, lane);  // accumulator and output in different phases
    return;
  }
  // whole destination vectors, and up to 15 bytes on either side: one element each for lanes 0.. and 16..
  uint32_t head = static_cast<uint32_t>((16 - (reinterpret_cast<uintptr_t>(t) & 15)) & 15);
  if (head > n) head = n;
  const uint32_t vecs = (n - head) >> 4;
  const uint32_t q = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(s + head) & 15);
  const uint32_t edge = lane < 16 ? lane * es : head + (vecs << 4) + (lane - 16) * es;
  const bool has_edge = lane < 16 ? edge < head : edge < n;
  uint32_t ev = 0, ea = 0;
  if (has_edge) {
    if (RED == TCPXB_U8) ev = s[edge];
    if (RED == TCPXB_BF16) { ev = *reinterpret_cast<const uint16_t*>(s + edge); ea = *reinterpret_cast<const uint16_t*>(a + edge); }
    if (RED == TCPXB_F32) { ev = *reinterpret_cast<const uint32_t*>(s + edge); ea = *reinterpret_cast<const uint32_t*>(a + edge); }
  }
  const uint8_t* sv = s + head - q;  // aligned; with q != 0 the vectors are taken out of one more source vector
  const uint32_t loads = vecs + (q != 0 && vecs != 0 ? 1 : 0);
  for (uint32_t base = 0; base < vecs; base += 32 * U) {
    uint4 v[U], c[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint32_t i = base + u * 32 + lane;
      v[u] = i < loads ? ld_v4_hint(sv + ((uint64_t)i << 4), pool_policy) : make_uint4(0, 0, 0, 0);
    }
    if (RED) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const uint32_t i = base + u * 32 + lane;
        c[u] = i < vecs ? ld_v4(a + head + ((uint64_t)i << 4)) : make_uint4(0, 0, 0, 0);
      }
    }
    if (q != 0) {
      const uint32_t after = base + 32 * U;  // the vector behind this step's last
      const uint4 beyond = after < loads ? ld_v4_hint(sv + ((uint64_t)after << 4), pool_policy) : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const uint4& nb = u + 1 < U ? v[u + 1 < U ? u + 1 : u] : beyond;
        uint4 next = make_uint4(__shfl_down_sync(0xffffffffu, v[u].x, 1), __shfl_down_sync(0xffffffffu, v[u].y, 1),
                                __shfl_down_sync(0xffffffffu, v[u].z, 1), __shfl_down_sync(0xffffffffu, v[u].w, 1));
        const uint4 wrap = make_uint4(__shfl_sync(0xffffffffu, nb.x, 0), __shfl_sync(0xffffffffu, nb.y, 0),
                                      __shfl_sync(0xffffffffu, nb.z, 0), __shfl_sync(0xffffffffu, nb.w, 0));
        if (lane == 31) next = wrap;
        v[u] = take_vec(v[u], next, q >> 2, (q & 3) * 8);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint32_t i = base + u * 32 + lane;
      if (i < vecs) *reinterpret_cast<uint4*>(t + head + ((uint64_t)i << 4)) = RED ? add_vec<RED>(c[u], v[u]) : v[u];
    }
  }
  if (has_edge) {
    if (RED == TCPXB_U8) t[edge] = static_cast<uint8_t>(ev);
    if (RED == TCPXB_BF16)
      *reinterpret_cast<__nv_bfloat16*>(t + edge) = __float2bfloat16_rn(__uint_as_float(ev << 16) + __uint_as_float(ea << 16));
    if (RED == TCPXB_F32) *reinterpret_cast<float*>(t + edge) = __uint_as_float(ev) + __uint_as_float(ea);
  }
}

template <int RED>
__global__ void __launch_bounds__(kWideThreads, RED == TCPXB_U8 ? 4 : 3)
unpack_wide_kernel(const __grid_constant__ UnpackParams p) {
  const uint32_t idx = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;  // neighbours in the list go to different SMs
  const uint64_t pool_policy = policy_evict_first();
  if (idx >= p.count) return;
  pdl_wait();
  pdl_launch_dependents();
  wide_record<RED>(p, ld_v4(&p.descs[idx]), idx, pool_policy, threadIdx.x & 31);
}

// A small request of a polling host: its records ride in the launch's parameters, which saves the trip over PCIe that
// fetching them costs, and one CTA needs neither shared memory nor a count of CTAs to say that it is done.  All
// latency: the launch, one read of the pool, the write of the completion word.  all_reduce with the ring kernel -> with
// this one: 1 KiB 46.8 -> 43.9 us, 4 KiB 47.4 -> 44.8, 16 KiB 49.2 -> 47.4; more than 8 records (64 KiB: 59.8 both) stay there.
constexpr int kFewRecords = kWideWarps;
struct FewParams {
  UnpackParams p;
  uint4 recs[kFewRecords];
};
template <int RED>
__global__ void __launch_bounds__(kWideThreads, 1) unpack_few_kernel(const __grid_constant__ FewParams q) {
  const uint32_t warp = threadIdx.x >> 5;
  const uint64_t pool_policy = policy_evict_first();
  pdl_wait();
  if (warp < q.p.count) wide_record<RED>(q.p, q.recs[warp], warp, pool_policy, threadIdx.x & 31);
  __syncthreads();
  if (threadIdx.x == 0 && q.p.done_flag != nullptr) {
    __threadfence_system();
    st_release_sys(q.p.done_flag, q.p.done_value);
  }
}

// Bounded wait for peer completion flags; one warp, lane i watches flags[i].
__global__ void wait_flags_kernel(const uint32_t* flags, int n, uint32_t value, uint64_t wait_ns,
                                  uint32_t* status) {
  // Lets nothing in: a kernel behind this one would hold SMs while this one waits for a peer.
  const int i = threadIdx.x;
  pdl_wait();
  if (i >= n) return;
  uint64_t t0 = globaltimer_ns();
  for (;;) {
    uint32_t v = ld_acquire_sys(&flags[i]);
    if ((int32_t)(v - value) >= 0) return;
    if (globaltimer_ns() - t0 > wait_ns) {
      report(status, TCPXB_ST_TIMEOUT, (uint32_t)i);
      return;
    }
    __nanosleep(100);
  }
}

struct SignalParams {
  uint32_t* flags[TCPXB_MAX_PEERS + 1];
  int n;
  uint32_t value;
};
__global__ void signal_flags_kernel(const __grid_constant__ SignalParams p) {
  const int i = threadIdx.x;
  pdl_wait();
  pdl_launch_dependents();
  if (i < p.n && p.flags[i] != nullptr) {
    __threadfence_system();
    st_release_sys(p.flags[i], p.value);
  }
}

// Device memory -> mapped host memory, then a flag.  Bound by the latency of the launch and of one PCIe write:
// one CTA moves all of it (up to 64 KiB in the engine), so that the flag needs no counting of CTAs.  Against the
// copy engine behind an event, with a stream memory operation as the flag, and the same for the unpack kernel's
// end: an all_reduce of 1 KiB 53 -> 49 us, of 64 KiB 66 -> 60 us.
constexpr int kStageThreads = 1024;
__global__ void __launch_bounds__(kStageThreads)
stage_out_kernel(const uint8_t* src, uint8_t* dst, uint64_t bytes, uint32_t* flag, uint32_t value) {
  const uint64_t vecs = ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15) == 0 ? bytes >> 4 : 0;
  pdl_wait();
#pragma unroll 4
  for (uint64_t i = threadIdx.x; i < vecs; i += blockDim.x) *reinterpret_cast<uint4*>(dst + (i << 4)) = ld_v4(src + (i << 4));
  for (uint64_t i = (vecs << 4) + threadIdx.x; i < bytes; i += blockDim.x) dst[i] = src[i];
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence_system();
    st_release_sys(flag, value);
  }
}

// out[i] = sum_r srcs[r][shard_off + i], fp32 adds.
constexpr int kMaxSources = TCPXB_MAX_PEERS + 1;
struct PeerReduceParams {
  const uint8_t* srcs[kMaxSources];
  uint8_t* out;
  uint64_t shard_off;
  uint64_t vecs;
};
// Sum of one vector of every source, in the order of the sources.
template <int RED, int N>
__device__ __forceinline__ uint4 sum_sources(const uint4 (&v)[N]) {
  if (RED == TCPXB_BF16) {
    float acc[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] = 0.f;
#pragma unroll
    for (int r = 0; r < N; ++r) {
      const uint32_t w[4] = {v[r].x, v[r].y, v[r].z, v[r].w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        acc[2 * j] += __uint_as_float(w[j] << 16);
        acc[2 * j + 1] += __uint_as_float(w[j] & 0xffff0000u);
      }
    }
    uint32_t o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const __nv_bfloat162 t = __floats2bfloat162_rn(acc[2 * j], acc[2 * j + 1]);
      o[j] = *reinterpret_cast<const uint32_t*>(&t);
    }
    return make_uint4(o[0], o[1], o[2], o[3]);
  }
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int r = 0; r < N; ++r) {
    acc.x += __uint_as_float(v[r].x); acc.y += __uint_as_float(v[r].y);
    acc.z += __uint_as_float(v[r].z); acc.w += __uint_as_float(v[r].w);
  }
  return make_uint4(__float_as_uint(acc.x), __float_as_uint(acc.y), __float_as_uint(acc.z), __float_as_uint(acc.w));
}

// Bound by HBM (or NVLink, for peers' memory).  A thread sums 32 bytes of every source where all addresses allow it
// (WIDE), 16 otherwise; as many CTAs as that takes, so that no round of a persistent grid is part-filled.  One variant
// per number of sources N: registers for absent ones would cost warps in flight, predicates on a number that only the
// launch knows cost load slots.  Measured inside CUDA graphs, 16-byte loads in a persistent grid of 8 x 256 threads per SM ->
// this, out of HBM and (in brackets) out of L2: four bf16 sources of 16 MiB 14.5 -> 13.4 us (8.0 -> 6.4), 0.95 of the
// copy rate; eight fp32 ones of 4 MiB 7.5 -> 6.9 (3.6 -> 3.3); five of 16 MiB 16.4 -> 15.7 (11.4 -> 11.0), where one
// variant for up to nine took 17.6 (14.7).
constexpr int kPeerThreads = 256;
template <int RED, int N, bool WIDE>
__global__ void __launch_bounds__(kPeerThreads) peer_reduce_kernel(const __grid_constant__ PeerReduceParams p) {
  const uint64_t i = ((uint64_t)blockIdx.x * kPeerThreads + threadIdx.x) * (WIDE ? 2 : 1);
  if (i >= p.vecs) return;
  const uint64_t off = p.shard_off + (i << 4);
  pdl_wait();
  pdl_launch_dependents();
  if (WIDE && i + 1 < p.vecs) {
    uint4 lo[N], hi[N];
#pragma unroll
    for (int r = 0; r < N; ++r) {
      const Vec32 v = ld_v8(p.srcs[r] + off);
      lo[r] = v.lo;
      hi[r] = v.hi;
    }
    __syncwarp(__activemask());  // keeps the adds behind all of the loads: the compiler would wait for the first source first
    const Vec32 o = {sum_sources<RED, N>(lo), sum_sources<RED, N>(hi)};
    st_v8(p.out + (i << 4), o);
    return;
  }
  uint4 v[N];
#pragma unroll
  for (int r = 0; r < N; ++r) v[r] = ld_v4(p.srcs[r] + off);
  __syncwarp(__activemask());
  *reinterpret_cast<uint4*>(p.out + (i << 4)) = sum_sources<RED, N>(v);
}

using PeerReduceKernel = void (*)(PeerReduceParams);
template <int RED, int N>
PeerReduceKernel peerReduceKernelFrom(int nsrcs, bool wide) {
  if (nsrcs == N) return wide ? peer_reduce_kernel<RED, N, true> : peer_reduce_kernel<RED, N, false>;
  if constexpr (N < kMaxSources) return peerReduceKernelFrom<RED, N + 1>(nsrcs, wide);
  return nullptr;
}
PeerReduceKernel peerReduceKernel(int dtype, int nsrcs, bool wide) {
  return dtype == TCPXB_BF16 ? peerReduceKernelFrom<TCPXB_BF16, 1>(nsrcs, wide) : peerReduceKernelFrom<TCPXB_F32, 1>(nsrcs, wide);
}

// Checksum: per-block partial sums into scratch; the last block to arrive adds them.
// The sum is over 64-bit integers (wrapping), so its value depends neither on the order
// of the additions nor on scheduling.
constexpr int kCsumBlocks = 592;  // 4 per SM on a 148-SM part
constexpr int kCsumThreads = 256;
struct CsumScratch {
  uint32_t ticket;
  uint32_t pad;
  uint64_t partial[kCsumBlocks];
};
__global__ void __launch_bounds__(kCsumThreads)
checksum_kernel(const uint8_t* buf, uint64_t bytes, uint64_t* out, CsumScratch* scratch) {
  pdl_wait();
  pdl_launch_dependents();
  const uint64_t words = bytes >> 2;
  const uint32_t* w = reinterpret_cast<const uint32_t*>(buf);
  uint64_t sum = 0;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool vec_ok = (reinterpret_cast<uintptr_t>(buf) & 15) == 0;
  const uint64_t vecs = vec_ok ? (words >> 2) : 0;
  // Eight independent 16-byte streaming loads per thread and trip: at four CTAs of 256
  // threads per SM that is 128 KiB in flight per SM, several times what the HBM latency
  // asks for; one load per trip (16 KiB per SM) left the kernel latency-bound at a third
  // of the copy rate.  The data is read once: `ld.global.cs` keeps it from displacing L2 lines.
  const uint4* v16 = reinterpret_cast<const uint4*>(buf);
  uint64_t i = tid;
  constexpr int kUnroll = 8;
  for (; i + (kUnroll - 1) * stride < vecs; i += kUnroll * stride) {
    uint4 v[kUnroll];
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      // volatile: the eight loads are issued back to back, ahead of the first add
      asm volatile("ld.global.cs.v4.u32 {%0, %1, %2, %3}, [%4];"
                   : "=r"(v[u].x), "=r"(v[u].y), "=r"(v[u].z), "=r"(v[u].w)
                   : "l"(v16 + i + (uint64_t)u * stride));
    }
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) sum += (uint64_t)v[u].x + v[u].y + v[u].z + v[u].w;
  }
  for (; i < vecs; i += stride) {
    const uint4 v = __ldcs(v16 + i);
    sum += (uint64_t)v.x + v.y + v.z + v.w;
  }
  for (uint64_t i = (vecs << 2) + tid; i < words; i += stride) sum += w[i];
  if (tid == 0 && (bytes & 3)) {
    uint32_t last = 0;
    for (uint32_t b = 0; b < (bytes & 3); ++b) last |= (uint32_t)buf[(words << 2) + b] << (8 * b);
    sum += last;
  }
  __shared__ uint64_t red[kCsumThreads / 32];
  __shared__ uint32_t is_last;
  auto block_sum = [&](uint64_t v) -> uint64_t {  // valid in thread 0
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    __syncthreads();  // red[] may still be read from the previous use
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    uint64_t s = 0;
    if (threadIdx.x == 0)
      for (int i = 0; i < kCsumThreads / 32; ++i) s += red[i];
    return s;
  };
  const uint64_t mine = block_sum(sum);
  if (threadIdx.x == 0) {
    scratch->partial[blockIdx.x] = mine;
    __threadfence();
    is_last = atomicAdd(&scratch->ticket, 1u) == gridDim.x - 1 ? 1u : 0u;
  }
  __syncthreads();
  if (is_last) {
    // The last block to arrive adds the partial sums, all threads at once: one thread
    // walking 592 dependent-latency loads cost 20 us, twice the time of the 64 MiB pass.
    __threadfence();
    uint64_t part = 0;
    for (uint32_t b = threadIdx.x; b < gridDim.x; b += blockDim.x)
      part += *reinterpret_cast<volatile uint64_t*>(&scratch->partial[b]);
    const uint64_t total = block_sum(part);
    if (threadIdx.x == 0) {
      *out = total;
      scratch->ticket = 0;
    }
  }
}

// Scratch of the allocation-free checksum entry point: one CsumScratch per GPU,
// resident from library load to process exit.
static_assert(sizeof(CsumScratch) <= TCPXB_CHECKSUM_NOALLOC_SCRATCH_BYTES, "stated scratch size");
static __device__ __align__(256) unsigned char g_csum_static[TCPXB_CHECKSUM_NOALLOC_SCRATCH_BYTES];

// ------------------------------------------------------------------ host side
thread_local char g_err[256] = "";
int fail(int code, const char* fmt, const char* a = "") {
  snprintf(g_err, sizeof g_err, fmt, a);
  return code;
}
#define CUDA_TRY(expr)                                                  \
  do {                                                                  \
    cudaError_t e_ = (expr);                                            \
    if (e_ != cudaSuccess) return fail(TCPXB_K_CUDA, #expr ": %s", cudaGetErrorString(e_)); \
  } while (0)

constexpr int kMaxDevices = 64;
struct DeviceInfo {
  int sms = 0;
  bool attr_done[3][2][3] = {};
};
DeviceInfo g_dev[kMaxDevices];

// Applies the shared-memory attribute of one variant on `dev` (this also makes the
// runtime load the kernel) and records that it is done.
template <int RED, bool L2RED, int FAN>
int prepareVariant(int dev) {
  using C = Cfg<RED, L2RED, FAN>;
  DeviceInfo& di = g_dev[dev];
  if (di.attr_done[RED][L2RED][FAN]) return TCPXB_K_OK;
  CUDA_TRY(cudaFuncSetAttribute(unpack_kernel<RED, L2RED, FAN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                C::kSmemBytes));
  di.attr_done[RED][L2RED][FAN] = true;
  return TCPXB_K_OK;
}

int deviceInfo(int* dev_out) {
  int dev = 0;
  CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) return fail(TCPXB_K_INVALID, "device ordinal out of range");
  if (g_dev[dev].sms == 0) {
    int sms = 0;
    CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    g_dev[dev].sms = sms;
  }
  *dev_out = dev;
  return TCPXB_K_OK;
}

// Every launch may be scheduled while its predecessor in the stream still runs (programmatic dependent launch): the
// kernels wait for that predecessor on the device before they touch any memory, so results do not change and
// back-to-back launches save about 0.6 us each.  When a predecessor lets it in is that kernel's affair, since what
// waiting CTAs hold is not free for other streams:
//  - only after its own wait: at most one launch of a stream waits at a time, and a successor that reads something
//    before it waits still finds all that was written up to the kernel before this one;
//  - a kernel that waits for the host or another GPU (streamed records, flags), or that keeps to a part of the GPU, lets
//    its successor in when its work is done or not at all: that successor could take the SMs which the producer, or the
//    work beside a confined launch, needs.  At the end is early enough: 1 MiB requests on 16 CTAs, back to back, take
//    25.0 us with it as with a successor let in at once, 26.6 us if launched without.
template <typename Kernel, typename... Args>
int launchDependent(Kernel kernel, unsigned ctas, unsigned threads, size_t smem, cudaStream_t stream, const Args&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, args...));
  return TCPXB_K_OK;
}

template <int RED, bool L2RED, int FAN>
int launch(const UnpackParams& p, int max_ctas, cudaStream_t stream) {
  using C = Cfg<RED, L2RED, FAN>;
  int dev = 0;
  int rc = deviceInfo(&dev);
  if (rc) return rc;
  rc = prepareVariant<RED, L2RED, FAN>(dev);
  if (rc) return rc;
  if (p.count == 0) return TCPXB_K_OK;
  const int sms = g_dev[dev].sms;
  const bool whole_gpu = max_ctas <= 0 || max_ctas >= sms, asked = p.let_in != 0;
  if constexpr (FAN == FAN_NONE && !L2RED) {
    // Up to one record per ring warp the ring kernel is ahead (4 MiB in pages: 2.4 against 3.2 us, its bulk
    // copies need one instruction per page); beyond that its second, part-filled round costs more than it saves.
    // Ring -> register kernel, buffers out of HBM: 1777 whole pages copied 4.8 -> 4.5 us, summed 6.6 -> 5.4; 3000 of 1448
    // bytes copied 4.1 -> 3.4, summed 5.1 -> 4.3; 16384 pages 24.6 -> 23.3 and 34.0 -> 31.9.  Where the ring stays ahead: whole
    // pages copied within L2 (3000: 3.7 -> 4.4), 5000 to 10000 copies of 1448 to 3000 bytes (up to 10 %).  A pool in pinned
    // host memory, 8 MiB: pages 169 -> 167 us, sums of 1448-byte fragments 178 -> 184, copies of them 176 -> 186 (their edges are
    // read twice over PCIe); packing from HBM into host memory 172 -> 170.  Telling host memory apart would cost every
    // launch a driver query of half a microsecond.
    // A launch confined to a few CTAs, streamed or asked to publish its completion stays with the ring.
    if (whole_gpu && p.ready == nullptr && p.flag_value == 0 && p.done_flag == nullptr && p.count > (uint32_t)(sms * kWarps))
      return launchDependent(unpack_wide_kernel<RED>, (p.count + kWideWarps - 1) / kWideWarps, kWideThreads, 0, stream, p);
  }
  // As many SMs as there are records before any SM gets a second one: a record is one warp's work, and 12 of
  // them on one SM share its bulk-copy engine (256 records: 3.1 us on 22 SMs, 1.9 us on 148).
  const int cap = whole_gpu ? sms : max_ctas;
  const int ctas = p.count < (uint32_t)cap ? (int)p.count : cap;
  UnpackParams q = p;
  q.let_in = p.ready == nullptr && (whole_gpu || asked) ? 1 : 0;
  return launchDependent(unpack_kernel<RED, L2RED, FAN>, (unsigned)ctas, kThreads, C::kSmemBytes, stream, q);
}

// Device address of the allocation-free checksum's scratch on `dev` (the current
// device).  In host code `g_csum_static` is only a handle for the runtime, not an
// address a kernel could use, so the address is resolved once per device and kept.
int csumStaticScratch(int dev, void** out) {
  static std::mutex mu;
  static void* scratch_of_device[kMaxDevices] = {};
  std::lock_guard<std::mutex> l(mu);
  if (scratch_of_device[dev] == nullptr) {
    void* p = nullptr;
    CUDA_TRY(cudaGetSymbolAddress(&p, g_csum_static));
    scratch_of_device[dev] = p;
  }
  *out = scratch_of_device[dev];
  return TCPXB_K_OK;
}

template <int FAN>
int prepareFan(int dev) {
  int rc = prepareVariant<TCPXB_U8, false, FAN>(dev);
  if (!rc) rc = prepareVariant<TCPXB_BF16, false, FAN>(dev);
  if (!rc) rc = prepareVariant<TCPXB_BF16, true, FAN>(dev);
  if (!rc) rc = prepareVariant<TCPXB_F32, false, FAN>(dev);
  if (!rc) rc = prepareVariant<TCPXB_F32, true, FAN>(dev);
  return rc;
}

template <int FAN>
int dispatch(const UnpackParams& p, int dtype, int impl, int max_ctas, cudaStream_t s) {
  const bool l2 = (impl == TCPXB_REDUCE_L2);
  switch (dtype) {
    case TCPXB_U8: return launch<TCPXB_U8, false, FAN>(p, max_ctas, s);
    case TCPXB_BF16:
      return l2 ? launch<TCPXB_BF16, true, FAN>(p, max_ctas, s)
                : launch<TCPXB_BF16, false, FAN>(p, max_ctas, s);
    case TCPXB_F32:
      return l2 ? launch<TCPXB_F32, true, FAN>(p, max_ctas, s)
                : launch<TCPXB_F32, false, FAN>(p, max_ctas, s);
    default: return fail(TCPXB_K_INVALID, "unknown dtype");
  }
}

int fill(UnpackParams& p, const void* pool, uint64_t pool_bytes, const void* acc, void* dst,
         void* mc_dst, uint64_t dst_bytes, void* const* peers, int npeers,
         const tcpxbLoadMeta* descs, uint32_t count, uint32_t* status,
         const tcpxbUnpackOpts* opts) {
  memset(&p, 0, sizeof p);
  if (count != 0 && (pool == nullptr || dst == nullptr || descs == nullptr))
    return fail(TCPXB_K_INVALID, "null pool, dst or descriptor pointer");
  if (npeers < 0 || npeers > TCPXB_MAX_PEERS) return fail(TCPXB_K_INVALID, "npeers out of range");
  if (npeers > 0 && peers == nullptr) return fail(TCPXB_K_INVALID, "null peer table");
  if (reinterpret_cast<uintptr_t>(descs) & 15)
    return fail(TCPXB_K_INVALID, "descriptor array must be 16-byte aligned");
  p.pool = static_cast<const uint8_t*>(pool);
  p.pool_bytes = pool_bytes;
  p.dst = static_cast<uint8_t*>(dst);
  p.dst_bytes = dst_bytes;
  p.acc = static_cast<const uint8_t*>(acc ? acc : dst);
  p.mc_dst = static_cast<uint8_t*>(mc_dst);
  p.descs = descs;
  p.count = count;
  p.npeers = npeers;
  const uintptr_t base_mis = reinterpret_cast<uintptr_t>(dst) & 15;
  for (int i = 0; i < npeers; ++i) {
    if (peers[i] == nullptr) return fail(TCPXB_K_INVALID, "null peer pointer");
    // The fast path decides alignment from the local address; peers must agree.
    if ((reinterpret_cast<uintptr_t>(peers[i]) & 15) != base_mis)
      return fail(TCPXB_K_INVALID, "peer buffers must share the local buffer's 16-byte phase");
    p.peers[i] = static_cast<uint8_t*>(peers[i]);
  }
  if (mc_dst != nullptr && (reinterpret_cast<uintptr_t>(mc_dst) & 15) != base_mis)
    return fail(TCPXB_K_INVALID, "multicast mapping must share the local buffer's 16-byte phase");
  p.status = status;
  if (opts != nullptr) {
    p.ready = opts->ready_count;
    p.let_in = opts->early_launch != 0;
    p.wait_ns = opts->wait_ns;
    p.flag_value = opts->flag_value;
    p.ticket = opts->ticket;
    for (int i = 0; i < TCPXB_MAX_PEERS; ++i) p.peer_flags[i] = opts->peer_flags[i];
  }
  return TCPXB_K_OK;
}

}  // namespace

extern "C" {

const char* tcpxb_kernel_last_error(void) { return g_err; }

int tcpxb_kernels_preload(void) {
  static std::mutex mu;
  static bool done[kMaxDevices] = {};
  std::lock_guard<std::mutex> l(mu);
  int dev = 0;
  int rc = deviceInfo(&dev);
  if (rc) return rc;
  if (done[dev]) return TCPXB_K_OK;
  rc = prepareFan<FAN_NONE>(dev);
  if (!rc) rc = prepareFan<FAN_PEER>(dev);
  if (!rc) rc = prepareFan<FAN_NVLS>(dev);
  if (rc) return rc;
  // Setting an attribute does not make the runtime load a kernel; an empty launch
  // does.  Every kernel runs once with nothing to do, on a private stream.
  cudaStream_t s = nullptr;
  CUDA_TRY(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
  UnpackParams p;
  memset(&p, 0, sizeof p);
#define TCPXB_DRY(RED, L2, FAN) \
  unpack_kernel<RED, L2, FAN><<<1, kThreads, Cfg<RED, L2, FAN>::kSmemBytes, s>>>(p)
#define TCPXB_DRY_FAN(FAN)                                                      \
  TCPXB_DRY(TCPXB_U8, false, FAN); TCPXB_DRY(TCPXB_BF16, false, FAN); TCPXB_DRY(TCPXB_BF16, true, FAN); \
  TCPXB_DRY(TCPXB_F32, false, FAN); TCPXB_DRY(TCPXB_F32, true, FAN)
  TCPXB_DRY_FAN(FAN_NONE);
  TCPXB_DRY_FAN(FAN_PEER);
  TCPXB_DRY_FAN(FAN_NVLS);
#undef TCPXB_DRY_FAN
  unpack_wide_kernel<TCPXB_U8><<<1, kWideThreads, 0, s>>>(p);
  unpack_wide_kernel<TCPXB_BF16><<<1, kWideThreads, 0, s>>>(p);
  unpack_wide_kernel<TCPXB_F32><<<1, kWideThreads, 0, s>>>(p);
  FewParams few;
  memset(&few, 0, sizeof few);
  unpack_few_kernel<TCPXB_U8><<<1, kWideThreads, 0, s>>>(few);
  unpack_few_kernel<TCPXB_BF16><<<1, kWideThreads, 0, s>>>(few);
  unpack_few_kernel<TCPXB_F32><<<1, kWideThreads, 0, s>>>(few);
#undef TCPXB_DRY
  wait_flags_kernel<<<1, 32, 0, s>>>(nullptr, 0, 0, 1, nullptr);
  SignalParams sp;
  memset(&sp, 0, sizeof sp);
  signal_flags_kernel<<<1, 32, 0, s>>>(sp);
  PeerReduceParams pp;
  memset(&pp, 0, sizeof pp);
  for (int n = 1; n <= kMaxSources; ++n)
    for (const int dtype : {TCPXB_BF16, TCPXB_F32})
      for (const bool wide : {false, true}) peerReduceKernel(dtype, n, wide)<<<1, kPeerThreads, 0, s>>>(pp);
  // The checksum kernel and the address of the allocation-free entry point's scratch:
  // one launch over zero bytes, its result written into the scratch itself, so that
  // the first real tcpxb_checksum_noalloc on this device only clears and launches.
  void* cs = nullptr;
  rc = csumStaticScratch(dev, &cs);
  if (rc) return rc;
  CUDA_TRY(cudaMemsetAsync(cs, 0, 8, s));
  checksum_kernel<<<1, kCsumThreads, 0, s>>>(nullptr, 0, &static_cast<CsumScratch*>(cs)->partial[kCsumBlocks - 1],
                                             static_cast<CsumScratch*>(cs));
  stage_out_kernel<<<1, kStageThreads, 0, s>>>(nullptr, nullptr, 0, &static_cast<CsumScratch*>(cs)->pad, 0);
  CUDA_TRY(cudaGetLastError());
  CUDA_TRY(cudaStreamSynchronize(s));
  CUDA_TRY(cudaStreamDestroy(s));
  done[dev] = true;
  return TCPXB_K_OK;
}

int tcpxb_unpack_copy(const void* pool, uint64_t pool_bytes, void* dst, uint64_t dst_bytes,
                      const tcpxbLoadMeta* descs, uint32_t count, uint32_t* status,
                      const tcpxbUnpackOpts* opts, void* stream) {
  UnpackParams p;
  int rc = fill(p, pool, pool_bytes, nullptr, dst, nullptr, dst_bytes, nullptr, 0, descs, count,
                status, opts);
  if (rc) return rc;
  return dispatch<FAN_NONE>(p, TCPXB_U8, 0, opts ? opts->max_ctas : 0,
                            static_cast<cudaStream_t>(stream));
}

int tcpxb_unpack_reduce(const void* pool, uint64_t pool_bytes, const void* acc, void* dst,
                        uint64_t dst_bytes, const tcpxbLoadMeta* descs, uint32_t count, int dtype,
                        int impl, uint32_t* status, const tcpxbUnpackOpts* opts, void* stream) {
  if (dtype != TCPXB_BF16 && dtype != TCPXB_F32)
    return fail(TCPXB_K_INVALID, "reduce needs dtype bf16 or f32");
  if (impl == TCPXB_REDUCE_L2 && acc != nullptr && acc != dst)
    return fail(TCPXB_K_INVALID, "the L2 reduce form is in place: acc must be NULL or dst");
  UnpackParams p;
  int rc = fill(p, pool, pool_bytes, acc, dst, nullptr, dst_bytes, nullptr, 0, descs, count, status,
                opts);
  if (rc) return rc;
  return dispatch<FAN_NONE>(p, dtype, impl, opts ? opts->max_ctas : 0,
                            static_cast<cudaStream_t>(stream));
}

int tcpxb_unpack_fanout(const void* pool, uint64_t pool_bytes, void* dst, uint64_t dst_bytes,
                        void* const* peers, int npeers, const tcpxbLoadMeta* descs, uint32_t count,
                        uint32_t* status, const tcpxbUnpackOpts* opts, void* stream) {
  UnpackParams p;
  int rc = fill(p, pool, pool_bytes, nullptr, dst, nullptr, dst_bytes, peers, npeers, descs, count,
                status, opts);
  if (rc) return rc;
  return dispatch<FAN_PEER>(p, TCPXB_U8, 0, opts ? opts->max_ctas : 0,
                            static_cast<cudaStream_t>(stream));
}

int tcpxb_unpack_reduce_fanout(const void* pool, uint64_t pool_bytes, const void* acc, void* dst,
                               uint64_t dst_bytes, void* const* peers, int npeers,
                               const tcpxbLoadMeta* descs, uint32_t count, int dtype, int impl,
                               uint32_t* status, const tcpxbUnpackOpts* opts, void* stream) {
  if (dtype != TCPXB_BF16 && dtype != TCPXB_F32)
    return fail(TCPXB_K_INVALID, "reduce needs dtype bf16 or f32");
  if (impl == TCPXB_REDUCE_L2 && acc != nullptr && acc != dst)
    return fail(TCPXB_K_INVALID, "the L2 reduce form is in place: acc must be NULL or dst");
  UnpackParams p;
  int rc = fill(p, pool, pool_bytes, acc, dst, nullptr, dst_bytes, peers, npeers, descs, count,
                status, opts);
  if (rc) return rc;
  return dispatch<FAN_PEER>(p, dtype, impl, opts ? opts->max_ctas : 0,
                            static_cast<cudaStream_t>(stream));
}

int tcpxb_unpack_fanout_nvls(const void* pool, uint64_t pool_bytes, void* dst, void* mc_dst,
                             uint64_t dst_bytes, void* const* peers, int npeers,
                             const tcpxbLoadMeta* descs, uint32_t count, uint32_t* status,
                             const tcpxbUnpackOpts* opts, void* stream) {
  if (mc_dst == nullptr) return fail(TCPXB_K_INVALID, "null multicast mapping");
  UnpackParams p;
  int rc = fill(p, pool, pool_bytes, nullptr, dst, mc_dst, dst_bytes, peers, npeers, descs, count,
                status, opts);
  if (rc) return rc;
  return dispatch<FAN_NVLS>(p, TCPXB_U8, 0, opts ? opts->max_ctas : 0,
                            static_cast<cudaStream_t>(stream));
}

int tcpxb_unpack_reduce_fanout_nvls(const void* pool, uint64_t pool_bytes, const void* acc,
                                    void* dst, void* mc_dst, uint64_t dst_bytes,
                                    void* const* peers, int npeers, const tcpxbLoadMeta* descs,
                                    uint32_t count, int dtype, uint32_t* status,
                                    const tcpxbUnpackOpts* opts, void* stream) {
  if (mc_dst == nullptr) return fail(TCPXB_K_INVALID, "null multicast mapping");
  if (dtype != TCPXB_BF16 && dtype != TCPXB_F32)
    return fail(TCPXB_K_INVALID, "reduce needs dtype bf16 or f32");
  UnpackParams p;
  int rc = fill(p, pool, pool_bytes, acc, dst, mc_dst, dst_bytes, peers, npeers, descs, count,
                status, opts);
  if (rc) return rc;
  // acc == NULL selects the reduce-into-all form (multimem.red into every accumulator).
  return dispatch<FAN_NVLS>(p, dtype, acc == nullptr ? TCPXB_REDUCE_L2 : TCPXB_REDUCE_SM,
                            opts ? opts->max_ctas : 0, static_cast<cudaStream_t>(stream));
}

int tcpxb_unpack_request(const void* pool, uint64_t pool_bytes, const void* acc, void* dst, void* mc_dst, uint64_t dst_bytes,
                         void* const* peers, int npeers, const tcpxbLoadMeta* descs, const tcpxbLoadMeta* descs_host, uint32_t count,
                         int dtype, int impl, uint32_t* status, const tcpxbUnpackOpts* opts, uint32_t* done_flag, uint32_t done_value,
                         void* stream) {
  if (done_flag == nullptr || opts == nullptr || opts->ticket == nullptr)
    return fail(TCPXB_K_INVALID, "a completion word and its ticket are needed");
  if (acc != nullptr && dtype != TCPXB_BF16 && dtype != TCPXB_F32)
    return fail(TCPXB_K_INVALID, "reduce needs dtype bf16 or f32");
  if (impl == TCPXB_REDUCE_L2 && acc != nullptr && (acc != dst || mc_dst != nullptr))
    return fail(TCPXB_K_INVALID, "the L2 reduce form is in place: acc must be dst");
  UnpackParams p;
  int rc = fill(p, pool, pool_bytes, acc, dst, mc_dst, dst_bytes, peers, npeers, descs, count, status, opts);
  if (rc) return rc;
  p.done_flag = done_flag;
  p.done_value = done_value;
  const int dt = acc != nullptr ? dtype : TCPXB_U8;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (mc_dst != nullptr) return dispatch<FAN_NVLS>(p, dt, TCPXB_REDUCE_SM, opts->max_ctas, s);
  if (npeers > 0) return dispatch<FAN_PEER>(p, dt, impl, opts->max_ctas, s);
  // a warp per record in one CTA: beyond its eight warps the ring's bulk copies are as fast
  if (descs_host != nullptr && count != 0 && count <= (uint32_t)kFewRecords && impl == TCPXB_REDUCE_SM && p.ready == nullptr && p.flag_value == 0) {
    FewParams few;
    few.p = p;
    memset(few.recs, 0, sizeof few.recs);
    memcpy(few.recs, descs_host, count * sizeof(tcpxbLoadMeta));
    return launchDependent(dt == TCPXB_U8 ? unpack_few_kernel<TCPXB_U8> : dt == TCPXB_BF16 ? unpack_few_kernel<TCPXB_BF16> : unpack_few_kernel<TCPXB_F32>,
                           1, count * 32, 0, s, few);
  }
  return dispatch<FAN_NONE>(p, dt, impl, opts->max_ctas, s);
}

int tcpxb_wait_flags(const uint32_t* flags, int n, uint32_t value, uint64_t wait_ns,
                     uint32_t* status, void* stream) {
  if (flags == nullptr || n < 0 || n > 32) return fail(TCPXB_K_INVALID, "bad flag table");
  if (n == 0) return TCPXB_K_OK;
  return launchDependent(wait_flags_kernel, 1, 32, 0, static_cast<cudaStream_t>(stream), flags, n, value,
                         wait_ns ? wait_ns : kDefaultWaitNs, status);
}

int tcpxb_signal_flags(uint32_t* const* peer_flags, int n, uint32_t value, void* stream) {
  if (n < 0 || n > TCPXB_MAX_PEERS + 1 || (n > 0 && peer_flags == nullptr))
    return fail(TCPXB_K_INVALID, "bad flag table");
  if (n == 0) return TCPXB_K_OK;
  SignalParams p;
  memset(&p, 0, sizeof p);
  for (int i = 0; i < n; ++i) p.flags[i] = peer_flags[i];
  p.n = n;
  p.value = value;
  return launchDependent(signal_flags_kernel, 1, 32, 0, static_cast<cudaStream_t>(stream), p);
}

int tcpxb_stage_out(const void* src, void* host_dst, uint64_t bytes, uint32_t* flag, uint32_t value, void* stream) {
  if (flag == nullptr || (bytes != 0 && (src == nullptr || host_dst == nullptr)))
    return fail(TCPXB_K_INVALID, "null source, destination or flag");
  const unsigned threads = bytes <= kStageThreads * 16 / 4 ? kStageThreads / 4 : kStageThreads;
  return launchDependent(stage_out_kernel, 1, threads, 0, static_cast<cudaStream_t>(stream), static_cast<const uint8_t*>(src),
                         static_cast<uint8_t*>(host_dst), bytes, flag, value);
}

int tcpxb_peer_reduce(void* out, void* const* srcs, int nsrcs, uint64_t shard_off, uint64_t bytes,
                      int dtype, void* stream) {
  if (out == nullptr || srcs == nullptr || nsrcs < 1 || nsrcs > TCPXB_MAX_PEERS + 1)
    return fail(TCPXB_K_INVALID, "bad source table");
  if (dtype != TCPXB_BF16 && dtype != TCPXB_F32)
    return fail(TCPXB_K_INVALID, "reduce needs dtype bf16 or f32");
  if ((bytes & 15) || (shard_off & 15) || (reinterpret_cast<uintptr_t>(out) & 15))
    return fail(TCPXB_K_INVALID, "peer_reduce works on 16-byte aligned spans");
  PeerReduceParams p;
  memset(&p, 0, sizeof p);
  for (int i = 0; i < nsrcs; ++i) {
    if (srcs[i] == nullptr || (reinterpret_cast<uintptr_t>(srcs[i]) & 15))
      return fail(TCPXB_K_INVALID, "null or misaligned source");
    p.srcs[i] = static_cast<const uint8_t*>(srcs[i]);
  }
  p.out = static_cast<uint8_t*>(out);
  p.shard_off = shard_off;
  p.vecs = bytes >> 4;
  if (p.vecs == 0) return TCPXB_K_OK;
  uintptr_t at = reinterpret_cast<uintptr_t>(out);
  for (int i = 0; i < nsrcs; ++i) at |= reinterpret_cast<uintptr_t>(p.srcs[i]) + shard_off;
  const bool wide = (at & 31) == 0;
  const uint64_t ctas = ((wide ? (p.vecs + 1) / 2 : p.vecs) + kPeerThreads - 1) / kPeerThreads;
  if (ctas > 0x7fffffffull) return fail(TCPXB_K_INVALID, "span beyond the largest grid");
  return launchDependent(peerReduceKernel(dtype, nsrcs, wide), (unsigned)ctas, kPeerThreads, 0, static_cast<cudaStream_t>(stream), p);
}

size_t tcpxb_checksum_scratch_bytes(void) { return sizeof(CsumScratch); }

int tcpxb_checksum(const void* buf, uint64_t bytes, uint64_t* out, void* partials, void* stream) {
  if (out == nullptr || partials == nullptr || (buf == nullptr && bytes != 0))
    return fail(TCPXB_K_INVALID, "null buffer, output or scratch");
  if (reinterpret_cast<uintptr_t>(buf) & 3)
    return fail(TCPXB_K_INVALID, "checksum buffer must be 4-byte aligned");
  uint64_t want = (bytes / 16 + kCsumThreads - 1) / kCsumThreads;
  int blocks = (int)(want < 1 ? 1 : (want > (uint64_t)kCsumBlocks ? kCsumBlocks : want));
  return launchDependent(checksum_kernel, (unsigned)blocks, kCsumThreads, 0, static_cast<cudaStream_t>(stream),
                         static_cast<const uint8_t*>(buf), bytes, out, static_cast<CsumScratch*>(partials));
}

int tcpxb_checksum_noalloc(const void* buf, uint64_t bytes, uint64_t* out, void* stream) {
  if (out == nullptr || (buf == nullptr && bytes != 0))
    return fail(TCPXB_K_INVALID, "null buffer or output");
  if (reinterpret_cast<uintptr_t>(buf) & 3)
    return fail(TCPXB_K_INVALID, "checksum buffer must be 4-byte aligned");
  if (bytes > TCPXB_CHECKSUM_NOALLOC_MAX_BYTES)
    return fail(TCPXB_K_TOO_LARGE,
                "tcpxb_checksum_noalloc handles at most 16 GiB per call; split the buffer or use tcpxb_checksum");
  int dev = 0;
  CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) return fail(TCPXB_K_INVALID, "device ordinal out of range");
  void* scratch = nullptr;
  const int rc = csumStaticScratch(dev, &scratch);  // a table look-up after tcpxb_kernels_preload or a first call
  if (rc) return rc;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // the completion counter must start at zero even if an earlier launch was cut short
  CUDA_TRY(cudaMemsetAsync(scratch, 0, 8, s));
  uint64_t want = (bytes / 16 + kCsumThreads - 1) / kCsumThreads;
  int blocks = (int)(want < 1 ? 1 : (want > (uint64_t)kCsumBlocks ? kCsumBlocks : want));
  return launchDependent(checksum_kernel, (unsigned)blocks, kCsumThreads, 0, s, static_cast<const uint8_t*>(buf), bytes, out,
                         static_cast<CsumScratch*>(scratch));
}

}  // extern "C"
