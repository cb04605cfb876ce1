// nvshm_core.cuh -- device-side building blocks of the virtual-PE library.
//
// Everything on the hot path is here as inline functions taking the arena
// configuration explicitly, so the library's own kernels get it through the
// kernel parameter bank and inline every call, while the public extern "C"
// device API (device_api.cu) forwards to the same code with the __constant__
// copy.
//
// Memory layout (one B200):
//   arena = npes slices of `stride` bytes (stride a power of two), slice p at
//   arena + p*stride.  A symmetric address names an object by its offset in
//   its slice, so translating it to PE `pe` needs no table:
//       arena + pe*stride + ((addr - arena) & (stride - 1)).
//   (The prototype looked the peer base up in a __constant__ table of IPC
//   mappings, nvshmem_device.cu:446-447, which serialises lanes that name
//   different PEs; the shift/mask form is uniform-cost.)
#pragma once

#include <stdint.h>
#include <cuda_runtime.h>
#include "nvshmemx.h"

namespace nvshm {

// Arena configuration visible to device code.  One copy lives in __constant__
// memory for the public API; library kernels receive it by value.
struct Cfg {
  char *arena;
  unsigned long long arena_bytes;  // npes << log2_stride
  unsigned long long mask;         // stride - 1
  unsigned long long slice_bytes;  // mapped (usable) bytes at the start of each slice
  int log2_stride;
  int npes;
  int *status;                     // [0] code, [1] pe, [2..3] 64-bit detail
  unsigned long long *coll_bar;    // collective-launch ticket counter
  unsigned long long *pe_bar;      // per-PE ticket counters [npes]
  long long wait_timeout_ns;
  nvshmemx_trace_record *trace;    // npes * trace_cap records, or nullptr
  unsigned long long *trace_head;  // per-PE record counters
  unsigned int trace_cap;          // power of two
  int proc_pe;                     // process-per-PE mode: this process's PE; -1
                                   // when all PEs share one collective launch
};

// ---------------------------------------------------------------- PTX helpers
__device__ __forceinline__ unsigned long long gtimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ int ld_acquire(const int *p) {
  int v;
  asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned long long ld_acquire_u64(const unsigned long long *p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned int ld_relaxed_b32(const void *p) {
  unsigned int v;
  asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned long long ld_relaxed_b64(const void *p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed_b32(void *p, unsigned int v) {
  asm volatile("st.relaxed.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void st_relaxed_b64(void *p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ void st_release_b32(void *p, unsigned int v) {
  asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned long long atom_add_acq_rel_u64(unsigned long long *p,
                                                                   unsigned long long v) {
  unsigned long long old;
  asm volatile("atom.add.acq_rel.gpu.global.u64 %0, [%1], %2;"
               : "=l"(old) : "l"(p), "l"(v) : "memory");
  return old;
}
__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

__device__ __forceinline__ unsigned smem_u32(const void *p) {
  return (unsigned)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ unsigned lane_number() {
  unsigned l;
  asm("mov.u32 %0, %%laneid;" : "=r"(l));
  return l;
}

// ------------------------------------------------------------- PE / addresses
// The calling PE: blockIdx.z of a collective launch, or the process's PE when
// every PE is a process of its own.
__device__ __forceinline__ int my_pe(const Cfg &c) { return c.proc_pe >= 0 ? c.proc_pe : (int)blockIdx.z; }

__device__ __forceinline__ bool in_arena(const Cfg &c, const void *p) {
  return (unsigned long long)((const char *)p - c.arena) < c.arena_bytes;
}

__device__ __forceinline__ unsigned long long slice_off(const Cfg &c, const void *sym) {
  return (unsigned long long)((const char *)sym - c.arena) & c.mask;
}

__device__ __forceinline__ char *xlate(const Cfg &c, const void *sym, int pe) {
  return c.arena + ((unsigned long long)(unsigned)pe << c.log2_stride) + slice_off(c, sym);
}

// Records the first device-side error; later ones are dropped.
__device__ __forceinline__ void record_error(const Cfg &c, int code, long long detail) {
  if (atomicCAS(c.status, 0, code) == 0) {
    c.status[1] = my_pe(c);
    *(volatile long long *)(c.status + 2) = detail;
  }
}

// A symmetric range [sym, sym+bytes) on `pe` is valid when sym lies in the
// arena, pe is a PE and the range stays inside the mapped part of one slice.
__device__ __forceinline__ bool check_remote(const Cfg &c, const void *sym, unsigned long long bytes,
                                             int pe) {
  bool ok = in_arena(c, sym) && (unsigned)pe < (unsigned)c.npes &&
            slice_off(c, sym) + bytes <= c.slice_bytes;
  if (!ok) record_error(c, NVSHMEMX_ERR_BOUNDS, (long long)((const char *)sym - c.arena));
  return ok;
}

// A local operand may point anywhere in device memory; if it points into the
// arena's address range it must stay inside the mapped part of its slice
// (the rest of each slice's stride is reserved address space, not memory).
__device__ __forceinline__ bool check_local(const Cfg &c, const void *p, unsigned long long bytes) {
  if (!in_arena(c, p)) return true;
  bool ok = slice_off(c, p) + bytes <= c.slice_bytes;
  if (!ok) record_error(c, NVSHMEMX_ERR_BOUNDS, (long long)((const char *)p - c.arena));
  return ok;
}

// ------------------------------------------------------------------- tracing
__device__ __forceinline__ void trace_rec(const Cfg &c, int op, const void *local,
                                          const void *remote, unsigned long long bytes, int peer,
                                          unsigned long long t0, unsigned long long t1) {
  int pe = my_pe(c);
  if ((unsigned)pe >= (unsigned)c.npes) pe = 0;
  unsigned long long idx = atomicAdd(&c.trace_head[pe], 1ull);
  nvshmemx_trace_record *r =
      c.trace + (size_t)pe * c.trace_cap + (size_t)(idx & (unsigned long long)(c.trace_cap - 1));
  r->t_ns = (long long)t0;
  r->spin_ns = (long long)(t1 - t0);
  r->local_addr = (unsigned long long)local;
  r->remote_addr = (unsigned long long)remote;
  r->bytes = (unsigned)bytes;
  r->op = (unsigned short)op;
  r->pe = (unsigned short)pe;
  r->peer = (unsigned short)peer;
  r->tid = (unsigned short)(threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z));
  r->block = blockIdx.x + gridDim.x * blockIdx.y;
}

// --------------------------------------------------------------- copy engines
template <int VB> struct VecT;
template <> struct VecT<16> { typedef uint4 T; };
template <> struct VecT<8> { typedef uint2 T; };
template <> struct VecT<4> { typedef unsigned int T; };
template <> struct VecT<1> { typedef unsigned char T; };

// Asks the TMA unit to stage [p, p + bytes) in L2 (16-byte aligned address,
// size a multiple of 16; nothing to wait for -- later loads just hit L2).
// Only for addresses in global memory: callers ask __isGlobal of a source that
// an application named.
__device__ __forceinline__ void l2_prefetch_bulk(uintptr_t p, unsigned bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes));
}

// 16 bytes whose address is only LB-byte aligned.  LB 4 stands for addresses
// that are 4 modulo 8 (one that is 0 modulo 8 takes LB 8), so the middle two
// words are one 8-byte load; LB 1 for addresses that are not 0 modulo 4.
template <int LB>
__device__ __forceinline__ uint4 load16(const char *p) {
  if (LB == 16) return *reinterpret_cast<const uint4 *>(p);
  uint4 v;
  if (LB == 1) {
    // the five words that hold the 16 bytes, shifted; each of them holds at
    // least one of the bytes, so none lies outside the source's words
    const unsigned *q = reinterpret_cast<const unsigned *>((uintptr_t)p & ~(uintptr_t)3);
    const unsigned sh = ((unsigned)(uintptr_t)p & 3u) * 8u;
    const unsigned w0 = q[0], w1 = q[1], w2 = q[2], w3 = q[3], w4 = q[4];
    v.x = __funnelshift_r(w0, w1, sh), v.y = __funnelshift_r(w1, w2, sh);
    v.z = __funnelshift_r(w2, w3, sh), v.w = __funnelshift_r(w3, w4, sh);
  } else if (LB == 8) {
    const uint2 a = *reinterpret_cast<const uint2 *>(p), b = *reinterpret_cast<const uint2 *>(p + 8);
    v.x = a.x, v.y = a.y, v.z = b.x, v.w = b.y;
  } else {
    v.x = *reinterpret_cast<const unsigned *>(p);
    const uint2 m = *reinterpret_cast<const uint2 *>(p + 4);
    v.y = m.x, v.z = m.y;
    v.w = *reinterpret_cast<const unsigned *>(p + 12);
  }
  return v;
}

// The first `have` of U vectors 512 bytes apart; the loads' width follows the
// relative alignment `mis` (the same for the whole warp), in one set of
// registers for the three widths.
template <int U>
__device__ __forceinline__ void load_row(uint4 *v, const char *s, unsigned mis, unsigned have) {
  if ((mis & 15) == 0) {
#pragma unroll
    for (unsigned u = 0; u < U; ++u)
      if (u < have) v[u] = load16<16>(s + u * 512);
  } else if ((mis & 7) == 0) {
#pragma unroll
    for (unsigned u = 0; u < U; ++u)
      if (u < have) v[u] = load16<8>(s + u * 512);
  } else if ((mis & 3) == 0) {
#pragma unroll
    for (unsigned u = 0; u < U; ++u)
      if (u < have) v[u] = load16<4>(s + u * 512);
  } else if (U <= 4) {
#pragma unroll
    for (unsigned u = 0; u < U; ++u)
      if (u < have) v[u] = load16<1>(s + u * 512);
  }
}

// One VB-byte vector of a source that is LB-byte aligned (LB < VB: VB is 16).
template <int VB, int LB>
__device__ __forceinline__ typename VecT<VB>::T load_vec(const typename VecT<VB>::T *p) {
  return *p;
}
template <>
__device__ __forceinline__ uint4 load_vec<16, 8>(const uint4 *p) {
  return load16<8>(reinterpret_cast<const char *>(p));
}
template <>
__device__ __forceinline__ uint4 load_vec<16, 4>(const uint4 *p) {
  return load16<4>(reinterpret_cast<const char *>(p));
}

// Copies `bytes` with `nthr` cooperating threads (this one is `r`), VB-byte
// stores for the body aligned to the destination and U accesses in flight per
// thread.  LB is the alignment of the source there: with LB < VB a vector is
// put together from two or three narrower loads, so a copy between arrays
// that lie 4, 8 or 12 bytes apart modulo 16 still stores whole vectors and
// keeps 16 bytes in flight per access (before, it went by 4- or 8-byte
// accesses both ways: 1500 one-CTA puts of 140 KB at 4-byte offsets took
// 148 us, now 95 us; the narrower loads of one vector share L1 sectors, so
// L2 and DRAM see each byte once).
//
// PFI > 0: a copy by one thread or one warp is bound by the latency of its
// loads (U accesses per thread per round).  Its thread 0 keeps an L2
// prefetch of the source PFI rounds in front of the loads (never past the
// source range), so the loads hit L2 instead of DRAM.  Copies shorter than
// twice that distance skip it.
template <int VB, int U, unsigned PFI = 0, int LB = VB>
__device__ __forceinline__ void copy_body(char *__restrict__ dst, const char *__restrict__ src,
                                          unsigned long long bytes, unsigned r, unsigned nthr) {
  typedef typename VecT<VB>::T V;
  unsigned long long head = (VB - ((uintptr_t)dst & (VB - 1))) & (VB - 1);
  if (head > bytes) head = bytes;
  for (unsigned long long i = r; i < head; i += nthr) dst[i] = src[i];
  const unsigned long long nv = (bytes - head) / VB;
  const V *s = reinterpret_cast<const V *>(src + head);
  V *d = reinterpret_cast<V *>(dst + head);
  unsigned long long i = r;
  const unsigned long long step = (unsigned long long)nthr * U;
  const unsigned long long dist = (unsigned long long)PFI * step * VB;  // bytes ahead
  const bool pf_on = PFI > 0 && r == 0 && nthr <= 32 && bytes >= 2 * dist && __isGlobal(src);
  const uintptr_t pf_end = ((uintptr_t)src + bytes) & ~(uintptr_t)15;
  uintptr_t pf = ((uintptr_t)src + 15) & ~(uintptr_t)15;  // next source byte to stage
  if (nv >= (unsigned long long)(U - 1) * nthr) {
#pragma unroll 1
    for (; i + (unsigned long long)(U - 1) * nthr < nv; i += step) {
      V v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) v[u] = load_vec<VB, LB>(s + i + (unsigned long long)u * nthr);
      // between this iteration's loads and its stores: the stores of one
      // iteration and the loads of the next stay free to interleave
      // (measured: placed before the loads, the prefetch cost 15-23% on
      // copies already in L2)
      if (pf_on) {
        uintptr_t want = ((uintptr_t)(s + i) + dist) & ~(uintptr_t)15;
        if (want > pf_end) want = pf_end;
        if (want >= pf + 4096 || (want == pf_end && want > pf)) {
          const unsigned n = (unsigned)(want - pf < 65536 ? want - pf : 65536);
          l2_prefetch_bulk(pf, n);
          pf += n;
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) d[i + (unsigned long long)u * nthr] = v[u];
    }
  }
  // copies too short for U accesses per thread still get 4 in flight
  if (U > 4) {
#pragma unroll 1
    for (; i + 3ull * nthr < nv; i += 4ull * nthr) {
      V v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = load_vec<VB, LB>(s + i + (unsigned long long)u * nthr);
#pragma unroll
      for (int u = 0; u < 4; ++u) d[i + (unsigned long long)u * nthr] = v[u];
    }
  }
#pragma unroll 1
  for (; i < nv; i += nthr) d[i] = load_vec<VB, LB>(s + i);
  for (unsigned long long j = head + nv * VB + r; j < bytes; j += nthr) dst[j] = src[j];
}

// The body of a copy by whole warps (n >= 32 threads, of which the full warps
// take part): nv 16-byte vectors from an LB-byte aligned source, in tiles of
// U x 32 consecutive vectors, a warp per tile.  Within a tile every access is
// at a constant distance from the first, so a lane holds two addresses and U
// vectors (a stride known only at run time costs an address pair for each of
// the U accesses both ways: 72 instead of 60 registers for U = 8).
// PFI > 0: a lone warp keeps an L2 prefetch PFI tiles ahead (see copy_body).
//
// Tiles go in whole rounds of the block's warps; what is left would occupy some
// of them only (a message of 16 KiB is three of the all-to-all's tiles: 64 PEs
// 53 us a round by strides of the block, 68 with a tile to a warp, 45 so) and
// goes in rows.  EVEN deals the rows out over all warps, for a CTA that has its
// SM to itself (messages of 4100 bytes 48 -> 41 us a round); without it a warp
// takes four at a time, so that short copies occupy few warps where many CTAs
// share an SM (100,000 puts and gets of median 2 KiB, a CTA each: 272 us, 285
// with the rows dealt out).
template <int U, unsigned PFI, bool EVEN>
__device__ __forceinline__ void copy_tiles(char *__restrict__ dst, const char *__restrict__ src,
                                           unsigned long long nv, unsigned mis, unsigned r, unsigned n) {
  constexpr unsigned TB = U * 512;  // bytes per tile
  const unsigned nw = n >> 5, w = r >> 5, lane = r & 31u;
  if (w >= nw) return;
  const char *s = src + w * TB + lane * 16u;
  char *d = dst + w * TB + lane * 16u;
  long long left = (long long)nv;  // vectors from the round's (then the row's) first on
  const bool pf_on = PFI > 0 && n == 32 && lane == 0 && nv >= 2ull * PFI * U * 32 && __isGlobal(src);
  int staged = 16;  // bytes from s on that are on their way to L2
  // operands a number of bytes apart: in rows of four only (load_row)
  if ((mis & 3) == 0) {
#pragma unroll 1
    for (; left >= (long long)(nw * (U * 32)); left -= nw * (U * 32)) {
      uint4 v[U];
      load_row<U>(v, s, mis, U);
      if (pf_on) {
        int k = (int)(PFI * TB) - staged;
        if (left < (long long)(PFI * U * 32)) k = (int)left * 16 - 16 - staged;
        if (k >= 4096) {
          l2_prefetch_bulk(((uintptr_t)s & ~(uintptr_t)15) + staged, k);
          staged += k;
        }
        staged -= TB;
      }
#pragma unroll
      for (int u = 0; u < U; ++u) *reinterpret_cast<uint4 *>(d + u * 512) = v[u];
      s += nw * TB;
      d += nw * TB;
    }
  }
  // the vectors after the last round of tiles: up to 4 rows of 32 at a time
  const unsigned q = !EVEN || left > nw * 96 ? 128 : left > nw * 64 ? 96 : left > nw * 32 ? 64 : 32;
  s += (int)(w * q * 16) - (int)(w * TB);
  d += (int)(w * q * 16) - (int)(w * TB);
  left -= w * q;
#pragma unroll 1
  for (; left > 0; left -= nw * q) {
    uint4 v[4];
    const unsigned rows = left < q ? (unsigned)left : q;              // vectors of this round
    const unsigned have = rows > lane ? (rows - lane + 31) / 32 : 0;  // this lane's
    load_row<4>(v, s, mis, have);
#pragma unroll
    for (unsigned u = 0; u < 4; ++u)
      if (u < have) *reinterpret_cast<uint4 *>(d + u * 512) = v[u];
    s += nw * q * 16;
    d += nw * q * 16;
  }
}

// The bytes before and after the 16-byte vectors of the destination: fewer than
// 32, one each for the threads r of a warp or block.  Returns how many come
// before.
__device__ __forceinline__ unsigned copy_edges(char *dst, const char *src, unsigned long long bytes, unsigned r) {
  unsigned head = (unsigned)(16 - ((uintptr_t)dst & 15)) & 15u;
  if (head > bytes) head = (unsigned)bytes;
  const unsigned tail = (unsigned)(bytes - head) & 15u;
  if (r < head) dst[r] = src[r];
  if (r >= 16 && r - 16 < tail) {
    const unsigned long long j = bytes - tail + (r - 16);
    dst[j] = src[j];
  }
  return head;
}

// One thread, one warp or a block copies `bytes`: 16-byte stores, with loads
// as wide as the relative alignment of dst and src allows.  MAXV caps the
// width of both (4 and 8: the batch engine's narrow configurations).
// EVEN: see copy_tiles.
template <int MAXV = 16, int U = 4, unsigned PFI = 0, bool EVEN = false>
__device__ __forceinline__ void copy_coop(char *dst, const char *src, unsigned long long bytes,
                                          unsigned r, unsigned nthr) {
  const unsigned mis = (unsigned)((uintptr_t)dst ^ (uintptr_t)src);
  if (MAXV < 16) {
    if (MAXV == 8 && (mis & 7) == 0)
      copy_body<8, U, PFI>(dst, src, bytes, r, nthr);
    else if ((mis & 3) == 0)
      copy_body<4, U, PFI>(dst, src, bytes, r, nthr);
    else
      copy_body<1, U, PFI>(dst, src, bytes, r, nthr);
    return;
  }
  if (nthr < 32) {
    if ((mis & 3) != 0)
      copy_body<1, 4>(dst, src, bytes, r, nthr);
    else if ((mis & 15) == 0)
      copy_body<16, U, PFI>(dst, src, bytes, r, nthr);
    else if ((mis & 7) == 0)
      copy_body<16, U, PFI, 8>(dst, src, bytes, r, nthr);
    else
      copy_body<16, U, PFI, 4>(dst, src, bytes, r, nthr);
    return;
  }
  const unsigned head = copy_edges(dst, src, bytes, r);
  copy_tiles<U, PFI, EVEN>(dst + head, src + head, (bytes - head) >> 4, mis, r, nthr);
}

// One warp or a block copies `bytes` for the public calls, whose registers are
// those of an application's kernel, so they decide how many threads it may have
// and how many of its CTAs run at once: at most 64 for a kernel that does little
// else (with copy_coop such a kernel had 86 to 94 and did not run with 1024
// threads; 592 CTAs of 256 threads took two waves).  U vectors in flight where the
// operands are equal modulo 16, V where the loads are narrower.
template <int U, int V, unsigned PFI>
__device__ __forceinline__ void copy_group(char *dst, const char *src, unsigned long long bytes, unsigned r,
                                           unsigned n) {
  const unsigned mis = (unsigned)((uintptr_t)dst ^ (uintptr_t)src);
  if (n < 32) {
    if ((mis & 3) != 0)
      copy_body<1, 4>(dst, src, bytes, r, n);
    else if ((mis & 15) == 0)
      copy_body<16, 4>(dst, src, bytes, r, n);
    else
      copy_body<4, 4>(dst, src, bytes, r, n);
    return;
  }
  const unsigned head = copy_edges(dst, src, bytes, r);
  const unsigned long long nv = (bytes - head) >> 4;
  if ((mis & 15) == 0)
    copy_tiles<U, PFI, true>(dst + head, src + head, nv, 0, r, n);
  else
    copy_tiles<V, PFI, true>(dst + head, src + head, nv, mis, r, n);
}

// ----------------------------------------------- one copy per thread, shared
// A long copy by a whole warp: U vectors in flight per lane and the source
// prefetched into L2 `kAhead` bytes in front of the loads, which a lone warp
// waits for in every round.  Copies the whole rounds of U * 32 vectors and
// returns how many vectors that was.  (Two or three sets of 8 vectors in
// rotation, so that loads stay in flight while a set is stored, measured no
// better: they need the registers of U = 16 or 24 at once.)
constexpr unsigned kAhead = 32768;

template <int U>
__device__ __forceinline__ unsigned copy_warp_long(unsigned lane, char *dst, const char *src, unsigned nv,
                                                   unsigned mis) {
  const unsigned rounds = nv / (U * 32);
  const bool pf_on = lane == 0 && __isGlobal(src);
  const uintptr_t pf_end = ((uintptr_t)src + (unsigned long long)nv * 16u) & ~(uintptr_t)15;
  uintptr_t pf = ((uintptr_t)src + 15) & ~(uintptr_t)15;
  const char *s = src + 16u * lane;
  char *d = dst + 16u * lane;
#pragma unroll 1
  for (unsigned k = 0; k < rounds; ++k) {
    uint4 v[U];
    load_row<U>(v, s, mis, U);
    if (pf_on) {
      uintptr_t want = ((uintptr_t)s + kAhead) & ~(uintptr_t)15;
      if (want > pf_end) want = pf_end;
      if (want >= pf + 4096) {
        l2_prefetch_bulk(pf, (unsigned)(want - pf));
        pf = want;
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) *reinterpret_cast<uint4 *>(d + u * 512) = v[u];
    s += U * 512;
    d += U * 512;
  }
  return rounds * U * 32;
}

// The calling lanes' copies of one load alignment as one stream of 16-byte
// vectors: the lanes of `mask` (this one is number `r` of `nl`) take the
// messages of `todo` one after the other, nl vectors of one message per slot
// and U slots in flight, so U short messages or U * nl vectors of a long one
// are read at once.  dst / src / nv are this lane's own message.  One pass per
// alignment: with the width chosen per slot instead, the branches between the
// loads keep them from overlapping (25,000 calls: 215 us against 115-140 us).
template <int LB, int U>
__device__ __forceinline__ void copy_lanes_body(unsigned mask, unsigned todo, unsigned r, unsigned nl, char *dst,
                                                const char *src, unsigned nv) {
  unsigned long long cd = 0, cs = 0;  // the current message, at this lane's vector
  unsigned left = 0;                  // its vectors from lane 0's on
#pragma unroll 1
  while (left > 0 || todo) {
    uint4 v[U];
    uint4 *d[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      d[u] = nullptr;
      if (left == 0 && todo) {
        const int o = __ffs(todo) - 1;
        todo &= todo - 1;
        cd = __shfl_sync(mask, (unsigned long long)dst, o) + 16ull * r;
        cs = __shfl_sync(mask, (unsigned long long)src, o) + 16ull * r;
        left = __shfl_sync(mask, nv, o);
      }
      if (r < left) {
        d[u] = reinterpret_cast<uint4 *>(cd);
        v[u] = load16<LB>(reinterpret_cast<const char *>(cs));
      }
      cd += 16ull * nl;
      cs += 16ull * nl;
      left = left > nl ? left - nl : 0;
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (d[u]) *d[u] = v[u];
  }
}

// kLong: from this many vectors on (16 KiB) a copy is a long one; kTogether:
// fewer lanes than this copy alone (together they would have less in flight than
// each with 16 accesses of its own).
constexpr unsigned kLong = 1024, kTogether = 16;

// One copy by a warp, its long part with U vectors in flight per lane.
template <int U>
__device__ __forceinline__ void copy_warp(char *dst, const char *src, unsigned long long bytes, unsigned lane) {
  const unsigned mis = (unsigned)((uintptr_t)dst ^ (uintptr_t)src);
  if (bytes >= kLong * 16 && (mis & 3) == 0) {
    const unsigned head = (unsigned)(16 - ((uintptr_t)dst & 15)) & 15u;
    if (lane < head) dst[lane] = src[lane];
    const unsigned nv = (unsigned)((bytes - head) >> 4);
    const unsigned long long done = head + 16ull * copy_warp_long<U>(lane, dst + head, src + head, nv, mis);
    dst += done;
    src += done;
    bytes -= done;
  }
  copy_coop<16, 8>(dst, src, bytes, lane, 32);
}

template <int LB, unsigned N>
__device__ __forceinline__ void copy_own(char *dst, const char *src, unsigned nv) {
  uint4 v[N];
#pragma unroll
  for (unsigned k = 0; k < N; ++k)
    if (k < nv) v[k] = load16<LB>(src + 16 * k);
#pragma unroll
  for (unsigned k = 0; k < N; ++k)
    if (k < nv) reinterpret_cast<uint4 *>(dst)[k] = v[k];
}

// Whether the lanes of `mask` (nl of them, with copies of `bytes` bytes between
// operands `mis` apart) are sooner done each on its own, 16 accesses in flight,
// than together, SU * 32.  With less than two
// warps to an SM latency decides, not the memory's bandwidth, and copies of about
// one length are sooner done so (a round of lanes on their own takes half as
// long again as one together); with more warps only short ones are.  Us a launch,
// 32 lanes of every warp together and on their own: one warp to an SM, 260 bytes
// 8.5, 6.5, 4100 bytes 33, 27; four, 260 bytes 10.4, 8.3, 4100 bytes 43, 48;
// sixteen, 132 bytes 18, 14, 260 bytes 15, 22.
template <int SU, unsigned OWN>
__device__ __forceinline__ bool better_alone(unsigned mask, unsigned nl, unsigned long long bytes, unsigned mis) {
  const unsigned mine = bytes < kLong * 16 ? (unsigned)bytes >> 4 : kLong;
  if (!__any_sync(mask, mine > OWN)) return false;
  unsigned sms;
  asm("mov.u32 %0, %%nsmid;" : "=r"(sms));
  const unsigned warps = gridDim.x * gridDim.y * gridDim.z * ((blockDim.x * blockDim.y * blockDim.z + 31) >> 5);
  const unsigned most = __reduce_max_sync(mask, (mis & 15) == 0 || ((mis & 3) == 0 && mine <= 32) ? mine : kLong);
  const unsigned slots = __reduce_add_sync(mask, (mine + nl - 1) / nl);
  return most < kLong && most * 3 * SU < slots * 32 &&
         (warps < 2 * sms || (unsigned long long)warps * most < 96ull * sms);
}

// One copy per calling thread (the thread forms of put and get).  Lanes of a
// warp that arrive together carry their copies out together: a lane alone
// keeps at most 16 accesses in flight and touches a line of its own each
// time, while the group reads whole lines and has its accesses wherever there
// is work (see copy_lanes_body).  25,000 calls of log-normal sizes (median
// 2 KiB, up to 3 MiB, 282 MB moved) took 1240-2060 us with every lane on its
// own, as long as the longest call takes one thread; together 115-140 us.
// A lane whose copy has at most OWN vectors (one round trip, in parallel with
// the other lanes), or operands that are not 4-byte aligned, copies it itself,
// as do fewer than kTogether lanes, and a lane with an operand in its own local
// memory, where the same address names another array in every other lane.  LU /
// SU: the vectors in flight per lane for long and short copies.  FULL: the
// caller knows that all 32 lanes are here, with operands in the heap; without
// it the lanes also ask better_alone.
//
// The first __syncwarp makes what a lane wrote before its call visible to the
// lanes that copy for it, the last one makes their stores the calling lane's
// (its later fences and signals order them like its own).
template <int LU, int SU, bool FULL = false, unsigned OWN = 4>
__device__ __forceinline__ void copy_lanes(char *dst, const char *src, unsigned long long bytes) {
  unsigned mask = 0xffffffffu;
  bool local = false;
  if (!FULL) {
    local = __isLocal(dst) || __isLocal(src);
    mask = __ballot_sync(__activemask(), !local);
  }
  const unsigned nl = FULL ? 32u : __popc(mask);
  const unsigned mis = (unsigned)((uintptr_t)dst ^ (uintptr_t)src);
  if (!FULL && (local || nl < kTogether || better_alone<SU, OWN>(mask, nl, bytes, mis))) {
    // one thread: 16 vector accesses in flight (measured 2.6x the bandwidth of
    // 4 for a 1 MiB put) and an L2 prefetch 64 rounds (16 KiB) ahead: 1 MiB
    // from DRAM 0.90 -> 1.36 GB/s, from L2 1.89 -> 1.81 GB/s
    copy_coop<16, 16, 64>(dst, src, bytes, 0, 1);
    return;
  }
  __syncwarp(mask);
  unsigned nv = 0;
  if (((mis | (unsigned)(uintptr_t)dst | (unsigned)bytes) & 3) != 0) {
    copy_coop<16, 4>(dst, src, bytes, 0, 1);
  } else {
    // the words before and after the 16-byte vectors of the destination
    unsigned head = (unsigned)(16 - ((uintptr_t)dst & 15)) & 15u;
    if (head > bytes) head = (unsigned)bytes;
    nv = (unsigned)((bytes - head) >> 4);
    const unsigned tail = (unsigned)(bytes - head) & 15u;
    const char *ts = src + (bytes - tail);
    char *td = dst + (bytes - tail);
    unsigned w[6];
#pragma unroll
    for (unsigned k = 0; k < 3; ++k) {
      if (4 * k < head) w[k] = reinterpret_cast<const unsigned *>(src)[k];
      if (4 * k < tail) w[3 + k] = reinterpret_cast<const unsigned *>(ts)[k];
    }
#pragma unroll
    for (unsigned k = 0; k < 3; ++k) {
      if (4 * k < head) reinterpret_cast<unsigned *>(dst)[k] = w[k];
      if (4 * k < tail) reinterpret_cast<unsigned *>(td)[k] = w[3 + k];
    }
    dst += head;
    src += head;
    if (nv <= OWN) {
      if ((mis & 15) == 0)
        copy_own<16, OWN>(dst, src, nv);
      else if ((mis & 7) == 0)
        copy_own<8, OWN>(dst, src, nv);
      else
        copy_own<4, OWN>(dst, src, nv);
      nv = 0;
    }
  }
  const unsigned r = __popc(mask & ((1u << lane_number()) - 1u));
  if (mask == 0xffffffffu) {
#pragma unroll 1
    for (unsigned todo = __ballot_sync(mask, nv >= kLong); todo; todo &= todo - 1) {
      const int o = __ffs(todo) - 1;
      char *d = (char *)__shfl_sync(mask, (unsigned long long)dst, o);
      const char *p = (const char *)__shfl_sync(mask, (unsigned long long)src, o);
      const unsigned k = copy_warp_long<LU>(r, d, p, __shfl_sync(mask, nv, o), __shfl_sync(mask, mis, o));
      if ((int)r == o) {
        nv -= k;
        dst += 16ull * k;
        src += 16ull * k;
      }
    }
  }
  const unsigned lb = (mis & 15) == 0 ? 16 : ((mis & 7) == 0 ? 8 : 4);
  const unsigned t16 = __ballot_sync(mask, nv && lb == 16), t8 = __ballot_sync(mask, nv && lb == 8),
                 t4 = __ballot_sync(mask, nv && lb == 4);
  copy_lanes_body<16, SU>(mask, t16, r, nl, dst, src, nv);
  copy_lanes_body<8, SU>(mask, t8, r, nl, dst, src, nv);
  copy_lanes_body<4, SU>(mask, t4, r, nl, dst, src, nv);
  __syncwarp(mask);
}

__device__ __forceinline__ unsigned block_rank() {
  return threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z);
}
__device__ __forceinline__ unsigned block_size() { return blockDim.x * blockDim.y * blockDim.z; }

// ------------------------------------------------- TMA bulk (cp.async.bulk) ring
__device__ __forceinline__ void mbar_init(unsigned long long *m, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(m)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_inval(unsigned long long *m) {
  asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(smem_u32(m)) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long *m, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(m)),
               "r"(bytes)
               : "memory");
}
// Bounded wait on an mbarrier phase; returns false when `deadline` passed.
__device__ __forceinline__ bool mbar_wait(unsigned long long *m, unsigned parity,
                                          unsigned long long deadline) {
  unsigned addr = smem_u32(m);
  for (unsigned it = 0;; ++it) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(addr), "r"(parity)
        : "memory");
    if (ok) return true;
    if ((it & 63) == 63 && gtimer() > deadline) return false;
  }
}
__device__ __forceinline__ void bulk_g2s(void *smem_dst, const void *gsrc, unsigned bytes,
                                         unsigned long long *m) {
  asm volatile(
      "cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_u32(smem_dst)),
      "l"(gsrc), "r"(bytes), "r"(smem_u32(m))
      : "memory");
}
__device__ __forceinline__ void bulk_s2g(void *gdst, const void *smem_src, unsigned bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(gdst),
               "r"(smem_u32(smem_src)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// at most one bulk group (the newest store) may still be reading shared memory
__device__ __forceinline__ void bulk_wait_read1() {
  asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
}
// no bulk group may still be reading shared memory
__device__ __forceinline__ void bulk_wait_read_all() {
  asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}
__device__ __forceinline__ void bulk_wait_all() {
  asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  asm volatile("fence.proxy.async.global;" ::: "memory");
}

// Shared-memory layout of a bulk ring: up to 8 mbarriers in the first 128
// bytes, then `stages` buffers of `stage_bytes` (a multiple of 16).
struct BulkRing {
  unsigned long long *mbar;
  char *buf;
  unsigned stages;
  unsigned stage_bytes;
};

__device__ __forceinline__ BulkRing make_ring(void *smem, unsigned smem_bytes, unsigned want_stages) {
  BulkRing r;
  r.mbar = reinterpret_cast<unsigned long long *>(smem);
  r.buf = reinterpret_cast<char *>(smem) + 128;
  unsigned avail = smem_bytes > 128 ? smem_bytes - 128 : 0;
  unsigned st = want_stages < 2 ? 2 : (want_stages > 8 ? 8 : want_stages);
  unsigned sb = (avail / st) & ~127u;
  r.stages = st;
  r.stage_bytes = sb;
  return r;
}

// Single-thread bulk pipeline for a 16-byte aligned body (dst, src 16-aligned,
// bytes a multiple of 16): loads run up to `stages` - 1 ahead of the stores,
// and a stage is reloaded one store later than it could be, so the issuing
// thread never waits on the store it has just started (measured against
// reloading the stage of the newest store: one CTA's 1 MiB put 51 -> 60 GB/s,
// the 16 MiB all-to-all 6350 -> 6565 GB/s with 6 stages).
// Returns false if an mbarrier wait passed `deadline` (the copy is then
// incomplete; every issued store is still drained before returning).
__device__ __forceinline__ bool bulk_copy_1t(const BulkRing &ring, char *dst, const char *src,
                                             unsigned long long bytes, unsigned long long deadline) {
  if (bytes == 0) return true;
  const unsigned S = ring.stages, SB = ring.stage_bytes;
  const unsigned long long nch = (bytes + SB - 1) / SB;
  for (unsigned s = 0; s < S; ++s) mbar_init(ring.mbar + s, 1);
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  const unsigned long long pre = nch < S ? nch : S;
  for (unsigned long long c = 0; c < pre; ++c) {
    unsigned len = (unsigned)((bytes - c * SB) < SB ? (bytes - c * SB) : SB);
    mbar_expect_tx(ring.mbar + c, len);
    bulk_g2s(ring.buf + (size_t)c * SB, src + c * SB, len, ring.mbar + c);
  }
  bool ok = true;
  for (unsigned long long c = 0; c < nch; ++c) {
    const unsigned s = (unsigned)(c % S);
    const unsigned parity = (unsigned)((c / S) & 1);
    if (!mbar_wait(ring.mbar + s, parity, deadline)) {
      ok = false;
      break;
    }
    unsigned len = (unsigned)((bytes - c * SB) < SB ? (bytes - c * SB) : SB);
    bulk_s2g(dst + c * SB, ring.buf + (size_t)s * SB, len);
    bulk_commit();
    // refill the stage the previous store read, not this one: that store has
    // had a whole load wait to finish reading, while this one just started
    const unsigned long long n = c - 1 + S;
    if (c >= 1 && n < nch) {
      bulk_wait_read1();
      const unsigned ps = (unsigned)((c - 1) % S);
      unsigned nlen = (unsigned)((bytes - n * SB) < SB ? (bytes - n * SB) : SB);
      mbar_expect_tx(ring.mbar + ps, nlen);
      bulk_g2s(ring.buf + (size_t)ps * SB, src + n * SB, nlen, ring.mbar + ps);
    }
  }
  bulk_wait_all();
  if (ok) {
    for (unsigned s = 0; s < S; ++s) mbar_inval(ring.mbar + s);
  }
  return ok;
}

// Block-cooperative bulk copy: thread 0 drives the TMA ring over the
// 16-aligned body while the other threads copy the unaligned head and tail.
// Falls back to the generic copy when dst/src alignments differ mod 16, an
// operand is not in global memory or the ring has no room.  Every thread of the block must call it.
// One issuer per CTA streams the body as one sequential range: measured on
// B200 this keeps DRAM accesses more local than splitting the range across
// per-warp rings (which lost 6-7% on 16-256 MiB all-to-all rounds).
__device__ __forceinline__ void bulk_copy_block(const Cfg &c, char *dst, const char *src,
                                                unsigned long long bytes, void *smem,
                                                unsigned smem_bytes) {
  const unsigned r = block_rank(), n = block_size();
  BulkRing ring = make_ring(smem, smem_bytes, 6);
  if ((((uintptr_t)dst ^ (uintptr_t)src) & 15) != 0 || ring.stage_bytes < 1024 || bytes < 4096 ||
      n < 64 || !__isGlobal(dst) || !__isGlobal(src)) {
    copy_coop<16, 4>(dst, src, bytes, r, n);
    __syncthreads();
    return;
  }
  unsigned long long head = (16 - ((uintptr_t)dst & 15)) & 15;
  unsigned long long body = (bytes - head) & ~15ull;
  unsigned long long tail = bytes - head - body;
  if (r == 0) {
    unsigned long long deadline = gtimer() + (unsigned long long)c.wait_timeout_ns;
    if (!bulk_copy_1t(ring, dst + head, src + head, body, deadline))
      record_error(c, NVSHMEMX_ERR_TIMEOUT, -2);
  } else if (r >= 32) {
    // warps 1.. handle head and tail bytes
    unsigned rr = r - 32, nn = n - 32;
    for (unsigned long long i = rr; i < head; i += nn) dst[i] = src[i];
    for (unsigned long long i = rr; i < tail; i += nn) dst[head + body + i] = src[head + body + i];
  }
  __syncthreads();
}

// ---------------------------------------------------------------- waits
__device__ __forceinline__ bool cmp_ok(int v, int cmp, int x) {
  switch (cmp) {
    case NVSHMEMX_CMP_EQ: return v == x;
    case NVSHMEMX_CMP_NE: return v != x;
    case NVSHMEMX_CMP_GT: return v > x;
    case NVSHMEMX_CMP_GE: return v >= x;
    case NVSHMEMX_CMP_LT: return v < x;
    default: return v <= x;
  }
}

// Polls *p with ld.acquire.gpu until cmp_ok; tight polling first, then
// __nanosleep backoff (32 ns doubling to 256 ns) so idle waiters leave L2
// bandwidth to the copies.  Gives up after timeout_ns (library default when
// <= 0), records NVSHMEMX_ERR_TIMEOUT and returns it.
__device__ __forceinline__ int wait_cmp(const Cfg &c, const int *p, int cmp, int val,
                                        long long timeout_ns) {
  if (((uintptr_t)p & 3) != 0 || (in_arena(c, p) && slice_off(c, p) + 4 > c.slice_bytes)) {
    record_error(c, NVSHMEMX_ERR_BOUNDS, (long long)((const char *)p - c.arena));
    return NVSHMEMX_ERR_BOUNDS;
  }
  if (cmp_ok(ld_acquire(p), cmp, val)) return NVSHMEMX_SUCCESS;
  if (timeout_ns <= 0) timeout_ns = c.wait_timeout_ns;
  const unsigned long long t0 = gtimer();
  unsigned ns = 0;
  for (unsigned spins = 1;; ++spins) {
    if (cmp_ok(ld_acquire(p), cmp, val)) return NVSHMEMX_SUCCESS;
    if (spins > 64) {
      ns = ns == 0 ? 32 : (ns >= 256 ? 256 : ns * 2);
      __nanosleep(ns);
    }
    if ((spins & 15) == 0 && (long long)(gtimer() - t0) > timeout_ns) {
      record_error(c, NVSHMEMX_ERR_TIMEOUT, (long long)((const char *)p - c.arena));
      return NVSHMEMX_ERR_TIMEOUT;
    }
  }
}

// ---------------------------------------------------------------- barriers
// Ticket barrier over P CTAs on a monotonically increasing 64-bit counter:
// each CTA's leader adds 1 (acq_rel) and the CTAs of episode e = ticket / P
// leave once the counter reaches (e+1)*P.  One atomic per CTA and no reset
// between episodes; P must stay the same for the counter's lifetime (the
// launcher zeroes it before each launch).
__device__ __forceinline__ int ticket_barrier(const Cfg &c, unsigned long long *ctr,
                                              unsigned long long P) {
  __syncthreads();
  int rc = 0;
  if (block_rank() == 0) {
    // bar.sync orders the CTA's earlier writes before this thread's
    // operations; the acq_rel atomic releases them at GPU scope (cumulative),
    // so no separate fence is needed.
    const unsigned long long t = atom_add_acq_rel_u64(ctr, 1ull);
    const unsigned long long target = (t / P + 1ull) * P;
    if (ld_acquire_u64(ctr) < target) {
      const unsigned long long t0 = gtimer();
      for (unsigned spins = 1;; ++spins) {
        if (ld_acquire_u64(ctr) >= target) break;
        if (spins > 256) __nanosleep(64);
        if ((spins & 15) == 0 && (long long)(gtimer() - t0) > c.wait_timeout_ns) {
          record_error(c, NVSHMEMX_ERR_TIMEOUT, -1);
          rc = NVSHMEMX_ERR_TIMEOUT;
          break;
        }
      }
    }
  }
  rc = __syncthreads_or(rc) ? NVSHMEMX_ERR_TIMEOUT : 0;
  return rc;
}

__device__ __forceinline__ void red_add_release_u64(unsigned long long *p, unsigned long long v) {
  asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// The same barrier when every CTA knows which barrier of the launch this is
// (episode 0, 1, 2 ...): the leader arrives with a fire-and-forget
// red.release and polls for (episode+1)*P, so the last arriver does not wait
// for an atomic's return value before its first poll -- one L2 round trip
// less on the critical path.  Interoperates with ticket_barrier on the same
// counter as long as every CTA passes the true episode number.
__device__ __forceinline__ int episode_barrier(const Cfg &c, unsigned long long *ctr, unsigned long long P,
                                               unsigned long long episode) {
  __syncthreads();
  int rc = 0;
  if (block_rank() == 0) {
    red_add_release_u64(ctr, 1ull);  // releases the CTA's writes (see ticket_barrier)
    const unsigned long long target = (episode + 1ull) * P;
    if (ld_acquire_u64(ctr) < target) {
      const unsigned long long t0 = gtimer();
      for (unsigned spins = 1;; ++spins) {
        if (ld_acquire_u64(ctr) >= target) break;
        if (spins > 256) __nanosleep(64);
        if ((spins & 15) == 0 && (long long)(gtimer() - t0) > c.wait_timeout_ns) {
          record_error(c, NVSHMEMX_ERR_TIMEOUT, -1);
          rc = NVSHMEMX_ERR_TIMEOUT;
          break;
        }
      }
    }
  }
  rc = __syncthreads_or(rc) ? NVSHMEMX_ERR_TIMEOUT : 0;
  return rc;
}

__device__ __forceinline__ int barrier_all(const Cfg &c) {
  const unsigned long long P = (unsigned long long)gridDim.x * gridDim.y * gridDim.z;
  return ticket_barrier(c, c.coll_bar, P);
}

__device__ __forceinline__ int barrier_pe(const Cfg &c) {
  int pe = my_pe(c);
  if ((unsigned)pe >= (unsigned)c.npes) pe = 0;
  const unsigned long long P = (unsigned long long)gridDim.x * gridDim.y;
  return ticket_barrier(c, c.pe_bar + (size_t)pe * 16, P);  // counters 128 bytes apart
}

// ------------------------------------------------------- typed RMA (one thread)
// Scalar accesses must be naturally aligned; a misaligned address is recorded
// as a bounds error and skipped rather than executed (it would fault).
__device__ __forceinline__ bool check_align(const Cfg &c, const void *p, unsigned width) {
  if (((uintptr_t)p & (width - 1)) == 0) return true;
  record_error(c, NVSHMEMX_ERR_BOUNDS, (long long)((const char *)p - c.arena));
  return false;
}

template <typename T>
__device__ __forceinline__ void p_one(const Cfg &c, T *target, T value, int pe) {
  if (!check_remote(c, target, sizeof(T), pe) || !check_align(c, target, sizeof(T))) return;
  char *dst = xlate(c, target, pe);
  if (sizeof(T) == 8) {
    st_relaxed_b64(dst, *reinterpret_cast<unsigned long long *>(&value));
  } else {
    st_relaxed_b32(dst, *reinterpret_cast<unsigned int *>(&value));
  }
}

template <typename T>
__device__ __forceinline__ T g_one(const Cfg &c, const T *source, int pe) {
  if (!check_remote(c, source, sizeof(T), pe) || !check_align(c, source, sizeof(T))) return T(0);
  const char *src = xlate(c, source, pe);
  if (sizeof(T) == 8) {
    unsigned long long v = ld_relaxed_b64(src);
    return *reinterpret_cast<T *>(&v);
  } else {
    unsigned int v = ld_relaxed_b32(src);
    return *reinterpret_cast<T *>(&v);
  }
}

// Bytes of a put/get of `len` elements; a negative len copies nothing, as the
// prototype's `for (i = 0; i < len; i++)` loop.
template <typename T>
__device__ __forceinline__ unsigned long long elem_bytes(int len) {
  return len > 0 ? (unsigned long long)len * sizeof(T) : 0ull;
}

}  // namespace nvshm
