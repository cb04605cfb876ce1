// ops.cu -- host-callable operations (nvshmemx_ops.h): what an application of
// the prototype writes by hand, in one collective launch in which blockIdx.z is
// the PE.  The kernels call nvshmem_int_p, nvshmem_int_wait_until, nvshmem_quiet
// and the barriers of the public device API; their puts and gets have its checks,
// results and trace records and copy in the kernel itself.
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdio.h>

#include <algorithm>
#include <vector>

#include "nvshmem_device.h"
#include "nvshmemx.h"
#include "nvshmemx_ops.h"
#include "procs.h"
#include "runtime.h"

namespace nvshm {

namespace cg = cooperative_groups;

// Grow-only device scratch owned by the library (request uploads, results).
struct DevScratch {
  void *p = nullptr;
  size_t n = 0;
  void *get(size_t bytes) {
    if (bytes > n) {
      if (p) cudaFree(p);
      p = nullptr;
      n = 0;
      if (cudaMalloc(&p, bytes) != cudaSuccess) return nullptr;
      n = bytes;
    }
    return p;
  }
};
static DevScratch g_req_buf, g_out_buf;

// Times an operation on a stream with two events.  A host thread keeps its
// pair from operation to operation (creating and destroying them cost a call
// 3 us), one pair per thread, for the device that it last used.
struct EventTimer {
  struct Pair {
    cudaEvent_t a = nullptr, b = nullptr;
    int dev = -1;
    bool busy = false;
    void drop() {
      if (a) cudaEventDestroy(a);
      if (b) cudaEventDestroy(b);
      a = b = nullptr;
      dev = -1;
    }
    ~Pair() { drop(); }
  };
  static Pair &kept() {
    static thread_local Pair p;
    return p;
  }
  cudaEvent_t a = nullptr, b = nullptr;
  bool from_kept = false;
  EventTimer() {
    Pair &p = kept();
    int dev = 0;
    cudaGetDevice(&dev);
    if (!p.busy) {
      if (p.dev != dev) {
        p.drop();
        cudaEventCreate(&p.a);
        cudaEventCreate(&p.b);
        p.dev = dev;
      }
      p.busy = from_kept = true;
      a = p.a;
      b = p.b;
    } else {
      cudaEventCreate(&a);
      cudaEventCreate(&b);
    }
  }
  ~EventTimer() {
    if (from_kept) {
      kept().busy = false;
    } else {
      cudaEventDestroy(a);
      cudaEventDestroy(b);
    }
  }
  EventTimer(const EventTimer &) = delete;
  EventTimer &operator=(const EventTimer &) = delete;
  void start(cudaStream_t s = 0) { cudaEventRecord(a, s); }
  void stop(cudaStream_t s = 0) { cudaEventRecord(b, s); }
  float ms() {
    float m = 0;
    cudaEventSynchronize(b);
    cudaEventElapsedTime(&m, a, b);
    return m;
  }
};

__device__ __forceinline__ char *slice_ptr(const Cfg &c, int pe, unsigned long long off) {
  return c.arena + ((unsigned long long)(unsigned)pe << c.log2_stride) + off;
}

// ------------------------------------------------------------ request lists
// One caller unit per request: a thread (MODE_THREAD), a warp (MODE_WARP) or
// a CTA (MODE_BLOCK / MODE_BULK).  The symmetric operand is named by PE 0's
// copy of the object (any slice names the same object).

// A PUT or GET: the checks, translation, copy and trace record of the public
// put and get, written once for all operations and types.  In the thread form
// the lanes of a warp so reach the shared copy together (branching to the six
// typed calls would split them into groups); in the other forms the copy is
// part of the kernel, which has registers for more accesses in flight.
//
// In the thread form the warps of a cluster of CTAs share the long copies: one
// warp's copy moves 20-25 GB/s, so the longest of them decided when the kernel
// ended (25,000 calls of log-normal sizes, 282 MB moved, 110 and 132 us for two
// seeds; 83 us for both since).  A copy of kShareFrom bytes on is listed in
// its CTA's shared memory, and each warp, done with its shorter copies, claims
// pieces from its CTA's list and then from the others'.  (With 32 requests to a
// warp: 88-90 us; one CTA of 192 threads instead of four of 128 95 and 102 us,
// two of 96 threads 89 and 94, eight of 192 95 us; pieces of half the size,
// copies from 32 KiB on, 97-100 us, since each piece starts with loads that no
// prefetch has covered.)
constexpr int kShareThreads = 128, kShareCtas = 4;
constexpr unsigned kSharePiece = 32768, kShareFrom = 65536;

struct SharedCopies {
  unsigned long long dst[kShareThreads], src[kShareThreads], bytes[kShareThreads];
  unsigned next[kShareThreads];  // pieces of the copy claimed so far
  unsigned count;
};

// Lists a thread's copy.
__device__ __forceinline__ void share_copy(SharedCopies &l, char *dst, const char *src, unsigned long long bytes) {
  const unsigned k = atomicAdd(&l.count, 1u);
  l.dst[k] = (unsigned long long)dst;
  l.src[k] = (unsigned long long)src;
  l.bytes[k] = bytes;
  l.next[k] = 0;
}

// A warp's part of the copies that the cluster's CTAs have listed.
__device__ __forceinline__ void run_shared(SharedCopies *own, unsigned lane) {
  const cg::cluster_group cluster = cg::this_cluster();
  const unsigned rank = cluster.block_rank(), ctas = cluster.num_blocks();
#pragma unroll 1
  for (unsigned i = 0; i < ctas; ++i) {
    SharedCopies *l = cluster.map_shared_rank(own, (rank + i) % ctas);
    const unsigned count = l->count;
#pragma unroll 1
    for (unsigned k = 0; k < count; ++k) {
      const unsigned long long bytes = l->bytes[k], dst = l->dst[k], src = l->src[k];
#pragma unroll 1
      for (;;) {
        unsigned p = 0;
        if (lane == 0) p = atomicAdd(&l->next[k], 1u);
        const unsigned long long at = (unsigned long long)__shfl_sync(0xffffffffu, p, 0) * kSharePiece;
        if (at >= bytes) break;
        copy_warp<16>(reinterpret_cast<char *>(dst + at), reinterpret_cast<const char *>(src + at),
                      bytes - at < kSharePiece ? bytes - at : kSharePiece, lane);
      }
    }
  }
}

template <int MODE>
__device__ __forceinline__ void copy_request(const Cfg &c, const nvshmemx_request &r, char *smem, unsigned bulk_smem,
                                             SharedCopies *list = nullptr) {
  const bool put = r.op == NVSHMEMX_REQ_PUT;
  unsigned long long bytes = r.dtype == NVSHMEMX_DT_DOUBLE                                  ? r.bytes & ~7u
                             : r.dtype < NVSHMEMX_DT_DOUBLE || MODE == NVSHMEMX_MODE_BULK ? r.bytes & ~3u
                                                                                           : (r.bytes >> 2) * 8ull;
  char *near = slice_ptr(c, put ? r.src_pe : r.dst_pe, put ? r.src_off : r.dst_off);
  const char *sym = c.arena + (put ? r.dst_off : r.src_off);
  const int pe = put ? r.dst_pe : r.src_pe;
  bool ok = r.op <= NVSHMEMX_REQ_GET;
  ok = ok && check_remote(c, sym, bytes, pe) && check_local(c, near, bytes);
  if (MODE == NVSHMEMX_MODE_THREAD) {
    if (!ok) bytes = 0;
  } else if (!ok) {
    return;
  }
  char *far = xlate(c, sym, pe);
  char *dst = put ? far : near;
  const char *src = put ? near : far;
  const bool rec = ok && c.trace && MODE != NVSHMEMX_MODE_BULK &&
                   (MODE == NVSHMEMX_MODE_THREAD ||
                    (MODE == NVSHMEMX_MODE_WARP ? (threadIdx.x & 31) == 0 : threadIdx.x == 0));
  const unsigned long long t0 = rec ? gtimer() : 0;
  if (MODE == NVSHMEMX_MODE_THREAD) {
    // a traced copy stays with its warp: the record times it
    if (bytes >= kShareFrom && !c.trace) {
      share_copy(*list, dst, src, bytes);
      bytes = 0;
    }
    cg::this_cluster().sync();
    copy_lanes<16, 12, true>(dst, src, bytes);
    run_shared(list, threadIdx.x & 31);
    cg::this_cluster().sync();  // nobody claims from this CTA's list any more
  } else if (MODE == NVSHMEMX_MODE_WARP)
    copy_warp<12>(dst, src, bytes, threadIdx.x & 31);
  else if (MODE == NVSHMEMX_MODE_BLOCK)
    copy_coop<16, 8>(dst, src, bytes, threadIdx.x, blockDim.x);
  else
    bulk_copy_block(c, dst, src, bytes, smem, bulk_smem);
  if (rec) {
    const int op = (put ? NVSHMEMX_TRACE_PUT_INT : NVSHMEMX_TRACE_GET_INT) + (r.dtype < 2 ? (int)r.dtype : 2);
    trace_rec(c, op, near, far, bytes, pe, t0, gtimer());
  }
}

// CTAs of two warps in the warp form: a CTA's place frees up with its longest
// request.  It runs 20 warps per SM with 12 vectors in flight each: 100,000
// requests 255-270 us, against 300-360 us with 24 warps of 8 vectors in CTAs of
// eight (its largest request, one warp's, is a third of that time).  Sharing
// the long copies as in the thread form, in CTAs of two to eight warps, took
// 278-299 us where this takes 257: a warp then waits for its CTA's others.
//
// The CTA forms have two shapes.  A CTA spends about 2 us on a short request
// (its descriptor, then its data), so many requests want many CTAs: 128 threads,
// seven to an SM (block form, 100,000 requests of median 2 KiB 505 -> 291 us,
// 20,000 125 -> 93 us; TMA form 510 -> 308 us and 126 -> 100 us).  With fewer
// the longest requests decide, and three CTAs of 256 threads are ahead (block
// form, 1500 requests of median 64 KiB 110 against 122 us, 4100 of 16 KiB 107
// against 113; the TMA form, whose ring shrinks with the CTA, 6000 of 16 KiB
// 121 against 139 us).
constexpr int kManyBlock = 6144, kManyBulk = 12288;

template <int MODE, int THREADS>
__global__ void __launch_bounds__(THREADS, MODE == NVSHMEMX_MODE_THREAD ? 384 / THREADS
                                           : MODE == NVSHMEMX_MODE_WARP ? 10
                                           : THREADS == 128             ? 7
                                                                        : 3)
    exec_requests_kernel(Cfg c, const nvshmemx_request *__restrict__ reqs, int n, unsigned bulk_smem,
                         unsigned lanes) {
  extern __shared__ __align__(128) char smem[];
  long long u;
  if (MODE == NVSHMEMX_MODE_THREAD)
    // `lanes` of a warp have a request (see launch_exec_requests)
    u = (threadIdx.x & 31) < lanes
            ? (((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * lanes + (threadIdx.x & 31)
            : n;
  else if (MODE == NVSHMEMX_MODE_WARP)
    u = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  else
    u = blockIdx.x;
  nvshmemx_request r;
  if (MODE == NVSHMEMX_MODE_THREAD) {
    // every thread takes part in the copies, those without a request too
    r.op = 0xff;
    r.bytes = 0;
    r.dtype = 0;
    r.src_pe = r.dst_pe = 0;
    r.src_off = r.dst_off = 0;
    if (u < n) r = reqs[u];
  } else {
    if (u >= n) return;
    r = reqs[u];
  }
  const bool leader = MODE == NVSHMEMX_MODE_THREAD || (MODE == NVSHMEMX_MODE_WARP ? (threadIdx.x & 31) == 0
                                                                                 : threadIdx.x == 0);
  const int w = r.dtype == NVSHMEMX_DT_DOUBLE ? 8 : 4;
  switch (r.op) {
    case NVSHMEMX_REQ_PUT:
    case NVSHMEMX_REQ_GET:
      if (MODE != NVSHMEMX_MODE_THREAD) copy_request<MODE>(c, r, smem, bulk_smem);
      break;
    case NVSHMEMX_REQ_SIGNAL:
      if (leader) nvshmemx_int_signal((int *)(c.arena + r.dst_off), r.value, r.dst_pe);
      break;
    case NVSHMEMX_REQ_P:
      if (leader) {
        char *sym = c.arena + r.dst_off;
        if (r.dtype == NVSHMEMX_DT_INT) nvshmem_int_p((int *)sym, (int)(unsigned)r.src_off, r.dst_pe);
        else if (r.dtype == NVSHMEMX_DT_FLOAT)
          nvshmem_float_p((float *)sym, __uint_as_float((unsigned)r.src_off), r.dst_pe);
        else nvshmem_double_p((double *)sym, __longlong_as_double((long long)r.src_off), r.dst_pe);
      }
      break;
    case NVSHMEMX_REQ_G:
      if (leader) {
        char *sym = c.arena + r.src_off;
        char *dst = slice_ptr(c, r.dst_pe, r.dst_off);
        if (check_local(c, dst, w) && check_align(c, dst, w)) {
          if (r.dtype == NVSHMEMX_DT_INT) *(int *)dst = nvshmem_int_g((int *)sym, r.src_pe);
          else if (r.dtype == NVSHMEMX_DT_FLOAT) *(float *)dst = nvshmem_float_g((float *)sym, r.src_pe);
          else *(double *)dst = nvshmem_double_g((double *)sym, r.src_pe);
        }
      }
      break;
    default:
      if (leader && u < n) record_error(c, NVSHMEMX_ERR_INVALID, (long long)u);
  }
  if (MODE == NVSHMEMX_MODE_THREAD) {
    // last: the request's other fields need no registers during the copies
    __shared__ SharedCopies list;
    if (threadIdx.x == 0) list.count = 0;
    __syncthreads();
    copy_request<MODE>(c, r, smem, bulk_smem, &list);
  }
}

// ---------------------------------------------------------------- fill etc.
__device__ __forceinline__ unsigned long long splitmix64(unsigned long long x) {
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}
// Word w of PE p's slice for `seed`: the stream is keyed on (seed, pe) so
// every PE and every seed gets independent contents.
__device__ __forceinline__ unsigned long long fill_word(unsigned long long seed, int pe, unsigned long long w) {
  return splitmix64(splitmix64(seed ^ ((unsigned long long)pe << 48)) + w);
}

__global__ void fill_random_kernel(char *slice, unsigned long long off, unsigned long long bytes,
                                   unsigned long long seed, int pe) {
  // byte b (slice offset off+b) takes byte (off+b)%8 of word (off+b)/8
  const unsigned long long first_w = off >> 3, last_w = (off + bytes + 7) >> 3;
  const unsigned long long nthr = (unsigned long long)gridDim.x * blockDim.x;
  for (unsigned long long w = first_w + blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; w < last_w;
       w += nthr) {
    unsigned long long v = fill_word(seed, pe, w);
    unsigned long long lo = w << 3, hi = lo + 8;
    if (lo >= off && hi <= off + bytes) {
      *(unsigned long long *)(slice + lo) = v;
    } else {
      for (unsigned long long b = lo; b < hi; ++b)
        if (b >= off && b < off + bytes) slice[b] = (char)((v >> (8 * (b - lo))) & 0xff);
    }
  }
}

__global__ void compare_kernel(const unsigned char *a, const unsigned char *b, unsigned long long bytes,
                               unsigned long long *mismatches) {
  unsigned long long local = 0;
  const unsigned long long nthr = (unsigned long long)gridDim.x * blockDim.x;
  const unsigned long long tid = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x;
  if ((((uintptr_t)a | (uintptr_t)b) & 15) == 0) {
    const unsigned long long nv = bytes >> 4;
    const uint4 *a4 = (const uint4 *)a, *b4 = (const uint4 *)b;
    for (unsigned long long i = tid; i < nv; i += nthr) {
      uint4 x = a4[i], y = b4[i];
      if (x.x != y.x || x.y != y.y || x.z != y.z || x.w != y.w) {
        for (int k = 0; k < 16; ++k) local += a[i * 16 + k] != b[i * 16 + k];
      }
    }
    for (unsigned long long i = (nv << 4) + tid; i < bytes; i += nthr) local += a[i] != b[i];
  } else {
    for (unsigned long long i = tid; i < bytes; i += nthr) local += a[i] != b[i];
  }
  for (int o = 16; o > 0; o >>= 1) local += __shfl_xor_sync(0xffffffffu, local, o);
  if ((threadIdx.x & 31) == 0 && local) atomicAdd(mismatches, local);
}

__global__ void checksum_kernel(const unsigned long long *p, unsigned long long nwords, unsigned long long *out) {
  unsigned long long local = 0;
  const unsigned long long nthr = (unsigned long long)gridDim.x * blockDim.x;
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < nwords; i += nthr)
    local += splitmix64(p[i] ^ (i * 0x9E3779B97F4A7C15ull));
  for (int o = 16; o > 0; o >>= 1) local += __shfl_xor_sync(0xffffffffu, local, o);
  if ((threadIdx.x & 31) == 0) atomicAdd(out, local);
}

// ------------------------------------------------------------- C1 ping-pong
// The put + flag exchange of microbench/shmem_latency.cu:48-81 (and, with
// len == 0, the flag-only one of shmem_sync_latency.cu:48-78), with the PE
// taken from the launch instead of a kernel argument and the local copies of
// the symmetric objects named through nvshmemx_local_ptr.  PE 0 puts its data
// and sets PE 1's flag to i+1; PE 1 waits for its flag to leave i
// (nvshmem_int_wait), puts its data back and echoes i+1 into PE 0's flag.
// Each side has one value in flight, so no flag value can be overwritten
// before it is seen (the microbench's alternating equality waits can miss an
// i+1 that the peer already replaced with i+2).
// Each PE has one thread, so the put is that thread's own copy, written into
// the kernel with the checks and the trace record of nvshmem_int_put: the call
// would save and restore the registers of its group copy (exchanges of
// 4, 68 and 1020 bytes 3.35, 3.71 and 8.5 us with the call, 2.94, 3.05 and 7.7
// without).  Whole vectors go straight to the copy: the branches around the
// words outside them cost a short exchange more than those words (16, 64 and
// 256 bytes 2.29, 2.28 and 2.38 us an exchange through them, 2.20, 2.20 and
// 2.27 straight).
__device__ __forceinline__ void put_ints_alone(const Cfg &c, int *target, const int *source, int len, int pe) {
  const unsigned long long bytes = elem_bytes<int>(len);
  if (!check_remote(c, target, bytes, pe) || !check_local(c, source, bytes)) return;
  char *dst = xlate(c, target, pe);
  const unsigned long long t0 = c.trace ? gtimer() : 0;
  const char *src = reinterpret_cast<const char *>(source);
  const uintptr_t at = (uintptr_t)dst | (uintptr_t)src;
  if ((at & 3) != 0 || ((at | bytes) & 15) == 0) {
    copy_coop<16, 16, 64>(dst, src, bytes, 0, 1);
  } else {
    // the words outside the destination's vectors, loaded before those
    unsigned head = (unsigned)(16 - ((uintptr_t)dst & 15)) & 15u;
    if (head > bytes) head = (unsigned)bytes;
    const unsigned tail = (unsigned)(bytes - head) & 15u;
    const unsigned *hs = reinterpret_cast<const unsigned *>(src), *ts = hs + (bytes - tail) / 4;
    unsigned *hd = reinterpret_cast<unsigned *>(dst), *td = hd + (bytes - tail) / 4;
    unsigned w[6];
#pragma unroll
    for (unsigned k = 0; k < 3; ++k) {
      if (4 * k < head) w[k] = hs[k];
      if (4 * k < tail) w[3 + k] = ts[k];
    }
    if (bytes - head >= 16) copy_coop<16, 16, 64>(dst + head, src + head, bytes - head - tail, 0, 1);
#pragma unroll
    for (unsigned k = 0; k < 3; ++k) {
      if (4 * k < head) hd[k] = w[k];
      if (4 * k < tail) td[k] = w[3 + k];
    }
  }
  if (c.trace) trace_rec(c, NVSHMEMX_TRACE_PUT_INT, source, dst, bytes, pe, t0, gtimer());
}

// DATA: a payload goes before the flag.  Without one the kernel is a flag's
// round trip alone, in 26 registers instead of 220 (760 -> 704 ns).
template <bool DATA>
__global__ void pingpong_kernel(Cfg c, int *data, int *flag, int len, int iters, int skip, long long *cycles,
                                unsigned long long *gt) {
  const int pe = nvshmemx_my_pe();
  if (pe > 1 || threadIdx.x != 0 || blockIdx.x != 0) return;
  int *my_flag = (int *)nvshmemx_local_ptr(flag);
  int *my_data = (int *)nvshmemx_local_ptr(data);
  unsigned long long g0 = 0;
  for (int i = 0; i < iters + skip; ++i) {
    if (i == skip) g0 = nvshm::gtimer();
    long long t = clock64();
    if (pe == 0) {
      if (DATA) {
        put_ints_alone(c, data, my_data, len, 1);
        nvshmem_quiet();
      }
      nvshmem_int_p(flag, i + 1, 1);
      nvshmem_int_wait(my_flag, i);
    } else {
      nvshmem_int_wait(my_flag, i);
      if (DATA) {
        put_ints_alone(c, data, my_data, len, 0);
        nvshmem_quiet();
      }
      nvshmem_int_p(flag, i + 1, 0);
    }
    if (pe == 0 && i >= skip) cycles[i - skip] = clock64() - t;
  }
  if (pe == 0) gt[0] = nvshm::gtimer() - g0;
}

// ------------------------------------------------------------ barrier latency
__global__ void barrier_latency_kernel(int iters, int counted, long long *cycles, unsigned long long *gt) {
  const bool rec = blockIdx.x == 0 && blockIdx.z == 0 && threadIdx.x == 0;
  unsigned long long g0 = nvshm::gtimer();
  long long t = clock64();
  for (int i = 0; i < iters; ++i) {
    if (counted)
      nvshmemx_barrier_all_ep((unsigned long long)i);
    else
      nvshmemx_barrier_all();
    if (rec) {
      long long t1 = clock64();
      cycles[i] = t1 - t;
      t = t1;
    }
  }
  if (rec) gt[0] = nvshm::gtimer() - g0;
}

// -------------------------------------------------------------- C2 all-to-all
// Where message k of the share starts: its destination and source.
__device__ __forceinline__ void a2a_message(const Cfg &c, int op, int pe, unsigned long long so, unsigned long long ro,
                                            unsigned long long bytes, unsigned long long k, char **dst,
                                            const char **src) {
  const int q = (pe + 1 + (int)k) % c.npes;
  if (op == NVSHMEMX_REQ_PUT) {
    *dst = xlate(c, c.arena + ro + (unsigned long long)pe * bytes, q);
    *src = slice_ptr(c, pe, so + (unsigned long long)q * bytes);
  } else {
    *dst = slice_ptr(c, pe, ro + (unsigned long long)q * bytes);
    *src = xlate(c, c.arena + so + (unsigned long long)pe * bytes, q);
  }
}

// A CTA's share of the all-to-all rounds: in each, [b, e) of the PE's (npes-1)
// * `bytes` outgoing (put) or incoming (get) bytes, streamed by one thread
// through one TMA ring of kA2aStages stages.  The ring runs across message
// boundaries, so a share that spans two messages is loaded and stored without
// draining the ring between them (a cooperative bulk copy per message fills
// and drains its ring once per message), and, where no round's destinations
// overlap any round's sources (`ahead`), across rounds: the loads of the next
// round's first chunks are issued before this round's barrier, so a round no
// longer starts by waiting for its first load (8 PEs, us a round with a ring
// per round and now: 4 KiB messages 3.0 and 2.76, 256 KiB 8.2 and 7.2, 1 MiB
// 21.6 and 20.9).  Every chunk stays inside one message; all addresses are
// 16-byte aligned (the caller checks).  Stage reuse lags one store behind, as
// in bulk_copy_1t.
// Shared memory: 8 mbarriers, the destination and length of each stage's chunk
// (256 bytes), then the stages.
constexpr unsigned kA2aStages = 6;
constexpr unsigned kLastOfRound = 1u << 31;  // in a stage's length: the share's last chunk

struct A2aRing {
  unsigned long long *mbar, *sdst;
  unsigned *slen;
  char *buf;
  unsigned SB;
  unsigned issued, stored;       // chunks loaded and stored so far, over all rounds
  // the next chunk to load: in round `lr`, at `off` of message k, `left` bytes
  // of the round's share from there
  int lr;
  unsigned long long k, off, left;
  char *dbase;
  const char *sbase;
};

// The share and the buffers it moves between (the same for every round).
struct A2aShare {
  int op, pe, nsets;
  unsigned long long send, recv, stride, bytes, b, e;
};

__device__ __forceinline__ void a2a_round_start(const Cfg &c, A2aRing &g, const A2aShare &h, int round) {
  const unsigned long long set = (unsigned long long)(round % h.nsets) * h.stride;
  g.lr = round;
  g.k = h.b / h.bytes;
  g.off = h.b - g.k * h.bytes;
  g.left = h.e - h.b;
  a2a_message(c, h.op, h.pe, h.send + set, h.recv + set, h.bytes, g.k, &g.dbase, &g.sbase);
}

// Loads the next chunk into the next stage (which must be free).  The issuing
// thread walks the share message by message (one division per round, none per
// chunk): at tens of GB/s per CTA a 10 KiB chunk leaves it a few hundred cycles.
__device__ __forceinline__ void a2a_load(const Cfg &c, A2aRing &g, const A2aShare &h) {
  unsigned long long len = h.bytes - g.off;
  if (len > g.left) len = g.left;
  if (len > g.SB) len = g.SB;
  const unsigned s = g.issued % kA2aStages;
  g.sdst[s] = (unsigned long long)(g.dbase + g.off);
  g.slen[s] = (unsigned)len | (g.left == len ? kLastOfRound : 0u);
  mbar_expect_tx(g.mbar + s, (unsigned)len);
  bulk_g2s(g.buf + (size_t)s * g.SB, g.sbase + g.off, (unsigned)len, g.mbar + s);
  ++g.issued;
  g.off += len;
  g.left -= len;
  if (g.off == h.bytes && g.left) {
    const unsigned long long set = (unsigned long long)(g.lr % h.nsets) * h.stride;
    g.off = 0;
    a2a_message(c, h.op, h.pe, h.send + set, h.recv + set, h.bytes, ++g.k, &g.dbase, &g.sbase);
  }
}

// One thread: the stores of round `round`, with loads running ahead up to the
// end of round `last_load`.  Returns false if an mbarrier wait passed
// `deadline`; every store it issued is complete when it returns.
__device__ __forceinline__ bool a2a_round_1t(const Cfg &c, A2aRing &g, const A2aShare &h, int round, int last_load,
                                             unsigned long long deadline) {
  auto more = [&]() -> bool {
    if (g.left == 0 && g.lr < last_load) a2a_round_start(c, g, h, g.lr + 1);
    return g.left != 0;
  };
  if (g.lr < round) a2a_round_start(c, g, h, round);
  while (g.issued - g.stored < kA2aStages && more()) a2a_load(c, g, h);
  bool last = false;
  for (unsigned i = 0; !last; ++i) {
    const unsigned s = g.stored % kA2aStages;
    if (!mbar_wait(g.mbar + s, (g.stored / kA2aStages) & 1u, deadline)) {
      bulk_wait_all();
      return false;
    }
    const unsigned len = g.slen[s];
    last = (len & kLastOfRound) != 0;
    bulk_s2g(reinterpret_cast<void *>(g.sdst[s]), g.buf + (size_t)s * g.SB, len & ~kLastOfRound);
    bulk_commit();
    ++g.stored;
    // refill the stage the previous store read, not this one (see bulk_copy_1t)
    if (i >= 1 && more()) {
      bulk_wait_read1();
      a2a_load(c, g, h);
    }
  }
  bulk_wait_all();
  // every stage is free now: the next round's loads pass the barrier
  while (g.issued - g.stored < kA2aStages && more()) a2a_load(c, g, h);
  return true;
}

// Rounds in the CTA-wide TMA mode when everything is 16-byte aligned: a
// kernel of its own, so that the ring's state has the registers (in one kernel
// with the unaligned copies it spilled, which cost 1.1 us a round).
__global__ void __launch_bounds__(256, 3) alltoall_ring_kernel(Cfg c, A2aShare share, int rounds, unsigned bulk_smem,
                                                               int device_barrier, int ahead) {
  extern __shared__ __align__(128) char smem[];
  const unsigned long long total = (unsigned long long)(c.npes - 1) * share.bytes;
  const unsigned long long seg = (((total + gridDim.x - 1) / gridDim.x) + 15) & ~15ull;
  share.pe = blockIdx.z;
  share.b = blockIdx.x * seg;
  share.e = share.b + seg < total ? share.b + seg : total;
  A2aRing ring;
  ring.mbar = reinterpret_cast<unsigned long long *>(smem);
  ring.sdst = reinterpret_cast<unsigned long long *>(smem + 64);
  ring.slen = reinterpret_cast<unsigned *>(smem + 128);
  ring.buf = smem + 256;
  ring.SB = ((bulk_smem - 256) / kA2aStages) & ~127u;
  ring.issued = ring.stored = 0;
  ring.lr = -1;
  ring.left = 0;
  bool run = threadIdx.x == 0 && share.b < share.e;
  if (run) {
    for (unsigned s = 0; s < kA2aStages; ++s) mbar_init(ring.mbar + s, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  for (int r = 0; r < rounds; ++r) {
    if (run && !a2a_round_1t(c, ring, share, r, ahead && r + 1 < rounds ? r + 1 : r,
                             gtimer() + (unsigned long long)c.wait_timeout_ns)) {
      record_error(c, NVSHMEMX_ERR_TIMEOUT, -2);
      run = false;
    }
    if (device_barrier) {
      nvshmemx_barrier_all_ep((unsigned long long)r);
    } else {
      __syncthreads();
      if (threadIdx.x == 0) nvshmem_quiet();
    }
  }
}

// Message k (0..npes-2) of PE p goes to / comes from peer q = (p+1+k) % npes.
// For the cooperative modes the PE's (npes-1)*bytes are cut into one
// contiguous, 16-byte-rounded segment per caller unit (warp or CTA), so every
// unit streams one range; MODE_THREAD has one thread per message, as the
// per-thread put and get (whose copies a warp's lanes share).
// Bounds: as many threads and CTAs per SM as its callers may ask for: a thread
// per message up to 129 PEs and (kThreadMany) up to 289, two CTAs, in the
// CTA-wide TMA mode three.
constexpr int kThreadMany = 4;  // MODE_THREAD for more than 129 PEs
constexpr int kUnaligned = 5;   // MODE_BULK with buffers that are not 16-byte aligned

template <int MODE>
__global__ void __launch_bounds__(MODE == NVSHMEMX_MODE_THREAD ? 128 : MODE == kThreadMany ? 288 : 256,
                                  MODE == kUnaligned ? 3 : 2)
    alltoall_kernel(Cfg c, int op, int dtype, unsigned long long send_off,
                                unsigned long long recv_off, unsigned long long bytes, int rounds, int nsets,
                                unsigned long long set_stride, int device_barrier) {
  const int pe = blockIdx.z, np = c.npes;
  const unsigned long long total = (unsigned long long)(np - 1) * bytes;
  unsigned long long unit, nunits;
  constexpr bool by_thread = MODE == NVSHMEMX_MODE_THREAD || MODE == kThreadMany;
  if (by_thread) {
    unit = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
    nunits = (unsigned long long)(np - 1);
  } else if (MODE == NVSHMEMX_MODE_WARP) {
    unit = ((unsigned long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    nunits = (unsigned long long)gridDim.x * (blockDim.x >> 5);
  } else {
    unit = blockIdx.x;
    nunits = gridDim.x;
  }
  const unsigned long long seg = (((total + nunits - 1) / nunits) + 15) & ~15ull;  // a unit's share of a round
  for (int r = 0; r < rounds; ++r) {
    const unsigned long long so = send_off + (unsigned long long)(r % nsets) * set_stride;
    const unsigned long long ro = recv_off + (unsigned long long)(r % nsets) * set_stride;
    if (by_thread) {
      // the copies of nvshmem_{T}_put / _get by one thread per message; the
      // lanes without a message help (copy_lanes)
      char *dst = nullptr;
      const char *src = nullptr;
      const bool mine = unit < nunits;
      if (mine) a2a_message(c, op, pe, so, ro, bytes, unit, &dst, &src);
      const bool rec = mine && c.trace;
      const unsigned long long t0 = rec ? gtimer() : 0;
      copy_lanes<MODE == NVSHMEMX_MODE_THREAD ? 8 : 4, MODE == NVSHMEMX_MODE_THREAD ? 8 : 2, true>(dst, src, mine ? bytes : 0);
      if (rec)
        trace_rec(c, (op == NVSHMEMX_REQ_PUT ? NVSHMEMX_TRACE_PUT_INT : NVSHMEMX_TRACE_GET_INT) + dtype,
                  op == NVSHMEMX_REQ_PUT ? src : dst, op == NVSHMEMX_REQ_PUT ? dst : src, bytes,
                  (pe + 1 + (int)unit) % np, t0, gtimer());
    } else {
      unsigned long long b = unit * seg;
      const unsigned long long e = b + seg < total ? b + seg : total;
      while (b < e) {
        const unsigned long long k = b / bytes, off = b - k * bytes;
        const unsigned long long len = (e - b) < (bytes - off) ? (e - b) : (bytes - off);
        char *dst;
        const char *src;
        a2a_message(c, op, pe, so, ro, bytes, k, &dst, &src);
        dst += off;
        src += off;
        const bool rec = c.trace && (MODE == NVSHMEMX_MODE_WARP ? (threadIdx.x & 31) == 0
                                                                : MODE == NVSHMEMX_MODE_BLOCK && threadIdx.x == 0);
        const unsigned long long t0 = rec ? gtimer() : 0;
        if (MODE == NVSHMEMX_MODE_WARP)
          copy_coop<16, 8, 4>(dst, src, len, threadIdx.x & 31, 32);
        else  // one CTA per SM: 12 vectors in flight per lane (16 MiB a round 302 us, 317 with 8)
          copy_coop<16, MODE == NVSHMEMX_MODE_BLOCK ? 12 : 8, 0, true>(dst, src, len, threadIdx.x, blockDim.x);
        if (rec)
          trace_rec(c, op == NVSHMEMX_REQ_PUT ? NVSHMEMX_TRACE_PUT_INT : NVSHMEMX_TRACE_GET_INT,
                    op == NVSHMEMX_REQ_PUT ? src : dst, op == NVSHMEMX_REQ_PUT ? dst : src, len,
                    (pe + 1 + (int)k) % np, t0, gtimer());
        b += len;
      }
    }
    // the barrier's __syncthreads orders every thread's stores before the
    // leader, whose release (without a barrier: quiet) covers them all
    if (device_barrier) {
      nvshmemx_barrier_all_ep((unsigned long long)r);
    } else {
      __syncthreads();
      if (threadIdx.x == 0) nvshmem_quiet();
    }
  }
}

// ------------------------------------------------------------------ C3 halo
// Face d (0..5 = -x,+x,-y,+y,-z,+z) of the sender goes to the neighbour in
// direction d, into that neighbour's ghost buffer for direction d^1.  A face
// is n rows of n doubles; one warp moves one row per step.
__device__ __forceinline__ int halo_nbr(int pe, int d, int px, int py, int pz) {
  int x = pe % px, y = (pe / px) % py, z = pe / (px * py);
  const int s = (d & 1) ? 1 : -1;
  if (d < 2) x = (x + s + px) % px;
  else if (d < 4) y = (y + s + py) % py;
  else z = (z + s + pz) % pz;
  return x + px * (y + py * z);
}

// `iters` iterations numbered from it0 (signal values it0 + it + 1); with
// device_barrier each iteration ends at the device barrier, without it the
// caller follows the launch with nvshmem_barrier_all_offload (one iteration
// per launch, the prototype's own structure).
// The face rows are 2 KiB warp copies; they use the same checks and
// translation as nvshmemx_putmem_warp, inlined with a 4-deep copy loop (the
// public call is a shared out-of-line helper with a deeper loop tuned for
// long copies, which costs this short-row kernel registers and a call).
__device__ __forceinline__ void halo_row_put(const Cfg &c, double *dst_sym, const double *src, size_t bytes, int pe,
                                             unsigned lane) {
  if (!check_remote(c, dst_sym, bytes, pe) || !check_local(c, src, bytes)) return;
  char *dst = xlate(c, dst_sym, pe);
  const unsigned long long t0 = (c.trace && lane == 0) ? gtimer() : 0;
  if ((((uintptr_t)dst ^ (uintptr_t)src) & 15) == 0)
    copy_body<16, 4>(dst, reinterpret_cast<const char *>(src), bytes, lane, 32);
  else
    copy_body<8, 4>(dst, reinterpret_cast<const char *>(src), bytes, lane, 32);
  if (c.trace && lane == 0) trace_rec(c, NVSHMEMX_TRACE_PUT_INT, src, dst, bytes, pe, t0, gtimer());
}

// One x-face row: n doubles at stride n (src[k * n]) to n contiguous doubles
// at dst_sym on PE pe, with the checks of nvshmem_double_p made once for the
// row.  The gather is bound by DRAM access latency (every element is in its
// own row of the block), so each lane keeps 8 loads in flight, read through
// the non-coherent path without L1 allocation (the block is not written
// during the exchange), before storing them; stores are relaxed, ordered by
// the release that follows the faces.  `meanwhile` runs once, with the first
// loads in flight.
template <typename F>
__device__ __forceinline__ void halo_xrow_put(const Cfg &c, double *dst_sym, const double *src, int n, int pe,
                                              unsigned lane, F &&meanwhile) {
  const unsigned long long bytes = (unsigned long long)n * 8ull;
  const bool ok = check_remote(c, dst_sym, bytes, pe) && check_local(c, src, (unsigned long long)(n - 1) * bytes + 8);
  unsigned long long *dst = reinterpret_cast<unsigned long long *>(xlate(c, dst_sym, pe));
  const unsigned long long *s = reinterpret_cast<const unsigned long long *>(src);
  const long long stride = n;
  if (ok && c.trace && lane == 0) {
    const unsigned long long t = gtimer();
    trace_rec(c, NVSHMEMX_TRACE_PUT_DOUBLE, src, dst, bytes, pe, t, t);
  }
  if (!ok) n = 0;
  for (int k0 = 0; k0 < n || k0 == 0; k0 += 256) {
    unsigned long long v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int k = k0 + u * 32 + (int)lane;
      if (k < n)
        asm volatile("ld.global.nc.L1::no_allocate.L2::64B.b64 %0, [%1];" : "=l"(v[u]) : "l"(s + k * stride));
    }
    if (k0 == 0) meanwhile();
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int k = k0 + u * 32 + (int)lane;
      if (k < n) st_relaxed_b64(dst + k, v[u]);
    }
  }
}

// Bytes of shared memory in which a warp stages y and z rows.
constexpr unsigned kHaloStage = 4096;

// The face exchange.  What bounds an iteration at n = 256 is the gather of
// the x faces: a million 8-byte elements, each in a DRAM page of its own
// (20 us; 16 us at strides up to 512 bytes, where two share a page).  Its data
// take half of the memory's bandwidth meanwhile, so the contiguous rows of
// the y and z faces go along with it: every warp starts its rows as TMA loads
// into shared memory, gathers its x row, and sends the rows on while the
// gather's loads are in flight (32.4 us an iteration with every row through
// registers in turn, 29.0 now; n = 128: 11.8 and 10.9).  Rows of an odd number of doubles, not 16-byte aligned, and
// rows below kHaloTmaN doubles, which a TMA round trip only delays, are copied
// through registers after the x faces.
//
// The meeting at the end: every CTA releases its writes with one add on its
// PE's counter; only the PE's first CTA waits for all of them, sets the
// neighbours' signals and waits for its own; then the barrier over all PEs.
constexpr int kHaloTmaN = 96;

// Rows of n doubles that a warp's stage holds; 0: rows go through registers.
__host__ __device__ __forceinline__ int halo_rows(int n) {
  return (n & 1) == 0 && n >= kHaloTmaN ? (int)(kHaloStage / (8u * (unsigned)n)) : 0;
}

__global__ void __launch_bounds__(256, 4) halo_kernel(Cfg c, int px, int py, int pz, int n, unsigned long long block_off,
                            unsigned long long ghost_off, unsigned long long sig_off, int iters, int it0,
                            int device_barrier) {
  extern __shared__ __align__(128) char smem[];
  const int pe = blockIdx.z;
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const unsigned long long row_bytes = (unsigned long long)n * 8ull, face_bytes = row_bytes * n;
  const long long gw = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
  const double *blk = (const double *)slice_ptr(c, pe, block_off);
  int *my_sig = (int *)slice_ptr(c, pe, sig_off);
  unsigned long long *mbar = reinterpret_cast<unsigned long long *>(smem) + warp;
  char *stage = smem + 128 + warp * kHaloStage;
  const int fit = halo_rows(n);
  unsigned phase = 0;
  if (fit) {
    if (lane == 0) {
      mbar_init(mbar, 1);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncwarp();
  }
  // the y and z rows begin with the warps that have no x row
  const long long yu0 = gw >= 2ll * n % nw ? gw - 2ll * n % nw : gw - 2ll * n % nw + nw;
  // row u of the y and z faces: where it starts and which ghost row takes it
  auto yz_row = [&](long long u, const double **src, double **sym) -> int {
    const int d = 2 + (int)((unsigned)u / (unsigned)n), j = (int)((unsigned)u % (unsigned)n);
    *sym = (double *)(c.arena + ghost_off + (unsigned long long)(d ^ 1) * face_bytes + j * row_bytes);
    // y face: row j is z = j; z face: row j is y = j of its plane
    *src = d < 4 ? blk + ((long long)j * n + ((d & 1) ? n - 1 : 0)) * n
                 : blk + ((long long)((d & 1) ? n - 1 : 0) * n + j) * n;
    return halo_nbr(pe, d, px, py, pz);
  };
  for (int it = 0; it < iters; ++it) {
    long long yu = yu0;  // the warp's next y / z row
    auto load_rows = [&]() {
      if (lane != 0) return;
      unsigned k = 0;
      while ((int)k < fit && yu + k * nw < 4ll * n) ++k;
      if (k == 0) return;
      bulk_wait_read_all();  // the stage's earlier rows are on their way
      mbar_expect_tx(mbar, k * (unsigned)row_bytes);
      for (unsigned i = 0; i < k; ++i) {
        const double *src;
        double *sym;
        yz_row(yu + i * nw, &src, &sym);
        bulk_g2s(stage + i * row_bytes, src, (unsigned)row_bytes, mbar);
      }
    };
    auto send_rows = [&]() {
      if (lane == 0 && yu < 4ll * n) {
        if (!mbar_wait(mbar, phase & 1u, gtimer() + (unsigned long long)c.wait_timeout_ns)) {
          record_error(c, NVSHMEMX_ERR_TIMEOUT, -2);
        } else {
          for (int i = 0; i < fit && yu + i * nw < 4ll * n; ++i) {
            const double *src;
            double *sym;
            const int nb = yz_row(yu + i * nw, &src, &sym);
            char *dst = xlate(c, sym, nb);
            bulk_s2g(dst, stage + i * row_bytes, (unsigned)row_bytes);
            if (c.trace) {
              const unsigned long long t = gtimer();
              trace_rec(c, NVSHMEMX_TRACE_PUT_INT, src, dst, row_bytes, nb, t, t);
            }
          }
          bulk_commit();
        }
        ++phase;
      }
      yu += fit * nw;
    };
    if (fit) load_rows();
    bool sent = fit == 0;
    // x faces: units pair them row by row (unit 2j reads element x = 0 and
    // unit 2j+1 element x = n-1 of the same rows, on neighbouring warps at
    // about the same time); row z=j gathers element (z=j, y=k), at
    // blk[(j*n + k)*n + x0], into consecutive doubles on the neighbour
    for (long long u = gw; u < 2ll * n; u += nw) {
      const int d = (int)(u & 1), j = (int)(u >> 1);
      double *sym = (double *)(c.arena + ghost_off + (unsigned long long)(d ^ 1) * face_bytes + j * row_bytes);
      halo_xrow_put(c, sym, blk + (long long)j * n * n + (d ? n - 1 : 0), n, halo_nbr(pe, d, px, py, pz), lane, [&]() {
        if (!sent) {
          send_rows();
          sent = true;
        }
      });
    }
    if (fit) {
      if (!sent) send_rows();
      while (yu < 4ll * n) {
        load_rows();
        send_rows();
      }
      if (lane == 0) bulk_wait_all();
      __syncwarp();
    } else {
      for (long long u = yu0; u < 4ll * n; u += nw) {
        const double *src;
        double *sym;
        const int nb = yz_row(u, &src, &sym);
        halo_row_put(c, sym, src, row_bytes, nb, lane);
      }
    }
    // the CTA's writes are released by its leader's add, after the CTA's barrier
    __syncthreads();
    if (threadIdx.x == 0) red_add_release_u64(c.pe_bar + (size_t)pe * 16, 1ull);
    if (blockIdx.x == 0) {
      if (threadIdx.x == 0) {
        const unsigned long long want = (unsigned long long)(it + 1) * gridDim.x, t0 = gtimer();
        for (unsigned spins = 1; ld_acquire_u64(c.pe_bar + (size_t)pe * 16) < want; ++spins)
          if ((spins & 15) == 0 && (long long)(gtimer() - t0) > c.wait_timeout_ns) {
            record_error(c, NVSHMEMX_ERR_TIMEOUT, -1);
            break;
          }
      }
      __syncthreads();
      if (threadIdx.x < 6) {
        const int d = threadIdx.x;
        nvshmem_quiet();
        nvshmem_int_p((int *)(c.arena + sig_off) + (d ^ 1), it0 + it + 1, halo_nbr(pe, d, px, py, pz));
        nvshmem_int_wait_until(my_sig + d, 0, it0 + it + 1);
      }
    }
    if (device_barrier) nvshmemx_barrier_all_ep((unsigned long long)it);
  }
}

// ------------------------------------------------ strided-read ceiling
// What the halo's x faces cost at best: every PE reads nsets x rows 8-byte
// elements, element i of set t at slice offset off + t * set_off +
// i * stride, with ctas_per_pe CTAs per PE and 8 loads in flight per lane
// (the access pattern of halo_xrow_put without its stores; consecutive
// threads take the sets of one row in turn, as the halo pairs its two x
// faces), and adds them into one word per warp so that nothing is optimised
// away.
__global__ void __launch_bounds__(256) strided_read_kernel(Cfg c, unsigned long long off, unsigned long long set_off,
                                                           int nsets, unsigned long long rows,
                                                           unsigned long long stride, unsigned long long *sink) {
  const int pe = blockIdx.y;
  const char *base = slice_ptr(c, pe, off);
  const unsigned long long total = (unsigned long long)nsets * rows;
  const unsigned long long nthr = (unsigned long long)gridDim.x * blockDim.x;
  const unsigned long long t0 = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
  unsigned long long acc = 0;
  for (unsigned long long i0 = t0; i0 < total; i0 += 8 * nthr) {
    unsigned long long v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const unsigned long long i = i0 + (unsigned long long)u * nthr;
      v[u] = 0;
      if (i < total) {
        const unsigned long long set = i % (unsigned long long)nsets, row = i / (unsigned long long)nsets;
        const char *p = base + set * set_off + row * stride;
        asm volatile("ld.global.nc.L1::no_allocate.L2::64B.b64 %0, [%1];" : "=l"(v[u]) : "l"(p));
      }
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) acc += v[u];
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) atomicAdd(sink, acc);
}

// ------------------------------------------------------- failure detection
__global__ void wait_test_kernel(Cfg c, int *flag, int value, long long timeout_ns, int *out) {
  if (threadIdx.x == 0) out[0] = wait_cmp(c, flag, NVSHMEMX_CMP_EQ, value, timeout_ns);
}

__global__ void barrier_fault_kernel(Cfg c, int skip_pe, int *out) {
  if ((int)blockIdx.z == skip_pe) return;  // this PE never arrives
  int rc = barrier_all(c);
  if (threadIdx.x == 0 && rc) atomicMax(out, rc);
}

}  // namespace nvshm

using namespace nvshm;

static int need_started() {
  if (!is_started()) return fail(NVSHMEMX_ERR_STATE, "operation before nvstart_pes");
  // Drop a non-sticky error left by an earlier, unrelated runtime call so the
  // launch checks below report only this operation's own failures (sticky
  // device errors persist and are still reported).
  (void)cudaGetLastError();
  return 0;
}

// The C1-C3 operations run every PE in one collective launch and meet at
// device barriers; with one process per PE those barriers would see only
// this process's CTAs, so the operations refuse instead.
static int need_collective() {
  int rc;
  if ((rc = need_started())) return rc;
  if (proc_mode())
    return fail(NVSHMEMX_ERR_STATE, "operation needs every PE in one process (one process per PE is active)");
  return 0;
}

static int last_launch(const char *what) {
  return check_cuda(cudaGetLastError(), what);
}

// [off, off + bytes) lies inside [0, limit).  Arguments come from the caller
// as size_t, so the test never forms a sum that could wrap.
static bool range_ok(size_t off, size_t bytes, size_t limit) { return off <= limit && bytes <= limit - off; }

// *out = a * b, false when the product does not fit a size_t.
static bool mul_ok(size_t a, size_t b, size_t *out) {
  if (a != 0 && b > (size_t)-1 / a) return false;
  *out = a * b;
  return true;
}

// Shared memory of the halo kernel: mbarriers and a stage for each of its 8
// warps, none where it does not stage rows.
static unsigned halo_smem(int n) { return halo_rows(n) ? 128 + 8 * kHaloStage : 0; }

// Shared memory for the CTA-wide TMA copies: a 64 KiB ring (six stages)
// plus 128 bytes of mbarriers (three CTAs fit an SM).
static const unsigned kBulkSmem = 4 * 16384 + 128;
// ... and the ring of the CTAs of 128 threads (exec_requests_kernel): seven
// CTAs fit an SM.
static const unsigned kBulkSmemMany = 30 * 1024 + 128;

namespace nvshm {
int launch_exec_requests(int mode, const nvshmemx_request *dr, int n, cudaStream_t s) {
  const Cfg c = rt().cfg;
  if (n <= 0) return 0;
  switch (mode) {
    case NVSHMEMX_MODE_THREAD: {
      // Requests to a warp: no more than keep the warps of two CTAs to an SM
      // busy (up to 38,000 requests; 4100 of median 16 KiB took 322 us with 32
      // to a warp in CTAs of 64 threads, 110 so; 600 of 64 KiB 527 and 76 us;
      // 1000 of 2 KiB 47 and 30; for one CTA to an SM 116, 96 and 30 us).
      const long long warps = (long long)rt().sm_count * (2 * kShareThreads / 32);
      const unsigned lanes = (unsigned)std::min<long long>(32, (n + warps - 1) / warps);
      const long long per = (long long)lanes * (kShareThreads / 32) * kShareCtas;
      cudaLaunchAttribute at = {};
      at.id = cudaLaunchAttributeClusterDimension;
      at.val.clusterDim.x = kShareCtas;
      at.val.clusterDim.y = at.val.clusterDim.z = 1;
      cudaLaunchConfig_t lc = {};
      lc.gridDim = dim3((unsigned)((n + per - 1) / per) * kShareCtas);
      lc.blockDim = dim3(kShareThreads);
      lc.stream = s;
      lc.attrs = &at;
      lc.numAttrs = 1;
      const cudaError_t e =
          cudaLaunchKernelEx(&lc, exec_requests_kernel<NVSHMEMX_MODE_THREAD, kShareThreads>, c, dr, n, 0u, lanes);
      if (e != cudaSuccess) return check_cuda(e, "exec_requests launch");
      break;
    }
    case NVSHMEMX_MODE_WARP:
      exec_requests_kernel<NVSHMEMX_MODE_WARP, 64><<<(n + 1) / 2, 64, 0, s>>>(c, dr, n, 0, 0);
      break;
    case NVSHMEMX_MODE_BLOCK:
      if (n > kManyBlock)
        exec_requests_kernel<NVSHMEMX_MODE_BLOCK, 128><<<n, 128, 0, s>>>(c, dr, n, 0, 0);
      else
        exec_requests_kernel<NVSHMEMX_MODE_BLOCK, 256><<<n, 256, 0, s>>>(c, dr, n, 0, 0);
      break;
    default: {
      const bool many = n > kManyBulk;
      const auto fn = many ? exec_requests_kernel<NVSHMEMX_MODE_BULK, 128> : exec_requests_kernel<NVSHMEMX_MODE_BULK, 256>;
      const unsigned smem = many ? kBulkSmemMany : kBulkSmem;
      cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      fn<<<n, many ? 128 : 256, smem, s>>>(c, dr, n, smem, 0);
    }
  }
  return check_cuda(cudaGetLastError(), "exec_requests launch");
}
}  // namespace nvshm

extern "C" {

int nvshmemx_exec_requests(const nvshmemx_request *reqs, int n, int mode, float *out_ms) {
  int rc;
  if ((rc = need_started())) return rc;
  if (n < 0 || mode < 0 || mode > NVSHMEMX_MODE_BULK) return fail(NVSHMEMX_ERR_INVALID, "exec_requests: bad n/mode");
  if (out_ms) *out_ms = 0.f;
  if (n == 0) return 0;
  const Runtime &r = rt();
  for (int i = 0; i < n; ++i) {
    const nvshmemx_request &q = reqs[i];
    if (q.src_pe >= r.npes || q.dst_pe >= r.npes || q.op > NVSHMEMX_REQ_G || q.dtype > NVSHMEMX_DT_DOUBLE)
      return fail(NVSHMEMX_ERR_INVALID, "exec_requests: request %d has a bad pe/op/dtype", i);
  }
  void *d = g_req_buf.get((size_t)n * sizeof(nvshmemx_request));
  if (!d) return fail(NVSHMEMX_ERR_NOMEM, "exec_requests: cannot allocate request buffer");
  if ((rc = check_cuda(cudaMemcpy(d, reqs, (size_t)n * sizeof(nvshmemx_request), cudaMemcpyHostToDevice),
                       "cudaMemcpy(requests)")))
    return rc;
  const nvshmemx_request *dr = (const nvshmemx_request *)d;
  EventTimer t;
  t.start();
  rc = launch_exec_requests(mode, dr, n, 0);
  t.stop();
  if (rc) return rc;
  float ms = t.ms();
  if (out_ms) *out_ms = ms;
  return check_cuda(cudaDeviceSynchronize(), "exec_requests");
}

int nvshmemx_fill_random(int pe, size_t off, size_t bytes, uint64_t seed) {
  int rc;
  if ((rc = need_started())) return rc;
  const Runtime &r = rt();
  if (pe < 0 || pe >= r.npes || off > r.heap_bytes || bytes > r.heap_bytes - off)
    return fail(NVSHMEMX_ERR_INVALID, "fill_random: range outside the slice");
  if (bytes == 0) return 0;
  fill_random_kernel<<<r.sm_count * 8, 256>>>(r.arena + (size_t)pe * r.stride, off, bytes, seed, pe);
  if ((rc = last_launch("fill_random"))) return rc;
  return check_cuda(cudaDeviceSynchronize(), "fill_random");
}

int nvshmemx_compare(int a_pe, size_t a_off, int b_pe, size_t b_off, size_t bytes, unsigned long long *out) {
  int rc;
  if ((rc = need_started())) return rc;
  const Runtime &r = rt();
  if (a_pe < 0 || a_pe >= r.npes || b_pe < 0 || b_pe >= r.npes || a_off > r.heap_bytes ||
      bytes > r.heap_bytes - a_off || b_off > r.heap_bytes || bytes > r.heap_bytes - b_off)
    return fail(NVSHMEMX_ERR_INVALID, "compare: range outside the slice");
  unsigned long long *d = (unsigned long long *)g_out_buf.get(64);
  if (!d) return fail(NVSHMEMX_ERR_NOMEM, "compare: scratch");
  cudaMemset(d, 0, 8);
  if (bytes)
    compare_kernel<<<r.sm_count * 8, 256>>>((const unsigned char *)(r.arena + (size_t)a_pe * r.stride + a_off),
                                            (const unsigned char *)(r.arena + (size_t)b_pe * r.stride + b_off),
                                            bytes, d);
  if ((rc = last_launch("compare"))) return rc;
  return check_cuda(cudaMemcpy(out, d, 8, cudaMemcpyDeviceToHost), "compare result");
}

int nvshmemx_checksum(int pe, size_t off, size_t bytes, unsigned long long *out) {
  int rc;
  if ((rc = need_started())) return rc;
  const Runtime &r = rt();
  if (pe < 0 || pe >= r.npes || off > r.heap_bytes || bytes > r.heap_bytes - off || (bytes & 7) || (off & 7))
    return fail(NVSHMEMX_ERR_INVALID, "checksum: range outside the slice or not 8-byte aligned");
  unsigned long long *d = (unsigned long long *)g_out_buf.get(64);
  if (!d) return fail(NVSHMEMX_ERR_NOMEM, "checksum: scratch");
  cudaMemset(d, 0, 8);
  if (bytes)
    checksum_kernel<<<r.sm_count * 8, 256>>>((const unsigned long long *)(r.arena + (size_t)pe * r.stride + off),
                                             bytes / 8, d);
  if ((rc = last_launch("checksum"))) return rc;
  return check_cuda(cudaMemcpy(out, d, 8, cudaMemcpyDeviceToHost), "checksum result");
}

int nvshmemx_op_pingpong(size_t flag_off, size_t data_off, int len_elems, int iters, int skip, double *out_ns,
                         double *out_total_ns) {
  int rc;
  if ((rc = need_collective())) return rc;
  const Runtime &r = rt();
  if (r.npes < 2) return fail(NVSHMEMX_ERR_INVALID, "pingpong needs at least 2 PEs");
  if (iters < 1 || skip < 0 || len_elems < 0 || !range_ok(flag_off, 4, r.heap_bytes) ||
      !range_ok(data_off, (size_t)len_elems * 4, r.heap_bytes))
    return fail(NVSHMEMX_ERR_INVALID, "pingpong: bad arguments");
  long long *cyc = (long long *)g_out_buf.get((size_t)iters * 8 + 64);
  if (!cyc) return fail(NVSHMEMX_ERR_NOMEM, "pingpong scratch");
  unsigned long long *gt = (unsigned long long *)(cyc + iters);
  int *data = (int *)(r.arena + data_off);
  int *flag = (int *)(r.arena + flag_off);
  // both flag words start at 0, whatever an earlier exchange left there
  for (int pe = 0; pe < 2; ++pe)
    if ((rc = check_cuda(cudaMemsetAsync(r.arena + (size_t)pe * r.stride + flag_off, 0, 4, 0), "pingpong flags")))
      return rc;
  Cfg c = r.cfg;
  void *args[] = {&c, &data, &flag, &len_elems, &iters, &skip, &cyc, &gt};
  const void *fn = len_elems > 0 ? (const void *)pingpong_kernel<true> : (const void *)pingpong_kernel<false>;
  if ((rc = launch_collective(fn, dim3(1), dim3(32), args, 0, 0))) return rc;
  if ((rc = check_cuda(cudaDeviceSynchronize(), "pingpong"))) return rc;
  std::vector<long long> h(iters);
  unsigned long long total = 0;
  cudaMemcpy(h.data(), cyc, (size_t)iters * 8, cudaMemcpyDeviceToHost);
  cudaMemcpy(&total, gt, 8, cudaMemcpyDeviceToHost);
  double sum = 0;
  for (long long v : h) sum += (double)v;
  const double ns_per_cycle = sum > 0 ? (double)total / sum : 0.0;
  if (out_ns)
    for (int i = 0; i < iters; ++i) out_ns[i] = (double)h[i] * ns_per_cycle;
  if (out_total_ns) *out_total_ns = (double)total;
  return 0;
}

int nvshmemx_op_barrier_latency(int ctas_per_pe, int iters, int counted, double *out_ns, double *out_total_ns) {
  int rc;
  if ((rc = need_collective())) return rc;
  if (ctas_per_pe < 1 || iters < 1) return fail(NVSHMEMX_ERR_INVALID, "barrier_latency: bad arguments");
  long long *cyc = (long long *)g_out_buf.get((size_t)iters * 8 + 64);
  if (!cyc) return fail(NVSHMEMX_ERR_NOMEM, "barrier scratch");
  unsigned long long *gt = (unsigned long long *)(cyc + iters);
  void *args[] = {&iters, &counted, &cyc, &gt};
  if ((rc = launch_collective((const void *)barrier_latency_kernel, dim3(ctas_per_pe), dim3(128), args, 0, 0)))
    return rc;
  if ((rc = check_cuda(cudaDeviceSynchronize(), "barrier_latency"))) return rc;
  std::vector<long long> h(iters);
  unsigned long long total = 0;
  cudaMemcpy(h.data(), cyc, (size_t)iters * 8, cudaMemcpyDeviceToHost);
  cudaMemcpy(&total, gt, 8, cudaMemcpyDeviceToHost);
  double sum = 0;
  for (long long v : h) sum += (double)v;
  const double ns_per_cycle = sum > 0 ? (double)total / sum : 0.0;
  if (out_ns)
    for (int i = 0; i < iters; ++i) out_ns[i] = (double)h[i] * ns_per_cycle;
  if (out_total_ns) *out_total_ns = (double)total;
  return 0;
}

int nvshmemx_op_offload_barrier(int iters, double *out_us_per_call) {
  int rc;
  if ((rc = need_collective())) return rc;
  if (iters < 1) return fail(NVSHMEMX_ERR_INVALID, "offload_barrier: iters < 1");
  nvshmem_barrier_all_offload();  // warm-up
  if ((rc = check_cuda(cudaDeviceSynchronize(), "offload barrier"))) return rc;
  EventTimer t;
  t.start();
  for (int i = 0; i < iters; ++i) nvshmem_barrier_all_offload();
  t.stop();
  float ms = t.ms();
  if (out_us_per_call) *out_us_per_call = 1000.0 * ms / iters;
  return check_cuda(cudaDeviceSynchronize(), "offload barrier");
}

// Validates the arguments and picks the kernel, grid and block of an
// all-to-all in `mode`.
// CTAs per PE for an operation called with 0: NVSHMEM_CTAS_PER_PE when it is
// set to a positive count, else the operation's own choice `fallback`.
static int default_ctas_per_pe(int fallback) {
  const char *v = getenv("NVSHMEM_CTAS_PER_PE");
  const int k = v ? atoi(v) : 0;
  return k > 0 ? k : fallback;
}

static int alltoall_setup(int op, int dtype, size_t send_off, size_t recv_off, size_t bytes, int rounds, int nsets,
                          size_t set_stride, int mode, int ctas_per_pe, const void **fn, dim3 *grid, dim3 *block,
                          unsigned *smem) {
  int rc;
  if ((rc = need_collective())) return rc;
  const Runtime &r = rt();
  // 0: one CTA per PE per 1/npes of the SMs (18 for 8 PEs on 148 SMs: one
  // ring-driving CTA per SM measured fastest from 4 MiB messages on)
  if (ctas_per_pe == 0) ctas_per_pe = default_ctas_per_pe(r.sm_count / r.npes > 0 ? r.sm_count / r.npes : 1);
  if ((op != NVSHMEMX_REQ_PUT && op != NVSHMEMX_REQ_GET) || dtype < 0 || dtype > NVSHMEMX_DT_DOUBLE ||
      mode < 0 || mode > NVSHMEMX_MODE_BULK || rounds < 1 || nsets < 1 || ctas_per_pe < 1 || r.npes < 2)
    return fail(NVSHMEMX_ERR_INVALID, "alltoall: bad arguments");
  const int w = dtype == NVSHMEMX_DT_DOUBLE ? 8 : 4;
  if (bytes % w) return fail(NVSHMEMX_ERR_INVALID, "alltoall: bytes not a multiple of the element width");
  if (mode == NVSHMEMX_MODE_THREAD && bytes / w > 0x7fffffffull)
    return fail(NVSHMEMX_ERR_INVALID, "alltoall: message too long for an int element count");
  // every set of send and receive buffers, [off + s * set_stride, + npes * bytes)
  // for s < nsets, must lie inside the heap; no product or sum may wrap
  size_t span = 0, last = 0;
  if (!mul_ok((size_t)r.npes, bytes, &span) || !mul_ok((size_t)(nsets - 1), set_stride, &last) ||
      !range_ok(last, span, r.heap_bytes) || !range_ok(send_off, last + span, r.heap_bytes) ||
      !range_ok(recv_off, last + span, r.heap_bytes))
    return fail(NVSHMEMX_ERR_INVALID, "alltoall: buffers exceed the heap");
  *smem = mode == NVSHMEMX_MODE_BULK ? kBulkSmem : 0;
  *grid = dim3(ctas_per_pe);
  *block = dim3(256);
  switch (mode) {
    case NVSHMEMX_MODE_THREAD:
      // CTAs of up to 128 threads have the registers for 8 vectors in flight per
      // lane, larger ones for 4 and 2 (with more they spill).  Us a round with 4096
      // bytes to a message, with each lane on its own, with 4 in flight, and now:
      // 34 PEs 25.6, 44.5, 16.4; 64 PEs 52.7, 90.7, 26.9; 128 PEs 105, 115, 37.6;
      // (4 and 2) 160 PEs 183, 123, 90; 200 PEs 324, 136, 98
      *fn = r.npes <= 129 ? (const void *)alltoall_kernel<NVSHMEMX_MODE_THREAD>
                         : (const void *)alltoall_kernel<kThreadMany>;
      *grid = dim3(1);
      *block = dim3(32 * ((r.npes - 1 + 31) / 32));
      break;
    case NVSHMEMX_MODE_WARP: *fn = (const void *)alltoall_kernel<NVSHMEMX_MODE_WARP>; break;
    case NVSHMEMX_MODE_BLOCK: *fn = (const void *)alltoall_kernel<NVSHMEMX_MODE_BLOCK>; break;
    default: {
      // the ring that runs across rounds needs every buffer 16-byte aligned
      const bool aligned = ((bytes | send_off | recv_off | (nsets > 1 ? set_stride : 0)) & 15) == 0;
      // (without it the block form's copies are ahead of a TMA ring per message,
      // which only some messages can use: 1,048,580 bytes 26.1 against 33.1 us a
      // round, 12,000,008 bytes 235 against 301; the mode still records no puts)
      *fn = aligned ? (const void *)alltoall_ring_kernel : (const void *)alltoall_kernel<kUnaligned>;
      if (!aligned) *smem = 0;
    }
  }
  return 0;
}

// One collective launch of `rounds` rounds from buffer sets at send / recv.
static int alltoall_launch(const void *fn, dim3 grid, dim3 block, unsigned smem, int op, int dtype, size_t send,
                           size_t recv, size_t bytes, int rounds, int nsets, size_t stride, int device_barrier) {
  Cfg c = rt().cfg;
  unsigned long long so = send, ro = recv, by = bytes, ss = stride;
  if (fn != (const void *)alltoall_ring_kernel) {
    void *args[] = {&c, &op, &dtype, &so, &ro, &by, &rounds, &nsets, &ss, &device_barrier};
    return launch_collective(fn, grid, block, args, smem, 0);
  }
  A2aShare share = {op, 0, nsets, so, ro, ss, by, 0, 0};
  // a round's sources may be read before the round in front of it is over when
  // no round writes them: the send and receive buffers lie apart
  const size_t span = (size_t)(nsets - 1) * stride + (size_t)rt().npes * bytes;
  int ahead = send + span <= recv || recv + span <= send;
  void *args[] = {&c, &share, &rounds, &smem, &device_barrier, &ahead};
  return launch_collective(fn, grid, block, args, smem, 0);
}

int nvshmemx_op_alltoall(int op, int dtype, size_t send_off, size_t recv_off, size_t bytes, int rounds, int nsets,
                         size_t set_stride, int mode, int ctas_per_pe, float *out_ms) {
  int rc;
  const void *fn;
  dim3 grid, block;
  unsigned smem;
  if ((rc = alltoall_setup(op, dtype, send_off, recv_off, bytes, rounds, nsets, set_stride, mode, ctas_per_pe, &fn,
                           &grid, &block, &smem)))
    return rc;
  EventTimer t;
  t.start();
  if ((rc = alltoall_launch(fn, grid, block, smem, op, dtype, send_off, recv_off, bytes, rounds, nsets, set_stride, 1)))
    return rc;
  t.stop();
  float ms = t.ms();
  if (out_ms) *out_ms = ms;
  return check_cuda(cudaDeviceSynchronize(), "alltoall");
}

int nvshmemx_op_alltoall_host(int op, int dtype, size_t send_off, size_t recv_off, size_t bytes, int rounds,
                              int nsets, size_t set_stride, int mode, int ctas_per_pe, float *out_ms) {
  int rc;
  const void *fn;
  dim3 grid, block;
  unsigned smem;
  if ((rc = alltoall_setup(op, dtype, send_off, recv_off, bytes, rounds, nsets, set_stride, mode, ctas_per_pe, &fn,
                           &grid, &block, &smem)))
    return rc;
  EventTimer t;
  t.start();
  for (int rd = 0; rd < rounds; ++rd) {
    const size_t set = (size_t)(rd % nsets) * set_stride;
    if ((rc = alltoall_launch(fn, grid, block, smem, op, dtype, send_off + set, recv_off + set, bytes, 1, 1, 0, 0)))
      return rc;
    nvshmem_barrier_all();
    if ((rc = last_launch("alltoall_host round"))) return rc;
  }
  t.stop();
  float ms = t.ms();
  if (out_ms) *out_ms = ms;
  return check_cuda(cudaDeviceSynchronize(), "alltoall_host");
}

// ctas_per_pe 0: NVSHMEM_CTAS_PER_PE if set, else as many CTAs per PE as stay
// co-resident (the exchange is latency-bound, so more warps in flight help).
static int halo_check(int px, int py, int pz, int n, size_t block_off, size_t ghost_off, size_t sig_off, int iters,
                      int *ctas_per_pe) {
  int rc;
  if ((rc = need_collective())) return rc;
  const Runtime &r = rt();
  if (*ctas_per_pe == 0) *ctas_per_pe = default_ctas_per_pe(max_ctas_per_pe((const void *)halo_kernel, 256, halo_smem(n)));
  if (px < 1 || py < 1 || pz < 1 || px * py * pz != r.npes || n < 1 || iters < 1 || *ctas_per_pe < 1)
    return fail(NVSHMEMX_ERR_INVALID, "halo: grid %dx%dx%d does not match %d PEs", px, py, pz, r.npes);
  const size_t nn = (size_t)n;
  size_t face = 0, block = 0, ghosts = 0;
  if (!mul_ok(nn * 8, nn, &face) || !mul_ok(face, nn, &block) || !mul_ok(face, 6, &ghosts) ||
      !range_ok(block_off, block, r.heap_bytes) || !range_ok(ghost_off, ghosts, r.heap_bytes) ||
      !range_ok(sig_off, 24, r.heap_bytes) || (block_off | ghost_off) % 16 || sig_off % 4)
    return fail(NVSHMEMX_ERR_INVALID, "halo: buffers exceed the heap or are misaligned");
  return 0;
}

int nvshmemx_op_halo(int px, int py, int pz, int n, size_t block_off, size_t ghost_off, size_t sig_off, int iters,
                     int ctas_per_pe, float *out_ms) {
  int rc;
  if ((rc = halo_check(px, py, pz, n, block_off, ghost_off, sig_off, iters, &ctas_per_pe))) return rc;
  Cfg c = rt().cfg;
  unsigned long long bo = block_off, go = ghost_off, so = sig_off;
  int it0 = 0, device_barrier = 1;
  void *args[] = {&c, &px, &py, &pz, &n, &bo, &go, &so, &iters, &it0, &device_barrier};
  EventTimer t;
  t.start();
  if ((rc = launch_collective((const void *)halo_kernel, dim3(ctas_per_pe), dim3(256), args, halo_smem(n), 0))) return rc;
  t.stop();
  float ms = t.ms();
  if (out_ms) *out_ms = ms;
  return check_cuda(cudaDeviceSynchronize(), "halo");
}

int nvshmemx_op_halo_offload(int px, int py, int pz, int n, size_t block_off, size_t ghost_off, size_t sig_off,
                             int iters, int ctas_per_pe, float *out_ms) {
  int rc;
  if ((rc = halo_check(px, py, pz, n, block_off, ghost_off, sig_off, iters, &ctas_per_pe))) return rc;
  Cfg c = rt().cfg;
  unsigned long long bo = block_off, go = ghost_off, so = sig_off;
  int one = 1, device_barrier = 0;
  EventTimer t;
  t.start();
  for (int it = 0; it < iters; ++it) {
    void *args[] = {&c, &px, &py, &pz, &n, &bo, &go, &so, &one, &it, &device_barrier};
    if ((rc = launch_collective((const void *)halo_kernel, dim3(ctas_per_pe), dim3(256), args, halo_smem(n), 0))) return rc;
    nvshmem_barrier_all_offload();
    if ((rc = last_launch("halo_offload barrier"))) return rc;
  }
  t.stop();
  float ms = t.ms();
  if (out_ms) *out_ms = ms;
  return check_cuda(cudaDeviceSynchronize(), "halo_offload");
}

int nvshmemx_op_strided_read(size_t off, size_t set_off, int nsets, size_t rows, size_t stride, int ctas_per_pe,
                             int iters, float *out_ms) {
  int rc;
  if ((rc = need_started())) return rc;
  const Runtime &r = rt();
  size_t span = 0, last = 0;
  if (nsets < 1 || ctas_per_pe < 1 || iters < 1 || rows < 1 || stride < 8 || (off | set_off | stride) % 8 ||
      !mul_ok(rows - 1, stride, &span) || !mul_ok((size_t)(nsets - 1), set_off, &last) ||
      span > r.heap_bytes ||  // so that span + 8 cannot wrap
      !range_ok(last, span + 8, r.heap_bytes) || !range_ok(off, last + span + 8, r.heap_bytes))
    return fail(NVSHMEMX_ERR_INVALID, "strided_read: bad arguments or elements outside the heap");
  unsigned long long *sink = (unsigned long long *)g_out_buf.get(64);
  if (!sink) return fail(NVSHMEMX_ERR_NOMEM, "strided_read scratch");
  EventTimer t;
  t.start();
  for (int i = 0; i < iters; ++i)
    strided_read_kernel<<<dim3(ctas_per_pe, r.npes), 256>>>(r.cfg, off, set_off, nsets, rows, stride, sink);
  t.stop();
  if ((rc = last_launch("strided_read"))) return rc;
  float ms = t.ms();
  if (out_ms) *out_ms = ms;
  return check_cuda(cudaDeviceSynchronize(), "strided_read");
}

int nvshmemx_op_wait_test(size_t flag_off, int value, long long timeout_ns, int *out_status) {
  int rc;
  if ((rc = need_collective())) return rc;
  const Runtime &r = rt();
  if (!range_ok(flag_off, 4, r.heap_bytes) || flag_off % 4)
    return fail(NVSHMEMX_ERR_INVALID, "wait_test: bad flag offset");
  int *d = (int *)g_out_buf.get(64);
  if (!d) return fail(NVSHMEMX_ERR_NOMEM, "wait_test scratch");
  cudaMemset(d, 0, 4);
  wait_test_kernel<<<1, 32>>>(r.cfg, (int *)(r.arena + flag_off), value, timeout_ns, d);
  if ((rc = last_launch("wait_test"))) return rc;
  return check_cuda(cudaMemcpy(out_status, d, 4, cudaMemcpyDeviceToHost), "wait_test result");
}

int nvshmemx_op_barrier_fault_test(int skip_pe, long long timeout_ns, int *out_status) {
  int rc;
  if ((rc = need_collective())) return rc;
  const Runtime &r = rt();
  if (skip_pe < 0 || skip_pe >= r.npes || timeout_ns <= 0) return fail(NVSHMEMX_ERR_INVALID, "barrier_fault_test");
  int *d = (int *)g_out_buf.get(64);
  if (!d) return fail(NVSHMEMX_ERR_NOMEM, "barrier_fault_test scratch");
  cudaMemset(d, 0, 4);
  Cfg c = r.cfg;
  c.wait_timeout_ns = timeout_ns;
  void *args[] = {&c, &skip_pe, &d};
  if ((rc = launch_collective((const void *)barrier_fault_kernel, dim3(1), dim3(32), args, 0, 0))) return rc;
  if ((rc = check_cuda(cudaDeviceSynchronize(), "barrier_fault_test"))) return rc;
  return check_cuda(cudaMemcpy(out_status, d, 4, cudaMemcpyDeviceToHost), "barrier_fault_test result");
}

}  // extern "C"

