// Carries out lists of requests with the public device calls of
// nvshmem_device.h and nvshmemx.h, the way an application's kernels call them.
//
//   device_calls IN OUT
//
// IN: npes and the number of lists (int32), the heap's bytes (uint64), every
// PE's heap; then for each list its form, lane mask, count and operand (int32)
// and the requests (nvshmemx_request).  OUT: every PE's heap after the last
// list.  The lists run one after the other.
//
// Forms: 0 one thread per request, the lanes of the mask in every warp; 1 warp,
// 2 CTA, 3 CTA through the TMA ring.  Operand: where the local side of a put or
// get lies: 0 the heap, 1 an array of the thread's own, 2 shared memory (a part
// for each thread), 3 shared memory (one source for all requests); forms 1 to 3
// take 0 and 3.
#include <cuda_runtime.h>
#include <stdio.h>
#include <stdlib.h>

#include <vector>

#include "nvshmem.h"
#include "nvshmem_device.h"
#include "nvshmemx.h"
#include "nvshmemx_ops.h"

static const int kWords = 68;        // of a thread's own array
static const int kSource = 24 << 10;  // bytes of the source for all threads
static const int kRing = 20 << 10;

__device__ void call(const nvshmemx_request &r, void *sym, void *near, bool put) {
  const int pe = put ? r.dst_pe : r.src_pe;
  if (r.dtype == NVSHMEMX_DT_INT) {
    if (put) nvshmem_int_put((int *)sym, (int *)near, r.bytes / 4, pe);
    else nvshmem_int_get((int *)near, (int *)sym, r.bytes / 4, pe);
  } else if (r.dtype == NVSHMEMX_DT_FLOAT) {
    if (put) nvshmem_float_put((float *)sym, (float *)near, r.bytes / 4, pe);
    else nvshmem_float_get((float *)near, (float *)sym, r.bytes / 4, pe);
  } else {
    if (put) nvshmem_double_put((double *)sym, (double *)near, r.bytes / 8, pe);
    else nvshmem_double_get((double *)near, (double *)sym, r.bytes / 8, pe);
  }
}

__device__ void copy_words(int *dst, const int *src, unsigned bytes) {
  for (unsigned i = 0; i < bytes / 4; ++i) dst[i] = src[i];
}

// The first request's source in shared memory, by all threads.
__device__ void load_source(char *shared, char *arena, const nvshmemx_request &r) {
  const char *src = (const char *)nvshmemx_ptr(arena + r.src_off, r.src_pe);
  for (unsigned i = threadIdx.x; i < r.bytes; i += blockDim.x) shared[i] = src[i];
  __syncthreads();
}

__global__ void by_thread(char *arena, const nvshmemx_request *reqs, int n, unsigned lanes, int operand) {
  __shared__ __align__(16) char shared[kSource];
  __align__(16) int own[kWords];
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const int k = (int)(blockIdx.x * (blockDim.x >> 5) + warp) * __popc(lanes) + __popc(lanes & ((1u << lane) - 1u));
  if (operand == 3) load_source(shared, arena, reqs[0]);
  if ((lanes >> lane & 1u) && k < n) {
    const nvshmemx_request r = reqs[k];
    const bool put = r.op == NVSHMEMX_REQ_PUT;
    char *sym = arena + (put ? r.dst_off : r.src_off);
    char *near = (char *)nvshmemx_ptr(arena + (put ? r.src_off : r.dst_off), put ? r.src_pe : r.dst_pe);
    if (operand == 0) {
      call(r, sym, near, put);
    } else if (operand == 3) {
      call(r, sym, shared, put);
    } else {
      int *at = operand == 1 ? own : (int *)shared + threadIdx.x * kWords;
      at += (r.src_off >> 2) & 3;
      if (put) copy_words(at, (const int *)near, r.bytes);
      call(r, sym, at, put);
      if (!put) copy_words((int *)near, at, r.bytes);
    }
  }
  __syncwarp();
}

__global__ void by_group(char *arena, const nvshmemx_request *reqs, int n, int form, int operand) {
  extern __shared__ __align__(128) char ring[];
  __shared__ __align__(16) char shared[kSource];
  if (operand == 3) load_source(shared, arena, reqs[0]);
  const int k = form == 1 ? (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5) : (int)blockIdx.x;
  if (k >= n) return;
  const nvshmemx_request r = reqs[k];
  const bool put = r.op == NVSHMEMX_REQ_PUT;
  char *sym = arena + (put ? r.dst_off : r.src_off);
  void *near = operand == 3 ? shared : nvshmemx_ptr(arena + (put ? r.src_off : r.dst_off), put ? r.src_pe : r.dst_pe);
  const int pe = put ? r.dst_pe : r.src_pe;
  if (form == 3) {
    if (put) nvshmemx_putmem_bulk_block(sym, near, r.bytes, pe, ring, kRing);
    else nvshmemx_getmem_bulk_block(near, sym, r.bytes, pe, ring, kRing);
    return;
  }
#define TYPED(Name, Type)                                                                                   \
  if (form == 1) {                                                                                          \
    if (put) nvshmemx_##Name##_put_warp((Type *)sym, (Type *)near, (int)(r.bytes / sizeof(Type)), pe);      \
    else nvshmemx_##Name##_get_warp((Type *)near, (Type *)sym, (int)(r.bytes / sizeof(Type)), pe);          \
  } else {                                                                                                  \
    if (put) nvshmemx_##Name##_put_block((Type *)sym, (Type *)near, (int)(r.bytes / sizeof(Type)), pe);     \
    else nvshmemx_##Name##_get_block((Type *)near, (Type *)sym, (int)(r.bytes / sizeof(Type)), pe);         \
  }
  if (r.dtype == NVSHMEMX_DT_INT) {
    TYPED(int, int)
  } else if (r.dtype == NVSHMEMX_DT_FLOAT) {
    TYPED(float, float)
  } else {
    TYPED(double, double)
  }
}

#define CHECK(call)                                              \
  do {                                                           \
    const cudaError_t e = (call);                                \
    if (e != cudaSuccess) {                                      \
      fprintf(stderr, "%s: %s\n", #call, cudaGetErrorString(e)); \
      return 3;                                                  \
    }                                                            \
  } while (0)

int main(int argc, char **argv) {
  if (argc < 3) return 2;
  FILE *f = fopen(argv[1], "rb");
  if (!f) return 2;
  int head[2];
  unsigned long long heap = 0;
  if (fread(head, sizeof head, 1, f) != 1 || fread(&heap, sizeof heap, 1, f) != 1) return 2;
  const int npes = head[0], lists = head[1];
  nvshmemx_set_error_mode(NVSHMEMX_ERRORS_RETURN);
  if (nvshmemx_init_attr(npes, heap)) return 4;
  char *arena = (char *)nvshmemx_arena_base();
  std::vector<char> h(heap);
  for (int pe = 0; pe < npes; ++pe) {
    if (fread(h.data(), 1, heap, f) != heap) return 2;
    CHECK(cudaMemcpy(nvshmem_ptr(arena, pe), h.data(), heap, cudaMemcpyHostToDevice));
  }
  for (int l = 0; l < lists; ++l) {
    int s[4];  // form, lanes, requests, operand
    if (fread(s, sizeof s, 1, f) != 1 || s[2] < 1) return 2;
    std::vector<nvshmemx_request> r(s[2]);
    if (fread(r.data(), sizeof(nvshmemx_request), s[2], f) != (size_t)s[2]) return 2;
    nvshmemx_request *d = nullptr;
    CHECK(cudaMalloc(&d, s[2] * sizeof *d));
    CHECK(cudaMemcpy(d, r.data(), s[2] * sizeof *d, cudaMemcpyHostToDevice));
    if (s[0] == 0) {
      const int per = __builtin_popcount((unsigned)s[1]) * 2;  // of a CTA of two warps
      by_thread<<<(s[2] + per - 1) / per, 64>>>(arena, d, s[2], (unsigned)s[1], s[3]);
    } else {
      by_group<<<s[0] == 1 ? (s[2] + 3) / 4 : s[2], 128, s[0] == 3 ? kRing : 0>>>(arena, d, s[2], s[0], s[3]);
    }
    CHECK(cudaGetLastError());
    CHECK(cudaDeviceSynchronize());
    CHECK(cudaFree(d));
    if (nvshmemx_status()) return 5;
  }
  fclose(f);
  f = fopen(argv[2], "wb");
  if (!f) return 2;
  for (int pe = 0; pe < npes; ++pe) {
    CHECK(cudaMemcpy(h.data(), nvshmem_ptr(arena, pe), heap, cudaMemcpyDeviceToHost));
    fwrite(h.data(), 1, heap, f);
  }
  fclose(f);
  nvstop_pes();
  return 0;
}
