// mlp.cu -- the learned variant picker (nvshmemx_picker.h): an FP32 MLP
// 6 -> 64 -> 64 -> 64 -> 12 (ReLU) with this library's own forward, backward
// and Adam kernels, and the executor of the 12 transfer variants it chooses
// between.
//
// Kernel shape: a CTA of 256 threads per tile of 16 rows, weights and
// activations in shared memory.  Rows of 64 values lie 68 floats apart, so
// the 16-byte reads of eight lanes (eight weight rows, or one row's
// consecutive columns) fall into different banks.  The network is tiny (9,548
// parameters), so it is bound by latency: shared-memory reads within a tile
// (a 64 x 64 layer's weights are read once per row group) and
// what has to be exchanged between tiles.  It stays in FP32 on the CUDA
// cores: the tensor cores have no FP32 form, and a tile is 16 rows.
//
// Training is a chain of small steps, so it runs as one launch of one
// thread-block cluster (train_cluster_kernel): the weights stay in shared
// memory from step to step, the partial gradients are read by their owners
// through distributed shared memory, and a step costs two cluster barriers
// instead of three launches.  800 rows, batch 128: 75 us a step as a memset, a
// gradient kernel (64 threads per 32 rows) and an Adam kernel, 11 us now, half of
// it the tile and half the exchange of gradients and weights.
#include <cuda_runtime.h>
#include <math.h>
#include <string.h>

#include <algorithm>
#include <mutex>
#include <vector>

#include "batch.h"
#include "nvshmemx_picker.h"

namespace nvshm {

constexpr int NI = NVSHMEMX_PICKER_NIN, NH = NVSHMEMX_PICKER_HIDDEN, NO = NVSHMEMX_PICKER_VARIANTS;
constexpr int OFF_W1 = 0, OFF_B1 = OFF_W1 + NH * NI, OFF_W2 = OFF_B1 + NH, OFF_B2 = OFF_W2 + NH * NH,
              OFF_W3 = OFF_B2 + NH, OFF_B3 = OFF_W3 + NH * NH, OFF_W4 = OFF_B3 + NH, OFF_B4 = OFF_W4 + NO * NH,
              NPARAM = OFF_B4 + NO;
// The gradient in shared memory has the rows of W1 padded to 8, so that every
// group of four values is one 16-byte access there and in the network.
constexpr int NPAD = NPARAM + NH * 2;
__host__ __device__ constexpr int padded(int p) { return p < OFF_B1 ? (p / NI) * 8 + p % NI : p + NH * 2; }
static_assert(NPAD % 4 == 0 && padded(OFF_W2) % 4 == 0 && padded(OFF_W4) % 4 == 0, "16-byte groups");
constexpr int kThreads = 256;
constexpr int kRows = 16;       // rows of a tile of the grid kernels
constexpr int kTrainRows = 8;   // rows of a CTA's tile in a training cluster
constexpr int LD = NH + 4;  // floats between rows of 64
constexpr int LDX = 12;     // floats between rows of 6 (padded with zeros to 8)
static_assert(NI <= 8 && NH == 64 && NO == 12, "the thread mappings below are for these sizes");

// Shared memory in floats.
template <int R>
struct Net {
  float W1[NH * LDX], W2[NH * LD], W3[NH * LD], W4[NO * LD];
  float b1[NH], b2[NH], b3[NH], b4[16];
  float X[R * LDX];
  float A1[R * LD], A2[R * LD], A3[R * LD];
  float O[R * 16];  // outputs, then dL/dO
};
template <int R>
struct NetGrad : Net<R> {
  float Y[R * NO], M[R * NO];
  float D1[R * LD], D2[R * LD], D3[R * LD];  // dL/dz of the hidden layers
  float G[NPAD];                             // gradient (padded order)
  float loss;
};

// Where the value at padded position q lies in the net's shared memory, in
// floats from its start.
__host__ __device__ __forceinline__ int net_slot(int q) {
  constexpr int sW2 = NH * LDX, sW3 = sW2 + NH * LD, sW4 = sW3 + NH * LD, sb1 = sW4 + NO * LD, sb2 = sb1 + NH,
                sb3 = sb2 + NH, sb4 = sb3 + NH;
  if (q < NH * 8) return (q / 8) * LDX + q % 8;
  if (q < padded(OFF_W2)) return sb1 + (q - padded(OFF_B1));
  if (q < padded(OFF_B2)) return sW2 + ((q - padded(OFF_W2)) / NH) * LD + (q - padded(OFF_W2)) % NH;
  if (q < padded(OFF_W3)) return sb2 + (q - padded(OFF_B2));
  if (q < padded(OFF_B3)) return sW3 + ((q - padded(OFF_W3)) / NH) * LD + (q - padded(OFF_W3)) % NH;
  if (q < padded(OFF_W4)) return sb3 + (q - padded(OFF_B3));
  if (q < padded(OFF_B4)) return sW4 + ((q - padded(OFF_W4)) / NH) * LD + (q - padded(OFF_W4)) % NH;
  return sb4 + (q - padded(OFF_B4));
}

__device__ __forceinline__ float4 ld4(const float *p) { return *reinterpret_cast<const float4 *>(p); }

template <int R>
__device__ __forceinline__ void load_net(Net<R> &s, const float *__restrict__ P) {
  const int t = threadIdx.x;
  for (int i = t; i < NH * LDX; i += kThreads) s.W1[i] = 0.f;
  for (int i = t; i < R * LDX; i += kThreads) s.X[i] = 0.f;
  __syncthreads();
  float *base = s.W1;
  for (int p = t; p < NPARAM; p += kThreads) base[net_slot(padded(p))] = P[p];
}

// out[r][j] = relu(b[j] + sum_k W[j][k] in[r][k]): a warp takes 32 outputs
// (one per lane) of R / 4 rows.
template <int R, int K4>
__device__ __forceinline__ void forward_layer(const float *W, int ldw, const float *b, const float *in, int ldin,
                                              float *out) {
  constexpr int N = R / 4;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int j = (w & 1) * 32 + lane, r0 = (w >> 1) * N;
  float a[N];
#pragma unroll
  for (int r = 0; r < N; ++r) a[r] = b[j];
#pragma unroll 8
  for (int k = 0; k < K4; ++k) {
    const float4 x = ld4(W + j * ldw + 4 * k);
#pragma unroll
    for (int r = 0; r < N; ++r) {
      const float4 y = ld4(in + (r0 + r) * ldin + 4 * k);
      a[r] += x.x * y.x;
      a[r] += x.y * y.y;
      a[r] += x.z * y.z;
      a[r] += x.w * y.w;
    }
  }
#pragma unroll
  for (int r = 0; r < N; ++r) out[(r0 + r) * LD + j] = fmaxf(a[r], 0.f);
}

// The outputs of a warp's R / 8 rows, one per lane.
template <int R>
__device__ __forceinline__ bool output_of(int *row, int *k) {
  const int lane = threadIdx.x & 31;
  *row = (threadIdx.x >> 5) * (R / 8) + lane / NO;
  *k = lane % NO;
  return lane < R / 8 * NO;
}
template <int R>
__device__ __forceinline__ float output_value(const Net<R> &s, int row, int k) {
  float a = s.b4[k];
#pragma unroll 8
  for (int i = 0; i < NH; i += 4) {
    const float4 x = ld4(s.W4 + k * LD + i), y = ld4(s.A3 + row * LD + i);
    a += x.x * y.x;
    a += x.y * y.y;
    a += x.z * y.z;
    a += x.w * y.w;
  }
  return a;
}

// Hidden layers of the tile in s.X; ends with a barrier.
template <int R>
__device__ __forceinline__ void forward_hidden(Net<R> &s) {
  forward_layer<R, 2>(s.W1, LDX, s.b1, s.X, LDX, s.A1);
  __syncthreads();
  forward_layer<R, 16>(s.W2, LD, s.b2, s.A1, LD, s.A2);
  __syncthreads();
  forward_layer<R, 16>(s.W3, LD, s.b3, s.A2, LD, s.A3);
  __syncthreads();
}

__device__ __forceinline__ void put_grad(float *g, float v, bool first) { *g = first ? v : *g + v; }
__device__ __forceinline__ void put_grad4(float *g, const float *v, bool first) {
  float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
  if (!first) o = ld4(g);
  *reinterpret_cast<float4 *>(g) = make_float4(o.x + v[0], o.y + v[1], o.z + v[2], o.w + v[3]);
}

// G += D^T A (64 x 64) and its bias gradient: a 4 x 4 block per thread.
template <int R>
__device__ __forceinline__ void weight_grad(const float *D, const float *A, float *gw, float *gb, bool first) {
  const int i4 = (threadIdx.x & 15) * 4, j4 = (threadIdx.x >> 4) * 4;
  float g[4][4] = {}, sb[4] = {};
#pragma unroll 4
  for (int r = 0; r < R; ++r) {
    const float4 d = ld4(D + r * LD + j4), a = ld4(A + r * LD + i4);
    const float dv[4] = {d.x, d.y, d.z, d.w}, av[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      sb[j] += dv[j];
#pragma unroll
      for (int i = 0; i < 4; ++i) g[j][i] += dv[j] * av[i];
    }
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) put_grad4(gw + (j4 + j) * NH + i4, g[j], first);
  if (i4 == 0) put_grad4(gb + j4, sb, first);
}

// out = (D W) where A > 0: R / 8 rows per warp, half of the sum per half
// warp, four columns per lane.
template <int R>
__device__ __forceinline__ void input_grad(const float *D, const float *W, const float *A, float *out) {
  constexpr int N = R / 8;
  const int lane = threadIdx.x & 31, i4 = (lane & 15) * 4, half = lane >> 4, r0 = (threadIdx.x >> 5) * N;
  float a[N][4] = {};
#pragma unroll 4
  for (int j = half * 32; j < half * 32 + 32; j += 4) {
    float e[N][4];
#pragma unroll
    for (int r = 0; r < N; ++r) {
      const float4 d = ld4(D + (r0 + r) * LD + j);
      e[r][0] = d.x, e[r][1] = d.y, e[r][2] = d.z, e[r][3] = d.w;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const float4 w = ld4(W + (j + u) * LD + i4);
      const float wv[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
      for (int r = 0; r < N; ++r)
#pragma unroll
        for (int i = 0; i < 4; ++i) a[r][i] += e[r][u] * wv[i];
    }
  }
#pragma unroll
  for (int r = 0; r < N; ++r)
#pragma unroll
    for (int i = 0; i < 4; ++i) a[r][i] += __shfl_xor_sync(0xffffffffu, a[r][i], 16);
  // both halves hold every sum: of two rows each writes one, of one row the
  // first writes it
  const int r = N == 2 ? half : 0;
  if (N == 2 || half == 0) {
    const float *m = A + (r0 + r) * LD + i4;
    float v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = m[i] > 0.f ? a[N == 2 && half ? N - 1 : 0][i] : 0.f;
    *reinterpret_cast<float4 *>(out + (r0 + r) * LD + i4) = make_float4(v[0], v[1], v[2], v[3]);
  }
}

// Forward and backward of the tile in s.X, s.Y, s.M (`rows` valid rows):
// adds its loss to s.loss and its gradient to s.G (`first`: replaces it).
// Begins and ends with every thread past a barrier for the inputs / not yet
// past one for s.G.
template <int R>
__device__ __forceinline__ void tile_gradient(NetGrad<R> &s, int rows, float inv_count, bool first) {
  const int t = threadIdx.x;
  forward_hidden(s);
  int row, k;
  float l = 0.f;
  if (output_of<R>(&row, &k)) {
    float d = 0.f;
    if (row < rows) {
      const float m = s.M[row * NO + k], diff = output_value(s, row, k) - s.Y[row * NO + k];
      d = 2.f * m * diff * inv_count;
      l = m * diff * diff;
    }
    s.O[row * 16 + k] = d;
  }
  for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
  if ((t & 31) == 0) atomicAdd(&s.loss, l * inv_count);
  __syncthreads();
  // layer 4: four columns of one output per thread; the output's bias
  if (t < NO * 16) {
    const int q = t >> 4, i4 = (t & 15) * 4;
    float g[4] = {};
#pragma unroll 4
    for (int r = 0; r < R; ++r) {
      const float d = s.O[r * 16 + q];
      const float4 a = ld4(s.A3 + r * LD + i4);
      g[0] += d * a.x;
      g[1] += d * a.y;
      g[2] += d * a.z;
      g[3] += d * a.w;
    }
    put_grad4(s.G + padded(OFF_W4) + q * NH + i4, g, first);
  } else if (t < NO * 16 + NO) {
    float g = 0.f;
    for (int r = 0; r < R; ++r) g += s.O[r * 16 + (t - NO * 16)];
    put_grad(s.G + padded(OFF_B4) + (t - NO * 16), g, first);
  }
  if (t < R * 16) {
    const int r = t >> 4, i4 = (t & 15) * 4;
    float a[4] = {};
#pragma unroll
    for (int q = 0; q < NO; ++q) {
      const float d = s.O[r * 16 + q];
      const float4 w = ld4(s.W4 + q * LD + i4);
      a[0] += d * w.x;
      a[1] += d * w.y;
      a[2] += d * w.z;
      a[3] += d * w.w;
    }
    const float4 m = ld4(s.A3 + r * LD + i4);
    *reinterpret_cast<float4 *>(s.D3 + r * LD + i4) = make_float4(
        m.x > 0.f ? a[0] : 0.f, m.y > 0.f ? a[1] : 0.f, m.z > 0.f ? a[2] : 0.f, m.w > 0.f ? a[3] : 0.f);
  }
  __syncthreads();
  weight_grad<R>(s.D3, s.A2, s.G + padded(OFF_W3), s.G + padded(OFF_B3), first);
  input_grad<R>(s.D3, s.W3, s.A2, s.D2);
  __syncthreads();
  weight_grad<R>(s.D2, s.A1, s.G + padded(OFF_W2), s.G + padded(OFF_B2), first);
  input_grad<R>(s.D2, s.W2, s.A1, s.D1);
  __syncthreads();
  // layer 1: one output's inputs f and f + 4 per thread; the bias where
  // there is no f + 4 within the six
  {
    const int j = t & 63, f = t >> 6;
    float g0 = 0.f, g1 = 0.f, sb = 0.f;
    for (int r = 0; r < R; ++r) {
      const float d = s.D1[r * LD + j];
      g0 += d * s.X[r * LDX + f];
      if (f + 4 < NI) g1 += d * s.X[r * LDX + f + 4];
      sb += d;
    }
    put_grad(s.G + j * 8 + f, g0, first);
    if (f + 4 < NI) put_grad(s.G + j * 8 + f + 4, g1, first);
    if (f == 3) put_grad(s.G + padded(OFF_B1) + j, sb, first);
  }
}

__device__ __forceinline__ float adam_step(float p, float g, float *m, float *v, float lr, float c1, float c2) {
  const float mi = 0.9f * *m + 0.1f * g;
  const float vi = 0.999f * *v + 0.001f * g * g;
  *m = mi;
  *v = vi;
  return p - lr * (mi / c1) / (sqrtf(vi / c2) + 1e-8f);
}

// Y[n][12] of X[n][6], 16 rows at a time per CTA.
__global__ void __launch_bounds__(kThreads) mlp_forward_kernel(const float *__restrict__ P, const float *__restrict__ X,
                                                               int n, const float *__restrict__ norm,
                                                               float *__restrict__ out) {
  extern __shared__ __align__(16) char sm[];
  Net<kRows> &s = *reinterpret_cast<Net<kRows> *>(sm);
  load_net(s, P);
  for (long long s0 = (long long)blockIdx.x * kRows; s0 < n; s0 += (long long)gridDim.x * kRows) {
    __syncthreads();
    if (threadIdx.x < kRows * NI) {
      const int r = threadIdx.x / NI, f = threadIdx.x % NI;
      s.X[r * LDX + f] = s0 + r < n ? (X[(s0 + r) * NI + f] - norm[f]) / norm[NI + f] : 0.f;
    }
    __syncthreads();
    forward_hidden(s);
    int row, k;
    if (output_of<kRows>(&row, &k) && s0 + row < n) out[(s0 + row) * NO + k] = output_value(s, row, k);
  }
}

// Loss and gradient of n rows (rows idx[0..n) when idx is given), added to
// *loss and grad: every CTA sums its tiles in shared memory and adds them once.
__global__ void __launch_bounds__(kThreads) mlp_grad_kernel(const float *__restrict__ P, const float *__restrict__ X,
                                                            const float *__restrict__ Y, const float *__restrict__ M,
                                                            const int *__restrict__ idx, int n,
                                                            const float *__restrict__ norm, float inv_count,
                                                            float *__restrict__ grad, float *__restrict__ loss) {
  extern __shared__ __align__(16) char sm[];
  NetGrad<kRows> &s = *reinterpret_cast<NetGrad<kRows> *>(sm);
  const int t = threadIdx.x;
  load_net(s, P);
  if (t == 0) s.loss = 0.f;
  bool first = true;
  for (long long s0 = (long long)blockIdx.x * kRows; s0 < n; s0 += (long long)gridDim.x * kRows) {
    const int rows = n - s0 < kRows ? (int)(n - s0) : kRows;
    __syncthreads();
    if (t < kRows * NO) {
      const int r = t / NO, k = t % NO;
      const long long g = r < rows ? (idx ? idx[s0 + r] : s0 + r) : 0;
      s.Y[t] = r < rows ? Y[g * NO + k] : 0.f;
      s.M[t] = r < rows ? M[g * NO + k] : 0.f;
    }
    if (t < kRows * NI) {
      const int r = t / NI, f = t % NI;
      const long long g = r < rows ? (idx ? idx[s0 + r] : s0 + r) : 0;
      s.X[r * LDX + f] = r < rows ? (X[g * NI + f] - norm[f]) / norm[NI + f] : 0.f;
    }
    __syncthreads();
    tile_gradient(s, rows, inv_count, first);
    first = false;
  }
  __syncthreads();
  if (first) return;
  for (int p = t; p < NPARAM; p += kThreads) atomicAdd(&grad[p], s.G[padded(p)]);
  if (t == 0) atomicAdd(loss, s.loss);
}

__global__ void adam_kernel(float *P, const float *G, float *m, float *v, int n, float lr, float c1, float c2) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) P[i] = adam_step(P[i], G[i], m + i, v + i, lr, c1, c2);
}

// ------------------------------------------------ training in one cluster
// One tile of a training run: up to 8 rows for each CTA of the cluster.
struct TrainTile {
  int first, rows;   // rows idx[first .. first + rows)
  float inv_count;   // 1 / mask sum of its batch
  float c1, c2;      // Adam's bias corrections of its batch's step
  int flags;         // kFirst: begins a batch; kLast: ends it
  int epoch;
  int pad;
};
enum { kFirst = 1, kLast = 2 };
constexpr int kCluster = 16;                                          // CTAs (8 took 14.4 us a step, 16 12.0 us; 11.0 with 16-byte exchanges)
constexpr int kTileRows = kCluster * kTrainRows;                           // rows of a tile
constexpr int kOwned = (NPAD / 4 + kCluster - 1) / kCluster;          // 16-byte groups that a CTA updates,
static_assert(kOwned <= kThreads, "");                                // one of them per thread
// A batch of more rows is spread over more SMs than a cluster has.  Us a step in
// the cluster and as three spread-out launches: 256 rows 17.7 and 32.9, 384 24.1
// and 33.6, 512 30.6 and 34.0; 640 rows are another tile of some 6 us for the
// cluster, and 34.8 spread out.
constexpr int kClusterBatch = 512;

__device__ __forceinline__ unsigned peer_addr(const void *p, unsigned rank) {
  unsigned a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
  return a;
}
__device__ __forceinline__ float ld_peer(unsigned a) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ float4 ld_peer4(unsigned a) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(a)
               : "memory");
  return v;
}
__device__ __forceinline__ void st_peer4(unsigned a, float4 v) {
  asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
               : "memory");
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}

// Every CTA holds the whole network and takes 8 of a tile's 128 rows.  After
// a batch's last tile, CTA c sums the cluster's gradients of the 16-byte groups
// [c * kOwned, (c + 1) * kOwned) in rank order (so training is reproducible),
// updates those parameters (their moments stay in its registers) and writes
// the new values into every CTA's network.  The next tile's rows, and the row numbers
// of the one after, are fetched while a tile is computed.
__global__ void __launch_bounds__(kThreads) train_cluster_kernel(float *__restrict__ P, float *__restrict__ Am,
                                                                 float *__restrict__ Av, const float *__restrict__ X,
                                                                 const float *__restrict__ Y,
                                                                 const float *__restrict__ M,
                                                                 const int *__restrict__ idx,
                                                                 const TrainTile *__restrict__ tiles, int ntiles,
                                                                 const float *__restrict__ norm, float lr,
                                                                 float *__restrict__ losses) {
  extern __shared__ __align__(16) char sm[];
  NetGrad<kTrainRows> &s = *reinterpret_cast<NetGrad<kTrainRows> *>(sm);
  const int t = threadIdx.x, rank = blockIdx.x;
  load_net(s, P);
  if (t == 0) s.loss = 0.f;
  // this thread's group of parameters: padded positions q .. q + 3, and their
  // numbers (-1: padding, or no group)
  const int q = (rank * kOwned + t) * 4;
  const bool own = t < kOwned && q < NPAD;
  float p[4], m[4], v[4];
  int num[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    num[i] = !own ? -1 : q < NH * 8 ? ((q + i) % 8 < NI ? (q + i) / 8 * NI + (q + i) % 8 : -1) : q + i - NH * 2;
    p[i] = num[i] >= 0 ? P[num[i]] : 0.f;
    m[i] = num[i] >= 0 ? Am[num[i]] : 0.f;
    v[i] = num[i] >= 0 ? Av[num[i]] : 0.f;
  }
  const float *const g_at = s.G + (own ? q : 0), *const p_at = s.W1 + net_slot(own ? q : 0);
  if (t < NH * 2) s.G[t / 2 * 8 + NI + t % 2] = 0.f;  // the padding of W1's gradient
  // this thread's part of a tile: one output of one row, one input of one row
  const int yr = t / NO, yk = t % NO, xr = t / NI, xf = t % NI;
  const bool has_y = t < kTrainRows * NO, has_x = t < kTrainRows * NI;
  const float mean = has_x ? norm[xf] : 0.f, sd = has_x ? norm[NI + xf] : 1.f;
  auto row_of = [&](const TrainTile &d, int r) { return rank * kTrainRows + r < d.rows ? idx[d.first + rank * kTrainRows + r] : -1; };
  TrainTile cur = tiles[0], nxt = tiles[ntiles > 1 ? 1 : 0];
  int gy = has_y ? row_of(cur, yr) : -1, gx = has_x ? row_of(cur, xr) : -1;
  float y = gy >= 0 ? Y[(size_t)gy * NO + yk] : 0.f, mk = gy >= 0 ? M[(size_t)gy * NO + yk] : 0.f;
  float x = gx >= 0 ? X[(size_t)gx * NI + xf] : 0.f;
  int ny = has_y ? row_of(nxt, yr) : -1, nx = has_x ? row_of(nxt, xr) : -1;
  float epoch_loss = 0.f;  // rank 0, thread 0
  cluster_barrier();
  for (int i = 0; i < ntiles; ++i) {
    if (has_y) {
      s.Y[t] = y;
      s.M[t] = mk;
    }
    if (has_x) s.X[xr * LDX + xf] = gx >= 0 ? (x - mean) / sd : 0.f;
    __syncthreads();
    const TrainTile d = cur;
    const TrainTile after = tiles[i + 2 < ntiles ? i + 2 : ntiles - 1];
    y = ny >= 0 ? Y[(size_t)ny * NO + yk] : 0.f;
    mk = ny >= 0 ? M[(size_t)ny * NO + yk] : 0.f;
    x = nx >= 0 ? X[(size_t)nx * NI + xf] : 0.f;
    gx = nx;
    cur = nxt;
    nxt = after;
    ny = has_y ? row_of(after, yr) : -1;
    nx = has_x ? row_of(after, xr) : -1;
    int rows = d.rows - rank * kTrainRows;
    rows = rows < 0 ? 0 : (rows > kTrainRows ? kTrainRows : rows);
    tile_gradient(s, rows, d.inv_count, (d.flags & kFirst) != 0);
    if (!(d.flags & kLast)) {
      __syncthreads();
      continue;
    }
    cluster_barrier();  // every CTA's gradient and loss of the batch are there
    if (rank == 0 && t == 0) {
      float l = 0.f;
      for (unsigned r = 0; r < kCluster; ++r) l += ld_peer(peer_addr(&s.loss, r));
      epoch_loss += l;
      if (i + 1 == ntiles || cur.epoch != d.epoch) {
        losses[d.epoch] = epoch_loss;
        epoch_loss = 0.f;
      }
    }
    if (own) {
      float4 part[kCluster];
#pragma unroll
      for (unsigned r = 0; r < kCluster; ++r) part[r] = ld_peer4(peer_addr(g_at, r));
      float g[4] = {part[0].x, part[0].y, part[0].z, part[0].w};
#pragma unroll
      for (int r = 1; r < kCluster; ++r) {
        g[0] += part[r].x;
        g[1] += part[r].y;
        g[2] += part[r].z;
        g[3] += part[r].w;
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) p[k] = adam_step(p[k], g[k], &m[k], &v[k], lr, d.c1, d.c2);
#pragma unroll
      for (unsigned r = 0; r < kCluster; ++r) st_peer4(peer_addr(p_at, r), make_float4(p[0], p[1], p[2], p[3]));
    }
    cluster_barrier();  // the new weights are everywhere, nobody reads G or loss any more
    if (t == 0) s.loss = 0.f;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (num[i] >= 0) {
      P[num[i]] = p[i];
      Am[num[i]] = m[i];
      Av[num[i]] = v[i];
    }
  }
}

// Deterministic host RNG for initialisation and shuffles.
static unsigned long long mix64(unsigned long long x) {
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}

}  // namespace nvshm

using namespace nvshm;

// Memory of a network: its own arrays and kSlotWork bytes for the host arrays
// of a call.  The first kSlots networks of a device live in an array of the
// library (the device's allocator takes 0.3-0.6 ms to map a first block and
// as long to give it back, several times what training a table of 800
// classes for some epochs takes); further ones are allocated.
constexpr size_t pad256(size_t x) { return (x + 255) / 256 * 256; }
constexpr size_t kParBytes = pad256(NPARAM * 4), kNormBytes = pad256(2 * NI * 4);
constexpr size_t kNetBytes = 4 * kParBytes + kNormBytes + 256, kSlotWork = 256u << 10;
constexpr int kSlots = 2, kMaxDevices = 64;
static __device__ __align__(256) unsigned char g_mlp_slots[kSlots][kNetBytes + kSlotWork];
static std::mutex g_slot_mu;
static bool g_slot_used[kMaxDevices][kSlots];

// Takes a free slot of device `dev` (the current one): its number and address,
// or -1.
static int take_slot(int dev, char **p) {
  if (dev < 0 || dev >= kMaxDevices) return -1;
  std::lock_guard<std::mutex> lk(g_slot_mu);
  for (int k = 0; k < kSlots; ++k) {
    if (g_slot_used[dev][k]) continue;
    void *base = nullptr;
    if (cudaGetSymbolAddress(&base, g_mlp_slots) != cudaSuccess) {
      (void)cudaGetLastError();
      return -1;
    }
    g_slot_used[dev][k] = true;
    *p = (char *)base + k * (kNetBytes + kSlotWork);
    return k;
  }
  return -1;
}

static void give_slot(int dev, int k) {
  std::lock_guard<std::mutex> lk(g_slot_mu);
  g_slot_used[dev][k] = false;
}

struct nvshmemx_mlp {
  char *block = nullptr;  // everything below in one allocation
  float *P = nullptr, *norm = nullptr, *Am = nullptr, *Av = nullptr, *G = nullptr, *loss = nullptr;
  long long step = 0;
  int sms = 0;
  int cluster = -1;  // whether a training cluster fits the device (-1: not asked yet)
  int dev = 0, slot = -1;
  // Device copies of the host arrays of a call, kept between calls up to
  // kKeep bytes; a larger call allocates its own.  `mu` is held for the whole of
  // every call but destroy, so calls on one network from several threads run
  // one after the other.
  mutable std::mutex mu;
  char *work = nullptr;
  size_t work_bytes = 0;
  bool work_own = false;  // allocated (else part of a slot)
};

static const size_t kKeep = 16u << 20;

// Device memory for one call, held under the network's lock.
struct Work {
  std::lock_guard<std::mutex> lk;
  char *p = nullptr;
  char *own = nullptr;
  explicit Work(nvshmemx_mlp *m) : lk(m->mu) {}
  ~Work() {
    if (own) cudaFree(own);
  }
  int get(nvshmemx_mlp *m, size_t bytes) {
    if (bytes > kKeep) {
      if (cudaMalloc(&own, bytes) != cudaSuccess) return fail(NVSHMEMX_ERR_NOMEM, "mlp: cudaMalloc");
      p = own;
      return 0;
    }
    if (bytes > m->work_bytes) {
      size_t want = 64u << 10;
      while (want < bytes) want *= 2;
      if (m->work_own) cudaFree(m->work);
      m->work = nullptr;
      m->work_bytes = 0;
      m->work_own = false;
      if (cudaMalloc(&m->work, want) != cudaSuccess) return fail(NVSHMEMX_ERR_NOMEM, "mlp: cudaMalloc");
      m->work_own = true;
      m->work_bytes = want;
    }
    p = m->work;
    return 0;
  }
};

static int upload(void *d, const void *h, size_t bytes) {
  return bytes ? check_cuda(cudaMemcpy(d, h, bytes, cudaMemcpyHostToDevice), "mlp: upload") : 0;
}

static int launch_forward(nvshmemx_mlp *m, const float *dX, int n, float *dY) {
  cudaFuncSetAttribute(mlp_forward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Net<kRows>));
  const int blocks = std::min((n - 1) / kRows + 1, 3 * m->sms);
  mlp_forward_kernel<<<blocks, kThreads, sizeof(Net<kRows>)>>>(m->P, dX, n, m->norm, dY);
  return check_cuda(cudaGetLastError(), "mlp forward kernel");
}

static int launch_grad(nvshmemx_mlp *m, const float *dX, const float *dY, const float *dM, const int *didx, int n,
                       float inv_count) {
  cudaFuncSetAttribute(mlp_grad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(NetGrad<kRows>));
  const int blocks = std::min((n - 1) / kRows + 1, m->sms);
  mlp_grad_kernel<<<blocks, kThreads, sizeof(NetGrad<kRows>)>>>(m->P, dX, dY, dM, didx, n, m->norm, inv_count, m->G, m->loss);
  return check_cuda(cudaGetLastError(), "mlp gradient kernel");
}

// The launch of the training cluster (`attr`: room for its attribute).
static cudaLaunchConfig_t train_launch(cudaLaunchAttribute *attr) {
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3(kCluster);
  lc.blockDim = dim3(kThreads);
  lc.dynamicSmemBytes = sizeof(NetGrad<kTrainRows>);
  attr->id = cudaLaunchAttributeClusterDimension;
  attr->val.clusterDim.x = kCluster;
  attr->val.clusterDim.y = 1;
  attr->val.clusterDim.z = 1;
  lc.attrs = attr;
  lc.numAttrs = 1;
  return lc;
}

// Whether the device runs a cluster of this size (16 CTAs are more than every
// device promises); asked once per network.
static bool cluster_fits(nvshmemx_mlp *m) {
  if (m->cluster < 0) {
    cudaLaunchAttribute attr;
    cudaLaunchConfig_t lc = train_launch(&attr);
    int clusters = 0;
    const bool ok =
        cudaFuncSetAttribute(train_cluster_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)lc.dynamicSmemBytes) == cudaSuccess &&
        cudaFuncSetAttribute(train_cluster_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
        cudaOccupancyMaxActiveClusters(&clusters, train_cluster_kernel, &lc) == cudaSuccess && clusters > 0;
    if (!ok) (void)cudaGetLastError();
    m->cluster = ok ? 1 : 0;
  }
  return m->cluster == 1;
}

static int launch_train(nvshmemx_mlp *m, const float *dX, const float *dY, const float *dM, const int *didx,
                        const TrainTile *dtiles, int ntiles, float lr, float *dlosses) {
  cudaLaunchAttribute attr;
  cudaLaunchConfig_t lc = train_launch(&attr);
  return check_cuda(cudaLaunchKernelEx(&lc, train_cluster_kernel, m->P, m->Am, m->Av, dX, dY, dM, didx, dtiles, ntiles,
                                       (const float *)m->norm, lr, dlosses),
                    "mlp training kernel");
}

extern "C" {

int nvshmemx_mlp_num_params(void) { return NPARAM; }

int nvshmemx_mlp_create(unsigned long long seed, nvshmemx_mlp **out) {
  if (!out) return fail(NVSHMEMX_ERR_INVALID, "mlp_create: null out");
  nvshmemx_mlp *m = new nvshmemx_mlp();
  const size_t np = kParBytes, nn = kNormBytes;
  int rc;
  if ((rc = check_cuda(cudaGetDevice(&m->dev), "cudaGetDevice")) ||
      (rc = check_cuda(cudaDeviceGetAttribute(&m->sms, cudaDevAttrMultiProcessorCount, m->dev),
                       "cudaDeviceGetAttribute"))) {
    nvshmemx_mlp_destroy(m);
    return rc;
  }
  m->slot = take_slot(m->dev, &m->block);
  if (m->slot >= 0) {
    m->work = m->block + kNetBytes;
    m->work_bytes = kSlotWork;
  } else if ((rc = check_cuda(cudaMalloc(&m->block, kNetBytes), "cudaMalloc(mlp)"))) {
    nvshmemx_mlp_destroy(m);
    return rc;
  }
  m->P = (float *)m->block;
  m->norm = (float *)(m->block + np);
  m->Am = (float *)(m->block + np + nn);
  m->Av = (float *)(m->block + 2 * np + nn);
  m->G = (float *)(m->block + 3 * np + nn);
  m->loss = (float *)(m->block + 4 * np + nn);
  // He initialisation: N(0, 2 / fan_in) by Box-Muller on a splitmix64 stream
  std::vector<float> p((np + nn) / 4, 0.f);  // weights, then the normalisation
  unsigned long long ctr = seed;
  auto normal = [&]() {
    const double u1 = ((mix64(ctr++) >> 11) + 1.0) * (1.0 / 9007199254740993.0);
    const double u2 = (mix64(ctr++) >> 11) * (1.0 / 9007199254740992.0);
    return sqrt(-2.0 * log(u1)) * cos(6.283185307179586 * u2);
  };
  auto fill = [&](int off, int count, int fan_in) {
    const double sd = sqrt(2.0 / fan_in);
    for (int i = 0; i < count; ++i) p[off + i] = (float)(sd * normal());
  };
  fill(OFF_W1, NH * NI, NI);
  fill(OFF_W2, NH * NH, NH);
  fill(OFF_W3, NH * NH, NH);
  fill(OFF_W4, NO * NH, NH);
  for (int i = 0; i < NI; ++i) p[np / 4 + NI + i] = 1.f;
  if ((rc = upload(m->block, p.data(), np + nn)) ||
      (rc = check_cuda(cudaMemset(m->Am, 0, 3 * np + 256), "cudaMemset(mlp)"))) {
    nvshmemx_mlp_destroy(m);
    return rc;
  }
  *out = m;
  return check_cuda(cudaDeviceSynchronize(), "mlp_create");
}

int nvshmemx_mlp_destroy(nvshmemx_mlp *m) {
  if (!m) return 0;
  if (m->work_own) cudaFree(m->work);
  if (m->slot >= 0) {
    // nothing of this network runs any more (a free would wait too): the wait
    // is for the network's device, whichever is current
    int now = m->dev;
    cudaGetDevice(&now);
    if (now != m->dev) cudaSetDevice(m->dev);
    cudaStreamSynchronize(0);
    if (now != m->dev) cudaSetDevice(now);
    give_slot(m->dev, m->slot);
  } else if (m->block) {
    cudaFree(m->block);
  }
  delete m;
  return 0;
}

int nvshmemx_mlp_get_params(const nvshmemx_mlp *m, float *h) {
  if (!m || !h) return fail(NVSHMEMX_ERR_INVALID, "mlp_get_params");
  std::lock_guard<std::mutex> lk(m->mu);
  return check_cuda(cudaMemcpy(h, m->P, NPARAM * 4, cudaMemcpyDeviceToHost), "mlp_get_params");
}

int nvshmemx_mlp_set_params(nvshmemx_mlp *m, const float *h) {
  if (!m || !h) return fail(NVSHMEMX_ERR_INVALID, "mlp_set_params");
  std::lock_guard<std::mutex> lk(m->mu);
  return check_cuda(cudaMemcpy(m->P, h, NPARAM * 4, cudaMemcpyHostToDevice), "mlp_set_params");
}

int nvshmemx_mlp_set_normalization(nvshmemx_mlp *m, const float *mean, const float *sd) {
  if (!m || !mean || !sd) return fail(NVSHMEMX_ERR_INVALID, "mlp_set_normalization");
  float h[2 * NI];
  for (int i = 0; i < NI; ++i) {
    h[i] = mean[i];
    h[NI + i] = sd[i] > 1e-12f ? sd[i] : 1.f;
  }
  std::lock_guard<std::mutex> lk(m->mu);
  return check_cuda(cudaMemcpy(m->norm, h, sizeof h, cudaMemcpyHostToDevice), "mlp_set_normalization");
}

int nvshmemx_mlp_forward(nvshmemx_mlp *m, const float *X, int n, float *Y) {
  if (!m || n < 0 || (n && (!X || !Y))) return fail(NVSHMEMX_ERR_INVALID, "mlp_forward");
  if (n == 0) return 0;
  Work w(m);
  const size_t xb = pad256((size_t)n * NI * 4), yb = (size_t)n * NO * 4;
  int rc;
  if ((rc = w.get(m, xb + yb)) || (rc = upload(w.p, X, (size_t)n * NI * 4))) return rc;
  if ((rc = launch_forward(m, (float *)w.p, n, (float *)(w.p + xb)))) return rc;
  return check_cuda(cudaMemcpy(Y, w.p + xb, yb, cudaMemcpyDeviceToHost), "mlp_forward");
}

int nvshmemx_mlp_loss_grad(nvshmemx_mlp *m, const float *X, const float *Y, const float *M, int n, float *loss,
                           float *grad) {
  if (!m || n < 1 || !X || !Y || !M) return fail(NVSHMEMX_ERR_INVALID, "mlp_loss_grad");
  double cnt = 0;
  for (size_t i = 0; i < (size_t)n * NO; ++i) cnt += M[i];
  if (cnt <= 0) return fail(NVSHMEMX_ERR_INVALID, "mlp_loss_grad: empty mask");
  Work w(m);
  const size_t xb = pad256((size_t)n * NI * 4), yb = pad256((size_t)n * NO * 4);
  int rc;
  if ((rc = w.get(m, xb + 2 * yb)) || (rc = upload(w.p, X, (size_t)n * NI * 4)) ||
      (rc = upload(w.p + xb, Y, (size_t)n * NO * 4)) || (rc = upload(w.p + xb + yb, M, (size_t)n * NO * 4)))
    return rc;
  cudaMemset(m->G, 0, NPARAM * 4);
  cudaMemset(m->loss, 0, 4);
  if ((rc = launch_grad(m, (float *)w.p, (float *)(w.p + xb), (float *)(w.p + xb + yb), nullptr, n,
                        (float)(1.0 / cnt))))
    return rc;
  if (loss && (rc = check_cuda(cudaMemcpy(loss, m->loss, 4, cudaMemcpyDeviceToHost), "mlp loss"))) return rc;
  if (grad) return check_cuda(cudaMemcpy(grad, m->G, NPARAM * 4, cudaMemcpyDeviceToHost), "mlp grad");
  return 0;
}

int nvshmemx_mlp_train(nvshmemx_mlp *m, const float *X, const float *Y, const float *M, int n, int epochs, int batch,
                       float lr, unsigned long long seed, float *curve) {
  if (!m || n < 1 || epochs < 1 || batch < 1 || !X || !Y || !M) return fail(NVSHMEMX_ERR_INVALID, "mlp_train");
  std::vector<double> rowm(n, 0.0);
  for (int i = 0; i < n; ++i)
    for (int k = 0; k < NO; ++k) rowm[i] += M[(size_t)i * NO + k];
  Work w(m);
  const bool one_cluster = batch <= kClusterBatch && cluster_fits(m);
  const int nb = (n - 1) / batch + 1;  // batches of an epoch
  // epochs to a launch: at most 4 MiB of row numbers
  const int per = one_cluster ? (int)std::min<size_t>((size_t)epochs, std::max<size_t>(1, (1u << 20) / (size_t)n)) : 1;
  const size_t tiles_epoch = (size_t)nb * ((std::min(n, batch) - 1) / kTileRows + 1);
  // one block: features, targets, masks, row numbers, tiles, losses
  const size_t xb = pad256((size_t)n * NI * 4), yb = pad256((size_t)n * NO * 4), ib = pad256((size_t)per * n * 4),
               tb = one_cluster ? pad256(per * tiles_epoch * sizeof(TrainTile)) : 0, lb = pad256((size_t)epochs * 4);
  int rc;
  if ((rc = w.get(m, xb + 2 * yb + ib + tb + lb))) return rc;
  float *dX = (float *)w.p, *dY = (float *)(w.p + xb), *dM = (float *)(w.p + xb + yb);
  int *dI = (int *)(w.p + xb + 2 * yb);
  TrainTile *dT = (TrainTile *)(w.p + xb + 2 * yb + ib);
  float *dL = (float *)(w.p + xb + 2 * yb + ib + tb);
  // A table of the usual size goes up in one copy with the first launch's
  // rows and tiles; a large one array by array.
  const bool together = one_cluster && n <= 8192;
  std::vector<char> up((together ? xb + 2 * yb : 0) + ib + tb);
  if (together) {
    memcpy(up.data(), X, (size_t)n * NI * 4);
    memcpy(up.data() + xb, Y, (size_t)n * NO * 4);
    memcpy(up.data() + xb + yb, M, (size_t)n * NO * 4);
  } else if ((rc = upload(dX, X, (size_t)n * NI * 4)) || (rc = upload(dY, Y, (size_t)n * NO * 4)) ||
             (rc = upload(dM, M, (size_t)n * NO * 4))) {
    return rc;
  }
  char *const hrows = up.data() + (together ? xb + 2 * yb : 0);
  if ((rc = check_cuda(cudaMemsetAsync(dL, 0, lb), "cudaMemsetAsync(losses)"))) return rc;
  for (int e0 = 0; e0 < epochs; e0 += per) {
    const int e1 = std::min(epochs, e0 + per);
    int *perm = (int *)hrows;
    TrainTile *tiles = (TrainTile *)(hrows + ib);
    size_t nt = 0;
    for (int e = e0; e < e1; ++e, perm += n) {
      for (int i = 0; i < n; ++i) perm[i] = i;
      unsigned long long st = seed * 0x100000001b3ull + (unsigned long long)e;
      for (int i = n - 1; i > 0; --i) std::swap(perm[i], perm[mix64(st++) % (unsigned long long)(i + 1)]);
      if (!one_cluster) {
        if ((rc = upload(dI, perm, (size_t)n * 4))) return rc;
        cudaMemsetAsync(m->loss, 0, 4);
      }
      for (int b0 = 0; b0 < n; b0 += batch) {
        const int cnt = std::min(batch, n - b0);
        double c = 0;
        for (int i = b0; i < b0 + cnt; ++i) c += rowm[perm[i]];
        if (c <= 0) continue;
        ++m->step;
        const float c1 = 1.f - powf(0.9f, (float)m->step), c2 = 1.f - powf(0.999f, (float)m->step);
        if (one_cluster) {
          for (int k = 0; k < cnt; k += kTileRows) {
            const bool last = cnt - k <= kTileRows;
            tiles[nt++] = TrainTile{(e - e0) * n + b0 + k, std::min(cnt - k, kTileRows), (float)(1.0 / c), c1, c2,
                                    (k == 0 ? kFirst : 0) | (last ? kLast : 0), e, 0};
          }
        } else {
          cudaMemsetAsync(m->G, 0, NPARAM * 4);
          if ((rc = launch_grad(m, dX, dY, dM, dI + b0, cnt, (float)(1.0 / c)))) return rc;
          adam_kernel<<<(NPARAM + 255) / 256, 256>>>(m->P, m->G, m->Am, m->Av, NPARAM, lr, c1, c2);
        }
      }
      if (!one_cluster && curve &&
          (rc = check_cuda(cudaMemcpy(&curve[e], m->loss, 4, cudaMemcpyDeviceToHost), "mlp loss")))
        return rc;
    }
    if (!one_cluster) continue;
    const bool first_up = together && e0 == 0;
    if ((rc = first_up ? upload(w.p, up.data(), xb + 2 * yb + ib + nt * sizeof(TrainTile))
                       : upload(dI, hrows, ib + nt * sizeof(TrainTile))))
      return rc;
    if (nt && (rc = launch_train(m, dX, dY, dM, dI, dT, (int)nt, lr, dL))) return rc;
  }
  if (one_cluster && curve &&
      (rc = check_cuda(cudaMemcpy(curve, dL, (size_t)epochs * 4, cudaMemcpyDeviceToHost), "mlp losses")))
    return rc;
  if (curve)
    for (int e = 0; e < epochs; ++e) curve[e] /= (float)nb;
  return check_cuda(cudaDeviceSynchronize(), "mlp_train");
}

int nvshmemx_mlp_pick(nvshmemx_mlp *m, const float *X, int n, int *variant, float *margin) {
  if (!m || n < 0 || (n && (!X || !variant))) return fail(NVSHMEMX_ERR_INVALID, "mlp_pick");
  std::vector<float> y((size_t)n * NO);
  int rc;
  if ((rc = nvshmemx_mlp_forward(m, X, n, y.data()))) return rc;
  for (int i = 0; i < n; ++i) {
    const float *r = &y[(size_t)i * NO];
    int best = 0;
    for (int k = 1; k < NO; ++k)
      if (r[k] < r[best]) best = k;
    float second = 1e30f;
    for (int k = 0; k < NO; ++k)
      if (k != best && r[k] < second) second = r[k];
    variant[i] = best;
    if (margin) margin[i] = second - r[best];
  }
  return 0;
}

// ------------------------------------------------------------------ variants
int nvshmemx_variant_describe(int v, int *percall_mode, nvshmemx_batch_config *cfg) {
  if (v < 0 || v >= NO) return NVSHMEMX_ERR_INVALID;
  nvshmemx_batch_config c;
  nvshmemx_batch_default_config(&c);
  int mode = -1;
  struct Shape {
    int chunk, unroll, threads, grab, stages, stage, minb;
  };
  static const Shape shapes[8] = {
      {4096, 4, 1024, 4, 0, 8192, 512},   {16384, 8, 256, 2, 0, 8192, 512},   {65536, 4, 256, 2, 0, 8192, 512},
      {16384, 4, 128, 2, 2, 8192, 2048},  {16384, 4, 256, 2, 3, 8192, 512},   {16384, 4, 128, 2, 4, 4096, 512},
      {65536, 4, 256, 2, 3, 8192, 512},   {65536, 4, 128, 2, 2, 16384, 2048},
  };
  if (v < 4) {
    mode = v;  // NVSHMEMX_MODE_THREAD, WARP, BLOCK, BULK
  } else {
    const Shape &s = shapes[v - 4];
    c.vec_bytes = 16;
    c.chunk_bytes = s.chunk;
    c.unroll = s.unroll;
    c.threads = s.threads;
    c.ctas_per_sm = 0;
    c.grab = s.grab;
    c.tma_stages = s.stages;
    c.tma_stage_bytes = s.stage;
    c.tma_min_bytes = s.minb;
  }
  if (percall_mode) *percall_mode = mode;
  if (cfg) *cfg = c;
  return 0;
}

int nvshmemx_variant_time(nvshmemx_batch *b, int v, int reps, size_t flush_bytes, float *out_ms) {
  int mode;
  nvshmemx_batch_config c, saved;
  if (!b || reps < 1 || nvshmemx_variant_describe(v, &mode, &c)) return fail(NVSHMEMX_ERR_INVALID, "variant_time");
  nvshmemx_batch_get_config(b, &saved);
  int rc = 0;
  if (mode < 0 && (rc = nvshmemx_batch_set_config(b, &c))) return rc;
  std::vector<float> t;
  for (int r = 0; r <= reps && rc == 0; ++r) {  // r == 0 warms up (graph build)
    if ((rc = l2_flush(flush_bytes))) break;
    float ms = 0;
    rc = mode >= 0 ? nvshmemx_batch_execute_percall(b, mode, 1, &ms) : nvshmemx_batch_execute(b, 1, &ms);
    if (r > 0) t.push_back(ms);
  }
  nvshmemx_batch_set_config(b, &saved);
  if (rc) return rc;
  std::sort(t.begin(), t.end());
  if (out_ms) *out_ms = t[t.size() / 2];
  return 0;
}

}  // extern "C"
