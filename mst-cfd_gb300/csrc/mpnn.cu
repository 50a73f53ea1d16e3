// The learned initial field: a message-passing network over the cell
// adjacency whose dense layers run on the tensor cores (tc_gemm.cuh).
// This file holds the GEMM launcher and its C-ABI check entry point.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdlib>
#include <mutex>
#include <string>
#include <vector>

#include "ctx.hpp"
#include "tc_gemm.cuh"
#include "tc_gemm_tma.cuh"
#include "vec8.cuh"

namespace mst {
namespace tc {

// Descriptor strides of the no-swizzle K-major layout of k_gemm_bf16's
// tiles: core matrices adjacent along K are 128 bytes apart (leading
// dimension), 8-row groups 1024 bytes apart (stride dimension).
constexpr uint32_t kLBO = 128, kSBO = 1024;

// polls of the GEMM's bounded mbarrier waits (mst_set_wait_limit)
std::atomic<long long> g_wait_limit{-1};

// cuTensorMapEncodeTiled, through the runtime's driver entry point (no
// link-time dependency on the driver library)
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_tiled() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault,
                                         &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  });
  return fn;
}

// tensor map of a row-major [rows][cols] BF16 matrix in boxes of box_rows rows
// x 64 columns, 128-byte swizzle; what lies beyond the matrix reads as zeros
bool bf16_tile_map(CUtensorMap* map, const void* base, int rows, int cols, int box_rows) {
  EncodeTiledFn fn = encode_tiled();
  if (!fn) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)cols * 2};
  const cuuint32_t box[2] = {(cuuint32_t)kBK, (cuuint32_t)box_rows};
  const cuuint32_t es[2] = {1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides,
            box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) ==
         CUDA_SUCCESS;
}

// MSTCFD_GEMM_TMA=0 keeps every GEMM on k_gemm_bf16 (for comparisons)
bool use_tma() {
  static const bool on = [] {
    const char* v = std::getenv("MSTCFD_GEMM_TMA");
    return !v || std::atoi(v) != 0;
  }();
  return on;
}

unsigned spin_limit() {
  const long long lim = g_wait_limit.load(std::memory_order_relaxed);
  return lim < 0 ? kSpinLimit : (unsigned)std::min<long long>(lim, 0xFFFFFFFFll);
}

// tensor map of an FP32 [rows][ld] matrix's first cols columns in boxes of 32 x
// 32, 128-byte swizzle: the staged result tiles (stores clip at the matrix)
bool f32_tile_map(CUtensorMap* map, const float* base, int rows, int cols, int ld) {
  EncodeTiledFn fn = encode_tiled();
  if (!fn || (ld & 3) || (reinterpret_cast<uintptr_t>(base) & 15)) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)ld * 4};
  const cuuint32_t box[2] = {32, 32};
  const cuuint32_t es[2] = {1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(base), dims, strides, box,
            es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) ==
         CUDA_SUCCESS;
}

// The persistent TMA kernel where it applies (whole K per CTA, K <= 256 in
// tiles of 64, 16-byte-aligned operands; fewer than 128 outputs use one
// 128-wide tile whose missing rows of B the copy fills with zeros); false:
// the caller launches k_gemm_bf16 instead
bool gemm_tma(const GemmArgs& a, cudaStream_t s, cudaError_t* err) {
  *err = cudaSuccess;
  if (a.k_chunk > 0 || a.K % kBK != 0 || a.K / kBK > kTmaMaxKT || a.M <= 0 || a.N <= 0 ||
      (reinterpret_cast<uintptr_t>(a.A) & 15) || (reinterpret_cast<uintptr_t>(a.B) & 15))
    return false;
  CUtensorMap ma, mb;
  if (!bf16_tile_map(&ma, a.A, a.M, a.K, kBM) || !bf16_tile_map(&mb, a.B, a.N, a.K, kBM))
    return false;
  static std::atomic<uint64_t> attr_done{0};
  const int kt = a.K / kBK;
  *err = ensure_smem_limit(k_gemm_tma, tma_smem_bytes(kTmaMaxKT), attr_done);
  if (*err != cudaSuccess) return true;
  // resident CTAs of the device (SMs x CTAs per SM at this K), per K
  static std::atomic<int> resident[kTmaMaxKT + 1];
  int slots = resident[kt].load(std::memory_order_relaxed);
  if (slots <= 0) {
    int dev = 0, sms = 0, per_sm = 0;
    if ((*err = cudaGetDevice(&dev)) != cudaSuccess ||
        (*err = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) !=
            cudaSuccess ||
        (*err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_gemm_tma, kTmaThreads,
                                                              tma_smem_bytes(kt))) != cudaSuccess)
      return true;
    slots = std::max(1, sms * per_sm);
    resident[kt].store(slots, std::memory_order_relaxed);
  }
  TmaGemm t;
  t.g = a;
  t.kt = kt;
  CUtensorMap mc = ma, mi = ma;  // (not used unless staged)
  t.staged = (!a.C || f32_tile_map(&mc, a.C, a.M, a.N, a.ldc)) &&
             (!a.Cin || f32_tile_map(&mi, a.Cin, a.M, a.N, a.ldc)) &&
             (!a.Cb || ((a.ldcb & 7) == 0 && (reinterpret_cast<uintptr_t>(a.Cb) & 15) == 0 &&
                        a.N % 32 == 0)) &&
             (!a.gate || a.N % 32 == 0);
  t.n_ntiles = (a.N + kBN - 1) / kBN;
  t.m_tiles = (a.M + kBM - 1) / kBM;
  // one wave of resident CTAs, each column block with the same number
  int grid = std::min(slots, t.n_ntiles * t.m_tiles);
  grid = std::max(t.n_ntiles, grid / t.n_ntiles * t.n_ntiles);
  k_gemm_tma<<<grid, kTmaThreads, tma_smem_bytes(kt), s>>>(ma, mb, mc, mi, t);
  *err = cudaGetLastError();
  return true;
}

template <bool ROWS>
cudaError_t launch_split(const CUtensorMap& ma, const CUtensorMap& mb, const GemmArgs& a,
                         cudaStream_t s) {
  static std::atomic<uint64_t> attr_done{0};
  const cudaError_t e = ensure_smem_limit(k_gemm_tma_split<ROWS>, split_smem_bytes(), attr_done);
  if (e != cudaSuccess) return e;
  const dim3 grid((a.M + kBM - 1) / kBM, (a.N + kBN - 1) / kBN, (a.K + a.k_chunk - 1) / a.k_chunk);
  k_gemm_tma_split<ROWS><<<grid, kSplitThreads, split_smem_bytes(), s>>>(ma, mb, a);
  return cudaGetLastError();
}

// The split-K TMA kernel where it applies (K and the chunk in tiles of 64,
// 16-byte-aligned operands); false: the caller launches k_gemm_bf16
bool gemm_tma_split(const GemmArgs& a, cudaStream_t s, cudaError_t* err) {
  *err = cudaSuccess;
  if (a.k_chunk <= 0 || a.k_chunk % kBK != 0 || a.K % kBK != 0 || a.M <= 0 || a.N <= 0 ||
      (reinterpret_cast<uintptr_t>(a.A) & 15) || (reinterpret_cast<uintptr_t>(a.B) & 15))
    return false;
  CUtensorMap ma, mb;
  if (!bf16_tile_map(&ma, a.A, a.M, a.K, kBM) || !bf16_tile_map(&mb, a.B, a.N, a.K, kBM))
    return false;
  *err = launch_split<false>(ma, mb, a, s);
  return true;
}

// The same with operands [n_rows][a_cols] and [n_rows][b_cols] (K = the rows,
// M <= a_cols, N <= b_cols); false: the caller transposes
bool gemm_tma_rows(const GemmArgs& a, int n_rows, int a_cols, int b_cols, cudaStream_t s,
                   cudaError_t* err) {
  *err = cudaSuccess;
  if (!use_tma() || a.k_chunk <= 0 || a.k_chunk % kBK != 0 || a.K % kBK != 0 ||
      a_cols % 8 != 0 || b_cols % 8 != 0 || (reinterpret_cast<uintptr_t>(a.A) & 15) ||
      (reinterpret_cast<uintptr_t>(a.B) & 15))
    return false;
  CUtensorMap ma, mb;
  if (!bf16_tile_map(&ma, a.A, n_rows, a_cols, kBK) ||
      !bf16_tile_map(&mb, a.B, n_rows, b_cols, kBK))
    return false;
  GemmArgs g = a;
  g.spin_limit = spin_limit();
  *err = launch_split<true>(ma, mb, g, s);
  return true;
}

cudaError_t gemm(const GemmArgs& a0, cudaStream_t s) {
  static std::atomic<uint64_t> attr_done{0}, attr_done16{0};
  const bool narrow = a0.N <= 16;
  cudaError_t e = narrow ? ensure_smem_limit(k_gemm_bf16<16>, smem_bytes<16>(), attr_done16)
                         : ensure_smem_limit(k_gemm_bf16<kBN>, kSmemBytes, attr_done);
  if (e != cudaSuccess) return e;
  GemmArgs a = a0;
  a.spin_limit = spin_limit();
  if (a.lbo == 0 && use_tma()) {
    cudaError_t te;
    if (a.k_chunk > 0 ? gemm_tma_split(a, s, &te) : gemm_tma(a, s, &te)) return te;
  }
  if (a.lbo == 0) {
    a.lbo = kLBO;
    a.sbo = kSBO;
  }
  const int splits = a.k_chunk > 0 ? (a.K + a.k_chunk - 1) / a.k_chunk : 1;
  if (narrow) {
    dim3 grid((a.M + kBM - 1) / kBM, 1, splits);
    k_gemm_bf16<16><<<grid, kGemmThreads, smem_bytes<16>(), s>>>(a);
    return cudaGetLastError();
  }
  dim3 grid((a.M + kBM - 1) / kBM, (a.N + kBN - 1) / kBN, splits);
  k_gemm_bf16<kBN><<<grid, kGemmThreads, kSmemBytes, s>>>(a);
  return cudaGetLastError();
}

// C[M][N] = sum over z of part[z][M][N], in a fixed order (deterministic): the
// kReduceRows threads of an output each add a run of z, then the runs are added
// in order.  (One thread an output: a chain of 293 loads, 16 us.)
constexpr int kReduceRows = 8;
__global__ void __launch_bounds__(32 * kReduceRows)
    k_reduce_splits(const float* __restrict__ part, int splits, size_t mn, float* __restrict__ c) {
  __shared__ float red[kReduceRows][32];
  const size_t i = blockIdx.x * (size_t)32 + threadIdx.x;
  const int run = (splits + kReduceRows - 1) / kReduceRows;
  const int z1 = min(splits, (int)(threadIdx.y + 1) * run);
  float s = 0.f;
  if (i < mn) {
#pragma unroll 8
    for (int z = threadIdx.y * run; z < z1; ++z) s += part[(size_t)z * mn + i];
  }
  red[threadIdx.y][threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.y == 0 && i < mn) {
    for (int q = 1; q < kReduceRows; ++q) s += red[q][threadIdx.x];
    c[i] = s;
  }
}

cudaError_t reduce_splits(const float* part, int splits, size_t mn, float* c) {
  k_reduce_splits<<<(unsigned)((mn + 31) / 32), dim3(32, kReduceRows)>>>(part, splits, mn, c);
  return cudaGetLastError();
}

}  // namespace tc
}  // namespace mst

// ---------------------------------------------------------------------------
// The network.  Per cell c of a mesh graph (interior-face neighbours N(c)):
//   h0 = relu(We x + be)                                 x: 16 features (K 64)
//   h_{l+1} = h_l + relu(Wl [h_l, mean_{j in N(c)} h_j] + bl),  l = 0..2
//   y = Wd h3 + bd                                       4 outputs
// Width 128.  GEMM operands are BF16 (weights and activations rounded once
// per use), accumulation and the residual stream FP32; master weights and
// Adam moments FP32.  Training minimises the mean squared error of y.
// ---------------------------------------------------------------------------
namespace {

constexpr int kW = 128;       // hidden width
constexpr int kIn = 16;       // input features
constexpr int kInK = 64;      // padded K of the first layer
constexpr int kOut = 4;
constexpr int kLayers = 3;
constexpr int kZ = 2 * kW;    // [h, mean of neighbours]
constexpr int kMaxSplits = 320;  // split-K CTAs of a weight-gradient GEMM

// Cells are walked by half warps, each lane eight of the 128 columns (32-byte
// loads; four columns a lane and a warp a cell took twice the instructions: 49
// and 82 us where this takes 41 and 72).  A block takes a run of consecutive
// cells (neighbours' rows meet in its L1), its kCellWarps warps in turn, so that a
// cell's neighbour ids are there when its rows are read.
constexpr int kCellWarps = 8;
constexpr int kHalf = 16;  // lanes of a cell
constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ uint2 bf16x4(float4 v) {
  const __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
  return make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
}
struct F8 {
  float x[8];
};
__device__ __forceinline__ F8 ld8(const float* p) {
  F8 r;
  mst::load8(p, r.x);
  return r;
}
__device__ __forceinline__ void st_bf16x8(__nv_bfloat16* p, const F8& v) {
  const uint2 lo = bf16x4(make_float4(v.x[0], v.x[1], v.x[2], v.x[3])),
              hi = bf16x4(make_float4(v.x[4], v.x[5], v.x[6], v.x[7]));
  *reinterpret_cast<uint4*>(p) = make_uint4(lo.x, lo.y, hi.x, hi.y);
}

// x / d for a cell's degree d, r = 1 / d: the product with the reciprocal and
// one residual correction (Markstein 1990), equal to the correctly rounded
// quotient for every x of normal range and d = 1..256 (all significands
// compared).  The division itself takes four times the instructions, and its
// slow path wherever a numerator is zero, as relu outputs often are: 20 us of
// k_build_z's 75 at 168,594 cells.
__device__ __forceinline__ F8 div_deg(F8 v, float d, float r) {
  float m = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) m = fmaxf(m, fabsf(v.x[i]));
  // (d = 0: a neighbour whose own list is empty)
  if (m == __int_as_float(0x7f800000) || !(d >= 1.f && d <= 256.f)) {
#pragma unroll
    for (int i = 0; i < 8; ++i) v.x[i] /= d;
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float q = v.x[i] * r;
      v.x[i] = fmaf(fmaf(-q, d, v.x[i]), r, q);
    }
  }
  return v;
}

// The cells of one half warp, every 2 kCellWarps-th: their neighbour ranges and
// ids (lane i the i-th) read one cell ahead
struct CellWalk {
  const int *ptr, *nbr;
  int n, sub, b, e, id, nb, ne, nid;
  __device__ __forceinline__ void fetch(int c) {
    nb = ne = 0;
    if (c < n) {
      nb = ptr[c];
      ne = ptr[c + 1];
    }
    nid = nb + sub < ne ? nbr[nb + sub] : 0;
  }
  __device__ __forceinline__ void next() {
    b = nb;
    e = ne;
    id = nid;
  }
};

// add(k, whether the cell has a k-th neighbour, it, its row) in list order; both
// halves of a warp go through the longer list.  (Rows loaded two or three at a
// time cost registers and with them warps: 78 and 85 us for 72 in k_back.)
template <class Load, class Add>
__device__ __forceinline__ void walk_neighbours(const CellWalk& w, Load load, Add add) {
  const int deg = w.e - w.b, most = max(deg, __shfl_xor_sync(kFull, deg, kHalf));
  for (int k = 0; k < most; ++k) {
    int id = __shfl_sync(kFull, w.id, k & (kHalf - 1), kHalf);
    if (k >= kHalf && k < deg) id = w.nbr[w.b + k];
    F8 v{};
    if (k < deg) v = load(id);
    add(k, k < deg, id, v);
  }
}

// Z = [bf16(h_c), bf16(mean_{j in N(c)} h_j)] (rows >= n: zero), the neighbours
// summed in list order
__global__ void __launch_bounds__(32 * kCellWarps, 4)
    k_build_z(const float* __restrict__ h, const int* __restrict__ ptr,
              const int* __restrict__ nbr, int n, int n_pad, __nv_bfloat16* __restrict__ z) {
  const int sub = threadIdx.x & (kHalf - 1), k = sub * 8;
  const int chunk = (n_pad + gridDim.x - 1) / gridDim.x;
  const int last = min(n_pad, (int)(blockIdx.x + 1) * chunk);
  int c = blockIdx.x * chunk + threadIdx.x / kHalf;
  CellWalk w{ptr, nbr, n, sub};
  w.fetch(c);
  // (a warp leaves together)
  for (; c - (int)(threadIdx.x / kHalf & 1) < last; c += 2 * kCellWarps) {
    w.next();
    w.fetch(c + 2 * kCellWarps);
    F8 a{}, hc{};
    if (c < min(n, last)) hc = ld8(h + (size_t)c * kW + k);
    walk_neighbours(
        w, [&](int j) { return ld8(h + (size_t)j * kW + k); },
        [&](int, bool there, int, const F8& v) {
          if (there) {
#pragma unroll
            for (int i = 0; i < 8; ++i) a.x[i] += v.x[i];
          }
        });
    if (w.e > w.b) {
      const float d = (float)(w.e - w.b);
      a = div_deg(a, d, 1.f / d);
    }
    if (c < last) {
      st_bf16x8(z + (size_t)c * kZ + k, hc);
      st_bf16x8(z + (size_t)c * kZ + kW + k, a);
    }
  }
}

// dst[w][n_pad] = transpose of src[n][w] (BF16), zero for rows >= n: the
// operands of the GEMMs that k_gemm_bf16 takes over
__global__ void k_transpose_bf16(const __nv_bfloat16* __restrict__ src, int n, int w,
                                 int n_pad, __nv_bfloat16* __restrict__ dst) {
  __shared__ __nv_bfloat16 t[32][33];
  const int r0 = blockIdx.x * 32, c0 = blockIdx.y * 32;
  for (int i = threadIdx.y; i < 32; i += blockDim.y) {
    const int r = r0 + i, c = c0 + threadIdx.x;
    t[i][threadIdx.x] = (r < n && c < w) ? src[(size_t)r * w + c] : __float2bfloat16_rn(0.f);
  }
  __syncthreads();
  for (int i = threadIdx.y; i < 32; i += blockDim.y) {
    const int c = c0 + i, r = r0 + threadIdx.x;
    if (c < w && r < n_pad) dst[(size_t)c * n_pad + r] = t[threadIdx.x][i];
  }
}

// loss and dY = 2 (y - t) / (n * kOut), the latter as the BF16 operand [np][64]
// (columns >= 4 and rows >= n zero); per-block partial losses and column sums.
// 64 cells a block.
__global__ void __launch_bounds__(256)
    k_mse(const float* __restrict__ y, const float* __restrict__ t, int n,
          __nv_bfloat16* __restrict__ dyb, double* __restrict__ part, float* __restrict__ cpart) {
  __shared__ double red[256];
  __shared__ float dy[256];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double l = 0.0;
  float g = 0.f;
  if (i < n * kOut) {
    const float d = y[i] - t[i];
    g = 2.f * d / (float)(n * kOut);
    l = (double)d * d;
  }
  red[threadIdx.x] = l;
  dy[threadIdx.x] = g;
  __syncthreads();
  for (int q = threadIdx.x; q < 64 * (kInK / 8); q += 256) {
    const int r = q / (kInK / 8), c = q % (kInK / 8);
    uint4 o = make_uint4(0u, 0u, 0u, 0u);
    if (c == 0) {
      const uint2 b = bf16x4(make_float4(dy[4 * r], dy[4 * r + 1], dy[4 * r + 2], dy[4 * r + 3]));
      o.x = b.x;
      o.y = b.y;
    }
    reinterpret_cast<uint4*>(dyb)[((size_t)blockIdx.x * 64 + r) * (kInK / 8) + c] = o;
  }
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) {
      red[threadIdx.x] += red[threadIdx.x + w];
      if (w >= kOut) dy[threadIdx.x] += dy[threadIdx.x + w];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = red[0];
  if (threadIdx.x < kOut) cpart[(size_t)blockIdx.x * kOut + threadIdx.x] = dy[threadIdx.x];
}

// One backward step between two dense products.  AGG: dH_l = dH_{l+1} +
// dZ[:, :kW] + sum_{c in N(j)} dZ[c, kW:] / |N(c)| (neighbours in list order),
// stored to dh if a further layer needs it; otherwise dH is read.  Then dP =
// dH (.) [relu output > 0] (the gate bits of the forward product) as the BF16
// operand (rows >= n zero), and its FP32 column sums per block -- the bias
// gradient -- without an FP32 dP in memory.  Bound by its bytes: dH and dZ in,
// dH and dP out.
template <bool AGG>
__global__ void __launch_bounds__(32 * kCellWarps, 4)
    k_back(const float* __restrict__ dhn, const float* __restrict__ dz,
           const int* __restrict__ ptr, const int* __restrict__ nbr,
           const uint8_t* __restrict__ gate, int n, int n_pad, float* __restrict__ dh,
           __nv_bfloat16* __restrict__ dpb, float* __restrict__ cpart) {
  __shared__ float red[2 * kCellWarps][kW];
  const int sub = threadIdx.x & (kHalf - 1), k = sub * 8;
  const int chunk = (n_pad + gridDim.x - 1) / gridDim.x;
  const int last = min(n_pad, (int)(blockIdx.x + 1) * chunk);
  int j = blockIdx.x * chunk + threadIdx.x / kHalf;
  F8 s{};
  CellWalk w{ptr, nbr, n, sub};
  if (AGG) w.fetch(j);
  // (a warp leaves together)
  for (; j - (int)(threadIdx.x / kHalf & 1) < last; j += 2 * kCellWarps) {
    F8 v{};
    unsigned g = 0;
    const bool live = j < min(n, last);
    if (AGG) {
      w.next();
      w.fetch(j + 2 * kCellWarps);
    }
    if (live) {
      g = gate[(size_t)j * (kW / 8) + sub];
      v = ld8(dhn + (size_t)j * kW + k);
    }
    if (AGG) {
      // lane i: the degree of the i-th neighbour and its reciprocal
      const float dl = sub < w.e - w.b ? (float)(ptr[w.id + 1] - ptr[w.id]) : 1.f, rl = 1.f / dl;
      if (live) {
        const F8 y = ld8(dz + (size_t)j * kZ + k);
#pragma unroll
        for (int i = 0; i < 8; ++i) v.x[i] += y.x[i];
      }
      walk_neighbours(
          w, [&](int c) { return ld8(dz + (size_t)c * kZ + kW + k); },
          [&](int i, bool there, int c, const F8& u) {
            float d = __shfl_sync(kFull, dl, i & (kHalf - 1), kHalf);
            float r = __shfl_sync(kFull, rl, i & (kHalf - 1), kHalf);
            if (!there) return;
            if (i >= kHalf) {
              d = (float)(ptr[c + 1] - ptr[c]);
              r = 1.f / d;
            }
            const F8 q = div_deg(u, d, r);
#pragma unroll
            for (int t = 0; t < 8; ++t) v.x[t] += q.x[t];
          });
      if (dh && live) mst::store8(dh + (size_t)j * kW + k, v.x);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      v.x[i] = (g >> i & 1u) ? v.x[i] : 0.f;
      s.x[i] += v.x[i];
    }
    if (j < last) st_bf16x8(dpb + (size_t)j * kW + k, v);
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) red[threadIdx.x / kHalf][k + i] = s.x[i];
  __syncthreads();
  if (threadIdx.x < kW) {
    float a = red[0][threadIdx.x];
    for (int q = 1; q < 2 * kCellWarps; ++q) a += red[q][threadIdx.x];
    cpart[(size_t)blockIdx.x * kW + threadIdx.x] = a;
  }
}

// out[w] = column sums of the blocks' partials part[blocks][w], w <= 128, in a
// fixed order: thread (r, c) of a block takes every 32nd partial of column c
__global__ void __launch_bounds__(1024) k_colsum_parts(const float* __restrict__ part, int blocks,
                                                       int w, float* __restrict__ out) {
  __shared__ float red[32][33];
  const int c = blockIdx.x * 32 + (threadIdx.x & 31), r = threadIdx.x >> 5;
  float acc = 0.f;
  if (c < w) {
#pragma unroll 8
    for (int b = r; b < blocks; b += 32) acc += part[(size_t)b * w + c];
  }
  red[r][threadIdx.x & 31] = acc;
  __syncthreads();
  if (r == 0 && c < w) {
    for (int q = 1; q < 32; ++q) acc += red[q][threadIdx.x];
    out[c] = acc;
  }
}

// the transposes of the weights that the data gradients need, in one launch
// (blockIdx.z: which); dst[cols][rows_pad], zero for rows >= rows
struct WeightT {
  const __nv_bfloat16* src[kLayers + 1];
  __nv_bfloat16* dst[kLayers + 1];
  int rows[kLayers + 1], cols[kLayers + 1], pad[kLayers + 1];
};
__global__ void k_transpose_weights(const WeightT t) {
  __shared__ __nv_bfloat16 s[32][33];
  const int z = blockIdx.z, r0 = blockIdx.x * 32, c0 = blockIdx.y * 32;
  const int R = t.rows[z], W = t.cols[z], pad = t.pad[z];
  for (int i = threadIdx.y; i < 32; i += blockDim.y) {
    const int r = r0 + i, c = c0 + threadIdx.x;
    s[i][threadIdx.x] = (r < R && c < W) ? t.src[z][(size_t)r * W + c] : __float2bfloat16_rn(0.f);
  }
  __syncthreads();
  for (int i = threadIdx.y; i < 32; i += blockDim.y) {
    const int c = c0 + i, r = r0 + threadIdx.x;
    if (c < W && r < pad) t.dst[z][(size_t)c * pad + r] = s[threadIdx.x][i];
  }
}

struct AdamTensors {  // blockIdx.y: which
  float *w[2 * (kLayers + 2)], *m[2 * (kLayers + 2)], *v[2 * (kLayers + 2)];
  const float* g[2 * (kLayers + 2)];
  __nv_bfloat16* wb[2 * (kLayers + 2)];
  int n[2 * (kLayers + 2)];
};
__global__ void k_adam(const AdamTensors t, float lr, float b1, float b2, float c1, float c2) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, q = blockIdx.y;
  if (i >= t.n[q]) return;
  const float gi = t.g[q][i];
  const float mi = b1 * t.m[q][i] + (1.f - b1) * gi;
  const float vi = b2 * t.v[q][i] + (1.f - b2) * gi * gi;
  t.m[q][i] = mi;
  t.v[q][i] = vi;
  const float x = t.w[q][i] - lr * (mi / c1) / (sqrtf(vi / c2) + 1e-8f);
  t.w[q][i] = x;
  t.wb[q][i] = __float2bfloat16_rn(x);
}

}  // namespace

// One parameter tensor: FP32 master, BF16 copy (GEMM operand), gradient,
// Adam moments.  Weights are [rows = outputs][cols = inputs], the B
// operand layout of the GEMM.
struct MpnnParam {
  int rows = 0, cols = 0;
  float *w = nullptr, *g = nullptr, *m = nullptr, *v = nullptr;
  __nv_bfloat16* wb = nullptr;
  int size() const { return rows * cols; }
};

struct mst_mpnn {
  MpnnParam W[2 * (kLayers + 2)];  // We, be, Wl0, bl0, ..., Wd, bd
  // the tensors of W lie one after another in these
  float *w = nullptr, *g = nullptr, *m1 = nullptr, *v1 = nullptr;
  __nv_bfloat16* wb = nullptr;
  int step = 0;
  // work buffers for up to cap cells
  int cap = 0;
  int* err = nullptr;
  double* lpart = nullptr;
  std::vector<void*> bufs;
  float* H[kLayers] = {};          // FP32 residual stream (the last only as Hb)
  __nv_bfloat16 *X = nullptr, *Z[kLayers] = {}, *Hb = nullptr;
  uint16_t* gate[kLayers + 1] = {};  // [cap][8] bits: the layer's relu output > 0
  float *Y = nullptr, *T = nullptr, *dH = nullptr, *dHn = nullptr, *dZ = nullptr;
  __nv_bfloat16 *dPb = nullptr, *dYb = nullptr, *WdT = nullptr, *WlT[kLayers] = {};
  __nv_bfloat16 *tA = nullptr, *tB = nullptr;  // transposed operands, where they are needed
  float* part = nullptr;  // split-K partial products of the weight gradients
  float* feat = nullptr;  // the graph's FP32 features [cap][16]
  int *ptr = nullptr, *nbr = nullptr;
  int n_nbr_cap = 0;
  int n = 0;  // cells of the current graph
  // live timing of the tensor-core GEMM launches (mst_mpnn_profile): one
  // event pair per launch on the network's stream, with the launch's
  // 2MNK flops and its operand/result bytes
  struct GemmRec {
    cudaEvent_t a = nullptr, b = nullptr;
    double flops = 0.0, bytes = 0.0;
  };
  bool prof = false;
  std::vector<GemmRec> recs;
  size_t n_recs = 0;
};

namespace {

MpnnParam& P(mst_mpnn* m, int i) { return m->W[i]; }
enum { kWe = 0, kBe = 1, kWd = 2 * kLayers + 2, kBd = 2 * kLayers + 3 };
int wl(int l) { return 2 + 2 * l; }
int bl(int l) { return 3 + 2 * l; }

template <class T>
cudaError_t nalloc(mst_mpnn* m, T** p, size_t count) {
  cudaError_t e = cudaMalloc((void**)p, std::max<size_t>(count, 1) * sizeof(T));
  if (e == cudaSuccess) {
    m->bufs.push_back(*p);
    e = cudaMemset(*p, 0, std::max<size_t>(count, 1) * sizeof(T));
  }
  return e;
}

int pad128(int n) { return (n + 127) / 128 * 128; }
int pad64(int n) { return (n + 63) / 64 * 64; }

cudaError_t ensure_cap(mst_mpnn* m, int n, int n_nbr) {
  cudaError_t e = cudaSuccess;
  if (n_nbr > m->n_nbr_cap) {
    if (m->nbr) cudaFree(m->nbr);
    e = cudaMalloc(&m->nbr, sizeof(int) * (size_t)n_nbr);
    m->n_nbr_cap = n_nbr;
  }
  if (e != cudaSuccess || n <= m->cap) return e;
  // grow: free the old work buffers (parameters live in m->W)
  for (void* p : m->bufs) cudaFree(p);
  m->bufs.clear();
  const int np = pad128(n);
  m->cap = n;
  m->tA = m->tB = nullptr;
  for (int l = 0; l < kLayers && e == cudaSuccess; ++l) e = nalloc(m, &m->H[l], (size_t)np * kW);
  for (int l = 0; l < kLayers && e == cudaSuccess; ++l) e = nalloc(m, &m->Z[l], (size_t)np * kZ);
  for (int l = 0; l <= kLayers && e == cudaSuccess; ++l)
    e = nalloc(m, &m->gate[l], (size_t)np * (kW / 16));
  if (e == cudaSuccess) e = nalloc(m, &m->X, (size_t)np * kInK);
  if (e == cudaSuccess) e = nalloc(m, &m->Hb, (size_t)np * kW);
  if (e == cudaSuccess) e = nalloc(m, &m->Y, (size_t)np * kOut);
  if (e == cudaSuccess) e = nalloc(m, &m->T, (size_t)np * kOut);
  if (e == cudaSuccess) e = nalloc(m, &m->dYb, (size_t)np * kInK);
  if (e == cudaSuccess) e = nalloc(m, &m->dH, (size_t)np * kW);
  if (e == cudaSuccess) e = nalloc(m, &m->dHn, (size_t)np * kW);
  if (e == cudaSuccess) e = nalloc(m, &m->dPb, (size_t)np * kW);
  if (e == cudaSuccess) e = nalloc(m, &m->dZ, (size_t)np * kZ);
  if (e == cudaSuccess) e = nalloc(m, &m->ptr, (size_t)n + 1);
  if (e == cudaSuccess) e = nalloc(m, &m->lpart, (size_t)(np * kOut + 255) / 256 + 1);
  if (e == cudaSuccess) e = nalloc(m, &m->err, 1);
  if (e == cudaSuccess) e = nalloc(m, &m->WdT, (size_t)kW * kInK);
  for (int l = 0; l < kLayers && e == cudaSuccess; ++l)
    e = nalloc(m, &m->WlT[l], (size_t)kZ * kW);
  if (e == cudaSuccess) e = nalloc(m, &m->part, (size_t)kMaxSplits * kW * kZ);
  if (e == cudaSuccess) e = nalloc(m, &m->feat, (size_t)n * kIn);
  return e;
}

// brackets one GEMM launch with an event pair when profiling is on
struct GemmTimer {
  mst_mpnn* m;
  mst_mpnn::GemmRec* r = nullptr;
  GemmTimer(mst_mpnn* mm, double flops, double bytes) : m(mm) {
    if (!m->prof) return;
    if (m->n_recs == m->recs.size()) {
      mst_mpnn::GemmRec g;
      if (cudaEventCreate(&g.a) != cudaSuccess || cudaEventCreate(&g.b) != cudaSuccess) return;
      m->recs.push_back(g);
    }
    r = &m->recs[m->n_recs++];
    r->flops = flops;
    r->bytes = bytes;
    cudaEventRecord(r->a, 0);
  }
  ~GemmTimer() {
    if (r) cudaEventRecord(r->b, 0);
  }
};

// what a product writes beside (or instead of) C
struct Side {
  const float* Cin = nullptr;  // residual added
  __nv_bfloat16* Cb = nullptr;
  uint16_t* gate = nullptr;
};

cudaError_t gemm(mst_mpnn* m, const __nv_bfloat16* A, const __nv_bfloat16* B, float* C, int M,
                 int N, int K, int ldc, const float* bias, int relu, const Side& side = Side()) {
  GemmTimer timer(m, 2.0 * M * N * K,
                  2.0 * ((double)M * K + (double)N * K) + (C ? 4.0 * M * N : 0.0) +
                      (side.Cin ? 4.0 * M * N : 0.0) + (side.Cb ? 2.0 * M * N : 0.0) +
                      (side.gate ? M * N / 8.0 : 0.0));
  mst::tc::GemmArgs g{};
  g.A = A;
  g.B = B;
  g.C = C;
  g.Cin = side.Cin;
  g.Cb = side.Cb;
  g.gate = side.gate;
  g.bias = bias;
  g.M = M;
  g.N = N;
  g.K = K;
  g.ldc = ldc;
  g.ldcb = ldc;
  g.relu = relu;
  g.err = m->err;
  return mst::tc::gemm(g, 0);
}

cudaError_t transpose(const __nv_bfloat16* src, int n, int w, int n_pad, __nv_bfloat16* dst) {
  dim3 grid((n_pad + 31) / 32, (w + 31) / 32), block(32, 8);
  k_transpose_bf16<<<grid, block>>>(src, n, w, n_pad, dst);
  return cudaGetLastError();
}

// SMs of the device (read once, thread-safe; it only sizes grids)
int sm_count() {
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    n = 152;
  return n;
}

// Weight gradients C[M][N] = A^T B over the n cells: A [n][a_cols], B
// [n][b_cols] with M <= a_cols, N <= b_cols (<= 256).  Split over up to
// kMaxSplits CTAs per output tile, then add the partial products in a fixed
// order.
cudaError_t gemm_wgrad(mst_mpnn* m, const __nv_bfloat16* A, int a_cols, const __nv_bfloat16* B,
                       int b_cols, float* C, int M, int N, int n, int ldc) {
  const int K = pad64(n);
  const int kt = K / mst::tc::kBK;  // K tiles
  // about two CTAs per SM over the output tiles, each with at least 4 K tiles
  static const int sms = sm_count();
  const int n_tiles = ((M + mst::tc::kBM - 1) / mst::tc::kBM) * ((N + mst::tc::kBN - 1) / mst::tc::kBN);
  const int splits =
      std::min(kMaxSplits, std::max(1, std::min(2 * sms / std::max(1, n_tiles), kt / 4)));
  const int chunk = ((kt + splits - 1) / splits) * mst::tc::kBK;
  const int used = (K + chunk - 1) / chunk;
  mst::tc::GemmArgs g{};
  g.A = A;
  g.B = B;
  g.C = m->part;
  g.M = M;
  g.N = N;
  g.K = K;
  g.ldc = ldc;
  g.err = m->err;
  g.k_chunk = chunk;
  cudaError_t e;
  {
    GemmTimer timer(m, 2.0 * M * N * K,
                    2.0 * ((double)M * K + (double)N * K) + 4.0 * used * M * N);
    if (!mst::tc::gemm_tma_rows(g, n, a_cols, b_cols, 0, &e)) {
      // k_gemm_bf16 reads [M][K] and [N][K]
      const size_t nk = pad64(m->cap);
      e = cudaSuccess;
      if (!m->tA) e = nalloc(m, &m->tA, kZ * nk);
      if (e == cudaSuccess && !m->tB) e = nalloc(m, &m->tB, kZ * nk);
      if (e == cudaSuccess) e = transpose(A, n, a_cols, K, m->tA);
      if (e == cudaSuccess) e = transpose(B, n, b_cols, K, m->tB);
      g.A = m->tA;
      g.B = m->tB;
      if (e == cudaSuccess) e = mst::tc::gemm(g, 0);
    }
  }
  if (e != cudaSuccess) return e;
  const size_t mn = (size_t)M * ldc;
  return mst::tc::reduce_splits(m->part, used, mn, C);
}

// bias gradient from the blocks' column sums in the split-K partial buffer
// (free between weight-gradient GEMMs)
void colsum(mst_mpnn* m, int blocks, int w, float* out) {
  k_colsum_parts<<<(w + 31) / 32, 1024>>>(m->part, blocks, w, out);
}

// blocks of the kernels that walk cells by warps: up to 8 an SM, so that a warp
// has several cells where there are many
int cell_blocks(int n_pad) {
  static const int sms = sm_count();
  return std::min((n_pad + 2 * kCellWarps - 1) / (2 * kCellWarps), 8 * sms);
}

// forward over the graph loaded in m (n cells); Y = outputs
cudaError_t forward(mst_mpnn* m, int n) {
  const int np = pad128(n);
  Side side;
  side.gate = m->gate[0];
  cudaError_t e =
      gemm(m, m->X, P(m, kWe).wb, m->H[0], np, kW, kInK, kW, P(m, kBe).w, 1, side);
  for (int l = 0; l < kLayers && e == cudaSuccess; ++l) {
    k_build_z<<<cell_blocks(np), 32 * kCellWarps>>>(m->H[l], m->ptr, m->nbr, n, np, m->Z[l]);
    // h_{l+1}: the next layer reads it in FP32, the decoder as its BF16 operand
    const bool last = l + 1 == kLayers;
    side.Cin = m->H[l];
    side.gate = m->gate[l + 1];
    side.Cb = last ? m->Hb : nullptr;
    e = gemm(m, m->Z[l], P(m, wl(l)).wb, last ? nullptr : m->H[l + 1], np, kW, kZ, kW,
             P(m, bl(l)).w, 1, side);
  }
  if (e == cudaSuccess)
    e = gemm(m, m->Hb, P(m, kWd).wb, m->Y, np, kOut, kW, kOut, P(m, kBd).w, 0);
  return e == cudaSuccess ? cudaGetLastError() : e;
}

// backward of the mean squared error against m->T; gradients into W[].g;
// returns the loss through *loss
cudaError_t backward(mst_mpnn* m, int n, double* loss) {
  const int np = pad128(n), nb = np / 64, cb = cell_blocks(np);
  cudaError_t e = cudaSuccess;
  {
    WeightT t;
    for (int l = 0; l < kLayers; ++l) {  // Wl^T [256][128]
      t.src[l] = P(m, wl(l)).wb;
      t.dst[l] = m->WlT[l];
      t.rows[l] = t.pad[l] = kW;
      t.cols[l] = kZ;
    }
    t.src[kLayers] = P(m, kWd).wb;  // Wd^T [128][64], K = 4 padded with zeros
    t.dst[kLayers] = m->WdT;
    t.rows[kLayers] = kOut;
    t.cols[kLayers] = kW;
    t.pad[kLayers] = kInK;
    k_transpose_weights<<<dim3(kW / 32, kZ / 32, kLayers + 1), dim3(32, 8)>>>(t);
  }
  // decoder: dWd = dY^T H3, dbd = colsum dY, dH3 = dY Wd
  k_mse<<<nb, 256>>>(m->Y, m->T, n, m->dYb, m->lpart, m->part);
  colsum(m, nb, kOut, P(m, kBd).g);
  e = gemm_wgrad(m, m->dYb, kInK, m->Hb, kW, P(m, kWd).g, kOut, kW, n, kW);
  if (e == cudaSuccess) e = gemm(m, m->dYb, m->WdT, m->dH, np, kW, kInK, kW, nullptr, 0);
  if (e == cudaSuccess)
    k_back<false><<<cb, 32 * kCellWarps>>>(m->dH, nullptr, nullptr, nullptr,
                                           reinterpret_cast<const uint8_t*>(m->gate[kLayers]), n,
                                           np, nullptr, m->dPb, m->part);
  for (int l = kLayers - 1; l >= 0 && e == cudaSuccess; --l) {
    // dbl, dWl = dP^T Z, dZ = dP Wl, then dH_l and the dP below it
    colsum(m, cb, kW, P(m, bl(l)).g);
    e = gemm_wgrad(m, m->dPb, kW, m->Z[l], kZ, P(m, wl(l)).g, kW, kZ, n, kZ);
    if (e == cudaSuccess) e = gemm(m, m->dPb, m->WlT[l], m->dZ, np, kZ, kW, kZ, nullptr, 0);
    if (e != cudaSuccess) break;
    std::swap(m->dH, m->dHn);  // dHn = dH_{l+1}
    k_back<true><<<cb, 32 * kCellWarps>>>(m->dHn, m->dZ, m->ptr, m->nbr,
                                          reinterpret_cast<const uint8_t*>(m->gate[l]), n, np,
                                          l > 0 ? m->dH : nullptr, m->dPb, m->part);
    e = cudaGetLastError();
  }
  // encoder: dbe, dWe = dP0^T X
  if (e == cudaSuccess) {
    colsum(m, cb, kW, P(m, kBe).g);
    e = gemm_wgrad(m, m->dPb, kW, m->X, kInK, P(m, kWe).g, kW, kInK, n, kInK);
  }
  if (e != cudaSuccess) return e;
  std::vector<double> part(nb);
  e = cudaMemcpy(part.data(), m->lpart, sizeof(double) * nb, cudaMemcpyDeviceToHost);
  double l = 0.0;
  for (double x : part) l += x;
  *loss = l / (double)(n * kOut);
  return e == cudaSuccess ? cudaGetLastError() : e;
}

}  // namespace
namespace {

// features [n][16] FP32 -> X [np][64] BF16 (zero padding), eight columns a thread
__global__ void k_features(const float* __restrict__ f, int n, int np,
                           __nv_bfloat16* __restrict__ x) {
  constexpr int kPer = kInK / 8;
  const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i >= (size_t)np * kPer) return;
  const int r = (int)(i / kPer), c = (int)(i % kPer) * 8;
  uint2 lo = make_uint2(0u, 0u), hi = lo;
  if (r < n && c < kIn) {
    const float4* p = reinterpret_cast<const float4*>(f + (size_t)r * kIn + c);
    lo = bf16x4(p[0]);
    hi = bf16x4(p[1]);
  }
  reinterpret_cast<uint4*>(x)[i] = make_uint4(lo.x, lo.y, hi.x, hi.y);
}

// xorshift64* uniform in [-1, 1)
double urand(uint64_t& s) {
  s ^= s >> 12;
  s ^= s << 25;
  s ^= s >> 27;
  const uint64_t r = s * 2685821657736338717ull;
  return (double)(r >> 11) * (2.0 / 9007199254740992.0) - 1.0;
}

}  // namespace

extern "C" {

int mst_mpnn_num_params(void) {
  return kW * kInK + kW + kLayers * (kW * kZ + kW) + kOut * kW + kOut;
}

mst_status mst_mpnn_create(uint64_t seed, mst_mpnn** out) {
  if (!out) return mst_internal_fail(MST_EINVAL, "NULL argument");
  mst_mpnn* m = new mst_mpnn();
  const int shapes[2 * (kLayers + 2)][2] = {{kW, kInK}, {1, kW}, {kW, kZ}, {1, kW}, {kW, kZ},
                                            {1, kW},   {kW, kZ}, {1, kW}, {kOut, kW}, {1, kOut}};
  uint64_t st = seed * 0x9E3779B97F4A7C15ull + 1;
  const size_t all = (size_t)mst_mpnn_num_params();
  cudaError_t e = cudaSuccess;
  for (float** q : {&m->w, &m->g, &m->m1, &m->v1}) {
    if (e == cudaSuccess) e = cudaMalloc(q, all * 4);
    if (e == cudaSuccess) e = cudaMemset(*q, 0, all * 4);
  }
  if (e == cudaSuccess) e = cudaMalloc(&m->wb, all * 2);
  size_t off = 0;
  for (int i = 0; i < 2 * (kLayers + 2) && e == cudaSuccess; ++i) {
    MpnnParam& p = m->W[i];
    p.rows = shapes[i][0];
    p.cols = shapes[i][1];
    const size_t n = (size_t)p.size();
    std::vector<float> w(n, 0.f);
    if (p.rows > 1) {
      // Glorot-uniform over the real fan-in (the first layer's is 16)
      const int fan_in = (i == kWe) ? kIn : p.cols;
      const double a = std::sqrt(6.0 / (fan_in + p.rows));
      for (int r = 0; r < p.rows; ++r)
        for (int c = 0; c < p.cols; ++c)
          w[(size_t)r * p.cols + c] = (i == kWe && c >= kIn) ? 0.f : (float)(a * urand(st));
    }
    std::vector<__nv_bfloat16> wb(n);
    for (size_t k = 0; k < n; ++k) wb[k] = __float2bfloat16_rn(w[k]);
    // (every tensor but the last is a multiple of 8 values: 16-byte operands)
    p.w = m->w + off;
    p.g = m->g + off;
    p.m = m->m1 + off;
    p.v = m->v1 + off;
    p.wb = m->wb + off;
    off += n;
    e = cudaMemcpy(p.w, w.data(), n * 4, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(p.wb, wb.data(), n * 2, cudaMemcpyHostToDevice);
  }
  if (e != cudaSuccess) {
    mst_mpnn_destroy(m);
    return mst_internal_fail(MST_ECUDA, std::string("mpnn create: ") + cudaGetErrorString(e));
  }
  *out = m;
  return MST_OK;
}

mst_status mst_mpnn_destroy(mst_mpnn* m) {
  if (!m) return MST_OK;
  cudaDeviceSynchronize();
  for (float* p : {m->w, m->g, m->m1, m->v1}) cudaFree(p);
  cudaFree(m->wb);
  for (void* p : m->bufs) cudaFree(p);
  cudaFree(m->nbr);
  for (auto& r : m->recs) {
    cudaEventDestroy(r.a);
    cudaEventDestroy(r.b);
  }
  delete m;
  return MST_OK;
}

mst_status mst_mpnn_profile(mst_mpnn* m, int on) {
  if (!m) return mst_internal_fail(MST_EINVAL, "NULL network");
  m->prof = on != 0;
  m->n_recs = 0;
  return MST_OK;
}

mst_status mst_mpnn_profile_read(mst_mpnn* m, double out[4]) {
  if (!m || !out) return mst_internal_fail(MST_EINVAL, "NULL argument");
  cudaError_t e = cudaDeviceSynchronize();
  if (e != cudaSuccess)
    return mst_internal_fail(MST_ECUDA, std::string("mpnn profile: ") + cudaGetErrorString(e));
  double ms = 0.0, fl = 0.0, by = 0.0;
  for (size_t i = 0; i < m->n_recs; ++i) {
    float t = 0.f;
    e = cudaEventElapsedTime(&t, m->recs[i].a, m->recs[i].b);
    if (e != cudaSuccess)
      return mst_internal_fail(MST_ECUDA, std::string("mpnn profile: ") + cudaGetErrorString(e));
    ms += t;
    fl += m->recs[i].flops;
    by += m->recs[i].bytes;
  }
  out[0] = ms;
  out[1] = fl;
  out[2] = by;
  out[3] = (double)m->n_recs;
  m->n_recs = 0;
  return MST_OK;
}

mst_status mst_mpnn_set_graph(mst_mpnn* m, int n, const float* features, const int* nbr_ptr,
                              const int* nbr) {
  if (!m || n <= 0 || !features || !nbr_ptr || !nbr)
    return mst_internal_fail(MST_EINVAL, "bad graph arguments");
  const int n_nbr = nbr_ptr[n];
  int bad = nbr_ptr[0] < 0;  // (no early exit: the loops vectorise)
  for (int i = 0; i < n; ++i) bad |= nbr_ptr[i + 1] < nbr_ptr[i];
  if (bad) return mst_internal_fail(MST_EINVAL, "nbr_ptr not ascending from 0 on");
  for (int i = 0; i < n_nbr; ++i) bad |= (unsigned)nbr[i] >= (unsigned)n;
  if (bad) return mst_internal_fail(MST_EINVAL, "neighbour id out of range");
  cudaError_t e = ensure_cap(m, n, std::max(n_nbr, 1));
  float* df = m->feat;
  if (e == cudaSuccess)
    e = cudaMemcpy(df, features, sizeof(float) * (size_t)n * kIn, cudaMemcpyHostToDevice);
  if (e == cudaSuccess)
    e = cudaMemcpy(m->ptr, nbr_ptr, sizeof(int) * ((size_t)n + 1), cudaMemcpyHostToDevice);
  if (e == cudaSuccess && n_nbr)
    e = cudaMemcpy(m->nbr, nbr, sizeof(int) * (size_t)n_nbr, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    const int np = pad128(n);
    const size_t cnt = (size_t)np * (kInK / 8);
    k_features<<<(unsigned)((cnt + 255) / 256), 256>>>(df, n, np, m->X);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaDeviceSynchronize();
  if (e != cudaSuccess) return mst_internal_fail(MST_ECUDA, std::string("mpnn graph: ") + cudaGetErrorString(e));
  m->n = n;
  return MST_OK;
}

mst_status mst_mpnn_set_targets(mst_mpnn* m, const float* t) {
  if (!m || !t || m->n <= 0) return mst_internal_fail(MST_EINVAL, "no graph or NULL targets");
  cudaError_t e = cudaMemcpy(m->T, t, sizeof(float) * (size_t)m->n * kOut, cudaMemcpyHostToDevice);
  if (e != cudaSuccess) return mst_internal_fail(MST_ECUDA, cudaGetErrorString(e));
  return MST_OK;
}

mst_status mst_mpnn_forward(mst_mpnn* m, float* y) {
  if (!m || m->n <= 0) return mst_internal_fail(MST_EINVAL, "no graph");
  cudaError_t e = cudaMemset(m->err, 0, sizeof(int));
  if (e == cudaSuccess) e = forward(m, m->n);
  int herr = 0;
  if (e == cudaSuccess) e = cudaMemcpy(&herr, m->err, sizeof(int), cudaMemcpyDeviceToHost);
  if (e == cudaSuccess && y)
    e = cudaMemcpy(y, m->Y, sizeof(float) * (size_t)m->n * kOut, cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) return mst_internal_fail(MST_ECUDA, std::string("mpnn forward: ") + cudaGetErrorString(e));
  if (herr == 2)
    return mst_internal_fail(MST_ECUDA, "mpnn forward: shared memory not 1024-byte aligned for TMA");
  if (herr) return mst_internal_fail(MST_ETIMEOUT, "mpnn forward: a tensor-core wait timed out");
  return MST_OK;
}

mst_status mst_mpnn_backward(mst_mpnn* m, double* loss) {
  if (!m || m->n <= 0) return mst_internal_fail(MST_EINVAL, "no graph");
  double l = 0.0;
  cudaError_t e = backward(m, m->n, &l);
  int herr = 0;
  if (e == cudaSuccess) e = cudaMemcpy(&herr, m->err, sizeof(int), cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) return mst_internal_fail(MST_ECUDA, std::string("mpnn backward: ") + cudaGetErrorString(e));
  if (herr == 2)
    return mst_internal_fail(MST_ECUDA, "mpnn backward: shared memory not 1024-byte aligned for TMA");
  if (herr) return mst_internal_fail(MST_ETIMEOUT, "mpnn backward: a tensor-core wait timed out");
  if (loss) *loss = l;
  return MST_OK;
}

// all parameters (which = 0) or gradients (1), in the order We, be, W0, b0,
// W1, b1, W2, b2, Wd, bd, each row-major [outputs][inputs]
mst_status mst_mpnn_get(mst_mpnn* m, int which, float* out) {
  if (!m || !out) return mst_internal_fail(MST_EINVAL, "NULL argument");
  const cudaError_t e = cudaMemcpy(out, which ? m->g : m->w, sizeof(float) * mst_mpnn_num_params(),
                                   cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) return mst_internal_fail(MST_ECUDA, cudaGetErrorString(e));
  return MST_OK;
}

mst_status mst_mpnn_set_weights(mst_mpnn* m, const float* w) {
  if (!m || !w) return mst_internal_fail(MST_EINVAL, "NULL argument");
  size_t off = 0;
  for (auto& p : m->W) {
    const size_t n = (size_t)p.size();
    std::vector<__nv_bfloat16> wb(n);
    for (size_t k = 0; k < n; ++k) wb[k] = __float2bfloat16_rn(w[off + k]);
    cudaError_t e = cudaMemcpy(p.w, w + off, n * 4, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(p.wb, wb.data(), n * 2, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) return mst_internal_fail(MST_ECUDA, cudaGetErrorString(e));
    off += n;
  }
  return MST_OK;
}

mst_status mst_mpnn_adam_step(mst_mpnn* m, float lr) {
  if (!m) return mst_internal_fail(MST_EINVAL, "NULL network");
  m->step += 1;
  const float b1 = 0.9f, b2 = 0.999f;
  const float c1 = 1.f - std::pow(b1, (float)m->step), c2 = 1.f - std::pow(b2, (float)m->step);
  AdamTensors t;
  int most = 0;
  for (int i = 0; i < 2 * (kLayers + 2); ++i) {
    const MpnnParam& p = m->W[i];
    t.w[i] = p.w;
    t.m[i] = p.m;
    t.v[i] = p.v;
    t.g[i] = p.g;
    t.wb[i] = p.wb;
    t.n[i] = p.size();
    most = std::max(most, p.size());
  }
  k_adam<<<dim3((most + 255) / 256, 2 * (kLayers + 2)), 256>>>(t, lr, b1, b2, c1, c2);
  cudaError_t e = cudaDeviceSynchronize();
  if (e != cudaSuccess) return mst_internal_fail(MST_ECUDA, cudaGetErrorString(e));
  return MST_OK;
}


mst_status mst_set_wait_limit(long long polls) {
  mst::tc::g_wait_limit.store(polls < 0 ? -1 : polls, std::memory_order_relaxed);
  return MST_OK;
}

mst_status mst_tc_gemm_check(const uint16_t* A, const uint16_t* B, const float* bias, float* C,
                             int M, int N, int K, int relu, int layout) {
  if (!A || !B || !C || M <= 0 || N <= 0 || K <= 0 || K % mst::tc::kBK != 0)
    return mst_internal_fail(MST_EINVAL, "bad GEMM arguments (K must be a multiple of 64)");
  __nv_bfloat16 *dA = nullptr, *dB = nullptr;
  float *dC = nullptr, *dbias = nullptr;
  int* derr = nullptr;
  auto cleanup = [&]() {
    cudaFree(dA);
    cudaFree(dB);
    cudaFree(dC);
    cudaFree(dbias);
    cudaFree(derr);
  };
  cudaError_t e = cudaMalloc(&dA, sizeof(uint16_t) * (size_t)M * K);
  if (e == cudaSuccess) e = cudaMalloc(&dB, sizeof(uint16_t) * (size_t)N * K);
  if (e == cudaSuccess) e = cudaMalloc(&dC, sizeof(float) * (size_t)M * N);
  if (e == cudaSuccess && bias) e = cudaMalloc(&dbias, sizeof(float) * N);
  if (e == cudaSuccess) e = cudaMalloc(&derr, sizeof(int));
  if (e == cudaSuccess) e = cudaMemcpy(dA, A, sizeof(uint16_t) * (size_t)M * K, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(dB, B, sizeof(uint16_t) * (size_t)N * K, cudaMemcpyHostToDevice);
  if (e == cudaSuccess && bias) e = cudaMemcpy(dbias, bias, sizeof(float) * N, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemset(derr, 0, sizeof(int));
  if (e == cudaSuccess) {
    mst::tc::GemmArgs g{};
    g.A = dA;
    g.B = dB;
    g.C = dC;
    g.bias = dbias;
    g.M = M;
    g.N = N;
    g.K = K;
    g.ldc = N;
    g.relu = relu;
    g.err = derr;
    if (layout == 1) {  // the other assignment of the two strides
      g.lbo = mst::tc::kSBO;
      g.sbo = mst::tc::kLBO;
    }
    if (layout >= mst::tc::kBK && layout % mst::tc::kBK == 0 && !bias && !relu) {
      // split K in chunks of `layout`, partial products reduced in order
      const int splits = (K + layout - 1) / layout;
      float* part = nullptr;
      e = cudaMalloc(&part, sizeof(float) * (size_t)splits * M * N);
      if (e == cudaSuccess) {
        g.C = part;
        g.k_chunk = layout;
        e = mst::tc::gemm(g, 0);
        const size_t mn = (size_t)M * N;
        if (e == cudaSuccess) e = mst::tc::reduce_splits(part, splits, mn, dC);
        if (e == cudaSuccess) e = cudaDeviceSynchronize();
        cudaFree(part);
      }
    } else {
      e = mst::tc::gemm(g, 0);
    }
  }
  int herr = 0;
  if (e == cudaSuccess) e = cudaDeviceSynchronize();
  if (e == cudaSuccess) e = cudaMemcpy(&herr, derr, sizeof(int), cudaMemcpyDeviceToHost);
  if (e == cudaSuccess) e = cudaMemcpy(C, dC, sizeof(float) * (size_t)M * N, cudaMemcpyDeviceToHost);
  cleanup();
  if (e != cudaSuccess) return mst_internal_fail(MST_ECUDA, std::string("gemm: ") + cudaGetErrorString(e));
  if (herr == 2)
    return mst_internal_fail(MST_ECUDA, "gemm: shared memory not 1024-byte aligned for TMA");
  if (herr) return mst_internal_fail(MST_ETIMEOUT, "gemm: a tensor-core wait timed out");
  return MST_OK;
}

}  // extern "C"
