// Expert layers over dense fp16 weights [E, N, K] on the 5th-generation tensor cores.
//
//   out^T tile [128 weight rows x up to 256 batch rows] = W_tile [128 x K] * x_tile^T [K x 256]
//
// Bound: HBM (the experts' weights) at small batches, the tensor pipe at large ones: one tcgen05.mma of
// width N takes N / 2 clocks (N = 16: 9, 32: 16, 64: 32, 128: 64, 256: 128).  Both operands come from
// shared memory, staged by TMA in the 128-byte swizzled K-major layout; the accumulator sits in 256
// tensor-memory columns.
//
//   warp 0  weights: one TMA tile of 128 rows x 64 k per block
//   warp 1  MMA: four per 64-k block, by an elected thread; commits recycle both rings
//   warp 3  x: one TMA tile of 64 k x nb batch rows per block; rows past m read zero
//   warps 4..11  two groups of four warps (128 TMEM lanes each) drain one half of the batch columns
//           each: one rounding to fp16, transpose through shared memory, whole-line stores.
// Tiles are walked persistently, batch tiles fastest, so CTAs running together share a weight
// tile in L2.  Every wait is bounded and reports through the device status word.
//
// The dense form of src/runtime/contrib/cutlass/fp16_group_gemm.cu:39-64.
#include "umma_gemm.h"

#include <cuda.h>

#include <cstring>

#include "dequant.cuh"
#include "gemv_cluster.cuh"
#include "tensormap.h"
#include "umma_common.cuh"

namespace rb200 {
namespace um {

constexpr int kDrainWarps = 8;
constexpr int kFirstDrainWarp = 4;
constexpr int kThreads = (kFirstDrainWarp + kDrainWarps) * 32;
constexpr int kTileRows = 128;
constexpr int kKBlock = 64;                 // k per MMA block (4 x K=16)
constexpr int kWStageBytes = kTileRows * kKBlock * 2;
constexpr int kWStages = 3;
constexpr int kMaxXStages = 8;
constexpr int kTmemCols = 256;              // the accumulator
constexpr int kMaxNb = 256;
constexpr int kEpiStageBytes = 2 * 2 * 16 * kTileRows * 2;  // per group: two 16 x 128 fp16 buffers

constexpr int kMaxExperts = 64;

struct Params {
  GemvParams g;
  int nb;          // batch rows per tile = MMA N (multiple of 32, <= 256)
  int x_stages;
  // rows [indptr[e-1], indptr[e]) of x / out belong to expert e (indptr: device, end offsets)
  const int64_t* indptr;
  int indptr_has_prev;      // the first group starts at indptr[-1] (a sub-range of a longer table), not at row 0
  int num_experts;
};

inline size_t smem_bytes(int nb, int x_stages) {
  return 1024 + (size_t)x_stages * nb * 128 + (size_t)kWStages * kWStageBytes + kEpiStageBytes +
         (size_t)(2 * kWStages + 2 * kMaxXStages + 4) * 8 + 16 + (3 * kMaxExperts + 4) * sizeof(int);
}

using gc::tma_load_2d;
using ug::make_b_desc;
using ug::tc_commit;
using ug::tc_fence_after;
using ug::tc_fence_before;
using ug::tc_ld16;
using ug::elect_one;
using ug::tmem_alloc;
using ug::tmem_dealloc;
using ug::tmem_relinquish;

// D[tmem] (+)= A[smem desc] * B[smem desc]; kind::f16, fp32 accumulate
__device__ __forceinline__ void tc_mma_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                          uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d(void* smem_dst, const CUtensorMap* map, int c0, int c1, int c2,
                                            uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
          smem_u32(smem_dst)),
      "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(smem_u32(bar))
      : "memory");
}

// Work item: one (expert, 128-row weight tile, batch tile).  Items are numbered expert by expert,
// batch tiles fastest; the tables live in shared memory (built once per CTA from indptr).
struct Tile {
  int e, n_tile;
  int m0, m_end;  // first batch row of the tile, end of the expert's rows
};
struct TileTables {
  int base[kMaxExperts + 1];
  int row_begin[kMaxExperts];
  int row_end[kMaxExperts];
};
__device__ __forceinline__ Tile get_tile(const TileTables& tt, int num_experts, int nb, int t) {
  int e = 0;
  while (e + 1 < num_experts && t >= tt.base[e + 1]) ++e;
  const int local = t - tt.base[e];
  const int rows = tt.row_end[e] - tt.row_begin[e];
  const int mt = (rows + nb - 1) / nb;
  Tile tl;
  tl.e = e;
  tl.n_tile = local / mt;
  tl.m0 = tt.row_begin[e] + (local % mt) * nb;
  tl.m_end = tt.row_end[e];
  return tl;
}

__global__ void __launch_bounds__(kThreads, 1)
    umma_gemm_kernel(const Params pp, const __grid_constant__ CUtensorMap tmap_x,
                     const __grid_constant__ CUtensorMap tmap_w) {
  extern __shared__ uint8_t smem_raw[];
  const GemvParams& p = pp.g;
  // 1 KB alignment as an offset from the array (a pointer rebuilt from an integer would turn
  // every shared-memory access of the drain warps into a generic one)
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const int nb = pp.nb;
  const int x_stages = pp.x_stages;
  const int x_stage_bytes = nb * 128;
  uint8_t* x_ring = smem;
  uint8_t* w_ring = smem + (size_t)x_stages * x_stage_bytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(w_ring + (size_t)kWStages * kWStageBytes + kEpiStageBytes);
  uint64_t* w_full = bars;
  uint64_t* w_empty = w_full + kWStages;
  uint64_t* x_full = w_empty + kWStages;
  uint64_t* x_empty = x_full + kMaxXStages;
  uint64_t* d_full = x_empty + kMaxXStages;
  uint64_t* d_empty = d_full + 1;
  uint64_t* e_bar = d_empty + 1;  // one per drain group: epilogue staging hand-over
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(e_bar + 2);
  TileTables& tt = *reinterpret_cast<TileTables*>(tmem_holder + 4);
  __half* e_stage = reinterpret_cast<__half*>(w_ring + (size_t)kWStages * kWStageBytes);  // [2 groups][2][16][128]

  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;

  if (tid == 0) {
    for (int s = 0; s < kWStages; ++s) {
      mbar_init(&w_full[s], 1);
      mbar_init(&w_empty[s], 1);
    }
    for (int s = 0; s < x_stages; ++s) {
      mbar_init(&x_full[s], 1);
      mbar_init(&x_empty[s], 1);
    }
    mbar_init(d_full, 1);
    mbar_init(d_empty, kDrainWarps);
    mbar_init(&e_bar[0], 4);
    mbar_init(&e_bar[1], 4);
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_holder, kTmemCols);
    tmem_relinquish();
  }
  const int n_tiles = p.n / kTileRows;
  if (tid < pp.num_experts) {
    const int64_t r0 = (tid || pp.indptr_has_prev) ? pp.indptr[tid - 1] : 0;
    int64_t r1 = pp.indptr[tid];
    if (r1 > p.m) r1 = p.m;  // never past the rows x / out hold
    tt.row_begin[tid] = (int)r0;
    tt.row_end[tid] = r1 > r0 ? (int)r1 : (int)r0;
  }
  tc_fence_before();
  __syncthreads();
  if (tid == 0) {
    int acc = 0;
    for (int e = 0; e < pp.num_experts; ++e) {
      tt.base[e] = acc;
      acc += n_tiles * ((tt.row_end[e] - tt.row_begin[e] + pp.nb - 1) / pp.nb);
    }
    tt.base[pp.num_experts] = acc;
  }
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;

  const int kb_total = p.k / kKBlock;             // MMA blocks along k
  const int total_tiles = tt.base[pp.num_experts];
  const int ne = pp.num_experts;
  bool ok = true;

  if (warp == 0) {
    // ============================================================ weight tiles (TMA)
    int ws = 0;
    uint32_t wph = 0;
    for (int t = blockIdx.x; ok && t < total_tiles; t += gridDim.x) {
      const Tile tile = get_tile(tt, ne, nb, t);
      for (int kb = 0; kb < kb_total; ++kb) {
        if (!mbar_wait_parked(&w_empty[ws], wph ^ 1u, p.status)) {
          ok = false;
          break;
        }
        if (lane == 0) {
          mbar_arrive_expect_tx(&w_full[ws], (uint32_t)kWStageBytes);
          tma_load_3d(w_ring + (size_t)ws * kWStageBytes, &tmap_w, kb * kKBlock, tile.n_tile * kTileRows, tile.e, &w_full[ws]);
        }
        __syncwarp();
        if (++ws == kWStages) {
          ws = 0;
          wph ^= 1u;
        }
      }
    }
  } else if (warp == 1) {
    // ============================================================ MMA issuer (one elected thread)
    // The whole warp runs the loop and waits; elect.sync picks the issuing thread, from which the compiler
    // knows that operands may stay in uniform registers (with `if (lane == 0)` and descriptors rebuilt per
    // instruction the issue loop itself took 108 clocks per MMA).
    const uint32_t idesc = (1u << 4) | ((uint32_t)(nb >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
    const bool leader = elect_one();
    const uint64_t x_desc0 = make_b_desc(smem_u32(x_ring));
    const uint64_t w_desc0 = make_b_desc(smem_u32(w_ring));
    uint64_t x_desc = x_desc0;
    int xs = 0;
    uint32_t xph = 0;
    uint32_t dph = 1;          // accumulator hand-back phase
    int ws = 0;
    uint32_t wph = 0;
    for (int t = blockIdx.x; ok && t < total_tiles; t += gridDim.x, dph ^= 1u) {
      if (!mbar_wait_parked(d_empty, dph, p.status)) {
        ok = false;
        break;
      }
      tc_fence_after();
      uint32_t acc_on = 0u;
      for (int kb = 0; kb < kb_total; ++kb) {
        if (!mbar_wait_parked(&x_full[xs], xph, p.status) || !mbar_wait_parked(&w_full[ws], wph, p.status)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint64_t w_desc = w_desc0 + (uint64_t)(ws * (kWStageBytes >> 4));
        if (leader) {
          tc_mma_ss(tmem_base, w_desc, x_desc, idesc, acc_on);
#pragma unroll
          for (int j = 1; j < 4; ++j) tc_mma_ss(tmem_base, w_desc + j * 2, x_desc + j * 2, idesc, 1u);
          tc_commit(&w_empty[ws]);
          tc_commit(&x_empty[xs]);
        }
        if (++ws == kWStages) {
          ws = 0;
          wph ^= 1u;
        }
        acc_on = 1u;
        x_desc += (uint64_t)(x_stage_bytes >> 4);
        if (++xs == x_stages) {
          xs = 0;
          xph ^= 1u;
          x_desc = x_desc0;
        }
      }
      if (ok && leader) tc_commit(d_full);
      __syncwarp();
    }
  } else if (warp == 3) {
    // ============================================================ x tiles (TMA)
    int xs = 0;
    uint32_t xph = 0;
    for (int t = blockIdx.x; ok && t < total_tiles; t += gridDim.x) {
      const int m0 = get_tile(tt, ne, nb, t).m0;
      for (int kb = 0; kb < kb_total; ++kb) {
        if (!mbar_wait_parked(&x_empty[xs], xph ^ 1u, p.status)) {
          ok = false;
          break;
        }
        if (lane == 0) {
          mbar_arrive_expect_tx(&x_full[xs], (uint32_t)x_stage_bytes);
          tma_load_2d(x_ring + (size_t)xs * x_stage_bytes, &tmap_x, kb * kKBlock, m0, &x_full[xs]);
        }
        __syncwarp();
        if (++xs == x_stages) {
          xs = 0;
          xph ^= 1u;
        }
      }
    }
  } else if (warp >= kFirstDrainWarp) {
    // ============================================================ drain warps
    const int dw = warp - kFirstDrainWarp;
    const int grp = dw >> 2;
    const int w4 = warp & 3;             // TMEM lane quadrant of this warp
    const int row = 32 * w4 + lane;      // weight row held by this thread's TMEM lane
    const uint32_t lane_taddr = (uint32_t)(32 * w4) << 16;
    uint32_t tile_i = 0;
    uint32_t estep = 0;  // staging steps done by this group
    for (int t = blockIdx.x; ok && t < total_tiles; t += gridDim.x, ++tile_i) {
      const Tile tile = get_tile(tt, ne, nb, t);
      const int n_tile = tile.n_tile;
      if (!mbar_wait_parked(d_full, tile_i & 1u, p.status)) {
        ok = false;
        break;
      }
      tc_fence_after();
      const int64_t m0 = tile.m0;
      const int64_t m_end = tile.m_end;
      const int c_begin = grp * (nb / 2), c_end = c_begin + nb / 2;
      const int gj = (dw & 3) * 32 + lane;  // thread index inside the group
      for (int c0 = c_begin; c0 < c_end; c0 += 16, ++estep) {
        if (m0 + c0 >= m_end) break;
        float v[16];
        tc_ld16(lane_taddr | (tmem_base + c0), v);
        // transpose through shared memory: 16 batch rows x 128 weight rows of fp16 (rounded once), so
        // that global stores are whole 256-byte row segments
        __half* st = e_stage + ((grp * 2 + (estep & 1u)) * 16) * kTileRows;
#pragma unroll
        for (int i = 0; i < 16; ++i) st[i * kTileRows + row] = __float2half_rn(v[i]);
        __syncwarp();
        if (lane == 0) mbar_arrive(&e_bar[grp]);
        if (!mbar_wait_parked(&e_bar[grp], estep & 1u, p.status)) {
          ok = false;
          break;
        }
#pragma unroll
        for (int pass = 0; pass < 2; ++pass) {
          const int mi = pass * 8 + (gj >> 4), ch = gj & 15;
          const int64_t m = m0 + c0 + mi;
          if (m < m_end) {
            *reinterpret_cast<uint4*>(p.out + m * p.ldo + (int64_t)n_tile * kTileRows + ch * 8) =
                *reinterpret_cast<const uint4*>(st + mi * kTileRows + ch * 8);
          }
        }
      }
      if (!ok) break;
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(d_empty);
    }
  }

  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

}  // namespace um

int umma_group_gemm_run(const GemvParams& p, int sm_count, const int64_t* indptr, int indptr_has_prev, int num_experts,
                        int64_t w_expert_bytes, cudaStream_t stream) {
  using namespace um;
  RB200_CHECK(indptr != nullptr, "indptr must be non-NULL");
  // coverage: whole 128-row tiles, whole 64-k blocks, TMA-loadable x, 16-byte row stores
  RB200_CHECK(p.n % kTileRows == 0 && p.k % kKBlock == 0 && (reinterpret_cast<uintptr_t>(p.x) & 15u) == 0 &&
                  (p.ldx * 2) % 16 == 0 && (reinterpret_cast<uintptr_t>(p.out) & 15u) == 0 && (p.ldo * 2) % 16 == 0,
              "grouped GEMM needs n %% 128 == 0, k %% 64 == 0 and 16-byte aligned x / out rows (n=%d, k=%d)", p.n, p.k);
  RB200_CHECK(num_experts >= 1 && num_experts <= kMaxExperts, "num_experts=%d outside [1, %d]", num_experts, kMaxExperts);

  Params pp;
  memset(&pp, 0, sizeof(pp));
  pp.g = p;
  pp.indptr = indptr;
  pp.indptr_has_prev = indptr_has_prev;
  pp.num_experts = num_experts;
  // The split of the rows is known only on the device, and an MMA costs its width whether its rows exist
  // or not: 128 or 192 batch rows when the rows, spread evenly over the experts, stay well inside that (an
  // expert above the width takes a second tile), 256 otherwise.
  const long long even = p.m / num_experts;
  if (p.m < kMaxNb) pp.nb = (p.m + 31) / 32 * 32;
  else pp.nb = even <= 96 ? 128 : (even <= 160 ? 192 : kMaxNb);

  const size_t budget = (size_t)227 * 1024;
  pp.x_stages = kMaxXStages;
  while (pp.x_stages > 2 && smem_bytes(pp.nb, pp.x_stages) > budget) --pp.x_stages;

  CUtensorMap tx, tw;
  if (make_tensor_map_2d(&tx, p.x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, (unsigned long long)p.k, (unsigned long long)p.m,
                         (unsigned long long)p.ldx * 2, kKBlock, (unsigned)pp.nb, CU_TENSOR_MAP_SWIZZLE_128B) != 0)
    return -1;
  const unsigned long long dims[3] = {(unsigned long long)p.k, (unsigned long long)p.n, (unsigned long long)num_experts};
  const unsigned long long strides[2] = {(unsigned long long)p.k * 2, (unsigned long long)w_expert_bytes};
  const unsigned box[3] = {kKBlock, kTileRows, 1};
  if (make_tensor_map(&tw, p.w, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B) != 0)
    return -1;

  static thread_local int configured_device = -1;
  int dev = 0;
  RB200_CUDA(cudaGetDevice(&dev));
  if (configured_device != dev) {
    RB200_CUDA(cudaFuncSetAttribute(umma_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    configured_device = dev;
  }
  // one persistent CTA per SM
  umma_gemm_kernel<<<sm_count, kThreads, smem_bytes(pp.nb, pp.x_stages), stream>>>(pp, tx, tw);
  RB200_CUDA(cudaGetLastError());
  return 0;
}

}  // namespace rb200
