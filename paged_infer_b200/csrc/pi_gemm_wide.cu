// Tensor-core GEMM of f32 activations with bf16 weights.
//
//   out[m][r] = row_factor[m] * sum_k W[r][k] * y[m][k]
//
// Activations as in pi_gemm_tc.cu: three bf16 planes whose sum is the f32 value, fetched as ONE tile of 3 x 64 rows, so
// that one product of N 192 per 16 K elements leaves W*p0, W*p1, W*p2 in three groups of accumulator columns.  The
// weights need no widening, so both operands come by TMA and are read from shared memory; sizes need not be multiples of
// the tile (what lies past K, N or M reads as zero).  The CUDA-core kernel reads the matrix once per four activation
// rows; this one once per 64.
//
// The cut: one CTA per SM walks an equal share of the launch's K blocks (tile after tile, K innermost), so that no wave is
// partly filled and loads and products of the next tile run during the epilogue of the last.  A tile cut by a share's
// end is summed over the CTAs that hold it: each parks its part in a workspace and takes a ticket, the last one adds the
// parts in CTA order (the sum does not depend on who is last) and runs the epilogue.  Nobody waits for another CTA.
//
// The sums: two accumulators of one K block each take turns, and the epilogue warps add them up in registers.  The
// tensor pipe cuts its running sum towards zero at every step of 16 K elements, about 1.5e-8 of the sum a step: one chain
// over K 2048 is off by 2e-6 of the result, sums of single K blocks by 1.0e-7 to 1.3e-7, the CUDA-core kernel by 1.2e-7
// (K 5600: 1.7e-7 and 1.8e-7).
//
// What bounds it: hand-overs.  A wait on an mbarrier takes about 190 cycles even when the phase is complete, so the issuing
// threads ask for the next stage before they work on this one.  24000 x 5600, alone, with the split: 83 us for 64 rows, 76 us for 5
// (42 us is the matrix out of HBM); the CUDA-core kernel takes 755 and 104.
//
// Warps 0-7: epilogue; 8: TMA; 9: tensor memory and MMA issue.  Waits are bounded; one that runs out sets the context's error
// word and ends the CTA's other waits, and tickets are taken all the same, so that the counters are zero again behind every
// launch.
#include <algorithm>

#include "pi_common.cuh"

#include "pi_gemm_tc.cuh"
#include "pi_gemm_wide.cuh"

namespace {
using namespace pi_tc;
using pi_wide::Cut;
using pi_wide::cut_at;
using pi_wide::kGivenUp;

constexpr int kWR = pi_wide::kRows, kWC = pi_wide::kCols, kWK = pi_wide::kBlock;
constexpr int kStages = 4, kDrain = 8, kWideThreads = (kDrain + 2) * 32;
constexpr int kDCols = kPlanes * kWC;                // 192 columns of an accumulator
constexpr int kBBytes = kDCols * 128, kStageBytes = kBBytes + kWR * 128;
constexpr int kTileFloats = kWR * kWC;
constexpr size_t kWideSmem = (size_t)kStages * kStageBytes + (size_t)kTileFloats * sizeof(float) + 1024;
static_assert(2 * kDCols <= 512, "TMEM holds 512 columns");
static_assert(kWideSmem >= kMinSmem && kWideSmem <= 225 * 1024, "one CTA per SM");

__device__ __forceinline__ void umma_f16_ss(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}

__global__ void __launch_bounds__(kWideThreads, 1)
gemm_wide_kernel(const GemmParams p, const Cut cut, float* __restrict__ parked, int* __restrict__ tickets,
                 const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_act) {
  constexpr int kTma = kDrain, kMma = kTma + 1;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  float* tile_out = reinterpret_cast<float*>(smem + (size_t)kStages * kStageBytes);   // [64 activation rows][128 weight rows]
  __shared__ __align__(8) unsigned long long bars[2 * kStages + 4];
  __shared__ uint32_t s_tmem;
  __shared__ volatile int s_weight;
  __shared__ EpiPlace s_place[kWC];
  __shared__ int s_n, s_slots[pi_wide::kMaxHolders];

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int cta = blockIdx.x;
  const int pos0 = cut_at(cut, cta), pos1 = cut_at(cut, cta + 1);     // this CTA's K blocks, tile by tile
  const int nkb = cut.nkb, mtiles = cut.mtiles;
  const uint32_t full = smem_u32(&bars[0]), empty = smem_u32(&bars[kStages]), d_full = smem_u32(&bars[2 * kStages]), d_empty = d_full + 16;

  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(full + 8 * s, 1);
      mbar_init(empty + 8 * s, 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(d_full + 8 * b, 1);
      mbar_init(d_empty + 8 * b, kDrain);
    }
    s_weight = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == kMma) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  pi_grid_launch_dependents();   // only now that this CTA holds its tensor memory
  const uint32_t tmem = s_tmem, smem_base = smem_u32(smem);

  auto wait = [&](uint32_t bar, uint32_t parity) {
    return pi_wide::wait_for([&] { return mbar_test(bar, parity); }, &s_weight);
  };
  auto give_up = [&](int code) {
    if (s_weight != kGivenUp && p.err_flag) atomicExch(p.err_flag, code);
    s_weight = kGivenUp;   // the copying thread's 1 is not ahead of us: only waits that counted can run out
  };

  if (warp == kTma) {
    if (pi_elect()) {
      int tile = pos0 / nkb, kb = pos0 % nkb;
      auto load_w = [&](int it, int t, int k) {
        mbar_arrive_expect_tx(full + 8 * (it % kStages), kStageBytes);
        asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
                         smem_base + (it % kStages) * kStageBytes + kBBytes),
                     "l"(&map_w), "r"(full + 8 * (it % kStages)), "r"(k * kWK), "r"(t / mtiles * kWR)
                     : "memory");
      };
      auto load_x = [&](int it, int t, int k) {   // {64 K, 64 rows, 3 planes}
        asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(
                         smem_base + (it % kStages) * kStageBytes),
                     "l"(&map_act), "r"(full + 8 * (it % kStages)), "r"(k * kWK), "r"(t % mtiles * kWC), "r"(0)
                     : "memory");
      };
      const int n = pos1 - pos0, ahead = min(n, kStages);
      for (int it = 0; it < ahead; ++it) load_w(it, (pos0 + it) / nkb, (pos0 + it) % nkb);   // weights never depend on the preceding kernel
      pi_grid_dependency_wait();
      s_weight = 1;
      int it = 0;
      bool free_next = false;   // the next stage is known to be free
      for (; it < n; ++it) {
        if (it >= ahead) {
          if ((!free_next && !wait(empty + 8 * (it % kStages), ((it / kStages) & 1) ^ 1)) || s_weight == kGivenUp) {
            give_up(32);
            break;
          }
          load_w(it, tile, kb);
        }
        free_next = it + 1 >= ahead && mbar_test(empty + 8 * ((it + 1) % kStages), (((it + 1) / kStages) & 1) ^ 1);
        load_x(it, tile, kb);
        if (++kb == nkb) {
          kb = 0;
          ++tile;
        }
      }
      if (s_weight == kGivenUp)   // no copy of this CTA may still be in flight when it leaves
        for (int i = max(0, it - kStages); i < it; ++i) mbar_wait(full + 8 * (i % kStages), (i / kStages) & 1);
    }
  } else if (warp == kMma) {
    // ---- kind::f16, D = f32, A and B in shared memory, K-major bf16, M = 128, N = 192 ---------------------------------
    if (pi_elect()) {
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kDCols >> 3) << 17) | ((uint32_t)(kWR >> 4) << 24);
      const int n = pos1 - pos0;
      bool full_next = false, d_next = true;   // the next stage, the next accumulator are known to be ready
      for (int it = 0; it < n; ++it) {
        const int s = it % kStages, buf = it & 1;
        if ((!d_next && !wait(d_empty + 8 * buf, ((it >> 1) & 1) ^ 1)) ||
            (!full_next && !wait(full + 8 * s, (it / kStages) & 1)) || s_weight == kGivenUp) {
          give_up(33);
          if (it > 0) mbar_wait(d_full + 8 * (buf ^ 1), ((it - 1) >> 1) & 1);   // products under way still use the tensor memory
          break;
        }
        full_next = mbar_test(full + 8 * ((it + 1) % kStages), ((it + 1) / kStages) & 1);
        d_next = it < 1 || mbar_test(d_empty + 8 * (buf ^ 1), (((it + 1) >> 1) & 1) ^ 1);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t stage = smem_base + s * kStageBytes, d = tmem + (uint32_t)(buf * kDCols);
        const uint64_t db = smem_desc(stage), da = smem_desc(stage + kBBytes);
#pragma unroll
        for (int ks = 0; ks < kWK / 16; ++ks)   // 16 K elements: 32 bytes of every row
          umma_f16_ss(d, da + (uint64_t)((ks * 32) >> 4), db + (uint64_t)((ks * 32) >> 4), idesc, ks ? 1u : 0u);
        umma_commit(empty + 8 * s);
        umma_commit(d_full + 8 * buf);
      }
    }
  } else {
    // ---- epilogue: warp w reads TMEM lanes 32 (w % 4).., columns 32 (w / 4).. of each plane: thread = a weight row, 32 columns ---
    const int row = (warp & 3) * 32 + lane, c0 = (warp >> 2) * 32;
    const uint32_t my_d = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c0;
    pi_grid_dependency_wait();   // reads and writes what the preceding kernels use
    int it = 0;
    for (int pos = pos0; pos < pos1;) {
      const int tile = pos / nkb, first = tile * nkb, end = min(first + nkb, pos1);
      const int rt = tile / mtiles, m0 = tile % mtiles * kWC;
      float acc[32];
#pragma unroll
      for (int j = 0; j < 32; ++j) acc[j] = 0.f;
      for (int left = end - pos; left > 0; --left, ++it) {
        const int buf = it & 1;
        int got = 0;
        if (lane == 0) {
          got = (wait(d_full + 8 * buf, (it >> 1) & 1) && s_weight != kGivenUp) ? 1 : 0;
          if (!got) give_up(35);
        }
        got = __shfl_sync(0xffffffffu, got, 0);
        if (!got) continue;   // the parts of this tile stay short, the error word says so
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        uint32_t r[kPlanes][32];
#pragma unroll
        for (int i = 0; i < kPlanes; ++i)
#pragma unroll
          for (int c = 0; c < 32; c += 16) tmem_ld16_issue(my_d + (uint32_t)(buf * kDCols + i * kWC + c), &r[i][c]);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(d_empty + 8 * buf);   // before the sums: the products behind it may start
        // An infinite weight makes infinities or NaN of all products with the second plane, whose values are finite: the row's
        // first column shows it.  Its product with an activation is the first plane's then (inf * 0 of the others is not).  For
        // the warp as a whole: chosen row by row it costs a tenth of the launch.
        if (__any_sync(0xffffffffu, (r[1][0] & 0x7f800000u) == 0x7f800000u)) {
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            const float p0 = __uint_as_float(r[0][j]);
            acc[j] += isinf(p0) ? p0 : (p0 + __uint_as_float(r[1][j])) + __uint_as_float(r[2][j]);
          }
          continue;
        }
#pragma unroll
        for (int j = 0; j < 32; ++j) acc[j] += (__uint_as_float(r[0][j]) + __uint_as_float(r[1][j])) + __uint_as_float(r[2][j]);
      }
      bool finish = true;
      if (pos != first || end != first + nkb) {
        // park this part (slot 0: the share's first tile, slot 1: its last), take a ticket
        float* dst = parked + (size_t)(cta * 2 + (pos0 >= first ? 0 : 1)) * kTileFloats + row * 4;
#pragma unroll
        for (int j = 0; j < 32; j += 4)
          if (m0 + c0 + j < p.M) __stcg(reinterpret_cast<float4*>(dst + (size_t)(c0 + j) * kWR), make_float4(acc[j], acc[j + 1], acc[j + 2], acc[j + 3]));
        __threadfence();
        asm volatile("bar.sync 1, %0;" ::"n"(kDrain * 32) : "memory");
        if (tid == 0) {
          int j0 = 0;
          const int n = pi_wide::holders(cut, cta, tile, s_slots, &j0);
          const bool last = atomicAdd(tickets + j0, 1) == n - 1;
          if (last) tickets[j0] = 0;
          __threadfence();
          s_n = last ? n : 0;
        }
        asm volatile("bar.sync 1, %0;" ::"n"(kDrain * 32) : "memory");
        const int n = s_n;
        finish = n > 0;
        if (finish) {
#pragma unroll
          for (int j = 0; j < 32; ++j) acc[j] = 0.f;
          for (int i = 0; i < n; ++i) {     // in CTA order
            const float* src = parked + (size_t)s_slots[i] * kTileFloats + row * 4;
            float4 t[8];
#pragma unroll
            for (int u = 0; u < 8; ++u)
              t[u] = m0 + c0 + u * 4 < p.M ? __ldcg(reinterpret_cast<const float4*>(src + (size_t)(c0 + u * 4) * kWR)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int u = 0; u < 8; ++u) {
              acc[u * 4] += t[u].x; acc[u * 4 + 1] += t[u].y; acc[u * 4 + 2] += t[u].z; acc[u * 4 + 3] += t[u].w;
            }
          }
        }
      }
      if (finish) {
        // through shared memory: four adjacent output columns per thread, as the epilogues want them
        EpiRows rows;
        epi_rows_load(p, rt * kWR, lane, rows);
        if (tid < kWC) epi_place(p, m0 + tid, s_place[tid]);
#pragma unroll
        for (int j = 0; j < 32; ++j) tile_out[(c0 + j) * kWR + row] = acc[j];
        asm volatile("bar.sync 1, %0;" ::"n"(kDrain * 32) : "memory");
        for (int c = warp; c < kWC && m0 + c < p.M; c += 4 * kDrain) {
          float4 old[4];     // four rows' residuals in flight at once
#pragma unroll
          for (int u = 0; u < 4; ++u) old[u] = epi_old(p, rows, m0 + c + u * kDrain);
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (m0 + c + u * kDrain < p.M)
              epi_row(p, rows, rt, m0 + c + u * kDrain, s_place[c + u * kDrain],
                      *reinterpret_cast<const float4*>(tile_out + (c + u * kDrain) * kWR + lane * 4), old[u], lane);
        }
        asm volatile("bar.sync 1, %0;" ::"n"(kDrain * 32) : "memory");   // tile_out and s_place are free again
      }
      pos = end;
    }
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == kMma) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
  }
}

}  // namespace

void pi_gemm_wide_reserve(pi_ctx* ctx, const pi_linear* lin, int rows) {
  if (lin->kind != PI_BF16 || !pi_tc::wide_fits(lin)) return;
  // The tickets and the parts of cut tiles: of one size for every launch of the context; the tickets start and stay at zero
  // between launches.
  if (!ctx->gemm_parked.ptr) {
    const size_t tickets = pi_wide::ticket_bytes(ctx->sm_count), bytes = tickets + (size_t)ctx->sm_count * 2 * kTileFloats * sizeof(float);
    void* ptr = nullptr;
    if (cudaMalloc(&ptr, bytes) != cudaSuccess) {
      cudaGetLastError();
      return;
    }
    if (cudaMemsetAsync(ptr, 0, tickets, ctx->stream) != cudaSuccess) {
      cudaGetLastError();
      cudaFree(ptr);
      return;
    }
    ctx->gemm_parked.ptr = ptr;
    ctx->gemm_parked.bytes = bytes;
  }
  const size_t want = pi_wide::planes_bytes(std::min(rows, pi_wide::portion_limit(lin->cols)), lin->cols);
  if (want <= ctx->wide_planes.bytes) return;
  void* ptr = nullptr;
  if (cudaStreamSynchronize(ctx->stream) != cudaSuccess || cudaMalloc(&ptr, want) != cudaSuccess) {   // what there is stays
    cudaGetLastError();
    return;
  }
  if (ctx->wide_planes.ptr) cudaFree(ctx->wide_planes.ptr);
  ctx->wide_planes.ptr = ptr;
  ctx->wide_planes.bytes = want;
}

pi_status pi_tc::run_gemm_wide(pi_ctx* ctx, const pi_linear* lin, const pi_linear_args& a, const pi_act_planes& in) {
  GemmParams p;
  CUtensorMap act, w;
  PI_TRY(build_gemm_params(ctx, lin, a, in, kWC, &p, &act));
  {
    const cuuint64_t dims[2] = {(cuuint64_t)lin->cols, (cuuint64_t)lin->rows};
    const cuuint64_t strides[1] = {(cuuint64_t)lin->ld * sizeof(__nv_bfloat16)};
    const cuuint32_t box[2] = {kWK, kWR}, estr[2] = {1, 1};
    const CUresult r = encode_tiled_fn()(&w, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, lin->w, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                         CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return pi_fail(ctx, PI_ERR_CUDA, "cuTensorMapEncodeTiled failed with %d", (int)r);
  }
  const Cut cut = pi_wide::make_cut((int)lin->rows, a.M, (int)lin->cols, ctx->sm_count);
  static pi_smem_grant granted;
  if (kWideSmem > granted.of(ctx)) {
    PI_CUDA(ctx, cudaFuncSetAttribute(gemm_wide_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWideSmem));
    granted.of(ctx) = kWideSmem;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cut.ctas);
  cfg.blockDim = dim3(kWideThreads);
  cfg.dynamicSmemBytes = kWideSmem;
  cfg.stream = ctx->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = ctx->opt_pdl ? 1 : 0;
  int* tickets = static_cast<int*>(ctx->gemm_parked.ptr);
  float* parked = reinterpret_cast<float*>(static_cast<unsigned char*>(ctx->gemm_parked.ptr) + pi_wide::ticket_bytes(ctx->sm_count));
  const cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_wide_kernel, p, cut, parked, tickets, w, act);
  if (e != cudaSuccess) return pi_fail(ctx, PI_ERR_CUDA, "wide tensor-core GEMM launch failed: %s", cudaGetErrorString(e));
  ctx->launches++;
  return PI_OK;
}
