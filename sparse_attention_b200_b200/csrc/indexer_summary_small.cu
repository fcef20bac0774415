// R1 / R4 summary selector for problems that do not fill the GPU, and for every problem of up to 2048 KV blocks whose
// scores are wanted or that the tensor-core forms refuse: the arithmetic of indexer_summary.cu, cut so that a problem of
// 64 lists fills the GPU.
//
//   pool_small_kernel   one CTA per descriptor: the 128/R token rows (contiguous in
//                       memory) are fetched into shared memory in ONE round trip by all
//                       threads, then 64 threads add them in token order (the canonical
//                       sequential fp32 sum, so the descriptors are bit-identical with
//                       pool_kernel, which keeps 16 lanes per descriptor and pays one
//                       memory round trip per 8 tokens).
//   score_rows_kernel   16 to 64 query descriptors (one or several lists of a KV head) per cluster of 1 - 8 CTAs.
// Same results as pool_blocks / descriptor_dot / reduce_topk
// (indexers/r1_r4/gpu_ops.py:6-49): ids in score-descending order, ties to the lower id.
#include "internal.h"
#include "ptx.cuh"
#include "topk.cuh"
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <type_traits>

namespace sb {
namespace {

namespace cg = cooperative_groups;

// ---------------------------------------------------------------- pooling
// Descriptors 0 .. first - 1 come from x, the rest from x2 (queries and keys in one launch).
__global__ void __launch_bounds__(256) pool_small_kernel(const __nv_bfloat16* __restrict__ x,
                                                         __nv_bfloat16* __restrict__ desc, long long first,
                                                         const __nv_bfloat16* __restrict__ x2,
                                                         __nv_bfloat16* __restrict__ desc2, int n) {
  extern __shared__ uint4 tile[];                 // n token rows x 16 uint4
  long long vec = blockIdx.x;
  if (vec >= first) {
    vec -= first;
    x = x2;
    desc = desc2;
  }
  const uint4* src = reinterpret_cast<const uint4*>(x + vec * n * 128);
  for (int i = threadIdx.x; i < n * 16; i += blockDim.x) tile[i] = __ldcs(src + i);
  __syncthreads();
  if (threadIdx.x < 64) {
    const __nv_bfloat162* rows = reinterpret_cast<const __nv_bfloat162*>(tile) + threadIdx.x;
    float2 acc = make_float2(0.f, 0.f);
#pragma unroll 8
    for (int t = 0; t < n; ++t) {
      const float2 f = __bfloat1622float2(rows[t * 64]);
      acc.x += f.x;
      acc.y += f.y;
    }
    const float inv = 1.0f / static_cast<float>(n);
    reinterpret_cast<__nv_bfloat162*>(desc + vec * 128)[threadIdx.x] = __floats2bfloat162_rn(acc.x * inv, acc.y * inv);
  }
}

// ---------------------------------------------------------------- score + top-k
// A row tile is ROWS = 16 QT query descriptors (QT = 1, 2 or 4): L lists (query blocks of one KV head) of MP descriptors
// each (MP = group heads x R rounded up to a power of two, padding repeats a list's first descriptor: the maximum is
// unchanged). A cluster of C CTAs (C = 1, 2, 4 or 8) shares the row tile: CTA `rank` scores the key chunks rank,
// rank + C, ... of 64 KG descriptors, and owns the lists l with l % C == rank: every score goes straight into the owner's
// shared memory. QT x 4 KG register tile per thread, the next chunk's bytes requested before the arithmetic of this one (the
// exact score is defined by fp32 sums in feature order). The tiles stay bf16 in shared memory, two features to a word, and are
// widened by the reader: half the bytes of fp32 tiles, whose reads (8 wavefronts of a warp and feature for 4 x 4) bounded the
// loop at 8192 cycles per 64 x 64 unit against 4096 of FMAs. Products go two keys at a time through fma.rn.f32x2 (each half
// is fmaf), the same sums with half the instructions; KG = 2 (64 rows x 128 keys, 4 x 8 per thread) shares the widened
// queries among twice the keys. Now bound by the FMA pipe (60 % of its cycles busy, its throttle the largest stall; shared
// memory 39 %). Whole selector, us, fp32 4 x 4 -> this: 1024 lists of 64 x 8192 3790 -> 3390, 128 of 64 x 2048 166 -> 152,
// 64 of 64 x 512 29.6 -> 28.1. 4 x 8 with scalar FMAs took 3811; with fp32 keys 3309, but 96 KiB of shared memory: 4096 lists
// of 1 x 2048 332 us instead of 310, and sorts of 1024 x 2048 361 instead of 243; 4 x 4 with packed FMAs 4062. QT, KG, L and
// C are chosen by plan_rows().
constexpr int KD = 64;
constexpr int SCORE_BYTES_MAX = 40 * 1024;
constexpr size_t SMEM_PER_SM = 228 * 1024;       // of which 1 KiB per CTA is the system's

__device__ __forceinline__ unsigned score_key(float s) {      // order of the floats; both zeros are one value
  const unsigned b = __float_as_uint(s + 0.f);
  return b ^ ((b >> 31) ? 0xffffffffu : 0x80000000u);
}

// [feature pair][ROWS] words of two bf16 in shared memory. Odd 8-feature pieces are stored with bit 4 of the column flipped
// (tiles of at least 32 columns), so that a warp which holds two neighbouring pieces of 16 rows (whole 32-byte sectors of
// global memory) stores without bank conflicts.
template <int ROWS>
__device__ __forceinline__ void stage_piece(uint32_t* tile, int row, int c, const uint4& raw) {
  uint32_t* dst = tile + c * 4 * ROWS + (ROWS > 16 ? row ^ ((c & 1) << 4) : row);
  dst[0] = raw.x;
  dst[ROWS] = raw.y;
  dst[2 * ROWS] = raw.z;
  dst[3 * ROWS] = raw.w;
}

// feature F (0 or 1) of a pair of bf16
template <int F>
__device__ __forceinline__ float feature(uint32_t pair) {
  return __uint_as_float(F ? pair & 0xffff0000u : pair << 16);
}

struct RowsParams {
  const __nv_bfloat16 *qd, *kd;
  float* scores_out;         // [lists][nt] or null
  int32_t* ids;
  int32_t* fallback_counter; // three words to reset, or null
  int hq, hkv, qt, nt, r, topk;
  int lists_per_cta, tiles_per_head, mp_log2;
  int tile_words;            // words of shared memory before the scores
};

// QT = rows per thread, LPT = lists that they belong to: 1 (MP >= QT) or QT / MP, KG = groups of 64 keys in a chunk
template <int QT, int LPT, int KG>
__global__ void __launch_bounds__(256, QT < 4 ? 4 : KG == 1 ? 3 : 2) score_rows_kernel(const RowsParams p) {
  constexpr int ROWS = 16 * QT, KEYS = KD * KG;
  extern __shared__ __align__(16) float smem[];
  uint32_t* q_s = reinterpret_cast<uint32_t*>(smem);      // [64][ROWS]
  uint32_t* k_s = q_s + 64 * ROWS;           // [KG][64][KD]
  float* scores = smem + p.tile_words;       // [lists owned by this CTA][nt]

  cg::cluster_group cluster = cg::this_cluster();
  const int rank = static_cast<int>(cluster.block_rank()), csize = static_cast<int>(cluster.num_blocks());
  const int c_log2 = 31 - __clz(csize);
  const int tile = blockIdx.x >> c_log2;
  const int group = p.hq / p.hkv, m_real = group * p.r;
  const int bk = tile / p.tiles_per_head;
  const int b = bk / p.hkv, kvh = bk - b * p.hkv;
  const int qtile0 = (tile - bk * p.tiles_per_head) * p.lists_per_cta;
  const int lists = min(p.lists_per_cta, p.qt - qtile0);
  const int n_keys = p.nt * p.r;
  const int tid = threadIdx.x;
  // staging role: 16-byte pieces piece0 + 2 i of row `srow` (i = 0 .. 3, both parities of a piece pair in a warp); for
  // the queries QT pieces qpiece0 + 2 i of row `qrow`
  const int srow = (tid >> 1) & 63, piece0 = (tid & 1) | ((tid >> 7) << 3);
  const int qrow = (tid >> 1) & (ROWS - 1), qpiece0 = (tid & 1) | (tid / (2 * ROWS)) * (2 * QT);

  asm volatile("griddepcontrol.wait;" ::: "memory");      // the descriptors of the pooling kernel are visible from here
  // every list is exact here: no fallback, no violated bound, no largest difference
  if (p.fallback_counter && blockIdx.x == 0 && tid < 3) p.fallback_counter[tid] = 0;
  const uint4* kbase = reinterpret_cast<const uint4*>(p.kd + static_cast<long long>(bk) * n_keys * 128);
  uint4 raw[KG][4];
  auto fetch_keys = [&](int base) {
#pragma unroll
    for (int g = 0; g < KG; ++g) {
      const int key = base + g * KD + srow;
#pragma unroll
      for (int i = 0; i < 4; ++i)
        raw[g][i] = key < n_keys ? __ldg(kbase + static_cast<long long>(key) * 16 + piece0 + 2 * i) : make_uint4(0u, 0u, 0u, 0u);
    }
  };
  {
    const int l = qrow >> p.mp_log2, m = qrow & ((1 << p.mp_log2) - 1);
    const int mm = m < m_real ? m : 0;
    const int g = mm / p.r, rq = mm - g * p.r;
    const long long row = ((static_cast<long long>(b) * p.hq + kvh * group + g) * p.qt + qtile0 + (l < lists ? l : 0)) * p.r + rq;
    const uint4* src = reinterpret_cast<const uint4*>(p.qd + row * 128);
    uint4 qraw[QT];
#pragma unroll
    for (int i = 0; i < QT; ++i) qraw[i] = __ldg(src + qpiece0 + 2 * i);
    fetch_keys(rank * KEYS);
#pragma unroll
    for (int i = 0; i < QT; ++i) stage_piece<ROWS>(q_s, qrow, qpiece0 + 2 * i, qraw[i]);
  }
  if (csize > 1) cluster.sync();               // all CTAs of the cluster run: their shared memory may be addressed
  const float scale = 0.08838834764831845f;   // fp32(128^-0.5)
  const int tq = tid & 15, tk = tid >> 4;
  float* owner_scores[LPT];                    // where the scores of this thread's lists go (null: not a real list)
#pragma unroll
  for (int x = 0; x < LPT; ++x) {
    const int l = (tq * QT + x * (QT / LPT)) >> p.mp_log2;
    const bool speaks = LPT > 1 || ((tq * QT) & ((1 << p.mp_log2) - 1)) == 0;
    owner_scores[x] = speaks && l < lists ? cluster.map_shared_rank(scores, l & (csize - 1)) + (l >> c_log2) * p.nt : nullptr;
  }

  for (int base = rank * KEYS; base < n_keys; base += csize * KEYS) {
#pragma unroll
    for (int g = 0; g < KG; ++g)
#pragma unroll
      for (int i = 0; i < 4; ++i) stage_piece<KD>(k_s + g * 64 * KD, srow, piece0 + 2 * i, raw[g][i]);
    __syncthreads();                           // tiles staged
    if (base + csize * KEYS < n_keys) fetch_keys(base + csize * KEYS);
    unsigned long long acc[QT][2 * KG];        // two neighbouring keys each
#pragma unroll
    for (int i = 0; i < QT; ++i)
#pragma unroll
      for (int j = 0; j < 2 * KG; ++j) acc[i][j] = 0ull;
    const int pairs = base + (tid >> 5) * 8 < n_keys ? 64 : 0;          // a warp's keys may all be padding
#pragma unroll 1
    for (int d0 = 0; d0 < pairs; d0 += 8) {
#pragma unroll
      for (int dd = 0; dd < 8; ++dd) {
        const int flip = (dd >> 2) << 4;
        uint4 kw[KG];
#pragma unroll
        for (int g = 0; g < KG; ++g)
          kw[g] = *reinterpret_cast<const uint4*>(k_s + g * 64 * KD + (d0 + dd) * KD + ((tk * 4) ^ flip));
        const uint32_t* qsrc = q_s + (d0 + dd) * ROWS + (QT > 1 ? (tq * QT) ^ flip : tq);
        uint32_t qw[QT];
        if constexpr (QT == 4) {
          const uint4 qv = *reinterpret_cast<const uint4*>(qsrc);
          qw[0] = qv.x; qw[1] = qv.y; qw[2] = qv.z; qw[3] = qv.w;
        } else if constexpr (QT == 2) {
          const uint2 qv = *reinterpret_cast<const uint2*>(qsrc);
          qw[0] = qv.x; qw[1] = qv.y;
        } else {
          qw[0] = *qsrc;
        }
        auto step = [&](auto which) {
          constexpr int F = decltype(which)::value;
          unsigned long long kp[2 * KG];
#pragma unroll
          for (int g = 0; g < KG; ++g) {
            kp[2 * g] = f32x2_pack(feature<F>(kw[g].x), feature<F>(kw[g].y));
            kp[2 * g + 1] = f32x2_pack(feature<F>(kw[g].z), feature<F>(kw[g].w));
          }
#pragma unroll
          for (int i = 0; i < QT; ++i) {
            const float q = feature<F>(qw[i]);
            const unsigned long long qq = f32x2_pack(q, q);
#pragma unroll
            for (int j = 0; j < 2 * KG; ++j) acc[i][j] = f32x2_fma(qq, kp[j], acc[i][j]);
          }
        };
        step(std::integral_constant<int, 0>{});
        step(std::integral_constant<int, 1>{});
      }
    }
    // one score per (list, KV block): maximum over the list's rows and the block's R descriptors, then the scale. As in
    // the exact kernel the maximum starts at -inf: a NaN product never wins, and no score is NaN.
#pragma unroll
    for (int g = 0; g < KG; ++g) {
#pragma unroll
      for (int x = 0; x < LPT; ++x) {
        float best[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) best[j] = -CUDART_INF_F;
#pragma unroll
        for (int i = 0; i < QT / LPT; ++i) {
          float s0, s1, s2, s3;
          f32x2_unpack(acc[x * (QT / LPT) + i][2 * g], s0, s1);
          f32x2_unpack(acc[x * (QT / LPT) + i][2 * g + 1], s2, s3);
          best[0] = fmaxf(best[0], s0);
          best[1] = fmaxf(best[1], s1);
          best[2] = fmaxf(best[2], s2);
          best[3] = fmaxf(best[3], s3);
        }
        if (p.r > 1) { best[0] = fmaxf(best[0], best[1]); best[2] = fmaxf(best[2], best[3]); }
        if (p.r > 2) best[0] = fmaxf(best[0], best[2]);
        if (LPT == 1) {
          for (int dlt = 1; dlt < (1 << p.mp_log2) / QT; dlt <<= 1) {
#pragma unroll
            for (int j = 0; j < 4; ++j) best[j] = fmaxf(best[j], __shfl_xor_sync(0xffffffffu, best[j], dlt));
          }
        }
        if (owner_scores[x]) {
          const int first = base + g * KD + tk * 4;       // a multiple of R
          float* dst = owner_scores[x] + first / p.r;
          if (first < n_keys) dst[0] = best[0] * scale;
          if (p.r == 1) {
#pragma unroll
            for (int j = 1; j < 4; ++j)
              if (first + j < n_keys) dst[j] = best[j] * scale;
          } else if (p.r == 2) {
            if (first + 2 < n_keys) dst[1] = best[2] * scale;
          }
        }
      }
    }
    __syncthreads();                           // k_s free again
  }
  if (csize > 1) cluster.sync();               // every score is in its owner's shared memory
  const int own = (lists - rank + csize - 1) >> c_log2;     // lists rank, rank + C, ... of the tile
  if (own <= 0) return;
  const long long list0 = static_cast<long long>(bk) * p.qt + qtile0 + rank;
  if (p.scores_out)
    for (int e = tid; e < own * p.nt; e += blockDim.x) {
      const int l = e / p.nt;
      p.scores_out[(list0 + static_cast<long long>(l) * csize) * p.nt + (e - l * p.nt)] = scores[e];
    }
  // (score descending, id ascending) is a total order: no score is NaN
  if (p.nt <= 256 && ((own * p.nt + 255) >> 8) * p.nt <= 512 * ((own + 7) >> 3)) {
    // Short lists: every score counts the scores that beat it, the count is its rank. The right-hand side is what
    // the threshold search of a warp below takes in the same unit, scores read by a thread (whole selector, us, with as
    // many lists in a CTA: 64 lists of 256 271 by counting, 60 by searching; 32 lists of 32 20 and 25).
    for (int e = tid; e < own * p.nt; e += blockDim.x) {
      const int l = e / p.nt, j = e - l * p.nt;
      const float* s = scores + l * p.nt;
      const float mine = s[j];
      int place = 0;
#pragma unroll 4
      for (int i = 0; i < p.nt; ++i) place += better(s[i], i, mine, j) ? 1 : 0;
      if (place < p.topk) p.ids[(list0 + static_cast<long long>(l) * csize) * p.topk + place] = j;
    }
    return;
  }
  const int lane = tid & 31, warp = tid >> 5;
  if (p.topk <= 128) {
    // one warp per list: k-th largest score bit by bit, then ranks among the k that reach it
    float* cand_s = smem + warp * 256;
    int* cand_i = reinterpret_cast<int*>(cand_s + 128);
    for (int l = warp; l < own; l += 8) {
      const float* s = scores + l * p.nt;
      unsigned T = 0;
      for (int bit = 31; bit >= 0; --bit) {
        const unsigned trial = T | (1u << bit);
        int cnt = 0;
#pragma unroll 8
        for (int j = lane; j < p.nt; j += 32) cnt += score_key(s[j]) >= trial ? 1 : 0;
        cnt = __reduce_add_sync(0xffffffffu, cnt);
        if (cnt >= p.topk) T = trial;
        if (cnt == p.topk) break;              // exactly the wanted ones pass: `trial` separates as well as the k-th score
      }
      int above = 0;
      for (int j = lane; j < p.nt; j += 32) above += score_key(s[j]) > T ? 1 : 0;
      above = __reduce_add_sync(0xffffffffu, above);
      const unsigned below = (1u << lane) - 1u;
      int written = 0, ties = 0;
      for (int j0 = 0; j0 < p.nt; j0 += 32) {
        const int j = j0 + lane;
        const unsigned u = j < p.nt ? score_key(s[j]) : 0u;
        const bool eq = j < p.nt && u == T;
        const unsigned eqs = __ballot_sync(0xffffffffu, eq);
        const bool take = j < p.nt && (u > T || (eq && ties + __popc(eqs & below) < p.topk - above));
        const unsigned takes = __ballot_sync(0xffffffffu, take);
        if (take) {
          const int pos = written + __popc(takes & below);
          cand_s[pos] = s[j];
          cand_i[pos] = j;
        }
        written += __popc(takes);
        ties += __popc(eqs);
      }
      __syncwarp();
      for (int c = lane; c < p.topk; c += 32) {
        const float mine = cand_s[c];
        const int id = cand_i[c];
        int place = 0;
#pragma unroll 4
        for (int i = 0; i < p.topk; ++i) place += better(cand_s[i], cand_i[i], mine, id) ? 1 : 0;
        p.ids[(list0 + static_cast<long long>(l) * csize) * p.topk + place] = id;
      }
      __syncwarp();
    }
    return;
  }
  // k > 128: the lists are sorted, as many at a time as fit the tiles' 40 to 64 KiB (bitonic, 64-bit keys of score and
  // inverted id, so that the order is score descending, id ascending; padding sorts last). Rounds of block-wide
  // arg-max, k per list and list after list, took 1320 us for 64 lists of 512 with k = 256, this 44 with 64 lists to a
  // tile and 20 with 14 (whole selector).
  unsigned long long* keys = reinterpret_cast<unsigned long long*>(smem);
  int p_log2 = 1;
  while ((1 << p_log2) < p.nt) ++p_log2;
  const int batch = (p.tile_words / 2) >> p_log2, half = 1 << (p_log2 - 1);
  for (int l0 = 0; l0 < own; l0 += batch) {
    const int nl = min(batch, own - l0);
    for (int e = tid; e < nl << p_log2; e += blockDim.x) {
      const int l = e >> p_log2, j = e & (2 * half - 1);
      keys[e] = j < p.nt ? (static_cast<unsigned long long>(score_key(scores[(l0 + l) * p.nt + j])) << 32) | (0xffffffffu - j) : 0ull;
    }
    __syncthreads();
    for (int k = 1; k <= p_log2; ++k) {
      for (int d = k - 1; d >= 0; --d) {
        for (int c = tid; c < nl * half; c += blockDim.x) {
          const int i = ((c >> d) << (d + 1)) | (c & ((1 << d) - 1));      // bit d clear; i + 2^d is its partner
          const bool descending = k == p_log2 || ((i >> k) & 1) == 0;
          const unsigned long long x = keys[i], y = keys[i + (1 << d)];
          if ((x < y) == descending) {
            keys[i] = y;
            keys[i + (1 << d)] = x;
          }
        }
        __syncthreads();
      }
    }
    for (int e = tid; e < nl * p.topk; e += blockDim.x) {
      const int l = e / p.topk, place = e - l * p.topk;
      p.ids[(list0 + static_cast<long long>(l0 + l) * csize) * p.topk + place] =
          static_cast<int32_t>(0xffffffffu - static_cast<unsigned>(keys[(l << p_log2) + place]));
    }
    __syncthreads();
  }
}

template <int QT, int LPT, int KG>
int launch_rows(const RowsParams& p, int grid, int csize, size_t smem, DeviceCtx* ctx, int slot, cudaStream_t stream) {
  if (!(ctx->small_attr & (1 << slot))) {
    cudaError_t e = cudaFuncSetAttribute(score_rows_kernel<QT, LPT, KG>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (QT * 16 + KD) * 512 + SCORE_BYTES_MAX);
    if (e != cudaSuccess) return set_error(SB_ERR_CUDA, cudaGetErrorString(e));
    ctx->small_attr |= (1 << slot);
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(grid));
  cfg.blockDim = dim3(256);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = static_cast<unsigned>(csize);
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  cudaError_t e = cudaLaunchKernelEx(&cfg, score_rows_kernel<QT, LPT, KG>, p);
  return e == cudaSuccess ? SB_OK : set_error(SB_ERR_CUDA, cudaGetErrorString(e));
}

struct RowsPlan {
  int lists, tiles, csize, qt, kg;   // lists per row tile, row tiles per KV head, cluster size, rows per thread, key groups
  int tile_words;                    // of shared memory, before the scores
  size_t smem;
};

// How the lists of a KV head are cut into row tiles and how many CTAs share one: the cheapest by an estimate in cycles of
// an SM. Few lists are spread over the SMs in smaller tiles; many are packed, as far as the scores of the lists that a CTA
// owns fit its share of shared memory, which for long lists takes a large cluster. Whole selector with scores, us, always
// 64-row tiles packed as densely as the rows hold -> this: 64 lists of 1 x 128 descriptors, which ran on two CTAs,
// 49.9 -> 11.5; 16 of 1 x 64 16.9 -> 9.6; 4 of 1 x 8 11.6 -> 8.1; 2048 of 1 x 2048, five lists to a tile, 662 -> 161;
// 1024 of 8 x 8192 2237 -> 1948. (A cluster of 8 CTAs per list and 16 descriptors, which was used for up to 148 lists before
// the row tiles, took 15.1, 10.7 and 9.1 us for the first three; on a few lists of 65 to 128 keys it was 1 us faster.)
// The constants were fitted to the times of all plans of 673 problems (1 to 1448 lists of 1 to 64 x 8 to 8192, whole selector with
// scores): the choice is 1.0 % behind the best plan (geometric mean) and 6.6 % ahead of fp32 tiles with a plan of their own. It is
// more than 2 % behind those on 21 problems, more than 5 % on three (1204 lists of 3 x 291 64.5 -> 69.4 us, 744 of 4 x 1038 63.3 ->
// 67.7, 171 of 16 x 1218 64.7 -> 68.2). With 128 keys to a chunk wherever there is a second half, and constants from fewer
// problems, 82 were more than 2 % behind and 55 more than 5 (3 lists of 48 x 96 9.5 -> 11.8 us, now 8.9; 58 of 24 x 688 23.6 ->
// 26.1, 21.9; 160 of 16 x 1024 71.3 -> 77.8, 71.3). On 200 further problems 6 and 1 are (23 and 13).
RowsPlan plan_rows(long long heads, int qt, int nt, int r, int topk, int mp_log2, int sm_count) {
  const float nf = static_cast<float>(nt);
  float sort_stage = 0.f, stages = 0.f;        // k > 128: cycles per list and stage beside others, number of stages
  int p_log2 = 1;
  while ((1 << p_log2) < nt) ++p_log2;
  stages = 0.5f * p_log2 * (p_log2 + 1);
  sort_stage = 25.f * (1 << p_log2) / 512.f;
  const float search = 1300.f + 5.2f * nf + 0.25f * static_cast<float>(topk) * static_cast<float>(topk);
  RowsPlan best{};
  float best_cost = 0.f;
  int full = 64 >> mp_log2;
  if (full > qt) full = qt;
  for (int n = full;; n = (n + 1) / 2) {
    const int tiles = (qt + n - 1) / n, lists = (qt + tiles - 1) / tiles;
    const int rows = lists << mp_log2, per_thread = rows <= 16 ? 1 : rows <= 32 ? 2 : 4;
    for (int i = 0; i < 8; ++i) {
      const int c = 8 >> (i >> 1), kg = 1 + (i & 1);
      if (kg == 2 && (per_thread < 4 || nt * r <= KD)) continue;       // no empty second half
      const int own = (lists + c - 1) / c, chunks = (nt * r + KD * kg - 1) / (KD * kg);
      if ((c > 1 && c / 2 >= chunks) || own * nt * 4 > SCORE_BYTES_MAX) continue;
      // k > 128: room to sort as many lists at a time as fp32 tiles would leave
      const int tile_words = topk > 128 ? (16 * per_thread + KD) * 128 : (16 * per_thread + KD * kg) * 64;
      const size_t smem = (static_cast<size_t>(tile_words) + static_cast<size_t>(own) * nt) * 4;
      const long long ctas = heads * tiles * c;
      const int most = per_thread < 4 ? 4 : kg == 1 ? 3 : 2;
      const int resident = static_cast<int>(SMEM_PER_SM / (smem + 1024)) < most ? static_cast<int>(SMEM_PER_SM / (smem + 1024)) : most;
      const float load = static_cast<float>((ctas + sm_count - 1) / sm_count);       // CTAs of an SM in all
      const float rounds = static_cast<float>(ctas) / static_cast<float>(resident * sm_count);
      // a chunk of 64 keys (128 with kg = 2), cycles of an SM
      float chunk = per_thread == 1 ? 2920.f : per_thread == 2 ? 3870.f : kg == 1 ? 5520.f : 10580.f;
      // clusters of a second round wait until all their slots are free
      if (c >= 4 && rounds > 1.f) chunk *= 1.f + (c == 8 ? 0.15f : 0.12f) * (rounds < 2.f ? rounds - 1.f : 1.f);
      const float share = static_cast<float>(lists) / static_cast<float>(c);
      float alone, among;                      // ranking: of the busiest CTA by itself, of the average one beside others
      if (nt <= 256 && ((own * nt + 255) >> 8) * nt <= 512 * ((own + 7) >> 3)) {
        alone = static_cast<float>((own * nt + 255) >> 8) * nf * 14.f;
        among = share * nf * nf * (7.f / 256.f);
      } else if (topk <= 128) {
        alone = search * (own > 5 ? 0.34f * static_cast<float>(own) : 1.7f);
        among = search * 0.28f * share;
      } else {
        alone = stages * (own * sort_stage > 80.f ? own * sort_stage : 80.f) * 7.3f;
        among = stages * share * sort_stage * 1.3f;
      }
      const float ranking = alone > load * among ? alone : load * among;
      const float start = c == 1 ? 3240.f : c == 2 ? 4010.f : c == 4 ? 4910.f : 6690.f;
      const float cost = (rounds > 1.f ? rounds : 1.f) * start + load * chunk * static_cast<float>((chunks + c - 1) / c) + ranking;
      if (best.lists == 0 || cost < best_cost) {
        best = RowsPlan{lists, tiles, c, per_thread, kg, tile_words, smem};
        best_cost = cost;
      }
    }
    if (n == 1) break;
  }
  return best;
}

}  // namespace

// Small problems only: at most four waves of 16-descriptor CTAs of pool_kernel.
bool pool_small_eligible(long long num_desc) {
  DeviceCtx* ctx = device_ctx();
  return ctx && (num_desc + 15) / 16 < 4LL * ctx->sm_count;
}

int launch_pool_small(const void* x, void* desc, long long num_desc, int tokens_per_desc, cudaStream_t stream) {
  return launch_pool_small_pair(x, desc, num_desc, nullptr, nullptr, 0, tokens_per_desc, stream);
}

// Two tensors in one launch (x2 may be null with num_desc2 = 0).
int launch_pool_small_pair(const void* x, void* desc, long long num_desc, const void* x2, void* desc2,
                           long long num_desc2, int tokens_per_desc, cudaStream_t stream) {
  pool_small_kernel<<<static_cast<unsigned>(num_desc + num_desc2), 256, static_cast<size_t>(tokens_per_desc) * 256,
                      stream>>>(static_cast<const __nv_bfloat16*>(x), static_cast<__nv_bfloat16*>(desc), num_desc,
                                static_cast<const __nv_bfloat16*>(x2), static_cast<__nv_bfloat16*>(desc2),
                                tokens_per_desc);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? SB_OK : set_error(SB_ERR_CUDA, cudaGetErrorString(e));
}

// Returns 1 when the problem is not a small one (the caller then takes the other kernels). force: whatever its size, up
// to 2048 blocks (scores wanted, or problems the tensor-core forms do not take). Against score_topk_kernel, us, that one ->
// this: 512 lists of 4 x 512 89 -> 66, 2048 of 1 x 2048 420 -> 161, 1024 of 64 x 8192 5370 -> 3370; behind it only on
// problems of a few microseconds (262 of 4 x 136 with k = 1 16.8 -> 21.3, 202 of 16 x 342 55 -> 61 were the worst of 680).
int launch_summary_small(const void* qd, const void* kd, float* scores, int32_t* ids, int32_t* fallback_counter,
                         int batch, int hq, int hkv, int qt, int nt, int r, int topk, cudaStream_t stream, bool force) {
  DeviceCtx* ctx = device_ctx();
  if (!ctx) return SB_ERR_CUDA;
  const int m = (hq / hkv) * r;
  if (nt > 2048 || m > 64) return 1;
  int mp_log2 = 0;
  while ((1 << mp_log2) < m) ++mp_log2;
  const long long heads = static_cast<long long>(batch) * hkv;
  // 64 x 64 units of the problem: lists packed as densely as a cluster of 8 allows
  int packed = 64 >> mp_log2;
  if (packed > 8 * (SCORE_BYTES_MAX / (4 * nt))) packed = 8 * (SCORE_BYTES_MAX / (4 * nt));
  const long long units = heads * ((qt + packed - 1) / packed) * ((nt * r + KD - 1) / KD);
  // Against the tensor-core forms (their selection phase costs about 16 us per round of eight lists whatever the
  // length, a unit of 64 rows x 64 keys here about 5 us of an SM; select_summary with pooling, us, tensor-core form ->
  // this one): below 16 descriptors per list those pack more than a round of lists into one CTA and leave most SMs
  // idle (256 lists of 1 x 32 blocks 65 -> 10, 512 of 4 x 512 131 -> 68, 2048 of 1 x 256 269 -> 56); from 16 on only
  // when the lists do not fill the GPU (64 lists of 64 x 512 key rows 42 -> 32, 128 of 16 x 1024 75 -> 67). Beyond four
  // units per SM the tensor cores win (320 of 16 x 600: 85 against 100; 128 of 64 x 2048: 62 against 167).
  if (!force && !((m < 16 || heads * qt <= ctx->sm_count) && units <= 4LL * ctx->sm_count)) return 1;
  const RowsPlan plan = plan_rows(heads, qt, nt, r, topk, mp_log2, ctx->sm_count);
  RowsParams p{};
  p.qd = static_cast<const __nv_bfloat16*>(qd);
  p.kd = static_cast<const __nv_bfloat16*>(kd);
  p.scores_out = scores;
  p.ids = ids;
  p.fallback_counter = fallback_counter;
  p.hq = hq; p.hkv = hkv; p.qt = qt; p.nt = nt; p.r = r; p.topk = topk;
  p.lists_per_cta = plan.lists;
  p.tiles_per_head = plan.tiles;
  p.mp_log2 = mp_log2;
  p.tile_words = plan.tile_words;
  const int grid = static_cast<int>(heads) * plan.tiles * plan.csize;
  if (plan.qt == 1) return launch_rows<1, 1, 1>(p, grid, plan.csize, plan.smem, ctx, 0, stream);
  if (plan.qt == 2 && mp_log2 == 0) return launch_rows<2, 2, 1>(p, grid, plan.csize, plan.smem, ctx, 1, stream);
  if (plan.qt == 2) return launch_rows<2, 1, 1>(p, grid, plan.csize, plan.smem, ctx, 2, stream);
  if (plan.kg == 2) {
    if (mp_log2 == 0) return launch_rows<4, 4, 2>(p, grid, plan.csize, plan.smem, ctx, 6, stream);
    if (mp_log2 == 1) return launch_rows<4, 2, 2>(p, grid, plan.csize, plan.smem, ctx, 7, stream);
    return launch_rows<4, 1, 2>(p, grid, plan.csize, plan.smem, ctx, 8, stream);
  }
  if (mp_log2 == 0) return launch_rows<4, 4, 1>(p, grid, plan.csize, plan.smem, ctx, 3, stream);
  if (mp_log2 == 1) return launch_rows<4, 2, 1>(p, grid, plan.csize, plan.smem, ctx, 4, stream);
  return launch_rows<4, 1, 1>(p, grid, plan.csize, plan.smem, ctx, 5, stream);
}

}  // namespace sb
