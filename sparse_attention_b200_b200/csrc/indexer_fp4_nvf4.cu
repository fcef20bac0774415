// Tensor-core path of the NVFP4 indexer on NVFP4 tensor-core MMAs: the same block ids as the
// exact scorer followed by tile top-k, bit for bit.
//
// tcgen05.mma kind::mxf4nvf4.block_scale multiplies the packed e2m1 codes of a key page
// (M = 128 rows) and of a query tile (N) straight from shared memory, with the ue4m3 scale of every
// 16-element group read from tensor memory: no dequantised copy exists anywhere. Operands: 64 bytes
// of codes per row, TMA-loaded with the 64-byte swizzle; K = 64 per instruction, so two
// instructions cover the 128 features. The scales of a 128-row tile are re-ordered by the producer
// warp into the 512-byte "32 x (4 row groups x 4 scales)" chunks the instruction reads
// (byte (r % 32) * 16 + (r / 32) * 4 + j = scale j of row r) and copied to tensor memory with
// tcgen05.cp.32x128b.warpx4 by the elected lane of the MMA warp. One 128 x 128 accumulator, two key-scale slots and the
// query scales take 152 tensor-memory columns (256 allocated), so two CTAs share an SM and the
// epilogue of one runs under the MMAs of the other. (N = 64 halves of the query tile with three
// accumulators per CTA were measured slower: an M128 N64 K64 instruction takes nearly as long as
// an N128 one, both being bound by the shared-memory reads of their operands.)
//
// Each product and each 16-element group sum is exact; only the accumulation of the eight scaled
// group sums is done in the tensor core's own order and precision instead of the fixed group order
// that defines a score. The MMA result is therefore a PRE-FILTER, as in the summary indexer:
// approximate and exact score differ by at most delta = 2^-18 * min(max_q ||q||_1 * max|k|,
// max_q ||q||_2 * max_k ||k||_2) (see EPS below; the pruning kernel, which serves small problems, takes
// max|k| <= 6 x the largest key scale of its pages instead of a pass over the keys); candidates more
// than 2 delta apart are ordered by their
// approximate scores for certain, the others are re-scored exactly, a tile whose pre-filter cannot be
// proven safe is scored exactly in full. Whenever both values of a score are in hand the kernels
// also CHECK the bound: a difference above delta sends the tile to the exact path and is counted.
// Same role as Fp4IndexerStagedMmaSm100 + Fp4IndexerScaleReorderSm100 + tile_max_topk16_kernel
// (indexers/fp4/vendor_minimax_msa/src/sm100/fp4_indexer.py:83-198, 201-1108,
// indexers/fp4/tile_topk.cu:38-126).
#include "ptx.cuh"
#include "internal.h"
#include "topk.cuh"
#include "fp4_exact.cuh"
#include <algorithm>

namespace sb {
namespace fnv {

constexpr int CODE_BYTES = 128 * 64;              // one operand tile: 128 rows of 64 bytes of codes
constexpr int SF_BYTES = 1024;                    // its scales: two 512-byte chunks (features 0-63, 64-127)
constexpr int STAGE_BYTES = CODE_BYTES + SF_BYTES;
constexpr int A_STAGES = 6;                       // at most (see Layout)
constexpr int C_MAX = 192;
constexpr int NUM_THREADS = 320;
constexpr int TMA_WARP = 8, MMA_WARP = 9;
// Bound on |tensor-core dot - canonical dot| relative to B = sum_g |t_g| (t_g = scaled group sum, each
// exact in fp32): eight terms added by the hardware in an unknown order with at worst a truncating
// 24-bit datapath give <= 8 * 2^-22 * B, the canonical fp32 sum itself is within 7 * 2^-24 * B of the
// real value: together < 2^-18 * B, and B <= min(||q||_1 * max|k|, ||q||_2 * ||k||_2). Measured on
// stress inputs the difference stays below 2^-24 * that bound (the tests print the ratio), and the
// kernels check it on every score they hold twice.
constexpr float EPS = 3.814697265625e-06f;        // 2^-18
constexpr int MAX_TILES = 16384;                  // 64 KiB of scores
constexpr int ACC_STAGES = 1;                     // accumulators of 128 columns (a whole query tile)

constexpr int OFF_A = 0;
// Shared memory of the scorers by the number of pages in flight: six, or four where the selection kernel's scores (4 bytes a
// page) leave no room for a second CTA on the SM beside six; the staging ring then shares the candidate arrays' place.
template <int STAGES>
struct Layout {
  static constexpr int B = STAGES * STAGE_BYTES;            // query tile: codes + scales
  static constexpr int RAW = B + STAGE_BYTES;               // staging ring: the scales of a page as they are in memory
  static constexpr int RAW_STAGES = STAGES == A_STAGES ? 4 : 3;     // pages whose scales are on their way
  static constexpr int CAND = STAGES == A_STAGES ? RAW + RAW_STAGES * SF_BYTES : RAW;     // arrays of the selection phase
  static constexpr int SCORES = CAND + 4 * C_MAX * 4;
  static_assert(STAGES == A_STAGES || RAW_STAGES * SF_BYTES <= SCORES - CAND, "staging ring");
  // the selection phase re-uses [0, CAND) for int8 rows and fp32 scales of a query tile and a key page
  static_assert(2 * 128 * FP4_ROW_WORDS * 4 + 2 * 128 * 8 * 4 <= CAND, "staging area of the exact scorer does not fit");
};
// tensor memory columns
constexpr int TM_ACC = 0;
constexpr int TM_SFA = ACC_STAGES * 128;           // 2 slots x 8 columns (two K halves of 4 columns)
constexpr int TM_SFB = TM_SFA + 16;               // 8 columns
constexpr int TM_COLS = 256;
static_assert(TM_SFB + 8 <= TM_COLS, "tensor memory map");

// barrier indices
enum { A_FULL = 0, A_EMPTY = A_STAGES, B_FULL = 2 * A_STAGES, ACC_FULL = 2 * A_STAGES + 1,
       ACC_EMPTY = ACC_FULL + ACC_STAGES, NUM_BARS = ACC_EMPTY + ACC_STAGES };

// kind::mxf4nvf4 instruction descriptor: e2m1 A and B (format 1), ue4m3 scales (0), both K-major,
// dense, K = 64; N >> 3 in bits 17-22, M >> 4 in bits 24-28.
__host__ __device__ constexpr uint32_t idesc_nvf4(int m, int n) {
  return (1u << 7) | (1u << 10) | (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(m >> 4) << 24);
}
// K-major operand of 64-byte rows, 64-byte swizzle (layout type 4): 8-row atoms 512 bytes apart.
__device__ __forceinline__ uint64_t desc_sw64_kmajor(uint32_t addr) {
  return desc_field(addr) | (desc_field(512) << 32) | (1ULL << 46) | (4ULL << 61);
}
// one 512-byte scale chunk: 32 rows of 16 bytes, no swizzle, 8-row groups 128 bytes apart
__device__ __forceinline__ uint64_t desc_scale_chunk(uint32_t addr) {
  return desc_field(addr) | (desc_field(128) << 32) | (1ULL << 46);
}
__device__ __forceinline__ void mma_nvf4(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t sfa, uint32_t sfb,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.block16 [%0], %1, %2, %3, [%5], [%6], p;\n\t"
      "}" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(sfa), "r"(sfb)
      : "memory");
}
// 32 rows x 16 bytes of shared memory -> 4 tensor-memory columns of lanes 0-31, repeated for the
// other three lane quarters
__device__ __forceinline__ void tmem_cp_scales(uint32_t taddr, uint64_t sdesc) {
  asm volatile("tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], %1;" ::"r"(taddr), "l"(sdesc) : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst),
      "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ int f2ord(float f) {
  const int i = __float_as_int(f);
  return i >= 0 ? i : i ^ 0x7fffffff;
}
// maximum of a warp's floats in one instruction; a NaN counts only when all are (as with fmaxf)
__device__ __forceinline__ float warp_max(float v) {
  float m;
  asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(m) : "f"(v));
  return m;
}
__device__ __forceinline__ float ord2f(int i) { return __int_as_float(i >= 0 ? i : i ^ 0x7fffffff); }

// 8 bytes of global memory to shared memory, asynchronously; groups of a thread's copies and a wait for all but the newest N
__device__ __forceinline__ void cp_async8(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Largest |dequantised element| and largest squared L2 norm over all key vectors -> stats[0], stats[1]
// (zeroed by the caller). Sixteen adjacent threads hold one row.
__global__ void __launch_bounds__(256) key_stats_kernel(const uint8_t* __restrict__ codes, const uint8_t* __restrict__ scales,
                                                        long long rows, float* __restrict__ stats) {
  __shared__ float red_m[8], red_n[8];
  const long long gid = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const long long row = gid >> 4;
  const int w = static_cast<int>(gid & 15);
  float amax = 0.f, squares = 0.f;
  if (row < rows) {
    const uint32_t word = __ldg(reinterpret_cast<const uint32_t*>(codes + row * 64 + w * 4));
    const float sc = 0.5f * e4m3_to_float(scales[row * 8 + (w >> 1)] & 0x7fu);
    const unsigned long long lut = 0x0C08060403020100ULL;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const uint32_t c = (word >> (4 * e)) & 7u;
      const float f = static_cast<float>((lut >> (8 * c)) & 0xFFu) * sc;
      amax = fmaxf(amax, f);
      squares = fmaf(f, f, squares);
    }
  }
#pragma unroll
  for (int d = 8; d > 0; d >>= 1) squares += __shfl_xor_sync(0xffffffffu, squares, d);   // the row's 16 threads
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, d));
    squares = fmaxf(squares, __shfl_xor_sync(0xffffffffu, squares, d));
  }
  if ((threadIdx.x & 31) == 0) {
    red_m[threadIdx.x >> 5] = amax;
    red_n[threadIdx.x >> 5] = squares;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 1; i < 8; ++i) {
      amax = fmaxf(amax, red_m[i]);
      squares = fmaxf(squares, red_n[i]);
    }
    atomicMax(reinterpret_cast<int*>(stats), __float_as_int(amax));
    atomicMax(reinterpret_cast<int*>(stats + 1), __float_as_int(squares));
  }
}

// Largest byte of eight packed e4m3 scale words (codes 0x00..0x7e grow with the value; the sign bit,
// which a valid scale does not carry, is masked off).
__device__ __forceinline__ uint32_t max_scale_bytes(uint32_t acc, uint32_t w) { return __vmaxu4(acc, w & 0x7f7f7f7fu); }
__device__ __forceinline__ uint32_t top_byte(uint32_t w) {
  return max(max(w & 0xffu, (w >> 8) & 0xffu), max((w >> 16) & 0xffu, w >> 24));
}
// |dequantised element| <= 6 * scale
__device__ __forceinline__ float key_bound_from_scale_byte(uint32_t byte) {
  return 6.0f * e4m3_to_float(static_cast<uint8_t>(byte)) * 1.0001f;
}

// The eight scales of rows lane, lane + 32, lane + 64, lane + 96 of a 128-row tile (row pitch in bytes).
struct ScaleRegs { uint2 r[4]; };
__device__ __forceinline__ ScaleRegs load_scales(const uint8_t* base, long long pitch, int lane) {
  ScaleRegs s;
#pragma unroll
  for (int i = 0; i < 4; ++i) s.r[i] = __ldg(reinterpret_cast<const uint2*>(base + (lane + 32 * i) * pitch));
  return s;
}
// ... written as the two 512-byte chunks the MMA reads: one 16-byte store per lane and chunk.
__device__ __forceinline__ void store_scale_chunks(unsigned char* dst, const ScaleRegs& s, int lane) {
  *reinterpret_cast<uint4*>(dst + lane * 16) = make_uint4(s.r[0].x, s.r[1].x, s.r[2].x, s.r[3].x);
  *reinterpret_cast<uint4*>(dst + 512 + lane * 16) = make_uint4(s.r[0].y, s.r[1].y, s.r[2].y, s.r[3].y);
}

// Problem geometry shared by the two kernels.
struct Geometry {
  const uint8_t *qp, *qs, *kp, *ks;   // public NVFP4 layout (codes, e4m3 scales)
  int batch, hidx, hk, len_q, tiles;
};

// ---------------------------------------------------------------- producer and MMA roles
// A page takes about 430 cycles of an SM with two CTAs on it, against 128 cycles of MMAs: the serial work of lone warps
// (waits, scale copies, hand-overs) bounds it, in the producer, the MMA warp and the epilogue alike: leaving out any one of
// maxima, accumulator reads, TMA copies or scale stores changes nothing. 440 when the producer loaded the scales into
// registers, in a loop unrolled over the pages in flight, 450 when it also fenced its scale stores for the async proxy (a fence
// takes 300 cycles, and waits for the loads in flight; now the MMA warp does it, when a page has landed), 520 when one lane
// issued under `if (lane == 0)`, see elect_one(). No faster: one CTA per SM with three accumulators and one to four producer
// warps (540 to 720), two or three producer warps per CTA here (450), three accumulators of 64 columns per CTA (450).
// Producer warp: query tile once, then key pages page0 + (t + rot) % wrap for t = 0 .. num_tiles - 1 (num_tiles <= wrap,
// rot < wrap).
template <int STAGES>
__device__ __forceinline__ void producer_role(const Geometry& g, const CUtensorMap* q_map, const CUtensorMap* k_map,
                                              uint32_t base, unsigned char* gbase, uint32_t bar0, const Guard& guard,
                                              int b, int h, int hk_idx, long long q_row0, int page0, int num_tiles,
                                              int rot, int wrap, int lane, int code0) {
  using L = Layout<STAGES>;
  auto bar = [&](int i) { return bar0 + 8u * i; };
  auto page_of = [&](int t) { return page0 + (t + rot >= wrap ? t + rot - wrap : t + rot); };
  auto key_row = [&](int pg) { return ((static_cast<long long>(b) * g.tiles + pg) * g.hk + hk_idx) * 128; };
  if (lane == 0) {
    mbar_expect_tx(bar(B_FULL), CODE_BYTES);
    tma_load_3d(base + L::B, q_map, 0, h, static_cast<int>(q_row0), bar(B_FULL));
  }
  {
    const ScaleRegs s = load_scales(g.qs + (q_row0 * g.hidx + h) * 8, static_cast<long long>(g.hidx) * 8, lane);
    store_scale_chunks(gbase + L::B + CODE_BYTES, s, lane);
    fence_async_smem();
    __syncwarp();
    if (lane == 0) mbar_arrive(bar(B_FULL));
  }
  // The scales of a page are staged RAW_STAGES pages ahead by asynchronous copies, a lane its rows lane, lane + 32, .., and
  // re-ordered from there. (Loads into registers need the loop unrolled over the pages in flight.)
  auto raw = [&](int t) { return L::RAW + (t % L::RAW_STAGES) * SF_BYTES + lane * 8; };
  auto fetch = [&](int t) {
    if (t < num_tiles) {
      const uint8_t* src = g.ks + key_row(page_of(t)) * 8 + lane * 8;
#pragma unroll
      for (int i = 0; i < 4; ++i) cp_async8(base + raw(t) + i * 256, src + i * 256);
    }
    cp_async_commit();
  };
#pragma unroll 1
  for (int t = 0; t < L::RAW_STAGES; ++t) fetch(t);
  bool ok = true;
#pragma unroll 1
  for (int t = 0; t < num_tiles; ++t) {
    const int s = t % STAGES, use = t / STAGES;
    if (use > 0) ok = mbar_wait_warp(bar(A_EMPTY + s), (use - 1) & 1, guard, code0 + s);
    if (!ok) break;
    if (lane == 0) {
      mbar_expect_tx(bar(A_FULL + s), CODE_BYTES);
      tma_load_2d(base + OFF_A + s * STAGE_BYTES, k_map, 0, static_cast<int>(key_row(page_of(t))), bar(A_FULL + s));
    }
    cp_async_wait<L::RAW_STAGES - 1>();
    ScaleRegs regs;
#pragma unroll
    for (int i = 0; i < 4; ++i) regs.r[i] = *reinterpret_cast<const uint2*>(gbase + raw(t) + i * 256);
    store_scale_chunks(gbase + OFF_A + s * STAGE_BYTES + CODE_BYTES, regs, lane);
    __syncwarp();
    if (lane == 0) mbar_arrive(bar(A_FULL + s));
    fetch(t + L::RAW_STAGES);
  }
  cp_async_wait<0>();
  if (!ok)
    for (int t = max(0, num_tiles - STAGES); t < num_tiles; ++t)
      mbar_wait_drain(bar(A_FULL + t % STAGES), (t / STAGES) & 1);
}

// MMA warp: page t against the whole query tile into accumulator t % ACC_STAGES. The key scales of
// page t go to slot t & 1, copied as soon as the page has landed: the slot was last read by the MMAs of
// page t - 2, which had completed (their accumulator had been read out and released) before the MMAs
// of page t - 1 were issued; this holds for one or two accumulators.
static_assert(ACC_STAGES <= 2, "the two key-scale slots are protected by the accumulator hand-over only up to two accumulators");
template <int STAGES>
__device__ __forceinline__ void mma_role(uint32_t base, uint32_t bar0, uint32_t tmem, const Guard& guard, int num_tiles,
                                         int code0) {
  auto bar = [&](int i) { return bar0 + 8u * i; };
  constexpr uint32_t IDESC = idesc_nvf4(128, 128);
  const bool lead = elect_one();
  if (!mbar_wait_warp(bar(B_FULL), 0, guard, code0)) return;
  tc_fence_after();
  if (lead) {
    tmem_cp_scales(tmem + TM_SFB, desc_scale_chunk(base + Layout<STAGES>::B + CODE_BYTES));
    tmem_cp_scales(tmem + TM_SFB + 4, desc_scale_chunk(base + Layout<STAGES>::B + CODE_BYTES + 512));
  }
  const uint64_t b0 = desc_sw64_kmajor(base + Layout<STAGES>::B);
  for (int t = 0; t < num_tiles; ++t) {
    const int s = t % STAGES, st = t % ACC_STAGES;
    if (!mbar_wait_warp(bar(A_FULL + s), (t / STAGES) & 1, guard, code0 + 1 + s)) return;
    fence_async_smem();              // the producer's scale stores, for the copies below
    tc_fence_after();
    // the scale copy does not touch the accumulator: it goes out before the accumulator hand-over is awaited
    const uint64_t a0 = desc_sw64_kmajor(base + OFF_A + s * STAGE_BYTES);
    const uint32_t sfa = tmem + TM_SFA + (t & 1) * 8;
    if (lead) {
      tmem_cp_scales(sfa, desc_scale_chunk(base + OFF_A + s * STAGE_BYTES + CODE_BYTES));
      tmem_cp_scales(sfa + 4, desc_scale_chunk(base + OFF_A + s * STAGE_BYTES + CODE_BYTES + 512));
    }
    if (t >= ACC_STAGES) {
      if (!mbar_wait_warp(bar(ACC_EMPTY + st), ((t / ACC_STAGES) - 1) & 1, guard, code0 + 8 + st)) return;
      tc_fence_after();
    }
    if (lead) {
      // second K = 64: 32 bytes further along every row, its scales in the next four columns
#pragma unroll
      for (int kh = 0; kh < 2; ++kh)
        mma_nvf4(tmem + TM_ACC + st * 128, a0 + kh * 2, b0 + kh * 2, IDESC, sfa + kh * 4, tmem + TM_SFB + kh * 4, kh);
      tc_commit(bar(ACC_FULL + st));
      tc_commit(bar(A_EMPTY + s));
    }
  }
}

// L1 norm and squared L2 norm (both rounded up a little) of dequantised query row `row` of the tile.
__device__ __forceinline__ void query_row_norms(const Geometry& g, long long q_row0, int h, int row, float& l1, float& l2) {
  const long long r = (q_row0 + row) * g.hidx + h;
  const uint4* codes = reinterpret_cast<const uint4*>(g.qp + r * 64);
  const uint2 sc = __ldg(reinterpret_cast<const uint2*>(g.qs + r * 8));
  const unsigned long long lut = 0x0C08060403020100ULL;
  l1 = 0.f;
  l2 = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint4 v = __ldg(codes + i);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int gq = 0; gq < 2; ++gq) {
      const int grp = i * 2 + gq;
      const float unit = 0.5f * e4m3_to_float(static_cast<uint8_t>(((grp < 4 ? sc.x : sc.y) >> (8 * (grp & 3))) & 0x7fu));
      int sum = 0, squares = 0;
#pragma unroll
      for (int ww = 0; ww < 2; ++ww)
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const int m = static_cast<int>((lut >> (8 * ((w[gq * 2 + ww] >> (4 * e)) & 7u))) & 0xFFu);
          sum += m;
          squares += m * m;
        }
      l1 += static_cast<float>(sum) * unit;
      l2 += static_cast<float>(squares) * unit * unit;
    }
  }
  l1 *= 1.0001f;
  l2 *= 1.0001f;
}

struct Params {
  Geometry g;
  int* stats;                         // [0] CTAs run (counter), [1] tiles scored exactly in full, [3] bound violations,
                                      // [4] largest observed |approximate - exact| / delta (float bits); all cumulative
  const float* key_stats;             // [0] largest |key element|, [1] largest squared key norm (key_stats_kernel)
  int32_t* ids;                       // [B, Hidx, Qt, topk]
  int* status;
  int* fallbacks;                     // tiles scored exactly in full
  int* violations;                    // re-scored candidates whose two scores differed by more than delta
  int topk, cand;
};

// One CTA per (batch, index head, query tile), two CTAs per SM up to 16304 pages (the exact re-scoring of one
// overlaps the tensor-core scoring of the other): approximate tile scores of every key
// page on the tensor cores, then candidate selection and exact re-scoring.
// Warps 0-7 epilogue (lane quarter = warp & 3, query half = warp >> 2), warp 8 producer,
// warp 9 MMA issue (its elected lane).
template <int STAGES>
__global__ void __launch_bounds__(NUM_THREADS, 2)
fp4_nv_select_kernel(const __grid_constant__ CUtensorMap q_map, const __grid_constant__ CUtensorMap k_map, const Params p) {
  using L = Layout<STAGES>;
  extern __shared__ unsigned char smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  unsigned char* gbase = smem_raw + (base - raw);
  const Geometry& g = p.g;
  int* scores = reinterpret_cast<int*>(gbase + L::SCORES);
  const int score_bytes = (g.tiles * 4 + 15) & ~15;
  unsigned char* aux = gbase + L::SCORES + score_bytes;
  const uint32_t bar0 = base + L::SCORES + score_bytes;
  volatile int* misc = reinterpret_cast<volatile int*>(aux + 128);   // tmem base, abort, unsafe, l1q bits, l2q bits, k-th bound
  float* scratch_f = reinterpret_cast<float*>(aux + 192);            // [16]
  int* scratch_i = reinterpret_cast<int*>(aux + 256);                // [16]
  auto bar = [&](int i) { return bar0 + 8u * i; };

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int qt = g.len_q >> 7;
  const int qtile = blockIdx.x % qt;
  const int bh = blockIdx.x / qt;
  const int h = bh % g.hidx, b = bh / g.hidx;
  const int hk_idx = g.hk > 1 ? h : 0;
  const long long q_row0 = static_cast<long long>(b) * g.len_q + static_cast<long long>(qtile) * 128;
  const int num_tiles = g.tiles;
  const int rot = static_cast<int>((static_cast<unsigned>(qtile) * 37u) % static_cast<unsigned>(num_tiles));
  Guard guard{misc + 1, p.status};

  if (threadIdx.x == 0) {
    misc[1] = 0;
    for (int i = 0; i < STAGES; ++i) {
      mbar_init(bar(A_FULL + i), 2);      // the TMA transaction of the codes + the producer warp's scale stores
      mbar_init(bar(A_EMPTY + i), 1);
    }
    for (int i = 0; i < ACC_STAGES; ++i) {
      mbar_init(bar(ACC_FULL + i), 1);
      mbar_init(bar(ACC_EMPTY + i), 8);
    }
    mbar_init(bar(B_FULL), 2);
    fence_mbar_init();
  }
  if (warp == MMA_WARP) {
    tmem_alloc(smem_u32(const_cast<int*>(misc)), TM_COLS);
    tmem_relinquish();
  }
  for (int j = threadIdx.x; j < g.tiles; j += NUM_THREADS) scores[j] = static_cast<int>(0x80000000u);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = static_cast<uint32_t>(misc[0]);

  if (warp == TMA_WARP) {
    producer_role<STAGES>(g, &q_map, &k_map, base, gbase, bar0, guard, b, h, hk_idx, q_row0, 0, num_tiles, rot, num_tiles, lane,
                  0x500);
  } else if (warp == MMA_WARP) {
    mma_role<STAGES>(base, bar0, tmem, guard, num_tiles, 0x510);
    __syncwarp();
  } else {
    // epilogue: thread = key row of the page, this warp's 64-query half of the tile
    const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const int half = warp >> 2;
    bool ok = true;
    for (int t = 0; ok && t < num_tiles; ++t) {
      const int st = t % ACC_STAGES;
      bool w = mbar_wait(bar(ACC_FULL + st), (t / ACC_STAGES) & 1, guard, 0x540 + st);
      ok = __all_sync(0xffffffffu, w);
      if (!ok) break;
      tc_fence_after();
      const uint32_t t_acc = tmem + lane_base + TM_ACC + st * 128 + half * 64;
      uint32_t v[4][16];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld16(t_acc + c * 16, v[c]);
      tc_wait_ld();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(ACC_EMPTY + st));
      float m4[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        float m5[5];
#pragma unroll
        for (int jj = 0; jj < 5; ++jj)
          m5[jj] = max3(__uint_as_float(v[c][3 * jj]), __uint_as_float(v[c][3 * jj + 1]), __uint_as_float(v[c][3 * jj + 2]));
        m4[c] = fmaxf(max3(m5[0], m5[1], m5[2]), max3(m5[3], m5[4], __uint_as_float(v[c][15])));
      }
      const float m = warp_max(fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])));
      const int at = t + rot >= num_tiles ? t + rot - num_tiles : t + rot;
      if (lane == 0) atomicMax(&scores[at], f2ord(m));
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == MMA_WARP) {
    tc_fence_after();
    tmem_dealloc(tmem, TM_COLS);
  }
  if (misc[1]) return;

  // ------------------------------------------------------------- selection
  uint32_t* q_i8 = reinterpret_cast<uint32_t*>(gbase + OFF_A);
  uint32_t* k_i8 = q_i8 + 128 * FP4_ROW_WORDS;
  float* q_sc = reinterpret_cast<float*>(k_i8 + 128 * FP4_ROW_WORDS);
  float* k_sc = q_sc + 128 * 8;
  int32_t* cand_ids = reinterpret_cast<int32_t*>(gbase + L::CAND);
  int* cand_ex = reinterpret_cast<int*>(cand_ids + C_MAX);
  float* cand_apx = reinterpret_cast<float*>(cand_ex + C_MAX);     // approximate tile scores of the candidates
  int* near_s = reinterpret_cast<int*>(cand_apx + C_MAX);          // candidate needs its exact score
  const int C = p.cand;

  int32_t* out = p.ids + (static_cast<long long>(bh) * qt + qtile) * p.topk;

  fp4_stage_rows(q_i8, q_sc, g.qp + (q_row0 * g.hidx + h) * 64, static_cast<long long>(g.hidx) * 64,
                 g.qs + (q_row0 * g.hidx + h) * 8, static_cast<long long>(g.hidx) * 8, 0.25f);
  if (threadIdx.x == 0) { misc[2] = 0; misc[3] = 0; misc[4] = 0; misc[5] = __float_as_int(-INFINITY); atomicAdd(p.stats, 1); }
  for (int c = threadIdx.x; c < C_MAX; c += NUM_THREADS) cand_ex[c] = static_cast<int>(0x80000000u);
  __syncthreads();
  if (threadIdx.x < 128) {
    float l1, l2;
    query_row_norms(g, q_row0, h, threadIdx.x, l1, l2);
    atomicMax(const_cast<int*>(misc + 3), __float_as_int(l1));
    atomicMax(const_cast<int*>(misc + 4), __float_as_int(l2));
  }
  float thr = 0.f;
  if (warp == 0) {
    // C-th largest approximate score and the candidate set (ties at the threshold in index order)
    const unsigned* keys = reinterpret_cast<const unsigned*>(scores);
    const unsigned lt_mask = (1u << lane) - 1u;
    unsigned T = 0;
    for (int bit = 31; bit >= 0; --bit) {
      const unsigned trial = T | (1u << bit);
      int cnt = 0;
      for (int j = lane; j < g.tiles; j += 32) cnt += ((keys[j] ^ 0x80000000u) >= trial) ? 1 : 0;
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, d);
      if (cnt >= C) T = trial;
    }
    int n_gt = 0;
    for (int j = lane; j < g.tiles; j += 32) n_gt += ((keys[j] ^ 0x80000000u) > T) ? 1 : 0;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) n_gt += __shfl_xor_sync(0xffffffffu, n_gt, d);
    const int need_eq = C - n_gt;
    int out_run = 0, eq_run = 0;
    for (int base_j = 0; base_j < g.tiles; base_j += 32) {
      const int j = base_j + lane;
      const unsigned u = j < g.tiles ? (keys[j] ^ 0x80000000u) : 0u;
      const bool is_gt = j < g.tiles && u > T;
      const bool is_eq = j < g.tiles && u == T;
      const unsigned eq_ballot = __ballot_sync(0xffffffffu, is_eq);
      const bool take = is_gt || (is_eq && eq_run + __popc(eq_ballot & lt_mask) < need_eq);
      const unsigned take_ballot = __ballot_sync(0xffffffffu, take);
      if (take) {
        const int pos = out_run + __popc(take_ballot & lt_mask);
        cand_ids[pos] = j;
        cand_apx[pos] = ord2f(static_cast<int>(u ^ 0x80000000u));
      }
      out_run += __popc(take_ballot);
      eq_run += __popc(eq_ballot);
    }
    thr = ord2f(static_cast<int>(T ^ 0x80000000u));
  }
  __syncthreads();
  // exact tile score of one page: max over the 128 x 128 dots, whole CTA
  auto exact_page = [&](int pg) -> float {
    const long long page = (static_cast<long long>(b) * g.tiles + pg) * g.hk + hk_idx;
    fp4_stage_rows(k_i8, k_sc, g.kp + page * 128 * 64, 64, g.ks + page * 128 * 8, 8, 1.0f);
    __syncthreads();
    float m = -INFINITY;
    if (threadIdx.x < 256) m = fp4_block_max_mma(q_i8, q_sc, k_i8, k_sc, warp, lane);
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, d));
    return m;                              // per-warp maximum; lane 0 publishes it
  };
  // Approximate and exact tile score differ by at most delta (the sum of |q_d k_d| bounded by
  // Hoelder and by Cauchy-Schwarz), so candidates more than 2 delta apart are ordered by their
  // approximate scores for certain: only a candidate with another one within 2 delta is re-scored.
  const float delta = EPS * fminf(__int_as_float(misc[3]) * p.key_stats[0],
                                  sqrtf(__int_as_float(misc[4])) * sqrtf(p.key_stats[1] * 1.0001f));
  const float two = 2.f * delta;
  for (int c = threadIdx.x; c < C; c += NUM_THREADS) {
    const float a = cand_apx[c];
    int near = 0;
#pragma unroll 4
    for (int j = 0; j < C; ++j) near |= static_cast<int>(j != c) & static_cast<int>(!(fabsf(a - cand_apx[j]) > two));
    near_s[c] = near;
  }
  __syncthreads();
  for (int c = 0; c < C; ++c) {
    if (!near_s[c]) continue;
    const float m = exact_page(cand_ids[c]);
    if (lane == 0) atomicMax(&cand_ex[c], f2ord(m));
    __syncthreads();
  }
  // The bound checks itself: both scores of a re-scored candidate are in hand. A difference above
  // delta (the tensor core did not behave as assumed) sends the tile to the exact path below.
  for (int c = threadIdx.x; c < C; c += NUM_THREADS)
    if (near_s[c]) {
      const float diff = fabsf(cand_apx[c] - ord2f(cand_ex[c]));
      if (delta > 0.f) atomicMax(p.stats + 4, __float_as_int(diff / delta));
      if (!(diff <= delta)) {
        misc[2] = 1;
        atomicAdd(p.violations, 1);
      }
    }
  // rank of a candidate = number of candidates that beat it in (exact score descending, page
  // ascending): by the approximate scores when more than 2 delta apart, else by the exact ones
  for (int c = threadIdx.x; c < C; c += NUM_THREADS) {
    const float a = cand_apx[c], e = ord2f(cand_ex[c]);
    const int id = cand_ids[c];
    int rank = 0;
#pragma unroll 4
    for (int j = 0; j < C; ++j) {
      const float d = cand_apx[j] - a, ej = ord2f(cand_ex[j]);
      const int gt = static_cast<int>(d > two), lt = static_cast<int>(d < -two);
      const int exact = static_cast<int>(ej > e) | (static_cast<int>(ej == e) & static_cast<int>(cand_ids[j] < id));
      rank += gt | (((gt | lt) ^ 1) & exact);
    }
    if (rank < p.topk) out[rank] = id;
    if (rank == p.topk - 1) misc[5] = __float_as_int(near_s[c] ? e : a - delta);   // lower bound of the k-th exact score
  }
  __syncthreads();
  if (threadIdx.x == 0 && !misc[2]) misc[2] = ((C >= g.tiles) || (__int_as_float(misc[5]) > thr + delta)) ? 0 : 1;
  __syncthreads();
  if (misc[2]) {
    float* row = reinterpret_cast<float*>(scores);
    for (int pg = 0; pg < g.tiles; ++pg) {
      const float m = exact_page(pg);
      if (lane == 0) scratch_f[warp] = m;
      __syncthreads();
      if (threadIdx.x == 0) {
        float mm = scratch_f[0];
        for (int w = 1; w < NUM_THREADS / 32; ++w) mm = fmaxf(mm, scratch_f[w]);
        row[pg] = mm;
      }
      __syncthreads();
    }
    block_topk(row, g.tiles, p.topk, out, scratch_f, scratch_i);
    if (threadIdx.x == 0 && p.fallbacks) atomicAdd(p.fallbacks, 1);
  }
}

// ---------------------------------------------------------------- exact tile scores by pruning
// The exact score of a (query tile, key page) pair is the maximum of 128 x 128 exact dots. The
// tensor cores give every dot within delta of its exact value, so only the elements whose
// approximate value reaches (largest approximate value - 2 delta) can hold the exact maximum:
// any other element is below the exact value of the approximate arg-max. Those few elements
// (usually one) are queued with the other fifteen of their group of columns and evaluated, when the queue fills up and at
// the end, with the canonical arithmetic (integer group sums, scaled and added in group order) straight from the codes in
// global memory. Same scores, bit for bit, as fp4_score_mma_kernel, which evaluates all 16384 elements of a pair exactly.
// The exact maximum of every evaluated group is also compared with its approximate one: a difference above delta is
// counted and the pair is re-done by evaluating all of its elements.
struct PruneParams {
  Geometry g;
  int* stats;                         // as in Params
  float* tile_scores;                 // [B, Hidx, Qt, tiles]
  int* status;
  int* violations;
  int pages_per_cta, chunks;
};

// Integer dot of one 16-element scale group straight from the e2m1 codes (two words per row):
// magnitudes 2 |value| through a byte-permute table, the sign of each product from the xor of
// the code sign bits, products of either sign summed apart with dp4a.
__device__ __forceinline__ int fp4_group_sum(uint32_t q0, uint32_t q1, uint32_t k0, uint32_t k1) {
  constexpr uint32_t LUT_LO = 0x03020100u, LUT_HI = 0x0C080604u;      // 2 |value| of codes 0..7
  int pos = 0, neg = 0;
#pragma unroll
  for (int w = 0; w < 2; ++w) {
    const uint32_t wq = w ? q1 : q0, wk = w ? k1 : k0;
    const uint32_t sg = ((wq ^ wk) >> 3) & 0x11111111u;               // 1 where the product is negative
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
      const uint32_t mq = __byte_perm(LUT_LO, LUT_HI, (wq >> (16 * hh)) & 0x7777u);
      const uint32_t mk = __byte_perm(LUT_LO, LUT_HI, (wk >> (16 * hh)) & 0x7777u);
      const uint32_t ng = __byte_perm(0x0000FF00u, 0u, (sg >> (16 * hh)) & 0x1111u);
      pos = __dp4a(static_cast<int>(mq & ~ng), static_cast<int>(mk), pos);
      neg = __dp4a(static_cast<int>(mq & ng), static_cast<int>(mk), neg);
    }
  }
  return pos - neg;
}

// canonical dot of a query row and a key row (16 code words and 8 e4m3 scales each); everything
// is requested from memory before the first use
__device__ __forceinline__ float fp4_exact_dot(const uint8_t* __restrict__ q_codes, const uint8_t* __restrict__ q_scales,
                                               const uint8_t* __restrict__ k_codes, const uint8_t* __restrict__ k_scales) {
  uint4 qw[4], kw[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    qw[i] = __ldg(reinterpret_cast<const uint4*>(q_codes) + i);
    kw[i] = __ldg(reinterpret_cast<const uint4*>(k_codes) + i);
  }
  const uint2 qs8 = __ldg(reinterpret_cast<const uint2*>(q_scales));
  const uint2 ks8 = __ldg(reinterpret_cast<const uint2*>(k_scales));
  const uint32_t* q32 = reinterpret_cast<const uint32_t*>(qw);
  const uint32_t* k32 = reinterpret_cast<const uint32_t*>(kw);
  float acc = 0.f;
#pragma unroll
  for (int gq = 0; gq < 8; ++gq) {
    const int sum = fp4_group_sum(q32[2 * gq], q32[2 * gq + 1], k32[2 * gq], k32[2 * gq + 1]);
    const uint8_t qb = static_cast<uint8_t>(((gq < 4 ? qs8.x : qs8.y) >> (8 * (gq & 3))) & 0xFFu);
    const uint8_t kb = static_cast<uint8_t>(((gq < 4 ? ks8.x : ks8.y) >> (8 * (gq & 3))) & 0xFFu);
    const float c = (0.25f * e4m3_to_float(qb)) * e4m3_to_float(kb);
    acc = fmaf(static_cast<float>(sum), c, acc);
  }
  return acc;
}

constexpr int PR_QCAP = 2048;                // queued groups of elements per CTA
// A queue that has grown beyond this is emptied at the next page's meeting: there always is room for all 1024 groups of a
// page. (Emptied at the end only, every page behind two all-equal ones, or behind 2000 others, had to be evaluated in full.
// Selection of 160 lists, us: 4096 pages 232000 -> 3150, 1024 pages, four of zeros, 113000 -> 1580.)
constexpr int PR_DRAIN = PR_QCAP - 1024;
constexpr int PR_PAGES_MAX = 3072;           // pages of a CTA: the results of more would leave one CTA to an SM
constexpr int PR_OFF_AUX = Layout<A_STAGES>::CAND;         // barriers (128 bytes), misc (128 bytes)
constexpr int PR_OFF_QUEUE = PR_OFF_AUX + 256;            // [PR_QCAP] groups waiting for their exact values
constexpr int PR_OFF_APX = PR_OFF_QUEUE + PR_QCAP * 4;     // [PR_QCAP] their largest approximate values
constexpr int PR_OFF_RES = PR_OFF_APX + PR_QCAP * 4;       // [pages per CTA] exact maxima as ordered ints
                                                           // then [pages per CTA] flags: pair to be re-done in full
static_assert(2 * (PR_OFF_RES + PR_PAGES_MAX * 8 + 1024 + 1024) <= 228 * 1024, "two CTAs of the pruning scorer to an SM");

// One CTA per (batch, index head, query tile, chunk of key pages), two CTAs per SM. Warps 0-7 epilogue (lane
// quarter = warp & 3, query half = warp >> 2), warp 8 producer, warp 9 MMA issue. The epilogue
// warps meet once per page at a named barrier (largest approximate value of the page) and twice
// more where they empty the queue; a warp whose bounded wait gave up keeps
// taking part in those meetings, so nobody is left waiting for it.
__global__ void __launch_bounds__(NUM_THREADS, 2)
fp4_nv_prune_kernel(const __grid_constant__ CUtensorMap q_map, const __grid_constant__ CUtensorMap k_map,
                    const PruneParams p) {
  extern __shared__ unsigned char smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  unsigned char* gbase = smem_raw + (base - raw);
  const Geometry& g = p.g;
  unsigned char* aux = gbase + PR_OFF_AUX;
  const uint32_t bar0 = base + PR_OFF_AUX;
  // tmem base, abort flag, L1 bits, largest key scale byte, queue length, largest |approximate - exact| / delta (float bits)
  volatile int* misc = reinterpret_cast<volatile int*>(aux + 128);
  // three slots for a page each: its largest approximate value, and whether the queue is to be emptied before the page
  // queues anything (one word, so that everybody reads both at once)
  volatile int* peak = misc + 6;
  auto peak_word = [&](int slot) { return reinterpret_cast<volatile unsigned long long*>(peak + slot); };
  constexpr unsigned long long NO_PEAK = 0x80000000ull;
  int* queue = reinterpret_cast<int*>(gbase + PR_OFF_QUEUE);
  float* queue_apx = reinterpret_cast<float*>(gbase + PR_OFF_APX);
  int* res = reinterpret_cast<int*>(gbase + PR_OFF_RES);
  int* redo = res + p.pages_per_cta;
  auto bar = [&](int i) { return bar0 + 8u * i; };

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int qt = g.len_q >> 7;
  const int chunk = blockIdx.x % p.chunks;
  const int list = blockIdx.x / p.chunks;            // (batch * Hidx + head) * Qt + query tile
  const int qtile = list % qt;
  const int bh = list / qt;
  const int h = bh % g.hidx, b = bh / g.hidx;
  const int hk_idx = g.hk > 1 ? h : 0;
  const long long q_row0 = static_cast<long long>(b) * g.len_q + static_cast<long long>(qtile) * 128;
  const int page0 = chunk * p.pages_per_cta;
  const int num_tiles = min(p.pages_per_cta, g.tiles - page0);
  Guard guard{misc + 1, p.status};
  // The top-k kernel that follows is launched as a programmatic dependent: its CTAs may be placed as
  // soon as resources free up; they wait for this whole grid (griddepcontrol.wait) before reading scores.
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  if (threadIdx.x == 0) {
    misc[1] = 0;
    misc[2] = 0;
    misc[3] = 0;
    misc[4] = 0;
    misc[5] = 0;
    for (int i = 0; i < 3; ++i) *peak_word(2 * i) = NO_PEAK;
    for (int i = 0; i < A_STAGES; ++i) {
      mbar_init(bar(A_FULL + i), 2);
      mbar_init(bar(A_EMPTY + i), 1);
    }
    for (int i = 0; i < ACC_STAGES; ++i) {
      mbar_init(bar(ACC_FULL + i), 1);
      mbar_init(bar(ACC_EMPTY + i), 8);
    }
    mbar_init(bar(B_FULL), 2);
    fence_mbar_init();
  }
  if (warp == MMA_WARP) {
    tmem_alloc(smem_u32(const_cast<int*>(misc)), TM_COLS);
    tmem_relinquish();
  }
  for (int t = threadIdx.x; t < num_tiles; t += NUM_THREADS) {
    res[t] = INT_MIN;
    redo[t] = 0;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = static_cast<uint32_t>(misc[0]);

  if (warp == TMA_WARP) {
    producer_role<A_STAGES>(g, &q_map, &k_map, base, gbase, bar0, guard, b, h, hk_idx, q_row0, page0, num_tiles, 0, num_tiles, lane,
                  0x580);
  } else if (warp == MMA_WARP) {
    mma_role<A_STAGES>(base, bar0, tmem, guard, num_tiles, 0x590);
    __syncwarp();
  } else {
    // epilogue: thread = key row of the page, this warp's 64-query half of the tile
    auto meet = [&]() { asm volatile("bar.sync 1, 256;" ::: "memory"); };
    if (threadIdx.x == 0) atomicAdd(p.stats, 1);
    if (threadIdx.x < 128) {
      float l1, l2;
      query_row_norms(g, q_row0, h, threadIdx.x, l1, l2);
      atomicMax(const_cast<int*>(misc + 2), __float_as_int(l1));
    }
    {
      // largest scale among this CTA's key pages: 64 threads per page, 16 bytes each
      uint32_t seen = 0;
      for (int t0 = threadIdx.x >> 6; t0 < num_tiles; t0 += 32) {     // eight pages' loads in flight
        uint4 w[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int t = t0 + 4 * i;
          const long long page = (static_cast<long long>(b) * g.tiles + page0 + t) * g.hk + hk_idx;
          w[i] = make_uint4(0u, 0u, 0u, 0u);
          if (t < num_tiles) w[i] = __ldg(reinterpret_cast<const uint4*>(g.ks + page * 1024) + (threadIdx.x & 63));
        }
#pragma unroll
        for (int i = 0; i < 8; ++i)
          seen = max_scale_bytes(max_scale_bytes(max_scale_bytes(max_scale_bytes(seen, w[i].x), w[i].y), w[i].z), w[i].w);
      }
      uint32_t m = top_byte(seen);
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, d));
      if (lane == 0) atomicMax(const_cast<int*>(misc + 3), static_cast<int>(m));
    }
    meet();
    const float delta = EPS * __int_as_float(misc[2]) * key_bound_from_scale_byte(static_cast<uint32_t>(misc[3]));
    const float two = 2.f * delta;
    const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const int half = warp >> 2;
    const int key_row = (warp & 3) * 32 + lane;
    // the queued groups, sixteen threads each: exact values of the group's elements into the page's maximum
    auto evaluate_queue = [&]() {
      const int queued = misc[4];
      for (int i = static_cast<int>(threadIdx.x) >> 4; i < ((queued + 15) & ~15); i += 16) {
        const bool live = i < queued;
        const int e = live ? queue[i] : 0, t = e >> 10, krow = (e >> 3) & 127;
        float m = -INFINITY;
        if (live) {
          const long long page = (static_cast<long long>(b) * g.tiles + page0 + t) * g.hk + hk_idx;
          const long long qrow = (q_row0 + (e & 7) * 16 + (threadIdx.x & 15)) * g.hidx + h;
          const float x = fp4_exact_dot(g.qp + qrow * 64, g.qs + qrow * 8, g.kp + (page * 128 + krow) * 64,
                                        g.ks + (page * 128 + krow) * 8);
          if (x == x) m = x;
        }
#pragma unroll
        for (int d = 8; d > 0; d >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, d));
        if (live && (threadIdx.x & 15) == 0 && m > -INFINITY) {
          atomicMax(res + t, f2ord(m));
          // the largest value of a group, exact and approximate, differ by at most delta, as its elements do
          const float diff = fabsf(queue_apx[i] - m);
          if (delta > 0.f) atomicMax(const_cast<int*>(misc + 5), __float_as_int(diff / delta));
          if (!(diff <= delta)) {
            redo[t] = 1;
            atomicAdd(p.violations, 1);
          }
        }
      }
    };
    bool ok = true;
    for (int t = 0; t < num_tiles; ++t) {
      const int st = t % ACC_STAGES, slot = 2 * (t % 3);
      if (ok) {
        bool w = mbar_wait(bar(ACC_FULL + st), (t / ACC_STAGES) & 1, guard, 0x5c0 + st);
        ok = __all_sync(0xffffffffu, w);
      }
      uint32_t v[4][16];
      float m4[4], mine = -INFINITY;
      if (ok) {
        tc_fence_after();
        const uint32_t t_acc = tmem + lane_base + TM_ACC + st * 128 + half * 64;
#pragma unroll
        for (int c = 0; c < 4; ++c) tmem_ld16(t_acc + c * 16, v[c]);
        tc_wait_ld();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(ACC_EMPTY + st));
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          float m5[5];
#pragma unroll
          for (int jj = 0; jj < 5; ++jj)
            m5[jj] = max3(__uint_as_float(v[c][3 * jj]), __uint_as_float(v[c][3 * jj + 1]), __uint_as_float(v[c][3 * jj + 2]));
          m4[c] = fmaxf(max3(m5[0], m5[1], m5[2]), max3(m5[3], m5[4], __uint_as_float(v[c][15])));
        }
        mine = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3]));
        const float m = warp_max(mine);
        if (lane == 0) atomicMax(const_cast<int*>(peak + slot), f2ord(m));
      }
      meet();
      const unsigned long long top = *peak_word(slot);
      // the slot of the page before is free now (everyone read it before this meeting); it is
      // next written for page t + 2, after the meeting of page t + 1
      if (threadIdx.x == 0 && t > 0) *peak_word(2 * ((t - 1) % 3)) = NO_PEAK;
      if ((top >> 32) != 0) {                  // everybody, and nobody queues anything until all are through
        evaluate_queue();
        meet();
        if (threadIdx.x == 0) misc[4] = 0;
        meet();
      }
      if (ok) {
        const float thr = ord2f(static_cast<int>(top)) - two;
        // Groups of sixteen columns of this key row that hold an element that may be the maximum. Everyone waits for this
        // at the page's next meeting, and a lone lane does it: the column is left to the evaluation (looking for it here,
        // with its approximate value, took the lane longer than the page took everyone: 1070 cycles of an SM per page).
        if (!(mine < thr)) {
#pragma unroll
          for (int c = 0; c < 4; ++c)
            if (!(m4[c] < thr)) {
              const int at = atomicAdd(const_cast<int*>(misc + 4), 1);
              queue[at] = (t << 10) | (key_row << 3) | (half * 4 + c);
              queue_apx[at] = m4[c];
              if (at >= PR_DRAIN) peak[2 * ((t + 1) % 3) + 1] = 1;
            }
        }
      }
    }
    meet();
    evaluate_queue();
    meet();
    if (threadIdx.x == 0 && misc[5] > 0) atomicMax(p.stats + 4, misc[5]);      // one global atomic per CTA
    // a pair whose bound was violated: every one of its 16384 elements, exactly (256 threads)
    for (int t = 0; t < num_tiles; ++t) {
      if (!redo[t]) continue;
      const long long page = (static_cast<long long>(b) * g.tiles + page0 + t) * g.hk + hk_idx;
      float m = -INFINITY;
      for (int e = threadIdx.x; e < 128 * 128; e += 256) {
        const long long qrow = (q_row0 + (e & 127)) * g.hidx + h;
        m = fmaxf(m, fp4_exact_dot(g.qp + qrow * 64, g.qs + qrow * 8, g.kp + (page * 128 + (e >> 7)) * 64,
                                   g.ks + (page * 128 + (e >> 7)) * 8));
      }
      atomicMax(res + t, f2ord(m));
    }
    meet();
    if (ok)
      for (int t = threadIdx.x; t < num_tiles; t += 256)
        p.tile_scores[static_cast<long long>(list) * g.tiles + page0 + t] = ord2f(res[t]);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == MMA_WARP) {
    tc_fence_after();
    tmem_dealloc(tmem, TM_COLS);
  }
}

// ---------------------------------------------------------------- host side
static int make_maps(CUtensorMap* qm, CUtensorMap* km, const void* qp, const void* kp, int batch, int hidx, int len_q,
                     long long k_rows) {
  {
    const cuuint64_t dims[3] = {64, static_cast<cuuint64_t>(hidx), static_cast<cuuint64_t>(batch) * len_q};
    const cuuint64_t strides[2] = {64, static_cast<cuuint64_t>(hidx) * 64};
    const cuuint32_t box[3] = {64, 1, 128};
    const cuuint32_t steps[3] = {1, 1, 1};
    if (encode_tiled(qm, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(qp), dims, strides, box, steps,
                     CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B))
      return set_error(SB_ERR_CUDA, "cuTensorMapEncodeTiled failed for the query codes");
  }
  {
    const cuuint64_t dims[2] = {64, static_cast<cuuint64_t>(k_rows)};
    const cuuint64_t strides[1] = {64};
    const cuuint32_t box[2] = {64, 128};
    const cuuint32_t steps[2] = {1, 1};
    if (encode_tiled(km, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(kp), dims, strides, box, steps,
                     CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B))
      return set_error(SB_ERR_CUDA, "cuTensorMapEncodeTiled failed for the key codes");
  }
  return SB_OK;
}

static bool aligned(const void* p, uintptr_t a) { return (reinterpret_cast<uintptr_t>(p) & (a - 1)) == 0; }


// ---------------------------------------------------------------- per-query page scores (ragged / paged / causal)
// scores[h, page, query] = max over the visible keys of a page, straight off the NVFP4 MMA: the output the
// reference's scorer produces (indexers/fp4/vendor_minimax_msa/src/sm100/fp4_indexer.py:201-1108, decode form
// :1110-1229), values in the tensor core's own accumulation order (within delta of the canonical ones; the
// reference's gate for this output is rtol 1e-4 / atol 1e-3, benchmarks/ch4_selectors/harness.py:33-42).
// Here the QUERY tile is the M operand (one tensor-memory lane = one query, so the maximum over the keys of a
// page is a maximum along a lane) and the key pages stream through as the N operand.
// An item is a (request, query tile, head) -- or, packed (decode batches), a (request, KV head, block of 16 group heads)
// with rows = (query, head) pairs; its pages are the visible ones of its request. The pages of all items, one after
// the other, are cut into equal runs, one per CTA: two CTAs per SM (160 tensor-memory columns each) stay for the whole
// launch, whatever the lengths, which only the device knows. With a CTA per (item, 16 to 64 pages) the last round was
// nearly empty and every CTA paid its start (descriptors, first loads: 4000 cycles) for 16 pages of 1000.
// Launches of few CTAs give each a share of one item's pages instead, found by division (RUNS = false): there a run levels
// nothing, and the way to its place is longer than the rest of the start (see the host side).
// Warps 0-3 epilogue (lane quarter = warp), warp 4 copies the codes, warp 6 brings the scales, warp 5 issues the MMAs (its
// elected lane).
struct QueryScoreParams {
  const uint8_t *qp, *qs, *kp, *ks;
  const int32_t *cu_q, *cu_k, *cu_pages, *kv_indices, *qo_offset;
  float* out;                          // [Hq, tiles_out, total_q], pre-filled with -inf
  int* status;
  int batch, hq, hk, total_q, total_pages, qt_max, tiles_out, causal;
  int group, subs;                     // query heads of a KV head; items of a KV head (heads, or blocks of 16 of them)
  int share, shares;                   // launches without runs: pages of a CTA, CTAs of an item
};
constexpr int QS_THREADS = 224;
constexpr int QS_PACK_Q = 8, QS_PACK_HEADS = 16;
constexpr int QS_AHEAD = 4;            // pages whose scales are on their way to their staging ring
// Shared memory and barriers: eight pages in flight and two query tiles. With shares of packed items (THREE) one query tile and
// four pages (and 80 registers) leave room for a third CTA on the SM, which is set up by the time one of the other two gives up
// its tensor memory: 1300 of the 4900 to 8600 cycles of a CTA. One-token requests in a graph, us: 1024 of 100 to 400 keys 17.6 ->
// 16.6, 2048 30.6 -> 28.5, 1500 of 10 to 128 19.5 -> 17.2, 600 of 500 to 900 16.9 -> 17.5; six pages, which leave less L1, 17.2,
// 29.3, 17.5 and 18.0. Not for query tiles of one head, whose launches of shares are one round: 16 requests 7.2 -> 8.8.
template <bool THREE>
struct QsMap {
  static constexpr int STAGES = THREE ? 4 : 8, Q_TILES = THREE ? 1 : 2;
  static constexpr int Q = STAGES * STAGE_BYTES;             // query tiles: codes + scales
  static constexpr int RAW = Q + Q_TILES * STAGE_BYTES;      // staging ring: the scales of a page as they are in memory
  static constexpr int AUX = RAW + QS_AHEAD * SF_BYTES;      // barriers, misc (64 bytes), sums (64)
  enum { K_FULL = 0, K_EMPTY = STAGES, Q_FULL = 2 * STAGES, Q_EMPTY = Q_FULL + Q_TILES, BAR_ACC_FULL = Q_EMPTY + Q_TILES,
         BAR_ACC_EMPTY, BARS };
  static constexpr int BAR_BYTES = (BARS * 8 + 63) & ~63;
  static constexpr int SMEM = AUX + BAR_BYTES + 128 + 1024;
};
static_assert(3 * (QsMap<true>::SMEM + 1024) <= 228 * 1024, "three CTAs to an SM");
// tensor memory: the accumulator, two slots of key scales, two of query scales
constexpr int QS_SFK = 128, QS_SFQ = 144;
static_assert(QS_SFQ + 16 <= TM_COLS, "tensor memory map");

// What a request means for the scorer; qtiles is 0 where there is nothing to score.
struct Request {
  int q_begin, q_len, q_rows, k_len, page_begin, pages, offset, qtiles;     // q_rows: query rows that exist in q
  template <bool PACKED>
  static __device__ __forceinline__ Request load(const QueryScoreParams& p, int b) {
    Request r;
    r.q_begin = p.cu_q[b];
    r.q_len = p.cu_q[b + 1] - r.q_begin;
    r.k_len = p.cu_k[b + 1] - p.cu_k[b];
    r.page_begin = p.cu_pages[b];
    r.pages = min(min((r.k_len + 127) >> 7, p.tiles_out), p.cu_pages[b + 1] - r.page_begin);
    r.q_rows = min(r.q_len, p.total_q - r.q_begin);
    if (PACKED) r.q_rows = min(r.q_rows, QS_PACK_Q);
    r.offset = p.causal ? (p.qo_offset ? p.qo_offset[b] : r.k_len - r.q_len) : 0;
    const bool nothing = r.q_begin < 0 || r.q_rows <= 0 || r.k_len <= 0 || r.page_begin < 0 || r.pages <= 0;
    r.qtiles = nothing ? 0 : min((r.q_rows + 127) >> 7, p.qt_max);
    return r;
  }
  // pages that query tile j sees: up to its last live query's horizon
  __device__ __forceinline__ int visible(const QueryScoreParams& p, int j) const {
    if (!p.causal) return pages;
    const long long horizon = min(static_cast<long long>(j) * 128 + 128, static_cast<long long>(q_rows)) - 1 + offset;
    return horizon < 0 ? 0 : static_cast<int>(min(static_cast<long long>(pages), (horizon >> 7) + 1));
  }
  // sum of visible() over all tiles: a full tile j sees max(0, min(pages, j + c)), c = ((127 + offset) >> 7) + 1
  __device__ __forceinline__ long long total(const QueryScoreParams& p) const {
    if (qtiles == 0) return 0;
    const long long n = qtiles - 1, last = visible(p, qtiles - 1);
    if (!p.causal) return n * pages + last;
    const long long c = ((127LL + offset) >> 7) + 1;
    const long long a = min(n, max(0LL, 1 - c)), sat = min(n, max(a, pages - c));    // tiles from a on see some, from sat all
    return (a + sat - 1 + 2 * c) * (sat - a) / 2 + (n - sat) * pages + last;
  }
};

// A role's place in the CTA's run of pages: the same items in the same order in every role.
template <bool PACKED, bool RUNS>
struct ScoreWalk {
  int left;                      // pages of the run from the current item's `page` on
  int b, j, kvh, sub;            // item: request, query tile, KV head, query head or head block of it
  int page, end;                 // next page, visible pages of the item
  Request r;
  ScoreWalk() = default;
  __device__ __forceinline__ ScoreWalk(const QueryScoreParams& p, volatile const int* start) {
    if constexpr (RUNS) {
      left = start[5];
      b = start[0];
      j = start[1];
      kvh = start[2];
      sub = start[3];
      page = start[4];
      r = Request::load<PACKED>(p, b);
      end = r.visible(p, j);
    } else {                         // `left` is 0 where the share is empty
      int rest = static_cast<int>(blockIdx.x) / p.shares;
      page = (static_cast<int>(blockIdx.x) - rest * p.shares) * p.share;
      const int items = p.hk * p.subs;               // of a query tile
      b = rest / items;
      rest -= b * items;
      kvh = rest / p.subs;
      sub = rest - kvh * p.subs;
      j = 0;
      if (!PACKED) {
        rest = b;
        b = rest / p.qt_max;
        j = rest - b * p.qt_max;
      }
      r = Request::load<PACKED>(p, b);
      end = j < r.qtiles ? r.visible(p, j) : 0;
      left = max(0, min(p.share, end - page));
    }
  }
  // pages of the run in the current item
  __device__ __forceinline__ int count() const { return min(left, end - page); }
  __device__ __forceinline__ void next(const QueryScoreParams& p) {
    if constexpr (!RUNS) {
      left = 0;
      return;
    }
    left -= count();
    page = 0;
    if (left <= 0 || ++sub < p.subs) return;
    sub = 0;
    if (++kvh < p.hk) return;
    kvh = 0;
    do {
      ++j;
      while (j >= r.qtiles) {
        if (++b >= p.batch) {
          left = 0;
          return;
        }
        r = Request::load<PACKED>(p, b);
        j = 0;
      }
      end = r.visible(p, j);
    } while (end == 0);
  }
  __device__ __forceinline__ int head0(const QueryScoreParams& p) const {      // head of row 0
    return kvh * p.group + (PACKED ? sub * QS_PACK_HEADS : sub);
  }
};

// n / d, both positive; mostly by the short division
__device__ __forceinline__ long long quotient(long long n, long long d) {
  return ((n | d) >> 32) == 0 ? static_cast<long long>(static_cast<uint32_t>(n) / static_cast<uint32_t>(d)) : n / d;
}

// Where the run of this CTA begins: request, query tile, KV head, item of it, page; number of pages (0: nothing). All threads,
// each with a slice of the requests, once; then the warp that has the run's request looks through its slice. (One warp, 32
// requests to a step and up to twice over all of them, took 250 steps of dependent loads for 4096 requests while the others
// waited. One-token requests of 100 to 400 keys in a graph, us: 256 15.0 -> 10.9, 1024 40.4 -> 19.5, 4096 160 -> 59, 16384 788 -> 231.)
template <bool PACKED>
__device__ __forceinline__ void find_run(const QueryScoreParams& p, volatile int* start, volatile long long* warp_sums, int warp,
                                         int lane) {
  const int heads = p.hk * p.subs;
  auto scan = [&](long long v) {
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const long long o = __shfl_up_sync(0xffffffffu, v, d);
      if (lane >= d) v += o;
    }
    return v;
  };
  const int slice = (p.batch + QS_THREADS - 1) / QS_THREADS;
  const int lo = min(static_cast<int>(threadIdx.x) * slice, p.batch), hi = min(lo + slice, p.batch);
  long long mine = 0;
#pragma unroll 4
  for (int b = lo; b < hi; ++b) mine += Request::load<PACKED>(p, b).total(p);
  mine *= heads;
  const long long sum = scan(mine);
  if (lane == 31) warp_sums[warp] = sum;
  if (threadIdx.x == 0) start[5] = 0;
  __syncthreads();
  long long total = 0, before = sum - mine;        // pages of all requests, pages before this thread's slice
#pragma unroll
  for (int w = 0; w < QS_THREADS / 32; ++w) {
    const long long ws = warp_sums[w];
    if (w < warp) before += ws;
    total += ws;
  }
  const long long per = max(2LL, quotient(total + gridDim.x - 1, gridDim.x)), first = per * blockIdx.x;
  if (first >= total) return;
  const unsigned owner = __ballot_sync(0xffffffffu, first >= before && first < before + mine);
  if (owner == 0) return;
  const int at = __ffs(owner) - 1, end = __shfl_sync(0xffffffffu, hi, at);
  int begin = __shfl_sync(0xffffffffu, lo, at);
  long long rest = first - __shfl_sync(0xffffffffu, before, at);
  while (slice > 1) {                              // which request of the slice
    if (begin >= end) return;
    const int b = begin + lane;
    const long long pages_b = b < end ? heads * Request::load<PACKED>(p, b).total(p) : 0LL, upto = scan(pages_b);
    const unsigned hit = __ballot_sync(0xffffffffu, upto > rest);
    if (hit != 0) {
      const int in_slice = __ffs(hit) - 1;
      begin += in_slice;
      rest -= __shfl_sync(0xffffffffu, upto - pages_b, in_slice);
      break;
    }
    rest -= __shfl_sync(0xffffffffu, upto, 31);
    begin += 32;
  }
  const Request r = Request::load<PACKED>(p, begin);
  for (int j0 = 0; j0 < r.qtiles; j0 += 32) {
    const int j = j0 + lane;
    const long long pages = j < r.qtiles ? r.visible(p, j) : 0, sum_j = scan(pages * heads);
    const unsigned in = __ballot_sync(0xffffffffu, sum_j > rest);
    if (in == 0) {
      rest -= __shfl_sync(0xffffffffu, sum_j, 31);
      continue;
    }
    if (lane == __ffs(in) - 1) {
      const long long local = rest - (sum_j - pages * heads);
      start[0] = begin;
      start[1] = j;
      const int h = static_cast<int>(quotient(local, pages)), kvh = h / p.subs;
      start[2] = kvh;
      start[3] = h - kvh * p.subs;
      start[4] = static_cast<int>(local - h * pages);
      start[5] = static_cast<int>(min(per, total - first));
    }
    return;
  }
}

template <bool PACKED, bool RUNS>
__global__ void __launch_bounds__(QS_THREADS, PACKED && !RUNS ? 3 : 2)
fp4_nv_query_scores_kernel(const __grid_constant__ CUtensorMap q_map, const __grid_constant__ CUtensorMap k_map,
                           const QueryScoreParams p) {
  using M = QsMap<PACKED && !RUNS>;
  extern __shared__ unsigned char smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  unsigned char* gbase = smem_raw + (base - raw);
  const uint32_t bar0 = base + M::AUX;
  volatile int* misc = reinterpret_cast<volatile int*>(gbase + M::AUX + M::BAR_BYTES);   // tmem base, abort, start of the run
  auto bar = [&](int i) { return bar0 + 8u * i; };
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  Guard guard{misc + 1, p.status};

  if (threadIdx.x == 0) {
    misc[1] = 0;
    for (int i = 0; i < M::STAGES; ++i) {
      mbar_init(bar(M::K_FULL + i), 2);          // the TMA transaction of the codes + the producer warp's scale stores
      mbar_init(bar(M::K_EMPTY + i), 1);
    }
    for (int i = 0; i < M::Q_TILES; ++i) {
      mbar_init(bar(M::Q_FULL + i), 2);
      mbar_init(bar(M::Q_EMPTY + i), 1);
    }
    mbar_init(bar(M::BAR_ACC_FULL), 1);
    mbar_init(bar(M::BAR_ACC_EMPTY), 4);
    fence_mbar_init();
  }
  if (warp == 5) {
    tmem_alloc(smem_u32(const_cast<int*>(misc)), TM_COLS);
    tmem_relinquish();
  }
  ScoreWalk<PACKED, RUNS> place;
  if constexpr (RUNS) find_run<PACKED>(p, misc + 2, reinterpret_cast<volatile long long*>(misc + 16), warp, lane);
  else place = ScoreWalk<PACKED, RUNS>(p, nullptr);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = static_cast<uint32_t>(misc[0]);
  int total;
  if constexpr (RUNS) total = misc[7];
  else total = place.left;
  auto first_item = [&]() {
    if constexpr (RUNS) return ScoreWalk<PACKED, RUNS>(p, misc + 2);
    else return place;
  };

  if (total > 0) {
  if (warp == 4) {
    // ----------------------------------------------------------- codes (TMA); page ids 32 at a time
    ScoreWalk<PACKED, RUNS> walk = first_item();
    int items = 0, left = 0, pg = 0, ids = 0;     // items begun, pages left in the current one
    int pushed = 0;
    bool ok = true;
    for (int t = 0; t < total; ++t) {
      if (left == 0 || (pg & 31) == 0) {
        const int i = ((left == 0 ? walk.page : pg) & ~31) + lane;
        ids = i < walk.r.pages ? __ldg(p.kv_indices + walk.r.page_begin + i) : 0;
      }
      if (left == 0) {
        const int slot = items & (M::Q_TILES - 1);
        if (items >= 2) ok = mbar_wait_warp(bar(M::Q_EMPTY + slot), ((items >> 1) - 1) & 1, guard, 0x630 + slot);
        if (!ok) break;
        ++items;
        if (lane == 0) {
          mbar_expect_tx(bar(M::Q_FULL + slot), CODE_BYTES);
          // packed: box {64 bytes, 16 heads, 8 queries}, row = query * 16 + head; else box {64 bytes, 1 head, 128 queries}
          tma_load_3d(base + M::Q + slot * STAGE_BYTES, &q_map, 0, walk.head0(p), walk.r.q_begin + walk.j * 128,
                      bar(M::Q_FULL + slot));
        }
        left = walk.count();
        pg = walk.page;
      }
      const int s = t % M::STAGES, use = t / M::STAGES;
      if (use > 0) ok = mbar_wait_warp(bar(M::K_EMPTY + s), (use - 1) & 1, guard, 0x600 + s);
      if (!ok) break;
      const int ph = __shfl_sync(0xffffffffu, ids, pg & 31);
      if (lane == 0) {
        mbar_expect_tx(bar(M::K_FULL + s), CODE_BYTES);
        tma_load_2d(base + OFF_A + s * STAGE_BYTES, &k_map, 0, ((ph < 0 || ph >= p.total_pages ? 0 : ph) * p.hk + walk.kvh) * 128,
                    bar(M::K_FULL + s));
      }
      ++pushed;
      ++pg;
      if (--left == 0) walk.next(p);
    }
    if (!ok) {
      // let copies in flight land before the CTA gives up its shared memory
      for (int t = max(0, pushed - M::STAGES); t < pushed; ++t)
        mbar_wait_drain(bar(M::K_FULL + t % M::STAGES), (t / M::STAGES) & 1);
      for (int i = max(0, items - 2); i < items; ++i) mbar_wait_drain(bar(M::Q_FULL + (i & 1)), (i >> 1) & 1);
    }
  } else if (warp == 6) {
    // ----------------------------------------------------------- scales: staged QS_AHEAD pages ahead, then re-ordered
    // (asynchronous copies, not loads into registers: those need the loop unrolled over the pages in flight, and its
    // instructions alone, fetched for the first time, took 7000 cycles before the first page)
    ScoreWalk<PACKED, RUNS> ahead_walk = first_item(), walk = first_item();
    int ids = 0, ahead_left = 0, ahead_pg = 0;    // of the walk ahead: 32 page ids, pages left in its item, next page
    auto raw = [&](int t) { return M::RAW + (t % QS_AHEAD) * SF_BYTES + lane * 8; };
    auto fetch = [&](int t) {                     // rows lane, lane + 32, .. of page t; one group per page
      if (t < total) {
        const bool first = ahead_left == 0;
        if (first) {
          ahead_left = ahead_walk.count();
          ahead_pg = ahead_walk.page;
        }
        if (first || (ahead_pg & 31) == 0) {
          const int i = (ahead_pg & ~31) + lane;
          ids = i < ahead_walk.r.pages ? __ldg(p.kv_indices + ahead_walk.r.page_begin + i) : 0;
        }
        const int ph = __shfl_sync(0xffffffffu, ids, ahead_pg & 31);
        const long long row = ((ph < 0 || ph >= p.total_pages ? 0 : ph) * p.hk + ahead_walk.kvh) * 128LL;
        const uint8_t* src = p.ks + row * 8 + lane * 8;
#pragma unroll
        for (int i = 0; i < 4; ++i) cp_async8(base + raw(t) + i * 256, src + i * 256);
        ++ahead_pg;
        if (--ahead_left == 0) ahead_walk.next(p);
      }
      cp_async_commit();
    };
    bool ok = true;
#pragma unroll 1
    for (int t = 0; t < QS_AHEAD; ++t) fetch(t);
    int items = 0, left = 0;
#pragma unroll 1
    for (int t = 0; t < total; ++t) {
      if (left == 0) {
        const int slot = items & (M::Q_TILES - 1);
        const int h0 = walk.head0(p), q0 = walk.j * 128;
        const int rows_live = walk.r.q_rows - q0, heads_here = PACKED ? p.group - walk.sub * QS_PACK_HEADS : 1;
        ScaleRegs s;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int r = lane + 32 * i, q = PACKED ? r >> 4 : r, h = PACKED ? r & (QS_PACK_HEADS - 1) : 0;
          s.r[i] = make_uint2(0u, 0u);
          if (q < rows_live && h < heads_here)
            s.r[i] = __ldg(reinterpret_cast<const uint2*>(
                p.qs + ((static_cast<long long>(walk.r.q_begin) + q0 + q) * p.hq + h0 + h) * 8));
        }
        if (items >= 2) ok = mbar_wait_warp(bar(M::Q_EMPTY + slot), ((items >> 1) - 1) & 1, guard, 0x634 + slot);
        if (!ok) break;
        ++items;
        store_scale_chunks(gbase + M::Q + slot * STAGE_BYTES + CODE_BYTES, s, lane);
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(M::Q_FULL + slot));
        left = walk.count();
      }
      const int s = t % M::STAGES, use = t / M::STAGES;
      if (use > 0) ok = mbar_wait_warp(bar(M::K_EMPTY + s), (use - 1) & 1, guard, 0x608 + s);
      if (!ok) break;
      cp_async_wait<QS_AHEAD - 1>();              // this lane's rows of page t have landed
      ScaleRegs regs;
#pragma unroll
      for (int i = 0; i < 4; ++i) regs.r[i] = *reinterpret_cast<const uint2*>(gbase + raw(t) + i * 256);
      store_scale_chunks(gbase + OFF_A + s * STAGE_BYTES + CODE_BYTES, regs, lane);
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(M::K_FULL + s));
      fetch(t + QS_AHEAD);
      if (--left == 0) walk.next(p);
    }
    cp_async_wait<0>();
  } else if (warp == 5) {
    // ----------------------------------------------------------- MMA issue (elected lane of a converged warp)
    constexpr uint32_t IDESC = idesc_nvf4(128, 128);
    const bool lead = elect_one();
    ScoreWalk<PACKED, RUNS> walk = first_item();
    bool ok = true;
    int items = 0, left = 0;
    for (int t = 0; t < total; ++t) {
      const int slot = (items - (left ? 1 : 0)) & 1;       // of the current item's query tile
      const uint32_t q_tile = base + M::Q + slot * STAGE_BYTES;
      const uint32_t sfq = tmem + QS_SFQ + slot * 8;       // query scales: the A operand here
      if (left == 0) {
        ok = mbar_wait_warp(bar(M::Q_FULL + slot), (items >> 1) & 1, guard, 0x610 + slot);
        if (!ok) break;
        fence_async_smem();            // the producer's scale stores, for the copies below
        tc_fence_after();
        if (lead) {
          tmem_cp_scales(sfq, desc_scale_chunk(q_tile + CODE_BYTES));
          tmem_cp_scales(sfq + 4, desc_scale_chunk(q_tile + CODE_BYTES + 512));
        }
        ++items;
        left = walk.count();
        walk.next(p);
      }
      const int s = t % M::STAGES;
      ok = mbar_wait_warp(bar(M::K_FULL + s), (t / M::STAGES) & 1, guard, 0x612 + s);
      if (!ok) break;
      fence_async_smem();              // the producer's scale stores, for the copies below
      tc_fence_after();
      const uint64_t a0 = desc_sw64_kmajor(q_tile), b0 = desc_sw64_kmajor(base + OFF_A + s * STAGE_BYTES);
      const uint32_t sfk = tmem + QS_SFK + (t & 1) * 8;
      if (lead) {
        tmem_cp_scales(sfk, desc_scale_chunk(base + OFF_A + s * STAGE_BYTES + CODE_BYTES));
        tmem_cp_scales(sfk + 4, desc_scale_chunk(base + OFF_A + s * STAGE_BYTES + CODE_BYTES + 512));
      }
      if (t >= 1) {
        ok = mbar_wait_warp(bar(M::BAR_ACC_EMPTY), (t - 1) & 1, guard, 0x61a);
        if (!ok) break;
        tc_fence_after();
      }
      --left;
      if (lead) {
#pragma unroll
        for (int kh = 0; kh < 2; ++kh)
          mma_nvf4(tmem + TM_ACC, a0 + kh * 2, b0 + kh * 2, IDESC, sfq + kh * 4, sfk + kh * 4, kh);
        tc_commit(bar(M::BAR_ACC_FULL));
        tc_commit(bar(M::K_EMPTY + s));
        if (left == 0) tc_commit(bar(M::Q_EMPTY + slot));
      }
    }
    __syncwarp();
  } else {
    // ----------------------------------------------------------- epilogue: one lane = one query row
    // The fill kernel before this one on the stream has written its -inf (scoring begins under it: everything else here
    // only reads the inputs, and those were complete before the fill kernel began).
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint32_t lane_base = static_cast<uint32_t>(warp * 32) << 16;
    const int row = warp * 32 + lane;
    ScoreWalk<PACKED, RUNS> walk = first_item();
    bool ok = true;
    int t = 0;
    while (ok && walk.left > 0) {
      const int qi = PACKED ? row >> 4 : walk.j * 128 + row, head = PACKED ? row & (QS_PACK_HEADS - 1) : 0;
      const int h0 = walk.head0(p);
      const bool alive = qi < walk.r.q_rows && (!PACKED || walk.sub * QS_PACK_HEADS + head < p.group);
      float* dst = p.out + static_cast<long long>(h0 + head) * p.tiles_out * p.total_q + walk.r.q_begin + qi;
      // last visible key of this query (inclusive), relative to the request
      const long long last_key = p.causal ? min(static_cast<long long>(walk.r.k_len) - 1, static_cast<long long>(qi) + walk.r.offset)
                                          : static_cast<long long>(walk.r.k_len) - 1;
      const int stop = walk.page + walk.count();
      for (int pg = walk.page; pg < stop; ++pg, ++t) {
        const int ph = __ldg(p.kv_indices + walk.r.page_begin + pg);      // (the page stays -inf where it is out of range)
        bool w = mbar_wait(bar(M::BAR_ACC_FULL), t & 1, guard, 0x620);
        ok = __all_sync(0xffffffffu, w);
        if (!ok) break;
        tc_fence_after();
        const long long visible = last_key - static_cast<long long>(pg) * 128 + 1;     // visible keys of this page
        float m = -INFINITY;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          uint32_t v[4][16];
#pragma unroll
          for (int c = 0; c < 4; ++c) tmem_ld16(tmem + lane_base + TM_ACC + half * 64 + c * 16, v[c]);
          tc_wait_ld();
          if (half == 1) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(M::BAR_ACC_EMPTY));
          }
          if (visible >= (half + 1) * 64) {
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              float m5[5];
#pragma unroll
              for (int jj = 0; jj < 5; ++jj)
                m5[jj] = max3(__uint_as_float(v[c][3 * jj]), __uint_as_float(v[c][3 * jj + 1]), __uint_as_float(v[c][3 * jj + 2]));
              m = fmaxf(m, fmaxf(max3(m5[0], m5[1], m5[2]), max3(m5[3], m5[4], __uint_as_float(v[c][15]))));
            }
          } else if (visible > half * 64) {
            const int n = static_cast<int>(visible) - half * 64;           // 1 .. 63 visible columns of this half
#pragma unroll
            for (int c = 0; c < 4; ++c)
#pragma unroll
              for (int jj = 0; jj < 16; ++jj)
                if (c * 16 + jj < n) m = fmaxf(m, __uint_as_float(v[c][jj]));
          }
        }
        if (alive && ph >= 0 && ph < p.total_pages) dst[static_cast<long long>(pg) * p.total_q] = m;
      }
      walk.next(p);
    }
  }
  } else {
    // nothing to score: the grid must still not be complete before the fill kernel is
    asm volatile("griddepcontrol.wait;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 5) {
    tc_fence_after();
    tmem_dealloc(tmem, TM_COLS);
  }
}

// -inf everywhere; 16-byte stores from the first aligned element on
__global__ void __launch_bounds__(256) fill_neg_inf_kernel(float* out, long long n) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const long long head = min(n, static_cast<long long>((16u - (reinterpret_cast<uintptr_t>(out) & 15u)) & 15u) >> 2);
  const long long gid = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
  const long long n4 = (n - head) >> 2;
  float4* body = reinterpret_cast<float4*>(out + head);
  const float4 v = make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
  for (long long i = gid; i < n4; i += stride) body[i] = v;
  if (gid < head) out[gid] = -INFINITY;
  if (gid < n - head - 4 * n4) out[head + 4 * n4 + gid] = -INFINITY;
}

}  // namespace fnv

// aux (32 bytes, zeroed once by the owner of the workspace; every word accumulates over calls): [0] CTAs of the
// tensor-core kernels that ran (int), [1] tiles that took the exact path (int), [2] unused, [3] scores whose
// tensor-core value differed from the exact one by more than delta (int), [4] largest observed
// |tensor-core value - exact value| / delta (float); [5], [6] scratch of the page pre-filter (largest |key
// element| and largest squared key norm, rewritten by every call).
// Returns SB_OK when the tensor-core path ran, 1 when the problem is not eligible.
int launch_fp4_indexer_tc(const void* qp, const void* qs, const void* kp, const void* ks, void* aux, int32_t* ids,
                          int batch, int hidx, int hk, int len_q, int len_kv, int topk, cudaStream_t stream) {
  using namespace fnv;
  const int tiles = len_kv / 128, qt = len_q / 128;
  const int extra = topk / 4 > 16 ? topk / 4 : 16;
  int cand = topk + extra;
  if (cand > tiles) cand = tiles;
  if (cand > C_MAX || tiles > MAX_TILES) return 1;
  // Every candidate is re-scored exactly by one CTA per list, while the pruning scorer spreads
  // pages over the whole GPU: the pre-filter pays off only when candidates are a small share
  // of the pages.
  if (8 * cand > tiles) return 1;
  const long long q_rows = static_cast<long long>(batch) * len_q * hidx;
  const long long k_rows = static_cast<long long>(batch) * tiles * hk * 128;
  if (q_rows >= (1LL << 31) || k_rows >= (1LL << 31)) return 1;
  if (!aligned(qp, 16) || !aligned(kp, 16) || !aligned(qs, 8) || !aligned(ks, 8)) return 1;
  DeviceCtx* ctx = device_ctx();
  if (!ctx) return SB_ERR_CUDA;
  // key statistics for the error bound: one pass over codes and scales (microseconds next to the scoring)
  float* key_stats = static_cast<float*>(aux) + 5;
  if (cudaMemsetAsync(key_stats, 0, 8, stream) != cudaSuccess) return set_error(SB_ERR_CUDA, "memset failed");
  key_stats_kernel<<<static_cast<unsigned>((k_rows * 16 + 255) / 256), 256, 0, stream>>>(
      static_cast<const uint8_t*>(kp), static_cast<const uint8_t*>(ks), k_rows, key_stats);
  CUtensorMap qm, km;
  int rc = make_maps(&qm, &km, qp, kp, batch, hidx, len_q, k_rows);
  if (rc) return rc;
  Params p{};
  p.key_stats = key_stats;
  p.g = Geometry{static_cast<const uint8_t*>(qp), static_cast<const uint8_t*>(qs), static_cast<const uint8_t*>(kp),
                 static_cast<const uint8_t*>(ks), batch, hidx, hk, len_q, tiles};
  p.stats = static_cast<int*>(aux);
  p.fallbacks = reinterpret_cast<int*>(aux) + 1;
  p.violations = reinterpret_cast<int*>(aux) + 3;
  p.ids = ids;
  p.status = ctx->status;
  p.topk = topk; p.cand = cand;
  // shared memory beside the layout's: scores, barriers and scratch, slack of the alignment
  const size_t rest = ((static_cast<size_t>(tiles) * 4 + 15) & ~static_cast<size_t>(15)) + 320 + 1024;
  // Two CTAs to an SM with 1 KiB of the system's each: with six stages up to 10672 pages, with four up to 16304. 1024 lists of
  // 12000 pages, ms: six stages and one CTA 30.8, four and two 18.8; of 10000 pages six and two 15.6.
  const bool six = 2 * (Layout<A_STAGES>::SCORES + rest + 1024) <= 228 * 1024;
  auto kernel = six ? fp4_nv_select_kernel<A_STAGES> : fp4_nv_select_kernel<4>;
  const int configured = six ? 1 << 8 : 1 << 21;
  if (!(ctx->tc_attr & configured)) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    if (e != cudaSuccess) return set_error(SB_ERR_CUDA, cudaGetErrorString(e));
    ctx->tc_attr |= configured;
  }
  kernel<<<batch * hidx * qt, NUM_THREADS, (six ? Layout<A_STAGES>::SCORES : Layout<4>::SCORES) + rest, stream>>>(qm, km, p);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? SB_OK : set_error(SB_ERR_CUDA, cudaGetErrorString(e));
}

// Exact tile scores [B, Hidx, Qt, tiles] through fp4_nv_prune_kernel. Returns SB_OK, or 1 when the
// problem is not eligible (the caller then runs the exact mma.sync scorer). aux as above.
int launch_fp4_scores_prune(const void* qp, const void* qs, const void* kp, const void* ks, void* aux, float* tile_scores,
                            int batch, int hidx, int hk, int len_q, int len_kv, cudaStream_t stream) {
  using namespace fnv;
  const int tiles = len_kv / 128, qt = len_q / 128;
  const long long q_rows = static_cast<long long>(batch) * len_q * hidx;
  const long long k_rows = static_cast<long long>(batch) * tiles * hk * 128;
  const long long lists = static_cast<long long>(batch) * hidx * qt;
  if (q_rows >= (1LL << 31) || k_rows >= (1LL << 31) || lists * tiles >= (1LL << 31)) return 1;
  if (!aligned(qp, 16) || !aligned(kp, 16) || !aligned(qs, 8) || !aligned(ks, 16)) return 1;
  DeviceCtx* ctx = device_ctx();
  if (!ctx) return SB_ERR_CUDA;
  CUtensorMap qm, km;
  int rc = make_maps(&qm, &km, qp, kp, batch, hidx, len_q, k_rows);
  if (rc) return rc;
  PruneParams p{};
  p.g = Geometry{static_cast<const uint8_t*>(qp), static_cast<const uint8_t*>(qs), static_cast<const uint8_t*>(kp),
                 static_cast<const uint8_t*>(ks), batch, hidx, hk, len_q, tiles};
  p.stats = static_cast<int*>(aux);
  p.violations = reinterpret_cast<int*>(aux) + 3;
  p.tile_scores = tile_scores;
  p.status = ctx->status;
  // Two CTAs fit an SM: while one waits for its accumulator the other uses the tensor pipe. As many
  // CTAs as fit at once when the lists are few; a CTA keeps its query tile and takes a run of pages.
  long long chunks = (2LL * ctx->sm_count) / lists;
  if (chunks > tiles) chunks = tiles;
  if (chunks < (tiles + PR_PAGES_MAX - 1) / PR_PAGES_MAX) chunks = (tiles + PR_PAGES_MAX - 1) / PR_PAGES_MAX;
  p.pages_per_cta = static_cast<int>((tiles + chunks - 1) / chunks);
  p.chunks = (tiles + p.pages_per_cta - 1) / p.pages_per_cta;
  if (lists * p.chunks >= (1LL << 31)) return 1;
  if (!(ctx->tc_attr & (1 << 11))) {
    cudaError_t e = cudaFuncSetAttribute(fp4_nv_prune_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(fp4_nv_prune_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    if (e != cudaSuccess) return set_error(SB_ERR_CUDA, cudaGetErrorString(e));
    ctx->tc_attr |= (1 << 11);
  }
  const size_t smem = PR_OFF_RES + static_cast<size_t>(p.pages_per_cta) * 8 + 1024;
  fp4_nv_prune_kernel<<<static_cast<unsigned>(lists * p.chunks), NUM_THREADS, smem, stream>>>(qm, km, p);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? SB_OK : set_error(SB_ERR_CUDA, cudaGetErrorString(e));
}

// Per-query page scores of a ragged batch on the NVFP4 tensor cores. Returns SB_OK, or 1 when the inputs do not
// meet the alignment the TMA path needs (the caller then runs the exact scorer).
int launch_fp4_scores_varlen_nv(const void* qp, const void* qs, const void* kp, const void* ks, const int32_t* cu_q,
                                const int32_t* cu_k, const int32_t* cu_pages, const int32_t* kv_indices,
                                const int32_t* qo_offset, float* out, int batch, int hq, int hk, int total_q,
                                int total_pages, int max_seqlen_q, int max_seqlen_k, int causal, cudaStream_t stream) {
  using namespace fnv;
  if (!aligned(qp, 16) || !aligned(kp, 16) || !aligned(qs, 8) || !aligned(ks, 8)) return 1;
  const long long k_rows = static_cast<long long>(total_pages) * hk * 128;
  if (k_rows >= (1LL << 31) || static_cast<long long>(total_q) >= (1LL << 31)) return 1;
  DeviceCtx* ctx = device_ctx();
  if (!ctx) return SB_ERR_CUDA;
  QueryScoreParams p{};
  p.qp = static_cast<const uint8_t*>(qp); p.qs = static_cast<const uint8_t*>(qs);
  p.kp = static_cast<const uint8_t*>(kp); p.ks = static_cast<const uint8_t*>(ks);
  p.cu_q = cu_q; p.cu_k = cu_k; p.cu_pages = cu_pages; p.kv_indices = kv_indices; p.qo_offset = qo_offset;
  p.out = out;
  p.status = ctx->status;
  p.batch = batch; p.hq = hq; p.hk = hk; p.total_q = total_q; p.total_pages = total_pages;
  p.qt_max = (max_seqlen_q + 127) / 128;
  p.tiles_out = (max_seqlen_k + 127) / 128;
  p.causal = causal;
  const bool packed = max_seqlen_q <= QS_PACK_Q && hq / hk > 1;
  p.group = hq / hk;
  p.subs = packed ? (p.group + QS_PACK_HEADS - 1) / QS_PACK_HEADS : p.group;
  const long long items = packed ? static_cast<long long>(batch) * hk * p.subs
                                 : static_cast<long long>(batch) * p.qt_max * hq;
  if (items > 0x7fffffffLL) return set_error(SB_ERR_INVALID, "too many (request, query tile, head) items");
  const long long n = static_cast<long long>(hq) * p.tiles_out * total_q;
  const long long fill_blocks = std::min<long long>((n / 4 + 255) / 256 + 1, 8LL * ctx->sm_count);
  fill_neg_inf_kernel<<<static_cast<unsigned>(fill_blocks), 256, 0, stream>>>(out, n);
  const cudaError_t filled = cudaGetLastError();
  if (filled != cudaSuccess) return set_error(SB_ERR_CUDA, cudaGetErrorString(filled));
  if (items == 0 || p.tiles_out == 0) return SB_OK;
  // two CTAs per SM, at least two pages each
  const long long most = (items * p.tiles_out + 1) / 2;
  long long ctas = std::min<long long>(2LL * ctx->sm_count, most);
  // Up to four CTAs to an SM, the longest lengths taken for all, each gets a share of one item's pages instead of a run: the
  // call has no last round to level, and a run's place costs 1.5 to 3 us to find. In a graph, us, runs -> shares (and before
  // there were runs): one token of one request 6.9 -> 5.1 (5.5), of 64 requests of 100 to 400 keys 8.9 -> 5.3 (5.8), of 256 11.1 ->
  // 9.0 (9.4), prefill of eight requests of up to 300 8.5 -> 6.3 (7.2). Beyond, runs are faster (64 requests of 1000 to 4000
  // keys 11.1, shares 13.2) unless a request is one item of a few pages, where a run changes its item every other page: 600
  // requests of 500 to 900 keys 18.9 -> 17.5 (16.2), 1024 of 100 to 400 20.1 -> 16.6 (16.0), 2048 32.6 -> 28.5 (26.3).
  int share = 64;
  while (share > 2 && items * ((p.tiles_out + share - 1) / share) < 4LL * ctx->sm_count) share >>= 1;
  const long long shared = items * ((p.tiles_out + share - 1) / share);
  const bool single = packed && items == batch;      // one item to a request
  const bool runs = shared > (single && p.tiles_out <= 8 ? 16 : 4) * ctx->sm_count;
  if (!runs) {
    p.share = share;
    p.shares = (p.tiles_out + share - 1) / share;
    ctas = shared;
  }
  const dim3 grid(static_cast<unsigned>(ctas));
  CUtensorMap qm, km;
  {
    const cuuint64_t dims[3] = {64, static_cast<cuuint64_t>(hq), static_cast<cuuint64_t>(total_q)};
    const cuuint64_t strides[2] = {64, static_cast<cuuint64_t>(hq) * 64};
    const cuuint32_t box_tile[3] = {64, 1, 128}, box_packed[3] = {64, QS_PACK_HEADS, QS_PACK_Q};
    const cuuint32_t steps[3] = {1, 1, 1};
    if (encode_tiled(&qm, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(qp), dims, strides,
                     packed ? box_packed : box_tile, steps, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B))
      return set_error(SB_ERR_CUDA, "cuTensorMapEncodeTiled failed for the query codes");
  }
  {
    const cuuint64_t dims[2] = {64, static_cast<cuuint64_t>(k_rows)};
    const cuuint64_t strides[1] = {64};
    const cuuint32_t box[2] = {64, 128};
    const cuuint32_t steps[2] = {1, 1};
    if (encode_tiled(&km, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(kp), dims, strides, box, steps,
                     CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B))
      return set_error(SB_ERR_CUDA, "cuTensorMapEncodeTiled failed for the key codes");
  }
  if (!(ctx->tc_attr & (1 << 12))) {
    for (auto kernel : {fp4_nv_query_scores_kernel<false, false>, fp4_nv_query_scores_kernel<false, true>,
                        fp4_nv_query_scores_kernel<true, false>, fp4_nv_query_scores_kernel<true, true>}) {
      cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, QsMap<false>::SMEM);
      if (e != cudaSuccess) return set_error(SB_ERR_CUDA, cudaGetErrorString(e));
    }
    ctx->tc_attr |= (1 << 12);
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(QS_THREADS);
  cfg.dynamicSmemBytes = packed && !runs ? QsMap<true>::SMEM : QsMap<false>::SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  auto kernel = packed ? (runs ? fp4_nv_query_scores_kernel<true, true> : fp4_nv_query_scores_kernel<true, false>)
                       : (runs ? fp4_nv_query_scores_kernel<false, true> : fp4_nv_query_scores_kernel<false, false>);
  cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, qm, km, p);
  return e == cudaSuccess ? SB_OK : set_error(SB_ERR_CUDA, cudaGetErrorString(e));
}

}  // namespace sb
