// Persistent bf16 GEMM for sm_100a: TMA -> 128B-swizzled shared memory -> tcgen05.mma with
// fp32 accumulators in TMEM -> tcgen05.ld epilogue with fused bias / GELU / residual / fp32
// accumulate.  C[M,N] = sum_k A(m,k) * B(n,k).
//
// Operand layouts (runtime): each operand is either K-major (stored [rows, K], K contiguous)
// or MN-major (stored [K, rows], rows contiguous), so forward (X.W^T), dgrad (dY.W) and wgrad
// (dY^T.X) all run on the same kernel without any transposed copies.
//
// Warp roles (192 threads): warp 0 = TMA producer, warp 1 = MMA issuer (+TMEM owner),
// warps 2..5 = epilogue (TMEM lane quarter = warp_id % 4).  The accumulator is double-buffered
// in TMEM (2 x BN columns) so the epilogue of tile i overlaps the main loop of tile i+1.
//
// kCtaGroup == 2 pairs two CTAs of a cluster on one 256 x BN tile (tcgen05 cta_group::2): each
// CTA loads its own 128 rows of A and its own half of B; the leader CTA issues the MMAs.
#include "launch.cuh"
#include "tc05.cuh"
#include "peer.cuh"

#include <atomic>
#include <string.h>

extern "C" void pb_count_launch(int n);

namespace pb {

struct GemmParams {
  int M, N, K;
  void* C;
  long long ldc;
  const __nv_bfloat16* bias;      // [N] or null
  const __nv_bfloat16* residual;  // [M, ldr] or null
  long long ldr;
  __nv_bfloat16* aux;  // optional pre-activation output [M, ldc] (bf16), written when act != 0
  int act;             // 0 none, 1 gelu(tanh)
  int out_fp32;        // C is float (else bf16)
  int accumulate;      // C += result (fp32 output only)
  int a_mn, b_mn;      // operand majors
  int* err;
  int num_m_tiles, num_n_tiles, num_k_blocks;
  int group_m;
  // ---- fused tensor-parallel modes (0 = plain GEMM)
  //   1: all-gather -> GEMM.  A is the row-wise concatenation of `world` shards of `chunk_rows` rows; this rank's
  //      shard is read in place (tmA), the others from a local gathered copy (tmA2) that copy CTAs of this same
  //      grid fill from the peers' shards while GEMM CTAs already work on the rows that have arrived.
  //   2: GEMM -> reduce-scatter.  Output rows are owned chunk-wise by the ranks; tiles of a foreign chunk are stored
  //      straight into the owner's staging slot (P2P stores), the own chunk into `C`; when everything has been
  //      sent the grid reduces own partial + received partials into `rs_out`.
  int fused;
  int rank, world, chunk_rows;
  long long lda_elems;  // row pitch (elements) of the shards and of the gathered buffer
  int m_rot;         // rotation of the M-tile order (tiles): own chunk first (mode 1) / last (mode 2)
  int gemm_ctas;     // CTAs running the GEMM roles; the rest of the grid copies (mode 1)
  int epoch;
  int* tile_flags;   // local [num_m_tiles]: rows of that M tile have landed in the gathered buffer (mode 1)
  int* counters;     // local scratch, zeroed before launch: [0] grid barrier, [1 + peer] copy CTAs done with peer
  int* flags[8];     // every rank's flag block (peer mapped): [0,W) ready, [W,2W) done / sent
  const __nv_bfloat16* peer_src[8];  // mode 1: every rank's shard [chunk_rows, K] (row pitch lda)
  __nv_bfloat16* gathered;           // mode 1: local [world * chunk_rows, K] (row pitch lda)
  __nv_bfloat16* rs_staging[8];      // mode 2: every rank's staging [world, chunk_rows, N]
  __nv_bfloat16* rs_out;             // mode 2: local result [chunk_rows, N] (row pitch ldc)
  const __nv_bfloat16* rs_residual;  // mode 2: optional [chunk_rows, N] added in the final reduce
  // ---- grouped modes (0 = plain GEMM): the rows of one operand dimension belong to `n_groups` groups (the
  // experts of a mixture-of-experts layer) whose sizes are only known on the device.  Group g occupies rows
  // [group_start[g], group_start[g] + group_rows[g]); every group_start is a multiple of 256.
  //   1: the M rows of A and C are grouped; each group multiplies its own B: a K-major B is the row-wise stack of
  //      the groups' [b_group_stride, K] matrices, an MN-major B the stack of their [b_group_stride (= K), N]
  //      matrices.  Only tiles that hold rows of a group run; output rows of such a tile beyond the group's end
  //      are written as zeros, so that a later contraction over the rows can run to the next multiple of 64.
  //   2: the contraction dimension is grouped (both operands MN-major, stored [rows, M] and [rows, N]); group g
  //      writes (or accumulates into) its own C block at C + g * c_group_stride elements.  The contraction of a
  //      group runs over whole 64-row blocks: rows between the group's end and the next multiple of 64 must be
  //      zero in one operand and finite in the other.
  int grouped;
  int n_groups;
  const int* group_rows;
  const int* group_start;
  int b_group_stride;
  long long c_group_stride;
  // ---- split contraction (plain GEMMs): tiles from `dp_tiles` on are cut into `splits` ranges of k-blocks, one work
  // item each.  Every item leaves its fp32 partial tile in `split_ws`; the one that arrives last at the tile's counter
  // (per 32 rows) adds the partials in range order, so the result does not depend on which one that was, and runs
  // the epilogue.  Nobody waits.  A counter holds the launch's tag | arrivals (low 4 bits); under any other tag it counts
  // as zero, so that what a launch that gave up left behind means nothing to the next one.
  int dp_tiles, splits;
  float* split_ws;
  unsigned long long* split_counters;
  unsigned long long split_tag;
};

constexpr int MAX_GROUPS = 8;

// Group table in shared memory, built by every CTA from the device-side sizes.
struct GroupTable {
  int prefix[MAX_GROUPS + 1];  // mode 1: M tiles before group g
  int start[MAX_GROUPS];
  int rows[MAX_GROUPS];
};

constexpr int BK = 64;
constexpr int BM_CTA = 128;

__device__ __forceinline__ float4 add4(const float4& a, const float4& b) {
  return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
}
__device__ __forceinline__ float4 bf16x4_to_float4(uint2 u) {
  const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
  const float2 hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
  return make_float4(lo.x, lo.y, hi.x, hi.y);
}
__device__ __forceinline__ uint2 float4_to_bf16x4(const float4& v) {
  const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
  return make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
}
__device__ __forceinline__ void prefetch_l2(const void* p, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}
template <bool V>
struct Flag {
  static constexpr bool value = V;
};

__device__ __forceinline__ float gelu_tanh(float x) {
  const float k0 = 0.7978845608028654f, k1 = 0.044715f;
  float u = k0 * (x + k1 * x * x * x);
  float t;
  asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(u));
  return 0.5f * x * (1.f + t);
}

__device__ __forceinline__ void tile_coords(int tile, const GemmParams& p, int num_m_tiles, int& tm, int& tn) {
  const int per_group = p.group_m * p.num_n_tiles;
  const int g = tile / per_group;
  const int first_m = g * p.group_m;
  const int gsz = min(p.group_m, num_m_tiles - first_m);
  const int r = tile - g * per_group;
  tm = first_m + r % gsz;
  tn = r / gsz;
  if (p.fused == 1) {
    tm += p.m_rot;
    if (tm >= p.num_m_tiles) tm -= p.num_m_tiles;
  } else if (p.fused == 2) {
    // reduce-scatter: walk the owners round-robin, one tile group at a time, starting with the next rank, so the
    // stores to each peer are spread over the whole kernel instead of bursting at its start
    const int tiles_per_chunk = p.num_m_tiles / p.world;
    if (tiles_per_chunk % p.group_m == 0) {
      const int grp = tm / p.group_m, within = tm % p.group_m;
      const int chunk = (p.rank + 1 + grp) % p.world;
      tm = chunk * tiles_per_chunk + (grp / p.world) * p.group_m + within;
    } else {
      tm += p.m_rot;
      if (tm >= p.num_m_tiles) tm -= p.num_m_tiles;
    }
  }
}

template <int kCtaGroup, int BN, int kStages>
__global__ void __launch_bounds__(192, 1)
gemm_bf16_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                 const __grid_constant__ CUtensorMap tmA2, GemmParams p) {
  constexpr int A_BYTES = BM_CTA * BK * 2;
  constexpr int BN_CTA = BN / kCtaGroup;  // B rows loaded by this CTA
  constexpr int B_BYTES = BN_CTA * BK * 2;
  constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  constexpr int TMEM_COLS = 2 * BN >= 512 ? 512 : (2 * BN <= 32 ? 32 : 2 * BN);

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sA = smem;
  uint8_t* sB = smem + kStages * A_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kStages * STAGE_BYTES);
  uint64_t* full = bars;
  uint64_t* empty = bars + kStages;
  uint64_t* tfull = bars + 2 * kStages;
  uint64_t* tempty = bars + 2 * kStages + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kStages + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  GroupTable* gt = reinterpret_cast<GroupTable*>(smem + kStages * STAGE_BYTES + 152);  // 100 bytes of the 256
  static_assert((2 * kStages + 4) * 8 + 8 <= 152, "barriers overlap the group table");
  uint8_t* sEpi = smem + kStages * STAGE_BYTES + 256;  // 4 epilogue warps x 32 rows x (128 + 16) bytes

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t cta_rank = (kCtaGroup == 2) ? cluster_ctarank() : 0;
  const bool leader = (cta_rank == 0);

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tfull[a], 1);
      mbar_init(&tempty[a], 4 * kCtaGroup);
    }
    *abort_flag = 0;
    mbar_fence_init();
    if (p.grouped) {
      int acc_tiles = 0;
      for (int g = 0; g < MAX_GROUPS; ++g) {
        const int rows = g < p.n_groups ? p.group_rows[g] : 0;
        gt->prefix[g] = acc_tiles;
        gt->start[g] = g < p.n_groups ? p.group_start[g] : 0;
        gt->rows[g] = rows;
        acc_tiles += (rows + BM_CTA * kCtaGroup - 1) / (BM_CTA * kCtaGroup);
      }
      gt->prefix[MAX_GROUPS] = acc_tiles;
    }
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
  }
  if (warp == 1) tmem_alloc<kCtaGroup>(tmem_slot, TMEM_COLS);
  tc_fence_before_sync();
  __syncthreads();
  if constexpr (kCtaGroup == 2) cluster_sync_all();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;

  const int unit = blockIdx.x / kCtaGroup;
  const int num_units = (p.fused == 1 ? p.gemm_ctas : (int)gridDim.x) / kCtaGroup;
  const bool copy_cta = (p.fused == 1) && ((int)blockIdx.x >= p.gemm_ctas);
  // grouped mode 1 only knows its M tiles now; mode 2 runs the full [M, N] tile grid once per group
  const int num_m_tiles = (p.grouped == 1) ? gt->prefix[MAX_GROUPS] : p.num_m_tiles;
  const int tiles_per_group = num_m_tiles * p.num_n_tiles;
  // work items: whole tiles, then the ranges of the split ones
  const int num_tiles = (p.grouped == 2)   ? tiles_per_group * p.n_groups
                        : (p.splits > 1) ? p.dp_tiles + (tiles_per_group - p.dp_tiles) * p.splits
                                         : tiles_per_group;
  constexpr int TILE_M_ALL = BM_CTA * kCtaGroup;
  // Where a tile lives.  Every role calls this with the same arguments, so all agree on the rows, the group and
  // the contraction range (kb0 <= kb < kb1; an empty range means the tile is skipped by everybody).
  auto locate = [&](int tile, int& tn, int& row0, int& m_limit, int& grp, int& kb0, int& kb1) {
    int tm;
    grp = 0;
    kb0 = 0;
    kb1 = p.num_k_blocks;
    if (p.splits > 1 && tile >= p.dp_tiles) {
      const int item = tile - p.dp_tiles, range = item % p.splits;
      tile = p.dp_tiles + item / p.splits;
      kb0 = (int)((long long)p.num_k_blocks * range / p.splits);
      kb1 = (int)((long long)p.num_k_blocks * (range + 1) / p.splits);
    }
    if (p.grouped == 2) {
      grp = tile / tiles_per_group;
      tile -= grp * tiles_per_group;
      kb0 = gt->start[grp] / BK;
      kb1 = (gt->start[grp] + gt->rows[grp] + BK - 1) / BK;
      if (gt->rows[grp] == 0) kb1 = kb0;
    }
    tile_coords(tile, p, num_m_tiles, tm, tn);
    row0 = tm * TILE_M_ALL;
    m_limit = p.M;
    if (p.grouped == 1) {
      while (grp + 1 < MAX_GROUPS && tm >= gt->prefix[grp + 1]) ++grp;
      row0 = gt->start[grp] + (tm - gt->prefix[grp]) * TILE_M_ALL;
      m_limit = min(p.M, gt->start[grp] + gt->rows[grp]);
    }
  };

  if (copy_cta) {
    // ------------------------------------------------------------ all-gather copy role (mode 1)
    using namespace pbp;
    const int n_copy = (int)gridDim.x - p.gemm_ctas;
    const int me = (int)blockIdx.x - p.gemm_ctas;
    const int W = p.world;
    constexpr int TILE_M = BM_CTA * kCtaGroup;
    const int blocks_per_chunk = (p.chunk_rows + TILE_M - 1) / TILE_M;
    __shared__ int s_ok;
    uint32_t copy_issue = 0, copy_done = 0;
    if (me == 0 && threadIdx.x < W && (int)threadIdx.x != p.rank)
      st_release_sys(p.flags[threadIdx.x] + p.rank, p.epoch);  // my shard is complete (stream order)
    for (int q = 1; q < W; ++q) {
      const int peer = (p.rank + q) % W;
      if (threadIdx.x == 0) s_ok = wait_flag_sys(p.flags[p.rank] + peer, p.epoch, p.err, ERR_PEER_TIMEOUT) ? 1 : 0;
      __syncthreads();
      if (!s_ok) break;
      const __nv_bfloat16* src = p.peer_src[peer];
      // One thread streams the rows through a ring of shared-memory slots with bulk copies (peer -> smem -> local):
      // up to kStages pieces of 32 KiB are in flight per copy CTA, enough to cover the NVLink round trip.
      if (threadIdx.x == 0) {
        constexpr uint32_t PIECE = 32768;
        bool good = true;
        for (int blk = me; blk < blocks_per_chunk && good; blk += n_copy) {
          const int r0 = blk * TILE_M;
          const int rows = min(TILE_M, p.chunk_rows - r0);
          const long long bytes_total = (long long)rows * p.lda_elems * 2;
          const char* gsrc = reinterpret_cast<const char*>(src + (long long)r0 * p.lda_elems);
          char* gdst = reinterpret_cast<char*>(p.gathered + ((long long)peer * p.chunk_rows + r0) * p.lda_elems);
          const int n_pieces = (int)((bytes_total + PIECE - 1) / PIECE);
          int issued = 0, stored = 0;
          while (stored < n_pieces) {
            while (issued < n_pieces && issued - stored < kStages) {
              const uint32_t slot = copy_issue % kStages;
              const long long off = (long long)issued * PIECE;
              const uint32_t nb = (uint32_t)min((long long)PIECE, bytes_total - off);
              mbar_expect_tx(&full[slot], nb);
              bulk_load(smem + slot * PIECE, gsrc + off, nb, &full[slot]);
              ++copy_issue;
              ++issued;
            }
            const uint32_t slot = copy_done % kStages;
            if (!mbar_wait(&full[slot], (copy_done / kStages) & 1, abort_flag)) {
              good = false;
              atomicExch(p.err, ERR_WAIT_TIMEOUT);
              break;
            }
            const long long off = (long long)stored * PIECE;
            const uint32_t nb = (uint32_t)min((long long)PIECE, bytes_total - off);
            bulk_store(gdst + off, smem + slot * PIECE, nb);
            tma_store_commit();
            tma_store_wait_read<0>();  // the slot may be refilled once the store has read it
            ++copy_done;
            ++stored;
          }
          if (!good) break;
          tma_store_wait<0>();  // rows are in local memory
          __threadfence();
          st_release_gpu(p.tile_flags + (peer * p.chunk_rows + r0) / TILE_M, p.epoch);
        }
      }
      __syncthreads();
      if (threadIdx.x == 0) {
        // the last copy CTA to finish with this peer tells it that its shard may be overwritten
        __threadfence();
        if (atomicAdd(p.counters + 1 + peer, 1) == n_copy - 1) st_release_sys(p.flags[peer] + W + p.rank, p.epoch);
      }
    }
    if (me == 0) {
      // do not return before every peer has finished reading my shard
      bool ok = true;
      if (threadIdx.x < W && (int)threadIdx.x != p.rank)
        ok = wait_flag_sys(p.flags[p.rank] + W + threadIdx.x, p.epoch, p.err, ERR_PEER_TIMEOUT);
      __syncthreads_and(ok);
    }
  } else if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (whole warp, one elected lane issues)
    {
      uint32_t stage = 0, phase = 0;
      bool ok = true;
      const uint32_t full0_remote = (kCtaGroup == 2) ? mapa_u32(smem_u32(&full[0]), 0) : 0;
      for (int tile = unit; tile < num_tiles && ok; tile += num_units) {
        int tn, row0, m_limit, grp, kb0, kb1;
        locate(tile, tn, row0, m_limit, grp, kb0, kb1);
        const int tm = row0 / TILE_M_ALL;  // fused modes only (never grouped)
        int m0 = row0 + cta_rank * BM_CTA;
        const int n0 = tn * BN + cta_rank * BN_CTA;
        // a grouped-M GEMM reads group `grp`'s own B: a row offset for a K-major B, a k offset for an MN-major one
        const int bn_off = (p.grouped == 1 && !p.b_mn) ? grp * p.b_group_stride : 0;
        const int bk_off = (p.grouped == 1 && p.b_mn) ? grp * p.b_group_stride : 0;
        const CUtensorMap* tma_a = &tmA;
        if (p.fused == 1) {
          const int chunk = (tm * (BM_CTA * kCtaGroup)) / p.chunk_rows;
          if (chunk == p.rank) {
            m0 -= chunk * p.chunk_rows;  // own shard, read in place
          } else {
            tma_a = &tmA2;
            // the verdict is the warp's: lanes that went different ways would wait for one another below
            ok = __all_sync(0xffffffffu, pbp::wait_flag_gpu(p.tile_flags + tm, p.epoch, p.err, ERR_PEER_TIMEOUT));
            if (!ok) break;
            asm volatile("fence.proxy.async.global;" ::: "memory");  // copied rows -> visible to the TMA engine
          }
        }
        for (int kb = kb0; kb < kb1; ++kb) {
          ok = __all_sync(0xffffffffu, mbar_wait(&empty[stage], phase ^ 1, abort_flag));
          if (!ok) break;
          uint8_t* a_dst = sA + stage * A_BYTES;
          uint8_t* b_dst = sB + stage * B_BYTES;
          const int k0 = kb * BK;
          if (elect_one()) {
            if constexpr (kCtaGroup == 1) {
              mbar_expect_tx(&full[stage], STAGE_BYTES);
              if (!p.a_mn) {
                tma_load_2d(a_dst, tma_a, &full[stage], k0, m0);
              } else {
#pragma unroll
                for (int i = 0; i < BM_CTA / 64; ++i) tma_load_2d(a_dst + i * 8192, tma_a, &full[stage], m0 + i * 64, k0);
              }
              if (!p.b_mn) {
                tma_load_2d(b_dst, &tmB, &full[stage], k0, n0 + bn_off);
              } else {
#pragma unroll
                for (int i = 0; i < BN_CTA / 64; ++i)
                  tma_load_2d(b_dst + i * 8192, &tmB, &full[stage], n0 + i * 64, k0 + bk_off);
              }
            } else {
              if (leader) mbar_expect_tx(&full[stage], STAGE_BYTES * 2);
              const uint32_t bar = full0_remote + stage * 8;
              if (!p.a_mn) {
                tma_load_2d_pair(a_dst, tma_a, bar, k0, m0);
              } else {
#pragma unroll
                for (int i = 0; i < BM_CTA / 64; ++i) tma_load_2d_pair(a_dst + i * 8192, tma_a, bar, m0 + i * 64, k0);
              }
              if (!p.b_mn) {
                tma_load_2d_pair(b_dst, &tmB, bar, k0, n0 + bn_off);
              } else {
#pragma unroll
                for (int i = 0; i < BN_CTA / 64; ++i)
                  tma_load_2d_pair(b_dst + i * 8192, &tmB, bar, n0 + i * 64, k0 + bk_off);
              }
            }
          }
          __syncwarp();
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
      if (!ok && lane == 0) atomicExch(p.err, ERR_WAIT_TIMEOUT);
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    // The whole warp walks the loop (waits included) so that control flow stays warp-uniform; one elected lane issues.
    // Under `lane == 0` issuing set the pace: a 64-deep k-block took 512 to 570 cycles with every tile shape, although
    // its four MMAs run in 256 (128 x 128 tiles).  Elected in both issuing warps, of this kernel on a B200:
    // 4096 x 4096 x 8192 weight gradient 235 -> 224 us, 8192 x 4096 x 4096 207 -> 201 us, 77 x 4096 x 4096 26.4 -> 23.7 us;
    // a pair's k-block takes 518 cycles from the first operands to the accumulator of an 8192 x 4096 x 4096 tile, where its
    // 128 x 256 per CTA need 512 at the tensor rate.
    if (leader) {
      const uint32_t idesc = make_idesc_bf16(BM_CTA * kCtaGroup, BN, p.a_mn, p.b_mn);
      // K-major: 16 k-elements = 32 B inside the swizzled row; MN-major: 16 k-rows of 128 B
      const uint32_t a_kstep = p.a_mn ? 2048 : 32;
      const uint32_t b_kstep = p.b_mn ? 2048 : 32;
      const uint32_t a_lbo = p.a_mn ? 8192 : 16;
      const uint32_t b_lbo = p.b_mn ? 8192 : 16;
      uint32_t stage = 0, phase = 0, acc = 0, acc_phase = 0;
      bool ok = true;
      for (int tile = unit; tile < num_tiles && ok; tile += num_units) {
        int tn_, row0_, ml_, grp_, kb0, kb1;
        locate(tile, tn_, row0_, ml_, grp_, kb0, kb1);
        if (kb1 <= kb0) continue;  // empty group: no accumulator is produced, the epilogue skips the tile too
        ok = __all_sync(0xffffffffu, mbar_wait(&tempty[acc], acc_phase ^ 1, abort_flag));
        if (!ok) break;
        tc_fence_after_sync();
        const uint32_t d_tmem = tmem_base + acc * BN;
        for (int kb = kb0; kb < kb1; ++kb) {
          ok = __all_sync(0xffffffffu, mbar_wait(&full[stage], phase, abort_flag));
          if (!ok) break;
          tc_fence_after_sync();
          const uint64_t da = make_smem_desc(smem_u32(sA + stage * A_BYTES), a_lbo, 1024);
          const uint64_t db = make_smem_desc(smem_u32(sB + stage * B_BYTES), b_lbo, 1024);
          if (elect_one()) {
            // descriptors of the steps differ only in the start address (low 14 bits, in 16-byte units)
#pragma unroll
            for (int k = 0; k < BK / 16; ++k)
              umma_ss<kCtaGroup>(d_tmem, da + ((k * a_kstep) >> 4), db + ((k * b_kstep) >> 4), idesc,
                                 (kb != kb0) || (k != 0));
            if constexpr (kCtaGroup == 1) umma_commit(&empty[stage]);
            else umma_commit_pair(&empty[stage], 3);
          }
          __syncwarp();
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (!ok) break;
        if (elect_one()) {
          if constexpr (kCtaGroup == 1) umma_commit(&tfull[acc]);
          else umma_commit_pair(&tfull[acc], 3);
        }
        __syncwarp();
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1;
      }
      if (!ok && lane == 0) atomicExch(p.err, ERR_WAIT_TIMEOUT);
    }
  } else {
    // ------------------------------------------------------------ epilogue
    const int quarter = warp & 3;
    uint32_t acc = 0, acc_phase = 0;
    uint32_t peer_ready_mask = 0;
    bool ok = true;
    if (p.fused == 2 && blockIdx.x == 0 && warp == 2 && lane < p.world && lane != p.rank)
      pbp::st_release_sys(p.flags[lane] + p.rank, p.epoch);  // "my previous reduce is over": peers may write to me
    const bool vec_ok = (p.ldc % 8 == 0) && (p.residual == nullptr || p.ldr % 8 == 0) &&
                        (((reinterpret_cast<uintptr_t>(p.C) | reinterpret_cast<uintptr_t>(p.residual) |
                           reinterpret_cast<uintptr_t>(p.bias) | reinterpret_cast<uintptr_t>(p.aux)) &
                          15) == 0);
    for (int tile = unit; tile < num_tiles && ok; tile += num_units) {
      int tn, row0, m_limit, grp, kb0, kb1;
      locate(tile, tn, row0, m_limit, grp, kb0, kb1);
      if (kb1 <= kb0) continue;
      const int tm = row0 / TILE_M_ALL;  // fused modes only
      int row = row0 + cta_rank * BM_CTA + quarter * 32 + lane;
      const int n0 = tn * BN;
      void* c_base = p.C;
      if (p.grouped == 2)
        c_base = p.out_fp32 ? static_cast<void*>(reinterpret_cast<float*>(p.C) + grp * p.c_group_stride)
                            : static_cast<void*>(reinterpret_cast<__nv_bfloat16*>(p.C) + grp * p.c_group_stride);
      // grouped M: rows of this tile past the group's end are written as zeros (bf16 outputs)
      const bool zero_tail = (p.grouped == 1) && !p.out_fp32 && row >= m_limit && row < p.M;
      bool peer_tile = false;
      if (p.fused == 2) {
        const int chunk = (tm * (BM_CTA * kCtaGroup)) / p.chunk_rows;
        m_limit = (row < p.M) ? p.chunk_rows : 0;
        row -= chunk * p.chunk_rows;
        if (chunk != p.rank) {
          c_base = p.rs_staging[chunk] + (long long)p.rank * p.chunk_rows * p.ldc;  // my slot in the owner's staging
          // Tiles that leave over NVLink go out as whole 128-byte row pieces: a lane owns a row, so its direct
          // stores are 16-byte pieces 32 rows apart, which use a fraction of the link; two 32-column chunks are
          // staged in shared memory and written back with 8 lanes per row instead.
          peer_tile = vec_ok && !p.out_fp32 && (n0 + BN <= p.N) && (p.M % 32 == 0) && p.bias == nullptr &&
                      p.act == 0 && p.residual == nullptr;
          if (!(peer_ready_mask & (1u << chunk))) {
            // the owner must have finished reducing the previous call's partials before they are overwritten
            bool rdy = true;
            if (lane == 0) rdy = pbp::wait_flag_sys(p.flags[p.rank] + chunk, p.epoch, p.err, ERR_PEER_TIMEOUT);
            rdy = __shfl_sync(0xffffffffu, rdy, 0);
            if (!rdy) {
              ok = false;
              break;
            }
            peer_ready_mask |= 1u << chunk;
          }
        }
      }
      // Warps whose 32 rows all exist take whole 32-column chunks through `fast` code below.  What bounds an epilogue is
      // latency: four warps, one per scheduler, so that every branch, every wait and every round trip to memory
      // adds up (with a bounds test per row and the fused operands tested per chunk, a plain bf16 chunk took 1 400
      // cycles and an fp32 read-modify-write one 4 000).  So the variants are compiled separately, without tests inside;
      // the rows of an operand that the epilogue will read are requested into L2 when the tile starts, one
      // instruction for 32 rows, and read one chunk ahead.  Chunks are turned in shared memory, so that 8 lanes
      // access consecutive 16-byte pieces of one row instead of 32 lanes 32 different rows.
      // On a B200, against one lane per row with the tests inside: 4096 x 14336 x 1024 into fp32 230 -> 145 us (3.2 TB/s of
      // reads and writes), 768 x 3072 x 2048 into fp32 29.5 -> 19.2 us, 2048 x 3072 x 768 23.7 -> 16.3 us, 2048 x 768 x 768 with
      // residual 19.7 -> 12.6 us, 8192 x 4096 x 4096 201 -> 182 us (1 510 TFLOP/s).
      const int row_w = row - lane;  // first of this warp's 32 rows
      const bool fast = vec_ok && p.fused != 2 && row_w + 32 <= m_limit;
      int fast_chunks = fast ? min(BN, p.N - n0) / 32 : 0;
      const bool acc_c = p.accumulate && p.out_fp32 && p.residual == nullptr && p.bias == nullptr && p.act == 0;
      const bool plain_bf16 = !p.out_fp32 && p.residual == nullptr && p.act == 0;
      const bool res_bf16 = !p.out_fp32 && p.residual != nullptr && p.act == 0;
      const int sub_row = lane >> 3, part = lane & 7;
      uint8_t* const stage_w = sEpi + (warp - 2) * 32 * 144;
      if (fast_chunks > 0) {
        if (acc_c)
          prefetch_l2(reinterpret_cast<const float*>(c_base) + (long long)row * p.ldc + n0, fast_chunks * 128);
        else if (res_bf16)
          prefetch_l2(p.residual + (long long)row * p.ldr + n0, fast_chunks * 64);
      }
      // the verdict is the warp's: a lane that left alone would keep the others at the exchanges below for good
      ok = __all_sync(0xffffffffu, mbar_wait(&tfull[acc], acc_phase, abort_flag));
      if (!ok) break;
      tc_fence_after_sync();
      const uint32_t t_row = tmem_base + acc * BN + (static_cast<uint32_t>(quarter * 32) << 16);
      int c_done = 0;
      // split tile: partials of one warp's 32 rows lie as [chunk][float4 of the row][lane], so that both the stores and
      // the reads of a warp are contiguous
      const bool is_split = p.splits > 1 && tile >= p.dp_tiles;
      const int range = is_split ? (tile - p.dp_tiles) % p.splits : 0;
      constexpr long long PART = 32 * BN;                       // floats of one warp's partial
      constexpr long long ITEM = 4 * kCtaGroup * PART;          // floats of one work item
      const float4* parts = nullptr;                            // this warp's partial of range 0
      bool finish = true;
      if (is_split) {
        const int first_item = tile - p.dp_tiles - range;
        const long long slot = (cta_rank * 4 + quarter) * PART;
        parts = reinterpret_cast<const float4*>(p.split_ws + first_item * ITEM + slot);
        finish = false;
        if (row_w < m_limit) {
          float4* own = reinterpret_cast<float4*>(p.split_ws + (first_item + range) * ITEM + slot);
          unsigned long long* counter =
              p.split_counters + (first_item / p.splits) * (4 * kCtaGroup) + cta_rank * 4 + quarter;
          unsigned long long seen = 0;
          if (lane == 0) seen = __ldcg(counter);  // a guess for the exchange below, there by the time it is needed
#pragma unroll 1
          for (int c = 0; c < BN / 32 && n0 + c * 32 < p.N; ++c) {
            uint32_t r[32];
            tmem_ld_32x32(t_row + c * 32, r);
            tmem_ld_wait();
#pragma unroll
            for (int q = 0; q < 8; ++q)
              __stcg(own + (c * 8 + q) * 32 + lane,
                     make_float4(__uint_as_float(r[q * 4]), __uint_as_float(r[q * 4 + 1]),
                                 __uint_as_float(r[q * 4 + 2]), __uint_as_float(r[q * 4 + 3])));
          }
          __threadfence();
          __syncwarp();
          int arrived = 0;
          if (lane == 0) {
            for (int attempt = 0; attempt < 16; ++attempt) {  // fails only when another of the <= 8 ranges got in first
              const unsigned long long base = (seen & ~15ull) == p.split_tag ? seen : p.split_tag;
              const unsigned long long old = atomicCAS(counter, seen, base + 1);
              if (old == seen) {
                arrived = (int)(base & 15ull);
                break;
              }
              seen = old;
            }
          }
          arrived = __shfl_sync(0xffffffffu, arrived, 0);
          finish = arrived == p.splits - 1;
          if (finish) __threadfence();
        }
      }
      if (!finish) {
        c_done = BN / 32;
        fast_chunks = 0;
      }
      // sum of the partials of chunk c in range order (this item's own ones are read back with the others)
      auto gather = [&](int c, uint32_t(&r)[32]) {
        float4 sum[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) sum[q] = __ldcg(parts + (c * 8 + q) * 32 + lane);
        const float4* next = parts + ITEM / 4;
#pragma unroll 3
        for (int i = 1; i < p.splits; ++i, next += ITEM / 4) {
          float4 t[8];
#pragma unroll
          for (int q = 0; q < 8; ++q) t[q] = __ldcg(next + (c * 8 + q) * 32 + lane);
#pragma unroll
          for (int q = 0; q < 8; ++q) sum[q] = add4(sum[q], t[q]);
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          r[q * 4] = __float_as_uint(sum[q].x);
          r[q * 4 + 1] = __float_as_uint(sum[q].y);
          r[q * 4 + 2] = __float_as_uint(sum[q].z);
          r[q * 4 + 3] = __float_as_uint(sum[q].w);
        }
      };
      // this warp's 32 x 32 block of chunk c, turned: v[q] = columns [4 part, +4) of row 4 q + sub_row
      auto turned = [&](int c, float4(&v)[8]) {
        uint32_t r[32];
        if (is_split) {
          gather(c, r);
        } else {
          tmem_ld_32x32(t_row + c * 32, r);
          tmem_ld_wait();
        }
        float4* mine = reinterpret_cast<float4*>(stage_w + lane * 144);
#pragma unroll
        for (int q = 0; q < 8; ++q)
          mine[q] = make_float4(__uint_as_float(r[q * 4]), __uint_as_float(r[q * 4 + 1]), __uint_as_float(r[q * 4 + 2]),
                                __uint_as_float(r[q * 4 + 3]));
        __syncwarp();
        const uint8_t* src = stage_w + sub_row * 144 + part * 16;
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = *reinterpret_cast<const float4*>(src + q * 4 * 144);
        __syncwarp();  // the next chunk may overwrite the stage
      };
      if (fast_chunks > 0 && acc_c) {
        float* cp = reinterpret_cast<float*>(c_base) + (long long)(row_w + sub_row) * p.ldc + n0 + part * 4;
        const long long step = 4 * p.ldc;
        float4 next[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) next[q] = __ldcg(reinterpret_cast<const float4*>(cp + q * step));
#pragma unroll 1
        for (; c_done < fast_chunks; ++c_done, cp += 32) {
          float4 v[8], old[8];
#pragma unroll
          for (int q = 0; q < 8; ++q) old[q] = next[q];
          if (c_done + 1 < fast_chunks) {
#pragma unroll
            for (int q = 0; q < 8; ++q) next[q] = __ldcg(reinterpret_cast<const float4*>(cp + 32 + q * step));
          }
          turned(c_done, v);
#pragma unroll
          for (int q = 0; q < 8; ++q) *reinterpret_cast<float4*>(cp + q * step) = add4(old[q], v[q]);
        }
      } else if (fast_chunks > 0 && (plain_bf16 || res_bf16)) {
        auto bf16_chunks = [&](auto with_bias, auto with_res) {
          __nv_bfloat16* cp = reinterpret_cast<__nv_bfloat16*>(c_base) + (long long)(row_w + sub_row) * p.ldc + n0 + part * 4;
          const __nv_bfloat16* rp =
              with_res.value ? p.residual + (long long)(row_w + sub_row) * p.ldr + n0 + part * 4 : nullptr;
          const __nv_bfloat16* bp = with_bias.value ? p.bias + n0 + part * 4 : nullptr;
          const long long step = 4 * p.ldc, rstep = 4 * p.ldr;
          uint2 next[8];
          uint2 bnext = make_uint2(0u, 0u);
          if constexpr (with_res.value) {
#pragma unroll
            for (int q = 0; q < 8; ++q) next[q] = __ldg(reinterpret_cast<const uint2*>(rp + q * rstep));
          }
          if constexpr (with_bias.value) bnext = __ldg(reinterpret_cast<const uint2*>(bp));
#pragma unroll 1
          for (; c_done < fast_chunks; ++c_done, cp += 32) {
            float4 v[8];
            uint2 res[8];
            const uint2 b = bnext;
            if constexpr (with_res.value) {
#pragma unroll
              for (int q = 0; q < 8; ++q) res[q] = next[q];
            }
            if (c_done + 1 < fast_chunks) {
              if constexpr (with_res.value) {
                rp += 32;
#pragma unroll
                for (int q = 0; q < 8; ++q) next[q] = __ldg(reinterpret_cast<const uint2*>(rp + q * rstep));
              }
              if constexpr (with_bias.value) {
                bp += 32;
                bnext = __ldg(reinterpret_cast<const uint2*>(bp));
              }
            }
            turned(c_done, v);
#pragma unroll
            for (int q = 0; q < 8; ++q) {
              if constexpr (with_bias.value) v[q] = add4(v[q], bf16x4_to_float4(b));
              if constexpr (with_res.value) v[q] = add4(v[q], bf16x4_to_float4(res[q]));
              *reinterpret_cast<uint2*>(cp + q * step) = float4_to_bf16x4(v[q]);
            }
          }
        };
        if (p.bias) {
          if (res_bf16) bf16_chunks(Flag<true>{}, Flag<true>{});
          else bf16_chunks(Flag<true>{}, Flag<false>{});
        } else {
          if (res_bf16) bf16_chunks(Flag<false>{}, Flag<true>{});
          else bf16_chunks(Flag<false>{}, Flag<false>{});
        }
      } else if (fast_chunks > 0 && !p.out_fp32 && p.act == 1 && p.bias && p.aux && p.residual == nullptr) {
        // bias + GELU with the pre-activation kept (the first projection of a GPT-2 MLP in training)
        const long long off = (long long)(row_w + sub_row) * p.ldc + n0 + part * 4;
        __nv_bfloat16* cp = reinterpret_cast<__nv_bfloat16*>(c_base) + off;
        __nv_bfloat16* ap = p.aux + off;
        const __nv_bfloat16* bp = p.bias + n0 + part * 4;
        const long long step = 4 * p.ldc;
#pragma unroll 1
        for (; c_done < fast_chunks; ++c_done, cp += 32, ap += 32, bp += 32) {
          const float4 b = bf16x4_to_float4(__ldg(reinterpret_cast<const uint2*>(bp)));
          float4 v[8];
          turned(c_done, v);
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            v[q] = add4(v[q], b);
            *reinterpret_cast<uint2*>(ap + q * step) = float4_to_bf16x4(v[q]);
            v[q] = make_float4(gelu_tanh(v[q].x), gelu_tanh(v[q].y), gelu_tanh(v[q].z), gelu_tanh(v[q].w));
            *reinterpret_cast<uint2*>(cp + q * step) = float4_to_bf16x4(v[q]);
          }
        }
      }
      // everything else: rows that end inside the warp, the ragged right edge, unaligned outputs, other combinations
      // of fused operands, and the reduce-scatter mode
#pragma unroll 1
      for (int c = c_done; c < BN / 32; ++c) {
        const int col0 = n0 + c * 32;
        if (col0 >= p.N) break;  // uniform across the warp
        uint32_t r[32];
        if (is_split) {
          gather(c, r);
        } else {
          tmem_ld_32x32(t_row + c * 32, r);
          tmem_ld_wait();
        }
        if (zero_tail) {
          __nv_bfloat16* zp = reinterpret_cast<__nv_bfloat16*>(c_base) + (long long)row * p.ldc + col0;
          if (col0 + 32 <= p.N && vec_ok) {
#pragma unroll
            for (int q = 0; q < 4; ++q) reinterpret_cast<uint4*>(zp)[q] = make_uint4(0u, 0u, 0u, 0u);
          } else {
            for (int j = 0; j < 32 && col0 + j < p.N; ++j) zp[j] = __float2bfloat16(0.f);
          }
        }
        if (row < m_limit) {
          float v[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
          const bool full_chunk = (col0 + 32 <= p.N) && vec_ok;
          if (full_chunk) {
            if (p.bias) {
              const uint4* bp = reinterpret_cast<const uint4*>(p.bias + col0);
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                uint4 b4 = __ldg(bp + q);
                const __nv_bfloat162* bb = reinterpret_cast<const __nv_bfloat162*>(&b4);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                  float2 f = __bfloat1622float2(bb[e]);
                  v[q * 8 + e * 2] += f.x;
                  v[q * 8 + e * 2 + 1] += f.y;
                }
              }
            }
            if (p.act == 1) {
              if (p.aux) {
                uint4* ap = reinterpret_cast<uint4*>(p.aux + (long long)row * p.ldc + col0);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                  uint4 o;
                  __nv_bfloat162* ob = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
                  for (int e = 0; e < 4; ++e) ob[e] = __floats2bfloat162_rn(v[q * 8 + e * 2], v[q * 8 + e * 2 + 1]);
                  ap[q] = o;
                }
              }
#pragma unroll
              for (int j = 0; j < 32; ++j) v[j] = gelu_tanh(v[j]);
            }
            if (p.residual) {
              const uint4* rp = reinterpret_cast<const uint4*>(p.residual + (long long)row * p.ldr + col0);
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                uint4 r4 = __ldg(rp + q);
                const __nv_bfloat162* rb = reinterpret_cast<const __nv_bfloat162*>(&r4);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                  float2 f = __bfloat1622float2(rb[e]);
                  v[q * 8 + e * 2] += f.x;
                  v[q * 8 + e * 2 + 1] += f.y;
                }
              }
            }
            if (p.out_fp32) {
              float4* cp = reinterpret_cast<float4*>(reinterpret_cast<float*>(c_base) + (long long)row * p.ldc + col0);
              if (p.accumulate) {
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                  float4 o = cp[q];
                  o.x += v[q * 4];
                  o.y += v[q * 4 + 1];
                  o.z += v[q * 4 + 2];
                  o.w += v[q * 4 + 3];
                  cp[q] = o;
                }
              } else {
#pragma unroll
                for (int q = 0; q < 8; ++q) cp[q] = make_float4(v[q * 4], v[q * 4 + 1], v[q * 4 + 2], v[q * 4 + 3]);
              }
            } else {
              uint4* cp =
                  peer_tile
                      ? reinterpret_cast<uint4*>(sEpi + ((warp - 2) * 32 + lane) * 144 + (c & 1) * 64)
                      : reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(c_base) + (long long)row * p.ldc +
                                                 col0);
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                uint4 o;
                __nv_bfloat162* ob = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
                for (int e = 0; e < 4; ++e) ob[e] = __floats2bfloat162_rn(v[q * 8 + e * 2], v[q * 8 + e * 2 + 1]);
                cp[q] = o;
              }
            }
          } else {
            // ragged edge: scalar path
            for (int j = 0; j < 32; ++j) {
              const int col = col0 + j;
              if (col >= p.N) break;
              float x = v[j];
              if (p.bias) x += __bfloat162float(p.bias[col]);
              if (p.act == 1) {
                if (p.aux) p.aux[(long long)row * p.ldc + col] = __float2bfloat16(x);
                x = gelu_tanh(x);
              }
              if (p.residual) x += __bfloat162float(p.residual[(long long)row * p.ldr + col]);
              if (p.out_fp32) {
                float* cp = reinterpret_cast<float*>(c_base) + (long long)row * p.ldc + col;
                *cp = p.accumulate ? (*cp + x) : x;
              } else {
                reinterpret_cast<__nv_bfloat16*>(c_base)[(long long)row * p.ldc + col] = __float2bfloat16(x);
              }
            }
          }
        }
        if (peer_tile && (c & 1)) {
          // 32 rows x 128 bytes staged by this warp: piece i = q * 32 + lane is bytes [16 * (i % 8), +16) of row i / 8
          __syncwarp();
          const int row_w = row - lane;  // first row of this warp's block, relative to the owner's chunk
          const uint8_t* stage = sEpi + (warp - 2) * 32 * 144;
          __nv_bfloat16* dst0 = reinterpret_cast<__nv_bfloat16*>(c_base) + n0 + (c - 1) * 32;
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const int i = q * 32 + lane;
            const int rr = i >> 3, part = i & 7;
            if (row_w + rr < m_limit && row_w + rr >= 0) {
              const uint4 val = *reinterpret_cast<const uint4*>(stage + rr * 144 + part * 16);
              *reinterpret_cast<uint4*>(dst0 + (long long)(row_w + rr) * p.ldc + part * 8) = val;
            }
          }
          __syncwarp();
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) {
        if constexpr (kCtaGroup == 1) mbar_arrive(&tempty[acc]);
        else mbar_arrive_cluster(&tempty[acc], 0);
      }
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1;
    }
    if (!ok && lane == 0) atomicExch(p.err, ERR_WAIT_TIMEOUT);
  }

  // ---------------------------------------------------------------- teardown
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag) {
    // give copies still in flight time to land before shared memory is released
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
  }
  __syncwarp();
  if constexpr (kCtaGroup == 2) cluster_sync_all();
  tc_fence_after_sync();
  __syncwarp();
  if (warp == 1) tmem_dealloc<kCtaGroup>(tmem_base, TMEM_COLS);

  if (p.fused == 2) {
    // ------------------------------------------------------------ reduce-scatter tail: sum what arrived
    using namespace pbp;
    const int W = p.world;
    __threadfence_system();
    if (!grid_barrier(p.counters, (int)gridDim.x, p.err, ERR_PEER_TIMEOUT)) return;
    if (blockIdx.x == 0 && (int)threadIdx.x < W && (int)threadIdx.x != p.rank)
      st_release_sys(p.flags[threadIdx.x] + W + p.rank, p.epoch);  // everything I owed you has been stored
    bool ok = true;
    if ((int)threadIdx.x < W && (int)threadIdx.x != p.rank)
      ok = wait_flag_sys(p.flags[p.rank] + W + threadIdx.x, p.epoch, p.err, ERR_PEER_TIMEOUT);
    if (!__syncthreads_and(ok)) return;
    const __nv_bfloat16* mine = reinterpret_cast<const __nv_bfloat16*>(p.C);
    const __nv_bfloat16* stag = p.rs_staging[p.rank];
    const int vec_per_row = p.N / 8;
    const long long total = (long long)p.chunk_rows * vec_per_row;
    // Four output vectors per thread and trip, all their loads issued before the first use: with one vector in
    // flight per thread this pass ran at a fraction of the HBM rate.
    constexpr int RU = 4;
    const long long nthr = (long long)gridDim.x * blockDim.x;
    auto add8 = [](float* accv, const uint4& u) {
      const __nv_bfloat162* b2 = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 f = __bfloat1622float2(b2[e]);
        accv[2 * e] += f.x;
        accv[2 * e + 1] += f.y;
      }
    };
    for (long long i0 = blockIdx.x * (long long)blockDim.x + threadIdx.x; i0 < total; i0 += nthr * RU) {
      long long off[RU];
      uint4 own[RU], res[RU];
#pragma unroll
      for (int u = 0; u < RU; ++u) {
        const long long i = i0 + u * nthr;
        off[u] = -1;
        if (i < total) {
          off[u] = (i / vec_per_row) * p.ldc + (i % vec_per_row) * 8;
          own[u] = *reinterpret_cast<const uint4*>(mine + off[u]);
          if (p.rs_residual) res[u] = *reinterpret_cast<const uint4*>(p.rs_residual + off[u]);
        }
      }
      float accv[RU][8];
#pragma unroll
      for (int u = 0; u < RU; ++u) {
#pragma unroll
        for (int e = 0; e < 8; ++e) accv[u][e] = 0.f;
        if (off[u] >= 0) {
          add8(accv[u], own[u]);
          if (p.rs_residual) add8(accv[u], res[u]);
        }
      }
      for (int src = 0; src < W; ++src) {
        if (src == p.rank) continue;
        const __nv_bfloat16* base = stag + (long long)src * p.chunk_rows * p.ldc;
        uint4 v[RU];
#pragma unroll
        for (int u = 0; u < RU; ++u)
          if (off[u] >= 0) v[u] = *reinterpret_cast<const uint4*>(base + off[u]);
#pragma unroll
        for (int u = 0; u < RU; ++u)
          if (off[u] >= 0) add8(accv[u], v[u]);
      }
#pragma unroll
      for (int u = 0; u < RU; ++u) {
        if (off[u] < 0) continue;
        uint4 o;
        __nv_bfloat162* ob = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
        for (int e = 0; e < 4; ++e) ob[e] = __floats2bfloat162_rn(accv[u][2 * e], accv[u][2 * e + 1]);
        *reinterpret_cast<uint4*>(p.rs_out + off[u]) = o;
      }
    }
  }
}

// Tile order knob: output tiles are walked in bands of `group_m` row tiles, row-fastest inside a band (0 = default).
static int g_group_m = 0;

template <int kCtaGroup, int BN, int kStages>
static int launch_gemm(const CUtensorMap& tmA, const CUtensorMap& tmB, GemmParams p, int sm_count,
                       cudaStream_t stream, const CUtensorMap* tmA2 = nullptr, int copy_ctas = 0,
                       int tile_multiplier = 1) {
  constexpr int A_BYTES = BM_CTA * BK * 2;
  constexpr int B_BYTES = (BN / kCtaGroup) * BK * 2;
  constexpr int SMEM = kStages * (A_BYTES + B_BYTES) + 1024 + 256 + 4 * 32 * 144;
  constexpr auto kern = gemm_bf16_kernel<kCtaGroup, BN, kStages>;
  if (cudaError_t e = pb::allow_smem<kern, SMEM>(); e != cudaSuccess) return (int)e;
  const int tile_m = BM_CTA * kCtaGroup;
  p.num_m_tiles = (p.M + tile_m - 1) / tile_m;
  p.num_n_tiles = (p.N + BN - 1) / BN;
  p.num_k_blocks = (p.K + BK - 1) / BK;
  p.group_m = kCtaGroup == 1 ? 16 : 8;
  if (g_group_m > 0 && !p.fused) p.group_m = g_group_m;
  // grouped M: up to one partial tile per group on top of the dense count (p.M is the buffers' row capacity)
  int tiles = (p.num_m_tiles + (p.grouped == 1 ? p.n_groups : 0)) * p.num_n_tiles * tile_multiplier;
  if (p.splits > 1) tiles = p.dp_tiles + (tiles - p.dp_tiles) * p.splits;
  int units = (sm_count - copy_ctas) / kCtaGroup;
  if (units > tiles) units = tiles;
  if (units < 1) units = 1;
  if (p.fused) {
    const int tiles_per_chunk = p.chunk_rows / tile_m;
    // own chunk first when gathering (its rows need no transfer), last when scattering (foreign tiles leave early)
    p.m_rot = (p.fused == 1 ? p.rank : (p.rank + 1) % p.world) * tiles_per_chunk;
    p.gemm_ctas = units * kCtaGroup;
  }
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(units * kCtaGroup + (p.fused == 1 ? copy_ctas : 0), 1, 1);
  cfg.blockDim = dim3(192, 1, 1);
  cfg.dynamicSmemBytes = SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = kCtaGroup;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, tmA, tmB, tmA2 ? *tmA2 : tmA, p);
  pb_count_launch(1);
  return (int)e;
}

}  // namespace pb

static int g_sm_reserve = 0;

namespace {

// How a plain GEMM is cut: kernel variant, tiles that run whole, ranges that each remaining tile is split into.
struct GemmPlan {
  int variant, dp_tiles, splits;
  int items;  // split work items (0: no workspace needed)
  double cycles;
};

constexpr long long SPLIT_ITEM_BYTES = 128 * 256 * 4;  // partial of one CTA, largest variant
constexpr int SPLIT_COUNTERS = 1024;                   // 4 per CTA of a split tile, at most 148 CTAs
std::atomic<unsigned long long> g_split_calls{0};      // source of the launches' tags (never 0: cleared counters)

// Estimated SM cycles of `variant` and the best split of its last wave.  Tiles run in waves of one per worker (CTA or
// CTA pair).  When r tiles are left for the last wave they are cut into s ranges of k-blocks, r * s <= workers: the
// wave takes 1/s of the time, plus the partial tiles' way through L2.
//
// Constants measured on a B200.  A 64-deep k-block takes about 480 cycles with 128 x 128 tiles, 640 with 128 x 256, 500
// with pairs (2 % below their tensor rate of 512, which long main loops run at).  The epilogue is charged once, as that of a
// plain bf16 output: one of an fp32 read-modify-write pair tile takes 9 000 to 14 000 cycles, and the waves of such a
// weight gradient with K below about 1 200 to 1 800 are bound by it, which the rule does not see.  Start, first operands, last MMAs and the last tile's epilogue add
// 7 000, 9 500 and 14 000.  Splitting costs 6 000 + 2 000 s with 128 x 128 tiles and 9 000 + 5 000 s with 256 columns.
// Against the best unsplit variant, us: 77 x 4096 x 11008 46.1 -> 25.2 (s = 4), 77 x 4096 x 4096 20.6 -> 16.3 (4),
// 2048 x 768 x 50304 192 -> 118 (3), 2999 x 5120 x 13824 321 -> 291 (4), 4096 x 4096 x 8192 205 -> 192 (2); on the other
// side of the line 768 x 768 x 2048 14.4 -> 16.3 (3), 4095 x 4096 x 4096 97.1 -> 98.5 (2).  Variants where none is
// split: 2048 x 768 x 768 11.4 with pairs, 8.6 with 128 x 128; 2048 x 50304 x 768 135 and 167.
GemmPlan plan_variant(int variant, int M, int N, int K, int sms, bool may_split) {
  const int ctas = variant == 2 ? 2 : 1, bn = variant == 3 ? 128 : 256;
  const int units = sms / ctas;
  const int tiles = ((M + 128 * ctas - 1) / (128 * ctas)) * ((N + bn - 1) / bn);
  const int kb = (K + 63) / 64;
  const double per_kb = variant == 2 ? 500 : (variant == 1 ? 640 : 480);
  const double edge = variant == 2 ? 14000 : (variant == 1 ? 9500 : 7000);
  const double split_fixed = variant == 3 ? 6000 : 9000, split_each = variant == 3 ? 2000 : 5000;
  const int whole = tiles / units, rest = tiles - whole * units;
  GemmPlan best{variant, tiles, 1, 0, edge + (whole + (rest ? 1 : 0)) * kb * per_kb};
  if (may_split && rest) {
    for (int s = 2; s <= 8 && rest * s <= units && s * 4 <= kb; ++s) {
      const double c = edge + whole * kb * per_kb + ((kb + s - 1) / s) * per_kb + split_fixed + split_each * s;
      if (c < 0.99 * best.cycles) best = GemmPlan{variant, whole * units, s, rest * s, c};
    }
  }
  return best;
}

// The cheapest variant.  N <= 128 leaves half of a 256-column tile empty, M <= 128 the second CTA of a pair.
GemmPlan plan_gemm(int M, int N, int K, int sms, bool may_split) {
  GemmPlan plan = plan_variant(3, M, N, K, sms, may_split);
  if (N > 128) {
    const GemmPlan wide = plan_variant(1, M, N, K, sms, may_split);
    if (wide.cycles < plan.cycles) plan = wide;
    if (M > 128) {
      const GemmPlan pair = plan_variant(2, M, N, K, sms, may_split);
      if (pair.cycles < plan.cycles) plan = pair;
    }
  }
  return plan;
}

}  // namespace

extern "C" {

// Leaves `n` SMs out of the persistent GEMM grid (for communication kernels that must run beside it).
void pb_set_sm_reserve(int n) { g_sm_reserve = n < 0 ? 0 : n; }
int pb_get_sm_reserve() { return g_sm_reserve; }

// Rows of output tiles per band of the tile order of the plain and grouped GEMMs (0 restores the default).
void pb_set_gemm_group_m(int n) { pb::g_group_m = n < 0 ? 0 : n; }

// C[M,N] = A.B^T with fused epilogue.  A: a_mn ? [K, M] (ld = lda) : [M, K];  B: b_mn ? [K, N] : [N, K].
// variant: 0 = automatic, 1 = single-CTA tiles (128 x 256), 2 = CTA-pair tiles (256 x 256),
//          3 = single-CTA 128 x 128.
// Returns 0 on success, a negative value for an argument error, a positive CUDA error otherwise.
// `split_ws`: pb_gemm_split_ws_bytes() bytes that no other stream uses, its last 8 KB (the counters) cleared before the
// first call; null = the contraction is never split.  A call under capture bakes its tag into the graph, which therefore
// has to clear the counters itself before the kernel.  With `ask_ws` != 0 the call returns
// PB_GEMM_WANTS_WS, without launching anything, where a split needs a workspace and none is given, or the given one
// (which outlives the call) would become part of a graph under capture.
#define PB_GEMM_WANTS_WS (-100)
long long pb_gemm_split_ws_bytes() { return 148LL * SPLIT_ITEM_BYTES + SPLIT_COUNTERS * 8; }

// out: variant, whole tiles, ranges per split tile, split work items
void pb_gemm_plan(int M, int N, int K, int sms, int may_split, int* out) {
  const GemmPlan plan = plan_gemm(M, N, K, sms, may_split != 0);
  out[0] = plan.variant;
  out[1] = plan.dp_tiles;
  out[2] = plan.splits;
  out[3] = plan.items;
}

int pb_gemm_bf16_ws(const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb,
                    long long ldc, int a_mn, int b_mn, const void* bias, const void* residual, long long ldr, void* aux,
                    int act, int out_fp32, int accumulate, int variant, void* split_ws, int ask_ws, int* err_dev,
                    void* stream_) {
  using namespace pb;
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  if (M <= 0 || N <= 0 || K <= 0) return -1;
  if ((lda % 8) || (ldb % 8)) return -2;  // TMA needs 16-byte row pitch
  if ((reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(B) & 15)) return -3;
  if (accumulate && !out_fp32) return -4;
  static int sm_count = 0;
  if (!sm_count) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev);
  }
  int sms = sm_count - g_sm_reserve;
  if (sms < 2) sms = 2;
  GemmPlan plan{variant, 0, 1, 0, 0.0};
  if (variant == 0) {
    plan = plan_gemm(M, N, K, sms, (split_ws != nullptr || ask_ws) && sms <= 148);  // the workspace is sized for 148
    if (plan.splits > 1 && ask_ws) {
      cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
      cudaError_t e = split_ws ? cudaStreamIsCapturing(stream, &capture) : cudaSuccess;
      if (e != cudaSuccess) return (int)e;
      if (split_ws == nullptr || capture != cudaStreamCaptureStatusNone) return PB_GEMM_WANTS_WS;
    }
    variant = plan.variant;
  }
  const int bn = (variant == 3) ? 128 : 256;
  const int b_rows = (variant == 2) ? bn / 2 : bn;

  CUtensorMap tmA, tmB;
  int r;
  if (!a_mn) r = make_tmap_bf16_2d(&tmA, A, (uint64_t)K, (uint64_t)M, (uint64_t)lda, 64, 128);
  else r = make_tmap_bf16_2d(&tmA, A, (uint64_t)M, (uint64_t)K, (uint64_t)lda, 64, 64);
  if (r) return -1000 - r;  // tensor map of A refused: -1000 - CUresult (or +1 when the encoder is missing)
  if (!b_mn) r = make_tmap_bf16_2d(&tmB, B, (uint64_t)K, (uint64_t)N, (uint64_t)ldb, 64, (uint32_t)b_rows);
  else r = make_tmap_bf16_2d(&tmB, B, (uint64_t)N, (uint64_t)K, (uint64_t)ldb, 64, 64);
  if (r) return -2000 - r;  // tensor map of B refused

  GemmParams p;
  memset(&p, 0, sizeof(p));
  p.M = M;
  p.N = N;
  p.K = K;
  p.C = C;
  p.ldc = ldc;
  p.bias = reinterpret_cast<const __nv_bfloat16*>(bias);
  p.residual = reinterpret_cast<const __nv_bfloat16*>(residual);
  p.ldr = ldr;
  p.aux = reinterpret_cast<__nv_bfloat16*>(aux);
  p.act = act;
  p.out_fp32 = out_fp32;
  p.accumulate = accumulate;
  p.a_mn = a_mn;
  p.b_mn = b_mn;
  p.err = err_dev;
  p.dp_tiles = plan.dp_tiles;
  p.splits = plan.splits;
  p.split_ws = reinterpret_cast<float*>(split_ws);
  if (plan.splits > 1) {
    p.split_counters =
        reinterpret_cast<unsigned long long*>(reinterpret_cast<char*>(split_ws) + 148LL * SPLIT_ITEM_BYTES);
    p.split_tag = (g_split_calls.fetch_add(1, std::memory_order_relaxed) + 1) << 4;
  }
  switch (variant) {
    case 1: return launch_gemm<1, 256, 4>(tmA, tmB, p, sms, stream);
    case 2: return launch_gemm<2, 256, 6>(tmA, tmB, p, sms, stream);
    case 3: return launch_gemm<1, 128, 6>(tmA, tmB, p, sms, stream);
    default: return -5;
  }
}

// Grouped GEMMs of a mixture-of-experts layer: ONE launch covers all local experts, and the group sizes stay on the
// device (group_rows / group_start: int[n_groups] in device memory, group_start[g] a multiple of 256).
//   mode 1 (rows grouped):  C[r, :] = A[r, :] . B_g^T for the rows r of group g.  A: [M, K] K-major, M = the row
//       capacity of the buffers.  B: b_mn ? the groups' [K, N] matrices stacked to [n_groups * K, N]
//                                         : the groups' [N, K] matrices stacked to [n_groups * N, K].
//       C: [M, N] bf16.  Rows of a computed tile beyond its group's end are set to zero; tiles without rows of any
//       group are not computed and their part of C is left untouched.  b_mn needs K % 64 == 0.
//   mode 2 (contraction grouped):  C_g[M, N] (+)= sum over the rows r of group g of A[r, m] * B[r, n].
//       A: [rows, M], B: [rows, N] (both MN-major), C: n_groups stacked [M, N] blocks (fp32 accumulate or bf16).
//       Rows from a group's end to the next multiple of 64 take part: they must be zero in A or in B and finite in
//       the other (mode 1 outputs satisfy this).
int pb_gemm_grouped(int mode, const void* A, const void* B, void* C, int M, int N, int K, long long lda,
                    long long ldb, long long ldc, int b_mn, int n_groups, const int* group_rows,
                    const int* group_start, int out_fp32, int accumulate, int* err_dev, void* stream_) {
  using namespace pb;
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  if (mode != 1 && mode != 2) return -1;
  if (M <= 0 || N <= 0 || K <= 0 || n_groups < 1 || n_groups > MAX_GROUPS) return -1;
  if ((lda % 8) || (ldb % 8) || (ldc % 8)) return -2;
  if ((reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(B) & 15)) return -3;
  if (accumulate && !out_fp32) return -4;
  if (mode == 1 && (out_fp32 || (b_mn && K % 64 != 0))) return -6;
  static int sm_count = 0;
  if (!sm_count) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev);
  }
  CUtensorMap tmA, tmB;
  int r;
  if (mode == 1) {
    r = make_tmap_bf16_2d(&tmA, A, (uint64_t)K, (uint64_t)M, (uint64_t)lda, 64, 128);
    if (r) return -10;
    if (!b_mn) r = make_tmap_bf16_2d(&tmB, B, (uint64_t)K, (uint64_t)n_groups * N, (uint64_t)ldb, 64, 128);
    else r = make_tmap_bf16_2d(&tmB, B, (uint64_t)N, (uint64_t)n_groups * K, (uint64_t)ldb, 64, 64);
    if (r) return -11;
  } else {
    r = make_tmap_bf16_2d(&tmA, A, (uint64_t)M, (uint64_t)K, (uint64_t)lda, 64, 64);
    if (r) return -10;
    r = make_tmap_bf16_2d(&tmB, B, (uint64_t)N, (uint64_t)K, (uint64_t)ldb, 64, 64);
    if (r) return -11;
  }
  GemmParams p;
  memset(&p, 0, sizeof(p));
  p.M = M;
  p.N = N;
  p.K = K;
  p.C = C;
  p.ldc = ldc;
  p.out_fp32 = out_fp32;
  p.accumulate = accumulate;
  p.a_mn = mode == 2;
  p.b_mn = mode == 2 ? 1 : b_mn;
  p.err = err_dev;
  p.grouped = mode;
  p.n_groups = n_groups;
  p.group_rows = group_rows;
  p.group_start = group_start;
  p.b_group_stride = b_mn ? K : N;
  p.c_group_stride = (long long)M * ldc;
  int sms = sm_count - g_sm_reserve;
  if (sms < 2) sms = 2;
  return launch_gemm<2, 256, 6>(tmA, tmB, p, sms, stream, nullptr, 0, mode == 2 ? n_groups : 1);
}


// Tensor-parallel fused GEMMs over peer memory (CTA-pair tiles, 256 x 256).
//   mode 1 (all-gather -> GEMM):  C[world*chunk_rows, N] = concat_r(shard_r)[.., K] . B^T.  `a_local` is this rank's
//       shard, `peer_src[r]` every rank's shard (peer mapped), `gathered` a local [world*chunk_rows, K] buffer.
//   mode 2 (GEMM -> reduce-scatter): partial = A[world*chunk_rows, K] . B^T; rank r ends up with
//       rs_out[chunk_rows, N] = sum over ranks of their partial rows [r*chunk_rows, (r+1)*chunk_rows) (+ residual).
//       `C` is local scratch [chunk_rows, N]; `rs_staging[r]` every rank's [world, chunk_rows, N] staging buffer.
// chunk_rows must be a multiple of 256; K, N multiples of 8; flags[r]: every rank's int[2*world] block;
// tile_flags: local int[world*chunk_rows/256]; counters: local int[16]. All flag memory starts at zero and `epoch`
// grows by one per call on every rank.
int pb_gemm_tp_fused(int mode, const void* a_local, const void* B, void* C, int N, int K, long long lda,
                     long long ldb, long long ldc, int b_mn, int rank, int world, int chunk_rows, int epoch,
                     void** peer_src, void* gathered, void** rs_staging, void* rs_out, const void* rs_residual,
                     int** flags, int* tile_flags, int* counters, int copy_ctas, int* err_dev, void* stream_) {
  using namespace pb;
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  if (mode != 1 && mode != 2) return -1;
  if (world < 2 || world > 8 || chunk_rows % 256 != 0) return -2;
  if ((lda % 8) || (ldb % 8) || (ldc % 8) || (N % 8) || (K % 8)) return -3;
  if (mode == 1 && lda != K) return -4;  // shards are streamed as contiguous byte ranges
  static int sm_count = 0;
  if (!sm_count) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev);
  }
  const int M = world * chunk_rows;
  CUtensorMap tmA, tmA2, tmB;
  if (mode == 1) {
    if (make_tmap_bf16_2d(&tmA, a_local, (uint64_t)K, (uint64_t)chunk_rows, (uint64_t)lda, 64, 128)) return -10;
    if (make_tmap_bf16_2d(&tmA2, gathered, (uint64_t)K, (uint64_t)M, (uint64_t)lda, 64, 128)) return -10;
  } else {
    if (make_tmap_bf16_2d(&tmA, a_local, (uint64_t)K, (uint64_t)M, (uint64_t)lda, 64, 128)) return -10;
    tmA2 = tmA;
  }
  int r;
  if (!b_mn) r = make_tmap_bf16_2d(&tmB, B, (uint64_t)K, (uint64_t)N, (uint64_t)ldb, 64, 128);
  else r = make_tmap_bf16_2d(&tmB, B, (uint64_t)N, (uint64_t)K, (uint64_t)ldb, 64, 64);
  if (r) return -11;
  GemmParams p;
  memset(&p, 0, sizeof(p));
  p.M = M;
  p.N = N;
  p.K = K;
  p.C = C;
  p.ldc = ldc;
  p.b_mn = b_mn;
  p.err = err_dev;
  p.fused = mode;
  p.rank = rank;
  p.world = world;
  p.chunk_rows = chunk_rows;
  p.lda_elems = lda;
  p.epoch = epoch;
  p.tile_flags = tile_flags;
  p.counters = counters;
  for (int i = 0; i < world; ++i) {
    p.flags[i] = flags[i];
    if (peer_src) p.peer_src[i] = reinterpret_cast<const __nv_bfloat16*>(peer_src[i]);
    if (rs_staging) p.rs_staging[i] = reinterpret_cast<__nv_bfloat16*>(rs_staging[i]);
  }
  p.gathered = reinterpret_cast<__nv_bfloat16*>(gathered);
  p.rs_out = reinterpret_cast<__nv_bfloat16*>(rs_out);
  p.rs_residual = reinterpret_cast<const __nv_bfloat16*>(rs_residual);
  cudaError_t e = cudaMemsetAsync(counters, 0, 16 * sizeof(int), stream);
  if (e != cudaSuccess) return (int)e;
  int sms = sm_count - g_sm_reserve;
  if (copy_ctas < 2) copy_ctas = 2;
  copy_ctas &= ~1;
  // every CTA of this grid waits on others of the same grid: it must be fully resident
  return launch_gemm<2, 256, 6>(tmA, tmB, p, sms, stream, &tmA2, mode == 1 ? copy_ctas : 0);
}

}  // extern "C"
