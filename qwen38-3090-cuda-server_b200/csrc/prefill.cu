// Prefill W4A16 GEMM for sm_100a:  C[M, out_f] = A[M, in_f] @ W^T  (bf16 in/out, fp32 accumulate)
// with the dequantisation fused into the tensor-core pipeline.
//
// Replaces gemm_w4a16 of the reference (src/kernels/gemm_w4a16.cu:63-88), which expands a
// weight tile to bf16 in a 256 MB workspace (k_dequant_rows) and calls cublasGemmEx. Here no
// bf16 copy of the weights ever touches global or shared memory:
//   * a pair of CTAs (cta_group::2) computes a tile of 256 output rows x TN tokens: each CTA holds the weights
//     and the fp32 accumulator of its own 128 rows in tensor memory and HALF of the tile's tokens in shared
//     memory. A CTA alone (128 rows x 256 tokens) pulls 72 KB through L2 per k group and 1024 tensor
//     cycles; a pair's CTA pulls 41 KB for the same math, which leaves room for four
//     group stages of activations instead of two;
//   * a producer thread per CTA streams the packed int4 blocks of its row tile through a ring of
//     shared-memory stages with 1-D bulk async copies (cp.async.bulk + mbarrier);
//   * sixteen dequant warps per CTA (one output row per thread; four teams take the k groups in
//     turn) turn 64 bytes of nibbles into bf16 weights in registers - (128+q) by LOP3,
//     minus (128+zp) and times the group scale with packed bf16 arithmetic, which is exactly
//     bf16(float(q-zp)*float(s)), the value w4a16_dequant_rows produces - and store them as the A operand
//     into tensor memory (tcgen05.st);
//   * a second producer thread per CTA brings its half of the activation tile in with tiled TMA loads
//     (cp.async.bulk.tensor, 128-byte swizzle), which is the K-major B operand as is; both CTAs' loads
//     complete on the leader's mbarrier;
//   * one thread of the leader CTA issues tcgen05.mma (256 x N x 16, kind::f16) per 16-k slab for both
//     CTAs, and one commit per group tells both CTAs that the A columns and the stage are free;
//   * eight epilogue warps per CTA read the accumulator back with tcgen05.ld into shared memory, hand it back to the
//     issuer, and store C in 256-byte rows while the next tile's main loop runs;
//   * few tiles (short prompts, narrow layers): a cluster of 2 S CTAs splits K S ways; the splits' fp32 tiles
//     are added through distributed shared memory, always in split order (bitwise reproducible).
//
// What bounds it: long prompts run at the tensor cores' rate under the power cap (256 x 256 x 16 per 128 cycles: 1024
// cycles per k group; tensor pipe 87 % active over a 4096-token launch), short ones by no single role: a CTA and k group takes
// 640 to 700 cycles (5120 x 17408 at M = 77: issue slots 52 %, ALU pipe 41 % on average and 52 % on the busiest SM, tensor pipe 43 % of active
// cycles), where HBM would allow 386.
// In us, weights cold, against one CTA per tile of 128 x 256 with eight dequant warps (by box and temperature: 2 to 10 %):
//   34816 x 5120, M = 4096: 1264 -> 922 (1583 TFLOP/s); 5120 x 17408, M = 4096: 698 -> 488 (1497)
//   34816 x 5120, M = 777:   300 -> 208;                5120 x 8192, M = 777:   110 -> 54
//   34816 x 5120, M = 77:     73 -> 34;                 5120 x 17408, M = 77:   105 -> 23;     8192 x 5120, M = 77: 45 -> 13
// and on the way, 34816 x 5120 at M = 4096 on one device: half groups as the unit of every hand-off 1134 (the first shape; the
// issuing thread is the limit), whole groups 1063, two teams of dequant warps (four since) and C through shared memory 890. A warp's vote on
// its waits took another 9 % off short prompts (34816 x 5120 at M = 77: 40.8 -> 37.1) by keeping the loops warp-uniform.
// Programmatic dependent launch (the next launch sets up, streams and expands its first weights as this one's CTAs leave) took
// the four layers of a block from 104.8 to 96.5 us at M = 77 (5120 -> 8192, 6144 -> 5120, MLP) and from 562.5 to 546.7 at M = 777.
#include <cuda.h>
#include <cstring>
#include <mutex>

#include "common.cuh"

namespace w4a16 {
namespace {

constexpr int PW = 16;                      // dequant warps: 4 TMEM lane quarters x 4 groups
constexpr int EW = 8;                       // epilogue warps: two per lane quarter, each half of the tokens
constexpr int kWEpi0 = PW, kWWeights = PW + EW, kWIssue = kWWeights + 1, kWActs = kWIssue + 1;
constexpr int kPWarps = kWActs + 1;
constexpr int kPRows = 2 * kTileRows;       // output rows of a CTA pair's tile
constexpr int kPMaxTN = 256;                // tokens of a tile: a multiple of 32 (the pair's MMA needs N % 32 == 0)
constexpr int kPMaxSplit = 4;               // 2 S <= 8 CTAs: the portable cluster size
constexpr int kPSteps = 4;                  // activation stages, each one k group of the CTA's TN / 2 tokens
constexpr int kPDone = 8;                   // ring of "group multiplied" barriers: at least kPSteps and the A slots
constexpr int kPMaxWD = 16;                 // weight ring stages (one k group each), at most
constexpr uint32_t kPTmemCols = 512;
constexpr uint32_t kPSpin = 1u << 20;
constexpr uint32_t kMagicP = 0x43004300u, kNibMaskP = 0x000F000Fu;
constexpr int kPTeams = 4;                  // teams of dequant warps
constexpr int kPMaxA = 6;                   // A slots, at most
constexpr int kPBars = 2 * kPMaxWD + kPDone + kPMaxA + kPSteps + 2;
// Tensor memory: the accumulator's TN columns, the rest are slots of the A operand, 64 columns per k group.
__host__ __device__ constexpr int a_slots(int tn) { return tn <= 128 ? 6 : 4; }
static_assert(128 + 6 * 64 <= 512 && 256 + 4 * 64 <= 512 && kPMaxA <= kPDone && kPSteps <= kPDone, "ring depths");

struct PrefillParams {
  CUtensorMap amap;   // A as [M][K] bf16, box 64 k x TN / 2 tokens, 128-byte swizzle, zero fill
  const uint8_t* stream;
  uint16_t* C;        // [M][ldc] bf16; this launch's rows land in columns [col0, col0 + N)
  int M, N, K, G, row_tiles, pairs;  // pairs: row tiles in twos (an odd last one repeats the last tile and stores nothing)
  int tn, splits, wdepth;            // wdepth is a multiple of four: a stage is always read by the same dequant warps
  int full_tt, tiles;                // token tiles of TN tokens; tiles in all (the ragged token tile's come last)
  long long ldc;
  int wide;                          // C (and every peer's) takes 16-byte stores: base, ldc and col0 are multiples of that
  int col0;
  int* status;
  // column-sharded call: the other ranks' C (peer-mapped) receive the same tile, then the completion flag
  int npeers;
  uint16_t* C_peers[8];
  unsigned* comm_local;
  unsigned* comm_peers[8];
  int comm_n, comm_rank;
};

__device__ __forceinline__ uint32_t fma_bf16x2(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}

// ---- CTA pairs and clusters --------------------------------------------------------------
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t map_to_rank(uint32_t saddr, uint32_t rank) {
  uint32_t d;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(d) : "r"(saddr), "r"(rank));
  return d;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Arrival on a barrier of any CTA of the cluster (a mapped address). What it hands over is tensor memory, ordered by
// the tcgen05 fences around it, so the barrier needs no cluster-scope release (which costs a memory fence).
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ float4 ld_cluster_f32x4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(addr)
               : "memory");
  return v;
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t smem_dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(ncols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// D[both CTAs' tmem] (+)= A[both CTAs' tmem] * B[half of the columns from each CTA's shared memory]
__device__ __forceinline__ void umma_bf16_ts_pair(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                                  uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
      "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// One arrival on the barrier at this offset in every CTA of `mask` once all MMAs issued so far have completed.
__device__ __forceinline__ void umma_commit_pair(uint32_t bar, uint16_t mask) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
      "h"(mask)
      : "memory");
}
// Tiled TMA load of a 64 x TN / 2 box (k, token) into this CTA's shared memory; completion on the pair leader's mbarrier.
__device__ __forceinline__ void tma_load_pair(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::
          "r"(dst),
      "l"(map), "r"(x), "r"(y), "r"(bar)
      : "memory");
}
// K-major operand descriptor for a 128-byte-swizzled tile ([row][128 B], 8-row groups 1024 B apart)
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t saddr) {
  return static_cast<uint64_t>((saddr >> 4) & 0x3FFFu) | (static_cast<uint64_t>(1) << 16) |
         (static_cast<uint64_t>(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}

// A tile: its row pair, first token and the tokens it multiplies (a multiple of 32; the ragged token tile has fewer).
struct PTile {
  int pair, tok0, n;
};
__device__ __forceinline__ PTile tile_of(const PrefillParams& p, int tile) {
  const int nfull = p.pairs * p.full_tt;
  PTile t;
  if (tile < nfull) {  // token tiles of one row pair are neighbours: its weights stay in L2
    t.pair = tile / p.full_tt;
    t.tok0 = (tile - t.pair * p.full_tt) * p.tn;
    t.n = p.tn;
  } else {
    t.pair = tile - nfull;
    t.tok0 = p.full_tt * p.tn;
    t.n = (p.M - t.tok0 + 31) & ~31;
  }
  return t;
}

__global__ void __launch_bounds__(kPWarps * 32, 1) k_prefill(const __grid_constant__ PrefillParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int xbytes = p.tn * 128;  // one activation stage: two swizzled tiles of TN / 2 tokens x 64 k
  uint8_t* xbuf = smem;          // 128-byte-swizzled TMA tiles start on 1024-byte boundaries
  uint8_t* cbuf = xbuf + kPSteps * xbytes;  // [TN tokens][128 rows] bf16: the finished tile on its way out
  uint8_t* ring = cbuf + p.tn * (kTileRows * 2);
  uint64_t* bars = reinterpret_cast<uint64_t*>(ring + p.wdepth * kTileGroupBytes);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + kPBars);

  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const uint32_t rank = cluster_rank(), leader = rank & ~1u;
  const int half = static_cast<int>(rank & 1u), split = static_cast<int>(rank >> 1);
  const int WD = p.wdepth, S = p.splits;
  const int na = a_slots(p.tn);
  const uint32_t ring_a = smem_u32(ring), xbuf_a = smem_u32(xbuf);
  const uint32_t wfull_a = smem_u32(bars);               // [WD] weights of a group landed
  const uint32_t wempty_a = wfull_a + kPMaxWD * 8;       // [WD] read by the 4 dequant warps
  const uint32_t done_a = wempty_a + kPMaxWD * 8;        // [kPDone] group j % 8 multiplied (both CTAs get the commit)
  const uint32_t dfull_a = done_a + kPDone * 8;          // accumulator complete (both CTAs)
  const uint32_t afull_a = dfull_a + 8;                  // [na] leader: a group's A operand written (4 warps of each CTA)
  const uint32_t xfull_a = afull_a + kPMaxA * 8;         // [kPSteps] leader: both CTAs' activations of a group landed
  const uint32_t dempty_a = xfull_a + kPSteps * 8;       // leader: accumulator read out (the epilogue warps of both CTAs)

  if (tid == 0) {
    for (int i = 0; i < kPMaxWD; ++i) {
      mbar_init(wfull_a + i * 8, 1);
      mbar_init(wempty_a + i * 8, 4);
    }
    for (int i = 0; i < kPDone; ++i) mbar_init(done_a + i * 8, 1);
    for (int i = 0; i < kPSteps; ++i) mbar_init(xfull_a + i * 8, 1);
    for (int i = 0; i < kPMaxA; ++i) mbar_init(afull_a + i * 8, 8);
    mbar_init(dfull_a, 1);
    mbar_init(dempty_a, 2 * EW);
    fence_mbar_init();
  }
  if (warp == kWIssue) tmem_alloc_pair(smem_u32(tmem_slot), kPTmemCols);
  tc_fence_before();
  __syncthreads();
  cluster_sync();  // the other CTAs' barriers exist from here on
  // The next launch's CTAs may take over each SM as this one's leave it: set-up, first weights and their expansion then run
  // under the rest of this launch. Its activations and everything behind them wait for this launch's end (griddepcontrol.wait).
  pdl_launch_dependents();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t tmem_a = tmem + (p.tn <= 128 ? 128 : 256);

  const int cluster = blockIdx.x / (2 * S), nclusters = gridDim.x / (2 * S);
  const int g0 = p.G * split / S, g1 = p.G * (split + 1) / S;  // this split's k groups (S <= G)
  bool dead = false;

  if (warp == kWWeights) {
    // ================================================================ weight producer
    if (lane == 0) {
      int st = 0;
      uint32_t ph = 1;
      for (int tile = cluster; !dead && tile < p.tiles; tile += nclusters) {
        const int rt = min(2 * tile_of(p, tile).pair + half, p.row_tiles - 1);
        const uint8_t* src = p.stream + (static_cast<size_t>(rt) * p.G + g0) * kTileGroupBytes;
        for (int g = g0; g < g1; ++g, src += kTileGroupBytes) {
          if (!mbar_wait_bounded_relaxed(wempty_a + st * 8, ph, kPSpin)) {
            atomicExch(p.status, W4A16_ETIMEOUT);
            dead = true;
            break;
          }
          mbar_expect_tx(wfull_a + st * 8, kTileGroupBytes);
          bulk_g2s(ring_a + st * kTileGroupBytes, src, kTileGroupBytes, wfull_a + st * 8);
          if (++st == WD) {
            st = 0;
            ph ^= 1;
          }
        }
      }
      if (dead) {  // the copies in flight still have to land
        for (int i = 0; i < WD; ++i) mbar_wait_bounded_relaxed(wfull_a + i * 8, i < st ? ph ^ 1u : ph, 1u << 10);
      }
    }
  } else if (warp == kWIssue) {
    // ================================================================ MMA issuer (leader CTA only)
    // The whole warp walks (so that the operands stay in uniform registers), one elected lane issues.
    if (half == 0) {
      const uint16_t both = static_cast<uint16_t>(3u << rank);
      const uint64_t desc0 = umma_desc_sw128(xbuf_a);
      const uint32_t x16 = static_cast<uint32_t>(xbytes) >> 4;
      uint32_t j = 0, aph = 0, dph = 1;
      int a = 0;
      for (int tile = cluster; !dead && tile < p.tiles; tile += nclusters, dph ^= 1) {
        const uint32_t idesc = umma_idesc_bf16(kPRows, tile_of(p, tile).n);
        if (!warp_agrees(mbar_wait_bounded(dempty_a, dph, kPSpin))) dead = true;  // (passes on the first tile)
        for (int g = g0; !dead && g < g1; ++g, ++j) {
          const uint32_t st = j & (kPSteps - 1);
          if (!warp_waits(xfull_a + st * 8, (j / kPSteps) & 1u, afull_a + a * 8, aph, kPSpin)) {
            dead = true;
            break;
          }
          tc_fence_after();
          // B operand of the group: two swizzled tiles of 128-byte rows, one per token; a 16-k slab is 32 bytes
          // further along them
          const uint64_t b0 = desc0 + st * x16, b1 = b0 + (x16 >> 1);
          const uint32_t at = tmem_a + a * 64;
          if (elect_one()) {
#pragma unroll
            for (int s = 0; s < 8; ++s)
              umma_bf16_ts_pair(tmem, at + s * 8, (s < 4 ? b0 : b1) + 2 * (s & 3), idesc, s > 0 || g > g0);
            umma_commit_pair(done_a + (j & (kPDone - 1)) * 8, both);
            if (g == g1 - 1) umma_commit_pair(dfull_a, both);
          }
          __syncwarp();
          if (++a == na) {
            a = 0;
            aph ^= 1;
          }
        }
      }
      if (dead && lane == 0) atomicExch(p.status, W4A16_ETIMEOUT);
    }
  } else if (warp == kWActs) {
    // ================================================================ activation producer
    // Two tiled TMA loads per k group (64 k each) into this CTA's half of the token tile; rows past M are zero-filled. The
    // leader's barrier expects both CTAs' bytes.
    if (lane == 0) {
      const uint32_t xfull_l = map_to_rank(xfull_a, leader);
      pdl_wait();  // the previous kernel produced the activations (the weights never depend on it)
      uint32_t j = 0;
      for (int tile = cluster; !dead && tile < p.tiles; tile += nclusters) {
        const PTile t = tile_of(p, tile);
        const int y = t.tok0 + half * (t.n >> 1);
        for (int g = g0; g < g1; ++g, ++j) {
          const uint32_t st = j & (kPSteps - 1);
          const uint32_t jd = j - kPSteps;
          if (j >= kPSteps && !mbar_wait_bounded_relaxed(done_a + (jd & (kPDone - 1)) * 8, (jd / kPDone) & 1u, kPSpin)) {
            atomicExch(p.status, W4A16_ETIMEOUT);
            dead = true;
            break;
          }
          if (half == 0) mbar_expect_tx(xfull_a + st * 8, 2 * xbytes);
          tma_load_pair(xbuf_a + st * xbytes, &p.amap, g * kGroup, y, xfull_l + st * 8);
          tma_load_pair(xbuf_a + st * xbytes + (xbytes >> 1), &p.amap, g * kGroup + 64, y, xfull_l + st * 8);
        }
      }
      if (dead && half == 0) {
        for (uint32_t i = j < kPSteps ? 0 : j - kPSteps; i < j; ++i)
          mbar_wait_bounded_relaxed(xfull_a + (i & (kPSteps - 1)) * 8, (i / kPSteps) & 1u, 1u << 10);
      }
    }
  } else if (warp < PW) {
    // ================================================================ dequant warps
    // The walk over tiles does not matter here: the groups come in the order of the weight ring.
    // Four teams of four warps (one output row per thread) take the groups in turn: one group's waits, shared-memory loads and
    // tensor-memory stores run beside the others' arithmetic. (The weight ring's depth is a multiple of four and the ring of
    // "group multiplied" barriers has eight, so a barrier's consecutive phases belong to one team; a parity wait could
    // not tell them apart otherwise.)
    // A team of eight warps with half a row each paid every wait, vote and arrival twice: 34816 x 5120 at M = 17 / 77 31.8 / 36.0 us
    // with two teams of eight, 29.6 / 34.7 with four of four (M = 777, four layers of a block: 546 and 533).
    const int q = warp & 3, team = warp >> 2;
    const int row = q * 32 + lane;
    const uint32_t a_t = tmem_a + (static_cast<uint32_t>(q * 32) << 16);
    const uint32_t afull_l = map_to_rank(afull_a, leader);
    const int ntiles = cluster < p.tiles ? (p.tiles - 1 - cluster) / nclusters + 1 : 0;
    const uint32_t ngroups = static_cast<uint32_t>(ntiles) * static_cast<uint32_t>(g1 - g0);
    const uint32_t off_e = weight_slot(row, 0) * 16, off_o = kChunkBytes + weight_slot(row, 1) * 16;  // even and odd 32-k chunks
    int st = team, a = team;  // weight stage and A slot
    uint32_t wph = 0;
    for (uint32_t j = team; j < ngroups; j += kPTeams) {
      const bool landed = mbar_wait_bounded(wfull_a + st * 8, wph, kPSpin);
      const uint8_t* blk = ring + st * kTileGroupBytes;
      const uint4 w[4] = {*reinterpret_cast<const uint4*>(blk + off_e), *reinterpret_cast<const uint4*>(blk + off_o),
                          *reinterpret_cast<const uint4*>(blk + off_e + 2 * kChunkBytes),
                          *reinterpret_cast<const uint4*>(blk + off_o + 2 * kChunkBytes)};
      const uint32_t zp = blk[kTgZpOff + row];
      const uint32_t sc = reinterpret_cast<const uint16_t*>(blk + kTgScaleOff)[row];
      const uint32_t zpair = __byte_perm(zp, 0x43434343u, 0x4040);  // bf16 pair (128+zp, 128+zp)
      const uint32_t spair = sc | (sc << 16);
      // Nibbles 0 and 4 of a word become (128 + q) - (128 + zp) by one OR and a subtraction. Nibbles 1 and 5 are left where they
      // are: as a bf16 pair w & 0x00F000F0 is q 2^-129 (subnormals, and the first normal binade goes on where they end), so
      // one packed FMA makes (q - zp) / 4 of it, exactly, and 4 s is exact too: the same product, rounded once. The ALU pipe
      // (shifts and LOP3) is the busiest: 80 of its instructions per row and group instead of 112. Four layers of a block at M = 30 /
      // 77: 77.7 / 85.0 us with a shift per nibble position, 76.5 / 83.8 with this (74.1 / 81.7 without the test for large scales).
      const uint32_t zquarter = fma_bf16x2(zpair, 0xBE80BE80u, 0x42004200u);  // -zp / 4 = 32 - (128 + zp) / 4
      const uint32_t s4 = mul_bf16x2(spair, 0x40804080u);
      auto expand = [&](const uint4& c, uint32_t(&v)[16]) {
        const uint32_t cw[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint32_t w8 = cw[i] >> 8;
          v[4 * i] = mul_bf16x2(sub_bf16x2((cw[i] & kNibMaskP) | kMagicP, zpair), spair);
          v[4 * i + 1] = mul_bf16x2(fma_bf16x2(cw[i] & 0x00F000F0u, 0x7F007F00u, zquarter), s4);
          v[4 * i + 2] = mul_bf16x2(sub_bf16x2((w8 & kNibMaskP) | kMagicP, zpair), spair);
          v[4 * i + 3] = mul_bf16x2(fma_bf16x2(w8 & 0x00F000F0u, 0x7F007F00u, zquarter), s4);
        }
      };
      // ... unless 4 s overflows, from 2^126 on
      auto expand_large = [&](const uint4& c, uint32_t(&v)[16]) {
        const uint32_t cw[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int pp = 0; pp < 4; ++pp)
            v[4 * i + pp] = mul_bf16x2(sub_bf16x2(((cw[i] >> (4 * pp)) & kNibMaskP) | kMagicP, zpair), spair);
      };
      uint32_t v0[16], v1[16];
      expand(w[0], v0);
      expand(w[1], v1);
      bool large = false;
      if (!warp_agrees(landed && (sc & 0x7FFFu) - 0x7E80u >= 0x100u)) {
        if (!warp_agrees(landed)) {
          dead = true;
          break;
        }
        large = true;
        expand_large(w[0], v0);
        expand_large(w[1], v1);
      }
      // The second half of the row is in registers but used only below: a vote orders no memory accesses, __syncwarp does, so
      // that the next bulk copy into the stage cannot pass another lane's loads.
      __syncwarp();
      if (lane == 0) mbar_arrive(wempty_a + st * 8);
      // only now the wait for the A slot: the MMAs that read it last, na groups ago, must have completed
      const uint32_t jd = j - na;
      if (!warp_agrees(j < static_cast<uint32_t>(na) ||
                       mbar_wait_bounded(done_a + (jd & (kPDone - 1)) * 8, (jd / kPDone) & 1u, kPSpin))) {
        dead = true;
        break;
      }
      tc_fence_after();
      tmem_st16(a_t + a * 64, v0);
      tmem_st16(a_t + a * 64 + 16, v1);
      if (large) {
        expand_large(w[2], v0);
        expand_large(w[3], v1);
      } else {
        expand(w[2], v0);
        expand(w[3], v1);
      }
      tmem_st16(a_t + a * 64 + 32, v0);
      tmem_st16(a_t + a * 64 + 48, v1);
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(afull_l + a * 8);
      if ((a += kPTeams) >= na) a -= na;
      if ((st += kPTeams) >= WD) {
        st -= WD;
        wph ^= 1;
      }
    }
    if (dead && lane == 0) atomicExch(p.status, W4A16_ETIMEOUT);
  } else if (S == 1) {
    // ================================================================ epilogue warps
    // The next tile's MMAs wait for the accumulator, so it is read out into shared memory (as bf16) and handed back;
    // the stores to C, 256 bytes per token, run beside the next tile's main loop.
    const int q = warp & 3, eh = (warp - kWEpi0) >> 2, et = tid - kWEpi0 * 32;
    const uint32_t lane_t = tmem + (static_cast<uint32_t>(q * 32) << 16);
    const uint32_t dempty_l = map_to_rank(dempty_a, leader);
    uint32_t dph = 0;
    for (int tile = cluster; tile < p.tiles; tile += nclusters, dph ^= 1) {
      const PTile t = tile_of(p, tile);
      uint16_t* cs = reinterpret_cast<uint16_t*>(cbuf);
      if (!dead && !warp_agrees(mbar_wait_bounded_relaxed(dfull_a, dph, kPSpin))) {
        dead = true;
        if (lane == 0) atomicExch(p.status, W4A16_ETIMEOUT);
      }
      if (!dead) {
        tc_fence_after();
#pragma unroll 2
        for (int c = eh * 16; c < t.n; c += EW / 4 * 16) {
          float v[16];
          tmem_ld<16>(lane_t + c, v);
          tmem_wait_ld();
#pragma unroll
          for (int i = 0; i < 16; ++i) cs[(c + i) * kTileRows + q * 32 + lane] = float_to_bf16_bits(v[i]);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(dempty_l);
      }
      named_bar_sync(1, EW * 32);  // every epilogue warp comes here for every tile, dead or not
      const int r0 = (2 * t.pair + half) * kTileRows;
      const int rows = min(kTileRows, p.N - r0);                     // (<= 0: an odd last row tile's second half)
      const int toks = dead ? 0 : min(t.n, p.M - t.tok0);
      if (p.wide) {
        const int rl = (et & 15) * 8;  // eight rows of one token per thread
        if (rl < rows) {
          for (int c = et >> 4; c < toks; c += EW * 2) {
            const uint4 v = *reinterpret_cast<const uint4*>(cs + c * kTileRows + rl);
            const size_t o = static_cast<size_t>(t.tok0 + c) * p.ldc + p.col0 + r0 + rl;
            *reinterpret_cast<uint4*>(p.C + o) = v;
            for (int pq = 0; pq < p.npeers; ++pq) *reinterpret_cast<uint4*>(p.C_peers[pq] + o) = v;  // fused all-gather over NVLink
          }
        }
      } else {
        for (int i = et; i < toks * kTileRows; i += EW * 32) {
          const int rl = i & (kTileRows - 1);
          if (rl < rows) {
            const size_t o = static_cast<size_t>(t.tok0 + i / kTileRows) * p.ldc + p.col0 + r0 + rl;
            p.C[o] = cs[i];
            for (int pq = 0; pq < p.npeers; ++pq) p.C_peers[pq][o] = cs[i];
          }
        }
      }
      named_bar_sync(1, EW * 32);  // the next tile overwrites the staged one
    }
  }

  if (S > 1) {
    // ================================================================ split K: one tile per cluster
    // Every split's fp32 tile goes to its own shared memory (the activation stages: all MMAs have read them, and
    // [TN tokens][128 rows] floats are exactly their size), then split s adds up and stores the s-th share
    // of the tokens, reading the others' tiles through the cluster.
    const PTile t = tile_of(p, cluster);
    if (warp >= kWEpi0 && warp < kWEpi0 + EW) {
      const int q = warp & 3;
      const uint32_t lane_t = tmem + (static_cast<uint32_t>(q * 32) << 16);
      if (warp_agrees(mbar_wait_bounded(dfull_a, 0, kPSpin))) {
        tc_fence_after();
        float* tile_s = reinterpret_cast<float*>(xbuf) + q * 32 + lane;
#pragma unroll 1
        for (int c = ((warp - kWEpi0) >> 2) * 16; c < t.n; c += EW / 4 * 16) {
          float v[16];
          tmem_ld<16>(lane_t + c, v);
          tmem_wait_ld();
#pragma unroll
          for (int i = 0; i < 16; ++i) tile_s[(c + i) * kTileRows] = v[i];
        }
      } else if (lane == 0) {
        atomicExch(p.status, W4A16_ETIMEOUT);
      }
    }
    __syncwarp();
    cluster_sync();
    if (warp < PW + EW) {
      // Four rows of a token per thread: 16-byte loads from every split's tile, 256 contiguous bytes of C per warp. (One row per
      // thread, 4-byte loads and 64-byte runs of C took 1.6 us of a 5120 x 6144 launch at M = 77. The four layers of a block at M = 77,
      // three of which split: 85.1 -> 83.8 us, at M = 40 80.7 -> 79.9.)
      const int c0 = t.n * split / S, n4 = (t.n * (split + 1) / S - c0) * (kTileRows / 4);
      const int r0 = (2 * t.pair + half) * kTileRows;
      uint32_t src[kPMaxSplit];
#pragma unroll
      for (int s = 0; s < kPMaxSplit; ++s)
        src[s] = map_to_rank(xbuf_a, static_cast<uint32_t>(2 * min(s, S - 1) + half)) + c0 * (kTileRows * 4);
#pragma unroll 2
      for (int i = tid; i < n4; i += (PW + EW) * 32) {
        const int r = r0 + 4 * (i & (kTileRows / 4 - 1)), tok = t.tok0 + c0 + i / (kTileRows / 4);
        float4 part[kPMaxSplit];
#pragma unroll
        for (int s = 0; s < kPMaxSplit; ++s)
          if (s < S) part[s] = ld_cluster_f32x4(src[s] + i * 16);
        float4 acc = part[0];
#pragma unroll
        for (int s = 1; s < kPMaxSplit; ++s)
          if (s < S) {
            acc.x += part[s].x;
            acc.y += part[s].y;
            acc.z += part[s].z;
            acc.w += part[s].w;
          }
        if (r < p.N && tok < p.M) {  // (N is a multiple of 16)
          const size_t o = static_cast<size_t>(tok) * p.ldc + p.col0 + r;
          const uint2 v = make_uint2(float_to_bf16_bits(acc.x) | (static_cast<uint32_t>(float_to_bf16_bits(acc.y)) << 16),
                                     float_to_bf16_bits(acc.z) | (static_cast<uint32_t>(float_to_bf16_bits(acc.w)) << 16));
          auto store = [&](uint16_t* c) {
            if (p.wide) {
              *reinterpret_cast<uint2*>(c) = v;
            } else {
              c[0] = static_cast<uint16_t>(v.x);
              c[1] = static_cast<uint16_t>(v.x >> 16);
              c[2] = static_cast<uint16_t>(v.y);
              c[3] = static_cast<uint16_t>(v.y >> 16);
            }
          };
          store(p.C + o);
          for (int pq = 0; pq < p.npeers; ++pq) store(p.C_peers[pq] + o);
        }
      }
    }
  }

  // Nobody leaves while the other CTAs of the cluster may still reach its barriers, shared or tensor memory.
  tc_fence_before();
  __syncwarp();
  cluster_sync();
  if (warp == kWIssue) {
    tc_fence_after();
    tmem_dealloc_pair(tmem, kPTmemCols);
  }
  // every store of this CTA was issued before the barrier above: its share of the launch's completion signal
  if (p.comm_local && tid == 0) signal_cta_done(p.comm_local, p.comm_peers, p.comm_n, p.comm_rank);
}

// ------------------------------------------------------------------ the plan of a launch
struct PrefillPlan {
  int tn = 0, splits = 1, full_tt = 0, tiles = 0, clusters = 0, wdepth = 0, smem = 0;
};

int prefill_smem(int tn, int wdepth) {
  return 1024 + kPSteps * tn * 128 + tn * kTileRows * 2 + wdepth * kTileGroupBytes + kPBars * 8 + 16;
}

// Tokens per tile and K splits. A cluster's time for a tile is its k groups times the slower of the tensor cores
// (4 TN cycles per group for a pair) and the expansion of the weights (kExpand cycles per group), plus
// what is paid once per tile (pipeline fill, read-out of the accumulator, the exchange of split K). Tiles go to
// the clusters in turn, dearest first, so cluster 0 has the longest list: its total is what is minimised.
// The constants rank the shapes, they do not predict times: a group of a short prompt takes about one and a half times kExpand (see
// above). Against every other (TN, S), on 22 shapes of 1024..34816 rows, 4096..17408 columns and 17..1500 tokens: the choice was the
// fastest on 17. 5120 x 17408 at M = 24: 32 tokens and three splits 20.1 us, two 25.7, one 45.0; 6144 x 5120 at M = 100: two
// splits 13.2, one 15.7; 34816 x 5120 at M = 520: 192 tokens 141, 224 149, 160 161, 128 182. Where kExpand misleads it, tiles
// come out too narrow: 12288 x 4096 at M = 200 96 tokens 30.7 us, 224 23.2; 8192 x 5120 at M = 777 96 tokens 69.1, 224 55.1; 34816 x 5120
// at M = 1024 128 tokens 285, 256 271; 1024 x 4096 at M = 64 32 tokens in four splits 6.6, 64 tokens 5.8. Too wide: 34816 x 5120 at M = 777
// 224 tokens 208, 160 203.
// `only` > 0 asks for that number of splits. The choice goes by what a B200 of 148 SMs runs (index S: clusters of 2 S CTAs
// at once, as cudaOccupancyMaxActiveClusters answers on two of them), not by what this device's GPCs happen to fit, so that a
// row has the same bits on every GPU; the device only rules out clusters it cannot run at all and sizes the grid.
PrefillPlan plan_prefill(int M, int pairs, int G, const int* device_clusters, int smem_optin, int only) {
  constexpr int kClusters[kPMaxSplit + 1] = {0, 74, 33, 22, 15};
  constexpr int kExpand = 420, kFill = 2500, kReduce = 4000;
  PrefillPlan best;
  long long best_cost = -1;
  for (int S = 1; S <= kPMaxSplit && S <= G; ++S) {
    const int slots = kClusters[S];
    if (device_clusters[S] < 1 || (only > 0 && S != only)) continue;
    for (int tn = 32; tn <= kPMaxTN; tn += 32) {
      const int full = M / tn, rest = M - full * tn;
      if (full == 0 && tn - 32 >= rest) break;  // one token tile: the smallest that holds M
      const long long nfull = static_cast<long long>(pairs) * full, tiles = nfull + (rest ? pairs : 0);
      if (S > 1 && tiles > slots) continue;     // split clusters take one tile each
      const int groups = (G + S - 1) / S;
      auto cost = [&](int n) {
        const long long loop = static_cast<long long>(groups) * (4 * n > kExpand ? 4 * n : kExpand);
        return loop + (S > 1 ? kFill + kReduce : kFill / 2);
      };
      const long long cf = cost(tn), cr = cost((rest + 31) & ~31);
      const long long wf = (nfull + slots - 1) / slots, wa = (tiles + slots - 1) / slots;
      const long long total = wf * cf + (wa - wf) * cr;
      if (best_cost < 0 || total < best_cost) {
        best_cost = total;
        best.tn = tn;
        best.splits = S;
        best.full_tt = full;
        best.tiles = static_cast<int>(tiles);
        best.clusters = static_cast<int>(S > 1 || tiles < device_clusters[S] ? tiles : device_clusters[S]);
      }
    }
  }
  // A multiple of the teams: tiles of 224 tokens keep four stages of the six that would fit, of 128 twelve of fourteen. Two teams and six
  // (fourteen) stages -> four teams and four (twelve), in us: 34816 x 5120 at M = 200 55.8 -> 55.4, 16384 x 5120 at M = 210 28.48 -> 28.43, 5120 x
  // 17408 at M = 209 35.3 -> 34.8; at 128 tokens 16384 x 5120 at M = 112 20.0 -> 19.1, 34816 x 5120 at M = 128 39.4 -> 37.7.
  best.wdepth = kPMaxWD;
  while (best.wdepth > kPTeams && prefill_smem(best.tn, best.wdepth) > smem_optin) best.wdepth -= kPTeams;
  best.smem = prefill_smem(best.tn, best.wdepth);
  return best;
}

}  // namespace
}  // namespace w4a16

using namespace w4a16;

extern "C" {

int w4a16_workspace_alloc(w4a16_workspace_t* ws, size_t bytes) {
  W4_REQUIRE(ws != nullptr, "workspace_alloc: null struct");
  memset(ws, 0, sizeof *ws);
  // The fused kernel needs no dequantised tile; keep a small valid allocation because the
  // reference's callers free `wbuf` themselves (src/model/model.cu:440-441).
  (void)bytes;
  void* p = nullptr;
  W4_CUDA(cudaMalloc(&p, 4096));
  ws->wbuf = static_cast<uint16_t*>(p);
  ws->bytes = 4096;
  return W4A16_OK;
}

int w4a16_workspace_free(w4a16_workspace_t* ws) {
  W4_REQUIRE(ws != nullptr, "workspace_free: null struct");
  cudaFree(ws->wbuf);
  memset(ws, 0, sizeof *ws);
  return W4A16_OK;
}

namespace {
void cluster_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* at, int splits, int clusters, int smem) {
  cfg.gridDim = dim3(2 * splits * clusters);
  cfg.blockDim = dim3(kPWarps * 32);
  cfg.dynamicSmemBytes = smem;
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 2 * splits;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
}

// How many clusters of 2 S CTAs (one CTA per SM) the device runs at once, index S; asked for once per device.
// The kernel's shared-memory attribute is set on the way. Returns nullptr (and sets the error) on failure.
const int* cluster_slots(int dev, const DeviceInfo* di) {
  struct Slots {
    bool ready = false;
    int n[kPMaxSplit + 1] = {};
  };
  static std::mutex mu;
  static Slots all[64];
  std::lock_guard<std::mutex> lk(mu);
  Slots& s = all[dev & 63];
  if (!s.ready) {
    cudaError_t e = cudaFuncSetAttribute(k_prefill, cudaFuncAttributeMaxDynamicSharedMemorySize, di->smem_optin);
    for (int S = 1; S <= kPMaxSplit && e == cudaSuccess; ++S) {
      cudaLaunchConfig_t cfg = {};
      cudaLaunchAttribute at[1];
      cluster_config(cfg, at, S, 1, prefill_smem(kPMaxTN, kPTeams));
      e = cudaOccupancyMaxActiveClusters(&s.n[S], k_prefill, &cfg);
    }
    if (e != cudaSuccess || s.n[1] < 1) {
      fail(W4A16_ECUDA, "gemm_prefill: the device runs no CTA pair of the kernel (%s)", cudaGetErrorString(e));
      return nullptr;
    }
    s.ready = true;
  }
  return s.n;
}

// The current device's plan for M tokens through `row_tiles` row tiles and G k groups of a layer of `layer_tiles` row
// tiles. A shard is split as the whole layer would be, so that a row has the same bits sharded and unsharded; as its
// tiles are fewer, they always fit the clusters that the layer's would. (What the shard's own choice would save is left.)
int current_plan(PrefillPlan& plan, int M, int row_tiles, int layer_tiles, int G) {
  const DeviceInfo* di = device_info();
  if (!di) return W4A16_ECUDA;
  const int* slots = cluster_slots(di->device, di);
  if (!slots) return W4A16_ECUDA;
  plan = plan_prefill(M, (layer_tiles + 1) / 2, G, slots, di->smem_optin, 0);
  if (row_tiles < layer_tiles && plan.tn > 0)
    plan = plan_prefill(M, (row_tiles + 1) / 2, G, slots, di->smem_optin, plan.splits);
  W4_REQUIRE(plan.tn > 0, "gemm_prefill: no launch shape for M = %d, %d row tiles x %d k groups", M, row_tiles, G);
  return W4A16_OK;
}

int launch_prefill(PrefillParams& p, uint16_t* C, const w4a16_weights_t* w, const uint16_t* A, int M, w4a16_workspace_t* ws,
                   void* stream) {
  if (int rc = check_weights(w)) return rc;
  W4_REQUIRE(C != nullptr && A != nullptr, "gemm_prefill: null matrix");
  W4_REQUIRE((reinterpret_cast<uintptr_t>(A) & 15) == 0, "gemm_prefill: A not 16-byte aligned");
  W4_REQUIRE(M >= 1, "gemm_prefill: M = %d", M);
  W4_REQUIRE(ws != nullptr, "gemm_prefill: null workspace");
  const DeviceInfo* di = device_info();
  if (!di) return W4A16_ECUDA;
  p.stream = reinterpret_cast<const uint8_t*>(w->qweight);
  p.C = C;
  p.M = M;
  p.N = w->out_f;
  p.K = w->in_f;
  p.G = w->num_groups;
  p.row_tiles = (w->out_f + kTileRows - 1) / kTileRows;
  p.pairs = (p.row_tiles + 1) / 2;
  PrefillPlan plan;
  const int layer_tiles = static_cast<int>((p.ldc + kTileRows - 1) / kTileRows);
  if (int rc = current_plan(plan, M, p.row_tiles, layer_tiles, p.G)) return rc;
  p.tn = plan.tn;
  p.splits = plan.splits;
  p.wdepth = plan.wdepth;
  p.full_tt = plan.full_tt;
  p.tiles = plan.tiles;
  p.status = di->status;
  p.wide = (reinterpret_cast<uintptr_t>(C) & 15) == 0 && p.ldc % 8 == 0 && p.col0 % 8 == 0;
  for (int q = 0; q < p.npeers; ++q)
    if (reinterpret_cast<uintptr_t>(p.C_peers[q]) & 15) p.wide = 0;
  {
    // driver entry point for the tensor-map encoder (no link-time dependency on libcuda)
    typedef CUresult (*EncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                 const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static EncodeFn encode = nullptr;
    if (!encode) {
      void* fn = nullptr;
      cudaDriverEntryPointQueryResult qres;
      W4_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres));
      W4_REQUIRE(fn != nullptr && qres == cudaDriverEntryPointSuccess, "gemm_prefill: cuTensorMapEncodeTiled unavailable");
      encode = reinterpret_cast<EncodeFn>(fn);
    }
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(w->in_f), static_cast<cuuint64_t>(M)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(w->in_f) * 2};
    const cuuint32_t box[2] = {64, static_cast<cuuint32_t>(plan.tn / 2)};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult cr = encode(&p.amap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<uint16_t*>(A), dims, strides,
                               box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (cr != CUDA_SUCCESS) return fail(W4A16_ECUDA, "gemm_prefill: cuTensorMapEncodeTiled failed (%d)", int(cr));
  }
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[2];
  cluster_config(cfg, at, plan.splits, plan.clusters, plan.smem);
  const bool behind_write = take_weight_write(static_cast<cudaStream_t>(stream));
  if (!behind_write && pdl_enabled()) {
    // (behind a weight write the launch is fully ordered: the weights are read before the wait)
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.numAttrs = 2;
  }
  cfg.stream = static_cast<cudaStream_t>(stream);
  const cudaError_t e = cudaLaunchKernelEx(&cfg, k_prefill, p);
  if (e == cudaSuccess) return W4A16_OK;
  if (behind_write) note_weight_write(static_cast<cudaStream_t>(stream));
  return fail(W4A16_ECUDA, "gemm_prefill: launch: %s", cudaGetErrorString(e));
}
}  // namespace

int w4a16_gemm_prefill(uint16_t* C, const w4a16_weights_t* w, const uint16_t* A, int M, w4a16_workspace_t* ws,
                       void* stream) {
  PrefillParams p = {};
  p.ldc = w ? w->out_f : 0;
  return launch_prefill(p, C, w, A, M, ws, stream);
}

int w4a16_prefill_plan(int M, int out_f, int in_f, int* tokens_per_tile, int* k_splits) {
  W4_REQUIRE(tokens_per_tile != nullptr && k_splits != nullptr, "prefill_plan: null output");
  W4_REQUIRE(M >= 1 && out_f > 0 && out_f % kRowGranule == 0 && in_f > 0 && in_f % kGroup == 0,
             "prefill_plan: M = %d, %d x %d", M, out_f, in_f);
  PrefillPlan plan;
  const int row_tiles = (out_f + kTileRows - 1) / kTileRows;
  if (int rc = current_plan(plan, M, row_tiles, row_tiles, in_f / kGroup)) return rc;
  *tokens_per_tile = plan.tn;
  *k_splits = plan.splits;
  return W4A16_OK;
}

int w4a16_gemm_prefill_sharded(uint16_t* const* C_peers, const w4a16_comm_t* comm, int out_f_total, int row_begin,
                               const w4a16_weights_t* w_shard, const uint16_t* A, int M, w4a16_workspace_t* ws,
                               void* stream) {
  W4_REQUIRE(C_peers != nullptr && comm != nullptr && w_shard != nullptr, "gemm_prefill_sharded: null argument");
  if (comm->nranks < 1 || comm->nranks > 8 || comm->rank < 0 || comm->rank >= comm->nranks)
    return fail(W4A16_ECOMM, "gemm_prefill_sharded: rank %d of %d (1..8 ranks)", comm->rank, comm->nranks);
  if (row_begin < 0 || row_begin % kRowGranule != 0 || row_begin + w_shard->out_f > out_f_total)
    return fail(W4A16_ECOMM, "gemm_prefill_sharded: rows [%d,%d) outside [0,%d)", row_begin, row_begin + w_shard->out_f,
                out_f_total);
  PrefillParams p = {};
  p.ldc = out_f_total;
  p.col0 = row_begin;
  for (int r = 0; r < comm->nranks; ++r) {
    if (C_peers[r] == nullptr || comm->blocks[r] == nullptr)
      return fail(W4A16_ECOMM, "gemm_prefill_sharded: null output or flag block of rank %d", r);
    p.comm_peers[r] = comm->blocks[r];
    if (r != comm->rank) p.C_peers[p.npeers++] = C_peers[r];
  }
  p.comm_local = comm->blocks[comm->rank];
  p.comm_n = comm->nranks;
  p.comm_rank = comm->rank;
  return launch_prefill(p, C_peers[comm->rank], w_shard, A, M, ws, stream);
}

}  // extern "C"
