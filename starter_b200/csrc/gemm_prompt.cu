// Projections of the prompt pass: Y[M,N] = X[M,K] . W[N,K]^T for hundreds to thousands of
// activation rows, on CTA pairs (tcgen05.mma.cta_group::2), with the layer's element-wise work
// as the epilogue (reference: engine/prefill.py:40-52 calls library GEMMs and separate kernels).
//
// A pair of CTAs (a cluster of two, one SM each) owns an output tile of 256 rows x 256 columns:
// each CTA brings in its 128 activation rows and HALF of the tile's weight rows per 64-k step,
// the leader's one MMA thread multiplies over both shared memories, and each CTA's tensor memory
// ends up with its own 128 rows x 256 columns in fp32. What bounds this kernel is operand traffic
// from L2 into shared memory: per 64 k an SM reads 32 KB for 128 x 256 outputs, two thirds of the
// bytes per product of the one-CTA kernel of gemm_tc.cu (weights 128 x rows 256 per SM), which is
// why prompts leave that kernel: 1.4 - 1.5 PFLOP/s against 1.0. O and down, whose 2560 columns are ten such tiles
// only, take tiles of 160 columns where these fill the last wave better (a CTA's 80 weight rows come in one or two
// copies, with a tensor map for each multiple of 16 rows; in five copies of 16 rows they ran at 0.66 PFLOP/s).
//
// The epilogue's thread owns one activation row (tensor-memory lane) and walks the columns, so all of these are thread-local:
//   EPI_F32     fp32 sums                          (before a tensor-parallel all-reduce)
//   EPI_RESID   x = bf16(x + bf16(sum))            (O and down projections, in place)
//   EPI_SWIGLU  act = bf16(bf16(silu(bf16 g)) * bf16 u): the tile's columns are 128 gate columns
//               (the leader's weight half) and the matching 128 up columns (the peer's half)
//   EPI_ROPE    bf16 q|k|v, head norm + RoPE on q and k heads (128 columns each), q to
//               [row][head][128], k and v rows into their pages
// The rounding points are those of the consumers in fused_ops.cu.
//
// Roles per CTA (320 threads): warp 0 producer (one lane), warp 1 MMA issuer (the leader's one
// lane), warps 2-9 epilogue, which drain one of two accumulators while the MMAs fill the other: two
// warps per 32 rows, each for two runs of 64 columns (four warps took as long for head norm + RoPE
// as the MMAs for a tile with K = 2560). What the epilogue reads besides the accumulator is
// requested before it waits for it, or one step ahead.
// The `full` barriers live in the leader: both CTAs' copies complete there (a stage is 2 x its
// bytes); commits release stages and hand over accumulators in both CTAs at once. Every wait is
// bounded as in gemm_tc.cu and reports in the same status word (codes 5-8).
//
// Work split: tiles in raster order (row tiles fastest inside groups of `group`, so that the tiles in
// flight share both operands in L2). Whole waves of one tile per pair come first; what is left over
// - up to two tiles' work per pair - is cut evenly by k steps over all pairs (`split`), since a
// projection with N = 2560 has 40 tiles at 1024 rows and 80 at 2048 for 74 pairs. A pair that ends
// up with a part of a tile stores its fp32 accumulator in the caller's scratch, draws a ticket, and
// the LAST of a tile's pairs adds the parts in k order (its own included, so the sum does not depend
// on who is last), puts the total back into tensor memory and runs the epilogue. Nobody waits. The
// unit of all this is a warp: 32 rows x 2 x 64 columns. A launch that gives up leaves tickets drawn, so
// the prompt pass clears them before each run of layers.
#include "tc.cuh"

int* q_tc_status_addr();

namespace {

constexpr int PG_THREADS = 320;
constexpr int PG_EPI_WARPS = 8;
constexpr int PG_TILE_K = 64;
constexpr int PG_A_BYTES = 128 * PG_TILE_K * 2;            // 16 KB of activations per CTA and stage
constexpr int PG_BN = 256, PG_HALF = 128;                  // columns of a tile, weight rows per CTA
constexpr int PG_NARROW = 160;                             // ... of a narrow tile: weight rows in runs of 16, see prompt_plan
__host__ __device__ constexpr uint32_t pg_stage(int bn) { return PG_A_BYTES + bn / 2 * PG_TILE_K * 2; }
__host__ __device__ constexpr int pg_stages(int bn) { return bn == PG_BN ? 7 : 8; }                     // 224 KB, 208 KB
constexpr size_t pg_smem(int bn) { return 1024 + pg_stages(bn) * pg_stage(bn) + (2 * pg_stages(bn) + 4) * 8 + 16; }
constexpr int PG_MAX_PAIRS = 128;
constexpr int PG_SPLIT_STEPS = 60;                         // what a split costs, in k steps
// scratch: tickets (16 warps per tile, at most two tiles per pair), then two parts per pair
constexpr size_t PG_TICKET_BYTES = PG_MAX_PAIRS * 2 * 16 * 4;
static_assert(PG_TICKET_BYTES == 16384, "stated in qdecode.h");
constexpr size_t PG_PART_FLOATS = 256 * 256;

enum { EPI_F32 = 0, EPI_RESID = 1, EPI_SWIGLU = 2, EPI_ROPE = 3 };

struct PromptShape {
  int M, N, KT;         // rows, output columns (EPI_SWIGLU: inter), k tiles
  int mt, nt;           // tiles along rows (256) and columns (256; EPI_SWIGLU 128 gate + 128 up)
  int wrows;            // weight rows per copy (a power of two that divides every copy's start)
  int group;            // row tiles of a raster group
  int waves;            // tiles that each pair takes whole
  int share;            // k steps of the remaining tiles per pair: whole tiles, or an even split
};

// First row of the 128 that a CTA loads for rows [row0, row0 + 128): the last block is moved up so
// that it holds no rows past M (copies that fill in zeros are slow), and a block that has no rows at
// all loads some others; neither computes anything twice that is stored.
__device__ __forceinline__ int first_row(int row0, int M) { return row0 >= M ? 0 : max(0, min(row0, M - 128)); }

// The pieces of a pair in order: (tile, k steps [k0, k1)).
struct Walk {
  int i, u, u1;
  __device__ __forceinline__ void start(const PromptShape& sh, int pair, int pairs) {
    i = 0;
    const int rest = (sh.mt * sh.nt - sh.waves * pairs) * sh.KT;
    u = min(rest, pair * sh.share);
    u1 = min(rest, u + sh.share);
  }
  __device__ __forceinline__ bool next(const PromptShape& sh, int pair, int pairs, int& t, int& k0, int& k1) {
    if (i < sh.waves) {
      t = pair + i++ * pairs;
      k0 = 0;
      k1 = sh.KT;
      return true;
    }
    if (u >= u1) return false;
    const int rel = u / sh.KT;
    t = sh.waves * pairs + rel;
    k0 = u - rel * sh.KT;
    k1 = min(sh.KT, k0 + u1 - u);
    u += k1 - k0;
    return true;
  }
};

// The tiled weight with boxes of wrows rows; narrow tiles: of 16, 32, .. 80 rows, since a run of 80 weight rows
// crosses at most one boundary of a 128-row block.
template <int BN>
struct WeightMaps { CUtensorMap m[BN == PG_BN ? 1 : BN / 32]; };

struct RopeArgs {
  const bf16* q_gain; const bf16* k_gain; const bf16* cos; const bf16* sin;
  const int32_t* pos; char* kpool; char* vpool; const int32_t* block_table;
  int pages_per_seq, T, nq, nkv;
  float eps;
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// The address, in the cluster's shared window, of the leader's copy of a local address.
__device__ __forceinline__ uint32_t leader_addr(uint32_t addr) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(addr));
  return r;
}
// (not the .aligned form: single lanes of a warp come here from their role's loop)
__device__ __forceinline__ void cluster_sync_all() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
  __syncwarp();
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Copies into this CTA's shared memory that complete on the leader's barrier.
__device__ __forceinline__ void pair_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 "
      "[%0], [%1, {%2, %3}], [%4];"
      ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
__device__ __forceinline__ void pair_load_4d(uint32_t dst, const CUtensorMap* map, int x, int y, int z, int w,
                                             uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 "
      "[%0], [%1, {%2, %3, %4, %5}], [%6];"
      ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(w), "r"(bar) : "memory");
}
__device__ __forceinline__ void pair_mma(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
// One arrival on the barrier at this offset in both CTAs of the pair once the MMAs so far are done.
__device__ __forceinline__ void pair_commit(uint32_t bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
      ::"r"(bar), "h"((uint16_t)3) : "memory");
}
// 2 x 16 columns of this warp's 32 lanes; the wait is part of the statement.
__device__ __forceinline__ void tc_ld16x2(uint32_t a, uint32_t b, float (&v)[16], float (&w)[16]) {
  uint32_t r[16], s[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%32];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%33];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5]), "=r"(s[6]), "=r"(s[7]),
        "=r"(s[8]), "=r"(s[9]), "=r"(s[10]), "=r"(s[11]), "=r"(s[12]), "=r"(s[13]), "=r"(s[14]), "=r"(s[15])
      : "r"(a), "r"(b) : "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) { v[i] = __uint_as_float(r[i]); w[i] = __uint_as_float(s[i]); }
}

__device__ __forceinline__ void tc_st16x2(uint32_t a, uint32_t b, const float (&v)[16], const float (&w)[16]) {
#define Q_R(x, i) "f"(x[i]), "f"(x[i + 1]), "f"(x[i + 2]), "f"(x[i + 3]), "f"(x[i + 4]), "f"(x[i + 5]), "f"(x[i + 6]), "f"(x[i + 7])
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
               ::"r"(a), Q_R(v, 0), Q_R(v, 8) : "memory");
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
               ::"r"(b), Q_R(w, 0), Q_R(w, 8) : "memory");
#undef Q_R
}

// 32 bytes (16 bf16) at a 32-byte boundary: whole sectors, since neighbouring lanes hold other rows.
__device__ __forceinline__ void ld32B(const void* p, uint32_t (&r)[8]) {
  asm volatile("ld.global.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "l"(p));
}
__device__ __forceinline__ void st32B(void* p, const uint32_t (&r)[8]) {
  asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
               ::"l"(p), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
__device__ __forceinline__ void pack16(const float (&v)[16], uint32_t (&r)[8]) {
#pragma unroll
  for (int i = 0; i < 8; ++i) r[i] = pack_bf16(v[2 * i], v[2 * i + 1]);
}
__device__ __forceinline__ void unpack16(const uint32_t (&r)[8], float (&v)[16]) {
#pragma unroll
  for (int i = 0; i < 8; ++i) { v[2 * i] = bf_lo(r[i]); v[2 * i + 1] = bf_hi(r[i]); }
}
// 16 gains, the same for all lanes
__device__ __forceinline__ void ld_gain16(const bf16* p, uint32_t (&r)[8]) {
  const uint4 a = __ldg(reinterpret_cast<const uint4*>(p)), b = __ldg(reinterpret_cast<const uint4*>(p) + 1);
  r[0] = a.x; r[1] = a.y; r[2] = a.z; r[3] = a.w; r[4] = b.x; r[5] = b.y; r[6] = b.z; r[7] = b.w;
}
__device__ __forceinline__ uint32_t mul2(uint32_t a, uint32_t b) {
  const __nv_bfloat162 p = __hmul2_rn(*reinterpret_cast<__nv_bfloat162*>(&a), *reinterpret_cast<__nv_bfloat162*>(&b));
  return *reinterpret_cast<const uint32_t*>(&p);
}

// k / v row of a page: the 32 bytes of dims d..d+15 (d a multiple of 16) are one aligned pair of
// 16-byte chunks whose order depends on the token's parity (chunk index XOR-ed with r & 7).
__device__ __forceinline__ void st_page16(char* row, int r, int d, const uint32_t (&a)[8]) {
  uint32_t b[8];
  const bool swap = r & 1;
#pragma unroll
  for (int i = 0; i < 4; ++i) { b[i] = swap ? a[i + 4] : a[i]; b[i + 4] = swap ? a[i] : a[i + 4]; }
  st32B(row + (((d >> 3) ^ (r & 6)) << 4), b);
}

// Rotary rows of 16 dims and of their partners 64 on.
struct RotRow { uint32_t c0[8], c1[8], s0[8], s1[8]; };
__device__ __forceinline__ void ld_rot(RotRow& r, const bf16* cs, const bf16* sn) {
  ld32B(cs, r.c0);
  ld32B(cs + 64, r.c1);
  ld32B(sn, r.s0);
  ld32B(sn + 64, r.s1);
}

// One 128-column head of one row: `taddr` is the head's first column in tensor memory, `rot` already
// holds the rotary rows of dims 0..15 and 64..79.
__device__ __forceinline__ void rope_head(uint32_t taddr, const RopeArgs& ra, bf16* Q, int m, bool live, int head,
                                          RotRow& rot, const bf16* cs, const bf16* sn, char* krow, char* vrow, int r) {
  const bool is_q = head < ra.nq, is_v = head >= ra.nq + ra.nkv;     // warp-uniform
  const int kh = is_v ? head - ra.nq - ra.nkv : head - ra.nq;
  const size_t hoff = is_q ? 0 : (size_t)kh * (Q_PAGE_TOKENS * 256);
  if (is_v) {
#pragma unroll 1
    for (int d = 0; d < 64; d += 16) {
      float lo[16], hi[16];
      tc_ld16x2(taddr + d, taddr + 64 + d, lo, hi);
      uint32_t a[8], b[8];
      pack16(lo, a);
      pack16(hi, b);
      if (live) {
        st_page16(vrow + hoff, r, d, a);
        st_page16(vrow + hoff, r, 64 + d, b);
      }
    }
    return;
  }
  // The head as bf16 pairs: one pass over tensor memory. The products below are of two bf16 values
  // and rounded to bf16, which the packed multiply does in one instruction.
  uint32_t xl[4][8], xh[4][8];
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float lo[16], hi[16];
    tc_ld16x2(taddr + 16 * i, taddr + 64 + 16 * i, lo, hi);
    pack16(lo, xl[i]);
    pack16(hi, xh[i]);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      ss += bf_lo(xl[i][e]) * bf_lo(xl[i][e]) + bf_hi(xl[i][e]) * bf_hi(xl[i][e]);
      ss += bf_lo(xh[i][e]) * bf_lo(xh[i][e]) + bf_hi(xh[i][e]) * bf_hi(xh[i][e]);
    }
  }
  const float inv = rsqrtf(ss / 128.f + ra.eps);
  const bf16* gain = is_q ? ra.q_gain : ra.k_gain;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int d = 16 * i;
    uint32_t g0[8], g1[8], o[8], p[8];
    ld_gain16(gain + d, g0);
    ld_gain16(gain + 64 + d, g1);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const uint32_t lo = mul2(pack_bf16(bf_lo(xl[i][e]) * inv, bf_hi(xl[i][e]) * inv), g0[e]);
      const uint32_t hi = mul2(pack_bf16(bf_lo(xh[i][e]) * inv, bf_hi(xh[i][e]) * inv), g1[e]);
      const uint32_t a = mul2(lo, rot.c0[e]), b = mul2(hi, rot.s0[e]);
      const uint32_t c = mul2(hi, rot.c1[e]), f = mul2(lo, rot.s1[e]);
      o[e] = pack_bf16(bf_lo(a) - bf_lo(b), bf_hi(a) - bf_hi(b));
      p[e] = pack_bf16(bf_lo(c) + bf_lo(f), bf_hi(c) + bf_hi(f));
    }
    if (i < 3) ld_rot(rot, cs + d + 16, sn + d + 16);
    if (live) {
      if (is_q) {
        bf16* dst = Q + ((size_t)m * ra.nq + head) * 128 + d;
        st32B(dst, o);
        st32B(dst + 64, p);
      } else {
        st_page16(krow + hoff, r, d, o);
        st_page16(krow + hoff, r, 64 + d, p);
      }
    }
  }
}

// A warp's part (32 rows x 64 columns at `ta` and at `tb`) of tile `rel` of the split ones. True: this
// was the tile's last part and tensor memory now holds the sum of all parts, added in k order.
__device__ __forceinline__ bool merge_parts(const PromptShape& sh, unsigned char* scratch, uint32_t ta, uint32_t tb,
                                            int pair, int rel, int warp_of_tile, int lane) {
  const int first = rel * sh.KT / sh.share, last = ((rel + 1) * sh.KT - 1) / sh.share;
  int* ticket = reinterpret_cast<int*>(scratch) + rel * 16 + warp_of_tile;
  float* parts = reinterpret_cast<float*>(scratch + PG_TICKET_BYTES);
  // a pair has at most two parts: the rest of a tile it did not begin, the beginning of its last one;
  // columns 4 j .. 4 j + 3 of run b of a lane are the float4 at ((b * 16 + j) * 32 + lane)
  auto part = [&](int p) {
    return reinterpret_cast<float4*>(parts + (size_t)(2 * p + (p * sh.share > rel * sh.KT ? 0 : 1)) * PG_PART_FLOATS +
                                     warp_of_tile * (32 * 128)) + lane;
  };
  int drawn = 0;
  if (lane == 0) drawn = *reinterpret_cast<volatile int*>(ticket);
  drawn = __shfl_sync(0xffffffffu, drawn, 0);
  if (drawn != last - first) {                    // not known to be the last one: leave the part in memory
    float4* dst = part(pair);
#pragma unroll
    for (int c = 0; c < 64; c += 16) {
      float v[16], w[16];
      tc_ld16x2(ta + c, tb + c, v, w);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        __stcg(dst + (c / 4 + j) * 32, make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]));
        __stcg(dst + (16 + c / 4 + j) * 32, make_float4(w[4 * j], w[4 * j + 1], w[4 * j + 2], w[4 * j + 3]));
      }
    }
    __threadfence();
    __syncwarp();
    if (lane == 0) drawn = atomicAdd(ticket, 1);
    drawn = __shfl_sync(0xffffffffu, drawn, 0);
    if (drawn != last - first) return false;
  }
  __syncwarp();
  __threadfence();
  if (lane == 0) *ticket = 0;                     // ready for the next launch
#pragma unroll 1
  for (int b = 0; b < 2; ++b) {
    // 64 columns at a time: 16 loads of a part are in flight together
    const uint32_t t = b ? tb : ta;
    float v[4][16];
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int e = 0; e < 16; ++e) v[c][e] = 0.f;
#pragma unroll 1
    for (int p = first; p <= last; ++p) {
      if (p == pair) {
#pragma unroll
        for (int c = 0; c < 4; c += 2) {
          float x[16], y[16];
          tc_ld16x2(t + 16 * c, t + 16 * c + 16, x, y);
#pragma unroll
          for (int e = 0; e < 16; ++e) { v[c][e] += x[e]; v[c + 1][e] += y[e]; }
        }
        continue;
      }
      const float4* src = part(p) + b * (16 * 32);
      float4 a[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) a[j] = __ldcg(src + j * 32);
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        float* d = v[j >> 2] + 4 * (j & 3);
        d[0] += a[j].x; d[1] += a[j].y; d[2] += a[j].z; d[3] += a[j].w;
      }
    }
    tc_st16x2(t, t + 16, v[0], v[1]);
    tc_st16x2(t + 32, t + 48, v[2], v[3]);
  }
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
  return true;
}

template <int EPI, int BN>
__global__ void __launch_bounds__(PG_THREADS, 1)
k_gemm_prompt(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ WeightMaps<BN> wmaps,
              void* __restrict__ out, PromptShape sh, const __grid_constant__ RopeArgs ra, unsigned char* scratch, int* status,
              unsigned long long* tl) {
  constexpr int PG_STAGES = pg_stages(BN), HALF = BN / 2;
  constexpr uint32_t PG_STAGE = pg_stage(BN);
  constexpr bool NARROW = BN != PG_BN;
  extern __shared__ unsigned char smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  unsigned char* smem = smem_raw + (base - raw);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + PG_STAGES * PG_STAGE);
  // full[stages] (leader's) | empty[stages] | acc_full[2] | acc_empty[2] (leader's)
  const uint32_t bar_full = smem_u32(bars), bar_empty = bar_full + 8u * PG_STAGES;
  const uint32_t bar_acc_full = bar_empty + 8u * PG_STAGES, bar_acc_empty = bar_acc_full + 16u;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * PG_STAGES + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  tl_begin(tl);
  pdl_launch_dependents();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t rank = cluster_rank();
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;

  if (tid == 0) {
    for (int s = 0; s < PG_STAGES; ++s) {
      mbar_init(bar_full + 8 * s, 1);
      mbar_init(bar_empty + 8 * s, 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(bar_acc_full + 8 * b, 1);
      mbar_init(bar_acc_empty + 8 * b, 2 * PG_EPI_WARPS);   // of both CTAs
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 0 && lane == 0) {
    if (!NARROW) prefetch_map(&wmaps.m[0]);
    prefetch_map(&xmap);
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                                       // the peer's barriers exist
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  // (row tile, column tile) of a tile number
  auto locate = [&](int t, int& mi, int& ni) {
    const int per = sh.group * sh.nt;
    const int g = t / per, in = t - g * per;
    const int rows = min(sh.group, sh.mt - g * sh.group);
    ni = in / rows;
    mi = g * sh.group + in - ni * rows;
  };

  if (warp == 0) {
    // ---------------- producer ----------------
    if (lane == 0) {
      const uint32_t full0 = leader_addr(bar_full);
      const int nload = NARROW ? 0 : PG_HALF / sh.wrows;
      const uint32_t wbytes = (uint32_t)sh.wrows * 128u;
      int st = 0;
      uint32_t parity = 1;                                  // an untouched stage is free
      bool ok = true, waited = false;
      int issued = 0;
      Walk walk;
      walk.start(sh, pair, pairs);
      int t, k0, k1;
      while (ok && walk.next(sh, pair, pairs, t, k0, k1)) {
        int mi, ni;
        locate(t, mi, ni);
        const int row = first_row(mi * 256 + (int)rank * 128, sh.M);
        // first weight row of this CTA's half
        const int n0 = EPI == EPI_SWIGLU ? (int)rank * sh.N + ni * PG_HALF : ni * BN + (int)rank * HALF;
        // narrow: the rows up to the end of their 128-row block, then the rest
        const int run = min(HALF, 128 - (n0 & 127));
        for (int kt = k0; kt < k1; ++kt) {
          if (!mbar_wait(bar_empty + 8 * st, parity, abort_flag)) {
            atomicExch(status, 5);
            *abort_flag = 1;
            ok = false;
            break;
          }
          const uint32_t full = full0 + 8u * st, dst = base + st * PG_STAGE;
          if (rank == 0) mbar_expect_tx(bar_full + 8 * st, 2 * PG_STAGE);
          if (NARROW) {
            pair_load_4d(dst + PG_A_BYTES, &wmaps.m[(run >> 4) - 1], 0, n0 & 127, kt, n0 >> 7, full);
            if (run < HALF)
              pair_load_4d(dst + PG_A_BYTES + run * 128, &wmaps.m[((HALF - run) >> 4) - 1], 0, 0, kt, (n0 >> 7) + 1, full);
          }
          for (int j = 0; j < nload; ++j) {
            const int n = n0 + j * sh.wrows;
            pair_load_4d(dst + PG_A_BYTES + j * wbytes, &wmaps.m[0], 0, n & 127, kt, n >> 7, full);
          }
          if (!waited) {                                    // weights do not depend on the previous kernel
            pdl_wait();
            tl_waited(tl);
            waited = true;
          }
          pair_load_2d(dst, &xmap, kt * PG_TILE_K, row, full);
          ++issued;
          if (++st == PG_STAGES) { st = 0; parity ^= 1u; }
        }
      }
      // Every copy must have landed before the CTAs may leave: the leader waits for the last fill
      // of each stage (both CTAs' bytes), the cluster barrier at the end holds the peer.
      if (rank == 0)
        for (int s = 0; s < PG_STAGES && s < issued; ++s) {
          const int last = (issued - 1 - s) / PG_STAGES;
          if (!mbar_wait_plain(bar_full + 8 * s, last & 1)) atomicExch(status, 8);
        }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (leader) ----------------
    // (the whole warp walks the loop and one elected lane issues, so that descriptors live in uniform
    // registers)
    if (rank == 0) {
      pdl_wait();                                           // as in gemm_tc.cu: the wait limit starts here
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | (16u << 24);
      const uint32_t stage_units = PG_STAGE >> 4;
      const uint64_t desc0 = smem_desc(base);
      auto warp_wait = [&](uint32_t b, uint32_t par) {
        return __all_sync(0xffffffffu, mbar_wait(b, par, abort_flag) ? 1 : 0) != 0;
      };
      int st = 0, seg = 0;
      uint32_t parity = 0;
      bool ok = true;
      Walk walk;
      walk.start(sh, pair, pairs);
      int t, k0, k1;
      for (; ok && walk.next(sh, pair, pairs, t, k0, k1); ++seg) {
        const int buf = seg & 1;
        if (!warp_wait(bar_acc_empty + 8 * buf, ((seg >> 1) & 1) ^ 1)) { ok = false; break; }
        tc_fence_after();
        const uint32_t dacc = tmem_base + (uint32_t)buf * 256u;
        for (int kt = k0; kt < k1; ++kt) {
          if (!warp_wait(bar_full + 8 * st, parity)) { ok = false; break; }
          tc_fence_after();
          const uint64_t a_desc = desc0 + (uint64_t)(st * stage_units);
          const uint64_t b_desc = a_desc + (PG_A_BYTES >> 4);
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < PG_TILE_K / 16; ++k)
              pair_mma(dacc, a_desc + 2u * k, b_desc + 2u * k, idesc, (kt > k0 || k) ? 1u : 0u);
            pair_commit(bar_empty + 8 * st);
          }
          __syncwarp();
          if (++st == PG_STAGES) { st = 0; parity ^= 1u; }
        }
        if (ok && elect_one()) pair_commit(bar_acc_full + 8 * buf);
        __syncwarp();
      }
      if (!ok && lane == 0) {
        atomicExch(status, 6);
        *abort_flag = 1;
      }
    }
  } else {
    // ---------------- epilogue (warps 2..9) ----------------
    pdl_wait();
    const int q = warp & 3, h = (warp - 2) >> 2;
    // the warp's two runs of 64 columns: gate and up columns that belong together, or one head
    const int ca = EPI == EPI_SWIGLU ? 64 * h : HALF * h, cb = EPI == EPI_SWIGLU ? PG_HALF + 64 * h : ca + 64;
    constexpr int RUNS = HALF / 16;                         // runs of 16 columns of a warp (not EPI_SWIGLU)
    const uint32_t acc_empty0 = leader_addr(bar_acc_empty);
    int seg = 0;
    Walk walk;
    walk.start(sh, pair, pairs);
    int t, k0, k1;
    for (; walk.next(sh, pair, pairs, t, k0, k1); ++seg) {
      const int buf = seg & 1;
      int mi, ni;
      locate(t, mi, ni);
      const int row0 = mi * 256 + (int)rank * 128;
      const int m = first_row(row0, sh.M) + q * 32 + lane;
      const bool live = m >= row0 && m < sh.M;
      const int n0 = EPI == EPI_SWIGLU ? ni * PG_HALF + ca : ni * BN + ca;      // output column of run a
      // operands besides the accumulator: requested now, used after the wait
      uint32_t res[EPI == EPI_RESID ? (RUNS + 1) / 2 * 2 : 1][8];
      bf16* x = reinterpret_cast<bf16*>(out) + (size_t)(live ? m : 0) * sh.N + n0;
      if (EPI == EPI_RESID) {
#pragma unroll
        for (int j = 0; j < RUNS; ++j)
          if (n0 + 16 * j < sh.N) ld32B(x + 16 * j, res[j]);
      }
      RotRow rot;
      const bf16 *cs = nullptr, *sn = nullptr;
      char *krow = nullptr, *vrow = nullptr;
      int r = 0;
      if (EPI == EPI_ROPE) {
        const int mm = live ? m : 0;
        const int b = mm / ra.T, pos = ra.pos[0] + mm - b * ra.T;
        const int page = ra.block_table[(size_t)b * ra.pages_per_seq + pos / Q_PAGE_TOKENS];
        r = pos % Q_PAGE_TOKENS;
        const size_t row = (size_t)page * ra.nkv * (Q_PAGE_TOKENS * 256) + (size_t)r * 256;
        krow = ra.kpool + row;
        vrow = ra.vpool + row;
        cs = ra.cos + (size_t)pos * 128;
        sn = ra.sin + (size_t)pos * 128;
        ld_rot(rot, cs, sn);
      }
      const int landed = mbar_wait(bar_acc_full + 8 * buf, (seg >> 1) & 1, abort_flag) ? 1 : 0;
      if (!__all_sync(0xffffffffu, landed)) {
        if (lane == 0) {
          atomicExch(status, 7);
          *abort_flag = 1;
        }
        break;
      }
      tc_fence_after();
      const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)buf * 256u;
      const uint32_t ta = taddr + ca, tb = taddr + cb;
      // (a part of a tile that is not the last one: another pair finishes the tile)
      const bool whole = NARROW || k1 - k0 == sh.KT ||
                         merge_parts(sh, scratch, ta, tb, pair, t - sh.waves * pairs, ((int)rank * 4 + q) * 2 + h, lane);
      if (whole && n0 < sh.N) {
        if (EPI == EPI_F32) {
          float* dst = reinterpret_cast<float*>(out) + (size_t)m * sh.N + n0;
#pragma unroll 2
          for (int c = 0; c < HALF && n0 + c < sh.N; c += 32) {            // N is a multiple of 32
            float v[16], w[16];
            tc_ld16x2(ta + c, ta + c + 16, v, w);
            const bool second = c + 16 < HALF && (!NARROW || n0 + c + 16 < sh.N);
            if (live) {
#pragma unroll
              for (int j = 0; j < 16; j += 8) {
                uint32_t a[8], b[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) { a[e] = __float_as_uint(v[j + e]); b[e] = __float_as_uint(w[j + e]); }
                st32B(dst + c + j, a);
                if (second) st32B(dst + c + 16 + j, b);
              }
            }
          }
        } else if (EPI == EPI_RESID) {
#pragma unroll
          for (int j = 0; j < RUNS; j += 2) {
            if (n0 + 16 * j < sh.N) {
              const bool second = j + 1 < RUNS && (!NARROW || n0 + 16 * j + 16 < sh.N);
              float v[16], w[16], a[16];
              tc_ld16x2(ta + 16 * j, ta + 16 * j + 16, v, w);
              unpack16(res[j], a);
#pragma unroll
              for (int e = 0; e < 16; ++e) v[e] = a[e] + bf16_round(v[e]);
              unpack16(res[j + 1], a);
#pragma unroll
              for (int e = 0; e < 16; ++e) w[e] = a[e] + bf16_round(w[e]);
              uint32_t o0[8], o1[8];
              pack16(v, o0);
              pack16(w, o1);
              if (live) {
                st32B(x + 16 * j, o0);
                if (second) st32B(x + 16 * j + 16, o1);
              }
            }
          }
        } else if (EPI == EPI_SWIGLU) {
          bf16* act = reinterpret_cast<bf16*>(out) + (size_t)m * sh.N + n0;
#pragma unroll 1
          for (int c = 0; c < 64 && n0 + c < sh.N; c += 16) {              // inter is a multiple of 16
            float g[16], u[16];
            uint32_t w[8];
            tc_ld16x2(ta + c, tb + c, g, u);
#pragma unroll
            for (int e = 0; e < 16; ++e) {
              const float gb = bf16_round(g[e]);
              g[e] = bf16_round(gb / (1.0f + expf(-gb))) * bf16_round(u[e]);
            }
            pack16(g, w);
            if (live) st32B(act + c, w);
          }
        } else {
          rope_head(ta, ra, reinterpret_cast<bf16*>(out), m, live, n0 >> 7, rot, cs, sn, krow, vrow, r);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(acc_empty0 + 8 * buf);
    }
  }

  __syncwarp();
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                 // the peer no longer reads this CTA's memory or barriers
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
  }
  tl_end(tl);
}

int pair_count() {
  const int sms = q_sm_count();
  const int pairs = (sms > 0 ? sms : 148) / 2;
  return pairs < PG_MAX_PAIRS ? pairs : PG_MAX_PAIRS;
}

// `N` as in PromptShape; the weight has `wN` rows. Tiles and their split for a shape; `pairs` in: of the device, out: of the launch. False: too many tiles.
bool prompt_plan(int epi, int M, int N, int wN, int K, bool scratch, PromptShape* plan, int* pairs_io, bool* narrow) {
  PromptShape& sh = *plan;
  sh.M = M; sh.N = N;
  // A raster group reads the whole weight once. Where the weight does not stay in L2 from one group to the next,
  // fewer and taller groups: gate|up (100 MB) in groups of 4 / 8 / 16 / 32 row tiles 609 / 597 / 586 / 580 us at
  // 8192 rows, 534 / 527 / 516 / 512 at 7000 (in a loop under the power cap), but down (50 MB) 328 / 333 / 335 / 351
  // and O (21 MB) 143 / 141 / 143 / 152.
  sh.group = (long long)wN * K * 2 > (64ll << 20) ? 32 : 8;
  sh.KT = (K + PG_TILE_K - 1) / PG_TILE_K;
  sh.mt = (M + 255) / 256;
  const int cols = epi == EPI_SWIGLU ? PG_HALF : PG_BN;
  sh.nt = (N + cols - 1) / cols;
  const long long tiles = (long long)sh.mt * sh.nt;
  if (tiles * sh.KT >= (1ll << 30)) return false;
  sh.wrows = 128;
  while (epi == EPI_SWIGLU && N % sh.wrows) sh.wrows >>= 1;
  const int pairs = *pairs_io;
  *narrow = false;
  // Whole tiles only, or the last wave and the remainder cut evenly: the split saves the idle part of
  // a wave (k steps of ~0.4 us each) and costs parts through L2, tickets, the merge and a late epilogue.
  // Split / whole, us: QKV at 1024 rows (52 against 80 steps) 39.3 / 34.9, O at 400 (9 against 64)
  // 29.4 / 25.3, down at 1500 (123 against 152) 70.2 / 58.8, but down at 1024 (83 against 152) 50.3 / 57.0.
  const int full = (int)(tiles / pairs), rest = (int)(tiles % pairs);
  sh.waves = full;
  sh.share = sh.KT;
  if (scratch && rest) {
    const int whole = full > 0 ? full - 1 : 0;
    const int left = (int)(tiles - (long long)whole * pairs);
    const int share = (left * sh.KT + pairs - 1) / pairs;
    if (share + PG_SPLIT_STEPS < (full - whole + 1) * sh.KT) {
      sh.waves = whole;
      sh.share = share;
    }
  }
  if (epi == EPI_RESID || epi == EPI_F32) {
    // Narrow tiles (whole ones) where they leave less of a wave idle. Both sides in k steps of a wide tile: a narrow
    // step takes 0.71 (0.63 the columns, the same activations); a nearly empty wave down to 0.5 of a full one, a narrow
    // one 0.7; a split 3 steps for each part of a tile and 31 (17 with fp32 sums, which wait for no residual), behind
    // whole waves 5. Wide / narrow, us, weights cold: O at 257 rows 26.3 / 20.3, 1024 27.8 / 21.4, 2048 49.6 / 40.3, but
    // 1280 27.8 / 34.7, 4096 80.0 / 81.7, 8192 143 / 154; down at 600 45.4 / 42.2, 1024 54.7 / 45.4, 2103 105 / 101, but
    // 1900 96.1 / 100.3, 2500 117 / 150; down's fp32 sums at 1024 51.1 / 47.6, but 600 39.9 / 44.1, 2048 88.0 / 101. Of
    // 780 shapes (N 896 - 5120, K 512 - 17408, 257 - 8192 rows, both epilogues) two lose more than 1 % (28.3 / 28.8, 2.4 %).
    PromptShape nr = sh;
    nr.nt = (N + PG_NARROW - 1) / PG_NARROW;
    const long long nt = (long long)nr.mt * nr.nt;
    const double busy = (double)rest / pairs, nbusy = (double)(nt % pairs) / pairs;
    const double tail = sh.share != sh.KT ? sh.share + (sh.waves ? 5.0 : (epi == EPI_F32 ? 17 : 31) + 3.0 * sh.KT / sh.share)
                        : rest ? sh.KT * (0.5 + 0.5 * busy) : 0;
    const double wide = (double)sh.waves * sh.KT + tail;
    const double cost = 0.71 * sh.KT * ((double)(nt / pairs) + (nt % pairs ? 0.7 + 0.3 * nbusy : 0.0));
    if (cost < wide) {
      nr.waves = (int)(nt / pairs);
      nr.share = nr.KT;
      if (nt < pairs) *pairs_io = (int)nt;
      sh = nr;
      *narrow = true;
      return true;
    }
  }
  if (sh.share == sh.KT && tiles < pairs) *pairs_io = (int)tiles;
  return true;
}

template <int EPI, int BN>
int launch_tiles(const void* x, const void* w_tc, void* out, int M, int wN, int K, PromptShape sh, int pairs,
                 const RopeArgs& ra, void* scratch, int* status, void* stream, const char* who) {
  CUtensorMap xmap;
  WeightMaps<BN> wmaps;
  {
    const cuuint64_t dim[2] = {(cuuint64_t)K, (cuuint64_t)M};
    const cuuint64_t stride[1] = {(cuuint64_t)K * 2};
    const cuuint32_t box[2] = {(cuuint32_t)PG_TILE_K, 128};
    int rc = tc_encode(&xmap, x, 2, dim, stride, box, CU_TENSOR_MAP_SWIZZLE_128B, who);
    if (rc) return rc;
  }
  for (size_t i = 0; i < sizeof(wmaps.m) / sizeof(wmaps.m[0]); ++i) {
    // the tiled weight as (64 k, 128 rows, k tiles, row blocks): tiles are already swizzled images
    const cuuint64_t dim[4] = {64, 128, (cuuint64_t)sh.KT, (cuuint64_t)((wN + 127) / 128)};
    const cuuint64_t stride[3] = {128, 16384, (cuuint64_t)sh.KT * 16384};
    const cuuint32_t box[4] = {64, BN == PG_BN ? (cuuint32_t)sh.wrows : 16 * (cuuint32_t)(i + 1), 1, 1};
    int rc = tc_encode(&wmaps.m[i], w_tc, 4, dim, stride, box, CU_TENSOR_MAP_SWIZZLE_NONE, who);
    if (rc) return rc;
  }
  static size_t smem_done[64] = {0};
  Q_CHECK_CUDA(q_ensure_smem(k_gemm_prompt<EPI, BN>, pg_smem(BN), smem_done));
  Q_CHECK_CUDA(q_launch_cluster(k_gemm_prompt<EPI, BN>, dim3(2 * pairs), dim3(PG_THREADS), pg_smem(BN),
                                (cudaStream_t)stream, 2, xmap, wmaps, out, sh, ra, (unsigned char*)scratch, status,
                                q_tl_next(Q_TL_GEMM_TC)));
  return Q_OK;
}

template <int EPI>
int launch_prompt(const void* x, const void* w_tc, void* out, int M, int N, int wN, int K, const RopeArgs& ra,
                  void* scratch, void* stream, const char* who) {
  Q_CHECK_ARG(x && w_tc && out, "%s: null pointer", who);
  Q_CHECK_ARG(M >= 1 && N >= 32 && N % 32 == 0 && K >= 32 && K % 32 == 0,
              "%s: need rows, N and K multiples of 32 (M=%d N=%d K=%d)", who, M, N, K);
  Q_CHECK_ARG(((uintptr_t)x & 15) == 0 && ((uintptr_t)w_tc & 1023) == 0 && ((uintptr_t)out & 31) == 0 &&
                  ((uintptr_t)scratch & 15) == 0,
              "%s: x and scratch must be 16-byte, the output 32-byte and the tiled weight 1024-byte aligned", who);
  int* status = q_tc_status_addr();
  if (!status) { q_set_error("%s: could not locate the device status word", who); return Q_ERR_CUDA; }
  PromptShape sh;
  int pairs = pair_count();
  bool narrow = false;
  Q_CHECK_ARG(prompt_plan(EPI, M, N, wN, K, scratch != nullptr, &sh, &pairs, &narrow), "%s: too many tiles", who);
  if constexpr (EPI == EPI_RESID || EPI == EPI_F32) {
    if (narrow) return launch_tiles<EPI, PG_NARROW>(x, w_tc, out, M, wN, K, sh, pairs, ra, scratch, status, stream, who);
  }
  return launch_tiles<EPI, PG_BN>(x, w_tc, out, M, wN, K, sh, pairs, ra, scratch, status, stream, who);
}

}  // namespace

int64_t q_gemm_prompt_ticket_bytes() { return (int64_t)PG_TICKET_BYTES; }

extern "C" int64_t q_gemm_prompt_scratch_bytes(void) {
  return (int64_t)(PG_TICKET_BYTES + (size_t)pair_count() * 2 * PG_PART_FLOATS * 4);
}

extern "C" int q_gemm_prompt_columns(int M, int N, int K, int residual) {
  PromptShape sh;
  int pairs = pair_count();
  bool narrow = false;
  if (M < 1 || N < 32 || N % 32 || K < 32 || K % 32 ||
      !prompt_plan(residual ? EPI_RESID : EPI_F32, M, N, N, K, true, &sh, &pairs, &narrow)) return 0;
  return narrow ? PG_NARROW : PG_BN;
}

extern "C" int q_gemm_prompt_f32(const void* d_x, const void* d_w_tc, float* d_out, int M, int N, int K,
                                 void* d_scratch, void* stream) {
  return launch_prompt<EPI_F32>(d_x, d_w_tc, d_out, M, N, N, K, RopeArgs(), d_scratch, stream, "q_gemm_prompt_f32");
}

extern "C" int q_gemm_prompt_add(const void* d_x, const void* d_w_tc, void* d_resid, int M, int N, int K,
                                 void* d_scratch, void* stream) {
  Q_CHECK_ARG(d_x != d_resid, "q_gemm_prompt_add: the residual cannot be the projection's input");
  return launch_prompt<EPI_RESID>(d_x, d_w_tc, d_resid, M, N, N, K, RopeArgs(), d_scratch, stream, "q_gemm_prompt_add");
}

extern "C" int q_gemm_prompt_swiglu(const void* d_x, const void* d_w_tc, void* d_act, int M, int inter, int K,
                                    void* d_scratch, void* stream) {
  return launch_prompt<EPI_SWIGLU>(d_x, d_w_tc, d_act, M, inter, 2 * inter, K, RopeArgs(), d_scratch, stream,
                                   "q_gemm_prompt_swiglu");
}

extern "C" int q_gemm_prompt_qkv(const void* d_x, const void* d_w_tc, const void* d_q_gain, const void* d_k_gain,
                                 const void* d_cos, const void* d_sin, const int32_t* d_pos, void* d_q_out,
                                 const q_kv_layout_t* kv, int batch, int T, int n_q_heads, int K, float eps,
                                 void* d_scratch, void* stream) {
  const char* who = "q_gemm_prompt_qkv";
  Q_CHECK_ARG(d_q_gain && d_k_gain && d_cos && d_sin && d_pos && kv, "%s: null pointer", who);
  Q_CHECK_ARG(kv->d_kpool && kv->d_vpool && kv->d_block_table && kv->pages_per_seq >= 1 && kv->n_kv_heads >= 1,
              "%s: incomplete KV layout", who);
  Q_CHECK_ARG(batch >= 1 && T >= 1 && n_q_heads >= 1 && (long long)batch * T < (1ll << 30),
              "%s: bad batch / T / heads", who);
  Q_CHECK_ALIGN(d_q_gain, 16, who); Q_CHECK_ALIGN(d_k_gain, 16, who);
  Q_CHECK_ALIGN(d_cos, 32, who); Q_CHECK_ALIGN(d_sin, 32, who);
  Q_CHECK_ALIGN(kv->d_kpool, 32, who); Q_CHECK_ALIGN(kv->d_vpool, 32, who);
  RopeArgs ra;
  ra.q_gain = (const bf16*)d_q_gain; ra.k_gain = (const bf16*)d_k_gain;
  ra.cos = (const bf16*)d_cos; ra.sin = (const bf16*)d_sin; ra.pos = d_pos;
  ra.kpool = (char*)kv->d_kpool; ra.vpool = (char*)kv->d_vpool; ra.block_table = kv->d_block_table;
  ra.pages_per_seq = kv->pages_per_seq; ra.T = T; ra.nq = n_q_heads; ra.nkv = kv->n_kv_heads; ra.eps = eps;
  const int N = (n_q_heads + 2 * kv->n_kv_heads) * 128;
  return launch_prompt<EPI_ROPE>(d_x, d_w_tc, d_q_out, batch * T, N, N, K, ra, d_scratch, stream, who);
}
