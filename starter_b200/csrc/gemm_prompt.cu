// Projections of the prompt pass: Y[M,N] = X[M,K] . W[N,K]^T for hundreds to thousands of
// activation rows, on CTA pairs (tcgen05.mma.cta_group::2), with the layer's element-wise work
// as the epilogue (reference: engine/prefill.py:40-52 calls library GEMMs and separate kernels).
//
// A pair of CTAs (a cluster of two, one SM each) owns an output tile of 256 rows x `bn` columns:
// each CTA brings in its 128 activation rows and HALF of the tile's weight rows per 64-k step,
// the leader's one MMA thread multiplies over both shared memories, and each CTA's tensor memory
// ends up with its own 128 rows x bn columns in fp32. What bounds this kernel is operand traffic
// from L2 into shared memory: per 64 k an SM reads 16 KB + bn/2 x 128 B for 128 x bn outputs, at
// bn = 256 two thirds of the bytes per product of the one-CTA kernel of gemm_tc.cu (weights 128 x
// rows 256 per SM), which is why prompts leave that kernel.
//
// One accumulator holds the whole K range of a tile, so nothing is split, no fp32 partials
// travel through memory, and the epilogue can apply the consumer right away. Its thread owns one
// activation row (tensor-memory lane) and walks the columns, so all of these are thread-local:
//   EPI_F32     fp32 sums                          (before a tensor-parallel all-reduce)
//   EPI_RESID   x = bf16(x + bf16(sum))            (O and down projections, in place)
//   EPI_SWIGLU  act = bf16(bf16(silu(bf16 g)) * bf16 u): the tile's columns are bn/2 gate columns
//               (the leader's weight half) and the matching bn/2 up columns (the peer's half)
//   EPI_ROPE    bf16 q|k|v, head norm + RoPE on q and k heads (128 columns each), q to
//               [row][head][128], k and v rows into their pages
// The rounding points are those of the consumers in fused_ops.cu.
//
// Roles per CTA (192 threads): warp 0 producer (one lane), warp 1 MMA issuer (the leader's one
// lane), warps 2-5 epilogue, which drains one of two accumulators while the MMAs fill the other.
// The `full` barriers live in the leader: both CTAs' copies complete there (a stage is 2 x its
// bytes); commits release stages and hand over accumulators in both CTAs at once. Every wait is
// bounded as in gemm_tc.cu and reports in the same status word (codes 5-8).
//
// Tiles go to pairs in a fixed order (tile = pair + i * pairs): row tiles fastest inside groups of
// eight, so that the tiles in flight share both operands in L2.
#include "tc.cuh"

int* q_tc_status_addr();

namespace {

constexpr int PG_THREADS = 192;
constexpr int PG_TILE_K = 64;
constexpr int PG_A_BYTES = 128 * PG_TILE_K * 2;            // 16 KB of activations per CTA and stage
constexpr int PG_SMEM_BUDGET = 224 * 1024;
constexpr int PG_GROUP = 8;                                // row tiles per raster group

enum { EPI_F32 = 0, EPI_RESID = 1, EPI_SWIGLU = 2, EPI_ROPE = 3 };

struct PromptShape {
  int M, N, KT;         // rows, output columns (EPI_SWIGLU: inter), k tiles
  int mt, nt;           // tiles along rows (256) and columns (bn; EPI_SWIGLU bn/2)
  int bn;               // MMA N: 128 .. 256, multiple of 32
  int wrows;            // weight rows per copy (a power of two that divides every copy's start)
  int stages;
};

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

// 32 bytes (16 bf16) at a 32-byte boundary: whole sectors, since neighbouring lanes hold other rows.
__device__ __forceinline__ void ld32B(const void* p, uint32_t (&r)[8]) {
  asm volatile("ld.global.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "l"(p) : "memory");
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
__device__ __forceinline__ void ld_gain16(const bf16* p, float (&v)[16]) {
  const uint4 a = __ldg(reinterpret_cast<const uint4*>(p)), b = __ldg(reinterpret_cast<const uint4*>(p) + 1);
  const uint32_t r[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
  unpack16(r, v);
}

// k / v row of a page: the 32 bytes of dims d..d+15 (d a multiple of 16) are one aligned pair of
// 16-byte chunks whose order depends on the token's parity (chunk index XOR-ed with r & 7).
__device__ __forceinline__ void st_page16(char* row, int r, int d, const float (&v)[16]) {
  uint32_t a[8], b[8];
  pack16(v, a);
  const bool swap = r & 1;
#pragma unroll
  for (int i = 0; i < 4; ++i) { b[i] = swap ? a[i + 4] : a[i]; b[i + 4] = swap ? a[i] : a[i + 4]; }
  st32B(row + (((d >> 3) ^ (r & 6)) << 4), b);
}

// One 128-column head of one row: `taddr` is the head's first column in tensor memory.
__device__ __forceinline__ void rope_head(uint32_t taddr, const RopeArgs& ra, bf16* Q, int m, bool live, int head,
                                          int pos, char* krow, char* vrow, int r) {
  const bool is_q = head < ra.nq, is_v = head >= ra.nq + ra.nkv;     // warp-uniform
  const int kh = is_v ? head - ra.nq - ra.nkv : head - ra.nq;
  const size_t hoff = is_q ? 0 : (size_t)kh * (Q_PAGE_TOKENS * 256);
  if (is_v) {
    for (int d = 0; d < 64; d += 16) {
      float lo[16], hi[16];
      tc_ld16x2(taddr + d, taddr + 64 + d, lo, hi);
      if (live) {
        st_page16(vrow + hoff, r, d, lo);
        st_page16(vrow + hoff, r, 64 + d, hi);
      }
    }
    return;
  }
  float ss = 0.f;
#pragma unroll 1
  for (int d = 0; d < 64; d += 16) {
    float lo[16], hi[16];
    tc_ld16x2(taddr + d, taddr + 64 + d, lo, hi);
#pragma unroll
    for (int e = 0; e < 16; ++e) {
      const float a = bf16_round(lo[e]), b = bf16_round(hi[e]);
      ss += a * a + b * b;
    }
  }
  const float inv = rsqrtf(ss / 128.f + ra.eps);
  const bf16* gain = is_q ? ra.q_gain : ra.k_gain;
  const bf16* cs = ra.cos + (size_t)pos * 128;
  const bf16* sn = ra.sin + (size_t)pos * 128;
#pragma unroll 1
  for (int d = 0; d < 64; d += 16) {
    float lo[16], hi[16], g[16], c[16], s[16], o[16];
    uint32_t w[8];
    tc_ld16x2(taddr + d, taddr + 64 + d, lo, hi);
    ld_gain16(gain + d, g);
#pragma unroll
    for (int e = 0; e < 16; ++e) lo[e] = bf16_round(bf16_round(bf16_round(lo[e]) * inv) * g[e]);
    ld_gain16(gain + 64 + d, g);
#pragma unroll
    for (int e = 0; e < 16; ++e) hi[e] = bf16_round(bf16_round(bf16_round(hi[e]) * inv) * g[e]);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      ld32B(cs + 64 * h + d, w);
      unpack16(w, c);
      ld32B(sn + 64 * h + d, w);
      unpack16(w, s);
#pragma unroll
      for (int e = 0; e < 16; ++e)
        o[e] = h == 0 ? bf16_round(lo[e] * c[e]) + bf16_round(-hi[e] * s[e])
                      : bf16_round(hi[e] * c[e]) + bf16_round(lo[e] * s[e]);   // rounded at the store
      if (live) {
        if (is_q) {
          pack16(o, w);
          st32B(Q + ((size_t)m * ra.nq + head) * 128 + 64 * h + d, w);
        } else {
          st_page16(krow + hoff, r, 64 * h + d, o);
        }
      }
    }
  }
}

template <int EPI>
__global__ void __launch_bounds__(PG_THREADS, 1)
k_gemm_prompt(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap, void* __restrict__ out,
              PromptShape sh, const __grid_constant__ RopeArgs ra, int* status, unsigned long long* tl) {
  extern __shared__ unsigned char smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  unsigned char* smem = smem_raw + (base - raw);
  const int half = sh.bn >> 1;                              // weight rows per CTA and stage
  const uint32_t stage_bytes = PG_A_BYTES + (uint32_t)half * 128u;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + (size_t)sh.stages * stage_bytes);
  // full[stages] (leader's) | empty[stages] | acc_full[2] | acc_empty[2] (leader's)
  const uint32_t bar_full = smem_u32(bars), bar_empty = bar_full + 8u * sh.stages;
  const uint32_t bar_acc_full = bar_empty + 8u * sh.stages, bar_acc_empty = bar_acc_full + 16u;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * sh.stages + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  tl_begin(tl);
  pdl_launch_dependents();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t rank = cluster_rank();
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const int total = sh.mt * sh.nt;

  if (tid == 0) {
    for (int s = 0; s < sh.stages; ++s) {
      mbar_init(bar_full + 8 * s, 1);
      mbar_init(bar_empty + 8 * s, 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(bar_acc_full + 8 * b, 1);
      mbar_init(bar_acc_empty + 8 * b, 8);                  // four epilogue warps of each CTA
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
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
    const int per = PG_GROUP * sh.nt;
    const int g = t / per, in = t - g * per;
    const int rows = min(PG_GROUP, sh.mt - g * PG_GROUP);
    ni = in / rows;
    mi = g * PG_GROUP + in - ni * rows;
  };

  if (warp == 0) {
    // ---------------- producer ----------------
    if (lane == 0) {
      const uint32_t full0 = leader_addr(bar_full);
      const int nload = half / sh.wrows;
      const uint32_t wbytes = (uint32_t)sh.wrows * 128u;
      int st = 0;
      uint32_t parity = 1;                                  // an untouched stage is free
      bool ok = true, waited = false;
      int issued = 0;
      for (int t = pair; ok && t < total; t += pairs) {
        int mi, ni;
        locate(t, mi, ni);
        const int row = mi * 256 + (int)rank * 128;
        // first weight row of this CTA's half
        const int n0 = EPI == EPI_SWIGLU ? (int)rank * sh.N + ni * half : ni * sh.bn + (int)rank * half;
        for (int kt = 0; kt < sh.KT; ++kt) {
          if (!mbar_wait(bar_empty + 8 * st, parity, abort_flag)) {
            atomicExch(status, 5);
            *abort_flag = 1;
            ok = false;
            break;
          }
          const uint32_t full = full0 + 8u * st, dst = base + st * stage_bytes;
          if (rank == 0) mbar_expect_tx(bar_full + 8 * st, 2 * stage_bytes);
          for (int j = 0; j < nload; ++j) {
            const int n = n0 + j * sh.wrows;
            pair_load_4d(dst + PG_A_BYTES + j * wbytes, &wmap, 0, n & 127, kt, n >> 7, full);
          }
          if (!waited) {                                    // weights do not depend on the previous kernel
            pdl_wait();
            tl_waited(tl);
            waited = true;
          }
          pair_load_2d(dst, &xmap, kt * PG_TILE_K, row, full);
          ++issued;
          if (++st == sh.stages) { st = 0; parity ^= 1u; }
        }
      }
      // Every copy must have landed before the CTAs may leave: the leader waits for the last fill
      // of each stage (both CTAs' bytes), the cluster barrier at the end holds the peer.
      if (rank == 0)
        for (int s = 0; s < sh.stages && s < issued; ++s) {
          const int last = (issued - 1 - s) / sh.stages;
          if (!mbar_wait_plain(bar_full + 8 * s, last & 1)) atomicExch(status, 8);
        }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (leader) ----------------
    if (rank == 0 && lane == 0) {
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(sh.bn >> 3) << 17) | (16u << 24);
      const uint32_t stage_units = stage_bytes >> 4;
      const uint64_t desc0 = smem_desc(base);
      int st = 0, seg = 0;
      uint32_t parity = 0;
      bool ok = true;
      for (int t = pair; ok && t < total; t += pairs, ++seg) {
        const int buf = seg & 1;
        if (!mbar_wait(bar_acc_empty + 8 * buf, ((seg >> 1) & 1) ^ 1, abort_flag)) { ok = false; break; }
        tc_fence_after();
        const uint32_t dacc = tmem_base + (uint32_t)buf * 256u;
        for (int kt = 0; kt < sh.KT; ++kt) {
          if (!mbar_wait(bar_full + 8 * st, parity, abort_flag)) { ok = false; break; }
          tc_fence_after();
          const uint64_t a_desc = desc0 + (uint64_t)(st * stage_units);
          const uint64_t b_desc = a_desc + (PG_A_BYTES >> 4);
#pragma unroll
          for (int k = 0; k < PG_TILE_K / 16; ++k)
            pair_mma(dacc, a_desc + 2u * k, b_desc + 2u * k, idesc, (kt | k) ? 1u : 0u);
          pair_commit(bar_empty + 8 * st);
          if (++st == sh.stages) { st = 0; parity ^= 1u; }
        }
        if (ok) pair_commit(bar_acc_full + 8 * buf);
      }
      if (!ok) {
        atomicExch(status, 6);
        *abort_flag = 1;
      }
    }
  } else {
    // ---------------- epilogue (warps 2..5) ----------------
    pdl_wait();
    const int q = warp & 3;
    const uint32_t acc_empty0 = leader_addr(bar_acc_empty);
    int seg = 0;
    for (int t = pair; t < total; t += pairs, ++seg) {
      const int buf = seg & 1;
      int mi, ni;
      locate(t, mi, ni);
      const int m = mi * 256 + (int)rank * 128 + q * 32 + lane;
      const bool live = m < sh.M;
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
      if (EPI == EPI_F32) {
        float* dst = reinterpret_cast<float*>(out) + (size_t)m * sh.N + ni * sh.bn;
        for (int c = 0; c < sh.bn && ni * sh.bn + c < sh.N; c += 32) {   // N is a multiple of 32
          float v[16], w[16];
          tc_ld16x2(taddr + c, taddr + c + 16, v, w);
          if (live) {
#pragma unroll
            for (int j = 0; j < 16; j += 8) {
              uint32_t a[8], b[8];
#pragma unroll
              for (int e = 0; e < 8; ++e) { a[e] = __float_as_uint(v[j + e]); b[e] = __float_as_uint(w[j + e]); }
              st32B(dst + c + j, a);
              st32B(dst + c + 16 + j, b);
            }
          }
        }
      } else if (EPI == EPI_RESID) {
        bf16* x = reinterpret_cast<bf16*>(out) + (size_t)(live ? m : 0) * sh.N + ni * sh.bn;
#pragma unroll 2
        for (int c = 0; c < sh.bn && ni * sh.bn + c < sh.N; c += 32) {
          float v[16], w[16], a[16];
          uint32_t r0[8], r1[8];
          ld32B(x + c, r0);
          ld32B(x + c + 16, r1);
          tc_ld16x2(taddr + c, taddr + c + 16, v, w);
          unpack16(r0, a);
#pragma unroll
          for (int e = 0; e < 16; ++e) v[e] = a[e] + bf16_round(v[e]);
          unpack16(r1, a);
#pragma unroll
          for (int e = 0; e < 16; ++e) w[e] = a[e] + bf16_round(w[e]);
          pack16(v, r0);
          pack16(w, r1);
          if (live) {
            st32B(x + c, r0);
            st32B(x + c + 16, r1);
          }
        }
      } else if (EPI == EPI_SWIGLU) {
        bf16* act = reinterpret_cast<bf16*>(out) + (size_t)m * sh.N + ni * half;
        for (int c = 0; c < half && ni * half + c < sh.N; c += 16) {     // inter is a multiple of 16
          float g[16], u[16];
          uint32_t r[8];
          tc_ld16x2(taddr + c, taddr + half + c, g, u);
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            const float gb = bf16_round(g[e]);
            g[e] = bf16_round(gb / (1.0f + expf(-gb))) * bf16_round(u[e]);
          }
          pack16(g, r);
          if (live) st32B(act + c, r);
        }
      } else {
        const int mm = live ? m : 0;
        const int b = mm / ra.T, pos = ra.pos[0] + mm - b * ra.T;
        const int page = ra.block_table[(size_t)b * ra.pages_per_seq + pos / Q_PAGE_TOKENS];
        const int r = pos % Q_PAGE_TOKENS;
        const size_t row = (size_t)page * ra.nkv * (Q_PAGE_TOKENS * 256) + (size_t)r * 256;
        for (int c = 0; c < sh.bn && ni * sh.bn + c < sh.N; c += 128)
          rope_head(taddr + c, ra, reinterpret_cast<bf16*>(out), m, live, (ni * sh.bn + c) >> 7, pos, ra.kpool + row,
                    ra.vpool + row, r);
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

// Column width of a tile: 256 unless a narrower tile saves waves. `sms`/2 pairs take one tile
// each per wave, and a tile costs about its operand traffic, 256 + bn rows of 128 bytes per 64 k.
int pick_bn(int mt, int N, int sms, int step) {
  int best = 256;
  long long cost = -1;
  for (int bn = 256; bn >= 128; bn -= step) {
    const long long tiles = (long long)mt * ((N + bn - 1) / bn);
    const long long waves = (tiles + sms / 2 - 1) / (sms / 2);
    const long long c = waves * (256 + bn);
    if (cost < 0 || c < cost) { cost = c; best = bn; }
  }
  return best;
}

// `N` as in PromptShape; the weight has `wN` rows.
template <int EPI>
int launch_prompt(const void* x, const void* w_tc, void* out, int M, int N, int wN, int K, const RopeArgs& ra,
                  void* stream, const char* who) {
  Q_CHECK_ARG(x && w_tc && out, "%s: null pointer", who);
  Q_CHECK_ARG(M >= 1 && N >= 32 && N % 32 == 0 && K >= 32 && K % 32 == 0,
              "%s: need rows, N and K multiples of 32 (M=%d N=%d K=%d)", who, M, N, K);
  Q_CHECK_ARG(((uintptr_t)x & 15) == 0 && ((uintptr_t)w_tc & 1023) == 0 && ((uintptr_t)out & 31) == 0,
              "%s: x must be 16-byte, the output 32-byte and the tiled weight 1024-byte aligned", who);
  int* status = q_tc_status_addr();
  if (!status) { q_set_error("%s: could not locate the device status word", who); return Q_ERR_CUDA; }
  const int sms = q_sm_count();
  PromptShape sh;
  sh.M = M; sh.N = N;
  sh.KT = (K + PG_TILE_K - 1) / PG_TILE_K;
  sh.mt = (M + 255) / 256;
  // gate and up halves stay whole 128-row blocks; heads are 128 columns
  sh.bn = EPI == EPI_SWIGLU ? 256 : pick_bn(sh.mt, N, sms, EPI == EPI_ROPE ? 128 : 32);
  const int cols = EPI == EPI_SWIGLU ? sh.bn / 2 : sh.bn;
  sh.nt = (N + cols - 1) / cols;
  Q_CHECK_ARG((long long)sh.mt * sh.nt < (1ll << 30), "%s: too many tiles", who);
  sh.wrows = 128;
  while ((sh.bn / 2) % sh.wrows || (EPI == EPI_SWIGLU && N % sh.wrows)) sh.wrows >>= 1;
  const uint32_t stage = PG_A_BYTES + sh.bn / 2 * 128;
  sh.stages = PG_SMEM_BUDGET / stage;
  if (sh.stages > 12) sh.stages = 12;
  CUtensorMap xmap, wmap;
  {
    const cuuint64_t dim[2] = {(cuuint64_t)K, (cuuint64_t)M};
    const cuuint64_t stride[1] = {(cuuint64_t)K * 2};
    const cuuint32_t box[2] = {(cuuint32_t)PG_TILE_K, 128};
    int rc = tc_encode(&xmap, x, 2, dim, stride, box, CU_TENSOR_MAP_SWIZZLE_128B, who);
    if (rc) return rc;
  }
  {
    // the tiled weight as (64 k, 128 rows, k tiles, row blocks): tiles are already swizzled images
    const cuuint64_t dim[4] = {64, 128, (cuuint64_t)sh.KT, (cuuint64_t)((wN + 127) / 128)};
    const cuuint64_t stride[3] = {128, 16384, (cuuint64_t)sh.KT * 16384};
    const cuuint32_t box[4] = {64, (cuuint32_t)sh.wrows, 1, 1};
    int rc = tc_encode(&wmap, w_tc, 4, dim, stride, box, CU_TENSOR_MAP_SWIZZLE_NONE, who);
    if (rc) return rc;
  }
  const size_t smem = 1024 + (size_t)sh.stages * stage + (2 * sh.stages + 4) * 8 + 16;
  static size_t smem_done[64] = {0};
  Q_CHECK_CUDA(q_ensure_smem(k_gemm_prompt<EPI>, smem, smem_done));
  const int tiles = sh.mt * sh.nt;
  const int pairs = tiles < sms / 2 ? tiles : sms / 2;
  Q_CHECK_CUDA(q_launch_cluster(k_gemm_prompt<EPI>, dim3(2 * pairs), dim3(PG_THREADS), smem, (cudaStream_t)stream, 2,
                                xmap, wmap, out, sh, ra, status, q_tl_next(Q_TL_GEMM_TC)));
  return Q_OK;
}

}  // namespace

extern "C" int q_gemm_prompt_f32(const void* d_x, const void* d_w_tc, float* d_out, int M, int N, int K,
                                 void* stream) {
  return launch_prompt<EPI_F32>(d_x, d_w_tc, d_out, M, N, N, K, RopeArgs(), stream, "q_gemm_prompt_f32");
}

extern "C" int q_gemm_prompt_add(const void* d_x, const void* d_w_tc, void* d_resid, int M, int N, int K,
                                 void* stream) {
  Q_CHECK_ARG(d_x != d_resid, "q_gemm_prompt_add: the residual cannot be the projection's input");
  return launch_prompt<EPI_RESID>(d_x, d_w_tc, d_resid, M, N, N, K, RopeArgs(), stream, "q_gemm_prompt_add");
}

extern "C" int q_gemm_prompt_swiglu(const void* d_x, const void* d_w_tc, void* d_act, int M, int inter, int K,
                                    void* stream) {
  return launch_prompt<EPI_SWIGLU>(d_x, d_w_tc, d_act, M, inter, 2 * inter, K, RopeArgs(), stream,
                                   "q_gemm_prompt_swiglu");
}

extern "C" int q_gemm_prompt_qkv(const void* d_x, const void* d_w_tc, const void* d_q_gain, const void* d_k_gain,
                                 const void* d_cos, const void* d_sin, const int32_t* d_pos, void* d_q_out,
                                 const q_kv_layout_t* kv, int batch, int T, int n_q_heads, int K, float eps,
                                 void* stream) {
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
  return launch_prompt<EPI_ROPE>(d_x, d_w_tc, d_q_out, batch * T, N, N, K, ra, stream, who);
}
