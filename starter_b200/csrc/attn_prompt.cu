// Causal attention over a whole prompt on the 5th-generation tensor cores (the prompt pass;
// reference: engine/prefill.py:45-52 calls the library's scaled-dot-product attention there).
//
// A work item is one (sequence, kv head, block of prompt tokens): two query tiles of 128 rows each
// (row = token, query head of the group: 128 / G tokens x G heads), which share every K/V tile of
// 128 keys (two pages). Per tile S = Q K^T (M = 128 query rows, N = 128 keys, fp32 in tensor
// memory), the softmax warps read their rows, write P as bf16 over S, and O += P V takes P from
// tensor memory and V from shared memory (keys are the K dimension there, so V is the operand whose
// other dimension is contiguous). Tensor memory is exactly S and O of the two query tiles.
//
// What bounds it: per query tile and key tile 16384 exponentials (16 per clock and SM: 1024 cycles)
// and 2 x 128 x 128 x 128 products (1024 cycles). Two query tiles let the tensor cores work on one
// while the softmax of the other runs; a CTA is persistent and starts the next item's first
// products under the current one's last softmax, since an item is only ~9 tiles long at 1-2 K keys.
//
// Warps 0-7 / 8-15: softmax and epilogue of query tile 0 / 1 (TILES = 1: all of one tile). Two (four) threads
// share a row (64 or 32 scores, then as many dims of O each) and exchange its maximum through shared memory: a step is a chain - scores,
// softmax, P V, next scores - and with one thread per row it took 4500 cycles, of which the softmax
// of 128 scores was more than half.
// Warp 16: producer lane. Warp 17: MMA issue; the whole warp walks the loop and one elected lane
// issues, so that descriptors live in uniform registers: an MMA of 128 x 128 x 16 takes 64 cycles,
// about what a single diverged lane needs to assemble its operands.
// O is rescaled only when some row of the warp has a new maximum. (Moving the maximum only after
// it had grown by 2^8 measured 367 against 390 us at 7000 tokens, but the largest probability of a
// row is then no longer exactly 1 in bf16: error against fp64 2.1e-3 instead of 1.77e-3 where scores
// keep growing.) Cast boundaries as in attention.cu: fp32 scores and statistics, P rounded to bf16,
// fp32 accumulation, one rounding of the result.
//
// Tiles are read through tensor maps whose boxes undo the 256-byte row pitch of a page: a box of
// 64 rows x 64 dims lands as rows of 128 bytes, and the pages' own chunk swizzle (chunk ^ row & 7)
// is then the 128-byte swizzle the MMA descriptors name. Every wait is bounded.
#include "tc.cuh"

int* q_attn_status_addr();

namespace {

constexpr int AP_THREADS = 576;                            // 16 softmax warps, producer, MMA
constexpr int AP_KEYS = 128;                               // keys per tile
constexpr uint32_t AP_HALF = 128 * 128;                    // bytes of 128 rows x 64 dims
constexpr uint32_t AP_TILE = 2 * AP_HALF;                  // 128 rows x 128 dims
constexpr uint32_t AP_Q = 0, AP_K = 2 * AP_TILE, AP_V = AP_K + 2 * AP_TILE;
constexpr uint32_t AP_BARS = AP_V + 2 * AP_TILE;           // 192 KB in
constexpr uint32_t AP_RED = AP_BARS + 24 * 8 + 16;         // row exchange: [3][2 tiles x 2 or 4 parts][128] floats
constexpr size_t AP_SMEM = 1024 + AP_RED + 3 * 2 * 2 * 128 * 4;

enum { B_QF = 0, B_QE = 2, B_KF = 4, B_KE = 6, B_VF = 8, B_VE = 10, B_SF = 12, B_P = 14, B_OF = 18, B_OE = 20 };

struct AttnShape {
  int batch, T, G, gshift, nq, nkv, pages_per_seq;
  int tokens;        // prompt tokens per query tile: 128 / G
  int tiles;         // query tiles per work item: 2, or 1 where there are at most two for an SM
  int blocks;        // work items per (sequence, kv head)
  int items;
  int wide;          // the output is 32-byte aligned
  float scale_log2;
};

struct Item { int b, kh, q0, n, max_limit; };

__device__ __forceinline__ Item item_at(const AttnShape& sh, int w, int pos) {
  Item it;
  const int heads = sh.batch * sh.nkv;
  const int blk = w / heads, bh = w - blk * heads;
  it.b = bh / sh.nkv;
  it.kh = bh - it.b * sh.nkv;
  it.q0 = (sh.blocks - 1 - blk) * sh.tiles * sh.tokens;           // latest blocks (most keys) first
  it.max_limit = pos + min(it.q0 + sh.tiles * sh.tokens, sh.T);
  it.n = (it.max_limit + AP_KEYS - 1) / AP_KEYS;
  return it;
}
// The items of a CTA: rounds of gridDim.x, every other round backwards, so that the lengths (which
// fall with the item number) even out.
__device__ __forceinline__ int item_of(int round) {
  const int g = gridDim.x;
  return round * g + ((round & 1) ? g - 1 - (int)blockIdx.x : (int)blockIdx.x);
}

__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, int x, int y, int z, int w,
                                            uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%2, %3, %4, %5}], [%6];"
      ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(w), "r"(bar) : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%2, %3, %4}], [%5];"
      ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar) : "memory");
}
// D[tmem] (+)= A[tmem] . B[smem desc]
__device__ __forceinline__ void tc_mma_ta(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                          uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
// 32 columns of the warp's lanes; valid after tc_wait_ld and tc_pin32.
__device__ __forceinline__ void tc_ld32(uint32_t taddr, float* v) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]),
        "=f"(v[8]), "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15]),
        "=f"(v[16]), "=f"(v[17]), "=f"(v[18]), "=f"(v[19]), "=f"(v[20]), "=f"(v[21]), "=f"(v[22]), "=f"(v[23]),
        "=f"(v[24]), "=f"(v[25]), "=f"(v[26]), "=f"(v[27]), "=f"(v[28]), "=f"(v[29]), "=f"(v[30]), "=f"(v[31])
      : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// Keeps the compiler from using loaded registers before the wait.
__device__ __forceinline__ void tc_pin32(float* v) {
#pragma unroll
  for (int i = 0; i < 32; i += 8)
    asm volatile("" : "+f"(v[i]), "+f"(v[i + 1]), "+f"(v[i + 2]), "+f"(v[i + 3]), "+f"(v[i + 4]), "+f"(v[i + 5]),
                      "+f"(v[i + 6]), "+f"(v[i + 7]));
}
__device__ __forceinline__ void tc_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// Two fp32 lanes per instruction, each rounded like the scalar one; and the largest of three.
__device__ __forceinline__ unsigned long long pair2(float a, float b) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpair2(unsigned long long r, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(r));
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

template <int TILES>
__global__ void __launch_bounds__(AP_THREADS, 1)
k_attn_prompt(const __grid_constant__ CUtensorMap qmap, const __grid_constant__ CUtensorMap kmap,
              const __grid_constant__ CUtensorMap vmap, const int32_t* __restrict__ block_table,
              const int32_t* __restrict__ pos_ptr, bf16* __restrict__ out, AttnShape sh, int* status) {
  constexpr int WARPS = TILES == 2 ? 8 : 16;               // softmax warps of a query tile
  constexpr int PER_ROW = WARPS / 4, COLS = 128 / PER_ROW; // threads of a row, scores (and dims of O) of each
  extern __shared__ unsigned char smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  unsigned char* smem = smem_raw + (base - raw);
  const uint32_t bars = base + AP_BARS;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + AP_BARS + 24 * 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  auto bar = [&](int kind, int i) { return bars + 8u * (uint32_t)(kind + i); };

  pdl_launch_dependents();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int i = 0; i < 24; ++i) {
      const bool warps = i >= B_P && i < B_P + 4;          // half a tile's softmax warps arrive (all at the epilogue)
      mbar_init(bars + 8u * i, i >= B_OE && i < B_OE + 2 ? WARPS : warps ? WARPS / 2 : 1);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 16 && lane == 0) {
    prefetch_map(&qmap);
    prefetch_map(&kmap);
    prefetch_map(&vmap);
  }
  if (warp == 17) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  // All 512 columns are this CTA's, so its tensor memory starts at column 0.
  constexpr uint32_t tmem = 0;
  // q, this pass's K/V rows, and also the position and the block table: a caller's own kernel before this
  // one may write those. All are requested at once, behind the wait: reading position and pages before
  // it, as the decode kernel does, gained 1 us in a prompt of 64 tokens (12 layers, 1128.7 / 1129.6 us).
  pdl_wait();
  const int pos = *reinterpret_cast<const volatile int32_t*>(pos_ptr);
  int first_page[2] = {0, 0};
  if (warp == 16) {                                        // the grid has at most one CTA per item
    const volatile int32_t* table = block_table + (size_t)item_at(sh, item_of(0), 0).b * sh.pages_per_seq;
    first_page[0] = table[0];
    first_page[1] = table[min(1, sh.pages_per_seq - 1)];
  }

  if (warp == 16) {
    // ---------------- producer ----------------
    if (lane == 0) {
      uint32_t step = 0;                                   // K/V tiles requested so far
      uint32_t nitems = 0;
      bool ok = true;
      auto fail = [&]() { atomicExch(status, 7); *abort_flag = 1; ok = false; };
      for (int r = 0; ok && r * (int)gridDim.x < sh.items; ++r) {
        const int w = item_of(r);
        if (w >= sh.items) continue;
        const Item it = item_at(sh, w, pos);
        for (int i = 0; ok && i < TILES; ++i) {
          if (!mbar_wait(bar(B_QE, i), (nitems & 1) ^ 1, abort_flag)) { fail(); break; }
          const int tok = it.b * sh.T + it.q0 + i * sh.tokens;
          mbar_expect_tx(bar(B_QF, i), AP_TILE);
          for (int h = 0; h < 2; ++h)
            tma_load_3d(base + AP_Q + i * AP_TILE + h * AP_HALF, &qmap, 64 * h, it.kh * sh.G, tok, bar(B_QF, i));
        }
        const int32_t* table = block_table + (size_t)it.b * sh.pages_per_seq;
        const int npages = (it.max_limit + Q_PAGE_TOKENS - 1) / Q_PAGE_TOKENS;
        for (int j = 0; ok && j < it.n; ++j, ++step) {
          const int s = step & 1;
          const uint32_t parity = ((step >> 1) & 1) ^ 1;
          const int np = min(2, npages - 2 * j);
          const int page0 = step ? table[2 * j] : first_page[0];
          const int page1 = np < 2 ? 0 : step ? table[2 * j + 1] : first_page[1];
          for (int kv = 0; kv < 2; ++kv) {
            if (!mbar_wait(bar(kv ? B_VE : B_KE, s), parity, abort_flag)) { fail(); break; }
            const uint32_t full = bar(kv ? B_VF : B_KF, s);
            const uint32_t dst = base + (kv ? AP_V : AP_K) + s * AP_TILE;
            mbar_expect_tx(full, (uint32_t)np * AP_HALF);
            for (int p = 0; p < np; ++p)
              for (int h = 0; h < 2; ++h)
                tma_load_4d(dst + h * AP_HALF + p * (AP_HALF / 2), kv ? &vmap : &kmap, 0, h, 0,
                            (p ? page1 : page0) * sh.nkv + it.kh, full);
          }
        }
        ++nitems;
      }
      // copies in flight must land before the CTA may leave
      for (int i = 0; i < 2; ++i) {
        if (nitems > 0 && i < TILES) mbar_wait_plain(bar(B_QF, i), (nitems - 1) & 1);
        if (step > (uint32_t)i) {
          const uint32_t last = ((step - 1 - i) >> 1) & 1;
          mbar_wait_plain(bar(B_KF, (step - 1 - i) & 1), last);
          mbar_wait_plain(bar(B_VF, (step - 1 - i) & 1), last);
        }
      }
      if (!ok) {                                           // ... also those of a step that was given up half-way
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000) __nanosleep(1000);
      }
    }
  } else if (warp == 17) {
    // ---------------- MMA issuer ----------------
    {
      const uint32_t f16 = (1u << 4) | (1u << 7) | (1u << 10) | (16u << 17) | (8u << 24);   // 128 x 128, fp32 sums
      const uint32_t idesc_s = f16, idesc_pv = f16 | (1u << 16);      // V: the non-contracted dimension is contiguous
      const uint64_t q_desc = smem_desc(base + AP_Q), k_desc = smem_desc(base + AP_K);
      // V: leading offset = the other 64 dims, stride offset = the next 8 keys
      const uint64_t v_desc = (uint64_t)(((base + AP_V) & 0x3FFFFu) >> 4) | ((uint64_t)(AP_HALF >> 4) << 16) |
                              (64ull << 32) | (1ull << 46) | (2ull << 61);
      uint32_t kstep = 0, vstep = 0, nitems = 0;
      bool ok = true;
      auto wait = [&](uint32_t b, uint32_t parity) {
        const int landed = mbar_wait(b, parity, abort_flag) ? 1 : 0;
        if (!__all_sync(0xffffffffu, landed)) {
          if (elect_one()) { atomicExch(status, 8); *abort_flag = 1; }
          ok = false;
        }
        tc_fence_after();
        return ok;
      };
      auto scores = [&](int i) {                           // S_i = Q_i K^T of the K tile at kstep
        const uint64_t a = q_desc + (uint64_t)(i * (AP_TILE >> 4)), b = k_desc + (uint64_t)((kstep & 1) * (AP_TILE >> 4));
        if (!elect_one()) return;
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {
          const uint32_t off = (uint32_t)(ks >> 2) * (AP_HALF >> 4) + (ks & 3) * 2;
          tc_mma(tmem + 128u * i, a + off, b + off, idesc_s, ks ? 1u : 0u);
        }
        tc_commit(bar(B_SF, i));
      };
      int r = 0;
      Item cur = item_at(sh, item_of(0), pos);             // the grid has at most one CTA per item
      for (int i = 0; i < TILES && ok; ++i) {
        if (!wait(bar(B_QF, i), 0) || (i == 0 && !wait(bar(B_KF, 0), 0))) break;
        scores(i);
        if (elect_one() && cur.n == 1) tc_commit(bar(B_QE, i));
        __syncwarp();
      }
      if (ok) {
        if (elect_one()) tc_commit(bar(B_KE, 0));
        ++kstep;
      }
      while (ok) {
        // the item after this one
        bool more = false;
        Item nxt = cur;
        for (++r; r * (int)gridDim.x < sh.items; ++r) {
          const int w = item_of(r);
          if (w < sh.items) { nxt = item_at(sh, w, pos); more = true; break; }
        }
        for (int j = 0; ok && j < cur.n; ++j) {
          const bool last = j + 1 == cur.n, ahead = !last || more;
          const int vs = vstep & 1;
          if (!wait(bar(B_VF, vs), (vstep >> 1) & 1)) break;
          for (int i = 0; i < TILES && ok; ++i) {
            if (j == 0 && !wait(bar(B_OE, i), (nitems & 1) ^ 1)) break;
            // P comes in two halves of 64 keys, from different warps
            if (!wait(bar(B_P, 2 * i), vstep & 1) || !wait(bar(B_P, 2 * i + 1), vstep & 1)) break;
            const int keys = cur.max_limit - j * AP_KEYS;      // in the last tile, k steps past the newest key are left out
            if (elect_one()) {
              if (keys >= AP_KEYS) {
#pragma unroll
                for (int ks = 0; ks < 8; ++ks)
                  tc_mma_ta(tmem + 256u + 128u * i, tmem + 128u * i + 8u * ks,
                            v_desc + (uint64_t)(vs * (AP_TILE >> 4) + ks * (2048 >> 4)), idesc_pv, (j | ks) ? 1u : 0u);
              } else {
#pragma unroll 1
                for (int ks = 0; 16 * ks < keys; ++ks)
                  tc_mma_ta(tmem + 256u + 128u * i, tmem + 128u * i + 8u * ks,
                            v_desc + (uint64_t)(vs * (AP_TILE >> 4) + ks * (2048 >> 4)), idesc_pv, (j | ks) ? 1u : 0u);
              }
            }
            __syncwarp();
            if (!ok) break;
            if (last && elect_one()) tc_commit(bar(B_OF, i));
            if (ahead) {
              if (i == 0 && !wait(bar(B_KF, kstep & 1), (kstep >> 1) & 1)) break;
              if (last && !wait(bar(B_QF, i), (nitems + 1) & 1)) break;
              scores(i);
              if (elect_one() && (last ? nxt.n == 1 : j + 2 == cur.n)) tc_commit(bar(B_QE, i));
              __syncwarp();
            }
          }
          if (!ok) break;
          // (not after the last tile: nobody waits for it any more, and the arrival could find that the
          // CTA has left)
          if (ahead && elect_one()) {
            tc_commit(bar(B_VE, vs));
            tc_commit(bar(B_KE, kstep & 1));
          }
          __syncwarp();
          ++vstep;
          if (ahead) ++kstep;
        }
        ++nitems;
        if (!more) break;
        cur = nxt;
      }
    }
  } else {
    // ---------------- softmax and epilogue: query tile `i`, half (a quarter) of a row per thread ----------------
    const int i = TILES == 2 ? warp >> 3 : 0, part = TILES == 2 ? (warp >> 2) & 1 : warp >> 2;
    const int row = tid & 127;
    float* red = reinterpret_cast<float*>(smem + AP_RED) + i * 256;        // [buffer * 512 + part * 128 + row]
    auto tile_sync = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(1 + i), "n"(WARPS * 32) : "memory"); };
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t s_addr = tmem + lanes + 128u * i + (uint32_t)(COLS * part), p_addr = tmem + lanes + 128u * i + (uint32_t)(COLS / 2 * part);
    const uint32_t o_addr = tmem + lanes + 256u + 128u * i + (uint32_t)(COLS * part);
    // A scale that is not positive (the maximum would sit elsewhere) is multiplied in first.
    const bool plain = sh.scale_log2 > 0.f;
    const float c = plain ? sh.scale_log2 : 1.f;
    uint32_t step = 0, nitems = 0;
    // A warp whose wait ran out keeps coming to the tile's barriers; at the item's end all its tile's
    // warps learn of it and leave together.
    bool broken = false;
    auto wait = [&](uint32_t b, uint32_t parity) {
      const int landed = broken || mbar_wait(b, parity, abort_flag) ? 1 : 0;
      if (!__all_sync(0xffffffffu, landed)) {
        if (lane == 0) { atomicExch(status, 9); *abort_flag = 1; }
        broken = true;
      }
      tc_fence_after();
    };
    for (int r = 0; r * (int)gridDim.x < sh.items; ++r) {
      const int w = item_of(r);
      if (w >= sh.items) continue;
      const Item it = item_at(sh, w, pos);
      const int t = it.q0 + i * sh.tokens + (row >> sh.gshift);
      const int limit = t < sh.T ? pos + t + 1 : 0;        // a row past the prompt sees nothing
      // keys that every row of this warp sees: tiles inside them need no mask
      const int t_first = it.q0 + i * sh.tokens + (((warp & 3) * 32) >> sh.gshift);
      const int t_last = it.q0 + i * sh.tokens + (((warp & 3) * 32 + 31) >> sh.gshift);
      const int free_keys = t_last < sh.T ? pos + t_first + 1 : 0;
      float m = -INFINITY, l = 0.f;
      for (int j = 0; j < it.n; ++j, ++step) {
        wait(bar(B_SF, i), step & 1);
        float v[COLS];
        if constexpr (TILES == 2) {
          tc_ld32(s_addr, v);
          tc_ld32(s_addr + 32, v + 32);
          tc_wait_ld();
          tc_pin32(v);
          tc_pin32(v + 32);
        } else {
          float lo[16], hi[16];
          tc_ld16(s_addr, lo);
          tc_ld16(s_addr + 16, hi);
#pragma unroll
          for (int k = 0; k < 16; ++k) { v[k] = lo[k]; v[k + 16] = hi[k]; }
        }
        const int key_base = j * AP_KEYS;
        if (!plain) {
#pragma unroll
          for (int k = 0; k < COLS; ++k) v[k] *= sh.scale_log2;
        }
        if (key_base + AP_KEYS > free_keys) {
          const int vis = limit - key_base - COLS * part;
#pragma unroll
          for (int k = 0; k < COLS; ++k) v[k] = k < vis ? v[k] : -INFINITY;
        }
        if (tid < 128 && key_base + AP_KEYS > it.max_limit && (it.max_limit & 15)) {
          // V rows past the newest key hold stale bits (0 * garbage could be NaN): clear those of its
          // k step before the first product with this tile may start
          wait(bar(B_VF, step & 1), (step >> 1) & 1);
          unsigned char* vt = smem + AP_V + (step & 1) * AP_TILE;
          const int live = it.max_limit - key_base;
          for (int q = tid; !broken && q < ((16 - live) & 15) * 16; q += 128) {
            const int kr = live + (q >> 4);
            *reinterpret_cast<uint4*>(vt + (q & 8 ? AP_HALF : 0u) + kr * 128 + ((q & 7) << 4)) = make_uint4(0, 0, 0, 0);
          }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
        }
        float mx[4] = {v[0], v[1], v[2], v[3]};
#pragma unroll
        for (int k = 4; k < COLS - 4; k += 8)
#pragma unroll
          for (int e = 0; e < 4; ++e) mx[e] = max3(mx[e], v[k + e], v[k + 4 + e]);
        float m_tile = max3(max3(mx[0], mx[1], mx[2]), mx[3], fmaxf(max3(v[COLS - 4], v[COLS - 3], v[COLS - 2]), v[COLS - 1]));
        // the row's other parts; this barrier also says that all of S is in registers, so that P may
        // overwrite it
        red[(step & 1) * 512 + part * 128 + row] = m_tile;
        tc_fence_before();
        tile_sync();
        tc_fence_after();
#pragma unroll
        for (int e = 1; e < PER_ROW; ++e) m_tile = fmaxf(m_tile, red[(step & 1) * 512 + (part ^ e) * 128 + row]);
        if (j == 0) {
          m = m_tile;
        } else {
          if (__any_sync(0xffffffffu, m_tile > m)) {
            // the products up to the tile before are complete: this tile's scores came after them
            const float m_new = fmaxf(m, m_tile);
            const float f = m_new == m ? 1.f : ex2((m - m_new) * c);
            l *= f;
            m = m_new;
#pragma unroll 1
            for (int k = 0; k < COLS / 16; ++k) {
              float o[16];
              uint32_t u[16];
              tc_ld16(o_addr + 16 * k, o);
#pragma unroll
              for (int e = 0; e < 16; ++e) u[e] = __float_as_uint(o[e] * f);
              tc_st16(o_addr + 16 * k, u);
            }
            tc_wait_st();
          }
        }
        const float mc = m == -INFINITY ? 0.f : m * c;
        const unsigned long long c2 = pair2(c, c), mc2 = pair2(-mc, -mc);
        unsigned long long sum[2] = {0ull, 0ull};
#pragma unroll
        for (int h = 0; h < COLS / 32; ++h) {
          uint32_t p[16];
#pragma unroll
          for (int k = 0; k < 16; ++k) {
            float a, b;
            unpair2(fma2(pair2(v[32 * h + 2 * k], v[32 * h + 2 * k + 1]), c2, mc2), a, b);
            a = ex2(a);
            b = ex2(b);
            sum[k & 1] = add2(sum[k & 1], pair2(a, b));
            p[k] = pack_bf16(a, b);
          }
          tc_st16(p_addr + 16 * h, p);
        }
        tc_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(B_P, 2 * i + part / (PER_ROW / 2)));
        __syncwarp();
        float s_lo, s_hi;
        unpair2(add2(sum[0], sum[1]), s_lo, s_hi);
        l += s_lo + s_hi;
      }
      red[1024 + part * 128 + row] = l;
      int give_up;
      asm volatile(
          "{\n\t.reg .pred p, q;\n\t"
          "setp.ne.u32 q, %1, 0;\n\t"
          "barrier.cta.red.or.pred p, %2, %3, q;\n\t"
          "selp.u32 %0, 1, 0, p;\n\t}"
          : "=r"(give_up) : "r"((int)broken), "r"(1 + i), "n"(WARPS * 32) : "memory");
      if (give_up) break;
      {
        float all = red[1024 + row];                       // (in the same order in all threads of a row)
#pragma unroll
        for (int e = 1; e < PER_ROW; ++e) all += red[1024 + e * 128 + row];
        l = all;
      }
      wait(bar(B_OF, i), nitems & 1);
      if (broken) { ++nitems; continue; }
      const float inv = l > 0.f ? 1.f / l : (l == 0.f ? 0.f : l);      // NaN stays NaN
      bf16* dst = out + (((size_t)it.b * sh.T + t) * sh.nq + it.kh * sh.G + (row & (sh.G - 1))) * 128 + COLS * part;
#pragma unroll 1
      for (int k = 0; k < COLS / 16; ++k) {
        float o[16];
        tc_ld16(o_addr + 16 * k, o);
        if (t < sh.T) {
          uint32_t u[8];
#pragma unroll
          for (int q = 0; q < 8; ++q) u[q] = pack_bf16(o[2 * q] * inv, o[2 * q + 1] * inv);
          if (sh.wide) {
            asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                         ::"l"(dst + 16 * k), "r"(u[0]), "r"(u[1]), "r"(u[2]), "r"(u[3]), "r"(u[4]), "r"(u[5]),
                         "r"(u[6]), "r"(u[7]) : "memory");
          } else {
#pragma unroll
            for (int q = 0; q < 8; ++q) *reinterpret_cast<uint32_t*>(dst + 16 * k + 2 * q) = u[q];
          }
        }
        __syncwarp();
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(B_OE, i));
      __syncwarp();
      ++nitems;
    }
  }

  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 17) {
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
}

}  // namespace

extern "C" int q_attention_prefill(const void* d_q, const q_kv_layout_t* kv, const int32_t* d_pos,
                                   void* d_out, int batch, int T, int n_q_heads, float scale,
                                   void* stream) {
  const char* who = "q_attention_prefill";
  Q_CHECK_ARG(d_q && kv && d_pos && d_out, "q_attention_prefill: null pointer");
  Q_CHECK_ARG(kv->d_kpool && kv->d_vpool && kv->d_block_table && kv->pages_per_seq >= 1 &&
                  kv->n_kv_heads >= 1,
              "q_attention_prefill: incomplete KV layout");
  const int nkv = kv->n_kv_heads;
  Q_CHECK_ARG(batch >= 1 && batch <= 65535 && nkv <= 65535 && T >= 1 && n_q_heads >= nkv &&
                  n_q_heads % nkv == 0,
              "q_attention_prefill: bad batch/T/heads");
  const int G = n_q_heads / nkv;
  Q_CHECK_ARG(G <= 8 && (G & (G - 1)) == 0,
              "q_attention_prefill: %d query heads per kv head (1, 2, 4 or 8 supported)", G);
  Q_CHECK_ALIGN(d_q, 16, who); Q_CHECK_ALIGN(d_out, 4, who);
  Q_CHECK_ALIGN(kv->d_kpool, 16, who); Q_CHECK_ALIGN(kv->d_vpool, 16, who);
  int* status = q_attn_status_addr();
  if (!status) { q_set_error("%s: could not locate the device status word", who); return Q_ERR_CUDA; }
  AttnShape sh;
  sh.batch = batch; sh.T = T; sh.G = G; sh.nq = n_q_heads; sh.nkv = nkv; sh.pages_per_seq = kv->pages_per_seq;
  sh.gshift = 0;
  while ((1 << sh.gshift) < G) ++sh.gshift;
  sh.tokens = 128 >> sh.gshift;
  // Two tiles of a CTA hide each other's latencies; one tile has all 16 softmax warps, four threads to a row, and a
  // shorter chain. Up to two tiles per SM the one is faster. One tile / two, us: 1 x 592 tokens 15.5 / 18.8, 1 x 1024
  // 22.8 / 26.4, 1 x 1184 (296 tiles) 28.8 / 30.7, 3 x 250 10.2 / 12.8, 9 x 128 10.2 / 10.5, but 1 x 1200 32.4 / 31.8,
  // 3 x 400 (312) 19.4 / 17.0, 2 x 701 26.9 / 22.8. (With half of the warps idle, one tile took 17.1 at 592.)
  const int sms = q_sm_count();
  sh.tiles = (long long)((T + sh.tokens - 1) / sh.tokens) * batch * nkv <= 2ll * sms ? 1 : 2;
  sh.blocks = (T + sh.tiles * sh.tokens - 1) / (sh.tiles * sh.tokens);
  const long long items = (long long)sh.blocks * batch * nkv;
  Q_CHECK_ARG(items < (1ll << 30) && (long long)batch * T < (1ll << 31), "q_attention_prefill: too many rows");
  sh.items = (int)items;
  sh.wide = ((uintptr_t)d_out & 31) == 0;
  sh.scale_log2 = scale * 1.4426950408889634f;
  CUtensorMap qmap, kmap, vmap;
  {
    const cuuint64_t dim[3] = {128, (cuuint64_t)n_q_heads, (cuuint64_t)batch * T};
    const cuuint64_t stride[2] = {256, (cuuint64_t)n_q_heads * 256};
    const cuuint32_t box[3] = {64, (cuuint32_t)G, (cuuint32_t)sh.tokens};
    int rc = tc_encode(&qmap, d_q, 3, dim, stride, box, CU_TENSOR_MAP_SWIZZLE_128B, who);
    if (rc) return rc;
  }
  for (int i = 0; i < 2; ++i) {
    // (64 dims, half, token row, page x head): the number of pages is the caller's, bounded by memory
    const cuuint64_t dim[4] = {64, 2, Q_PAGE_TOKENS, 1u << 24};
    const cuuint64_t stride[3] = {128, 256, Q_PAGE_TOKENS * 256};
    const cuuint32_t box[4] = {64, 1, Q_PAGE_TOKENS, 1};
    int rc = tc_encode(i ? &vmap : &kmap, i ? kv->d_vpool : kv->d_kpool, 4, dim, stride, box, CU_TENSOR_MAP_SWIZZLE_NONE,
                       who);
    if (rc) return rc;
  }
  static size_t done[2][64] = {{0}};
  auto kern = sh.tiles == 2 ? k_attn_prompt<2> : k_attn_prompt<1>;
  Q_CHECK_CUDA(q_ensure_smem(kern, AP_SMEM, done[sh.tiles - 1]));
  const int grid = sh.items < sms ? sh.items : sms;
  Q_CHECK_CUDA(q_launch(kern, dim3(grid), dim3(AP_THREADS), AP_SMEM, (cudaStream_t)stream, qmap, kmap, vmap,
                        kv->d_block_table, d_pos, (bf16*)d_out, sh, status));
  return Q_OK;
}
