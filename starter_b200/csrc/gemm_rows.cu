// Projections of a step with 1 .. 64 activation rows whose outputs are complete when the kernel ends: no
// split-K slots in memory, the layer's element-wise work before and after the product inside the kernel
// (reference: engine/decode_step.py:43-59 runs norm, projection, add, norm, projection, SwiGLU, projection).
//
//   EPI_F32      out fp32 [M][N]                                        (q|k|v)
//   EPI_RESID    x = bf16(x + bf16(sum)) in place, and the sums of squares of the new x  (O, down)
//   EPI_SWIGLU   act = bf16(bf16(silu(bf16 g)) * bf16 u)                (gate|up, weight [gate; up])
//   NORM         the activations are the residual x: RMSNorm is applied to every 64-k slice in shared
//                memory on its way to the tensor cores, with the sums of squares that EPI_RESID left
// so that a layer is QKV, attention, O, gate|up, down: five launches instead of the eight of gemm_tc.cu with
// k_add_rmsnorm and k_swiglu between the projections (4 - 5 us each, of which under 1 us is work).
//
// What bounds it is the weight stream from HBM. The activations are the A operand (M = 64 rows of the
// instruction; rows past the batch hold leftovers of shared memory and are never read back), the weight rows
// the B operand: there a CTA's share is any number of 8-row atoms (1 KB for 64 k) of the 128 x 64 tiles of
// gemm_tc.cu, copied as they lie. A cluster of S CTAs owns a run of atoms and splits K; at the end every CTA
// sends its fp32 sums to the cluster CTA that owns the row (rows are dealt out in S runs) through
// distributed shared memory, where they are added in rank order and finished.
//
// Roles (384 threads): warp 0 weight copies (a ring's worth before anything the previous kernel wrote is
// needed), warp 1 MMA issuer, warp 2 activation slices by TMA after the dependency wait, warps 4-11 norm of the
// slices (four warps to each of a stage's two k tiles), then the epilogue. What each role's loop costs per stage
// is what limits short tiles - 250 ns a stage with nothing to copy and nothing to multiply -, hence two k tiles a
// stage, whole warps that walk their loop and elect the lane that issues, and a hardware barrier, not an mbarrier
// that eight warps poll, to wake the epilogue. (While it was built, with clusters of at most four, down alone at 16 rows:
// one k tile a stage 13.9 us, two 10.9; the loop inside one lane's branch 14.3, polls by one lane 12.6. With a ring of
// half an SM, so that the next kernel's CTA could start beside this one, there is too little in flight at 64 rows: 12
// layers 1228 against 1044 us; 922 / 908 at 16.)
// Decode step of 12 layers, gemm_tc.cu and its consumers / this, us: 16 x 1000 keys 1032 / 870, 32 x 2000
// 1402 / 1249, 64 x 333 1251 / 1004; inside the step a layer's QKV, O, gate|up, down at 16 rows 8.8, 7.4, 18.8, 11.4 us,
// of which the weights take 4.8, 3.2, 15.2, 7.6.
// Every wait is bounded as in gemm_tc.cu and reports in the same status word (codes 10-13).
#include "tc.cuh"

int* q_tc_status_addr();

namespace {

constexpr int GR_THREADS = 384;
constexpr int GR_EPI = 256;                       // threads of warps 4-11
constexpr int GR_MISC = (64 + GR_EPI) * 4;        // bytes: 1 / rms of the rows, then partial sums of squares
constexpr int GR_ATOM = 1024;                     // 8 weight rows x 64 k
constexpr int GR_TILE = 16 * GR_ATOM;             // one 128 x 64 tile
constexpr int GR_MAX_COLS = 256;                  // accumulator columns of a CTA
constexpr int GR_MAX_STAGES = 12;
constexpr size_t GR_SMEM = 224 * 1024;            // one CTA per SM
constexpr size_t GR_SMEM_MAX = 227 * 1024;        // what a kernel is allowed (always the same: no launch lowers another's)

enum { EPI_F32 = 0, EPI_RESID = 1, EPI_SWIGLU = 2 };

struct RowsShape {
  int M, KT;           // activation rows, k tiles
  int units, clusters; // 8-row atoms (EPI_SWIGLU: pairs of a gate and an up atom) dealt out over the clusters:
  int each, more;      // `each` to a cluster, one more to the first `more`
  int S, log_s;        // CTAs of a cluster: K is split S ways
  int up_atom;         // EPI_SWIGLU: first up atom of the weight
  int ldo;             // columns of a row of the output
  int ar;              // rows of the activation slice in shared memory (M rounded up to 8)
  int rpr;             // rows that a cluster CTA finishes
  int ld;              // floats of a row of the receive area
  int tile_bytes;      // one k tile in the ring: activation slice, then weight atoms
  int stages, stage_bytes;  // a ring stage holds two k tiles
  int recv_off, misc_off;   // bytes from the start of shared memory
};
struct RowsNorm {
  const bf16* gain;    // [K]
  const float* ss;     // [parts][M] sums of squares
  int parts;
  float k, eps;
};

__device__ __forceinline__ void gr_cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void gr_cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ void epi_sync() { asm volatile("bar.sync 1, %0;" ::"n"(GR_EPI) : "memory"); }
__device__ __forceinline__ uint32_t norm2(uint32_t x, float inv, uint32_t g) {
  // (two bf16 rounded to bf16 in one packed instruction; their product is exact in fp32, so the result is the same)
  const uint32_t n = pack_bf16(bf_lo(x) * inv, bf_hi(x) * inv);
  const __nv_bfloat162 p = __hmul2_rn(*reinterpret_cast<const __nv_bfloat162*>(&n), *reinterpret_cast<const __nv_bfloat162*>(&g));
  return *reinterpret_cast<const uint32_t*>(&p);
}

template <int EPI, bool NORM>
__global__ void __launch_bounds__(GR_THREADS, 1)
k_gemm_rows(const __grid_constant__ CUtensorMap xmap, const unsigned char* __restrict__ W, void* __restrict__ out,
            float* __restrict__ ss_out, const RowsShape sh, const RowsNorm nm, int* status, unsigned long long* tl) {
  extern __shared__ unsigned char smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  unsigned char* smem = smem_raw + (base - raw);
  float* recv = reinterpret_cast<float*>(smem + sh.recv_off);               // [S][rpr][ld]
  float* inv_s = reinterpret_cast<float*>(smem + sh.misc_off);              // [64], then [GR_EPI] partial sums
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + sh.misc_off + GR_MISC);
  // full[stages] | empty[stages] | ready[stages] | acc_full
  const uint32_t bar_full = smem_u32(bars), bar_empty = bar_full + 8u * GR_MAX_STAGES;
  const uint32_t bar_ready = bar_empty + 8u * GR_MAX_STAGES, bar_acc = bar_ready + 8u * GR_MAX_STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 3 * GR_MAX_STAGES + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  bf16* gain_s = reinterpret_cast<bf16*>(tmem_slot + 2);                    // NORM: this CTA's k range
  float* ss_s = reinterpret_cast<float*>(tmem_slot + 2);                    // EPI_RESID (never with NORM): [rpr][8-column chunks]

  tl_begin(tl);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = blockIdx.x & (sh.S - 1), cl = blockIdx.x >> sh.log_s;     // (ranks follow x inside a cluster)
  const int u0 = cl * sh.each + min(cl, sh.more), nu = sh.each + (cl < sh.more ? 1 : 0);
  const int kt0 = (rank * sh.KT) >> sh.log_s, nk = (((rank + 1) * sh.KT) >> sh.log_s) - kt0;
  // Every CTA starts somewhere else in its k range: in step, all SMs would ask the same L2 slices for the same
  // activation slice at the same time.
  const int rot = nk > 0 ? cl % nk : 0;
  const int cols = nu * (EPI == EPI_SWIGLU ? 16 : 8);                        // accumulator columns
  uint32_t tcols = 32;
  while ((int)tcols < cols) tcols <<= 1;

  // Nobody but warp 0 waits for the first weight copies to be issued, and they wait for nothing but the barriers:
  // tensor memory is allocated, and gains are fetched, meanwhile.
  const uint32_t a_bytes = (uint32_t)sh.ar * 128u;
  // the runs of atoms as pieces that end at a 128-row block: a run of 32 atoms has up to three, the gate
  // and the up run of at most 16 two each
  constexpr int PIECES = EPI == EPI_SWIGLU ? 4 : 3;
  const unsigned char* src[PIECES];
  uint32_t off[PIECES], bytes[PIECES];
  int issued = 0, kt = rot;                                  // ring stages filled, next k tile
  // weights of the next stage; sources move on (the whole warp keeps the addresses, so that they stay in uniform
  // registers, and one elected lane issues)
  auto weights = [&](uint32_t dst, uint32_t full, uint64_t policy) {
    const bool two = issued * 2 + 1 < nk;
    const ptrdiff_t next = kt + 1 == nk ? GR_TILE - (ptrdiff_t)nk * GR_TILE : GR_TILE;
    if (elect_one()) {
      mbar_expect_tx(full, (uint32_t)cols * (two ? 256u : 128u));
#pragma unroll
      for (int p = 0; p < PIECES; ++p)
        if (bytes[p]) bulk_g2s(dst + off[p], src[p], bytes[p], full, policy);
      if (two) {
#pragma unroll
        for (int p = 0; p < PIECES; ++p)
          if (bytes[p]) bulk_g2s(dst + sh.tile_bytes + off[p], src[p] + next, bytes[p], full, policy);
      }
    }
    __syncwarp();
    const bool wrap = kt + 2 >= nk;                     // (past the end after the last stage)
    kt += wrap ? 2 - nk : 2;
#pragma unroll
    for (int p = 0; p < PIECES; ++p) src[p] += ((ptrdiff_t)2 - (wrap ? nk : 0)) * GR_TILE;
    ++issued;
  };
  const int n_fill = (nk + 1) >> 1;       // ring stages this CTA fills in all
  if (tid == 0) {
    for (int s = 0; s < sh.stages; ++s) {
      mbar_init(bar_full + 8 * s, 2);            // weights and activations
      mbar_init(bar_empty + 8 * s, 1);
      mbar_init(bar_ready + 8 * s, 8);
    }
    mbar_init(bar_acc, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
  if (sh.S > 1) gr_cluster_arrive();                         // (waited for before the first remote store)
  uint32_t tmem = 0;                                         // warp 1's; the epilogue reads it when it is woken
  if (warp == 0) {
    int a = u0, left = nu, part = 0;
    uint32_t o = a_bytes;
#pragma unroll
    for (int p = 0; p < PIECES; ++p) {
      if (left == 0 && EPI == EPI_SWIGLU && part == 0) { a = sh.up_atom + u0; left = nu; part = 1; }
      const int n = min(left, 16 - (a & 15));
      src[p] = W + ((size_t)(a >> 4) * sh.KT + kt0 + rot) * GR_TILE + (size_t)(a & 15) * GR_ATOM;
      off[p] = o;
      bytes[p] = (uint32_t)n * GR_ATOM;
      o += bytes[p];
      a += n;
      left -= n;
    }
    const uint64_t policy = stream_policy();
    for (int s = 0; s < sh.stages && s < n_fill; ++s) weights(base + s * sh.stage_bytes, bar_full + 8 * s, policy);
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_u32(tmem_slot)), "r"(tcols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    __syncwarp();
    tmem = *reinterpret_cast<volatile uint32_t*>(tmem_slot);
  }
  if (warp == 2 && lane == 0) prefetch_map(&xmap);
  if (NORM && warp >= 4)                                     // (read after the barriers among warps 4-11 below)
    for (int i = tid - 128; i < nk * 8; i += GR_EPI)
      *reinterpret_cast<uint4*>(gain_s + 8 * i) = __ldg(reinterpret_cast<const uint4*>(nm.gain + kt0 * 64) + i);
  auto warp_wait = [&](uint32_t b, uint32_t par) {
    return __all_sync(0xffffffffu, mbar_wait(b, par, abort_flag) ? 1 : 0) != 0;
  };

  if (warp == 0) {
    // ---------------- weights: the stages after the first ring ----------------
    if (issued < n_fill) pdl_wait();                         // as in gemm_tc.cu: the wait limit starts here
    const uint64_t policy = stream_policy();
    int st = 0;
    uint32_t parity = 0;
    while (issued < n_fill) {
      if (!warp_wait(bar_empty + 8 * st, parity)) {
        if (lane == 0) {
          atomicExch(status, 10);
          *abort_flag = 1;
        }
        break;
      }
      weights(base + st * sh.stage_bytes, bar_full + 8 * st, policy);
      if (++st == sh.stages) { st = 0; parity ^= 1u; }
    }
    // From here on this CTA asks for no more weights: the next kernel's CTAs may take the SMs that become free.
    if (elect_one()) pdl_launch_dependents();
    __syncwarp();
    // copies in flight must land before the CTA may exit, also when a role gave up
    pdl_wait();
    tl_waited(tl);
    for (int s = 0; s < sh.stages && s < issued; ++s)
      if (!mbar_wait_plain(bar_full + 8 * s, ((issued - 1 - s) / sh.stages) & 1) && lane == 0) atomicExch(status, 13);
  } else if (warp == 2) {
    // ---------------- activations ----------------
    pdl_wait();                         // they are complete from here on
    int st = 0, filled = 0;
    uint32_t parity = 1;
    for (int i = 0; i < nk; i += 2) {
      if (filled++ >= sh.stages && !warp_wait(bar_empty + 8 * st, parity)) break;    // (warp 0 waits for the same and reports)
      const bool two = i + 1 < nk;
      const int k1 = kt + 1 == nk ? 0 : kt + 1;
      if (elect_one()) {
        mbar_expect_tx(bar_full + 8 * st, two ? 2 * a_bytes : a_bytes);
        tma_load_2d(base + st * sh.stage_bytes, &xmap, (kt0 + kt) * 64, 0, bar_full + 8 * st);
        if (two) tma_load_2d(base + st * sh.stage_bytes + sh.tile_bytes, &xmap, (kt0 + k1) * 64, 0, bar_full + 8 * st);
      }
      __syncwarp();
      kt += 2;
      if (kt >= nk) kt -= nk;
      if (++st == sh.stages) { st = 0; parity ^= 1u; }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    // (the whole warp walks the loop and one elected lane issues: descriptors stay in uniform registers)
    pdl_wait();                         // as in gemm_tc.cu: the wait limit starts here
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(cols >> 3) << 17) | (4u << 24);
    const uint64_t desc0 = smem_desc(base);
    const uint32_t stage_units = (uint32_t)sh.stage_bytes >> 4, a_units = a_bytes >> 4, tile_units = (uint32_t)sh.tile_bytes >> 4;
    bool ok = true;
    int st = 0;
    uint32_t parity = 0;
    for (int i = 0; i < nk; i += 2) {
      if (!warp_wait(bar_full + 8 * st, parity) || (NORM && !warp_wait(bar_ready + 8 * st, parity))) { ok = false; break; }
      tc_fence_after();
      const bool two = i + 1 < nk;
      const uint64_t a_desc = desc0 + (uint64_t)(st * stage_units), b_desc = a_desc + a_units;
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < 4; ++k) tc_mma(tmem, a_desc + 2u * k, b_desc + 2u * k, idesc, (i || k) ? 1u : 0u);
        if (two) {
#pragma unroll
          for (int k = 0; k < 4; ++k) tc_mma(tmem, a_desc + tile_units + 2u * k, b_desc + tile_units + 2u * k, idesc, 1u);
        }
        tc_commit(bar_empty + 8 * st);
      }
      __syncwarp();
      if (++st == sh.stages) { st = 0; parity ^= 1u; }
    }
    // The epilogue is woken through a hardware barrier: eight warps that polled an mbarrier all along slowed the
    // roles above down.
    if (ok && nk > 0) {
      if (elect_one()) tc_commit(bar_acc);
      __syncwarp();
      ok = warp_wait(bar_acc, 0);
    }
    if (!ok && lane == 0) {
      atomicExch(status, 11);
      *abort_flag = 1;
    }
    tc_fence_before();
    __syncwarp();
    asm volatile("bar.arrive 2, %0;" ::"n"(GR_EPI + 32) : "memory");
  } else if (warp >= 4) {
    // ---------------- norm of the slices, then the epilogue (warps 4..11) ----------------
    const int et = tid - 128, half = et >> 7;
    pdl_wait();
    bool ok = true;
    if (NORM) {
      // 1 / rms of every row: the parts of a row are added by 256 / (rows rounded up) threads
      int mp = 8;
      while (mp < sh.M) mp <<= 1;
      const int groups = GR_EPI / mp, r = et & (mp - 1), g = et / mp;
      float s = 0.f;
      if (r < sh.M) {
#pragma unroll 8
        for (int p = g; p < nm.parts; p += groups) s += nm.ss[p * sh.M + r];
      }
      inv_s[64 + et] = s;
      epi_sync();
      if (et < sh.M) {
        float t = 0.f;
        for (int j = 0; j < groups; ++j) t += inv_s[64 + j * mp + et];
        inv_s[et] = rsqrtf(t / nm.k + nm.eps);            // (rounded as the row norm rounds it)
      }
      epi_sync();
      // A thread has one 16-byte chunk of rows r0, r0 + 16, ...: r0 % 8 is r % 8 of all of them, so that the
      // swizzled position stands for the same 8 columns in each.
      const int r0 = (et & 127) >> 3, pos = et & 7, chunk = pos ^ (r0 & 7);
      float inv[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) inv[j] = r0 + 16 * j < sh.M ? inv_s[r0 + 16 * j] : 0.f;
      // Each group has one of a stage's two tiles. (Both wait for every stage: a group that skipped a phase of a
      // barrier could take the one before it for the one it waits for.)
      int st = 0, kt = rot;
      uint32_t parity = 0;
      for (int i = 0; i < nk; i += 2) {
        if (!warp_wait(bar_full + 8 * st, parity)) { ok = false; break; }
        if (i + half < nk) {
          int k = kt + half;
          if (k >= nk) k -= nk;
          unsigned char* a = smem + st * sh.stage_bytes + half * sh.tile_bytes + r0 * 128 + pos * 16;
          const uint4 gv = *reinterpret_cast<const uint4*>(gain_s + k * 64 + chunk * 8);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if (r0 + 16 * j < sh.M) {
              uint4* p = reinterpret_cast<uint4*>(a + j * 2048);
              uint4 v = *p;
              v.x = norm2(v.x, inv[j], gv.x);
              v.y = norm2(v.y, inv[j], gv.y);
              v.z = norm2(v.z, inv[j], gv.z);
              v.w = norm2(v.w, inv[j], gv.w);
              *p = v;
            }
          }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_ready + 8 * st);
        kt += 2;
        if (kt >= nk) kt -= nk;
        if (++st == sh.stages) { st = 0; parity ^= 1u; }
      }
      if (!ok && lane == 0) {
        atomicExch(status, 12);
        *abort_flag = 1;
      }
    }
    // The residual of this thread's first items is asked for before the sums are there.
    const int row0 = rank * sh.rpr, nrow = min(sh.rpr, sh.M - row0);         // rows finished here (may be <= 0)
    const int items = nrow > 0 ? nrow * nu : 0;                              // (row, 8 output columns)
    uint4 res[2];
    if (EPI == EPI_RESID) {
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int it = et + j * GR_EPI;
        if (it < items)
          res[j] = *reinterpret_cast<const uint4*>(reinterpret_cast<const bf16*>(out) +
                                                   (size_t)(row0 + it / nu) * sh.ldo + (u0 + it % nu) * 8);
      }
    }
    asm volatile("bar.sync 2, %0;" ::"n"(GR_EPI + 32) : "memory");         // the MMA warp arrives in every case
    ok = __all_sync(0xffffffffu, *abort_flag == 0 ? 1 : 0) != 0;
    tmem = *reinterpret_cast<volatile uint32_t*>(tmem_slot);
    tc_fence_after();
    if (sh.S > 1) {
      __syncwarp();
      gr_cluster_wait();                                                     // every CTA of the cluster has started
    }
    // tensor memory -> the receive area of the CTA that finishes the row. With M = 64 a warp's first 16
    // lanes hold 16 rows.
    const int q = warp & 3;
    if (ok && q * 16 < sh.M) {
      const int m = q * 16 + lane;
      const bool live = lane < 16 && m < sh.M;
      const int owner = live ? m / sh.rpr : 0;
      uint32_t dst = smem_u32(recv + ((size_t)rank * sh.rpr + (live ? m - owner * sh.rpr : 0)) * sh.ld);
      if (sh.S > 1) asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(dst) : "r"(dst), "r"(owner));
      for (int c = 16 * half; c < cols; c += 32) {
        float v[16];
        if (nk > 0) {
          tc_ld16(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)c, v);
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] = 0.f;
        }
        if (live) {
#pragma unroll
          for (int j = 0; j < 16; j += 4)
            if (c + j < cols)
              asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};"
                           ::"r"(dst + (uint32_t)(c + j) * 4u), "f"(v[j]), "f"(v[j + 1]), "f"(v[j + 2]), "f"(v[j + 3])
                           : "memory");
        }
      }
    }
    tc_fence_before();
    if (sh.S > 1) {
      __syncwarp();
      gr_cluster_arrive();
      gr_cluster_wait();
    } else {
      epi_sync();
    }
    // ---- the rows this CTA owns: add the ranks' sums in order and finish ----
    for (int j = 0, it = et; it < items; ++j, it += GR_EPI) {
      const int r = it / nu, c = it - r * nu;
      auto column = [&](int first, float (&v)[8]) {
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = 0.f;
        for (int s = 0; s < sh.S; ++s) {
          const float4* p = reinterpret_cast<const float4*>(recv + ((size_t)s * sh.rpr + r) * sh.ld + first);
          const float4 a = p[0], b = p[1];
          v[0] += a.x; v[1] += a.y; v[2] += a.z; v[3] += a.w;
          v[4] += b.x; v[5] += b.y; v[6] += b.z; v[7] += b.w;
        }
      };
      float v[8];
      column(c * 8, v);
      const size_t at = (size_t)(row0 + r) * sh.ldo + (u0 + c) * 8;
      if (EPI == EPI_F32) {
        float4* dst = reinterpret_cast<float4*>(reinterpret_cast<float*>(out) + at);
        dst[0] = make_float4(v[0], v[1], v[2], v[3]);
        dst[1] = make_float4(v[4], v[5], v[6], v[7]);
      } else if (EPI == EPI_SWIGLU) {
        float u[8];
        column((nu + c) * 8, u);
        uint32_t w[4];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float gb = bf16_round(v[e]);
          v[e] = bf16_round(gb / (1.0f + expf(-gb))) * bf16_round(u[e]);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) w[e] = pack_bf16(v[2 * e], v[2 * e + 1]);
        *reinterpret_cast<uint4*>(reinterpret_cast<bf16*>(out) + at) = make_uint4(w[0], w[1], w[2], w[3]);
      } else {
        uint4* x = reinterpret_cast<uint4*>(reinterpret_cast<bf16*>(out) + at);
        const uint4 old = j == 0 ? res[0] : j == 1 ? res[1] : *x;
        const uint32_t ow[4] = {old.x, old.y, old.z, old.w};
        uint32_t w[4];
        float sq = 0.f;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          w[e] = pack_bf16(bf_lo(ow[e]) + bf16_round(v[2 * e]), bf_hi(ow[e]) + bf16_round(v[2 * e + 1]));
          sq += bf_lo(w[e]) * bf_lo(w[e]) + bf_hi(w[e]) * bf_hi(w[e]);
        }
        *x = make_uint4(w[0], w[1], w[2], w[3]);
        ss_s[it] = sq;
      }
    }
    if (EPI == EPI_RESID) {
      epi_sync();
      if (et < nrow) {
        float s = 0.f;
        for (int c = 0; c < nu; ++c) s += ss_s[et * nu + c];
        ss_out[cl * sh.M + row0 + et] = s;
      }
    }
  }

  if (warp < 4 && sh.S > 1) {           // the barriers that warps 4-11 passed above
    __syncwarp();
    gr_cluster_wait();
    gr_cluster_arrive();
    gr_cluster_wait();
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tcols) : "memory");
  }
  tl_end(tl);
}

// Clusters of S CTAs, one CTA per SM, that the current device holds at once (a cluster stays inside one
// GPC); without a device what the SM count alone would allow.
template <int EPI, bool NORM>
int rows_clusters(int S, int sms) {
  static int cached[64][9];
  if (S == 1) return sms;
  const int dev = q_device_index();
  if (dev < 0) return sms / S;
  int& n = cached[dev][S];
  if (n == 0) {
    static size_t done[64] = {0};
    int got = 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(S);
    cfg.blockDim = dim3(GR_THREADS);
    cfg.dynamicSmemBytes = 200 * 1024;           // one CTA per SM
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = S; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    cfg.attrs = at; cfg.numAttrs = 1;
    cudaError_t e = q_ensure_smem(k_gemm_rows<EPI, NORM>, GR_SMEM_MAX, done);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&got, k_gemm_rows<EPI, NORM>, &cfg);
    if (e != cudaSuccess) { cudaGetLastError(); got = sms / S; }
    n = got < sms / S ? got : sms / S;
    if (n < 1) n = 1;
  }
  return n;
}

// N output columns (EPI_SWIGLU: inter) over the device; false where the kernel does not take the shape.
template <int EPI, bool NORM>
bool rows_shape(int M, int N, int K, RowsShape* sh, size_t* smem) {
  if (M < 1 || M > Q_MAX_ROWS || N < 8 || N % 8 || K < 64 || K % 64) return false;
  int sms = q_sm_count();
  if (sms <= 0) sms = 148;
  const int per = EPI == EPI_SWIGLU ? 16 : 8;
  sh->M = M;
  sh->KT = K / 64;
  sh->units = N / 8;
  sh->up_atom = N / 8;
  sh->ldo = N;
  sh->ar = (M + 7) / 8 * 8;
  sh->S = 0;
  // K is split so that a CTA's time comes out least, in bytes at the HBM rate of an SM: its weights, half of its
  // activation slices (from L2), 11 KB a ring stage (250 ns) and 40 KB for the exchange. Clusters of 8 leave a quarter of
  // the SMs idle and still win by the stages and, since O and down then leave half as many sums of squares, in the next
  // norm; towards 64 rows their receive area does not fit (33 rows still take them). Step of 12 layers, at most 4 / 8 CTAs
  // a cluster, when that was chosen, us: 9 x 300 keys 790 / 771, 16 x 1024 896 / 883, 32 x 500 904 / 902.
  long long best = -1;
  for (int S = 1; S <= 8; S *= 2) {
    RowsShape t = *sh;
    const int ncl = rows_clusters<EPI, NORM>(S, sms);
    t.S = S;
    t.log_s = S == 8 ? 3 : S == 4 ? 2 : S - 1;
    t.clusters = t.units < ncl ? t.units : ncl;
    t.each = t.units / t.clusters;
    t.more = t.units - t.each * t.clusters;
    const int cols = (t.each + (t.more ? 1 : 0)) * per;
    if (cols > GR_MAX_COLS) continue;
    t.rpr = (M + S - 1) / S;
    t.ld = cols + 4;
    t.tile_bytes = t.ar * 128 + cols * 128;
    t.stage_bytes = 2 * t.tile_bytes;
    const int kts = (t.KT + S - 1) / S;
    const size_t recv = ((size_t)S * t.rpr * t.ld * 4 + 15) / 16 * 16;
    const size_t misc = GR_MISC + (3 * GR_MAX_STAGES + 1) * 8 + 8 + (NORM ? (size_t)kts * 128 : (size_t)t.rpr * (cols / 8) * 4);
    const size_t fixed = 1024 + misc + (S > 1 ? recv : 0);             // S == 1: received where the ring was
    if (fixed + 3 * (size_t)t.stage_bytes > GR_SMEM) continue;
    t.stages = (int)((GR_SMEM - fixed) / t.stage_bytes);
    if (t.stages > GR_MAX_STAGES) t.stages = GR_MAX_STAGES;
    size_t ring = (size_t)t.stages * t.stage_bytes + (t.tile_bytes > 8192 ? 0 : 8192 - t.tile_bytes);   // 64 rows are read
    if (S == 1 && ring < recv) ring = recv;
    t.recv_off = S > 1 ? (int)ring : 0;
    t.misc_off = (int)((ring + (S > 1 ? recv : 0) + 15) / 16 * 16);
    const size_t bytes = 1024 + t.misc_off + misc;
    if (bytes > GR_SMEM_MAX) continue;
    const long long cost = (long long)kts * (cols * 128 + t.ar * 64) + (kts + 1) / 2 * 11000 + (S > 1 ? 40000 : 0);
    if (best < 0 || cost < best) { best = cost; *sh = t; *smem = bytes; }
  }
  return sh->S != 0;
}

template <int EPI, bool NORM>
int launch_rows(const void* x, const void* w_tc, void* out, float* ss_out, const RowsNorm& nm, int M, int N, int K,
                void* stream, const char* who) {
  Q_CHECK_ARG(x && w_tc && out, "%s: null pointer", who);
  Q_CHECK_ARG(((uintptr_t)x & 15) == 0 && ((uintptr_t)w_tc & 1023) == 0 && ((uintptr_t)out & 15) == 0 &&
                  ((uintptr_t)nm.gain & 15) == 0 && ((uintptr_t)nm.ss & 3) == 0 && ((uintptr_t)ss_out & 3) == 0,
              "%s: x, gain and output must be 16-byte, the tiled weight 1024-byte aligned", who);
  RowsShape sh;
  size_t smem = 0;
  Q_CHECK_ARG((rows_shape<EPI, NORM>(M, N, K, &sh, &smem)), "%s: shape not supported (M=%d N=%d K=%d)", who, M, N, K);
  int* status = q_tc_status_addr();
  if (!status) { q_set_error("%s: could not locate the device status word", who); return Q_ERR_CUDA; }
  CUtensorMap map;
  const cuuint64_t dim[2] = {(cuuint64_t)K, (cuuint64_t)M};
  const cuuint64_t stride[1] = {(cuuint64_t)K * 2};
  const cuuint32_t box[2] = {64, (cuuint32_t)sh.ar};
  int rc = tc_encode(&map, x, 2, dim, stride, box, CU_TENSOR_MAP_SWIZZLE_128B, who);
  if (rc) return rc;
  static size_t done[64] = {0};
  Q_CHECK_CUDA(q_ensure_smem(k_gemm_rows<EPI, NORM>, GR_SMEM_MAX, done));
  const dim3 grid(sh.clusters * sh.S), block(GR_THREADS);
  if (sh.S > 1)
    Q_CHECK_CUDA(q_launch_cluster(k_gemm_rows<EPI, NORM>, grid, block, smem, (cudaStream_t)stream, (unsigned)sh.S, map,
                                  (const unsigned char*)w_tc, out, ss_out, sh, nm, status, q_tl_next(Q_TL_GEMM_ROWS)));
  else
    Q_CHECK_CUDA(q_launch(k_gemm_rows<EPI, NORM>, grid, block, smem, (cudaStream_t)stream, map,
                          (const unsigned char*)w_tc, out, ss_out, sh, nm, status, q_tl_next(Q_TL_GEMM_ROWS)));
  return Q_OK;
}

int norm_args(const void* gain, const float* ss, int parts, int K, float eps, RowsNorm* nm, const char* who) {
  Q_CHECK_ARG(!gain || (ss && parts >= 1), "%s: the norm needs the sums of squares", who);
  nm->gain = (const bf16*)gain;
  nm->ss = ss;
  nm->parts = parts;
  nm->k = (float)K;
  nm->eps = eps;
  return Q_OK;
}

}  // namespace

extern "C" int q_gemm_rows_parts(int M, int N, int K) {
  RowsShape sh;
  size_t smem = 0;
  return rows_shape<EPI_RESID, false>(M, N, K, &sh, &smem) ? sh.clusters : 0;
}

extern "C" int q_gemm_rows_splits(int M, int N, int K, int add) {
  RowsShape sh;
  size_t smem = 0;
  return (add ? rows_shape<EPI_RESID, false>(M, N, K, &sh, &smem) : rows_shape<EPI_F32, false>(M, N, K, &sh, &smem)) ? sh.S : 0;
}

extern "C" int q_gemm_rows_supported(int M, int hidden, int inter, int q_cols, int qkv_cols) {
  RowsShape sh;
  size_t smem = 0;
  if (qkv_cols < q_sm_count()) return 0;          // (the steps keep up to one part per SM and row behind one QKV slot)
  return rows_shape<EPI_F32, true>(M, qkv_cols, hidden, &sh, &smem) && rows_shape<EPI_F32, false>(M, qkv_cols, hidden, &sh, &smem) &&
         rows_shape<EPI_RESID, false>(M, hidden, q_cols, &sh, &smem) && rows_shape<EPI_RESID, false>(M, hidden, inter, &sh, &smem) &&
         rows_shape<EPI_SWIGLU, true>(M, inter, hidden, &sh, &smem);
}

extern "C" int q_gemm_rows_f32(const void* d_x, const void* d_gain, const float* d_ss, int parts, const void* d_w_tc,
                               float* d_out, int M, int N, int K, float eps, void* stream) {
  RowsNorm nm;
  int rc = norm_args(d_gain, d_ss, parts, K, eps, &nm, "q_gemm_rows_f32");
  if (rc) return rc;
  if (d_gain) return launch_rows<EPI_F32, true>(d_x, d_w_tc, d_out, nullptr, nm, M, N, K, stream, "q_gemm_rows_f32");
  return launch_rows<EPI_F32, false>(d_x, d_w_tc, d_out, nullptr, nm, M, N, K, stream, "q_gemm_rows_f32");
}

extern "C" int q_gemm_rows_add(const void* d_x, const void* d_w_tc, void* d_resid, float* d_ss, int M, int N, int K,
                               void* stream) {
  Q_CHECK_ARG(d_ss && d_x != d_resid, "q_gemm_rows_add: needs room for the sums of squares, and the residual cannot "
              "be the projection's input");
  RowsNorm nm = {};
  return launch_rows<EPI_RESID, false>(d_x, d_w_tc, d_resid, d_ss, nm, M, N, K, stream, "q_gemm_rows_add");
}

extern "C" int q_gemm_rows_swiglu(const void* d_x, const void* d_gain, const float* d_ss, int parts, const void* d_w_tc,
                                  void* d_act, int M, int inter, int K, float eps, void* stream) {
  Q_CHECK_ARG(d_gain, "q_gemm_rows_swiglu: null pointer");
  RowsNorm nm;
  int rc = norm_args(d_gain, d_ss, parts, K, eps, &nm, "q_gemm_rows_swiglu");
  if (rc) return rc;
  return launch_rows<EPI_SWIGLU, true>(d_x, d_w_tc, d_act, nullptr, nm, M, inter, K, stream, "q_gemm_rows_swiglu");
}
