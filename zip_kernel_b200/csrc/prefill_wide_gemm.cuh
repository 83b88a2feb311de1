// Kernel 2b: tensor-core fused GEMM on wide token tiles, the library's own route for many tokens.
//
// The arithmetic is that of prefill_gemm_kernel's e4m3 form, step by step and in the same order, so the
// outputs have the same bits:
//
//   Y[n,t] = fp16( sx[t] * ( sum_g s[n,g] * acc[g,n,t] + w * sum_blk s[n,bc] * acc_hi[blk,n,t] - Z[n,t] ) )
//   Z[n,t] = sum_g (s*z)[n,g] * sumX[t,g]
//
// What bounds prefill_gemm_kernel: per K-step of 128 a CTA moves a weight tile and an activation tile from L2 and
// hands one accumulator round (commit -> tcgen05.ld -> FMA -> next MMAs into that buffer) between warps.  On a
// 128 x 128 tile that is 650-700 clk per step (prepared weights; 1000-1100 on packed ones) for 256 clk of MMAs,
// and about 11000 clk per tile before the first and after the last step.  Here the tile is 128 rows x 256
// tokens: one hand-over and one weight tile per 512 clk of MMAs, and half as many tiles.  Measured (B200, 1.9 GHz,
// gate_up 4096 -> 28672, 4096 tokens, 5 % residual blocks, prepared weights): 1100-1200 clk per step, 4300 clk of
// epilogue.  What bounds it now is the fold: 128 columns x 128 rows per warp quarter in fp32 FMAs take about
// 1050 clk per step with the MMAs removed, the MMAs and copies 550 clk with the fold removed.
//
// To fit, two things moved out of the way:
//   * two accumulators of 256 columns fill tensor memory, so the zero-point term has no accumulator of its
//     own: its tf32 products (one K-step per window of 16 groups) run after the last K-step, all into one of
//     the buffers, and the fold subtracts that buffer once;
//   * their operand tiles have no shared memory of their own either: four helper warps write them into ring
//     slots, where a copy would have landed.
// The fold warps read their scales from a table of 16 steps, double buffered, that the helper warps keep
// ahead of them (dense groups and residual blocks alike), so the fold's loop has no window hand-over, no
// global load and no block-wide barrier.
//
// Weights: PREP reads e4m3 bytes prepared at load time (16 KB per step, the A operand as it lands).  Without
// them the packed nibbles land in the lower half of the slot (8 KB) and the helper warps widen them in place:
// every thread takes its row's 64 bytes into registers, the four warps meet, and the row goes back as 128
// e4m3 bytes.  A tile twice as wide halves that work per multiply-add, and the accumulators arrive as floats,
// without the int -> float conversions of the s8 form.
//
// Registers: the fold keeps 128 fp32 sums per thread.  The block is launched with 128 registers a thread
// (512 x 128 = 65536) and re-deals them between its warpgroups: 56 + 88 + 184 + 184 = 4 x 128.  (192 or more for
// the fold makes ptxas spill in every role: +16 % time.)
#pragma once

#include "prefill_gemm.cuh"

namespace w4a4 {
namespace wide {

constexpr int ROWS = 128;
constexpr int WARP_W = 0, WARP_X = 1, WARP_MMA = 2, WARP_HELP0 = 4, WARP_FOLD0 = 8;
constexpr int N_HELP = 4, N_FOLD = 8;
constexpr int THREADS = (WARP_FOLD0 + N_FOLD) * 32;
constexpr int REG_ISSUE = 56, REG_HELP = 88, REG_FOLD = 184;
static_assert(REG_ISSUE + REG_HELP + 2 * REG_FOLD <= 4 * 128, "the warpgroups share the registers of the launch");
constexpr int W_BYTES = ROWS * BCOL;              // one e4m3 weight tile
constexpr int TAB = 16;                           // K-steps per scale table = groups per zero-point product

constexpr int TN = 256;                           // tokens per tile
constexpr int X_BYTES = TN * BCOL;
constexpr int SLOT = W_BYTES + X_BYTES;
constexpr int STAGES = 4;
constexpr int ACC_BUFS = 2;
constexpr int COLS = TN / 2;                      // tokens of a fold thread
struct Layout {
  static constexpr size_t tab = (size_t)STAGES * SLOT;                 // float [2][TAB][128]
  static constexpr size_t sxs = tab + (size_t)2 * TAB * ROWS * 4;      // float [TN]
  static constexpr size_t bars = sxs + (size_t)TN * 4;
  static constexpr size_t total = bars + 256;
  static_assert(1024 + total <= 232448, "shared memory of one SM");
  static_assert((size_t)ROWS * (TN + 4) * 4 <= tab, "the ring takes the tile's sums in the epilogue");
  static_assert(ACC_BUFS * TN <= pre::TMEM_COLS, "tensor memory capacity");
  static_assert(ACC_BUFS < STAGES, "the fold warps' arrival for step n + ACC_BUFS must fall into that step's barrier phase");
  static_assert(STAGES % 2 == 0, "an issuing thread takes every other step");
};
inline size_t smem_bytes() { return 1024 + Layout::total; }

enum : int { SITE_WIDE_W = 72, SITE_WIDE_X, SITE_WIDE_READY, SITE_WIDE_PACKED, SITE_WIDE_TAB, SITE_WIDE_Z, SITE_WIDE_ACC };

__device__ __forceinline__ void mbar_arrive_n(uint64_t* bar, uint32_t n) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(n) : "memory");
}
// instruction descriptors without the token count (bits 17..22: N / 8), M = 128
constexpr uint32_t IDESC_F8_M = (1u << 4) | ((uint32_t)(ROWS >> 4) << 24);
constexpr uint32_t IDESC_TF32_M = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(ROWS >> 4) << 24);

// Bounded wait whose polls may sleep in hardware (up to 20 us each): the roles of this kernel wait for hundreds of
// clocks at a time, and polling takes issue slots and instruction fetches from the fold warps of the same
// scheduler (-2 % time against plain polling).  The hint bounds a poll from above only - a poll that misses returns
// after about 4 us on B200 - so the count of polls alone (65536: 0.26 s) does not say how long the wait lasts: it
// gives up after WAIT_POLLS polls AND WAIT_NS nanoseconds (a count too, because the timer also runs while another
// process has the GPU).
constexpr uint32_t WAIT_POLLS = 1u << 16;
constexpr uint64_t WAIT_NS = 1000000000;
__device__ __forceinline__ uint64_t timer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ bool try_wait_suspend(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity), "r"(20000) : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool wait_suspend(uint64_t* bar, uint32_t parity, int site) {
  if (try_wait_suspend(bar, parity)) return true;
  const uint64_t t0 = timer_ns();
  for (uint32_t i = 0; i < WAIT_POLLS || timer_ns() - t0 < WAIT_NS; ++i)
    if (try_wait_suspend(bar, parity)) return true;
  record_error(site, parity);
  return false;
}

// `count` <= 32 * P neighbouring outputs that may start at any element, by one warp.  Straight-line code, all reads before
// the first store: 4-byte stores between single elements need half as many, and branches that take longer.
// Measured, 2048 tokens 4096 -> 28673 prepared, token-major: 8 single halves per thread, 16 bytes apart, 460 us; a
// loop of 2-byte stores 390; 4-byte stores with branches 402; this 341 (28672: 335).
template <int P>
__device__ __forceinline__ void store_run(__half* dst, uint32_t src, int count, int lane, const float (&scale)[P]) {
  float v[P];
#pragma unroll
  for (int k = 0; k < P; ++k) v[k] = lds_f1(src + (lane + 32 * k) * 4);
#pragma unroll
  for (int k = 0; k < P; ++k)
    if (lane + 32 * k < count) dst[lane + 32 * k] = __float2half_rn(v[k] * scale[k]);
}

template <bool PREP>
__global__ void __launch_bounds__(THREADS, 1)
prefill_wide_gemm_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_wh,
                         const pre::Params p) {
  using L = Layout;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* sm = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* w_full = reinterpret_cast<uint64_t*>(sm + L::bars);   // [STAGES] packed weights have landed
  // everything the MMAs of ring entry q need is in place: operand tiles, and the accumulator has been folded
  uint64_t* ready = w_full + STAGES;                              // [STAGES]
  uint64_t* done = ready + STAGES;                                // [STAGES] the MMAs of entry q have completed
  uint64_t* z_free = done + STAGES;                               // [STAGES] the helper warps may fill this slot
  uint64_t* tab_full = z_free + STAGES;                           // [2]
  uint64_t* tab_empty = tab_full + 2;                             // [2]
  uint64_t* z_done = tab_empty + 2;                               // all zero-point products have completed
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(z_done + 1);

  grid_launch_dependents();
#ifdef W4A4_TRACE
  const long long t_start = clock64();
#endif
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // CTA order: bands of `band` token tiles, token tile first (see prefill_gemm_kernel)
  const int lin = blockIdx.x + blockIdx.y * gridDim.x;
  const int per_band = gridDim.x * p.band;
  const int band_i = lin / per_band, band_rem = lin - band_i * per_band;
  const int band_h = min(p.band, (int)gridDim.y - band_i * p.band);
  const int r = band_rem / band_h;
  const int row0 = r * ROWS;
  const int tok0 = (band_i * p.band + band_rem % band_h) * TN;
  const int live = min(TN, p.T - tok0);           // tokens of this tile
  const int n_mma = (live + 15) & ~15;            // columns that are copied and multiplied

  if (tid == 0) {
    for (int i = 0; i < STAGES; ++i) {
      mbar_init(&w_full[i], 1);
      mbar_init(&ready[i], (PREP ? 2 : 1 + N_HELP) + N_FOLD);
      mbar_init(&done[i], 1);
      mbar_init(&z_free[i], 1);
    }
    mbar_init(z_done, 1);
    for (int i = 0; i < 2; ++i) { mbar_init(&tab_full[i], N_HELP); mbar_init(&tab_empty[i], N_FOLD); }
    mbar_fence_init();
    tma_prefetch_desc(&tm_w);
    tma_prefetch_desc(&tm_wh);
  }
  if (warp == WARP_MMA) pre::tmem_alloc(tmem_slot, pre::TMEM_COLS);
  pre::tc_fence_before();
  __syncthreads();
  pre::tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  int b_lo = 0, b_hi = 0;
  if (p.sparse_on) {
    b_lo = ld_plain(p.hp_row_offsets + r);
    b_hi = ld_plain(p.hp_row_offsets + r + 1);
  }
  const int n_steps = p.nd + (b_hi - b_lo);
  // ring entries 0 .. n_steps - 1 are K-steps, n_steps .. n_steps + n_z - 1 the zero-point products
  const int n_z = p.sumxf != nullptr ? (p.nd + TAB - 1) / TAB : 0;
  bool ok = true;                                 // no wait of this thread has given up

  if (warp < WARP_HELP0) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REG_ISSUE));
    if (warp == WARP_W && lane == 0) {
      // ---------------------------------------------------------- weight copies
      int s = 0;
      uint32_t ph = 1;
      for (int n = 0; n < n_steps; ++n) {
        // From here on this role waits for MMAs, and they for the preceding kernel's output: that time is not
        // this kernel's, so no bounded wait runs during it (here and in the roles below).
        if (n == STAGES) grid_dependency_wait();
        if (n >= STAGES) ok = wait_suspend(&done[s], ph, SITE_WIDE_W);
        if (!ok) break;
        uint64_t* bar = PREP ? &ready[s] : &w_full[s];
        TRACE(0, n);
        mbar_arrive_expect_tx(bar, PREP ? W_BYTES : W_BYTES / 2);
        if (n < p.nd) tma_load_2d(sm + s * SLOT, &tm_w, n * (PREP ? BCOL : GROUP_BYTES), row0, bar);
        else          tma_load_2d(sm + s * SLOT, &tm_wh, 0, (b_lo + n - p.nd) * BROW, bar);
        if (++s == STAGES) { s = 0; ph ^= 1; }
      }
    } else if (warp == WARP_X && lane == 0) {
      // ---------------------------------------------------------- activation copies
      grid_dependency_wait_for_async_reads();     // the expanded codes are written by the preceding kernel
      const int8_t* src0 = p.XE + (size_t)tok0 * BCOL;
      const size_t gstride = (size_t)p.t_pad * BCOL;
      const uint32_t bytes = (uint32_t)n_mma * BCOL;     // rows up to the 16-token padding: inside the buffer
      int s = 0;
      uint32_t ph = 1;
      for (int n = 0; n < n_steps; ++n) {
        const int g = n < p.nd ? n : ld_plain(p.hp_col_indices + b_lo + n - p.nd);
        if (n >= STAGES) ok = wait_suspend(&done[s], ph, SITE_WIDE_X);
        if (!ok) break;
        TRACE(1, n);
        mbar_arrive_expect_tx(&ready[s], bytes);
        bulk_load_1d(sm + s * SLOT + W_BYTES, src0 + g * gstride, bytes, &ready[s]);
        if (++s == STAGES) { s = 0; ph ^= 1; }
      }
      // The entries the helper warps fill.  They do not follow the ring from step to step, so a wait of theirs on
      // a `done` barrier could mistake an earlier phase for the one it means; this thread walks the ring in
      // order and passes every free slot on through a barrier that completes once per use.
      for (int q = n_steps; ok && q < n_steps + n_z; ++q) {
        if (q >= STAGES) ok = wait_suspend(&done[s], ph, SITE_WIDE_X);
        if (ok) mbar_arrive(&z_free[s]);
        if (++s == STAGES) { s = 0; ph ^= 1; }
      }
    } else if (warp >= WARP_MMA && lane == 0) {
      // ---------------------------------------------------------- MMA issuers: even and odd K-steps
      const int par = warp - WARP_MMA;
      const uint32_t ncol = (uint32_t)(n_mma >> 3) << 17;
      const uint64_t a0 = pre::smem_desc_sw128(sm), b0 = pre::smem_desc_sw128(sm + W_BYTES);
      int s = par, buf = par;
      uint32_t ph = 0;
      grid_dependency_wait();
      for (int n = par; n < n_steps; n += 2) {
        ok = wait_suspend(&ready[s], ph, SITE_WIDE_READY);
        if (!ok) break;
        pre::tc_fence_after();
        TRACE(2, n);
        const uint64_t off = (uint64_t)(s * (SLOT >> 4));
        const uint32_t d = tmem_base + buf * TN;
#pragma unroll
        for (int j = 0; j < 4; ++j) pre::umma_f8(d, a0 + off + 2 * j, b0 + off + 2 * j, j > 0, IDESC_F8_M | ncol);
        pre::umma_commit(&done[s]);
        TRACE(3, n);
        s += 2;
        if (s >= STAGES) { s -= STAGES; ph ^= 1; }
        buf += 2;
        if (buf >= ACC_BUFS) buf -= ACC_BUFS;
      }
      // zero-point products: entry n_steps belongs to the thread of its parity, which now stands at it
      if (ok && (n_steps & 1) == par) {
        const uint32_t d = tmem_base + buf * TN;
        for (int k = 0; k < n_z; ++k) {
          ok = wait_suspend(&ready[s], ph, SITE_WIDE_Z);
          if (!ok) break;
          pre::tc_fence_after();
          const uint64_t off = (uint64_t)(s * (SLOT >> 4));
#pragma unroll
          for (int j = 0; j < 4; ++j) pre::umma_tf32(d, a0 + off + 2 * j, b0 + off + 2 * j, (k > 0 || j > 0) ? 1u : 0u, IDESC_TF32_M | ncol);
          pre::umma_commit(&done[s]);
          if (k == n_z - 1) pre::umma_commit(z_done);
          if (++s == STAGES) { s = 0; ph ^= 1; }
        }
      }
    }
  } else if (warp < WARP_FOLD0) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REG_HELP));
    // ------------------------------------------------------------ helper warps: thread = weight row
    const int hr = tid - WARP_HELP0 * 32;
    const int row = row0 + hr;
    const uint32_t ring_a = smem_u32(sm), tab_a = smem_u32(sm + L::tab);
    const int n_tab = (n_steps + TAB - 1) / TAB;
    const __half* srow = p.scale_u4 + (size_t)min(row, p.N - 1) * p.ng;
    const bool row_live = row < p.N;
    // scale factors of the 16 steps of table k: dense groups in order, then the residual blocks' groups
    auto load_tab = [&](int k, float (&f)[TAB]) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int n0 = k * TAB + 8 * h;
        if (p.sz_vec && n0 + 8 <= p.nd) {
          const uint4 v = ld_plain(reinterpret_cast<const uint4*>(srow + n0));
          const __half2* hv = reinterpret_cast<const __half2*>(&v);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float2 t = __half22float2(hv[i]);
            f[8 * h + 2 * i] = t.x;
            f[8 * h + 2 * i + 1] = t.y;
          }
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int n = n0 + i;
            float v = 0.f;
            if (n < p.nd) v = __half2float(ld_plain(srow + n));
            else if (n < n_steps) v = __half2float(ld_plain(srow + ld_plain(p.hp_col_indices + b_lo + n - p.nd))) * p.sparse_weight;
            f[8 * h + i] = v;
          }
        }
      }
    };
    auto store_tab = [&](int k, const float (&f)[TAB]) {
      if (PREP && k == 2) grid_dependency_wait();          // packed weights: after the step STAGES, below
      if (ok && k >= 2) ok = __all_sync(0xffffffffu, wait_suspend(&tab_empty[k & 1], ((k >> 1) - 1) & 1, SITE_WIDE_TAB));
      if (!ok) return;
#pragma unroll
      for (int i = 0; i < TAB; ++i) sts_f1(tab_a + (((k & 1) * TAB + i) * ROWS + hr) * 4, row_live ? f[i] : 0.f);
      __syncwarp();
      if (lane == 0) mbar_arrive(&tab_full[k & 1]);
    };
    float f[TAB];
    if (n_tab > 0) load_tab(0, f);
    if (PREP) {
      for (int k = 0; k < n_tab; ++k) {
        store_tab(k, f);
        if (k + 1 < n_tab) load_tab(k + 1, f);
      }
    } else {
      int s = 0;
      uint32_t ph = 0;
      for (int n = 0; n < n_steps; ++n) {
        if ((n & (TAB - 1)) == 0) {
          store_tab(n / TAB, f);
          if (n / TAB + 1 < n_tab) load_tab(n / TAB + 1, f);
        }
        if (n == STAGES) grid_dependency_wait();           // the first STAGES weight copies depend on nothing
        if (ok) ok = __all_sync(0xffffffffu, wait_suspend(&w_full[s], ph, SITE_WIDE_PACKED));
        const uint32_t slot = ring_a + s * SLOT;
        // the row's 64 packed bytes: 16-byte chunks stored at chunk ^ ((row >> 1) & 3) by the 64-byte swizzle
        uint4 w[4];
        if (ok) {
#pragma unroll
          for (int c = 0; c < 4; ++c) w[c] = lds_v4(slot + hr * GROUP_BYTES + ((c ^ ((hr >> 1) & 3)) << 4));
        }
        asm volatile("bar.sync 2, %0;" ::"n"(N_HELP * 32) : "memory");      // every row has been read
        if (ok) {
          // codes in their natural order; operand row of 128 bytes, chunk c at c ^ (row & 7)
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            uint4 lo, hi;
            nib8_to_e4m3(w[c].x, lo.x, lo.y);
            nib8_to_e4m3(w[c].y, lo.z, lo.w);
            nib8_to_e4m3(w[c].z, hi.x, hi.y);
            nib8_to_e4m3(w[c].w, hi.z, hi.w);
            sts_v4(slot + hr * BCOL + (((2 * c) ^ (hr & 7)) << 4), lo);
            sts_v4(slot + hr * BCOL + (((2 * c + 1) ^ (hr & 7)) << 4), hi);
          }
          fence_proxy_async_smem();
        }
        __syncwarp();
        if (ok && lane == 0) mbar_arrive(&ready[s]);
        if (++s == STAGES) { s = 0; ph ^= 1; }
      }
    }
    // ------------------------------------------------------------ operand tiles of the zero-point products
    // A: the weight row's scale * zero of 16 groups (exact in fp32), split into two 11-bit halves; B: the tokens'
    // group sums (below 2^11), twice - all of them tf32 values.  Rows of 32 values, 16-byte chunks swizzled by row.
    if (n_z > 0) grid_dependency_wait();          // the group sums are written by the preceding kernel
    for (int k = 0; k < n_z; ++k) {
      const int s = (n_steps + k) % STAGES, g0 = k * TAB;
      float c16[TAB];
#pragma unroll
      for (int i = 0; i < TAB; ++i) {
        const bool in = row_live && p.zero_u4 != nullptr && g0 + i < p.ng;
        c16[i] = in ? __half2float(ld_plain(srow + g0 + i)) * __half2float(ld_plain(p.zero_u4 + (size_t)row * p.ng + g0 + i)) : 0.f;
      }
      if (ok) ok = __all_sync(0xffffffffu, wait_suspend(&z_free[s], (k / STAGES) & 1, SITE_WIDE_Z));
      const uint32_t at = ring_a + s * SLOT, bt = at + W_BYTES;
      if (ok) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          float hi[4], lo[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            hi[i] = __uint_as_float(__float_as_uint(c16[4 * c + i]) & 0xFFFFE000u);
            lo[i] = c16[4 * c + i] - hi[i];
          }
          sts_v4(at + hr * 128 + ((c ^ (hr & 7)) << 4),
                 make_uint4(__float_as_uint(hi[0]), __float_as_uint(hi[1]), __float_as_uint(hi[2]), __float_as_uint(hi[3])));
          sts_v4(at + hr * 128 + (((c + 4) ^ (hr & 7)) << 4),
                 make_uint4(__float_as_uint(lo[0]), __float_as_uint(lo[1]), __float_as_uint(lo[2]), __float_as_uint(lo[3])));
        }
#pragma unroll
        for (int h = 0; h < TN / 128; ++h) {
          const int t = h * 128 + hr, tok = tok0 + t;
          if (t >= n_mma) continue;
          float v[TAB];
#pragma unroll
          for (int i = 0; i < TAB; ++i)
            v[i] = (tok < p.T && g0 + i < p.ng) ? ld_plain(p.sumxf + ((size_t)(tok >> 4) * p.ng + g0 + i) * 16 + (tok & 15)) : 0.f;
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const uint4 u = make_uint4(__float_as_uint(v[4 * c]), __float_as_uint(v[4 * c + 1]), __float_as_uint(v[4 * c + 2]), __float_as_uint(v[4 * c + 3]));
            sts_v4(bt + t * 128 + ((c ^ (t & 7)) << 4), u);
            sts_v4(bt + t * 128 + (((c + 4) ^ (t & 7)) << 4), u);
          }
        }
        fence_proxy_async_smem();
      }
      asm volatile("bar.sync 2, %0;" ::"n"(N_HELP * 32) : "memory");
      // in the place of the copies and helper arrivals of a K-step, and of the fold warps' once those have no step left
      if (ok && hr == 0) mbar_arrive_n(&ready[s], (PREP ? 2 : 1 + N_HELP) + (k >= ACC_BUFS ? N_FOLD : 0));
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REG_FOLD));
    // ------------------------------------------------------------ fold warps
    const int ft = tid - WARP_FOLD0 * 32;
    const int quarter = warp & 3;                 // TMEM lanes this warp may read
    const int c0 = ((warp - WARP_FOLD0) >> 2) * COLS;
    const int rl = quarter * 32 + lane;
    float* sxs = reinterpret_cast<float*>(sm + L::sxs);
    const uint32_t tab_a = smem_u32(sm + L::tab);
    const uint32_t t_lane = tmem_base + ((uint32_t)(quarter * 32) << 16) + c0;
    // Last ring entry.  The first zero-point product needs a free accumulator; the fold warps arrive for the first
    // ACC_BUFS of them all the same, so that the ring cannot lap a fold warp that is still at the last K-steps.
    const int last_q = n_steps + n_z - 1;
    grid_dependency_wait();
    for (int i = ft; i < TN; i += N_FOLD * 32)
      sxs[i] = (tok0 + i < p.T && p.scale_x) ? __half2float(ld_plain(p.scale_x + tok0 + i)) : 0.f;

    float y[COLS];
#pragma unroll
    for (int i = 0; i < COLS; ++i) y[i] = 0.f;
    // the accumulators start out free
    if (lane == 0)
      for (int i = 0; i < ACC_BUFS && i <= last_q; ++i) mbar_arrive(&ready[i]);
    int s = 0, s_next = ACC_BUFS % STAGES, buf = 0;
    uint32_t ph = 0;
#pragma unroll 1
    for (int n = 0; n < n_steps; ++n) {
      const int k = n / TAB, j = n & (TAB - 1);
      if (j == 0 && ok) ok = __all_sync(0xffffffffu, wait_suspend(&tab_full[k & 1], (k >> 1) & 1, SITE_WIDE_TAB));
      const float f = lds_f1(tab_a + (((k & 1) * TAB + j) * ROWS + rl) * 4);
      if (ok) ok = __all_sync(0xffffffffu, wait_suspend(&done[s], ph, SITE_WIDE_ACC));
      if (ft == 0) TRACE(4, n);
      if (ok) {
        pre::tc_fence_after();
        // Straight-line code: columns past the live tokens are folded too (into sums nobody stores), because branches
        // between the pieces cost more than they save - the schedulers then wait for instructions.
#pragma unroll
        for (int cc = 0; cc < COLS; cc += 32) {
          uint32_t a[32];
          pre::tmem_ld32(t_lane + buf * TN + cc, a);
          if (cc + 32 == COLS) {
            // the accumulator has been read: it belongs to step n + ACC_BUFS from here on
            pre::tc_fence_before();
            __syncwarp();
            if (lane == 0 && n + ACC_BUFS <= last_q) mbar_arrive(&ready[s_next]);
          }
#pragma unroll
          for (int i = 0; i < 32; ++i) y[cc + i] = __fmaf_rn(__uint_as_float(a[i]), f, y[cc + i]);
        }
        if (j == TAB - 1) {
          __syncwarp();
          if (lane == 0) mbar_arrive(&tab_empty[k & 1]);
        }
      }
      if (ft == 0) TRACE(5, n);
      if (++s == STAGES) { s = 0; ph ^= 1; }
      if (++s_next == STAGES) s_next = 0;
      if (++buf == ACC_BUFS) buf = 0;
    }
    if (n_z > 0) {
      if (ok) ok = __all_sync(0xffffffffu, wait_suspend(z_done, 0, SITE_WIDE_ACC));
      if (ok) {
        pre::tc_fence_after();
#pragma unroll
        for (int cc = 0; cc < COLS; cc += 32) {
          uint32_t a[32];
          pre::tmem_ld32(t_lane + buf * TN + cc, a);
#pragma unroll
          for (int i = 0; i < 32; ++i) y[cc + i] = __fsub_rn(y[cc + i], __uint_as_float(a[i]));
        }
      }
    }
    if (ft == 0) TRACE(6, 0);
    // ------------------------------------------------------------ epilogue
    // The ring has no copy or MMA in flight any more: it takes the tile's sums, in the order the output has in
    // memory, and a rolled loop of 16-byte stores drains them (storing straight from the registers is 128
    // two-byte stores per thread and several times the code, executed once: about 12000 clk on this tile).
    // Where the output's rows do not all start on 16 bytes, a warp stores a row of the tile at a time (store_run).
    const uint32_t stage = smem_u32(sm);
    asm volatile("bar.sync 1, %0;" ::"n"(N_FOLD * 32) : "memory");       // every fold warp has seen the last MMAs complete
    if (p.y_stride_n == 1) {
      // token-major: [token][128 rows]
#pragma unroll
      for (int i = 0; i < COLS; ++i) sts_f1(stage + ((c0 + i) * ROWS + rl) * 4, y[i]);
      asm volatile("bar.sync 1, %0;" ::"n"(N_FOLD * 32) : "memory");
      const bool vec = (p.y_stride_t & 7) == 0 && (reinterpret_cast<uintptr_t>(p.Y) & 15) == 0;
      if (!vec) {
        const int count = min(ROWS, p.N - row0);
#pragma unroll 2
        for (int t = warp - WARP_FOLD0; ok && t < live; t += N_FOLD) {
          const float sx[ROWS / 32] = {sxs[t], sxs[t], sxs[t], sxs[t]};
          store_run<ROWS / 32>(p.Y + (size_t)(tok0 + t) * p.y_stride_t + row0, stage + t * ROWS * 4, count, lane, sx);
        }
      }
#pragma unroll 1
      for (int i = ft; vec && ok && i < live * (ROWS / 8); i += N_FOLD * 32) {
        const int t = i >> 4, r8 = (i & 15) * 8;
        const float4 u = lds_f4(stage + (t * ROWS + r8) * 4), v = lds_f4(stage + (t * ROWS + r8 + 4) * 4);
        const float sx = sxs[t];
        __align__(16) __half2 h[4] = {__floats2half2_rn(u.x * sx, u.y * sx), __floats2half2_rn(u.z * sx, u.w * sx),
                                      __floats2half2_rn(v.x * sx, v.y * sx), __floats2half2_rn(v.z * sx, v.w * sx)};
        // (the stride, N, is a multiple of 8: no ragged eight)
        if (row0 + r8 < p.N) *reinterpret_cast<uint4*>(p.Y + (size_t)(tok0 + t) * p.y_stride_t + row0 + r8) = *reinterpret_cast<uint4*>(h);
      }
    } else {
      // row-major: [row][TN tokens], consecutive rows 4 banks apart
      constexpr int PITCH = TN + 4;
#pragma unroll
      for (int i = 0; i < COLS; i += 4)
        sts_v4(stage + (rl * PITCH + c0 + i) * 4, make_uint4(__float_as_uint(y[i]), __float_as_uint(y[i + 1]), __float_as_uint(y[i + 2]), __float_as_uint(y[i + 3])));
      asm volatile("bar.sync 1, %0;" ::"n"(N_FOLD * 32) : "memory");
      const bool vec = (p.y_stride_n & 7) == 0 && (reinterpret_cast<uintptr_t>(p.Y) & 15) == 0;
      const int rows = min(ROWS, p.N - row0);
      if (!vec) {
        float sx[TN / 32];
#pragma unroll
        for (int k = 0; k < TN / 32; ++k) sx[k] = sxs[lane + 32 * k];
#pragma unroll 2
        for (int q = warp - WARP_FOLD0; ok && q < rows; q += N_FOLD)
          store_run<TN / 32>(p.Y + (size_t)(row0 + q) * p.y_stride_n + tok0, stage + q * PITCH * 4, live, lane, sx);
      }
#pragma unroll 1
      for (int i = ft; vec && ok && i < rows * (TN / 8); i += N_FOLD * 32) {
        const int q = i / (TN / 8), t8 = (i % (TN / 8)) * 8;
        if (t8 >= live) continue;
        const float4 u = lds_f4(stage + (q * PITCH + t8) * 4), v = lds_f4(stage + (q * PITCH + t8 + 4) * 4);
        const float4 a = lds_f4(smem_u32(sxs + t8)), b = lds_f4(smem_u32(sxs + t8 + 4));
        __align__(16) __half2 h[4] = {__floats2half2_rn(u.x * a.x, u.y * a.y), __floats2half2_rn(u.z * a.z, u.w * a.w),
                                      __floats2half2_rn(v.x * b.x, v.y * b.y), __floats2half2_rn(v.z * b.z, v.w * b.w)};
        // (the stride, T, is a multiple of 8: no ragged eight)
        *reinterpret_cast<uint4*>(p.Y + (size_t)(row0 + q) * p.y_stride_n + tok0 + t8) = *reinterpret_cast<uint4*>(h);
      }
    }
  }

#ifdef W4A4_TRACE
  if (tid == WARP_FOLD0 * 32) { TRACE(8, 0); if (lin == p.trace_cta) p.trace[8 * 64 + 1] = t_start; }
#endif
  // Common exit: every role falls through to here, then the allocating warp frees tensor memory.  After a wait that
  // gave up copies and MMAs may still be in flight, on barriers that also count arrivals which will not come: the
  // block then stays for a millisecond, many times what they need, before its memory is handed on.
  pre::tc_fence_before();
  if (__syncthreads_or(!ok)) {
    if (tid == 0)
      for (const uint64_t t0 = timer_ns(); timer_ns() - t0 < 1000000;) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == WARP_MMA) {
    pre::tc_fence_after();
    pre::tmem_dealloc(tmem_base, pre::TMEM_COLS);
  }
}

}  // namespace wide
}  // namespace w4a4
