// FP64 grouped block GEMM on the tensor cores (sm_103a) by error-free slicing (Ozaki,
// Ogita, Oishi, Rump 2012: "Error-free transformations of matrix multiplication").
//
// GB300's FP64 pipe does 2.1 fused multiply-adds per clock and SM, its tensor cores two
// thousand times as many in bf16.  An operand row is scaled by a power of two 2^e to its
// largest magnitude (|x| < 2^e) and cut into seven signed base-256 digits,
//   x = 2^e sum_p d_p 2^(-7 - 8 (p - 1)),  |d_p| <= 128,
// each exact in bf16: 56 bits under the row maximum.  Digit products d_p d_q are summed
// exactly by the FP32 accumulators, all products of one weight (p + q = t + 2, t = 0..7)
// in one accumulator: at most 7 x 160 products of 2^14 for a contraction of 160, below
// 2^24 but for the last weights, where a rounding is under the dropped products.  The 34
// products with p + q <= 9 are kept.  An operand is off by at most half a unit of 2^(e-55) (e
// the exponent of its row), the sum of a group of 160 by half a unit of 2^(e-55) (e the sum of
// both exponents), what is dropped is below 2^-61 of 2^e: a sum of K products by at most
// K 2^-53 of (row maximum x column maximum).  FP64 multiply-adds are off by at most K 2^-53 of
// the sum of magnitudes, which is less where large elements of a row meet small ones of a
// column.
//
// Contractions are balanced for that reason: the elements at k are multiplied by 2^s_k in
// one operand and 2^-s_k in the other while they are sliced, s_k the exponent of the largest
// magnitude at k of the wavefunction (for both of its indices) or of a site tensor
// (oz_scale_kernel).  Largest error of an element of H_eff*psi relative to its sum of magnitudes,
// without / with / FP64 pipe: on converged Hubbard bonds (M=32, 64) 5e-13 .. 6e-10 / 1.4e-15 ..
// 1e-13 / 2.5e-16; on wavefunctions graded over four decades, Hubbard M=33..101 5e-15 .. 1e-14 /
// 3e-16 .. 7e-16 / 3e-16 .. 5e-16, QC M=40, 60 2e-16 / 2e-16 / 5e-16; rms values below the FP64
// pipe's but for the converged bonds (1e-16 .. 6e-15 / 5e-17).  It costs the launch of the maxima
// and 6 of some 50 instructions an element of the packing: 55 -> 57 us at Hubbard M=64, 136 -> 143
// at M=512, 7.68 -> 7.92 ms at QC n=20 M=512.  An eigenproblem, whose operators are sliced once and
// whose vectors enter through norms and dot products, does not balance.
//
// A K step of 16 is seven MMAs: digit p of A times the stacked digits [B_1; ..; B_n] as
// one operand, written at the accumulator columns of weight p - 1, so that every product
// lands in its weight's columns: A_1 and A_2 take all seven digits of B, A_p 9 - p.
// What bounds the kernel is shared memory (operand reads of the MMAs and the bulk copies),
// hence wide MMAs; a 128 x 32 tile keeps two accumulators of 8 x 32 columns, so that the
// epilogue (integer recombination and three FP64 additions per element) runs while the
// next group of K steps issues.
//
// H_eff*psi at the C2 size (QC n=20 M=512, 88 GFLOP): 91.5 ms on the FP64 pipe (0.96 TFLOP/s,
// 89 % of cuBLAS DGEMM), 7.9 ms sliced (11 TFLOP/s; GEMMs 5.5 ms, packing 2.4), 143 us against
// 1.25 ms at Hubbard M=512.
//
// GEMM CTA (640 threads, warp-specialised, persistent over the tile list): warp 0 lane 0
// copies operand slices (one bulk copy each of A and B per K step) into a six-stage
// ring; warp 1 lane 0 issues the MMAs; warps 4-19 are the epilogue (warp 4 + 4 c + q:
// tensor-memory lanes 32 q.., output columns 8 c..).
//
// A row with a value that is not finite or of 2^480 and above, or of values below 2^-480 that
// are not all zero, sets the operand's flag; the kernel then computes its tiles from the FP64
// operands directly (plain loops: such operands do not occur in a converging sweep, but give
// what FP64 arithmetic gives).
#include <cuda_runtime.h>

#include <cstdint>

#include "kernels.hpp"
#include "launch.hpp"
#include "tc.hpp"

namespace mpsxx {

namespace {

constexpr int OM = kOzTileM, ON = kOzTileN, OKS = kOzTileK, ND = kOzDigits, NW = 8;
constexpr int NTHREADS = 640;
constexpr int EPI_THREADS = 512;  // warps 4-19
constexpr int EPI_COLS = 8;       // output columns of an epilogue warp
constexpr int STAGES = 6;
constexpr uint32_t A_BYTES = ND * OM * OKS * 2;  // 28 KB
constexpr uint32_t B_BYTES = ND * ON * OKS * 2;  // 7 KB
constexpr uint32_t STAGE_BYTES = A_BYTES + B_BYTES;
// Row and column exponents of a pair, copied with its first slice into a slot with its own
// "landed" barrier.  When a pair's copy is issued, at most STAGES + 3 pairs (ring and
// accumulators) are between it and the last one that the epilogue has finished, so that the
// slot, last used EXP_SLOTS pairs ago, is free without another barrier.
constexpr int EXP_SLOTS = 16;
static_assert(EXP_SLOTS > STAGES + 3, "a pair's exponents would be overwritten while in use");
constexpr uint32_t EXP_BYTES = (OM + ON) * 4;
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + EXP_SLOTS * EXP_BYTES + 1024;
constexpr uint32_t ACC_COLS = NW * ON;  // 256
constexpr uint32_t TMEM_COLS = 2 * ACC_COLS;

__host__ __device__ constexpr uint32_t bf16_idesc(int m, int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

__device__ __forceinline__ void mma_bf16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
      "l"(a), "l"(b), "r"(idesc), "r"(acc));
}

// K steps of a pair's groups: as even as possible, at most kOzGroupSteps each
__device__ __forceinline__ int group_steps(int nks) {
  const int ng = (nks + kOzGroupSteps - 1) / kOzGroupSteps;
  return (nks + ng - 1) / ng;
}

// The weights' integer sums of one element -> its value 2^(e - 55) S rounded to FP64; ew
// is e << 20 (e = row exponent + column exponent).  S is exact but for the two lowest
// weights' bits under 1 (rounded).  All in integer arithmetic: the FP64 pipe (15 clocks of
// an SM per warp instruction) takes only the additions to the running sums.
__device__ __forceinline__ double oz_value(const float (&v)[NW], int ew) {
  int a[5];
#pragma unroll
  for (int t = 0; t < 5; ++t) a[t] = __float2int_rn(v[t]);
  const float z = fmaf(fmaf(v[7], 0x1p-8f, v[6]), 0x1p-7f, 2.0f * v[5]);
  const int ht = a[0] * 256 + a[1], hl = a[2] * 256 + a[3];
  long long S = (long long)__float2int_rn(z) + (long long)a[4] * 512;
  S += (long long)hl * 131072;
  S += (long long)((unsigned long long)(uint32_t)ht << 33);
  // normalise |S| to 64 bits, round to 53, place the exponent
  const int neg = (int)(S >> 63);
  const unsigned long long u = (unsigned long long)((S ^ (long long)neg) - (long long)neg);
  const int n = __clzll((long long)u);
  const unsigned long long m = ((u << n) >> 11) + ((u << n) >> 10 & 1);  // (a carry out of 53 bits moves the exponent)
  const int hi = (int)(m >> 32) + ew + ((1085 - 55 - n) << 20);
  return u == 0 ? 0.0 : __hiloint2double(hi | (neg & (int)0x80000000u), (int)(uint32_t)m);
}

__device__ __forceinline__ void oz_store(double* dst, double v, int assign) {
  if (assign)
    *dst = v;
  else
    *dst += v;
}

// First element of a tile of a tiled intermediate (DOzTiled).
__device__ __forceinline__ int64_t oz_tile_off(const DOzTiled& p, int tm, int tn) {
  return p.base + ((int64_t)tm * p.ntn + tn) * (OM * ON);
}

// Tile from the FP64 operands by plain sums (flagged operands).
__device__ void oz_plain_tile(const DTile& t, const OzGemmArgs& g) {
  for (int e = threadIdx.x; e < OM * ON; e += blockDim.x) {
    const int row = e / ON, col = e % ON;
    if (col >= t.nt || row >= t.h64) continue;
    int task = t.task, r = t.tm * OM + row, p0 = t.p0, p1 = t.p1;
    if (g.row_map != nullptr) {
      const int64_t m = g.row_map[(int64_t)g.pairs[t.p0].map + r];
      if (m < 0) continue;
      task = static_cast<int>(m >> 32);
      r = static_cast<int>(m & 0xffffffffll);
      p0 = g.tasks[task].p0;
      p1 = p0 + 1;
    }
    const DGemmTask tk = g.tasks[task];
    const int c = t.tn * ON + col;
    const int i = g.swap ? c : r, j = g.swap ? r : c;  // element of the task's result
    double s = 0.0;
    if (i < tk.m && j < tk.n)
      for (int p = p0; p < p1; ++p) {
        const DGemmPair pr = g.fpairs[p];
        for (int k = 0; k < pr.k; ++k) {
          double a;
          if (g.tiled_in) {
            const DOzTiled tl = g.pairs_tiled[p];
            const int pr_row = tl.row0 + i;
            a = g.A[oz_tile_off(tl, pr_row / OM, k / ON) + (pr_row % OM) * ON + k % ON];
          } else {
            a = g.ta ? g.A[pr.a_off + (int64_t)k * pr.lda + i] : g.A[pr.a_off + (int64_t)i * pr.lda + k];
          }
          const double b = g.tb ? g.B[pr.b_off + (int64_t)j * pr.ldb + k] : g.B[pr.b_off + (int64_t)k * pr.ldb + j];
          s = fma(a, b, s);
        }
      }
    if (g.tiled_out)
      g.C[oz_tile_off(g.pairs_tiled[t.p0], t.tm, t.tn) + e] = s;
    else if (t.slot >= 0)
      g.partial[(int64_t)t.slot * (OM * ON) + e] = s;
    else if (i < tk.m && j < tk.n)
      oz_store(g.C + tk.c_off + (int64_t)i * tk.ldc + j, g.alpha * s, g.assign);
  }
}

__global__ void __launch_bounds__(NTHREADS, 1) gemm_oz_kernel(const OzGemmArgs g) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* exps = ring + STAGES * STAGE_BYTES;
  __shared__ __align__(8) uint64_t full_bar[STAGES];
  __shared__ __align__(8) uint64_t empty_bar[STAGES];
  __shared__ __align__(8) uint64_t exp_bar[EXP_SLOTS];
  __shared__ __align__(8) uint64_t drain_bar;
  __shared__ __align__(8) uint64_t accf_bar[2];
  __shared__ __align__(8) uint64_t acce_bar[2];
  __shared__ uint32_t tmem_slot;
  __shared__ volatile int abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                 "r"(TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (threadIdx.x == 32) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(smem_u32(&full_bar[s]), 1);
      mbar_init(smem_u32(&empty_bar[s]), 1);
    }
    for (int e = 0; e < EXP_SLOTS; ++e) mbar_init(smem_u32(&exp_bar[e]), 1);
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&accf_bar[b]), 1);
      mbar_init(smem_u32(&acce_bar[b]), EPI_THREADS);
    }
    mbar_init(smem_u32(&drain_bar), 1);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = tmem_slot;
  chain_wait();
  const bool plain = *g.flag_a == g.seq_a || *g.flag_b == g.seq_b;
  const uint64_t deadline = deadline_in(g.timeout_ns);
  // Persistent: the CTA walks its list of tiles (balanced on the host); every role walks the
  // same sequence, so stage and accumulator counters continue across tiles.
  const int ti0 = g.cta_ptr[blockIdx.x], ti1 = plain ? ti0 : g.cta_ptr[blockIdx.x + 1];
  if (plain)
    for (int ti = ti0; ti < g.cta_ptr[blockIdx.x + 1]; ++ti) oz_plain_tile(g.tiles[ti], g);
  if (warp == 0) {
    // ---------------- producer ----------------
    if (lane == 0) {
      int slice = 0, s = 0, np = 0;
      uint32_t ph = 1;  // parity of the stage's "empty" phase to wait for
      DTile t_next = ti0 < ti1 ? g.tiles[ti0] : DTile{};
      for (int ti = ti0; ti < ti1 && !abort_flag; ++ti) {
        const DTile t = t_next;
        if (ti + 1 < ti1) t_next = g.tiles[ti + 1];
        // a tail tile's slices are packed compact; the row tiles before it are full
        const uint32_t at = A_BYTES / OM * t.h64, bt = B_BYTES / ON * t.nt;
        DOzPair pr_next = t.p0 < t.p1 ? g.pairs[t.p0] : DOzPair{};
        for (int p = t.p0; p < t.p1 && !abort_flag; ++p) {
          const DOzPair pr = pr_next;
          if (p + 1 < t.p1) pr_next = g.pairs[p + 1];
          const uint8_t* as = g.Apk + pr.a_pk + (int64_t)t.tm * pr.nks * A_BYTES;
          const uint8_t* bs = g.Bpk + pr.b_pk + (int64_t)t.tn * pr.nks * B_BYTES;
          const uint32_t ae = t.h64 * 4, be = t.nt * 4;
          const uint32_t es = smem_u32(exps + (np % EXP_SLOTS) * EXP_BYTES);
          for (int ks = 0; ks < pr.nks; ++ks) {
            if (!mbar_wait(smem_u32(&empty_bar[s]), ph, deadline, &abort_flag)) break;
            const uint32_t fb = smem_u32(&full_bar[s]);
            if (ks == 0) {
              const uint32_t eb = smem_u32(&exp_bar[np % EXP_SLOTS]);
              mbar_expect_tx(eb, ae + be);
              bulk_g2s(es, g.Aexp + pr.a_exp + t.tm * OM, ae, eb);
              bulk_g2s(es + OM * 4, g.Bexp + pr.b_exp + t.tn * ON, be, eb);
              ++np;
            }
            mbar_expect_tx(fb, at + bt);
            const uint32_t dst = smem_u32(ring + s * STAGE_BYTES);
            bulk_g2s(dst, as + (int64_t)ks * at, at, fb);
            bulk_g2s(dst + A_BYTES, bs + (int64_t)ks * bt, bt, fb);
            ++slice;
            if (++s == STAGES) {
              s = 0;
              ph ^= 1u;
            }
          }
        }
      }
      // every bulk copy issued lands before the kernel exits (after an abort the
      // consumers no longer wait for them): the last STAGES slices' phases
      const uint64_t dl = deadline_in(DRAIN_NS);
      for (int k = slice - STAGES < 0 ? 0 : slice - STAGES; k < slice; ++k)
        mbar_drain(smem_u32(&full_bar[k % STAGES]), (uint32_t)(k / STAGES) & 1u, dl);
      for (int k = np - EXP_SLOTS < 0 ? 0 : np - EXP_SLOTS; k < np; ++k)
        mbar_drain(smem_u32(&exp_bar[k % EXP_SLOTS]), (uint32_t)(k / EXP_SLOTS) & 1u, dl);
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    if (lane == 0) {
      const uint32_t lbo = 128, sbo = 256;  // core matrices: 128 B apart along K, 256 B along rows
      const uint64_t d0 = smem_desc(smem_u32(ring), lbo, sbo);
      int s = 0, gc = 0;
      uint32_t ph = 0;
      bool ok = true;
      DTile t_next = ti0 < ti1 ? g.tiles[ti0] : DTile{};
      for (int ti = ti0; ti < ti1 && ok; ++ti) {
        const DTile t = t_next;
        if (ti + 1 < ti1) t_next = g.tiles[ti + 1];
        const int mt = t.h64 <= 64 ? 64 : OM, nt = t.nt;
        const uint64_t da = (uint64_t)(t.h64 * OKS * 2) >> 4;  // one digit of A
        const uint64_t db6 = (uint64_t)(6 * nt * OKS * 2) >> 4;  // digit 7 of B
        const uint32_t id7 = bf16_idesc(mt, 7 * nt), id6 = bf16_idesc(mt, 6 * nt), id1 = bf16_idesc(mt, nt);
        const uint32_t idstep = (uint32_t)(nt >> 3) << 17;
        int nks_next = t.p0 < t.p1 ? g.pairs[t.p0].nks : 0;
        for (int p = t.p0; p < t.p1 && ok; ++p) {
          const int nks = nks_next;
          if (p + 1 < t.p1) nks_next = g.pairs[p + 1].nks;
          const int gs = group_steps(nks);
          for (int k0 = 0; k0 < nks && ok; k0 += gs, ++gc) {
            const int b = gc & 1;
            if (!mbar_wait(smem_u32(&acce_bar[b]), ((gc >> 1) & 1u) ^ 1u, deadline, &abort_flag)) {
              ok = false;
              break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;");
            const uint32_t d = tmem + b * ACC_COLS;
            const int k1 = k0 + gs < nks ? k0 + gs : nks;
            for (int ks = k0; ks < k1; ++ks) {
              if (!mbar_wait(smem_u32(&full_bar[s]), ph, deadline, &abort_flag)) {
                ok = false;
                break;
              }
              asm volatile("tcgen05.fence::after_thread_sync;");
              const uint64_t a = d0 + ((uint64_t)(s * STAGE_BYTES) >> 4);
              const uint64_t bd = a + (A_BYTES >> 4);
              if (ks == k0) {
                // the group's first step: A_1 starts weights 0..6, A_2 B_7 weight 7
                mma_bf16(d, a, bd, id7, 0u);
                mma_bf16(d + nt, a + da, bd, id6, 1u);
                mma_bf16(d + 7 * nt, a + da, bd + db6, id1, 0u);
              } else {
                mma_bf16(d, a, bd, id7, 1u);
                mma_bf16(d + nt, a + da, bd, id7, 1u);
              }
#pragma unroll
              for (int q = 2; q < ND; ++q) mma_bf16(d + q * nt, a + q * da, bd, id6 - (q - 2) * idstep, 1u);
              mma_commit(smem_u32(&empty_bar[s]));  // stage free once these MMAs completed
              if (++s == STAGES) {
                s = 0;
                ph ^= 1u;
              }
            }
            if (!ok) break;
            mma_commit(smem_u32(&accf_bar[b]));
          }
        }
      }
      // every MMA issued has completed before tensor memory is freed
      mma_commit(smem_u32(&drain_bar));
      mbar_drain(smem_u32(&drain_bar), 0u, deadline_in(DRAIN_NS));
    }
  } else if (warp >= 4) {
    // ---------------- epilogue ----------------
    const int q = (warp - 4) & 3;    // tensor-memory lane quarter (warp id mod 4)
    const int ch = (warp - 4) >> 2;  // output columns [8 ch, 8 ch + 8)
    int gc = 0, np = 0;
    bool ok = true;
    // what a tile needs from global memory is loaded while the tile before it is worked on,
    // one dependent load at a time: the tile, its first pair, the row map, the task
    auto tile_row = [&](const DTile& t) {
      // M = 128: lane 32 q + i holds row 32 q + i; M = 64: row 16 q + i for i < 16
      const int row = t.h64 <= 64 ? (lane < 16 ? q * 16 + lane : OM) : q * 32 + lane;
      return row < t.h64 ? row : -1;
    };
    auto map_row = [&](const DTile& t, const DOzPair& pr) -> int64_t {
      // task << 32 | row of this lane's tile row, -1: none
      const int row = tile_row(t);
      if (row < 0) return -1;
      const int r = t.tm * OM + row;
      return g.row_map != nullptr ? g.row_map[(int64_t)pr.map + r] : (int64_t)t.task << 32 | r;
    };
    DTile t_n = ti0 < ti1 ? g.tiles[ti0] : DTile{};
    DOzPair pr_n = ti0 < ti1 ? g.pairs[t_n.p0] : DOzPair{};
    int64_t m_n = ti0 < ti1 ? map_row(t_n, pr_n) : -1;
    for (int ti = ti0; ti < ti1 && ok; ++ti) {
      const DTile t = t_n;
      const int64_t m = m_n;
      const int nks0 = pr_n.nks;
      const bool more = ti + 1 < ti1;
      if (more) t_n = g.tiles[ti + 1];
      const int nt = t.nt, c0 = EPI_COLS * ch, row = tile_row(t);
      const int r = static_cast<int>(m & 0xffffffffll);
      DGemmTask tk{};
      if (m >= 0) tk = g.tasks[m >> 32];
      bool live = false, work = false;
      double acc[EPI_COLS];
      bool first = true;
      int nks_n = nks0;
      for (int p = t.p0; p < t.p1 && ok; ++p, ++np) {
        const int nks = nks_n, gs = group_steps(nks);
        if (p + 1 < t.p1) nks_n = g.pairs[p + 1].nks;
        if (more && p == t.p0) pr_n = g.pairs[t_n.p0];
        const int* es = reinterpret_cast<const int*>(exps + (np % EXP_SLOTS) * EXP_BYTES);
        for (int k0 = 0; k0 < nks; k0 += gs, ++gc) {
          const int b = gc & 1;
          if (!mbar_wait(smem_u32(&accf_bar[b]), (gc >> 1) & 1u, deadline, &abort_flag)) {
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;");
          if (first) {
            // warps without rows or columns only hand the accumulators back
            live = m >= 0 && r < (g.swap ? tk.n : tk.m);
            work = c0 < nt && __any_sync(0xffffffffu, live);
          }
          if (k0 == 0 && work &&
              !mbar_wait(smem_u32(&exp_bar[np % EXP_SLOTS]), (uint32_t)(np / EXP_SLOTS) & 1u, deadline, &abort_flag)) {
            ok = false;
            break;
          }
          if (work) {
            const int ea = (row >= 0 ? es[row] : 0) << 20;
            const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + b * ACC_COLS + c0;
#pragma unroll
            for (int h = 0; h < EPI_COLS; h += 4) {
              float v[NW][4];
#pragma unroll
              for (int w = 0; w < NW; ++w) tmem_ld4(taddr + w * nt + h, v[w]);
              asm volatile("tcgen05.wait::ld.sync.aligned;");
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                float x[NW];
#pragma unroll
                for (int w = 0; w < NW; ++w) x[w] = v[w][i];
                const double y = oz_value(x, ea + (es[OM + c0 + h + i] << 20));
                acc[h + i] = first ? y : acc[h + i] + y;
              }
            }
          }
          asm volatile("tcgen05.fence::before_thread_sync;");
          mbar_arrive(smem_u32(&acce_bar[b]));
          first = false;
        }
      }
      if (!ok) break;
      if (more) m_n = map_row(t_n, pr_n);
      if (!work || row < 0) continue;
      if (t.slot >= 0 || g.tiled_out) {
        // a whole tile row: 64 contiguous bytes a lane
        double* base = g.tiled_out ? g.C + oz_tile_off(g.pairs_tiled[t.p0], t.tm, t.tn)
                                   : g.partial + (int64_t)t.slot * (OM * ON);
        double2* part = reinterpret_cast<double2*>(base + row * ON + c0);
#pragma unroll
        for (int j = 0; j < EPI_COLS / 2; ++j) part[j] = make_double2(acc[2 * j], acc[2 * j + 1]);
      } else if (live) {
        const int n0 = t.tn * ON + c0, cols = g.swap ? tk.m : tk.n;
        double* dst = g.C + tk.c_off + (g.swap ? (int64_t)n0 * tk.ldc + r : (int64_t)r * tk.ldc + n0);
        const int64_t cs = g.swap ? tk.ldc : 1;
        // all old values before the first store: the compiler cannot tell that the columns do
        // not overlap, and a load after each store would wait for it (a Hubbard M=512 gradient
        // with its two products written that way took 617 us instead of 415)
        double old[EPI_COLS] = {};
        if (!g.assign)
#pragma unroll
          for (int j = 0; j < EPI_COLS; ++j)
            if (n0 + j < cols) old[j] = dst[j * cs];
#pragma unroll
        for (int j = 0; j < EPI_COLS; ++j)
          if (n0 + j < cols) dst[j * cs] = old[j] + g.alpha * acc[j];
      }
    }
  }
  chain_next();
  __syncthreads();
  if (threadIdx.x == 0 && abort_flag) report_timeout(g.err);
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS));
}

// Split-K partials of one tile summed into C in slot order, one thread per valid element.
__global__ void __launch_bounds__(256) oz_reduce_kernel(const DReduce* __restrict__ red, const OzGemmArgs g) {
  chain_wait();
  chain_next();
  const DReduce rd = red[blockIdx.x];
  const DGemmTask tk = g.tasks[rd.task];
  const int rows = g.swap ? tk.n : tk.m, cols = g.swap ? tk.m : tk.n;
  const int m0 = rd.tm * OM, n0 = rd.tn * ON;
  const int vm = min(OM, rows - m0), vn = min(ON, cols - n0);
  const int e = blockIdx.y * blockDim.x + threadIdx.x;
  if (vm <= 0 || vn <= 0 || e >= vm * vn) return;
  constexpr int64_t SLOT = OM * ON;
  const int r = e / vn, c = e - r * vn;
  const double* __restrict__ p = g.partial + (int64_t)rd.slot0 * SLOT + r * ON + c;
  double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
  int k = 0;
  for (; k + 4 <= rd.nslot; k += 4) {
    s0 += p[(k + 0) * SLOT];
    s1 += p[(k + 1) * SLOT];
    s2 += p[(k + 2) * SLOT];
    s3 += p[(k + 3) * SLOT];
  }
  for (; k < rd.nslot; ++k) s0 += p[k * SLOT];
  const int i = g.swap ? n0 + c : m0 + r, j = g.swap ? m0 + r : n0 + c;
  oz_store(g.C + tk.c_off + (int64_t)i * tk.ldc + j, g.alpha * ((s0 + s1) + (s2 + s3)), g.assign);
}

// Exponent that scales a row whose largest magnitude has the biased exponent field m: 0
// for a zero (or subnormal) row.
__device__ __forceinline__ int row_exponent(int m) { return m == 0 ? 0 : max(m - 1022, -kOzMaxExponent); }

// One value's 56-bit fixed point under its row's exponent, rounded to nearest (zeros and
// subnormals shift out), plus the digits' bias.
__device__ __forceinline__ unsigned long long biased56(double x, int e1022) {
  const int hi = __double2hiint(x);
  const unsigned long long m =
      ((unsigned long long)(uint32_t)((hi & 0xfffff) | 0x100000) << 32) | (uint32_t)__double2loint(x);
  const int s = min(e1022 - ((hi >> 20) & 0x7ff), 63);  // x 2^(55 - e) = m 2^(2 - s), s >= 0
  const long long h = (long long)((((m << 3) >> s) + 1) >> 1);
  const long long neg = (long long)(hi >> 31);
  return (unsigned long long)((h ^ neg) - neg) + 0x80808080808080ull;
}

// Packs FP64 rows as digit tiles: a CTA takes up to 128 rows of an operand block over all of K
// (about kOzPackElems elements), finds each row's exponent and writes the digits in the
// K-major core-matrix layout (8 rows x 16 bytes) slice by slice: digit p of a tile's slice k at
// (k ND + p) tile_rows 32 bytes.  A thread holds 8 consecutive K of a row per item, so that a warp
// reads whole sectors and its stores fill 128-byte lines; up to kHold items stay in registers
// between the two steps, what a long row has beyond is read again (from L2).  HBM moves 8 + 14
// bytes per element; the integer pipe works about 50 instructions on one (45 without powers of
// two), which is why the digits are cut by byte permutes and one FP32 addition each.  Neither is
// saturated (HBM 65 %, issue 50 %): warps in flight decide.  Four CTAs an SM (64 registers) against
// three, and against five with one item held, whose second reads cost more: 7.68, 7.88, 7.97 ms
// for H_eff*psi at QC n=20 M=512 (unbalanced).
constexpr int kHold = 2;
template <bool kScaled>
__global__ void __launch_bounds__(256, 4) oz_pack_kernel(const __grid_constant__ OzPackJobs jobs) {
  constexpr int kExp = kScaled ? 16 : 20;  // row_max holds an exponent from this bit on
  __shared__ long long row_off[kOzPackRows];
  __shared__ int row_ks[kOzPackRows];
  __shared__ int row_max[kOzPackRows];
  chain_wait();
  chain_next();
  int first = 0, jb = 0;  // the CTA's operand and its place among that operand's packs
  while (jb + 1 < jobs.n && (int)blockIdx.x - first >= jobs.job[jb].npacks) first += jobs.job[jb++].npacks;
  const OzPackJob& job = jobs.job[jb];
  const DOzSeg* __restrict__ segs = job.segs;
  const double* __restrict__ src = job.src;
  uint8_t* __restrict__ dst = job.dst;
  const DOzPack pk = job.packs[blockIdx.x - first];
  if (threadIdx.x < pk.rows) {
    const int r = threadIdx.x;
    long long off = -1;
    int ks = 1;
    for (int i = 0; i < pk.nseg; ++i) {
      const DOzSeg sg = segs[pk.seg0 + i];
      if (r >= sg.row && r < sg.row + sg.n) {
        off = sg.src_off + (long long)(r - sg.row) * sg.rstride;
        ks = sg.kstride;
      }
    }
    row_off[r] = off;
    row_ks[r] = ks;
    row_max[r] = 0;
  }
  __syncthreads();
  const int G = 2 * pk.nks;  // groups of 8 K
  const int items = pk.rows * G;
  // item -> (row group of 8, K group, row in group)
  auto place = [&](int it, int& r, int& kg) {
    const int rg = (it >> 3) / G;
    r = rg * 8 + (it & 7);
    kg = (it >> 3) - rg * G;
  };
  auto fetch = [&](int r, int kg, double (&x)[8]) {
    const long long off = row_off[r];
    const int ks = row_ks[r], n = off < 0 ? 0 : pk.k - kg * 8;  // elements with data
    if (ks == 0) {  // tiled source: 64 contiguous bytes
      const double2* p = reinterpret_cast<const double2*>(src + off + (long long)(kg >> 2) * (OM * ON) + (kg & 3) * 8);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const double2 y = 2 * i < n ? p[i] : make_double2(0.0, 0.0);
        x[2 * i] = y.x;
        x[2 * i + 1] = 2 * i + 1 < n ? y.y : 0.0;
      }
      return;
    }
    const double* p = src + off + (long long)(kg * 8) * ks;
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = i < n ? p[(long long)i * ks] : 0.0;
  };
  // the 8 powers of two of a K group as bytes
  auto powers = [&](int kg) {
    uint2 p = make_uint2(0, 0);
    if (kScaled) {
      p = *reinterpret_cast<const uint2*>(job.scales + pk.scale + kg * 8);
      if (job.sign < 0) p = make_uint2(__vneg4(p.x), __vneg4(p.y));
    }
    return p;
  };
  auto power = [](const uint2& p, int i) { return (int)(int8_t)((i < 4 ? p.x : p.y) >> (8 * (i & 3))); };
  auto top = [&](const double (&x)[8], int r, int kg) {
    int m = 0, low = 0;
    const uint2 p = powers(kg);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      int h = __double2hiint(x[i]) & 0x7fffffff;
      if (kScaled && h != 0) h = max((h >> 4) + power(p, i) * (1 << kExp), 1);  // (>> 4: room for the largest)
      m = max(m, h);
      low |= __double2loint(x[i]);
    }
    if (m == 0 && low != 0) m = 1;  // (the smallest subnormal numbers)
    if (m) atomicMax(&row_max[r], m);
  };
  auto emit = [&](const double (&x)[8], int r, int kg) {
    const int e1022 = row_exponent(row_max[r] >> kExp) + 1022;
    const uint2 pw = powers(kg);
    uint32_t lo[8], hi[8];  // bytes: digit + 128 (the leading one in the upper 16 bits)
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const unsigned long long d = biased56(x[i], kScaled ? e1022 - power(pw, i) : e1022);
      lo[i] = (uint32_t)d;
      hi[i] = (uint32_t)(d >> 32);
    }
    const int tile = (pk.row0 + r) >> pk.tile_log2, tr = pk.row0 + r - (tile << pk.tile_log2);
    const int tile_rows = tile == pk.last ? pk.tail : 1 << pk.tile_log2;
    uint8_t* out = dst + pk.dst_off +
                   (((long long)tile * pk.nks << pk.tile_log2) + (kg >> 1) * tile_rows) * (ND * OKS * 2) +
                   ((tr >> 3) * 2 + (kg & 1)) * 128 + (tr & 7) * 16;
#pragma unroll
    for (int p = 0; p < ND; ++p) {
      // digit -> 2^23 + 128 + digit as FP32 by placing its byte, minus the constant; an
      // integer of at most 8 bits is exact in bf16: the upper half of its FP32 form
      const uint32_t sel = p == 0 ? 0x7432u : p == 1 ? 0x7441u : p == 2 ? 0x7440u : 0x7440u + (6 - p);
      uint32_t u[8];
#pragma unroll
      for (int i = 0; i < 8; ++i)
        u[i] = __float_as_uint(__uint_as_float(__byte_perm(p < 3 ? hi[i] : lo[i], 0x4b000000u, sel)) - 8388736.0f);
      *reinterpret_cast<uint4*>(out + p * tile_rows * (OKS * 2)) =
          make_uint4(__byte_perm(u[0], u[1], 0x7632), __byte_perm(u[2], u[3], 0x7632), __byte_perm(u[4], u[5], 0x7632),
                     __byte_perm(u[6], u[7], 0x7632));
    }
  };
  double x[kHold][8];
  int rr[kHold], kk[kHold];
#pragma unroll
  for (int h = 0; h < kHold; ++h) {
    const int it = threadIdx.x + h * 256;
    if (it < items) {
      place(it, rr[h], kk[h]);
      fetch(rr[h], kk[h], x[h]);
    }
  }
#pragma unroll
  for (int h = 0; h < kHold; ++h)
    if (threadIdx.x + h * 256 < items) top(x[h], rr[h], kk[h]);
  for (int it = threadIdx.x + kHold * 256; it < items; it += 256) {
    double y[8];
    int r, kg;
    place(it, r, kg);
    fetch(r, kg, y);
    top(y, r, kg);
  }
  __syncthreads();
  if (threadIdx.x < pk.rows) {
    const int m = row_max[threadIdx.x], e = row_exponent(m >> kExp);
    job.exps[pk.exp0 + threadIdx.x] = e;
    // out of range: the largest magnitude 2^480 or above (also of a value that is not finite),
    // or below 2^-480 and not zero
    if (e > kOzMaxExponent || (m != 0 && (m >> kExp) - 1022 < -kOzMaxExponent)) atomicMax(job.flag, job.seq);
  }
#pragma unroll
  for (int h = 0; h < kHold; ++h)
    if (threadIdx.x + h * 256 < items) emit(x[h], rr[h], kk[h]);
  for (int it = threadIdx.x + kHold * 256; it < items; it += 256) {
    double y[8];
    int r, kg;
    place(it, r, kg);
    fetch(r, kg, y);
    emit(y, r, kg);
  }
}

// 32 entries of a contraction's powers of two (DOzScale).  A launch of a few CTAs whose time is
// its latency, hence 32 warps each: where the elements of an entry are contiguous a warp takes
// an entry, else a lane does.
__global__ void __launch_bounds__(1024) oz_scale_kernel(const __grid_constant__ OzScaleJobs jobs) {
  __shared__ int top[32];
  chain_wait();
  chain_next();
  const int jb = jobs.n > 1 && (int)blockIdx.x >= jobs.job[0].ntasks;
  const OzScaleJob& job = jobs.job[jb];
  const DOzScale t = job.tasks[blockIdx.x - (jb ? jobs.job[0].ntasks : 0)];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x < 32) top[threadIdx.x] = 0;
  __syncthreads();
  for (int b = t.b0; b < t.b1; ++b) {
    const DOzScaleBlock bl = job.blocks[b];
    const bool by_lane = bl.istride == 1;
    const int i = t.i0 + (by_lane ? lane : warp);
    int m = 0;
    if (i < t.dim) {
      const double* p = job.src + bl.off + (long long)i * bl.istride;
#pragma unroll 4
      for (int l = by_lane ? warp : lane; l < bl.len; l += 32)
        m = max(m, __double2hiint(p[(long long)l * bl.lstride]) & 0x7fffffff);
    }
    if (!by_lane) m = __reduce_max_sync(0xffffffffu, m);
    if (m != 0 && (by_lane || lane == 0)) atomicMax(&top[by_lane ? lane : warp], m);
  }
  __syncthreads();
  const int i = t.i0 + (int)threadIdx.x;
  if (threadIdx.x >= 32 || i >= t.dim) return;
  const int m = top[threadIdx.x];
  const int e = m == 0 ? -127 : min(max((m >> 20) - 1022, -127), 127);
  for (int r = 0; r < t.repeat; ++r) job.out[t.out + r * t.dim + i] = (int8_t)e;
}

}  // namespace

void launch_oz_scale(const OzScaleJobs& jobs, cudaStream_t st) {
  int n = 0;
  for (int i = 0; i < jobs.n; ++i) n += jobs.job[i].ntasks;
  if (n > 0) launch_chained(oz_scale_kernel, dim3(n), 1024, 0, st, jobs);
}

void launch_gemm_oz(const OzGemmArgs& a, cudaStream_t st) {
  if (a.nctas <= 0) return;
  allow_smem<gemm_oz_kernel>(SMEM_BYTES);
  launch_chained(gemm_oz_kernel, dim3(a.nctas), NTHREADS, SMEM_BYTES, st, a);
}

void launch_oz_reduce(const DReduce* red, int nred, const OzGemmArgs& a, cudaStream_t st) {
  if (nred <= 0) return;
  launch_chained(oz_reduce_kernel, dim3(nred, (OM * ON) / 256), 256, 0, st, red, a);
}

void launch_oz_pack(const OzPackJobs& jobs, cudaStream_t st) {
  int n = 0;
  for (int i = 0; i < jobs.n; ++i) n += jobs.job[i].npacks;
  if (n <= 0) return;
  launch_chained(jobs.job[0].scales ? oz_pack_kernel<true> : oz_pack_kernel<false>, dim3(n), 256, 0, st, jobs);
}

}  // namespace mpsxx
