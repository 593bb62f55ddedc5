// Batched GEMV: several sequences against one weight matrix on the 5th-generation tensor cores
// (tcgen05.mma kind::i8), for every integer tensor-core layout.
//
// Same arithmetic as the warp-level units (gemv_units.cuh): the activations of a 256-block are four
// signed base-256 digits of a 32-bit fixed-point number, products and block sums are exact integers,
// lut_linear's loop over sequences (src/kernels/lut_gemm_scalar.cpp:76) becomes the N dimension:
//     D[128 rows][4 digits x sequences] = A[128 rows][256 columns] x B[256][4 x sequences]   (s32)
// A: weight codes, expanded to bytes in registers (a mask per word: the tile layout is the operand
//    fragment order, which is also the 16x128b register shape of tcgen05.st) and stored to TMEM.
// B: digits, written once per launch by k_prepare_batched in the no-swizzle core-matrix order, so that a
//    block's operand and its scales arrive with one bulk copy.
// D: TMEM, read back per 256-block (every block has scales of its own) and accumulated in fp32 per row.
//
// What bounds it: warp-level IMMA re-read the weights once per 8 sequences and spent 16 MMAs, their
// operand loads and the scaling of every (32 rows x 2 sequences) in the same warps; here the weights are
// read once per 8, 16 or 32 sequences and the tensor work leaves the warps, which keep the byte expansion
// (64 masks per 32 x 256 codes) and the scaling (9 instructions per row, sequence and block).  Ternary
// 8192 x 28672, 16 sequences: 133 us before, 44 us with this kernel (9.9 us of HBM time).  Measured on the way
// and not taken: two warps per tile (46 us; 24 instead of 19 us at 8192 x 8192).  With an eighth of the MMAs,
// of the scaling or of the TMEM stores it takes 38 to 43 us, with an eighth of all three 27 us, with an eighth
// of the bytes 42 us: what is left is the chain of expansion, hand-over and scaling inside a warp.
//
// Work split: the (row group, block) units of all jobs of a launch are one flat list, cut into equal
// contiguous ranges, one per CTA; how many CTAs, and how many passes over the sequences, plan_batched
// decides.  A row group whose blocks lie in several CTAs is added up, in CTA order, by the warp that arrives last.
//
// Roles: 4 * H worker warps (a 32-row tile each), one producer thread (bulk copies), one MMA thread.
// Every wait is bounded: on expiry the kernel raises the context's fault flag and leaves in order.
#include <algorithm>

#include "decode_device.cuh"
#include "gemv_units.cuh"

namespace lmb {

namespace {

constexpr int BT_MAX_JOBS = 4;
constexpr int BT_MAX_STAGES = 8;
constexpr unsigned BT_DRAIN_POLLS = 1u << 20;  // bound of the waits on the way out
constexpr int BT_MAX_SEQS = 32;           // sequences per pass: 4 digits each = 128 accumulator columns
constexpr size_t BT_SEQ_BYTES = 1024 + 16;  // one sequence's share of a block's operand image: digits and {scale, digit sums}

struct BtJob {
  const uint8_t *tiles;
  float *y;
  const float *bias, *residual;
  int M, row_tiles, rg_first;  // rg_first: first row group of the job in the launch
  unsigned y_stride;
#ifdef LMB_DEBUG_BOUNDS
  size_t tiles_bytes, y_floats;
#endif
};

struct BtParams {
  BtJob job[BT_MAX_JOBS];
  int njobs, n_rg, bpr, batch, ns, n_stages;
  unsigned stage_bytes;
  const uint8_t *img;   // [pass][block] operand images of ns * BT_SEQ_BYTES bytes
  float *scratch;       // [pass][CTA][its first / last row group][ns][rows of a group]: partial sums
  unsigned *counters;   // [pass][row group][tile of the group]
  unsigned *fault;
  unsigned spin_limit;
  int extra_arrivals;   // test hook: the operand barriers expect this many arrivals too many
  unsigned long long *dbg;  // this launch's slot of the launch timeline (debugging), or null
#ifdef LMB_DEBUG_BOUNDS
  size_t scratch_floats;
#endif
};

// Row tiles per CTA = 4 * H: B is fetched once per row group, so the narrow kinds take 256 rows (with 128
// the operand images would be twice the weight bytes); the wide ones have 4 to 8 KiB per tile anyway.
__host__ __device__ constexpr int bt_halves(int kind) { return kind_is_wide(kind) ? 1 : 2; }
__host__ __device__ constexpr int bt_planes(int kind) { return kind == DK_INT2_MMA ? 2 : 1; }
__host__ __device__ constexpr int bt_threads(int kind) { return (4 * bt_halves(kind) + 2) * 32; }
// accumulators are double buffered where TMEM has room
__host__ __device__ constexpr bool bt_double(int nsmax) { return nsmax <= 16; }
__host__ __device__ constexpr int bt_tmem_cols(int kind, int nsmax) {
  const int need = bt_halves(kind) * (2 * 64 + (bt_double(nsmax) ? 2 : 1) * 4 * nsmax);
  return need <= 128 ? 128 : need <= 256 ? 256 : 512;
}

// ---- tcgen05 -----------------------------------------------------------------------------------------------
__device__ __forceinline__ void tc_alloc(uint32_t *dst, unsigned cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr_u32(dst)), "r"(cols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
__device__ __forceinline__ void tc_dealloc(uint32_t base, unsigned cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(cols));
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint64_t *bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr_u32(bar)) : "memory");
}
// 16 lanes x 16 columns: registers 4k..4k+3 = {row g, row g+8, row g (+4 columns), row g+8 (+4 columns)} of k-step k
__device__ __forceinline__ void tc_st_16x128b_x4(uint32_t addr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.16x128b.x4.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]),
               "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]));
}
// this lane's row, 32 columns; complete when the statement is (the results depend on the wait inside it)
__device__ __forceinline__ void tc_ld_32x32b_x32(uint32_t addr, int (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(addr));
}
__device__ __forceinline__ void tc_mma_i8(uint32_t d, uint32_t a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d), "r"(a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr_u32(bar)) : "memory");
}

// ---- byte expansion ------------------------------------------------------------------------------------------
// The registers of k-steps 2q and 2q+1 for rows 16 * hl .. 16 * hl + 15 of a tile (tc_st_16x128b_x4 order).
// Codes may keep their field's offset inside the byte (row_mult / plane shifts in `Row` undo it).
template <int KIND> __device__ __forceinline__ void expand(const uint4 (&t)[kind_info(KIND).chunks], int hl, int q, int plane, uint32_t (&r)[8]) {
  if constexpr (KIND == DK_TERNARY_MMA || KIND == DK_INT2_MMA) {
    const uint4 w = t[q];
    uint32_t m0, m1;
    if constexpr (KIND == DK_TERNARY_MMA) {
      m0 = 0x03030303u << (4 * hl);
      m1 = 0x0C0C0C0Cu << (4 * hl);
    } else {
      m0 = 0x01010101u << (4 * hl + plane);
      m1 = 0x04040404u << (4 * hl + plane);
    }
    r[0] = w.x & m0; r[1] = w.x & m1; r[2] = w.y & m0; r[3] = w.y & m1;
    r[4] = w.z & m0; r[5] = w.z & m1; r[6] = w.w & m0; r[7] = w.w & m1;
  } else if constexpr (KIND == LMB_INT4) {
    const uint4 w = t[hl * 4 + q];
    constexpr uint32_t LO = 0x0F0F0F0Fu, HI = 0xF0F0F0F0u;
    r[0] = w.x & LO; r[1] = w.x & HI; r[2] = w.y & LO; r[3] = w.y & HI;
    r[4] = w.z & LO; r[5] = w.z & HI; r[6] = w.w & LO; r[7] = w.w & HI;
  } else if constexpr (KIND == DK_INT8_MMA) {
    const uint4 a = t[hl * 8 + 2 * q], b = t[hl * 8 + 2 * q + 1];
    r[0] = a.x; r[1] = a.y; r[2] = a.z; r[3] = a.w;
    r[4] = b.x; r[5] = b.y; r[6] = b.z; r[7] = b.w;
  } else {
    // bit planes in the DK_BINARY_MMA arrangement (bit m + 4 kh of a byte), with low nibbles under them for 5 and 6 bits
    constexpr bool NIB = KIND == LMB_INT5 || KIND == LMB_INT6;
    constexpr int NPL = KIND == DK_BINARY_MMA ? 1 : KIND == DK_INT3_MMA ? 3 : KIND == LMB_INT5 ? 1 : 2;
    constexpr int P0 = NIB ? 4 : 0, NC = NIB ? 8 : 0;
    uint32_t pa[NPL], pb[NPL];
#pragma unroll
    for (int pl = 0; pl < NPL; ++pl) {
      const uint4 v = t[NC + 2 * pl + (q >> 1)];
      pa[pl] = (q & 1) ? v.z : v.x;
      pb[pl] = (q & 1) ? v.w : v.y;
    }
    uint4 n = make_uint4(0u, 0u, 0u, 0u);
    if constexpr (NIB) n = t[hl * 4 + q];
#pragma unroll
    for (int kh = 0; kh < 2; ++kh)
#pragma unroll
      for (int ab = 0; ab < 2; ++ab)
#pragma unroll
        for (int mm = 0; mm < 2; ++mm) {
          const int s = 2 * hl + mm + 4 * kh;
          const uint32_t nw = kh ? (ab ? n.w : n.z) : (ab ? n.y : n.x);
          uint32_t code = NIB ? ((mm ? nw >> 4 : nw) & 0x0F0F0F0Fu) : 0u;
#pragma unroll
          for (int pl = 0; pl < NPL; ++pl) code |= (((ab ? pb[pl] : pa[pl]) >> s) & 0x01010101u) << (P0 + pl);
          r[kh * 4 + ab * 2 + mm] = code;
        }
  }
}

// How a row of a tile turns its integer sums into values: field multiplier and zero point.
template <int KIND> struct Row {
  // plus-minus-one planes: 2 x - d
  static constexpr bool PM1 = KIND == DK_INT2_MMA || KIND == DK_BINARY_MMA;
  static __device__ __forceinline__ int mult(int m, int plane) {
    return KIND == DK_TERNARY_MMA ? 1 << (2 * m) : KIND == DK_INT2_MMA ? 1 << (2 * m + plane) : KIND == LMB_INT4 ? 1 << (4 * (m & 1)) : 1;
  }
  static constexpr int ZERO = KIND == DK_TERNARY_MMA ? 1 : KIND == LMB_INT4 ? 8 : KIND == DK_INT3_MMA ? 4 : KIND == LMB_INT5 ? 16
                            : KIND == LMB_INT6 ? 32 : 0;
};

// CTA that owns unit u when `total` units are cut into g contiguous ranges [c * total / g, (c + 1) * total / g)
__device__ __forceinline__ int owner_of(long long u, long long total, long long g) { return int(((u + 1) * g - 1) / total); }

template <int KIND, int NSMAX>
__global__ void __launch_bounds__(bt_threads(KIND), 512 / bt_tmem_cols(KIND, NSMAX) > 1 ? 2 : 1) k_gemm_batched(const __grid_constant__ BtParams p) {
  constexpr int H = bt_halves(KIND), P = bt_planes(KIND), W = 4 * H;
  constexpr bool DD = bt_double(NSMAX);
  constexpr unsigned TB = unsigned(tile_bytes(KIND));
  constexpr unsigned COLS = bt_tmem_cols(KIND, NSMAX);
  constexpr uint32_t D0 = H * 128;
  constexpr int ROWS = W * TILE_ROWS;
  extern __shared__ __align__(128) uint8_t stages[];
  __shared__ __align__(8) uint64_t full[BT_MAX_STAGES], empty[BT_MAX_STAGES], a_full[H][2], d_full[H][2], drain;
  __shared__ uint32_t tmem_base;
  __shared__ volatile int gave_up;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    tl_min(p.dbg, 0);
    gave_up = 0;
    for (int s = 0; s < p.n_stages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], W);
    }
    for (int h = 0; h < H; ++h)
      for (int b = 0; b < 2; ++b) {
        mbar_init(&a_full[h][b], unsigned(4 + p.extra_arrivals));
        mbar_init(&d_full[h][b], 1);
      }
    mbar_init(&drain, 1);
  }
  if (warp == W + 1) tc_alloc(&tmem_base, COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  // Only now: a successor that is let in earlier could take the SM's TMEM before this CTA has its own, and
  // would hold it while waiting for this kernel to finish.
  pdl_launch_dependents();
  const uint32_t tmem = tmem_base;

  const long long total = (long long)p.n_rg * p.bpr;
  const long long u0 = (long long)blockIdx.x * total / gridDim.x, u1 = (long long)(blockIdx.x + 1) * total / gridDim.x;
  const int n = int(u1 - u0);  // (row group, block) units of this CTA
  const int rg0 = int(u0 / p.bpr), b_first = int(u0 - (long long)rg0 * p.bpr);
  const int pass = blockIdx.y;
  const unsigned img_bytes = unsigned(p.ns) * unsigned(BT_SEQ_BYTES);
  const uint8_t *img = p.img + size_t(pass) * p.bpr * img_bytes;
  constexpr unsigned B_OFF = (W * TB + 127) / 128 * 128;

  auto wait = [&](uint64_t *bar, unsigned parity) -> bool {
    unsigned spins = 0;
    while (!mbar_try_wait(bar, parity)) {
      if (gave_up || ++spins > p.spin_limit) {
        gave_up = 1;
        *p.fault = 1u;
        return false;
      }
    }
    return true;
  };
  auto job_of = [&](int rg) {
    int j = 0;
    while (j + 1 < p.njobs && rg >= p.job[j + 1].rg_first) ++j;
    return j;
  };

  if (warp == W) {
    // The whole warp issues: lane 0 the expected bytes, lanes 0 .. W-1 a weight tile each, lane W the operand
    // image.  Positions advance by one unit at a time: the divisions of a flat index, per unit, held this warp
    // below the rate of the tensor cores.
    struct Cursor {
      int rg, b, st;
    };
    auto advance = [&](Cursor &c) {
      if (++c.b == p.bpr) {
        c.b = 0;
        ++c.rg;
      }
      if (++c.st == p.n_stages) c.st = 0;
    };
    int rg_of = -1, nt = 0;
    const uint8_t *src = nullptr;  // this lane's tile row
    auto weights = [&](const Cursor &c) {
      if (c.rg != rg_of) {
        rg_of = c.rg;
        const BtJob &jb = p.job[job_of(c.rg)];
        const int rt0 = (c.rg - jb.rg_first) * W;
        nt = min(W, jb.row_tiles - rt0);
        src = jb.tiles + size_t(rt0 + lane) * p.bpr * TB;
#ifdef LMB_DEBUG_BOUNDS
        const size_t end = (size_t(rt0 + lane + 1) * p.bpr) * TB;
        const bool ok = lane >= nt || LMB_IN_BOUNDS(end <= jb.tiles_bytes, BOUNDS_WEIGHT_TILE, end);
        nt = __ffs(~__ballot_sync(0xffffffffu, ok && lane < nt)) - 1;  // a tile row that would leave its buffer is not fetched
#endif
      }
      if (lane == 0) mbar_arrive_expect_tx(&full[c.st], unsigned(nt) * TB + img_bytes);
      __syncwarp();
      if (lane < nt) bulk_copy_g2s(stages + size_t(c.st) * p.stage_bytes + lane * TB, src + size_t(c.b) * TB, TB, &full[c.st]);
    };
    auto operand = [&](const Cursor &c) {
      if (lane == W) bulk_copy_g2s(stages + size_t(c.st) * p.stage_bytes + B_OFF, img + size_t(c.b) * img_bytes, img_bytes, &full[c.st]);
    };
    const Cursor first{rg0, b_first, 0};
    // weights do not depend on the preceding kernel, the operand images do
    const int ahead = min(n, p.n_stages);
    Cursor c = first;
    for (int i = 0; i < ahead; ++i, advance(c)) weights(c);
    pdl_wait();
    Cursor o = first;
    for (int i = 0; i < ahead; ++i, advance(o)) operand(o);
    int issued = ahead;
    unsigned par = 0;
    for (int i = ahead; i < n; ++i) {
      if (!__all_sync(0xffffffffu, wait(&empty[c.st], par))) break;
      weights(c);
      operand(c);
      issued = i + 1;
      advance(c);
      if (c.st == 0) par ^= 1u;
    }
    // own copies in flight (after a wait that expired): they land before the shared memory goes away
    for (int i = max(0, issued - p.n_stages); i < issued; ++i)
      for (unsigned s = 0; s < BT_DRAIN_POLLS && !mbar_try_wait(&full[i % p.n_stages], unsigned(i / p.n_stages) & 1u); ++s) {}
  } else if (warp == W + 1) {
    // Nothing to do before the operand copies, which wait for the preceding kernels: polling earlier would charge
    // those kernels' run time (another rank's lateness among it) to this kernel's limit.
    pdl_wait();
    if (lane == 0) {
      tl_min(p.dbg, 1);
      tl_max(p.dbg, 2);
      const unsigned groups = unsigned(p.ns) / 2;  // 8-row groups of B: two sequences x four digits
      const uint32_t idesc = (2u << 4) | (KIND == DK_INT8_MMA ? 1u << 7 : 0u) | (1u << 10) | ((unsigned(p.ns) * 4u >> 3) << 17) | (8u << 24);
      const uint64_t lbo = groups * 128u >> 4, sbo = 128u >> 4;  // core matrices: [16-column chunk][8-row group][8 rows][16 bytes]
      bool ok = true;
      int st = 0;
      unsigned st_par = 0;
      for (int i = 0; i < n && ok; ++i) {
        ok = wait(&full[st], st_par);
        if (i == 0) tl_max(p.dbg, 3);  // stamped here, not by the workers: they have no register to spare
        const uint64_t bdesc0 = (uint64_t(1) << 46) | (sbo << 32) | (lbo << 16) |
                                uint64_t((smem_addr_u32(stages) + unsigned(st) * p.stage_bytes + B_OFF) >> 4);
        for (int pl = 0; pl < P && ok; ++pl) {
          const int u = i * P + pl, buf = u & 1;
          for (int h = 0; h < H && ok; ++h) {
            ok = wait(&a_full[h][buf], unsigned(u >> 1) & 1u);
            if (!ok) break;
            tc_fence_after();
            const uint32_t d = tmem + D0 + uint32_t(h * (DD ? 2 : 1) + (DD ? buf : 0)) * (4 * NSMAX), a = tmem + uint32_t(h * 2 + buf) * 64;
#pragma unroll
            for (int s = 0; s < 8; ++s) tc_mma_i8(d, a + 8 * s, bdesc0 + uint64_t(2 * s) * lbo, idesc, s > 0);
            tc_commit(&d_full[h][buf]);
          }
        }
        if (++st == p.n_stages) {
          st = 0;
          st_par ^= 1u;
        }
      }
      // no MMA is in flight when the TMEM is given back, whatever the workers have waited for
      tc_commit(&drain);
      for (unsigned s = 0; s < BT_DRAIN_POLLS && !mbar_try_wait(&drain, 0); ++s) {}
      tl_max(p.dbg, 4);
    }
  } else {
    pdl_wait();
    const int h = warp >> 2;
    const uint32_t lanes = uint32_t(warp & 3) << 21;  // this warp's 32 TMEM lanes
    const int m = lane >> 3, sc_at = 4 * (lane & 7) + m;
    // low and high digit pairs of up to 8 blocks, and the sum of what they were before: two levels keep the fp32
    // error of a long row below that of the short slices a single-sequence launch cuts it into
    float2 acc[NSMAX];
    float sum[NSMAX];
#pragma unroll
    for (int q = 0; q < NSMAX; ++q) {
      acc[q] = make_float2(0.0f, 0.0f);
      sum[q] = 0.0f;
    }
    int in_acc = 0;
    auto fold = [&]() {
#pragma unroll
      for (int q = 0; q < NSMAX; ++q) {
        sum[q] += acc[q].x + 65536.0f * acc[q].y;
        acc[q] = make_float2(0.0f, 0.0f);
      }
      in_acc = 0;
    };
    const int nb = min(p.ns, p.batch - pass * p.ns);

    // finished row group (or this CTA's part of it)
    auto flush = [&](int rg) {
      const BtJob &jb = p.job[job_of(rg)];
      const int rt = (rg - jb.rg_first) * W + warp, row = rt * TILE_ROWS + lane;
      float v[NSMAX];
#pragma unroll
      for (int q = 0; q < NSMAX; ++q) {
        v[q] = sum[q];
        sum[q] = 0.0f;
      }
      if (rt >= jb.row_tiles) return;  // uniform over the warp
      const int c0 = owner_of((long long)rg * p.bpr, total, gridDim.x), c1 = owner_of((long long)rg * p.bpr + p.bpr - 1, total, gridDim.x);
      const int parts = c1 - c0 + 1;
      if (parts > 1) {
        // CTA c0 has this row group last in its range, the others have it first
        const size_t part_floats = size_t(p.ns) * ROWS;
        float *scr = p.scratch + (size_t(pass) * gridDim.x + c0) * 2 * part_floats + warp * TILE_ROWS + lane;
        auto part = [&](int k) { return scr + size_t(k == 0 ? 1 : 2 * k) * part_floats; };
        float *mine = part(int(blockIdx.x) - c0);
#pragma unroll
        for (int q = 0; q < NSMAX; ++q)
          if (q < nb) {
#ifdef LMB_DEBUG_BOUNDS
            if (!LMB_IN_BOUNDS(size_t(mine - p.scratch) + size_t(q) * ROWS < p.scratch_floats, BOUNDS_SCRATCH, mine - p.scratch)) continue;
#endif
            mine[size_t(q) * ROWS] = v[q];
          }
        __syncwarp();
        unsigned before = 0;
        unsigned *ctr = p.counters + (size_t(pass) * p.n_rg + rg) * W + warp;
        if (lane == 0) {
          // release: this warp's partial sums; acquire: those of the parts that arrived earlier
          asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(before) : "l"(ctr) : "memory");
          if (before == unsigned(parts - 1)) *ctr = 0u;  // ready for the next launch
        }
        before = __shfl_sync(0xffffffffu, before, 0);
        if (before != unsigned(parts - 1)) return;
        __syncwarp();
        // Parts are added in pairs and fours, which shortens the serial fp32 chain over them: with one addition per
        // part, few rows over a long K (dozens of parts) had up to 1.5 times the error of a single sequence's short slices.
#pragma unroll
        for (int q0 = 0; q0 < NSMAX; q0 += 8) {
          if (q0 < nb) {
#pragma unroll
            for (int q = 0; q < 8; ++q) v[q0 + q] = 0.0f;
            for (int k0 = 0; k0 < parts; k0 += 4) {  // 32 loads in flight per lane
              float t[4][8];
#pragma unroll
              for (int k = 0; k < 4; ++k)
#pragma unroll
                for (int q = 0; q < 8; ++q)
                  t[k][q] = (k0 + k < parts && q0 + q < nb) ? __ldcg(part(k0 + k) + size_t(q0 + q) * ROWS) : 0.0f;
#pragma unroll
              for (int q = 0; q < 8; ++q) v[q0 + q] += (t[0][q] + t[1][q]) + (t[2][q] + t[3][q]);
            }
          }
        }
      }
      if (row >= jb.M) return;
      const float bias = jb.bias ? jb.bias[row] : 0.0f;
      const size_t at0 = size_t(pass) * p.ns * jb.y_stride + row;
#pragma unroll
      for (int q0 = 0; q0 < NSMAX; q0 += 8) {
        if (q0 < nb) {
          float res[8];
#pragma unroll
          for (int q = 0; q < 8; ++q) res[q] = (jb.residual && q0 + q < nb) ? jb.residual[at0 + size_t(q0 + q) * jb.y_stride] : 0.0f;
#pragma unroll
          for (int q = 0; q < 8; ++q)
            if (q0 + q < nb) {
              float o = v[q0 + q];
              if (jb.bias) o += bias;
              if (jb.residual) o += res[q];
              const size_t at = at0 + size_t(q0 + q) * jb.y_stride;
#ifdef LMB_DEBUG_BOUNDS
              if (!LMB_IN_BOUNDS(at < jb.y_floats, BOUNDS_OUTPUT, at)) continue;
#endif
              jb.y[at] = o;
            }
        }
      }
    };

    // accumulator of unit u (block i = u / P) -> fp32
    int rg = rg0, b = b_first, st_r = 0;  // where the read-out stands
    auto readout = [&](int u, bool last_unit) -> bool {
      const int plane = u % P, st = st_r, buf = u & 1;
      if (!__all_sync(0xffffffffu, wait(&d_full[h][buf], unsigned(u >> 1) & 1u))) return false;
      tc_fence_after();
      const uint8_t *stage = stages + size_t(st) * p.stage_bytes;
      const float rs = reinterpret_cast<const float *>(stage + warp * TB + kind_info(KIND).chunks * 512 + plane * 128)[sc_at];
      const int4 *aux = reinterpret_cast<const int4 *>(stage + B_OFF + size_t(p.ns) * 1024);
      const int mult = Row<KIND>::mult(m, plane);
      const float scale = rs * __uint_as_float(uint32_t(127 - (31 - __clz(mult))) << 23);  // / mult, exact
      const uint32_t zm = uint32_t(Row<KIND>::PM1 ? mult : Row<KIND>::ZERO * mult);
      const uint32_t d = tmem + lanes + D0 + uint32_t(h * (DD ? 2 : 1) + (DD ? buf : 0)) * (4 * NSMAX);
#pragma unroll
      for (int q0 = 0; q0 < NSMAX; q0 += 8) {
        if (q0 < p.ns) {
          int r[32];
          tc_ld_32x32b_x32(d + 4 * q0, r);
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const int4 ax = aux[q0 + q];  // {block scale, digit-pair sums}; beyond p.ns: unused columns
            // modular arithmetic: the results fit 32 bits
            uint32_t lo = uint32_t(r[4 * q]) + 256u * uint32_t(r[4 * q + 1]), hi = uint32_t(r[4 * q + 2]) + 256u * uint32_t(r[4 * q + 3]);
            if constexpr (Row<KIND>::PM1) {
              lo = 2u * lo - zm * uint32_t(ax.y);
              hi = 2u * hi - zm * uint32_t(ax.z);
            } else if constexpr (Row<KIND>::ZERO != 0) {
              lo -= zm * uint32_t(ax.y);
              hi -= zm * uint32_t(ax.z);
            }
            const float s = __int_as_float(ax.x) * scale;
            fma2(acc[q0 + q], make_float2(float(int(lo)), float(int(hi))), make_float2(s, s));
          }
        }
      }
      if (plane == P - 1) {
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[st]);
        if (++st_r == p.n_stages) st_r = 0;
        const bool row_end = ++b == p.bpr;
        if (++in_acc == 8 || last_unit || row_end) fold();
        if (last_unit || row_end) flush(rg);
        if (row_end) {
          b = 0;
          ++rg;
        }
      }
      return true;
    };

    bool ok = true;
    int st_w = 0;
    unsigned par_w = 0;
    for (int i = 0; i < n && ok; ++i) {
      ok = __all_sync(0xffffffffu, wait(&full[st_w], par_w));
      if (!ok) break;
      const uint4 *tile = reinterpret_cast<const uint4 *>(stages + size_t(st_w) * p.stage_bytes + warp * TB);
      uint4 raw[kind_info(KIND).chunks];
#pragma unroll
      for (int k = 0; k < kind_info(KIND).chunks; ++k) raw[k] = tile[k * 32 + lane];
      if (++st_w == p.n_stages) {
        st_w = 0;
        par_w ^= 1u;
      }
#pragma unroll
      for (int pl = 0; pl < P; ++pl) {
        const int u = i * P + pl, buf = u & 1;
        // this A buffer was last read by the MMAs of unit u - 2, whose results this warp has read
        const uint32_t a = tmem + lanes + uint32_t(h * 2 + buf) * 64;
#pragma unroll
        for (int hl = 0; hl < 2; ++hl)
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            uint32_t r[8];
            expand<KIND>(raw, hl, q, pl, r);
            tc_st_16x128b_x4(a + (uint32_t(hl) << 20) + 16 * q, r);
          }
        tc_wait_st();
        // one accumulator: its last unit is read before the next MMAs are let go
        if (!DD && u > 0) ok = readout(u - 1, false);
        if (!ok) break;
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&a_full[h][buf]);
        if (DD && u > 0) ok = readout(u - 1, false);
        if (!ok) break;
      }
    }
    if (ok && n > 0) readout(n * P - 1, true);
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == W + 1) {
    tc_dealloc(tmem, COLS);
    if (lane == 0) {
      tl_max(p.dbg, 5);
      tl_min(p.dbg, 6);
    }
  }
}

// Operand images of a launch's activations: normalised / gated / rotated and cut into digits once.  One warp
// per (sequence, block); grid = (ceil(bpr / 8), sequences).
constexpr int BT_PREP_THREADS = 256;
__global__ void __launch_bounds__(BT_PREP_THREADS) k_prepare_batched(const float *x, const float *x2, unsigned x_len, unsigned x_stride, int bpr,
                                                                     int xmode, int rotate, float eps, int ns, uint8_t *img,
                                                                     unsigned long long *dbg) {
  pdl_launch_dependents();
  if (threadIdx.x == 0) tl_min(dbg, 0);
  __shared__ float red[8];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q = blockIdx.y;
  const float *xq = x + size_t(q) * x_stride;
  pdl_wait();
  if (threadIdx.x == 0) {
    tl_min(dbg, 1);
    tl_max(dbg, 2);
  }
  float inv_rms = 1.0f;
  if (xmode == XMODE_RMSNORM) {  // src/layers/norm.cpp:18-34
    float ss = 0.0f;
    for (unsigned i = threadIdx.x; i < x_len; i += BT_PREP_THREADS) {
      const float v = xq[i];
      ss += v * v;
    }
#pragma unroll
    for (int k = 16; k > 0; k >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, k);
    if (lane == 0) red[warp] = ss;
    __syncthreads();
    ss = 0.0f;
#pragma unroll
    for (int k = 0; k < 8; ++k) ss += red[k];
    inv_rms = 1.0f / sqrtf(ss / float(x_len) + eps);
  }
  const int bl = blockIdx.x * 8 + warp;
  if (bl >= bpr) return;
  float v[8], w8[8];
  load_x8(xq, x_len, size_t(bl), lane, v);
  if (xmode == XMODE_RMSNORM) {
    load_x8(x2, x_len, size_t(bl), lane, w8);
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = v[e] * inv_rms * w8[e];
  } else if (xmode == XMODE_SILU_MUL || xmode == XMODE_GELU_MUL) {
    load_x8(x2 + size_t(q) * x_stride, x_len, size_t(bl), lane, w8);
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = (xmode == XMODE_GELU_MUL ? gelu_tanh(v[e]) : v[e] / (1.0f + expf(-v[e]))) * w8[e];
  }
  if (threadIdx.x == 0) tl_max(dbg, 3);
  if (rotate) fwht256_warp(v, lane);
  MmaDigits dg;
  mma_digits(v, dg);
  const int pass = q / ns, sq = q - pass * ns;
  uint8_t *im = img + (size_t(pass) * bpr + bl) * ns * BT_SEQ_BYTES;
  // columns 8 lane .. 8 lane + 7 are half a 16-byte row of chunk lane / 2; rows 4 sq + digit
  uint8_t *dst = im + (size_t(lane >> 1) * (ns / 2) + (sq >> 1)) * 128 + (sq & 1) * 64 + (lane & 1) * 8;
#pragma unroll
  for (int d = 0; d < 4; ++d) *reinterpret_cast<uint2 *>(dst + d * 16) = make_uint2(dg.words[d][0], dg.words[d][1]);
  if (lane == 0)
    *reinterpret_cast<int4 *>(im + size_t(ns) * 1024 + sq * 16) = make_int4(__float_as_int(dg.bscale), dg.d01, dg.d23, 0);
  if (threadIdx.x == 0) {
    tl_max(dbg, 4);
    tl_max(dbg, 5);
    tl_min(dbg, 6);
  }
}

struct BtPlan {
  int passes, ns, n_rg, ctas, n_stages, nsmax;
  unsigned stage_bytes;
  size_t scratch, counters, img_records;
  float us;  // estimated time of both kernels of the launch
};

// Shared memory of one SM (228 KiB) less what the driver and the static part take.
constexpr size_t BT_SMEM = 220 * 1024;

// Estimate of a launch in microseconds, fitted to 14,700 timed launches (64 to 28672 rows x 300 to 28672 columns,
// 4 to 32 sequences, every split).  What a CTA takes per unit of work in the forms for 8, 16 and 32 sequences:
constexpr float BT_PART_US[3] = {0.137f, 0.295f, 0.58f};  // reading one part of a row group back
constexpr float BT_FORM_US[3] = {0.0f, 1.1f, 3.7f};       // fixed part beyond the smallest form's
constexpr float BT_MERGE_US = 1.5f, BT_FLAT_US = 2.0f, BT_WAVE_US = 3.5f;
constexpr float BT_SHARED_SM = 1.3f;  // a unit's time with a second CTA on the SM
// two launches, operand images, first copies
constexpr float BT_BASE_US = 4.0f, BT_BASE_INT2_US = 4.4f, BT_BASE_INT8_US = 2.7f;
float bt_unit_us(int kind, int form) {
  switch (kind) {
  case DK_INT2_MMA: return form == 0 ? 2.0f : form == 1 ? 2.1f : 3.2f;    // two planes
  case DK_INT3_MMA: return form == 0 ? 1.45f : form == 1 ? 1.5f : 1.95f;  // three bit planes put together in registers
  case DK_INT8_MMA: return 1.3f;                                          // 128 rows of 8 KiB a tile
  case LMB_INT5:
  case LMB_INT6: return form == 0 ? 1.0f : 1.5f;
  default: return form == 2 ? 1.4f : 1.07f;
  }
}

// Sequences per pass and CTAs per pass.  More passes than the 32 sequences a pass can hold need read the weights
// again (from L2 when the passes run side by side) but fill the GPU where rows are few and take the leaner forms.
// A row group is cut into equal parts, as many as balance the units of a CTA against reading the parts back
// (about sqrt(blocks x 0.14) units); or all units into as many ranges as CTAs fit (flat), where that shortens the
// longest range by more than the second merge of a CTA that then holds the end of one row group and the start of the next.
// Against one pass of all sequences and at least two units per CTA, in us: ternary 64 x 1536, 32 sequences 13.1 -> 7.2;
// 512 x 28672, 32 sequences 50.4 -> 21.4; 2-bit 1536 x 8960, 32 sequences 30.8 -> 21.3; 4-bit 8192 x 1536, 16 sequences
// 9.9 -> 9.5.  The measured best over all splits is 0.7 % less on average.
// force_seqs, force_ctas: sequences and CTAs per pass of the test hook (0: free choice).
BtPlan plan_batched(int kind, const size_t *row_tiles, int njobs, size_t bpr, size_t batch, int sm_count, int force_seqs, int force_ctas) {
  const int W = 4 * bt_halves(kind);
  size_t n_rg = 0;
  for (int j = 0; j < njobs; ++j) n_rg += (row_tiles[j] + W - 1) / W;
  const size_t total = n_rg * bpr;
  const float base = kind == DK_INT8_MMA ? BT_BASE_INT8_US : kind == DK_INT2_MMA ? BT_BASE_INT2_US : BT_BASE_US;
  BtPlan best{};
  for (int form = 0; form < 3; ++form) {
    const size_t most = force_seqs ? size_t(force_seqs) : size_t(8) << form;
    if (force_seqs ? form > 0 : form > 0 && batch <= most / 2) break;  // the form before holds all sequences
    BtPlan pl{};
    pl.n_rg = int(n_rg);
    pl.passes = int((batch + most - 1) / most);
    const size_t per = (batch + pl.passes - 1) / pl.passes;
    pl.ns = int((per + 3) / 4 * 4);
    const int f = pl.ns <= 8 ? 0 : pl.ns <= 16 ? 1 : 2;
    pl.nsmax = 8 << f;
    // the 128 bytes behind an image keep the reads of unused columns' scales inside the stage
    pl.stage_bytes = unsigned((W * tile_bytes(kind) + 127) / 128 * 128 + (size_t(pl.ns) * BT_SEQ_BYTES + 128 + 127) / 128 * 128);
    const size_t tmem_ctas = 512 / size_t(bt_tmem_cols(kind, pl.nsmax));
    // two CTAs per SM where TMEM and shared memory hold two with two stages each
    const size_t per_sm = tmem_ctas > 1 && 2 * pl.stage_bytes * 2 + 8192 <= BT_SMEM ? 2 : 1;
    pl.n_stages = int(std::min<size_t>(BT_MAX_STAGES, (BT_SMEM / per_sm - 2048) / pl.stage_bytes));
    const size_t slots = size_t(sm_count) * per_sm, mine = std::max<size_t>(1, slots / size_t(pl.passes));
    auto consider = [&](size_t ctas, size_t units, size_t parts, bool flat) {
      const size_t all = ctas * size_t(pl.passes), waves = (all + slots - 1) / slots;
      const float unit = bt_unit_us(kind, f) * (all > size_t(sm_count) ? BT_SHARED_SM : 1.0f);
      const float us = base + 0.015f * float(batch) + BT_FORM_US[f] + float(waves * units) * unit +
                       (parts > 1 ? BT_MERGE_US + BT_PART_US[f] * float(parts) : 0.0f) + (flat ? BT_FLAT_US : 0.0f) +
                       BT_WAVE_US * float(waves - 1);
      if (best.ctas == 0 || us < best.us) {
        best = pl;
        best.ctas = int(ctas);
        best.us = us;
      }
    };
    if (force_ctas) {
      consider(std::min(total, size_t(force_ctas)), 1, 1, false);
      continue;
    }
    for (size_t parts = 1; parts <= bpr && n_rg * parts <= mine;) {
      const size_t units = (bpr + parts - 1) / parts;
      consider(n_rg * parts, units, parts, false);
      if (units == 1) break;
      parts = (bpr + units - 2) / (units - 1);  // the next shorter longest part
    }
    const size_t ctas = std::min(mine, total), units = (total + ctas - 1) / ctas;
    if (ctas % n_rg != 0) consider(ctas, units, std::min(bpr, (bpr + total / ctas - 1) / (total / ctas) + 1), true);
  }
  best.scratch = best.ctas > 1 ? size_t(best.passes) * best.ctas * 2 * best.ns * W * TILE_ROWS : 0;
  best.counters = size_t(best.passes) * best.n_rg * W;
  best.img_records = size_t(best.passes) * best.ns * bpr;
  return best;
}

template <int KIND, int NSMAX> int launch_one(lmb_ctx *ctx, const BtParams &p, const BtPlan &pl) {
  const size_t smem = size_t(pl.n_stages) * pl.stage_bytes;
  static_assert(bt_tmem_cols(KIND, NSMAX) >= bt_halves(KIND) * (128 + (bt_double(NSMAX) ? 2 : 1) * 4 * NSMAX), "TMEM");
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(pl.ctas), unsigned(pl.passes));
  cfg.blockDim = dim3(bt_threads(KIND));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = ctx->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = ctx->pdl ? 1 : 0;
  LMB_CUDA(cudaLaunchKernelEx(&cfg, k_gemm_batched<KIND, NSMAX>, p));
  ctx->launches++;
  return LMB_OK;
}
template <int KIND> int launch_kind(lmb_ctx *ctx, const BtParams &p, const BtPlan &pl) {
  return pl.nsmax == 8 ? launch_one<KIND, 8>(ctx, p, pl) : pl.nsmax == 16 ? launch_one<KIND, 16>(ctx, p, pl) : launch_one<KIND, 32>(ctx, p, pl);
}
template <int KIND> int configure_kind() {
  LMB_CUDA(cudaFuncSetAttribute(k_gemm_batched<KIND, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(BT_SMEM)));
  LMB_CUDA(cudaFuncSetAttribute(k_gemm_batched<KIND, 16>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(BT_SMEM)));
  LMB_CUDA(cudaFuncSetAttribute(k_gemm_batched<KIND, 32>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(BT_SMEM)));
  return LMB_OK;
}

}  // namespace

int configure_batched() {
  int st = configure_kind<LMB_INT4>();
  if (st == LMB_OK) st = configure_kind<DK_TERNARY_MMA>();
  if (st == LMB_OK) st = configure_kind<DK_INT2_MMA>();
  if (st == LMB_OK) st = configure_kind<DK_BINARY_MMA>();
  if (st == LMB_OK) st = configure_kind<LMB_INT5>();
  if (st == LMB_OK) st = configure_kind<LMB_INT6>();
  if (st == LMB_OK) st = configure_kind<DK_INT8_MMA>();
  if (st == LMB_OK) st = configure_kind<DK_INT3_MMA>();
  return st;
}

// Whether the batched kernel can serve a launch: several sequences, an integer tensor-core layout, one input for
// all jobs, ordinary output.
bool batched_possible(const LinearArgs *args, int njobs) {
  if (!kind_is_mma(args[0].w->kind) || args[0].batch < 3 || njobs > BT_MAX_JOBS) return false;
  for (int j = 0; j < njobs; ++j)
    if (args[j].to_peers || args[j].prep_in || args[j].next_prep || args[j].x != args[0].x || args[j].x2 != args[0].x2 ||
        args[j].x_len != args[0].x_len || args[j].x_stride != args[0].x_stride || args[j].w->bpr != args[0].w->bpr)
      return false;
  return true;
}

// LMB_ERR_LIMIT, and nothing launched: the estimate is above limit_us, or the workspaces would have to grow while
// the stream is capturing.
int launch_batched(lmb_ctx *ctx, const LinearArgs *args, int njobs, bool rotate, int xmode, float eps, float limit_us) {
  const int kind = args[0].w->kind, W = 4 * bt_halves(kind);
  size_t row_tiles[BT_MAX_JOBS];
  for (int j = 0; j < njobs; ++j) row_tiles[j] = args[j].w->row_tiles;
  const BtPlan pl = plan_batched(kind, row_tiles, njobs, args[0].w->bpr, args[0].batch, ctx->sm_count, ctx->batched_force_seqs, ctx->batched_force_ctas);
  if (pl.n_stages < 2 || pl.us > limit_us) return LMB_ERR_LIMIT;
  if (pl.scratch > ctx->scratch_floats || pl.counters > ctx->n_counters || pl.img_records > ctx->xprep_blocks) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    LMB_CUDA(cudaStreamIsCapturing(ctx->stream, &cs));
    if (cs != cudaStreamCaptureStatusNone) return LMB_ERR_LIMIT;
    LMB_CUDA(cudaStreamSynchronize(ctx->stream));
    int st = ensure_scratch(ctx, pl.scratch, pl.counters);
    if (st == LMB_OK) st = ensure_xprep(ctx, pl.img_records);
    if (st != LMB_OK) return st;
  }
  BtParams p{};
  p.njobs = njobs;
  p.n_rg = pl.n_rg;
  p.bpr = int(args[0].w->bpr);
  p.batch = int(args[0].batch);
  p.ns = pl.ns;
  p.n_stages = pl.n_stages;
  p.stage_bytes = pl.stage_bytes;
  p.img = reinterpret_cast<const uint8_t *>(ctx->xprep);
  p.scratch = ctx->scratch;
  p.counters = ctx->counters;
  p.fault = ctx->d_fault;
  p.spin_limit = ctx->batched_spin_limit;
  p.extra_arrivals = ctx->batched_extra_arrivals;
#ifdef LMB_DEBUG_BOUNDS
  p.scratch_floats = pl.scratch;
#endif
  int rg = 0;
  for (int j = 0; j < njobs; ++j) {
    const lmb_weight *w = args[j].w;
    BtJob &jb = p.job[j];
    jb.tiles = w->d_tiles;
    jb.y = args[j].y;
    jb.bias = args[j].bias;
    jb.residual = args[j].residual;
    jb.M = int(w->M);
    jb.row_tiles = int(w->row_tiles);
    jb.rg_first = rg;
    jb.y_stride = unsigned(args[j].y_stride);
#ifdef LMB_DEBUG_BOUNDS
    jb.tiles_bytes = w->bytes > g_bounds_shrink ? w->bytes - g_bounds_shrink : 0;
    jb.y_floats = (args[j].batch - 1) * args[j].y_stride + w->M;
#endif
    rg += int((w->row_tiles + W - 1) / W);
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned((p.bpr + 7) / 8), unsigned(p.batch));
  cfg.blockDim = dim3(BT_PREP_THREADS);
  cfg.stream = ctx->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = ctx->pdl ? 1 : 0;
  LMB_CUDA(cudaLaunchKernelEx(&cfg, k_prepare_batched, args[0].x, args[0].x2, unsigned(args[0].x_len), unsigned(args[0].x_stride), p.bpr, xmode,
                              rotate ? 1 : 0, eps, p.ns, reinterpret_cast<uint8_t *>(ctx->xprep), timeline_slot(ctx)));
  ctx->launches++;
  p.dbg = timeline_slot(ctx);
  switch (kind) {
  case LMB_INT4: return launch_kind<LMB_INT4>(ctx, p, pl);
  case DK_TERNARY_MMA: return launch_kind<DK_TERNARY_MMA>(ctx, p, pl);
  case DK_INT2_MMA: return launch_kind<DK_INT2_MMA>(ctx, p, pl);
  case DK_BINARY_MMA: return launch_kind<DK_BINARY_MMA>(ctx, p, pl);
  case LMB_INT5: return launch_kind<LMB_INT5>(ctx, p, pl);
  case LMB_INT6: return launch_kind<LMB_INT6>(ctx, p, pl);
  case DK_INT8_MMA: return launch_kind<DK_INT8_MMA>(ctx, p, pl);
  case DK_INT3_MMA: return launch_kind<DK_INT3_MMA>(ctx, p, pl);
  default: return LMB_ERR_ARG;
  }
}

}  // namespace lmb

extern "C" int lmb_debug_batched_plan(lmb_ctx *ctx, int seqs_per_pass, int ctas) {
  LMB_REQUIRE(ctx && seqs_per_pass >= 0 && seqs_per_pass <= lmb::BT_MAX_SEQS && seqs_per_pass % 4 == 0 && ctas >= 0,
              "lmb_debug_batched_plan: bad argument");
  ctx->batched_force_seqs = seqs_per_pass;
  ctx->batched_force_ctas = ctas;
  return LMB_OK;
}

extern "C" int lmb_debug_batched_waits(lmb_ctx *ctx, int extra_arrivals, unsigned spin_limit) {
  LMB_REQUIRE(ctx && extra_arrivals >= 0, "lmb_debug_batched_waits: bad argument");
  ctx->batched_extra_arrivals = extra_arrivals;
  ctx->batched_spin_limit = spin_limit ? spin_limit : (1u << 22);
  return LMB_OK;
}
