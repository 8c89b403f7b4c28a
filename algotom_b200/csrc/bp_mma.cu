// Back-projection of slice stacks on the fifth-generation tensor cores.
//
// All slices of a stack share angles and centre, so for one angle the
// back-projection of a pixel tile is a product
//     out[pixel][slice] += W[pixel][bin] * s[bin][slice]
// whose matrix W holds the two interpolation weights (1 - f, f) of every
// pixel and is the same for all slices (the sums of algotom's
// back-projectors, algotom/rec/reconstruction.py:156-359).  A tile of 8 x 8
// pixels sees at most 12 neighbouring detector bins at any angle, so one
// tcgen05.mma of K = 16 covers an angle.  The gather kernel
// (backproject.cu) reads one 8-byte interpolation pair from shared memory
// for every update, which bounds it at 16 updates per clock and SM whatever
// the number of slices; here the weights of a pixel are formed once and
// serve up to 32 slices.
//
// Precision.  Both factors are split in two float16 terms:
// - positions are 32-bit fixed point (2^-26 bins) from an FP64 origin per
//   (tile, angle), their fraction rounded to 20 bits: 10 for the high weight
//   (integers 1024 - u and u in units of 2^-10) and 10 for the low one
//   (-v, v in units of 2^-20); the weights are exact in float16 and sum to 1;
// - samples, scaled per slice by a power of two to below 2^15, are hi + lo
//   float16: 22 bits down to 2^-17 of the slice's largest sample, and a fixed
//   2^-40 of that sample below.
// The accumulator tile has 128 rows, 64 pixels x (high, low weight), and 2 S
// columns, S slices x (hi, lo): all four partial products.  The tensor cores
// add in FP32 with truncation (measured: a relative bias of 5e-8 over 8
// additions, 1.3e-7 over 16, 2.5e-5 over 1024), so the sums leave TMEM every 16
// angles (8 with edge padding and where the angles are many for the image) and are
// added with Kahan compensation in registers; the other three products, below 2^-10 of the high terms' one, stay
// in TMEM to the end.  A pixel is rounded once, after the small terms joined.
// Error against FP64 at 901 x 1024: 1.4e-7 (2.3e-7 with the gather kernel,
// whose positions carry 1e-5 bins of FP32 rounding).
//
// A stack that holds a non-finite sample (0 times an infinity must stay out of
// the pixels that do not read it), or so faint ones beside its largest that 2^-40
// of that shows, is left to the gather kernel: the scan for the slices' largest
// magnitudes and the packing see it (bp_left_to_gather), this kernel's CTAs leave
// at once and the gather kernel's CTAs, launched behind a gate, run.
//
// One CTA (one per SM) owns 16 x 16 pixels, four tiles, and walks the angles in
// chunks of 8:
// - staging warps form the angle parameters (FP64) and request the region's
//   bins by TMA, 28 bins of all slices per angle, four chunks in flight.  The
//   sinogram is repacked before as [angle][8 slices][bin][8], so that shared
//   memory holds an MN-major operand without swizzle, in which a window may
//   start at any bin;
// - each tile's four weight warps build one row of W per thread (16 float16,
//   two of them non-zero) for 4 angles and store them to TMEM (two slots);
// - one warp per tile issues its MMAs;
// - four warps read each tile's sums, zero them and keep the compensated
//   totals, in registers that the other warps give up.
// The tiles' sums end in turn, so that one tile's read is covered by the
// others' MMAs.  What bounds it: the weight warps' issue (69 % of all issue slots
// taken, the integer pipe 58 %), which is why the cost of a launch hardly depends
// on the number of slices; the tensor cores are busy 46 % of the time.  Under
// sustained load the power cap sets the clock (1.70 GHz).
// Measured, 1801 angles of 2560 bins, 32 slices, no mask: 55.7 ms against
// 100.5 ms with the gather kernel (6.8e12 and 3.8e12 updates/s); 901 x 1280: 6.0
// against 10.0 ms with 24 slices, 5.4 against 6.8 with 16.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <cstring>
#include <mutex>
#include <type_traits>

#include "bp.cuh"
#include "common.cuh"

namespace {

constexpr int kTile = 8;                  // tile edge (pixels)
constexpr int kRegion = 2 * kTile;        // region edge: four tiles
constexpr int kBins = 28;                 // bins staged per angle: 12 (the largest offset of a tile) + 16
constexpr int kChunk = 8;                 // angles per chunk
constexpr int kRing = 4;                  // chunks in flight
constexpr int kStep = 4;                  // angles per weight slot
// Steps between two reads of an accumulator: 16 angles, or 8 (fold_steps)
constexpr int kFoldLong = 4, kFoldShort = 2;
// warps 0-15 form the weights (four for each tile), 16-19 keep the totals,
// 20-23 issue a tile's MMAs each, 25-27 stage (every third chunk each: one warp
// alone, waiting for its FP64 results, takes 2.29 ms at 361 x 1024 with 32
// slices where three take 1.81; four, with warp 24, 1.86)
constexpr int kTotals = 16, kIssuers = 20, kProducers = 24;
constexpr int kThreads = 28 * 32;
// registers per thread of the three kinds: 512 x 64 + 128 x 168 + 256 x 40 =
// 896 x 72, what the block is launched with
constexpr int kRegsWeights = 64, kRegsTotals = 168, kRegsHelpers = 40;
constexpr int kFrac = 26;                 // fraction bits of a position
constexpr float kTolBins = 2e-3f;         // as the gather kernel's edge decision
constexpr int kHeader = 512;              // workspace bytes before the packed samples: the gate's words
static_assert(atb::kGateWords * sizeof(unsigned) <= kHeader, "the gate fits its header");
constexpr int kNowhere = 11 << kFrac;     // a position whose weights are both zero

__device__ int g_mma_status;  // bit 0: a CTA gave up waiting
constexpr unsigned long long kWaitLimit = 1000000000ull;  // ns: about a second, against microseconds in normal operation

struct MmaArgs {
  const unsigned *maxbits;  // [S] largest |sample| of each slice, as bits
  const unsigned *gate;     // bp_left_to_gather, for ngate slices
  int ngate;
  const double2 *trig;
  int nrow, ncol, nsl;  // nsl: live slices (<= S)
  double center;
  int edge_pad;
  double mask_r2;
  float scale;
  float *out;
  long long ors, oss;
  double interior;  // >= 0: only the blocks of bp_interior (centre groups)
  int inject;       // test only: CTA (0, 0) arms its first copies for 16 bytes
                    // more than they deliver
};

// parameters of one (angle, tile)
struct __align__(16) TilePrm {
  int base, c, s;  // fixed-point position of the tile's first pixel in its window, and its steps
  int off;         // the window's shared-memory address / 16; bit 30: checked
};
struct EdgePrm {
  int qlo, qmax;  // fixed-point positions of bins 0 and ncol - 1
};

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t *bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t *bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, unsigned bytes) {
  asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_test(uint64_t *bar, unsigned parity) {
  unsigned done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return done != 0;
}
// Waits for the phase of the given parity; gives up after kWaitLimit, or at once
// when another thread of the CTA has (*bad).  Then nothing more is requested, the
// other warps walk on to the end without waiting, over parameters that keep every
// access inside its buffer whatever has arrived, and no pixel is written.  (With
// a vote and a way out of the loop after each wait the kernel takes 8-12 % longer.)
__device__ __forceinline__ void mbar_wait(uint64_t *bar, unsigned parity, volatile int *bad) {
  unsigned long long t0 = 0, t;
  for (int n = 1; !mbar_test(bar, parity); ++n) {
    if (n & 63) continue;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    if (t0 == 0) t0 = t;
    if (*bad || t - t0 > kWaitLimit) {
      *bad = 1;
      return;
    }
  }
}
__device__ __forceinline__ void tma_load_3d(void *dst, const CUtensorMap *map, int x, int y, int z, uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
      "[%5];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ bool elect_one() {
  unsigned p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
  return p != 0;
}
__device__ __forceinline__ void commit(uint64_t *bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}
// D[d] (+)= A[a] B with A [128 x 16] in TMEM, B [16 x N] in shared memory
__device__ __forceinline__ void mma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t add) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d),
      "r"(a), "l"(b), "r"(idesc), "r"(add)
      : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t t, const uint32_t *w) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(t),
      "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]), "r"(w[8]), "r"(w[9]), "r"(w[10]), "r"(w[11]), "r"(w[12]), "r"(w[13]), "r"(w[14]), "r"(w[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t t, const uint32_t *w) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(t), "r"(w[0]),
               "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
               : "memory");
}
// S columns, complete on return
template <int S> __device__ __forceinline__ void tmem_ld(uint32_t t, float *r);
template <> __device__ __forceinline__ void tmem_ld<8>(uint32_t t, float *r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7])
      : "r"(t)
      : "memory");
}
template <> __device__ __forceinline__ void tmem_ld<16>(uint32_t t, float *r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7]), "=f"(r[8]), "=f"(r[9]), "=f"(r[10]), "=f"(r[11]), "=f"(r[12]), "=f"(r[13]), "=f"(r[14]), "=f"(r[15])
      : "r"(t)
      : "memory");
}
template <> __device__ __forceinline__ void tmem_ld<24>(uint32_t t, float *r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%24];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%16, %17, %18, %19, %20, %21, %22, %23}, [%25];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7]), "=f"(r[8]), "=f"(r[9]), "=f"(r[10]), "=f"(r[11]), "=f"(r[12]), "=f"(r[13]), "=f"(r[14]), "=f"(r[15]), "=f"(r[16]), "=f"(r[17]), "=f"(r[18]), "=f"(r[19]), "=f"(r[20]), "=f"(r[21]), "=f"(r[22]), "=f"(r[23])
      : "r"(t), "r"(t + 16u)
      : "memory");
}
template <> __device__ __forceinline__ void tmem_ld<32>(uint32_t t, float *r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7]), "=f"(r[8]), "=f"(r[9]), "=f"(r[10]), "=f"(r[11]), "=f"(r[12]), "=f"(r[13]), "=f"(r[14]), "=f"(r[15]), "=f"(r[16]), "=f"(r[17]), "=f"(r[18]), "=f"(r[19]), "=f"(r[20]), "=f"(r[21]), "=f"(r[22]), "=f"(r[23]), "=f"(r[24]), "=f"(r[25]), "=f"(r[26]), "=f"(r[27]), "=f"(r[28]), "=f"(r[29]), "=f"(r[30]), "=f"(r[31])
      : "r"(t)
      : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float &lo, float &hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long sub2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  const unsigned long long m1 = 0xbf800000bf800000ull;  // -1, -1: a - b in one rounding
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(b), "l"(m1), "l"(a));
  return r;
}

__device__ __forceinline__ __half2 as_half2(uint32_t v) { return *reinterpret_cast<const __half2 *>(&v); }

// Where the two halves of V = (1 - f, f) go in a row of W, for each bin j the
// selectors of six byte permutes: bin b takes the first half (0x10) where it is
// j, the second (0x32) where it is j + 1, else zero (0x44).  Row 11 (kNowhere)
// takes neither.
struct BinSelect {
  uint4 w03[12];
  uint4 w45[12];  // (two words used: one index serves both loads)
};
__device__ __forceinline__ uint32_t select_bytes(int j, int word) {
  uint32_t v = 0x4444u;
  for (int t = 0; t < 2; ++t) {
    const int b = j + t - 2 * word;
    if (j < 11 && b >= 0 && b < 2) v ^= (t ? 0x76u : 0x54u) << (8 * b);
  }
  return v;
}
// a row of the table by its shared-memory address (it is written once, before
// the warps part)
__device__ __forceinline__ void load_select(uint32_t addr, uint32_t *x) {
  asm("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(x[0]), "=r"(x[1]), "=r"(x[2]), "=r"(x[3]) : "r"(addr));
  asm("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(x[4]), "=r"(x[5]) : "r"(addr + (uint32_t)(12 * sizeof(uint4))));
}
// bytes of v (0-3) and zero bytes (4); __byte_perm masks the selector first
__device__ __forceinline__ uint32_t permute(uint32_t v, uint32_t select) {
  uint32_t r;
  asm("prmt.b32 %0, %1, 0, %2;" : "=r"(r) : "r"(v), "r"(select));
  return r;
}

template <int S>
struct MmaCfg {
  static constexpr int N = 2 * S, G = N / 8;
  static constexpr int kAngleBytes = G * kBins * 16;  // one angle's bins: [G][kBins][8] float16
  static constexpr size_t kRingBytes = (size_t)kRing * kChunk * kAngleBytes;
  static constexpr size_t kPrmBytes = (size_t)kRing * kChunk * 4 * sizeof(TilePrm);
  static constexpr size_t kEdgeBytes = (size_t)kRing * kChunk * 4 * sizeof(EdgePrm);
  static constexpr size_t kSmem = kRingBytes + kPrmBytes + kEdgeBytes + 128;
  static_assert(kRingBytes >= (size_t)768 * (S + 1) * sizeof(float), "the epilogue's totals fit the ring");
};

// Parameters of one (angle, tile) of the region whose first pixel is
// (x0, y0), the angle's bins staged at shared-memory address bins; returns the
// first staged bin (the same for the four tiles).
__device__ __forceinline__ int angle_params(const MmaArgs &a, int i, int x0, int y0, int tile, uint32_t bins,
                                            TilePrm &prm, EdgePrm &edge) {
  const double ic = 0.5 * (double)(a.ncol - 1), last = (double)(a.ncol - 1);
  double2 cs = make_double2(0.0, 0.0);
  if (i < a.nrow) cs = a.trig[i];
  const double P0 = ((double)x0 - ic) * cs.x + ((double)y0 - ic) * cs.y + a.center;
  prm = {kNowhere, 0, 0, (int)(bins >> 4)};
  edge = {0, 0};
  if (i >= a.nrow || !isfinite(P0) || !(fabs(cs.x) <= 1.0) || !(fabs(cs.y) <= 1.0)) return -1;
  const double rmin = P0 + fmin(0.0, (kRegion - 1) * cs.x) + fmin(0.0, (kRegion - 1) * cs.y);
  const double rmax = P0 + fmax(0.0, (kRegion - 1) * cs.x) + fmax(0.0, (kRegion - 1) * cs.y);
  int rlo;
  if (rmax < 0.0) rlo = -1;               // every position left of the detector: bin 0
  else if (rmin > last) rlo = a.ncol - 2; // right of it: bin ncol - 1
  else rlo = (int)floor(rmin - 1e-6);
  constexpr double kOne = (double)(1 << kFrac);
  constexpr int kHalfUlp = 1 << (kFrac - 21);  // rounds the fraction to 20 bits
  const double Pt = P0 + (double)((tile & 1) * kTile) * cs.x + (double)((tile >> 1) * kTile) * cs.y;
  const double pmin = Pt + fmin(0.0, (kTile - 1) * cs.x) + fmin(0.0, (kTile - 1) * cs.y);
  const double pmax = Pt + fmax(0.0, (kTile - 1) * cs.x) + fmax(0.0, (kTile - 1) * cs.y);
  // the window of 16 bins inside the staged ones: a tile's positions span at
  // most 9.9 bins, so the weights lie in the first 12; the window of a tile
  // beyond the detector whose edge sample is wanted still holds that
  double want = floor(pmin - 1e-6);
  if (pmax < 0.0) want = -1.0;
  if (pmin > last) want = last - 1.0;
  const int off = (int)fmin(fmax(want - (double)rlo, 0.0), (double)(kBins - 16));
  const int lo = rlo + off;
  prm.off = (int)(bins >> 4) + off;
  edge.qlo = (int)(fmin(fmax((double)-lo, -16.0), 16.0) * kOne);
  edge.qmax = (int)(fmin(fmax(last - (double)lo, -16.0), 31.0) * kOne);
  if (pmax < -1e-2 || pmin > last + 1e-2) {
    if (a.edge_pad) prm.base = pmax < 0.0 ? edge.qlo : edge.qmax;  // one edge sample for the whole tile
  } else {
    prm.base = __double2int_rn((Pt - (double)lo) * kOne) + kHalfUlp;
    prm.c = __double2int_rn(cs.x * kOne);
    prm.s = __double2int_rn(cs.y * kOne);
    if (pmin < 1e-2 || pmax > last - 1e-2) prm.off |= 1 << 30;
  }
  return rlo;
}

template <int S, int F>
__global__ void __launch_bounds__(kThreads, 1) bp_mma_kernel(MmaArgs a, const __grid_constant__ CUtensorMap tmap) {
  using K = MmaCfg<S>;
  constexpr int N = K::N;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned char *smem = smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u);
  TilePrm *prm = reinterpret_cast<TilePrm *>(smem + K::kRingBytes);      // [kRing][kChunk][4]
  EdgePrm *edge = reinterpret_cast<EdgePrm *>(smem + K::kRingBytes + K::kPrmBytes);
  __shared__ __align__(8) uint64_t full[kRing], empty[kRing], wfull[4][2], wdone[4][2], ddone[4], dfree[4];
  __shared__ unsigned checked_s[kRing];
  __shared__ uint32_t tmem_slot;
  __shared__ int bad_s;
  __shared__ BinSelect sel;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int x0 = blockIdx.x * kRegion, y0 = blockIdx.y * kRegion;
  const int ncol = a.ncol, cm = ncol / 2;
  if (atb::bp_left_to_gather(a.gate, a.ngate, a.nrow)) return;
  if (a.interior >= 0.0 && !atb::bp_interior(x0, y0, ncol, a.interior)) return;
  // a region wholly outside the circle mask is zero
  if (a.mask_r2 >= 0.0) {
    const long long dx = max(0, max(x0 - cm, cm - (x0 + kRegion - 1)));
    const long long dy = max(0, max(y0 - cm, cm - (y0 + kRegion - 1)));
    if ((double)(dx * dx + dy * dy) > a.mask_r2) {
      for (int e = tid; e < kRegion * kRegion * a.nsl; e += kThreads) {
        const int x = x0 + (e & (kRegion - 1)), r = e / kRegion;
        const int k = r % a.nsl, y = y0 + r / a.nsl;
        if (x < ncol && y < ncol) a.out[y * a.ors + k * a.oss + x] = 0.f;
      }
      return;
    }
  }
  if (tid == 0) {
    for (int r = 0; r < kRing; ++r) {
      mbar_init(&full[r], kChunk + 32);
      mbar_init(&empty[r], 4);  // one per issuer
    }
    for (int q = 0; q < 4; ++q) {
      for (int t = 0; t < 2; ++t) {
        mbar_init(&wfull[q][t], 4);
        mbar_init(&wdone[q][t], 1);
      }
      mbar_init(&ddone[q], 1);
      mbar_init(&dfree[q], 2);  // the two warps of the high rows
    }
    if (a.inject && blockIdx.x == 0 && blockIdx.y == 0) mbar_expect_tx(&full[0], 16u);
    bad_s = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (tid < 12) {
    sel.w03[tid] = make_uint4(select_bytes(tid, 0), select_bytes(tid, 1), select_bytes(tid, 2), select_bytes(tid, 3));
    sel.w45[tid] = make_uint4(select_bytes(tid, 4), select_bytes(tid, 5), 0u, 0u);
  }
  // parameters that no chunk has written yet: no weights, a window inside the ring
  if (tid < kRing * kChunk * 4) {
    prm[tid] = {kNowhere, 0, 0, (int)(smem_u32(smem) >> 4)};
    edge[tid] = {0, 0};
  }
  if (tid < kRing) checked_s[tid] = 0u;
  if (warp == kProducers) {
    asm volatile(
        "tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;\n\t"
        "tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::"r"(smem_u32(&tmem_slot))
        : "memory");
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t *>(&tmem_slot);
  volatile int *bad = &bad_s;
  const int nchunk = (a.nrow + kChunk - 1) / kChunk;

  const int nstep = nchunk * (kChunk / kStep);

  if (warp >= kIssuers) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsHelpers));
  if (warp >= kProducers) {
    // lane = angle of the chunk and tile
    const int ai = lane >> 2;
    for (int k = warp - kProducers - 1; warp > kProducers && k < nchunk; k += 3) {
      const int r = k % kRing;
      if (k >= kRing) {
        mbar_wait(&empty[r], (unsigned)((k / kRing - 1) & 1), bad);
        // (full[r] may still be short of bytes: another arrival would fault)
        if (__any_sync(0xffffffffu, *bad)) break;
      }
      unsigned char *dst = smem + (size_t)(r * kChunk + ai) * K::kAngleBytes;
      const int e = r * kChunk * 4 + lane;
      const int rlo = angle_params(a, k * kChunk + ai, x0, y0, lane & 3, smem_u32(dst), prm[e], edge[e]);
      unsigned chk = prm[e].off & (1 << 30) ? 1u << (lane & 3) : 0u;
      chk = __reduce_or_sync(0xffffffffu, chk);
      if (lane == 0) checked_s[r] = chk;
      mbar_arrive(&full[r]);  // this lane's parameters
      if ((lane & 3) == 0) {
        mbar_arrive_expect_tx(&full[r], K::kAngleBytes);
        tma_load_3d(dst, &tmap, rlo * 8, 0, k * kChunk + ai, &full[r]);
      }
    }
    __syncwarp();
  } else if (warp >= kIssuers) {
    // one warp issues the MMAs of one tile (alone it issues one in 45 clocks,
    // the tensor cores take 32).  All lanes walk the loop, which keeps the
    // operands in uniform registers; one of them issues
    const int q = warp - kIssuers;
    // D float32; A, B float16; B MN-major; N, M
    const uint32_t idesc = (1u << 4) | (1u << 16) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
    // no swizzle; 8 bins are 128 bytes (leading), 8 slices kBins * 16 (stride)
    const uint64_t bdesc = ((uint64_t)(128 >> 4) << 16) | ((uint64_t)((kBins * 16) >> 4) << 32) | (1ull << 46);
    const uint32_t dcol = tmem + (uint32_t)(q * N), wcol = tmem + 256u + (uint32_t)(q * 2 * 8 * kStep);
    const bool elected = elect_one();
#pragma unroll 1
    for (int k = 0; k < nchunk; ++k) {
      const int r = k % kRing;
      mbar_wait(&full[r], (unsigned)((k / kRing) & 1), bad);
#pragma unroll
      for (int st = 0; st < kChunk / kStep; ++st) {
        const int slot = st & 1, step = k * (kChunk / kStep) + st;
        uint64_t b[kStep];
#pragma unroll
        for (int u = 0; u < kStep; ++u)
          b[u] = bdesc | (uint64_t)(prm[(r * kChunk + st * kStep + u) * 4 + q].off & 0x3fff);
        mbar_wait(&wfull[q][slot], (unsigned)((step >> 1) & 1), bad);
        // a sum ends with step F i + q % F (the tiles take turns); before the
        // next one starts its accumulator has been read and zeroed
        if (step == 0 || step % F == (q + 1) % F)
          mbar_wait(&dfree[q], (unsigned)((step == 0 ? 0 : (step - q % F - 1) / F + 1) & 1), bad);
        fence_after();
        if (elected) {
#pragma unroll
          for (int u = 0; u < kStep; ++u) mma_ts(dcol, wcol + (uint32_t)(8 * (slot * kStep + u)), b[u], idesc, 1u);
          commit(&wdone[q][slot]);
          if (step % F == q % F || step == nstep - 1) commit(&ddone[q]);
          if (st == kChunk / kStep - 1) commit(&empty[r]);
        }
        __syncwarp();
      }
    }
  } else if (warp >= kTotals) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsTotals));
    // Rows 0-63 and 64-127 of an accumulator hold a tile's high and low
    // weights, the other way round in odd tiles; its columns the hi and the lo
    // samples.  Only the product of the two high terms is summed here: the
    // other three weigh 2^-10 and less of it, and stay in the accumulator to
    // the end.  thread = lane of TMEM = high row of tiles t0 and t0 + 2
    const int row = tid & 127, px = row & 63, t0 = row >> 6;
    const uint32_t dlane = tmem + ((uint32_t)((row >> 5) * 32) << 16);
    uint32_t zero[16];
#pragma unroll
    for (int z = 0; z < 16; ++z) zero[z] = 0u;
    for (int c = 0; c < 4 * N; c += 16) tmem_st16(dlane + (uint32_t)c, zero);
    tmem_wait_st();
    fence_before();
    asm volatile("bar.sync 1, 128;" ::: "memory");
    if (lane == 0) {
      mbar_arrive(&dfree[t0]);
      mbar_arrive(&dfree[t0 + 2]);
    }
    unsigned long long sum[2][S / 2], comp[2][S / 2];
#pragma unroll
    for (int g = 0; g < S / 2; ++g) sum[0][g] = sum[1][g] = comp[0][g] = comp[1][g] = 0ull;
    auto fold = [&](int q, unsigned long long *s, unsigned long long *c) {
      fence_after();
      const uint32_t dcol = dlane + (uint32_t)(q * N);
      float d[S];
      tmem_ld<S>(dcol, d);
#pragma unroll
      for (int p = 0; p < S / 8; ++p) tmem_st8(dcol + 8u * p, zero);
      tmem_wait_st();
      fence_before();
      if (lane == 0) mbar_arrive(&dfree[q]);
#pragma unroll
      for (int g = 0; g < S / 2; ++g) {
        const unsigned long long y = sub2(pack2(d[2 * g], d[2 * g + 1]), c[g]), t = add2(s[g], y);
        c[g] = sub2(sub2(t, s[g]), y);
        s[g] = t;
      }
    };
#pragma unroll 1
    for (int i = 0; F * (i - 1) + t0 % F < nstep - 1 || i == 0; ++i) {
      // sum i of the first tile, and of the second where it has one
      mbar_wait(&ddone[t0], (unsigned)(i & 1), bad);
      fold(t0, sum[0], comp[0]);
      if (i == 0 || F * (i - 1) + (t0 + 2) % F < nstep - 1) {
        mbar_wait(&ddone[t0 + 2], (unsigned)(i & 1), bad);
        fold(t0 + 2, sum[1], comp[1]);
      }
    }
    asm volatile("bar.sync 1, 128;" ::: "memory");  // every MMA is done (or given up)
    fence_after();
    // totals to the ring, which nothing reads any more:
    // [high sums, the rest of them, low][pixel of 4 tiles][S + 1]
#pragma unroll 1
    for (int q = 0; q < 4; ++q) {
      const bool high = (q & 1) == t0;
      float *dst = reinterpret_cast<float *>(smem) + (q * 64 + px) * (S + 1);
      const uint32_t dcol = dlane + (uint32_t)(q * N);
#pragma unroll
      for (int p = 0; p < S / 8; ++p) {
        float hi[8], lo[8];
        tmem_ld<8>(dcol + 8u * p, hi);
        tmem_ld<8>(dcol + S + 8u * p, lo);
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          const int n = 4 * p + g;
          if (high) {
            float c0, c1;
            unpack2(q < 2 ? sum[0][n] : sum[1][n], dst[2 * n], dst[2 * n + 1]);
            unpack2(q < 2 ? comp[0][n] : comp[1][n], c0, c1);
            dst[256 * (S + 1) + 2 * n] = lo[2 * g] - c0;
            dst[256 * (S + 1) + 2 * n + 1] = lo[2 * g + 1] - c1;
          } else {
            dst[512 * (S + 1) + 2 * n] = hi[2 * g] + lo[2 * g];
            dst[512 * (S + 1) + 2 * n + 1] = hi[2 * g + 1] + lo[2 * g + 1];
          }
        }
      }
    }
    fence_before();
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsWeights));
    // thread = row of one tile's W
    const int quad = warp >> 2, row = tid & 127;
    const int px = row & 63, tx = px & 7, ty = px >> 3;
    const bool high = (row < 64) == ((quad & 1) == 0);
    const uint32_t up = high ? 1u << (32 - kFrac) : 1u << (42 - kFrac);  // the fraction's ten bits to the top
    const uint32_t selbase = smem_u32(&sel);
    const __half2 minus = __halves2half2(__float2half_rn(high ? -1024.f : -2048.f), __float2half_rn(-1024.f));
    const uint32_t wcol = tmem + ((uint32_t)((row >> 5) * 32) << 16) + 256u + (uint32_t)(quad * 2 * 8 * kStep);

    // The weights of kStep angles from ring entry e (angle i of the launch).  How
    // these loops lie in the instruction cache, which 28 warps share, matters: with
    // the rarer checked form rolled up and a chunk's two steps unrolled, 901 x 1280
    // takes 5.38 (16 slices), 6.01 (24) and 6.36 ms (32); both forms unrolled and
    // the steps rolled up, 5.93, 6.47 and 6.76.
    auto weights = [&](auto checked_tag, int e, int i, uint32_t col) {
      constexpr bool kChecked = decltype(checked_tag)::value;
      const TilePrm *pp = prm + e * 4 + quad;
#pragma unroll (kChecked ? 1 : 2)
      for (int u2 = 0; u2 < kStep; u2 += 2) {
        uint32_t w[16];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const TilePrm p = pp[4 * (u2 + u)];
          int q = p.base + tx * p.c + ty * p.s;
          if constexpr (kChecked) {
            if (p.off & (1 << 30)) {  // the tile reaches an edge of the detector
              const EdgePrm ed = edge[(e + u2 + u) * 4 + quad];
              bool in = true;
              if (!a.edge_pad) {
                in = q >= ed.qlo && q <= ed.qmax + (1 << (kFrac - 21));
                constexpr int kTol = (int)(kTolBins * (float)(1 << kFrac));
                if (abs(q - ed.qlo) < kTol || abs(q - ed.qmax) < kTol) {
                  // the reference's expression and rounding order in FP64
                  const double ic = 0.5 * (double)(ncol - 1);
                  const double2 cs = a.trig[min(i + u2 + u, a.nrow - 1)];  // (past it only after a wait gave up)
                  const double xq = x0 + (quad & 1) * kTile + tx, yq = y0 + (quad >> 1) * kTile + ty;
                  const double pe =
                      __dadd_rn(__dadd_rn(__dmul_rn(xq - ic, cs.x), __dmul_rn(yq - ic, cs.y)), a.center);
                  in = pe >= 0.0 && pe <= (double)(ncol - 1);
                }
              }
              q = in ? min(max(q, ed.qlo), ed.qmax) : kNowhere;
            }
          }
          // ten bits of the fraction: the float16 pair (1024 - f, f), in the
          // low weights (-f, f), from (1024 + 1024 - f, 1024 + f)
          const uint32_t f = ((uint32_t)q * up) >> 22;
          const __half2 v = __hadd2(as_half2(f * 65535u + (0x64006400u + 1024u)), minus);
          const uint32_t V = *reinterpret_cast<const uint32_t *>(&v);
          uint32_t x[6];
          load_select(selbase + 16u * ((uint32_t)q >> kFrac), x);
#pragma unroll
          for (int z = 0; z < 6; ++z) w[8 * u + z] = permute(V, x[z]);
          w[8 * u + 6] = w[8 * u + 7] = 0u;
        }
        tmem_st16(col + 8u * u2, w);
      }
    };

    int step = 0;  // slot step & 1, use step >> 1
#pragma unroll 1
    for (int k = 0; k < nchunk; ++k) {
      const int r = k % kRing;
      mbar_wait(&full[r], (unsigned)((k / kRing) & 1), bad);
      const bool chk = (checked_s[r] >> quad) & 1u;
#pragma unroll
      for (int st = 0; st < kChunk / kStep; ++st, ++step) {
        const int slot = step & 1;
        // the MMAs that read this slot two steps ago are done
        if (step >= 2) mbar_wait(&wdone[quad][slot], (unsigned)(((step >> 1) - 1) & 1), bad);
        fence_after();
        const int e = r * kChunk + st * kStep;
        const uint32_t col = wcol + (uint32_t)(slot * 8 * kStep);
        if (chk) weights(std::true_type{}, e, step * kStep, col);
        else weights(std::false_type{}, e, 0, col);
        tmem_wait_st();
        fence_before();
        if (lane == 0) mbar_arrive(&wfull[quad][slot]);
      }
    }
  }
  fence_before();
  __syncthreads();
  if (*bad) {
    if (tid == 0) atomicOr(&g_mma_status, 1);
    // this CTA's memory stays its own until what is in flight has ended: copies
    // and MMAs, at worst all of them (128 clocks an angle)
    for (int n = 0; n < 64 + a.nrow / 128; ++n) __nanosleep(16000);
    __syncthreads();
  }
  if (!*bad && tid < 3 * kRegion * kRegion) {
    // thread = pixel of the region, and every third slice
    const int xr = tid & (kRegion - 1), yr = (tid / kRegion) & (kRegion - 1);
    const int x = x0 + xr, y = y0 + yr;
    const int q = yr / kTile * 2 + xr / kTile, px = (yr % kTile) * kTile + xr % kTile;
    bool keep = true;
    if (a.mask_r2 >= 0.0) {
      const long long dx = x - cm, dy = y - cm;
      keep = (double)(dx * dx + dy * dy) <= a.mask_r2;
    }
    if (x < ncol && y < ncol) {
      const float *total = reinterpret_cast<const float *>(smem) + (q * 64 + px) * (S + 1);
      float *dst = a.out + y * a.ors + x;
      for (int n = tid / (kRegion * kRegion); n < a.nsl; n += 3) {
        // the small terms first, so that the pixel is rounded once; then undo
        // the sample scale and the weights' 2^10
        const float rest = fmaf(total[512 * (S + 1) + n], 0x1p-10f, total[256 * (S + 1) + n]);
        const float t = __fadd_rn(total[n], rest);
        const float f = ldexpf(t, -(atb::bp_sample_exponent(a.maxbits[n]) + 10));
        dst[n * a.oss] = keep ? f * a.scale : 0.f;
      }
    }
  }
  if (warp == kProducers) {
    fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
  }
}

// Adds a warp's faint pairs (a sample and the one before it, both scaled) to
// *pairs.  Every lane calls it.
__device__ __forceinline__ void count_faint(float v, float before, bool valid, unsigned *pairs) {
  const unsigned n = __popc(__ballot_sync(
      0xffffffffu, valid && fabsf(v) < atb::kFaint && fabsf(before) < atb::kFaint && (v != 0.f || before != 0.f)));
  if (n > 0u && (threadIdx.x & 31) == 0) atomicAdd(pairs, n);
}

// The S "slices" of a centre group: slice m is the one row of each angle, read m
// spacing bins further on.  One word of maxbits serves them all (the others
// repeat it).  count: the first group of a call, which counts the row's faint
// pairs.
__global__ void __launch_bounds__(256) pack_centers_kernel(const float *sino, long long srs, int ncol, int nsl, int S,
                                                           int spacing, bool count, unsigned *maxbits, uint4 *dst) {
  const int i = blockIdx.y, g = blockIdx.z;
  const unsigned bits = maxbits[0];
  if (i == 0 && blockIdx.x == 0 && threadIdx.x < 8) maxbits[S + 8 * g + threadIdx.x] = bits;
  const float sc = __int_as_float((atb::bp_sample_exponent(bits) + 127) << 23);
  const float *row = sino + i * srs;
  uint4 *hi = dst + ((long long)i * (S / 4) + g) * ncol, *lo = hi + (long long)(S / 8) * ncol;
  const int d = blockIdx.x * 256 + threadIdx.x;
  if (count && g == 0) {
    const float v = d < ncol ? __ldg(row + d) * sc : 0.f, before = d > 0 && d < ncol ? __ldg(row + d - 1) * sc : v;
    count_faint(v, before, d > 0 && d < ncol, maxbits + atb::kGatePairs);
  }
  if (d < ncol) {
    unsigned h[4], l[4];
#pragma unroll
    for (int u = 0; u < 8; u += 2) {
      float v[2];
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        const int m = 8 * g + u + t, b = d + m * spacing;
        v[t] = m < nsl && b < ncol ? __ldg(row + b) * sc : 0.f;
      }
      const __half2 hh = __floats2half2_rn(v[0], v[1]);
      const float2 hf = __half22float2(hh);
      const __half2 ll = __floats2half2_rn(v[0] - hf.x, v[1] - hf.y);
      h[u / 2] = *reinterpret_cast<const unsigned *>(&hh);
      l[u / 2] = *reinterpret_cast<const unsigned *>(&ll);
    }
    hi[d] = make_uint4(h[0], h[1], h[2], h[3]);
    lo[d] = make_uint4(l[0], l[1], l[2], l[3]);
  }
}

// largest |sample| of each slice as float bits (monotonic; a NaN ranks above
// infinity).  grid (row blocks, slices), atomics on zeroed words.
template <typename T>
__global__ void __launch_bounds__(256) absmax_kernel(const T *sino, long long srs, long long sss, int nrow, int ncol,
                                                     unsigned *maxbits) {
  const int k = blockIdx.y;
  unsigned m = 0u;
  for (int i = blockIdx.x; i < nrow; i += gridDim.x) {
    const T *row = sino + i * srs + k * sss;
    for (int d = threadIdx.x; d < ncol; d += 256) m = max(m, __float_as_uint(atb::load_as_float(row + d)) & 0x7fffffffu);
  }
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0) atomicMax(maxbits + k, m);
}

// [angle][slice][bin] samples -> [angle][G][bin][8] float16, groups of 8
// slices: first the hi parts of all S slices, then the lo parts.  Counts the
// slices' faint pairs (of 16-bit samples, which one term holds, too).
template <typename T>
__global__ void __launch_bounds__(256) pack_kernel(const T *sino, long long srs, long long sss, int nrow, int ncol,
                                                   int nsl, int S, unsigned *gate, uint4 *dst) {
  const int i = blockIdx.y, g = blockIdx.z, lane = threadIdx.x & 31;
  const T *row = sino + i * srs + 8 * g * sss;
  uint4 *hi = dst + ((long long)i * (S / 4) + g) * ncol, *lo = hi + (long long)(S / 8) * ncol;
  const int d = blockIdx.x * 256 + threadIdx.x;
  unsigned h[4], l[4];
#pragma unroll
  for (int u = 0; u < 8; u += 2) {
    float v[2];
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const int k = 8 * g + u + t;
      v[t] = 0.f;
      if (k >= nsl) continue;
      const float sc = __int_as_float((atb::bp_sample_exponent(gate[k]) + 127) << 23);
      const T *p = row + (u + t) * sss;
      if (d < ncol) v[t] = atb::load_as_float(p + d) * sc;
      float before = __shfl_up_sync(0xffffffffu, v[t], 1);
      if (lane == 0 && d > 0 && d < ncol) before = atb::load_as_float(p + d - 1) * sc;
      count_faint(v[t], before, d > 0 && d < ncol, gate + atb::kGatePairs + k);
    }
    const __half2 hh = __floats2half2_rn(v[0], v[1]);
    const float2 hf = __half22float2(hh);
    const __half2 ll = __floats2half2_rn(v[0] - hf.x, v[1] - hf.y);
    h[u / 2] = *reinterpret_cast<const unsigned *>(&hh);
    l[u / 2] = *reinterpret_cast<const unsigned *>(&ll);
  }
  if (d < ncol) {
    hi[d] = make_uint4(h[0], h[1], h[2], h[3]);
    lo[d] = make_uint4(l[0], l[1], l[2], l[3]);
  }
}

PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  });
  return fn;
}

// The packed samples as a tensor: false where the driver has no tensor maps, and
// the gather kernel takes the stack (as it stages without them).
bool packed_map(int S, int nrow, int ncol, void *packed, CUtensorMap *map) {
  auto encode = tensor_map_encoder();
  std::memset(map, 0, sizeof(*map));
  const cuuint64_t G = (cuuint64_t)S / 4;
  const cuuint64_t dims[3] = {(cuuint64_t)ncol * 8, G, (cuuint64_t)nrow};
  const cuuint64_t strides[2] = {(cuuint64_t)ncol * 16, (cuuint64_t)ncol * 16 * G};
  const cuuint32_t box[3] = {kBins * 8, (cuuint32_t)G, 1u};
  const cuuint32_t estr[3] = {1u, 1u, 1u};
  return encode && encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, packed, dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int S, int F>
int launch_mma(const MmaArgs &a, const CUtensorMap &map, cudaStream_t st) {
  using K = MmaCfg<S>;
  static_assert(K::G == S / 4, "as packed_map");
  auto fn = bp_mma_kernel<S, F>;
  const int rc = atb::ensure_smem(fn, K::kSmem, "atb_backproject_stack", kThreads, 512);
  if (rc != ATB_OK) return rc;
  const int n = (a.ncol + kRegion - 1) / kRegion;
  fn<<<dim3(n, n), kThreads, K::kSmem, st>>>(a, map);
  return atb::check_launch("atb_backproject_stack");
}

// Steps between two reads of an accumulator.  The truncations add up to a bias,
// the same for every pixel, that the angles do not average out: after 16 angles
// 1.4e-7 of an image, after 8 0.7e-7 (half of it at 200 pixels).  The gather
// kernel's error, from its positions, falls as the angles and grows with the
// image, 2.2e-7 (ncol / 1024) sqrt(901 / nrow), so that 16 angles are the less
// exact choice from nrow = ncol^2 / 450 on.  Errors of filtered sinograms
// against FP64 with 16 angles, with 8, and with the gather kernel (1e-8):
//   901 x 200: 10.1, 3.8, 6.5;  901 x 512: 13.6, 6.2, 12.0;  901 x 1024: 14.1,
//   7.8, 22.5;  1801 x 320: 11.8, 4.9, 6.2;  1801 x 720: 13.8, 6.5, 11.6
// 8 angles cost 1801 x 2560 with 32 slices 59.1 ms instead of 56.1.  With edge
// padding (BPF) the samples have one sign, so that the bias is the larger, and the
// 2-D ramp filter magnifies it: BPF of 901 x 1280 has 4.0e-6 with 8 and 4.1e-6
// with 16 angles (4.2e-6 with the gather kernel).
int fold_steps(const MmaArgs &a) {
  return a.edge_pad || (long long)a.ncol * a.ncol < 500ll * a.nrow ? kFoldShort : kFoldLong;
}

int launch(const MmaArgs &a, int S, const CUtensorMap &map, cudaStream_t st) {
  if (fold_steps(a) == kFoldShort)
    return S == 16   ? launch_mma<16, kFoldShort>(a, map, st)
           : S == 24 ? launch_mma<24, kFoldShort>(a, map, st)
                     : launch_mma<32, kFoldShort>(a, map, st);
  return S == 16   ? launch_mma<16, kFoldLong>(a, map, st)
         : S == 24 ? launch_mma<24, kFoldLong>(a, map, st)
                   : launch_mma<32, kFoldLong>(a, map, st);
}

template <typename T>
int prepare(const void *sino, long long srs, long long sss, int nrow, int nsl, int ncol, int S, void *work,
            cudaStream_t st) {
  unsigned *maxbits = static_cast<unsigned *>(work);
  uint4 *packed = reinterpret_cast<uint4 *>(static_cast<unsigned char *>(work) + kHeader);
  const T *src = static_cast<const T *>(sino);
  if (cudaMemsetAsync(work, 0, kHeader, st) != cudaSuccess)
    return atb::fail(ATB_ECUDA, "atb_backproject_stack: %s", cudaGetErrorString(cudaGetLastError()));
  const int rows = nrow < 64 ? nrow : 64;
  absmax_kernel<T><<<dim3(rows, nsl), 256, 0, st>>>(src, srs, sss, nrow, ncol, maxbits);
  int rc = atb::check_launch("atb_backproject_stack (scan)");
  if (rc != ATB_OK) return rc;
  pack_kernel<T><<<dim3((ncol + 255) / 256, nrow, S / 8), 256, 0, st>>>(src, srs, sss, nrow, ncol, nsl, S, maxbits,
                                                                       packed);
  return atb::check_launch("atb_backproject_stack (pack)");
}

// slices of the next launch of a stack with n left: 0 if the gather kernel is
// the faster one for all of them.  A launch costs the same for 16 as for 10
// slices, at 901 x 1280 5.4 ms, and the gather kernel 0.43 ms per slice, 6.0 for
// 14; but at 2560 pixels and fewer angles the two meet at 15 and 16
// (fewest_angles).  bfloat16 samples stay with the gather kernel, whose
// interpolation differences are bfloat16 too: a user's results would move by
// that rounding (2e-4) for a faster kernel.  So do stacks of more angles than the
// truncations bear, whose sums the gather kernel, averaging over its positions'
// errors, holds the better (1e-8, 8 angles between two reads, and gather): 7201 x
// 320: 4.7, 3.8; x 512: 5.8, 4.9; 30001 x 200: 4.4, 2.7 (the small products, which
// stay in TMEM to the end, then show).
int next_group(int sino_dtype, int nrow, int ncol, int n) {
  if (sino_dtype == ATB_BF16 || nrow > 8192 || (nrow > 2048 && (long long)ncol * ncol < 120ll * nrow)) return 0;
  if (n >= 32) return 32;
  return n >= 15 ? n : 0;
}
int padded(int n) { return (n + 7) / 8 * 8; }

// Angles from which a group of n slices is worth its scan, packing and launch
// (the gather kernel has one launch, of a cost per slice).  Time against the
// gather kernel's by angles, read off 15 to 32 slices of 32 to 2560 pixels:
//   up to 160 pixels  16 slices: 1.15 (16), 0.85 (24); 32 slices: 1.07 (24), 0.96
//                     (32); whole calls, with three launches more: 1.2 (33)
//   24 slices         512: 1.11 (32), 0.95 (48); 1536: 1.08 (48), 0.94 (64)
//   32                800: 1.06 (24), 1.00 (32), 0.85 (48)
//   21                1536: 1.03 (64), 0.91 (96); 2560: 1.05 (64), 0.93 (96)
//   18, 20            1536: 1.03 (96), 0.96 (128); 2560: 1.05 (96), 0.98 (128)
//   17                800: 1.00 (64); 1536: 1.02 (128), 0.94 (192)
//   16                320: 1.01 (64); 800: 0.98 (128); 1536: 1.01 (256); 2560: 1.00 (384)
//   15                800: 0.94 (64); 1536: 0.99 (256); 2560: 1.00 (384): the two more
//                     launches of the gather kernel's remainder weigh less and less
int fewest_angles(int n, int ncol) {
  if (ncol <= 160) return 64;
  if (n >= 18) return n >= 28 ? 48 : n >= 24 ? 56 : n >= 21 ? 72 : 120;
  const int w = ncol < 1536 ? ncol : 1536;
  const int by_size = n == 17 ? 168 * w / 1536 : n == 16 ? 320 * w / 1536 : 320 * w / 1536 * w / 1536;
  return by_size > 24 ? by_size : 24;
}
// The same for a group of n centres, whose gather kernel reads one sinogram for
// all of them and whose ring stays with it.
//   15  512: 1.06 (16), 0.89 (32); 800: 1.01 (64), 0.89 (128); 1536: 1.06 (128), 0.91 (192)
//   16  320: 1.26 (512); 700: 0.91 (192), 0.87 (361); 1100: 0.95 (361)
//   20  200: 1.15 (512); 400: 0.94 (512); 512: 1.02 (96), 0.93 (128)
//   28  320: 1.02 (512); 400: 0.95 (192); 700: 0.95 (96)
//   32  200: 1.13 (512); 400: 0.97 (512); 700: 0.92 (96); 1536: 0.79 (96)
// Without a remainder of 1 to 3 centres the gather kernel has one launch, and
// small images are mostly ring.
bool centers_worth(int n, int nrow, int ncol) {
  if (n % 4) return nrow >= (ncol > 144 ? ncol / 6 : 24);
  if (n == 16) return nrow >= 256 && ncol >= 640;
  return nrow >= 128 && ncol >= 400;
}

}  // namespace

namespace atb {
int bp_mma_status(int reset) {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_mma_status, sizeof(int)) != cudaSuccess) return -1;
  if (reset && v) {
    const int zero = 0;
    if (cudaMemcpyToSymbol(g_mma_status, &zero, sizeof(int)) != cudaSuccess) return -1;
  }
  return v;
}
}  // namespace atb

extern "C" int64_t atb_backproject_stack_workspace(int sino_dtype, int nrow, int nslice, int ncol) {
  if (nrow < 1 || nslice < 1 || ncol < 1 || nrow > 65535 || ncol > (1 << 16)) return 0;
  const int n = next_group(sino_dtype, nrow, ncol, nslice);
  const int64_t packed = n ? kHeader + (int64_t)nrow * ncol * padded(n) * 4 : 0;
  // the gather kernel's angle groups: of 32 slices, and of what is left over
  const int left = nslice % 32;
  int64_t split = 0;
  if (left && !next_group(sino_dtype, nrow, ncol, left)) split = atb::bp_gather_workspace(nrow, left, ncol);
  if (nslice >= 32 && n == 0) {
    const int64_t whole = atb::bp_gather_workspace(nrow, 32, ncol);
    if (whole > split) split = whole;
  }
  return packed > split ? packed : split;
}

extern "C" int atb_backproject_stack(const void *sino, int sino_dtype, int64_t sino_row_stride,
                                     int64_t sino_slice_stride, int nrow, int nslice, int ncol, const double *trig,
                                     double center, int edge_pad, double mask_r2, float scale, float *out,
                                     int64_t out_row_stride, int64_t out_slice_stride, int flags, void *workspace,
                                     int64_t workspace_bytes, void *stream) {
  if (flags & ~240) return atb::fail(ATB_EINVAL, "atb_backproject_stack: unknown flags %d", flags);
  const bool always = flags & 64, no_maps = flags & 128;
  flags &= ~192;
  cudaStream_t st = atb::as_stream(stream);
  const int64_t need = atb_backproject_stack_workspace(sino_dtype, nrow, nslice, ncol);
  const int esize = sino_dtype == ATB_F32 ? 4 : 2;
  int first = 0;
  const bool work_ok = need > 0 && workspace && workspace_bytes >= need && reinterpret_cast<uintptr_t>(workspace) % 128 == 0;
  const bool args_ok = sino && trig && out && (sino_dtype == ATB_F32 || sino_dtype == ATB_F16 || sino_dtype == ATB_BF16) &&
                       center >= 0.0 && center < (double)ncol;
  if (args_ok && work_ok) {
    for (int n; (n = next_group(sino_dtype, nrow, ncol, nslice - first)) > 0; first += n) {
      if (!always && nrow < fewest_angles(n, ncol)) break;
      const int S = padded(n);
      void *packed = static_cast<unsigned char *>(workspace) + kHeader;
      CUtensorMap map;
      if (no_maps || !packed_map(S, nrow, ncol, packed, &map)) break;
      const char *src = static_cast<const char *>(sino) + (int64_t)first * sino_slice_stride * esize;
      float *dst = out + (int64_t)first * out_slice_stride;
      int rc = sino_dtype == ATB_F32
                   ? prepare<float>(src, sino_row_stride, sino_slice_stride, nrow, n, ncol, S, workspace, st)
                   : prepare<__half>(src, sino_row_stride, sino_slice_stride, nrow, n, ncol, S, workspace, st);
      if (rc != ATB_OK) return rc;
      MmaArgs a;
      a.maxbits = a.gate = static_cast<const unsigned *>(workspace);
      a.ngate = n;
      a.trig = reinterpret_cast<const double2 *>(trig);
      a.nrow = nrow; a.ncol = ncol; a.nsl = n;
      a.center = center; a.edge_pad = edge_pad ? 1 : 0; a.mask_r2 = mask_r2; a.scale = scale;
      a.out = dst; a.ors = out_row_stride; a.oss = out_slice_stride;
      a.interior = -1.0;
      a.inject = (flags >> 5) & 1;
      rc = launch(a, S, map, st);
      if (rc != ATB_OK) return rc;
      // runs only where bp_left_to_gather
      rc = atb::bp_gather(src, sino_dtype, sino_row_stride, sino_slice_stride, nrow, n, ncol, trig, center, edge_pad,
                          mask_r2, scale, dst, out_row_stride, out_slice_stride, flags & 16, a.gate, nullptr, stream);
      if (rc != ATB_OK) return rc;
    }
    if (first == nslice) return ATB_OK;
    // the gather kernel: whole launches of 32 slices, then the rest, so that a
    // slice's bits depend on its place among them and not on how many follow
    auto gather = [&](int n, bool split) {
      const int rc = atb::bp_gather(static_cast<const char *>(sino) + (int64_t)first * sino_slice_stride * esize,
                                    sino_dtype, sino_row_stride, sino_slice_stride, nrow, n, ncol, trig, center,
                                    edge_pad, mask_r2, scale, out + (int64_t)first * out_slice_stride, out_row_stride,
                                    out_slice_stride, flags, nullptr, split ? workspace : nullptr, stream);
      first += n;
      return rc;
    };
    const auto groups = [&](int n) {
      return n > 0 && next_group(sino_dtype, nrow, ncol, n) == 0 && atb::bp_gather_workspace(nrow, n, ncol) > 0;
    };
    const int left = (nslice - first) % 32;
    const bool split = groups(32), split_left = groups(left);
    if (!split && !split_left) return gather(nslice - first, false);  // (one launch has the same bits)
    while (nslice - first > left) {
      const int rc = gather(split ? 32 : nslice - first - left, split);
      if (rc != ATB_OK) return rc;
    }
    return left ? gather(left, split_left) : ATB_OK;
  }
  return atb::bp_gather(sino, sino_dtype, sino_row_stride, sino_slice_stride, nrow, nslice, ncol, trig, center, edge_pad,
                        mask_r2, scale, out, out_row_stride, out_slice_stride, flags, nullptr, nullptr, stream);
}

extern "C" int64_t atb_backproject_centers_workspace(int nrow, int ncol, int ncenter) {
  if (nrow < 1 || ncol < 1 || ncenter < 1 || nrow > 65535 || ncol > (1 << 16)) return 0;
  const int n = next_group(ATB_F32, nrow, ncol, ncenter);
  return n ? kHeader + (int64_t)nrow * ncol * padded(n) * 4 : 0;
}

extern "C" int atb_backproject_centers_stack(const float *sino, int64_t sino_row_stride, int nrow, int ncol,
                                             const double *trig, double center, int spacing, int ncenter,
                                             int edge_pad, double mask_r2, float scale, float *out,
                                             int64_t out_row_stride, int64_t out_center_stride, int flags,
                                             void *workspace, int64_t workspace_bytes, void *stream) {
  cudaStream_t st = atb::as_stream(stream);
  const int64_t need = atb_backproject_centers_workspace(nrow, ncol, ncenter);
  const bool always = flags & 64;
  flags &= ~64;
  int first = 0;
  // (arguments that atb_backproject_centers refuses go there)
  if (sino && trig && out && spacing >= 1 && spacing <= 56 && center >= 0.0 &&
      center + (double)(ncenter - 1) * (double)spacing < (double)ncol && need > 0 && workspace &&
      workspace_bytes >= need && reinterpret_cast<uintptr_t>(workspace) % 128 == 0) {
    unsigned *maxbits = static_cast<unsigned *>(workspace);
    uint4 *packed = reinterpret_cast<uint4 *>(static_cast<unsigned char *>(workspace) + kHeader);
    int rc;
    for (int n; (n = next_group(ATB_F32, nrow, ncol, ncenter - first)) > 0; first += n) {
      const int S = padded(n);
      const double c0 = center + (double)first * (double)spacing, c1 = c0 + (double)(n - 1) * (double)spacing;
      const double reach = (c0 < (double)(ncol - 1) - c1 ? c0 : (double)(ncol - 1) - c1) - 1e-2;
      // (nor where hardly a block lies within the reach)
      if (!always && !(centers_worth(n, nrow, ncol) && reach > 0.125 * (double)ncol)) break;
      CUtensorMap map;
      if (!packed_map(S, nrow, ncol, packed, &map)) break;
      if (first == 0) {
        if (cudaMemsetAsync(workspace, 0, kHeader, st) != cudaSuccess)
          return atb::fail(ATB_ECUDA, "atb_backproject_centers_stack: %s", cudaGetErrorString(cudaGetLastError()));
        absmax_kernel<float><<<dim3(nrow < 256 ? nrow : 256, 1), 256, 0, st>>>(sino, sino_row_stride, 0, nrow, ncol,
                                                                              maxbits);
        rc = atb::check_launch("atb_backproject_centers_stack (scan)");
        if (rc != ATB_OK) return rc;
      }
      // samples of the first centre's frame: later centres read further on
      pack_centers_kernel<<<dim3((ncol + 255) / 256, nrow, S / 8), 256, 0, st>>>(sino, sino_row_stride, ncol, n, S,
                                                                                spacing, first == 0, maxbits, packed);
      rc = atb::check_launch("atb_backproject_centers_stack (pack)");
      if (rc != ATB_OK) return rc;
      MmaArgs a;
      a.maxbits = maxbits + S;
      a.gate = maxbits;
      a.ngate = 1;
      a.trig = reinterpret_cast<const double2 *>(trig);
      a.nrow = nrow; a.ncol = ncol; a.nsl = n;
      a.center = c0; a.edge_pad = edge_pad ? 1 : 0; a.mask_r2 = mask_r2; a.scale = scale;
      a.out = out + (int64_t)first * out_center_stride; a.ors = out_row_stride; a.oss = out_center_stride;
      a.interior = reach > 0.0 ? reach : 0.0;
      a.inject = 0;
      rc = launch(a, S, map, st);
      if (rc != ATB_OK) return rc;
      // the blocks whose positions reach an edge of the detector for some
      // centre: each centre has its own edges there
      rc = atb::bp_gather_centers(sino, sino_row_stride, nrow, ncol, trig, c0, spacing, n, edge_pad, mask_r2, scale,
                                  a.out, out_row_stride, out_center_stride, flags, a.gate, a.ngate, a.interior, stream);
      if (rc != ATB_OK) return rc;
    }
    if (first == ncenter) return ATB_OK;
  }
  return atb::bp_gather_centers(sino, sino_row_stride, nrow, ncol, trig, center + (double)first * (double)spacing,
                                spacing, ncenter - first, edge_pad, mask_r2, scale,
                                out ? out + (int64_t)first * out_center_stride : out, out_row_stride,
                                out_center_stride, flags, nullptr, 0, -1.0, stream);
}
