// Block-sparse products at FP64 accuracy on the tensor cores: the stored
// couplings of the far field (double-float pairs) and the dense leaves (FP64),
// real and complex, times blocks of right-hand sides
// (H2DenseProduct.hpp:107-135, the dense and the low-rank leaves).
//
// GB300's FP64 pipe runs at 1/64 of its FP32 rate and the double-float
// product on the FP32 pipes costs 12 operations per multiply-add, so the
// product is done in exact integer arithmetic on the FP16 tensor cores
// (Ozaki's error-free splitting, fixed-point variant). Real couplings are
// stored as 8 digits of one byte, the bytes an FP64 entry or a double-float
// pair takes; complex ones (FP32 pairs of the far field, FP64 leaf blocks) are
// split into digits on the way:
//  - row i of a block row has an exponent e_i with |A_ij| <= 2^(e_i - 1) over
//    the whole block row, column c an exponent f_c with |x_jc| <= 2^(f_c - 1)
//    over all rows of the segment (one FMM level, or the near field);
//  - A_ij = 2^e_i sum_s a_s 2^(-7 (s + 1)) and x_jc likewise, 8 signed digits
//    of 7 bits each (|a_s| <= 64: exact in FP16);
//  - acc_d = sum_j sum_{s + t = d} a_s x_t for d = 0 .. 7 in FP32 tensor
//    memory. A product is at most 2^12 and a diagonal holds at most 8 per j,
//    so over 512 source rows acc_d is an exact integer below 2^24, whatever
//    the order and rounding of the tensor cores' accumulation;
//  - the epilogue adds the diagonals into one 64-bit fixed-point sum per
//    output entry and converts it once to FP64.
// The error is absolute in 2^(e_i + f_c), which is 4 to 16 times max |A_i| max
// |x_c|: per term below 2^-55.2 for the dropped digits (seven products of 2^12
// at 2^-70) and 2^-57 for the rounding of A and x (FP32 pairs: 2^-54.8); these
// are of either sign, about 2^-57.8 each, and grow with the root of the n
// terms. A plain FP64 sum errs by up to n 2^-53 of S = sum_j |A_ij| |x_jc|
// instead. The digits lose to it where S is small against 2^(e_i + f_c): an x of
// very different sizes, a kernel that decays within the row.
// Near field: the epilogue bounds S from below by the norms of x over 8 rows
// and the floors of A over 8 columns and 36 rows, and marks the columns of a block row
// where four times the digits' error could pass the plain sum's bound; the CTA
// sums those in FP64 at its end (plain_columns). Columns of normal or smooth
// values have S some 50 times above the line (B = 4 .. 64). Maxwell's blocks
// (B = 72) hold small entries among the others, and with one floor for all their
// rows half of the block rows had marks for normal x (sphere M = 3, mixed, 3
// columns: floors 0.9 to 1.2 times the line, S 200 times; 305 -> 350 us). Two groups
// of rows give 2.6 times and the old time back. At M = 4 (8 columns) the product
// still takes 2083 us, 1120 without the fallback; groups of 4 rows do not change
// that (2089), so its cause is another one, not found yet. All columns marked
// cost what the FP64 pipe did: sphere M = 5, P = 2, 32 columns 1.76 ms (1.49 on
// the pipe, 0.23 unmarked), torus M = 3, 16 complex ones 2.03 (2.59, 0.30).
// Far field: no row is marked. What an entry loses there is relative to the
// row's largest coupling times the column's largest x; that x reaches the entry
// too, through a block of this or another level or the near field, and with a
// coupling of similar size as long as kernel and surface measure vary little.
// So the loss stays below n 2^-48 of |A| |x|, the bound of the double-float sums
// that the digits replace; couplings that spread further within a row keep
// those sums (kFarSpread in bg_capi.cu).
//
// MMA (tcgen05.mma kind::f16, cta_group::1, M = 128, K = 16): the rows of the
// couplings are the M rows (rows beyond B produce accumulator lanes nobody
// reads), the digits of x the N columns, ordered (digit t, column c). For
// coupling digit s one MMA with N = (8 - s) NC covers x digits t = 0 .. 7 - s,
// whose accumulators d = s + t are consecutive in tensor memory too. Complex
// blocks add four such products, Re A Re x, Re A Im x, -Im A Im x (the
// instruction descriptor's negation of A) and Im A Re x, with the columns
// [Re | Im] of 16 right-hand sides.
//
// Roles of a CTA (persistent, one per SM, walking a list of block rows):
//  warps 0-7   epilogue: tensor-memory quadrant w % 4, half of the columns; warps
//              0 and 4 also mark the columns that are summed in FP64
//  warp 8      TMA (1-D bulk copies): the couplings of a stage into the raw
//              ring, the x digit panels into the stage
//  warp 9      MMA issue
//  warps 10-23 converters: expand a stage's digit bytes to FP16 (a byte permute
//              and a packed subtraction per two digits), or split its entries,
//              into the UMMA K-major layout
// A stage is one block's slice of up to 48 source rows (both parts of a
// complex block are stages of their own); two to four stages, a raw ring of up
// to eight slices, two accumulator buffers. Every wait is bounded; on timeout
// the kernel records an error code, the roles stop, and the tensor memory is
// freed.
#include <cuda_fp16.h>

#include <algorithm>
#include <cfloat>
#include <climits>
#include <cstdint>

#include "bg_kernels.cuh"
#include "bg_oz.cuh"
#include "bg_tcgen05.cuh"

namespace bg {

long bsr_oz_tile_stride(int B) { return ((long)B * B * 8 + 15) / 16 * 16; }

namespace {

using namespace tc;

constexpr int kEpiWarps = 8;
constexpr int kConvWarps = 14, kConvLanes = 32 * kConvWarps;
constexpr int kTmaWarp = kEpiWarps, kMmaWarp = kEpiWarps + 1, kConvWarp0 = kEpiWarps + 2;
constexpr int kOzThreads = 32 * (kEpiWarps + 2 + kConvWarps);  // 24 warps: 80 registers a thread
constexpr uint32_t kTmemCols = 512;  // two accumulator buffers of 8 diagonals x 32 columns
// stored couplings: digit bytes (real), FP32 pairs (complex, Re then Im at
// im_off), FP64 (complex, interleaved)
enum { kDigits = 0, kPairsC = 1, kF64C = 2 };
constexpr int kMaxStages = 4, kMaxRaws = 8;
constexpr uint32_t kOzSmem = 224 * 1024;
constexpr uint32_t kPlainSmem = kOzThreads * 8 * sizeof(double);  // partial sums of plain_columns

// the stage geometry of block size B (rows and columns of a block)
struct OzGeom {
  int B, rg;           // rows, 8-row groups stored
  int nks, kw, nch;    // 16-column K steps of a block, per full chunk, chunks
  int bps;             // blocks per stage (more than one only where a block is one K step)
  int nc;              // columns per digit in a panel: 32 (complex: 16 + 16) or 16
  uint32_t slice;      // bytes of one digit's coupling tile of a full chunk
  uint32_t x_bytes, stage, raw, raw_off;
  int stages, raws;
  uint32_t smem;
  uint32_t panel;      // bytes of a cluster's digit panels and norms
  int chunk_blocks;    // blocks whose diagonals stay exact
};

// bytes of a cluster's digits, ahead of the norms of its rows: [2 nks][nc] FP32,
// sum of |x_jc| 2^-f_c over 8 rows (complex: of the real and of the imaginary parts)
__host__ __device__ constexpr uint32_t oz_norms_at(int nc, int nks) { return 8u * nc * nks * 32u; }

// esz: bytes of a stored entry of a raw slice (FP64 complex: both parts, 16)
bool oz_geom(int B, bool cplx, int ncols, int esz, OzGeom* g) {
  // squares only (n_p^2, 4^m p^2): the last group of 8 columns is full or has 1 or 4
  if (B < 1 || B > 128 || (B % 8 != 0 && B % 8 != 1 && B % 8 != 4)) return false;
  g->B = B;
  g->rg = (B + 7) / 8;
  g->nks = (B + 15) / 16;
  g->nc = cplx || ncols > 16 ? 32 : 16;
  g->panel = oz_norms_at(g->nc, g->nks) + (uint32_t)g->nc * g->nks * 2u * sizeof(float);
  g->chunk_blocks = std::max(1, 512 / (B * (cplx ? 2 : 1)));
  // a stage holds up to three K steps, as many as the converters take in one
  // go: 2 kw groups of 8 columns for each of the B rows
  const int kmax = std::max(1, std::min(3, kConvLanes / (2 * B)));
  const int nch = (g->nks + kmax - 1) / kmax;
  g->kw = (g->nks + nch - 1) / nch;
  g->nch = (g->nks + g->kw - 1) / g->kw;
  // small blocks: three per stage, which is what a stage costs beside its MMAs
  // (M = 5, P = 1, B = 16 near field, 32 columns: 134 -> 96 us)
  g->bps = g->nks == 1 ? 3 : 1;
  g->chunk_blocks = std::max(g->bps, g->chunk_blocks / g->bps * g->bps);
  const int steps = g->kw * g->bps;  // K steps of a full stage
  g->slice = (uint32_t)g->rg * steps * 256u;
  g->x_bytes = 8u * g->nc * steps * 32u;
  g->stage = 8u * g->slice + g->x_bytes;
  g->raw = (uint32_t)(g->bps > 1 ? g->bps * (B * B * esz + 15) : std::min(B, 16 * g->kw) * B * esz + 15);
  g->raw = (g->raw + 127u) / 128u * 128u;
  // the MMA reads 16 row groups of every digit tile: the last tiles' reads
  // run into what follows them, which has to stay inside the allocation
  const uint32_t over = (uint32_t)(16 - g->rg) * steps * 256u;
  auto need = [&]() {
    const uint32_t after = g->x_bytes + g->raws * g->raw;
    return std::max(kPlainSmem, g->stages * g->stage + g->raws * g->raw + (over > after ? over - after : 0u));
  };
  for (g->stages = kMaxStages; g->stages >= 2; --g->stages)
    for (g->raws = kMaxRaws; g->raws >= 3; --g->raws)
      if (need() <= kOzSmem) {
        g->raw_off = g->stages * g->stage;
        g->smem = need();
        return true;
      }
  return false;
}

// Fixed point of the row sums: 2^-unit of the leading digit product. A sum
// over n source entries is below 2^(12 + log2 n) (1 + 2^-6) of it, which with
// unit bits below the point has to fit 63 bits.
constexpr int kOzMinUnit = 30;
// pairs: rows whose largest entry is below 2^-111 are split as if it were
// that, which keeps the scale 2^(14 - e) a normal FP32 number
constexpr int kMinPairExp = -110;
int oz_unit(int B, bool cplx, int max_row_blocks) {
  const long n = (long)std::max(1, max_row_blocks) * B * (cplx ? 2 : 1);
  int lg = 0;
  while ((1l << lg) < n) ++lg;
  return std::min(48, 49 - lg);
}

// ---- digits of the couplings ----
// Four 14-bit groups, each two biased 7-bit digits (digit + 64), most
// significant first; bits above the group are garbage except in the first.
struct Groups {
  uint32_t u[4];
};

// v = hi + lo (FP32 pair), scale = 2^(14 - e) with |v| <= 2^(e - 1): groups
// by round-to-integer (adding 1.5 2^23, plus the digits' bias) and exact
// remainders; what is left of hi and lo below the second group is summed in
// FP32, which keeps the pair's bits to 2^-53 of the row's largest entry. The
// bits of a rounded sum are those of 1.5 2^23 + 8256 + n; what a group has
// above its 14 bits is carried into the one before it.
__device__ __forceinline__ Groups split_pair(float hi, float lo, float scale) {
  constexpr float kM = 12582912.0f + 8256.0f;
  constexpr int kBits = 0x4B400000 >> 14;
  const float v = hi * scale, m1 = v + kM, r1 = v - (m1 - kM);
  const float m2 = fmaf(r1, 16384.0f, kM), r2 = fmaf(r1, 16384.0f, kM - m2);
  const float t = fmaf(lo * scale, 16384.0f, r2);
  const float m3 = fmaf(t, 16384.0f, kM), r3 = fmaf(t, 16384.0f, kM - m3);
  const float m4 = fmaf(r3, 16384.0f, kM);
  Groups g;
  int u = __float_as_int(m4);
  g.u[3] = (uint32_t)u;
  u = __float_as_int(m3) + (u >> 14) - kBits;
  g.u[2] = (uint32_t)u;
  u = __float_as_int(m2) + (u >> 14) - kBits;
  g.u[1] = (uint32_t)u;
  g.u[0] = (uint32_t)(__float_as_int(m1) + (u >> 14) - kBits);
  return g;
}

// FP64 v, bmax = e + 1021 the largest biased exponent of the row:
// round(|v| 2^(56 - e)) in 64-bit integers, with the sign, plus 64 in every digit
__device__ __forceinline__ Groups split_double(double v, int bmax) {
  const uint32_t h = (uint32_t)__double2hiint(v), l = (uint32_t)__double2loint(v);
  const int be = (int)((h >> 20) & 0x7FF);
  const unsigned long long mant =
      ((unsigned long long)((h & 0xFFFFFu) | (be ? 0x100000u : 0u)) << 32 | l) << 3;
  const int q = max(0, min(bmax - max(be, 1), 63));
  long long V = (long long)(((mant >> q) + 1) >> 1);
  V = (int)h < 0 ? -V : V;
  const unsigned long long U = (unsigned long long)V + 0x0081020408102040ull;
  return {{(uint32_t)(U >> 42), (uint32_t)(U >> 28), (uint32_t)(U >> 14), (uint32_t)U}};
}

// the FP16 digits 2 g, 2 g + 1 of two values as packed pairs
__device__ __forceinline__ void digit_pair(uint32_t ua, uint32_t ub, bool top, uint32_t* first, uint32_t* second) {
  const uint32_t w = __byte_perm(ua, ub, 0x5410);
  const uint32_t hi = ((w >> 7) & (top ? 0x00FF00FFu : 0x007F007Fu)) | 0x64006400u;  // 1024 + digit + 64
  const uint32_t lo = (w & 0x007F007Fu) | 0x64006400u;
  const __half2 off = __float2half2_rn(1088.0f);
  const __half2 a = __hsub2(*reinterpret_cast<const __half2*>(&hi), off);
  const __half2 b = __hsub2(*reinterpret_cast<const __half2*>(&lo), off);
  *first = *reinterpret_cast<const uint32_t*>(&a);
  *second = *reinterpret_cast<const uint32_t*>(&b);
}

// bytes ahead of group jg (8 columns) of a block's digit bytes: a full group
// is [4][B][16 bytes], quad q of a row holding digits 2 q and 2 q + 1 of the 8
// columns; a last group of 4 columns [2][B][16], digits 4 q .. 4 q + 3 of 4
// columns; of 1 column [B][8]. A byte is a digit + 64.
__device__ __forceinline__ uint32_t group_bytes(int B, int jg) { return (uint32_t)(jg * 64 * B); }

// the bytes of two digits of 8 columns (bytes b0: columns 0-3, b1: 4-7) as FP16
__device__ __forceinline__ uint4 expand_digit(uint32_t b0, uint32_t b1) {
  const __half2 off = __float2half2_rn(1088.0f);
  uint32_t w[4] = {__byte_perm(b0, 0x64646464u, 0x4140), __byte_perm(b0, 0x64646464u, 0x4342),
                   __byte_perm(b1, 0x64646464u, 0x4140), __byte_perm(b1, 0x64646464u, 0x4342)};
#pragma unroll
  for (int q = 0; q < 4; ++q) {  // 1024 + digit + 64, minus 1088
    const __half2 h = __hsub2(*reinterpret_cast<const __half2*>(&w[q]), off);
    w[q] = *reinterpret_cast<const uint32_t*>(&h);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// entry (row i, column j) of a block, from its digit bytes and row exponent
__device__ double digit_value(const unsigned char* t, int B, int i, int j, int e) {
  const int jg = j >> 3, c = j & 7, nv = min(8, B - 8 * jg);
  const unsigned char* p = t + group_bytes(B, jg);
  long long V = 0;
  for (int s = 0; s < 8; ++s) {
    const int o = nv == 8 ? ((s >> 1) * B + i) * 16 + (s & 1) * 8 + c : nv == 4 ? ((s >> 2) * B + i) * 16 + (s & 3) * 4 + c : i * 8 + s;
    V = V * 128 + ((int)p[o] - 64);
  }
  return oz_to_double(V, e - 56);
}

// position in a ring of n barriers: consumers wait for parity `phase` of the
// full barrier, producers for phase ^ 1 of the empty one (which a fresh
// barrier passes). No division: these sit on the critical path of every stage.
struct Ring {
  int slot;
  uint32_t phase;
  __device__ __forceinline__ void next(int n) {
    if (++slot == n) {
      slot = 0;
      phase ^= 1u;
    }
  }
};

// a walk over the stages of a CTA: items, blocks, K chunks, parts
struct Cursor {
  int item, seg, row, pass;
  int k, ke, chunk, part;
  bool done;
};

// WARP: the whole warp walks together and what it loads is made warp-uniform
template <bool WARP>
__device__ __forceinline__ int uniform(int v) {
  return WARP ? __shfl_sync(0xffffffffu, v, 0) : v;
}
template <bool WARP = false>
__device__ __forceinline__ bool open_item(const OzArgs& a, Cursor& c) {
  for (; c.item < a.nitems; c.item += gridDim.x) {
    const int w = c.item % a.nwork;
    c.pass = c.item / a.nwork;
    if (a.work) {
      const int2 it = __ldg(a.work + w);
      c.seg = uniform<WARP>(it.x);
      c.row = uniform<WARP>(it.y);
    } else {
      c.seg = 0;
      c.row = w;
    }
    c.k = uniform<WARP>(__ldg(a.seg[c.seg].row_ptr + c.row));
    c.ke = uniform<WARP>(__ldg(a.seg[c.seg].row_ptr + c.row + 1));
    c.chunk = c.part = 0;
    if (c.k < c.ke) return true;
  }
  c.done = true;
  return false;
}
template <int PARTS, bool WARP = false>
__device__ __forceinline__ void next_stage(const OzArgs& a, Cursor& c) {
  if (++c.part < PARTS) return;
  c.part = 0;
  if (++c.chunk < a.nch) return;
  c.chunk = 0;
  c.k += a.bps;
  if (c.k < c.ke) return;
  c.item += gridDim.x;
  open_item<WARP>(a, c);
}

// blocks of the cursor's stage, and its K steps
__device__ __forceinline__ int stage_blocks(const OzArgs& a, const Cursor& c) { return min(a.bps, c.ke - c.k); }
__device__ __forceinline__ int stage_steps(const OzArgs& a, const Cursor& c) {
  return a.bps > 1 ? stage_blocks(a, c) : min(a.kw, a.nks - c.chunk * a.kw);
}

__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}\n" : "=r"(p));
  return p != 0;
}

__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n.reg .pred p;\nmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(done)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return done != 0;
}

// bounded wait, the common case (already complete) without reading the clock
__device__ __forceinline__ bool mbar_wait_fast(uint64_t* bar, uint32_t parity) {
  return mbar_test(bar, parity) || mbar_wait(bar, parity);
}

// a wait that leaves the issue slots to the other warps
__device__ __forceinline__ bool mbar_wait_idle(uint64_t* bar, uint32_t parity) {
  const uint32_t a = smem_u32(bar);
  const long long t0 = clock64();
  while (true) {
    uint32_t done;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    if (done) return true;
    if (clock64() - t0 > kWaitCycles) return false;
    __nanosleep(100);
  }
}

// tcgen05.mma kind::f16 with the descriptors' low words (addresses) and high
// words (strides) apart
__device__ __forceinline__ void mma_f16_lo(uint32_t d, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi,
                                           uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p;\n.reg .b64 a, b;\nmov.b64 a, {%1, %2};\nmov.b64 b, {%3, %4};\nsetp.ne.b32 p, %6, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %5, p;\n}\n" ::"r"(d),
      "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate));
}

// operands of a stage's MMAs: low descriptor words of coupling digit 0 and of
// the x panel, steps to the next coupling digit, the next K step of the panel
// and its imaginary half, high words
struct StageOps {
  uint32_t a_lo, a_hi, x_lo, x_hi, a_digit, x_step, x_half;
};

// The MMAs of a stage with KC K steps, fully unrolled: with N = 16 .. 256 an
// MMA takes 45 .. 128 cycles (measured), so issuing it may cost a few
// instructions only
template <bool C, int NC, int KC>
__device__ __forceinline__ void stage_mmas(uint32_t dd, StageOps o, int part, bool fresh) {
#pragma unroll
  for (int s = 0; s < 8; ++s, o.a_lo += o.a_digit) {
    if constexpr (!C) {
#pragma unroll
      for (int ks = 0; ks < KC; ++ks)
        mma_f16_lo(dd + (uint32_t)(s * NC), o.a_lo + 16 * ks, o.a_hi, o.x_lo + ks * o.x_step, o.x_hi,
                   idesc_f16(128, (8 - s) * NC), (s == 0 && ks == 0 && fresh) ? 0u : 1u);
    } else {
      constexpr uint32_t neg = 1u << 13;
      // part 0: Re += Re A Re x, Im += Re A Im x; part 1: Re -= Im A Im x (A negated), Im += Im A Re x
      const uint32_t id = idesc_f16(128, (8 - s) * 16), id_re = part ? id | neg : id;
      const uint32_t x_re = part ? o.x_lo + o.x_half : o.x_lo, x_im = part ? o.x_lo : o.x_lo + o.x_half;
#pragma unroll
      for (int ks = 0; ks < KC; ++ks)
        mma_f16_lo(dd + (uint32_t)(s * 16), o.a_lo + 16 * ks, o.a_hi, x_re + ks * o.x_step, o.x_hi, id_re,
                   (s == 0 && ks == 0 && fresh) ? 0u : 1u);
#pragma unroll
      for (int ks = 0; ks < KC; ++ks)
        mma_f16_lo(dd + (uint32_t)(s * 16) + 128u, o.a_lo + 16 * ks, o.a_hi, x_im + ks * o.x_step, o.x_hi, id,
                   (s == 0 && ks == 0 && fresh) ? 0u : 1u);
    }
  }
}
template <bool C, int NC>
__device__ __forceinline__ void stage_mmas(int kc, uint32_t dd, const StageOps& o, int part, bool fresh) {
  if (kc == 3) stage_mmas<C, NC, 3>(dd, o, part, fresh);
  else if (kc == 2) stage_mmas<C, NC, 2>(dd, o, part, fresh);
  else stage_mmas<C, NC, 1>(dd, o, part, fresh);
}

// 32 lanes x 2 consecutive FP32 columns of tensor memory, without the wait
__device__ __forceinline__ void tmem_ld2(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0,%1}, [%2];\n" : "=r"(r[0]), "=r"(r[1]) : "r"(taddr));
}

// |v| 2^-e in FP32, rounded down, for |v| < 2^(e + 128); what is below the range
// of FP32 counts as its smallest number
__device__ __forceinline__ float scaled_magnitude(double v, int e) {
  const uint32_t h = (uint32_t)__double2hiint(v) & 0x7FFFFFFFu, l = (uint32_t)__double2loint(v);
  const int ex = (int)(h >> 20) - e - 896;
  if ((h | l) == 0u) return 0.0f;
  return ex <= 0 || h < 0x100000u ? FLT_MIN : __uint_as_float((uint32_t)ex << 23 | (h & 0xFFFFFu) << 3 | l >> 29);
}

// The columns (bits 0 .. 15) of half h of a pass (complex: of the pass) that have
// to be summed in FP64 in block row `row`: those with Inf or NaN, and those
// where the bound of S = sum |A| |x| (in units of 2^(e + f)) is below the line
// that the head of this file derives; columns whose x is zero wherever the row
// has blocks are exact anyway. Lanes hold 16 columns and every second block each.
template <int SRC>
__device__ __noinline__ uint32_t careful_columns(const OzArgs& a, const OzSeg& g, int row, int seg, int pass, int h) {
  constexpr bool C = SRC != kDigits;
  const int lane = threadIdx.x & 31, per = C ? 16 : a.nc, first = C ? 0 : 16 * h;
  const int ncol = min(16, min(per, a.ncols - pass * per) - first), c = first + (lane & 15);
  const int kb = g.row_ptr[row], ke = g.row_ptr[row + 1], ng = (a.B + 7) / 8;
  bool care = a.fmax[(pass * a.nseg + seg) * 32 + c] == 2047;
  if (a.care > 0.0f && kb < ke) {
    const int nh = oz_row_groups(a.B);
    float least = FLT_MAX, most = 0.0f;
    for (int r = 0; r < nh; ++r) {
      float sum = 0.0f;
      for (int k = kb + (lane >> 4); k < ke; k += 2) {
        const float* nx = reinterpret_cast<const float*>(g.panels + (size_t)pass * a.pass_panels +
                                                         (size_t)g.col[k] * a.panel + oz_norms_at(a.nc, a.nks)) + c;
        const float* fl = g.floors + ((long)k * nh + r) * ng;
#pragma unroll 4
        for (int q = 0; q < ng; ++q) {
          float v = nx[q * a.nc];
          if (C) v = 0.7071f * (v + nx[q * a.nc + 16]);  // at most the sum of the moduli
          sum = fmaf(fl[q], v, sum);
          most = fmaxf(most, v);
        }
      }
      sum += __shfl_xor_sync(0xffffffffu, sum, 16);
      least = sum < least ? sum : (sum == sum ? least : sum);
    }
    most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, 16));
    const float n = (float)(ke - kb) * (float)(a.B * (C ? 2 : 1));
    const float roundings = (float)((ke - kb + a.chunk_blocks - 1) / a.chunk_blocks);  // of the fixed-point sum
    const float line = a.care * (0.15f * rsqrtf(n) + roundings * exp2f((float)(39 - a.unit)) / n);
    care |= !(least >= line) && most > 0.0f;
  }
  return __ballot_sync(0xffffffffu, care) & ((1u << max(ncol, 0)) - 1u);
}

template <int SRC>
__device__ __forceinline__ double stored_entry(const OzArgs& a, const OzSeg& g, long k, int part, int i, int j, int e) {
  const unsigned char* t = g.tiles + k * g.tstride;
  const long q = (long)j * a.B + i;
  if constexpr (SRC == kDigits) return g.exact ? g.exact[k * g.exact_stride + q] : digit_value(t, a.B, i, j, e);
  else if constexpr (SRC == kF64C) return reinterpret_cast<const double*>(t)[2 * q + part];
  else {
    const float2 v = reinterpret_cast<const float2*>(t + (part ? g.im_off : 0))[q];
    return (double)v.x + (double)v.y;
  }
}
// Plain FP64 sums of block row `row` in the columns of mask (from col0 on), by a
// whole CTA: a thread owns a row, four columns, which share the entries they
// read, and every nsp-th block; the shares are added in order. Bound by the FP64
// pipe, like the products that the digits replace.
template <int SRC>
__device__ void plain_columns(const OzArgs& a, const OzSeg& g, int row, int col0, uint32_t mask, double* sums) {
  constexpr bool C = SRC != kDigits;
  constexpr int W = C ? 2 : 1;
  const int kb = g.row_ptr[row], ke = g.row_ptr[row + 1], left = __popc(mask), nq = (left + 3) / 4;
  for (int q0 = 0; q0 < nq; q0 += kOzThreads / a.B) {
    const int nqs = min(nq - q0, kOzThreads / a.B), units = a.B * nqs, nsp = kOzThreads / units;
    const int sp = threadIdx.x / units, unit = threadIdx.x - sp * units, i = unit % a.B, quad = q0 + unit / a.B;
    int col[4];
    double acc[4 * W];
#pragma unroll
    for (int u = 0; u < 4; ++u) col[u] = col0 + __fns(mask, 0, min(4 * quad + u, left - 1) + 1);
#pragma unroll
    for (int u = 0; u < 4 * W; ++u) acc[u] = 0.0;
    if (sp < nsp) {
      const int e = SRC == kDigits ? g.rexp[(long)row * a.B + i] : 0;
      for (int k = kb + sp; k < ke; k += nsp) {
        const double* x = g.x + (long)g.col[k] * a.B * a.ldx * W;
#pragma unroll 2
        for (int j = 0; j < a.B; ++j, x += (long)a.ldx * W) {
          const double ar = stored_entry<SRC>(a, g, k, 0, i, j, e);
          if constexpr (C) {
            const double ai = stored_entry<SRC>(a, g, k, 1, i, j, e);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const double2 v = reinterpret_cast<const double2*>(x)[col[u]];
              acc[2 * u] = fma(ar, v.x, fma(-ai, v.y, acc[2 * u]));
              acc[2 * u + 1] = fma(ar, v.y, fma(ai, v.x, acc[2 * u + 1]));
            }
          } else {
#pragma unroll
            for (int u = 0; u < 4; ++u) acc[u] = fma(ar, x[col[u]], acc[u]);
          }
        }
      }
#pragma unroll
      for (int u = 0; u < 4 * W; ++u) sums[(sp * 4 * W + u) * units + unit] = acc[u];
    }
    __syncthreads();
    if (sp == 0) {
      double* y = g.y + ((long)row * a.B + i) * a.ldx * W;
#pragma unroll
      for (int u = 0; u < 4 * W; ++u) {
        double v = 0.0;
        for (int t = 0; t < nsp; ++t) v += sums[(t * 4 * W + u) * units + unit];
        y[W * col[u / W] + u % W] = v;  // fewer than four columns: the last one again
      }
    }
    __syncthreads();
  }
}

}  // namespace

// Row exponents of FP64 blocks (column-major, complex interleaved): e[r B + i]
// with |A_ij| <= 2^(e - 1) over block row r. A thread owns one row of the
// blocks and a share of their columns. spread, if given: the most that the
// exponents of a row's entries (complex: of the larger parts) differ, with its
// own value; at least 2046 in rows of complex couplings that FP32 pairs cannot
// hold, and 2047 in rows with Inf or NaN.
template <bool C>
__global__ void k_oz_rows(const int* __restrict__ row_ptr, const double* __restrict__ blocks, long bstride, int B,
                          int* __restrict__ e, int* spread) {
  __shared__ int top[128], low[128];
  const int r = blockIdx.x, i = threadIdx.x % B, jg = threadIdx.x / B, nj = blockDim.x / B;
  for (int t = threadIdx.x; t < B; t += blockDim.x) {
    top[t] = 0;
    low[t] = 2047;
  }
  __syncthreads();
  int m = 0, least = 2047;
  const int kb = row_ptr[r], ke = row_ptr[r + 1];
  for (int k = kb; k < ke; ++k)
    for (int j = jg; j < B; j += nj) {
      const long o = k * bstride + (long)j * B + i;
      if constexpr (C) {
        const double2 v = reinterpret_cast<const double2*>(blocks)[o];
        const int be = max((__double2hiint(v.x) >> 20) & 0x7FF, (__double2hiint(v.y) >> 20) & 0x7FF);
        m = max(m, be);
        least = min(least, be);
      } else {
        const int be = (__double2hiint(blocks[o]) >> 20) & 0x7FF;
        m = max(m, be);
        least = min(least, be);
      }
    }
  atomicMax(&top[i], m);
  atomicMin(&low[i], least);
  __syncthreads();
  for (int t = threadIdx.x; t < B; t += blockDim.x) {
    e[(long)r * B + t] = top[t] - 1021;
    const int most = top[t] == 2047 ? 2047 : C && top[t] - 1023 > 126 ? 2046 : top[t] - low[t];
    if (spread && kb < ke) atomicMax(spread, most);
  }
}

// floors[k][r][q]: lower bounds of |A_ij| 2^-e_i (complex: of the larger part)
// over columns 8 q .. 8 q + 7 and rows 36 r .. 36 r + 35 of block k. A warp per
// group of columns and rows.
template <bool C>
__global__ void k_oz_floors(const int* __restrict__ row_ptr, const double* __restrict__ blocks, long bstride, int B,
                            const int* __restrict__ e, float* __restrict__ floors) {
  const int r = blockIdx.x, ng = (B + 7) / 8, per = ng * oz_row_groups(B), lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int kb = row_ptr[r], n = (row_ptr[r + 1] - kb) * per;
  for (int u = threadIdx.x >> 5; u < n; u += nw) {
    const long k = kb + u / per;
    const int j0 = 8 * (u % ng), nv = min(8, B - j0), i0 = kOzGroupRows * (u % per / ng);
    float m = FLT_MAX;
    for (int i = i0 + lane; i < min(B, i0 + kOzGroupRows); i += 32) {
      const int ei = e[(long)r * B + i];
      for (int c = 0; c < nv; ++c) {
        const long o = k * bstride + (long)(j0 + c) * B + i;
        if constexpr (C) {
          const double2 v = reinterpret_cast<const double2*>(blocks)[o];
          m = fminf(m, fmaxf(scaled_magnitude(v.x, ei), scaled_magnitude(v.y, ei)));
        } else {
          m = fminf(m, scaled_magnitude(blocks[o], ei));
        }
      }
    }
    const int bits = __reduce_min_sync(0xffffffffu, __float_as_int(m));  // not negative: ordered as integers
    if (lane == 0) floors[kb * (long)per + u] = __int_as_float(bits);
  }
}

// Digit bytes of real FP64 blocks (layout: group_bytes). A thread takes 8
// columns of one row.
__global__ void k_oz_tiles(const int* __restrict__ row_ptr, const double* __restrict__ blocks, long bstride, int B,
                           const int* __restrict__ e, unsigned char* __restrict__ tiles, long tstride) {
  const int r = blockIdx.x, ng = (B + 7) / 8;
  const int kb = row_ptr[r], ke = row_ptr[r + 1];
  for (long u = threadIdx.x + (long)blockIdx.y * blockDim.x; u < (long)(ke - kb) * ng * B;
       u += (long)blockDim.x * gridDim.y) {
    const int i = (int)(u % B);
    const long q = u / B;
    const int jg = (int)(q % ng);
    const long k = kb + q / ng;
    const int nv = min(8, B - 8 * jg), bmax = e[(long)r * B + i] + 1021;
    uint32_t w[8][2];  // digit s: bytes of columns 0-3, 4-7
#pragma unroll
    for (int s = 0; s < 8; ++s) w[s][0] = w[s][1] = 0;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const double v = c < nv ? blocks[k * bstride + (long)(8 * jg + c) * B + i] : 0.0;
      const Groups g = split_double(v, bmax);
#pragma unroll
      for (int d = 0; d < 4; ++d) {
        w[2 * d][c >> 2] |= ((g.u[d] >> 7) & (d ? 0x7Fu : 0xFFu)) << (8 * (c & 3));
        w[2 * d + 1][c >> 2] |= (g.u[d] & 0x7Fu) << (8 * (c & 3));
      }
    }
    unsigned char* t = tiles + k * tstride + group_bytes(B, jg);
    if (nv == 8) {
#pragma unroll
      for (int h = 0; h < 4; ++h)
        *reinterpret_cast<uint4*>(t + (h * B + i) * 16) =
            make_uint4(w[2 * h][0], w[2 * h][1], w[2 * h + 1][0], w[2 * h + 1][1]);
    } else if (nv == 4) {
#pragma unroll
      for (int h = 0; h < 2; ++h)
        *reinterpret_cast<uint4*>(t + (h * B + i) * 16) =
            make_uint4(w[4 * h][0], w[4 * h + 1][0], w[4 * h + 2][0], w[4 * h + 3][0]);
    } else {
      uint32_t lo = 0, hi = 0;
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        lo |= (w[s][0] & 0xFFu) << (8 * s);
        hi |= (w[4 + s][0] & 0xFFu) << (8 * s);
      }
      *reinterpret_cast<uint2*>(t + i * 8) = make_uint2(lo, hi);
    }
  }
}

// One right-hand side, y = A x from the digit bytes in double-float arithmetic
// on the FP32 pipes (for callers without scratch for the digit panels; x
// arrives as FP32 (hi, lo) pairs). An entry's digits
// are summed in three exact FP32 integers (21, 21 and 14 bits) and folded into
// a pair of the row's units 2^(e - 56), products and sums as in k_bsr_df
// (about 1e-14). A CTA per block row, lanes over its rows and warps over the
// blocks' groups of 8 columns.
__global__ void __launch_bounds__(256) k_digits_one(OzSeg g, const float2* __restrict__ x, int B) {
  extern __shared__ double sums[];  // [warps][B]
  const int r = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int kb = g.row_ptr[r], ke = g.row_ptr[r + 1], ng = (B + 7) / 8;
  for (int i = lane; i < B; i += 32) {
    float sum = 0.0f, comp = 0.0f;
    int k = kb + warp / ng, jg = warp % ng;
    for (; k < ke; jg += nw, k += jg / ng, jg %= ng) {
      const int nv = min(8, B - 8 * jg);
      const float2* xp = x + (long)g.col[k] * B + 8 * jg;
      const unsigned char* t = g.tiles + (long)k * g.tstride + group_bytes(B, jg);
      uint32_t w[8][2];
      if (nv == 8) {
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          const uint4 v = __ldg(reinterpret_cast<const uint4*>(t + (h * B + i) * 16));
          w[2 * h][0] = v.x; w[2 * h][1] = v.y; w[2 * h + 1][0] = v.z; w[2 * h + 1][1] = v.w;
        }
      } else if (nv == 4) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint4 v = __ldg(reinterpret_cast<const uint4*>(t + (h * B + i) * 16));
          w[4 * h][0] = v.x; w[4 * h + 1][0] = v.y; w[4 * h + 2][0] = v.z; w[4 * h + 3][0] = v.w;
        }
      } else {
        const uint2 v = __ldg(reinterpret_cast<const uint2*>(t + i * 8));
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          w[q][0] = (v.x >> (8 * q)) & 0xFFu;
          w[4 + q][0] = (v.y >> (8 * q)) & 0xFFu;
        }
      }
#pragma unroll
      for (int c = 0; c < 8; ++c)
        if (c < nv) {
          int d[8];
#pragma unroll
          for (int q = 0; q < 8; ++q) d[q] = (int)((w[q][c >> 2] >> (8 * (c & 3))) & 0xFFu) - 64;
          const float a = (float)((d[0] * 128 + d[1]) * 128 + d[2]), b = (float)((d[3] * 128 + d[4]) * 128 + d[5]);
          const float hi = fmaf(a, 2097152.0f, b), rest = fmaf(a, 2097152.0f, -hi) + b;  // exact
          const float lo = fmaf((float)(d[6] * 128 + d[7]), 1.0f / 16384.0f, rest);
          const float2 v = xp[c];
          const float p = hi * v.x;
          float err = fmaf(hi, v.x, -p);
          err = fmaf(hi, v.y, err);
          err = fmaf(lo, v.x, err);
          const float ts = sum + p, z = ts - sum;
          comp += ((sum - (ts - z)) + (p - z)) + err;
          sum = ts;
        }
    }
    sums[warp * B + i] = (double)sum + (double)comp;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < B; i += blockDim.x) {
    double v = 0.0;
    for (int w = 0; w < nw; ++w) v += sums[w * B + i];
    // units of 2^(e - 42): the first six digits are integers
    g.y[(long)r * B + i] = ldexp(v, g.rexp[(long)r * B + i] - 42);
  }
}

// red[c] = the largest biased exponent of column c of a pass over this CTA's
// share (part of nparts) of the rows of segment g, of both parts if complex
template <bool C>
__device__ __forceinline__ void column_maxima(const OzArgs& a, const OzSeg& g, int pass, int part, int nparts, int* red) {
  const int per = C ? 16 : a.nc, col0 = a.c0 + pass * per, ncol = min(per, a.c0 + a.ncols - col0);
  const int c = threadIdx.x % ncol, rows = blockDim.x / ncol;  // rows of x a round
  if (threadIdx.x < 32) red[threadIdx.x] = 0;
  __syncthreads();
  int m = 0;
  if ((int)threadIdx.x < rows * ncol)
#pragma unroll 4
    for (long r = (long)part * rows + threadIdx.x / ncol; r < (long)g.ncl * a.B; r += (long)nparts * rows) {
      const long o = r * a.ldx + col0 + c;
      if constexpr (C) {
        const double2 v = reinterpret_cast<const double2*>(g.x)[o];
        m = max(m, max((__double2hiint(v.x) >> 20) & 0x7FF, (__double2hiint(v.y) >> 20) & 0x7FF));
      } else {
        m = max(m, (__double2hiint(g.x[o]) >> 20) & 0x7FF);
      }
    }
  if (m) atomicMax(&red[c], m);
  __syncthreads();
}

// Column exponents of every segment and pass: fmax[(pass nseg + seg) 32 + c]
// = the largest biased exponent of column c (complex: of both parts, for
// columns c and c + 16). Zeroed before.
template <bool C>
__global__ void k_oz_cols(OzArgs a) {
  __shared__ int red[32];
  const OzSeg& g = a.seg[blockIdx.y];
  const int pass = blockIdx.z, per = C ? 16 : a.nc;
  column_maxima<C>(a, g, pass, blockIdx.x, gridDim.x, red);
  if (threadIdx.x < per && red[threadIdx.x]) {
    int* f = a.fmax + (pass * a.nseg + blockIdx.y) * 32;
    atomicMax(f + threadIdx.x, red[threadIdx.x]);
    if (C) atomicMax(f + 16 + threadIdx.x, red[threadIdx.x]);
  }
}

// Digit panels of x: cluster J of segment s at panels + pass a.pass_panels +
// J panel; in it K chunk by K chunk, rows (t, c) (complex: [Re (t, c)] [Im (t,
// c)]) K-major. A thread takes 8 consecutive source rows of one column;
// columns and rows beyond the data get zeros. It also writes their norm where
// care is to be taken. OWN: few rows, and every CTA finds the column exponents
// itself instead of a launch (and a memset) before.
template <bool C, bool OWN>
__global__ void k_oz_panels(OzArgs a) {
  __shared__ int red[32];
  const OzSeg& g = a.seg[blockIdx.y];
  const int pass = blockIdx.z, ng = 2 * a.nks, per = C ? 16 : a.nc, col0 = a.c0 + pass * per;
  int* fmax = a.fmax + (pass * a.nseg + blockIdx.y) * 32;
  if (OWN) {
    column_maxima<C>(a, g, pass, 0, 1, red);
    if (blockIdx.x == 0 && threadIdx.x < 32) fmax[threadIdx.x] = red[threadIdx.x % per];
  }
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long)g.ncl * ng * a.nc) return;
  const int c = (int)(t % a.nc);
  const long q = t / a.nc;
  const int kg = (int)(q % ng);
  const long J = q / ng;
  const int half = C ? c >> 4 : 0, cc = C ? c & 15 : c;
  const bool live = col0 + cc < a.c0 + a.ncols;
  const int f = (OWN ? red[cc] : fmax[cc]) - 1021;
  float norm = 0.0f;
  uint32_t w[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int j = kg * 8 + i;
    double v = 0.0;
    if (live && j < a.B) {
      const long o = (J * a.B + j) * a.ldx + col0 + cc;
      v = C ? g.x[2 * o + half] : g.x[o];
    }
    if (a.care > 0.0f) norm += scaled_magnitude(v, f);
    int d[8];
    oz_digits(v, f, d);
#pragma unroll
    for (int s = 0; s < 8; ++s) {
      const uint32_t h = (uint32_t)__half_as_ushort(__int2half_rn(d[s]));
      if (i & 1) w[s][i >> 1] |= h << 16;
      else w[s][i >> 1] = h;
    }
  }
  const int chunk = kg / (2 * a.kw), kc = min(a.kw, a.nks - chunk * a.kw);
  const uint32_t sbo = (uint32_t)kc * 256u;
  unsigned char* base = g.panels + (size_t)pass * a.pass_panels + (size_t)J * a.panel;
  if (a.care > 0.0f) reinterpret_cast<float*>(base + oz_norms_at(a.nc, a.nks))[kg * a.nc + c] = norm;
  base += (size_t)chunk * a.kw * a.nc * 8u * 32u + (uint32_t)(kg - chunk * 2 * a.kw) * 128u;
#pragma unroll
  for (int s = 0; s < 8; ++s) {
    const int r = C ? half * 128 + s * 16 + cc : s * a.nc + c;
    *reinterpret_cast<uint4*>(base + (uint32_t)(r >> 3) * sbo + (uint32_t)(r & 7) * 16u) =
        make_uint4(w[s][0], w[s][1], w[s][2], w[s][3]);
  }
}

// What bounds it: shared memory. An MMA reads its 4 KB of couplings and up to 8
// KB of x digits in 45 .. 128 cycles, on top of which come the converters'
// loads and stores and the copies (far field of sphere M = 4, 32 columns: the
// tensor cores' reads take 42 % of the cycles and the converters' accesses 39 %,
// with an SM active in 80 %; tensor pipe 44 %, DRAM 27 %); a stage of 16 MMAs (B = 81) takes about 1900 cycles,
// 1240 of them MMAs back to back. Large stages amortise what a stage costs
// beside its MMAs (barriers, commit: about 500 cycles of the issuing warp).
// Storing digits for real couplings saves the splitting (300 against 110
// instructions per 8 couplings): 1.80 -> 1.53 ms below.
// Measured (GB300), with the panels of x, against what it replaces: sphere M =
// 5, P = 2, n_p = 9, 32 columns: far field (67 944 blocks of 81) 9.68 (double-
// float) -> 1.53 ms, near field (16 872 blocks of 36) 1.49 (FP64 pipe) -> 0.22
// ms; one column 1.68 -> 1.31 ms far. Torus M = 3, n_p = 10, 16 complex
// columns: far 9.65 -> 1.85 ms, near 2.58 -> 0.30 ms. Relative error of a
// product against exact sums 3e-16 (double-float far field: 5e-14).
template <int SRC>
__global__ void __launch_bounds__(kOzThreads, 1) k_bsr_oz(const __grid_constant__ OzArgs a) {
  constexpr bool C = SRC != kDigits;
  constexpr int PARTS = C ? 2 : 1;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ uint64_t full[kMaxStages], empty[kMaxStages], acc_full[2], acc_free[2], fin_bar;
  __shared__ uint64_t raw_full[kMaxRaws], raw_empty[kMaxRaws];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag, any_careful, conv_left, conv_stages[kConvWarps];
  volatile int* abort_v = &abort_flag;
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int S = a.stages;

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_slot)),
                 "r"(kTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
  }
  if (tid == 0) {
    for (int b = 0; b < S; ++b) {
      mbar_init(&full[b], kConvWarps + 1);  // the converters and the panel's copy
      mbar_init(&empty[b], 1);
    }
    for (int b = 0; b < a.raws; ++b) {
      mbar_init(&raw_full[b], 1);
      mbar_init(&raw_empty[b], kConvWarps);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_free[b], kEpiWarps);
    }
    mbar_init(&fin_bar, 1);
    abort_flag = any_careful = conv_left = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const uint32_t tmem = tmem_slot;
  Cursor cur{};
  cur.item = blockIdx.x;

  if (warp >= kConvWarp0) {
    // ---- converters ----
    // this lane's row and column group of every stage, one after another
    // where the stage has more than the lanes
    const int u0 = 32 * (warp - kConvWarp0) + lane, jg0 = u0 / a.B, i0 = u0 - jg0 * a.B;
    Ring sr{0, 0u}, rr{0, 0u};
    int item = -1, ex0 = 0;  // the exponent of row i0 (pairs and FP64 entries are split here)
    int stages = 0;          // handed over
    for (open_item(a, cur); !cur.done; next_stage<PARTS>(a, cur)) {
      const int slot = sr.slot, raw = rr.slot;
      const int* rexp = a.seg[cur.seg].rexp + (long)cur.row * a.B;
      if (SRC != kDigits && item != cur.item) {
        item = cur.item;
        ex0 = __ldg(rexp + i0);
      }
      int ok = 1;
      if (lane == 0) {
        const bool r = mbar_test(&raw_full[raw], rr.phase), f = mbar_test(&empty[slot], sr.phase ^ 1u);
        ok = !*abort_v && (r || mbar_wait(&raw_full[raw], rr.phase)) && (f || mbar_wait(&empty[slot], sr.phase ^ 1u));
      }
      ok = __shfl_sync(0xffffffffu, ok, 0);
      if (!ok) {
        if (lane == 0) {
          *abort_v = 1;
          atomicExch(a.err, 21);
        }
        break;
      }
      const int kc = stage_steps(a, cur), g0 = cur.chunk * a.kw * 2;
      const uint32_t sbo = (uint32_t)kc * 256u, sl = (uint32_t)a.rg * sbo;
      const unsigned char* src = smem + a.raw_off + (uint32_t)raw * a.raw;
      unsigned char* tiles = smem + (uint32_t)slot * a.stage;
      int jg = jg0, i = i0;
      for (int u = u0; u < 2 * kc * a.B; u += kConvLanes) {
        if (u != u0) {
          jg = u / a.B;
          i = u - jg * a.B;
        }
        // the group and the columns of its block from it on (with several
        // blocks of one K step per stage, block jg / 2)
        const int gb = a.bps > 1 ? jg & 1 : jg;
        const int nv = a.B - 8 * (a.bps > 1 ? gb : g0 + jg);
        const unsigned char* p = src + (a.bps > 1 ? (uint32_t)(jg >> 1) * a.tstride : 0u);
        unsigned char* dst = tiles + (uint32_t)(i >> 3) * sbo + (uint32_t)jg * 128u + (uint32_t)(i & 7) * 16u;
        if constexpr (SRC != kDigits) {
          const int ex = u == u0 ? ex0 : __ldg(rexp + i);
          Groups gr[8];
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const int at = (8 * gb + q) * a.B + i;
            if constexpr (SRC == kPairsC) {
              const float2 v = q < nv ? reinterpret_cast<const float2*>(p)[at] : make_float2(0.0f, 0.0f);
              gr[q] = split_pair(v.x, v.y, __int_as_float((127 + 14 - max(ex, kMinPairExp)) << 23));
            } else {
              gr[q] = split_double(q < nv ? reinterpret_cast<const double*>(p)[2 * at + cur.part] : 0.0, ex + 1021);
            }
          }
#pragma unroll
          for (int d = 0; d < 4; ++d) {
            uint32_t w0[4], w1[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) digit_pair(gr[2 * q].u[d], gr[2 * q + 1].u[d], d == 0, &w0[q], &w1[q]);
            *reinterpret_cast<uint4*>(dst + (2 * d) * sl) = make_uint4(w0[0], w0[1], w0[2], w0[3]);
            *reinterpret_cast<uint4*>(dst + (2 * d + 1) * sl) = make_uint4(w1[0], w1[1], w1[2], w1[3]);
          }
          continue;
        }
        p += group_bytes(a.B, gb);
        if (nv >= 8) {
#pragma unroll
          for (int h = 0; h < 4; ++h) {
            const uint4 v = *reinterpret_cast<const uint4*>(p + (h * a.B + i) * 16);
            *reinterpret_cast<uint4*>(dst + (2 * h) * sl) = expand_digit(v.x, v.y);
            *reinterpret_cast<uint4*>(dst + (2 * h + 1) * sl) = expand_digit(v.z, v.w);
          }
        } else if (nv == 4) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const uint4 v = *reinterpret_cast<const uint4*>(p + (h * a.B + i) * 16);
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int q = 0; q < 4; ++q) *reinterpret_cast<uint4*>(dst + (4 * h + q) * sl) = expand_digit(w[q], 0x40404040u);
          }
        } else {
          const uint2 v = nv == 1 ? *reinterpret_cast<const uint2*>(p + i * 8) : make_uint2(0x40404040u, 0x40404040u);
#pragma unroll
          for (int s = 0; s < 8; ++s)
            *reinterpret_cast<uint4*>(dst + s * sl) =
                expand_digit(0x40404000u | (((s < 4 ? v.x : v.y) >> (8 * (s & 3))) & 0xFFu), 0x40404040u);
        }
      }
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
      __syncwarp();
      // a slice of FP64 complex entries serves both parts
      const bool last = SRC != kF64C || cur.part == 1;
      if (lane == 0) {
        mbar_arrive(&full[slot]);
        if (last) mbar_arrive(&raw_empty[raw]);
      }
      ++stages;
      sr.next(S);
      if (last) rr.next(a.raws);
    }
    if (lane == 0) {
      conv_stages[warp - kConvWarp0] = stages;
      __threadfence_block();
      atomicAdd(&conv_left, 1);
    }
  } else if (warp == kTmaWarp) {
    // ---- copies: one thread fills the raw ring and the panel slots, each as
    // soon as its next one is free ----
    if (lane == 0) {
      Cursor cr{};
      cr.item = blockIdx.x;
      open_item(a, cr);
      open_item(a, cur);
      Ring rr{0, 0u}, sr{0, 0u};
      int panels = 0;  // stages whose panels are under way or there
      long long t0 = clock64();
      while (!(cr.done && cur.done)) {
        bool moved = false;
        if (!cr.done && mbar_test(&raw_empty[rr.slot], rr.phase ^ 1u)) {
          const int raw = rr.slot;
          const OzSeg& g = a.seg[cr.seg];
          constexpr uint32_t EB = SRC == kF64C ? 16u : 8u;
          const int j0 = cr.chunk * a.kw * 16, cols = min(a.B - j0, a.kw * 16);
          // rounded up to 16 bytes: a block of odd size is followed by 8 padding bytes
          const uint32_t bytes = a.bps > 1 ? (uint32_t)stage_blocks(a, cr) * a.tstride
                                           : ((uint32_t)(cols * a.B) * EB + 15u) / 16u * 16u;
          mbar_expect_tx(&raw_full[raw], bytes);
          bulk_g2s(smem + a.raw_off + (uint32_t)raw * a.raw,
                   g.tiles + (SRC == kPairsC && cr.part ? g.im_off : 0) + cr.k * g.tstride + (long)j0 * a.B * EB, bytes,
                   &raw_full[raw]);
          if (SRC == kF64C) next_stage<PARTS>(a, cr);
          rr.next(a.raws);
          next_stage<PARTS>(a, cr);
          moved = true;
        }
        const int slot = sr.slot;
        if (!cur.done && mbar_test(&empty[slot], sr.phase ^ 1u)) {
          const OzSeg& g = a.seg[cur.seg];
          const int nb = stage_blocks(a, cur), kc = a.bps > 1 ? 1 : stage_steps(a, cur);
          const uint32_t bytes = 8u * a.nc * (uint32_t)kc * 32u;
          mbar_expect_tx(&full[slot], (uint32_t)nb * bytes);
          for (int b = 0; b < nb; ++b)
            bulk_g2s(smem + (uint32_t)slot * a.stage + 8u * a.slice + (uint32_t)b * bytes,
                     g.panels + (size_t)cur.pass * a.pass_panels + (size_t)__ldg(g.col + cur.k + b) * a.panel +
                         (size_t)cur.chunk * a.kw * a.nc * 8u * 32u,
                     bytes, &full[slot]);
          ++panels;
          sr.next(S);
          next_stage<PARTS>(a, cur);
          moved = true;
        }
        if (moved) {
          t0 = clock64();
        } else if (*abort_v || clock64() - t0 > kWaitCycles) {
          if (!*abort_v) atomicExch(a.err, 22);
          *abort_v = 1;
          break;
        }
      }
      // after an abort, the copies still in flight land before the CTA exits.
      // A panel's barrier counts the converters' arrivals too: once they have
      // left (their waits are bounded), this thread arrives for those that had
      // not reached the stage, and the phase ends with the copy.
      if (*abort_v) {
        for (int q = 0; q < a.raws; ++q) mbar_wait(&raw_full[q], q < rr.slot ? rr.phase : rr.phase ^ 1u);
        const long long t1 = clock64();
        volatile int* left = &conv_left;
        while (*left < kConvWarps && clock64() - t1 < 4 * kWaitCycles) {
        }
        if (*left == kConvWarps) {
          __threadfence_block();
          volatile int* done = conv_stages;
          for (int n = max(0, panels - S); n < panels; ++n) {
            for (int w = 0; w < kConvWarps; ++w)
              if (done[w] <= n) mbar_arrive(&full[n % S]);
            mbar_wait(&full[n % S], (uint32_t)(n / S) & 1u);
          }
        }
      }
    }
  } else if (warp == kMmaWarp) {
    // ---- MMA issue: the warp walks together, one elected thread issues ----
    const bool leader = elect_one();
    const uint32_t base = smem_u32(smem);
    Ring sr{0, 0u}, ar{0, 0u};
    int in_acc = 0;  // blocks in the accumulator so far
    bool issued = false, fresh = true, ready = false;
    open_item<true>(a, cur);
    while (!cur.done) {
      const int slot = sr.slot, buf = ar.slot;
      bool ok = !fresh || mbar_wait_fast(&acc_free[buf], ar.phase ^ 1u);
      ok = ok && (ready || (!*abort_v && mbar_wait_fast(&full[slot], sr.phase)));
      if (!__all_sync(0xffffffffu, ok)) {
        if (leader) {
          *abort_v = 1;
          atomicExch(a.err, 24);
        }
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      const int kc = stage_steps(a, cur);
      const uint32_t sa = base + (uint32_t)slot * a.stage, sx = sa + 8u * a.slice;
      const uint32_t dd = tmem + 256u * (uint32_t)buf;
      // K-major, no swizzle: LBO 128; SBO 256 bytes a K step of the tile (with
      // several blocks per stage a panel has one K step of its own); panel rows
      // of complex operands are [Re (t, c)][Im (t, c)], 16 row groups per half
      const uint32_t sbo = (uint32_t)kc * 256u, xsbo = a.bps > 1 ? 256u : sbo;
      const uint64_t ad = umma_desc(sa, 128, sbo), xd = umma_desc(sx, 128, xsbo);
      const StageOps ops{(uint32_t)ad, (uint32_t)(ad >> 32), (uint32_t)xd, (uint32_t)(xd >> 32),
                         (uint32_t)a.rg * (sbo >> 4), a.bps > 1 ? 16u * a.nc : 16u, xsbo};
      // whether the next stage is full already: looked up ahead of this
      // stage's MMAs, which hide the time the answer takes
      sr.next(S);
      ready = mbar_test(&full[sr.slot], sr.phase);
      // a finished block: the accumulators are handed over after chunk_blocks
      // blocks and at the end of the row
      bool hand = false;
      if (cur.part == PARTS - 1 && cur.chunk == a.nch - 1) {
        in_acc += a.bps;
        hand = in_acc == a.chunk_blocks || cur.k + a.bps >= cur.ke;
      }
      if (leader) {
        if (C || a.nc == 32) stage_mmas<C, 32>(kc, dd, ops, cur.part, fresh);
        else stage_mmas<C, 16>(kc, dd, ops, cur.part, fresh);
        mma_commit(&empty[slot]);
        if (hand) mma_commit(&acc_full[buf]);
      }
      __syncwarp();
      issued = true;
      fresh = hand;
      if (hand) {
        ar.next(2);
        in_acc = 0;
      }
      next_stage<PARTS, true>(a, cur);
    }
    if (issued && leader) {
      // every MMA of this CTA complete before the tensor memory is freed
      mma_commit(&fin_bar);
      if (!mbar_wait(&fin_bar, 0)) atomicExch(a.err, 25);
    }
  } else {
    // ---- epilogue: lanes 32 q .. + 31 (rows of the block row), columns 16 h .. + 15 ----
    const int q = warp & 3, h = warp >> 2, i = 32 * q + lane;
    const bool work = 32 * q < a.B && 16 * h < a.nc;
    // column 16 h of diagonal 0; diagonals nc apart (complex: the two halves hold 16-column diagonals)
    const uint32_t ta0 = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(C ? 128 * h : 16 * h);
    const uint32_t dstep = C ? 16u : (uint32_t)a.nc;
    Ring ar{0, 0u};
    bool stop = false;
    for (int item = blockIdx.x; item < a.nitems && !stop; item += gridDim.x) {
      const int w = item % a.nwork, pass = item / a.nwork;
      const int2 it = a.work ? __ldg(a.work + w) : make_int2(0, w);
      const OzSeg& g = a.seg[it.x];
      const int kb = __ldg(g.row_ptr + it.y), ke = __ldg(g.row_ptr + it.y + 1);
      // looked up while the first accumulator fills
      if (q == 0 && work && !(C && h)) {
        const uint32_t m = careful_columns<SRC>(a, g, it.y, it.x, pass, h);
        if (lane == 0) a.careful[2 * item + h] = (unsigned short)m;
        if (m && lane == 0) any_careful = 1;
      }
      long long P[16];
#pragma unroll
      for (int c = 0; c < 16; ++c) P[c] = 0;
      for (int cb = kb; cb < ke; cb += a.chunk_blocks, ar.next(2)) {
        const int buf = ar.slot;
        int got = 0;
        if (lane == 0 && !*abort_v) got = mbar_wait_idle(&acc_full[buf], ar.phase) ? 1 : 0;
        got = __shfl_sync(0xffffffffu, got, 0);
        if (!got) {
          if (lane == 0) {
            *abort_v = 1;
            atomicExch(a.err, 26);
          }
          stop = true;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        if (work) {
          const int s0 = a.unit - 14, s1 = a.unit - 35, s2 = 49 - a.unit;
#pragma unroll
          for (int c = 0; c < 16; c += 2) {
            uint32_t v[8][2];
#pragma unroll
            for (int d = 0; d < 8; ++d) tmem_ld2(ta0 + 256u * buf + d * dstep + c, v[d]);
            asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              int n[8];
#pragma unroll
              for (int d = 0; d < 8; ++d) n[d] = __float2int_rn(__uint_as_float(v[d][u]));  // exact, below 2^24
              // diagonals 0-2, 3-5 and 6-7 in units of 2^-14, 2^-35 and 2^-49
              const long long t0 = ((long long)n[0] << 14) + ((long long)n[1] << 7) + n[2];
              const long long t1 = ((long long)n[3] << 14) + ((long long)n[4] << 7) + n[5];
              const long long t2 = ((long long)n[6] << 7) + n[7];
              P[c + u] += (t0 << s0) + (s1 >= 0 ? t1 << s1 : (t1 + (1ll << (-s1 - 1))) >> -s1) +
                          ((t2 + (1ll << (s2 - 1))) >> s2);
            }
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(&acc_free[buf]);
      }
      if (stop || !work || i >= a.B) continue;
      // y rows row B .. row B + B - 1
      const int per = C ? 16 : a.nc, col0 = a.c0 + pass * per, ncol = min(per, a.c0 + a.ncols - col0);
      const int* f = a.fmax + (pass * a.nseg + it.x) * 32;
      const int e0 = kb < ke ? __ldg(g.rexp + (long)it.y * a.B + i) : 0, er = SRC == kPairsC ? max(e0, kMinPairExp) : e0;
      const long ro = ((long)it.y * a.B + i) * a.ldx + col0;
#pragma unroll
      for (int c = 0; c < 16; ++c) {
        const int cc = C ? c : 16 * h + c;
        if (cc < ncol) {
          const double out = oz_to_double(P[c], er + (f[cc] - 1021) - 14 - a.unit);
          if (C) g.y[2 * (ro + cc) + h] = out;
          else g.y[ro + cc] = out;
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(kTmemCols));
  // the block rows and columns that the digits do not serve, over what was written above
  if (!any_careful || abort_flag) return;
  for (int item = blockIdx.x; item < a.nitems; item += gridDim.x) {
    // halves 0 and 1 of the columns (complex: both halves hold the same ones; 16 columns: one half)
    const uint32_t m = a.careful[2 * item] | (C || a.nc == 16 ? 0u : (uint32_t)a.careful[2 * item + 1] << 16);
    if (!m) continue;
    const int pass = item / a.nwork, w = item - pass * a.nwork;
    const int2 it = a.work ? __ldg(a.work + w) : make_int2(0, w);
    plain_columns<SRC>(a, a.seg[it.x], it.y, a.c0 + pass * (C ? 16 : a.nc), m, reinterpret_cast<double*>(smem));
  }
}

bool bsr_oz_supported(int B, bool cplx, bool pairs, int max_row_blocks) {
  OzGeom g;
  return oz_geom(B, cplx, 32, cplx && !pairs ? 16 : 8, &g) && oz_unit(B, cplx, max_row_blocks) >= kOzMinUnit;
}

size_t bsr_oz_panel_bytes(int B, bool cplx) {
  OzGeom g;
  return oz_geom(B, cplx, 32, 8, &g) ? (size_t)g.panel : 0;
}

cudaError_t launch_bsr_oz_rows(bool cplx, const int* row_ptr, const void* blocks, long bstride, int nrows, int B,
                               int* rexp, int* spread, cudaStream_t s) {
  if (nrows == 0) return cudaSuccess;
  if (B < 1 || B > 128) return cudaErrorInvalidValue;
  const int threads = std::max(1, 384 / B) * B;
  const double* f = static_cast<const double*>(blocks);
  if (cplx) k_oz_rows<true><<<nrows, threads, 0, s>>>(row_ptr, f, bstride, B, rexp, spread);
  else k_oz_rows<false><<<nrows, threads, 0, s>>>(row_ptr, f, bstride, B, rexp, spread);
  return cudaGetLastError();
}
cudaError_t launch_bsr_oz_tiles(const int* row_ptr, const double* blocks, long bstride, int nrows, int B,
                                const int* rexp, void* tiles, cudaStream_t s) {
  if (nrows == 0) return cudaSuccess;
  if (B < 1 || B > 128) return cudaErrorInvalidValue;
  // a row's blocks are shared by enough CTAs to fill the GPU
  const dim3 grid(nrows, (unsigned)std::min<long>(16, std::max<long>(1, (long)8 * 152 / nrows)));
  k_oz_tiles<<<grid, 256, 0, s>>>(row_ptr, blocks, bstride, B, rexp, static_cast<unsigned char*>(tiles),
                                  bsr_oz_tile_stride(B));
  return cudaGetLastError();
}

cudaError_t launch_bsr_oz_floors(bool cplx, const int* row_ptr, const void* blocks, long bstride, int nrows, int B,
                                 const int* rexp, float* floors, cudaStream_t s) {
  if (nrows == 0) return cudaSuccess;
  if (B < 1 || B > 128) return cudaErrorInvalidValue;
  const double* f = static_cast<const double*>(blocks);
  if (cplx) k_oz_floors<true><<<nrows, 512, 0, s>>>(row_ptr, f, bstride, B, rexp, floors);
  else k_oz_floors<false><<<nrows, 512, 0, s>>>(row_ptr, f, bstride, B, rexp, floors);
  return cudaGetLastError();
}

cudaError_t launch_digits_one(const OzSeg& g, const void* x_pairs, int nrows, int B, cudaStream_t s) {
  if (nrows == 0) return cudaSuccess;
  if (B < 1 || B > 128) return cudaErrorInvalidValue;
  k_digits_one<<<nrows, 256, (size_t)8 * B * sizeof(double), s>>>(g, static_cast<const float2*>(x_pairs), B);
  return cudaGetLastError();
}

cudaError_t launch_bsr_oz(bool cplx, bool pairs, OzArgs a, int max_row_blocks, int max_passes, cudaStream_t s) {
  OzGeom g;
  if (!oz_geom(a.B, cplx, a.ncols, cplx && !pairs ? 16 : 8, &g) || a.nseg < 1 || a.nseg > kOzMaxSegs || max_passes < 1)
    return cudaErrorInvalidValue;
  if (a.nwork == 0 || a.ncols == 0) return cudaSuccess;
  a.unit = oz_unit(a.B, cplx, max_row_blocks);
  if (a.unit < kOzMinUnit) return cudaErrorInvalidValue;
  a.rg = g.rg;
  a.nks = g.nks;
  a.kw = g.kw;
  a.bps = g.bps;
  a.tstride = (uint32_t)a.seg[0].tstride;
  a.nch = g.nch;
  a.nc = g.nc;
  a.slice = g.slice;
  a.stage = g.stage;
  a.stages = g.stages;
  a.raws = g.raws;
  a.raw = g.raw;
  a.raw_off = g.raw_off;
  a.panel = g.panel;
  a.chunk_blocks = g.chunk_blocks;
  int dev = 0, nsm = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  int ncl = 0;
  for (int q = 0; q < a.nseg; ++q) ncl = std::max(ncl, a.seg[q].ncl);
  const int per = cplx ? 16 : g.nc;
  const int c_end = a.c0 + a.ncols;
  for (int c0 = a.c0; c0 < c_end; c0 += per * max_passes) {
    OzArgs b = a;
    b.c0 = c0;
    b.ncols = std::min(per * max_passes, c_end - c0);
    const int np = (b.ncols + per - 1) / per;
    b.nitems = np * b.nwork;
    // up to 8192 values of x a segment, 64 a thread, the panels' CTAs find the
    // column exponents themselves (sphere M = 2, P = 1: 34 -> 27 us)
    const bool own = (long)ncl * b.B * std::min(per, b.ncols) <= 8192;
    if (!own) {
      e = cudaMemsetAsync(b.fmax, 0, (size_t)np * b.nseg * 32 * sizeof(int), s);
      if (e != cudaSuccess) return e;
    }
    const dim3 gc((unsigned)std::max<long>(1, std::min<long>(2 * nsm, ((long)ncl * b.B + 15) / 16)), b.nseg, np);
    const long nt = std::max<long>(1, (long)ncl * 2 * g.nks * g.nc);
    const dim3 gp((unsigned)((nt + 127) / 128), b.nseg, np);
    const int grid = std::min(b.nitems, nsm);
    auto run = [&](auto cols, auto panels, auto own_panels, auto product) {
      if (!own) cols<<<gc, 256, 0, s>>>(b);
      if (own) own_panels<<<gp, 128, 0, s>>>(b);
      else panels<<<gp, 128, 0, s>>>(b);
      const cudaError_t r = smem_limit(product, g.smem);
      if (r == cudaSuccess) product<<<grid, kOzThreads, g.smem, s>>>(b);
      return r;
    };
    if (cplx && pairs) e = run(k_oz_cols<true>, k_oz_panels<true, false>, k_oz_panels<true, true>, k_bsr_oz<kPairsC>);
    else if (cplx) e = run(k_oz_cols<true>, k_oz_panels<true, false>, k_oz_panels<true, true>, k_bsr_oz<kF64C>);
    else e = run(k_oz_cols<false>, k_oz_panels<false, false>, k_oz_panels<false, true>, k_bsr_oz<kDigits>);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace bg
