// Tensor-core (tcgen05) ImageProximity path for sm_100a.
//
// The product term of SqrDistance[_Norm] and CrossCorr[_Norm]
// (cl-files/ImageProximity.cl :44, :122, :290, :375),
//   C(x, y) = sum_h sum_w S(x + w - ax, y + h - ay) * T(w, h),
// is computed per channel and strip of P = 128 S output positions by one
// chain of MMAs per source row. TMEM lane m holds the S positions
// x0 + S m + p (p < S). R (template rows rounded up to 16, 32 or 64) and S
// satisfy S R = 128: S = 8, 4, 2. An MMA instruction (M = 128, K = 16) takes
// the same time for any N up to 256, so the kernel makes N as wide as the
// accumulators in TMEM allow.
//
// A operand (shared memory, no per-lane copies). Lane m's K window is the
// staged row itself, A[m][k] = raw(S m + k): a Hankel matrix. In the
// canonical K-major SWIZZLE_NONE layout a core matrix row is 16 bytes, so the
// row is stored once more per S pixels: buffer row q holds raw elements
// S q .. S q + 7 (BF16) or .. + 15 (i8), and core matrix c of lane m is buffer
// row m + c (8/S) [(16/S) for i8]: one descriptor per MMA with SBO = 128 and
// LBO = the distance of the next K core matrix.
//
// F32 and U16 sources are split into BF16 hi + lo (U16 exactly) and three
// products hi*Thi + hi*Tlo + lo*Thi accumulate in FP32. They are packed into
// MMAs of K = 16 by pairing core matrices along K: (hi_c, lo_c) x (Tlo_c, Thi_c)
// for every chunk c, then (hi_2i, hi_2i+1) x (Thi_2i, Thi_2i+1). U8 sources use
// the i8 MMA with s32 accumulation (exact).
//
// B operand: N = S R = 128 rows; the row of phase p and slot j holds template
// row th - 1 - j shifted by p and by the staged row's lead: T(k - p - lead,
// th - 1 - j). Source row t then adds to output-row slots t .. t + R - 1 (slot u
// is the output row whose last template row is source row u). The rows stand in
// two halves, phases p < S/2 and p >= S/2, each S/2 rows a slot, so that
// each half of the positions has TMEM columns of its own.
//
// Blocks. The steps (source rows) of an item are cut into blocks of
// B = 16 / S steps. Step q of a block adds into TMEM columns (S/2) q + [0, 64)
// of each half of the block's partial buffer: MMAs of N' = 2 * 72 columns
// with B read (S/2) q rows later (B is stored with zero rows in front of, between
// and behind the halves), so the block's partial sums of its B + R - 1 slots
// end up at columns (S/2) j + p of their half. The block's first MMA does not
// accumulate, which clears the buffer. Partial buffers are double-buffered: the
// epilogue reads block k while the tensor cores fill block k + 1.
//
// Running sums, F32 and U16. The epilogue adds each block's partials to the running sums of
// the open slots, 64 registers of each thread (FP32 round-to-nearest). The first 8 columns of a half are the B slots the block
// completes; the sums move down 8 registers a block as they are added to. The
// tensor cores' FP32 accumulation into one value thus never spans more than
// one block: that accumulator rounds every addition with a bias that grows with
// the number of additions, so the chains of a whole window (th rows x K
// chunks) would cost accuracy.
//
// U8. Integer sums are exact in any order, so they need neither partials nor running
// sums: the MMAs accumulate in TMEM over the whole window, in a ring of 512 columns
// that a block's 144-column window moves along by 16 columns (in two parts where it
// wraps; the slots then stand S columns each, without halves). The epilogue takes
// the 16 columns that a block completes and clears them; the MMAs may run up to 24
// blocks ahead of it, and the row energies of blocks of 2 or 4 steps are fetched
// three blocks ahead. A batch of 60 U8 maps of 1024 x 1024 (templates of 8 to 64 a
// side, SqrDistance) went from 426 to 381 us.
//
// Window energies sum S^2 of each position (measures other than CrossCorr):
// a separate pre-pass (row_energy.cu) writes the row energies R(x, r) =
// sum_{w < tw} S^2(x + w - ax, r) of every source row (int32 for U8, FP32
// otherwise); the epilogue keeps each position's window energy as a running
// sum (FP64; int32 for U8) over the rows it walks (add R of the row a slot
// completes, drop R of the row th back), loading a block's R values before it
// waits for the block's MMAs. Exact for U8; for F32 and U16 one rounding of
// 2^-24 per row energy, as far as row_energy.cu states. F32 and U16 sources:
// SqrDistance = E_S - 2C + E_T is formed in FP64, the _Norm scale in FP32 for
// an F32 map and in FP64 for an F64 one. U8: as the plain path does them (the
// results are bit-identical to it).
//
// Roles (12 warps; one CTA per SM, which holds all 512 TMEM columns):
//   warps 0-2  builders: each loads (TMA, zero fill outside the image) and
//              builds whole rows of the A operand (split into hi/lo);
//   warp 3     MMA issue (one commit per block of rows: the block's partial
//              and its A stages are free once it completes);
//   warps 4-11 epilogue, two per TMEM sub-partition, one for each half of the
//              positions: running sums, window energies, score map.
//
// Bound: an MMA of M = 128, N = 144 takes the tensor pipe 72 cycles and reads
// 8.7 KB of operands from shared memory in them, 120 of the 128 bytes a cycle
// that shared memory and L1 give, so what the other warps read and write there
// (staged rows, A operand, energies, maps) slows the MMAs. 4096 x 4096 F32, 31 x 31
// under the profiler: CrossCorr 253 thousand cycles for 259 steps of 8 MMAs (576
// cycles), about 930 a step, shared memory 92 percent busy (54 the MMAs, 38 the
// rest); SqrDistance_Norm 346 thousand, 1290 a step, shared memory 58 percent: with
// energies the epilogue's chain binds (conversions to FP64, its warps wait as much
// for the arithmetic pipes as for memory). By the same count a step took 1240 and
// 1600 with a wait per step, one warp per sub-partition in the epilogue, the running
// sums in TMEM and FP64 scores. CrossCorr_Norm of that image went from 234 to 208 us
// (row energies included), the 3840 x 2160 x 4 U16 map with 64 x 64 from 1296 to 1085.
//
// Every wait is bounded: a wait that gives up sets the CTA's abort flag, the
// roles leave their loops, the MMA and TMA threads drain what they issued,
// and the kernel raises the context's error flag.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstring>
#include <map>
#include <mutex>
#include <tuple>
#include <type_traits>
#include <vector>

#include "sm100.cuh"
#include "tensor.h"
#include "row_energy.h"

namespace ocipb {
namespace {

using namespace sm100;

constexpr int kM = 128;                 // TMEM lanes = A rows
constexpr int kBuilders = 3;
constexpr int kEpilogue = 8;            // two warps per TMEM sub-partition
constexpr int kMmaWarp = kBuilders;
constexpr int kFirstEpilogue = kMmaWarp + 1;  // a multiple of 4: warp mod 4 is its sub-partition
constexpr int kWarps = kFirstEpilogue + kEpilogue;  // 3 a scheduler, so 168 registers a thread
constexpr int kThreads = kWarps * 32;
constexpr int kMaxRaw = 18;             // staged source rows at most (TMA stages of one row)
constexpr int kMaxAB = 4;               // blocks of A operand stages at most
constexpr int kSR = 128;                // S R: template rows x positions per lane
constexpr int kN = kSR;                 // B rows (MMA N without the slide)
constexpr int kHalfN = kN / 2;          // of each half of the positions
constexpr int kHalf = kHalfN + 8;       // columns of a half: a block's slides fit in 8 more
constexpr int kNp = 2 * kHalf;          // MMA N
constexpr int kPartCols = kNp;          // TMEM columns per partial buffer (two of them)
constexpr int kRingChunks = kHalfN / 8; // open slots of a half: 8 chunks of 8 columns
// U8: the sums of all open slots accumulate in TMEM, in a ring of 32 chunks of 16
// columns; a block's MMAs cover 9 of them.
constexpr int kU8Chunks = 32, kU8Window = kNp / 16, kU8Group = 8, kU8Groups = kU8Chunks / kU8Group;
constexpr int kMaxBlk = kU8Chunks;      // "block full" barriers at most
// U8: row energies of the next blocks on their way in shared memory (2 KB a warp and
// block). The MMAs of a block of 2 to 8 steps take less than a load's latency.
constexpr int kU8Ahead = 4;
constexpr int kU8Energies = 2048;
constexpr int kTmemCols = 512;
constexpr int kMinSmem = 120 * 1024;    // keeps one CTA per SM (it takes all of TMEM)
constexpr int kMaxDynSmem = 226 * 1024; // opt-in dynamic shared memory limit of the kernel
constexpr long long kSpinLimit = 4000000000LL;  // about 2 s of SM clock
constexpr int kTmplBatch = 8;           // template loads a thread has in flight

enum Elem { kF32 = 0, kU8 = 1, kU16 = 2 };

// Staged rows (multiples of the builders, so that a stage belongs to one of
// them) and blocks of A stages. A step of a U8 item is
// one to three MMAs (72 cycles each), of a split item 4 to 16, so the U8 rows
// are loaded and built further ahead: a load takes about 2000 cycles to land,
// a row about 500 to build.
__host__ __device__ constexpr int raw_stages(bool split) { return split ? 9 : 18; }
__host__ __device__ constexpr int a_blocks(bool split) { return split ? 2 : 4; }

template <int ELEM>
struct ElemTraits {
  static constexpr bool split = ELEM != kU8;  // BF16 hi/lo operands
  static constexpr int size = ELEM == kF32 ? 4 : ELEM == kU16 ? 2 : 1;
  static constexpr int inner = 16 / size;     // elements per 16-byte TMA group
  static constexpr int cmk = split ? 8 : 16;  // K elements per core-matrix row
  static constexpr int raw = raw_stages(split);
  static constexpr int ab = a_blocks(split);
};

// Positions per TMEM lane for a template of R rows (S R = 128), and the steps
// of a block (S B = 16: a block's completed slots are one 16-column chunk).
__host__ __device__ constexpr int s_for(int R) { return kSR / R; }
__host__ __device__ constexpr int block_steps(int S) { return 16 / S; }

// Geometry of one work item (host and device).
struct Geo {
  int S, P, R, B;
  int NB;          // B-operand rows stored per core matrix
  int KC;          // core matrices of one K segment
  int nmma;        // MMAs per source row
  int cma;         // A core matrices addressed per lane (hi, incl. the pairing's spare)
  int QR;          // buffer rows of one A plane
  int lbok;        // bytes between K-adjacent core matrices of A
  int nraw;        // staged elements the windows cover (lead + P - 1 + tw)
  int NA;          // A operand stages: a_blocks() blocks of steps
};

__host__ __device__ inline Geo make_geo(bool split, int R, int tw, int lead) {
  Geo g;
  g.S = s_for(R);
  g.P = kM * g.S;
  g.R = R;
  g.B = block_steps(g.S);
  g.NB = split ? kNp + 8 - g.S / 2 : kNp + 16 - g.S;
  const int cmk = split ? 8 : 16;
  const int keff = tw + g.S - 1 + lead;
  g.KC = (keff + cmk - 1) / cmk;
  if (split) {
    g.nmma = g.KC + (g.KC + 1) / 2;
    g.cma = 2 * ((g.KC + 1) / 2);
  } else {
    g.nmma = (g.KC + 1) / 2;
    g.cma = 2 * g.nmma;
  }
  g.lbok = 16 * (cmk / g.S);
  g.QR = kM + (cmk / g.S) * (g.cma - 1);
  g.nraw = lead + g.P - 1 + tw;
  g.NA = a_blocks(split) * g.B;
  return g;
}

// Staged elements of one row: the last buffer row's end, and every element
// of the strip's windows.
__host__ __device__ inline int staged_elems(const Geo& g, bool split) {
  const int a = g.S * (g.QR - 1) + (split ? 8 : 16);
  return a > g.nraw ? a : g.nraw;
}

// One work item: one channel of one strip x band of rows of one
// (image, template) pair.
struct ItemArgs {
  const CUtensorMap* tmap;  // source planes (rank 4: group, groups, rows, channel)
  int W, H;
  int tw, th, R;
  int ax, ay;    // window anchor: output (x, y) reads S(x + w - ax, y + h - ay)
  int nch, ch;
  int xs_out;    // strip covers outputs [xs_out, xs_out + P)
  int y0, yend;  // band of output rows
  int nbox;      // 16-byte groups per staged row (box_split loads of box_part)
  const char* tmpl;
  size_t tmpl_pitch;
  char* dst;
  size_t dst_pitch;
  int dst_f64;
  int measure;
  // Row energies (measures other than CrossCorr): int32 (U8) or FP32 planes
  // of R(x, r), plane ch at energy + ch * e_plane bytes, rows e_pitch apart.
  const char* energy;
  size_t e_pitch, e_plane;
  int dst_nch, dst_ch;  // channels of the destination, and the item's
  int raw;       // U8 product sums as int32 bits (the tiles of a larger template)
  // Best match (ocipProximityIndx): -1 none, else the index reduction
  // (0 min, 1 max, 2 min |v|, 3 max |v|) of the F32 scores; each epilogue warp
  // writes one IdxRecord per item to idx_out[item * kEpilogue + warp]. dst may
  // then be null (no map written).
  int idx_op;
  char* idx_out;
};

// Best score of an epilogue warp's positions in one item. Among equal values
// the smallest key wins: key = (reference work-group index << 12) |
// (bit-reversed work-item id << 4) | pixel index within the work-item, the
// order in which the reference's index reduction resolves ties
// (cl-files/Statistics.cl REDUCE_POS: a strict scan of 16 pixels per
// work-item, a tree fold over work-items that keeps the left one on ties, a
// strict fold over work-groups). NaN scores are only flagged: with a NaN in
// the map the reference's answer depends on where it lies, so the caller
// takes the map path then.
struct IdxRecord {
  float v;
  int have;
  unsigned long long key;
  int nan;
  int pad;
};

// Shared-memory layout, identical on host and device.
struct Layout {
  int row_bytes, raw_stage, raw, b, a_stage, a, energies, bars, total;
};

__host__ __device__ inline int align128(int x) { return (x + 127) & ~127; }

// A staged row of nbox 16-byte groups is loaded by box_split(nbox) TMA copies
// of box_part(nbox) groups each: a box dimension holds at most 256, and every
// copy's shared-memory destination must be 128-byte aligned, so a part is a
// multiple of 8 groups.
__host__ __device__ inline int box_split(int nbox) { return (nbox + 255) / 256; }
__host__ __device__ inline int box_part(int nbox) {
  return ((nbox + box_split(nbox) - 1) / box_split(nbox) + 7) & ~7;
}

__host__ __device__ inline Layout make_layout(bool split, const Geo& g, int nbox) {
  Layout L;
  L.row_bytes = box_split(nbox) * box_part(nbox) * 16;
  L.raw_stage = align128(L.row_bytes);
  L.raw = 0;
  L.b = L.raw + raw_stages(split) * L.raw_stage;
  L.a = L.b + align128(2 * g.nmma * g.NB * 16);
  L.a_stage = align128(g.QR * 16 * (split ? 2 : 1));
  L.energies = L.a + g.NA * L.a_stage;
  L.bars = L.energies + (split ? 0 : kEpilogue * kU8Ahead * kU8Energies);
  // raw full; A block ready, A block free; block full, sums read; done.
  L.total = L.bars + align128(8 * (kMaxRaw + 2 * kMaxAB + kMaxBlk + kU8Groups + 1));
  return L;
}

// CTA state that outlives one work item.
struct CtaState {
  uint32_t tmem;  // TMEM base address (all 512 columns)
  int abort;      // set by a wait that gave up; the CTA stops taking items
  int next;       // work item fetched from the queue
  double et[kWarps];  // template energy of the item's channel, one part per warp
};

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float bf16lo_f(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16hi_f(uint32_t w) { return __uint_as_float(w & 0xFFFF0000u); }

// Template element (w, h) of channel c as a float (exact for every type).
template <int ELEM>
__device__ __forceinline__ float tmpl_at(const ItemArgs& a, int h, int w, int c) {
  const char* row = a.tmpl + (size_t)h * a.tmpl_pitch;
  const int i = w * a.nch + c;
  if (ELEM == kF32) return __ldg(reinterpret_cast<const float*>(row) + i);
  if (ELEM == kU16) return __ldg(reinterpret_cast<const uint16_t*>(row) + i);
  return __ldg(reinterpret_cast<const uint8_t*>(row) + i);
}

// S staged elements from element e0, a multiple of S, as floats (F32, U16).
template <int ELEM, int S>
__device__ __forceinline__ void load_s(const unsigned char* row, int e0, float (&f)[S]) {
  if (ELEM == kF32) {
    if (S % 4 == 0) {
#pragma unroll
      for (int j = 0; j < S / 4; ++j) {
        const float4 u = reinterpret_cast<const float4*>(row + 4 * e0)[j];
        f[(4 * j) % S] = u.x;
        f[(4 * j + 1) % S] = u.y;
        f[(4 * j + 2) % S] = u.z;
        f[(4 * j + 3) % S] = u.w;
      }
    } else {
      const float2 u = *reinterpret_cast<const float2*>(row + 4 * e0);
      f[0] = u.x;
      f[1] = u.y;
    }
  } else {
    uint32_t w[S / 2];
    if (S == 8) {
      const uint4 u = *reinterpret_cast<const uint4*>(row + 2 * e0);
      memcpy(w, &u, sizeof(w));
    } else if (S == 4) {
      const uint2 u = *reinterpret_cast<const uint2*>(row + 2 * e0);
      memcpy(w, &u, sizeof(w));
    } else {
      w[0] = *reinterpret_cast<const uint32_t*>(row + 2 * e0);
    }
#pragma unroll
    for (int j = 0; j < S / 2; ++j) {
      f[2 * j] = static_cast<float>(w[j] & 0xFFFFu);
      f[2 * j + 1] = static_cast<float>(w[j] >> 16);
    }
  }
}

// Running best of one lane (the fused best match): the value, its key and
// flags. A value replaces the best when strictly better, or equal with a
// smaller key; NaN values are only flagged.
struct IdxState {
  float v;
  unsigned long long key;
  int have, nan;
};

__device__ __forceinline__ unsigned long long idx_key_of(int x, int y, int ngx) {
  const unsigned lid = ((unsigned)(y & 15) << 4) | (unsigned)(x & 15);
  const unsigned long long grp = (unsigned long long)(y >> 4) * ngx + (x >> 8);
  return (grp << 12) | ((unsigned long long)(__brev(lid) >> 24) << 4) | (unsigned)((x & 255) >> 4);
}

__device__ __forceinline__ void idx_state_update(IdxState& st, float v, int x, int y, int op,
                                                 int ngx) {
  const float c = op >= 2 ? fabsf(v) : v;
  if (c != c) {
    st.nan = 1;
    return;
  }
  const bool is_min = op == 0 || op == 2;
  if (st.have && (is_min ? c > st.v : c < st.v)) return;
  const unsigned long long k = idx_key_of(x, y, ngx);
  if (st.have && c == st.v && k > st.key) return;
  st.v = c;
  st.key = k;
  st.have = 1;
}

// num / sqrt(es * ei) of exact integers, rounded to FP32 through FP64 as
// (float)(num / sqrt(es * ei)) with each FP64 operation correctly rounded. That
// chain (a divide and a square root, about 220 cycles of a warp with no
// overlap) is the true quotient within 2^-51, so an estimate within 2^-41
// gives the same FP32 value unless a rounding boundary lies that near.
// norm_near gives the estimate and whether it decides the value; norm_exact
// is the chain, for the others (one value in 2^14, and zero energies).
// es, ei < 2^31, |num| < 2^31; ret ~ 1 / sqrt(ei).
__device__ __forceinline__ float norm_near(int num, int es, int ei, float ret, bool& decided) {
  auto f64 = [](int v) {  // exact, without a conversion (8 cycles of a quarter of the SM)
    return __hiloint2double(0x43300000, v ^ 0x80000000) - 4503601774854144.0;  // 2^52 + 2^31
  };
  const double x = f64(es) * f64(ei);
  const double r = rsqrtf((float)es) * ret;   // 1 / sqrt(x) within 2^-21
  const double q = f64(num) * (r * fma(-0.5 * x * r, r, 1.5));  // a Newton step: 2^-41
  const int low = __double2loint(q) & 0x1fffffff;  // the bits FP32 drops
  decided = es > 0 && ei > 0 && abs(low - 0x10000000) > 0x4000;
  return (float)q;
}
__device__ __forceinline__ float norm_exact(int num, int es, int ei) {
  return (float)__ddiv_rn((double)num, __dsqrt_rn(__dmul_rn((double)es, (double)ei)));
}

// U8 _Norm: float arithmetic where the plain path's float sums are exact.
__device__ __forceinline__ bool u8_norm_in_float(int tw, int th) {
  return (double)tw * th * 65025.0 <= 16777216.0;
}

template <bool SPLIT>
struct Sums {
  typedef typename std::conditional<SPLIT, float, int>::type A;   // product sums
  typedef typename std::conditional<SPLIT, double, int>::type E;  // window energies
  typedef typename std::conditional<SPLIT, float, int>::type R;   // row energies
};

// Scores of one position from its product sum cv and window energy ev (etd:
// template energy, ret ~ 1 / sqrt(etd)). Split sources: SqrDistance's terms
// cancel near a match, so its numerator is formed in FP64; the _Norm scale of
// an F32 map is taken in FP32 (relative error a few 1e-7), of an F64 map in
// FP64. U8: the plain path's float or double formulas (bit-identical) on
// integers exact in int32, as each of C, E_S, E_T <= 64 * 64 * 255^2 < 2^28.
template <bool SPLIT, int M>
__device__ __forceinline__ float score_f(typename Sums<SPLIT>::A cv, typename Sums<SPLIT>::E ev,
                                         double etd, float ret, bool u8_float) {
  constexpr bool product = M == kCrossCorr || M == kCrossCorrNorm;
  if constexpr (SPLIT) {
    float num;
    if (product)
      num = cv;
    else
      num = (float)(ev - 2.0 * (double)cv + etd);
    return M == kCrossCorr || M == kSqrDistance ? num : num * (rsqrtf((float)ev) * ret);
  } else {
    const int eti = static_cast<int>(etd);
    const int num = product ? cv : ev - 2 * cv + eti;
    if (M == kCrossCorr || M == kSqrDistance) return __int2float_rn(num);
    if (u8_float) return __fdiv_rn((float)num, __fsqrt_rn(__fmul_rn((float)ev, (float)eti)));
    return norm_exact(num, ev, eti);
  }
}

// score_f of eight positions, independent of one another.
template <bool SPLIT, int M>
__device__ __forceinline__ void scores8(float (&out)[8], const typename Sums<SPLIT>::A (&val)[8],
                                        const typename Sums<SPLIT>::E (&es)[8], double etd,
                                        float ret, bool u8_float) {
  if constexpr (!SPLIT && (M == kCrossCorrNorm || M == kSqrDistanceNorm)) {
    if (!u8_float) {
      const int eti = static_cast<int>(etd);
      bool all = true;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        bool decided;
        out[i] = norm_near(M == kCrossCorrNorm ? val[i] : es[i] - 2 * val[i] + eti, es[i], eti, ret,
                           decided);
        all = all && decided;
      }
      if (all) return;
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) out[i] = score_f<SPLIT, M>(val[i], es[i], etd, ret, u8_float);
}

template <bool SPLIT, int M>
__device__ __forceinline__ double score_d(typename Sums<SPLIT>::A cv, typename Sums<SPLIT>::E ev,
                                          double etd, bool u8_float) {
  constexpr bool product = M == kCrossCorr || M == kCrossCorrNorm;
  if constexpr (SPLIT) {
    const double num = product ? (double)cv : ev - 2.0 * (double)cv + etd;
    return M == kCrossCorr || M == kSqrDistance ? num : num * rsqrt(ev * etd);
  } else {
    const int eti = static_cast<int>(etd);
    const int num = product ? cv : ev - 2 * cv + eti;
    if (M == kCrossCorr || M == kSqrDistance) return (double)num;
    if (u8_float)
      return (double)__fdiv_rn((float)num, __fsqrt_rn(__fmul_rn((float)ev, (float)eti)));
    return __ddiv_rn((double)num, __dsqrt_rn(__dmul_rn((double)ev, (double)eti)));
  }
}

// Scores and stores of one slot that is not a whole run of a one-channel F32
// map's row: F64 maps, several channels, the right edge. v: the F32 scores, for the best match.
template <int ELEM, int SH, int M>
__device__ __noinline__ void store_slot(const ItemArgs& a, int xl, char* orow,
                           const typename Sums<ElemTraits<ELEM>::split>::A* val,
                           const typename Sums<ElemTraits<ELEM>::split>::E* esum, double etd,
                           float* v) {
  constexpr bool SPLIT = ElemTraits<ELEM>::split;
  const bool u8_float = u8_norm_in_float(a.tw, a.th);
  if (a.dst_f64) {
    double* o = reinterpret_cast<double*>(orow) + (size_t)xl * a.dst_nch + a.dst_ch;
#pragma unroll
    for (int p = 0; p < SH; ++p) {
      if (xl + p >= a.W) break;
      o[p * a.dst_nch] = score_d<SPLIT, M>(val[p], esum[p], etd, u8_float);
    }
    return;
  }
  const float ret = (float)(1.0 / sqrt(etd));
#pragma unroll
  for (int p = 0; p < SH; ++p) {
    v[p] = score_f<SPLIT, M>(val[p], esum[p], etd, ret, u8_float);
    if (!SPLIT && a.raw) v[p] = __int_as_float(static_cast<int>(val[p]));
    if (xl + p < a.W && a.dst != nullptr)
      reinterpret_cast<float*>(orow)[(size_t)(xl + p) * a.dst_nch + a.dst_ch] = v[p];
  }
}

// Epilogue of an item, one of two warps of each TMEM sub-partition: warp
// 4 + 4 h + s takes positions [h S/2, (h + 1) S/2) of lanes 32 s .. 32 s + 31,
// which have their own 72 columns of the partials (U8: S/2 of every S columns of the
// ring). One warp is a chain of dependent steps (TMEM round trips, conversions,
// energies), so the block's time is its latency; with one warp per sub-partition, FP64
// scores of every measure and a wait per 16 columns, the 31 x 31 F32 kernel's
// step took 1170-1410 cycles here against 580 of the MMAs.
template <int ELEM, int S, bool IDX, int M>
__device__ __forceinline__ void run_epilogue(const ItemArgs& a, CtaState& cs, uint32_t tmem_base,
                                             uint64_t* blk_full, uint64_t* buf_free, int r_begin,
                                             int nsteps, unsigned char* energies) {
  constexpr bool SPLIT = ElemTraits<ELEM>::split;
  constexpr int R = kSR / S;
  constexpr int BS = block_steps(S);
  constexpr int SH = S / 2;
  constexpr bool kE = M != kCrossCorr;  // the measure needs window energies
  // U8 blocks of 2 and 4 steps: energies fetched blocks ahead. Blocks of 8 steps last
  // long enough (1920 x 1080 48 x 40 took 72.1 us with it, 70.6 without).
  constexpr bool kAhead = kE && !SPLIT && S > 2;
  typedef typename Sums<SPLIT>::A AT;
  typedef typename Sums<SPLIT>::E ET;
  typedef typename Sums<SPLIT>::R RT;
  volatile int* abort_flag = &cs.abort;
  const int ew = (threadIdx.x >> 5) - kFirstEpilogue, lane = threadIdx.x & 31;
  const int half = ew >> 2;
  const uint32_t lane_base = tmem_base + (static_cast<uint32_t>((ew & 3) * 32) << 16);
  // The item's fields in registers: the item lives in shared memory, and
  // the score loop would otherwise reload them on every slot.
  const int W = a.W, H = a.H, th = a.th, nch = a.dst_nch;
  const int idx_op = IDX ? a.idx_op : -1;
  const int xl = a.xs_out + S * ((ew & 3) * 32 + lane) + half * SH;  // first position
  const bool whole = xl + SH <= W;
  const bool f32 = !a.dst_f64, raw = !SPLIT && a.raw;
  double etd = 0.0;  // template energy
#pragma unroll
  for (int w = 0; w < kWarps; ++w) etd += cs.et[w];
  const float ret = (float)(1.0 / sqrt(etd));  // 1 / sqrt(E_T)
  const bool u8_float = u8_norm_in_float(a.tw, th);
  // Best-match state of this lane (ocipProximityIndx).
  IdxState ib;
  ib.v = 0.f;
  ib.key = 0ull;
  ib.have = 0;
  ib.nan = 0;
  const int idx_ngx = (W + 255) >> 8;

  // Row energies of the rows a block's slots complete (entering: staged row u;
  // leaving: staged row u - th), loaded before the block's MMAs are waited
  // for. The window energy of each position is a running sum over the slots,
  // in order (FP64, exact int32 for U8). Positions past the last column read
  // the rows' pitch (a multiple of 32 values) and are not stored.
  uint32_t rin[BS][SH] = {}, rout[BS][SH] = {};
  ET esum[SH];
#pragma unroll
  for (int p = 0; p < SH; ++p) esum[p] = ET(0);
  auto add_energy = [&](int g, int p) {
    if constexpr (SPLIT)
      esum[p] += (double)__uint_as_float(rin[g][p]) - (double)__uint_as_float(rout[g][p]);
    else
      esum[p] += static_cast<int>(rin[g][p] - rout[g][p]);
  };
  const char* e_row = nullptr;  // the row entering with the block's first slot
  size_t e_pitch = 0, e_back = 0;
  if (kE) {
    e_pitch = a.e_pitch;
    e_back = (size_t)th * e_pitch;
    e_row = a.energy + (size_t)a.ch * a.e_plane + (size_t)xl * sizeof(RT) +
            (ptrdiff_t)r_begin * (ptrdiff_t)e_pitch;
  }
  auto load_row = [&](uint32_t (&v)[SH], const char* at, bool ok) {
    if (SH == 4) {
      const uint4 q = ok ? *reinterpret_cast<const uint4*>(at) : make_uint4(0u, 0u, 0u, 0u);
      memcpy(v, &q, sizeof(v));
    } else if (SH == 2) {
      const uint2 q = ok ? *reinterpret_cast<const uint2*>(at) : make_uint2(0u, 0u);
      memcpy(v, &q, sizeof(v));
    } else {
      v[0] = ok ? *reinterpret_cast<const uint32_t*>(at) : 0u;
    }
  };
  // Running sums of the open slots (FP32 round-to-nearest): 8 chunks of BS slots,
  // chunk 0 the next block's completed one.
  // U8: they are in TMEM.
  AT ring[SPLIT ? kRingChunks : 1][8];
  if constexpr (SPLIT) {
#pragma unroll
    for (int c = 0; c < kRingChunks; ++c)
#pragma unroll
      for (int j = 0; j < 8; ++j) ring[c][j] = AT(0);
  }
  // The row energies come from the launch before this one, which this kernel
  // may overlap up to here (launch_items).
  if (kE) cudaGridDependencySynchronize();
  char* orow = a.dst + (ptrdiff_t)(a.y0 - R + 1) * (ptrdiff_t)a.dst_pitch;  // of slot 0
  const size_t dst_pitch = a.dst_pitch;
  const bool has_dst = a.dst != nullptr;
  // U8: block k's row energies by cp.async into slot k mod kU8Ahead, each lane its
  // own (entering rows, then leaving ones), one commit group a block.
  auto slot_of = [&](int k, int i) {
    return reinterpret_cast<uint32_t*>(energies + (ew * kU8Ahead + k % kU8Ahead) * kU8Energies) +
           (i * 32 + lane) * SH;
  };
  auto prefetch = [&](int k) {
    if (k * BS < nsteps) {
#pragma unroll
      for (int g = 0; g < BS; ++g) {
        const int u = k * BS + g, r = r_begin + u;
        const bool in = u < nsteps && xl < W;
        const char* at = e_row + g * e_pitch;
        const bool enter = in && r >= 0 && r < H, leave = in && u >= th && r >= th && r - th < H;
        cp_async_zfill<4 * SH>(slot_of(k, g), enter ? at : a.energy, enter);
        cp_async_zfill<4 * SH>(slot_of(k, BS + g), leave ? at - e_back : a.energy, leave);
      }
      e_row += BS * e_pitch;
    }
    cp_async_commit();
  };
  if constexpr (kAhead) {
#pragma unroll
    for (int k = 0; k < kU8Ahead - 1; ++k) prefetch(k);
  }
  for (int k = 0; k * BS < nsteps; ++k) {
    const int t0 = k * BS;
    if constexpr (kAhead) prefetch(k + kU8Ahead - 1);
    if (kE && !kAhead) {
#pragma unroll
      for (int g = 0; g < BS; ++g) {
        const int u = t0 + g, r = r_begin + u;
        const bool in = u < nsteps && xl < W;
        load_row(rin[g], e_row + g * e_pitch, in && r >= 0 && r < H);
        load_row(rout[g], e_row + g * e_pitch - e_back, in && u >= th && r >= th && r - th < H);
      }
      e_row += BS * e_pitch;
    }
    constexpr int NBLK = SPLIT ? 2 : kU8Chunks;
    const bool ok = mbar_wait(&blk_full[k % NBLK], (k / NBLK) & 1, abort_flag, kSpinLimit);
    // tcgen05.ld/st are warp-collective: the whole warp takes one branch.
    if (!__all_sync(0xffffffffu, ok)) break;
    tc_fence_after();
    AT val[8];
    if constexpr (SPLIT) {
      const uint32_t part = lane_base + (k & 1) * kPartCols + half * kHalf;
      // Chunk 0 of the partial completes the BS slots t0 .. t0 + BS - 1; chunk c
      // belongs to the open sums c - 1 of the next block (the sums move down a
      // chunk as they are added to). Three chunks are in flight together.
      auto chunks = [&](auto first) {
        constexpr int C0 = decltype(first)::value, N = 3;
        uint32_t vp[N][8];
#pragma unroll
        for (int c = 0; c < N; ++c) tmem_ld8x(part + 8 * (C0 + c), vp[c]);
        tmem_ld_wait();
#pragma unroll
        for (int c = 0; c < N; ++c)
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const AT old = C0 + c < kRingChunks ? ring[(C0 + c) % kRingChunks][j] : AT(0);
            const AT v = __fadd_rn(old, __uint_as_float(vp[c][j]));
            if (C0 + c == 0)
              val[j] = v;
            else
              ring[(C0 + c + kRingChunks - 1) % kRingChunks][j] = v;
          }
      };
      chunks(std::integral_constant<int, 0>());
      chunks(std::integral_constant<int, 3>());
      chunks(std::integral_constant<int, 6>());
      // The partial has been read: the MMAs may refill it (block k + 2).
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&buf_free[k & 1]);
    } else {
      // The chunk of the block's BS completed slots, column S g + p; this warp
      // takes its half of the positions and clears those columns for the slots
      // 512 / S later.
      const uint32_t chunk = lane_base + 16 * (k % kU8Chunks);
      uint32_t v[16];
      tmem_ld16x(chunk, v);
      tmem_ld_wait();
#pragma unroll
      for (int g = 0; g < BS; ++g) {
#pragma unroll
        for (int p = 0; p < SH; ++p)
          val[g * SH + p] = static_cast<int>(half ? v[S * g + SH + p] : v[S * g + p]);
        tmem_st_zero<SH>(chunk + S * g + SH * half);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&buf_free[(k / kU8Group) % kU8Groups]);
    }
    if constexpr (kAhead) {
      cp_async_wait<kU8Ahead - 1>();
#pragma unroll
      for (int g = 0; g < BS; ++g) {
        memcpy(rin[g], __builtin_assume_aligned(slot_of(k, g), 4 * SH), 4 * SH);
        memcpy(rout[g], __builtin_assume_aligned(slot_of(k, BS + g), 4 * SH), 4 * SH);
      }
      __syncwarp();
    }
    if (kE && !kAhead) {
      // The loaded energies are first used here: without this the compiler
      // converts them where they were loaded, and waits for the loads there
      // (about 900 cycles a step).
#pragma unroll
      for (int g = 0; g < BS; ++g)
#pragma unroll
        for (int p = 0; p < SH; ++p) asm volatile("" : "+r"(rin[g][p]), "+r"(rout[g][p]));
    }
    // The block's completed slots: window energies, scores and stores.
    const bool rows = t0 >= R - 1 && t0 + BS <= nsteps;  // every slot is an output row
    if (f32 && rows) {
      // Straight-line independent work.
      float out[8];
      ET es[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int g = i / SH, p = i % SH;
        if (kE) add_energy(g, p);
        es[i] = esum[p];
      }
      scores8<SPLIT, M>(out, val, es, etd, ret, u8_float);
      if (M == kCrossCorr && raw) {
#pragma unroll
        for (int i = 0; i < 8; ++i) out[i] = __int_as_float(static_cast<int>(val[i]));
      }
#pragma unroll
      for (int g = 0; g < BS; ++g) {
        if (IDX && idx_op >= 0) {
#pragma unroll
          for (int p = 0; p < SH; ++p)
            if (xl + p < W)
              idx_state_update(ib, out[g * SH + p], xl + p, a.y0 + t0 + g - R + 1, idx_op, idx_ngx);
        }
        if (IDX && !has_dst) {
        } else if (!whole || nch > 1) {
          float* o = reinterpret_cast<float*>(orow) + (size_t)xl * nch + a.dst_ch;
#pragma unroll
          for (int p = 0; p < SH; ++p)
            if (xl + p < W) o[p * nch] = out[g * SH + p];
        } else {
          float* o = reinterpret_cast<float*>(orow) + xl;
          if (SH == 4)
            *reinterpret_cast<float4*>(o) =
                make_float4(out[g * SH], out[(g * SH + 1) % 8], out[(g * SH + 2) % 8],
                            out[(g * SH + 3) % 8]);
          else if (SH == 2)
            *reinterpret_cast<float2*>(o) = make_float2(out[g * SH], out[(g * SH + 1) % 8]);
          else
            o[0] = out[g];
        }
        orow += dst_pitch;
      }
    } else {
#pragma unroll
      for (int g = 0; g < BS; ++g) {
        const int u = t0 + g;
        if (kE) {
#pragma unroll
          for (int p = 0; p < SH; ++p) add_energy(g, p);
        }
        if (u >= R - 1 && u < nsteps && xl < W) {
          // (Copies: arrays whose address a call takes live in local memory.)
          float v[SH];
          AT cv[SH];
          ET ev[SH];
#pragma unroll
          for (int p = 0; p < SH; ++p) {
            cv[p] = val[g * SH + p];
            ev[p] = esum[p];
          }
          store_slot<ELEM, SH, M>(a, xl, orow, cv, ev, etd, v);
          if (IDX && idx_op >= 0) {
#pragma unroll
            for (int p = 0; p < SH; ++p)
              if (xl + p < W)
                idx_state_update(ib, v[p], xl + p, a.y0 + u - R + 1, idx_op, idx_ngx);
          }
        }
        orow += dst_pitch;
      }
    }
  }
  if (kAhead) cp_async_wait<0>();  // none is left in flight after a wait that gave up
  if (IDX && idx_op >= 0) {
    // The warp's best: same rule, then lane 0 writes the warp's record.
    const bool is_min = idx_op == 0 || idx_op == 2;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, ib.v, d);
      const unsigned long long ok2 = __shfl_xor_sync(0xffffffffu, ib.key, d);
      const int oh = __shfl_xor_sync(0xffffffffu, ib.have, d);
      ib.nan |= __shfl_xor_sync(0xffffffffu, ib.nan, d);
      const bool take = oh && (!ib.have || (is_min ? ov < ib.v : ov > ib.v) ||
                               (ov == ib.v && ok2 < ib.key));
      if (take) {
        ib.v = ov;
        ib.key = ok2;
        ib.have = 1;
      }
    }
    if (lane == 0) {
      const int item = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
      IdxRecord r;
      r.v = ib.v;
      r.have = ib.have;
      r.key = ib.key;
      r.nan = ib.nan;
      r.pad = 0;
      reinterpret_cast<IdxRecord*>(a.idx_out)[item * kEpilogue + ew] = r;
    }
  }
}

// Runs one work item with all 12 warps of the CTA. The caller has
// synchronised the CTA; TMEM (512 columns) is allocated. Barriers are
// initialised here and invalidated at the end, so consecutive items may use
// different layouts.
template <int ELEM, int S, bool IDX>
__device__ __forceinline__ void run_item(const ItemArgs& a, unsigned char* smem, CtaState& cs) {
  typedef ElemTraits<ELEM> TR;
  constexpr bool SPLIT = TR::split;
  constexpr int R = kSR / S;
  constexpr int BS = block_steps(S);
  constexpr int CMK = TR::cmk;
  constexpr int NR = TR::raw;
  constexpr int AB = TR::ab;
  constexpr int SH = S / 2;             // positions of a half
  static_assert(SH * BS == 8, "a half's completed slots of a block are one chunk");
  static_assert(SH * (BS + R - 1) <= kHalf, "a block's open slots do not fit the partial");
  const int lead = (TR::inner - a.ax % TR::inner) % TR::inner;
  const Geo G = make_geo(SPLIT, R, a.tw, lead);
  const Layout L = make_layout(SPLIT, G, a.nbox);

  uint64_t* raw_full = reinterpret_cast<uint64_t*>(smem + L.bars);
  // Block k's A stages (k mod AB) hold its rows; its MMAs have completed, so
  // the builders may refill them (block k + AB).
  uint64_t* ready = raw_full + kMaxRaw;
  uint64_t* a_free = ready + kMaxAB;
  uint64_t* blk_full = a_free + kMaxAB;    // block's MMAs complete (a buffer or chunk each)
  uint64_t* buf_free = blk_full + kMaxBlk;  // block's buffer read by the epilogue; U8: the
                                            // chunks of a group of 8 blocks read and cleared
  uint64_t* done_bar = buf_free + kU8Groups;
  constexpr int NBLK = SPLIT ? 2 : kU8Chunks, NFREE = SPLIT ? 2 : kU8Groups;
  volatile int* abort_flag = &cs.abort;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int ch = a.ch;
  const int r_begin = a.y0 - a.ay - (R - a.th);
  const int nsteps = (a.yend - a.y0) + R - 1;
  const int nblk = (nsteps + BS - 1) / BS;

  if (threadIdx.x == 0) {
    for (int i = 0; i < NR; ++i) mbar_init(&raw_full[i], 1);
    for (int i = 0; i < AB; ++i) {
      mbar_init(&ready[i], BS);
      mbar_init(&a_free[i], 1);
    }
    for (int i = 0; i < NBLK; ++i) mbar_init(&blk_full[i], 1);
    for (int i = 0; i < NFREE; ++i) mbar_init(&buf_free[i], SPLIT ? kEpilogue : kEpilogue * kU8Group);
    mbar_init(done_bar, 1);
    fence_barrier_init();
  }

  // The template is staged once (at the A stages, which nothing uses yet): row
  // h holds elements T(i - o, h) at i, zero outside the template, as BF16 hi
  // and lo (split) or bytes. All loads of a group of kTmplBatch are in flight
  // together, and each thread squares what it loads for the template energy:
  // gathering B's elements and the energy straight from global memory, one
  // dependent load after another, took 25-30 us of every launch.
  const int o = S - 1 + lead;
  const int tpitch = G.KC * CMK + o;
  const int tplane = (a.th * tpitch + 7) & ~7;  // elements of one staged array
  {
    double e = 0.0;
    const int total = a.th * tpitch;
    for (int base = threadIdx.x; base < total; base += kTmplBatch * kThreads) {
      float v[kTmplBatch];
#pragma unroll
      for (int u = 0; u < kTmplBatch; ++u) {
        const int idx = base + u * kThreads;
        const int h = idx / tpitch, w = idx - h * tpitch - o;
        v[u] = (idx < total && w >= 0 && w < a.tw) ? tmpl_at<ELEM>(a, h, w, ch) : 0.f;
      }
#pragma unroll
      for (int u = 0; u < kTmplBatch; ++u) {
        const int idx = base + u * kThreads;
        if (idx >= total) break;
        e = fma((double)v[u], (double)v[u], e);
        if (SPLIT) {
          const __nv_bfloat16 hi = __float2bfloat16_rn(v[u]);
          __nv_bfloat16* st = reinterpret_cast<__nv_bfloat16*>(smem + L.a);
          st[idx] = hi;
          st[tplane + idx] = __float2bfloat16_rn(v[u] - __bfloat162float(hi));
        } else {
          smem[L.a + idx] = static_cast<uint8_t>(v[u]);
        }
      }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) e += __shfl_xor_sync(0xffffffffu, e, d);
    if (lane == 0) cs.et[warp] = e;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  // Loads of row t into its stage, by the builder that owns it (one lane).
  auto load_stage = [&](int t) {
    const int st = t % NR, part = box_part(a.nbox), nsplit = box_split(a.nbox);
    const int gx = (a.xs_out - a.ax - lead) / TR::inner;  // exact: a multiple of inner
    mbar_arrive_expect_tx(&raw_full[st], L.row_bytes);
    for (int j = 0; j < nsplit; ++j)
      tma_load_4d(smem + L.raw + st * L.raw_stage + j * part * 16, a.tmap, 0, gx + j * part,
                  r_begin + t, ch, &raw_full[st]);
  };
  if (warp < kBuilders && lane == 0) {
    tma_prefetch_desc(a.tmap);
    for (int t = warp; t < min(NR, nsteps); t += kBuilders) load_stage(t);
  }
  {
    // Template operand B: per core matrix (two per MMA, in issue order) NB rows
    // of 16 bytes, a thread per row; rows zp .. zp + 63 hold the first half of the positions,
    // rows zp + 72 .. zp + 135 the second, the rest are zero.
    // U8: rows zp + S j + p, slot after slot.
    constexpr int zp = SPLIT ? 8 - SH : 16 - S;
    constexpr int NB = kNp + zp;
    const int total = 2 * G.nmma * NB;
    for (int idx = threadIdx.x; idx < total; idx += kThreads) {
      const int cm = idx / NB, r = idx - cm * NB - zp;
      const int half = SPLIT && r >= kHalf;
      const int n = r - half * kHalf;        // row of its half (U8: of all)
      constexpr int rows = SPLIT ? SH : S;   // rows of a slot
      // Which part (0 zero, 1 Thi, 2 Tlo; U8: 1) and which K chunk.
      int part, c;
      if (SPLIT) {
        const int j = cm >> 1, half = cm & 1;
        if (j < G.KC) {
          c = j;
          part = half ? 1 : 2;  // (hi_c, lo_c) x (Tlo_c, Thi_c)
        } else {
          c = 2 * (j - G.KC) + half;
          part = c < G.KC ? 1 : 0;
        }
      } else {
        c = cm;
        part = c < G.KC ? 1 : 0;
      }
      const int h = a.th - 1 - n / rows;
      uint4 q = make_uint4(0u, 0u, 0u, 0u);
      if (part && n >= 0 && n < (SPLIT ? kHalfN : kN) && h >= 0) {
        // Elements w = c CMK - p - lead .. + CMK - 1 of template row h.
        const int at = h * tpitch + c * CMK + S - 1 - (half * SH + n % rows);
        uint32_t w4[4];
        if (SPLIT) {
          const uint16_t* st =
              reinterpret_cast<const uint16_t*>(smem + L.a) + (part == 2 ? tplane : 0) + at;
#pragma unroll
          for (int j = 0; j < 4; ++j) w4[j] = st[2 * j] | (uint32_t)st[2 * j + 1] << 16;
        } else {
          const uint8_t* st = smem + L.a + at;
#pragma unroll
          for (int j = 0; j < 4; ++j)
            w4[j] = st[4 * j] | (uint32_t)st[4 * j + 1] << 8 | (uint32_t)st[4 * j + 2] << 16 |
                    (uint32_t)st[4 * j + 3] << 24;
        }
        q = make_uint4(w4[0], w4[1], w4[2], w4[3]);
      }
      *reinterpret_cast<uint4*>(smem + L.b + idx * 16) = q;
    }
    if constexpr (!SPLIT) {
      // Every MMA accumulates: the ring of sums starts at zero (each epilogue warp
      // clears half of the columns of its lanes).
      if (warp >= kFirstEpilogue) {
        const int ew = warp - kFirstEpilogue;
        const uint32_t at = cs.tmem + (static_cast<uint32_t>((ew & 3) * 32) << 16) + (ew >> 2) * 256;
        uint32_t zero[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) zero[i] = 0u;
#pragma unroll 4
        for (int i = 0; i < 256; i += 16) tmem_st16(at + i, zero);
        tmem_st_wait();
      }
    }
    // B is complete, and the staged template read, for the MMA and builder warps.
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
  }
  const uint32_t tmem_base = cs.tmem;

  if (warp == kMmaWarp) {
    // ---- MMA issue --------------------------------------------------------------
    // The whole warp walks the blocks on warp-uniform values (taken from lane 0)
    // and one elected lane issues. An MMA of N = 144 takes the tensor pipe 72
    // cycles (N / 2), and the pipe queues only two or three, so what the issuing
    // lane does between MMAs counts: with the lane alone in a divergent branch,
    // a wait per step and descriptors in per-lane registers an MMA went out
    // every 95-130 cycles; this form measured 73-76 (steps of 8 MMAs).
    {
      const uint32_t idesc = idesc_bf16_f32(kM, kNp);
      auto uniform = [](uint32_t v) { return __shfl_sync(0xffffffffu, v, 0); };
      const uint32_t tm = uniform(tmem_base);
      const uint32_t a0 = uniform(smem_u32(smem + L.a));
      const uint32_t b0 = uniform(smem_u32(smem + L.b));
      const uint32_t bstride = G.NB * 16;  // between B core matrices
      const uint32_t dhi = desc_hi(128);   // every descriptor: SBO 128 bytes
      const uint32_t astep = uniform(G.lbok >> 4), bstep = (2 * bstride) >> 4;  // 16-byte units
      const int a_stage = uniform(L.a_stage), a_hl = uniform(G.QR * 16), lbok = uniform(G.lbok);
      const int kc = uniform(G.KC), nmma = uniform(G.nmma), nst = uniform(nsteps),
                nb = uniform(nblk);
      const bool issuer = elect_one();
      for (int k = 0; k < nb; ++k) {
        // The buffer of block k was read by the epilogue (block k - 2). U8: the chunks
        // that the next 8 blocks' windows reach for the first time were cleared (the
        // blocks 24 to 17 back).
        bool ok = true;
        if (SPLIT) {
          ok = k < 2 || mbar_wait(&buf_free[k & 1], ((k >> 1) - 1) & 1, abort_flag, kSpinLimit);
        } else if (k % kU8Group == 0 && k >= 3 * kU8Group) {
          const int g = k / kU8Group - 3;
          ok = mbar_wait(&buf_free[g % kU8Groups], (g / kU8Groups) & 1, abort_flag, kSpinLimit);
        }
        ok = ok && mbar_wait(&ready[k % AB], (k / AB) & 1, abort_flag, kSpinLimit);
        if (!__all_sync(0xffffffffu, ok)) break;
        tc_fence_after();
        const uint32_t d = tm + (k & 1) * kPartCols;  // the block's partial
        // U8: its window of the ring, in two parts where it wraps.
        const int c0 = k % kU8Chunks, n1 = min(kU8Window, kU8Chunks - c0);
        const uint32_t id1 = idesc_u8_s32(kM, 16 * n1), id2 = idesc_u8_s32(kM, kNp - 16 * n1);
        if (issuer) {
#pragma unroll
          for (int q = 0; q < BS; ++q) {
            if (k * BS + q < nst) {
              const uint32_t ah = a0 + ((k % AB) * BS + q) * a_stage;
              // Descriptors advance by one add of their low word per MMA: B by
              // two core matrices, A by one (split, hi/lo pairs) or two K core
              // matrices. The block's first MMA overwrites all kNp columns.
              uint32_t bl = desc_lo(b0 + 16 * (SPLIT ? SH : S) * (BS - 1 - q), bstride);
              uint32_t acc = q == 0 ? 0u : 1u;
              if (SPLIT) {
                uint32_t al = desc_lo(ah, a_hl);
                for (int c = 0; c < kc; ++c) {
                  mma_bf16_h(d, al, dhi, bl, dhi, idesc, acc);
                  acc = 1u;
                  al += astep;
                  bl += bstep;
                }
                al = desc_lo(ah, lbok);
                for (int j = kc; j < nmma; ++j) {
                  mma_bf16_h(d, al, dhi, bl, dhi, idesc, 1u);
                  al += 2 * astep;
                  bl += bstep;
                }
              } else {
                (void)acc;
                uint32_t al = desc_lo(ah, lbok);
                for (int j = 0; j < nmma; ++j) {
                  mma_i8_h(tm + 16 * c0, al, dhi, bl, dhi, id1, 1u);
                  if (n1 < kU8Window) mma_i8_h(tm, al, dhi, bl + 16 * n1, dhi, id2, 1u);
                  al += 2 * astep;
                  bl += bstep;
                }
              }
            }
          }
          // The block's partial for the epilogue, its A stages for the builders.
          mma_commit(&blk_full[k % NBLK]);
          // (The last blocks' stages are not refilled: no arrival is left pending.)
          if (k + AB < nb) mma_commit(&a_free[k % AB]);
        }
        __syncwarp();
      }
      // Every MMA issued has completed before the item ends.
      if (issuer) mma_commit(done_bar);
      __syncwarp();
      volatile int no_abort = 0;
      mbar_wait(done_bar, 0, &no_abort, kSpinLimit);
    }
  } else if (warp < kBuilders) {
    // ---- Builders: A operand ------------------------------------------------------
    // One warp per row, so that three rows are in flight: the waits, shared-memory
    // round trips and proxy fence of a row are a chain of hundreds of cycles.
    // The warp that has read a staged row loads the stage's next one.
    // Rows past the last step only arrive (a block completes with BS arrivals).
    int t = warp;
    for (; t < nblk * BS; t += kBuilders) {
      const int kb = t / BS, st = t % NR, i = t % (AB * BS);
      bool ok = kb < AB || mbar_wait(&a_free[kb % AB], (kb / AB - 1) & 1, abort_flag, kSpinLimit);
      ok = ok && (t >= nsteps || mbar_wait(&raw_full[st], (t / NR) & 1, abort_flag, kSpinLimit));
      if (!__all_sync(0xffffffffu, ok)) break;
      if (t >= nsteps) {
        if (lane == 0) mbar_arrive(&ready[kb % AB]);
        continue;
      }
      const unsigned char* row = smem + L.raw + st * L.raw_stage;
      unsigned char* ahi = smem + L.a + i * L.a_stage;
      if constexpr (SPLIT) {
        // Row q is the S pixels of "lane" q and of the 8 / S - 1 after it. Each
        // pixel is read and split once (the MMAs use 120 of the 128 bytes a
        // cycle that shared memory gives); rows take their neighbours'
        // pixels by shuffles.
        constexpr int NG = (kM + 31) / 32 + (S == 2 ? 2 : 1);  // row groups: QR <= 164, 160
        constexpr int NL = NG + (S == 4 ? 1 : 0);              // pixel groups
        constexpr int SP = S / 2;                              // packed pairs a lane reads
        const int qlast = G.QR + 8 / S - 2;                    // last pixel group of a row
        uint32_t hi[NL][SP], lo[NL][SP];
#pragma unroll
        for (int j = 0; j < NL; ++j) {
          float f[S];
          load_s<ELEM, S>(row, S * min(lane + 32 * j, qlast), f);
#pragma unroll
          for (int i = 0; i < SP; ++i) {
            hi[j][i] = pack_bf16(f[2 * i], f[2 * i + 1]);
            lo[j][i] = pack_bf16(f[2 * i] - bf16lo_f(hi[j][i]), f[2 * i + 1] - bf16hi_f(hi[j][i]));
          }
        }
#pragma unroll
        for (int j = 0; j < NG; ++j) {
          uint32_t h4[4], l4[4];
#pragma unroll
          for (int d = 0; d < 8 / S; ++d)
#pragma unroll
            for (int i = 0; i < SP; ++i) {
              if (d == 0) {
                h4[i] = hi[j][i];
                l4[i] = lo[j][i];
              } else {
                // Lane + d: of this group, or of the next one past lane 31.
                const int jn = j + 1 < NL ? j + 1 : j;
                const int from = (lane + d) & 31;
                h4[d * SP + i] = __shfl_sync(0xffffffffu, lane < d ? hi[jn][i] : hi[j][i], from);
                l4[d * SP + i] = __shfl_sync(0xffffffffu, lane < d ? lo[jn][i] : lo[j][i], from);
              }
            }
          const int q = lane + 32 * j;
          if (q < G.QR) {
            *reinterpret_cast<uint4*>(ahi + q * 16) = make_uint4(h4[0], h4[1], h4[2], h4[3]);
            *reinterpret_cast<uint4*>(ahi + G.QR * 16 + q * 16) =
                make_uint4(l4[0], l4[1], l4[2], l4[3]);
          }
        }
      } else {
        // Bytes S q .. S q + 15 (S q is a multiple of 4 when S is).
        constexpr int NW = S % 4 == 0 ? 4 : 5;
        auto get = [&](int q, uint32_t (&w)[NW]) {
          const uint32_t* w32 = reinterpret_cast<const uint32_t*>(row + ((S * q) & ~3));
#pragma unroll
          for (int j = 0; j < NW; ++j) w[j] = w32[j];
        };
        auto put = [&](int q, const uint32_t (&w)[NW]) {
          const uint32_t sh = ((S * q) & 3) * 8;
          uint32_t v[4];
#pragma unroll
          for (int j = 0; j < 4; ++j)
            v[j] = S % 4 == 0 ? w[j] : __funnelshift_r(w[j], w[(j + 1) % NW], sh);
          *reinterpret_cast<uint4*>(ahi + q * 16) = make_uint4(v[0], v[1], v[2], v[3]);
        };
        uint32_t w[kM / 32][NW];
#pragma unroll
        for (int j = 0; j < kM / 32; ++j) get(lane + 32 * j, w[j]);
#pragma unroll
        for (int j = 0; j < kM / 32; ++j) put(lane + 32 * j, w[j]);
        for (int q = kM + lane; q < G.QR; q += 32) {
          get(q, w[0]);
          put(q, w[0]);
        }
      }
      fence_async_smem();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&ready[kb % AB]);
        if (t + NR < nsteps) load_stage(t + NR);
      }
    }
    // After a wait that gave up: every load issued lands before the item ends.
    if (lane == 0) {
      volatile int no_abort = 0;
      for (int r = t; r < min(t + NR, nsteps); r += kBuilders)
        mbar_wait(&raw_full[r % NR], (r / NR) & 1, &no_abort, kSpinLimit);
    }
  } else {
    // ---- Epilogue ---------------------------------------------------------------
    const uint32_t tm = tmem_base;
    switch (a.measure) {
      case kSqrDistance:
        run_epilogue<ELEM, S, IDX, kSqrDistance>(a, cs, tm, blk_full, buf_free, r_begin, nsteps,
                                                smem + L.energies);
        break;
      case kSqrDistanceNorm:
        run_epilogue<ELEM, S, IDX, kSqrDistanceNorm>(a, cs, tm, blk_full, buf_free, r_begin,
                                                     nsteps, smem + L.energies);
        break;
      case kCrossCorrNorm:
        run_epilogue<ELEM, S, IDX, kCrossCorrNorm>(a, cs, tm, blk_full, buf_free, r_begin, nsteps,
                                                   smem + L.energies);
        break;
      default:
        run_epilogue<ELEM, S, IDX, kCrossCorr>(a, cs, tm, blk_full, buf_free, r_begin, nsteps,
                                                smem + L.energies);
        break;
    }
  }

  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (threadIdx.x == 0) {
    for (int i = 0; i < NR; ++i) mbar_inval(&raw_full[i]);
    for (int i = 0; i < AB; ++i) {
      mbar_inval(&ready[i]);
      mbar_inval(&a_free[i]);
    }
    for (int i = 0; i < NBLK; ++i) mbar_inval(&blk_full[i]);
    for (int i = 0; i < NFREE; ++i) mbar_inval(&buf_free[i]);
    mbar_inval(done_bar);
  }
}

// Template classes: R in {16, 32, 64} (template rows rounded up); the strip
// width is 128 S positions.
inline int class_of(int th) { return th <= 16 ? 0 : th <= 32 ? 1 : 2; }
__host__ __device__ inline int class_r(int cls) { return 16 << cls; }
template <int ELEM>
int strip_width(int cls) {
  return kM * s_for(class_r(cls));
}

template <int ELEM, bool IDX>
__device__ __forceinline__ void dispatch(const ItemArgs& a, unsigned char* smem, CtaState& cs) {
  if (a.R == 16)
    run_item<ELEM, 8, IDX>(a, smem, cs);
  else if (a.R == 32)
    run_item<ELEM, 4, IDX>(a, smem, cs);
  else
    run_item<ELEM, 2, IDX>(a, smem, cs);
}

// Batch tables (device memory).
struct BatchImage {
  int W, H, nch;
};
struct BatchTemplate {
  const char* ptr;
  size_t pitch;
  int tw, th, cls;  // cls: template rows class (R = 16 << cls)
};
struct BatchDest {
  char* ptr;
  size_t pitch;
  int f64;
};
struct BatchItem {
  int img, tpl, dst;  // indices into the tables
  int energy;         // index into the energy maps, -1 for CrossCorr
  int ch, strip, y0, yend;
};
// Window-energy map of one (image, template size) pair of a batch.
struct BatchEnergy {
  const char* ptr;
  size_t pitch, plane;
};

// A tile of a template larger than 64 x 64.
struct TemplateTile {
  const char* tmpl;
  int tw, th, ax, ay;
};
constexpr int kMaxTiles = 16;  // of one launch

struct TensorLaunch {
  CUtensorMap map;     // single-image mode: the source planes
  int mode;            // 0: one (image, template) pair, items from blockIdx; 1: work queue
  int measure;
  int nbox;            // 16-byte groups per staged row (all tensor maps of the launch)
  int* err;
  // mode 0
  unsigned* ticket;    // best match: CTAs done (0 between launches)
  Context::HostPage::Index* index;  // and its result
  ItemArgs base;       // fields common to every item
  int BH;
  int ntiles;          // > 0: CTA z = (tile, channel), each with its own map of product sums
  size_t tile_plane;   // bytes between those maps (base.dst)
  TemplateTile tiles[kMaxTiles];
  // mode 1
  const CUtensorMap* maps;  // one per image (64-byte aligned)
  const BatchImage* imgs;
  const BatchTemplate* tpls;
  const BatchDest* dsts;
  const BatchItem* items;
  const BatchEnergy* energies;
  int nitems;
  int* counter;        // next item; reset to 0 before every launch
};

// Best match: the last CTA to finish folds every CTA's records (each value with
// the smallest key among equals, so the order does not matter) into the host's
// result.
__device__ void fold_records(const TensorLaunch& P) {
  __shared__ bool last;
  __shared__ IdxRecord part[kWarps];
  const unsigned ncta = gridDim.x * gridDim.y * gridDim.z;
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(P.ticket, 1u) == ncta - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  const bool is_min = P.base.idx_op == 0 || P.base.idx_op == 2;
  auto better = [&](float v, unsigned long long key, int have, const IdxRecord& r) {
    return have && (!r.have || (is_min ? v < r.v : v > r.v) || (v == r.v && key < r.key));
  };
  IdxRecord best;
  best.v = 0.f;
  best.key = 0ull;
  best.have = best.nan = best.pad = 0;
  const IdxRecord* rec = reinterpret_cast<const IdxRecord*>(P.base.idx_out);
  for (unsigned i = threadIdx.x; i < ncta * kEpilogue; i += kThreads) {
    const float v = __ldcg(&rec[i].v);
    const unsigned long long key = __ldcg(&rec[i].key);
    const int have = __ldcg(&rec[i].have);
    best.nan |= __ldcg(&rec[i].nan);
    if (better(v, key, have, best)) {
      best.v = v;
      best.key = key;
      best.have = 1;
    }
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    const float v = __shfl_xor_sync(0xffffffffu, best.v, d);
    const unsigned long long key = __shfl_xor_sync(0xffffffffu, best.key, d);
    const int have = __shfl_xor_sync(0xffffffffu, best.have, d);
    best.nan |= __shfl_xor_sync(0xffffffffu, best.nan, d);
    if (better(v, key, have, best)) {
      best.v = v;
      best.key = key;
      best.have = 1;
    }
  }
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = best;
  __syncthreads();
  if (threadIdx.x != 0) return;
  for (int w = 1; w < kWarps; ++w) {
    best.nan |= part[w].nan;
    if (better(part[w].v, part[w].key, part[w].have, best)) best = IdxRecord{part[w].v, 1, part[w].key, best.nan, 0};
  }
  // Key -> pixel: group, bit-reversed work-item id, pixel index in the work-item.
  const unsigned long long grp = best.key >> 12;
  const unsigned lid = __brev((unsigned)(best.key >> 4) & 255u) >> 24;
  const int ngx = (P.base.W + 255) >> 8;
  volatile Context::HostPage::Index* out = P.index;
  out->v = best.v;
  out->x = (int)(grp % ngx) * 256 + (int)(lid & 15) + 16 * (int)(best.key & 15);
  out->y = (int)(grp / ngx) * 16 + (int)(lid >> 4);
  out->nan = best.nan || !best.have;
  __threadfence_system();
  *P.ticket = 0;
}

// One kernel per element type. Mode 0 (one image and template): CTA
// (x, y, z) = (strip, band, channel). Mode 1 (batch): one persistent CTA per
// SM takes items from a global counter until none are left.
template <int ELEM, bool IDX = false>
__global__ void __launch_bounds__(kThreads, 1)
    prox_tensor_kernel(const __grid_constant__ TensorLaunch P) {
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ CtaState cs;
  const int warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) cs.abort = 0;
  if (warp == 0) tmem_alloc(&cs.tmem, kTmemCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();

  // The item's arguments live in shared memory: read where they are used,
  // they take no registers from the roles' accumulators.
  __shared__ ItemArgs item;
  if (P.mode == 0) {
    if (threadIdx.x == 0) {
      item = P.base;
      item.tmap = &P.map;
      item.ch = item.dst_ch = blockIdx.z;
      if (P.ntiles > 0) {
        const TemplateTile t = P.tiles[blockIdx.z / item.nch];
        item.ch = blockIdx.z % item.nch;
        item.dst_ch = 0;
        item.dst += blockIdx.z * P.tile_plane;
        item.tmpl = t.tmpl;
        item.tw = t.tw;
        item.th = t.th;
        item.ax = t.ax;
        item.ay = t.ay;
      }
      item.xs_out = blockIdx.x * kM * s_for(item.R);
      item.y0 = blockIdx.y * P.BH;
      item.yend = min(item.H, item.y0 + P.BH);
    }
    __syncthreads();
    dispatch<ELEM, IDX>(item, smem, cs);
  } else {
    for (;;) {
      if (threadIdx.x == 0) {
        const int it = cs.abort ? P.nitems : atomicAdd(P.counter, 1);
        cs.next = it;
        if (it < P.nitems) {
          const BatchItem bi = P.items[it];
          const BatchImage im = P.imgs[bi.img];
          const BatchTemplate tp = P.tpls[bi.tpl];
          const BatchDest ds = P.dsts[bi.dst];
          item.tmap = P.maps + bi.img;
          item.W = im.W;
          item.H = im.H;
          item.tw = tp.tw;
          item.th = tp.th;
          item.R = class_r(tp.cls);
          item.ax = tp.tw / 2;
          item.ay = tp.th / 2;
          item.nch = im.nch;
          item.ch = bi.ch;
          item.xs_out = bi.strip * kM * s_for(item.R);
          item.y0 = bi.y0;
          item.yend = bi.yend;
          item.nbox = P.nbox;
          item.tmpl = tp.ptr;
          item.tmpl_pitch = tp.pitch;
          item.dst = ds.ptr;
          item.dst_pitch = ds.pitch;
          item.dst_f64 = ds.f64;
          item.measure = P.measure;
          item.dst_nch = im.nch;
          item.dst_ch = bi.ch;
          item.raw = 0;
          item.idx_op = -1;
          item.idx_out = nullptr;
          item.energy = nullptr;
          item.e_pitch = item.e_plane = 0;
          if (bi.energy >= 0) {
            const BatchEnergy be = P.energies[bi.energy];
            item.energy = be.ptr;
            item.e_pitch = be.pitch;
            item.e_plane = be.plane;
          }
        }
      }
      __syncthreads();
      const int it = cs.next;
      if (it >= P.nitems) break;
      dispatch<ELEM, IDX>(item, smem, cs);
      __syncthreads();  // every thread has read the item before it is replaced
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(cs.tmem, kTmemCols);
  }
  if (threadIdx.x == 0 && cs.abort) {
    *reinterpret_cast<volatile int*>(P.err) = 1;
    __threadfence_system();
  }
  if (IDX) fold_records(P);
}

// Interleaved channels -> planes: plane c holds channel c of every pixel, rows
// at `plane_pitch`, planes `plane_bytes` apart. Columns W .. pw - 1 (the pitch
// tail, which the TMA view reads in whole 16-byte groups) are written as zeros.
template <typename T>
__global__ void split_channels_kernel(const char* src, size_t src_pitch, char* planes,
                                      size_t plane_pitch, size_t plane_bytes, int W, int pw,
                                      int H, int nch) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int y = blockIdx.y;
  if (x >= pw || y >= H) return;
  const T* s = reinterpret_cast<const T*>(src + (size_t)y * src_pitch) + (size_t)x * nch;
  for (int c = 0; c < nch; ++c)
    reinterpret_cast<T*>(planes + c * plane_bytes + (size_t)y * plane_pitch)[x] =
        x < W ? s[c] : T(0);
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(f);
  }
  return fn;
}

// Band height: the fewest waves of CTAs times the steps per band (output
// rows plus the R - 1 rows of ramp), over all band counts.
int band_height(int H, int R, long long columns, int sm_count) {
  long long best = LLONG_MAX;
  int best_bh = H;
  for (int nb = 1; nb <= std::max(1, H / 8); ++nb) {
    const int bh = (H + nb - 1) / nb;
    const int nbe = (H + bh - 1) / bh;
    const long long waves = (columns * nbe + sm_count - 1) / sm_count;
    const long long cost = waves * (bh + R - 1);
    if (cost < best) {
      best = cost;
      best_bh = bh;
    }
  }
  return best_bh;
}

// Lead of the staged row (elements before the first window pixel, so that
// the TMA copy starts on a 16-byte group).
template <int ELEM>
int lead_for(int ax) {
  const int inner = ElemTraits<ELEM>::inner;
  return (inner - ax % inner) % inner;
}

template <int ELEM>
Geo geo_for(int cls, int tw, int ax) {
  return make_geo(ElemTraits<ELEM>::split, class_r(cls), tw, lead_for<ELEM>(ax));
}

// 16-byte groups a staged row needs for a template of this class and width.
template <int ELEM>
int nbox_for(int cls, int tw, int ax) {
  typedef ElemTraits<ELEM> TR;
  const Geo g = geo_for<ELEM>(cls, tw, ax);
  return (staged_elems(g, TR::split) + TR::inner - 1) / TR::inner;
}

template <int ELEM>
int smem_for(int cls, int tw, int ax, int nbox) {
  return std::max(make_layout(ElemTraits<ELEM>::split, geo_for<ELEM>(cls, tw, ax), nbox).total,
                  kMinSmem);
}

// Rank-4 view of source planes: 16-byte groups (dim 0), groups along the row
// (dim 1), rows (dim 2), channels (dim 3). A staged row (the strip plus the
// template width, nbox groups) is box_split(nbox) boxes of box_part(nbox)
// groups and one row. The last group of a row may reach into the row pitch,
// which is zero (image creation zero-fills device buffers; the channel split
// writes zeros there).
template <int ELEM>
cudaError_t encode_planes(CUtensorMap* map, const void* planes, int W, int H, int nch,
                          size_t plane_pitch, size_t plane_bytes, int nbox) {
  typedef ElemTraits<ELEM> TR;
  EncodeTiledFn enc = encode_fn();
  if (!enc) return cudaErrorNotSupported;
  const CUtensorMapDataType dt = ELEM == kF32   ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32
                                 : ELEM == kU16 ? CU_TENSOR_MAP_DATA_TYPE_UINT16
                                                : CU_TENSOR_MAP_DATA_TYPE_UINT8;
  const cuuint64_t gdim[4] = {(cuuint64_t)TR::inner, (cuuint64_t)((W + TR::inner - 1) / TR::inner),
                              (cuuint64_t)H, (cuuint64_t)nch};
  const cuuint64_t gstride[3] = {16, (cuuint64_t)plane_pitch, (cuuint64_t)plane_bytes};
  const cuuint32_t box[4] = {(cuuint32_t)TR::inner, (cuuint32_t)box_part(nbox), 1, 1};
  const cuuint32_t estride[4] = {1, 1, 1, 1};
  CUresult r = enc(map, dt, 4, const_cast<void*>(planes), gdim, gstride, box, estride,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

// Splits an nch-channel image into planes at `planes` (row pitch rounded up
// to 128 bytes). Returns the plane pitch.
template <int ELEM>
size_t split_channels(const DevImage& src, char* planes, cudaStream_t stream, bool count = true) {
  typedef ElemTraits<ELEM> TR;
  const size_t plane_pitch = ((size_t)src.width * TR::size + 127) / 128 * 128;
  const size_t plane_bytes = plane_pitch * src.height;
  typedef typename std::conditional<TR::size == 4, uint32_t,
                                    typename std::conditional<TR::size == 2, uint16_t,
                                                              uint8_t>::type>::type PT;
  const int pw = static_cast<int>(plane_pitch / TR::size);  // row length incl. the tail
  dim3 sg((pw + 255) / 256, src.height);
  split_channels_kernel<PT><<<sg, 256, 0, stream>>>((const char*)src.ptr, src.pitch, planes,
                                                    plane_pitch, plane_bytes, src.width, pw,
                                                    src.height, src.nch);
  if (count) count_launches(1);
  return plane_pitch;
}

size_t plane_set_bytes(const DevImage& s) {
  const size_t pitch = ((size_t)s.width * type_bytes(s.type) + 127) / 128 * 128;
  return pitch * s.height * s.nch;
}

// Channel planes of a source: the image itself for one channel, else a split
// copy in the context's scratch.
struct Planes {
  const char* ptr;
  size_t pitch, bytes;  // between rows, between planes
};

template <int ELEM>
Planes source_planes(Context& ctx, const DevImage& src) {
  Planes p{(const char*)src.ptr, src.pitch, src.pitch * src.height};
  if (src.nch > 1) {
    char* pl = reinterpret_cast<char*>(ctx.scratch(Context::kPlanes, plane_set_bytes(src)));
    p.pitch = split_channels<ELEM>(src, pl, ctx.stream);
    p.bytes = p.pitch * src.height;
    p.ptr = pl;
  }
  return p;
}

RowEnergyJob energy_job(const Planes& p, const DevImage& src, int tw, int ax, char* dst) {
  const size_t pitch = row_energy_pitch(src.width);
  return RowEnergyJob{p.ptr, p.pitch, p.bytes, dst, pitch, pitch * src.height, src.width,
                      src.height, src.nch, tw, ax};
}

cudaError_t launch_energy(RowEnergyJob j, char* dst, int type, cudaStream_t stream,
                          bool count = true) {
  j.dst = dst;
  if (count) count_launches(1);
  return launch_row_energies(type, j.tw, j, nullptr, 1, j.W, j.H, stream);
}

// One launch of `n` templates of one rows class over a source: a measure's map
// (n = 1), or the product sums of the tiles of a larger template. With row
// energies the kernel is a programmatic dependent of the launch that writes
// them (the one before it on the stream): it starts as that one's blocks leave,
// and only the epilogue waits for the energies, so its start (TMEM, template
// operand, first rows: 6 us) runs in the tail of that launch. Whatever was on
// the stream before the energies has completed, as that launch is an ordinary
// one. 1920 x 1080 U8 48 x 40 CrossCorr_Norm 73.9 -> 70.6 us, 4096 x 4096 F32 31 x 31
// 214 -> 211.
template <int ELEM>
cudaError_t launch_items(Context& ctx, TensorLaunch& P, const DevImage& src, const Planes& planes,
                         int cls, int n, int smem_bytes) {
  ItemArgs& a = P.base;
  const int R = class_r(cls);
  const int sw = strip_width<ELEM>(cls);
  const int nstrips = (src.width + sw - 1) / sw;
  P.mode = 0;
  P.err = &ctx.page->error;
  P.BH = ctx.band_rows > 0
             ? std::min(ctx.band_rows, src.height)
             : band_height(src.height, R, (long long)nstrips * src.nch * n, ctx.sm_count);
  a.W = src.width;
  a.H = src.height;
  a.R = R;
  a.nch = src.nch;
  a.nbox = P.nbox;
  if (smem_bytes > kMaxDynSmem) return cudaErrorInvalidValue;
  cudaError_t e = encode_planes<ELEM>(&P.map, planes.ptr, src.width, src.height, src.nch,
                                      planes.pitch, planes.bytes, P.nbox);
  if (e != cudaSuccess) return e;
  auto kern = a.idx_op >= 0 ? prox_tensor_kernel<ELEM, true> : prox_tensor_kernel<ELEM, false>;
  e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynSmem);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(nstrips, (src.height + P.BH - 1) / P.BH, src.nch * n);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem_bytes;
  cfg.stream = ctx.stream;
  cudaLaunchAttribute attr = {};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = a.energy ? 1 : 0;
  e = cudaLaunchKernelEx(&cfg, kern, P);
  count_launches(1);
  return e != cudaSuccess ? e : cudaGetLastError();
}

template <int ELEM>
cudaError_t launch_one(Context& ctx, Measure m, const DevImage& src, const DevImage& tmpl,
                       const DevImage& dst, int ax, int ay, int idx_op = -1,
                       void* idx_out = nullptr) {
  const int cls = class_of(tmpl.height);
  TensorLaunch P;
  std::memset(&P, 0, sizeof(P));
  P.measure = m;
  P.nbox = nbox_for<ELEM>(cls, tmpl.width, ax);
  ItemArgs& a = P.base;
  a.tw = tmpl.width;
  a.th = tmpl.height;
  a.ax = ax;
  a.ay = ay;
  a.tmpl = (const char*)tmpl.ptr;
  a.tmpl_pitch = tmpl.pitch;
  a.dst = (char*)dst.ptr;
  a.dst_pitch = dst.pitch;
  a.dst_f64 = dst.type == F64;
  a.dst_nch = src.nch;
  a.measure = m;
  a.idx_op = idx_op;
  a.idx_out = reinterpret_cast<char*>(idx_out);
  if (idx_op >= 0) {
    P.ticket = reinterpret_cast<unsigned*>(ctx.scratch(Context::kTickets, 256));
    P.index = &ctx.page->index;
  }
  const Planes planes = source_planes<ELEM>(ctx, src);
  // Row energies of every source row, for the measures that use them.
  if (m != kCrossCorr) {
    const RowEnergyJob j = energy_job(planes, src, tmpl.width, ax, nullptr);
    char* emap =
        reinterpret_cast<char*>(ctx.scratch(Context::kEnergyMap, j.dst_plane * src.nch));
    const cudaError_t e = launch_energy(j, emap, src.type, ctx.stream);
    if (e != cudaSuccess) return e;
    a.energy = emap;
    a.e_pitch = j.dst_pitch;
    a.e_plane = j.dst_plane;
  }
  return launch_items<ELEM>(ctx, P, src, planes, cls, 1,
                            smem_for<ELEM>(cls, tmpl.width, ax, P.nbox));
}

// ---- Batches ------------------------------------------------------------------

// Autotuned band heights, per (element type, template class, channels).
std::mutex g_tune_mutex;
std::map<std::tuple<int, int, int>, int> g_tuned_bh;

}  // namespace

struct TensorBatch {
  Context* ctx = nullptr;
  int elem = 0;
  int measure = 0;
  int nbox = 0;
  int smem = 0;
  int nitems = 0;
  void* tables = nullptr;  // maps, images, templates, dests, items, counter
  char* planes = nullptr;  // channel planes of multi-channel images
  std::vector<std::pair<int, size_t>> plane_offsets;  // per image: (split?, offset)
  std::vector<DevImage> images;
  TensorLaunch launch;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  std::map<int, int> bh;  // class -> band height used
  // Row-energy maps, one per (image, template width) of the batch (measures
  // other than CrossCorr), recomputed by every run.
  // One launch per staged width of the kernel (energy_groups) over the device
  // table ejobs, sorted by template width.
  std::vector<RowEnergyJob> ejobs;
  RowEnergyJob* ejobs_dev = nullptr;
  char* emaps = nullptr;
};

namespace {

// Channel splits, window energies, queue reset, persistent launch. `count`
// is false while the work is recorded into a graph (counted when the graph
// is launched).
template <int ELEM>
cudaError_t batch_record(TensorBatch& b, cudaStream_t stream, bool count) {
  for (size_t i = 0; i < b.images.size(); ++i) {
    if (b.plane_offsets[i].first)
      split_channels<ELEM>(b.images[i], b.planes + b.plane_offsets[i].second, stream, count);
  }
  // Row energies: the narrow templates' maps in one launch, the others' in a
  // second one (rows of 256 + tw - 1 pixels: 288 or 320 staged).
  for (size_t i = 0; i < b.ejobs.size();) {
    size_t n = i;
    int W = 0, H = 0;
    while (n < b.ejobs.size() && (b.ejobs[n].tw <= 33) == (b.ejobs[i].tw <= 33)) {
      W = std::max(W, b.ejobs[n].W);
      H = std::max(H, b.ejobs[n].H);
      ++n;
    }
    const cudaError_t ee =
        launch_row_energies(b.images[0].type, b.ejobs[n - 1].tw, b.ejobs[i], b.ejobs_dev + i,
                            (int)(n - i), W, H, stream);
    if (ee != cudaSuccess) return ee;
    if (count) count_launches(1);
    i = n;
  }
  cudaError_t e = cudaMemsetAsync(b.launch.counter, 0, sizeof(int), stream);
  if (e != cudaSuccess) return e;
  auto kern = prox_tensor_kernel<ELEM>;
  kern<<<b.ctx->sm_count, kThreads, b.smem, stream>>>(b.launch);
  if (count) count_launches(1);
  return cudaGetLastError();
}

// Builds the item list of a batch: every (image, template) pair, channel,
// strip and band; the largest items first, so the queue ends on small ones.
template <int ELEM>
std::vector<BatchItem> make_items(const std::vector<DevImage>& imgs,
                                  const std::vector<DevImage>& tpls,
                                  const std::vector<int>& pair_img,
                                  const std::vector<int>& pair_tpl,
                                  const std::vector<int>& pair_dst,
                                  const std::vector<int>& pair_energy,
                                  const std::map<int, int>& bh) {
  std::vector<std::pair<long long, BatchItem>> v;
  for (size_t p = 0; p < pair_img.size(); ++p) {
    const DevImage& s = imgs[pair_img[p]];
    const DevImage& t = tpls[pair_tpl[p]];
    const int cls = class_of(t.height);
    const int R = class_r(cls);
    const Geo g = geo_for<ELEM>(cls, t.width, t.width / 2);
    const int BH = bh.at(cls);
    const int sw = strip_width<ELEM>(cls);
    const int nstrips = (s.width + sw - 1) / sw;
    for (int c = 0; c < s.nch; ++c)
      for (int st = 0; st < nstrips; ++st)
        for (int y0 = 0; y0 < s.height; y0 += BH) {
          BatchItem it;
          it.img = pair_img[p];
          it.tpl = pair_tpl[p];
          it.dst = pair_dst[p];
          it.energy = pair_energy[p];
          it.ch = c;
          it.strip = st;
          it.y0 = y0;
          it.yend = std::min(s.height, y0 + BH);
          // steps x MMA work per step (MMAs of Np columns, plus a fixed part)
          const long long cost = (long long)(it.yend - y0 + R - 1) * (g.nmma * kNp + 512);
          v.push_back({cost, it});
        }
  }
  std::stable_sort(v.begin(), v.end(),
                   [](const std::pair<long long, BatchItem>& a,
                      const std::pair<long long, BatchItem>& b) { return a.first > b.first; });
  std::vector<BatchItem> out;
  out.reserve(v.size());
  for (auto& x : v) out.push_back(x.second);
  return out;
}

// Device tables of a batch in one allocation; returns the TensorLaunch
// pointers into it.
template <int ELEM>
cudaError_t upload_tables(TensorBatch& b, const std::vector<CUtensorMap>& maps,
                          const std::vector<BatchImage>& bimgs,
                          const std::vector<BatchTemplate>& btpls,
                          const std::vector<BatchDest>& bdsts,
                          const std::vector<BatchItem>& items,
                          const std::vector<BatchEnergy>& benergy, void** mem) {
  auto al = [](size_t x) { return (x + 255) / 256 * 256; };
  const size_t o_maps = 0;
  const size_t o_imgs = al(o_maps + maps.size() * sizeof(CUtensorMap));
  const size_t o_tpls = al(o_imgs + bimgs.size() * sizeof(BatchImage));
  const size_t o_dsts = al(o_tpls + btpls.size() * sizeof(BatchTemplate));
  const size_t o_items = al(o_dsts + bdsts.size() * sizeof(BatchDest));
  const size_t o_en = al(o_items + items.size() * sizeof(BatchItem));
  const size_t o_ctr = al(o_en + benergy.size() * sizeof(BatchEnergy));
  const size_t total = o_ctr + 256;
  std::vector<char> host(total, 0);
  std::memcpy(host.data() + o_maps, maps.data(), maps.size() * sizeof(CUtensorMap));
  std::memcpy(host.data() + o_imgs, bimgs.data(), bimgs.size() * sizeof(BatchImage));
  std::memcpy(host.data() + o_tpls, btpls.data(), btpls.size() * sizeof(BatchTemplate));
  std::memcpy(host.data() + o_dsts, bdsts.data(), bdsts.size() * sizeof(BatchDest));
  std::memcpy(host.data() + o_items, items.data(), items.size() * sizeof(BatchItem));
  if (!benergy.empty())
    std::memcpy(host.data() + o_en, benergy.data(), benergy.size() * sizeof(BatchEnergy));
  char* d = nullptr;
  cudaError_t e = cudaMalloc(&d, total);
  if (e != cudaSuccess) return e;
  e = cudaMemcpy(d, host.data(), total, cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    cudaFree(d);
    return e;
  }
  *mem = d;
  TensorLaunch& P = b.launch;
  P.maps = reinterpret_cast<const CUtensorMap*>(d + o_maps);
  P.imgs = reinterpret_cast<const BatchImage*>(d + o_imgs);
  P.tpls = reinterpret_cast<const BatchTemplate*>(d + o_tpls);
  P.dsts = reinterpret_cast<const BatchDest*>(d + o_dsts);
  P.items = reinterpret_cast<const BatchItem*>(d + o_items);
  P.energies = reinterpret_cast<const BatchEnergy*>(d + o_en);
  P.nitems = static_cast<int>(items.size());
  P.counter = reinterpret_cast<int*>(d + o_ctr);
  return cudaSuccess;
}

// Autotuner: for one template class, times the persistent kernel on the
// probe pair (first image and template of that class) replicated so that
// every band height sees the same total work and enough items for all SMs,
// and keeps the band height with the least time per pair. The candidates
// span the trade-off between ramp rows (R - 1 per band, favouring tall
// bands) and load balance (favouring short ones).
template <int ELEM>
int autotune_bh(Context& ctx, int measure, const DevImage& img, const CUtensorMap& map,
                const Planes& planes, const DevImage& tpl, int cls, int nbox, int smem,
                char* probe_dst, size_t probe_pitch) {
  const int R = class_r(cls);
  std::vector<int> cand;
  for (int bh : {64, 128, 192, 256, 384, 512, 768, 1024})
    if (bh >= R && bh < img.height) cand.push_back(bh);
  cand.push_back(img.height);
  const int sw = strip_width<ELEM>(cls);
  const int nstrips = (img.width + sw - 1) / sw;
  const long long units = (long long)nstrips * img.nch;
  // Replicas so that the shortest candidate has at least 4 items per SM.
  const int min_bh = cand.front();
  const long long items_min = units * ((img.height + min_bh - 1) / min_bh);
  const int reps = (int)std::max<long long>(
      1, std::min<long long>(64, (4LL * ctx.sm_count + items_min - 1) / items_min));
  std::vector<CUtensorMap> maps(1, map);
  std::vector<BatchImage> bimgs(1, BatchImage{img.width, img.height, img.nch});
  std::vector<BatchTemplate> btpls(1, BatchTemplate{(const char*)tpl.ptr, tpl.pitch, tpl.width,
                                                    tpl.height, cls});
  std::vector<BatchDest> bdsts(1, BatchDest{probe_dst, probe_pitch, 0});
  // The probe pair's row energies, computed once for every candidate.
  std::vector<BatchEnergy> benergy;
  char* probe_e = nullptr;
  if (measure != kCrossCorr) {
    const RowEnergyJob j = energy_job(planes, img, tpl.width, tpl.width / 2, nullptr);
    if (cudaMalloc(&probe_e, j.dst_plane * img.nch) != cudaSuccess) return cand.back();
    if (launch_energy(j, probe_e, img.type, ctx.stream) != cudaSuccess) {
      cudaFree(probe_e);
      return cand.back();
    }
    benergy.push_back(BatchEnergy{probe_e, j.dst_pitch, j.dst_plane});
  }
  float best = 1e30f;
  int best_bh = cand.back();
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  for (int bh : cand) {
    std::vector<int> pi(reps, 0), pt(reps, 0), pd(reps, 0), pe(reps, probe_e ? 0 : -1);
    std::map<int, int> m1{{cls, bh}};
    std::vector<BatchItem> items = make_items<ELEM>({img}, {tpl}, pi, pt, pd, pe, m1);
    TensorBatch tb;
    tb.ctx = &ctx;
    std::memset(&tb.launch, 0, sizeof(tb.launch));
    tb.launch.mode = 1;
    tb.launch.measure = measure;
    tb.launch.nbox = nbox;
    tb.launch.err = &ctx.page->error;
    tb.smem = smem;
    void* mem = nullptr;
    if (upload_tables<ELEM>(tb, maps, bimgs, btpls, bdsts, items, benergy, &mem) != cudaSuccess)
      break;
    float ms = 1e30f;
    for (int rep = 0; rep < 3; ++rep) {
      cudaEventRecord(e0, ctx.stream);
      batch_record<ELEM>(tb, ctx.stream, true);
      cudaEventRecord(e1, ctx.stream);
      cudaEventSynchronize(e1);
      float t = 0.f;
      cudaEventElapsedTime(&t, e0, e1);
      if (rep > 0) ms = std::min(ms, t);  // the first run warms up
    }
    cudaFree(mem);
    if (ms < best) {
      best = ms;
      best_bh = bh;
    }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (probe_e) {
    cudaStreamSynchronize(ctx.stream);
    cudaFree(probe_e);
  }
  return best_bh;
}

template <int ELEM>
TensorBatch* batch_create(Context& ctx, Measure m, const std::vector<DevImage>& imgs,
                          const std::vector<DevImage>& tpls, const std::vector<DevImage>& dsts,
                          cudaError_t* err) {
  TensorBatch* b = new TensorBatch();
  b->ctx = &ctx;
  b->elem = ELEM;
  b->measure = m;
  // One staged-row width for every tensor map of the batch: the widest need.
  b->nbox = 1;
  for (const DevImage& t : tpls)
    b->nbox = std::max(b->nbox, nbox_for<ELEM>(class_of(t.height), t.width, t.width / 2));
  b->images = imgs;
  std::memset(&b->launch, 0, sizeof(b->launch));
  cudaError_t e = cudaSuccess;
  auto fail = [&](cudaError_t code) {
    *err = code;
    tensor_batch_destroy(b);
    return static_cast<TensorBatch*>(nullptr);
  };

  // Channel planes of multi-channel images (owned by the batch).
  size_t plane_total = 0;
  for (const DevImage& s : imgs) {
    b->plane_offsets.push_back({s.nch > 1 ? 1 : 0, plane_total});
    if (s.nch > 1) plane_total += plane_set_bytes(s);
  }
  if (plane_total) {
    e = cudaMalloc(&b->planes, plane_total);
    if (e != cudaSuccess) return fail(e);
  }
  std::vector<CUtensorMap> maps(imgs.size());
  std::vector<Planes> planes;
  for (size_t i = 0; i < imgs.size(); ++i) {
    const DevImage& s = imgs[i];
    Planes p{(const char*)s.ptr, s.pitch, s.pitch * s.height};
    if (s.nch > 1) {
      p.ptr = b->planes + b->plane_offsets[i].second;
      p.bytes = plane_set_bytes(s) / s.nch;
      p.pitch = p.bytes / s.height;
    }
    planes.push_back(p);
    e = encode_planes<ELEM>(&maps[i], p.ptr, s.width, s.height, s.nch, p.pitch, p.bytes, b->nbox);
    if (e != cudaSuccess) return fail(e);
  }
  std::vector<BatchImage> bimgs;
  for (const DevImage& s : imgs) bimgs.push_back(BatchImage{s.width, s.height, s.nch});
  std::vector<BatchTemplate> btpls;
  for (const DevImage& t : tpls)
    btpls.push_back(BatchTemplate{(const char*)t.ptr, t.pitch, t.width, t.height,
                                  class_of(t.height)});
  std::vector<BatchDest> bdsts;
  for (const DevImage& d : dsts) bdsts.push_back(BatchDest{(char*)d.ptr, d.pitch, d.type == F64});

  auto kern = prox_tensor_kernel<ELEM>;
  e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynSmem);
  if (e != cudaSuccess) return fail(e);
  // Shared memory: the largest need of any template (per class, the widest).
  std::map<int, int> cls_smem;
  for (const DevImage& t : tpls) {
    const int c = class_of(t.height);
    const int sm = smem_for<ELEM>(c, t.width, t.width / 2, b->nbox);
    if (sm > kMaxDynSmem) return fail(cudaErrorInvalidValue);
    cls_smem[c] = std::max(cls_smem[c], sm);
  }

  // Multi-channel probes read the planes: split them once before tuning.
  for (size_t i = 0; i < imgs.size(); ++i)
    if (b->plane_offsets[i].first)
      split_channels<ELEM>(imgs[i], b->planes + b->plane_offsets[i].second, ctx.stream);

  // Band height per template class: autotuned once per (type, class,
  // channels) and kept for the process.
  std::map<int, int> bh;
  for (size_t j = 0; j < tpls.size(); ++j) {
    const int cls = btpls[j].cls;
    if (bh.count(cls)) continue;
    const auto key = std::make_tuple(ELEM, cls, imgs[0].nch);
    {
      std::lock_guard<std::mutex> lk(g_tune_mutex);
      auto it = g_tuned_bh.find(key);
      if (it != g_tuned_bh.end()) {
        bh[cls] = it->second;
        continue;
      }
    }
    const DevImage& probe = imgs[0];
    char* pd = nullptr;
    const size_t pp = ((size_t)probe.width * probe.nch * 4 + 127) / 128 * 128;
    e = cudaMalloc(&pd, pp * probe.height);
    if (e != cudaSuccess) return fail(e);
    const int v = autotune_bh<ELEM>(ctx, m, probe, maps[0], planes[0], tpls[j], cls, b->nbox,
                                    cls_smem[cls], pd, pp);
    cudaStreamSynchronize(ctx.stream);
    cudaFree(pd);
    e = cudaGetLastError();
    if (e != cudaSuccess) return fail(e);
    bh[cls] = v;
    std::lock_guard<std::mutex> lk(g_tune_mutex);
    g_tuned_bh[key] = v;
  }
  b->bh = bh;

  // Row-energy maps: one per (image, template width) for the measures that
  // use them, laid out back to back in one allocation owned by the batch.
  std::map<std::pair<int, int>, int> eidx;
  std::vector<BatchEnergy> benergy;
  if (m != kCrossCorr) {
    std::vector<int> widths;
    for (const DevImage& t : tpls) widths.push_back(t.width);
    std::sort(widths.begin(), widths.end());
    widths.erase(std::unique(widths.begin(), widths.end()), widths.end());
    size_t total = 0;
    std::vector<size_t> at;
    for (int w : widths)
      for (size_t i = 0; i < imgs.size(); ++i) {
        eidx[std::make_pair((int)i, w)] = (int)b->ejobs.size();
        b->ejobs.push_back(energy_job(planes[i], imgs[i], w, w / 2, nullptr));
        at.push_back(total);
        total += b->ejobs.back().dst_plane * imgs[i].nch;
      }
    e = cudaMalloc(&b->emaps, total);
    if (e != cudaSuccess) return fail(e);
    for (size_t k = 0; k < b->ejobs.size(); ++k) {
      RowEnergyJob& j = b->ejobs[k];
      j.dst = b->emaps + at[k];
      benergy.push_back(BatchEnergy{j.dst, j.dst_pitch, j.dst_plane});
    }
    const size_t jb = b->ejobs.size() * sizeof(RowEnergyJob);
    e = cudaMalloc(&b->ejobs_dev, jb);
    if (e != cudaSuccess) return fail(e);
    e = cudaMemcpy(b->ejobs_dev, b->ejobs.data(), jb, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) return fail(e);
  }
  std::vector<int> pi, pt, pd, pe;
  for (size_t i = 0; i < imgs.size(); ++i)
    for (size_t j = 0; j < tpls.size(); ++j) {
      pi.push_back((int)i);
      pt.push_back((int)j);
      pd.push_back((int)(i * tpls.size() + j));
      pe.push_back(m != kCrossCorr ? eidx[std::make_pair((int)i, tpls[j].width)] : -1);
    }
  std::vector<BatchItem> items = make_items<ELEM>(imgs, tpls, pi, pt, pd, pe, bh);
  b->launch.mode = 1;
  b->launch.measure = m;
  b->launch.nbox = b->nbox;
  b->launch.err = &ctx.page->error;
  e = upload_tables<ELEM>(*b, maps, bimgs, btpls, bdsts, items, benergy, &b->tables);
  if (e != cudaSuccess) return fail(e);
  b->nitems = b->launch.nitems;
  b->smem = 0;
  for (const auto& kv : cls_smem) b->smem = std::max(b->smem, kv.second);

  // Capture the batch (splits, queue reset, persistent launch) as a graph.
  e = cudaStreamSynchronize(ctx.stream);
  if (e != cudaSuccess) return fail(e);
  e = cudaStreamBeginCapture(ctx.stream, cudaStreamCaptureModeThreadLocal);
  if (e != cudaSuccess) return fail(e);
  const cudaError_t re = batch_record<ELEM>(*b, ctx.stream, false);
  e = cudaStreamEndCapture(ctx.stream, &b->graph);
  if (re != cudaSuccess) return fail(re);
  if (e != cudaSuccess) return fail(e);
  e = cudaGraphInstantiate(&b->exec, b->graph, 0);
  if (e != cudaSuccess) return fail(e);
  *err = cudaSuccess;
  return b;
}

}  // namespace

namespace {

// One thread waits on an mbarrier that nothing arrives on, with the bounded
// wait of the tensor kernels: the wait expires, sets the abort flag, and the
// kernel raises the context's error flag and returns.
__global__ void bounded_wait_probe_kernel(long long limit, int* err) {
  __shared__ uint64_t bar;
  __shared__ int abort_flag;
  if (threadIdx.x == 0) {
    abort_flag = 0;
    mbar_init(&bar, 1);
    fence_barrier_init();
    const bool ok = mbar_wait(&bar, 0, &abort_flag, limit);
    if (!ok) {
      *reinterpret_cast<volatile int*>(err) = 1;
      __threadfence_system();
    }
    mbar_inval(&bar);
  }
}

}  // namespace

cudaError_t launch_bounded_wait_probe(Context& ctx, long long limit_cycles) {
  int* err = &ctx.page->error;
  bounded_wait_probe_kernel<<<1, 32, 0, ctx.stream>>>(limit_cycles, err);
  count_launches(1);
  return cudaGetLastError();
}

bool tensor_supports(Measure m, const DevImage& src, const DevImage& tmpl, const DevImage& dst,
                     bool forced) {
  if (m == kAbsDistance) return false;
  if (src.nch != tmpl.nch || src.nch != dst.nch || src.nch < 1 || src.nch > 4) return false;
  // Templates beyond 64 x 64 run as tiles of at most 64 x 64 (tensor_large.cu);
  // the row energies take templates up to 1024 columns.
  if (tmpl.width > 1024) return false;
  if (src.type == U8) return true;
  // F32 and U16 use the BF16 hi + lo split: about 16 bits of each F32 operand
  // (all 16 of a U16), so one product can be off by ~3e-5 relative; the 1e-5
  // bar needs the errors of many terms to average, and tiny templates gain
  // nothing from the MMA. Taken only when asked for.
  if (src.type == F32 || src.type == U16) return forced && tmpl.width * tmpl.height >= 64;
  return false;
}

cudaError_t launch_proximity_tensor(Context& ctx, Measure m, const DevImage& src,
                                    const DevImage& tmpl, const DevImage& dst) {
  if (tmpl.width > 64 || tmpl.height > 64) return launch_proximity_tensor_large(ctx, m, src, tmpl, dst);
  return launch_proximity_tensor_anchored(ctx, m, src, tmpl, dst, tmpl.width / 2,
                                          tmpl.height / 2);
}

cudaError_t launch_proximity_tensor_anchored(Context& ctx, Measure m, const DevImage& src,
                                             const DevImage& tmpl, const DevImage& dst, int ax,
                                             int ay) {
  if (src.type == U8) return launch_one<kU8>(ctx, m, src, tmpl, dst, ax, ay);
  if (src.type == U16) return launch_one<kU16>(ctx, m, src, tmpl, dst, ax, ay);
  return launch_one<kF32>(ctx, m, src, tmpl, dst, ax, ay);
}

size_t tensor_index_records_bytes(const Context& ctx, const DevImage& src, const DevImage& tmpl) {
  (void)ctx;
  const int cls = class_of(tmpl.height);
  const int sw = kM * s_for(class_r(cls));
  const size_t nstrips = (src.width + sw - 1) / sw;
  // At most one band per row (a fixed band height of 1).
  const size_t nbands = src.height;
  return nstrips * nbands * src.nch * kEpilogue * sizeof(IdxRecord);
}

cudaError_t launch_proximity_tensor_indexed(Context& ctx, Measure m, const DevImage& src,
                                            const DevImage& tmpl, const DevImage& dst, int idx_op,
                                            void* records, float* best, int* bx, int* by,
                                            bool* has_nan) {
  cudaError_t e;
  const int ax = tmpl.width / 2, ay = tmpl.height / 2;
  if (src.type == U8)
    e = launch_one<kU8>(ctx, m, src, tmpl, dst, ax, ay, idx_op, records);
  else if (src.type == U16)
    e = launch_one<kU16>(ctx, m, src, tmpl, dst, ax, ay, idx_op, records);
  else
    e = launch_one<kF32>(ctx, m, src, tmpl, dst, ax, ay, idx_op, records);
  if (e != cudaSuccess) return e;
  e = cudaStreamSynchronize(ctx.stream);
  if (e != cudaSuccess) return e;
  const volatile Context::HostPage::Index* r = &ctx.page->index;
  *best = r->v;
  *bx = r->x;
  *by = r->y;
  *has_nan = r->nan != 0;
  return cudaSuccess;
}

namespace {
template <int ELEM>
cudaError_t launch_tiles(Context& ctx, const DevImage& src, const std::vector<TensorTile>& tiles,
                         const TensorPlanes& planes, char* maps, size_t pitch) {
  TensorLaunch P;
  std::memset(&P, 0, sizeof(P));
  P.measure = kCrossCorr;
  int rows = 0;
  for (const TensorTile& t : tiles) rows = std::max(rows, t.tmpl.height);
  const int cls = class_of(rows);
  P.nbox = 1;
  for (const TensorTile& t : tiles)
    P.nbox = std::max(P.nbox, nbox_for<ELEM>(cls, t.tmpl.width, t.ax));
  int smem = 0;
  for (const TensorTile& t : tiles)
    smem = std::max(smem, smem_for<ELEM>(cls, t.tmpl.width, t.ax, P.nbox));
  P.ntiles = (int)tiles.size();
  for (int i = 0; i < P.ntiles; ++i)
    P.tiles[i] = TemplateTile{(const char*)tiles[i].tmpl.ptr, tiles[i].tmpl.width,
                              tiles[i].tmpl.height, tiles[i].ax, tiles[i].ay};
  P.tile_plane = pitch * src.height;
  ItemArgs& a = P.base;
  a.tmpl_pitch = tiles[0].tmpl.pitch;
  a.dst = maps;
  a.dst_pitch = pitch;
  a.dst_nch = 1;
  a.raw = src.type == U8;
  a.measure = kCrossCorr;
  a.idx_op = -1;
  return launch_items<ELEM>(ctx, P, src, Planes{planes.ptr, planes.pitch, planes.bytes}, cls,
                            P.ntiles, smem);
}
}  // namespace

TensorPlanes tensor_source_planes(Context& ctx, const DevImage& src) {
  const Planes p = src.type == U8    ? source_planes<kU8>(ctx, src)
                   : src.type == U16 ? source_planes<kU16>(ctx, src)
                                     : source_planes<kF32>(ctx, src);
  return TensorPlanes{p.ptr, p.pitch, p.bytes};
}

int tensor_max_tiles() { return kMaxTiles; }

cudaError_t launch_tensor_tiles(Context& ctx, const DevImage& src,
                                const std::vector<TensorTile>& tiles, const TensorPlanes& planes,
                                char* maps, size_t pitch) {
  if (src.type == U8) return launch_tiles<kU8>(ctx, src, tiles, planes, maps, pitch);
  if (src.type == U16) return launch_tiles<kU16>(ctx, src, tiles, planes, maps, pitch);
  return launch_tiles<kF32>(ctx, src, tiles, planes, maps, pitch);
}

TensorBatch* tensor_batch_create(Context& ctx, Measure m, const std::vector<DevImage>& imgs,
                                 const std::vector<DevImage>& tpls,
                                 const std::vector<DevImage>& dsts, cudaError_t* err) {
  if (imgs[0].type == U8) return batch_create<kU8>(ctx, m, imgs, tpls, dsts, err);
  if (imgs[0].type == U16) return batch_create<kU16>(ctx, m, imgs, tpls, dsts, err);
  return batch_create<kF32>(ctx, m, imgs, tpls, dsts, err);
}

cudaError_t tensor_batch_run(TensorBatch* b) {
  // Launches of the graph: splits, row energies (at most two groups), the kernel.
  const bool two = !b->ejobs.empty() && b->ejobs.front().tw <= 33 && b->ejobs.back().tw > 33;
  count_launches(1 + (b->ejobs.empty() ? 0 : two ? 2 : 1) +
                 std::count_if(b->plane_offsets.begin(), b->plane_offsets.end(),
                               [](const std::pair<int, size_t>& p) { return p.first != 0; }));
  return cudaGraphLaunch(b->exec, b->ctx->stream);
}

int tensor_batch_items(const TensorBatch* b) { return b->nitems; }

int tensor_batch_band_height(const TensorBatch* b, int tw, int th) {
  (void)tw;
  auto it = b->bh.find(class_of(th));
  return it == b->bh.end() ? 0 : it->second;
}

void tensor_batch_destroy(TensorBatch* b) {
  if (!b) return;
  if (b->ctx) cudaStreamSynchronize(b->ctx->stream);
  if (b->exec) cudaGraphExecDestroy(b->exec);
  if (b->graph) cudaGraphDestroy(b->graph);
  if (b->tables) cudaFree(b->tables);
  if (b->planes) cudaFree(b->planes);
  if (b->emaps) cudaFree(b->emaps);
  if (b->ejobs_dev) cudaFree(b->ejobs_dev);
  delete b;
}

}  // namespace ocipb
