// CSR SpMM  C = A B  for sm_100a (A sparse M x K in CSR, B dense K x N row-major).
//
// The launch reuses the SpMV unit plan (plan.cu), built with the SpMM window
// cap (64) and chunk (256).  One kernel, k_spmm_team, serves every width: teams
// of lanes own a column tile of B and C and take equal shares of the nonzeros
// of a run of rows; long rows run as chunks whose partials are joined in order.
// Rows of whole aligned 16-byte slices give each lane one slice; other widths
// give it up to four smaller pieces (Slice).
//
// Accumulation: fp32 for half / bfloat16 / fp32 values (half and bfloat16
// products are exact in fp32), fp64 for fp64, componentwise for complex.
// FSB_SPMM_COMPENSATED switches every sum to Dot2 compensated accumulation.
// Every sum runs in a fixed order, so results are bitwise reproducible.
//
// The same file holds that kernel fused with an SpMV (the batched step) and
// the one-launch backward of Y = A X
// (k_spmm_bwd: dX = A^T dY and the SDDMM dvals from one gather of dY).
//
// Replaces _triton_spmm_csr_impl / _spmm_csr_real_kernel / the complex kernel
// (sparse_operations/spmm_csr.py:3373-3466, 144-339) and the bucketed
// alg1 / alg2 / opt kernels (spmm_csr.py:1091-2449, spmm_csr_opt_alg2.py) of
// flagos-ai/FlagSparse.
#include <atomic>
#include <cstring>
#include <type_traits>

#include "fsb_common.cuh"

namespace fsb {
namespace {

// Warps per block, one work item (or unit) per warp.  Items are uneven, and a
// block's place is free only when its last warp ends: blocks of 2 warps instead
// of 8 keep more warps resident (1 M-row power-law matrix, 128 columns: bf16
// 1.54 -> 1.30 ms, fp32 2.35 -> 2.16 ms; single warps: 1.25 / 2.90 ms).
// spmm_block_warps has the exceptions.
constexpr int kSpmmWarps = 2, kMaxSpmmWarps = 8;
// Rows of at least this many bytes, made of whole 32-byte slices on 32-byte
// boundaries, give each lane a 32-byte slice: half the lanes per row, so a warp
// instruction loads, addresses and tests twice the nonzeros.  At 2 warps per
// block (300,000 rows of Poisson(20)): bf16, 128 columns 205 -> 172 us; fp32,
// 128 columns 364 -> 330 us, 32 columns 99 -> 92 us; fp64 64 columns on a
// 300,000-row Zipf matrix 386 -> 337 us.  64-byte rows lose (fp32 68 -> 75 us:
// teams of two lanes, and the wider sums at row ends), except in the fused
// kernel, which also gathers x once per lane of a team (256 uneven matrices,
// 16 columns: 1.90 -> 1.75 ms with two slices ahead; four: 2.00 ms).
// Real types; compensated sums only in fp64 (64 columns 520 -> 472 us; fp32, 128
// columns lose, 531 against 559 us, their pairs of sums spilling); the fused
// kernel only in fp32.
template <bool FUSED>
constexpr int kSlice32Row = FUSED ? 64 : 128;
template <int DT, bool COMP, bool FUSED>
constexpr bool kSlice32 = FUSED ? DT == FSB_F32 && !COMP : !VT<DT>::kComplex && (!COMP || DT == FSB_F64);
constexpr int kSpmmBatch = 128;    // chunks of long rows are whole multiples of it
constexpr int kSpmmMaxCap = 64;    // row blocks hold < 2*cap <= kSpmmBatch nonzeros
// B slices a team loads ahead of its sums: 4; 6 in one-team warps; 2 of 32
// bytes in the fused kernel, whose x gathers and y sums need the registers
constexpr int kSpmmAhead = 4, kOneTeamAhead = 6, kFused32Ahead = 2;
template <int BYTES> struct RawT;
template <> struct RawT<2> { using T = unsigned short; };
template <> struct RawT<4> { using T = unsigned int; };
template <> struct RawT<8> { using T = uint2; };
template <> struct RawT<16> { using T = uint4; };
struct Raw32 { uint32_t r[8]; };
template <> struct RawT<32> { using T = Raw32; };

// A lane's share of a team's column tile: P pieces of E consecutive elements,
// a team's T lanes side by side in each piece, piece q of lane tl starting at
// tile column (q * T + tl) * E.  Aligned rows take one 16- or 32-byte piece
// (P = 1, see kSlice32Row).
// Other widths take pieces of one element or, where N, the leading dimensions
// and the addresses allow, of 4 or 8 bytes; each piece lies wholly inside or
// outside the N columns.
template <typename S, int E, int P>
struct Slice {
  static constexpr int V = E * P;
  static constexpr bool kWhole = P == 1 && E * int(sizeof(S)) >= 16;
  using Raw = typename RawT<E * int(sizeof(S))>::T;
  int off[P];  // this lane's first column of each piece, any valid column for pieces past N
  int nv;      // valid pieces

  __device__ __forceinline__ void set(int64_t tile, int T, int tl, int64_t n) {
    nv = 0;
#pragma unroll
    for (int q = 0; q < P; ++q) {
      const int64_t c = (tile * (int64_t(T) * P) + q * T + tl) * E;
      const bool ok = c < n;
      off[q] = ok ? static_cast<int>(c) : 0;
      nv += ok ? 1 : 0;
    }
  }
  // first column's address: whole slices carry their offset in it
  __device__ __forceinline__ const S* base(const S* B) const { return kWhole ? B + off[0] : B; }
  // slice of row `row` (whole slices: ldb < 2^32, a single wide 32 x 32-bit multiply)
  __device__ __forceinline__ void load(const S* __restrict__ base, uint32_t row, int64_t ldb, S (&out)[V]) const {
    const S* r = base + (kWhole ? static_cast<uint64_t>(row) * static_cast<uint32_t>(ldb)
                                : static_cast<uint64_t>(row) * static_cast<uint64_t>(ldb));
#pragma unroll
    for (int q = 0; q < P; ++q) {
      Raw w;
      if constexpr (sizeof(Raw) == 32)
        asm("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
            : "=r"(w.r[0]), "=r"(w.r[1]), "=r"(w.r[2]), "=r"(w.r[3]), "=r"(w.r[4]), "=r"(w.r[5]), "=r"(w.r[6]),
              "=r"(w.r[7])
            : "l"(r));
      else
        w = __ldg(reinterpret_cast<const Raw*>(r + (kWhole ? 0 : off[q])));
      memcpy(&out[q * E], &w, sizeof(Raw));
    }
  }
  // slice of the row at `row`, read once: a streaming (evict-first) load
  __device__ __forceinline__ void load_once(const S* __restrict__ row, S (&out)[V]) const {
    static_assert(kWhole, "whole slices");
    Raw w;
    if constexpr (sizeof(Raw) == 32)
      asm("ld.global.cs.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
          : "=r"(w.r[0]), "=r"(w.r[1]), "=r"(w.r[2]), "=r"(w.r[3]), "=r"(w.r[4]), "=r"(w.r[5]), "=r"(w.r[6]),
            "=r"(w.r[7])
          : "l"(row + off[0]));
    else
      w = __ldcs(reinterpret_cast<const Raw*>(row + off[0]));
    memcpy(out, &w, sizeof(Raw));
  }
  // streaming (evict-first) stores: the output is written once
  __device__ __forceinline__ void store(S* __restrict__ row, const S (&v)[V]) const {
#pragma unroll
    for (int q = 0; q < P; ++q)
      if (q < nv) {
        Raw w;
        memcpy(&w, &v[q * E], sizeof(Raw));
        if constexpr (sizeof(Raw) == 32)
          asm volatile("st.global.cs.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(row + off[q]), "r"(w.r[0]),
                       "r"(w.r[1]), "r"(w.r[2]), "r"(w.r[3]), "r"(w.r[4]), "r"(w.r[5]), "r"(w.r[6]), "r"(w.r[7])
                       : "memory");
        else
          __stcs(reinterpret_cast<Raw*>(row + off[q]), w);
      }
  }
};

__device__ __forceinline__ __half spmm_store(float v, __half*) { return __float2half_rn(v); }
__device__ __forceinline__ __nv_bfloat16 spmm_store(float v, __nv_bfloat16*) { return __float2bfloat16_rn(v); }
__device__ __forceinline__ float spmm_store(float v, float*) { return v; }
__device__ __forceinline__ double spmm_store(double v, double*) { return v; }

// c0 += a * b0, c1 += a * b1 in one packed fp32x2 FMA (sm_100a); each half is
// rounded exactly as a scalar fma.rn, so results equal the scalar loop's.
__device__ __forceinline__ void ffma2(float& c0, float& c1, float a, float b0, float b1) {
  unsigned long long cc, aa, bb;
  asm("mov.b64 %0, {%1, %2};" : "=l"(cc) : "f"(c0), "f"(c1));
  asm("mov.b64 %0, {%1, %2};" : "=l"(aa) : "f"(a), "f"(a));
  asm("mov.b64 %0, {%1, %2};" : "=l"(bb) : "f"(b0), "f"(b1));
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(cc) : "l"(aa), "l"(bb));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(c0), "=f"(c1) : "l"(cc));
}

// (c0, c1) += (a * lo(b), a * hi(b)) for a 16-bit a and two packed 16-bit
// values b: sm_100a's mixed-precision fma.rn.f32.{bf16,f16} multiplies the
// 16-bit inputs exactly (the product fits fp32) and rounds each sum once, so
// the results equal widening to fp32 and calling fmaf, with no widening
// instructions.
template <typename S>
__device__ __forceinline__ void fma_mixed2(float& c0, float& c1, S a, unsigned b) {
  unsigned short ab;
  memcpy(&ab, &a, 2);
  if constexpr (std::is_same<S, __nv_bfloat16>::value) {
    asm("{\n .reg .b16 bl, bh;\n mov.b32 {bl, bh}, %3;\n fma.rn.f32.bf16 %0, %2, bl, %0;\n"
        " fma.rn.f32.bf16 %1, %2, bh, %1;\n}"
        : "+f"(c0), "+f"(c1) : "h"(ab), "r"(b));
  } else {
    asm("{\n .reg .b16 bl, bh;\n mov.b32 {bl, bh}, %3;\n fma.rn.f32.f16 %0, %2, bl, %0;\n"
        " fma.rn.f32.f16 %1, %2, bh, %1;\n}"
        : "+f"(c0), "+f"(c1) : "h"(ab), "r"(b));
  }
}

// Per-lane accumulator of V output elements.
template <int DT, bool COMP, int V>
struct SpmmAcc {
  using Vt = VT<DT>;
  using S = typename Vt::Store;
  using R = typename Vt::Real;
  static constexpr bool kCplx = Vt::kComplex;
  static constexpr int kNC = kCplx ? 2 : 1;            // real components per element
  using Sum = typename std::conditional<COMP, Comp<R>, Plain<R>>::type;
  Sum s[kNC][V];

  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int c = 0; c < kNC; ++c)
#pragma unroll
      for (int j = 0; j < V; ++j) s[c][j].zero();
  }

  __device__ __forceinline__ static void term(Sum& acc, R a, R b) {
    if constexpr (COMP && Vt::kExactProduct) acc.add(mul_rn(a, b));  // exact product
    else acc.add_prod(a, b);
  }

  __device__ __forceinline__ void add(S a, const S (&b)[V]) {
    if constexpr (kCplx) {
#pragma unroll
      for (int j = 0; j < V; ++j) {
        term(s[0][j], a.x, b[j].x);
        term(s[0][j], -a.y, b[j].y);
        term(s[1][j], a.x, b[j].y);
        term(s[1][j], a.y, b[j].x);
      }
    } else {
      const R ar = to_real(a);
      if constexpr (!COMP && sizeof(S) == 2 && V % 2 == 0) {
        unsigned bw[V / 2];
        memcpy(bw, b, sizeof(bw));
#pragma unroll
        for (int j = 0; j < V; j += 2) fma_mixed2(s[0][j].hi, s[0][j + 1].hi, a, bw[j / 2]);
      } else if constexpr (!COMP && std::is_same<R, float>::value && V % 2 == 0) {
#pragma unroll
        for (int j = 0; j < V; j += 2) ffma2(s[0][j].hi, s[0][j + 1].hi, ar, to_real(b[j]), to_real(b[j + 1]));
      } else {
#pragma unroll
        for (int j = 0; j < V; ++j) term(s[0][j], ar, to_real(b[j]));
      }
    }
  }

  __device__ __forceinline__ void result(S (&out)[V]) const {
#pragma unroll
    for (int j = 0; j < V; ++j) {
      if constexpr (kCplx) {
        out[j].x = s[0][j].value();
        out[j].y = s[1][j].value();
      } else {
        out[j] = spmm_store(s[0][j].value(), static_cast<S*>(nullptr));
      }
    }
  }

  // scratch layout per element: (hi, lo) per real component
  __device__ __forceinline__ void store_partial(R* p) const {
#pragma unroll
    for (int j = 0; j < V; ++j)
#pragma unroll
      for (int c = 0; c < kNC; ++c) {
        p[(j * kNC + c) * 2] = s[c][j].hi;
        if constexpr (COMP) p[(j * kNC + c) * 2 + 1] = s[c][j].lo;
        else p[(j * kNC + c) * 2 + 1] = R(0);
      }
  }

  __device__ __forceinline__ void add_partial(const R* p) {
#pragma unroll
    for (int j = 0; j < V; ++j)
#pragma unroll
      for (int c = 0; c < kNC; ++c)
        s[c][j].add_comp(__ldcg(p + (j * kNC + c) * 2), __ldcg(p + (j * kNC + c) * 2 + 1));
  }
};

// Blocks per SM that the backward's register budget is sized for: 10 (96
// registers) with 32-byte slices, 12 (80) with 16-byte ones.  Training step on a
// 500,000-node Chung-Lu graph, bf16, 128 columns: 1087 us at 96 registers, 1080
// at 128, 1616 at 80 (spills); 16-byte slices 1160 at 80, 1320 at 72.
template <int DT, int E>
struct SpmmBwdBlocks {
  static constexpr int value = E * int(sizeof(typename VT<DT>::Store)) == 32 ? 10 : 12;
};

// Gather of x for the fused y sums: L2-only.
template <typename T> __device__ __forceinline__ T ld_gather(const T* p) { return __ldcg(p); }
template <> __device__ __forceinline__ __half ld_gather<__half>(const __half* p) {
  return __ushort_as_half(__ldcg(reinterpret_cast<const unsigned short*>(p)));
}
template <> __device__ __forceinline__ __nv_bfloat16 ld_gather<__nv_bfloat16>(const __nv_bfloat16* p) {
  return __ushort_as_bfloat16(__ldcg(reinterpret_cast<const unsigned short*>(p)));
}
__device__ __forceinline__ void put_y(__half& o, float v) { o = __float2half_rn(v); }
__device__ __forceinline__ void put_y(__nv_bfloat16& o, float v) { o = __float2bfloat16_rn(v); }
__device__ __forceinline__ void put_y(float& o, float v) { o = v; }
__device__ __forceinline__ void put_y(double& o, double v) { o = v; }

// y accumulator of the fused SpMM + SpMV.  For 2- and 4-byte values every
// product is exact in fp64, so an fp64 sum is at least as accurate as Dot2 in
// fp32 and costs one DFMA per term; fp64 values keep the Dot2 pair.  A
// long-row partial takes the two real slots of the column after the team's.
template <typename R> struct YAcc;
template <> struct YAcc<float> {
  double s;
  __device__ __forceinline__ void zero() { s = 0.0; }
  __device__ __forceinline__ void add_prod(float a, float b) { s = __fma_rn(double(a), double(b), s); }
  __device__ __forceinline__ void shfl_join(int m) { s = __dadd_rn(s, __shfl_xor_sync(0xffffffffu, s, m)); }
  __device__ __forceinline__ void shfl_up(int d) { s = __shfl_up_sync(0xffffffffu, s, d); }
  __device__ __forceinline__ void combine(const YAcc& o) { s = __dadd_rn(s, o.s); }
  __device__ __forceinline__ void store(float* p) const { *reinterpret_cast<double*>(p) = s; }
  __device__ __forceinline__ void add_stored(const float* p) {
    s = __dadd_rn(s, __ldcg(reinterpret_cast<const double*>(p)));
  }
  __device__ __forceinline__ float value() const { return __double2float_rn(s); }
};
template <> struct YAcc<double> {
  Comp<double> c;
  __device__ __forceinline__ void zero() { c.zero(); }
  __device__ __forceinline__ void add_prod(double a, double b) { c.add_prod(a, b); }
  __device__ __forceinline__ void shfl_join(int m) {
    const double oh = __shfl_xor_sync(0xffffffffu, c.hi, m), ol = __shfl_xor_sync(0xffffffffu, c.lo, m);
    c.add_comp(oh, ol);
  }
  __device__ __forceinline__ void shfl_up(int d) {
    c.hi = __shfl_up_sync(0xffffffffu, c.hi, d);
    c.lo = __shfl_up_sync(0xffffffffu, c.lo, d);
  }
  __device__ __forceinline__ void combine(const YAcc& o) { c.add_comp(o.c.hi, o.c.lo); }
  __device__ __forceinline__ void store(double* p) const { p[0] = c.hi; p[1] = c.lo; }
  __device__ __forceinline__ void add_stored(const double* p) { c.add_comp(__ldcg(p), __ldcg(p + 1)); }
  __device__ __forceinline__ double value() const { return c.value(); }
};

template <typename T> __device__ __forceinline__ T ld_once(const T* p) { return __ldcs(p); }
template <> __device__ __forceinline__ __half ld_once<__half>(const __half* p) {
  return __ushort_as_half(__ldcs(reinterpret_cast<const unsigned short*>(p)));
}
template <> __device__ __forceinline__ __nv_bfloat16 ld_once<__nv_bfloat16>(const __nv_bfloat16* p) {
  return __ushort_as_bfloat16(__ldcs(reinterpret_cast<const unsigned short*>(p)));
}

// Asynchronous global -> shared copies of one 4-, 8- or 16-byte element
// (cp.async): every copy of a staging pass is in flight at once, with no
// registers held; cp_async_wait_all() then __syncwarp() before reading.
template <int BYTES>
__device__ __forceinline__ void cp_async(void* dst, const void* src) {
  const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
  if constexpr (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(d), "l"(src), "n"(BYTES) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Stages values and columns [s0, s0 + cnt) (cnt <= MAXN) into the warp's
// shared slices by cp.async, every copy in flight at once; returns the
// offset of value s0 in sh_a (the values start at sh_a + the offset).  2-byte
// values move as 4-byte words from the word boundary at or below value s0's
// address (offset 1 when that is a value earlier: an odd position, or an array
// that itself starts off a word; the slice holds MAXN + 2 values).  A last value
// left alone in its word is copied by itself, and so is value 0 of an array
// that starts inside a word, so nothing before the array or past value
// s0 + cnt - 1 is read.  The caller's __syncwarp() makes the slices visible to
// all lanes.
template <typename S, int MAXN>
__device__ __forceinline__ int stage_nz(S* sh_a, int32_t* sh_c, const S* __restrict__ data,
                                        const int32_t* __restrict__ col, int64_t s0, int cnt, int lane) {
  int shift = 0;
  for (int k = lane; k < cnt; k += 32) cp_async<4>(sh_c + k, col + s0 + k);
  if constexpr (sizeof(S) >= 4) {
    for (int k = lane; k < cnt; k += 32) cp_async<int(sizeof(S))>(sh_a + k, data + s0 + k);
  } else if (cnt > 0) {
    shift = static_cast<int>(reinterpret_cast<uintptr_t>(data + s0) >> 1 & 1);
    const S* base = data + (s0 - shift);
    const int words = (cnt + shift) >> 1;
    const int alone = s0 < shift ? 1 : 0;  // value 0's word begins before the array
    for (int w = lane + alone; w < words; w += 32) cp_async<4>(sh_a + 2 * w, base + 2 * w);
    if (alone && lane == 1) sh_a[1] = ld_once(data);
    if (((cnt + shift) & 1) && lane == 0) sh_a[cnt + shift - 1] = ld_once(data + s0 + cnt - 1);
  }
  cp_async_wait_all();
  return shift;
}

// The same with values read through perm: value k of the stage is
// vals[perm[s0 + k]]; sh_p, where given, keeps those positions.  4- and 8-byte
// values are copied asynchronously too: the only waits are for their positions,
// which come four at a time (eight spill in the kernels below; through registers
// the values cost 5 % on fp64 rows of 512 bytes).  2-byte values go through
// registers, two at a time (four: bf16 backward of 128 columns, 200,000 rows of
// Poisson(20), 216 against 203 us), past L1 (201 us).
template <typename S>
__device__ __forceinline__ void stage_perm(S* sh_a, int32_t* sh_c, int32_t* sh_p, const S* __restrict__ vals,
                                           const int32_t* __restrict__ perm, const int32_t* __restrict__ col,
                                           int64_t s0, int cnt, int lane) {
  for (int k = lane; k < cnt; k += 32) cp_async<4>(sh_c + k, col + s0 + k);
  constexpr int kU = sizeof(S) >= 4 ? 4 : 2;
  for (int k0 = lane; k0 < cnt; k0 += 32 * kU) {
    int32_t q[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u)
      if (k0 + 32 * u < cnt) q[u] = ld_once(perm + s0 + k0 + 32 * u);
    if constexpr (sizeof(S) >= 4) {
#pragma unroll
      for (int u = 0; u < kU; ++u)
        if (k0 + 32 * u < cnt) cp_async<int(sizeof(S))>(sh_a + k0 + 32 * u, vals + q[u]);
    } else {
      S v[kU];
#pragma unroll
      for (int u = 0; u < kU; ++u)
        if (k0 + 32 * u < cnt) v[u] = ld_gather(vals + q[u]);
#pragma unroll
      for (int u = 0; u < kU; ++u)
        if (k0 + 32 * u < cnt) sh_a[k0 + 32 * u] = v[u];
    }
#pragma unroll
    for (int u = 0; u < kU; ++u)
      if (k0 + 32 * u < cnt && sh_p) sh_p[k0 + 32 * u] = q[u];
  }
  cp_async_wait_all();
}

// Run-local row offsets off[i] = ptr[r0 + i] - s0 for i <= nr (nr < MAXR),
// every load issued before the first store.
template <int MAXR>
__device__ __forceinline__ void stage_offsets(int32_t* sh_off, const int64_t* __restrict__ ptr, int64_t r0, int nr,
                                              int64_t s0, int lane) {
  constexpr int kQ = (MAXR + 32) / 32;
  int64_t v[kQ];
#pragma unroll
  for (int q = 0; q < kQ; ++q) {
    const int i = lane + 32 * q;
    if (i <= nr) v[q] = __ldg(ptr + r0 + i);
  }
#pragma unroll
  for (int q = 0; q < kQ; ++q) {
    const int i = lane + 32 * q;
    if (i <= nr) sh_off[i] = static_cast<int32_t>(v[q] - s0);
  }
}

// Rows of more than this many nonzeros accumulate compensated in the types
// whose sums run in fp32 (f16, bf16, f32), whatever the plan's flags: their
// sums are the long ones.  Shorter rows keep the plan's accumulation.  The
// forward kernel uses Dot2, blocked Dot2 or fp64 sums (ChunkAcc), the backward
// fp64 sums of the exact products.
constexpr int64_t kCompensateAbove = 1024;
template <int DT, bool COMP>
constexpr bool kCompLong = !COMP && (DT == FSB_F16 || DT == FSB_BF16 || DT == FSB_F32);

// ---------------------------------------------------------------------------
// The team kernel.  Teams of T lanes (1 to 32) own a column tile, G = 32 / T
// teams per warp: T slices of 16 or 32 bytes of aligned rows, T * P pieces of
// others (Slice).
// Rows wider than the tile run as several column tiles; the tile is the
// slowest work dimension, so while one tile is in flight only that tile's
// slice of B is being gathered, and a slice that fits in L2 is read from HBM
// about once.
//
// Persistent warps stride over the work items of every tile in tile order.
// An item is either
//  * a row group: up to kRowUnits consecutive row-block units, split into runs
//    of adjacent rows.  A run (<= 256 rows, < 512 nonzeros) is staged in the
//    warp's shared memory and every team takes an equal share of its nonzeros,
//    whatever the row lengths: it finds its first row by a binary search of the
//    row offsets, sums nonzeros and writes a row at its end.  A row that
//    spans teams is finished by a segmented scan over the teams' partial sums
//    (keys: row indices) in team order;
//  * a long-row chunk: team g takes nonzeros g, g+G, ...; the team partials
//    are combined by xor-shuffles over the team index, then the chunk is
//    stored directly (one-chunk rows) or as a slot partial whose ticket's
//    last taker adds the partials in chunk order.
// FUSED: every lane also gathers x[col] beside B's row and sums y = A x for
// the team's rows (identical sums on the team's lanes; lane 0 writes y).
// PERM: value q of the matrix is data[perm[q]], as the gradient dX = A^T dY
// reads A's values; its rows over kCompensateAbove nonzeros sum in fp64.
// ---------------------------------------------------------------------------
constexpr int kRowUnits = 4;                            // row-block units per row group
constexpr int kRowStage = kRowUnits * 2 * kSpmmMaxCap;  // staged nonzeros of a run (< 512)
constexpr int kRowRows = kRowUnits * kSpmmMaxCap;       // rows of a run (<= 256)
static_assert(kSpmmBatch <= kRowStage, "the long-row batch must fit the run staging");

// Per-warp slice: staged values, columns and run-local row offsets, then
// (16-byte aligned) one parked accumulator per lane.
template <typename S>
constexpr int spmm_team_vals_bytes() {
  return ((kRowStage + 2) * int(sizeof(S)) + 15) & ~15;  // 2-byte values may start one element early
}
template <typename S>
constexpr int spmm_team_park_offset() {
  return (spmm_team_vals_bytes<S>() + kRowStage * 4 + (kRowRows + 1) * 4 + 15) & ~15;
}
template <int DT, bool COMP, int V>
constexpr int spmm_team_warp_smem_bytes() {
  using S = typename VT<DT>::Store;
  return spmm_team_park_offset<S>() + 32 * int(sizeof(SpmmAcc<DT, COMP, V>));
}

// Resident warps the register budget is sized for, in units of 8: 4 (64
// registers) for plain sums of 2- and 4-byte values, 3 (80) for 8-byte values,
// for compensated or fused sums, for 32-byte slices (bf16, 128 columns: 172
// against 195 us at 2.5 and 2 slices ahead in 242 us at 4) and for three or
// four pieces per lane (80 against 87 us at 4: 47 columns of fp32, a
// 170,001-row Chung-Lu graph) and for narrow 16-bit rows whose values come
// through perm (8 columns 60 against 51 us at 4); 2 for complex fp64 and 32-byte
// slices of fp64.
template <int DT, bool COMP, bool FUSED, int KP, int E, int P, bool PERM>
struct SpmmTeamWarps8 {
  static constexpr bool k8 = DT == FSB_F64 || DT == FSB_C64;
  static constexpr bool k32 = E * int(sizeof(typename VT<DT>::Store)) == 32;
  static constexpr bool kPerm2 = PERM && KP == kSpmmAhead && sizeof(typename VT<DT>::Store) == 2;
  static constexpr int value =
      DT == FSB_C128 ? 2 : k32 ? (k8 ? 2 : 3) : (!COMP && !FUSED && P < 3 && !k8 && !kPerm2) ? 4 : 3;
};

// Stages nonzeros [s0, s0 + cnt), cnt <= kRowStage, and returns the first value's place.
template <typename S, bool PERM>
__device__ __forceinline__ const S* stage(S* sh_a, int32_t* sh_c, const S* __restrict__ data,
                                          const int32_t* __restrict__ perm, const int32_t* __restrict__ col, int64_t s0,
                                          int cnt, int lane) {
  if constexpr (PERM) {
    stage_perm<S>(sh_a, sh_c, nullptr, data, perm, col, s0, cnt, lane);
    return sh_a;
  } else {
    return sh_a + stage_nz<S, kRowStage>(sh_a, sh_c, data, col, s0, cnt, lane);
  }
}

template <int DT, bool COMP, int V>
__device__ __forceinline__ void acc_shfl_add(SpmmAcc<DT, COMP, V>& a, int m) {
#pragma unroll
  for (int c = 0; c < SpmmAcc<DT, COMP, V>::kNC; ++c)
#pragma unroll
    for (int j = 0; j < V; ++j) {
      const auto hi = __shfl_xor_sync(0xffffffffu, a.s[c][j].hi, m);
      if constexpr (COMP) {
        const auto lo = __shfl_xor_sync(0xffffffffu, a.s[c][j].lo, m);
        a.s[c][j].add_comp(hi, lo);
      } else {
        a.s[c][j].add(hi);
      }
    }
}

// b = the accumulator of the lane `delta` below (the lane itself where there is none)
template <int DT, bool COMP, int V>
__device__ __forceinline__ void acc_shfl_up(const SpmmAcc<DT, COMP, V>& a, SpmmAcc<DT, COMP, V>& b, int delta) {
#pragma unroll
  for (int c = 0; c < SpmmAcc<DT, COMP, V>::kNC; ++c)
#pragma unroll
    for (int j = 0; j < V; ++j) {
      b.s[c][j].hi = __shfl_up_sync(0xffffffffu, a.s[c][j].hi, delta);
      if constexpr (COMP) b.s[c][j].lo = __shfl_up_sync(0xffffffffu, a.s[c][j].lo, delta);
    }
}

template <int DT, bool COMP, int V>
__device__ __forceinline__ void acc_combine(SpmmAcc<DT, COMP, V>& a, const SpmmAcc<DT, COMP, V>& b) {
#pragma unroll
  for (int c = 0; c < SpmmAcc<DT, COMP, V>::kNC; ++c)
#pragma unroll
    for (int j = 0; j < V; ++j) {
      if constexpr (COMP) a.s[c][j].add_comp(b.s[c][j].hi, b.s[c][j].lo);
      else a.s[c][j].add(b.s[c][j].hi);
    }
}

// a += t elementwise, each add an error-free TwoSum into the compensated a
template <int DT, int V>
__device__ __forceinline__ void acc_fold(SpmmAcc<DT, true, V>& a, const SpmmAcc<DT, false, V>& t) {
#pragma unroll
  for (int c = 0; c < SpmmAcc<DT, true, V>::kNC; ++c)
#pragma unroll
    for (int j = 0; j < V; ++j) a.s[c][j].add(t.s[c][j].hi);
}

// fp64 accumulator for a long row of a real type accumulated in fp32 (bf16,
// f16, f32): each product is exact in fp64 and the fp64 sum of n of them is
// within n 2^-53 sum|a||b| of the exact sum -- inside the Dot2 bound of the
// compensated fp32 sum for rows under 2^26 nonzeros, at one DFMA per term and
// no temporaries.  Partials keep the (hi, lo) fp32 pairs of SpmmAcc<DT, true>.
template <int DT, int V>
struct WideAcc {
  using S = typename VT<DT>::Store;
  using R = typename VT<DT>::Real;
  static_assert(std::is_same<R, float>::value, "fp32-accumulated real types only");
  static constexpr int kNC = 1;  // real components per element
  double s[V];

  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int j = 0; j < V; ++j) s[j] = 0.0;
  }
  __device__ __forceinline__ void add(S a, const S (&b)[V]) {
    const double ad = to_real(a);
#pragma unroll
    for (int j = 0; j < V; ++j) s[j] = fma(ad, double(to_real(b[j])), s[j]);
  }
  __device__ __forceinline__ void shfl_add(int m) {
#pragma unroll
    for (int j = 0; j < V; ++j) s[j] += __shfl_xor_sync(0xffffffffu, s[j], m);
  }
  __device__ __forceinline__ void result(S (&out)[V]) const {
#pragma unroll
    for (int j = 0; j < V; ++j) out[j] = spmm_store(__double2float_rn(s[j]), static_cast<S*>(nullptr));
  }
  __device__ __forceinline__ void store_partial(R* p) const {
#pragma unroll
    for (int j = 0; j < V; ++j) {
      const float hi = __double2float_rn(s[j]);
      p[j * 2] = hi;
      p[j * 2 + 1] = __double2float_rn(s[j] - double(hi));
    }
  }
  __device__ __forceinline__ void add_partial(const R* p) {
#pragma unroll
    for (int j = 0; j < V; ++j) s[j] += double(__ldcg(p + j * 2)) + double(__ldcg(p + j * 2 + 1));
  }
};

template <int DT, int V>
__device__ __forceinline__ void acc_shfl_add(WideAcc<DT, V>& a, int m) { a.shfl_add(m); }

// Accumulation of a long-row chunk: MODE 0 plain sums; 1 Dot2 on every term
// (plans with FSB_SPMM_COMPENSATED); 2 blocked compensation: each step's
// KA products of a team are summed plainly, then folded into a Dot2
// accumulator, so the error is at most gamma_(KA+1) * sum|a||b| plus
// the final rounding whatever the row length (the chunk and team partials
// are combined compensated as well); 3 fp64 sums of the exact products
// (WideAcc), far inside that bound.  The fp32-accumulated types' rows over
// kCompensateAbove nonzeros use 3 in column tiles of 512 bytes and in widths off
// the slices (against mode 1 there, 400,000-row Zipf matrix: fp32, 47 columns 324
// -> 297 us; bf16, 98 columns 529 -> 436 us), 2 in the other slices (fp64 sums
// cost 3-5 % on 256-byte rows).
template <int DT, int MODE, int V>
struct ChunkAcc;
template <int DT, int V>
struct ChunkAcc<DT, 0, V> { using T = SpmmAcc<DT, false, V>; };
template <int DT, int V>
struct ChunkAcc<DT, 1, V> { using T = SpmmAcc<DT, true, V>; };
template <int DT, int V>
struct ChunkAcc<DT, 2, V> { using T = SpmmAcc<DT, true, V>; };
template <int DT, int V>
struct ChunkAcc<DT, 3, V> { using T = WideAcc<DT, V>; };

// How a long row's chunk partials are joined, in fixed order.  Up to
// kJoinChunks chunks: the warp that takes the row's last ticket adds them all.
// More: the last of each group of kJoinChunks adds its group's partials into
// the group's first slot, and the last group adds the groups', so the longest
// rows (50,000 nonzeros: 196 chunks) end after two short sums instead of one
// warp's long one.  A row's ticket counts at its first slot, a group's at the
// group's second slot (a group of one takes none).
constexpr int kJoinChunks = 16;
struct ChunkJoin {
  int64_t group_slot;  // first slot of the chunk's group
  int group_size;      // chunks in it
  int members;         // partials of the row's final sum
  int64_t step;        // their distance in slots
  __device__ __forceinline__ ChunkJoin(int nch, int chunk, int64_t first) {
    const int g = chunk / kJoinChunks;
    const bool split = nch > kJoinChunks;
    group_slot = first + int64_t(g) * kJoinChunks;
    group_size = split ? min(kJoinChunks, nch - g * kJoinChunks) : 1;
    members = split ? (nch + kJoinChunks - 1) / kJoinChunks : nch;
    step = split ? kJoinChunks : 1;
  }
  __device__ __forceinline__ bool grouped() const { return group_size > 1; }
  __device__ __forceinline__ int64_t group_ticket() const { return group_slot + 1; }
};

// The warp's partial is stored: take a ticket; true for the last of `count`,
// after which every partial can be read and the ticket is zero again.
__device__ __forceinline__ bool join_ticket(int32_t* counter, int count, int lane) {
  __threadfence();
  __syncwarp();
  int ticket = 0;
  if (lane == 0) ticket = atomicAdd(counter, 1);
  ticket = __shfl_sync(0xffffffffu, ticket, 0);
  if (ticket != count - 1) return false;
  __threadfence();
  if (lane == 0) *counter = 0;  // ready for the next call
  return true;
}

// One long-row chunk of the team kernel: team g takes nonzeros g, g+G, ...,
// KA B-row slices in flight; the team partials are combined by xor-shuffles
// over the team index, then the chunk is stored directly (one-chunk rows) or
// as a slot partial whose ticket's last taker adds the partials in chunk order.
template <int DT, int MODE, bool FUSED, int KA, int E, int P, bool PERM>
__device__ __forceinline__ void team_chunk(const typename VT<DT>::Store* __restrict__ data,
                                           const int32_t* __restrict__ col,
                                           const typename VT<DT>::Store* __restrict__ B, int64_t ldb, int64_t n,
                                           typename VT<DT>::Store* __restrict__ C, int64_t ldc,
                                           const fsb_spmv_plan& plan, const fsb_spmv_unit* ud, int T, int64_t tile,
                                           const Slice<typename VT<DT>::Store, E, P>& sl, int64_t pstride,
                                           int64_t cps,
                                           const typename VT<DT>::Store* __restrict__ x,
                                           typename VT<DT>::Store* __restrict__ y, const int32_t* __restrict__ perm,
                                           typename VT<DT>::Store* sh_a, int32_t* sh_c) {
  using S = typename VT<DT>::Store;
  using R = typename VT<DT>::Real;
  constexpr int V = E * P;
  using Acc = typename ChunkAcc<DT, MODE, V>::T;
  constexpr int kER = Acc::kNC * 2;
  const int lane = threadIdx.x & 31;
  const int G = 32 / T, team = lane / T;
  const int64_t c0 = (tile * T + lane % T) * V;  // this lane's place in a slot's partials
  const int64_t s0 = __ldg(&ud->nnz_begin), s1 = __ldg(&ud->nnz_end);
  const int32_t row = __ldg(&ud->row), tag = __ldg(&ud->tag);
  const int32_t nch = __ldg(&ud->n_chunks), slot = __ldg(&ud->slot);
  const S* Bl = sl.base(B);
  Acc acc;
  acc.zero();
  YAcc<R> yacc;
  yacc.zero();
  for (int64_t b0 = s0; b0 < s1; b0 += kRowStage) {
    const int cnt = static_cast<int>(s1 - b0 < kRowStage ? s1 - b0 : int64_t(kRowStage));
    __syncwarp();
    const S* sv = stage<S, PERM>(sh_a, sh_c, data, perm, col, b0, cnt, lane);
    __syncwarp();
    for (int k = 0; k < cnt; k += KA * G) {
      S bv[KA][V];
      S xv[KA];
#pragma unroll
      for (int q = 0; q < KA; ++q) {
        const int kk = k + q * G + team;
        sl.load(Bl, static_cast<uint32_t>(sh_c[kk < cnt ? kk : cnt - 1]), ldb, bv[q]);
      }
      if constexpr (FUSED) {
        // the y terms of these KA * G items, one per lane in order
#pragma unroll
        for (int q = 0; q * 32 < KA * G; ++q) {
          const int kk = k + q * 32 + lane;
          if (q * 32 + lane < KA * G && kk < cnt) xv[q] = ld_gather(x + sh_c[kk]);
        }
      }
      if constexpr (MODE == 2) {
        SpmmAcc<DT, false, V> step;
        step.zero();
#pragma unroll
        for (int q = 0; q < KA; ++q) {
          const int kk = k + q * G + team;
          if (kk < cnt) step.add(sv[kk], bv[q]);
        }
        acc_fold(acc, step);
      } else {
#pragma unroll
        for (int q = 0; q < KA; ++q) {
          const int kk = k + q * G + team;
          if (kk < cnt) acc.add(sv[kk], bv[q]);
        }
      }
      if constexpr (FUSED) {
#pragma unroll
        for (int q = 0; q * 32 < KA * G; ++q) {
          const int kk = k + q * 32 + lane;
          if (q * 32 + lane < KA * G && kk < cnt) yacc.add_prod(to_real(sv[kk]), to_real(xv[q]));
        }
      }
    }
  }
  for (int m = T; m < 32; m <<= 1) acc_shfl_add(acc, m);  // every team now holds the chunk's sum
  if constexpr (FUSED) {
    // every lane's y terms, joined over the warp in a fixed order
    for (int m = 1; m < 32; m <<= 1) yacc.shfl_join(m);
  }
  if (nch == 1) {
    if (team == 0 && sl.nv > 0) {
      S o[V];
      acc.result(o);
      sl.store(C + int64_t(row) * ldc, o);
    }
    if constexpr (FUSED)
      if (lane == 0 && tile == 0) put_y(y[row], yacc.value());
    return;
  }
  R* part = static_cast<R*>(plan.partials);
  const int64_t first = int64_t(slot) + (tag + 1);  // slot of the row's first chunk
  // y's partial takes the column after the team's, which no lane's share reaches,
  // idle lanes (past column n) included: a fused row is at most 256 bytes, so a
  // team covers at most 128 columns of the slot's 256
  [[maybe_unused]] const int64_t yc = int64_t(T) * V;
  if (team == 0) acc.store_partial(part + (int64_t(slot) * pstride + c0) * kER);
  if constexpr (FUSED) {
    if (lane == 0 && tile == 0) yacc.store(part + (int64_t(slot) * pstride + yc) * kER);
  }
  // the sum of partials from, from + step, ... (count of them) in this order,
  // on every team
  auto total = [&](int64_t from, int64_t step, int count) {
    Acc fin;
    fin.zero();
#pragma unroll 4
    for (int c = team; c < count; c += G) fin.add_partial(part + ((from + c * step) * pstride + c0) * kER);
    for (int m = T; m < 32; m <<= 1) acc_shfl_add(fin, m);
    return fin;
  };
  auto total_y = [&](int64_t from, int64_t step, int count) {
    YAcc<R> fy;
    fy.zero();
    for (int c = 0; c < count; ++c) fy.add_stored(part + ((from + c * step) * pstride + yc) * kER);
    return fy;
  };
  const ChunkJoin join(nch, -(tag + 1), first);
  if (join.grouped()) {
    if (!join_ticket(plan.counters + join.group_ticket() * cps + tile, join.group_size, lane)) return;
    const Acc g = total(join.group_slot, 1, join.group_size);
    if (team == 0) g.store_partial(part + (join.group_slot * pstride + c0) * kER);
    if constexpr (FUSED)
      if (lane == 0 && tile == 0) total_y(join.group_slot, 1, join.group_size).store(part + (join.group_slot * pstride + yc) * kER);
  }
  if (!join_ticket(plan.counters + first * cps + tile, join.members, lane)) return;
  const Acc fin = total(first, join.step, join.members);
  if (team == 0 && sl.nv > 0) {
    S o[V];
    fin.result(o);
    sl.store(C + int64_t(row) * ldc, o);
  }
  if constexpr (FUSED)
    if (lane == 0 && tile == 0) put_y(y[row], total_y(first, join.step, join.members).value());
}

template <int DT, bool COMP, bool FUSED, int KP, int E, int P, bool PERM>
__global__ void __launch_bounds__(kMaxSpmmWarps * 32, SpmmTeamWarps8<DT, COMP, FUSED, KP, E, P, PERM>::value * 8 / kMaxSpmmWarps)
k_spmm_team(const typename VT<DT>::Store* __restrict__ data, const int32_t* __restrict__ col,
            const int64_t* __restrict__ ptr, const typename VT<DT>::Store* __restrict__ B, int64_t ldb, int64_t n,
            typename VT<DT>::Store* __restrict__ C, int64_t ldc, fsb_spmv_plan plan, int T, int64_t tiles,
            int64_t pstride, int64_t cps, const typename VT<DT>::Store* __restrict__ x,
            typename VT<DT>::Store* __restrict__ y, const int32_t* __restrict__ perm) {
  using S = typename VT<DT>::Store;
  using R = typename VT<DT>::Real;
  constexpr int V = E * P;
  using Acc = SpmmAcc<DT, COMP, V>;
  constexpr int kP = KP;
  // the KP = 6 instantiation runs 32-lane teams only (one team per warp): a
  // run's rows all end inside the team, so it has no scan and parks nothing
  constexpr bool kOneTeam = KP == kOneTeamAhead;

  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int G = 32 / T, team = lane / T, tl = lane % T;
  unsigned char* wbase = smem_raw + warp * spmm_team_warp_smem_bytes<DT, COMP, V>();
  S* sh_a = reinterpret_cast<S*>(wbase);
  int32_t* sh_c = reinterpret_cast<int32_t*>(wbase + spmm_team_vals_bytes<S>());
  int32_t* sh_off = sh_c + kRowStage;
  Acc* sh_park = reinterpret_cast<Acc*>(wbase + spmm_team_park_offset<S>()) + lane;

  const int64_t nb = plan.n_block_units;
  const uint32_t n_groups = static_cast<uint32_t>(ceil_div(nb, kRowUnits));
  const uint32_t n_items = n_groups + static_cast<uint32_t>(plan.n_units - nb);
  const uint32_t total = n_items * static_cast<uint32_t>(tiles);
  const uint32_t block_warps = blockDim.x >> 5, nwarps = gridDim.x * block_warps;

  for (uint32_t it = blockIdx.x * block_warps + warp; it < total; it += nwarps) {
    const uint32_t tile = it / n_items, item = it - tile * n_items;
    Slice<S, E, P> sl;  // pieces past N load column 0 and are not stored
    sl.set(tile, T, tl, n);
    const S* Bl = sl.base(B);
    __syncwarp();  // the staging slice of the previous item is free

    if (item < n_groups) {
      // ---------------------------------------------------------- row group
      // lanes 0 .. kRowUnits-1 hold the group's unit descriptors
      const int64_t ua = int64_t(item) * kRowUnits;
      const int nu = static_cast<int>(nb - ua < kRowUnits ? nb - ua : int64_t(kRowUnits));
      int64_t d_s0 = 0, d_s1 = 0;
      int32_t d_row = 0, d_tag = 0;
      if (lane < nu) {
        const int4* p = reinterpret_cast<const int4*>(plan.units + ua + lane);
        const int4 a = __ldg(p), b = __ldg(p + 1);
        d_s0 = (int64_t)(uint32_t)a.x | ((int64_t)a.y << 32);
        d_s1 = (int64_t)(uint32_t)a.z | ((int64_t)a.w << 32);
        d_row = b.x;
        d_tag = b.y;
      }
      int u = 0;
      while (u < nu) {
        // the run: units u .. v-1 whose rows join up (a long row between two
        // units, listed among the chunks, breaks the run)
        const int32_t r0 = __shfl_sync(0xffffffffu, d_row, u);
        const int64_t s0 = __shfl_sync(0xffffffffu, d_s0, u);
        int32_t r1 = __shfl_sync(0xffffffffu, d_tag, u);
        int64_t s1 = __shfl_sync(0xffffffffu, d_s1, u);
        int v = u + 1;
        for (; v < nu; ++v) {
          if (__shfl_sync(0xffffffffu, d_row, v) != r1) break;
          r1 = __shfl_sync(0xffffffffu, d_tag, v);
          s1 = __shfl_sync(0xffffffffu, d_s1, v);
        }
        u = v;
        const int nr = r1 - r0;
        const int cnt = static_cast<int>(s1 - s0);
        __syncwarp();
        const S* sv = stage<S, PERM>(sh_a, sh_c, data, perm, col, s0, cnt, lane);
        stage_offsets<kRowRows>(sh_off, ptr, r0, nr, s0, lane);
        __syncwarp();
        // empty rows get zero slices (one team each)
        for (int i0 = 0; i0 < nr; i0 += 32) {
          const int i = i0 + lane;
          const bool empty = i < nr && sh_off[i] == sh_off[i + 1];
          unsigned m = __ballot_sync(0xffffffffu, empty);
          for (int q = 0; m; ++q) {
            const int b = __ffs(m) - 1;
            m &= m - 1;
            if (q % G == team) {
              if (sl.nv > 0) {
                Acc z;
                z.zero();
                S o[V];
                z.result(o);
                sl.store(C + (int64_t(r0) + i0 + b) * ldc, o);
              }
              if constexpr (FUSED)
                if (tl == 0 && tile == 0) put_y(y[int64_t(r0) + i0 + b], 0.0f);
            }
          }
        }
        __syncwarp();

        // team g sums nonzeros [jb, je) of the run: an equal share whatever the
        // row lengths.  A row is written by the team holding its last nonzero;
        // the partials of a row spanning several teams are totalled by a
        // segmented scan over the teams (keys: run-local rows).
        const int per = (cnt + G - 1) / G;
        const int jb = min(team * per, cnt), je = min(jb + per, cnt);
        Acc acc;
        acc.zero();
        YAcc<R> yacc, ypark;
        yacc.zero();
        ypark.zero();
        int cur = 0;  // the row of nonzero jb: the last row whose offset is <= jb
        {
          int lo = 0, hi = nr - 1;
          while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (sh_off[mid] <= jb) lo = mid; else hi = mid - 1;
          }
          cur = lo;
        }
        int next_end = jb < je ? sh_off[cur + 1] : 0;  // where row cur ends
        bool open_start = jb < je && sh_off[cur] < jb;  // row cur began in an earlier team
        int park_row = -1;
        auto put_row = [&](const Acc& a, const YAcc<R>& ya, int r) {
          if (sl.nv > 0) {
            S o[V];
            a.result(o);
            sl.store(C + (int64_t(r0) + r) * ldc, o);
          }
          if constexpr (FUSED)
            if (tl == 0 && tile == 0) put_y(y[int64_t(r0) + r], ya.value());
        };
        for (int j0 = jb; j0 < je; j0 += kP) {
          S bv[kP][V];
          S xv[kP];
#pragma unroll
          for (int q = 0; q < kP; ++q) {  // past je: the last nonzero again, loaded and not summed
            const int j = j0 + q < je ? j0 + q : je - 1;
            sl.load(Bl, static_cast<uint32_t>(sh_c[j]), ldb, bv[q]);
            if constexpr (FUSED) xv[q] = ld_gather(x + sh_c[j]);
          }
#pragma unroll
          for (int q = 0; q < kP; ++q) {
            const int j = j0 + q;
            if (j < je) {
              if (j == next_end) {  // row cur ended before nonzero j
                if (!kOneTeam && open_start) {
                  *sh_park = acc;  // finished after the scan
                  ypark = yacc;
                  park_row = cur;
                  open_start = false;
                } else {
                  put_row(acc, yacc, cur);
                }
                acc.zero();
                yacc.zero();
                do {  // past the empty rows (already zeroed) to the row of nonzero j
                  ++cur;
                  next_end = sh_off[cur + 1];
                } while (next_end == j);
              }
              const S a = sv[j];
              acc.add(a, bv[q]);
              if constexpr (FUSED) yacc.add_prod(to_real(a), to_real(xv[q]));
            }
          }
        }
        if constexpr (kOneTeam) {  // one team walked the whole run: its last row ends here
          if (jb < je) put_row(acc, yacc, cur);
          __syncwarp();
          continue;
        }
        const bool open_end = jb < je && next_end > je;  // row cur goes on in later teams
        // inclusive segmented scan of the open-ended partials over the teams
        const int key = open_end ? cur : -1;
        Acc sc = acc;
        YAcc<R> ysc = yacc;
        if (!open_end) {
          sc.zero();
          ysc.zero();
        }
        for (int o = 1; o < G; o <<= 1) {
          Acc other;
          acc_shfl_up(sc, other, o * T);
          YAcc<R> oy = ysc;
          if constexpr (FUSED) oy.shfl_up(o * T);
          const int okey = __shfl_up_sync(0xffffffffu, key, o * T);
          if (team >= o && key >= 0 && okey == key) {
            acc_combine(sc, other);
            if constexpr (FUSED) ysc.combine(oy);
          }
        }
        Acc carry;
        acc_shfl_up(sc, carry, T);
        YAcc<R> ycarry = ysc;
        if constexpr (FUSED) ycarry.shfl_up(T);
        // the partials of earlier teams belong to the row this team began inside
        if (park_row >= 0) {
          Acc f = *sh_park;
          acc_combine(f, carry);
          if constexpr (FUSED) ypark.combine(ycarry);
          put_row(f, ypark, park_row);
        }
        if (jb < je && !open_end) {
          if (open_start) {  // this team holds the end of a row begun before it
            acc_combine(acc, carry);
            if constexpr (FUSED) yacc.combine(ycarry);
          }
          put_row(acc, yacc, cur);
        }
        __syncwarp();  // the staging slice is rewritten by the next run
      }
      continue;
    }

    // ------------------------------------------------------------ long-row chunk
    const fsb_spmv_unit* ud = plan.units + nb + (item - n_groups);
    const int32_t nch = __ldg(&ud->n_chunks);
    // rows of more than kCompensateAbove nonzeros sum compensated in the
    // fp32-accumulated types, partials and all (see ChunkAcc)
    auto chunk = [&](auto mode) {
      team_chunk<DT, decltype(mode)::value, FUSED, KP, E, P, PERM>(data, col, B, ldb, n, C, ldc, plan, ud, T, tile,
                                                                   sl, pstride, cps, x, y, perm, sh_a, sh_c);
    };
    if constexpr (COMP) {
      chunk(std::integral_constant<int, 1>());
      continue;
    }
    if constexpr (kCompLong<DT, COMP>) {
      if (int64_t(nch) * plan.chunk_nnz > kCompensateAbove) {
        constexpr bool k32 = E * int(sizeof(S)) == 32;
        if constexpr (kOneTeam || PERM || !Slice<S, E, P>::kWhole) {
          chunk(std::integral_constant<int, 3>());
        } else {
          if (k32 && !FUSED && T == 16) chunk(std::integral_constant<int, k32 && !FUSED ? 3 : 2>());
          else chunk(std::integral_constant<int, 2>());
        }
        continue;
      }
    }
    chunk(std::integral_constant<int, 0>());
  }
}

// ---------------------------------------------------------------------------
// Backward of Y = A X in one launch, over the unit plan of A^T (built with the
// SpMM window and chunk).  Nonzero q of A^T sits in row c (a column of A) and
// column r (a row of A) and is nonzero p = perm[q] of A:
//   dX[c]   += vals[p] * dY[r]      A^T dY, laid out as in k_spmm_team
//   dvals[p] = <dY[r], X[c]>        the SDDMM of dY and X on A's pattern
// The dY row slice of each nonzero is gathered once and serves both sums; A's
// values are read through perm (no transposed copy).  Work is cut as in
// k_spmm_team: teams of T lanes take equal shares of the nonzeros of a run of
// up to 4 units, whatever the row lengths (one team per row left the teams of
// short rows waiting for the longest of theirs, and single units paid the
// perm -> value -> dY chain every 50 nonzeros: bf16 training step on a
// 500,000-node Chung-Lu graph, 128 columns, 1232 -> 1087 us with 32-byte slices;
// 200,000 nodes, 64 columns 190 -> 146 us; fp32, 64 columns 210 -> 187 us; fp32,
// 128 columns on the large graph is bound by its dY traffic, 1.75 ms either
// way).  A team holds the X slice of
// its current row and loads the next row's beside the dY slices of the step in
// which the row changes.  The dot products of a step reduce across the team by
// a transpose butterfly (log2 of the step's size halving steps, then plain xor
// steps) in a fixed order; the lanes left holding a finished product write it.
// (dX alone is k_spmm_team over A^T, see spmm_backward.)  X is read with streaming loads
// and dX written with streaming stores, which keep more of the gathered dY
// rows in L2 (measured 0.5 % faster).
// ---------------------------------------------------------------------------
// dY row slices loaded ahead of the sums: 4, and 8 where one 32-lane team of
// 16-byte slices has the warp to itself (80 registers; Poisson(20) on 200,000
// rows, 4 / 8: fp32 of 100 columns 435 / 363 us, bf16 of 200 466 / 398, fp64 of
// 50 621 / 575)
constexpr int kBwdAhead = 4, kBwdOneTeamAhead = 8;

// Per-warp slice: staged values, columns, positions in A and run-local row
// offsets, then (16-byte aligned) one parked accumulator per lane.
template <typename S>
constexpr int spmm_bwd_park_offset() {
  return (spmm_team_vals_bytes<S>() + 2 * kRowStage * 4 + (kRowRows + 1) * 4 + 15) & ~15;
}
template <int DT, int V>
constexpr int spmm_bwd_warp_smem_bytes() {
  return spmm_bwd_park_offset<typename VT<DT>::Store>() + 32 * int(sizeof(SpmmAcc<DT, false, V>));
}

// Reduces d[0..M) of every lane across the T lanes of its team.  On return the
// lane holds the team sums of items first .. first + held - 1 in d[0..held),
// and `writer` is set on exactly one lane of each group holding the same items.
template <typename R, int M>
__device__ __forceinline__ void team_transpose_sum(R (&d)[M], int T, int tl, int& first, int& held, bool& writer) {
  first = 0;
  held = M;
  int m = T >> 1;
#pragma unroll
  for (int h = M / 2; h >= 1; h >>= 1) {
    if (m == 0) break;  // teams narrower than M keep M / T items per lane
    const bool up = (tl & m) != 0;
#pragma unroll
    for (int i = 0; i < h; ++i) {
      const R keep = up ? d[i + h] : d[i];
      const R send = up ? d[i] : d[i + h];
      d[i] = keep + __shfl_xor_sync(0xffffffffu, send, m);
    }
    if (up) first += h;
    held = h;
    m >>= 1;
  }
  const int rest = m;  // lanes tl and tl ^ j (j < 2 * rest) now hold the same items
  for (; m > 0; m >>= 1) d[0] += __shfl_xor_sync(0xffffffffu, d[0], m);
  writer = (tl & (2 * rest - 1)) == 0 || rest == 0;
}

// (c0, c1) += (a0 * b0, a1 * b1) in one packed fp32x2 FMA, each half rounded
// as a scalar fma.rn.
__device__ __forceinline__ void ffma2x(float& c0, float& c1, float a0, float a1, float b0, float b1) {
  unsigned long long cc, aa, bb;
  asm("mov.b64 %0, {%1, %2};" : "=l"(cc) : "f"(c0), "f"(c1));
  asm("mov.b64 %0, {%1, %2};" : "=l"(aa) : "f"(a0), "f"(a1));
  asm("mov.b64 %0, {%1, %2};" : "=l"(bb) : "f"(b0), "f"(b1));
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(cc) : "l"(aa), "l"(bb));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(c0), "=f"(c1) : "l"(cc));
}

// (c0, c1) += (lo(x) * lo(b), hi(x) * hi(b)) for packed 16-bit x and b, one
// rounding each (see fma_mixed2).
template <typename S>
__device__ __forceinline__ void fma_mixed2x(float& c0, float& c1, unsigned x, unsigned b) {
  if constexpr (std::is_same<S, __nv_bfloat16>::value) {
    asm("{\n .reg .b16 xl, xh, bl, bh;\n mov.b32 {xl, xh}, %2;\n mov.b32 {bl, bh}, %3;\n"
        " fma.rn.f32.bf16 %0, bl, xl, %0;\n fma.rn.f32.bf16 %1, bh, xh, %1;\n}"
        : "+f"(c0), "+f"(c1) : "r"(x), "r"(b));
  } else {
    asm("{\n .reg .b16 xl, xh, bl, bh;\n mov.b32 {xl, xh}, %2;\n mov.b32 {bl, bh}, %3;\n"
        " fma.rn.f32.f16 %0, bl, xl, %0;\n fma.rn.f32.f16 %1, bh, xh, %1;\n}"
        : "+f"(c0), "+f"(c1) : "r"(x), "r"(b));
  }
}

// Partial dot product of one dY slice with this lane's X slice.
template <typename S, typename R, int V>
__device__ __forceinline__ R slice_dot(const S (&b)[V], const S (&x)[V]) {
  if constexpr (sizeof(S) == 2 && V % 2 == 0) {
    unsigned xw[V / 2], bw[V / 2];
    memcpy(xw, x, sizeof(xw));
    memcpy(bw, b, sizeof(bw));
    float s0 = 0.f, s1 = 0.f;
#pragma unroll
    for (int j = 0; j < V / 2; ++j) fma_mixed2x<S>(s0, s1, xw[j], bw[j]);
    return s0 + s1;
  } else if constexpr (std::is_same<R, float>::value && V % 2 == 0) {
    float s0 = 0.f, s1 = 0.f;
#pragma unroll
    for (int j = 0; j < V; j += 2) ffma2x(s0, s1, to_real(b[j]), to_real(b[j + 1]), to_real(x[j]), to_real(x[j + 1]));
    return s0 + s1;
  } else {
    R s = R(0);
#pragma unroll
    for (int j = 0; j < V; ++j) s = fma(to_real(b[j]), to_real(x[j]), s);
    return s;
  }
}

// Team sums of d, each written once to dvals[perm of its staged entry]; item u
// of the group is staged entry base + u * stride, present when below limit.
template <typename S, typename R, int KA>
__device__ __forceinline__ void bwd_put_dots(R (&d)[KA], int base, int stride, int limit, int T, int tl,
                                             const int32_t* sh_p, S* __restrict__ dvals) {
  int first, held;
  bool writer;
  team_transpose_sum<R, KA>(d, T, tl, first, held, writer);
  if (!writer) return;
#pragma unroll
  for (int i = 0; i < KA; ++i) {
    const int k = base + (first + i) * stride;
    if (i < held && k < limit) dvals[sh_p[k]] = spmm_store(d[i], static_cast<S*>(nullptr));
  }
}

template <int DT, int E, int KP>
__global__ void __launch_bounds__(kSpmmWarps * 32, SpmmBwdBlocks<DT, E>::value)
k_spmm_bwd(const typename VT<DT>::Store* __restrict__ vals, const int32_t* __restrict__ perm,
           const int32_t* __restrict__ col, const int64_t* __restrict__ ptr,
           const typename VT<DT>::Store* __restrict__ dY, int64_t lddy, int64_t n,
           const typename VT<DT>::Store* __restrict__ X, int64_t ldx, typename VT<DT>::Store* __restrict__ dX,
           int64_t lddx, typename VT<DT>::Store* __restrict__ dvals, fsb_spmv_plan plan, int T, int64_t pstride,
           int64_t cps) {
  using S = typename VT<DT>::Store;
  using R = typename VT<DT>::Real;
  constexpr int V = E, kP = KP;
  using Acc = SpmmAcc<DT, false, V>;

  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int G = 32 / T, team = lane / T, tl = lane % T;
  unsigned char* wbase = smem_raw + warp * spmm_bwd_warp_smem_bytes<DT, V>();
  S* sh_a = reinterpret_cast<S*>(wbase);
  int32_t* sh_c = reinterpret_cast<int32_t*>(wbase + spmm_team_vals_bytes<S>());
  int32_t* sh_p = sh_c + kRowStage;
  int32_t* sh_off = sh_p + kRowStage;
  Acc* sh_park = reinterpret_cast<Acc*>(wbase + spmm_bwd_park_offset<S>()) + lane;

  const int64_t nb = plan.n_block_units;
  const uint32_t n_groups = static_cast<uint32_t>(ceil_div(nb, kRowUnits));
  const uint32_t item = blockIdx.x * kSpmmWarps + warp;
  if (item >= n_groups + static_cast<uint32_t>(plan.n_units - nb)) return;  // whole warp leaves together
  Slice<S, E, 1> sl;  // lanes past N load column 0, take no part in the dots and store nothing
  sl.set(0, T, tl, n);
  const S* Bl = sl.base(dY);
  auto load_x = [&](int64_t row, S (&out)[V]) { sl.load_once(X + row * ldx, out); };
  auto dot = [&](const S (&b)[V], const S (&x)[V]) { return sl.nv > 0 ? slice_dot<S, R, V>(b, x) : R(0); };

  if (item < n_groups) {
    // ------------------------------------------------------------ row group
    const int64_t ua = int64_t(item) * kRowUnits;
    const int nu = static_cast<int>(nb - ua < kRowUnits ? nb - ua : int64_t(kRowUnits));
    int64_t d_s0 = 0, d_s1 = 0;
    int32_t d_row = 0, d_tag = 0;
    if (lane < nu) {
      const int4* p = reinterpret_cast<const int4*>(plan.units + ua + lane);
      const int4 a = __ldg(p), b = __ldg(p + 1);
      d_s0 = (int64_t)(uint32_t)a.x | ((int64_t)a.y << 32);
      d_s1 = (int64_t)(uint32_t)a.z | ((int64_t)a.w << 32);
      d_row = b.x;
      d_tag = b.y;
    }
    int u = 0;
    while (u < nu) {  // runs of units whose rows join up, as in k_spmm_team
      const int32_t r0 = __shfl_sync(0xffffffffu, d_row, u);
      const int64_t s0 = __shfl_sync(0xffffffffu, d_s0, u);
      int32_t r1 = __shfl_sync(0xffffffffu, d_tag, u);
      int64_t s1 = __shfl_sync(0xffffffffu, d_s1, u);
      int v = u + 1;
      for (; v < nu; ++v) {
        if (__shfl_sync(0xffffffffu, d_row, v) != r1) break;
        r1 = __shfl_sync(0xffffffffu, d_tag, v);
        s1 = __shfl_sync(0xffffffffu, d_s1, v);
      }
      u = v;
      const int nr = r1 - r0;
      const int cnt = static_cast<int>(s1 - s0);
      __syncwarp();  // the staging slice of the previous run is free
      stage_offsets<kRowRows>(sh_off, ptr, r0, nr, s0, lane);
      stage_perm<S>(sh_a, sh_c, sh_p, vals, perm, col, s0, cnt, lane);
      __syncwarp();
      auto put_row = [&](const Acc& a, int r) {
        if (sl.nv > 0) {
          S o[V];
          a.result(o);
          sl.store(dX + (int64_t(r0) + r) * lddx, o);
        }
      };
      for (int i0 = 0; i0 < nr; i0 += 32) {  // empty rows get zero slices (one team each)
        const int i = i0 + lane;
        unsigned m = __ballot_sync(0xffffffffu, i < nr && sh_off[i] == sh_off[i + 1]);
        for (int q = 0; m; ++q) {
          const int b = __ffs(m) - 1;
          m &= m - 1;
          if (q % G == team) {
            Acc z;
            z.zero();
            put_row(z, i0 + b);
          }
        }
      }
      if (cnt == 0) continue;

      // team g takes nonzeros [jb, je) of the run (see k_spmm_team)
      const int per = (cnt + G - 1) / G;
      const int jb = min(team * per, cnt), je = min(jb + per, cnt);
      Acc acc;
      acc.zero();
      int cur = 0;  // the row of nonzero jb: the last row whose offset is <= jb
      {
        int lo = 0, hi = nr - 1;
        while (lo < hi) {
          const int mid = (lo + hi + 1) >> 1;
          if (sh_off[mid] <= jb) lo = mid; else hi = mid - 1;
        }
        cur = lo;
      }
      int next_end = jb < je ? sh_off[cur + 1] : cnt;
      bool open_start = jb < je && sh_off[cur] < jb;
      int park_row = -1;
      S xa[V], xb[V];
      if (jb < je) load_x(int64_t(r0) + cur, xa);
      // every team takes the same number of steps: the butterflies are warp-wide
      for (int t = 0; t < per; t += kP) {
        const int j0 = jb + t;
        S bv[kP][V];
        R d[kP];
#pragma unroll
        for (int q = 0; q < kP; ++q)  // past je: some nonzero, loaded and not summed
          sl.load(Bl, static_cast<uint32_t>(sh_c[min(j0 + q, max(je - 1, 0))]), lddy, bv[q]);
        int xrow = -1;
        if (next_end < je && next_end < j0 + kP) {  // the row changes in this step
          xrow = cur + 1;
          while (sh_off[xrow + 1] == next_end) ++xrow;
          load_x(int64_t(r0) + xrow, xb);
        }
#pragma unroll
        for (int q = 0; q < kP; ++q) {
          const int j = j0 + q;
          d[q] = R(0);
          if (j < je) {
            if (j == next_end) {  // row cur ended before nonzero j
              if (open_start) {
                *sh_park = acc;  // finished after the scan
                park_row = cur;
                open_start = false;
              } else {
                put_row(acc, cur);
              }
              acc.zero();
              do {
                ++cur;
                next_end = sh_off[cur + 1];
              } while (next_end == j);
              if (cur == xrow) memcpy(xa, xb, sizeof(xa));
              else load_x(int64_t(r0) + cur, xa);
            }
            acc.add(sh_a[j], bv[q]);
            d[q] = dot(bv[q], xa);
          }
        }
        bwd_put_dots<S, R, kP>(d, j0, 1, je, T, tl, sh_p, dvals);
      }
      // inclusive segmented scan of the open-ended partials over the teams
      const bool open_end = jb < je && next_end > je;  // row cur goes on in later teams
      const int key = open_end ? cur : -1;
      Acc sc = acc;
      if (!open_end) sc.zero();
      for (int o = 1; o < G; o <<= 1) {
        Acc other;
        acc_shfl_up(sc, other, o * T);
        const int okey = __shfl_up_sync(0xffffffffu, key, o * T);
        if (team >= o && key >= 0 && okey == key) acc_combine(sc, other);
      }
      Acc carry;
      acc_shfl_up(sc, carry, T);
      if (park_row >= 0) {
        Acc f = *sh_park;
        acc_combine(f, carry);
        put_row(f, park_row);
      }
      if (jb < je && !open_end) {
        if (open_start) acc_combine(acc, carry);
        put_row(acc, cur);
      }
    }
    return;
  }

  // ------------------------------------------------------------ long-row chunk
  const fsb_spmv_unit* ud = plan.units + nb + (item - n_groups);
  const int64_t s0 = __ldg(&ud->nnz_begin), s1 = __ldg(&ud->nnz_end);
  const int32_t row = __ldg(&ud->row), tag = __ldg(&ud->tag);
  const int32_t nch = __ldg(&ud->n_chunks), slot = __ldg(&ud->slot);
  const int64_t c0 = int64_t(tl) * V;  // this lane's place in a slot's partials
  S xs[V];
  load_x(row, xs);
  // WIDE (rows over kCompensateAbove nonzeros, see kCompLong): fp64 sums of the
  // exact products; else plain sums
  auto run_chunk = [&](auto wide) {
    using A2 = typename std::conditional<decltype(wide)::value, WideAcc<DT, V>, Acc>::type;
    constexpr int kER = A2::kNC * 2;
    A2 acc;
    acc.zero();
    for (int64_t b0 = s0; b0 < s1; b0 += kRowStage) {
      const int cnt = static_cast<int>(s1 - b0 < kRowStage ? s1 - b0 : int64_t(kRowStage));
      __syncwarp();
      stage_perm<S>(sh_a, sh_c, sh_p, vals, perm, col, b0, cnt, lane);
      __syncwarp();
      for (int k = 0; k < cnt; k += kP * G) {
        S bv[kP][V];
        R d[kP];
#pragma unroll
        for (int q = 0; q < kP; ++q) {
          const int kk = k + q * G + team;
          sl.load(Bl, static_cast<uint32_t>(sh_c[kk < cnt ? kk : cnt - 1]), lddy, bv[q]);
        }
#pragma unroll
        for (int q = 0; q < kP; ++q) {
          const int kk = k + q * G + team;
          if (kk < cnt) acc.add(sh_a[kk], bv[q]);
          d[q] = dot(bv[q], xs);
        }
        bwd_put_dots<S, R, kP>(d, k + team, G, cnt, T, tl, sh_p, dvals);
      }
    }
    for (int m = T; m < 32; m <<= 1) acc_shfl_add(acc, m);  // every team now holds the chunk's sum
    auto put = [&](const A2& a) {
      if (team == 0 && sl.nv > 0) {
        S o[V];
        a.result(o);
        sl.store(dX + int64_t(row) * lddx, o);
      }
    };
    if (nch == 1) {
      put(acc);
      return;
    }
    R* part = static_cast<R*>(plan.partials);
    const int64_t first = int64_t(slot) + (tag + 1);
    if (team == 0) acc.store_partial(part + (int64_t(slot) * pstride + c0) * kER);
    auto total = [&](int64_t from, int64_t stride, int count) {
      A2 fin;
      fin.zero();
#pragma unroll 4
      for (int c = team; c < count; c += G) fin.add_partial(part + ((from + c * stride) * pstride + c0) * kER);
      for (int m = T; m < 32; m <<= 1) acc_shfl_add(fin, m);
      return fin;
    };
    const ChunkJoin join(nch, -(tag + 1), first);
    if (join.grouped()) {
      if (!join_ticket(plan.counters + join.group_ticket() * cps, join.group_size, lane)) return;
      const A2 g = total(join.group_slot, 1, join.group_size);
      if (team == 0) g.store_partial(part + (join.group_slot * pstride + c0) * kER);
    }
    if (!join_ticket(plan.counters + first * cps, join.members, lane)) return;
    put(total(first, join.step, join.members));
  };
  if constexpr (kCompLong<DT, false>) {
    if (int64_t(nch) * plan.chunk_nnz > kCompensateAbove) {
      run_chunk(std::true_type());
      return;
    }
  }
  run_chunk(std::false_type());
}

}  // namespace
}  // namespace fsb

namespace fsb {
namespace {

inline int64_t spmm_real_bytes(int dtype) {
  switch (dtype) {
    case FSB_F16: case FSB_BF16: case FSB_F32: case FSB_C64: return 4;
    case FSB_F64: case FSB_C128: return 8;
    default: return -1;
  }
}

inline int64_t spmm_elem_bytes(int dtype) {
  switch (dtype) {
    case FSB_F16: case FSB_BF16: return 2;
    case FSB_F32: return 4;
    case FSB_F64: case FSB_C64: return 8;
    case FSB_C128: return 16;
    default: return -1;
  }
}

inline int64_t spmm_pstride(int64_t n) { return ceil_div(n, 256) * 256; }
// Tickets per slot: one per column tile.  The narrowest tile of any kernel is
// one 16-byte slice, so ceil(n * elem / 16) covers every tiling.
inline int64_t spmm_cps_bytes(int64_t n, int64_t elem) { return n > 0 ? ceil_div(n * elem, 16) : 1; }
template <int DT>
inline int64_t spmm_cps(int64_t n) { return spmm_cps_bytes(n, sizeof(typename VT<DT>::Store)); }

// Column tile of the team kernel, in bytes (a power of two, 16 .. 512).  The
// default is the whole row (rounded up to a power of two of 16-byte slices) up
// to 512 bytes.  A positive `hint` (fsb_spmv_plan.tile_bytes) asks for
// narrower tiles: then only a tile's slice of B (n_cols x tile bytes) is
// gathered at a time, which stays in L2 when it fits, at the cost of reading
// A once per tile.  On B200 the whole-row tile measured faster for every
// width up to 512 bytes on 1,000,000-row matrices (fp32 N = 128: 2.4 ms
// against 3.6 ms at 128-byte and 5.5 ms at 64-byte tiles), so narrow tiles
// are opt-in.
inline int spmm_team_tile_bytes(int64_t row_bytes, int32_t hint) {
  int w = 16;
  while (w < row_bytes && w < 512) w *= 2;
  if (hint > 0) {
    int h = 16;
    while (h < hint && h < 512) h *= 2;
    return h < w ? h : w;
  }
  return w;
}

// Warps per block of the team kernel (see kSpmmWarps).  Eight in the fused kernel
// of the batched step: its persistent grid levels the items itself (256 uneven
// matrices: 1.90 against 2.02 ms at 2).  More than two also in these 16-byte
// slices of 8- and 16-byte values, whose rows begin inside 32-byte sectors or
// take one or two: blocks of two fill the SM's shared memory with warps and leave
// L1 too small to hold a sector until its other half is read.  us at 2 / 4 / 8
// warps; Poisson(20) on 200,000 rows, or Poisson(8) on 1 M rows (*):
//  * fp64 but for rows of 96 bytes: 2 columns 45 / 46 / 41, 8 columns 187 / 188 /
//    133 *, 14 columns 351 / 352 / 233 *, 98 columns 658 / 659 / 510, Dot2 742 / 746
//    / 671; 12 columns 64 / 64 / 72 and 201 / 204 / 219 *.  In between two can be
//    the faster while B is in L2 (34 columns 177 / 178 / 203, 10 columns 62 / 62 /
//    68 but 269 / 271 / 204 *);
//  * c64 rows under 128 bytes: 2 columns 45 / 45 / 41, 8 columns 184 / 184 / 135 *;
//    24 columns 108 / 109 / 119;
//  * narrow tiles of wide rows (tile_bytes): fp64 98 columns 1034 / 1033 / 698, c64
//    1002 / 1002 / 702;
//  * c128 rows of one or two slices: 2 columns 145 / 123 / 128 *; and of more than
//    one tile off the sectors: 97 columns 1401 / 1293 / 1312; Dot2 1863 / 1881 /
//    1923, 8 columns 285 / 301 / 307 *.
template <int DT, bool COMP, bool FUSED, int E, int P>
inline int spmm_block_warps(int T, int64_t tiles, int64_t n, int64_t ldb) {
  constexpr int s = int(sizeof(typename VT<DT>::Store));
  if constexpr (FUSED) return kMaxSpmmWarps;
  if constexpr (s == 16) {
    const bool off = tiles > 1 && (n % 2 != 0 || ldb % 2 != 0);
    return !COMP && (n <= 2 || off) ? 4 : kSpmmWarps;
  }
  if constexpr (s == 8 && P == 1 && E * s == 16) {
    const bool tiled = tiles > 1 && T < 32;
    if (tiled || (DT == FSB_F64 ? n * s != 96 : n * s < 128)) return kMaxSpmmWarps;
  }
  return kSpmmWarps;
}

// The team kernel: one work item per warp, the items of every tile in tile
// order (tiles of T slices), so the blocks of one tile run together; with
// FSB_SPMM_PERSISTENT, the resident blocks, whose warps stride over the items
// in the same order.
template <int DT, bool COMP, bool FUSED = false, int E = 16 / int(sizeof(typename VT<DT>::Store)), int P = 1,
          bool PERM = false>
int spmm_launch_team(const void* data, const int32_t* idx, const int64_t* ptr, const void* B, int64_t ldb, int64_t n,
                     void* C, int64_t ldc, const fsb_spmv_plan& plan, int T, int64_t tiles, cudaStream_t st,
                     const void* x = nullptr, void* y = nullptr, const int32_t* perm = nullptr) {
  using S = typename VT<DT>::Store;
  constexpr bool kAligned = P == 1 && E * int(sizeof(S)) >= 16, k32 = E * int(sizeof(S)) == 32;
  const int warps = spmm_block_warps<DT, COMP, FUSED, E, P>(T, tiles, n, ldb);
  constexpr size_t kWarpSmem = size_t(spmm_team_warp_smem_bytes<DT, COMP, E * P>());
  const size_t smem = kWarpSmem * warps;
  const int wide = (kAligned && !k32 && !FUSED && T == 32) ? 1 : 0;
  auto kern = k_spmm_team<DT, COMP, FUSED, FUSED && k32 ? kFused32Ahead : kSpmmAhead, E, P, PERM>;
  if constexpr (kAligned && !k32 && !FUSED)
    if (wide) kern = k_spmm_team<DT, COMP, FUSED, kOneTeamAhead, E, P, PERM>;
  if (smem > 48 * 1024) {  // opt in to the larger dynamic shared memory once per kernel and device
    static std::atomic<uint64_t> done[2];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
      (void)cudaGetLastError();
      return FSB_ERR_CUDA;
    }
    const uint64_t bit = uint64_t(1) << (dev & 63);
    if (!(done[wide].load(std::memory_order_acquire) & bit)) {
      if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               int(kWarpSmem * kMaxSpmmWarps)) != cudaSuccess) {
        (void)cudaGetLastError();
        return FSB_ERR_CUDA;
      }
      done[wide].fetch_or(bit, std::memory_order_release);
    }
  }
  const int64_t nb = plan.n_block_units;
  const int64_t items = (ceil_div(nb, kRowUnits) + (plan.n_units - nb)) * tiles;
  int64_t blocks = ceil_div(items, warps);  // one work item per warp, tiles in block order
  if (items >= (int64_t(1) << 32) || blocks > INT32_MAX || (kAligned && ldb > UINT32_MAX)) return FSB_ERR_UNSUPPORTED;
  if (blocks < 1) return FSB_OK;
  if (plan.flags & FSB_SPMM_PERSISTENT) {  // the resident blocks; warps stride over the items
    static std::atomic<int64_t> resident[2][kMaxSpmmWarps + 1][64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
      (void)cudaGetLastError();
      return FSB_ERR_CUDA;
    }
    int64_t r = resident[wide][warps][dev].load(std::memory_order_acquire);
    if (r == 0) {
      int per_sm = 0, sms = 0;
      if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, warps * 32, smem) != cudaSuccess ||
          cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || per_sm < 1 ||
          sms < 1) {
        (void)cudaGetLastError();
        return FSB_ERR_CUDA;
      }
      r = int64_t(per_sm) * sms;
      resident[wide][warps][dev].store(r, std::memory_order_release);
    }
    if (blocks > r) blocks = r;
  }
  kern<<<(unsigned)blocks, warps * 32, smem, st>>>(
      static_cast<const S*>(data), idx, ptr, static_cast<const S*>(B), ldb, n,
      static_cast<S*>(C), ldc, plan, T, tiles, spmm_pstride(n), spmm_cps<DT>(n), static_cast<const S*>(x),
      static_cast<S*>(y), perm);
  FSB_LAUNCH_CHECK();
  return FSB_OK;
}

// Whether the rows of B and C are whole slices of `bytes` bytes on such boundaries.
template <typename S>
bool spmm_whole_slices(int bytes, int64_t n, const void* B, int64_t ldb, const void* C, int64_t ldc) {
  const int64_t v = bytes / int64_t(sizeof(S));
  return n % v == 0 && ldb % v == 0 && ldc % v == 0 && reinterpret_cast<uintptr_t>(B) % bytes == 0 &&
         reinterpret_cast<uintptr_t>(C) % bytes == 0;
}

// C = A B and y = A x in one launch: the team kernel with the fused y sums.
// Real types, whole aligned slices and rows of at most 256 bytes, which leave
// y's long-row partial a column of its own in the scratch slots (team_chunk).
template <int DT>
int spmm_spmv_fused(const void* data, const int32_t* idx, const int64_t* ptr, const void* B, int64_t ldb, int64_t n,
                    void* C, int64_t ldc, const void* x, void* y, const fsb_spmv_plan& plan, cudaStream_t st) {
  using S = typename VT<DT>::Store;
  constexpr int kVmax = 16 / int(sizeof(S));
  if constexpr (VT<DT>::kComplex) {
    return FSB_ERR_UNSUPPORTED;
  } else {
    if (!(n * int64_t(sizeof(S)) <= 256 && spmm_whole_slices<S>(16, n, B, ldb, C, ldc)))
      return FSB_ERR_UNSUPPORTED;
    if constexpr (kSlice32<DT, false, true>) {
      if (!(plan.flags & FSB_SPMM_COMPENSATED) && n * int64_t(sizeof(S)) >= kSlice32Row<true> &&
          spmm_whole_slices<S>(32, n, B, ldb, C, ldc)) {
        int T = 1;
        while (int64_t(T) * 2 * kVmax < n) T *= 2;
        return spmm_launch_team<DT, false, true, 2 * kVmax>(data, idx, ptr, B, ldb, n, C, ldc, plan, T, 1, st, x, y);
      }
    }
    int T = 1;
    while (int64_t(T) * kVmax < n) T *= 2;
    if (plan.flags & FSB_SPMM_COMPENSATED)
      return spmm_launch_team<DT, true, true>(data, idx, ptr, B, ldb, n, C, ldc, plan, T, 1, st, x, y);
    return spmm_launch_team<DT, false, true>(data, idx, ptr, B, ldb, n, C, ldc, plan, T, 1, st, x, y);
  }
}

// dX = A^T dY and dvals = SDDMM(dY, X) on A's pattern in one launch of
// k_spmm_bwd; without dvals, k_spmm_team over A^T with A's values read through
// perm, the same sums in the same order.  (The dots' kernel without its dots held
// the positions and fewer warps for nothing: Poisson(20) on 200,000 rows, fp64 of
// 64 columns 424 -> 266 us, fp32 of 100 columns 293 -> 239 us, bf16 of 200 290 ->
// 241 us; 16-bit rows of up to 64 bytes 49 -> 51 us at 8 columns.)  Real types,
// 16-byte aligned rows of at most 512 bytes whose width n is a multiple of 16 /
// sizeof(value); plain sums, fp64 sums on rows over kCompensateAbove nonzeros for
// the fp32-accumulated types.
template <int DT>
int spmm_backward(const void* vals, const int32_t* perm, const int32_t* idx, const int64_t* ptr, const void* dY,
                  int64_t lddy, const void* X, int64_t ldx, int64_t n, void* dX, int64_t lddx, void* dvals,
                  const fsb_spmv_plan& plan, cudaStream_t st) {
  using S = typename VT<DT>::Store;
  constexpr int kVmax = 16 / int(sizeof(S));
  if constexpr (VT<DT>::kComplex) {
    return FSB_ERR_UNSUPPORTED;
  } else {
    auto whole = [&](int bytes) {
      return spmm_whole_slices<S>(bytes, n, dY, lddy, dX, lddx) &&
             (!dvals || (ldx * int64_t(sizeof(S)) % bytes == 0 && reinterpret_cast<uintptr_t>(X) % bytes == 0));
    };
    if (n * int64_t(sizeof(S)) > 512 || lddy > UINT32_MAX || !whole(16) || (plan.flags & FSB_SPMM_COMPENSATED))
      return FSB_ERR_UNSUPPORTED;
    auto run = [&](auto e) {
      constexpr int E = decltype(e)::value;
      int T = 1;
      while (int64_t(T) * E < n) T *= 2;
      if (!dvals)
        return spmm_launch_team<DT, false, false, E, 1, true>(vals, idx, ptr, dY, lddy, n, dX, lddx, plan, T, 1, st,
                                                              nullptr, nullptr, perm);
      const int64_t items = ceil_div(plan.n_block_units, kRowUnits) + (plan.n_units - plan.n_block_units);
      const unsigned blocks = (unsigned)ceil_div(items, kSpmmWarps);
      const size_t smem = size_t(spmm_bwd_warp_smem_bytes<DT, E>()) * kSpmmWarps;
      auto kern = k_spmm_bwd<DT, E, kBwdAhead>;
      if constexpr (E == kVmax)
        if (T == 32) kern = k_spmm_bwd<DT, E, kBwdOneTeamAhead>;
      kern<<<blocks, kSpmmWarps * 32, smem, st>>>(
          static_cast<const S*>(vals), perm, idx, ptr, static_cast<const S*>(dY), lddy, n, static_cast<const S*>(X),
          ldx, static_cast<S*>(dX), lddx, static_cast<S*>(dvals), plan, T, spmm_pstride(n), spmm_cps<DT>(n));
      FSB_LAUNCH_CHECK();
      return int(FSB_OK);
    };
    if (n * int64_t(sizeof(S)) >= kSlice32Row<false> && whole(32)) return run(std::integral_constant<int, 2 * kVmax>());
    return run(std::integral_constant<int, kVmax>());
  }
}

// Rows of E-element pieces (see Slice): teams of T lanes with P pieces of at
// most 16 bytes together, as few lanes as hold a tile's pieces, so that a warp
// runs as many teams as it can; at most 32 * kMaxP pieces per column tile,
// spread evenly over the tiles.  One warp per unit and 32-column tile, which
// this replaced, left most lanes idle on narrow rows and ran two passes at 33
// to 64 columns (fp32 on a 170,001-row Chung-Lu graph, 47 columns: 208 -> 89
// us; 300,000 rows, 5 columns: 219 -> 84 us; 129 columns: 1543 -> 872 us).
template <int DT, bool COMP, int E>
int spmm_launch_pieces(const void* data, const int32_t* idx, const int64_t* ptr, const void* B, int64_t ldb, int64_t n,
                       void* C, int64_t ldc, const fsb_spmv_plan& plan, cudaStream_t st) {
  constexpr int kFit = 16 / (E * int(sizeof(typename VT<DT>::Store)));
  constexpr int kMaxP = kFit < 4 ? kFit : 4;
  const int64_t pieces = n / E;
  const int per = static_cast<int>(ceil_div(pieces, ceil_div(pieces, 32 * kMaxP)));
  int T = 1;
  while (T * kMaxP < per) T *= 2;
  const int P = (per + T - 1) / T;
  const int64_t tiles = ceil_div(pieces, int64_t(T) * P);
  if (n > INT32_MAX || tiles * T * P * E > spmm_pstride(n)) return FSB_ERR_UNSUPPORTED;
  if constexpr (kMaxP >= 4) {
    if (P == 4) return spmm_launch_team<DT, COMP, false, E, 4>(data, idx, ptr, B, ldb, n, C, ldc, plan, T, tiles, st);
    if (P == 3) return spmm_launch_team<DT, COMP, false, E, 3>(data, idx, ptr, B, ldb, n, C, ldc, plan, T, tiles, st);
  }
  if constexpr (kMaxP >= 2)
    if (P == 2) return spmm_launch_team<DT, COMP, false, E, 2>(data, idx, ptr, B, ldb, n, C, ldc, plan, T, tiles, st);
  return spmm_launch_team<DT, COMP, false, E, 1>(data, idx, ptr, B, ldb, n, C, ldc, plan, T, tiles, st);
}

template <int DT, bool COMP>
int spmm_dispatch(const void* data, const int32_t* idx, const int64_t* ptr, const void* B, int64_t ldb, int64_t n,
                  void* C, int64_t ldc, const fsb_spmv_plan& plan, cudaStream_t st) {
  using S = typename VT<DT>::Store;
  constexpr int kVmax = 16 / int(sizeof(S));
  // rows of whole, aligned slices: teams of T lanes over column tiles of T
  // slices (spmm_team_tile_bytes)
  if (spmm_whole_slices<S>(16, n, B, ldb, C, ldc) && ldb <= UINT32_MAX && n <= INT32_MAX) {
    const int w = spmm_team_tile_bytes(n * int64_t(sizeof(S)), plan.tile_bytes);
    if constexpr (kSlice32<DT, COMP, false>)
      if (w >= kSlice32Row<false> && spmm_whole_slices<S>(32, n, B, ldb, C, ldc))
        return spmm_launch_team<DT, COMP, false, 2 * kVmax>(data, idx, ptr, B, ldb, n, C, ldc, plan, w / 32,
                                                            ceil_div(n, int64_t(w / 32) * 2 * kVmax), st);
    const int T = w / 16;
    return spmm_launch_team<DT, COMP>(data, idx, ptr, B, ldb, n, C, ldc, plan, T, ceil_div(n, int64_t(T) * kVmax),
                                      st);
  }
  // other widths and addresses: pieces of 8 or 4 bytes where everything is a
  // multiple of them, else of one element
  auto fits = [&](int e) {
    const uintptr_t a = uintptr_t(e) * sizeof(S);
    return n % e == 0 && ldb % e == 0 && ldc % e == 0 && reinterpret_cast<uintptr_t>(B) % a == 0 &&
           reinterpret_cast<uintptr_t>(C) % a == 0;
  };
  if constexpr (sizeof(S) == 2) {
    if (fits(4)) return spmm_launch_pieces<DT, COMP, 4>(data, idx, ptr, B, ldb, n, C, ldc, plan, st);
    if (fits(2)) return spmm_launch_pieces<DT, COMP, 2>(data, idx, ptr, B, ldb, n, C, ldc, plan, st);
  } else if constexpr (sizeof(S) == 4) {
    if (fits(2)) return spmm_launch_pieces<DT, COMP, 2>(data, idx, ptr, B, ldb, n, C, ldc, plan, st);
  }
  if constexpr (sizeof(S) == 16) return FSB_ERR_UNSUPPORTED;  // an element is a slice: B or C is misaligned
  else return spmm_launch_pieces<DT, COMP, 1>(data, idx, ptr, B, ldb, n, C, ldc, plan, st);
}

template <int DT>
int spmm_mode(const void* data, const int32_t* idx, const int64_t* ptr, const void* B, int64_t ldb, int64_t n,
              void* C, int64_t ldc, const fsb_spmv_plan& plan, cudaStream_t st) {
  if (plan.flags & FSB_SPMM_COMPENSATED)
    return spmm_dispatch<DT, true>(data, idx, ptr, B, ldb, n, C, ldc, plan, st);
  return spmm_dispatch<DT, false>(data, idx, ptr, B, ldb, n, C, ldc, plan, st);
}

}  // namespace
}  // namespace fsb

using namespace fsb;

extern "C" {

int32_t fsb_spmm_default_cap(int dtype) { (void)dtype; return kSpmmMaxCap; }

int32_t fsb_spmm_default_chunk(int dtype) { (void)dtype; return 2 * kSpmmBatch; }

int fsb_spmm_scratch_layout(int dtype, int64_t n, int64_t* partial_bytes_per_slot, int64_t* tickets_per_slot) {
  const int64_t rb = spmm_real_bytes(dtype);
  if (rb < 0) return FSB_ERR_UNSUPPORTED;
  if (n < 0 || !partial_bytes_per_slot || !tickets_per_slot) return FSB_ERR_INVALID_ARG;
  const int64_t comps = (dtype == FSB_C64 || dtype == FSB_C128) ? 2 : 1;
  *partial_bytes_per_slot = spmm_pstride(n) * comps * 2 * rb;
  *tickets_per_slot = spmm_cps_bytes(n, spmm_elem_bytes(dtype));
  return FSB_OK;
}

int fsb_spmm_csr(int dtype, const void* data, const int32_t* indices, const int64_t* indptr, int64_t n_rows,
                 int64_t n_cols, const void* B, int64_t ldb, int64_t n, void* C, int64_t ldc,
                 const fsb_spmv_plan* plan, void* stream) {
  if (!plan || n_rows < 0 || n_cols < 0 || n < 0 || ldb < n || ldc < n) return FSB_ERR_INVALID_ARG;
  if (n_rows == 0 || n == 0) return FSB_OK;
  if (!indptr || !C || !plan->units || plan->n_units < 1 || plan->cap < 1 || plan->cap > kSpmmMaxCap ||
      plan->chunk_nnz < kSpmmBatch || plan->chunk_nnz % kSpmmBatch != 0 || plan->n_slots < 0 ||
      (plan->n_slots > 0 && (!plan->partials || !plan->counters)))
    return FSB_ERR_INVALID_ARG;
  if (n_cols > 0 && !B) return FSB_ERR_INVALID_ARG;
  if (plan->n_units >= INT32_MAX) return FSB_ERR_UNSUPPORTED;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  switch (dtype) {
    case FSB_F16: return spmm_mode<FSB_F16>(data, indices, indptr, B, ldb, n, C, ldc, *plan, st);
    case FSB_BF16: return spmm_mode<FSB_BF16>(data, indices, indptr, B, ldb, n, C, ldc, *plan, st);
    case FSB_F32: return spmm_mode<FSB_F32>(data, indices, indptr, B, ldb, n, C, ldc, *plan, st);
    case FSB_F64: return spmm_mode<FSB_F64>(data, indices, indptr, B, ldb, n, C, ldc, *plan, st);
    case FSB_C64: return spmm_mode<FSB_C64>(data, indices, indptr, B, ldb, n, C, ldc, *plan, st);
    case FSB_C128: return spmm_mode<FSB_C128>(data, indices, indptr, B, ldb, n, C, ldc, *plan, st);
    default: return FSB_ERR_UNSUPPORTED;
  }
}

int fsb_spmm_spmv_csr(int dtype, const void* data, const int32_t* indices, const int64_t* indptr, int64_t n_rows,
                      int64_t n_cols, const void* B, int64_t ldb, int64_t n, void* C, int64_t ldc, const void* x,
                      void* y, const fsb_spmv_plan* plan, void* stream) {
  if (!plan || n_rows < 0 || n_cols < 0 || n < 1 || ldb < n || ldc < n || !x || !y) return FSB_ERR_INVALID_ARG;
  if (n_rows == 0) return FSB_OK;
  if (!indptr || !C || !plan->units || plan->n_units < 1 || plan->cap < 1 || plan->cap > kSpmmMaxCap ||
      plan->chunk_nnz < kSpmmBatch || plan->chunk_nnz % kSpmmBatch != 0 || plan->n_slots < 0 ||
      (plan->n_slots > 0 && (!plan->partials || !plan->counters)))
    return FSB_ERR_INVALID_ARG;
  if (n_cols > 0 && !B) return FSB_ERR_INVALID_ARG;
  if (plan->n_units >= INT32_MAX) return FSB_ERR_UNSUPPORTED;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  switch (dtype) {
    case FSB_F16: return spmm_spmv_fused<FSB_F16>(data, indices, indptr, B, ldb, n, C, ldc, x, y, *plan, st);
    case FSB_BF16: return spmm_spmv_fused<FSB_BF16>(data, indices, indptr, B, ldb, n, C, ldc, x, y, *plan, st);
    case FSB_F32: return spmm_spmv_fused<FSB_F32>(data, indices, indptr, B, ldb, n, C, ldc, x, y, *plan, st);
    case FSB_F64: return spmm_spmv_fused<FSB_F64>(data, indices, indptr, B, ldb, n, C, ldc, x, y, *plan, st);
    default: return FSB_ERR_UNSUPPORTED;
  }
}

int fsb_spmm_csr_backward(int dtype, const void* vals, const int32_t* perm, const int32_t* t_indices,
                          const int64_t* t_indptr, int64_t n_rows, int64_t n_cols, const void* dY, int64_t lddy,
                          const void* X, int64_t ldx, int64_t n, void* dX, int64_t lddx, void* dvals,
                          const fsb_spmv_plan* t_plan, void* stream) {
  const fsb_spmv_plan* plan = t_plan;
  if (!plan || n_rows < 0 || n_cols < 0 || n < 0 || lddy < n || lddx < n || !dX || (dvals && (!X || ldx < n)))
    return FSB_ERR_INVALID_ARG;
  if (n == 0) return FSB_ERR_UNSUPPORTED;  // dvals would be all zero: left to the separate kernels
  if (n_cols == 0) return FSB_OK;
  if (!t_indptr || !plan->units || plan->n_units < 1 || plan->cap < 1 || plan->cap > kSpmmMaxCap ||
      plan->chunk_nnz < kSpmmBatch || plan->chunk_nnz % kSpmmBatch != 0 || plan->n_slots < 0 ||
      (plan->n_slots > 0 && (!plan->partials || !plan->counters)))
    return FSB_ERR_INVALID_ARG;
  if (n_rows > 0 && !dY) return FSB_ERR_INVALID_ARG;
  if (plan->n_units >= INT32_MAX) return FSB_ERR_UNSUPPORTED;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  switch (dtype) {
    case FSB_F16:
      return spmm_backward<FSB_F16>(vals, perm, t_indices, t_indptr, dY, lddy, X, ldx, n, dX, lddx, dvals, *plan, st);
    case FSB_BF16:
      return spmm_backward<FSB_BF16>(vals, perm, t_indices, t_indptr, dY, lddy, X, ldx, n, dX, lddx, dvals, *plan,
                                     st);
    case FSB_F32:
      return spmm_backward<FSB_F32>(vals, perm, t_indices, t_indptr, dY, lddy, X, ldx, n, dX, lddx, dvals, *plan, st);
    case FSB_F64:
      return spmm_backward<FSB_F64>(vals, perm, t_indices, t_indptr, dY, lddy, X, ldx, n, dX, lddx, dvals, *plan, st);
    default: return FSB_ERR_UNSUPPORTED;
  }
}

}  // extern "C"
