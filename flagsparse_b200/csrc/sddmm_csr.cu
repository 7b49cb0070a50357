// CSR SDDMM  out[p] = alpha * <x[row(p)], y[col(p)]> + beta * in[p]  for sm_100a.
//
// x is M x K and y is N x K, both row-major; the sparsity pattern comes as the
// per-nonzero row ids and column indices (the reference's own prepared
// layout).  Every warp owns 32 consecutive nonzeros: it loads their row ids
// and columns with one coalesced read each, then walks them four at a time.
// The lanes own consecutive K-slices of V elements (16-byte loads when K and
// the leading dimensions allow it); the x and y slices of four nonzeros are
// loaded before any product is formed, and the four dot products are reduced
// together with a transpose butterfly (6 shuffles for 4 results instead of
// 20).  Consecutive nonzeros mostly share a row, so the x slice is an L1 hit.
//
// That generic kernel serves every shape; K-rows of up to 1,024 bytes in whole
// pieces of 8 bytes or more (512 bytes in pieces of 4, 256 of 2: sddmm_try_team)
// take the team kernel below, several nonzeros per warp instruction, which keeps
// the x row per team.  (Narrow rows left most lanes of the generic kernel idle,
// and rows off the 16-byte slices ran it too: fp32 on a 300,000-node graph, 8
// columns 342 -> 42 us, 16 columns 340 -> 60 us, 37 columns 416 -> 158 us.)
//
// Accumulation: fp32 for half / bfloat16 / fp32, fp64 for fp64 (fp64 for every
// type with FSB_SDDMM_ACC64, which the reference's "acc64" variants select),
// in a fixed order, so results are bitwise reproducible.
//
// Replaces _sddmm_csr_real_kernel (sparse_operations/sddmm_csr.py:121-162)
// launched by _run_sddmm_prepared (sddmm_csr.py:291-384) of flagos-ai/FlagSparse.
#include <cstring>
#include <type_traits>

#include "fsb_common.cuh"

namespace fsb {
namespace {

// Warps per block.  Team kernel: 2 rather than 8, since a block's place is free
// when its last warp ends (64 columns of fp32 on a 500,000-node graph: 311
// against 361 us at 8).  Generic kernel, Poisson(20) on 200,000 rows: 8 where
// lanes load single 2- or 4-byte elements (fp32 of 513 columns 1875 against 2315
// us at 2, of 37 columns with fp64 sums 360 against 402 us), 2 in fp64 (257
// columns 1992 against 2981 us at 8) and with vectors (bf16 of 128 columns with
// fp64 sums 491 against 604 us, fp32 of 512 columns 1573 against 1657 us).
constexpr int kSddmmWarps = 2;
template <int DT, int V>
constexpr int kSddmmGenericWarps = DT != FSB_F64 && V == 1 ? 8 : 2;
constexpr int kSddmmGroup = 4;  // nonzeros reduced together
// K-rows of at least this many bytes take 32-byte pieces where they can: half
// the lanes per row and half the instructions per nonzero of 16-byte ones (64
// columns of fp32 on that graph 441 -> 311 us; fp64, 32 columns 213 -> 180 us).
constexpr int kSlice32 = 128;

template <int BYTES> struct SRaw;
template <> struct SRaw<2> { using T = unsigned short; };
template <> struct SRaw<4> { using T = unsigned int; };
template <> struct SRaw<8> { using T = uint2; };
template <> struct SRaw<16> { using T = uint4; };

template <typename S, int V>
__device__ __forceinline__ void sload(const S* p, int nv, S (&out)[V]) {
  if (nv == V) {
    using Raw = typename SRaw<int(sizeof(S)) * V>::T;
    Raw r = __ldg(reinterpret_cast<const Raw*>(p));
    memcpy(out, &r, sizeof(Raw));
  } else {
#pragma unroll
    for (int j = 0; j < V; ++j) {
      if (j < nv) out[j] = p[j];
      else memset(&out[j], 0, sizeof(S));
    }
  }
}

__device__ __forceinline__ __half sddmm_out(float v, const __half*) { return __float2half_rn(v); }
__device__ __forceinline__ __nv_bfloat16 sddmm_out(float v, const __nv_bfloat16*) { return __float2bfloat16_rn(v); }
__device__ __forceinline__ float sddmm_out(float v, const float*) { return v; }
__device__ __forceinline__ double sddmm_out(double v, const double*) { return v; }
__device__ __forceinline__ __half sddmm_out(double v, const __half*) { return __double2half(v); }
__device__ __forceinline__ __nv_bfloat16 sddmm_out(double v, const __nv_bfloat16*) { return __double2bfloat16(v); }
__device__ __forceinline__ float sddmm_out(double v, const float*) { return __double2float_rn(v); }

__device__ __forceinline__ double to_acc64(float v) { return static_cast<double>(v); }
__device__ __forceinline__ double to_acc64(double v) { return v; }

// grid: one warp per 32 nonzeros.  ACC64: accumulate in fp64 whatever the
// value type; OUT64: write fp64 results (only with ACC64).
template <int DT, int V, bool ACC64, bool OUT64>
__global__ void __launch_bounds__(kSddmmGenericWarps<DT, V> * 32)
k_sddmm_csr(const int32_t* __restrict__ row_ids, const int32_t* __restrict__ col, int64_t nnz,
            const typename VT<DT>::Store* __restrict__ x, int64_t ldx, const typename VT<DT>::Store* __restrict__ y,
            int64_t ldy, int64_t k, const typename VT<DT>::Store* __restrict__ in, double alpha, double beta,
            typename std::conditional<OUT64, double, typename VT<DT>::Store>::type* __restrict__ out) {
  using S = typename VT<DT>::Store;
  using R = typename std::conditional<ACC64, double, typename VT<DT>::Real>::type;
  const int lane = threadIdx.x & 31;
  const int64_t base = (int64_t(blockIdx.x) * kSddmmGenericWarps<DT, V> + (threadIdx.x >> 5)) * 32;
  if (base >= nnz) return;  // whole warp leaves together
  const int cnt = nnz - base < 32 ? static_cast<int>(nnz - base) : 32;
  int my_r = 0, my_c = 0;
  if (lane < cnt) {
    my_r = __ldcs(row_ids + base + lane);
    my_c = __ldcs(col + base + lane);
  }
  const R a = static_cast<R>(alpha), b = static_cast<R>(beta);
  const int64_t tile_w = int64_t(32) * V;
  const int n_tiles = static_cast<int>((k + tile_w - 1) / tile_w);

  for (int g = 0; g < cnt; g += kSddmmGroup) {
    R part[kSddmmGroup];
#pragma unroll
    for (int q = 0; q < kSddmmGroup; ++q) part[q] = R(0);
    int rq[kSddmmGroup], cq[kSddmmGroup];
#pragma unroll
    for (int q = 0; q < kSddmmGroup; ++q) {
      const int src = g + q < cnt ? g + q : g;
      rq[q] = __shfl_sync(0xffffffffu, my_r, src);
      cq[q] = __shfl_sync(0xffffffffu, my_c, src);
    }
    for (int t = 0; t < n_tiles; ++t) {
      const int64_t j0 = int64_t(t) * tile_w + int64_t(lane) * V;
      const int nv = static_cast<int>(k - j0 >= V ? int64_t(V) : (k > j0 ? k - j0 : int64_t(0)));
      S xs[kSddmmGroup][V], ys[kSddmmGroup][V];
#pragma unroll
      for (int q = 0; q < kSddmmGroup; ++q) {
        const int w = g + q < cnt ? nv : 0;
        sload<S, V>(x + int64_t(rq[q]) * ldx + j0, w, xs[q]);
        sload<S, V>(y + int64_t(cq[q]) * ldy + j0, w, ys[q]);
      }
#pragma unroll
      for (int q = 0; q < kSddmmGroup; ++q)
#pragma unroll
        for (int j = 0; j < V; ++j) {
          if constexpr (ACC64) part[q] = fma(to_acc64(to_real(xs[q][j])), to_acc64(to_real(ys[q][j])), part[q]);
          else part[q] = fma(to_real(xs[q][j]), to_real(ys[q][j]), part[q]);
        }
    }
    // Transpose butterfly: after the xor-16 step lanes 0-15 hold items {0,1}
    // and lanes 16-31 items {2,3}; after xor-8 each quarter of the warp holds
    // one item (quarter index = item index); xor 4, 2, 1 finish the sums.
    const bool hi16 = lane & 16, hi8 = lane & 8;
    R s0 = hi16 ? part[2] : part[0], s1 = hi16 ? part[3] : part[1];
    const R o0 = hi16 ? part[0] : part[2], o1 = hi16 ? part[1] : part[3];
    s0 += __shfl_xor_sync(0xffffffffu, o0, 16);
    s1 += __shfl_xor_sync(0xffffffffu, o1, 16);
    R v = hi8 ? s1 : s0;
    v += __shfl_xor_sync(0xffffffffu, hi8 ? s0 : s1, 8);
    v += __shfl_xor_sync(0xffffffffu, v, 4);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    const int q = lane >> 3;
    if ((lane & 7) == 0 && g + q < cnt) {
      const int64_t p = base + g + q;
      R res = v * a;
      if (in) res += static_cast<R>(to_real(in[p])) * b;
      out[p] = sddmm_out(res, out);
    }
  }
}

// ---------------------------------------------------------------------------
// Team kernel.  Teams of T lanes (2 to 32) own a K-row as P pieces of E
// consecutive elements per lane, a team's lanes side by side in each piece.
// A team walks U = 4 consecutive nonzeros per round with their y slices in
// flight together, and keeps its current x row, loaded when the row changes
// (holding the round's first and last row instead, loaded beside the y slices,
// measured slower: 364 against 311 us below, its registers and branches cost
// more than the wait).  The four
// dot products are reduced across the team by a transpose butterfly: after the
// T/2 step a lane holds 2 items, after T/4 one, then log2(T/4) plain steps.
// ---------------------------------------------------------------------------
constexpr int kTeamU = 4;

// acc += lo(x) * lo(y), then acc += hi(x) * hi(y) for two packed 16-bit
// values each: sm_100a's mixed-precision fma.rn.f32.{bf16,f16} multiplies the
// 16-bit inputs exactly (their product fits fp32) and rounds the sum once,
// so the result equals widening both to fp32 and calling fmaf, in the same
// order, with no widening instructions.
template <typename S>
__device__ __forceinline__ float fma_pair16(unsigned xw, unsigned yw, float acc) {
  if constexpr (std::is_same<S, __nv_bfloat16>::value) {
    asm("{\n .reg .b16 xl, xh, yl, yh;\n mov.b32 {xl, xh}, %1;\n mov.b32 {yl, yh}, %2;\n"
        " fma.rn.f32.bf16 %0, xl, yl, %0;\n fma.rn.f32.bf16 %0, xh, yh, %0;\n}"
        : "+f"(acc) : "r"(xw), "r"(yw));
  } else {
    asm("{\n .reg .b16 xl, xh, yl, yh;\n mov.b32 {xl, xh}, %1;\n mov.b32 {yl, yh}, %2;\n"
        " fma.rn.f32.f16 %0, xl, yl, %0;\n fma.rn.f32.f16 %0, xh, yh, %0;\n}"
        : "+f"(acc) : "r"(xw), "r"(yw));
  }
  return acc;
}

// A lane's elements of a K-row: piece q is columns (q * T + tl) * E .. + E,
// wholly inside K or (zero) outside it.
template <typename S, int E, int P>
struct KSlice {
  static constexpr int V = E * P, kBytes = E * int(sizeof(S));
  S v[V];
  __device__ __forceinline__ void load(const S* __restrict__ row, int T, int tl, int k) {
#pragma unroll
    for (int q = 0; q < P; ++q) {
      const int c = (q * T + tl) * E;
      if (c < k) {
        if constexpr (kBytes == 32) {
          uint32_t r[8];
          asm("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
              : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
              : "l"(row + c));
          memcpy(&v[q * E], r, 32);
        } else {
          using Raw = typename SRaw<kBytes>::T;
          const Raw r = __ldg(reinterpret_cast<const Raw*>(row + c));
          memcpy(&v[q * E], &r, kBytes);
        }
      } else {
        memset(&v[q * E], 0, kBytes);
      }
    }
  }
  // the dot product of two slices, one chain in element order (pairs of 4-byte
  // values: two chains, added)
  template <typename R>
  __device__ __forceinline__ R dot(const KSlice& o) const {
    if constexpr (sizeof(S) == 2 && V % 2 == 0) {
      float acc = 0.f;
      unsigned a[V / 2], b[V / 2];
      memcpy(a, v, sizeof(a));
      memcpy(b, o.v, sizeof(b));
#pragma unroll
      for (int j = 0; j < V / 2; ++j) acc = fma_pair16<S>(a[j], b[j], acc);
      return acc;
    } else if constexpr (std::is_same<S, float>::value && V % 2 == 0) {
      unsigned long long acc = 0;
#pragma unroll
      for (int j = 0; j < V; j += 2) {
        unsigned long long a, b;
        asm("mov.b64 %0, {%1, %2};" : "=l"(a) : "f"(v[j]), "f"(v[j + 1]));
        asm("mov.b64 %0, {%1, %2};" : "=l"(b) : "f"(o.v[j]), "f"(o.v[j + 1]));
        asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
      }
      float lo, hi;
      asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(acc));
      return lo + hi;
    } else {
      R acc = R(0);
#pragma unroll
      for (int j = 0; j < V; ++j) acc = fma(to_real(v[j]), to_real(o.v[j]), acc);
      return acc;
    }
  }
};

// Blocks per SM the register budget is sized for, by a lane's bytes of a row: 80
// registers for four 32-byte slices in flight (64 spill: 525 against 375 us on
// the graph above, before the rest of this kernel's changes), else 64.
constexpr int sddmm_blocks(int bytes) { return (bytes > 16 ? 24 : 32) / kSddmmWarps; }

template <int DT, int T, int E, int P>
__global__ void __launch_bounds__(kSddmmWarps * 32, sddmm_blocks(E * P * int(sizeof(typename VT<DT>::Store))))
k_sddmm_team(const int32_t* __restrict__ row_ids, const int32_t* __restrict__ col, int64_t nnz,
             const typename VT<DT>::Store* __restrict__ x, int64_t ldx, const typename VT<DT>::Store* __restrict__ y,
             int64_t ldy, int k, const typename VT<DT>::Store* __restrict__ in, double alpha, double beta,
             typename VT<DT>::Store* __restrict__ out) {
  using S = typename VT<DT>::Store;
  using R = typename VT<DT>::Real;
  using Sl = KSlice<S, E, P>;
  constexpr int G = 32 / T;                              // teams per warp
  constexpr int kRound = G * kTeamU;                     // nonzeros per warp round
  constexpr int kOwn = kRound > 32 ? kRound : 32, kW = kOwn / 32;  // nonzeros per warp
  static_assert(T >= 2 && T <= 32, "team size");
  const int lane = threadIdx.x & 31;
  const int team = lane / T, tl = lane % T;
  const int64_t base = (int64_t(blockIdx.x) * kSddmmWarps + (threadIdx.x >> 5)) * kOwn;
  if (base >= nnz) return;  // whole warp leaves together
  const int cnt = nnz - base < kOwn ? static_cast<int>(nnz - base) : kOwn;
  int my_r[kW], my_c[kW];
#pragma unroll
  for (int w = 0; w < kW; ++w) {  // past the end: the last nonzero again, computed and not written
    const int i = min(w * 32 + lane, cnt - 1);
    my_r[w] = __ldcs(row_ids + base + i);
    my_c[w] = __ldcs(col + base + i);
  }
  const R a = static_cast<R>(alpha), b = static_cast<R>(beta);
  Sl xs;
  int cur = -1;  // the row that xs holds

  for (int r0 = 0; r0 < cnt; r0 += kRound) {
    const int first = r0 + team * kTeamU;  // this team's items: first .. first+3
    int rq[kTeamU], cq[kTeamU];
#pragma unroll
    for (int u = 0; u < kTeamU; ++u) {
      const int src = (first + u) & 31;
      rq[u] = __shfl_sync(0xffffffffu, my_r[0], src);
      cq[u] = __shfl_sync(0xffffffffu, my_c[0], src);
#pragma unroll
      for (int w = 1; w < kW; ++w) {
        const int r = __shfl_sync(0xffffffffu, my_r[w], src), c = __shfl_sync(0xffffffffu, my_c[w], src);
        if (((first + u) >> 5) == w) {
          rq[u] = r;
          cq[u] = c;
        }
      }
    }
    Sl ys[kTeamU];
#pragma unroll
    for (int u = 0; u < kTeamU; ++u) ys[u].load(y + int64_t(cq[u]) * ldy, T, tl, k);
    R part[kTeamU];
#pragma unroll
    for (int u = 0; u < kTeamU; ++u) {
      if (rq[u] != cur) {  // uniform inside the team
        cur = rq[u];
        xs.load(x + int64_t(cur) * ldx, T, tl, k);
      }
      part[u] = xs.template dot<R>(ys[u]);
    }
    // transpose butterfly inside the team
    constexpr int H = T / 2, Q = T / 4;
    const bool hb = tl & H, qb = Q > 0 && (tl & Q);
    R s0 = hb ? part[2] : part[0], s1 = hb ? part[3] : part[1];
    s0 += __shfl_xor_sync(0xffffffffu, hb ? part[0] : part[2], H);
    s1 += __shfl_xor_sync(0xffffffffu, hb ? part[1] : part[3], H);
    auto put = [&](int item, R v) {
      if (item < cnt) {
        const int64_t p = base + item;
        R res = v * a;
        if (in) res += to_real(in[p]) * b;
        out[p] = sddmm_out(res, out);
      }
    };
    if constexpr (Q == 0) {  // two lanes: two finished items each
      put(first + (hb ? 2 : 0), s0);
      put(first + (hb ? 3 : 1), s1);
    } else {
      R v = qb ? s1 : s0;
      v += __shfl_xor_sync(0xffffffffu, qb ? s0 : s1, Q);
#pragma unroll
      for (int m = Q / 2; m > 0; m >>= 1) v += __shfl_xor_sync(0xffffffffu, v, m);
      if ((tl & (Q - 1)) == 0) put(first + (hb ? 2 : 0) + (qb ? 1 : 0), v);
    }
  }
}

template <int DT, int T, int E, int P>
int sddmm_launch_team(const int32_t* row_ids, const int32_t* col, int64_t nnz, const void* x, int64_t ldx,
                      const void* y, int64_t ldy, int64_t k, const void* in, double alpha, double beta, void* out,
                      cudaStream_t st) {
  using S = typename VT<DT>::Store;
  constexpr int kOwn = 32 / T * kTeamU > 32 ? 32 / T * kTeamU : 32;
  const int64_t blocks = ceil_div(ceil_div(nnz, kOwn), kSddmmWarps);
  if (blocks > INT32_MAX) return FSB_ERR_UNSUPPORTED;
  k_sddmm_team<DT, T, E, P><<<(unsigned)blocks, kSddmmWarps * 32, 0, st>>>(
      row_ids, col, nnz, static_cast<const S*>(x), ldx, static_cast<const S*>(y), ldy, static_cast<int>(k),
      static_cast<const S*>(in), alpha, beta, static_cast<S*>(out));
  FSB_LAUNCH_CHECK();
  return FSB_OK;
}

// A row as `pieces` pieces of E elements, P per lane.
template <int DT, int E, int P, int T = 32>
int sddmm_launch_pieces(int pieces, const int32_t* row_ids, const int32_t* col, int64_t nnz, const void* x,
                        int64_t ldx, const void* y, int64_t ldy, int64_t k, const void* in, double alpha, double beta,
                        void* out, cudaStream_t st) {
  if constexpr (T > 2)
    if (pieces <= T / 2 * P)
      return sddmm_launch_pieces<DT, E, P, T / 2>(pieces, row_ids, col, nnz, x, ldx, y, ldy, k, in, alpha, beta, out,
                                                  st);
  return sddmm_launch_team<DT, T, E, P>(row_ids, col, nnz, x, ldx, y, ldy, k, in, alpha, beta, out, st);
}

// The team kernel where 32 lanes hold a K-row: returns 1 when it launched (rc
// set).  Pieces are the widest of 32 (rows of at least kSlice32 bytes), 16, 8, 4
// and 2 bytes that divide K, the leading dimensions and the addresses; a lane
// holds 32 bytes of a row at most (four pieces of 8, two of 16), and four pieces
// of 4 or 2, so rows of up to 1,024, 512 and 256 bytes.
template <int DT>
int sddmm_try_team(const int32_t* row_ids, const int32_t* col, int64_t nnz, const void* x, int64_t ldx,
                   const void* y, int64_t ldy, int64_t k, const void* in, double alpha, double beta, void* out,
                   int* rc, cudaStream_t st) {
  using S = typename VT<DT>::Store;
  constexpr int s = int(sizeof(S));
  auto whole = [&](int bytes) {
    const int e = bytes / s;
    return k % e == 0 && ldx % e == 0 && ldy % e == 0 && reinterpret_cast<uintptr_t>(x) % bytes == 0 &&
           reinterpret_cast<uintptr_t>(y) % bytes == 0;
  };
  auto run = [&](auto e, auto p) {
    constexpr int E = decltype(e)::value, P = decltype(p)::value;
    if (k > int64_t(32) * P * E) return 0;
    *rc = sddmm_launch_pieces<DT, E, P>(static_cast<int>(k / E), row_ids, col, nnz, x, ldx, y, ldy, k, in, alpha, beta,
                                        out, st);
    return 1;
  };
#define FSB_I(n) std::integral_constant<int, (n)>()
  if (k < 1) return 0;
  if (k * s >= kSlice32 && whole(32)) return run(FSB_I(32 / s), FSB_I(1));
  if (whole(16)) return k * s <= 512 ? run(FSB_I(16 / s), FSB_I(1)) : run(FSB_I(16 / s), FSB_I(2));
  if constexpr (s <= 8)
    if (whole(8)) return run(FSB_I(8 / s), FSB_I(2)) || run(FSB_I(8 / s), FSB_I(4));
  if constexpr (s <= 4)
    if (whole(4)) return run(FSB_I(4 / s), FSB_I(4));
  if constexpr (s <= 2)
    if (whole(2)) return run(FSB_I(1), FSB_I(4));
#undef FSB_I
  return 0;
}

template <int DT, int V, bool ACC64, bool OUT64>
int sddmm_launch_mode(const int32_t* row_ids, const int32_t* col, int64_t nnz, const void* x, int64_t ldx,
                      const void* y, int64_t ldy, int64_t k, const void* in, double alpha, double beta, void* out,
                      cudaStream_t st) {
  using S = typename VT<DT>::Store;
  using O = typename std::conditional<OUT64, double, S>::type;
  const int64_t blocks = ceil_div(ceil_div(nnz, 32), kSddmmGenericWarps<DT, V>);
  if (blocks > INT32_MAX) return FSB_ERR_UNSUPPORTED;
  k_sddmm_csr<DT, V, ACC64, OUT64><<<(unsigned)blocks, kSddmmGenericWarps<DT, V> * 32, 0, st>>>(
      row_ids, col, nnz, static_cast<const S*>(x), ldx, static_cast<const S*>(y), ldy, k,
      static_cast<const S*>(in), alpha, beta, static_cast<O*>(out));
  FSB_LAUNCH_CHECK();
  return FSB_OK;
}

template <int DT, int V>
int sddmm_launch_v(const int32_t* row_ids, const int32_t* col, int64_t nnz, const void* x, int64_t ldx,
                   const void* y, int64_t ldy, int64_t k, const void* in, double alpha, double beta, void* out,
                   int flags, cudaStream_t st) {
  if constexpr (DT != FSB_F64) {
    if (flags & FSB_SDDMM_OUT64)
      return sddmm_launch_mode<DT, V, true, true>(row_ids, col, nnz, x, ldx, y, ldy, k, in, alpha, beta, out, st);
    if (flags & FSB_SDDMM_ACC64)
      return sddmm_launch_mode<DT, V, true, false>(row_ids, col, nnz, x, ldx, y, ldy, k, in, alpha, beta, out, st);
  }
  return sddmm_launch_mode<DT, V, false, false>(row_ids, col, nnz, x, ldx, y, ldy, k, in, alpha, beta, out, st);
}

template <int DT>
int sddmm_dispatch(const int32_t* row_ids, const int32_t* col, int64_t nnz, const void* x, int64_t ldx,
                   const void* y, int64_t ldy, int64_t k, const void* in, double alpha, double beta, void* out,
                   int flags, cudaStream_t st) {
  using S = typename VT<DT>::Store;
  constexpr int kVmax = 16 / int(sizeof(S));
  if (!(flags & (FSB_SDDMM_ACC64 | FSB_SDDMM_OUT64)) || DT == FSB_F64) {
    int rc = FSB_OK;
    if (sddmm_try_team<DT>(row_ids, col, nnz, x, ldx, y, ldy, k, in, alpha, beta, out, &rc, st)) return rc;
  }
  int v = 1;
  while (v < kVmax && int64_t(32) * v < k) v *= 2;
  auto ok = [&](int w) {
    const uintptr_t al = uintptr_t(w) * sizeof(S);
    return reinterpret_cast<uintptr_t>(x) % al == 0 && reinterpret_cast<uintptr_t>(y) % al == 0 && ldx % w == 0 &&
           ldy % w == 0;
  };
  while (v > 1 && !ok(v)) v /= 2;
  if constexpr (kVmax >= 8)
    if (v == 8) return sddmm_launch_v<DT, 8>(row_ids, col, nnz, x, ldx, y, ldy, k, in, alpha, beta, out, flags, st);
  if constexpr (kVmax >= 4)
    if (v == 4) return sddmm_launch_v<DT, 4>(row_ids, col, nnz, x, ldx, y, ldy, k, in, alpha, beta, out, flags, st);
  if constexpr (kVmax >= 2)
    if (v == 2) return sddmm_launch_v<DT, 2>(row_ids, col, nnz, x, ldx, y, ldy, k, in, alpha, beta, out, flags, st);
  return sddmm_launch_v<DT, 1>(row_ids, col, nnz, x, ldx, y, ldy, k, in, alpha, beta, out, flags, st);
}

// row_ids[p] = the row of nonzero p: one thread per nonzero, upper bound on indptr.
template <typename PT>
__global__ void k_csr_row_ids(const PT* __restrict__ ptr, int64_t n_rows, int64_t nnz, int32_t* __restrict__ rows) {
  const int64_t stride = int64_t(gridDim.x) * blockDim.x;
  for (int64_t p = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; p < nnz; p += stride) {
    int64_t lo = 0, hi = n_rows - 1;  // last row r with ptr[r] <= p
    while (lo < hi) {
      const int64_t mid = (lo + hi + 1) >> 1;
      if (ld_ptr(ptr, mid) <= p) lo = mid; else hi = mid - 1;
    }
    rows[p] = static_cast<int32_t>(lo);
  }
}

}  // namespace
}  // namespace fsb

using namespace fsb;

extern "C" {

int fsb_csr_row_ids(const void* indptr, int ptr_is_64, int64_t n_rows, int64_t nnz, int32_t* row_ids, void* stream) {
  if (!indptr || n_rows < 0 || nnz < 0 || (nnz > 0 && (!row_ids || n_rows == 0))) return FSB_ERR_INVALID_ARG;
  if (n_rows > INT32_MAX) return FSB_ERR_UNSUPPORTED;
  if (nnz == 0) return FSB_OK;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int64_t blocks = ceil_div(nnz, 256);
  if (blocks > 148 * 64) blocks = 148 * 64;
  if (ptr_is_64)
    k_csr_row_ids<int64_t><<<(unsigned)blocks, 256, 0, st>>>(static_cast<const int64_t*>(indptr), n_rows, nnz, row_ids);
  else
    k_csr_row_ids<int32_t><<<(unsigned)blocks, 256, 0, st>>>(static_cast<const int32_t*>(indptr), n_rows, nnz, row_ids);
  FSB_LAUNCH_CHECK();
  return FSB_OK;
}

int fsb_sddmm_csr(int dtype, const int32_t* row_ids, const int32_t* indices, int64_t nnz, const void* x, int64_t ldx,
                  const void* y, int64_t ldy, int64_t k, const void* in, double alpha, double beta, void* out,
                  int flags, void* stream) {
  if ((flags & FSB_SDDMM_OUT64) && !(flags & FSB_SDDMM_ACC64)) return FSB_ERR_INVALID_ARG;
  if (nnz < 0 || k < 0 || ldx < k || ldy < k) return FSB_ERR_INVALID_ARG;
  if (nnz == 0) return FSB_OK;
  if (!row_ids || !indices || !out || (k > 0 && (!x || !y))) return FSB_ERR_INVALID_ARG;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  switch (dtype) {
    case FSB_F16: return sddmm_dispatch<FSB_F16>(row_ids, indices, nnz, x, ldx, y, ldy, k, in, alpha, beta, out, flags, st);
    case FSB_BF16: return sddmm_dispatch<FSB_BF16>(row_ids, indices, nnz, x, ldx, y, ldy, k, in, alpha, beta, out, flags, st);
    case FSB_F32: return sddmm_dispatch<FSB_F32>(row_ids, indices, nnz, x, ldx, y, ldy, k, in, alpha, beta, out, flags, st);
    case FSB_F64: return sddmm_dispatch<FSB_F64>(row_ids, indices, nnz, x, ldx, y, ldy, k, in, alpha, beta, out, flags, st);
    default: return FSB_ERR_UNSUPPORTED;
  }
}

}  // extern "C"
