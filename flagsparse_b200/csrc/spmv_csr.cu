// CSR SpMV y = A x for sm_100a.
//
// Every warp executes work units of the plan built by fsb_spmv_plan_build
// (plan.cu); a unit's 32-byte descriptor carries its nonzero range, so the
// warp issues its value / column loads immediately.  The plan lists the two
// kinds of unit apart, and each kind runs as its own launch:
//
//  * row-block units: a run of rows with < 2*cap nonzeros.  Persistent warps
//    stride over the units.  Every lane owns kP consecutive nonzeros of a pass
//    (one or two wide loads of values and of columns), gathers x for them and
//    sums them in order, closing a row wherever the pass's end marks say one
//    ends; a segmented shuffle scan joins rows that span lanes.  The end marks
//    are one byte per nonzero in the warp's shared memory, so the sums have no
//    per-lane row walk and no divergence.
//  * long-row chunks: `chunk_nnz` nonzeros of one row with > cap nonzeros, in
//    256-nonzero batches whose column loads are issued one batch ahead; no
//    shared memory; launched as a programmatic dependent of the row-block
//    launch so it overlaps that grid's tail.  A one-chunk row is written directly; otherwise the warp
//    publishes a partial sum and the warp whose atomic ticket completes the
//    row adds all partials in a fixed order and resets the ticket, so results
//    are deterministic.
//
// x is gathered with L2-only loads (ld.global.cg): random gathers have no reuse
// in L1 (row blocks of a 2 M-row Zipf matrix 94.0 us, 94.4 with plain loads).
//
// Replaces _spmv_csr_real_kernel / _spmv_csr_complex_kernel
// (sparse_operations/spmv_csr.py:179-240) and the bucketed CSR-vector kernels
// (spmv_csr.py:247-368) of flagos-ai/FlagSparse.
#include <algorithm>
#include <cstring>
#include <mutex>

#include <cuda.h>
#include <type_traits>

#include "fsb_common.cuh"

namespace fsb {

template <int DT>
struct SpmvTraits {
  using V = VT<DT>;
  using S = typename V::Store;
  using R = typename V::Real;
  static constexpr bool kLo = !V::kExactProduct;  // a product has a rounding error of its own
};

template <typename S> __device__ __forceinline__ S to_store(float v);
template <> __device__ __forceinline__ __half to_store<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 to_store<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }
template <> __device__ __forceinline__ float to_store<float>(float v) { return v; }
template <typename S> __device__ __forceinline__ S to_store(double v) { return v; }

// Row accumulator.  COMP = true: Dot2 compensated sums (Comp); COMP = false:
// plain sums in the real type (Plain), used only where the caller opts in.
template <int DT, bool COMP, bool CPLX = VT<DT>::kComplex>
struct SpmvAcc;

template <int DT, bool COMP>
struct SpmvAcc<DT, COMP, false> {
  using Tr = SpmvTraits<DT>;
  using S = typename Tr::S;
  using R = typename Tr::R;
  static constexpr int kPartialReals = 2;
  using Sum = typename std::conditional<COMP, Comp<R>, Plain<R>>::type;
  Sum c;
  __device__ __forceinline__ void zero() { c.zero(); }
  __device__ __forceinline__ void add_prod(S a, S x) {
    if constexpr (COMP) {
      if constexpr (Tr::kLo) c.add_prod(to_real(a), to_real(x));
      else c.add(mul_rn(to_real(a), to_real(x)));
    } else {
      c.add_prod(to_real(a), to_real(x));
    }
  }
  __device__ __forceinline__ void combine(const SpmvAcc& o) {
    if constexpr (COMP) c.add_comp(o.c.hi, o.c.lo);
    else c.add(o.c.hi);
  }
  __device__ __forceinline__ void shfl_combine(int m) {
    SpmvAcc o = *this;
    o.c.hi = __shfl_xor_sync(0xffffffffu, c.hi, m);
    if constexpr (COMP) o.c.lo = __shfl_xor_sync(0xffffffffu, c.lo, m);
    combine(o);
  }
  __device__ __forceinline__ void shfl_up(int o) {
    c.hi = __shfl_up_sync(0xffffffffu, c.hi, o);
    if constexpr (COMP) c.lo = __shfl_up_sync(0xffffffffu, c.lo, o);
  }
  __device__ __forceinline__ void from_lane(int l) {
    c.hi = __shfl_sync(0xffffffffu, c.hi, l);
    if constexpr (COMP) c.lo = __shfl_sync(0xffffffffu, c.lo, l);
  }
  __device__ __forceinline__ S result() const { return to_store<S>(c.value()); }
  __device__ __forceinline__ void store(R* p) const {
    p[0] = c.hi;
    if constexpr (COMP) p[1] = c.lo;
  }
  __device__ __forceinline__ void load_cg(const R* p) {
    c.hi = __ldcg(p);
    if constexpr (COMP) c.lo = __ldcg(p + 1);
  }
};

// Short rows of the 2- and 4-byte real types: fp64 sums of the exact products
// (their products are exact in fp64, and the fp64 sum of a row-block row is
// far inside the Dot2 bound) at one DFMA per term.
template <int DT>
struct SpmvWide {
  using S = typename VT<DT>::Store;
  double c;
  __device__ __forceinline__ void zero() { c = 0.0; }
  __device__ __forceinline__ void add_prod(S a, S x) { c = __fma_rn(double(to_real(a)), double(to_real(x)), c); }
  __device__ __forceinline__ void combine(const SpmvWide& o) { c = __dadd_rn(c, o.c); }
  __device__ __forceinline__ void shfl_up(int o) { c = __shfl_up_sync(0xffffffffu, c, o); }
  __device__ __forceinline__ void from_lane(int l) { c = __shfl_sync(0xffffffffu, c, l); }
  __device__ __forceinline__ S result() const { return to_store<S>(__double2float_rn(c)); }
};

template <int DT, bool COMP>
struct SpmvAcc<DT, COMP, true> {
  using Tr = SpmvTraits<DT>;
  using S = typename Tr::S;
  using R = typename Tr::R;
  static constexpr int kPartialReals = 4;
  using Sum = typename std::conditional<COMP, Comp<R>, Plain<R>>::type;
  Sum re, im;
  __device__ __forceinline__ void zero() { re.zero(); im.zero(); }
  __device__ __forceinline__ void add_prod(S a, S x) {
    re.add_prod(a.x, x.x); re.add_prod(-a.y, x.y);
    im.add_prod(a.x, x.y); im.add_prod(a.y, x.x);
  }
  __device__ __forceinline__ void combine(const SpmvAcc& o) {
    if constexpr (COMP) { re.add_comp(o.re.hi, o.re.lo); im.add_comp(o.im.hi, o.im.lo); }
    else { re.add(o.re.hi); im.add(o.im.hi); }
  }
  __device__ __forceinline__ void shfl_combine(int m) {
    SpmvAcc o = *this;
    o.re.hi = __shfl_xor_sync(0xffffffffu, re.hi, m);
    o.im.hi = __shfl_xor_sync(0xffffffffu, im.hi, m);
    if constexpr (COMP) {
      o.re.lo = __shfl_xor_sync(0xffffffffu, re.lo, m);
      o.im.lo = __shfl_xor_sync(0xffffffffu, im.lo, m);
    }
    combine(o);
  }
  __device__ __forceinline__ void shfl_up(int o) {
    re.hi = __shfl_up_sync(0xffffffffu, re.hi, o);
    im.hi = __shfl_up_sync(0xffffffffu, im.hi, o);
    if constexpr (COMP) {
      re.lo = __shfl_up_sync(0xffffffffu, re.lo, o);
      im.lo = __shfl_up_sync(0xffffffffu, im.lo, o);
    }
  }
  __device__ __forceinline__ void from_lane(int l) {
    re.hi = __shfl_sync(0xffffffffu, re.hi, l);
    im.hi = __shfl_sync(0xffffffffu, im.hi, l);
    if constexpr (COMP) {
      re.lo = __shfl_sync(0xffffffffu, re.lo, l);
      im.lo = __shfl_sync(0xffffffffu, im.lo, l);
    }
  }
  __device__ __forceinline__ S result() const {
    S s; s.x = re.value(); s.y = im.value(); return s;
  }
  __device__ __forceinline__ void store(R* p) const {
    p[0] = re.hi; p[1] = re.lo; p[2] = im.hi; p[3] = im.lo;
  }
  __device__ __forceinline__ void load_cg(const R* p) {
    re.hi = __ldcg(p); re.lo = __ldcg(p + 1); im.hi = __ldcg(p + 2); im.lo = __ldcg(p + 3);
  }
};

template <typename T> __device__ __forceinline__ T ld_stream(const T* p) { return __ldcs(p); }
template <> __device__ __forceinline__ __half ld_stream<__half>(const __half* p) {
  unsigned short v = __ldcs(reinterpret_cast<const unsigned short*>(p));
  return __ushort_as_half(v);
}
template <> __device__ __forceinline__ __nv_bfloat16 ld_stream<__nv_bfloat16>(const __nv_bfloat16* p) {
  unsigned short v = __ldcs(reinterpret_cast<const unsigned short*>(p));
  return __ushort_as_bfloat16(v);
}
// Gather of x: L2-only, no L1 allocation.
template <typename T> __device__ __forceinline__ T ld_x(const T* p) { return __ldcg(p); }
template <> __device__ __forceinline__ __half ld_x<__half>(const __half* p) {
  return __ushort_as_half(__ldcg(reinterpret_cast<const unsigned short*>(p)));
}
template <> __device__ __forceinline__ __nv_bfloat16 ld_x<__nv_bfloat16>(const __nv_bfloat16* p) {
  return __ushort_as_bfloat16(__ldcg(reinterpret_cast<const unsigned short*>(p)));
}

constexpr int kSpmvWarps = 8;     // warps per block; a unit at a time per warp
constexpr int kSpmvItems = 8;     // nonzeros per lane per long-row batch
constexpr int kSpmvBatch = 32 * kSpmvItems;

// Row-block units: kP consecutive nonzeros per lane and pass (one wide load of
// columns, one or two of values), kCap the largest window: a unit holds <= cap
// rows, whose local indices fit the end marks' bytes, and < 2*cap nonzeros.
// A large window fills more of a unit's last pass and spreads its fixed chain of
// loads over more rows: against 224 for the 2- and 4-byte types and 128 for the
// wider ones, 252 takes a 1 M-row stencil from 37 to 33 us in fp64 and 26.7 to
// 22.6 in fp32, Poisson(16) from 39 to 31 us in fp64 (300,000 rows) and 71.8 to
// 70.3 in fp32 (1 M rows), fp64 Zipf (1 M rows) from 139 to 123 us.
// Four per lane rather than eight: the next pass's run is held in registers
// beside the current one, and eight spill at 64 registers (2 M-row Zipf(2)
// matrix: 94 against 135 us for this launch, 107 us for the product staging
// and merge path it replaced; 1 M rows of Poisson(16): 72 against 106 and 84).
// Two per lane measured slower in fp64 (41 against 37.5 us on a 1 M-row stencil)
// and in complex fp64 (Poisson(16) on 500,000 rows 115 against 78 us, Poisson(60)
// on 200,000 rows 187 against 131 us, the stencil 81 against 57 us; the staged
// kernel took 115, 165 and 82).
struct SpmvRow {
  static constexpr int kP = 4;
  static constexpr int kPass = 32 * kP;
  static constexpr int kCap = 252;
  static constexpr int kMarkBytes = (2 * kCap + 2 * kP + 15) & ~15;
  static_assert(kCap < 255, "local row index + 1 is one byte");
  static_assert(kP == 4, "a run's marks are one 32-bit word");
};

// N consecutive elements at p (aligned to their size or to 32 bytes), read
// once: 32-byte loads where there are that many.
template <typename T, int N>
__device__ __forceinline__ void ld_run(const T* p, T (&out)[N]) {
  constexpr int kBytes = int(sizeof(T)) * N;
  if constexpr (kBytes >= 32) {
    static_assert(kBytes % 32 == 0, "whole 32-byte loads");
#pragma unroll
    for (int c = 0; c < kBytes / 32; ++c) {
      uint32_t r[8];
      asm volatile("ld.global.cs.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                   : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                   : "l"(reinterpret_cast<const char*>(p) + 32 * c));
      memcpy(reinterpret_cast<char*>(out) + 32 * c, r, 32);
    }
  } else if constexpr (kBytes == 16) {
    const uint4 r = __ldcs(reinterpret_cast<const uint4*>(p));
    memcpy(out, &r, 16);
  } else {
    static_assert(kBytes == 8, "8, 16 or whole 32-byte runs");
    const uint2 r = __ldcs(reinterpret_cast<const uint2*>(p));
    memcpy(out, &r, 8);
  }
}

struct UnitRegs { int64_t s0, s1; int32_t row, tag, nch, slot; };

__device__ __forceinline__ UnitRegs load_unit(const fsb_spmv_unit* u) {
  const int4* p = reinterpret_cast<const int4*>(u);
  int4 a = __ldg(p), b = __ldg(p + 1);
  UnitRegs r;
  r.s0 = (int64_t)(uint32_t)a.x | ((int64_t)a.y << 32);
  r.s1 = (int64_t)(uint32_t)a.z | ((int64_t)a.w << 32);
  r.row = b.x;
  r.tag = b.y;
  r.nch = b.z;
  r.slot = b.w;
  return r;
}

// Resident blocks per SM the register budgets are sized for.  Row blocks: 4 (64
// registers; fp64 spills 44 bytes there and still gains on 3 blocks: 37.5
// against 45.6 us on a 1 M-row stencil, where each unit is a chain of dependent
// loads and more warps hide more of it; 5 blocks of fp32 spill, 121 against 94
// us on the Zipf matrix), 2 for complex fp64.  Long rows: 8-byte reals and
// complex values need more registers than fp32 / half types.
template <int DT>
struct SpmvRowMinBlocks { static constexpr int value = (DT == FSB_C128) ? 2 : 4; };
template <int DT>
struct SpmvMinBlocks { static constexpr int value = (DT == FSB_C128) ? 2 : (DT == FSB_F64 || DT == FSB_C64) ? 3 : 4; };
// The long-row kernel keeps fewer values live (no pass ahead, columns one batch
// ahead): the 2- and 4-byte real types with 32-bit columns fit 5 blocks per SM
// without spills.
template <int DT, typename IT>
struct SpmvLongMinBlocks {
  static constexpr int value =
      ((DT == FSB_F16 || DT == FSB_BF16 || DT == FSB_F32) && sizeof(IT) == 4) ? 5 : SpmvMinBlocks<DT>::value;
};

// The long-row launch may start while the row-block launch before it still
// runs (programmatic dependent launch); pdl_join_primary makes its grid
// complete only after both have, so work later in the stream sees every y row.
__device__ __forceinline__ void spmv_long_join() { pdl_join_primary(); }

// Long-row chunks units[unit0, unit1): no shared memory.
template <int DT, typename IT>
__global__ void __launch_bounds__(kSpmvWarps * 32, SpmvLongMinBlocks<DT, IT>::value)
k_spmv_long(const typename VT<DT>::Store* __restrict__ data, const IT* __restrict__ col,
            const typename VT<DT>::Store* __restrict__ x, typename VT<DT>::Store* __restrict__ y, fsb_spmv_plan plan,
            int64_t unit0, int64_t unit1) {
  using Tr = SpmvTraits<DT>;
  using S = typename Tr::S;
  using R = typename Tr::R;
  using Acc = SpmvAcc<DT, true>;  // long rows: always compensated

  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t unit = unit0 + int64_t(blockIdx.x) * kSpmvWarps + warp;
  if (unit >= unit1) return;  // whole warp leaves together

  const UnitRegs u = load_unit(plan.units + unit);
  // Offsets within the chunk are 32-bit (chunk_nnz < 2^31).  Columns run one
  // batch ahead; values are loaded beside the x gathers they pair with.
  Acc acc;
  acc.zero();
  const S* dp = data + u.s0;
  const IT* cp = col + u.s0;
  const int n = static_cast<int>(u.s1 - u.s0);
  IT cv[kSpmvItems];
#pragma unroll
  for (int k = 0; k < kSpmvItems; ++k) {
    const int i = k * 32 + lane;
    if (i < n) cv[k] = ld_stream(cp + i);
  }
  for (int base = 0; base < n; base += kSpmvBatch) {
    S av[kSpmvItems], xv[kSpmvItems];
#pragma unroll
    for (int k = 0; k < kSpmvItems; ++k) {
      const int i = base + k * 32 + lane;
      if (i < n) { xv[k] = ld_x(x + cv[k]); av[k] = ld_stream(dp + i); }
    }
    IT cn[kSpmvItems];
#pragma unroll
    for (int k = 0; k < kSpmvItems; ++k) {
      const int i = base + kSpmvBatch + k * 32 + lane;
      if (i < n) cn[k] = ld_stream(cp + i);
    }
#pragma unroll
    for (int k = 0; k < kSpmvItems; ++k) {
      if (base + k * 32 + lane < n) acc.add_prod(av[k], xv[k]);
    }
#pragma unroll
    for (int k = 0; k < kSpmvItems; ++k) cv[k] = cn[k];
  }
#pragma unroll
  for (int m = 16; m > 0; m >>= 1) acc.shfl_combine(m);
  if (u.nch == 1) {
    if (lane == 0) y[u.row] = acc.result();
    spmv_long_join();
    return;
  }
  const int64_t s0 = int64_t(u.slot) + (u.tag + 1);  // slot of this row's first chunk
  R* part = static_cast<R*>(plan.partials);
  int ticket = 0;
  if (lane == 0) {
    acc.store(part + int64_t(u.slot) * Acc::kPartialReals);
    __threadfence();
    ticket = atomicAdd(plan.counters + s0, 1);
  }
  ticket = __shfl_sync(0xffffffffu, ticket, 0);
  if (ticket != u.nch - 1) {
    spmv_long_join();
    return;
  }
  __threadfence();
  Acc fin;
  fin.zero();
  for (int64_t c = lane; c < u.nch; c += 32) {
    Acc p;
    p.load_cg(part + (s0 + c) * Acc::kPartialReals);
    fin.combine(p);
  }
#pragma unroll
  for (int m = 16; m > 0; m >>= 1) fin.shfl_combine(m);
  if (lane == 0) {
    y[u.row] = fin.result();
    plan.counters[s0] = 0;  // ready for the next call
  }
  spmv_long_join();
}

// Row-block units [0, n_units).  Persistent warps: units unit, unit + stride,
// ...; the next pass's values and columns (the next unit's at a unit's end)
// are loaded while the current pass's x gathers are in flight.  VEC: values and columns start
// on 32-byte boundaries, so a lane's run is read with wide loads.
template <int DT, typename IT, typename PT, bool SHORT_COMP, bool VEC>
__global__ void __launch_bounds__(kSpmvWarps * 32, SpmvRowMinBlocks<DT>::value)
k_spmv_rows(const typename VT<DT>::Store* __restrict__ data, const IT* __restrict__ col,
            const PT* __restrict__ ptr, const typename VT<DT>::Store* __restrict__ x,
            typename VT<DT>::Store* __restrict__ y, const fsb_spmv_unit* __restrict__ units, int64_t n_units,
            int64_t n_rows) {
  using S = typename VT<DT>::Store;
  using Row = SpmvRow;
  constexpr int kP = Row::kP;
  using Acc = typename std::conditional<(sizeof(S) <= 4), SpmvWide<DT>, SpmvAcc<DT, SHORT_COMP>>::type;
  __shared__ __align__(16) uint8_t sh_mark[kSpmvWarps][Row::kMarkBytes];
  // The long-row launch that follows is independent of this one (other rows,
  // its own scratch): let it start on the SMs this grid leaves.
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t unit = int64_t(blockIdx.x) * kSpmvWarps + warp;
  if (unit >= n_units) return;  // whole warp leaves together
  uint8_t* mark = sh_mark[warp];
  const int64_t nnz = ld_ptr(ptr, n_rows);  // wide loads stay below it
  const int64_t stride = int64_t(gridDim.x) * kSpmvWarps;
  UnitRegs u = load_unit(units + unit);
  S av[kP];
  IT cv[kP];
  // the lane's run of unit w's pass at p0 (positions from a0, w.s0 rounded down
  // to a whole run); entries outside the unit are left unset or unused
  auto load_run = [&](const UnitRegs& w, int p0) {
    const int64_t a0 = w.s0 & ~int64_t(kP - 1);
    const int64_t q = a0 + p0 + lane * kP;
    if (q >= w.s1) return;
    if (VEC && q + kP <= nnz) {
      ld_run<IT, kP>(col + q, cv);
      ld_run<S, kP>(data + q, av);
    } else {
#pragma unroll
      for (int k = 0; k < kP; ++k)
        if (q + k >= w.s0 && q + k < w.s1) {
          cv[k] = ld_stream(col + q + k);
          av[k] = ld_stream(data + q + k);
        }
    }
  };
  load_run(u, 0);
  for (int64_t uid = unit; uid < n_units; uid += stride) {
    const bool more = uid + stride < n_units;
    UnitRegs nxt = u;
    if (more) nxt = load_unit(units + uid + stride);
    const int64_t r0 = u.row;
    const int nr = u.tag - u.row;
    const int64_t a0 = u.s0 & ~int64_t(kP - 1);
    const int begin = static_cast<int>(u.s0 - a0), end = u.s1 > u.s0 ? static_cast<int>(u.s1 - a0) : 0;
    Acc open;  // the sum so far of the row that is open at the pass's start
    open.zero();
    for (int p0 = 0; p0 == 0 || p0 < end; p0 += Row::kPass) {
      const int p = p0 + lane * kP;
      S xv[kP], at[kP];
#pragma unroll
      for (int k = 0; k < kP; ++k) {
        if (p + k >= begin && p + k < end) {
          xv[k] = ld_x(x + cv[k]);
          at[k] = av[k];
        } else {  // no term: 0 * 0
          memset(&xv[k], 0, sizeof(S));
          memset(&at[k], 0, sizeof(S));
        }
      }
      // while x arrives: the next pass's run, or the next unit's first
      const bool last = p0 + Row::kPass >= end;
      if (!last) load_run(u, p0 + Row::kPass);
      else if (more) load_run(nxt, 0);
      if (p0 == 0) {
        // end marks: byte of a row's last nonzero = its local index + 1
        for (int i = lane; i < Row::kMarkBytes / 16; i += 32)
          reinterpret_cast<uint4*>(mark)[i] = make_uint4(0, 0, 0, 0);
        __syncwarp();
        for (int i = lane; i < nr; i += 32) {
          const int64_t b = ld_ptr(ptr, r0 + i), e = ld_ptr(ptr, r0 + i + 1);
          if (e > b) {
            mark[e - 1 - a0] = static_cast<uint8_t>(i + 1);
          } else {
            Acc z;
            z.zero();
            y[r0 + i] = z.result();
          }
        }
        __syncwarp();
      }
      uint32_t marks = 0;
      if (p < end) memcpy(&marks, __builtin_assume_aligned(mark + p, kP), kP);
      // sums in order; the first row that ends in the run may have begun before it
      Acc acc, first;
      acc.zero();
      first.zero();
      int first_row = 0;
#pragma unroll
      for (int k = 0; k < kP; ++k) {
        acc.add_prod(at[k], xv[k]);
        const int m = (marks >> (8 * k)) & 255;
        if (m) {
          if (first_row == 0) {
            first = acc;
            first_row = m;
          } else {
            y[r0 + m - 1] = acc.result();
          }
          acc.zero();
        }
      }
      if (lane == 0) {
        if (first_row) {
          Acc t = open;
          t.combine(first);
          first = t;
        } else {
          open.combine(acc);
          acc = open;
        }
      }
      // segmented inclusive scan of what each lane leaves open; a lane in which a
      // row ended starts a segment.  Only as many rounds as the longest segment
      // needs: short rows span few lanes.
      const unsigned closed = __ballot_sync(0xffffffffu, first_row != 0);
      const unsigned below = closed & (0xffffffffu >> (31 - lane));
      const int reach = below ? lane - (31 - __clz(below)) : lane;
      const int far = static_cast<int>(__reduce_max_sync(0xffffffffu, static_cast<unsigned>(reach)));
      for (int o = 1; o <= far; o <<= 1) {
        Acc other = acc;
        other.shfl_up(o);
        if (o <= reach) {
          other.combine(acc);
          acc = other;
        }
      }
      Acc carry = acc;
      carry.shfl_up(1);
      if (first_row) {
        if (lane > 0) {
          carry.combine(first);
          first = carry;
        }
        y[r0 + first_row - 1] = first.result();
      }
      open = acc;
      open.from_lane(31);
    }
    __syncwarp();  // the marks are rewritten by the next unit
    u = nxt;
  }
}

template <int DT, typename IT, typename PT, bool SHORT_COMP>
static int spmv_launch_mode(const void* data, const void* idx, const void* ptr, const void* x, void* y,
                            int64_t n_rows, const fsb_spmv_plan& plan, cudaStream_t st) {
  using S = typename VT<DT>::Store;
  const int64_t nb = plan.n_block_units, nu = plan.n_units;
  if (nb > 0) {
    const bool vec = (reinterpret_cast<uintptr_t>(data) | reinterpret_cast<uintptr_t>(idx)) % 32 == 0;
    auto kern = vec ? k_spmv_rows<DT, IT, PT, SHORT_COMP, true> : k_spmv_rows<DT, IT, PT, SHORT_COMP, false>;
    // persistent: at most the resident blocks (148 SMs); one block per 8 units
    // measured slower (92 against 88 us on 1 M rows of Poisson(16))
    const int64_t blocks = std::min<int64_t>(ceil_div(nb, kSpmvWarps), int64_t(148) * SpmvRowMinBlocks<DT>::value);
    kern<<<(unsigned)blocks, kSpmvWarps * 32, 0, st>>>(
        static_cast<const S*>(data), static_cast<const IT*>(idx), static_cast<const PT*>(ptr),
        static_cast<const S*>(x), static_cast<S*>(y), plan.units, nb, n_rows);
    FSB_LAUNCH_CHECK();
  }
  if (nu > nb) {  // long-row chunks: no shared memory
    // after a row-block launch: a programmatic dependent launch, so its blocks
    // fill the SMs the row-block grid's tail leaves (see spmv_long_join)
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ceil_div(nu - nb, kSpmvWarps));
    cfg.blockDim = dim3(kSpmvWarps * 32);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = nb > 0 ? 1 : 0;
    if (cudaLaunchKernelEx(&cfg, k_spmv_long<DT, IT>, static_cast<const S*>(data), static_cast<const IT*>(idx),
                           static_cast<const S*>(x), static_cast<S*>(y), plan, nb, nu) != cudaSuccess) {
      (void)cudaGetLastError();
      return FSB_ERR_LAUNCH;
    }
  }
  return FSB_OK;
}

template <int DT, typename IT, typename PT>
static int spmv_launch(const void* data, const void* idx, const void* ptr, const void* x, void* y,
                       int64_t n_rows, const fsb_spmv_plan& plan, cudaStream_t st) {
  // any window up to kCap fits the end marks (<= cap rows, < 2*cap nonzeros)
  if (plan.cap < 1 || plan.cap > SpmvRow::kCap || plan.chunk_nnz % kSpmvBatch != 0) return FSB_ERR_INVALID_ARG;
  // plain sums of the short rows on request; the 2- and 4-byte types sum them in fp64 at no more cost
  if constexpr (sizeof(typename VT<DT>::Store) > 4)
    if (plan.flags & FSB_SPMV_FAST_SHORT_ROWS)
      return spmv_launch_mode<DT, IT, PT, false>(data, idx, ptr, x, y, n_rows, plan, st);
  return spmv_launch_mode<DT, IT, PT, true>(data, idx, ptr, x, y, n_rows, plan, st);
}

template <int DT>
static int spmv_dispatch_idx(const void* data, const void* idx, int i64, const void* ptr, int p64, const void* x,
                             void* y, int64_t n_rows, const fsb_spmv_plan& plan, cudaStream_t st) {
  if (i64) {
    return p64 ? spmv_launch<DT, int64_t, int64_t>(data, idx, ptr, x, y, n_rows, plan, st)
               : spmv_launch<DT, int64_t, int32_t>(data, idx, ptr, x, y, n_rows, plan, st);
  }
  return p64 ? spmv_launch<DT, int32_t, int64_t>(data, idx, ptr, x, y, n_rows, plan, st)
             : spmv_launch<DT, int32_t, int32_t>(data, idx, ptr, x, y, n_rows, plan, st);
}

// ---------------------------------------------------------------------------
// The x-gather floor of a CSR SpMV (measurement only): out[b] = sum of
// data[i] * x[col[i]] over block b's grid-stride share of all nnz nonzeros,
// fp64 sums.  It moves the SpMV's values, columns and x gathers with the same
// load flavours (streaming values / columns, L2-only x) and 8 gathers in
// flight per thread, without the row structure: its time bounds what any
// CSR SpMV of the same pattern can reach.
// ---------------------------------------------------------------------------
constexpr int kFloorThreads = 256;
constexpr int kFloorItems = 8;

template <int DT, typename IT>
__global__ void __launch_bounds__(kFloorThreads)
k_gather_floor(const typename VT<DT>::Store* __restrict__ data, const IT* __restrict__ col, int64_t nnz,
               const typename VT<DT>::Store* __restrict__ x, double* __restrict__ out) {
  using S = typename VT<DT>::Store;
  __shared__ double red[kFloorThreads / 32];
  double acc = 0.0;
  const int64_t step = int64_t(gridDim.x) * kFloorThreads * kFloorItems;
  for (int64_t base = int64_t(blockIdx.x) * kFloorThreads * kFloorItems; base < nnz; base += step) {
    S av[kFloorItems], xv[kFloorItems];
#pragma unroll
    for (int q = 0; q < kFloorItems; ++q) {
      const int64_t i = base + q * kFloorThreads + threadIdx.x;
      if (i < nnz) {
        av[q] = ld_stream(data + i);
        xv[q] = ld_x(x + ld_stream(col + i));
      }
    }
#pragma unroll
    for (int q = 0; q < kFloorItems; ++q)
      if (base + q * kFloorThreads + threadIdx.x < nnz) acc = fma(double(to_real(av[q])), double(to_real(xv[q])), acc);
  }
#pragma unroll
  for (int m = 16; m > 0; m >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, m);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < kFloorThreads / 32; ++w) t += red[w];
    out[blockIdx.x] = t;
  }
}

template <int DT>
static int gather_floor_launch(const void* data, const void* idx, int i64, int64_t nnz, const void* x, double* out,
                               int64_t blocks, cudaStream_t st) {
  using S = typename VT<DT>::Store;
  if (i64)
    k_gather_floor<DT, int64_t><<<(unsigned)blocks, kFloorThreads, 0, st>>>(
        static_cast<const S*>(data), static_cast<const int64_t*>(idx), nnz, static_cast<const S*>(x), out);
  else
    k_gather_floor<DT, int32_t><<<(unsigned)blocks, kFloorThreads, 0, st>>>(
        static_cast<const S*>(data), static_cast<const int32_t*>(idx), nnz, static_cast<const S*>(x), out);
  FSB_LAUNCH_CHECK();
  return FSB_OK;
}

// ---------------------------------------------------------------------------
// Built-in long-row scratch of fsb_spmv_csr_static_scratch: partial sums of
// the widest type (c128, 32 bytes) for every slot, then one int32 ticket per
// slot.  Zero at module load; every call clears the tickets it uses.
// ---------------------------------------------------------------------------
constexpr int64_t kStaticSlots = FSB_SPMV_STATIC_MAX_SLOTS;
constexpr int64_t kStaticPartialBytes = 4 * sizeof(double);
constexpr int64_t kStaticTicketOffset = kStaticSlots * kStaticPartialBytes;
static __device__ __align__(256) unsigned char g_spmv_static_scratch[kStaticTicketOffset + kStaticSlots * sizeof(int32_t)];

constexpr int kStaticMaxDevices = 256;
struct StaticScratchEntry {
  unsigned long long ctx_id;  // the context the address was resolved in (0: none yet)
  void* addr;
};
static StaticScratchEntry g_static_cache[kStaticMaxDevices];
static std::mutex g_static_mu;

// Unique id of the calling thread's current context, 0 if there is none or the
// driver cannot tell.  A device reset (or a new primary context) gives a new
// id, so an address resolved in an earlier context is never reused.
typedef CUresult (*PfnCtxGetCurrent)(CUcontext*);
typedef CUresult (*PfnCtxGetId)(CUcontext, unsigned long long*);
static unsigned long long current_context_id() {
  static PfnCtxGetCurrent get_current = nullptr;
  static PfnCtxGetId get_id = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      get_current = reinterpret_cast<PfnCtxGetCurrent>(p);
    else
      (void)cudaGetLastError();
    p = nullptr;
    if (cudaGetDriverEntryPoint("cuCtxGetId", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      get_id = reinterpret_cast<PfnCtxGetId>(p);
    else
      (void)cudaGetLastError();
  });
  if (!get_current || !get_id) return 0;
  CUcontext ctx = nullptr;
  unsigned long long id = 0;
  if (get_current(&ctx) != CUDA_SUCCESS || !ctx) return 0;
  if (get_id(ctx, &id) != CUDA_SUCCESS) return 0;
  return id;
}

// Device address of the current device's scratch.  cudaGetSymbolAddress runs
// once per device and context: on the first call, and again only after the
// device's context changed (a device reset).  `st` must belong to the current
// device: the scratch of another device is not reachable through it.
static int static_scratch_address(cudaStream_t st, void** out) {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    (void)cudaGetLastError();
    return FSB_ERR_CUDA;
  }
  if (dev < 0 || dev >= kStaticMaxDevices) return FSB_ERR_UNSUPPORTED;
  int sdev = -1;
  if (cudaStreamGetDevice(st, &sdev) != cudaSuccess) {
    (void)cudaGetLastError();
    return FSB_ERR_INVALID_ARG;
  }
  if (sdev != dev) return FSB_ERR_INVALID_ARG;
  const unsigned long long ctx = current_context_id();
  std::lock_guard<std::mutex> lock(g_static_mu);
  StaticScratchEntry& e = g_static_cache[dev];
  if (!e.addr || (ctx != 0 && e.ctx_id != ctx)) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_spmv_static_scratch) != cudaSuccess || !p) {
      (void)cudaGetLastError();
      return FSB_ERR_CUDA;
    }
    e.addr = p;
    e.ctx_id = current_context_id();  // the symbol lookup made the device's context current
  }
  *out = e.addr;
  return FSB_OK;
}

}  // namespace fsb

using namespace fsb;

extern "C" {

int64_t fsb_spmv_partial_bytes(int dtype) {
  switch (dtype) {
    case FSB_F16: case FSB_BF16: case FSB_F32: return 2 * sizeof(float);
    case FSB_F64: return 2 * sizeof(double);
    case FSB_C64: return 4 * sizeof(float);
    case FSB_C128: return 4 * sizeof(double);
    default: return -1;
  }
}

int fsb_spmv_csr(int dtype, const void* data, const void* indices, int idx_is_64, const void* indptr, int ptr_is_64,
                 int64_t n_rows, int64_t n_cols, const void* x, void* y, const fsb_spmv_plan* plan, void* stream) {
  if (!plan || n_rows < 0 || n_cols < 0) return FSB_ERR_INVALID_ARG;
  if (n_rows == 0 || plan->n_units == 0) return FSB_OK;
  if (!indptr || !y || !plan->units || plan->cap < 1 || plan->chunk_nnz < 1 || plan->n_slots < 0 ||
      plan->n_block_units < 0 || plan->n_block_units > plan->n_units ||
      (plan->n_slots > 0 && (!plan->partials || !plan->counters)))
    return FSB_ERR_INVALID_ARG;
  if (plan->n_units >= INT32_MAX) return FSB_ERR_UNSUPPORTED;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  switch (dtype) {
    case FSB_F16: return spmv_dispatch_idx<FSB_F16>(data, indices, idx_is_64, indptr, ptr_is_64, x, y, n_rows, *plan, st);
    case FSB_BF16: return spmv_dispatch_idx<FSB_BF16>(data, indices, idx_is_64, indptr, ptr_is_64, x, y, n_rows, *plan, st);
    case FSB_F32: return spmv_dispatch_idx<FSB_F32>(data, indices, idx_is_64, indptr, ptr_is_64, x, y, n_rows, *plan, st);
    case FSB_F64: return spmv_dispatch_idx<FSB_F64>(data, indices, idx_is_64, indptr, ptr_is_64, x, y, n_rows, *plan, st);
    case FSB_C64: return spmv_dispatch_idx<FSB_C64>(data, indices, idx_is_64, indptr, ptr_is_64, x, y, n_rows, *plan, st);
    case FSB_C128: return spmv_dispatch_idx<FSB_C128>(data, indices, idx_is_64, indptr, ptr_is_64, x, y, n_rows, *plan, st);
    default: return FSB_ERR_UNSUPPORTED;
  }
}

int fsb_spmv_gather_floor(int dtype, const void* data, const void* indices, int idx_is_64, int64_t nnz,
                          const void* x, double* out, int64_t n_out, void* stream) {
  if (nnz < 0 || n_out < 1 || !out || (nnz > 0 && (!data || !indices || !x))) return FSB_ERR_INVALID_ARG;
  const int64_t blocks = std::min<int64_t>(n_out, int64_t(148) * 8);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  switch (dtype) {
    case FSB_F16: return gather_floor_launch<FSB_F16>(data, indices, idx_is_64, nnz, x, out, blocks, st);
    case FSB_BF16: return gather_floor_launch<FSB_BF16>(data, indices, idx_is_64, nnz, x, out, blocks, st);
    case FSB_F32: return gather_floor_launch<FSB_F32>(data, indices, idx_is_64, nnz, x, out, blocks, st);
    case FSB_F64: return gather_floor_launch<FSB_F64>(data, indices, idx_is_64, nnz, x, out, blocks, st);
    default: return FSB_ERR_UNSUPPORTED;
  }
}

int fsb_spmv_csr_static_scratch(int dtype, const void* data, const void* indices, int idx_is_64, const void* indptr,
                                int ptr_is_64, int64_t n_rows, int64_t n_cols, const void* x, void* y,
                                const fsb_spmv_plan* plan, void* stream) {
  if (!plan || n_rows < 0 || n_cols < 0 || plan->n_slots < 0) return FSB_ERR_INVALID_ARG;
  if (plan->n_slots > kStaticSlots) return FSB_ERR_TOO_LARGE;
  if (fsb_spmv_partial_bytes(dtype) < 0) return FSB_ERR_UNSUPPORTED;
  if (n_rows == 0 || plan->n_units == 0) return FSB_OK;
  fsb_spmv_plan p = *plan;
  p.partials = nullptr;
  p.counters = nullptr;
  if (p.n_slots > 0) {
    void* base = nullptr;
    const int rc = static_scratch_address(static_cast<cudaStream_t>(stream), &base);
    if (rc != FSB_OK) return rc;
    p.partials = base;
    p.counters = reinterpret_cast<int32_t*>(static_cast<unsigned char*>(base) + kStaticTicketOffset);
    if (cudaMemsetAsync(p.counters, 0, size_t(p.n_slots) * sizeof(int32_t), static_cast<cudaStream_t>(stream)) !=
        cudaSuccess) {
      (void)cudaGetLastError();
      return FSB_ERR_CUDA;
    }
  }
  return fsb_spmv_csr(dtype, data, indices, idx_is_64, indptr, ptr_is_64, n_rows, n_cols, x, y, &p, stream);
}

}  // extern "C"
