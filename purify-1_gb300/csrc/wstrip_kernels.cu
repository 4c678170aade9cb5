// sm_103a kernels of the row-factor operators on the tensor cores (see
// wplan.h WStripPlan): G, G^H and the sum of the task windows.
//
// A row K = sum_e A_e B_e^T touches S x S cells, so a run of rows whose
// footprints start in the same 8 x 8 cells is a matrix product over a few
// 8 x 8 blocks of the grid.  Both kernels give a warp such runs and use
// mma.m16n8k16 with BF16 operands: the 16 rows are the real and the imaginary
// parts of 8 values, the columns the real and the imaginary parts of 8 terms.
//
// Precision.  Every operand x is split into three pieces of 8 bits, x = x1 + x2 +
// x3, each the BF16 nearest to what the ones before it leave (a split of FP32
// into narrower pieces whose products are summed in FP32: Markidis et al. 2018,
// Ootomo and Yokota 2022).  The split is exact, 24 bits in all.  Six of the nine
// products are summed, the smallest first:
//   a3 b1, a1 b3, a2 b2, a1 b2, a2 b1, a1 b1;
// what is left out (a2 b3, a3 b2, a3 b3) is below 2^-24 of a product, 2^-27 in the
// mean.  The 16 columns of an instruction hold both halves of a complex product:
// 8 terms times real parts, 8 times imaginary parts.  The unit truncates its
// sums, so each block's product starts from zero and is added to the FP32 sums
// outside with rounding.
//
// Error of G and of G^H alone, random values, 10^6 rows of 4 to 24 taps (relative L2
// against FP64): 7.7e-8 and 1.16e-7; the band kernels of wkernels.cu 8.3e-8 and
// 1.66e-7.
//
// What bounds them: on paper the mma rate, measured 0.5 a cycle and SM.  A 1024^2
// image with 10^6 rows of 4 to 24 taps takes 215 us (G) and 280 (G^H), 269 and 542
// with the band kernels, 187 and 261 with two TF32 pieces of 11 bits, which lost
// precision (1.0e-7 in G).  The registers of the blocks and shared memory leave
// 10 to 14 warps an SM, whose chains of dependent products and splits are the
// limit.
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "cplx_ops.cuh"
#include "pdl.cuh"
#include "wstrip_kernels.h"

namespace pg {
namespace {

using dev::add2;
using dev::fma2;

// Warps of a G^H CTA; they share nothing but the shared-memory array.
constexpr int kStripWarps = 2;

// The three pieces of two values, the first in the lower halves: two columns of
// an operand, so that the terms t and t + 4 of a lane are columns 2 t and 2 t + 1.
struct Pieces {
  uint32_t p[3];
};
__device__ __forceinline__ uint32_t pack_bf16(float x, float y) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(y), "f"(x));
  return r;
}
// Two complex values: the pieces of their real and of their imaginary parts.
struct Split {
  Pieces re, im;
};
// what the pieces p leave of the values
__device__ __forceinline__ void split_rest(float2 &v0, float2 &v1, uint32_t re, uint32_t im) {
  const float2 minus = make_float2(-1.f, -1.f);
  v0 = fma2(make_float2(__uint_as_float(re << 16), __uint_as_float(im << 16)), minus, v0);
  v1 = fma2(make_float2(__uint_as_float(re & 0xffff0000u), __uint_as_float(im & 0xffff0000u)),
            minus, v1);
}
template <bool UP>
__device__ __forceinline__ Split split(float2 v0, float2 v1) {
  // x (1 + kTrunc): one operand of each product makes up for what the unit's
  // truncation takes from a product on average (measured 3.5 to 4.0e-8 of it:
  // random, same-sign and nearly equal operands, 1 to 8 terms).
  constexpr float kTrunc = 4.0e-8f;
  const float2 x0 = v0, x1 = v1;
  Split s;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    s.re.p[k] = pack_bf16(v0.x, v1.x);
    s.im.p[k] = pack_bf16(v0.y, v1.y);
    if (k < 2) split_rest(v0, v1, s.re.p[k], s.im.p[k]);
    if (UP && k == 0) {
      v0 = fma2(x0, make_float2(kTrunc, kTrunc), v0);
      v1 = fma2(x1, make_float2(kTrunc, kTrunc), v1);
    }
  }
  return s;
}

// d = a b (16 x 16 by 16 x 8), and d += a b
__device__ __forceinline__ void mma0(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                     uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
      "{%8, %9}, {%10, %10, %10, %10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ void mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                    uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
      "{%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// The left operand: rows g and g + 8 at the columns of the real parts, rows g
// and g + 8 at those of the imaginary parts.
struct Rows {
  uint32_t p[3][4];
};
__device__ __forceinline__ Rows rows(const Pieces &re0, const Pieces &im0, const Pieces &re1,
                                     const Pieces &im1) {
  Rows r;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    r.p[k][0] = re0.p[k];
    r.p[k][1] = im0.p[k];
    r.p[k][2] = re1.p[k];
    r.p[k][3] = im1.p[k];
  }
  return r;
}
__device__ __forceinline__ Pieces negate(Pieces x) {
#pragma unroll
  for (int k = 0; k < 3; ++k) x.p[k] ^= 0x80008000u;
  return x;
}
// d = left operand times right operand for TV blocks, independent chains of
// six products: of the blocks i, left operand a(i) and right operand b(i).
template <int TV, typename A, typename B>
__device__ __forceinline__ void multiply(float (&d)[TV][4], A a, B b) {
  constexpr int order[6][2] = {{2, 0}, {0, 2}, {1, 1}, {0, 1}, {1, 0}, {0, 0}};
#pragma unroll
  for (int k = 0; k < 6; ++k)
#pragma unroll
    for (int i = 0; i < TV; ++i) {
      const uint32_t(&l)[4] = a(i).p[order[k][0]];
      const uint32_t re = b(i).re.p[order[k][1]], im = b(i).im.p[order[k][1]];
      if (k == 0)
        mma0(d[i], l[0], l[1], l[2], l[3], re, im);
      else
        mma(d[i], l[0], l[1], l[2], l[3], re, im);
    }
}
// One factor pair (WTerm) as a lane needs it.
struct Term {
  const float2 *A, *B;
  int S, dv, du, rank, m, blocks;
  float2 w;
};
// A term as loaded, decoded where it is used: decoding it at the load would
// wait for it there.
struct RawTerm {
  int4 x, y;
};
__device__ __forceinline__ RawTerm load_raw(const WStripArgs &a, int64_t k) {
  const int4 *p = reinterpret_cast<const int4 *>(a.terms + k);
  RawTerm r;
  asm volatile("ld.global.nc.v4.s32 {%0, %1, %2, %3}, [%4];"
               : "=r"(r.x.x), "=r"(r.x.y), "=r"(r.x.z), "=r"(r.x.w)
               : "l"(p));
  asm volatile("ld.global.nc.v4.s32 {%0, %1, %2, %3}, [%4];"
               : "=r"(r.y.x), "=r"(r.y.y), "=r"(r.y.z), "=r"(r.y.w)
               : "l"(p + 1));
  return r;
}
__device__ __forceinline__ Term decode(const WStripArgs &a, const RawTerm &r) {
  int4 x = r.x, y = r.y;
  asm volatile("" : "+r"(x.x), "+r"(x.y), "+r"(x.z), "+r"(x.w), "+r"(y.x), "+r"(y.y), "+r"(y.z), "+r"(y.w));
  Term t;
  const int64_t off = (int64_t(x.y) << 32) | uint32_t(x.x);
  t.A = static_cast<const float2 *>(a.factors) + off;
  t.B = t.A + x.z;
  t.m = x.w;
  t.w = make_float2(__int_as_float(y.x), __int_as_float(y.y));
  t.dv = y.z & 15;
  t.du = (y.z >> 4) & 15;
  t.S = (y.z >> 8) & 255;
  t.rank = y.z >> 16;
  t.blocks = y.w;
  return t;
}
__device__ __forceinline__ Term load_term(const WStripArgs &a, int64_t k) {
  return decode(a, load_raw(a, k));
}
// 8 bytes from global to shared memory, zeros where !there.
__device__ __forceinline__ void cp_async8_zfill(unsigned smem, const void *gmem, bool there) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(smem), "l"(gmem),
               "r"(there ? 8 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async16(unsigned smem, const void *gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}
__device__ __forceinline__ unsigned smem_address(const void *p) {
  return static_cast<unsigned>(__cvta_generic_to_shared(p));
}
// Eight terms of G^H: lane (g, t) holds A of the terms t and t + 4 at the rows
// 8 i + g, times conj(weight) y, and B of the same terms at the columns
// 8 j + g.  Adds scale conj(A) conj(B) z to TV x tu window blocks from block
// row H on: with conj(A) z = r + i s, (r + i s) (B.x - i B.y) is the product of
// the rows (r, s) with B's real parts and (s, -r) with its imaginary parts.  The
// blocks of a column are independent chains.
template <int H, int TV, int TM>
__device__ __forceinline__ void grid_column(float2 (&acc)[TM + 1][TM][2], const Rows (&a)[TM],
                                            const Split &b, float scale, int j) {
  float c[TV][4];
  multiply<TV>(c, [&](int i) -> const Rows & { return a[i]; },
               [&](int) -> const Split & { return b; });
#pragma unroll
  for (int i = 0; i < TV; ++i)
#pragma unroll
    for (int h = 0; h < 2; ++h)
      acc[H + i][j][h] = fma2(make_float2(c[i][2 * h], c[i][2 * h + 1]), make_float2(scale, scale),
                              acc[H + i][j][h]);
}
template <int N>
using Int = std::integral_constant<int, N>;
// Calls f(Int<H>, Int<TV>) for the shape of an octet.
template <int H, int TM, typename F>
__device__ __forceinline__ void with_shape(int tv, F f) {
  if constexpr (TM >= 4)
    if (tv == 4) return f(Int<H>(), Int<4>());
  if constexpr (TM >= 3)
    if (tv == 3) return f(Int<H>(), Int<3>());
  if constexpr (TM >= 2)
    if (tv == 2) return f(Int<H>(), Int<2>());
  f(Int<H>(), Int<1>());
}
// At TM = 4 the columns are outside and the shape is looked at for each: with
// every shape's columns unrolled, splits and all, the code outgrows the
// instruction cache (warps of one SM are in different shapes).
template <int TM>
__device__ __forceinline__ void grid_oct(float2 (&acc)[TM + 1][TM][2], const float4 (*A)[32],
                                         const float4 (*B)[32], float2 z0, float2 z1, float scale,
                                         bool half, int tv, int tu) {
  Rows a[TM];
  auto split_column = [&](int j) {
    const float4 v = B[j][0];
    return split<true>(make_float2(v.x, v.y), make_float2(v.z, v.w));
  };
  auto split_rows = [&](int i) {
    const float4 v = A[i][0];
    const Split x = split<false>(
        make_float2(fmaf(v.x, z0.x, v.y * z0.y), fmaf(v.x, z0.y, -(v.y * z0.x))),
        make_float2(fmaf(v.z, z1.x, v.w * z1.y), fmaf(v.z, z1.y, -(v.w * z1.x))));
    a[i] = rows(x.re, x.im, x.im, negate(x.re));
  };
  if constexpr (TM >= 4) {
#pragma unroll
    for (int i = 0; i < TM; ++i)
      if (i < tv) split_rows(i);
#pragma unroll
    for (int j = 0; j < TM; ++j)
      if (j < tu) {
        const Split b = split_column(j);
        auto column = [&](auto h, auto n) {
          grid_column<decltype(h)::value, decltype(n)::value, TM>(acc, a, b, scale, j);
        };
        if (half)
          with_shape<1, TM>(tv, column);
        else
          with_shape<0, TM>(tv, column);
      }
  } else {
    auto columns = [&](auto h, auto n) {
      constexpr int H = decltype(h)::value, TV = decltype(n)::value;
#pragma unroll
      for (int i = 0; i < TV; ++i) split_rows(i);
#pragma unroll
      for (int j = 0; j < TM; ++j)
        if (j < tu) {
          const Split b = split_column(j);
          grid_column<H, TV, TM>(acc, a, b, scale, j);
        }
    };
    if (half)
      with_shape<1, TM>(tv, columns);
    else
      with_shape<0, TM>(tv, columns);
  }
}

// The same eight terms cell by cell: only cells of a term's footprint are
// touched, so an infinite or NaN visibility stays inside it (in the products
// above, zero factors outside would turn it into NaN).
template <int TM>
__device__ __noinline__ void grid_oct_scalar(float2 (*acc)[TM][2], const WStripArgs &a,
                                             int64_t term0, float2 z0, float2 z1, int lane) {
  const int g = lane >> 2, t = lane & 3;
  for (int u = 0; u < kOctTerms; ++u) {
    const Term x = load_term(a, term0 + u);
    const float2 mine = u < 4 ? z0 : z1;
    const float2 z = make_float2(__shfl_sync(0xffffffffu, mine.x, u & 3),
                                 __shfl_sync(0xffffffffu, mine.y, u & 3));
    const int half = (x.blocks >> 8) & 1;
    for (int i = 0; i < TM; ++i) {
      const int jv = 8 * i + g - x.dv;
      if (unsigned(jv) >= unsigned(x.S)) continue;
      const float2 av = x.A[jv];
      for (int j = 0; j < TM; ++j)
        for (int c = 0; c < 2; ++c) {
          const int ju = 8 * j + 2 * t + c - x.du;
          if (unsigned(ju) >= unsigned(x.S)) continue;
          const float2 bv = x.B[ju];
          const float2 bz = make_float2(bv.x * z.x + bv.y * z.y, bv.x * z.y - bv.y * z.x);
          float2 &re = acc[half + i][j][0], &im = acc[half + i][j][1];
          const float vr = av.x * bz.x + av.y * bz.y, vi = av.x * bz.y - av.y * bz.x;
          if (c == 0) {
            re.x += vr;
            im.x += vi;
          } else {
            re.y += vr;
            im.y += vi;
          }
        }
    }
  }
}

// Visibilities this small or large are scaled to about 1 for the products:
// exponents below 2^-60 or above 2^60 (0 is neither).
__device__ __forceinline__ bool far_from_one(unsigned top) {
  return top - 0x21800000u > 0x5d800000u - 0x21800000u && top != 0;
}

// G^H, one warp per task.  The warp keeps the window's blocks over the
// current group and the TM - 1 to its right in registers (two halves of the
// strip: TM + 1 block rows).  After a group the leftmost block column is
// complete and is stored; the others move one place to the left.  The factors
// and visibilities of kGridAhead octs are on their way by cp.async, each lane
// copying the operands it will use itself (8 lanes read 64 contiguous bytes
// of one row), so that no lane waits for another.
constexpr int kGridAhead = 2;
template <int TM>
struct GridStage {
  float4 A[TM][32], B[TM][32];  // the terms t and t + 4
  float4 y[32], w[32];          // their visibilities and weights
  int blocks[32];
};
template <int TM>
struct GridShared {
  GridStage<TM> stages[kGridAhead];
  // the terms of oct o at place o mod 4, copied two octs before they are used
  // (a load into registers would share its scoreboard with the loop's other
  // loads, which then wait for it)
  int4 terms[4][2 * kOctTerms];
};
template <int TM>
__global__ void __launch_bounds__(kStripWarps * 32, 5) wstrip_grid_kernel(const WStripArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  dev::pdl_launch_next();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  GridShared<TM> &shared = reinterpret_cast<GridShared<TM> *>(smem_raw)[warp];
  GridStage<TM> *stages = shared.stages;
  const int slot = int(blockIdx.x) * kStripWarps + warp;
  if (slot >= a.ntasks) {
    dev::pdl_wait();
    return;
  }
  const WStripTask tk = a.tasks[a.order[slot]];
  const int32_t *goct = a.group_oct + tk.oct0;
  const int oend = goct[tk.groups];
  const float2 *vis = static_cast<const float2 *>(a.vis_in);
  float2 acc[TM + 1][TM][2];
#pragma unroll
  for (int i = 0; i <= TM; ++i)
#pragma unroll
    for (int j = 0; j < TM; ++j) acc[i][j][0] = acc[i][j][1] = make_float2(0.f, 0.f);
  int o = goct[0];  // the oct computed next
  int o1 = o;       // the oct copied next
  auto copy_terms = [&](int oct) {
    if (lane < 2 * kOctTerms && oct < oend)
      cp_async16(smem_address(&shared.terms[oct & 3][lane]),
                 reinterpret_cast<const int4 *>(a.terms + int64_t(oct) * kOctTerms) + lane);
  };
  auto term_at = [&](int oct, int k) {
    const RawTerm r{shared.terms[oct & 3][2 * k], shared.terms[oct & 3][2 * k + 1]};
    return decode(a, r);
  };
  auto issue = [&](GridStage<TM> &st) {
    if (o1 < oend) {
      const Term n0 = term_at(o1, t), n1 = term_at(o1, t + 4);
      const int tv = n0.blocks & 15, tu = (n0.blocks >> 4) & 15;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const Term &x = e ? n1 : n0;
        const int jv = g - x.dv, ju = g - x.du;
        const float2 *pa = x.A + jv, *pb = x.B + ju;
        const int la = x.S - jv, lb = x.S - ju;
        const unsigned sa = smem_address(&st.A[0][lane]) + 8 * e, sb = smem_address(&st.B[0][lane]) + 8 * e;
#pragma unroll
        for (int i = 0; i < TM; ++i) {
          if (i < tv) cp_async8_zfill(sa + 512 * i, pa + 8 * i, la > 8 * i && (i > 0 || jv >= 0));
          if (i < tu) cp_async8_zfill(sb + 512 * i, pb + 8 * i, lb > 8 * i && (i > 0 || ju >= 0));
        }
        cp_async8_zfill(smem_address(&st.y[lane]) + 8 * e, vis + max(x.m, 0), x.m >= 0);
      }
      st.w[lane] = make_float4(n0.w.x, n0.w.y, n1.w.x, n1.w.y);
      st.blocks[lane] = n0.blocks;
      copy_terms(o1 + 2);
      ++o1;
    }
    cp_async_commit();
  };
  copy_terms(o);
  copy_terms(o + 1);
  cp_async_commit();
  cp_async_wait<0>();
  __syncwarp();
  dev::pdl_wait();  // the visibilities are the previous kernel's output
#pragma unroll 1
  for (int k = 0; k < kGridAhead; ++k) issue(stages[k]);
  int place = 0;
  float2 *win = static_cast<float2 *>(a.windows) + tk.window;
  int oe = goct[1];
  for (int grp = 0; grp < tk.groups; ++grp) {
    const int oe1 = grp + 1 < tk.groups ? goct[grp + 2] : 0;
    for (; o < oe; ++o) {
      static_assert(kGridAhead == 2, "the places of the terms count on two octs ahead");
      cp_async_wait<kGridAhead - 1>();
      __syncwarp();  // the terms copied with this oct's operands, by other lanes
      GridStage<TM> &st = stages[place];
      place = place + 1 == kGridAhead ? 0 : place + 1;
      const float4 y = st.y[lane], w = st.w[lane];
      const int blocks = st.blocks[lane];
      // z = conj(weight) y
      float2 z0 = make_float2(fmaf(w.x, y.x, w.y * y.y), fmaf(w.x, y.y, -(w.y * y.x)));
      float2 z1 = make_float2(fmaf(w.z, y.z, w.w * y.w), fmaf(w.z, y.w, -(w.w * y.z)));
      const unsigned top0 = max(__float_as_uint(fabsf(z0.x)), __float_as_uint(fabsf(z0.y)));
      const unsigned top1 = max(__float_as_uint(fabsf(z1.x)), __float_as_uint(fabsf(z1.y)));
      const int tv = blocks & 15, tu = (blocks >> 4) & 15;
      float scale = 1.f;
      if (__any_sync(0xffffffffu, far_from_one(top0) || far_from_one(top1))) {
        const unsigned top = __reduce_max_sync(0xffffffffu, max(top0, top1));
        if (top >= 0x7f800000u) {
          // through a copy, so that acc itself stays in registers
          float2 copy[TM + 1][TM][2];
#pragma unroll
          for (int i = 0; i <= TM; ++i)
#pragma unroll
            for (int j = 0; j < TM; ++j)
#pragma unroll
              for (int e = 0; e < 2; ++e) copy[i][j][e] = acc[i][j][e];
          grid_oct_scalar<TM>(copy, a, int64_t(o) * kOctTerms, z0, z1, lane);
#pragma unroll
          for (int i = 0; i <= TM; ++i)
#pragma unroll
            for (int j = 0; j < TM; ++j)
#pragma unroll
              for (int e = 0; e < 2; ++e) acc[i][j][e] = copy[i][j][e];
          issue(st);
          continue;
        }
        // by powers of two, kept where both are normal
        const unsigned e = min(max(top >> 23, 1u), 253u);
        const float up = __uint_as_float((254u - e) << 23);
        scale = __uint_as_float(e << 23);
        z0 = make_float2(z0.x * up, z0.y * up);
        z1 = make_float2(z1.x * up, z1.y * up);
      }
      const float4(*sa)[32] = reinterpret_cast<const float4(*)[32]>(&st.A[0][lane]);
      const float4(*sb)[32] = reinterpret_cast<const float4(*)[32]>(&st.B[0][lane]);
      grid_oct<TM>(acc, sa, sb, z0, z1, scale, (blocks >> 8) & 1, tv, tu);
      issue(st);
    }
    oe = oe1;
    // store the leftmost block column (after the last group, all of them);
    // shift the others
    const bool last = grp + 1 == tk.groups;
#pragma unroll
    for (int j = 0; j < TM; ++j) {
      if (j > 0 && !last) break;
      float2 *col = win + 8 * (grp + j) + 2 * t;
#pragma unroll
      for (int i = 0; i <= TM; ++i) {
        const int row = 8 * i + g;
        if (row < a.rows)
          *reinterpret_cast<float4 *>(col + size_t(row) * tk.width) = make_float4(
              acc[i][j][0].x, acc[i][j][1].x, acc[i][j][0].y, acc[i][j][1].y);
      }
    }
#pragma unroll
    for (int i = 0; i <= TM; ++i)
#pragma unroll
      for (int j = 0; j < TM; ++j) {
        acc[i][j][0] = j + 1 < TM ? acc[i][j + 1 < TM ? j + 1 : j][0] : make_float2(0.f, 0.f);
        acc[i][j][1] = j + 1 < TM ? acc[i][j + 1 < TM ? j + 1 : j][1] : make_float2(0.f, 0.f);
      }
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");
}

// Element (row, column of its block of 8) of a block column in shared memory:
// the two halves of odd row pairs are swapped, so that the 16 lanes of a
// half-warp (4 rows, 4 columns) fall on 16 different bank pairs.
__device__ __forceinline__ int block_at(int row, int c) {
  return row * 8 + (c ^ ((row & 2) << 1));
}
__device__ __forceinline__ void cp_async8(void *smem, const void *gmem) {
  const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem) : "memory");
}

// T[term][row] = sum over columns of B x grid for TV block rows from row0 on
// (lane: term g, rows 8 i + 2 t and 8 i + 2 t + 1; real parts, imaginary
// parts) and tu block columns, `ring` the block columns from place `base` on.
// The factors (term g, columns 8 j + t and 8 j + t + 4) are the 16 x 8
// operand, the grid's real and then its imaginary parts the 8 x 8 one.  The
// TV blocks are independent chains, unrolled together.
template <bool SCALED, int TV, int TM>
__device__ __forceinline__ void degrid_oct_rows(float2 (&T)[TM][2], const float4 (*B)[32],
                                                const float2 (*ring)[8 * (TM + 1) * 8], int base,
                                                int row0, int tu, int g, int t, float up) {
  // not unrolled: with every shape's columns unrolled the code outgrows the
  // instruction cache
#pragma unroll 1
  for (int j = 0; j < tu; ++j) {
    int place = base + j;
    if (place >= TM + 1) place -= TM + 1;
    const float2 *blk = ring[place] + block_at(row0 + g, t);  // block_at(row + 8, c): 64 further
    const int other = block_at(g, t + 4) - block_at(g, t);
    const float4 v = B[j][0];
    const Split f = split<true>(make_float2(v.x, v.y), make_float2(v.z, v.w));
    // (bx + i by) (gr + i gi): the rows (bx, by) times gr, (-by, bx) times gi
    const Rows a = rows(f.re, f.im, negate(f.im), f.re);
    float2 g0[TV], g1[TV];
#pragma unroll
    for (int i = 0; i < TV; ++i) {
      g0[i] = blk[64 * i];
      g1[i] = blk[64 * i + other];
    }
    if constexpr (SCALED) {
#pragma unroll
      for (int i = 0; i < TV; ++i) {
        g0[i] = make_float2(g0[i].x * up, g0[i].y * up);
        g1[i] = make_float2(g1[i].x * up, g1[i].y * up);
      }
    }
    Split grid[TV];
#pragma unroll
    for (int i = 0; i < TV; ++i) grid[i] = split<false>(g0[i], g1[i]);
    float c[TV][4];
    multiply<TV>(c, [&](int) -> const Rows & { return a; },
                 [&](int i) -> const Split & { return grid[i]; });
#pragma unroll
    for (int i = 0; i < TV; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        T[i][h] = add2(T[i][h], make_float2(c[i][2 * h], c[i][2 * h + 1]));
  }
}

// G, kDegridWarps warps per task.  The grid blocks over the current group and
// the TM - 1 to its right are in shared memory, a ring of TM + 1 block columns
// of which one is on its way (cp.async).  Per oct of terms: T = B x grid
// (mma), then y = sum over rows of A x T in FP32, over a lane's rows and a
// butterfly over the 4 lanes of a term.  The factors are copied ahead
// (kOctsAhead octs, each lane its own operands, by cp.async).
constexpr int kOctsAhead = 2;
constexpr int kDegridWarps = 2;  // warps of a task, which share the grid blocks
template <int TM>
struct OctStage {
  float4 A[TM][32], B[TM][32];
  int4 term[32];  // weight, visibility, blocks | rank << 16
};
template <int TM>
struct DegridShared {
  float2 ring[TM + 1][8 * (TM + 1) * 8];
  OctStage<TM> stages[kDegridWarps][kOctsAhead];
};
template <int TM>
__global__ void __launch_bounds__(kDegridWarps * 32, 14 / kDegridWarps) wstrip_degrid_kernel(const WStripArgs a) {
  constexpr int ROWS = 8 * (TM + 1), RING = TM + 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  DegridShared<TM> &shared = *reinterpret_cast<DegridShared<TM> *>(smem_raw);
  dev::pdl_launch_next();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const WStripTask tk = a.tasks[a.order[blockIdx.x]];
  const int32_t *goct = a.group_oct + tk.oct0;
  float2(*ring)[ROWS * 8] = shared.ring;
  OctStage<TM> *stages = shared.stages[warp];
  const float2 *grid = static_cast<const float2 *>(a.grid);
  float2 *out = static_cast<float2 *>(a.vis_out);
  // block column b of the task (columns Q + 8 b ...), rows and columns
  // wrapped; two cells at a time where every row is 16-byte aligned
  const bool wide = a.wide;
  auto load_block = [&](int b, int place) {
    if (wide) {
      const int c = 2 * (threadIdx.x & 3);
      int q = tk.Q + 8 * b + c;
      while (q >= a.Nu) q -= a.Nu;
      int p = tk.P + (threadIdx.x >> 2);
      for (int row = threadIdx.x >> 2; row < ROWS; row += 8 * kDegridWarps, p += 8 * kDegridWarps) {
        while (p >= a.Nv) p -= a.Nv;
        cp_async16(smem_address(&ring[place][block_at(row, c)]), grid + size_t(p) * a.Nu + q);
      }
      return;
    }
    const int c = threadIdx.x & 7;
    int q = tk.Q + 8 * b + c;
    while (q >= a.Nu) q -= a.Nu;
    int p = tk.P + (threadIdx.x >> 3);
    for (int row = threadIdx.x >> 3; row < ROWS; row += 4 * kDegridWarps, p += 4 * kDegridWarps) {
      while (p >= a.Nv) p -= a.Nv;
      cp_async8(&ring[place][block_at(row, c)], grid + size_t(p) * a.Nu + q);
    }
  };
  const int oend = goct[tk.groups];
  // a warp takes every kDegridWarps-th oct; o1: the oct of `raw`, copied next
  int o1 = goct[0] + warp;
  RawTerm raw{};
  if (o1 < oend) raw = load_raw(a, int64_t(o1) * kOctTerms + g);
  // term g's columns 8 j + t and 8 j + t + 4 of B, its rows 8 i + 2 t and
  // 8 i + 2 t + 1 of A
  auto issue = [&](OctStage<TM> &st) {
    if (o1 < oend) {
      const Term next = decode(a, raw);
      const int tv = next.blocks & 15, tu = (next.blocks >> 4) & 15;
      const int jv = 2 * t - next.dv, ju = t - next.du;
      const float2 *pa = next.A + jv, *pb = next.B + ju;
      const int la = next.S - jv, lb = next.S - ju;
      const unsigned sa = smem_address(&st.A[0][lane]), sb = smem_address(&st.B[0][lane]);
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        if (i < tv) {
          cp_async8_zfill(sa + 512 * i, pa + 8 * i, la > 8 * i && (i > 0 || jv >= 0));
          cp_async8_zfill(sa + 512 * i + 8, pa + 8 * i + 1, la > 8 * i + 1 && (i > 0 || jv + 1 >= 0));
        }
        if (i < tu) {
          cp_async8_zfill(sb + 512 * i, pb + 8 * i, lb > 8 * i && (i > 0 || ju >= 0));
          cp_async8_zfill(sb + 512 * i + 8, pb + 8 * i + 4, lb > 8 * i + 4 && (i > 0 || ju + 4 >= 0));
        }
      }
      st.term[lane] = make_int4(__float_as_int(next.w.x), __float_as_int(next.w.y), next.m,
                                next.blocks | (next.rank << 16));
      o1 += kDegridWarps;
      if (o1 < oend) raw = load_raw(a, int64_t(o1) * kOctTerms + g);
    }
    cp_async_commit();
  };
  dev::pdl_wait();  // the grid is the previous kernel's output
  for (int b = 0; b < TM; ++b) load_block(b, b);
#pragma unroll 1
  for (int k = 0; k < kOctsAhead; ++k) issue(stages[k]);  // the window travels with the first
  int base = 0;   // ring place of the current group's first block column
  int place = 0;  // stage of the current oct
  int o = goct[0] + warp, oe = goct[1];
  int before = 1;  // octs that this warp took from the last group
  float up = 1.f;   // scale of the grid's values
  int looked = -1;  // the group in which `top`, the largest of them, was looked up
  unsigned top = 0;
  for (int grp = 0; grp < tk.groups; ++grp) {
    const int oe1 = grp + 1 < tk.groups ? goct[grp + 2] : 0;
    // the block column that this group adds was committed a group ago, before
    // that group's octs issued theirs (if it had any)
    if (before == 0)
      cp_async_wait<0>();
    else
      cp_async_wait<1>();
    // ... is visible, and every warp is done with the one that is replaced
    __syncthreads();
    if (grp + 1 < tk.groups) load_block(grp + TM, base == 0 ? RING - 1 : base - 1);
    cp_async_commit();
    before = 0;
    for (; o < oe; o += kDegridWarps) {
      static_assert(kOctsAhead == 2, "the waits count on two octs ahead");
      cp_async_wait<1>();
      ++before;
      OctStage<TM> &st = stages[place];
      place ^= 1;
      const float4(*B)[32] = reinterpret_cast<const float4(*)[32]>(&st.B[0][lane]);
      const int4 term = st.term[lane];
      const int tv = term.w & 15, tu = (term.w >> 4) & 15, row0 = (term.w >> 8) & 1 ? 8 : 0;
      const float2(*rg)[ROWS * 8] = ring;
      float2 y;
      bool cells = false;  // each term again over its own cells
#pragma unroll 1
      for (;;) {
        float2 T[TM][2];
#pragma unroll
        for (int i = 0; i < TM; ++i) T[i][0] = T[i][1] = make_float2(0.f, 0.f);
        auto product = [&](auto scaled) {
          constexpr bool SCALED = decltype(scaled)::value;
          if constexpr (TM >= 4)
            if (tv == 4) return degrid_oct_rows<SCALED, 4, TM>(T, B, rg, base, row0, tu, g, t, up);
          if constexpr (TM >= 3)
            if (tv == 3) return degrid_oct_rows<SCALED, 3, TM>(T, B, rg, base, row0, tu, g, t, up);
          if constexpr (TM >= 2)
            if (tv == 2) return degrid_oct_rows<SCALED, 2, TM>(T, B, rg, base, row0, tu, g, t, up);
          degrid_oct_rows<SCALED, 1, TM>(T, B, rg, base, row0, tu, g, t, up);
        };
        if (up == 1.f)
          product(std::false_type());
        else
          product(std::true_type());
        y = make_float2(0.f, 0.f);
#pragma unroll
        for (int i = 0; i < TM; ++i) {
          if (i >= tv) break;  // the rest of the stage is an older oct's
          const float4 A = st.A[i][lane];
          y.x = fmaf(A.x, T[i][0].x, fmaf(-A.y, T[i][1].x, y.x));
          y.y = fmaf(A.x, T[i][1].x, fmaf(A.y, T[i][0].x, y.y));
          y.x = fmaf(A.z, T[i][0].y, fmaf(-A.w, T[i][1].y, y.x));
          y.y = fmaf(A.z, T[i][1].y, fmaf(A.w, T[i][0].y, y.y));
        }
#pragma unroll
        for (int s = 1; s <= 2; s <<= 1) {
          y.x += __shfl_xor_sync(0xffffffffu, y.x, s);
          y.y += __shfl_xor_sync(0xffffffffu, y.y, s);
        }
        // Sums of 2^-80 up to 2^120, or 0 beside such sums, had all the bits of
        // their operands' pieces.  Others: see whether the grid's values are
        // scaled as they should be (by a power of two that brings the largest
        // of them to 1, kept for the octs that follow).  10^6 rows on a
        // 1024^2 image, values of 10^-30: 245 us, 215 of order 1; with each such
        // oct's terms summed cell by cell 1,092.
        const unsigned size = max(__float_as_uint(fabsf(y.x)), __float_as_uint(fabsf(y.y)));
        const bool off = size - 0x17800000u >= 0x7b800000u - 0x17800000u && size != 0;
        const bool any_off = __any_sync(0xffffffffu, off);
        if (!any_off && __any_sync(0xffffffffu, size != 0)) break;
        if (looked != grp) {
          looked = grp;
          top = 0;
          for (int j = 0; j < TM; ++j) {
            int place = base + j;
            if (place >= RING) place -= RING;
            for (int k = lane; k < ROWS * 8; k += 32) {
              const float2 v = ring[place][k];
              top = max(top, max(__float_as_uint(fabsf(v.x)), __float_as_uint(fabsf(v.y))));
            }
          }
          top = __reduce_max_sync(0xffffffffu, top);
        }
        if (top == 0) break;
        const float fit = __uint_as_float((254u - min(max(top >> 23, 1u), 253u)) << 23);
        if (top < 0x7f800000u && fit != up) {
          up = fit;
          continue;
        }
        // an infinite or NaN grid value, which zero factors have spread over
        // the oct, or a term whose own cells are far below the largest
        cells = any_off;
        break;
      }
      issue(st);
      // 1 / up
      const float down = __uint_as_float((254u << 23) - __float_as_uint(up));
      y = make_float2(y.x * down, y.y * down);
      if (cells) {
        for (int u = 0; u < kOctTerms; ++u) {
          const Term x = load_term(a, int64_t(o) * kOctTerms + u);
          float2 sum = make_float2(0.f, 0.f);
          for (int k = lane; k < x.S * x.S; k += 32) {
            const int jv = k / x.S, ju = k - jv * x.S, q = x.du + ju;
            int place = base + (q >> 3);
            if (place >= RING) place -= RING;
            const float2 v = ring[place][block_at(row0 + x.dv + jv, q & 7)];
            const float2 av = x.A[jv], bv = x.B[ju];
            const float2 bg = make_float2(bv.x * v.x - bv.y * v.y, bv.x * v.y + bv.y * v.x);
            sum.x += av.x * bg.x - av.y * bg.y;
            sum.y += av.x * bg.y + av.y * bg.x;
          }
          for (int s = 16; s > 0; s >>= 1) {
            sum.x += __shfl_xor_sync(0xffffffffu, sum.x, s);
            sum.y += __shfl_xor_sync(0xffffffffu, sum.y, s);
          }
          if (g == u) y = sum;
        }
      }
      // the terms of a row follow its first one
      const float2 d1 = make_float2(__shfl_down_sync(0xffffffffu, y.x, 4), __shfl_down_sync(0xffffffffu, y.y, 4));
      const float2 d2 = make_float2(__shfl_down_sync(0xffffffffu, y.x, 8), __shfl_down_sync(0xffffffffu, y.y, 8));
      const int rank = term.w >> 16;
      if (rank > 1) y = add2(y, d1);
      if (rank > 2) y = add2(y, d2);
      const float2 w = make_float2(__int_as_float(term.x), __int_as_float(term.y));
      if (t == 0 && rank > 0)
        out[term.z] = make_float2(y.x * w.x - y.y * w.y, y.x * w.y + y.y * w.x);
    }
    base = base + 1 == RING ? 0 : base + 1;
    oe = oe1;
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");
}

// Each grid cell sums the windows that cover it: strips upwards from its own
// (then those that wrap around the last row), in each strip the groups to the
// left of its own (then those that wrap), each task once.  A thread takes 8
// rows of one half strip, which the same windows cover but for the last rows
// of a window, so that one look-up serves eight loads.
constexpr int kFoldRows = 8;
static_assert(kStripRows % kFoldRows == 0, "a thread's rows start in one strip");
__global__ void __launch_bounds__(128) wstrip_fold_kernel(const WStripFoldArgs f) {
  dev::pdl_launch_next();
  dev::pdl_wait();  // the windows are the previous kernel's output
  const int q = int(blockIdx.x) * 32 + int(threadIdx.x);
  const int p = (int(blockIdx.y) * 4 + int(threadIdx.y)) * kFoldRows;
  if (q >= f.Nu || p >= f.Nv) return;
  const float2 *win = static_cast<const float2 *>(f.windows);
  float2 sum[kFoldRows];
#pragma unroll
  for (int k = 0; k < kFoldRows; ++k) sum[k] = make_float2(0.f, 0.f);
  for (int wv = 0; wv < 2; ++wv) {
    const int pp = p + wv * f.Nv;
    // strips that reach the first of the rows; pp >= Nv lies below every strip
    for (int s = min(pp / kStripRows, f.strips - 1); s >= 0 && pp - s * kStripRows < f.rows;
         --s) {
      const int r = pp - s * kStripRows;
      const int k1 = min(kFoldRows, f.rows - r);
      for (int wu = 0; wu < 2; ++wu) {
        const int qq = q + wu * f.Nu;
        int done = -1;  // the last task list summed
        for (int c = min(qq / kStripCols, f.cols - 1);
             c >= 0 && qq - c * kStripCols < kStripCols * f.tiles; --c) {
          const int2 own = __ldg(f.owner + size_t(s) * f.cols + c);
          if (own.x == own.y || own.x == done) continue;
          done = own.x;
          for (int n = own.x; n < own.y; ++n) {
            const int4 t = __ldg(reinterpret_cast<const int4 *>(f.tasks + n));
            const int width = __ldg(&f.tasks[n].width);
            const int64_t base = (int64_t(t.y) << 32) | uint32_t(t.x);
            const float2 *v = win + base + int64_t(r) * width + (qq - t.w);
            if (k1 == kFoldRows) {
              float2 x[kFoldRows];
#pragma unroll
              for (int k = 0; k < kFoldRows; ++k) x[k] = __ldcs(v + k * width);
#pragma unroll
              for (int k = 0; k < kFoldRows; ++k) sum[k] = add2(sum[k], x[k]);
            } else {
#pragma unroll
              for (int k = 0; k < kFoldRows; ++k)
                if (k < k1) sum[k] = add2(sum[k], __ldcs(v + k * width));
            }
          }
        }
      }
    }
  }
  float2 *grid = static_cast<float2 *>(f.grid) + size_t(p) * f.Nu + q;
#pragma unroll
  for (int k = 0; k < kFoldRows; ++k)
    if (p + k < f.Nv) grid[size_t(k) * f.Nu] = sum[k];
}

template <int TM>
cudaError_t launch_strip(bool degrid, const WStripArgs &a, cudaStream_t s) {
  auto fn = degrid ? wstrip_degrid_kernel<TM> : wstrip_grid_kernel<TM>;
  const size_t smem = degrid ? sizeof(DegridShared<TM>) : kStripWarps * sizeof(GridShared<TM>);
  const dim3 blocks(degrid ? a.ntasks : (a.ntasks + kStripWarps - 1) / kStripWarps);
  const dim3 threads(32 * (degrid ? kDegridWarps : kStripWarps));
  if (smem > 48 * 1024) {
    const cudaError_t e =
        cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
    if (e != cudaSuccess) return e;
  }
  return launch_chain_if(a.early, fn, blocks, threads, smem, s, a);
}
cudaError_t launch_tiles(bool degrid, const WStripArgs &a, cudaStream_t s) {
  if (a.ntasks == 0) return cudaSuccess;
  switch (a.tiles) {
    case 1: return launch_strip<1>(degrid, a, s);
    case 2: return launch_strip<2>(degrid, a, s);
    case 3: return launch_strip<3>(degrid, a, s);
    case 4: return launch_strip<4>(degrid, a, s);
  }
  return cudaErrorInvalidValue;
}

}  // namespace

cudaError_t launch_wstrip_degrid(const WStripArgs &a, cudaStream_t s) {
  WStripArgs b = a;
  // a caller's grid need only be aligned as complex<float> is
  b.wide = a.Nu % 2 == 0 && reinterpret_cast<uintptr_t>(a.grid) % 16 == 0;
  return launch_tiles(true, b, s);
}
cudaError_t launch_wstrip_grid(const WStripArgs &a, cudaStream_t s) {
  return launch_tiles(false, a, s);
}
cudaError_t launch_wstrip_fold(const WStripFoldArgs &f, cudaStream_t s) {
  const int rows = 4 * kFoldRows;
  return launch_chain(wstrip_fold_kernel, dim3((f.Nu + 31) / 32, (f.Nv + rows - 1) / rows), dim3(32, 4),
                      0, s, f);
}

}  // namespace pg
