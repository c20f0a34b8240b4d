/*
 * fdtd_flow.cu -- many whole FDTD steps in one persistent launch (sm_103a):
 * the H and E half-steps of fdtd_tma.cu as items of one ordered queue, kept
 * in step by counters in device memory instead of kernel boundaries.
 *
 * Why.  One step as separate kernels (H, E, E's CPML X pass, two TF/SF face
 * passes, the probe gather) pays a launch gap, a ramp and a drained last wave
 * per kernel.  Here an item waits only for the tiles it touches, so nothing
 * drains between half-steps, and everything a cell takes in a half-step (curl,
 * CPML X, Y, Z, TF/SF, current source) runs in its item.
 *
 * Order and waits.  Tickets are taken from a global counter in order: step by
 * step, the H items by z-chunk and tile, then the E items.  Item (half, step,
 * chunk c, tile row ty, tile column) waits for
 *   H of step n: E of step n-1 in the rows (c, ty), (c, ty+1), (c+1, ty), (c+1, ty+1);
 *   E of step n: H of step n   in the rows (c, ty), (c, ty-1), (c-1, ty), (c-1, ty-1),
 * every tile column of a row counted together.  Those rows hold what the item
 * reads, and every reader of what it overwrites.  The fourth holds no cell that
 * the item uses, but H has no cells at j = J-1 and k = K-1: where a row of E
 * items holds just these (J-1 and K-1 multiples of the tile's height and of the
 * item's planes), the fourth is the only one there is, and orders such an item
 * after itself of step n-1 (as a wait of its own it cost 1 % on 64^3 and
 * 131x117x109).  All of these are earlier in the
 * order, so the earliest unfinished item can always run and no ticket waits
 * for a block that is not running.  A row's counter counts finished tiles
 * and is never reset within a launch (`base` steps were counted before
 * it).  Waits are bounded like every wait of the pipelines.
 *
 * Memory order.  A consumer warp's stores are released (gpu scope) by the
 * publishing warp into the row's counter; the producer warp of a later item
 * acquires the counters, fences the async proxy and issues the TMA loads; the
 * "full" mbarrier passes that order on to the group's consumers, whose few
 * direct loads (psi pairs, the H plane below an item) bypass L1.
 *
 * What bounds it.  At 64^3 and below the chain of waits (about 6 us a half-
 * step); above, instruction supply: a loop of straight-line code takes 1.04
 * cycles an instruction and warp up to 24 KB, 1.20 at 32 KB, 2.6 from 48 to 128
 * KB and 6.0 at 192 KB (multiply-adds, a warp a scheduler; with four 4.0 and
 * from 48 KB on 5.4 to 6.3), and the groups of a block are at different places
 * of the kernel.  28 of the 32 instances spill 4 to 40 bytes a thread (8 to 40
 * bytes of stack).  Code size therefore decides more than instruction count:
 * loops specialised by CPML axis, a face pass in batches of cells and psi loads
 * a whole plane ahead each took fewer cycles a plane and were 5-30 % slower as
 * a whole, while one kernel per mode family and coefficient layout (75-82 KB
 * instead of 91) gained 10 % at 256^3 with an oblique wave, and rolled set-up
 * loops, one psi load for three axes and 32-bit cell offsets (75 to 71 KB) 8 %
 * from 96^3 to 192^3.
 *
 * Measured (us a step, separate kernels / this): 64^3 mode 3 27.7/13.2;
 * 131x117x109 mode 5 64.8/52.0; 176x160x129 mode 4 with coefficient arrays
 * 120/76; 256^3 mode 5 281/220; 400x360x120 with a current 314/226;
 * 512x512x448 mode 1 1492/1354.  From 256^3 on that is 80-90 % of the measured
 * copy bandwidth for two passes over the fields a step (74 B a cell and the
 * pairs); running the E items a few chunks behind the H items of the same step,
 * to find their operands in L2, waited longer than it saved (512x512x448: 1452
 * at best against 1400).
 *
 * Results.  Every cell goes through the same per-cell arithmetic in the same
 * order as in the half-step kernels, so the fields, psi pairs and probe
 * record equal theirs (and the reference's).  They do so bit for bit but for the
 * sign of a zero: in the Y and Z slabs the E cells at i = 0 and I-1, which have
 * no pairs, take a correction of 0, and -0 becomes +0 there.  Leaving those cells
 * out cost 3-15 % of a step up to 200^3 (three values kept over the recurrences
 * 160x144x130 61 -> 65.5 us, pairs set to -0 63; 200x185x168 97 -> 111).
 */
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

#include <type_traits>

#include "fdtd_device.cuh"
#include "fdtd_internal.h"
#include "fdtd_pipe.cuh"
#include "fdtd_tile.cuh"

using namespace fdtd;
using namespace fdtd_pipe;
using namespace fdtd_tile;

extern "C" void fdtdk_count_launches(unsigned long long n);

namespace {

// A block fills an SM: NG independent groups of CW consumer warps, each with
// its own ring and producer warp, and one warp that publishes the finished
// items of all of them.  A consumer thread owns four cells in a row of its
// tile: 16-byte shared-memory and field accesses and one 32-byte access per
// psi axis, so that addresses, barriers and path tests are paid once per four
// cells (with one cell per access the kernels issued about 340 instructions a
// cell and step and were bound by that).
constexpr int CW = 4;  // consumer warps of a group: 128 threads x 4 cells = a tile
constexpr int NS = 4;  // ring stages of a group
constexpr int ND = 4;  // items of a group between their first load and their release
// Per-cell H coefficients take more registers: two groups of 168 each a thread
// where the fields fit L2, three of 128 where memory latency is what a step
// waits for (two / three, mode 1: 96^3 23/25 us, 320^3 527/462).
template <bool MU, bool AHEAD>
constexpr int kGroups = MU && !AHEAD ? 2 : 3;
template <int NG>
constexpr int kThreads = (NG * (CW + 1) + 1) * 32;
struct Ctrl {
  uint64_t full[NS], empty[NS];  // ring stages
  uint64_t done[ND], freed[ND];  // items: computed by every warp; released
  uint64_t sync[2];              // the consumer warps, before a face or current pass
  int4 meta[2 * NS];             // see the producer
  uint32_t row[ND];              // the items' row counters (kNoRow: no more items)
};
constexpr int kTabRow = 8;  // floats per row of the shared coefficient table (two aligned loads)
constexpr uint32_t kNoRow = 0xffffffffu;
// A ring stage: three components' tiles, three with the halo (and for E the
// material ids), each family one TMA box.
template <class G>
struct Stage {
  static constexpr int TILES = 3 * G::TILE_B;
  static constexpr int HALOS = (3 * G::HALO_B + 127) / 128 * 128;
  static constexpr int E_HALO = TILES;          // E items: E tiles, H with halo, ids
  static constexpr int E_MAT = E_HALO + HALOS;
  static constexpr int H_TILES = HALOS;         // H items: E with halo, H tiles
  static constexpr int BYTES = E_MAT + G::MAT_B;
  static constexpr int C1 = G::HALO_B / 4;      // floats per component with halo
};
struct FlowMaps {
  CUtensorMap m[FDTD_FLOW_MAPS];  // E, H tiles; E, H with halo; ids
};
template <int NG, class G>
struct FG {
  static constexpr int STAGE = Stage<G>::BYTES;
  static constexpr int RING = NS * STAGE;
  static constexpr int TAB = NG * RING;  // the coefficient table
  static constexpr int CTRL = TAB + kSmemTabMax * kTabRow * 4;
  static constexpr int SMEM = CTRL + NG * (int)sizeof(Ctrl);
  static_assert(STAGE % 128 == 0 && sizeof(Ctrl) % 16 == 0, "alignment");
  static_assert(SMEM + 2048 <= 228 * 1024, "one block per SM");
};

// Division by a launch constant: n / d for 0 <= n < 2^31 as (n * m) >> s with
// s = 31 + ceil(log2 d), m = floor(2^s / d) + 1 (T. Granlund, P. Montgomery,
// PLDI 1994).
struct Div {
  uint32_t d, m, s;
  __device__ __forceinline__ int of(int n) const {
    return (int)(((uint64_t)(uint32_t)n * m) >> s);
  }
};
inline Div make_div(int d) {
  uint32_t l = 0;
  while ((1u << l) < (uint32_t)d) ++l;
  const uint32_t s = 31 + l;
  return Div{(uint32_t)d, (uint32_t)((1ull << s) / (uint32_t)d + 1), s};
}

// One launch.
struct Flow {
  int n_steps, first;       // steps of this launch; the first one's index
  uint32_t base;            // steps already counted by the row counters
  int n_tickets;
  int32_t *work;            // [0] next ticket, [1] finished producers
  uint32_t *cnt;            // row counters
  int32_t *err;             // device error word
  int zc, nch_h, nch_e;     // z-planes per item; chunks of H and of E
  int tx_h, ty_h, tx_e, ty_e;
  int tiles, per_half;      // tickets per chunk and per half-step
  Div by_step, by_tiles, by_tx;
  const int32_t *probe_first;  // [tiles * K + 1] first entry of each tile's planes
  const int2 *probe_at;     // {probe, cell} in that order
  int n_probes;             // probe entries (0: none)
};

__device__ __forceinline__ uint32_t ld_acquire(const uint32_t *p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void red_release(uint32_t *p, uint32_t v) {
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// Has the phase of this parity completed?  (Does not suspend the thread.)
__device__ __forceinline__ bool mbar_test(uint64_t *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ void proxy_fence_all() {
  asm volatile("fence.proxy.async;" ::: "memory");
}

// One poll in line, the rest of a wait out of line: the waits are at many
// places, and code size counts (see above).
__device__ __noinline__ bool wait_more(uint64_t *bar, uint32_t parity) {
  return mbar_wait(bar, parity);
}
__device__ __forceinline__ bool wait_on(uint64_t *bar, uint32_t parity) {
  return mbar_try_wait(bar, parity) || wait_more(bar, parity);
}

// Waits until every lane's counter *p has reached want (p null: nothing to
// wait for); the whole warp calls it.  False when it gave up: after kWaitNs,
// or when another block has reported an error.
__device__ __forceinline__ bool wait_rows(const uint32_t *p, uint32_t want, const int32_t *err) {
  bool done = !p || (int32_t)(ld_acquire(p) - want) >= 0;
  if (__all_sync(0xffffffffu, done)) return true;
  const unsigned long long t0 = global_ns();
#pragma unroll 1
  for (unsigned it = 1;; ++it) {
    if (!done) done = (int32_t)(ld_acquire(p) - want) >= 0;
    if (__all_sync(0xffffffffu, done)) return true;
    if ((it & 255u) == 0u) {
      const bool bad = global_ns() - t0 > kWaitNs || (err && *(const volatile int32_t *)err);
      if (__any_sync(0xffffffffu, bad)) return false;
    }
  }
}

// ------------------------------------------------------------- four cells

// Four cells' values as two packed pairs: the differences and products go two
// per instruction (each rounded as its scalar form).
struct Q4 {
  float2 a, b;
};
__device__ __forceinline__ Q4 q4(float4 v) { return Q4{{v.x, v.y}, {v.z, v.w}}; }
__device__ __forceinline__ Q4 all4(float v) { return Q4{{v, v}, {v, v}}; }
template <int C>
__device__ __forceinline__ float &el(Q4 &q) {
  return C == 0 ? q.a.x : (C == 1 ? q.a.y : (C == 2 ? q.b.x : q.b.y));
}
__device__ __forceinline__ float get(const Q4 &q, int c) {
  return c == 0 ? q.a.x : (c == 1 ? q.a.y : (c == 2 ? q.b.x : q.b.y));
}
__device__ __forceinline__ void set(Q4 &q, int c, float v) {
  if (c == 0) q.a.x = v;
  else if (c == 1) q.a.y = v;
  else if (c == 2) q.b.x = v;
  else q.b.y = v;
}
__device__ __forceinline__ Q4 lds4(const float *p) {
  return q4(*reinterpret_cast<const float4 *>(p));
}
__device__ __forceinline__ void stg4(float *p, const Q4 &q) {
  *reinterpret_cast<float4 *>(p) = make_float4(q.a.x, q.a.y, q.b.x, q.b.y);
}
#define FDTD_PACKED2(name, op)                                                          \
  __device__ __forceinline__ float2 name(float2 x, float2 y) {                          \
    float2 r;                                                                           \
    asm("{\n\t.reg .b64 p, q, r;\n\tmov.b64 p, {%2, %3};\n\tmov.b64 q, {%4, %5};\n\t" op \
        ".rn.f32x2 r, p, q;\n\tmov.b64 {%0, %1}, r;\n\t}"                               \
        : "=f"(r.x), "=f"(r.y)                                                          \
        : "f"(x.x), "f"(x.y), "f"(y.x), "f"(y.y));                                      \
    return r;                                                                           \
  }
FDTD_PACKED2(sub2, "sub")
FDTD_PACKED2(mul2, "mul")
#undef FDTD_PACKED2
__device__ __forceinline__ Q4 sub4(const Q4 &x, const Q4 &y) {
  return Q4{sub2(x.a, y.a), sub2(x.b, y.b)};
}
// Sums and differences with products among their operands: scalar, since the
// compiler contracts a packed product and a packed sum into a fused
// multiply-add whatever their rounding modifiers say (measured: 27 % of the
// sums of random products differ from the separately rounded ones).
__device__ __forceinline__ Q4 add4(const Q4 &x, const Q4 &y) {
  return Q4{{x.a.x + y.a.x, x.a.y + y.a.y}, {x.b.x + y.b.x, x.b.y + y.b.y}};
}
__device__ __forceinline__ Q4 sub4s(const Q4 &x, const Q4 &y) {
  return Q4{{x.a.x - y.a.x, x.a.y - y.a.y}, {x.b.x - y.b.x, x.b.y - y.b.y}};
}
__device__ __forceinline__ Q4 mul4(const Q4 &x, const Q4 &y) {
  return Q4{mul2(x.a, y.a), mul2(x.b, y.b)};
}
// The psi pairs of four cells: one 32-byte access (rows padded to match); not
// kept in L1, where no line of them is read twice.
struct P4 {
  float2 c[4];
};
__device__ __forceinline__ P4 ldp4(const float2 *p) {
  P4 r;
  asm volatile("ld.global.L1::no_allocate.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=f"(r.c[0].x), "=f"(r.c[0].y), "=f"(r.c[1].x), "=f"(r.c[1].y),
                 "=f"(r.c[2].x), "=f"(r.c[2].y), "=f"(r.c[3].x), "=f"(r.c[3].y)
               : "l"(p)
               : "memory");
  return r;
}
// Starts bringing a line to L2.
__device__ __forceinline__ void to_l2(const void *p) {
  asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}
__device__ __forceinline__ void stp4(float2 *p, const P4 &r) {
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p),
               "f"(r.c[0].x), "f"(r.c[0].y), "f"(r.c[1].x), "f"(r.c[1].y), "f"(r.c[2].x),
               "f"(r.c[2].y), "f"(r.c[3].x), "f"(r.c[3].y)
               : "memory");
}

__device__ __noinline__ float2 div_pair(float2 a, float dx) {
  return make_float2(div_ieee(a.x, dx), div_ieee(a.y, dx));
}
// RN(a / dx) of small numerators (|a| < 1, where div_small), y = RN(1/dx): v, the
// quotient of a*2^100, scaled back.  Where that rounds a second time (subnormal quotients)
// the result differs from the right one only if v lies half way between two
// subnormals without being exact; the remainder of v tells the side.  q: the
// quotient of a*2^64, for the others.
__device__ __forceinline__ float quot_small(float a, float q, float dx, float y) {
  const float s = a * 0x1p100f, q0 = s * y;
  const float v = __fmaf_rn(__fmaf_rn(q0, dx, -s), -y, q0);
  const float r = __fmaf_rn(v, dx, -s);  // > 0: v is above the quotient
  const float w = v * 0x1p-100f, t = __fmaf_rn(w, -0x1p100f, v);
  const bool other = fabsf(t) == 0x1p-50f && r != 0.f && (r > 0.f) != (t > 0.f);
  return fabsf(a) < 1.f ? w + (other ? copysignf(0x1p-149f, t) : copysignf(0.f, w)) : q * 0x1p-64f;
}
__device__ __noinline__ float2 quot_pair(float2 a, float2 q, float dx, float y) {
  return make_float2(quot_small(a.x, q.x, dx, y), quot_small(a.y, q.y, dx, y));
}

// All eight quotients of a recurrence in one call.
struct F8 {
  float2 v[4];
};
__device__ __noinline__ F8 quot_all(F8 a, F8 q, float dx, float y, bool divide) {
  if (divide) {
#pragma unroll
    for (int n = 0; n < 4; ++n) a.v[n] = div_pair(a.v[n], dx);
    return a;
  }
#pragma unroll
  for (int n = 0; n < 4; ++n)
    q.v[n] = make_float2(quot_small(a.v[n].x, q.v[n].x, dx, y), quot_small(a.v[n].y, q.v[n].y, dx, y));
  return q;
}

// The recurrences of four cells' pairs, psi = b*psi + c*difference/dx, old
// values in and new ones out.  The quotient is div_by's corrected product,
// taken for every numerator a on a*2^64: exact where lo2 <= |a| < hi*2^-64,
// and the sum undoes the scaling exactly (q*2^-64 is a normal number there).
// So the tiny values ahead of a wave front need no other path; telling them
// apart, as div_by does, cost 60 % of a step while a front was in the CPML
// (176x160x129, 200 steps from rest: 143 us a step, from a filled state 84).
// With the remainder taken as q0*dx - a, zeros come out with their sign too.
// The rest (subnormal quotients, huge numerators, infinities) goes out of line.
// ONE: in one call, which takes 1.5 KB less of the loops and more registers
// across it; the kernels choose by what they measured (kOneCall).
template <bool ONE>
__device__ __forceinline__ P4 recur(const fdtd_dev &d, P4 ps, const Q4 &b, const Q4 &c,
                                    const Q4 &da, const Q4 &db) {
  const float2 dx = {d.dx, d.dx}, ny = {-d.rdx, -d.rdx}, s = {-0x1p64f, -0x1p64f};
  const float2 a[4] = {mul2(c.a, da.a), mul2(c.b, da.b), mul2(c.a, db.a), mul2(c.b, db.b)};
  float2 q[4];
  uint32_t least = ~0u;  // of 2*bits(|a|) - 1: zeros count as large
  float most = 0.f;
#pragma unroll
  for (int n = 0; n < 4; ++n) {
    least = min(least, min(__float_as_uint(a[n].x) * 2u - 1u, __float_as_uint(a[n].y) * 2u - 1u));
    most = fmaxf(most, fmaxf(fabsf(a[n].x), fabsf(a[n].y)));
    const float2 na = mul2(a[n], s), q0 = mul2(na, ny);
    q[n] = __ffma2_rn(__ffma2_rn(q0, dx, na), ny, q0);
  }
  float u = 0x1p-64f;
  if (least < __float_as_uint(d.div_lo2) * 2u - 1u || most >= d.div_hi * 0x1p-64f) {
    u = 1.f;
    const bool divide = most >= d.div_hi * 0x1p-64f || !d.div_small;
    if (ONE) {
      F8 x, z;
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        x.v[n] = a[n];
        z.v[n] = q[n];
      }
      z = quot_all(x, z, d.dx, d.rdx, divide);
#pragma unroll
      for (int n = 0; n < 4; ++n) q[n] = z.v[n];
    } else {
#pragma unroll
      for (int n = 0; n < 4; ++n)
        q[n] = divide ? div_pair(a[n], d.dx) : quot_pair(a[n], q[n], d.dx, d.rdx);
    }
  }
#pragma unroll
  for (int n = 0; n < 4; ++n) {
    const float2 o = mul2(make_float2(get(b, n), get(b, n)), ps.c[n]);
    const float qa = n & 1 ? q[n / 2].y : q[n / 2].x, qb = n & 1 ? q[2 + n / 2].y : q[2 + n / 2].x;
    ps.c[n] = make_float2(__fmaf_rn(qa, u, o.x), __fmaf_rn(qb, u, o.y));
  }
  return ps;
}
// Self-check of the recurrences' quotients over all float bit patterns, eight
// of them at once, or seven beside a subnormal numerator (so that the special
// path takes them): psi = -0 and b = c = 1 leave the bare quotient.
template <bool ONE>
__global__ void k_check_recurrence(const __grid_constant__ fdtd_dev d, int tiny,
                                   unsigned long long *out) {
  unsigned long long bad = 0;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x, per = tiny ? 7 : 8;
  for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t * per < 1ull << 32;
       t += stride) {
    Q4 a, b;
    float v[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      v[e] = __uint_as_float(tiny && e == 7 ? 1u : (uint32_t)(t * per + e));
      set(e < 4 ? a : b, e & 3, v[e]);
    }
    P4 ps;
#pragma unroll
    for (int e = 0; e < 4; ++e) ps.c[e] = make_float2(-0.f, -0.f);
    ps = recur<ONE>(d, ps, all4(1.f), all4(1.f), a, b);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float got = e < 4 ? ps.c[e].x : ps.c[e - 4].y, want = v[e] / d.dx;
      bad += __float_as_uint(got) != __float_as_uint(want) && !(got != got && want != want);
    }
  }
  for (int o = 16; o > 0; o >>= 1) bad += __shfl_xor_sync(0xffffffffu, bad, o);
  if ((threadIdx.x & 31) == 0 && bad) atomicAdd(out, bad);
}

// b, c of the four cells from i at their X slab positions (0 where the slab
// function is negative, and the cell's bit in the result).
template <class S>
__device__ __forceinline__ uint32_t grading_x(const float *tb, const float *tc, int i, S slab,
                                              Q4 &b, Q4 &c) {
  uint32_t out = 0;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int px = slab(i + e);
    set(b, e, px >= 0 ? tb[px] : 0.f);
    set(c, e, px >= 0 ? tc[px] : 0.f);
    out |= (uint32_t)(px < 0) << e;
  }
  return out;
}
// to = from in the cells of the mask.
__device__ __forceinline__ void put_back(Q4 &to, const Q4 &from, uint32_t mask) {
#pragma unroll
  for (int e = 0; e < 4; ++e)
    if (mask >> e & 1) set(to, e, get(from, e));
}

// The H coefficients of four cells from n (a multiple of 4; rows are padded, and
// the ids and arrays there belong to the allocation): ids in one load and three
// per table row, or one load per array (cell by cell it was seven loads each:
// 160x144x130 63 us a step, now 60).
struct H4 {
  Q4 a[3], c[3];  // Chh.., Che..
};
__device__ __forceinline__ H4 hcoef4(const fdtd_dev &d, int n) {
  H4 h;
  if (d.hcoef_mode == 2) {
    const ushort4 id = __ldg(reinterpret_cast<const ushort4 *>(d.hmat + n));
    const int ids[4] = {id.x, id.y, id.z, id.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 *r = reinterpret_cast<const float2 *>(d.hmat_tab + ids[e] * 6);
      const float2 r0 = __ldg(r), r1 = __ldg(r + 1), r2 = __ldg(r + 2);
      set(h.a[0], e, r0.x);
      set(h.a[1], e, r0.y);
      set(h.a[2], e, r1.x);
      set(h.c[0], e, r1.y);
      set(h.c[1], e, r2.x);
      set(h.c[2], e, r2.y);
    }
  } else {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      h.a[a] = q4(__ldg(reinterpret_cast<const float4 *>(d.hc + a * d.cells + n)));
      h.c[a] = q4(__ldg(reinterpret_cast<const float4 *>(d.hc + (3 + a) * d.cells + n)));
    }
  }
  return h;
}

// f +- (C * psi) * dx with the pairs' first (N = 0) or second element.
template <bool PLUS, int N>
__device__ __forceinline__ void corr4(Q4 &f, const Q4 &C, const P4 &ps, float dx) {
  const Q4 v = N == 0 ? Q4{{ps.c[0].x, ps.c[1].x}, {ps.c[2].x, ps.c[3].x}}
                      : Q4{{ps.c[0].y, ps.c[1].y}, {ps.c[2].y, ps.c[3].y}};
  const Q4 t = mul4(mul4(C, v), all4(dx));
  f = PLUS ? add4(f, t) : sub4s(f, t);
}

// Position of the cells i..i+3 (i a multiple of 4, some of them in a slab) in
// a row of X pairs.
__device__ __forceinline__ int psi_x4(int I, int p, int i) {
  return i < p ? i : ((p + 3) & ~3) + i - ((I - p) & ~3);
}

// ------------------------------------------- passes over an item's cells
//
// TF/SF corrections and the current source come after everything else a cell
// takes in a half-step (fdtd_flow_ok), so they are applied to the item's few
// cells concerned once its planes are done, every thread of the group taking
// cells, instead of under a test and a divergent branch in every plane.

struct Box {
  int x0, x1, y0, y1, z0, z1;  // inclusive
};
__device__ __forceinline__ int pick3(int a, int x, int y, int z) {
  return a == 0 ? x : (a == 1 ? y : z);
}
__device__ __forceinline__ bool meets(const Box &t, int x0, int x1, int y0, int y1, int z0,
                                      int z1) {
  return t.x0 <= x1 && t.x1 >= x0 && t.y0 <= y1 && t.y1 >= y0 && t.z0 <= z1 && t.z1 >= z0;
}
// The incident value that corrects component E_ce / H_ch across the face of
// axis ax on one side at the cell (x0, x1, x2): hfam 1: the E wave (component
// ce) on the face plane; 0: the H wave (component ch) half a cell outside.
template <bool OB>
__device__ __forceinline__ float incident(const fdtd_dev &d, int hfam, int mode,
                                          const float *row, int ax, int side, int ce, int ch,
                                          int x0, int x1, int x2) {
  const int lo = pick3(ax, d.i0, d.j0, d.k0), hi = pick3(ax, d.i1, d.j1, d.k1);
  const int at = side ? hi : lo - 1 + hfam;
  const int y0 = ax == 0 ? at : x0, y1 = ax == 1 ? at : x1, y2 = ax == 2 ? at : x2;
  if (!OB) return row[mode < 3 ? y2 : y0];
  const float p0 = (float)y0 + ((hfam ? ce == 0 : ch != 0) ? 0.5f : 0.f);
  const float p1 = (float)y1 + ((hfam ? ce == 1 : ch != 1) ? 0.5f : 0.f);
  const float p2 = (float)y2 + ((hfam ? ce == 2 : ch != 2) ? 0.5f : 0.f);
  const float x = ob_coord(d, p0, p1, p2);
  const float amp = hfam ? (ce == 0 ? d.ob_e[0] : (ce == 1 ? d.ob_e[1] : d.ob_e[2]))
                         : (ch == 0 ? d.ob_h[0] : (ch == 1 ? d.ob_h[1] : d.ob_h[2]));
  return amp * ob_interp(row, hfam ? x : x - 0.5f, d.ob_w);
}

// The corrections that an E element of an oblique wave takes after the one of
// its first face (axis ax, side low or high): the high face of ax when both lie
// on one plane, then the faces of ch (the pair with the other sign).
__device__ __noinline__ float other_faces(const fdtd_dev &d, const float *row, int ax, int ce,
                                          int ch, bool plus, int x0, int x1, int x2, float c,
                                          float val) {
  if (pick3(ax, d.i0, d.j0, d.k0) == pick3(ax, d.i1, d.j1, d.k1)) {
    const float w = c * incident<true>(d, 0, FDTD_MODE_OBLIQUE, row, ax, 1, ce, ch, x0, x1, x2);
    val = plus ? val - w : val + w;
  }
  const int xh = pick3(ch, x0, x1, x2);
#pragma unroll 1
  for (int side = 0; side < 2; ++side) {
    if (xh != (side ? pick3(ch, d.i1, d.j1, d.k1) : pick3(ch, d.i0, d.j0, d.k0))) continue;
    const float w = c * incident<true>(d, 0, FDTD_MODE_OBLIQUE, row, ch, side, ce, ax, x0, x1, x2);
    val = (ce == (ch + 1) % 3) == (side == 0) ? val + w : val - w;
  }
  return val;
}

// One face plane of the pass, q = 0..11 in the order (axis, side, pair p: 0
// E_u with H_v, 1 E_v with H_u; u, v the axes after the axis), and its cells in
// a tile: `only` the planes that a mode corrects on.  The axis modes are the
// cases with one incident E component (y, x, z, y in modes 1-4) and one H
// component (x, y, y, z).
struct Face {
  int ax, side, p, ce, ch, a0, a1, b0, b1, c0, c1;
  bool any;
};
template <bool OB>
__device__ __forceinline__ Face face_of(const fdtd_dev &d, int hfam, int mode, int q,
                                        const Box &t) {
  Face f;
  f.ax = q >> 2;
  f.side = (q >> 1) & 1;
  f.p = q & 1;
  const int u = f.ax == 2 ? 0 : f.ax + 1, v = f.ax == 0 ? 2 : f.ax - 1;
  f.ce = f.p == 0 ? u : v;
  f.ch = f.p == 0 ? v : u;
  const int only = hfam ? (mode == 2 ? 0 : (mode == 3 ? 2 : 1))
                        : (mode == 1 ? 0 : (mode == 4 ? 2 : 1));
  const int lo = pick3(f.ax, d.i0, d.j0, d.k0), hi = pick3(f.ax, d.i1, d.j1, d.k1);
  const int own = f.side ? hi : lo - hfam;
  // [lo, hi-1] along ce, [lo, hi] along ch
  f.a0 = f.ax == 0 ? own : max(t.x0, d.i0);
  f.a1 = f.ax == 0 ? own : min(t.x1, d.i1 - (f.ce == 0));
  f.b0 = f.ax == 1 ? own : max(t.y0, d.j0);
  f.b1 = f.ax == 1 ? own : min(t.y1, d.j1 - (f.ce == 1));
  f.c0 = f.ax == 2 ? own : max(t.z0, d.k0);
  f.c1 = f.ax == 2 ? own : min(t.z1, d.k1 - (f.ce == 2));
  f.any = (OB || (hfam ? f.ce : f.ch) == only) &&
          (hfam || !f.side || lo != hi) &&  // both E faces on one plane: the low one's
          f.a0 >= t.x0 && f.a1 <= t.x1 && f.b0 >= t.y0 && f.b1 <= t.y1 && f.c0 >= t.z0 &&
          f.c1 <= t.z1 && f.a0 <= f.a1 && f.b0 <= f.b1 && f.c0 <= f.c1;
  return f;
}

// The corrections of the item's face cells, plane after plane (mask: those
// with cells in the tile), as ob_plane: an E element on two faces belongs to
// the first plane in the order, which applies both corrections.  The E
// corrections of modes 2 and 4 are negated (src/simulation.h:493-570).  A
// thread's cells follow from its number by shifts (the tile's extents are
// powers of two).
template <bool OB, bool TAB, class G>
__device__ __forceinline__ void face_pass(const fdtd_dev &d, const float *stab, int hfam, int mode,
                                          int step, const Box &t, int tid, uint32_t mask) {
  const float *row = OB ? d.ob_inc[hfam ? 0 : 1] + (int64_t)step * d.ob_w
                        : (hfam ? inc_h_row(d, mode, step) : inc_e_row(d, mode, step));
  const bool flip = !OB && !hfam && (mode == 2 || mode == 4);
#pragma unroll 1
  for (; mask; mask &= mask - 1) {
    const Face f = face_of<OB>(d, hfam, mode, __ffs(mask) - 1, t);
    const bool plus = ((f.p == 0) == (f.side == 0)) != flip;
    const bool flat = OB && !hfam &&
                      pick3(f.ax, d.i0, d.j0, d.k0) == pick3(f.ax, d.i1, d.j1, d.k1);
    const int fast = f.ax == 0 ? G::BY : G::BX, bits = f.ax == 0 ? G::LY : G::LX;
    const int total = f.ax == 2 ? 512 : fast * (t.z1 - t.z0 + 1);
    float *const field = d.f[hfam ? 3 + f.ch : f.ce];
#pragma unroll 1
    for (int r = tid; r < total; r += CW * 32) {
      const int lo = r & (fast - 1), hi = r >> bits;
      const int x0 = f.ax == 0 ? f.a0 : t.x0 + lo;
      const int x1 = f.ax == 0 ? t.y0 + lo : (f.ax == 1 ? f.b0 : t.y0 + hi);
      const int x2 = f.ax == 2 ? f.c0 : t.z0 + hi;
      if (x0 < f.a0 || x0 > f.a1 || x1 < f.b0 || x1 > f.b1 || x2 < f.c0 || x2 > f.c1) continue;
      const int xh = pick3(f.ch, x0, x1, x2);
      const bool h_face = OB && !hfam && (xh == pick3(f.ch, d.i0, d.j0, d.k0) ||
                                          xh == pick3(f.ch, d.i1, d.j1, d.k1));
      if (h_face && f.ch < f.ax) continue;  // a face of ch owns it
      const int64_t n = x0 + (int64_t)x1 * d.Ip + (int64_t)x2 * d.plane;
      float *at = field + n;
      float val = __ldcg(at);
      float c;
      if (hfam) c = hche_at(d, n, f.ch);
      else if (TAB) c = stab[(int)__ldg(d.mat + n) * kTabRow + 3 + f.ce];
      else if (d.coef_mode == 0) c = __ldg(d.ce[3 + f.ce] + n);
      else c = __ldg(d.mat_tab + (int)__ldg(d.mat + n) * 6 + 3 + f.ce);
      const float w =
          c * incident<OB>(d, hfam, mode, row, f.ax, f.side, f.ce, f.ch, x0, x1, x2);
      val = plus ? val + w : val - w;
      if (h_face || flat) val = other_faces(d, row, f.ax, f.ce, f.ch, plus, x0, x1, x2, c, val);
      *at = val;
    }
  }
}

// The corrections of modes 1-4 on a thread's four cells of a plane, within the
// planes' loop: f the components of H (or E) and C their Che (or Cexh..).  A
// half-step corrects the two components that are not `only`, each on the faces
// of the remaining axis.  For grids whose steps are a chain of waits this saves
// the item's second visit to its cells (us a step, afterwards / here: 48^3
// 14.4/12.2, 64^3 15.0/13.4); otherwise the code costs more than the visit (96^3
// 21/28).
template <bool H>
__device__ __forceinline__ void axis_faces(const fdtd_dev &d, int mode, const float *row, int i,
                                           int j, int k, Q4 *const f[3], const Q4 *const C[3]) {
  const int only = H ? (mode == 2 ? 0 : (mode == 3 ? 2 : 1)) : (mode == 1 ? 0 : (mode == 4 ? 2 : 1));
  const bool flip = !H && (mode == 2 || mode == 4);
#pragma unroll
  for (int t = 0; t < 3; ++t) {
    if (t == only) continue;
    const int ax = 3 - t - only, ce = H ? only : t;
    const bool first = ce == (ax == 2 ? 0 : ax + 1);  // the pair (E_u, H_v)
    const int lo = pick3(ax, d.i0, d.j0, d.k0), hi = pick3(ax, d.i1, d.j1, d.k1);
#pragma unroll 1
    for (int side = 0; side < 2; ++side) {
      const int own = side ? hi : lo - H;
      const int a0 = ax == 0 ? own : d.i0, a1 = ax == 0 ? own : d.i1 - (ce == 0);
      const int b0 = ax == 1 ? own : d.j0, b1 = ax == 1 ? own : d.j1 - (ce == 1);
      const int c0 = ax == 2 ? own : d.k0, c1 = ax == 2 ? own : d.k1 - (ce == 2);
      if (j < b0 || j > b1 || k < c0 || k > c1 || i + 3 < a0 || i > a1) continue;
      const int at = side ? hi : lo - 1 + H;
      const bool plus = (first == (side == 0)) != flip;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        if (i + e < a0 || i + e > a1) continue;
        const float v = row[mode < 3 ? (ax == 2 ? at : k) : (ax == 0 ? at : i + e)];
        const float w = get(*C[t], e) * v;
        set(*f[t], e, plus ? get(*f[t], e) + w : get(*f[t], e) - w);
      }
    }
  }
}

// The same for mode 5: component t is corrected on the faces of the other two
// axes in their order, which is the order of ob_plane's owner (us a step,
// afterwards / here: 24^3 37/19, 48^3 25/19, 64^3 26/20; 96^3 at two planes an
// item 35/39).  The cells go one by one, which keeps the code small.
template <bool H>
__device__ __forceinline__ void oblique_faces(const fdtd_dev &d, const float *row, int i, int j,
                                              int k, Q4 *const f[3], const Q4 *const C[3]) {
#pragma unroll
  for (int t = 0; t < 3; ++t) {
#pragma unroll 1
    for (int face = 0; face < 4; ++face) {
      const int side = face & 1, ax = face < 2 ? (t == 0 ? 1 : 0) : (t == 2 ? 1 : 2);
      const int ce = H ? 3 - ax - t : t, ch = H ? t : 3 - ax - t;
      const bool first = ce == (ax == 2 ? 0 : ax + 1);  // the pair (E_u, H_v)
      const int lo = pick3(ax, d.i0, d.j0, d.k0), hi = pick3(ax, d.i1, d.j1, d.k1);
      const int own = side ? hi : lo - H;
      const int a0 = ax == 0 ? own : d.i0, a1 = ax == 0 ? own : d.i1 - (ce == 0);
      const int b0 = ax == 1 ? own : d.j0, b1 = ax == 1 ? own : d.j1 - (ce == 1);
      const int c0 = ax == 2 ? own : d.k0, c1 = ax == 2 ? own : d.k1 - (ce == 2);
      if (j < b0 || j > b1 || k < c0 || k > c1) continue;
      const bool plus = first == (side == 0);
#pragma unroll 1
      for (int e = max(a0 - i, 0); e <= min(a1 - i, 3); ++e) {
        const float w = get(*C[t], e) * incident<true>(d, H, FDTD_MODE_OBLIQUE, row, ax, side, ce,
                                                       ch, i + e, j, k);
        const float v = get(*f[t], e);
        set(*f[t], e, plus ? v + w : v - w);
      }
    }
  }
}

// The current source on the item's cells in the box (gpu.h:55-82).
__device__ __noinline__ void current_pass(const fdtd_dev &d, const fdtd_op &op, int step, Box t,
                                          int tid) {
  const int *b = op.cur_box;
  const int x0 = max(t.x0, b[0]), x1 = min(t.x1, b[1]), y0 = max(t.y0, b[2]);
  const int y1 = min(t.y1, b[3]), z0 = max(t.z0, b[4]), z1 = min(t.z1, b[5]);
  const int na = x1 - x0 + 1, nb = y1 - y0 + 1, total = na * nb * (z1 - z0 + 1);
  const int cm = op.cur_mode;
  const float src = d.src[step], dx = d.dx;
#pragma unroll 1
  for (int r = tid; r < total; r += CW * 32) {
    const int rb = r / na;
    const int64_t n = x0 + r - rb * na + (int64_t)(y0 + rb % nb) * d.Ip +
                      (int64_t)(z0 + rb / nb) * d.plane;
    const float c = d.coef_mode == 0
                        ? __ldg(d.ce[2 + cm] + n)
                        : __ldg(d.mat_tab + (int64_t)__ldg(d.mat + n) * 6 + 2 + cm);
    float *f = d.f[cm - 1] + n;
    *f = __ldcg(f) - c * src * dx / dx / dx;
  }
}

// The publishing warp: lane g takes group g's items in order.  When every
// consumer warp has computed one (its stores are ordered before its arrival),
// the item's row counter is raised with gpu-scope release, so that the
// consumers never wait for their stores to land.  Gives up without progress
// for twice the waits' limit, or when a block has reported an error.
// Polling without a pause between costs the others nothing measurable and gains
// 1-2 % up to 200^3 (131x117x109 52.9 -> 52.0 us a step, 128^3 36.7 -> 35.8).
template <int NG>
__device__ __forceinline__ void release_items(Ctrl *ctrl, uint32_t *cnt, const int32_t *err,
                                              int lane) {
  bool live = lane < NG;
  Ctrl &c = ctrl[live ? lane : 0];
  int item = 0;
  unsigned long long t0 = global_ns();
#pragma unroll 1
  for (unsigned it = 1; __any_sync(0xffffffffu, live); ++it) {
    const int slot = item % ND;
    const bool ready = live && mbar_test(&c.done[slot], (uint32_t)((item / ND) & 1));
    if (__any_sync(0xffffffffu, ready)) {
      if (ready) {
        const uint32_t row = c.row[slot];
        if (row == kNoRow) {
          live = false;
        } else {
          red_release(cnt + row, 1);
          mbar_arrive(&c.freed[slot]);
          ++item;
        }
      }
      t0 = global_ns();
    }
    if ((it & 1023u) == 0u) {
      const bool bad = global_ns() - t0 > 2 * kWaitNs || (err && *(const volatile int32_t *)err);
      if (__any_sync(0xffffffffu, bad)) return;
    }
    __syncwarp();
  }
}

// What a ticket stands for: an item of half-step `e` of step n of the launch.
struct Item {
  bool valid, e;
  int n, x0, y0, kb, np;
  int c, ty;  // z-chunk and tile row
};

template <class G>
__device__ __forceinline__ Item decode(const Flow &f, int K, int w) {
  Item it;
  it.n = f.by_step.of(w);
  int t = w - it.n * 2 * f.per_half;
  it.e = t >= f.per_half;
  if (it.e) t -= f.per_half;
  it.c = f.by_tiles.of(t);
  const int tile = t - it.c * f.tiles;
  it.ty = f.by_tx.of(tile);
  const int tx = tile - it.ty * f.tx_e;
  it.valid = it.e || (it.c < f.nch_h && it.ty < f.ty_h && tx < f.tx_h);
  it.x0 = tx * G::BX;
  it.y0 = it.ty * G::BY;
  it.kb = it.c * f.zc;
  it.np = min(f.zc, (it.e ? K : K - 1) - it.kb);
  return it;
}

// The probes in an H item's cells (a list per tile and plane, `first` at the
// item's): E and H at the start of the step (nothing of it has been overwritten
// yet), by the producer warp.  With one list per plane, which every tile's item
// looked through, a dense plane of probes cost more than the separate gather (us
// a step, separate kernels / so / with a list per tile: 64^3 and 2304 probes in a
// plane 35/49/19, 128^3 and 8100 85/108/37, 200^3 and 10000 207/216/108).
__device__ __noinline__ void gather_probes(const fdtd_dev &d, const int32_t *first,
                                           const int2 *pat, int row, int np, int lane) {
  const int a = first[0], b = first[np];
  if (row >= d.T) return;
#pragma unroll 1
  for (int t = a + lane; t < b; t += 32) {
    const int2 e = pat[t];
    float *o = d.probes + ((int64_t)row * d.num_ant + e.x) * 6;
    float v[6];
#pragma unroll
    for (int c = 0; c < 6; ++c) v[c] = __ldcg(d.f[c] + e.y);
#pragma unroll
    for (int c = 0; c < 6; ++c) o[c] = v[c];
  }
}

// A pair at a time / one call (us a step): mode 1 160^3 61.4/58.7, 192^3
// 92.9/90.9; coefficient arrays 192^3 133/121, 320^3 530/503, but 128^3 45.3/47.1;
// mode 5 128^3 49.6/47.2, but 256^3 226/233.
template <bool OB, bool TAB, bool AHEAD>
constexpr bool kOneCall = OB ? !AHEAD : (TAB || AHEAD);

// MU: per-cell H coefficients (fdtd_set_magnetic).
// OB: mode 5.  TAB: material ids with a table that fits shared memory.  One
// kernel each, since what a step does not need would cost it instruction cache.
// SIZE: big, the pairs of the next plane are brought to L2 a plane ahead, for
// grids that do not stay there (fdtd_flow::ahead); small, axis_faces and
// oblique_faces.
constexpr int kSmall = 0, kMid = 1, kBig = 2;
template <int NG, bool MU, bool OB, bool TAB, int SIZE, class G>
__global__ void __launch_bounds__(kThreads<NG>, 1)
    k_flow(const __grid_constant__ fdtd_dev d, const __grid_constant__ fdtd_op op,
           const __grid_constant__ FlowMaps mp, const __grid_constant__ Flow f) {
  extern __shared__ __align__(128) unsigned char smem_all[];
  using L = FG<NG, G>;
  using S = Stage<G>;
  constexpr int ST = L::STAGE;
  constexpr bool AHEAD = SIZE == kBig, IN_PLANE = SIZE == kSmall;
  constexpr bool kOne = kOneCall<OB, TAB, AHEAD>;
  float *stab = reinterpret_cast<float *>(smem_all + L::TAB);
  Ctrl *ctrl = reinterpret_cast<Ctrl *>(smem_all + L::CTRL);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // the CPML grading, indexed per lane: a shared-memory copy (the
  // by-value descriptor's would be divergent constant-bank loads)
  __shared__ float s_bc[4][2 * FDTD_MAX_PML];  // bH cH bE cE
#pragma unroll 1
  for (int t = threadIdx.x; t < 2 * FDTD_MAX_PML; t += kThreads<NG>) {
    s_bc[0][t] = d.bH[t];
    s_bc[1][t] = d.cH[t];
    s_bc[2][t] = d.bE[t];
    s_bc[3][t] = d.cE[t];
  }
  if (threadIdx.x < NG) {
    Ctrl &c = ctrl[threadIdx.x];
#pragma unroll 1
    for (int s = 0; s < NS; ++s) {
      mbar_init(&c.full[s], 1);
      mbar_init(&c.empty[s], CW);
    }
#pragma unroll 1
    for (int s = 0; s < ND; ++s) {
      mbar_init(&c.done[s], CW);
      mbar_init(&c.freed[s], 1);
    }
    mbar_init(&c.sync[0], CW);
    mbar_init_fence();
  }
  if (TAB)
#pragma unroll 1
    for (int t = threadIdx.x; t < d.n_mat * 6; t += kThreads<NG>)
      stab[t / 6 * kTabRow + t % 6] = __ldg(d.mat_tab + t);
  __syncthreads();

  if (warp == NG * (CW + 1)) {
    release_items<NG>(ctrl, f.cnt, f.err, lane);
    return;
  }
  const int grp = warp < NG * CW ? warp / CW : warp - NG * CW;
  Ctrl &cg = ctrl[grp];
  uint64_t *full = cg.full, *empty = cg.empty;
  int4 *meta = cg.meta;
  unsigned char *smem = smem_all + grp * L::RING;

  if (warp >= NG * CW) {  // ----------------------------------- producer
    const int row0 = f.n_probes ? *d.probe_row : 0;
    int q = 0, item = 0;
    bool ok = true;
    int w = lane == 0 ? atomicAdd(&f.work[0], 1) : 0;
    w = __shfl_sync(0xffffffffu, w, 0);
#pragma unroll 1
    while (w < f.n_tickets) {
      // the next ticket's round trip runs under this item's work
      int wn = lane == 0 ? atomicAdd(&f.work[0], 1) : 0;
      const Item it = decode<G>(f, d.K, w);
      if (it.valid) {
        const uint32_t cnt_e = (uint32_t)f.nch_h * f.ty_h;  // E's counters follow H's
        // the rows this item waits for, one per lane
        const uint32_t *p = nullptr;
        uint32_t want;
        if (it.e) {
          want = (uint32_t)f.tx_h * (f.base + it.n + 1);
          const int c = it.c - (lane >> 1), y = it.ty - (lane & 1);
          if (lane < 4 && c >= 0 && y >= 0 && c < f.nch_h && y < f.ty_h)
            p = f.cnt + c * f.ty_h + y;
        } else {
          want = (uint32_t)f.tx_e * (f.base + it.n);
          const int c = it.c + (lane >> 1), y = it.ty + (lane & 1);
          if (lane < 4 && it.n > 0 && c < f.nch_e && y < f.ty_e)
            p = f.cnt + cnt_e + c * f.ty_e + y;
        }
        if (!(ok = wait_rows(p, want, f.err))) break;
        // what lanes 0 to 3 have acquired holds for the warp (a vote alone is
        // not documented to order memory)
        __syncwarp();
        if (!it.e && f.n_probes) {
          gather_probes(d, f.probe_first + (it.ty * f.tx_e + it.x0 / G::BX) * d.K + it.kb,
                        f.probe_at, row0 + it.n, it.np, lane);
          __syncwarp();
        }
        if (lane == 0) {
          proxy_fence_all();
          const CUtensorMap *mm = mp.m;
          const bool um = TAB || d.coef_mode == 1;
          const int step = f.first + it.n;
          // E: the item's planes upwards; H: the plane above the item (its Ex
          // and Ey), then the item's planes downwards
          const int loads = it.e ? it.np : it.np + 1;
          const int slot = item % ND;
          if (item >= ND) ok = wait_on(&cg.freed[slot], (uint32_t)(((item / ND) - 1) & 1));
          if (ok) cg.row[slot] = it.e ? cnt_e + it.c * f.ty_e + it.ty : it.c * f.ty_h + it.ty;
#pragma unroll 1
          for (int t = 0; t < loads && ok; ++t, ++q) {
            const int s = q % NS;
            if (q >= NS) ok = wait_on(&empty[s], (uint32_t)(((q / NS) - 1) & 1));
            if (!ok) break;
            // for the item's first stage: {half, item slot, planes, first plane},
            // {-, x0, y0, step}
            if (t == 0) {
              meta[2 * s] = make_int4(it.e ? 1 : 0, slot, it.np, it.kb);
              meta[2 * s + 1] = make_int4(0, it.x0, it.y0, step);
            }
            unsigned char *st = smem + s * ST;
            // one arrive per phase: the stage's whole byte count at once
            const bool above = !it.e && t == 0;
            const uint32_t bytes = it.e ? 3 * G::TILE_B + 3 * G::HALO_B + (um ? G::MAT_B : 0)
                                  : (above ? 3 * G::HALO_B : 3 * G::HALO_B + 3 * G::TILE_B);
            mbar_expect_tx(&full[s], bytes);
            if (it.e) {
              const int k = it.kb + t;
              tma_load_4d(st, &mm[0], &full[s], it.x0, it.y0, k, 0);
              tma_load_4d(st + S::E_HALO, &mm[3], &full[s], it.x0 - 4, it.y0 - 1, k, 0);
              if (um) tma_load_3d(st + S::E_MAT, &mm[4], &full[s], it.x0, it.y0, k);
            } else {
              const int k = it.kb + it.np - t;
              tma_load_4d(st, &mm[2], &full[s], it.x0, it.y0, k, 0);
              if (!above) tma_load_4d(st + S::H_TILES, &mm[1], &full[s], it.x0, it.y0, k, 0);
            }
          }
        }
        ++item;
        ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
        if (!ok) break;
      }
      w = __shfl_sync(0xffffffffu, wn, 0);
    }
    if (lane == 0) {
      // the last producer rewinds the queue and advances the probe row
      __threadfence();
      if (atomicAdd(&f.work[1], 1) == (int)gridDim.x * NG - 1) {
        atomicExch(&f.work[0], 0);
        atomicExch(&f.work[1], 0);
        if (f.n_probes) *d.probe_row = row0 + f.n_steps;
      }
      if (ok) {  // sentinel: no more work
        const int s = q % NS, slot = item % ND;
        if (item >= ND) ok = wait_on(&cg.freed[slot], (uint32_t)(((item / ND) - 1) & 1));
        if (ok && q >= NS) ok = wait_on(&empty[s], (uint32_t)(((q / NS) - 1) & 1));
        if (ok) {
          cg.row[slot] = kNoRow;
          meta[2 * s] = make_int4(-1, slot, 0, 0);
          mbar_arrive(&full[s]);
          ++q;
        }
      }
      if (!ok && f.err) atomicExch(f.err, 3);
      // drain: every copy issued by this block has landed before it retires
#pragma unroll 1
      for (int r = (q > NS ? q - NS : 0); r < q; ++r)
        wait_on(&full[r % NS], (uint32_t)((r / NS) & 1));
    }
    return;
  }

  // ------------------------------------------------------------ consumers
  const int tid = (int)threadIdx.x - grp * CW * 32;
  const int xo = 4 * (tid % (G::BX / 4)), ry = tid / (G::BX / 4);
  int q = 0;
  uint32_t syncs = 0;
  // every warp of the group has stored its cells (bounded, as the other waits)
  const auto group_sync = [&]() {
    __syncwarp();
    if (lane == 0) mbar_arrive(&cg.sync[0]);
    return wait_on(&cg.sync[0], syncs++ & 1u);
  };
#pragma unroll 1
  for (;;) {
    int s = q % NS;
    if (!wait_on(&full[s], (uint32_t)((q / NS) & 1))) {
      if (f.err) atomicExch(f.err, 2);
      return;
    }
    const int4 m = meta[2 * s], m1 = meta[2 * s + 1];
    if (m.x < 0) {  // sentinel
      if (lane == 0) mbar_arrive(&cg.done[m.y]);
      return;
    }
    const int np = m.z, kb = m.w, step = m1.w;
    const int i = m1.y + xo, j = m1.z + ry;
    const int I = d.I, J = d.J, K = d.K, p = d.p;
    const float dx = d.dx;
    const float *tb = s_bc[m.x ? 2 : 0];
    const float *tc = s_bc[m.x ? 3 : 1];
    // the thread's psi pairs, as 32-bit offsets (fdtd_flow_ok): Y and X of its
    // first plane with their plane strides, Z of slab position 0
    const int oz = i + j * d.Ip, plane = (int)d.plane;
    const int sY = 2 * p * d.Ip, sX = fdtd_psi_x_pitch(I, p) * J;
    // does the item reach the TF/SF faces (of either kind)?
    const bool faces =
        IN_PLANE && op.tfsf_mode && m1.y <= d.i1 && m1.y + G::BX >= d.i0 && m1.z <= d.j1 &&
        m1.z + G::BY >= d.j0 && kb <= d.k1 && kb + np >= d.k0 &&
        !(m1.y > d.i0 && m1.y + G::BX <= d.i1 && m1.z > d.j0 && m1.z + G::BY <= d.j1 &&
          kb > d.k0 && kb + np <= d.k1);
    bool good;
    if (m.x == 0) {
      // ------------------------------------------------------------ H item
      const Q4 Chh = all4(d.Chh), Che = all4(d.Che);
      const int nv = j < J - 1 ? min(I - 1 - i, 4) : 0;  // H cells of this thread
      const int py = nv > 0 ? slab_h(j, J, p) : -1;
      const bool sy = py >= 0, sx = nv > 0 && (i < p || i + 3 >= I - p);
      const int k1 = kb + np - 1;
      int oy = i + (py + k1 * 2 * p) * d.Ip;
      int ox = psi_x4(I, p, i) + (j + k1 * J) * fdtd_psi_x_pitch(I, p);
      int n = oz + k1 * plane;
      Q4 ex1, ey1;
      {
        const float *sE = reinterpret_cast<const float *>(smem + s * ST) + ry * G::HW + xo;
        ex1 = lds4(sE);
        ey1 = lds4(sE + S::C1);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[s]);
      ++q;
      // The psi pairs of a plane's first CPML axis are loaded while the plane
      // before it finishes and its own tiles are waited for.
      P4 ps;
      const auto first_pairs = [&](int k) {
        const int pz = slab_h(k, K, p);
        const float2 *at = sy ? psi_pairs(d, PSI_HY) + oy : psi_pairs(d, PSI_HX) + ox;
        if (!sy && !sx) at = psi_pairs(d, PSI_HZ) + (oz + pz * plane);
        if (sy || sx || (nv > 0 && pz >= 0)) ps = ldp4(at);
      };
      // The next plane's pairs are on their way to L2 meanwhile.
      const auto ahead = [&](int k, int y, int x) {
        const int pz = slab_h(k, K, p);
        if (sy) to_l2(psi_pairs(d, PSI_HY) + y);
        if (sx) to_l2(psi_pairs(d, PSI_HX) + x);
        if (nv > 0 && pz >= 0) to_l2(psi_pairs(d, PSI_HZ) + (oz + pz * plane));
      };
      // An item with nothing but the curl for this warp (all its cells H cells
      // outside the CPML) has a loop of its own: about 110 instructions a plane
      // against 300 and a call, and no path test.
      const auto planes = [&](auto curl_only) {
        constexpr bool kCurl = decltype(curl_only)::value;
        if constexpr (!kCurl) first_pairs(k1);
#pragma unroll 1
        for (int k = k1; k >= kb; --k, ++q) {
          s = q % NS;
          if (!wait_on(&full[s], (uint32_t)((q / NS) & 1))) {
            return false;
          }
          const float *sE = reinterpret_cast<const float *>(smem + s * ST) + ry * G::HW + xo;
          const float *sH =
              reinterpret_cast<const float *>(smem + s * ST + S::H_TILES) + ry * G::BX + xo;
          constexpr int C1 = S::C1;
          const Q4 ex = lds4(sE), ey = lds4(sE + C1), ez = lds4(sE + 2 * C1);
          const float ey_r = sE[C1 + 4], ez_r = sE[2 * C1 + 4];
          Q4 dEz_y = sub4(lds4(sE + 2 * C1 + G::HW), ez), dEx_y = sub4(lds4(sE + G::HW), ex);
          Q4 dEz_x = {{ez.a.y - ez.a.x, ez.b.x - ez.a.y}, {ez.b.y - ez.b.x, ez_r - ez.b.y}};
          Q4 dEy_x = {{ey.a.y - ey.a.x, ey.b.x - ey.a.y}, {ey.b.y - ey.b.x, ey_r - ey.b.y}};
          Q4 dEy_z = sub4(ey1, ey), dEx_z = sub4(ex1, ex);
          ex1 = ex;
          ey1 = ey;
          Q4 hx = lds4(sH), hy = lds4(sH + 512), hz = lds4(sH + 1024);
          Q4 Cx = Che, Cy = Che, Cz = Che;
          if (MU) {
            const H4 hc = hcoef4(d, kCurl || nv > 0 ? n : 0);
            const Q4 Ax = hc.a[0], Ay = hc.a[1], Az = hc.a[2];
            Cx = hc.c[0];
            Cy = hc.c[1];
            Cz = hc.c[2];
            hx = mul4(Ax, hx);
            hy = mul4(Ay, hy);
            hz = mul4(Az, hz);
          } else {
            hx = mul4(Chh, hx);
            hy = mul4(Chh, hy);
            hz = mul4(Chh, hz);
          }
          hx = add4(hx, mul4(Cx, sub4(dEy_z, dEz_y)));
          hy = add4(hy, mul4(Cy, sub4(dEz_x, dEx_z)));
          hz = add4(hz, mul4(Cz, sub4(dEx_y, dEy_x)));
          if constexpr (!kCurl) {
            // CPML Y, X, Z (gpu.h:644-685, :604-642, :687-725)
            const int pz = slab_h(k, K, p);
            const bool sz = nv > 0 && pz >= 0;
            if (AHEAD && k > kb) ahead(k - 1, oy - sY, ox - sX);
            if (nv < 4) {  // cells past the last H cell: no recurrence
              const Q4 none = all4(0.f);
              const uint32_t past = 0xfu << max(nv, 0);
              put_back(dEz_y, none, past);
              put_back(dEx_y, none, past);
              put_back(dEz_x, none, past);
              put_back(dEy_x, none, past);
              put_back(dEy_z, none, past);
              put_back(dEx_z, none, past);
            }
            if (sy) {
              ps = recur<kOne>(d, ps, all4(tb[py]), all4(tc[py]), dEz_y, dEx_y);
              corr4<false, 0>(hx, Cx, ps, dx);
              corr4<true, 1>(hz, Cz, ps, dx);
              stp4(psi_pairs(d, PSI_HY) + oy, ps);
            }
            if (sx) {
              if (sy) ps = ldp4(psi_pairs(d, PSI_HX) + ox);
              Q4 b, c;
              const Q4 hy0 = hy, hz0 = hz;
              const uint32_t out =
                  grading_x(tb, tc, i, [&](int v) { return slab_h(v, I, p); }, b, c);
              ps = recur<kOne>(d, ps, b, c, dEz_x, dEy_x);
              corr4<true, 0>(hy, Cy, ps, dx);
              corr4<false, 1>(hz, Cz, ps, dx);
              put_back(hy, hy0, out);
              put_back(hz, hz0, out);
              stp4(psi_pairs(d, PSI_HX) + ox, ps);
            }
            if (sz) {
              float2 *Z = psi_pairs(d, PSI_HZ) + (oz + pz * plane);
              if (sy || sx) ps = ldp4(Z);
              ps = recur<kOne>(d, ps, all4(tb[pz]), all4(tc[pz]), dEy_z, dEx_z);
              corr4<true, 0>(hx, Cx, ps, dx);
              corr4<false, 1>(hy, Cy, ps, dx);
              stp4(Z, ps);
            }
            if (nv < 4) {  // the cells past it keep their value
              const uint32_t past = 0xfu << max(nv, 0);
              put_back(hx, lds4(sH), past);
              put_back(hy, lds4(sH + 512), past);
              put_back(hz, lds4(sH + 1024), past);
            }
          }
          if constexpr (IN_PLANE && !kCurl) {
            if (faces && nv > 0) {
              Q4 *const ff[3] = {&hx, &hy, &hz};
              const Q4 *const cc[3] = {&Cx, &Cy, &Cz};
              if constexpr (OB)
                oblique_faces<true>(d, d.ob_inc[0] + (int64_t)step * d.ob_w, i, j, k, ff, cc);
              else
                axis_faces<true>(d, op.tfsf_mode, inc_h_row(d, op.tfsf_mode, step), i, j, k, ff, cc);
            }
          }
          if (kCurl || nv > 0) {
            stg4(d.f[3] + n, hx);
            stg4(d.f[4] + n, hy);
            stg4(d.f[5] + n, hz);
          }
          n -= plane;
          if constexpr (!kCurl) {
            oy -= sY;
            ox -= sX;
            if (k > kb) first_pairs(k - 1);
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(&empty[s]);
        }
        return true;
      };
      good = __all_sync(0xffffffffu, nv == 4 && !sy && !sx) && !faces && kb >= p && k1 < K - p
                 ? planes(std::true_type{})
                 : planes(std::false_type{});
    } else {
      // ------------------------------------------------------------ E item
      const int nv = j < J ? min(I - i, 4) : 0;
      // slabs exclude the first and last planes of the other axes
      // (gpu.h:776-777, :800-801, :839-840)
      const bool j_in = j >= 1 && j <= J - 2;
      const int py = nv > 0 ? slab_e(j, J, p) : -1;
      const bool sx_ = nv > 0 && j_in && (i < p || i + 3 >= I - p);
      const bool use_mat = TAB || d.coef_mode == 1;
      int oy = i + (py + kb * 2 * p) * d.Ip;
      int ox = psi_x4(I, p, i) + (j + kb * J) * fdtd_psi_x_pitch(I, p);
      int n = oz + kb * plane;
      Q4 hx_km = all4(0.f), hy_km = hx_km;
      if (kb > 0 && nv > 0) {
        hx_km = q4(__ldcg(reinterpret_cast<const float4 *>(d.f[3] + (n - plane))));
        hy_km = q4(__ldcg(reinterpret_cast<const float4 *>(d.f[4] + (n - plane))));
      }
      // The first axis's pairs and the loop for the curl alone, as for H.
      P4 ps;
      const auto first_pairs = [&](int k) {
        const int pz = slab_e(k, K, p);
        const bool k_in = k >= 1 && k <= K - 2;
        const bool y = py >= 0 && k_in, z = nv > 0 && j_in && pz >= 0, x = sx_ && k_in;
        const float2 *at = y ? psi_pairs(d, PSI_EY) + oy : psi_pairs(d, PSI_EX) + ox;
        if (!y && z) at = psi_pairs(d, PSI_EZ) + (oz + pz * plane);
        if (y || z || x) ps = ldp4(at);
      };
      const auto ahead = [&](int k, int y, int x) {
        const int pz = slab_e(k, K, p);
        if (py >= 0) to_l2(psi_pairs(d, PSI_EY) + y);
        if (sx_) to_l2(psi_pairs(d, PSI_EX) + x);
        if (nv > 0 && pz >= 0) to_l2(psi_pairs(d, PSI_EZ) + (oz + pz * plane));
      };
      const auto planes = [&](auto curl_only) {
        constexpr bool kCurl = decltype(curl_only)::value;
        if constexpr (!kCurl) first_pairs(kb);
#pragma unroll 1
        for (int k = kb; k < kb + np; ++k, ++q) {
          s = q % NS;
          if (k > kb && !wait_on(&full[s], (uint32_t)((q / NS) & 1))) {
            return false;
          }
          const unsigned char *st = smem + s * ST;
          const float *sE = reinterpret_cast<const float *>(st) + ry * G::BX + xo;
          const float *sH =
              reinterpret_cast<const float *>(st + S::E_HALO) + (ry + 1) * G::HW + xo + 4;
          Q4 Ax, Ay, Az, Cx, Cy, Cz;  // Cexe.. and Cexh..
          if (use_mat) {
            const ushort4 id = *reinterpret_cast<const ushort4 *>(
                reinterpret_cast<const uint16_t *>(st + S::E_MAT) + ry * G::BX + xo);
            const int ids[4] = {id.x, id.y, id.z, id.w};
            if (TAB) {
#pragma unroll
              for (int c = 0; c < 4; ++c) {
                const float4 r0 = *reinterpret_cast<const float4 *>(stab + ids[c] * kTabRow);
                const float2 r1 = *reinterpret_cast<const float2 *>(stab + ids[c] * kTabRow + 4);
                set(Ax, c, r0.x);
                set(Ay, c, r0.y);
                set(Az, c, r0.z);
                set(Cx, c, r0.w);
                set(Cy, c, r1.x);
                set(Cz, c, r1.y);
              }
            } else {
#pragma unroll
              for (int c = 0; c < 4; ++c) {
                const float2 *r = reinterpret_cast<const float2 *>(d.mat_tab + ids[c] * 6);
                const float2 r0 = r[0], r1 = r[1], r2 = r[2];
                set(Ax, c, r0.x);
                set(Ay, c, r0.y);
                set(Az, c, r1.x);
                set(Cx, c, r1.y);
                set(Cy, c, r2.x);
                set(Cz, c, r2.y);
              }
            }
          } else {
            const int nc = kCurl || nv > 0 ? n : 0;
            Ax = q4(__ldg(reinterpret_cast<const float4 *>(d.ce[0] + nc)));
            Ay = q4(__ldg(reinterpret_cast<const float4 *>(d.ce[1] + nc)));
            Az = q4(__ldg(reinterpret_cast<const float4 *>(d.ce[2] + nc)));
            Cx = q4(__ldg(reinterpret_cast<const float4 *>(d.ce[3] + nc)));
            Cy = q4(__ldg(reinterpret_cast<const float4 *>(d.ce[4] + nc)));
            Cz = q4(__ldg(reinterpret_cast<const float4 *>(d.ce[5] + nc)));
          }
          constexpr int C1 = S::C1;
          const Q4 hx = lds4(sH), hy = lds4(sH + C1), hz = lds4(sH + 2 * C1);
          const float hy_l = sH[C1 - 1], hz_l = sH[2 * C1 - 1];
          Q4 dHz_y = sub4(hz, lds4(sH + 2 * C1 - G::HW)), dHx_y = sub4(hx, lds4(sH - G::HW));
          const Q4 dHz_x = {{hz.a.x - hz_l, hz.a.y - hz.a.x}, {hz.b.x - hz.a.y, hz.b.y - hz.b.x}};
          const Q4 dHy_x = {{hy.a.x - hy_l, hy.a.y - hy.a.x}, {hy.b.x - hy.a.y, hy.b.y - hy.b.x}};
          Q4 dHy_z = sub4(hy, hy_km), dHx_z = sub4(hx, hx_km);
          hx_km = hx;
          hy_km = hy;
          Q4 ex = add4(mul4(Ax, lds4(sE)), mul4(Cx, sub4(dHz_y, dHy_z)));
          Q4 ey = add4(mul4(Ay, lds4(sE + 512)), mul4(Cy, sub4(dHx_z, dHz_x)));
          Q4 ez = add4(mul4(Az, lds4(sE + 1024)), mul4(Cz, sub4(dHy_x, dHx_y)));
          if constexpr (!kCurl) {
            if (i == 0 || j == 0 || k == 0) {  // the curl's guards (gpu.h:727-763)
              if (i == 0) {
                ey.a.x = sE[512];
                ez.a.x = sE[1024];
              }
              if (j == 0 || k == 0) ex = lds4(sE);
              if (k == 0) ey = lds4(sE + 512);
              if (j == 0) ez = lds4(sE + 1024);
            }
            // CPML Y, Z, X (gpu.h:790-827, :829-868, :765-788)
            const bool k_in = k >= 1 && k <= K - 2;
            const int pz = slab_e(k, K, p);
            const bool sy = py >= 0 && k_in, sz = nv > 0 && pz >= 0 && j_in, sx = sx_ && k_in;
            if (AHEAD && k + 1 < kb + np) ahead(k + 1, oy + sY, ox + sX);
            if (i == 0 || i + 3 > I - 2) {  // Y, Z: 1 <= i <= I-2
              const Q4 none = all4(0.f);
              const uint32_t off = (i == 0 ? 1u : 0u) | 0xfu << min(max(I - 1 - i, 0), 4);
              put_back(dHz_y, none, off);
              put_back(dHx_y, none, off);
              put_back(dHy_z, none, off);
              put_back(dHx_z, none, off);
            }
            if (sy) {
              ps = recur<kOne>(d, ps, all4(tb[py]), all4(tc[py]), dHz_y, dHx_y);
              corr4<true, 0>(ex, Cx, ps, dx);
              corr4<false, 1>(ez, Cz, ps, dx);
              stp4(psi_pairs(d, PSI_EY) + oy, ps);
            }
            if (sz) {
              float2 *Z = psi_pairs(d, PSI_EZ) + (oz + pz * plane);
              if (sy) ps = ldp4(Z);
              ps = recur<kOne>(d, ps, all4(tb[pz]), all4(tc[pz]), dHy_z, dHx_z);
              corr4<false, 0>(ex, Cx, ps, dx);
              corr4<true, 1>(ey, Cy, ps, dx);
              stp4(Z, ps);
            }
            if (sx) {
              if (sy || sz) ps = ldp4(psi_pairs(d, PSI_EX) + ox);
              Q4 b, c;
              const Q4 ey0 = ey, ez0 = ez;
              const uint32_t out =
                  grading_x(tb, tc, i, [&](int v) { return slab_e(v, I, p); }, b, c);
              ps = recur<kOne>(d, ps, b, c, dHz_x, dHy_x);
              corr4<false, 0>(ey, Cy, ps, dx);
              corr4<true, 1>(ez, Cz, ps, dx);
              put_back(ey, ey0, out);
              put_back(ez, ez0, out);
              stp4(psi_pairs(d, PSI_EX) + ox, ps);
            }
            if (nv < 4) {
              const uint32_t past = 0xfu << max(nv, 0);
              put_back(ex, lds4(sE), past);
              put_back(ey, lds4(sE + 512), past);
              put_back(ez, lds4(sE + 1024), past);
            }
          }
          if constexpr (IN_PLANE && !kCurl) {
            if (faces && nv > 0) {
              Q4 *const ff[3] = {&ex, &ey, &ez};
              const Q4 *const cc[3] = {&Cx, &Cy, &Cz};
              if constexpr (OB)
                oblique_faces<false>(d, d.ob_inc[1] + (int64_t)step * d.ob_w, i, j, k, ff, cc);
              else
                axis_faces<false>(d, op.tfsf_mode, inc_e_row(d, op.tfsf_mode, step), i, j, k, ff, cc);
            }
          }
          if (kCurl || nv > 0) {
            stg4(d.f[0] + n, ex);
            stg4(d.f[1] + n, ey);
            stg4(d.f[2] + n, ez);
          }
          n += plane;
          if constexpr (!kCurl) {
            oy += sY;
            ox += sX;
            if (k + 1 < kb + np) first_pairs(k + 1);
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(&empty[s]);
        }
        return true;
      };
      good = __all_sync(0xffffffffu, nv == 4 && py < 0 && !sx_ && i > 0 && j > 0) && !faces &&
                     kb >= p && kb + np <= K - p
                 ? planes(std::true_type{})
                 : planes(std::false_type{});
    }
    if (!good) {
      if (f.err) atomicExch(f.err, m.x ? 1 : 2);
      return;
    }
    // the item's face cells, then its source cells
    const Box t = {m1.y, m1.y + G::BX - 1, m1.z, m1.z + G::BY - 1, kb, kb + np - 1};
    bool ok = true;
    if (!IN_PLANE && op.tfsf_mode) {
      const uint32_t mask = __ballot_sync(
          0xffffffffu, lane < 12 && face_of<OB>(d, m.x == 0, op.tfsf_mode, lane, t).any);
      if (mask) {
        ok = group_sync();
        if (ok) face_pass<OB, TAB, G>(d, stab, m.x == 0, op.tfsf_mode, step, t, tid, mask);
      }
    }
    if (m.x && op.cur_mode &&
        meets(t, op.cur_box[0], op.cur_box[1], op.cur_box[2], op.cur_box[3], op.cur_box[4],
              op.cur_box[5])) {
      ok = ok && group_sync();
      if (ok) current_pass(d, op, step, t, tid);
    }
    if (!ok) {
      if (f.err) atomicExch(f.err, 4);
      return;
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&cg.done[m.y]);  // after the warp's stores
  }
}

// Blocks of a kernel on the current device (one per SM), its shared memory
// opted in once.
template <class K>
int prepare(K kern, int threads, int smem, int *cached) {
  if (*cached > 0) return 0;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return (int)e;
  int per_sm = 0, sms = 0, dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem);
  if (e != cudaSuccess) return (int)e;
  *cached = (per_sm > 0 ? per_sm : 1) * (sms > 0 ? sms : 1);
  return 0;
}

template <bool MU, bool OB, bool TAB, int SIZE, class G>
int launch(const fdtd_dev *d, const fdtd_maps_flow *m, const fdtd_op *op, const fdtd_flow *w,
           cudaStream_t s) {
  static_assert(sizeof(FlowMaps) == sizeof(((fdtd_maps_flow *)0)->bytes), "map layout");
  static int cached = 0;
  constexpr int NG = kGroups<MU, SIZE == kBig>;
  constexpr int smem = FG<NG, G>::SMEM;
  auto kern = k_flow<NG, MU, OB, TAB, SIZE, G>;
  if (const int e = prepare(kern, kThreads<NG>, smem, &cached)) return e;
  FlowMaps mp;
  memcpy(&mp, m->bytes, sizeof(FlowMaps));
  Flow f;
  memset(&f, 0, sizeof(f));
  f.n_steps = w->n_steps;
  f.first = w->first;
  f.base = w->base;
  f.work = d->work;
  f.cnt = w->cnt;
  f.err = w->err;
  f.zc = w->zc;
  f.nch_h = (d->K - 1 + w->zc - 1) / w->zc;
  f.nch_e = (d->K + w->zc - 1) / w->zc;
  f.tx_h = (d->I - 1 + G::BX - 1) / G::BX;
  f.ty_h = (d->J - 1 + G::BY - 1) / G::BY;
  f.tx_e = (d->I + G::BX - 1) / G::BX;
  f.ty_e = (d->J + G::BY - 1) / G::BY;
  f.tiles = f.tx_e * f.ty_e;
  f.per_half = f.tiles * f.nch_e;
  f.by_step = make_div(2 * f.per_half);
  f.by_tiles = make_div(f.tiles);
  f.by_tx = make_div(f.tx_e);
  const long long tickets = 2ll * f.per_half * w->n_steps;
  if (tickets > (1ll << 30) || tickets < 1) return (int)cudaErrorInvalidValue;
  f.n_tickets = (int)tickets;
  f.probe_first = w->probe_first;
  f.probe_at = reinterpret_cast<const int2 *>(w->probe_at);
  f.n_probes = w->n_probes;
  const long long want = (2ll * f.tiles * f.nch_e + NG - 1) / NG;  // a step's items
  int blocks = want < cached ? (int)want : cached;
  if (w->blocks > 0 && w->blocks < blocks) blocks = w->blocks;
  kern<<<blocks, kThreads<NG>, smem, s>>>(*d, *op, mp, f);
  fdtdk_count_launches(1);
  return (int)cudaGetLastError();
}

template <bool MU, bool OB, bool TAB>
int launch_tiled(const fdtd_dev *d, const fdtd_maps_flow *m, const fdtd_op *op, const fdtd_flow *w,
                 cudaStream_t s) {
  if (w->tile == 0) return launch<MU, OB, TAB, kBig, GS>(d, &m[0], op, w, s);
  if (w->ahead) return launch<MU, OB, TAB, kBig, GB>(d, &m[1], op, w, s);
  if (w->zc == 1 && op->tfsf_mode) return launch<MU, OB, TAB, kSmall, GB>(d, &m[1], op, w, s);
  return launch<MU, OB, TAB, kMid, GB>(d, &m[1], op, w, s);
}
template <bool MU, bool OB>
int launch_coef(const fdtd_dev *d, const fdtd_maps_flow *m, const fdtd_op *op, const fdtd_flow *w,
                cudaStream_t s) {
  return d->coef_mode == 1 && d->n_mat <= kSmemTabMax ? launch_tiled<MU, OB, true>(d, m, op, w, s)
                                                      : launch_tiled<MU, OB, false>(d, m, op, w, s);
}

template <class G>
int make_maps(const fdtd_dev *d, int64_t fstride, fdtd_maps_flow *m) {
  m->valid = 0;
  if (((d->Ip * 4) % 16) || ((d->Ip * 2) % 16) || (fstride * 4) % 16)
    return (int)cudaErrorInvalidValue;
  if (!d->mat || ((uintptr_t)d->mat) % 16 || ((uintptr_t)d->f[0]) % 16 ||
      ((uintptr_t)d->f[3]) % 16)
    return (int)cudaErrorInvalidValue;
  for (int c = 1; c < 3; ++c)
    if (d->f[c] != d->f[0] + c * fstride || d->f[3 + c] != d->f[3] + c * fstride)
      return (int)cudaErrorInvalidValue;
  CUtensorMap *t = reinterpret_cast<CUtensorMap *>(m->bytes);
  int e = encode3(&t[0], d->f[0], d, fstride, G::BX, G::BY);
  if (!e) e = encode3(&t[1], d->f[3], d, fstride, G::BX, G::BY);
  if (!e) e = encode3(&t[2], d->f[0], d, fstride, G::HW, G::HH);
  if (!e) e = encode3(&t[3], d->f[3], d, fstride, G::HW, G::HH);
  if (!e) e = encode(&t[4], (void *)d->mat, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, d, G::BX, G::BY);
  if (!e) m->valid = 1;
  return e;
}

}  // namespace

extern "C" {

int fdtdk_make_maps_flow(const fdtd_dev *d, int tile, int64_t fstride, fdtd_maps_flow *m) {
  switch (tile) {
    case 0: return make_maps<GS>(d, fstride, m);
    case 1: return make_maps<GB>(d, fstride, m);
  }
  m->valid = 0;
  return (int)cudaErrorInvalidValue;
}

int fdtdk_flow(const fdtd_dev *d, const fdtd_maps_flow *m, const fdtd_op *op, const fdtd_flow *w,
               cudaStream_t s) {
  const bool ob = op->tfsf_mode == FDTD_MODE_OBLIQUE;
  if (d->hcoef_mode)
    return ob ? launch_coef<true, true>(d, m, op, w, s) : launch_coef<true, false>(d, m, op, w, s);
  return ob ? launch_coef<false, true>(d, m, op, w, s) : launch_coef<false, false>(d, m, op, w, s);
}

int fdtdk_check_recurrence(fdtd_div_plan p, unsigned long long *out, cudaStream_t s) {
  fdtd_dev d;
  memset(&d, 0, sizeof(d));
  d.dx = p.dx;
  d.rdx = p.rdx;
  d.div_lo = p.lo;
  d.div_hi = p.hi;
  d.div_lo2 = p.lo2;
  d.div_small = p.small;
  for (int tiny = 0; tiny < 2; ++tiny) {
    k_check_recurrence<true><<<152 * 8, 256, 0, s>>>(d, tiny, out);
    k_check_recurrence<false><<<152 * 8, 256, 0, s>>>(d, tiny, out);
  }
  fdtdk_count_launches(4);
  return (int)cudaGetLastError();
}

int64_t fdtdk_flow_counters(int32_t J, int32_t K) {
  const int64_t rows = (J + 3) / 4;  // the flattest tile is 4 rows high
  return 2 * rows * K;
}

}  // extern "C"
