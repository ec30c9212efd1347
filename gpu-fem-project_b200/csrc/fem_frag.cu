// Warp-fragment assembly kernel: FP64 residual + Jacobian assembly, LINEAR strain at
// orders 2 to 4 and NONLINEAR (Green) strain at orders 2 and 3; FEM_PRECISION_MIXED at
// order 3 with the element stiffness as BF16x6 tensor-core products (which paths use
// it: frag_supported and b16_stiffness at the end of this file).  Launch forms: one
// list-position range (plans, drop-in), up to four ranges (the band-split launches of
// fem_plan_assemble_host), tile queues (batches, the server).
//
// The element kernel in fem_device.cuh stages every element's coordinates,
// states and scaled gradients in shared memory and reads them back for each
// stage; at p = 3 that is ~400 shared-memory wavefronts per element and the
// L1 data pipe, not HBM, bounds it.  Here a warp assembles two elements per
// step and keeps their data in registers laid out as FP64 tensor-core
// (mma.m8n8k4) fragments:
//
//   1. gather    lane (g, t) (g = lane/4, t = lane%4) loads component c = g%4
//                (x, y, u, v) of node 4ks + t of element g/4: that register IS
//                the B fragment of step 2 (columns = 2 elements x 4 components,
//                k = element nodes).  Node ids are read two steps ahead, the
//                coordinates/states one step ahead.
//   2. J stage   C_d[q][(e,c)] = sum_a dN_d(a, q) X[a][(e,c)]: the isoparametric
//                Jacobian and the reference-space state gradient of both
//                elements at every quadrature point (8 points per tile), with the
//                derivative table as A fragments (shared memory, lane order).
//   3. points    lane (g, t) holds J (t even) or grad u (t odd) of element t/2 at its
//                tiles' points q = 8tm + g; one xor-1 exchange per pair of tiles hands
//                each lane all eight values of one point.  It forms det J, sqrt|s| J^-1
//                (s = w det J t) and the weak stress in FP64 and stores the ~8 doubles
//                of q to shared memory.
//   4. fragments lane (g, t) builds G-hat_i(q, a) = sqrt|s| (dN(a,q) J^-1)_i for
//                q = 4ks + t from sqrt|s| J^-1 and the table: the A and B fragments
//                of M_ij[a][b] = sum_q s G_ai G_bj.
//   5. residual  R_(a,i) = sum_q sum_j G-hat_j S-hat_ij on the FP64 pipe from the
//                same fragments, reduced over the lanes of a node by shuffles.
//   6. stiffness component-major node tiles (a = 8T + pi(g), pi(g) = 4(g%2) + g/2;
//                pairs TA <= TB, four (i, j) tiles sharing fragments, k-steps
//                outermost): lane (g, t) ends with WHOLE 2x2 blocks (a, b = 8TB +
//                4h + t), so the plane-stress combination needs no shuffle and a
//                warp store covers eight runs of four consecutive blocks.  Orders 2
//                and 4 (9 and 25 nodes) leave the last node out of the tiles; its row
//                and column take the FP64 pipe.  Order 4 runs its six tile pairs in
//                two passes of twelve accumulator tiles (an earlier form, 28 tiles of
//                interleaved rows r = 2a + i in five groups, formed 19 instead of 5
//                fragment pairs per k-step and exchanged the two rows of every block
//                between lanes: 256^2 703 -> 507 us, now 486; the same at two CTAs per SM
//                and 255 registers: 537 against 507 us).  Blocks above the diagonal are also written
//                transposed.
//
// Writes.  Plan mode: a launch is one colour; the first contributor of a block
// stores it (one 256-bit store); a later colour adds its 2x2 blocks with
// asynchronous bulk reductions (cp.reduce.async.bulk .add.f64 from shared memory)
// instead of four FP64 L2 atomics per block -- at p = 3 staged by row run, one
// 128-byte reduction per run of four adjacent blocks.  Drop-in mode (reference
// element map, accumulate-into) adds every block that way.  Residual rows: first
// writer stores, others add with atomics.  The arithmetic is the closed form of
// the reference's per-column forward AD (element/FEKernels.h:286-315, 884-976)
// that the element kernel documents.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "fem_common.h"
#include "fem_device.cuh"
#include "fem_launch.h"

// Resident CTAs per SM the register budget is sized for: 3 (168 registers) at
// p = 3, where the 12 live stiffness accumulators need them, and in p = 4 plans; 4 (128)
// at p = 2; 2 (255) in the p = 4 drop-in Jacobian, whose map entries are in flight beside
// the accumulators and whose reductions, not its warps, set the time (200 x 199 485 us, with
// 3 CTAs 511; the plan, whose blocks leave one by one, loses: 256^2 507, with 2 CTAs 537).
// The residual alone, without stiffness accumulators: 6 (85 registers) at
// p = 2, 3 (800 x 512 p = 2: 175 / 159 / 152 us with 4 / 5 / 6; 600 x 590 p = 3: 172 / 162 /
// 160 us), 4 at p = 4 (256^2: 102 / 107 / 115 us).
#ifndef FEM_FRAG_MINB
#define FEM_FRAG_MINB ((MODE & kJac) == 0 ? (P == 4 ? 4 : 6) : P == 2 ? 4 : P == 4 && (MODE & kPlan) == 0 ? 2 : 3)
#endif

namespace fem {
namespace dev {

template <int P>
struct FragDims {
  static constexpr int P1 = P + 1, NN = P1 * P1, NQ = NN;
  static constexpr int K4 = (NN + 3) / 4;   // node k-steps = quadrature k-steps
  static constexpr int NQP = 4 * K4;        // padded quadrature points
  static constexpr int QT = 2 * ((NQ + 15) / 16);  // J-stage row tiles (8 quadrature points each), in pairs
  static constexpr int NTM = NN / 8;        // node tiles of the component-major stiffness product
  static constexpr bool EX = NN % 8 == 1;   // orders 2, 4: the last node is in no tile (FP64 pipe)
  static constexpr int NPASS = NTM == 3 ? 2 : 1;  // stiffness passes (at most 12 accumulator tiles each)
  static constexpr int CS = Dims<P>::CS;    // plan code record bytes per element
  static constexpr int WARPS = 4;           // warps per CTA
  static_assert(P >= 2 && P <= 4 && (NN == 8 * NTM || EX), "fragment kernel: orders 2 to 4");
  // Local node at position m of the tiles: m, but at order 4, where four x-neighbours sit at
  // positions 4r .. 4r + 3 (grid row r) and then the last column: the blocks of a row's
  // four columns, and the residual rows of a quadruple of lanes, are adjacent in memory
  // wherever the numbering follows the grid.  (Not the plan's Jacobian, whose blocks leave
  // one by one: 381 x 379 1034 us, permuted 1075.)
  __host__ __device__ static constexpr int node(int m) {
    return P < 4 ? m : (m < 20 ? 5 * (m >> 2) + (m & 3) : (m < 24 ? 5 * (m - 20) + 4 : 24));
  }
  // Node-tile pair k = (ta, tb) of a pass: pass 0 the pairs of tiles 0 and 1 (order 2: of
  // tile 0), pass 1 those of tile 2.
  static constexpr int NPAIR = NTM == 1 ? 1 : 3;
  __host__ __device__ static constexpr int ta(int pass, int k) { return pass ? k : (k == 2 ? 1 : 0); }
  __host__ __device__ static constexpr int tb(int pass, int k) { return pass ? 2 : (k == 0 ? 0 : 1); }
};

template <int V>
using IC = std::integral_constant<int, V>;

// Shared memory: CTA tables, then one region per warp.  DROP: drop-in mode (the
// stage holds the reference element map rows, NN*NN ints per element, instead of
// plan code records).  B16: the BF16x6 stiffness table follows the CTA tables.
// JAC = false (residual only): no block staging slots.
template <int P, bool DROP = false, bool NL = false, bool B16 = false, bool JAC = true>
struct FragLayout {
  using F = FragDims<P>;
  static constexpr int K4 = F::K4, NQP = F::NQP, NN = F::NN;
  // staged bytes per element (drop-in order 4: none, the issuing lanes load their entries)
  static constexpr int CS = !DROP ? F::CS : (P == 4 ? 0 : 4 * NN * NN);
  // Slot of quadrature point q of an element's arrays, and the slots between the two
  // elements: a quarter-warp of the quadrature stage stores points q, q + 1 of two
  // tiles of both elements (slots g, g + 10, g + PS, g + PS + 10 with PS = 4 mod 8:
  // eight distinct 16-byte bank groups); the fragment loads read four consecutive slots.
  static constexpr int PS = (NQP + 2 * ((NQP - 1) / 8) + 11) / 8 * 8 - 4;
  __host__ __device__ static constexpr int slot(int q) { return q + 2 * (q >> 3); }
  static constexpr size_t tabJ = 0;                          // double2 [K4][QT][32]
  static constexpr size_t tabF = tabJ + 16 * K4 * F::QT * 32;  // double2 [K4][NTM][32]
  static constexpr size_t tabX = tabF + 16 * K4 * F::NTM * 32;  // double2 [NQP]: dN of the node outside the tiles
  static constexpr int NQT = 8 * F::QT;                       // points of the J stage's tiles
  static constexpr size_t wq = tabX + (F::EX ? 16 * NQP : 0);  // double [NQT]
  static constexpr size_t csum = align16(wq + 8 * NQT);       // double2 [NQT]: sum_a dN(a, q)
  static constexpr size_t tabB = align16(csum + 16 * NQT);    // double2 [8][32]: BF16x6 stiffness operands
  // uint32: runs (order 3: 64; drop-in orders 2 and 4: DR per pass)
  static constexpr int DR = !DROP || !JAC ? 0 : (P == 2 ? 32 : P == 4 ? 96 : 0);
  static constexpr size_t tabR = align16(tabB + (B16 ? 16 * 8 * 32 : 0));
  static constexpr size_t warps = align16(tabR + 4 * (P == 3 ? 64 : DR * F::NPASS));
  // warp-relative; [2] = the two elements of the step, point q at slot(q) of PS
  // (residual alone: s sigma J^-T, rows x and y, in WI0 and WI1, and no more)
  static constexpr size_t WI0 = 0;                  // double2 [2][PS]: sqrt|s| (J^-1_0x, J^-1_1x)
  static constexpr size_t WI1 = WI0 + 16 * 2 * PS;  // double2 [2][PS]: sqrt|s| (J^-1_0y, J^-1_1y)
  static constexpr size_t WS0 = WI1 + 16 * 2 * PS;  // double2 [2][PS]: (S-hat_xx, S-hat_xy)
  static constexpr size_t WS1 = WS0 + (JAC ? 16 * 2 * PS : 0);  // double2 [2][PS]: (S-hat_xy, S-hat_yy)
  static constexpr size_t SG = WS1 + (JAC ? 16 * 2 * PS : 0);   // double [2][NQP]: sign of s (0 on padding)
  static constexpr size_t MC = align16(SG + (JAC ? 8 * 2 * NQP : 0));  // double2: the mesh's (+-sqrt|t| or |t mu|, lam / mu)
  static constexpr size_t NID = MC + 16;            // int [2][NN]: node ids
  static constexpr size_t RB = align16(NID + 4 * 2 * NN);  // int [2][NN]: rowp[node]
  static constexpr size_t STAGE = align16(RB + 4 * 2 * NN);  // [2 buffers][2 elements][CS] code records
  // staging slots: p = 3, 3 node-tile pairs x 2 halves, direct and transposed; p = 2, 4, the
  // blocks one lane has in flight; drop-in p = 4 a pass's pairs and node XN's blocks
  static constexpr int NSLOT = P == 3 ? 8 : (P == 4 && DROP ? 11 : 4);
  static constexpr size_t REDS = align16(STAGE + 2 * 2 * CS);  // double4 [NSLOT][32]: bulk-reduction sources
  // NONLINEAR: sign(s) x tangent modulus, double [2][NQP][2 (l)][8 (i, k, n)]
  static constexpr size_t AT = align16(REDS + (JAC ? 32 * NSLOT * 32 : 0));
  static constexpr size_t warp_bytes = align16(AT + (NL && JAC ? 8 * 2 * NQP * 16 : 0));
  static constexpr size_t total = warps + F::WARPS * warp_bytes;
};

// D = A B, the first product of an accumulator (no zeroed registers needed).
__device__ __forceinline__ void dmma_first(double &c0, double &c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%4,%4};"
               : "=d"(c0), "=d"(c1)
               : "d"(a), "d"(b), "d"(0.0));
}

// D += A B, m16n8k16, BF16 operands, FP32 accumulate.
__device__ __forceinline__ void bmma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// v ~ hi + mid + lo, three BF16 parts (8 significant bits each, 24 together): the
// FP32 value and its two successive remainders, each rounded to nearest.
__device__ __forceinline__ void split3(double v, uint32_t &hi, uint32_t &mid, uint32_t &lo) {
  const float f = __double2float_rn(v);
  const __nv_bfloat16 h = __float2bfloat16_rn(f);
  const float r1 = f - __bfloat162float(h);
  const __nv_bfloat16 m = __float2bfloat16_rn(r1);
  const __nv_bfloat16 l = __float2bfloat16_rn(r1 - __bfloat162float(m));
  hi = __bfloat16_as_ushort(h);
  mid = __bfloat16_as_ushort(m);
  lo = __bfloat16_as_ushort(l);
}

// Run r of staging slot sl (see frag_slot): four blocks of one matrix row `row` with four
// consecutive element-local columns from col0, staged from position pos0 of the slot.
// Packed as row NN + col0 (a code record offset) | first staged double << 16.
__device__ __forceinline__ uint32_t frag_run(int sl, int r) {
  const int k = sl < 2 ? 0 : (sl < 6 ? 1 : 2);
  const int h = sl < 2 ? sl : (sl < 6 ? (sl - 2) >> 1 : sl - 6);
  const int w = (sl >= 2 && sl < 6) ? ((sl - 2) & 1) : 0;
  const int TA = k == 2 ? 1 : 0, TB = k == 0 ? 0 : 1;
  int row, col0, pos0;
  if (w == 0) {
    row = 8 * TA + 4 * (r & 1) + (r >> 1);  // pi(r)
    col0 = 8 * TB + 4 * h;
    pos0 = 4 * r;
  } else {
    const int tt = r >> 1, half = r & 1;
    row = 8 * TB + 4 * h + tt;
    col0 = 8 * TA + 4 * half;
    pos0 = 8 * tt + 4 * half;
  }
  return (uint32_t)(row * 16 + col0) | (uint32_t)(128 * sl + 4 * pos0) << 16;
}

// Drop-in orders 2 and 4, entry i of a pass: up to four staged blocks of one matrix row,
// packed as row NN + first column | (columns 5 apart) << 10 | (blocks - 1) << 11 |
// staged position << 13; 0xffffffff: none.  Staging slots: a pass's node-tile pairs
// (direct: position 4r + t of row pi(r), transposed: 8t + pi(g)), then node XN's row and
// column, (XN, m) and (m, XN), and its diagonal block.
template <int P>
__host__ __device__ __forceinline__ uint32_t drop_run(int pass, int i) {
  using F = FragDims<P>;
  constexpr int NN = F::NN, XN = NN - 1;
  auto pack = [](int row, int col0, bool five, int n, int src) {
    return (uint32_t)(row * NN + col0) | (uint32_t)five << 10 | (uint32_t)(n - 1) << 11 | (uint32_t)src << 13;
  };
  auto pi = [](int r) { return 4 * (r & 1) + (r >> 1); };
  auto quad = [&](int row, int m0, int src) { return pack(row, F::node(m0), m0 == 20, 4, src); };
  if constexpr (P == 2) {
    if (i < 16) return quad(pi(i & 7), 4 * (i >> 3), 32 * (i >> 3) + 4 * (i & 7));
    if (i < 18) return quad(XN, 4 * (i - 16), 64 + 4 * (i - 16));
    if (i < 26) return pack(i - 18, XN, false, 1, 64 + 8 + i - 18);
    return i == 26 ? pack(XN, XN, false, 1, 64 + 16) : 0xffffffffu;
  } else if constexpr (P == 4) {
    const int s = i >> 3, r = i & 7, np = pass ? 80 : 64;
    if (i < np) {
      const int k = pass ? (s < 8 ? s >> 2 : 2) : (s < 2 ? 0 : s < 6 ? 1 : 2);
      const int h = pass ? (s < 8 ? (s >> 1) & 1 : s - 8) : (s < 2 ? s : s < 6 ? (s - 2) >> 1 : s - 6);
      const bool w = pass ? (s < 8 && (s & 1)) : (s >= 2 && s < 6 && (s & 1));
      const int TA = F::ta(pass, k), TB = F::tb(pass, k);
      if (!w) return quad(F::node(8 * TA + pi(r)), 8 * TB + 4 * h, 32 * s + 4 * r);
      const int tt = r >> 1, half = r & 1;
      return quad(F::node(8 * TB + 4 * h + tt), 8 * TA + 4 * half, 32 * s + 8 * tt + 4 * half);
    }
    const int j = i - np, sx = 4 * np;  // node XN's slot follows the pairs'
    const int nq = pass ? 2 : 4, nm = pass ? 8 : 16, m0 = pass ? 16 : 0;
    if (j < nq) return quad(XN, m0 + 4 * j, sx + 4 * j);
    if (j < nq + nm) return pack(F::node(m0 + j - nq), XN, false, 1, sx + nm + j - nq);
    return pass && j == nq + nm ? pack(XN, XN, false, 1, sx + 2 * nm) : 0xffffffffu;
  }
  return 0xffffffffu;
}

// Drop-in: the blocks staged from `src` on are added at map offsets m[0..3] (n = 1 or 4
// of them), each maximal stretch of blocks adjacent in the matrix with one reduction;
// FP64 atomics where a block is not 16-byte aligned (the matrix is not, or the caller's map
// has an odd offset).  n = 0: none.
__device__ __forceinline__ void drop_issue(double *mat, const int (&m)[4], int n, const double *src) {
  if (((reinterpret_cast<uintptr_t>(mat) | 8u * (unsigned)(m[0] | m[1] | m[2] | m[3])) & 15u) != 0) {
    for (int j = 0; j < n; j++)
      for (int c = 0; c < 4; c++) atomicAdd(mat + m[j] + c, src[4 * j + c]);
    return;
  }
  const int c1 = n == 4 && m[1] == m[0] + 4, c2 = n == 4 && m[2] == m[1] + 4, c3 = n == 4 && m[3] == m[2] + 4;
  const int b[4] = {n ? 32 * (1 + c1 * (1 + c2 * (1 + c3))) : 0, n == 4 && !c1 ? 32 * (1 + c2 * (1 + c3)) : 0,
                    n == 4 && !c2 ? 32 * (1 + c3) : 0, n == 4 && !c3 ? 32 : 0};
  const unsigned sa = (unsigned)__cvta_generic_to_shared(src);
#pragma unroll
  for (int j = 0; j < 4; j++)
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "setp.ne.s32 p, %2, 0;\n\t"
                 "@p cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f64 [%0], [%1], %2;\n\t}" ::"l"(mat + m[j]),
                 "r"(sa + 32 * j), "r"(b[j])
                 : "memory");
}

// Whether the four blocks of an entry are all apart.
__device__ __forceinline__ bool drop_apart(const int (&m)[4], int n) {
  return n == 4 && m[1] != m[0] + 4 && m[2] != m[1] + 4 && m[3] != m[2] + 4;
}

// drop_issue at order 4 for an element whose entries' blocks are mostly apart (a mesh
// numbered at random): those by FP64 atomics, four lanes to a block, which is faster there
// than four reductions of 32 bytes (90 x 89 184 / 165 us, 200 x 199 866 / 800; the element
// kernel's atomics 175 and 917).  A grid's last columns are apart too (8 of 32 entries):
// reductions are faster for those (200 x 199 485 / 513 us).
__device__ __forceinline__ void drop_issue_scattered(double *mat, const int (&m)[4], int n, const double *redsW, int src,
                                                     int lane) {
  const bool apart = drop_apart(m, n);
  drop_issue(mat, m, apart ? 0 : n, redsW + src);
  __syncwarp();
#pragma unroll 1
  for (int g = 0; g < 4; g++) {  // the entries of lanes 8g .. 8g + 7
    const int from = 8 * g + (lane >> 2), c = lane & 3;
    const bool add = __shfl_sync(0xffffffffu, (int)apart, from) != 0;
    const int s0 = __shfl_sync(0xffffffffu, src, from);
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int off = __shfl_sync(0xffffffffu, m[j], from);
      if (add) atomicAdd(mat + off + c, redsW[s0 + 4 * j + c]);
    }
  }
}

template <int P, int MODE>
__device__ __forceinline__ void frag_prologue(unsigned char *smem) {
  constexpr bool B16 = (MODE & kB16) != 0, SQRTW = (MODE & kNL) == 0 && (MODE & kJac) != 0;
  using F = FragDims<P>;
  using L = FragLayout<P, (MODE & kPlan) == 0, (MODE & kNL) != 0, B16, (MODE & kJac) != 0>;
  constexpr int P1 = F::P1, NN = F::NN, NQ = F::NQ, K4 = F::K4, QT = F::QT, NTM = F::NTM;
  double2 *tabJ = reinterpret_cast<double2 *>(smem + L::tabJ);
  double2 *tabF = reinterpret_cast<double2 *>(smem + L::tabF);
  double *wq = reinterpret_cast<double *>(smem + L::wq);
  // the 1D basis at the 1D points, [point][node] (N, dN), in the first warp's region: a
  // thread per entry, where evaluating it per 2D entry meant ten divergent constant loads
  // and two polynomials each (a large part of a small launch's time)
  double2 *b1 = reinterpret_cast<double2 *>(smem + L::warps);
  for (int i = threadIdx.x; i < P1 * P1; i += blockDim.x) {
    double N, dN1;
    lag1d(P, kGX[P][i / P1], i % P1, N, dN1);
    b1[i] = make_double2(N, dN1);
  }
  __syncthreads();
  // dN(a, q) = (N_y dN_x, N_x dN_y) with the rounding of the element kernel's table
  auto dN = [&](int a, int q) {
    const double2 x = b1[(q % P1) * P1 + a % P1], y = b1[(q / P1) * P1 + a / P1];
    return make_double2(__dmul_rn(y.x, x.y), __dmul_rn(x.x, y.y));
  };
  // J-stage A fragments: lane (g, t) of (ks, tm) holds dN(a = 4ks + t, q = 8tm + g)
  for (int i = threadIdx.x; i < K4 * QT * 32; i += blockDim.x) {
    const int lane = i & 31, blk = i >> 5, ks = blk / QT, tm = blk - ks * QT;
    const int a = 4 * ks + (lane & 3), q = 8 * tm + (lane >> 2);
    tabJ[i] = (a < NN && q < NQ) ? dN(a, q) : make_double2(0.0, 0.0);
  }
  // stiffness fragments at (ks, T): lane (g, t) holds dN(node(8T + pi(g)), q = 4ks + t)
  for (int i = threadIdx.x; i < K4 * NTM * 32; i += blockDim.x) {
    const int lane = i & 31, blk = i >> 5, ks = blk / NTM, T = blk - ks * NTM;
    const int g = lane >> 2, t = lane & 3, m = 8 * T + 4 * (g & 1) + (g >> 1), q = 4 * ks + t;
    const int a = (MODE & (kPlan | kJac)) == (kPlan | kJac) ? m : F::node(m);
    tabF[i] = q < NQ ? dN(a, q) : make_double2(0.0, 0.0);
  }
  if constexpr (F::EX) {
    double2 *tabX = reinterpret_cast<double2 *>(smem + L::tabX);
    for (int q = threadIdx.x; q < F::NQP; q += blockDim.x) tabX[q] = q < NQ ? dN(NN - 1, q) : make_double2(0.0, 0.0);
  }
  for (int q = threadIdx.x; q < L::NQT; q += blockDim.x) {
    const double w = q < NQ ? __dmul_rn(kGW[P][q % P1], kGW[P][q / P1]) : 0.0;
    wq[q] = SQRTW ? sqrt(w) : w;  // LINEAR Jacobians: the square root
  }
  // BF16x6 stiffness (order 3): entry (2k + h, lane (g, t)) holds dN(a, q) for the
  // node a = 8h + pi(g) and quadrature point q = 2t + (k & 1) + 8 (k >> 1) that lane
  // (g, t) places in its m16n8k16 fragments
  if constexpr (B16) {
    double2 *tabB = reinterpret_cast<double2 *>(smem + L::tabB);
    for (int i = threadIdx.x; i < 8 * 32; i += blockDim.x) {
      const int lane = i & 31, k = (i >> 5) >> 1, h = (i >> 5) & 1, g = lane >> 2, t = lane & 3;
      const int a = 8 * h + 4 * (g & 1) + (g >> 1), q = 2 * t + (k & 1) + 8 * (k >> 1);
      tabB[i] = (a < NN && q < NQ) ? dN(a, q) : make_double2(0.0, 0.0);
    }
  }
  if constexpr (P == 3) {
    for (int i = threadIdx.x; i < 64; i += blockDim.x)
      reinterpret_cast<uint32_t *>(smem + L::tabR)[i] = frag_run(i >> 3, i & 7);
  }
  for (int i = threadIdx.x; i < L::DR * F::NPASS; i += blockDim.x)
    reinterpret_cast<uint32_t *>(smem + L::tabR)[i] = drop_run<P>(i / (L::DR ? L::DR : 1), i % (L::DR ? L::DR : 1));
  // sum_a dN(a, q): zero in exact arithmetic, a few ulp of the table entries in
  // FP64; summed with Neumaier compensation (error ~1e-30 absolute) over the J-stage
  // table entries written above instead of evaluating the basis again
  __syncthreads();
  double2 *csum = reinterpret_cast<double2 *>(smem + L::csum);
  for (int q = threadIdx.x; q < L::NQT; q += blockDim.x) {
    double s0 = 0.0, c0 = 0.0, s1 = 0.0, c1 = 0.0;
    if (q < NQ) {
#pragma unroll
      for (int a = 0; a < NN; a++) {
        const double2 d = tabJ[((a >> 2) * QT + (q >> 3)) * 32 + 4 * (q & 7) + (a & 3)];
        const double t0 = s0 + d.x, t1 = s1 + d.y;
        c0 += fabs(s0) >= fabs(d.x) ? (s0 - t0) + d.x : (d.x - t0) + s0;
        c1 += fabs(s1) >= fabs(d.y) ? (s1 - t1) + d.y : (d.y - t1) + s1;
        s0 = t0;
        s1 = t1;
      }
    }
    csum[q] = make_double2(s0 + c0, s1 + c1);
  }
  __syncthreads();
}

// Staging slot of node-tile pair k (0: (0,0), 1: (0,1), 2: (1,1)), half h, and
// direct (0) / transposed (1) blocks.
__host__ __device__ constexpr int frag_slot(int k, int h, int w) { return k == 0 ? h : (k == 1 ? 2 + 2 * h + w : 6 + h); }

// The block (a, b) of element el (or its transpose (b, a) with w = 1), where `act`: plan
// mode stores it when this element is its first contributor (code bit 7, where `m80`
// has it); otherwise (and in drop-in mode always) it goes to its staging position for
// frag_issue_run.
// Predicated, without a branch: the lanes of a warp mix the two.  Returns the code (0 in
// drop-in mode), so that the caller knows whether any block was staged.
template <int P, bool PLAN>
__device__ __forceinline__ uint32_t frag_put(const Out &O, int el, int a, int b, int w, bool act, uint32_t m80, double kxx,
                                             double kxy, double kyx, double kyy, double *stg) {
  constexpr int NN = Dims<P>::NN, CS = Dims<P>::CS;
  const int r0 = w ? b : a, c0 = w ? a : b;
  const double v0 = kxx, v1 = w ? kyx : kxy, v2 = w ? kxy : kyx, v3 = kyy;
  const unsigned sa = (unsigned)__cvta_generic_to_shared(stg);
  if constexpr (PLAN) {
    const uint32_t code = O.codes[el * CS + r0 * NN + c0];
    double *blk = O.mat + 4 * ((int64_t)O.rbase[el * NN + r0] + (code & 0x7f));
    asm volatile("{\n\t.reg .pred f, s;\n\t"
                 "setp.ne.u32 f, %6, 0;\n\t"
                 "setp.ne.u32 s, %7, 0;\n\t"
                 "@f st.global.v4.f64 [%0], {%2, %3, %4, %5};\n\t"
                 "@s st.shared.v2.f64 [%1], {%2, %3};\n\t"
                 "@s st.shared.v2.f64 [%1 + 16], {%4, %5};\n\t}" ::"l"(blk),
                 "r"(sa), "d"(v0), "d"(v1), "d"(v2), "d"(v3), "r"(act ? code & m80 : 0u), "r"((uint32_t)(act && !(code & m80)))
                 : "memory");
    return act ? code : 0x80u;
  } else {
    if (act) {
      reinterpret_cast<double2 *>(stg)[0] = make_double2(v0, v1);
      reinterpret_cast<double2 *>(stg)[1] = make_double2(v2, v3);
    }
    return 0;
  }
}

// frag_put at order 3 with the code and the row's address in registers: one predicate.
template <int OFF>
__device__ __forceinline__ void frag_put_row(const double *row, uint32_t code, uint32_t m80, unsigned stg, double v0,
                                             double v1, double v2, double v3) {
  const double *blk = row + 4 * (code & 0x7f);
  asm volatile("{\n\t.reg .pred f;\n\t"
               "setp.ne.u32 f, %6, 0;\n\t"
               "@f st.global.v4.f64 [%0], {%2, %3, %4, %5};\n\t"
               "@!f st.shared.v2.f64 [%1 + %7], {%2, %3};\n\t"
               "@!f st.shared.v2.f64 [%1 + %8], {%4, %5};\n\t}" ::"l"(blk),
               "r"(stg), "d"(v0), "d"(v1), "d"(v2), "d"(v3), "r"(code & m80), "n"(OFF), "n"(OFF + 16)
               : "memory");
}

// Before the second element of a step writes.  In a plan's pair layout it shares an
// edge with the first: where the first stored a shared block (a generic-proxy
// 256-bit store) the second adds to it with a bulk reduction (async proxy, maybe
// another lane), and where both add (an earlier colour stored it) the first one's
// reduction must land first, or the two would round in either order.  So: wait
// for this lane's reductions to complete, order the lanes, order the proxies.
// Residual rows go generic store or atomic, then atomics: the barrier orders them.
// The order-3 writers, which store first and reduce last, take the two halves
// apart (pair_first_landed before, pair_first_visible after the barrier that
// precedes their reductions) so that the first element's reductions have the second
// element's stores to land in.
__device__ __forceinline__ void pair_first_landed() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void pair_first_visible() { asm volatile("fence.proxy.async.global;" ::: "memory"); }
__device__ __forceinline__ void pair_order_fence() {
  pair_first_landed();
  __syncwarp();
  pair_first_visible();
}

// A node's residual row: `act` lanes store it (first writer) or add to it, without a branch.
__device__ __forceinline__ void residual_put(double *dst, bool act, bool first, double x, double y) {
  asm volatile("{\n\t.reg .pred f, s;\n\t"
               "setp.ne.u32 f, %3, 0;\n\t"
               "setp.ne.u32 s, %4, 0;\n\t"
               "@f st.global.v2.f64 [%0], {%1, %2};\n\t"
               "@s red.global.add.f64 [%0], %1;\n\t"
               "@s red.global.add.f64 [%0 + 8], %2;\n\t}" ::"l"(dst),
               "d"(x), "d"(y), "r"((uint32_t)(act && first)), "r"((uint32_t)(act && !first))
               : "memory");
}

__device__ __forceinline__ void bulk_add(double *gdst, const double *src, int bytes) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(src);
  asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f64 [%0], [%1], %2;" ::"l"(gdst), "r"(sa),
               "r"(bytes)
               : "memory");
}

// Blocks of a run to add: drop-in, every block; plan, the blocks whose code is not a
// first store.  One 128-byte reduction when all four are added and adjacent in the
// matrix, else 32 bytes per block (four FP64 atomics for a block whose address is not
// 16-byte aligned).  Order 3 (16 nodes: a run's four code bytes are one word).
template <int P, bool PLAN>
__device__ __forceinline__ void frag_issue_run(const Out &O, int el, uint32_t run, const double *redsW) {
  constexpr int NN = Dims<P>::NN, CS = Dims<P>::CS;
  static_assert(NN == 16, "runs: order 3");
  const int off = run & 0xffff, row = off >> 4, col0 = off & 15;
  const double *src = redsW + (run >> 16);
  if constexpr (PLAN) {
    // most runs hold first stores only, most of the others add four adjacent blocks (or,
    // where a strip leaves the run's last block to its right neighbour, three)
    const uint32_t w4 = *reinterpret_cast<const uint32_t *>(O.codes + el * CS + off);
    const uint32_t addm = ~w4 & 0x80808080u;
    double *d0 = O.mat + 4 * ((int64_t)O.rbase[el * NN + row] + (w4 & 0x7f));
    const bool four = addm == 0x80808080u && w4 == (w4 & 0xff) * 0x01010101u + 0x03020100u;
    const bool three = addm == 0x00808080u && (w4 & 0xffffffu) == (w4 & 0xff) * 0x010101u + 0x020100u;
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "setp.ne.s32 p, %2, 0;\n\t"
                 "@p cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f64 [%0], [%1], %2;\n\t}" ::"l"(d0),
                 "r"((unsigned)__cvta_generic_to_shared(src)), "r"(four ? 128 : three ? 96 : 0)
                 : "memory");
    if (!__any_sync(0xffffffffu, addm != 0 && !four && !three)) return;
    if (addm == 0 || four || three) return;
  }
  double *dst[4];
  bool add[4];
  bool all = true, adj = true;
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const int col = col0 + j;
    if constexpr (PLAN) {
      const uint8_t code = O.codes[el * CS + row * NN + col];
      add[j] = !(code & 0x80);
      dst[j] = O.mat + 4 * ((int64_t)O.rbase[el * NN + row] + (code & 0x7f));
    } else {
      add[j] = true;
      dst[j] = O.mat + O.map[(el * NN + row) * NN + col];
    }
    all = all && add[j];
    if (j > 0) adj = adj && dst[j] == dst[0] + 4 * j;
  }
  if (all && adj && (reinterpret_cast<uintptr_t>(dst[0]) & 15u) == 0) {
    bulk_add(dst[0], src, 128);
    return;
  }
#pragma unroll
  for (int j = 0; j < 4; j++) {
    if (!add[j]) continue;
    if ((reinterpret_cast<uintptr_t>(dst[j]) & 15u) == 0) {
      bulk_add(dst[j], src + 4 * j, 32);
    } else {
      atomicAdd(dst[j] + 0, src[4 * j + 0]);
      atomicAdd(dst[j] + 1, src[4 * j + 1]);
      atomicAdd(dst[j] + 2, src[4 * j + 2]);
      atomicAdd(dst[j] + 3, src[4 * j + 3]);
    }
  }
}

// Per-block writer of plans at orders 2 and 4, where four consecutive element-local nodes
// straddle grid rows and row runs rarely merge: block (r0, c0) of element `el`, where
// `act`.  The first contributor stores it, a later one stages it in `slot` (this lane's,
// its previous bulk read complete) for bulk_add_block.  Without a branch.  Returns
// whether it staged the block, with its address.
template <int P>
__device__ __forceinline__ bool frag_put_block(const Out &O, int el, int r0, int c0, bool act, double v0, double v1,
                                               double v2, double v3, double *slot, double *&blk) {
  constexpr int NN = Dims<P>::NN, CS = Dims<P>::CS;
  if (!act) r0 = c0 = 0;
  const uint32_t code = O.codes[el * CS + r0 * NN + c0];
  blk = O.mat + 4 * ((int64_t)O.rbase[el * NN + r0] + (code & 0x7f));
  const uint32_t first = code & 0x80;
  const bool add = act && !first;
  asm volatile("{\n\t.reg .pred f, s;\n\t"
               "setp.ne.u32 f, %6, 0;\n\t"
               "setp.ne.u32 s, %7, 0;\n\t"
               "@f st.global.v4.f64 [%0], {%2, %3, %4, %5};\n\t"
               "@s st.shared.v2.f64 [%1], {%2, %3};\n\t"
               "@s st.shared.v2.f64 [%1 + 16], {%4, %5};\n\t}" ::"l"(blk),
               "r"((unsigned)__cvta_generic_to_shared(slot)), "d"(v0), "d"(v1), "d"(v2), "d"(v3),
               "r"(act ? first : 0u), "r"((uint32_t)add)
               : "memory");
  return add;
}

__device__ __forceinline__ void bulk_add_block(double *blk, const double *slot, bool add) {
  asm volatile("{\n\t.reg .pred p;\n\t"
               "setp.ne.u32 p, %2, 0;\n\t"
               "@p cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f64 [%0], [%1], 32;\n\t}" ::"l"(blk),
               "r"((unsigned)__cvta_generic_to_shared(slot)), "r"((uint32_t)add)
               : "memory");
}

// The element pairs a warp assembles, in order.
struct PairCursor {
  int mesh;
  int ne;  // 0 ends the warp's loop
  int64_t k0;
  int tile = -1;      // dependency-ordered launches: the pair's tile
  bool last = false;  // ... and whether it is the tile's last pair
  int fl = 0;         // strips: kHalo | kCarry | kRight
};


// Single mesh, order-4 plans: units p, p + stride, ... of list positions [begin, end), all of
// `unit` elements (their kernel, short of registers, is slower with the next form: 381 x 379
// 999 -> 1054 us).
struct UnitStride {
  static constexpr bool kBatched = false, kSched = false, kStrip = false;
  int64_t begin, end, p, stride;
  int unit;
  __device__ PairCursor next(int) {
    PairCursor c{0, 0, begin + unit * p};
    if (c.k0 < end) c.ne = (int)min((int64_t)unit, end - c.k0);
    p += stride;
    return c;
  }
};

// Single mesh: units p, p + stride, ... of `units`, the first `pairs` of them pairs of list
// positions from `begin` on, the others single elements.
struct PairStride {
  static constexpr bool kBatched = false, kSched = false, kStrip = false;
  int64_t begin;
  unsigned p, stride, pairs, units;
  __device__ PairCursor next(int) {
    PairCursor c{0, (p < pairs) + (p < units), begin + (p + min(p, pairs))};
    p += stride;
    return c;
  }
};

// One mesh, up to kMaxRanges list-position ranges of one launch (the band-split
// launches of fem_plan_assemble_host that share a schedule step): pairs p, p +
// stride, ... of their concatenation; a pair never straddles two ranges.
struct PairRanges {
  static constexpr bool kBatched = false, kSched = false, kStrip = false;
  RangeList r;
  int64_t p, stride;
  __device__ PairCursor next(int) {
    PairCursor c{0, 0, 0};
    int64_t q = p;
    for (int i = 0; i < r.n; i++) {
      const int64_t np = (r.count[i] + 1) / 2;
      if (q < np) {
        c.k0 = r.begin[i] + 2 * q;
        c.ne = (int)min((int64_t)2, r.begin[i] + r.count[i] - c.k0);
        break;
      }
      q -= np;
    }
    p += stride;
    return c;
  }
};

// One mesh, strips (HostPlan::strips) of up to kMaxRanges ranges of one launch: a warp
// takes strips p, p + stride, ... of their concatenation whole, two listed elements per
// step; the next strip's header is read one strip ahead.
struct StripRanges {
  static constexpr bool kBatched = false, kSched = false, kStrip = true;
  const Strip *strips;
  const RangeList &r;  // the kernel's __grid_constant__ parameter
  int64_t p, stride;
  Strip ahead{0, 0, 0, 0};
  int pos = 0, end = 0, flags = 0;
  __device__ void fetch() {
    ahead.count = 0;
    int64_t q = p;
#pragma unroll
    for (int i = 0; i < kMaxRanges; i++) {
      if (i >= r.n) break;
      if (q < r.count[i]) {
        const int4 v = __ldg(reinterpret_cast<const int4 *>(strips + r.begin[i] + q));
        ahead = Strip{v.x, v.y, v.z, v.w};
        break;
      }
      q -= r.count[i];
    }
    p += stride;
  }
  __device__ PairCursor next(int) {
    PairCursor c{0, 0, 0};
    int fl = kCarry;
    if (pos >= end) {
      if (ahead.count == 0) return c;
      pos = ahead.begin;
      end = ahead.begin + ahead.count;
      flags = ahead.flags;
      fl = (flags & kHalo);
      fetch();
    }
    c.k0 = pos;
    c.ne = min(2, end - pos);
    pos += c.ne;
    c.fl = fl | ((pos < end || (flags & kRight)) ? kRight : 0);
    return c;
  }
};

// Many meshes: the pairs of the warp's tiles -- tile w of the launch's list first, then
// the ones it pulls from the launch's queue (one atomic counter per launch; tiles hold
// even element counts except at the end of a colour range, so pairs never straddle
// tiles).  A warp asks for its next tile when it hands out the last pair of the one it
// has, no earlier: a small launch has about as many tiles as warps, and a warp that
// holds tiles in advance (as every warp did, from its start) leaves others idle.
struct PairQueue {
  static constexpr bool kBatched = true, kSched = false, kStrip = false;
  const Tile *tiles;
  int ntiles;
  int *counter;
  int warps;      // of the launch
  int idx;        // lane 0: the next tile
  int mesh = 0;
  int64_t pos = 0, tend = 0;
  bool done = false;
  __device__ PairCursor next(int lane) {
    PairCursor c{0, 0, 0};
    if (done) return c;
    if (pos >= tend) {
      const int t = __shfl_sync(0xffffffffu, idx, 0);
      if (t >= ntiles) {
        done = true;
        return c;
      }
      const int4 tl = __ldg(reinterpret_cast<const int4 *>(tiles + t));  // mesh, count, begin
      mesh = tl.x;
      pos = ((int64_t)tl.w << 32) | (uint32_t)tl.z;
      tend = pos + tl.y;
    }
    c.mesh = mesh;
    c.k0 = pos;
    c.ne = (int)min((int64_t)2, tend - pos);
    pos += 2;
    if (pos >= tend && lane == 0) idx = warps + atomicAdd(counter, 1);
    return c;
  }
};

__device__ __forceinline__ int ld_acquire_gpu(const int *p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Waits (one lane) until group g of the schedule has finished all its tiles.  The
// wait is bounded: after S.waitLimitNs (or 2^22 polls, should the timer stall) it
// counts itself in status[0] and returns, and once any wait has run out no later
// wait starts, so a launch whose dependencies can never be met still ends within
// about one limit.  The tile then writes regardless; the host reports the count.
__device__ __noinline__ void sched_wait(const SchedArgs *S, int g) {
  const int target = S->groupTiles[g] + (g == S->stallGroup ? 1 : 0);
  const int *done = S->status + 2 + g;
  if (ld_acquire_gpu(done) >= target) return;
  const unsigned long long t0 = global_ns();
  for (unsigned it = 0;; it++) {
    __nanosleep(100);
    if (ld_acquire_gpu(done) >= target) return;
    if (ld_acquire_gpu(S->status) != 0) return;
    if (global_ns() - t0 > (unsigned long long)S->waitLimitNs || it >= (1u << 22)) {
      atomicAdd(S->status, 1);
      return;
    }
  }
}

// Dependency-ordered: warps pull tiles in dispatch order from one counter
// (status[1]); one mesh, or (BATCHED) the tiles of many meshes of one order, each
// tile naming its mesh.  Before the first write of a tile's pairs the warp waits for the
// groups its tile's group depends on (acquire); after the last pair of a tile it
// completes its writes -- the asynchronous bulk reductions included -- and counts
// the tile in its group (release).  A warp holds at most the tiles it has pulled,
// in dispatch order, and every dependency of a tile is an earlier group, so the
// earliest unfinished tile can always proceed: no wait is circular, whether or not
// every CTA of the grid is resident.
template <bool BATCHED>
struct PairSchedT {
  static constexpr bool kBatched = BATCHED, kSched = true, kStrip = false;
  const SchedArgs *S;  // the kernel's __grid_constant__ parameter
  int tile = -1, held = -1, mesh = 0;
  int64_t pos = 0, tend = 0;
  bool done = false;
  __device__ PairCursor next(int lane) {
    PairCursor c{0, 0, 0};
    while (!done && pos >= tend) {
      int t = 0;
      if (lane == 0) t = atomicAdd(S->status + 1, 1);
      t = __shfl_sync(0xffffffffu, t, 0);
      if (t >= S->ntiles) {
        done = true;
      } else {
        const SchedTile tl = S->tiles[t];
        tile = t;
        if (BATCHED) mesh = tl.mesh;
        pos = tl.begin;
        tend = tl.begin + tl.count;
      }
    }
    if (done) return c;
    c.mesh = mesh;
    c.k0 = pos;
    c.ne = (int)min((int64_t)2, tend - pos);
    c.tile = tile;
    pos += 2;
    c.last = pos >= tend;
    return c;
  }
  __device__ void acquire(const PairCursor &c, int lane) {
    if (c.tile == held) return;
    held = c.tile;
    if (lane == 0) {
      const int g = S->tiles[c.tile].group;
      for (int i = S->depPtr[g]; i < S->depPtr[g + 1]; i++) sched_wait(S, S->deps[i]);
      __threadfence();
    }
    __syncwarp();
    // later bulk reductions (async proxy) are ordered after what the wait observed
    asm volatile("fence.proxy.async.global;" ::: "memory");
  }
  __device__ void release(const PairCursor &c, int lane) {
    asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    asm volatile("fence.proxy.async.global;" ::: "memory");
    __threadfence();
    __syncwarp();
    if (lane == 0) atomicAdd(S->status + 2 + S->tiles[c.tile].group, 1);
  }
};
using PairSched = PairSchedT<false>;

// One warp's assembly loop over the pairs its generator yields.  `single` is the
// single-mesh kernel's argument block; batched generators read meshes[c.mesh].
template <int P, int MODE, typename Gen>
__device__ __forceinline__ void frag_loop(unsigned char *smem, Gen &gen, const AsmArgs &single,
                                          const AsmArgs *__restrict__ meshes) {
  constexpr bool PLAN = (MODE & kPlan) != 0;
  constexpr bool NL = (MODE & kNL) != 0;
  constexpr bool B16 = (MODE & kB16) != 0;  // BF16x6 element stiffness
  using F = FragDims<P>;
  constexpr bool STRIP = Gen::kStrip;
  using L = FragLayout<P, !PLAN, NL, B16, (MODE & kJac) != 0>;
  constexpr int NN = F::NN, NQ = F::NQ, K4 = F::K4, QT = F::QT, NTM = F::NTM, NQP = F::NQP, PS = L::PS, CS = F::CS;
  constexpr bool EX = F::EX;  // node XN is in no tile
  constexpr int XN = NN - 1, NPAIR = F::NPAIR;
  constexpr int STG = L::CS;  // staged bytes per element: plan code record or map rows
  constexpr bool RES = (MODE & kRes) != 0, JAC = (MODE & kJac) != 0;
  constexpr bool RUNS = (P == 3);  // order 3: staged row runs, one bulk reduction per adjacent run
  static_assert(!NL || P < 4, "NONLINEAR strain: orders 2 and 3");
  static_assert(PLAN || !Gen::kBatched, "drop-in mode assembles one mesh");
  static_assert(!STRIP || (PLAN && JAC && !NL && P == kStripOrder), "strips: LINEAR Jacobians of plans, order 3");
  static_assert(!B16 || (!NL && P == 3), "BF16x6 stiffness: LINEAR, order 3");
  // LINEAR FP64: mu is folded into the gradients (G-hat carries sqrt|s mu|), so a block
  // is four FMAs of M with the one constant lam / mu.  (B16 keeps sqrt|s|: the BF16
  // split rounds the operands.)
  constexpr bool SCALED = !NL && !B16;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int e_ld = g >> 2, c_ld = g & 3;  // element / component this lane gathers
  const double2 *tabJ = reinterpret_cast<const double2 *>(smem + L::tabJ);
  const double2 *tabF = reinterpret_cast<const double2 *>(smem + L::tabF);
  const double2 *tabX = reinterpret_cast<const double2 *>(smem + L::tabX);
  const double *wqs = reinterpret_cast<const double *>(smem + L::wq);
  const double2 *csum = reinterpret_cast<const double2 *>(smem + L::csum);
  const double2 *tabB = reinterpret_cast<const double2 *>(smem + L::tabB);
  const uint32_t *tabR = reinterpret_cast<const uint32_t *>(smem + L::tabR);
  unsigned char *ws = smem + L::warps + warp * L::warp_bytes;
  double2 *WI0 = reinterpret_cast<double2 *>(ws + L::WI0);
  double2 *WI1 = reinterpret_cast<double2 *>(ws + L::WI1);
  double2 *WS0 = reinterpret_cast<double2 *>(ws + L::WS0);
  double2 *WS1 = reinterpret_cast<double2 *>(ws + L::WS1);
  double *SGs = reinterpret_cast<double *>(ws + L::SG);
  volatile double2 *MC = reinterpret_cast<volatile double2 *>(ws + L::MC);
  int *nid = reinterpret_cast<int *>(ws + L::NID);
  int *rb = reinterpret_cast<int *>(ws + L::RB);
  unsigned char *stage = ws + L::STAGE;
  double *redsW = reinterpret_cast<double *>(ws + L::REDS);  // staging slot s at redsW + 128 s
  double *ATs = reinterpret_cast<double *>(ws + L::AT);      // NONLINEAR tangent
  double crx = 0.0, cry = 0.0;                               // strips: carried residual rows
  // order 2, NONLINEAR: half of the lane's staging slots that the next blocks use.  It
  // turns with every bulk group and is kept from step to step, so the one group that a
  // put's wait leaves unfinished always reads the other half.
  [[maybe_unused]] int half = 0;
  [[maybe_unused]] bool scattered = false;  // drop-in, order 4: drop_issue_scattered adds the blocks

  // Mesh arguments are read through `mtab` (for one mesh, a pointer to the kernel
  // parameter).  At p = 4 it is laundered once per step: the compiler then reloads
  // the arguments where they are used instead of hoisting ~20 loop-invariant values
  // into registers for the whole loop, which pushed the residual + Jacobian kernel
  // into 400 bytes of spills (3.4 against 3.0 ms on a 512^2 mesh).  At p = 2 the
  // reloads cost more than they save (1.80 against 1.60 ms on the annulus).
  const AsmArgs *mtab = meshes;
  auto args = [&](const PairCursor &c) -> const AsmArgs & {
    if constexpr (Gen::kBatched) {
      return mtab[c.mesh];
    } else {
      return *mtab;
    }
  };
  // node ids (two pairs ahead) and coordinate/state values (one pair ahead)
  int nodeA[K4] = {}, nodeB[K4] = {}, rbB[K4] = {};
  double valB[K4] = {};
  // Lanes past the element's nodes or the pair's elements read the last ones again: their
  // values meet zero table entries, their ids are not kept.
  auto load_nodes = [&](const PairCursor &c, int *node) {
    if (c.ne <= 0) return;
    const int64_t k = c.k0 + (c.ne > 1 ? e_ld : 0);
    const int *src;
    if constexpr (PLAN) src = args(c).connList + k * NN;
    else src = args(c).conn + __ldg(args(c).connPtr + k);
#pragma unroll
    for (int ks = 0; ks < K4; ks++) node[ks] = __ldg(src + (4 * ks + 3 < NN ? 4 * ks + t : min(4 * ks + t, NN - 1)));
  };
  auto load_values = [&](const PairCursor &c, const int *node, double *val, int *rbv) {
    if (c.ne <= 0) return;
    const AsmArgs &M = args(c);
    const double *src = (c_ld < 2 ? M.coords : M.states) + (c_ld & 1);
#pragma unroll
    for (int ks = 0; ks < K4; ks++) {
      val[ks] = __ldg(src + 2 * (int64_t)node[ks]);
      if (PLAN && JAC) rbv[ks] = __ldg(M.rowp + node[ks]);
    }
  };
  auto stage_codes = [&](const PairCursor &c, int buf) {
    if (c.ne > 0) {
      unsigned char *dst = stage + buf * 2 * STG;
      if constexpr (PLAN && JAC) {
        const unsigned char *src = args(c).blockCode + c.k0 * CS;
#pragma unroll
        for (int i0 = 0; i0 < 2 * CS / 16; i0 += 32) {
          const int i = i0 + lane;
          if (i < c.ne * CS / 16) cp_async16(dst + 16 * i, src + 16 * i);
        }
      } else if constexpr (PLAN) {
        // the first-writer bytes of the residual rows alone
        constexpr int B0 = NN * NN / 16, NB = (NN * NN + NN - 1) / 16 - B0 + 1;
        const int e = lane / NB, i = B0 + lane - e * NB;
        if (e < c.ne) cp_async16(dst + e * CS + 16 * i, args(c).blockCode + (c.k0 + e) * CS + 16 * i);
      } else if constexpr (JAC && STG > 0) {
        // element map rows: 16-byte copies when a row set is a multiple of 16 bytes
        const int *src = args(c).map + c.k0 * NN * NN;
        if ((NN * NN) % 4 == 0 && (reinterpret_cast<uintptr_t>(src) & 15u) == 0) {
          for (int i = lane; i < c.ne * NN * NN / 4; i += 32) cp_async16(dst + 16 * i, src + 4 * i);
        } else {
          for (int i = lane; i < c.ne * NN * NN; i += 32) cp_async4(dst + 4 * i, src + i);
        }
      }
    }
    cp_async_commit();
  };

  // the mesh's constants of the quadrature stage and of the blocks (LINEAR)
  auto mesh_constants = [&](const AsmArgs &M) {
    if constexpr (!NL) {
      const double ts = SCALED ? M.t * M.mu : M.t;
      if (lane == 0) {
        MC->x = ts < 0.0 ? -sqrt(-ts) : sqrt(ts);
        MC->y = M.mu != 0.0 ? M.lam / M.mu : 0.0;
      }
      __syncwarp();
    }
  };
  if constexpr (NL && JAC && NQP > NQ) {  // the padded points' tangents: zero
    for (int i = lane; i < 2 * (NQP - NQ) * 16; i += 32)
      ATs[(i / ((NQP - NQ) * 16) * NQP + NQ) * 16 + i % ((NQP - NQ) * 16)] = 0.0;
  }
  int meshC = -1;
  // a grid launched after this one with programmatic serialization may start its CTAs
  // as this one's retire; it waits (griddepcontrol.wait) before it writes
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  bool dep_ready = false;
  PairCursor cur = gen.next(lane);
  PairCursor nxt = gen.next(lane);
  load_nodes(cur, nodeB);
  load_values(cur, nodeB, valB, rbB);
  load_nodes(nxt, nodeA);
  stage_codes(cur, 0);
  int buf = 0;

  for (; cur.ne > 0; buf ^= 1) {
    if constexpr (P == 4) asm volatile("" : "+l"(mtab));
    const int ne = cur.ne;
    const AsmArgs &M = args(cur);
    const double mu = M.mu, lam = M.lam, c11 = lam + 2.0 * mu;
    if (cur.mesh != meshC) {
      mesh_constants(M);
      meshC = cur.mesh;
    }
    // 0. commit this pair's gathered data
    double val[K4];
#pragma unroll
    for (int ks = 0; ks < K4; ks++) {
      val[ks] = valB[ks];
      const int a = 4 * ks + t;
      // nid by the lanes of component 0, rb by those of component 1
      if ((4 * ks + 3 < NN || a < NN) && c_ld < (PLAN && JAC ? 2 : 1))
        (c_ld == 0 ? nid : rb)[e_ld * NN + a] = c_ld == 0 ? nodeB[ks] : rbB[ks];
    }
    cp_async_wait_all();
    __syncwarp();
    // issue the following pairs' loads
    const PairCursor nn2 = gen.next(lane);
    stage_codes(nxt, buf ^ 1);
#pragma unroll
    for (int ks = 0; ks < K4; ks++) nodeB[ks] = nodeA[ks];
    load_values(nxt, nodeB, valB, rbB);
    load_nodes(nn2, nodeA);

    // 1. J stage: rows = quadrature points (8 per tile), columns = (element, component):
    //    lane (g, t) ends with component pair (x, y) (t even) or (u, v) (t odd) of element
    //    t/2 at points q = 8tm + g, derivative d of each.
    //    J = sum_a x_a dN_a cancels by ~h/|x| (1e-4 on a 10x10 square of 1024^2
    //    elements), so the coordinates enter relative to the element's node 0 (an
    //    exact subtraction for nearby values) and x_0 sum_a dN_a is added back: the
    //    same sum, evaluated without the cancellation.
    const int e_q = t >> 1, odd = t & 1;
    const double xq = __shfl_sync(0xffffffffu, val[0], 16 * e_q), yq = __shfl_sync(0xffffffffu, val[0], 16 * e_q + 4);
    const double xn0 = __shfl_sync(0xffffffffu, val[0], lane & ~3);
    const double x0 = c_ld < 2 ? xn0 : 0.0;
#pragma unroll
    for (int ks = 0; ks < K4; ks++) val[ks] -= x0;
    double cj[QT][2][2];  // [tile][d][component of the pair]
#pragma unroll
    for (int ks = 0; ks < K4; ks++)
#pragma unroll
      for (int tm = 0; tm < QT; tm++) {
        const double2 d = tabJ[(ks * QT + tm) * 32 + lane];
        if (ks == 0) {
          dmma_first(cj[tm][0][0], cj[tm][0][1], d.x, val[ks]);
          dmma_first(cj[tm][1][0], cj[tm][1][1], d.y, val[ks]);
        } else {
          dmma(cj[tm][0][0], cj[tm][0][1], d.x, val[ks]);
          dmma(cj[tm][1][0], cj[tm][1][1], d.y, val[ks]);
        }
      }

    // 2. per pair m of tiles: lanes t, t^1 exchange halves, so that each takes one
    //    quadrature point, q = 16m + 8 (t%2) + g of element t/2, with J and the
    //    reference gradient of the state
    unsigned negm = 0;  // lanes whose point has s (mu) < 0
#pragma unroll
    for (int m = 0; m < QT / 2; m++) {
      double jm[2][2], um[2][2];  // [d][component]
#pragma unroll
      for (int d = 0; d < 2; d++)
#pragma unroll
        for (int c = 0; c < 2; c++) {
          const double lo = cj[2 * m][d][c], hi = cj[2 * m + 1][d][c];
          const double r = __shfl_xor_sync(0xffffffffu, odd ? lo : hi, 1);
          jm[d][c] = odd ? r : lo;
          um[d][c] = odd ? hi : r;
        }
      const int q = 16 * m + 8 * odd + g;
      const int o = e_q * PS + L::slot(q);
      const bool in = 8 * F::QT == NQ || q < NQ;  // a point of the rule: the others store zeros
      const double2 cs = csum[q];
      const double j00 = fma(xq, cs.x, jm[0][0]), j01 = fma(xq, cs.y, jm[1][0]);
      const double j10 = fma(yq, cs.x, jm[0][1]), j11 = fma(yq, cs.y, jm[1][1]);
      const double g00 = um[0][0], g01 = um[1][0], g10 = um[0][1], g11 = um[1][1];
      const double det = j00 * j11 - j01 * j10;
      const bool keep = q < NQP;  // the point has a slot
      if constexpr (!JAC) {
        // residual alone: R_(a,i) = sum_q sum_d T_id dN_d(a, q) with T = s sigma J^-T, so
        // the nodal gradients are not formed: w t sigma adj(J)^T
        const double inv = in ? 1.0 / det : 0.0;
        const double ux0 = (g00 * j11 - g01 * j10) * inv, ux1 = (g01 * j00 - g00 * j01) * inv;
        const double uy0 = (g10 * j11 - g11 * j10) * inv, uy1 = (g11 * j00 - g10 * j01) * inv;
        double pxx, pxy, pyx, pyy;
        if constexpr (NL) {
          const double F[2][2] = {{1.0 + ux0, ux1}, {uy0, 1.0 + uy1}};
          const double e00 = 0.5 * (2.0 * ux0 + ux0 * ux0 + uy0 * uy0);
          const double e01 = 0.5 * (ux1 + uy0 + ux0 * ux1 + uy0 * uy1);
          const double e11 = 0.5 * (2.0 * uy1 + ux1 * ux1 + uy1 * uy1);
          const double tr = lam * (e00 + e11), s00 = 2.0 * mu * e00 + tr, s01 = 2.0 * mu * e01, s11 = 2.0 * mu * e11 + tr;
          pxx = F[0][0] * s00 + F[0][1] * s01, pxy = F[0][0] * s01 + F[0][1] * s11;
          pyx = F[1][0] * s00 + F[1][1] * s01, pyy = F[1][0] * s01 + F[1][1] * s11;
        } else {
          const double tr = lam * (ux0 + uy1);
          pxx = 2.0 * mu * ux0 + tr, pyy = 2.0 * mu * uy1 + tr;
          pxy = pyx = mu * (ux1 + uy0);
        }
        const double wt = wqs[q] * M.t;
        if (keep) {
          WI0[o] = make_double2(wt * (pxx * j11 - pxy * j01), wt * (pxy * j00 - pxx * j10));
          WI1[o] = make_double2(wt * (pyx * j11 - pyy * j01), wt * (pyy * j00 - pyx * j10));
        }
      } else if constexpr (NL) {
        const double inv = in ? 1.0 / det : 0.0;
        const double i00 = j11 * inv, i01 = -j01 * inv, i10 = -j10 * inv, i11 = j00 * inv;
        const double st = wqs[q] * det * M.t;
        const double rs = sqrt(fabs(st));
        const double sg = st < 0.0 ? -1.0 : 1.0;
        const double sw = sg * rs;
        const double uxx = g00 * i00 + g01 * i10, uxy = g00 * i01 + g01 * i11;
        const double uyx = g10 * i00 + g11 * i10, uyy = g10 * i01 + g11 * i11;
        // Green strain E = 1/2 (g + g^T + g^T g), S = 2 mu E + lam tr(E) I, first Piola
        // P = F S (F = I + g); tangent A_{il,kn} = delta_ik S_ln + mu F_in F_kl
        // + mu (F F^T)_ik delta_ln + lam F_il F_kn (element/FEKernels.h:286-315,
        // NONLINEAR), stored times sign(s) as [l][i][k][n]
        const double F[2][2] = {{1.0 + uxx, uxy}, {uyx, 1.0 + uyy}};
        const double e00 = 0.5 * (2.0 * uxx + uxx * uxx + uyx * uyx);
        const double e01 = 0.5 * (uxy + uyx + uxx * uxy + uyx * uyy);
        const double e11 = 0.5 * (2.0 * uyy + uxy * uxy + uyy * uyy);
        const double trE = e00 + e11;
        const double Sm[2][2] = {{2.0 * mu * e00 + lam * trE, 2.0 * mu * e01}, {2.0 * mu * e01, 2.0 * mu * e11 + lam * trE}};
        if (keep) {
          WI0[o] = make_double2(rs * i00, rs * i10);
          WI1[o] = make_double2(rs * i01, rs * i11);
          // (P-hat_x0, P-hat_y0), (P-hat_x1, P-hat_y1)
          WS0[o] = make_double2(sw * (F[0][0] * Sm[0][0] + F[0][1] * Sm[1][0]), sw * (F[1][0] * Sm[0][0] + F[1][1] * Sm[1][0]));
          WS1[o] = make_double2(sw * (F[0][0] * Sm[0][1] + F[0][1] * Sm[1][1]), sw * (F[1][0] * Sm[0][1] + F[1][1] * Sm[1][1]));
          double *at = ATs + (e_q * NQP + q) * 16;
          if (in) {
#pragma unroll
          for (int ll = 0; ll < 2; ll++)
#pragma unroll
            for (int ii2 = 0; ii2 < 2; ii2++)
#pragma unroll
              for (int kk = 0; kk < 2; kk++) {
                double v2[2];
#pragma unroll
                for (int nn = 0; nn < 2; nn++) {
                  const double bik = F[ii2][0] * F[kk][0] + F[ii2][1] * F[kk][1];
                  double v = mu * F[ii2][nn] * F[kk][ll] + lam * F[ii2][ll] * F[kk][nn];
                  if (ii2 == kk) v += Sm[ll][nn];
                  if (ll == nn) v += mu * bik;
                  v2[nn] = sg * v;
                }
                *reinterpret_cast<double2 *>(at + ll * 8 + ii2 * 4 + kk * 2) = make_double2(v2[0], v2[1]);
              }
          }
        }
      } else {
        // s = w det t, J^-1 = adj(J) / det: sqrt|s| J^-1 = +-c adj(J) with
        // c = sqrt|w t| / sqrt|det| (the sign leaves every product of two gradients
        // alone), grad u = g adj(J) / det, and s sigma G = (+-c sigma(g adj(J))) (c adj(J) dN):
        // one reciprocal square root instead of a division and a square root.
        // A singular point (det = 0) gives NaN.
        const double2 mc = make_double2(MC->x, MC->y);
        const double r = det != 0.0 ? rsqrt(fabs(det)) : __longlong_as_double(0x7ff8000000000000LL);
        const double c = in ? wqs[q] * fabs(mc.x) * r : 0.0;
        const bool ng = in && e_q < ne && (det < 0.0) != (mc.x < 0.0);
        const double sg = ng ? -1.0 : 1.0;
        const double cw = sg * c;
        const double uxx = g00 * j11 - g01 * j10, uxy = g01 * j00 - g00 * j01;
        const double uyx = g10 * j11 - g11 * j10, uyy = g11 * j00 - g10 * j01;
        const double m1 = SCALED ? 1.0 : mu, lt = (SCALED ? mc.y : lam) * (uxx + uyy);
        const double sxy = cw * (m1 * (uxy + uyx));
        if (keep) {
          WI0[o] = make_double2(c * j11, -(c * j10));
          WI1[o] = make_double2(-(c * j01), c * j00);
          WS0[o] = make_double2(cw * fma(2.0 * m1, uxx, lt), sxy);
          WS1[o] = make_double2(sxy, cw * fma(2.0 * m1, uyy, lt));
          SGs[e_q * NQP + q] = sg;
        }
        if constexpr (SCALED) negm |= __ballot_sync(0xffffffffu, ng);
      }
    }
    __syncwarp();

    // the warp's first writes wait for the grid launched before this one (programmatic
    // dependent launch: its gathers and element arithmetic ran while that grid drained)
    if (!dep_ready) {
      asm volatile("griddepcontrol.wait;" ::: "memory");
      dep_ready = true;
    }
    if constexpr (Gen::kSched) gen.acquire(cur, lane);
    const Out O{M.mat, M.residual, stage + buf * 2 * STG, rb, reinterpret_cast<const int *>(stage + buf * 2 * STG)};
    // the 2x2 block of M (LINEAR: the plane-stress combination, divided by mu where
    // the gradients carry sqrt mu; NONLINEAR: the product is the block)
    const double lm = SCALED ? MC->y : 0.0, lm2 = lm + 2.0;
    auto block = [&](double mxx, double mxy, double myx, double myy, double &kxx, double &kxy, double &kyx, double &kyy) {
      if constexpr (NL) {
        kxx = mxx, kxy = mxy, kyx = myx, kyy = myy;
      } else if constexpr (SCALED) {
        kxx = fma(lm2, mxx, myy);
        kxy = fma(lm, mxy, myx);
        kyx = fma(lm, myx, mxy);
        kyy = fma(lm2, myy, mxx);
      } else {
        kxx = c11 * mxx + mu * myy, kxy = lam * mxy + mu * myx;
        kyx = lam * myx + mu * mxy, kyy = c11 * myy + mu * mxx;
      }
    };
    // order 3: the staged blocks of an element leave as row runs, two per lane, after one
    // proxy fence; nothing to do when no lane staged any (a launch of first contributors)
    auto issue_runs = [&](const Out &out, int el, bool staged) {
      if (!__any_sync(0xffffffffu, staged)) return;
      if (PLAN && !STRIP && el > 0) pair_first_landed();
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (PLAN && !STRIP && el > 0) pair_first_visible();
#pragma unroll
      for (int u = 0; u < 2; u++) if constexpr (RUNS) frag_issue_run<P, PLAN>(out, el, tabR[lane + 32 * u], redsW);
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    };
    // all k-steps; the form with the points' signs is rarely run and stays rolled
    auto kstep_all = [&](auto &kstep, bool neg) {
      if (SCALED && neg) {
        kstep(0, std::true_type{}, std::true_type{});
#pragma unroll 1
        for (int ks = 1; ks < K4; ks++) kstep(ks, std::false_type{}, std::true_type{});
      } else {
        kstep(0, std::true_type{}, std::false_type{});
#pragma unroll
        for (int ks = 1; ks < K4; ks++) kstep(ks, std::false_type{}, std::false_type{});
      }
    };
    // strips: the right edge's residual rows go to the next element's left edge
    auto residual_carry = [&](double &sx, double &sy, bool in) {
      if (in && g < 2) sx += crx, sy += cry;
      crx = __shfl_down_sync(0xffffffffu, sx, 24);
      cry = __shfl_down_sync(0xffffffffu, sy, 24);
    };
    if constexpr (!JAC) {
      // residual alone: rows (element, component) m = g%4 (twice), columns the nodes of a
      // tile, k = points: R_(a,i) = sum_(q,d) T_id(q) dN_d(a, q); the node outside the tiles
      // on the FP64 pipe.  Forming the nodal gradients first, as the Jacobian does, took
      // 8 shared loads and 16 FMAs per k-step and element instead of this pair's 3 loads
      // and 4 MMAs (order 3; residual 600 x 590 order 3 248 -> 160 us, 800 x 512 order
      // 2 239 -> 152, 256^2 order 4 170 -> 102).
      const double2 *Ts = ((g & 1) ? WI1 : WI0) + ((g >> 1) & 1) * PS;
      double c[NTM][2], xr = 0.0;
#pragma unroll
      for (int ks = 0; ks < K4; ks++) {
        const double2 tv = Ts[L::slot(4 * ks) + t];
#pragma unroll
        for (int T = 0; T < NTM; T++) {
          const double2 d = tabF[(ks * NTM + T) * 32 + lane];
          if (ks == 0) dmma_first(c[T][0], c[T][1], tv.x, d.x);
          else dmma(c[T][0], c[T][1], tv.x, d.x);
          dmma(c[T][0], c[T][1], tv.y, d.y);
        }
        if constexpr (EX) {
          const double2 d = tabX[4 * ks + t];
          xr = fma(tv.x, d.x, fma(tv.y, d.y, xr));
        }
      }
      // lane (g, t) holds component i = g%2 of nodes 8T + t, 8T + 4 + t; lanes g, g^1 swap,
      // and each keeps node 8T + 4i + t; the copies g >= 4 take the odd tiles (the last
      // one of orders 2 and 4: node XN)
      const int i = g & 1, e = (g >> 1) & 1, up = g >> 2;
      if constexpr (EX) {
        xr += __shfl_xor_sync(0xffffffffu, xr, 1);
        xr += __shfl_xor_sync(0xffffffffu, xr, 2);
      }
      constexpr int NR = (NTM + (EX ? 1 : 0) + 1) / 2;
      double sx[NR], sy[NR];
      double *dst[NR];
      bool act[NR], first[NR];
#pragma unroll
      for (int x = 0; x < NR; x++) {
        const int T = 2 * x;
        double v0 = c[T][0], v1 = c[T][1];
        if (up) {
          v0 = T + 1 < NTM ? c[T + 1 < NTM ? T + 1 : T][0] : xr;
          v1 = T + 1 < NTM ? c[T + 1 < NTM ? T + 1 : T][1] : xr;
        }
        const double r = __shfl_xor_sync(0xffffffffu, i ? v0 : v1, 4);
        sx[x] = i ? r : v0;
        sy[x] = i ? v1 : r;
        const bool xl = EX && T + 1 == NTM && up;
        const int a = xl ? XN : F::node(8 * (T + up) + 4 * i + t);
        act[x] = e < ne && (!xl || (i == 0 && t == 0));
        dst[x] = M.residual + 2 * (int64_t)nid[e * NN + a];
        first[x] = PLAN && O.codes[e * CS + NN * NN + a];
      }
      if constexpr (PLAN) {
        // pair layout: the first element's rows before the second's
#pragma unroll
        for (int x = 0; x < NR; x++) residual_put(dst[x], act[x] && e == 0, first[x], sx[x], sy[x]);
        __syncwarp();
#pragma unroll
        for (int x = 0; x < NR; x++) residual_put(dst[x], act[x] && e == 1, first[x], sx[x], sy[x]);
      } else {
#pragma unroll
        for (int x = 0; x < NR; x++) residual_put(dst[x], act[x], false, sx[x], sy[x]);
      }
    } else {
      const int pa = 4 * (g & 1) + (g >> 1);  // pi(g)
      // nodes of a lane's row (8T + pi(g)) and column (8T + 4h + t) positions (FragDims::node,
      // drop-in)
      constexpr bool PERM = P == 4 && !PLAN;
      const int p0 = !PERM ? pa : 5 * (g & 1) + (g >> 1);
      const int p2 = !PERM ? 16 + pa : ((g & 1) ? 5 * (g >> 1) + 4 : 20 + (g >> 1));
      auto row_node = [&](int T) { return T == 2 ? p2 : (PERM ? 10 : 8) * T + p0; };
      auto col_node = [&](int T, int h) {
        return !PERM ? 8 * T + 4 * h + t : T == 2 ? (h ? 5 * t + 4 : 20 + t) : 5 * (2 * T + h) + t;
      };
      for (int el = 0; el < ne; el++) {
        // Strips: the blocks of an edge's nodes among themselves and their residual rows
        // belong to the element right of it; lanes (g = 6, 7; t = 3) hold exactly those
        // blocks of an element's right edge, lanes (g = 0, 1; t = 0) its left edge's, in
        // the same order.
        const bool halo = STRIP && el == 0 && (cur.fl & kHalo);
        const bool cin = STRIP && (el > 0 || (cur.fl & kCarry));
        const bool right = STRIP && (el + 1 < ne || (cur.fl & kRight));
        // The give lanes stage their blocks like blocks to add (which the codes say they are
        // not, so no run takes them), the take lanes of the next element add them from
        // there; a halo stages everything and issues nothing.
        const bool give = STRIP && right && (lane & ~4) == 27, take = STRIP && cin && (lane & ~4) == 0;
        const uint32_t m80 = give || halo ? 0u : 0x80u;
        // pair layout: the first element's residual writes before the second's
        if (PLAN && !STRIP && el > 0) __syncwarp();
        if constexpr (B16) {
          // BF16x6 element stiffness: M_ij = sum_q s G_i(q, a) G_j(q, b) as m16n8k16
          // products (k = quadrature points 0-15; rows a and columns b of the two node
          // tiles, a = 8h + pi(g) and b = 8h' + pi(n)); each FP64 operand is split into
          // three BF16 parts and six part products accumulate in FP32 (hi*hi, hi*mid,
          // mid*hi, hi*lo, lo*hi, mid*mid: ~FP32 accuracy; the two-way BF16x3 split
          // leaves ~4e-6 relative error in K).  Lane (g, t) holds the values of the
          // quadrature points q_k = 2t + (k & 1) + 8 (k >> 1) of nodes 8h + pi(g).
          double gv[2][4][2];  // [i][k][h]: G-hat_i(q_k, 8h + pi(g)) = sqrt|s| (dN J^-1)_i
          double sgk[4];
          double rx[2] = {0.0, 0.0}, ry[2] = {0.0, 0.0};
#pragma unroll
          for (int k = 0; k < 4; k++) {
            const int q = 2 * t + (k & 1) + 8 * (k >> 1);
            const int o = el * PS + L::slot(q);
            const bool qv = q < NQ;
            const double2 w0 = qv ? WI0[o] : make_double2(0.0, 0.0), w1 = qv ? WI1[o] : make_double2(0.0, 0.0);
            sgk[k] = qv ? SGs[el * NQP + q] : 0.0;
            double2 s0 = make_double2(0.0, 0.0), s1 = make_double2(0.0, 0.0);
            if (RES && qv) {
              s0 = WS0[o];
              s1 = WS1[o];
            }
#pragma unroll
            for (int h = 0; h < 2; h++) {
              const double2 d = tabB[(2 * k + h) * 32 + lane];
              gv[0][k][h] = fma(w0.x, d.x, w0.y * d.y);
              gv[1][k][h] = fma(w1.x, d.x, w1.y * d.y);
              if constexpr (RES) {
                rx[h] = fma(gv[0][k][h], s0.x, fma(gv[1][k][h], s1.x, rx[h]));
                ry[h] = fma(gv[0][k][h], s0.y, fma(gv[1][k][h], s1.y, ry[h]));
              }
            }
          }
          if constexpr (RES) {
            // sum over the four lanes t of node 8h + pi(g); lane t = h writes it
#pragma unroll
            for (int h = 0; h < 2; h++) {
              rx[h] += __shfl_xor_sync(0xffffffffu, rx[h], 1);
              ry[h] += __shfl_xor_sync(0xffffffffu, ry[h], 1);
              rx[h] += __shfl_xor_sync(0xffffffffu, rx[h], 2);
              ry[h] += __shfl_xor_sync(0xffffffffu, ry[h], 2);
            }
            const int a = 8 * t + pa;
            double sx = t ? rx[1] : rx[0], sy = t ? ry[1] : ry[0];
            if constexpr (STRIP) residual_carry(sx, sy, cin);
            {
              const bool act = t < 2 && !halo && !(right && g >= 6);
              const int an = t < 2 ? a : 0;
              residual_put(M.residual + 2 * (int64_t)nid[el * NN + an], act, PLAN && O.codes[el * CS + NN * NN + an], sx, sy);
            }
          }
          if constexpr (JAC) {
            // split operands: B[part][j][h][r] (column node 8h + pi(g)), A = sign(s) B
            // packed as row fragments: A[part][i][r] (rows pi(g), 8 + pi(g))
            uint32_t pb[3][2][4][2];  // [part][i][k][h] raw BF16 bits
#pragma unroll
            for (int i = 0; i < 2; i++)
#pragma unroll
              for (int k = 0; k < 4; k++)
#pragma unroll
                for (int h = 0; h < 2; h++) split3(gv[i][k][h], pb[0][i][k][h], pb[1][i][k][h], pb[2][i][k][h]);
            uint32_t Af[3][2][4], Bf[3][2][2][2];
#pragma unroll
            for (int pt = 0; pt < 3; pt++)
#pragma unroll
              for (int i = 0; i < 2; i++) {
                auto sv = [&](int k, int h) { return pb[pt][i][k][h] ^ (sgk[k] < 0.0 ? 0x8000u : 0u); };
                Af[pt][i][0] = sv(0, 0) | (sv(1, 0) << 16);
                Af[pt][i][1] = sv(0, 1) | (sv(1, 1) << 16);
                Af[pt][i][2] = sv(2, 0) | (sv(3, 0) << 16);
                Af[pt][i][3] = sv(2, 1) | (sv(3, 1) << 16);
#pragma unroll
                for (int h = 0; h < 2; h++) {
                  Bf[pt][i][h][0] = pb[pt][i][0][h] | (pb[pt][i][1][h] << 16);
                  Bf[pt][i][h][1] = pb[pt][i][2][h] | (pb[pt][i][3][h] << 16);
                }
              }
            float acc[2][2][2][4];  // [i][j][h (column tile)][c]
#pragma unroll
            for (int i = 0; i < 2; i++)
#pragma unroll
              for (int j = 0; j < 2; j++)
#pragma unroll
                for (int h = 0; h < 2; h++) {
#pragma unroll
                  for (int c = 0; c < 4; c++) acc[i][j][h][c] = 0.0f;
                  // smallest terms first
                  bmma(acc[i][j][h], Af[2][i], Bf[0][j][h][0], Bf[0][j][h][1]);
                  bmma(acc[i][j][h], Af[0][i], Bf[2][j][h][0], Bf[2][j][h][1]);
                  bmma(acc[i][j][h], Af[1][i], Bf[1][j][h][0], Bf[1][j][h][1]);
                  bmma(acc[i][j][h], Af[1][i], Bf[0][j][h][0], Bf[0][j][h][1]);
                  bmma(acc[i][j][h], Af[0][i], Bf[1][j][h][0], Bf[1][j][h][1]);
                  bmma(acc[i][j][h], Af[0][i], Bf[0][j][h][0], Bf[0][j][h][1]);
                }
            // lane (g, t): c = 2 r + u holds M_ij[a = 8r + pi(g)][b = 8h + 4u + t]: whole
            // 2x2 blocks, four consecutive columns across the lanes t.  Blocks to add go
            // to the staging slots of the FP64 layout (node-tile pair (r, h) = (TA, TB);
            // the pair (1, 0) is the transposed half of (0, 1)) and leave as row runs.
            asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
            __syncwarp();
            uint32_t allfirst = 0x80u;
#pragma unroll
            for (int r = 0; r < 2; r++)
#pragma unroll
              for (int h = 0; h < 2; h++)
#pragma unroll
                for (int u = 0; u < 2; u++) {
                  const int a = 8 * r + pa, b = 8 * h + 4 * u + t, c = 2 * r + u;
                  {
                    const double mxx = acc[0][0][h][c], mxy = acc[0][1][h][c];
                    const double myx = acc[1][0][h][c], myy = acc[1][1][h][c];
                    double kxx, kxy, kyx, kyy;
                    block(mxx, mxy, myx, myy, kxx, kxy, kyx, kyy);
                    const int sl = (r == 1 && h == 0) ? frag_slot(1, g & 1, 1) : frag_slot(r + h, u, 0);
                    const int pos = (r == 1 && h == 0) ? 8 * (g >> 1) + 4 * u + t : 4 * g + t;
                    double *stg = redsW + 128 * sl + 4 * pos;
                    if (take) {  // from lane + 27's staging position
                      const double *cs = stg + 4 * (r == 1 && h == 0 ? 8 * 3 + 3 : 27);
                      kxx += cs[0], kxy += cs[1];
                      kyx += cs[2], kyy += cs[3];
                    }
                    if constexpr (STRIP) __syncwarp();
                    if constexpr (PLAN) {
                      const uint32_t code = O.codes[el * CS + a * NN + b];
                      frag_put_row<0>(O.mat + 4 * (int64_t)O.rbase[el * NN + a], code, m80,
                                      (unsigned)__cvta_generic_to_shared(stg), kxx, kxy, kyx, kyy);
                      allfirst &= code;
                    } else {
                      allfirst &= frag_put<P, PLAN>(O, el, a, b, 0, true, m80, kxx, kxy, kyx, kyy, stg);
                    }
                  }
                }
            issue_runs(O, el, !halo && (allfirst & 0x80u) == 0);
          }
          continue;
        }
        // 3.-5. quadrature k-steps outermost: per step each lane forms its fragments
        // G-hat_i(q = 4ks + t, a = 8T + pi(g)), adds its residual partials and issues
        // the 4 NPAIR independent stiffness MMAs of the pass's node-tile pairs.  Orders 2
        // and 4: the node outside the tiles has its row and column on the FP64 pipe, each
        // lane forming its G-hat(q, XN) itself (order 4: 168 instead of the 280 MMAs of a
        // fourth node tile).
        // whether a point of this element has s (mu) < 0 (inverted element or negative
        // thickness or modulus): only then do the A fragments take the points' signs
        const bool neg = SCALED && (negm & (el ? 0xccccccccu : 0x33333333u)) != 0;
        // a strip's halo: the blocks and residual rows of its right edge alone, as one 8 x 8
        // tile (rows and columns (edge node, component)) instead of twelve; short strips of
        // small meshes are half halos (43 x 37 18.4 -> 14.5 us, 128^2 53.3 -> 50.0, 512^2
        // 547 -> 537)
        if constexpr (STRIP && !B16) {
          if (halo) {
            const int ay = g >> 1, i = g & 1;
            double c0, c1, px = 0.0, py = 0.0;
#pragma unroll
            for (int ks = 0; ks < K4; ks++) {
              const int o = el * PS + L::slot(4 * ks) + t;
              const double2 w = i ? WI1[o] : WI0[o];
              const double2 d = tabF[(ks * NTM + (ay >> 1)) * 32 + 4 * (6 + (ay & 1)) + t];
              const double fr = fma(w.x, d.x, w.y * d.y);
              if constexpr (RES) {
                const double2 sj = i ? WS1[o] : WS0[o];  // (S-hat_xi, S-hat_yi)
                px = fma(fr, sj.x, px);
                py = fma(fr, sj.y, py);
              }
              const double af = neg ? SGs[el * NQP + 4 * ks + t] * fr : fr;
              if (ks == 0) dmma_first(c0, c1, af, fr);
              else dmma(c0, c1, af, fr);
            }
            // lane (g, t): (M_i0, M_i1) of edge nodes (ay, by = t); the other row from lane^4
            const double o0 = __shfl_xor_sync(0xffffffffu, c0, 4), o1 = __shfl_xor_sync(0xffffffffu, c1, 4);
            const double mxx = i ? o0 : c0, mxy = i ? o1 : c1, myx = i ? c0 : o0, myy = i ? c1 : o1;
            double kxx, kxy, kyx, kyy;
            block(mxx, mxy, myx, myy, kxx, kxy, kyx, kyy);
            // to the give lanes' staging positions, where the next element takes them
            asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
            __syncwarp();
            if ((ay >> 1) <= (t >> 1)) {
              const int k = (ay >> 1) + (t >> 1);  // pairs (0, 0), (0, 1), (1, 1)
              const int sl = k == 0 ? (t & 1) : k == 1 ? 2 + 2 * (t & 1) : 6 + (t & 1);
              double2 *x = reinterpret_cast<double2 *>(redsW + 128 * sl + 4 * (27 + 4 * (ay & 1)));
              x[i] = i ? make_double2(kyx, kyy) : make_double2(kxx, kxy);
            }
            if constexpr (RES) {
#pragma unroll
              for (int x = 1; x <= 4; x <<= 1) {
                px += __shfl_xor_sync(0xffffffffu, px, x);
                py += __shfl_xor_sync(0xffffffffu, py, x);
              }
              const int src = 8 * (2 * (t >> 1) + (g & 1));
              crx = __shfl_sync(0xffffffffu, px, src);
              cry = __shfl_sync(0xffffffffu, py, src);
            }
            __syncwarp();
            continue;
          }
        }
        auto pass = [&](auto passc) {
          constexpr int PASS = decltype(passc)::value;
          // fragments of tiles [0, NF); residual slots: tiles RT0 and RT1, NTM = node XN;
          // xs[0], xs[1]: M[XN][tile] (orders 2: tile 0; 4: tiles 0, 1 | 2) and M[XN][XN]
          constexpr int NF = PASS ? 3 : (NTM == 1 ? 1 : 2);
          [[maybe_unused]] constexpr int RT0 = PASS ? 2 : 0, RT1 = PASS || NTM == 1 ? NTM : 1;
          double acc[NPAIR][4][2];
          [[maybe_unused]] double rp[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
          [[maybe_unused]] double xs[2][4] = {{0.0, 0.0, 0.0, 0.0}, {0.0, 0.0, 0.0, 0.0}};
          auto kstep = [&](int ks, auto firstc, auto negc) {
            constexpr bool FIRST = decltype(firstc)::value, NEG = decltype(negc)::value;
            const int o = el * PS + L::slot(4 * ks) + t;
            const double2 w0 = WI0[o], w1 = WI1[o];
            double fr[NTM][2];
#pragma unroll
            for (int T = 0; T < NF; T++) {
              const double2 d = tabF[(ks * NTM + T) * 32 + lane];
              fr[T][0] = fma(w0.x, d.x, w0.y * d.y);
              fr[T][1] = fma(w1.x, d.x, w1.y * d.y);
            }
            [[maybe_unused]] double h0 = 0.0, h1 = 0.0;  // G-hat(q, XN)
            if constexpr (EX) {
              const double2 d = tabX[4 * ks + t];
              h0 = fma(w0.x, d.x, w0.y * d.y);
              h1 = fma(w1.x, d.x, w1.y * d.y);
            }
            if constexpr (RES) {
              // LINEAR: the stress is symmetric, S-hat_yx = S-hat_xy
              const double2 s0 = WS0[o];
              const double s1y = WS1[o].y, s1x = NL ? WS1[o].x : s0.y;
#pragma unroll
              for (int x = 0; x < 2; x++) {
                const int T = x ? RT1 : RT0;
                const double f0 = T == NTM ? h0 : fr[T < NTM ? T : 0][0], f1 = T == NTM ? h1 : fr[T < NTM ? T : 0][1];
                rp[x][0] = fma(f0, s0.x, fma(f1, s1x, rp[x][0]));
                rp[x][1] = fma(f0, s0.y, fma(f1, s1y, rp[x][1]));
              }
            }
            if constexpr (NL) {
              // K_ik[a][b] = sum over (q, l) of G-hat_l(q, a) B_ikl(q, b),
              // B_ikl = sign(s) sum_n A_{il,kn} G-hat_n(q, b): 4 (i, k) x 2 (l) MMAs per pair
              const double *at = ATs + (el * NQP + 4 * ks + t) * 16;
#pragma unroll
              for (int ll = 0; ll < 2; ll++) {
                double C[2][2][2];  // [i][k][n]
#pragma unroll
                for (int j = 0; j < 4; j++) {
                  const double2 v = *reinterpret_cast<const double2 *>(at + ll * 8 + 2 * j);
                  C[j >> 1][j & 1][0] = v.x;
                  C[j >> 1][j & 1][1] = v.y;
                }
#pragma unroll
                for (int k = 0; k < NPAIR; k++) {
                  const int TA = F::ta(PASS, k), TB = F::tb(PASS, k);
#pragma unroll
                  for (int ik = 0; ik < 4; ik++) {
                    const double bv = fma(C[ik >> 1][ik & 1][0], fr[TB][0], C[ik >> 1][ik & 1][1] * fr[TB][1]);
                    if (FIRST && ll == 0) dmma_first(acc[k][ik][0], acc[k][ik][1], fr[TA][ll], bv);
                    else dmma(acc[k][ik][0], acc[k][ik][1], fr[TA][ll], bv);
                  }
                }
                if constexpr (EX) {
                  const double hl = ll ? h1 : h0;
#pragma unroll
                  for (int ik = 0; ik < 4; ik++) {
                    xs[0][ik] = fma(hl, fma(C[ik >> 1][ik & 1][0], fr[0][0], C[ik >> 1][ik & 1][1] * fr[0][1]), xs[0][ik]);
                    xs[1][ik] = fma(hl, fma(C[ik >> 1][ik & 1][0], h0, C[ik >> 1][ik & 1][1] * h1), xs[1][ik]);
                  }
                }
              }
            }
            if constexpr (!NL) {
              double sg = 1.0;
              if constexpr (NEG) sg = SGs[el * NQP + 4 * ks + t];
              double af[NTM][2];  // A fragments: times the point's sign
#pragma unroll
              for (int T = 0; T < NF; T++) af[T][0] = NEG ? sg * fr[T][0] : fr[T][0], af[T][1] = NEG ? sg * fr[T][1] : fr[T][1];
#pragma unroll
              for (int k = 0; k < NPAIR; k++) {
                const int TA = F::ta(PASS, k), TB = F::tb(PASS, k);
#pragma unroll
                for (int ij = 0; ij < 4; ij++) {
                  if constexpr (FIRST) dmma_first(acc[k][ij][0], acc[k][ij][1], af[TA][ij >> 1], fr[TB][ij & 1]);
                  else dmma(acc[k][ij][0], acc[k][ij][1], af[TA][ij >> 1], fr[TB][ij & 1]);
                }
              }
              if constexpr (EX) {
                const double s0 = NEG ? sg * h0 : h0, s1 = NEG ? sg * h1 : h1;
#pragma unroll
                for (int x = 0; x < 2; x++) {
                  const int T = x ? RT1 : RT0;
                  const double f0 = T == NTM ? h0 : fr[T < NTM ? T : 0][0], f1 = T == NTM ? h1 : fr[T < NTM ? T : 0][1];
                  xs[x][0] = fma(s0, f0, xs[x][0]);
                  xs[x][1] = fma(s0, f1, xs[x][1]);
                  xs[x][2] = fma(s1, f0, xs[x][2]);
                  xs[x][3] = fma(s1, f1, xs[x][3]);
                }
              }
            }
          };
          // drop-in order 4: the lane's map entries of this pass, in flight during the products
          int mp[L::DR ? L::DR / 32 : 1][4];
          if constexpr (!PLAN && P == 4) {
            const int *row = M.map + (cur.k0 + el) * (int64_t)(NN * NN);
#pragma unroll
            for (int x = 0; x < L::DR / 32; x++) {
              const uint32_t e = tabR[PASS * L::DR + 32 * x + lane];
              const int o = e == 0xffffffffu ? 0 : e & 0x3ff, n = e == 0xffffffffu ? 0 : (e >> 11) & 3;
#pragma unroll
              for (int j = 0; j < 4; j++) mp[x][j] = __ldg(row + o + (j <= n ? j : 0) * (e >> 10 & 1 ? 5 : 1));
            }
          }
          kstep_all(kstep, neg);
          // residual: sum over the four lanes t of a node (reduce-scatter over the two slots)
          [[maybe_unused]] const int Tm = t >> 1, To = Tm ^ 1;
          if constexpr (RES) {
            double sx = (Tm ? rp[1][0] : rp[0][0]) + __shfl_xor_sync(0xffffffffu, To ? rp[1][0] : rp[0][0], 2);
            double sy = (Tm ? rp[1][1] : rp[0][1]) + __shfl_xor_sync(0xffffffffu, To ? rp[1][1] : rp[0][1], 2);
            sx += __shfl_xor_sync(0xffffffffu, sx, 1);
            sy += __shfl_xor_sync(0xffffffffu, sy, 1);
            if constexpr (STRIP) residual_carry(sx, sy, cin);
            const int an = Tm == 0 ? row_node(RT0) : (RT1 == NTM ? XN : row_node(RT1));
            const bool act = (t & 1) == 0 && (Tm == 0 || RT1 < NTM || g == 0) && !halo && !(right && g >= 6);
            residual_put(M.residual + 2 * (int64_t)nid[el * NN + an], act, PLAN && O.codes[el * CS + NN * NN + an], sx, sy);
          }
          if constexpr (RUNS) {
            // acc becomes the blocks (xx, xy, yx, yy)
#pragma unroll
            for (int k = 0; k < NPAIR; k++)
#pragma unroll
              for (int h = 0; h < 2; h++) {
                double kxx, kxy, kyx, kyy;
                block(acc[k][0][h], acc[k][1][h], acc[k][2][h], acc[k][3][h], kxx, kxy, kyx, kyy);
                acc[k][0][h] = kxx, acc[k][1][h] = kxy, acc[k][2][h] = kyx, acc[k][3][h] = kyy;
              }
            // every lane's previous bulk reads of the staging slots are complete
            asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
            __syncwarp();
            double *stg = redsW + 4 * lane;  // direct blocks: position 4g + t of their slot
            if constexpr (STRIP) {
              if (take) {
#pragma unroll
                for (int k = 0; k < NPAIR; k++)
#pragma unroll
                  for (int h = 0; h < 2; h++) {
                    const double2 *cs = reinterpret_cast<const double2 *>(stg + 128 * frag_slot(k, h, 0) + 4 * 27);
                    acc[k][0][h] += cs[0].x, acc[k][1][h] += cs[0].y;
                    acc[k][2][h] += cs[1].x, acc[k][3][h] += cs[1].y;
                  }
              }
              __syncwarp();
            }
            uint32_t allfirst = 0x80u;
            if constexpr (PLAN && !NL) {
              // the lane's code bytes and row addresses first: rows pi(g) and 8 + pi(g) hold
              // its direct blocks, rows 8 + 4h + t the transposed ones of pair (0, 1)
              const uint8_t *rec = O.codes + el * CS;
              const int *rbe = O.rbase + el * NN;
              uint32_t cd[NPAIR][2], ct[2];
#pragma unroll
              for (int k = 0; k < NPAIR; k++)
#pragma unroll
                for (int h = 0; h < 2; h++) cd[k][h] = rec[pa * NN + t + (k == 2 ? 8 * NN : 0) + (k == 0 ? 0 : 8) + 4 * h];
#pragma unroll
              for (int h = 0; h < 2; h++) ct[h] = rec[t * NN + pa + (8 + 4 * h) * NN];
              const double *r0 = O.mat + 4 * (int64_t)rbe[pa], *r1 = O.mat + 4 * (int64_t)rbe[8 + pa];
              const double *rt0 = O.mat + 4 * (int64_t)rbe[8 + t], *rt1 = O.mat + 4 * (int64_t)rbe[12 + t];
              const unsigned sd = (unsigned)__cvta_generic_to_shared(stg);
              const unsigned st = (unsigned)__cvta_generic_to_shared(redsW + 4 * (8 * t + pa));
              auto direct = [&](auto kc, auto hc) {
                constexpr int k = decltype(kc)::value, h = decltype(hc)::value;
                frag_put_row<1024 * frag_slot(k, h, 0)>(k == 2 ? r1 : r0, cd[k][h], m80, sd, acc[k][0][h], acc[k][1][h],
                                                        acc[k][2][h], acc[k][3][h]);
                allfirst &= cd[k][h];
              };
              direct(IC<0>{}, IC<0>{});
              direct(IC<0>{}, IC<1>{});
              direct(IC<1>{}, IC<0>{});
              direct(IC<1>{}, IC<1>{});
              frag_put_row<1024 * frag_slot(1, 0, 1)>(rt0, ct[0], m80, st, acc[1][0][0], acc[1][2][0], acc[1][1][0], acc[1][3][0]);
              frag_put_row<1024 * frag_slot(1, 1, 1)>(rt1, ct[1], m80, st, acc[1][0][1], acc[1][2][1], acc[1][1][1], acc[1][3][1]);
              direct(IC<2>{}, IC<0>{});
              direct(IC<2>{}, IC<1>{});
              allfirst &= ct[0] & ct[1];
            } else {
#pragma unroll
              for (int k = 0; k < NPAIR; k++) {
                {
                  const int TA = F::ta(0, k), TB = F::tb(0, k);
                  const int a = 8 * TA + pa;
#pragma unroll
                  for (int h = 0; h < 2; h++) {
                    const int b = 8 * TB + 4 * h + t;
                    const double kxx = acc[k][0][h], kxy = acc[k][1][h], kyx = acc[k][2][h], kyy = acc[k][3][h];
                    // NONLINEAR diagonal tiles: (a, b) for a <= b and, for a < b, its exact
                    // transpose (b, a) at the staging position the (b, a) lane would use
                    const bool diag = NL && TA == TB;
                    allfirst &= frag_put<P, PLAN>(O, el, a, b, 0, !diag || a <= b, m80, kxx, kxy, kyx, kyy,
                                                  stg + 128 * frag_slot(k, h, 0));
                    if (TA < TB) {
                      allfirst &= frag_put<P, PLAN>(O, el, a, b, 1, true, m80, kxx, kxy, kyx, kyy,
                                                    redsW + 128 * frag_slot(k, h, 1) + 4 * (8 * t + pa));
                    } else if (diag) {
                      const int xb = b - 8 * TA, xa = a - 8 * TA;  // pi(g') = xb; a = 8T + 4h' + t'
                      const int gb = 2 * (xb & 3) + (xb >> 2);
                      allfirst &= frag_put<P, PLAN>(O, el, a, b, 1, a < b, m80, kxx, kxy, kyx, kyy,
                                                    redsW + 128 * frag_slot(k, xa >> 2, 0) + 4 * (4 * gb + (xa & 3)));
                    }
                  }
                }
              }
            }
            issue_runs(O, el, !halo && (allfirst & 0x80u) == 0);
          }
          // stiffness blocks, orders 2 and 4: lane (g, t) writes (8TA + pi(g), 8TB + 4h + t) of
          // each pair and, for TA < TB, its transpose (NONLINEAR diagonal pairs: for a <= b,
          // and the exact transpose); then the row and column of node XN: of the two slots of
          // xs, lanes t/2 = x take slot x, t even (XN, a), t odd its transpose.  First stores
          // go out at once, the blocks to add are staged and leave FL at a time after one
          // proxy fence, as one bulk group.  Fewer fences and groups, against waiting for the
          // group before: order 4 takes all four slots at a time (256^2 486 us; two from each
          // half of the slots in turn 503), order 2 an element's three (512 x 2048 annulus 1178
          // us, from two sets of slots in turn 1184), its NONLINEAR blocks two (500 x 512 770 us,
          // four 808).
          if constexpr (EX && PLAN) {
            constexpr int FL = P == 4 ? 4 : (NL ? 2 : 3), HALF = FL == 2 ? 2 : 0;
            double *reds = redsW + 4 * lane;
            double *dst[FL];
            bool add[FL];
            int n = 0;
            auto flush = [&](int m) {
              bool any = false;
#pragma unroll
              for (int x = 0; x < FL; x++) any = any || (x < m && add[x]);
              if (!__any_sync(0xffffffffu, any)) return;
              if (el > 0) pair_first_landed();
              asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
              if (el > 0) {
                __syncwarp();
                pair_first_visible();
              }
#pragma unroll
              for (int x = 0; x < FL; x++)
                if (x < m) bulk_add_block(dst[x], reds + 128 * (HALF * half + x), add[x]);
              asm volatile("cp.async.bulk.commit_group;" ::: "memory");
              half ^= 1;
            };
            auto put = [&](int r, int c, bool act, double v0, double v1, double v2, double v3) {
              // the bulk reads of the slots used next are complete
              if (n == 0) {
                if constexpr (HALF) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
                else asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
              }
              add[n] = frag_put_block<P>(O, el, r, c, act, v0, v1, v2, v3, reds + 128 * (HALF * half + n), dst[n]);
              if (++n == FL) {
                flush(FL);
                n = 0;
              }
            };
            double kxx, kxy, kyx, kyy;
#pragma unroll
            for (int k = 0; k < NPAIR; k++)
#pragma unroll
              for (int h = 0; h < 2; h++) {
                const int TA = F::ta(PASS, k), TB = F::tb(PASS, k);
                const int a = row_node(TA), b = col_node(TB, h);
                const bool diag = NL && TA == TB;
                block(acc[k][0][h], acc[k][1][h], acc[k][2][h], acc[k][3][h], kxx, kxy, kyx, kyy);
                put(a, b, !diag || a <= b, kxx, kxy, kyx, kyy);
                if (TA < TB || diag) put(b, a, !diag || a < b, kxx, kyx, kxy, kyy);
              }
            double xv[4];
#pragma unroll
            for (int c = 0; c < 4; c++) {
              xv[c] = (Tm ? xs[1][c] : xs[0][c]) + __shfl_xor_sync(0xffffffffu, To ? xs[1][c] : xs[0][c], 2);
              xv[c] += __shfl_xor_sync(0xffffffffu, xv[c], 1);
            }
            block(xv[0], xv[1], xv[2], xv[3], kxx, kxy, kyx, kyy);
            const int xa = Tm == 0 ? row_node(RT0) : (RT1 == NTM ? XN : row_node(RT1));
            const bool tr = t & 1;
            put(tr ? xa : XN, tr ? XN : xa, Tm == 0 || RT1 < NTM || (g == 0 && !tr), kxx, tr ? kyx : kxy, tr ? kxy : kyx, kyy);
            if (n) flush(n);
          }
          // drop-in, orders 2 and 4: every block is staged (drop_run), and each lane adds its
          // entries' stretches of adjacent blocks.  A reduction of 32 bytes per block bounded
          // these launches: 200 x 201 order 4, with the element kernel's FP64 atomics 987 us
          // for the driver's two calls, with 32-byte reductions 1082, with stretches 648;
          // 501 x 500 order 2 597 -> 496
          if constexpr (EX && !PLAN) {
            asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
            __syncwarp();
            auto stage_at = [&](int block, double v0, double v1, double v2, double v3) {
              double2 *x = reinterpret_cast<double2 *>(redsW + 4 * block);
              x[0] = make_double2(v0, v1);
              x[1] = make_double2(v2, v3);
            };
            double kxx, kxy, kyx, kyy;
            int sl = 0;  // slots in the order of drop_run
#pragma unroll
            for (int k = 0; k < NPAIR; k++)
#pragma unroll
              for (int h = 0; h < 2; h++) {
                const int TA = F::ta(PASS, k), TB = F::tb(PASS, k);
                block(acc[k][0][h], acc[k][1][h], acc[k][2][h], acc[k][3][h], kxx, kxy, kyx, kyy);
                if constexpr (NL) {  // order 2: (a, b) for a <= b and its exact transpose
                  const int b = 4 * h + t;
                  if (pa <= b) stage_at(32 * h + 4 * g + t, kxx, kxy, kyx, kyy);
                  if (pa < b) stage_at(32 * (pa >> 2) + 4 * (2 * (b & 3) + (b >> 2)) + (pa & 3), kxx, kyx, kxy, kyy);
                } else {
                  stage_at(32 * sl++ + 4 * g + t, kxx, kxy, kyx, kyy);
                  if (TA < TB) stage_at(32 * sl++ + 8 * t + pa, kxx, kyx, kxy, kyy);
                }
              }
            double xv[4];
#pragma unroll
            for (int c = 0; c < 4; c++) {
              xv[c] = (Tm ? xs[1][c] : xs[0][c]) + __shfl_xor_sync(0xffffffffu, To ? xs[1][c] : xs[0][c], 2);
              xv[c] += __shfl_xor_sync(0xffffffffu, xv[c], 1);
            }
            block(xv[0], xv[1], xv[2], xv[3], kxx, kxy, kyx, kyy);
            constexpr int SX = 32 * (P == 2 ? 2 : PASS ? 10 : 8), NM = RT1 < NTM ? 16 : 8;
            const bool tr = t & 1, xd = RT1 == NTM && Tm == 1;  // xd: the diagonal block's lanes
            if (!xd || (g == 0 && !tr))
              stage_at(SX + (xd ? 2 * NM : (tr ? NM : 0) + 8 * Tm + pa), kxx, tr ? kyx : kxy, tr ? kxy : kyx, kyy);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            auto entry = [&](int x, int (&m)[4], int &src) {
              const uint32_t e = tabR[PASS * L::DR + 32 * x + lane];
              src = 4 * (e >> 13 & 0x1ff);
              if constexpr (P == 4) {
#pragma unroll
                for (int j = 0; j < 4; j++) m[j] = mp[x][j];
              } else {
                const int *row = O.map + el * NN * NN + (e == 0xffffffffu ? 0 : e & 0x3ff);
#pragma unroll
                for (int j = 0; j < 4; j++) m[j] = row[j < (int)((e >> 11) & 3) + 1 ? j : 0];
              }
              return e == 0xffffffffu ? 0 : (int)((e >> 11) & 3) + 1;
            };
            int m[4], src;
            if (P == 4 && PASS == 0) {
              const int n = entry(0, m, src);
              scattered = 2 * __popc(__ballot_sync(0xffffffffu, drop_apart(m, n))) > __popc(__ballot_sync(0xffffffffu, n == 4));
            }
            if (P == 4 && scattered) {
#pragma unroll
              for (int x = 0; x < L::DR / 32; x++) {
                const int n = entry(x, m, src);
                drop_issue_scattered(O.mat, m, n, redsW, src, lane);
              }
            } else {
#pragma unroll
              for (int x = 0; x < L::DR / 32; x++) {
                const int n = entry(x, m, src);
                drop_issue(O.mat, m, n, redsW + src);
              }
            }
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          }
        };
        pass(IC<0>{});
        if constexpr (F::NPASS == 2) {
          // keeps each pass's table loads inside the pass (registers)
          asm volatile("" ::: "memory");
          pass(IC<1>{});
        }
      }
    }
    if constexpr (Gen::kSched) {
      if (cur.last) gen.release(cur, lane);
    }
    __syncwarp();
    cur = nxt;
    nxt = nn2;
  }
  cp_async_wait_all();
  // bulk reductions complete (shared-memory reads and global writes) before exit
  asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

// One mesh: plan mode, list positions [A.begin, A.begin + A.count) of one colour;
// drop-in mode, elements [A.begin, A.begin + A.count) through the reference map.  split: the
// pairs (PairStride), for order-4 plans the elements of a unit (UnitStride).
template <int P, int MODE>
__global__ void __launch_bounds__(32 * FragDims<P>::WARPS, FEM_FRAG_MINB) frag_kernel(const __grid_constant__ AsmArgs A,
                                                                                             int split) {
  extern __shared__ __align__(16) unsigned char smem[];
  frag_prologue<P, MODE>(smem);
  const int warp = threadIdx.x >> 5;
  if constexpr (P == 4 && (MODE & kPlan) != 0) {
    UnitStride gen{A.begin, A.begin + A.count, (int64_t)blockIdx.x * FragDims<P>::WARPS + warp,
                   (int64_t)gridDim.x * FragDims<P>::WARPS, split};
    frag_loop<P, MODE>(smem, gen, A, &A);
  } else {
    PairStride gen{A.begin, blockIdx.x * FragDims<P>::WARPS + warp, gridDim.x * FragDims<P>::WARPS, (unsigned)split,
                   (unsigned)A.count - (unsigned)split};
    frag_loop<P, MODE>(smem, gen, A, &A);
  }
}

// One mesh, several list-position ranges (plan mode).
template <int P, int MODE>
__global__ void __launch_bounds__(32 * FragDims<P>::WARPS, FEM_FRAG_MINB)
    frag_ranges_kernel(const __grid_constant__ AsmArgs A, const RangeList R) {
  extern __shared__ __align__(16) unsigned char smem[];
  frag_prologue<P, MODE>(smem);
  const int warp = threadIdx.x >> 5;
  PairRanges gen{R, (int64_t)blockIdx.x * FragDims<P>::WARPS + warp, (int64_t)gridDim.x * FragDims<P>::WARPS};
  frag_loop<P, MODE>(smem, gen, A, &A);
}

// One mesh, strips of several ranges of its strip list (plan mode, LINEAR Jacobian).  The
// order-3 assembly is bound by its writes: a probe that stores every block once at its
// real address took 568 us for 512^2 in the pair layout's order (four colours, x-neighbours
// written in different launches: lines leave L2 half written), 466 us with each element row
// in one launch (linear fill: 378-400).  512^2: 668 -> 537 us, 1024^2 2.63 -> 2.18 ms.
template <int P, int MODE>
__global__ void __launch_bounds__(32 * FragDims<P>::WARPS, FEM_FRAG_MINB)
    frag_strip_kernel(const __grid_constant__ AsmArgs A, const __grid_constant__ RangeList R,
                      const Strip *__restrict__ strips) {
  extern __shared__ __align__(16) unsigned char smem[];
  frag_prologue<P, MODE>(smem);
  const int warp = threadIdx.x >> 5;
  StripRanges gen{strips, R, (int64_t)blockIdx.x * FragDims<P>::WARPS + warp, (int64_t)gridDim.x * FragDims<P>::WARPS};
  gen.fetch();
  frag_loop<P, MODE>(smem, gen, A, &A);
}

// One mesh, all colours in one dependency-ordered persistent launch (plan mode).
template <int P, int MODE>
__global__ void __launch_bounds__(32 * FragDims<P>::WARPS, FEM_FRAG_MINB)
    frag_sched_kernel(const __grid_constant__ AsmArgs A, const __grid_constant__ SchedArgs S) {
  extern __shared__ __align__(16) unsigned char smem[];
  frag_prologue<P, MODE>(smem);
  PairSched gen{&S};
  frag_loop<P, MODE>(smem, gen, A, &A);
}

// Many meshes of one order, all colours in one dependency-ordered persistent launch:
// the tiles of every (mesh, colour) group, colours outermost, each group waiting
// for its mesh's previous colour.
template <int P, int MODE>
__global__ void __launch_bounds__(32 * FragDims<P>::WARPS, FEM_FRAG_MINB)
    frag_batched_sched_kernel(const AsmArgs *__restrict__ meshes, const __grid_constant__ SchedArgs S) {
  extern __shared__ __align__(16) unsigned char smem[];
  frag_prologue<P, MODE>(smem);
  PairSchedT<true> gen{&S};
  frag_loop<P, MODE>(smem, gen, meshes[0], meshes);
}

// Many meshes of one order (one colour each): warps pull tiles from the launch's queue.
template <int P, int MODE>
__global__ void __launch_bounds__(32 * FragDims<P>::WARPS, FEM_FRAG_MINB)
    frag_batched_kernel(const AsmArgs *__restrict__ meshes, const Tile *__restrict__ tiles, int ntiles, int *counter) {
  extern __shared__ __align__(16) unsigned char smem[];
  frag_prologue<P, MODE>(smem);
  constexpr int W = FragDims<P>::WARPS;
  PairQueue gen{tiles, ntiles, counter, (int)gridDim.x * W, (int)blockIdx.x * W + (int)(threadIdx.x >> 5)};
  frag_loop<P, MODE>(smem, gen, meshes[0], meshes);
}

// A launch whose grid may begin while the kernel before it on the stream drains
// (programmatic dependent launch): consecutive colour or band launches of one
// assembly overlap one's tail with the next one's table setup, gathers and element
// arithmetic; the fragment kernel waits for the previous grid before it writes.
template <typename K, typename... Args>
cudaError_t pdl_launch(K kernel, int grid, int nt, size_t smem, cudaStream_t s, const Args &...args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)nt);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// chained: the launch follows this assembly's previous fragment-kernel launch on the
// stream (a later colour or band), whose outputs are the only ones it may read
// early, so it may start as that one drains; a first launch follows the caller's
// work, which may have produced its inputs, and launches in stream order.
// single: the listed elements are independent (not the pair layout's), so that a small
// launch may take them one by one.
template <int P, int MODE>
int launch_frag_p(const AsmArgs &a, cudaStream_t s, bool chained, bool single) {
  using F = FragDims<P>;
  constexpr int NT = 32 * F::WARPS;
  auto kernel = frag_kernel<P, MODE>;
  const size_t smem = FragLayout<P, (MODE & kPlan) == 0, (MODE & kNL) != 0, (MODE & kB16) != 0, (MODE & kJac) != 0>::total;
  LaunchInfo li;
  int st = launch_info(kernel, NT, smem, li);
  if (st) return st;
  // Order-3 drop-in Jacobian (every block added through the element map, one launch
  // whose elements share blocks): two CTAs per SM.  At 1024^2 the kernel took 3.90 ms
  // with two resident CTAs per SM against 4.35 ms with three (the bulk reductions of
  // more warps contend in L2); at order 2 (four CTAs) halving them cost 2.04 -> 3.46
  // ms on the 512x2048 annulus, so it keeps its occupancy.
  const int perSm =
      (P == 3 && (MODE & kPlan) == 0 && (MODE & kJac) != 0) ? std::min(li.grid_per_sm, 2) : li.grid_per_sm;
  const int64_t cap = (int64_t)perSm * li.num_sms;
  // A launch whose elements all find a warp of their own takes one per warp instead of a
  // pair: the warp's step is what the launch takes, and one element's stiffness and writes
  // are most of half of it (33 x 31 order 4 63.5 -> 38.9 us, order 3 NONLINEAR
  // 44.1 -> 22.6; order 2, bound by its four launches, 18.5 -> 18.4), and so does the last
  // wave of the warps as far as its elements go around (order-4 drop-in 90 x 89 122 -> 112
  // us, order-3 drop-in 80 x 79 34.8 -> 32.8, order-3 NONLINEAR plan 90 x 89 63.5 -> 58.4;
  // not in order-4 plans, see UnitStride).
  // Not the residual alone, where both elements of a step are rows of the same products
  // (90 x 89 in the colour layout, order 2 one / two per warp 20.5 / 14.4, order 3 22.0 / 16.4).
  [[maybe_unused]] const int64_t per = cap * F::WARPS, left = a.count % (2 * per);
  int split;
  int64_t units;
  if constexpr (P == 4 && (MODE & kPlan) != 0) {
    split = single && (MODE & kJac) != 0 && a.count <= per ? 1 : 2;
    units = (a.count + split - 1) / split;
  } else {
    const int64_t pairs =
        single && (MODE & kJac) != 0 ? (a.count - left) / 2 + std::max<int64_t>(left - per, 0) : a.count / 2;
    split = (int)pairs;
    units = a.count - pairs;
  }
  const int64_t need = (units + F::WARPS - 1) / F::WARPS;
  const int grid = (int)(need < cap ? need : cap);
  if (grid <= 0) return FEM_SUCCESS;
  cudaError_t err;
  if (chained) {
    err = pdl_launch(kernel, grid, NT, smem, s, a, split);
  } else {
    kernel<<<grid, NT, smem, s>>>(a, split);
    err = cudaGetLastError();
  }
  if (err != cudaSuccess) return cuda_fail(err, "frag_kernel launch");
  return FEM_SUCCESS;
}

template <int P, int MODE>
int launch_frag_ranges_p(const AsmArgs &a, const RangeList &r, cudaStream_t s, bool chained) {
  using F = FragDims<P>;
  constexpr int NT = 32 * F::WARPS;
  auto kernel = frag_ranges_kernel<P, MODE>;
  const size_t smem = FragLayout<P, false, (MODE & kNL) != 0, (MODE & kB16) != 0, (MODE & kJac) != 0>::total;
  LaunchInfo li;
  int st = launch_info(kernel, NT, smem, li);
  if (st) return st;
  int64_t pairs = 0;
  for (int i = 0; i < r.n; i++) pairs += (r.count[i] + 1) / 2;
  const int64_t need = (pairs + F::WARPS - 1) / F::WARPS;
  const int64_t cap = (int64_t)li.grid_per_sm * li.num_sms;
  const int grid = (int)(need < cap ? need : cap);
  if (grid <= 0) return FEM_SUCCESS;
  cudaError_t err;
  if (chained) {
    err = pdl_launch(kernel, grid, NT, smem, s, a, r);
  } else {
    kernel<<<grid, NT, smem, s>>>(a, r);
    err = cudaGetLastError();
  }
  if (err != cudaSuccess) return cuda_fail(err, "frag_ranges_kernel launch");
  return FEM_SUCCESS;
}

template <int P, int MODE>
int launch_frag_strips_p(const AsmArgs &a, const RangeList &r, const Strip *strips, cudaStream_t s, bool chained) {
  using F = FragDims<P>;
  constexpr int NT = 32 * F::WARPS;
  auto kernel = frag_strip_kernel<P, MODE>;
  const size_t smem = FragLayout<P, false, (MODE & kNL) != 0, (MODE & kB16) != 0, (MODE & kJac) != 0>::total;
  LaunchInfo li;
  int st = launch_info(kernel, NT, smem, li);
  if (st) return st;
  int64_t n = 0;
  for (int i = 0; i < r.n; i++) n += r.count[i];
  const int64_t need = (n + F::WARPS - 1) / F::WARPS;
  const int64_t cap = (int64_t)li.grid_per_sm * li.num_sms;
  const int grid = (int)(need < cap ? need : cap);
  if (grid <= 0) return FEM_SUCCESS;
  cudaError_t err;
  if (chained) {
    err = pdl_launch(kernel, grid, NT, smem, s, a, r, strips);
  } else {
    kernel<<<grid, NT, smem, s>>>(a, r, strips);
    err = cudaGetLastError();
  }
  if (err != cudaSuccess) return cuda_fail(err, "frag_strip_kernel launch");
  return FEM_SUCCESS;
}

template <int P, int MODE>
int launch_frag_batched_p(const AsmArgs *meshes, const Tile *tiles, int ntiles, int *counter, cudaStream_t s) {
  using F = FragDims<P>;
  constexpr int NT = 32 * F::WARPS;
  auto kernel = frag_batched_kernel<P, MODE>;
  const size_t smem = FragLayout<P, false, false, (MODE & kB16) != 0>::total;
  LaunchInfo li;
  int st = launch_info(kernel, NT, smem, li);
  if (st) return st;
  const int64_t need = (ntiles + F::WARPS - 1) / F::WARPS;
  const int64_t cap = (int64_t)li.grid_per_sm * li.num_sms;
  const int grid = (int)(need < cap ? need : cap);
  if (grid <= 0) return FEM_SUCCESS;
  kernel<<<grid, NT, smem, s>>>(meshes, tiles, ntiles, counter);
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) return cuda_fail(err, "frag_batched_kernel launch");
  return FEM_SUCCESS;
}

template <int P, int MODE>
int launch_frag_batched_sched_p(const AsmArgs *meshes, const SchedArgs &sa, cudaStream_t s) {
  using F = FragDims<P>;
  constexpr int NT = 32 * F::WARPS;
  auto kernel = frag_batched_sched_kernel<P, MODE>;
  const size_t smem = FragLayout<P, false, false, (MODE & kB16) != 0>::total;
  LaunchInfo li;
  int st = launch_info(kernel, NT, smem, li);
  if (st) return st;
  const int64_t need = ((int64_t)sa.ntiles + F::WARPS - 1) / F::WARPS;
  const int64_t cap = (int64_t)li.grid_per_sm * li.num_sms;
  const int grid = (int)(need < cap ? need : cap);
  if (grid <= 0) return FEM_SUCCESS;
  kernel<<<grid, NT, smem, s>>>(meshes, sa);
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) return cuda_fail(err, "frag_batched_sched_kernel launch");
  return FEM_SUCCESS;
}

template <int P, int MODE>
int launch_frag_sched_p(const AsmArgs &a, const SchedArgs &sa, cudaStream_t s) {
  using F = FragDims<P>;
  constexpr int NT = 32 * F::WARPS;
  auto kernel = frag_sched_kernel<P, MODE>;
  const size_t smem = FragLayout<P, false, (MODE & kNL) != 0, (MODE & kB16) != 0, (MODE & kJac) != 0>::total;
  LaunchInfo li;
  int st = launch_info(kernel, NT, smem, li);
  if (st) return st;
  const int64_t need = ((int64_t)sa.ntiles + F::WARPS - 1) / F::WARPS;
  const int64_t cap = (int64_t)li.grid_per_sm * li.num_sms;
  const int grid = (int)(need < cap ? need : cap);
  if (grid <= 0) return FEM_SUCCESS;
  kernel<<<grid, NT, smem, s>>>(a, sa);
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) return cuda_fail(err, "frag_sched_kernel launch");
  return FEM_SUCCESS;
}

template <int MODE>
int launch_frag_mode(int order, const AsmArgs &a, cudaStream_t s, bool chained, bool single) {
  switch (order) {
    case 2:
      if constexpr ((MODE & kB16) != 0) return fail(FEM_ERR_INVALID_ORDER, "fragment kernel, BF16x6: order 2");
      else return launch_frag_p<2, MODE>(a, s, chained, single);
    case 3: return launch_frag_p<3, MODE>(a, s, chained, single);
    case 4:
      if constexpr ((MODE & (kNL | kB16)) != 0) return fail(FEM_ERR_INVALID_ORDER, "fragment kernel, mode %d: order 4", MODE);
      else return launch_frag_p<4, MODE>(a, s, chained, single);
    default: return fail(FEM_ERR_INVALID_ORDER, "fragment kernel: order %d", order);
  }
}

}  // namespace dev

// MIXED, LINEAR, order 3: the Jacobian's element stiffness runs as BF16x6 tensor-core
// products (kB16); everything else of the kernel stays FP64.  Order 2 pads 9 nodes and
// 9 quadrature points to 16 in both operands and ran slower than FP64 (2.0 against
// 1.4 ms on the 512x2048 annulus), so MIXED keeps the FP64 kernel there.
bool b16_stiffness(int order, int precision, int strain) {
  return precision == FEM_PRECISION_MIXED && strain == FEM_STRAIN_LINEAR && order == 3;
}

// FP64, LINEAR: orders 2 to 4 in every mode (one 512^2 order-4 mesh took 3.00 ms with the
// element kernel and 2.03 with this one; drop-in, 400 x 390 with its residual call 3.80
// against 2.40 ms).  Plans and batches must run the same kernel (a mesh's batched result
// equals its single-mesh plan result bit for bit).
// MIXED at orders 2 and 3 also runs this kernel (faster than the FP32 element
// products there: 3.1 against 3.8 ms at 1024^2 p = 3): at order 3 with the element
// stiffness as BF16x6 tensor-core products (b16_stiffness), at order 2 in FP64 (the
// FP64 result, as order-1 row assembly gives).  MIXED at order 4 keeps the FP32 element
// kernel, whose results its callers have.
bool frag_supported(int order, int precision, int strain) {
  if (strain == FEM_STRAIN_NONLINEAR) return precision == FEM_PRECISION_FP64 && (order == 2 || order == 3);
  if (strain != FEM_STRAIN_LINEAR) return false;
  if (precision == FEM_PRECISION_MIXED) return order == 2 || order == 3;
  if (precision != FEM_PRECISION_FP64) return false;
  return order >= 2 && order <= 4;
}

int launch_frag(int order, int precision, int mode, const dev::AsmArgs &a, cudaStream_t s, int strain, bool chained,
                bool single) {
  using namespace dev;
  if (strain == FEM_STRAIN_NONLINEAR) mode |= kNL;
  if (b16_stiffness(order, precision, strain) && (mode & kJac)) mode |= kB16;
  switch (mode) {
    case kPlan | kJac | kB16: return launch_frag_mode<kPlan | kJac | kB16>(order, a, s, chained, single);
    case kPlan | kRes | kJac | kB16: return launch_frag_mode<kPlan | kRes | kJac | kB16>(order, a, s, chained, single);
    case kJac | kB16: return launch_frag_mode<kJac | kB16>(order, a, s, chained, single);
    case kRes | kJac | kB16: return launch_frag_mode<kRes | kJac | kB16>(order, a, s, chained, single);
    case kPlan | kRes: return launch_frag_mode<kPlan | kRes>(order, a, s, chained, single);
    case kPlan | kJac: return launch_frag_mode<kPlan | kJac>(order, a, s, chained, single);
    case kPlan | kRes | kJac: return launch_frag_mode<kPlan | kRes | kJac>(order, a, s, chained, single);
    case kRes: return launch_frag_mode<kRes>(order, a, s, chained, single);
    case kJac: return launch_frag_mode<kJac>(order, a, s, chained, single);
    case kRes | kJac: return launch_frag_mode<kRes | kJac>(order, a, s, chained, single);
    case kNL | kPlan | kRes: return launch_frag_mode<kNL | kPlan | kRes>(order, a, s, chained, single);
    case kNL | kPlan | kJac: return launch_frag_mode<kNL | kPlan | kJac>(order, a, s, chained, single);
    case kNL | kPlan | kRes | kJac: return launch_frag_mode<kNL | kPlan | kRes | kJac>(order, a, s, chained, single);
    case kNL | kRes: return launch_frag_mode<kNL | kRes>(order, a, s, chained, single);
    case kNL | kJac: return launch_frag_mode<kNL | kJac>(order, a, s, chained, single);
    case kNL | kRes | kJac: return launch_frag_mode<kNL | kRes | kJac>(order, a, s, chained, single);
    default: return fail(FEM_ERR_INVALID_ARGUMENT, "fragment kernel: mode %d", mode);
  }
}

int launch_frag_ranges(int order, int precision, int mode, const dev::AsmArgs &a, const dev::RangeList &r,
                       cudaStream_t s, int strain, bool chained) {
  using namespace dev;
  if (strain == FEM_STRAIN_NONLINEAR) mode |= kNL;
  if (b16_stiffness(order, precision, strain) && (mode & kJac)) mode |= kB16;
  auto go = [&](auto mc) -> int {
    constexpr int M = decltype(mc)::value;
    switch (order) {
      case 2:
        if constexpr ((M & kB16) != 0) return fail(FEM_ERR_INVALID_ORDER, "fragment kernel, BF16x6: order 2");
        else return launch_frag_ranges_p<2, M>(a, r, s, chained);
      case 3: return launch_frag_ranges_p<3, M>(a, r, s, chained);
      case 4:
        if constexpr ((M & (kNL | kB16)) != 0) return fail(FEM_ERR_INVALID_ORDER, "fragment kernel, mode %d: order 4", M);
        else return launch_frag_ranges_p<4, M>(a, r, s, chained);
      default: return fail(FEM_ERR_INVALID_ORDER, "fragment kernel: order %d", order);
    }
  };
  switch (mode) {
    case kPlan | kRes: return go(IC<kPlan | kRes>{});
    case kPlan | kRes | kJac: return go(IC<kPlan | kRes | kJac>{});
    case kPlan | kRes | kJac | kB16: return go(IC<kPlan | kRes | kJac | kB16>{});
    case kNL | kPlan | kRes: return go(IC<kNL | kPlan | kRes>{});
    case kNL | kPlan | kRes | kJac: return go(IC<kNL | kPlan | kRes | kJac>{});
    default: return fail(FEM_ERR_INVALID_ARGUMENT, "fragment kernel, ranges: mode %d", mode);
  }
}

// Strips: LINEAR Jacobians of order-kStripOrder plans.
int launch_frag_strips(int order, int precision, int mode, const dev::AsmArgs &a, const dev::RangeList &r,
                       const dev::Strip *strips, cudaStream_t s, int strain, bool chained) {
  using namespace dev;
  if (order != kStripOrder || strain != FEM_STRAIN_LINEAR)
    return fail(FEM_ERR_INVALID_ORDER, "fragment kernel, strips: order %d, strain %d", order, strain);
  if (b16_stiffness(order, precision, strain) && (mode & kJac)) mode |= kB16;
  switch (mode) {
    case kPlan | kJac: return launch_frag_strips_p<kStripOrder, kPlan | kJac>(a, r, strips, s, chained);
    case kPlan | kRes | kJac: return launch_frag_strips_p<kStripOrder, kPlan | kRes | kJac>(a, r, strips, s, chained);
    case kPlan | kJac | kB16: return launch_frag_strips_p<kStripOrder, kPlan | kJac | kB16>(a, r, strips, s, chained);
    case kPlan | kRes | kJac | kB16:
      return launch_frag_strips_p<kStripOrder, kPlan | kRes | kJac | kB16>(a, r, strips, s, chained);
    default: return fail(FEM_ERR_INVALID_ARGUMENT, "fragment kernel, strips: mode %d", mode);
  }
}

int launch_frag_sched(int order, int precision, int mode, const dev::AsmArgs &a, const dev::SchedArgs &sa,
                      cudaStream_t s, int strain) {
  using namespace dev;
  if (strain == FEM_STRAIN_NONLINEAR) mode |= kNL;
  if (b16_stiffness(order, precision, strain) && (mode & kJac)) mode |= kB16;
  auto go = [&](auto mc) -> int {
    constexpr int M = decltype(mc)::value;
    switch (order) {
      case 2:
        if constexpr ((M & kB16) != 0) return fail(FEM_ERR_INVALID_ORDER, "fragment kernel, BF16x6: order 2");
        else return launch_frag_sched_p<2, M>(a, sa, s);
      case 3: return launch_frag_sched_p<3, M>(a, sa, s);
      case 4:
        if constexpr ((M & (kNL | kB16)) != 0) return fail(FEM_ERR_INVALID_ORDER, "fragment kernel, mode %d: order 4", M);
        else return launch_frag_sched_p<4, M>(a, sa, s);
      default: return fail(FEM_ERR_INVALID_ORDER, "fragment kernel: order %d", order);
    }
  };
  switch (mode) {
    case kPlan | kRes: return go(IC<kPlan | kRes>{});
    case kPlan | kJac: return go(IC<kPlan | kJac>{});
    case kPlan | kRes | kJac: return go(IC<kPlan | kRes | kJac>{});
    case kPlan | kJac | kB16: return go(IC<kPlan | kJac | kB16>{});
    case kPlan | kRes | kJac | kB16: return go(IC<kPlan | kRes | kJac | kB16>{});
    case kNL | kPlan | kRes: return go(IC<kNL | kPlan | kRes>{});
    case kNL | kPlan | kJac: return go(IC<kNL | kPlan | kJac>{});
    case kNL | kPlan | kRes | kJac: return go(IC<kNL | kPlan | kRes | kJac>{});
    default: return fail(FEM_ERR_INVALID_ARGUMENT, "fragment kernel, schedule: mode %d", mode);
  }
}

int launch_frag_batched_sched(int order, int precision, const dev::AsmArgs *meshes, const dev::SchedArgs &sa,
                              cudaStream_t s) {
  using namespace dev;
  constexpr int M = kPlan | kRes | kJac;
  const bool b16 = b16_stiffness(order, precision, FEM_STRAIN_LINEAR);
  switch (order) {
    case 2: return launch_frag_batched_sched_p<2, M>(meshes, sa, s);
    case 3: return b16 ? launch_frag_batched_sched_p<3, M | kB16>(meshes, sa, s)
                       : launch_frag_batched_sched_p<3, M>(meshes, sa, s);
    case 4: return launch_frag_batched_sched_p<4, M>(meshes, sa, s);
    default: return fail(FEM_ERR_INVALID_ORDER, "fragment kernel: order %d", order);
  }
}

int launch_frag_batched(int order, int precision, const dev::AsmArgs *meshes, const dev::Tile *tiles, int ntiles,
                        int *counter, cudaStream_t s) {
  using namespace dev;
  constexpr int M = kPlan | kRes | kJac;
  const bool b16 = b16_stiffness(order, precision, FEM_STRAIN_LINEAR);
  switch (order) {
    case 2: return launch_frag_batched_p<2, M>(meshes, tiles, ntiles, counter, s);
    case 3: return b16 ? launch_frag_batched_p<3, M | kB16>(meshes, tiles, ntiles, counter, s)
                       : launch_frag_batched_p<3, M>(meshes, tiles, ntiles, counter, s);
    case 4: return launch_frag_batched_p<4, M>(meshes, tiles, ntiles, counter, s);
    default: return fail(FEM_ERR_INVALID_ORDER, "fragment kernel: order %d", order);
  }
}

}  // namespace fem
