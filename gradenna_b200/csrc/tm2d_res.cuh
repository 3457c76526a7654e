// 2D TM time loop, register-resident tiles (included by tm2d.cu inside
// namespace gdn::tm2d).
//
// Same arithmetic as tb_body, bit for bit, organised so that the state stays
// on the chip:
//
//   * A CTA owns one rectangle of the grid for a whole SEGMENT of time steps
//     (up to SEG_MAX), one CTA per SM. A warp holds R rows and 32 * V columns
//     of Ez, Hx and Hy of the rectangle and its halo of TB cells in registers
//     (V adjacent columns a lane); ca, cb and the CPML psi sit in shared
//     memory. Horizontal neighbours come from warp shuffles, vertical ones
//     from registers, one row per warp and half step through shared memory.
//   * After each block of TB = 4 steps the CTA sends its frame (the cells that
//     neighbours hold as halo) as 16-byte words that carry their own block
//     number, and polls its halo cells' words: one trip through L2, no fence,
//     no flag, no launch. The whole grid is one cooperative launch, so every
//     rectangle is resident and the words always come. Interior state goes to
//     memory only at a segment's end.
//   * The tile kernels round E differently in general tiles (near a slab or
//     the PEC ring) than in interior ones, halo included. Rectangles therefore
//     never span both classes, and their class is that of the tiles they are
//     cut from (Cfg), which keeps every bit.
//   * Point work belongs to the thread that holds the cell: the host sorts
//     every rectangle's points by thread. Source values of a segment are
//     tabulated beforehand (tm_values), so CW synthesis stays off the step's
//     path. DFT samples go from registers to a ring of one slot per step of
//     the segment; tm_seg_fold adds them up afterwards, in the same 32-step
//     partial sums as tm_dft_fold.
//
// What bounds it: not memory (the state stays in registers; only ring, frame
// and value traffic is left: 4 MB of DRAM a block at 1024 x 1024) but a block's
// chain. At 1024 x 1024 f32 with a 512 x 512 design monitor and contour currents a
// block of four steps takes 21 us, 12 us with one source: half steps, the row
// exchange and two barriers a step, about 4 us for send and receive, then points
// and ring stores.
// Measured on B200 against the tile kernels alone, whole calls:
//   70 x 53 f32, 300 steps, 2 frequencies                  2.8 ms -> 1.5 ms
//   140 x 140 f32 gradient, 2 x 3500 steps                41.9 ms -> 20.1 ms
//   280 x 280 f64 gradient, 2 x 7000 steps                  84 ms -> 54 ms
//   517 x 384 f32, 2000 steps, 8 frequencies, whole grid  18.3 ms -> 9.7 ms
//   1024 x 1024 f32 gradient, 2 x 8000 steps               143 ms -> 100 ms
#pragma once

namespace res {

constexpr int TB = 4;
constexpr int SEG_MAX = 1024;        // steps per segment
constexpr int FOLD = 32;             // steps per partial DFT sum
constexpr int POLLS = 1 << 22;       // polls of a word before a CTA gives up (seconds)

// A rectangle of owned cells, all of one class.
struct Rect {
  int i0, j0, h, w, gen;
};

// A port or probe copy in the thread that holds its cell: `m` its own index; w
// packs register r * V + k (8 bits), kind (2 bits: 1 = owner for ports) and a
// port's number in the rectangle (22 bits), which is also that of its value.
struct __align__(8) RPt {
  int m;
  unsigned w;
  __host__ __device__ int reg() const { return int(w & 255); }
  __host__ __device__ int kind() const { return int(w >> 8 & 3); }
  __host__ __device__ int val() const { return int(w >> 10); }
};
// A thread's entries of its rectangle: first, then the counts of Mx/My, Jz,
// ports and probes (16 bits each). Currents are added by masks of the registers
// whose cells have one: the values follow one another from index v of the
// rectangle's on, Hx then Hy by register, then Jz (from v plus the count of
// Mx/My). Cells with several currents have the second ones in another layer of
// masks, and so on: `how` bit 1 (3) says that magnetic (electric) layers follow as
// {Hx mask, Hy mask} ({Ez mask, 0}) in the class's entries up to a pair of zeros;
// bit 0 that the values are not staged. us for 160 steps at 1024 x 1024 f32, an
// entry at a time, each value through an index -> by layers, values in order,
// staged by asynchronous copies (tile kernels): 150 x 150 Jz 4209 -> 833 (1926),
// 16 x 16 Jz named twice 3246 -> 576 (989). A row's values loaded together first
// spilled (F32E: 72 -> 440 bytes) and cost the 1024 x 1024 gradient an eighth.
struct __align__(16) RHdr {
  int first;
  unsigned n01, n23, how;
  unsigned m_hx, m_hy, m_e, v;
};
constexpr int MAXE = 512;  // entries of a rectangle staged in shared memory
// Words of 32 monitor parts that a thread keeps masks of, past the first. Walked by
// every thread instead, 200 monitors of 3 x 3 cells in a rectangle took 10.1 ms for
// 160 steps at 1024 x 1024 f32, with masks 1.2 (tile kernels 4.3).
constexpr int MOREW = 16;

// Everything a rectangle needs besides Dev: one per run.
template <typename T>
struct RDev {
  Dev<T> d;
  uint4* xch;          // words in flight: [parity][NF + 2 NP][padded plane]
  const T* pv;         // [step - seg0][n_vals] injected values, by rectangle
  int n_vals;
  // A rectangle's first val_cap injections are staged in shared memory, from
  // element val_at on. As many as the largest rectangle holds wherever they fit:
  // fetched from pv entry by entry instead, past a fixed 256 of them, the 360 of
  // a rectangle that a flux contour crosses set the pace of the whole 1024 x 1024
  // adjoint run (38.1 us a block of four steps; staged 17.8).
  int val_at, val_cap;
  const int* vl_off;   // per rectangle CSR over vl: its values
  const int* vl;       // their injection (Jz, Mx, My, ports)
  const RHdr* hdr;     // [slot][NT]
  const int* pts_off;  // [slot] CSR over pts
  const RPt* pts;
};

// A CTA of a launch: a rectangle and its index, header slot or -1.
struct RTile {
  int idx, slot, i0, j0, h, w, gen;
};

template <typename T>
struct RArgs {
  const RDev<T>* dev;
  const RTile* tiles;
  int* err;
  int blk0, blk1, seg0;  // blocks [blk0, blk1); ring and value slot 0 is step seg0
  int polls;             // polls of a word before a CTA gives up
  int hold;              // tests: rectangle 0 keeps this block's words back (-1: none)
};

// NW warps of R rows, V columns a lane.
template <typename T_, int NW_, int R_, int V_>
struct Shape {
  using T = T_;
  static constexpr int NW = NW_, R = R_, V = V_, NT = NW * 32;
  static constexpr int EH = NW * R, EW = 32 * V;        // extended cells
  static constexpr int TI = EH - 2 * TB, TJ = EW - 2 * TB;  // most owned cells
  static constexpr int MREG = R * V <= 8 ? 3 : 1;  // monitor parts a thread keeps in registers
  // Words of a cell: NF of fields {Ez, Hx, Hy, block} (float) or {value,
  // block} each (double); NP per psi pair (ezx, hyx), (ezy, hxy).
  static constexpr int NF = sizeof(T) == 4 ? 1 : 3, NP = sizeof(T) == 4 ? 1 : 2;
  // Dynamic shared memory, in elements: first Ez row and last Hy row of every
  // warp, staged frame or halo cells (Ez, Hx, Hy: eight rows of EW, then eight
  // columns of the rows between them), ca, cb; general rectangles add
  // coefficients and psi. The injected values of a block follow (RDev).
  static constexpr int NB = 2 * TB * (EH + EW);
  static constexpr int O_Y = NW * EW, O_B = 2 * NW * EW, O_C = O_B + 3 * NB;
  static constexpr int O_GEN = O_C + 2 * EH * EW;
  using K = Coef<T, EH, EW>;
  static constexpr int KE = int((sizeof(K) + 15) / 16 * 16 / sizeof(T));
};

// Kinds of launches, smallest rectangles first: few cells a thread finish a
// step soonest and are taken while every rectangle has an SM of its own. A
// kind has a shape for interior rectangles and one for general ones, whose
// cells cost about twice as much. (16 warps of 128 registers: 32 warps of 64
// spilled, and eight rows a warp of 32 x 64 tiles left general rectangles three
// to ten times slower than interior ones.)
using F32A = Shape<float, 16, 2, 1>;    // 24 x 24 owned cells
using F32B = Shape<float, 16, 4, 1>;    // 56 x 24
using F32C = Shape<float, 16, 4, 2>;    // 56 x 56
using F32CG = Shape<float, 16, 2, 2>;   // 24 x 56
using F32D = Shape<float, 16, 4, 4>;    // 56 x 120
using F32DG = Shape<float, 16, 3, 3>;   // 40 x 88
using F32E = Shape<float, 16, 6, 4>;    // 88 x 120
using F32EG = Shape<float, 16, 4, 3>;   // 56 x 88
using F64A = Shape<double, 16, 2, 1>;   // 24 x 24
using F64B = Shape<double, 16, 4, 1>;   // 56 x 24
using F64C = Shape<double, 16, 4, 2>;   // 56 x 56
using F64CG = Shape<double, 16, 2, 2>;  // 24 x 56
constexpr int NKIND = 5;                // float kinds A .. E; double A .. C

// Rows (columns) of the extended rectangle [lo, lo + n) inside the low and
// high CPML slab of an axis of `len` nodes: E- and H-type samples together are
// nodes 0 .. m and len - 1 - m .. len - 2.
struct Slab {
  int a0, a1, b0, b1;  // [a0, a1) low, [b0, b1) high, relative to lo
  __host__ __device__ bool has(int c) const { return (c >= a0 && c < a1) || (c >= b0 && c < b1); }
  // psi storage covers [first, end): both slabs and what lies between them
  // where a rectangle meets both.
  __host__ __device__ int first() const { return a1 > a0 ? a0 : b0; }
  __host__ __device__ int end() const { return b1 > b0 ? b1 : (a1 > a0 ? a1 : b0); }
};
__host__ __device__ __forceinline__ Slab slab_range(int lo, int n, int len, int m) {
  Slab s{0, 0, 0, 0};
  if (m <= 0) return s;
  const int h0 = len - 1 - m;
  s.a0 = 0 > lo ? -lo : 0;
  s.a1 = m + 1 - lo < n ? m + 1 - lo : n;
  if (s.a1 < s.a0) s.a1 = s.a0;
  s.b0 = h0 > lo ? h0 - lo : 0;
  s.b1 = len - 1 - lo < n ? len - 1 - lo : n;
  if (s.b1 < s.b0) s.b1 = s.b0;
  return s;
}
// psi storage in elements: two x arrays (rows x EW), two y arrays (EH x the
// columns of the lanes that the slabs touch, v columns a lane).
__host__ __device__ __forceinline__ int psi_elems(const Slab& x, const Slab& y, int eh, int ew) {
  const int v = ew / 32, lanes = y.end() > y.first() ? (y.end() - 1) / v - y.first() / v + 1 : 0;
  return 2 * (x.end() - x.first()) * ew + 2 * eh * lanes * v;
}

// 16-byte words between tiles: single accesses at GPU scope, so a word's
// payload and its block number arrive together and no fence is needed.
__device__ __forceinline__ void put_word(uint4* p, const uint4& v) {
  asm volatile(
      "{\n\t.reg .b64 lo, hi;\n\t.reg .b128 w;\n\t"
      "mov.b64 lo, {%1, %2};\n\tmov.b64 hi, {%3, %4};\n\tmov.b128 w, {lo, hi};\n\t"
      "st.relaxed.gpu.global.b128 [%0], w;\n\t}" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
      : "memory");
}
__device__ __forceinline__ uint4 get_word(const uint4* p) {
  uint4 v;
  asm volatile(
      "{\n\t.reg .b64 lo, hi;\n\t.reg .b128 w;\n\t"
      "ld.relaxed.gpu.global.b128 w, [%4];\n\tmov.b128 {lo, hi}, w;\n\t"
      "mov.b64 {%0, %1}, lo;\n\tmov.b64 {%2, %3}, hi;\n\t}"
      : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
      : "l"(p)
      : "memory");
  return v;
}
// Words of one cell: NF field words, NP words per psi pair; `n` words apart.
__device__ __forceinline__ void put_cell(uint4* p, int, float e, float x, float y, unsigned blk) {
  put_word(p, make_uint4(__float_as_uint(e), __float_as_uint(x), __float_as_uint(y), blk));
}
__device__ __forceinline__ void put_one(uint4* p, double v, unsigned blk) {
  put_word(p, make_uint4(unsigned(__double2loint(v)), unsigned(__double2hiint(v)), blk, blk));
}
__device__ __forceinline__ void put_cell(uint4* p, int n, double e, double x, double y, unsigned blk) {
  put_one(p, e, blk);
  put_one(p + n, x, blk);
  put_one(p + 2 * n, y, blk);
}
__device__ __forceinline__ void put_pair(uint4* p, int, float u, float v, unsigned blk) {
  put_word(p, make_uint4(__float_as_uint(u), __float_as_uint(v), blk, blk));
}
__device__ __forceinline__ void put_pair(uint4* p, int n, double u, double v, unsigned blk) {
  put_one(p, u, blk);
  put_one(p + n, v, blk);
}
// The same the other way; the result is 0 when every block number is `blk`.
__device__ __forceinline__ unsigned get_cell(const uint4* p, int, float& e, float& x, float& y, unsigned blk) {
  const uint4 w = get_word(p);
  e = __uint_as_float(w.x);
  x = __uint_as_float(w.y);
  y = __uint_as_float(w.z);
  return w.w ^ blk;
}
__device__ __forceinline__ unsigned get_one(const uint4* p, double& v, unsigned blk) {
  const uint4 w = get_word(p);
  v = __hiloint2double(int(w.y), int(w.x));
  return w.z ^ blk;
}
__device__ __forceinline__ unsigned get_cell(const uint4* p, int n, double& e, double& x, double& y, unsigned blk) {
  return get_one(p, e, blk) | get_one(p + n, x, blk) | get_one(p + 2 * n, y, blk);
}
__device__ __forceinline__ unsigned get_pair(const uint4* p, int, float& u, float& v, unsigned blk) {
  const uint4 w = get_word(p);
  u = __uint_as_float(w.x);
  v = __uint_as_float(w.y);
  return w.z ^ blk;
}
__device__ __forceinline__ unsigned get_pair(const uint4* p, int n, double& u, double& v, unsigned blk) {
  return get_one(p, u, blk) | get_one(p + n, v, blk);
}
// One value from memory to shared memory, not waited for.
template <typename T>
__device__ __forceinline__ void copy_async(T* dst, const T* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(unsigned(__cvta_generic_to_shared(dst))),
               "l"(src), "n"(int(sizeof(T)))
               : "memory");
}
// V adjacent values between registers and memory: for V of 2 and 4 one access
// (the address is a multiple of V values).
template <typename T, int V>
__device__ __forceinline__ void lds(T (&v)[V], const T* p) {
  if constexpr (sizeof(T) * V == 16 && V == 4) {
    const float4 q = *reinterpret_cast<const float4*>(p);
    v[0] = q.x;
    v[1] = q.y;
    v[2] = q.z;
    v[3] = q.w;
  } else if constexpr (V == 2) {
    struct __align__(2 * sizeof(T)) Two {
      T a, b;
    };
    const Two q = *reinterpret_cast<const Two*>(p);
    v[0] = q.a;
    v[1] = q.b;
  } else {
#pragma unroll
    for (int k = 0; k < V; ++k) v[k] = p[k];
  }
}
template <typename T, int V>
__device__ __forceinline__ void sts(T* p, const T (&v)[V]) {
  if constexpr (sizeof(T) * V == 16 && V == 4) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  } else if constexpr (V == 2) {
    struct __align__(2 * sizeof(T)) Two {
      T a, b;
    };
    *reinterpret_cast<Two*>(p) = Two{v[0], v[1]};
  } else {
#pragma unroll
    for (int k = 0; k < V; ++k) p[k] = v[k];
  }
}

// Explicitly rounded operations: the same roundings, in the same places, that
// the tile kernels are compiled to, so both give the same bits.
__device__ __forceinline__ float mul_(float x, float y) { return __fmul_rn(x, y); }
__device__ __forceinline__ double mul_(double x, double y) { return __dmul_rn(x, y); }
__device__ __forceinline__ float sub_(float x, float y) { return __fsub_rn(x, y); }
__device__ __forceinline__ double sub_(double x, double y) { return __dsub_rn(x, y); }
__device__ __forceinline__ float fma_(float x, float y, float z) { return __fmaf_rn(x, y, z); }
__device__ __forceinline__ double fma_(double x, double y, double z) { return __fma_rn(x, y, z); }

// A monitor part in a rectangle: extended rows [a0, a1) and columns [b0, b1);
// the ring index of extended cell (r, c) is base + r * w + c.
struct Part {
  int a0, a1, b0, b1, base, w, comp, pad;
  __device__ Part() {}
  __device__ Part(const MonW& m, int ie, int je)
      : a0(m.a0 - ie), a1(m.a1 - ie), b0(m.b0 - je), b1(m.b1 - je),
        base(int(m.base + (long long)ie * m.w + je)), w(m.w), comp(m.comp), pad(0) {}
};

// What a CTA knows about its rectangle, in shared memory: read where it is
// needed instead of held in registers, which the fields take.
template <typename T>
struct TileInfo {
  int ie, je;          // cell of extended (0, 0)
  int wb, nw;          // monitor parts
  int vb, nv, nvs;     // injections; the first nvs are staged in shared memory
  int pb, np;          // entries; the first MAXE are staged
  int fail;
  // General rectangles: slabs, psi at xo + row * EW + column, yo + row * yrow +
  // column (ezx, ezy; hyx, hxy xd, yd further).
  Slab sx, sy;
  int xo, xd, yo, yd, yrow;
  Part mw[MAXW];
  RPt pts[MAXE];
  T eb[MAXP];          // Ez^n at owned port records
};

template <class S, bool GEN>
__device__ __forceinline__ void body(const RDev<typename S::T>& D, const RTile& tl,
                                     const RArgs<typename S::T>& a, TileInfo<typename S::T>& U) {
  using T = typename S::T;
  constexpr int R = S::R, V = S::V, EW = S::EW, EH = S::EH, NW = S::NW, MREG = S::MREG;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* const sm = reinterpret_cast<T*>(smem_raw);
  const Dev<T>& d = D.d;
  int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // Kept in registers: recomputed from threadIdx they cost a special-register
  // read in front of every access.
  asm volatile("" : "+r"(lane), "+r"(warp));
  // This thread: rows r0 .. r0 + R - 1, columns c0 .. c0 + V - 1 of the
  // extended rectangle; `row` its place in the rows that warps exchange.
  const int r0 = warp * R, c0 = lane * V;
  int row = warp * EW + c0;
  asm volatile("" : "+r"(row));
  typename S::K* const K = reinterpret_cast<typename S::K*>(sm + S::O_GEN);

  if (threadIdx.x == 0) {
    U.ie = tl.i0 - TB;
    U.je = tl.j0 - TB;
    U.wb = U.nw = U.vb = U.nv = U.fail = U.pb = U.np = 0;
    if (tl.slot >= 0) {
      U.pb = D.pts_off[tl.slot];
      U.np = D.pts_off[tl.slot + 1] - U.pb;
    }
    if (d.n_mons > 0) {
      U.wb = d.mw_off[tl.idx];
      U.nw = d.mw_off[tl.idx + 1] - U.wb;
    }
    if (D.vl_off) {
      U.vb = D.vl_off[tl.idx];
      U.nv = D.vl_off[tl.idx + 1] - U.vb;
    }
    U.nvs = min(U.nv, D.val_cap);
    if constexpr (GEN) {
      U.sx = slab_range(U.ie, EH, d.nx, d.npml);
      U.sy = slab_range(U.je, EW, d.ny, d.npml);
      const int la = U.sy.first() / V, lanes = U.sy.end() > U.sy.first() ? (U.sy.end() - 1) / V - la + 1 : 0;
      U.xo = S::O_GEN + S::KE - U.sx.first() * EW;
      U.xd = (U.sx.end() - U.sx.first()) * EW;
      U.yrow = lanes * V;
      U.yo = S::O_GEN + S::KE + 2 * U.xd - la * V;
      U.yd = EH * U.yrow;
    }
  }
  __syncthreads();
  for (int q = threadIdx.x; q < min(U.nw, MAXW); q += S::NT) U.mw[q] = Part(d.mw[U.wb + q], U.ie, U.je);
  for (int q = threadIdx.x; q < min(U.np, MAXE); q += S::NT) U.pts[q] = D.pts[U.pb + q];
  if constexpr (GEN) fill_coef<T, EH, EW, S::NT>(d, *K, U.ie, U.je, threadIdx.x);
  __syncthreads();

  // Rows (the same for the whole warp) and columns of this thread: bit r (k)
  // owned, 8 + r in use, 16 + r owned and within TB of the rectangle's edge;
  // rows of general rectangles also 24 + r.
  unsigned rows = 0, cols = 0;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int q = r0 + r - TB;
    rows |= unsigned(q >= 0 && q < tl.h) << r | unsigned(q < tl.h + TB) << (8 + r) |
            unsigned(q >= 0 && q < tl.h && (q < TB || q >= tl.h - TB)) << (16 + r);
  }
#pragma unroll
  for (int k = 0; k < V; ++k) {
    const int q = c0 + k - TB;
    cols |= unsigned(q >= 0 && q < tl.w) << k | unsigned(q < tl.w + TB) << (8 + k) |
            unsigned(q >= 0 && q < tl.w && (q < TB || q >= tl.w - TB)) << (16 + k);
  }
  const bool live = rows >> 8 & 255;  // the warp has rows in use
  auto owned = [&](int r, int k) { return (rows >> r & cols >> k & 1) != 0; };
  auto in_use = [&](int r, int k) { return (rows >> (8 + r) & cols >> (8 + k) & 1) != 0; };
  auto in_frame = [&](int r, int k) {
    return owned(r, k) && ((rows >> (16 + r) | cols >> (16 + k)) & 1);
  };
  // Flags: 1 Mx/My, 2 Jz, 4 ports, 8 probes, 16 monitors, 32 a port in the warp,
  // 64 a y slab in the warp, 128 values not staged, 256 (1024) more magnetic
  // (electric) layers.
  unsigned flags = 0;
  int hd_first = 0;
  unsigned n01 = 0, n23 = 0;
  if (tl.slot >= 0) {
    const RHdr hd = D.hdr[(long long)tl.slot * S::NT + threadIdx.x];
    hd_first = hd.first;
    n01 = hd.n01;
    n23 = hd.n23;
    flags |= (n01 & 0xffff ? 1u : 0u) | (n01 >> 16 ? 2u : 0u) | (n23 & 0xffff ? 4u : 0u) |
             (n23 >> 16 ? 8u : 0u) | hd.how << 7;
  }
  // Entry q of this thread's list; begin and end of a class in it.
  auto entry = [&](int q) {
    if (q < MAXE) return U.pts[q];
    const int2 p = __ldg(reinterpret_cast<const int2*>(D.pts + U.pb + q));
    return RPt{p.x, unsigned(p.y)};
  };
  auto at_jz = [&]() { return hd_first + int(n01 & 0xffff); };
  auto at_port = [&]() { return at_jz() + int(n01 >> 16); };
  auto at_probe = [&]() { return at_port() + int(n23 & 0xffff); };
  auto at_end = [&]() { return at_probe() + int(n23 >> 16); };
  if (__any_sync(0xffffffffu, flags & 4)) flags |= 32;
  // Probes: of a thread's only one its index, and its register in bits 24 .. 31 of
  // flags; of several in as many registers (flag 512) the mask of these.
  int probe = -1;
  if ((flags & 8) && n23 >> 16 == 1) {
    const RPt q = entry(at_probe());
    probe = q.m;
    flags |= unsigned(q.reg()) << 24;
  } else if (flags & 8) {
    unsigned mask = 0;
    int last = -1;
    bool once = true;
    for (int q = at_probe(); q < at_end(); ++q) {
      const int reg = entry(q).reg();
      once = once && reg > last && reg < 32;
      mask |= 1u << (reg & 31);
      last = reg;
    }
    if (once) {
      flags |= 512;
      probe = int(mask);
    }
  }
  // Monitor parts (of the first 32) that this thread's owned cells touch. Up to
  // MREG of those that cover all of them are kept in registers: ring index of
  // the thread's first cell, row pitch, component; `pmask` keeps the others.
  // Masks of the next 32 * MOREW parts lie in the thread's local memory.
  unsigned pmask = 0, mcomp = 0, more[MOREW];
  int moff[MREG], mw[MREG], mregs = 0;
#pragma unroll
  for (int u = 0; u < MREG; ++u) moff[u] = mw[u] = 0;
  if ((rows & 255) && (cols & 255)) {
    for (int q = 0; q < min(U.nw, 32); ++q) {
      const Part w = q < MAXW ? U.mw[q] : Part(d.mw[U.wb + q], U.ie, U.je);
      if (!(r0 < w.a1 && r0 + R > w.a0 && c0 < w.b1 && c0 + V > w.b0)) continue;
      bool all = true;
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (rows >> r & 1) all = all && r0 + r >= w.a0 && r0 + r < w.a1;
#pragma unroll
      for (int k = 0; k < V; ++k)
        if (cols >> k & 1) all = all && c0 + k >= w.b0 && c0 + k < w.b1;
      if (all && mregs < MREG) {
#pragma unroll
        for (int u = 0; u < MREG; ++u)
          if (u == mregs) {
            moff[u] = w.base + r0 * w.w + c0;
            mw[u] = w.w;
          }
        mcomp |= unsigned(w.comp) << (2 * mregs);
        ++mregs;
      } else {
        pmask |= 1u << q;
      }
    }
    unsigned any = mregs | pmask | unsigned(U.nw > 32 * (MOREW + 1));
#pragma unroll 1
    for (int u = 0; u < min(MOREW, (U.nw - 1) / 32); ++u) {
      unsigned mask = 0;
      for (int q = 0; q < min(32, U.nw - 32 * (u + 1)); ++q) {
        const Part w(d.mw[U.wb + 32 * (u + 1) + q], U.ie, U.je);
        mask |= unsigned(r0 < w.a1 && r0 + R > w.a0 && c0 < w.b1 && c0 + V > w.b0) << q;
      }
      more[u] = mask;
      any |= mask;
    }
    if (any) flags |= 16;
  }

  // General rectangles. x psi (slab rows): ezx at xp + r * EW + k, hyx xd
  // further; y psi (lanes that touch a slab): ezy at yp + r * yrow + k, hxy yd
  // further; all offsets into sm. Bits of rgen (rows): r Hy psi, 8 + r Ez psi,
  // 16 + r in the slab, 24 + r Ez rows inside the PEC ring; of cgen the same for
  // columns with Hx psi.
  int xp = 0, xd = 0, yp = 0, yd = 0, yrow = 0;
  unsigned rgen = 0, cgen = 0;
  if constexpr (GEN) {
    const Slab sx = U.sx, sv = U.sy;
    xp = U.xo + r0 * EW + c0;
    xd = U.xd;
    yrow = U.yrow;
    yp = U.yo + r0 * yrow + c0;
    yd = U.yd;
#pragma unroll
    for (int r = 0; r < R; ++r)
      rgen |= unsigned(K->x_h[r0 + r]) << r | unsigned(K->x_e[r0 + r]) << (8 + r) |
              unsigned(sx.has(r0 + r)) << (16 + r) | unsigned(K->r_e[r0 + r]) << (24 + r);
    const int m = d.npml, ny = d.ny;
#pragma unroll
    for (int k = 0; k < V; ++k) {
      const int j = U.je + c0 + k;
      const bool h = j >= 0 && j < ny - 1 && (j < m || j >= ny - 1 - m);
      const bool e = j >= 1 && j < ny - 1 && (j <= m || j >= ny - 1 - m);
      cgen |= unsigned(h) << k | unsigned(e) << (8 + k) | unsigned(sv.has(c0 + k)) << (16 + k) |
              unsigned(K->c_e[c0 + k]) << (24 + k);
    }
    // Columns that share a lane with slab columns keep a psi of zero.
    if (cgen >> 16 & 255) {
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int k = 0; k < V; ++k) sm[yp + r * yrow + k] = sm[yp + yd + r * yrow + k] = T(0);
    }
    if (__any_sync(0xffffffffu, cgen >> 16 & 255)) flags |= 64;  // the warp meets a y slab
  }

  T e[R][V], hx[R][V], hy[R][V];
  // The cells in use (owned = false) or owned ones, between registers and
  // state slot `par`; psi of the same cells. ca and cb come with the load.
  auto load = [&](int par) {
    const T* const src = d.state[par];
    const T* const gp = d.psi[par];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int q0 = int(cell_at(d.ld, U.ie + r0 + r, U.je + c0));  // planes hold < 2^31 cells
#pragma unroll
      for (int k = 0; k < V; ++k) {
        const int q = q0 + k;
        const bool in = in_use(r, k);
        e[r][k] = in ? __ldcg(src + q) : T(0);
        hx[r][k] = in ? __ldcg(src + d.plane + q) : T(0);
        hy[r][k] = in ? __ldcg(src + 2 * d.plane + q) : T(0);
        sm[S::O_C + (r0 + r) * EW + c0 + k] = in ? __ldcg(d.ca + q) : T(0);
        sm[S::O_C + EH * EW + (r0 + r) * EW + c0 + k] = in ? __ldcg(d.cb + q) : T(0);
        if constexpr (GEN) {
          if (rgen >> (16 + r) & 1) {
            sm[xp + r * EW + k] = in ? __ldcg(gp + q) : T(0);
            sm[xp + xd + r * EW + k] = in ? __ldcg(gp + 2 * d.plane + q) : T(0);
          }
          if (cgen >> (16 + k) & 1) {
            sm[yp + r * yrow + k] = in ? __ldcg(gp + d.plane + q) : T(0);
            sm[yp + yd + r * yrow + k] = in ? __ldcg(gp + 3 * d.plane + q) : T(0);
          }
        }
      }
    }
  };
  auto store = [&](int par) {
    T* const dst = d.state[par];
    T* const gp = d.psi[par];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int q0 = int(cell_at(d.ld, U.ie + r0 + r, U.je + c0));
#pragma unroll
      for (int k = 0; k < V; ++k)
        if (owned(r, k)) {
          const int q = q0 + k;
          __stcg(dst + q, e[r][k]);
          __stcg(dst + d.plane + q, hx[r][k]);
          __stcg(dst + 2 * d.plane + q, hy[r][k]);
          if constexpr (GEN) {
            if (rgen >> (16 + r) & 1) {
              __stcg(gp + q, sm[xp + r * EW + k]);
              __stcg(gp + 2 * d.plane + q, sm[xp + xd + r * EW + k]);
            }
            if (cgen >> (16 + k) & 1) {
              __stcg(gp + d.plane + q, sm[yp + r * yrow + k]);
              __stcg(gp + 3 * d.plane + q, sm[yp + yd + r * yrow + k]);
            }
          }
        }
    }
  };
  // Exchange units: unit u < 8 V is 32 cells of edge row u / V (0 .. 3 the
  // rectangle's first rows, 4 .. 7 its last), the others eight edge columns of
  // four rows. Calls f(staged index, row, column) for this lane's cell of every
  // unit of its warp; h x w is the frame's owned rectangle or, with the halo,
  // the extended one.
  auto unit = [&](int u, int h, int w, auto&& f) {
    if (u < 8 * V) {
      const int t = u / V, c = (u - t * V) * 32 + lane;
      const int r = t < TB ? t : h - 2 * TB + t;
      if (c < w && r < h && (t < TB || r >= TB)) f(t * EW + c, r, c);
    } else {
      const int r = TB + (u - 8 * V) * 4 + (lane >> 3), q = lane & 7;
      const int c = q < TB ? q : w - 2 * TB + q;
      if (r < h - TB && c < w && (q < TB || c >= TB)) f(8 * EW + r * 8 + q, r, c);
    }
  };
  // The frame as words of block `blk`: from the owners' registers through
  // shared memory, so that all warps share the stores.
  auto send = [&](uint4* x, unsigned blk) {
    T* const st = sm + S::O_B;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (!(rows >> r & 1)) continue;
      const int q = r0 + r - TB;
      if (rows >> (16 + r) & 1) {
        const int t = q < TB ? q : q - tl.h + 2 * TB;
#pragma unroll
        for (int k = 0; k < V; ++k)
          if (cols >> k & 1) {
            const int o = t * EW + c0 + k - TB;
            st[o] = e[r][k];
            st[S::NB + o] = hx[r][k];
            st[2 * S::NB + o] = hy[r][k];
          }
      } else if (cols >> 16 & 255) {
#pragma unroll
        for (int k = 0; k < V; ++k)
          if (cols >> (16 + k) & 1) {
            const int c = c0 + k - TB;
            const int o = 8 * EW + q * 8 + (c < TB ? c : c - tl.w + 2 * TB);
            st[o] = e[r][k];
            st[S::NB + o] = hx[r][k];
            st[2 * S::NB + o] = hy[r][k];
          }
      }
    }
    __syncthreads();
    const int n = int(d.plane);
    x += cell_at(d.ld, tl.i0, tl.j0);
    const int units = 8 * V + max(0, tl.h - 2 * TB + 3) / 4;
    for (int u = warp; u < units; u += NW)
      unit(u, tl.h, tl.w, [&](int o, int r, int c) {
        uint4* const p = x + r * d.ld + c;
        put_cell(p, n, st[o], st[S::NB + o], st[2 * S::NB + o], blk);
        if constexpr (GEN) {
          const int er = r + TB, ec = c + TB;
          if (U.sx.has(er)) {
            const int q = U.xo + er * EW + ec;
            put_pair(p + (long long)S::NF * n, n, sm[q], sm[q + U.xd], blk);
          }
          if (U.sy.has(ec)) {
            const int q = U.yo + er * U.yrow + ec;
            put_pair(p + (long long)(S::NF + S::NP) * n, n, sm[q], sm[q + U.yd], blk);
          }
        }
      });
  };
  // Halo cells from their owners' words of block `blk`, all warps sharing the
  // polls, up to B units in flight; false when a word did not come in time or
  // another CTA gave up (every rectangle then leaves, and the host makes the
  // run's outputs NaN).
  auto receive = [&](const uint4* x, unsigned blk) -> bool {
    T* const st = sm + S::O_B;
    const int n = int(d.plane), h = tl.h + 2 * TB, w = tl.w + 2 * TB;
    const int units = 8 * V + (tl.h + 3) / 4;
    constexpr int B = sizeof(T) == 4 ? 4 : 2;
    x += cell_at(d.ld, U.ie, U.je);
    for (int u0 = warp; u0 < units; u0 += B * NW) {
      int o[B], er[B], ec[B];  // o < 0: no cell; bit 30: outside the grid
#pragma unroll
      for (int q = 0; q < B; ++q) {
        o[q] = -1;
        er[q] = ec[q] = 0;
        if (u0 + q * NW < units)
          unit(u0 + q * NW, h, w, [&](int o_, int r, int c) {
            o[q] = o_;
            er[q] = r;
            ec[q] = c;
            if (GEN && (U.ie + r < 0 || U.ie + r >= d.nx || U.je + c < 0 || U.je + c >= d.ny)) o[q] |= 1 << 30;
          });
      }
      int i = 0;
      unsigned bad;
      do {
        bad = 0;
        T ve[B], vx[B], vy[B];
#pragma unroll
        for (int q = 0; q < B; ++q) {
          ve[q] = vx[q] = vy[q] = T(0);
          if (o[q] >= 0 && o[q] < 1 << 30)
            bad |= get_cell(x + er[q] * d.ld + ec[q], n, ve[q], vx[q], vy[q], blk);
        }
#pragma unroll
        for (int q = 0; q < B; ++q)
          if (o[q] >= 0) {
            T* const t = st + (o[q] & ~(1 << 30));
            t[0] = ve[q];
            t[S::NB] = vx[q];
            t[2 * S::NB] = vy[q];
          }
        if constexpr (GEN) {
#pragma unroll
          for (int q = 0; q < B; ++q)
            if (o[q] >= 0 && o[q] < 1 << 30) {
              const uint4* const p = x + er[q] * d.ld + ec[q];
              T v0, v1;
              if (U.sx.has(er[q])) {
                bad |= get_pair(p + (long long)S::NF * n, n, v0, v1, blk);
                const int t = U.xo + er[q] * EW + ec[q];
                sm[t] = v0;
                sm[t + U.xd] = v1;
              }
              if (U.sy.has(ec[q])) {
                bad |= get_pair(p + (long long)(S::NF + S::NP) * n, n, v0, v1, blk);
                const int t = U.yo + er[q] * U.yrow + ec[q];
                sm[t] = v0;
                sm[t + U.yd] = v1;
              }
            }
        }
        if (bad && (++i >= a.polls || ((i & 255) == 0 && *reinterpret_cast<const volatile int*>(a.err))))
          return false;
      } while (bad);
    }
    return true;
  };
  // The staged halo cells into registers.
  auto unpack = [&]() {
    const T* const st = sm + S::O_B;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (!(rows >> (8 + r) & 1)) continue;
      if (!(rows >> r & 1)) {
        const int er = r0 + r, t = er < TB ? er : er - tl.h;
#pragma unroll
        for (int k = 0; k < V; ++k)
          if (cols >> (8 + k) & 1) {
            const int o = t * EW + c0 + k;
            e[r][k] = st[o];
            hx[r][k] = st[S::NB + o];
            hy[r][k] = st[2 * S::NB + o];
          }
      } else if ((cols >> 8 & 255) != (cols & 255)) {
#pragma unroll
        for (int k = 0; k < V; ++k)
          if ((cols >> (8 + k) & 1) && !(cols >> k & 1)) {
            const int c = c0 + k;
            const int o = 8 * EW + (r0 + r) * 8 + (c < TB ? c : c - tl.w);
            e[r][k] = st[o];
            hx[r][k] = st[S::NB + o];
            hy[r][k] = st[2 * S::NB + o];
          }
      }
    }
  };
  auto publish_e = [&]() {
    sts(sm + row, e[0]);
  };

  const T dt_mu = d.dt_mu, inv_dx = d.inv_dx, inv_dy = d.inv_dy;
#pragma unroll 1
  for (int b = a.blk0; b < min(a.blk1, (d.n_steps + TB - 1) / TB); ++b) {
    // Injected values of the block, [sub-step][value], while the halo comes.
    for (int s = 0; s < min(TB, d.n_steps - b * TB); ++s) {
      const T* const src = D.pv + (long long)(b * TB + s - a.seg0) * D.n_vals + U.vb;
      for (int q = threadIdx.x; q < U.nvs; q += S::NT) copy_async(sm + D.val_at + s * U.nvs + q, src + q);
    }
    if (b == a.blk0) {
      load(b & 1);
    } else {
      if (!receive(D.xch + (long long)(b & 1) * (S::NF + 2 * S::NP) * d.plane, unsigned(b))) U.fail = 1;
      __syncthreads();
      unpack();
    }
    publish_e();
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    if (U.fail) {
      if (threadIdx.x == 0) atomicExch(a.err, 1);
      return;
    }

    const int n_end = min(b * TB + TB, d.n_steps);
#pragma unroll 1
    for (int n = b * TB; n < n_end; ++n) {
      // Opaque to the compiler: otherwise it takes every bit test and address
      // of the unrolled sweeps out of the loops, each into a register.
      asm volatile("" : "+r"(rows), "+r"(cols), "+r"(flags));
      if constexpr (GEN) asm volatile("" : "+r"(rgen), "+r"(cgen), "+r"(xp), "+r"(xd), "+r"(yp), "+r"(yd), "+r"(yrow));
      // ---- H sweep (fdtd2d.py:416-428) ----
      if (live) {
        T el[V];  // first Ez row of the warp below
        lds(el, sm + row + EW);  // past the last warp: Hy rows, never used
        T kb[GEN ? V : 1], kc[GEN ? V : 1], kk[GEN ? V : 1];
        if (GEN && (flags & 64)) {
#pragma unroll
          for (int k = 0; k < (GEN ? V : 1); ++k) {
            kb[k] = K->cb_h[c0 + k];
            kc[k] = K->cc_h[c0 + k];
            kk[k] = K->ck_h[c0 + k];
          }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const T en = __shfl_down_sync(0xffffffffu, e[r][0], 1);
          T dy_[V], dx_[V];
#pragma unroll
          for (int k = 0; k < V; ++k) {
            dy_[k] = mul_(sub_(k + 1 < V ? e[r][k + 1 < V ? k + 1 : k] : en, e[r][k]), inv_dy);
            dx_[k] = mul_(sub_(r + 1 < R ? e[r + 1 < R ? r + 1 : r][k] : el[k], e[r][k]), inv_dx);
          }
          if constexpr (GEN) {
            if (cgen & 0xff) {
              T q[V];
              lds(q, sm + yp + yd + r * yrow);
#pragma unroll
              for (int k = 0; k < V; ++k) {
                const bool in = cgen >> k & 1;
                q[k] = fma_(kb[k], q[k], mul_(kc[k], dy_[k]));
                dy_[k] = in ? fma_(dy_[k], kk[k], q[k]) : dy_[k];
                q[k] = in ? q[k] : T(0);
              }
              sts(sm + yp + yd + r * yrow, q);
            }
            if (rgen >> r & 1) {
              const T rb = K->rb_h[r0 + r], rc = K->rc_h[r0 + r], rk = K->rk_h[r0 + r];
              T q[V];
              lds(q, sm + xp + xd + r * EW);
#pragma unroll
              for (int k = 0; k < V; ++k) {
                q[k] = fma_(rc, dx_[k], mul_(rb, q[k]));
                dx_[k] = fma_(dx_[k], rk, q[k]);
              }
              sts(sm + xp + xd + r * EW, q);
            }
          }
#pragma unroll
          for (int k = 0; k < V; ++k) {
            hx[r][k] = fma_(-dt_mu, dy_[k], hx[r][k]);
            hy[r][k] = fma_(dt_mu, dx_[k], hy[r][k]);
          }
        }
      }
      // The rectangle's values of this step, staged or in memory.
      const T* const staged = sm + D.val_at + (n - b * TB) * U.nvs;
      auto in_memory = [&]() { return D.pv + (long long)(n - a.seg0) * D.n_vals + U.vb; };
      // f -= value in the registers of a mask, values from v on.
      auto add = [&](T (&f)[R][V], unsigned mask, int& v) {
        if (flags & 128) {
          const T* q = in_memory() + v;
#pragma unroll
          for (int r = 0; r < R; ++r)
#pragma unroll
            for (int k = 0; k < V; ++k)
              if (mask >> (r * V + k) & 1) f[r][k] += -__ldg(q++);
        } else {
          const T* q = staged + v;
#pragma unroll
          for (int r = 0; r < R; ++r)
#pragma unroll
            for (int k = 0; k < V; ++k)
              if (mask >> (r * V + k) & 1) f[r][k] += -*q++;
        }
        v += __popc(mask);
      };
      if (flags & 1) {  // Mx / My
        const RHdr& hd = D.hdr[(long long)tl.slot * S::NT + threadIdx.x];
        unsigned mx = hd.m_hx, my = hd.m_hy;
        int v = int(hd.v);
#pragma unroll 1
        for (int q = hd_first;; ++q) {
          add(hx, mx, v);
          add(hy, my, v);
          if (!(flags & 256) || q >= at_jz()) break;
          const RPt p = entry(q);
          mx = unsigned(p.m);
          my = p.w;
          if (!(mx | my)) break;
        }
      }
      sts(sm + S::O_Y + row, hy[R - 1]);
      __syncthreads();
      // ---- E sweep (fdtd2d.py:438-443) ----
      if (live) {
        T hu[V];  // last Hy row of the warp above
        lds(hu, sm + S::O_Y + row - EW);  // before the first: Ez rows, never used
        T kb[GEN ? V : 1], kc[GEN ? V : 1], kk[GEN ? V : 1];
        if (GEN && (flags & 64)) {
#pragma unroll
          for (int k = 0; k < (GEN ? V : 1); ++k) {
            kb[k] = K->cb_e[c0 + k];
            kc[k] = K->cc_e[c0 + k];
            kk[k] = K->ck_e[c0 + k];
          }
        }
        if (flags & 32) {  // port current on H^{n+1/2} and Ez^n (fdtd2d.py:430-436)
          T hl[R];
#pragma unroll
          for (int r = 0; r < R; ++r) hl[r] = __shfl_up_sync(0xffffffffu, hx[r][V - 1], 1);
          for (int q = at_port(); q < at_probe(); ++q) {
            const RPt p = entry(q);
            if (!p.kind()) continue;
            T eb = 0, y1 = 0, y0 = 0, x1 = 0, x0 = 0;
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
              for (int k = 0; k < V; ++k)
                if (p.reg() == r * V + k) {
                  eb = e[r][k];
                  y1 = hy[r][k];
                  y0 = r > 0 ? hy[r > 0 ? r - 1 : 0][k] : hu[k];
                  x1 = hx[r][k];
                  x0 = k > 0 ? hx[r][k > 0 ? k - 1 : 0] : hl[r];
                }
            if (p.val() < MAXP)
              U.eb[p.val()] = eb;
            else
              d.out_v[(long long)n * d.n_ports + p.m] = eb;
            d.out_i[(long long)n * d.n_ports + p.m] = fma_(sub_(y1, y0), d.dy, -mul_(sub_(x1, x0), d.dx));
          }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const T hl = __shfl_up_sync(0xffffffffu, hx[r][V - 1], 1);
          if constexpr (GEN) {
            T tx_[V], ty_[V];
#pragma unroll
            for (int k = 0; k < V; ++k) {
              tx_[k] = mul_(sub_(hy[r][k], r > 0 ? hy[r > 0 ? r - 1 : 0][k] : hu[k]), inv_dx);
              ty_[k] = mul_(sub_(hx[r][k], k > 0 ? hx[r][k > 0 ? k - 1 : 0] : hl), inv_dy);
            }
            if (rgen >> (8 + r) & 1) {
              const T rb = K->rb_e[r0 + r], rc = K->rc_e[r0 + r], rk = K->rk_e[r0 + r];
              T q[V];
              lds(q, sm + xp + r * EW);
#pragma unroll
              for (int k = 0; k < V; ++k) {
                q[k] = fma_(rc, tx_[k], mul_(rb, q[k]));
                tx_[k] = fma_(tx_[k], rk, q[k]);
              }
              sts(sm + xp + r * EW, q);
            }
            if (cgen & 0xff00) {
              T q[V];
              lds(q, sm + yp + r * yrow);
#pragma unroll
              for (int k = 0; k < V; ++k) {
                const bool in = cgen >> (8 + k) & 1;
                q[k] = fma_(kb[k], q[k], mul_(kc[k], ty_[k]));
                ty_[k] = in ? fma_(ty_[k], kk[k], q[k]) : ty_[k];
                q[k] = in ? q[k] : T(0);
              }
              sts(sm + yp + r * yrow, q);
            }
            T ca[V], cb[V];
            lds(ca, sm + S::O_C + (r0 + r) * EW + c0);
            lds(cb, sm + S::O_C + EH * EW + (r0 + r) * EW + c0);
#pragma unroll
            for (int k = 0; k < V; ++k) {
              const T ne = fma_(ca[k], e[r][k], mul_(cb[k], sub_(tx_[k], ty_[k])));
              e[r][k] = rgen >> (24 + r) & cgen >> (24 + k) & 1 ? ne : e[r][k];
            }
          } else {
            T ca[V], cb[V];
            lds(ca, sm + S::O_C + (r0 + r) * EW + c0);
            lds(cb, sm + S::O_C + EH * EW + (r0 + r) * EW + c0);
#pragma unroll
            for (int k = 0; k < V; ++k) {
              const T d1 = sub_(hy[r][k], r > 0 ? hy[r > 0 ? r - 1 : 0][k] : hu[k]);
              const T d2 = sub_(hx[r][k], k > 0 ? hx[r][k > 0 ? k - 1 : 0] : hl);
              e[r][k] = fma_(ca[k], e[r][k], mul_(cb[k], fma_(d1, inv_dx, -mul_(d2, inv_dy))));
            }
          }
        }
      }
      if (flags & 31) {
        // Jz (fdtd2d.py:444), then the RVS ports' injections, then their V for
        // owned records (fdtd2d.py:446-451).
        if (flags & 2) {
          const RHdr& hd = D.hdr[(long long)tl.slot * S::NT + threadIdx.x];
          unsigned me = hd.m_e;
          int v = int(hd.v + (n01 & 0xffff));
#pragma unroll 1
          for (int q = at_jz();; ++q) {
            add(e, me, v);
            if (!(flags & 1024) || q >= at_port()) break;
            me = unsigned(entry(q).m);
            if (!me) break;
          }
        }
        if (flags & 4) {
          for (int q = at_port(); q < at_probe(); ++q) {
            const RPt p = entry(q);
            const T v = p.val() < U.nvs ? staged[p.val()] : in_memory()[p.val()];
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
              for (int k = 0; k < V; ++k)
                if (p.reg() == r * V + k) e[r][k] += -v;
          }
        }
        if (flags & 4) {
          for (int q = at_port(); q < at_probe(); ++q) {
            const RPt p = entry(q);
            if (!p.kind()) continue;
            T ev = 0;
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
              for (int k = 0; k < V; ++k)
                if (p.reg() == r * V + k) ev = e[r][k];
            T* const ov = d.out_v + (long long)n * d.n_ports + p.m;
            // Past MAXP the snapshot waits in the record itself (volatile: not
            // to be fetched for the others, which would wait for DRAM).
            T eb;
            if (p.val() < MAXP)
              eb = U.eb[p.val()];
            else
              eb = *const_cast<volatile T*>(ov);
            *ov = T(-0.5) * d.dz * (eb + ev);
          }
        }
        if (flags & 8) {  // probes
          auto record = [&](int m, int reg) {
            T ev = 0;
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
              for (int k = 0; k < V; ++k)
                if (reg == r * V + k) ev = e[r][k];
            d.out_probe[(long long)n * d.n_probes + m] = ev;
          };
          if (flags & 512) {
            T* const o = d.out_probe + (long long)n * d.n_probes;
            int q = at_probe();
#pragma unroll
            for (int r = 0; r < R; ++r) {
              int m[V];  // a row's indices in flight together
#pragma unroll
              for (int k = 0; k < V; ++k)
                if (unsigned(probe) >> (r * V + k) & 1) m[k] = entry(q++).m;
#pragma unroll
              for (int k = 0; k < V; ++k)
                if (unsigned(probe) >> (r * V + k) & 1) o[m[k]] = e[r][k];
            }
          } else if (probe >= 0)
            record(probe, flags >> 24);
          else
            for (int q = at_probe(); q < at_end(); ++q) record(entry(q).m, entry(q).reg());
        }
        // ---- DFT samples of the step (every monitored owned cell) ----
        if (flags & 16) {
          T* const slot = d.mring + (long long)(n - a.seg0) * d.mon_cells;
#pragma unroll
          for (int u = 0; u < MREG; ++u)
            if (u < mregs) {
              T* const o = slot + moff[u];
              const unsigned comp = mcomp >> (2 * u) & 3;
#pragma unroll
              for (int r = 0; r < R; ++r)
                if (rows >> r & 1) {
                  T v[V];
#pragma unroll
                  for (int k = 0; k < V; ++k) v[k] = comp == 0 ? e[r][k] : (comp == 1 ? hx[r][k] : hy[r][k]);
                  if ((cols & 255) == (1u << V) - 1) {
                    sts(o + r * mw[u], v);  // ring rows are padded: whole vectors are aligned
                  } else {
#pragma unroll
                    for (int k = 0; k < V; ++k)
                      if (cols >> k & 1) o[r * mw[u] + k] = v[k];
                  }
                }
            }
          auto part = [&](const Part& w) {
            T* const o = slot + (w.base + r0 * w.w + c0);
            // rows [lo, hi) of this thread, columns by mask
            const int lo = w.a0 - r0, hi = w.a1 - r0;
            unsigned cm = 0;
#pragma unroll
            for (int k = 0; k < V; ++k) cm |= unsigned(c0 + k >= w.b0 && c0 + k < w.b1) << k;
            if (!cm) return;
#pragma unroll
            for (int r = 0; r < R; ++r)
              if (r >= lo && r < hi) {
                T v[V];
#pragma unroll
                for (int k = 0; k < V; ++k) v[k] = w.comp == 0 ? e[r][k] : (w.comp == 1 ? hx[r][k] : hy[r][k]);
                if (cm == (1u << V) - 1) {
                  sts(o + r * w.w, v);
                } else {
#pragma unroll
                  for (int k = 0; k < V; ++k)
                    if (cm >> k & 1) o[r * w.w + k] = v[k];
                }
              }
          };
          for (unsigned mk = pmask; mk; mk &= mk - 1) {
            const int q = __ffs(mk) - 1;
            if (q < MAXW)
              part(U.mw[q]);
            else
              part(Part(d.mw[U.wb + q], U.ie, U.je));
          }
#pragma unroll 1
          for (int u = 0; u < min(MOREW, (U.nw - 1) / 32); ++u)
            for (unsigned mk = more[u]; mk; mk &= mk - 1)
              part(Part(d.mw[U.wb + 32 * (u + 1) + __ffs(mk) - 1], U.ie, U.je));
          for (int q = 32 * (MOREW + 1); q < U.nw; ++q) part(Part(d.mw[U.wb + q], U.ie, U.je));
        }
      }
      if (n + 1 < n_end) {
        publish_e();
        __syncthreads();
      }
    }

    // ---- the frame to the neighbours; at the segment's end every owned cell
    // to the other state slot ----
    if (b + 1 == min(a.blk1, (d.n_steps + TB - 1) / TB))
      store((b & 1) ^ 1);
    else if (tl.idx != 0 || b + 1 != a.hold)
      send(D.xch + (long long)((b & 1) ^ 1) * (S::NF + 2 * S::NP) * d.plane, unsigned(b + 1));
    __syncthreads();
  }
}

// S, S2: the shapes of interior and of general rectangles.
template <class S, class S2>
__global__ void __launch_bounds__(S::NT, 1) tm_res(RArgs<typename S::T> a) {
  using T = typename S::T;
  static_assert(S::NT == S2::NT, "one block size");
  __shared__ __align__(16) unsigned char sdev[sizeof(RDev<T>)];
  __shared__ TileInfo<T> U;
  const RTile tl = a.tiles[blockIdx.x];
  // A rectangle of an earlier segment (or of this one) gave up: nothing to do.
  if (__syncthreads_or(*reinterpret_cast<const volatile int*>(a.err))) return;
  const int* src = reinterpret_cast<const int*>(a.dev);
  for (int q = threadIdx.x; q < int(sizeof(RDev<T>) / sizeof(int)); q += S::NT)
    reinterpret_cast<int*>(sdev)[q] = src[q];
  __syncthreads();
  const RDev<T>& D = *reinterpret_cast<const RDev<T>*>(sdev);
  if (tl.gen)
    body<S2, true>(D, tl, a, U);
  else
    body<S, false>(D, tl, a, U);
}

// Headers to their places among all threads' (zeroed beforehand). Uploaded for
// every thread, 16 KB a rectangle that holds points, they were most of what a run
// of a few steps with scattered points took.
__global__ void tm_headers(const RHdr* in, const int* at, int n, RHdr* out) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q < n) out[at[q]] = in[q];
}

// Injected values of steps [seg0, seg0 + cnt): one thread per value and FOLD steps
// (blockIdx.y). The products are formed like the tile kernels' (src_term, mx_term,
// my_term and the port term), for every rectangle that an injection reaches, in the
// order in which the rectangles read them.
template <typename T>
__global__ void __launch_bounds__(128) tm_values(const RDev<T>* dev, int seg0, int seg) {
  const RDev<T>& D = *dev;
  const Dev<T>& d = D.d;
  const int id = blockIdx.x * blockDim.x + threadIdx.x;
  if (id >= D.n_vals) return;
  const int inj = D.vl[id];
  const int t0 = blockIdx.y * FOLD;
  const int cnt = min(FOLD, min(seg, d.n_steps - seg0) - t0);
  T* const out = const_cast<T*>(D.pv) + (long long)t0 * D.n_vals + id;
  for (int t = 0; t < cnt; ++t) {
    const int n = seg0 + t0 + t;
    int m = inj;
    T v;
    if (m < d.n_src) {
      v = src_term(d, m, n);
    } else if ((m -= d.n_src) < d.n_mx) {
      v = mx_term(d, m, n);
    } else if ((m -= d.n_mx) < d.n_my) {
      v = my_term(d, m, n);
    } else {
      m -= d.n_my;
      v = d.cb_vs[m] * d.port_vs[(long long)n * d.n_ports + m];
    }
    out[(long long)t * D.n_vals] = v;
  }
}

// Threads of a CTA of tm_seg_fold, and CTAs an SM that it is compiled for: as
// many as its registers allow without spills, in steps of 128 threads where 256
// are too coarse (more waits are hidden; see the figures at the kernel).
template <typename T, typename A>
constexpr int fold_threads(int km) {
  return (km == 8 && sizeof(A) == 8) || (km == 16 && sizeof(T) == 4 && sizeof(A) == 4) ? 128 : 256;
}
template <typename T, typename A>
constexpr int fold_ctas(int km) {
  if (fold_threads<T, A>(km) == 128) return 5;
  if (km <= 8) return sizeof(T) == 4 ? 4 : 3;
  return sizeof(T) == 8 && sizeof(A) == 8 ? 1 : 2;
}

// Running DFT of a segment: per monitored cell and FOLD steps one partial sum
// in A, added to the accumulator (the sums and their order are tm_dft_fold's).
// One thread a cell; the next eight samples come while eight are summed. The
// accumulators are read and written once per FOLD steps: kept in registers for
// the segment, beside the partial sums, they left one CTA an SM, and several
// cells a thread did not make up for it. Bound by the ring's bytes for few tones
// and by the multiply-adds for many. us for a ring of about 256 MB (of 32 steps
// at 1024 x 1024), kept in registers -> here (tm_dft_fold, 32 steps a launch):
//   full grid 140 x 140, 1024 steps, 8 tones, float samples and sums  329 -> 207 (463)
//   400 x 400, 128 steps, 8 tones, float, float                       249 -> 136 (223)
//   400 x 400, 128 steps, 16 tones, float, double                    1511 -> 474 (950)
//   400 x 400, 64 steps, 8 tones, double, double                      253 -> 123 (159)
//   1024 x 1024, 32 steps, 4 tones, float, float                      329 -> 165 (191)
//   1024 x 1024, 32 steps, 16 tones, float, float                     726 -> 560 (576)
template <typename T, typename A, int KM>
__global__ void __launch_bounds__(fold_threads<T, A>(KM), fold_ctas<T, A>(KM))
    tm_seg_fold(Dev<T> d, int seg0, int seg) {
  constexpr int NT = fold_threads<T, A>(KM);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  using C = typename Cplx<A>::type;
  C* const sph = reinterpret_cast<C*>(smem_raw);  // [2 tables][FOLD][K]
  const int K = d.n_freq, total = min(seg, d.n_steps - seg0);
  const int r = int(blockIdx.x) * NT + int(threadIdx.x);  // a ring slot holds < 2^31 cells
  int lo = 0, hi = d.n_mons - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (d.mons[mid].off <= r)
      lo = mid;
    else
      hi = mid - 1;
  }
  const MonD mon = d.mons[lo];
  const unsigned loc = unsigned(r - int(mon.off));
  const int row = int(loc / unsigned(mon.pitch));
  const int col = int(loc - unsigned(row) * unsigned(mon.pitch)) - mon.pad;
  const bool live = r < d.mon_cells && row < mon.h && col >= 0 && col < mon.w;
  C* const acc = static_cast<C*>(mon.out) + ((long long)row * mon.w + col);
  const int tab = mon.comp == 0 ? 0 : FOLD * K;
  const T* const ring = d.mring + r;
  for (int b0 = 0; b0 < total; b0 += FOLD) {
    const int cnt = min(FOLD, total - b0);
    __syncthreads();
    for (int q = threadIdx.x; q < cnt * K; q += NT) {
      const double2 pe = d.ph_e[(long long)(seg0 + b0) * K + q];
      const double2 ph = d.ph_h[(long long)(seg0 + b0) * K + q];
      sph[q].x = A(pe.x);
      sph[q].y = A(pe.y);
      sph[FOLD * K + q].x = A(ph.x);
      sph[FOLD * K + q].y = A(ph.y);
    }
    __syncthreads();
    if (!live) continue;
    C part[KM];
#pragma unroll
    for (int k = 0; k < KM; ++k) part[k].x = part[k].y = A(0);
    const T* const base = ring + b0 * d.mon_cells;
    T x[8], next[8];
    auto fetch = [&](T (&v)[8], int t0) {
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = t0 + u < cnt ? base[(t0 + u) * d.mon_cells] : T(0);
    };
    fetch(next, 0);
    for (int t0 = 0; t0 < cnt; t0 += 8) {
#pragma unroll
      for (int u = 0; u < 8; ++u) x[u] = next[u];
      if (t0 + 8 < cnt) fetch(next, t0 + 8);
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        if (t0 + u < cnt) {
          const C* const p0 = sph + tab + (t0 + u) * K;
#pragma unroll
          for (int k = 0; k < KM; ++k)
            if (k < K) {
              const C p = p0[k];
              part[k].x += p.x * A(x[u]);
              part[k].y += p.y * A(x[u]);
            }
        }
      }
    }
#pragma unroll
    for (int k = 0; k < KM; ++k)
      if (k < K) {
        C v = acc[(long long)k * mon.count];
        v.x += part[k].x;
        v.y += part[k].y;
        acc[(long long)k * mon.count] = v;
      }
  }
}

}  // namespace res
