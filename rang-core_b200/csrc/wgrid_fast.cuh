// The single-precision gridder and degridder on the tensor cores, and the
// fixed-point grid that makes gridding exact and order-independent.
//
// Included by wgrid_plan.cu inside its anonymous namespace (it uses the scan,
// binning and device helpers defined there).
//
// Records. The binning's count pass writes one 32-byte record per active
// visibility at its own index: the tap arguments of u, v and w, the
// visibility's index, its shift phase, its offset inside its sub-tile's
// window, its first plane and its bin. The per-visibility FP64 arithmetic
// (coordinates, getpix, minplane, the phase's argument reduction) is thus
// done once per plan, and the gridder and degridder read records through
// the sorted indices.
//
// Exact gridding. Every grid cell is an int64 fixed-point sum (a pair per
// complex cell) of the footprint terms kw * ku * (value * kv). The gridder
// forms both factors as 23-bit integers, A = rint(kw ku 2^22) and
// B = rint(value kv 2^sb), splits each into three balanced 8-bit limbs
// (x = x2 2^16 + x1 2^8 + x0, x0 and x1 in [-128, 127]) and contracts the
// limbs on the integer tensor cores (mma.sync m16n8k32, s8 x s8 -> s32),
// keeping the limb products of weight 2^32, 2^24 and 2^16: the kept sums are
// exact integers and the dropped terms (weight 2^8 and 1, zero-mean) are
// below 2^-21 of the largest term. Integer sums do not depend on the order
// of their terms, so the result is bit for bit the same whatever the order
// of the visibilities in the sorted layout, however they are split among
// warps and blocks, and whatever the order of the atomic adds into the
// grid: a call is reproducible and a one-pass PSF equals a separate call.
// The grid is converted to floating point once, before the FFTs.

namespace fast {

// A grid cell in fixed point: value = (re + i im) * 2^-q.
struct FixCell {
  long long re, im;
};

// The fixed-point scales of one gridding pass (written on the device).
struct FixScale {
  int sb;         // B = rint(value * kv * 2^sb) in the integer gridder
  int q;          // cell value = int64 * 2^-q
  int nonfinite;  // an active value or tap was not finite: the planes are NaN
  int pad;
};

// Largest |value| of a pass (device scalars, the scan's or k_value_max's).
struct ValueBound {
  unsigned long long vmax_bits;  // max |vis| |wgt| (as the bits of a non-negative double)
  unsigned long long wmax_bits;  // max |wgt|
};

__device__ __forceinline__ void atomic_max_double(unsigned long long* a, double v) {
  if (v > 0.0) atomicMax(a, (unsigned long long)__double_as_longlong(v));
}

// max |vis| |wgt| and max |wgt| over visibilities [i0, i1) that the plan
// keeps (key != INACTIVE), for gridding data other than the plan's own.
template <class T>
__global__ void k_value_max(uint64_t i0, uint64_t i1, Inputs in, const uint32_t* __restrict__ key, ValueBound* vb) {
  double vm = 0.0, wm = 0.0;
  for (uint64_t i = i0 + blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < i1;
       i += (uint64_t)gridDim.x * blockDim.x) {
    if (key[i] == INACTIVE) continue;
    const double w = fabs((double)wgt_get<T>(in, i));
    const double a = value_bound_sq(vis_get<T>(in, i), w);
    // NaN compares false and is dropped here; the gridder flags it.
    vm = a > vm ? a : vm;
    wm = w > wm ? w : wm;
  }
  for (int o = 16; o > 0; o >>= 1) {
    vm = fmax(vm, __shfl_down_sync(0xffffffffu, vm, o));
    wm = fmax(wm, __shfl_down_sync(0xffffffffu, wm, o));
  }
  if ((threadIdx.x & 31) == 0) {
    vm = sqrt(vm);
    atomic_max_double(&vb->vmax_bits, vm);
    atomic_max_double(&vb->wmax_bits, wm);
  }
}

__global__ void k_bound_init(ValueBound* vb, unsigned long long vmax_bits, unsigned long long wmax_bits) {
  vb->vmax_bits = vmax_bits;
  vb->wmax_bits = wmax_bits;
}

// The scales of one pass from the value maxima of `values`. `unit`: unit
// values (the PSF), bounded by max |wgt|; otherwise max |vis| |wgt|. The
// integer gridder's terms are at most 2^28 grid units (q = sb + 6), so int64
// holds 2^34 of them. For the floating-point gridders a cell sums at most
// nvis terms, each at most max |value| (taps are at most 1 + eps), and q
// leaves 2 bits of headroom over that bound in the cell's width (64 bits in
// single precision; 94 bits of hi * 2^32 + lo in double, where the unit is
// 2^-(92 - log2 nvis) of the largest value, 2^-60 or finer: a 64-bit cell's
// unit would sit about 2^-48 below the largest term, which the wide-field
// correction factors amplify past double precision's accuracy). The scales
// depend on nothing but the values and the active count, so a plan split
// into row chunks grids to the same bits as one without.
// The exponent the scales take from `values`: vmax < 2^(ev + 1) (clamped,
// so that the scales stay finite floats).
__device__ __forceinline__ int bound_exponent(const ValueBound* values, int unit) {
  double vmax = __longlong_as_double((long long)(unit ? values->wmax_bits : values->vmax_bits));
  if (!(vmax > 0.0) || !isfinite(vmax)) vmax = 1.0;
  return min(max(ilogb(vmax), -90), 90);
}

__device__ __forceinline__ FixScale scale_of(int ev, unsigned long long nvis, int integer, int wide) {
  FixScale r;
  r.nonfinite = 0;
  r.pad = 0;
  if (integer) {
    r.sb = 21 - ev;  // |B| < 2^22
    r.q = r.sb + 6;
  } else {
    r.sb = 0;
    // nvis * vmax * 2^q < 2^62 (int64 cells), < 2^94 (hi * 2^32 + lo cells)
    r.q = (wide ? 92 : 60) - ev - ilogb((double)max(nvis, 1ull));
  }
  return r;
}

__global__ void k_fix_scale(const ValueBound* values, int unit, unsigned long long nvis, int integer, int wide,
                            FixScale* fs) {
  *fs = scale_of(bound_exponent(values, unit), nvis, integer, wide);
}

// Gridding row chunks as they arrive, before the bound of all the values
// is known: the scale depends on the bound only through its exponent, so
// the chunks are gridded with the exponent of the values seen so far, and
// when a chunk changes it, the planes are cleared and the chunks before it
// gridded again (`redo`, which their launches test). After the last chunk
// the exponent, and every term, is the one-pass gridding's.
struct SpecState {
  int ev;
  int redo;
};
__global__ void k_spec_scale(const ValueBound* values, int first, int unit, unsigned long long nvis, int integer,
                             int wide, SpecState* st, FixScale* fs) {
  const int ev = bound_exponent(values, unit);
  if (first || ev != st->ev) {
    st->redo = first ? 0 : 1;
    st->ev = ev;
    *fs = scale_of(ev, nvis, integer, wide);
  } else {
    st->redo = 0;
  }
}

// Zeroes n planes' rows as zero_touched does, when *flag is set.
template <class Cell>
__global__ void k_zero_touched_if(const int* __restrict__ flag, Cell* __restrict__ grids, int n, int nu, int nv,
                                  int rows) {
  if (*flag == 0) return;
  const uint64_t prow = rows == 0 ? (uint64_t)nu : 2ull * rows;  // rows cleared per plane
  const uint64_t total = (uint64_t)n * prow * nv;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < total;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t p = i / (prow * nv), r = (i / nv) % prow, c = i % nv;
    const uint64_t row = (rows == 0 || r < (uint64_t)rows) ? r : (uint64_t)nu - 2ull * rows + r;
    grids[(p * nu + row) * nv + c] = Cell{};
  }
}

__device__ __forceinline__ void fix_add(FixCell* cell, long long re, long long im) {
  if (re) atomicAdd(reinterpret_cast<unsigned long long*>(&cell->re), (unsigned long long)re);
  if (im) atomicAdd(reinterpret_cast<unsigned long long*>(&cell->im), (unsigned long long)im);
}

// A double-precision grid value in fixed point: hi * 2^32 + lo, two int64
// words, and a complex cell of two of them. A term, x * 2^q rounded once to
// an integer t, is split as t_hi = floor(t / 2^32) and t_lo = t - t_hi 2^32 in
// [0, 2^32]; the words sum their parts independently, so adding a term is two
// integer adds that need no carry and no returned value (red.global.add),
// exact in any order. lo stays below 2^63 for fewer than 2^31 terms per cell
// (runs, not visibilities, are the terms), hi below 2^62 by the scale's
// headroom (k_fix_scale).
struct FixWide {
  long long lo, hi;
};
struct FixCell2 {
  FixWide re, im;
};

__device__ __forceinline__ void fix_add_wide(FixWide* cell, FixWide v) {
  if (v.lo) atomicAdd(reinterpret_cast<unsigned long long*>(&cell->lo), (unsigned long long)v.lo);
  if (v.hi) atomicAdd(reinterpret_cast<unsigned long long*>(&cell->hi), (unsigned long long)v.hi);
}

// The fixed-point cell and accumulator of each working precision.
template <class T>
struct FixTraits;
template <>
struct FixTraits<float> {
  using Cell = FixCell;
  using Acc = long long;
  static constexpr int wide = 0;
  // x * 2^q rounded to an integer (sc = 2^q)
  static __device__ __forceinline__ float scale(int q) { return ldexpf(1.0f, q); }
  static __device__ __forceinline__ Acc term(float x, float sc) { return __float2ll_rn(x * sc); }
  static __device__ __forceinline__ Acc zero() { return 0; }
  static __device__ __forceinline__ Acc add(Acc a, Acc b) { return a + b; }
  static __device__ __forceinline__ bool nonzero(Acc a) { return a != 0; }
  static __device__ __forceinline__ void flush(Cell* c, Acc re, Acc im) { fix_add(c, re, im); }
  static __device__ __forceinline__ double value(long long v, int q) { return ldexp((double)v, -q); }
};
template <>
struct FixTraits<double> {
  using Cell = FixCell2;
  using Acc = FixWide;
  static constexpr int wide = 1;
  // sc = 2^(q - 32): y = x * sc (exact), hi = floor(y) (exact; every double
  // from 2^52 up is an integer), lo = rint((y - hi) 2^32) (the fraction is
  // exact, the one rounding is to the grid's unit).
  static __device__ __forceinline__ double scale(int q) { return ldexp(1.0, q - 32); }
  static __device__ __forceinline__ Acc term(double x, double sc) {
    const double y = x * sc, h = floor(y);
    return FixWide{__double2ll_rn((y - h) * 4294967296.0), __double2ll_rn(h)};
  }
  static __device__ __forceinline__ Acc zero() { return FixWide{0ll, 0ll}; }
  static __device__ __forceinline__ Acc add(Acc a, Acc b) { return FixWide{a.lo + b.lo, a.hi + b.hi}; }
  static __device__ __forceinline__ bool nonzero(Acc a) { return (a.lo | a.hi) != 0; }
  static __device__ __forceinline__ void flush(Cell* c, Acc re, Acc im) {
    fix_add_wide(&c->re, re);
    fix_add_wide(&c->im, im);
  }
  static __device__ __forceinline__ double value(FixWide v, int q) {
    return ldexp((double)v.hi, 32 - q) + ldexp((double)v.lo, -q);
  }
};

// Planes (one per blockIdx.y) of the fixed-point grid to floating point: rows
// [0, rows) and [nu - rows, nu) (every row when rows is 0), each cell rounded
// once.
template <class T>
__global__ void k_fix_to_plane(const typename FixTraits<T>::Cell* __restrict__ fix, int nu, int nv, int rows,
                               const FixScale* fs, cplx<T>* __restrict__ out) {
  fix += (size_t)blockIdx.y * nu * nv;
  out += (size_t)blockIdx.y * nu * nv;
  const int q = fs->q;
  const bool nan = fs->nonfinite != 0;
  const int nr = rows == 0 ? nu : 2 * rows;
  const uint64_t n = (uint64_t)nr * nv;
  for (uint64_t c = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; c < n; c += (uint64_t)gridDim.x * blockDim.x) {
    const int r = (int)(c / nv);
    const uint64_t cell = (uint64_t)(rows == 0 || r < rows ? r : nu - 2 * rows + r) * nv + (c - (uint64_t)r * nv);
    const auto f = fix[cell];
    cplx<T> v;
    if (nan) {
      v = {(T)__longlong_as_double(0x7ff8000000000000ll), (T)__longlong_as_double(0x7ff8000000000000ll)};
    } else {
      v = {(T)FixTraits<T>::value(f.re, q), (T)FixTraits<T>::value(f.im, q)};
    }
    out[cell] = v;
  }
}

// ------------------------------------------------------------------ records

struct VisRecord {
  float x0, y0, xw;  // tap arguments (taps_uv, w_factor's locz of the first plane)
  uint32_t idx;      // visibility index, row * nchan + channel
  float ph_re, ph_im;  // shift phase (shift_phase with sign +1), (1, 0) without shifts
  uint32_t meta;     // dv << 4 | (w was flipped) << 8 | su mod 8 << 9 | first plane << 16
  uint32_t bin;      // the sorted key (chunk * nbins + bin)
};
static_assert(sizeof(VisRecord) == 32, "records are one 32-byte sector");

// The loads of one visibility of the count pass: its word of the scan's
// active bits, its row's coordinates and its channel's f / c, issued an
// iteration ahead of their use (the pass otherwise waited on them).
struct CountIn {
  uint32_t word = 0;
  double4 b = {0.0, 0.0, 0.0, 0.0};  // the row's coordinates and phase (k_row_coords)
  double f = 0.0;
};
__device__ __forceinline__ CountIn count_in(const uint32_t* __restrict__ bits, const double4* __restrict__ rowc,
                                            const double* __restrict__ foc, uint64_t i, uint32_t row, uint32_t ch) {
  CountIn c;
  c.word = bits[i >> 5];
  c.b = rowc[row];
  c.f = foc[ch];
  return c;
}

// Each row's coordinates as the binning uses them (row_coord: flips,
// recentring, w made non-negative; w negated here where that flipped it) and
// its shift phase in turns per f / c (shift_phase with sign +1), once per row:
// the count pass then reads them instead of forming them for every channel
// (the same doubles, so the same keys and records).
__global__ void k_row_coords(uint64_t nrow, const double* __restrict__ uvw, double fu, double fv, double fw,
                             double r_l, double r_m, double lshift, double mshift, double nshift,
                             double4* __restrict__ out) {
  for (uint64_t r = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; r < nrow;
       r += (uint64_t)gridDim.x * blockDim.x) {
    double b[3];
    const double sgn = row_coord(uvw, r, fu, fv, fw, r_l, r_m, b);
    const double turns = sgn * (b[0] * lshift + b[1] * mshift + b[2] * nshift);
    out[r] = make_double4(b[0], b[1], copysign(b[2], sgn), turns);
  }
}

// The count pass of the counting sort (k_bin_count) for single precision,
// writing as well the record of each active visibility at its own index
// (coalesced): its coordinates and taps' arguments are formed here once. The
// scatter then moves only the 4-byte indices, and the gridder and degridder
// read each record through the sorted index. The active set comes from the
// scan's bits (bit i: visibility i), one word per 32 visibilities. The
// plan's uniform choices (w-planes, phase shift, row chunks) are template
// arguments: tested in the loop they cost branches and reloads of the plan's
// constants on every visibility. Three blocks per SM (at most 85 registers)
// measured 9.20 ms per call at 1.06 G visibilities, four 9.32, five 9.61. It is
// bound by issue (80 % of the slots; the conversion unit 60 %, FP64 20 %):
// 17.5 ms for two calls became 16.1 with the phase formed once per row in turns.
constexpr int COUNT_BLOCKS = 3;
template <bool WPL, bool SHIFT, bool CHUNKED>
__global__ void __launch_bounds__(256, COUNT_BLOCKS)
    k_bin_count_rec(const __grid_constant__ Geom<float> g, const double4* __restrict__ rowc,
                    const double* __restrict__ foc, const uint32_t* __restrict__ bits, uint32_t* __restrict__ key,
                    uint32_t* __restrict__ counts, VisRecord* __restrict__ rec, uint32_t rows_per_chunk,
                    uint32_t nbins, uint64_t i0, uint64_t n, uint32_t koff) {
  // Visibilities [i0, n); bin k is counted in counts[k - koff].
  const uint64_t nround = i0 + ((n - i0 + 31) & ~31ull);
  const uint32_t tmask = (1u << g.log2tile) - 1u;
  const uint32_t se = (uint32_t)g.sube, sdiv = (65536u + se - 1u) / se;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  uint64_t i = i0 + blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  RowCh rc(i, (uint32_t)g.nchan, stride);
  CountIn cur = i < n ? count_in(bits, rowc, foc, i, rc.row, rc.ch) : CountIn{};
  for (; i < nround; i += stride) {
    RowCh nrc = rc;
    nrc.next((uint32_t)g.nchan);
    const CountIn nxt = i + stride < n ? count_in(bits, rowc, foc, i + stride, nrc.row, nrc.ch) : CountIn{};
    bool act = false;
    uint32_t k = INACTIVE;
    if (i < n) {
      act = ((cur.word >> (i & 31)) & 1u) != 0;
      if (act) {
        const double f = cur.f;
        const double u = cur.b.x * f, v = cur.b.y * f, w = fabs(cur.b.z) * f;
        double uf, vf;
        int iu0, iv0;
        getpix(g, u, v, uf, vf, iu0, iv0);
        const uint32_t su = (uint32_t)shifted(iu0, g.nu), sv = (uint32_t)shifted(iv0, g.nv);
        // (x / sube) for x < 32 as a multiply and shift (exact: the error of
        // ceil(2^16 / sube) stays below 2^-11 over 32 steps)
        const uint32_t sa = ((su & tmask) * sdiv) >> 16, sb = ((sv & tmask) * sdiv) >> 16;
        const int mp = WPL ? minplane(g, w) : 0;
        // The key of bin_of_rc (Setup::locate refined by the sub-tile).
        k = (((su >> g.log2tile) * (uint32_t)g.ntv + (sv >> g.log2tile)) * (uint32_t)g.nbuckets + (uint32_t)mp) *
                (uint32_t)g.nsub + sb * (uint32_t)g.nsub_side + sa;
        if (CHUNKED) k += (rc.row / rows_per_chunk) * nbins;
        // The record's two 16-byte halves, formed in registers (VisRecord's
        // field order).
        const double s1 = (double)g.supp - 1.0;
        const float x0 = (float)(-uf * 2.0 + s1);
        const float y0 = (float)(-vf * 2.0 + s1);
        float xw = 0.0f;
        if (WPL) {  // w_factor's argument for the first plane (nth 0)
          const float z = (float)(g.xdw * ((g.wmin + (double)mp * g.dw) - w));
          xw = z * 2.0f + (float)s1;
        }
        float ph_re = 1.0f, ph_im = 0.0f;
        if (SHIFT) {
          const cplx<float> ph = cis_turns(cur.b.w * f, 0.0f);
          ph_re = ph.re;
          ph_im = ph.im;
        }
        const uint32_t meta = (((sv & tmask) - sb * se) << 4) |
                              (signbit(cur.b.z) ? 256u : 0u) | ((su & 7u) << 9) | ((uint32_t)mp << 16);
        reinterpret_cast<uint4*>(rec + i)[0] =
            make_uint4(__float_as_uint(x0), __float_as_uint(y0), __float_as_uint(xw), (uint32_t)i);
        reinterpret_cast<uint4*>(rec + i)[1] = make_uint4(__float_as_uint(ph_re), __float_as_uint(ph_im), meta, k);
      }
      key[i] = k;
    }
    warp_aggregated_count(counts, k - koff, act);
    cur = nxt;
    rc = nrc;
  }
}

// The taps of one axis at x (the reference's eval_taps, one of the two axes
// of eval_taps2).
template <int S, class T>
__device__ __forceinline__ void eval_taps1(const T* __restrict__ c, T x, T* r) {
  constexpr int ne = coeff_rows(S);
  constexpr int H = (S + 1) / 2;
  const T x2 = x * x;
  T e[H], o[H];
#pragma unroll
  for (int i = 0; i < H; i++) {
    e[i] = c[i];
    o[i] = c[ne * S + i];
  }
#pragma unroll
  for (int k = 1; k < ne; k++)
#pragma unroll
    for (int i = 0; i < H; i++) {
      e[i] = fma_t(e[i], x2, c[k * S + i]);
      o[i] = fma_t(o[i], x2, c[(ne + k) * S + i]);
    }
#pragma unroll
  for (int i = 0; i < H; i++) r[i] = fma_t(o[i], x, e[i]);
#pragma unroll
  for (int i = 0; i < S - H; i++) r[S - 1 - i] = fma_t(o[i], -x, e[i]);
}

// The kernel's polynomials for evaluation two coefficients at a time: even and
// odd coefficient k of tap i (of the first ceil(S / 2)) side by side, for the
// packed FP32 multiply-add (fma.rn.f32x2, each half rounded as fmaf rounds):
// a tap costs half the instructions, and the kernels below are bound by them.
template <int S>
struct TapPairs {
  static constexpr int NE = coeff_rows(S), H = (S + 1) / 2;
  float2 c[NE * H];
  explicit TapPairs(const float* coeff) {
    for (int k = 0; k < NE; k++)
      for (int i = 0; i < H; i++) c[k * H + i] = make_float2(coeff[k * S + i], coeff[(NE + k) * S + i]);
  }
};
__device__ __forceinline__ unsigned long long pack2(float x, float y) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// The taps of one axis at x (eval_taps1 in pairs, the same roundings).
template <int S>
__device__ __forceinline__ void eval_taps_pairs(const TapPairs<S>& tp, float x, float* r) {
  constexpr int ne = TapPairs<S>::NE, H = TapPairs<S>::H;
  const float x2 = x * x;
  const unsigned long long xx = pack2(x2, x2);
  unsigned long long eo[H];
#pragma unroll
  for (int i = 0; i < H; i++) eo[i] = pack2(tp.c[i].x, tp.c[i].y);
#pragma unroll
  for (int k = 1; k < ne; k++)
#pragma unroll
    for (int i = 0; i < H; i++) eo[i] = fma2(eo[i], xx, pack2(tp.c[k * H + i].x, tp.c[k * H + i].y));
#pragma unroll
  for (int i = 0; i < H; i++) {
    const float2 v = unpack2(eo[i]);
    r[i] = fmaf(v.y, x, v.x);
    if (i < S - H) r[S - 1 - i] = fmaf(v.y, -x, v.x);
  }
}

// The stored value of a record's visibility (unit_value, data_value,
// wgridder.rs:1414-1435): value = vis * phase * wgt with the imaginary part
// negated where w was flipped; the phase alone times wgt for unit values.
__device__ __forceinline__ cplx<float> record_value(const VisRecord& r, const Inputs& in, int mode) {
  const float flip = (r.meta & 256u) ? -1.0f : 1.0f;
  float pr = r.ph_re, pi = r.ph_im;
  if (in.wgt_kind != WGT_NONE) {
    const float w = wgt_get<float>(in, r.idx);
    pr *= w;
    pi *= w;
  }
  if (mode == VALUE_DATA) {
    const cplx<float> v = vis_get<float>(in, r.idx);
    const float dr = v.re * pr - v.im * pi, di = v.re * pi + v.im * pr;
    return {dr, di * flip};
  }
  return {pr, pi * flip};
}

// The window of a bin key: its first row on the shifted indices (rb), the grid
// row and column of its cell (0, 0) (the sub-tile's first cell; windows are
// 8 x 8) and its first plane. Within a tile, first plane and sub-tile column
// (a strip) the keys ascend along u.
template <class T>
__device__ __forceinline__ void window_of(const Geom<T>& g, uint32_t key, uint32_t nbins, int& rb, int& su0,
                                          int& sv0, int& mp) {
  const uint32_t bin = key % nbins;
  const uint32_t sub = bin % (uint32_t)g.nsub, t = bin / (uint32_t)g.nsub;
  mp = (int)(t % (uint32_t)g.nbuckets);
  const uint32_t tile = t / (uint32_t)g.nbuckets;
  const uint32_t tu = tile / (uint32_t)g.ntv, tv = tile - tu * (uint32_t)g.ntv;
  // Tiles are laid out on the shifted indices (i0 + n/2) mod n; the grid is
  // stored unshifted.
  rb = (int)((tu << g.log2tile) + (sub % (uint32_t)g.nsub_side) * (uint32_t)g.sube);
  su0 = (int)(((uint32_t)rb + (uint32_t)(g.nu - g.nu / 2)) % (uint32_t)g.nu);
  sv0 = (int)(((tv << g.log2tile) + (sub / (uint32_t)g.nsub_side) * (uint32_t)g.sube + (uint32_t)(g.nv - g.nv / 2)) %
              (uint32_t)g.nv);
}

// A warp's window as it moves from bin to bin of the sorted order. Its rows
// sit at u mod 8 (on the shifted indices), so that the next bin of the same
// strip, a few rows further along u, keeps every row the two windows share in
// place: only the rows that leave are written out (gridding), only those that
// enter are read (degridding).
struct Window {
  uint32_t key = INACTIVE, strip = INACTIVE;  // the bin, and its strip (key / nsub_side)
  int rb = 0, su0 = 0, sv0 = 0, mp = 0;       // window_of
};
// Moves to bin `key`; returns the rows the move leaves behind (8: all).
template <class T>
__device__ __forceinline__ int window_step(const Geom<T>& g, const Window& w, uint32_t key, uint32_t nbins,
                                           Window& n) {
  n.key = key;
  n.strip = key / (uint32_t)g.nsub_side;
  if (n.strip == w.strip) {
    const int adv = (int)(key - w.key) * g.sube;
    n.rb = w.rb + adv;
    n.su0 = w.su0 + adv;
    if (n.su0 >= g.nu) n.su0 -= g.nu;
    n.sv0 = w.sv0;
    n.mp = w.mp;
    return min(adv, 8);
  }
  window_of(g, key, nbins, n.rb, n.su0, n.sv0, n.mp);
  return 8;
}

// The taps t[0..S) placed at rows [off, off + S) of an 8-row window, zero
// elsewhere, in registers (off < 9 - S is a runtime value, the candidates
// compile-time: selects instead of indexed stores).
template <int S, class V>
__device__ __forceinline__ void place8(const V (&t)[S], int off, V zero, V (&row)[8]) {
#pragma unroll
  for (int j = 0; j < 8; j++) {
    V x = zero;
#pragma unroll
    for (int d = 0; d < 9 - S; d++)
      if (j - d >= 0 && j - d < S && off == d) x = t[(j - d >= 0 && j - d < S) ? j - d : 0];
    row[j] = x;
  }
}

// The taps t[0..S) at rows (r + i) mod 8 of a window, zero elsewhere, in
// registers (r is a runtime value: three conditional rotations).
template <int S>
__device__ __forceinline__ void rotate8(const float (&t)[S], int r, float (&row)[8]) {
  float a[8], b[8];
#pragma unroll
  for (int j = 0; j < 8; j++) a[j] = j < S ? t[j < S ? j : 0] : 0.0f;
#pragma unroll
  for (int j = 0; j < 8; j++) b[j] = (r & 1) ? a[(j + 7) & 7] : a[j];
#pragma unroll
  for (int j = 0; j < 8; j++) a[j] = (r & 2) ? b[(j + 6) & 7] : b[j];
#pragma unroll
  for (int j = 0; j < 8; j++) row[j] = (r & 4) ? a[(j + 4) & 7] : a[j];
}

// ------------------------------------------------------------------ prefetch

// The inputs of one staged record, copied asynchronously (cp.async) into
// shared memory a round ahead of their use, so that the gathers of records,
// visibilities and weights are in flight while the previous round is
// contracted and take no registers.
struct Prefetched {
  uint4 rec[2];  // the record
  uint4 vis;     // the visibility: complex64 in .x, .y or complex128
  uint2 wgt;     // the weight: float32 in .x, float64, or the two float32 factors
};

__device__ __forceinline__ void cp_async(void* dst, const void* src, int bytes) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  if (bytes == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src));
  else if (bytes == 8)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src));
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(src));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// Starts the copies of record `idx` (at sorted position k) and (with_vis,
// with_wgt) its value's inputs.
__device__ __forceinline__ void prefetch(Prefetched* dst, const VisRecord* __restrict__ rec, const Inputs& in,
                                         bool with_vis, bool with_wgt, uint32_t idx, uint64_t k) {
  const uint4* r = reinterpret_cast<const uint4*>(rec + idx);
  cp_async(&dst->rec[0], r, 16);
  cp_async(&dst->rec[1], r + 1, 16);
  if (with_vis) {
    if (in.vis_kind == VIS_SORTED)
      cp_async(&dst->vis, reinterpret_cast<const float2*>(in.vis) + k, 8);
    else if (in.vis_kind == VIS_C64)
      cp_async(&dst->vis, reinterpret_cast<const float2*>(in.vis) + idx, 8);
    else if (in.vis_kind == VIS_C128)
      cp_async(&dst->vis, reinterpret_cast<const double2*>(in.vis) + idx, 16);
  }
  if (with_wgt) {
    if (in.wgt_kind == WGT_F64) {
      cp_async(&dst->wgt, reinterpret_cast<const double*>(in.wgt) + idx, 8);
    } else if (in.wgt_kind == WGT_F32 || in.wgt_kind == WGT_F32_PRODUCT) {
      cp_async(&dst->wgt.x, reinterpret_cast<const float*>(in.wgt) + idx, 4);
      if (in.wgt_kind == WGT_F32_PRODUCT) cp_async(&dst->wgt.y, reinterpret_cast<const float*>(in.wgt2) + idx, 4);
    }
  }
}

__device__ __forceinline__ VisRecord prefetched_record(const Prefetched& p) {
  const uint4 a = p.rec[0], b = p.rec[1];
  return VisRecord{__uint_as_float(a.x), __uint_as_float(a.y), __uint_as_float(a.z), a.w,
                   __uint_as_float(b.x), __uint_as_float(b.y), b.z, b.w};
}
// Weights::get and VisData::get (wgridder.rs:950-1005) of the copied values.
__device__ __forceinline__ float prefetched_wgt(const Prefetched& p, const Inputs& in) {
  switch (in.wgt_kind) {
    case WGT_F32:
      return __uint_as_float(p.wgt.x);
    case WGT_F64:
      return (float)__longlong_as_double((long long)(((unsigned long long)p.wgt.y << 32) | p.wgt.x));
    case WGT_F32_PRODUCT:
      return __uint_as_float(p.wgt.x) * __uint_as_float(p.wgt.y);
    default:
      return 1.0f;
  }
}
__device__ __forceinline__ cplx<float> prefetched_vis(const Prefetched& p, const Inputs& in) {
  if (in.vis_kind == VIS_C64 || in.vis_kind == VIS_SORTED) return {__uint_as_float(p.vis.x), __uint_as_float(p.vis.y)};
  if (in.vis_kind == VIS_C128)
    return {(float)__longlong_as_double((long long)(((unsigned long long)p.vis.y << 32) | p.vis.x)),
            (float)__longlong_as_double((long long)(((unsigned long long)p.vis.w << 32) | p.vis.z))};
  return {1.0f, 0.0f};
}

// ------------------------------------------------------------------ integer gridder

// Warps per block: each takes some of the support's plane pairs, and the block
// stages its records once, one per thread.
__host__ __device__ constexpr int i8_warps(int S) { return S >= 7 ? 2 : 1; }
__host__ __device__ constexpr int i8_pairs(int S) { return ((S + 1) / 2 + i8_warps(S) - 1) / i8_warps(S); }
// Blocks per SM: 12 blocks (168 registers) up to support 6; 54 M visibilities at
// support 8 took 6.18 ms at 9 blocks of two warps (registers spilt) and 6.12 at 8.
__host__ __device__ constexpr int i8_blocks(int S) { return S <= 4 ? 16 : S <= 6 ? 12 : 8; }  // per SM
constexpr float I8_ASCALE = 4194304.0f;  // 2^22
// A's integers (w tap x u tap x 2^22) are formed without a conversion
// instruction: y = x + 2^23 + 0x8080 lies in [2^23, 2^24), where FP32 spacing is
// 1, so the FFMA that forms x rounds it to the nearest integer, and the low
// three bytes of y's bits are those of rint(x) + 0x8080, the offset the
// balanced limbs need. The taps of every kernel of the table are positive on
// [-1, 1] and at most 1 + eps, so x lies far inside [-0x8080, 2^23 - 0x8080).
constexpr float I8_AOFF = 8421504.0f;  // 2^23 + 0x8080
// One staged record, in words: value * v taps placed on the window's 8 columns
// (rint(value kv 2^sb) + 0x8080, re and im; the offset elsewhere), the w taps
// times 2^22 (8, read as pairs of planes), the u taps placed on the window's 8
// rows (zero elsewhere). With a stride that is 2 mod 8 the reads of the eight
// records of a lane quad (slots 4 tq + j) fall in distinct banks.
constexpr int I8_SLOT = 42, I8_KW = 18, I8_KU = 28;  // stride; where the w and u taps start
// Staging of one round: N records and their bin keys. Slot N stays zero.
template <int N>
struct I8Slots {
  uint32_t* slot;  // [N + 1][I8_SLOT]
  uint32_t* key;   // [N + 1]
  __host__ __device__ static constexpr size_t bytes() { return ((size_t)(N + 1) * (I8_SLOT + 1) * 4 + 15) / 16 * 16; }
  __device__ void carve(unsigned char* base) {
    slot = reinterpret_cast<uint32_t*>(base);
    key = slot + (N + 1) * I8_SLOT;
  }
};

// Three balanced 8-bit limbs of four integers y - 0x8080 (y = x + 0x8080,
// |x| < 2^22 + 2^15), packed per limb (byte j of limb register L holds limb
// L of x[j]): bytes 0 and 1 of y are the low limbs plus 128, y >> 16 (byte 2
// of y, as a signed byte) is the top limb.
__device__ __forceinline__ void limbs4(uint32_t y0, uint32_t y1, uint32_t y2, uint32_t y3, uint32_t& l0, uint32_t& l1,
                                       uint32_t& l2) {
  const uint32_t a01 = __byte_perm(y0, y1, 0x5140), a23 = __byte_perm(y2, y3, 0x5140);  // b0 b0' b1 b1'
  l0 = __byte_perm(a01, a23, 0x5410) ^ 0x80808080u;
  l1 = __byte_perm(a01, a23, 0x7632) ^ 0x80808080u;
  l2 = __byte_perm(__byte_perm(y0, y1, 0x0062), __byte_perm(y2, y3, 0x0062), 0x5410);
}

__device__ __forceinline__ void imma(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                     uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void imma16(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};\n"
      : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
      : "r"(a0), "r"(a1), "r"(b0));
}

// Adds the first `leave` rows of a window's exact sums to the fixed-point grid
// and clears them. acc[h][c][g][r]: plane pair h0 + h, component c (re, im), limb
// group g (weights 2^32, 2^24, 2^16: the grid unit is 2^16 of the products),
// fragment element r (rows gq / gq + 8 of the MMA are planes 2h / 2h + 1 at the
// window row that is gq mod 8; columns 2tq, 2tq + 1).
//
// The atomics are what bounds sparse bins: L2 takes about one 32-byte sector
// per slice and clock, whatever the number of words added in it. Straight
// from the fragments every 8-byte add was a sector of its own (8 x 8 cells of
// every plane per bin: 19.6 ms for 1.8 M bins of support 8). Through `buf` a
// half-warp adds one row of one plane, 128 contiguous bytes, and only the
// rows the window leaves are added.
constexpr int I8_FLUSH_BYTES = 8 * 2 * 8 * 16;  // [row][plane of the pair][column] cells
template <int NP>
__device__ __forceinline__ void i8_flush(const Geom<float>& g, FixCell* __restrict__ grids, int pg0, int npg,
                                         const Window& w, int leave, int h0, int (&acc)[NP][2][3][4],
                                         unsigned long long* buf) {
  const int lane = threadIdx.x & 31, gq = lane >> 2, tq = lane & 3;
  const int o = (gq - w.rb) & 7;  // this lane's row of the window
  const int e = lane >> 4, word = lane & 15;
  int col = w.sv0 + (word >> 1);
  if (col >= g.nv) col -= g.nv;
  const size_t plane = (size_t)g.nu * g.nv;
#pragma unroll
  for (int h = 0; h < NP; h++) {
    if (o < leave) {
#pragma unroll
      for (int r = 0; r < 4; r++) {
        const long long re = ((long long)acc[h][0][0][r] << 16) + ((long long)acc[h][0][1][r] << 8) + acc[h][0][2][r];
        const long long im = ((long long)acc[h][1][0][r] << 16) + ((long long)acc[h][1][1][r] << 8) + acc[h][1][2][r];
        reinterpret_cast<longlong2*>(buf)[(o * 2 + (r >> 1)) * 8 + 2 * tq + (r & 1)] = make_longlong2(re, im);
#pragma unroll
        for (int q = 0; q < 3; q++) acc[h][0][q][r] = acc[h][1][q][r] = 0;
      }
    }
    __syncwarp();
    const int p = w.mp + 2 * (h0 + h) + e;
    const bool ok = p >= pg0 && p < pg0 + npg;
    unsigned long long* base = reinterpret_cast<unsigned long long*>(grids + (size_t)(ok ? p - pg0 : 0) * plane + col) +
                               (word & 1);
    for (int i = 0; i < leave; i++) {
      const unsigned long long v = buf[i * 32 + lane];
      int row = w.su0 + i;
      if (row >= g.nu) row -= g.nu;
      if (ok && v) atomicAdd(base + (size_t)row * g.nv * 2, v);
    }
    __syncwarp();
  }
}

// The limb products of a run's first 16 HF records (slots q .. q + len - 1, the
// zero slot past them; FULL: all 16 HF of them) added to the window's fragments.
template <int NP, int HF, bool FULL, int N>
__device__ __forceinline__ void i8_contract(const I8Slots<N>& st, int q, int len, int h0, int (&acc)[NP][2][3][4]) {
  const int lane = threadIdx.x & 31, gq = lane >> 2, tq = lane & 3;
  // This lane's records: k = 4tq + j and 16 + 4tq + j, j < 4.
  int rec[4 * HF];  // where their slots start
  const int first = (q + 4 * tq) * I8_SLOT;
#pragma unroll
  for (int j = 0; j < 4 * HF; j++) {
    const int k = j < 4 ? j : 12 + j;  // past 4tq
    rec[j] = FULL || 4 * tq + k < len ? first + k * I8_SLOT : N * I8_SLOT;
  }
  float kuv[4 * HF];
  uint32_t b[2][3][HF];  // B limbs per component: registers for k 4tq.. and 16 + 4tq..
#pragma unroll
  for (int hf = 0; hf < HF; hf++) {
    uint2 bvv[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      kuv[4 * hf + j] = __uint_as_float(st.slot[rec[4 * hf + j] + I8_KU + gq]);
      bvv[j] = *reinterpret_cast<const uint2*>(st.slot + rec[4 * hf + j] + 2 * gq);
    }
    limbs4(bvv[0].x, bvv[1].x, bvv[2].x, bvv[3].x, b[0][0][hf], b[0][1][hf], b[0][2][hf]);
    limbs4(bvv[0].y, bvv[1].y, bvv[2].y, bvv[3].y, b[1][0][hf], b[1][1][hf], b[1][2][hf]);
  }
#pragma unroll
  for (int h = 0; h < NP; h++) {
    uint32_t a[3][2 * HF];  // per limb: rows gq (plane 2h), gq + 8 (plane 2h + 1) x k halves
#pragma unroll
    for (int hf = 0; hf < HF; hf++) {
      uint32_t x[4], y[4];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const float2 w = *reinterpret_cast<const float2*>(st.slot + rec[4 * hf + j] + I8_KW + 2 * (h0 + h));
        x[j] = __float_as_uint(fmaf(w.x, kuv[4 * hf + j], I8_AOFF));
        y[j] = __float_as_uint(fmaf(w.y, kuv[4 * hf + j], I8_AOFF));
      }
      limbs4(x[0], x[1], x[2], x[3], a[0][2 * hf], a[1][2 * hf], a[2][2 * hf]);
      limbs4(y[0], y[1], y[2], y[3], a[0][2 * hf + 1], a[1][2 * hf + 1], a[2][2 * hf + 1]);
    }
#pragma unroll
    for (int c = 0; c < 2; c++) {
      // weight 2^32: a2 b2; 2^24: a2 b1 + a1 b2; 2^16: a2 b0 + a1 b1 + a0 b2
#pragma unroll
      for (int gr = 0; gr < 3; gr++)
#pragma unroll
        for (int i = 0; i <= gr; i++) {
          const uint32_t (&av)[2 * HF] = a[2 - i];
          const uint32_t (&bl)[HF] = b[c][2 - gr + i];
          if constexpr (HF == 2)
            imma(acc[h][c][gr], av[0], av[1], av[2], av[3], bl[0], bl[1]);
          else
            imma16(acc[h][c][gr], av[0], av[1], bl[0]);
        }
    }
  }
}

// A barrier of W warps.
template <int W>
__device__ __forceinline__ void block_sync() {
  if constexpr (W == 1)
    __syncwarp();
  else
    __syncthreads();
}

// Gridding of records [kbase, kend) (single precision): each block takes
// `chunk` consecutive sorted records, stages one per thread at a time, and per run
// of one bin forms the integer limbs of A (rows: w tap x placed u tap of
// planes 2h and 2h + 1, columns: the run's records) and B (rows: records,
// columns: value x placed v tap) and adds their limb products into int32
// fragments on the tensor cores; when the window moves to the next bin, the
// rows it leaves are combined into int64 and added to the grid. Records
// outside the run read the zero slot; runs of at most 16 take the MMAs of
// half the depth. The next round's records and values are loaded while the
// current round is contracted.
//
// It is bound by the latency of its own chains at 11 warps per SM: on 106 M
// active visibilities of support 6 54 % of the issue slots and 24 % of the
// integer tensor pipe are used. 1.06 G visibilities of support 6 took
// 31.3 ms while every bin flushed its whole window and staging ran on scalar
// multiply-adds in blocks of 8192 records, 26.2 now; 54 M of support 8, where
// bins are sparse and the flush's atomics were the bound, 19.6 and 6.1.
template <int S>
__global__ void __launch_bounds__(32 * i8_warps(S), i8_blocks(S))
    k_grid_i8(const __grid_constant__ Geom<float> g, Inputs in, int mode, const VisRecord* __restrict__ rec,
              const uint32_t* __restrict__ sorted, uint64_t kbase, uint64_t kend, uint32_t chunk, uint32_t nbins,
              FixCell* __restrict__ grids, int pg0, int npg, FixScale* __restrict__ fs,
              const int* __restrict__ run, const __grid_constant__ TapPairs<S> taps) {
  static_assert(S >= 1 && S <= 8, "8 x 8 windows");
  if (run && *run == 0) return;  // a speculative pass's regridding, not needed
  constexpr int W = i8_warps(S), N = 32 * W;
  constexpr int NP = i8_pairs(S);  // plane pairs of each warp
  extern __shared__ __align__(16) unsigned char smem[];
  const int tid = threadIdx.x, lane = tid & 31, h0 = (tid >> 5) * NP;
  unsigned long long* flush_buf = reinterpret_cast<unsigned long long*>(smem + (tid >> 5) * I8_FLUSH_BYTES);
  I8Slots<N> st;
  st.carve(smem + W * I8_FLUSH_BYTES);
  // the zero slot: u and w taps 0, B columns at the offset (value 0)
  if (tid < I8_SLOT) st.slot[N * I8_SLOT + tid] = tid < 16 ? 0x8080u : 0u;
  if (I8_SLOT > 32 * W && tid + 32 * W < I8_SLOT) st.slot[N * I8_SLOT + tid + 32 * W] = 0u;
  if (tid == 0) st.key[N] = INACTIVE;
  const uint64_t k0 = kbase + (uint64_t)blockIdx.x * chunk;
  const uint64_t k1 = min(kend, k0 + chunk);
  const float bscale = ldexpf(1.0f, fs->sb);
  float bad = 0.0f;  // NaN once a value or a tap's argument was not finite

  int acc[NP][2][3][4];
#pragma unroll
  for (int h = 0; h < NP; h++)
#pragma unroll
    for (int c = 0; c < 2; c++)
#pragma unroll
      for (int q = 0; q < 3; q++)
#pragma unroll
        for (int r = 0; r < 4; r++) acc[h][c][q][r] = 0;
  Window win;

  // Rounds ahead: this round's inputs are in pre (copied asynchronously),
  // nidx is the next round's index.
  Prefetched* pre = reinterpret_cast<Prefetched*>(smem + W * I8_FLUSH_BYTES + I8Slots<N>::bytes()) + tid;
  const bool with_vis = mode == VALUE_DATA && in.vis_kind != VIS_UNIT, with_wgt = in.wgt_kind != WGT_NONE;
  if (k0 + tid < k1) prefetch(pre, rec, in, with_vis, with_wgt, sorted[k0 + tid], k0 + tid);
  cp_async_commit();
  uint32_t nidx = (k0 + N + tid < k1) ? sorted[k0 + N + tid] : 0u;

  for (uint64_t kb = k0; kb < k1; kb += N) {
    const int nb = (int)min((uint64_t)N, k1 - kb);
    cp_async_wait_all();
    block_sync<W>();
    if (tid < nb) {  // staging, one record per thread
      const VisRecord r = prefetched_record(*pre);
      const float wt = prefetched_wgt(*pre, in);
      const cplx<float> vv = with_vis ? prefetched_vis(*pre, in) : cplx<float>{1.0f, 0.0f};
      float ku[S], kv[S], kw[S];
      eval_taps_pairs<S>(taps, r.x0, ku);
      eval_taps_pairs<S>(taps, r.y0, kv);
      if (g.do_wgridding) eval_taps_pairs<S>(taps, r.xw, kw);
      // record_value: value = vis * phase * wgt, imaginary part negated where w was flipped.
      const float flip = (r.meta & 256u) ? -1.0f : 1.0f;
      const float pr = r.ph_re * wt, pi = r.ph_im * wt;
      const float vr = vv.re * pr - vv.im * pi, vi = (vv.re * pi + vv.im * pr) * flip;
      // Zero times anything that is not finite is NaN, and stays.
      bad = fmaf(vr, 0.0f, fmaf(vi, 0.0f, fmaf(r.x0, 0.0f, fmaf(r.y0, 0.0f, fmaf(r.xw, 0.0f, bad)))));
      const uint32_t ur = (r.meta >> 9) & 7u, dv = (r.meta >> 4) & 15u;
      const float br = vr * bscale, bi = vi * bscale;
      uint32_t* rec = st.slot + tid * I8_SLOT;
      // The value's columns dv .. dv + S - 1, the offset in the others. Planes
      // outside this pass's are left to the flush, which drops them.
      uint2* cb = reinterpret_cast<uint2*>(rec);
#pragma unroll
      for (int i = S; i < 8; i++) cb[(dv + i) & 7u] = make_uint2(0x8080u, 0x8080u);
      cb += dv;
#pragma unroll
      for (int i = 0; i < S; i++)
        cb[i] = make_uint2((uint32_t)(__float2int_rn(br * kv[i]) + 0x8080), (uint32_t)(__float2int_rn(bi * kv[i]) + 0x8080));
      float urow[8];
      rotate8<S>(ku, (int)ur, urow);
      float2* cu = reinterpret_cast<float2*>(rec + I8_KU);
      float2* cw = reinterpret_cast<float2*>(rec + I8_KW);
#pragma unroll
      for (int j = 0; j < 4; j++) {
        cu[j] = make_float2(urow[2 * j], urow[2 * j + 1]);
        float2 w = make_float2(0.0f, 0.0f);
        if (g.do_wgridding) {
          if (2 * j < S) w.x = kw[2 * j < S ? 2 * j : 0] * I8_ASCALE;
          if (2 * j + 1 < S) w.y = kw[2 * j + 1 < S ? 2 * j + 1 : 0] * I8_ASCALE;
        } else if (j == 0) {
          w.x = I8_ASCALE;
        }
        cw[j] = w;
      }
      st.key[tid] = r.bin;
    }
    // The next round's record and value, in flight while this one is contracted.
    block_sync<W>();
    if (kb + N + tid < k1) prefetch(pre, rec, in, with_vis, with_wgt, nidx, kb + N + tid);
    cp_async_commit();
    if (kb + 2 * N + tid < k1) nidx = sorted[kb + 2 * N + tid];
    int q = 0;
    while (q < nb) {
      const uint32_t gk = st.key[q];
      if (gk != win.key) {
        Window next;
        const int leave = window_step(g, win, gk, nbins, next);
        if (win.key != INACTIVE) i8_flush<NP>(g, grids, pg0, npg, win, leave, h0, acc, flush_buf);
        win = next;
      }
      // The run: slots [q, q + len) of bin gk, at most 32.
      const unsigned m = __ballot_sync(0xffffffffu, q + lane < nb && st.key[q + lane] == gk);
      const int len = __popc(m);
      if (len == 32)
        i8_contract<NP, 2, true>(st, q, len, h0, acc);
      else if (len > 16)
        i8_contract<NP, 2, false>(st, q, len, h0, acc);
      else
        i8_contract<NP, 1, false>(st, q, len, h0, acc);
      q += len;
    }
  }
  if (win.key != INACTIVE) i8_flush<NP>(g, grids, pg0, npg, win, 8, h0, acc, flush_buf);
  if (__any_sync(0xffffffffu, bad != 0.0f) && lane == 0) atomicOr(&fs->nonfinite, 1);
}

// ------------------------------------------------------------------ tensor-core degridder

constexpr int H16_BATCH = 32;
constexpr float H16_BSCALE = 16384.0f;  // 2^14: v taps stay clear of FP16 subnormals
constexpr int h16_blocks(int S) { return S <= 6 ? 24 : 16; }  // one-warp blocks per SM
constexpr int H16_KU = 10;  // u taps placed on the window's 8 rows (read as float2)
constexpr int H16_KV = 10;  // v taps * 2^14 placed on the 8 columns (read as float2)
constexpr int H16_KW = 12;  // w taps (8, read as float4)

struct H16Slots {
  float4* out;    // [H16_BATCH + 1]: conj(phase) * wgt (re, im), imflip, index bits
  float* kw;      // [H16_BATCH + 1][H16_KW]: w taps (zero outside the pass's planes)
  float* kv;      // [H16_BATCH + 1][H16_KV]
  float* ku;      // [H16_BATCH + 1][H16_KU]
  uint32_t* key;  // [H16_BATCH + 1]
  __host__ __device__ static constexpr size_t bytes() {
    return ((size_t)(H16_BATCH + 1) * (16 + H16_KW * 4 + H16_KV * 4 + H16_KU * 4 + 4) + 15) / 16 * 16;
  }
  // out and kw are read as float4, kv and ku as float2: their offsets are aligned.
  __device__ void carve(unsigned char* base) {
    out = reinterpret_cast<float4*>(base);
    kw = reinterpret_cast<float*>(out + (H16_BATCH + 1));
    kv = kw + (H16_BATCH + 1) * H16_KW;
    ku = kv + (H16_BATCH + 1) * H16_KV;
    key = reinterpret_cast<uint32_t*>(ku + (H16_BATCH + 1) * H16_KU);
  }
};

// (x0, x1) as FP16 hi + lo (x - hi is exact in FP32; lo rounds it to FP16).
__device__ __forceinline__ void split_h2(float x0, float x1, uint32_t& hi, uint32_t& lo) {
  const __half2 h = __floats2half2_rn(x0, x1);
  const float2 hf = __half22float2(h);
  const __half2 l = __floats2half2_rn(x0 - hf.x, x1 - hf.y);
  hi = *reinterpret_cast<const uint32_t*>(&h);
  lo = *reinterpret_cast<const uint32_t*>(&l);
}

__device__ __forceinline__ void hmma_zero(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};\n"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a0), "r"(a1), "r"(b0), "f"(0.0f));
}
__device__ __forceinline__ void hmma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(b0));
}

// Where the degridder's results go. DEGRID_TO_VIS: vis[visibility index],
// times the weights of the call. The two other modes write the plan's stored
// values, indexed by sorted position, for the gridder to read back
// (Prepared::residual, wgridder.rs:3297-3395): DEGRID_GRAM stores w A x
// (the prediction times the weight of `data`), DEGRID_RESIDUAL stores
// w (d - A x) with d the visibility of `data`; both add w |stored / w|^2 into
// an FP64 partial per block (partials[block0 + block], summed by the warp in
// a fixed order) and the largest |stored| into `bound`.
enum DegridMode : int { DEGRID_TO_VIS = 0, DEGRID_GRAM = 1, DEGRID_RESIDUAL = 2 };
struct DegridOut {
  int mode = DEGRID_TO_VIS;
  cplx<float>* vis = nullptr;     // DEGRID_TO_VIS
  cplx<float>* stored = nullptr;  // the other modes
  Inputs data;                    // weights (and visibilities) of the stored modes
  int sorted_data = 0;            // data and weights by sorted position, not by visibility index
  double* partials = nullptr;
  uint32_t block0 = 0;
  ValueBound* bound = nullptr;
};

// Degridding of records [kbase, kend) (single precision, degrid_task_body,
// wgridder.rs:2793-2901): the warp holds the current bin's 8 x 8 window of
// each plane as FP16 hi + lo fragments, each row (of all planes) scaled by a
// power of two to its largest value; per block of sixteen records the v
// contraction T[k][u] = sum_v kv_k[v - dv_k] G_p[u][v] of each plane runs on
// the tensor cores as hi*hi + hi*lo + lo*hi (mma.sync m16n8k8, records along M,
// window rows along N, FP32 accumulation, each block from zero); the u and w
// contractions and the final phase and weight (wgridder.rs:3146-3159) run on
// the CUDA cores, reduced over the four lanes that hold a record's window
// rows. Window rows sit at u mod 8, so the next bin of a strip reads only the
// rows it adds. Each output depends only on its own record and its window
// rows, so the result does not depend on the grouping. With plane groups
// (first / last) the partial sums accumulate in `vis` and the final factor is
// applied with the last group. The next round's records are copied while the
// current round is contracted. `out` says where the results go (DegridOut). Up
// to support 6, 24 warps per SM (80 registers) measured 4 % faster than 16 (122
// registers) and 20 (96), and as fast as 28. The w contraction before the u
// taps and one output lane per record (two lanes of each quad) measured 10 %
// faster than u first and one lane writing both records. From support 7, 16
// (128 registers) against 12 took 5.5 ms against 6.1 at 54 M visibilities. That
// call took 12.5 ms while a warp read the whole window of every bin; 1.06 G
// visibilities of support 6, 27.6 then and 26.3 now. It is bound by issue and the
// FP16 tensor pipe: 65 % of the slots and 51 % of the pipe on 106 M active
// visibilities of support 6.
template <int S>
__global__ void __launch_bounds__(H16_BATCH, h16_blocks(S))
    k_degrid_h(const __grid_constant__ Geom<float> g, Inputs wts, const VisRecord* __restrict__ rec,
               const uint32_t* __restrict__ sorted, uint64_t kbase, uint64_t kend, uint32_t chunk, uint32_t nbins,
               const cplx<float>* __restrict__ grids, int pg0, int npg, const __grid_constant__ DegridOut out,
               int first, int last, const uint32_t* __restrict__ kb_ptr, const uint32_t* __restrict__ ke_ptr,
               const __grid_constant__ TapPairs<S> taps) {
  static_assert(S >= 1 && S <= 8, "8 x 8 windows");
  if (kb_ptr) {  // a range the device computed: the grid covers its largest size
    kbase = *kb_ptr;
    kend = *ke_ptr;
    if (kbase + (uint64_t)blockIdx.x * chunk >= kend) return;
  }
  extern __shared__ __align__(16) unsigned char smem[];
  H16Slots st;
  st.carve(smem);
  const int lane = threadIdx.x, gq = lane >> 2, tq = lane & 3;
  {  // the zero slot
    if (lane < H16_KW) st.kw[H16_BATCH * H16_KW + lane] = 0.0f;
    if (lane < H16_KV) st.kv[H16_BATCH * H16_KV + lane] = 0.0f;
    if (lane < H16_KU) st.ku[H16_BATCH * H16_KU + lane] = 0.0f;
    if (lane == 0) {
      st.key[H16_BATCH] = INACTIVE;
      st.out[H16_BATCH] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
  }
  const uint64_t k0 = kbase + (uint64_t)blockIdx.x * chunk;
  const uint64_t k1 = min(kend, k0 + chunk);
  const size_t plane = (size_t)g.nu * g.nv;

  uint32_t bhi[S][2], blo[S][2];  // [plane][re/im]: window row gq (mod 8), columns 2tq, 2tq + 1
  float inv = 0.0f;               // 1 / (row gq's scale * 2^14)
  float2 invp = {0.0f, 0.0f};     // the same of rows 2tq, 2tq + 1
  Window win;
  double part = 0.0, vmax = 0.0;  // the stored modes' misfit partial and largest |stored|

  Prefetched* pre = reinterpret_cast<Prefetched*>(smem + H16Slots::bytes()) + lane;
  const bool with_wgt = wts.wgt_kind != WGT_NONE;
  if (k0 + lane < k1) prefetch(pre, rec, wts, false, with_wgt, sorted[k0 + lane], k0 + lane);
  cp_async_commit();
  uint32_t nidx = (k0 + H16_BATCH + lane < k1) ? sorted[k0 + H16_BATCH + lane] : 0u;

  for (uint64_t kb = k0; kb < k1; kb += H16_BATCH) {
    const int nb = (int)min((uint64_t)H16_BATCH, k1 - kb);
    cp_async_wait_all();
    __syncwarp();
    if (lane < nb) {
      const VisRecord r = prefetched_record(*pre);
      const float tw = prefetched_wgt(*pre, wts);
      float ku[S], kv[S], kw[S];
      eval_taps_pairs<S>(taps, r.x0, ku);
      eval_taps_pairs<S>(taps, r.y0, kv);
      if (g.do_wgridding) eval_taps_pairs<S>(taps, r.xw, kw);
      const int ur = (int)((r.meta >> 9) & 7u), dv = (int)((r.meta >> 4) & 15u);
#pragma unroll
      for (int i = 0; i < S; i++) kv[i] *= H16_BSCALE;
      float urow[8], vrow[8], wrow[8];
      rotate8<S>(ku, ur, urow);
      place8<S>(kv, dv, 0.0f, vrow);
#pragma unroll
      for (int j = 0; j < 8; j++) {
        // Planes outside this pass's are zero in the window.
        float w = 0.0f;
        if (g.do_wgridding) {
          if (j < S) w = kw[j < S ? j : 0];
        } else if (j == 0) {
          w = 1.0f;
        }
        wrow[j] = w;
      }
      float2* cu = reinterpret_cast<float2*>(st.ku + lane * H16_KU);
      float2* cv = reinterpret_cast<float2*>(st.kv + lane * H16_KV);
      float4* cw = reinterpret_cast<float4*>(st.kw + lane * H16_KW);
#pragma unroll
      for (int j = 0; j < 4; j++) {
        cu[j] = make_float2(urow[2 * j], urow[2 * j + 1]);
        cv[j] = make_float2(vrow[2 * j], vrow[2 * j + 1]);
      }
      cw[0] = make_float4(wrow[0], wrow[1], wrow[2], wrow[3]);
      cw[1] = make_float4(wrow[4], wrow[5], wrow[6], wrow[7]);
      // The final factor conj(phase) * wgt (shift_phase with sign -1).
      st.out[lane] = make_float4(r.ph_re * tw, -r.ph_im * tw, (r.meta & 256u) ? -1.0f : 1.0f,
                                 __uint_as_float(r.idx));
      st.key[lane] = r.bin;
    }
    __syncwarp();
    if (kb + H16_BATCH + lane < k1) prefetch(pre, rec, wts, false, with_wgt, nidx, kb + H16_BATCH + lane);
    cp_async_commit();
    if (kb + 2 * H16_BATCH + lane < k1) nidx = sorted[kb + 2 * H16_BATCH + lane];
    int q = 0;
    while (q < nb) {
      const uint32_t gk = st.key[q];
      if (gk != win.key) {  // read the rows that bin gk adds to the window, as FP16 fragments
        Window next;
        const int enter = window_step(g, win, gk, nbins, next);
        win = next;
        const int o = (gq - win.rb) & 7;  // this lane's row of the window
        const bool mine = o >= 8 - enter;
        int row = win.su0 + o;
        if (row >= g.nu) row -= g.nu;
        int c0 = win.sv0 + 2 * tq, c1 = c0 + 1;
        if (c0 >= g.nv) c0 -= g.nv;
        if (c1 >= g.nv) c1 -= g.nv;
        cplx<float> v[S][2];  // [plane][column]
        float m = 0.0f;
#pragma unroll
        for (int p = 0; p < S; p++) {
          const int pp = win.mp + p;
          const bool ok = mine && pp >= pg0 && pp < pg0 + npg && (g.do_wgridding || pp == 0);
          const cplx<float>* src = grids + (size_t)(ok ? pp - pg0 : 0) * plane + (size_t)row * g.nv;
          v[p][0] = ok ? src[c0] : cplx<float>{0.0f, 0.0f};
          v[p][1] = ok ? src[c1] : cplx<float>{0.0f, 0.0f};
          m = fmaxf(m, fmaxf(fmaxf(fabsf(v[p][0].re), fabsf(v[p][0].im)), fmaxf(fabsf(v[p][1].re), fabsf(v[p][1].im))));
        }
        m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
        m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
        if (mine) {
          // The row's largest value to about 2^14 (FP16 tops out at 65504).
          const int e = (m > 0.0f && isfinite(m)) ? max(ilogbf(m), -100) : 0;
          const float sc = ldexpf(1.0f, 14 - e);
          inv = ldexpf(1.0f, e - 14) / H16_BSCALE;
#pragma unroll
          for (int p = 0; p < S; p++) {
            split_h2(v[p][0].re * sc, v[p][1].re * sc, bhi[p][0], blo[p][0]);
            split_h2(v[p][0].im * sc, v[p][1].im * sc, bhi[p][1], blo[p][1]);
          }
        }
        invp.x = __shfl_sync(0xffffffffu, inv, 8 * tq);
        invp.y = __shfl_sync(0xffffffffu, inv, 8 * tq + 4);
      }
      const unsigned mk = __ballot_sync(0xffffffffu, lane >= q && lane < nb && st.key[lane] == gk);
      const int len = __popc(mk);
      // Blocks of sixteen records of the run: rows gq and gq + 8 of the MMA.
      for (int k16 = q; k16 < q + len; k16 += 16) {
        int sr[2];
        uint32_t ahi[2], alo[2];
        float2 kup[2];
        float kwv[2][8];
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int k = k16 + gq + 8 * h;
          sr[h] = (k < q + len) ? k : H16_BATCH;
          const float2 kvp = *reinterpret_cast<const float2*>(st.kv + sr[h] * H16_KV + 2 * tq);
          split_h2(kvp.x, kvp.y, ahi[h], alo[h]);
          kup[h] = *reinterpret_cast<const float2*>(st.ku + sr[h] * H16_KU + 2 * tq);
          const float4 w0 = *reinterpret_cast<const float4*>(st.kw + sr[h] * H16_KW);
          const float4 w1 = *reinterpret_cast<const float4*>(st.kw + sr[h] * H16_KW + 4);
          kwv[h][0] = w0.x;
          kwv[h][1] = w0.y;
          kwv[h][2] = w0.z;
          kwv[h][3] = w0.w;
          kwv[h][4] = w1.x;
          kwv[h][5] = w1.y;
          kwv[h][6] = w1.z;
          kwv[h][7] = w1.w;
        }
        // The w contraction first (per window row, over the planes), then the
        // u taps: two FMAs per plane and output instead of three.
        float wr[2][2] = {{0.0f, 0.0f}, {0.0f, 0.0f}}, wi[2][2] = {{0.0f, 0.0f}, {0.0f, 0.0f}};
#pragma unroll
        for (int p = 0; p < S; p++) {
          float dre[4], dim[4];
          hmma_zero(dre, ahi[0], ahi[1], bhi[p][0]);
          hmma(dre, ahi[0], ahi[1], blo[p][0]);
          hmma(dre, alo[0], alo[1], bhi[p][0]);
          hmma_zero(dim, ahi[0], ahi[1], bhi[p][1]);
          hmma(dim, ahi[0], ahi[1], blo[p][1]);
          hmma(dim, alo[0], alo[1], bhi[p][1]);
          // d[0], d[1]: record gq, window rows 2tq, 2tq + 1; d[2], d[3]: record gq + 8
#pragma unroll
          for (int h = 0; h < 2; h++)
#pragma unroll
            for (int c = 0; c < 2; c++) {
              wr[h][c] = fmaf(kwv[h][p], dre[2 * h + c], wr[h][c]);
              wi[h][c] = fmaf(kwv[h][p], dim[2 * h + c], wi[h][c]);
            }
        }
        float tr[2], ti[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
          tr[h] = fmaf(kup[h].x, wr[h][0] * invp.x, kup[h].y * (wr[h][1] * invp.y));
          ti[h] = fmaf(kup[h].x, wi[h][0] * invp.x, kup[h].y * (wi[h][1] * invp.y));
        }
        // Odd lanes of a quad take record gq + 8, even ones record gq: each
        // gives the other's half away, then the two halves of its own are added.
        const bool odd = tq & 1;
        float sr_ = odd ? tr[1] : tr[0], si_ = odd ? ti[1] : ti[0];
        sr_ += __shfl_xor_sync(0xffffffffu, odd ? tr[0] : tr[1], 1);
        si_ += __shfl_xor_sync(0xffffffffu, odd ? ti[0] : ti[1], 1);
        sr_ += __shfl_xor_sync(0xffffffffu, sr_, 2);
        si_ += __shfl_xor_sync(0xffffffffu, si_, 2);
        const int slot = odd ? sr[1] : sr[0];
        if (tq < 2 && slot != H16_BATCH) {
          {
            const float4 fo = st.out[slot];
            const uint32_t idx = __float_as_uint(fo.w);
            const uint64_t k = kb + (uint64_t)slot;
            cplx<float>* dst = out.mode == DEGRID_TO_VIS ? out.vis + idx : out.stored + k;
            cplx<float> accv{sr_, si_ * fo.z};
            if (!first) {
              const cplx<float> prev = *dst;
              accv = {accv.re + prev.re, accv.im + prev.im};
            }
            if (last) {
              accv = {accv.re * fo.x - accv.im * fo.y, accv.re * fo.y + accv.im * fo.x};
              if (out.mode != DEGRID_TO_VIS) {
                const uint64_t di = out.sorted_data ? k : (uint64_t)idx;
                const float w = wgt_get<float>(out.data, di);
                if (out.mode == DEGRID_RESIDUAL) {
                  const cplx<float> d = vis_get<float>(out.data, di);
                  accv = {d.re - accv.re, d.im - accv.im};
                }
                part += (double)w * ((double)accv.re * (double)accv.re + (double)accv.im * (double)accv.im);
                accv = {accv.re * w, accv.im * w};
                vmax = fmax(vmax, sqrt((double)accv.re * (double)accv.re + (double)accv.im * (double)accv.im));
              }
            }
            *dst = accv;
          }
        }
      }
      q += len;
    }
  }
  if (out.mode != DEGRID_TO_VIS && last) {
    for (int o = 16; o > 0; o >>= 1) {
      part += __shfl_down_sync(0xffffffffu, part, o);
      vmax = fmax(vmax, __shfl_down_sync(0xffffffffu, vmax, o));
    }
    if (lane == 0) {
      out.partials[out.block0 + blockIdx.x] = part;
      atomic_max_double(&out.bound->vmax_bits, vmax);
    }
  }
}

// ------------------------------------------------------------------ residual without a model, and sums

constexpr uint32_t STORE_CHUNK = 8192;  // sorted positions per block of k_store_values
constexpr int STORE_THREADS = 256;

// Fixed-order sum of one value per thread of a block into thread 0.
__device__ __forceinline__ double block_sum(double v, double* sh) {
  sh[threadIdx.x] = v;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
    __syncthreads();
  }
  return sh[0];
}

// The residual of the data alone (no model): stored[k] = w d for the
// visibility at sorted position k, w |d|^2 summed into partials[block]
// (each block takes STORE_CHUNK positions, each thread a fixed stride of
// them, then a fixed tree), and the largest |stored| into `bound`.
__global__ void __launch_bounds__(STORE_THREADS)
    k_store_values(uint64_t n, const uint32_t* __restrict__ sorted, Inputs data, int sorted_data,
                   cplx<float>* __restrict__ stored, double* __restrict__ partials, ValueBound* bound) {
  __shared__ double sh[STORE_THREADS];
  const uint64_t k0 = (uint64_t)blockIdx.x * STORE_CHUNK, k1 = min(n, k0 + STORE_CHUNK);
  double part = 0.0, vmax = 0.0;
  for (uint64_t k = k0 + threadIdx.x; k < k1; k += STORE_THREADS) {
    const uint64_t di = sorted_data ? k : (uint64_t)sorted[k];
    const float w = wgt_get<float>(data, di);
    const cplx<float> d = vis_get<float>(data, di);
    part += (double)w * ((double)d.re * (double)d.re + (double)d.im * (double)d.im);
    const cplx<float> v{d.re * w, d.im * w};
    vmax = fmax(vmax, sqrt((double)v.re * (double)v.re + (double)v.im * (double)v.im));
    stored[k] = v;
  }
  const double sum = block_sum(part, sh);
  if (threadIdx.x == 0) partials[blockIdx.x] = sum;
  for (int o = 16; o > 0; o >>= 1) vmax = fmax(vmax, __shfl_down_sync(0xffffffffu, vmax, o));
  if ((threadIdx.x & 31) == 0) atomic_max_double(&bound->vmax_bits, vmax);
}

// out = sum of partials[0, n) in a fixed order (one block).
__global__ void __launch_bounds__(STORE_THREADS) k_sum_partials(const double* __restrict__ partials, uint32_t n,
                                                                 double* out) {
  __shared__ double sh[STORE_THREADS];
  double v = 0.0;
#pragma unroll 8
  for (uint32_t i = threadIdx.x; i < n; i += STORE_THREADS) v += partials[i];
  const double s = block_sum(v, sh);
  if (threadIdx.x == 0) *out = s;
}

}  // namespace fast
