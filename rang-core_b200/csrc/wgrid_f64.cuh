// The double-precision gridder and degridder on the FP64 tensor cores.
//
// Included by wgrid_plan.cu inside its anonymous namespace, after
// wgrid_fast.cuh (it uses the fixed-point grid, the windows and the device
// helpers defined there).
//
// A double-precision plan's sorted order is stable (a radix sort by bin key,
// so the visibilities of a bin keep their index order) and every warp takes
// a fixed range of it, so each warp meets the same records in the same
// order on every call. Per run of one bin the warp accumulates the bin's
// 8 x 8 window of each of its S planes on the FP64 tensor cores
// (mma.sync m16n8k8: rows the window's u cells on two planes, columns its v
// cells, k eight records: A = w tap x placed u taps, B = value x placed v taps),
// so the run's sums are formed in one fixed order, in FP64 as the reference forms them.
// When the window moves on, the rows it leaves are added to the 128-bit
// fixed-point grid (each sum rounded once into the grid's unit; integer adds,
// exact in any order), so the result does not depend on how the warps' atomic
// adds interleave: a call is reproducible bit for bit.

namespace fast {

constexpr int F64_BATCH = 32;        // records staged per round, one per lane
constexpr int F64_BLOCKS = 12;       // one-warp blocks per SM
// Doubles per staged row of 8: the odd stride spreads the lanes' stores over
// the banks; the w taps' rows are read as double2.
constexpr int F64_ROW = 9, F64_KW = 10;
constexpr int F64_FLUSH_BYTES = 4 * 8 * 8 * 16;  // four planes' sums, [plane][row][column][re, im]

// Per slot (record): the u taps placed on the window's 8 rows, Re and Im of
// value x v taps placed on its 8 columns, the w taps of the S planes (zero
// outside the pass's planes) and the bin key. Slot F64_BATCH stays zero.
struct F64Slots {
  double* ku;
  double* bre;
  double* bim;
  double* kw;
  uint32_t* key;
  __host__ __device__ static constexpr size_t bytes() {
    return ((size_t)(F64_BATCH + 1) * ((3 * F64_ROW + F64_KW) * 8 + 4) + 15) / 16 * 16;
  }
  __device__ void carve(unsigned char* base) {
    kw = reinterpret_cast<double*>(base);
    ku = kw + (F64_BATCH + 1) * F64_KW;
    bre = ku + (F64_BATCH + 1) * F64_ROW;
    bim = bre + (F64_BATCH + 1) * F64_ROW;
    key = reinterpret_cast<uint32_t*>(bim + (F64_BATCH + 1) * F64_ROW);
  }
};

// The inputs of one staged visibility, copied asynchronously (cp.async) a
// round ahead of their use: its row's uvw, its channel's f / c, its value,
// its weight and its bin key.
struct Prefetched64 {
  double uvw[3];
  double foc;
  uint4 vis;  // complex128, or complex64 in .x, .y
  uint2 wgt;  // float64, float32 in .x, or the two float32 factors
  uint32_t key;
  uint32_t idx;
};
static_assert(sizeof(Prefetched64) == 64, "one 64-byte slot per lane");

__device__ __forceinline__ void prefetch64(Prefetched64* dst, const double* __restrict__ uvw,
                                           const double* __restrict__ foc, const Inputs& in, bool with_vis,
                                           bool with_wgt, const uint32_t* __restrict__ key, uint32_t idx,
                                           uint32_t nchan) {
  const uint32_t row = idx / nchan, ch = idx - row * nchan;
  const double* u = uvw + 3 * (size_t)row;
  cp_async(&dst->uvw[0], u, 8);
  cp_async(&dst->uvw[1], u + 1, 8);
  cp_async(&dst->uvw[2], u + 2, 8);
  cp_async(&dst->foc, foc + ch, 8);
  if (with_vis) {
    if (in.vis_kind == VIS_C128)
      cp_async(&dst->vis, reinterpret_cast<const double2*>(in.vis) + idx, 16);
    else if (in.vis_kind == VIS_C64)
      cp_async(&dst->vis, reinterpret_cast<const float2*>(in.vis) + idx, 8);
  }
  if (with_wgt) {
    if (in.wgt_kind == WGT_F64) {
      cp_async(&dst->wgt, reinterpret_cast<const double*>(in.wgt) + idx, 8);
    } else {
      cp_async(&dst->wgt.x, reinterpret_cast<const float*>(in.wgt) + idx, 4);
      if (in.wgt_kind == WGT_F32_PRODUCT) cp_async(&dst->wgt.y, reinterpret_cast<const float*>(in.wgt2) + idx, 4);
    }
  }
  cp_async(&dst->key, key + idx, 4);
  dst->idx = idx;
}

// Weights::get and VisData::get (wgridder.rs:950-1005) in double precision.
__device__ __forceinline__ double prefetched_wgt64(const Prefetched64& p, const Inputs& in) {
  switch (in.wgt_kind) {
    case WGT_F64:
      return __longlong_as_double((long long)(((unsigned long long)p.wgt.y << 32) | p.wgt.x));
    case WGT_F32:
      return (double)__uint_as_float(p.wgt.x);
    case WGT_F32_PRODUCT:
      return (double)(__uint_as_float(p.wgt.x) * __uint_as_float(p.wgt.y));
    default:
      return 1.0;
  }
}
__device__ __forceinline__ cplx<double> prefetched_vis64(const Prefetched64& p, const Inputs& in) {
  if (in.vis_kind == VIS_C128)
    return {__longlong_as_double((long long)(((unsigned long long)p.vis.y << 32) | p.vis.x)),
            __longlong_as_double((long long)(((unsigned long long)p.vis.w << 32) | p.vis.z))};
  if (in.vis_kind == VIS_C64) return {(double)__uint_as_float(p.vis.x), (double)__uint_as_float(p.vis.y)};
  return {1.0, 0.0};
}

// FP64 matrix products, d += a b: eight rows and four of the sum, and sixteen
// rows and four or eight (rows gq, gq + 8; k tq, tq + 4; columns 2 tq, 2 tq + 1).
__device__ __forceinline__ void dmma8x4(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}
__device__ __forceinline__ void dmma16x4(double (&d)[4], double a0, double a1, double b) {
  asm volatile("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};\n"
               : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
               : "d"(a0), "d"(a1), "d"(b));
}
__device__ __forceinline__ void dmma16x8(double (&d)[4], double a0, double a1, double a2, double a3, double b0,
                                         double b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
      : "d"(a0), "d"(a1), "d"(a2), "d"(a3), "d"(b0), "d"(b1));
}

// Adds the first `leave` rows of a window's sums to the 128-bit grid and clears
// them: acc[h][c][2 e + i] is plane mp + 2 h + e, component c, column 2 tq + i of
// the window row that is gq mod 8. As in i8_flush the adds go through shared
// memory, a warp adding one row of one plane (256 contiguous bytes): straight
// from the fragments each 8-byte add was a 32-byte sector of its own in L2
// (4 x 512 adds per bin of support 8). The sums are rounded into the grid's unit
// on the way out, a word per lane, in a loop: rounded by the four lanes that
// hold a row, unrolled over the planes, the code outgrew the instruction cache
// (4.8 of 11 cycles per instruction waiting for it).
template <int S>
__device__ __forceinline__ void f64_flush(const Geom<double>& g, FixCell2* __restrict__ grids, int pg0, int npg,
                                          const Window& w, int leave, double sc, double (&acc)[(S + 1) / 2][2][4],
                                          double* buf) {
  const int lane = threadIdx.x & 31, gq = lane >> 2, tq = lane & 3;
  const int o = (gq - w.rb) & 7;  // this lane's row of the window
  int col = w.sv0 + (lane >> 2);
  if (col >= g.nv) col -= g.nv;
  const size_t plane = (size_t)g.nu * g.nv;
  // This lane's word of a cell: the low or high part of re or im.
  unsigned long long* base =
      reinterpret_cast<unsigned long long*>(grids + (size_t)w.su0 * g.nv + col) + (lane & 3);
#pragma unroll
  for (int p4 = 0; p4 < S; p4 += 4) {
    if (o < leave) {
#pragma unroll
      for (int p = p4; p < p4 + 4 && p < S; p++) {
        double(&re)[4] = acc[p / 2][0];
        double(&im)[4] = acc[p / 2][1];
        const int e = 2 * (p & 1);
        double2* d = reinterpret_cast<double2*>(buf + ((p - p4) * 8 + o) * 16 + 4 * tq);
        d[0] = make_double2(re[e], im[e]);
        d[1] = make_double2(re[e + 1], im[e + 1]);
        re[e] = re[e + 1] = im[e] = im[e + 1] = 0.0;
      }
    }
    __syncwarp();
#pragma unroll 1
    for (int q = 0; q < min(4, S - p4); q++) {
      const int p = w.mp + p4 + q;
      if (p < pg0 || p >= pg0 + npg) continue;
      unsigned long long* cell = base + (size_t)(p - pg0) * plane * 4;
      const double* sum = buf + q * 128 + (lane >> 1);
      int wrap = g.nu - w.su0;  // rows until the grid's last
#pragma unroll 1
      for (int i = 0; i < leave; i++) {
        const double y = sum[16 * i] * sc, h = floor(y);  // FixTraits<double>::term
        const long long v = __double2ll_rn((lane & 1) ? h : (y - h) * 4294967296.0);
        if (v != 0) atomicAdd(cell, (unsigned long long)v);
        cell += (size_t)g.nv * 4;
        if (--wrap == 0) cell -= plane * 4;
      }
    }
    __syncwarp();
  }
}

// Gridding of sorted records [kbase, kend) in double precision (the
// reference's grid_task_body, wgridder.rs:2102-2156, on windows): each warp
// takes `chunk` consecutive sorted visibilities, stages F64_BATCH at a time
// (coordinates, taps and value from uvw and the data, as k_grid does) and
// contracts each run of one bin eight records at a time. It is bound by
// latency at 12 warps per SM, which its registers allow (DMMA 25 % busy): 16.5 M
// visibilities of support 8 took 5.7 ms while every bin flushed its whole
// window, 3.5 with windows that move, 3.3 with the flush in a loop (unrolled it
// outgrew the instruction cache). 8, 10 and 16 warps measured no faster.
template <int S>
__global__ void __launch_bounds__(F64_BATCH, F64_BLOCKS)
    k_grid_f64(const __grid_constant__ Geom<double> g, Inputs in, int mode, const double* __restrict__ uvw,
               const double* __restrict__ foc, const uint32_t* __restrict__ key, const uint32_t* __restrict__ sorted,
               uint64_t kbase, uint64_t kend, uint32_t chunk, uint32_t nbins, FixCell2* __restrict__ grids, int pg0, int npg,
               FixScale* __restrict__ fs) {
  static_assert(S >= 1 && S <= 8, "8 x 8 windows");
  extern __shared__ __align__(16) unsigned char smem[];
  double* flush_buf = reinterpret_cast<double*>(smem);
  F64Slots st;
  st.carve(smem + F64_FLUSH_BYTES);
  const int lane = threadIdx.x, gq = lane >> 2, tq = lane & 3;
  if (lane < 8) {
    st.ku[F64_BATCH * F64_ROW + lane] = 0.0;
    st.bre[F64_BATCH * F64_ROW + lane] = 0.0;
    st.bim[F64_BATCH * F64_ROW + lane] = 0.0;
    st.kw[F64_BATCH * F64_KW + lane] = 0.0;
  }
  if (lane == 0) st.key[F64_BATCH] = INACTIVE;
  const uint64_t k0 = kbase + (uint64_t)blockIdx.x * chunk;
  const uint64_t k1 = min(kend, k0 + chunk);
  const double sc = FixTraits<double>::scale(fs->q);
  const uint32_t nchan = (uint32_t)g.nchan;
  const uint32_t tmask = (1u << g.log2tile) - 1u;
  const bool with_wgt = in.wgt_kind != WGT_NONE;
  bool bad = false;

  constexpr int NP = (S + 1) / 2;  // plane pairs
  double acc[NP][2][4];
#pragma unroll
  for (int h = 0; h < NP; h++)
#pragma unroll
    for (int c = 0; c < 2; c++)
#pragma unroll
      for (int i = 0; i < 4; i++) acc[h][c][i] = 0.0;
  Window win;

  // This round's inputs are in pre (copied asynchronously); nidx is the next
  // round's index.
  Prefetched64* pre = reinterpret_cast<Prefetched64*>(smem + F64_FLUSH_BYTES + F64Slots::bytes()) + lane;
  const bool with_vis = mode == VALUE_DATA && in.vis_kind != VIS_UNIT;
  if (k0 + lane < k1) prefetch64(pre, uvw, foc, in, with_vis, with_wgt, key, sorted[k0 + lane], nchan);
  cp_async_commit();
  uint32_t nidx = (k0 + F64_BATCH + lane < k1) ? sorted[k0 + F64_BATCH + lane] : 0u;

  for (uint64_t kb = k0; kb < k1; kb += F64_BATCH) {
    const int nb = (int)min((uint64_t)F64_BATCH, k1 - kb);
    cp_async_wait_all();
    __syncwarp();
    if (lane < nb) {  // staging, one record per lane
      const Prefetched64& pr = *pre;
      double b[3];
      const double imflip = row_coord_of(pr.uvw[0], pr.uvw[1], pr.uvw[2], g.fu, g.fv, g.fw, g.r_l, g.r_m, b);
      const double f = pr.foc;
      const double u = b[0] * f, v = b[1] * f, w = b[2] * f;
      double uf, vf;
      int iu0, iv0;
      getpix(g, u, v, uf, vf, iu0, iv0);
      const int mp = minplane(g, w);
      const uint32_t su = (uint32_t)shifted(iu0, g.nu) & tmask, sv = (uint32_t)shifted(iv0, g.nv) & tmask;
      const int ur = (int)(su & 7u), dv = (int)(sv % (uint32_t)g.sube);
      double ku[S], kv[S];
      eval_taps2<double, S>(g.coeff, g.ne, -uf * 2.0 + ((double)S - 1.0), -vf * 2.0 + ((double)S - 1.0), ku, kv);
      cplx<double> val = unit_value<double>(g, b, imflip, f, with_wgt, prefetched_wgt64(pr, in));
      if (mode == VALUE_DATA) val = data_value<double>(prefetched_vis64(pr, in), val, imflip);
      bad |= !isfinite(val.re) || !isfinite(val.im) || !isfinite(uf) || !isfinite(vf) || !isfinite(w);
      double* cu = st.ku + lane * F64_ROW;
      double* cr = st.bre + lane * F64_ROW;
      double* ci = st.bim + lane * F64_ROW;
      double* cw = st.kw + lane * F64_KW;
      // The u taps at rows (su + i) mod 8, zero elsewhere.
#pragma unroll
      for (int j = 0; j < 8; j++) cu[(ur + j) & 7] = j < S ? ku[j < S ? j : 0] : 0.0;
      double kwt[S];
      if (g.do_wgridding) {  // the w taps from the first plane's argument (w_factor)
        const double z = g.xdw * ((g.wmin + (double)mp * g.dw) - w);
        eval_taps1<S>(g.coeff, z * 2.0 + ((double)S - 1.0), kwt);
      }
#pragma unroll
      for (int j = 0; j < 8; j++) {
        double br = 0.0, bi = 0.0;
#pragma unroll
        for (int d = 0; d < 9 - S; d++) {
          if (j - d >= 0 && j - d < S && dv == d) {
            const int t = (j - d >= 0 && j - d < S) ? j - d : 0;
            br = val.re * kv[t];
            bi = val.im * kv[t];
          }
        }
        cr[j] = br;
        ci[j] = bi;
        double kwj = 0.0;
        if (j < S) {
          if (g.do_wgridding) {
            if (mp + j >= pg0 && mp + j < pg0 + npg) kwj = kwt[j < S ? j : 0];
          } else if (j == 0 && pg0 == 0) {
            kwj = 1.0;
          }
        }
        cw[j] = kwj;
      }
      st.key[lane] = pr.key;
    }
    // The next round's inputs, in flight while this one is contracted.
    __syncwarp();
    if (kb + F64_BATCH + lane < k1) prefetch64(pre, uvw, foc, in, with_vis, with_wgt, key, nidx, nchan);
    cp_async_commit();
    if (kb + 2 * F64_BATCH + lane < k1) nidx = sorted[kb + 2 * F64_BATCH + lane];
    int q = 0;
    while (q < nb) {
      const uint32_t gk = st.key[q];
      if (gk != win.key) {
        Window next;
        const int leave = window_step(g, win, gk, nbins, next);
        if (win.key != INACTIVE) f64_flush<S>(g, grids, pg0, npg, win, leave, sc, acc, flush_buf);
        win = next;
      }
      const unsigned m = __ballot_sync(0xffffffffu, lane >= q && lane < nb && st.key[lane] == gk);
      const int len = __popc(m);
      for (int k8 = q; k8 < q + len; k8 += 8) {
        const int s0 = k8 + tq < q + len ? k8 + tq : F64_BATCH, s1 = k8 + 4 + tq < q + len ? k8 + 4 + tq : F64_BATCH;
        const double u0 = st.ku[s0 * F64_ROW + gq];  // A: row gq, k tq
        const double re0 = st.bre[s0 * F64_ROW + gq], im0 = st.bim[s0 * F64_ROW + gq];  // B: k tq, column gq
        const double2* w0 = reinterpret_cast<const double2*>(st.kw + s0 * F64_KW);
        if (k8 + 4 < q + len) {
          const double u1 = st.ku[s1 * F64_ROW + gq];
          const double re1 = st.bre[s1 * F64_ROW + gq], im1 = st.bim[s1 * F64_ROW + gq];
          const double2* w1 = reinterpret_cast<const double2*>(st.kw + s1 * F64_KW);
#pragma unroll
          for (int h = 0; h < NP; h++) {
            const double2 wa = w0[h], wb = w1[h];
            const double a0 = u0 * wa.x, a1 = u0 * wa.y, a2 = u1 * wb.x, a3 = u1 * wb.y;
            dmma16x8(acc[h][0], a0, a1, a2, a3, re0, re1);
            dmma16x8(acc[h][1], a0, a1, a2, a3, im0, im1);
          }
        } else {
#pragma unroll
          for (int h = 0; h < NP; h++) {
            const double2 wa = w0[h];
            const double a0 = u0 * wa.x, a1 = u0 * wa.y;
            dmma16x4(acc[h][0], a0, a1, re0);
            dmma16x4(acc[h][1], a0, a1, im0);
          }
        }
      }
      q += len;
    }
  }
  if (win.key != INACTIVE) f64_flush<S>(g, grids, pg0, npg, win, 8, sc, acc, flush_buf);
  if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(&fs->nonfinite, 1);
}

// ------------------------------------------------------------------ degridder

// Per slot (record): the v taps placed on the window's 8 columns, the u taps on
// its 8 rows, the w taps of the S planes, conj(phase) * wgt with the sign of
// the w flip, and the visibility's index and bin key. Slot F64_BATCH stays zero.
struct F64DegridSlots {
  double* kw;
  double4* out;  // re, im of the final factor, the flip's sign, unused
  double* ku;
  double* kv;
  uint32_t* idx;
  uint32_t* key;
  __host__ __device__ static constexpr size_t bytes() {
    return ((size_t)(F64_BATCH + 1) * ((2 * F64_ROW + F64_KW) * 8 + 32 + 8) + 15) / 16 * 16;
  }
  __device__ void carve(unsigned char* base) {
    out = reinterpret_cast<double4*>(base);
    kw = reinterpret_cast<double*>(out + (F64_BATCH + 1));
    ku = kw + (F64_BATCH + 1) * F64_KW;
    kv = ku + (F64_BATCH + 1) * F64_ROW;
    idx = reinterpret_cast<uint32_t*>(kv + (F64_BATCH + 1) * F64_ROW);
    key = idx + (F64_BATCH + 1);
  }
};

// Degridding of sorted records [kbase, kend) in double precision on the FP64
// tensor cores (degrid_task_body, wgridder.rs:2793-2901): as k_degrid_h, the
// warp holds the current bin's 8 x 8 window of each plane (here as the doubles
// themselves) with its rows at u mod 8, reads only the rows a bin adds, and
// per block of sixteen records contracts along v on the tensor cores (records
// along M, window columns along K, window rows along N), then over the planes
// and along u with FMAs. Blocks of at most eight records take the 8-row MMA.
// One thread per visibility over a tile's window in shared memory, which
// this replaces for supports up to 8, read every cell of every footprint from
// shared memory: 2.91 ms for 16.5 M visibilities of support 8, 2.36 now (the
// FP64 tensor pipe is busy 44 % of the time, 11 warps per SM by registers).
template <int S>
__global__ void __launch_bounds__(F64_BATCH, F64_BLOCKS)
    k_degrid_f64(const __grid_constant__ Geom<double> g, Inputs wts, const double* __restrict__ uvw,
                 const double* __restrict__ foc, const uint32_t* __restrict__ key,
                 const uint32_t* __restrict__ sorted, uint64_t kbase, uint64_t kend, uint32_t chunk, uint32_t nbins,
                 const cplx<double>* __restrict__ grids, int pg0, int npg, cplx<double>* __restrict__ vis, int first,
                 int last) {
  static_assert(S >= 1 && S <= 8, "8 x 8 windows");
  extern __shared__ __align__(16) unsigned char smem[];
  F64DegridSlots st;
  st.carve(smem);
  const int lane = threadIdx.x, gq = lane >> 2, tq = lane & 3;
  if (lane < 8) {
    st.ku[F64_BATCH * F64_ROW + lane] = 0.0;
    st.kv[F64_BATCH * F64_ROW + lane] = 0.0;
    st.kw[F64_BATCH * F64_KW + lane] = 0.0;
  }
  if (lane == 0) st.key[F64_BATCH] = INACTIVE;
  const uint64_t k0 = kbase + (uint64_t)blockIdx.x * chunk;
  const uint64_t k1 = min(kend, k0 + chunk);
  const uint32_t nchan = (uint32_t)g.nchan;
  const uint32_t tmask = (1u << g.log2tile) - 1u;
  const bool with_wgt = wts.wgt_kind != WGT_NONE;
  const size_t plane = (size_t)g.nu * g.nv;

  cplx<double> win_v[S][2];  // [plane]: window row gq (mod 8), columns tq and tq + 4
#pragma unroll
  for (int p = 0; p < S; p++) win_v[p][0] = win_v[p][1] = cplx<double>{0.0, 0.0};
  Window win;

  Prefetched64* pre = reinterpret_cast<Prefetched64*>(smem + F64DegridSlots::bytes()) + lane;
  if (k0 + lane < k1) prefetch64(pre, uvw, foc, wts, false, with_wgt, key, sorted[k0 + lane], nchan);
  cp_async_commit();
  uint32_t nidx = (k0 + F64_BATCH + lane < k1) ? sorted[k0 + F64_BATCH + lane] : 0u;

  for (uint64_t kb = k0; kb < k1; kb += F64_BATCH) {
    const int nb = (int)min((uint64_t)F64_BATCH, k1 - kb);
    cp_async_wait_all();
    __syncwarp();
    if (lane < nb) {  // staging, one record per lane
      const Prefetched64& pr = *pre;
      double b[3];
      const double imflip = row_coord_of(pr.uvw[0], pr.uvw[1], pr.uvw[2], g.fu, g.fv, g.fw, g.r_l, g.r_m, b);
      const double f = pr.foc;
      const double u = b[0] * f, v = b[1] * f, w = b[2] * f;
      double uf, vf;
      int iu0, iv0;
      getpix(g, u, v, uf, vf, iu0, iv0);
      const int mp = minplane(g, w);
      const uint32_t su = (uint32_t)shifted(iu0, g.nu) & tmask, sv = (uint32_t)shifted(iv0, g.nv) & tmask;
      const uint32_t ur = su & 7u, dv = sv % (uint32_t)g.sube;
      double ku[S], kv[S];
      eval_taps2<double, S>(g.coeff, g.ne, -uf * 2.0 + ((double)S - 1.0), -vf * 2.0 + ((double)S - 1.0), ku, kv);
      double* cu = st.ku + lane * F64_ROW;
      double* cv = st.kv + lane * F64_ROW;
      double* cw = st.kw + lane * F64_KW;
#pragma unroll
      for (int j = 0; j < 8; j++) {
        cu[(ur + j) & 7u] = j < S ? ku[j < S ? j : 0] : 0.0;
        cv[(dv + j) & 7u] = j < S ? kv[j < S ? j : 0] : 0.0;
      }
      double kwt[S];
      if (g.do_wgridding) {  // the w taps from the first plane's argument (w_factor)
        const double z = g.xdw * ((g.wmin + (double)mp * g.dw) - w);
        eval_taps1<S>(g.coeff, z * 2.0 + ((double)S - 1.0), kwt);
      }
      // Planes outside this pass's are zero in the window.
#pragma unroll
      for (int j = 0; j < 8; j++)
        cw[j] = g.do_wgridding ? (j < S ? kwt[j < S ? j : 0] : 0.0) : (j == 0 ? 1.0 : 0.0);
      double4 fin = make_double4(1.0, 0.0, imflip, 0.0);
      if (last) {  // wgridder.rs:3146-3159
        const double tw = prefetched_wgt64(pr, wts);
        fin.x = tw;
        if (g.shifting) {
          const cplx<double> ph = shift_phase<double>(g, b, imflip, f, -1.0);
          fin.x = ph.re * tw;
          fin.y = ph.im * tw;
        }
      }
      st.out[lane] = fin;
      st.idx[lane] = pr.idx;
      st.key[lane] = pr.key;
    }
    __syncwarp();
    if (kb + F64_BATCH + lane < k1) prefetch64(pre, uvw, foc, wts, false, with_wgt, key, nidx, nchan);
    cp_async_commit();
    if (kb + 2 * F64_BATCH + lane < k1) nidx = sorted[kb + 2 * F64_BATCH + lane];
    int q = 0;
    while (q < nb) {
      const uint32_t gk = st.key[q];
      if (gk != win.key) {  // read the rows that bin gk adds to the window
        Window next;
        const int enter = window_step(g, win, gk, nbins, next);
        win = next;
        const int o = (gq - win.rb) & 7;  // this lane's row of the window
        if (o >= 8 - enter) {
          int row = win.su0 + o;
          if (row >= g.nu) row -= g.nu;
          int c0 = win.sv0 + tq, c1 = c0 + 4;
          if (c0 >= g.nv) c0 -= g.nv;
          if (c1 >= g.nv) c1 -= g.nv;
#pragma unroll
          for (int p = 0; p < S; p++) {
            const int pp = win.mp + p;
            const bool ok = pp >= pg0 && pp < pg0 + npg && (g.do_wgridding || pp == 0);
            const double2* src =
                reinterpret_cast<const double2*>(grids + (size_t)(ok ? pp - pg0 : 0) * plane + (size_t)row * g.nv);
            const double2 x0 = ok ? src[c0] : make_double2(0.0, 0.0), x1 = ok ? src[c1] : make_double2(0.0, 0.0);
            win_v[p][0] = {x0.x, x0.y};
            win_v[p][1] = {x1.x, x1.y};
          }
        }
      }
      const unsigned mk = __ballot_sync(0xffffffffu, lane >= q && lane < nb && st.key[lane] == gk);
      const int len = __popc(mk);
      for (int k16 = q; k16 < q + len; k16 += 16) {
        const bool two = k16 + 8 < q + len;  // records gq + 8 too
        int sr[2];
        double av[2][2];  // [record gq, gq + 8][column tq, tq + 4]
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int k = k16 + gq + 8 * h;
          sr[h] = k < q + len ? k : F64_BATCH;
          av[h][0] = st.kv[sr[h] * F64_ROW + tq];
          av[h][1] = st.kv[sr[h] * F64_ROW + tq + 4];
        }
        double wr[2][2] = {{0.0, 0.0}, {0.0, 0.0}}, wi[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
#pragma unroll
        for (int p = 0; p < S; p++) {
          double dre[4] = {0.0, 0.0, 0.0, 0.0}, dim[4] = {0.0, 0.0, 0.0, 0.0};
          const cplx<double> x0 = win_v[p][0], x1 = win_v[p][1];
          if (two) {
            dmma16x8(dre, av[0][0], av[1][0], av[0][1], av[1][1], x0.re, x1.re);
            dmma16x8(dim, av[0][0], av[1][0], av[0][1], av[1][1], x0.im, x1.im);
          } else {
            dmma8x4(dre[0], dre[1], av[0][0], x0.re);
            dmma8x4(dre[0], dre[1], av[0][1], x1.re);
            dmma8x4(dim[0], dim[1], av[0][0], x0.im);
            dmma8x4(dim[0], dim[1], av[0][1], x1.im);
          }
#pragma unroll
          for (int h = 0; h < 2; h++) {
            if (h == 1 && !two) break;
            const double kw = st.kw[sr[h] * F64_KW + p];
#pragma unroll
            for (int c = 0; c < 2; c++) {
              wr[h][c] = fma(kw, dre[2 * h + c], wr[h][c]);
              wi[h][c] = fma(kw, dim[2 * h + c], wi[h][c]);
            }
          }
        }
        double tr[2], ti[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const double u0 = st.ku[sr[h] * F64_ROW + 2 * tq], u1 = st.ku[sr[h] * F64_ROW + 2 * tq + 1];
          tr[h] = fma(u0, wr[h][0], u1 * wr[h][1]);
          ti[h] = fma(u0, wi[h][0], u1 * wi[h][1]);
        }
        // Odd lanes of a quad take record gq + 8, even ones record gq.
        const bool odd = tq & 1;
        double re = odd ? tr[1] : tr[0], im = odd ? ti[1] : ti[0];
        re += __shfl_xor_sync(0xffffffffu, odd ? tr[0] : tr[1], 1);
        im += __shfl_xor_sync(0xffffffffu, odd ? ti[0] : ti[1], 1);
        re += __shfl_xor_sync(0xffffffffu, re, 2);
        im += __shfl_xor_sync(0xffffffffu, im, 2);
        const int slot = odd ? sr[1] : sr[0];
        if (tq < 2 && slot != F64_BATCH) {
          const double4 fin = st.out[slot];
          cplx<double>* dst = vis + st.idx[slot];
          cplx<double> acc{re, im * fin.z};
          if (!first) {
            const cplx<double> prev = *dst;
            acc = {acc.re + prev.re, acc.im + prev.im};
          }
          if (last) acc = {acc.re * fin.x - acc.im * fin.y, acc.re * fin.y + acc.im * fin.x};
          *dst = acc;
        }
      }
      q += len;
    }
  }
}

}  // namespace fast
