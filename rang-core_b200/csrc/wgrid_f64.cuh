// The double-precision gridder on the FP64 tensor cores.
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
// (mma.sync m8n8k4: rows the window's u cells, columns its v cells, k four
// records: A = w tap x placed u taps, B = value x placed v taps), so the run's
// sums are formed in one fixed order, in FP64 as the reference forms them.
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
constexpr int F64_FLUSH_BYTES = 2 * 8 * 8 * 32;  // two planes' cells, [plane][row][column]

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

__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

// Adds the first `leave` rows of a window's sums to the 128-bit grid and clears
// them: acc[p][c][i] is plane mp + p, component c, column 2 tq + i of the window
// row that is gq mod 8. As in i8_flush the adds go through shared memory, a
// warp adding one row of one plane (256 contiguous bytes): straight from the
// fragments each 8-byte add was a 32-byte sector of its own in L2, which
// bound the kernel (4 x 512 adds per bin of support 8).
template <int S>
__device__ __forceinline__ void f64_flush(const Geom<double>& g, FixCell2* __restrict__ grids, int pg0, int npg,
                                          const Window& w, int leave, double sc, double (&acc)[S][2][2],
                                          unsigned long long* buf) {
  const int lane = threadIdx.x & 31, gq = lane >> 2, tq = lane & 3;
  const int o = (gq - w.rb) & 7;  // this lane's row of the window
  int col = w.sv0 + (lane >> 2);
  if (col >= g.nv) col -= g.nv;
  const size_t plane = (size_t)g.nu * g.nv;
#pragma unroll
  for (int p2 = 0; p2 < S; p2 += 2) {
    if (o < leave) {
#pragma unroll
      for (int e = 0; e < 2; e++) {
        if (p2 + e >= S) break;
#pragma unroll
        for (int i = 0; i < 2; i++) {
          const FixWide re = FixTraits<double>::term(acc[p2 + e][0][i], sc);
          const FixWide im = FixTraits<double>::term(acc[p2 + e][1][i], sc);
          longlong2* d = reinterpret_cast<longlong2*>(buf + (e * 8 + o) * 32 + (2 * tq + i) * 4);
          d[0] = make_longlong2(re.lo, re.hi);
          d[1] = make_longlong2(im.lo, im.hi);
          acc[p2 + e][0][i] = acc[p2 + e][1][i] = 0.0;
        }
      }
    }
    __syncwarp();
#pragma unroll
    for (int e = 0; e < 2; e++) {
      const int p = w.mp + p2 + e;
      if (p2 + e >= S || p < pg0 || p >= pg0 + npg) continue;
      unsigned long long* base =
          reinterpret_cast<unsigned long long*>(grids + (size_t)(p - pg0) * plane + col) + (lane & 3);
      for (int i = 0; i < leave; i++) {
        const unsigned long long v = buf[(e * 8 + i) * 32 + lane];
        int row = w.su0 + i;
        if (row >= g.nu) row -= g.nu;
        if (v) atomicAdd(base + (size_t)row * g.nv * 4, v);
      }
    }
    __syncwarp();
  }
}

// Gridding of sorted records [kbase, kend) in double precision (the
// reference's grid_task_body, wgridder.rs:2102-2156, on windows): each warp
// takes `chunk` consecutive sorted visibilities, stages F64_BATCH at a time
// (coordinates, taps and value from uvw and the data, as k_grid does) and
// contracts each run of one bin four records at a time.
template <int S>
__global__ void __launch_bounds__(F64_BATCH, F64_BLOCKS)
    k_grid_f64(const __grid_constant__ Geom<double> g, Inputs in, int mode, const double* __restrict__ uvw,
               const double* __restrict__ foc, const uint32_t* __restrict__ key, const uint32_t* __restrict__ sorted,
               uint64_t kbase, uint64_t kend, uint32_t chunk, uint32_t nbins, FixCell2* __restrict__ grids, int pg0, int npg,
               FixScale* __restrict__ fs) {
  static_assert(S >= 1 && S <= 8, "8 x 8 windows");
  extern __shared__ __align__(16) unsigned char smem[];
  unsigned long long* flush_buf = reinterpret_cast<unsigned long long*>(smem);
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

  double acc[S][2][2];
#pragma unroll
  for (int p = 0; p < S; p++)
#pragma unroll
    for (int c = 0; c < 2; c++) acc[p][c][0] = acc[p][c][1] = 0.0;
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
      for (int k4 = q; k4 < q + len; k4 += 4) {
        const int kk = k4 + tq;
        const int slot = kk < q + len ? kk : F64_BATCH;
        const double kur = st.ku[slot * F64_ROW + gq];   // A: row gq, k tq
        const double bre = st.bre[slot * F64_ROW + gq];  // B: k tq, column gq
        const double bim = st.bim[slot * F64_ROW + gq];
        const double2* kw2 = reinterpret_cast<const double2*>(st.kw + slot * F64_KW);
#pragma unroll
        for (int p = 0; p < S; p += 2) {
          const double2 kw = kw2[p / 2];
          const double a0 = kur * kw.x;
          dmma(acc[p][0], a0, bre);
          dmma(acc[p][1], a0, bim);
          if (p + 1 < S) {
            const double a1 = kur * kw.y;
            dmma(acc[p + 1 < S ? p + 1 : 0][0], a1, bre);
            dmma(acc[p + 1 < S ? p + 1 : 0][1], a1, bim);
          }
        }
      }
      q += len;
    }
  }
  if (win.key != INACTIVE) f64_flush<S>(g, grids, pg0, npg, win, 8, sc, acc, flush_buf);
  if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(&fs->nonfinite, 1);
}

}  // namespace fast
