// 2D LF / WENO5-JS stage of the fp64 and mixed variants as an x-line sweep
// plus y runs (included by jb_kernels.cuh inside the variant's namespace):
//   k_sweep_x  one thread per (y line, x segment of seg cells, field pack;
//              seg chosen by the host for whole waves): register windows of
//              the split fluxes' differences walk the segment's faces and
//              write twice the x flux difference F_{i+1/2} - F_{i-1/2}
//   k_flux_y   one block per segment of 128 cells of a column: split fluxes
//              of all packs on the segment and its 3 + 3 halo cells in
//              shared memory, the 129 y faces as register-window runs of
//              four (or two) faces per thread, then the RK combination with
//              the x part and the temperature solve of the new state
// A pack V is one float64 field (fp64: 12 packs) or a pair of float32 fields
// (mixed: (rho, rho u), (rho v, rho E), (rho Y_1, rho Y_2), ... as sm_100's
// paired float32 instructions FFMA2 / FADD2 / FMUL2, 6 packs).  The RK
// combination and the temperature solve are float64 in both.  The stage
// state's u, v, p come from the kernel that finished that state
// (prims[3][ncell], in the pack's scalar type).  The x differences wait in the
// stage's own output: pack j of a cell in the 8 bytes that field W j of that
// cell takes, which only the thread that combines the cell reads, before it
// writes them (k_flux_y reads them through out, which is neither Uk nor Un).
typedef float2 f2;
template <class V> struct VT;
template <> struct VT<double> {
  typedef double S;
  static constexpr int W = 1, NP = 12;
};
template <> struct VT<float> {  // 1D lines only
  typedef float S;
  static constexpr int W = 1;
};
template <> struct VT<f2> {
  typedef float S;
  static constexpr int W = 2, NP = 6;
};

template <class V> __device__ __forceinline__ V vset(typename VT<V>::S a);
template <> __device__ __forceinline__ double vset<double>(double a) { return a; }
template <> __device__ __forceinline__ f2 vset<f2>(float a) { return make_float2(a, a); }
template <class V> __device__ __forceinline__ V vmake(typename VT<V>::S a, typename VT<V>::S b);
template <> __device__ __forceinline__ double vmake<double>(double a, double) { return a; }
template <> __device__ __forceinline__ f2 vmake<f2>(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ double vget(double a, int) { return a; }
__device__ __forceinline__ float vget(f2 a, int i) { return i ? a.y : a.x; }
__device__ __forceinline__ double vadd(double a, double b) { return a + b; }
__device__ __forceinline__ double vsub(double a, double b) { return a - b; }
__device__ __forceinline__ float vsub(float a, float b) { return a - b; }
__device__ __forceinline__ double vmul(double a, double b) { return a * b; }
__device__ __forceinline__ double vfma(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float vfma(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ f2 vadd(f2 a, f2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ f2 vsub(f2 a, f2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ f2 vmul(f2 a, f2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ f2 vfma(f2 a, f2 b, f2 c) { return __ffma2_rn(a, b, c); }

// The float32 weno_side for a pair of fields.  The bound on the ratios keeps
// den and num * den in range (|f| < 1e17), so that both sides of a face share
// one reciprocal.  Paired instructions where both operands are pairs; sums with
// a sign and products with a constant are taken per component, whose scalar
// forms carry signs and immediates (a paired one needs its constant in a
// register pair: with those the sweep issued 200 instructions per face).
__device__ __forceinline__ void weno_side(f2 dmm, f2 dm, f2 dp, f2 dpp, f2 Da, f2 Db, f2 Dc, f2& num, f2& den) {
  const f2 t1 = make_float2(fmaf(3.f, dm.x, -dmm.x), fmaf(3.f, dm.y, -dmm.y));
  const f2 t2 = vadd(dm, dp);
  const f2 t3 = make_float2(fmaf(3.f, dp.x, -dpp.x), fmaf(3.f, dp.y, -dpp.y));
  const f2 e1 = vfma(t1, t1, Da), e2 = vfma(t2, t2, Db), e3 = vfma(t3, t3, Dc);
  f2 r1 = vmul(e2, make_float2(rcp_fast(e1.x), rcp_fast(e1.y)));
  f2 r3 = vmul(e2, make_float2(rcp_fast(e3.x), rcp_fast(e3.y)));
  r1 = make_float2(fminf(r1.x, 6.5e4f), fminf(r1.y, 6.5e4f));
  r3 = make_float2(fminf(r3.x, 6.5e4f), fminf(r3.y, 6.5e4f));
  const f2 a1 = vmul(r1, r1);
  f2 a3 = vmul(r3, r3);
  a3 = make_float2(3.f * a3.x, 3.f * a3.y);
  const f2 q1 = make_float2(fmaf(2.f, t1.x, -dm.x), fmaf(2.f, t1.y, -dm.y));
  f2 q2 = vadd(t2, dp);
  q2 = make_float2(6.f * q2.x, 6.f * q2.y);
  num = vfma(a3, vadd(t3, dp), vfma(a1, q1, q2));
  den = vadd(make_float2(a1.x + 6.f, a1.y + 6.f), a3);
}

// Twice the face flux L(H+) + R(H-) from the two sides' base values and
// corrections (the right-biased value is taken along the reversed axis, which
// flips the sign of its differences); the factor 1/2 goes into the
// divergence.
__device__ __forceinline__ double face_value(double bl, double nl, double dl, double br, double nr, double dr) {
  // each side's value rounded by itself, as the reference rounds L and R
  return fma(1.0 / 6.0, nl * rcp_nr(dl), bl) + fma(-1.0 / 6.0, nr * rcp_nr(dr), br);
}
__device__ __forceinline__ float face_value(float bl, float nl, float dl, float br, float nr, float dr) {
  return fmaf(1.f / 6.f, fmaf(nl, dr, -(nr * dl)) * rcp_fast(dl * dr), bl + br);
}
__device__ __forceinline__ f2 face_value(f2 bl, f2 nl, f2 dl, f2 br, f2 nr, f2 dr) {
  const f2 dd = vmul(dl, dr), nd = vmul(nr, dl), b = vadd(bl, br);
  const f2 c = vmul(make_float2(fmaf(nl.x, dr.x, -nd.x), fmaf(nl.y, dr.y, -nd.y)),
                    make_float2(rcp_fast(dd.x), rcp_fast(dd.y)));
  return make_float2(fmaf(1.f / 6.f, c.x, b.x), fmaf(1.f / 6.f, c.y, b.y));
}

// Register window of one split flux along a line: before cell n enters, the
// values of cells n-2, n-1, the differences d_{n-7/2} .. d_{n-3/2} and the
// curvature terms of cells n-3, n-2.  Each enters once per cell and serves
// three faces.
template <class V>
struct Win {
  V f0, f1, d0, d1, d2, D0, D1;
};
__device__ __forceinline__ double weno_curv(double da, double db) { return weno_curv(da, db, 16e-6); }
__device__ __forceinline__ float weno_curv(float da, float db) { return weno_curv(da, db, 16e-6f); }
__device__ __forceinline__ f2 weno_curv(f2 da, f2 db) {
  return make_float2(weno_curv(da.x, db.x, 16e-6f), weno_curv(da.y, db.y, 16e-6f));
}
// cells n-4 .. n-1
template <class V>
__device__ __forceinline__ void win_init(Win<V>& w, V g0, V g1, V g2, V g3) {
  w.d0 = vsub(g1, g0);
  w.d1 = vsub(g2, g1);
  w.d2 = vsub(g3, g2);
  w.f0 = g2;
  w.f1 = g3;
  w.D0 = weno_curv(w.d0, w.d1);
  w.D1 = weno_curv(w.d1, w.d2);
}
// Cell n enters: base value f_{n-2} and correction of the left-biased value
// behind cell n-2 (LEFT), or of the right-biased value before it.
template <bool LEFT, class V>
__device__ __forceinline__ void win_push(Win<V>& w, V fn, V& base, V& num, V& den) {
  const V d3 = vsub(fn, w.f1), D2 = weno_curv(w.d2, d3);
  base = w.f0;
  if (LEFT) weno_side(w.d0, w.d1, w.d2, d3, w.D0, w.D1, D2, num, den);
  else weno_side(d3, w.d2, w.d1, w.d0, D2, w.D1, w.D0, num, den);
  w.f0 = w.f1;
  w.f1 = fn;
  w.d0 = w.d1;
  w.d1 = w.d2;
  w.d2 = d3;
  w.D0 = w.D1;
  w.D1 = D2;
}

// Doubled split fluxes of pack j at one cell for direction dir:
// F = vel q (+ p in the normal momentum, + vel p in rho E), H' = F +- alpha q.
__device__ __forceinline__ void split_pack(int j, int dir, double q, double vel, double p, double al, double& hp,
                                           double& hm) {
  double F = vel * q;
  if (j == 1 + dir) F = fma(vel, q, p);
  if (j == 3) F = fma(vel, p, F);
  hp = fma(al, q, F);
  hm = fma(-al, q, F);
}
__device__ __forceinline__ void split_pack(int j, int dir, f2 q, float vel, float p, float al, f2& hp, f2& hm) {
  // pack 0 = (rho, rho u), pack 1 = (rho v, rho E)
  f2 c = make_float2(0.f, 0.f);
  if (j == 0 && dir == 0) c.y = p;
  if (j == 1) {
    if (dir == 1) c.x = p;
    c.y = vel * p;
  }
  const f2 F = make_float2(fmaf(vel, q.x, c.x), fmaf(vel, q.y, c.y));
  hp = make_float2(fmaf(al, q.x, F.x), fmaf(al, q.y, F.y));
  hm = make_float2(fmaf(-al, q.x, F.x), fmaf(-al, q.y, F.y));
}

// pack j of the float64 state at cell index c, with the sign flips of a ghost
template <class V>
__device__ __forceinline__ V load_pack(const double* __restrict__ U, long long nc, long long c, int j, int flip);
template <>
__device__ __forceinline__ double load_pack<double>(const double* __restrict__ U, long long nc, long long c, int j,
                                                    int flip) {
  const double v = U[j * nc + c];
  return ((flip >> j) & 1) ? -v : v;
}
template <>
__device__ __forceinline__ f2 load_pack<f2>(const double* __restrict__ U, long long nc, long long c, int j, int flip) {
  const float v0 = (float)U[2 * j * nc + c], v1 = (float)U[(2 * j + 1) * nc + c];
  return make_float2(((flip >> (2 * j)) & 1) ? -v0 : v0, ((flip >> (2 * j + 1)) & 1) ? -v1 : v1);
}

// Pack j, the normal velocity of direction DIR and the pressure of padded
// cell (x, y): interior and copied ghosts from the state and the primitives,
// outlet / injector ghosts and ghost layers from their buffers.
template <int DIR, class V>
__device__ __forceinline__ void pack_load(const MP& m, const Grid& g, const double* __restrict__ Uk,
                                          const typename VT<V>::S* __restrict__ prims,
                                          const double* __restrict__ strips, int x, int y, int j, V& q,
                                          typename VT<V>::S& vel, typename VT<V>::S& p) {
  typedef typename VT<V>::S R;
  const long long nc = g.ncell;
  const Src s = map_cell<2>(g, x, y);
  if (s.kind == 0) {
    const long long src = (long long)s.xs * g.ny + s.ys;
    q = load_pack<V>(Uk, nc, src, j, s.flip);
    vel = prims[(DIR == 0 ? 0 : nc) + src];
    if (s.flip & (DIR == 0 ? 2 : 4)) vel = -vel;
    p = prims[2 * nc + src];
  } else if (s.kind == 1) {
    R qa[12];
#pragma unroll
    for (int i = 0; i < 12; ++i) qa[i] = (R)ghost(g, strips, s, i);
    R rho, u, v;
    flux_prims<2>(m, qa, (R)ghost(g, strips, s, 13), rho, u, v, p);
    vel = DIR == 0 ? u : v;
    constexpr int W = VT<V>::W;
    q = vmake<V>((R)ghost(g, strips, s, W * j), (R)ghost(g, strips, s, W * j + W - 1));
  } else {
    q = vset<V>((R)1);
    vel = (R)1;
    p = (R)1;
  }
}

constexpr int SX_NT = 128;
// blocks per SM: 72 registers for float32 pairs, 96 for float64 (80 at 6: the
// channel 715 against 710 us for two steps)
#ifndef JB_SX_MINB
#define JB_SX_MINB 7
#endif
#ifndef JB_SXD_MINB
#define JB_SXD_MINB 5
#endif
template <class V>
__global__ void __launch_bounds__(SX_NT, VT<V>::W == 2 ? JB_SX_MINB : JB_SXD_MINB)
    k_sweep_x(MP m, Grid g, const double* __restrict__ Uk, const typename VT<V>::S* __restrict__ prims,
              const double* __restrict__ strips, const Slots* slots, int aidx, V* __restrict__ dfx, int nlb,
              int seg_len) {
  typedef typename VT<V>::S R;
  constexpr int W = VT<V>::W, NP = VT<V>::NP;
  const int j = blockIdx.x % NP;
  const int rest = blockIdx.x / NP;
  const int y = (rest % nlb) * SX_NT + threadIdx.x, seg = rest / nlb;
  if (y >= g.ny) return;
  const long long nc = g.ncell;
  const double* u0 = Uk + (long long)W * j * nc;
  const R al = (R)bitsd(slots->ax[aidx]);
  const bool need_p = W == 2 ? j < 2 : (j == 1 || j == 3);  // the packs whose flux has a pressure term
  const int a0 = seg * seg_len, a1 = min(a0 + seg_len, g.nx);  // cells [a0, a1), faces a0 .. a1
  Win<V> wp, wm;
  V hp_next;  // H+ of the cell behind the newest H-
  {
    V hp[5], hm[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      V q;
      R vel, p;
      pack_load<0, V>(m, g, Uk, prims, strips, a0 - 3 + k, y, j, q, vel, p);
      split_pack(j, 0, q, vel, p, al, hp[k], hm[k]);
    }
    win_init(wp, hp[0], hp[1], hp[2], hp[3]);
    win_init(wm, hm[1], hm[2], hm[3], hm[4]);
    hp_next = hp[4];
  }
  // The hi-side ghost cells nx .. nx+2 of the line (the last segment's
  // window reaches them) go to this thread's column of shared memory first,
  // so that the face loop's fetch is a plain load: the ghost mapping stays
  // out of the unrolled loop body.
  __shared__ R gh[3][W + 2][SX_NT];
  if (a1 + 2 >= g.nx) {
#pragma unroll 1
    for (int k = 0; k < 3; ++k) {
      V q;
      R vel, p;
      pack_load<0, V>(m, g, Uk, prims, strips, g.nx + k, y, j, q, vel, p);
#pragma unroll
      for (int i = 0; i < W; ++i) gh[k][i][threadIdx.x] = vget(q, i);
      gh[k][W][threadIdx.x] = vel;
      gh[k][W + 1][threadIdx.x] = p;
    }
  }
  // the cell about to enter the window, fetched one face ahead and left
  // untouched until then so that its loads overlap the WENO arithmetic
  double n0 = 0.0, n1 = 0.0;
  R nv = (R)0, np = (R)0;
  auto fetch = [&](int a) {
    if (a < g.nx) {
      const long long src = (long long)a * g.ny + y;
      n0 = u0[src];
      if (W == 2) n1 = u0[nc + src];
      nv = prims[src];
      if (need_p) np = prims[2 * nc + src];
    } else {
      const int k = a - g.nx;
      n0 = gh[k][0][threadIdx.x];
      if (W == 2) n1 = gh[k][W - 1][threadIdx.x];
      nv = gh[k][W][threadIdx.x];
      np = gh[k][W + 1][threadIdx.x];
    }
  };
  fetch(a0 + 2);
  V* out = dfx + (long long)W * j * nc + y;
  V Fprev = vset<V>((R)0);
#pragma unroll 4  // the windows shift by renaming inside the unrolled bodies
  for (int fa = a0; fa <= a1; ++fa) {
    V hp, hm, bl, nl, dl, br, nr, dr;
    split_pack(j, 0, vmake<V>((R)n0, (R)n1), nv, np, al, hp, hm);  // cell fa+2
    if (fa < a1) fetch(fa + 3);
    // face fa (cells fa-1 | fa): H+ of cells fa-3 .. fa+1, H- of fa-2 .. fa+2
    win_push<true>(wp, hp_next, bl, nl, dl);
    win_push<false>(wm, hm, br, nr, dr);
    hp_next = hp;
    const V F = face_value(bl, nl, dl, br, nr, dr);
    if (fa > a0) out[(long long)(fa - 1) * g.ny] = vsub(F, Fprev);
    Fprev = F;
  }
}

// Slot i of a row of shared memory sits at i + i / 4, so that the runs'
// stride of four slots (two for the last packs of the float32 pairs) spreads
// over the banks.  y runs: blocks of 128 threads on 128 cells of a column.
constexpr int YR_S = 128;
__host__ __device__ constexpr int yr_at(int i) { return i + (i >> 2); }
constexpr int YR_C = yr_at(YR_S + 6), YR_F = yr_at(YR_S) + 1;
template <class V>
__host__ __device__ constexpr size_t yr_smem() {
  return sizeof(V) * VT<V>::NP * (2 * (size_t)YR_C + YR_F);
}

// N faces k0 .. k0 + N - 1 of one pack's row
template <int N, class V>
__device__ __forceinline__ void yr_run(const V* hp, const V* hm, V* f, int k0) {
  Win<V> wp, wm;
  win_init(wp, hp[yr_at(k0)], hp[yr_at(k0 + 1)], hp[yr_at(k0 + 2)], hp[yr_at(k0 + 3)]);
  win_init(wm, hm[yr_at(k0 + 1)], hm[yr_at(k0 + 2)], hm[yr_at(k0 + 3)], hm[yr_at(k0 + 4)]);
#pragma unroll
  for (int k = 0; k < N; ++k) {
    V bl, nl, dl, br, nr, dr;
    win_push<true>(wp, hp[yr_at(k0 + k + 4)], bl, nl, dl);
    win_push<false>(wm, hm[yr_at(k0 + k + 5)], br, nr, dr);
    f[yr_at(k0 + k)] = face_value(bl, nl, dl, br, nr, dr);
  }
}

// float32 pairs at 7 blocks per SM (72 registers, no spills): annulus 1600 x
// 1000 1236 us a step, 1292 at 8 (64 registers), 1258 at 6; channel 1024 x 256
// 455, 461, 461 us for two.  float64 at 4 (128 registers): 710 us, 717 at 5.
#ifndef JB_YR_MINB
#define JB_YR_MINB 7
#endif
#ifndef JB_YRD_MINB
#define JB_YRD_MINB 4
#endif
// STAGE 0: out = dt_arg * total flux (flux_func); 1..3 the RK stages, dt from
// the slots.
template <int STAGE, class V, bool VISC>
__global__ void __launch_bounds__(YR_S, VT<V>::W == 2 ? JB_YR_MINB : JB_YRD_MINB)
    k_flux_y(MP m, Grid g, const double* __restrict__ Uk, const double* __restrict__ auxk,
             const double* __restrict__ Un, const typename VT<V>::S* __restrict__ prims,
             const double* __restrict__ strips, double* __restrict__ out, Slots* slots, int aidx, jb_fin fin,
             double dt_arg, int nsy) {
  typedef typename VT<V>::S R;
  constexpr int W = VT<V>::W, NP = VT<V>::NP;
  extern __shared__ __align__(128) unsigned char smraw[];
  V* sHp = reinterpret_cast<V*>(smraw);  // [NP][YR_C]: cell y0 - 3 + i in slot i
  V* sHm = sHp + NP * YR_C;
  V* sF = sHm + NP * YR_C;  // [NP][YR_F]: face y0 + k (cells y0+k-1 | y0+k)
  const int t = threadIdx.x;
  const long long nc = g.ncell;
  const int x = blockIdx.x / nsy, y0 = (blockIdx.x % nsy) * YR_S;
  const int nin = min(YR_S, g.ny - y0);  // cells of the segment, faces 0 .. nin
  const R al = (R)bitsd(slots->ay[aidx]);
  // ---- split fluxes on the window: the segment's own cells one per thread,
  // the 3 + 3 halo cells as 6 NP (cell, pack) items
  if (t < nin) {
    const long long cell = (long long)x * g.ny + y0 + t;
    const R vel = prims[nc + cell], p = prims[2 * nc + cell];
    V q[NP];
#pragma unroll
    for (int i = 0; i < NP; ++i) q[i] = load_pack<V>(Uk, nc, cell, i, 0);
    const int jj = yr_at(t + 3);
#pragma unroll
    for (int i = 0; i < NP; ++i) split_pack(i, 1, q[i], vel, p, al, sHp[i * YR_C + jj], sHm[i * YR_C + jj]);
  }
#pragma unroll 1
  for (int i = t; i < 6 * NP; i += YR_S) {
    const int h = i / NP, pk = i % NP;
    const int jj = h < 3 ? h : nin + h;
    V q;
    R vel, p;
    pack_load<1, V>(m, g, Uk, prims, strips, x, y0 - 3 + jj, pk, q, vel, p);
    split_pack(pk, 1, q, vel, p, al, sHp[pk * YR_C + yr_at(jj)], sHm[pk * YR_C + yr_at(jj)]);
  }
  __syncthreads();
  // ---- faces 0 .. 127 of every pack as runs: warp w takes packs w, w + 4,
  // ... as 32 runs of four faces; the last two of six packs as 64 runs of two
  {
    const int w = t >> 5, l = t & 31;
    if (4 * l <= nin) {
#pragma unroll 1
      for (int pk = w; pk < (NP & ~3); pk += 4) yr_run<4>(sHp + pk * YR_C, sHm + pk * YR_C, sF + pk * YR_F, 4 * l);
    }
    if (NP & 3) {
      const int pk = (NP & ~3) + (t >> 6), k0 = 2 * (t & 63);
      if (k0 <= nin) yr_run<2>(sHp + pk * YR_C, sHm + pk * YR_C, sF + pk * YR_F, k0);
    }
    // face 128 of a full segment
    if (nin == YR_S && t < NP) yr_run<1>(sHp + t * YR_C, sHm + t * YR_C, sF + t * YR_F, YR_S);
  }
  __syncthreads();
  // ---- RK combination (float64) and update_aux of the new state
  unsigned bits = 0;
  double amx = 0.0, amy = 0.0, dtm = __longlong_as_double(0x7ff0000000000000LL);
  if (t < nin) {
    const long long cell = (long long)x * g.ny + y0 + t;
    const double dt = STAGE == 0 ? dt_arg : slots->dt;
    const double hx = 0.5 * g.idx, hy = 0.5 * g.idy;  // the face values are doubled
    double q[12];
#pragma unroll
    for (int i = 0; i < NP; ++i) {
      const V dF = reinterpret_cast<const V*>(out)[(long long)W * i * nc + cell];  // own planes, stored below
      const V dG = vsub(sF[i * YR_F + yr_at(t + 1)], sF[i * YR_F + yr_at(t)]);
#pragma unroll
      for (int h = 0; h < W; ++h) {
        const int f = W * i + h;
        const double L =
            visc_add<VISC>(g, f, cell, -fma((double)vget(dF, h), hx, __dmul_rn((double)vget(dG, h), hy)));
        // Uk is read again (L1): no registers held across the WENO
        const double r = STAGE == 0 ? dt * L
                                    : rk_stage<STAGE>(STAGE == 1 ? 0.0 : Un[f * nc + cell], Uk[f * nc + cell], dt, L);
        out[f * nc + cell] = r;
        q[f] = r;
      }
    }
    if (STAGE > 0)
      bits = finish_state<2, W == 2>(m, g, fin, q, auxk[nc + cell], cell, amx, amy, dtm, slots);
  }
  if (STAGE > 0) finish_reduce(fin, amx, amy, dtm, bits, slots);
}

// ---------------------------------------------------------------------------
// 1D LF / WENO5-JS stage
// ---------------------------------------------------------------------------
// One tile [x0, x0 + S) of a 1D stage by a block of NT threads (see k_flux_y;
// V: float64 or, in the mixed variant, float32): one thread per padded cell
// loads it, forms its primitives and writes the split fluxes of the 11 fields
// to shared memory; the S + 1 faces of the 11 fields are runs of R faces
// spread over all threads; one thread per cell combines the RK stage and
// finishes the new state's temperature as fin says.  Two block barriers a
// tile (a loop over the fields with three barriers each, one face and one
// cell per thread, took 15 us a launch at any small size).  Every thread of
// the block must call it.  Pointers are plain (not restrict) because the
// persistent ensemble kernel calls it on buffers written by other blocks of
// the same launch.  Returns the thread's mask / status bits as finish_state.
constexpr int L1_NF = 11;
// runs of R faces covering the S + 1 faces, and the row lengths they reach
template <int S>
struct LineShape {
  static constexpr int R = S >= 48 ? 4 : 1, NRUN = (S + R) / R;
  static constexpr int C = yr_at(NRUN * R + 4) + 1, F = yr_at(NRUN * R - 1) + 1;
};
template <class V, int S>
__host__ __device__ constexpr size_t line_smem() {
  return sizeof(V) * L1_NF * (2 * (size_t)LineShape<S>::C + LineShape<S>::F);
}
template <int STAGE, class V, int NT, int S, bool VISC = false>
__device__ __forceinline__ unsigned line_tile(const MP& m, const Grid& g, const double* Uk, const double* auxk,
                                              const double* Un, double* out, const jb_fin& fin,
                                              const double* strips, double alpha, double dt, int x0,
                                              unsigned char* smraw, double& amx, double& dtm, Slots* slots) {
  constexpr int R = LineShape<S>::R, NRUN = LineShape<S>::NRUN, C = LineShape<S>::C, F = LineShape<S>::F;
  V* sHp = reinterpret_cast<V*>(smraw);  // [11][C]: cell x0 - 3 + i in slot i
  V* sHm = sHp + L1_NF * C;
  V* sF = sHm + L1_NF * C;  // [11][F]: twice the flux at face x0 + k
  const int tid = threadIdx.x;
  const long long nc = g.ncell;
  const V al = (V)alpha;
  const int nin = min(S, g.nx - x0);
  for (int i = tid; i < nin + 6; i += NT) {
    const Src s = map_cell<1>(g, x0 + i - 3, 0);
    V q[L1_NF], T;
    if (s.kind == 0) {
#pragma unroll
      for (int f = 0; f < L1_NF; ++f) {
        const double v = Uk[f * nc + s.xs];
        q[f] = (V)(((s.flip >> f) & 1) ? -v : v);
      }
      T = (V)auxk[nc + s.xs];
    } else {
#pragma unroll
      for (int f = 0; f < L1_NF; ++f) q[f] = (V)ghost(g, strips, s, f);
      T = (V)ghost(g, strips, s, L1_NF + 1);
    }
    V rho, u, v, p;
    flux_prims<1>(m, q, T, rho, u, v, p);
    const int at = yr_at(i);
#pragma unroll
    for (int f = 0; f < L1_NF; ++f) {
      V Fl = u * q[f];
      if (f == 1) Fl = vfma(u, q[f], p);
      if (f == 2) Fl = vfma(u, p, Fl);
      sHp[f * C + at] = vfma(al, q[f], Fl);
      sHm[f * C + at] = vfma(-al, q[f], Fl);
    }
  }
  __syncthreads();
  for (int i = tid; i < L1_NF * NRUN; i += NT) {
    const int f = i / NRUN, k0 = R * (i % NRUN);
    if (k0 <= nin) yr_run<R>(sHp + f * C, sHm + f * C, sF + f * F, k0);
  }
  __syncthreads();
  unsigned bits = 0;
  if (tid < nin) {
    const long long cell = x0 + tid;
    const double hx = 0.5 * g.idx;
    double q[L1_NF];
#pragma unroll
    for (int f = 0; f < L1_NF; ++f) {
      const double dF = (double)(sF[f * F + yr_at(tid + 1)] - sF[f * F + yr_at(tid)]);
      const double L = visc_add<VISC>(g, f, cell, __dmul_rn(-dF, hx));
      q[f] = STAGE == 0 ? dt * L
                        : rk_stage<STAGE>(STAGE == 1 ? 0.0 : Un[f * nc + cell], Uk[f * nc + cell], dt, L);
    }
#pragma unroll
    for (int f = 0; f < L1_NF; ++f) out[f * nc + cell] = q[f];
    if (STAGE > 0) {
      double amy = 0.0;
      bits = finish_state<1, sizeof(V) == 4>(m, g, fin, q, auxk[nc + cell], cell, amx, amy, dtm, slots);
    }
  }
  __syncthreads();  // the tile's shared memory is reused by the next tile
  return bits;
}

template <int STAGE, class V, int NT, int S, bool VISC>
__global__ void __launch_bounds__(NT) k_line(MP m, Grid g, const double* __restrict__ Uk,
                                             const double* __restrict__ auxk, const double* __restrict__ Un,
                                             double* __restrict__ out, const double* __restrict__ strips,
                                             Slots* slots, int aidx, jb_fin fin, double dt_arg) {
  extern __shared__ __align__(128) unsigned char smraw[];
  const double dt = STAGE == 0 ? dt_arg : slots->dt;
  double amx = 0.0, dtm = __longlong_as_double(0x7ff0000000000000LL);
  const unsigned bits =
      line_tile<STAGE, V, NT, S, VISC>(m, g, Uk, auxk, Un, out, fin, strips, bitsd(slots->ax[aidx]), dt,
                                       blockIdx.x * S, smraw, amx, dtm, slots);
  if (STAGE > 0) finish_reduce(fin, amx, 0.0, dtm, bits, slots);
}
