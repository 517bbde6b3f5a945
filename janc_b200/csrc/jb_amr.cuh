// Block-structured AMR stepping on blocks with their ghost layers
// (src/janc_v2/simulation/time_step/TVD_RK3.py:15-36 advance_one_step_amr,
// with the block functions of simulation/set_simulator.py:37-42 and
// :97-113): the block layer (the external jaxamr package) fills each
// block's 3-cell ghost layers; the reference then applies, per block,
//   flux_func(U, aux) = pad(dt * total_flux(U, aux), 3)   (vmapped)
//   update_func       = update_aux                          (vmapped)
// on the ghost-padded block, and after the three stages the chemistry and
// update_aux on the unpadded blocks.  vmap makes every reduction per block:
// the LF wave-speed maxima are nanmax over the block's padded array, and the
// temperature solve stops when the block's own max |res| <= tol (JAX's
// batched while_loop keeps each block's carry once its predicate is false).
//
// Layout: blocks [nb][nv + 2][PX][PY] float64, C-contiguous (the reference's
// blk_data: U fields then gamma, T), PX = bx + 6, PY = by + 6 for padded
// blocks; the chemistry takes unpadded blocks [nb][nv + 2][bx][by].
//
// One CTA per block, so each block's reductions stay inside its CTA:
//   k_amr_stage   alpha of the padded block; the interior in tiles of
//                 tx x ty cells, a shape the host picks per block size so
//                 that few tiles cover the block (20 x 20 blocks: one) (LF + WENO5-JS
//                 / MUSCL faces in shared memory, the RK combination); every
//                 ghost entry takes the combination with a zero right-hand
//                 side (the reference pads the rhs with zeros); update_aux
//                 over the whole padded block
//   k_amr_update  update_aux of blocks alone
// update_aux runs the reference's loop in lockstep over the block: one
// Halley iteration of every cell per round, the block's OR of "residual
// above tol" / "residual NaN" deciding whether another round follows (the
// iterates live in the output's gamma / T slots), so a cell is evaluated
// once per iteration the block takes.
//   k_amr_chem    point-implicit chemistry, one thread per cell of all
//                 blocks, U + S; k_amr_update then solves the temperatures

namespace {  // internal linkage

constexpr int AMR_NT = 256;
// Shared doubles of a tx x ty tile: rho, u, v, p of its padded cells, and of
// two fields at a time the split fluxes along both axes and the face values.
__host__ __device__ constexpr int amr_tile_doubles(int tx, int ty) {
  return 4 * (tx + 6) * (ty + 6) + 4 * ((tx + 6) * ty + tx * (ty + 6)) + 2 * ((tx + 1) * ty + tx * (ty + 1));
}
constexpr int AMR_SMEM_DOUBLES = 72 * 1024 / 8;  // three blocks an SM

// Items i = tid, tid + AMR_NT, ... of an array with rows of w entries as (row,
// column), stepped without a division.
struct AmrIt {
  int r, c, dr, dc, w;
  __device__ __forceinline__ AmrIt(int tid, int w_) : r(tid / w_), c(tid % w_), dr(AMR_NT / w_), dc(AMR_NT % w_), w(w_) {}
  __device__ __forceinline__ void next() {
    r += dr;
    c += dc;
    if (c >= w) {
      c -= w;
      ++r;
    }
  }
};

struct AmrBlocks {
  int nb, bx, by, tx, ty;  // blocks, block cells, interior tile of k_amr_stage
  double dx, dy, idx, idy;
};

// Block-wide reductions (all threads of the CTA call them).
__device__ __forceinline__ void amr_block_max2(double& a, double& b) {
  __shared__ double ra[32], rb[32];
  a = warp_max(a);
  b = warp_max(b);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) { ra[w] = a; rb[w] = b; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 1; i < (int)(blockDim.x >> 5); ++i) { a = fmax(a, ra[i]); b = fmax(b, rb[i]); }
    ra[0] = a;
    rb[0] = b;
  }
  __syncthreads();
  a = ra[0];
  b = rb[0];
  __syncthreads();
}

__device__ __forceinline__ unsigned amr_block_or(unsigned v) {
  __shared__ unsigned ro[32];
  v = warp_or(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) ro[w] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 1; i < (int)(blockDim.x >> 5); ++i) v |= ro[i];
    ro[0] = v;
  }
  __syncthreads();
  v = ro[0];
  __syncthreads();
  return v;
}

// e, Y and R of a 2D state cell c (field stride nc): update_aux
// (solver_2D/aux_func.py:21-29) as the select pass forms them.
__device__ __forceinline__ void amr_eYR(const MP& m, const double* Ub, long long nc, long long c, double& e,
                                        double* Yf, double& R) {
  constexpr int nY = 4;
  const double rho = Ub[c];
  double Y8[NR];
#if JB_FAST
  const double ri = 1.0 / rho;
  const double u = Ub[nc + c] * ri, v = Ub[2 * nc + c] * ri;
  e = Ub[3 * nc + c] * ri - 0.5 * (u * u + v * v);
#pragma unroll
  for (int k = 0; k < NR; ++k) Y8[k] = Ub[(nY + k) * nc + c] * ri;
#else
  const double u = Ub[nc + c] / rho, v = Ub[2 * nc + c] / rho;
  e = Ub[3 * nc + c] / rho - 0.5 * (u * u + v * v);
#pragma unroll
  for (int k = 0; k < NR; ++k) Y8[k] = Ub[(nY + k) * nc + c] / rho;
#endif
  fill_Y(Y8, Yf);
  R = get_R(m, Yf);
}

// update_aux of the nc cells of one block (state Ub, initial temperatures
// T0b, result into Ab = [gamma][T]) with the block's global stop
// (thermo_model.py:135-153 on the vmapped block): round i evaluates the
// residual at every cell's i-th iterate; the loop ends when no residual
// exceeds tol, when one is NaN (jnp.max is then NaN and the test false) or
// after 5 iterations.  T0b may equal Ab + nc.
__device__ void amr_update_block(const MP& m, const double* Ub, const double* T0b, double* Ab, long long nc,
                                 unsigned& st) {
  double* Tn = Ab;       // each cell's next iterate (the gamma slot until the end)
  double* Tc = Ab + nc;  // its current iterate
  for (long long c = threadIdx.x; c < nc; c += blockDim.x) Tc[c] = T0b[c];
  for (int i = 0;; ++i) {
    unsigned bits = 0;
    for (long long c = threadIdx.x; c < nc; c += blockDim.x) {
      double e, Yf[NS], R;
      amr_eYR(m, Ub, nc, c, e, Yf, R);
      const double T = Tc[c];
      const Th t = thermo_mix(m, T, Yf);
      const double res = (t.h - R * T) - e;
      const double d1 = t.cp - R, d2 = t.dcp;
      if (fabs(res) > HALLEY_TOL) bits |= 1u;
      if (res != res) bits |= 2u;
      Tn[c] = T + ((-2.0 * res) * d1) / ((2.0 * (d1 * d1)) - res * d2);
    }
    bits = amr_block_or(bits);
    if (!(bits & 1u) || (bits & 2u) || i == HALLEY_MAX) break;
    for (long long c = threadIdx.x; c < nc; c += blockDim.x) Tc[c] = Tn[c];
  }
  for (long long c = threadIdx.x; c < nc; c += blockDim.x) {
    double e, Yf[NS], R;
    amr_eYR(m, Ub, nc, c, e, Yf, R);
    const double T = Tc[c];
    const double cp = cp_mix(m, T, Yf);
    Ab[c] = cp / (cp - R);
    if (!(T == T)) st |= JB_ERR_NONFINITE;
  }
}

typedef jb_amr_io AmrIO;  // the stage call's block arrays (jb_ops.h)

// STAGE 1..3: one SSP-RK3 stage of every padded block (TVD_RK3.py:17-35):
// out = a U0 + b (G + pad(dt L(G))) and its update_aux started from G's T.
// STAGE 0: the block flux function alone, out = pad(dt L(G))
// (set_simulator.py:37-40).  G: the stage input with its ghost layers
// filled; U0: the step's first stage input.
template <int STAGE>
#ifndef JB_AMR_MINB
#define JB_AMR_MINB 3
#endif
__global__ void __launch_bounds__(AMR_NT, JB_AMR_MINB) k_amr_stage(MP m, Grid g, AmrBlocks B, AmrIO io, Slots* slots,
                                                    double dt) {
  extern __shared__ __align__(128) unsigned char smraw[];
  constexpr int nv = 12;
  const int TX = B.tx, TY = B.ty, APX = TX + 6, APY = TY + 6, AQ = APX * APY;
  const int HX = APX * TY, HY = TX * APY;
  const int NFX = (TX + 1) * TY, NFY = TX * (TY + 1);
  double* sP = reinterpret_cast<double*>(smraw);  // [4][APX][APY]: rho, u, v, p
  double* sHx = sP + 4 * AQ;                       // [2 fields][H+, H-][APX][TY]
  double* sHy = sHx + 4 * HX;                      // [2][2][TX][APY]
  double* sFx = sHy + 4 * HY;                      // [2][TX+1][TY]
  double* sFy = sFx + 2 * NFX;                     // [2][TX][TY+1]
  const int tid = threadIdx.x;
  const int PX = B.bx + 6, PY = B.by + 6;
  const long long nc = (long long)PX * PY;
  const long long b = blockIdx.x;
  const double* gU = io.gU + b * io.gsU;
  const double* gA = io.gA + b * io.gsA;
  const double* u0 = STAGE >= 2 ? io.u0 + b * io.u0s : nullptr;
  double* oU = io.oU + b * io.osU;
  unsigned st = 0;

  // ---- LF wave speeds: nanmax(|u| + a), nanmax(|v| + a) over the padded
  // block (flux_splitting/LF.py:11-12 on the vmapped block)
  double ax = 0.0, ay = 0.0;
  for (long long c = tid; c < nc; c += AMR_NT) {
    double q[nv];
#pragma unroll
    for (int f = 0; f < nv; ++f) q[f] = gU[f * nc + c];
    const Prim<2> pr = u_to_prim<2>(m, q, gA[c], gA[nc + c]);
    ax = fmax(ax, fabs(pr.u) + pr.a);
    ay = fmax(ay, fabs(pr.v) + pr.a);
  }
  amr_block_max2(ax, ay);

  // ---- the interior, tile by tile
  const int ntx = (B.bx + TX - 1) / TX, nty = (B.by + TY - 1) / TY;
  for (int t = 0; t < ntx * nty; ++t) {
    const int x0 = (t / nty) * TX, y0 = (t % nty) * TY;  // interior coordinates of the tile
    // primitives of the padded tile (block padded rows x0 .. x0 + APX - 1,
    // columns y0 .. y0 + APY - 1); cells beyond the padded block are read
    // only by faces of cells outside the block
    for (int i = tid; i < AQ; i += AMR_NT) {
      const int px = x0 + i / APY, py = y0 + i % APY;
      double rho = 1.0, u = 1.0, v = 1.0, p = 1.0;
      if (px < PX && py < PY) {
        const long long c = (long long)px * PY + py;
        double q[nv];
#pragma unroll
        for (int f = 0; f < nv; ++f) q[f] = gU[f * nc + c];
        flux_prims<2>(m, q, gA[nc + c], rho, u, v, p);
      }
      sP[i] = rho;
      sP[AQ + i] = u;
      sP[2 * AQ + i] = v;
      sP[3 * AQ + i] = p;
    }
    __syncthreads();
    // two fields at a time, two barriers a pair
    for (int f0 = 0; f0 < nv; f0 += 2) {
      // split fluxes H+- = 0.5 (F +- alpha U) (flux_splitting/LF.py:4-16) of
      // tile cell (px, py) along dir into h[field][sign][n] at position k
      auto split = [&](int dir, int px, int py, double al, double* h, int n, int k) {
        const int c = px * APY + py;
        const bool in = x0 + px < PX && y0 + py < PY;
        const long long gc = (long long)(x0 + px) * PY + (y0 + py);
#if !JB_FAST
        const double E = in ? gU[3 * nc + gc] : 1.0;
#endif
#pragma unroll
        for (int d = 0; d < 2; ++d) {
          const int f = f0 + d;
          const double qf = in ? gU[f * nc + gc] : 1.0;
#if JB_FAST
          // F = vel q + pressure terms: the reference's LF flux regrouped
          const double vel = sP[(1 + dir) * AQ + c];
          double F = vel * qf;
          if (f == 1 + dir) F += sP[3 * AQ + c];
          if (f == 3) F += vel * sP[3 * AQ + c];
#else
          const double F = lf_flux<2>(f, dir, qf, sP[c], sP[AQ + c], sP[2 * AQ + c], sP[3 * AQ + c], E);
#endif
          h[(2 * d) * n + k] = 0.5 * (F + al * qf);
          h[(2 * d + 1) * n + k] = 0.5 * (F - al * qf);
        }
      };
      int k = tid;
      for (AmrIt i(tid, TY); i.r < APX; i.next(), k += AMR_NT) split(0, i.r, i.c + 3, ax, sHx, HX, k);
      k = tid;
      for (AmrIt i(tid, APY); i.r < TX; i.next(), k += AMR_NT) split(1, i.r + 3, i.c, ay, sHy, HY, k);
      __syncthreads();
      // face values F = L(H+) + R(H-) (flux.py:56-68, WENO5_JS.py / MUSCL.py)
      auto face = [&](const double* hp, const double* hm, int s) {
        return recon_L(g, hp[0], hp[s], hp[2 * s], hp[3 * s], hp[4 * s]) +
               recon_R(g, hm[s], hm[2 * s], hm[3 * s], hm[4 * s], hm[5 * s]);
      };
#pragma unroll 1
      for (int d = 0; d < 2; ++d) {
        const double* hp = sHx + 2 * d * HX;
#pragma unroll 1
        for (k = tid; k < NFX; k += AMR_NT) sFx[d * NFX + k] = face(hp + k, hp + HX + k, TY);
        const double* gp = sHy + 2 * d * HY;
        k = tid;
#pragma unroll 1
        for (AmrIt i(tid, TY + 1); i.r < TX; i.next(), k += AMR_NT) {
          const double* p = gp + i.r * APY + i.c;
          sFy[d * NFY + k] = face(p, p + HY, 1);
        }
      }
      __syncthreads();
      // divergence and the RK combination (TVD_RK3.py:17, 24, 31); the next
      // pair's split fluxes do not touch the face values
      for (AmrIt i(tid, TY); i.r < TX; i.next()) {
        const int gx = x0 + i.r, gy = y0 + i.c;
        if (gx >= B.bx || gy >= B.by) continue;
        const long long cell = (long long)(gx + 3) * PY + (gy + 3);
#pragma unroll
        for (int d = 0; d < 2; ++d) {
          const int f = f0 + d;
          const double* Fx = sFx + d * NFX + i.r * TY + i.c;
          const double* Fy = sFy + d * NFY + i.r * (TY + 1) + i.c;
          const double dF = Fx[TY] - Fx[0], dG = Fy[1] - Fy[0];
#if JB_FAST
          const double rhs = dt * (-(dF * B.idx + dG * B.idy));
#else
          const double rhs = dt * (-(dF / B.dx + dG / B.dy));
#endif
          const double uk = gU[f * nc + cell];
          double r;
          if (STAGE == 0) r = rhs;
          else if (STAGE == 1) r = uk + rhs;
          else if (STAGE == 2) r = 3.0 / 4.0 * u0[f * nc + cell] + 1.0 / 4.0 * (uk + rhs);
          else r = 1.0 / 3.0 * u0[f * nc + cell] + 2.0 / 3.0 * (uk + rhs);
          oU[f * nc + cell] = r;
        }
      }
    }
    __syncthreads();  // the next tile's primitives replace this one's
  }
  // ---- ghost entries: the combination with the zero-padded rhs
  for (long long c = tid; c < nc; c += AMR_NT) {
    const int px = (int)(c / PY), py = (int)(c % PY);
    if (px >= 3 && px < PX - 3 && py >= 3 && py < PY - 3) continue;
    for (int f = 0; f < nv; ++f) {
      const double rhs = 0.0;
      double r;
      if (STAGE == 0) r = rhs;
      else if (STAGE == 1) r = gU[f * nc + c] + rhs;
      else if (STAGE == 2) r = 3.0 / 4.0 * u0[f * nc + c] + 1.0 / 4.0 * (gU[f * nc + c] + rhs);
      else r = 1.0 / 3.0 * u0[f * nc + c] + 2.0 / 3.0 * (gU[f * nc + c] + rhs);
      oU[f * nc + c] = r;
    }
  }
  if (!(ax == ax) || !(ay == ay)) st |= JB_ERR_NONFINITE;
#if !JB_FAST
  if (STAGE > 0) {
    __syncthreads();
    // ---- update_aux of the padded block from G's temperatures (the fast
    // variants' launcher runs k_amr_update_cells on the result instead)
    amr_update_block(m, oU, gA + nc, io.oA + b * io.osA, nc, st);
  }
#endif
  st = amr_block_or(st);
  if (tid == 0 && st) atomicOr(&slots->status, st);
}

// update_aux of every block (vmap(update_aux), set_simulator.py:41) with
// each block's own stop: U [nb][nv][X][Y] (field stride nc, block stride
// su), aux_in / aux_out [nb][2][X][Y] (block strides sai, sao).
template <int UNUSED>
__global__ void __launch_bounds__(AMR_NT) k_amr_update(MP m, long long nc, const double* U, long long su,
                                                     const double* aux_in, long long sai, double* aux_out,
                                                     long long sao, Slots* slots) {
  const long long b = blockIdx.x;
  unsigned st = 0;
  amr_update_block(m, U + b * su, aux_in + b * sai + nc, aux_out + b * sao, nc, st);
  st = amr_block_or(st);
  if (threadIdx.x == 0 && st) atomicOr(&slots->status, st);
}

#if JB_FAST
// The same with each thread's CPT cells held in registers across the rounds:
// energy, gas constant, temperature and the six coefficients of the mixture
// enthalpy (mix_h; every species switches NASA7 ranges at the same
// temperature), so a round is one Horner pass and one block-wide vote
// instead of the species sums over a state read again.  676-cell padded
// blocks (20 x 20 + ghosts), 300 of them: half of the stage's 160 us before.
constexpr int AMR_UNT = 512, AMR_UCPT = 4;  // blocks of up to 2048 cells
template <int CPT>
__global__ void __launch_bounds__(AMR_UNT) k_amr_update_cells(MP m, long long nc, const double* U, long long su,
                                                           const double* aux_in, long long sai, double* aux_out,
                                                           long long sao, Slots* slots) {
  const long long b = blockIdx.x;
  const double* Ub = U + b * su;
  const double* T0 = aux_in + b * sai + nc;
  double* Ab = aux_out + b * sao;
  const double Tcr = m.Tcr[0];
  double T[CPT], e[CPT], R[CPT], H[CPT][6], cp[CPT];
  unsigned lo = 0, st = 0;
  auto cell = [&](int k) { return (long long)threadIdx.x + (long long)k * blockDim.x; };
#pragma unroll
  for (int k = 0; k < CPT; ++k) {
    const long long c = cell(k);
    if (c < nc) {
      double Yf[NS];
      amr_eYR(m, Ub, nc, c, e[k], Yf, R[k]);
      T[k] = T0[c];
      if (T[k] < Tcr) lo |= 1u << k;
      mix_h(m, Yf, T[k] < Tcr, H[k]);
    }
  }
  for (int i = 0;; ++i) {
    double Tn[CPT];
    unsigned bits = 0;
#pragma unroll
    for (int k = 0; k < CPT; ++k) {
      if (cell(k) < nc) {
        double h, dcp;
        poly6_d2(H[k], T[k], h, cp[k], dcp);
        const double res = (h - R[k] * T[k]) - e[k], d1 = cp[k] - R[k];
        if (fabs(res) > HALLEY_TOL) bits |= 1u;
        if (res != res) bits |= 2u;
        Tn[k] = halley_next(T[k], res, d1, dcp);
      }
    }
    const int go = __syncthreads_or(bits & 1u), bad = __syncthreads_or(bits & 2u);
    if (!go || bad || i == HALLEY_MAX) break;
#pragma unroll
    for (int k = 0; k < CPT; ++k) {
      const long long c = cell(k);
      if (c < nc) {
        T[k] = Tn[k];
        if ((T[k] < Tcr) != (bool)((lo >> k) & 1u)) {  // the iterate crossed the range boundary (rare)
          lo ^= 1u << k;
          double ek, Yf[NS], Rk;
          amr_eYR(m, Ub, nc, c, ek, Yf, Rk);
          mix_h(m, Yf, T[k] < Tcr, H[k]);
        }
      }
    }
  }
#pragma unroll
  for (int k = 0; k < CPT; ++k) {
    const long long c = cell(k);
    if (c < nc) {
      Ab[c] = cp[k] / (cp[k] - R[k]);
      Ab[nc + c] = T[k];
      if (!(T[k] == T[k])) st |= JB_ERR_NONFINITE;
    }
  }
  st = amr_block_or(st);
  if (threadIdx.x == 0 && st) atomicOr(&slots->status, st);
}
#endif

// Chemistry of every cell of nb unpadded blocks (the vmapped
// reaction_source_terms of set_simulator.py:109-111): out = U + S(U, T, dt),
// the flow fields copied; one thread per cell.  out may equal blk.
// GEN: the specialised chemistry (CHEM_SH shared doubles per thread).
template <bool GEN>
__global__ void __launch_bounds__(128, 3) k_amr_chem(MP m, AmrBlocks B, const double* blk, double* out,
                                                     Slots* slots, double dt) {
  extern __shared__ double shc[];
  constexpr int nY = 4, nv = 12;
  const long long nc = (long long)B.bx * B.by;
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  unsigned st = 0;
  if (i < nc * B.nb) {
    const long long b = i / nc, c = i % nc;
    const double* Ib = blk + b * (nv + 2) * nc;
    double* Ob = out + b * (nv + 2) * nc;
    const double T = Ib[(nv + 1) * nc + c];
    const double rho = Ib[c];
    double Y8[NR], S[NR];
#if JB_FAST
    const double ri = 1.0 / rho;
#pragma unroll
    for (int k = 0; k < NR; ++k) Y8[k] = Ib[(nY + k) * nc + c] * ri;
    if (GEN) chem_cell_gen(m, rho, Y8, T, dt, S, st, shc + threadIdx.x, blockDim.x);
    else chem_cell(m, rho, Y8, T, dt, S, st);
#else
#pragma unroll
    for (int k = 0; k < NR; ++k) Y8[k] = Ib[(nY + k) * nc + c] / rho;
    chem_cell(m, rho, Y8, T, dt, S, st);
#endif
#pragma unroll
    for (int f = 0; f < nY; ++f) Ob[f * nc + c] = Ib[f * nc + c];
#pragma unroll
    for (int k = 0; k < NR; ++k) Ob[(nY + k) * nc + c] = Ib[(nY + k) * nc + c] + S[k];
  }
  block_reduce_store(0.0, 0.0, 0.0, st << 16, slots, 0, false, false, -1);
}

}  // namespace
