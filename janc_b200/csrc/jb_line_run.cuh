// A whole run of 1D LF / WENO5-JS steps with chemistry as ONE persistent
// cooperative launch (included by jb_variant.inc in the LINE part of the fast
// variants).  A short line's step is a chain of short latencies; as separate
// launches (8 a step in mixed, 9 in fp64, plus the outlet strips) the host's
// 4-6 us per launch and the launch gaps outweigh it: 500 cells in fp64 took
// 69 us a step, 12000 cells in mixed with an outlet 68 us, against 52 us and
// 36 us here.
//
// Each CTA owns one tile of S cells through every phase, so the passes that
// only touch a cell's own state follow each other without a barrier; the
// reductions (alpha per stage, the CFL minimum, the global Halley mask) and
// the neighbours' halo cells need one of all CTAs:
//   mixed  stage 1 | stage 2 | stage 3, chemistry |               3 a step
//   fp64   stage 1 | select 1 | stage 2 | select 2 | stage 3 | chemistry |
//          select 4 |  (global stop, as advance_impl's sequence)   7 a step
// The arithmetic is the single launches' own (line_tile, select_cell,
// chem_cell_step), so the results are bitwise theirs.  Outlet ghost states
// have three buffers, one per state whose ghosts are read (pos 0..2 of a
// strip row), so that the CTA that writes one never races with a neighbour
// still reading another.  The slot sets alternate between even and odd steps.
//
// Every wait is bounded, after which the run is abandoned.  The first barrier
// waits for CTAs that may not be resident yet, because other streams' kernels
// (a long ensemble run, say) hold their places: up to 60 s.  After it every CTA
// is resident, and a wait is 2 s at most.  Of an abandoned run the last CTA to
// leave fills the outputs and the time steps with NaN and sets JB_ERR_TIMEOUT;
// it clears the barrier words and slot sets for the next launch in any case.
struct LineRun {
  const double *U, *aux;
  double *U_out, *aux_out, *W0, *W1, *A0, *A1, *cand, *strips;
  Slots *slots, *sets;  // the handle's slots (status), two alternating sets
  unsigned* bar;        // arrivals, departures, abort
  double dt_fixed, cfl;
  int nsteps;
  double* dt_hist;
  unsigned arrivals;             // CTAs that a barrier waits for
  unsigned count0;               // the arrival count before the first
  unsigned long long start_ns;   // how long the first may wait,
  unsigned long long limit_ns;   // and the others
};

namespace {

constexpr int LR_NT = 128;
constexpr unsigned long long LR_START_NS = 60000000000ull, LR_LIMIT_NS = 2000000000ull;
constexpr long long LR_SPIN_MAX = 1LL << 28;

__device__ __forceinline__ unsigned lr_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Barrier of all CTAs (every thread calls it); false when the run is abandoned.
__device__ __forceinline__ bool lr_sync(const LineRun& a, unsigned& target, unsigned long long limit_ns) {
  __shared__ int s_go;
  __syncthreads();
  if (a.arrivals == 1) return true;
  unsigned* bar = a.bar;
  if (threadIdx.x == 0) {
    int go = 1;
    target += a.arrivals;
    __threadfence();
    atomicAdd(&bar[0], 1u);
    unsigned long long t0 = 0;
    for (long long it = 0; !jb_arrived(lr_acquire(&bar[0]), target); ++it) {
      if (*(volatile unsigned*)&bar[2]) { go = 0; break; }
      if ((it & 63) == 0) {
        unsigned long long now;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
        if (it == 0) t0 = now;
        if (it >= LR_SPIN_MAX || now - t0 > limit_ns) {
          atomicExch(&bar[2], 1u);
          go = 0;
          break;
        }
      }
      __nanosleep(20);
    }
    __threadfence();
    s_go = go;
  }
  __syncthreads();
  return s_go != 0;
}

__device__ __forceinline__ void lr_clear(Slots* s) {
  for (int i = 0; i < 4; ++i) { s->ax[i] = 0ull; s->ay[i] = 0ull; s->mask[i] = 0u; }
  s->dtmin_next = 0x7ff0000000000000ull;
  s->dtnan = 0u;
  s->dt = 0.0;
}

// Outlet ghost states of the tile's boundary cells' new (U, gamma, T), their
// wave speeds folded into amx.
__device__ __forceinline__ void lr_strips(const MP& m, const Grid& g, int x0, int nin, const double* U,
                                          const double* aux, double* strips, double& amx) {
  if ((x0 != 0 || g.bc[0] != JB_BC_PRESSURE_OUTLET) && (x0 + nin != g.nx || g.bc[1] != JB_BC_PRESSURE_OUTLET))
    return;
  __syncthreads();
  const int side = threadIdx.x;
  if (side < 2 && g.bc[side] == JB_BC_PRESSURE_OUTLET && (side == 0 ? x0 == 0 : x0 + nin == g.nx)) {
    double amy = 0.0;
    strip_one<1>(m, g, U, aux, strips, side, 0, amx, amy);
  }
}

// 168 registers, three CTAs an SM (the chemistry's shape)
template <class V, int S>
__global__ void __launch_bounds__(LR_NT, 3)
    k_line_run(const __grid_constant__ MP m, const __grid_constant__ Grid g, const __grid_constant__ LineRun a) {
  extern __shared__ __align__(128) unsigned char smraw[];
  constexpr bool CELL = sizeof(V) == 4;
  const int tid = threadIdx.x, x0 = blockIdx.x * S, nin = min(S, g.nx - x0);
  const bool live = tid < nin;
  const long long c = x0 + tid, nc = g.ncell;
  // S == 32: the cell of the thread's lane, for the split chemistry
  const bool live32 = (tid & 31) < nin;
  const long long cl = x0 + min(tid & 31, nin - 1);
  (void)live32, (void)cl;
  const bool use_cfl = a.cfl > 0.0;
  const double inf = __longlong_as_double(0x7ff0000000000000LL);
  double* sh = reinterpret_cast<double*>(smraw) + tid;
  unsigned target = a.count0;
  bool go = true;
  {  // alpha and CFL minimum of the initial state (set 1 plays the previous step)
    double amx = 0.0, amy = 0.0, dtm = inf;
    unsigned st = 0;
    if (live)
      select_cell<1, false, true, true>(m, g, a.U, a.aux, nullptr, nullptr, a.strips, &a.sets[1], 0u, c, amx, amy,
                                        dtm, st);
    block_reduce_store(amx, amy, dtm, st << 16, &a.sets[1], 3, true, use_cfl, -1);
    go = lr_sync(a, target, a.start_ns);
  }
#pragma unroll 1
  for (int step = 0; go && step < a.nsteps; ++step) {
    Slots* cur = a.sets + (step & 1);
    Slots* prv = a.sets + ((step & 1) ^ 1);
    const double* U = step ? a.U_out : a.U;
    const double* aux = step ? a.aux_out : a.aux;
    const double dt = use_cfl ? a.cfl * (__ldcg(&prv->dtnan) ? __longlong_as_double(0x7ff8000000000000LL)
                                                             : bitsd(__ldcg(&prv->dtmin_next)))
                              : a.dt_fixed;
    if (a.dt_hist && blockIdx.x == 0 && tid == 0) a.dt_hist[step] = dt;
    if constexpr (CELL) {
      unsigned bits = 0, st = 0;
      double amx = 0.0, amy = 0.0, dtm = inf;
      // stage 1: U1 = U + L(U), (gamma, T)_1 and alpha 1
      const jb_fin f1 = jb_fin_cell(a.A0, nullptr, 1, 0);
      bits = line_tile<1, V, LR_NT, S>(m, g, U, aux, U, a.W0, f1, a.strips, bitsd(__ldcg(&prv->ax[3])), dt, x0, smraw,
                                       amx, dtm, cur);
      lr_strips(m, g, x0, nin, a.W0, a.A0, a.strips + 1, amx);
      finish_reduce(f1, amx, 0.0, dtm, bits, cur);
      if (!(go = lr_sync(a, target, a.limit_ns))) break;
      if (blockIdx.x == 0 && tid == 0) lr_clear(prv);  // every CTA has read it
      // stage 2: U2 = 3/4 U + 1/4 (U1 + L(U1))
      amx = 0.0;
      const jb_fin f2 = jb_fin_cell(a.A1, nullptr, 2, 0);
      bits = line_tile<2, V, LR_NT, S>(m, g, a.W0, a.A0, U, a.W1, f2, a.strips + 1, bitsd(__ldcg(&cur->ax[1])), dt, x0,
                                       smraw, amx, dtm, cur);
      lr_strips(m, g, x0, nin, a.W1, a.A1, a.strips + 2, amx);
      finish_reduce(f2, amx, 0.0, dtm, bits, cur);
      if (!(go = lr_sync(a, target, a.limit_ns))) break;
      // stage 3: U3 = 1/3 U + 2/3 (U2 + L(U2)); then the chemistry of the own cells
      amx = 0.0;
      bits = line_tile<3, V, LR_NT, S>(m, g, a.W1, a.A1, U, a.W0, jb_fin_cell(a.A0, nullptr, -1, 0), a.strips + 2,
                                       bitsd(__ldcg(&cur->ax[2])), dt, x0, smraw, amx, dtm, cur);
      const jb_fin f4 = jb_fin_cell(a.aux_out, nullptr, 3, use_cfl);
      if constexpr (S == 32) {
        // the other warps read what warp 0 wrote in stage 3 (line_tile ends in a block barrier)
        chem_split_step<1, false, true>(m, g, a.W0, a.A0[nc + cl], a.U_out, f4, cl, live32, dt,
                                        reinterpret_cast<double*>(smraw), bits, st, amx, amy, dtm, cur);
      } else if (live) {
        chem_cell_step<1, false, true, true>(m, g, a.W0, a.A0[nc + c], a.U_out, f4, c, dt, sh, bits, st, amx, amy,
                                             dtm, cur);
      }
      lr_strips(m, g, x0, nin, a.U_out, a.aux_out, a.strips, amx);
      finish_reduce(f4, amx, 0.0, dtm, bits | (st << 16), cur);
      go = lr_sync(a, target, a.limit_ns);
    } else {
      unsigned bits = 0, st = 0;
      double amx = 0.0, amy = 0.0, dtm = inf;
      auto select = [&](const double* Us, double* As, int midx, int aidx) {
        amx = 0.0;
        st = 0;
        if (live)
          select_cell<1, true, true, false>(m, g, Us, nullptr, a.cand, As, a.strips, cur, __ldcg(&cur->mask[midx]), c,
                                            amx, amy, dtm, st);
        block_reduce_store(amx, 0.0, inf, st << 16, cur, aidx, true, false, -1);
        return lr_sync(a, target, a.limit_ns);
      };
      // stage 1: U1 = U + L(U)
      bits = line_tile<1, V, LR_NT, S>(m, g, U, aux, U, a.W0, jb_fin_cand(a.cand, 0), a.strips,
                                       bitsd(__ldcg(&prv->ax[3])), dt, x0, smraw, amx, dtm, cur);
      finish_reduce(jb_fin_cand(a.cand, 0), 0.0, 0.0, inf, bits, cur);
      if (!(go = lr_sync(a, target, a.limit_ns))) break;
      if (blockIdx.x == 0 && tid == 0) lr_clear(prv);  // every CTA has read it
      if (!(go = select(a.W0, a.A0, 0, 1))) break;
      // stage 2: U2 = 3/4 U + 1/4 (U1 + L(U1))
      bits = line_tile<2, V, LR_NT, S>(m, g, a.W0, a.A0, U, a.W1, jb_fin_cand(a.cand, 1), a.strips,
                                       bitsd(__ldcg(&cur->ax[1])), dt, x0, smraw, amx, dtm, cur);
      finish_reduce(jb_fin_cand(a.cand, 1), 0.0, 0.0, inf, bits, cur);
      if (!(go = lr_sync(a, target, a.limit_ns))) break;
      if (!(go = select(a.W1, a.A1, 1, 2))) break;
      // stage 3: U3 = 1/3 U + 2/3 (U2 + L(U2))
      bits = line_tile<3, V, LR_NT, S>(m, g, a.W1, a.A1, U, a.W0, jb_fin_cand(a.cand, 2), a.strips,
                                       bitsd(__ldcg(&cur->ax[2])), dt, x0, smraw, amx, dtm, cur);
      finish_reduce(jb_fin_cand(a.cand, 2), 0.0, 0.0, inf, bits, cur);
      if (!(go = lr_sync(a, target, a.limit_ns))) break;
      // chemistry at the selected stage-3 iterate
      bits = st = 0;
      const long long n3 = halley_count(__ldcg(&cur->mask[2])) * nc;
      if constexpr (S == 32) {
        chem_split_step<1, false, false>(m, g, a.W0, a.cand[n3 + cl], a.U_out, jb_fin_cand(a.cand, 3), cl, live32, dt,
                                         reinterpret_cast<double*>(smraw), bits, st, amx, amy, dtm, nullptr);
      } else if (live) {
        chem_cell_step<1, false, true, false>(m, g, a.W0, a.cand[n3 + c], a.U_out, jb_fin_cand(a.cand, 3), c, dt, sh,
                                              bits, st, amx, amy, dtm, nullptr);
      }
      finish_reduce(jb_fin_cand(a.cand, 3), 0.0, 0.0, inf, bits | (st << 16), cur);
      if (!(go = lr_sync(a, target, a.limit_ns))) break;
      amx = 0.0;
      dtm = inf;
      st = 0;
      if (live)
        select_cell<1, true, true, true>(m, g, a.U_out, nullptr, a.cand, a.aux_out, a.strips, cur,
                                         __ldcg(&cur->mask[3]), c, amx, amy, dtm, st);
      block_reduce_store(amx, 0.0, dtm, st << 16, cur, 3, true, use_cfl, -1);
      go = lr_sync(a, target, a.limit_ns);
    }
  }
  __shared__ int s_gone;
  __syncthreads();
  if (tid == 0) {
    s_gone = 0;
    __threadfence();
    if (atomicAdd(&a.bar[1], 1u) == gridDim.x - 1) {  // the last to leave: no CTA waits any more
      __threadfence();
      unsigned st = atomicExch(&a.sets[0].status, 0u) | atomicExch(&a.sets[1].status, 0u);
      if (atomicExch(&a.bar[2], 0u)) {
        st |= JB_ERR_TIMEOUT;
        s_gone = 1;
      }
      if (st) atomicOr(&a.slots->status, st);
      lr_clear(&a.sets[0]);
      lr_clear(&a.sets[1]);
      a.bar[0] = 0u;
      a.bar[1] = 0u;
    }
  }
  __syncthreads();
  if (s_gone) {  // half a run is no result
    const double nan = __longlong_as_double(0x7ff8000000000000LL);
    for (long long i = tid; i < L1_NF * nc; i += LR_NT) a.U_out[i] = nan;
    for (long long i = tid; i < 2 * nc; i += LR_NT) a.aux_out[i] = nan;
    if (a.dt_hist)
      for (int i = tid; i < a.nsteps; i += LR_NT) a.dt_hist[i] = nan;
  }
}

// CTAs of k_line_run<V, S> the current device holds at once (0: no cooperative
// launch), queried once per device.
template <class V, int S>
int lr_resident(size_t sm) {
  static PerDevice known;
  return known.get([sm](int dev) {
    int n = 0, coop = 0;
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    cudaFuncSetAttribute(k_line_run<V, S>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (!coop || cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_line_run<V, S>, LR_NT, sm) != cudaSuccess) n = 0;
    return n * sm_count();
  });
}

// Launch with tiles of S cells; false, and nothing launched, where their CTAs
// do not fit the device, or not the part of it that this process may use (an
// MPS share, a green context), which only the launch itself can tell.
template <class V, int S>
bool lr_try(const MP& m, const Grid& g, LineRun& a, const jb_line_io& io, cudaStream_t st, cudaError_t& err) {
  constexpr size_t chem = sizeof(double) * (S == 32 ? CHEM_SPLIT_SH : CHEM_SH * LR_NT), line = line_smem<V, S>(), sm = chem > line ? chem : line;
  const int nb = (g.nx + S - 1) / S;
  const int fit = lr_resident<V, S>(sm);
  if (!fit || (nb > fit && !io.oversize)) return false;
  a.arrivals = (unsigned)nb + io.missing;
  void* args[] = {(void*)&m, (void*)&g, (void*)&a};
  err = cudaLaunchCooperativeKernel((void*)k_line_run<V, S>, dim3(nb), dim3(LR_NT), args, sm, st);
  if (err != cudaErrorCooperativeLaunchTooLarge) return true;
  (void)cudaGetLastError();  // refused, not failed: the next launch check must not find it
  err = cudaSuccess;
  return false;
}

}  // namespace

// The run as one launch where one tile per resident CTA covers the line (32
// cells a tile while that suffices, one per lane with the chemistry split over
// the four warps; then 58, then 122); false, and nothing launched, where it does not,
// the driver refuses the launch, or the stream is being captured (the separate
// launches are plain graph nodes).
template <class V>
static bool line_run_t(const MP& m, const Grid& g, const jb_line_io& io, cudaStream_t st, cudaError_t& err) {
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (!m.gen_ok || cudaStreamIsCapturing(st, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) return false;
  LineRun a;
  a.U = io.U; a.aux = io.aux; a.U_out = io.U_out; a.aux_out = io.aux_out;
  a.W0 = io.W0; a.W1 = io.W1; a.A0 = io.A0; a.A1 = io.A1; a.cand = io.cand; a.strips = io.strips;
  a.slots = io.slots; a.sets = io.slots + 1; a.bar = io.bar;
  a.dt_fixed = io.dt_fixed; a.cfl = io.cfl; a.nsteps = io.nsteps; a.dt_hist = io.dt_hist;
  a.count0 = io.count0;
  const unsigned long long ns = (unsigned long long)(io.wait_ms * 1e6);
  a.start_ns = ns ? ns : LR_START_NS;
  a.limit_ns = ns ? ns : LR_LIMIT_NS;
  return lr_try<V, 32>(m, g, a, io, st, err) || lr_try<V, 58>(m, g, a, io, st, err) ||
         lr_try<V, 122>(m, g, a, io, st, err);
}
bool line_run(bool mixed, const MP& m, const Grid& g, const jb_line_io& io, cudaStream_t st, cudaError_t& err) {
  return mixed ? line_run_t<float>(m, g, io, st, err) : line_run_t<double>(m, g, io, st, err);
}
