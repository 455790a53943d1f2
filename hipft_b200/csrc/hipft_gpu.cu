// hipft_gpu.cu -- host side of the B200 flux-transport library (C ABI in
// include/hipft_gpu.h).  Owns all device state behind an opaque handle and
// sequences the kernels of kernels.cuh the way HipFT's Fortran routines
// sequence their do-concurrent loops (src/hipft.f90).
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <cfloat>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <string>
#include <unordered_map>
#include <vector>

#include "../../include/hipft_gpu.h"
#include "kernels.cuh"
#include "sts_march.cuh"
#include "adv_march.cuh"
#include "adjoint.cuh"
#include "adj_march.cuh"
#include "graph_step.cuh"

using namespace hipft;

namespace {

// Constants of the reference (src/hipft.f90:83-136).
constexpr double c_pi = 3.1415926535897932;
constexpr double c_pi_i = 0.3183098861837907;
constexpr double c_twopi = 6.2831853071795864;
constexpr double c_pi_two = 1.5707963267948966;
constexpr double c_threepi_two = 4.71238898038469;
constexpr double c_d2r = 0.017453292519943295;
constexpr double c_rsun_cm2 = 4.84416e21;
constexpr double c_km_s_to_rs_hr = 0.005172413793103448;
constexpr double c_m_s_to_rs_hr = 5.172413793103448e-06;
constexpr double c_safety = 0.95;
constexpr double c_three_quarter = 0.75;
constexpr double c_quarter = 0.25;
constexpr double c_sixth = 0.16666666666666666;
constexpr double c_two_third = 0.66666666666666666;
constexpr double c_third = 0.33333333333333333;

constexpr int kNBuf = 6;  // current field + scratch: u0, dty0, two inputs and two outputs of a pass

int round_up(int a, int b) { return (a + b - 1) / b * b; }

double pow3(double c) { return c * c * c; }
double pow5(double c) { return c * c * c * c * c; }

}  // namespace

// ------------------------------------------------------------- adjoint tape
namespace {
// One RKG2 super-step of the replay.  With q == 0 the tape holds every stage:
// slots t0 = u0, t0+1 = dty0, t0+1+k = Y_k (k = 1..s-1).  With stage
// checkpoints (q > 0, even) it holds u0, dty0 and, for each block start
// c = 1, 1+q, 1+2q, ..., the pair (Y_{c-1}, Y_c) (b = block index; Y_0 = u0 is
// not stored twice); the reverse pass recomputes the stages of one block at a
// time from its pair.
struct AdjSub {
  double dtl;
  int64_t s;
  std::vector<double> uj, vj, ubj, gj;
  size_t t0;
  int64_t q = 0;
  std::vector<int64_t> cstart;        // block starts c
  std::vector<size_t> ck_prev, ck_cur;  // tape slots of Y_{c-1} (SIZE_MAX: u0) and Y_c
};

// One taped (recorded) flux_transport_step: its tape slots sit on the tape's
// stack from `first`.
struct AdjRec {
  double dt = 0.0;
  size_t first = 0;
  size_t ta1[4] = {}, ta2[4] = {};  // SSPRK(4,3) stage inputs of the advection calls
  std::vector<AdjSub> subs;         // RKG2 super-steps
};
}  // namespace

struct hipft_gpu {
  int dev = 0;
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  int ntm = 0, npm = 0, npm1 = 0, nt = 0, np = 0, nr = 0, ldt = 0, ldv = 0;
  int64_t plane = 0;
  size_t fieldn = 0;
  hipft_params P{};
  std::vector<double> Dc;
  int adv_time = 3, adv_space = 2;
  // host mesh, 1-based (element 0 unused)
  std::vector<double> t, p, th, ph, dt, dth, dp, dph, dt_i, dth_i, dp_i, dph_i, st, sth, ct, cth, st_i, sth_i;
  std::vector<void *> allocs;
  size_t dev_bytes = 0;
  unsigned char *slab = nullptr;  // unused rest of the chunk dsmall carves from
  size_t slab_left = 0;
  Mesh M{};
  DiffCoef DC{};
  Weno W{};
  Flow FL{};
  double bc_flow_n = 0, bc_flow_s = 0, bc_diff_n = 0, bc_diff_s = 0;
  // fields
  double *buf[kNBuf] = {};
  int nbuf = kNBuf;         // allocated fields
  int cur = 0;
  bool field_set = false;
  // flows
  bool have_flow = false, flow_needs_updating = false, flow2d = false, atten_set = false;
  bool have_file_flow = false;               // flows from files are the base of vt, vp
  double *d_vtf = nullptr, *d_vpf = nullptr;  // [npm][nt+1], [np][ntm+1]
  double *d_fterms = nullptr;                 // analytic terms applied over the file flow
  hipft_flow_def fdef{};
  std::vector<double> f_p0, f_p2, f_p4, f_p1, f_p3, f_p5, f_att;
  double *d_vt1 = nullptr, *d_vp1 = nullptr, *d_at1 = nullptr, *d_ap1 = nullptr;
  double *d_vt = nullptr, *d_vp = nullptr, *d_at = nullptr, *d_ap = nullptr;
  double *d_trig = nullptr, *d_atten = nullptr;
  // diffusion
  double dt_euler = 0.0;
  bool auto_sc = false;
  int64_t sts_s = 0, n_euler = 0, subcycles_state = 0;
  std::vector<double> sts_uj, sts_vj, sts_ubj, sts_gj, sts_b;
  // scratch
  double *d_ringbuf[2] = {};           // diffusion ring of a stage's input / output (fused path)
  int ring_cur = 0;
  bool dring_valid = false;            // d_ringbuf[ring_cur] holds the ring of the current field
  double *d_rpart = nullptr;
  unsigned int *d_rcount = nullptr;
  int nkb = 0;
  PairTables ptab{};        // coefficient tables of the RKG2/RKL2 passes
  int m_strips = 0, m_slots = 0;         // theta strips, resident warps of k_sts_march
  double *d_pscratch = nullptr;          // strips of k_sts_poles_any
  // adjoint: fields of one taped forward step, folded work fields (seam
  // columns stay zero), per-block partial sums and pole sums
  std::vector<double *> tape;             // tape slots (allocated in chunks, see adj_slot)
  std::vector<void *> tape_chunks;
  size_t adj_top = 0;                     // first free tape slot (recorded steps sit below, a stack)
  size_t adj_top_max = 0;                 // most tape slots in use at once since the last release
  std::vector<AdjRec> adj_recs;           // recorded steps, oldest first
  std::vector<double *> adj_block;        // stage fields of one recomputed block
  int64_t adj_tape_limit = 0;             // fields the tape may use (0: half the free memory)
  int64_t adj_force_q = 0;                // stage-checkpoint spacing forced by the caller (0: automatic)
  size_t adj_free_seen = 0;               // free device memory + 1 as seen at the run's first record (0: not yet)
  double *adjw[8] = {};
  double *d_dpart = nullptr, *d_gring = nullptr, *d_gpart[2] = {};
  double *d_dpole = nullptr;  // [nr][adj_nch] D partials of the pole-row chunks
  int adj_nch = 1;            // phi-column chunks of k_adj_pole2
  int dpart_per_r = 0;
  double *d_jpart = nullptr;  // D partials of the marching passes, [nr][jpart_per_r]
  int jpart_per_r = 0;        // 0: the grid is not theirs
  int pass_clusters = 0;         // clusters of a merged pass that the GPU holds; 0: not on this grid
  int j_strips = 0, j_cols = 0;  // their theta strips and columns per warp
  bool adj_ready = false;        // adj_ensure has succeeded
  // ragged batches: every realization keeps the schedule it would have if run
  // alone (Euler limit, CFL substeps, PTL subcycles, stage counts)
  bool ragged = false;
  std::vector<double> r_dt_euler, r_dtmax;
  bool r_dtmax_valid = false;
  int *d_rlist_dif = nullptr, *d_rlist_adv = nullptr;  // [nr] realization lists of the launches
  StageCoef *d_rcoef = nullptr;                         // [passes][nr][4] coefficients of a super-step
  size_t rcoef_passes = 0;
  double *d_rlen = nullptr;                             // [nr] super-step lengths
  double *d_rdt = nullptr;                              // [nr] advection substeps
  unsigned long long *d_rbits = nullptr;                // [2*nr] per-realization reductions
  std::vector<int64_t> r_s, r_cycles, r_substeps;       // the last step's schedule
  int64_t rkg2_cell_stages = 0;  // unique cells x stages k >= 2 advanced (both modes)
  // steps run as one CUDA graph each (hipft_gpu_set_graph)
  bool graph_on = false;
  cudaGraph_t g_graph = nullptr;
  cudaGraphExec_t g_exec = nullptr;
  cudaStream_t g_side[3] = {};      // streams the step (and its loop bodies) are captured on
  GArrays GA{};                     // device schedule arrays
  int g_cur = -1;                   // buffer the capture used as the field
  bool g_pdl = true;                // programmatic launches inside the captured pass loop
  std::vector<unsigned char> g_key; // launch parameters the capture baked in
  GState g_last{};                  // statistics of the last graph-run step
  bool g_stats_valid = true;        // g_last read back since the last launch
  hipft_allreduce_cb red_cb = nullptr;  // scalar all-reduce over ranks (plain-mode sharding)
  void *red_user = nullptr;
  mutable std::vector<const void *> smem_set;  // kernels whose shared-memory limit this handle has set
  int *d_err = nullptr;   // set by kernels whose bounded waits gave up
  int num_sms = 148;
  unsigned long long *d_bits = nullptr;
  double *d_part = nullptr;
  size_t part_cap = 0;
  double *h_pin = nullptr;
  // analysis
  double *d_anw = nullptr;
  double *d_adj_delta = nullptr;  // increment of a balanced assimilation, recomputed by its reverse
  unsigned char *d_masks = nullptr;
  std::vector<double> da_t, da_p;
  int vmode = 0;
  double *d_fval_u0 = nullptr, *d_vscale = nullptr, *d_vgauss = nullptr;
  double vwidth = 0.03, vt_const = 0.0, vp_omega = 0.0, vtime_start = 0.0;
  // assimilation
  double *d_da = nullptr, *d_daopt = nullptr;
  double *d_daw = nullptr;                   // mu^power weight planes
  int *d_dawidx = nullptr;                   // [nr+1] plane of each realization
  double *d_dawkey = nullptr;                // [nr][2] power and limit of each plane
  size_t daw_cap = 0;
  // sources: file term (one plane), two RFE frames, the blended source
  double *d_src_file = nullptr, *d_rfe[2] = {}, *d_src = nullptr, *d_rnd = nullptr, *d_rfe_aux = nullptr;
  bool src_set = false;
  int *d_tidx = nullptr;
  std::string err;
  int64_t launches = 0, cell_updates = 0;
  int64_t rkg2_stages = 0;  // RKG2/RKL2 stages k >= 2 run (fused kernels)
  // optional per-kernel event timing
  bool profiling = false;
  std::vector<cudaEvent_t> ev_pool;
  std::vector<std::pair<cudaEvent_t, cudaEvent_t>> ev_pending[HIPFT_K_NKINDS];
  double prof_ms[HIPFT_K_NKINDS] = {};
  int64_t prof_n[HIPFT_K_NKINDS] = {};
};

static void graph_release(hipft_gpu *h);

// Event pair around one launch when profiling (returns the stop event).
struct ProfScope {
  hipft_gpu *h;
  int kind;
  cudaEvent_t a = nullptr, b = nullptr;
  static cudaEvent_t take(hipft_gpu *h) {
    if (!h->ev_pool.empty()) {
      cudaEvent_t e = h->ev_pool.back();
      h->ev_pool.pop_back();
      return e;
    }
    cudaEvent_t e = nullptr;
    if (cudaEventCreate(&e) != cudaSuccess) return nullptr;
    return e;
  }
  ProfScope(hipft_gpu *hh, int k) : h(hh), kind(k) {
    if (!h->profiling) return;
    a = take(h);
    b = take(h);
    if (a) cudaEventRecord(a, h->stream);
  }
  ~ProfScope() {
    if (!h->profiling || !a || !b) return;
    cudaEventRecord(b, h->stream);
    h->ev_pending[kind].push_back({a, b});
  }
};

// ------------------------------------------------------------------ errors
static int fail(hipft_gpu *h, int code, const char *fmt, ...) {
  char msg[512];
  va_list ap;
  va_start(ap, fmt);
  std::vsnprintf(msg, sizeof msg, fmt, ap);
  va_end(ap);
  if (h) h->err = msg;
  return code;
}

#define CK(h, call)                                                                         \
  do {                                                                                      \
    cudaError_t e_ = (call);                                                                \
    if (e_ != cudaSuccess)                                                                  \
      return fail((h), HIPFT_ECUDA, "%s:%d %s: %s", __FILE__, __LINE__, #call,              \
                  cudaGetErrorString(e_));                                                  \
  } while (0)

#define LAUNCHED(h)                                                                         \
  do {                                                                                      \
    (h)->launches++;                                                                        \
    cudaError_t e_ = cudaPeekAtLastError();                                                 \
    if (e_ != cudaSuccess)                                                                  \
      return fail((h), HIPFT_ECUDA, "%s:%d kernel launch: %s", __FILE__, __LINE__,          \
                  cudaGetErrorString(e_));                                                  \
  } while (0)

// MIN/MAX of a scalar over the ranks sharing a run; a no-op on one process
static int allreduce(hipft_gpu *h, int op, double *v) {
  if (!h->red_cb) return HIPFT_OK;
  if (h->red_cb(h->red_user, op, v) != 0) return fail(h, HIPFT_ECOMM, "all-reduce callback failed");
  return HIPFT_OK;
}

template <typename T>
static int dalloc(hipft_gpu *h, T **p, size_t n) {
  size_t bytes = std::max<size_t>(n, 1) * sizeof(T);
  cudaError_t e = cudaMalloc((void **)p, bytes);
  if (e != cudaSuccess) {
    cudaGetLastError();  // reported here: a later launch does not take it for its own
    return fail(h, HIPFT_ENOMEM, "cudaMalloc(%zu bytes): %s", bytes, cudaGetErrorString(e));
  }
  h->allocs.push_back((void *)*p);
  h->dev_bytes += bytes;
  return HIPFT_OK;
}

template <typename T>
static int upload(hipft_gpu *h, T *d, const std::vector<T> &v) {
  CK(h, cudaMemcpyAsync(d, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, h->stream));
  return HIPFT_OK;
}

#define TRY(x)                 \
  do {                         \
    int rc_ = (x);             \
    if (rc_ != HIPFT_OK) return rc_; \
  } while (0)

// A small array that lives as long as the handle, from a chunk shared with
// others: an allocation and its release take 60 us or more each, and a handle
// has some thirty of them.
template <typename T>
static int dsmall(hipft_gpu *h, T **p, size_t n) {
  constexpr size_t kChunk = (size_t)1 << 18, kAlign = 256;
  const size_t bytes = (std::max<size_t>(n, 1) * sizeof(T) + kAlign - 1) / kAlign * kAlign;
  if (bytes > kChunk / 4) return dalloc(h, p, n);
  if (bytes > h->slab_left) {
    TRY(dalloc(h, &h->slab, kChunk));
    h->slab_left = kChunk;
  }
  *p = reinterpret_cast<T *>(h->slab);
  h->slab += bytes;
  h->slab_left -= bytes;
  return HIPFT_OK;
}

// An array made on first use; one that an earlier call got before it ran out of
// memory is kept.
template <typename T>
static int once(hipft_gpu *h, T **p, size_t n) {
  return *p ? HIPFT_OK : dsmall(h, p, n);
}

// Fields that live as long as the handle, several per allocation while they
// are small (at most 256 MB each, as the tape's chunks); those that an earlier
// call got before it ran out of memory are kept.
static int dfields(hipft_gpu *h, double **f, int n) {
  const size_t per = std::max<size_t>(1, ((size_t)256 << 20) / (h->fieldn * sizeof(double)));
  int b = 0;
  while (b < n && f[b]) ++b;
  while (b < n) {
    const int c = (int)std::min<size_t>(per, (size_t)(n - b));
    double *q = nullptr;
    TRY(dalloc(h, &q, h->fieldn * c));
    for (int e = 0; e < c; ++e) f[b + e] = q + e * h->fieldn;
    CK(h, cudaMemsetAsync(q, 0, h->fieldn * c * sizeof(double), h->stream));
    b += c;
  }
  return HIPFT_OK;
}

// ------------------------------------------------------------- set_mesh
// src/hipft.f90:6495-6653, restated on 1-based host vectors.
static int set_mesh(hipft_gpu *h, const double *tin, const double *pin) {
  const double eps = 1.e-5;
  int ntm = h->ntm, npm = h->npm, nt = h->nt, np = h->np, npm1 = h->npm1, ntm1 = h->ntm;
  auto &t = h->t, &p = h->p;
  t.assign(ntm + 1, 0.0);
  p.assign(npm + 1, 0.0);
  for (int j = 1; j <= ntm; ++j) t[j] = tin[j - 1];
  for (int k = 1; k <= npm1; ++k) p[k] = pin[k - 1];
  p[npm1 + 1] = p[2] + c_twopi;
  if (std::fabs(t[1]) > eps || std::fabs(t[ntm] - c_pi) > eps || std::fabs(p[1]) > eps ||
      std::fabs(p[npm - 1] - c_twopi) > eps)
    return fail(h, HIPFT_EINVAL, "set_mesh: the mesh does not cover the sphere (t in [0,pi], p in [0,2pi])");
  h->th.assign(nt + 1, 0); h->dth.assign(nt + 1, 0); h->dth_i.assign(nt + 1, 0);
  h->sth.assign(nt + 1, 0); h->sth_i.assign(nt + 1, 0); h->cth.assign(nt + 1, 0);
  h->dt.assign(ntm + 1, 0); h->dt_i.assign(ntm + 1, 0); h->st.assign(ntm + 1, 0);
  h->st_i.assign(ntm + 1, 0); h->ct.assign(ntm + 1, 0);
  h->ph.assign(np + 1, 0); h->dph.assign(np + 1, 0); h->dph_i.assign(np + 1, 0);
  h->dp.assign(npm + 1, 0); h->dp_i.assign(npm + 1, 0);
  auto &th = h->th, &dth = h->dth, &dt = h->dt, &ph = h->ph, &dph = h->dph, &dp = h->dp;
  for (int i = 2; i <= ntm1; ++i) {
    th[i] = 0.5 * (t[i] + t[i - 1]);
    dth[i] = t[i] - t[i - 1];
  }
  th[1] = th[2] - dth[2];
  th[nt] = th[ntm1] + dth[ntm1];
  dth[1] = dth[2];
  dth[nt] = dth[ntm1];
  for (int i = 1; i <= nt; ++i) h->dth_i[i] = 1.0 / dth[i];
  for (int i = 1; i <= ntm; ++i) {
    dt[i] = th[i + 1] - th[i];
    h->dt_i[i] = 1.0 / dt[i];
  }
  for (int i = 1; i <= ntm; ++i) h->st[i] = std::sin(t[i]);
  h->st[1] = 0.0;
  h->st[ntm] = 0.0;
  for (int i = 1; i <= ntm; ++i) h->ct[i] = std::cos(t[i]);
  h->ct[1] = 1.0;
  h->ct[ntm] = 1.0;
  for (int i = 2; i <= ntm - 1; ++i) h->st_i[i] = 1.0 / h->st[i];
  for (int i = 1; i <= nt; ++i) h->sth[i] = std::sin(std::fabs(th[i]));
  for (int i = 2; i <= ntm1; ++i) h->sth_i[i] = 1.0 / h->sth[i];
  for (int i = 1; i <= nt; ++i) h->cth[i] = std::cos(th[i]);
  for (int i = 2; i <= np; ++i) {
    ph[i] = 0.5 * (p[i] + p[i - 1]);
    dph[i] = p[i] - p[i - 1];
  }
  ph[1] = ph[npm1] - c_twopi;
  dph[1] = dph[npm1];
  for (int i = 1; i <= np; ++i) h->dph_i[i] = 1.0 / dph[i];
  for (int i = 1; i <= npm - 1; ++i) dp[i] = ph[i + 1] - ph[i];
  dp[npm] = dp[2];
  for (int i = 1; i <= npm; ++i) h->dp_i[i] = 1.0 / dp[i];
  return HIPFT_OK;
}

// load_weno grid weights (src/hipft.f90:6893-6932); 7 theta + 7 phi arrays.
static void weno_weights(const hipft_gpu *h, std::vector<double> wt[7], std::vector<double> wp[7]) {
  int nt = h->nt, np = h->np, ntm = h->ntm, npm = h->npm;
  for (int q = 0; q < 7; ++q) {
    wt[q].assign(nt + 2, 0.0);
    wp[q].assign(np + 2, 0.0);
  }
  for (int j = 1; j <= ntm; ++j) wt[6][j] = (h->P.weno_eps <= 0.0) ? h->dt[j] : h->P.weno_eps;
  for (int k = 1; k <= npm; ++k) wp[6][k] = (h->P.weno_eps <= 0.0) ? h->dp[k] : h->P.weno_eps;
  auto fill = [](std::vector<double> *w, const std::vector<double> &d, int lo, int hi) {
    for (int j = lo; j <= hi; ++j) {
      double tot = d[j - 1] + d[j] + d[j + 1];
      w[0][j] = d[j] / (d[j] + d[j + 1]);          // D_C_CP
      w[1][j] = d[j] / (d[j - 1] + d[j]);          // D_C_MC
      w[2][j] = d[j - 1] / tot;                    // D_M_T
      w[3][j] = (d[j] + d[j + 1]) / tot;           // D_CP_T
      w[4][j] = d[j + 1] / tot;                    // D_P_T
      w[5][j] = (d[j - 1] + d[j]) / tot;           // D_MC_T
    }
  };
  fill(wt, h->dt, 2, nt - 2);
  fill(wp, h->dp, 2, np - 1);
  for (int q = 0; q < 6; ++q) {
    wp[q][1] = wp[q][np - 1];
    wp[q][np] = wp[q][2];
  }
}

// Scratch buffer n (0,1,2) other than the current field.
static int scratch(const hipft_gpu *h, int n) {
  int c = 0;
  for (int b = 0; b < h->nbuf; ++b) {
    if (b == h->cur) continue;
    if (c == n) return b;
    ++c;
  }
  return -1;
}

static dim3 stage_grid(const hipft_gpu *h, int tj, int tk) {
  return dim3((unsigned)((h->ntm + tj - 1) / tj), (unsigned)((h->npm - 2 + tk - 1) / tk), (unsigned)h->nr);
}

static int ensure_part(hipft_gpu *h, size_t n) {
  if (n <= h->part_cap) return HIPFT_OK;
  if (h->d_part) {
    cudaFree(h->d_part);
    h->allocs.erase(std::remove(h->allocs.begin(), h->allocs.end(), (void *)h->d_part), h->allocs.end());
  }
  h->d_part = nullptr;
  h->part_cap = 0;
  TRY(dalloc(h, &h->d_part, n));
  h->part_cap = n;
  return HIPFT_OK;
}

static int sync_read(hipft_gpu *h, const void *dsrc, size_t bytes) {
  CK(h, cudaMemcpyAsync(h->h_pin, dsrc, bytes, cudaMemcpyDeviceToHost, h->stream));
  CK(h, cudaStreamSynchronize(h->stream));
  return HIPFT_OK;
}

// ------------------------------------------------------------- kernels glue
static int ring_diffusion(hipft_gpu *h, const double *x, double *ring) {
  ProfScope ps(h, HIPFT_K_RING);
  k_ring_diffusion<<<h->nr, 256, 0, h->stream>>>(h->M, h->DC, x, ring);
  LAUNCHED(h);
  return HIPFT_OK;
}

// Diffusion ring sums of the current field, reused while the field is
// unchanged (the fused stages leave the ring of their output behind).
static int current_dring(hipft_gpu *h, const double **ring) {
  if (!h->dring_valid) {
    TRY(ring_diffusion(h, h->buf[h->cur], h->d_ringbuf[h->ring_cur]));
    h->dring_valid = true;
  }
  *ring = h->d_ringbuf[h->ring_cur];
  return HIPFT_OK;
}

constexpr int kKPT3 = 4;  // phi columns per thread of the explicit Euler kernel (two rows per thread)

// One explicit Euler step, k_euler_step; leaves the ring sums of its output
// for the next.
static int euler_step(hipft_gpu *h, const double *x, double *out, double dte) {
  const int nkb = (h->npm - 2 + kKPT3 - 1) / kKPT3;
  RingOut ro{h->d_ringbuf[1 - h->ring_cur], h->d_rpart, h->d_rcount, nkb};
  {
    ProfScope ps(h, HIPFT_K_OTHER);
    // odd ntm: keep the thread owning row ntm off lane 0 (row ntm-1 is its left neighbour)
    const int jshift = (h->ntm % 2 == 1 && ((h->ntm - 1) / 2) % 32 == 0) ? 1 : 0;
    const int nthr = (h->ntm + 2 * jshift + 1) / 2;
    dim3 grd((unsigned)((nthr + 127) / 128), (unsigned)nkb, (unsigned)h->nr);
    k_euler_step<kKPT3><<<grd, 128, 0, h->stream>>>(h->M, h->DC.dfac, x, out, h->d_ringbuf[h->ring_cur],
                                                    h->bc_diff_n, h->bc_diff_s, dte, ro, jshift);
    LAUNCHED(h);
  }
  h->ring_cur = 1 - h->ring_cur;  // the output's ring is now current
  return HIPFT_OK;
}

// HIPFT_PDL=0 turns off the programmatic (overlapping) launches.
static bool ws_pdl() {
  static int v = -1;
  if (v < 0) {
    const char *e = std::getenv("HIPFT_PDL");
    v = (e && std::atoi(e) == 0) ? 0 : 1;
  }
  return v == 1;
}

static int check_wait_flag(hipft_gpu *h, const char *what);

// ------------------------------------------------ four stages per pass
// The fixed part of a pass's arguments.
static MarchArgs march_args(const hipft_gpu *h, const double *u0, const double *dty0) {
  MarchArgs a{};
  a.u = u0;
  a.d = dty0;
  a.nreal = h->nr;
  a.strips = h->m_strips;
  a.dfac = h->DC.dfac;
  a.bcn = h->bc_diff_n;
  a.bcs = h->bc_diff_s;
  a.err = h->d_err;
  return a;
}

// The pole strips in one launch, a column per thread (k_sts_poles), or stage by
// stage (k_sts_poles_any, and k_sts_whole on a low grid).
static bool poles_by_column(const hipft_gpu *h) {
  return h->ntm >= kMMinRows && poles_threads(h->npm - 2) <= kPMaxThreads;
}

// Places of k_sts_march's blocks that one realization's strips take: a block of
// the widest takes an SM; none where the strips' launches are over by then.
static int pole_places(int n2) {
  if (poles_threads(n2) > kPMaxThreads) return 0;
  return 2 * poles_ranks(n2) * (poles_threads(n2) > kPMidThreads ? kMBlocks : 1);
}

static int march_columns(const hipft_gpu *h, int nreal) {
  const int n2 = h->npm - 2;
  return march_cols(n2, h->m_strips, nreal, h->m_slots, pole_places(n2));
}

static int64_t march_blocks(const hipft_gpu *h, int nreal) {
  return march_units(h->npm - 2, h->m_strips, march_columns(h, nreal), kMWarps) * nreal;
}

// Before a kernel's first launch by this handle: the most dynamic shared memory
// that it takes.  The limit is the kernel's, not the handle's, so `bytes` is the
// most that any grid takes; setting it loads the kernel, which is why a handle
// does it for the kernels it runs and not for all it might (0.5 ms in a process).
static cudaError_t smem_limit(const hipft_gpu *h, const void *kernel, size_t bytes) {
  if (std::find(h->smem_set.begin(), h->smem_set.end(), kernel) != h->smem_set.end()) return cudaSuccess;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess) h->smem_set.push_back(kernel);
  return e;
}

// k_sts_march for these arguments; byte offsets in 32 bits while a plane has them.
typedef void (*MarchKernel)(Mesh, MarchArgs, PairTables);
template <typename Off>
static MarchKernel march_kernel(bool table, bool keep) {
  if (keep) return table ? k_sts_march<true, true, Off, false> : k_sts_march<false, true, Off, false>;
  return table ? k_sts_march<true, false, Off, false> : k_sts_march<false, false, Off, false>;
}
static MarchKernel march_kernel(bool table, bool keep, bool wide) {
  return wide ? march_kernel<uint64_t>(table, keep) : march_kernel<uint32_t>(table, keep);
}

// Both parts of a pass in one launch, where the host knows its realizations, and
// the columns per warp with which the GPU holds all of it at once; 0 columns: two
// launches.
static MarchKernel pass_kernel(bool table, bool keep) {
  return table ? (keep ? k_sts_march<true, true, uint32_t, true> : k_sts_march<true, false, uint32_t, true>)
               : (keep ? k_sts_march<false, true, uint32_t, true> : k_sts_march<false, false, uint32_t, true>);
}
static int pass_columns(const hipft_gpu *h, const MarchArgs &a) {
  if (!h->pass_clusters || a.dctr) return 0;
  const int n2 = h->npm - 2, nc = poles_ranks(n2), nw = poles_threads(n2) / 32;
  const int64_t free = ((int64_t)h->pass_clusters - 2 * a.nreal) * nc;
  if (free < 1) return 0;
  const int64_t nch = free / a.nreal * nw / h->m_strips;
  if (nch < 1) return 0;
  const int64_t c = ((n2 + nch - 1) / nch + kMGroup - 1) / kMGroup * kMGroup;
  return c <= kPassColsMax ? (int)c : 0;
}

// k_sts_march of a pass, on the stream of cfg behind the strips' launches.
static cudaError_t launch_march(const hipft_gpu *h, cudaLaunchConfig_t cfg, cudaLaunchAttribute *attr,
                                const MarchArgs &a, int64_t blocks, bool pdl) {
  attr[0].val.programmaticStreamSerializationAllowed = pdl ? 1 : 0;
  cfg.numAttrs = 1;
  cfg.gridDim = dim3((unsigned)blocks);
  cfg.blockDim = dim3(32 * kMWarps);
  cfg.dynamicSmemBytes = kMSmem;
  const MarchKernel kernel = march_kernel(a.rc || a.cols > kMGroup, a.o[0] || a.o[1], h->plane >= (int64_t)1 << 29);
  const cudaError_t e = smem_limit(h, (const void *)kernel, kMSmem);
  return e == cudaSuccess ? cudaLaunchKernelEx(&cfg, kernel, h->M, a, h->ptab) : e;
}

// One pass on stream s.  after_pass: the launch before it on the stream is
// the previous pass, whose end it waits for on the device, so it may be
// launched programmatically.  blocks: k_sts_march's grid (0: for a.nreal
// realizations, and so its columns per warp).
static cudaError_t launch_pass(const hipft_gpu *h, cudaStream_t s, MarchArgs a, bool pdl, bool after_pass,
                               int64_t blocks = 0) {
  if (!blocks) {
    blocks = march_blocks(h, a.nreal);
    a.cols = march_columns(h, a.nreal);
  }
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const int n2 = h->npm - 2, nc = poles_ranks(n2);
  if (!poles_by_column(h)) {
    const bool low = h->ntm < kMMinRows;
    cfg.gridDim = dim3((unsigned)poles_any_blocks(n2), low ? 1 : 2, (unsigned)a.nreal);
    cfg.blockDim = dim3(kPAThreads);
    const int s0 = after_pass ? 0 : -1;
    int step = 1;
    if (cfg.gridDim.x <= kPACluster) {
      step = kMS - s0;
      attr[1].id = cudaLaunchAttributeClusterDimension;
      attr[1].val.clusterDim.x = cfg.gridDim.x;
      attr[1].val.clusterDim.y = 1;
      attr[1].val.clusterDim.z = 1;
      cfg.numAttrs = cfg.gridDim.x > 1 ? 2 : 1;
    }
    for (int st = s0; st < kMS; st += step) {
      attr[0].val.programmaticStreamSerializationAllowed = (pdl && (after_pass || st > s0)) ? 1 : 0;
      const cudaError_t e = cudaLaunchKernelEx(&cfg, low ? k_sts_whole : k_sts_poles_any, h->M, a, h->ptab,
                                               h->d_pscratch, st, st + step);
      if (e != cudaSuccess) return e;
    }
    return low ? cudaSuccess : launch_march(h, cfg, attr, a, blocks, pdl);
  }
  attr[0].val.programmaticStreamSerializationAllowed = (pdl && after_pass) ? 1 : 0;
  if (const int pc = pass_columns(h, a)) {
    a.cols = pc;
    const int64_t mb = march_units(n2, h->m_strips, pc, poles_threads(n2) / 32) * a.nreal;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)nc;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.numAttrs = 2;
    cfg.gridDim = dim3((unsigned)(2 * a.nreal * nc + (mb + nc - 1) / nc * nc));
    cfg.blockDim = dim3((unsigned)poles_threads(n2));
    cfg.dynamicSmemBytes = pass_smem(poles_threads(n2));
    const MarchKernel kernel = pass_kernel(a.rc || pc > kMGroup, a.o[0] || a.o[1]);
    const cudaError_t e = smem_limit(h, (const void *)kernel, pass_smem(kPassThreads));
    return e == cudaSuccess ? cudaLaunchKernelEx(&cfg, kernel, h->M, a, h->ptab) : e;
  }
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)nc;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.numAttrs = 2;
  cfg.gridDim = dim3((unsigned)(2 * a.nreal * nc));
  cfg.blockDim = dim3((unsigned)poles_threads(n2));
  cfg.dynamicSmemBytes = poles_smem(poles_threads(n2));
  // a march that leaves places free does not compete with the pole strips' registers
  const bool roomy = blocks + 3 * (int64_t)cfg.gridDim.x <= (int64_t)kMBlocks * h->num_sms;
  const MarchKernel poles = poles_threads(n2) > kPMidThreads    ? k_sts_poles<kPMaxThreads, 1>
                            : poles_threads(n2) <= kPMinThreads ? k_sts_poles<kPMinThreads, 3>
                            : roomy                             ? k_sts_poles<kPMidThreads, 1>
                                                                : k_sts_poles<kPMidThreads, 3>;
  cudaError_t e = smem_limit(h, (const void *)poles, poles_smem(poles_most_threads(n2)));
  if (e != cudaSuccess) return e;
  e = cudaLaunchKernelEx(&cfg, poles, h->M, a, h->ptab);
  return e == cudaSuccess ? launch_march(h, cfg, attr, a, blocks, pdl) : e;
}

static int pass_launches(const hipft_gpu *h, const MarchArgs &a, bool after_pass) {
  if (poles_by_column(h)) return pass_columns(h, a) ? 1 : 2;
  const int strips = poles_any_blocks(h->npm - 2) <= kPACluster ? 1 : kMS + (after_pass ? 0 : 1);
  return strips + (h->ntm < kMMinRows ? 0 : 1);
}

static int sts_pass(hipft_gpu *h, const MarchArgs &a, bool after_pass) {
  ProfScope ps(h, HIPFT_K_STS);
  const cudaError_t e = launch_pass(h, h->stream, a, ws_pdl(), after_pass);
  if (e != cudaSuccess) return fail(h, HIPFT_ECUDA, "RKG2 pass launch: %s", cudaGetErrorString(e));
  h->launches += pass_launches(h, a, after_pass);
  return HIPFT_OK;
}

// The seam columns of a field whose core columns the passes wrote.
static int seam(hipft_gpu *h, double *f) {
  ProfScope ps(h, HIPFT_K_OTHER);
  k_seam<<<dim3((unsigned)((h->ntm + 127) / 128), (unsigned)h->nr), 128, 0, h->stream>>>(h->M, h->ntm, h->ldt, f);
  LAUNCHED(h);
  return HIPFT_OK;
}

// dty0 = dtl * A u0 from A u0 (src/hipft.f90:5211), for all realizations or
// for the n of a list with a length each.
static int scale_dty0(hipft_gpu *h, const double *af, double *dty0, double dtl, const int *rlist = nullptr, int n = 0,
                      const double *rlen = nullptr) {
  ProfScope ps(h, HIPFT_K_OTHER);
  const unsigned chunks = (unsigned)std::min<int64_t>((h->plane / 2 + 255) / 256, 4 * h->num_sms);
  k_scale<<<dim3(chunks, (unsigned)(rlist ? n : h->nr)), 256, 0, h->stream>>>(h->plane, af, dty0, dtl, rlist, rlen);
  LAUNCHED(h);
  return HIPFT_OK;
}

// chained: the launch before it on the stream is a diffusion stage too.
template <int MODE>
static int diffusion_stage(hipft_gpu *h, const double *x, const double *ykm2, const double *u0, const double *dty0,
                           double *out, double *out2, StageCoef sc, bool chained) {
  ProfScope ps(h, MODE == MODE_STSK ? HIPFT_K_STS : HIPFT_K_OTHER);
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = (ws_pdl() && chained) ? 1 : 0;
  cfg.stream = h->stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cfg.gridDim = stage_grid(h, 32, 8 * kDCols);
  const int prows = pole_grid_rows(h->npm - 2, cfg.gridDim.x);
  cfg.gridDim.y += prows;
  cfg.blockDim = dim3(32, 8);
  CK(h, cudaLaunchKernelEx(&cfg, k_diffusion_stage<MODE>, h->M, h->DC, x, ykm2, u0, dty0, out, out2, h->bc_diff_n,
                           h->bc_diff_s, sc, prows));
  LAUNCHED(h);
  return HIPFT_OK;
}

// Grid of k_ax and k_ptl over n realizations.
static dim3 ax_grid(const hipft_gpu *h, int n) {
  return dim3((unsigned)((h->ntm + 31) / 32), (unsigned)((h->npm - 2 + 8 * kAxCols - 1) / (8 * kAxCols)), (unsigned)n);
}

// Maxima of k_ax's blocks.
static unsigned long long *ax_block_max(const hipft_gpu *h) { return h->d_bits + 4; }

// A u0 of the current field into scratch buffer 0 and, with absmax, the largest
// |A u0| of all realizations or of each of the n in rlist (per_real).
static int apply_lap(hipft_gpu *h, unsigned long long *absmax, const int *rlist, int n, int per_real) {
  const double *ring;
  TRY(current_dring(h, &ring));
  ProfScope ps(h, HIPFT_K_OTHER);
  k_ax<<<ax_grid(h, n), dim3(32, 8), 0, h->stream>>>(h->M, h->DC, h->buf[h->cur], h->buf[scratch(h, 0)], ring,
                                                     h->bc_diff_n, h->bc_diff_s, absmax, ax_block_max(h), rlist,
                                                     per_real);
  LAUNCHED(h);
  return HIPFT_OK;
}
static int ptl_cells(hipft_gpu *h, const unsigned long long *absmax, unsigned long long *ptl, const int *rlist, int n,
                     int per_real) {
  ProfScope ps(h, HIPFT_K_OTHER);
  k_ptl<<<ax_grid(h, n), dim3(32, 8), 0, h->stream>>>(h->M, h->buf[h->cur], h->buf[scratch(h, 0)], absmax,
                                                      ax_block_max(h), ptl, rlist, per_real);
  LAUNCHED(h);
  return HIPFT_OK;
}

// One explicit advection stage over nz realization slots (rlist maps slot z
// to a realization when non-null; rdt scales each realization's step), on
// stream s.  chained: the launch before it on the stream is the stage before.
typedef void (*AdvKernel)(Mesh, Flow, Weno, AdvArgs);
template <typename Off, bool BOTH, int HB>
static AdvKernel adv_kernel(bool flow2d, bool mode) {
  return flow2d ? (mode ? k_adv_march<true, 1, Off, BOTH, HB> : k_adv_march<true, 0, Off, BOTH, HB>)
                : (mode ? k_adv_march<false, 1, Off, BOTH, HB> : k_adv_march<false, 0, Off, BOTH, HB>);
}
static AdvKernel adv_kernel(bool flow2d, bool mode, bool wide, bool both, int hb) {
  if (wide) return adv_kernel<uint64_t, false, 1>(flow2d, mode);
  if (!both) return adv_kernel<uint32_t, false, 1>(flow2d, mode);
  return hb == 2 ? adv_kernel<uint32_t, true, 2>(flow2d, mode) : adv_kernel<uint32_t, true, 1>(flow2d, mode);
}

static cudaError_t launch_adv_stage(const hipft_gpu *h, cudaStream_t s, unsigned nz, const double *x, const double *f0,
                                    double *out, AdvCombine cb, const int *rlist, const double *rdt, bool pdl,
                                    bool chained) {
  if (h->adv_space != 2) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = (pdl && chained) ? 1 : 0;
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cfg.gridDim = dim3((unsigned)((h->ntm + 31) / 32), (unsigned)((h->npm - 2 + 7) / 8), nz);
    const int prows = pole_grid_rows(h->npm - 2, cfg.gridDim.x);
    cfg.gridDim.y += prows;
    cfg.blockDim = dim3(33, 9);  // (TJ+1) x (TK+1) threads for a 32 x 8 tile
    const bool many = (int64_t)cfg.gridDim.x * cfg.gridDim.y * nz > (int64_t)16 * h->num_sms;
    return cudaLaunchKernelEx(&cfg, many ? k_adv_upwind<32, 8, 6> : k_adv_upwind<32, 8, 4>, h->M, h->FL, x, f0, out,
                              h->bc_flow_n, h->bc_flow_s, cb, rlist, rdt, prows);
  }
  AdvArgs a{x, f0, out, cb, rlist, rdt, 0, 0, h->bc_flow_n, h->bc_flow_s, adv_pole_blocks(h->npm - 2, (int)nz), 0, 0};
  const int n2 = h->npm - 2;
  const bool wide = std::max(h->plane, h->FL.vplane) >= (int64_t)1 << 29;
  a.pgrid = wide ? 2 * a.poles : adv_pole_grid(n2, (int)nz);  // eight such planes do not fit the GPU
  a.share = (n2 + a.poles - 1) / a.poles;
  const int slots = kABlocks * kAWarps * h->num_sms;
  const int hb = a.pgrid == 1 ? adv_halves(h->ntm) : 1;
  a.strips = adv_strips(h->ntm, hb);
  a.cols = adv_cols(n2, a.strips, (int)nz, slots, hb);
  const int nch = (n2 + a.cols - 1) / a.cols;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = (pdl && chained) ? 1 : 0;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cfg.gridDim = dim3((unsigned)(a.pgrid + a.strips * ((nch + hb * kAWarps - 1) / (hb * kAWarps))), nz);
  cfg.blockDim = dim3(32 * kAWarps);
  cfg.dynamicSmemBytes = adv_smem(h->FL.flow2d, hb);
  const AdvKernel kernel = adv_kernel(h->FL.flow2d, cb.mode != 0, wide, a.pgrid == 1, hb);
  const cudaError_t e = smem_limit(h, (const void *)kernel, adv_smem(h->FL.flow2d, hb));
  return e == cudaSuccess ? cudaLaunchKernelEx(&cfg, kernel, h->M, h->FL, h->W, a) : e;
}

static int advection_stage(hipft_gpu *h, const double *x, const double *f0, double *out, AdvCombine cb,
                           bool chained, int n = 0, const int *rlist = nullptr, const double *rdt = nullptr) {
  ProfScope ps(h, HIPFT_K_ADV);
  if (!n) n = h->nr;
  const cudaError_t e = launch_adv_stage(h, h->stream, (unsigned)n, x, f0, out, cb, rlist, rdt, ws_pdl(), chained);
  if (e != cudaSuccess) return fail(h, HIPFT_ECUDA, "advection stage launch: %s", cudaGetErrorString(e));
  h->launches += 1;
  h->cell_updates += (int64_t)h->ntm * (h->npm - 2) * n;
  return HIPFT_OK;
}

extern "C" int hipft_gpu_create(const hipft_grid *g, const hipft_params *prm, hipft_gpu **out) {
  if (!g || !prm || !out || !g->t || !g->p) return HIPFT_EINVAL;
  *out = nullptr;
  if (g->ntm < 4 || g->npm1 < 5 || g->nr < 1) return HIPFT_EINVAL;
  if (prm->advance_diffusion && !prm->diffusion_coef_constants) return HIPFT_EINVAL;
  if (prm->advance_flow && (prm->flow_num_method < 1 || prm->flow_num_method > 4)) return HIPFT_EINVAL;
  if (prm->advance_diffusion && (prm->diffusion_num_method < 1 || prm->diffusion_num_method > 3))
    return HIPFT_EINVAL;
  hipft_gpu *h = new hipft_gpu();
  h->dev = g->device;
  h->P = *prm;
  h->P.diffusion_coef_constants = nullptr;
  h->ntm = g->ntm;
  h->npm1 = g->npm1;
  h->npm = g->npm1 + 1;
  h->nt = g->ntm + 1;
  h->np = g->npm1 + 1;
  h->nr = g->nr;
  h->ldt = round_up(h->ntm, 16);
  h->ldv = round_up(h->nt, 16);
  h->plane = (int64_t)h->ldt * h->npm;
  h->fieldn = (size_t)h->plane * h->nr;
  // the per-realization constants also set validation run 1's decay rate
  // (src/hipft.f90:3156-3159), diffusion or not
  if (prm->diffusion_coef_constants)
    h->Dc.assign(prm->diffusion_coef_constants, prm->diffusion_coef_constants + g->nr);
  int fm = prm->flow_num_method;
  h->adv_time = (fm == 1) ? 1 : (fm == 4 ? 3 : 2);
  h->adv_space = (fm <= 2) ? 1 : 2;
  h->subcycles_state = prm->diffusion_subcycles;
  auto bail = [&](int rc) {
    std::string e = h->err;
    hipft_gpu_destroy(h);
    (void)e;
    return rc;
  };
  cudaError_t ce = cudaSetDevice(h->dev);
  if (ce != cudaSuccess) {
    fail(h, HIPFT_ECUDA, "cudaSetDevice(%d): %s", h->dev, cudaGetErrorString(ce));
    return bail(HIPFT_ECUDA);
  }
  ce = cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking);
  if (ce != cudaSuccess) return bail(HIPFT_ECUDA);
  h->own_stream = true;
  int rc = set_mesh(h, g->t, g->p);
  if (rc) return bail(rc);
  int ntm = h->ntm, npm = h->npm, nt = h->nt, np = h->np, nr = h->nr;

  // 1-D mesh arrays on the device (one allocation, 1-based slices)
  std::vector<const std::vector<double> *> arrs = {&h->dt_i, &h->dth_i, &h->dp_i, &h->dph_i, &h->st_i,
                                                   &h->sth,  &h->dp,    &h->dth,  &h->dph};
  size_t tot = 0;
  for (auto *a : arrs) tot += a->size();
  double *dm = nullptr;
  if ((rc = dsmall(h, &dm, tot))) return bail(rc);
  std::vector<double> packed;
  packed.reserve(tot);
  std::vector<size_t> offs;
  for (auto *a : arrs) {
    offs.push_back(packed.size());
    packed.insert(packed.end(), a->begin(), a->end());
  }
  if ((rc = upload(h, dm, packed))) return bail(rc);
  h->M.ntm = ntm; h->M.npm = npm; h->M.nt = nt; h->M.np = np; h->M.nr = nr; h->M.ldt = h->ldt;
  h->M.plane = h->plane;
  h->M.dt_i = dm + offs[0]; h->M.dth_i = dm + offs[1]; h->M.dp_i = dm + offs[2]; h->M.dph_i = dm + offs[3];
  h->M.st_i = dm + offs[4]; h->M.sth = dm + offs[5]; h->M.dp = dm + offs[6]; h->M.dth = dm + offs[7];
  h->M.dph = dm + offs[8];

  // the field, A u0 and the four of the RKG2 passes
  if ((rc = dfields(h, h->buf, h->nbuf))) return bail(rc);
  h->nkb = (npm - 2 + kKPT3 - 1) / kKPT3;  // partial slots for the smaller phi block
  if ((rc = dsmall(h, &h->d_ringbuf[0], 2 * (size_t)nr))) return bail(rc);
  if ((rc = dsmall(h, &h->d_ringbuf[1], 2 * (size_t)nr))) return bail(rc);
  if ((rc = dsmall(h, &h->d_rpart, 2 * (size_t)nr * h->nkb))) return bail(rc);
  if ((rc = dsmall(h, &h->d_rcount, (size_t)nr))) return bail(rc);
  if ((rc = dsmall(h, &h->d_err, 1))) return bail(rc);
  if (cudaMemsetAsync(h->d_err, 0, sizeof(int), h->stream) != cudaSuccess) return bail(HIPFT_ECUDA);
  if (prm->advance_diffusion && prm->diffusion_num_method >= 2 && !prm->diffusion_coef_grid && poles_by_column(h) &&
      npm - 2 >= kPassColumns && poles_threads(npm - 2) <= kPassThreads && h->plane < (int64_t)1 << 29) {
    const int pt = poles_threads(npm - 2);
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)poles_ranks(npm - 2);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)poles_ranks(npm - 2));
    cfg.blockDim = dim3((unsigned)pt);
    cfg.dynamicSmemBytes = pass_smem(pt);
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const MarchKernel kernel = pass_kernel(true, false);  // all four take two blocks per SM
    if (smem_limit(h, (const void *)kernel, pass_smem(kPassThreads)) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&h->pass_clusters, kernel, &cfg) != cudaSuccess) {
      cudaGetLastError();
      h->pass_clusters = 0;
    }
  }
  if (cudaDeviceGetAttribute(&h->num_sms, cudaDevAttrMultiProcessorCount, h->dev) != cudaSuccess || h->num_sms < 1)
    h->num_sms = 148;
  if (cudaMemsetAsync(h->d_rcount, 0, sizeof(unsigned int) * nr, h->stream) != cudaSuccess) return bail(HIPFT_ECUDA);
  {  // two reduction slots and the maxima of k_ax's blocks
    const dim3 g = ax_grid(h, nr);
    if ((rc = dsmall(h, &h->d_bits, 4 + (size_t)g.x * g.y * g.z))) return bail(rc);
  }
  if (cudaMallocHost((void **)&h->h_pin, sizeof(double) * std::max<size_t>(64, (size_t)nr * kNPart)) !=
      cudaSuccess)
    return bail(fail(h, HIPFT_ENOMEM, "cudaMallocHost failed"));

  // diffusion: D constants, Gershgorin dt (load_diffusion, src/hipft.f90:6655-6844)
  std::vector<double> dfac(nr + 1, 0.0);
  if (prm->advance_diffusion)
    for (int i = 1; i <= nr; ++i)
      dfac[i] = prm->diffusion_coef_grid ? h->Dc[i - 1] : prm->diffusion_coef_factor * h->Dc[i - 1];
  double *d_dfac = nullptr;
  if ((rc = dsmall(h, &d_dfac, nr + 1))) return bail(rc);
  if ((rc = upload(h, d_dfac, dfac))) return bail(rc);
  h->DC.dfac = d_dfac;
  h->DC.factor = prm->diffusion_coef_factor;
  h->DC.grid = prm->diffusion_coef_grid;
  if (prm->advance_diffusion && !prm->diffusion_coef_grid) {
    PairTables &pt = h->ptab;
    pt.LR = round_up(ntm + 4, 2);  // even: the column table behind the rows stays 16-byte aligned
    pt.LC = npm + 2 + 2 * kColPad;
    h->m_strips = std::max(1, (ntm - 2 * kMS + kMOwn - 1) / kMOwn);
    h->m_slots = kMBlocks * kMWarps * h->num_sms;
    if (!poles_by_column(h) &&
        (rc = dalloc(h, &h->d_pscratch, (size_t)nr * poles_any_doubles(npm - 2))))
      return bail(rc);
    double *tab = nullptr;
    const size_t nrow = (size_t)nr * pt.LR * 3, ncol = (size_t)nr * pt.LC * 2;
    if ((rc = dsmall(h, &tab, nrow + ncol))) return bail(rc);
    pt.row = tab;
    pt.col = tab + nrow + 2 * kColPad;
    k_pair_tables<<<2 * h->num_sms, 256, 0, h->stream>>>(h->M, d_dfac, pt.LR, pt.LC, tab, tab + nrow);
    h->launches++;
    if (cudaPeekAtLastError() != cudaSuccess) return bail(fail(h, HIPFT_ECUDA, "k_pair_tables launch failed"));
  }
  h->bc_diff_n = c_pi_i * h->dth_i[2] * h->dth_i[2];
  h->bc_diff_s = c_pi_i * h->dth_i[nt - 1] * h->dth_i[nt - 1];
  h->auto_sc = (prm->diffusion_subcycles == 0);
  if (prm->advance_diffusion) {
    if (cudaMemsetAsync(h->d_bits, 0, sizeof(unsigned long long), h->stream) != cudaSuccess) return bail(HIPFT_ECUDA);
    dim3 blk(32, 8);
    dim3 grd((unsigned)((ntm - 2 + 31) / 32), (unsigned)((npm - 2 + 7) / 8), (unsigned)nr);
    k_gershgorin<<<grd, blk, 0, h->stream>>>(h->M, h->DC, h->d_bits);
    h->launches++;
    if (cudaPeekAtLastError() != cudaSuccess) return bail(fail(h, HIPFT_ECUDA, "k_gershgorin launch failed"));
    if ((rc = sync_read(h, h->d_bits, sizeof(unsigned long long)))) return bail(rc);
    unsigned long long bits;
    std::memcpy(&bits, h->h_pin, 8);
    double max_eig;
    std::memcpy(&max_eig, &bits, 8);
    h->dt_euler = c_safety * (2.0 / max_eig);
  }

  // flows and WENO (load_flows src/hipft.f90:2535-2564, load_weno 6846)
  h->bc_flow_n = 2.0 * h->dth_i[2] * c_pi_i;
  h->bc_flow_s = 2.0 * h->dth_i[nt - 1] * c_pi_i;
  if (prm->advance_flow) {
    std::vector<double> wt[7], wp[7];
    weno_weights(h, wt, wp);
    std::vector<double> pk;
    std::vector<size_t> wo;
    for (int q = 0; q < 7; ++q) { wo.push_back(pk.size()); pk.insert(pk.end(), wt[q].begin(), wt[q].end()); }
    for (int q = 0; q < 7; ++q) { wo.push_back(pk.size()); pk.insert(pk.end(), wp[q].begin(), wp[q].end()); }
    // phi-face rows of the marching advection stage (Weno::ptab): faces
    // 2..npm, face npm with face 2's weights (src/hipft.f90:7882)
    const size_t tab0 = (pk.size() + 1) & ~(size_t)1;  // 16-byte aligned rows
    pk.resize(tab0 + (size_t)(npm - 1) * kPhiTab, 0.0);
    for (int kf = 2; kf <= npm; ++kf) {
      const int kw = (kf >= npm) ? 2 : kf;
      double *row = pk.data() + tab0 + (size_t)(kf - 2) * kPhiTab;
      const double v[10] = {wp[1][kw - 1], wp[1][kw], wp[0][kw - 1], wp[0][kw], wp[4][kw - 1],
                            wp[5][kw - 1], wp[2][kw], wp[3][kw],     wp[6][kw - 1], wp[6][kw]};
      row[12] = 1.0 + v[0];
      row[13] = 1.0 + v[3];
      for (int q = 0; q < 10; ++q) row[q] = v[q];
      row[10] = weno_consts_ok(v[4], v[5], v[6], v[7], v[8], v[9]) ? 1.0 : 0.0;
      row[11] = (kf <= npm - 1) ? h->dp_i[kf] : 0.0;
    }
    double *dw = nullptr;
    if ((rc = dsmall(h, &dw, pk.size()))) return bail(rc);
    if ((rc = upload(h, dw, pk))) return bail(rc);
    h->W.cpt = dw + wo[0]; h->W.mct = dw + wo[1]; h->W.mt = dw + wo[2]; h->W.cptt = dw + wo[3];
    h->W.pt = dw + wo[4]; h->W.mctt = dw + wo[5]; h->W.epst = dw + wo[6];
    h->W.cpp = dw + wo[7]; h->W.mcp = dw + wo[8]; h->W.mp = dw + wo[9]; h->W.cptp = dw + wo[10];
    h->W.pp = dw + wo[11]; h->W.mctp = dw + wo[12]; h->W.epsp = dw + wo[13];
    h->W.ptab = dw + tab0;
    if ((rc = dsmall(h, &h->d_vt1, (size_t)nr * (nt + 1)))) return bail(rc);
    if ((rc = dsmall(h, &h->d_vp1, (size_t)nr * (ntm + 1)))) return bail(rc);
    if ((rc = dsmall(h, &h->d_at1, (size_t)nr * (ntm + 1)))) return bail(rc);
    if ((rc = dsmall(h, &h->d_ap1, (size_t)nr * (ntm + 1)))) return bail(rc);
    h->FL.vt1 = h->d_vt1; h->FL.vp1 = h->d_vp1; h->FL.at1 = h->d_at1; h->FL.ap1 = h->d_ap1;
    h->FL.ldv = h->ldv;
    h->FL.vplane = (int64_t)h->ldv * npm;
    h->FL.upwind = prm->upwind;
    // zero flow until set_flow
    std::vector<double> z1((size_t)nr * (nt + 1), 0.0), z2((size_t)nr * (ntm + 1), 0.0);
    if ((rc = upload(h, h->d_vt1, z1)) || (rc = upload(h, h->d_vp1, z2)) || (rc = upload(h, h->d_at1, z2)) ||
        (rc = upload(h, h->d_ap1, z2)))
      return bail(rc);
  }

  // analysis weights (src/hipft.f90:3230-3257; get_flux 8712-8732)
  {
    std::vector<double> w(6 * (size_t)(std::max(ntm, npm) + 1), 0.0);
    size_t L = (size_t)std::max(ntm, npm) + 1;
    double *da_t = &w[0], *sn_t = &w[L], *cs_t = &w[2 * L], *da_p = &w[3 * L], *cs_p = &w[4 * L], *sn_p = &w[5 * L];
    for (int j = 1; j <= ntm; ++j) {
      double tav, sn, cs, d;
      if (j == 1) {
        tav = 0.5 * (h->t[1] + h->t[2]);
        sn = std::sin(tav); cs = std::cos(tav); d = h->dth[2];
        da_t[j] = 0.25 * sn * d;
      } else if (j == ntm) {
        tav = 0.5 * (h->t[ntm] + h->t[ntm - 1]);
        sn = std::sin(tav); cs = std::cos(tav); d = h->dth[ntm];
        da_t[j] = 0.25 * sn * d;
      } else {
        sn = std::sin(h->t[j]); cs = std::cos(h->t[j]); d = h->dt[j];
        da_t[j] = sn * d;
      }
      sn_t[j] = sn;
      cs_t[j] = cs;
    }
    for (int k = 1; k <= npm - 1; ++k) {
      if (k == 1) da_p[k] = 0.5 * h->dph[1];
      else if (k == npm - 1) da_p[k] = 0.5 * h->dph[npm - 1];
      else da_p[k] = h->dp[k];
      cs_p[k] = std::cos(h->p[k]);
      sn_p[k] = std::sin(h->p[k]);
    }
    h->da_t.assign(da_t, da_t + ntm + 1);
    h->da_p.assign(da_p, da_p + npm);
    if ((rc = dsmall(h, &h->d_anw, w.size()))) return bail(rc);
    if ((rc = upload(h, h->d_anw, w))) return bail(rc);
    std::vector<unsigned char> masks(2 * (size_t)(ntm + 1), 0);
    for (int j = 1; j <= ntm; ++j) {
      masks[j] = (h->t[j] <= prm->pole_flux_lat_limit * c_d2r) ? 1 : 0;
      masks[ntm + 1 + j] = (h->t[j] >= c_pi - prm->pole_flux_lat_limit * c_d2r) ? 1 : 0;
    }
    if ((rc = dsmall(h, &h->d_masks, masks.size()))) return bail(rc);
    if (cudaMemcpyAsync(h->d_masks, masks.data(), masks.size(), cudaMemcpyHostToDevice, h->stream) != cudaSuccess)
      return bail(HIPFT_ECUDA);
    if ((rc = dsmall(h, &h->d_vscale, nr + 1))) return bail(rc);
  }
  if (cudaStreamSynchronize(h->stream) != cudaSuccess) return bail(fail(h, HIPFT_ECUDA, "create: sync failed"));
  *out = h;
  return HIPFT_OK;
}

extern "C" int hipft_gpu_destroy(hipft_gpu *h) {
  if (!h) return HIPFT_OK;
  cudaSetDevice(h->dev);
  if (h->stream) cudaStreamSynchronize(h->stream);
  for (auto &v : h->ev_pending)
    for (auto &pr : v) {
      cudaEventDestroy(pr.first);
      cudaEventDestroy(pr.second);
    }
  for (auto e : h->ev_pool) cudaEventDestroy(e);
  graph_release(h);
  for (auto s : h->g_side)
    if (s) cudaStreamDestroy(s);
  for (void *p : h->allocs) cudaFree(p);
  if (h->h_pin) cudaFreeHost(h->h_pin);
  if (h->own_stream && h->stream) cudaStreamDestroy(h->stream);
  delete h;
  return HIPFT_OK;
}

extern "C" int hipft_gpu_last_error(const hipft_gpu *h, char *buf, size_t len) {
  if (!buf || !len) return HIPFT_EINVAL;
  const char *m = h ? h->err.c_str() : "no handle";
  std::snprintf(buf, len, "%s", m);
  return HIPFT_OK;
}

extern "C" const char *hipft_gpu_version(void) { return "hipft_b200 0.1.0 (sm_100a, fp64)"; }

// ------------------------------------------------------------- field I/O
extern "C" int hipft_gpu_set_field(hipft_gpu *h, const double *f) {
  if (!h || !f) return HIPFT_EINVAL;
  CK(h, cudaSetDevice(h->dev));
  CK(h, cudaMemcpy2DAsync(h->buf[h->cur], (size_t)h->ldt * sizeof(double), f, (size_t)h->ntm * sizeof(double),
                          (size_t)h->ntm * sizeof(double), (size_t)h->npm * h->nr, cudaMemcpyHostToDevice,
                          h->stream));
  h->field_set = true;
  h->dring_valid = false;
  return HIPFT_OK;
}

extern "C" int hipft_gpu_get_field(hipft_gpu *h, double *f) {
  if (!h || !f) return HIPFT_EINVAL;
  CK(h, cudaSetDevice(h->dev));
  CK(h, cudaMemcpy2DAsync(f, (size_t)h->ntm * sizeof(double), h->buf[h->cur], (size_t)h->ldt * sizeof(double),
                          (size_t)h->ntm * sizeof(double), (size_t)h->npm * h->nr, cudaMemcpyDeviceToHost,
                          h->stream));
  CK(h, cudaStreamSynchronize(h->stream));
  return HIPFT_OK;
}

// get_flux of a host (ntm,npm) slab (src/hipft.f90:8706-8738).
static void host_flux(const hipft_gpu *h, const double *map, double &fp, double &fm) {
  fp = 0.0;
  fm = 0.0;
  for (int k = 1; k <= h->npm - 1; ++k)
    for (int j = 1; j <= h->ntm; ++j) {
      double fv = map[(size_t)(k - 1) * h->ntm + (j - 1)] * h->da_t[j] * h->da_p[k];
      if (fv > 0.0) fp = fp + fv; else fm = fm + fv;
    }
}

extern "C" int hipft_gpu_load_initial_map(hipft_gpu *h, const double *map_pt, int flux_balance, double mult_fac) {
  if (!h || !map_pt) return HIPFT_EINVAL;
  int ntm = h->ntm, npm = h->npm, npm1 = h->npm1, nr = h->nr;
  std::vector<double> f((size_t)ntm * npm * nr);
  auto F = [&](int j, int k, int i) -> double & { return f[((size_t)(i - 1) * npm + (k - 1)) * ntm + (j - 1)]; };
  for (int i = 1; i <= nr; ++i)
    for (int k = 1; k <= npm1; ++k)
      for (int j = 1; j <= ntm; ++j) F(j, k, i) = map_pt[((size_t)(i - 1) * ntm + (j - 1)) * npm1 + (k - 1)];
  for (int i = 1; i <= nr; ++i)
    for (int j = 1; j <= ntm; ++j) {
      F(j, 1, i) = 0.5 * (F(j, 1, i) + F(j, npm1, i));
      F(j, npm1, i) = F(j, 1, i);
      F(j, npm1 + 1, i) = F(j, 2, i);
    }
  for (int i = 1; i <= nr; ++i) {
    double fn1 = 0.0, fs1 = 0.0;
    for (int k = 2; k <= npm - 1; ++k) {
      fn1 = fn1 + F(1, k, i) * h->dp[k];
      fs1 = fs1 + F(ntm, k, i) * h->dp[k];
    }
    for (int k = 1; k <= npm; ++k) {
      F(1, k, i) = fn1 * 0.15915494309189535;
      F(ntm, k, i) = fs1 * 0.15915494309189535;
    }
  }
  if (flux_balance)
    for (int i = 1; i <= nr; ++i) {
      double *slab = &f[(size_t)(i - 1) * npm * ntm];
      double fp, fm;
      host_flux(h, slab, fp, fm);
      if (fm + fp == 0.0) continue;
      double ratio = std::sqrt(std::fabs(fp / fm));
      for (size_t q = 0; q < (size_t)npm * ntm; ++q) slab[q] = (slab[q] > 0) ? slab[q] / ratio : slab[q] * ratio;
    }
  for (auto &v : f) v = mult_fac * v;
  return hipft_gpu_set_field(h, f.data());
}

// ------------------------------------------------------------------ flows
extern "C" int hipft_gpu_set_flow(hipft_gpu *h, const hipft_flow_def *def) {
  if (!h || !def) return HIPFT_EINVAL;
  if (!h->P.advance_flow) return fail(h, HIPFT_ESTATE, "set_flow: advance_flow is off for this handle");
  int nr = h->nr;
  auto take = [&](std::vector<double> &v, const double *src, double dflt) {
    v.assign(nr, dflt);
    if (src) std::copy(src, src + nr, v.begin());
  };
  if ((def->flow_dr_model == 1 && (!def->dr_p0 || !def->dr_p2 || !def->dr_p4)) ||
      (def->flow_mf_model == 1 && (!def->mf_p1 || !def->mf_p3 || !def->mf_p5)) ||
      (def->flow_attenuate && !def->flow_attenuate_values))
    return fail(h, HIPFT_EINVAL, "set_flow: missing per-realization coefficients");
  take(h->f_p0, def->dr_p0, 0); take(h->f_p2, def->dr_p2, 0); take(h->f_p4, def->dr_p4, 0);
  take(h->f_p1, def->mf_p1, 0); take(h->f_p3, def->mf_p3, 0); take(h->f_p5, def->mf_p5, 0);
  take(h->f_att, def->flow_attenuate_values, 0);
  h->atten_set = false;
  h->fdef = *def;
  h->have_flow = true;
  h->flow_needs_updating = true;
  // a flow from files, set before or after, stays the base of vt, vp
  h->flow2d = h->have_file_flow || def->flow_attenuate || def->flow_rigid_omega != 0.0;
  return HIPFT_OK;
}

// 1-D analytic parts of vt (theta faces) and vp (phi faces), per
// realization, in the order update_flow adds them (src/hipft.f90:3409-3437).
static void analytic_profiles(const hipft_gpu *h, std::vector<double> &vt1, std::vector<double> &vp1) {
  int nt = h->nt, ntm = h->ntm, nr = h->nr;
  const hipft_flow_def &d = h->fdef;
  vt1.assign((size_t)nr * (nt + 1), 0.0);
  vp1.assign((size_t)nr * (ntm + 1), 0.0);
  for (int i = 1; i <= nr; ++i) {
    double *vt = &vt1[(size_t)(i - 1) * (nt + 1)];
    double *vp = &vp1[(size_t)(i - 1) * (ntm + 1)];
    if (d.flow_mf_model == 1)
      for (int j = 1; j <= nt; ++j) {
        double c = h->cth[j];
        vt[j] = vt[j] - c_m_s_to_rs_hr * h->sth[j] *
                            (h->f_p1[i - 1] * c + h->f_p3[i - 1] * pow3(c) + h->f_p5[i - 1] * pow5(c));
      }
    if (d.flow_dr_model == 1)
      for (int j = 1; j <= ntm; ++j) {
        double c = h->ct[j];
        double c2 = c * c, c4 = c2 * c2;
        vp[j] = vp[j] + c_m_s_to_rs_hr * h->st[j] * (h->f_p0[i - 1] + h->f_p2[i - 1] * c2 + h->f_p4[i - 1] * c4);
      }
    if (d.flow_vp_rigid_omega != 0.0)
      for (int j = 1; j <= ntm; ++j) vp[j] = vp[j] + d.flow_vp_rigid_omega * c_km_s_to_rs_hr * h->st[j];
    if (d.flow_vt_const != 0.0)
      for (int j = 1; j <= nt; ++j) vt[j] = vt[j] + d.flow_vt_const * c_km_s_to_rs_hr;
  }
}

extern "C" int hipft_gpu_set_allreduce(hipft_gpu *h, hipft_allreduce_cb cb, void *user) {
  if (!h) return HIPFT_EINVAL;
  h->red_cb = cb;
  h->red_user = user;
  if (h->P.advance_diffusion) TRY(allreduce(h, HIPFT_RED_MIN, &h->dt_euler));  // src/hipft.f90:5036
  return HIPFT_OK;
}

extern "C" int hipft_gpu_set_flow_from_files(hipft_gpu *h, const double *vt_pt, const double *vp_pt,
                                             int at_load) {
  if (!h || !vt_pt || !vp_pt) return HIPFT_EINVAL;
  if (!h->P.advance_flow) return fail(h, HIPFT_ESTATE, "set_flow_from_files: advance_flow is off for this handle");
  CK(h, cudaSetDevice(h->dev));
  const int nt = h->nt, ntm = h->ntm, npm = h->npm, np = h->np, npm1 = h->npm1;
  std::vector<double> vt((size_t)npm * (nt + 1), 0.0), vp((size_t)np * (ntm + 1), 0.0);
  auto T = [&](int j, int k) -> double & { return vt[(size_t)(k - 1) * (nt + 1) + j]; };
  auto P = [&](int j, int k) -> double & { return vp[(size_t)(k - 1) * (ntm + 1) + j]; };
  for (int k = 1; k <= npm1; ++k)
    for (int j = 1; j <= nt; ++j) T(j, k) = c_m_s_to_rs_hr * vt_pt[(size_t)(j - 1) * npm1 + (k - 1)];
  for (int k = 1; k <= np; ++k)
    for (int j = 1; j <= ntm; ++j) P(j, k) = c_m_s_to_rs_hr * vp_pt[(size_t)(j - 1) * np + (k - 1)];
  if (at_load) {
    for (int j = 1; j <= nt; ++j) T(j, npm) = T(j, 2);  // src/hipft.f90:3789
  } else {                                             // set_periodic_bc_3d, src/hipft.f90:3604, 3634
    for (int j = 1; j <= nt; ++j) { T(j, 1) = T(j, npm - 1); T(j, npm) = T(j, 2); }
    for (int j = 1; j <= ntm; ++j) { P(j, 1) = P(j, np - 1); P(j, np) = P(j, 2); }
  }
  TRY(once(h, &h->d_vtf, vt.size()));
  TRY(once(h, &h->d_vpf, vp.size()));
  TRY(upload(h, h->d_vtf, vt));
  TRY(upload(h, h->d_vpf, vp));
  CK(h, cudaStreamSynchronize(h->stream));  // the host staging vectors go out of scope
  h->have_file_flow = true;
  h->flow2d = true;
  h->flow_needs_updating = true;
  return HIPFT_OK;
}

extern "C" int hipft_gpu_update_flow(hipft_gpu *h, int *updated) {
  if (!h) return HIPFT_EINVAL;
  if (updated) *updated = 0;
  if (!(h->have_flow || h->have_file_flow) || !h->flow_needs_updating) return HIPFT_OK;
  CK(h, cudaSetDevice(h->dev));
  int nt = h->nt, ntm = h->ntm, nr = h->nr, npm = h->npm;
  bool again = false;  // the flow changes before every step
  std::vector<double> vt1, vp1;
  analytic_profiles(h, vt1, vp1);
  TRY(upload(h, h->d_vt1, vt1));
  TRY(upload(h, h->d_vp1, vp1));
  if (!h->flow2d) {
    // set_lf_alpha on theta-only profiles (src/hipft.f90:6968-7037)
    std::vector<double> at1((size_t)nr * (ntm + 1), 0.0), ap1((size_t)nr * (ntm + 1), 0.0);
    for (int i = 1; i <= nr; ++i) {
      const double *vt = &vt1[(size_t)(i - 1) * (nt + 1)];
      const double *vp = &vp1[(size_t)(i - 1) * (ntm + 1)];
      double *at = &at1[(size_t)(i - 1) * (ntm + 1)];
      double *ap = &ap1[(size_t)(i - 1) * (ntm + 1)];
      auto A = [&](int j) { return std::fabs(vt[j]); };
      for (int j = 3; j <= nt - 3; ++j)
        at[j] = std::max(std::max(std::max(std::max(std::max(A(j - 2), A(j - 1)), A(j)), A(j + 1)), A(j + 2)), A(j + 3));
      at[1] = std::max(std::max(std::max(A(1), A(2)), A(3)), A(4));
      at[2] = std::max(std::max(std::max(std::max(A(1), A(2)), A(3)), A(4)), A(5));
      { int j = nt - 2; at[j] = std::max(std::max(std::max(std::max(A(j - 2), A(j - 1)), A(j)), A(j + 1)), A(j + 2)); }
      { int j = nt - 1; at[j] = std::max(std::max(std::max(A(j - 2), A(j - 1)), A(j)), A(j + 1)); }
      for (int j = 2; j <= ntm - 1; ++j) ap[j] = std::fabs(vp[j]);
    }
    TRY(upload(h, h->d_at1, at1));
    TRY(upload(h, h->d_ap1, ap1));
    h->FL.flow2d = 0;
  } else {
    if (!h->d_atten) {  // the last of them
      size_t n2 = (size_t)h->ldv * npm * nr;
      TRY(once(h, &h->d_vt, n2));
      TRY(once(h, &h->d_vp, n2));
      TRY(once(h, &h->d_at, n2));
      TRY(once(h, &h->d_ap, n2));
      CK(h, cudaMemsetAsync(h->d_at, 0, n2 * sizeof(double), h->stream));
      CK(h, cudaMemsetAsync(h->d_ap, 0, n2 * sizeof(double), h->stream));
      // cos(p), sin(p), cos(ph), theta metrics (1-based), attenuation factors
      size_t L = (size_t)std::max(npm, nt) + 2;
      std::vector<double> trig(7 * L, 0.0);
      for (int k = 1; k <= npm; ++k) {
        trig[k] = std::cos(h->p[k]);
        trig[L + k] = std::sin(h->p[k]);
        trig[2 * L + k] = std::cos(h->ph[k]);
      }
      for (int j = 1; j <= nt; ++j) { trig[3 * L + j] = h->cth[j]; trig[4 * L + j] = h->sth[j]; }
      for (int j = 1; j <= ntm; ++j) { trig[5 * L + j] = h->ct[j]; trig[6 * L + j] = h->st[j]; }
      TRY(once(h, &h->d_trig, trig.size()));
      TRY(upload(h, h->d_trig, trig));
      TRY(dsmall(h, &h->d_atten, nr + 1));
    }
    if (h->have_flow && !h->atten_set) {
      std::vector<double> att(nr + 1, 0.0);
      for (int i = 1; i <= nr; ++i)
        att[i] = (h->f_att[i - 1] > 0.0) ? 1.0 / h->f_att[i - 1] : DBL_MAX;
      TRY(upload(h, h->d_atten, att));
      h->atten_set = true;
    }
    if (h->fdef.flow_attenuate && !h->field_set) return fail(h, HIPFT_ESTATE, "update_flow: attenuation needs the field");
    size_t L = (size_t)std::max(npm, nt) + 2;
    Flow2DBuild b{};
    b.vt1 = h->d_vt1; b.vp1 = h->d_vp1;
    b.cosp = h->d_trig; b.sinp = h->d_trig + L; b.cosph = h->d_trig + 2 * L;
    b.cth = h->d_trig + 3 * L; b.sth = h->d_trig + 4 * L; b.ct = h->d_trig + 5 * L; b.st = h->d_trig + 6 * L;
    b.vrigid = h->fdef.flow_rigid_omega * c_km_s_to_rs_hr;
    b.attenuate = h->fdef.flow_attenuate;
    b.atten_i = h->d_atten;
    if (h->have_file_flow) {
      // the analytic terms one by one, as update_flow adds them over the
      // file flow (src/hipft.f90:3416-3437, 7219-7285)
      const hipft_flow_def &d = h->fdef;
      const size_t nT = (size_t)nr * (nt + 1), nP = (size_t)nr * (ntm + 1);
      std::vector<double> terms(nT + nP + (size_t)(ntm + 1), 0.0);
      double *tmf = terms.data(), *vdr = tmf + nT, *vrg = vdr + nP;
      for (int i = 1; i <= nr; ++i) {
        for (int j = 1; j <= nt; ++j) {
          double c = h->cth[j];
          tmf[(size_t)(i - 1) * (nt + 1) + j] =
              c_m_s_to_rs_hr * h->sth[j] * (h->f_p1[i - 1] * c + h->f_p3[i - 1] * pow3(c) + h->f_p5[i - 1] * pow5(c));
        }
        for (int j = 1; j <= ntm; ++j) {
          double c = h->ct[j];
          double c2 = c * c, c4 = c2 * c2;
          vdr[(size_t)(i - 1) * (ntm + 1) + j] =
              c_m_s_to_rs_hr * h->st[j] * (h->f_p0[i - 1] + h->f_p2[i - 1] * c2 + h->f_p4[i - 1] * c4);
        }
      }
      for (int j = 1; j <= ntm; ++j) vrg[j] = d.flow_vp_rigid_omega * c_km_s_to_rs_hr * h->st[j];
      if (!h->d_fterms) TRY(dalloc(h, &h->d_fterms, terms.size()));
      TRY(upload(h, h->d_fterms, terms));
      b.vtf = h->d_vtf;
      b.vpf = h->d_vpf;
      b.tmf = (d.flow_mf_model == 1) ? h->d_fterms : nullptr;
      b.vdr = (d.flow_dr_model == 1) ? h->d_fterms + nT : nullptr;
      b.vrg = (d.flow_vp_rigid_omega != 0.0) ? h->d_fterms + nT + nP : nullptr;
      b.vtc = (d.flow_vt_const != 0.0) ? d.flow_vt_const * c_km_s_to_rs_hr : 0.0;
    }
    dim3 blk(32, 8), grd((unsigned)((nt + 31) / 32), (unsigned)((npm + 7) / 8), (unsigned)nr);
    k_flow_build<<<grd, blk, 0, h->stream>>>(h->M, b, h->ldv, h->buf[h->cur], h->d_vt, h->d_vp);
    LAUNCHED(h);
    again = h->have_file_flow;  // src/hipft.f90:3423
    if (h->fdef.flow_attenuate) {
      k_seam<<<dim3((unsigned)((nt + 127) / 128), (unsigned)nr), 128, 0, h->stream>>>(h->M, nt, h->ldv, h->d_vt);
      LAUNCHED(h);
      k_seam<<<dim3((unsigned)((ntm + 127) / 128), (unsigned)nr), 128, 0, h->stream>>>(h->M, ntm, h->ldv, h->d_vp);
      LAUNCHED(h);
      again = true;  // Br changes every step (src/hipft.f90:3514)
    }
    if (h->adv_space == 2) {
      dim3 g2((unsigned)((ntm + 31) / 32), (unsigned)((npm + 7) / 8), (unsigned)nr);
      k_lf_alpha<<<g2, blk, 0, h->stream>>>(h->M, h->ldv, h->d_vt, h->d_vp, h->d_at, h->d_ap);
      LAUNCHED(h);
    }
    h->FL.vt = h->d_vt; h->FL.vp = h->d_vp; h->FL.at = h->d_at; h->FL.ap = h->d_ap;
    h->FL.flow2d = 1;
  }
  // only now: a call that failed leaves the flow to be built
  h->flow_needs_updating = again;
  h->r_dtmax_valid = false;
  if (updated) *updated = 1;
  return HIPFT_OK;
}

extern "C" int hipft_gpu_flow_dtmax(hipft_gpu *h, double *dtmax) {
  if (!h || !dtmax) return HIPFT_EINVAL;
  if (!h->P.advance_flow) return fail(h, HIPFT_ESTATE, "flow_dtmax: advance_flow is off");
  CK(h, cudaSetDevice(h->dev));
  unsigned long long init = 0x7fefffffffffffffULL;  // DBL_MAX bits
  CK(h, cudaMemcpyAsync(h->d_bits + 1, &init, 8, cudaMemcpyHostToDevice, h->stream));
  dim3 blk(32, 8), grd((unsigned)((h->ntm - 2 + 31) / 32),
                       (unsigned)((h->npm - 2 + 8 * kAxCols - 1) / (8 * kAxCols)), (unsigned)h->nr);
  k_flow_dtmax<<<grd, blk, 0, h->stream>>>(h->M, h->FL, h->d_bits + 1);
  LAUNCHED(h);
  TRY(sync_read(h, h->d_bits + 1, 8));
  double d;
  std::memcpy(&d, h->h_pin, 8);
  d = c_safety * d;
  if (h->P.strang_splitting) d = 2.0 * d;
  if (h->adv_time == 3) d = 2.0 * d;
  TRY(allreduce(h, HIPFT_RED_MIN, &d));  // src/hipft.f90:7345
  *dtmax = d;
  return HIPFT_OK;
}

// ------------------------------------------------------------- advection
static int ragged_advection_step(hipft_gpu *h, double dt);

static int plain_advection_step(hipft_gpu *h, double dt) {
  h->dring_valid = false;
  double *f = h->buf[h->cur];
  int ia = scratch(h, 0), ib = scratch(h, 1);
  double *A = h->buf[ia], *B = h->buf[ib];
  if (h->adv_time == 1) {  // FE (src/hipft.f90:7440-7444)
    TRY(advection_stage(h, f, nullptr, A, AdvCombine{0, 0.0, 0.0, dt}, false));
    h->cur = ia;
  } else if (h->adv_time == 2) {  // SSPRK(3,3) (7486-7505)
    TRY(advection_stage(h, f, nullptr, A, AdvCombine{0, 0.0, 0.0, dt}, false));
    TRY(advection_stage(h, A, f, B, AdvCombine{1, c_three_quarter, c_quarter, c_quarter * dt}, true));
    TRY(advection_stage(h, B, f, f, AdvCombine{1, c_third, c_two_third, c_two_third * dt}, true));
  } else {  // SSPRK(4,3) (7552-7574)
    TRY(advection_stage(h, f, nullptr, A, AdvCombine{0, 0.0, 0.0, 0.5 * dt}, false));
    TRY(advection_stage(h, A, nullptr, B, AdvCombine{0, 0.0, 0.0, 0.5 * dt}, true));
    TRY(advection_stage(h, B, f, A, AdvCombine{1, c_two_third, c_third, c_sixth * dt}, true));
    TRY(advection_stage(h, A, nullptr, f, AdvCombine{0, 0.0, 0.0, 0.5 * dt}, true));
  }
  return HIPFT_OK;
}

extern "C" int hipft_gpu_advection_step(hipft_gpu *h, double dt) {
  if (!h) return HIPFT_EINVAL;
  if (!h->field_set) return fail(h, HIPFT_ESTATE, "advection_step before set_field");
  if (!h->P.advance_flow) return fail(h, HIPFT_ESTATE, "advection_step: advance_flow is off");
  CK(h, cudaSetDevice(h->dev));
  if (h->ragged) return ragged_advection_step(h, dt);
  return plain_advection_step(h, dt);
}

// ------------------------------------------------------------- diffusion
// Stage count and coefficients of one RKL2 (method 2) or RKG2 (method 3)
// super-step, load_sts_rkl2 / load_sts_rkg2 (src/hipft.f90:5244-5475).
struct StsTable {
  int64_t s = 0;
  std::vector<double> uj, vj, ubj, gj, b;
};
static void sts_coefs(int method, double dtl, double dt_euler, StsTable &T) {
  const int64_t s = sts_count(method, dtl, dt_euler);
  T.s = s;
  T.b.assign(s + 1, 0); T.uj.assign(s + 1, 0); T.vj.assign(s + 1, 0); T.ubj.assign(s + 1, 0); T.gj.assign(s + 1, 0);
  for (int64_t j = 1; j <= s; ++j) {
    T.b[j] = sts_b(method, j);
    sts_stage(method, s, j, T.uj[j], T.vj[j], T.ubj[j], T.gj[j]);
  }
}

static void load_sts(hipft_gpu *h, double dtl) {
  StsTable T;
  sts_coefs(h->P.diffusion_num_method, dtl, h->dt_euler, T);
  h->sts_s = T.s;
  h->sts_b = std::move(T.b);
  h->sts_uj = std::move(T.uj);
  h->sts_vj = std::move(T.vj);
  h->sts_ubj = std::move(T.ubj);
  h->sts_gj = std::move(T.gj);
}

// diffusion_step_sts_cd (src/hipft.f90:5163-5242).  have_lap: scratch buffer 0
// holds A u0 (not with a grid-dependent D).
static int sts_super_step(hipft_gpu *h, double dtl, bool have_lap) {
  load_sts(h, dtl);
  const int u0 = h->cur, idty = scratch(h, 0);
  const int64_t cells = (int64_t)h->ntm * (h->npm - 2) * h->nr;
  h->rkg2_stages += h->sts_s - 1;
  h->rkg2_cell_stages += cells * (h->sts_s - 1);
  h->cell_updates += cells * h->sts_s;
  if (!h->DC.grid) {
    if (!have_lap) TRY(apply_lap(h, nullptr, nullptr, h->nr, 0));
    TRY(scale_dty0(h, h->buf[idty], h->buf[idty], dtl));
    const int R[4] = {scratch(h, 1), scratch(h, 2), scratch(h, 3), scratch(h, 4)};
    MarchArgs a = march_args(h, h->buf[u0], h->buf[idty]);
    const int64_t np = sts_passes(h->sts_s);
    for (int64_t p = 0; p < np; ++p) {
      const int in = (p & 1) ? 0 : 2, out = 2 - in;
      a.x2 = h->buf[R[in]];
      a.x1 = h->buf[R[in + 1]];
      a.o[2] = h->buf[R[out]];
      a.o[3] = h->buf[R[out + 1]];
      a.first = p == 0;
      for (int q = 0; q < kMS; ++q) a.c[q] = sts_slot(h->P.diffusion_num_method, h->sts_s, kMS * p + q, dtl);
      TRY(sts_pass(h, a, p > 0));
      h->cur = R[out + 1];
    }
    h->dring_valid = false;
    return seam(h, h->buf[h->cur]);
  }
  const int ia = scratch(h, 1), ib = scratch(h, 2);
  TRY(diffusion_stage<MODE_STS1>(h, h->buf[u0], nullptr, nullptr, nullptr, h->buf[ia], h->buf[idty],
                                 StageCoef{dtl, h->sts_ubj[1], 0, 0, 0}, false));
  int ykm1 = ia, ykm2 = u0;
  for (int64_t k = 2; k <= h->sts_s; ++k) {
    const int out = (ykm2 == u0) ? ib : ykm2;
    const double uj = h->sts_uj[k], vj = h->sts_vj[k];
    TRY(diffusion_stage<MODE_STSK>(h, h->buf[ykm1], h->buf[ykm2], h->buf[u0], h->buf[idty], h->buf[out], nullptr,
                                   StageCoef{uj, vj, 1.0 - uj - vj, h->sts_ubj[k] * dtl, h->sts_gj[k]}, true));
    ykm2 = ykm1;
    ykm1 = out;
  }
  h->cur = ykm1;
  h->dring_valid = false;
  return HIPFT_OK;
}

// diffusion_step_fe_cd (src/hipft.f90:7352-7407).
static int euler_steps(hipft_gpu *h, double dtl) {
  int64_t n = (int64_t)std::ceil(dtl / h->dt_euler);
  h->n_euler = n;
  double dte = dtl / (double)n;
  for (int64_t c = 0; c < n; ++c) {
    int o = scratch(h, 0);
    if (!h->DC.grid) {
      const double *r0;
      TRY(current_dring(h, &r0));
      TRY(euler_step(h, h->buf[h->cur], h->buf[o], dte));
      h->cur = o;
      h->dring_valid = true;
    } else {
      TRY(diffusion_stage<MODE_EULER>(h, h->buf[h->cur], nullptr, nullptr, nullptr, h->buf[o], nullptr,
                                      StageCoef{dte, 0, 0, 0, 0}, c > 0));
      h->cur = o;
      h->dring_valid = false;
    }
  }
  h->cell_updates += (int64_t)h->ntm * (h->npm - 2) * h->nr * n;
  return HIPFT_OK;
}

// get_dtime_diffusion_ptl (src/hipft.f90:5042-5161).
// Reads and clears the flag that kernels set when a bounded wait gave up;
// HIPFT_ETIMEOUT if it was set (the context stays usable).
static int check_wait_flag(hipft_gpu *h, const char *what) {
  int ev = 0;
  CK(h, cudaMemcpyAsync(&ev, h->d_err, sizeof(int), cudaMemcpyDeviceToHost, h->stream));
  CK(h, cudaStreamSynchronize(h->stream));
  if (!ev) return HIPFT_OK;
  CK(h, cudaMemsetAsync(h->d_err, 0, sizeof(int), h->stream));
  CK(h, cudaMemsetAsync(h->d_rcount, 0, sizeof(unsigned int) * h->nr, h->stream));
  return fail(h, HIPFT_ETIMEOUT, "%s", what);
}

// Both results come back in one read, unless the maximum over the processes of
// a job is needed in between.
static int ptl_dt(hipft_gpu *h, double *dtl) {
  double dtime_in = *dtl;
  const unsigned long long init[2] = {0ULL, 0x7fefffffffffffffULL};
  CK(h, cudaMemcpyAsync(h->d_bits, init, 16, cudaMemcpyHostToDevice, h->stream));
  TRY(apply_lap(h, h->d_bits, nullptr, h->nr, 0));
  double axabsmax, d = DBL_MAX, ptl;
  if (h->red_cb) {  // src/hipft.f90:5103: the PTL cells are those at the global maximum
    TRY(sync_read(h, h->d_bits, 8));
    std::memcpy(&axabsmax, h->h_pin, 8);
    TRY(allreduce(h, HIPFT_RED_MAX, &axabsmax));
    if (!(axabsmax > 0.0)) {
      *dtl = d;
      return HIPFT_OK;
    }
    CK(h, cudaMemcpyAsync(h->d_bits, &axabsmax, 8, cudaMemcpyHostToDevice, h->stream));
    CK(h, cudaStreamSynchronize(h->stream));
  }
  TRY(ptl_cells(h, h->d_bits, h->d_bits + 1, nullptr, h->nr, 0));
  TRY(sync_read(h, h->d_bits, 16));
  std::memcpy(&axabsmax, h->h_pin, 8);
  std::memcpy(&ptl, h->h_pin + 1, 8);
  if (axabsmax > 0.0) {
    d = ptl;
    TRY(allreduce(h, HIPFT_RED_MIN, &d));  // src/hipft.f90:5141
    d = 0.95 * d;
    if (d < dtime_in) d = dtime_in;
  }
  *dtl = d;
  return HIPFT_OK;
}

// ================================================================ ragged
// Ragged batches (no counterpart in the reference, which keeps one dt, one
// Euler limit, one stage count and one PTL subcycle sequence for all
// realizations through global MIN/MAX reductions, src/hipft.f90:5036, 5103,
// 5141, 7345).  In a ragged batch every realization gets the schedule it would
// have if it were run alone: its own Gershgorin limit, its own PTL subcycles
// and RKG2/RKL2 stage counts, and, when the step is longer than its own CFL
// limit, its own number of advection substeps.  Launches still cover many
// realizations at once: a launch walks a list of realizations sorted by the
// work they still need, and the realizations that are done drop off its end.

// per-realization Euler limits, get_dtime_diffusion_euler (src/hipft.f90:
// 5019-5025) of each realization alone
static int ragged_gershgorin(hipft_gpu *h) {
  const int nr = h->nr;
  CK(h, cudaMemsetAsync(h->d_rbits, 0, sizeof(unsigned long long) * nr, h->stream));
  dim3 blk(32, 8);
  dim3 grd((unsigned)((h->ntm - 2 + 31) / 32), (unsigned)((h->npm - 2 + 7) / 8), (unsigned)nr);
  k_gershgorin<<<grd, blk, 0, h->stream>>>(h->M, h->DC, h->d_rbits, 1);
  LAUNCHED(h);
  std::vector<unsigned long long> bits(nr);
  CK(h, cudaMemcpyAsync(bits.data(), h->d_rbits, sizeof(unsigned long long) * nr, cudaMemcpyDeviceToHost,
                        h->stream));
  CK(h, cudaStreamSynchronize(h->stream));
  h->r_dt_euler.assign(nr, 0.0);
  for (int i = 0; i < nr; ++i) {
    double max_eig;
    std::memcpy(&max_eig, &bits[i], 8);
    h->r_dt_euler[i] = c_safety * (2.0 / max_eig);
  }
  return HIPFT_OK;
}

// per-realization CFL limits, get_flow_dtmax (src/hipft.f90:7287-7350) of each
// realization alone
static int ragged_dtmax(hipft_gpu *h) {
  if (h->r_dtmax_valid) return HIPFT_OK;
  const int nr = h->nr;
  std::vector<unsigned long long> bits(nr, 0x7fefffffffffffffULL);
  CK(h, cudaMemcpyAsync(h->d_rbits, bits.data(), sizeof(unsigned long long) * nr, cudaMemcpyHostToDevice,
                        h->stream));
  dim3 blk(32, 8), grd((unsigned)((h->ntm - 2 + 31) / 32),
                       (unsigned)((h->npm - 2 + 8 * kAxCols - 1) / (8 * kAxCols)), (unsigned)nr);
  k_flow_dtmax<<<grd, blk, 0, h->stream>>>(h->M, h->FL, h->d_rbits, 1);
  LAUNCHED(h);
  CK(h, cudaMemcpyAsync(bits.data(), h->d_rbits, sizeof(unsigned long long) * nr, cudaMemcpyDeviceToHost,
                        h->stream));
  CK(h, cudaStreamSynchronize(h->stream));
  h->r_dtmax.assign(nr, 0.0);
  for (int i = 0; i < nr; ++i) {
    double d;
    std::memcpy(&d, &bits[i], 8);
    d = c_safety * d;
    if (h->P.strang_splitting) d = 2.0 * d;
    if (h->adv_time == 3) d = 2.0 * d;
    h->r_dtmax[i] = d;
  }
  h->r_dtmax_valid = true;
  return HIPFT_OK;
}

// realizations `act` ordered by decreasing work (ties by index), uploaded
static int upload_list(hipft_gpu *h, int *dlist, std::vector<int> &act, const std::vector<int64_t> &work) {
  std::stable_sort(act.begin(), act.end(), [&](int a, int b) { return work[a] > work[b]; });
  CK(h, cudaMemcpyAsync(dlist, act.data(), sizeof(int) * act.size(), cudaMemcpyHostToDevice, h->stream));
  return HIPFT_OK;
}

// PTL time steps (src/hipft.f90:5042-5161) of the realizations in `act`,
// each from its own max |Af| and its own argmax cells; dtl[i] is the
// realization's previous subcycle (the floor), replaced by the new one.
static int ragged_ptl(hipft_gpu *h, std::vector<int> act, std::vector<double> &dtl) {
  const int nr = h->nr, na = (int)act.size();
  std::vector<int64_t> none(nr, 0);
  TRY(upload_list(h, h->d_rlist_dif, act, none));
  std::vector<unsigned long long> init(2 * (size_t)nr, 0ULL);
  for (int i = 0; i < nr; ++i) init[nr + i] = 0x7fefffffffffffffULL;
  CK(h, cudaMemcpyAsync(h->d_rbits, init.data(), sizeof(unsigned long long) * 2 * nr, cudaMemcpyHostToDevice,
                        h->stream));
  TRY(apply_lap(h, h->d_rbits, h->d_rlist_dif, na, 1));
  TRY(ptl_cells(h, h->d_rbits, h->d_rbits + nr, h->d_rlist_dif, na, 1));
  std::vector<unsigned long long> bits(2 * (size_t)nr);
  CK(h, cudaMemcpyAsync(bits.data(), h->d_rbits, sizeof(unsigned long long) * 2 * nr, cudaMemcpyDeviceToHost,
                        h->stream));
  CK(h, cudaStreamSynchronize(h->stream));
  for (int i : act) {
    double axabsmax, ptl;
    std::memcpy(&axabsmax, &bits[i], 8);
    std::memcpy(&ptl, &bits[nr + i], 8);
    double d = DBL_MAX;
    if (axabsmax > 0.0) {
      d = 0.95 * ptl;
      if (d < dtl[i]) d = dtl[i];
    }
    dtl[i] = d;
  }
  return HIPFT_OK;
}

// One RKG2/RKL2 super-step of every realization in `act`, realization i over
// dtl[i] with its own stage count s_i (src/hipft.f90:5163-5242 per
// realization).  Pass p covers the realizations with more than p passes;
// afterwards every realization's field is gathered into one buffer, which
// becomes the current field.  Scratch buffer 0 holds A u0 of the realizations.
static int ragged_super_step(hipft_gpu *h, std::vector<int> act, const std::vector<double> &dtl) {
  const int nr = h->nr, method = h->P.diffusion_num_method;
  std::vector<int64_t> s(nr, 0);
  int64_t smax = 0;
  for (int i : act) {
    s[i] = sts_count(method, dtl[i], h->r_dt_euler[i]);
    h->r_s[i] = s[i];
    smax = std::max(smax, s[i]);
  }
  TRY(upload_list(h, h->d_rlist_dif, act, s));
  const int na = (int)act.size();
  const int64_t np = sts_passes(smax);
  if ((size_t)np > h->rcoef_passes) {
    if (h->d_rcoef) {
      CK(h, cudaStreamSynchronize(h->stream));
      cudaFree(h->d_rcoef);
      h->allocs.erase(std::remove(h->allocs.begin(), h->allocs.end(), (void *)h->d_rcoef), h->allocs.end());
      h->d_rcoef = nullptr;
      h->rcoef_passes = 0;
    }
    const size_t cap = (size_t)np + 32;
    TRY(dalloc(h, &h->d_rcoef, cap * nr * kMS));
    h->rcoef_passes = cap;
  }
  std::vector<StageCoef> pc((size_t)np * nr * kMS, StageCoef{});
  for (int i : act)
    for (int64_t q = 0; q < kMS * sts_passes(s[i]); ++q)
      pc[((size_t)(q / kMS) * nr + i) * kMS + q % kMS] = sts_slot(method, s[i], q, dtl[i]);
  CK(h, cudaMemcpyAsync(h->d_rcoef, pc.data(), sizeof(StageCoef) * pc.size(), cudaMemcpyHostToDevice, h->stream));
  CK(h, cudaMemcpyAsync(h->d_rlen, dtl.data(), sizeof(double) * nr, cudaMemcpyHostToDevice, h->stream));

  const int u0 = h->cur, idty = scratch(h, 0);
  const int R[4] = {scratch(h, 1), scratch(h, 2), scratch(h, 3), scratch(h, 4)};
  TRY(scale_dty0(h, h->buf[idty], h->buf[idty], 0.0, h->d_rlist_dif, na, h->d_rlen));
  std::vector<int> fin(nr, u0);  // buffer holding each realization's result
  const int64_t cells = (int64_t)h->ntm * (h->npm - 2);
  MarchArgs a = march_args(h, h->buf[u0], h->buf[idty]);
  a.rlist = h->d_rlist_dif;
  int dst = u0;
  for (int64_t p = 0; p < np; ++p) {
    int n = 0;  // realizations with pass p
    while (n < na && sts_passes(s[act[n]]) > p) ++n;
    const int in = (p & 1) ? 0 : 2, out = 2 - in;
    a.x2 = h->buf[R[in]];
    a.x1 = h->buf[R[in + 1]];
    a.o[2] = h->buf[R[out]];
    a.o[3] = h->buf[R[out + 1]];
    a.first = p == 0;
    a.nreal = n;
    a.rc = h->d_rcoef + (size_t)p * nr * kMS;
    TRY(sts_pass(h, a, p > 0));
    h->rkg2_stages += kMS;
    dst = R[out + 1];
    for (int e = 0; e < n; ++e)
      if (sts_passes(s[act[e]]) == p + 1) fin[act[e]] = dst;
  }
  // gather: realizations that finished earlier, and those not in this
  // super-step at all (still in u0), into the last pass's output
  const size_t pbytes = (size_t)h->plane * sizeof(double);
  for (int i = 0; i < nr; ++i)
    if (fin[i] != dst)
      CK(h, cudaMemcpyAsync(h->buf[dst] + (size_t)i * h->plane, h->buf[fin[i]] + (size_t)i * h->plane, pbytes,
                            cudaMemcpyDeviceToDevice, h->stream));
  TRY(seam(h, h->buf[dst]));
  h->cur = dst;
  h->dring_valid = false;
  int64_t tot = 0;
  for (int i : act) tot += s[i];
  h->cell_updates += cells * tot;
  h->rkg2_cell_stages += cells * (tot - na);
  return HIPFT_OK;
}

// diffusion_step (src/hipft.f90:4551-4695) with every realization's own
// subcycle sequence (PTL) and stage counts.
static int ragged_diffusion_step(hipft_gpu *h, double dtl, hipft_diffusion_info *info) {
  const int nr = h->nr, max_sc = 60;
  const int64_t stages0 = h->cell_updates;
  std::vector<double> ts(nr, 0.0), d(nr, h->auto_sc ? 0.0 : dtl / (double)h->P.diffusion_subcycles);
  std::vector<int> act(nr);
  for (int i = 0; i < nr; ++i) act[i] = i;
  h->r_s.assign(nr, 0);
  h->r_cycles.assign(nr, 0);
  int cyc = 1;
  int64_t smax = 0;
  while (!act.empty()) {
    if (h->auto_sc) TRY(ragged_ptl(h, act, d));
    else TRY(apply_lap(h, nullptr, nullptr, h->nr, 0));
    std::vector<int> done;
    for (int i : act) {
      bool fin = false;
      if (h->auto_sc && ts[i] + d[i] >= dtl) {
        d[i] = dtl - ts[i];
        fin = true;
      }
      if (h->auto_sc && cyc == max_sc - 1) {
        d[i] = dtl - ts[i];
        fin = true;
      }
      if (!h->auto_sc && cyc == h->P.diffusion_subcycles) fin = true;
      if (fin) done.push_back(i);
    }
    TRY(ragged_super_step(h, act, d));
    for (int i : act) {
      ts[i] = ts[i] + d[i];
      h->r_cycles[i] = cyc;
      smax = std::max(smax, h->r_s[i]);
    }
    std::vector<int> next;
    for (int i : act)
      if (std::find(done.begin(), done.end(), i) == done.end()) next.push_back(i);
    act.swap(next);
    cyc = cyc + 1;
  }
  TRY(check_wait_flag(h, "diffusion_step: a bounded wait for ring sums gave up"));
  h->sts_s = smax;
  h->subcycles_state = cyc - 1;
  if (info) {
    info->dtime_diffusion_euler = *std::min_element(h->r_dt_euler.begin(), h->r_dt_euler.end());
    info->sts_s = smax;
    info->subcycles = cyc - 1;
    const int64_t cells = (int64_t)h->ntm * (h->npm - 2) * h->nr;
    info->total_stages = cells ? (h->cell_updates - stages0) / cells : 0;
  }
  return HIPFT_OK;
}

// advection_step (src/hipft.f90:4509-4549) with every realization's own
// substep count: realization i takes n_i = ceil(dt / its own CFL limit)
// substeps of dt / n_i (one substep when dt is within its limit, which is
// the plain step).
static int plain_advection_step(hipft_gpu *h, double dt);

static int ragged_advection_step(hipft_gpu *h, double dt) {
  const int nr = h->nr;
  TRY(ragged_dtmax(h));
  // the CFL limit bounds a whole split step: a Strang half step may use half of it
  const double scale = h->P.strang_splitting ? 2.0 : 1.0;
  std::vector<int64_t> n(nr, 1);
  int64_t nmax = 1;
  for (int i = 0; i < nr; ++i) {
    const double r = dt * scale / h->r_dtmax[i];
    n[i] = (r > 1.0) ? (int64_t)std::ceil(r) : 1;
    nmax = std::max(nmax, n[i]);
  }
  h->r_substeps = n;
  if (nmax == 1) return plain_advection_step(h, dt);
  std::vector<int> act(nr);
  for (int i = 0; i < nr; ++i) act[i] = i;
  TRY(upload_list(h, h->d_rlist_adv, act, n));
  std::vector<double> rdt(nr);
  for (int i = 0; i < nr; ++i) rdt[i] = dt / (double)n[i];
  CK(h, cudaMemcpyAsync(h->d_rdt, rdt.data(), sizeof(double) * nr, cudaMemcpyHostToDevice, h->stream));
  h->dring_valid = false;
  double *f = h->buf[h->cur];
  double *A = h->buf[scratch(h, 0)], *B = h->buf[scratch(h, 1)];
  for (int64_t q = 0; q < nmax; ++q) {
    int na = 0;
    while (na < nr && n[act[na]] > q) ++na;
    if (h->adv_time == 2) {  // SSPRK(3,3) (src/hipft.f90:7486-7505)
      TRY(advection_stage(h, f, nullptr, A, AdvCombine{0, 0.0, 0.0, 1.0}, false, na, h->d_rlist_adv, h->d_rdt));
      TRY(advection_stage(h, A, f, B, AdvCombine{1, c_three_quarter, c_quarter, c_quarter}, true, na, h->d_rlist_adv, h->d_rdt));
      TRY(advection_stage(h, B, f, f, AdvCombine{1, c_third, c_two_third, c_two_third}, true, na, h->d_rlist_adv, h->d_rdt));
    } else {  // SSPRK(4,3) (src/hipft.f90:7552-7574)
      TRY(advection_stage(h, f, nullptr, A, AdvCombine{0, 0.0, 0.0, 0.5}, false, na, h->d_rlist_adv, h->d_rdt));
      TRY(advection_stage(h, A, nullptr, B, AdvCombine{0, 0.0, 0.0, 0.5}, true, na, h->d_rlist_adv, h->d_rdt));
      TRY(advection_stage(h, B, f, A, AdvCombine{1, c_two_third, c_third, c_sixth}, true, na, h->d_rlist_adv, h->d_rdt));
      TRY(advection_stage(h, A, nullptr, f, AdvCombine{0, 0.0, 0.0, 0.5}, true, na, h->d_rlist_adv, h->d_rdt));
    }
  }
  return HIPFT_OK;
}

static int ragged_arrays(hipft_gpu *h) {
  const size_t nr = (size_t)h->nr;
  TRY(once(h, &h->d_rbits, 2 * nr));
  TRY(once(h, &h->d_rlist_dif, nr));
  TRY(once(h, &h->d_rlist_adv, nr));
  TRY(once(h, &h->d_rlen, nr));
  TRY(once(h, &h->d_rdt, nr));
  return HIPFT_OK;
}

extern "C" int hipft_gpu_set_ragged(hipft_gpu *h, int on) {
  if (!h) return HIPFT_EINVAL;
  CK(h, cudaSetDevice(h->dev));
  if (!on) {
    h->ragged = false;
    return HIPFT_OK;
  }
  if (h->red_cb) return fail(h, HIPFT_ESTATE, "set_ragged: a ragged batch has no shared schedule to reduce over ranks");
  if (h->P.advance_diffusion && (h->DC.grid || h->P.diffusion_num_method == 1))
    return fail(h, HIPFT_EINVAL, "set_ragged: needs RKG2 or RKL2 with per-realization constant diffusion coefficients");
  if (h->P.advance_flow && h->adv_time == 1)
    return fail(h, HIPFT_EINVAL, "set_ragged: needs SSPRK(3,3) or SSPRK(4,3) advection");
  const int nr = h->nr;
  TRY(ragged_arrays(h));
  if (h->P.advance_diffusion) TRY(ragged_gershgorin(h));
  h->r_dtmax_valid = false;
  h->r_s.assign(nr, 0);
  h->r_cycles.assign(nr, 0);
  h->r_substeps.assign(nr, 1);
  h->ragged = true;
  return HIPFT_OK;
}

extern "C" int hipft_gpu_flow_dtmax_each(hipft_gpu *h, double *dtmax) {
  if (!h || !dtmax) return HIPFT_EINVAL;
  if (!h->P.advance_flow) return fail(h, HIPFT_ESTATE, "flow_dtmax_each: advance_flow is off");
  CK(h, cudaSetDevice(h->dev));
  TRY(ragged_arrays(h));
  h->r_dtmax_valid = false;
  TRY(ragged_dtmax(h));
  std::copy(h->r_dtmax.begin(), h->r_dtmax.end(), dtmax);
  return HIPFT_OK;
}

extern "C" int hipft_gpu_ragged_schedule(hipft_gpu *h, int64_t *sts_s, int64_t *subcycles, int64_t *adv_substeps,
                                         double *dt_euler) {
  if (!h) return HIPFT_EINVAL;
  if (!h->ragged) return fail(h, HIPFT_ESTATE, "ragged_schedule: the handle is not in ragged mode");
  if (h->graph_on && h->GA.nr) {
    // the device's record of the last graph-run step
    const int nr = h->nr;
    std::vector<long long> s(nr);
    std::vector<int> c(nr), q(nr);
    CK(h, cudaMemcpyAsync(s.data(), h->GA.s_last, sizeof(long long) * nr, cudaMemcpyDeviceToHost, h->stream));
    CK(h, cudaMemcpyAsync(c.data(), h->GA.cycles_i, sizeof(int) * nr, cudaMemcpyDeviceToHost, h->stream));
    CK(h, cudaMemcpyAsync(q.data(), h->GA.nsub_i, sizeof(int) * nr, cudaMemcpyDeviceToHost, h->stream));
    CK(h, cudaStreamSynchronize(h->stream));
    for (int i = 0; i < nr; ++i) {
      h->r_s[i] = s[i];
      h->r_cycles[i] = c[i];
      h->r_substeps[i] = q[i] > 0 ? q[i] : 1;
    }
  }
  for (int i = 0; i < h->nr; ++i) {
    if (sts_s) sts_s[i] = h->r_s.empty() ? 0 : h->r_s[i];
    if (subcycles) subcycles[i] = h->r_cycles.empty() ? 0 : h->r_cycles[i];
    if (adv_substeps) adv_substeps[i] = h->r_substeps.empty() ? 1 : h->r_substeps[i];
    if (dt_euler) dt_euler[i] = h->r_dt_euler.empty() ? 0.0 : h->r_dt_euler[i];
  }
  return HIPFT_OK;
}

extern "C" int hipft_gpu_diffusion_step(hipft_gpu *h, double dtl, hipft_cycle_cb cb, void *user,
                                        hipft_diffusion_info *info) {
  if (!h) return HIPFT_EINVAL;
  if (!h->field_set) return fail(h, HIPFT_ESTATE, "diffusion_step before set_field");
  if (!h->P.advance_diffusion) return fail(h, HIPFT_ESTATE, "diffusion_step: advance_diffusion is off");
  CK(h, cudaSetDevice(h->dev));
  if (h->ragged) return ragged_diffusion_step(h, dtl, info);
  // the ring sums of the step's input are summed afresh (as in ragged
  // batches and in a graph-run step), also when the previous step left the
  // fused kernels' ring sums of the same field
  h->dring_valid = false;
  const int max_sc = 60;
  int64_t stages0 = h->cell_updates;
  int i = 1;
  bool done = false;
  double time_stepped = 0.0;
  double dtl2 = h->auto_sc ? 0.0 : dtl / (double)h->P.diffusion_subcycles;
  for (;;) {
    if (h->auto_sc) TRY(ptl_dt(h, &dtl2));
    if (h->auto_sc && time_stepped + dtl2 >= dtl) {
      dtl2 = dtl - time_stepped;
      done = true;
    }
    if (h->auto_sc && i == max_sc - 1) {
      dtl2 = dtl - time_stepped;
      done = true;
    }
    if (h->auto_sc && h->P.verbose > 0) h->subcycles_state = (int64_t)std::ceil((dtl - time_stepped) / dtl2);
    if (h->P.diffusion_num_method == 1) TRY(euler_steps(h, dtl2));
    else TRY(sts_super_step(h, dtl2, h->auto_sc));
    time_stepped = time_stepped + dtl2;
    if (cb) {
      CK(h, cudaStreamSynchronize(h->stream));
      cb(user, i, time_stepped, dtl2, h->P.diffusion_num_method == 1 ? h->n_euler : h->sts_s, h->subcycles_state);
    }
    if (!h->auto_sc && i == h->P.diffusion_subcycles) done = true;
    if (done) break;
    i = i + 1;
  }
  if (h->auto_sc) h->subcycles_state = i;
  TRY(check_wait_flag(h, "diffusion_step: a bounded wait for ring sums gave up"));
  if (info) {
    info->dtime_diffusion_euler = h->dt_euler;
    info->sts_s = (h->P.diffusion_num_method == 1) ? h->n_euler : h->sts_s;
    info->subcycles = h->subcycles_state;
    int64_t cells = (int64_t)h->ntm * (h->npm - 2) * h->nr;
    info->total_stages = cells ? (h->cell_updates - stages0) / cells : 0;
  }
  return HIPFT_OK;
}

// ================================================================ graph mode
// hipft_gpu_set_graph: every flux_transport_step runs as one launch of a
// captured CUDA graph.  The schedule decisions that the host-driven step
// makes between launches (PTL subcycles, stage counts, advection substeps)
// are made on the device by the schedule kernels of graph_step.cuh, and the
// loops they size are WHILE nodes.  The capture fixes the buffers: the field
// stays in buffer g_cur; stage outputs rotate through four others with fixed
// roles (an even pass reads (R2, R3) and writes (R0, R1), an odd one the other
// way round); each realization's result is gathered back into the field buffer
// after its super-step.

static void graph_release(hipft_gpu *h) {
  if (h->g_exec) cudaGraphExecDestroy(h->g_exec);
  if (h->g_graph) cudaGraphDestroy(h->g_graph);
  h->g_exec = nullptr;
  h->g_graph = nullptr;
}

template <typename T>
static void dfree(hipft_gpu *h, T *&p) {
  if (p) {
    cudaFree((void *)p);
    h->allocs.erase(std::remove(h->allocs.begin(), h->allocs.end(), (void *)p), h->allocs.end());
  }
  p = nullptr;
}

// Schedule arrays for the handle's realizations and `passcap` passes.
static int graph_alloc(hipft_gpu *h, int passcap) {
  GArrays &g = h->GA;
  const size_t nr = (size_t)h->nr;
  if (!g.nr) {  // set last
    double *de = nullptr, *dm = nullptr;
    TRY(once(h, &g.st, 1));
    TRY(once(h, &g.ts, nr));
    TRY(once(h, &g.d, nr));
    TRY(dsmall(h, &de, nr));
    TRY(dsmall(h, &dm, nr));
    TRY(once(h, &g.rdt, nr));
    TRY(once(h, &g.act, nr));
    TRY(once(h, &g.fin, nr));
    TRY(once(h, &g.rl_ptl, nr));
    TRY(once(h, &g.rl_dif, nr));
    TRY(once(h, &g.rl_adv, nr));
    TRY(once(h, &g.rl_adv_all, nr));
    TRY(once(h, &g.nsub_i, nr));
    TRY(once(h, &g.cycles_i, nr));
    TRY(once(h, &g.s_i, nr));
    TRY(once(h, &g.s_last, nr));
    TRY(once(h, &g.bits, 2 * nr));
    g.dt_euler = de;
    g.dtmax = dm;
    CK(h, cudaMemsetAsync(g.st, 0, sizeof(GState), h->stream));
    CK(h, cudaMemsetAsync(g.s_last, 0, nr * sizeof(long long), h->stream));
    CK(h, cudaMemsetAsync(g.cycles_i, 0, nr * sizeof(int), h->stream));
    CK(h, cudaMemsetAsync(g.nsub_i, 0, nr * sizeof(int), h->stream));
    g.nr = h->nr;
  }
  if (passcap > g.passcap) {
    dfree(h, g.nactp);
    dfree(h, g.colsp);
    dfree(h, g.rc);
    g.passcap = 0;
    TRY(dalloc(h, &g.nactp, (size_t)passcap));
    TRY(dalloc(h, &g.colsp, (size_t)passcap));
    TRY(dalloc(h, &g.rc, (size_t)passcap * nr * kMS));
    g.passcap = passcap;
  }
  return HIPFT_OK;
}

// Passes (with the pass loop's slack) a step of length dt can need: one
// subcycle over the whole step at the smallest Euler limit bounds every
// realization's stage count.
static int graph_passes_needed(const hipft_gpu *h, double dt) {
  if (!h->P.advance_diffusion) return kGUnrollMax;
  double dte = h->dt_euler;
  if (h->ragged)
    for (double v : h->r_dt_euler) dte = std::min(dte, v);
  const int64_t s = sts_count(h->P.diffusion_num_method, dt, dte);
  return (int)sts_passes(s) + kGUnrollMax;
}

// Launch parameters a capture bakes in besides the buffers; any change (new
// flows, ragged mode, larger tables) means a new capture.
static std::vector<unsigned char> graph_key(const hipft_gpu *h) {
  std::vector<unsigned char> k;
  auto add = [&](const void *p, size_t n) {
    const unsigned char *c = static_cast<const unsigned char *>(p);
    k.insert(k.end(), c, c + n);
  };
  add(&h->FL, sizeof(h->FL));
  add(&h->DC, sizeof(h->DC));
  add(&h->ptab, sizeof(h->ptab));
  const double bc[4] = {h->bc_flow_n, h->bc_flow_s, h->bc_diff_n, h->bc_diff_s};
  add(bc, sizeof(bc));
  const int flags[6] = {h->ragged ? 1 : 0, h->cur, h->GA.passcap, h->g_pdl ? 1 : 0, h->auto_sc ? 1 : 0,
                        (int)h->P.diffusion_subcycles};
  add(flags, sizeof(flags));
  return k;
}

// A conditional handle on the graph that stream s is capturing into.
static cudaError_t g_handle(cudaStream_t s, cudaGraphConditionalHandle *hc) {
  cudaStreamCaptureStatus cs;
  cudaGraph_t cg = nullptr;
  cudaError_t e = cudaStreamGetCaptureInfo(s, &cs, nullptr, &cg, nullptr, nullptr);
  if (e != cudaSuccess) return e;
  if (cs != cudaStreamCaptureStatusActive) return cudaErrorStreamCaptureInvalidated;
  return cudaGraphConditionalHandleCreate(hc, cg, 0, 0);
}

// A WHILE node on handle hc at stream s's capture point; returns its body.
static cudaError_t g_while(cudaStream_t s, cudaGraphConditionalHandle hc, cudaGraph_t *body) {
  cudaStreamCaptureStatus cs;
  cudaGraph_t cg = nullptr;
  const cudaGraphNode_t *deps = nullptr;
  size_t nd = 0;
  cudaError_t e = cudaStreamGetCaptureInfo(s, &cs, nullptr, &cg, &deps, &nd);
  if (e != cudaSuccess) return e;
  if (cs != cudaStreamCaptureStatusActive) return cudaErrorStreamCaptureInvalidated;
  cudaGraphNodeParams p = {};
  p.type = cudaGraphNodeTypeConditional;
  p.conditional.handle = hc;
  p.conditional.type = cudaGraphCondTypeWhile;
  p.conditional.size = 1;
  cudaGraphNode_t node;
  e = cudaGraphAddNode(&node, cg, deps, nd, &p);
  if (e != cudaSuccess) return e;
  *body = p.conditional.phGraph_out[0];
  return cudaStreamUpdateCaptureDependencies(s, &node, 1, cudaStreamSetCaptureDependencies);
}

// Captures the split step: the host-driven step's kernels, grids and
// argument values (ragged or plain), with realization lists, coefficients
// and substep lengths read from the schedule arrays.
static int graph_capture(hipft_gpu *h) {
  graph_release(h);
  for (auto &s : h->g_side)
    if (!s) CK(h, cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
  const int nr = h->nr;
  GArrays &G = h->GA;
  G.method = h->P.diffusion_num_method;
  G.auto_sc = h->auto_sc ? 1 : 0;
  G.subcycles = (int)h->P.diffusion_subcycles;
  G.ragged = h->ragged ? 1 : 0;
  G.strang = h->P.strang_splitting ? 1 : 0;
  G.n2 = h->npm - 2;
  G.strips = h->m_strips;
  G.slots = h->m_slots;
  G.poles = pole_places(h->npm - 2);
  G.nadv = (h->adv_time == 1) ? 1 : ((h->adv_time == 2) ? 3 : 4);
  {
    const char *e = std::getenv("HIPFT_GRAPH_UNROLL");
    const int u = e ? std::atoi(e) : kGUnrollMax;  // each iteration boundary costs ~11 us (tick, node relaunch)
    G.unroll = std::max(2, std::min(kGUnrollMax, u - u % 2));
  }
  const GArrays g = G;
  h->g_cur = h->cur;
  double *F = h->buf[h->cur];
  double *Bd = h->buf[scratch(h, 0)];  // A u0, then dty0
  double *R[4] = {h->buf[scratch(h, 1)], h->buf[scratch(h, 2)], h->buf[scratch(h, 3)], h->buf[scratch(h, 4)]};
  const Mesh M = h->M;
  const int64_t nfield = (int64_t)h->fieldn;
  const int cblocks = 4 * h->num_sms;
  double *ring = h->d_ringbuf[0];
  cudaError_t first = cudaSuccess;
  auto ok = [&](cudaError_t e) {
    if (e != cudaSuccess && first == cudaSuccess) first = e;
  };
  auto peek = [&]() { ok(cudaPeekAtLastError()); };
  // captured on a stream of its own (the handle's stream may be the legacy
  // default stream, which cannot capture); launched on the handle's stream
  cudaStream_t s0 = h->g_side[2], s1 = h->g_side[0], s2 = h->g_side[1];
  // the body of a WHILE node at stream s's capture point, captured on stream b
  auto begin_body = [&](cudaStream_t s, cudaGraphConditionalHandle hc, cudaStream_t b) {
    cudaGraph_t body = nullptr;
    ok(g_while(s, hc, &body));
    if (first == cudaSuccess)
      ok(cudaStreamBeginCaptureToGraph(b, body, nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed));
  };
  auto end_body = [&](cudaStream_t b) {
    cudaGraph_t gdone = nullptr;
    ok(cudaStreamEndCapture(b, &gdone));
  };

  // ---- advection_step over frac * dt (src/hipft.f90:4509-4549)
  auto adv_stage = [&](cudaStream_t s, const double *x, const double *f0, double *out, AdvCombine cb) {
    // the first stage reads the field, after a kernel that is not a stage
    ok(launch_adv_stage(h, s, (unsigned)nr, x, f0, out, cb, g.rl_adv, g.rdt, h->g_pdl, x != F));
  };
  auto advection = [&](double frac) {
    cudaGraphConditionalHandle hc{};
    ok(g_handle(s0, &hc));
    if (first != cudaSuccess) return;
    k_g_adv_plan<<<1, 256, 0, s0>>>(g, frac, hc);
    peek();
    begin_body(s0, hc, s1);
    if (first != cudaSuccess) return;
    double *A = R[0], *B = R[1];
    if (h->adv_time == 1) {  // FE (src/hipft.f90:7440-7444), then back into the field
      adv_stage(s1, F, nullptr, A, AdvCombine{0, 0.0, 0.0, 1.0});
      k_g_copy<<<cblocks, 256, 0, s1>>>(F, A, nfield);
      peek();
    } else if (h->adv_time == 2) {  // SSPRK(3,3) (src/hipft.f90:7486-7505)
      adv_stage(s1, F, nullptr, A, AdvCombine{0, 0.0, 0.0, 1.0});
      adv_stage(s1, A, F, B, AdvCombine{1, c_three_quarter, c_quarter, c_quarter});
      adv_stage(s1, B, F, F, AdvCombine{1, c_third, c_two_third, c_two_third});
    } else {  // SSPRK(4,3) (src/hipft.f90:7552-7574)
      adv_stage(s1, F, nullptr, A, AdvCombine{0, 0.0, 0.0, 0.5});
      adv_stage(s1, A, nullptr, B, AdvCombine{0, 0.0, 0.0, 0.5});
      adv_stage(s1, B, F, A, AdvCombine{1, c_two_third, c_third, c_sixth});
      adv_stage(s1, A, nullptr, F, AdvCombine{0, 0.0, 0.0, 0.5});
    }
    k_g_adv_tick<<<1, 256, 0, s1>>>(g, (h->adv_time == 1) ? 3 : g.nadv + 1, hc);
    peek();
    end_body(s1);
  };

  // ---- one pass of the loop body: pass q of the iteration.  Its grid covers
  // any number of realizations that may still take part.
  int64_t pass_blocks = 1;
  for (int n = 1; n <= nr && h->P.advance_diffusion; ++n) pass_blocks = std::max(pass_blocks, march_blocks(h, n));
  auto pass = [&](cudaStream_t s, int q, bool after_pass) {
    const int in = (q & 1) ? 0 : 2, out = 2 - in;
    MarchArgs a = march_args(h, F, Bd);
    a.x2 = R[in];
    a.x1 = R[in + 1];
    a.o[2] = R[out];
    a.o[3] = R[out + 1];
    a.rlist = g.rl_dif;
    a.rc = g.rc;
    a.dctr = &g.st->pctr;
    a.doff = q;
    a.dnact = g.nactp;
    a.dstride = kMS * nr;
    a.dcols = g.colsp;
    ok(launch_pass(h, s, a, h->g_pdl, after_pass, pass_blocks));
  };

  // ---- diffusion_step over dt (src/hipft.f90:4551-4695)
  auto diffusion = [&]() {
    cudaGraphConditionalHandle hsub{};
    ok(g_handle(s0, &hsub));
    if (first != cudaSuccess) return;
    k_g_dif_begin<<<1, 256, 0, s0>>>(g, 0, hsub);
    peek();
    begin_body(s0, hsub, s1);
    if (first != cudaSuccess) return;
    int body_kernels = 3;  // ring sums, A u0 and the subcycle tick
    k_ring_diffusion<<<nr, 256, 0, s1>>>(M, h->DC, F, ring);
    peek();
    const dim3 blk(32, 8), grd = ax_grid(h, nr);
    unsigned long long *bblk = ax_block_max(h);
    const int pr = h->ragged ? 1 : 0;
    unsigned long long *bmax = g.bits, *bmin = g.bits + (h->ragged ? nr : 1);
    if (h->auto_sc) {
      k_g_ptl_reset<<<1, 256, 0, s1>>>(g);
      peek();
    }
    k_ax<<<grd, blk, 0, s1>>>(M, h->DC, F, Bd, ring, h->bc_diff_n, h->bc_diff_s, h->auto_sc ? bmax : nullptr, bblk,
                              g.rl_ptl, pr);
    peek();
    if (h->auto_sc) {  // PTL (src/hipft.f90:5042-5161) of the active realizations
      k_ptl<<<grd, blk, 0, s1>>>(M, F, Bd, bmax, bblk, bmin, g.rl_ptl, pr);
      peek();
      ++body_kernels;
    }
    cudaGraphConditionalHandle hpass{};
    ok(g_handle(s1, &hpass));
    if (first != cudaSuccess) return;
    k_g_plan<<<1, 256, 0, s1>>>(g, hpass);
    peek();
    const int64_t ncoef = (int64_t)g.passcap * nr;
    k_g_coefs<<<(unsigned)((ncoef + 255) / 256), 256, 0, s1>>>(g);
    peek();
    k_scale<<<dim3((unsigned)std::min<int64_t>((h->plane / 2 + 255) / 256, cblocks), (unsigned)nr), 256, 0, s1>>>(
        h->plane, Bd, Bd, 0.0, g.rl_dif, g.d);
    peek();
    ++body_kernels;
    begin_body(s1, hpass, s2);
    if (first != cudaSuccess) return;
    int pass_kernels = 0;
    for (int q = 0; q < g.unroll; ++q) {
      pass(s2, q, q > 0);
      MarchArgs a{};
      a.dctr = &g.st->pctr;
      pass_kernels += pass_launches(h, a, q > 0);
    }
    k_g_pass_tick<<<1, 1, 0, s2>>>(g, pass_kernels, hpass);
    peek();
    end_body(s2);
    // the result of each realization back into the field: Y_s is in R1 after
    // an even last pass, in R3 after an odd one
    k_g_gather<<<dim3((unsigned)nr, 64u), 256, 0, s1>>>(g, M, F, R[1], R[3]);
    peek();
    k_g_sub_tick<<<1, 256, 0, s1>>>(g, body_kernels, hsub);
    peek();
    end_body(s1);
  };

  ok(cudaStreamBeginCapture(s0, cudaStreamCaptureModeThreadLocal));
  if (first == cudaSuccess) {
    k_g_step_begin<<<1, 32, 0, s0>>>(g);
    peek();
    const double fa = h->P.strang_splitting ? 0.5 : 1.0;
    if (h->P.advance_flow) advection(fa);
    if (h->P.advance_diffusion && first == cudaSuccess) diffusion();
    if (h->P.strang_splitting && h->P.advance_flow && first == cudaSuccess) advection(0.5);
  }
  // a failed body capture may leave a side stream capturing
  for (cudaStream_t s : {s1, s2}) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &cs) == cudaSuccess && cs != cudaStreamCaptureStatusNone) {
      cudaGraph_t gd = nullptr;
      cudaStreamEndCapture(s, &gd);
      if (first == cudaSuccess) first = cudaErrorStreamCaptureInvalidated;
    }
  }
  cudaGraph_t graph = nullptr;
  cudaError_t ee = cudaStreamEndCapture(s0, &graph);
  if (first == cudaSuccess) first = ee;
  if (first == cudaSuccess) first = cudaGraphInstantiate(&h->g_exec, graph, 0);
  if (first != cudaSuccess) {
    if (graph) cudaGraphDestroy(graph);
    h->g_exec = nullptr;
    cudaGetLastError();
    return fail(h, HIPFT_ECUDA, "graph capture of the step: %s", cudaGetErrorString(first));
  }
  h->g_graph = graph;
  h->g_key = graph_key(h);
  return HIPFT_OK;
}

// Statistics of the last graph-run step into the handle's counters.
static int graph_collect(hipft_gpu *h) {
  if (h->g_stats_valid) return HIPFT_OK;
  CK(h, cudaMemcpyAsync(h->h_pin, h->GA.st, sizeof(GState), cudaMemcpyDeviceToHost, h->stream));
  CK(h, cudaStreamSynchronize(h->stream));
  std::memcpy(&h->g_last, h->h_pin, sizeof(GState));
  h->g_stats_valid = true;
  const GState &st = h->g_last;
  const int64_t cells = (int64_t)h->ntm * (h->npm - 2);
  h->cell_updates += cells * (st.stage_sum + st.adv_slices);
  h->rkg2_cell_stages += cells * st.rkg2_sum;
  h->launches += st.kernels;
  if (h->P.advance_diffusion) {
    h->sts_s = st.smax;
    h->subcycles_state = st.cycles;
  }
  if (st.err == 1) return fail(h, HIPFT_ECUDA, "graph-run step: the stage tables were too small");
  if (st.err == 2) return fail(h, HIPFT_ECUDA, "graph-run step: a loop ran past its iteration limit");
  return HIPFT_OK;
}

// One split step as one graph launch.
static int graph_step(hipft_gpu *h, double dt, hipft_diffusion_info *info) {
  TRY(graph_collect(h));
  const int need = graph_passes_needed(h, dt);
  const bool grow = need > h->GA.passcap;
  TRY(graph_alloc(h, grow ? need + need / 4 : need));
  if (h->cur != h->g_cur && h->g_cur >= 0) {
    // another entry point left the field elsewhere: back into the captured buffer
    CK(h, cudaMemcpyAsync(h->buf[h->g_cur], h->buf[h->cur], h->fieldn * sizeof(double), cudaMemcpyDeviceToDevice,
                          h->stream));
    h->cur = h->g_cur;
  }
  // per-realization limits (ragged: each its own; plain: the shared ones)
  const int nr = h->nr;
  std::vector<double> de(nr, h->dt_euler), dm(nr, 0.0);
  if (h->ragged) {
    if (h->P.advance_diffusion) de = h->r_dt_euler;
    if (h->P.advance_flow) {
      TRY(ragged_dtmax(h));
      dm = h->r_dtmax;
    }
  }
  CK(h, cudaMemcpyAsync(const_cast<double *>(h->GA.dt_euler), de.data(), sizeof(double) * nr,
                        cudaMemcpyHostToDevice, h->stream));
  CK(h, cudaMemcpyAsync(const_cast<double *>(h->GA.dtmax), dm.data(), sizeof(double) * nr, cudaMemcpyHostToDevice,
                        h->stream));
  if (!h->g_exec || graph_key(h) != h->g_key) TRY(graph_capture(h));
  CK(h, cudaMemcpyAsync(&h->GA.st->dt, &dt, sizeof(double), cudaMemcpyHostToDevice, h->stream));
  CK(h, cudaGraphLaunch(h->g_exec, h->stream));
  h->g_stats_valid = false;
  h->dring_valid = false;
  h->ring_cur = 0;
  if (info) {
    TRY(graph_collect(h));
    TRY(check_wait_flag(h, "graph-run step: a bounded wait for ring sums gave up"));
    info->dtime_diffusion_euler = h->dt_euler;
    if (h->ragged && !h->r_dt_euler.empty())
      info->dtime_diffusion_euler = *std::min_element(h->r_dt_euler.begin(), h->r_dt_euler.end());
    info->sts_s = h->g_last.smax;
    info->subcycles = h->g_last.cycles;
    info->total_stages = nr ? h->g_last.stage_sum / nr : 0;
  }
  return HIPFT_OK;
}

extern "C" int hipft_gpu_set_graph(hipft_gpu *h, int on) {
  if (!h) return HIPFT_EINVAL;
  CK(h, cudaSetDevice(h->dev));
  if (!on) {
    TRY(graph_collect(h));
    h->graph_on = false;
    graph_release(h);
    return HIPFT_OK;
  }
  if (h->red_cb) return fail(h, HIPFT_ESTATE, "set_graph: a step shared over ranks reduces on the host");
  if (h->P.advance_source) return fail(h, HIPFT_EINVAL, "set_graph: sources are not part of a graph-run step");
  if (h->P.advance_diffusion && (h->DC.grid || h->P.diffusion_num_method == 1))
    return fail(h, HIPFT_EINVAL, "set_graph: needs RKG2 or RKL2 with per-realization constant diffusion coefficients");
  if (h->nbuf < 6) return fail(h, HIPFT_ESTATE, "set_graph: needs six field buffers");
  const char *e = std::getenv("HIPFT_GRAPH_PDL");
  h->g_pdl = ws_pdl() && !(e && std::atoi(e) == 0);
  h->graph_on = true;
  return HIPFT_OK;
}

extern "C" int hipft_gpu_flux_transport_step(hipft_gpu *h, double dt, hipft_cycle_cb cb, void *user,
                                             hipft_diffusion_info *info) {
  if (!h) return HIPFT_EINVAL;
  if (h->graph_on) {
    if (cb) return fail(h, HIPFT_ESTATE, "flux_transport_step: subcycle callbacks need the host-driven step");
    if (!h->field_set) return fail(h, HIPFT_ESTATE, "flux_transport_step before set_field");
    CK(h, cudaSetDevice(h->dev));
    return graph_step(h, dt, info);
  }
  if (h->P.strang_splitting) {
    double half = dt * 0.5;
    if (h->P.advance_source) TRY(hipft_gpu_source_step(h, half));
    if (h->P.advance_flow) TRY(hipft_gpu_advection_step(h, half));
    if (h->P.advance_diffusion) TRY(hipft_gpu_diffusion_step(h, dt, cb, user, info));
    if (h->P.advance_flow) TRY(hipft_gpu_advection_step(h, half));
    if (h->P.advance_source) TRY(hipft_gpu_source_step(h, half));
  } else {
    if (h->P.advance_flow) TRY(hipft_gpu_advection_step(h, dt));
    if (h->P.advance_diffusion) TRY(hipft_gpu_diffusion_step(h, dt, cb, user, info));
    if (h->P.advance_source) TRY(hipft_gpu_source_step(h, dt));
  }
  return HIPFT_OK;
}

// ----------------------------------------------------------------- sources
static int ensure_sources(hipft_gpu *h) {
  if (h->d_src) return HIPFT_OK;
  TRY(dalloc(h, &h->d_src, h->fieldn));
  CK(h, cudaMemsetAsync(h->d_src, 0, h->fieldn * sizeof(double), h->stream));
  return HIPFT_OK;
}

extern "C" int hipft_gpu_set_source_file(hipft_gpu *h, const double *data_tp) {
  if (!h || !data_tp) return HIPFT_EINVAL;
  CK(h, cudaSetDevice(h->dev));
  TRY(ensure_sources(h));
  if (!h->d_src_file) TRY(dalloc(h, &h->d_src_file, (size_t)h->ldt * h->npm));
  CK(h, cudaMemcpy2DAsync(h->d_src_file, (size_t)h->ldt * sizeof(double), data_tp, (size_t)h->ntm * sizeof(double),
                          (size_t)h->ntm * sizeof(double), (size_t)h->npm, cudaMemcpyHostToDevice, h->stream));
  CK(h, cudaStreamSynchronize(h->stream));
  return HIPFT_OK;
}

static int balance_buffer(hipft_gpu *h, double *a);

extern "C" int hipft_gpu_set_rfe_frame(hipft_gpu *h, int slot, int model, const double *rnd_tp, const double *uf) {
  if (!h || !rnd_tp || !uf || slot < 0 || slot > 1 || model < 1 || model > 2) return HIPFT_EINVAL;
  CK(h, cudaSetDevice(h->dev));
  TRY(ensure_sources(h));
  const int ntm = h->ntm, npm = h->npm, nr = h->nr;
  if (!h->d_rfe[slot]) {
    TRY(dalloc(h, &h->d_rfe[slot], h->fieldn));
    CK(h, cudaMemsetAsync(h->d_rfe[slot], 0, h->fieldn * sizeof(double), h->stream));
  }
  TRY(once(h, &h->d_rnd, (size_t)ntm * npm));
  TRY(once(h, &h->d_rfe_aux, (size_t)(nr + 1) + (ntm + 1)));
  // da_ti per theta row, model 1 (src/hipft.f90:8840-8853)
  std::vector<double> aux((size_t)(nr + 1) + (ntm + 1), 0.0);
  for (int i = 1; i <= nr; ++i) aux[i] = uf[i - 1];
  double *dati = aux.data() + (nr + 1);
  for (int j = 1; j <= ntm; ++j) {
    if (j == 1 || j == ntm) {
      const double tav = (j == 1) ? 0.5 * (h->t[1] + h->t[2]) : 0.5 * (h->t[ntm] + h->t[ntm - 1]);
      const double sn_t = std::sin(tav), d_t = (j == 1) ? h->dth[2] : h->dth[ntm];
      dati[j] = 1.0 / (0.25 * sn_t * d_t);
    } else {
      dati[j] = h->st_i[j] * h->dt_i[j];
    }
  }
  TRY(upload(h, h->d_rfe_aux, aux));
  CK(h, cudaMemcpyAsync(h->d_rnd, rnd_tp, (size_t)ntm * npm * sizeof(double), cudaMemcpyHostToDevice, h->stream));
  double *fr = h->d_rfe[slot];
  dim3 blk(32, 8), grd((unsigned)((ntm + 31) / 32), (unsigned)((npm - 2 + 7) / 8), (unsigned)nr);
  k_rfe_frame<<<grd, blk, 0, h->stream>>>(h->M, model, h->d_rnd, h->d_rfe_aux, h->d_rfe_aux + (nr + 1), fr);
  LAUNCHED(h);
  k_seam<<<dim3((unsigned)((ntm + 127) / 128), (unsigned)nr), 128, 0, h->stream>>>(h->M, ntm, h->ldt, fr);
  LAUNCHED(h);
  k_rfe_poles<<<nr, 128, 0, h->stream>>>(h->M, fr);
  LAUNCHED(h);
  TRY(balance_buffer(h, fr));
  return HIPFT_OK;
}

extern "C" int hipft_gpu_update_source(hipft_gpu *h, int use_file, int use_rfe, int slot1, int slot2,
                                       double alpha) {
  if (!h || slot1 < 0 || slot1 > 1 || slot2 < 0 || slot2 > 1) return HIPFT_EINVAL;
  if ((use_file && !h->d_src_file) || (use_rfe && (!h->d_rfe[slot1] || !h->d_rfe[slot2])))
    return fail(h, HIPFT_ESTATE, "update_source: source file or RFE frame not set");
  CK(h, cudaSetDevice(h->dev));
  TRY(ensure_sources(h));
  dim3 blk(32, 8), grd((unsigned)((h->ntm + 31) / 32), (unsigned)((h->npm + 7) / 8), (unsigned)h->nr);
  k_source_blend<<<grd, blk, 0, h->stream>>>(h->M, use_file ? h->d_src_file : nullptr,
                                             use_rfe ? h->d_rfe[slot1] : nullptr, use_rfe ? h->d_rfe[slot2] : nullptr,
                                             alpha, h->d_src);
  LAUNCHED(h);
  h->src_set = true;
  return HIPFT_OK;
}

extern "C" int hipft_gpu_source_step(hipft_gpu *h, double dt) {
  if (!h) return HIPFT_EINVAL;
  if (!h->field_set) return fail(h, HIPFT_ESTATE, "source_step before set_field");
  if (!h->src_set) return fail(h, HIPFT_ESTATE, "source_step before update_source");
  CK(h, cudaSetDevice(h->dev));
  dim3 blk(32, 8), grd((unsigned)((h->ntm + 31) / 32), (unsigned)((h->npm + 7) / 8), (unsigned)h->nr);
  k_source_step<<<grd, blk, 0, h->stream>>>(h->M, h->d_src, dt, h->buf[h->cur]);
  LAUNCHED(h);
  h->dring_valid = false;
  return HIPFT_OK;
}

// ------------------------------------------------------------ assimilation
// Uploads one observed map and the per-realization blend options
// (assimilate_new_data's inputs, src/hipft.f90:4083-4146; lat-limit indices
// of load_data_assimilation, 4066-4079) and fills the kernels' arguments.
static int da_args(hipft_gpu *h, const double *data3_pt, const hipft_da_opts *o, DAArgs &a) {
  int ntm = h->ntm, npm1 = h->npm1, nr = h->nr;
  size_t nd = (size_t)npm1 * ntm * 3;
  TRY(once(h, &h->d_da, nd));
  TRY(once(h, &h->d_daopt, 3 * (size_t)(nr + 1)));
  TRY(once(h, &h->d_tidx, 2 * (size_t)(nr + 1)));
  std::vector<double> opt(3 * (size_t)(nr + 1), 0.0);
  std::vector<int> tidx(2 * (size_t)(nr + 1), -1);
  for (int i = 1; i <= nr; ++i) {
    opt[i] = o->mu_power ? o->mu_power[i - 1] : 0.0;
    opt[(nr + 1) + i] = o->mu_limit ? o->mu_limit[i - 1] : 0.0;
    opt[2 * (nr + 1) + i] = o->lat_limit[i - 1];
    int t0 = -1, t1 = -1;
    for (int j = 1; j <= ntm; ++j)
      if (h->t[j] >= o->lat_limit[i - 1] * c_d2r && t0 == -1) t0 = j;
    for (int j = ntm; j >= 1; --j)
      if (h->t[j] <= (c_pi - o->lat_limit[i - 1] * c_d2r) && t1 == -1) t1 = j;
    tidx[i] = t0;
    tidx[(nr + 1) + i] = t1;
  }
  TRY(upload(h, h->d_daopt, opt));
  CK(h, cudaMemcpyAsync(h->d_tidx, tidx.data(), tidx.size() * sizeof(int), cudaMemcpyHostToDevice, h->stream));
  if (o->custom_from_mu && (!o->mu_power || !o->mu_limit))
    return fail(h, HIPFT_EINVAL, "assimilate: custom_from_mu needs mu_power and mu_limit");
  const size_t slice = (size_t)npm1 * ntm;
  if (o->custom_from_mu) {
    // mu^power weights (src/hipft.f90:4246-4252), one plane per distinct
    // (power, limit), evaluated on the device while the data slice is still
    // on its way; the map's own weight slice is not read and not copied.
    std::vector<double> keys;  // power, limit of each plane
    std::vector<int> widx((size_t)nr + 1, 0);
    for (int i = 1; i <= nr; ++i) {
      size_t u = 0;
      while (2 * u < keys.size() && !(keys[2 * u] == o->mu_power[i - 1] && keys[2 * u + 1] == o->mu_limit[i - 1])) ++u;
      if (2 * u == keys.size()) {
        keys.push_back(o->mu_power[i - 1]);
        keys.push_back(o->mu_limit[i - 1]);
      }
      widx[i] = (int)u;
    }
    const size_t np = keys.size() / 2;
    if (np * slice > h->daw_cap) {
      if (h->d_daw) {
        CK(h, cudaStreamSynchronize(h->stream));
        cudaFree(h->d_daw);
        h->allocs.erase(std::remove(h->allocs.begin(), h->allocs.end(), (void *)h->d_daw), h->allocs.end());
        h->d_daw = nullptr;
        h->daw_cap = 0;
      }
      TRY(dalloc(h, &h->d_daw, np * slice));
      h->daw_cap = np * slice;
    }
    TRY(once(h, &h->d_dawidx, (size_t)nr + 1));
    TRY(once(h, &h->d_dawkey, 2 * (size_t)nr));
    TRY(upload(h, h->d_dawkey, keys));
    CK(h, cudaMemcpyAsync(h->d_dawidx, widx.data(), widx.size() * sizeof(int), cudaMemcpyHostToDevice, h->stream));
    CK(h, cudaMemcpyAsync(h->d_da + 2 * slice, data3_pt + 2 * slice, slice * sizeof(double), cudaMemcpyHostToDevice,
                          h->stream));
    k_da_mu_weights<<<dim3((unsigned)((slice + 255) / 256), (unsigned)np), 256, 0, h->stream>>>(
        (int64_t)slice, h->d_da + 2 * slice, h->d_dawkey, h->d_daw);
    LAUNCHED(h);
    CK(h, cudaMemcpyAsync(h->d_da, data3_pt, slice * sizeof(double), cudaMemcpyHostToDevice, h->stream));
    CK(h, cudaStreamSynchronize(h->stream));  // the caller's map and the vectors above are free again
  } else {
    CK(h, cudaMemcpyAsync(h->d_da, data3_pt, 2 * slice * sizeof(double), cudaMemcpyHostToDevice, h->stream));
  }
  a = DAArgs{};
  a.data = h->d_da;
  a.mu_power = h->d_daopt;
  a.mu_limit = h->d_daopt + (nr + 1);
  a.lat_limit = h->d_daopt + 2 * (nr + 1);
  a.tidx0 = h->d_tidx;
  a.tidx1 = h->d_tidx + (nr + 1);
  a.add = o->add;
  a.custom_from_mu = o->custom_from_mu;
  a.mult_fac = o->mult_fac;
  a.wmap = h->d_daw;
  a.widx = h->d_dawidx;
  return HIPFT_OK;
}

extern "C" int hipft_gpu_assimilate(hipft_gpu *h, const double *data3_pt, const hipft_da_opts *o) {
  if (!h || !data3_pt || !o) return HIPFT_EINVAL;
  if (!h->field_set) return fail(h, HIPFT_ESTATE, "assimilate before set_field");
  if (!o->lat_limit || (o->custom_from_mu && (!o->mu_power || !o->mu_limit)))
    return fail(h, HIPFT_EINVAL, "assimilate: missing per-realization options");
  CK(h, cudaSetDevice(h->dev));
  int ntm = h->ntm, npm1 = h->npm1, nr = h->nr;
  DAArgs a;
  TRY(da_args(h, data3_pt, o, a));
  double *f = h->buf[h->cur], *delta = h->buf[scratch(h, 0)];
  dim3 blk(32, 8), grd((unsigned)((ntm + 31) / 32), (unsigned)((npm1 + 31) / 32), (unsigned)nr);
  k_da_delta<<<grd, blk, 0, h->stream>>>(h->M, a, f, delta);
  LAUNCHED(h);
  const double *ratio = nullptr;
  if (o->balance_flux) {
    int cpb = 16, nb = (h->npm - 1 + cpb - 1) / cpb;
    TRY(ensure_part(h, (size_t)nr * nb * 2 + (nr + 1)));
    double *da_t = h->d_anw, *da_p = h->d_anw + 3 * ((size_t)std::max(ntm, h->npm) + 1);
    k_flux_partial<<<dim3((unsigned)nb, (unsigned)nr), 256, 0, h->stream>>>(h->M, da_t, da_p, delta, 1, h->d_part,
                                                                            cpb);
    LAUNCHED(h);
    std::vector<double> part((size_t)nr * nb * 2);
    CK(h, cudaMemcpyAsync(part.data(), h->d_part, part.size() * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    CK(h, cudaStreamSynchronize(h->stream));
    std::vector<double> r(nr + 1, 1.0);
    for (int i = 0; i < nr; ++i) {
      double fp = 0.0, fm = 0.0;
      for (int b = 0; b < nb; ++b) {
        fp = fp + part[((size_t)i * nb + b) * 2];
        fm = fm + part[((size_t)i * nb + b) * 2 + 1];
      }
      r[i + 1] = (fm + fp == 0.0) ? 1.0 : std::sqrt(std::fabs(fp / fm));
    }
    double *dr = h->d_part + (size_t)nr * nb * 2;
    TRY(upload(h, dr, r));
    ratio = dr;
  }
  dim3 g2((unsigned)((ntm + 31) / 32), (unsigned)((h->npm + 7) / 8), (unsigned)nr);
  k_da_apply<<<g2, blk, 0, h->stream>>>(h->M, delta, f, ratio);
  LAUNCHED(h);
  h->dring_valid = false;
  return HIPFT_OK;
}

// ------------------------------------------------------------ diagnostics
extern "C" int hipft_gpu_set_validation(hipft_gpu *h, int mode, const double *fval_u0_pt, double width,
                                        double vt_const, double vp_omega, double time_start) {
  if (!h || mode < 0 || mode > 2) return HIPFT_EINVAL;
  CK(h, cudaSetDevice(h->dev));
  h->vmode = mode;
  h->vwidth = width;
  h->vt_const = vt_const;
  h->vp_omega = vp_omega;
  h->vtime_start = time_start;
  if (mode == 1) {
    if (!fval_u0_pt) return HIPFT_EINVAL;
    if ((int)h->Dc.size() != h->nr)
      return fail(h, HIPFT_ESTATE, "validation 1 needs the diffusion coefficient constants");
    size_t n = (size_t)h->npm1 * h->ntm * h->nr;
    if (!h->d_fval_u0) TRY(dalloc(h, &h->d_fval_u0, n));
    CK(h, cudaMemcpyAsync(h->d_fval_u0, fval_u0_pt, n * sizeof(double), cudaMemcpyHostToDevice, h->stream));
  }
  if (mode == 2 && !h->d_vgauss) {
    // theta scale, phi scale and st_i (1-based) for the analytic Gaussians
    size_t L = (size_t)std::max(h->npm, h->nt) + 2;
    std::vector<double> v(3 * L, 0.0);
    for (int j = 1; j <= h->ntm; ++j) {
      v[j] = h->t[j];
      v[2 * L + j] = h->st_i[j];
    }
    for (int k = 1; k <= h->npm; ++k) v[L + k] = h->p[k];
    TRY(dalloc(h, &h->d_vgauss, v.size()));
    TRY(upload(h, h->d_vgauss, v));
  }
  return HIPFT_OK;
}

// Fortran MODULO for reals.
static double fmodulo(double a, double p) { return a - std::floor(a / p) * p; }

extern "C" int hipft_gpu_analysis(hipft_gpu *h, double time, double *hist) {
  if (!h || !hist) return HIPFT_EINVAL;
  if (!h->field_set) return fail(h, HIPFT_ESTATE, "analysis before set_field");
  CK(h, cudaSetDevice(h->dev));
  int ntm = h->ntm, npm = h->npm, nr = h->nr;
  AnalysisArgs a{};
  size_t L = (size_t)std::max(ntm, npm) + 1;
  a.da_t = h->d_anw; a.sn_t = h->d_anw + L; a.cs_t = h->d_anw + 2 * L;
  a.da_p = h->d_anw + 3 * L; a.cs_p = h->d_anw + 4 * L; a.sn_p = h->d_anw + 5 * L;
  a.pn = h->d_masks; a.ps = h->d_masks + (ntm + 1);
  a.vmode = h->vmode;
  if (h->vmode == 1) {
    // fval = fval_u0 * exp(-42 D factor (time - time_start))  (src/hipft.f90:3156-3159)
    std::vector<double> sc(nr + 1, 0.0);
    for (int i = 1; i <= nr; ++i)
      sc[i] = std::exp(-42.0 * h->Dc[i - 1] * h->P.diffusion_coef_factor * (time - h->vtime_start));
    TRY(upload(h, h->d_vscale, sc));
    a.fval_u0 = h->d_fval_u0;
    a.vscale = h->d_vscale;
  } else if (h->vmode == 2) {
    size_t G = (size_t)std::max(h->npm, h->nt) + 2;
    a.t = h->d_vgauss; a.p = h->d_vgauss + G; a.st_i = h->d_vgauss + 2 * G;
    a.vtt = h->vt_const * c_km_s_to_rs_hr * (time - h->vtime_start);
    a.vpt = h->vp_omega * c_km_s_to_rs_hr * (time - h->vtime_start);
    a.p1 = fmodulo(c_pi_two + a.vpt, c_twopi);
    a.p2 = fmodulo(c_threepi_two + a.vpt, c_twopi);
    a.width = h->vwidth;
  }
  const int cpb = 8;
  int nb = (npm - 1 + cpb - 1) / cpb;
  TRY(ensure_part(h, (size_t)nr * nb * kNPart + (size_t)nr * kNPart));
  double *fin = h->d_part + (size_t)nr * nb * kNPart;
  k_analysis_partial<256><<<dim3((unsigned)nb, (unsigned)nr), 256, 0, h->stream>>>(h->M, a, h->buf[h->cur],
                                                                                    h->d_part, cpb);
  LAUNCHED(h);
  k_analysis_final<<<(nr * kNPart + 127) / 128, 128, 0, h->stream>>>(nb, nr, h->d_part, fin);
  LAUNCHED(h);
  TRY(sync_read(h, fin, (size_t)nr * kNPart * sizeof(double)));
  for (int i = 0; i < nr; ++i) {
    const double *v = h->h_pin + (size_t)i * kNPart;
    double *o = hist + (size_t)i * 14;
    o[0] = v[0]; o[1] = v[1]; o[2] = v[2];
    double verr = v[3], sumfval2 = v[4];
    o[13] = (sumfval2 == 0.0) ? std::sqrt(verr / (double)((int64_t)ntm * (npm - 1))) : std::sqrt(verr / sumfval2);
    o[3] = c_rsun_cm2 * v[5]; o[4] = c_rsun_cm2 * v[6];
    o[5] = c_rsun_cm2 * v[7]; o[6] = c_rsun_cm2 * v[8];
    o[7] = c_rsun_cm2 * v[9]; o[8] = c_rsun_cm2 * v[10];
    o[9] = c_rsun_cm2 * v[11]; o[10] = c_rsun_cm2 * v[12];
    o[12] = c_three_quarter * c_pi_i * v[15];
    double e1 = c_three_quarter * c_pi_i * v[13], e2 = c_three_quarter * c_pi_i * v[14];
    o[11] = std::sqrt(e1 * e1 + e2 * e2);
  }
  return HIPFT_OK;
}

static int flux_of(hipft_gpu *h, const double *a, std::vector<double> &fp, std::vector<double> &fm) {
  int nr = h->nr;
  const int cpb = 16;
  int nb = (h->npm - 1 + cpb - 1) / cpb;
  TRY(ensure_part(h, (size_t)nr * nb * 2 + (nr + 1)));
  size_t L = (size_t)std::max(h->ntm, h->npm) + 1;
  k_flux_partial<<<dim3((unsigned)nb, (unsigned)nr), 256, 0, h->stream>>>(h->M, h->d_anw, h->d_anw + 3 * L, a, 0,
                                                                          h->d_part, cpb);
  LAUNCHED(h);
  std::vector<double> part((size_t)nr * nb * 2);
  CK(h, cudaMemcpyAsync(part.data(), h->d_part, part.size() * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
  CK(h, cudaStreamSynchronize(h->stream));
  fp.assign(nr, 0.0);
  fm.assign(nr, 0.0);
  for (int i = 0; i < nr; ++i)
    for (int b = 0; b < nb; ++b) {
      fp[i] = fp[i] + part[((size_t)i * nb + b) * 2];
      fm[i] = fm[i] + part[((size_t)i * nb + b) * 2 + 1];
    }
  return HIPFT_OK;
}

extern "C" int hipft_gpu_get_flux(hipft_gpu *h, double *flux_p, double *flux_m) {
  if (!h || !flux_p || !flux_m) return HIPFT_EINVAL;
  if (!h->field_set) return fail(h, HIPFT_ESTATE, "get_flux before set_field");
  CK(h, cudaSetDevice(h->dev));
  std::vector<double> fp, fm;
  TRY(flux_of(h, h->buf[h->cur], fp, fm));
  std::copy(fp.begin(), fp.end(), flux_p);
  std::copy(fm.begin(), fm.end(), flux_m);
  return HIPFT_OK;
}

// balance_flux (src/hipft.f90:8752-8807) of every realization of `a`
static int balance_buffer(hipft_gpu *h, double *a) {
  std::vector<double> fp, fm;
  TRY(flux_of(h, a, fp, fm));
  std::vector<double> r(h->nr + 1, 1.0);
  for (int i = 0; i < h->nr; ++i) r[i + 1] = (fm[i] + fp[i] == 0.0) ? 1.0 : std::sqrt(std::fabs(fp[i] / fm[i]));
  size_t L = (size_t)h->nr * ((h->npm - 1 + 15) / 16) * 2;
  double *dr = h->d_part + L;
  TRY(upload(h, dr, r));
  dim3 blk(32, 8), grd((unsigned)((h->ntm + 31) / 32), (unsigned)((h->npm + 7) / 8), (unsigned)h->nr);
  k_scale_balance<<<grd, blk, 0, h->stream>>>(h->M, a, dr);
  LAUNCHED(h);
  CK(h, cudaStreamSynchronize(h->stream));
  return HIPFT_OK;
}

extern "C" int hipft_gpu_balance_flux(hipft_gpu *h) {
  if (!h) return HIPFT_EINVAL;
  if (!h->field_set) return fail(h, HIPFT_ESTATE, "balance_flux before set_field");
  CK(h, cudaSetDevice(h->dev));
  TRY(balance_buffer(h, h->buf[h->cur]));
  h->dring_valid = false;
  return HIPFT_OK;
}

extern "C" int hipft_gpu_info(const hipft_gpu *h, hipft_info *info) {
  if (!h || !info) return HIPFT_EINVAL;
  info->ntm = h->ntm;
  info->npm = h->npm;
  info->nr = h->nr;
  info->ldt = h->ldt;
  info->dtime_diffusion_euler = h->dt_euler;
  info->sts_s = (h->P.diffusion_num_method == 1) ? h->n_euler : h->sts_s;
  info->kernel_launches = h->launches;
  info->cell_stage_updates = h->cell_updates;
  info->device_bytes = h->dev_bytes;
  info->rkg2_stages = h->rkg2_stages;
  info->rkg2_cell_stages = h->rkg2_cell_stages;
  return HIPFT_OK;
}

// "ws-quad" stands for passes of four stages by independent warps (k_sts_march).
extern "C" int hipft_gpu_describe(hipft_gpu *h, char *buf, size_t len) {
  if (!h || !buf || !len) return HIPFT_EINVAL;
  const char *k = "none";
  if (h->P.advance_diffusion) {
    MarchArgs a{};
    a.nreal = h->nr;
    if (h->P.diffusion_num_method == 1) k = "explicit Euler steps";
    else if (h->DC.grid) k = "one stage per launch (k_diffusion_stage)";
    else if (h->ntm < kMMinRows) k = "four stages per pass, all rows as pole rows (k_sts_whole)";
    else if (!poles_by_column(h)) k = "ws-quad (four stages per pass): k_sts_march, pole strips stage by stage (k_sts_poles_any)";
    else if (pass_columns(h, a) && !h->graph_on) k = "ws-quad (four stages per pass): k_sts_march and pole strips in one launch";
    else k = "ws-quad (four stages per pass): k_sts_march, pole strips beside it (k_sts_poles)";
  }
  std::snprintf(buf, len, "schedule=%s; diffusion kernels: %s", h->ragged ? "ragged" : "shared", k);
  return HIPFT_OK;
}

extern "C" int hipft_gpu_set_stream(hipft_gpu *h, void *s) {
  if (!h) return HIPFT_EINVAL;
  CK(h, cudaStreamSynchronize(h->stream));
  if (s) {
    if (h->own_stream) cudaStreamDestroy(h->stream);
    h->own_stream = false;
    h->stream = (cudaStream_t)s;
  } else if (!h->own_stream) {
    CK(h, cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking));
    h->own_stream = true;
  }
  return HIPFT_OK;
}

extern "C" int hipft_gpu_expire_wait(hipft_gpu *h, unsigned int limit) {
  if (!h || limit == 0 || limit > (1u << 22)) return HIPFT_EINVAL;
  CK(h, cudaSetDevice(h->dev));
  k_wait_selftest<<<1, 32, 0, h->stream>>>(limit, h->d_err);
  LAUNCHED(h);
  return HIPFT_OK;
}

extern "C" int hipft_gpu_check_bounded_wait(hipft_gpu *h, unsigned int limit) {
  if (!h || limit == 0 || limit > (1u << 22)) return HIPFT_EINVAL;
  CK(h, cudaSetDevice(h->dev));
  TRY(hipft_gpu_expire_wait(h, limit));
  return check_wait_flag(h, "check_bounded_wait: the wait gave up as intended");
}

extern "C" int hipft_gpu_field_device_ptr(hipft_gpu *h, double **ptr, int *ldt) {
  if (!h || !ptr || !ldt) return HIPFT_EINVAL;
  if (!h->field_set) return fail(h, HIPFT_ESTATE, "field_device_ptr before set_field");
  CK(h, cudaSetDevice(h->dev));
  CK(h, cudaStreamSynchronize(h->stream));  // the field is complete when the pointer is handed out
  *ptr = h->buf[h->cur];
  *ldt = h->ldt;
  return HIPFT_OK;
}

extern "C" int hipft_gpu_synchronize(hipft_gpu *h) {
  if (!h) return HIPFT_EINVAL;
  CK(h, cudaStreamSynchronize(h->stream));
  return HIPFT_OK;
}

// Folds finished event pairs into the per-kind totals.
static int prof_collect(hipft_gpu *h) {
  CK(h, cudaStreamSynchronize(h->stream));
  for (int k = 0; k < HIPFT_K_NKINDS; ++k) {
    for (auto &pr : h->ev_pending[k]) {
      float ms = 0.f;
      CK(h, cudaEventElapsedTime(&ms, pr.first, pr.second));
      h->prof_ms[k] += ms;
      h->prof_n[k] += 1;
      h->ev_pool.push_back(pr.first);
      h->ev_pool.push_back(pr.second);
    }
    h->ev_pending[k].clear();
  }
  return HIPFT_OK;
}

extern "C" int hipft_gpu_set_profiling(hipft_gpu *h, int on) {
  if (!h) return HIPFT_EINVAL;
  TRY(prof_collect(h));
  for (int k = 0; k < HIPFT_K_NKINDS; ++k) {
    h->prof_ms[k] = 0.0;
    h->prof_n[k] = 0;
  }
  h->profiling = on != 0;
  return HIPFT_OK;
}

extern "C" int hipft_gpu_kernel_time(hipft_gpu *h, int kind, int64_t *launches, double *total_ms) {
  if (!h || kind < 0 || kind >= HIPFT_K_NKINDS || !launches || !total_ms) return HIPFT_EINVAL;
  TRY(prof_collect(h));
  *launches = h->prof_n[kind];
  *total_ms = h->prof_ms[kind];
  return HIPFT_OK;
}

// ======================================================================
// hipft_get_flux_noalloc: get_flux (src/hipft.f90:8672) for callers that
// cannot allocate GPU memory.
//
// Some callers own every byte of device memory themselves: a Fortran code
// that keeps its maps device-resident through OpenMP `target enter data`
// mappings (HipFT's own model) and hands over `use_device_ptr` addresses, or
// a host application that runs the GPU from a fixed, pre-reserved arena.
// They cannot let a library call cudaMalloc.  This entry point takes the
// field as a device pointer and keeps all of its scratch -- the mesh scales,
// the cell-area weights, the per-block partial sums and the per-realization
// results -- in one file-scope __device__ array, g_na_scratch, of fixed size
// (kNaScratchDoubles doubles, about 1.6 MB), which every GPU that loads this
// library holds until the process exits.
//
// Limits: ntm <= kNaMaxNtm, npm1 <= kNaMaxNpm1, nr <= kNaMaxNr, and the
// partial sums (2 * nr * ceil((npm1)/16)) must fit kNaMaxPart; larger
// requests return HIPFT_EINVAL.  The array is shared by every call on a
// device and keeps the last call's contents, so calls that overlap on the GPU
// (different streams, or different host threads) race; serialise them.
// The first call on a device looks up the array's device address with
// cudaGetSymbolAddress (with that device current) and caches it; make that
// first call before any stream capture.
// ======================================================================
#include <mutex>

namespace {
constexpr int kNaMaxNtm = 16384;
constexpr int kNaMaxNpm1 = 16384;
constexpr int kNaMaxNr = 2000;
constexpr int kNaMaxPart = 1 << 17;
constexpr int kNaMaxDevices = 64;
// layout (doubles): t[kNaMaxNtm+2] p[kNaMaxNpm1+2] da_t[kNaMaxNtm+2] da_p[kNaMaxNpm1+2] part[kNaMaxPart] out[2*kNaMaxNr]
constexpr size_t kNaOffT = 0;
constexpr size_t kNaOffP = kNaOffT + kNaMaxNtm + 2;
constexpr size_t kNaOffDaT = kNaOffP + kNaMaxNpm1 + 2;
constexpr size_t kNaOffDaP = kNaOffDaT + kNaMaxNtm + 2;
constexpr size_t kNaOffPart = kNaOffDaP + kNaMaxNpm1 + 2;
constexpr size_t kNaOffOut = kNaOffPart + kNaMaxPart;
constexpr size_t kNaScratchDoubles = kNaOffOut + 2 * kNaMaxNr;
std::mutex g_na_mutex;
double *g_na_dev_ptr[kNaMaxDevices] = {};
}  // namespace

static __device__ __align__(256) double g_na_scratch[kNaScratchDoubles];

// Cell-area weights of get_flux (src/hipft.f90:8712-8732) from the raw
// scales, computed with set_mesh's definitions (6579-6641); 1-based.
__global__ void k_na_weights(int ntm, int npm1, const double *t, const double *p, double *da_t, double *da_p) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x + 1;
  if (n <= ntm) {
    const int j = n;
    double v;
    if (j == 1) {
      v = 0.25 * sin(0.5 * (t[1] + t[2])) * (t[2] - t[1]);
    } else if (j == ntm) {
      v = 0.25 * sin(0.5 * (t[ntm] + t[ntm - 1])) * (t[ntm] - t[ntm - 1]);
    } else {
      double thj = 0.5 * (t[j] + t[j - 1]), thj1 = 0.5 * (t[j + 1] + t[j]);
      v = sin(t[j]) * (thj1 - thj);
    }
    da_t[j] = v;
  }
  if (n <= npm1) {
    const int k = n;
    double v;
    if (k == 1 || k == npm1) {
      v = 0.5 * (p[npm1] - p[npm1 - 1]);
    } else {
      double phk = 0.5 * (p[k] + p[k - 1]), phk1 = 0.5 * (p[k + 1] + p[k]);
      v = phk1 - phk;
    }
    da_p[k] = v;
  }
}

// Per-realization totals of the block partials, in block order.
__global__ void k_na_flux_final(int nb, int nr, const double *part, double *out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nr) return;
  double fp = 0.0, fm = 0.0;
  for (int b = 0; b < nb; ++b) {
    fp = fp + part[((int64_t)i * nb + b) * 2];
    fm = fm + part[((int64_t)i * nb + b) * 2 + 1];
  }
  out[2 * i] = fp;
  out[2 * i + 1] = fm;
}

static int na_fail(char *err, size_t len, int code, const char *msg) {
  if (err && len) std::snprintf(err, len, "hipft_get_flux_noalloc: %s", msg);
  return code;
}

extern "C" int hipft_get_flux_noalloc(const double *f_dev, int ntm, int npm1, int nr, int ldt, const double *t,
                                      const double *p, double *flux_p, double *flux_m, void *cuda_stream,
                                      char *err, size_t err_len) {
  if (!f_dev || !t || !p || !flux_p || !flux_m) return na_fail(err, err_len, HIPFT_EINVAL, "null argument");
  if (ntm < 4 || npm1 < 5 || nr < 1 || ldt < ntm)
    return na_fail(err, err_len, HIPFT_EINVAL, "sizes out of range (ntm >= 4, npm1 >= 5, nr >= 1, ldt >= ntm)");
  const int cpb = 16;
  const int npm = npm1 + 1;
  const int nb = (npm - 1 + cpb - 1) / cpb;
  if (ntm > kNaMaxNtm || npm1 > kNaMaxNpm1 || nr > kNaMaxNr || (size_t)2 * nr * nb > (size_t)kNaMaxPart)
    return na_fail(err, err_len, HIPFT_EINVAL,
                   "grid too large for the fixed scratch (ntm <= 16384, npm1 <= 16384, nr <= 2000, "
                   "2*nr*ceil(npm1/16) <= 131072)");
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kNaMaxDevices)
    return na_fail(err, err_len, HIPFT_ECUDA, "no usable current device");
  double *base = nullptr;
  {
    std::lock_guard<std::mutex> lk(g_na_mutex);
    if (!g_na_dev_ptr[dev]) {
      double *ptr = nullptr;
      cudaError_t e = cudaGetSymbolAddress((void **)&ptr, g_na_scratch);
      if (e != cudaSuccess || !ptr) return na_fail(err, err_len, HIPFT_ECUDA, cudaGetErrorString(e));
      g_na_dev_ptr[dev] = ptr;
    }
    base = g_na_dev_ptr[dev];
  }
  cudaStream_t s = (cudaStream_t)cuda_stream;
  double *dt = base + kNaOffT, *dp = base + kNaOffP, *dat = base + kNaOffDaT, *dap = base + kNaOffDaP;
  double *part = base + kNaOffPart, *out = base + kNaOffOut;
  // 1-based scales
  if (cudaMemcpyAsync(dt + 1, t, sizeof(double) * ntm, cudaMemcpyHostToDevice, s) != cudaSuccess ||
      cudaMemcpyAsync(dp + 1, p, sizeof(double) * npm1, cudaMemcpyHostToDevice, s) != cudaSuccess)
    return na_fail(err, err_len, HIPFT_ECUDA, "copy of the scales failed");
  int nmax = ntm > npm1 ? ntm : npm1;
  k_na_weights<<<(nmax + 255) / 256, 256, 0, s>>>(ntm, npm1, dt, dp, dat, dap);
  Mesh m{};
  m.ntm = ntm;
  m.npm = npm;
  m.nt = ntm + 1;
  m.np = npm;
  m.nr = nr;
  m.ldt = ldt;
  m.plane = (int64_t)ldt * npm;
  k_flux_partial<<<dim3((unsigned)nb, (unsigned)nr), 256, 0, s>>>(m, dat, dap, f_dev, 0, part, cpb);
  k_na_flux_final<<<(nr + 127) / 128, 128, 0, s>>>(nb, nr, part, out);
  {
    cudaError_t le = cudaGetLastError();
    if (le != cudaSuccess) {
      char msg[256];
      std::snprintf(msg, sizeof msg, "kernel launch failed: %s", cudaGetErrorString(le));
      return na_fail(err, err_len, HIPFT_ECUDA, msg);
    }
  }
  if (cudaMemcpy2DAsync(flux_p, sizeof(double), out, 2 * sizeof(double), sizeof(double), (size_t)nr,
                        cudaMemcpyDeviceToHost, s) != cudaSuccess ||
      cudaMemcpy2DAsync(flux_m, sizeof(double), out + 1, 2 * sizeof(double), sizeof(double), (size_t)nr,
                        cudaMemcpyDeviceToHost, s) != cudaSuccess)
    return na_fail(err, err_len, HIPFT_ECUDA, "copy of the results failed");
  cudaError_t e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return na_fail(err, err_len, HIPFT_ECUDA, cudaGetErrorString(e));
  return HIPFT_OK;
}

// ------------------------------------------------------------------ adjoint
// Discrete adjoint of one flux_transport_step (no reference counterpart):
// the step is replayed from its input with every stage input kept (the
// "tape"), then run backwards through the transposed stages.  The schedule
// of the replay (PTL subcycle dts, RKG2 stage counts) is the forward's own,
// computed by the same routines from the same field, and is held fixed:
// the gradient is that of the discrete map at this schedule.



// Stage spacing of the stage checkpoints for a super-step of s stages:
// 0 (keep every stage) when s + 1 fields fit the tape budget, else an even
// q near sqrt(2 s), which keeps about 2 sqrt(2 s) fields.
static int64_t adj_stage_spacing(hipft_gpu *h, int64_t s) {
  int64_t budget = h->adj_tape_limit;
  if (budget <= 0) {
    if (h->adj_free_seen == 0) {  // once per run (reset by hipft_adj_clear / hipft_adj_release)
      size_t fr = 0, tot = 0;
      if (cudaMemGetInfo(&fr, &tot) != cudaSuccess) fr = 0;
      h->adj_free_seen = fr + 1;
    }
    budget = (int64_t)((h->adj_free_seen - 1) / 2 / (h->fieldn * sizeof(double)));
  }
  if (h->adj_force_q > 0) return h->adj_force_q;
  if (s + 1 <= budget) return 0;
  int64_t q = (int64_t)std::ceil(std::sqrt(2.0 * (double)s));
  if (q % 2) ++q;
  return std::max<int64_t>(q, 2);
}

// Tape slot n; slots are allocated in chunks of up to 32 fields (at most
// 256 MB per chunk), so that taping many steps needs few allocations.
static int adj_slot(hipft_gpu *h, size_t n, double **p) {
  while (h->tape.size() <= n) {
    const size_t fb = h->fieldn * sizeof(double);
    const size_t per = std::max<size_t>(1, std::min<size_t>(32, (size_t)(256u << 20) / fb));
    double *q = nullptr;
    TRY(dalloc(h, &q, h->fieldn * per));
    h->tape_chunks.push_back(q);
    for (size_t e = 0; e < per; ++e) h->tape.push_back(q + e * h->fieldn);
  }
  *p = h->tape[n];
  return HIPFT_OK;
}

typedef void (*AdjPassKernel)(Mesh, AdjPassArgs, PairTables);
static AdjPassKernel adj_march_kernel(int ns, bool wide) {
  if (wide) return ns == 4 ? k_adj_march<4, uint64_t> : k_adj_march<2, uint64_t>;
  return ns == 4 ? k_adj_march<4, uint32_t> : k_adj_march<2, uint32_t>;
}
static AdjPassKernel adj_poles_kernel(int ns, int threads) {
  if (threads > kPMidThreads) return ns == 4 ? k_adj_poles<4, kPMaxThreads> : k_adj_poles<2, kPMaxThreads>;
  return ns == 4 ? k_adj_poles<4, kPMidThreads> : k_adj_poles<2, kPMidThreads>;
}

// ns reverse stages (four or two) as the strips' and the march's launches;
// after_pass: the launch before them on the stream is such a pass too.
static int adj_pass(hipft_gpu *h, AdjPassArgs a, int ns, bool after_pass) {
  const int n2 = h->npm - 2, nc = poles_ranks(n2);
  a.dpart = h->d_jpart;
  a.dstride = h->jpart_per_r;
  a.strips = h->j_strips;
  a.cols = h->j_cols;
  a.dfac = h->DC.dfac;
  a.bcn = h->bc_diff_n;
  a.bcs = h->bc_diff_s;
  a.err = h->d_err;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = (ws_pdl() && after_pass) ? 1 : 0;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)nc;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.stream = h->stream;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  cfg.gridDim = dim3((unsigned)(2 * h->nr * nc));
  cfg.blockDim = dim3((unsigned)poles_threads(n2));
  cfg.dynamicSmemBytes = adj_poles_smem(ns, poles_threads(n2));
  const AdjPassKernel poles = adj_poles_kernel(ns, poles_threads(n2));
  const int most = std::max(kPMidThreads, poles_most_threads(n2));
  CK(h, smem_limit(h, (const void *)poles, adj_poles_smem(ns, most)));
  CK(h, cudaLaunchKernelEx(&cfg, poles, h->M, a, h->ptab));
  LAUNCHED(h);
  const int nch = (n2 + a.cols - 1) / a.cols;
  attr[0].val.programmaticStreamSerializationAllowed = ws_pdl() ? 1 : 0;
  cfg.numAttrs = 1;
  cfg.gridDim = dim3((unsigned)((int64_t)a.strips * ((nch + kJWarps - 1) / kJWarps) * h->nr));
  cfg.blockDim = dim3(32 * kJWarps);
  cfg.dynamicSmemBytes = adj_march_smem(ns);
  const AdjPassKernel march = adj_march_kernel(ns, h->plane >= (int64_t)1 << 29);
  CK(h, smem_limit(h, (const void *)march, adj_march_smem(ns)));
  CK(h, cudaLaunchKernelEx(&cfg, march, h->M, a, h->ptab));
  LAUNCHED(h);
  return HIPFT_OK;
}

// Work arrays of the reverse pass.  A call that failed may be repeated: it goes
// on with what is missing, and nothing is ready before everything is there.
static int adj_ensure(hipft_gpu *h) {
  if (h->adj_ready) return HIPFT_OK;
  TRY(dfields(h, h->adjw, (int)(sizeof(h->adjw) / sizeof(h->adjw[0]))));
  dim3 g = stage_grid(h, 32, 8);
  h->dpart_per_r = (int)(g.x * g.y);
  TRY(once(h, &h->d_dpart, (size_t)h->dpart_per_r * h->nr));
  h->adj_nch = (h->npm - 2 + 255) / 256;
  TRY(once(h, &h->d_gring, 2 * (size_t)h->nr * h->adj_nch));
  TRY(once(h, &h->d_dpole, (size_t)h->nr * h->adj_nch));
  for (auto &gp : h->d_gpart) TRY(once(h, &gp, 2 * (size_t)g.y * h->nr));
  const int n2 = h->npm - 2;
  if (h->ntm >= kJMinRows && poles_by_column(h)) {
    h->j_strips = adj_strips(h->ntm);
    // a strip's block leaves no room for the march's on its SM; with those SMs counted in,
    // 512x1024 took a second wave and 34 us per pass instead of 20
    const int sms = std::max(h->num_sms - 2 * h->nr * poles_ranks(n2), h->num_sms / 2);
    h->j_cols = adj_cols(n2, h->j_strips, h->nr, kJWarps * kJBlocks * sms);
    const int per_r = h->j_strips * ((n2 + h->j_cols - 1) / h->j_cols) + 2 * poles_ranks(n2);
    TRY(once(h, &h->d_jpart, (size_t)per_r * h->nr));
    h->jpart_per_r = per_r;
  }
  h->adj_ready = true;
  return HIPFT_OK;
}

// SSPRK(4,3) with its four stage inputs kept (src/hipft.f90:7552-7574);
// the result replaces the current field.
static int adj_adv_fwd(hipft_gpu *h, double dtl, size_t &nt, size_t t[4]) {
  double *T[4];
  for (int q = 0; q < 4; ++q) {
    t[q] = nt;
    TRY(adj_slot(h, nt++, &T[q]));
  }
  double *f = h->buf[h->cur];
  CK(h, cudaMemcpyAsync(T[0], f, h->fieldn * sizeof(double), cudaMemcpyDeviceToDevice, h->stream));
  TRY(advection_stage(h, T[0], nullptr, T[1], AdvCombine{0, 0.0, 0.0, 0.5 * dtl}, false));
  TRY(advection_stage(h, T[1], nullptr, T[2], AdvCombine{0, 0.0, 0.0, 0.5 * dtl}, true));
  TRY(advection_stage(h, T[2], T[0], T[3], AdvCombine{1, c_two_third, c_third, c_sixth * dtl}, true));
  TRY(advection_stage(h, T[3], nullptr, f, AdvCombine{0, 0.0, 0.0, 0.5 * dtl}, true));
  h->dring_valid = false;
  return HIPFT_OK;
}

// diffusion_step (src/hipft.f90:4551-4695) with RKG2 super-steps whose
// stage fields are kept; same subcycle logic as hipft_gpu_diffusion_step.
static int adj_diff_fwd(hipft_gpu *h, double dtl, size_t &nt, std::vector<AdjSub> &subs) {
  const int max_sc = 60;
  int i = 1;
  bool done = false;
  double time_stepped = 0.0;
  double dtl2 = h->auto_sc ? 0.0 : dtl / (double)h->P.diffusion_subcycles;
  for (;;) {
    if (h->auto_sc) TRY(ptl_dt(h, &dtl2));
    if (h->auto_sc && time_stepped + dtl2 >= dtl) {
      dtl2 = dtl - time_stepped;
      done = true;
    }
    if (h->auto_sc && i == max_sc - 1) {
      dtl2 = dtl - time_stepped;
      done = true;
    }
    load_sts(h, dtl2);
    AdjSub S;
    S.dtl = dtl2;
    S.s = h->sts_s;
    S.uj = h->sts_uj;
    S.vj = h->sts_vj;
    S.ubj = h->sts_ubj;
    S.gj = h->sts_gj;
    S.t0 = nt;
    S.q = adj_stage_spacing(h, S.s);
    double *u0, *dty0;
    TRY(adj_slot(h, nt++, &u0));
    TRY(adj_slot(h, nt++, &dty0));
    std::vector<double *> Y((size_t)S.s + 1, nullptr);
    Y[0] = u0;
    if (S.q == 0) {
      for (int64_t k = 1; k <= S.s - 1; ++k) TRY(adj_slot(h, nt++, &Y[k]));
    } else {
      // block starts c = 1, 1+q, ... below s; their pairs (Y_{c-1}, Y_c) are
      // tape slots; of the other stages a pass keeps its last two, which the
      // next pass reads, in a rotating scratch set
      for (int64_t c = 1; c <= S.s - 1; c += S.q) S.cstart.push_back(c);
      for (size_t b = 0; b < S.cstart.size(); ++b) {
        const int64_t c = S.cstart[b];
        S.ck_prev.push_back(SIZE_MAX);
        if (c > 1) {
          S.ck_prev.back() = nt;
          TRY(adj_slot(h, nt++, &Y[c - 1]));
        }
        S.ck_cur.push_back(nt);
        TRY(adj_slot(h, nt++, &Y[c]));
      }
      while (h->adj_block.size() < 4) {
        double *q = nullptr;
        TRY(dalloc(h, &q, h->fieldn));
        h->adj_block.push_back(q);
      }
    }
    Y[S.s] = h->buf[h->cur];
    CK(h, cudaMemcpyAsync(u0, h->buf[h->cur], h->fieldn * sizeof(double), cudaMemcpyDeviceToDevice, h->stream));
    // the passes of sts_super_step, with the tape's stages kept
    if (!h->auto_sc) TRY(apply_lap(h, nullptr, nullptr, h->nr, 0));
    TRY(scale_dty0(h, h->buf[scratch(h, 0)], dty0, dtl2));
    MarchArgs a = march_args(h, u0, dty0);
    const int64_t np = sts_passes(S.s), pad = kMS * np - S.s;
    for (int64_t p = 0; p < np; ++p) {
      for (int q = 0; q < kMS; ++q) {
        const int64_t k = kMS * p + q + 1 - pad;
        a.c[q] = sts_slot(h->P.diffusion_num_method, S.s, kMS * p + q, dtl2);
        a.o[q] = (k >= 1) ? Y[k] : nullptr;
        if (q >= 2 && !a.o[q]) a.o[q] = S.q ? h->adj_block[2 * (p & 1) + q - 2] : h->buf[scratch(h, q - 1)];
      }
      a.first = p == 0;
      TRY(sts_pass(h, a, p > 0));
      a.x2 = a.o[kMS - 2];
      a.x1 = a.o[kMS - 1];
    }
    TRY(seam(h, Y[S.s]));
    h->dring_valid = false;
    h->cell_updates += (int64_t)h->ntm * (h->npm - 2) * h->nr * S.s;
    subs.push_back(std::move(S));
    time_stepped = time_stepped + dtl2;
    if (!h->auto_sc && i == h->P.diffusion_subcycles) done = true;
    if (done) break;
    i = i + 1;
  }
  return HIPFT_OK;
}

// a work field other than those in `busy`
static double *adj_free(hipft_gpu *h, std::initializer_list<const double *> busy) {
  for (double *w : h->adjw) {
    bool used = false;
    for (const double *b : busy) used = used || (b == w);
    if (!used) return w;
  }
  return nullptr;
}

static int adj_adv_rev(hipft_gpu *h, double dtl, const size_t t[4], double *&W, double *gflow) {
  const dim3 blk(32, 8), grd = stage_grid(h, 32, 8);
  double *g[5];
  for (int q = 0; q < 5; ++q) g[q] = gflow + (size_t)q * h->fieldn;
  auto stage = [&](const double *x, const double *w, double sigma, double alpha, const double *base, double beta,
                   double *out) -> int {
    k_adj_pole_sums<<<h->nr, 256, 0, h->stream>>>(h->M, w, h->d_gring);
    LAUNCHED(h);
    k_adj_adv<<<grd, blk, 0, h->stream>>>(h->M, h->FL, h->W, x, w, base, out, h->d_gring,
                                          AdjAdvArgs{sigma, alpha, beta, h->bc_flow_n, h->bc_flow_s}, g[0], g[1],
                                          g[2], g[3], g[4]);
    LAUNCHED(h);
    return HIPFT_OK;
  };
  double *b3 = adj_free(h, {W});
  double *b2 = adj_free(h, {W, b3});
  double *b1 = adj_free(h, {W, b3, b2});
  const double *T0 = h->tape[t[0]], *T1 = h->tape[t[1]], *T2 = h->tape[t[2]], *T3 = h->tape[t[3]];
  TRY(stage(T3, W, -0.5 * dtl, 1.0, nullptr, 0.0, b3));
  TRY(stage(T2, b3, -c_sixth * dtl, c_third, nullptr, 0.0, b2));
  TRY(stage(T1, b2, -0.5 * dtl, 1.0, nullptr, 0.0, b1));
  TRY(stage(T0, b1, -0.5 * dtl, 1.0, b3, c_two_third, W));
  return HIPFT_OK;
}

// Reverse of one RKG2 super-step: W (cotangent of Y_s) becomes the
// cotangent of u0; dacc[i] += the diffusion-coefficient terms
// sum mu~_k dt <A^T Wbar_k, Y_{k-1}> (+ dt <A^T dbar, u0>).  One launch per
// stage: each leaves the pole-row partials of its output for the next.
// Recomputes the stages Y_{c+1}..Y_e of stage-checkpoint block b (e = the
// block's last stage input, at most s-1) from its pair (Y_{c-1}, Y_c); the
// values do not depend on how the stages are grouped into passes, so they are
// bitwise those of the replay.  Y receives the block's fields.
static int adj_block_recompute(hipft_gpu *h, const AdjSub &S, size_t b, std::vector<const double *> &Y) {
  const int64_t c = S.cstart[b], e = std::min(c + S.q - 1, S.s - 1);
  while ((int64_t)h->adj_block.size() < S.q + kMS - 1) {
    double *q = nullptr;
    TRY(dalloc(h, &q, h->fieldn));
    h->adj_block.push_back(q);
  }
  const double *u0 = h->tape[S.t0], *dty0 = h->tape[S.t0 + 1];
  std::vector<double *> Yw((size_t)(e + kMS) + 1, nullptr);
  Yw[c - 1] = (S.ck_prev[b] == SIZE_MAX) ? const_cast<double *>(u0) : h->tape[S.ck_prev[b]];
  Yw[c] = h->tape[S.ck_cur[b]];
  for (int64_t k = c + 1; k < e + kMS; ++k) Yw[k] = h->adj_block[k - c - 1];
  MarchArgs a = march_args(h, u0, dty0);
  const int64_t pad = kMS * sts_passes(S.s) - S.s;
  for (int64_t k = c + 1; k <= e; k += kMS) {
    a.x2 = Yw[k - 2];
    a.x1 = Yw[k - 1];
    for (int q = 0; q < kMS; ++q) {
      a.c[q] = sts_slot(h->P.diffusion_num_method, S.s, k + q - 1 + pad, S.dtl);
      a.o[q] = Yw[k + q];
    }
    TRY(sts_pass(h, a, k > c + 1));
  }
  for (int64_t q = c - 1; q <= e; ++q) Y[q] = Yw[q];
  h->dring_valid = false;
  return HIPFT_OK;
}

// HIPFT_ADJ_PAIR=0 runs the reverse RKG2 stages one per launch (A/B timing).
static bool adj_pairs_enabled() {
  static int v = -1;
  if (v < 0) {
    const char *e = std::getenv("HIPFT_ADJ_PAIR");
    v = (e && std::atoi(e) == 0) ? 0 : 1;
  }
  return v == 1;
}

static int adj_diff_rev(hipft_gpu *h, const AdjSub &S, double *&W, double *dacc) {
  const dim3 blk(32, 8), grd = stage_grid(h, 32, 8);
  const double dtl = S.dtl;
  double *ub = adj_free(h, {W});
  double *db = adj_free(h, {W, ub});
  CK(h, cudaMemsetAsync(ub, 0, h->fieldn * sizeof(double), h->stream));
  CK(h, cudaMemsetAsync(db, 0, h->fieldn * sizeof(double), h->stream));
  CK(h, cudaMemsetAsync(h->d_dpart, 0, (size_t)h->dpart_per_r * h->nr * sizeof(double), h->stream));
  CK(h, cudaMemsetAsync(h->d_dpole, 0, (size_t)h->adj_nch * h->nr * sizeof(double), h->stream));
  // stage inputs Y_k: all on the tape (q == 0) or one recomputed block at a time
  std::vector<const double *> Yr((size_t)S.s + 1, nullptr);
  Yr[0] = h->tape[S.t0];
  if (S.q == 0)
    for (int64_t k = 1; k <= S.s - 1; ++k) Yr[k] = h->tape[S.t0 + 1 + k];
  int64_t curb = -1;
  auto Yt = [&](int64_t k) -> const double * { return Yr[k]; };
  const double *gin = h->d_gring;
  int npin = 1, pp = 0;
  auto pole_sums = [&](const double *w) -> int {
    k_adj_pole_sums<<<h->nr, 256, 0, h->stream>>>(h->M, w, h->d_gring);
    LAUNCHED(h);
    gin = h->d_gring;
    npin = 1;
    return HIPFT_OK;
  };
  auto stage = [&](const double *w, const double *wp, const double *y, double *out, double *u, double *d,
                   AdjDiffCoef ac) -> int {
    double *gout = h->d_gpart[pp];
    k_adj_diff<<<grd, blk, 0, h->stream>>>(h->M, h->DC, w, wp, y, out, u, d, gin, npin, gout, h->bc_diff_n,
                                           h->bc_diff_s, ac, h->d_dpart, h->ptab);
    LAUNCHED(h);
    gin = gout;
    npin = (int)grd.y;
    pp ^= 1;
    return HIPFT_OK;
  };
  double *Wk = W, *Wk1 = nullptr;
  int64_t k = S.s;
  // four or two reverse stages per pass, whose stage inputs lie in one
  // stage-checkpoint block
  if (h->jpart_per_r) {
    CK(h, cudaMemsetAsync(h->d_jpart, 0, (size_t)h->jpart_per_r * h->nr * sizeof(double), h->stream));
    bool after = false;
    while (k >= 3 && adj_pairs_enabled()) {
      if (S.q > 0 && (k - 2) / S.q != curb) {
        curb = (k - 2) / S.q;
        TRY(adj_block_recompute(h, S, (size_t)curb, Yr));
        after = false;
      }
      const int64_t room = S.q > 0 ? (k - 2) % S.q + 1 : k - 1;  // stages whose inputs are at hand
      if (room < 2) break;
      const int ns = room >= kMS ? kMS : 2;
      AdjPassArgs a{};
      a.w0 = Wk;
      a.w1 = Wk1 ? Wk1 : Wk;
      a.o0 = adj_free(h, {Wk, Wk1, ub, db});
      a.o1 = adj_free(h, {Wk, Wk1, ub, db, a.o0});
      a.ub = ub;
      a.db = db;
      for (int q = 0; q < ns; ++q) {
        const int64_t K = k - q;
        const double nu = (K < S.s) ? S.vj[K + 1] : 0.0;
        a.c[q] = AdjStage{S.uj[K], nu, S.ubj[K] * dtl, 1.0 - S.uj[K] - S.vj[K], S.gj[K], S.ubj[K] * dtl};
        a.y[q] = Yt(K - 1);
      }
      TRY(adj_pass(h, a, ns, after));
      after = true;
      Wk1 = a.o0;
      Wk = a.o1;
      k -= ns;
    }
  }
  if (k >= 2) TRY(pole_sums(Wk));
  // two reverse stages per launch (k_adj_diff2 + k_adj_pole2) while both of
  // their stage inputs Y_{k-1}, Y_{k-2} lie in one stage-checkpoint block
  // A pair launch follows the previous pair's k_adj_pole2 programmatically
  // (its interior tiles start while that kernel runs); its outputs then avoid
  // the previous pair's W_k as well, which that kernel still reads.
  double *Wprev = nullptr;
  bool after_pole2 = false;
  const dim3 grd2((unsigned)((h->ntm + kA2J - 1) / kA2J), (unsigned)((h->npm - 2 + kA2K - 1) / kA2K), (unsigned)h->nr);
  while (adj_pairs_enabled() && k >= 3 && (S.q == 0 || (k - 2) / S.q == (k - 3) / S.q)) {
    if (S.q > 0 && (k - 3) / S.q != curb) {
      curb = (k - 3) / S.q;
      TRY(adj_block_recompute(h, S, (size_t)curb, Yr));
      after_pole2 = false;
    }
    double *Wm1 = adj_free(h, {Wk, Wk1, ub, db, Wprev});
    double *Wm2 = adj_free(h, {Wk, Wk1, ub, db, Wprev, Wm1});
    const double u1 = S.uj[k], v1 = S.vj[k], u2 = S.uj[k - 1], v2 = S.vj[k - 1];
    const double nu1 = (k < S.s) ? S.vj[k + 1] : 0.0;
    const AdjDiff2Coef ac{u1, nu1, S.ubj[k] * dtl, 1.0 - u1 - v1, S.gj[k], S.ubj[k] * dtl,
                          u2, v1, S.ubj[k - 1] * dtl, 1.0 - u2 - v2, S.gj[k - 1], S.ubj[k - 1] * dtl};
    double *gpart = h->d_gpart[pp];
    {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = grd2;
      cfg.blockDim = dim3(kA2J, kA2K);
      cfg.stream = h->stream;
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      attr[0].val.programmaticStreamSerializationAllowed = (ws_pdl() && after_pole2) ? 1 : 0;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      const double *y1 = Yt(k - 1), *y2 = Yt(k - 2);
      CK(h, cudaLaunchKernelEx(&cfg, k_adj_diff2, h->M, h->DC, (const double *)Wk, (const double *)Wk1, y1, y2, Wm1,
                               Wm2, ub, db, gin, npin, gpart, h->bc_diff_n, h->bc_diff_s, ac, h->d_dpart,
                               h->dpart_per_r, h->ptab));
      LAUNCHED(h);
    }
    k_adj_pole2<<<dim3((unsigned)h->nr, (unsigned)h->adj_nch), 256, 0, h->stream>>>(
        h->M, h->DC, Wk, Wm1, Yt(k - 2), Wm2, gpart, (int)grd2.y, h->d_gring, h->bc_diff_n, h->bc_diff_s, ac, h->d_dpole,
        h->ptab);
    LAUNCHED(h);
    after_pole2 = true;
    gin = h->d_gring;
    npin = h->adj_nch;
    pp ^= 1;
    Wprev = Wk;
    Wk1 = Wm1;
    Wk = Wm2;
    k -= 2;
  }
  for (; k >= 2; --k) {
    if (S.q > 0 && (k - 2) / S.q != curb) {
      curb = (k - 2) / S.q;  // the block holding Y_{k-1}
      TRY(adj_block_recompute(h, S, (size_t)curb, Yr));
    }
    double *Wm = adj_free(h, {Wk, Wk1, ub, db});
    const double uj = S.uj[k], vj = S.vj[k];
    const double nu1 = (k < S.s) ? S.vj[k + 1] : 0.0;
    TRY(stage(Wk, Wk1, Yt(k - 1), Wm, ub, db,
              AdjDiffCoef{uj, nu1, S.ubj[k] * dtl, 1.0 - uj - vj, S.gj[k], S.ubj[k] * dtl}));
    Wk1 = Wk;
    Wk = Wm;
  }
  // Y_1 = u0 + mu~_1 dty0 and Y_0 = u0 (read by stage 2 with nu_2)
  k_adj_axpy2<<<grd, blk, 0, h->stream>>>(h->M, ub, 1.0, Wk, S.vj[2], Wk1);
  LAUNCHED(h);
  k_adj_axpy2<<<grd, blk, 0, h->stream>>>(h->M, db, S.ubj[1], Wk, 0.0, nullptr);
  LAUNCHED(h);
  // dty0 = dt A u0
  TRY(pole_sums(db));
  TRY(stage(db, ub, Yt(0), ub, nullptr, nullptr, AdjDiffCoef{0.0, 1.0, dtl, 0.0, 0.0, dtl}));
  k_adj_dsum<<<h->nr, 256, 0, h->stream>>>(h->d_dpart, h->dpart_per_r, h->d_dpole, h->adj_nch, 1.0, dacc);
  LAUNCHED(h);
  if (h->jpart_per_r) {
    k_adj_dsum<<<h->nr, 256, 0, h->stream>>>(h->d_jpart, h->jpart_per_r, nullptr, 0, 1.0, dacc);
    LAUNCHED(h);
  }
  W = ub;
  return HIPFT_OK;
}

static int adj_check(hipft_gpu *h) {
  if (!h->field_set) return fail(h, HIPFT_ESTATE, "adjoint step before set_field");
  if (h->P.advance_flow && (h->adv_time != 3 || h->adv_space != 2))
    return fail(h, HIPFT_ESTATE, "adjoint: advection must be WENO3+SSPRK(4,3)");
  // flows from files (with or without analytic parts) do not depend on the
  // field; attenuated flows do (through |Br|), and the rotated rigid rotation
  // is NaN on most grids
  if (h->P.advance_flow && h->have_flow && (h->fdef.flow_attenuate || h->fdef.flow_rigid_omega != 0.0))
    return fail(h, HIPFT_ESTATE, "adjoint: attenuated or rotated flows are not differentiated");
  if (h->P.advance_diffusion && (h->P.diffusion_num_method != 3 || h->DC.grid))
    return fail(h, HIPFT_ESTATE, "adjoint: diffusion must be RKG2 with per-realization constant coefficients");
  if (h->P.advance_source) return fail(h, HIPFT_ESTATE, "adjoint: sources are not differentiated");
  if (h->ragged) return fail(h, HIPFT_ESTATE, "adjoint: replays the shared (plain) schedule only");
  return HIPFT_OK;
}

// One flux_transport_step of the current field with its tape pushed on the
// tape stack (the field becomes the step's output).
static int adj_record(hipft_gpu *h, double dt) {
  TRY(adj_ensure(h));
  h->dring_valid = false;
  AdjRec R;
  R.dt = dt;
  R.first = h->adj_top;
  size_t nt = h->adj_top;
  const bool strang = h->P.strang_splitting != 0;
  const double da = strang ? 0.5 * dt : dt;
  if (h->P.advance_flow) TRY(adj_adv_fwd(h, da, nt, R.ta1));
  if (h->P.advance_diffusion) TRY(adj_diff_fwd(h, dt, nt, R.subs));
  if (strang && h->P.advance_flow) TRY(adj_adv_fwd(h, da, nt, R.ta2));
  h->adj_top = nt;
  h->adj_top_max = std::max(h->adj_top_max, nt);
  h->adj_recs.push_back(std::move(R));
  return HIPFT_OK;
}

// Reverse of the most recently recorded step (popped from the stack).
static int adj_reverse(hipft_gpu *h, double *fbar, double *dacc, double *gflow) {
  if (h->adj_recs.empty() || !h->adj_ready) return fail(h, HIPFT_ESTATE, "adjoint reverse: no recorded step");
  const AdjRec &R = h->adj_recs.back();
  const size_t bytes = h->fieldn * sizeof(double);
  const bool strang = h->P.strang_splitting != 0;
  const double da = strang ? 0.5 * R.dt : R.dt;
  double *W = h->adjw[0];
  CK(h, cudaMemcpyAsync(W, fbar, bytes, cudaMemcpyDeviceToDevice, h->stream));
  if (strang && h->P.advance_flow) TRY(adj_adv_rev(h, da, R.ta2, W, gflow));
  for (size_t q = R.subs.size(); q-- > 0;) TRY(adj_diff_rev(h, R.subs[q], W, dacc));
  if (h->P.advance_flow) TRY(adj_adv_rev(h, da, R.ta1, W, gflow));
  CK(h, cudaMemcpyAsync(fbar, W, bytes, cudaMemcpyDeviceToDevice, h->stream));
  h->adj_top = R.first;
  h->adj_recs.pop_back();
  h->dring_valid = false;
  return HIPFT_OK;
}

extern "C" int hipft_adj_step(hipft_gpu *h, double dt, const double *f_in, double *fbar, double *dacc,
                              double *gflow) {
  if (!h || !f_in || !fbar || !dacc || !gflow) return HIPFT_EINVAL;
  TRY(adj_check(h));
  CK(h, cudaSetDevice(h->dev));
  CK(h, cudaMemcpyAsync(h->buf[h->cur], f_in, h->fieldn * sizeof(double), cudaMemcpyDeviceToDevice, h->stream));
  TRY(adj_record(h, dt));
  TRY(adj_reverse(h, fbar, dacc, gflow));
  CK(h, cudaStreamSynchronize(h->stream));
  CK(h, cudaGetLastError());
  return check_wait_flag(h, "adj_step: a bounded wait for ring sums gave up");
}

extern "C" int hipft_adj_record(hipft_gpu *h, double dt) {
  if (!h) return HIPFT_EINVAL;
  TRY(adj_check(h));
  CK(h, cudaSetDevice(h->dev));
  TRY(adj_record(h, dt));
  CK(h, cudaGetLastError());
  const int rc = check_wait_flag(h, "adj_record: a bounded wait for ring sums gave up");
  if (rc != HIPFT_OK) {  // a step that is not right is not kept
    h->adj_top = h->adj_recs.back().first;
    h->adj_recs.pop_back();
  }
  return rc;
}

extern "C" int hipft_adj_reverse(hipft_gpu *h, double *fbar, double *dacc, double *gflow) {
  if (!h || !fbar || !dacc || !gflow) return HIPFT_EINVAL;
  CK(h, cudaSetDevice(h->dev));
  TRY(adj_reverse(h, fbar, dacc, gflow));
  CK(h, cudaGetLastError());
  return check_wait_flag(h, "adj_reverse: a bounded wait for ring sums gave up");
}

extern "C" int hipft_adj_clear(hipft_gpu *h) {
  if (!h) return HIPFT_EINVAL;
  h->adj_recs.clear();
  h->adj_top = 0;
  h->adj_free_seen = 0;
  return HIPFT_OK;
}

extern "C" int hipft_adj_recorded(hipft_gpu *h, int64_t *n, int64_t *slots_used) {
  if (!h || !n) return HIPFT_EINVAL;
  *n = (int64_t)h->adj_recs.size();
  if (slots_used) *slots_used = (int64_t)h->adj_top;
  return HIPFT_OK;
}

extern "C" int hipft_adj_tape_fields(hipft_gpu *h, int64_t *n) {
  if (!h || !n) return HIPFT_EINVAL;
  *n = (int64_t)(h->adj_top_max + h->adj_block.size());
  return HIPFT_OK;
}

extern "C" int hipft_adj_set_tape_limit(hipft_gpu *h, int64_t max_fields, int64_t stage_spacing) {
  if (!h || max_fields < 0 || stage_spacing < 0 || stage_spacing % 2) return HIPFT_EINVAL;
  h->adj_tape_limit = max_fields;
  h->adj_force_q = stage_spacing;
  return HIPFT_OK;
}

extern "C" int hipft_adj_release(hipft_gpu *h) {
  if (!h) return HIPFT_EINVAL;
  CK(h, cudaSetDevice(h->dev));
  CK(h, cudaStreamSynchronize(h->stream));
  auto drop = [&](void *p) {
    if (!p) return;
    cudaFree(p);
    h->allocs.erase(std::remove(h->allocs.begin(), h->allocs.end(), p), h->allocs.end());
    h->dev_bytes -= h->fieldn * sizeof(double);
  };
  {
    const size_t fb = h->fieldn * sizeof(double);
    const size_t per = std::max<size_t>(1, std::min<size_t>(32, (size_t)(256u << 20) / fb));
    for (void *q : h->tape_chunks) {
      if (!q) continue;
      cudaFree(q);
      h->allocs.erase(std::remove(h->allocs.begin(), h->allocs.end(), q), h->allocs.end());
      h->dev_bytes -= per * fb;
    }
  }
  for (double *q : h->adj_block) drop(q);
  h->tape.clear();
  h->tape_chunks.clear();
  h->adj_block.clear();
  h->adj_recs.clear();
  h->adj_top = 0;
  h->adj_top_max = 0;
  h->adj_free_seen = 0;
  return HIPFT_OK;
}

extern "C" int hipft_adj_assimilate(hipft_gpu *h, const double *data3_pt, const hipft_da_opts *o, double *fbar) {
  if (!h || !data3_pt || !o || !fbar) return HIPFT_EINVAL;
  if (!o->lat_limit || (o->custom_from_mu && (!o->mu_power || !o->mu_limit)))
    return fail(h, HIPFT_EINVAL, "adj_assimilate: missing per-realization options");
  if (o->balance_flux) return fail(h, HIPFT_ESTATE, "adj_assimilate: the balanced increment is not differentiated");
  CK(h, cudaSetDevice(h->dev));
  DAArgs a;
  TRY(da_args(h, data3_pt, o, a));
  dim3 blk(32, 8), grd((unsigned)((h->ntm + 31) / 32), (unsigned)((h->npm - 2 + 7) / 8), (unsigned)h->nr);
  k_adj_da<<<grd, blk, 0, h->stream>>>(h->M, a, fbar);
  LAUNCHED(h);
  CK(h, cudaStreamSynchronize(h->stream));
  return HIPFT_OK;
}

extern "C" int hipft_adj_assimilate_at(hipft_gpu *h, const double *data3_pt, const hipft_da_opts *o,
                                       const double *f_pre, double *fbar) {
  if (!h || !data3_pt || !o || !fbar) return HIPFT_EINVAL;
  if (!o->balance_flux || o->add) {
    // the plain blend, or an increment that does not depend on f
    hipft_da_opts o2 = *o;
    o2.balance_flux = 0;
    return hipft_adj_assimilate(h, data3_pt, &o2, fbar);
  }
  if (!f_pre) return fail(h, HIPFT_EINVAL, "adj_assimilate_at: the balanced increment needs the field it was applied to");
  if (!o->lat_limit || (o->custom_from_mu && (!o->mu_power || !o->mu_limit)))
    return fail(h, HIPFT_EINVAL, "adj_assimilate_at: missing per-realization options");
  CK(h, cudaSetDevice(h->dev));
  const int ntm = h->ntm, npm1 = h->npm1, nr = h->nr;
  DAArgs a;
  TRY(da_args(h, data3_pt, o, a));
  if (!h->d_adj_delta) TRY(dalloc(h, &h->d_adj_delta, h->fieldn));
  double *delta = h->d_adj_delta;
  dim3 blk(32, 8), grd((unsigned)((ntm + 31) / 32), (unsigned)((npm1 + 31) / 32), (unsigned)nr);
  k_da_delta<<<grd, blk, 0, h->stream>>>(h->M, a, f_pre, delta);
  LAUNCHED(h);
  // F+, F- exactly as the forward's balance (same kernel, same block order),
  // then SP, SN over the core columns
  const int cpb = 16, nb = (h->npm - 1 + cpb - 1) / cpb, nb2 = (h->npm - 2 + cpb - 1) / cpb;
  TRY(ensure_part(h, (size_t)nr * (nb + nb2) * 2 + 4 * (size_t)nr));
  const double *da_t = h->d_anw, *da_p = h->d_anw + 3 * ((size_t)std::max(ntm, h->npm) + 1);
  double *pf = h->d_part, *ps = h->d_part + (size_t)nr * nb * 2, *dcoef = ps + (size_t)nr * nb2 * 2;
  k_flux_partial<<<dim3((unsigned)nb, (unsigned)nr), 256, 0, h->stream>>>(h->M, da_t, da_p, delta, 1, pf, cpb);
  LAUNCHED(h);
  k_adj_bal_partial<<<dim3((unsigned)nb2, (unsigned)nr), 256, 0, h->stream>>>(h->M, delta, fbar, cpb, ps);
  LAUNCHED(h);
  std::vector<double> part((size_t)nr * (nb + nb2) * 2);
  CK(h, cudaMemcpyAsync(part.data(), h->d_part, part.size() * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
  CK(h, cudaStreamSynchronize(h->stream));
  std::vector<double> coef(4 * (size_t)nr);
  for (int i = 0; i < nr; ++i) {
    double fp = 0.0, fm = 0.0, sp = 0.0, sn = 0.0;
    for (int q = 0; q < nb; ++q) {
      fp = fp + part[((size_t)i * nb + q) * 2];
      fm = fm + part[((size_t)i * nb + q) * 2 + 1];
    }
    const double *p2 = part.data() + (size_t)nr * nb * 2;
    for (int q = 0; q < nb2; ++q) {
      sp = sp + p2[((size_t)i * nb2 + q) * 2];
      sn = sn + p2[((size_t)i * nb2 + q) * 2 + 1];
    }
    double *c = coef.data() + 4 * (size_t)i;
    if (fm + fp == 0.0) {  // the forward leaves the increment as it is
      c[0] = c[1] = 1.0;
      c[2] = c[3] = 0.0;
      continue;
    }
    if (fp == 0.0 || fm == 0.0)
      return fail(h, HIPFT_ESTATE, "adj_assimilate_at: realization %d: one-signed balanced increment", i + 1);
    const double r = std::sqrt(std::fabs(fp / fm));
    const double S = -sp / (r * r) + sn;
    c[0] = 1.0 / r;
    c[1] = r;
    c[2] = S * r / (2.0 * fp);
    c[3] = -S * r / (2.0 * fm);
  }
  TRY(upload(h, dcoef, coef));
  dim3 g2((unsigned)((ntm + 31) / 32), (unsigned)((h->npm - 2 + 7) / 8), (unsigned)nr);
  k_adj_da_bal<<<g2, blk, 0, h->stream>>>(h->M, a, delta, da_t, da_p, dcoef, fbar);
  LAUNCHED(h);
  CK(h, cudaStreamSynchronize(h->stream));
  return HIPFT_OK;
}

extern "C" int hipft_gpu_set_field_device(hipft_gpu *h, const double *f_dev) {
  if (!h || !f_dev) return HIPFT_EINVAL;
  if (!h->field_set) return fail(h, HIPFT_ESTATE, "set_field_device before set_field");
  CK(h, cudaSetDevice(h->dev));
  CK(h, cudaMemcpyAsync(h->buf[h->cur], f_dev, h->fieldn * sizeof(double), cudaMemcpyDeviceToDevice, h->stream));
  h->dring_valid = false;
  CK(h, cudaStreamSynchronize(h->stream));
  return HIPFT_OK;
}
