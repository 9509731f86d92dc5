// deb_adjoint.cu -- the discrete-adjoint kernel and its C ABI
// (deb_plan_create_adjoint, deb_adjoint in include/discoeb_gb300.h).
//
// One block of four warps per work item (cotangent seed, k-mode), pulled from
// a device queue in order of recorded step counts, longest first
// (deb_adjoint_block.cuh).  A block integrates its mode backwards segment by
// segment: it recomputes the segment's states from the checkpoint the recorded
// forward solve stored, then steps back through them.  As much of an item's
// state as fits lives in shared memory, the rest in a global workspace
// (L2-resident for the blocks in flight).  Replaces the reference's jax.jacfwd
// through diffrax (perturbations.py:765) by one reverse sweep per mode.

#include <cuda_runtime.h>

#include <cstring>
#include <mutex>

#include "deb_adjoint_block.cuh"
#include "deb_internal.h"
#include "discoeb_gb300.h"

namespace {

__constant__ deb::Tab c_tab;
__constant__ deb::Rodas c_rodas;

struct AParams {
  const double* tables;      // [ncosmo, blob_len]
  const double* tables_pm;   // [ncosmo * 2 npar, blob_len]
  int ncosmo, npar, blob_len;
  const double* eps;         // [ncosmo, npar]
  const double* k;
  const int* cosmo;
  int nmode, nseed, nout;
  const double* tau_out;     // [ncosmo, nout]
  const double* tau_pm;      // [ncosmo * 2 npar, nout]
  const double* rec;
  int rec_len;
  const int* nrec;
  const double* ckpt;
  int ck_cap;
  const long long* ckoff;    // null: mode m's slots from m * ck_cap
  const int* ckstride;
  const double* gy;          // [nseed, nmode, nout, 20]
  double* gth;               // [nseed, nmode, npar]
  int* status;               // [nseed * nmode]
  double* ws;
  long wslot;
  int seg_cap;
  int* queue;
  const int* order;          // modes, most recorded steps first
  deb::Dims D;
  int level;                 // what of an item's state lives in shared memory (adj_smem_doubles)
};

constexpr int kAdjWarps = 4, kAdjThreads = 32 * kAdjWarps;
using AdjBlk = deb::AdjBlk<kAdjWarps>;

// per-block workspace in global memory, in doubles, after the slot, the
// adjoint vectors and the segment states: theta differences and table sets
constexpr long kThetaLen = (long)deb::NB * 9 * deb::MAXPAR;
constexpr long kSetLen = (long)((2 * deb::MAXPAR * sizeof(deb::SetCtx) + 7) / 8);

// doubles of dynamic shared memory: the scratch, the stages' momentum-bin
// coefficients and, by level, 1: the slot without the stage vectors,
// 2: and the stage vectors, 3: and the NSHV hottest adjoint vectors, 4: and
// all adjoint vectors
long adj_smem_doubles(const deb::Dims& D, int level) {
  long d = deb::SC_LEN + (21L + 48L) * D.nq;
  if (level >= 1) d += deb::hot_len(D);
  if (level >= 2) d += deb::stage_len(D);
  if (level == 3) d += (long)deb::NSHV * D.n;
  if (level == 4) d += (long)deb::NAV * D.n;
  return d;
}

// Two blocks per SM at 254 registers: eight warps of FP64 work hide each
// other's latencies, and a register limit for more spills.  Measured against
// one warp per item (one likelihood gradient from Python): nvar 323, 128 k, 8
// outputs: 935 -> 229 ms; nvar 1098, 96 k, 64 outputs: 799 -> 230 ms.
__global__ void __launch_bounds__(kAdjThreads, 2) adjoint_kernel(AParams P) {
  extern __shared__ double smem[];
  __shared__ __align__(16) unsigned char raw[sizeof(deb::AdjS)];   // no constructor runs
  deb::AdjS& S = *reinterpret_cast<deb::AdjS*>(raw);
  const int tid = threadIdx.x;
  const int n = P.D.n, nq = P.D.nq;
  double* const g = P.ws + (long)blockIdx.x * P.wslot;             // this block's global workspace
  double* const g_av = g + deb::slot_len(P.D);
  double* const g_seg = g_av + (long)deb::NAV * n;
  double* const g_th = g_seg + (long)P.seg_cap * n;
  double* sh = smem;
  double* const sc = sh; sh += deb::SC_LEN;
  double* const vqs = sh; sh += 21 * nq;
  double* const vv = sh; sh += 48 * nq;
  deb::AWS<32> A;
  A.w.n = n;
  A.w.misc0 = deb::V_K0 * n;
  A.w.dp = nullptr;
  A.w.p = P.level >= 1 ? sh : g;
  if (P.level >= 1) sh += deb::hot_len(P.D);
  A.w.kp = P.level >= 2 ? sh : g + deb::hot_len(P.D);
  if (P.level >= 2) sh += deb::stage_len(P.D);
  A.av = P.level == 4 ? sh : g_av;
  A.shv = P.level == 3 ? sh : nullptr;
  A.seg = g_seg;
  A.seg_cap = P.seg_cap;
  A.sc = sc;
  A.n = n;
  deb::Blk<kAdjWarps> B{S.blk, A.w, vqs, P.D, c_rodas, tid, tid >> 5, tid & 31};
  AdjBlk J{S, B, P.D, c_rodas, tid, tid >> 5, tid & 31};
  J.lam = A.vec(deb::A_LAM).p; J.rb = A.vec(deb::A_RB).p; J.rbn = A.vec(deb::A_YOUT).p; J.ub = A.vec(deb::A_UB).p;
  J.yh = A.vec(deb::A_YH).p; J.ye = A.vec(deb::A_YE).p; J.rho = A.vec(deb::A_RHO).p; J.u = A.vec(deb::A_TMP).p;
  J.yo2 = A.vec(deb::A_YO2).p; J.kb = A.vec(deb::A_KB0).p;
  J.vv = vv;
  J.dth = g_th;
  J.dth1 = g_th + (long)deb::NB * 8 * deb::MAXPAR;
  J.sets = reinterpret_cast<deb::SetCtx*>(g_th + kThetaLen);
  B.init_tables(c_tab);
  J.init_lists();
  const long items = (long)P.nmode * P.nseed;
  for (;;) {
    if (tid == 0) S.blk.q = atomicAdd(P.queue, 1);
    __syncthreads();
    const int q = S.blk.q;
    __syncthreads();
    if (q >= items) break;
    const int j = q / P.nseed, seed = q - j * P.nseed;
    const int m = P.order ? P.order[j] : j;
    if (m < 0 || m >= P.nmode) continue;
    const long item = (long)seed * P.nmode + m;
    double* gth = P.gth + item * P.npar;
    const int ci = P.cosmo ? P.cosmo[m] : 0;
    const double km = P.k[m];
    int st = deb::ST_BAD_INPUT;
    deb::AdjItem it;
    if (ci >= 0 && ci < P.ncosmo && km > 0.0 && isfinite(km)) {
      it.blob0 = P.tables + (long)ci * P.blob_len;
      it.blobs = P.tables_pm + (long)ci * 2 * P.npar * P.blob_len;
      it.blob_len = P.blob_len;
      it.npar = P.npar;
      it.eps = P.eps + (long)ci * P.npar;
      it.tau0 = P.tau_out + (long)ci * P.nout;
      it.taus = P.tau_pm + (long)ci * 2 * P.npar * P.nout;
      it.rec = P.rec + (long)m * P.rec_len;
      it.nrec = P.nrec[m];
      it.ck = P.ckpt + (P.ckoff ? (long)P.ckoff[m] : (long)m * P.ck_cap) * n;
      it.ck_stride = it.nrec >= 1 ? P.ckstride[m] : 1;
      it.gy = P.gy + item * P.nout * deb::NFIELD;
      it.k = km;
      if (it.nrec >= 1 && it.nrec <= P.rec_len - 1) st = J.run(it, P.nout, A, g_seg, P.seg_cap, gth);
    }
    if (tid == 0) {
      P.status[item] = st;
      if (st != deb::ST_OK)
        for (int p = 0; p < P.npar; ++p) gth[p] = __longlong_as_double(0x7ff8000000000000LL);
    }
    __syncthreads();
  }
}

// order[rank(i)] = i by key descending (ties by index), as the replay orders its work
__global__ void rank_desc_adj_kernel(const int* key, int n, int* order) {
  __shared__ int tile[256];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int ki = i < n ? key[i] : 0;
  int r = 0;
  for (int base = 0; base < n; base += blockDim.x) {
    const int j = base + (int)threadIdx.x;
    tile[threadIdx.x] = j < n ? key[j] : 0;
    __syncthreads();
    const int lim = n - base < (int)blockDim.x ? n - base : (int)blockDim.x;
    for (int t = 0; t < lim; ++t) {
      const int kj = tile[t];
      r += (kj > ki) || (kj == ki && base + t < i);
    }
    __syncthreads();
  }
  if (i < n) order[r] = i;
}

std::mutex g_adj_mu;
unsigned long long g_adj_ctx[64] = {0};

// constant tables of this translation unit, once per context
int adj_upload_constants() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return DEB_ERR_CUDA;
  unsigned long long ctx = deb_internal::current_ctx_id();
  if (ctx == 0) {
    if (cudaFree(nullptr) != cudaSuccess) return DEB_ERR_CUDA;
    ctx = deb_internal::current_ctx_id();
  }
  std::lock_guard<std::mutex> lock(g_adj_mu);
  if (dev >= 0 && dev < 64 && ctx != 0 && g_adj_ctx[dev] == ctx) return DEB_OK;
  deb::Tab T;
  deb::Rodas R;
  deb::fill_tables(T);
  deb::fill_rodas(R);
  const deb::LeadInv& L = deb::host_linv();
  if (!L.ok) return DEB_ERR_INVALID;
  if (cudaMemcpyToSymbol(c_tab, &T, sizeof(T)) != cudaSuccess) return DEB_ERR_CUDA;
  if (cudaMemcpyToSymbol(c_rodas, &R, sizeof(R)) != cudaSuccess) return DEB_ERR_CUDA;
  if (cudaMemcpyToSymbol(deb::c_linv, &L, sizeof(L)) != cudaSuccess) return DEB_ERR_CUDA;
  if (dev >= 0 && dev < 64) g_adj_ctx[dev] = ctx;
  return DEB_OK;
}

deb_internal::SmemLimit g_adj_smem;

// Launch shape, by the items of the launch (not by the plan's room for them):
// two blocks per SM (the registers' limit) when there are more items than SMs,
// else one, each with the highest shared-memory level that leaves room.  ms with
// one / two per SM on 152 SMs (likelihood gradients of one cosmology): nvar 323
// 171 / 181 at 152 items, 166 / 173 at 153, 168 / 236 at 304, 166 / 229 at 400,
// 247 / 249 at 608; nvar 1098 175 / 198, 174 / 197, 216 / 244, 253 / 253, 389 /
// 308.  Two win where a launch has several items per SM; the line lies low, one
// would still be as fast at up to 2.6.
int adj_launch_blocks(const deb_plan* p, long items) { return (int)(items < p->adj_blocks ? items : p->adj_blocks); }
int adj_two_per_sm(const deb_plan* p, int blocks) { return blocks > p->nsm ? 1 : 0; }

}  // namespace

extern "C" {

int deb_plan_create_adjoint(const deb_dims* dims, int max_items, int seg_cap, deb_plan** out) {
  if (!dims || !out || max_items <= 0 || seg_cap < 1) return DEB_ERR_INVALID;
  *out = nullptr;
  // the lead rows' sources must not alias (lmax >= 5), the scratch block
  // holds up to 64 outputs and 64 momentum bins
  if (dims->lmaxg < 5 || dims->lmaxgp < 5 || dims->lmaxr < 5 || dims->lmaxnu < 3 || dims->nqmax < 1 ||
      dims->nqmax > 64 || dims->nout < 1 || dims->nout > 64)
    return DEB_ERR_INVALID;
  if (dims->lmaxg > deb::LMAX_TABLE || dims->lmaxgp > deb::LMAX_TABLE || dims->lmaxr > deb::LMAX_TABLE ||
      dims->lmaxnu > deb::LMAX_TABLE)
    return DEB_ERR_INVALID;
  if (dims->linear_solver != DEB_SOLVE_STRUCTURED || dims->return_full) return DEB_ERR_INVALID;
  int rc = adj_upload_constants();
  if (rc) return rc;
  int dev = 0, nsm = 0, optin = 0, sm_bytes = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return DEB_ERR_CUDA;
  if (cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sm_bytes, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev) != cudaSuccess)
    return DEB_ERR_CUDA;
  const deb::Dims Dm = deb::make_dims(dims->lmaxg, dims->lmaxgp, dims->lmaxr, dims->lmaxnu, dims->nqmax);
  const long fixed = (long)sizeof(deb::AdjS);
  int level[2];
  long smem[2];
  for (int i = 0; i < 2; ++i) {
    for (level[i] = 4; level[i] > 0; --level[i]) {
      const long bytes = adj_smem_doubles(Dm, level[i]) * (long)sizeof(double);
      if (bytes + fixed <= optin && (i + 1) * (bytes + fixed + 1024) <= sm_bytes) break;
    }
    smem[i] = adj_smem_doubles(Dm, level[i]) * (long)sizeof(double);
    if (smem[i] + fixed > optin) return DEB_ERR_INVALID;
    if (g_adj_smem.raise(adjoint_kernel, smem[i]) != cudaSuccess) return DEB_ERR_CUDA;
  }
  deb_plan* p = new deb_plan();
  for (int i = 0; i < 2; ++i) { p->adj_smem[i] = smem[i]; p->adj_level[i] = level[i]; }
  p->D = deb::make_dims(dims->lmaxg, dims->lmaxgp, dims->lmaxr, dims->lmaxnu, dims->nqmax);
  p->nout = dims->nout;
  p->exec_mode = DEB_EXEC_WARP;
  p->max_modes = max_items;
  p->nsm = nsm;
  p->slot_len = deb::slot_len(p->D);
  p->adj = 1;
  p->adj_seg_cap = seg_cap;
  p->adj_wslot = p->slot_len + (long)(deb::NAV + seg_cap) * p->D.n + kThetaLen + kSetLen;
  p->adj_wslot += p->adj_wslot & 1;
  // blocks in flight: what the SMs hold, capped by the items and by 32 GiB
  long blocks = (long)nsm * 2;
  const long mem_cap = (32L << 30) / (p->adj_wslot * 8);
  if (blocks > mem_cap) blocks = mem_cap;
  if (blocks > max_items) blocks = max_items;
  if (blocks < 1) { delete p; return DEB_ERR_NOMEM; }
  p->adj_blocks = (int)blocks;
  p->ws_bytes = (size_t)blocks * p->adj_wslot * sizeof(double);
  if (cudaMalloc(&p->adj_ws, p->ws_bytes) != cudaSuccess) { delete p; return DEB_ERR_NOMEM; }
  if (cudaMalloc(&p->queue, sizeof(int) * 4) != cudaSuccess) { cudaFree(p->adj_ws); delete p; return DEB_ERR_NOMEM; }
  if (cudaMalloc(&p->order_dev, sizeof(int) * (size_t)max_items) != cudaSuccess) {
    cudaFree(p->adj_ws); cudaFree(p->queue); delete p; return DEB_ERR_NOMEM;
  }
  *out = p;
  return DEB_OK;
}

int deb_adjoint_launch_info(const deb_plan* p, int items, deb_launch_cfg* cfg, int* items_in_flight) {
  if (!p || !p->adj || items < 1 || !cfg || !items_in_flight) return DEB_ERR_INVALID;
  if (items > p->max_modes) return DEB_ERR_CAPACITY;
  const int blocks = adj_launch_blocks(p, items), two = adj_two_per_sm(p, blocks), level = p->adj_level[two];
  cfg->stage_vectors = level >= 2 ? DEB_STAGE_SHARED : level == 1 ? DEB_STAGE_GLOBAL : DEB_STAGE_ALL_GLOBAL;
  cfg->modes_per_sm = 1 + two;
  *items_in_flight = blocks;
  return DEB_OK;
}

int deb_adjoint(deb_plan* p, const double* d_tables, const double* d_tables_pm, int ncosmo, int npar, int blob_len,
                const double* d_eps, const double* d_k, const int* d_cosmo_of_mode, int nmode,
                const double* d_tau_out, const double* d_tau_out_pm, const double* d_record, int rec_len,
                const int* d_nrec, const double* d_ckpt, int ck_cap, const long long* d_ckoff, const int* d_ckstride,
                const double* d_gy, int nseed, double* d_gtheta, int* d_status, void* stream) {
  if (!p || !p->adj || ncosmo <= 0 || npar < 1 || npar > 12 || nmode < 0 || nseed < 1 || blob_len <= deb::HDR_LEN)
    return DEB_ERR_INVALID;
  if (nmode == 0) return DEB_OK;
  if (!d_tables || !d_tables_pm || !d_eps || !d_k || !d_tau_out || !d_tau_out_pm || !d_record || !d_nrec || !d_ckpt ||
      !d_ckstride || !d_gy || !d_gtheta || !d_status || rec_len < 2 || (!d_ckoff && ck_cap < 2))
    return DEB_ERR_INVALID;
  if ((long)nmode * nseed > p->max_modes || nmode > p->max_modes) return DEB_ERR_CAPACITY;
  int rc = adj_upload_constants();
  if (rc) return rc;
  cudaStream_t s = (cudaStream_t)stream;
  AParams P{};
  P.tables = d_tables; P.tables_pm = d_tables_pm; P.ncosmo = ncosmo; P.npar = npar; P.blob_len = blob_len;
  P.eps = d_eps; P.k = d_k; P.cosmo = d_cosmo_of_mode; P.nmode = nmode; P.nseed = nseed; P.nout = p->nout;
  P.tau_out = d_tau_out; P.tau_pm = d_tau_out_pm; P.rec = d_record; P.rec_len = rec_len; P.nrec = d_nrec;
  P.ckpt = d_ckpt; P.ck_cap = ck_cap; P.ckoff = d_ckoff; P.ckstride = d_ckstride; P.gy = d_gy; P.gth = d_gtheta; P.status = d_status;
  P.ws = p->adj_ws; P.wslot = p->adj_wslot; P.seg_cap = p->adj_seg_cap; P.queue = p->queue; P.order = p->order_dev;
  P.D = p->D;
  const long items = (long)nmode * nseed;
  const int blocks = adj_launch_blocks(p, items), two = adj_two_per_sm(p, blocks);
  P.level = p->adj_level[two];
  if (g_adj_smem.raise(adjoint_kernel, p->adj_smem[two]) != cudaSuccess) return DEB_ERR_CUDA;
  if (cudaMemsetAsync(p->queue, 0, sizeof(int), s) != cudaSuccess) return DEB_ERR_CUDA;
  rank_desc_adj_kernel<<<(nmode + 255) / 256, 256, 0, s>>>(d_nrec, nmode, p->order_dev);
  adjoint_kernel<<<blocks, kAdjThreads, (size_t)p->adj_smem[two], s>>>(P);
  return cudaGetLastError() == cudaSuccess ? DEB_OK : DEB_ERR_CUDA;
}

}  // extern "C"
