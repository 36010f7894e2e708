// salsa_chain.cu -- the kernels of the gradient harness that advance the state, and its C-ABI.
//
// They keep the plain operations and CUDA's functions: over many steps the condensation
// magnifies a last-bit difference by orders of magnitude.
#define SALSA_MATH_PLAIN
#include "salsa_chain_impl.cuh"

namespace salsa {
// the kernels of salsa_chain_taped.cu and salsa_chain_rev.cu
const void *chain_taped_entry();
const void *chain_rev_entry();
}  // namespace salsa

// =======================================================================================
// C-ABI entry points of the chain
// =======================================================================================
namespace {
using salsa::DevParams;
using salsa::ChainArgs;

int chain_params(salsa_handle_t *h, const salsa_chain_t *c, DevParams *P, ChainArgs *A, cudaStream_t *st, void *stream,
                 int *nsm) {
  int dev = 0;
  cudaStream_t hs;
  if (!h || !c || !salsa::handle_params(h, P, &hs, &dev, nsm)) return SALSA_E_ARG;
  const salsa_config_t *g = salsa::handle_config(h);
  if (g->level != 4) return SALSA_E_UNSUPPORTED;
  if (c->ncell <= 0 || c->nsub <= 0 || !(c->dt > 0.) || c->dt > 1.2) return SALSA_E_ARG;
  if (!c->temp || !c->press || !c->rs || !c->dn || !c->kappa || !c->ssat) return SALSA_E_ARG;
  if (cudaSetDevice(dev) != cudaSuccess) return SALSA_E_NODEV;
  *st = stream ? (cudaStream_t)stream : hs;
  P->level = 4; P->lcharge = 0; P->initialize = 0; P->dt = c->dt; P->has_kappa = 1;
  P->lscgaa = g->lscgaa; P->lscgcc = g->lscgcc; P->lscgca = g->lscgca; P->lscgpc = g->lscgpc; P->lscgpa = g->lscgpa;
  P->lscgpp = g->lscgpp; P->lscgia = P->lscgic = P->lscgii = P->lscgip = 0;
  P->lscndh2oae = g->lscndh2oae; P->lscndh2ocl = g->lscndh2ocl; P->lscndh2oic = 0;
  memset(A, 0, sizeof *A);
  A->ncell = c->ncell; A->nsub = c->nsub; A->dt = c->dt;
  A->NL = P->nliquid; A->NW = P->nwet; A->nstate = A->NL * (1 + A->NW); A->n1a = P->fn1a - P->in1a + 1;
  A->temp = c->temp; A->press = c->press; A->rs = c->rs; A->dn = c->dn; A->kappa = c->kappa; A->ssat = c->ssat;
  A->every = 1;
  unsigned long long *err = (unsigned long long *)salsa::handle_scratch(h, 3, 64);
  if (!err) return SALSA_E_CUDA;
  A->err = err;
  if (cudaMemsetAsync(err, 0, sizeof(unsigned long long), *st) != cudaSuccess) return SALSA_E_CUDA;
  return SALSA_OK;
}

template <typename R>
int ws_doubles(int NL, int NW) {
  return (int)(((size_t)salsa::chain_ws_entries(NL, NW) * sizeof(R) + 7) / 8) + 32;
}

template <typename K>
int launch_chain(K kernel, const DevParams &P, const ChainArgs &A, cudaStream_t st, int nsm, int wpb) {
  size_t smem = sizeof(double) * ((size_t)P.tab_doubles + (size_t)wpb * A.ws_doubles);
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    return SALSA_E_CUDA;
  int bps = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, kernel, 32 * wpb, smem) != cudaSuccess || bps <= 0)
    return SALSA_E_CUDA;
  long long grid = (long long)bps * nsm * 4;
  long long need = (A.ncell + wpb - 1) / wpb;
  if (grid > need) grid = need;
  kernel<<<(int)grid, 32 * wpb, smem, st>>>(P, A);
  return cudaGetLastError() == cudaSuccess ? SALSA_OK : SALSA_E_CUDA;
}

int chain_finish(const ChainArgs &A, cudaStream_t st) {
  unsigned long long nerr = 0;
  if (cudaMemcpyAsync(&nerr, A.err, sizeof nerr, cudaMemcpyDeviceToHost, st) != cudaSuccess) return SALSA_E_CUDA;
  if (cudaStreamSynchronize(st) != cudaSuccess) return SALSA_E_CUDA;
  return nerr ? SALSA_E_NUMERIC : SALSA_OK;
}
}  // namespace

extern "C" {

int salsa_gb300_chain_state_size(const salsa_handle_t *h) {
  DevParams P;
  cudaStream_t s;
  int dev, nsm;
  if (!salsa::handle_params(h, &P, &s, &dev, &nsm)) return 0;
  return salsa::handle_config(h)->level == 4 ? P.nliquid * (1 + P.nwet) : 0;
}

long long salsa_gb300_chain_adjoint_bytes(const salsa_handle_t *h, int ncell, int nsub, double dt,
                                          int ckpt_every) {
  DevParams P;
  cudaStream_t s;
  int dev, nsm;
  if (!salsa::handle_params(h, &P, &s, &dev, &nsm) || salsa::handle_config(h)->level != 4) return -1;
  if (ncell <= 0 || nsub <= 0 || ckpt_every <= 0 || !(dt > 0.)) return -1;
  const long long ns = (long long)P.nliquid * (1 + P.nwet);
  const salsa::TapeLayout tl = salsa::tape_layout(P.nliquid, P.nwet, P.fn1a - P.in1a + 1, salsa::tape_maxit(dt));
  const long long nseg = (nsub + ckpt_every - 1) / ckpt_every;
  long long d = nseg * ncell * ns + (long long)ncell * tl.total;   // checkpoints, tape
  if (ckpt_every > 1) d += (long long)ckpt_every * ncell * ns;      // states of one segment
  return d * (long long)sizeof(double) + (nseg + 2LL * nsub) * (long long)sizeof(unsigned) + 64;
}

int salsa_gb300_chain_forward(salsa_handle_t *h, const salsa_chain_t *c, const double *x0, double *xN, double *ckpt,
                              int ckpt_every, void *stream) {
  DevParams P;
  ChainArgs A;
  cudaStream_t st;
  int nsm = 0;
  int rc = chain_params(h, c, &P, &A, &st, stream, &nsm);
  if (rc) return rc;
  if (!x0 || !xN || (ckpt && ckpt_every <= 0)) return SALSA_E_ARG;
  A.x0 = x0; A.xN = xN; A.ckpt = ckpt; A.every = ckpt ? ckpt_every : 1;
  A.ws_doubles = ws_doubles<double>(A.NL, A.NW);
  rc = launch_chain(salsa::chain_fwd_kernel<double, false>, P, A, st, nsm, 4);
  if (rc) return rc;
  return chain_finish(A, st);
}

int salsa_gb300_chain_tlm(salsa_handle_t *h, const salsa_chain_t *c, const double *x0, const double *dx0,
                          const double *dkappa, const double *dssat, double *xN, double *dxN, void *stream) {
  DevParams P;
  ChainArgs A;
  cudaStream_t st;
  int nsm = 0;
  int rc = chain_params(h, c, &P, &A, &st, stream, &nsm);
  if (rc) return rc;
  if (!x0 || !xN || !dxN) return SALSA_E_ARG;
  A.x0 = x0; A.xN = xN; A.dx0 = dx0; A.dkappa = dkappa; A.dssat = dssat; A.dxN = dxN;
  A.ws_doubles = ws_doubles<salsa::Dual<1>>(A.NL, A.NW);
  rc = launch_chain(salsa::chain_fwd_kernel<salsa::Dual<1>, true>, P, A, st, nsm, 4);
  if (rc) return rc;
  return chain_finish(A, st);
}

int salsa_gb300_chain_adjoint(salsa_handle_t *h, const salsa_chain_t *c, const double *ckpt, int ckpt_every,
                              const double *xbarN, double *xbar0, double *kappabar, double *ssatbar, void *stream) {
  DevParams P;
  ChainArgs A;
  cudaStream_t st;
  int nsm = 0;
  int rc = chain_params(h, c, &P, &A, &st, stream, &nsm);
  if (rc) return rc;
  if (!ckpt || ckpt_every <= 0 || !xbarN || !xbar0 || !kappabar || !ssatbar) return SALSA_E_ARG;
  A.ckpt = const_cast<double *>(ckpt); A.every = ckpt_every;
  A.xbarN = xbarN; A.xbar0 = xbar0; A.kappabar = kappabar; A.ssatbar = ssatbar;
  const int NL = A.NL, NW = A.NW, ns = A.nstate, wpb = 4;
  const salsa::TapeLayout tl = salsa::tape_layout(NL, NW, A.n1a, salsa::tape_maxit(A.dt));
  A.tape = (double *)salsa::handle_scratch(h, 0, (size_t)A.ncell * tl.total * sizeof(double));
  A.seg = ckpt_every > 1
              ? (double *)salsa::handle_scratch(h, 1, (size_t)ckpt_every * A.ncell * ns * sizeof(double))
              : nullptr;
  if (!A.tape || (ckpt_every > 1 && !A.seg)) return SALSA_E_CUDA;
  // one work counter per launch: segment recomputes, then a taped and a reverse step each
  const int nseg = (A.nsub + A.every - 1) / A.every;
  const size_t nctr = (size_t)nseg + 2 * (size_t)A.nsub;
  unsigned *ctr = (unsigned *)salsa::handle_scratch(h, 2, nctr * sizeof(unsigned));
  if (!ctr || cudaMemsetAsync(ctr, 0, nctr * sizeof(unsigned), st) != cudaSuccess) return SALSA_E_CUDA;
  // per-kernel shared memory (doubles per warp) and grids
  const int ws_fwd = salsa::chain_ws_entries(NL, NW) + 32;
  const int ws_tap = ws_fwd + 9 * NL;
  const int ws_rev = ns + 6 * NL + salsa::adj_ws_doubles(NL, NW) + ns + salsa::chain_tri(NL);
  auto config = [&](const void *kernel, int wsd, int *grid, size_t *smem) -> bool {
    *smem = sizeof(double) * ((size_t)P.tab_doubles + (size_t)wpb * wsd);
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)*smem) != cudaSuccess)
      return false;
    int bps = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, kernel, 32 * wpb, *smem) != cudaSuccess || bps <= 0)
      return false;
    long long g = (long long)bps * nsm, need = (A.ncell + wpb - 1) / wpb;
    *grid = (int)(g < need ? g : need);
    return true;
  };
  int g_seg = 0, g_tap = 0, g_rev = 0;
  size_t s_seg = 0, s_tap = 0, s_rev = 0;
  if (!config((const void *)salsa::chain_seg_kernel, ws_fwd, &g_seg, &s_seg) ||
      !config(salsa::chain_taped_entry(), ws_tap, &g_tap, &s_tap) ||
      !config(salsa::chain_rev_entry(), ws_rev, &g_rev, &s_rev))
    return SALSA_E_CUDA;
  salsa::chain_adj_units<<<4 * nsm, 256, 0, st>>>(P, A, 1);
  for (int sg = nseg - 1; sg >= 0; sg--) {
    const int k0 = sg * A.every, k1 = A.nsub < k0 + A.every ? A.nsub : k0 + A.every;
    if (k1 - k0 > 1) {
      A.ws_doubles = ws_fwd;
      salsa::chain_seg_kernel<<<g_seg, 32 * wpb, s_seg, st>>>(P, A, sg, ctr + sg);
    }
    for (int k = k1 - 1; k >= k0; k--) {
      const double *src = k == k0 ? A.ckpt + (size_t)sg * A.ncell * ns : A.seg + (size_t)(k - k0) * A.ncell * ns;
      A.ws_doubles = ws_tap;
      unsigned *c_k = ctr + nseg + 2 * k;
      void *tap_args[] = {&P, &A, &src, &c_k};
      if (cudaLaunchKernel(salsa::chain_taped_entry(), dim3(g_tap), dim3(32 * wpb), tap_args, s_tap, st) != cudaSuccess)
        return SALSA_E_CUDA;
      A.ws_doubles = ws_rev;
      unsigned *c_r = c_k + 1;
      void *rev_args[] = {&P, &A, &c_r};
      if (cudaLaunchKernel(salsa::chain_rev_entry(), dim3(g_rev), dim3(32 * wpb), rev_args, s_rev, st) != cudaSuccess)
        return SALSA_E_CUDA;
    }
  }
  salsa::chain_adj_units<<<4 * nsm, 256, 0, st>>>(P, A, 0);
  if (cudaGetLastError() != cudaSuccess) return SALSA_E_CUDA;
  return chain_finish(A, st);
}

}  // extern "C"
