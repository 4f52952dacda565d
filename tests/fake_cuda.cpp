// The host side of the solver (fim_solver.cpp, included here) over a fake CUDA
// runtime: device memory is host memory under a budget, copies are memcpy, and
// the staging kernels are loops that fill and overwrite what the kernels do.
// For tests of allocation failures and of the route a call takes, which need
// no GPU that way.
#include FIM_SOLVER_CPP

#include <cstdlib>
#include <map>

namespace {
struct Fake {
  size_t budget = ~size_t(0), live = 0, peak = 0;
  std::map<void *, size_t> blocks;
  cudaError_t last = cudaSuccess;
  int d2h = 0, launches = 0;
  int other_device = 0;  // what cudaPointerGetAttributes says of memory that is not in blocks
  const double *metric_fib = nullptr;
} F;
cudaError_t ok() { ++F.launches; return F.last; }  // a launch reports the last error, as the wrappers do
}  // namespace

extern "C" {
cudaError_t cudaMalloc(void **p, size_t n)
{
  *p = nullptr;
  if (n > F.budget || F.live > F.budget - n) return F.last = cudaErrorMemoryAllocation;
  if (!(*p = std::malloc(n))) return F.last = cudaErrorMemoryAllocation;
  std::memset(*p, 0xab, n);
  F.blocks[*p] = n;
  F.live += n;
  F.peak = std::max(F.peak, F.live);
  return cudaSuccess;
}
cudaError_t cudaFree(void *p)
{
  auto it = F.blocks.find(p);
  if (it == F.blocks.end()) std::abort();
  F.live -= it->second;
  F.blocks.erase(it);
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaGetLastError() { const cudaError_t e = F.last; F.last = cudaSuccess; return e; }
const char *cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "error"; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind k, cudaStream_t)
{
  if (k == cudaMemcpyDeviceToHost) ++F.d2h;
  std::memmove(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind k) { return cudaMemcpyAsync(d, s, n, k, nullptr); }
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t) { std::memset(p, v, n); return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p)
{
  *a = cudaPointerAttributes{};
  a->type = cudaMemoryTypeDevice;
  a->device = F.other_device;
  for (const auto &b : F.blocks)
    if (p >= b.first && p < static_cast<const char *>(b.first) + b.second) a->device = 0;
  return cudaSuccess;
}
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { *v = 1; return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = nullptr; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaErrorNotSupported; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *) { return cudaErrorNotSupported; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *, cudaGraph_t, unsigned long long) { return cudaErrorNotSupported; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorNotSupported; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 0.f; return cudaSuccess; }
}

namespace fimgb {

const ShapeDesc kShapes[kNumShapes] = {};
cudaError_t solve_prepare(int, int, int, int *g) { *g = 1; return cudaSuccess; }

template <typename Id>
cudaError_t launch_stage_check(int64_t nV, int64_t nT, const Id *tets, const double *xyz, uint32_t *first,
                               StageCtl *ctl, cudaStream_t)
{
  *ctl = StageCtl{~0ull, ~0ull, ~0ull, 0, 0, 0};
  if (first) std::fill(first, first + nV, ~0u);
  for (int64_t e = 0; e < nT; ++e) {
    Id v[4];
    std::copy(tets + 4 * e, tets + 4 * e + 4, v);
    for (int j = 3; j >= 0; --j)
      if (v[j] < 0 || v[j] >= nV) ctl->bad_id = std::min<unsigned long long>(ctl->bad_id, 4 * e + j);
    std::sort(v, v + 4);
    if (v[0] < 0 || v[3] >= nV) continue;
    if (v[0] == v[1] || v[1] == v[2] || v[2] == v[3]) ctl->bad_tet = std::min<unsigned long long>(ctl->bad_tet, e);
    else if (first)
      for (int j = 0; j < 4; ++j) first[v[j]] = std::min<uint32_t>(first[v[j]], (uint32_t)(4 * e + j));
  }
  for (int64_t i = 0; i < 3 * nV; ++i)
    if (!std::isfinite(xyz[i])) ctl->bad_xyz = std::min<unsigned long long>(ctl->bad_xyz, i);
  return ok();
}
template <typename Id>
cudaError_t launch_stage_slots(int64_t nT, const Id *tets, const uint32_t *first, int32_t *slots, cudaStream_t)
{
  for (int64_t e = 0; e < nT; ++e) {
    std::copy(tets + 4 * e, tets + 4 * e + 4, slots + 4 * e);
    std::sort(slots + 4 * e, slots + 4 * e + 4, [&](int32_t a, int32_t b) { return first[a] < first[b]; });
  }
  return ok();
}
template cudaError_t launch_stage_check(int64_t, int64_t, const int64_t *, const double *, uint32_t *, StageCtl *, cudaStream_t);
template cudaError_t launch_stage_check(int64_t, int64_t, const int32_t *, const double *, uint32_t *, StageCtl *, cudaStream_t);
template cudaError_t launch_stage_slots(int64_t, const int64_t *, const uint32_t *, int32_t *, cudaStream_t);
template cudaError_t launch_stage_slots(int64_t, const int32_t *, const uint32_t *, int32_t *, cudaStream_t);
cudaError_t launch_stage_lists(int64_t nL, int64_t nT, const StageLists &x, StageCtl *, cudaStream_t)
{
  std::vector<std::vector<int32_t>> nb(nL);
  std::vector<int64_t> deg(nL, 0);
  // every buffer that the kernels overwrite, in full
  std::fill(x.cnt, x.cnt + nL, -7);
  std::fill(x.big_list, x.big_list + nL, -7);
  std::fill(x.mark, x.mark + nL, -7);
  std::fill(x.keys, x.keys + 4 * nT, 0x77777777u);
  std::fill(x.scratch, x.scratch + 16 * nT, -7);
  std::fill(x.tile_sum, x.tile_sum + nL, -7);
  for (int64_t e = 0; e < nT; ++e)
    for (int t = 0; t < 4; ++t) {
      const int32_t v = x.cslots[4 * e + t];
      ++deg[v];
      for (int k = 0; k < 4; ++k) nb[v].push_back(x.cslots[4 * e + k]);
    }
  x.cptr[0] = x.nptr[0] = 0;
  for (int64_t v = 0; v < nL; ++v) {
    nb[v].push_back((int32_t)v);
    std::sort(nb[v].begin(), nb[v].end());
    nb[v].erase(std::unique(nb[v].begin(), nb[v].end()), nb[v].end());
    x.cptr[v + 1] = x.cptr[v] + deg[v];
    x.nptr[v + 1] = x.nptr[v] + (int64_t)nb[v].size();
    if (deg[v]) std::copy(nb[v].begin(), nb[v].end(), x.scratch + 4 * x.cptr[v]);
  }
  std::vector<int64_t> fill(x.cptr, x.cptr + nL);
  for (int64_t e = 0; e < nT; ++e)
    for (int t = 0; t < 4; ++t) {
      const int64_t c = fill[x.cslots[4 * e + t]]++;
      x.cidx[4 * e + t] = c;
      for (int w = 0; w < kCrecWords; ++w) x.crec[kCrecWords * c + w] = uint4{(unsigned)e, (unsigned)t, 0u, 0u};
    }
  return ok();
}
cudaError_t launch_stage_compact(int64_t nL, const StageLists &x, int32_t *nbr, cudaStream_t)
{
  for (int64_t v = 0; v < nL; ++v) {
    if (x.cptr[v + 1] == x.cptr[v]) nbr[x.nptr[v]] = (int32_t)v;
    else std::copy(x.scratch + 4 * x.cptr[v], x.scratch + 4 * x.cptr[v] + (x.nptr[v + 1] - x.nptr[v]), nbr + x.nptr[v]);
  }
  return ok();
}
cudaError_t launch_stage_in_tet(int64_t nV, const int64_t *cptr, uint8_t *in_tet, cudaStream_t)
{
  for (int64_t v = 0; v < nV; ++v) in_tet[v] = cptr[v + 1] > cptr[v];
  return ok();
}
cudaError_t launch_edge_vectors(const int32_t *slots, const double *xyz, int64_t nT, double *evec, StageCtl *ctl,
                                cudaStream_t)
{
  double m;
  std::memcpy(&m, &ctl->max_edge2, sizeof m);
  for (int64_t e = 0; e < nT; ++e)
    for (int i = 0; i < 4; ++i)
      for (int j = 0; j < i; ++j) {
        double l = 0.0;
        for (int a = 0; a < 3; ++a) {
          const double d = xyz[3 * (int64_t)slots[4 * e + i] + a] - xyz[3 * (int64_t)slots[4 * e + j] + a];
          l += d * d;
        }
        m = std::max(m, l);
      }
  std::memcpy(&ctl->max_edge2, &m, sizeof m);
  if (evec) std::fill(evec, evec + 18 * nT, 1.0);
  return ok();
}
cudaError_t launch_metric(const int32_t *, const int64_t *, const double *, const double *, int64_t, const double *fib,
                          const double *, const double *, int64_t, int64_t, double *, float *, uint4 *,
                          unsigned long long *, cudaStream_t)
{
  F.metric_fib = fib;
  return ok();
}
cudaError_t launch_solve(const FimDev &d, const FimParams &, int, int, int, cudaStream_t)
{
  const int64_t n = d.gptr ? d.nG : d.nV;
  double *phi = d.gptr ? d.phi_out : d.phi;
  uint8_t *st = d.gptr ? d.st_out : d.st;
  for (int64_t v = 0; v < n; ++v) { phi[v] = 0.5 * (double)v; st[v] = (uint8_t)(v % 6); }
  ++F.launches;
  return cudaSuccess;  // (cudaLaunchKernelEx returns its own status)
}
cudaError_t launch_widen(const uint8_t *s, int32_t *d, int64_t n, cudaStream_t) { std::copy(s, s + n, d); return ok(); }
cudaError_t launch_copy(const double *s, double *d, int64_t n, cudaStream_t) { std::copy(s, s + n, d); return ok(); }
cudaError_t launch_support_check(const FimDev &, double, const uint8_t *, cudaStream_t) { return ok(); }
cudaError_t launch_mark_seeds(const FimDev &, uint8_t *, cudaStream_t) { return ok(); }
cudaError_t launch_warm_reset(const FimDev &, double, cudaStream_t) { return ok(); }
cudaError_t noalloc_scratch(int, NoallocScratch *) { return cudaErrorNotSupported; }
cudaError_t launch_noalloc_seeds(const NoallocScratch &, int32_t, const int64_t *, const int32_t *, const int64_t *, cudaStream_t) { return ok(); }
size_t features_scratch(int nV) { return (size_t)nV; }
float features_scale(const unsigned int *) { return 0.f; }
cudaError_t launch_features(int, int64_t, const double *, const int32_t *, const double *, const double *, const double *, int,
                            const int32_t *, const double *, float *, unsigned int **, void *, cudaStream_t) { return ok(); }

}  // namespace fimgb

// what the tests set and read
extern "C" {
void fake_budget(size_t b) { F.budget = b; F.peak = F.live; }
size_t fake_live() { return F.live; }
size_t fake_peak() { return F.peak; }
int fake_d2h() { const int n = F.d2h; F.d2h = 0; return n; }
void fake_other_device(int d) { F.other_device = d; }
int fake_metric_reads(const double *p) { return F.metric_fib == p; }
size_t fake_bytes(const fim_solver *s, int k)
{
  const size_t b[4] = {s->stage.n, s->arena.n, s->nbr.n * sizeof(int32_t), s->evec.n * sizeof(double)};
  return b[k];
}
double fake_front_width(const fim_solver *s) { return s->front_width; }
// the staged lists, in one order: slots, corner offsets and indices, records, neighbourhoods, coordinates, seeds' flags
void fake_lists(const fim_solver *s, unsigned long long *sum)
{
  unsigned long long h = 1469598103934665603ull;
  const auto add = [&](const void *p, size_t n) {
    for (size_t i = 0; i < n; ++i) h = (h ^ static_cast<const unsigned char *>(p)[i]) * 1099511628211ull;
  };
  add(s->tslots.p, sizeof(int32_t) * 4 * s->nT);
  add(s->cptr.p, sizeof(int64_t) * (s->nL + 1));
  add(s->cidx.p, sizeof(int64_t) * s->nC);
  add(s->crec.p, sizeof(uint4) * kCrecWords * s->nC);
  add(s->nptr.p, sizeof(int64_t) * (s->nL + 1));
  add(s->nbr.p, sizeof(int32_t) * s->nptr.p[s->nL]);
  add(s->xyz.p, sizeof(double) * 3 * s->nV);
  add(s->in_tet.data(), s->in_tet.size());
  if (s->gptr.p) { add(s->gptr.p, sizeof(int64_t) * (s->nV + 1)); add(s->gcopy.p, sizeof(int32_t) * s->nL); }
  *sum = h;
}
}
