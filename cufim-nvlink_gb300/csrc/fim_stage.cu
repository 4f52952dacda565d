// fim_stage.cu -- mesh staging on the device (fim_set_mesh): checks of the
// tets, the reference's slot order of a mesh with one submesh, corner lists
// and first-read records, vertex neighbourhoods, edge vectors.
//
// The staging is a handful of passes over the tets and vertices, bound by
// scattered 4- to 32-byte accesses that the 129 MB L2 mostly serves.  On
// the host (loops over tets, of which only the neighbourhoods ran on several
// threads) fim_set_mesh took 49.8 ms for a 135k-vertex slab and 420 ms for a
// 1.03M-vertex one, 18 times the solve itself; here, with one allocation for
// the per-mesh arrays instead of 35, it takes 0.67 ms for the former, of
// which 0.2 ms are the upload.
#include "fim_internal.h"

#include <climits>

namespace fimgb {

namespace {

constexpr int kStageThreads = 256;

unsigned stage_grid(int64_t n, int per_block)
{
  int64_t g = (n + per_block - 1) / per_block;
  if (g < 1) g = 1;
  return (unsigned)(g > 152 * 32 ? 152 * 32 : g);
}

__device__ __forceinline__ void cswap(int &a, int &b)
{
  const int lo = min(a, b), hi = max(a, b);
  a = lo; b = hi;
}
__device__ __forceinline__ void cswap_by(uint32_t &ka, int &a, uint32_t &kb, int &b)
{
  if (kb < ka) {
    const uint32_t k = ka; ka = kb; kb = k;
    const int t = a; a = b; b = t;
  }
}

// The four ids of tet e, of 64 or 32 bits.
__device__ __forceinline__ void load_ids(const int64_t *tets, int64_t e, long long *id)
{
  const longlong2 *p = reinterpret_cast<const longlong2 *>(tets);
  const longlong2 a = __ldg(p + 2 * e), b = __ldg(p + 2 * e + 1);
  id[0] = a.x; id[1] = a.y; id[2] = b.x; id[3] = b.y;
}
__device__ __forceinline__ void load_ids(const int32_t *tets, int64_t e, long long *id)
{
  const int4 a = __ldg(reinterpret_cast<const int4 *>(tets) + e);
  id[0] = a.x; id[1] = a.y; id[2] = a.z; id[3] = a.w;
}

// Tets: every id in [0, nV), no vertex twice; the first offender of each
// kind goes to ctl.  first[v] receives the smallest 4 e + (position of v
// among tet e's ids in ascending order): the order of first appearance by
// which the reference numbers a submesh's vertices (types.cpp:331-345).
template <typename Id>
__global__ void check_tets_kernel(int64_t nV, int64_t nT, const Id *__restrict__ tets, uint32_t *first, StageCtl *ctl)
{
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < nT; e += (int64_t)gridDim.x * blockDim.x) {
    long long id[4];
    load_ids(tets, e, id);
    bool in = true;
#pragma unroll
    for (int j = 3; j >= 0; --j)
      if (id[j] < 0 || id[j] >= nV) {
        in = false;
        atomicMin(&ctl->bad_id, (unsigned long long)(4 * e + j));
      }
    if (!in) continue;
    int v[4] = {(int)id[0], (int)id[1], (int)id[2], (int)id[3]};
    cswap(v[0], v[1]); cswap(v[2], v[3]); cswap(v[0], v[2]); cswap(v[1], v[3]); cswap(v[1], v[2]);
    if (v[0] == v[1] || v[1] == v[2] || v[2] == v[3]) {
      atomicMin(&ctl->bad_tet, (unsigned long long)e);
      continue;
    }
    if (first) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t key = (uint32_t)(4 * e + j);
        if (__ldcg(first + v[j]) > key) atomicMin(first + v[j], key);
      }
    }
  }
}

__global__ void check_xyz_kernel(int64_t n, const double *__restrict__ xyz, StageCtl *ctl)
{
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    if (((unsigned long long)__double_as_longlong(xyz[i]) & 0x7ff0000000000000ull) == 0x7ff0000000000000ull)
      atomicMin(&ctl->bad_xyz, (unsigned long long)i);
}

// One submesh: the slots of every tet are its ids in the order of first
// appearance (types.cpp:383-398, 473).
template <typename Id>
__global__ void slots_kernel(int64_t nT, const Id *__restrict__ tets, const uint32_t *__restrict__ first,
                             int4 *__restrict__ slots)
{
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < nT; e += (int64_t)gridDim.x * blockDim.x) {
    long long id[4];
    load_ids(tets, e, id);
    int v[4] = {(int)id[0], (int)id[1], (int)id[2], (int)id[3]};
    uint32_t k[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) k[j] = __ldg(first + v[j]);
    cswap_by(k[0], v[0], k[1], v[1]); cswap_by(k[2], v[2], k[3], v[3]);
    cswap_by(k[0], v[0], k[2], v[2]); cswap_by(k[1], v[1], k[3], v[3]);
    cswap_by(k[1], v[1], k[2], v[2]);
    slots[e] = make_int4(v[0], v[1], v[2], v[3]);
  }
}

__global__ void count_corners_kernel(int64_t nC, const int32_t *__restrict__ cslots, int32_t *cnt)
{
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nC; i += (int64_t)gridDim.x * blockDim.x)
    atomicAdd(cnt + __ldg(cslots + i), 1);
}

// Exclusive prefix sums of n int32 counts into n + 1 int64 offsets, in three
// launches: sums of kScanTile counts per block, their prefix in one block,
// the prefix inside every tile.
constexpr int kScanThreads = 256, kScanItems = 16, kScanTile = kScanThreads * kScanItems;

// inclusive prefix of x over the block (kScanThreads threads)
__device__ __forceinline__ long long block_scan(long long x, long long *wsum)
{
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const long long u = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += u;
  }
  if (lane == 31) wsum[w] = x;
  __syncthreads();
  for (int k = 0; k < w; ++k) x += wsum[k];
  __syncthreads();
  return x;
}

__global__ void __launch_bounds__(kScanThreads) scan_sums_kernel(int64_t n, const int32_t *__restrict__ cnt,
                                                                 long long *tile_sum)
{
  __shared__ long long wsum[kScanThreads / 32];
  const int64_t i0 = blockIdx.x * (int64_t)kScanTile;
  long long s = 0;
  for (int k = 0; k < kScanItems; ++k) {
    const int64_t i = i0 + k * kScanThreads + threadIdx.x;
    if (i < n) s += cnt[i];
  }
  s = block_scan(s, wsum);
  if (threadIdx.x == kScanThreads - 1) tile_sum[blockIdx.x] = s;
}

__global__ void __launch_bounds__(kScanThreads) scan_tiles_kernel(int tiles, long long *tile_sum)
{
  __shared__ long long wsum[kScanThreads / 32];
  __shared__ long long carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int i0 = 0; i0 < tiles; i0 += kScanThreads) {
    const int i = i0 + threadIdx.x;
    const long long x = i < tiles ? tile_sum[i] : 0;
    const long long inc = block_scan(x, wsum), base = carry;
    if (i < tiles) tile_sum[i] = base + inc - x;
    __syncthreads();
    if (threadIdx.x == kScanThreads - 1) carry = base + inc;
    __syncthreads();
  }
}

__global__ void __launch_bounds__(kScanThreads) scan_apply_kernel(int64_t n, const int32_t *__restrict__ cnt,
                                                                  const long long *__restrict__ tile_sum,
                                                                  int64_t *__restrict__ out)
{
  __shared__ long long wsum[kScanThreads / 32];
  const int64_t i0 = blockIdx.x * (int64_t)kScanTile + threadIdx.x * kScanItems;
  int32_t c[kScanItems];
  long long s = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    c[k] = i0 + k < n ? cnt[i0 + k] : 0;
    s += c[k];
  }
  long long x = tile_sum[blockIdx.x] + block_scan(s, wsum) - s;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    if (i0 + k < n) out[i0 + k] = x;
    x += c[k];
    if (i0 + k == n - 1) out[n] = x;
  }
}

// Corner keys 4 e + t in the run of their vertex copy, in any order
// (lists_kernel sorts each run); cur counts every run down to 0.
__global__ void fill_corners_kernel(int64_t nC, const int32_t *__restrict__ cslots, const int64_t *__restrict__ cptr,
                                    int32_t *cur, uint32_t *__restrict__ keys)
{
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nC; i += (int64_t)gridDim.x * blockDim.x) {
    const int32_t v = __ldg(cslots + i);
    keys[__ldg(cptr + v) + atomicSub(cur + v, 1) - 1] = (uint32_t)i;
  }
}

// Per vertex copy, one warp: its corners in increasing tet index (ids of the
// first-read records, corner index of every slot) and its neighbourhood,
// sorted and with the copy itself.  The neighbour candidates (three per
// corner) are sorted in the warp's part of shared memory (a bitonic sort of
// the next power of two); a copy with more than kListCorners corners, rare
// in a tetrahedral mesh (about 24 corners each), goes to big_list instead.
// The neighbourhood is written to scratch at 4 cptr[v] (it has at most
// 3 deg + 1 <= 4 deg entries) and its length to ncnt; compact_kernel moves it.
constexpr int kListWarps = 8, kListCap = 1024, kListCorners = (kListCap - 1) / 3;
constexpr int kSortMax = 2048;  // longer corner runs stay in the order of the fill (the solve takes any)

__global__ void __launch_bounds__(32 * kListWarps) lists_kernel(int64_t nL, const int4 *__restrict__ cslots,
                                                                const int64_t *__restrict__ cptr,
                                                                const uint32_t *__restrict__ keys, uint4 *__restrict__ crec,
                                                                int64_t *__restrict__ cidx, int32_t *__restrict__ scratch,
                                                                int32_t *__restrict__ ncnt, int32_t *big_list, StageCtl *ctl)
{
  __shared__ int32_t s_cand[kListWarps][kListCap];
  const int lane = threadIdx.x & 31;
  int32_t *cand = s_cand[threadIdx.x >> 5];
  const int64_t stride = (int64_t)gridDim.x * kListWarps;
  for (int64_t v = blockIdx.x * (int64_t)kListWarps + (threadIdx.x >> 5); v < nL; v += stride) {
    const int64_t c0 = __ldg(cptr + v);
    const int64_t deg64 = __ldg(cptr + v + 1) - c0;
    const int deg = (int)deg64;
    const bool small = deg <= kListCorners;
    const bool sort = deg <= kSortMax;
    for (int i0 = 0; i0 < deg; i0 += 32) {
      const int i = i0 + lane;
      const uint32_t key = i < deg ? __ldg(keys + c0 + i) : 0xffffffffu;
      int rank = sort ? 0 : i;
      if (sort)
        for (int j0 = 0; j0 < deg; j0 += 32) {
          const uint32_t o = j0 == i0 ? key : (j0 + lane < deg ? __ldg(keys + c0 + j0 + lane) : 0xffffffffu);
          const int m = min(32, deg - j0);
          for (int j = 0; j < m; ++j) rank += __shfl_sync(0xffffffffu, o, j) < key ? 1 : 0;
        }
      if (i < deg) {
        const uint32_t e = key >> 2, t = key & 3u;
        const int4 s = __ldg(cslots + e);
        // the other slots t+1, t+2, t+3 (mod 4)
        const int a = t == 0 ? s.y : (t == 1 ? s.z : (t == 2 ? s.w : s.x));
        const int b = t == 0 ? s.z : (t == 1 ? s.w : (t == 2 ? s.x : s.y));
        const int c = t == 0 ? s.w : (t == 1 ? s.x : (t == 2 ? s.y : s.z));
        uint4 *r = crec + kCrecWords * (c0 + rank);
        r[0] = make_uint4((unsigned)a, (unsigned)b, (unsigned)c, 0u);
        r[1] = make_uint4(0u, 0u, 0u, 0u);
        cidx[key] = c0 + rank;
        if (small) { cand[3 * i] = a; cand[3 * i + 1] = b; cand[3 * i + 2] = c; }
      }
    }
    if (deg == 0) {
      if (lane == 0) ncnt[v] = 1;
      continue;
    }
    if (!small) {
      if (lane == 0) big_list[atomicAdd(&ctl->n_big, 1)] = (int32_t)v;
      continue;
    }
    const int n = 3 * deg + 1;
    int np = 32;
    while (np < n) np <<= 1;
    for (int i = n - 1 + lane; i < np; i += 32) cand[i] = i == n - 1 ? (int)v : INT_MAX;
    __syncwarp();
    for (int k = 2; k <= np; k <<= 1)
      for (int j = k >> 1; j > 0; j >>= 1) {
        for (int p = lane; p < (np >> 1); p += 32) {
          const int i = 2 * p - (p & (j - 1)), q = i + j;
          const int x = cand[i], y = cand[q];
          if ((x > y) == ((i & k) == 0)) { cand[i] = y; cand[q] = x; }
        }
        __syncwarp();
      }
    int m = 0;
    for (int i0 = 0; i0 < n; i0 += 32) {
      const int i = i0 + lane;
      const int x = i < n ? cand[i] : INT_MAX;
      const bool keep = i < n && (i == 0 || cand[i - 1] != x);
      const unsigned msk = __ballot_sync(0xffffffffu, keep);
      if (keep) scratch[4 * c0 + m + __popc(msk & ((1u << lane) - 1u))] = x;
      m += __popc(msk);
    }
    if (lane == 0) ncnt[v] = m;
    __syncwarp();  // the next copy overwrites the candidates
  }
}

// Neighbourhoods of the copies with very many corners: one block, one copy
// after another, duplicates found by a stamp per copy (their order is that
// of the appends; the marking takes any).
__global__ void __launch_bounds__(1024) big_lists_kernel(int64_t nL, const int4 *__restrict__ cslots,
                                                         const int64_t *__restrict__ cptr,
                                                         const uint32_t *__restrict__ keys, int32_t *__restrict__ scratch,
                                                         int32_t *__restrict__ ncnt, const int32_t *__restrict__ big_list,
                                                         int32_t *mark, const StageCtl *__restrict__ ctl)
{
  const int nb = ctl->n_big;
  if (nb == 0) return;
  __shared__ int s_n;
  for (int64_t v = threadIdx.x; v < nL; v += blockDim.x) mark[v] = -1;
  for (int b = 0; b < nb; ++b) {
    const int32_t v = big_list[b];
    const int64_t c0 = cptr[v], deg = cptr[v + 1] - c0;
    if (threadIdx.x == 0) s_n = 0;
    __syncthreads();
    for (int64_t i = threadIdx.x; i < deg; i += blockDim.x) {
      const int4 s = __ldg(cslots + (keys[c0 + i] >> 2));  // the copy itself among them
      const int u[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (atomicExch(mark + u[k], v) != v) scratch[4 * c0 + atomicAdd(&s_n, 1)] = u[k];
    }
    __syncthreads();
    if (threadIdx.x == 0) ncnt[v] = s_n;
    __syncthreads();
  }
}

__global__ void compact_kernel(int64_t nL, const int64_t *__restrict__ cptr, const int64_t *__restrict__ nptr,
                               const int32_t *__restrict__ scratch, int32_t *__restrict__ nbr)
{
  const int sub = threadIdx.x & 15;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x / 16;
  for (int64_t v = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / 16; v < nL; v += stride) {
    const int64_t a = __ldg(nptr + v), n = __ldg(nptr + v + 1) - a;
    const int64_t c0 = __ldg(cptr + v);
    const bool alone = __ldg(cptr + v + 1) == c0;
    for (int64_t i = sub; i < n; i += 16) nbr[a + i] = alone ? (int32_t)v : __ldg(scratch + 4 * c0 + i);
  }
}

__global__ void in_tet_kernel(int64_t nV, const int64_t *__restrict__ cptr, uint8_t *__restrict__ in_tet)
{
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < nV; v += (int64_t)gridDim.x * blockDim.x)
    in_tet[v] = cptr[v + 1] > cptr[v] ? 1 : 0;
}

// Edge vectors of every tet in the metric kernel's edge order, x_a - x_b
// for (a, b) = (0,1) (0,2) (1,2) (0,3) (1,3) (2,3) of its slots
// (load_edge, types.h:210-216): they depend on the mesh only, so
// fim_set_mesh stages them once and every conduction upload saves their 18
// FP64 subtractions per tet.  Layout: evec[(3 k + axis) nT + e] (nullptr:
// not stored).  The largest squared edge length goes to ctl (the
// reference's front width, compute_dwf, cuda_fim.h:1536-1576).
__global__ void __launch_bounds__(kStageThreads) edge_vector_kernel(const int4 *__restrict__ tslots,
                                                                    const double *__restrict__ xyz, int64_t nT,
                                                                    double *__restrict__ evec, StageCtl *ctl)
{
  double m = 0.0;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < nT; e += (int64_t)gridDim.x * blockDim.x) {
    const int4 s = __ldg(tslots + e);
    const int32_t va[6] = {s.x, s.x, s.y, s.x, s.y, s.z};
    const int32_t vb[6] = {s.y, s.z, s.z, s.w, s.w, s.w};
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      double x[3];
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        x[a] = __ldg(xyz + 3 * (int64_t)va[k] + a) - __ldg(xyz + 3 * (int64_t)vb[k] + a);
        if (evec) evec[(3 * k + a) * nT + e] = x[a];
      }
      const double l = x[0] * x[0] + x[1] * x[1] + x[2] * x[2];
      // non-negative: the order of the bit patterns is that of the values
      if (__double_as_longlong(l) > __double_as_longlong(m)) m = l;
    }
  }
  unsigned long long b = (unsigned long long)__double_as_longlong(m);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) b = max(b, __shfl_xor_sync(0xffffffffu, b, o));
  __shared__ unsigned long long s_b[kStageThreads / 32];
  if ((threadIdx.x & 31) == 0) s_b[threadIdx.x >> 5] = b;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kStageThreads / 32; ++w) b = max(b, s_b[w]);
    atomicMax(&ctl->max_edge2, b);
  }
}

cudaError_t scan(int64_t n, const int32_t *cnt, int64_t *out, long long *tile_sum, cudaStream_t st)
{
  const int64_t tiles = (n + kScanTile - 1) / kScanTile;
  scan_sums_kernel<<<(unsigned)tiles, kScanThreads, 0, st>>>(n, cnt, tile_sum);
  scan_tiles_kernel<<<1, kScanThreads, 0, st>>>((int)tiles, tile_sum);
  scan_apply_kernel<<<(unsigned)tiles, kScanThreads, 0, st>>>(n, cnt, tile_sum, out);
  return cudaGetLastError();
}

}  // namespace

template <typename Id>
cudaError_t launch_stage_check(int64_t nV, int64_t nT, const Id *tets, const double *xyz, uint32_t *first,
                               StageCtl *ctl, cudaStream_t st)
{
  cudaError_t e;
  if ((e = cudaMemsetAsync(ctl, 0xff, offsetof(StageCtl, max_edge2), st)) != cudaSuccess) return e;
  if ((e = cudaMemsetAsync(&ctl->max_edge2, 0, sizeof(StageCtl) - offsetof(StageCtl, max_edge2), st)) != cudaSuccess)
    return e;
  if (first && (e = cudaMemsetAsync(first, 0xff, sizeof(uint32_t) * (size_t)nV, st)) != cudaSuccess) return e;
  check_tets_kernel<<<stage_grid(nT, kStageThreads), kStageThreads, 0, st>>>(nV, nT, tets, first, ctl);
  check_xyz_kernel<<<stage_grid(3 * nV, kStageThreads), kStageThreads, 0, st>>>(3 * nV, xyz, ctl);
  return cudaGetLastError();
}

template <typename Id>
cudaError_t launch_stage_slots(int64_t nT, const Id *tets, const uint32_t *first, int32_t *slots, cudaStream_t st)
{
  slots_kernel<<<stage_grid(nT, kStageThreads), kStageThreads, 0, st>>>(nT, tets, first,
                                                                        reinterpret_cast<int4 *>(slots));
  return cudaGetLastError();
}

template cudaError_t launch_stage_check(int64_t, int64_t, const int64_t *, const double *, uint32_t *, StageCtl *,
                                        cudaStream_t);
template cudaError_t launch_stage_check(int64_t, int64_t, const int32_t *, const double *, uint32_t *, StageCtl *,
                                        cudaStream_t);
template cudaError_t launch_stage_slots(int64_t, const int64_t *, const uint32_t *, int32_t *, cudaStream_t);
template cudaError_t launch_stage_slots(int64_t, const int32_t *, const uint32_t *, int32_t *, cudaStream_t);

cudaError_t launch_stage_lists(int64_t nL, int64_t nT, const StageLists &x, StageCtl *ctl, cudaStream_t st)
{
  const int64_t nC = 4 * nT;
  const auto *cs4 = reinterpret_cast<const int4 *>(x.cslots);
  cudaError_t e;
  if ((e = cudaMemsetAsync(x.cnt, 0, sizeof(int32_t) * (size_t)nL, st)) != cudaSuccess) return e;
  count_corners_kernel<<<stage_grid(nC, kStageThreads), kStageThreads, 0, st>>>(nC, x.cslots, x.cnt);
  if ((e = scan(nL, x.cnt, x.cptr, x.tile_sum, st)) != cudaSuccess) return e;
  fill_corners_kernel<<<stage_grid(nC, kStageThreads), kStageThreads, 0, st>>>(nC, x.cslots, x.cptr, x.cnt, x.keys);
  lists_kernel<<<stage_grid(nL, kListWarps), 32 * kListWarps, 0, st>>>(nL, cs4, x.cptr, x.keys, x.crec, x.cidx,
                                                                       x.scratch, x.cnt, x.big_list, ctl);
  big_lists_kernel<<<1, 1024, 0, st>>>(nL, cs4, x.cptr, x.keys, x.scratch, x.cnt, x.big_list, x.mark, ctl);
  return scan(nL, x.cnt, x.nptr, x.tile_sum, st);
}

cudaError_t launch_stage_compact(int64_t nL, const StageLists &x, int32_t *nbr, cudaStream_t st)
{
  compact_kernel<<<stage_grid(nL, kStageThreads / 16), kStageThreads, 0, st>>>(nL, x.cptr, x.nptr, x.scratch, nbr);
  return cudaGetLastError();
}

cudaError_t launch_stage_in_tet(int64_t nV, const int64_t *cptr, uint8_t *in_tet, cudaStream_t st)
{
  in_tet_kernel<<<stage_grid(nV, kStageThreads), kStageThreads, 0, st>>>(nV, cptr, in_tet);
  return cudaGetLastError();
}

cudaError_t launch_edge_vectors(const int32_t *tslots, const double *xyz, int64_t nT, double *evec, StageCtl *ctl,
                                cudaStream_t stream)
{
  if (nT <= 0) return cudaSuccess;
  edge_vector_kernel<<<stage_grid(nT, kStageThreads), kStageThreads, 0, stream>>>(
      reinterpret_cast<const int4 *>(tslots), xyz, nT, evec, ctl);
  return cudaGetLastError();
}

}  // namespace fimgb
