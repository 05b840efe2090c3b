// sg_noalloc.cu - force evaluation that allocates no device memory.
//
// Some callers cannot call cudaMalloc: code running under another framework's memory manager,
// which owns the device heap and forbids raw allocations; code that must not stall other work
// on the device with the implicit synchronisation of cudaMalloc/cudaFree; plugins that may not
// grow the process's device footprint per call.  sg_compute_forces_noalloc serves them: the
// caller passes device buffers for the inputs and outputs, and every intermediate of the
// evaluation (cell counts and starts, sorted atoms, neighbour lists, EAM densities, the
// parameter block) lives in one file-scope static device array of
// SG_NOALLOC_SCRATCH_BYTES, which every GPU that loads the library holds until the process
// exits.
//
// The work is that of sg_build_lists + sg_compute_forces of a context: atoms sorted by cell,
// neighbour list, EAM density, metal and carbon forces, in five launches.
#include <cuda_runtime.h>

#include <cstddef>
#include <cstring>
#include <mutex>

#include "sg_api.h"
#include "sg_device.cuh"
#include "sg_engine.h"
#include "sg_kernels.h"

using namespace sg;

namespace {

constexpr size_t kScratchBytes = SG_NOALLOC_SCRATCH_BYTES;
constexpr int kBs = 128;
// home atoms per work item of the list build: 4, so that a small system's warps have little to do in
// sequence (a call on 2,217 / 15,883 atoms: 54.8 / 67.2 us; 8 as in the step, 56.7 / 67.7)
constexpr int kItem = kMinItemAtoms;
constexpr int kSortCells = 512;         // cells per block of the sort
constexpr int kSortThreads = 1024;
constexpr int kBuildBlocks = 7 * 152;  // the list build's: its blocks resident at once on a GB300
static_assert(SG_NOALLOC_MAX_ATOMS < (1 << 15) && kSortCells <= (1 << 16), "the sort packs cell and atom in a word");

// The scratch of every call on this device.  Host code must not take its address directly:
// the host-side name is only a stand-in; the device address comes from cudaGetSymbolAddress.
static __device__ __align__(256) unsigned char g_scratch[kScratchBytes];

// Carving of the scratch array (offsets in bytes, each 256-byte aligned).
struct Carve {
  size_t rc, st, cellStart;
  size_t cellOf, sortIdx, nn, ns, sl, sortPos, rho, posF, Fv, fric, nbl, nrl, rl, active, heavy, work, total;
};
constexpr size_t up(size_t x) { return (x + 255) & ~size_t(255); }
constexpr Carve carve() {
  Carve c{};
  size_t o = 0;
  const size_t N = SG_NOALLOC_MAX_ATOMS;
  c.rc = o; o += up(sizeof(RepConst));
  c.st = o; o += up(sizeof(RepState));
  c.cellStart = o; o += up(SG_NOALLOC_MAX_CELLS * sizeof(int));
  c.cellOf = o; o += up(N * sizeof(int));
  c.sortIdx = o; o += up(N * sizeof(int));
  c.nn = o; o += up(N * sizeof(int));
  c.ns = o; o += up(N * sizeof(int));
  c.sl = o; o += up(N * kShortMax * sizeof(int));
  c.sortPos = o; o += up(N * sizeof(float4));
  c.rho = o; o += up(N * sizeof(float));
  c.posF = o; o += up(N * sizeof(float4));
  c.Fv = o; o += up(N * sizeof(float));
  c.fric = o; o += up(N * sizeof(float));
  c.nbl = o; o += up(N * SG_NOALLOC_MAX_NEBR * sizeof(int));
  c.nrl = o; o += up(N * sizeof(int));
  c.rl = o; o += up(N * kRelMax * sizeof(unsigned));
  c.active = o; o += up(SG_NOALLOC_MAX_CELLS * sizeof(int));
  // a cell of n > t atoms (t = kItem) gives ceil(n / t) items: at most N / t + N / (t + 1) in all
  c.heavy = o; o += up(((size_t)N / kItem + (size_t)N / (kItem + 1) + 16) * sizeof(int2));
  c.work = o; o += up(4 * sizeof(int));
  c.total = o;
  return c;
}
constexpr Carve kCarve = carve();
static_assert(kCarve.total <= kScratchBytes, "scratch layout exceeds the static array");

// Device address of g_scratch per device ordinal, set up once per device.  The address belongs
// to the context that was current at set-up: the device's primary context, the one the CUDA
// runtime uses.  A caller that resets the device (cudaDeviceReset) or drives the device through
// another driver-API context is outside what this cache supports.
constexpr int kMaxDevices = 64;
unsigned char *g_base[kMaxDevices] = {};
std::mutex g_mu;

// Block 0 writes the parameter block and clears the state block and the list build's counters: what must
// start fresh on every call.  The others find the cells of kSortThreads atoms each (-1: outside the grid; past the last atom one that no cell
// has, up to a multiple of four).
constexpr int kNoCell = 1 << 30;
__global__ void __launch_bounds__(kSortThreads) k_noalloc_setup(const __grid_constant__ RepConst P, RepState *st,
                                                                RepConst *rc, int *work, const float4 *__restrict__ pos,
                                                                int *__restrict__ cellOf, int *__restrict__ nn,
                                                                int *__restrict__ ns, int *__restrict__ nrl) {
  asm volatile("griddepcontrol.launch_dependents;");  // the sort's few blocks may take their places now
  const int t = threadIdx.x, n = blockDim.x;
  if (blockIdx.x > 0) {
    const int g = (blockIdx.x - 1) * kSortThreads + t;
    if (g < P.nMol) {
      const float4 r = pos[g];
      const int c = cellIndex(P, r.x, r.y, r.z);
      cellOf[g] = c;
      if (c < 0) nn[g] = ns[g] = nrl[g] = 0;  // no list (the reference clears its NN)
    } else if (g < (P.nMol + 3 & ~3)) {
      cellOf[g] = kNoCell;
    }
    return;
  }
  for (int q = t; q < (int)(sizeof(RepConst) / 4); q += n)
    reinterpret_cast<int *>(rc)[q] = reinterpret_cast<const int *>(&P)[q];
  for (int q = t; q < (int)(sizeof(RepState) / 4); q += n)
    reinterpret_cast<int *>(st)[q] = q == (int)(offsetof(RepState, nebrNow) / 4) ? 1 : 0;
  if (t < 4) work[t] = 0;
}

// The atoms in cell order, ascending index inside a cell (sortIdx, sortPos), the cell starts and the
// list build's work items, in one pass: a block per kSortCells cells looks at every atom's cell (at
// most SG_NOALLOC_MAX_ATOMS, four of four a thread), counts those of earlier cells (its offset), keeps
// its own in shared memory, groups them by cell there and ranks each among its cell's.  The passes it
// replaces (count, three of a prefix sum, scatter, rank) were six launches of 3 to 9 us, each waiting
// for the one before: 32 us of the 87 us of kernels of a 2,217-atom call, 35 of 107 us at 15,883 atoms;
// now 8 and 12 us (ncu).  The whole call, with the two force passes in one launch and programmatic
// dependent launch: 105 -> 55 us and 129 -> 67 us.
// Dynamic shared memory: two words an atom.
__global__ void __launch_bounds__(kSortThreads) k_noalloc_sort(int nMol, int ncells, RepState *st,
                                                               const float4 *__restrict__ pos, const int *__restrict__ cellOf,
                                                               int *__restrict__ cellStart, int cap,
                                                               int2 *__restrict__ heavy, int *__restrict__ active,
                                                               int *__restrict__ work, int *__restrict__ sortIdx,
                                                               float4 *__restrict__ sortPos) {
  extern __shared__ unsigned sAtoms[];  // {cell of the block << 15 | atom} as met, then by cell
  __shared__ int sCount[kSortCells], sStart[kSortCells + 1], sBefore[kSortThreads / 32], sWarp[kSortCells / 32], sMine;
  unsigned *met = sAtoms, *byCell = sAtoms + nMol;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, c0 = blockIdx.x * kSortCells;
  if (tid < kSortCells) sCount[tid] = 0;
  if (tid == 0) sMine = 0;
  __syncthreads();
  pdlEnter();
  int before = 0, outside = 0;
#pragma unroll 4
  for (int q = tid; 4 * q < nMol; q += kSortThreads) {
    const int4 v = reinterpret_cast<const int4 *>(cellOf)[q];
    const int c[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int u = 0; u < 4; u++) {
      outside += c[u] < 0 ? 1 : 0;
      before += c[u] >= 0 && c[u] < c0 ? 1 : 0;
      if (c[u] >= c0 && c[u] < c0 + kSortCells) {
        atomicAdd(&sCount[c[u] - c0], 1);
        met[atomicAdd(&sMine, 1)] = (unsigned)(c[u] - c0) << 15 | (unsigned)(4 * q + u);
      }
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    before += __shfl_xor_sync(0xffffffffu, before, o);
    outside += __shfl_xor_sync(0xffffffffu, outside, o);
  }
  if (lane == 0) sBefore[wid] = before;
  __syncthreads();
  // prefix sum of the block's cells, a thread each
  const int n = tid < kSortCells ? sCount[tid] : 0;
  int incl = n;
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (tid < kSortCells && lane == 31) sWarp[wid] = incl;
  int base = sBefore[lane];  // kSortThreads / 32 = 32 warps
  for (int o = 16; o > 0; o >>= 1) base += __shfl_xor_sync(0xffffffffu, base, o);
  __syncthreads();
  if (tid < kSortCells) {
    int start = incl - n;
    for (int q = 0; q < wid; q++) start += sWarp[q];
    sStart[tid] = start;
    if (tid == kSortCells - 1) sStart[kSortCells] = start + n;
    if (c0 + tid <= ncells) cellStart[c0 + tid] = base + start;
    sCount[tid] = 0;  // arrivals of the grouping below
  }
  __syncthreads();
  // the work items: places in the lists asked for now, used at the end
  const bool live = n > 0 && c0 + tid < ncells;
  const int nHeavy = live && n > kItem ? (n + kItem - 1) / kItem : 0, nLight = live && n <= kItem ? 1 : 0;
  int preH = nHeavy, preL = nLight, occ = n, over = n > cap ? 1 : 0, atH = 0, atL = 0;
  if (tid < kSortCells) {
    for (int o = 1; o < 32; o <<= 1) {
      const int yh = __shfl_up_sync(0xffffffffu, preH, o), yl = __shfl_up_sync(0xffffffffu, preL, o);
      if (lane >= o) {
        preH += yh;
        preL += yl;
      }
    }
    for (int o = 16; o > 0; o >>= 1) {
      occ = max(occ, __shfl_xor_sync(0xffffffffu, occ, o));
      over += __shfl_xor_sync(0xffffffffu, over, o);
    }
    if (lane == 31) {
      if (preL) atL = atomicAdd(&work[1], preL);
      if (preH) atH = atomicAdd(&work[2], preH);
      if (occ) atomicMax(&st->maxCellOcc, occ);
      if (over) {
        atomicAdd(&st->cellOverflow, over);
        setFlag(st, 11 /*SG_ERR_CELL_OVERFLOW*/);
      }
    }
  }
  if (blockIdx.x == 0 && lane == 0 && outside) atomicAdd(&st->cellRange, outside);
  const int mine = sMine;
  for (int q = tid; q < mine; q += kSortThreads) {
    const unsigned v = met[q];
    byCell[sStart[v >> 15] + atomicAdd(&sCount[v >> 15], 1)] = v;
  }
  __syncthreads();
  for (int q = tid; q < mine; q += kSortThreads) {
    const unsigned v = byCell[q];
    const int c = v >> 15, g = v & 0x7fff, b = sStart[c], e = sStart[c + 1];
    float4 r = pos[g];
    int rank = 0;
    for (int k = b; k < e; k++) rank += byCell[k] < v ? 1 : 0;  // the same cell: compares atoms
    r.w = __int_as_float(g);
    sortIdx[base + b + rank] = g;
    sortPos[base + b + rank] = r;
  }
  if (tid >= kSortCells) return;
  atH = __shfl_sync(0xffffffffu, atH, 31) + preH - nHeavy;
  atL = __shfl_sync(0xffffffffu, atL, 31) + preL - nLight;
  for (int j = 0; j < nHeavy; j++) {
    const int h0 = j * n / nHeavy, h1 = (j + 1) * n / nHeavy;
    heavy[atH + j] = make_int2(c0 + tid, h0 << 16 | (h1 - h0));
  }
  if (nLight) active[atL] = c0 + tid;
}

RepConst constFor(const sg_simparams &p) {
  RepConst P;
  memset(&P, 0, sizeof(P));
  P.region[0] = p.region.x; P.region[1] = p.region.y; P.region[2] = p.region.z;
  P.invWidth[0] = p.invWidth.x; P.invWidth[1] = p.invWidth.y; P.invWidth[2] = p.invWidth.z;
  P.cells[0] = p.cells.x; P.cells[1] = p.cells.y; P.cells[2] = p.cells.z;
  P.ncells = p.cells.x * p.cells.y * p.cells.z;
  P.ncellsPad = ((P.ncells + 1 + kCellTile - 1) / kCellTile) * kCellTile;
  P.nMol = p.nMol; P.nMolMe = p.nMolMe;
  P.nRedBlocks = (p.nMol + kRedElems - 1) / kRedElems;
  P.deltaT = p.deltaT; P.rrNebr = p.rrNebr; P.rNebrShell = p.rNebrShell;
  const float rs = p.rCutC + p.rNebrShell;
  P.rrShort = rs * rs;
  P.rei = p.rei; P.rhoei = p.rhoei; P.rhoe = p.rhoe; P.fe = p.fe; P.alpha = p.alpha; P.beta = p.beta;
  P.A = p.A; P.B = p.B; P.kappa = p.kappa; P.lambda = p.lambda;
  for (int i = 0; i < 4; i++) { P.Fn[i] = p.Fn[i]; P.F[i] = p.F[i]; }
  P.eta = p.eta; P.Fe = p.Fe; P.massMe = p.massMe; P.rrCutEam = p.rrCutEam;
  P.rrCutC = p.rrCutC; P.mu_r = p.mu_r; P.theta_0 = p.theta_0; P.mu_theta = p.mu_theta; P.mu_p = p.mu_p;
  P.z_0 = p.z_0; P.sigmaLJ = p.sigmaLJ; P.epsLJ = p.epsLJ; P.rrCutLJ = p.rrCutLJ;
  P.hasFric = (p.iRegime != 0 && p.nMolMe != 0) ? 1 : 0;
  P.iRegime = p.iRegime;
  return P;
}

}  // namespace

extern "C" int sg_compute_forces_noalloc(const sg_simparams *p, sg_float4 *d_pos, sg_float4 *d_acc, void *stream) {
  if (!p || !d_pos || !d_acc) return sg_fail(SG_ERR_INVALID, "sg_compute_forces_noalloc: null argument");
  if (p->nMol <= 0 || p->nMolMe < 0 || p->nMolMe > p->nMol || p->cells.x < 1 || p->cells.y < 1 || p->cells.z < 1)
    return sg_fail(SG_ERR_INVALID, "sg_compute_forces_noalloc: inconsistent parameter block");
  // the cell count in 64 bits: a parameter block from outside may hold any extents, and an int
  // product could wrap to a small value that passes the limit
  const long long ncells64 = (long long)p->cells.x * p->cells.y * p->cells.z;
  const long long ncellsPad64 = ((ncells64 + 1 + kCellTile - 1) / kCellTile) * kCellTile;
  if (p->nMol > SG_NOALLOC_MAX_ATOMS || ncellsPad64 > SG_NOALLOC_MAX_CELLS || p->iNebrMax > SG_NOALLOC_MAX_NEBR ||
      p->iNebrMax < 1)
    return sg_fail(SG_ERR_INVALID,
                   "sg_compute_forces_noalloc: system exceeds the static scratch (nMol %d of max %d, "
                   "padded cells %lld of max %d, iNebrMax %d of max %d)",
                   p->nMol, SG_NOALLOC_MAX_ATOMS, ncellsPad64, SG_NOALLOC_MAX_CELLS, p->iNebrMax, SG_NOALLOC_MAX_NEBR);
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= kMaxDevices)
    return sg_fail(SG_ERR_NO_DEVICE, "sg_compute_forces_noalloc: no current device");
  unsigned char *base;
  {
    std::lock_guard<std::mutex> lk(g_mu);
    if (!g_base[dev]) {  // set-up, once per device, with that device current
      void *ptr = nullptr;
      e = cudaGetSymbolAddress(&ptr, g_scratch);
      if (e != cudaSuccess)
        return sg_fail(SG_ERR_CUDA, "cudaGetSymbolAddress(scratch): %s", cudaGetErrorString(e));
      // the sort's shared memory at the largest system
      e = cudaFuncSetAttribute(k_noalloc_sort, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)(2 * sizeof(unsigned) * SG_NOALLOC_MAX_ATOMS));
      if (e != cudaSuccess)
        return sg_fail(SG_ERR_CUDA, "cudaFuncSetAttribute(k_noalloc_sort): %s", cudaGetErrorString(e));
      g_base[dev] = (unsigned char *)ptr;
    }
    base = g_base[dev];
  }
  cudaStream_t s = (cudaStream_t)stream;
  const Carve &K = kCarve;
  RepConst *rc = (RepConst *)(base + K.rc);
  RepState *st = (RepState *)(base + K.st);
  int *cellStart = (int *)(base + K.cellStart);
  int *cellOf = (int *)(base + K.cellOf), *sortIdx = (int *)(base + K.sortIdx), *nn = (int *)(base + K.nn), *ns = (int *)(base + K.ns);
  int *sl = (int *)(base + K.sl);
  float4 *sortPos = (float4 *)(base + K.sortPos);
  float *rho = (float *)(base + K.rho), *Fv = (float *)(base + K.Fv);
  float *fric = (float *)(base + K.fric);
  float4 *posF = (float4 *)(base + K.posF);
  int *nbl = (int *)(base + K.nbl), *nrl = (int *)(base + K.nrl);
  unsigned *rl = (unsigned *)(base + K.rl);
  int *active = (int *)(base + K.active), *work = (int *)(base + K.work);
  int2 *heavy = (int2 *)(base + K.heavy);
  float4 *pos = (float4 *)d_pos, *acc = (float4 *)d_acc;

  const RepConst P = constFor(*p);
  const int N = p->nMol;
  const int nMetalBlk = (p->nMolMe + kMetalPerBlock - 1) / kMetalPerBlock;
  const int nCarbBlk = (N - p->nMolMe + kCarbonPerBlock - 1) / kCarbonPerBlock;
  const BlockTab metalTab{nullptr, nullptr, nMetalBlk, nullptr, 0, kMetalPerBlock, p->nMolMe};
  const BlockTab carbTab{nullptr, nullptr, nCarbBlk, nullptr, p->nMolMe, kCarbonPerBlock, N};
  const int rowStride = (p->iNebrMax + 3) & ~3;
  const size_t sortSmem = 2 * sizeof(unsigned) * N;

  k_noalloc_setup<<<1 + (N + kSortThreads + 3) / kSortThreads, kSortThreads, 0, s>>>(P, st, rc, work,
                                                                                     pos, cellOf, nn, ns, nrl);
  launchK(true, k_noalloc_sort, P.ncells / kSortCells + 1, kSortThreads, sortSmem, s, N, P.ncells, st, pos, cellOf, cellStart,
          (int)p->blockSize, heavy, active, work, sortIdx, sortPos);
  launchK(true, k_build_nebr, kBuildBlocks, kNebrWarps * 32, 0, s, nullptr, active, heavy, work, rc, st, cellStart, sortPos, nn,
          nbl, ns, sl, nrl, rl, rowStride, p->iNebrMax, 0, nullptr, 0);
  if (nMetalBlk)
    launchK(true, k_rho, nMetalBlk, kBs, 0, s, metalTab, rc, pos, nn, nbl, rho, posF, Fv, rowStride);
  launchK(true, k_force_both, nMetalBlk + nCarbBlk, kBs, 0, s, metalTab, carbTab, rc, pos, acc, nn, nbl, ns, sl, nrl, rl, posF, Fv,
          fric, rowStride);
  e = cudaGetLastError();
  if (e != cudaSuccess) return sg_fail(SG_ERR_CUDA, "sg_compute_forces_noalloc launch: %s", cudaGetErrorString(e));
  int flags = 0;
  e = cudaMemcpyAsync(&flags, &st->flags, sizeof(int), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return sg_fail(SG_ERR_CUDA, "sg_compute_forces_noalloc: %s", cudaGetErrorString(e));
  for (int code = 1; code < 31; code++)
    if (flags & (1 << code)) return sg_fail(code, "sg_compute_forces_noalloc: device reported condition %d", code);
  return SG_OK;
}
