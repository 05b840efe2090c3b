// sg_adjoint.cu - the differentiation form: the metal part of the model (EAM with B-spline
// pair functions, metal-carbon Lennard-Jones) as a function of 66 fit parameters, its forces,
// and the gradients of the frame energies and of a force-matching loss from a hand-written
// adjoint pass.  No counterpart in the reference (its potentials are fixed analytic forms).
//
// Parameters theta: [0] epsilon, [1] sigma of the metal-carbon LJ; [2, 34) the cubic B-spline
// coefficients of phi(r); [34, 66) those of f(r), on 29 equal intervals from 0.6 r_e to the EAM
// cutoff.  On interval k (x = (r - r0) / h, t = x - k) a spline is sum_m c[k + m] b_m(t) with the
// uniform cubic B-spline weights b_0 = (1-t)^3/6, b_1 = (3t^3 - 6t^2 + 4)/6,
// b_2 = (-3t^3 + 3t^2 + 3t + 1)/6, b_3 = t^3/6: linear in the coefficients, C2 in r.
//
// Force matching.  With the residual e_i = 2 (F_i - F_ref,i) / (3N) held fixed,
//   dL/dtheta = -d/dtheta D,   D = sum_i e_i . dE/dr_i
//             = 1/2 sum_{i,j metal} phi'(r_ij) w_ij + sum_i F'(rho_i) g_i + sum_{MC} U'(r) w,
//   w_ij = rhat_ij . (e_i - e_j),  g_i = sum_j f'(r_ij) w_ij  (the change of rho_i along e),
// so  dD/dc_phi,k = 1/2 sum B_k'(r) w,   dD/dc_f,k = sum_i [F''(rho_i) g_i sum_j B_k(r_ij)
// + F'(rho_i) sum_j B_k'(r_ij) w_ij],  dD/d(eps, sigma) = sum_MC d U'(r)/d(eps, sigma) w.
// Four passes: densities (F' and F'' of every metal atom), forces or residuals, g_i with the w of every
// pair (k_diff_along), and these sums over each metal pair once.  What a pair keeps between evaluations
// is its geometry alone.
//
// Pair arithmetic in FP32 (FMA on).  Sums that grow with the set of frames pass to FP64 after a few dozen
// terms (a thread's spline coefficients, an atom's pairs) or are compensated (LongSum: losses, the LJ
// parameters), so that their error does not grow with it; energies, losses and gradients are summed in
// FP64 across blocks.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "sg_api.h"
#include "sg_device.cuh"
#include "sg_engine.h"
#include "sg_kernels.h"

namespace sg {

constexpr int kDP = SG_DIFF_NPARAM;
constexpr int kSC = SG_DIFF_SPLINE_COEFFS;
constexpr int kSI = SG_DIFF_SPLINE_INTERVALS;
constexpr int kPhi = 2, kDen = 2 + kSC;  // offsets of the two splines in theta
static_assert(kSC == kSI + 3 && kDP == 2 + 2 * kSC, "spline layout");

constexpr int kDT = 128;    // threads per block but for the passes over work lists
// The passes over work lists: warps per slice of 32 atoms, and pairs a thread loads together (a bulk
// metal atom has 42 to 48, 6 a thread), with what it gathers for them fewer for the sake of registers:
// 64, four blocks an SM.  Over 64 frames of 20,432 atoms a force-matching evaluation takes 202 us with
// 8 warps and 3 pairs (6 pairs: 228), 215 with 4 warps, 242 with 16; over 4 frames of 2,217 atoms 49,
// 60 and 49.
constexpr int kParts = 8, kLoads = 6, kGathers = 3, kPassThreads = 32 * kParts, kPassBlocks = 4;

// The model of one call: epsilon, sigma and both splines as one cubic per interval, in s = r - knot
// with knot the interval's first knot rounded to float: the coefficients are theta's, expanded around
// that float in FP64, and s is an exact difference for any r near the interval, so no rounding of
// knots or widths enters a value or slope.  In device memory, copied there ahead of the passes: as a
// kernel parameter of this size, every block's read of it took 5 to 12 us of misses in the constant
// cache.
struct DiffModel {
  float4 phi[kSI], den[kSI];
  float2 knot[kSI];          // {knot, its interval coordinate t (0 but for its rounding)}
  float r0, invH;            // first knot, 1 / interval width
  float eps, sig6, invSig;   // epsilon, sigma^6, 1 / sigma
  float pad;
};
static_assert(sizeof(DiffModel) % 16 == 0, "copied as 16-byte words");
__device__ __forceinline__ void loadModel(const DiffModel *__restrict__ model, DiffModel &m) {
  const float4 *src = reinterpret_cast<const float4 *>(model);
  float4 *dst = reinterpret_cast<float4 *>(&m);
  for (int q = threadIdx.x; q < (int)(sizeof(DiffModel) / 16); q += blockDim.x) dst[q] = src[q];
  __syncthreads();
}

// Interval of r (the end pieces continue past the ends).
__device__ __forceinline__ int interval(const DiffModel &m, float r) {
  return max(0, min((int)floorf((r - m.r0) * m.invH), kSI - 1));
}
__device__ __forceinline__ float cubic(const float4 &c, float s) { return c.x + s * (c.y + s * (c.z + s * c.w)); }
__device__ __forceinline__ float slope(const float4 &c, float s) { return c.y + s * (2.f * c.z + 3.f * s * c.w); }

// The reference's embedding function (SurfaceGrowth.cu:72-126 forms) with its first and second
// derivatives.
__device__ __forceinline__ void embedAll(const RepConst &P, float rho, float &F, float &Fp, float &Fpp) {
  const float rhon = 0.85f * P.rhoe, rhoo = 1.15f * P.rhoe;
  if (rho < rhon) {
    const float s = P.rhoei * 1.176471f, x = rho * s - 1.f;
    F = P.Fn[0] + x * (P.Fn[1] + x * (P.Fn[2] + x * P.Fn[3]));
    Fp = s * (P.Fn[1] + x * (2.f * P.Fn[2] + 3.f * x * P.Fn[3]));
    Fpp = s * s * (2.f * P.Fn[2] + 6.f * x * P.Fn[3]);
  } else if (rho < rhoo) {
    const float s = P.rhoei, x = rho * s - 1.f;
    F = P.F[0] + x * (P.F[1] + x * (P.F[2] + x * P.F[3]));
    Fp = s * (P.F[1] + x * (2.f * P.F[2] + 3.f * x * P.F[3]));
    Fpp = s * s * (2.f * P.F[2] + 6.f * x * P.F[3]);
  } else {
    const float y = rho * P.rhoei, ly = logf(y), yeta = powf(y, P.eta);
    F = P.Fe * (1.f - P.eta * ly) * yeta;
    Fp = -P.Fe * P.eta * P.eta * P.rhoei * yeta / y * ly;
    Fpp = -P.Fe * P.eta * P.eta * P.rhoei * P.rhoei * yeta / (y * y) * ((P.eta - 1.f) * ly + 1.f);
  }
}

// The sums of an evaluation, the 66 parameters' and the loss, in kSumCopies copies that blocks add
// to in turn (the host adds the copies): FP64 additions to one address follow one another at about
// 20 ns, and 912 blocks on one copy ended in 20 us of them.
constexpr int kSumCopies = 32, kSumStride = kDP + 1, kSums = kSumCopies * kSumStride;
__device__ __forceinline__ double *sumsCopy(double *sums) { return sums + kSumStride * (blockIdx.x % kSumCopies); }
__device__ __forceinline__ float warpSumF(float x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}
__device__ __forceinline__ double warpSumD(double x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}
// A thread's FP32 sum of any number of terms, with what each addition rounds off carried into the next
// (W. Kahan, "Further remarks on reducing truncation errors", 1965): wrong by two roundings whatever
// their number, where a plain sum's error grows with it and FP64 runs at 1/64 of the rate.  A sum that
// has left the finite numbers carries nothing.
struct LongSum {
  float s = 0.f, c = 0.f;
  __device__ __forceinline__ void add(float x) {
    const float y = __fsub_rn(x, c), t = __fadd_rn(s, y);
    c = fabsf(t) <= 3.4028234664e38f ? __fsub_rn(__fsub_rn(t, s), y) : 0.f;
    s = t;
  }
};
// ---- pair lists ----------------------------------------------------------------------------
// Positions are set once for many evaluations of a fit, so everything that follows from them alone
// is laid out then: which pairs an evaluation needs (a metal atom's metal entries within the EAM
// cutoff and its carbon entries within the LJ cutoff, and those of the few carbon atoms that have
// metal within it, out of rows built to the larger cutoff over every species) and each pair's
// distance and direction, in the order the passes read them.  An evaluation streams
// them and gathers only what depends on theta.  Before, every pass gathered positions and derived
// distances anew (about 75 instructions a pair), and a thread per carbon atom walked its whole row
// (195 us of the 733 us of kernels of a force-matching evaluation over 64 frames of 20,432 atoms).
//
// The work lists go in slices of 32 atoms, a lane each, and a slice's pairs are interleaved: pair j
// of lane l at first + 32 j + l, so that a warp's load of its atoms' j-th pairs is one contiguous
// piece.  (With 4 to 16 lanes an atom, whose pairs lay in a row, the same passes took 2 to 3 times
// as long: shorter loops with more remainders, the embedding function for 2 to 8 atoms a warp, and
// three waves of blocks, each a chain of dependent loads.)
//
// Per-atom values are kept in slots: positions in the cell order the list build sorts the atoms
// into.  The atoms of a warp then share most of their neighbours, and a gather touches few cache
// lines (metal atoms are numbered by distance from their cluster's centre, which scatters them).

// slotOf[atom] (-1: outside the grid, or no lists yet; such an atom has no pair).
__global__ void k_diff_slots(BlockTab tab, const RepConst *__restrict__ rc, const int *__restrict__ cellStart,
                             const int *__restrict__ sortIdx, int *__restrict__ slotOf) {
  const RepConst &P = rc[tab.rep[blockIdx.x]];
  const int s = tab.start[blockIdx.x] + threadIdx.x;
  if (s < cellStart[P.cellOff + P.ncells]) slotOf[sortIdx[s]] = s;
}
// A warp per atom: its row packed to metal entries of higher slots, the other metal entries and
// carbon entries, with their numbers in seg[slot] (all metal, carbon, metal of higher slots);
// paired[atom] set for every metal atom in the grid and for a carbon atom of any LJ pair.  oneSided:
// rows that did not hold all their entries, of which a pair may be in one only; every metal entry then
// counts as one of a higher slot (k_diff_sums takes each for its own side).
__global__ void __launch_bounds__(kDT) k_diff_pack(BlockTab tab, const RepConst *__restrict__ rc,
                                                   const float4 *__restrict__ pos, const int *__restrict__ nn,
                                                   const int *__restrict__ slotOf, int *__restrict__ nbl, int rowStride,
                                                   int restStride, int4 *__restrict__ seg,
                                                   unsigned char *__restrict__ paired, bool oneSided) {
  extern __shared__ int sRow[];
  const unsigned full = 0xffffffffu;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int per = 128 / (blockDim.x / 32);  // blocks per table entry (128 atoms)
  const RepConst &P = rc[tab.rep[blockIdx.x / per]];
  const int i = tab.start[blockIdx.x / per] + (blockIdx.x % per) * (blockDim.x / 32) + w;
  if (i >= P.atomOff + P.nMol || slotOf[i] < 0) return;
  const int metalEnd = P.atomOff + P.nMolMe, own = slotOf[i];
  const bool metal = i < metalEnd;
  // what does not go to the front of the row: lower metal entries from the start, carbon from the
  // end (backwards); together at most the row's entries
  int *rest = sRow + w * restStride;
  const float4 A = pos[i];
  int *row = nbl + (size_t)i * rowStride;
  const int len = nn[i];
  int nh = 0, nl = 0, nc = 0;
  for (int base = 0; base < len; base += 32) {
    const int k = base + lane < len ? row[base + lane] : -1;
    bool e = false, c = false;
    int slot = 0;
    if (k >= 0 && (metal || k < metalEnd)) {
      const float4 B = pos[k];
      const float dx = minImg(A.x - B.x, P.region[0]), dy = minImg(A.y - B.y, P.region[1]),
                  dz = minImg(A.z - B.z, P.region[2]);
      const float rr = dx * dx + dy * dy + dz * dz;
      if (metal && k < metalEnd) e = rr < P.rrCutEam;
      else c = rr < P.rrCutLJ;
      if (c) paired[metal ? k : i] = 1;  // seen from either side
      slot = slotOf[k];
    }
    const unsigned lower = (1u << lane) - 1u;
    const unsigned bh = __ballot_sync(full, e && slot > own), bl = __ballot_sync(full, e && slot < own),
                   bc = __ballot_sync(full, c);
    // every lane has read its entry of this and all earlier words: the packed row ends before them
    if (e && slot > own) row[nh + __popc(bh & lower)] = slot;
    else if (e) rest[nl + __popc(bl & lower)] = slot;
    else if (c) rest[restStride - 1 - nc - __popc(bc & lower)] = slot;
    nh += __popc(bh);
    nl += __popc(bl);
    nc += __popc(bc);
    __syncwarp();
  }
  for (int q = lane; q < nl; q += 32) row[nh + q] = rest[q];
  for (int q = lane; q < nc; q += 32) row[nh + nl + q] = rest[restStride - 1 - q];
  if (lane == 0) {
    seg[own] = make_int4(nh + nl, nc, oneSided ? nh + nl : nh, 0);
    if (metal) paired[i] = 1;
  }
}
// An atom of a work list: its slot (-1: a metal atom outside the grid, which has no pair but still
// its F(0); or none, filling the last slice), its frame (-1: none), its numbers of metal pairs and
// of carbon pairs after them; the first nh, those with metal atoms of higher slots, are the metal
// pairs counted once.
struct DiffWork {
  int slot, rep, ne, nc, nh, pad[3];
};
static_assert(sizeof(DiffWork) == 32, "read in 16-byte words");
// Appends the lanes with `on` to a work list in lane order.
__device__ __forceinline__ void appendWork(bool on, int slot, int rep, const int4 *__restrict__ seg,
                                           DiffWork *__restrict__ list, int *__restrict__ count) {
  const unsigned full = 0xffffffffu, b = __ballot_sync(full, on);
  const int lane = threadIdx.x & 31;
  int at = 0;
  if (lane == 0 && b) at = atomicAdd(count, __popc(b));
  at = __shfl_sync(full, at, 0) + __popc(b & ((1u << lane) - 1u));
  if (!on) return;
  const int4 c = slot >= 0 ? seg[slot] : make_int4(0, 0, 0, 0);
  list[at] = DiffWork{slot, rep, c.x, c.y, c.z};
}
// The work lists: metal atoms, and carbon atoms with an LJ pair (counts[0], counts[1]).
__global__ void k_diff_lists(BlockTab tab, const RepConst *__restrict__ rc, const int *__restrict__ cellStart,
                             const int *__restrict__ sortIdx, const int *__restrict__ slotOf, bool built,
                             const unsigned char *__restrict__ paired, const int4 *__restrict__ seg,
                             DiffWork *__restrict__ metal, DiffWork *__restrict__ carbon, int *__restrict__ counts) {
  const int rep = tab.rep[blockIdx.x], s = tab.start[blockIdx.x] + threadIdx.x;
  const RepConst &P = rc[rep];
  const int metalEnd = P.atomOff + P.nMolMe;
  const int atom = built && s < cellStart[P.cellOff + P.ncells] ? sortIdx[s] : -1;
  appendWork(atom >= 0 && atom < metalEnd, s, rep, seg, metal, &counts[0]);
  appendWork(s < metalEnd && slotOf[s] < 0, -1, rep, seg, metal, &counts[0]);
  appendWork(atom >= metalEnd && paired[atom], s, rep, seg, carbon, &counts[1]);
}

// A slice of 32 atoms of a work list: where its pairs start, the most metal and carbon pairs of an
// atom (an atom's carbon pairs follow the most metal ones), and where its metal pairs counted once do.
struct DiffSlice {
  int first, most, mostC, once;
};
// A warp per slice; totals: places taken by the pairs of all slices, metal pairs counted once.  The
// last slice is filled.
__global__ void __launch_bounds__(kDT) k_diff_slices(DiffWork *__restrict__ list, int n, DiffSlice *__restrict__ slices,
                                                     unsigned long long *__restrict__ totals) {
  const unsigned full = 0xffffffffu;
  const int s = blockIdx.x * (kDT / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31, u = 32 * s + lane;
  if (32 * s >= n) return;
  DiffWork w{-1, -1, 0, 0, 0};
  if (u < n) w = list[u];
  else list[u] = w;
  const int most = __reduce_max_sync(full, w.ne), mostC = __reduce_max_sync(full, w.nc), once = __reduce_add_sync(full, w.nh);
  if (lane == 0)
    slices[s] = DiffSlice{(int)atomicAdd(&totals[0], 32ull * (most + mostC)), most, mostC,
                          (int)atomicAdd(&totals[1], (unsigned long long)once)};
}

// Pairs as the passes read them: the other atom's slot, the distance, and the direction (from the
// other atom to this one).
struct DiffPairs {
  int *slot;
  float *r;
  float4 *dir;  // w: the distance again
  float *w;     // of an evaluation
  int2 *both;   // the metal pairs counted once: both slots, the distance, the place of its w
  float *rOnce;
  int *place;
};
// A warp per atom of a work list.
__global__ void __launch_bounds__(kDT) k_diff_pairs(const DiffWork *__restrict__ list, const DiffSlice *__restrict__ slices,
                                                    int n, const RepConst *__restrict__ rc,
                                                    const float4 *__restrict__ slotPos, const int *__restrict__ nbl,
                                                    int rowStride, DiffPairs pr) {
  const int u = blockIdx.x * (kDT / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (u >= n || list[u].slot < 0) return;
  const DiffWork a = list[u];
  const DiffSlice sl = slices[u / 32];
  const RepConst &P = rc[a.rep];
  const float4 A = slotPos[a.slot];
  const int *row = nbl + (size_t)__float_as_int(A.w) * rowStride;
  for (int j = lane; j < a.ne + a.nc; j += 32) {
    const int k = row[j];
    const float4 B = slotPos[k];
    const float dx = minImg(A.x - B.x, P.region[0]), dy = minImg(A.y - B.y, P.region[1]),
                dz = minImg(A.z - B.z, P.region[2]);
    const float r = sqrtf(dx * dx + dy * dy + dz * dz);
    const int at = sl.first + 32 * (j < a.ne ? j : sl.most + j - a.ne) + u % 32;
    pr.slot[at] = k;
    pr.r[at] = r;
    pr.dir[at] = make_float4(dx / r, dy / r, dz / r, r);
  }
}
// A warp per slice: its metal pairs counted once, in the order of their places, so that what is read
// at the places of neighbouring ones lies together.
__global__ void __launch_bounds__(kDT) k_diff_once(const DiffWork *__restrict__ list, const DiffSlice *__restrict__ slices,
                                                   int n, DiffPairs pr) {
  const int s = blockIdx.x * (kDT / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (32 * s >= n) return;
  const DiffWork a = list[32 * s + lane];
  const DiffSlice sl = slices[s];
  int at = sl.once;
  for (int j = 0; j < sl.most; j++) {
    const unsigned b = __ballot_sync(0xffffffffu, j < a.nh);
    if (j < a.nh) {
      const int place = sl.first + 32 * j + lane, q = at + __popc(b & ((1u << lane) - 1u));
      pr.both[q] = make_int2(a.slot, pr.slot[place]);
      pr.rOnce[q] = pr.r[place];
      pr.place[q] = place;
    }
    at += __popc(b);
  }
}

// ---- evaluation ----------------------------------------------------------------------------
// All passes over work lists: a lane per atom, a slice a block at a time, kParts warps that take every
// kParts-th pair each; their sums meet in shared memory.  A load that misses L1 takes 0.5 us here, and
// what a pass costs is the number of such loads that wait for one another: a thread loads several pairs
// together, and the next slice's work entries while this one is evaluated.  A block walks the slices
// with a grid stride, so that it loads the model once.
struct DiffAtom {
  int slot, rep, ne, nc, nh;  // as DiffWork; slot -1, no pairs and rep -1 past the end of the list
  int first, most, mostC;           // as DiffSlice
};
__device__ __forceinline__ DiffAtom diffAtom(const DiffWork *__restrict__ list, const DiffSlice *__restrict__ slices, int n,
                                             int slice) {
  if (32 * slice >= n) return DiffAtom{-1, -1, 0, 0, 0, 0, 0, 0};
  const DiffWork *w = list + 32 * slice + (threadIdx.x & 31);
  const int4 w0 = *reinterpret_cast<const int4 *>(w), s = *reinterpret_cast<const int4 *>(slices + slice);
  return DiffAtom{w0.x, w0.y, w0.z, w0.w, w->nh, s.x, s.y, s.z};
}
// Sums of x over the parts, for part 0 (warp 0).  Two buffers in turn: the others may write the next
// slice's while part 0 still reads this one's.
template <int N>
__device__ __forceinline__ void sumParts(int turn, float (&x)[N]) {
  __shared__ float s[2][kParts][N][32];
  const int part = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < N; k++) s[turn & 1][part][k][lane] = x[k];
  __syncthreads();
  if (part != 0) return;
#pragma unroll
  for (int k = 0; k < N; k++) {
    x[k] = 0.f;
#pragma unroll
    for (int p = 0; p < kParts; p++) x[k] += s[turn & 1][p][k][lane];
  }
}
// f(u, j) over a thread's share of its atom's n pairs j (at first + 32 j + lane), the most of any lane
// of the slice being `most`; U at a time, load(u, place) for all of them first.
template <int U, typename Load, typename F>
__device__ __forceinline__ void overPairs(int first, int n, int most, Load load, F f) {
  const int lane = threadIdx.x & 31;
  for (int j0 = threadIdx.x >> 5; j0 < most; j0 += U * kParts) {
#pragma unroll
    for (int u = 0; u < U; u++)
      if (j0 + u * kParts < n) load(u, first + 32 * (j0 + u * kParts) + lane);
#pragma unroll
    for (int u = 0; u < U; u++)
      if (j0 + u * kParts < n) f(u, j0 + u * kParts);
  }
}
// (sigma / r)^6 of an LJ pair
__device__ __forceinline__ float ljSix(float sig6, float r) {
  const float i2 = 1.f / (r * r);
  return sig6 * (i2 * i2 * i2);
}

// Densities: F'(rho) and F''(rho) of every metal atom (emb, by slot); with ENERGY also the frame
// energies (to which it only adds), else the launch clears the sums of the evaluation (sums), and
// its first refBlocks blocks fetch the reference forces of the atoms with pairs (into refOf, by slot)
// for the force pass, which a read over the host link by each of its atoms would hold up.
template <bool ENERGY>
__global__ void __launch_bounds__(kPassThreads) k_diff_rho(const DiffModel *__restrict__ model, const DiffWork *__restrict__ metal,
                                                  const DiffSlice *__restrict__ slices, int nMetal,
                                                  const RepConst *__restrict__ rc, const float *__restrict__ pairR,
                                                  float2 *__restrict__ emb, double *__restrict__ energy,
                                                  double *__restrict__ sums, const float *__restrict__ ref, int n,
                                                  const unsigned char *__restrict__ paired, const int *__restrict__ slotOf,
                                                  float4 *__restrict__ refOf, int refBlocks) {
  __shared__ __align__(16) DiffModel m;
  pdlEnter();
  if (!ENERGY && blockIdx.x == 0)
    for (int q = threadIdx.x; q < kSums; q += blockDim.x) sums[q] = 0.0;
  const int block = (int)blockIdx.x - refBlocks;
  if (!ENERGY && block < 0) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += refBlocks * blockDim.x)
      if (paired[i]) refOf[slotOf[i]] = make_float4(ref[3 * (size_t)i], ref[3 * (size_t)i + 1], ref[3 * (size_t)i + 2], 0.f);
    return;
  }
  const int grid = gridDim.x - refBlocks, nSlices = (nMetal + 31) / 32, lane = threadIdx.x & 31;
  DiffAtom next = diffAtom(metal, slices, nMetal, block);
  loadModel(model, m);
  for (int slice = block, turn = 0; slice < nSlices; slice += grid, turn++) {
    const DiffAtom a = next;
    next = diffAtom(metal, slices, nMetal, slice + grid);
    float x[2] = {0.f, 0.f};  // rho, pair energy
    float r[kLoads];
    auto load = [&](int u, int p) { r[u] = pairR[p]; };
    overPairs<kLoads>(a.first, a.ne, a.most, load, [&](int u, int) {
      const int i = interval(m, r[u]);
      const float s = r[u] - m.knot[i].x;
      x[0] += cubic(m.den[i], s);
      if (ENERGY) x[1] += 0.5f * cubic(m.phi[i], s);
    });
    if (ENERGY)
      overPairs<kLoads>(a.first + 32 * a.most, a.nc, a.mostC, load, [&](int u, int) {
        const float s6 = ljSix(m.sig6, r[u]);
        x[1] += 4.f * m.eps * (s6 * s6 - s6);  // the whole pair, from the metal side
      });
    sumParts(turn, x);
    if (threadIdx.x >= 32) continue;
    float F = 0.f, Fd, Fdd;
    if (a.rep >= 0) embedAll(rc[a.rep], x[0], F, Fd, Fdd);
    if (a.slot >= 0) emb[a.slot] = make_float2(Fd, Fdd);
    if (ENERGY) {
      // the slice's atoms of one frame in one sum; a slice whose atoms are of several adds them singly
      const int rep = __shfl_sync(0xffffffffu, a.rep, 0);
      const double u = (double)x[1] + (double)F;
      if (__all_sync(0xffffffffu, a.rep < 0 || a.rep == rep)) {
        const double all = warpSumD(u);
        if (lane == 0 && rep >= 0) atomicAdd(&energy[rep], all);
      } else if (a.rep >= 0) {
        atomicAdd(&energy[a.rep], u);
      }
    }
  }
}

// Sum over the block (all threads), in thread 0: FP32 in a warp, FP64 over the warps.  (FP64 runs at
// 1/64 of the FP32 rate here: with the warps' sums in FP64 too, a block of 8 warps kept the SM's FP64
// pipe busy for 1,700 cycles, and this sum took half of the force pass.)
__device__ __forceinline__ double blockSum(float x) {
  __shared__ float s[32];
  x = warpSumF(x);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = x;
  __syncthreads();
  double y = 0.0;
  if (threadIdx.x == 0)
    for (int q = 0; q < (int)blockDim.x / 32; q++) y += (double)s[q];
  return y;
}

// |F_ref|^2 summed over the atoms without a pair (their force is zero), for block b of nb: the
// reference forces stream in place, from host memory where the device reads it directly.
__device__ __forceinline__ float refSquares(const float *__restrict__ ref, int n, const unsigned char *__restrict__ paired,
                                            int b, int nb) {
  const long long n3 = 3LL * n;
  const bool aligned = (reinterpret_cast<uintptr_t>(ref) & 15) == 0;
  const long long n4 = aligned ? n3 / 4 : 0, stride = (long long)nb * blockDim.x;
  LongSum s;
  for (long long q = (long long)b * blockDim.x + threadIdx.x; q < n4; q += 2 * stride) {
    float4 v[2];
#pragma unroll
    for (int u = 0; u < 2; u++)
      v[u] = q + u * stride < n4 ? reinterpret_cast<const float4 *>(ref)[q + u * stride] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int u = 0; u < 2; u++) {
      // floats f .. f + 3 belong to atoms a and a + 1, split at atom a + 1's first float
      const long long f = min(4 * (q + u * stride), n3 - 1);
      const int a = (int)(f / 3), cut = (int)(3LL * (a + 1) - f);  // 1..3 floats of atom a
      // selected, not weighted with 0 and 1: a square may be infinite
      const bool wa = !paired[a], wb = a + 1 < n && !paired[a + 1];
      s.add((wa ? v[u].x * v[u].x : 0.f) + ((cut > 1 ? wa : wb) ? v[u].y * v[u].y : 0.f) +
            ((cut > 2 ? wa : wb) ? v[u].z * v[u].z : 0.f) + (wb ? v[u].w * v[u].w : 0.f));
    }
  }
  for (long long f = 4 * n4 + (long long)b * blockDim.x + threadIdx.x; f < n3; f += stride)
    if (!paired[f / 3]) s.add(ref[f] * ref[f]);
  return s.s;
}
__global__ void __launch_bounds__(kDT) k_diff_ref(const float *__restrict__ ref, int n,
                                                  const unsigned char *__restrict__ paired, double *__restrict__ lossPart) {
  const double s = blockSum(refSquares(ref, n, paired, blockIdx.x, gridDim.x));
  if (threadIdx.x == 0) lossPart[blockIdx.x] = s;
}

// Forces of the metal atoms (EAM and LJ) and of the paired carbon atoms (LJ), slices of the
// metal list first.  LOSS: the residual e = scale (F - F_ref) of each (resid, by slot; F_ref on
// entry) and sum |F - F_ref|^2 (sums), the last refBlocks blocks of the grid summing the atoms without
// a pair (refPart); else the forces, packed (out).
template <bool LOSS>
__global__ void __launch_bounds__(kPassThreads, kPassBlocks) k_diff_force(const DiffModel *__restrict__ model, const DiffWork *__restrict__ metal,
                                                    const DiffSlice *__restrict__ metalSlices, int nMetal,
                                                    const DiffWork *__restrict__ carbon,
                                                    const DiffSlice *__restrict__ carbonSlices, int nCarbon,
                                                    const int *__restrict__ sortIdx, DiffPairs pr,
                                                    const float2 *__restrict__ emb, float *__restrict__ out,
                                                    const float *__restrict__ ref, float scale,
                                                    float4 *__restrict__ resid, double *__restrict__ sums,
                                                    double *__restrict__ refPart, int n,
                                                    const unsigned char *__restrict__ paired, int refBlocks) {
  __shared__ __align__(16) DiffModel m;
  pdlEnter();
  const int grid = gridDim.x - refBlocks;
  if (LOSS && (int)blockIdx.x >= grid) {
    const double s = blockSum(refSquares(ref, n, paired, blockIdx.x - grid, refBlocks));
    if (threadIdx.x == 0) refPart[blockIdx.x - grid] = s;
    return;
  }
  const int metalN = (nMetal + 31) / 32, nSlices = metalN + (nCarbon + 31) / 32;
  auto atomOf = [&](int slice) {
    return slice < metalN ? diffAtom(metal, metalSlices, nMetal, slice)
                          : diffAtom(carbon, carbonSlices, nCarbon, slice - metalN);
  };
  DiffAtom next = atomOf(blockIdx.x);
  loadModel(model, m);
  LongSum loss;
  for (int slice = blockIdx.x, turn = 0; slice < nSlices; slice += grid, turn++) {
    const DiffAtom a = next;
    next = atomOf(slice + grid);
    float x[3] = {0.f, 0.f, 0.f};
    const float Fpi = a.ne ? emb[a.slot].x : 0.f;
    float4 D[kGathers];
    float Fk[kGathers];
    overPairs<kGathers>(
        a.first, a.ne, a.most,
        [&](int u, int p) {
          D[u] = pr.dir[p];
          Fk[u] = emb[pr.slot[p]].x;
        },
        [&](int u, int) {
          const int i = interval(m, D[u].w);
          const float s = D[u].w - m.knot[i].x;
          const float f = -(slope(m.phi[i], s) + slope(m.den[i], s) * (Fpi + Fk[u]));
          x[0] += f * D[u].x; x[1] += f * D[u].y; x[2] += f * D[u].z;
        });
    overPairs<kGathers>(
        a.first + 32 * a.most, a.nc, a.mostC, [&](int u, int p) { D[u] = pr.dir[p]; },
        [&](int u, int) {
          const float s6 = ljSix(m.sig6, D[u].w), s12 = s6 * s6;
          const float f = 24.f * m.eps * (2.f * s12 - s6) / D[u].w;  // -U'(r)
          x[0] += f * D[u].x; x[1] += f * D[u].y; x[2] += f * D[u].z;
        });
    sumParts(turn, x);
    if (threadIdx.x < 32 && a.slot >= 0) {
      if (LOSS) {
        const float4 want = resid[a.slot];
        const float ex = x[0] - want.x, ey = x[1] - want.y, ez = x[2] - want.z;
        resid[a.slot] = make_float4(scale * ex, scale * ey, scale * ez, 0.f);
        loss.add(ex * ex + ey * ey + ez * ez);
      } else {
        const size_t f = 3 * (size_t)sortIdx[a.slot];
        out[f] = x[0];
        out[f + 1] = x[1];
        out[f + 2] = x[2];
      }
    }
  }
  if (LOSS && threadIdx.x < 32) {
    const float all = warpSumF(loss.s);
    if (threadIdx.x == 0) atomicAdd(sumsCopy(sums) + kDP, (double)all);
  }
}

// Parameter sums.  A pair adds to four consecutive coefficients of each spline.  Every thread has
// a column of its own in shared memory ({phi, f} of coefficient c at [c][thread], 32 KB a block,
// no bank shared between lanes), so an addition is a plain load and store; a float atomicAdd in
// shared memory is a compare-and-swap loop whose lanes collide, since neighbours sit at few
// distances.  The blocks are few and walk many atoms, because each ends with 66 FP64 additions to
// the same 66 totals: a block per 8 atoms took 16,000 x 66 of them.
struct DiffSums {
  float2 c[kSC][kDT];
};
// A pair at interval coordinate t of interval k adds p0 b_m + p1 b'_m to phi's coefficient k + m
// and d0 b_m + d1 b'_m to f's: b, b' the B-spline weights at t and their t-derivatives.
template <bool VAL, bool DER>
__device__ __forceinline__ void addPair(DiffSums &S, int k, float t, float p0, float p1, float d0, float d1) {
  const float u = 1.f - t, t2 = t * t, u2 = u * u;
  const float b[4] = {u2 * (u * (1.f / 6.f)), fmaf(t2, fmaf(0.5f, t, -1.f), 2.f / 3.f),
                      fmaf(u2, fmaf(0.5f, u, -1.f), 2.f / 3.f), t2 * (t * (1.f / 6.f))};
  const float db[4] = {-0.5f * u2, t * fmaf(1.5f, t, -2.f), -u * fmaf(1.5f, u, -2.f), 0.5f * t2};
#pragma unroll
  for (int q = 0; q < 4; q++) {
    float2 v = S.c[k + q][threadIdx.x];
    if (VAL) v.x += p0 * b[q];
    if (DER) v.x += p1 * db[q];
    v.y += d0 * b[q];
    if (DER) v.y += d1 * db[q];
    S.c[k + q][threadIdx.x] = v;
  }
}
__device__ __forceinline__ void clearSums(DiffSums &S) {
#pragma unroll 8
  for (int q = 0; q < kSC; q++) S.c[q][threadIdx.x] = make_float2(0.f, 0.f);
}
// The block's columns into the totals.
__device__ __forceinline__ void flushSums(const DiffSums &S, double *__restrict__ grad) {
  __syncthreads();
  grad = sumsCopy(grad);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int q = w; q < kSC; q += kDT / 32) {
    float px = 0.f, py = 0.f;
#pragma unroll
    for (int u = 0; u < kDT / 32; u++) {
      const float2 v = S.c[q][lane + 32 * u];
      px += v.x;
      py += v.y;
    }
    px = warpSumF(px);
    py = warpSumF(py);
    if (lane == 0) {
      if (px != 0.f) atomicAdd(&grad[kPhi + q], (double)px);
      if (py != 0.f) atomicAdd(&grad[kDen + q], (double)py);
    }
  }
}

// The LJ parameters' share of an evaluation's gradient, and with LOSS what the metal pairs' share
// needs of each atom and pair: {F'(rho_i), F''(rho_i) g_i} (emb) and w (pr.w, pairs counted once).
template <bool LOSS>
__global__ void __launch_bounds__(kPassThreads, kPassBlocks) k_diff_along(const DiffModel *__restrict__ model, const DiffWork *__restrict__ metal,
                                                    const DiffSlice *__restrict__ slices, int nMetal, DiffPairs pr,
                                                    const float4 *__restrict__ resid, float2 *__restrict__ emb,
                                                    double *__restrict__ sums) {
  __shared__ __align__(16) DiffModel m;
  pdlEnter();
  const int nSlices = (nMetal + 31) / 32;
  DiffAtom next = diffAtom(metal, slices, nMetal, blockIdx.x);
  loadModel(model, m);
  LongSum sumE, sumS;
  for (int slice = blockIdx.x, turn = 0; slice < nSlices; slice += gridDim.x, turn++) {
    const DiffAtom a = next;
    next = diffAtom(metal, slices, nMetal, slice + gridDim.x);
    float ge = 0.f, gs = 0.f;  // the slice's
    if (LOSS) {
      const float4 Ei = a.slot >= 0 ? resid[a.slot] : make_float4(0.f, 0.f, 0.f, 0.f);
      const float Fdd = a.slot >= 0 ? emb[a.slot].y : 0.f;
      float x[1] = {0.f};  // g
      float4 D[kGathers], E[kGathers];
      auto load = [&](int u, int p) {
        D[u] = pr.dir[p];
        E[u] = resid[pr.slot[p]];
      };
      auto along = [&](int u) {  // w = rhat . (e_i - e_k)
        return D[u].x * (Ei.x - E[u].x) + D[u].y * (Ei.y - E[u].y) + D[u].z * (Ei.z - E[u].z);
      };
      overPairs<kGathers>(a.first, a.ne, a.most, load, [&](int u, int j) {
        const float w = along(u);
        const int i = interval(m, D[u].w);
        x[0] += slope(m.den[i], D[u].w - m.knot[i].x) * w;
        if (j < a.nh) pr.w[a.first + 32 * j + (threadIdx.x & 31)] = w;
      });
      overPairs<kGathers>(a.first + 32 * a.most, a.nc, a.mostC, load, [&](int u, int) {
        const float w = along(u);
        const float s6 = ljSix(m.sig6, D[u].w), s12 = s6 * s6;
        ge += 24.f * (s6 - 2.f * s12) / D[u].w * w;                          // dU'/d eps
        gs += 144.f * m.eps * (s6 - 4.f * s12) / D[u].w * m.invSig * w;  // dU'/d sigma
      });
      sumParts(turn, x);
      if (threadIdx.x < 32 && a.slot >= 0) emb[a.slot].y = Fdd * x[0];
    } else {
      float r[kLoads];
      overPairs<kLoads>(a.first + 32 * a.most, a.nc, a.mostC, [&](int u, int p) { r[u] = pr.r[p]; },
                       [&](int u, int) {
                         const float s6 = ljSix(m.sig6, r[u]), s12 = s6 * s6;
                         ge += 4.f * (s12 - s6);                                // dU / d eps
                         gs += 24.f * m.eps * (2.f * s12 - s6) * m.invSig;  // dU / d sigma
                       });
    }
    sumE.add(ge);
    sumS.add(gs);
  }
  const double e = blockSum(sumE.s), q = blockSum(sumS.s);
  if (threadIdx.x == 0 && e != 0.0) atomicAdd(sumsCopy(sums), e);
  if (threadIdx.x == 0 && q != 0.0) atomicAdd(sumsCopy(sums) + 1, q);
}

// w of the metal pairs counted once (pr.w) alone, where the pairs were laid out anew since k_diff_along.
__global__ void __launch_bounds__(kDT) k_diff_w(DiffPairs pr, int nPairs, const float4 *__restrict__ resid) {
  for (long long p = (long long)blockIdx.x * kDT + threadIdx.x; p < nPairs; p += (long long)gridDim.x * kDT) {
    const int2 k = pr.both[p];
    const int place = pr.place[p];
    const float4 D = pr.dir[place], Ei = resid[k.x], Ek = resid[k.y];
    pr.w[place] = D.x * (Ei.x - Ek.x) + D.y * (Ei.y - Ek.y) + D.z * (Ei.z - Ek.z);
  }
}

// The spline coefficients' share, a thread per metal pair counted once (its two sides' terms are
// alike: r and w are the same from both, and only F' and F'' g differ).
//   energy: phi B(r), f (F'_i + F'_j) B(r)
//   loss (LOSS; the adjoint of sum e . dE/dr): phi w B'(r), f (F''_i g_i + F''_j g_j) B(r) +
//   (F'_i + F'_j) w B'(r).
// ONE_SIDED: a side's terms of each entry, half of phi's and atom i's F' and F'' g.
constexpr int kSumLoads = 4;   // pairs a thread loads together
constexpr int kSumRounds = 8;  // rounds of them (32 pairs) after which the columns pass to the totals
template <bool LOSS, bool ONE_SIDED>
__global__ void __launch_bounds__(kDT) k_diff_sums(const DiffModel *__restrict__ model, DiffPairs pr, int nPairs,
                                                   const float2 *__restrict__ emb, double *__restrict__ grad) {
  __shared__ __align__(16) DiffModel m;
  __shared__ DiffSums S;
  clearSums(S);
  loadModel(model, m);
  pdlEnter();
  const int stride = gridDim.x * kDT;
  for (int b0 = blockIdx.x * kDT, round = 1; b0 < nPairs; b0 += kSumLoads * stride, round++) {
    const int p0 = b0 + threadIdx.x;
    float r[kSumLoads], w[kSumLoads];
    int at[kSumLoads];
    int2 k[kSumLoads];
    float2 a[kSumLoads], b[kSumLoads];
#pragma unroll
    for (int q = 0; q < kSumLoads; q++) {
      const int p = p0 + q * stride;
      if (p < nPairs) {
        k[q] = pr.both[p];
        r[q] = pr.rOnce[p];
        if (LOSS) at[q] = pr.place[p];
      }
    }
#pragma unroll
    for (int q = 0; q < kSumLoads; q++)
      if (p0 + q * stride < nPairs) {
        a[q] = emb[k[q].x];
        b[q] = ONE_SIDED ? make_float2(0.f, 0.f) : emb[k[q].y];
        if (LOSS) w[q] = pr.w[at[q]];
      }
#pragma unroll
    for (int q = 0; q < kSumLoads; q++) {
      if (p0 + q * stride >= nPairs) continue;
      const int i = interval(m, r[q]);
      const float t = fmaf(r[q] - m.knot[i].x, m.invH, m.knot[i].y), Fd = a[q].x + b[q].x;
      if (LOSS) {
        const float wh = w[q] * m.invH;
        addPair<false, true>(S, i, t, 0.f, ONE_SIDED ? 0.5f * wh : wh, a[q].y + b[q].y, Fd * wh);
      } else {
        addPair<true, false>(S, i, t, ONE_SIDED ? 0.5f : 1.f, 0.f, Fd, 0.f);
      }
    }
    if (round % kSumRounds == 0) {
      flushSums(S, grad);
      __syncthreads();
      clearSums(S);
    }
  }
  flushSums(S, grad);
}

// Most blocks of a pass: those resident at once.  Blocks of a second wave would start when the first
// has done nearly all the work.
template <typename K>
static int mostBlocks(K kernel, int threads, int numSMs) {
  int n = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, threads, 0) != cudaSuccess || n < 1) n = 1;
  return n * numSMs;
}
struct DiffGrids {
  int rho, energy, residual, force, along, lj, lossSums, energySums;
  explicit DiffGrids(int sms)
      : rho(mostBlocks(k_diff_rho<false>, kPassThreads, sms)), energy(mostBlocks(k_diff_rho<true>, kPassThreads, sms)),
        residual(mostBlocks(k_diff_force<true>, kPassThreads, sms)), force(mostBlocks(k_diff_force<false>, kPassThreads, sms)),
        along(mostBlocks(k_diff_along<true>, kPassThreads, sms)), lj(mostBlocks(k_diff_along<false>, kPassThreads, sms)),
        lossSums(mostBlocks(k_diff_sums<true, false>, kDT, sms)),
        energySums(mostBlocks(k_diff_sums<false, false>, kDT, sms)) {}
};

}  // namespace sg

using namespace sg;

// A run of slices whose pairs are laid out together: the first atom (a multiple of 32) and the number of
// atoms of each work list, and the metal pairs counted once.
struct DiffBatch {
  int metal, nMetal, carbon, nCarbon, nOnce;
};
// Most places of pairs laid out at once: they and the threads' strides over them are 32-bit numbers.
constexpr unsigned long long kMostPlaces = (1ull << 31) - (1ull << 24);

struct sg_diff {
  sg_ctx *ctx = nullptr;
  int nFrames = 0, n = 0;
  DiffGrids most;
  explicit sg_diff(int sms) : most(sms) {}
  double r0 = 0, h = 0;  // first knot and interval width of the splines
  bool listed = false;                          // has work lists (of positions, or of none yet)
  bool oneSided = false;                        // rows were truncated: a pair may be in one of two only
  void *arena = nullptr, *pairArena = nullptr, *pinned = nullptr;  // what the arrays below lie in
  int *slotOf = nullptr;                        // slot of each atom
  unsigned char *paired = nullptr;              // per atom: has a slot in a work list
  DiffWork *metal = nullptr, *carbon = nullptr;  // the work lists and their slices
  DiffSlice *metalSlices = nullptr, *carbonSlices = nullptr;
  int *counts = nullptr, nMetal = 0;
  unsigned long long *totals = nullptr;         // places of all pairs, metal pairs counted once
  int4 *seg = nullptr;                          // per slot: its row's segments (k_diff_pack)
  DiffPairs pairs{};
  unsigned long long pairCap = 0, onceCap = 0;  // pairs the arrays hold
  // One batch of all slices, laid out with the positions; or several, where that is more than memory
  // holds, that each pass lays out in turn.
  std::vector<DiffBatch> batches;
  unsigned long long mostPlaces = kMostPlaces;
  int broken = SG_OK;                           // what the last set of positions failed with: no lists
  float2 *emb = nullptr;                        // per slot: F', then F'' or F'' g
  float4 *resid = nullptr;                      // per slot
  // results on the device and page-locked on the host: the copies of the sums, then the
  // frame energies or the sums of squares of the blocks of k_diff_ref
  double *out = nullptr, *hostOut = nullptr;
  DiffModel *model = nullptr, *hostModel = nullptr;  // of the call, on the device and page-locked
  int outCap = 0;
};

#define DCK(call)                                                                              \
  do {                                                                                         \
    cudaError_t e_ = (call);                                                                   \
    if (e_ != cudaSuccess) return sg_fail(SG_ERR_CUDA, "%s: %s", #call, cudaGetErrorString(e_)); \
  } while (0)

// phi(r) and f(r) of the Zhou-Wadley-Johnson forms (SurfaceGrowth.cu:46-69) in FP64
static void eamAnalytic(const sg_simparams &p, double r, double &phi, double &f) {
  const double x = r * p.rei;
  const double eA = std::exp(-(double)p.alpha * (x - 1.0)), eB = std::exp(-(double)p.beta * (x - 1.0));
  const double dA = 1.0 + std::pow(x - p.kappa, 20.0), dB = 1.0 + std::pow(x - p.lambda, 20.0);
  phi = p.A * eA / dA - p.B * eB / dB;
  f = p.fe * eB / dB;
}

// First knot and interval width of a metal's splines.
static void splineKnots(const sg_simparams &p, double &r0, double &h) {
  r0 = 0.6 / p.rei;
  h = (std::sqrt((double)p.rrCutEam) - r0) / kSI;
}

extern "C" int sg_diff_frame_params(const sg_simparams *in, sg_simparams *out) {
  if (!in || !out) return sg_fail(SG_ERR_INVALID, "sg_diff_frame_params: null argument");
  sg_simparams q = *in;
  const double rl = std::sqrt((double)std::max(q.rrCutEam, q.rrCutLJ));
  q.rrNebr = std::max(q.rrCutEam, q.rrCutLJ);
  q.cells.x = (int)(q.region.x / rl);
  q.cells.y = (int)(q.region.y / rl);
  q.cells.z = (int)(q.region.z / rl);
  if (q.cells.x < 3 || q.cells.y < 3 || q.cells.z < 3)
    return sg_fail(SG_ERR_INVALID, "box too small for the LJ cutoff (fewer than 3 cells in a direction)");
  q.invWidth = sg_float3{q.cells.x / q.region.x, q.cells.y / q.region.y, q.cells.z / q.region.z};
  q.gridSize = (unsigned)(q.cells.x * q.cells.y * q.cells.z);
  q.maxMol = (int)q.gridSize * (int)q.blockSize;
  q.iNebrMax = std::max(q.iNebrMax, 192);
  q.nebrNow = 1;
  *out = q;
  return SG_OK;
}

// Blocks per SM that stream the reference forces of atoms without a pair: 2 keep the host link
// busy and leave the SMs to the passes that run beside them.
constexpr int kRefBlocks = 2;
// From this many atoms the stream gets a launch of its own beside the passes; below, it is a few
// blocks of the force pass, which saves the launch and two event waits.  A fit's evaluation of frames of
// 6,444 atoms (300 metal), launch of its own / blocks of the force pass: 12,888 atoms 47.3 / 44.8 us,
// 64,440 atoms 50.9 / 47.1, 103,104 atoms 58.7 / 50.9, 206,208 atoms 59.5 / 61.2; 1.3 million atoms 204 in
// its own launch.  With these frames the two meet near 180,000 atoms.
constexpr int kRefOwnLaunch = 65536;

// The sums of an evaluation just read back.
static double sumOf(const sg_diff *d, int q) {
  double s = 0.0;
  for (int c = 0; c < kSumCopies; c++) s += d->hostOut[c * kSumStride + q];
  return s;
}

// Lays arrays out one after another (256-byte aligned) from base on; with base null only counts.
struct Carver {
  char *base;
  size_t used = 0;
  template <typename T> void take(T *&p, size_t n) {
    if (base) p = reinterpret_cast<T *>(base + used);
    used += (n * sizeof(T) + 255) & ~size_t(255);
  }
};

static void freePairs(sg_diff *d) {
  cudaFree(d->pairArena);
  d->pairArena = nullptr;
  d->pairCap = d->onceCap = 0;
}
// Memory for the arrays of so many pairs and metal pairs counted once, in place of what there was.
static bool pairMemory(sg_diff *d, unsigned long long all, unsigned long long once) {
  auto lay = [&](Carver v) {
    v.take(d->pairs.dir, all);
    v.take(d->pairs.slot, all);
    v.take(d->pairs.r, all);
    v.take(d->pairs.w, all);
    v.take(d->pairs.both, once);
    v.take(d->pairs.rOnce, once);
    v.take(d->pairs.place, once);
    return v.used;
  };
  freePairs(d);
  if (cudaMalloc(&d->pairArena, lay(Carver{nullptr})) != cudaSuccess) {
    cudaGetLastError();
    d->pairArena = nullptr;
    return false;
  }
  lay(Carver{static_cast<char *>(d->pairArena)});
  d->pairCap = all;
  d->onceCap = once;
  return true;
}
constexpr size_t kPlaceBytes = sizeof(float4) + sizeof(int) + 2 * sizeof(float);   // dir, slot, r, w
constexpr size_t kOnceBytes = sizeof(int2) + sizeof(float) + sizeof(int);          // both, rOnce, place

// The pairs of a batch into the arrays.
static int layPairs(sg_diff *d, const DiffBatch &b) {
  sg_ctx *c = d->ctx;
  const DiffWork *lists[2] = {d->metal + b.metal, d->carbon + b.carbon};
  const DiffSlice *slices[2] = {d->metalSlices + b.metal / 32, d->carbonSlices + b.carbon / 32};
  const int n[2] = {b.nMetal, b.nCarbon};
  for (int l = 0; l < 2; l++)
    if (n[l])
      k_diff_pairs<<<(n[l] + kDT / 32 - 1) / (kDT / 32), kDT, 0, c->stream>>>(lists[l], slices[l], n[l], c->rc, c->sortPos,
                                                                              c->nbl, c->rowStride, d->pairs);
  if (b.nOnce) k_diff_once<<<(n[0] + kDT - 1) / kDT, kDT, 0, c->stream>>>(lists[0], slices[0], n[0], d->pairs);
  DCK(cudaGetLastError());
  return SG_OK;
}

// The slices in batches that fit the memory there is (n: the atoms of the two work lists; needed: places
// of all pairs), each batch's slices numbered from its own first place.
static int splitPairs(sg_diff *d, const int n[2], unsigned long long needed) {
  sg_ctx *c = d->ctx;
  DiffWork *lists[2] = {d->metal, d->carbon};
  DiffSlice *slices[2] = {d->metalSlices, d->carbonSlices};
  std::vector<DiffSlice> all((n[0] + 31) / 32 + (n[1] + 31) / 32);  // metal slices first
  const int metalN = (n[0] + 31) / 32;
  DCK(cudaMemcpyAsync(all.data(), slices[0], sizeof(DiffSlice) * metalN, cudaMemcpyDeviceToHost, c->stream));
  DCK(cudaMemcpyAsync(all.data() + metalN, slices[1], sizeof(DiffSlice) * (all.size() - metalN), cudaMemcpyDeviceToHost,
                      c->stream));
  DCK(cudaStreamSynchronize(c->stream));
  auto places = [](const DiffSlice &s) { return 32ull * (s.most + s.mostC); };
  unsigned long long largest = 1;
  for (const DiffSlice &s : all) largest = std::max(largest, places(s));
  freePairs(d);
  size_t freeBytes = 0, total = 0;
  DCK(cudaMemGetInfo(&freeBytes, &total));
  // nine tenths of what is free, and less where that cannot be had in one piece; every place may be of a
  // metal pair counted once
  unsigned long long cap = std::min<unsigned long long>(freeBytes / (kPlaceBytes + kOnceBytes) / 10 * 9,
                                                        std::min(d->mostPlaces, needed));
  for (; cap >= largest && !pairMemory(d, cap, cap); cap /= 2) {
  }
  if (cap < largest) return sg_fail(SG_ERR_NOMEM, "sg_diff: memory for %llu pairs", largest);
  d->batches.clear();
  for (size_t s = 0; s < all.size();) {
    const size_t s0 = s;
    for (unsigned long long sum = 0; s < all.size() && sum + places(all[s]) <= cap; s++) sum += places(all[s]);
    const int m0 = 32 * (int)std::min(s0, (size_t)metalN), m1 = std::min(32 * (int)std::min(s, (size_t)metalN), n[0]);
    const int c0 = 32 * (int)(std::max(s0, (size_t)metalN) - metalN);
    const int c1 = std::min(32 * (int)(std::max(s, (size_t)metalN) - metalN), n[1]);
    d->batches.push_back(DiffBatch{m0, std::max(m1 - m0, 0), c0, std::max(c1 - c0, 0), 0});
  }
  for (DiffBatch &b : d->batches) {
    const int at[2] = {b.metal, b.carbon}, count[2] = {b.nMetal, b.nCarbon};
    DCK(cudaMemsetAsync(d->totals, 0, 2 * sizeof(unsigned long long), c->stream));
    for (int l = 0; l < 2; l++)
      if (count[l])
        k_diff_slices<<<(count[l] + kDT - 1) / kDT, kDT, 0, c->stream>>>(lists[l] + at[l], count[l], slices[l] + at[l] / 32,
                                                                         d->totals);
    DCK(cudaGetLastError());
    unsigned long long pairs[2];
    DCK(cudaMemcpyAsync(pairs, d->totals, sizeof pairs, cudaMemcpyDeviceToHost, c->stream));
    DCK(cudaStreamSynchronize(c->stream));
    b.nOnce = (int)pairs[1];
  }
  return d->batches.size() == 1 ? layPairs(d, d->batches[0]) : SG_OK;
}

// The packed rows, work lists and pairs of the positions and lists of d's context (built: it has
// lists; truncated: not all of them whole).
static int packLists(sg_diff *d, bool built, bool truncated) try {
  sg_ctx *c = d->ctx;
  d->oneSided = truncated;
  DCK(cudaMemsetAsync(d->paired, 0, d->n, c->stream));
  DCK(cudaMemsetAsync(d->counts, 0, 2 * sizeof(int), c->stream));
  DCK(cudaMemsetAsync(d->totals, 0, 2 * sizeof(unsigned long long), c->stream));
  DCK(cudaMemsetAsync(d->slotOf, 0xff, sizeof(int) * d->n, c->stream));
  if (built) {
    k_diff_slots<<<c->atomTab.n, 128, 0, c->stream>>>(c->atomTab.view(), c->rc, c->cellStart, c->sortIdx, d->slotOf);
    // a row's entries per warp in shared memory: one warp a block where they are very many.  A row has
    // fewer than its frame has atoms, and what the longest one has is looked up only where that, too,
    // is more than a block can hold.
    constexpr int kMostRest = 227 * 1024 / sizeof(int);
    int rest = 1;
    for (const RepConst &P : c->hrc) rest = std::max(rest, std::min(c->rowStride, P.nMol));
    if (rest > kMostRest) {
      int longest = 1;
      for (int f = 0; f < d->nFrames; f++) {
        RepState S;
        if (int rc = sg_read_state(c, f, &S)) return rc;
        longest = std::max(longest, S.maxNeighbours);
      }
      rest = std::min(rest, longest);
    }
    const int warps = rest <= 3072 ? kDT / 32 : 1;
    const size_t smem = sizeof(int) * warps * rest;
    if (smem > 48 * 1024)
      DCK(cudaFuncSetAttribute(k_diff_pack, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    k_diff_pack<<<c->atomTab.n * (128 / warps), 32 * warps, smem, c->stream>>>(
        c->atomTab.view(), c->rc, c->pos, c->nn, d->slotOf, c->nbl, c->rowStride, rest, d->seg, d->paired, truncated);
  }
  k_diff_lists<<<c->atomTab.n, 128, 0, c->stream>>>(c->atomTab.view(), c->rc, c->cellStart, c->sortIdx, d->slotOf, built,
                                                    d->paired, d->seg, d->metal, d->carbon, d->counts);
  DCK(cudaGetLastError());
  int counts[2];
  DCK(cudaMemcpyAsync(counts, d->counts, sizeof counts, cudaMemcpyDeviceToHost, c->stream));
  DCK(cudaStreamSynchronize(c->stream));
  DiffWork *lists[2] = {d->metal, d->carbon};
  DiffSlice *slices[2] = {d->metalSlices, d->carbonSlices};
  for (int l = 0; l < 2; l++)
    if (counts[l])
      k_diff_slices<<<(counts[l] + kDT - 1) / kDT, kDT, 0, c->stream>>>(lists[l], counts[l], slices[l], d->totals);
  DCK(cudaGetLastError());
  unsigned long long pairs[2];
  DCK(cudaMemcpyAsync(pairs, d->totals, sizeof pairs, cudaMemcpyDeviceToHost, c->stream));
  DCK(cudaStreamSynchronize(c->stream));
  d->nMetal = counts[0];
  if (pairs[0] <= d->mostPlaces) {
    // an eighth more than asked: a later set of positions rarely has as many more
    if ((pairs[0] <= d->pairCap && pairs[1] <= d->onceCap) ||
        pairMemory(d, pairs[0] + pairs[0] / 8 + 1, pairs[1] + pairs[1] / 8 + 1)) {
      d->batches.assign(1, DiffBatch{0, counts[0], 0, counts[1], (int)pairs[1]});
      return built ? layPairs(d, d->batches[0]) : SG_OK;
    }
  }
  return splitPairs(d, counts, pairs[0]);
} catch (const std::bad_alloc &) {
  return sg_fail(SG_ERR_NOMEM, "sg_diff: host memory for the batches of pairs");
}
// The same; without lists, every evaluation returns the error until a set of positions has them again.
static int setLists(sg_diff *d, bool built, bool truncated) {
  d->broken = packLists(d, built, truncated);
  d->listed = d->broken == SG_OK;
  return d->broken;
}

// Most places of pairs laid out at once, for the sets of positions to come (0: as many as there can be).
int sg_diff_limit_places(sg_diff *d, unsigned long long places) {
  d->mostPlaces = places && places < kMostPlaces ? places : kMostPlaces;
  return SG_OK;
}

extern "C" int sg_diff_create(const sg_simparams *frames, int n, int device, sg_diff **out) {
  if (!frames || n < 1 || !out) return sg_fail(SG_ERR_INVALID, "sg_diff_create: bad arguments");
  *out = nullptr;
  std::vector<sg_simparams> q(n);
  for (int f = 0; f < n; f++) {
    if (frames[f].rei != frames[0].rei || frames[f].rrCutEam != frames[0].rrCutEam)
      return sg_fail(SG_ERR_INVALID, "sg_diff_create: frames must share the metal");
    if (int rc = sg_diff_frame_params(&frames[f], &q[f])) return rc;
  }
  sg_options o;
  sg_default_options(&o);
  o.use_graphs = 0;
  o.force_rebuild = 1;
  o.device = device;
  sg_ctx *c = nullptr;
  if (int rc = sg_create(q.data(), n, &o, &c)) return rc;
  size_t M = 0;
  for (const RepConst &P : c->hrc) M += P.nMolMe;
  sg_diff *d = new sg_diff(c->numSMs);
  d->ctx = c;
  d->nFrames = n;
  d->n = sg_num_atoms(c, -1);
  splineKnots(q[0], d->r0, d->h);
  const size_t N = d->n;
  d->outCap = kSums + std::max(n, c->numSMs * kRefBlocks);
  auto lay = [&](Carver v) {
    v.take(d->metal, M + 32);
    v.take(d->carbon, N + 32);
    v.take(d->metalSlices, M / 32 + 1);
    v.take(d->carbonSlices, N / 32 + 1);
    v.take(d->seg, N);
    v.take(d->emb, N);
    v.take(d->resid, N);
    v.take(d->slotOf, N);
    v.take(d->paired, N);
    v.take(d->counts, 2);
    v.take(d->totals, 2);
    v.take(d->out, d->outCap);
    v.take(d->model, 1);
    return v.used;
  };
  auto layHost = [&](Carver v) {
    v.take(d->hostModel, 1);
    v.take(d->hostOut, d->outCap);
    return v.used;
  };
  cudaError_t e = cudaMalloc(&d->arena, lay(Carver{nullptr}));
  if (e == cudaSuccess) e = cudaMallocHost(&d->pinned, layHost(Carver{nullptr}));
  if (e != cudaSuccess) {
    sg_diff_destroy(d);
    return sg_fail(SG_ERR_NOMEM, "sg_diff_create: %s", cudaGetErrorString(e));
  }
  lay(Carver{static_cast<char *>(d->arena)});
  layHost(Carver{static_cast<char *>(d->pinned)});
  *out = d;
  return SG_OK;
}

extern "C" int sg_diff_destroy(sg_diff *d) {
  if (!d) return SG_OK;
  cudaFree(d->arena);
  cudaFree(d->pairArena);
  cudaFreeHost(d->pinned);
  if (d->ctx) sg_destroy(d->ctx);
  delete d;
  return SG_OK;
}

extern "C" int sg_diff_num_atoms(const sg_diff *d) { return d ? d->n : 0; }

extern "C" int sg_diff_set_positions(sg_diff *d, const sg_float4 *r) {
  if (!d || !r) return sg_fail(SG_ERR_INVALID, "sg_diff_set_positions: null argument");
  if (int rc = sg_set_state(d->ctx, -1, r, nullptr, nullptr)) return rc;
  const int built = sg_build_lists(d->ctx);  // a list that overflowed is used truncated
  const std::string why = built ? sg_last_error() : "";
  if (int rc = setLists(d, true, built != SG_OK)) return rc;
  return built ? sg_fail(built, "%s", why.c_str()) : SG_OK;
}

extern "C" int sg_diff_init_theta(const sg_simparams *pp, double *theta) {
  if (!pp || !theta) return sg_fail(SG_ERR_INVALID, "sg_diff_init_theta: null argument");
  const sg_simparams &p = *pp;
  theta[0] = p.epsLJ;
  theta[1] = p.sigmaLJ;
  // least squares on 40 points per interval, normal equations solved by Cholesky in FP64
  double r0, h;
  splineKnots(p, r0, h);
  const int ns = 40 * kSI;
  std::vector<double> M(kSC * kSC, 0.0), rp(kSC, 0.0), rf(kSC, 0.0);
  for (int s = 0; s < ns; s++) {
    const double r = r0 + (s + 0.5) * (kSI * h) / ns;
    const double x = (r - r0) / h;
    const int k = std::max(0, std::min((int)std::floor(x), kSI - 1));
    const double t = x - k, u = 1.0 - t;
    const double b[4] = {u * u * u / 6, (3 * t * t * t - 6 * t * t + 4) / 6,
                         (-3 * t * t * t + 3 * t * t + 3 * t + 1) / 6, t * t * t / 6};
    double phi, f;
    eamAnalytic(p, r, phi, f);
    for (int a = 0; a < 4; a++) {
      rp[k + a] += b[a] * phi;
      rf[k + a] += b[a] * f;
      for (int c2 = 0; c2 < 4; c2++) M[(k + a) * kSC + k + c2] += b[a] * b[c2];
    }
  }
  for (int j = 0; j < kSC; j++) {  // Cholesky M = L L^T in place (lower triangle)
    for (int k = 0; k < j; k++) M[j * kSC + j] -= M[j * kSC + k] * M[j * kSC + k];
    M[j * kSC + j] = std::sqrt(M[j * kSC + j]);
    for (int i = j + 1; i < kSC; i++) {
      for (int k = 0; k < j; k++) M[i * kSC + j] -= M[i * kSC + k] * M[j * kSC + k];
      M[i * kSC + j] /= M[j * kSC + j];
    }
  }
  for (int which = 0; which < 2; which++) {
    std::vector<double> y = which == 0 ? rp : rf;
    for (int i = 0; i < kSC; i++) {
      for (int k = 0; k < i; k++) y[i] -= M[i * kSC + k] * y[k];
      y[i] /= M[i * kSC + i];
    }
    for (int i = kSC - 1; i >= 0; i--) {
      for (int k = i + 1; k < kSC; k++) y[i] -= M[k * kSC + i] * y[k];
      y[i] /= M[i * kSC + i];
    }
    for (int i = 0; i < kSC; i++) theta[(which == 0 ? kPhi : kDen) + i] = y[i];
  }
  return SG_OK;
}

// theta as the kernels read it, on its way to the device.  (Every call ends with its stream empty, so
// the page-locked copy is free again.)
static int uploadModel(sg_diff *d, const double *theta) {
  if (d->broken) return sg_fail(d->broken, "sg_diff: no pair lists, sg_diff_set_positions failed");
  if (!d->listed)  // no positions yet: every metal atom without a pair
    if (int rc = setLists(d, false, false)) return rc;
  DiffModel &m = *d->hostModel;
  m.r0 = (float)d->r0;
  m.invH = (float)(1.0 / d->h);
  m.eps = (float)theta[0];
  m.sig6 = (float)std::pow(theta[1], 6.0);
  m.invSig = (float)(1.0 / theta[1]);
  for (int k = 0; k < kSI; k++) {
    const float knot = (float)(d->r0 + k * d->h);
    const double t = (knot - d->r0) / d->h - k;  // the knot's own interval coordinate
    m.knot[k] = make_float2(knot, (float)t);
    for (int s = 0; s < 2; s++) {
      // the B-spline sum of the interval as a cubic in t, moved to the rounded knot, per length
      const double *c = theta + (s == 0 ? kPhi : kDen) + k;
      const double a0 = (c[0] + 4.0 * c[1] + c[2]) / 6.0, a1 = (c[2] - c[0]) / 2.0, a2 = (c[0] - 2.0 * c[1] + c[2]) / 2.0,
                   a3 = (c[3] - c[0] + 3.0 * (c[1] - c[2])) / 6.0;
      (s == 0 ? m.phi : m.den)[k] = make_float4((float)(a0 + t * (a1 + t * (a2 + t * a3))), (float)((a1 + t * (2.0 * a2 + 3.0 * t * a3)) / d->h),
                                 (float)((a2 + 3.0 * t * a3) / (d->h * d->h)), (float)(a3 / (d->h * d->h * d->h)));
    }
  }
  DCK(cudaMemcpyAsync(d->model, &m, sizeof m, cudaMemcpyHostToDevice, d->ctx->stream));
  return SG_OK;
}

// Slices of a work list of n atoms, a block each.
static int slicesOf(int n) { return (n + 31) / 32; }

// f(batch) for every batch, its pairs in the arrays.
template <typename F> static int overBatches(sg_diff *d, F f) {
  for (const DiffBatch &b : d->batches) {
    if (d->batches.size() > 1)
      if (int rc = layPairs(d, b)) return rc;
    if (int rc = f(b)) return rc;
  }
  return SG_OK;
}

// F'(rho) of the metal atoms, then the forces: packed into `force`, or (ref) the residuals and the
// loss, with refBlocks blocks for the atoms without a pair (their sums at out + kSums) in the same
// launch or (own) in one on the side stream.  That one starts when the reference forces of the atoms
// with pairs are there: a fetch beside it would share the host link and hold up the force pass by
// most of the transfer (64 frames of 20,432 atoms: 281 us an evaluation instead of 236).
static int forces(sg_diff *d, float *force, const float *ref, float scale, int refBlocks, bool own) {
  sg_ctx *c = d->ctx;
  // k_diff_rho also clears the sums, so it runs (one block) without metal too
  int refGather = ref ? std::min((d->n + kPassThreads - 1) / kPassThreads, c->numSMs * kRefBlocks) : 0;
  int rc = overBatches(d, [&](const DiffBatch &b) {
    DCK(launchK(false, k_diff_rho<false>, std::max(1, std::min(slicesOf(b.nMetal), d->most.rho) + refGather), kPassThreads, 0,
                c->stream, d->model, d->metal + b.metal, d->metalSlices + b.metal / 32, b.nMetal, c->rc, d->pairs.r, d->emb,
                nullptr, d->out, ref, d->n, d->paired, d->slotOf, d->resid, refGather));
    refGather = 0;  // with the first batch
    return (int)SG_OK;
  });
  if (rc) return rc;
  if (own) {
    DCK(cudaEventRecord(c->evFork, c->stream));
    DCK(cudaStreamWaitEvent(c->side, c->evFork, 0));
    k_diff_ref<<<refBlocks, kDT, 0, c->side>>>(ref, d->n, d->paired, d->out + kSums);
    DCK(cudaGetLastError());
    DCK(cudaEventRecord(c->evJoin, c->side));
    refBlocks = 0;
  }
  return overBatches(d, [&](const DiffBatch &b) {
    const int blocks =
        std::min(slicesOf(b.nMetal) + slicesOf(b.nCarbon), ref ? d->most.residual : d->most.force) + refBlocks;
    if (blocks > 0)
      DCK(launchK(true, ref ? k_diff_force<true> : k_diff_force<false>, blocks, kPassThreads, 0, c->stream, d->model,
                  d->metal + b.metal, d->metalSlices + b.metal / 32, b.nMetal, d->carbon + b.carbon,
                  d->carbonSlices + b.carbon / 32, b.nCarbon, c->sortIdx, d->pairs, d->emb, force, ref, scale, d->resid,
                  d->out, d->out + kSums, d->n, d->paired, refBlocks));
    refBlocks = 0;  // with the first batch
    return (int)SG_OK;
  });
}

// The parameter sums of an energy or loss evaluation, after its densities (and residuals).
template <bool LOSS>
static int parameterSums(sg_diff *d) {
  sg_ctx *c = d->ctx;
  auto along = [&](const DiffBatch &b) {
    if (b.nMetal)
      DCK(launchK(true, k_diff_along<LOSS>, std::min(slicesOf(b.nMetal), LOSS ? d->most.along : d->most.lj), kPassThreads, 0,
                  c->stream, d->model, d->metal + b.metal, d->metalSlices + b.metal / 32, b.nMetal, d->pairs, d->resid,
                  d->emb, d->out));
    return (int)SG_OK;
  };
  auto sums = [&](const DiffBatch &b) {
    const int most = LOSS ? d->most.lossSums : d->most.energySums, blocks = std::min((b.nOnce + kDT - 1) / kDT, most);
    if (b.nOnce && LOSS && d->batches.size() > 1) k_diff_w<<<blocks, kDT, 0, c->stream>>>(d->pairs, b.nOnce, d->resid);
    if (b.nOnce)
      DCK(launchK(true, d->oneSided ? k_diff_sums<LOSS, true> : k_diff_sums<LOSS, false>, blocks, kDT, 0, c->stream, d->model,
                  d->pairs, b.nOnce, d->emb, d->out));
    return (int)SG_OK;
  };
  if (d->batches.size() == 1 || !LOSS)
    return overBatches(d, [&](const DiffBatch &b) {
      const int rc = along(b);
      return rc ? rc : sums(b);
    });
  // the sums need F'' g of both atoms of a pair, which may lie in different batches
  const int rc = overBatches(d, along);
  return rc ? rc : overBatches(d, sums);
}

extern "C" int sg_diff_energy(sg_diff *d, const double *theta, double *energy, double *grad) {
  if (!d || !theta) return sg_fail(SG_ERR_INVALID, "sg_diff_energy: null argument");
  sg_ctx *c = d->ctx;
  if (int rc = uploadModel(d, theta)) return rc;
  const size_t bytes = sizeof(double) * (kSums + d->nFrames);
  DCK(cudaMemsetAsync(d->out, 0, bytes, c->stream));
  if (d->nMetal) {
    int rc = overBatches(d, [&](const DiffBatch &b) {
      if (b.nMetal)
        DCK(launchK(false, k_diff_rho<true>, std::min(slicesOf(b.nMetal), d->most.energy), kPassThreads, 0, c->stream,
                    d->model, d->metal + b.metal, d->metalSlices + b.metal / 32, b.nMetal, c->rc, d->pairs.r, d->emb,
                    d->out + kSums, d->out, nullptr, d->n, d->paired, d->slotOf, d->resid, 0));
      return (int)SG_OK;
    });
    if (!rc && grad) rc = parameterSums<false>(d);
    if (rc) return rc;
  }
  DCK(cudaMemcpyAsync(d->hostOut, d->out, bytes, cudaMemcpyDeviceToHost, c->stream));
  DCK(cudaStreamSynchronize(c->stream));
  if (energy) memcpy(energy, d->hostOut + kSums, sizeof(double) * d->nFrames);
  if (grad)
    for (int q = 0; q < kDP; q++) grad[q] = sumOf(d, q);
  return SG_OK;
}

extern "C" int sg_diff_forces(sg_diff *d, const double *theta, float *out) {
  if (!d || !theta || !out) return sg_fail(SG_ERR_INVALID, "sg_diff_forces: null argument");
  sg_ctx *c = d->ctx;
  DCK(cudaMemsetAsync(c->stage, 0, sizeof(float) * 3 * d->n, c->stream));  // atoms without a pair
  if (int rc = uploadModel(d, theta)) return rc;
  if (int rc = forces(d, c->stage, nullptr, 0.f, 0, false)) return rc;
  sg_populate(out, sizeof(float) * 3 * d->n);  // while the passes run
  DCK(cudaMemcpyAsync(out, c->stage, sizeof(float) * 3 * d->n, cudaMemcpyDeviceToHost, c->stream));
  DCK(cudaStreamSynchronize(c->stream));
  return SG_OK;
}

// The reference forces are read in place where the device reads host memory directly (their
// transfer then overlaps the passes: only the paired atoms' are needed early), else, or at an address
// that is no multiple of four, copied first.
extern "C" int sg_diff_force_matching(sg_diff *d, const double *theta, const float *ref, double *loss,
                                      double *grad) {
  if (!d || !theta || !ref) return sg_fail(SG_ERR_INVALID, "sg_diff_force_matching: null argument");
  sg_ctx *c = d->ctx;
  if (int rc = uploadModel(d, theta)) return rc;
  const double inv3N = 1.0 / (3.0 * d->n);
  const float *src = ref;
  if (!c->hostDirect || (reinterpret_cast<uintptr_t>(ref) & 3) != 0) {
    DCK(cudaMemcpyAsync(c->stage, ref, sizeof(float) * 3 * d->n, cudaMemcpyHostToDevice, c->stream));
    src = c->stage;
  }
  const bool own = d->n >= kRefOwnLaunch;
  const int refBlocks = std::max(1, std::min((d->n * 3 / 4 + kDT - 1) / kDT, c->numSMs * kRefBlocks));
  int rc = forces(d, nullptr, src, (float)(2.0 * inv3N), refBlocks, own);
  if (!rc && grad) rc = parameterSums<true>(d);
  // joined whatever happened: the stream reads the caller's array until k_diff_ref is done
  if (own) DCK(cudaStreamWaitEvent(c->stream, c->evJoin, 0));
  if (!rc) DCK(cudaMemcpyAsync(d->hostOut, d->out, sizeof(double) * (kSums + refBlocks), cudaMemcpyDeviceToHost, c->stream));
  DCK(cudaStreamSynchronize(c->stream));
  if (rc) return rc;
  if (loss) {
    double s = sumOf(d, kDP);
    for (int b = 0; b < refBlocks; b++) s += d->hostOut[kSums + b];
    *loss = s * inv3N;
  }
  if (grad)
    for (int q = 0; q < kDP; q++) grad[q] = -sumOf(d, q);  // dL/dtheta = -dD/dtheta
  return SG_OK;
}
