// Differentiable decode: the real-valued decode operator D and its adjoint D^T on sm_100a.
//
// D maps the dequantised zfp-domain coefficients of every brick to the decoded grid, the
// reference decode (Core/idx2Decode.cpp:141-320) with the integer inverse zfp replaced by its
// real counterpart (Core/Zfp.h:181 ILift with exact halvings in place of the arithmetic shifts;
// the bit-exact decode differs from D only by those floors, about 2^(EMax-59) per block):
//   per level, coarsest first, per brick: the parent's values on the low band
//   (Core/idx2Decode.cpp:285-293), the inverse zfp of every coded block written over them (in
//   3D the full low-band blocks are not coded below the coarsest level and the rest lie outside
//   the parent's 16^3 part; in 2D every low-band block is coded on every level,
//   Core/idx2Decode.cpp:126-130 against BlockDims3 = 4^3, so the parent's values are all
//   overwritten), de-normalisation and the one-level inverse CDF5/3 along each axis
//   (Core/Wavelet.cpp:144-203), then the brick goes to its children or, on the finest level,
//   to the grid.
// D is linear; D^T applies the transposed steps in the reverse order, finest level first, the
// low-band gradient of every child flowing into its parent's gradient brick (children cover
// disjoint 16^3 parts of the parent).
//
// Coefficient tensor of one field: levels 0 (finest) .. L-1; on each level the bricks in
// row-major order of their coordinates (x fastest); each brick 33^3 values (33^2 for 2D)
// indexed (z * 33 + y) * 33 + x, the coefficient of a block at the position of the sample it
// transforms (natural order inside the block). Positions of blocks that are not coded on a
// level (3D: the full low-band blocks below the coarsest level) are unused; their gradient is 0.
// The bit-exact decode leaves a block that had no bit plane above the tolerance unwritten; D
// writes every coded block, so in 2D, where such a block would keep the parent's values, D
// and the decode agree only where every low-band block below the coarsest level is decoded.
//
// Kernels. A 3D brick lies in shared memory whole (float, one CTA) or over a cluster of two CTAs
// (double: planes 0-15 and 16-32), rows 34 and planes 34 x 34 samples apart. The inverse zfp
// takes a lane per 4^3 block, 64 samples in registers: a warp's 32 blocks are the 8 parities of
// the 4 blocks of a row along x, whose samples at one place in the block lie in 32 different
// banks (8 t + hx + 2 hy + 4 hz). Samples at x = 32, y = 32 and z = 32 (blocks of extent 1 on an
// axis) go as 4-point lines, one axis after the other. The forward pass writes the parent's
// values over the uncoded blocks, the adjoint hands theirs to the parent and clears them. The
// one-level CDF5/3 runs along y, x (rows read two samples at a time, which an even row length
// of 17 pairs leaves free of conflicts) and z; the Z pass writes the grid (finest level) or the
// kept brick straight from registers, and in the adjoint reads the grid's gradient the same way;
// the cluster's two halves meet in it only, through distributed shared memory. The next brick is
// prefetched into L2 while this one is worked on. A 2D brick is one CTA: X pass inside, Y pass as
// the column pass. The order of the three CDF passes differs from the decode's Z, Y, X: they act
// on different axes and commute, the results differ by rounding only.
//
// What bounds it: per brick 26 K cycles forward, of which the shared-memory pipe is busy half
// (some 10 accesses a sample) and the issue slots a third (38 K warp instructions), with the load
// of a brick and the store of its grid not overlapped (one brick fills an SM). For 32 float fields
// of 256^3 (gpu__time_duration, both levels) 1.72 ms forward and 2.03 ms adjoint; with the Y and
// the X sweep taken over all rows of the brick and a barrier between them, instead of a warp doing
// both in its own plane (cdf_plane), 1.86 and 2.18 ms; that form over clusters of two CTAs, two
// clusters per SM pair, 2.09 and 2.26 ms; clusters of four CTAs with every zfp pass and every
// sweep through shared memory 3.09 and 2.69 ms.
#include "codec_device.cuh"
#include "device.h"
#include "encoder.h"
#include "format.h"

#include <cooperative_groups.h>

#include <cstring>
#include <vector>

namespace cg = cooperative_groups;

namespace idx2g
{

namespace
{

constexpr int kPlane = 33 * 33;
constexpr int kRow = 34;            // samples between rows of a brick in shared memory
constexpr int kLayer = 34 * kRow;   // and between its planes
constexpr int kSynThreads2 = 320;   // 2D bricks

// 3D: CTAs per brick, threads per CTA (the 1,089 lines of a sweep, or a half's 561, take two
// rounds)
template <typename T>
struct syn3
{
  static constexpr int CS = sizeof(T) == 4 ? 1 : 2;
  static constexpr int threads = sizeof(T) == 4 ? 576 : 288;
  static constexpr size_t smem = (size_t)(sizeof(T) == 4 ? 33 : 17) * kLayer * sizeof(T);
};

struct syn_brick
{
  int b3[3];
  int valid[3];   // samples of the grid in the brick (finest level)
  int parent;     // index of the parent brick on the coarser level (all fields)
  int pos[3];     // position inside the parent (0/1 per axis)
  int field;
  long long coff; // offset of the brick in its field's coefficient tensor (elements)
};

template <typename T>
struct syn_args
{
  int nbricks, coarsest, finest, norm_mask;
  double inv_weight[8];
  int nb[3], npb[3];     // bricks per axis of one field on this level and on the coarser one
  long long cbase;       // first element of the level in a field's coefficient tensor
  long long cstride;     // elements of one field's coefficient tensor
  long long gstride;     // elements of one field's grid
  long long gdims[3];
  // forward: in = coefficients, out = grid (finest level), bricks_out = kept bricks (other
  // levels), parents = kept bricks of the coarser level. adjoint: in = gradient of the grid
  // (finest level) or this level's gradient bricks, out = gradient of the coefficients,
  // pgrad = the coarser level's gradient bricks (or null).
  const T* in;
  T* out;
  const T* parents;
  T* pgrad;
  T* bricks_out;
};

// Brick bi of the launch: the fields one after the other, row-major bricks (x fastest) in each.
template <typename T>
__device__ __forceinline__ syn_brick brick_at(const syn_args<T>& a, int bi, bool is2d)
{
  syn_brick b;
  const int per = a.nb[0] * a.nb[1] * a.nb[2];
  b.field = bi / per;
  const int i = bi - b.field * per, r = i / a.nb[0];
  b.b3[0] = i - r * a.nb[0];
  b.b3[2] = r / a.nb[1];
  b.b3[1] = r - b.b3[2] * a.nb[1];
  for (int k = 0; k < 3; ++k)
  {
    const int side = is2d && k == 2 ? 1 : 32;
    const long long left = a.gdims[k] - (long long)b.b3[k] * side;
    b.valid[k] = (int)(left < side ? left : side);
    b.pos[k] = is2d && k == 2 ? 0 : b.b3[k] & 1;
  }
  const int pz = is2d ? b.b3[2] : b.b3[2] >> 1;
  b.parent = b.field * (a.npb[0] * a.npb[1] * a.npb[2]) + (pz * a.npb[1] + (b.b3[1] >> 1)) * a.npb[0] + (b.b3[0] >> 1);
  b.coff = a.cbase + (long long)i * (is2d ? kPlane : 33 * kPlane);
  return b;
}

// a * k + b for a power of two k: the product is exact, so this is the sum's one rounding
__device__ __forceinline__ float axpb(float a, float k, float b) { return __fmaf_rn(a, k, b); }
__device__ __forceinline__ double axpb(double a, double k, double b) { return __fma_rn(a, k, b); }

// Real inverse zfp lifting of one 4-point line (Core/Zfp.h:181 ILift, halvings exact).
template <typename T>
__device__ __forceinline__ void rilift4(T& x, T& y, T& z, T& w)
{
  y = axpb(w, T(0.5), y);
  w = axpb(y, T(-0.5), w);
  y += w;
  w = axpb(w, T(2), -y);
  z += x;
  x = axpb(x, T(2), -z);
  y += z;
  z = axpb(z, T(2), -y);
  w += x;
  x = axpb(x, T(2), -w);
}

// Its transpose: the elementary steps of rilift4 transposed, in reverse order.
template <typename T>
__device__ __forceinline__ void rilift4_adj(T& x, T& y, T& z, T& w)
{
  w -= x;
  x = axpb(x, T(2), w);
  y -= z;
  z = axpb(z, T(2), y);
  z -= x;
  x = axpb(x, T(2), z);
  y -= w;
  w = axpb(w, T(2), y);
  y = axpb(w, T(-0.5), y);
  w = axpb(y, T(0.5), w);
}

template <typename T, bool ADJ>
__device__ __forceinline__ void lift4(T& x, T& y, T& z, T& w)
{
  if constexpr (ADJ)
    rilift4_adj(x, y, z, w);
  else
    rilift4(x, y, z, w);
}

// the same on samples s apart in shared memory
template <typename T, bool ADJ>
__device__ __forceinline__ void lift4_at(T* q, int s)
{
  T x = q[0], y = q[s], z = q[2 * s], w = q[3 * s];
  lift4<T, ADJ>(x, y, z, w);
  q[0] = x;
  q[s] = y;
  q[2 * s] = z;
  q[3 * s] = w;
}

// One-level inverse CDF5/3 of a 33-sample line (Core/Wavelet.h:250 ILiftCdf53, D = 33) and
// its transpose.
template <typename T>
__device__ __forceinline__ void rilift33(T (&v)[33])
{
#pragma unroll
  for (int x = 1; x < 33; x += 2)
  {
    v[x - 1] = axpb(v[x], T(-0.25), v[x - 1]);
    v[x + 1] = axpb(v[x], T(-0.25), v[x + 1]);
  }
#pragma unroll
  for (int x = 1; x < 33; x += 2)
    v[x] = axpb(v[x - 1] + v[x + 1], T(0.5), v[x]);
}

template <typename T>
__device__ __forceinline__ void rilift33_adj(T (&g)[33])
{
  g[32] = axpb(g[31], T(0.5), g[32]);
  g[30] = axpb(g[31], T(0.5), g[30]);
#pragma unroll
  for (int x = 1; x < 31; x += 2)
  {
    g[x - 1] = axpb(g[x], T(0.5), g[x - 1]);
    g[x + 1] = axpb(g[x], T(0.5), g[x + 1]);
  }
  g[31] = axpb(g[30] + g[32], T(-0.25), g[31]);
#pragma unroll
  for (int x = 1; x < 31; x += 2)
    g[x] = axpb(g[x - 1] + g[x + 1], T(-0.25), g[x]);
}

template <typename T, bool ADJ>
__device__ __forceinline__ void lift33(T (&v)[33])
{
  if constexpr (ADJ)
    rilift33_adj(v);
  else
    rilift33(v);
}

// Subband of a sample from its parities (the subband order of the format: 3D hx hy hz, 2D hx hy).
template <bool IS2D>
__device__ __forceinline__ int parity_index(int x, int y, int z)
{
  if constexpr (IS2D)
    return ((x & 1) << 1) | (y & 1);
  else
    return ((x & 1) << 2) | ((y & 1) << 1) | (z & 1);
}

// De-normalisation factors per subband in shared memory (1 where the subband is not weighted:
// a multiplication by 1 is exact), staged once per CTA.
template <typename T>
__device__ __forceinline__ void stage_weights(const syn_args<T>& a, T* sw, int tid)
{
  if (tid < 8)
    sw[tid] = ((a.norm_mask >> tid) & 1) ? (T)a.inv_weight[tid] : T(1);
  __syncthreads();
}

template <int CS>
__device__ __forceinline__ void cluster_sync()
{
  if constexpr (CS > 1)
    cg::this_cluster().sync();
  else
    __syncthreads();
}

template <typename T>
__device__ __forceinline__ void copy_async(T* dst, const T* src)
{
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  if constexpr (sizeof(T) == 4)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
}

__device__ __forceinline__ void copy_wait()
{
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
}

__device__ __forceinline__ void prefetch_l2(const void* p)
{
  asm volatile("prefetch.global.L2 [%0];\n" ::"l"(p));
}

// In-place inverse zfp (or its transpose) lines of a 2D brick, rows of 33: along y and x, per
// parity h, blocks k = 0..3 at h + 8k + 2j; the fifth block of the 17-sample low half has extent 1
// and no line.
template <typename T, bool ADJ>
__device__ __forceinline__ void zfp_y2(T* S, int tid)
{
  for (int L = tid; L < 8 * 33; L += kSynThreads2)
  {
    const int x = L % 33, g = L / 33;
    lift4_at<T, ADJ>(S + ((g & 1) + 8 * (g >> 1)) * 33 + x, 66);
  }
}

template <typename T, bool ADJ>
__device__ __forceinline__ void zfp_x2(T* S, int tid)
{
  for (int L = tid; L < 8 * 33; L += kSynThreads2)
  {
    const int row = L % 33, g = L / 33;
    lift4_at<T, ADJ>(S + row * 33 + (g & 1) + 8 * (g >> 1), 2);
  }
}

// CDF5/3 lines along x of a 2D brick; the de-normalisation comes before the lift (forward) or
// after the transposed lift (adjoint).
template <typename T, bool ADJ>
__device__ __forceinline__ void cdf_x2(const T* sw, T* S, int tid)
{
  for (int y = tid; y < 33; y += kSynThreads2)
  {
    T* row = S + y * 33;
    T v[33];
#pragma unroll
    for (int x = 0; x < 33; ++x)
      v[x] = !ADJ ? row[x] * sw[parity_index<true>(x, y, 0)] : row[x];
    lift33<T, ADJ>(v);
#pragma unroll
    for (int x = 0; x < 33; ++x)
      row[x] = ADJ ? v[x] * sw[parity_index<true>(x, y, 0)] : v[x];
  }
}

// The inverse zfp (or its transpose) of the 4^3 blocks of block row (yb, zb), a lane per block.
// `low`: the blocks of the first subband are coded too.
template <typename T, bool ADJ>
__device__ __forceinline__ void zfp_blocks(T* S, int yb, int zb, bool low, int lane)
{
  const int t = lane & 3, hx = (lane >> 2) & 1, hy = (lane >> 3) & 1, hz = lane >> 4;
  T* b = S + (8 * zb + hz) * kLayer + (8 * yb + hy) * kRow + 8 * t + hx;
  T q[64];
#pragma unroll
  for (int j = 0; j < 64; ++j)
    q[j] = b[(j >> 4) * 2 * kLayer + ((j >> 2) & 3) * 2 * kRow + (j & 3) * 2];
#pragma unroll
  for (int pass = 0; pass < 3; ++pass)
  {
    const int s = (ADJ ? pass : 2 - pass) == 0 ? 1 : ((ADJ ? pass : 2 - pass) == 1 ? 4 : 16);
#pragma unroll
    for (int i = 0; i < 16; ++i)
    {
      const int o = s == 1 ? 4 * i : (s == 4 ? (i & 3) + 16 * (i >> 2) : i);
      lift4<T, ADJ>(q[o], q[o + s], q[o + 2 * s], q[o + 3 * s]);
    }
  }
  if (!low && hx + hy + hz == 0)
    return;
#pragma unroll
  for (int j = 0; j < 64; ++j)
    b[(j >> 4) * 2 * kLayer + ((j >> 2) & 3) * 2 * kRow + (j & 3) * 2] = q[j];
}

// Lines of the blocks of extent 1 on an axis, the CTA's `np` planes (8 nzb of them in whole
// blocks along z; `top`: the last one is plane 32).
template <typename T, bool ADJ>
__device__ __forceinline__ void face_z(T* S, int nzb, int tid, int nt)
{
  for (int L = tid; L < 65 * 2 * nzb; L += nt)
  {
    const int c = L % 65, g = L / 65;
    const int x = c < 33 ? 32 : c - 33, y = c < 33 ? c : 32;
    lift4_at<T, ADJ>(S + (8 * (g >> 1) + (g & 1)) * kLayer + y * kRow + x, 2 * kLayer);
  }
}

template <typename T, bool ADJ>
__device__ __forceinline__ void face_y(T* S, int np, bool top, int tid, int nt)
{
  const int n = np + (top ? 32 : 0);  // x = 32 on every plane, then plane 32
  for (int L = tid; L < 8 * n; L += nt)
  {
    const int c = L % n, g = L / n;
    const int x = c < np ? 32 : c - np, p = c < np ? c : np - 1;
    lift4_at<T, ADJ>(S + p * kLayer + (8 * (g >> 1) + (g & 1)) * kRow + x, 2 * kRow);
  }
}

template <typename T, bool ADJ>
__device__ __forceinline__ void face_x(T* S, int np, bool top, int tid, int nt)
{
  const int n = np + (top ? 32 : 0);  // y = 32 on every plane, then plane 32
  for (int L = tid; L < 8 * n; L += nt)
  {
    const int c = L % n, g = L / n;
    const int y = c < np ? 32 : c - np, p = c < np ? c : np - 1;
    lift4_at<T, ADJ>(S + p * kLayer + y * kRow + 8 * (g >> 1) + (g & 1), 2);
  }
}

// One 33-sample line over the lanes of a warp: lane k holds samples 2k (k <= 16) and 2k + 1
// (k <= 15); the operations of rilift33 / rilift33_adj, in their order.
template <typename T, bool ADJ>
__device__ __forceinline__ void lift33_lanes(T& e, T& o, int lane)
{
  const T prev = __shfl_up_sync(0xffffffffu, o, 1);
  constexpr T k = ADJ ? T(0.5) : T(-0.25);
  if (ADJ && lane == 15)  // (rilift33_adj starts with the last odd sample)
    e = axpb(o, k, e);
  if (lane > 0)
    e = axpb(prev, k, e);
  if (lane < (ADJ ? 15 : 16))
    e = axpb(o, k, e);
  const T next = __shfl_down_sync(0xffffffffu, e, 1);
  o = axpb(e + next, ADJ ? T(-0.25) : T(0.5), o);
}

// The CDF5/3 sweeps inside plane z of the brick (at S), by a warp: along y with the
// de-normalisation before it, then along x (forward), or along x, then along y with the
// de-normalisation after it (adjoint). A lane per column or row, their 33rd over the lanes; rows two
// samples an access (the 34th is padding).
template <typename T, bool ADJ>
__device__ __forceinline__ void cdf_plane(const T* sw, T* S, int z, int lane)
{
  struct alignas(2 * sizeof(T)) pair_t
  {
    T a, b;
  };
  const int l16 = lane < 16 ? lane : 16, l15 = lane < 15 ? lane : 15;
  auto along_y = [&]() {
    T e = S[2 * l16 * kRow + 32], o = S[(2 * l15 + 1) * kRow + 32];
    T v[33];
    const T w0 = sw[parity_index<false>(lane, 0, z)], w1 = sw[parity_index<false>(lane, 1, z)];
    const T u0 = sw[parity_index<false>(32, 0, z)], u1 = sw[parity_index<false>(32, 1, z)];
#pragma unroll
    for (int y = 0; y < 33; ++y)
      v[y] = !ADJ ? S[y * kRow + lane] * ((y & 1) ? w1 : w0) : S[y * kRow + lane];
    if (!ADJ)
    {
      e *= u0;
      o *= u1;
    }
    lift33_lanes<T, ADJ>(e, o, lane);
    lift33<T, ADJ>(v);
    if (ADJ)
    {
      e *= u0;
      o *= u1;
    }
#pragma unroll
    for (int y = 0; y < 33; ++y)
      S[y * kRow + lane] = ADJ ? v[y] * ((y & 1) ? w1 : w0) : v[y];
    if (lane < 17)
      S[2 * lane * kRow + 32] = e;
    if (lane < 16)
      S[(2 * lane + 1) * kRow + 32] = o;
  };
  auto along_x = [&]() {
    pair_t* row = reinterpret_cast<pair_t*>(S + lane * kRow);
    pair_t last = reinterpret_cast<pair_t*>(S + 32 * kRow)[l16];
    T v[33];
#pragma unroll
    for (int x = 0; x < 17; ++x)
    {
      const pair_t r = row[x];
      v[2 * x] = r.a;
      if (x < 16)
        v[2 * x + 1] = r.b;
    }
    lift33_lanes<T, ADJ>(last.a, last.b, lane);
    lift33<T, ADJ>(v);
#pragma unroll
    for (int x = 0; x < 17; ++x)
      row[x] = pair_t{ v[2 * x], x < 16 ? v[2 * x + 1] : T(0) };
    if (lane < 17)
      reinterpret_cast<pair_t*>(S + 32 * kRow)[lane] = last;
  };
  if constexpr (!ADJ)
  {
    along_y();
    __syncwarp();
    along_x();
  }
  else
  {
    along_x();
    __syncwarp();
    along_y();
  }
}

// Offset of the brick's first sample in a batch of grids.
template <typename T>
__device__ __forceinline__ size_t grid_offset(const syn_args<T>& a, const syn_brick& br, bool is2d)
{
  return (size_t)br.field * (size_t)a.gstride +
         (size_t)(((long long)br.b3[2] * (is2d ? 1 : 32)) * a.gdims[1] + (long long)br.b3[1] * 32) *
           (size_t)a.gdims[0] +
         (size_t)br.b3[0] * 32;
}

// Shared-memory address of sample (z, c) of the brick, c the offset in a plane, in the CTA of the
// cluster that holds plane z.
template <typename T>
__device__ __forceinline__ unsigned sample_addr(const unsigned* base, int z, int c)
{
  const int r = z < 16 ? 0 : 1;
  return base[r] + (unsigned)(((z - 16 * r) * kLayer + c) * (int)sizeof(T));
}

template <typename T, bool ADJ>
__global__ void __launch_bounds__(syn3<T>::threads, 1) k_synth3(const syn_args<T> a)
{
  extern __shared__ __align__(16) unsigned char syn_smem[];
  __shared__ T sw[8];
  __shared__ syn_brick sb[2];  // this brick and the next (made by one thread: some divisions)
  T* S = reinterpret_cast<T*>(syn_smem);
  constexpr int CS = syn3<T>::CS, NT = syn3<T>::threads, NW = NT / 32;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  stage_weights(a, sw, tid);
  int rank = 0;
  unsigned base[2] = { 0, 0 };  // the cluster's brick halves, as shared::cluster addresses
  if constexpr (CS > 1)
  {
    rank = (int)cg::this_cluster().block_rank();
    base[0] = dev::cluster_addr(S, 0);
    base[1] = dev::cluster_addr(S, 1);
    cluster_sync<CS>();  // every CTA of the cluster has started before any remote access
  }
  const int z0 = rank * 16;
  const int np = CS == 1 ? 33 : 16 + rank;
  const int nzb = CS == 1 ? 4 : 2;
  const bool top = rank == CS - 1;
  const int nclusters = gridDim.x / CS;
  const size_t zs = (size_t)a.gdims[1] * (size_t)a.gdims[0];
  if (tid == 0)
    sb[0] = brick_at(a, (int)blockIdx.x / CS, false);
  __syncthreads();
  int cur = 0;
  for (int bi = blockIdx.x / CS; bi < a.nbricks; bi += nclusters, cur ^= 1)
  {
    const syn_brick& br = sb[cur];
    const int next = bi + nclusters;
    if (tid == 0 && next < a.nbricks)
      sb[cur ^ 1] = brick_at(a, next, false);  // read after the next barrier
    const size_t cat = (size_t)br.field * (size_t)a.cstride + (size_t)br.coff + (size_t)z0 * kPlane;
    if constexpr (!ADJ)
    {
      // the coefficients, a warp per row, the 33rd samples after them
      const T* src = a.in + cat;
      for (int y = warp; y < 33; y += NW)
      {
        const T* g = src + y * 33 + lane;
        T* d = S + y * kRow + lane;
#pragma unroll
        for (int p = 0; p < (CS == 1 ? 33 : 16); ++p)
          copy_async(d + p * kLayer, g + p * kPlane);
        if (CS > 1 && top)
          copy_async(d + 16 * kLayer, g + 16 * kPlane);
      }
      for (int r = tid; r < 33 * np; r += NT)
        copy_async(S + (r / 33) * kLayer + (r % 33) * kRow + 32, src + r * 33 + 32);
      copy_wait();
      __syncthreads();
      // inverse zfp: z, y, x
      if (warp < 4 * nzb)
        zfp_blocks<T, false>(S, warp & 3, warp >> 2, a.coarsest, lane);
      face_z<T, false>(S, nzb, tid, NT);
      if (!a.coarsest)
      {
        // the parent's values over the uncoded full low-band blocks (even samples below 32)
        const T* P = a.parents + (size_t)br.parent * (33 * kPlane);
        for (int i = tid; i < 4 * nzb * 256; i += NT)
        {
          const int x = i & 15, y = (i >> 4) & 15, k = i >> 8;
          S[2 * k * kLayer + 2 * y * kRow + 2 * x] =
            P[((br.pos[2] * 16 + (z0 >> 1) + k) * 33 + (br.pos[1] * 16 + y)) * 33 + (br.pos[0] * 16 + x)];
        }
      }
      __syncthreads();
      if (next < a.nbricks)
      {
        const syn_brick& nx = sb[cur ^ 1];
        const char* q = (const char*)(a.in + (size_t)nx.field * (size_t)a.cstride + (size_t)nx.coff +
                                      (size_t)z0 * kPlane);
        for (int k = tid * 128; k < np * kPlane * (int)sizeof(T); k += NT * 128)
          prefetch_l2(q + k);
      }
      face_y<T, false>(S, np, top, tid, NT);
      __syncthreads();
      face_x<T, false>(S, np, top, tid, NT);
      __syncthreads();
      for (int p = warp; p < np; p += NW)
        cdf_plane<T, false>(sw, S + p * kLayer, z0 + p, lane);
      cluster_sync<CS>();
      // Z pass over the brick: this CTA's share of the columns (the grid has those below 32)
      const int side = a.finest ? 32 : 33;
      for (int c = rank * NT + tid; c < side * side; c += CS * NT)
      {
        const int x = c % side, y = c / side, o = y * kRow + x;
        T v[33];
#pragma unroll
        for (int z = 0; z < 33; ++z)
        {
          if constexpr (CS == 1)
            v[z] = S[z * kLayer + o];
          else
            v[z] = dev::ld_cluster<T>(sample_addr<T>(base, z, o));
        }
        rilift33(v);
        if (a.finest)
        {
          if (x < br.valid[0] && y < br.valid[1])
          {
            T* g = a.out + grid_offset(a, br, false) + (size_t)y * (size_t)a.gdims[0] + x;
            if (br.valid[2] == 32)
            {
#pragma unroll
              for (int z = 0; z < 32; ++z, g += zs)
                *g = v[z];
            }
            else
            {
#pragma unroll
              for (int z = 0; z < 32; ++z, g += zs)
                if (z < br.valid[2])
                  *g = v[z];
            }
          }
        }
        else
        {
          T* out = a.bricks_out + (size_t)bi * (33 * kPlane) + c;
#pragma unroll
          for (int z = 0; z < 33; ++z)
            out[z * kPlane] = v[z];
        }
      }
      cluster_sync<CS>();
    }
    else
    {
      // transposed Z pass: this CTA's columns of the incoming gradient, into the cluster. The
      // grid has those below 32; the faces x = 32 and y = 32 start from zeros there.
      const int side = a.finest ? 32 : 33;
      if (a.finest)
        for (int i = tid; i < 65 * np; i += NT)
        {
          const int c = i % 65, p = i / 65;
          S[p * kLayer + (c < 33 ? c * kRow + 32 : 32 * kRow + c - 33)] = T(0);
        }
      for (int c = rank * NT + tid; c < side * side; c += CS * NT)
      {
        const int x = c % side, y = c / side, o = y * kRow + x;
        T v[33];
        if (a.finest)
        {
          const int nz = x < br.valid[0] && y < br.valid[1] ? br.valid[2] : 0;  // valid[2] <= 32
          const T* g = a.in + grid_offset(a, br, false) + (size_t)y * (size_t)a.gdims[0] + x;
          v[32] = T(0);
#pragma unroll
          for (int z = 0; z < 32; ++z, g += zs)
            v[z] = z < nz ? *g : T(0);
        }
        else
        {
          const T* gi = a.in + (size_t)bi * (33 * kPlane) + c;
#pragma unroll
          for (int z = 0; z < 33; ++z)
            v[z] = gi[z * kPlane];
        }
        rilift33_adj(v);
#pragma unroll
        for (int z = 0; z < 33; ++z)
        {
          if constexpr (CS == 1)
            S[z * kLayer + o] = v[z];
          else
            dev::st_cluster<T>(sample_addr<T>(base, z, o), v[z]);
        }
      }
      cluster_sync<CS>();
      if (next < a.nbricks && a.finest)
      {
        const syn_brick& nx = sb[cur ^ 1];
        for (int r = rank * NT + tid; r < nx.valid[1] * nx.valid[2]; r += CS * NT)
        {
          const T* g = a.in + grid_offset(a, nx, false) + (size_t)(r % nx.valid[1]) * (size_t)a.gdims[0] +
                       (size_t)(r / nx.valid[1]) * zs;
          prefetch_l2(g);
          prefetch_l2(g + nx.valid[0] - 1);
        }
      }
      for (int p = warp; p < np; p += NW)
        cdf_plane<T, true>(sw, S + p * kLayer, z0 + p, lane);
      __syncthreads();
      // transposed zfp: x, y, z; the low band over the uncoded blocks goes to the parent (and
      // nowhere else)
      face_x<T, true>(S, np, top, tid, NT);
      if (!a.coarsest)
      {
        T* P = a.pgrad + (size_t)br.parent * (33 * kPlane);
        for (int i = tid; i < 4 * nzb * 256; i += NT)
        {
          const int x = i & 15, y = (i >> 4) & 15, k = i >> 8;
          T* s = S + 2 * k * kLayer + 2 * y * kRow + 2 * x;
          P[((br.pos[2] * 16 + (z0 >> 1) + k) * 33 + (br.pos[1] * 16 + y)) * 33 + (br.pos[0] * 16 + x)] = *s;
          *s = T(0);
        }
      }
      __syncthreads();
      face_y<T, true>(S, np, top, tid, NT);
      __syncthreads();
      if (warp < 4 * nzb)
        zfp_blocks<T, true>(S, warp & 3, warp >> 2, a.coarsest, lane);
      face_z<T, true>(S, nzb, tid, NT);
      __syncthreads();
      T* dst = a.out + cat;
      for (int y = warp; y < 33; y += NW)
      {
        T* g = dst + y * 33 + lane;
        const T* d = S + y * kRow + lane;
#pragma unroll
        for (int p = 0; p < (CS == 1 ? 33 : 16); ++p)
          g[p * kPlane] = d[p * kLayer];
        if (CS > 1 && top)
          g[16 * kPlane] = d[16 * kLayer];
      }
      for (int r = tid; r < 33 * np; r += NT)
        dst[r * 33 + 32] = S[(r / 33) * kLayer + (r % 33) * kRow + 32];
      // the next brick's transposed Z pass writes into every CTA of the cluster
      cluster_sync<CS>();
    }
  }
}

// 2D bricks: a CTA each.
template <typename T, bool ADJ>
__global__ void __launch_bounds__(kSynThreads2, sizeof(T) == 4 ? 3 : 2) k_synth2(const syn_args<T> a)
{
  __shared__ T S[kPlane];
  __shared__ T sw[8];
  const int tid = threadIdx.x;
  stage_weights(a, sw, tid);
  for (int bi = blockIdx.x; bi < a.nbricks; bi += gridDim.x)
  {
    const syn_brick br = brick_at(a, bi, true);
    const size_t cat = (size_t)br.field * (size_t)a.cstride + (size_t)br.coff;
    if constexpr (!ADJ)
    {
      for (int i = tid; i < kPlane; i += kSynThreads2)
        copy_async(S + i, a.in + cat + i);
      copy_wait();
      __syncthreads();
      zfp_y2<T, false>(S, tid);
      __syncthreads();
      zfp_x2<T, false>(S, tid);
      __syncthreads();
      cdf_x2<T, false>(sw, S, tid);
      __syncthreads();
      // Y pass: one column per x
      if (tid < 33)
      {
        const int x = tid;
        T v[33];
#pragma unroll
        for (int y = 0; y < 33; ++y)
          v[y] = S[y * 33 + x];
        rilift33(v);
        if (a.finest)
        {
          if (x < br.valid[0])
          {
            T* g = a.out + grid_offset(a, br, true) + x;
#pragma unroll
            for (int y = 0; y < 32; ++y)
              if (y < br.valid[1])
                g[(size_t)y * (size_t)a.gdims[0]] = v[y];
          }
        }
        else
        {
          T* o = a.bricks_out + (size_t)bi * kPlane + x;
#pragma unroll
          for (int y = 0; y < 33; ++y)
            o[y * 33] = v[y];
        }
      }
      __syncthreads();
    }
    else
    {
      // transposed Y pass: one column per x of the incoming gradient
      if (tid < 33)
      {
        const int x = tid;
        T v[33];
        if (a.finest)
        {
          const T* g = a.in + grid_offset(a, br, true) + x;
#pragma unroll
          for (int y = 0; y < 33; ++y)
            v[y] = (x < br.valid[0] && y < 32 && y < br.valid[1]) ? g[(size_t)y * (size_t)a.gdims[0]] : T(0);
        }
        else
        {
          const T* gi = a.in + (size_t)bi * kPlane + x;
#pragma unroll
          for (int y = 0; y < 33; ++y)
            v[y] = gi[y * 33];
        }
        rilift33_adj(v);
#pragma unroll
        for (int y = 0; y < 33; ++y)
          S[y * 33 + x] = v[y];
      }
      __syncthreads();
      cdf_x2<T, true>(sw, S, tid);
      __syncthreads();
      zfp_x2<T, true>(S, tid);
      __syncthreads();
      zfp_y2<T, true>(S, tid);
      __syncthreads();
      for (int i = tid; i < kPlane; i += kSynThreads2)
        a.out[cat + i] = S[i];
      __syncthreads();
    }
  }
}

// Bricks and weights of every level of a format (levels finest first).
struct syn_level
{
  int nb[3];        // bricks per axis
  long long base;   // first element of the level in a field's coefficient tensor
  double inv_weight[8];
  int norm_mask;
};

// The kernels assume the block layout of an extended brick: subband s at the parities of its
// index (3D hx hy hz, 2D hx hy), 17 samples on a low and 16 on a high axis, blocks of 4 (the
// fifth of a low axis of extent 1), every block coded except, below the coarsest level, the
// full 4^3 low-band blocks (Core/idx2Decode.cpp:126-130). Checked against the coder's own
// block walk of every level.
bool uniform_blocks(const dataset_format& f, int level)
{
  const bool is2d = f.is2d();
  for (int s = 0; s < f.nsubbands(); ++s)
  {
    const subband& sb = f.subbands[(size_t)s];
    const int h[3] = { is2d ? (s >> 1) & 1 : (s >> 2) & 1, is2d ? s & 1 : (s >> 1) & 1, is2d ? 0 : s & 1 };
    const v3 ha(h[0], h[1], h[2]);
    if (!(sb.low_high == ha) || !(sb.g.from == ha))
      return false;
    const v3 want(17 - h[0], 17 - h[1], is2d ? 1 : 17 - h[2]);
    if (!(sb.g.dims == want))
      return false;
    const int nk[3] = { h[0] ? 4 : 5, h[1] ? 4 : 5, is2d ? 1 : (h[2] ? 4 : 5) };
    const size_t uncoded = s == 0 && level + 1 < f.nlevels && !is2d ? 64 : 0;
    bool seen[125] = {};
    std::vector<block_geom> g;
    subband_blocks(f, level, s, &g);
    if (g.size() + uncoded != (size_t)(nk[0] * nk[1] * nk[2]))
      return false;
    for (const block_geom& b : g)
    {
      if (b.dx >= nk[0] || b.dy >= nk[1] || b.dz >= nk[2])
        return false;
      const int bx = b.dx < 4 ? 4 : 1, by = b.dy < 4 ? 4 : 1, bz = is2d ? 1 : (b.dz < 4 ? 4 : 1);
      bool& at = seen[(b.dz * 5 + b.dy) * 5 + b.dx];
      if (at || b.bx != bx || b.by != by || b.bz != bz || (uncoded && bx == 4 && by == 4 && bz == 4))
        return false;
      at = true;
    }
  }
  return true;
}

long long build_levels(const dataset_format& f, std::vector<syn_level>* out)
{
  const int L = f.nlevels;
  const bool is2d = f.is2d();
  const int NB = is2d ? 33 * 33 : 33 * 33 * 33;
  if (L > 1 && !(f.group_brick3 == v3(2, 2, is2d ? 1 : 2)))
    return -1;
  out->assign((size_t)L, syn_level());
  long long base = 0;
  for (int l = 0; l < L; ++l)
  {
    if (!uniform_blocks(f, l))
      return -1;
    syn_level& sl = (*out)[(size_t)l];
    const v3 n3 = f.nbricks3[(size_t)l];
    sl.nb[0] = n3.x;
    sl.nb[1] = n3.y;
    sl.nb[2] = n3.z;
    sl.base = base;
    base += (long long)n3.x * n3.y * n3.z * NB;
    double w[8];
    level_weights(f, l, w, &sl.norm_mask);
    for (int s = 0; s < 8; ++s)
      sl.inv_weight[s] = s < f.nsubbands() ? 1.0 / w[s] : 1.0;
  }
  return base;
}

template <typename T, bool IS2D>
int launch_synth(device_ctx* ctx, const syn_args<T>& a, bool adjoint, cudaStream_t st)
{
  if (a.nbricks < 1)
    return NoError;
  if constexpr (IS2D)
  {
    const int grid = a.nbricks < 3 * ctx->num_sms ? a.nbricks : 3 * ctx->num_sms;
    (adjoint ? k_synth2<T, true> : k_synth2<T, false>)<<<grid, kSynThreads2, 0, st>>>(a);
    return cudaGetLastError() == cudaSuccess ? NoError : CudaError;
  }
  else
  {
    constexpr int CS = syn3<T>::CS;
    const size_t smem = syn3<T>::smem;
    void (*kern)(const syn_args<T>) = adjoint ? k_synth3<T, true> : k_synth3<T, false>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
      return CudaError;
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof cfg);
    cudaLaunchAttribute attr[1];
    cfg.blockDim = dim3(syn3<T>::threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    int nclusters = ctx->num_sms / CS;
    if (CS > 1)
    {
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = CS;
      attr[0].val.clusterDim.y = 1;
      attr[0].val.clusterDim.z = 1;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      cfg.gridDim = dim3(CS * nclusters);
      int active = 0;
      if (cudaOccupancyMaxActiveClusters(&active, kern, &cfg) == cudaSuccess && active > 0)
        nclusters = active;
    }
    if (nclusters > a.nbricks)
      nclusters = a.nbricks;
    cfg.gridDim = dim3(CS * nclusters);
    return cudaLaunchKernelEx(&cfg, kern, a) == cudaSuccess ? NoError : CudaError;
  }
}

template <typename T>
int run_synth(device_ctx* ctx, const dataset_format& f, int nbatch, const void* in, void* out, bool adjoint,
              double* kernel_ms)
{
  std::vector<syn_level> lv;
  const long long count = build_levels(f, &lv);
  if (count < 0)
    return OptionNotSupported;
  const int L = f.nlevels;
  const int NB = f.is2d() ? 33 * 33 : 33 * 33 * 33;
  cudaStream_t st = ctx->stream;
  const long long gcount = (long long)f.dims.x * f.dims.y * f.dims.z;
  T* prev = nullptr;  // forward: kept bricks of the coarser level; adjoint: this level's gradient bricks
  // an error return waits for the levels launched so far: they read and write the caller's arrays
  auto fail = [st](int e) {
    cudaStreamSynchronize(st);
    return e;
  };
  for (int step = 0; step < L; ++step)
  {
    const int l = adjoint ? step : L - 1 - step;
    const syn_level& sl = lv[(size_t)l];
    syn_args<T> a;
    memset(&a, 0, sizeof a);
    a.nbricks = sl.nb[0] * sl.nb[1] * sl.nb[2] * nbatch;
    a.coarsest = l + 1 == L;
    a.finest = l == 0;
    a.norm_mask = sl.norm_mask;
    memcpy(a.inv_weight, sl.inv_weight, sizeof a.inv_weight);
    memcpy(a.nb, sl.nb, sizeof a.nb);
    if (l + 1 < L)
      memcpy(a.npb, lv[(size_t)l + 1].nb, sizeof a.npb);
    a.cbase = sl.base;
    a.cstride = count;
    a.gstride = gcount;
    a.gdims[0] = f.dims.x;
    a.gdims[1] = f.dims.y;
    a.gdims[2] = f.dims.z;
    char nm[32];
    snprintf(nm, sizeof nm, "syn.lev%d", step & 1);
    if (!adjoint)
    {
      a.in = (const T*)in;
      a.parents = prev;
      if (l == 0)
        a.out = (T*)out;
      else
      {
        a.bricks_out = (T*)ctx->ws(nm, (size_t)a.nbricks * (size_t)NB * sizeof(T));
        if (!a.bricks_out)
          return fail(OutOfMemory);
      }
    }
    else
    {
      a.in = l == 0 ? (const T*)in : prev;
      a.out = (T*)out;
      if (l + 1 < L)
      {
        const size_t pn = (size_t)a.npb[0] * (size_t)a.npb[1] * (size_t)a.npb[2] * (size_t)nbatch * (size_t)NB;
        a.pgrad = (T*)ctx->ws(nm, pn * sizeof(T));
        if (!a.pgrad)
          return fail(OutOfMemory);
        cudaMemsetAsync(a.pgrad, 0, pn * sizeof(T), st);
      }
    }
    // the levels follow one another on the stream; the host waits once, after the last
    cudaEvent_t t0 = ctx->ev((size_t)(2 * step)), t1 = ctx->ev((size_t)(2 * step + 1));
    if (!t0 || !t1)
      return fail(CudaError);
    cudaEventRecord(t0, st);
    const int e = f.is2d() ? launch_synth<T, true>(ctx, a, adjoint, st) : launch_synth<T, false>(ctx, a, adjoint, st);
    cudaEventRecord(t1, st);
    if (e)
      return fail(e);
    prev = adjoint ? a.pgrad : a.bricks_out;
    ++ctx->launches;
    if (cudaGetLastError() != cudaSuccess)
      return fail(CudaError);
  }
  if (cudaStreamSynchronize(st) != cudaSuccess)
    return CudaError;
  float total = 0;
  for (int step = 0; step < L; ++step)
  {
    float ms = 0;
    cudaEventElapsedTime(&ms, ctx->ev((size_t)(2 * step)), ctx->ev((size_t)(2 * step + 1)));
    total += ms;
  }
  if (kernel_ms)
    *kernel_ms = total;
  return NoError;
}

} // namespace

long long synth_coeff_count(const dataset_format& f)
{
  std::vector<syn_level> lv;
  return build_levels(f, &lv);
}

int synth(device_ctx* ctx, const dataset_format& f, int nbatch, const void* d_in, void* d_out, bool adjoint,
          double* kernel_ms)
{
  if (f.brick_dims.x != 32 || f.brick_dims.y != 32 || (f.brick_dims.z != 32 && f.brick_dims.z != 1))
    return OptionNotSupported;
  cudaSetDevice(ctx->device);
  return f.type == dtype::float32 ? run_synth<float>(ctx, f, nbatch, d_in, d_out, adjoint, kernel_ms)
                                  : run_synth<double>(ctx, f, nbatch, d_in, d_out, adjoint, kernel_ms);
}

} // namespace idx2g
