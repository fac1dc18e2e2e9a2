// k_decode_bricks: the device decode of one level of 3D bricks from the bit planes of
// k_decode_planes (included by decode.cu inside an anonymous namespace, after
// decode_kernel.cuh).
//
// What bounds it: one brick is 729 zfp blocks (512 of them 4^3) and three sweeps over 33^3
// doubles (287 KB, more than an SM's shared memory). A warp working on one block at a time (as
// k_decode_level does) issues 350 K warp instructions per brick, most of them exchanges between
// the lanes that share a block, and the sweeps move the brick through L2 seven times.
//
// The split here:
//  * A lane owns a whole block. Its plane words are transposed to coefficients in registers (no
//    shuffles), and the inverse zfp runs on 64 registers of 32 bits: with at most 26 planes the
//    low word of every 64-bit coefficient stays zero through the three passes (each pass needs
//    two more bits, 26 + 6 = 32), so the high words alone give the 64-bit result exactly. Blocks
//    of 27 to 44 planes are the exact sum of two such transforms (planes 0-25 and 26-43): the
//    transform is linear where no halving loses a bit, which 64 - 44 - 6 > 0 spare bits ensure,
//    and where no halved value wraps around 64 bits, which the coder's blocks of finite samples
//    are far from and which is checked (may_wrap). Blocks of more planes, and those that may wrap
//    (a stream of another origin, or a damaged one), take the warp-per-block 64-bit form.
//  * A warp's 32 blocks are the 8 blocks along z (4 of each z parity) of 4 tiles in a row along
//    x, so the inverse CDF5/3 along z follows at once from shared memory, and the brick goes to
//    its slot in L2 once, already swept along z.
//  * Then a warp takes a z-plane at a time: the sweep along y reads the plane from L2 into
//    registers (a lane per column), the sweep along x takes it from shared memory (a lane per
//    row), and the rows leave as 16-byte stores. No barrier of the CTA inside.
//  * The samples at x = 32, y = 32 and z = 32 (blocks of extent 1 on an axis, 16 coefficients
//    or fewer) are rebuilt first, into three 33 x 33 faces in shared memory.
//
// Kept bricks are stored x fastest, 33^3 doubles, in natural order.
//
// Measured on one B200 (gpu__time_duration): the three levels of a 1024^3 float32 field at 1e-3
// 28.3 ms with k_decode_level, 6.2 ms now; one brick per CTA (8 bricks) 184 and 54 us. At level 0
// of 512^3 56 K warp instructions per brick (354 K before), 29% issue activity: what is left is
// latency at 16 warps per SM (128 registers a thread, 99 KB of shared memory per CTA). Not kept,
// as no faster: the next brick's parameters, exponents and tables fetched ahead (13% slower: more
// of the slots leave L2), plane words as 32-byte loads or marked evict-first, the next task's
// blocks looked up ahead, one CTA of 16 warps per SM in large launches.
#pragma once

constexpr int kFaceRow = 33;
constexpr int kFace = 33 * 33;
// A z-plane in a slot: four parity classes (hx, hy), each of rows of 17 samples: sample (x, y) at
// slot_xy(x, y). Rows of one class are read and written 16 lanes at a time, contiguous.
// (1,122 of them, padded to whole lines of 128 bytes)
constexpr int kSlotPlane = 1136;
constexpr int kSlotBrick = 33 * kSlotPlane;
// A warp's tile buffer: z sample (16 of even z, then 16 of odd z) major, 64 columns, the row
// padded to 65 words: lanes store with (tile, z block, parity) -> banks t + 4 zb + 16 hz.
constexpr int kTileRow = 65;
constexpr int kTileWords = 32 * kTileRow;
constexpr int kHighPlanes = 26;  // planes the high words alone hold exactly
constexpr int kLowBase = 14;     // bit of weight 1 in the second part's words
constexpr int kSplitPlanes = 44; // planes that the two parts hold together

template <int W>
struct brick_smem
{
  union alignas(16)
  {
    int32_t tile[kTileWords];  // rebuilt blocks of a task
    long long q[64];           // one block (more than kSplitPlanes planes)
    double plane[kFace];       // a z-plane between its y and x sweeps
    float rows[32 * 36];       // its rows cast to float, 144 bytes each
  } w[W];
  double face[3][kFace];       // samples at x = 32 ([z][y]), y = 32 ([z][x]), z = 32 ([y][x])
  double scale[W][32];    // dequantisation of the task's blocks, by lane
  uint8_t block[8][128];       // block of (zb * 5 + yb) * 5 + xb in the subband's walk, 255: not coded
  decode_target rq;
  decode_brick br;
  int sig;
};
static_assert(sizeof(brick_smem<1>::w[0]) % 16 == 0, "every warp's rows start 16-byte aligned");

__device__ __forceinline__ int slot_xy(int x, int y)
{
  return (x & 1) * (17 * 33) + (y & 1) * (17 * 17) + (y >> 1) * 17 + (x >> 1);
}

// One exchange round of the in-register bit transposes: rows a and b = a + J.
template <int J>
__device__ __forceinline__ void swap_bits(uint32_t& a, uint32_t& b)
{
  if constexpr (J == 16)
  {
    const uint32_t x = __byte_perm(a, b, 0x5410), y = __byte_perm(a, b, 0x7632);
    a = x;
    b = y;
  }
  else if constexpr (J == 8)
  {
    const uint32_t x = __byte_perm(a, b, 0x6240), y = __byte_perm(a, b, 0x7351);
    a = x;
    b = y;
  }
  else
  {
    constexpr uint32_t m = J == 4 ? 0x0f0f0f0fu : (J == 2 ? 0x33333333u : 0x55555555u);
    const uint32_t x = (a & m) | ((b << J) & ~m), y = ((a >> J) & m) | (b & ~m);
    a = x;
    b = y;
  }
}

template <int J, int N>
__device__ __forceinline__ void swap_round(uint32_t (&r)[N])
{
#pragma unroll
  for (int k = 0; k < N; ++k)
    if (!(k & J))
      swap_bits<J>(r[k], r[k + J]);
}

// bit i of word j <- bit j of word i: 32 x 32, or (N = 16) the two 16 x 16 halves side by side
template <int N>
__device__ __forceinline__ void transpose_bits(uint32_t (&r)[N])
{
  if constexpr (N == 32)
    swap_round<16>(r);
  swap_round<8>(r);
  swap_round<4>(r);
  swap_round<2>(r);
  swap_round<1>(r);
}

// Inverse zfp of one line (Core/Zfp.h:181 ILift) on 32-bit words, modulo 2^32.
__device__ __forceinline__ void ilift4_w(int32_t& x, int32_t& y, int32_t& z, int32_t& w)
{
  y += w >> 1;
  w -= y >> 1;
  y += w;
  w = (int32_t)((uint32_t)w << 1) - y;
  z += x;
  x = (int32_t)((uint32_t)x << 1) - z;
  y += z;
  z = (int32_t)((uint32_t)z << 1) - y;
  w += x;
  x = (int32_t)((uint32_t)x << 1) - w;
}

__device__ __forceinline__ void ilift4_ll(long long& x, long long& y, long long& z, long long& w)
{
  dev::inv_lift4_at(&x, &y, &z, &w);
}

// Negabinary digits to a two's complement word (Core/Zfp.h:520), bit 0 of even weight.
__device__ __forceinline__ int32_t from_negabinary(uint32_t u)
{
  return (int32_t)((u ^ 0xaaaaaaaau) - 0xaaaaaaaau);
}

// Coefficients of a 3D block from planes [first, first + count) of its row of plane words,
// count <= N: plane first + k becomes bit `top - k` of the coefficients' words. q in sample order.
template <int N>
__device__ __forceinline__ void block_words(const unsigned long long* row, int first, int count, int top,
                                            int32_t (&q)[64])
{
  // rows in the order that leaves the first plane in the words' highest bit
  uint32_t lo[N], hi[N];
#pragma unroll
  for (int k = 0; k < N; k += 2)
  {
    ulonglong2 v = make_ulonglong2(0ull, 0ull);
    if (k < count)
      v = __ldg(reinterpret_cast<const ulonglong2*>(row + first + k));
    const unsigned long long a = v.x, b = k + 1 < count ? v.y : 0ull;
    lo[N - 1 - k] = (uint32_t)a;
    hi[N - 1 - k] = (uint32_t)(a >> 32);
    lo[N - 2 - k] = (uint32_t)b;
    hi[N - 2 - k] = (uint32_t)(b >> 32);
  }
  transpose_bits(lo);
  transpose_bits(hi);
#pragma unroll
  for (int j = 0; j < 32; ++j)
  {
    uint32_t a, b;
    if constexpr (N == 32)
    {
      a = lo[j];
      b = hi[j];
    }
    else
    {
      a = j < 16 ? lo[j & 15] << 16 : lo[j & 15] & 0xffff0000u;
      b = j < 16 ? hi[j & 15] << 16 : hi[j & 15] & 0xffff0000u;
    }
    if (N == 32 && top != 31)
    {
      a >>= 31 - top;
      b >>= 31 - top;
    }
    q[dev::kPerm3d[j]] = from_negabinary(a);
    q[dev::kPerm3d[j + 32]] = from_negabinary(b);
  }
}

__device__ __forceinline__ void inverse_zfp3(int32_t (&q)[64])
{
#pragma unroll
  for (int i = 0; i < 16; ++i)
    ilift4_w(q[i], q[i + 16], q[i + 32], q[i + 48]);
#pragma unroll
  for (int i = 0; i < 16; ++i)
  {
    const int o = (i & 3) + 16 * (i >> 2);
    ilift4_w(q[o], q[o + 4], q[o + 8], q[o + 12]);
  }
#pragma unroll
  for (int i = 0; i < 16; ++i)
    ilift4_w(q[4 * i], q[4 * i + 1], q[4 * i + 2], q[4 * i + 3]);
}

// Whether a halved value of the inverse transform of the 64-bit coefficients q * 2^32 + l, the l
// (planes from kHighPlanes on) below 2^38, may come within 2^46 of the ends of the 64-bit range, so
// that the sum of the two parts' transforms could differ from the transform of the sum. A pass
// halves its w and y + w / 2; the passes before it give either at most 1.5^2 = 2.25 of any one
// coefficient (the largest entry of ILift's matrix is 6/4), so with the sum of the |q| at most
// 7 * 2^27 they stay below 0.985 * 2^31. Shifted down by 6 for the sum to fit, each rounded by less
// than 1. (The coder's blocks hold |q| < 2^27 before its transform, which averages: the sum of all 64
// coefficients is then at most 11.6 * 2^27, and 3 to 4 * 2^27 for white noise; one above the limit
// only takes the slower form. The check costs 0.6% where every block has 27 to 44 planes: 256^3 float64
// at 1e-7 1.048 -> 1.054 ms.)
__device__ __forceinline__ bool may_wrap(const int32_t (&q)[64])
{
  uint32_t sum = 0;
#pragma unroll
  for (int j = 0; j < 64; ++j)
    sum += (uint32_t)abs(q[j] >> 6);
  return sum > (7u << 21) - 64u;
}

// What a lane knows of a block: its decoded planes (0: nothing to rebuild) and their words.
struct lane_block
{
  int np, emax;
  const unsigned long long* row;
};

template <int W>
__device__ __forceinline__ lane_block find_block(const dec_args& a, const brick_smem<W>& sm, const decode_brick& br,
                                                 int bi, int s, int xb, int yb, int zb, bool there)
{
  lane_block lb;
  lb.np = 0;
  lb.emax = 0;
  lb.row = nullptr;
  const int b = there ? sm.block[s][(zb * 5 + yb) * 5 + xb] : 255;
  if (b == 255 || !((sm.rq.mask >> s) & 1))
    return lb;
  const unsigned long long uo = a.unit_off[(size_t)bi * 8 + (size_t)s];
  const size_t fs = (size_t)br.flat * 8 + (size_t)s;
  lb.emax = a.exps[fs * kMaxBlocksPerSubband + (size_t)b];
  if (uo == ~0ull)
    return lb;
  // blocks off the request's lattice are not rebuilt (the reference's BypassDecode)
  const int* sp = sm.rq.spacing[s];
  if ((sp[0] > 1 && (4 * xb) % sp[0]) || (sp[1] > 1 && (4 * yb) % sp[1]) || (sp[2] > 1 && (4 * zb) % sp[2]))
    return lb;
  lb.np = dev::coded_planes(lb.emax, sm.rq.etol, a.end_bp);
  lb.row = a.planes + (uo & kUnitOffMask) / 8 + (size_t)b * (size_t)(uo >> kUnitStrideShift);
  return lb;
}

// 1 / 2^k as the division of 1 by 2^k rounds it (0 once 2^k overflows)
__device__ __forceinline__ double dequant_scale(int nd, int emax)
{
  const int k = 63 - nd - 1 - emax;
  return k > 1023 ? 0.0 : dev::pow2(-k);
}

// The faces: 2D blocks (tasks 0-5: faces x, y, z, by the parity of the second axis), then the
// edges and the corner (task 6), a lane per block.
template <int W>
__device__ __forceinline__ void rebuild_face(const dec_args& a, brick_smem<W>& sm, const decode_brick& br, int bi,
                                             int task, int lane, bool sig_level)
{
  if (task < 6)
  {
    const int o = task >> 1, hv = task & 1, hu = lane >> 4, ub = lane & 3, vb = (lane >> 2) & 3;
    const int s = o == 0 ? 2 * hu + hv : (o == 1 ? 4 * hu + hv : 4 * hu + 2 * hv);
    const int xb = o == 0 ? 4 : ub, yb = o == 1 ? 4 : (o == 0 ? ub : vb), zb = o == 2 ? 4 : vb;
    const lane_block lb = find_block(a, sm, br, bi, s, xb, yb, zb, true);
    double* out = sm.face[o] + (hv + 8 * vb) * kFaceRow + hu + 8 * ub;
    if (lb.np == 0)
    {
#pragma unroll
      for (int j = 0; j < 16; ++j)
        out[2 * (j >> 2) * kFaceRow + 2 * (j & 3)] = 0.0;
      return;
    }
    if (a.sig && (s > 0 || sig_level))
      sm.sig = 1;
    const double scale = dequant_scale(2, lb.emax);
    // planes 0-15 in the words' high halves, 16-31 in the low ones; 32-63 in the second word
    auto words = [&](int first, uint32_t(&w)[16]) {
#pragma unroll
      for (int k = 0; k < 16; ++k)
      {
        const uint32_t hi = first + k < lb.np ? (uint32_t)__ldg(lb.row + first + k) : 0u;
        const uint32_t lo = first + 16 + k < lb.np ? (uint32_t)__ldg(lb.row + first + 16 + k) : 0u;
        w[15 - k] = (hi << 16) | (lo & 0xffffu);
      }
      transpose_bits(w);
    };
    uint32_t h[16];
    words(0, h);
    if (lb.np <= kHighPlanes)
    {
      int32_t q[16];
#pragma unroll
      for (int j = 0; j < 16; ++j)
        q[dev::kPerm2d[j]] = from_negabinary(h[j]);
#pragma unroll
      for (int i = 0; i < 4; ++i)
        ilift4_w(q[i], q[i + 4], q[i + 8], q[i + 12]);
#pragma unroll
      for (int i = 0; i < 4; ++i)
        ilift4_w(q[4 * i], q[4 * i + 1], q[4 * i + 2], q[4 * i + 3]);
#pragma unroll
      for (int j = 0; j < 16; ++j)
        out[2 * (j >> 2) * kFaceRow + 2 * (j & 3)] = __dmul_rn(scale, (double)q[j] * 4294967296.0);
      return;
    }
    uint32_t l[16];
    words(32, l);
    long long q[16];
#pragma unroll
    for (int j = 0; j < 16; ++j)
    {
      const unsigned long long u = ((unsigned long long)h[j] << 32) | l[j];
      q[dev::kPerm2d[j]] = (long long)((u ^ dev::kNegaMask) - dev::kNegaMask);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
      ilift4_ll(q[i], q[i + 4], q[i + 8], q[i + 12]);
#pragma unroll
    for (int i = 0; i < 4; ++i)
      ilift4_ll(q[4 * i], q[4 * i + 1], q[4 * i + 2], q[4 * i + 3]);
#pragma unroll
    for (int j = 0; j < 16; ++j)
      out[2 * (j >> 2) * kFaceRow + 2 * (j & 3)] = __dmul_rn(scale, __ll2double_rn(q[j]));
    return;
  }
  // edges along z, y, x (8 blocks each) and the corner
  const int e = lane >> 3, h = (lane >> 2) & 1, kb = lane & 3;
  const bool corner = lane == 24;
  if (lane > 24)
    return;
  const int s = corner ? 0 : (e == 0 ? h : (e == 1 ? 2 * h : 4 * h));
  const int xb = e == 2 ? kb : 4, yb = e == 1 ? kb : 4, zb = corner ? 4 : (e == 0 ? kb : 4);
  const lane_block lb = find_block(a, sm, br, bi, s, xb, yb, zb, true);
  if (a.sig && lb.np && (s > 0 || sig_level))
    sm.sig = 1;
  unsigned long long u[4] = { 0, 0, 0, 0 };
  for (int k = 0; k < lb.np; ++k)
  {
    const uint32_t x = (uint32_t)__ldg(lb.row + k);
#pragma unroll
    for (int j = 0; j < 4; ++j)
      u[j] |= (unsigned long long)((x >> j) & 1u) << (63 - k);
  }
  long long q[4];
#pragma unroll
  for (int j = 0; j < 4; ++j)
    q[j] = (long long)((u[j] ^ dev::kNegaMask) - dev::kNegaMask);
  const double scale = dequant_scale(corner ? 0 : 1, lb.emax);
  if (corner)
  {
    sm.face[0][32 * kFaceRow + 32] = lb.np ? __dmul_rn(scale, __ll2double_rn(q[0])) : 0.0;
    return;
  }
  ilift4_ll(q[0], q[1], q[2], q[3]);
#pragma unroll
  for (int j = 0; j < 4; ++j)
  {
    const int p = h + 2 * (4 * kb + j);
    const int at = e == 0 ? p * kFaceRow + 32 : 32 * kFaceRow + p;
    sm.face[e == 2 ? 1 : 0][at] = lb.np ? __dmul_rn(scale, __ll2double_rn(q[j])) : 0.0;
  }
}

// A 3D block of any number of planes, by the warp, raw to the slot (its column of samples at
// `dst`, the z-planes of one parity 2 * kSlotPlane apart).
__device__ __noinline__ void rebuild_block_wide(const unsigned long long* row, int np, int emax, long long* q,
                                                double* dst, int lane)
{
  const unsigned long long x0 = lane < np ? row[lane] : 0ull, x1 = lane + 32 < np ? row[lane + 32] : 0ull;
  const unsigned long long u0 =
    ((unsigned long long)__brev(dev::warp_transpose32((uint32_t)x0, lane)) << 32) |
    __brev(dev::warp_transpose32((uint32_t)x1, lane));
  const unsigned long long u1 =
    ((unsigned long long)__brev(dev::warp_transpose32((uint32_t)(x0 >> 32), lane)) << 32) |
    __brev(dev::warp_transpose32((uint32_t)(x1 >> 32), lane));
  __syncwarp();
  q[dev::perm(3, lane)] = (long long)((u0 ^ dev::kNegaMask) - dev::kNegaMask);
  q[dev::perm(3, lane + 32)] = (long long)((u1 ^ dev::kNegaMask) - dev::kNegaMask);
  __syncwarp();
  dev::warp_inv_zfp(q, 3, lane);
  const double scale = dequant_scale(3, emax);
#pragma unroll
  for (int k = 0; k < 2; ++k)
  {
    const int j = lane + 32 * k;
    dst[(j >> 4) * 2 * kSlotPlane + ((j >> 2) & 3) * 17 + (j & 3)] = __dmul_rn(scale, __ll2double_rn(q[j]));
  }
  __syncwarp();
}

// The z sweep of one column and its store to the slot.
__device__ __forceinline__ void lift_column(double (&v)[33], const dec_args& a, int s0, double* col)
{
  const bool n0 = (a.norm_mask >> s0) & 1, n1 = (a.norm_mask >> (s0 | 1)) & 1;
  const double w0 = a.inv_weight[s0], w1 = a.inv_weight[s0 | 1];
  if (n0)
#pragma unroll
    for (int z = 0; z < 33; z += 2)
      v[z] = __dmul_rn(v[z], w0);
  if (n1)
#pragma unroll
    for (int z = 1; z < 33; z += 2)
      v[z] = __dmul_rn(v[z], w1);
  ilift33(v);
#pragma unroll
  for (int z = 0; z < 33; ++z)
    col[z * kSlotPlane] = v[z];
}

// One task of the rebuild: parities (hx, hy) and block row yb, the 4 tiles along x: 32 blocks
// (a lane each: tile t, z block zb, z parity hz), then their 64 columns along z.
template <int W>
__device__ __forceinline__ void rebuild_tiles(const dec_args& a, brick_smem<W>& sm, const decode_brick& br, int bi,
                                              int task, double* F, int warp, int lane, bool sig_level)
{
  const int hx = task >> 3, hy = (task >> 2) & 1, yb = task & 3;
  const int s0 = 4 * hx + 2 * hy;
  int32_t* const tile = sm.w[warp].tile;
  bool staged = true;   // the blocks' words are in the tile buffer (else raw samples in the slot)
  bool empty = false;   // no block of the task was decoded
  // below the coarsest level the low band's full blocks are not coded: it comes from the parent
  const bool low = s0 == 0 && sm.block[0][0] == 255;
  {
    const int t = lane & 3, zb = (lane >> 2) & 3, hz = lane >> 4, s = s0 + hz;
    const lane_block lb = find_block(a, sm, br, bi, s, t, yb, zb, true);
    if (a.sig && lb.np && (s > 0 || sig_level))
      sm.sig = 1;
    const int most = __reduce_max_sync(0xffffffffu, lb.np);
    empty = most == 0;
    int32_t* const own = tile + (16 * hz + 4 * zb) * kTileRow + t;  // + z * kTileRow + 4 * (x + 4 y)
    auto put = [&](const int32_t(&q)[64]) {
#pragma unroll
      for (int j = 0; j < 64; ++j)
        own[(j >> 4) * kTileRow + 4 * ((j & 3) + 4 * ((j >> 2) & 3))] = q[j];
    };
    bool wide = most > kSplitPlanes;
    if (!empty && !wide)
    {
      int32_t q[64];
      if (most <= 16)
        block_words<16>(lb.row, 0, lb.np, 31, q);
      else
        block_words<32>(lb.row, 0, lb.np < kHighPlanes ? lb.np : kHighPlanes, 31, q);
      if (most > kHighPlanes)
        wide = __any_sync(0xffffffffu, may_wrap(q));
      if (!wide)
      {
        inverse_zfp3(q);
        put(q);
        sm.scale[warp][lane] = lb.np ? __dmul_rn(dequant_scale(3, lb.emax), 4294967296.0) : 0.0;
        if (most > kHighPlanes)
        {
          // the planes past the 26th, added to the first part as 64-bit words
          staged = false;
          block_words<32>(lb.row, kHighPlanes, lb.np - kHighPlanes, 63 - kHighPlanes - kLowBase, q);
          inverse_zfp3(q);
          const double scale = lb.np ? dequant_scale(3, lb.emax) : 0.0;
          double* dst = F + (size_t)(8 * zb + hz) * kSlotPlane + slot_xy(8 * t + hx, 8 * yb + hy);
#pragma unroll
          for (int j = 0; j < 64; ++j)
          {
            const int32_t h = own[(j >> 4) * kTileRow + 4 * ((j & 3) + 4 * ((j >> 2) & 3))];
            const long long u = (long long)(((unsigned long long)(uint32_t)h << 32) +
                                            ((unsigned long long)(long long)q[j] << kLowBase));
            dst[(j >> 4) * 2 * kSlotPlane + ((j >> 2) & 3) * 17 + (j & 3)] = __dmul_rn(scale, __ll2double_rn(u));
          }
        }
      }
    }
    if (wide)
    {
      staged = false;
      for (int r = 0; r < 32; ++r)
      {
        const int np = __shfl_sync(0xffffffffu, lb.np, r), emax = __shfl_sync(0xffffffffu, lb.emax, r);
        const unsigned long long* row =
          (const unsigned long long*)__shfl_sync(0xffffffffu, (unsigned long long)lb.row, r);
        double* dst = F + (size_t)(8 * ((r >> 2) & 3) + (r >> 4)) * kSlotPlane + slot_xy(8 * (r & 3) + hx, 8 * yb + hy);
        rebuild_block_wide(row, np, emax, sm.w[warp].q, dst, lane);
      }
    }
    __syncwarp();
  }
  const double* P = nullptr;
  if (low && br.parent >= 0 && a.parents && (sm.rq.mask & 1))
    P = a.parents + (size_t)br.parent * (33 * kFace) + ((size_t)(br.pos[2] * 16) * kFaceRow + br.pos[1] * 16) * kFaceRow +
        br.pos[0] * 16;
#pragma unroll 1
  for (int i = 0; i < 2; ++i)
  {
    const int t = (lane >> 2) & 3, yq = 2 * i + (lane >> 4);
    const int xi = 4 * t + (lane & 3), yi = 4 * yb + yq, x = 2 * xi + hx, y = 2 * yi + hy;
    double* const col = F + slot_xy(x, y);
    double v[33];
    v[32] = sm.face[2][y * kFaceRow + x];
    if (empty)
    {
      if (!P && !__any_sync(0xffffffffu, v[32] != 0.0))
      {
        // nothing of these columns was decoded
#pragma unroll
        for (int z = 0; z < 33; ++z)
          col[z * kSlotPlane] = 0.0;
        continue;
      }
#pragma unroll
      for (int z = 0; z < 32; ++z)
        v[z] = 0.0;
    }
    else if (staged)
    {
      const int32_t* src = tile + yq * 16 + 4 * (lane & 3) + t;
      const double* sc = sm.scale[warp] + t;
#pragma unroll
      for (int zb = 0; zb < 4; ++zb)
      {
        const double e = sc[4 * zb], o = sc[4 * zb + 16];
#pragma unroll
        for (int k = 0; k < 4; ++k)
        {
          v[8 * zb + 2 * k] = __dmul_rn(e, (double)src[(4 * zb + k) * kTileRow]);
          v[8 * zb + 2 * k + 1] = __dmul_rn(o, (double)src[(16 + 4 * zb + k) * kTileRow]);
        }
      }
    }
    else
    {
#pragma unroll
      for (int z = 0; z < 32; ++z)
        v[z] = col[z * kSlotPlane];
    }
    if (low)
    {
#pragma unroll
      for (int k = 0; k < 16; ++k)
        v[2 * k] = P ? P[(size_t)k * kFace + yi * kFaceRow + xi] : 0.0;
    }
    lift_column(v, a, s0, col);
  }
  __syncwarp();
}

// One 33-sample line lifted by a warp: lane k holds samples 2k (k <= 16) and 2k + 1 (k <= 15).
__device__ __forceinline__ void ilift33_lanes(double& e, double& o, int lane)
{
  const double V = __dmul_rn(o, 0.25);
  const double Vl = __shfl_up_sync(0xffffffffu, V, 1);
  if (lane > 0)
    e = __dsub_rn(e, Vl);
  if (lane < 16)
    e = __dsub_rn(e, V);
  const double r = __shfl_down_sync(0xffffffffu, e, 1);
  o = __dadd_rn(o, __dmul_rn(lane < 15 ? __dadd_rn(e, r) : __dadd_rn(r, e), 0.5));
}

template <int W>
__global__ void __launch_bounds__(32 * W, 16 / W) k_decode_bricks(const dec_args a)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  brick_smem<W>& sm = *reinterpret_cast<brick_smem<W>*>(smem_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double* const F = a.slots + (size_t)blockIdx.x * (size_t)kSlotBrick;
  const bool sig_level = a.level + 1 == a.nlevels;
  // the level's block walk, by block position
  for (int i = tid; i < 8 * 128; i += 32 * W)
    (&sm.block[0][0])[i] = 255;
  __syncthreads();
  for (int i = tid; i < 8 * kMaxBlocksPerSubband; i += 32 * W)
  {
    const int s = i / kMaxBlocksPerSubband, b = i % kMaxBlocksPerSubband;
    if (b >= a.nblocks[s])
      continue;
    const uint64_t g = a.geom[(size_t)s * kMaxBlocksPerSubband + b];
    const int xb = (int)(g & 0xff), yb = (int)((g >> 8) & 0xff), zb = (int)((g >> 16) & 0xff);
    if (xb < 5 && yb < 5 && zb < 5)
      sm.block[s][(zb * 5 + yb) * 5 + xb] = (uint8_t)b;
  }
  for (int bi = blockIdx.x; bi < a.nbricks; bi += gridDim.x)
  {
    // the brick's and its request's parameters to shared memory: read all through the brick,
    // between stores that would have them loaded from global memory again each time
    {
      static_assert(sizeof(decode_brick) % 4 == 0 && sizeof(decode_target) % 4 == 0, "copied as words");
      constexpr int nb = (int)(sizeof(decode_brick) / 4), nr = (int)(sizeof(decode_target) / 4);
      if (tid < nb)
        reinterpret_cast<uint32_t*>(&sm.br)[tid] = reinterpret_cast<const uint32_t*>(a.bricks + bi)[tid];
      for (int i = tid - 64; i >= 0 && i < nr; i += 32 * W)
        reinterpret_cast<uint32_t*>(&sm.rq)[i] = reinterpret_cast<const uint32_t*>(a.reqs + a.bricks[bi].req)[i];
    }
    if (tid == 0)
      sm.sig = 0;
    __syncthreads();
    const decode_target& rq = sm.rq;
    const decode_brick& br = sm.br;
    // 1: the faces
    if (warp < 7)
      rebuild_face(a, sm, br, bi, warp, lane, sig_level);
    __syncthreads();
    // 2: blocks and z sweep; the columns of the faces x = 32 and y = 32 (and their common one)
    for (int t = warp; t < 19; t += W)
    {
      if (t < 16)
      {
        rebuild_tiles(a, sm, br, bi, t, F, warp, lane, sig_level);
        continue;
      }
      const int x = t == 17 ? lane : 32, y = t == 16 ? lane : 32;
      if (t == 18 && lane > 0)
        continue;
      const double* f = t == 17 ? sm.face[1] + x : sm.face[0] + y;
      double v[33];
#pragma unroll
      for (int z = 0; z < 33; ++z)
        v[z] = f[z * kFaceRow];
      lift_column(v, a, ((x & 1) << 2) | ((y & 1) << 1), F + slot_xy(x, y));
    }
    __syncthreads();
    if (a.sig && tid == 0 && br.store >= 0)
      a.sig[br.store] = sm.sig;
    // 3: y and x sweeps, a warp per z-plane, and the rows' way out (Core/idx2Decode.cpp:431-442
    // CopyGridGrid on the output level)
    const bool vec4 = a.out_f32 && rq.is_output && br.dims[0] == 32 && br.src_from[0] == 0 && br.src_strd[0] == 1 &&
                      br.dst_strd[0] == 1 && br.dst_from[0] % 4 == 0 && rq.out_dims[0] % 4 == 0 &&
                      (reinterpret_cast<uintptr_t>(rq.out) & 15) == 0;
    const bool output = rq.is_output != 0;
    const int nplanes = output ? br.dims[2] : 33;
    // row r of output plane p goes to out0 + p * out_z + r * out_y (elements), from row
    // src_y + r * src_sy of the brick's plane src_z + p * src_sz
    const int nx = br.dims[0], ny = br.dims[1];
    const int src_y = br.src_from[1], src_sy = br.src_strd[1];
    const int src_z = br.src_from[2], src_sz = br.src_strd[2];
    const long long row_n = rq.out_dims[0], plane_n = row_n * rq.out_dims[1];
    const long long out_y = br.dst_strd[1] * row_n, out_z = br.dst_strd[2] * plane_n;
    const long long out0 = br.dst_from[2] * plane_n + br.dst_from[1] * row_n + br.dst_from[0];
    const int src_x = br.src_from[0] + lane * br.src_strd[0];
    const long long dst_x = (long long)lane * br.dst_strd[0];
    for (int p = warp; p < nplanes; p += W)
    {
      const int z = output ? src_z + p * src_sz : p;
      const double* const S = F + (size_t)z * kSlotPlane;
      double* const T = sm.w[warp].plane;
      {
        // column 32, a sample pair per lane
        double e = lane < 17 ? S[slot_xy(32, 0) + 17 * lane] : 0.0;
        double o = lane < 16 ? S[slot_xy(32, 1) + 17 * lane] : 0.0;
        const double* c = S + slot_xy(lane, 0);
        double v[33];
#pragma unroll
        for (int y = 0; y < 33; ++y)
          v[y] = c[(y & 1) * (17 * 17) + (y >> 1) * 17];
        // (column 32 is waited for with the others: left to the compiler its loads went after the
        // lift and a second round trip to L2; 1024^3 13.9 -> 13.3 ms)
        asm volatile("" : "+d"(e), "+d"(o));
        ilift33_lanes(e, o, lane);
        if (lane < 17)
          T[2 * lane * 33 + 32] = e;
        if (lane < 16)
          T[(2 * lane + 1) * 33 + 32] = o;
        ilift33(v);
#pragma unroll
        for (int y = 0; y < 33; ++y)
          T[y * 33 + lane] = v[y];
        // the plane is done with: its lines need not go to memory (1024^3: 13.9 against 14.3 ms)
        __syncwarp();
        for (int k = lane; k < kSlotPlane / 16; k += 32)
          asm volatile("discard.global.L2 [%0], 128;\n" ::"l"(S + 16 * k) : "memory");
      }
      __syncwarp();
      double v[33];
#pragma unroll
      for (int x = 0; x < 33; ++x)
        v[x] = T[lane * 33 + x];
      ilift33(v);
      if (!output)
      {
        double e = lane < 17 ? T[32 * 33 + 2 * lane] : 0.0;
        double o = lane < 16 ? T[32 * 33 + 2 * lane + 1] : 0.0;
        ilift33_lanes(e, o, lane);
        __syncwarp();
#pragma unroll
        for (int x = 0; x < 33; ++x)
          T[lane * 33 + x] = v[x];
        if (lane < 17)
          T[32 * 33 + 2 * lane] = e;
        if (lane < 16)
          T[32 * 33 + 2 * lane + 1] = o;
        __syncwarp();
        double* out = a.bricks_out + (size_t)br.store * (33 * kFace) + (size_t)z * kFace;
        for (int i = lane; i < kFace; i += 32)
          out[i] = T[i];
      }
      else
      {
        const long long at = out0 + p * out_z;
        __syncwarp();
        if (vec4)
        {
          float* R = sm.w[warp].rows;
#pragma unroll
          for (int x = 0; x < 32; x += 4)
            *reinterpret_cast<float4*>(R + lane * 36 + x) =
              make_float4(__double2float_rn(v[x]), __double2float_rn(v[x + 1]), __double2float_rn(v[x + 2]),
                          __double2float_rn(v[x + 3]));
          __syncwarp();
          // 4 rows at a time, 8 lanes each
          const float* r0 = R + (src_y + (lane >> 3) * src_sy) * 36 + 4 * (lane & 7);
          float* g = (float*)rq.out + at + (lane >> 3) * out_y + 4 * (lane & 7);
#pragma unroll
          for (int k = 0; k < 8; ++k)
            if (4 * k + (lane >> 3) < ny)
              __stcs(reinterpret_cast<float4*>(g + 4 * k * out_y),
                     *reinterpret_cast<const float4*>(r0 + 4 * k * src_sy * 36));
        }
        else
        {
#pragma unroll
          for (int x = 0; x < 33; ++x)
            T[lane * 33 + x] = v[x];
          __syncwarp();
          if (lane < nx)
          {
            const double* r0 = T + src_y * 33 + src_x;
            if (a.out_f32)
            {
              float* g = (float*)rq.out + at + dst_x;
#pragma unroll 8
              for (int r = 0; r < ny; ++r)
                __stcs(g + r * out_y, __double2float_rn(r0[r * src_sy * 33]));
            }
            else
            {
              double* g = (double*)rq.out + at + dst_x;
#pragma unroll 8
              for (int r = 0; r < ny; ++r)
                __stcs(g + r * out_y, r0[r * src_sy * 33]);
            }
          }
        }
      }
      __syncwarp();
    }
    __syncthreads();
  }
}
