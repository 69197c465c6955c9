// 3x3x3 convolutions of channels-last BF16 volumes on the sm_100a tensor cores
// (tcgen05), for the learned preconditioner's U-Net.
//
// Forward (and, with flipped / transposed weights, the input gradient) is an
// implicit GEMM: D[v][co] = sum_t sum_ci X[v + off(t)][ci] W[co][t][ci].
// A CTA owns a box of bj lines x bz voxels along z of bi planes along x and nt
// of the output channels.  It keeps its channels' weights of all 27 taps and a
// ring of input planes, each with a one-voxel halo in j and k, in shared
// memory in the canonical no-swizzle K-major layout (8 rows x 16 bytes per
// core matrix): the voxels of a haloed plane, line after line, are the rows,
// 16 bytes apart, one run of rows per 8-channel chunk.  A tap is then the
// same rows shifted by di planes, dj lines and dk rows, which is only another
// start address in the MMA's descriptor: every voxel is copied to shared
// memory once per plane ring and not once per tap, and the 27 taps of a plane
// are issued back to back.  M = 128 consecutive rows (the halo rows among
// them compute values that are not stored), N = nt, K = 16 channels per MMA.
// One elected thread issues tcgen05.mma.kind::f16 (BF16 operands, FP32
// accumulator in tensor memory) and commits a plane's MMAs to an mbarrier;
// meanwhile all threads copy the plane after next (cp.async, zero filled
// outside the volume) and write the previous plane's result: tcgen05.ld (warp
// w owns lanes 32w..32w+31 = rows), bias, ReLU, BF16 (and optionally FP32).
//
// What bounds it: MMAs of N = 16..64 are short, and their rate is that of the
// one thread that issues them and of the A operand's reads from shared memory
// (4 KB, 32 cycles), so the tensor pipe cannot fill at these channel counts; the
// box is chosen (conv_tile) so that enough CTAs run and few halo rows are
// computed.  A network forward at 64 x 72 x 128 took 1.89 ms with the voxels
// copied again for every tap, 1.14 ms without, and takes 0.84 ms now that the
// issuing thread only adds to its descriptors (forming them anew took longer
// than the MMAs: 80 -> 32 channels at 32^3 67.7 us, now 55.4; 16 -> 16 at 64 x 72
// x 128 80.1, now 58.5).
//
// The weight gradient dW[co][t][ci] = sum_v dY[v][co] X[v + off(t)][ci] reads
// the same images as MN-major operands (rows = voxels = K): A is the three
// planes' chunks of X side by side, so M runs over (di, ci), N over co, and a
// tap's (dj, dk) is again a row shift.
// On the FP32 pipes it was 14.0 of the 18.2 ms of the gradients of four 32^3
// crops; all of those take 3.5 ms now.
//
// Every mbarrier wait is bounded; a wait that gives up sets the caller's
// error word, waits (bounded) for the MMAs in flight and frees the tensor
// memory before returning.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

namespace efsi {
namespace conv {

constexpr int kTileM = 128;          // rows per MMA
constexpr int kThreads = 128;        // 4 warps: one TMEM lane quadrant each
constexpr long long kWaitLimit = 4000000000LL;  // ~2 s of clock64

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Shared-memory matrix descriptor (SWIZZLE_NONE, K-major, version 1).
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFFu);
  d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1 << 46;
  return d;
}

// Instruction descriptor of kind::f16: BF16 A and B (both K-major, or both
// MN-major), FP32 D.
__host__ __device__ constexpr uint32_t idesc_bf16(int m, int n, bool mn_major = false) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (mn_major ? (3u << 15) : 0u) | ((uint32_t)(n >> 3) << 17) |
         ((uint32_t)(m >> 4) << 24);
}

__device__ __forceinline__ void mbar_init(uint64_t* bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ bool mbar_test(uint64_t* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, unsigned parity) {
  if (mbar_test(bar, parity)) return true;
  const long long t0 = clock64();
  while (!mbar_test(bar, parity))
    if (clock64() - t0 > kWaitLimit) return false;
  return true;
}

// 16-byte asynchronous copy global -> shared; src_bytes = 0 writes zeros.
__device__ __forceinline__ void cp_async16(void* dst, const void* src, int src_bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(src_bytes)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tc_mma(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, int accum) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accum)
      : "memory");
}

__device__ __forceinline__ void tc_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

__device__ __forceinline__ void tc_ld16(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
      "%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int q = 0; q < 16; ++q) v[q] = __uint_as_float(r[q]);
}

// A volume's channels-last input, [n][cin]; with `coarse` the first ca channels
// come from the parent voxels of a ceil-halved volume (nearest-neighbour
// upsampling) and the other cin - ca from x, without the concatenation being
// stored.
struct ConvInput {
  const __nv_bfloat16* x;
  const __nv_bfloat16* coarse;
  int ca;
};

struct ConvArgs {
  int nx, ny, nz;
  int cin, cout;                 // multiples of 16
  ConvInput in;
  const __nv_bfloat16* w;        // [cout][27][cin]
  const float* bias;             // [cout] or null
  int relu;                      // apply ReLU in the epilogue
  __nv_bfloat16* y;              // [n][cout] or null
  float* yf;                     // [n][cout] FP32 copy or null
  int* error;                    // set to 1 when a wait gives up
};

// The box of one CTA and its shared-memory layout.
struct ConvTile {
  int bz, zp;        // output voxels per line, rows per line (bz + 2)
  int bj, bi;        // lines per plane, planes
  int nt;            // output channels (the last split may have fewer)
  int mt;            // 128-row MMA tiles per plane
  int slots;         // planes in the ring: 3 (bi == 1) or 4
  int nzb, njb, nib; // boxes along z, y, x
  int cs;            // bytes between the chunks of the input
  int woff;          // byte offset of the weights
  int smem;          // dynamic shared memory
  unsigned cols;     // tensor-memory columns
};

constexpr int kGuard = 128;  // bytes before the first row (tap -1 of row 0)

__host__ __device__ inline uint32_t tmem_columns(int n) {
  uint32_t c = 32;
  while ((int)c < n) c <<= 1;
  return c;
}

// Eight channels, or zeros: with kVec one 16-byte asynchronous copy, which
// needs an aligned source, otherwise a load per element.
template <bool kVec>
__device__ __forceinline__ void copy8(void* dst, const __nv_bfloat16* src, bool ok) {
  if (kVec) {
    cp_async16(dst, src, ok ? 16 : 0);
  } else {
    __align__(16) __nv_bfloat16 v[8];
    for (int q = 0; q < 8; ++q) v[q] = ok ? src[q] : __float2bfloat16_rn(0.0f);
    *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(v);
  }
}

__device__ __forceinline__ bool in_volume(int nx, int ny, int nz, int i, int j, int k) {
  return i >= 0 && i < nx && j >= 0 && j < ny && k >= 0 && k < nz;
}

// Channel ch of voxel (i, j, k) of the volume.
__device__ __forceinline__ const __nv_bfloat16* channel_at(const ConvInput& in, int ny, int nz, int cin, int i, int j,
                                                           int k, int ch) {
  if (ch < in.ca)
    return in.coarse + (((int64_t)(i >> 1) * ((ny + 1) >> 1) + (j >> 1)) * ((nz + 1) >> 1) + (k >> 1)) * in.ca + ch;
  return in.x + (((int64_t)i * ny + j) * nz + k) * (cin - in.ca) + (ch - in.ca);
}

// 16-byte chunk c of voxel (i, j, k), or zeros outside the volume.
template <bool kVec>
__device__ __forceinline__ void copy_chunk(unsigned char* dst, const ConvInput& in, int nx, int ny, int nz, int cin,
                                           int i, int j, int k, int c) {
  const bool ok = in_volume(nx, ny, nz, i, j, k);
  copy8<kVec>(dst, ok ? channel_at(in, ny, nz, cin, i, j, k, c * 8) : in.x, ok);
}

__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(cols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free(uint32_t tmem, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols) : "memory");
}

__global__ void __launch_bounds__(kThreads) k_conv3d_tc(ConvArgs A, ConvTile T) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t bars[2];
  __shared__ uint32_t tmem_slot;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int cin = A.cin, kch = cin / 8, nt = T.nt, zp = T.zp;
  int b = blockIdx.x;
  const int z0 = (b % T.nzb) * T.bz;
  b /= T.nzb;
  const int j0 = (b % T.njb) * T.bj, ib = (b / T.njb) * T.bi, ie = min(A.nx, ib + T.bi);
  const int n0 = blockIdx.y * nt;
  const int rows = (T.bj + 2) * zp, plane_bytes = rows * 16;
  unsigned char* sx = smem_raw + kGuard;
  unsigned char* sw = smem_raw + T.woff;

  if (tid == 0) {
    mbar_init(&bars[0]);
    mbar_init(&bars[1]);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) tmem_alloc(&tmem_slot, T.cols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;

  // plane p lives in slot (p - ib + 1) % slots
  auto load_plane = [&](int p) {
    unsigned char* dst = sx + ((p - ib + 1) % T.slots) * plane_bytes;
    for (int e = tid; e < rows * kch; e += kThreads) {
      const int row = e / kch, c = e - row * kch;
      const int line = row / zp, z = row - line * zp;
      copy_chunk<true>(dst + c * T.cs + row * 16, A.in, A.nx, A.ny, A.nz, cin, p, j0 - 1 + line, z0 - 1 + z, c);
    }
  };
  for (int q = tid; q < 27 * nt * kch; q += kThreads) {
    const int c = q % kch, r = q / kch, t = r % 27, co = r / 27;
    const bool in = n0 + co < A.cout;  // the last split may have fewer channels
    cp_async16(sw + ((t * kch + c) * nt + co) * 16, in ? A.w + ((int64_t)(n0 + co) * 27 + t) * cin + c * 8 : A.w,
               in ? 16 : 0);
  }
  for (int p = ib - 1; p <= ib + 1; ++p) load_plane(p);
  cp_async_commit();
  cp_async_wait<0>();
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncthreads();

  const uint32_t idesc = idesc_bf16(kTileM, nt);
  // The 27 taps of output plane i into accumulator set `buf`.  A descriptor's
  // low bits are the start address in 16-byte units, and a row is one: the
  // thread that issues only adds to the two descriptors.
  const uint64_t adesc = umma_desc(smem_u32(sx), (uint32_t)T.cs, 128);
  const uint64_t bdesc = umma_desc(smem_u32(sw), (uint32_t)(nt * 16), 128);
  auto issue = [&](int i, int buf) {
    tc_fence_after();
    for (int m = 0; m < T.mt; ++m) {
      const uint32_t acc = tmem + (uint32_t)((buf * T.mt + m) * nt);
      uint64_t b = bdesc;
      for (int di = 0; di < 3; ++di) {
        // (dj, dk) of the plane i + di - 1: rows dj * zp + dk - 1 on
        uint64_t plane = adesc + (uint64_t)(((i + di - ib) % T.slots) * rows + m * kTileM) - 1;
        for (int dj = 0; dj < 3; ++dj, plane += zp)
          for (int dk = 0; dk < 3; ++dk) {
            uint64_t a = plane + dk;
            for (int ks = 0; ks < kch / 2; ++ks, a += T.cs / 8, b += 2 * nt)
              tc_mma(acc, a, b, idesc, (b != bdesc) ? 1 : 0);
          }
      }
    }
    tc_commit(&bars[buf]);
  };
  auto epilogue = [&](int i, int buf) {
    tc_fence_after();
    for (int m = 0; m < T.mt; ++m) {
      const int row = m * kTileM + warp * 32 + lane;
      const int line = row / zp, z = row - line * zp;
      const int j = j0 + line, k = z0 + z - 1;
      const bool in = line < T.bj && z >= 1 && z <= T.bz && j < A.ny && k < A.nz;
      const int64_t at = (((int64_t)i * A.ny + j) * A.nz + k) * A.cout + n0;
      for (int c0 = 0; c0 < min(nt, A.cout - n0); c0 += 16) {
        float acc[16];
        tc_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)((buf * T.mt + m) * nt + c0), acc);
        if (!in) continue;
#pragma unroll
        for (int q = 0; q < 16; ++q) {
          const float a = acc[q] + (A.bias != nullptr ? __ldg(A.bias + n0 + c0 + q) : 0.0f);
          acc[q] = A.relu ? fmaxf(a, 0.0f) : a;
        }
        if (A.y != nullptr) {
          __align__(16) __nv_bfloat16 hb[16];
#pragma unroll
          for (int q = 0; q < 16; ++q) hb[q] = __float2bfloat16_rn(acc[q]);
          uint4* dst = reinterpret_cast<uint4*>(A.y + at + c0);
          dst[0] = reinterpret_cast<const uint4*>(hb)[0];
          dst[1] = reinterpret_cast<const uint4*>(hb)[1];
        }
        if (A.yf != nullptr) {
          float4* dst = reinterpret_cast<float4*>(A.yf + at + c0);
#pragma unroll
          for (int q = 0; q < 4; ++q) dst[q] = make_float4(acc[4 * q], acc[4 * q + 1], acc[4 * q + 2], acc[4 * q + 3]);
        }
      }
    }
    tc_fence_before();
  };
  // Plane i's MMAs run while plane i + 2 is copied and plane i - 1's result is
  // written.  Plane i + 2 takes the slot of plane i - 2, which the MMAs of
  // plane i - 1 read last; the rows past a plane's last line that an MMA tile
  // also covers may see it arrive, and are not stored.
  bool ok = true;
  int last = -1;  // last plane whose MMAs were issued, from ib
  for (int q = 0; q < ie - ib; ++q) {
    if (tid == 0) issue(ib + q, q & 1);
    last = q;
    bool good = true;
    if (q > 0) good = mbar_wait_bounded(&bars[(q - 1) & 1], (unsigned)(((q - 1) >> 1) & 1));
    if (good && q + 1 < ie - ib) load_plane(ib + q + 2);
    cp_async_commit();
    // (the same for all lanes of a warp: tcgen05.ld is a warp's instruction;
    // the exit is taken by all threads together, after the copies have landed)
    good = __all_sync(0xffffffffu, good);
    if (good && q > 0) epilogue(ib + q - 1, (q - 1) & 1);
    cp_async_wait<0>();
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (!__syncthreads_and(good)) {
      ok = false;
      break;
    }
  }
  const bool done = mbar_wait_bounded(&bars[last & 1], (unsigned)((last >> 1) & 1));
  ok = __syncthreads_and(ok && done);
  if (ok)
    epilogue(ib + last, last & 1);
  else if (tid == 0)
    atomicExch(A.error, 1);
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_free(tmem, T.cols);
  }
}

// ---------------------------------------------------------------------------
// Weight gradient: dw[co][t][ci] += sum_v dy[v][co] X[v + off(t)][ci].
// ---------------------------------------------------------------------------
struct WgradArgs {
  int nx, ny, nz;
  int cin, cout;            // multiples of 16
  ConvInput in;
  const __nv_bfloat16* dy;  // [n][cout]
  float* dw;                // [cout][27][cin]
  int* error;               // as in ConvArgs; null: dw[0] becomes NaN instead
};

// One CTA: one dj, `ndk` of the dk (grid y), mb of the 128-row blocks of
// (di, ci) and nt output channels (grid z), boxes of bj lines x bz voxels of a
// plane (grid x, strided).
struct WgradTile {
  int bz, zp, bj;
  int rows;         // K rows of a box, bj * zp rounded up to 16
  int nzb, njb;
  int items;        // boxes
  int ndk, mb, nmb, nt;
  int cs, ds;       // bytes between the chunks of x and of dy
  int doff;         // byte offset of dy
  int smem;
  unsigned cols;
};

// One CTA's share of dw[co][tap (di, dj, dk)][ci], product by product.  The
// row shifts of k_wgrad_tc pair zero rows of dy with voxels of x that are not
// theirs (the halo columns of a box): nothing while x is finite, a NaN where it
// is not.  A sum that came out infinite or NaN is formed again here.
__device__ __noinline__ float wgrad_direct(const WgradArgs& A, const WgradTile& T, int di, int dj, int dk, int ci,
                                           int co) {
  float s = 0.0f;
  for (int item = blockIdx.x; item < T.items; item += gridDim.x) {
    const int z0 = (item % T.nzb) * T.bz, rest = item / T.nzb;
    const int j0 = (rest % T.njb) * T.bj, i = rest / T.njb;
    const int j1 = min(A.ny, j0 + T.bj), k1 = min(A.nz, z0 + T.bz);
    for (int j = j0; j < j1; ++j)
      for (int k = z0; k < k1; ++k) {
        const float g = __bfloat162float(A.dy[(((int64_t)i * A.ny + j) * A.nz + k) * A.cout + co]);
        float x = 0.0f;  // (times a dy that is infinite: NaN)
        if (in_volume(A.nx, A.ny, A.nz, i + di, j + dj, k + dk))
          x = __bfloat162float(*channel_at(A.in, A.ny, A.nz, A.cin, i + di, j + dj, k + dk, ci));
        s = fmaf(g, x, s);
        if (isnan(s)) return s;
      }
  }
  return s;
}

// kVec: x and dy start on 16-byte boundaries (their rows are multiples of 32
// bytes); they may start at any element otherwise.
template <bool kVec>
__global__ void __launch_bounds__(kThreads) k_wgrad_tc(const __grid_constant__ WgradArgs A,
                                                       const __grid_constant__ WgradTile T) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t bar;
  __shared__ uint32_t tmem_slot;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int cin = A.cin, kch = cin / 8, nch = T.nt / 8, zp = T.zp;
  const int dj = (int)blockIdx.y % 3 - 1, dk0 = ((int)blockIdx.y / 3) * T.ndk - 1;
  const int m0 = ((int)blockIdx.z % T.nmb) * T.mb, n0 = ((int)blockIdx.z / T.nmb) * T.nt;
  // the chunks of the three planes this CTA's M blocks cover
  const int g0 = m0 * (kTileM / 8), g1 = min(3 * kch, g0 + T.mb * (kTileM / 8));
  unsigned char* sx = smem_raw + kGuard;
  unsigned char* sd = smem_raw + T.doff;

  if (tid == 0) {
    mbar_init(&bar);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) tmem_alloc(&tmem_slot, T.cols);
  // the row before the first and the row after the last of every chunk of x
  // meet zero rows of dy: they only have to be finite
  for (int g = tid; g < g1 - g0; g += kThreads) {
    *reinterpret_cast<uint4*>(sx + g * T.cs - 16) = make_uint4(0u, 0u, 0u, 0u);
    *reinterpret_cast<uint4*>(sx + g * T.cs + T.rows * 16) = make_uint4(0u, 0u, 0u, 0u);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  const uint32_t idesc = idesc_bf16(kTileM, T.nt, true);

  bool ok = true;
  int uses = 0;
  for (int item = blockIdx.x; item < T.items; item += gridDim.x, ++uses) {
    const int z0 = (item % T.nzb) * T.bz, rest = item / T.nzb;
    const int j0 = (rest % T.njb) * T.bj, i = rest / T.njb;
    // Row r of a box is voxel (line r / zp, z0 - 1 + r % zp): dy is zero on
    // the halo columns and beyond the box, x of line j + dj is what it is
    // there (zero outside the volume).
    for (int e = tid; e < T.rows * (g1 - g0); e += kThreads) {
      const int row = e / (g1 - g0), g = g0 + e - row * (g1 - g0);
      const int line = row / zp, z = row - line * zp, di = g / kch - 1, c = g % kch;
      copy_chunk<kVec>(sx + (g - g0) * T.cs + row * 16, A.in, A.nx, A.ny, A.nz, cin, i + di,
                 line < T.bj ? j0 + line + dj : -1, z0 - 1 + z, c);
    }
    for (int e = tid; e < T.rows * nch; e += kThreads) {
      const int row = e / nch, c = e - row * nch;
      const int line = row / zp, z = row - line * zp, j = j0 + line, k = z0 - 1 + z;
      const bool in = line < T.bj && z >= 1 && z <= T.bz && j < A.ny && k < A.nz;
      copy8<kVec>(sd + c * T.ds + row * 16,
                  in ? A.dy + (((int64_t)i * A.ny + j) * A.nz + k) * A.cout + n0 + c * 8 : A.dy, in);
    }
    cp_async_commit();
    cp_async_wait<0>();
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (tid == 0) {
      tc_fence_after();
      for (int d = 0; d < T.ndk; ++d)
        for (int m = 0; m < T.mb; ++m) {
          const uint32_t acc = tmem + (uint32_t)((d * T.mb + m) * T.nt);
          const uint32_t a0 = smem_u32(sx) + (uint32_t)(m * (kTileM / 8) * T.cs + (dk0 + d) * 16);
          for (int r = 0; r < T.rows; r += 16)
            tc_mma(acc, umma_desc(a0 + (uint32_t)(r * 16), 128, (uint32_t)T.cs),
                   umma_desc(smem_u32(sd) + (uint32_t)(r * 16), 128, (uint32_t)T.ds), idesc,
                   (uses > 0 || r > 0) ? 1 : 0);
        }
      tc_commit(&bar);
    }
    // the buffers are refilled for the next box once the MMAs have read them
    const bool good = mbar_wait_bounded(&bar, (unsigned)(uses & 1));
    if (!__syncthreads_and(good)) {
      ok = false;
      break;
    }
  }
  if (!ok && tid == 0) {
    if (A.error != nullptr)
      atomicExch(A.error, 1);
    else
      A.dw[0] = __int_as_float(0x7fc00000);
  }
  if (ok && uses > 0) {
    tc_fence_after();
    for (int d = 0; d < T.ndk; ++d)
      for (int m = 0; m < T.mb; ++m) {
        const int row = (m0 + m) * kTileM + warp * 32 + lane;  // of (di, ci)
        const int di = row / cin, ci = row - di * cin;
        const int t = di * 9 + (dj + 1) * 3 + dk0 + d + 1;
        for (int c0 = 0; c0 < T.nt; c0 += 16) {
          float acc[16];
          tc_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)((d * T.mb + m) * T.nt + c0), acc);
          if (di >= 3) continue;
          unsigned again = 0;
#pragma unroll
          for (int q = 0; q < 16; ++q) {
            if (!isfinite(acc[q]))
              again |= 1u << q;
            else if (acc[q] != 0.0f)
              atomicAdd(A.dw + ((int64_t)(n0 + c0 + q) * 27 + t) * cin + ci, acc[q]);
          }
          for (; again != 0; again &= again - 1) {
            const int co = n0 + c0 + __ffs(again) - 1;
            atomicAdd(A.dw + ((int64_t)co * 27 + t) * cin + ci, wgrad_direct(A, T, di - 1, dj, dk0 + d, ci, co));
          }
        }
      }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_free(tmem, T.cols);
  }
}

// ---------------------------------------------------------------------------
// Tiles
// ---------------------------------------------------------------------------
constexpr int kMaxSmem = 222 * 1024;

// Bytes between chunks: `bytes` rounded up to 64 past a multiple of 128, so
// that the two chunks of neighbouring voxels' copies fall on different banks.
inline int chunk_stride(int bytes) { return ((bytes + 127) & ~127) + 64; }

// The CTAs of one SM together may not ask for more than its 512 tensor-memory
// columns, and convolutions and weight gradients (of several networks, too)
// run beside each other: a launch takes the same share of the SM's 228 KB as
// of its columns, less the 1 KB the system keeps per CTA and 256 bytes, so that
// 512 / cols of them still fit.  The shares of all 512 columns leave at most
// 4 KB, and the smallest CTA takes 14: whichever launches meet on an SM, their
// columns fit it too.  (At the cap of kMaxSmem what is left holds no CTA.)
inline int smem_for(int bytes, unsigned cols) {
  const int share = 228 * 1024 / 512 * (int)cols - 1024 - 256;
  return std::max(bytes, std::min(share, kMaxSmem));
}

// The box of a convolution: among the line lengths, MMA tiles per plane,
// planes per CTA and channel splits that fit, the one with the least estimated
// cycles -- per SM, the CTAs it gets in turn, each a fixed start (about 4000
// cycles: launch, first copies, first MMA) and 250 a plane, its copies at 64
// bytes a cycle and its MMAs at 36 cycles (the A operand's shared-memory read).
// The estimate ranks boxes, it does not time them (the measured times are 2.5
// to 5 times as long).  Over 16530 boxes of 237 layer shapes, 2^3 to 96 x 96 x
// 64 voxels and 16 to 112 channels, its choice is 2.3% off the best box on
// average and 32% at worst; without the cycles per plane, which keep few CTAs
// from marching over many planes, it is 5% and 82%.
inline bool conv_tile(int nx, int ny, int nz, int cin, int cout, ConvTile& best) {
  double least = 1e300;
  const int kch = cin / 8;
  for (int zcap : {62, 30, 14, 6})
    for (int mt : {4, 2, 1})
      for (int nt = std::min(cout, 128) / 16 * 16; nt >= 16; nt -= 16) {
        const int splits = (cout + nt - 1) / nt;
        if (nt > 16 && (cout + nt - 17) / (nt - 16) == splits) continue;  // 16 channels fewer do as well
        for (int bi : {16, 8, 4, 2, 1, 0}) {  // 0: one plane of one line, the least shared memory
          if (bi > 1 && bi > nx) continue;
          ConvTile t;
          t.nt = nt;
          t.mt = mt;
          t.bi = std::max(bi, 1);
          t.slots = bi > 1 ? 4 : 3;
          t.nzb = (nz + zcap - 1) / zcap;
          t.bz = (nz + t.nzb - 1) / t.nzb;
          t.zp = t.bz + 2;
          t.bj = bi == 0 ? 1 : std::min(ny, mt * kTileM / t.zp);
          t.njb = (ny + t.bj - 1) / t.bj;
          t.bj = (ny + t.njb - 1) / t.njb;
          if ((mt - 1) * kTileM >= t.bj * t.zp) continue;  // a whole MMA tile without a row
          t.nib = (nx + t.bi - 1) / t.bi;
          const int rows = (t.bj + 2) * t.zp, w = 27 * kch * nt * 16;
          t.cs = chunk_stride(t.slots * rows * 16);
          // an MMA tile may reach past the last plane's rows: into the weights
          t.woff = (kGuard + kch * t.cs + 127) & ~127;
          const int used = t.woff + std::max(w, kTileM * 16 + 64);
          t.cols = tmem_columns((bi > 1 ? 2 : 1) * mt * nt);
          if (used > kMaxSmem || t.cols > 512) continue;
          t.smem = smem_for(used, t.cols);
          const int per_sm = std::max(1, 228 * 1024 / (t.smem + 1024));
          const double ctas = (double)t.nzb * t.njb * t.nib * splits;
          const double mma = (double)t.bi * mt * 27 * (kch / 2) * 36;
          const double copy = (w + (t.bi + 2.0) * rows * cin * 2) / 64;
          const double waves = std::max(1.0, std::ceil(ctas / (148.0 * per_sm)));
          const double cycles = waves * (4000 + 250.0 * t.bi) + std::ceil(ctas / 148.0) * std::max(mma, copy) +
                                (w + 3.0 * rows * cin * 2) / 64;
          if (cycles < least) {
            least = cycles;
            best = t;
          }
        }
      }
  return least < 1e300;
}

inline bool wgrad_tile(int nx, int ny, int nz, int cin, int cout, WgradTile& t) {
  const int blocks = (3 * cin + kTileM - 1) / kTileM;
  // as many (dk, M block, channel) accumulators as tensor memory holds, and
  // boxes of about 256 rows that fit the shared memory
  bool found = false;
  for (int ndk : {3, 1}) {
    for (int mb = std::min(blocks, 4); mb >= 1 && !found; --mb)
      for (int nt = std::min(cout, 128) / 16 * 16; nt >= 16 && !found; nt -= 16)
        if (cout % nt == 0 && ndk * mb * nt <= 256) {
          t.ndk = ndk;
          t.mb = mb;
          t.nt = nt;
          found = true;
        }
    if (found) break;
  }
  if (!found) return false;
  t.nmb = (blocks + t.mb - 1) / t.mb;
  t.cols = tmem_columns(t.ndk * t.mb * t.nt);
  for (int target : {512, 256, 128, 64, 32}) {
    t.nzb = (nz + 61) / 62;
    t.bz = (nz + t.nzb - 1) / t.nzb;
    if (t.bz + 2 > target) {
      t.nzb = (nz + target - 3) / (target - 2);
      t.bz = (nz + t.nzb - 1) / t.nzb;
    }
    t.zp = t.bz + 2;
    t.bj = std::max(1, std::min(ny, target / t.zp));
    t.njb = (ny + t.bj - 1) / t.bj;
    t.bj = (ny + t.njb - 1) / t.njb;
    t.rows = (t.bj * t.zp + 15) & ~15;
    t.items = nx * t.njb * t.nzb;
    t.cs = chunk_stride((t.rows + 2) * 16);
    t.ds = chunk_stride(t.rows * 16);
    // the last M block's rows beyond 3 cin lie past the last chunk of x
    t.doff = (kGuard + t.mb * (kTileM / 8) * t.cs + 127) & ~127;
    const int used = t.doff + (t.nt / 8) * t.ds + 128;
    if (used > 100 * 1024 && target > 32) continue;
    if (used > kMaxSmem) return false;
    t.smem = smem_for(used, t.cols);
    // large boxes only while every SM still gets work
    if (t.items * 3 * (3 / t.ndk) * t.nmb * (cout / t.nt) >= 2 * 148 || target == 64 || target == 32) return true;
  }
  return true;
}

}  // namespace conv
}  // namespace efsi
