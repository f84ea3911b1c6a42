// hmp_stabilize.cu -- frame stabiliser (hmp_stabilizer_* in include/hmpano.h).
//
// The reference ships it as a demo beside the stitcher (src/cuda/cudaStabilize.cu): Harris corners
// of the previous frame, sparse Lucas-Kanade flow of each into the next frame, the mean flow as the
// global motion, and the next frame translated by it. There every step round-trips through the
// host (the response map is copied out for thresholding, the features copied in, the flow copied
// out and averaged on the CPU) with a synchronize after each kernel and allocations per call. Here
// a stabiliser allocates once and every step stays on the device, asynchronous on the caller's
// stream:
//   harris      Sobel gradients and the 3x3 Harris response, four columns a thread, the gradient
//               products of three rows in registers;
//   corners     threshold + 3x3 non-maximum suppression as one bit a pixel with the rows' counts, one
//               CTA scans the counts, and a warp per row writes its corners at its offset, so the
//               list is in raster order as the reference's host loop builds it;
//   flow        Lucas-Kanade per feature, one thread each, the reference's sums in its order, by tiles
//               of the frame held in shared memory;
//   motion      the flow summed in feature order (the reference's host sum) by scans, and rounded;
//   warp        translation by the rounded mean, zero fill.
// Operation order follows the reference (this file is compiled with -fmad=false); where the
// reference reads memory it never defines, the values are fixed as the oracle documents
// (oracle/hmp_stabilize_oracle.c): gradients and responses outside the interior are 0, flow taps
// in column 0 or row 0 are skipped, and no corners means no motion.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstdint>
#include <cstdio>
#include <new>

#include "hmp_ordered_sum.h"
#include "hmpano.h"

namespace {

struct Motion {
  int corners;     // corners found (the list holds at most the stabiliser's capacity)
  float dx, dy;    // mean flow
  int sx, sy;      // its rounding, the translation applied
};

// A displacement rounded to whole pixels: the float-to-int conversion saturates and maps NaN to 0;
// the clamp at +-2^24 keeps the index sums in range (a shift that large leaves the frame either way).
__device__ __forceinline__ int shift_of(float v) {
  if (!(v == v)) return 0;
  return int(fminf(fmaxf(roundf(v), -16777216.0f), 16777216.0f));
}

// Harris response: a thread walks kHarrisRows rows of four columns. Per row it forms the gradients
// of its columns and the ones beside them (with the reference's sums, whose leading terms neighbours
// share) and their three products once each, and keeps the products of three rows in registers; a
// response is then 24 additions (the first row of each window sum is shared) and the determinant.
// Every column of the image is read through L1 by the threads around it, so nothing is staged and
// there is no barrier. Issue-bound at about 70 instructions a pixel. 3840x2160: 72 -> 31 us. The
// row counters of the corner pass are cleared on the way.
constexpr int kHarrisRows = 8, kHarrisCols = 4;

__global__ void __launch_bounds__(128) harris_kernel(const float* __restrict__ img, int w, int h, float k,
                                                     float* __restrict__ resp, int* __restrict__ row_cnt) {
  constexpr int C = kHarrisCols, N = C + 2;  // columns x .. x + 3 and one to each side
  const int x = (blockIdx.x * 32 + threadIdx.x) * C;
  const int y0 = (blockIdx.y * blockDim.y + threadIdx.y) * kHarrisRows;
  if (x >= w || y0 >= h) return;
  if (x == 0) {
    for (int y = y0; y < min(y0 + kHarrisRows, h); ++y) row_cnt[y] = 0;
  }
  bool col_in[N];  // gradients exist in the frame's interior
#pragma unroll
  for (int c = 0; c < N; ++c) col_in[c] = x - 1 + c > 0 && x - 1 + c < w - 1;
  float r[3][N + 2];  // three image rows, columns x - 2 .. x + 5
  const auto load = [&](float (&v)[N + 2], int y) {
    const bool in = y >= 0 && y < h;
    const float* row = img + (long long)y * w;
#pragma unroll
    for (int c = 0; c < N + 2; ++c) {
      const int xx = x - 2 + c;
      v[c] = in && xx >= 0 && xx < w ? __ldg(row + xx) : 0.f;
    }
  };
  float pxx[3][N], pxy[3][N], pyy[3][N];  // products of three gradient rows
  const auto products = [&](int s, const float (&a)[N + 2], const float (&m)[N + 2], const float (&b)[N + 2], int y) {
    const bool in = y > 0 && y < h - 1;
    float col[N + 2], row[N];
#pragma unroll
    for (int c = 0; c < N + 2; ++c) col[c] = a[c] + 2.0f * m[c] + b[c];
#pragma unroll
    for (int c = 0; c < N; ++c) row[c] = a[c] + 2.0f * a[c + 1] + a[c + 2];
#pragma unroll
    for (int c = 0; c < N; ++c) {
      float vx = col[c + 2] - a[c] - 2.0f * m[c] - b[c];
      float vy = row[c] - b[c] - 2.0f * b[c + 1] - b[c + 2];
      if (!(in && col_in[c])) vx = vy = 0.f;
      pxx[s][c] = vx * vx;
      pxy[s][c] = vx * vy;
      pyy[s][c] = vy * vy;
    }
  };
  load(r[0], y0 - 2);
  load(r[1], y0 - 1);
  load(r[2], y0);
  products(0, r[0], r[1], r[2], y0 - 1);
  load(r[0], y0 + 1);
  products(1, r[1], r[2], r[0], y0);
  // Row y0 + i: the image rows at hand are i + 2 and before, the product rows i + 1 and before.
#pragma unroll
  for (int i = 0; i < kHarrisRows; ++i) {
    const int y = y0 + i;
    if (y >= h) return;
    load(r[(i + 1) % 3], y + 2);
    products((i + 2) % 3, r[(i + 2) % 3], r[i % 3], r[(i + 1) % 3], y + 1);
    const int s0 = i % 3, s1 = (i + 1) % 3, s2 = (i + 2) % 3;
    float out[C];
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const auto sum = [&](const float (&p)[3][N]) {
        return 0.f + p[s0][c] + p[s0][c + 1] + p[s0][c + 2] + p[s1][c] + p[s1][c + 1] + p[s1][c + 2] + p[s2][c] +
               p[s2][c + 1] + p[s2][c + 2];
      };
      const float sxx = sum(pxx), sxy = sum(pxy), syy = sum(pyy);
      const float det = sxx * syy - sxy * sxy, tr = sxx + syy;
      out[c] = col_in[c + 1] && y > 0 && y < h - 1 ? det - k * tr * tr : 0.f;
    }
    float* o = resp + (long long)y * w + x;
    if (x + C <= w && (w & 3) == 0) {  // resp is 16-byte aligned
      *reinterpret_cast<float4*>(o) = make_float4(out[0], out[1], out[2], out[3]);
    } else {
#pragma unroll
      for (int c = 0; c < C; ++c)
        if (x + c < w) o[c] = out[c];
    }
  }
}

// Corners: threshold and 3x3 non-maximum suppression (a neighbour strictly above removes the pixel)
// of the response, four columns a thread over kCornerRows rows, as one bit a pixel in 32-bit words
// per row, and the rows' counts. The emit pass then reads the bits, not the response again.
// 3840x2160, count and emit: 94 -> 23 us.
constexpr int kCornerRows = 8;

__host__ __device__ inline int corner_words(int w) { return (w + 127) / 128 * 4; }  // per row

__global__ void __launch_bounds__(128) corner_bits_kernel(const float* __restrict__ resp, int w, int h, float thr,
                                                          uint32_t* __restrict__ bits, int* __restrict__ row_cnt) {
  const int lane = threadIdx.x, x = (blockIdx.x * 32 + lane) * 4;
  const int y0 = (blockIdx.y * blockDim.y + threadIdx.y) * kCornerRows;
  if (y0 >= h) return;
  float v[3][6];   // columns x - 1 .. x + 4
  float m3[3][4];  // the largest of three in a row
  const auto load = [&](int s, int y) {
    const bool in = y >= 0 && y < h;
    const float* row = resp + (long long)y * w;
#pragma unroll
    for (int c = 0; c < 6; ++c) {
      const int xx = x - 1 + c;
      v[s][c] = in && xx >= 0 && xx < w ? __ldg(row + xx) : 0.f;
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) m3[s][c] = fmaxf(fmaxf(v[s][c], v[s][c + 1]), v[s][c + 2]);
  };
  load(0, y0 - 1);
  load(1, y0);
#pragma unroll
  for (int i = 0; i < kCornerRows; ++i) {
    const int y = y0 + i;
    if (y >= h) return;
    load((i + 2) % 3, y + 1);
    unsigned b = 0;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      // fmaxf drops NaN neighbours, as the comparison with one does; the pixel itself never beats itself.
      const float r = v[(i + 1) % 3][c + 1];
      const float m = fmaxf(fmaxf(m3[i % 3][c], m3[(i + 1) % 3][c]), m3[(i + 2) % 3][c]);
      if (x + c >= 1 && x + c < w - 1 && y >= 1 && y < h - 1 && r > thr && !(m > r)) b |= 1u << c;
    }
    b <<= 4 * (lane & 7);
    const int n = __reduce_add_sync(0xFFFFFFFFu, __popc(b));
    b |= __shfl_xor_sync(0xFFFFFFFFu, b, 1);
    b |= __shfl_xor_sync(0xFFFFFFFFu, b, 2);
    b |= __shfl_xor_sync(0xFFFFFFFFu, b, 4);
    if ((lane & 7) == 0) bits[(long long)y * corner_words(w) + blockIdx.x * 4 + (lane >> 3)] = b;
    if (lane == 0 && n) atomicAdd(row_cnt + y, n);
  }
}

constexpr int kScanPerThread = 8;  // counts per thread in each pass of the scan

// One CTA: offsets (exclusive scan of the counts, kScanPerThread consecutive counts per
// thread, 1024 threads a pass) and the total (m; nullptr: not wanted).
__global__ void __launch_bounds__(1024) corner_scan_kernel(const int* seg_count, int segs, int* seg_off, Motion* m) {
  __shared__ int warp_sum[32];
  __shared__ int carry;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int base = 0; base < segs; base += 1024 * kScanPerThread) {
    const int i0 = base + threadIdx.x * kScanPerThread;
    int v[kScanPerThread];
    int t = 0;
#pragma unroll
    for (int e = 0; e < kScanPerThread; ++e) {
      v[e] = i0 + e < segs ? seg_count[i0 + e] : 0;
      t += v[e];
    }
    int s = t;  // inclusive scan of the threads' totals within the warp
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int u = __shfl_up_sync(0xFFFFFFFFu, s, d);
      if (lane >= d) s += u;
    }
    if (lane == 31) warp_sum[wid] = s;
    __syncthreads();
    if (wid == 0) {
      int ws = warp_sum[lane];
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int u = __shfl_up_sync(0xFFFFFFFFu, ws, d);
        if (lane >= d) ws += u;
      }
      warp_sum[lane] = ws;  // inclusive over warps
    }
    __syncthreads();
    int before = carry + (wid > 0 ? warp_sum[wid - 1] : 0) + s - t;
#pragma unroll
    for (int e = 0; e < kScanPerThread; ++e) {
      if (i0 + e < segs) seg_off[i0 + e] = before;
      before += v[e];
    }
    __syncthreads();
    if (threadIdx.x == 1023) carry = before;  // this pass's total added
    __syncthreads();
  }
  if (threadIdx.x == 0 && m != nullptr) m->corners = carry;
}

// A warp per row: its corners, in x order, at the row's offset (those within the capacity).
__global__ void __launch_bounds__(256) corner_emit_kernel(const uint32_t* __restrict__ bits, int w, int h,
                                                          const int* __restrict__ row_off, int2* xy, int cap) {
  const int lane = threadIdx.x & 31, y = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (y >= h) return;
  const int words = corner_words(w);
  int at = row_off[y];
  for (int w0 = 0; w0 < words; w0 += 32) {
    uint32_t b = w0 + lane < words ? __ldg(bits + (long long)y * words + w0 + lane) : 0u;
    const int n = __popc(b);
    int s = n;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int u = __shfl_up_sync(0xFFFFFFFFu, s, d);
      if (lane >= d) s += u;
    }
    for (int pos = at + s - n; b != 0u; b &= b - 1u, ++pos)
      if (pos < cap) xy[pos] = make_int2(32 * (w0 + lane) + __ffs(b) - 1, y);
    at += __shfl_sync(0xFFFFFFFFu, s, 31);
  }
}

// ---- Lucas-Kanade flow ----
//
// Per feature, 10 iterations over a window: the displacement so far rounded to whole pixels for
// sampling the next frame, five sums over the window's taps in raster order, and a step that the
// sums determine (the reference's scheme and sum order). The sums depend on the displacement only
// through its rounding, and 10 iterations visit about four roundings (a sub-pixel shift alternates
// between its neighbours), so the steps of the roundings a feature has met are kept while its
// iterations run, and a window is summed once per rounding.

// The step the sums of a window determine; bad: the determinant is too small, iterations end.
struct FlowStep {
  float x, y;
  bool bad;
};

__device__ __forceinline__ FlowStep flow_step(float sxx, float syy, float sxy, float stx, float sty) {
  FlowStep r;
  const float det = sxx * syy - sxy * sxy;
  r.bad = fabsf(det) < 1e-6f;
  r.x = (-syy * stx + sxy * sty) / det;
  r.y = (sxy * stx - sxx * sty) / det;
  return r;
}

// One feature's iterations: the displacement and how many were made (10 or more: done).
struct FlowState {
  float dx = 0.f, dy = 0.f;
  float ex = 0.f, ey = 0.f;  // the match the last step pointed at: its rounding plus the step
  int iter = 0;
  __device__ __forceinline__ void apply(const FlowStep& s, int rx, int ry) {
    if (s.bad) {
      iter = 10;
      return;
    }
    ex = float(rx) + s.x;
    ey = float(ry) + s.y;
    dx += s.x;
    dy += s.y;
    ++iter;
    if (sqrtf(s.x * s.x + s.y * s.y) < 0.01f) iter = 10;
  }
};

// Steps of a 2 x 2 block of roundings (x0..x0+1, y0..y0+1); `have`: the entries present.
struct FlowQuad {
  int x0 = 0, y0 = 0;
  unsigned have = 0, bad = 0;
  float x[4], y[4];
  __device__ __forceinline__ bool find(int rx, int ry, FlowStep& s) const {
    const int i = rx - x0, j = ry - y0;
    if ((i | j) & ~1) return false;
    const int q = i + 2 * j;
    if (!((have >> q) & 1u)) return false;
    s.x = j ? (i ? x[3] : x[2]) : (i ? x[1] : x[0]);
    s.y = j ? (i ? y[3] : y[2]) : (i ? y[1] : y[0]);
    s.bad = (bad >> q) & 1u;
    return true;
  }
  // The one rounding (rx, ry).
  __device__ __forceinline__ void set(int rx, int ry, const FlowStep& s) {
    x0 = rx;
    y0 = ry;
    have = 1u;
    bad = s.bad ? 1u : 0u;
    x[0] = s.x;
    y[0] = s.y;
  }
};

// The window's sums straight from the frames, taps outside them skipped.
__device__ __forceinline__ FlowStep window_global(const float* __restrict__ prev, const float* __restrict__ next, int2 p,
                                                  int rdx, int rdy, int half, int w, int h) {
  float sxx = 0.f, syy = 0.f, sxy = 0.f, stx = 0.f, sty = 0.f;
  for (int j = -half; j <= half; ++j)
    for (int i = -half; i <= half; ++i) {
      const int x = p.x + i, y = p.y + j, xn = x + rdx, yn = y + rdy;
      if (x < 1 || x >= w - 1 || y < 1 || y >= h - 1 || xn < 0 || xn >= w - 1 || yn < 0 || yn >= h - 1) continue;
      const long long o = (long long)y * w + x;
      const float ix = (__ldg(prev + o + 1) - __ldg(prev + o - 1)) * 0.5f;
      const float iy = (__ldg(prev + o + w) - __ldg(prev + o - w)) * 0.5f;
      const float it = __ldg(next + (long long)yn * w + xn) - __ldg(prev + o);
      sxx += ix * ix;
      syy += iy * iy;
      sxy += ix * iy;
      stx += ix * it;
      sty += iy * it;
    }
  return flow_step(sxx, syy, sxy, stx, sty);
}

// Any window: a thread per feature, every tap from the frames. The last four roundings' steps are
// kept. Windows of 3 too: nine taps cost less than listing the features by tile and staging the tiles
// (a call on 3840x2160, 231,000 features 430 -> 300 us; 4000 at 12 px on 1920x1080 112 -> 62).
__global__ void __launch_bounds__(256) flow_kernel(const float* __restrict__ prev, const float* __restrict__ next,
                                                   const int2* xy, const Motion* m, int cap, int w, int h, int half,
                                                   float2* flow) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= min(m->corners, cap)) return;
  const int2 p = xy[f];
  FlowState st;
  FlowQuad kept[4];
  while (st.iter < 10) {
    const int rx = shift_of(st.dx), ry = shift_of(st.dy);
    FlowStep s;
    bool found = false;
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (!found && kept[k].find(rx, ry, s)) found = true;
    if (!found) {
      s = window_global(prev, next, p, rx, ry, half, w, h);
#pragma unroll
      for (int k = 3; k > 0; --k) kept[k] = kept[k - 1];
      kept[0].set(rx, ry, s);
    }
    st.apply(s, rx, ry);
  }
  flow[f] = make_float2(st.dx, st.dy);
}

// Windows of 5 to 21 pixels: a CTA per 64 x 64 tile of the frame (and 128 features), one to a thread, the
// tile of `prev` (with the window's halo and the gradients') and of `next` (with the window's halo
// and flow_margin pixels of motion) in shared memory. Features of a warp sit at scattered places, so
// their taps are 4-byte accesses at unrelated addresses: from L1 each costs a wavefront per lane,
// from shared memory one per bank conflict. Both tiles have a pitch of 96 words (a multiple of 32),
// so a tap's bank depends on its column alone, and the tile's features are dealt out to the warps
// in the order of their columns' banks: the lanes of a warp then read nearly distinct banks.
//
// A feature's first window (no displacement) gives all five sums. The sums of the gradients are the
// same for every displacement of a window inside both frames, so each later pass over such a window
// sums only the two that hold the time difference, for the four roundings around the displacement
// at once (the gradients of a tap are formed once for the four). Windows across the frame's border
// are summed tap by tap with the taps outside skipped. When the features' mean displacement is past half
// the margin, `next` is staged again around it; windows beyond the margin take `prev` from its tile and
// `next` from the frame, by rows (window_far).
// The gradients are summed without their factor 1/2, which scales every product and partial sum by a
// power of two: exact, unless a sum nears either end of the FP32 range, and then the window is summed
// from the frames as written. Bound by the additions' issue (about 24 instructions a tap and pass).
// 231,000 features at 3840x2160, window 15, a thread per feature reading the frames every iteration:
// 1840 us whatever the motion; so: 175 to 385 us for motions up to 4 px, 900 at 6 px, 1290 at 12 px, 1200 at
// 30 px (1900 with the windows beyond the margin tap by tap from both frames), and 16 us to list the
// features by tile.
constexpr int kFlowTile = 64, kFlowPitch = 96, kFlowThreads = 128;
constexpr int kFlowMinHalf = 2, kFlowMaxHalf = 10, kFlowFewFar = 6;
// Pixels of motion staged around a tile of `next`, so that it is 96 x 96: 9 at window 15, 6 at 21.
__host__ __device__ constexpr int flow_margin(int half) { return (kFlowPitch - kFlowTile) / 2 - half; }
__host__ __device__ constexpr int flow_prev_rows(int half) { return kFlowTile + 2 * half + 2; }
__host__ __device__ constexpr int flow_smem(int half) {
  return (flow_prev_rows(half) + kFlowPitch) * kFlowPitch * int(sizeof(float));
}

__device__ __forceinline__ void copy_async4(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(uint32_t(__cvta_generic_to_shared(dst))), "l"(src));
}

// frame[oy ..][ox ..] into rows x cols of a tile, 0 outside the frame (never used: those taps are
// skipped).
__device__ __forceinline__ void stage_frame(float* t, const float* __restrict__ frame, int ox, int oy, int rows, int cols,
                                            int w, int h) {
  const int lane = threadIdx.x & 31;
  for (int r = threadIdx.x >> 5; r < rows; r += kFlowThreads / 32) {
    const int y = oy + r;
    const bool row_in = y >= 0 && y < h;
    const float* src = frame + (long long)y * w;
#pragma unroll
    for (int c = lane; c < kFlowPitch; c += 32) {
      const int x = ox + c;
      if (row_in && c < cols && x >= 0 && x < w)
        copy_async4(t + r * kFlowPitch + c, src + x);
      else
        t[r * kFlowPitch + c] = 0.f;
    }
  }
}

__device__ __forceinline__ void stage_wait() {
  asm volatile("cp.async.commit_group;\n" ::: "memory");
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();
}

// The five sums of a W x W window, of doubled gradients: a at the tap above and left of the window's first in `prev`'s
// tile, b at the first tap in `next`'s. kMask: only taps of set bits (columns cm, rows rm).
template <int W, bool kMask>
__device__ __forceinline__ void window_sums(const float* a, const float* b, unsigned cm, unsigned rm, float& sxx, float& syy,
                                            float& sxy, float& stx, float& sty) {
  float up[W + 2], mid[W + 2], dn[W + 2];
#pragma unroll
  for (int c = 0; c < W + 2; ++c) up[c] = a[c], mid[c] = a[kFlowPitch + c];
  sxx = syy = sxy = stx = sty = 0.f;
#pragma unroll 1
  for (int j = 0; j < W; ++j) {
    const float* d = a + (j + 2) * kFlowPitch;
    const float* n = b + j * kFlowPitch;
#pragma unroll
    for (int c = 0; c < W + 2; ++c) dn[c] = d[c];
    const unsigned row = kMask ? (((rm >> j) & 1u) ? cm : 0u) : 0u;
#pragma unroll
    for (int i = 0; i < W; ++i) {
      const float ix = mid[i + 2] - mid[i];
      const float iy = dn[i + 1] - up[i + 1];
      const float it = n[i] - mid[i + 1];
      if (!kMask || ((row >> i) & 1u)) {
        sxx += ix * ix;
        syy += iy * iy;
        sxy += ix * iy;
        stx += ix * it;
        sty += iy * it;
      }
    }
#pragma unroll
    for (int c = 0; c < W + 2; ++c) up[c] = mid[c], mid[c] = dn[c];
  }
}

// The two time sums of a window, of doubled gradients, for the displacements b, b + 1 column, b + 1 row and both.
template <int W>
__device__ __forceinline__ void window_time_sums(const float* a, const float* b, float (&stx)[4], float (&sty)[4]) {
  float up[W + 2], mid[W + 2], dn[W + 2], n0[W + 1], n1[W + 1];
#pragma unroll
  for (int c = 0; c < W + 2; ++c) up[c] = a[c], mid[c] = a[kFlowPitch + c];
#pragma unroll
  for (int c = 0; c < W + 1; ++c) n0[c] = b[c];
#pragma unroll
  for (int q = 0; q < 4; ++q) stx[q] = sty[q] = 0.f;
#pragma unroll 3
  for (int j = 0; j < W; ++j) {
    const float* d = a + (j + 2) * kFlowPitch;
    const float* n = b + (j + 1) * kFlowPitch;
#pragma unroll
    for (int c = 0; c < W + 2; ++c) dn[c] = d[c];
#pragma unroll
    for (int c = 0; c < W + 1; ++c) n1[c] = n[c];
#pragma unroll
    for (int i = 0; i < W; ++i) {
      const float ix = mid[i + 2] - mid[i];
      const float iy = dn[i + 1] - up[i + 1];
      const float c = mid[i + 1];
      const float it[4] = {n0[i] - c, n0[i + 1] - c, n1[i] - c, n1[i + 1] - c};
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        stx[q] += ix * it[q];
        sty[q] += iy * it[q];
      }
    }
#pragma unroll
    for (int c = 0; c < W + 2; ++c) up[c] = mid[c], mid[c] = dn[c];
#pragma unroll
    for (int c = 0; c < W + 1; ++c) n0[c] = n1[c];
  }
}

// W values of a row of a frame from value L on, by aligned 16-byte loads (a warp's windows lie scattered:
// a load of four values costs the L1 what one of a single value does); inside: every chunk lies in the
// frame's `total` values, else value by value, 0 outside.
template <int W>
struct FarRow {
  static constexpr int NC = (W + 6) / 4;  // chunks: up to 3 values before the row's first
  static_assert(W + 3 <= 4 * NC, "whole rows");
  float4 c[NC];
  int off;
  __device__ __forceinline__ void load(const float* __restrict__ frame, long long total, long long L) {
    off = int(reinterpret_cast<uintptr_t>(frame + L) >> 2) & 3;
    const long long at = L - off;
    if (at >= 0 && at + 4 * NC <= total) {
#pragma unroll
      for (int k = 0; k < NC; ++k) c[k] = __ldg(reinterpret_cast<const float4*>(frame + at) + k);
    } else {
      const auto one = [&](long long i) { return i >= 0 && i < total ? __ldg(frame + i) : 0.f; };
#pragma unroll
      for (int k = 0; k < NC; ++k) {
        const long long i = at + 4 * k;
        c[k] = make_float4(one(i), one(i + 1), one(i + 2), one(i + 3));
      }
    }
  }
  __device__ __forceinline__ void values(float (&v)[W]) const {
    const auto at = [&](int i) {
      const float4 q = c[i >> 2];
      return (i & 3) == 0 ? q.x : (i & 3) == 1 ? q.y : (i & 3) == 2 ? q.z : q.w;
    };
#pragma unroll
    for (int i = 0; i < W; ++i) {
      const float lo = off & 1 ? at(i + 1) : at(i), hi = off & 1 ? at(i + 3) : at(i + 2);
      v[i] = off & 2 ? hi : lo;
    }
  }
};

// The sums of a window whose displacement the staged part of `next` does not cover: `prev` from its tile
// (a as above), `next` from the frame, its window's first tap at (x0, y0), a row ahead of the sums. Without
// kMask, of a window inside both frames: the time sums only; with it all five, over the taps of set bits.
template <int W, bool kMask>
__device__ __forceinline__ void window_far(const float* a, const float* __restrict__ next, int x0, int y0, int w, int h,
                                           unsigned cm, unsigned rm, float& sxx, float& syy, float& sxy, float& stx,
                                           float& sty) {
  constexpr bool kAhead = W <= 15;  // larger windows have no registers for two rows of `next`
  const long long total = (long long)w * h;
  float up[W + 2], mid[W + 2], dn[W + 2], n[W];
  FarRow<W> ahead;
  const auto request = [&](int j) {
    if (!kMask || ((rm >> j) & 1u)) ahead.load(next, total, (long long)(y0 + j) * w + x0);
  };
  if (kAhead) request(0);
#pragma unroll
  for (int c = 0; c < W + 2; ++c) up[c] = a[c], mid[c] = a[kFlowPitch + c];
  if (kMask) sxx = syy = sxy = 0.f;
  stx = sty = 0.f;
#pragma unroll 1
  for (int j = 0; j < W; ++j) {
    const float* d = a + (j + 2) * kFlowPitch;
#pragma unroll
    for (int c = 0; c < W + 2; ++c) dn[c] = d[c];
    const unsigned row = kMask ? (((rm >> j) & 1u) ? cm : 0u) : 0u;
    if (!kAhead) request(j);
    ahead.values(n);
    if (kAhead && j + 1 < W) request(j + 1);
#pragma unroll
    for (int i = 0; i < W; ++i) {
      const float ix = mid[i + 2] - mid[i];
      const float iy = dn[i + 1] - up[i + 1];
      const float it = n[i] - mid[i + 1];
      if (!kMask || ((row >> i) & 1u)) {
        if (kMask) {
          sxx += ix * ix;
          syy += iy * iy;
          sxy += ix * iy;
        }
        stx += ix * it;
        sty += iy * it;
      }
    }
#pragma unroll
    for (int c = 0; c < W + 2; ++c) up[c] = mid[c], mid[c] = dn[c];
  }
}

// The step of sums of doubled gradients. in_range: the sums proper have the same bits. Doubling scales
// every product and partial sum exactly except past the ends of the FP32 range: sums that may have
// overflowed doubled are refused, and so are tiny ones, whose products may be subnormal. (Subnormal
// products inside a larger sum lie 2^-18 of its last place below it: they can only tip a tie.)
__device__ __forceinline__ FlowStep flow_step_doubled(float sxx, float syy, float sxy, float stx, float sty,
                                                      bool& in_range) {
  const auto tiny = [](float v) { return v != 0.f && fabsf(v) < 1e-30f; };
  in_range = fmaxf(fmaxf(sxx, syy), fmaxf(fabsf(stx), fabsf(sty))) < 1e37f && stx == stx && sty == sty &&
             !(tiny(sxx) || tiny(syy) || tiny(sxy) || tiny(stx) || tiny(sty));
  return flow_step(sxx * 0.25f, syy * 0.25f, sxy * 0.25f, stx * 0.5f, sty * 0.5f);
}

// Bits [lo, hi) of a W-bit mask.
__device__ __forceinline__ unsigned range_mask(int lo, int hi, int W) {
  lo = max(lo, 0);
  hi = min(hi, W);
  return hi > lo ? ((1u << hi) - 1u) & ~((1u << lo) - 1u) : 0u;
}

// The plain window where the tiled kernel seldom needs it, out of its way.
__device__ __noinline__ FlowStep window_global_call(const float* __restrict__ prev, const float* __restrict__ next, int2 p,
                                                    int rdx, int rdy, int half, int w, int h) {
  return window_global(prev, next, p, rdx, rdy, half, w, h);
}

// What the tiled flow's kernels share besides the features: per tile the count of its features and where
// they end in `order`; the work items, a tile and which kFlowThreads of its features, so that a crowded tile
// is shared by many CTAs (20,000 features in one: 2100 us for a call as rounds of one CTA, 127 so).
struct FlowItems {
  int* cnt;
  int* at;
  int* order;
  int2* items;
  int* n_items;  // [0] the number, [1] how many were taken besides the CTAs' first ones
};

template <int HALF>
__global__ void __launch_bounds__(kFlowThreads, 3)
    flow_tile_kernel(const float* __restrict__ prev, const float* __restrict__ next, const int2* __restrict__ xy,
                     const __grid_constant__ FlowItems q, int tiles_x, int w, int h, float2* flow) {
  constexpr int W = 2 * HALF + 1, M = flow_margin(HALF), P = kFlowPitch;
  extern __shared__ float tiles[];
  float* sp = tiles;                             // prev, origin (X0 - HALF - 1, Y0 - HALF - 1)
  float* sn = tiles + flow_prev_rows(HALF) * P;  // next, origin (X0 - HALF + cx - M, Y0 - HALF + cy - M)
  __shared__ int bank_cnt[32], slot[kFlowThreads], mean_sum[3], taken;
  const int tid = threadIdx.x, lane = tid & 31;
  if (int(blockIdx.x) >= q.n_items[0]) return;
  for (bool first_item = true;; first_item = false) {  // item blockIdx.x, then the next that no CTA has
    __syncthreads();  // the last item is done with shared memory
    if (tid == 0) taken = first_item ? int(blockIdx.x) : int(gridDim.x) + atomicAdd(q.n_items + 1, 1);
    if (tid < 32) bank_cnt[tid] = 0;
    if (tid < 3) mean_sum[tid] = 0;
    slot[tid] = -1;
    __syncthreads();
    if (taken >= q.n_items[0]) return;
    const int2 item = q.items[taken];
    const int total = q.cnt[item.x], rounds = (total + kFlowThreads - 1) / kFlowThreads;
    const int per = (total + rounds - 1) / rounds, r0 = item.y * per, nc = min(per, total - r0);
    const int first = q.at[item.x] - total + r0;
    const int X0 = item.x % tiles_x * kFlowTile, Y0 = item.x / tiles_x * kFlowTile;
    int cx = 0, cy = 0;  // the displacement `next` is staged around
    stage_frame(sp, prev, X0 - HALF - 1, Y0 - HALF - 1, flow_prev_rows(HALF), flow_prev_rows(HALF), w, h);
    stage_frame(sn, next, X0 - HALF - M, Y0 - HALF - M, P, P, w, h);
    // Deal the features out by bank.
    int mine = -1, bank = 0, rank = 0;
    if (tid < nc) {
      mine = q.order[first + tid];
      bank = xy[mine].x & 31;
      rank = atomicAdd(&bank_cnt[bank], 1);
    }
    __syncthreads();
    if (tid < 32) {
      const int c = bank_cnt[lane];
      int s = c;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int u = __shfl_up_sync(0xFFFFFFFFu, s, d);
        if (lane >= d) s += u;
      }
      bank_cnt[lane] = s - c;
    }
    __syncthreads();
    if (mine >= 0) {
      const int warps = (nc + 31) >> 5, pos = bank_cnt[bank] + rank;
      slot[(pos % warps) * 32 + pos / warps] = mine;
    }
    stage_wait();  // the tiles and the slots
    const bool has = slot[tid] >= 0;
    const int2 p = has ? xy[slot[tid]] : make_int2(X0, Y0);
    const int own = (p.y - Y0) * P + p.x - X0;  // the feature's place in the tile
    const float* a = sp + own;
    const bool inside = p.x - HALF >= 1 && p.x + HALF < w - 1 && p.y - HALF >= 1 && p.y + HALF < h - 1;
    // Bits of the window's taps that lie inside both frames under displacement (rx, ry).
    const auto masks = [&](int rx, int ry, unsigned& cm, unsigned& rm) {
      cm = range_mask(max(1, -rx) - (p.x - HALF), min(w - 1, w - 1 - rx) - (p.x - HALF), W);
      rm = range_mask(max(1, -ry) - (p.y - HALF), min(h - 1, h - 1 - ry) - (p.y - HALF), W);
    };
    FlowState st;
    FlowStep zero{0.f, 0.f, true};
    FlowQuad qa, qb;
    float sxx = 0.f, syy = 0.f, sxy = 0.f;
    if (!has) st.iter = 10;
    if (has) {
      float stx, sty;
      const float* b = sn + own + M * P + M;
      if (__all_sync(__activemask(), inside)) {
        window_sums<W, false>(a, b, 0u, 0u, sxx, syy, sxy, stx, sty);
      } else {
        unsigned cm, rm;
        masks(0, 0, cm, rm);
        window_sums<W, true>(a, b, cm, rm, sxx, syy, sxy, stx, sty);
      }
      bool in_range;
      zero = flow_step_doubled(sxx, syy, sxy, stx, sty, in_range);
      if (!in_range) zero = window_global_call(prev, next, p, 0, 0, HALF, w, h);
    }
    bool recentred = false;
    while (true) {
      // As far as the steps at hand go.
      int rx = 0, ry = 0;
      while (st.iter < 10) {
        rx = shift_of(st.dx);
        ry = shift_of(st.dy);
        FlowStep s = zero;
        if (!(rx == 0 && ry == 0) && !qa.find(rx, ry, s) && !qb.find(rx, ry, s)) break;
        st.apply(s, rx, ry);
      }
      const bool need = st.iter < 10;
      if (!recentred) {
        // The mean displacement wanted: staged again around it when it is past half the margin.
        recentred = true;
        const int vx = need ? min(max(rx, -1024), 1024) : 0, vy = need ? min(max(ry, -1024), 1024) : 0;
        const int sx = __reduce_add_sync(0xFFFFFFFFu, vx), sy = __reduce_add_sync(0xFFFFFFFFu, vy);
        const int sc = __reduce_add_sync(0xFFFFFFFFu, need ? 1 : 0);
        if (lane == 0 && sc > 0) {
          atomicAdd(&mean_sum[0], sx);
          atomicAdd(&mean_sum[1], sy);
          atomicAdd(&mean_sum[2], sc);
        }
        __syncthreads();
        const int c = max(mean_sum[2], 1), mx = mean_sum[0] / c, my = mean_sum[1] / c;
        if (max(abs(mx), abs(my)) > M / 2) {
          cx = mx;
          cy = my;
          stage_frame(sn, next, X0 - HALF + cx - M, Y0 - HALF + cy - M, P, P, w, h);
          stage_wait();
        }
      }
      if (!__any_sync(0xFFFFFFFFu, need)) break;
      // A warp's windows beyond the staged part wait for those inside it, where they are more than a few: then
      // they are summed together, not beside one of the others pass after pass (3840x2160, 12 px: 1640 -> 1540 us
      // a call). A few outliers are not worth the others' wait: 3 to 4 % of the flow at window 21 and 3 px.
      const bool near1 = abs(rx - cx) <= M && abs(ry - cy) <= M;
      const unsigned far_lanes = __ballot_sync(0xFFFFFFFFu, need && !near1);
      const bool defer = __any_sync(0xFFFFFFFFu, need && near1) && __popc(far_lanes) > kFlowFewFar;
      if (!need || (defer && !near1)) continue;
      // The rounding and its neighbours toward the match the last step pointed at: iterations near a
      // match add the same step until the rounding crosses to that side.
      const int bx = st.ex < float(rx) ? rx - 1 : rx, by = st.ey < float(ry) ? ry - 1 : ry;
      const bool near4 = near1 && bx - cx >= -M && bx + 1 - cx <= M && by - cy >= -M && by + 1 - cy <= M;
      qb = qa;
      if (inside && near4 && p.x - HALF + bx >= 0 && p.x + HALF + bx + 1 < w - 1 && p.y - HALF + by >= 0 &&
          p.y + HALF + by + 1 < h - 1) {
        float stx[4], sty[4];
        window_time_sums<W>(a, sn + own + (by - cy + M) * P + bx - cx + M, stx, sty);
        qa.x0 = bx;
        qa.y0 = by;
        qa.have = 15u;
        qa.bad = 0u;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          bool in_range;
          FlowStep s = flow_step_doubled(sxx, syy, sxy, stx[q], sty[q], in_range);
          if (!in_range) s = window_global_call(prev, next, p, bx + (q & 1), by + (q >> 1), HALF, w, h);
          qa.x[q] = s.x;
          qa.y[q] = s.y;
          if (s.bad) qa.bad |= 1u << q;
        }
      } else if (near1) {
        unsigned cm, rm;
        masks(rx, ry, cm, rm);
        float a0, a1, a2, stx, sty;
        window_sums<W, true>(a, sn + own + (ry - cy + M) * P + rx - cx + M, cm, rm, a0, a1, a2, stx, sty);
        bool in_range;
        FlowStep s = flow_step_doubled(a0, a1, a2, stx, sty, in_range);
        if (!in_range) s = window_global_call(prev, next, p, rx, ry, HALF, w, h);
        qa.set(rx, ry, s);
      } else {
        const int x0 = p.x - HALF + rx, y0 = p.y - HALF + ry;
        float a0 = sxx, a1 = syy, a2 = sxy, stx, sty;
        if (inside && x0 >= 0 && x0 + W < w && y0 >= 0 && y0 + W < h) {
          window_far<W, false>(a, next, x0, y0, w, h, 0u, 0u, a0, a1, a2, stx, sty);
        } else {
          unsigned cm, rm;
          masks(rx, ry, cm, rm);
          window_far<W, true>(a, next, x0, y0, w, h, cm, cm != 0u ? rm : 0u, a0, a1, a2, stx, sty);
        }
        bool in_range;
        FlowStep s = flow_step_doubled(a0, a1, a2, stx, sty, in_range);
        if (!in_range) s = window_global_call(prev, next, p, rx, ry, HALF, w, h);
        qa.set(rx, ry, s);
      }
    }
    if (has) flow[slot[tid]] = make_float2(st.dx, st.dy);
  }
}

// Grids of the per-feature passes: the feature count is known on the device only and the capacity
// may be every pixel, so a few CTAs per SM walk the features.
constexpr unsigned kFeatureBlocks = 152 * 4;
constexpr unsigned kFlowBlocks = 152 * 3;  // flow_tile_kernel's, as many as are resident

// Features by tile: their counts and the work items (each kFlowThreads-th feature of a tile opens one),
// then (after corner_scan_kernel's offsets) their indices, tile by tile. The order inside a tile is left to
// the atomics; a feature's flow does not depend on it.
__global__ void __launch_bounds__(256) tile_count_kernel(const int2* xy, const Motion* m, int cap, int tiles_x,
                                                         const __grid_constant__ FlowItems q) {
  const int n = min(m->corners, cap);
  for (int f = blockIdx.x * blockDim.x + threadIdx.x; f < n; f += gridDim.x * blockDim.x) {
    const int2 p = xy[f];
    const int tile = (p.y / kFlowTile) * tiles_x + p.x / kFlowTile, i = atomicAdd(q.cnt + tile, 1);
    if (i % kFlowThreads == 0) q.items[atomicAdd(q.n_items, 1)] = make_int2(tile, i / kFlowThreads);
  }
}

__global__ void __launch_bounds__(256) tile_fill_kernel(const int2* xy, const Motion* m, int cap, int tiles_x,
                                                        const __grid_constant__ FlowItems q) {
  const int n = min(m->corners, cap);
  for (int f = blockIdx.x * blockDim.x + threadIdx.x; f < n; f += gridDim.x * blockDim.x) {
    const int2 p = xy[f];
    q.order[atomicAdd(&q.at[(p.y / kFlowTile) * tiles_x + p.x / kFlowTile], 1)] = f;
  }
}

// The global motion: the flow summed in feature order (as the reference's host loop), its mean and
// the rounded translation; a CTA per component. The sum's bits are those of one dependent chain of
// additions, found by scans of whole units (hmp_ordered_sum.h): a chunk of kMotionChunk features is
// staged in shared memory and scanned at once, up to the first partial sum that leaves the binade;
// from there `run` elements are added one by one by the thread that found it, and the scan resumes.
// A scan costs about as much as 1500 plain additions (3.4 us against 2.2 ns each), so `run` starts at a
// third of that, doubles while scans end within kMotionFar elements of where they began (sums hovering at
// a power of two or at zero), and falls back when one gets far; up to kMotionSmall features are summed
// plainly. 11 elements a thread: an odd stride keeps the blocked shared-memory reads free of bank conflicts.
// Bound by the scans. One dependent chain against this, 231,000 features at 3840x2160: a moving pair 746
// and 108 us, a still one, whose sums hover, 839 and about 800; 20,000 unsteady flows 67 and about 70.
constexpr int kMotionThreads = 1024, kMotionPer = 11, kMotionChunk = kMotionThreads * kMotionPer;
constexpr int kMotionRunMin = 512, kMotionRunMax = 8192, kMotionFar = 256, kMotionSmall = 4096;

// Inclusive scan of a warp's runs. Runs without ties (both increments alike in every lane, the usual
// case) are plain sums: a shuffle and an addition a step instead of two shuffles and a composition
// (motion_kernel 124 -> 116 us at 231,496 features).
__device__ __forceinline__ hmp::OrderedRun motion_scan(hmp::OrderedRun r, int lane) {
  if (__all_sync(0xFFFFFFFFu, r.d0 == r.d1)) {
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int u = __shfl_up_sync(0xFFFFFFFFu, r.d0, d);
      if (lane >= d) r.d0 = int(unsigned(u) + unsigned(r.d0));
    }
    r.d1 = r.d0;
    return r;
  }
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    hmp::OrderedRun u;
    u.d0 = __shfl_up_sync(0xFFFFFFFFu, r.d0, d);
    u.d1 = __shfl_up_sync(0xFFFFFFFFu, r.d1, d);
    if (lane >= d) r = hmp::ordered_then(u, r);
  }
  return r;
}

__global__ void __launch_bounds__(kMotionThreads) motion_kernel(const float2* __restrict__ flow, int cap, Motion* m) {
  __shared__ float xs[kMotionChunk];
  __shared__ hmp::OrderedRun warp_run[kMotionThreads / 32];
  __shared__ int first_fail;
  __shared__ float sum_after;
  const int comp = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n = min(m->corners, cap);
  const float* f = reinterpret_cast<const float*>(flow) + comp;
  float next[kMotionPer];
  const auto fetch = [&](int base) {
#pragma unroll
    for (int k = 0; k < kMotionPer; ++k) {
      const int i = base + k * kMotionThreads + tid;
      next[k] = i < n ? __ldg(f + 2LL * i) : 0.f;
    }
  };
  float s = 0.f;  // the same in every thread
  int run = n <= kMotionSmall ? kMotionSmall : kMotionRunMin, last = 0;  // last: the element the present scan began at
  fetch(0);
  for (int base = 0; base < n; base += kMotionChunk) {
    const int cnt = min(kMotionChunk, n - base);
    __syncthreads();  // the previous chunk is done with xs
#pragma unroll
    for (int k = 0; k < kMotionPer; ++k) xs[k * kMotionThreads + tid] = next[k];
    if (base + kMotionChunk < n) fetch(base + kMotionChunk);
    int pos = 0;
    while (pos < cnt) {
      if (tid == 0) first_fail = cnt;
      __syncthreads();  // xs, first_fail; the last pass is done with warp_run and sum_after
      float scale = 0.f, unit = 0.f;
      const bool scan = hmp::ordered_scale(s, scale, unit);
      float before = s;  // the sum before this thread's first failing element
      int fail = cnt;
      float total = s;  // the sum if nothing fails
      if (scan) {
        const int S = int(s * scale);
        // This thread's elements from `lead` on (the ones past the chunk's end are zeros): without
        // ties their partial sums are whole units from the start, so the extremes tell whether all
        // stay inside the binade; with ties (or elements too large) the pairs are composed.
        const int lead = pos - tid * kMotionPer;
        // (No branch per element: the ones before `lead` count as zeros, and whether any is a tie or
        // too large is one flag for the thread.)
        int sum = 0, lo = 0, hi = 0;
        bool plain = true;
#pragma unroll
        for (int k = 0; k < kMotionPer; ++k) {
          const float r = k >= lead ? xs[tid * kMotionPer + k] * scale : 0.f;
          hmp::OrderedRun e;
          plain = hmp::ordered_plain(r, e.d0) && plain;
          sum = int(unsigned(sum) + unsigned(e.d0));
          lo = min(lo, sum);
          hi = max(hi, sum);
        }
        hmp::OrderedRun mine{sum, sum};
        if (!plain) {
          mine.d0 = mine.d1 = 0;
          for (int k = max(lead, 0); k < kMotionPer; ++k) {
            hmp::OrderedRun e;
            if (hmp::ordered_element(xs[tid * kMotionPer + k] * scale, e)) mine = hmp::ordered_then(mine, e);
          }
        }
        const hmp::OrderedRun incl = motion_scan(mine, lane);
        if (lane == 31) warp_run[warp] = incl;
        hmp::OrderedRun excl;
        excl.d0 = __shfl_up_sync(0xFFFFFFFFu, incl.d0, 1);
        excl.d1 = __shfl_up_sync(0xFFFFFFFFu, incl.d1, 1);
        if (lane == 0) excl.d0 = excl.d1 = 0;
        __syncthreads();
        const hmp::OrderedRun w = motion_scan(warp_run[lane], lane);
        hmp::OrderedRun all, wbefore;
        all.d0 = __shfl_sync(0xFFFFFFFFu, w.d0, 31);
        all.d1 = __shfl_sync(0xFFFFFFFFu, w.d1, 31);
        wbefore.d0 = __shfl_sync(0xFFFFFFFFu, w.d0, warp > 0 ? warp - 1 : 0);
        wbefore.d1 = __shfl_sync(0xFFFFFFFFu, w.d1, warp > 0 ? warp - 1 : 0);
        total = float(hmp::ordered_apply(all, S)) * unit;
        int P = warp > 0 ? hmp::ordered_apply(wbefore, S) : S;
        P = hmp::ordered_apply(excl, P);
        const int plo = int(unsigned(P) + unsigned(lo)), phi = int(unsigned(P) + unsigned(hi));
        if (lead < kMotionPer &&
            !(plain && hmp::ordered_inside(plo) && hmp::ordered_inside(phi) && (plo ^ phi) >= 0)) {
          // Partial sums one by one, up to the first outside the binade.
          for (int k = max(lead, 0); k < kMotionPer && fail == cnt; ++k) {
            hmp::OrderedRun e{0, 0};
            const bool can = hmp::ordered_element(xs[tid * kMotionPer + k] * scale, e);
            const int q = hmp::ordered_apply(e, P);
            if (!can || !hmp::ordered_inside(q)) {
              fail = tid * kMotionPer + k;
              before = float(P) * unit;
            } else {
              P = q;
            }
          }
        }
      } else {
        // Zero, or too small or not finite to scan: a zero sum stays zero over zeros.
#pragma unroll
        for (int k = 0; k < kMotionPer; ++k) {
          const int i = tid * kMotionPer + k;
          if (i >= pos && i < cnt && fail == cnt && !(s == 0.f && xs[i] == 0.f)) fail = i;
        }
      }
      const int wf = __reduce_min_sync(0xFFFFFFFFu, fail);
      if (lane == 0 && wf < cnt) atomicMin(&first_fail, wf);
      __syncthreads();
      const int at = first_fail;
      if (at >= cnt) {
        s = total;
        break;
      }
      const int end = min(at + run, cnt);
      if (fail == at) {  // its thread adds the run as it stands
        float v = before, c[16];
        int i = at;
        if (end - at >= 16) {
#pragma unroll
          for (int k = 0; k < 16; ++k) c[k] = xs[at + k];
          for (; i + 32 <= end; i += 16) {  // the next 16 elements' loads fly during these additions
            float d[16];
#pragma unroll
            for (int k = 0; k < 16; ++k) d[k] = xs[i + 16 + k];
#pragma unroll
            for (int k = 0; k < 16; ++k) v += c[k];
#pragma unroll
            for (int k = 0; k < 16; ++k) c[k] = d[k];
          }
#pragma unroll
          for (int k = 0; k < 16; ++k) v += c[k];
          i += 16;
        }
        for (; i < end; ++i) v += xs[i];
        sum_after = v;
      }
      __syncthreads();
      s = sum_after;
      run = base + at - last < kMotionFar ? min(2 * run, kMotionRunMax) : kMotionRunMin;
      last = base + end;
      pos = end;
    }
  }
  if (tid == 0) {
    const float mean = n > 0 ? s / float(n) : 0.f;
    if (comp == 0) {
      m->dx = mean;
      m->sx = shift_of(mean);
    } else {
      m->dy = mean;
      m->sy = shift_of(mean);
    }
  }
}

// Translation by the motion, zero fill, four pixels a thread (one 16-byte store where rows allow).
// 3840x2160: 27 -> 11 us.
__global__ void __launch_bounds__(256) warp_kernel(const float* __restrict__ in, float* __restrict__ out, int w, int h,
                                                   const Motion* m) {
  const int x = (blockIdx.x * 64 + threadIdx.x) * 4, y = blockIdx.y * 4 + threadIdx.y;
  if (x >= w || y >= h) return;
  const int u = x - m->sx, v = y - m->sy;
  const bool row_in = v >= 0 && v < h;
  const float* row = in + (long long)v * w;
  float q[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) q[c] = row_in && u + c >= 0 && u + c < w ? __ldg(row + u + c) : 0.f;
  float* o = out + (long long)y * w + x;
  if (x + 4 <= w && (reinterpret_cast<uintptr_t>(o) & 15u) == 0) {
    *reinterpret_cast<float4*>(o) = make_float4(q[0], q[1], q[2], q[3]);
  } else {
#pragma unroll
    for (int c = 0; c < 4; ++c)
      if (x + c < w) o[c] = q[c];
  }
}

__global__ void copy_kernel(const float* __restrict__ in, float* __restrict__ out, long long n) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = in[i];
}

hmp_status status_of(int code, const char* msg) {
  hmp_status s;
  s.code = code;
  std::snprintf(s.message, sizeof(s.message), "%s", msg);
  return s;
}

hmp_status cuda_failure(cudaError_t e, const char* what) {
  hmp_status s;
  s.code = int(e);
  std::snprintf(s.message, sizeof(s.message), "%s: %s", what, cudaGetErrorString(e));
  return s;
}

}  // namespace

struct hmp_stabilizer {
  int w = 0, h = 0, cap = 0, device = -1;
  float* resp = nullptr;
  uint32_t* corner_bits = nullptr;  // one bit a pixel, corner_words(w) words a row
  int* row_cnt = nullptr;           // corners per row, and where each row's start in the list
  int* row_off = nullptr;
  int2* xy = nullptr;
  float2* flow = nullptr;
  Motion* motion = nullptr;
  float* temp = nullptr;  // an in-place warp's output before the copy back
  int tiles_x = 0, tiles = 0;  // flow tiles of the frame
  FlowItems items{};           // one allocation: items, order, at, cnt and n_items (cleared together)
  ~hmp_stabilizer() {
    for (void* p : {static_cast<void*>(resp), static_cast<void*>(corner_bits), static_cast<void*>(row_cnt),
                    static_cast<void*>(row_off), static_cast<void*>(xy), static_cast<void*>(flow),
                    static_cast<void*>(motion), static_cast<void*>(temp), static_cast<void*>(items.items)})
      if (p) cudaFree(p);
  }
  int most_items() const { return tiles + cap / kFlowThreads; }
  hmp_status check(const void* a, const void* b) const {
    int dev = -1;
    cudaGetDevice(&dev);
    if (dev != device) return status_of(HMP_ERR_INVALID_VALUE, "stabilizer used on another device");
    if (!a || !b) return status_of(HMP_ERR_INVALID_DEVICE_POINTER, "frame is null");
    return status_of(HMP_OK, "");
  }
};

namespace {

// flow_tile_kernel by half window (nullptr: none).
template <int HALF>
void launch_flow_tile(const hmp_stabilizer& st, const float* prev, const float* next, cudaStream_t cs) {
  const unsigned grid = std::min(unsigned(st.most_items()), kFlowBlocks);
  flow_tile_kernel<HALF><<<grid, kFlowThreads, flow_smem(HALF), cs>>>(prev, next, st.xy, st.items, st.tiles_x, st.w,
                                                                      st.h, st.flow);
}

using FlowTileLaunch = void (*)(const hmp_stabilizer&, const float*, const float*, cudaStream_t);
constexpr FlowTileLaunch kFlowTileLaunch[kFlowMaxHalf + 1] = {
    nullptr,             nullptr,             launch_flow_tile<2>, launch_flow_tile<3>, launch_flow_tile<4>,
    launch_flow_tile<5>, launch_flow_tile<6>, launch_flow_tile<7>, launch_flow_tile<8>, launch_flow_tile<9>,
    launch_flow_tile<10>};

template <int HALF = kFlowMaxHalf>
cudaError_t flow_tile_init() {
  const cudaError_t e =
      cudaFuncSetAttribute(flow_tile_kernel<HALF>, cudaFuncAttributeMaxDynamicSharedMemorySize, flow_smem(HALF));
  if constexpr (HALF > kFlowMinHalf) {
    return e == cudaSuccess ? flow_tile_init<HALF - 1>() : e;
  } else {
    return e;
  }
}

}  // namespace

extern "C" {

HMP_API hmp_status hmp_stabilizer_create(int width, int height, int max_features, hmp_stabilizer** out) {
  if (!out) return status_of(HMP_ERR_INVALID_VALUE, "out is null");
  *out = nullptr;
  if (width < 3 || height < 3 || width > (1 << 15) || height > (1 << 15))
    return status_of(HMP_ERR_INVALID_VALUE, "frames must be 3..32768 pixels per side");
  const long long interior = (long long)(width - 2) * (height - 2);
  if (max_features < 0) return status_of(HMP_ERR_INVALID_VALUE, "max_features must be >= 0 (0: every interior pixel)");
  hmp_stabilizer* st = new (std::nothrow) hmp_stabilizer();
  if (!st) return status_of(HMP_ERR_MEMORY_ALLOCATION, "out of host memory");
  st->w = width;
  st->h = height;
  st->cap = int(max_features == 0 ? interior : std::min<long long>(max_features, interior));
  st->tiles_x = (width + kFlowTile - 1) / kFlowTile;
  st->tiles = st->tiles_x * ((height + kFlowTile - 1) / kFlowTile);
  cudaError_t e = cudaGetDevice(&st->device);
  const size_t px = size_t(width) * height;
  if (e == cudaSuccess) e = cudaMalloc(&st->resp, px * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&st->corner_bits, size_t(corner_words(width)) * height * sizeof(uint32_t));
  if (e == cudaSuccess) e = cudaMalloc(&st->row_cnt, size_t(height) * sizeof(int));
  if (e == cudaSuccess) e = cudaMalloc(&st->row_off, size_t(height) * sizeof(int));
  if (e == cudaSuccess) e = cudaMalloc(&st->xy, size_t(std::max(st->cap, 1)) * sizeof(int2));
  if (e == cudaSuccess) e = cudaMalloc(&st->flow, size_t(std::max(st->cap, 1)) * sizeof(float2));
  if (e == cudaSuccess) e = cudaMalloc(&st->motion, sizeof(Motion));
  if (e == cudaSuccess) e = cudaMalloc(&st->temp, px * sizeof(float));
  if (e == cudaSuccess)
    e = cudaMalloc(&st->items.items, size_t(st->most_items()) * sizeof(int2) +
                                         (size_t(std::max(st->cap, 1)) + 2 * size_t(st->tiles) + 2) * sizeof(int));
  if (e == cudaSuccess) {
    st->items.order = reinterpret_cast<int*>(st->items.items + st->most_items());
    st->items.at = st->items.order + std::max(st->cap, 1);
    st->items.cnt = st->items.at + st->tiles;
    st->items.n_items = st->items.cnt + st->tiles;
  }
  if (e == cudaSuccess) e = flow_tile_init();
  if (e == cudaSuccess) e = cudaMemset(st->motion, 0, sizeof(Motion));
  if (e != cudaSuccess) {
    delete st;
    return cuda_failure(e, "stabilizer allocation");
  }
  *out = st;
  return status_of(HMP_OK, "");
}

HMP_API void hmp_stabilizer_destroy(hmp_stabilizer* st) { delete st; }

HMP_API hmp_status hmp_stabilizer_corners(hmp_stabilizer* st, const float* img, float k, float threshold,
                                          void* stream) {
  if (!st) return status_of(HMP_ERR_INVALID_VALUE, "stabilizer is null");
  hmp_status s = st->check(img, img);
  if (s.code) return s;
  const cudaStream_t cs = static_cast<cudaStream_t>(stream);
  const dim3 block(32, 4);
  harris_kernel<<<dim3((st->w + 127) / 128, (st->h + 4 * kHarrisRows - 1) / (4 * kHarrisRows)), block, 0, cs>>>(
      img, st->w, st->h, k, st->resp, st->row_cnt);
  corner_bits_kernel<<<dim3((st->w + 127) / 128, (st->h + 4 * kCornerRows - 1) / (4 * kCornerRows)), block, 0, cs>>>(
      st->resp, st->w, st->h, threshold, st->corner_bits, st->row_cnt);
  corner_scan_kernel<<<1, 1024, 0, cs>>>(st->row_cnt, st->h, st->row_off, st->motion);
  corner_emit_kernel<<<(st->h + 7) / 8, 256, 0, cs>>>(st->corner_bits, st->w, st->h, st->row_off, st->xy, st->cap);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? status_of(HMP_OK, "") : cuda_failure(e, "corner launch");
}

HMP_API hmp_status hmp_stabilizer_flow(hmp_stabilizer* st, const float* prev, const float* next, int window_size,
                                       void* stream) {
  if (!st) return status_of(HMP_ERR_INVALID_VALUE, "stabilizer is null");
  hmp_status s = st->check(prev, next);
  if (s.code) return s;
  if (window_size < 1 || window_size > 255) return status_of(HMP_ERR_INVALID_VALUE, "window_size must be in 1..255");
  const cudaStream_t cs = static_cast<cudaStream_t>(stream);
  const unsigned blocks = unsigned((std::max(st->cap, 1) + 255) / 256);
  const int half = window_size / 2;
  if (half >= kFlowMinHalf && half <= kFlowMaxHalf) {
    cudaError_t e = cudaMemsetAsync(st->items.cnt, 0, size_t(st->tiles + 2) * sizeof(int), cs);
    if (e != cudaSuccess) return cuda_failure(e, "flow set-up");
    const unsigned strided = std::min(blocks, kFeatureBlocks);
    tile_count_kernel<<<strided, 256, 0, cs>>>(st->xy, st->motion, st->cap, st->tiles_x, st->items);
    corner_scan_kernel<<<1, 1024, 0, cs>>>(st->items.cnt, st->tiles, st->items.at, nullptr);
    tile_fill_kernel<<<strided, 256, 0, cs>>>(st->xy, st->motion, st->cap, st->tiles_x, st->items);
    kFlowTileLaunch[half](*st, prev, next, cs);
  } else {
    flow_kernel<<<blocks, 256, 0, cs>>>(prev, next, st->xy, st->motion, st->cap, st->w, st->h, half, st->flow);
  }
  motion_kernel<<<2, kMotionThreads, 0, cs>>>(st->flow, st->cap, st->motion);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? status_of(HMP_OK, "") : cuda_failure(e, "flow launch");
}

HMP_API hmp_status hmp_stabilizer_warp(hmp_stabilizer* st, const float* frame, float* out, void* stream) {
  if (!st) return status_of(HMP_ERR_INVALID_VALUE, "stabilizer is null");
  hmp_status s = st->check(frame, out);
  if (s.code) return s;
  const cudaStream_t cs = static_cast<cudaStream_t>(stream);
  const dim3 grid((st->w + 255) / 256, (st->h + 3) / 4), block(64, 4);
  const long long px = (long long)st->w * st->h;
  if (out == frame) {
    warp_kernel<<<grid, block, 0, cs>>>(frame, st->temp, st->w, st->h, st->motion);
    copy_kernel<<<unsigned((px + 255) / 256), 256, 0, cs>>>(st->temp, out, px);
  } else {
    warp_kernel<<<grid, block, 0, cs>>>(frame, out, st->w, st->h, st->motion);
  }
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? status_of(HMP_OK, "") : cuda_failure(e, "warp launch");
}

HMP_API hmp_status hmp_stabilizer_run(hmp_stabilizer* st, const float* prev, const float* next, float* out, float k,
                                      float threshold, int window_size, void* stream) {
  hmp_status s = hmp_stabilizer_corners(st, prev, k, threshold, stream);
  if (s.code == HMP_OK) s = hmp_stabilizer_flow(st, prev, next, window_size, stream);
  if (s.code == HMP_OK) s = hmp_stabilizer_warp(st, next, out, stream);
  return s;
}

HMP_API hmp_status hmp_stabilizer_get_features(hmp_stabilizer* st, int* xy, float* flow, int capacity,
                                               hmp_stabilize_info* info, void* stream) {
  if (!st || !info || capacity < 0 || (capacity > 0 && (!xy || !flow)))
    return status_of(HMP_ERR_INVALID_VALUE, "invalid argument");
  const cudaStream_t cs = static_cast<cudaStream_t>(stream);
  cudaError_t e = cudaStreamSynchronize(cs);
  Motion m{};
  if (e == cudaSuccess) e = cudaMemcpy(&m, st->motion, sizeof(m), cudaMemcpyDeviceToHost);
  const int n = std::min({m.corners, st->cap, capacity});
  if (e == cudaSuccess && n > 0) e = cudaMemcpy(xy, st->xy, size_t(n) * sizeof(int2), cudaMemcpyDeviceToHost);
  if (e == cudaSuccess && n > 0) e = cudaMemcpy(flow, st->flow, size_t(n) * sizeof(float2), cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) return cuda_failure(e, "feature copy");
  info->corners = m.corners;
  info->kept = std::min(m.corners, st->cap);
  info->dx = m.dx;
  info->dy = m.dy;
  info->shift_x = m.sx;
  info->shift_y = m.sy;
  return status_of(HMP_OK, "");
}

HMP_API hmp_status hmp_stabilizer_get_response(hmp_stabilizer* st, float* out, size_t capacity, void* stream) {
  if (!st || !out) return status_of(HMP_ERR_INVALID_VALUE, "invalid argument");
  const size_t px = size_t(st->w) * st->h;
  if (capacity < px) return status_of(HMP_ERR_INVALID_VALUE, "capacity below width * height");
  const cudaStream_t cs = static_cast<cudaStream_t>(stream);
  cudaError_t e = cudaStreamSynchronize(cs);
  if (e == cudaSuccess) e = cudaMemcpy(out, st->resp, px * sizeof(float), cudaMemcpyDeviceToHost);
  return e == cudaSuccess ? status_of(HMP_OK, "") : cuda_failure(e, "response copy");
}

HMP_API hmp_status hmp_stabilizer_set_features(hmp_stabilizer* st, const int* xy, int n, void* stream) {
  if (!st || n < 0 || (n > 0 && !xy)) return status_of(HMP_ERR_INVALID_VALUE, "invalid argument");
  if (n > st->cap) return status_of(HMP_ERR_INVALID_VALUE, "more features than the stabilizer holds");
  for (int i = 0; i < n; ++i)  // the window's index sums stay in range for points on the frame
    if (xy[2 * i] < 0 || xy[2 * i] >= st->w || xy[2 * i + 1] < 0 || xy[2 * i + 1] >= st->h)
      return status_of(HMP_ERR_INVALID_VALUE, "feature outside the frame");
  const cudaStream_t cs = static_cast<cudaStream_t>(stream);
  Motion m{};
  m.corners = n;
  cudaError_t e = cudaSuccess;
  if (n > 0) e = cudaMemcpyAsync(st->xy, xy, size_t(n) * sizeof(int2), cudaMemcpyHostToDevice, cs);
  if (e == cudaSuccess) e = cudaMemcpyAsync(st->motion, &m, sizeof(m), cudaMemcpyHostToDevice, cs);
  if (e == cudaSuccess) e = cudaStreamSynchronize(cs);  // the host arrays may go once this returns
  return e == cudaSuccess ? status_of(HMP_OK, "") : cuda_failure(e, "feature upload");
}

}  // extern "C"
