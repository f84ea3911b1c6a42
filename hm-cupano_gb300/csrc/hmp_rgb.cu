// hmp_rgb.cu -- the stitch of RGB8 frames (uchar3): CudaStitchPano*<uchar3, float3>.
//
// The structure is the RGBA8 path's (hmp_gather.cu, hmp_pyramid_kernels.cuh): a canvas gather of
// resolved table entries beside a three-launch pyramid (down, coarse, fine) over the blocks near a
// seam. RGB pixels have no alpha, which makes three things simpler:
//   - every pixel of a level counts, mapped or not (unmapped ones are 0): means and upsamples are
//     plain, and the blends have no alpha tests (src/cuda/cudaBlend.cu:46-144, 389-455, 520-672;
//     cudaBlend3.cu:376-531; cudaBlendN.cu:199-288, 372-447);
//   - 8-bit samples under 2x2 means and bilinear taps stay short dyadic fractions (8 + 2l bits at
//     level l, two more in a tap), so every Gaussian level and Laplacian is exact in FP32 whatever
//     the order of its sums; only blended values round, and their sums keep the reference's order;
//   - where the labels are one image's over a pixel's whole support the result is that image's
//     level-0 pixel whatever the frames hold, so the copied blocks need no per-call check.
// A pixel is three bytes at any address: it is read as the two aligned words around it (one by one
// only where those would leave the frame) and written as whole words assembled in shared memory.
// Two 5K frames onto 8500x3300, six levels: 82 us a frame; five cameras onto 4999x1201, five levels:
// 62 us (as level-by-level kernels over float4 levels in HBM: 315 and 476 us). Now the gather and the
// latency of the three-launch chain bound it, as for RGBA8.
#include "hmp_pyramid_kernels.cuh"

namespace hmp {
namespace {

// A frame's bytes: [begin, end), from its first pixel to its last (the last row may end before the
// pitch).
struct RgbFrame {
  const unsigned char* begin;
  const unsigned char* end;
};
__device__ __forceinline__ RgbFrame rgb_frame(const SrcSet& S, int o, int b) {
  RgbFrame f;
  f.begin = reinterpret_cast<const unsigned char*>(S.ptr[o]) + b * S.bstride[o];
  f.end = f.begin + (long long)(S.h[o] - 1) * S.pitch[o] + 3LL * S.w[o];
  return f;
}

// Where a pixel's bytes lie: p (nullptr: none, the pixel is 0) and whether both aligned words around
// them lie in the frame.
struct RgbAt {
  const unsigned char* p;
  bool words;
};
__device__ __forceinline__ RgbAt rgb_at(const RgbFrame& f, long long off) {
  RgbAt r;
  r.p = f.begin + off;
  const unsigned char* w = r.p - (reinterpret_cast<uintptr_t>(r.p) & 3u);
  r.words = w >= f.begin && w + 8 <= f.end;
  return r;
}

// N pixels as 0x00BBGGRR: the word loads of all of them are in flight together (predicated, no
// branch); the few at a frame's ends follow byte by byte.
template <int N>
__device__ __forceinline__ void rgb_load(const RgbAt (&at)[N], uint32_t (&v)[N]) {
  uint32_t lo[N], hi[N];
  bool ends = false;
#pragma unroll
  for (int u = 0; u < N; ++u) {
    const uint32_t* w = reinterpret_cast<const uint32_t*>(at[u].p - (reinterpret_cast<uintptr_t>(at[u].p) & 3u));
    const bool in = at[u].p != nullptr && at[u].words;
    lo[u] = in ? __ldg(w) : 0u;
    hi[u] = in ? __ldg(w + 1) : 0u;
    ends = ends || (at[u].p != nullptr && !at[u].words);
  }
#pragma unroll
  for (int u = 0; u < N; ++u)
    v[u] = __funnelshift_r(lo[u], hi[u], unsigned(reinterpret_cast<uintptr_t>(at[u].p)) * 8u) & 0xFFFFFFu;
  if (ends) {
#pragma unroll
    for (int u = 0; u < N; ++u)
      if (at[u].p != nullptr && !at[u].words)
        v[u] = uint32_t(__ldg(at[u].p)) | uint32_t(__ldg(at[u].p + 1)) << 8 | uint32_t(__ldg(at[u].p + 2)) << 16;
  }
}

// Where the level-0 pixel of a looked-up (owner, packed entry) lies; none outside the table or the
// frame.
__device__ __forceinline__ RgbAt rgb_find(const SrcSet& S, int n, int o, uint32_t e, int b) {
  const int sx = int(e & 0xFFFFu), sy = int(e >> 16);
  if (o >= n || sx >= S.w[o] || sy >= S.h[o]) return RgbAt{nullptr, false};
  return rgb_at(rgb_frame(S, o, b), (long long)sy * S.pitch[o] + 3LL * sx);
}

// Tile (tx, ty) and frame b of this CTA: the dense grid, or entry blockIdx.x of the work list, the
// frames of a call fastest.
__device__ __forceinline__ void rgb_tile(const PyrArgs& a, int& tx, int& ty, int& b) {
  if (a.tiles != nullptr) {
    const int i = int(blockIdx.x) / a.list_frames;
    b = int(blockIdx.x) - i * a.list_frames;
    const uint32_t t = __ldg(a.tiles + i);
    tx = int(t & 0xFFFFu);
    ty = int((t >> 16) & 0x7FFFu);
  } else {
    tx = int(blockIdx.x);
    ty = int(blockIdx.y);
    b = int(blockIdx.z);
  }
}

// The slots whose plane meets [x0, x1) x [y0, y1) of the blend region, four bits each, at most cap.
__device__ __forceinline__ int rgb_active(const PyrArgs& a, int x0, int y0, int x1, int y1, int cap, uint32_t& list,
                                          uint32_t& cmap) {
  int na = 0;
  list = 0u;
  cmap = 0xFFFFFFFFu;
  for (int k = 0; k < a.n; ++k) {
    const PlaneDev& P = a.slot[k];
    if (x0 < P.x0 + P.w && P.x0 < x1 && y0 < P.y0 + P.h && P.y0 < y1 && na < cap) {
      list |= uint32_t(k) << (4 * na);
      cmap = (cmap & ~(0xFu << (4 * k))) | (uint32_t(na) << (4 * k));
      ++na;
    }
  }
  return na;
}

// Gaussian levels 1..L-1 of one TD x TD level-0 tile of every slot that meets it (the 2x2 mean has
// no halo). Level 0 is gathered into shared memory, table entries first, then their pixels, all of
// a thread's loads in flight together; levels 1 and 2 come from one pass over 4x4 pixel blocks with
// the channels summed as packed integers, deeper ones from the level before in shared memory.
template <int TD>
__global__ void __launch_bounds__(256) rgb_down_kernel(const __grid_constant__ PyrArgs a) {
  extern __shared__ float4 sm[];
  constexpr int T1 = TD / 2, T2 = TD / 4, A2 = T2 * T2, NJ = TD / 32, ROWS = TD / 8;
  constexpr int kBatch = ROWS * NJ < 8 ? ROWS * NJ : 8;  // loads in flight per thread and step
  int tx, ty, b;
  rgb_tile(a, tx, ty, b);
  const int cap = a.slots_cap, L = a.levels;
  uint32_t* pix = reinterpret_cast<uint32_t*>(sm);  // level 0: [cap][TD][TD]
  float4* bufA = sm;                                // levels 3, 5: [cap][T1*T1], over level 0
  float4* bufB = sm + cap * T1 * T1;                // levels 2, 4, 6: [cap][A2]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int X0 = tx * TD, Y0 = ty * TD;
  const int lw0 = a.lw[0], lh0 = a.lh[0], lw1 = a.lw[1], lh1 = a.lh[1];
  uint32_t list, cmap;
  const int na = rgb_active(a, X0, Y0, X0 + TD, Y0 + TD, cap, list, cmap);
#pragma unroll 1
  for (int c = 0; c < na; ++c) {
    const int k = (list >> (4 * c)) & 15u;
    const PlaneDev& P = a.slot[k];
    uint32_t* pk = pix + c * TD * TD;
#pragma unroll
    for (int g = 0; g < ROWS * NJ; g += kBatch) {
      uint32_t e[kBatch], v[kBatch];
      int o[kBatch];
#pragma unroll
      for (int u = 0; u < kBatch; ++u) {
        const int r = warp + 8 * ((g + u) / NJ), xl = lane + 32 * ((g + u) % NJ);
        const int x = X0 + xl, y = Y0 + r, rx = x - P.x0, ry = y - P.y0;
        const bool in = x < lw0 && y < lh0 && (unsigned)rx < (unsigned)P.w && (unsigned)ry < (unsigned)P.h;
        e[u] = in ? __ldg(P.map + (long long)ry * P.map_pitch + rx) : 0xFFFFFFFFu;
        o[u] = k;
        if (P.owner != nullptr) o[u] = in ? int(__ldg(P.owner + (long long)ry * P.owner_pitch + rx)) : 0xFF;
      }
      RgbAt at[kBatch];
      if (P.owner == nullptr) {  // image k's frame, once
        const RgbFrame f = rgb_frame(a.S, k, b);
        const int fw = a.S.w[k], fh = a.S.h[k];
        const long long pitch = a.S.pitch[k];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
          const int sx = int(e[u] & 0xFFFFu), sy = int(e[u] >> 16);
          at[u] = rgb_at(f, sy * pitch + 3 * sx);
          if (sx >= fw || sy >= fh) at[u].p = nullptr;
        }
      } else {
#pragma unroll
        for (int u = 0; u < kBatch; ++u) at[u] = rgb_find(a.S, a.n, o[u], e[u], b);
      }
      rgb_load(at, v);
#pragma unroll
      for (int u = 0; u < kBatch; ++u) {
        const int r = warp + 8 * ((g + u) / NJ), xl = lane + 32 * ((g + u) % NJ);
        pk[r * TD + xl] = v[u];
      }
    }
  }
  __syncthreads();
  const bool has2 = L > 2;
  const int lw2 = a.lw[has2 ? 2 : 1], lh2 = a.lh[has2 ? 2 : 1];
#pragma unroll 1
  for (int it = tid; it < na * A2; it += 256) {
    const int c = it / A2, j = it - c * A2, k = (list >> (4 * c)) & 15u;
    const int tx2 = j % T2, ty2 = j / T2;
    const int gx2 = (X0 >> 2) + tx2, gy2 = (Y0 >> 2) + ty2;
    const uint32_t* pk = pix + c * TD * TD;
    float4* G1 = static_cast<float4*>(a.G[k][1]) + (long long)b * lw1 * lh1;
    float s0 = 0.f, s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int x1 = 2 * tx2 + (q & 1), y1 = 2 * ty2 + (q >> 1);
      const int gx = (X0 >> 1) + x1, gy = (Y0 >> 1) + y1;
      if (gx < lw1 && gy < lh1) {
        // Pixels past the level are 0 in the tile, so only the count knows the edge.
        const uint2 r0 = *reinterpret_cast<const uint2*>(pk + (2 * y1) * TD + 2 * x1);
        const uint2 r1 = *reinterpret_cast<const uint2*>(pk + (2 * y1 + 1) * TD + 2 * x1);
        const uint32_t rb = (r0.x & 0xFF00FFu) + (r0.y & 0xFF00FFu) + (r1.x & 0xFF00FFu) + (r1.y & 0xFF00FFu);
        const uint32_t g = ((r0.x >> 8) & 0xFFu) + ((r0.y >> 8) & 0xFFu) + ((r1.x >> 8) & 0xFFu) + ((r1.y >> 8) & 0xFFu);
        const float inv = (2 * gx + 1 < lw0 ? 0.5f : 1.f) * (2 * gy + 1 < lh0 ? 0.5f : 1.f);
        // Sums below 2^10 in the low bits of 2^23.
        const float v0 = (__uint_as_float(0x4B000000u | (rb & 0xFFFFu)) - 8388608.0f) * inv;
        const float v1 = (__uint_as_float(0x4B000000u | g) - 8388608.0f) * inv;
        const float v2 = (__uint_as_float(0x4B000000u | (rb >> 16)) - 8388608.0f) * inv;
        G1[(long long)gy * lw1 + gx] = make_float4(v0, v1, v2, 0.f);
        s0 += v0;
        s1 += v1;
        s2 += v2;
      }
    }
    if (has2) {
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (gx2 < lw2 && gy2 < lh2) {
        const float inv = (2 * gx2 + 1 < lw1 ? 0.5f : 1.f) * (2 * gy2 + 1 < lh1 ? 0.5f : 1.f);
        v = make_float4(s0 * inv, s1 * inv, s2 * inv, 0.f);
        static_cast<float4*>(a.G[k][2])[(long long)b * lw2 * lh2 + (long long)gy2 * lw2 + gx2] = v;
      }
      bufB[c * A2 + j] = v;
    }
  }
  __syncthreads();
#pragma unroll
  for (int l = 3; l < kL; ++l) {
    if (l >= L) break;
    const int Tp = TD >> (l - 1), Tn = TD >> l, area = Tn * Tn;
    const float4* src = (l & 1) ? bufB : bufA;
    float4* dst = (l & 1) ? bufA : bufB;
    const int sstride = (l & 1) ? A2 : T1 * T1, dstride = (l & 1) ? T1 * T1 : A2;
    const int lwl = a.lw[l], lhl = a.lh[l], lwp = a.lw[l - 1], lhp = a.lh[l - 1];
#pragma unroll 1
    for (int it = tid; it < na * area; it += 256) {
      const int c = it / area, j = it - c * area, k = (list >> (4 * c)) & 15u;
      const int x = j % Tn, y = j / Tn, gx = (X0 >> l) + x, gy = (Y0 >> l) + y;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (gx < lwl && gy < lhl) {
        const float4* s = src + c * sstride + 2 * y * Tp + 2 * x;  // pixels past the level are 0
        const float4 p = s[0], q = s[1], r = s[Tp], t = s[Tp + 1];
        const float inv = (2 * gx + 1 < lwp ? 0.5f : 1.f) * (2 * gy + 1 < lhp ? 0.5f : 1.f);
        v = make_float4((p.x + q.x + r.x + t.x) * inv, (p.y + q.y + r.y + t.y) * inv, (p.z + q.z + r.z + t.z) * inv, 0.f);
        static_cast<float4*>(a.G[k][l])[(long long)b * lwl * lhl + (long long)gy * lwl + gx] = v;
      }
      dst[c * dstride + j] = v;
    }
    __syncthreads();
  }
}

// Bilinear upsample at parity (ox, oy) from the taps t[i], t[i + dx], t[i + dy], t[i + dy + dx], in
// the reconstruction's order ((v00 w00 + v10 w10) + v01 w01) + v11 w11 (a tap of weight 0 adds 0);
// Laplacians use it too, where every order gives the same exact value.
__device__ __forceinline__ float3 rgb_up(const float4* t, int i, int dx, int dy, bool ox, bool oy) {
  const float4 p = t[i];
  if (!ox && !oy) return make_float3(p.x, p.y, p.z);
  if (ox != oy) {
    const float4 q = t[i + (ox ? dx : dy)];
    return make_float3(p.x * 0.5f + q.x * 0.5f, p.y * 0.5f + q.y * 0.5f, p.z * 0.5f + q.z * 0.5f);
  }
  const float4 q = t[i + dx], r = t[i + dy], s = t[i + dy + dx];
  return make_float3(((p.x * 0.25f + q.x * 0.25f) + r.x * 0.25f) + s.x * 0.25f,
                     ((p.y * 0.25f + q.y * 0.25f) + r.y * 0.25f) + s.y * 0.25f,
                     ((p.z * 0.25f + q.z * 0.25f) + r.z * 0.25f) + s.z * 0.25f);
}

// Blend of the Laplacians lap(c) of a tile's listed slots (zero for the others) with fractional
// weights mk[0..K).
template <int RULE, class Lap>
__device__ __forceinline__ float3 rgb_blend(int n, uint32_t cmap, const float* mk, Lap lap) {
  const auto of = [&](int k) {
    const uint32_t c = (cmap >> (4 * k)) & 15u;
    return c < 15u ? lap(int(c)) : make_float3(0.f, 0.f, 0.f);
  };
  if constexpr (RULE == kRuleTwo) {
    const float m = __ldg(mk), w = 1.f - m;
    const float3 p = of(0), q = of(1);
    return make_float3(m * p.x + w * q.x, m * p.y + w * q.y, m * p.z + w * q.z);
  } else if constexpr (RULE == kRuleThree) {
    const float m0 = __ldg(mk), m1 = __ldg(mk + 1), m2 = __ldg(mk + 2);
    const float3 p = of(0), q = of(1), r = of(2);
    return make_float3((m0 * p.x + m1 * q.x) + m2 * r.x, (m0 * p.y + m1 * q.y) + m2 * r.y,
                       (m0 * p.z + m1 * q.z) + m2 * r.z);
  } else {
    float sum = 0.f;
    for (int k = 0; k < n; ++k) sum += __ldg(mk + k);
    float3 acc = make_float3(0.f, 0.f, 0.f);
    for (int k = 0; k < n; ++k) {
      float w = __ldg(mk + k);
      if (sum > 0.f && sum != 1.f) w /= sum;  // masks sum to 1 unless a label has no image
      if (w == 0.f) continue;
      const float3 p = of(k);
      acc.x += w * p.x;
      acc.y += w * p.y;
      acc.z += w * p.z;
    }
    return acc;
  }
}

// The blended Laplacian of one pixel at level l >= 1: one image's where the mask class says so.
template <int RULE, class Lap>
__device__ __forceinline__ float3 rgb_level_blend(int n, uint32_t cmap, int hot, const float* mk, Lap lap) {
  if (hot < 16) {
    const uint32_t c = (cmap >> (4 * hot)) & 15u;
    return c < 15u ? lap(int(c)) : make_float3(0.f, 0.f, 0.f);
  }
  if (hot == kHotNone) return make_float3(0.f, 0.f, 0.f);
  return rgb_blend<RULE>(n, cmap, mk, lap);
}

// R^1 of one T1 x T1 tile of level-1 pixels: levels 2..L-1 of the slots that meet the tile's
// footprint (with the upsample's halo) are copied into shared memory together, then blended and
// reconstructed from the coarsest level down (pyr_coarse_n_kernel's walk).
template <int RULE, int T1>
__global__ void __launch_bounds__(256) rgb_coarse_kernel(const __grid_constant__ PyrArgs a) {
  extern __shared__ float4 sm[];
  char* smb = reinterpret_cast<char*>(sm);
  int tx, ty, b;
  rgb_tile(a, tx, ty, b);
  if (a.tiles == nullptr) tx += a.tx0, ty += a.ty0;
  const int n = a.n, K = a.K, cap = a.coarse_cap;
  const int X1 = tx * T1, Y1 = ty * T1, L = a.levels, c = L - 1, tid = threadIdx.x;
  const CoarseLayout lo = coarse_layout(cap, 0, T1, L, int(sizeof(float4)));
  int rax[kL], ray[kL], rbx[kL], rby[kL];
  int fx0, fy0, fx1, fy1;  // level-0 footprint of every region
  {
    int ax = X1, ay = Y1, bx = min(X1 + T1, a.lw[1]), by = min(Y1 + T1, a.lh[1]);
    fx0 = ax << 1, fy0 = ay << 1, fx1 = bx << 1, fy1 = by << 1;
#pragma unroll
    for (int l = 1; l < kL; ++l) {
      if (l > 1 && l < L) {
        ax >>= 1;
        ay >>= 1;
        bx = min(((bx - 1) >> 1) + 2, a.lw[l]);
        by = min(((by - 1) >> 1) + 2, a.lh[l]);
        fx0 = min(fx0, ax << l);
        fy0 = min(fy0, ay << l);
        fx1 = max(fx1, bx << l);
        fy1 = max(fy1, by << l);
      }
      rax[l] = ax;
      ray[l] = ay;
      rbx[l] = bx;
      rby[l] = by;
    }
  }
  uint32_t list, cmap;
  const int na = rgb_active(a, fx0, fy0, fx1, fy1, cap, list, cmap);
  // The mask classes of this thread's pixels at every level, before the wait for the levels.
  constexpr int HALF = T1 / 2, CLS = HALF * HALF, PER = T1 * T1 / 256;
  const int lw1 = a.lw[1], lh1 = a.lh[1];
  uint8_t hot[kL][2], hot1[PER];
#pragma unroll
  for (int l = 2; l < kL; ++l) {
    if (l >= L) break;
    const int CW = up_cw(T1, l - 1), QW = (CW + 1) / 2, QC = QW * QW;
    static_assert(4 * ((up_cw(T1, 1) + 1) / 2) * ((up_cw(T1, 1) + 1) / 2) <= 512, "two pixels a thread");
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int t = tid + 256 * i, cls = t / QC, j = t - cls * QC;
      const int px = rax[l] + 2 * (j % QW) + (cls & 1), py = ray[l] + 2 * (j / QW) + (cls >> 1);
      hot[l][i] = t < 4 * QC && px < rbx[l] && py < rby[l] ? __ldg(a.hotL[l] + (long long)py * a.lw[l] + px) : kHotNone;
    }
  }
#pragma unroll
  for (int p = 0; p < PER; ++p) {
    const int i = p * 256 + tid;
    const int px = X1 + 2 * ((i % CLS) % HALF) + ((i / CLS) & 1), py = Y1 + 2 * ((i % CLS) / HALF) + ((i / CLS) >> 1);
    hot1[p] = px < lw1 && py < lh1 ? __ldg(a.hotL[1] + (long long)py * lw1 + px) : kHotNone;
  }
  grid_dep_wait();  // G^l of rgb_down
#pragma unroll
  for (int l = 2; l < kL; ++l) {
    if (l >= L) break;
    const int CW = up_cw(T1, l - 1), CAP = CW * CW;
    const int lax = rax[l], lay = ray[l], rw = rbx[l] - lax, rh = rby[l] - lay;
    const int lw = a.lw[l], lh = a.lh[l];
#pragma unroll 1
    for (int ci = 0; ci < na; ++ci) {
      const float4* Gl = static_cast<const float4*>(a.G[(list >> (4 * ci)) & 15u][l]) + (long long)b * lw * lh;
      float4* gl = reinterpret_cast<float4*>(smb + lo.g[l]) + ci * CAP;
      for (int i = tid; i < CAP; i += 256) {
        const int x = i % CW, y = i / CW;
        if (x < rw && y < rh) cp_async<16>(gl + i, Gl + (long long)(lay + y) * lw + (lax + x));
      }
    }
  }
  // G^1 of this thread's own pixels, the one image's the class names, with the rest in flight.
  const long long boff = (long long)b * lw1 * lh1;
  float4 own1[PER];
#pragma unroll
  for (int p = 0; p < PER; ++p) {
    const int i = p * 256 + tid;
    const int px = X1 + 2 * ((i % CLS) % HALF) + ((i / CLS) & 1), py = Y1 + 2 * ((i % CLS) / HALF) + ((i / CLS) >> 1);
    own1[p] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (hot1[p] < n && ((cmap >> (4 * hot1[p])) & 15u) < 15u)
      own1[p] = load_dep(static_cast<const float4*>(a.G[hot1[p]][1]) + boff + (long long)py * lw1 + px);
  }
  cp_async_commit_wait_all();
  __syncthreads();
#pragma unroll
  for (int l = kL - 1; l >= 2; --l) {
    if (l > c) continue;
    const int CW = up_cw(T1, l - 1), CAP = CW * CW, QW = (CW + 1) / 2, QC = QW * QW;
    const int lax = rax[l], lay = ray[l], rw = rbx[l] - lax, rh = rby[l] - lay, lw = a.lw[l];
    const float4* gcur = reinterpret_cast<const float4*>(smb + lo.g[l]);
    float4* rcur = reinterpret_cast<float4*>(smb + lo.r[l]);
    const bool has_next = l < c;
    const int nl = l + 1 < kL ? l + 1 : l;
    const int CWN = up_cw(T1, nl - 1), CAPN = CWN * CWN, nax = rax[nl], nay = ray[nl];
    const int lwn = a.lw[nl], lhn = a.lh[nl];
    const float4* gnext = reinterpret_cast<const float4*>(smb + lo.g[nl]);
    const float4* rnext = reinterpret_cast<const float4*>(smb + lo.r[nl]);
#pragma unroll
    for (int it = 0; it < 2; ++it) {  // by parity class, so that a warp's upsamples agree
      const int t = tid + 256 * it;
      if (t >= 4 * QC) break;
      const int cls = t / QC, j = t - cls * QC;
      const int x = 2 * (j % QW) + (cls & 1), y = 2 * (j / QW) + (cls >> 1);
      if (x >= rw || y >= rh) continue;
      const int i = y * CW + x, px = lax + x, py = lay + y;
      const long long o = (long long)py * lw + px;
      const int gxi = px >> 1, gyi = py >> 1;
      const int un = (gyi - nay) * CWN + gxi - nax;
      const int dx = gxi + 1 < lwn ? 1 : 0, dy = gyi + 1 < lhn ? CWN : 0;
      const bool ox = (px & 1) != 0, oy = (py & 1) != 0;
      const auto lap = [&](int ci) {
        const float4 g = gcur[ci * CAP + i];
        float3 r = make_float3(g.x, g.y, g.z);
        if (has_next) {
          const float3 u = rgb_up(gnext + ci * CAPN, un, dx, dy, ox, oy);
          r.x -= u.x;
          r.y -= u.y;
          r.z -= u.z;
        }
        return r;
      };
      float3 r = rgb_level_blend<RULE>(n, cmap, hot[l][it], a.maskL[l] + o * K, lap);
      if (has_next) {
        const float3 u = rgb_up(rnext, un, dx, dy, ox, oy);
        r.x = u.x + r.x;
        r.y = u.y + r.y;
        r.z = u.z + r.z;
      }
      rcur[i] = make_float4(r.x, r.y, r.z, 0.f);
    }
    __syncthreads();
  }
  const bool has2 = c >= 2;
  const int CW2 = up_cw(T1, 1), CAP2 = CW2 * CW2, nax = rax[2], nay = ray[2];
  const int lw2 = a.lw[has2 ? 2 : 1], lh2 = a.lh[has2 ? 2 : 1];
  const float4* g2 = reinterpret_cast<const float4*>(smb + lo.g[2]);
  const float4* r2 = reinterpret_cast<const float4*>(smb + lo.r[2]);
#pragma unroll
  for (int p = 0; p < PER; ++p) {
    const int i = p * 256 + tid;
    const int px = X1 + 2 * ((i % CLS) % HALF) + ((i / CLS) & 1), py = Y1 + 2 * ((i % CLS) / HALF) + ((i / CLS) >> 1);
    if (px >= lw1 || py >= lh1) continue;
    const long long o = (long long)py * lw1 + px;
    const int gxi = px >> 1, gyi = py >> 1;
    const int un = (gyi - nay) * CW2 + gxi - nax;
    const int dx = gxi + 1 < lw2 ? 1 : 0, dy = gyi + 1 < lh2 ? CW2 : 0;
    const bool ox = (px & 1) != 0, oy = (py & 1) != 0;
    const auto lap = [&](int ci) {
      const int k = (list >> (4 * ci)) & 15u;
      const float4 g = k == hot1[p] ? own1[p] : load_dep(static_cast<const float4*>(a.G[k][1]) + boff + o);
      float3 r = make_float3(g.x, g.y, g.z);
      if (has2) {
        const float3 u = rgb_up(g2 + ci * CAP2, un, dx, dy, ox, oy);
        r.x -= u.x;
        r.y -= u.y;
        r.z -= u.z;
      }
      return r;
    };
    float3 r = rgb_level_blend<RULE>(n, cmap, hot1[p], a.maskL[1] + o * K, lap);
    if (has2) {
      const float3 u = rgb_up(r2, un, dx, dy, ox, oy);
      r.x = u.x + r.x;
      r.y = u.y + r.y;
      r.z = u.z + r.z;
    }
    a.R1[boff + o] = make_float4(r.x, r.y, r.z, 0.f);
  }
}

// Stores `count` bytes of shared memory s (s[i] goes to dst[i]; s is as far past a word boundary as
// dst) by the calling group of `threads` threads: whole words inside, single bytes at the ends.
__device__ __forceinline__ void store_bytes(unsigned char* dst, const unsigned char* s, int count, int t, int threads) {
  const int head = min(int(-reinterpret_cast<uintptr_t>(dst) & 3u), count), words = (count - head) >> 2;
  for (int w = t; w < words; w += threads)
    *reinterpret_cast<uint32_t*>(dst + head + 4 * w) = *reinterpret_cast<const uint32_t*>(s + head + 4 * w);
  const int tail = head + 4 * words;
  if (t < head) dst[t] = s[t];
  if (t < count - tail) dst[tail + t] = s[tail + t];
}

// Level 0 of the write rect: a CTA a 64 x 16 block, a thread a 2x2 quad. The label names the one
// image whose Laplacian a pixel takes (two-image seams other than 0 / 1 blend both), so a pixel is
// one table lookup and one fetch, issued before the wait for the levels. The block's bytes are
// assembled in shared memory and stored as words.
constexpr int kRgbRow = 200;  // bytes of a staged row: 64 pixels and up to 3 of misalignment, a multiple of 4

template <int RULE>
__global__ void __launch_bounds__(256) rgb_fine_kernel(const __grid_constant__ PyrArgs a) {
  extern __shared__ float4 fsm[];  // R^1 tile, then the G^1 tiles of the listed slots
  __shared__ __align__(16) unsigned char s_out[16][kRgbRow];
  int tx, ty, b;
  rgb_tile(a, tx, ty, b);
  const int n = a.n, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int bx0 = (a.wx0 & ~1) + tx * 64, by0 = (a.wy0 & ~1) + ty * 16;
  const int X = bx0 + 2 * lane, Y = by0 + 2 * warp;
  const bool has1 = a.levels > 1;
  const int lw0 = a.lw[0], lh0 = a.lh[0], lw1 = a.lw[1], lh1 = a.lh[1];
  float4* rs = fsm;
  float4* gs = fsm + kFineTA;
  uint32_t list, cmap;
  const int na = rgb_active(a, bx0, by0, bx0 + 66, by0 + 18, a.fine_cap, list, cmap);
  const auto lookup = [&](int k, int x, int y, int& o, uint32_t& e) { slot_lookup(a.slot[k], k, x, y, o, e); };
  bool live[4];
  int v[4], o[4];
  uint32_t e[4], px[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int x = X + (q & 1), y = Y + (q >> 1);
    live[q] = x < lw0 && y < lh0 && x >= a.wx0 && x < a.wx1 && y >= a.wy0 && y < a.wy1;
    int s = live[q] ? int(__ldg(a.mask0 + (long long)y * a.mask0_pitch + x)) : 0xFF;
    if (RULE == kRuleTwo && live[q]) s = s == 1 ? 0 : (s == 0 ? 1 : 0x100 + s);  // the slot, or a weight
    v[q] = s;
    o[q] = 0xFF;
    e[q] = 0xFFFFFFFFu;
    if (live[q] && s < n) lookup(s, x, y, o[q], e[q]);
  }
  {
    RgbAt at[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) at[q] = rgb_find(a.S, n, o[q], e[q], b);
    rgb_load(at, px);
  }
  if (has1) {
    grid_dep_wait();  // R^1 of rgb_coarse, G^1 of rgb_down
    const int tx0 = bx0 >> 1, ty0 = by0 >> 1;
    const long long fo = (long long)b * lw1 * lh1;
    for (int j = tid; j < kFineTA; j += 256) {
      const int y = min(ty0 + j / kFineTW, lh1 - 1), x = min(tx0 + j % kFineTW, lw1 - 1);
      const long long at = fo + (long long)y * lw1 + x;
      cp_async<16>(rs + j, a.R1 + at);
      for (int c = 0; c < na; ++c)
        cp_async<16>(gs + c * kFineTA + j, static_cast<const float4*>(a.G[(list >> (4 * c)) & 15u][1]) + at);
    }
    cp_async_commit_wait_all();
    __syncthreads();
  }
  const int ti = warp * kFineTW + lane;
  unsigned char* canvas = reinterpret_cast<unsigned char*>(a.C.ptr) + b * a.C.bstride;
  // Row r of the block starts at this canvas byte (before the write rect's columns are cut).
  const auto row_at = [&](int r) {
    return canvas + (long long)(by0 + r + a.cy_off) * a.C.pitch + 3LL * (bx0 + a.cx_off);
  };
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    if (!live[q]) continue;
    const bool ox = (q & 1) != 0, oy = (q >> 1) != 0;
    const auto lap = [&](int k, uint32_t p) {
      const float4 f = u32_to_f4(p);
      float3 r = make_float3(f.x, f.y, f.z);
      const uint32_t c = (cmap >> (4 * k)) & 15u;
      if (has1 && c < 15u) {
        const float3 u = rgb_up(gs + c * kFineTA, ti, 1, kFineTW, ox, oy);
        r.x -= u.x;
        r.y -= u.y;
        r.z -= u.z;
      }
      return r;
    };
    float3 r = make_float3(0.f, 0.f, 0.f);
    if (v[q] < n) {
      r = lap(v[q], px[q]);
    } else if (RULE == kRuleTwo) {
      const float m = float(v[q] - 0x100), w = 1.f - m;
      float3 p[2];
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        int ok;
        uint32_t ek;
        lookup(k, X + (q & 1), Y + (q >> 1), ok, ek);
        const RgbAt at[1] = {rgb_find(a.S, n, ok, ek, b)};
        uint32_t one[1];
        rgb_load(at, one);
        p[k] = lap(k, one[0]);
      }
      r = make_float3(m * p[0].x + w * p[1].x, m * p[0].y + w * p[1].y, m * p[0].z + w * p[1].z);
    }
    if (has1) {
      const float3 u = rgb_up(rs, ti, 1, kFineTW, ox, oy);
      r.x = u.x + r.x;
      r.y = u.y + r.y;
      r.z = u.z + r.z;
    }
    const int row = 2 * warp + (q >> 1);
    unsigned char* d = s_out[row] + (reinterpret_cast<uintptr_t>(row_at(row)) & 3u) + 3 * (2 * lane + (q & 1));
    d[0] = pack_u8(r.x);
    d[1] = pack_u8(r.y);
    d[2] = pack_u8(r.z);
  }
  __syncwarp();  // a warp's two rows are its own
  const int c0 = max(bx0, a.wx0) - bx0, c1 = min(min(bx0 + 64, a.wx1), lw0) - bx0;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int row = 2 * warp + i, y = by0 + row;
    if (y < a.wy0 || y >= a.wy1 || y >= lh0 || c1 <= c0) continue;
    unsigned char* dst = row_at(row);
    const unsigned char* src = s_out[row] + (reinterpret_cast<uintptr_t>(dst) & 3u);
    store_bytes(dst + 3 * c0, src + 3 * c0, 3 * (c1 - c0), lane, 32);
  }
}

// Canvas gather: a warp a 256-pixel row segment, lane l its pixels l + 32j. Resolved entries (byte
// offsets into the owner's frame, resolve_plane_kernel) are read once and serve every frame of the
// call; a segment of one owner without fills skips the tests per pixel. The segment's pixels are
// assembled into words in shared memory (each word takes two neighbouring pixels) so that the canvas
// is written in full lines; the words at a segment's ends, and those with a pixel the pyramid writes,
// are stored byte by byte. kPacked: frames past the offsets' range, from the packed entries.
// 4 (entry) + 3 + 3 bytes a pixel; bound by the issue of 57 instructions a pixel (70 % of the issue slots).
// 8500x3300 (27 Mpx of it): 181 -> 61 us alone, 4.4 TB/s.
constexpr uint32_t kRgbSkip = 0x80000000u;  // a staged pixel that is not stored

template <bool kPacked>
__global__ void __launch_bounds__(256, 5) rgb_gather_kernel(const __grid_constant__ GatherArgs a,
                                                            const __grid_constant__ SkipMap skip) {
  __shared__ uint32_t s_px[8][kSegPixels + 4];
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  const int x0 = blockIdx.x * kSegPixels, y = blockIdx.y * 8 + wp;
  const int W = a.C.w, H = a.C.h;
  if (y >= H) return;
  const bool row_skip = y >= a.skip_y0 && y < a.skip_y1;
  if (row_skip && x0 >= a.skip_x0 && x0 + kSegPixels <= a.skip_x1) return;
  constexpr int PJ = kSegPixels / 32;
  const int count = min(kSegPixels, W - x0);
  uint32_t e[PJ];
  const uint32_t* mrow = a.P.map + (long long)y * a.P.map_pitch;
#pragma unroll
  for (int j = 0; j < PJ; ++j) {
    const int x = x0 + lane + 32 * j;
    e[j] = x < W ? __ldg(mrow + x) : (kPacked ? 0xFFFFFFFFu : kOffZero);
  }
  const unsigned so = kPacked ? kSegMixed : __ldg(a.seg_owner + (long long)y * a.seg_pitch + blockIdx.x);
  const bool plain = so < kSegFills && count == kSegPixels && !(row_skip && x0 < a.skip_x1 && x0 + kSegPixels > a.skip_x0);
  uint32_t* s = s_px[wp];
  for (int b = 0; b < a.batch; ++b) {
    unsigned char* dst = reinterpret_cast<unsigned char*>(a.C.ptr) + b * a.C.bstride + (long long)y * a.C.pitch + 3LL * x0;
    const int mis = int(reinterpret_cast<uintptr_t>(dst) & 3u);
    __syncwarp();  // the previous frame's words are read
    bool fast = false;
    if (plain) {
      // One owner, no fills: byte offsets from the frame's word below its first byte.
      const RgbFrame f = rgb_frame(a.S, int(so), b);
      const unsigned fm = unsigned(reinterpret_cast<uintptr_t>(f.begin)) & 3u;
      const uint32_t* base = reinterpret_cast<const uint32_t*>(f.begin - fm);
      const unsigned first = fm ? 1u : 0u, last = unsigned((f.end - f.begin + fm) >> 2) - 2u;  // words a pixel may start in
      bool in = f.end - f.begin >= 16;
#pragma unroll
      for (int j = 0; j < PJ; ++j) in = in && ((e[j] + fm) >> 2) - first <= last - first;
      fast = __all_sync(0xFFFFFFFFu, in);
      if (fast) {
        uint32_t lo[PJ], hi[PJ];
#pragma unroll
        for (int j = 0; j < PJ; ++j) {
          const uint32_t* w = base + ((e[j] + fm) >> 2);
          lo[j] = __ldg(w);
          hi[j] = __ldg(w + 1);
        }
#pragma unroll
        for (int j = 0; j < PJ; ++j) s[lane + 32 * j] = __funnelshift_r(lo[j], hi[j], (e[j] + fm) * 8u) & 0xFFFFFFu;
      }
    }
    if (!fast) {
#pragma unroll
      for (int j = 0; j < PJ; j += 2) {
        RgbAt at[2];
        uint32_t v[2];
        bool drop[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int x = x0 + lane + 32 * (j + u);
          const uint32_t ej = e[j + u];
          drop[u] = row_skip && x >= a.skip_x0 && x < a.skip_x1;
          at[u] = RgbAt{nullptr, false};
          if (kPacked) {
            if (skip.map && x >= skip.wr_x0 && x < skip.wr_x1 && y >= skip.wr_y0 && y < skip.wr_y1)
              drop[u] = drop[u] || skip.map[(long long)((y - skip.y0) >> 4) * skip.pitch + ((x - skip.x0) >> 6)] != 0;
            const int o = x >= W ? 0xFF
                                 : (a.P.owner ? int(__ldg(a.P.owner + (long long)y * a.P.owner_pitch + x)) : a.P.default_owner);
            at[u] = rgb_find(a.S, a.n_owners, o, ej, b);
          } else {
            drop[u] = drop[u] || ej == kOffSkip;
            if (ej < kOffSkip) {
              const int o = so != kSegMixed ? int(so & (kSegFills - 1)) : int(ej >> kOwnerShift);
              at[u] = rgb_at(rgb_frame(a.S, o, b), ej & kOffMask);
            }
          }
        }
        rgb_load(at, v);
#pragma unroll
        for (int u = 0; u < 2; ++u) s[lane + 32 * (j + u)] = drop[u] ? kRgbSkip : v[u];
      }
    }
    __syncwarp();
    // Word w holds bytes 4w - mis .. 4w - mis + 3 of the segment.
    const int bytes = 3 * count;
    if (fast) {
      // 192 words; word w + 96 takes the pixels 128 past word w's. With mis, word 0 and the bytes past
      // word 191 are partial.
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const int w = lane + 32 * i, q = 4 * w - mis, p = (q + 3) / 3 - 1, f = q - 3 * p;
        uint32_t* d = reinterpret_cast<uint32_t*>(dst - mis) + w;
        if (q >= 0) __stcs(d, (s[p] >> (8 * f)) | (s[p + 1] << (24 - 8 * f)));
        __stcs(d + 96, (s[p + 128] >> (8 * f)) | (s[p + 129] << (24 - 8 * f)));
      }
      if (mis != 0 && lane < 4) {
        const int k = lane < 4 - mis ? lane : bytes - 4 + lane;
        dst[k] = (unsigned char)(s[k / 3] >> (8 * (k % 3)));
      }
      continue;
    }
    const int words = (bytes + mis + 3) >> 2;
    for (int w = lane; w < words; w += 32) {
      const int q = 4 * w - mis;
      const int p = max(q, 0) / 3, f = q - 3 * p;
      if (q >= 0 && q + 4 <= bytes) {
        const uint32_t lo = s[p], hi = s[p + 1];
        if (!((lo | hi) & kRgbSkip)) {
          __stcs(reinterpret_cast<uint32_t*>(dst + q), (lo >> (8 * f)) | (hi << (24 - 8 * f)));
          continue;
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int k = q + i;
        if (k < 0 || k >= bytes) continue;
        const uint32_t t = s[k / 3];
        if (!(t & kRgbSkip)) dst[k] = (unsigned char)(t >> (8 * (k % 3)));
      }
    }
  }
}

template <typename Kern>
void launch_chained(Kern k, dim3 grid, size_t smem, bool pdl, cudaStream_t stream, const PyrArgs& a) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(256);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = pdl ? 1 : 0;
  cudaLaunchKernelEx(&cfg, k, a);
}

}  // namespace

cudaError_t rgb_init() {
  constexpr int kMax = 227 * 1024;
  cudaFuncSetAttribute(rgb_down_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMax);
  cudaFuncSetAttribute(rgb_down_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMax);
  cudaFuncSetAttribute(rgb_coarse_kernel<kRuleTwo, 32>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMax);
  cudaFuncSetAttribute(rgb_coarse_kernel<kRuleThree, 32>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMax);
  cudaFuncSetAttribute(rgb_coarse_kernel<kRuleNway, 32>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMax);
  // Eight slots' G^1 tiles and the staged rows: 46 KB, close to the default limit.
  cudaFuncSetAttribute(rgb_fine_kernel<kRuleTwo>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMax - 8192);
  cudaFuncSetAttribute(rgb_fine_kernel<kRuleThree>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMax - 8192);
  cudaFuncSetAttribute(rgb_fine_kernel<kRuleNway>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMax - 8192);
  return cudaGetLastError();
}

cudaError_t launch_rgb_gather(const GatherArgs& a, bool packed, const SkipMap& skip, cudaStream_t stream) {
  const dim3 grid((a.C.w + kSegPixels - 1) / kSegPixels, (a.C.h + 7) / 8);
  if (packed)
    rgb_gather_kernel<true><<<grid, 256, 0, stream>>>(a, skip);
  else
    rgb_gather_kernel<false><<<grid, 256, 0, stream>>>(a, skip);
  return cudaGetLastError();
}

cudaError_t launch_rgb_down(const PyrArgs& a, dim3 grid, cudaStream_t stream) {
  const size_t smem = pyr_down_smem(a.slots_cap, a.tile);
  if (a.tile == 32)
    rgb_down_kernel<32><<<grid, 256, smem, stream>>>(a);
  else if (a.tile == 64)
    rgb_down_kernel<64><<<grid, 256, smem, stream>>>(a);
  else
    return cudaErrorInvalidValue;
  return cudaGetLastError();
}

cudaError_t launch_rgb_coarse(const PyrArgs& a, int rule, dim3 grid, size_t smem, cudaStream_t stream) {
  if (a.tile != 32) return cudaErrorInvalidValue;
  if (rule == kRuleTwo)
    launch_chained(rgb_coarse_kernel<kRuleTwo, 32>, grid, smem, true, stream, a);
  else if (rule == kRuleThree)
    launch_chained(rgb_coarse_kernel<kRuleThree, 32>, grid, smem, true, stream, a);
  else
    launch_chained(rgb_coarse_kernel<kRuleNway, 32>, grid, smem, true, stream, a);
  return cudaGetLastError();
}

cudaError_t launch_rgb_fine(const PyrArgs& a, int rule, dim3 grid, cudaStream_t stream) {
  const size_t smem = a.levels > 1 ? size_t(kFineTA) * sizeof(float4) * (1 + a.fine_cap) : 0;
  const bool pdl = a.levels > 1;
  if (rule == kRuleTwo)
    launch_chained(rgb_fine_kernel<kRuleTwo>, grid, smem, pdl, stream, a);
  else if (rule == kRuleThree)
    launch_chained(rgb_fine_kernel<kRuleThree>, grid, smem, pdl, stream, a);
  else
    launch_chained(rgb_fine_kernel<kRuleNway>, grid, smem, pdl, stream, a);
  return cudaGetLastError();
}

}  // namespace hmp
