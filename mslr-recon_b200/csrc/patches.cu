// patches.cu — image series ↔ patches: extraction, recombination and their
// adjoints (src/recon.jl:53-126), and the patch geometry on the host.
//
// All are bound by memory: patches in, images out or the reverse, once each.
// One thread has one voxel (of the image, or of a patch) for eight frames: its
// coordinates, covering patches and offsets — integer divisions, which bound
// these kernels when every element had its own — are worked out once, and the
// eight frames' accesses are in flight together.  Starts and covering ranges
// are arithmetic of the stride, so that a call without a context needs no
// tables on the device: allocating, filling and freeing them took longer than
// its kernels.  Measured on 35 × 29 × 21 voxels, 50 frames, 7³ patches at
// stride 4: extraction 48 -> 15 us, recombination 35 -> 17; recombination of
// 6³ patches at stride 3 of 48 × 48 × 32 × 128 (0.5 GB of patches): 302 -> 123 us.
#include <algorithm>

#include "internal.h"
#include "patchmap.cuh"

namespace mslr {

namespace {

constexpr int kFrames = 8;

// Patches along one axis that cover coordinate c, [lo, hi], empty when lo > hi
// (a stride above the patch size leaves gaps): starts are i·ss, the last one
// is at most n − ps.
__device__ __forceinline__ int2 covering(int c, int n, int ps, int ss, int cnt) {
  const int hi = c >= n - ps ? cnt - 1 : c / ss;
  const int lo = c < ps ? 0 : min((c - ps) / ss + 1, cnt - 1);
  return patch_start(lo, ss, n, ps) + ps > c ? make_int2(lo, hi) : make_int2(0, -1);
}

struct Cover {
  int x, y, z;
  int2 rx, ry, rz;
  float count;   // covering patches, 0 for a voxel in a gap
};

__device__ __forceinline__ Cover cover_of(const PatchMap& m, int64_t v) {
  Cover c;
  const int64_t r = v / m.Nx;
  c.x = (int)(v - r * m.Nx);
  c.z = (int)(r / m.Ny);
  c.y = (int)(r - (int64_t)c.z * m.Ny);
  c.rx = covering(c.x, m.Nx, m.psx, m.ssx, m.nx);
  c.ry = covering(c.y, m.Ny, m.psy, m.ssy, m.ny);
  c.rz = covering(c.z, m.Nz, m.psz, m.ssz, m.nz);
  c.count = (float)max(c.rx.y - c.rx.x + 1, 0) * (float)max(c.ry.y - c.ry.x + 1, 0) *
            (float)max(c.rz.y - c.rz.x + 1, 0);
  return c;
}

// img2patches: P[(ip*Nt + t)*p + l] = img[t][vox(ip, l)].
// grid (Np · ceil(p / threads), groups of frames), from block `first` on
__global__ void __launch_bounds__(256) k_img2patches(const cf* __restrict__ img, const PatchMap m,
                                                     cf* __restrict__ P, int lblocks, int64_t first) {
  const int64_t b = first + blockIdx.x, ip = b / lblocks;
  const int l = (int)(b - ip * lblocks) * blockDim.x + threadIdx.x;
  if (l >= m.p) return;
  const cf* src = img + patch_origin(m, ip) + patch_off(m, l);
  cf* dst = P + ip * m.Nt * (int64_t)m.p + l;
  for (int t0 = blockIdx.y * kFrames; t0 < m.Nt; t0 += gridDim.y * kFrames) {
    cf v[kFrames];
#pragma unroll
    for (int i = 0; i < kFrames; ++i)
      if (t0 + i < m.Nt) v[i] = src[(t0 + i) * m.nvox];
#pragma unroll
    for (int i = 0; i < kFrames; ++i)
      if (t0 + i < m.Nt) dst[(t0 + i) * (int64_t)m.p] = v[i];
  }
}

// Sum over the covering patches in ascending ip; MEAN (patches2img) divides
// by their Float32 count, clamped to 1 (src/recon.jl:113-124); without it the
// adjoint of img2patches.  Voxels in gaps get 0.  grid (voxels, groups of frames)
template <bool MEAN>
__global__ void __launch_bounds__(256) k_recombine(const cf* __restrict__ P, const PatchMap m,
                                                   cf* __restrict__ img) {
  const int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (v >= m.nvox) return;
  const Cover c = cover_of(m, v);
  const float cnt = fmaxf(c.count, 1.f);
  for (int t0 = blockIdx.y * kFrames; t0 < m.Nt; t0 += gridDim.y * kFrames) {
    cf acc[kFrames];
#pragma unroll
    for (int i = 0; i < kFrames; ++i) acc[i] = make_float2(0.f, 0.f);
    for (int iz = c.rz.x; iz <= c.rz.y; ++iz) {
      const int lz = c.z - patch_start(iz, m.ssz, m.Nz, m.psz);
      for (int iy = c.ry.x; iy <= c.ry.y; ++iy) {
        const int ly = c.y - patch_start(iy, m.ssy, m.Ny, m.psy);
        for (int ix = c.rx.x; ix <= c.rx.y; ++ix) {
          const int lx = c.x - patch_start(ix, m.ssx, m.Nx, m.psx);
          const int64_t ip = ix + (int64_t)m.nx * (iy + (int64_t)m.ny * iz);
          const cf* src = P + (ip * m.Nt + t0) * (int64_t)m.p + lx + m.psx * (ly + m.psy * lz);
          if (t0 + kFrames <= m.Nt) {
#pragma unroll
            for (int i = 0; i < kFrames; ++i) acc[i] = cadd(acc[i], src[i * (int64_t)m.p]);
          } else {
#pragma unroll
            for (int i = 0; i < kFrames; ++i)
              if (t0 + i < m.Nt) acc[i] = cadd(acc[i], src[i * (int64_t)m.p]);
          }
        }
      }
    }
#pragma unroll
    for (int i = 0; i < kFrames; ++i)
      if (t0 + i < m.Nt)
        img[(t0 + i) * m.nvox + v] = MEAN ? make_float2(acc[i].x / cnt, acc[i].y / cnt) : acc[i];
  }
}

// out = img / max(count, 1): the adjoint of patches2img's averaging, before the gather
__global__ void __launch_bounds__(256) k_div_count(const cf* __restrict__ img, const PatchMap m,
                                                   cf* __restrict__ out) {
  const int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (v >= m.nvox) return;
  const float cnt = fmaxf(cover_of(m, v).count, 1.f);
  for (int t0 = blockIdx.y * kFrames; t0 < m.Nt; t0 += gridDim.y * kFrames)
#pragma unroll
    for (int i = 0; i < kFrames; ++i)
      if (t0 + i < m.Nt) {
        const cf a = img[(t0 + i) * m.nvox + v];
        out[(t0 + i) * m.nvox + v] = make_float2(a.x / cnt, a.y / cnt);
      }
}

unsigned frame_groups(const PatchMap& m) {
  return (unsigned)std::min((m.Nt + kFrames - 1) / kFrames, 65535);
}

dim3 voxel_grid(const PatchMap& m) { return dim3((unsigned)((m.nvox + 255) / 256), frame_groups(m)); }

}  // namespace

int img2patches_launch(const cf* img, const PatchMap& m, int64_t np, cf* P, cudaStream_t st) {
  const int thr = std::min(256, (m.p + 31) / 32 * 32);
  const int lblocks = (m.p + thr - 1) / thr;
  const int64_t blocks = np * lblocks, most = 0x7fffffff;   // what the grid's first dimension holds
  for (int64_t b = 0; b < blocks; b += most) {
    const dim3 grid((unsigned)std::min(blocks - b, most), frame_groups(m));
    k_img2patches<<<grid, thr, 0, st>>>(img, m, P, lblocks, b);
    MSLR_CUDA_TRY(cudaGetLastError());
  }
  return MSLR_OK;
}

int patches2img_launch(const cf* P, const PatchMap& m, cf* img, cudaStream_t st) {
  k_recombine<true><<<voxel_grid(m), 256, 0, st>>>(P, m, img);
  MSLR_CUDA_TRY(cudaGetLastError());
  return MSLR_OK;
}

int patch_sum_launch(const cf* P, const PatchMap& m, cf* img, cudaStream_t st) {
  k_recombine<false><<<voxel_grid(m), 256, 0, st>>>(P, m, img);
  MSLR_CUDA_TRY(cudaGetLastError());
  return MSLR_OK;
}

int div_count_launch(const cf* img, const PatchMap& m, cf* out, cudaStream_t st) {
  k_div_count<<<voxel_grid(m), 256, 0, st>>>(img, m, out);
  MSLR_CUDA_TRY(cudaGetLastError());
  return MSLR_OK;
}

// Geometry of a scale from the requested patch sizes and strides (src/recon.jl:54-72).
int geom_build(const int N[3], int Nt, const int ps_in[3], const int ss_in[3], ScaleGeom* g) {
  int64_t Np = 1;
  g->h_starts.clear();
  bool partition = true;
  for (int d = 0; d < 3; ++d) {
    if (ps_in[d] <= 0 || ss_in[d] <= 0)
      return fail(MSLR_ERR_ARG, "patch sizes and strides must be positive");
    g->ps[d] = std::min(ps_in[d], N[d]);
    g->ss[d] = ss_in[d];
    // 64-bit: a stride may be anything up to 2^31 - 1
    const int64_t num = N[d] - g->ps[d], ss = g->ss[d];
    g->nsteps[d] = (int)((num + ss - 1) / ss);   // cld for num >= 0
    Np *= (g->nsteps[d] + 1);
    int prev = -1;
    for (int i = 0; i <= g->nsteps[d]; ++i) {
      const int s = (int)std::min(i * ss, num);
      g->h_starts.push_back(s);
      if (i == 0 && s != 0) partition = false;
      if (i > 0 && s - prev != g->ps[d]) partition = false;
      prev = s;
    }
    if (prev + g->ps[d] != N[d]) partition = false;
  }
  g->Np = Np;
  g->p = g->ps[0] * g->ps[1] * g->ps[2];
  g->n = std::min(g->p, Nt);
  g->L = std::max(g->p, Nt);
  g->tall = g->p >= Nt;
  g->partition = partition;
  g->global = (Np == 1 && g->ps[0] == N[0] && g->ps[1] == N[1] && g->ps[2] == N[2]);
  return MSLR_OK;
}

}  // namespace mslr
