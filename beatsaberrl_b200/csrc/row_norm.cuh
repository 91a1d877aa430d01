// LayerNorm of a few fp32 rows on their way to becoming an fp16 operand in shared memory, with the block tail kernel's
// statistics: each half of a row is summed in column order (one thread per half row), one of two groupings.  The same
// sums in the same order give the same bits, so a row does not depend on which kernel normalised it.
#pragma once
#include "kernels.cuh"

namespace bsrl {

// xs: rows of d floats, `pitch` floats apart (a multiple of 4, pitch / 4 odd: conflict-free); part: [2][rows]
__device__ __forceinline__ void row_norm_sums(const float* xs, int pitch, int rows, int d, bool quads, float2* part, int tid) {
  if (tid >= 2 * rows) return;
  const int row = tid < rows ? tid : tid - rows, half = tid < rows ? 0 : 1;
  const float4* v4 = reinterpret_cast<const float4*>(xs + row * pitch + half * (d >> 1));
  float sum = 0.f, sq = 0.f;
#pragma unroll 8
  for (int j = 0; j < d >> 3; ++j) {
    const float4 v = v4[j];
    if (quads) {              // as the kernel that wrote the row sums it in its drain
      sum += (v.x + v.y) + (v.z + v.w);
      sq = fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, fmaf(v.w, v.w, sq))));
    } else {                  // as it sums the rows between out-projection and FFN
      sum += v.x; sq = fmaf(v.x, v.x, sq);
      sum += v.y; sq = fmaf(v.y, v.y, sq);
      sum += v.z; sq = fmaf(v.z, v.z, sq);
      sum += v.w; sq = fmaf(v.w, v.w, sq);
    }
  }
  part[half * rows + row] = make_float2(sum, sq);
}

// eight normalised columns [c, c + 8) of a row as fp16
__device__ __forceinline__ uint4 row_norm_piece(const float* xr, int c, float2 a, float2 b, int d, const RowNorm& n) {
  const float inv_d = 1.0f / (float)d;
  const float mean = (a.x + b.x) * inv_d;
  const float rstd = rsqrtf(fmaxf((a.y + b.y) * inv_d - mean * mean, 0.f) + n.eps);
  const float shift = -mean * rstd;
  float y[8];
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const float4 v = *reinterpret_cast<const float4*>(xr + c + 4 * e);
    const float4 g = *reinterpret_cast<const float4*>(n.g + c + 4 * e), bb = *reinterpret_cast<const float4*>(n.b + c + 4 * e);
    y[4 * e] = fmaf(fmaf(v.x, rstd, shift), g.x, bb.x);
    y[4 * e + 1] = fmaf(fmaf(v.y, rstd, shift), g.y, bb.y);
    y[4 * e + 2] = fmaf(fmaf(v.z, rstd, shift), g.z, bb.z);
    y[4 * e + 3] = fmaf(fmaf(v.w, rstd, shift), g.w, bb.w);
  }
  return make_uint4(pack_half2(y[0], y[1]), pack_half2(y[2], y[3]), pack_half2(y[4], y[5]), pack_half2(y[6], y[7]));
}

}  // namespace bsrl
