// Weight refresh in a handful of launches, optionally fused with the optimizer step.
//
// The reference keeps fp32 masters and a flat fp16 replica that ONE cast kernel refreshes after every
// optimizer step (flat_refresh, python/fp16_linear.py:236-246; the trainer bumps the weights version
// after opt.step(), python/train_batch.py:2847-2854).  Here the replica is the packed arena, whose
// matrices are stacked, K-padded and -- for the fused attention kernel -- regrouped, so a refresh is a
// scatter: every master has a primary destination and possibly a few row ranges with a second one.
//
// multi_pack_kernel does that scatter for up to kMaxSegs masters per launch (the segment table travels
// by value in the kernel parameters: no device-side table, no host-to-device copy), and, when a master
// comes with a gradient, first applies an Adam / AdamW step to it in place:
//
//   g' = g * inv_scale;  p *= 1 - lr wd;  m = b1 m + (1 - b1) g';  v = b2 v + (1 - b2) g'^2
//   p -= (lr / (1 - b1^t)) m / (sqrt(v) / sqrt(1 - b2^t) + eps)        (torch.optim.AdamW)
//
// so the fp16 arena is produced by the optimizer kernel itself and no separate refresh pass runs.  In additive
// mode (step = 0 with gradients given) the "gradient" is an update direction and the step is p = p (1 - lr wd) + lr u: the last
// stage of an optimizer whose direction is computed elsewhere (the Muon half of the reference's hybrid optimizer
// orthogonalises its momentum with a chain of small matrix products first, python/train_batch.py:818-931; muon.cu).
#include <string.h>

#include "kernels.cuh"
#include "layout.h"

namespace bsrl {
namespace {

// Segments of one launch: the table is a kernel parameter (32,764 bytes at most), so that nearly every model's refresh
// is ONE launch (130-200 masters; it was nine launches of 20 masters, 94 us, at d = 256 and four blocks).
constexpr int kMaxSegs = 240;
constexpr int kBlockElems = 2048;     // elements per block: 256 threads, two 16-byte pieces each

struct Seg {
  float* p;                // master (rows, cols) f32
  const float* g;          // gradient, or nullptr: no update, scatter only
  float* m;                // exp_avg
  float* v;                // exp_avg_sq
  int64_t dst, dst2;       // primary and second (regrouped) destination in the arena (bytes)
  int n, cols;             // elements, elements per row (vectors: one row)
  int pitch, pitch2;       // fp16 matrices: elements per destination row; fp32 vectors: 0
  int group, gstride;      // second destination: row r -> (r / group) * gstride + r % group; group 0: none
  float lr, wd;
  int blk0;                // first block of this segment
  int vec;                 // 16-byte accesses are possible throughout
};
struct Table {
  Seg seg[kMaxSegs];
  int n_seg;
  float beta1, beta2, eps, bc1, rsqrt_bc2;   // bias corrections 1 - b1^t and 1 / sqrt(1 - b2^t)
  const float* inv_scale;                    // device scalar multiplying every gradient, or nullptr
  const float* found_inf;                    // device scalar: non-zero = skip every update (scatter still runs)
  int additive;                              // the gradients are update directions: p = p (1 - lr wd) + lr g
};
static_assert(sizeof(Table) + 16 <= 32764, "kernel parameter limit");

// one element's update; true when the master changes
struct Updater {
  float beta1, beta2, eps, rsqrt_bc2, inv_scale, step, decay, lr;
  bool additive;
  __device__ __forceinline__ float adam(float p, float g_in, float& m, float& v) const {
    const float g = g_in * inv_scale;
    m = beta1 * m + (1.f - beta1) * g;
    v = beta2 * v + (1.f - beta2) * g * g;
    return p * decay - step * m / (sqrtf(v) * rsqrt_bc2 + eps);
  }
  __device__ __forceinline__ float add(float p, float u) const { return fmaf(lr, u, p * decay); }
};

__device__ __forceinline__ void put(const Seg& s, uint8_t* arena, int r, int c, float val) {
  if (s.pitch) reinterpret_cast<__half*>(arena + s.dst)[(int64_t)r * s.pitch + c] = __float2half_rn(val);
  else reinterpret_cast<float*>(arena + s.dst)[c] = val;
  if (s.group) {
    const int row = s.pitch ? r : c;       // a vector's elements are its rows
    const int row2 = (row / s.group) * s.gstride + row % s.group;
    if (s.pitch) reinterpret_cast<__half*>(arena + s.dst2)[(int64_t)row2 * s.pitch2 + c] = __float2half_rn(val);
    else reinterpret_cast<float*>(arena + s.dst2)[row2] = val;
  }
}

// Bound by the masters', gradients' and moments' traffic once the launch is large enough to fill the GPU: every block
// takes kBlockElems consecutive elements of one segment (found by bisection over the segments' first blocks), so small
// vectors cost one block each and a large matrix is spread over as many as it has pieces.
__global__ void __launch_bounds__(256) multi_pack_kernel(const __grid_constant__ Table t, uint8_t* __restrict__ arena) {
  int lo = 0, hi = t.n_seg - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (t.seg[mid].blk0 <= (int)blockIdx.x) lo = mid; else hi = mid - 1;
  }
  const Seg& s = t.seg[lo];
  const bool update = s.g != nullptr && !(t.found_inf && *t.found_inf != 0.f);
  Updater u;
  u.beta1 = t.beta1; u.beta2 = t.beta2; u.eps = t.eps; u.rsqrt_bc2 = t.rsqrt_bc2;
  u.inv_scale = (update && t.inv_scale) ? *t.inv_scale : 1.f;
  u.step = s.lr / t.bc1; u.decay = 1.f - s.lr * s.wd; u.lr = s.lr;
  u.additive = t.additive != 0;
  const int i0 = ((int)blockIdx.x - s.blk0) * kBlockElems, i1 = min(s.n, i0 + kBlockElems);
  if (s.vec) {
#pragma unroll
    for (int k = 0; k < kBlockElems / 1024; ++k) {
      const int i = i0 + k * 1024 + threadIdx.x * 4;
      if (i >= i1) break;
      float4 p = *reinterpret_cast<const float4*>(s.p + i);
      if (update) {
        const float4 g = *reinterpret_cast<const float4*>(s.g + i);
        if (u.additive) {
          p = make_float4(u.add(p.x, g.x), u.add(p.y, g.y), u.add(p.z, g.z), u.add(p.w, g.w));
        } else {
          float4 m = *reinterpret_cast<const float4*>(s.m + i), v = *reinterpret_cast<const float4*>(s.v + i);
          p = make_float4(u.adam(p.x, g.x, m.x, v.x), u.adam(p.y, g.y, m.y, v.y), u.adam(p.z, g.z, m.z, v.z),
                          u.adam(p.w, g.w, m.w, v.w));
          *reinterpret_cast<float4*>(s.m + i) = m;
          *reinterpret_cast<float4*>(s.v + i) = v;
        }
        *reinterpret_cast<float4*>(s.p + i) = p;
      }
      if (s.pitch) {                         // matrix: cols, pitches and offsets are multiples of four
        const int r = i / s.cols, c = i - r * s.cols;
        const uint2 h = make_uint2(pack_half2(p.x, p.y), pack_half2(p.z, p.w));
        *reinterpret_cast<uint2*>(arena + s.dst + ((int64_t)r * s.pitch + c) * 2) = h;
        if (s.group) {
          const int row2 = (r / s.group) * s.gstride + r % s.group;
          *reinterpret_cast<uint2*>(arena + s.dst2 + ((int64_t)row2 * s.pitch2 + c) * 2) = h;
        }
      } else {
        const float e[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) put(s, arena, 0, i + j, e[j]);
      }
    }
    return;
  }
  for (int i = i0 + threadIdx.x; i < i1; i += 256) {
    float p = s.p[i];
    if (update) {
      if (u.additive) {
        p = u.add(p, s.g[i]);
      } else {
        float m = s.m[i], v = s.v[i];
        p = u.adam(p, s.g[i], m, v);
        s.m[i] = m;
        s.v[i] = v;
      }
      s.p[i] = p;
    }
    const int r = i / s.cols;
    put(s, arena, r, i - r * s.cols, p);
  }
}

}  // namespace

int multi_pack(const bsrl_config& cfg, const Layout& l, float* const* params, const float* const* grads,
               float* const* exp_avg, float* const* exp_avg_sq, const float* lr, const float* wd, float beta1,
               float beta2, float eps, int step, const float* inv_scale, const float* found_inf, void* arena,
               cudaStream_t stream) {
  const Plan& plan = plan_of(cfg);
  return multi_pack_slots(plan.slots, plan.copies, params, grads, exp_avg, exp_avg_sq, lr, wd, beta1, beta2, eps, step,
                          inv_scale, found_inf, arena, stream);
}

int multi_pack_slots(const std::vector<ParamSlot>& slots, const std::vector<CopySlot>& copies, float* const* params,
                     const float* const* grads, float* const* exp_avg, float* const* exp_avg_sq, const float* lr,
                     const float* wd, float beta1, float beta2, float eps, int step, const float* inv_scale,
                     const float* found_inf, void* arena, cudaStream_t stream) {
  Table t;
  memset(&t, 0, sizeof(t));
  t.beta1 = beta1; t.beta2 = beta2; t.eps = eps;
  t.bc1 = step > 0 ? 1.f - powf(beta1, (float)step) : 1.f;
  t.rsqrt_bc2 = step > 0 ? 1.f / sqrtf(1.f - powf(beta2, (float)step)) : 1.f;
  t.inv_scale = inv_scale;
  t.found_inf = found_inf;
  t.additive = (step == 0 && grads != nullptr) ? 1 : 0;
  std::vector<const CopySlot*> second(slots.size(), nullptr);
  for (const CopySlot& cs : copies) second[cs.param] = &cs;
  int blocks = 0;
  auto flush = [&]() -> int {
    if (t.n_seg == 0) return BSRL_OK;
    multi_pack_kernel<<<(unsigned)blocks, 256, 0, stream>>>(t, static_cast<uint8_t*>(arena));
    BSRL_LAUNCH_OK("multi_pack_kernel");
    t.n_seg = 0;
    blocks = 0;
    return BSRL_OK;
  };
  for (size_t i = 0; i < slots.size(); ++i) {
    const ParamSlot& ps = slots[i];
    if (t.n_seg == kMaxSegs) {
      int rc = flush();
      if (rc != BSRL_OK) return rc;
    }
    Seg& s = t.seg[t.n_seg++];
    s.p = params[i];
    s.g = grads ? grads[i] : nullptr;
    s.m = (s.g && exp_avg) ? exp_avg[i] : nullptr;
    s.v = (s.g && exp_avg_sq) ? exp_avg_sq[i] : nullptr;
    if (s.g && !t.additive && (!s.m || !s.v)) {
      set_error("adam_step_pack: parameter %s has a gradient but no optimizer state", ps.name.c_str());
      return BSRL_ERR_NULL;
    }
    s.n = (int)(ps.rows * ps.cols);
    s.cols = ps.half ? (int)ps.cols : s.n;
    s.dst = ps.dst;
    s.pitch = ps.half ? (int)ps.dst_pitch : 0;
    s.group = s.gstride = s.pitch2 = 0;
    s.dst2 = 0;
    if (const CopySlot* cs = second[i]) {
      s.group = cs->group_rows; s.gstride = cs->group_stride;
      s.dst2 = cs->dst; s.pitch2 = (int)cs->dst_pitch;
    }
    s.lr = lr ? lr[i] : (t.additive ? 1.f : 0.f);
    s.wd = wd ? wd[i] : 0.f;
    // 16-byte pieces: a piece must not cross a matrix row, and 8-byte fp16 stores need pitches of four elements
    s.vec = s.n % 4 == 0 && aligned16(s.p) && (!s.g || aligned16(s.g)) && (!s.m || aligned16(s.m)) && (!s.v || aligned16(s.v)) &&
            (!ps.half || (ps.cols % 4 == 0 && s.pitch % 4 == 0 && s.pitch2 % 4 == 0 && s.dst % 8 == 0 && s.dst2 % 8 == 0));
    s.blk0 = blocks;
    blocks += (s.n + kBlockElems - 1) / kBlockElems;
  }
  return flush();
}

}  // namespace bsrl
