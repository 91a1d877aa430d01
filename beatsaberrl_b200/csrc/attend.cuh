// Attention of one (env, head) pair from a q|k|v tile in shared memory: device functions shared by the fused
// projection + attention kernels.
#pragma once
#include "common.cuh"

namespace bsrl {
__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rcp_approx(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Byte offset of 16-byte piece p of row r of a tile of dense rows: the 8 rows of an ldmatrix hit 8 different 16-byte banks,
// and so do 8 consecutive pieces (with rows padded by 16 bytes instead, those took two turns of the pipe).
template <int DH>
__device__ __forceinline__ uint32_t tile_at(int r, int p) {
  return r * (DH * 2) + ((DH == 32 ? p ^ ((r >> 1) & 3) : DH == 48 ? p ^ ((r >> 2) & 1) : p ^ (r & 7)) << 4);
}

// Byte address of 16-byte piece `piece` of row `row` of a section (q, k or v): rows LDQ bytes apart, or, for LDQ = 128, a
// 128-byte-swizzled tile (piece p of row r at ((p ^ (r & 7)) << 4)) that starts on a 1024-byte boundary
template <int LDQ>
__device__ __forceinline__ uint32_t section_at(uint32_t base, int row, int piece) {
  return LDQ == 128 ? base + row * 128 + ((piece ^ (row & 7)) << 4) : base + row * LDQ + (piece << 4);
}

// Attention of one (env, head) pair from the shared q|k|v tile; one warp.  sq, sk, sv: byte addresses (shared window) of
// the env's first row in the three sections; query rows from q_row0, the head's columns from 16-byte piece piece0.
// The MT 16-row query tiles are processed side by side: two independent dependency chains per warp
// (the kernel is latency-bound here) and each K / V fragment is fetched once for both.
// OB: bytes per row of the staged group output (128: two heads of 32, swizzled; 96: one head of 48, dense)
// BODY: one more key outside the tile (the body token): x_lane = q_row . k_0 for row `lane` (raw), kb0 its
// base-2 key bias, v0 its DH values (shared memory, generic pointer); its score joins each row's softmax and its
// probability times v_0 starts the row's output.
// PACK: the env's keys are the n_keys rows from k_row0 of a tile of 128, in KT tiles of 16; what the last one holds beyond them
// belongs to other environments and must not show, whatever it is: its scores are replaced, its v rows cleared.  Chunks
// of keys that are left out would have added exact zeros.
template <int MT, int DH, int LDQ, int OB, bool BODY = false, bool PACK = false, int KT = 2>
__device__ __forceinline__ void attend_pair(uint32_t sq, uint32_t sk, uint32_t sv, int q_row0, int piece0, const float (&kb)[4][2],
                                            int n_q, __half* out_env, int ldo, int lane, uint8_t* so, int so_row0, int so_piece0,
                                            float x_lane = 0.f, float kb0 = 0.f, const __half* v0 = nullptr, int k_row0 = 0, int n_keys = 32) {
  const int g = lane >> 2, tig = lane & 3;
  auto in_tile = [](int row) { return PACK ? min(row, 127) : row; };
  const float scale = rsqrtf((float)DH) * 1.4426950408889634f;   // 1/sqrt(dh) * log2(e)
  float s[MT][2 * KT][4];
#pragma unroll
  for (int mt = 0; mt < MT; ++mt)
#pragma unroll
    for (int nt = 0; nt < 2 * KT; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) s[mt][nt][e] = 0.f;
#pragma unroll
  for (int ks = 0; ks < DH / 16; ++ks) {
    uint32_t a[MT][4];
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
      ldmatrix_x4(a[mt], section_at<LDQ>(sq, in_tile(q_row0 + mt * 16 + (lane & 15)), piece0 + ks * 2 + (lane >> 4)));
#pragma unroll
    for (int j = 0; j < KT; ++j) {
      uint32_t b[4];
      const int row = in_tile(k_row0 + j * 16 + (lane & 7) + ((lane >> 4) << 3));
      ldmatrix_x4(b, section_at<LDQ>(sk, row, piece0 + ks * 2 + ((lane >> 3) & 1)));
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) {
        mma_f16(s[mt][2 * j], a[mt], b[0], b[1]);
        mma_f16(s[mt][2 * j + 1], a[mt], b[2], b[3]);
      }
    }
  }
  uint32_t pa[MT][KT][4];
  float p0[MT][2];                    // BODY: the body key's probability for rows g and g + 8 of each query tile
#pragma unroll
  for (int mt = 0; mt < MT; ++mt) {
    float mx[2] = {-INFINITY, -INFINITY};
    if (BODY) {
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        p0[mt][r] = fmaf(__shfl_sync(0xffffffffu, x_lane, mt * 16 + g + r * 8), scale, kb0);
        mx[r] = p0[mt][r];
      }
    }
#pragma unroll
    for (int nt = 0; nt < 2 * KT; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        s[mt][nt][e] = fmaf(s[mt][nt][e], scale, kb[nt][e & 1]);   // base-2 logits: scale and key bias carry log2(e)
        if (PACK && kb[nt][e & 1] == -INFINITY) s[mt][nt][e] = -INFINITY;
        mx[e >> 1] = fmaxf(mx[e >> 1], s[mt][nt][e]);
      }
    float sum[2] = {0.f, 0.f};
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 1));
      mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 2));
    }
#pragma unroll
    for (int nt = 0; nt < 2 * KT; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        s[mt][nt][e] = ex2_approx(s[mt][nt][e] - mx[e >> 1]);
        sum[e >> 1] += s[mt][nt][e];
      }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], 1);
      sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], 2);
      if (BODY) {
        p0[mt][r] = ex2_approx(p0[mt][r] - mx[r]);
        sum[r] = rcp_approx(sum[r] + p0[mt][r]);
        p0[mt][r] *= sum[r];
      } else {
        sum[r] = rcp_approx(sum[r]);
      }
    }
#pragma unroll
    for (int ks = 0; ks < KT; ++ks) {
      pa[mt][ks][0] = pack_half2(s[mt][2 * ks][0] * sum[0], s[mt][2 * ks][1] * sum[0]);
      pa[mt][ks][1] = pack_half2(s[mt][2 * ks][2] * sum[1], s[mt][2 * ks][3] * sum[1]);
      pa[mt][ks][2] = pack_half2(s[mt][2 * ks + 1][0] * sum[0], s[mt][2 * ks + 1][1] * sum[0]);
      pa[mt][ks][3] = pack_half2(s[mt][2 * ks + 1][2] * sum[1], s[mt][2 * ks + 1][3] * sum[1]);
    }
  }
  uint32_t live[2];                   // PACK: which of this lane's v rows of the last 16 (tig * 2, + 1; 8 further) are the env's
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int left = n_keys - (KT - 1) * 16 - tig * 2 - 8 * e;
    live[e] = left > 1 ? 0xffffffffu : left == 1 ? 0xffffu : 0u;
  }
  float o[MT][DH / 8][4];
#pragma unroll
  for (int nt = 0; nt < DH / 8; ++nt) {
    float2 v = make_float2(0.f, 0.f);
    if (BODY) v = __half22float2(*reinterpret_cast<const __half2*>(v0 + nt * 8 + tig * 2));
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
      o[mt][nt][0] = BODY ? p0[mt][0] * v.x : 0.f;
      o[mt][nt][1] = BODY ? p0[mt][0] * v.y : 0.f;
      o[mt][nt][2] = BODY ? p0[mt][1] * v.x : 0.f;
      o[mt][nt][3] = BODY ? p0[mt][1] * v.y : 0.f;
    }
  }
#pragma unroll
  for (int ks = 0; ks < KT; ++ks) {
#pragma unroll
    for (int j = 0; j < DH / 16; ++j) {
      uint32_t b[4];
      const int row = in_tile(k_row0 + ks * 16 + (lane & 7) + ((lane >> 3) & 1) * 8);
      ldmatrix_x4_trans(b, section_at<LDQ>(sv, row, piece0 + j * 2 + (lane >> 4)));
      if (PACK && ks == KT - 1) {
        b[0] &= live[0]; b[2] &= live[0];
        b[1] &= live[1]; b[3] &= live[1];
      }
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) {
        mma_f16(o[mt][2 * j], pa[mt][ks], b[0], b[1]);
        mma_f16(o[mt][2 * j + 1], pa[mt][ks], b[2], b[3]);
      }
    }
  }
#pragma unroll
  for (int mt = 0; mt < MT; ++mt)
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int qrow = mt * 16 + g + r * 8;
      if (qrow < n_q && so) {
        // staged for the group's TMA store.  128-byte rows: 16-byte piece p of row r at ((p ^ (r & 7)) << 4),
        // the 8 rows of a store instruction hit 32 different banks; 96-byte rows: dense (2-way conflicts)
        const int row = so_row0 + qrow;
        uint8_t* orow = so + row * OB + tig * 4;
#pragma unroll
        for (int nt = 0; nt < DH / 8; ++nt)
          *reinterpret_cast<uint32_t*>(orow + (OB == 128 ? (((so_piece0 + nt) ^ (row & 7)) << 4) : ((so_piece0 + nt) << 4))) =
              pack_half2(o[mt][nt][r * 2], o[mt][nt][r * 2 + 1]);
      } else if (qrow < n_q) {
        __half* orow = out_env + (int64_t)qrow * ldo + tig * 2;
#pragma unroll
        for (int nt = 0; nt < DH / 8; ++nt)
          *reinterpret_cast<uint32_t*>(orow + nt * 8) = pack_half2(o[mt][nt][r * 2], o[mt][nt][r * 2 + 1]);
      }
    }
}

// One query row of an env on the CUDA cores (lane = key for the scores, lane = output column for the weighted sum):
// row q_row of section sq (as in attend_pair, generic pointers) against the NKEYS rows of sk and sv, the head's columns
// from piece0; kb_row: this lane's key bias in base 2, -inf past the last key.  The keys are the n_keys rows from k_row0.
template <int DH, int LDQ, int NKEYS>
__device__ __forceinline__ void attend_one_row(const uint8_t* sq, const uint8_t* sk, const uint8_t* sv, int q_row, int piece0, float kb_row,
                                               __half* orow, int lane, int k_row0 = 0, int n_keys = NKEYS) {
  const int krow = k_row0 + (lane < n_keys ? lane : 0);
  float sc = 0.f;
#pragma unroll
  for (int ch = 0; ch < DH / 8; ++ch) {
    const uint4 qv = *reinterpret_cast<const uint4*>(sq + section_at<LDQ>(0, q_row, piece0 + ch));
    const uint4 kv = *reinterpret_cast<const uint4*>(sk + section_at<LDQ>(0, krow, piece0 + ch));
    const __half2* qh = reinterpret_cast<const __half2*>(&qv);
    const __half2* kh = reinterpret_cast<const __half2*>(&kv);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 a = __half22float2(qh[e]), b = __half22float2(kh[e]);
      sc = fmaf(a.x, b.x, fmaf(a.y, b.y, sc));
    }
  }
  sc = fmaf(sc, rsqrtf((float)DH) * 1.4426950408889634f, kb_row);
  const float mx = warp_max(sc);
  const float pj = ex2_approx(sc - mx);
  const float inv = rcp_approx(warp_sum(pj));
#pragma unroll
  for (int dd = 0; dd < DH; dd += 32) {
    const int col = dd + lane;
    const int vc = col < DH ? col : 0;
    float acc = 0.f;
#pragma unroll 8
    for (int j = 0; j < n_keys; ++j)
      acc = fmaf(__shfl_sync(0xffffffffu, pj, j), __half2float(*reinterpret_cast<const __half*>(sv + section_at<LDQ>(0, k_row0 + j, piece0 + (vc >> 3)) + (vc & 7) * 2)), acc);
    if (col < DH) orow[col] = __float2half_rn(acc * inv);
  }
}

}  // namespace bsrl
