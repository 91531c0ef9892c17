// Generic CUDA-core forward: any dtype (bf16 / fp16 / fp32), any headdim <= 256, any strides,
// any softmax scale.  It covers the corners of the reference's test grid that the tensor-core
// kernel does not take (test/test_accuracy.py:24,28: fp32 inputs, headdim 18) and is the
// second, independently written implementation the tensor-core kernel is cross-checked against.
//
// One CTA = 32 or 64 query rows of one (q-block, q-head); four threads share a row, or a pair of rows 32 apart, and split
// the head dimension (thread s owns dims 16 j + 4 s ... 16 j + 4 s + 3).  K/V tiles of the active k-blocks are
// staged in shared memory as fp32; scores, online softmax and the output accumulate in fp32
// registers (the arithmetic of fwd_triton_fix_tile_size.py:157-192 without the bf16 rounding of P).
//
// Bound by the latency of staging K and V, then by FMAs and shared-memory reads along the keys of the longest rows.  fp32, d = 64,
// 4 samples of 200 to 1500 tokens, 8 heads: one row and single floats per thread (a shared-memory read for every FMA) 237 us a call;
// four dims per read and two rows per value (a read for eight FMAs) 227 us; staging loads in batches of eight as well 168 us (151 us in the final build).
#include "hbsa_common.cuh"

namespace hbsa {

template <typename T> __device__ __forceinline__ float load_f(const T* p);
template <> __device__ __forceinline__ float load_f<float>(const float* p) { return *p; }
template <> __device__ __forceinline__ float load_f<__half>(const __half* p) { return __half2float(*p); }
template <> __device__ __forceinline__ float load_f<__nv_bfloat16>(const __nv_bfloat16* p) { return __bfloat162float(*p); }

template <typename T> __device__ __forceinline__ void store_f(T* p, float x);
template <> __device__ __forceinline__ void store_f<float>(float* p, float x) { *p = x; }
template <> __device__ __forceinline__ void store_f<__half>(__half* p, float x) { *p = __float2half_rn(x); }
template <> __device__ __forceinline__ void store_f<__nv_bfloat16>(__nv_bfloat16* p, float x) { *p = __float2bfloat16_rn(x); }

struct Strides { long long q0, q1, q2, k0, k1, k2, v0, v1, v2, o0, o1, o2; };

constexpr int kRowGroups = 32;     // groups of four threads in a CTA, each with ROWS rows

template <typename T, int DQ, int KT, int ROWS>
__global__ void __launch_bounds__(128)
fwd_generic_kernel(Problem p, Workspace ws, const T* __restrict__ q, const T* __restrict__ k,
                   const T* __restrict__ v, T* __restrict__ o, float* __restrict__ lse, Strides st, int chunks_per_block,
                   int total_q) {
  constexpr int DPAD = DQ * 4;
  static_assert(KT * DPAD % (128 * 8) == 0, "staging in whole batches");
  if (ws.status[0] != HBSA_STATUS_OK) {
    zero_fill_output(o, st.o0, st.o1, st.o2, total_q, p.nhead_q, p.headdim, lse);
    return;
  }
  constexpr int kRowsPerCta = kRowGroups * ROWS;
  extern __shared__ __align__(16) float smem[];
  float* sK = smem;                  // [KT][DPAD]
  float* sV = smem + KT * DPAD;      // [KT][DPAD]

  const int qb = blockIdx.x / chunks_per_block;
  const int chunk = blockIdx.x % chunks_per_block;
  const int hq = blockIdx.y;
  const int hk = hq / p.group;
  const RowGeom g = row_geometry(p, ws.cnq, ws.cnk, ws.qb2b, qb);
  const int row0 = g.q_begin + chunk * kRowsPerCta;
  if (row0 >= g.q_end) return;

  const int tid = threadIdx.x;
  const int r = tid >> 2, sub = tid & 3;
  const float scale_log2 = p.scale * 1.4426950408889634f;

  // dim of a thread's element i
  auto dim_of = [sub](int i) { return 16 * (i >> 2) + 4 * sub + (i & 3); };
  float qreg[ROWS][DQ], acc[ROWS][DQ], m[ROWS], l[ROWS];
  int limit_row[ROWS];
#pragma unroll
  for (int w = 0; w < ROWS; ++w) {
    const int tok = row0 + r + w * kRowGroups;
#pragma unroll
    for (int i = 0; i < DQ; ++i) {
      const int d = dim_of(i);
      qreg[w][i] = (tok < g.q_end && d < p.headdim) ? load_f(q + tok * st.q0 + hq * st.q1 + d * st.q2) * scale_log2 : 0.f;
      acc[w][i] = 0.f;
    }
    m[w] = -INFINITY;
    l[w] = 0.f;
    limit_row[w] = g.k_len - 1;
    if (p.causal) limit_row[w] = min(limit_row[w], g.q_in0 + (tok - g.q_begin) + g.off);
  }

  // Active k-blocks of the row, in ascending order: bytes of the dense mask row, or the entries of the CSR row that
  // lie in the row's own sample below the causal reach.
  const bool csr = p.csr_ptr != nullptr;
  const uint8_t* mrow = csr ? nullptr : p.mask + hk * p.mask_s0 + qb * p.mask_s1;
  int e_begin = 0, n_src = g.n_reach;
  if (csr) {
    const long long row = (long long)hk * p.num_q_block + qb;
    const int e0 = p.csr_ptr[row], e1 = p.csr_ptr[row + 1];
    e_begin = lower_bound_i32(p.csr_idx, e0, e1, g.kb0);
    n_src = lower_bound_i32(p.csr_idx, e_begin, e1, g.kb0 + g.n_reach) - e_begin;
  }
  for (int e = 0; e < n_src; ++e) {
    int j = e;
    if (csr) j = p.csr_idx[e_begin + e] - g.kb0;
    else if (mrow[(long long)(g.kb0 + j) * p.mask_s2] == 0) continue;  // uniform over the CTA
    const int blk_k0 = j * p.kbs;
    const int blk_len = min(p.kbs, g.k_len - blk_k0);
    for (int t0 = 0; t0 < blk_len; t0 += KT) {
      const int nk = min(KT, blk_len - t0);
      __syncthreads();
      // eight loads of each in flight per thread: one after the other they cost a memory latency apiece
      for (int idx0 = tid; idx0 < KT * DPAD; idx0 += 128 * 8) {
        float kv[8], vv[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int key = (idx0 + 128 * i) / DPAD, d = (idx0 + 128 * i) % DPAD;
          kv[i] = vv[i] = 0.f;
          if (key < nk && d < p.headdim) {
            const long long ktok = g.k_begin + blk_k0 + t0 + key;
            kv[i] = load_f(k + ktok * st.k0 + hk * st.k1 + d * st.k2);
            vv[i] = load_f(v + ktok * st.v0 + hk * st.v1 + d * st.v2);
          }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          sK[idx0 + 128 * i] = kv[i];
          sV[idx0 + 128 * i] = vv[i];
        }
      }
      __syncthreads();
      const int key_base = blk_k0 + t0;
      for (int kk = 0; kk < nk; kk += 8) {
        float s[ROWS][8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const float4* kr = reinterpret_cast<const float4*>(sK + (kk + u) * DPAD) + sub;
          float part[ROWS] = {};
#pragma unroll
          for (int j = 0; j < DQ / 4; ++j) {
            const float4 x = kr[4 * j];
#pragma unroll
            for (int w = 0; w < ROWS; ++w) {
              part[w] = fmaf(qreg[w][4 * j], x.x, part[w]);
              part[w] = fmaf(qreg[w][4 * j + 1], x.y, part[w]);
              part[w] = fmaf(qreg[w][4 * j + 2], x.z, part[w]);
              part[w] = fmaf(qreg[w][4 * j + 3], x.w, part[w]);
            }
          }
#pragma unroll
          for (int w = 0; w < ROWS; ++w) {
            part[w] += __shfl_xor_sync(0xffffffffu, part[w], 1);
            part[w] += __shfl_xor_sync(0xffffffffu, part[w], 2);
            const bool allowed = (kk + u < nk) && (key_base + kk + u <= limit_row[w]);
            s[w][u] = allowed ? part[w] : -INFINITY;
          }
        }
#pragma unroll
        for (int w = 0; w < ROWS; ++w) {
          float mx = s[w][0];
#pragma unroll
          for (int u = 1; u < 8; ++u) mx = fmaxf(mx, s[w][u]);
          const float m_new = fmaxf(m[w], mx);
          const float m_use = m_new == -INFINITY ? 0.f : m_new;
          const float alpha = exp2f(m[w] - m_use);
          float psum = 0.f;
#pragma unroll
          for (int u = 0; u < 8; ++u) { s[w][u] = exp2f(s[w][u] - m_use); psum += s[w][u]; }
          l[w] = l[w] * alpha + psum;
          m[w] = m_new;
#pragma unroll
          for (int i = 0; i < DQ; ++i) acc[w][i] *= alpha;
        }
#pragma unroll
        for (int j = 0; j < DQ / 4; ++j) {
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            const float4 x = (reinterpret_cast<const float4*>(sV + (kk + u) * DPAD) + sub)[4 * j];
#pragma unroll
            for (int w = 0; w < ROWS; ++w) {
              acc[w][4 * j] = fmaf(s[w][u], x.x, acc[w][4 * j]);
              acc[w][4 * j + 1] = fmaf(s[w][u], x.y, acc[w][4 * j + 1]);
              acc[w][4 * j + 2] = fmaf(s[w][u], x.z, acc[w][4 * j + 2]);
              acc[w][4 * j + 3] = fmaf(s[w][u], x.w, acc[w][4 * j + 3]);
            }
          }
        }
      }
    }
  }
#pragma unroll
  for (int w = 0; w < ROWS; ++w) {
    const int tok = row0 + r + w * kRowGroups;
    if (tok >= g.q_end) continue;
    const float inv = l[w] > 0.f ? 1.f / l[w] : 0.f;      // rows that see no key are exact zeros
#pragma unroll
    for (int i = 0; i < DQ; ++i) {
      const int d = dim_of(i);
      if (d < p.headdim) store_f(o + tok * st.o0 + hq * st.o1 + d * st.o2, acc[w][i] * inv);
    }
    // scores are kept in the log2 domain: ln sum exp = ln 2 * (m + log2 l)
    if (lse != nullptr && sub == 0) lse[(long long)tok * p.nhead_q + hq] = l[w] > 0.f ? 0.6931471805599453f * (m[w] + log2f(l[w])) : -INFINITY;
  }
}

template <typename T>
static cudaError_t launch_typed(const Problem& p, const Workspace& ws, const hbsa_forward_args& a, cudaStream_t stream) {
  Strides st{a.q_stride[0], a.q_stride[1], a.q_stride[2], a.k_stride[0], a.k_stride[1], a.k_stride[2],
             a.v_stride[0], a.v_stride[1], a.v_stride[2], a.o_stride[0], a.o_stride[1], a.o_stride[2]};
  const T* q = static_cast<const T*>(a.q);
  const T* k = static_cast<const T*>(a.k);
  const T* v = static_cast<const T*>(a.v);
  T* o = static_cast<T*>(a.o);
  // Two rows a thread where a q-block has rows for them; above 128 dims their Q and O do not fit a thread's registers.
  const int rows = (p.qbs > kRowGroups && p.headdim <= 128 ? 2 : 1) * kRowGroups;
  const int cpb = (p.qbs + rows - 1) / rows;
  dim3 grid((unsigned)((long long)p.num_q_block * cpb), (unsigned)p.nhead_q);
#define HBSA_LAUNCH_GENERIC(DQ_, KT_, ROWS_)                                                            \
  fwd_generic_kernel<T, DQ_, KT_, ROWS_><<<grid, 128, 2 * KT_ * DQ_ * 4 * sizeof(float), stream>>>(p, ws, q, k, v, o, a.lse, st, cpb, a.total_q)
#define HBSA_LAUNCH_ROWS(DQ_) do { if (rows > kRowGroups) HBSA_LAUNCH_GENERIC(DQ_, 32, 2); else HBSA_LAUNCH_GENERIC(DQ_, 32, 1); } while (0)
  if (p.headdim <= 32) HBSA_LAUNCH_ROWS(8);
  else if (p.headdim <= 64) HBSA_LAUNCH_ROWS(16);
  else if (p.headdim <= 128) HBSA_LAUNCH_ROWS(32);
  else HBSA_LAUNCH_GENERIC(64, 16, 1);
#undef HBSA_LAUNCH_ROWS
#undef HBSA_LAUNCH_GENERIC
  return cudaGetLastError();
}

cudaError_t launch_forward_generic(const Problem& p, const Workspace& ws, const hbsa_forward_args& a,
                                   cudaStream_t stream) {
  switch (a.dtype) {
    case HBSA_DTYPE_BF16: return launch_typed<__nv_bfloat16>(p, ws, a, stream);
    case HBSA_DTYPE_F16: return launch_typed<__half>(p, ws, a, stream);
    default: return launch_typed<float>(p, ws, a, stream);
  }
}

}  // namespace hbsa
