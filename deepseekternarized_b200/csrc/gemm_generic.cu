// Generic ternary grouped GEMM on CUDA cores: covers every shape the C ABI accepts (any K, group,
// N, row count, 1..4 stacked terms, bf16 / f16 / int8 activations, f16 / f32 / bf16 scales).
// It is the kernel for shapes the two fast kernels do not cover (ragged K, short last group,
// group != 128) and the one the fast kernels are first validated against on the device. int8 activations with groups of
// whole 64-trit steps have a tensor-core form of their own (canonical_i8_kernel below).
//
// Work split of the plain form: one warp per output row n, eight rows per block, one block column per expert; the
// block walks its expert's token rows in tiles of TOK. Inside a scale group the lanes stride over k,
// so activation loads are coalesced and each lane keeps a partial group sum (exact int32 for int8
// activations); the lane multiplies its partial by the group scale and the warp reduces once per
// token tile. Same contract as the reference kernels
// (boilerplate/kernels/csrc/ternary_cuda_kernel.cu:44-99, boilerplate_cpu.cpp:109-127).
#include <algorithm>

#include "dst_common.cuh"

namespace dst {
namespace {

constexpr int WARPS = 8;
constexpr int TOK = 8;

template <int ACT>
struct ActT;
template <>
struct ActT<DST_ACT_BF16> { using type = __nv_bfloat16; using acc = float; };
template <>
struct ActT<DST_ACT_F16> { using type = __half; using acc = float; };
template <>
struct ActT<DST_ACT_I8> { using type = int8_t; using acc = int; };

template <int FMT, int ACT>
__global__ void __launch_bounds__(WARPS * 32)
generic_kernel(GemmArgs a) {
  using XT = typename ActT<ACT>::type;
  using AccT = typename ActT<ACT>::acc;
  __shared__ uint16_t lut[256];
  if (FMT == 1) {
    for (int i = threadIdx.x; i < 256; i += blockDim.x) lut[i] = (uint16_t)tq1_fields(i);
    __syncthreads();
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t e = blockIdx.y;
  const int64_t n = (int64_t)blockIdx.x * WARPS + warp;
  int64_t ra, rb;
  row_range(a.offsets, e, a.T, ra, rb);
  if (n >= a.N || ra >= rb) return;  // no block-wide barrier below this point
  const XT* __restrict__ x = static_cast<const XT*>(a.x);
  const int64_t K = a.K, G = a.G, group = a.group;

  for (int64_t row0 = ra; row0 < rb; row0 += TOK) {
    const int rows = (int)(rb - row0 < TOK ? rb - row0 : TOK);
    float y[TOK];
#pragma unroll
    for (int r = 0; r < TOK; ++r) y[r] = 0.f;
    for (int i = 0; i < a.terms.n; ++i) {
      const uint8_t* __restrict__ wrow = a.terms.packed[i] + (e * a.N + n) * a.Kp;
      const int64_t sbase = (e * a.N + n) * G;
      for (int64_t g = 0; g < G; ++g) {
        const int64_t k0 = g * group, k1 = k0 + group < K ? k0 + group : K;
        AccT acc[TOK];
#pragma unroll
        for (int r = 0; r < TOK; ++r) acc[r] = 0;
        for (int64_t k = k0 + lane; k < k1; k += 32) {
          int t;
          if (FMT == 2) {
            t = (int)((wrow[k >> 2] >> ((k & 3) * 2)) & 3) - 1;
          } else {
            const int64_t b = k / 5;
            t = (int)((lut[wrow[b]] >> ((int)(k - b * 5) * 2)) & 3) - 1;
          }
          if (t == 0) continue;
#pragma unroll
          for (int r = 0; r < TOK; ++r) {
            if (r < rows) {
              if (ACT == DST_ACT_I8) acc[r] += (AccT)t * (AccT)x[(row0 + r) * K + k];
              else acc[r] = (AccT)fmaf((float)t, (float)x[(row0 + r) * K + k], (float)acc[r]);
            }
          }
        }
        const float s = scale_to_float(a.terms.scale[i], sbase + g, a.scale_dtype);
#pragma unroll
        for (int r = 0; r < TOK; ++r) y[r] = fmaf(s, (float)acc[r], y[r]);
      }
    }
#pragma unroll
    for (int r = 0; r < TOK; ++r) {
      float v = y[r];
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
      y[r] = v;
    }
    if (lane == 0) {
#pragma unroll
      for (int r = 0; r < TOK; ++r) {
        if (r < rows) {
          const int64_t o = (row0 + r) * a.N + n;
          float v = y[r];
          if (a.row_scale) v *= a.row_scale[row0 + r];
          if (a.out_dtype == DST_OUT_F32) {
            float* out = static_cast<float*>(a.out);
            out[o] = a.accumulate ? out[o] + v : v;
          } else if (a.out_dtype == DST_OUT_BF16) {
            static_cast<__nv_bfloat16*>(a.out)[o] = __float2bfloat16_rn(v);
          } else {
            static_cast<__half*>(a.out)[o] = __float2half_rn(v);
          }
        }
      }
    }
  }
}

// ------------------------------------------------------------------------------------------ int8 activations
// The reference's CUDA contract (int8 activations, float scales, canonical weights) on mma.sync.m16n8k32 u8 x s8 -> s32:
// exact integer sums per 128 (64) trits, one fused multiply-add per (row, token) and step with the group's scale. Takes
// every K, N and row count; groups of a multiple of 64. Nothing is re-laid out: a lane reads 32 (16) consecutive trits of
// its weight row straight from the canonical bytes (TQ1 through a byte -> 2-bit-field table), and four ANDs of the 2-bit
// words ARE the A operands (digits t + 1; the sums of x, taken while the token rows are staged, remove the 1). The token
// rows are staged in shared memory in the lanes' order, so a B operand is half a 128-bit load.
// Eight warps per CTA; `wk` of them share 16 weight rows and split K between them (their sums meet in shared memory), so a
// small call still fills the GPU.
// What bounds it: memory latency at these sizes (an expert's 0.5-2 MB). The lane-per-trit kernel above spends ~4
// instructions per weight and token; measured with 16 experts, 96 rows, K = N = 2048, TQ2, float32 scales (19 MB):
// 308 us there, 23 us here.
constexpr int CI_WARPS = 8;
constexpr int CI_LUT_REPL = 8;  // copies of the table, a lane reads copy lane % 8: random bytes then rarely share a bank

struct CanonArgs {
  GemmArgs g;
  int wk;       // warps that split K (1, 2, 4 or 8)
  int chunk;    // K elements staged at a time (a multiple of STEP)
  int vec_x;    // token rows start 16-byte aligned
  int vec_w;    // TQ2 rows start 8-byte aligned and are whole 8-byte pieces
  int64_t packed_bytes;  // of one term, for the bounds of unaligned reads
};

__device__ __forceinline__ void mma_u8s8_acc(int* d, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// The four bytes at base + off as a word, off any value: bytes outside [0, total) read as 0.
__device__ __forceinline__ uint32_t load_bytes4(const uint8_t* base, int64_t off, int64_t total) {
  if (off >= 0 && off + 4 <= total && ((reinterpret_cast<uintptr_t>(base) + off) & 3) == 0) return *reinterpret_cast<const uint32_t*>(base + off);
  uint32_t v = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i)
    if (off + i >= 0 && off + i < total) v |= (uint32_t)base[off + i] << (8 * i);
  return v;
}
// n = 4 or 8 bytes at base + off, off of any alignment, through aligned words
template <int N>
__device__ __forceinline__ void load_unaligned(const uint8_t* base, int64_t off, int64_t total, uint32_t* out) {
  const int mis = (int)((reinterpret_cast<uintptr_t>(base) + off) & 3);
  uint32_t w[N / 4 + 1];
#pragma unroll
  for (int i = 0; i <= N / 4; ++i) w[i] = (i < N / 4 || mis) ? load_bytes4(base, off - mis + 4 * i, total) : 0u;
#pragma unroll
  for (int i = 0; i < N / 4; ++i) out[i] = __funnelshift_r(w[i], w[i + 1], 8 * mis);
}

// 16 W trits of a canonical row from trit k on as W words of 2-bit digits (trit j in bits 2 j, 2 j + 1); digits past the
// row's end are arbitrary (their activations are zero).
template <int FMT, int W>
__device__ __forceinline__ void load_trits(const CanonArgs& a, const uint8_t* packed, int64_t row, int k, const uint32_t* lut, uint32_t* out) {
  const int64_t off = row * a.g.Kp;
  if (FMT == 2) {
    const int b = k >> 2;
    if (a.vec_w) {
      if (W == 2) {
        const uint2 v = b < a.g.Kp ? *reinterpret_cast<const uint2*>(packed + off + b) : make_uint2(0u, 0u);
        out[0] = v.x;
        out[W - 1] = v.y;
      } else {
        out[0] = b < a.g.Kp ? *reinterpret_cast<const uint32_t*>(packed + off + b) : 0u;
      }
    } else {
      load_unaligned<4 * W>(packed, off + b, a.packed_bytes, out);
    }
  } else {
    // 5 trits per byte: the trits span 4 W bytes at most (r + 16 W <= 4 + 32 = 36 < 40 digits), ten bits of fields each
    const int b = k / 5, r = k - b * 5;
    uint32_t w[2];
    load_unaligned<4 * W>(packed, off + b, a.packed_bytes, w);
    auto fields = [&](uint32_t word, int i) { return lut[((word >> (8 * i)) & 0xffu) * CI_LUT_REPL]; };
    const uint64_t lo = (uint64_t)fields(w[0], 0) | ((uint64_t)fields(w[0], 1) << 10) | ((uint64_t)fields(w[0], 2) << 20) | ((uint64_t)fields(w[0], 3) << 30);
    if (W == 2) {
      const uint64_t hi = (uint64_t)fields(w[W - 1], 0) | ((uint64_t)fields(w[W - 1], 1) << 10) | ((uint64_t)fields(w[W - 1], 2) << 20) |
                          ((uint64_t)fields(w[W - 1], 3) << 30);
      const uint64_t v = ((lo | (hi << 40)) >> (2 * r)) | (r ? (hi >> 24) << (64 - 2 * r) : 0ull);
      out[0] = (uint32_t)v;
      out[W - 1] = (uint32_t)(v >> 32);
    } else {
      out[0] = (uint32_t)(lo >> (2 * r));
    }
  }
}

template <int FMT, int STEP, int NB>
__global__ void __launch_bounds__(CI_WARPS * 32)
canonical_i8_kernel(const CanonArgs a) {
  constexpr int W = STEP / 64;      // 2-bit words a lane holds of a row per step
  constexpr int TOK = 8 * NB;       // token rows per pass
  extern __shared__ __align__(16) uint8_t ci_smem[];
  __shared__ uint32_t lut_s[FMT == 1 ? 256 * CI_LUT_REPL : 1];
  const int xstride = a.chunk + 16;                                            // two rows read together hit all banks once
  uint8_t* xs = ci_smem;                                                       // [TOK][xstride], lane order
  int* xsum = reinterpret_cast<int*>(ci_smem + (size_t)TOK * xstride);         // [chunk / STEP][TOK]
  float* red = reinterpret_cast<float*>(ci_smem);                              // [warps][NB * 4][32], after the last chunk
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g8 = lane >> 2, c = lane & 3;
  if (FMT == 1)
    for (int i = tid; i < 256 * CI_LUT_REPL; i += CI_WARPS * 32) lut_s[i] = tq1_fields((uint32_t)i / CI_LUT_REPL);
  const uint32_t* lut = lut_s + (FMT == 1 ? (lane & (CI_LUT_REPL - 1)) : 0);
  const GemmArgs& g = a.g;
  const int64_t e = blockIdx.y, K = g.K, N = g.N, G = g.G;
  const int kp = warp % a.wk, wn = warp / a.wk, row_tiles = CI_WARPS / a.wk;
  const int64_t n_lo = ((int64_t)blockIdx.x * row_tiles + wn) * 16 + g8, n_hi = n_lo + 8;
  const int64_t r_lo = e * N + (n_lo < N ? n_lo : N - 1), r_hi = e * N + (n_hi < N ? n_hi : N - 1);  // rows beyond N are not stored
  const int8_t* __restrict__ x = static_cast<const int8_t*>(g.x);
  int64_t ra, rb;
  row_range(g.offsets, e, g.T, ra, rb);

  for (int64_t m0 = ra + (int64_t)blockIdx.z * TOK; m0 < rb; m0 += (int64_t)gridDim.z * TOK) {
    const int mc = (int)(rb - m0 < TOK ? rb - m0 : TOK);
    float y[NB][4];
#pragma unroll
    for (int b = 0; b < NB; ++b)
#pragma unroll
      for (int i = 0; i < 4; ++i) y[b][i] = 0.f;
    for (int64_t kc = 0; kc < K; kc += a.chunk) {
      const int left = (int)(K - kc < a.chunk ? K - kc : a.chunk);
      const int steps = (left + STEP - 1) / STEP;
      __syncthreads();  // the previous chunk (or pass) has been read
      // stage: a thread takes 16 elements of a token row, turns them into the four operand words (word f = elements f, 4 + f,
      // 8 + f, 12 + f) and adds them up; the 8 (4) threads of a step sit side by side
      const int per_row = steps * (STEP / 16);
      for (int i = tid; i < TOK * per_row; i += CI_WARPS * 32) {
        const int tok = i / per_row, q = i - tok * per_row;
        const int64_t k = kc + 16 * q;
        uint32_t in[4] = {0u, 0u, 0u, 0u};
        if (tok < mc && k < K) {
          const int8_t* src = x + (m0 + tok) * K + k;
          if (a.vec_x) {
            const uint4 v = *reinterpret_cast<const uint4*>(src);
            in[0] = v.x;
            in[1] = v.y;
            in[2] = v.z;
            in[3] = v.w;
          } else {
#pragma unroll
            for (int j = 0; j < 16; ++j)
              if (k + j < K) in[j >> 2] |= (uint32_t)(uint8_t)src[j] << (8 * (j & 3));
          }
        }
        int sum = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) sum = __dp4a((int)in[j], 0x01010101, sum);
        for (int off = STEP / 32; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
        const uint32_t l01 = __byte_perm(in[0], in[1], 0x5140), h01 = __byte_perm(in[0], in[1], 0x7362);
        const uint32_t l23 = __byte_perm(in[2], in[3], 0x5140), h23 = __byte_perm(in[2], in[3], 0x7362);
        const uint32_t f[4] = {__byte_perm(l01, l23, 0x5410), __byte_perm(l01, l23, 0x7632), __byte_perm(h01, h23, 0x5410), __byte_perm(h01, h23, 0x7632)};
        uint8_t* dst = xs + (size_t)tok * xstride + (W == 2 ? (q >> 1) * 32 + (q & 1) * 4 : q * 16);
#pragma unroll
        for (int j = 0; j < 4; ++j) *reinterpret_cast<uint32_t*>(dst + j * 4 * W) = f[j];
        if (q % (STEP / 16) == 0) xsum[(q / (STEP / 16)) * TOK + tok] = sum;
      }
      __syncthreads();
      for (int t = 0; t < g.terms.n; ++t) {
        const uint8_t* packed = g.terms.packed[t];
        uint32_t wl[W], wh[W];
        float sl, sh;
        auto fetch = [&](int st) {
          const int k = (int)kc + st * STEP;  // K <= 2^24
          load_trits<FMT, W>(a, packed, r_lo, k + c * 16 * W, lut, wl);
          load_trits<FMT, W>(a, packed, r_hi, k + c * 16 * W, lut, wh);
          const int grp = k / (int)g.group;
          sl = scale_to_float(g.terms.scale[t], r_lo * G + grp, g.scale_dtype);
          sh = scale_to_float(g.terms.scale[t], r_hi * G + grp, g.scale_dtype);
        };
        if (kp < steps) fetch(kp);
        for (int st = kp; st < steps; st += a.wk) {
          uint32_t cl[W], ch[W];
#pragma unroll
          for (int i = 0; i < W; ++i) {
            cl[i] = wl[i];
            ch[i] = wh[i];
          }
          const float s0 = sl, s1 = sh;
          if (st + a.wk < steps) fetch(st + a.wk);  // in flight under this step's MMAs
          constexpr uint32_t M = 0x03030303u;
#pragma unroll
          for (int b = 0; b < NB; ++b) {
            const uint8_t* xb = xs + (size_t)(8 * b + g8) * xstride + st * STEP + c * 16 * W;
            int acc[4] = {0, 0, 0, 0};
            const uint4 q0 = *reinterpret_cast<const uint4*>(xb);
            if (W == 2) {
              const uint4 q1 = *reinterpret_cast<const uint4*>(xb + 16);
              mma_u8s8_acc(acc, cl[0] & M, ch[0] & M, cl[W - 1] & M, ch[W - 1] & M, q0.x, q0.y);
              mma_u8s8_acc(acc, (cl[0] >> 2) & M, (ch[0] >> 2) & M, (cl[W - 1] >> 2) & M, (ch[W - 1] >> 2) & M, q0.z, q0.w);
              mma_u8s8_acc(acc, (cl[0] >> 4) & M, (ch[0] >> 4) & M, (cl[W - 1] >> 4) & M, (ch[W - 1] >> 4) & M, q1.x, q1.y);
              mma_u8s8_acc(acc, (cl[0] >> 6) & M, (ch[0] >> 6) & M, (cl[W - 1] >> 6) & M, (ch[W - 1] >> 6) & M, q1.z, q1.w);
            } else {
              mma_u8s8_acc(acc, cl[0] & M, ch[0] & M, (cl[0] >> 2) & M, (ch[0] >> 2) & M, q0.x, q0.y);
              mma_u8s8_acc(acc, (cl[0] >> 4) & M, (ch[0] >> 4) & M, (cl[0] >> 6) & M, (ch[0] >> 6) & M, q0.z, q0.w);
            }
            const int2 xs2 = *reinterpret_cast<const int2*>(xsum + st * TOK + 8 * b + 2 * c);
            y[b][0] = fmaf(s0, (float)(acc[0] - xs2.x), y[b][0]);
            y[b][1] = fmaf(s0, (float)(acc[1] - xs2.y), y[b][1]);
            y[b][2] = fmaf(s1, (float)(acc[2] - xs2.x), y[b][2]);
            y[b][3] = fmaf(s1, (float)(acc[3] - xs2.y), y[b][3]);
          }
        }
      }
    }
    if (a.wk > 1) {
      __syncthreads();  // the staged rows are no longer needed: the partial sums take their place
#pragma unroll
      for (int b = 0; b < NB; ++b)
#pragma unroll
        for (int i = 0; i < 4; ++i) red[(warp * NB * 4 + b * 4 + i) * 32 + lane] = y[b][i];
      __syncthreads();
      if (kp == 0) {
        for (int w = 1; w < a.wk; ++w)
#pragma unroll
          for (int b = 0; b < NB; ++b)
#pragma unroll
            for (int i = 0; i < 4; ++i) y[b][i] += red[((warp + w) * NB * 4 + b * 4 + i) * 32 + lane];
      }
    }
    if (kp == 0) {
#pragma unroll
      for (int b = 0; b < NB; ++b)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int tok = 8 * b + 2 * c + (i & 1);
          const int64_t n = i < 2 ? n_lo : n_hi;
          if (tok < mc && n < N) {
            const int64_t o = (m0 + tok) * N + n;
            const float v = g.row_scale ? y[b][i] * g.row_scale[m0 + tok] : y[b][i];
            if (g.out_dtype == DST_OUT_F32) {
              float* out = static_cast<float*>(g.out);
              out[o] = g.accumulate ? out[o] + v : v;
            } else if (g.out_dtype == DST_OUT_BF16) {
              static_cast<__nv_bfloat16*>(g.out)[o] = __float2bfloat16_rn(v);
            } else {
              static_cast<__half*>(g.out)[o] = __float2half_rn(v);
            }
          }
        }
    }
  }
}

template <int FMT, int STEP, int NB>
int launch_canonical(CanonArgs a, int64_t passes, cudaStream_t st) {
  constexpr int TOK = 8 * NB;
  const int64_t whole = cdiv64(a.g.K, STEP) * STEP;
  a.chunk = (int)std::min<int64_t>(whole, NB == 4 ? 2048 : 4096);
  // enough CTAs for two per SM where splitting K between warps can give them
  a.wk = 1;
  const int64_t tiles = cdiv64(a.g.N, 16) * std::min(a.g.E, a.g.T) * passes;
  const int64_t ctas = 2 * sm_count();
  while (a.wk < CI_WARPS && cdiv64(tiles * a.wk, CI_WARPS) < ctas && a.wk * STEP < whole) a.wk *= 2;
  const size_t stage = (size_t)TOK * (a.chunk + 16) + (size_t)TOK * (a.chunk / STEP) * 4;
  const size_t smem = std::max(stage, (size_t)CI_WARPS * NB * 4 * 32 * 4);
  auto kernel = canonical_i8_kernel<FMT, STEP, NB>;
  DST_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const dim3 grid((unsigned)cdiv64(a.g.N, 16 * (CI_WARPS / a.wk)), (unsigned)a.g.E, (unsigned)std::min<int64_t>(passes, 65535));
  kernel<<<grid, CI_WARPS * 32, smem, st>>>(a);
  DST_CUDA_TRY(cudaGetLastError());
  return DST_OK;
}

template <int FMT, int STEP>
int launch_canonical_rows(const CanonArgs& a, cudaStream_t st) {
  // token rows per pass by the rows an expert has (unknown on the host: twice the mean; a longer expert takes more passes)
  const int64_t rows = std::max<int64_t>(1, a.g.max_rows >= 0 ? a.g.max_rows : std::min(a.g.T, 2 * cdiv64(a.g.T, a.g.E)));
  if (rows <= 8) return launch_canonical<FMT, STEP, 1>(a, 1, st);
  if (rows <= 16) return launch_canonical<FMT, STEP, 2>(a, 1, st);
  return launch_canonical<FMT, STEP, 4>(a, cdiv64(rows, 32), st);
}

// Groups of whole 64-trit steps; anything else stays with the lane-per-trit kernel.
bool canonical_i8_supports(const GemmArgs& a) { return a.act_dtype == DST_ACT_I8 && a.group % 64 == 0 && a.E <= 65535; }

int launch_canonical_i8(const GemmArgs& g, cudaStream_t st) {
  CanonArgs a;
  a.g = g;
  a.wk = 1;
  a.chunk = 0;
  a.vec_x = g.K % 16 == 0 && (reinterpret_cast<uintptr_t>(g.x) & 15) == 0;
  a.vec_w = g.Kp % 8 == 0;
  for (int i = 0; i < g.terms.n; ++i) a.vec_w = a.vec_w && (reinterpret_cast<uintptr_t>(g.terms.packed[i]) & 7) == 0;
  a.packed_bytes = g.E * g.N * g.Kp;
  if (g.fmt == DST_FMT_TQ2) return g.group % 128 == 0 ? launch_canonical_rows<2, 128>(a, st) : launch_canonical_rows<2, 64>(a, st);
  return g.group % 128 == 0 ? launch_canonical_rows<1, 128>(a, st) : launch_canonical_rows<1, 64>(a, st);
}

template <int FMT>
int launch_fmt(const GemmArgs& a, dim3 grid, cudaStream_t st) {
  switch (a.act_dtype) {
    case DST_ACT_BF16: generic_kernel<FMT, DST_ACT_BF16><<<grid, WARPS * 32, 0, st>>>(a); break;
    case DST_ACT_F16: generic_kernel<FMT, DST_ACT_F16><<<grid, WARPS * 32, 0, st>>>(a); break;
    case DST_ACT_I8: generic_kernel<FMT, DST_ACT_I8><<<grid, WARPS * 32, 0, st>>>(a); break;
    default: return DST_ERR_BAD_ARG;
  }
  DST_CUDA_TRY(cudaGetLastError());
  return DST_OK;
}

}  // namespace

int launch_generic(const GemmArgs& a, cudaStream_t stream) {
  if (a.T == 0 || a.N == 0 || a.E == 0) return DST_OK;
  if (canonical_i8_supports(a)) return launch_canonical_i8(a, stream);
  const dim3 grid((unsigned)cdiv64(a.N, WARPS), (unsigned)a.E, 1);
  return a.fmt == DST_FMT_TQ2 ? launch_fmt<2>(a, grid, stream) : launch_fmt<1>(a, grid, stream);
}

}  // namespace dst
