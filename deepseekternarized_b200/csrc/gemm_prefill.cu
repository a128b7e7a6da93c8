// Prefill grouped ternary GEMM for sm_100a: tcgen05 MMA with TMEM accumulators, TMA-fed activations,
// warp-specialised dequantisation of packed trits straight into tensor memory.
//
// Problem (per expert e, rows ra..rb of the expert-sorted activations):
//     out[m, n] = row_scale[m] * sum_k x[m, k] * W_e[n, k],   W_e[n, k] = sum_i scale_i[e, n, k/128] * trit_i[e, n, k]
//
// Mapping ("swap AB"): the 128 weight rows of a tile are the MMA M dimension (TMEM lanes), the token rows of
// one expert (up to 320 per tile) are the MMA N dimension (TMEM columns), so tiles stay full when an expert
// has few rows and an expert with up to 320 rows has its weights dequantised ONCE per 128-row weight tile.
// Both operands are fp16, 64 K-elements per pipeline stage (128 for token tiles of at most 128 rows, the SMALL form):
//   A (weights)      packed 8 KB slabs of the tiled layout (layout_kernels.cu) arrive by cp.async.bulk in a
//                    small ring; the dequant warps turn them into scale * trit, exact in fp16, and write them
//                    with tcgen05.st straight into TENSOR MEMORY (lane = weight row, one 32-bit column = two
//                    consecutive K elements; 32 columns per 64 K): the MMA takes A from TMEM, so the
//                    dequantised tile never passes through shared memory
//   B (activations)  fp16 rows fetched by one thread with cp.async.bulk.tensor (TMA) into K-major,
//                    128-byte-swizzled shared-memory stages (one box for up to 256 rows, two for more)
//   D (accumulator)  fp32 in TMEM columns 0 .. tn_max - 1 (above 256 rows two MMAs per K step, each over half of the
//                    rows); the columns behind hold the A ring. A and B rings have their own depths (na, nb)
// What bounds it: up to ~128 token rows the instruction streams of the dequant warps and of the MMA issuer (130 to 500
// cycles of tensor work per 64 K, ~470 spent), above that the tensor pipe and the drain of the one accumulator. Measured
// on 96 experts of 4096 x 4096, one launch, this form / the one before (one 64-trit piece per group and step, two issuing
// warps on one ring of A and B slots, digit-field tables): TQ1 64 rows 310 / 629 us, 256 rows 599 / 736; TQ2 64 rows
// 319 / 577, 256 rows 590 / 689; two TQ2 terms 64 rows 502 / 869.
// Shared-memory bandwidth is what bounds this kernel when A goes through shared memory (measured: the MMA
// issuer stalled ~1100 cycles per 512-cycle stage); with A in TMEM only B is written and read there.
// bf16 activations are converted once to fp16 with a power-of-two factor per row (exact for every
// element within 2^-22 of the row's absolute maximum); the factor comes back through row_scale.
// tcgen05 kind::f16 refuses an fp16 A with a bf16 B (illegal instruction), hence the conversion.
//
// Warp roles (896 threads, one CTA per SM, persistent over tiles):
//   warp 0      TMA producer for B (one thread)
//   warp 1      MMA issuer (all lanes run the loop, the elected one issues); owns the TMEM allocation
//   warp 2      bulk-copy producer of the packed slabs (one thread)
//   warps 4-11  epilogue: TMEM -> registers -> global, two warps per TMEM lane quarter (warp id % 4) taking
//               alternate 32-column chunks
//   warps 12-27 dequant producers for A, in four groups of four warps: group g owns the 128-trit units with index = g
//               (mod 4), so four units are dequantised at once (each warp's instruction stream is a long dependent
//               chain); inside a group the warp with id % 4 == q owns the 32 weight rows of TMEM lane quarter q, one
//               thread per row. SMALL: the warps 8-11 are a fifth group, four epilogue warps drain
// The accumulator is drained by warps that do nothing else. A variant in which the 20 dequant warps also drained
// it (tcgen05.ld in the same, register-starved instruction stream as the dequantisation) raised "unspecified
// launch failure" on the GPU although the same code with extra progress stores passed; tcgen05.ld writes its
// destination registers asynchronously, so that role keeps few live registers and nothing between the load and
// tcgen05.wait::ld.
//
// Every mbarrier wait is bounded by elapsed clock cycles; on expiry the CTA raises its abort flag, all
// roles leave their loops, the CTA frees TMEM and the kernel records DST_ERR_TIMEOUT in the status word.
#include <cuda.h>

#include <atomic>
#include <cmath>
#include <cstring>

#include "dst_common.cuh"

namespace dst {
namespace {

constexpr int PF_CTRL_WARPS = 4;
constexpr int PF_EPI_WARPS = 8;              // accumulator drain, two warps per TMEM lane quarter
constexpr int PF_GROUPS = 4;                 // dequant warp groups (4 warps each, one per TMEM lane quarter)
constexpr int PF_DQ_WARPS = 4 * PF_GROUPS;
constexpr int PF_DQ_WARP0 = PF_CTRL_WARPS + PF_EPI_WARPS;
constexpr int PF_THREADS = 32 * (PF_DQ_WARP0 + PF_DQ_WARPS);
constexpr int PF_TN_MAX = 320;               // token rows per tile at most = accumulator columns in TMEM
constexpr int PF_A_COLS = 32;                // TMEM columns of one A stage: 64 fp16 per weight row
constexpr int PF_MAX_STAGES = 12;            // stage ring depth at most; tn_max + depth * 32 <= 512 TMEM columns
// Barriers of stage g (slab i): entry g % 16 (i % 16) of their ring, phase g / 16, whatever the number of data slots. A parity
// tells a phase from its neighbour only, and a dequant group jumps over the others' units to a stage up to 7 further on (a
// slab up to 6, in tiles of few K elements); sixteen entries keep every phase that a role waits for the next one of its entry.
constexpr uint32_t PF_BARS = 16;
constexpr int PF_SMALL_TN = 128;             // token tiles up to this many rows: the SMALL form of the kernel
// TQ1 selector tables (see tq1_stage_select): 64 KB where the token tiles leave room for it, else 32 KB
enum { PF_TABLE_NONE = 0, PF_TABLE_32K = 1, PF_TABLE_64K = 2 };
__host__ __device__ constexpr int pf_table(int fmt, int terms, bool small) {
  return fmt != 1 ? PF_TABLE_NONE : (small && terms <= 2 ? PF_TABLE_64K : PF_TABLE_32K);
}
constexpr int PF_SLAB = 8192;                // one (row tile, superblock) slab of packed weights
constexpr int PF_MAX_E = 1023;               // experts per launch: two int arrays of E + 1 entries live in shared memory
constexpr int PF_EPI_TILE = 2048;             // bytes of an epilogue warp's transposition tile (32 token rows x 32 columns x 2 bytes)
// Shared memory is planned in addresses of the shared window, because the selector tables sit at multiples of their size.
// The dynamic part starts behind the system's 1 KB and the static part (under 1 KB, the kernel checks it) and may reach up
// to PF_SMEM_END: 227 KB per CTA less the static part.
constexpr uint32_t PF_SMEM_FIRST = 1024, PF_SMEM_START = 2048, PF_SMEM_END = 232448;
constexpr long long PF_WAIT_CYCLES = 4000000000LL;  // ~2 s

__device__ int g_device_status = 0;
// Test hooks (dst_debug_prefill_timeout): the cycle limit of the bounded waits, and a switch that makes the epilogue
// warps keep their "accumulator drained" arrivals to themselves, so that the MMA warps' wait for the accumulator runs
// out by design at a CTA's second tile. Nothing faults or spins unbounded: the wait gives up, the abort flag goes up,
// every role leaves, the CTA frees its TMEM and the status word says DST_ERR_TIMEOUT.
__device__ long long g_wait_cycles = PF_WAIT_CYCLES;
__device__ int g_drop_drain_arrivals = 0;
int g_debug_max_ctas = 0;  // host side: caps the grid when positive (so one CTA is sure to own several tiles)

// Optional per-role cycle accounting (build with -DDST_ROLE_TIMERS): where each warp role of the tcgen05
// kernel spends its time, summed over CTAs. Read with dst_role_timers(). Off in the shipped library.
#ifdef DST_ROLE_TIMERS
__device__ unsigned long long g_role_timers[64];
#define RT_DECL(...) long long __VA_ARGS__
#define RT_NOW() clock64()
#define RT_ADD(slot, v) atomicAdd(&g_role_timers[slot], (unsigned long long)(v))
#define RT_WAIT(acc, call) [&]() { const long long t0__ = clock64(); const bool r__ = (call); acc += clock64() - t0__; return r__; }()
#define RT_SPAN(acc, t0) acc += clock64() - (t0)
#else
#define RT_DECL(...)
#define RT_NOW() 0
#define RT_ADD(slot, v)
#define RT_WAIT(acc, call) (call)
#define RT_SPAN(acc, t0)
#endif

// One tensor map per TMA box height (16, 32, ... 256 token rows), so half a stage or a whole one is one TMA instruction.
struct TmaMaps {
  CUtensorMap m[16];
};

struct PrefillParams {
  const uint8_t* tiled[DST_MAX_TERMS];
  const __half* scale[DST_MAX_TERMS];
  int n_terms;
  const float* row_scale;
  const int64_t* offsets;
  void* out;
  int out_dtype, accumulate;
  int E, T, N, K, G, NT, S, kstages;
  // chosen by the host from the shared-memory budget
  int tn_max;       // token rows per tile at most (a multiple of 32, <= PF_TN_MAX): accumulator columns 0 .. tn_max - 1, the A ring after them
  int rows_hint;    // most rows an expert is expected to have (host knowledge or the mean and three deviations), sizes tn_max
  int nb;           // B stages in shared memory
  int na;           // A slots in TMEM = length of the barrier rings (nb <= na): stage g uses A slot g % na and B stage g % nb
  int nslab;        // slots of the packed-slab ring, 2 or 3
  // places in the shared window (see plan_smem): B stage ring, packed slabs, tables and epilogue tiles, selector table
  uint32_t a_ring, a_slabs, a_front, a_table;
  int wide_drain;   // 16-bit outputs, N % 8 == 0, 16-byte aligned rows: the accumulator is drained with 128-bit stores (drain_tile_wide)
  // Scatter of the output rows (null: rows go to `out` in place). Row r is stored at row (row_target[r] & (2^48 - 1)) of
  // peer_out[row_target[r] >> 48]: the buffers of the GPUs whose tokens the rows belong to, written from the epilogue
  // with plain stores over NVLink while the tensor pipe works on the next tile. A negative target drops the row.
  const int64_t* row_target;
  void* peer_out[DST_MAX_PEERS];
  int n_peer_out;      // a target that names a buffer >= n_peer_out or a row >= peer_rows is dropped as well
  int64_t peer_rows;
};

// Entry d of the by-value pointer table, as a chain of selects over compile-time indices (indexing a parameter array
// with a run-time value copies the table into every thread's local memory).
__device__ __forceinline__ void* pf_peer_out(const PrefillParams& p, int d) {
  void* r = p.peer_out[0];
#pragma unroll
  for (int i = 1; i < DST_MAX_PEERS; ++i)
    if (d == i) r = p.peer_out[i];
  return r;
}

// ------------------------------------------------------------------------------------------ PTX helpers
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_n(uint32_t bar, uint32_t n) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(n) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// Up to PF_SPIN_TRIES try_waits in a loop written in PTX: three to five instructions per poll. The same loop in C++
// compiles to about nine (convergence bookkeeping around a divergent loop). A suspend-time hint does not reduce the polls
// (103 per 64 K elements with one of 20 us, 124 without).
#ifndef PF_SPIN_TRIES
#define PF_SPIN_TRIES 64
#endif
__device__ __forceinline__ bool mbar_spin(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n"
      ".reg .pred p, q;\n"
      ".reg .u32 n;\n"
      "mov.u32 n, %3;\n"
      "PF_SPIN:\n"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "@p bra PF_SPIN_DONE;\n"
      "sub.u32 n, n, 1;\n"
      "setp.ne.u32 q, n, 0;\n"
      "@q bra PF_SPIN;\n"
      "PF_SPIN_DONE:\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(done) : "r"(bar), "r"(parity), "n"(PF_SPIN_TRIES) : "memory");
  return done != 0;
}
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
               : "=r"(done) : "r"(bar), "r"(parity) : "memory");
  return done != 0;
}
// Bounded wait: false when the abort flag is up or ~2 s of clock cycles have passed.
// BACKOFF sleeps between polls: for roles that wait long.
template <bool BACKOFF = false>
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  if (mbar_test(bar, parity)) return true;
  const long long t0 = clock64();
  for (;;) {
    if (BACKOFF) {
#pragma unroll 1
      for (int i = 0; i < 16; ++i) {
        __nanosleep(200);
        if (mbar_test(bar, parity)) return true;
      }
    } else if (mbar_spin(bar, parity)) {
      return true;
    }
    if (*abort_flag) return false;
    if (clock64() - t0 > g_wait_cycles) {
      *abort_flag = 1;
      return false;
    }
  }
}

__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr) {
  // K-major, SWIZZLE_128B: start address >> 4, LBO unused (1), SBO = 1024 B (8 rows x 128 B), version 1.
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) |
         ((uint64_t)2 << 61);
}

// The four tcgen05.mma (K = 16 each) of 64 K elements: A from tensor memory (lane = row, 32-bit column = 2 K elements), B from
// shared memory. Executed by a whole (converged) warp, one elected lane issues. One block with one election: the issuing
// warp's instruction stream is what bounds tiles of few token rows (see the MMA issuer), and an election, two predicates
// and a descriptor assembled per instruction made it ~290 cycles per 64 K elements.
__device__ __forceinline__ void umma_f16_ts_64(uint32_t tmem_d, uint32_t tmem_a, uint32_t b_lo, uint32_t b_hi, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p, t, e;\n.reg .b32 a1, a2, a3, l1, l2, l3;\n.reg .b64 d0, d1, d2, d3;\n"
      "setp.ne.b32 p, %5, 0;\nsetp.eq.b32 t, %5, %5;\n"
      "add.u32 a1, %1, 8;\nadd.u32 a2, %1, 16;\nadd.u32 a3, %1, 24;\n"
      "add.u32 l1, %2, 2;\nadd.u32 l2, %2, 4;\nadd.u32 l3, %2, 6;\n"
      "mov.b64 d0, {%2, %3};\nmov.b64 d1, {l1, %3};\nmov.b64 d2, {l2, %3};\nmov.b64 d3, {l3, %3};\n"
      "elect.sync _|e, 0xffffffff;\n"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], d0, %4, p;\n"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [a1], d1, %4, t;\n"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [a2], d2, %4, t;\n"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [a3], d3, %4, t;\n}\n"
      ::"r"(tmem_d), "r"(tmem_a), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void umma_commit_elect(uint32_t bar) {
  asm volatile("{\n.reg .pred e;\nelect.sync _|e, 0xffffffff;\n"
               "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n" ::"r"(bar) : "memory");
}
// 8 consecutive 32-bit columns of this thread's TMEM lane
__device__ __forceinline__ void tmem_st_8(uint32_t taddr, const uint32_t* v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
               ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
               ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(bar) : "memory");
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}

#define TMEM_LD_32(v, taddr)                                                                                              \
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "                                                                  \
               "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,"   \
               "%28,%29,%30,%31}, [%32];"                                                                                 \
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),          \
                 "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),    \
                 "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),  \
                 "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])   \
               : "r"(taddr))
#define TMEM_LD_16(v, taddr)                                                                                             \
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"  \
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),         \
                 "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])    \
               : "r"(taddr))

// 16 TMEM lanes x 32 columns in the layout of an MMA accumulator fragment: registers 4 b + {0, 1} = lane t / 4 of the 16,
// columns 8 b + 2 (t % 4) + {0, 1}; registers 4 b + {2, 3} = lane t / 4 + 8, the same columns (t = lane of the warp).
#define TMEM_LD_16x256_X4(v, taddr)                                                                                        \
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"    \
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),           \
                 "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])      \
               : "r"(taddr))
// Four 8 x 8 matrices of 16-bit elements from registers (thread t: row t / 4, columns 2 (t % 4) + {0, 1} of each) to
// shared memory, TRANSPOSED: lanes 8 k .. 8 k + 7 give the addresses of the eight 16-byte rows of matrix k.
__device__ __forceinline__ void stmatrix_x4_trans(uint32_t addr, uint32_t r0, uint32_t r1, uint32_t r2, uint32_t r3) {
  asm volatile("stmatrix.sync.aligned.x4.trans.m8n8.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(r0), "r"(r1), "r"(r2), "r"(r3)
               : "memory");
}

// ------------------------------------------------------------------------------------------ tile walk
// Token rows a tile of `rows` rows occupies in the MMA N dimension: a multiple of 16 up to 256 (one MMA per K
// step), a multiple of 32 above (two MMAs, each over half of the rows, and N must be a multiple of 16).
__device__ __forceinline__ int tile_neff(int rows) { return rows <= 256 ? (rows + 15) & ~15 : (rows + 31) & ~31; }

// Tiles are numbered expert-major, then token tile, then weight-row tile (fastest), so the CTAs that run
// at the same time share an expert's activation rows in L2. The kernel keeps two int arrays in shared memory:
// offs[e] = first token row of expert e (clamped to [0, T]) and tpre[e] = number of tiles of the experts
// before e. A tile index is resolved with a short forward scan from the expert of the previous tile.
__device__ __forceinline__ int expert_tiles(const int* offs, int e, int tn_max, int NT) {
  const int n = offs[e + 1] - offs[e];
  return n > 0 ? (n + tn_max - 1) / tn_max * NT : 0;
}
// e: in = an expert at or before the tile's expert, out = the tile's expert. t must be < tpre[E].
__device__ __forceinline__ void tile_seek(const PrefillParams& p, const int* offs, const int* tpre, int t, int& e, int& nt, int& row0,
                                          int& rows) {
  while (tpre[e + 1] <= t) ++e;
  const int ra = offs[e], rb = offs[e + 1];  // rb > ra: the expert has tiles
  const int n = rb - ra;
  const int mt_count = (n + p.tn_max - 1) / p.tn_max;
  // an expert with more rows than one tile holds is split evenly, so no tile repeats the dequantisation
  // of the weights for a handful of left-over rows
  const int mt_rows = tile_neff((n + mt_count - 1) / mt_count);
  const unsigned local = (unsigned)(t - tpre[e]);
  const unsigned mt = local / (unsigned)p.NT;
  nt = (int)(local - mt * (unsigned)p.NT);
  row0 = ra + (int)mt * mt_rows;
  rows = rb - row0 < mt_rows ? rb - row0 : mt_rows;
}

// ------------------------------------------------------------------------------------------ dequant
__device__ __forceinline__ uint32_t h2_bits(__half2 h) { return *reinterpret_cast<uint32_t*>(&h); }
__device__ __forceinline__ __half2 bits_h2(uint32_t u) { return *reinterpret_cast<__half2*>(&u); }

// Field f (0..4) of a word that holds trit digits u = t + 1 as 2-bit fields, an even trit in bits [2f, 2f+1]
// and the odd trit after it in bits [16+2f, 17+2f]: (w & (0x00030003 << 2f)) | 0x64006400 is the fp16 pair
// 1024 + u * 4^f; one fused multiply-add maps it to u - 1 exactly.
template <int F>
__device__ __forceinline__ __half2 trit_pair(uint32_t w) {
  constexpr float m = F == 0 ? 1.f : F == 1 ? 0.25f : F == 2 ? 0.0625f : F == 3 ? 0.015625f : 0.00390625f;
  constexpr float a = F == 0 ? -1025.f : F == 1 ? -257.f : F == 2 ? -65.f : F == 3 ? -17.f : -5.f;
  return __hfma2(bits_h2((w & (0x00030003u << (2 * F))) | 0x64006400u), __floats2half2_rn(m, m), __floats2half2_rn(a, a));
}
__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}
template <bool FIRST>
__device__ __forceinline__ void put(__half2& acc, __half2 t, __half2 s2) {
  acc = FIRST ? __hmul2(t, s2) : __hfma2(t, s2, acc);  // the group scale is applied exactly (trit in {-1, 0, 1})
}

// TQ2, tiled word format: 16 trits, trit 2j in field j of the low half, trit 2j+1 in field j of the high half.
template <bool FIRST>
__device__ __forceinline__ void tq2_word(uint32_t w, __half2 s2, __half2* acc /* 8 */) {
  const uint32_t w2 = w >> 10;
  put<FIRST>(acc[0], trit_pair<0>(w), s2);
  put<FIRST>(acc[1], trit_pair<1>(w), s2);
  put<FIRST>(acc[2], trit_pair<2>(w), s2);
  put<FIRST>(acc[3], trit_pair<3>(w), s2);
  put<FIRST>(acc[4], trit_pair<4>(w), s2);
  put<FIRST>(acc[5], trit_pair<0>(w2), s2);
  put<FIRST>(acc[6], trit_pair<1>(w2), s2);
  put<FIRST>(acc[7], trit_pair<2>(w2), s2);
}

// TQ1, tiled grouping (layout_kernels.cu): the 64 trits of piece s of a row-superblock are the 12 bytes 12 s .. 12 s + 11
// (5 trits each) plus digit s of the 4 bytes 60..63. No arithmetic: an fp16 pair of scale * trit is ONE byte permutation of
// the four bytes {scale low, scale high, scale high with the sign flipped, 0}, and its selector (two bytes, one per trit: low
// nibble = source of the low byte, high nibble = source of the high byte) comes from a table in shared memory, 64 bits per
// byte value. A pair of bytes holds ten trits = five pairs, the third of them split between the two bytes.
//   64 KB table   an entry for either position in the pair, [byte value][position][16 replicas]: 256 bytes per byte value, so
//                 ONE byte permutation forms the address (the table sits at a multiple of 64 KB)
//                   first byte    x = trits 0, 1 | trit 4 in bits 16..23      y = trits 2, 3
//                   second byte   x = trits 6, 7 | trit 5 in bits 24..31      y = trits 8, 9
//   32 KB table   one entry for both, [byte value][16 replicas]: a shift and an AND-OR per address, two shifts per byte pair
//                   x = trits 0, 1, 2, 3      y = trits 3, 4, 1, 2
// (a permutation reads the low 16 bits of its selector). 16 replicas: the 64-bit reads of a half warp hit all banks once.
// A table of 2-bit digit fields expanded by fused multiply-adds (16 KB) took ~200 instructions per warp and 64 trits, this
// takes ~110: 96 experts of 4096 x 4096, 64 rows 457 -> 381 us in the form of the kernel of that time.
__host__ __device__ inline uint32_t tq1_select_byte(uint32_t digit) { return digit == 2u ? 0x10u : digit == 0u ? 0x20u : 0x33u; }
template <int TABLE>
__host__ __device__ inline void tq1_select_entry(uint32_t byte, int second, uint32_t& x, uint32_t& y) {
  const uint32_t f = tq1_fields(byte);
  uint32_t t[5];
#pragma unroll
  for (int d = 0; d < 5; ++d) t[d] = tq1_select_byte((f >> (2 * d)) & 3u);
  if (TABLE == PF_TABLE_64K) {
    x = second ? t[1] | (t[2] << 8) | (t[0] << 24) : t[0] | (t[1] << 8) | (t[4] << 16);
    y = second ? t[3] | (t[4] << 8) : t[2] | (t[3] << 8);
  } else {
    x = t[0] | (t[1] << 8) | (t[2] << 16) | (t[3] << 24);
    y = t[3] | (t[4] << 8) | (t[1] << 16) | (t[2] << 24);
  }
}
// where digit d of a byte is in its (first) entry
template <int TABLE>
__device__ __forceinline__ uint32_t tq1_select_place(int d) { return ((TABLE == PF_TABLE_64K ? 0x25410u : 0x53210u) >> (4 * d)) & 7u; }
// entry address of byte B of `word` for a lane whose replica of the first entry is at `base`
template <int TABLE, int B>
__device__ __forceinline__ uint32_t tq1_select_addr(uint32_t word, uint32_t base) {
  if (TABLE == PF_TABLE_64K) return __byte_perm(word, base, 0x7604 | (B << 4));  // the byte becomes bits 8..15 of base
  return ((B == 0 ? word << 7 : word >> (8 * B - 7)) & 0x7F80u) | base;          // ... bits 7..14
}
template <int SECOND>
__device__ __forceinline__ uint2 tq1_select_load(uint32_t addr) {
  uint2 v;
  if (SECOND) asm("ld.shared.v2.u32 {%0,%1}, [%2+128];" : "=r"(v.x), "=r"(v.y) : "r"(addr));
  else asm("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr));
  return v;
}
template <int TABLE, int B>
__device__ __forceinline__ uint32_t tq1_select_digit(uint32_t word, uint32_t base) {
  uint32_t v;
  asm("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(tq1_select_addr<TABLE, B>(word, base)));
  return v;
}
// prmt itself: __byte_perm masks every selector to three bits per nibble first, an instruction more for run-time selectors
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t d;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
  return d;
}
__device__ __forceinline__ void put_select(bool first, uint32_t& acc, uint32_t pool, uint32_t sel) {
  const uint32_t v = prmt(pool, pool, sel);
  acc = first ? v : h2_bits(__hadd2(bits_h2(acc), bits_h2(v)));
}
// The four source bytes of a scale (fp16 bits). A scale that is not finite makes NaN of its zero trits, as a product does.
__device__ __forceinline__ uint32_t tq1_select_pool(uint32_t h) {
  const uint32_t hi = h >> 8;
  return h | ((hi ^ 0x80u) << 16) | ((h & 0x7c00u) == 0x7c00u ? 0x7f000000u : 0u);
}
// One 64-trit piece of a row, all stacked terms, into 32 TMEM columns from `taddr` on, eight as soon as they are complete.
// w[i][0..2]: term i's 12 own bytes, w[i][3]: bytes 60..63 of the row-superblock; base: the lane's replica of the table;
// base_d: the same plus the place of the piece's digit inside an entry. n_terms <= TERMS.
template <int TABLE, int TERMS>
__device__ __forceinline__ void tq1_stage_select(const uint32_t (&w)[TERMS][4], int n_terms, uint32_t base, uint32_t base_d,
                                                 const uint32_t (&pool)[TERMS], uint32_t taddr) {
  uint32_t v[32];
#pragma unroll
  for (int q = 0; q < 6; ++q) {
#pragma unroll
    for (int i = 0; i < TERMS; ++i) {
      if (i < n_terms) {
        const uint32_t word = w[i][q >> 1];
        const uint2 a = tq1_select_load<0>((q & 1) ? tq1_select_addr<TABLE, 2>(word, base) : tq1_select_addr<TABLE, 0>(word, base));
        const uint2 b = tq1_select_load<TABLE == PF_TABLE_64K>((q & 1) ? tq1_select_addr<TABLE, 3>(word, base) : tq1_select_addr<TABLE, 1>(word, base));
        if (TABLE == PF_TABLE_64K) {
          put_select(i == 0, v[5 * q + 0], pool[i], a.x);
          put_select(i == 0, v[5 * q + 1], pool[i], a.y);
          put_select(i == 0, v[5 * q + 2], pool[i], __byte_perm(a.x, b.x, 0x0072));
          put_select(i == 0, v[5 * q + 3], pool[i], b.x);
          put_select(i == 0, v[5 * q + 4], pool[i], b.y);
        } else {
          put_select(i == 0, v[5 * q + 0], pool[i], a.x);
          put_select(i == 0, v[5 * q + 1], pool[i], a.x >> 16);
          put_select(i == 0, v[5 * q + 2], pool[i], __byte_perm(a.y, b.x, 0x0041));
          put_select(i == 0, v[5 * q + 3], pool[i], b.y >> 16);
          put_select(i == 0, v[5 * q + 4], pool[i], b.y);
        }
      }
    }
    if (q == 1) tmem_st_8(taddr, v);
    if (q == 3) tmem_st_8(taddr + 8, v + 8);
    if (q == 4) tmem_st_8(taddr + 16, v + 16);
  }
#pragma unroll
  for (int i = 0; i < TERMS; ++i) {  // trits 60..63
    if (i < n_terms) {
      put_select(i == 0, v[30], pool[i], tq1_select_digit<TABLE, 0>(w[i][3], base_d) | (tq1_select_digit<TABLE, 1>(w[i][3], base_d) << 8));
      put_select(i == 0, v[31], pool[i], tq1_select_digit<TABLE, 2>(w[i][3], base_d) | (tq1_select_digit<TABLE, 3>(w[i][3], base_d) << 8));
    }
  }
  tmem_st_8(taddr + 24, v + 24);
}

// Scale of group g (0..7 inside the 8 scales held in `sc`), as fp16 bits.
__device__ __forceinline__ uint32_t pick_scale_bits(const uint4& sc, int g) {
  const uint32_t w = (g & 4) ? ((g & 2) ? sc.w : sc.z) : ((g & 2) ? sc.y : sc.x);
  return (g & 1) ? (w >> 16) : (w & 0xFFFFu);
}
// Scale of group g (0..7 inside the 8 scales held in `sc`), as an fp16 pair.
__device__ __forceinline__ __half2 pick_scale(const uint4& sc, int g) {
  const uint32_t w = (g & 4) ? ((g & 2) ? sc.w : sc.z) : ((g & 2) ? sc.y : sc.x);
  const uint32_t h = (g & 1) ? (w >> 16) : (w & 0xFFFFu);
  return bits_h2(h | (h << 16));
}

// Drains a finished tile's accumulator: 32-column chunks col_first, col_first + col_step, ... of the warp's
// TMEM lane quarter -> registers -> global (thread = output column n, chunk column j = token row j).
__device__ __forceinline__ bool drain_tile(const PrefillParams& p, uint32_t tmem, int col_first, int col_step, int r, uint32_t tfull_bar,
                                        uint32_t tempty_bar, volatile int* abort_flag, int d_nt, int d_row0, int d_rows,
                                        uint32_t d_tile, const uint64_t* __restrict__ row_ptr) {
  const int lane = r & 31;
  const uint32_t lane_base = (uint32_t)(r & ~31) << 16;
  if (!mbar_wait<true>(tfull_bar, d_tile & 1u, abort_flag)) return false;
  // Lanes leave the polling loop (and its per-thread sleeps) one by one; the .sync.aligned tcgen05 instructions
  // below must be executed by the whole warp together.
  __syncwarp();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const int dn = d_nt * 128 + r;
  const bool n_ok = dn < p.N;
  const int n_eff = tile_neff(d_rows);
  // this thread owns output column dn; consecutive token rows are p.N elements apart
  const size_t esz = p.out_dtype == DST_OUT_F32 ? 4 : 2;
  const size_t ostep = (size_t)p.N * esz;
  uint8_t* obase = static_cast<uint8_t*>(p.out) + ((size_t)d_row0 * p.N + (n_ok ? dn : 0)) * esz;
  for (int c0 = col_first; c0 < n_eff; c0 += col_step) {
    const float rs_lane = (p.row_scale && c0 + lane < d_rows) ? p.row_scale[d_row0 + c0 + lane] : 1.f;
    uint32_t v[32];
    if (c0 + 32 <= n_eff) {
      TMEM_LD_32(v, tmem + lane_base + c0);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    } else {
      TMEM_LD_16(v, tmem + lane_base + c0);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
      for (int j = 16; j < 32; ++j) v[j] = 0u;
    }
    const int lim = n_ok ? d_rows - c0 : 0;  // token rows of this chunk that exist (and a column that exists)
    uint8_t* optr = obase + (size_t)c0 * ostep;
    if (row_ptr != nullptr) {
      // scatter form: row_ptr[j] = where token row j of the tile goes (0: nowhere), looked up by this role while it
      // waited for the accumulator; every thread stores its column of the row there
      const size_t col = (size_t)(n_ok ? dn : 0) * esz;
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        const float val = __uint_as_float(v[j]) * __shfl_sync(0xffffffffu, rs_lane, j);
        if (j < lim) {
          const uint64_t rowp = row_ptr[c0 + j];
          if (rowp != 0) {
            if (p.out_dtype == DST_OUT_BF16) *reinterpret_cast<__nv_bfloat16*>(rowp + col) = __float2bfloat16_rn(val);
            else *reinterpret_cast<__half*>(rowp + col) = __float2half_rn(val);
          }
        }
      }
    } else if (p.out_dtype == DST_OUT_BF16) {
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        const float val = __uint_as_float(v[j]) * __shfl_sync(0xffffffffu, rs_lane, j);
        if (j < lim) *reinterpret_cast<__nv_bfloat16*>(optr) = __float2bfloat16_rn(val);
        optr += ostep;
      }
    } else if (p.out_dtype == DST_OUT_F16) {
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        const float val = __uint_as_float(v[j]) * __shfl_sync(0xffffffffu, rs_lane, j);
        if (j < lim) *reinterpret_cast<__half*>(optr) = __float2half_rn(val);
        optr += ostep;
      }
    } else {
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        const float val = __uint_as_float(v[j]) * __shfl_sync(0xffffffffu, rs_lane, j);
        if (j < lim) {
          float* o = reinterpret_cast<float*>(optr);
          *o = p.accumulate ? *o + val : val;
        }
        optr += ostep;
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncwarp();
  if (lane == 0 && !g_drop_drain_arrivals) mbar_arrive(tempty_bar);
  return true;
}

// The same drain for 16-bit outputs with N % 8 == 0: 128-bit stores. A thread of the plain drain owns one output
// column and stores 2 bytes per token row, ~5 instructions each, and the drain of the single accumulator is on the
// critical path (a fifth of the second expert GEMM's time). Here the accumulator is read as MMA-style fragments
// (16 lanes x 256 bits), scaled, packed to pairs and turned by stmatrix.trans into a [32 token rows][32 columns] tile
// in this warp's 2 KB of shared memory (16-byte pieces XOR-swizzled by the row pair: no bank conflicts either way);
// every lane then moves four 16-byte pieces = eight adjacent columns of a token row each to global memory. The
// scatter form (row_ptr) needs one destination lookup per piece instead of one per element.
__device__ __forceinline__ bool drain_tile_wide(const PrefillParams& p, uint32_t tmem, int col_first, int col_step, int warp_q, int lane,
                                                uint32_t tfull_bar, uint32_t tempty_bar, volatile int* abort_flag, int d_nt, int d_row0,
                                                int d_rows, uint32_t d_tile, const uint64_t* __restrict__ row_ptr, uint8_t* tile_smem) {
  if (!mbar_wait<true>(tfull_bar, d_tile & 1u, abort_flag)) return false;
  __syncwarp();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const int n_eff = tile_neff(d_rows);
  const int n0 = d_nt * 128 + warp_q * 32;  // first output column of this warp's lane quarter
  const int t0 = lane & 3, t1 = lane >> 2;
  const uint32_t tile_a = smem_u32(tile_smem);
  // stmatrix: lane L addresses row r = L % 8 of matrix k = L / 8 of a group of four: (token block 2 x + k / 2, columns 16 h + 8 (k % 2) ..)
  const int st_r = lane & 7, st_g = (lane >> 3) & 1, st_b = lane >> 4;
  // read-back: piece q = 32 i + lane -> token row 8 i + lane / 4, columns 8 (lane % 4) ..
  const int rb_p = lane & 3, rb_t = lane >> 2;
  const size_t ostep = (size_t)p.N * 2;
  for (int c0 = col_first; c0 < n_eff; c0 += col_step) {
    const float rs_lane = (p.row_scale && c0 + lane < d_rows) ? p.row_scale[d_row0 + c0 + lane] : 1.f;
    float rs[8];  // of the token rows 8 b + 2 t0 + {0, 1} of the chunk
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      rs[2 * b] = __shfl_sync(0xffffffffu, rs_lane, 8 * b + 2 * t0);
      rs[2 * b + 1] = __shfl_sync(0xffffffffu, rs_lane, 8 * b + 2 * t0 + 1);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {  // lanes 16 h .. 16 h + 15 of the quarter = output columns n0 + 16 h ..
      uint32_t v[16];
      TMEM_LD_16x256_X4(v, tmem + ((uint32_t)(warp_q * 32 + 16 * h) << 16) + (uint32_t)c0);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      uint32_t m[8];  // m[2 b + g]: token block b, columns 16 h + 8 g ..: (row = column t1, pair = token rows 2 t0, 2 t0 + 1)
#pragma unroll
      for (int b = 0; b < 4; ++b)
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          const float lo = __uint_as_float(v[4 * b + 2 * g]) * rs[2 * b], hi = __uint_as_float(v[4 * b + 2 * g + 1]) * rs[2 * b + 1];
          if (p.out_dtype == DST_OUT_BF16) {
            const __nv_bfloat162 q = __floats2bfloat162_rn(lo, hi);
            m[2 * b + g] = *reinterpret_cast<const uint32_t*>(&q);
          } else {
            const __half2 q = __floats2half2_rn(lo, hi);
            m[2 * b + g] = *reinterpret_cast<const uint32_t*>(&q);
          }
        }
#pragma unroll
      for (int x = 0; x < 2; ++x) {  // token blocks 2 x, 2 x + 1
        const int tok = 8 * (2 * x + st_b) + st_r, piece = 2 * h + st_g;
        stmatrix_x4_trans(tile_a + (uint32_t)(tok * 64 + ((piece ^ ((tok >> 1) & 3)) << 4)), m[4 * x], m[4 * x + 1], m[4 * x + 2], m[4 * x + 3]);
      }
    }
    __syncwarp();
    const int n = n0 + 8 * rb_p;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int tok = 8 * i + rb_t;
      const uint4 q = *reinterpret_cast<const uint4*>(tile_smem + tok * 64 + ((rb_p ^ ((tok >> 1) & 3)) << 4));
      if (c0 + tok < d_rows && n < p.N) {
        if (row_ptr != nullptr) {
          const uint64_t rowp = row_ptr[c0 + tok];
          if (rowp != 0) *reinterpret_cast<uint4*>(rowp + (size_t)n * 2) = q;
        } else {
          *reinterpret_cast<uint4*>(static_cast<uint8_t*>(p.out) + (size_t)(d_row0 + c0 + tok) * ostep + (size_t)n * 2) = q;
        }
      }
    }
    __syncwarp();  // the tile is read before the next chunk overwrites it
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncwarp();
  if (lane == 0 && !g_drop_drain_arrivals) mbar_arrive(tempty_bar);
  return true;
}

// ------------------------------------------------------------------------------------------ the kernel
// Shared memory of a CTA (plan_smem places the parts):
//   B stage ring       nb stages of tn_max token rows x 64 (SMALL: 2 x 64) fp16, 1024-byte aligned
//   packed slabs       nslab x n_terms x 8 KB, slot-major
//   selector table     TQ1
//   front              offs[E + 1] and tpre[E + 1] (see tile_seek), the scatter form's row pointers, the epilogue warps' tiles
// SMALL: token tiles of at most PF_SMALL_TN rows: 128-K stages, four epilogue warps, five dequant groups.
template <int FMT, int TERMS, bool SMALL>
__global__ void __launch_bounds__(PF_THREADS, 1)
prefill_kernel(const __grid_constant__ TmaMaps xmaps, const PrefillParams p) {
  constexpr int SPB = FMT == 2 ? 4 : 5;  // 64-trit pieces per 64-byte row-superblock
  constexpr int TABLE = pf_table(FMT, TERMS, SMALL);
  constexpr int KH = SMALL ? 2 : 1;      // 64-K pieces per stage
  constexpr int EPI = SMALL ? 4 : PF_EPI_WARPS;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t NB = (uint32_t)p.nb, NA = (uint32_t)p.na;
  const uint32_t half_bytes = (uint32_t)p.tn_max * 128u, stage_bytes = half_bytes * KH;
  const uint32_t first = smem_u32(smem_raw);
  if (first < PF_SMEM_FIRST || first > PF_SMEM_START) {  // the plan does not fit this start of the dynamic part
    if (threadIdx.x == 0) atomicExch(&g_device_status, DST_ERR_UNSUPPORTED);
    return;
  }
  uint8_t* stages = smem_raw + (p.a_ring - first);
  uint8_t* slabs = smem_raw + (p.a_slabs - first);
  int* offs = reinterpret_cast<int*>(smem_raw + (p.a_front - first));
  int* tpre = offs + (PF_MAX_E + 1);
  // scatter form: destination of every token row of a tile, two tiles alternating (absent otherwise)
  constexpr int ROWS = SMALL ? PF_SMALL_TN : PF_TN_MAX;
  uint64_t* rowptr_s = reinterpret_cast<uint64_t*>(tpre + (PF_MAX_E + 1));
  uint8_t* epi_tiles = reinterpret_cast<uint8_t*>(rowptr_s + (p.row_target != nullptr ? 2 * ROWS : 0));  // EPI x 2 KB
  __shared__ uint64_t bar_full[PF_BARS], bar_empty[PF_BARS], bar_tfull[1], bar_tempty[1], bar_pfull[PF_BARS], bar_pempty[PF_BARS];
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_s;
  __shared__ uint64_t bar_epi;                      // scatter form: the epilogue warps' own barrier, once per tile
  volatile int* abort_flag = &abort_s;

  // the warp index as a broadcast: the compiler then knows it to be the same in all lanes and keeps what follows from it (the
  // MMA issuer's loop counters and addresses) in uniform registers
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  if (tid == 0) {
    abort_s = 0;
    for (int s = 0; s < (int)PF_BARS; ++s) {
      mbar_init(smem_u32(&bar_full[s]), 1 + 4);  // the TMA producer's expect_tx arrive + one arrive per warp of the dequant group that owns the stage
      mbar_init(smem_u32(&bar_empty[s]), 1);     // tcgen05.commit: the MMAs that read the stage are done
    }
    for (int a = 0; a < (int)PF_BARS; ++a) {
      mbar_init(smem_u32(&bar_pfull[a]), 1);         // bulk-copy producer's expect_tx arrive
      mbar_init(smem_u32(&bar_pempty[a]), 4 * SPB);  // one arrive per (piece of the superblock, warp of its group)
    }
    mbar_init(smem_u32(&bar_tfull[0]), 1);             // tcgen05.commit after the tile's last MMA
    mbar_init(smem_u32(&bar_tempty[0]), EPI);  // every epilogue warp has drained its share of the accumulator
    mbar_init(smem_u32(&bar_epi), EPI);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (TABLE != PF_TABLE_NONE) {
    // every entry is computed once (into the B ring, not in use yet), then copied to its 16 replicas
    constexpr int ENTRIES = TABLE == PF_TABLE_64K ? 512 : 256;
    uint2* once = reinterpret_cast<uint2*>(stages);
    for (int i = tid; i < ENTRIES; i += PF_THREADS) {
      uint2 v;
      tq1_select_entry<TABLE>(TABLE == PF_TABLE_64K ? (uint32_t)i >> 1 : (uint32_t)i, i & 1, v.x, v.y);
      once[i] = v;
    }
    __syncthreads();
    uint2* table = reinterpret_cast<uint2*>(smem_raw + (p.a_table - first));
    for (int i = tid; i < ENTRIES * 16; i += PF_THREADS) table[i] = once[i >> 4];
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the ring is written by bulk copies from here on
  }
  for (int i = tid; i <= p.E; i += PF_THREADS) {
    // offsets that were not validated on the host are clamped so no row index leaves [0, T)
    int64_t v = p.offsets ? p.offsets[i] : (i == 0 ? 0 : (int64_t)p.T);
    offs[i] = (int)(v < 0 ? 0 : (v > p.T ? p.T : v));
  }
  __syncthreads();
  if (warp == 0) {
    // tpre: exclusive prefix sum of the experts' tile counts; each lane takes a contiguous run of experts
    const int per = (p.E + 31) / 32, b0 = lane * per, b1 = b0 + per < p.E ? b0 + per : p.E;
    int sum = 0;
    for (int i = b0; i < b1; ++i) sum += expert_tiles(offs, i, p.tn_max, p.NT);
    int incl = sum;
    for (int d = 1; d < 32; d <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += up;
    }
    int run = incl - sum;
    for (int i = b0; i < b1; ++i) {
      tpre[i] = run;
      run += expert_tiles(offs, i, p.tn_max, p.NT);
    }
    if (lane == 31) tpre[p.E] = incl;
  } else if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)), "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_base_s;

  int e = 0, nt, row0, rows;
  const int nsb = (p.kstages + SPB - 1) / SPB;  // superblocks a tile touches
  const int t_step = (int)gridDim.x, n_tiles = tpre[p.E];

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer for B (activations)
    if (lane == 0) {
      uint32_t gst = 0, b = 0;  // stage, counted over all tiles of this CTA, and its place in the B ring
      bool ok = true;
      RT_DECL(w_empty = 0, n_it = 0, t_begin = RT_NOW());
      const uint32_t full0 = smem_u32(&bar_full[0]), empty0 = smem_u32(&bar_empty[0]), dst0 = smem_u32(stages);
      for (int t = (int)blockIdx.x; ok && t < n_tiles; t += t_step) {
        tile_seek(p, offs, tpre, t, e, nt, row0, rows);
        const int n_eff = tile_neff(rows);
        const int h = n_eff > 256 ? n_eff >> 1 : n_eff;  // token rows per TMA box and per MMA (a multiple of 16)
        const CUtensorMap* map = &xmaps.m[h / 16 - 1];
        const uint32_t bytes = (uint32_t)n_eff * 128u * KH;
        for (int ks = 0; ks < p.kstages; ks += KH) {
          const uint32_t prev = gst - NB;  // the stage whose place this is
          if (gst >= NB && !RT_WAIT(w_empty, mbar_wait(empty0 + prev % PF_BARS * 8, prev / PF_BARS & 1u, abort_flag))) { ok = false; break; }
          const uint32_t full = full0 + gst % PF_BARS * 8;
          mbar_arrive_expect_tx(full, bytes);
#pragma unroll
          for (int x = 0; x < KH; ++x) {
            const uint32_t dst = dst0 + b * stage_bytes + x * half_bytes;
            tma_load_2d(dst, map, (ks + x) * 64, row0, full);
            if (h != n_eff) tma_load_2d(dst + (uint32_t)h * 128u, map, (ks + x) * 64, row0 + h, full);
          }
          ++gst;
          if (++b == NB) b = 0;
#ifdef DST_ROLE_TIMERS
          ++n_it;
#endif
        }
      }
      RT_ADD(0, RT_NOW() - t_begin); RT_ADD(2, w_empty); RT_ADD(3, n_it); RT_ADD(4, 1);
    }
  } else if (warp == 2) {
    // ------------------------------------------------------------------ bulk-copy producer for the packed slabs
    if (lane == 0) {
      uint32_t gsl = 0, slot = 0;  // slab, counted over all tiles of this CTA, and its place
      bool ok = true;
      RT_DECL(w_pempty = 0, t_begin = RT_NOW());
      for (int t = (int)blockIdx.x; ok && t < n_tiles; t += t_step) {
        tile_seek(p, offs, tpre, t, e, nt, row0, rows);
        const int64_t off0 = ((int64_t)e * p.NT + nt) * p.S * PF_SLAB;
        for (int sb = 0; sb < nsb; ++sb) {
          const uint32_t prev = gsl - (uint32_t)p.nslab;  // the slab whose place this is
          if (gsl >= (uint32_t)p.nslab &&
              !RT_WAIT(w_pempty, mbar_wait<true>(smem_u32(&bar_pempty[prev % PF_BARS]), prev / PF_BARS & 1u, abort_flag))) { ok = false; break; }
          const uint32_t full = smem_u32(&bar_pfull[gsl % PF_BARS]);
          mbar_arrive_expect_tx(full, (uint32_t)p.n_terms * PF_SLAB);
          for (int i = 0; i < p.n_terms; ++i)
            bulk_load(smem_u32(slabs + ((size_t)slot * p.n_terms + i) * PF_SLAB), p.tiled[i] + off0 + (int64_t)sb * PF_SLAB, PF_SLAB, full);
          ++gsl;
          if (++slot == (uint32_t)p.nslab) slot = 0;
        }
      }
      RT_ADD(5, RT_NOW() - t_begin); RT_ADD(1, w_pempty);
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    // One warp, all of whose lanes run the loop (the elected lane issues). Next to the dequant warps its own instructions per
    // stage - a barrier wait, a vote, a commit and the MMAs - cost several hundred cycles whatever the number of token rows:
    // with a 64-K stage and every MMA elected by itself, 16 rows and 64 rows both took ~780 cycles per 64 K elements
    // (MMAs of 64 rows: 128; alone on the SM the same instructions take 166) and the dequant warps spent half of their
    // time waiting for a free A slot. Hence the 128-K stages of the small tiles and the one block per 64 K.
    {
      uint32_t gst = 0, s = 0, b = 0, tile = 0;  // stage, counted over all tiles of this CTA; its A slot and its place in the B ring
      bool ok = true;
      const uint64_t b_desc0 = umma_desc(smem_u32(stages));
      const uint32_t tmem_u = __shfl_sync(0xffffffffu, tmem, 0);
      const uint32_t b_desc_lo = (uint32_t)b_desc0, b_desc_hi = (uint32_t)(b_desc0 >> 32);
      RT_DECL(w_tempty = 0, w_full = 0, n_it = 0, t_begin = RT_NOW());
      for (int t = (int)blockIdx.x; ok && t < n_tiles; t += t_step) {
        tile_seek(p, offs, tpre, t, e, nt, row0, rows);
        // one accumulator: the previous tile must have been drained
        if (!__all_sync(0xffffffffu, RT_WAIT(w_tempty, mbar_wait(smem_u32(&bar_tempty[0]), (tile & 1u) ^ 1u, abort_flag)))) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t n_eff = __shfl_sync(0xffffffffu, (uint32_t)tile_neff(rows), 0);  // (uniform, as above)
        const bool two = n_eff > 256u;
        const uint32_t h = two ? n_eff >> 1 : n_eff;             // token rows per MMA (a multiple of 16, at most 256)
        // instruction descriptor: D f32, A f16, B f16, both K-major, N >> 3 at bit 17, M >> 4 at bit 24
        const uint32_t idesc = (1u << 4) | ((h >> 3) << 17) | ((128u >> 4) << 24);
        for (int ks = 0; ks < p.kstages; ks += KH) {
          if (!__all_sync(0xffffffffu, RT_WAIT(w_full, mbar_wait(smem_u32(&bar_full[gst % PF_BARS]), gst / PF_BARS & 1u, abort_flag)))) { ok = false; break; }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t a_tmem = tmem_u + (uint32_t)p.tn_max + s * (PF_A_COLS * KH);  // this stage's slot of the A ring
          const uint32_t b_lo = b_desc_lo + b * (stage_bytes >> 4);                  // start address of the B descriptor
#pragma unroll
          for (int x = 0; x < KH; ++x)
            umma_f16_ts_64(tmem_u, a_tmem + x * PF_A_COLS, b_lo + x * (half_bytes >> 4), b_desc_hi, idesc, (ks > 0 || x > 0) ? 1u : 0u);
          if (!SMALL && two) umma_f16_ts_64(tmem_u + h, a_tmem, b_lo + ((h * 128u) >> 4), b_desc_hi, idesc, ks > 0 ? 1u : 0u);
          umma_commit_elect(smem_u32(&bar_empty[gst % PF_BARS]));  // the MMAs have read the stage
          ++gst;
          if (++s == NA) s = 0;
          if (++b == NB) b = 0;
#ifdef DST_ROLE_TIMERS
          ++n_it;
#endif
        }
        if (ok) umma_commit_elect(smem_u32(&bar_tfull[0]));
        ++tile;
      }
      if (lane == 0) {
        RT_ADD(8, RT_NOW() - t_begin); RT_ADD(9, w_tempty); RT_ADD(10, w_full); RT_ADD(11, n_it); RT_ADD(12, 1); RT_ADD(13, tile);
      }
    }
  } else if (warp == 3) {
    // no role
  } else if (warp < PF_CTRL_WARPS + EPI) {
    // ------------------------------------------------------------------ epilogue: TMEM -> registers -> global
    const int r = (warp & 3) * 32 + lane;  // a warp may only read the TMEM lanes of its own quarter (warp id % 4)
    uint32_t tile = 0;
    const int epi_threads = 32 * EPI, epi_tid = tid - 32 * PF_CTRL_WARPS;
    for (int t = (int)blockIdx.x; t < n_tiles; t += t_step, ++tile) {
      tile_seek(p, offs, tpre, t, e, nt, row0, rows);
      const uint64_t* row_ptr = nullptr;
      if (p.row_target != nullptr) {
        // scatter form: while the tile is computed, look up where its token rows go (a global load and a pointer
        // per row, shared by the role's warps through shared memory; the buffer of the tile before stays intact for
        // warps still draining it, and nobody passes the barrier before all are done with the tile before that)
        uint64_t* rp = rowptr_s + (tile & 1u) * ROWS;
        const size_t ostep = (size_t)p.N * 2;
        for (int j = epi_tid; j < rows; j += epi_threads) {
          const int64_t tg = p.row_target[row0 + j];
          const int64_t dr = tg & 0xFFFFFFFFFFFFLL;
          const bool ok = tg >= 0 && (tg >> 48) < p.n_peer_out && dr < p.peer_rows;  // nothing is stored outside the buffers
          rp[j] = ok ? (uint64_t)reinterpret_cast<uintptr_t>(pf_peer_out(p, (int)(tg >> 48))) + (uint64_t)dr * ostep : 0ull;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&bar_epi));
        if (!mbar_wait(smem_u32(&bar_epi), tile & 1u, abort_flag)) break;
        __syncwarp();
        row_ptr = rp;
      }
      // the two warps of a lane quarter take alternate 32-column chunks
      const int col_first = ((warp - PF_CTRL_WARPS) >> 2) * 32, col_step = 32 * (EPI / 4);
      if (p.wide_drain) {
        if (!drain_tile_wide(p, tmem, col_first, col_step, warp & 3, lane, smem_u32(&bar_tfull[0]), smem_u32(&bar_tempty[0]), abort_flag, nt,
                             row0, rows, tile, row_ptr, epi_tiles + (warp - PF_CTRL_WARPS) * PF_EPI_TILE))
          break;
      } else if (!drain_tile(p, tmem, col_first, col_step, r, smem_u32(&bar_tfull[0]), smem_u32(&bar_tempty[0]), abort_flag, nt, row0,
                             rows, tile, row_ptr)) {
        break;
      }
    }
  } else {
    // ------------------------------------------------------------------ dequant producers (weights)
    // A warp may only touch the TMEM lanes of its own quarter (warp id % 4): it owns those 32 weight rows.
    const int q = warp & 3;
    const int r = q * 32 + lane;
    // groups 0..3: warps 12..27; with small token tiles warps 8..11 (epilogue warps otherwise) are group 4
    constexpr uint32_t n_groups = SMALL ? PF_GROUPS + 1 : PF_GROUPS;
    const uint32_t grp = warp >= PF_DQ_WARP0 ? (uint32_t)(warp - PF_DQ_WARP0) >> 2 : (uint32_t)PF_GROUPS;
    // logical word w of a row-superblock sits at physical word (((w & 3) ^ swizzle) << 2) | (w >> 2) of its 64 bytes
    const uint32_t slabs_a = smem_u32(slabs);
    uint32_t unit_off[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) unit_off[j] = (uint32_t)(r * 64 + ((j ^ ((r >> 1) & 3)) << 4));
    const uint32_t table_a = p.a_table + (uint32_t)(lane & 15) * 8u;
    const uint32_t lane_base = (uint32_t)(q * 32) << 16;
    const bool vec_scales = (p.G & 7) == 0;  // rows of 8 k scales are 16-byte aligned
    const int kstages = p.kstages;
    // A group takes 128 trits (two pieces: one scale group) at a time: unit `own`, counted over all tiles of this CTA. The
    // bookkeeping around a piece (barriers, slab slots, scale, loop) costs as much as its arithmetic and is paid once for two.
    const int units = kstages >> 1;
    uint32_t gst = grp * (2 / KH), s = gst % NA;  // the group's next unit's (first) stage, counted over all tiles of this CTA, and its A slot
    uint32_t gs0 = 0;                              // first slab of the current tile
    int g = (int)grp;                              // the group's next unit, from the current tile's first on
    bool ok = true;
    RT_DECL(w_pfull = 0, w_dempty = 0, w_drain = 0, w_comp = 0, w_st = 0, w_pre = 0, n_it = 0, t_begin = RT_NOW(), w_lds = 0, w_tail = 0, t_tail = RT_NOW());

    // scales of the row: 8 groups (8 units) per 128-bit load; when a block of 8 is taken into use the tile's next block is
    // prefetched into L1 (held in registers instead, it cost the two-term forms their spills)
    uint4 sc[TERMS];
    int cur_b = -1;                          // block of 8 groups held in sc, of the current tile
    const __half* srow[TERMS];               // the row's scales of the current tile (null: a row beyond N, scales read as 0)
    auto load_scales = [&](int g0, uint4* dst) {
#pragma unroll
      for (int i = 0; i < TERMS; ++i) {
        if (i < p.n_terms) {
          if (srow[i] == nullptr || g0 >= p.G) {
            dst[i] = make_uint4(0u, 0u, 0u, 0u);
          } else if (vec_scales) {
            dst[i] = *reinterpret_cast<const uint4*>(srow[i] + g0);
          } else {
            uint32_t h[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) h[j] = g0 + j < p.G ? (uint32_t)__half_as_ushort(srow[i][g0 + j]) : 0u;
            dst[i] = make_uint4(h[0] | (h[1] << 16), h[2] | (h[3] << 16), h[4] | (h[5] << 16), h[6] | (h[7] << 16));
          }
        }
      }
    };
    // SMALL TQ1: a group's units are ten pieces = two whole superblocks apart, so the pieces of all its units of a tile sit at
    // the same place of their superblocks and the words' offsets are found once per tile
    constexpr bool FIXED = SMALL && FMT == 1;
    static_assert(!FIXED || 2 * n_groups % SPB == 0, "units of a group at the same place of a superblock");
    uint32_t place[2][3] = {};  // FIXED: offsets of the words 3 sbk, 3 sbk + 1, 3 sbk + 2 of both pieces
    int sbk[2], sb0 = 0;        // piece inside its superblock; FIXED: the unit's first piece's superblock
    for (int t = (int)blockIdx.x; ok && t < n_tiles; t += t_step, g -= units, gs0 += (uint32_t)nsb) {
      if (g >= units) continue;  // a tile with fewer units than groups: none of them is this group's
      tile_seek(p, offs, tpre, t, e, nt, row0, rows);
      const int n = nt * 128 + r;
#pragma unroll
      for (int i = 0; i < TERMS; ++i)
        if (i < p.n_terms) srow[i] = n < p.N ? p.scale[i] + ((int64_t)e * p.N + n) * p.G : nullptr;
      cur_b = -1;
      if (FIXED) {
        sb0 = 2 * g / SPB;
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          sbk[x] = (2 * g + x) % SPB;
          const int k0 = 3 * sbk[x];
#pragma unroll
          for (int j = 0; j < 3; ++j) {
            const int lw = k0 + j;
            place[x][j] = (uint32_t)(r * 64 + (((lw & 3) ^ ((r >> 1) & 3)) << 4) + (lw >> 2) * 4);
          }
        }
      }
      for (; g < units; g += (int)n_groups) {
      RT_DECL(t_pre = RT_NOW());
      RT_SPAN(w_tail, t_tail);
      // scales
      const int blk = g >> 3;
      if (blk != cur_b) {
        load_scales(blk * 8, sc);
        cur_b = blk;
        if ((blk + 1) * 8 < p.G) {  // the tile's next block, needed a few of this warp's units from now
#pragma unroll
          for (int i = 0; i < TERMS; ++i)
            if (i < p.n_terms && srow[i] != nullptr) asm volatile("prefetch.global.L1 [%0];" ::"l"(srow[i] + (blk + 1) * 8));
        }
      }
      RT_SPAN(w_pre, t_pre);

      // packed words of this row for a piece, then (after the superblock's last piece of this group) the slab can go back to
      // the producer. One term: both pieces' words up front; more: a piece at a time (registers).
      constexpr int WX = TERMS == 1 ? 2 : 1;
      uint32_t w[WX][TERMS][4];
      auto load_piece = [&](int x, uint32_t (&dst)[TERMS][4]) -> bool {
        const int ks = 2 * g + x;
        int sb;
        if (FIXED) {
          sb = x == 0 ? sb0 : sb0 + (sbk[1] == 0);
        } else {
          sb = ks / SPB;
          sbk[x] = ks - sb * SPB;
        }
        const uint32_t gs = gs0 + (uint32_t)sb;
        const uint32_t slot = p.nslab == 2 ? (gs & 1u) : gs % 3u;
        const bool same = x == 1 && sbk[1] != 0;  // the first piece's slab
        if (!same && !RT_WAIT(w_pfull, mbar_wait(smem_u32(&bar_pfull[gs % PF_BARS]), gs / PF_BARS & 1u, abort_flag))) return false;
        RT_DECL(t_lds = RT_NOW());
#pragma unroll
        for (int i = 0; i < TERMS; ++i) {
          if (i < p.n_terms) {
            const uint32_t wp = slabs_a + ((uint32_t)slot * p.n_terms + i) * PF_SLAB;
            if (FMT == 2) {  // word 4 sbk + j
#pragma unroll
              for (int j = 0; j < 4; ++j) dst[i][j] = lds32(wp + unit_off[j] + sbk[x] * 4);
            } else if (FIXED) {
#pragma unroll
              for (int j = 0; j < 3; ++j) dst[i][j] = lds32(wp + place[x][j]);
              dst[i][3] = lds32(wp + unit_off[3] + 12);
            } else {         // words 3 sbk, 3 sbk + 1, 3 sbk + 2 and 15
              switch (sbk[x]) {
                case 0: dst[i][0] = lds32(wp + unit_off[0]); dst[i][1] = lds32(wp + unit_off[1]); dst[i][2] = lds32(wp + unit_off[2]); break;
                case 1: dst[i][0] = lds32(wp + unit_off[3]); dst[i][1] = lds32(wp + unit_off[0] + 4); dst[i][2] = lds32(wp + unit_off[1] + 4); break;
                case 2: dst[i][0] = lds32(wp + unit_off[2] + 4); dst[i][1] = lds32(wp + unit_off[3] + 4); dst[i][2] = lds32(wp + unit_off[0] + 8); break;
                case 3: dst[i][0] = lds32(wp + unit_off[1] + 8); dst[i][1] = lds32(wp + unit_off[2] + 8); dst[i][2] = lds32(wp + unit_off[3] + 8); break;
                default: dst[i][0] = lds32(wp + unit_off[0] + 12); dst[i][1] = lds32(wp + unit_off[1] + 12); dst[i][2] = lds32(wp + unit_off[2] + 12); break;
              }
              dst[i][3] = lds32(wp + unit_off[3] + 12);
            }
          }
        }
        // the slab goes back; the tile's last superblock may hold fewer than SPB pieces: make up for those that do not exist.
        // One term: both pieces' arrivals at once where they share the slab
        if (!(TERMS == 1 && x == 0 && sbk[0] != SPB - 1)) {
          __syncwarp();
          if (lane == 0)
            mbar_arrive_n(smem_u32(&bar_pempty[gs % PF_BARS]),
                          (uint32_t)((TERMS == 1 && same ? 2 : 1) + (ks == kstages - 1 ? nsb * SPB - kstages : 0)));
        }
#ifdef DST_ROLE_TIMERS
#pragma unroll
        for (int i = 0; i < TERMS; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) asm volatile("" : "+r"(dst[i][j]));
#endif
        RT_SPAN(w_lds, t_lds);
        return true;
      };
      if (TERMS == 1 && (!load_piece(0, w[0]) || !load_piece(1, w[WX - 1]))) { ok = false; break; }

#pragma unroll
      for (int x = 0; x < 2; ++x) {
        const int wx = TERMS == 1 ? x : 0;
        if (TERMS > 1 && !load_piece(x, w[0])) { ok = false; break; }
        if (!SMALL || x == 0) {
          // the A slot must be free (the MMAs that last read it are done); waited for before the arithmetic, so that the
          // dequantised words go to TMEM eight by eight as they come and need not all stay in registers
          // no sleep between polls here: these warps are the critical path, and a sleeping lane wakes up to a
          // microsecond late (the whole warp then waits for it at the next convergence point)
          const uint32_t prev = gst - NA;  // the stage whose A slot this is
          if (gst >= NA && !RT_WAIT(w_dempty, mbar_wait(smem_u32(&bar_empty[prev % PF_BARS]), prev / PF_BARS & 1u, abort_flag))) { ok = false; break; }
          __syncwarp();  // re-converge after the polling loop: tcgen05.st is .sync.aligned
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        }
        RT_DECL(t_c = RT_NOW());
        const uint32_t taddr = tmem + lane_base + (uint32_t)p.tn_max + s * (PF_A_COLS * KH) + (SMALL ? x * PF_A_COLS : 0);
        if constexpr (FMT == 1) {
          uint32_t pool[TERMS];
#pragma unroll
          for (int i = 0; i < TERMS; ++i) pool[i] = i < p.n_terms ? tq1_select_pool(pick_scale_bits(sc[i], g & 7)) : 0u;
          tq1_stage_select<TABLE, TERMS>(w[wx], TERMS <= 2 ? TERMS : p.n_terms, table_a, table_a + tq1_select_place<TABLE>(sbk[x]), pool, taddr);
        } else {
          __half2 s2[TERMS];
#pragma unroll
          for (int i = 0; i < TERMS; ++i) s2[i] = i < p.n_terms ? pick_scale(sc[i], g & 7) : __float2half2_rn(0.f);
#pragma unroll
          for (int j = 0; j < 4; ++j) {  // word by word, all terms, so eight words at a time are live
            __half2 acc[8];
#pragma unroll
            for (int i = 0; i < TERMS; ++i) {
              if (i < p.n_terms) {
                if (i == 0) tq2_word<true>(w[wx][i][j], s2[i], acc);
                else tq2_word<false>(w[wx][i][j], s2[i], acc);
              }
            }
            uint32_t v[8];
#pragma unroll
            for (int y = 0; y < 8; ++y) v[y] = h2_bits(acc[y]);
            tmem_st_8(taddr + 8 * j, v);
          }
        }
        RT_SPAN(w_comp, t_c);
        if (!SMALL || x == 1) {
          RT_DECL(t_st = RT_NOW());
          asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&bar_full[gst % PF_BARS]));
          RT_SPAN(w_st, t_st);
        }
        if (!SMALL && x == 0) {
          ++gst;
          if (++s == NA) s = 0;
        }
      }
      if (!ok) break;
#ifdef DST_ROLE_TIMERS
      ++n_it;
      t_tail = RT_NOW();
#endif
      constexpr uint32_t jump = SMALL ? n_groups : 2 * n_groups - 1;  // to the first stage of the group's next unit
      gst += jump;
      s += jump;
      while (s >= NA) s -= NA;
      if (FIXED) sb0 += 2 * (int)n_groups / SPB;
      }
    }
    if (warp == PF_DQ_WARP0 && lane == 0) {
      RT_ADD(24, RT_NOW() - t_begin); RT_ADD(25, w_pfull); RT_ADD(26, w_dempty); RT_ADD(27, n_it); RT_ADD(28, 1);
      RT_ADD(29, w_drain); RT_ADD(30, w_comp); RT_ADD(31, w_st); RT_ADD(32, w_pre); RT_ADD(33, w_lds); RT_ADD(34, w_tail);
    }
  }

  // ------------------------------------------------------------------ teardown
  if (*abort_flag) {
    // give copies and MMAs still in flight time to land before shared memory and TMEM are released
    const long long t0 = clock64();
    while (clock64() - t0 < 4000000LL) __nanosleep(1000);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
  }
  if (tid == 0 && abort_s) atomicExch(&g_device_status, DST_ERR_TIMEOUT);
}

// ------------------------------------------------------------------------------------------ activation conversion
// bf16 (or fp16) rows -> fp16 rows scaled by 2^-e with e = floor(log2(absmax)) - 7, so every row's
// largest magnitude lies in [128, 256); row_scale_out[m] = 2^e * row_scale_in[m].
template <typename XT>
__global__ void convert_rows_kernel(const XT* __restrict__ x, int64_t K, const float* __restrict__ rs_in, __half* __restrict__ y,
                                    float* __restrict__ rs_out) {
  __shared__ float red[32];
  const int64_t m = blockIdx.x;
  const XT* row = x + m * K;
  float amax = 0.f;
  for (int64_t k = threadIdx.x; k < K; k += blockDim.x) amax = fmaxf(amax, fabsf((float)row[k]));
  for (int off = 16; off > 0; off >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
  __syncthreads();
  if (threadIdx.x < 32) {
    float v = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.f;
    for (int off = 16; off > 0; off >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, off));
    if (threadIdx.x == 0) red[0] = v;
  }
  __syncthreads();
  amax = red[0];
  int ex = 0;
  if (amax > 0.f && isfinite(amax)) {
    (void)frexpf(amax, &ex);  // amax = f * 2^ex, f in [0.5, 1)
    ex -= 8;                  // amax * 2^-ex in [128, 256)
  }
  const float down = ldexpf(1.f, -ex);
  for (int64_t k = threadIdx.x; k < K; k += blockDim.x) y[m * K + k] = __float2half_rn((float)row[k] * down);
  if (threadIdx.x == 0) rs_out[m] = ldexpf(1.f, ex) * (rs_in ? rs_in[m] : 1.f);
}

using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                              const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                              CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeFn encode_fn() {
  static EncodeFn fn = nullptr;
  if (!fn) {
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeFn>(sym);
  }
  return fn;
}

// The kernel's dynamic shared memory starts where plan_smem reckons with (the kernel looks again, but can only leave without
// output): behind the system's part and at most 1 KB of the kernel's own static part.
template <typename Kernel>
int check_smem_start(Kernel kernel, std::atomic<int>& known) {
  if (known.load(std::memory_order_relaxed) == 0) {
    int dev = 0, reserved = 0;
    cudaFuncAttributes attr;
    DST_CUDA_TRY(cudaGetDevice(&dev));
    DST_CUDA_TRY(cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev));
    DST_CUDA_TRY(cudaFuncGetAttributes(&attr, kernel));
    const bool fits = (uint32_t)reserved >= PF_SMEM_FIRST && (size_t)reserved + ((attr.sharedSizeBytes + 127) & ~(size_t)127) <= PF_SMEM_START;
    known.store(fits ? 1 : 2, std::memory_order_relaxed);
  }
  return known.load(std::memory_order_relaxed) == 1 ? DST_OK : DST_ERR_UNSUPPORTED;
}

template <int FMT, int TERMS, bool SMALL>
int launch_plan(const TmaMaps& maps, const PrefillParams& p, size_t smem, cudaStream_t st) {
  auto kernel = prefill_kernel<FMT, TERMS, SMALL>;
  static std::atomic<int> smem_start{0};
  const int rc = check_smem_start(kernel, smem_start);
  if (rc != DST_OK) return rc;
  DST_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int dev = 0, sms = 148;
  DST_CUDA_TRY(cudaGetDevice(&dev));
  DST_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  // persistent CTAs, one per SM, fewer when there cannot be that many tiles
  long long tiles_upper = ((long long)cdiv64(p.T, p.tn_max) + p.E) * p.NT;
  if (tiles_upper >= (1LL << 30)) return DST_ERR_UNSUPPORTED;  // tile indices are 32-bit in the kernel
  if (tiles_upper < 1) tiles_upper = 1;
  unsigned grid = (unsigned)(tiles_upper < sms ? tiles_upper : sms);
  if (g_debug_max_ctas > 0 && grid > (unsigned)g_debug_max_ctas) grid = (unsigned)g_debug_max_ctas;
  kernel<<<grid, PF_THREADS, smem, st>>>(maps, p);
  DST_CUDA_TRY(cudaGetLastError());
  return DST_OK;
}

// Places the parts of a CTA's shared memory for p.tn_max, with at least min_nb B stages: sets nb, na, nslab and the
// addresses, returns the dynamic bytes (0: does not fit).
template <int FMT, int TERMS, bool SMALL>
size_t plan_smem(PrefillParams& p, int min_nb) {
  constexpr int TABLE = pf_table(FMT, TERMS, SMALL), KH = SMALL ? 2 : 1;
  const long long stage = p.tn_max * 128LL * KH, slab = (long long)p.n_terms * PF_SLAB;
  const long long front = 2 * (PF_MAX_E + 1) * 4 + (p.row_target ? 2 * (SMALL ? PF_SMALL_TN : PF_TN_MAX) * 8 : 0) +
                          (p.wide_drain ? (SMALL ? 4 : PF_EPI_WARPS) * PF_EPI_TILE : 0);
  const long long na = (512 - p.tn_max) / (PF_A_COLS * KH);
  p.na = (int)(na < PF_MAX_STAGES ? na : PF_MAX_STAGES);
  for (p.nslab = 3; p.nslab >= 2; --p.nslab) {
    const long long slabs = p.nslab * slab;
    long long ring_at, room;  // start of the ring, bytes for it
    if (TABLE == PF_TABLE_64K) {  // slabs, front | table at 64 KB | ring
      if (PF_SMEM_START + slabs + front > 0x10000) continue;
      ring_at = 0x20000;
      room = PF_SMEM_END - ring_at;
    } else if (TABLE == PF_TABLE_32K) {  // front | table at 32 KB | ring, slabs
      if (PF_SMEM_START + front > 0x8000) continue;
      ring_at = 0x10000;
      room = PF_SMEM_END - ring_at - slabs;
    } else {  // ring, slabs, front
      ring_at = PF_SMEM_START;
      room = PF_SMEM_END - ring_at - slabs - front;
    }
    long long nb = room / stage;
    if (nb > p.na) nb = p.na;
    if (nb < min_nb) continue;
    p.nb = (int)nb;
    const long long ring_end = ring_at + nb * stage;
    p.a_ring = (uint32_t)ring_at;
    p.a_table = TABLE == PF_TABLE_64K ? 0x10000u : 0x8000u;
    p.a_slabs = TABLE == PF_TABLE_64K ? PF_SMEM_START : (uint32_t)ring_end;
    p.a_front = TABLE == PF_TABLE_64K ? (uint32_t)(PF_SMEM_START + slabs) : TABLE == PF_TABLE_32K ? PF_SMEM_START : (uint32_t)(ring_end + slabs);
    const long long end = TABLE == PF_TABLE_64K ? ring_end : TABLE == PF_TABLE_32K ? ring_end + slabs : ring_end + slabs + front;
    return (size_t)(end - PF_SMEM_FIRST);
  }
  return 0;
}

// Chooses the token tile and places the CTA's shared memory: returns the dynamic bytes (0: not covered), p.tn_max and whether
// it is the SMALL form. one_matrix: all T rows of the call are one matrix's (a last run of one expert of many is not that).
template <int FMT, int TERMS>
size_t plan_tiles(PrefillParams& p, bool one_matrix, bool& small_form) {
  // The token tile is as large as the experts are expected to need (up to 320 rows) as long as a B ring of four 64-K stages
  // fits: that much hides the latency of the copies behind the MMAs of a stage. Then a third packed-slab slot if there is
  // room for it.
  int tn_cap = (p.rows_hint + 31) / 32 * 32;
  tn_cap = tn_cap < 64 ? 64 : (tn_cap > PF_TN_MAX ? PF_TN_MAX : tn_cap);
  int short_ring_tn = 0;  // the token tile that is taken with a ring of three stages
  if (one_matrix) {
    // One matrix: the row count is known, and few, large tiles may leave SMs idle. The token tile that gives the least (waves of
    // tiles) x (time of a 64-K stage, ns: fits of what 64 to 256 rows and one and two terms measured). 333 rows through
    // 4096 x 4096: 4 x 32 tiles of 84 rows instead of 2 x 32 of 167, kernel 30 -> 26 us; 2048 rows through 4096 x 11008, two terms: 203 -> 199 us per call.
    // The largest tile is weighed with three stages where four do not fit (TQ1, whose table takes 32 KB; a stage then takes up
    // to 1.3 times as long): 1200 rows through 4096 x 4096, TQ1, are one wave of 128 tiles of 300 rows instead of 160 of 240
    // rows in two, 55 -> 44 us (49 with the 16 KB table of the kernel before).
    const int sms = sm_count();
    float best = 0.f;
    int best_tn = 0;
    for (int tn = 64; tn <= tn_cap; tn += 32) {
      p.tn_max = tn;
      const bool small = tn <= PF_SMALL_TN;
      const bool fits = (small ? plan_smem<FMT, TERMS, true>(p, 2) : plan_smem<FMT, TERMS, false>(p, 4)) != 0;
      const bool short_ring = !fits && tn == PF_TN_MAX && plan_smem<FMT, TERMS, false>(p, 3) != 0;
      if (!fits && !short_ring) continue;
      const long long tiles = cdiv64(p.T, tn), rows = cdiv64(p.T, tiles);
      const float stage = (small ? 245.f + 0.9f * (float)(rows > 64 ? rows - 64 : 0) : 230.f + 0.9f * (float)rows) + 135.f * (float)(p.n_terms - 1);
      const float cost = (float)cdiv64(tiles * p.NT, sms) * stage * (short_ring ? 1.3f : 1.f);
      if (best_tn == 0 || cost < best) {
        best = cost;
        best_tn = tn;
        short_ring_tn = short_ring ? tn : 0;
      }
    }
    if (best_tn != 0) tn_cap = best_tn;
  }
  small_form = false;
  for (p.tn_max = tn_cap; p.tn_max > PF_SMALL_TN; p.tn_max -= 32)
    if (const size_t smem = plan_smem<FMT, TERMS, false>(p, p.tn_max == short_ring_tn ? 3 : 4)) return smem;
  small_form = true;
  for (; p.tn_max >= 64; p.tn_max -= 32)
    if (const size_t smem = plan_smem<FMT, TERMS, true>(p, 2)) return smem;
  return 0;
}
size_t plan_tiles(int fmt, PrefillParams& p, bool one_matrix, bool& small_form) {
  if (fmt == DST_FMT_TQ2)
    return p.n_terms == 1   ? plan_tiles<2, 1>(p, one_matrix, small_form)
           : p.n_terms == 2 ? plan_tiles<2, 2>(p, one_matrix, small_form)
                            : plan_tiles<2, 4>(p, one_matrix, small_form);
  return p.n_terms == 1   ? plan_tiles<1, 1>(p, one_matrix, small_form)
         : p.n_terms == 2 ? plan_tiles<1, 2>(p, one_matrix, small_form)
                          : plan_tiles<1, 4>(p, one_matrix, small_form);
}

// Tensor maps over the fp16 rows: [T, K], boxes of 64 K-elements x 16 i token rows, 128-byte swizzle, zero fill outside. One
// for every box height that the kernel can choose: the rows of a tile come from the offsets on the device, of which only
// the tile's size is certain here (the caller's host copy may differ).
int map_heights(int tn_max) { return (tn_max < 256 ? tn_max : 256) / 16; }
int encode_maps(TmaMaps& maps, const __half* rows, int64_t T, int64_t K, int heights) {
  const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)T};
  const cuuint64_t strides[1] = {(cuuint64_t)K * 2};
  const cuuint32_t estr[2] = {1, 1};
  for (int i = 0; i < heights; ++i) {
    const cuuint32_t box[2] = {64, (cuuint32_t)(16 * (i + 1))};
    const CUresult cr = encode_fn()(&maps.m[i], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<__half*>(rows), dims, strides, box, estr,
                                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (cr != CUDA_SUCCESS) return record_cuda_error(cudaErrorInvalidValue, "cuTensorMapEncodeTiled");
  }
  return DST_OK;
}

template <int FMT, int TERMS>
int launch_form(const TmaMaps& maps, const PrefillParams& p, bool small_form, size_t smem, cudaStream_t st) {
  return small_form ? launch_plan<FMT, TERMS, true>(maps, p, smem, st) : launch_plan<FMT, TERMS, false>(maps, p, smem, st);
}
int launch_run(int fmt, const __half* rows, PrefillParams& p, bool one_matrix, cudaStream_t st) {
  bool small_form = false;
  const size_t smem = plan_tiles(fmt, p, one_matrix, small_form);
  if (smem == 0) return DST_ERR_UNSUPPORTED;
  TmaMaps maps;
  const int rc = encode_maps(maps, rows, p.T, p.K, map_heights(p.tn_max));
  if (rc != DST_OK) return rc;
  if (fmt == DST_FMT_TQ2)
    return p.n_terms == 1   ? launch_form<2, 1>(maps, p, small_form, smem, st)
           : p.n_terms == 2 ? launch_form<2, 2>(maps, p, small_form, smem, st)
                            : launch_form<2, 4>(maps, p, small_form, smem, st);
  return p.n_terms == 1   ? launch_form<1, 1>(maps, p, small_form, smem, st)
         : p.n_terms == 2 ? launch_form<1, 2>(maps, p, small_form, smem, st)
                          : launch_form<1, 4>(maps, p, small_form, smem, st);
}

// The sizes of a launch: everything that plan_tiles looks at but the experts of the run (p.E)
void size_params(const GemmArgs& a, PrefillParams& p) {
  p.n_terms = a.terms.n;
  p.row_target = a.row_target;
  // 128-bit stores from the epilogue: two-byte outputs, whole 8-column pieces, 16-byte aligned rows
  p.wide_drain = (a.out_dtype != DST_OUT_F32 && !a.accumulate && a.N % 8 == 0 && (reinterpret_cast<uintptr_t>(a.out) & 15) == 0) ? 1 : 0;
  if (a.row_target != nullptr)
    for (int i = 0; i < DST_MAX_PEERS; ++i)
      if ((reinterpret_cast<uintptr_t>(a.peer_out[i]) & 15) != 0) p.wide_drain = 0;
  p.T = (int)a.T;
  p.N = (int)a.N;
  p.K = (int)a.K;
  p.G = (int)a.G;
  p.NT = (int)cdiv64(a.N, 128);
  p.S = (int)tiled_superblocks(a.fmt, a.K);
  p.kstages = (int)(a.K / 64);
  // Rows per expert: known when the caller passed host offsets, else three standard deviations of an even routing above the
  // mean. An expert with more is split into two tiles, which dequantises its weights twice; a tile sized for twice the mean
  // costs every expert the form of the kernel for larger tiles (96 rows on 96 experts of 4096 x 4096, TQ1, 428 against
  // 596 us). Under a skewed router (Zipf exponents 0, 0.3, 0.6, 1; 384 TQ1, 64 TQ2 and 128 two-term TQ2 experts) this size
  // against twice the mean took 0.88-0.95 of the time at 24 to 48 rows of the small TQ2 experts and the same elsewhere;
  // 0.94-1.00 even and up to 1.08 skewed at 64; 0.78-0.90 at 80 and 96 (two terms 0.91-1.03); 0.92-1.01 even and up to
  // 1.14 (TQ1, 128 rows, exponent 1) from 128 on.
  const int64_t mean = cdiv64(a.T, a.E);
  p.rows_hint = (int)(a.max_rows >= 0 ? a.max_rows : mean + (int64_t)ceil(3.0 * sqrt((double)mean)));
  if (p.rows_hint < 1) p.rows_hint = 1;
}
int run_experts_of(int64_t E, int64_t e0) { return (int)(E - e0 < PF_MAX_E ? E - e0 : PF_MAX_E); }


}  // namespace

size_t prefill_workspace_bytes(int act_dtype, int64_t T, int64_t K) {
  (void)act_dtype;  // fp16 activations are re-scaled per row as well, so every input type is converted
  return (size_t)T * (size_t)K * 2 + (((size_t)T * 4 + 255) & ~(size_t)255) + 256;
}

bool prefill_supports(const GemmArgs& a) {
  return a.weight_layout == DST_LAYOUT_TILED && a.group == 128 && a.K % 128 == 0 && a.scale_dtype == DST_SCALE_F16 &&
         ((a.act_dtype == DST_ACT_F16_NORM && a.row_scale != nullptr) ||
          ((a.act_dtype == DST_ACT_BF16 || a.act_dtype == DST_ACT_F16 || a.act_dtype == DST_ACT_I8) && a.workspace != nullptr &&
           a.workspace_bytes >= prefill_workspace_bytes(a.act_dtype, a.T, a.K))) &&
         a.T < (int64_t(1) << 30) &&
         a.N <= (int64_t(1) << 22) && encode_fn() != nullptr;
}

bool prefill_aligned(const GemmArgs& a) {
  const bool prenorm = a.act_dtype == DST_ACT_F16_NORM;
  if (!prenorm && (reinterpret_cast<uintptr_t>(a.workspace) & 255) != 0) return false;
  if (prenorm && (reinterpret_cast<uintptr_t>(a.x) & 15) != 0) return false;
  for (int i = 0; i < a.terms.n; ++i)
    if ((reinterpret_cast<uintptr_t>(a.terms.packed[i]) & 15) != 0 || (reinterpret_cast<uintptr_t>(a.terms.scale[i]) & 15) != 0) return false;
  return true;
}

int launch_prefill(const GemmArgs& a, cudaStream_t stream) {
  if (a.T == 0 || a.N == 0 || a.E == 0) return DST_OK;
  if (!prefill_supports(a)) return DST_ERR_UNSUPPORTED;
  if (!prefill_aligned(a)) return DST_ERR_ALIGNMENT;
  const bool prenorm = a.act_dtype == DST_ACT_F16_NORM;

  // 1. activations -> fp16 rows + per-row power-of-two factor, in the workspace
  //    (skipped when the caller hands in rows that are in that format already)
  const __half* xh = prenorm ? static_cast<const __half*>(a.x) : static_cast<const __half*>(a.workspace);
  const float* rs = prenorm ? a.row_scale
                            : reinterpret_cast<const float*>(static_cast<const uint8_t*>(a.workspace) + (((size_t)a.T * a.K * 2 + 255) & ~(size_t)255));
  if (prenorm) {
    // nothing to convert
  } else if (a.act_dtype == DST_ACT_BF16)
    convert_rows_kernel<__nv_bfloat16><<<(unsigned)a.T, 256, 0, stream>>>(static_cast<const __nv_bfloat16*>(a.x), a.K, a.row_scale,
                                                                          static_cast<__half*>(a.workspace), const_cast<float*>(rs));
  else if (a.act_dtype == DST_ACT_I8)
    // the int8-activation contract (per-token absmax quantisation, row_scale = the token's scale): int8 values are
    // exact in fp16, scale * trit is exact in fp16, every product is exact in fp32; only the fp32 accumulation
    // order differs from the reference's integer group sums (relative difference ~1e-6)
    convert_rows_kernel<int8_t><<<(unsigned)a.T, 256, 0, stream>>>(static_cast<const int8_t*>(a.x), a.K, a.row_scale,
                                                                   static_cast<__half*>(a.workspace), const_cast<float*>(rs));
  else
    convert_rows_kernel<__half><<<(unsigned)a.T, 256, 0, stream>>>(static_cast<const __half*>(a.x), a.K, a.row_scale,
                                                                   static_cast<__half*>(a.workspace), const_cast<float*>(rs));
  DST_CUDA_TRY(cudaGetLastError());

  // 2. one launch per run of experts
  PrefillParams p;
  for (int i = 0; i < DST_MAX_TERMS; ++i) {
    p.tiled[i] = i < a.terms.n ? a.terms.packed[i] : nullptr;
    p.scale[i] = i < a.terms.n ? static_cast<const __half*>(a.terms.scale[i]) : nullptr;
  }
  size_params(a, p);
  p.row_scale = rs;
  p.offsets = a.offsets;
  p.out = a.out;
  p.out_dtype = a.out_dtype;
  p.accumulate = a.accumulate;
  for (int i = 0; i < DST_MAX_PEERS; ++i) p.peer_out[i] = a.peer_out[i];
  p.n_peer_out = a.n_peer_out;
  p.peer_rows = a.peer_rows;
  if (a.row_target != nullptr && (a.out_dtype == DST_OUT_F32 || a.accumulate)) return DST_ERR_UNSUPPORTED;
  // The kernel keeps per-expert tables in shared memory: more experts than fit there are served by one launch
  // per run of PF_MAX_E experts (offsets are absolute token rows, so only the per-expert pointers move).
  const int64_t tiled_per_expert = (int64_t)p.NT * p.S * PF_SLAB, scales_per_expert = a.N * a.G;
  for (int64_t e0 = 0; e0 < a.E; e0 += PF_MAX_E) {
    p.E = run_experts_of(a.E, e0);
    p.offsets = a.offsets ? a.offsets + e0 : nullptr;
    for (int i = 0; i < a.terms.n; ++i) {
      p.tiled[i] = a.terms.packed[i] + e0 * tiled_per_expert;
      p.scale[i] = static_cast<const __half*>(a.terms.scale[i]) + e0 * scales_per_expert;
    }
    const int rc = launch_run(a.fmt, xh, p, a.E == 1, stream);
    if (rc != DST_OK) return rc;
  }
  return DST_OK;
}

}  // namespace dst

#ifdef DST_ROLE_TIMERS
// Profiling builds only: copies (and optionally clears) the 64 role-timer slots. Slots: 0-5 producers (B producer
// total cycles, slab producer wait slot free, B producer wait stage free, stages, threads, slab producer total),
// 8-13 MMA issuer (total, wait accumulator free, wait stage full, stages, threads, tiles), 24-30 one dequant warp
// (total, wait packed slab, wait stage free, own stages, threads, accumulator drain, dequant arithmetic, TMEM store +
// arrive, scale bookkeeping before the slab wait), 33 its reads of the packed words + slab hand-back, 34 loop tail and
// head (tile lookup included). The clock reads themselves cost: a build with them runs ~20 % slower.
extern "C" int dst_role_timers(unsigned long long* out, int reset) {
  DST_CUDA_TRY(cudaDeviceSynchronize());
  DST_CUDA_TRY(cudaMemcpyFromSymbol(out, dst::g_role_timers, sizeof(unsigned long long) * 64));
  if (reset) {
    unsigned long long z[64] = {0};
    DST_CUDA_TRY(cudaMemcpyToSymbol(dst::g_role_timers, z, sizeof(z)));
  }
  return DST_OK;
}
#endif

extern "C" int dst_debug_prefill_timeout(long long wait_cycles, int drop_drain_arrivals, int max_ctas) {
  const long long cycles = wait_cycles > 0 ? wait_cycles : dst::PF_WAIT_CYCLES;
  const int drop = drop_drain_arrivals ? 1 : 0;
  DST_CUDA_TRY(cudaDeviceSynchronize());
  DST_CUDA_TRY(cudaMemcpyToSymbol(dst::g_wait_cycles, &cycles, sizeof(cycles)));
  DST_CUDA_TRY(cudaMemcpyToSymbol(dst::g_drop_drain_arrivals, &drop, sizeof(drop)));
  dst::g_debug_max_ctas = max_ctas > 0 ? max_ctas : 0;
  return DST_OK;
}

extern "C" int dst_debug_prefill_plan(int fmt, int n_terms, int64_t E, int64_t T, int64_t N, int64_t K, int64_t max_rows, int out_dtype, int64_t first_expert,
                                      int* plan) {
  using namespace dst;
  if (!plan || (fmt != DST_FMT_TQ1 && fmt != DST_FMT_TQ2) || n_terms < 1 || n_terms > DST_MAX_TERMS || E < 1 || T < 1 || N < 1 || K < 128 ||
      K % 128 != 0 || first_expert < 0 || first_expert >= E || T >= (int64_t(1) << 30) || N > (int64_t(1) << 22) || K > (int64_t(1) << 24))
    return DST_ERR_BAD_ARG;
  GemmArgs a;
  memset(&a, 0, sizeof(a));
  a.terms.n = n_terms;
  a.E = E;
  a.T = T;
  a.N = N;
  a.K = K;
  a.G = K / 128;
  a.fmt = fmt;
  a.max_rows = max_rows;
  a.out_dtype = out_dtype;
  PrefillParams p;
  memset(&p, 0, sizeof(p));
  size_params(a, p);
  p.E = run_experts_of(E, first_expert / PF_MAX_E * PF_MAX_E);
  bool small_form = false;
  const size_t smem = plan_tiles(fmt, p, E == 1, small_form);
  if (smem == 0) return DST_ERR_UNSUPPORTED;
  const int values[DST_PREFILL_PLAN_INTS] = {p.tn_max, p.nb, p.na, p.nslab, small_form ? 1 : 0, (int)smem, map_heights(p.tn_max), p.E};
  memcpy(plan, values, sizeof(values));
  return DST_OK;
}

extern "C" int dst_check_device_status(dst_stream_t stream) {
  DST_CUDA_TRY(cudaStreamSynchronize(static_cast<cudaStream_t>(stream)));
  int st = 0;
  DST_CUDA_TRY(cudaMemcpyFromSymbol(&st, dst::g_device_status, sizeof(int)));
  if (st != 0) {
    const int zero = 0;
    DST_CUDA_TRY(cudaMemcpyToSymbol(dst::g_device_status, &zero, sizeof(int)));
  }
  int st_decode = 0;  // the decode kernel keeps a status word of its own
  const int rc = dst::decode_take_status(&st_decode);
  if (rc != DST_OK) return rc;
  int st_ep = 0;  // and so does the expert-parallel barrier
  const int rc2 = dst::ep_take_status(&st_ep);
  if (rc2 != DST_OK) return rc2;
  return st != 0 ? st : (st_decode != 0 || st_ep != 0) ? DST_ERR_TIMEOUT : DST_OK;  // the words hold the status itself
}

// ------------------------------------------------------------------------------------------ no-allocation entry
// Scratch for dst_ternary_grouped_gemm_noalloc: the fp16 copy of the activations and the per-row factors
// that the tcgen05 kernel otherwise keeps in a caller-provided workspace. It is part of the library
// image, so every GPU that loads the library holds these bytes until the process exits.
static __device__ __align__(256) unsigned char g_noalloc_scratch[DST_NOALLOC_SCRATCH_BYTES];

namespace dst {
namespace {
constexpr int kMaxDevices = 64;
void* g_noalloc_ptr[kMaxDevices] = {nullptr};  // device address of g_noalloc_scratch, per device ordinal
}  // namespace
}  // namespace dst

extern "C" int dst_ternary_grouped_gemm_noalloc(void* out, int out_dtype, int accumulate, const void* x, int act_dtype,
                                                const float* row_scale, const int64_t* offsets, const int64_t* offsets_host,
                                                const void* const* packed_tiled, const void* const* scales, int n_terms,
                                                int64_t E, int64_t T, int64_t N, int64_t K, int fmt, dst_stream_t stream) {
  using namespace dst;
  if (K <= 0 || (fmt != DST_FMT_TQ1 && fmt != DST_FMT_TQ2)) return DST_ERR_BAD_ARG;
  if (out_dtype < DST_OUT_F32 || out_dtype > DST_OUT_F16 || (act_dtype != DST_ACT_BF16 && act_dtype != DST_ACT_F16))
    return DST_ERR_BAD_ARG;
  if (n_terms < 1 || n_terms > DST_MAX_TERMS || E < 0 || T < 0 || N < 0) return DST_ERR_BAD_ARG;
  if (accumulate && out_dtype != DST_OUT_F32) return DST_ERR_BAD_ARG;
  if (E > DST_MAX_EXPERTS || K > (int64_t(1) << 24) || N > (int64_t(1) << 22) || T >= (int64_t(1) << 30)) return DST_ERR_BAD_SHAPE;
  if (K % 128 != 0) return DST_ERR_UNSUPPORTED;
  if (E != 1 && E != 0 && offsets == nullptr) return DST_ERR_BAD_ARG;
  if (offsets_host) {
    if (offsets_host[0] != 0 || offsets_host[E] != T) return DST_ERR_BAD_OFFSETS;
    for (int64_t e = 0; e < E; ++e)
      if (offsets_host[e + 1] < offsets_host[e]) return DST_ERR_BAD_OFFSETS;
  }
  if (E == 0) return T == 0 ? DST_OK : DST_ERR_BAD_OFFSETS;
  if (T == 0 || N == 0) return DST_OK;
  if (!out || !x || !packed_tiled || !scales) return DST_ERR_BAD_ARG;
  // The whole scratch need of this call must fit the static array: refuse anything larger.
  if (prefill_workspace_bytes(act_dtype, T, K) > (size_t)DST_NOALLOC_SCRATCH_BYTES) return DST_ERR_TOO_LARGE;

  // Set-up, once per device, with that device current: in host code the array's name is only a
  // stand-in for the symbol, so ask the runtime for its device address and hand THAT to the kernels.
  int dev = -1;
  DST_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) return DST_ERR_UNSUPPORTED;
  if (g_noalloc_ptr[dev] == nullptr) {
    void* ptr = nullptr;
    DST_CUDA_TRY(cudaGetSymbolAddress(&ptr, g_noalloc_scratch));
    if (ptr == nullptr) return record_cuda_error(cudaErrorInvalidSymbol, "cudaGetSymbolAddress(g_noalloc_scratch)");
    g_noalloc_ptr[dev] = ptr;
  }

  GemmArgs a;
  memset(&a, 0, sizeof(a));
  a.out = out;
  a.out_dtype = out_dtype;
  a.accumulate = accumulate;
  a.x = x;
  a.act_dtype = act_dtype;
  a.row_scale = row_scale;
  a.offsets = offsets;
  a.terms.n = n_terms;
  for (int i = 0; i < n_terms; ++i) {
    if (!packed_tiled[i] || !scales[i]) return DST_ERR_BAD_ARG;
    a.terms.packed[i] = static_cast<const uint8_t*>(packed_tiled[i]);
    a.terms.scale[i] = scales[i];
  }
  a.scale_dtype = DST_SCALE_F16;
  a.E = E;
  a.T = T;
  a.N = N;
  a.K = K;
  a.group = 128;
  a.Kp = cdiv64(K, fmt == DST_FMT_TQ2 ? 4 : 5);
  a.G = K / 128;
  a.fmt = fmt;
  a.max_rows = -1;
  a.weight_layout = DST_LAYOUT_TILED;
  a.workspace = g_noalloc_ptr[dev];
  a.workspace_bytes = DST_NOALLOC_SCRATCH_BYTES;
  return launch_prefill(a, static_cast<cudaStream_t>(stream));
}
