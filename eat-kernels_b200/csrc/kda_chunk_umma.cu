// Fused KDA chunk kernel on the 5th-generation tensor core (tcgen05 + tensor memory), sm_100a.
//
// One CTA walks the 32-token chunks of one (token run, head) task.  The fp32 state St [V=128][K=128] (value-first) never
// leaves tensor memory between chunks, and the whole per-chunk chain is tensor-core work issued by one elected lane:
//
//   MMA1  [W | O] = St [kd ; qd]^T          tf32: A = St read straight from its accumulator columns, N = 64, K = 128
//   MMA2  U  = v^T Tbh^T - W Tb^T           bf16 (A = v tile, MN-major) then tf32 (A = W columns, B negated), N = 32, K = 32
//   MMA3  St += U kr ,  O += U M^T          tf32: A = U columns; kr MN-major (N = 128), M K-major (N = 32)
//
// with kd = k 2^G, qd = scale q 2^G, kr = k 2^(G31-G), Tb = (I + diag(beta) tril(kd' ki'^T,-1))^-1 diag(beta),
// M = tril(qd' ki'^T) (G = inclusive cumulative log2-decay of the chunk; primed operands are taken relative to the
// exponent after token 15 so that every exponent is bounded by the decay of 16 tokens).  This is the chunked form of
// kda/b200/reference.py:30-37.  No accumulator makes a round trip through registers on the chain; the only register
// pass is the per-chunk decay St <- St diag(2^G31), done by the eight tensor-memory warps between MMA1 and MMA3, off
// the MMA warp's issue path.  Because tf32 operands keep 10 mantissa bits, the state enters the products more accurately
// than a bf16 copy would.
//
// Warp roles (28 warps):
//    0      MMA issuer (+ tensor-memory allocation); the whole warp runs the issue loop on warp-uniform values
//    1-2    triangular inverse, alternating chunks
//    3      loader: one lane polls three TMA copy streams (g / q,k / v); v goes straight into the consumer stage
//    4-11   tensor-memory warps: state load, per-chunk decay, checkpoints, final store, and O -> bf16 -> global; each
//           warp serves half of the columns of one lane quarter
//    12-27  operand preparation in two groups of eight warps that alternate chunks: gate + cumsum, L2 norm, decayed
//           operand tiles, intra-chunk products on mma.sync
// Roles hand off through mbarriers; every wait is bounded (see kda_umma.cuh): on a timeout the CTA keeps its control
// flow, waits (bounded again) for its copies and tensor-core work in flight, frees tensor memory and reports an error
// code in status[2].
//
// Measured alternative, not kept: the intra-chunk products as one bf16 tcgen05.mma over interleaved q / k tiles with
// the two results pulled out of tensor memory by the inverse warps.  It halves the work of the preparation warps, but
// the tensor-core round trip (issue, commit, barrier, tensor-memory load) and the extraction sit on the chain
// tiles -> products -> inverse -> MMA2, which with two operand stages is what sets the per-chunk time: 3-13 % slower.
//
// What bounds it: with 28 warps every warp issues about one instruction per ten cycles, so a chunk lasts as long as the chain
// [kd ; qd] free -> operand tiles -> intra-chunk products -> inverse -> MMA2 over the two stages; the tensor pipe needs 970
// cycles of it (the MMAs of a chunk depend on one another and still issue back to back).  Whole calls on a B200, with the
// cumulative sums through shared memory and three barriers per chunk / as it is (two boxes): prepared launches of 8 x 1024 tokens at 64 heads,
// raw 415 / 345 us, of 1 x 32768 at 16 heads with checkpoints, raw 985 / 883, of 48 requests at 64 heads, plain 2041 / 1920 (under the
// power cap); one-shot calls of 1 x 8192 at 96 heads, raw 789 / 608, of 16 x U[128, 4096] at 32 heads, plain 625 / 571; a graph of
// 512 x 64 tokens at 64 heads, plain 2345 / 2314 (start and end of a task).  The preparation warps react to where their code
// lies: other text in a function that is never called there has moved long raw runs by 2.5 %.
#include "kda_common.cuh"
#include "kda_plan.cuh"
#include "kda_tma.cuh"
#include "kda_umma.cuh"

namespace kda {
using namespace umma;

namespace u {

constexpr int WARPS = 28;
constexpr int THREADS = WARPS * 32;
constexpr int W_MMA = 0, W_INV0 = 1, W_LOAD = 3, W_SCALE0 = 4, W_PREP0 = 12;
constexpr int PREP_GROUPS = 2;                 // group g prepares the chunks c with c % 2 == g, in stage g
constexpr int PREP_WARPS = 8, PREP_THREADS = 256;   // per group

// ---- shared memory map (bytes); operand tiles are 1024-byte aligned.  A stage holds the operands of one chunk: what the
// tensor core reads (CS_*) and the bf16 k tile of the intra-chunk products (KI).
constexpr int CS_KDQD = 0, CS_KR = 32768, CS_V = 49152, CS_TB = 57344, CS_M = 61440;
constexpr int KI = 65536, STAGE = KI + 8192;
// Raw tiles: a ring of gate tiles and a ring of q / k tiles in 64 KB (the decayed bf16 tiles of the intra-chunk products
// replace q and k in place).  bf16 gates (8 KB) leave room for a third q / k stage.
template <int FE> struct Raw {
  static constexpr int G_BYTES = FE == 1 ? 16384 : 8192, NQK = FE == 1 ? 2 : 3;
  // The full barriers belong to chunks c, c + NFULL, ..: always the same preparation group waits on one, so it sees every
  // phase of it (a group that skipped a phase could take an older one of the same parity for its own).
  static constexpr int NFULL = NQK == 3 ? 6 : 2;
  static constexpr int OFF_G = 2 * STAGE, OFF_QK = OFF_G + 2 * G_BYTES;      // q, then k, of a stage
  static_assert(2 * G_BYTES + NQK * 16384 == 65536, "raw tiles");
};
constexpr int OFF_NORM = 2 * STAGE + 65536;                   // raw gates: partial square sums, 2 x [channel half]{q, k}[token]
constexpr int OFF_TBH = OFF_NORM + 1024;                      // 2 x 2048 (bf16, 64-byte swizzle)
constexpr int LS = 40;                                        // row stride of L in floats: rows 8 banks apart, 16-byte aligned
constexpr int OFF_L = OFF_TBH + 4096;                         // 2 x fp32 [32][LS]
constexpr int OFF_DEC = OFF_L + 2 * C * LS * 4;               // 4 x 512 (a slot is rewritten four chunks later)
constexpr int OFF_BETA = OFF_DEC + 2048;                      // beta of a chunk: 2 groups x 2 (alternating) x 128
constexpr int OFF_BAR = OFF_BETA + 512;                       // mbarriers
constexpr int NUM_BARS = 42;
constexpr int OFF_MISC = OFF_BAR + NUM_BARS * 8;              // +0 tmem slot, +8 abort code, +12 range flag, +16 wait limit (ns)
constexpr int SMEM_BYTES = OFF_MISC + 64;
static_assert(SMEM_BYTES <= 227 * 1024 && STAGE % 1024 == 0 && OFF_MISC % 8 == 0, "shared memory budget");

// mbarrier indices
constexpr int B_G_FULL = 0, B_G_EMPTY = 2, B_CONS_EMPTY = 4, B_P1_FULL = 6, B_INV_FULL = 8, B_L_FULL = 10,
              B_L_EMPTY = 12, B_O_FULL = 14, B_O_EMPTY = 16, B_MMA1_DONE = 18, B_S_READY = 19, B_DRAIN = 20, B_V_EMPTY = 21,
              B_QK_FULL = 23, B_QK_EMPTY = 29, B_V_FULL = 32, B_KDQD_EMPTY = 34,
              B_MMA1_DONE_T = 36, B_S_READY_T = 37,   // second chain of a dual-chain task
              B_NORM = 38,                            // partial square sums of q and k (raw gates only)
              B_KDQD_FULL = 40;                       // [kd ; qd] written: MMA1 may start before the rest of the stage is

// tensor-memory columns
constexpr uint32_t TM_COLS = 512, TM_S = 0, TM_WO = 128, TM_U = 256;
constexpr uint32_t TD_S0 = 0, TD_S1 = 128, TD_WO0 = 256, TD_WO1 = 320, TD_U0 = 384, TD_U1 = 448;   // dual-chain tasks

// error codes written to status[2] when a bounded wait gives up (which role, which barrier)
constexpr int E_LOAD = 0x40, E_PREP = 0x80, E_INV = 0xc0, E_MMA = 0x100, E_SCALE = 0x140, E_EPI = 0x180, E_DRAIN = 0x1c0;

#ifdef KDA_PROF
#define PROF_STAMP(role, slot) do { if ((threadIdx.x & 31) == 0 && blockIdx.x == 0 && x.prof != nullptr) { const long long _t = clock64(); atomicAdd(x.prof + (role) * 128 + 64 + (slot), (unsigned long long)(_t - prof_last)); prof_last = _t; } } while (0)
#define PROF_BEGIN long long prof_last = clock64()
#else
#define PROF_STAMP(role, slot) do { } while (0)
#define PROF_BEGIN do { } while (0)
#endif

// Byte offset of element (row, col) of a raw / decayed bf16 [32][128] tile as the copy engine lays it out with the
// 128-byte swizzle: two halves of 64 channels, each 32 rows of 128 bytes, 16-byte chunks XOR-ed with (row % 8).
// ldmatrix phases (8 rows, one chunk) are bank-conflict free in this layout.
__device__ __forceinline__ uint32_t rawtile_off(int row, int col) {
  return (uint32_t)((col >> 6) * 4096 + row * 128 + (((((col & 63) >> 3) ^ (row & 7))) << 4) + ((col & 7) << 1));
}

#ifndef KDA_SLEEP_NS
#define KDA_SLEEP_NS 32
#endif
constexpr unsigned kSleepNs = KDA_SLEEP_NS;   // back-off of waiting warps (not of the MMA issuer)

struct Ctx {
  uint8_t* smem;
  uint32_t bars;              // shared address of barrier 0
  volatile int* abort_flag;
  int h, len, nchunks;
  long long t0;
  __device__ __forceinline__ uint32_t bar(int i) const { return bars + 8u * (uint32_t)i; }
#ifdef KDA_PROF
  unsigned long long* prof;   // [role 0..7][wait on barrier 0..63 | 64 + stamp slot | 126 = total, 127 = warps] cycle
                              // counters of CTA 0 (profiling builds only; a buffer of its own, see kda_debug_configure)
  __device__ __forceinline__ void wait(int i, uint32_t parity, int code, unsigned sleep_ns = kSleepNs) const {
    const long long t = clock64();
    mbar_wait(bar(i), parity, abort_flag, code + i, sleep_ns);
    if ((threadIdx.x & 31) == 0 && blockIdx.x == 0 && prof != nullptr)
      atomicAdd(prof + ((code >> 6) * 128 + i), (unsigned long long)(clock64() - t));
  }
#else
  __device__ __forceinline__ void wait(int i, uint32_t parity, int code, unsigned sleep_ns = kSleepNs) const {
    mbar_wait(bar(i), parity, abort_flag, code + i, sleep_ns);
  }
#endif
};

// ------------------------------------------------------------------------------------------------ loader warp
// One elected lane drives the copy engine: per chunk it arms the stage's mbarrier with the byte count and issues the
// tile copies (g, q, k into the raw stage, v straight into the MMA2 operand slot of the consumer stage, whose
// MN-major 128-byte-swizzled layout is exactly what the engine writes).
// Rare paths of the loader, out of line: its polling loop sits on the refill latency of every tile, and anything that
// adds live state or code to it costs measurable time per chunk.
__device__ __noinline__ bool loader_idle_expired(unsigned long long idle_ns, volatile int* abort_flag) {
  if (idle_ns <= wait_limit_of(abort_flag)) return false;
  atomicCAS(const_cast<int*>(abort_flag), 0, E_LOAD);
  return true;
}
// Before the CTA may leave, every copy the loader issued has landed (on the normal path the consumers saw to that
// long ago and these waits return at once; after a give-up they keep the copy engine from writing into a dead CTA).
// A stage's full barrier is not re-armed after its last copy, so the parity of that last phase is still testable.
__device__ __noinline__ void loader_drain(uint32_t bars, volatile int* abort_flag, int cg, int cq, int cv, int nfull) {
#pragma unroll 1
  for (int st = 0; st < 3; st++) {
    const int issued = st == 0 ? cg : (st == 1 ? cq : cv);
    const int fb = st == 0 ? B_G_FULL : (st == 1 ? B_QK_FULL : B_V_FULL);
    const int nb = st == 1 ? nfull : 2;
    for (int c = max(0, issued - nb); c < issued; c++)
      if (!mbar_wait_drain(bars + 8u * (uint32_t)(fb + c % nb), (uint32_t)((c / nb) & 1), abort_flag))
        atomicCAS(const_cast<int*>(abort_flag), 0, E_DRAIN + fb);
  }
}

template <int FE>
__device__ void role_loader(const ChunkParams& p, const TmaMaps& m, const Ctx& x, int lane) {
  // Three independent copy streams (g; q and k; v), each with its own full / empty barriers: the gate tile is free after
  // step A of the chunk two back, q / k after step C of the chunk that had the stage (two back, three back with raw
  // gates), v only once MMA2 has read it.  ONE lane
  // serves all three by polling the empty barriers without blocking: a blocking wait of one stream (or of a second
  // lane of this warp, which shares the warp's single scheduling slot) would delay the refill of the others by its
  // suspend time, and the refill latency of q / k sits on the chain  copy -> step B -> step C -> inverse -> MMA2.
  if (lane != 0) return;
  const int n = x.nchunks;
  typedef Raw<FE> R;
  int cg = 0, cq = 0, cv = 0;                 // next chunk of each stream
  int sq = 0;                                 // q / k stage of chunk cq, and the parity of its empty barrier
  uint32_t pq = 1;
  unsigned idle = 0;
  unsigned long long t_idle = 0;
#pragma unroll 1
  while (cg < n || cq < n || cv < n) {
    bool progressed = false;
    if (cq < n) {
      if (mbar_test_wait(x.bar(B_QK_EMPTY + sq), pq)) {
        const uint32_t raw = smem_u32(x.smem + R::OFF_QK + sq * 16384);
        const int tok0 = (int)(x.t0 + (long long)cq * C);
        const uint32_t full = x.bar(B_QK_FULL + cq % R::NFULL);
        tma::mbar_arrive_expect_tx(full, 2u * 8192u);
        tma::load_tile(raw, &m.q, x.h, tok0, full);
        tma::load_tile(raw + 8192, &m.k, x.h, tok0, full);
        cq++;
        if (++sq == R::NQK) { sq = 0; pq ^= 1; }
        progressed = true;
      }
    }
    if (cg < n) {
      const int s = cg & 1;
      if (mbar_test_wait(x.bar(B_G_EMPTY + s), (uint32_t)(((cg >> 1) & 1) ^ 1))) {
        const int tok0 = (int)(x.t0 + (long long)cg * C);
        const uint32_t full = x.bar(B_G_FULL + s);
        tma::mbar_arrive_expect_tx(full, (uint32_t)R::G_BYTES);
        tma::load_tile(smem_u32(x.smem + R::OFF_G + s * R::G_BYTES), &m.g, x.h, tok0, full);
        cg++;
        progressed = true;
      }
    }
    if (cv < n) {
      const int s = cv & 1;
      if (mbar_test_wait(x.bar(B_V_EMPTY + s), (uint32_t)(((cv >> 1) & 1) ^ 1))) {
        const int tok0 = (int)(x.t0 + (long long)cv * C);
        tma::mbar_arrive_expect_tx(x.bar(B_V_FULL + s), 8192u);
        tma::load_tile(smem_u32(x.smem + s * STAGE + CS_V), &m.v, x.h, tok0, x.bar(B_V_FULL + s));
        cv++;
        progressed = true;
      }
    }
    if (progressed) {
      idle = 0;
      t_idle = 0;
    } else {
      // nothing to refill yet: back off briefly; give up like every other wait of the kernel does
      __nanosleep(32);
      if (*x.abort_flag != 0) break;
      if ((++idle & 1023u) == 0) {
        const unsigned long long now = global_timer_ns();
        if (t_idle == 0) t_idle = now;
        else if (loader_idle_expired(now - t_idle, x.abort_flag)) break;
      }
    }
  }
  loader_drain(x.bars, x.abort_flag, cg, cq, (p.debug_flags & DBG_STALL_V_STREAM) ? 0 : cv, R::NFULL);
}

// Beta of one token row of a chunk: the raw bits are fetched a chunk of the group ahead, the activation follows at their use
// (right behind the load it would hold the warp for the latency of global memory).
template <int FE>
__device__ __forceinline__ uint32_t load_beta(const ChunkParams& p, const Ctx& x, int c, int row) {
  if (row >= x.len - c * C) return 0;
  const long long at = (x.t0 + (long long)c * C + row) * p.ldbeta + x.h;
  return FE == 1 ? reinterpret_cast<const uint32_t*>(p.beta)[at] : reinterpret_cast<const uint16_t*>(p.beta)[at];
}
template <int FE>
__device__ __forceinline__ float activate_beta(uint32_t raw) { return FE == 1 ? __uint_as_float(raw) : sigmoidf_rel(bf16_lo(raw)); }

// ------------------------------------------------------------------------------------------------ prep warps
// Step A's exponents, clamped, of a chunk (its first token: t0) in which a gate decays without bound or is not a number.
// Taking the sum of such a gate's token group off the inclusive one has cancelled what precedes the group: here that is added
// up apart, so that the tokens in front keep their exponents.  Out of line and from the gates in global memory (the tile may
// be refilled by now), since elsewhere both forms are as good and any other code in step A is felt: with the same sums
// beside the others 1 x 8192 at 96 heads took 621 us instead of 609.  1 x 4096 at 96 heads, fp32 gates: 243 us in range, 253
// with a reset in every sixteenth chunk.
template <int FE>
__device__ __noinline__ void wide_exponents(const ChunkParams& p, long long t0, int nvalid, int h, int ptid, float2 (&e)[4][2]) {
  const int lane = ptid & 31, ch = 16 * (ptid >> 5) + 4 * (lane & 3);
  const long long ld = p.ldg, at = t0 * ld + (long long)h * D + ch;
  const void* g = FE == 1 ? static_cast<const void*>(static_cast<const float*>(p.g) + at) : static_cast<const void*>(static_cast<const __nv_bfloat16*>(p.g) + at);
  const float* dt_bias = p.dt_bias + h * D + ch;
  const int tg = lane >> 2, sw = ((tg ^ (tg >> 1)) & 1) << 1;
  const bool first = tg < 4, p1 = (tg & 3) >= 1, p2 = (tg & 3) >= 2;
  const float2 zero = make_float2(0.0f, 0.0f), unit = FE == 1 ? make_float2(LOG2E, LOG2E) : make_float2(p.lower_bound * LOG2E, p.lower_bound * LOG2E);
  const float m1 = FE == 0 ? -LOG2E * __expf(p.A_log[h]) : 0.0f;
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const int tok = (4 * tg + sw) ^ j;
    e[j][0] = e[j][1] = zero;
    if (tok >= nvalid) continue;
    if (FE == 1) {
      const float4 f = *reinterpret_cast<const float4*>(static_cast<const float*>(g) + tok * ld);
      e[j][0] = make_float2(f.x, f.y);
      e[j][1] = make_float2(f.z, f.w);
    } else {
      const uint2 f = *reinterpret_cast<const uint2*>(static_cast<const __nv_bfloat16*>(g) + tok * ld);
#pragma unroll
      for (int i = 0; i < 2; i++) {
        const uint32_t w = i ? f.y : f.x;
        e[j][i] = make_float2(rcpf(1.0f + ex2f(fmaf(bf16_lo(w), m1, m1 * dt_bias[2 * i]))), rcpf(1.0f + ex2f(fmaf(bf16_hi(w), m1, m1 * dt_bias[2 * i + 1]))));
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 2; i++) {
    e[0][i] = mul2(e[0][i], unit);
    e[1][i] = fma2(e[1][i], unit, e[0][i]);
    e[2][i] = mul2(e[2][i], unit);
    e[3][i] = fma2(e[3][i], unit, e[2][i]);
    float2 inc = add2(e[1][i], e[3][i]), base = zero, t;
    t.x = __shfl_up_sync(0xffffffffu, inc.x, 4);
    t.y = __shfl_up_sync(0xffffffffu, inc.y, 4);
    if (p1) { inc = add2(inc, t); base = t; }
    t.x = __shfl_up_sync(0xffffffffu, inc.x, 8);
    t.y = __shfl_up_sync(0xffffffffu, inc.y, 8);
    if (p2) { inc = add2(inc, t); base = add2(base, t); }
    t.x = __shfl_sync(0xffffffffu, inc.x, (lane & 19) | 12);
    t.y = __shfl_sync(0xffffffffu, inc.y, (lane & 19) | 12);
    if (first) base = make_float2(base.x - t.x, base.y - t.y);
    const float2 b0 = add2(base, sw ? e[3][i] : zero), b1 = add2(base, sw ? zero : e[1][i]);
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const float2 x = add2(e[j][i], j < 2 ? b0 : b1);
      e[j][i] = first ? make_float2(fminf(x.x, 126.0f), fminf(x.y, 126.0f)) : make_float2(fmaxf(x.x, -126.0f), fmaxf(x.y, -126.0f));
    }
  }
}

// Operand preparation.  A warp owns 16 channels of all 32 tokens, a lane four channels (its quad) of four tokens (its token
// group): the cumulative decay then runs along the lanes of one warp and never leaves registers, so a chunk costs the group
// ONE barrier (in front of the intra-chunk products, which contract over all channels).  Of the four tokens of a lane, token
// (j ^ sw) comes j-th, sw = 0 or 2 by token group: with that order every 16- and 8-byte access to the swizzled tiles is free
// of bank conflicts (the eight or sixteen lanes of one phase touch rows that differ in the swizzle bits), and the address of
// step j is that of step 0 with j flipped into the row and chunk bits.
// (A layout of four tokens x 128 channels per warp sent the cumulative sums through shared memory and two more barriers.)
template <int FE>
__device__ void role_prep(const ChunkParams& p, const Ctx& x, int grp, int ptid) {
  const int pw = ptid >> 5, lane = ptid & 31;
  const int quad = lane & 3, tg = lane >> 2;
  const int sw = ((tg ^ (tg >> 1)) & 1) << 1;
  const int tok0 = 4 * tg + sw;                        // token of step j: tok0 ^ j
  const bool first = tg < 4;                           // tokens 0-15
  const int s = grp;                                   // the group's stage
  const int bar_id = 1 + grp;
  typedef Raw<FE> R;
  uint8_t* st = x.smem + s * STAGE;
  const uint8_t* g_tile = x.smem + R::OFF_G + s * R::G_BYTES;
  float* norm = reinterpret_cast<float*>(x.smem + OFF_NORM) + s * 128;
  int sq = grp, fq = grp;                              // q / k stage of the chunk, its full barrier and parity
  uint32_t pq = 0;
  // offsets of step 0 (step j: ^ j * 0x90 for rows of 128 bytes, ^ j * 0xa0 for kr).  kr is MN-major in the 128-byte swizzle
  // with 32-byte base: token rows of 32 channels, 32-byte pieces XOR-ed with (token % 4), four rows to a 512-byte atom,
  // atoms 512 bytes apart along the channels and 2048 along the tokens.  (Written out: through a helper with the general
  // form the raw-gate instantiations spill 16 bytes more and 1 x 32768 with checkpoints takes 5 % longer.)
  const uint32_t off_f32 = (uint32_t)(tok0 * 128 + (((4 * (pw & 1) + quad) ^ (tok0 & 7)) << 4));
  const uint32_t off_g = FE == 1 ? (uint32_t)((pw >> 1) * 4096) + off_f32 : 0u;
  const uint32_t off_kd = (uint32_t)((pw >> 1) * 8192) + off_f32;
  const uint32_t off_b16 = (uint32_t)((pw >> 2) * 4096 + tok0 * 128 + (((2 * (pw & 3) + (quad >> 1)) ^ (tok0 & 7)) << 4) + (quad & 1) * 8);
  const uint32_t off_kr = (uint32_t)((pw >> 1) * 512 + tg * 2048 + sw * 128 + (((2 * (pw & 1) + (quad >> 1)) ^ sw) << 5) + (quad & 1) * 16);
  float m1 = 0.0f;
  float2 m0[2];
  if (FE == 0) {
    m1 = -LOG2E * __expf(p.A_log[x.h]);
    const float* b = p.dt_bias + x.h * D + 16 * pw + 4 * quad;       // (any alignment)
    m0[0] = make_float2(m1 * b[0], m1 * b[1]);
    m0[1] = make_float2(m1 * b[2], m1 * b[3]);
  }
  const float scale = p.scale;
  volatile int* range_flag = reinterpret_cast<volatile int*>(x.smem + OFF_MISC + 12);
  // Warps 1 and 5 have no block of the intra-chunk products: 5 looks after beta and zeroes, once, the upper right block of M.
  const bool no_block = (pw & 3) == 1;
  uint32_t beta_next = 0;                              // one own chunk ahead
  if (pw == 5) {
    if (grp < x.nchunks) beta_next = load_beta<FE>(p, x, grp, lane);
    const uint4 z = make_uint4(0u, 0u, 0u, 0u);
    *reinterpret_cast<uint4*>(st + CS_M + kmajor_f32_off(lane & 15, 16 + 4 * (lane >> 4), 0)) = z;
    *reinterpret_cast<uint4*>(st + CS_M + kmajor_f32_off(lane & 15, 24 + 4 * (lane >> 4), 0)) = z;
  }
#pragma unroll 1
  for (int c = grp; c < x.nchunks; c += PREP_GROUPS) {
    const uint32_t par = (uint32_t)((c >> 1) & 1);
    const int nvalid = min(C, x.len - c * C);
    // alternates so that step C of the chunk before may still read the other half
    float* beta_s = reinterpret_cast<float*>(x.smem + OFF_BETA) + (2 * s + (int)par) * 32;
    uint8_t* qk = x.smem + R::OFF_QK + sq * 16384;       // q, then k
    PROF_BEGIN;
    if (FE == 0) {
      x.wait(B_QK_FULL + fq, pq, E_PREP);
      // Square sums of the rows: the diagonal of rows x rows^T on mma.sync, whose B operand is the A operand's registers.
      // Warp w takes the 16 rows (w & 1) of q (w & 2: of k) over half of the channels; exact products, fp32 sums.  They
      // travel to the other warps while the gates are worked out.
      const int row = 16 * (pw & 1) + (lane & 15);
      const uint32_t tile = smem_u32(qk + ((pw & 2) ? 8192 : 0)) + (uint32_t)((pw >> 2) * 4096 + row * 128);
      float d0[4] = {0.0f, 0.0f, 0.0f, 0.0f}, d1[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
      for (int kt = 0; kt < 4; kt++) {
        uint32_t a[4];
        ldmatrix_x4(a, tile + (uint32_t)(((2 * kt + (lane >> 4)) ^ (row & 7)) << 4));
        mma_bf16(d0, a, a[0], a[2]);                     // columns = rows 0-7: diagonal in the first two registers
        mma_bf16(d1, a, a[1], a[3]);                     // columns = rows 8-15: diagonal in the last two
      }
      if ((tg >> 1) == quad) {                           // columns 2 quad, 2 quad + 1 against row tg
        float* n = norm + (pw >> 2) * 64 + ((pw & 2) ? 32 : 0) + 16 * (pw & 1) + tg;
        n[0] = (tg & 1) ? d0[1] : d0[0];
        n[8] = (tg & 1) ? d1[3] : d1[2];
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(x.bar(B_NORM + s));
    }
    x.wait(B_G_FULL + s, par, E_PREP);
    PROF_STAMP(2, 11);

    // ---- A: gate activation + cumulative log2-decay relative to r = the one after token 15 (tokens 0-15: own sum - r >= 0,
    // tokens 16-31: their own partial sum <= 0)
    float2 e[4][2], er[2], el[2];                        // exponents by step and channel pair; 2^r, 2^(G31 - r)
    {
      float2 unit;
      unit.x = unit.y = (FE == 1) ? LOG2E : p.lower_bound * LOG2E;
      float2 a[4][2];
      if (FE == 1) {
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const float4 f = *reinterpret_cast<const float4*>(g_tile + (off_g ^ (j * 0x90)));
          a[j][0] = make_float2(f.x, f.y);
          a[j][1] = make_float2(f.z, f.w);
        }
      } else {
        // log2-decay = lower_bound log2(e) sigmoid(x), x = exp(A_log) (g + dt_bias); sigmoid(x) = 1 / (1 + 2^(-x log2 e))
        // with the exponent argument formed by one fused multiply-add per element
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const uint2 f = *reinterpret_cast<const uint2*>(g_tile + (off_b16 ^ (j * 0x90)));
#pragma unroll
          for (int i = 0; i < 2; i++) {
            const uint32_t w = i ? f.y : f.x;
            const float2 y = fma2(make_float2(bf16_lo(w), bf16_hi(w)), make_float2(m1, m1), m0[i]);
            const float2 d = add2(make_float2(ex2f(y.x), ex2f(y.y)), make_float2(1.0f, 1.0f));
            a[j][i] = make_float2(rcpf(d.x), rcpf(d.y));
          }
        }
      }
      if (nvalid < C) {                                  // rows of the next sequence (last chunk only): no decay
#pragma unroll
        for (int j = 0; j < 4; j++)
          if ((tok0 ^ j) >= nvalid) a[j][0] = a[j][1] = make_float2(0.0f, 0.0f);
      }
      const bool p1 = (tg & 3) >= 1, p2 = (tg & 3) >= 2;
      float2 own[2], oth[2];                             // sums over this lane's half of the chunk and over the other half
#pragma unroll
      for (int i = 0; i < 2; i++) {
        // sums inside the two token pairs, the unit conversion fused into the additions
        e[0][i] = mul2(a[0][i], unit);
        e[1][i] = fma2(a[1][i], unit, e[0][i]);
        e[2][i] = mul2(a[2][i], unit);
        e[3][i] = fma2(a[3][i], unit, e[2][i]);
        const float2 sum = add2(e[1][i], e[3][i]);
        // inclusive sum over the four token groups of the half
        float2 inc = sum, t;
        t.x = __shfl_up_sync(0xffffffffu, inc.x, 4);
        t.y = __shfl_up_sync(0xffffffffu, inc.y, 4);
        if (p1) inc = add2(inc, t);
        t.x = __shfl_up_sync(0xffffffffu, inc.x, 8);
        t.y = __shfl_up_sync(0xffffffffu, inc.y, 8);
        if (p2) inc = add2(inc, t);
        own[i].x = __shfl_sync(0xffffffffu, inc.x, (lane & 19) | 12);
        own[i].y = __shfl_sync(0xffffffffu, inc.y, (lane & 19) | 12);
        oth[i].x = __shfl_sync(0xffffffffu, inc.x, ((lane & 19) | 12) ^ 16);
        oth[i].y = __shfl_sync(0xffffffffu, inc.y, ((lane & 19) | 12) ^ 16);
        // what precedes this group in its half, less r in the first half; the later token pair of the group adds the earlier one
        float2 base = make_float2(inc.x - sum.x, inc.y - sum.y);
        if (first) base = make_float2(base.x - own[i].x, base.y - own[i].y);
        const float2 zero = make_float2(0.0f, 0.0f);
        const float2 b0 = add2(base, sw ? e[3][i] : zero), b1 = add2(base, sw ? zero : e[1][i]);
        e[0][i] = add2(e[0][i], b0);
        e[1][i] = add2(e[1][i], b0);
        e[2][i] = add2(e[2][i], b1);
        e[3][i] = add2(e[3][i], b1);
      }
      // The gates are in registers: the tile may be refilled.  Not right behind the loads, which may sit behind hundreds of
      // cycles of other traffic: the shuffles behind `own` need every value that a lane has read.
      __syncwarp();
      if (lane == 0) mbar_arrive_after(x.bar(B_G_EMPTY + s), own[0].x);
      // Range of the primed operands: with gates <= 0 no exponent exceeds the decay of its half of the chunk.  Beyond 2^126
      // they are clamped and the intra-chunk products of this chunk are no longer exact: report it.  (A gate that is not a
      // number goes the same way, unreported: it shows from its own token on.)
      const float least = min_nan(min_nan(min_nan(own[0].x, own[0].y), min_nan(own[1].x, own[1].y)), min_nan(min_nan(oth[0].x, oth[0].y), min_nan(oth[1].x, oth[1].y)));
      if (__any_sync(0xffffffffu, !(least >= -126.0f))) {
        const float number = fminf(fminf(fminf(own[0].x, own[0].y), fminf(own[1].x, own[1].y)), fminf(fminf(oth[0].x, oth[0].y), fminf(oth[1].x, oth[1].y)));
        if (number < -126.0f) *range_flag = 1;
        // Down to -2048 what has cancelled is less than 2^-12 of an exponent: a clamp is enough (1 x 4096 with every chunk out
        // of range 251 us, 360 through the call).  Raw gates leave the range only under a lower bound of the caller's or as NaN.
        if (FE == 0 || __any_sync(0xffffffffu, !(least >= -2048.0f))) {
          float2 w[4][2];
          wide_exponents<FE>(p, x.t0 + (long long)c * C, nvalid, x.h, ptid, w);
#pragma unroll
          for (int j = 0; j < 4; j++) { e[j][0] = w[j][0]; e[j][1] = w[j][1]; }
        } else {
#pragma unroll
          for (int j = 0; j < 4; j++)
#pragma unroll
            for (int i = 0; i < 2; i++)
              e[j][i] = first ? make_float2(fminf(e[j][i].x, 126.0f), fminf(e[j][i].y, 126.0f)) : make_float2(fmaxf(e[j][i].x, -126.0f), fmaxf(e[j][i].y, -126.0f));
        }
      }
#pragma unroll
      for (int i = 0; i < 2; i++) {
        const float2 r = first ? own[i] : oth[i], l = first ? oth[i] : own[i];
        er[i] = make_float2(ex2f(r.x), ex2f(r.y));
        el[i] = make_float2(ex2f(l.x), ex2f(l.y));
      }
      if (tg == 0) {                                     // 2^G31 (the decay slot c & 3 was last read four chunks ago)
        const float2 d0 = mul2(er[0], el[0]), d1 = mul2(er[1], el[1]);
        *reinterpret_cast<float4*>(x.smem + OFF_DEC + (c & 3) * (D * 4) + (16 * pw + 4 * quad) * 4) = make_float4(d0.x, d0.y, d1.x, d1.y);
      }
    }
    PROF_STAMP(2, 12);
    if (pw == 5) {
      beta_s[lane] = lane < nvalid ? activate_beta<FE>(beta_next) : 0.0f;
      if (c + PREP_GROUPS < x.nchunks) beta_next = load_beta<FE>(p, x, c + PREP_GROUPS, lane);
    }

    // ---- B: L2 norm and decayed operand tiles.  [kd ; qd] is written as soon as MMA1 of the chunk two back has read the
    // stage; kr waits in registers until MMA3 has released the rest.
    float qinv = 1.0f, kinv = 1.0f;                      // of the token of step `quad`
    if (FE == 1) x.wait(B_QK_FULL + fq, pq, E_PREP);
    PROF_STAMP(2, 13);
    if (FE == 0) {
      x.wait(B_NORM + s, par, E_PREP);
      const float* n = norm + (tok0 ^ quad);
      qinv = rsqrtf(fmaxf(n[0] + n[64], 1e-12f));        // x / max(||x||, 1e-6)
      kinv = rsqrtf(fmaxf(n[32] + n[96], 1e-12f));
    }
    x.wait(B_KDQD_EMPTY + s, par ^ 1, E_PREP);
    PROF_STAMP(2, 14);
    float2 kr[4][2];
    {
      const float2 sc2 = make_float2(scale, scale);
      const float2 eq[2] = {mul2(er[0], sc2), mul2(er[1], sc2)};       // scale of q rides on 2^r here and on M below
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const uint32_t o = off_b16 ^ (j * 0x90);
        uint2 q2 = *reinterpret_cast<const uint2*>(qk + o), k2 = *reinterpret_cast<const uint2*>(qk + 8192 + o);
        if (nvalid < C && (tok0 ^ j) >= nvalid) { q2 = make_uint2(0u, 0u); k2 = make_uint2(0u, 0u); }   // rows of the next sequence
        float2 qn[2] = {make_float2(bf16_lo(q2.x), bf16_hi(q2.x)), make_float2(bf16_lo(q2.y), bf16_hi(q2.y))};
        float2 kn[2] = {make_float2(bf16_lo(k2.x), bf16_hi(k2.x)), make_float2(bf16_lo(k2.y), bf16_hi(k2.y))};
        if (FE == 0) {
          const float qi = __shfl_sync(0xffffffffu, qinv, (lane & 28) | j), ki = __shfl_sync(0xffffffffu, kinv, (lane & 28) | j);
#pragma unroll
          for (int i = 0; i < 2; i++) {
            qn[i] = mul2(qn[i], make_float2(qi, qi));
            kn[i] = mul2(kn[i], make_float2(ki, ki));
          }
        }
        float2 kd[2], qd[2], ki[2], kt[2], qt[2];
#pragma unroll
        for (int i = 0; i < 2; i++) {
          const float2 E = make_float2(ex2f(e[j][i].x), ex2f(e[j][i].y)), Ei = make_float2(ex2f(-e[j][i].x), ex2f(-e[j][i].y));
          kd[i] = mul2(kn[i], E);
          qd[i] = mul2(qn[i], E);
          ki[i] = mul2(kn[i], Ei);
          kt[i] = mul2(kd[i], er[i]);
          qt[i] = mul2(qd[i], eq[i]);
          kr[j][i] = mul2(ki[i], el[i]);
        }
        // in place: the decayed bf16 tiles of the intra-chunk products replace the raw q / k tiles
        *reinterpret_cast<uint2*>(qk + 8192 + o) = make_uint2(pack_bf16(kd[0].x, kd[0].y), pack_bf16(kd[1].x, kd[1].y));
        *reinterpret_cast<uint2*>(qk + o) = make_uint2(pack_bf16(qd[0].x, qd[0].y), pack_bf16(qd[1].x, qd[1].y));
        *reinterpret_cast<uint2*>(st + KI + o) = make_uint2(pack_bf16(ki[0].x, ki[0].y), pack_bf16(ki[1].x, ki[1].y));
        // tf32 operands of the state products: [kd ; qd] K-major (row = token, 32 + token), kr MN-major
        const uint32_t f = off_kd ^ (j * 0x90);
        *reinterpret_cast<float4*>(st + CS_KDQD + f) = make_float4(kt[0].x, kt[0].y, kt[1].x, kt[1].y);
        *reinterpret_cast<float4*>(st + CS_KDQD + 4096 + f) = make_float4(qt[0].x, qt[0].y, qt[1].x, qt[1].y);
      }
    }
    PROF_STAMP(2, 27);
    fence_proxy_async();
    __syncwarp();
    if (lane == 0) mbar_arrive(x.bar(B_KDQD_FULL + s));
    named_bar_sync(bar_id, PREP_THREADS);
    PROF_STAMP(2, 28);

    // ---- C: one 16x16 block of A = kd' ki'^T (warps 0-3) or M = qd' ki'^T (warps 4-7) per warp
    {
      const int which = pw >> 2, rb = (pw >> 1) & 1, cb = pw & 1;
      const int g = lane >> 2, t = lane & 3;
      const int i0 = 16 * rb + g, i1 = i0 + 8;
      float acc[2][4];
#pragma unroll
      for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = 0.0f;
      if (!no_block) {
        // K step kt reads 16-byte chunks 2 kt, 2 kt + 1 of a row: two bits of the swizzled address flipped, then the second block
        const uint32_t a_addr = smem_u32(qk + (which ? 0 : 8192)) + rawtile_off(16 * rb + (lane & 7) + ((lane >> 3) & 1) * 8, (lane >> 4) * 8);
        const uint32_t b_addr = smem_u32(st + KI) + rawtile_off(16 * cb + 8 * (lane >> 4) + (lane & 7), ((lane >> 3) & 1) * 8);
#pragma unroll
        for (int kh = 0; kh < 8; kh += 2) {
          uint32_t a[2][4], b[2][4];
#pragma unroll
          for (int i = 0; i < 2; i++) {
            const int kt = kh + i;
            ldmatrix_x4(a[i], (a_addr ^ ((kt & 3) << 5)) + (kt >> 2) * 4096);
            ldmatrix_x4(b[i], (b_addr ^ ((kt & 3) << 5)) + (kt >> 2) * 4096);
          }
#pragma unroll
          for (int i = 0; i < 2; i++) {
            mma_bf16(acc[0], a[i], b[i][0], b[i][1]);
            mma_bf16(acc[1], a[i], b[i][2], b[i][3]);
          }
        }
      }
      __syncwarp();
      // The q / k tiles are no longer read: the last product needs every fragment that the warp has loaded.
      if (lane == 0) mbar_arrive_after(x.bar(B_QK_EMPTY + sq), acc[0][0]);
      if (rb == cb) {                                          // diagonal block: strictly lower for A, lower for M
        const int m = g + which;
#pragma unroll
        for (int nt = 0; nt < 2; nt++) {
          const int j = 8 * nt + 2 * t;
          acc[nt][0] = j < m ? acc[nt][0] : 0.0f;
          acc[nt][1] = j + 1 < m ? acc[nt][1] : 0.0f;
          acc[nt][2] = j < m + 8 ? acc[nt][2] : 0.0f;
          acc[nt][3] = j + 1 < m + 8 ? acc[nt][3] : 0.0f;
        }
      }
      PROF_STAMP(2, 15);
      if (which == 0 && !no_block) {
        x.wait(B_L_EMPTY + s, par ^ 1, E_PREP);
        float* Lsm = reinterpret_cast<float*>(x.smem + OFF_L) + s * C * LS;
        const float b0 = beta_s[i0], b1 = beta_s[i1];
#pragma unroll
        for (int nt = 0; nt < 2; nt++) {
          const int j = 16 * cb + 8 * nt + 2 * t;
          *reinterpret_cast<float2*>(Lsm + i0 * LS + j) = make_float2(acc[nt][0] * b0, acc[nt][1] * b0);
          *reinterpret_cast<float2*>(Lsm + i1 * LS + j) = make_float2(acc[nt][2] * b1, acc[nt][3] * b1);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(x.bar(B_L_FULL + s));      // the inverse of this chunk may start
      }
      PROF_STAMP(2, 16);
      // ---- D: the operands of MMA3 go out once the tensor core has released the rest of the stage
      x.wait(B_CONS_EMPTY + s, par ^ 1, E_PREP);
      PROF_STAMP(2, 17);
#pragma unroll
      for (int j = 0; j < 4; j++)
        *reinterpret_cast<float4*>(st + CS_KR + (off_kr ^ (j * 0xa0))) = make_float4(kr[j][0].x, kr[j][0].y, kr[j][1].x, kr[j][1].y);
      if (which == 1 && !no_block) {
#pragma unroll
        for (int nt = 0; nt < 2; nt++) {
          const int j = 16 * cb + 8 * nt + 2 * t;
          *reinterpret_cast<float2*>(st + CS_M + kmajor_f32_off(i0, j, 0)) = make_float2(acc[nt][0] * scale, acc[nt][1] * scale);
          *reinterpret_cast<float2*>(st + CS_M + kmajor_f32_off(i1, j, 0)) = make_float2(acc[nt][2] * scale, acc[nt][3] * scale);
        }
      }
    }
    PROF_STAMP(2, 29);
    fence_proxy_async();
    __syncwarp();
    if (lane == 0) mbar_arrive(x.bar(B_P1_FULL + s));
    sq += PREP_GROUPS;
    if (sq >= R::NQK) sq -= R::NQK;
    fq += PREP_GROUPS;
    if (fq >= R::NFULL) { fq -= R::NFULL; pq ^= 1; }
  }
}

// ------------------------------------------------------------------------------------------------ inverse warps
// T = (I + L)^-1 for the strictly lower triangular fp32 L [32][32] of a chunk (row stride LS), by one warp:
//   1. the two 16x16 diagonal blocks by forward substitution in fp32 registers, one half-warp per block, lane = column
//      (16 dependent rows instead of 32), in place;
//   2. the off-diagonal block T10 = -(T11 L10) T00 as two 16x16x16 products on mma.sync (tf32 operands, fp32 accumulation; T
//      is consumed as a tf32 / bf16 tensor-core operand anyway).  The accumulators of the first product are the A operand of
//      the second as they lie: its contraction index is taken in the order 0, 2, 4, 6, 1, 3, 5, 7 on both sides.
// Then Tb = T diag(beta) goes out as the tf32 and bf16 operand tiles of MMA2: the diagonal blocks row by row, T10 from the
// accumulators; the upper right block is zeroed once.
__device__ void role_inverse(const Ctx& x, int which, int lane) {
  const int blk = lane >> 4, cl = lane & 15;
  const int g = lane >> 2, t = lane & 3;
  const int s = which;                                 // the warp's stage
  float* Lsm = reinterpret_cast<float*>(x.smem + OFF_L) + s * C * LS;
  uint8_t* tb = x.smem + s * STAGE + CS_TB;
  uint8_t* tbh = x.smem + OFF_TBH + s * 2048;
  {
    const uint4 z = make_uint4(0u, 0u, 0u, 0u);
    *reinterpret_cast<uint4*>(tb + kmajor_f32_off(cl, 16 + 4 * blk, 0)) = z;
    *reinterpret_cast<uint4*>(tb + kmajor_f32_off(cl, 24 + 4 * blk, 0)) = z;
    *reinterpret_cast<uint4*>(tbh + kmajor_b16_sw64_off(cl, 16 + 8 * blk)) = z;
  }
#pragma unroll 1
  for (int c = which; c < x.nchunks; c += 2) {
    const uint32_t par = (uint32_t)((c >> 1) & 1);
    x.wait(B_L_FULL + s, par, E_INV);
    // (beta of this chunk is replaced four chunks on, behind MMA3 of this one)
    const float* lbeta = reinterpret_cast<const float*>(x.smem + OFF_BETA) + (2 * s + (int)par) * 32;
    PROF_BEGIN;
    // ---- 1: diagonal blocks.  L is zero on and above its diagonal, so a row takes whole groups of four columns.
    {
      const float* Lb = Lsm + blk * 16 * LS + blk * 16;
      float2 T[8];
#pragma unroll
      for (int i = 0; i < 8; i++) T[i] = make_float2(2 * i == cl ? 1.0f : 0.0f, 2 * i + 1 == cl ? 1.0f : 0.0f);
#pragma unroll
      for (int i = 1; i < 16; i++) {
        float2 a0 = make_float2(0.0f, 0.0f), a1 = a0;
#pragma unroll
        for (int j = 0; j < i; j += 4) {
          const float4 l4 = *reinterpret_cast<const float4*>(Lb + i * LS + j);
          a0 = fma2(make_float2(l4.x, l4.y), T[j / 2], a0);
          a1 = fma2(make_float2(l4.z, l4.w), T[j / 2 + 1], a1);
        }
        const float2 a = add2(a0, a1);
        if (i & 1) T[i / 2].y -= a.x + a.y;
        else T[i / 2].x -= a.x + a.y;
      }
      __syncwarp();                                   // every lane has read its diagonal block
      float* Tb_ = Lsm + blk * 16 * LS + blk * 16;
#pragma unroll
      for (int i = 0; i < 16; i++) Tb_[i * LS + cl] = (i & 1) ? T[i / 2].y : T[i / 2].x;
    }
    PROF_STAMP(3, 25);
    __syncwarp();
    x.wait(B_CONS_EMPTY + s, par ^ 1, E_INV);         // MMA2 of the chunk two back has read Tb
    // ---- 2: T10 = -(T11 L10) T00
    float acc[2][4], out10[2][4];
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
      for (int j = 0; j < 4; j++) acc[i][j] = out10[i][j] = 0.0f;
    {
      const float* T11 = Lsm + 16 * LS + 16;
      const float* L10 = Lsm + 16 * LS;
#pragma unroll
      for (int kt = 0; kt < 2; kt++) {
        const uint32_t a[4] = {__float_as_uint(T11[g * LS + 8 * kt + t]), __float_as_uint(T11[(g + 8) * LS + 8 * kt + t]),
                               __float_as_uint(T11[g * LS + 8 * kt + t + 4]), __float_as_uint(T11[(g + 8) * LS + 8 * kt + t + 4])};
#pragma unroll
        for (int nt = 0; nt < 2; nt++)
          mma_tf32(acc[nt], a, __float_as_uint(L10[(8 * kt + t) * LS + 8 * nt + g]), __float_as_uint(L10[(8 * kt + t + 4) * LS + 8 * nt + g]));
      }
#pragma unroll
      for (int kt = 0; kt < 2; kt++) {
        const uint32_t a[4] = {__float_as_uint(acc[kt][0]), __float_as_uint(acc[kt][2]), __float_as_uint(acc[kt][1]), __float_as_uint(acc[kt][3])};
#pragma unroll
        for (int nt = 0; nt < 2; nt++)
          mma_tf32(out10[nt], a, __float_as_uint(Lsm[(8 * kt + 2 * t) * LS + 8 * nt + g]), __float_as_uint(Lsm[(8 * kt + 2 * t + 1) * LS + 8 * nt + g]));
      }
    }
    // Tb, diagonal blocks: lane = row
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const int c0 = 16 * blk + 8 * q;
      const float4 ta = *reinterpret_cast<const float4*>(Lsm + lane * LS + c0);
      const float4 tc = *reinterpret_cast<const float4*>(Lsm + lane * LS + c0 + 4);
      const float4 ba = *reinterpret_cast<const float4*>(lbeta + c0);
      const float4 bb = *reinterpret_cast<const float4*>(lbeta + c0 + 4);
      const float4 va = make_float4(ta.x * ba.x, ta.y * ba.y, ta.z * ba.z, ta.w * ba.w);
      const float4 vb = make_float4(tc.x * bb.x, tc.y * bb.y, tc.z * bb.z, tc.w * bb.w);
      *reinterpret_cast<float4*>(tb + kmajor_f32_off(lane, c0, 0)) = va;
      *reinterpret_cast<float4*>(tb + kmajor_f32_off(lane, c0 + 4, 0)) = vb;
      *reinterpret_cast<uint4*>(tbh + kmajor_b16_sw64_off(lane, c0)) =
          make_uint4(pack_bf16(va.x, va.y), pack_bf16(va.z, va.w), pack_bf16(vb.x, vb.y), pack_bf16(vb.z, vb.w));
    }
    PROF_STAMP(3, 26);
    // Tb, lower left block
#pragma unroll
    for (int nt = 0; nt < 2; nt++) {
      const int j = 8 * nt + 2 * t;
      const float2 b = *reinterpret_cast<const float2*>(lbeta + j);
      const float2 lo = make_float2(-out10[nt][0] * b.x, -out10[nt][1] * b.y), hi = make_float2(-out10[nt][2] * b.x, -out10[nt][3] * b.y);
      *reinterpret_cast<float2*>(tb + kmajor_f32_off(16 + g, j, 0)) = lo;
      *reinterpret_cast<float2*>(tb + kmajor_f32_off(24 + g, j, 0)) = hi;
      *reinterpret_cast<uint32_t*>(tbh + kmajor_b16_sw64_off(16 + g, j)) = pack_bf16(lo.x, lo.y);
      *reinterpret_cast<uint32_t*>(tbh + kmajor_b16_sw64_off(24 + g, j)) = pack_bf16(hi.x, hi.y);
    }
    // The v tile of a partial last chunk holds another sequence's rows (or worse) past the end of the run: zero them
    // so that they cannot poison MMA2 (their Tb columns are zero, but 0 * NaN is NaN).  MMA2 waits for this warp's
    // INV_FULL arrival.  (The wait for MMA3 of the chunk two back above implies that the v barrier has completed that
    // chunk's phase, so the wait here cannot be satisfied by an older one.)
    if (x.len - c * C < C) {
      x.wait(B_V_FULL + s, par, E_INV);
      const int nvalid = x.len - c * C;
      uint8_t* vt = x.smem + s * STAGE + CS_V;
      for (int i = lane; i < (C - nvalid) * 16; i += 32) {     // whole 128-byte lines of both 64-channel halves
        const int row = nvalid + (i >> 4), piece = i & 15;
        *reinterpret_cast<uint4*>(vt + (piece >> 3) * 4096 + row * 128 + (piece & 7) * 16) = make_uint4(0u, 0u, 0u, 0u);
      }
    }
    PROF_STAMP(3, 27);
    fence_proxy_async();
    __syncwarp();
    if (lane == 0) {
      mbar_arrive(x.bar(B_INV_FULL + s));
      mbar_arrive(x.bar(B_L_EMPTY + s));
    }
    PROF_STAMP(3, 28);
  }
}

// ------------------------------------------------------------------------------------------------ MMA issuer
// Runs on ALL lanes of warp 0 with warp-uniform values only; one elected lane issues the tensor-core instructions
// (predicated inside the asm).  Keeping the control flow convergent lets the compiler hold descriptors, tensor-memory
// addresses and barrier addresses in uniform registers, which is what makes issuing ~34 small MMAs per chunk cheap.
__device__ void role_mma(const Ctx& x, uint32_t tmem_any, bool v_zero_any) {
  const uint32_t go = elect_one();
  const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_any, 0);
  const bool v_zero = __shfl_sync(0xffffffffu, (int)v_zero_any, 0) != 0;
  const int nchunks = __shfl_sync(0xffffffffu, x.nchunks, 0);
  const uint32_t sb = smem_u32(x.smem);
  constexpr uint32_t ID1 = make_idesc(FMT_TF32, 128, 64, 0, 0, 0);
  constexpr uint32_t ID2A = make_idesc(FMT_BF16, 128, 32, 1, 0, 0);
  constexpr uint32_t ID2B = make_idesc(FMT_TF32, 128, 32, 0, 0, 1);
  constexpr uint32_t ID3A = make_idesc(FMT_TF32, 128, 128, 0, 1, 0);
  constexpr uint32_t ID3B = make_idesc(FMT_TF32, 128, 32, 0, 0, 0);
  const uint32_t tS = tmem + TM_S;
  // Descriptors of stage 0, built once; a stage or K step only moves the 14-bit start-address field (units of 16
  // bytes), so every other descriptor is one 64-bit add away.
  const uint64_t d_kdqd = make_sdesc(sb + CS_KDQD, 16, 1024, LAYOUT_SW128);
  const uint64_t d_v = make_sdesc(sb + CS_V, 4096, 1024, LAYOUT_SW128);
  const uint64_t d_tbh = make_sdesc(sb + OFF_TBH, 16, 512, LAYOUT_SW64);
  const uint64_t d_tb = make_sdesc(sb + CS_TB, 16, 1024, LAYOUT_SW128);
  const uint64_t d_kr = make_sdesc(sb + CS_KR, 512, 2048, LAYOUT_SW128_BASE32B);
  const uint64_t d_m = make_sdesc(sb + CS_M, 16, 1024, LAYOUT_SW128);
  x.wait(B_S_READY, 0, E_MMA, 0);                  // initial state is in tensor memory
#pragma unroll 1
  for (int c = 0; c < nchunks; c++) {
    const int s = c & 1;
    const uint32_t par = (uint32_t)((c >> 1) & 1);
    const uint64_t so = (uint64_t)(s * (STAGE >> 4));          // stage offset in the start-address field
    const uint64_t so_tbh = (uint64_t)(s * (2048 >> 4));
    const uint32_t tWO = tmem + TM_WO + 64 * s;
    const uint32_t tU = tmem + TM_U + 32 * s;             // U alternates too: MMA2 of the next chunk never overwrites
                                                          // columns that MMA3 of this chunk may still be reading
    x.wait(B_KDQD_FULL + s, par, E_MMA, 0);
    x.wait(B_O_EMPTY + s, par ^ 1, E_MMA, 0);
    tc_fence_after();
    PROF_BEGIN;
#pragma unroll
    for (int ks = 0; ks < 16; ks++)
      mma_ts_tf32_pred(tWO, tS + 8 * ks, d_kdqd + so + (uint64_t)(((ks >> 2) * 8192 + (ks & 3) * 32) >> 4), ID1, ks > 0, go);
    mma_commit_pred(x.bar(B_MMA1_DONE), go);              // the tensor-memory warps may rescale the state
    mma_commit_pred(x.bar(B_KDQD_EMPTY + s), go);         // [kd ; qd] of this stage may be rewritten
    PROF_STAMP(4, 26);
    x.wait(B_V_FULL + s, par, E_MMA, 0);                  // (over long before the inverse is; a wait costs some 150 cycles even so)
    x.wait(B_INV_FULL + s, par, E_MMA, 0);
    tc_fence_after();
    if (!v_zero) {
#pragma unroll
      for (int ks = 0; ks < 2; ks++)
        mma_ss_f16_pred(tU, d_v + so + (uint64_t)((2 * ks * 1024) >> 4), d_tbh + so_tbh + (uint64_t)((ks * 32) >> 4), ID2A, ks > 0, go);
    }
#pragma unroll
    for (int ks = 0; ks < 4; ks++)
      mma_ts_tf32_pred(tU, tWO + 8 * ks, d_tb + so + (uint64_t)((ks * 32) >> 4), ID2B, (ks > 0) || !v_zero, go);
    PROF_STAMP(4, 27);
    mma_commit_pred(x.bar(B_V_EMPTY + s), go);            // the v tile may be refilled once MMA2 has read it
    x.wait(B_P1_FULL + s, par, E_MMA, 0);                 // M and kr
    tc_fence_after();
#pragma unroll
    for (int ks = 0; ks < 4; ks++)                        // O += U M^T does not touch the state: issued before the wait
      mma_ts_tf32_pred(tWO + 32, tU + 8 * ks, d_m + so + (uint64_t)((ks * 32) >> 4), ID3B, 1, go);
    mma_commit_pred(x.bar(B_O_FULL + s), go);
    x.wait(B_S_READY, (uint32_t)((c + 1) & 1), E_MMA, 0); // decay St <- St diag(2^G31) finished
    tc_fence_after();
#pragma unroll
    for (int ks = 0; ks < 4; ks++)
      mma_ts_tf32_pred(tS, tU + 8 * ks, d_kr + so + (uint64_t)((ks * 4096) >> 4), ID3A, 1, go);
    PROF_STAMP(4, 28);
    mma_commit_pred(x.bar(B_CONS_EMPTY + s), go);
    PROF_STAMP(4, 29);
  }
  mma_commit_pred(x.bar(B_MMA1_DONE), go);         // the final state is complete
  mma_commit_pred(x.bar(B_DRAIN), go);
  // every tensor-core instruction has retired before tensor memory is freed, also after a give-up elsewhere
  if (!mbar_wait_drain(x.bar(B_DRAIN), 0, x.abort_flag)) atomicCAS(const_cast<int*>(x.abort_flag), 0, E_DRAIN + B_DRAIN);
}

// ------------------------------------------------------------------------------------------------ tensor-memory warps
template <typename OutT>
__device__ __forceinline__ void store_row_piece(OutT* dst_head, int key_first, int v, int col0, const uint32_t (&r)[32]);

template <>
__device__ __forceinline__ void store_row_piece<float>(float* dst, int key_first, int v, int col0, const uint32_t (&r)[32]) {
  if (!key_first) {
    float4* d = reinterpret_cast<float4*>(dst + v * D + col0);
#pragma unroll
    for (int i = 0; i < 8; i++)
      d[i] = make_float4(__uint_as_float(r[4 * i]), __uint_as_float(r[4 * i + 1]), __uint_as_float(r[4 * i + 2]), __uint_as_float(r[4 * i + 3]));
  } else {
#pragma unroll
    for (int i = 0; i < 32; i++) dst[(col0 + i) * D + v] = __uint_as_float(r[i]);
  }
}
template <>
__device__ __forceinline__ void store_row_piece<__nv_bfloat16>(__nv_bfloat16* dst, int key_first, int v, int col0, const uint32_t (&r)[32]) {
  if (!key_first) {
    uint4* d = reinterpret_cast<uint4*>(dst + v * D + col0);
#pragma unroll
    for (int i = 0; i < 4; i++)
      d[i] = make_uint4(pack_bf16(__uint_as_float(r[8 * i]), __uint_as_float(r[8 * i + 1])), pack_bf16(__uint_as_float(r[8 * i + 2]), __uint_as_float(r[8 * i + 3])),
                        pack_bf16(__uint_as_float(r[8 * i + 4]), __uint_as_float(r[8 * i + 5])), pack_bf16(__uint_as_float(r[8 * i + 6]), __uint_as_float(r[8 * i + 7])));
  } else {
#pragma unroll
    for (int i = 0; i < 32; i++) dst[(col0 + i) * D + v] = __float2bfloat16_rn(__uint_as_float(r[i]));
  }
}

// State columns [64 hf, 64 hf + 64) of this warp's 32 value rows: tensor memory -> final-state tensor and / or
// checkpoint row (either may be null).
template <int KF>
__device__ __noinline__ void store_state_rows(uint32_t tS, float* dst, void* ck, int ck_is_bf16, int v, int hf) {
#pragma unroll 1
  for (int j = 0; j < 2; j++) {
    const int col0 = 64 * hf + 32 * j;
    uint32_t r[32];
    tmem_ld32(tS + 32 * j, r);
    tmem_wait_ld();
    if (ck != nullptr) {
      if (ck_is_bf16) store_row_piece<__nv_bfloat16>(reinterpret_cast<__nv_bfloat16*>(ck), KF, v, col0, r);
      else store_row_piece<float>(reinterpret_cast<float*>(ck), KF, v, col0, r);
    }
    if (dst != nullptr) store_row_piece<float>(dst, KF, v, col0, r);
  }
}

// Decay St <- St diag(d) of a warp's 32 value rows x 64 state columns (at tS), on the serial chain MMA1 -> decay -> MMA3 ->
// MMA1 of the next chunk.  In the 16-lane form a thread holds columns 8 i + 2 (lane % 4), + 1 of every group of eight, so it
// needs 16 of the 64 factors (eight 8-byte loads; the 32-lane form takes sixteen 16-byte loads, all lanes the same).  Four
// pieces of 16 rows x 32 columns, the tensor-memory load of a piece in flight while the one before is scaled and stored.
__device__ __forceinline__ void scale_piece(uint32_t (&r)[16], const float2* d) {
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const float2 v = mul2(make_float2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1])), d[i >> 1]);
    r[2 * i] = __float_as_uint(v.x); r[2 * i + 1] = __float_as_uint(v.y);
  }
}
__device__ __forceinline__ void decay64(uint32_t tS, const float* dcol, int lane) {
  constexpr uint32_t ROWS16 = 16u << 16;
  uint32_t a[16], b[16];
  float2 d[8];
  tmem_ld16x32(tS, a);
#pragma unroll
  for (int i = 0; i < 8; i++) d[i] = *reinterpret_cast<const float2*>(dcol + 8 * i + 2 * (lane & 3));
  tmem_wait_ld();
  tmem_ld16x32(tS + 32, b);
  scale_piece(a, d);
  tmem_st16x32(tS, a);
  tmem_wait_ld();
  tmem_ld16x32(tS + ROWS16, a);
  scale_piece(b, d + 4);
  tmem_st16x32(tS + 32, b);
  tmem_wait_ld();
  tmem_ld16x32(tS + ROWS16 + 32, b);
  scale_piece(a, d);
  tmem_st16x32(tS + ROWS16, a);
  tmem_wait_ld();
  scale_piece(b, d + 4);
  tmem_st16x32(tS + ROWS16 + 32, b);
  tmem_wait_st();
}

// two neighbouring bf16 values of an output row
template <int PAIRS>
__device__ __forceinline__ void store_pair(__nv_bfloat16* at, uint32_t w) {
  if (PAIRS) {
    *reinterpret_cast<uint32_t*>(at) = w;
  } else {
    reinterpret_cast<uint16_t*>(at)[0] = (uint16_t)w;
    reinterpret_cast<uint16_t*>(at)[1] = (uint16_t)(w >> 16);
  }
}

// Eight warps own the tensor-memory traffic that goes through registers: warp (quarter q, half hf) serves the 32
// value rows [32 q, 32 q + 32) (the tensor-memory lanes a warp with id % 4 == q may touch) and, of those, the state
// columns [64 hf, 64 hf + 64) and the output tokens [16 hf, 16 hf + 16) of every chunk.  Per chunk:
//   wait MMA1 done -> (checkpoint row if due) -> St <- St diag(2^G31) for its columns -> signal S_READY        (on the chain)
//   wait MMA3 done -> O columns -> registers -> release the O buffer -> bf16 -> global                         (off the chain)
// plus the initial state load and the final state store for its columns.
template <int KF, int PAIRS>
__device__ void role_tmem(const ChunkParams& p, const Task& task, const Ctx& x, uint32_t tmem, int quarter, int hf, int lane) {
  const int v = 32 * quarter + lane;
  const uint32_t lane_base = (uint32_t)(32 * quarter) << 16;
  const uint32_t tS = tmem + TM_S + lane_base + 64 * hf;
  // ---- initial state -> tensor memory
#pragma unroll 1
  for (int j = 0; j < 2; j++) {
    const int col0 = 64 * hf + 32 * j;
    uint32_t r[32];
    if (task.flags & (TF_INIT_ZERO | TF_INIT_IDENTITY)) {
      const float one = (task.flags & TF_INIT_IDENTITY) ? 1.0f : 0.0f;
#pragma unroll
      for (int i = 0; i < 32; i++) r[i] = __float_as_uint((col0 + i == v) ? one : 0.0f);
    } else {
      const float* src = task.src + (size_t)x.h * STATE_ELEMS;
      if (!KF) {
        const float4* s4 = reinterpret_cast<const float4*>(src + v * D + col0);
#pragma unroll
        for (int i = 0; i < 8; i++) {
          const float4 f = s4[i];
          r[4 * i] = __float_as_uint(f.x); r[4 * i + 1] = __float_as_uint(f.y); r[4 * i + 2] = __float_as_uint(f.z); r[4 * i + 3] = __float_as_uint(f.w);
        }
      } else {
#pragma unroll
        for (int i = 0; i < 32; i++) r[i] = __float_as_uint(src[(col0 + i) * D + v]);
      }
    }
    tmem_st32(tS + 32 * j, r);
  }
  tmem_wait_st();
  tc_fence_before();
  __syncwarp();
  if (lane == 0) mbar_arrive(x.bar(B_S_READY));

  // Output: the two lanes of a pair exchange halves, so that a lane stores two neighbouring values of one token (even lanes
  // the even tokens) instead of one value of every token.  Rows that are not aligned to that (PAIRS = 0) are stored by value.
  const bool odd = lane & 1;
  const bool write_out = !(task.flags & TF_NO_OUT);
  const long long ldo = p.ldo;
  __nv_bfloat16* orow = ((task.flags & TF_OUT_AUX) ? p.out_aux : p.out) + (x.t0 + 16 * hf + (int)odd) * ldo + (long long)x.h * D + (v & ~1);
  const uint32_t sel = odd ? 0x3276u : 0x5410u;          // (own, other) packed token pairs -> this lane's token, lower value first
  int ck_left = (task.ck != nullptr && p.ck_every_chunks > 0) ? 0 : 0x7fffffff;     // chunks to the next checkpoint row
  const int nchunks = x.nchunks;
#pragma unroll 1
  for (int c = 0; c <= nchunks; c++, ck_left--, orow += C * ldo) {
    const int s = c & 1;
    const uint32_t par = (uint32_t)((c >> 1) & 1);
    const bool last = c == nchunks;
    x.wait(B_MMA1_DONE, (uint32_t)(c & 1), E_SCALE);
    tc_fence_after();
    // Checkpoint rows and the final state leave tensor memory through an out-of-line routine, so that their register
    // needs do not weigh on the per-chunk path below.
    const bool ck = ck_left == 0 && !last;
    if (ck || last) {
      float* dst = (last && task.dst != nullptr) ? task.dst + (size_t)x.h * STATE_ELEMS : nullptr;
      void* ckp = nullptr;
      if (ck) {
        const long long ck_off = (long long)(c / p.ck_every_chunks) * p.ck_row_stride + (long long)x.h * STATE_ELEMS;
        ckp = p.ck_is_bf16 ? static_cast<void*>(reinterpret_cast<__nv_bfloat16*>(task.ck) + ck_off)
                           : static_cast<void*>(reinterpret_cast<float*>(task.ck) + ck_off);
        ck_left = p.ck_every_chunks;
      }
      if (KF && (task.flags & TF_DST_VF)) store_state_rows<0>(tS, dst, ckp, p.ck_is_bf16, v, hf);   // transition maps
      else store_state_rows<KF>(tS, dst, ckp, p.ck_is_bf16, v, hf);
    }
    if (last) break;
    decay64(tS, reinterpret_cast<const float*>(x.smem + OFF_DEC) + (c & 3) * D + 64 * hf, lane);
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(x.bar(B_S_READY));

    // ---- output rows of this chunk
    x.wait(B_O_FULL + s, par, E_EPI);
    tc_fence_after();
    uint32_t o[16];
    tmem_ld16(tmem + TM_WO + 64 * s + 32 + 16 * hf + lane_base, o);
    tmem_wait_ld();
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(x.bar(B_O_EMPTY + s));
    if (write_out) {
      uint32_t w[8];
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const uint32_t own = pack_bf16(__uint_as_float(o[2 * i]), __uint_as_float(o[2 * i + 1]));
        w[i] = __byte_perm(own, __shfl_xor_sync(0xffffffffu, own, 1), sel);
      }
      const int left = x.len - c * C - 16 * hf - (int)odd;     // tokens of this run from this lane's first one on
      if (x.len - c * C >= C) {
#pragma unroll
        for (int i = 0; i < 8; i++) store_pair<PAIRS>(orow + (long long)(2 * i) * ldo, w[i]);
      } else {
#pragma unroll
        for (int i = 0; i < 8; i++)
          if (2 * i < left) store_pair<PAIRS>(orow + (long long)(2 * i) * ldo, w[i]);
      }
    }
  }
}

// ================================================================================================ dual-chain tasks
// Context parallelism and the cuts of long sequences need, for a token segment whose entering state is not known yet,
// TWO chains over the same tokens: chain L from S = 0 with the real v (o_loc, S_loc) and chain Tr from S = I with v = 0
// (Qt, P).  Everything the preparation warps, the loader and the inverse warps produce is the same for both, and the
// tensor pipe is busy a quarter of the time, so a task flagged TF_DUAL runs both chains over ONE operand preparation: a
// second state in tensor-memory columns 128-255, each MMA group issued twice, the tensor-memory warps serving both
// states (function of the reference's dual kernel, kda/b200/csrc/w3/base/cake_dual/kda_m128.cu:821-823,
// kda/b200/csrc/w3/base/dual.py:1-4).  The issuer and the tensor-memory warps have roles of their own for such a task
// (chosen once per CTA, so a launch mixes plain and dual tasks at no cost to the plain ones); the other roles do not
// know the difference.
// Tensor memory of a dual task: S_L 0-127, S_T 128-255, [W | O] of L 256-319, of T 320-383 (one buffer per chain: the
// other chain's work hides the read-out), U of L 384-447, of T 448-511 (two stages each).

__device__ void role_mma_dual(const Ctx& x, uint32_t tmem_any, bool v_zero_any) {
  const uint32_t go = elect_one();
  const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_any, 0);
  const bool v_zero = __shfl_sync(0xffffffffu, (int)v_zero_any, 0) != 0;
  const int nchunks = __shfl_sync(0xffffffffu, x.nchunks, 0);
  const uint32_t sb = smem_u32(x.smem);
  constexpr uint32_t ID1 = make_idesc(FMT_TF32, 128, 64, 0, 0, 0);
  constexpr uint32_t ID2A = make_idesc(FMT_BF16, 128, 32, 1, 0, 0);
  constexpr uint32_t ID2B = make_idesc(FMT_TF32, 128, 32, 0, 0, 1);
  constexpr uint32_t ID3A = make_idesc(FMT_TF32, 128, 128, 0, 1, 0);
  constexpr uint32_t ID3B = make_idesc(FMT_TF32, 128, 32, 0, 0, 0);
  const uint64_t d_kdqd = make_sdesc(sb + CS_KDQD, 16, 1024, LAYOUT_SW128);
  const uint64_t d_v = make_sdesc(sb + CS_V, 4096, 1024, LAYOUT_SW128);
  const uint64_t d_tbh = make_sdesc(sb + OFF_TBH, 16, 512, LAYOUT_SW64);
  const uint64_t d_tb = make_sdesc(sb + CS_TB, 16, 1024, LAYOUT_SW128);
  const uint64_t d_kr = make_sdesc(sb + CS_KR, 512, 2048, LAYOUT_SW128_BASE32B);
  const uint64_t d_m = make_sdesc(sb + CS_M, 16, 1024, LAYOUT_SW128);
  const uint32_t tS0 = tmem + TD_S0, tS1 = tmem + TD_S1, tWO1 = tmem + TD_WO1;
  x.wait(B_S_READY, 0, E_MMA, 0);                  // initial states are in tensor memory
  x.wait(B_S_READY_T, 0, E_MMA, 0);
#pragma unroll 1
  for (int c = 0; c < nchunks; c++) {
    const int s = c & 1;
    const uint32_t par = (uint32_t)((c >> 1) & 1), cpar = (uint32_t)(c & 1);
    const uint64_t so = (uint64_t)(s * (STAGE >> 4));
    const uint64_t so_tbh = (uint64_t)(s * (2048 >> 4));
    const uint32_t tU0 = tmem + TD_U0 + 32 * s, tU1 = tmem + TD_U1 + 32 * s;
    // [W | O]: one buffer per chain (one phase per chunk), not per stage as in the single-chain role
    const uint32_t tWO0 = tmem + TD_WO0;
    x.wait(B_KDQD_FULL + s, par, E_MMA, 0);
    x.wait(B_O_EMPTY + 0, cpar ^ 1, E_MMA, 0);
    tc_fence_after();
#pragma unroll
    for (int ks = 0; ks < 16; ks++)
      mma_ts_tf32_pred(tWO0, tS0 + 8 * ks, d_kdqd + so + (uint64_t)(((ks >> 2) * 8192 + (ks & 3) * 32) >> 4), ID1, ks > 0, go);
    mma_commit_pred(x.bar(B_MMA1_DONE), go);
    x.wait(B_O_EMPTY + 1, cpar ^ 1, E_MMA, 0);
    tc_fence_after();
#pragma unroll
    for (int ks = 0; ks < 16; ks++)
      mma_ts_tf32_pred(tWO1, tS1 + 8 * ks, d_kdqd + so + (uint64_t)(((ks >> 2) * 8192 + (ks & 3) * 32) >> 4), ID1, ks > 0, go);
    mma_commit_pred(x.bar(B_MMA1_DONE_T), go);
    mma_commit_pred(x.bar(B_KDQD_EMPTY + s), go);
    x.wait(B_V_FULL + s, par, E_MMA, 0);                  // (over long before the inverse is; a wait costs some 150 cycles even so)
    x.wait(B_INV_FULL + s, par, E_MMA, 0);
    tc_fence_after();
    if (!v_zero) {
#pragma unroll
      for (int ks = 0; ks < 2; ks++)
        mma_ss_f16_pred(tU0, d_v + so + (uint64_t)((2 * ks * 1024) >> 4), d_tbh + so_tbh + (uint64_t)((ks * 32) >> 4), ID2A, ks > 0, go);
    }
#pragma unroll
    for (int ks = 0; ks < 4; ks++)
      mma_ts_tf32_pred(tU0, tWO0 + 8 * ks, d_tb + so + (uint64_t)((ks * 32) >> 4), ID2B, (ks > 0) || !v_zero, go);
#pragma unroll
    for (int ks = 0; ks < 4; ks++)                      // the transition chain has v = 0: U = - W Tb^T
      mma_ts_tf32_pred(tU1, tWO1 + 8 * ks, d_tb + so + (uint64_t)((ks * 32) >> 4), ID2B, ks > 0, go);
    mma_commit_pred(x.bar(B_V_EMPTY + s), go);
    x.wait(B_P1_FULL + s, par, E_MMA, 0);
    tc_fence_after();
#pragma unroll
    for (int ks = 0; ks < 4; ks++)
      mma_ts_tf32_pred(tWO0 + 32, tU0 + 8 * ks, d_m + so + (uint64_t)((ks * 32) >> 4), ID3B, 1, go);
    mma_commit_pred(x.bar(B_O_FULL + 0), go);
#pragma unroll
    for (int ks = 0; ks < 4; ks++)
      mma_ts_tf32_pred(tWO1 + 32, tU1 + 8 * ks, d_m + so + (uint64_t)((ks * 32) >> 4), ID3B, 1, go);
    mma_commit_pred(x.bar(B_O_FULL + 1), go);
    x.wait(B_S_READY, (uint32_t)((c + 1) & 1), E_MMA, 0);
    tc_fence_after();
#pragma unroll
    for (int ks = 0; ks < 4; ks++)
      mma_ts_tf32_pred(tS0, tU0 + 8 * ks, d_kr + so + (uint64_t)((ks * 4096) >> 4), ID3A, 1, go);
    x.wait(B_S_READY_T, (uint32_t)((c + 1) & 1), E_MMA, 0);
    tc_fence_after();
#pragma unroll
    for (int ks = 0; ks < 4; ks++)
      mma_ts_tf32_pred(tS1, tU1 + 8 * ks, d_kr + so + (uint64_t)((ks * 4096) >> 4), ID3A, 1, go);
    mma_commit_pred(x.bar(B_CONS_EMPTY + s), go);
  }
  mma_commit_pred(x.bar(B_MMA1_DONE), go);         // the final states are complete
  mma_commit_pred(x.bar(B_MMA1_DONE_T), go);
  mma_commit_pred(x.bar(B_DRAIN), go);
  if (!mbar_wait_drain(x.bar(B_DRAIN), 0, x.abort_flag)) atomicCAS(const_cast<int*>(x.abort_flag), 0, E_DRAIN + B_DRAIN);
}

template <int KF>
__device__ void role_tmem_dual(const ChunkParams& p, const Task& task, const Ctx& x, uint32_t tmem, int quarter, int hf, int lane) {
  const int v = 32 * quarter + lane;
  const uint32_t lane_base = (uint32_t)(32 * quarter) << 16;
  const uint32_t tS0 = tmem + TD_S0 + lane_base + 64 * hf, tS1 = tmem + TD_S1 + lane_base + 64 * hf;
  // ---- initial states -> tensor memory: chain L as the task says, chain Tr the identity
#pragma unroll 1
  for (int ch = 0; ch < 2; ch++) {
#pragma unroll 1
    for (int j = 0; j < 2; j++) {
      const int col0 = 64 * hf + 32 * j;
      uint32_t r[32];
      if (ch == 1 || (task.flags & (TF_INIT_ZERO | TF_INIT_IDENTITY))) {
        const float one = (ch == 1 || (task.flags & TF_INIT_IDENTITY)) ? 1.0f : 0.0f;
#pragma unroll
        for (int i = 0; i < 32; i++) r[i] = __float_as_uint((col0 + i == v) ? one : 0.0f);
      } else {
        const float* src = task.src + (size_t)x.h * STATE_ELEMS;
        if (!KF) {
          const float4* s4 = reinterpret_cast<const float4*>(src + v * D + col0);
#pragma unroll
          for (int i = 0; i < 8; i++) {
            const float4 f = s4[i];
            r[4 * i] = __float_as_uint(f.x); r[4 * i + 1] = __float_as_uint(f.y); r[4 * i + 2] = __float_as_uint(f.z); r[4 * i + 3] = __float_as_uint(f.w);
          }
        } else {
#pragma unroll
          for (int i = 0; i < 32; i++) r[i] = __float_as_uint(src[(col0 + i) * D + v]);
        }
      }
      tmem_st32((ch ? tS1 : tS0) + 32 * j, r);
    }
    tmem_wait_st();
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(x.bar(ch ? B_S_READY_T : B_S_READY));
  }

  // Output of a dual-chain task: TILE-MAJOR scratch, [chunk][head][row v][32 tokens] bf16, Qt tiles at task.ck and the
  // o_loc tiles `oloc_tile_offset` elements behind them.  A lane owns one row v of the tile and 16 of its tokens, so
  // its share is 32 contiguous bytes (two 16-byte stores) instead of sixteen 2-byte stores 2 ldo bytes apart: the
  // tensor-memory warps are the busiest role of a dual task, and the output rows were a quarter of their time.  The
  // fix-up pass reads the tiles as they are (8 KB contiguous each) and writes the final rows.
  __nv_bfloat16* tiles = reinterpret_cast<__nv_bfloat16*>(task.ck) + (size_t)x.h * (D * C) + v * C + 16 * hf;
#pragma unroll 1
  for (int c = 0; c <= x.nchunks; c++) {
    const bool last = c == x.nchunks;
    const float* dcol = reinterpret_cast<const float*>(x.smem + OFF_DEC) + (c & 3) * D + 64 * hf;
#pragma unroll 1
    for (int ch = 0; ch < 2; ch++) {
      x.wait(ch ? B_MMA1_DONE_T : B_MMA1_DONE, (uint32_t)(c & 1), E_SCALE);
      tc_fence_after();
      const uint32_t tS = ch ? tS1 : tS0;
      if (last) {
        // final states: chain L in the launch's layout, the transition map always value-first
        float* dst = ch ? task.dst2 : task.dst;
        if (dst != nullptr) {
          dst += (size_t)x.h * STATE_ELEMS;
          if (ch == 1 || !KF || (task.flags & TF_DST_VF)) store_state_rows<0>(tS, dst, nullptr, 0, v, hf);
          else store_state_rows<KF>(tS, dst, nullptr, 0, v, hf);
        }
      } else {
        decay64(tS, dcol, lane);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(x.bar(ch ? B_S_READY_T : B_S_READY));
      }
    }
    if (last) break;
    // ---- output tiles of this chunk, chain L then chain Tr
#pragma unroll 1
    for (int ch = 0; ch < 2; ch++) {
      x.wait(B_O_FULL + ch, (uint32_t)(c & 1), E_EPI);       // one output buffer per chain (see role_mma_dual)
      tc_fence_after();
      uint32_t o[16];
      tmem_ld16(tmem + (ch ? TD_WO1 : TD_WO0) + 32 + 16 * hf + lane_base, o);
      tmem_wait_ld();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(x.bar(B_O_EMPTY + ch));
      if (!(task.flags & TF_NO_OUT)) {
        uint4* dst = reinterpret_cast<uint4*>(tiles + (ch ? 0 : p.oloc_tile_offset) + (size_t)c * p.H * (D * C));
        dst[0] = make_uint4(pack_bf16(__uint_as_float(o[0]), __uint_as_float(o[1])), pack_bf16(__uint_as_float(o[2]), __uint_as_float(o[3])),
                            pack_bf16(__uint_as_float(o[4]), __uint_as_float(o[5])), pack_bf16(__uint_as_float(o[6]), __uint_as_float(o[7])));
        dst[1] = make_uint4(pack_bf16(__uint_as_float(o[8]), __uint_as_float(o[9])), pack_bf16(__uint_as_float(o[10]), __uint_as_float(o[11])),
                            pack_bf16(__uint_as_float(o[12]), __uint_as_float(o[13])), pack_bf16(__uint_as_float(o[14]), __uint_as_float(o[15])));
      }
    }
  }
}

// ------------------------------------------------------------------------------------------------ kernel
template <int FE, int KF, int PAIRS>
__global__ void __launch_bounds__(THREADS, 1) kda_chunk_umma_kernel(const __grid_constant__ ChunkParams p, const __grid_constant__ TmaMaps maps) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = tid >> 5;
  const int H = p.H;
  const int rank = blockIdx.x / H, h = blockIdx.x % H;

  // Launched as a programmatic dependent of the planner (its CTAs become resident while the planner still runs): wait
  // here until the planner's writes (status, task table) are visible.  A no-op for an ordinary launch.
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  const int nt_word = *p.n_tasks;
  if (nt_word & NT_ZERO_FILL) {   // rejected cu_seqlens: all sequences empty, output rows zero-filled
    const long long rows = p.T * H;
    for (long long r = blockIdx.x; r < rows; r += gridDim.x)
      if (tid < 16) reinterpret_cast<uint4*>(p.out + (r / H) * p.ldo + (r % H) * D)[tid] = make_uint4(0, 0, 0, 0);
  }
  if (rank >= (nt_word & (NT_ZERO_FILL - 1))) return;
  const Task task = p.tasks[rank];
  Ctx x;
  x.smem = smem;
  x.bars = smem_u32(smem + OFF_BAR);
  x.abort_flag = reinterpret_cast<volatile int*>(smem + OFF_MISC + 8);
  x.h = h;
  x.len = task.len;
  x.nchunks = (task.len + C - 1) / C;
  x.t0 = task.t0;
#ifdef KDA_PROF
  x.prof = p.prof;
  const long long prof_t0 = clock64();
#endif

  const bool dual = (task.flags & TF_DUAL) != 0;   // both chains of a mapped segment in this task (see the dual-chain roles)
  if (x.nchunks == 0) {
    // empty run: the state passes through (source -> destination) without touching tensor memory; the transition map
    // of no tokens is the identity
    for (int ch = 0; ch < (dual ? 2 : 1); ch++) {
      float* dst = ch ? task.dst2 : task.dst;
      if (dst == nullptr) continue;
      dst += (size_t)h * STATE_ELEMS;
      const bool ident = ch == 1 || (task.flags & TF_INIT_IDENTITY);
      const float* src = (ch == 1 || (task.flags & (TF_INIT_ZERO | TF_INIT_IDENTITY))) ? nullptr : task.src + (size_t)h * STATE_ELEMS;
      if (src == dst) continue;
      for (int i = tid; i < STATE_ELEMS / 4; i += THREADS) {
        float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
        if (src != nullptr) f = reinterpret_cast<const float4*>(src)[i];
        else if (ident) {
          const int row = (4 * i) / D, col = (4 * i) % D;
          f = make_float4(row == col ? 1.f : 0.f, row == col + 1 ? 1.f : 0.f, row == col + 2 ? 1.f : 0.f, row == col + 3 ? 1.f : 0.f);
        }
        reinterpret_cast<float4*>(dst)[i] = f;
      }
    }
    return;
  }

  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + OFF_MISC);
  volatile int* range_flag = reinterpret_cast<volatile int*>(smem + OFF_MISC + 12);
  if (tid == 0) {
    *x.abort_flag = 0;
    *range_flag = 0;
    *reinterpret_cast<volatile unsigned long long*>(smem + OFF_MISC + 16) = p.wait_limit_ns ? p.wait_limit_ns : kWaitLimitNs;
  }
  if (warp == W_INV0) {
    // One lane per barrier (the issuer warp allocates tensor memory meanwhile): a task of one or two chunks notices the
    // forty serial initialisations.  Arrival counts: the eight warps of a preparation group or the eight tensor-memory
    // warps where a whole group signals, three for the L tile (its three blocks), one everywhere else.
    constexpr unsigned long long EIGHT = (3ull << B_G_EMPTY) | (3ull << B_P1_FULL) | (3ull << B_O_EMPTY) | (1ull << B_S_READY) |
                                         (7ull << B_QK_EMPTY) | (1ull << B_S_READY_T) | (3ull << B_NORM) | (3ull << B_KDQD_FULL);
    static_assert(PREP_WARPS == 8, "arrival counts of the group barriers");
    for (int i = lane; i < NUM_BARS; i += 32) {
      int count = ((EIGHT >> i) & 1ull) ? 8 : 1;
      if (i == B_L_FULL || i == B_L_FULL + 1) count = 3;
      // diagnostic switch: the v barriers expect one arrival more than they will ever get, so their waiters give up
      if ((i == B_V_FULL || i == B_V_FULL + 1) && (p.debug_flags & DBG_STALL_V_STREAM)) count = 2;
      mbar_init(x.bar(i), count);
    }
    fence_barrier_init();
  }
  if (warp == W_MMA) {
    tmem_alloc(smem_u32(tmem_slot), TM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const bool v_zero = (task.flags & TF_V_ZERO) != 0;

  if (warp == W_MMA) {
    if (dual) role_mma_dual(x, tmem, v_zero);
    else role_mma(x, tmem, v_zero);
    __syncwarp();
  } else if (warp == W_INV0 || warp == W_INV0 + 1) {
    role_inverse(x, warp - W_INV0, lane);
  } else if (warp == W_LOAD) {
    role_loader<FE>(p, maps, x, lane);
    __syncwarp();
  } else if (warp < W_PREP0) {
    if (dual) role_tmem_dual<KF>(p, task, x, tmem, warp & 3, (warp - W_SCALE0) >> 2, lane);
    else role_tmem<KF, PAIRS>(p, task, x, tmem, warp & 3, (warp - W_SCALE0) >> 2, lane);
  } else {
    const int pt = tid - W_PREP0 * 32;
    role_prep<FE>(p, x, pt / PREP_THREADS, pt % PREP_THREADS);
  }

#ifdef KDA_PROF
  if (lane == 0 && blockIdx.x == 0 && x.prof != nullptr) {
    const int role = warp == W_MMA ? 4 : (warp <= 2 ? 3 : (warp == W_LOAD ? 1 : (warp < W_PREP0 ? 5 : 2)));
    atomicAdd(x.prof + role * 128 + 126, (unsigned long long)(clock64() - prof_t0));
    atomicAdd(x.prof + role * 128 + 127, 1ull);
  }
#endif
  tc_fence_before();
  __syncthreads();
  if (tid == 0) {
    if (*x.abort_flag != 0) atomicCAS(p.status + 2, 0, *x.abort_flag);
    if (*range_flag != 0) atomicOr(p.status, KDA_BIT_RANGE);
  }
  if (warp == W_MMA) tmem_dealloc(tmem, TM_COLS);
}

}  // namespace u

cudaError_t launch_chunk_umma(const ChunkParams& p, const TmaMaps& maps, int n_task_cap, cudaStream_t stream, bool after_planner) {
  // One instantiation per (front-end, state layout).  Those of the third row are for Qt rows at an address that is no multiple
  // of four (value-first only, as every segment launch): a test of it per chunk cost the others up to 4 %.
  typedef void (*Kern)(const ChunkParams, const TmaMaps);
  static const Kern kerns[3][2] = {{u::kda_chunk_umma_kernel<0, 0, 1>, u::kda_chunk_umma_kernel<0, 1, 1>},
                                   {u::kda_chunk_umma_kernel<1, 0, 1>, u::kda_chunk_umma_kernel<1, 1, 1>},
                                   {u::kda_chunk_umma_kernel<0, 0, 0>, u::kda_chunk_umma_kernel<1, 0, 0>}};
  static int attr_dev_mask = 0;
  int dev = 0;
  cudaGetDevice(&dev);
  if (!(attr_dev_mask & (1 << (dev & 31)))) {
    for (int i = 0; i < 6; i++) {
      cudaError_t e = cudaFuncSetAttribute(kerns[i >> 1][i & 1], cudaFuncAttributeMaxDynamicSharedMemorySize, u::SMEM_BYTES);
      if (e != cudaSuccess) return e;
    }
    attr_dev_mask |= 1 << (dev & 31);
  }
  const long long blocks = (long long)n_task_cap * p.H;
  if (blocks <= 0) return cudaSuccess;
  // Chained behind the planner by programmatic dependent launch when it directly follows it in the stream (function
  // of kda/b200/csrc/w3/base/cake/launch_m128.cu:37-60): the launch latency hides under the planner.
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)blocks);
  cfg.blockDim = dim3(u::THREADS);
  cfg.dynamicSmemBytes = u::SMEM_BYTES;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = after_planner ? 1 : 0;
  const bool unpaired = (reinterpret_cast<uintptr_t>(p.out_aux) & 3) != 0;
  if (unpaired && p.key_first) return cudaErrorInvalidValue;
  return cudaLaunchKernelEx(&cfg, unpaired ? kerns[2][p.frontend ? 1 : 0] : kerns[p.frontend ? 1 : 0][p.key_first ? 1 : 0], p, maps);
}

}  // namespace kda
