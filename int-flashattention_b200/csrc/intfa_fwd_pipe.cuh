// INT8 attention forward (full-int8 and half-int8): ONE CTA per SM, one 128-row query tile at a time.
// (Included by intfa_fwd.cu inside namespace intfa, after the shared helpers.)
//
// 512 threads with two softmax groups, 640 with three (PipeCfg::NGRP):
//   warp 0        TMA producer (Q once per work item; K and V through rings of shared-memory stages); it also draws
//                 the work items: the CTA's own index first, then from a global counter
//   warp 1        MMA issuer for S = Q K^T (whole warp runs the loop, one elected lane issues): up to NSB (three or four) KV
//                 steps ahead of the softmax groups, into S buffer (step mod NSB)
//   warp 2        TMEM allocator; then loads the K scales (fp32 or fp16, rows of any alignment) into a ring of their own
//   warp 3        MMA issuer for O_j = P V
//   warps 4-7, 8-11 (, 12-15)   softmax groups 0, 1 (, 2): one thread per query row.  The groups take the KV steps in
//                 TURN (group g owns the steps whose running index is g mod NGRP), each with its own P buffer in shared
//                 memory (or with P over its scores in TMEM: PipeCfg::P_TMEM), so that on every scheduler one warp is in pass A (dequantise, row max: FMA pipe) while
//                 another is in pass B (exp2, P: exp2 unit).  The running max m of a row travels between the threads
//                 that own it through shared memory, once per step.
//   the last 4 warps   accumulator update and epilogue, one thread per query row:
//                 full-int8: A = A*alpha + fp32(O_j) with the fp32 row A in REGISTERS and O_j (int32) in TMEM;
//                 half-int8: P V (fp16 MMA) accumulates straight into an fp32 accumulator in TMEM, these warps
//                 multiply the row by alpha beforehand when some alpha of the warp's 32 rows is not 1.
//                 They also carry the row sum l = l*alpha + rowsum(P) (see PipeCfg::L_IN_ACC).
// TMEM columns: NSB S buffers of G | NO O_j buffers of D, or the half-int8 accumulator of D  (<= 512).
// S and O_j are int32 accumulators that start each KV step from the bit pattern of 1.5*2^23, written by a
// small fp16 MMA ahead of the int8 MMAs, so that the threads read fp32(S32) + 1.5*2^23 without a conversion.
// The arithmetic contract is at the top of intfa_fwd.cu.
#pragma once

constexpr int kPipeCorrThreads = 128;
constexpr int kPipeServiceRegs = 40;

// D: channels of V and of the accumulator that one pass covers (and the width the tensor-core tiles are built for);
// DQ: head dim of Q and K.  DQ == D except for full-int8 at head dim 256, which runs as DQ = 256, D = 128: every query tile
// is taken twice in a row by the same CTA, once per half of the V channels (the accumulator row of one thread holds 128
// channels); S, the running max and P are the same in both passes.  Half-int8 has its accumulator in TMEM, where 256
// channels fit next to three S buffers of 64, and takes them in one pass (batch 2, 16 heads, 4096 tokens, causal, fp16 V:
// 516 us for two passes).
// F8V: the half-int8 op with V (and therefore P) in float8_e5m2 (flash_atten_int8.py:55-56): one-byte P and V tiles laid
// out like the int8 ones, P V with kind::f8f6f4 accumulating in fp32 like the fp16 form.
template <int D, int G, bool FULL, int DQ = D, bool F8V = false>
struct PipeCfg {
  static_assert(!(FULL && F8V), "fp8 V belongs to the half-int8 op");
  static constexpr bool BYTE_PV = FULL || F8V;                     // P and V elements are one byte
  // P goes back into TMEM, over the first half of its own S buffer, and P V takes it from there (A operand in TMEM): no
  // P buffers in shared memory (32 KB each for fp16), which makes room for a third softmax group and four V stages, no swizzled
  // stores and no proxy fence.  Two groups with P in shared memory before: batch 4, 32 heads, 4096 tokens causal 733 -> 640 us,
  // batch 2 non-causal 659 -> 565 us, batch 2 causal at d=64 347 -> 308 us.  The S buffer goes back when the P V is done.  With
  // 64-column steps two groups stay the better (422 -> 398 us at d=64, three 401; 431 -> 421, 438 at d=128; 302 -> 288, 291 at d=256).
  // One-byte P: the same for fp8 V with 64-column steps (d=64 401 -> 380 us).  Three groups with small P buffers lose more from
  // the S buffer's later return than they gain: fp8 V 301 -> 322 us, full-int8 383 -> 388, 64-column steps 714 -> 737.
  static constexpr bool P_TMEM = !BYTE_PV || (F8V && G == 64);
  // Softmax groups of 128 threads.  Three (with 96 registers a thread, 16-column buffers) hide the hand-overs better than two
  // (152 registers, 32 columns) nearly everywhere (two -> three: full-int8 4 x 32 x 8192 4578 -> 4164 us, 2 x 32 x 4096 with 64-column
  // steps 802 -> 759, at d=64 634 -> 602 and 565 -> 527 with 128-column steps, 2 x 32 x 2048 causal at d=32 145 -> 134; half-int8
  // 487 -> 450, at d=64 460 -> 405; fp8 V 496 -> 448).  Half-int8 with 64-column steps does not gain (d=256 407 -> 407), full-int8 at
  // head dim 256 has no room for a third P buffer beside its K tiles.
  static constexpr int NGRP = (!BYTE_PV && G == 128) || (F8V && G == 128 && D == 128) || (FULL && DQ <= 128) ? 3 : 2;
  static constexpr int THREADS = 256 + 128 * NGRP;
  // Registers: the CTA is launched with LAUNCH_REGS per thread and setmaxnreg only moves registers around
  // INSIDE that allocation -- an increase beyond it would block for ever, hence the static_assert below.
  static constexpr int LAUNCH_REGS = (65536 / THREADS) / 8 * 8;
  static_assert(DQ == D || (DQ == 256 && D == 128), "head dims");
  static constexpr int NVH = DQ / D;                               // passes per query tile
  static constexpr int QK_ROWB = DQ < 128 ? DQ : 128;              // Q and K sit in shared memory as panels of [rows][QK_ROWB bytes]
  static constexpr int QK_PANELS = DQ / QK_ROWB;
  static constexpr int Q_BYTES = kBM * DQ;
  static constexpr int K_BYTES = G * DQ;
  static constexpr int V_BYTES = BYTE_PV ? G * D : G * D * 2;         // int8, or fp16 as D/64 boxes of [G keys][64 channels]
  static constexpr int P_BYTES = P_TMEM ? 0 : kBM * G;              // int8 or e5m2
  static constexpr int KS_BYTES = G * 4;
  static constexpr bool BIG = DQ > 128 && (G == 128 || D == 256);   // 32 KB K tiles, or 32 KB V tiles: three stages are what fits
  static constexpr int NSK = BIG ? 3 : 4;                          // K stages
  static constexpr int NSV = BIG ? 3 : 4;                          // V stages
  static constexpr int NKS = 8;                                    // K-scale slots (see the warp that fills them)
  // S buffers in TMEM.  Four where a step's buffer waits for its P V and there is room (d=64: 385 -> 371 us, d=128 at G=64 421 ->
  // 414; no gain at d=256).
  static constexpr int NSB = P_TMEM && G == 64 && D <= 128 ? 4 : 3;
  static constexpr int NRS = NSB == 4 ? 8 : 4;                     // row-sum slots: step j's is read at step j+1, when P V j+1 may be out
  static constexpr int P_PER_COL = BYTE_PV ? 4 : 2;                // P_TMEM: elements of P in a TMEM column
  static constexpr int NPB = P_TMEM ? NSB : NGRP;                  // P buffers
  // Where the accumulator is 256 channels wide, the way round P V -> rescaling -> next P V is the longest one: P V takes the channels
  // in two halves, and one is rescaled while P V of the other runs (2 x 16 x 4096 at d=256 432 -> 397 us, causal 267 -> 245).
  // (In two halves of the keys, so that P V of 128-column steps can begin before all of P is there: half-int8 443 -> 441 us, causal
  // 504 -> 547.)
  static constexpr int NOH = !FULL && D == 256 ? 2 : 1;
  static constexpr int NPBAR = P_TMEM ? 0 : NGRP;                  // ... and their barriers, where they are in shared memory
  // Who carries the row sum l = l*alpha + rowsum(P)?  Where a KV step is as wide as the head (G >= D) the accumulator
  // warps do, next to the accumulator row: the softmax groups then meet once per step (running max) instead of
  // twice.  Where the head is wider than the step (head_dim 128 at G = 64) the accumulator warps are the busier
  // side and the softmax groups keep l, handing it over like the running max (measured: 582 against 474 TOPS).
  static constexpr bool L_IN_ACC = G >= D;
  // A vectorised pass A for the causal diagonal band and the last, partial step (otherwise those take the general, scalar
  // path): compiled in for 128-column KV steps, where it measured +2..5 % on causal workloads, and for 32-column steps of
  // ragged lengths (batch 8, 32 heads, 1000 tokens causal at d=32: 273 -> 212 us, 64 x 32 x 250: 327 -> 224).  Elsewhere its
  // code costs the steps that need no mask more (instruction cache) than it gives (2 x 16 x 4096 at d=32: 573 -> 631).
  __host__ __device__ static constexpr bool band_fast(bool ragged) { return G == 128 || D == 256 || (G == 32 && ragged); }
  // instructions of never-executed filler between the softmax passes (see intfa_fwd_pipe_softmax.inc), the best of a sweep in
  // steps of 1 KB for each kind of instantiation (`ragged`: masks partial tiles; `steady`: see the kernel).  With three groups of
  // 128-column steps the sweep changed 1 to 3 % (steady 4157 to 4189 us but for 4361 at 256; causal 315 to 338); with 64-column steps and
  // at head dim 256 up to 20 % (half-int8 causal at d=128 406 to 520 us, at d=256 245 to 287).  These sweeps are older than the
  // votes inside the wait loops; of the kernels as they are only full-int8 at head dim 256, 64-column steps of ragged lengths, has been
  // swept (16 heads of 4001 498 to 549 us, causal 330 to 382).
  __host__ __device__ static constexpr int code_filler_of(bool ragged, bool steady) {
    if (P_TMEM) {
      if (G == 128) return ragged || D == 128 ? 64 : 192;
      return D == 256 ? (ragged ? 384 : 0) : !ragged ? 384 : D == 128 ? 256 : 128;
    }
    if (F8V) return 192;
    if (DQ == 256) return ragged ? (G == 64 ? 208 : 384) : 0;
    if (ragged) return G == 32 ? 384 : G == 128 ? 256 : D == 128 ? 0 : 128;
    return G < 128 ? 256 : steady ? 128 : 64;
  }
  // setmaxnreg split between the softmax and the accumulator warps, two groups.  The accumulator row of 128 channels fits either
  // way; with 128-column KV steps, and for half-int8 (no accumulator row in registers), the softmax passes gain more
  // from 16 further registers than the update loses (measured +2..3 %); full-int8 at head dim 256 with 64-column steps is the other
  // way round.
  static constexpr bool MORE_SOFTMAX_REGS = !FULL || G == 128;
  static constexpr int SOFTMAX_REGS = NGRP == 3 ? (FULL ? 96 : 112) : MORE_SOFTMAX_REGS ? 152 : 136;
  static constexpr int CORR_REGS = NGRP == 3 ? (FULL ? 152 : 96) : MORE_SOFTMAX_REGS ? 168 : 184;
  static_assert(128 * kPipeServiceRegs + 128 * NGRP * SOFTMAX_REGS + kPipeCorrThreads * CORR_REGS <= THREADS * LAUNCH_REGS,
                "setmaxnreg budget exceeds the registers the CTA is launched with");
  static constexpr int OFF_Q = 0;
  static constexpr int OFF_K = OFF_Q + Q_BYTES;
  static constexpr int OFF_V = OFF_K + NSK * K_BYTES;
  static constexpr int OFF_P = OFF_V + NSV * V_BYTES;             // a P buffer per softmax group
  static constexpr int OFF_KS = OFF_P + NGRP * P_BYTES;
  static constexpr int OFF_VSD = OFF_KS + NKS * KS_BYTES;         // s_v/127 per channel
  static constexpr int OFF_HM = OFF_VSD + D * 4;                  // [NGRP][128] float: running max after the group's latest step
  static constexpr int OFF_RS = OFF_HM + NGRP * 128 * 4;             // [NRS][128] float: row sum of P of step j, for the accumulator warps
                                                                   //   (!L_IN_ACC: [NGRP][128] float, l after the group's latest step)
  static constexpr int OFF_ALPHA = OFF_RS + NRS * 128 * 4;          // [4][128] float: alpha of step j, for the accumulator warps
  static constexpr int OFF_FIN = OFF_ALPHA + 4 * 128 * 4;         // [2][128] float2: final running max of a work item (.x)
  static constexpr int OFF_MAGIC = OFF_FIN + 2 * 128 * 8;          // 4 KB constant fp16 operand of the "arm" MMA
  static constexpr int MAGIC_BYTES = 4096;
  static constexpr int OFF_TILE = OFF_MAGIC + MAGIC_BYTES;         // [4] TileInfo: the work-item ring
  static constexpr int OFF_BAR = OFF_TILE + 4 * (int)sizeof(TileInfo);
  static constexpr int NUM_BARS = 14 + NPBAR + 2 * NSK + 2 * NSV + 12 + NSB + (NOH - 1);
  static constexpr int OFF_MISC = OFF_BAR + NUM_BARS * 8;
  static constexpr int SMEM_BYTES = OFF_MISC + 32 + 1024;
  // S buffer b at COL_S + b*G; then O_j (full-int8: the accumulator itself lives in registers) or the fp32
  // accumulator the second MMA adds into (half-int8)
  static constexpr int COL_S = 0, COL_O = NSB * G, COL_ACC = NSB * G;
  // full-int8: two O_j buffers where TMEM has the room (head dim 256, 64-column steps), so that P V of the next step does not wait for
  // the accumulator warps.  (Not with three groups: alpha and the row sums of a step would be overwritten too early.)
  static constexpr int NO = FULL && NGRP == 2 && NSB * G + 2 * D <= 512 ? 2 : 1;
  static_assert(NSB * G + NO * D <= 512, "TMEM columns");
  // The barrier on which an MMA warp waits for a step is a K or V stage's (see the kernel).  No arrival for step j may come before
  // the wait for the step that had the barrier before it: what arrives follows from that step's S, P or O_j buffer being free
  // again, so there must not be more of these than stages.
  static_assert(NSB <= NSK && NPB <= NSV && NO <= NSV, "ready barriers");
  static constexpr int TMEM_COLS = 512;
  static_assert(FULL || G >= 64, "half-int8");
  static constexpr uint64_t SWZ_QK = (QK_ROWB == 128) ? kSwz128 : (QK_ROWB == 64) ? kSwz64 : kSwz32;
  static constexpr uint32_t SBO_QK = 8 * QK_ROWB;
  // start-address offset (16-byte units) of the kk-th 32-byte K slice of a [ROWS][DQ] operand
  __host__ __device__ static constexpr uint32_t qk_slice(int kk, int rows) { return (uint32_t)((kk / 4) * ((rows * QK_ROWB) >> 4) + 2 * (kk % 4)); }
  static constexpr uint64_t SWZ_P = (G == 128) ? kSwz128 : (G == 64) ? kSwz64 : kSwz32;
  static constexpr uint32_t SBO_P = 8 * G;
  // V rows: boxes of at most 128 bytes of channels
  static constexpr int V_ROWB = D * (BYTE_PV ? 1 : 2) < 128 ? D * (BYTE_PV ? 1 : 2) : 128;
  static constexpr int PV_K = BYTE_PV ? 32 : 16, PV_STEPS = G / PV_K;     // keys of one P V MMA, and how many it takes
  static constexpr int V_BOXES = D * (BYTE_PV ? 1 : 2) / V_ROWB;
  static constexpr int V_BOXCH = D / V_BOXES;                      // channels of one box
  static constexpr uint64_t SWZ_V = (V_ROWB == 128) ? kSwz128 : (V_ROWB == 64) ? kSwz64 : kSwz32;
  static constexpr uint32_t SBO_V = 8 * V_ROWB;
  static constexpr uint32_t IDESC_QK = make_idesc(2, 1, 1, 0, 0, kBM, G);
  // (kind::f8f6f4: A / B format 1 = e5m2, D format 1 = f32)
  static constexpr int PV_N = D / NOH;                              // channels of one P V MMA
  static constexpr uint32_t IDESC_PV = FULL ? make_idesc(2, 1, 1, 0, 1, kBM, PV_N)
                                       : F8V ? make_idesc(1, 1, 1, 0, 1, kBM, PV_N) : make_idesc(1, 0, 0, 0, 1, kBM, PV_N);
  // fp16 x fp16 -> fp32, K = 16: writes the fp32 constant 1.5*2^23 into a whole accumulator tile
  static constexpr uint32_t IDESC_ARM_S = make_idesc(1, 0, 0, 0, 0, kBM, G);
  static constexpr uint32_t IDESC_ARM_O = make_idesc(1, 0, 0, 0, 0, kBM, D);
};

enum PipeWait { PW_TILE = 32, PW_QE, PW_KE, PW_VE, PW_QF, PW_QKRDY, PW_PVRDY, PW_SFULL,
                PW_PFREE, PW_HM, PW_OFULL, PW_FIN, PW_FINFREE, PW_HL, PW_AFULL };

// RAGGED: Nq / Nk are not multiples of 128 / G -- the last query tile and the last KV step are partial.  A separate
// instantiation, so that the code of the common case stays as small as it was (instruction cache).
// PROUND: how full-int8 rounds P (see PRound).
// STEADY: non-causal full-int8 with three groups, whose groups take the running max over before pass A (see the softmax warps).
template <int D, int G, bool FULL, int PROUND, bool RAGGED, int DQ = D, bool F8V = false, bool STEADY = false>
__global__ void __launch_bounds__((PipeCfg<D, G, FULL, DQ, F8V>::THREADS), 1)
intfa_fwd_pipe_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                      const __grid_constant__ CUtensorMap tmV, const KParams p) {
  using C = PipeCfg<D, G, FULL, DQ, F8V>;
  constexpr int NSK = C::NSK, NSV = C::NSV, NSB = C::NSB, NVH = C::NVH, NO = C::NO;
  extern __shared__ uint8_t smem_raw[];
  // (rounded up by an offset, not through an integer: the compiler then knows that all this is shared memory)
  uint8_t* smem = smem_raw + ((0u - smem_u32(smem_raw)) & 1023u);
  // (Uniform for the compiler: with the plain quotient every role's code is in a branch that it must take for divergent, and
  // all descriptors, barrier addresses and counters sit in vector registers.)
  const int warp = warp_uniform(threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;

  const uint32_t bar0 = smem_u32(smem + C::OFF_BAR);
  auto BAR = [&](int i) { return bar0 + 8u * i; };
  // mbarriers.  "commit" = arrived on by tcgen05.commit, i.e. when the MMAs issued so far are done.
  constexpr int NGRP = C::NGRP;
  constexpr int B_QFULL = 0;      // TMA: Q tile landed
  constexpr int B_QEMPTY = 1;     // commit: last Q K^T of the work item done
  constexpr int B_OFULL = 2;      // [NO] commit: O_j = P V in TMEM buffer (step mod NO) ([NOH]: P V of a half of the channels)
  constexpr int B_FIN = 4;        // [2] softmax (4 warps of one group): final (m, l) of the work item published; one
                                  //     barrier per slot, so that a short next work item cannot complete it twice
                                  //     before a slow accumulator warp has waited for the first completion
  constexpr int B_FINFREE = 6;    // [2] accumulator warps (4): they have read them
  constexpr int B_HM = 8;         // [NGRP] softmax group g (4 warps): running max after its step published
  constexpr int B_HL = 11;        // [NGRP] !L_IN_ACC: softmax group g (4 warps): row sum after its step published
  // What an MMA warp needs for step j arrives on ONE barrier, which belongs to the step's K or V stage: a wait that finds
  // everything there costs these warps 200 to 350 cycles, and three of them in a row were the longest part of the way from P to
  // the next S (half-int8, batch 2, 32 heads, 4096 tokens: 567 -> 518 us; full-int8 at head dim 32: 1131 -> 887 us).
  constexpr int B_QKRDY = 14;               // [NSK] TMA: K tile landed; softmax group of step j - NSB (4 warps): S buffer read out
                                            //     for good (P_TMEM: commit: the P V that read P from it is done)
  constexpr int B_KEMPTY = B_QKRDY + NSK;   // [NSK] commit: the Q K^T that read the stage is done
  constexpr int B_PVRDY = B_KEMPTY + NSK;   // [NSV] TMA: V tile landed; softmax group of step j (4 warps): P written; accumulator
                                            //     warps (4): O_j of step j - NO read out (half-int8: the accumulator row is at
                                            //     step j's running max)
  constexpr int B_VEMPTY = B_PVRDY + NSV;   // [NSV] commit: the P V that read the stage is done
  constexpr int B_PFREE = B_VEMPTY + NSV;   // [NPBAR] commit: the P V that read shared-memory P buffer b is done
  constexpr int B_TILE = B_PFREE + C::NPBAR, B_TDONE = B_TILE + 4;
  constexpr int B_AFULL = B_TDONE + 4;   // [4] half-int8: alpha of step j (slot j mod 4) published, for the accumulator warps
  constexpr int SFREE_ARRIVALS = C::P_TMEM ? 1 : 4;
  constexpr int B_SFULL = B_AFULL + 4;   // [NSB] commit: S = Q K^T in TMEM buffer b; scale loader: the step's K scales in
                                         //     shared memory (the arrival of the warp that wrote them is what lets the
                                         //     softmax warps see them)
  constexpr int B_OHI = B_SFULL + NSB;   // NOH == 2: accumulator warps (4): the upper half of the row is at step j's running max
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + C::OFF_MISC);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + C::OFF_MISC + 4);
  TileInfo* tile_slot = reinterpret_cast<TileInfo*>(smem + C::OFF_TILE);

  if (threadIdx.x == 0) {
    mbar_init(BAR(B_QFULL), 1);
    mbar_init(BAR(B_QEMPTY), 1);
    for (int b = 0; b < C::NPBAR; ++b) mbar_init(BAR(B_PFREE + b), 1);
    for (int b = 0; b < NGRP; ++b) {
      mbar_init(BAR(B_HM + b), 4);
      mbar_init(BAR(B_HL + b), 4);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(BAR(B_FINFREE + b), 4);
      mbar_init(BAR(B_FIN + b), 4);
    }
    for (int b = 0; b < (NO > C::NOH ? NO : C::NOH); ++b) mbar_init(BAR(B_OFULL + b), 1);
    if (C::NOH > 1) mbar_init(BAR(B_OHI), 4);
    for (int s = 0; s < NSK; ++s) {
      mbar_init(BAR(B_QKRDY + s), 1 + SFREE_ARRIVALS);
      mbar_init(BAR(B_KEMPTY + s), 1);
    }
    for (int s = 0; s < NSV; ++s) {
      mbar_init(BAR(B_PVRDY + s), 1 + 4 + 4);
      mbar_init(BAR(B_VEMPTY + s), 1);
    }
    for (int b = 0; b < NSB; ++b) mbar_init(BAR(B_SFULL + b), 2);         // Q K^T done; the K scales of the step are written
    // the very first step finds the running max (and l) handed over, the first steps their S and O_j buffers free
    mbar_arrive_n(BAR(B_HM + NGRP - 1), 4);
    mbar_arrive_n(BAR(B_HL + NGRP - 1), 4);
    for (int j = 0; j < NSB; ++j) mbar_arrive_n(BAR(B_QKRDY + j), SFREE_ARRIVALS);
    if (FULL)
      for (int j = 0; j < NO; ++j) mbar_arrive_n(BAR(B_PVRDY + j), 4);
    for (int i = 0; i < 4; ++i) {
      mbar_init(BAR(B_TILE + i), 1);
      mbar_init(BAR(B_TDONE + i), 7 + 4 * NGRP);       // 2 MMA warps, the scale loader, accumulator and softmax warps
      mbar_init(BAR(B_AFULL + i), 4);
    }
    abort_flag[0] = 0;
    abort_flag[1] = (int)((uint32_t)p.wait_limit_kcycles << 10);
    mbar_init_fence();
    fence_proxy_async_smem();
  }
  if (warp == 2) {
    tmem_alloc(smem_u32(tmem_slot), C::TMEM_COLS);
    tmem_relinquish();
    tc_fence_before();
  }
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = warp_uniform(*tmem_slot);
  const uint32_t tS = tmem_base + C::COL_S;
  const uint32_t tO = tmem_base + C::COL_O;
  const uint32_t tA = tmem_base + C::COL_ACC;
  const int code_hi = (int)(blockIdx.x << 8);
  const uint32_t sQ = smem_u32(smem + C::OFF_Q);
  const uint32_t sK = smem_u32(smem + C::OFF_K);
  const uint32_t sV = smem_u32(smem + C::OFF_V);
  const uint32_t sP = smem_u32(smem + C::OFF_P);

  // The int32 accumulator tiles start every KV step from the bit pattern of 1.5*2^23 (see kMagicI).  It is
  // written by the tensor core itself: an fp16 MMA (K = 16, no accumulate) of a constant operand with
  // itself.  Every 16-byte chunk of the operand holds (1024, 1024, 2048, 0, 0, 0, 0, 0), so whatever the
  // layout each row's 16 values are two such chunks and the dot product of any two rows is
  // 2*(2^20 + 2^20 + 2^22) = 12582912 = 1.5*2^23, exactly, in fp32.
  if (threadIdx.x < C::MAGIC_BYTES / 16) {
    reinterpret_cast<uint4*>(smem + C::OFF_MAGIC)[threadIdx.x] = make_uint4(0x64006400u, 0x00006800u, 0u, 0u);
    fence_proxy_async_smem();
  }
  __syncthreads();
  pdl_wait();            // everything above touches nothing outside this CTA
  // (No pdl_launch here: the next call's quantisers would take the SMs that finish first and wait there in front of nothing:
  // headline calls back to back 5231 -> 5287 us, half-int8 causal 1549 -> 1581 us.)
  const uint64_t descArm = make_smem_desc(smem_u32(smem + C::OFF_MAGIC), 128, 256, 0);

  // work items: drawn from a global counter by the producer, published in a 4-slot ring
  auto wait_tile = [&](uint32_t seq) { return mbar_wait_warp(BAR(B_TILE + (seq & 3u)), (seq >> 2) & 1u, abort_flag, p.status, code_hi | PW_TILE); };
  auto next_tile = [&](uint32_t& seq) -> TileInfo {
    const uint32_t slot = seq & 3u;
    TileInfo t;
    t.nsteps = -1;
    if (!wait_tile(seq)) return t;
    ++seq;
    const TileInfo& s = tile_slot[slot];
    t.b = warp_uniform(s.b);
    t.h = warp_uniform(s.h);
    t.hk = warp_uniform(s.hk);
    t.mb = warp_uniform(s.mb);
    t.bh = warp_uniform(s.bh);
    t.work = warp_uniform(s.work);
    t.vh = 0;
    t.nsteps = warp_uniform(s.nsteps);
    if (lane == 0) mbar_arrive(BAR(B_TDONE + slot));
    return t;
  };

  // registers (THREADS x LAUNCH_REGS at launch): the service warps give most of theirs to the others
  if (warp < 4) reg_dealloc<kPipeServiceRegs>();

  if (warp == 0) {
    {
      // ------------------------------------------------------------------ TMA producer
      // (the whole warp runs the loop, one lane issues: as in the MMA warps)
      if (lane == 0) {
        prefetch_tmap(&tmQ);
        prefetch_tmap(&tmK);
        prefetch_tmap(&tmV);
      }
      uint32_t kv_it = 0, tile_it = 0, tseq = 0;
      int drawn = 0, passes_left = 0;      // NVH > 1: the query tile in hand and how many of its passes are still to publish
      bool ok = true;
#pragma unroll 1
      while (ok) {
        if (tseq >= 4u) {
          ok = mbar_wait_warp(BAR(B_TDONE + (tseq & 3u)), ((tseq >> 2) - 1u) & 1u, abort_flag, p.status, code_hi | PW_TILE);
          if (!ok) break;
        }
        int tile;
        if (NVH > 1 && passes_left > 0) {
          tile = drawn * NVH + (NVH - passes_left);      // the next pass over the same query tile, on this CTA
          --passes_left;
        } else {
          if (tseq == 0) {
            tile = (int)blockIdx.x;
          } else {
            tile = p.num_tiles;
            if (p.tile_counter) {
              if (lane == 0) tile = (int)(gridDim.x + atomicAdd(p.tile_counter, 1u));
              tile = warp_uniform(tile);
            }
          }
          if (tile >= p.num_tiles) {
            tile = -1;
          } else if (NVH > 1) {
            drawn = tile;
            tile *= NVH;
            passes_left = NVH - 1;
          }
        }
        TileInfo t;
        t.nsteps = -1;
        if (tile >= 0) t = decode_tile<RAGGED, NVH>(p, tile, G);
        if (lane == 0) {
          tile_slot[tseq & 3u] = t;
          mbar_arrive(BAR(B_TILE + (tseq & 3u)));
        }
        ++tseq;
        if (tile < 0) break;
        if (t.nsteps == 0) continue;
        ok = mbar_wait_warp(BAR(B_QEMPTY), (tile_it & 1) ^ 1, abort_flag, p.status, code_hi | PW_QE);
        if (!ok) break;
        if (elect_one()) {
          mbar_expect_tx(BAR(B_QFULL), C::Q_BYTES);
#pragma unroll
          for (int pn = 0; pn < C::QK_PANELS; ++pn)
            tma_load_4d(sQ + pn * (kBM * C::QK_ROWB), &tmQ, BAR(B_QFULL), pn * C::QK_ROWB, t.mb * kBM, t.h, t.b);
        }
        __syncwarp();
#pragma unroll 1
        for (int j = 0; j < t.nsteps; ++j, ++kv_it) {
          const uint32_t s = kv_it % NSK, ph = (kv_it / NSK) & 1;
          ok = mbar_wait_warp(BAR(B_KEMPTY + s), ph ^ 1, abort_flag, p.status, code_hi | PW_KE);
          if (!ok) break;
          const int jb = kv_tile_of_step(p, j, t.nsteps);
          if ((p.skip_k_load == 0 || kv_it + 1 != (uint32_t)p.skip_k_load) && elect_one()) {      // (test hook: a K tile that never arrives)
            mbar_expect_tx(BAR(B_QKRDY + s), C::K_BYTES);
#pragma unroll
            for (int pn = 0; pn < C::QK_PANELS; ++pn)
              tma_load_4d(sK + s * C::K_BYTES + pn * (G * C::QK_ROWB), &tmK, BAR(B_QKRDY + s), pn * C::QK_ROWB, jb * G, t.hk, t.b);
          }
          const uint32_t sv = kv_it % NSV, phv = (kv_it / NSV) & 1;
          __syncwarp();
          ok = mbar_wait_warp(BAR(B_VEMPTY + sv), phv ^ 1, abort_flag, p.status, code_hi | PW_VE);
          if (!ok) break;
          if (elect_one()) {
            mbar_expect_tx(BAR(B_PVRDY + sv), C::V_BYTES);
#pragma unroll
            for (int c = 0; c < C::V_BOXES; ++c)
              tma_load_4d(sV + sv * C::V_BYTES + c * (G * C::V_ROWB), &tmV, BAR(B_PVRDY + sv), t.vh * D + c * C::V_BOXCH, jb * G, t.hk, t.b);
          }
          __syncwarp();
        }
        ++tile_it;
      }
      // The last CTA to get here leaves the counter words zero for the next launch that is given them.
      if (lane == 0 && p.tile_counter && atomicAdd(p.tile_counter + 1, 1u) + 1u == gridDim.x) {
        p.tile_counter[0] = 0u;
        p.tile_counter[1] = 0u;
      }
    }
    __syncwarp();
  } else if (warp == 2) {
    // -------------------------------------------------------------------- K scales
    // The scales of KV step it go into slot it mod NKS, and the softmax warps see them through S_FULL of the step, which they
    // wait for anyway.  This warp waits for S_FULL of the step NSB back first: so that its arrival counts for its own step, and
    // because the softmax groups are done with the step another NSB back by then, whose slot this is at the latest.
    // Plain loads, one step ahead of the wait: rows may start anywhere (a cache of odd length) and hold fp16 or fp32; columns
    // past Nk read as zero.
    static_assert(C::NKS >= 2 * NSB, "K-scale slots");
    uint32_t kv_it = 0, tseq = 0;
    bool ok = true;
#pragma unroll 1
    while (ok) {
      const TileInfo t = next_tile(tseq);
      if (t.nsteps < 0) break;
      const long long row = (long long)t.b * p.ks_sb + (long long)t.hk * p.ks_sh;
      float ks[G / 32];
#pragma unroll 1
      for (int j = -1; j < t.nsteps; ++j) {
        if (j >= 0) {
          const uint32_t s = kv_it % NSB, ph = (kv_it / NSB) & 1;
          ok = mbar_wait_warp(BAR(B_SFULL + s), ph ^ 1, abort_flag, p.status, code_hi | PW_SFULL);
          if (!ok) break;
          float* slot = reinterpret_cast<float*>(smem + C::OFF_KS + (kv_it % C::NKS) * C::KS_BYTES) + lane;
#pragma unroll
          for (int i = 0; i < G / 32; ++i) slot[32 * i] = ks[i];
          __syncwarp();
          if (lane == 0) mbar_arrive(BAR(B_SFULL + s));
          ++kv_it;
        }
        if (j + 1 < t.nsteps) {
          const int col0 = kv_tile_of_step(p, j + 1, t.nsteps) * G + lane;
#pragma unroll
          for (int i = 0; i < G / 32; ++i)
            ks[i] = !RAGGED || col0 + 32 * i < p.Nk ? ld_scale(p.ks, row + col0 + 32 * i, p.scale_f16 & INTFA_SCALE_F16_K) : 0.f;
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    {
      // ------------------------------------------------------------------ MMA issuer for S = Q K^T
      // The whole warp runs the loop and the waits (warp-uniform control flow keeps the descriptor arithmetic
      // off the per-thread path); one elected lane issues the tensor-core instructions.
      // Step it goes into S buffer it mod NSB as soon as the step NSB back has been read out of it and K has landed.  The K stage is handed back by the tensor core itself (the
      // K scales sit in a ring of their own).
      uint32_t kv_it = 0, tile_it = 0, tseq = 0, sb = 0;    // sb: kv_it mod NSB
      bool ok = true;
      // operand descriptors of stage 0 / K step 0; the start-address field (16-byte units) takes the offsets
      const uint64_t descQ0 = make_smem_desc(sQ, 16, C::SBO_QK, C::SWZ_QK);
      const uint64_t descK0 = make_smem_desc(sK, 16, C::SBO_QK, C::SWZ_QK);
#pragma unroll 1
      while (ok) {
        const TileInfo t = next_tile(tseq);
        if (t.nsteps < 0) break;
        if (t.nsteps == 0) continue;
        ok = mbar_wait_warp(BAR(B_QFULL), tile_it & 1, abort_flag, p.status, code_hi | PW_QF);
        if (!ok) break;
#pragma unroll 1
        for (int j = 0; j < t.nsteps; ++j, ++kv_it) {
          const uint32_t s = kv_it % NSK, ph = (kv_it / NSK) & 1;
          ok = mbar_wait_warp(BAR(B_QKRDY + s), ph, abort_flag, p.status, code_hi | PW_QKRDY);
          if (!ok) break;
          tc_fence_after();
          const uint64_t bd0 = descK0 + (uint64_t)(s * (C::K_BYTES >> 4));
          const uint32_t tSb = tS + sb * G;
          if (elect_one()) {
            umma_f16(tSb, descArm, descArm, C::IDESC_ARM_S, 0);
#pragma unroll
            for (int kk = 0; kk < DQ / 32; ++kk) umma_i8(tSb, descQ0 + C::qk_slice(kk, kBM), bd0 + C::qk_slice(kk, G), C::IDESC_QK, 1);
            umma_commit(BAR(B_SFULL + sb));
            umma_commit(BAR(B_KEMPTY + s));
            if (j + 1 == t.nsteps) umma_commit(BAR(B_QEMPTY));
          }
          __syncwarp();
          sb = sb + 1 == NSB ? 0 : sb + 1;
        }
        ++tile_it;
      }
    }
    __syncwarp();
  } else if (warp == 3) {
    {
      // ------------------------------------------------------------------ MMA issuer for O_j = P V
      // A warp of its own, so that a Q K^T whose S buffer is free never queues behind the wait for a P tile.
      uint32_t kv_it = 0, tseq = 0, b = 0;                   // b: kv_it mod NPB
      bool ok = true;
      const uint64_t descP0 = make_smem_desc(sP, 16, C::SBO_P, C::SWZ_P);
      const uint64_t descV0 = make_smem_desc(sV, C::V_BOXES > 1 ? G * C::V_ROWB : 16, C::SBO_V, C::SWZ_V);
      // P_TMEM: the MMAs of a step (8 TMEM columns of P each) into the accumulator columns from d on; fp16 or e5m2 P and V (MN-major)
      auto pv_tmem = [&](uint32_t d, uint32_t b, uint64_t vd, uint32_t keep) {
#pragma unroll
        for (int kk = 0; kk < C::PV_STEPS; ++kk) {
          const uint64_t vdk = vd + (uint64_t)(kk * ((C::PV_K * C::V_ROWB) >> 4));
          if constexpr (F8V) umma_f8_ts(d, tS + b * G + kk * 8, vdk, C::IDESC_PV, kk > 0 ? 1u : keep);
          else umma_f16_ts(d, tS + b * G + kk * 8, vdk, C::IDESC_PV, kk > 0 ? 1u : keep);
        }
      };
#pragma unroll 1
      while (ok) {
        const TileInfo t = next_tile(tseq);
        if (t.nsteps < 0) break;
#pragma unroll 1
        for (int j = 0; j < t.nsteps; ++j, ++kv_it) {
          const uint32_t s = kv_it % NSV, ph = (kv_it / NSV) & 1;
          ok = mbar_wait_warp(BAR(B_PVRDY + s), ph, abort_flag, p.status, code_hi | PW_PVRDY);
          if (!ok) break;
          tc_fence_after();
          const uint64_t ad0 = descP0 + (uint64_t)(b * (C::P_BYTES >> 4));
          const uint64_t vd0 = descV0 + (uint64_t)(s * (C::V_BYTES >> 4));
          if constexpr (C::NOH > 1) {
            // the lower half of the channels
            if (elect_one()) {
              pv_tmem(tA, b, vd0, (j > 0 || p.state_in) ? 1u : 0u);
              umma_commit(BAR(B_OFULL));
            }
            __syncwarp();
            ok = mbar_wait_warp(BAR(B_OHI), kv_it & 1, abort_flag, p.status, code_hi | PW_PVRDY);
            if (!ok) break;
            tc_fence_after();
          }
          if (elect_one()) {
            if constexpr (FULL) {
              const uint32_t tOj = tO + kv_it % NO * D;
              umma_f16(tOj, descArm, descArm, C::IDESC_ARM_O, 0);
#pragma unroll
              for (int kk = 0; kk < G / 32; ++kk) umma_i8(tOj, ad0 + 2 * kk, vd0 + kk * ((32 * C::V_ROWB) >> 4), C::IDESC_PV, 1);
            } else if constexpr (C::P_TMEM) {
              // straight into the fp32 accumulator; the first P V of a fresh work item overwrites it
              pv_tmem(tA + (C::NOH - 1) * C::PV_N, b, vd0 + (C::NOH - 1) * (C::V_BOXES / 2 * G * C::V_ROWB >> 4), (j > 0 || p.state_in) ? 1u : 0u);
            } else {
              // e5m2 P (shared memory) x e5m2 V: both one byte, laid out like the int8 tiles
              const uint32_t keep = (j > 0 || p.state_in) ? 1u : 0u;
#pragma unroll
              for (int kk = 0; kk < G / 32; ++kk) umma_f8(tA, ad0 + 2 * kk, vd0 + kk * ((32 * C::V_ROWB) >> 4), C::IDESC_PV, kk > 0 ? 1u : keep);
            }
            umma_commit(BAR(B_OFULL + (C::NOH > 1 ? 1 : kv_it % NO)));
            umma_commit(BAR(B_VEMPTY + s));
            umma_commit(C::P_TMEM ? BAR(B_QKRDY + (kv_it + NSB) % NSK) : BAR(B_PFREE + b));
          }
          __syncwarp();
          b = b + 1 == C::NPB ? 0 : b + 1;
        }
      }
    }
    __syncwarp();
  } else if (warp >= 4 && warp < 4 + 4 * NGRP) {
    reg_alloc<C::SOFTMAX_REGS>();
#include "intfa_fwd_pipe_softmax.inc"
  } else if (warp >= 4 + 4 * NGRP) {
    if constexpr (C::CORR_REGS > C::LAUNCH_REGS) reg_alloc<C::CORR_REGS>(); else reg_dealloc<C::CORR_REGS>();
#include "intfa_fwd_pipe_update.inc"
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 2) {
    tc_fence_after();
    tmem_dealloc(tmem_base, C::TMEM_COLS);
  }
}

