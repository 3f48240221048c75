// Persistent passes for row and column lengths L = 256*M (radices 16, M, 16).
//
// tall_static and wide_static spend more than half of their time outside the
// arithmetic: at 3200K a row CTA of 34 K cycles loads for 7.5 K, waits 3 K for
// its predecessor's carries and meets ten barriers, and with 1.4 waves the
// CTAs of an SM do all of it in step (clock stamps per phase; FP64 pipe 25 %
// busy).  At 18432K one CTA fits an SM and nothing overlaps its 7.9 K cycles
// of loads, 3.4 K of table copies and 3.2 K of waiting.  Here one CTA per SM
// stays for the whole pass:
//   * its shared memory is a ring of NS slots, each one unit (two rows, or the
//     two columns of a pair).  A slot is filled by the copy engine (TMA) while
//     other slots are worked on;
//   * NG groups of 32*M threads, 16 elements per thread, work on units of
//     their own with named barriers of their own, so that the phases of the
//     units of an SM drift apart;
//   * the transforms run in place in the slot: four barriers per unit;
//   * the stage twiddles are copied once per pass instead of once per unit;
//   * results leave by the copy engine too (the 16-byte stores of two rows per
//     element took 3-5 K of 30 K cycles per unit).
// Measured (us per iteration, launch per unit -> persistent): 3200K 61.4 ->
// 55.2, 8192K 141 -> 125, 18432K 366 -> 267, 32768K 796 -> 555; a row unit at
// 18432K 39.5 K -> 25 K cycles, a column unit 24.0 K -> 19.8 K.  What bounds
// them now is shared memory and the FP64 pipe in turn, 58 % and 49 % of the
// cycles in the columns of 3072: its one group of twelve warps does both in step.
//
// In-place order.  A transform takes elements t + r*TR (TR = 16*M, r < 16) in
// thread t and leaves outputs c + r*TR in thread c:
//   stage 0: radix 16 over r            (t, j0),    t = u + 16*v
//   stage 1: radix M over v             (j0, j1, u)
//   stage 2: radix 16 over u            c = j0 + 16*j1
// with input twiddles w_TR^(j0*v) and w_L^(c*u).  The first transform of a
// pass reads the slot in natural order (x = t + r*TR) and leaves block order:
// the 16 inputs of stage 2 of thread c are the block x = 16*j1 + TR*j0 ..+15,
// permuted by an exclusive-or with j0 so that the threads of a warp meet all
// banks.  The second transform starts from the registers, writes stage 0 into
// the block its thread has just read, and ends in natural order.

template <int M>
struct Pipe {
  static_assert(M >= 4, "rows and columns of 1024 and more");
  static constexpr int L = 256 * M, TR = 16 * M, TU = 2 * TR;
  // groups: 16 warps of 128 registers per SM where whole groups allow it
  static constexpr int NG = M == 4 ? 4 : M == 5 ? 3 : M <= 8 ? 2 : 1;
  static constexpr int NT = NG * TU;
  static constexpr int SLOT = 32 * L;                  // bytes of a unit
  static constexpr int SS = M | 1;                     // stride of the stage-1 twiddles (odd: bank spread)
  static constexpr int TW2 = 8 * TR, TW1 = 16 * SS;    // twiddle entries of stage 2 and stage 1
  static constexpr int TWN = TW2 + TW1;
  // the slots that fit beside the row pass's tables (the column pass needs less)
  static constexpr int FIT = (227 * 1024 - 128 - (16 * TWN + 24 * TR + 64)) / (SLOT + 32 * 41 + 8);
  static constexpr int NS = FIT > 2 * NG ? 2 * NG : FIT;
  static_assert(NS >= NG && NS >= 1, "a slot per group");
};

// Twiddle table of a length: entry e < 8 of thread c at [e*TR + c], cosine and
// tangent of the powers of z = w_L^c that dft16_tw takes: z^8, z^4, z^2,
// -i*z^2*w8, z, z*w16, -i*z*w8, -i*z*w16^3; then the stage-1 twiddles w_TR^(j0*v) at
// [8*TR + j0*SS + v].

// a + e*b and a - e*b in six fused operations; w.x is the cosine, w.y the
// tangent of the twiddle: e*b = c*(b + i*t*b), so each result has two
// roundings.  (With a - e*b as 2a - (a + e*b) it has three.)  e = i^Q * w,
// conjugated for SIGN < 0.
//
// Accuracy.  An error of the stored cosine scales both parts of the twiddle, so
// with cosine and tangent rounded each by itself the twiddle's own error has up
// to twice the variance of a rounded (cosine, sine) pair.  And what the errors of
// all twiddles and constants have in common, a gain of the whole transform, adds
// up over the two passes: at 3072 x 3072 the rms of all roundoffs was 0.02111,
// with products and dft16 0.02031.  So the table holds the pair of neighbouring
// values whose twiddle has the smallest error, entries 3, 6 and 7 are turned back
// by a quarter (tangents below one), and the twiddles aim at a length that
// cancels the gain (host side).  Squaring of random words by two transforms of
// length L, rms error in units of 2^-53 and the gain of the square, products /
// rounded singly / this: 2304 3.52, -0.4 / 3.68, -0.7 / 3.43, 0.0; 3072 3.43, -0.2 /
// 3.53, -0.5 / 3.37, 0.0; 4096 3.72, 1.3 / 3.73, 1.2 / 3.41, 0.0; the other lengths 2
// to 9 % below products too.
template <int SIGN, int Q>
__device__ __forceinline__ void bfly(double2 &a, double2 &b, double2 w) {
  const double c = Q & 2 ? -w.x : w.x, t = SIGN > 0 ? w.y : -w.y;
  const double ux = fma(-t, b.y, b.x), uy = fma(t, b.x, b.y);  // w*b = c*u, up to the sign of Q & 2
  const double rx = Q & 1 ? (SIGN > 0 ? -uy : uy) : ux, ry = Q & 1 ? (SIGN > 0 ? ux : -ux) : uy;
  b = make_double2(fma(-c, rx, a.x), fma(-c, ry, a.y));
  a = make_double2(fma(c, rx, a.x), fma(c, ry, a.y));
}

// 16-point DFT of v[r]*z^r in 192 fused operations (60 of complex products
// and 160 of dft16 before): radix-2 layers whose twiddles are powers of z
// times sixteenth roots, 8 different up to a power of i.  tw(e) gives entry e
// of the table above.  Output k is left in v[slot16(k)].
__device__ __forceinline__ constexpr int slot16(int k) {  // bit reversal
  return ((k & 1) << 3) | ((k & 2) << 1) | ((k & 4) >> 1) | ((k & 8) >> 3);
}
template <int SIGN, class TW>
__device__ __forceinline__ void dft16_tw(double2 *v, TW tw) {
  {
    const double2 w = tw(0);
#pragma unroll
    for (int j = 0; j < 8; ++j) bfly<SIGN, 0>(v[j], v[j + 8], w);
  }
  {
    const double2 w = tw(1);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      bfly<SIGN, 0>(v[j], v[j + 4], w);
      bfly<SIGN, 1>(v[8 + j], v[8 + j + 4], w);
    }
  }
  {
    const double2 w = tw(2), w8 = tw(3);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      bfly<SIGN, 0>(v[j], v[j + 2], w);
      bfly<SIGN, 1>(v[4 + j], v[4 + j + 2], w);
      bfly<SIGN, 1>(v[8 + j], v[8 + j + 2], w8);
      bfly<SIGN, 2>(v[12 + j], v[12 + j + 2], w8);
    }
  }
  // nodes k mod 8 = 0, 4 (rotated), 2, 6, 1, 5, 3, 7
  bfly<SIGN, 0>(v[0], v[1], tw(4));
  bfly<SIGN, 1>(v[2], v[3], tw(4));
  bfly<SIGN, 1>(v[4], v[5], tw(6));
  bfly<SIGN, 2>(v[6], v[7], tw(6));
  bfly<SIGN, 0>(v[8], v[9], tw(5));
  bfly<SIGN, 1>(v[10], v[11], tw(5));
  bfly<SIGN, 1>(v[12], v[13], tw(7));
  bfly<SIGN, 2>(v[14], v[15], tw(7));
}

// e^(2 pi i e/16), e a compile-time value after unrolling.
__device__ __forceinline__ double2 root16(int e) {
  constexpr double c[5] = {1.0, C16_1, SQH, S16_1, 0.0};
  const int q = e >> 2, f = e & 3;
  const double x = c[f], y = c[4 - f];
  return q == 0 ? make_double2(x, y) : q == 1 ? make_double2(-y, x) : q == 2 ? make_double2(-x, -y) : make_double2(y, -x);
}

// Barriers of a group (named barrier id, TU threads).
template <int M>
struct GroupSync {
  int id;
  __device__ __forceinline__ void operator()() const {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(Pipe<M>::TU) : "memory");
  }
};
// mbarriers of the slots: one arrival (the thread that issues the copies)
// plus the bytes of the copies.  One thread of a group finds out whether its
// next slot has come, before the barrier that ends the unit before; only if it
// had not come by then the group waits for that thread.  Since the group goes
// by one thread's word, a wait that runs out (it is bounded, sets the timeout
// fault bit and makes every later wait of the CTA give up at once) ends the
// group's work without leaving any of its threads behind at a barrier.  A
// group that gives up draws no more units and touches no slot; the copies that
// its CTA has asked for by then are waited for before the CTA leaves (drain).
constexpr int kNotYet = -9, kGaveUp = -10;
__device__ __forceinline__ uint32_t smem32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void slot_init(uint64_t *bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem32(bar)) : "memory");
}
__device__ __forceinline__ void slot_expect(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 _, [%0], %1;" ::"r"(smem32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool slot_full(uint64_t *bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cta.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}"
      : "=r"(done)
      : "r"(smem32(bar)), "r"(parity)
      : "memory");
  return done != 0;
}
// pos_of: the position that the slot was last filled for.  A group may come to
// a position while the slot's earlier one has not been filled yet (another
// group is behind); the parity alone would then take the phase before that for
// its own.
__device__ __forceinline__ bool slot_wait(uint64_t *bar, uint32_t parity, volatile int *pos_of, int pos, DevState *st,
                                          volatile int *dead, long long limit) {
  long long t0 = 0;
  for (int k = 0;; ++k) {
    if (*pos_of == pos && slot_full(bar, parity)) return true;
    if (*dead) return false;
    const long long now = clock64();
    if (k == 0) t0 = now;
    if (now - t0 > limit) {
      *dead = 1;
      atomicOr(&st->fault, 1u);
      return false;
    }
  }
}
// Waits (bounded) until the flag is up and takes it down.
__device__ __forceinline__ void await_extra(uint32_t *flag, DevState *st, volatile int *dead, long long limit) {
  long long t0 = 0;
  for (int k = 0;; ++k) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(flag) : "memory");
    if (v || *dead) break;
    const long long now = clock64();
    if (k == 0) t0 = now;
    if (now - t0 > limit || ((k & 1023) == 1023 && (*(volatile uint32_t *)&st->fault & 1u))) {
      *dead = 1;
      atomicOr(&st->fault, 1u);
      break;
    }
  }
  *flag = 0;
}
// After a wait has run out: the copy that the slot was last filled by has
// landed before the CTA leaves its shared memory to another one (one thread
// per slot, all fills issued; bounded by itself, whatever the limit of the
// other waits).  pos < 0: never filled.
__device__ __forceinline__ void drain(uint64_t *bar, int pos, int slots) {
  if (pos < 0) return;
  const long long t0 = clock64();
  while (!slot_full(bar, (uint32_t)(pos / slots) & 1u) && clock64() - t0 < kWaitCycles) {
  }
}
__device__ __forceinline__ void copy_bulk(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
  asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem32(dst)),
               "l"(src), "r"(bytes), "r"(smem32(bar))
               : "memory");
}
__device__ __forceinline__ void copy_tile(void *dst, const void *map, int x, int y, uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
          smem32(dst)),
      "l"(map), "r"(x), "r"(y), "r"(smem32(bar))
      : "memory");
}
// Stores of a slot by the copy engine: one group of copies per thread and
// unit; store_read() returns when the thread's copies have read the slot.
__device__ __forceinline__ void store_bulk(void *dst, const void *src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(smem32(src)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void store_tile(const void *map, int x, int y, const void *src) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%1, %2}], [%3];" ::"l"(map), "r"(x),
               "r"(y), "r"(smem32(src))
               : "memory");
}
__device__ __forceinline__ void store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void store_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
// the slot's earlier generic accesses come before the copy engine's
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// Cells of a slot.  Rows (wide pass) are interleaved as the copy engine
// leaves them, x*32 + row*16; columns (tall pass) lie one after the other.
// swz(j0): the exclusive-or on x that spreads a warp's blocks over the banks.
struct RowCells {
  static constexpr int XB = 32;
  uint32_t base;  // byte offset of the row's cell 0
  __device__ __forceinline__ uint32_t swz(int j0) const { return (uint32_t)(j0 & 3); }
};
struct ColCells {
  static constexpr int XB = 16;
  uint32_t base;
  int col;
  __device__ __forceinline__ uint32_t swz(int j0) const { return (uint32_t)(2 * (j0 & 3) + col); }
};
__device__ __forceinline__ double2 &cell(unsigned char *sm, uint32_t byte) {
  return *reinterpret_cast<double2 *>(sm + byte);
}

// Stage 1 of one row or column: radix M over v, in place up to the
// permutation within 16 cells (one half warp or warp).  BLOCK: from natural
// to block order, else back.
template <int M, int SIGN, bool BLOCK, class C>
__device__ __forceinline__ void pipe_stage1(unsigned char *sm, const C cells, const double2 *tw1, int it0) {
  constexpr int TR = 16 * M, SS = Pipe<M>::SS, NB = (16 + M - 1) / M;
#pragma unroll
  for (int b = 0; b < NB; ++b) {
    const int it = it0 + b * TR;
    if (256 % TR == 0 || it < 256) {
      const int lo = it & 15, hi = it >> 4;
      const int j0 = BLOCK ? hi : lo;
      const uint32_t row = cells.base + (uint32_t)(hi * TR) * C::XB;
      const uint32_t nat = row + (uint32_t)lo * C::XB, blk = row + ((uint32_t)lo ^ cells.swz(hi)) * C::XB;
      const uint32_t in = BLOCK ? nat : blk, out = BLOCK ? blk : nat;
      double2 v[M];
#pragma unroll
      for (int k = 0; k < M; ++k) v[k] = cell(sm, in + k * 16 * C::XB);
#pragma unroll
      for (int k = 1; k < M; ++k) {
        const double2 w = tw1[j0 * SS + k];
        v[k] = SIGN > 0 ? cmul(v[k], w) : cmulc(v[k], w);
      }
      sdft<M, SIGN>(v);
      // the 16 cells of a group belong to 16 neighbouring lanes (32 with the
      // rows interleaved); in columns of odd M a warp may hold the end of one
      // column and the start of the other
      if constexpr (C::XB == 32 || M % 2 == 0) __syncwarp();
      else __syncwarp(0xffffu << (threadIdx.x & 16));
#pragma unroll
      for (int k = 0; k < M; ++k) cell(sm, out + k * 16 * C::XB) = v[sslot<M>(k)];
    }
  }
}

// First transform, after stage 0 (v: its outputs j0 in register slots S0 of
// thread t): block order, outputs c + r*TR of thread c = t in o.
template <int M, int SIGN, class C, class SY, class SLOT0>
__device__ __forceinline__ void pipe_first(unsigned char *sm, const C cells, const double2 *tw, int t, const C cells1,
                                           int it0, double2 *v, SLOT0 s0, SY sync) {
  constexpr int TR = 16 * M;
#pragma unroll
  for (int r = 0; r < 16; ++r) cell(sm, cells.base + (uint32_t)(t + r * TR) * C::XB) = v[s0(r)];
  sync();
  pipe_stage1<M, SIGN, true>(sm, cells1, tw + Pipe<M>::TW2, it0);
  sync();
  const uint32_t blk = cells.base + (uint32_t)((t >> 4) * 16 + (t & 15) * TR) * C::XB;
  const uint32_t x = cells.swz(t & 15);
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = cell(sm, blk + (((uint32_t)i ^ x) * C::XB));
  dft16_tw<SIGN>(v, [&](int e) { return tw[e * TR + t]; });
}

// Second transform: stage-0 outputs in v (slots s0) of thread t, into the
// block that thread has read; outputs c + r*TR in natural order.
template <int M, int SIGN, class C, class SY, class SLOT0>
__device__ __forceinline__ void pipe_second(unsigned char *sm, const C cells, const double2 *tw, int t, const C cells1,
                                            int it0, double2 *v, SLOT0 s0, SY sync) {
  constexpr int TR = 16 * M;
  const uint32_t blk = cells.base + (uint32_t)((t >> 4) * 16 + (t & 15) * TR) * C::XB;
  const uint32_t x = cells.swz(t & 15);
#pragma unroll
  for (int i = 0; i < 16; ++i) cell(sm, blk + (((uint32_t)i ^ x) * C::XB)) = v[s0(i)];
  sync();
  pipe_stage1<M, SIGN, false>(sm, cells1, tw + Pipe<M>::TW2, it0);
  sync();
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = cell(sm, cells.base + (uint32_t)(t + i * TR) * C::XB);
  dft16_tw<SIGN>(v, [&](int e) { return tw[e * TR + t]; });
}

// ------------------------------------------------------------- tall pass --
// Constants of a column pair: for both columns the 16 factors g^r = w_N^(k*TR*r)
// of the column twiddles, and w_N^kA of the pairing.
constexpr int kPairConst = 33;

template <int M>
constexpr int tall_pipe_smem() {
  using P = Pipe<M>;
  return P::NS * P::SLOT + 16 * P::TWN + 32 * (P::NS + P::NG) * kPairConst + 8 * P::NS + 16;
}

template <int M>
__global__ void __launch_bounds__(Pipe<M>::NT, 1) tall_pipe(const __grid_constant__ TallArgs a) {
  using P = Pipe<M>;
  constexpr int H = P::L, TR = P::TR, TU = P::TU, NS = P::NS, NG = P::NG;
  extern __shared__ __align__(128) unsigned char smb[];
  double2 *tw = reinterpret_cast<double2 *>(smb + NS * P::SLOT);
  double2 *pc = tw + P::TWN;  // constants of the pairs, area position % (2*NS)
  double2 *raw = pc + 2 * NS * kPairConst;  // table entries of a group's next constants
  uint64_t *full = reinterpret_cast<uint64_t *>(raw + 2 * NG * kPairConst);
  __shared__ int s_dead, s_go[NG], s_pos[NS];
  const int W = a.W, units = W / 2;
  const int g = threadIdx.x / TU, idx = threadIdx.x - g * TU;
  // lanes 2q, 2q+1: thread q of column kA and its mirror TR-1-q of column kB
  const int col = idx & 1, t = col ? TR - 1 - (idx >> 1) : idx >> 1;
  const int col1 = idx / TR, it0 = idx - col1 * TR;  // stage 1: a column's items in order
  const GroupSync<M> sync{1 + g};

  for (int i = threadIdx.x; i < P::TWN; i += P::NT) cp_async16(&tw[i], &a.ptw[i]);
  if (threadIdx.x == 0) {
    s_dead = 0;
    for (int s = 0; s < NS; ++s) {
      s_pos[s] = -1;
      slot_init(&full[s]);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // Constants of pair u, entry i: product of two table entries, fetched into
  // shared memory (raw) while the unit before is worked on.
  auto constant_exp = [&](int u, int i) {
    if (i == 32) return u;
    return (i < 16 ? u : u == 0 ? W / 2 : W - u) * TR * (i & 15);
  };
  auto fill = [&](int u, int pos) {  // one thread
    const int slot = pos % NS;
    unsigned char *dst = smb + slot * P::SLOT;
    s_pos[slot] = pos;
    slot_expect(&full[slot], 32u * H);
    copy_bulk(dst, a.A + (size_t)u * H, 16u * H, &full[slot]);
    copy_bulk(dst + 16 * H, a.A + (size_t)(u == 0 ? W / 2 : W - u) * H, 16u * H, &full[slot]);
  };
  for (int i = threadIdx.x; i < NS * kPairConst; i += P::NT) {
    const int p = i / kPairConst, u = blockIdx.x + p * gridDim.x;
    if (u < units) pc[i] = omegaN(a.thi, a.tlo, a.ts, a.tmask, constant_exp(u, i - p * kPairConst));
  }
  // stage twiddle of the pairing that does not depend on the unit: w_H^tA
  const double2 wh = __ldg(&a.twH[col ? TR - 1 - t : t]);
  cp_async_wait_all();
  __syncthreads();
  griddep_wait();
  griddep_release();
  if (threadIdx.x == 0) {
    for (int s = 0; s < NS; ++s)
      if ((int)(blockIdx.x + s * gridDim.x) < units) fill(blockIdx.x + s * gridDim.x, s);
    if (blockIdx.x == 0) {
      const uint32_t o = a.st->offset;  // CUDALucas.cu:1882, once per iteration
      a.st->offset = (uint32_t)((2ull * o) % a.q);
    }
  }
  // refill of the group's last slot, once its stores have read it (the
  // thread that issued them)
  int refill_unit = -1, refill_pos = 0;
  auto refill = [&] {
    if (refill_unit >= 0) {
      store_read();
      fill(refill_unit, refill_pos);
      refill_unit = -1;
    }
  };
  for (int pos = g;; pos += NG) {
    const int u = blockIdx.x + pos * gridDim.x;
    if (u >= units) break;
    if (NS == NG) refill();
    const int slot = pos % NS;
    const double2 *cst = pc + (pos % (2 * NS)) * kPairConst;
    const bool special = u == 0;
    const int kA = u, kB = special ? W / 2 : W - u;
    const int k1 = col ? kB : kA;
    ColCells cells{(uint32_t)(slot * P::SLOT + col * 16 * H), col};
    ColCells cells1{(uint32_t)(slot * P::SLOT + col1 * 16 * H), col1};
    // column twiddle w_N^(k1*x), x = t + r*TR: base * g^r
    const int eb = k1 * t;
    // fetch the constants of the unit that will be loaded into this slot
    const int un = blockIdx.x + (pos + NS) * gridDim.x;
    for (int i = idx; i < kPairConst && un < units; i += TU) {
      const int e = constant_exp(un, i);
      double2 *rw = raw + 2 * (g * kPairConst + i);
      cp_async16(rw, &a.thi[e >> a.ts]);
      cp_async16(rw + 1, &a.tlo[e & a.tmask]);
    }
    const double2 bh = __ldg(&a.thi[eb >> a.ts]), bl = __ldg(&a.tlo[eb & a.tmask]);
    const uint32_t parity = (uint32_t)(pos / NS) & 1u;
    int go = pos == g ? kNotYet : s_go[g];
    if (go == kNotYet) {
      sync();
      if (idx == TU - 1) s_go[g] = slot_wait(&full[slot], parity, &s_pos[slot], pos, a.st, &s_dead, a.wait);
      sync();
      go = s_go[g];
    }
    if (!go) break;
    slot_full(&full[slot], parity);  // every thread sees the copies
    double2 v[16];
#pragma unroll
    for (int r = 0; r < 16; ++r) v[r] = cell(smb, cells.base + (uint32_t)(t + r * TR) * 16);
    const double2 *gc = cst + 16 * col;
    // each element times its own twiddle: folded into the transform's layers
    // the factors are products of four rounded ones
    const double2 base = cmul(bh, bl);
#pragma unroll
    for (int r = 0; r < 16; ++r) v[r] = cmul(v[r], cmul(base, gc[r]));
    dft16<+1>(v);
    auto ord16 = [](int r) { return out_slot<16>(r); };
    pipe_first<M, +1>(smb, cells, tw, t, cells1, it0, v, ord16, sync);
    if (NS > NG) refill();
    if (!special) {
      // bin c + r*TR of column kA pairs with bin (TR-1-c) + (15-r)*TR of
      // column kB, held by the neighbouring lane: each lane takes the lower
      // half of its own bins.  Swapping the two bins and conjugating w swaps
      // the results, so both lanes make the same call.
      const double2 wb = cmul(cst[32], wh);
      const double sg = col ? -1.0 : 1.0;
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        double2 z = v[slot16(15 - r)];
        z.x = __shfl_xor_sync(0xffffffffu, z.x, 1);
        z.y = __shfl_xor_sync(0xffffffffu, z.y, 1);
        // w_H^(r*TR) = w16^r; column kB: w16^(15-r)
        const double2 fr = root16(r), fm = root16(15 - r);
        double2 w = cmul(wb, make_double2(col ? fm.x : fr.x, col ? fm.y : fr.y));
        w.y *= sg;
        pair_square(v[slot16(r)], z, w);
        z.x = __shfl_xor_sync(0xffffffffu, z.x, 1);
        z.y = __shfl_xor_sync(0xffffffffu, z.y, 1);
        v[slot16(15 - r)] = z;
      }
    } else {
      // the self-paired columns 0 and W/2, by index through the slot
      sync();
#pragma unroll
      for (int r = 0; r < 16; ++r) cell(smb, cells.base + (uint32_t)(t + r * TR) * 16) = v[slot16(r)];
      sync();
      double2 *ca = reinterpret_cast<double2 *>(smb + slot * P::SLOT), *cb = ca + H;
      for (int i = idx; i <= H / 2; i += TU) {  // column 0: k2 <-> (H-k2) mod H
        const int p = (H - i) % H;
        double2 za = ca[i], zb = ca[p];
        pair_square(za, zb, __ldg(&a.twH[i]));
        ca[i] = za;
        if (p != i) ca[p] = zb;
      }
      const double2 wb = omegaN(a.thi, a.tlo, a.ts, a.tmask, W / 2);
      for (int i = idx; i < H / 2; i += TU) {  // column W/2: k2 <-> H-1-k2
        double2 za = cb[i], zb = cb[H - 1 - i];
        pair_square(za, zb, cmul(wb, __ldg(&a.twH[i])));
        cb[i] = za;
        cb[H - 1 - i] = zb;
      }
      sync();
#pragma unroll
      for (int r = 0; r < 16; ++r) v[slot16(r)] = cell(smb, cells.base + (uint32_t)(t + r * TR) * 16);
      sync();
    }
    {
      double2 w[16];
#pragma unroll
      for (int r = 0; r < 16; ++r) w[r] = v[slot16(r)];
      dft16<-1>(w);
#pragma unroll
      for (int r = 0; r < 16; ++r) v[r] = w[r];
    }
    pipe_second<M, -1>(smb, cells, tw, t, cells1, it0, v, ord16, sync);
    // the results go into the cells just read, and to memory by the copy engine
#pragma unroll
    for (int r = 0; r < 16; ++r)
      cell(smb, cells.base + (uint32_t)(t + r * TR) * 16) = cmulc(v[slot16(r)], cmul(base, gc[r]));
    if (un < units) {
      cp_async_wait_all();
      for (int i = idx; i < kPairConst; i += TU) {
        const double2 *rw = raw + 2 * (g * kPairConst + i);
        pc[((pos + NS) % (2 * NS)) * kPairConst + i] = cmul(rw[0], rw[1]);
      }
    }
    fence_async_smem();
    if (idx == TU - 1) {
      const int np = pos + NG, ns = np % NS;
      s_go[g] = *(volatile int *)&s_pos[ns] == np && slot_full(&full[ns], (uint32_t)(np / NS) & 1u) ? 1 : kNotYet;
    }
    sync();
    if (idx == 0) {
      store_bulk(a.A + (size_t)kA * H, smb + slot * P::SLOT, 16u * H);
      store_bulk(a.A + (size_t)kB * H, smb + slot * P::SLOT + 16 * H, 16u * H);
      store_commit();
      if (un < units) {
        refill_unit = un;
        refill_pos = pos + NS;
      }
    }
  }
  // a refill that is still due belongs to another group's next unit
  if (!*(volatile int *)&s_dead) refill();
  store_read();
  cp_async_wait_all();
  __syncthreads();
  if (s_dead && threadIdx.x < NS) drain(&full[threadIdx.x], s_pos[threadIdx.x], NS);
}

// ------------------------------------------------------------- wide pass --
template <int M>
constexpr int wide_pipe_smem() {
  using P = Pipe<M>;
  return P::NS * P::SLOT + 16 * P::TWN + 24 * P::TR + 96 * P::NS + 16 * P::NS + 64;
}

// Units (row groups of two rows) are worked on in the order of tickets, and a
// unit waits for the carries of the unit before it.  That unit has an earlier
// ticket, so it is being worked on already whichever CTAs are resident: no
// deadlock.  It should have been drawn well before, or every unit waits for
// its slowest neighbours (18432K: 8 to 15 K of 35 K cycles with consecutive
// tickets): the units form `chains` runs that advance side by side.  The first
// unit of a run, whose predecessor ends the run before, takes its carries from
// an extra ticket at the start, which computes that predecessor as far as its
// outgoing carries only (for unit 0 the last unit: the wrap, 2^q = 1); the
// predecessor itself is not stored before the extra ticket has read it.
struct RunOrder {
  int units, chains, len;  // runs of `len` units (the last ones shorter, or empty)
  // The unit of ticket k: run k % chains, its extra unit first; -1: none.
  __host__ __device__ __forceinline__ int unit(int k) const {
    const int i = k / chains, j = k - i * chains, first = j * len;
    if (first >= units) return -1;
    if (i == 0) return (j == 0 ? units : first) - 1;
    return first + i - 1 < units ? first + i - 1 : -1;
  }
  __host__ __device__ __forceinline__ int tickets() const { return chains * (len + 1); }
  __host__ __device__ __forceinline__ bool extra(int k) const { return k < chains; }
  // whether u ends its run, and the run whose extra ticket then reads it
  __host__ __device__ __forceinline__ bool tail(int u) const { return u % len == len - 1 || u == units - 1; }
  __host__ __device__ __forceinline__ int reader(int u) const { return u == units - 1 ? 0 : u / len + 1; }
};
// A multiple of the slots, about 32 runs, of four units or more each.
inline RunOrder run_order(int slots, int units) {
  const int chains = slots * std::max(1, std::min(32 / slots, units / (4 * slots)));
  return {units, chains, (units + chains - 1) / chains};
}
// What the pass relies on: every unit once; the unit before at an earlier ticket
// (else CTAs could wait for one that has not been drawn), or, at the start of a
// run, the run's extra ticket for it; that one before its unit is drawn, and
// flagged by the unit that ends the run.
inline bool run_order_ok(const RunOrder &o) {
  std::vector<int> at((size_t)o.units, -1);
  for (int k = o.chains; k < o.tickets(); ++k) {
    const int u = o.unit(k);
    if (u < 0) continue;
    if (u >= o.units || at[(size_t)u] >= 0) return false;
    at[(size_t)u] = k;
  }
  for (int u = 0; u < o.units; ++u) {
    const int before = u == 0 ? o.units - 1 : u - 1;
    if (at[(size_t)u] < 0) return false;
    if (u % o.len == 0) {
      const int k = u / o.len;
      if (k >= o.chains || o.unit(k) != before || k >= at[(size_t)before] || !o.tail(before) || o.reader(before) != k)
        return false;
    } else if (at[(size_t)before] >= at[(size_t)u] || o.tail(before)) {
      return false;
    }
  }
  return true;
}

template <int M>
__global__ void __launch_bounds__(Pipe<M>::NT, 1)
    wide_pipe(const __grid_constant__ TileMap map, const __grid_constant__ WideArgs a) {
  using P = Pipe<M>;
  constexpr int W = P::L, TR = P::TR, TU = P::TU, NS = P::NS, NG = P::NG;
  extern __shared__ __align__(128) unsigned char smb[];
  double2 *tw = reinterpret_cast<double2 *>(smb + NS * P::SLOT);
  double2 *cwt = tw + P::TWN;                                  // column weights 2^(colF/n), 2^(-colF/n)
  RowConst *rc = reinterpret_cast<RowConst *>(cwt + TR);       // row constants of the slots' units
  uint64_t *full = reinterpret_cast<uint64_t *>(rc + 2 * NS);
  int *cfe = reinterpret_cast<int *>(full + NS);               // column exponents
  int *unit_of = cfe + TR;  // ticket of the slot's unit, -1: no more, -2: a ticket without a unit
  __shared__ double s_two[NG][2];
  __shared__ uint32_t s_sub[NG][2];
  __shared__ int s_dead, s_first, s_go[NG], s_next[NG], s_pos[NS];
  const int g = threadIdx.x / TU, idx = threadIdx.x - g * TU;
  const int row = idx & 1, t = idx >> 1;
  const GroupSync<M> sync{1 + g};
  const int warp = idx >> 5, lane = threadIdx.x & 31;
  const int H = a.H, n = (int)a.n, units = H / 2;
  double *gcd = reinterpret_cast<double *>(a.carry);

  for (int i = threadIdx.x; i < P::TWN; i += P::NT) cp_async16(&tw[i], &a.ptw[i]);
  for (int i = threadIdx.x; i < TR; i += P::NT) {
    cwt[i] = make_double2(__ldg(&a.colW[i]), __ldg(&a.colWi[i]));
    cfe[i] = __ldg(&a.colF[i]);
  }
  if (threadIdx.x == 0) {
    s_dead = 0;
    for (int s = 0; s < NS; ++s) {
      s_pos[s] = -1;
      slot_init(&full[s]);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  const WordSize ws(a.lim, (int)a.qn);
  cp_async_wait_all();
  __syncthreads();
  griddep_wait();
  griddep_release();
  const RunOrder order{units, a.chains, a.chain_len};
  auto fill = [&](int k, int pos, int box, bool first) {
    const int slot = pos % NS;
    if (first) s_pos[slot] = pos;
    const int u = k < order.tickets() ? order.unit(k) : -1;
    if (u < 0) {
      if (first) {
        unit_of[slot] = k < order.tickets() ? -2 : -1;
        slot_expect(&full[slot], 0);
      }
      return;
    }
    if (first) {
      unit_of[slot] = k;
      slot_expect(&full[slot], 32u * W + 2 * (uint32_t)sizeof(RowConst));
      copy_bulk(&rc[2 * slot], &a.rowC[2 * u], 2 * (uint32_t)sizeof(RowConst), &full[slot]);
    }
    copy_tile(smb + slot * P::SLOT + box * 8192, &map, 4 * u, box * 256, &full[slot]);
  };
  // The first tickets, one per slot.  `chains` is a multiple of NS, so a
  // unit's predecessor sits in the same slot of another CTA: it is worked on
  // in the same round.
  if (threadIdx.x == 0) s_first = (int)atomicAdd(&a.st->pipe_ticket, (unsigned)NS);
  __syncthreads();
  if (lane == 0) {
    fill(s_first + g, g, warp, warp == 0);
    if (g < NS - NG) fill(s_first + NG + g, NG + g, warp, warp == 0);
  }
  if (idx == TU - 1) {  // seen by the group after the barriers of its first transform
    const MinusTwo two(__ldcg(&a.st->offset), a);
    s_sub[g][0] = two.m1;
    s_sub[g][1] = two.m2;
    s_two[g][0] = two.s0;
    s_two[g][1] = two.s1;
  }
  const uint32_t seen = __ldcg(&a.st->err_bits);
  Readings<> rd;
  // refill of the group's last slot, each warp its box, once the stores that
  // the warp has issued have read it
  int refill_pos = -1;
  auto refill = [&] {
    if (lane == 0 && refill_pos >= 0) {
      store_read();
      fill(s_next[g], refill_pos, warp, warp == 0);
    }
    refill_pos = -1;
  };
  for (int pos = g;; pos += NG) {
    const int slot = pos % NS;
    if (NS == NG) refill();
    const uint32_t parity = (uint32_t)(pos / NS) & 1u;
    int k = pos == g ? kNotYet : s_go[g];
    if (k == kNotYet) {
      sync();
      if (idx == TU - 1)
        s_go[g] = slot_wait(&full[slot], parity, &s_pos[slot], pos, a.st, &s_dead, a.wait) ? unit_of[slot] : kGaveUp;
      sync();
      k = s_go[g];
    }
    if (k == kGaveUp) break;
    if (k == -1) {
      // no more: pass that on to the group that takes this slot next
      if (idx == 0) {
        unit_of[slot] = -1;
        s_pos[slot] = pos + NS;
        slot_expect(&full[slot], 0);
      }
      refill();  // due to another group's next unit
      break;
    }
    // the next ticket of this slot, needed when the unit is done
    unsigned next = 0;
    if (idx == 0) next = *(volatile int *)&s_dead ? 0x7fffffffu : atomicAdd(&a.st->pipe_ticket, 1u);  // (no ticket: no fill)
    auto done = [&] {  // after a barrier since the last refill()
      if (idx == 0) s_next[g] = (int)min(next, 0x7fffffffu);
      fence_async_smem();
      if (idx == TU - 1) {
        const int np = pos + NG, ns = np % NS;
        s_go[g] = *(volatile int *)&s_pos[ns] == np && slot_full(&full[ns], (uint32_t)(np / NS) & 1u) ? unit_of[ns] : kNotYet;
      }
      sync();
      refill_pos = pos + NS;
    };
    if (k == -2) {  // a ticket without a unit (runs of unequal length)
      refill();
      sync();
      done();
      continue;
    }
    slot_full(&full[slot], parity);  // every thread sees the copies
    const bool extra = order.extra(k);
    const int u = order.unit(k);
    const RowCells cells{(uint32_t)(slot * P::SLOT + row * 16)};
    auto ord16 = [](int r) { return out_slot<16>(r); };
    double2 v[16];
#pragma unroll
    for (int r = 0; r < 16; ++r) v[r] = cell(smb, cells.base + (uint32_t)(t + r * TR) * 32);
    dft16<-1>(v);
    pipe_first<M, -1>(smb, cells, tw, t, cells, t, v, ord16, sync);
    // word s of element m1 = t + r*TR: exponent E_s - D_r, as in wide_body
    const RowConst rcn = rc[2 * slot + row];
    const int m2 = 2 * u + row;
    const int cf = cfe[t];
    const double2 cw = cwt[t];
    int E0 = rcn.e0 + cf, E1 = rcn.e1 + cf;
    const bool w0 = E0 >= n, w1 = E1 >= n;
    if (w0) E0 -= n;
    if (w1) E1 -= n;
    const uint32_t F0 = turn_fraction(E0, a.turn), F1 = turn_fraction(E1, a.turn);
    double2 *pk = v;  // (packed pair, outgoing carry) of element r in pk[slot16(r)]
    {
      const double Wi0 = rcn.wi0 * cw.y * (w0 ? 2.0 : 1.0), Wi1 = rcn.wi1 * cw.y * (w1 ? 2.0 : 1.0);
      const int r_sub = (int)s_sub[g][1] == m2 && (int)(s_sub[g][0] % TR) == t ? (int)(s_sub[g][0] / TR) : -1;
#pragma unroll
      for (int r = 0; r < 16; ++r) {
        const uint32_t D = a.colD[r];
        double P0, I0, P1, I1;
        ws.at(F0 - D, P0, I0);
        ws.at(F1 - D, P1, I1);
        const double2 z = v[slot16(r)];
        const double t0 = z.x * scale_exp(Wi0 * a.colSi[r], F0 < D ? -kExpOne : 0);
        const double t1 = z.y * scale_exp(Wi1 * a.colSi[r], F1 < D ? -kExpOne : 0);
        double r0 = rnd_int(t0), r1 = rnd_int(t1);
        rd.words(t0, r0, t1, r1);
        if (r == r_sub) {
          r0 -= s_two[g][0];
          r1 -= s_two[g][1];
        }
        carry_split(r0, r1, P0, I0, P1, I1, pk[slot16(r)].x, pk[slot16(r)].y);
      }
    }
    // The rows of an element sit in neighbouring lanes: row 1 takes row 0's
    // carries by shuffles, row 0 those of the unit before (unit 0 the last
    // unit's, shifted by one element).  The last unit of a run publishes
    // none: the run after it takes those of its extra ticket.
    const bool tail = order.tail(u);  // of its run
    if (row == 1 && (extra || !tail)) {
      double *out = gcd + (size_t)u * W + t;
#pragma unroll
      for (int r = 0; r < 16; ++r) put_carry(&out[r * TR], pk[slot16(r)].y);
    }
    if (NS > NG) refill();
    if (extra) {
      sync();
      // the extra ticket's unit has been read: the run before may store it
      if (idx == 0) asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(&a.flags[k]), "r"(1u) : "memory");
    } else {
      double cin[16];
#pragma unroll
      for (int r = 0; r < 16; ++r) cin[r] = __shfl_up_sync(0xffffffffu, pk[slot16(r)].y, 1);
      if (row == 0) {
        double *in = gcd + (size_t)(u == 0 ? units - 1 : u - 1) * W;
        take_carries<16>(cin, [&](int r) {
          const int m1 = t + r * TR;
          return in + (u == 0 ? (m1 == 0 ? W - 1 : m1 - 1) : m1);
        }, a.st, a.wait);
      }
      const double W0 = rcn.w0 * cw.x * (w0 ? 0.5 : 1.0), W1 = rcn.w1 * cw.x * (w1 ? 0.5 : 1.0);
      double2 x[16];
#pragma unroll
      for (int r = 0; r < 16; ++r) {
        const uint32_t D = a.colD[r];
        double P0, I0, d0, d1;
        ws.at(F0 - D, P0, I0);
        carry_join(pk[slot16(r)].x, cin[r], P0, I0, d0, d1);
        x[r] = make_double2(d0 * scale_exp(W0 * a.colS[r], F0 < D ? kExpOne : 0),
                            d1 * scale_exp(W1 * a.colS[r], F1 < D ? kExpOne : 0));
      }
      dft16<+1>(x);
      pipe_second<M, +1>(smb, cells, tw, t, cells, t, x, ord16, sync);
      // into the cells just read, and to memory by the copy engine
#pragma unroll
      for (int r = 0; r < 16; ++r) cell(smb, cells.base + (uint32_t)(t + r * TR) * 32) = x[slot16(r)];
    }
    if (!extra && tail && idx == 0) await_extra(&a.flags[order.reader(u)], a.st, &s_dead, a.wait);
    done();
    if (!extra && lane == 0) {
      store_tile(&map, 4 * u, warp * 256, smb + slot * P::SLOT + warp * 8192);
      store_commit();
    }
  }
  if (lane == 0) store_read();
  rd.publish(a.st, seen);
  __syncthreads();
  if (s_dead && threadIdx.x < NS) drain(&full[threadIdx.x], s_pos[threadIdx.x], NS);
  if (threadIdx.x == 0) {
    // the last CTA to leave puts the ticket counter back
    __threadfence();
    if (atomicInc(&a.st->pipe_exit, gridDim.x - 1) == gridDim.x - 1) a.st->pipe_ticket = 0;
  }
}
