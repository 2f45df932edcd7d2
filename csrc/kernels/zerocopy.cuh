// Zero-copy collective kernels: the peers' user buffers are read and written in place.
//
// A buffer qualifies when every rank can reach it: it lies in the symmetric heap (flagcxMemAlloc) or in a
// segment made peer-visible by flagcxCommRegister.  The reference gives registration the same meaning: a
// registered buffer skips the staging copy of its transport (flagcx/core/net.cc:150-168, 234-246) and, on one
// vendor's GPUs, is handed to the vendor library's own registration (flagcx/flagcx.cc:186-201).
//
// Protocol of every kind in this file (one launch, the same CTA count on every rank):
//   1. each CTA writes where its rank's buffers live (segment, offset) into a mailbox on every peer and
//      raises its flag there (release); it then waits for the same from the peers' CTA of the same index.
//      A peer's kernel having started means that everything queued before it on the peer's stream is done,
//      so after this barrier the peers' send buffers hold their data and their recv buffers may be written;
//   2. the data phase: loads from the peers' send buffers and/or stores into the peers' recv buffers, or
//      multimem.ld_reduce / multimem.st on the NVSwitch multicast alias when the buffers sit at the same
//      heap offset on every rank;
//   3. a second barrier: a rank leaves only when no peer CTA still reads or writes its buffers.
// Nothing is staged, so a message makes one pass over NVLink and at most one over local memory, and there
// is no size limit per launch.
//
#pragma once
#include "prims.cuh"

namespace fcxdev {

struct ZcPeers {
  const char *send[FCX_MAX_RANKS];  // rank p's send buffer as this rank addresses it (null: not peer-visible)
  char *recv[FCX_MAX_RANKS];
  const char *mcSend;               // multicast alias of the send buffers, null unless all ranks use one heap offset
  char *mcRecv;
  uint64_t x[FCX_MAX_RANKS], y[FCX_MAX_RANKS];  // two free words per source rank (all-to-all-v: displacement, count)
};

// Step 1 of the protocol.  `needSend` / `needRecv`: which buffers the kind will touch on the peers; a peer
// whose buffer is not visible, or a heap range that leaves the heap, ends the collective with a recorded
// FCX_ERR_BADARG instead of a wild access.  sendSpan / recvSpan are the bytes a peer may touch from the offset.
// xTo[p] / yTo[p]: two words handed to rank p (may be null).
__device__ __forceinline__ bool zcExchange(const FcxDevComm &dc, const FcxCollArgs &a, uint64_t seq, int cta, bool needSend,
                                           bool needRecv, size_t sendSpan, size_t recvSpan, const uint64_t *xTo,
                                           const uint64_t *yTo, ZcPeers *z) {
  const int n = dc.nranks, me = dc.rank, t = threadIdx.x;
  __syncthreads();
  bool ok = true;
  if (t < n && t != me) {
    FcxMail *mb = (FcxMail *)(dc.heap[t] + FCX_OFF_MAIL) + (seq & 1) * FCX_MAX_RANKS + me;
    stRelaxed(&mb->a, (uint64_t)(int64_t)a.sendSeg);
    stRelaxed(&mb->b, a.sendHeapOff);
    stRelaxed(&mb->c, (uint64_t)(int64_t)a.recvSeg);
    stRelaxed(&mb->d, a.recvHeapOff);
    stRelaxed(&mb->e, xTo ? xTo[t] : 0);
    stRelaxed(&mb->f, yTo ? yTo[t] : 0);
    stRelease(flagSlot(dc, t, cta, me), barrierValue(seq, 1));
    ok = waitGe(dc, flagSlot(dc, me, cta, t), barrierValue(seq, 1), t, FCX_WAIT_BARRIER, cta, seq);
  }
  if (!__syncthreads_and(ok)) return false;
  bool symS = a.sendSeg == FCX_SEG_HEAP, symR = a.recvSeg == FCX_SEG_HEAP, bad = false;
  int badPeer = me;
  for (int p = 0; p < n; p++) {
    int sseg, rseg;
    uint64_t soff, roff;
    if (p == me) {
      sseg = a.sendSeg; soff = a.sendHeapOff; rseg = a.recvSeg; roff = a.recvHeapOff;
      z->x[p] = xTo ? xTo[me] : 0;
      z->y[p] = yTo ? yTo[me] : 0;
      // this rank's own buffers are used through the pointers the caller gave
      z->send[p] = (const char *)a.send;
      z->recv[p] = (char *)a.recv;
      if ((needSend && (sseg == FCX_SEG_NONE || !a.send)) || (needRecv && (rseg == FCX_SEG_NONE || !a.recv))) { bad = true; badPeer = p; }
    } else {
      const FcxMail *mb = (const FcxMail *)(dc.heap[me] + FCX_OFF_MAIL) + (seq & 1) * FCX_MAX_RANKS + p;
      sseg = (int)(int64_t)ldRelaxed(&mb->a); soff = ldRelaxed(&mb->b);
      rseg = (int)(int64_t)ldRelaxed(&mb->c); roff = ldRelaxed(&mb->d);
      z->x[p] = ldRelaxed(&mb->e);
      z->y[p] = ldRelaxed(&mb->f);
      z->send[p] = needSend ? zcResolve(dc, sseg, soff, p) : nullptr;
      z->recv[p] = needRecv ? zcResolve(dc, rseg, roff, p) : nullptr;
      if ((needSend && !z->send[p]) || (needRecv && !z->recv[p])) { bad = true; badPeer = p; }
    }
    if (needSend && sseg == FCX_SEG_HEAP && (soff > dc.heapBytes || sendSpan > dc.heapBytes - soff)) { bad = true; badPeer = p; }
    if (needRecv && rseg == FCX_SEG_HEAP && (roff > dc.heapBytes || recvSpan > dc.heapBytes - roff)) { bad = true; badPeer = p; }
    symS = symS && sseg == FCX_SEG_HEAP && soff == a.sendHeapOff;
    symR = symR && rseg == FCX_SEG_HEAP && roff == a.recvHeapOff;
  }
  if (bad) {
    if (t == 0) giveUp(dc, FCX_ERR_BADARG, badPeer, FCX_WAIT_BARRIER, cta, 0, 0, seq);
    return false;
  }
  const bool mc = dc.mcHeap != nullptr && a.useMc;
  z->mcSend = (mc && symS && needSend && (a.sendHeapOff & 15u) == 0) ? dc.mcHeap + a.sendHeapOff : nullptr;
  z->mcRecv = (mc && symR && needRecv && (a.recvHeapOff & 15u) == 0) ? dc.mcHeap + a.recvHeapOff : nullptr;
  return true;
}

// multimem accesses are weak with respect to the generic proxy's ordinary loads and stores of the same
// addresses only through fences; a system-scope fence by every thread before the closing barrier makes the
// multicast stores visible to whatever the peers run next.
__device__ __forceinline__ void zcFenceBeforeClose() { __threadfence_system(); }

// ---------------------------------------------------------------- reducing kinds

// `cnt` 32-byte pieces from `first` on for exactly P ranks, everything 32-byte aligned, or (not WIDE) 16-byte aligned and
// each piece in two accesses.  A thread has eight loads of 32 bytes (pieces x ranks) in flight.  A GPU that stands in for all ranks at 25 MB (the loop alone, 16 CTAs per rank): 8 ranks 84 us with
// two alternating batches of eight 16-byte loads, 72 with one of eight 32-byte loads; 4 ranks 54 and 42.  Not 32-byte aligned, the
// whole all-reduce of 8 ranks: 112 us so, 126 in one batch of eight 16-byte loads, 92 in pieces of two.
template <typename TIn, int U, int P, bool WIDE>
__device__ __forceinline__ void zcReduceWide(const FcxCollArgs &a, const char *const *src, char *const *dst, int nd, size_t first, size_t cnt,
                                             size_t gtid, size_t gstride) {
  using Acc = typename Elem<TIn>::Acc;
  constexpr int G = 32 / (int)sizeof(TIn);
  const char *s[P];
#pragma unroll
  for (int p = 0; p < P; p++) s[p] = src[p];
  const size_t end = first + cnt;
  for (size_t u = first + gtid; u < end; u += U * gstride) {
    Vec32 raw[U][P];
#pragma unroll
    for (int i = 0; i < U; i++)
      if (u + i * gstride < end) {
#pragma unroll
        for (int p = 0; p < P; p++) {
          const char *at = s[p] + (u + i * gstride) * 32;
          if constexpr (WIDE) {
            raw[i][p] = ld32(at);
          } else {
            union { uint4 q[2]; Vec32 v; } w;
            w.q[0] = ld16(at);
            w.q[1] = ld16(at + 16);
            raw[i][p] = w.v;
          }
        }
      }
#pragma unroll
    for (int i = 0; i < U; i++)
      if (u + i * gstride < end) {
        Acc acc[G];
#pragma unroll
        for (int p = 0; p < P; p++) {
          union { Vec32 v; TIn t[G]; } w;
          w.v = raw[i][p];
#pragma unroll
          for (int e = 0; e < G; e++) {
            const Acc x = Elem<TIn>::up(w.t[e]);
            acc[e] = p == 0 ? x : applyOp<Acc>(acc[e], x, a.redop);
          }
        }
#pragma unroll
        for (int e = 0; e < G; e++) acc[e] = finish<Acc>(acc[e], a.redop, P, a.scale);
        union { uint4 q[2]; Vec32 v; } packed;
        packUnit<TIn, G>(acc, packed.q);
        for (int k = 0; k < nd; k++) {
          char *at = dst[k] + (u + i * gstride) * 32;
          if constexpr (WIDE) {
            st32(at, packed.v);
          } else {
            st16(at, packed.q[0]);
            st16(at + 16, packed.q[1]);
          }
        }
      }
  }
}

// Units [first, first + cnt) of 16 bytes for exactly P ranks whose buffers all start `m` bytes past a 16-byte boundary, into
// 16-byte aligned destinations.  A thread has U x P (eight) loads in flight.  With m > 0 a unit lies in two blocks of the source, the
// second of which the next lane has loaded: a warp takes 31 units and its last lane loads a block only (were it to load the 32nd unit's
// second block itself, that load would be waited for in the middle of the sums).  The block behind the last unit's must exist.
// Reduce-scatter, element by element (as all buffers that were not 16-byte aligned once were) / with that load in the middle / so, us:
// 4 x 1500001 fp32 on 16 CTAs 144 / 81 / 71, 4 x 113463 on 3 38 / 44 / 33, 8 x 158030 on 4 70 / 76 / 52, 8 x 200003 bf16 on 16 40 / 36 / 33.
template <typename TIn, int U, int P>
__device__ __forceinline__ void zcReduceShifted(const FcxCollArgs &a, const char *const *src, char *const *dst, int nd, size_t first, size_t cnt, int m,
                                                size_t gtid, size_t gstride) {
  using Acc = typename Elem<TIn>::Acc;
  constexpr int G = 16 / (int)sizeof(TIn);
  const size_t end = first + cnt, blocks = end + (m ? 1 : 0);
  const int lane = threadIdx.x & 31, lanes = m ? 31 : 32;
  const size_t mine = gtid / 32 * lanes + lane, stride = gstride / 32 * lanes;
  for (size_t u0 = first + mine; u0 - lane < end; u0 += U * stride) {  // a whole warp goes round together
    uint4 raw[U][P];
#pragma unroll
    for (int i = 0; i < U; i++)
      if (u0 + i * stride < blocks) {
#pragma unroll
        for (int p = 0; p < P; p++) raw[i][p] = ld16(src[p] - m + (u0 + i * stride) * 16);
      }
#pragma unroll
    for (int i = 0; i < U; i++) {
      const size_t u = u0 + i * stride;
      Acc acc[G];
#pragma unroll
      for (int p = 0; p < P; p++) {
        union { uint4 v; TIn t[G]; } w;
        w.v = raw[i][p];
        if (m) {
          uint4 hi;
          hi.x = __shfl_down_sync(0xffffffffu, w.v.x, 1);
          hi.y = __shfl_down_sync(0xffffffffu, w.v.y, 1);
          hi.z = __shfl_down_sync(0xffffffffu, w.v.z, 1);
          hi.w = __shfl_down_sync(0xffffffffu, w.v.w, 1);
          w.v = shiftBlocks(w.v, hi, m);
        }
#pragma unroll
        for (int e = 0; e < G; e++) {
          const Acc x = Elem<TIn>::up(w.t[e]);
          acc[e] = p == 0 ? x : applyOp<Acc>(acc[e], x, a.redop);
        }
      }
      if (lane < lanes && u < end) {
#pragma unroll
        for (int e = 0; e < G; e++) acc[e] = finish<Acc>(acc[e], a.redop, P, a.scale);
        uint4 packed;
        packUnit<TIn, G>(acc, &packed);
        for (int k = 0; k < nd; k++) st16(dst[k] + u * 16, packed);
      }
    }
  }
}

// out = finish(x_0 (op) x_1 ... (op) x_{n-1}) for `nElems` elements that start `srcOff` elements into every
// rank's send buffer.  The result goes `dstOff` elements into: this rank's recv buffer (toSelf), every other
// rank's recv buffer (toPeers), or both.  Ranks are combined in rank order, so the owner's result is the one
// every rank receives, bit for bit.
template <typename TIn, typename TOut>
__device__ __forceinline__ void zcReduceRange(const FcxDevComm &dc, const FcxCollArgs &a, const ZcPeers &z, size_t srcOff,
                                              size_t dstOff, size_t nElems, bool toSelf, bool toPeers, size_t gtid,
                                              size_t gstride) {
  using AI = typename Elem<TIn>::Acc;
  using AO = typename Elem<TOut>::Acc;
  constexpr int ESI = (int)sizeof(TIn), ESO = (int)sizeof(TOut);
  constexpr int G = 16 / (ESI < ESO ? ESI : ESO);
  constexpr int INB = G * ESI, OUTB = G * ESO;
  const int n = dc.nranks, me = dc.rank;
  if (!nElems) return;
  const char *src[FCX_MAX_RANKS];
  char *dst[FCX_MAX_RANKS];
  int nd = 0;
  uintptr_t orS = 0, apart = 0, orD = 0;  // low bits: how the buffers are aligned, and whether all sources alike
  for (int p = 0; p < n; p++) {
    src[p] = z.send[p] + srcOff * ESI;
    orS |= (uintptr_t)src[p];
    apart |= (uintptr_t)src[p] ^ (uintptr_t)src[0];
  }
  for (int k = 0; k < n; k++) {
    int p = (me + k) % n;  // own buffer first, then the peers starting with the right-hand neighbour
    if ((p == me && toSelf) || (p != me && toPeers)) {
      dst[nd] = z.recv[p] + dstOff * ESO;
      orD |= (uintptr_t)dst[nd];
      nd++;
    }
  }
  const bool alS = (orS & 15u) == 0, alD = (orD & 15u) == 0;
  const size_t nunits = (nElems + G - 1) / G;
  size_t firstPlain = 0;  // units below this index are done through the switch
  size_t edgeUnit = ~(size_t)0;  // but this one is not done yet

  if constexpr (ESI == ESO && Mm<TIn>::ok) {
    if (z.mcSend != nullptr && alS && alD && Mm<TIn>::opOk(a.redop)) {
      const char *mcs = z.mcSend + srcOff * ESI;
      char *mcd = (toSelf && toPeers && z.mcRecv != nullptr) ? z.mcRecv + dstOff * ESO : nullptr;
      const size_t nfull = nElems / G;
      constexpr int U = 8;
      size_t u = gtid;
      for (; u + (U - 1) * gstride < nfull; u += U * gstride) {
        uint4 r[U];
#pragma unroll
        for (int i = 0; i < U; i++) r[i] = Mm<TIn>::ldReduce(mcs + (u + i * gstride) * 16, a.redop);
#pragma unroll
        for (int i = 0; i < U; i++) {
          const uint4 f = mmFinish<TIn>(r[i], a.redop, n, a.scale);
          const size_t o = (u + i * gstride) * 16;
          if (mcd) mmStore(mcd + o, f);
          else
            for (int k = 0; k < nd; k++) st16(dst[k] + o, f);
        }
      }
      for (; u < nfull; u += gstride) {
        const uint4 f = mmFinish<TIn>(Mm<TIn>::ldReduce(mcs + u * 16, a.redop), a.redop, n, a.scale);
        if (mcd) mmStore(mcd + u * 16, f);
        else
          for (int k = 0; k < nd; k++) st16(dst[k] + u * 16, f);
      }
      firstPlain = nfull;  // at most one ragged unit is left for the plain path
    }
  }

  // Plain loads from peers are latency-bound (a load over NVLink takes microseconds): the bulk of the range keeps eight
  // loads per thread in flight (units x ranks), of 32 bytes where every buffer allows them.
  if constexpr (ESI == ESO && Mm<TIn>::ok) {  // the floating-point types of gradients and activations
    const int m = (int)((uintptr_t)src[0] & 15u);
    const size_t nfull = nElems / G;
    const bool ranks = n == 2 || n == 4 || n == 8;
    // 32-byte pieces once every thread has one: below, more threads with half of the work each are sooner done (8 ranks x 20000
    // bf16 25.4 us in units of 16 bytes, 26.6 in pieces of 32)
    if (ranks && alS && alD && firstPlain == 0 && nfull / 2 >= gstride) {
      const size_t cnt = nfull / 2;
      const bool wide = ((orS | orD) & 31u) == 0;
      if (n == 2) wide ? zcReduceWide<TIn, 4, 2, true>(a, src, dst, nd, 0, cnt, gtid, gstride) : zcReduceWide<TIn, 4, 2, false>(a, src, dst, nd, 0, cnt, gtid, gstride);
      else if (n == 4) wide ? zcReduceWide<TIn, 2, 4, true>(a, src, dst, nd, 0, cnt, gtid, gstride) : zcReduceWide<TIn, 2, 4, false>(a, src, dst, nd, 0, cnt, gtid, gstride);
      else wide ? zcReduceWide<TIn, 1, 8, true>(a, src, dst, nd, 0, cnt, gtid, gstride) : zcReduceWide<TIn, 1, 8, false>(a, src, dst, nd, 0, cnt, gtid, gstride);
      firstPlain = 2 * cnt;  // at most one whole and one ragged unit are left for the path below
    } else if (ranks && alD && (apart & 15u) == 0 && nfull > firstPlain && (m == 0 || nfull >= 3 * gstride)) {
      // With m > 0 the block before the first unit's bytes and the one behind the last unit's belong to the buffer's edges:
      // those units are left to the path below, which is the better one for all of them while a thread has less than three
      // (reduce of 27752 fp16 on 2 ranks, 2.3 units each, 15.7 us there, 16.7 here; reduce-scatter of 200003 bf16 on 8, 3.1 each, 40.4
      // and 32.5).
      const size_t lo = firstPlain, cnt = nfull - lo - (m ? 2 : 0);
      const size_t from = lo + (m ? 1 : 0);
      if (n == 2) zcReduceShifted<TIn, 4, 2>(a, src, dst, nd, from, cnt, m, gtid, gstride);
      else if (n == 4) zcReduceShifted<TIn, 2, 4>(a, src, dst, nd, from, cnt, m, gtid, gstride);
      else zcReduceShifted<TIn, 1, 8>(a, src, dst, nd, from, cnt, m, gtid, gstride);
      firstPlain = lo + cnt + (m ? 1 : 0);
      edgeUnit = m ? lo : ~(size_t)0;
    }
  }

  auto gather = [&](size_t u, AI *acc) {
    const int nv = (int)min((size_t)G, nElems - u * G);
    for (int p = 0; p < n; p++) {
      AI in[G];
      loadUnit<TIn, G>(src[p] + u * INB, alS, nv, in);
      if (p == 0) {
#pragma unroll
        for (int i = 0; i < G; i++) acc[i] = in[i];
      } else {
#pragma unroll
        for (int i = 0; i < G; i++) acc[i] = applyOp<AI>(acc[i], in[i], a.redop);
      }
    }
  };
  auto emit = [&](size_t u, const AI *acc) {
    const int nv = (int)min((size_t)G, nElems - u * G);
    AO res[G];
#pragma unroll
    for (int i = 0; i < G; i++) res[i] = accCast<AO, AI>(finish<AI>(acc[i], a.redop, n, a.scale));
    uint4 packed[OUTB / 16];
    packUnit<TOut, G>(res, packed);
    for (int k = 0; k < nd; k++) storeUnit<TOut, G>(dst[k] + u * OUTB, alD, nv, packed);
  };
  // the threads that had least of the bulk take what is left of it
  const size_t rest = firstPlain ? gstride - 1 - gtid : gtid;
  size_t u = firstPlain + rest;
  for (; u + gstride < nunits; u += 2 * gstride) {
    AI acc0[G], acc1[G];
    gather(u, acc0);
    gather(u + gstride, acc1);
    emit(u, acc0);
    emit(u + gstride, acc1);
  }
  bool edge = edgeUnit != ~(size_t)0 && rest == 3;  // up to three units lie behind the bulk
  while (u < nunits || edge) {
    const size_t v = u < nunits ? u : edgeUnit;
    edge = edge && u < nunits;
    u += gstride;
    AI acc[G];
    gather(v, acc);
    emit(v, acc);
  }
}

template <typename TIn, typename TOut>
__device__ void fcxZcReduceBody(const FcxDevComm &dc, const FcxCollArgs &a, int cta, int nctas) {
  constexpr int ESI = (int)sizeof(TIn), ESO = (int)sizeof(TOut);
  constexpr int G = 16 / (ESI < ESO ? ESI : ESO);
  const int n = dc.nranks, me = dc.rank;
  uint64_t seq;
  const size_t gtid = (size_t)cta * blockDim.x + threadIdx.x, gstride = (size_t)nctas * blockDim.x;
  if (!prologue(dc, cta, &seq)) return;
  ZcPeers z;
  const bool isAR = a.kind == FCX_K_AR_ZC, isRS = a.kind == FCX_K_RS_ZC;
  const size_t sendSpan = (isRS ? (size_t)(n - 1) * a.sendStride + a.count : a.count) * ESI;
  if (zcExchange(dc, a, seq, cta, true, isAR, sendSpan, a.count * ESO, nullptr, nullptr, &z)) {
    if (isAR) {
      // slices in pairs of units so that every slice starts as aligned as the buffer itself, up to 32 bytes
      const size_t totalUnits = (a.count + G - 1) / G, sliceUnits = ((totalUnits + n - 1) / n + 1) & ~(size_t)1;
      const size_t lo = min(a.count, (size_t)me * sliceUnits * G), hi = min(a.count, ((size_t)me + 1) * sliceUnits * G);
      zcReduceRange<TIn, TOut>(dc, a, z, lo, lo, hi - lo, true, true, gtid, gstride);
    } else if (isRS) {
      zcReduceRange<TIn, TOut>(dc, a, z, (size_t)me * a.sendStride, 0, a.count, true, false, gtid, gstride);
    } else if (me == a.root) {
      zcReduceRange<TIn, TOut>(dc, a, z, 0, 0, a.count, true, false, gtid, gstride);
    }
    if (z.mcSend || z.mcRecv) zcFenceBeforeClose();  // else the release of the closing barrier orders the CTA's stores
    ctaBarrier(dc, cta, barrierValue(seq, 2), seq);
  }
  epilogue(dc, seq, nctas);
}

// ---------------------------------------------------------------- byte-moving kinds

// One read of `src`, one store into each of dst[0..nd), so that local memory is read once whatever the number of peers.
// 32-byte aligned buffers move in four 32-byte accesses per thread and turn, others in four of 16 bytes at the destinations'
// alignment, for which a source that starts elsewhere in its 16-byte blocks is shifted out of two of them (the next lane has
// loaded the second).  Destinations of different alignments take a pass each.  Pieces of an odd number of bytes per rank, as
// an all-gather of any count has them, went byte by byte before: 8 ranks x 200003 bf16 120 us, 29 now; 4 x 1500001 284 and 35.
__device__ __forceinline__ void zcCopyShifted(char *const *dst, int nd, const char *src, size_t bytes, size_t gtid, size_t gstride) {
  constexpr int U = 4;
  const size_t head = min(bytes, (size_t)((16u - ((uintptr_t)dst[0] & 15u)) & 15u));  // bytes before the destinations' first block
  const char *s = src + head, *blocks = (const char *)((uintptr_t)s & ~(uintptr_t)15);
  const int m = (int)(s - blocks);
  // destination blocks [i0, i1) whose bytes lie in whole blocks of the source
  size_t i0 = 0, i1 = (bytes - head) / 16;
  if (m) {
    if (blocks < src) i0 = 1;
    const size_t have = (size_t)(src + bytes - blocks) / 16;  // whole blocks from `blocks` on
    i1 = min(i1, have ? have - 1 : (size_t)0);
    i0 = min(i0, i1);
  }
  const int lane = threadIdx.x & 31;
  for (size_t u = i0 + gtid; u - lane < i1; u += U * gstride) {  // a whole warp goes round together
    uint4 v[U];
#pragma unroll
    for (int i = 0; i < U; i++)
      if (u + i * gstride < i1 + (m ? 1 : 0)) v[i] = ld16(blocks + (u + i * gstride) * 16);
    if (m) {
#pragma unroll
      for (int i = 0; i < U; i++) {
        uint4 hi;
        hi.x = __shfl_down_sync(0xffffffffu, v[i].x, 1);
        hi.y = __shfl_down_sync(0xffffffffu, v[i].y, 1);
        hi.z = __shfl_down_sync(0xffffffffu, v[i].z, 1);
        hi.w = __shfl_down_sync(0xffffffffu, v[i].w, 1);
        if (lane == 31 && u + i * gstride < i1) hi = ld16(blocks + (u + i * gstride + 1) * 16);
        v[i] = shiftBlocks(v[i], hi, m);
      }
    }
    for (int k = 0; k < nd; k++) {
#pragma unroll
      for (int i = 0; i < U; i++)
        if (u + i * gstride < i1) st16(dst[k] + head + (u + i * gstride) * 16, v[i]);
    }
  }
  // the edges, byte by byte: at most 31 + 47 of them
  const size_t before = head + i0 * 16, after = head + i1 * 16;
  for (size_t j = gtid; j < before + (bytes - after); j += gstride) {
    const size_t at = j < before ? j : after + (j - before);
    const char c = src[at];
    for (int k = 0; k < nd; k++) dst[k][at] = c;
  }
}

__device__ __forceinline__ void zcCopyMulti(char *const *dst, int nd, const char *src, size_t bytes, size_t gtid, size_t gstride) {
  if (!bytes || !nd) return;
  bool wide = aligned32(src), alike = true;
  for (int k = 0; k < nd; k++) {
    wide = wide && aligned32(dst[k]);
    alike = alike && (((uintptr_t)dst[k] ^ (uintptr_t)dst[0]) & 15u) == 0;
  }
  if (wide) {
    constexpr int U = 4;
    const size_t nfull = bytes / 32;
    for (size_t u = gtid; u < nfull; u += U * gstride) {
      Vec32 v[U];
#pragma unroll
      for (int i = 0; i < U; i++)
        if (u + i * gstride < nfull) v[i] = ld32(src + (u + i * gstride) * 32);
      for (int k = 0; k < nd; k++) {
#pragma unroll
        for (int i = 0; i < U; i++)
          if (u + i * gstride < nfull) st32(dst[k] + (u + i * gstride) * 32, v[i]);
      }
    }
    for (size_t j = nfull * 32 + gtid; j < bytes; j += gstride) {
      const char c = src[j];
      for (int k = 0; k < nd; k++) dst[k][j] = c;
    }
    return;
  }
  const int together = alike ? nd : 1;
  for (int k = 0; k < nd; k += together) zcCopyShifted(dst + k, together, src, bytes, gtid, gstride);
}

// Store the 16-byte units of `src` through the multicast alias (every rank of the communicator receives
// them, this one included).  Returns the number of bytes covered; the ragged rest is left to plain stores.
__device__ __forceinline__ size_t zcMcPush(char *mcDst, const char *src, size_t bytes, size_t gtid, size_t gstride) {
  if (!aligned16(src) || !aligned16(mcDst)) return 0;
  const size_t nfull = bytes / 16;
  size_t u = gtid;
  for (; u + 3 * gstride < nfull; u += 4 * gstride) {
    uint4 v[4];
#pragma unroll
    for (int i = 0; i < 4; i++) v[i] = ld16(src + (u + i * gstride) * 16);
#pragma unroll
    for (int i = 0; i < 4; i++) mmStore(mcDst + (u + i * gstride) * 16, v[i]);
  }
  for (; u < nfull; u += gstride) mmStore(mcDst + u * 16, ld16(src + u * 16));
  return nfull * 16;
}

// One piece per rank: piece k is copied by `copy(k, gtid, gstride)`.  Where the CTAs divide by the ranks every rank's piece has CTAs of
// its own, so that short pieces are not one trip to memory after the other (8 ranks x 200000 bf16 41.3 us, 29.1 so).
template <typename Copy>
__device__ __forceinline__ void zcPieces(int n, int cta, int nctas, Copy copy) {
  if (nctas % n == 0)
    copy(cta % n, (size_t)(cta / n) * blockDim.x + threadIdx.x, (size_t)(nctas / n) * blockDim.x);
  else
    for (int k = 0; k < n; k++) copy(k, (size_t)cta * blockDim.x + threadIdx.x, (size_t)nctas * blockDim.x);
}

__device__ void fcxZcMoveBody(const FcxDevComm &dc, const FcxCollArgs &a, int cta, int nctas) {
  const int n = dc.nranks, me = dc.rank;
  uint64_t seq;
  const size_t gtid = (size_t)cta * blockDim.x + threadIdx.x, gstride = (size_t)nctas * blockDim.x;
  const size_t es = a.elemSize, bytes = a.count * es;
  const int mk = a.moveOp;
  if (!prologue(dc, cta, &seq)) return;
  const bool pull = mk == FCX_K_GATHER || mk == FCX_K_A2AV;
  size_t sendSpan = 0, recvSpan = 0;
  uint64_t xTo[FCX_MAX_RANKS], yTo[FCX_MAX_RANKS];
  for (int p = 0; p < n; p++) { xTo[p] = 0; yTo[p] = 0; }
  switch (mk) {
    case FCX_K_AG:
    case FCX_K_A2A: recvSpan = ((size_t)(n - 1) * a.recvStride + a.count) * es; break;
    case FCX_K_BCAST:
    case FCX_K_SCATTER: recvSpan = bytes; break;
    case FCX_K_GATHER: sendSpan = bytes; break;
    case FCX_K_A2AV:
      for (int p = 0; p < n; p++) {
        xTo[p] = a.sdispls[p] * es;
        yTo[p] = a.scounts[p] * es;
      }
      break;
    default: break;
  }
  ZcPeers z;
  if (a.ceOpen) {
    // Opening step of the copy-engine form: after this barrier every peer's receive buffer may be written;
    // the host's copies assume one heap offset on all ranks, which is checked here (a mismatch is recorded as a
    // bad argument; the copies then land at this rank's offset inside the peers' heaps, never outside them).
    if (zcExchange(dc, a, seq, cta, false, true, 0, recvSpan, nullptr, nullptr, &z)) {
      bool same = true;
      for (int p = 0; p < n; p++) same = same && (p == me || z.recv[p] == dc.heap[p] + a.recvHeapOff);
      if (!same && threadIdx.x == 0) giveUp(dc, FCX_ERR_BADARG, me, FCX_WAIT_BARRIER, cta, a.recvHeapOff, 0, seq);
    }
    epilogue(dc, seq, nctas);
    return;
  }
  if (zcExchange(dc, a, seq, cta, pull, !pull, sendSpan, recvSpan, xTo, yTo, &z)) {
    const char *send = (const char *)a.send;
    char *recv = (char *)a.recv;
    char *dst[FCX_MAX_RANKS];
    int nd = 0;
    switch (mk) {
      case FCX_K_AG: {
        const size_t off = (size_t)me * a.recvStride * es;
        size_t done = 0;
        if (z.mcRecv && (a.useMc & 2)) done = zcMcPush(z.mcRecv + off, send, bytes, gtid, gstride);
        // a multicast store reaches this rank too, so everybody, this rank included, still needs [done, bytes)
        if (recv + off != send) dst[nd++] = recv + off;
        for (int k = 1; k < n; k++) dst[nd++] = z.recv[(me + k) % n] + off;
        if (done < bytes) {
          char *d2[FCX_MAX_RANKS];
          for (int k = 0; k < nd; k++) d2[k] = dst[k] + done;
          zcCopyMulti(d2, nd, send + done, bytes - done, gtid, gstride);
        }
        break;
      }
      case FCX_K_BCAST: {
        if (me != a.root) break;
        size_t done = 0;
        if (z.mcRecv) done = zcMcPush(z.mcRecv, send, bytes, gtid, gstride);
        if (recv != send) dst[nd++] = recv;
        for (int k = 1; k < n; k++) dst[nd++] = z.recv[(me + k) % n];
        if (done < bytes) {
          char *d2[FCX_MAX_RANKS];
          for (int k = 0; k < nd; k++) d2[k] = dst[k] + done;
          zcCopyMulti(d2, nd, send + done, bytes - done, gtid, gstride);
        }
        break;
      }
      case FCX_K_SCATTER: {
        if (me != a.root) break;
        zcPieces(n, cta, nctas, [&](int k, size_t t, size_t stride) {
          const int p = (me + k) % n;
          const char *s = send + (size_t)p * a.sendStride * es;
          char *const d[1] = {p == me ? recv : z.recv[p]};
          if (d[0] != s) zcCopyMulti(d, 1, s, bytes, t, stride);
        });
        break;
      }
      case FCX_K_A2A: {
        zcPieces(n, cta, nctas, [&](int k, size_t t, size_t stride) {
          const int p = (me + k) % n;
          const char *s = send + (size_t)p * a.sendStride * es;
          char *const d[1] = {(p == me ? recv : z.recv[p]) + (size_t)me * a.recvStride * es};
          if (d[0] != s) zcCopyMulti(d, 1, s, bytes, t, stride);
        });
        break;
      }
      case FCX_K_GATHER: {
        if (me != a.root) break;
        zcPieces(n, cta, nctas, [&](int k, size_t t, size_t stride) {
          const int p = (me + k) % n;
          const char *s = p == me ? send : z.send[p];
          char *const d[1] = {recv + (size_t)p * a.recvStride * es};
          if (d[0] != s) zcCopyMulti(d, 1, s, bytes, t, stride);
        });
        break;
      }
      case FCX_K_A2AV: {
        for (int k = 0; k < n; k++) {
          const int p = (me + k) % n;
          const char *s = (p == me ? send : z.send[p]) + z.x[p];
          const size_t nb = min((size_t)z.y[p], (size_t)(a.rcounts[p] * es));
          char *const d[1] = {recv + a.rdispls[p] * es};
          if (nb && d[0] != s) zcCopyMulti(d, 1, s, nb, gtid, gstride);
        }
        break;
      }
      default: break;
    }
    if (z.mcSend || z.mcRecv) zcFenceBeforeClose();  // else the release of the closing barrier orders the CTA's stores
    ctaBarrier(dc, cta, barrierValue(seq, 2), seq);
  }
  epilogue(dc, seq, nctas);
}

}  // namespace fcxdev
