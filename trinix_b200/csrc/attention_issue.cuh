// Order of work of an issuing warp of attention_plain.cu, without any CUDA, so that a model on the host
// can run it too.
//
// The work is the sequence of one Q tile's visits over all items of the CTA. The Q K^T run one visit
// ahead of the P V, into the next item too:  .. P V(v), Q K(v + 1), P V(v + 1) ..  The K and V tiles of
// visits without this Q tile are only released. Nothing ahead of a pending P V is waited for: the ring may
// be held up by a V tile that this P V frees.
#pragma once

#ifdef __CUDACC__
#define TRX_ISSUE __device__ __forceinline__
#else
#define TRX_ISSUE inline
#endif

namespace trx {

constexpr int AP_STAGES = 4;  // K / V ring
static_assert((AP_STAGES & (AP_STAGES - 1)) == 0, "ring depth must be a power of two");

// Visits [lo, hi) of the n of an item are this Q tile's; v is the next one.
struct PlainCursor {
  int lo, hi, n, item, v;
};

// What the order is made of. `open` reads an item and says whether there is one; `*_there` ask without
// waiting; waits and `pv` return false when the CTA gives up.
template <class Open, class ItemThere, class WaitFill, class FillThere, class FreeFill, class WaitQ,
          class QThere, class Qk, class QDone, class WaitOFree, class Pv, class ODone>
struct PlainSteps {
  Open open;            // (cursor, item, ok) -> bool
  ItemThere item_there; // (item) -> bool
  WaitFill wait_fill;   // (fill) -> bool
  FillThere fill_there; // (fill) -> bool
  FreeFill free_fill;   // (fill)
  WaitQ wait_q;         // (parity) -> bool
  QThere q_there;       // (parity) -> bool
  Qk qk;                // (fill)
  QDone q_done;         // ()
  WaitOFree wait_o_free;  // (parity) -> bool
  Pv pv;                // (fill, accumulate) -> bool
  ODone o_done;         // ()
};
template <class... F>
PlainSteps(F...) -> PlainSteps<F...>;

// All items; false: the CTA gives up.
template <class Steps>
TRX_ISSUE bool plain_issue(Steps& s) {
  bool ok = true;
  unsigned qpar = 0;    // parity of the next Q tile
  bool s_busy = false;  // a Q K^T is issued whose P V is not
  unsigned keyed = 0;   // items with keys whose P V have begun
  int kf = 0, vf = 0;   // ring fill of the next Q K^T and of the next P V
  auto wait_fill = [&](int f) {
    if (ok) ok = s.wait_fill(f);
  };
  auto free_fill = [&](int f) {
    if (ok) s.free_fill(f);
  };
  auto qk = [&]() {
    s_busy = true;
    s.qk(kf);
  };
  auto pv = [&](unsigned acc) {
    ok = s.pv(vf, acc);
    s_busy = false;
  };
  auto step_qk = [&](PlainCursor& c) {
    const int v = c.v;
    wait_fill(kf);
    if (ok && v == c.lo && c.lo < c.hi) {
      ok = s.wait_q(qpar);
      qpar ^= 1u;
    }
    if (ok && v >= c.lo && v < c.hi) qk();
    if (ok && v == c.hi - 1 && c.lo < c.hi) s.q_done();
    free_fill(kf);
    kf += v == 0 && c.n > 1 ? 1 : 2;
    if (v + 1 == c.n) kf += c.n > 1 ? 1 : 0;
    c.v = v + 1;
  };
  auto step_pv = [&](PlainCursor& c) {
    const int v = c.v;
    wait_fill(vf);
    if (ok && v >= c.lo && v < c.hi) {
      // the epilogue is done with the last O (items without keys have none: it does not wait
      // for this warp there, so they must not count)
      if (v == c.lo && keyed++ > 0) ok = s.wait_o_free(keyed & 1);
      if (ok) pv(v == c.lo ? 0u : 1u);
      if (ok && v == c.hi - 1) s.o_done();
    }
    free_fill(vf);
    vf += v + 2 >= c.n ? 1 : 2;
    c.v = v + 1;
  };

  PlainCursor qc, pc, nc;  // of the Q K^T, of the P V, and the next item's
  bool more = s.open(qc, 0, ok);  // there may be another item
  pc = qc;
  vf = qc.n > 1 ? 2 : qc.n;  // V(0) comes behind K(1) of its item, if there is one
  bool known = false;        // nc is the item after pc's
#pragma unroll 1
  while (ok) {
    while (ok) {
      const bool behind = qc.item != pc.item || qc.v > pc.v;  // there is a P V step to take
      if (qc.v == qc.n) {
        if (qc.item > pc.item || !more) break;  // at the end of what it may go to
        const int i = qc.item + 1;
        if (pc.v < pc.n && !s.item_there(i)) break;
        more = s.open(nc, i, ok);
        if (!more) break;
        known = true;
        qc = nc;
        continue;
      }
      if (s_busy) break;
      // `fill_there` compares one bit of a phase count, so it answers for this fill only if the one
      // before it in its stage has been waited for. Behind the P V that need not be so: the next item's
      // K(0) shares a stage with V(n - 3), for which nothing has waited if its visit is not this Q tile's.
      // A fill that is really there was issued after this warp had released the one before it. (As a
      // test of its own 4 x 3001 with a window of 1024 takes 197.0 us, in one condition 193.9.)
      if (behind && (kf - vf >= AP_STAGES || !s.fill_there(kf))) break;
      if (behind && qc.v == qc.lo && !s.q_there(qpar)) break;
      step_qk(qc);
    }
    if (!ok) break;
    if (qc.item == pc.item && qc.v == pc.v + 1 && s_busy && pc.v > pc.lo) {
      const int last = pc.hi - 3;  // of the P V visits
#pragma unroll 1
      while (pc.v <= last) {
        wait_fill(vf);
        wait_fill(kf);
        if (ok) pv(1u);
        free_fill(vf);
        if (ok) qk();
        free_fill(kf);
        if (!ok) break;
        kf += 2;
        vf += 2;
        ++pc.v;
        ++qc.v;
      }
      if (!ok) break;
    }
    if (pc.v == pc.n) {
      // on to the next item, if there is one
      if (!known) break;
      pc = nc;
      known = false;
      vf += pc.n > 1 ? 2 : pc.n;
      continue;
    }
    if (pc.item != qc.item || pc.v < qc.v) step_pv(pc);
  }
  return ok;
}

}  // namespace trx
