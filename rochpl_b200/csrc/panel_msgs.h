// When the panel leaf's message barriers are waited on, armed and sent to
// (panel_fused.cu), apart from the instructions, so that the rules can be run on the
// host against a model of an mbarrier.
//
// A CTA has kBufs barriers; column kc's messages, one from every CTA, complete a phase
// of barrier kc % kBufs, which one arrival with the phase's byte count arms.  The next
// phase is armed only once this one has completed, and not at all once a wait of the
// CTA has expired: a second arrival in a phase is undefined, and the bytes expected
// would grow without end.  For the same reason such a CTA sends no more: the others'
// barriers then stay where they are until their own waits expire, and theirs are left
// with the few bytes that were on their way.
#pragma once

#ifdef __CUDACC__
#define HPLB_MSG_FN __device__ __forceinline__
#else
#define HPLB_MSG_FN inline
#endif

namespace hplb {

constexpr int kBufs = 4;  // message buffers and barriers, by column

// Ring: wait(buf, parity) until that phase has completed (or the budget is spent),
// expired() once a wait of this CTA has given up, arm(buf).

// Every thread waits for column kc's messages; true if they are all here.
template <class Ring>
HPLB_MSG_FN bool await_column(Ring& r, unsigned kc) {
  return r.wait((int)(kc % kBufs), (kc / kBufs) & 1u);
}
// One thread, after its own await_column and before it waits for column kc + kBufs.
template <class Ring>
HPLB_MSG_FN void rearm(Ring& r, unsigned kc, bool arrived) {
  if(arrived && !r.expired()) r.arm((int)(kc % kBufs));
}
template <class Ring>
HPLB_MSG_FN bool may_send(Ring& r) {
  return !r.expired();
}

}  // namespace hplb
