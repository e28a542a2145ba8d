// Order of memory operations in a slot exchange of the 2D PCG (ipc2d.cu): every CTA posts a value to its slot
// and polls the slots of all CTAs until they hold this exchange's values.  Posts, polls and clears are relaxed
// accesses; two kinds of exchange alternate:
//   FENCE (even epochs)   fence, post, poll, fence: what a CTA stored before is visible to all CTAs after it
//   else  (odd epochs)    post, poll, clear: an exchange of values alone, without a fence
// A slot is empty when its epoch begins because it rotates over SLOT_BUFFERS = 4 buffers and is cleared thus:
// a CTA that has polled the odd epoch e to its end knows that every CTA is past e - 1 (a post depends on the sums
// before it), so it clears its slots of e - 1 and e - 2, whose buffers e + 3 and e + 2 use next.  The fence before
// its post of e + 1 orders the clears before that post, and the fence after the poll of e + 1 orders the other CTAs'
// polls of e + 2 and later behind it: none of them can still read the value of e - 2 as that of e + 2.
// (With the clear between the even epoch's last fence and the odd epoch's post, in three buffers, that was
// possible: two relaxed stores to different slots.)  tests/test_slot_order_host.py runs this order under the
// memory model's views.
#pragma once

#if defined(__CUDACC__)
#define FIPC_SLOT_FN __device__ __forceinline__
#else
#define FIPC_SLOT_FN inline
#endif

namespace fipc {

constexpr int SLOT_BUFFERS = 4;

// Slots: fence(), post(buffer), poll(buffer) -> all arrived, clear(buffer), by one warp of the CTA; the same lane
// polls the same slots in every exchange
template <bool FENCE, class Slots>
FIPC_SLOT_FN bool slot_exchange(Slots& s, int epoch) {
    if (FENCE) s.fence();
    s.post(epoch & (SLOT_BUFFERS - 1));
    const bool all = s.poll(epoch & (SLOT_BUFFERS - 1));
    if (FENCE) {
        s.fence();
    } else {
        s.clear((epoch - 1) & (SLOT_BUFFERS - 1));
        s.clear((epoch - 2) & (SLOT_BUFFERS - 1));
    }
    return all;
}

}  // namespace fipc
