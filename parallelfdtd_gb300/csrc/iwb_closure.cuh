// IWB closure nodes (no counterpart in the reference): the inside nodes with
// a closed neighbour, whose update substitutes the node's own value for every
// closed neighbour.  The streaming TMA update leaves them alone and the
// sparse pass k_iwb_closure (dif.cu) updates them with iwb_closure_apply.
#pragma once

#include "common.cuh"

namespace pfdtd {

// One closure node, records in ascending flat-index order.  cls is the
// node's class (an index into the class table).
struct alignas(16) ClosureRec {
  int64_t idx;
  uint32_t mask;
  uint32_t cls;
};

// Per DIF class: a, b, c, g2 and the filter b0..b3, a1..a3 (11 values).
constexpr int kDifClassVals = 11;

// A DIF node's filter states and previous value, read and written as a whole.
template <typename A> struct alignas(16) DifState { A s1, s2, s3, prev; };

// Update of closure node i from its 3 x 3 x 3 neighbourhood m (closed
// neighbours already replaced by the centre's value) and P^{n-1} pp: the
// canonical sums give sw, then either the frequency-independent rule of class c or, for a
// node with a DIF state slot, the DIF update (operation for operation as
// k_dif_update), and the result is stored to Pp[i].  A DIF node without a
// slot stores its sw to iwb_sw for the separate DIF pass.
template <typename S>
__device__ __forceinline__ void iwb_closure_apply(const float (&m)[3][3][3], unsigned c, float pp,
                                                  ClassTab<float> tab, float l2, int32_t slot,
                                                  DifState<float> st, const float* __restrict__ dtab,
                                                  DifState<float>* __restrict__ dstate,
                                                  float* __restrict__ iwb_sw, int64_t i,
                                                  S* __restrict__ Pp) {
  using R = Rn<float>;
  using Sto = Store<S>;
  const float p = m[1][1][1];
  float s1, s2, s3;
  iwb_sums(m, s1, s2, s3);
  const float sw = R::mul(l2, R::add(R::add(R::mul(s1, 0.25f), R::mul(s2, 0.125f)),
                                     R::mul(s3, 0.0625f)));
  if (slot >= 0) {
    const float* t = dtab + (int64_t)kDifClassVals * c;
    const float num = R::sub(R::sub(R::add(sw, R::mul(t[1], p)), R::mul(t[2], st.prev)),
                             R::mul(t[3], st.s1));
    const float out = R::mul(t[0], num);
    const float xx = R::mul(R::sub(out, st.prev), 0.5f);
    const float yy = R::add(R::mul(t[4], xx), st.s1);
    dstate[slot] = DifState<float>{R::add(R::sub(R::mul(t[5], xx), R::mul(t[8], yy)), st.s2),
                                   R::add(R::sub(R::mul(t[6], xx), R::mul(t[9], yy)), st.s3),
                                   R::sub(R::mul(t[7], xx), R::mul(t[10], yy)), p};
    Pp[i] = Sto::store(out);
    return;
  }
  if (iwb_sw != nullptr && (__ldg(tab.pos + c) >> 31)) iwb_sw[i] = sw;
  const float out = R::mul(__ldg(tab.a + c), R::sub(R::add(sw, R::mul(__ldg(tab.b + c), p)),
                                                    R::mul(__ldg(tab.c + c), pp)));
  Pp[i] = Sto::store(out);
}

}  // namespace pfdtd
