// MPDATA step in a few launches under any boundary condition (declarations;
// kernels in stages_impl.cuh, instantiated per real type in stages_f32.cu and
// stages_f64.cu).
#pragma once

#include "state.cuh"

namespace mpdx {

constexpr int kStageEqns = 4;  // equations advanced by one launch

template <class T>
struct stage_engine {
  // work arrays of the equations after the first, where one launch takes several
  // (the first uses the state's own)
  struct work {
    field<T> tmp0[3], tmp1[3], beta_up, beta_dn, psi_min, psi_max;
  };
  std::vector<work> more;
  bool more_ready = false, one_by_one = false;  // `more` is allocated; it could not be

  // whether step() covers the configuration
  static bool covers(const mpdata_state<T> &st);
  // advances every equation by one step; `upwind_only`: the first pass alone
  void step(mpdata_state<T> &st, bool upwind_only);
  // equations that one launch takes
  int together(mpdata_state<T> &st);
  // one-dimensional problems with both ends open, or cyclic with consistent seams:
  // nt steps, several per launch (advances st.timestep)
  static bool line_covers(const mpdata_state<T> &st);
  void line(mpdata_state<T> &st, long long nt);
};

extern template struct stage_engine<float>;
extern template struct stage_engine<double>;

}  // namespace mpdx
