// Generated by gen_nl.py fx -- do not edit.  The Galerkin coupling as fixed-point products.
#pragma once
namespace mwf {
template <typename S_, typename LD> __device__ __forceinline__ void nl_fx_p_4(const S_& S, LD&& ld, FxAcc (&A)[4]) {
  { const FxLimbs d = ld(0);
    const FxLimbs e = fx_twice(d);
    fx_mac(A[0], S[0], e);
    fx_mac(A[1], S[1], e);
    fx_mac(A[2], S[2], e);
    fx_mac(A[3], S[3], e);
  }
  { const FxLimbs d = ld(1);
    const FxLimbs e = fx_twice(d);
    fx_mac(A[0], S[1], d);
    fx_mac(A[1], S[0], e);
    fx_msb(A[1], S[2], d);
    fx_msb(A[2], S[1], d);
    fx_mac(A[2], S[3], d);
    fx_mac(A[3], S[2], d);
  }
  { const FxLimbs d = ld(2);
    const FxLimbs e = fx_twice(d);
    fx_mac(A[0], S[2], d);
    fx_msb(A[1], S[1], d);
    fx_mac(A[1], S[3], d);
    fx_mac(A[2], S[0], e);
    fx_mac(A[3], S[1], d);
  }
  { const FxLimbs d = ld(3);
    const FxLimbs e = fx_twice(d);
    fx_mac(A[0], S[3], d);
    fx_mac(A[1], S[2], d);
    fx_mac(A[2], S[1], d);
    fx_mac(A[3], S[0], e);
  }
}
template <typename S_, typename LD> __device__ __forceinline__ void nl_fx_v_4(const S_& S, LD&& ld, FxAcc (&A)[4]) {
  { const FxLimbs d = ld(1);
    const FxLimbs e = fx_twice(d);
    fx_mac(A[1], S[0], e);
    fx_mac(A[1], S[2], d);
    fx_mac(A[2], S[1], d);
    fx_mac(A[2], S[3], d);
    fx_mac(A[3], S[2], d);
  }
  { const FxLimbs d = ld(2);
    const FxLimbs e = fx_twice(d);
    fx_mac(A[1], S[1], d);
    fx_mac(A[1], S[3], d);
    fx_mac(A[2], S[0], e);
    fx_msb(A[3], S[1], d);
  }
  { const FxLimbs d = ld(3);
    const FxLimbs e = fx_twice(d);
    fx_mac(A[1], S[2], d);
    fx_msb(A[2], S[1], d);
    fx_mac(A[3], S[0], e);
  }
}
template <typename S_, typename F_> __device__ __forceinline__ void nl_fx_yp_4(const S_& V, const F_& F, FxAcc (&A)[4]) {
  { const FxLimbs d = fx_times(F[1], 1);
    fx_mac(A[0], V[1], d);
    fx_mac(A[1], V[2], d);
    fx_mac(A[2], V[1], d);
    fx_mac(A[2], V[3], d);
    fx_mac(A[3], V[2], d);
  }
  { const FxLimbs d = fx_times(F[2], 2);
    fx_msb(A[0], V[2], d);
    fx_msb(A[1], V[1], d);
    fx_mac(A[1], V[3], d);
    fx_msb(A[3], V[1], d);
  }
  { const FxLimbs d = fx_times(F[3], 3);
    fx_mac(A[0], V[3], d);
    fx_msb(A[1], V[2], d);
    fx_mac(A[2], V[1], d);
  }
}
template <typename S_> __device__ __forceinline__ void nl_fx_yv_4(const S_& V, FxAcc (&A)[4]) {
  { const FxLimbs d = fx_times(V[1], 1);
    fx_msb(A[1], V[2], d);
    fx_msb(A[2], V[1], d);
    fx_mac(A[2], V[3], d);
    fx_mac(A[3], V[2], d);
  }
  { const FxLimbs d = fx_times(V[2], 2);
    fx_mac(A[1], V[1], d);
    fx_mac(A[1], V[3], d);
    fx_mac(A[3], V[1], d);
  }
  { const FxLimbs d = fx_times(V[3], 3);
    fx_msb(A[1], V[2], d);
    fx_msb(A[2], V[1], d);
  }
}
template <typename S_, typename LD> __device__ __forceinline__ void nl_fx_p_6(const S_& S, LD&& ld, FxAcc (&A)[6]) {
  { const FxLimbs d = ld(0);
    const FxLimbs e = fx_twice(d);
    fx_mac(A[0], S[0], e);
    fx_mac(A[1], S[1], e);
    fx_mac(A[2], S[2], e);
    fx_mac(A[3], S[3], e);
    fx_mac(A[4], S[4], e);
    fx_mac(A[5], S[5], e);
  }
  { const FxLimbs d = ld(1);
    const FxLimbs e = fx_twice(d);
    fx_mac(A[0], S[1], d);
    fx_mac(A[1], S[0], e);
    fx_msb(A[1], S[2], d);
    fx_msb(A[2], S[1], d);
    fx_mac(A[2], S[3], d);
    fx_mac(A[3], S[2], d);
    fx_msb(A[3], S[4], d);
    fx_msb(A[4], S[3], d);
    fx_mac(A[4], S[5], d);
    fx_mac(A[5], S[4], d);
  }
  { const FxLimbs d = ld(2);
    const FxLimbs e = fx_twice(d);
    fx_mac(A[0], S[2], d);
    fx_msb(A[1], S[1], d);
    fx_mac(A[1], S[3], d);
    fx_mac(A[2], S[0], e);
    fx_mac(A[2], S[4], d);
    fx_mac(A[3], S[1], d);
    fx_mac(A[3], S[5], d);
    fx_mac(A[4], S[2], d);
    fx_mac(A[5], S[3], d);
  }
  { const FxLimbs d = ld(3);
    const FxLimbs e = fx_twice(d);
    fx_mac(A[0], S[3], d);
    fx_mac(A[1], S[2], d);
    fx_msb(A[1], S[4], d);
    fx_mac(A[2], S[1], d);
    fx_mac(A[2], S[5], d);
    fx_mac(A[3], S[0], e);
    fx_msb(A[4], S[1], d);
    fx_mac(A[5], S[2], d);
  }
  { const FxLimbs d = ld(4);
    const FxLimbs e = fx_twice(d);
    fx_mac(A[0], S[4], d);
    fx_msb(A[1], S[3], d);
    fx_mac(A[1], S[5], d);
    fx_mac(A[2], S[2], d);
    fx_msb(A[3], S[1], d);
    fx_mac(A[4], S[0], e);
    fx_mac(A[5], S[1], d);
  }
  { const FxLimbs d = ld(5);
    const FxLimbs e = fx_twice(d);
    fx_mac(A[0], S[5], d);
    fx_mac(A[1], S[4], d);
    fx_mac(A[2], S[3], d);
    fx_mac(A[3], S[2], d);
    fx_mac(A[4], S[1], d);
    fx_mac(A[5], S[0], e);
  }
}
template <typename S_, typename LD> __device__ __forceinline__ void nl_fx_v_6(const S_& S, LD&& ld, FxAcc (&A)[6]) {
  { const FxLimbs d = ld(1);
    const FxLimbs e = fx_twice(d);
    fx_mac(A[1], S[0], e);
    fx_mac(A[1], S[2], d);
    fx_mac(A[2], S[1], d);
    fx_mac(A[2], S[3], d);
    fx_mac(A[3], S[2], d);
    fx_mac(A[3], S[4], d);
    fx_mac(A[4], S[3], d);
    fx_mac(A[4], S[5], d);
    fx_mac(A[5], S[4], d);
  }
  { const FxLimbs d = ld(2);
    const FxLimbs e = fx_twice(d);
    fx_mac(A[1], S[1], d);
    fx_mac(A[1], S[3], d);
    fx_mac(A[2], S[0], e);
    fx_msb(A[2], S[4], d);
    fx_msb(A[3], S[1], d);
    fx_mac(A[3], S[5], d);
    fx_mac(A[4], S[2], d);
    fx_msb(A[5], S[3], d);
  }
  { const FxLimbs d = ld(3);
    const FxLimbs e = fx_twice(d);
    fx_mac(A[1], S[2], d);
    fx_mac(A[1], S[4], d);
    fx_msb(A[2], S[1], d);
    fx_mac(A[2], S[5], d);
    fx_mac(A[3], S[0], e);
    fx_mac(A[4], S[1], d);
    fx_mac(A[5], S[2], d);
  }
  { const FxLimbs d = ld(4);
    const FxLimbs e = fx_twice(d);
    fx_mac(A[1], S[3], d);
    fx_mac(A[1], S[5], d);
    fx_mac(A[2], S[2], d);
    fx_mac(A[3], S[1], d);
    fx_mac(A[4], S[0], e);
    fx_msb(A[5], S[1], d);
  }
  { const FxLimbs d = ld(5);
    const FxLimbs e = fx_twice(d);
    fx_mac(A[1], S[4], d);
    fx_msb(A[2], S[3], d);
    fx_mac(A[3], S[2], d);
    fx_msb(A[4], S[1], d);
    fx_mac(A[5], S[0], e);
  }
}
template <typename S_, typename F_> __device__ __forceinline__ void nl_fx_yp_6(const S_& V, const F_& F, FxAcc (&A)[6]) {
  { const FxLimbs d = fx_times(F[1], 1);
    fx_mac(A[0], V[1], d);
    fx_mac(A[1], V[2], d);
    fx_mac(A[2], V[1], d);
    fx_mac(A[2], V[3], d);
    fx_mac(A[3], V[2], d);
    fx_mac(A[3], V[4], d);
    fx_mac(A[4], V[3], d);
    fx_mac(A[4], V[5], d);
    fx_mac(A[5], V[4], d);
  }
  { const FxLimbs d = fx_times(F[2], 2);
    fx_msb(A[0], V[2], d);
    fx_msb(A[1], V[1], d);
    fx_mac(A[1], V[3], d);
    fx_msb(A[2], V[4], d);
    fx_msb(A[3], V[1], d);
    fx_mac(A[3], V[5], d);
    fx_mac(A[4], V[2], d);
    fx_msb(A[5], V[3], d);
  }
  { const FxLimbs d = fx_times(F[3], 3);
    fx_mac(A[0], V[3], d);
    fx_msb(A[1], V[2], d);
    fx_mac(A[1], V[4], d);
    fx_mac(A[2], V[1], d);
    fx_mac(A[2], V[5], d);
    fx_mac(A[4], V[1], d);
    fx_mac(A[5], V[2], d);
  }
  { const FxLimbs d = fx_times(F[4], 4);
    fx_msb(A[0], V[4], d);
    fx_msb(A[1], V[3], d);
    fx_mac(A[1], V[5], d);
    fx_msb(A[2], V[2], d);
    fx_msb(A[3], V[1], d);
    fx_msb(A[5], V[1], d);
  }
  { const FxLimbs d = fx_times(F[5], 5);
    fx_mac(A[0], V[5], d);
    fx_msb(A[1], V[4], d);
    fx_mac(A[2], V[3], d);
    fx_msb(A[3], V[2], d);
    fx_mac(A[4], V[1], d);
  }
}
template <typename S_> __device__ __forceinline__ void nl_fx_yv_6(const S_& V, FxAcc (&A)[6]) {
  { const FxLimbs d = fx_times(V[1], 1);
    fx_msb(A[1], V[2], d);
    fx_msb(A[2], V[1], d);
    fx_mac(A[2], V[3], d);
    fx_mac(A[3], V[2], d);
    fx_msb(A[3], V[4], d);
    fx_msb(A[4], V[3], d);
    fx_mac(A[4], V[5], d);
    fx_mac(A[5], V[4], d);
  }
  { const FxLimbs d = fx_times(V[2], 2);
    fx_mac(A[1], V[1], d);
    fx_mac(A[1], V[3], d);
    fx_mac(A[2], V[4], d);
    fx_mac(A[3], V[1], d);
    fx_mac(A[3], V[5], d);
    fx_mac(A[4], V[2], d);
    fx_mac(A[5], V[3], d);
  }
  { const FxLimbs d = fx_times(V[3], 3);
    fx_msb(A[1], V[2], d);
    fx_msb(A[1], V[4], d);
    fx_msb(A[2], V[1], d);
    fx_mac(A[2], V[5], d);
    fx_msb(A[4], V[1], d);
    fx_mac(A[5], V[2], d);
  }
  { const FxLimbs d = fx_times(V[4], 4);
    fx_mac(A[1], V[3], d);
    fx_mac(A[1], V[5], d);
    fx_msb(A[2], V[2], d);
    fx_mac(A[3], V[1], d);
    fx_mac(A[5], V[1], d);
  }
  { const FxLimbs d = fx_times(V[5], 5);
    fx_msb(A[1], V[4], d);
    fx_msb(A[2], V[3], d);
    fx_msb(A[3], V[2], d);
    fx_msb(A[4], V[1], d);
  }
}
}  // namespace mwf
