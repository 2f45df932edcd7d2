// The order in which a GEMM launch works through its tiles; plain C++, so that the host can check it.
#pragma once

#ifdef __CUDACC__
#define FCX_HD __host__ __device__ __forceinline__
#else
#define FCX_HD inline
#endif

// The units (tile x K piece) that one worker (a CTA or a CTA pair) of n works on, in order.  One product: every n-th unit.
// Two products in one launch (`n1` > 0), the one with the longer units first: the workers that get one long unit fewer than
// the others make up for it with `extra` short ones, and the rest of the short units goes round as usual.
struct UnitIter {
  int me, n, n0, n1, extra;
  int i, longs, rem;
  FCX_HD UnitIter(int me_, int n_, int n0_, int n1_, int extraArg) : me(me_), n(n_), n0(n0_), n1(n1_), i(0) {
    rem = n0 % n;
    longs = n0 / n + (me < rem ? 1 : 0);
    extra = rem ? extraArg : 0;
  }
  FCX_HD bool next(int *prob, int *unit) {
    const int k = i++;
    if (k < longs) {
      *prob = 0;
      *unit = me + k * n;
      return true;
    }
    *prob = 1;
    int j = k - longs;
    if (me >= rem) {
      if (j < extra) {
        *unit = j * (n - rem) + me - rem;
        return *unit < n1;
      }
      j -= extra;
    }
    *unit = extra * (n - rem) + j * n + me;
    return *unit < n1;
  }
};
