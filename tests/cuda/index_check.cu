// Host check of the bounds-checked build's index arithmetic (mpdx::index_of): every slot
// of fields laid out as field<T>::alloc lays them out, padding included, against the
// indices that the slot was made from.  Prints the number of slots looked at.
#define MPDX_BOUNDS_CHECK
#include "../../libmpdataxx_b200/csrc/mpdx_common.cuh"

#include <cstdio>
#include <cstdlib>

template <class T>
static long long look(int nd, const int *lo, const int *hi) {
  const int align = int(128 / sizeof(T)), last = nd - 1;
  const int front = (-lo[last] + align - 1) / align * align;
  const long long pitch = (front + hi[last] + 1 + align - 1) / align * align;
  mpdx::dfield<T> f;
  long long s[3] = {0, 0, 0}, acc = pitch;
  s[last] = 1;
  for (int q = last - 1; q >= 0; --q) { s[q] = acc; acc *= hi[q] - lo[q] + 1; }
  f.s0 = s[0]; f.s1 = s[1]; f.s2 = s[2];
  for (int q = 0; q < 3; ++q) {
    f.lo[q] = q < nd ? lo[q] : -2147483647;
    f.hi[q] = q < nd ? hi[q] : 2147483647;
  }
  long long seen = 0;
  int c[3] = {0, 0, 0};
  for (c[0] = nd > 1 ? lo[0] - 1 : 0; c[0] <= (nd > 1 ? hi[0] + 1 : 0); ++c[0])
    for (c[1] = nd > 2 ? lo[1] : 0; c[1] <= (nd > 2 ? hi[1] : 0); ++c[1])
      for (int k = -front; k < pitch - front; ++k, ++seen) {
        long long want[3] = {c[0], c[1], 0}, got[3];
        want[last] = k;
        mpdx::index_of(f, c[0] * s[0] * (nd > 1) + c[1] * s[1] * (nd > 2) + k, got);
        for (int q = 0; q < 3; ++q)
          if (got[q] != want[q]) {
            std::printf("nd %d: (%lld %lld %lld) is not (%lld %lld %lld)\n", nd, got[0], got[1], got[2], want[0], want[1], want[2]);
            std::exit(1);
          }
      }
  return seen;
}

int main() {
  const int lo[][3] = {{-1, -1, -1}, {-2, -2, -2}, {-2, -1, -2}, {0, -2, -33}};
  const int hi[][3] = {{5, 6, 7}, {9, 4, 61}, {6, 7, 30}, {3, 2, 40}};
  long long seen = 0;
  for (int q = 0; q < 4; ++q)
    for (int nd = 1; nd <= 3; ++nd) seen += look<float>(nd, lo[q], hi[q]) + look<double>(nd, lo[q], hi[q]);
  std::printf("%lld\n", seen);
}
