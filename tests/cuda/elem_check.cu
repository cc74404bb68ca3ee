// Walking pointers of the bounds-checked build on the device: a field of 4 x 6 points with
// a halo of 1, read and written at every slot of a larger allocation around it.  Slots of
// the field go through; any other sets the record and lands on the field's first point.
// Prints "ok" or what differs.
#define MPDX_BOUNDS_CHECK
#include <cstdio>

#include "../../libmpdataxx_b200/csrc/mpdx_common.cuh"

__global__ void touch(mpdx::fptr<float> p, int first, int n, int *hit, float *seen) {
  for (int q = 0; q < n; ++q) {
    p.f.oob->hit = 0u;
    float &x = (p + first)[q];
    hit[q] = int(p.f.oob->hit);
    seen[q] = x;
  }
}

int main() {
  // rows of 64 slots (32 before index 0), 6 rows; the allocation has 4 rows more on each side
  const int pitch = 64, front = 32, rows = 6, spare = 4 * pitch, total = rows * pitch + 2 * spare;
  float *mem, *seen;
  int *hit;
  mpdx::oob_info *oob;
  cudaMallocManaged(&mem, total * sizeof(float));
  cudaMallocManaged(&seen, total * sizeof(float));
  cudaMallocManaged(&hit, total * sizeof(int));
  cudaMallocManaged(&oob, sizeof(mpdx::oob_info));
  for (int q = 0; q < total; ++q) mem[q] = float(q);
  mpdx::dfield<float> f;
  f.s0 = pitch; f.s1 = 1; f.s2 = 0;
  f.o = mem + spare + pitch + front;
  const int lo[2] = {-1, -1}, hi[2] = {4, 6};
  for (int d = 0; d < 2; ++d) { f.lo[d] = lo[d]; f.hi[d] = hi[d]; }
  f.lo[2] = -2147483647; f.hi[2] = 2147483647;
  f.oob = oob;
  touch<<<1, 1>>>(mpdx::pointer(f), int(mem - f.o), total, hit, seen);
  if (cudaDeviceSynchronize() != cudaSuccess) { std::printf("%s\n", cudaGetErrorString(cudaGetLastError())); return 1; }
  const float base = float(spare + front - 1);
  for (int q = 0; q < total; ++q) {
    const int row = q / pitch - spare / pitch - 1, col = q % pitch - front;
    const bool in = row >= lo[0] && row <= hi[0] && col >= lo[1] && col <= hi[1];
    if (hit[q] != int(!in) || seen[q] != (in ? float(q) : base)) {
      std::printf("slot %d: recorded %d, value %g\n", q, hit[q], seen[q]);
      return 1;
    }
  }
  std::printf("ok\n");
}
