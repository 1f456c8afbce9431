// Test harness of choose_fixed_slabs (csrc/host_math.h).
#include "host_math.h"

extern "C" void slabs_check(int timesteps, int channels, long long base_blocks, long long resident, int* out) {
  leapgb::choose_fixed_slabs(timesteps, channels, base_blocks, resident, out[0], out[1], out[2], out[3]);
}
