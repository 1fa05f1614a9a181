// A request's state slots set to zero before its first tokens: all layers' states of all new requests in one launch.
//
// Slots and state pointers travel as kernel arguments, so nothing is copied to the device and the host waits for nothing: by a list
// of slots copied to the device and a fill a state, a step with new requests waited for the step before it to end, and the device then idled
// until the host had launched again (60 to 210 us a step on B200: Nesezen, a prompt of 1,501 beside 24 requests, 1,881 -> 1,670; Tofilorn, 2,048 tokens, 3,158 -> 2,976).  The fill itself is bound by memory.
#include "common.cuh"

namespace vob {

constexpr int CLEAR_STATES = 16, CLEAR_SLOTS = 64, CLEAR_BLOCKS = 32;      // of a launch; blocks a (slot, state)

struct ClearList {
  char* state[CLEAR_STATES];
  long row_bytes[CLEAR_STATES];      // bytes of a slot
  int slot[CLEAR_SLOTS];
};

__global__ void __launch_bounds__(256)
clear_states_kernel(const __grid_constant__ ClearList list) {
  const int s = blockIdx.z, slot = list.slot[blockIdx.y];
  const long bytes = list.row_bytes[s], step = (long)CLEAR_BLOCKS * 256;
  char* row = list.state[s] + slot * bytes;
  long i = (long)blockIdx.x * 256 + threadIdx.x;
  if (bytes % 16 == 0 && (uintptr_t)row % 16 == 0) {
    for (; i < bytes / 16; i += step) reinterpret_cast<uint4*>(row)[i] = make_uint4(0u, 0u, 0u, 0u);
  } else {
    for (; i < bytes; i += step) row[i] = 0;
  }
}

}  // namespace vob

using namespace vob;

// Zeros in slot slots[j] of every state: states [n_states] pointers, row_bytes and num_slots [n_states] (arrays on the host, read before
// this returns).
VOB_API int vob_clear_states(const unsigned long long* states, const long* row_bytes, const long* num_slots, int n_states, const int* slots,
                             int n_slots, cudaStream_t stream) {
  for (int s = 0; s < n_states; ++s)
    for (int j = 0; j < n_slots; ++j)
      if (!states[s] || row_bytes[s] <= 0 || slots[j] < 0 || slots[j] >= num_slots[s]) return VOB_BAD_ARGUMENT;
  for (int s0 = 0; s0 < n_states; s0 += CLEAR_STATES)
    for (int j0 = 0; j0 < n_slots; j0 += CLEAR_SLOTS) {
      ClearList list = {};
      const int ns = n_states - s0 < CLEAR_STATES ? n_states - s0 : CLEAR_STATES;
      const int nj = n_slots - j0 < CLEAR_SLOTS ? n_slots - j0 : CLEAR_SLOTS;
      for (int s = 0; s < ns; ++s) {
        list.state[s] = (char*)states[s0 + s];
        list.row_bytes[s] = row_bytes[s0 + s];
      }
      for (int j = 0; j < nj; ++j) list.slot[j] = slots[j0 + j];
      // (a plain launch: the kernels of the step may read a state before they wait for the kernels ahead of them)
      clear_states_kernel<<<dim3(CLEAR_BLOCKS, nj, ns), 256, 0, stream>>>(list);
      const int code = launch_status();
      if (code != 0) return code;
    }
  return 0;
}
