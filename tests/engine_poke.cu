// Looks into an engine: what no call of the library lets a test set.
#include "jf_engine.h"

// The slot of instance m's particle at engine position k becomes `slot`; the one it had into *old.
extern "C" int poke_slot(jf_engine* e, int m, int k, int32_t slot, int32_t* old) {
  int32_t* at = e->p.slot + e->inst[m].p_off + k;
  cudaError_t err = cudaMemcpy(old, at, sizeof(int32_t), cudaMemcpyDeviceToHost);
  if (err == cudaSuccess) err = cudaMemcpy(at, &slot, sizeof(int32_t), cudaMemcpyHostToDevice);
  return (int)err;
}
