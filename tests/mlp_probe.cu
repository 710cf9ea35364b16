// Where a network's device status words are kept in its handle (MlpParams is its first member).
#include <cstddef>

#include "common.cuh"

extern "C" size_t err_offset() { return offsetof(cube::MlpParams, err); }
extern "C" int set_train_err(void *handle, int value) {
  int *const err = *reinterpret_cast<int **>(static_cast<char *>(handle) + err_offset());
  return cudaMemcpy(err + cube::kMlpErrTrain, &value, sizeof(int), cudaMemcpyHostToDevice);
}
