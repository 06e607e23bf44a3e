// A host build of the library's path decisions (phiray_b200/csrc/rules.cuh).
#include "../phiray_b200/csrc/rules.cuh"

extern "C" int probe_aligned16(const void* p) { return phx::aligned16(p) ? 1 : 0; }
