// Checks of the bindings: a failed one is a std::runtime_error, which pybind11 turns into RuntimeError. Messages are put
// together with std::to_string: a TORCH_CHECK whose message holds a number formats it through a stream, and where the
// extension is linked with its own copy of the C++ library (g++ of the CUDA image) that ends the process with SIGSEGV.
#pragma once
#include <stdexcept>
#include <string>

inline void need(bool ok, const char* what) {
  if (!ok) throw std::runtime_error(std::string("terra_b200: ") + what);
}
inline void rc_check(int rc, const char* what) {
  if (rc != 0) throw std::runtime_error(std::string("terra_b200: ") + what + " failed with code " + std::to_string(rc));
}
