// The copy threads of the pageable-operand path, in a small shared library of their own.
#include "../../cpu_ops_b200/csrc/host_copy.h"

extern "C" void probe_copy(uint8_t* dst, const uint8_t* src, size_t width, size_t rows, size_t pitch) {
  copy_threads().copy(RowCopy{dst, src, width, pitch, width, rows});
}
