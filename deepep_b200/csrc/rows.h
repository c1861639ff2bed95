// What every kernel assumes of the rows it reads and writes in 16-byte pieces, checked before a launch: an access off its boundary
// would end the process's CUDA context.
#pragma once
#include <cstdint>
#include <initializer_list>
#include <stdexcept>
#include <string>

namespace dep {

// `rows` rows at each address (none needs no memory, and a null address is another check's business).
inline void require_rows(long long rows, std::initializer_list<const void*> bases, const char* what) {
  for (const void* base : bases)
    if (rows > 0 && reinterpret_cast<uintptr_t>(base) % 16)
      throw std::invalid_argument(std::string(what) + ": rows must start on a 16-byte boundary");
}

}  // namespace dep
