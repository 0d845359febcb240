// Whether an array that kernels read or write where it lies is reached as a
// whole.  The runtime answers for one address; an array may be page-locked, or
// allocated, in its first part only, and a copy refuses such a range where a
// kernel would run past its end.  Host code only.
#pragma once

#include <cstdint>

#include <driver_types.h>

namespace hrt
{
namespace api
{

// `first` and `last`: the attributes of the first and the last of `bytes` bytes.
inline bool same_block(const cudaPointerAttributes& first, const cudaPointerAttributes& last, uint64_t bytes)
{
  return first.type == last.type && first.device == last.device && first.devicePointer && last.devicePointer &&
         (uint64_t)((uintptr_t)last.devicePointer - (uintptr_t)first.devicePointer) == bytes - 1;
}

}  // namespace api
}  // namespace hrt
