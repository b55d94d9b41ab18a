// How a field of a state is copied between device arrays (aqua_set_state,
// aqua_get_state).
#pragma once

#include <cstdint>

namespace aqua {

// By the kernel that copies all fields at once: memory of the context's
// device, at an address of whole words, while that device is current (a kernel
// runs on the current device).  Everything else goes by cudaMemcpyAsync, which
// takes any address and runs whichever device is current.
inline bool
copied_by_kernel(bool device_memory, int memory_device, int context_device,
                 int current_device, const void* address)
{
    return device_memory && memory_device == context_device &&
           current_device == context_device &&
           (reinterpret_cast<std::uintptr_t>(address) & 3) == 0;
}

}  // namespace aqua
