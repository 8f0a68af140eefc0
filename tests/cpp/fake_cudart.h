// Controls of the CUDA runtime without a device (fake_cudart.cpp).
#pragma once

#include <cstddef>
#include <functional>
#include <map>
#include <set>
#include <string>
#include <vector>

namespace fake {
struct Launch {
  std::string kernel;  // mangled name
  int grid, grid_y, threads;
};
extern std::vector<Launch> launches;
// launches of kernels with this in their name fail; calls of this name fail ("" for none)
extern std::string fail_kernel, fail_call;
// kernels of each module (translation unit)
std::map<void **, std::vector<std::string>> &modules();
extern size_t allocated;                   // bytes of device memory held
extern std::set<const void *> device_only;  // addresses the runtime takes for device memory
// called for each launch with the kernel's arguments
extern std::function<void(const std::string &, void **)> on_launch;
// duration of a launch, and of what the host does when a kernel is first used
extern std::function<double(const std::string &, const Launch &)> kernel_ms;
extern std::function<double(const std::string &)> first_use_ms;
}  // namespace fake
