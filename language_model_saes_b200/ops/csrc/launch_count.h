// Kernels that this process has launched (kernel_launch_count in sae_kernels.py): counted where they are launched, so that what an entry point
// launches is not written down a second time.
#pragma once
#include <atomic>

namespace lmsae {

inline std::atomic<long long> kernel_launches{0};

}  // namespace lmsae
