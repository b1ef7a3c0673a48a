// Module definition, library binding, device guard and status words of the native host path.
#include "host_common.h"

#include <mutex>

namespace cula_host {

Lib lib;

namespace {

void bind(const std::string& path) {
    void* h = dlopen(path.c_str(), RTLD_NOW | RTLD_LOCAL);
    if (!h) throw std::runtime_error(std::string("cannot load ") + path + ": " + dlerror());
#define CULA_KDA_LOAD(name)                                                                      \
    lib.name = reinterpret_cast<decltype(lib.name)>(dlsym(h, #name));                            \
    if (!lib.name) throw std::runtime_error(std::string("missing symbol ") + #name + " in " + path);
    CULA_KDA_ENTRIES(CULA_KDA_LOAD)
#undef CULA_KDA_LOAD
}

std::mutex status_mutex;
Tensor status_tensors[64];
std::atomic<int*> status_ptrs[64];
std::atomic<bool> blackwell[64];

const char* status_message(int code) {
    switch (code) {
        case 1: return "a bounded in-kernel wait timed out";
        case 2: return "a state-pool index lies past the end of the pool";
        case 3: return "a forward intermediate (w, u, kg, qg or Aqk) left the fp16 range or is not finite; "
                       "check the magnitude of v (|v| < 65504 is required) and of the gate";
        default: return "unknown";
    }
}

}  // namespace

void assert_blackwell(const Tensor& t) {
    const int dev = t.is_cuda() ? t.device().index() : -1;
    if (dev >= 0 && dev < 64 && blackwell[dev].load(std::memory_order_relaxed)) return;
    if (!at::globalContext().hasCUDA() || at::cuda::device_count() == 0)
        throw std::runtime_error("cula_b200 needs a CUDA device (B200, sm_100a); there is no CPU fallback.");
    if (dev < 0) throw std::runtime_error("cula_b200 operators take CUDA tensors.");
    const int major = at::cuda::getDeviceProperties(dev)->major;
    if (major != 10)
        throw std::runtime_error("cula_b200 kernels are built for sm_100a; found compute capability " + std::to_string(major) + ".x");
    if (dev < 64) blackwell[dev].store(true, std::memory_order_relaxed);
}

int* status_word(int dev) {
    TORCH_CHECK(dev >= 0 && dev < 64, "device index out of range");
    if (int* p = status_ptrs[dev].load(std::memory_order_acquire)) return p;
    std::lock_guard<std::mutex> lock(status_mutex);
    if (int* p = status_ptrs[dev].load(std::memory_order_acquire)) return p;
    c10::InferenceMode off(false);
    status_tensors[dev] = at::zeros({1}, at::TensorOptions().dtype(at::kInt).pinned_memory(true));
    status_ptrs[dev].store(status_tensors[dev].data_ptr<int>(), std::memory_order_release);
    return status_ptrs[dev].load();
}

void poll_status(int dev) {
    int* p = status_ptrs[dev].load(std::memory_order_acquire);
    if (!p) return;
    const int code = *reinterpret_cast<volatile int*>(p);
    if (code == 0) return;
    c10::cuda::CUDAGuard guard((c10::DeviceIndex)dev);
    c10::cuda::device_synchronize();               // whatever else is in flight reports now, not after the word is cleared
    *reinterpret_cast<volatile int*>(p) = 0;
    throw std::runtime_error("cula_b200 kernel status " + std::to_string(code) + ": " + status_message(code));
}

}  // namespace cula_host

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
    m.def("bind", &cula_host::bind);
    m.def("poll_status", &cula_host::poll_status);
    m.def("status_ptr", [](int dev) { return (int64_t)(intptr_t)cula_host::status_word(dev); });
    cula_host::bind_attention(m);
    cula_host::bind_layer_ops(m);
}
