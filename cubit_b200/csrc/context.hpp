// What the translation units behind the C ABI share: the context and elf handles and the error plumbing.
#pragma once
#include <map>
#include <memory>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

#include "../../include/cubit_b200.h"
#include "elf_text.hpp"
#include "flat_table.hpp"
#include "isa_table.hpp"
#include "sass_text.hpp"
#include "work_pool.hpp"

namespace cubit {
struct DeviceState;   // one GPU's share of a context (capi.cu)
}

struct cubit_ctx {
    cubit_ctx();
    ~cubit_ctx();
    cubit::IsaTable table;
    cubit::FlatTable flat;
    std::vector<std::unique_ptr<cubit::DeviceState>> devs;
    std::map<std::pair<std::string, std::string>, uint32_t> by_name;
    std::vector<std::vector<cubit_field_info>> field_infos;
    std::mutex err_mu;
    std::map<std::thread::id, std::string> errors;
    std::mutex synth_mu;
    // Host-side fault injection for tests (read from the environment when the context is made):
    // CUBIT_TEST_FAIL_SLOT=k makes the worker of device slot k report a failure instead of running,
    // CUBIT_TEST_FAIL_ALLOC=1 makes every growth of a staging buffer fail.  Nothing on a GPU is faulted.
    int test_fail_slot = -1;
    bool test_fail_alloc = false;
    std::unique_ptr<cubit::TextEncoder> text;          // built with the context; reads `table`
    std::vector<cubit::PrintPlan> print_plans;         // per variant
    cubit::WorkPool pool;                              // host threads of this context; joined when it is destroyed
};

struct cubit_elf {
    const uint8_t* bytes;
    uint64_t len;
    std::vector<cubit::TextSection> text;
};

namespace cubit {

// Records the message of the calling thread (for the context, or for calls without one) and returns the code.
int fail(const cubit_ctx* ctx, int code, const std::string& msg);
// What an exported function returns when an exception reaches its outermost handler: nothing
// may propagate into the caller's C frames.
int translate_exception(const cubit_ctx* ctx) noexcept;

// An array whose elements start out uninitialised (every one is written before it is read).
template <typename T>
struct RawArray {
    std::unique_ptr<T[]> p;
    RawArray() = default;
    explicit RawArray(size_t n) : p(new T[n ? n : 1]) {}
    T* data() const { return p.get(); }
    T& operator[](size_t i) const { return p[i]; }
};

}  // namespace cubit
