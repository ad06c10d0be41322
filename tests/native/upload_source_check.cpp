// CPU check of csrc/upload_source.h against a runtime whose copies run as late
// as the CUDA documentation allows: only when something waits for them, from
// the source as it then stands.  Prints the number of bytes that arrived wrong.
#include "upload_source.h"

#include <cstdio>
#include <cstring>
#include <functional>
#include <memory>
#include <vector>

namespace {
std::vector<std::function<void()>> queue;          // the one stream
void drain() {
    for (auto& f : queue) f();
    queue.clear();
}
}  // namespace
extern "C" {
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t n, cudaMemcpyKind, cudaStream_t) {
    queue.push_back([=] { memcpy(dst, src, n); });
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
    *e = reinterpret_cast<cudaEvent_t>(new int(0));
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) {
    drain();
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) {
    delete reinterpret_cast<int*>(e);
    return cudaSuccess;
}
}
namespace qg {
bool cudaFailed(cudaError_t e, const char*, const char*) { return e != cudaSuccess; }
}  // namespace qg

int main() {
    long wrong = 0, checked = 0;
    auto check = [&](const std::vector<char>& got, size_t n, char want) {
        for (size_t i = 0; i < n; ++i, ++checked) wrong += got[i] != want;
    };
    std::vector<char> a(5000, 1), b(9000, 1), c(300, 1);
    {
        qg::UploadSource src;
        // the second copy's source grows while the first one is queued, the
        // third is queued when the object goes
        memset(src.open(a.size(), "check"), 2, a.size());
        if (!src.copy(a.data(), nullptr, "check")) return 1;
        char* p = src.open(b.size(), "check");
        for (size_t i = 0; i < b.size(); ++i, ++checked) wrong += p[i] != 0;
        memset(p, 3, b.size());
        if (!src.copy(b.data(), nullptr, "check")) return 1;
        memset(src.open(c.size(), "check"), 4, c.size());
        if (!src.copy(c.data(), nullptr, "check")) return 1;
    }
    std::vector<std::unique_ptr<char[]>> reuse;    // whatever the freed memory is used for next
    for (int k = 0; k < 64; ++k) {
        reuse.emplace_back(new char[9000]);
        memset(reuse.back().get(), 7, 9000);
    }
    drain();
    check(a, a.size(), 2);
    check(b, b.size(), 3);
    check(c, c.size(), 4);
    printf("wrong %ld\nchecked %ld\n", wrong, checked);
    return 0;
}
