// upload_and_wait returns when the data is on the device: a reader on a
// non-blocking stream (here: the host, right after the call) finds it.
#include <cstdio>
#include <cstring>
#include <vector>

#include "../../gnss-1_b200/csrc/hostblock.h"

int main() {
    const size_t n = 300000;   // more than the 64 KB up to which a pageable copy is always complete on return
    std::vector<char> src(n), dst(n, 0);
    for (size_t i = 0; i < n; ++i) src[i] = (char)(i * 7 + 1);
    if (gnss::upload_and_wait(dst.data(), src.data(), n) != cudaSuccess) return 2;
    if (std::memcmp(dst.data(), src.data(), n)) {
        std::puts("the data had not arrived when the call returned");
        return 1;
    }
    std::puts("ok");
    return 0;
}
