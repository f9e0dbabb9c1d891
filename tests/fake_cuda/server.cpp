// The server of batch.cpp on the host runtime: one scenario per run, named by
// the first argument.
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "fake_ctx.h"
#include "fake_cuda.h"

#define EXPECT(x)                                             \
    do {                                                      \
        if (!(x)) {                                           \
            std::printf("line %d: %s\n", __LINE__, #x);       \
            return 1;                                         \
        }                                                     \
    } while (0)

static gnss_config config(int n, int device = 0) {
    gnss_config c{};
    c.nx = c.ny = c.nz = n;
    c.n_scalars = 1;
    c.precision = GNSS_FP32;
    c.device = device;
    return c;
}
static std::vector<char> state_of(const gnss_config &c) {
    return std::vector<char>((size_t)c.nx * c.ny * (c.nz / 2 + 1) * 8 * (3 + c.n_scalars), 1);
}
static gnss_server *server(int max_active, int device = 0) {
    gnss_server_config sc{};
    sc.budget_bytes = (size_t)1 << 34;
    sc.max_active = max_active;
    sc.steps_per_launch = 100;   // requests below: single launches
    sc.device = device;
    gnss_server *s = nullptr;
    return gnss_server_create(&sc, &s) == GNSS_OK ? s : nullptr;
}

// A request whose fourth step fails leaves three steps queued on its stream; its context must not serve another
// request.
static int failed_request() {
    const gnss_config c = config(8);
    const std::vector<char> st = state_of(c);
    gnss_server *s = server(4);
    long long id = 0;
    fake::fail_after = 3;
    EXPECT(gnss_server_submit(s, &c, st.data(), 12, &id) == GNSS_OK);
    EXPECT(gnss_server_wait(s, id, 10.0) == GNSS_OK);
    EXPECT(fake::fail_after < 0);
    long long id2 = 0;
    EXPECT(gnss_server_submit(s, &c, st.data(), 12, &id2) == GNSS_OK);
    EXPECT(gnss_server_wait(s, id2, 10.0) == GNSS_OK);
    EXPECT(fake::recycled_busy == 0);
    EXPECT(fake::recycled == 0);
    EXPECT(gnss_server_result(s, id, nullptr, nullptr, nullptr) == GNSS_ERR_CUDA);
    EXPECT(gnss_server_result(s, id2, nullptr, nullptr, nullptr) == GNSS_OK);
    // the second one ended well: a third request takes its context over
    EXPECT(gnss_server_submit(s, &c, st.data(), 12, &id) == GNSS_OK);
    EXPECT(gnss_server_wait(s, id, 10.0) == GNSS_OK);
    EXPECT(fake::recycled == 1 && fake::recycled_busy == 0);
    EXPECT(gnss_server_destroy(s) == GNSS_OK);
    EXPECT(fake::live == 0);
    return 0;
}

// After a burst of requests (of one geometry, then of several more) has been fetched, no more than 64 idle contexts
// are left; none was destroyed on the scheduler's thread, and the caller's device is as it was.
static int idle_contexts() {
    gnss_server *s = server(4);
    const int sizes[] = {8, 12, 16};
    for (int n : sizes) {
        const gnss_config c = config(n);
        const std::vector<char> st = state_of(c);
        std::vector<long long> ids(200);
        for (long long &id : ids) EXPECT(gnss_server_submit(s, &c, st.data(), 2, &id) == GNSS_OK);
        EXPECT(cudaSetDevice(1) == cudaSuccess);
        for (long long id : ids) {
            EXPECT(gnss_server_wait(s, id, 30.0) == GNSS_OK);
            EXPECT(gnss_server_result(s, id, nullptr, nullptr, nullptr) == GNSS_OK);
        }
        EXPECT(fake::current_device() == 1);
        EXPECT(fake::live <= 64);
    }
    EXPECT(fake::destroyed_elsewhere == 0);
    EXPECT(fake::recycled_busy == 0);
    EXPECT(gnss_server_destroy(s) == GNSS_OK);
    EXPECT(fake::live == 0);
    return 0;
}

// A submission that takes over an idle context leaves the calling thread on the server's device, as one that creates
// its context does; its pinned buffers belong there.
static int device_of_reuse() {
    const gnss_config c = config(8, 1);
    const std::vector<char> st = state_of(c);
    gnss_server *s = server(4, 1);
    long long a = 0, b = 0;
    EXPECT(gnss_server_submit(s, &c, st.data(), 2, &a) == GNSS_OK);
    EXPECT(fake::current_device() == 1 && fake::last_host_alloc_device() == 1);
    EXPECT(gnss_server_wait(s, a, 10.0) == GNSS_OK);   // not fetched: its pinned buffers are in use
    EXPECT(cudaSetDevice(0) == cudaSuccess);
    EXPECT(gnss_server_submit(s, &c, st.data(), 2, &b) == GNSS_OK);
    EXPECT(fake::recycled == 1);
    EXPECT(fake::last_host_alloc_device() == 1);
    EXPECT(fake::current_device() == 1);
    EXPECT(gnss_server_wait(s, b, 10.0) == GNSS_OK);
    EXPECT(gnss_server_destroy(s) == GNSS_OK);
    EXPECT(fake::live == 0);
    return 0;
}

// A state of several MB is copied in and out in parts, byte for byte.
static int large_state() {
    gnss_config c = config(96);
    c.nz = 64;   // 96 x 96 x 33 x 4 x 8 bytes, 9.7 MB
    std::vector<char> st = state_of(c), out(st.size(), 0);
    for (size_t i = 0; i < st.size(); ++i) st[i] = (char)(i * 31 + (i >> 13));
    gnss_server *s = server(2);
    long long id = 0;
    EXPECT(gnss_server_submit(s, &c, st.data(), 3, &id) == GNSS_OK);
    EXPECT(gnss_server_wait(s, id, 10.0) == GNSS_OK);
    EXPECT(gnss_server_result(s, id, out.data(), nullptr, nullptr) == GNSS_OK);
    EXPECT(st == out);
    EXPECT(gnss_server_destroy(s) == GNSS_OK);
    return 0;
}

int main(int argc, char **argv) {
    const std::string name = argc > 1 ? argv[1] : "";
    if (name == "failed_request") return failed_request();
    if (name == "idle_contexts") return idle_contexts();
    if (name == "device_of_reuse") return device_of_reuse();
    if (name == "large_state") return large_state();
    return 2;
}
