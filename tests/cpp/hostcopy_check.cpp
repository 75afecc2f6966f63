// Host-side checks of csrc/pt_hostcopy.cuh against the stand-in runtime, one per
// name given on the command line (tests/test_hostcopy.py).  Exit code 0: it holds.
#include "pt_hostcopy.cuh"

#include <cstdint>
#include <cstdio>
#include <string>
#include <sys/wait.h>
#include <unistd.h>

using pt::HostCopier;

namespace {

constexpr size_t kMb = 1u << 20;
const cudaStream_t kStream = reinterpret_cast<cudaStream_t>(1);
int failures = 0;

#define CHECK(x) \
    do { \
        if (!(x)) { \
            std::printf("line %d: %s\n", __LINE__, #x); \
            ++failures; \
        } \
    } while (0)

std::vector<char> bytes(size_t n, uint32_t seed)
{
    std::vector<char> v(n);
    for (size_t i = 0; i < n; ++i) {
        seed = seed * 1664525u + 1013904223u;
        v[i] = static_cast<char>(seed >> 24);
    }
    return v;
}

// One transfer of `a` to `b`; up: a is the host's.
cudaError_t move(HostCopier& c, std::vector<char>& a, std::vector<char>& b, bool up)
{
    const HostCopier::Piece p = up ? HostCopier::Piece{b.data(), a.data(), a.size()} : HostCopier::Piece{a.data(), b.data(), a.size()};
    cudaError_t e = up ? c.beginUpload(&p, 1, kStream) : c.beginDownload(&p, 1, kStream);
    const cudaError_t f = c.finish();
    return e != cudaSuccess ? e : f;
}

// A copier whose threads and pinned memory have been made.
HostCopier::Owner warm()
{
    HostCopier::Owner c(new HostCopier(0));
    std::vector<char> a(256 * kMb), b(256 * kMb);
    CHECK(move(*c, a, b, true) == cudaSuccess);
    CHECK(move(*c, a, b, true) == cudaSuccess);
    CHECK(fake::hostAllocs == 1);
    return c;
}

// The pinned memory is made once 96 MB of transfers of at least 12 MB have been
// copied plainly: few or small transfers never pay for it.
void stagingRule()
{
    HostCopier::Owner c(new HostCopier(0));
    auto moves = [&](size_t n, int times, bool up) {
        std::vector<char> a = bytes(n, static_cast<uint32_t>(n)), b(n);
        for (int k = 0; k < times; ++k) {
            std::fill(b.begin(), b.end(), 0);
            CHECK(move(*c, a, b, up) == cudaSuccess && a == b);
        }
    };
    moves(12 * kMb - 1, 40, true);
    moves(1, 3, false);
    CHECK(fake::hostAllocs == 0);
    moves(12 * kMb, 4, true);
    moves(12 * kMb, 4, false);
    CHECK(fake::hostAllocs == 0);
    const int before = fake::copies;
    moves(12 * kMb + 1, 1, true); // (13 slices)
    CHECK(fake::hostAllocs == 1 && fake::copies == before + 13);
    moves(12 * kMb - 1, 1, true);
    CHECK(fake::copies == before + 14);
    moves(40 * kMb + 77, 3, false);
    CHECK(fake::hostAllocs == 1 && fake::copies == before + 14 + 3 * 41);
    c.reset();
    CHECK(fake::hostFrees == 1);
}

// A forked child gives the copier back without its threads, and copies plainly.
void forkedChild()
{
    HostCopier::Owner c = warm();
    usleep(50000); // (the workers wait for the next transfer)
    const pid_t child = fork();
    if (child == 0) {
        alarm(20);
        std::vector<char> a = bytes(40 * kMb, 1), b(a.size());
        CHECK(move(*c, a, b, true) == cudaSuccess && a == b);
        c.reset();
        _exit(failures == 0 && fake::hostFrees == 0 ? 0 : 1);
    }
    int status = -1;
    CHECK(waitpid(child, &status, 0) == child);
    CHECK(WIFEXITED(status) && WEXITSTATUS(status) == 0);
    std::vector<char> a = bytes(40 * kMb, 2), b(a.size());
    CHECK(move(*c, a, b, true) == cudaSuccess && a == b);
    c.reset();
    CHECK(fake::hostFrees == 1);
}

} // namespace

int main(int argc, char** argv)
{
    for (int k = 1; k < argc; ++k) {
        const std::string name = argv[k];
        if (name == "forked_child") {
            forkedChild();
        } else if (name == "staging_rule") {
            stagingRule();
        } else {
            std::printf("no check named %s\n", name.c_str());
            ++failures;
        }
    }
    return failures == 0 ? 0 : 1;
}
