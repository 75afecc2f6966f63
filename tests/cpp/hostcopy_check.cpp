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
    HostCopier::Transfer t(c);
    const cudaError_t e = up ? t.upload(&p, 1, kStream) : t.download(&p, 1, kStream);
    const cudaError_t f = t.finish();
    return e != cudaSuccess ? e : f;
}

// A copier whose threads and pinned memory have been made.
std::shared_ptr<HostCopier> warm()
{
    std::shared_ptr<HostCopier> c = HostCopier::of(0);
    std::vector<char> a(256 * kMb), b(256 * kMb);
    const int allocs = fake::hostAllocs;
    CHECK(move(*c, a, b, true) == cudaSuccess);
    CHECK(move(*c, a, b, true) == cudaSuccess);
    CHECK(fake::hostAllocs == allocs + 1);
    return c;
}

// The pinned memory is made once 96 MB of transfers of at least 12 MB have been
// copied plainly: few or small transfers never pay for it.
void stagingRule()
{
    std::shared_ptr<HostCopier> c = HostCopier::of(0);
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
    std::shared_ptr<HostCopier> c = warm();
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

// Sixty-four holders on a device share one set of threads and pinned memory, and
// the last one gives it back; another device has its own.
void shared()
{
    std::vector<std::shared_ptr<HostCopier>> holders;
    for (int k = 0; k < 64; ++k) {
        holders.push_back(HostCopier::of(0));
        std::vector<char> a = bytes(30 * kMb, static_cast<uint32_t>(k)), b(a.size());
        CHECK(move(*holders.back(), a, b, k % 2 == 0) == cudaSuccess && a == b);
    }
    CHECK(fake::hostAllocs == 1 && fake::hostFrees == 0);
    CHECK(HostCopier::of(1) != holders[0]);
    while (holders.size() > 1) {
        holders.pop_back();
    }
    CHECK(fake::hostFrees == 0);
    holders.clear();
    CHECK(fake::hostFrees == 1);
    CHECK(warm() != nullptr);
    CHECK(fake::hostAllocs == 2 && fake::hostFrees == 2);
}

// Transfers of several threads at once: one of them is staged, the others are
// copied plainly without waiting for it.
void threads()
{
    std::shared_ptr<HostCopier> c = warm();
    std::vector<std::thread> t;
    for (uint32_t k = 0; k < 6; ++k) {
        t.emplace_back([k, c] {
            for (uint32_t i = 0; i < 5; ++i) {
                std::vector<char> a = bytes((13 + k) * kMb + i, 10 * k + i), b(a.size());
                CHECK(move(*c, a, b, (k + i) % 2 == 0) == cudaSuccess && a == b);
            }
        });
    }
    for (std::thread& x : t) {
        x.join();
    }
    std::vector<char> a = bytes(20 * kMb, 1), b(a.size()), d(a.size());
    const HostCopier::Piece p{b.data(), a.data(), a.size()}, q{d.data(), a.data(), a.size()};
    HostCopier::Transfer first(*c);
    CHECK(first.upload(&p, 1, kStream) == cudaSuccess); // (holds the copier until its end)
    const int before = fake::copies;
    std::thread([&] {
        HostCopier::Transfer second(*c);
        CHECK(second.upload(&q, 1, kStream) == cudaSuccess && second.finish() == cudaSuccess && a == d);
    }).join();
    CHECK(first.finish() == cudaSuccess && a == b);
    CHECK(fake::copies <= before + 21);
}

// Errors of a copy come out of finish(), and the copier works again afterwards;
// without pinned memory, from pinned sources and while the stream is captured
// everything is copied plainly.
void errorsAndPlainCopies()
{
    {
        fake::hostAllocFails = true;
        std::shared_ptr<HostCopier> c = HostCopier::of(0);
        std::vector<char> a = bytes(200 * kMb, 1), b(a.size());
        for (int k = 0; k < 3; ++k) {
            std::fill(b.begin(), b.end(), 0);
            CHECK(move(*c, a, b, true) == cudaSuccess && a == b);
        }
        CHECK(fake::hostAllocs == 1 && fake::hostFrees == 0);
        fake::hostAllocFails = false;
        fake::hostAllocs = 0;
    }
    std::shared_ptr<HostCopier> c = warm();
    std::vector<char> a = bytes(20 * kMb + 5, 3), b(a.size());
    for (bool up : {true, false}) {
        fake::failCopyAt = fake::copies + 7;
        CHECK(move(*c, a, b, up) == cudaErrorInvalidValue);
        fake::failCopyAt = -1;
        std::fill(b.begin(), b.end(), 0);
        CHECK(move(*c, a, b, up) == cudaSuccess && a == b);
    }
    int before = fake::copies;
    fake::pinned = a.data();
    CHECK(move(*c, a, b, true) == cudaSuccess && fake::copies == before + 1);
    fake::pinned = nullptr;
    fake::capturing = true;
    CHECK(move(*c, a, b, true) == cudaSuccess && fake::copies == before + 2);
    fake::capturing = false;
    {
        HostCopier::Transfer t(*c); // (ended with the object)
        const HostCopier::Piece p{b.data(), a.data(), a.size()};
        std::fill(b.begin(), b.end(), 0);
        CHECK(t.upload(&p, 1, kStream) == cudaSuccess);
    }
    CHECK(a == b);
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
        } else if (name == "shared") {
            shared();
        } else if (name == "threads") {
            threads();
        } else if (name == "errors_and_plain_copies") {
            errorsAndPlainCopies();
        } else {
            std::printf("no check named %s\n", name.c_str());
            ++failures;
        }
    }
    return failures == 0 ? 0 : 1;
}
