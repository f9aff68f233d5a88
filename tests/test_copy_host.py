"""The host side of the staged transfers (gale_b200/csrc/gg_copy.cu) and of the device memory
behind the handles (gg_alloc.cu) on the CPU: the files compiled for the host against a
stand-in for the CUDA runtime (tests/fake_cuda.cpp)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "gale_b200", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

PRELUDE = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <sys/wait.h>
#include <unistd.h>
#include <thread>
#include <vector>
#include "gg_handle.h"
#include "gg_kernels.cuh"
extern std::atomic<int> f_registers, f_unregisters, f_copies, f_syncs;
extern std::atomic<bool> f_refuse_register;
extern size_t f_capacity, f_used, f_registered;
struct FakeStream { int device; };
using namespace gg;
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); std::exit(1); } } while (0)
constexpr size_t MB = size_t(1) << 20;
struct H1 {  // a handle on a device
    FakeStream s;
    Handle H;
    explicit H1(int dev = 0) : s{dev} {
        H.stream = reinterpret_cast<cudaStream_t>(&s);
        H.device = dev;
        copy_handle_created();
    }
    ~H1() { H.stream = nullptr; copy_handle_destroyed(); }
};
static void fill(std::vector<char>& v, unsigned seed) {
    for (size_t i = 0; i < v.size(); i++) v[i] = (char)((i * 2654435761u + seed) >> 13);
}
// both ways, compared whole
static void round_trip(Handle& H, size_t n, unsigned seed) {
    std::vector<char> a(n), d(n), b(n);
    fill(a, seed);
    copy_to_device(H, d.data(), a.data(), n);
    CHECK(d == a);
    copy_to_host(H, b.data(), d.data(), n);
    CHECK(b == a);
}
"""


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None or not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")):
        pytest.skip("no host compiler or no CUDA headers")
    d = tmp_path_factory.mktemp("copy")
    flags = [cxx, "-std=c++17", "-O1", "-pthread", "-I", os.path.join(CUDA, "include"), "-I", CSRC, "-include", "atomic",
             *("-D__d%s_rn(a,b)=((a)%s(b))" % f for f in (("add", "+"), ("sub", "-"), ("mul", "*"), ("div", "/")))]
    for f in ("gg_copy", "gg_alloc"):
        subprocess.run([*flags, "-x", "c++", "-c", os.path.join(CSRC, f + ".cu"), "-o", str(d / (f + ".o"))], check=True)
    subprocess.run([*flags, "-c", os.path.join(HERE, "fake_cuda.cpp"), "-o", str(d / "fake.o")], check=True)
    objs = [str(d / f) for f in ("gg_copy.o", "gg_alloc.o", "fake.o")]

    def run(name, body):
        src = d / (name + ".cpp")
        src.write_text(PRELUDE + "int main() {\n" + body + "\nreturn 0;\n}\n")
        exe = str(d / name)
        subprocess.run([*flags, str(src), *objs, "-o", exe], check=True)
        r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
        assert r.returncode == 0, r.stdout + r.stderr
    return run


def test_handle_of_another_device(host):
    """A thread whose current device is not the handle's: the events of its slots would belong
    to the wrong device, so the copy goes the plain way and succeeds."""
    host("device", """
        H1 h(1);
        for (size_t n : {4 * MB, 32 * MB}) round_trip(h.H, n, 1);
        cudaSetDevice(1);
        for (size_t n : {4 * MB, 32 * MB}) round_trip(h.H, n, 2);
    """)


def test_refused_slots_are_not_asked_for_again(host):
    """Where the slots cannot be registered, one attempt is made while any handle lives."""
    host("refused", """
        f_refuse_register = true;
        {
            H1 a, b;
            for (int k = 0; k < 6; k++) round_trip(k & 1 ? a.H : b.H, 64 * MB + 4097 * k, k);
            CHECK(f_registers == 1 && f_unregisters == 0);
        }
        f_refuse_register = false;
        {
            H1 a;
            for (int k = 0; k < 3; k++) round_trip(a.H, 24 * MB, k);
            CHECK(f_registers == 2);
        }
        CHECK(f_unregisters == 1);
    """)


def test_small_slots_stay_where_large_ones_are_refused(host):
    host("small", """
        H1 a;
        round_trip(a.H, 32 * MB, 1);
        CHECK(f_registers == 1 && f_registered == 4 * MB);
        f_refuse_register = true;
        const int before = f_copies;
        for (int k = 0; k < 5; k++) round_trip(a.H, 64 * MB, k);
        CHECK(f_registers == 2 && f_unregisters == 0);       // asked for once
        CHECK(f_copies - before > 10 * 64 * 4 - 64);         // and every transfer in 256 KB pieces
    """)


def test_slots_are_made_when_the_transfers_have_earned_them(host):
    """Small slots from 8 MB down, or 32 MB up, or a sum of both, large ones from 128 MB; none
    for a handle that moves less, whatever its predecessors moved; given back with the last
    handle."""
    host("earned", """
        std::vector<char> a(128 * MB), b(128 * MB);
        for (int k = 0; k < 5; k++) {  // handles one after the other, 5 MB each
            H1 h;
            for (int t = 0; t < 2; t++) copy_to_host(h.H, a.data(), b.data(), 5 * MB / 2);
            copy_to_host(h.H, a.data(), b.data(), MB - 1);  // too small to count
            copy_to_device(h.H, a.data(), b.data(), 12 * MB - 1);
        }
        CHECK(f_registers == 0);
        {
            H1 h;
            for (int t = 0; t < 4; t++) {
                CHECK(f_registers == 0);
                copy_to_host(h.H, a.data(), b.data(), 2 * MB);
            }
            CHECK(f_registers == 1 && f_registered == 4 * MB);
            round_trip(h.H, 60 * MB + 5, 1);
            CHECK(f_registers == 1);
            copy_to_host(h.H, a.data(), b.data(), 50 * MB);  // 133 MB by now
            CHECK(f_registers == 2 && f_unregisters == 1 && f_registered == 16 * MB);
            round_trip(h.H, 33 * MB + 4099, 2);
            CHECK(f_registers == 2);
        }
        CHECK(f_unregisters == 2);
        {
            H1 h;
            copy_to_device(h.H, a.data(), b.data(), 31 * MB);
            CHECK(f_registers == 2);
            copy_to_device(h.H, a.data(), b.data(), 12 * MB);
            CHECK(f_registers == 3 && f_registered == 4 * MB);
        }
        {
            H1 h;
            copy_to_host(h.H, a.data(), b.data(), 128 * MB);
            CHECK(f_registers == 4 && f_registered == 16 * MB);
        }
        CHECK(f_unregisters == 4);
    """)


def test_threads_on_both_ways(host):
    """Transfers of several handles at once, uploads above their threshold among them: one has
    the slots, the others copy, and every array arrives whole."""
    host("threads", """
        H1 h[4];
        std::vector<std::thread> ts;
        for (int k = 0; k < 4; k++)
            ts.emplace_back([&, k] {
                for (int t = 0; t < 12; t++) round_trip(h[k].H, 12 * MB + 77773 * (k + 4 * t) - 1, k + t);
            });
        for (auto& t : ts) t.join();
        CHECK(f_registers == 2 && f_unregisters == 1);  // small, then large slots
    """)


def test_kept_point_scratch_is_lent(host):
    """Scratch that a handle keeps between calls is taken back when any handle of its device
    needs the memory, not while a call uses it, not from another device; beyond its bound it
    is not kept at all."""
    host("scratch", """
        const size_t GB = size_t(1) << 30;
        f_capacity = 4 * GB;
        H1 a, b;
        {
            PointScratch::Use use(a.H.point_scratch);
            a.H.point_scratch.coords.ensure(600 * MB);
            a.H.point_scratch.int_w.ensure(300 * MB);
            a.H.point_scratch.keep.ensure(MB);  // from the pool
        }
        CHECK(a.H.point_scratch.held() == 901 * MB);  // kept
        DBuf x;
        x.ensure(3 * GB);  // fits beside it
        CHECK(a.H.point_scratch.held() == 901 * MB);
        {
            PointScratch::Use use(a.H.point_scratch);
            DBuf y;
            bool refused = false;
            try { y.ensure(600 * MB); } catch (const CudaError&) { refused = true; }
            CHECK(refused && a.H.point_scratch.held() == 901 * MB);  // in use: not taken
        }
        cudaSetDevice(1);
        {
            DBuf y;
            bool refused = false;
            try { y.ensure(600 * MB); } catch (const CudaError&) { refused = true; }
            CHECK(refused && a.H.point_scratch.held() == 901 * MB);  // another device's
        }
        cudaSetDevice(0);
        DBuf y;
        y.ensure(600 * MB);  // by a handle or buffer that knows nothing of it
        CHECK(a.H.point_scratch.held() == 0 && y.p);
        y.release();
        x.release();
        const size_t before = f_used;
        {
            PointScratch::Use use(b.H.point_scratch);
            b.H.point_scratch.coords.ensure(GB);
            CHECK(b.H.point_scratch.held() == GB);
        }
        CHECK(b.H.point_scratch.held() == GB);
        {
            PointScratch::Use use(b.H.point_scratch);
            b.H.point_scratch.xi.ensure(8 * MB);
        }
        CHECK(b.H.point_scratch.held() == 0 && f_used == before);
    """)


def test_pool_chunk_takes_lent_scratch_back(host):
    """The same for a small buffer whose pool needs a new chunk, with small scratch that goes
    back to that pool."""
    host("chunk", """
        f_capacity = 200 * MB;
        H1 a;
        {
            PointScratch::Use use(a.H.point_scratch);
            a.H.point_scratch.coords.ensure(100 * MB);
            a.H.point_scratch.ps.ensure(3 * MB);
        }
        DBuf small[40];
        for (int k = 0; k < 16; k++) small[k].ensure(4 * MB - 1);  // the first chunk, and one block too many
        CHECK(a.H.point_scratch.held() == 0);
        for (int k = 16; k < 32; k++) small[k].ensure(4 * MB - 1);  // the second chunk and the returned block
        bool refused = false;
        try { small[32].ensure(4 * MB); small[33].ensure(200 * MB); } catch (const CudaError&) { refused = true; }
        CHECK(refused);
    """)


def test_results_past_the_caches_arrive_whole(host):
    """Sizes around the range that goes past the caches, into arrays at odd addresses, with
    nothing written outside them."""
    host("past", """
        H1 h;
        std::vector<char> src(33 * MB), dst(33 * MB + 256);
        fill(src, 3);
        copy_to_host(h.H, dst.data(), src.data(), 33 * MB);  // the slots are there from now on
        for (size_t n : {7 * MB / 4 - 1, 7 * MB / 4, 2 * MB + 13, 5 * MB + 63, 18 * MB - 1, 18 * MB, 20 * MB + 1})
            for (size_t off : {size_t(0), size_t(1), size_t(8), size_t(15), size_t(33)}) {
                std::memset(dst.data(), 0x5a, n + 256);
                copy_to_host(h.H, dst.data() + off, src.data() + 7, n);
                CHECK(std::memcmp(dst.data() + off, src.data() + 7, n) == 0);
                for (size_t k = 0; k < off; k++) CHECK(dst[k] == 0x5a);
                for (size_t k = off + n; k < n + 256; k++) CHECK(dst[k] == 0x5a);
            }
    """)


def test_forked_child_drops_its_handles(host):
    """A child of fork has the handles but not the copy threads: destroying the last handle
    there returns, and the parent's slots go on."""
    host("fork", """
        H1* h = new H1;
        round_trip(h->H, 32 * MB, 1);
        CHECK(f_registers == 1);
        const pid_t pid = fork();
        if (pid == 0) {
            alarm(20);  // ends a child that waits for threads it does not have
            delete h;
            H1 other;  // nor are there slots for a new one
            _exit(f_unregisters == 0 ? 0 : 2);
        }
        int status = 0;
        CHECK(waitpid(pid, &status, 0) == pid);
        CHECK(WIFEXITED(status) && WEXITSTATUS(status) == 0);
        round_trip(h->H, 32 * MB + 77, 2);
        delete h;
        CHECK(f_unregisters == 1);
    """)
