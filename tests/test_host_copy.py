"""The copying threads and the pinned block of pageable queries
(csrc/host_copy.h), built by itself with the two CUDA calls replaced: copies,
a forked child that destroys what it inherited, allocations that fail at each
place in turn, and memory that cannot be pinned."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

PROGRAM = r"""
#include "host_copy.h"

#include <dirent.h>
#include <sys/wait.h>

#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <new>
#include <string>

static bool pin_fails = false;
static int pinned = 0;
extern "C" cudaError_t cudaHostRegister(void*, size_t, unsigned) {
    if (pin_fails) return cudaErrorMemoryAllocation;
    ++pinned;
    return cudaSuccess;
}
extern "C" cudaError_t cudaHostUnregister(void*) {
    --pinned;
    return cudaSuccess;
}
extern "C" cudaError_t cudaGetLastError() { return cudaSuccess; }

static thread_local long allowed = -1;   // allocations of this thread before one fails; below 0: all pass
void* operator new(size_t n) {
    if (allowed == 0) throw std::bad_alloc();
    if (allowed > 0) --allowed;
    if (void* p = std::malloc(n)) return p;
    throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

// Whether this thread is alone (a joined one may be listed for a moment more).
static bool alone() {
    for (int k = 0; k < 2000; ++k) {
        int n = 0;
        DIR* d = opendir("/proc/self/task");
        while (readdir(d)) ++n;
        closedir(d);
        if (n == 3) return true;
        std::this_thread::sleep_for(std::chrono::milliseconds(1));
    }
    return false;
}

static bool copies(ilm::HostCopier& c) {
    for (size_t n : {size_t(0), size_t(1), size_t(65535), size_t(65536), size_t(65537), size_t(4) << 20}) {
        std::string from(n, 'x'), to(n + 1, '.');
        for (size_t k = 0; k < n; ++k) from[k] = (char)(k * 7 + (k >> 9));
        c.copy(&to[0], from.data(), n);
        if (to.compare(0, n, from) != 0 || to[n] != '.') return false;
    }
    return true;
}

int main(int, char** argv) {
    const std::string what = argv[1];
    alarm(60);
    if (what == "copy") {
        ilm::HostCopier c;
        for (int k = 0; k < 50; ++k)
            if (!copies(c)) return 1;
        return 0;
    }
    if (what == "fork") {
        auto* s = new ilm::HostStaging();
        ilm::HostCopier* c = s->copier.get();
        std::memset(s->block, 7, ilm::HostStaging::kBlockBytes);
        if (!copies(*c)) return 1;
        std::this_thread::sleep_for(std::chrono::milliseconds(200));   // the helpers sleep
        const pid_t child = fork();
        if (child == 0) {
            alarm(10);
            delete s;
            _exit(pinned == 1 ? 0 : 1);   // the parent's
        }
        int status = -1;
        waitpid(child, &status, 0);
        const bool ok = copies(*c) && static_cast<char*>(s->block)[ilm::HostStaging::kBlockBytes - 1] == 7;
        delete s;
        return status == 0 && ok && pinned == 0 ? 0 : 1;
    }
    if (what == "no_memory") {
        int made = 0;
        for (long k = 0; k < 40; ++k) {
            ilm::HostStaging* s = nullptr;
            allowed = k;
            try {
                s = new ilm::HostStaging();
            } catch (const std::bad_alloc&) {
            }
            allowed = -1;
            if (s) ++made;
            if (pinned != (s ? 1 : 0)) return 1;
            delete s;
            if (pinned != 0 || !alone()) return 2;
        }
        return made > 0 ? 0 : 3;
    }
    pin_fails = true;
    ilm::HostStaging s;
    return s.block == nullptr && alone() ? 0 : 1;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    if not shutil.which("g++") or not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")):
        pytest.skip("needs g++ and the CUDA headers")
    d = tmp_path_factory.mktemp("host_copy")
    src, exe = str(d / "t.cpp"), str(d / "t")
    with open(src, "w") as f:
        f.write(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O2", "-pthread", "-I" + os.path.join(ROOT, "rs_illume_b200", "csrc"),
                    "-I" + os.path.join(CUDA, "include"), src, "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("what", ["copy", "fork", "no_memory", "no_pinning"])
def test_host_copy(program, what):
    assert subprocess.run([program, what], timeout=120).returncode == 0
