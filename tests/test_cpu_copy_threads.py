"""The helper threads of the host copies (csrc/copy_threads.h): every row is copied once
whatever the number of rows, helpers and calls, also where no thread or no memory can be
had (nothing is thrown, the calling thread does the work) and in a forked child."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "subsecondpbs_b200" / "csrc"

PROGRAM = r"""
#include <dlfcn.h>
#include <errno.h>
#include <pthread.h>
#include <sys/wait.h>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <new>
#include <vector>
#include "copy_threads.h"

static int threadsLeft = 1000, newsLeft = 1 << 30;
extern "C" int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* x) {
    using Fn = int (*)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*);
    static Fn real = (Fn)dlsym(RTLD_NEXT, "pthread_create");
    return threadsLeft-- > 0 ? real(t, a, f, x) : EAGAIN;
}
void* operator new(size_t n) {
    if (newsLeft-- <= 0) throw std::bad_alloc();
    if (void* p = malloc(n ? n : 1)) return p;
    throw std::bad_alloc();
}
void operator delete(void* p) noexcept { free(p); }
void operator delete(void* p, size_t) noexcept { free(p); }

static bool copies(pbs::CopyThreads& t, size_t n, size_t bytes) {
    std::vector<int> seen(n, 0);
    int* s = seen.data();
    t.split(n, bytes, [&](size_t a, size_t b) {
        for (size_t i = a; i < b; ++i) ++s[i];
    });
    for (size_t i = 0; i < n; ++i)
        if (s[i] != 1) return false;
    return true;
}

int main(int argc, char** argv) {
    const char* mode = argv[1];
    bool ok = true;
    if (!strcmp(mode, "rows")) {
        pbs::CopyThreads t;
        const size_t sizes[] = {1, 2, 3, 4, 5, 7, 64, 1001};
        for (int k = 0; k < 300; ++k)
            for (size_t n : sizes) ok = ok && copies(t, n, (k % 5) * (size_t(64) << 10));
    } else if (!strcmp(mode, "threads")) {
        for (threadsLeft = 0; threadsLeft < 3;) {
            const int had = threadsLeft;
            pbs::CopyThreads t;
            for (int k = 0; k < 20; ++k) ok = ok && copies(t, 1001, size_t(1) << 20);
            threadsLeft = had + 1;
        }
    } else if (!strcmp(mode, "memory")) {
        // The state, then each thread's own allocation.
        for (int news = 1; news < 6; ++news) {
            pbs::CopyThreads t;
            newsLeft = news;  // the first one is the test's vector
            ok = ok && copies(t, 1001, size_t(1) << 20);
            newsLeft = 1 << 30;
            ok = ok && copies(t, 1001, size_t(1) << 20);
        }
    } else if (!strcmp(mode, "fork")) {
        pbs::CopyThreads t;
        ok = copies(t, 1001, size_t(1) << 20);
        const pid_t child = fork();
        ok = ok && copies(t, 1001, size_t(1) << 20);
        if (child == 0) return ok ? 0 : 1;  // destroys t
        int status = 1;
        waitpid(child, &status, 0);
        ok = ok && status == 0;
    }
    puts(ok ? "ok" : "wrong");
    return ok ? 0 : 1;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("no C++ compiler")
    d = tmp_path_factory.mktemp("copy_threads")
    (d / "t.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", str(CSRC), "-o", str(d / "t"), str(d / "t.cpp"), "-lpthread", "-ldl"],
                   check=True)
    return d / "t"


@pytest.mark.parametrize("mode", ["rows", "threads", "memory", "fork"])
def test_every_row_once(program, mode):
    r = subprocess.run([str(program), mode], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and "wrong" not in r.stdout, r.stdout + r.stderr
