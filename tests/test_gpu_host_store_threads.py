"""The threads that prepare the host store's slabs: a process that may start none goes on without them, and none outlives
the memory that it works for."""
import os
import subprocess
import sys
import textwrap

import pytest
import torch

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
MEMORY = textwrap.dedent("""
    import os, sys, ctypes
    sys.path.insert(0, %r)
    import torch
    from infllm_b200.attention import ContextManager, RotaryEmbeddingESM

    def memory(units):  # units of 2 MiB, 64 to a slab; the next slab is asked for from the 33rd on
        n = 64 + 256 + units * 128
        g = torch.Generator(device="cuda").manual_seed(1)
        q, k, v = (torch.randn((1, 32, n, 128), generator=g, device="cuda").to(torch.bfloat16) for _ in range(3))
        cm = ContextManager(RotaryEmbeddingESM(128, 1e6, 1.0), 64, 256, 128, 8, 8, 256, None, True, 2)
        torch.cuda.synchronize()
        return cm, cm.append(q, k, v, q, k, v)
""" % ROOT)


def _run(code, **env):
    r = subprocess.run([sys.executable, "-c", MEMORY + textwrap.dedent(code)], env={**os.environ, **env}, timeout=300,
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout


def test_a_process_that_can_start_no_thread(tmp_path):
    src, lib = tmp_path / "no_threads.c", tmp_path / "no_threads.so"
    src.write_text("""
        #define _GNU_SOURCE
        #include <dlfcn.h>
        #include <errno.h>
        #include <pthread.h>
        static int off, refused;
        void no_threads(int on) { off = on; }
        int threads_refused(void) { return refused; }
        int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* x) {
          static int (*real)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*);
          if (!real) real = dlsym(RTLD_NEXT, "pthread_create");
          if (off) return ++refused, EAGAIN;
          return real(t, a, f, x);
        }""")
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(lib), str(src), "-ldl"], check=True)
    out = _run("""
        cm, want = memory(40)
        torch.cuda.synchronize()
        del cm
        from infllm_b200.attention import release_idle_memories
        release_idle_memories()
        shim = ctypes.CDLL(None)
        shim.no_threads(1)
        cm, got = memory(40)
        torch.cuda.synchronize()
        print(shim.threads_refused(), cm.num_global_block, torch.equal(got, want))
        shim.no_threads(0)
    """, LD_PRELOAD=str(lib))
    refused, units, equal = out.split()[-3:]
    assert int(refused) >= 4 and int(units) == 40 and equal == "True"


def test_no_thread_outlives_its_memory():
    out = _run("""
        cm, _ = memory(20)
        torch.cuda.synchronize()
        del cm
        before = len(os.listdir("/proc/self/task"))
        cm, out = memory(33)
        del cm
        print(before, len(os.listdir("/proc/self/task")))
    """)
    before, after = map(int, out.split()[-2:])
    assert after <= before
