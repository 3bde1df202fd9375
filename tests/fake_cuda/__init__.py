"""Runs library calls on the host against fake_cudart.cpp (see there).

``run(body)`` executes Python source in a child process with the fake runtime
preloaded.  The source sees ``L`` (the library), ``F`` (the fake's controls),
``log()`` (the operations so far, split into fields), ``clear()``, and helpers for
buffers; it prints one JSON value with ``done(value)``, which ``run`` returns.
Results of device work are meaningless (kernels do nothing): only what the host
code allocates, queues, orders, refuses and frees can be looked at.
"""
import json
import os
import subprocess
import sys
import tempfile

HERE = os.path.dirname(os.path.abspath(__file__))

_PREAMBLE = '''
import ctypes as C, json, sys
F = C.CDLL({fake!r})
F.fake_log.restype = C.c_char_p
F.fake_used.restype = C.c_size_t
L = C.CDLL({lib!r})
L.catmsm_basis_create.restype = C.c_void_p
L.catmsm_server_create.restype = C.c_void_p
L.catmsm_server_submit_msm.restype = C.c_int64
L.catmsm_server_submit_fft.restype = C.c_int64
L.blst_p1_fft_with_domain.restype = C.c_bool
S = C.c_size_t
P = C.c_void_p
_keep = []
def log():
    return [l.split() for l in F.fake_log().decode().splitlines()]
def clear():
    F.fake_clear()
def limit(n):
    F.fake_limit(S(n))
def fail(name, nth=1):
    F.fake_fail(name.encode(), nth)
def buf(n):
    b = (C.c_char * n)()
    _keep.append(b)
    return C.c_void_p(C.addressof(b))
def aligned(n):
    b = buf(n + 64)
    return C.c_void_p((b.value + 63) & ~63)
def pin(b, n):
    F.fake_pin(b, S(n))
    return b
def sizes(v):
    return (S * len(v))(*v)
def domain(n):
    """A domain of n zero roots with the tag that the library asks for (n, Montgomery)."""
    b = buf(32 * (n + 2))
    r = 0x73eda753299d7d483339d80809a1d80553bda402fffe5bfeffffffff00000001
    C.memmove(b.value + 32 * (n + 1), (n * 2**256 % r).to_bytes(32, "little"), 32)
    return b
def kernels():
    return [l[2] for l in log() if l[0] == "launch"]
class Basis:
    def __init__(self, n, window, chunk=96):
        self.n = n
        self.h = P(L.catmsm_basis_create(buf(96 * n), S(n), S(window)))
        assert self.h.value and self.config(window, chunk) == 0
    def config(self, window, chunk):
        return L.catmsm_basis_set_config(self.h, S(window), S(chunk))
    def batch(self, counts, graph, scalars=None):
        return L.catmsm_basis_msm_batch(self.h, buf(144 * len(counts)), S(len(counts)), sizes(counts),
                                        scalars or buf(32 * sum(counts) + 32), 1 if graph else 0)
def done(v):
    print(json.dumps(v))
'''

_fake = None


def _build():
    global _fake
    if _fake is None:
        cuda = os.path.dirname(os.path.dirname(os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")))
        out = os.path.join(tempfile.mkdtemp(prefix="fake_cuda_"), "libfake_cudart.so")
        subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", "-O1", "-shared", "-fPIC",
                        "-I" + os.path.join(cuda, "include"), os.path.join(HERE, "fake_cudart.cpp"), "-o", out],
                       check=True)
        _fake = out
    return _fake


def run(lib_path, body, timeout=120):
    fake = _build()
    env = dict(os.environ, LD_PRELOAD=fake)
    r = subprocess.run([sys.executable, "-c", _PREAMBLE.format(fake=fake, lib=lib_path) + body],
                       capture_output=True, text=True, env=env, timeout=timeout)
    assert r.returncode == 0, r.stderr[-3000:] or r.returncode
    return json.loads(r.stdout.strip().splitlines()[-1])
