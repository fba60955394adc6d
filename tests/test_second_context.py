"""Kernels with more than 48 KB of dynamic shared memory in a second driver context of one process.

The limit is raised per context.  The calls run in a process of their own, which a context more does not disturb.
"""

import pathlib
import subprocess
import sys

import pytest

REPO = pathlib.Path(__file__).resolve().parent.parent

SCRIPT = """
import ctypes, torch, pygrog_b200
lib = pygrog_b200.load_library()
N, KW, K, C = 400000, 8, 3, 1  # chunks of 5,408 replicas: 64 KB of keys
R = N * KW
ns = lib.pgb_grog_expand_chunk(N, C, KW)
assert 4096 < ns * KW <= 8192
dev = torch.device("cuda", 0)
idx = torch.zeros(R, dtype=torch.int64, device=dev)
out = [torch.empty(R, dtype=torch.int32, device=dev) for _ in range(2)]
runs = torch.zeros(1, dtype=torch.int32, device=dev)
for _ in range(2):
    st = lib.pgb_grog_expand_order(idx.data_ptr(), N, KW, K, C, out[0].data_ptr(), out[1].data_ptr(), runs.data_ptr(), None)
    assert st == 0, lib.pgb_last_error()
torch.cuda.synchronize()
want = -(-N // ns)
assert int(runs) == 2 * want  # one operator: a run a chunk
cu = ctypes.CDLL("libcuda.so.1")
def do(name, *a):
    assert getattr(cu, name)(*a) == 0, name
ctx, dv = ctypes.c_void_p(), ctypes.c_int()
do("cuDeviceGet", ctypes.byref(dv), 0)
do("cuCtxCreate_v2", ctypes.byref(ctx), 0, dv)
mem = [ctypes.c_uint64() for _ in range(4)]
for m, n in zip(mem, (8 * R, 4 * R, 4 * R, 4)):
    do("cuMemAlloc_v2", ctypes.byref(m), ctypes.c_size_t(n))
    do("cuMemsetD8_v2", m, ctypes.c_ubyte(0), ctypes.c_size_t(n))
do("cuCtxSynchronize")
st = lib.pgb_grog_expand_order(mem[0].value, N, KW, K, C, mem[1].value, mem[2].value, mem[3].value, None)
assert st == 0, lib.pgb_last_error()
do("cuCtxSynchronize")
got = ctypes.c_int32()
do("cuMemcpyDtoH_v2", ctypes.byref(got), mem[3], ctypes.c_size_t(4))
assert got.value == want, (got.value, want)
for m in mem:
    do("cuMemFree_v2", m)
do("cuCtxDestroy_v2", ctx)
runs.zero_()  # and the first context again
st = lib.pgb_grog_expand_order(idx.data_ptr(), N, KW, K, C, out[0].data_ptr(), out[1].data_ptr(), runs.data_ptr(), None)
assert st == 0, lib.pgb_last_error()
assert int(runs) == want
print("done")
"""


@pytest.mark.gpu
def test_large_shared_memory_in_a_second_context(cuda):
    r = subprocess.run([sys.executable, "-c", SCRIPT], cwd=REPO, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "done" in r.stdout, r.stderr[-2000:]
