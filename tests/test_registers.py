"""Memory and streams of registers: what their device address may be used
for, where the memory of freed ones goes, calls that return with work queued."""
import ctypes as C
import os
import subprocess
import sys
import threading
from pathlib import Path

import numpy as np
import pytest

import yao_rs as Y
from helpers import layered_circuit, random_state
from yao_rs import _abi as A

pytestmark = pytest.mark.gpu


def device_ptr(reg):
    p = C.c_void_p()
    A.check(A.lib().yao_reg_device_ptr(reg.handle, C.byref(p)))
    return p.value


@pytest.mark.parametrize("n", [2, 10, 20, 24])
def test_address_can_be_shared_with_other_processes(n):
    """The address is plain device memory (cudaIpcGetMemHandle takes it), for
    new registers and for ones that reuse memory."""
    get = C.CDLL("libcuda.so.1").cuIpcGetMemHandle
    get.argtypes = [C.c_void_p, C.c_uint64]
    for _ in range(3):
        reg = Y.ArrayReg.zero_state(n)
        handle = (C.c_char * 64)()
        assert get(handle, device_ptr(reg)) == 0
        del reg


def test_memory_of_freed_registers():
    """Reused for registers of the same size in the order of the stream, from
    several threads, and at most 1 GiB of it kept."""
    torch = pytest.importorskip("torch")
    regs = [Y.ArrayReg.zero_state(23) for _ in range(16)]  # 2 GiB
    A.synchronize(0)
    free = torch.cuda.mem_get_info(0)[0]
    del regs
    A.synchronize(0)
    assert torch.cuda.mem_get_info(0)[0] - free >= (1 << 30)
    rng = np.random.default_rng(0)
    states = {n: random_state(rng, n) for n in (3, 12, 16, 20)}
    failed = []

    def work(seed):
        order = np.random.default_rng(seed)
        for _ in range(40):
            n = int(order.choice(list(states)))
            v = states[n] * np.exp(1j * seed)
            a = Y.ArrayReg.from_vec(n, v)
            b = Y.ArrayReg.zero_state(n)
            del b
            if not np.array_equal(a.state_vec(), v):
                failed.append((seed, n))
    threads = [threading.Thread(target=work, args=(t,)) for t in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed


def test_address_on_another_stream():
    """A register freed while another stream still reads its address: the free
    waits for that stream, also where the memory is used again."""
    torch = pytest.importorskip("torch")
    n = 24
    v = random_state(np.random.default_rng(1), n)
    reg = Y.ArrayReg.from_vec(n, v)
    side = torch.cuda.Stream()

    class Amplitudes:
        __cuda_array_interface__ = {"shape": (1 << n,), "typestr": "<c16", "data": (device_ptr(reg), False),
                                    "version": 3, "strides": None}
    src, big = torch.as_tensor(Amplitudes(), device="cuda"), torch.ones(1 << 27, device="cuda")
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        for _ in range(20):
            big.mul_(1.0001)
        got = src.clone()
    del reg
    other = Y.ArrayReg.zero_state(n)
    torch.cuda.synchronize()
    assert np.array_equal(got.cpu().numpy(), v) and other.norm() == 1.0


def test_plain_apply_returns_with_work_queued():
    """PLAIN waits for nothing: one host thread keeps several contexts busy."""
    torch = pytest.importorskip("torch")
    stream = torch.cuda.ExternalStream(A.stream_ptr(0), device=torch.device("cuda", 0))
    n = 27
    c, reg = layered_circuit(n, 4, seed=3), Y.ArrayReg.zero_state(n)
    Y.apply_inplace(c, reg)  # modules loaded, tables allocated
    A.synchronize(0)
    Y.apply_inplace(c, reg)
    assert not stream.query()  # 50 ms and more of work
    assert abs(reg.norm() - 1.0) < 1e-12
    rho = Y.DensityMatrix.from_reg(Y.ArrayReg.zero_state(12))
    layers = layered_circuit(12, 16, seed=4)
    A.synchronize(0)
    rho.apply(layers)
    assert not stream.query()
    assert abs(rho.trace() - 1.0) < 1e-12


def test_registers_of_two_contexts():
    """A mixture and a difference of registers of two contexts wait for the
    work queued on both, and memory freed afterwards is used again only once
    it has been read."""
    lib, n = A.lib(), 11
    ctx = C.c_void_p()
    A.check(lib.yao_ctx_create(0, C.byref(ctx)))
    c = layered_circuit(n, 400, seed=2)  # some milliseconds of work
    ref = Y.ArrayReg.zero_state(n)
    Y.apply_inplace(c, ref)
    want = Y.DensityMatrix.from_reg(ref).state_data().ravel()
    for _ in range(3):
        other, zero, rho = C.c_void_p(), C.c_void_p(), C.c_void_p()
        A.check(lib.yao_reg_zero_state(ctx, n, Y.C128, C.byref(other)))
        A.check(lib.yao_apply_inplace(c.handle, other))
        weights, regs = (C.c_double * 1)(1.0), (C.c_void_p * 1)(other)
        A.check(lib.yao_dm_mixed(A.context(0), weights, regs, 1, C.byref(rho)))
        lib.yao_reg_free(other)
        A.check(lib.yao_reg_zero_state(ctx, n, Y.C128, C.byref(zero)))  # the freed memory
        got = np.zeros(1 << (2 * n), dtype=np.complex128)
        A.check(lib.yao_dm_to_host(rho, got.ctypes.data_as(A.dptr)))
        assert np.max(np.abs(got - want)) < 1e-15
        A.check(lib.yao_apply_inplace(c.handle, zero))
        diff = C.c_double()
        A.check(lib.yao_reg_max_abs_diff(ref.handle, zero, C.byref(diff)))
        assert diff.value == 0.0
        lib.yao_reg_free(zero)
        lib.yao_dm_free(rho)
    A.check(lib.yao_ctx_destroy(ctx))


FULL = """
import ctypes as C
import numpy as np
import yao_rs as Y
from yao_rs import _abi as A
from helpers import layered_circuit, tfim
n, m = 25, 13  # registers of their own allocations
c, op = layered_circuit(n, 1, seed=1), tfim(n)
noisy = Y.Circuit.qubits(m, [Y.channel([q], Y.NoiseChannel.Depolarizing(1, 0.1)) for q in range(4)] * 2)
regs = [Y.ArrayReg.zero_state(n) for _ in range(3)]
rhos = [Y.DensityMatrix.zero_state(m) for _ in range(2)]
for e in c.elements:  # launches of their own, and shared passes: kernels loaded
    Y.apply_inplace(Y.Circuit.qubits(n, [e]), regs[0])
for e in noisy.elements:
    rhos[0].apply(Y.Circuit.qubits(m, [e]))
Y.apply_inplace(c, regs[1])
for x in (Y.OperatorPolynomial([1.0], [Y.OperatorString([(0, Y.Op.P0)])]), op):
    want = Y.expect_arrayreg(regs[1], x)
A.synchronize(0)
cu = C.CDLL("libcuda.so.1")
pool, held = C.c_void_p(), []
assert cu.cuDeviceGetDefaultMemPool(C.byref(pool), 0) == 0 and cu.cuMemPoolTrimTo(pool, C.c_size_t(0)) == 0
size = 64 << 30
while size >= 1 << 10:
    p = C.c_uint64()
    if cu.cuMemAlloc_v2(C.byref(p), C.c_size_t(size)) == 0:
        held.append(p)
    else:
        size //= 2
q = C.c_void_p()
status = A.lib().yao_reg_zero_state(A.context(0), 24, Y.C128, C.byref(q))
Y.apply_inplace(c, regs[2])
rhos[1].apply(noisy)
got = Y.expect_arrayreg(regs[1], op)
for p in held:
    cu.cuMemFree_v2(p)
assert regs[2].max_abs_diff(regs[1]) == 0.0 and abs(got - want) < 1e-12
assert np.array_equal(Y.probs(rhos[1]), Y.probs(rhos[0]))
print(status)
"""


def test_calls_that_need_no_memory_without_memory():
    """PLAIN on states and density matrices and expectation values on a GPU
    whose memory is taken: one launch a gate, a channel, a mask."""
    root = Path(__file__).resolve().parent.parent
    env = dict(os.environ, PYTHONPATH=f"{root / 'yao-rs_b200'}:{root / 'tests'}")
    r = subprocess.run([sys.executable, "-c", FULL], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert int(r.stdout.split()[0]) == A.YAO_ERR_OUT_OF_MEMORY
