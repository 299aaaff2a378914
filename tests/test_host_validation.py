"""Host-side argument checks of the Python mirror (no GPU needed): what the kernels would misread on
the device - a page table of the wrong dtype, on the wrong device or strided - is refused before any
launch, because a bad index on the GPU is an out-of-bounds read rather than an exception."""
import os
import subprocess
import sys
import textwrap
import threading

import pytest
import torch

from amd_optimization_challenge_b200 import submission as sub

CPU = torch.device("cpu")
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_index_tensor_checks():
    ok = torch.arange(9, dtype=torch.int32)
    sub._check_index_tensor("kv_indptr", ok, CPU, 2)
    sub._check_index_tensor("kv_indices", None, CPU)                       # optional arguments may be absent
    with pytest.raises(TypeError, match="int32"):
        sub._check_index_tensor("kv_indices", torch.arange(9), CPU)       # torch.arange defaults to int64
    with pytest.raises(TypeError, match="torch.Tensor"):
        sub._check_index_tensor("kv_indices", [0, 1, 2], CPU)
    with pytest.raises(ValueError, match="contiguous"):
        sub._check_index_tensor("kv_indices", torch.arange(18, dtype=torch.int32)[::2], CPU)
    with pytest.raises(ValueError, match="is on"):
        sub._check_index_tensor("kv_indices", torch.empty(9, dtype=torch.int32, device="meta"), CPU)
    with pytest.raises(ValueError, match="at least 10"):
        sub._check_index_tensor("kv_indices", ok, CPU, 10)


def test_plane_checks():
    sub._check_plane("kv[0]", torch.zeros(4, 1, 576, dtype=torch.uint8), CPU)
    sub._check_plane("scale", torch.zeros(1), CPU, torch.float32)
    with pytest.raises(TypeError, match="float32"):
        sub._check_plane("scale", torch.zeros(1, dtype=torch.float64), CPU, torch.float32)
    with pytest.raises(ValueError, match="unit stride"):
        sub._check_plane("kv[0]", torch.zeros(4, 576, dtype=torch.uint8).t(), CPU)
    with pytest.raises(ValueError, match="is on"):
        sub._check_plane("kv[0]", torch.empty(4, 576, dtype=torch.uint8, device="meta"), CPU)


def test_decode_refuses_cpu_tensors():
    q = torch.zeros(1, 16, 576, dtype=torch.bfloat16)
    with pytest.raises(RuntimeError, match="no CPU path"):
        sub.mla_decode(q, None, "fp8", (torch.zeros(4, 576, dtype=torch.uint8), torch.ones(1)),
                       torch.tensor([0, 4], dtype=torch.int32), sm_scale=1.0)


def test_generator_device_default_is_cpu_and_seeded():
    import amd_optimization_challenge_b200 as pkg
    a = pkg.generate_input(2, 1, 8, seed=3, formats=("fp8",), device="cpu")
    b = pkg.generate_input(2, 1, 8, seed=3, formats=("fp8",), device="cpu", generator_device="cpu")
    assert torch.equal(a[0], b[0]) and torch.equal(a[1]["fp8"][0].view(torch.uint8), b[1]["fp8"][0].view(torch.uint8))


def test_signature_sees_storage_and_shape():
    from amd_optimization_challenge_b200._host import signature
    t = torch.zeros(6, 4)
    old = t.detach()
    first = signature([t, None])
    assert first == signature((t, None)) != signature((t,))
    for change in (lambda: t.as_strided_((6, 2), (4, 1)), lambda: t.as_strided_((6, 2), (2, 1)), lambda: t.resize_(5, 2),
                   lambda: setattr(t, "data", torch.zeros(5, 2)), lambda: setattr(t, "data", torch.zeros(5, 2, dtype=torch.int32))):
        before = signature([t])
        change()
        assert signature([t]) != before
    assert signature([old, None]) == first
    with pytest.raises(RuntimeError):
        signature([torch.zeros(3, 3).to_sparse()])


def test_append_of_a_tensor_without_strides_raises():
    """Tensors that answer questions about themselves in Python, and may refuse: an exception, not the end of the process."""
    code = textwrap.dedent("""
        import torch
        from amd_optimization_challenge_b200 import submission as sub
        class T(torch.Tensor):
            @staticmethod
            def __new__(cls, shape, dtype):
                return torch.Tensor._make_wrapper_subclass(cls, shape, dtype=dtype, device="cuda", dispatch_sizes_strides_policy="strides")
            @classmethod
            def __torch_dispatch__(cls, f, types, args=(), kwargs=None):
                raise NotImplementedError("no strides")
        planes = T((9, 576), torch.uint8), T((1,), torch.float32)
        for call in (lambda: sub.kv_append(T((4, 576), torch.bfloat16), "fp8", planes), lambda: sub._host.signature(planes)):
            try:
                call()
            except NotImplementedError as e:
                print("RAISED", e)
    """)
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, cwd=ROOT)
    assert r.returncode == 0 and r.stdout.count("RAISED no strides") == 2, r.stdout + r.stderr


@pytest.mark.parametrize("base", [3.0, torch.tensor(3), 1 << 70])
def test_append_takes_what_int_takes_as_base_slot(base):
    with pytest.raises(ValueError, match="CUDA"):                # the rows are refused, not the slot
        sub.kv_append(torch.zeros(2, 576, dtype=torch.bfloat16), "fp8", (torch.zeros(9, 576, dtype=torch.uint8), torch.ones(1)), base_slot=base)


def test_remembering_replaces_and_evicts():
    cache = {i: i for i in range(4)}
    sub._remember(cache, 2, "new", limit=4)                      # a key that is there: nothing else leaves, and it is the newest
    assert cache == {0: 0, 1: 1, 3: 3, 2: "new"}
    for i in (7, 8, 9):
        sub._remember(cache, i, i, limit=4)
    assert list(cache) == [2, 7, 8, 9]


def test_plan_caches_with_threads(monkeypatch):
    """Calls of one tensor set with changing numbers, from threads that make each other's plans stale."""
    class Q:                                                     # what mla_decode looks at before it comes to the plan
        is_cuda = True
    q, ip = Q(), Q()
    plans = {}
    monkeypatch.setattr(sub, "_decode_plans", plans)

    class Stale:
        signature = refs = ()
        @property
        def scalars(self):                                       # another thread takes the plan out while this one looks at it
            plans.clear()
            return ()
    plans[(id(q), id(ip), id(None), "fp8", False)] = Stale()
    with pytest.raises(AttributeError):                          # past the plans, on to the arguments
        sub.mla_decode(q, None, "fp8", (), ip, sm_scale=1.0)
    cache, errors = {}, []

    def work(n):
        try:
            for i in range(20000):
                sub._remember(cache, (n, i % 50), i, limit=8)
                cache.pop((1 - n, i % 50), None)
        except Exception as e:
            errors.append(e)
    threads = [threading.Thread(target=work, args=(n,)) for n in (0, 1)]
    old = sys.getswitchinterval()
    sys.setswitchinterval(1e-6)
    [t.start() for t in threads]
    [t.join() for t in threads]
    sys.setswitchinterval(old)
    assert not errors


def test_append_arguments_of_the_c_entry():
    """What the reserved word holds does not matter; the flag that asks for the status word is part of kv_format."""
    from amd_optimization_challenge_b200 import _cabi
    a = _cabi.KvAppendArgs(rows_bf16=4096, n=3, row_stride=576, num_slots=10, kv_codes=4096, kv_codes_stride=576, base_slot=8, reserved=0x5A5A5A5A)
    for fmt, error in ((0, b"kv_scale"), (1, b"kv_block_scales"), (2, b"kv_scale"), (3, b"kv_format"), (256, b"status word"), (512, b"kv_format"), (-1, b"kv_format")):
        a.kv_format = fmt
        assert _cabi.lib.b200_mla_kv_append(a, None) == -1 and error in _cabi.lib.b200_mla_last_error(), fmt
    a.kv_format, a.kv_scale = 0, 4096
    for base in (-1, 8, 10, (1 << 63) - 1):                      # the last one plus three rows is negative in 64 bits
        a.base_slot = base
        assert _cabi.lib.b200_mla_kv_append(a, None) == -1 and b"do not fit" in _cabi.lib.b200_mla_last_error()
    a.kv_format, a.n = 0, 0
    assert _cabi.lib.b200_mla_kv_append(a, None) == 0
