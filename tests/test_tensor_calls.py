"""The native look at the tensors of a call: what it takes gives the results of the general path, what it leaves is answered there."""
import os
import sys

import pytest
import torch

gpu = pytest.mark.gpu


def test_cpu_tensors_are_left_to_the_general_path():
    from unified_ccl_b200.communicator import tensor_calls
    from unified_ccl_b200.ops import gemm_bf16

    x = torch.zeros(8, 8, dtype=torch.bfloat16)
    for taken in (tensor_calls.gemm(x, x, x, False), tensor_calls.norm(1, 0, x, x, x, 1e-6, x, x), tensor_calls.reduce_scatter(1, -1, 1, x, x),
                  tensor_calls.allgather(1, -1, 1, x, x), tensor_calls.allreduce_cast(1, -1, 1, x, x, 1.0, None),
                  tensor_calls.moe_dispatch(1, 0, 8, 8, x, x), tensor_calls.moe_combine(1, 0, 8, 8, 8, x, x), tensor_calls.gemm(),
                  tensor_calls.gemm(1, 2, 3, 4), tensor_calls.norm(2 ** 70, 0, x, x, x, 1e-6, x, x), tensor_calls.reduce_scatter(1, 2 ** 70, 1, x, x)):
        assert not taken
    with pytest.raises(ValueError):
        gemm_bf16(x, x, out=x)


class Sub(torch.Tensor):
    pass


@gpu
def test_taken_calls_equal_the_general_path(monkeypatch):
    os.environ.setdefault("UCCL_BOOTSTRAP_IFNAME", "lo")
    from unified_ccl_b200 import Communicator, communicator, ops
    from unified_ccl_b200.parallel import MoeDispatcher, allreduce_residual_rmsnorm

    native = communicator.tensor_calls
    assert native.__name__.endswith("_uccl_tensor_calls")
    users = [sys.modules["unified_ccl_b200." + m] for m in ("communicator", "ops.gemm", "parallel.tp", "parallel.moe")]
    comm = Communicator(0, 1)
    disp = MoeDispatcher(comm, 16, 256, 8, 2)
    g = torch.Generator(device="cuda").manual_seed(1)
    bf = lambda *s: torch.randn(*s, device="cuda", generator=g).to(torch.bfloat16)  # noqa: E731
    a, b, x, res, gamma = bf(16, 256), bf(64, 256), bf(16, 256), bf(16, 256), bf(256)
    idx = torch.randint(0, 8, (16, 2), device="cuda", generator=g, dtype=torch.int32)
    w = torch.rand(16, 2, device="cuda", generator=g)
    f32 = torch.randn(4096, device="cuda", generator=g)
    empty = lambda t, *s, dtype=None: torch.zeros(*(s or t.shape), device="cuda", dtype=dtype or t.dtype)  # noqa: E731
    fp8, fp16 = torch.float8_e4m3fn, torch.float16

    def norm(*t, **k):
        return allreduce_residual_rmsnorm(comm, *t, **k)

    def dispatch(t=x, i=idx):
        rows, scales, meta, counts = disp.dispatch(t, i)
        order = (meta[0, :, 0] * 2 + meta[0, :, 2]).argsort()
        return rows[0].view(torch.uint8)[order], scales[0][order], counts.clone()

    def combine(t=w, out=None):
        disp.dispatch(x, idx)
        disp.expert_out[0, :, :] = (disp.recv_meta[0, :, :1] * 2 + disp.recv_meta[0, :, 2:3]).to(torch.bfloat16)
        return disp.combine(t, out=empty(x) if out is None else out)

    taken = [
        lambda: ops.gemm_bf16(a, b, out=empty(a, 16, 64)), lambda: ops.gemm_bf16(a, b, out=empty(a, 16, 32), swiglu=True),
        lambda: ops.gemm_bf16(a[:, 8:136], b[:, 8:136], out=empty(a, 16, 80)[:, :64]),  # strides of their own
        lambda: norm(x, res.clone(), gamma, 1e-6, out=empty(x)), lambda: norm(x, res, gamma, out=empty(x), residual_out=empty(x)),
        lambda: comm.reduce_scatter(f32, empty(f32)), lambda: comm.allgather(f32.to(fp8), empty(f32, dtype=fp8)).view(torch.uint8),
        lambda: comm.reduce_scatter_cast(f32, empty(f32, dtype=fp16), 0.5)[0],
        lambda: comm.allreduce_cast(f32, empty(f32, dtype=fp8), 0.5, scales=empty(f32, 32))[1], dispatch, combine,
    ]
    left = [  # answered, or refused, as ever
        lambda: ops.gemm_bf16(a.as_subclass(Sub), b, out=empty(a, 16, 64)).as_subclass(torch.Tensor), lambda: ops.gemm_bf16(a, b, out=empty(a, 16, 32), swiglu=1),
        lambda: ops.gemm_bf16(a, b), lambda: ops.gemm_bf16(a.t(), b, out=empty(a, 16, 64)), lambda: ops.gemm_bf16(a, b, out=empty(a, 16, 63)),
        lambda: ops.gemm_bf16(a, b, out=empty(a, 64, 16).t()), lambda: ops.gemm_bf16(a.half(), b, out=empty(a, 16, 64)),
        lambda: ops.gemm_bf16(a[:, 1:129], b[:, :128], out=empty(a, 16, 64)), lambda: ops.gemm_bf16(a, b[:, :128], out=empty(a, 16, 64)),
        lambda: norm(x.t(), res, gamma, out=empty(x)), lambda: norm(x[0], res, gamma, out=empty(x)), lambda: norm(x.half(), res, gamma, out=empty(x)),
        lambda: norm(x, res, gamma, 0, out=empty(x), residual_out=empty(x)), lambda: norm(x, res, gamma, residual_out=empty(x)),
        lambda: comm.reduce_scatter(f32, empty(f32, 2048)), lambda: comm.reduce_scatter(f32, empty(f32, dtype=fp16)),
        lambda: comm.reduce_scatter(f32.int(), f32.int()), lambda: comm.reduce_scatter(f32[::2], empty(f32, 2048)),
        lambda: comm.reduce_scatter(f32, empty(f32), op="max"), lambda: comm.allgather(f32, f32.cpu()), lambda: comm.allgather(f32.long(), f32.long()),
        lambda: comm.reduce_scatter_cast(f32, empty(f32, dtype=torch.uint8)), lambda: comm.reduce_scatter_cast(f32[:100], empty(f32, 100, dtype=fp8)),
        lambda: comm.allreduce_cast(f32, empty(f32, dtype=fp8), scales=empty(f32, 31)), lambda: comm.allreduce_cast(f32, empty(f32, dtype=fp8), 2)[1],
        lambda: comm.allreduce_cast(f32, empty(f32, dtype=fp16), scales=empty(f32, 32))[0], lambda: comm.reduce_scatter_cast(f32[1:129], empty(f32, 128), 2.0)[0],
        lambda: dispatch(x.half()), lambda: dispatch(x, idx.long()), lambda: dispatch(x, idx[:, :1]), lambda: combine(w[:, :1]), lambda: combine(w.half()),
        lambda: combine(out=empty(x, 16 * 256)).view(16, 256),
    ]

    def answer(f):
        try:
            r = f()
        except Exception as e:
            return type(e), str(e)
        torch.cuda.synchronize()
        return [t.clone() for t in (r if isinstance(r, tuple) else (r,))]

    for i, f in enumerate(taken + left):
        for u in users:
            monkeypatch.setattr(u, "tensor_calls", communicator._GeneralPath)
        want = answer(f)
        for u in users:
            monkeypatch.setattr(u, "tensor_calls", native)
        got = answer(f)
        if isinstance(want, tuple):
            assert i >= len(taken) and got == want, (i, want, got)
        else:
            assert not isinstance(got, tuple), (i, got)
            assert len(got) == len(want) and all(torch.equal(p, q) for p, q in zip(got, want)), i
    # with the general path out of reach: these calls are taken
    for u in users:
        monkeypatch.setattr(u, "_C", None)
    for i, f in enumerate(taken):
        assert not isinstance(answer(f), tuple), (i, answer(f))
    monkeypatch.undo()
    gone = Communicator(0, 1)
    gone.destroy()
    with pytest.raises(RuntimeError):
        gone.reduce_scatter(f32, f32)
    disp.close()
    comm.destroy()


@pytest.mark.parametrize("name,value", [("__version__", "2.10.0+cu128"), ("git_version", "0" * 40)])
def test_module_of_another_torch_is_not_loaded(name, value):
    """Into a torch other than the one that it was built for the native module does not load, and says so once."""
    import subprocess

    code = (f"import warnings, torch; torch.version.{name} = {value!r}\n"
            "with warnings.catch_warnings(record=True) as w:\n"
            "    warnings.simplefilter('always')\n"
            "    from unified_ccl_b200 import communicator\n"
            "assert communicator.tensor_calls is communicator._GeneralPath\n"
            f"assert len(w) == 1 and {value!r} in str(w[0].message), [str(x.message) for x in w]\n"
            "assert 'unified_ccl_b200._uccl_tensor_calls' not in __import__('sys').modules\n")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    p = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr[-2000:]
