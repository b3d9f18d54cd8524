"""The operators' native call path and the Python checks take the same calls, with the same result, and refuse alike."""
import ctypes

import pytest
import torch

from oracle import attention as oracle
from tilecadence_b200 import cuda_runtime


def test_native_path_declines_what_it_cannot_take():
    """Tensors of the host, wrong counts and wrong types: declined with a number, never an exception or a crash."""
    native = cuda_runtime.fast_call()
    if native is None:
        pytest.skip("torch without CUDA")
    x = torch.zeros(1, 1, 32, 128, dtype=torch.bfloat16)
    assert native.decode(1, 32, *([x] * 10), 0, 1, True, 0) == -1
    assert native.prefill(1, 32, *([x] * 7), 0, 1, 0.1, True) == -1
    assert native.exchange(1, *([x] * 5), False) == -1
    for name in ("decode", "rope", "indexed", "prefill", "key_split", "exchange"):
        assert getattr(native, name)() == -1
        assert getattr(native, name)(*([None] * 17)) == -1
        assert getattr(native, name)(*(["x"] * 16)) == -1


@pytest.mark.parametrize("fault", ["no compiler", "compiler fails", "broken library"])
def test_operators_work_without_the_native_path(monkeypatch, tmp_path, fault):
    """Where the native path can be neither found nor built, the operators say so once and go through their checks."""
    if cuda_runtime.fast_call() is None:
        pytest.skip("torch without CUDA")
    library = next(cuda_runtime.BUILD_DIR.glob("tc_fast_call_*.so"))
    monkeypatch.setattr(cuda_runtime, "BUILD_DIR", tmp_path)
    if fault == "no compiler":
        monkeypatch.setattr(cuda_runtime.shutil, "which", lambda name: None)
    elif fault == "compiler fails":
        monkeypatch.setattr(cuda_runtime.subprocess, "run",
                            lambda *a, **k: cuda_runtime.subprocess.CompletedProcess(a, 1, "", "no headers"))
    else:
        for path in cuda_runtime.PACKAGE_ROOT.glob(f"_build/{library.name[:13]}*.so"):
            (tmp_path / path.name).write_bytes(b"not a library")

    class Prebuilt:
        addresses = {"tc_decode_forward_out_flags": 1}

        def has(self, prefix):
            return prefix == "tc_decode_"

    x = torch.zeros(1, 1, 32, 128, dtype=torch.bfloat16)
    cuda_runtime.fast_call.cache_clear()
    try:
        with pytest.warns(RuntimeWarning, match="checks in Python") as said:
            ops = cuda_runtime.ops_for(Prebuilt())
            for _ in range(2):
                with pytest.raises(RuntimeError, match="must be CUDA on the same device"):
                    ops.forward_out(*([x] * 10), 0, 1, True)
        assert len(said) == 1
    finally:
        cuda_runtime.fast_call.cache_clear()


def test_nothing_of_a_tensor_is_read_without_the_interpreter_lock():
    """Another thread may resize a tensor as soon as the lock is released: what the launch gets are numbers read before."""
    source = (cuda_runtime.PACKAGE_ROOT / "host" / "fast_call.cpp").read_text()
    released = source.split("Py_BEGIN_ALLOW_THREADS")[1:]
    assert len(released) == 1 and released[0].split("Py_END_ALLOW_THREADS")[0].split() == ["status", "=", "function(arguments...);"]
    assert "without_gil([" not in source  # a closure would read its captures after the release


def decode_state(device, batch=2, capacity=256):
    q, k, v, knew, vnew = (t.to(device) for t in oracle.seeded_normal(
        5, (batch, 1, 32, 128), (batch, capacity, 8, 128), (batch, capacity, 8, 128), (batch, 1, 8, 128), (batch, 1, 8, 128)))
    old = torch.arange(100, 100 + batch, dtype=torch.int32, device=device)
    ops = cuda_runtime.default_ops("decode")
    spec = ops.workspace_spec(q, k, old, 0, 1, True)
    results = [torch.empty_like(q), torch.empty((batch, 32, 1), device=device)]
    workspace = [torch.empty(n, device=device) for n in spec[1:]]
    return ops, [q, k, v, knew, vnew, old, *results, *workspace, 0, 1, True]


def calls(device, made_by=cuda_runtime.default_ops):
    """Operator, arguments and results of one call each; the operator objects called come from ``made_by``."""
    _, args = decode_state(device)
    ops = made_by("decode")
    table = torch.arange(8, dtype=torch.int32, device=device).view(2, 4)
    pages = [args[0], args[1].view(8, 64, 8, 128), args[2].view(8, 64, 8, 128), *args[3:]]
    cos = torch.rand(256, 64, device=device)
    q, k, v = (t.to(device) for t in oracle.seeded_normal(6, (1, 300, 32, 128), (1, 300, 8, 128), (1, 300, 8, 128)))
    prefill, out, lse = made_by("prefill"), torch.empty_like(q), torch.empty((1, 32, 300), device=device)
    none = torch.empty(0, device=device)
    split = torch.empty(cuda_runtime.default_ops("prefill").key_split_workspace_bytes(q), dtype=torch.uint8, device=device)
    tq = torch.randn(1, 64, 8, 128, device=device, dtype=torch.float16)
    two = made_by("exchange")
    return {
        "decode": (ops.forward_out, args, args[6:8]),
        "indexed": (lambda *a: ops.indexed_forward_out(*a, block_table=table), pages, args[6:8]),
        "rope": (lambda *a: ops.rope_forward_out(*a, cos, cos), args, args[6:8]),
        "prefill": (prefill.forward_out, [q, k, v, out, lse, none, none, 0, 1, 128 ** -0.5, True], [out, lse]),
        "key_split": (prefill.key_split_forward_out, [q, k, v, out, lse, split, 1, 128 ** -0.5, 2], [out, lse]),
        "exchange": (two.forward_out, [tq, tq.clone(), tq.clone(), torch.empty_like(tq),
                                       torch.empty(1, 8, 64, device=device), None, False], None),
    }


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["decode", "indexed", "rope", "prefill", "key_split", "exchange"])
def test_both_paths_agree(gpu_device, monkeypatch, name):
    call, args, results = calls(gpu_device)[name]
    results = args[3:5] if results is None else results
    native, taken = cuda_runtime.fast_call(), []

    class Recording:
        def __getattr__(self, operator):
            return lambda *a: taken.append(getattr(native, operator)(*a)) or taken[-1]

    monkeypatch.setattr(cuda_runtime, "fast_call", lambda: Recording())
    call(*args)
    assert taken == ([2] if name == "key_split" else [0])  # the native path made the call
    got = [t.clone() for t in results]
    monkeypatch.setattr(cuda_runtime, "fast_call", lambda: None)
    call(*args)
    torch.cuda.synchronize()
    for a, b in zip(got, results):
        assert torch.allclose(a, b, atol=1e-2) if name == "key_split" else torch.equal(a, b)
    # A tensor that the checks refuse is refused with the same words either way: one at a time, another type, a
    # longer last dimension's stride, autograd.
    for index, tensor in enumerate(args):
        if not isinstance(tensor, torch.Tensor) or not tensor.numel():
            continue
        bad = [tensor.to(torch.float64), torch.stack([tensor, tensor], -1)[..., 0]]
        if tensor.is_floating_point():
            bad.append(tensor.clone().requires_grad_())
        for wrong in bad:
            messages = []
            for path in (native, None):
                monkeypatch.setattr(cuda_runtime, "fast_call", lambda: path)
                changed = list(args)
                changed[index] = wrong
                try:
                    call(*changed)
                    messages.append("")
                except RuntimeError as error:
                    messages.append(str(error))
            assert messages[0] == messages[1]
    torch.cuda.synchronize()


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["decode", "indexed", "rope", "prefill", "key_split", "exchange"])
def test_both_paths_refuse_alike(gpu_device, monkeypatch, name):
    """Tensors of another device, of another shape (one entry more in the first dimension) and with a base that is not
    aligned, one at a time: both paths take the call or refuse it with the same words. All of them are refused on the
    host where a kernel could not take them."""
    call, args, _ = calls(gpu_device)[name]
    native, refused = cuda_runtime.fast_call(), 0
    for index, tensor in enumerate(args):
        if not isinstance(tensor, torch.Tensor) or not tensor.numel():
            continue
        shifted = torch.empty(tensor.numel() + 1, dtype=tensor.dtype, device=gpu_device)[1:].view(tensor.shape)
        longer = torch.cat([tensor, tensor[:1]])
        for wrong in (tensor.cpu(), longer, shifted.copy_(tensor)):
            messages = []
            for path in (native, None):
                monkeypatch.setattr(cuda_runtime, "fast_call", lambda: path)
                changed = list(args)
                changed[index] = wrong
                try:
                    call(*changed)
                    messages.append("")
                except RuntimeError as error:
                    messages.append(str(error))
            assert messages[0] == messages[1], (index, messages)
            refused += messages[0] != ""
        torch.cuda.synchronize()
    assert refused >= 2 * 5  # at least the five leading tensors, on another device and of another shape


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["decode", "indexed", "rope", "prefill", "key_split", "exchange"])
def test_a_call_that_fails_in_the_entry_point_is_made_once(gpu_device, name):
    """An error of the C ABI is raised from the native path; the call is not made again through ctypes. The entry point
    here is a stand-in that counts and launches nothing."""
    made = []
    stand_in = ctypes.CFUNCTYPE(ctypes.c_int)(lambda: made.append("native") or 2)
    real = cuda_runtime.default_library()

    class Failing:
        path, handle, symbols, fail, call = real.path, real.handle, real.symbols, cuda_runtime.Library.fail, cuda_runtime.Library.call
        addresses = dict.fromkeys(real.addresses, ctypes.cast(stand_in, ctypes.c_void_p).value)
        functions = dict.fromkeys(real.functions, lambda *a: made.append("ctypes") or 2)

    operator, args, _ = calls(gpu_device, lambda phase: cuda_runtime.ops_for(Failing(), phase))[name]
    with pytest.raises(RuntimeError, match=r"^tc_[a-z_]*_out: .*status 2"):
        operator(*args)
    assert made == ["native"]


@pytest.mark.gpu
def test_native_path_launches_on_the_current_stream(gpu_device):
    ops, args = decode_state(gpu_device)
    graph = torch.cuda.CUDAGraph()
    stream = torch.cuda.Stream(gpu_device)
    ops.forward_out(*args)
    torch.cuda.synchronize()
    want = args[6].clone()
    with torch.cuda.graph(graph, stream=stream):  # a launch on another stream would not be captured
        ops.forward_out(*args)
    args[6].zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(args[6], want)
