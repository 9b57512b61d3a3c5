"""GPU: the two bindings of the op surface - the torch extension `_C` (LibTorch stable ABI, the reference's
mechanism: csrc/reg.cpp:21-33, csrc/cuda/reg.cu:16-27) and the ctypes one - reach the same C ABI and give
the same bits; the extension's ops pass torch.library.opcheck."""
import os
import subprocess
import sys

import pytest
import torch

from conftest import PKG_ROOT, ROOT
from _util import check_close
from oracle import oracle as O

pytestmark = pytest.mark.gpu

_SCRIPT = r"""
import sys, torch
sys.path.insert(0, {pkg!r}); sys.path.insert(0, {root!r})
from minfer.kernels import KernelBackend
from minfer.kernels.torch_ext import ops
assert ops.BINDING == {binding!r}, ops.BINDING
kerns = KernelBackend("torch_ext")
g = torch.Generator().manual_seed(11)
q = torch.randn(2, 6, 300, 128, generator=g).half().cuda()
k = torch.randn(2, 2, 300, 128, generator=g).half().cuda()
v = torch.randn(2, 2, 300, 128, generator=g).half().cuda()
mask = (torch.rand(2, 1, 300, 300, generator=g) < 0.5).cuda()
lens = torch.tensor([300, 17], dtype=torch.int32).cuda()
o1, o2, o3 = torch.zeros_like(q), torch.zeros_like(q), torch.zeros(2, 6, 1, 128, dtype=torch.float16, device="cuda")
kerns.flash_attn_causal(q, k, v, o1)
kerns.flash_attn(1, 1, 2, q, k, v, mask, o2)
kerns.flash_attn_decode(q[:, :, :1].contiguous(), k, v, lens, o3)
with ops.prefill_cta_limit(7):
    o4 = torch.zeros_like(q)
    kerns.flash_attn_causal(q, k, v, o4)
ops.check_status()
torch.save([o1.cpu(), o2.cpu(), o3.cpu(), o4.cpu()], {out!r})
"""


def _run(binding, out):
    env = dict(os.environ, MINFER_ATTN_BINDING=binding)
    script = _SCRIPT.format(pkg=PKG_ROOT, root=ROOT, binding=binding, out=out)
    r = subprocess.run([sys.executable, "-c", script], env=env, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    return torch.load(out)


def test_stable_abi_extension_and_ctypes_binding_agree(tmp_path):
    from minfer.kernels.torch_ext import ops
    assert os.path.exists(os.path.join(PKG_ROOT, "minfer", "kernels", "torch_ext", "_C.abi3.so")), "the torch extension was not built"
    assert ops.BINDING == "stable", "the extension is present but the ops did not bind to it"
    a = _run("stable", str(tmp_path / "stable.pt"))
    b = _run("ctypes", str(tmp_path / "ctypes.pt"))
    for x, y in zip(a, b):
        assert torch.equal(x, y)
    assert torch.equal(a[0], a[3])
    g = torch.Generator().manual_seed(11)
    q = torch.randn(2, 6, 300, 128, generator=g).half()
    k = torch.randn(2, 2, 300, 128, generator=g).half()
    v = torch.randn(2, 2, 300, 128, generator=g).half()
    check_close(a[0], O.prefill_oracle(q, k, v, causal=True), "extension, causal")


def test_opcheck_on_the_extension_ops(kerns):
    g = torch.Generator().manual_seed(3)
    q = torch.randn(1, 4, 128, 64, generator=g).half().cuda()
    k = torch.randn(1, 2, 128, 64, generator=g).half().cuda()
    v = torch.randn(1, 2, 128, 64, generator=g).half().cuda()
    out = torch.zeros_like(q)
    lens = torch.tensor([100], dtype=torch.int32, device="cuda")
    torch.library.opcheck(torch.ops.minfer.flash_attn_decode.default, (q[:, :, :1].contiguous(), k, v, lens, out[:, :, :1].contiguous()),
                          test_utils=("test_schema", "test_faketensor"))
    pages = torch.randn(8, 2, 16, 64, generator=g).half().cuda()
    table = torch.arange(8, dtype=torch.int32, device="cuda").view(1, 8)
    torch.library.opcheck(torch.ops.minfer.flash_attn_decode_paged.default,
                          (q[:, :, :1].contiguous(), pages, pages.clone(), table, lens, out[:, :, :1].contiguous()),
                          test_utils=("test_schema", "test_faketensor"))


def test_extension_argument_errors_are_runtime_errors(kerns):
    q = torch.zeros(1, 4, 128, 128, dtype=torch.float16, device="cuda")
    k = torch.zeros(1, 2, 128, 128, dtype=torch.float16, device="cuda")
    with pytest.raises(RuntimeError):
        kerns.flash_attn_causal(q, k, k[:, :, :64], torch.zeros_like(q))          # k/v shapes differ
    with pytest.raises(RuntimeError):
        kerns.flash_attn_causal(q, k, k, torch.zeros(1, 4, 128, 64, dtype=torch.float16, device="cuda"))
    with pytest.raises(RuntimeError):
        kerns.flash_attn_decode(q[:, :, :1], k, k, torch.zeros(1, dtype=torch.int64, device="cuda"), torch.zeros_like(q[:, :, :1]))


def _op_calls():
    """Arguments of one small call per op (fresh tensors, the same values every time) and which of them it writes."""
    g = torch.Generator().manual_seed(21)
    r = lambda *s: torch.randn(*s, generator=g).half().cuda()  # noqa: E731
    B, H, Hkv, L, D, page = 2, 4, 2, 48, 64, 16
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")  # noqa: E731
    q, k, v, qd = r(B, H, L, D), r(B, Hkv, L, D), r(B, Hkv, L, D), r(B, H, 1, D)
    q8 = [O.q8_0_quantize(torch.randn(B, Hkv, L, D, generator=g).half()).cuda() for _ in range(2)]
    pools, table, lens = [r(6, Hkv, page, D) for _ in range(2)], i32([[5, 0, 2], [1, 4, 3]]), i32([48, 17])
    mask = (torch.rand(B, 1, L, L, generator=g) < 0.5).cuda()
    tok, kt, vt = r(B, 3, H, D), r(B, 3, Hkv, D), r(B, 3, Hkv, D)
    return {
        "flash_attn": ([1, 1, 2, q, k, v, mask, torch.zeros_like(q)], [7]),
        "flash_attn_causal": ([q, k, v, torch.zeros_like(q)], [3]),
        "flash_attn_decode": ([qd, k, v, lens, torch.zeros_like(qd)], [4]),
        "flash_attn_decode_q8": ([qd, *q8, lens, torch.zeros_like(qd)], [4]),
        "flash_attn_decode_paged": ([qd, *pools, table, lens, torch.zeros_like(qd)], [5]),
        "il_rope": ([D, 7, 10000.0, tok], [3]),
        "neox_rope": ([D, 7, 10000.0, tok], [3]),
        "rope_kv_append": ([D, 10000.0, 1, tok, kt, vt, k, v, i32([0, 40])], [3, 6, 7]),
        "rope_kv_append_q8": ([D, 10000.0, 0, tok, kt, vt, *q8, i32([0, 40])], [3, 6, 7]),
        "rope_kv_append_paged": ([D, 10000.0, 0, tok, kt, vt, *pools, table, i32([0, 40])], [3, 6, 7]),
    }


@pytest.mark.parametrize("name", ["flash_attn", "flash_attn_causal", "flash_attn_decode", "flash_attn_decode_q8", "flash_attn_decode_paged",
                                  "il_rope", "neox_rope", "rope_kv_append", "rope_kv_append_q8", "rope_kv_append_paged"])
def test_direct_entry_point_gives_the_bits_of_the_dispatched_op(name):
    from minfer.kernels.torch_ext import ops
    assert ops._direct is not None, "the direct entry points were not built"
    a, written = _op_calls()[name]
    b, _ = _op_calls()[name]
    assert getattr(ops._direct, name)(*a) is True
    getattr(torch.ops.minfer, name).default(*b)
    for i in written:
        assert torch.equal(a[i], b[i]), f"{name}: argument {i}"


def test_direct_entry_points_leave_everything_unusual_to_the_dispatcher(kerns):
    """Wrong arguments, autograd, modes and tracers: the direct call declines (and writes nothing), the façade behaves as the op."""
    from torch.utils._python_dispatch import TorchDispatchMode
    from minfer.kernels.torch_ext import ops
    f = ops._direct.flash_attn_decode
    q, k, v, lens, out = _op_calls()["flash_attn_decode"][0]
    out.fill_(7.0)
    assert f(q, k, v, lens.long(), out) is False and f(q, k, v, lens, out[..., :32]) is False and f(q, k, v, lens) is False
    assert f(q.cpu(), k, v, lens, out) is False and f(q.float(), k, v, lens, out) is False
    assert f(torch.nn.Parameter(q), k, v, lens, out) is False
    assert f(q.clone().requires_grad_(), k, v, lens, out) is False

    class Sees(TorchDispatchMode):
        seen = []

        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            self.seen.append(str(func))
            return func(*args, **(kwargs or {}))

    with Sees() as mode:
        assert f(q, k, v, lens, out) is False
        assert (out == 7.0).all()
        kerns.flash_attn_decode(q, k, v, lens, out)
        assert "minfer.flash_attn_decode.default" in mode.seen
    with torch.inference_mode():
        assert f(q, k, v, lens, torch.zeros_like(q)) is True
    out2 = torch.zeros_like(out)
    torch.compile(lambda o: kerns.flash_attn_decode(q, k, v, lens, o), fullgraph=True, backend="eager")(out2)
    assert torch.equal(out, out2)


_TWO_ROUTES = """
import sys, threading
sys.path.insert(0, sys.argv[1])
import torch
from minfer.kernels.torch_ext import ops
torch.cuda.memory._record_memory_history(context="all", stacks="python")
q = torch.randn(1, 4, 1, 64, device="cuda").half()
k = torch.randn(1, 2, 64, 64, device="cuda").half()
lens = torch.full((1,), 64, dtype=torch.int32, device="cuda")
outs = [torch.zeros_like(q) for _ in range(2)]
streams = [torch.cuda.Stream() for _ in range(32)]
torch.cuda.synchronize()
done = threading.Event()

def dispatched():      # a new stream each time: a scratch buffer is allocated, and the allocator records this stack
    for s in streams[2:]:
        with torch.cuda.stream(s):
            torch.ops.minfer.flash_attn_decode.default(q, k, k, lens, outs[0])
    done.set()

def direct():          # two streams in turn: the buffers are looked up in every call
    while not done.is_set():
        for s in streams[:2]:
            with torch.cuda.stream(s):
                assert ops._direct.flash_attn_decode(q, k, k, lens, outs[1])
            s.synchronize()

threads = [threading.Thread(target=f) for f in (direct, dispatched)]
[t.start() for t in threads]
[t.join() for t in threads]
torch.cuda.synchronize()
assert torch.equal(*outs)
print("both routes ended")
"""


def test_both_routes_at_once_while_the_allocator_records_python_stacks():
    """The direct route comes to the buffers' lock with the interpreter's lock held, and the allocator wants the interpreter's
    lock: no thread may allocate under the former.  (In a process of its own, which ends by the limit if two threads wait for each other.)"""
    r = subprocess.run([sys.executable, "-c", _TWO_ROUTES, PKG_ROOT], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "both routes ended" in r.stdout, r.stderr[-2000:]


_FULL_DEVICE = """
import sys
sys.path.insert(0, sys.argv[1])
import torch
from minfer.kernels import KernelBackend
from minfer.kernels.torch_ext import ops
kerns = KernelBackend("torch_ext")
F16 = (1, 1, 2)
L = 6000                                       # the tiles' bits: 4.5 MB, their classes: 2 KB
g = torch.Generator(device="cuda").manual_seed(5)
q, k, v = (torch.randn(1, h, L, 64, generator=g, device="cuda").half() for h in (2, 1, 1))
mask = torch.rand(1, 1, L, L, generator=g, device="cuda") < 0.5
outs = [torch.zeros_like(q) for _ in range(3)]
stream = torch.cuda.Stream()
torch.cuda.synchronize()
torch.cuda.empty_cache()
total = torch.cuda.get_device_properties(0).total_memory
torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (4 << 20)) / total)    # 4 MB left
try:
    with torch.cuda.stream(stream):            # (the allocator keeps a pool per stream)
        torch.empty(8 << 20, dtype=torch.uint8, device="cuda")
    raise SystemExit("the device is not full")
except torch.OutOfMemoryError:
    pass
calls = [lambda o: kerns.flash_attn(*F16, q, k, v, mask, o), lambda o: torch.ops.minfer.flash_attn.default(*F16, q, k, v, mask, o)]
with torch.cuda.stream(stream):
    for call, out in zip(calls, outs):
        for _ in range(3):
            call(out)
torch.cuda.synchronize()
torch.cuda.set_per_process_memory_fraction(1.0)
with torch.cuda.stream(stream):
    for _ in range(260):                       # room again: the larger scratch is asked for within 256 calls
        kerns.flash_attn(*F16, q, k, v, mask, outs[2])
torch.cuda.synchronize()
assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
assert torch.isfinite(outs[0]).all() and outs[0].abs().sum() > 0
print("served")
"""


@pytest.mark.parametrize("binding", ["auto", "ctypes"])
def test_dense_mask_on_a_full_device(binding):
    """The scratch for the mask tiles' bits cannot be had: the call is served with the tile classes alone, with the same bits."""
    r = subprocess.run([sys.executable, "-c", _FULL_DEVICE, PKG_ROOT], capture_output=True, text=True, timeout=240,
                       env={**os.environ, "MINFER_ATTN_BINDING": binding})
    assert r.returncode == 0 and "served" in r.stdout, r.stdout + r.stderr[-2000:]
