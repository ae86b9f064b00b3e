"""An output buffer that overlaps an operand of the plan: the operands are read
as they were before the call.  The result is that of separate buffers, bit for
bit (the same kernels on the same values)."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

from tenax_b200 import _capi, dense  # noqa: E402


def _execute(plan, ins, out, precision):
    ptrs = (C.c_void_p * len(ins))(*[t.data_ptr() for t in ins])
    _capi.check(_capi.LIB.tnx_plan_execute(plan.handle, ptrs, out.data_ptr(), _capi.PRECISIONS[precision], None, 0,
                                           torch.cuda.current_stream().cuda_stream))


@pytest.mark.parametrize("precision", ["fp64", "bf16x3"])
@pytest.mark.parametrize("subs,shapes", [
    ("mk,kn->mn", [(300, 300), (300, 300)]),
    ("km,nk->nm", [(97, 97), (97, 97)]),
    ("ab,bc,cd->da", [(130, 130), (130, 130), (130, 130)]),
    ("abc->cab", [(37, 41, 29)]),
])
@pytest.mark.parametrize("shift", [0, 5, -7])
def test_out_over_an_operand(precision, subs, shapes, shift):
    plan = dense._plan(subs, tuple(shapes), precision)
    n = int(np.prod(plan.out_shape))
    for which in range(len(shapes)):
        g = torch.Generator().manual_seed(which + 1)
        ins = [torch.randn(s, generator=g, dtype=torch.float64).cuda() for s in shapes]
        ref = torch.empty(n, dtype=torch.float64, device="cuda")
        _execute(plan, ins, ref, precision)
        # operand `which` inside a larger buffer, the output `shift` elements from it
        buf = torch.zeros(n + ins[which].numel() + 32, dtype=torch.float64, device="cuda")
        at = 16
        own = buf[at:at + ins[which].numel()].view(shapes[which])
        own.copy_(ins[which])
        out = buf[at + shift:at + shift + n]
        _execute(plan, [own if i == which else t for i, t in enumerate(ins)], out, precision)
        assert torch.equal(out, ref), (which, float((out - ref).abs().max()))
