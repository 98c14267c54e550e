"""What the operations tell their kernels about operands that may be read before the wait for earlier kernels: only what the
caller has said is no output of this step.  The kernels are replaced by a recorder, so nothing here needs a GPU."""
import pytest
import torch

from zinfer_b200 import ops


class Recorder:
    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        def call(*args):
            self.calls.append((name, args))
            return 0
        return call


@pytest.fixture
def recorder(monkeypatch):
    r = Recorder()
    monkeypatch.setattr(ops, "lib", lambda: r)
    monkeypatch.setattr(ops, "_stream", lambda: None)
    monkeypatch.setattr(ops, "_ptr", lambda t: None)
    return r


def early(recorder, name):
    (args,) = [a for n, a in recorder.calls if n == name]
    recorder.calls.clear()
    return args[-2]


def test_32_bit_products_read_weights_early_only_when_told(recorder):
    x, w = torch.zeros(3, 8), torch.zeros(4, 8)
    for said, want in ((None, 0), (True, 0), (False, 1)):
        ops.linear(x, w, fresh_weight=said)
        assert early(recorder, "zi_gemm_simt") == want
    ops.linear(x, w)
    assert early(recorder, "zi_gemm_simt") == 0
    ops.linear_swiglu(x, torch.zeros(256, 8))
    assert early(recorder, "zi_gemm_simt") == 0
    ops.linear_argmax(x, w)
    assert early(recorder, "zi_gemm_simt") == 0


def test_norms_of_updates_read_nothing_before_their_wait():
    """In the kernel itself: the wait for earlier kernels stands before the first read of an operand."""
    import os
    import re

    with open(os.path.join(os.path.dirname(ops.__file__), "csrc", "elementwise.cu")) as fh:
        body = fh.read().split("norm_residual_few_kernel(", 1)[1].split("{", 1)[1]
    before = body[:body.index("pdl_wait();")]
    assert not re.search(r"\b(w|bias|a_log|x|h|a|ap|b|bp)\s*\[|load\(", before)


def test_decays_read_weights_early_only_when_told(recorder):
    class OnGpu(torch.Tensor):
        is_cuda = True

    x, pair = torch.zeros(2, 4, dtype=torch.bfloat16).as_subclass(OnGpu), torch.zeros(8, 4, dtype=torch.bfloat16)
    for said, want in (({}, 0), ({"fresh_weights": True}, 0), ({"fresh_weights": False}, 1)):
        ops.low_rank_decay(x, pair, torch.zeros(8), None, 16.0, 4, **said)
        assert early(recorder, "zi_low_rank_decay") == want


def test_models_say_that_their_weights_are_weights():
    """Every product of a part with a bound weight by way of ``ops.linear`` says that it is one."""
    import glob
    import os
    import re

    for f in glob.glob(os.path.join(os.path.dirname(ops.__file__), "parts", "*.py")):
        with open(f) as fh:
            src = fh.read()
        for m in re.finditer(r"ops\.linear\(", src):
            depth, j = 1, m.end()
            while depth:
                depth += {"(": 1, ")": -1}.get(src[j], 0)
                j += 1
            assert src[m.start():j].endswith("fresh_weight=False)"), (os.path.basename(f), src[m.start():j])
