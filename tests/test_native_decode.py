"""Which decode steps the one-kernel path takes and what it is told, on the host (no GPU: the native call is recorded)."""

from types import SimpleNamespace

import pytest
import torch

from flashdecode_cuda_b200 import kernels as K
from flashdecode_cuda_b200.engine import native as N
from flashdecode_cuda_b200.engine.model import Workspace
from flashdecode_cuda_b200.parts import linear


class Weights:
    """What the native call asks of a tensor, with any address."""

    def __init__(self, address=1 << 20, elements=1 << 26, is_cuda=True, contiguous=True):
        self.address, self.elements, self.is_cuda, self.contiguous = address, elements, is_cuda, contiguous

    def data_ptr(self):
        return self.address

    def numel(self):
        return self.elements

    def element_size(self):
        return 2

    def is_contiguous(self):
        return self.contiguous


def _step(rows, bound=2048):
    """A step of one token each, and a native form of a model of one layer (the sizes of Qwen2.5-1.5B), on host memory."""
    ints = torch.zeros(rows, dtype=torch.int32)
    pool = torch.zeros(1, 4, 2, 16, 128, dtype=torch.bfloat16)
    group = SimpleNamespace(keys=pool, values=pool.clone(), table=torch.zeros(rows, 128, dtype=torch.int32))
    ctx = SimpleNamespace(T=rows, n_rows=rows, max_q_len=1, kv_len_bound=bound, tok_pos=ints, row_slot=ints, row_ctx_len=ints,
                          ws=Workspace(torch.device("cpu")), rt=SimpleNamespace(status=torch.zeros(1, dtype=torch.int32)),
                          cache=SimpleNamespace(num_blocks=4, block_size=16, groups=[group]))
    native = N.DensePrompts()
    native.layers, native.n, native.addresses, native.positions, native.all_write = [None], 1, [0], [], True
    native.exchange_words = {}
    native.hidden, native.inter, native.n_q, native.n_kv, native.d = 1536, 8960, 12, 2, 128
    native._current = lambda model: True
    return native, ctx


@pytest.fixture
def calls(monkeypatch):
    """What the native decode calls were given."""
    seen = []
    real = K.lib()

    class Lib:
        def __getattr__(self, name):
            return getattr(real, name)

        def fd_dense_decode(self, step, layers, n):
            s = N._Decode()
            N.ctypes.memmove(N.ctypes.addressof(s), step, N.ctypes.sizeof(s))
            seen.append(s)
            return 0

    monkeypatch.setattr(K, "lib", lambda lib=Lib(): lib)
    monkeypatch.setattr(K, "_stream", lambda: None)
    monkeypatch.setattr(K, "dense_decode_words", lambda *a, f=K.dense_decode_words: f(*a, 148, 232448))
    return seen


@pytest.mark.parametrize("upcoming,want", [
    (None, (None, 0)), (Weights(), (1 << 20, linear.UPCOMING_BYTES)), (Weights(elements=100), (1 << 20, 192)),
    (Weights(is_cuda=False), (None, 0)), (Weights(contiguous=False), (None, 0)), (Weights(address=(1 << 20) + 2), (None, 0))])
def test_only_memory_that_l2_can_be_asked_for(calls, upcoming, want):
    """What the step streams next is a hint: whole 16-byte words of contiguous device memory, and nothing of any other tensor."""
    native, ctx = _step(2)
    assert native.decodes(None, ctx)
    native.decode(ctx, torch.zeros(2, 1536), upcoming)
    assert [(s.next, s.next_bytes) for s in calls] == [want]


@pytest.mark.parametrize("gemm,most", [("auto", 24), ("tcgen05", 16), ("cublas", 16)])
def test_the_switch_for_products_rules_from_17_rows_on(calls, monkeypatch, gemm, most):
    """``linear.PROMPT_GEMM`` names the kernels of steps of more than 16 rows; a step that is to run on others is not one kernel."""
    monkeypatch.setattr(linear, "PROMPT_GEMM", gemm)
    assert [rows for rows in range(1, 26) if _step(rows)[0].decodes(None, _step(rows)[1])] == list(range(1, most + 1))


def test_steps_of_all_row_counts_share_their_exchange_memory(calls):
    """A workspace holds the words of the largest step so far, and no more splits of the attention than a step can have."""
    ws = Workspace(torch.device("cpu"))
    sizes = {rows: K.dense_decode_words(rows, 1536, 8960, 12, 2, 128) for rows in (24, 3, 17, 1)}
    for rows in sizes:
        native, ctx = _step(rows)
        ctx.ws = ws
        assert native.decodes(None, ctx)
        native.decode(ctx, torch.zeros(rows, 1536), None)
    assert len({s.exchange for s in calls}) == 1
    assert sum(b.numel() for (_, dtype), b in ws._bufs.items() if dtype == torch.int64) == sizes[24]
    # packets of a row: x twice, sums of squares, q, k and v, attention, activations, at most 4 slices' partial sums, 3 splits of 12 heads
    assert sizes[24] <= 24 * (1536 + 192 + 768 + 256 + 768 + 4480 + 4 * 1536 + 3 * 12 * 130) + 200
