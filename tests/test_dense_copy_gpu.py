"""GPU: the dense copy a layer keeps of its CSR weight always stands for the tensors it is asked with: after
every kind of change of them, in recorded calls, on other streams, and after saving and loading."""
import copy
import io

import pytest
import torch
from torch import nn

from intrasm_engine_b200.pytorch.huggingface_rewriter import SparseLinear
from intrasm_engine_b200.pytorch.utils import DenseCopy, dense_to_sparse_cuda

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _weight(m=128, k=256, density=0.5, seed=0):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    w = torch.randint(1, 4, (m, k), generator=g, device=DEV).half()
    return torch.where(torch.rand(m, k, generator=g, device=DEV) < density, w, torch.zeros_like(w))


def _csr(w):
    values, _ri, ro, ci = dense_to_sparse_cuda(w)
    return values, ro, ci


def test_follows_changes_in_place():
    w = _weight()
    values, ro, ci = _csr(w)
    kept = DenseCopy(*w.shape)
    first = kept.current(values, ro, ci)
    assert torch.equal(first, w) and kept.current(values, ro, ci) is first
    values.mul_(2)
    assert torch.equal(kept.current(values, ro, ci), 2 * w)
    w2 = w.roll(1, 0)  # rows moved: other offsets, columns and values of the same sizes, written in place
    for old, new in zip((values, ro, ci), _csr(w2)):
        old.copy_(new)
    assert torch.equal(kept.current(values, ro, ci), w2)


@pytest.mark.parametrize("which", ["values", "row_offsets", "column_indices"])
def test_follows_one_replaced_tensor(which):
    """One of the three tensors becomes another object at the same address and of the same version, after a
    change that left no trace in the counters."""
    w = _weight(seed=1)
    w[1] = w[0].flip(0)  # two rows of one length, other columns
    w[3] = 0
    csr = dict(zip(("values", "row_offsets", "column_indices"), _csr(w)))
    kept = DenseCopy(*w.shape)
    assert torch.equal(kept.current(**csr), w)
    same = csr[which].data
    if which == "values":
        same.mul_(2)
        w = 2 * w
    elif which == "row_offsets":  # row 2 becomes empty, row 3 gets its nonzeros
        same[3] = same[2]
        w[3], w[2] = w[2].clone(), 0
    else:  # rows 0 and 1 exchange their columns and keep their values
        ends = csr["row_offsets"][:3].tolist()
        first, second = same[ends[0]:ends[1]].clone(), same[ends[1]:ends[2]].clone()
        same[ends[0]:ends[1]], same[ends[1]:ends[2]] = second, first
        for r, cols in ((0, second), (1, first)):
            w[r] = 0
            w[r, cols.long()] = csr["values"][ends[r]:ends[r + 1]]
    csr[which] = same
    assert torch.equal(kept.current(**csr), w)


def test_parameter_registered_again():
    w = _weight()
    layer = SparseLinear(w)
    x = torch.randint(-2, 3, (4, w.size(1)), device=DEV).half()
    assert torch.equal(layer(x), (x.float() @ w.float().t()).half())
    data = layer.values.data
    address = data.data_ptr()
    del layer.values
    data.mul_(2)
    layer.values = nn.Parameter(data, requires_grad=False)
    assert layer.values.data_ptr() == address
    assert torch.equal(layer(x), (x.float() @ (2 * w).float().t()).half())
    layer.values.data = layer.values.data.clone() * 0.5  # the same Parameter, other storage
    assert torch.equal(layer(x), (x.float() @ w.float().t()).half())
    layer.values.data.mul_(2)  # leaves no trace: the layer has to be told
    layer.reset_dense_copy()
    assert torch.equal(layer(x), (x.float() @ (2 * w).float().t()).half())


def test_inference_tensors_get_no_copy():
    w = _weight()
    x = torch.randint(-2, 3, (4, w.size(1)), device=DEV).half()
    with torch.inference_mode():
        values, ro, ci = _csr(w)
        assert DenseCopy(*w.shape).current(values, ro, ci) is None
        layer = SparseLinear(w)
        assert torch.equal(layer(x), (x.float() @ w.float().t()).half())
        layer.values.mul_(2)
        assert torch.equal(layer(x), (x.float() @ (2 * w).float().t()).half())
    layer = SparseLinear(w)
    with torch.inference_mode():  # an ordinary layer keeps its copy in inference mode
        kept = layer.dense_copy()
        assert kept is not None and layer.dense_copy() is kept


@pytest.mark.parametrize("tokens", [1, 4, 300])
def test_recorded_call_reads_the_values_of_the_replay(tokens):
    w = _weight()
    layer = SparseLinear(w)
    x = torch.randint(-2, 3, (tokens, w.size(1)), device=DEV).half()
    layer(x)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.no_grad(), torch.cuda.graph(graph):
        y = layer(x)
    for factor in (1, 2, 3):
        layer.values.copy_(_csr(factor * w)[0])
        layer(x)  # the layer's own copy moves on in between
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, (x.float() @ (factor * w).float().t()).half())
    del graph


def test_copy_is_complete_for_other_streams():
    """A copy rebuilt behind a long wait on one stream is read on another at once."""
    w = _weight(512, 512)
    layer = SparseLinear(w)
    x = torch.randint(-2, 3, (8, 512), device=DEV).half()
    ref = (x.float() @ (2 * w).float().t()).half()
    one, two = torch.cuda.Stream(), torch.cuda.Stream()
    layer.values.mul_(2)
    torch.cuda.synchronize()
    with torch.cuda.stream(one):
        torch.cuda._sleep(50_000_000)
        a = layer(x)
    with torch.cuda.stream(two):
        b = layer(x)
    torch.cuda.synchronize()
    assert torch.equal(a, ref) and torch.equal(b, ref)


def test_replaced_copy_is_not_reused_while_another_stream_reads_it():
    w = _weight(2048, 2048)
    layer = SparseLinear(w)
    x = torch.randint(-1, 2, (16, 2048), device=DEV).half()
    ref = (x.float() @ w.float().t()).half()
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        torch.cuda._sleep(50_000_000)
        y = layer(x)  # waits on the side stream
    old = layer.dense_copy().data_ptr()
    layer.reset_dense_copy()  # on the main stream: the copy is let go ...
    grabbed = [torch.full((2048, 2048), 7.0, dtype=torch.float16, device=DEV) for _ in range(3)]
    assert all(t.data_ptr() != old for t in grabbed)  # ... but its memory is not handed out yet
    torch.cuda.synchronize()
    assert torch.equal(y, ref)


def test_saving_leaves_the_copy_out():
    w = _weight()
    layer = SparseLinear(w)
    x = torch.randint(-2, 3, (4, w.size(1)), device=DEV).half()
    size = []
    for kept in (True, False):
        if not kept:
            layer.reset_dense_copy()
        buf = io.BytesIO()
        torch.save(layer, buf)
        size.append(buf.tell())
        buf.seek(0)
        assert torch.equal(torch.load(buf, weights_only=False)(x), layer(x))
    assert abs(size[0] - size[1]) < 1024
    twin = copy.deepcopy(layer)
    twin.values.mul_(2)
    assert torch.equal(twin(x), 2 * layer(x))
    state = twin.__dict__.copy()
    del state["_dense"]  # a layer saved before there was a copy
    old = SparseLinear.__new__(SparseLinear)
    old.__setstate__(state)
    assert torch.equal(old(x), twin(x))
