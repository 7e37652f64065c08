"""Varlen tcgen05 attention against an fp32 PyTorch oracle."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from fms_acceleration_b200 import _native as NV
from fms_acceleration_b200.ops import attention as AT

DEV = "cuda"


def _rel(a, b):
    return ((a.float() - b.float()).norm() / b.float().norm().clamp(min=1e-12)).item()


def _make(T, nh, nkv, d, lens, dtype, seed=0):
    torch.manual_seed(seed)
    assert sum(lens) == T
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=DEV)
    ds, de = AT.doc_bounds_from_cu_seqlens(cu, T)
    qkv = torch.randn(T, (nh + 2 * nkv) * d, device=DEV, dtype=dtype)
    return qkv, ds, de


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("d", [128, 64])
@pytest.mark.parametrize("lens", [[128], [300], [100, 156, 7, 249], [513, 1, 254]])
def test_attention_forward(dtype, d, lens):
    T = sum(lens)
    nh, nkv = 4, 2
    qkv, ds, de = _make(T, nh, nkv, d, lens, dtype)
    q = qkv[:, : nh * d].view(T, nh, d)
    k = qkv[:, nh * d: (nh + nkv) * d].view(T, nkv, d)
    v = qkv[:, (nh + nkv) * d:].view(T, nkv, d)
    o = AT.varlen_attention(q, k, v, ds, de)
    NV.check_status()
    ref = AT.attention_ref(q, k, v, ds)
    assert _rel(o, ref) < 1.5e-2


@pytest.mark.parametrize("d", [128, 64])
@pytest.mark.parametrize("lens", [[1], [257], [129, 1, 1, 640], [900]])
def test_attention_forward_extreme_scores(d, lens):
    """Rows whose scores span hundreds (the running maximum advances block by block), rows with a single key, and tiles
    in which some rows have no key in a block.  P is rounded to 16 bits (half an ulp, 2^-9) and so is the result."""
    T, nh, nkv = sum(lens), 5, 1
    qkv, ds, de = _make(T, nh, nkv, d, lens, torch.bfloat16, seed=3)
    q = qkv[:, : nh * d].view(T, nh, d) * 4
    k = qkv[:, nh * d: (nh + nkv) * d].view(T, nkv, d) * (1 + torch.arange(T, device=DEV)[:, None, None] % 7).to(qkv.dtype)
    v = qkv[:, (nh + nkv) * d:].view(T, nkv, d)
    o = AT.varlen_attention(q, k, v, ds, de)
    NV.check_status()
    ref = AT.attention_ref(q, k, v, ds)
    assert torch.isfinite(o.float()).all()
    assert _rel(o, ref) < 2 * 2.0 ** -8


@pytest.mark.parametrize("d,dtype", [(128, torch.float16), (64, torch.float16), (128, torch.bfloat16)])
@pytest.mark.parametrize("lens", [[1], [127, 1], [1150], [129, 640, 1, 257]])
def test_attention_backward_ring_lengths(d, dtype, lens):
    """One to nine key blocks per query tile (the buffers and rings of the backward wrap at two), three query heads per
    key head, against fp32.  P and dS are rounded to 16 bits, sums are fp32: 4 ulp of the gradient in the 2-norm."""
    T, nh, nkv = sum(lens), 6, 2
    qkv, ds, de = _make(T, nh, nkv, d, lens, dtype, seed=5)
    q = qkv[:, : nh * d].reshape(T, nh, d).clone().requires_grad_()
    k = qkv[:, nh * d: (nh + nkv) * d].reshape(T, nkv, d).clone().requires_grad_()
    v = qkv[:, (nh + nkv) * d:].reshape(T, nkv, d).clone().requires_grad_()
    o = AT.varlen_attention(q, k, v, ds, de)
    g = torch.randn_like(o)
    got = torch.autograd.grad(o, (q, k, v), g)
    NV.check_status()
    qf, kf, vf = (t.detach().double().requires_grad_() for t in (q, k, v))
    rep = nh // nkv
    mask = (torch.arange(T, device=DEV)[None] <= torch.arange(T, device=DEV)[:, None]) & (
        torch.arange(T, device=DEV)[None] >= ds.long()[:, None])
    s = torch.einsum("thd,shd->hts", qf, kf.repeat_interleave(rep, 1)) * d ** -0.5
    ref = torch.einsum("hts,shd->thd", torch.softmax(s.masked_fill(~mask, float("-inf")), -1), vf.repeat_interleave(rep, 1))
    ulp = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    for a, r in zip(got, torch.autograd.grad(ref, (qf, kf, vf), g.double())):
        assert (a.double() - r).norm() <= 4 * ulp * r.norm() + 1e-6 * g.double().norm()


@pytest.mark.parametrize("d", [128, 64])
@pytest.mark.parametrize("lens", [[256], [100, 156, 7, 249], [640, 129, 255]])
def test_attention_backward(d, lens):
    T = sum(lens)
    nh, nkv = 4, 2
    dtype = torch.bfloat16
    qkv, ds, de = _make(T, nh, nkv, d, lens, dtype, seed=1)
    q = qkv[:, : nh * d].reshape(T, nh, d).clone().requires_grad_()
    k = qkv[:, nh * d: (nh + nkv) * d].reshape(T, nkv, d).clone().requires_grad_()
    v = qkv[:, (nh + nkv) * d:].reshape(T, nkv, d).clone().requires_grad_()
    o = AT.varlen_attention(q, k, v, ds, de)
    g = torch.randn_like(o)
    o.backward(g)
    NV.check_status()
    qf, kf, vf = (t.detach().float().requires_grad_() for t in (q, k, v))
    ref = AT.attention_ref(qf, kf, vf, ds)
    ref.backward(g.float())
    assert _rel(q.grad, qf.grad) < 3e-2
    assert _rel(k.grad, kf.grad) < 3e-2
    assert _rel(v.grad, vf.grad) < 3e-2


@pytest.mark.parametrize("d,nh,nkv", [(128, 8, 2), (64, 6, 2)])
def test_backward_on_ragged_documents_against_fp32(d, nh, nkv):
    """Backward kernels against the fp32 PyTorch statement on a longer packed batch with ragged documents
    (tile-crossing, single-token and tail documents)."""
    lens = [700, 1, 129, 1023, 64, 131]
    T = sum(lens)
    qkv, ds, de = _make(T, nh, nkv, d, lens, torch.bfloat16, seed=5)
    q, k, v = qkv[:, : nh * d], qkv[:, nh * d: (nh + nkv) * d], qkv[:, (nh + nkv) * d:]
    scale = d ** -0.5
    o, lse = AT._fwd(q, k, v, ds, de, nh, nkv, d, scale)
    do = torch.randn_like(o)
    got = AT._bwd(q, k, v, o, lse, do, ds, de, nh, nkv, d, scale)
    NV.check_status()
    qf, kf, vf = (t.float().reshape(T, -1, d).requires_grad_() for t in (q, k, v))
    ref = AT.attention_ref(qf, kf, vf, ds, scale)
    ref.backward(do.float().reshape(T, nh, d))
    for a, r in zip(got, (qf.grad, kf.grad, vf.grad)):
        assert _rel(a.reshape(T, -1, d), r) < 3e-2


def test_backward_is_bitwise_reproducible():
    """No gradient is accumulated with atomics: two runs of the same backward give the same bits."""
    lens = [700, 129, 1, 450]
    T, nh, nkv, d = sum(lens), 8, 2, 128
    qkv, ds, de = _make(T, nh, nkv, d, lens, torch.bfloat16, seed=3)
    grads = []
    for _ in range(2):
        q = qkv[:, : nh * d].reshape(T, nh, d).clone().requires_grad_()
        k = qkv[:, nh * d: (nh + nkv) * d].reshape(T, nkv, d).clone().requires_grad_()
        v = qkv[:, (nh + nkv) * d:].reshape(T, nkv, d).clone().requires_grad_()
        o = AT.varlen_attention(q, k, v, ds, de)
        torch.manual_seed(11)
        o.backward(torch.randn_like(o))
        NV.check_status()
        grads.append((o.detach().clone(), q.grad.clone(), k.grad.clone(), v.grad.clone()))
    for a, b in zip(*grads):
        assert torch.equal(a, b)


@pytest.mark.parametrize("dtype", [torch.int64, torch.int32])
@pytest.mark.parametrize("lens,lead", [([1], 0), ([1023, 1, 1025, 7], 0), ([5000, 3, 2], 0), ([1, 1, 1, 1], 0), ([2048, 2048], 0),
                                       ([100, 3000], 5), ([1500], 2100), ([], 1030)])
def test_doc_bounds_from_position_ids_equal_the_host_form(lens, lead, dtype):
    """Documents across and inside the 1024-token tiles; ``lead`` tokens before the first position 0 (or no 0 at all)."""
    pos = torch.cat([torch.arange(7, 7 + lead)] + [torch.arange(n) for n in lens]).to(dtype)
    got = AT.doc_bounds_from_position_ids(pos.to(DEV))
    cu = AT.cu_seqlens_from_position_ids(pos)
    ds, de = AT.doc_bounds_from_cu_seqlens(cu, pos.numel())
    assert torch.equal(got[0].cpu(), pos.to(torch.int32))
    assert torch.equal(got[1].cpu(), ds) and torch.equal(got[2].cpu(), de)


@pytest.mark.parametrize("scale", [0.0, 1e-30, 3e-25, 1e-3])
@pytest.mark.parametrize("d", [128, 64])
def test_attention_with_a_vanishing_scale_keeps_the_mask(d, scale):
    """Down to a scale of 0 (every key of a row weighs the same) no masked key has a weight: scores, outputs and the
    gradient of the values against fp32.  Tolerances of the other forward tests: one rounding of P and of the output."""
    T, nh, nkv = 330, 2, 1
    qkv, ds, de = _make(T, nh, nkv, d, [70, 1, 259], torch.bfloat16)
    q, k, v = (t.detach().requires_grad_() for t in (qkv[:, : nh * d].view(T, nh, d), qkv[:, nh * d: (nh + 1) * d].view(T, 1, d),
                                                     qkv[:, (nh + 1) * d:].view(T, 1, d)))
    o = AT._VarlenAttention.apply(q, k, v, ds, de, scale)
    g = torch.randn_like(o)
    got = torch.autograd.grad(o, [q, k, v], g)
    NV.check_status()
    t = [x.detach().float().requires_grad_() for x in (q, k, v)]
    ref = AT.attention_ref(*t, ds, scale or 1e-30)  # a scale of 0 asks the oracle for its default
    want = torch.autograd.grad(ref, t, g.float())
    assert _rel(o, ref) < 1.5e-2 and _rel(got[2], want[2]) < 1.5e-2
    assert all(torch.isfinite(x).all() for x in got)


@pytest.mark.parametrize("lens,lead", [([9217, 4], 5), ([30000, 2], 3000), ([20000, 1, 20000], 1023), ([1, 9300], 1),
                                       ([70000], 1024), ([], 11000), ([1100000, 5, 1050000], 0), ([1100000, 3], 1060000)])
def test_doc_bounds_of_long_documents_and_leads(lens, lead):
    """Documents and leads of many tiles, and (beyond 1024 tiles) of more than one step of the search over them."""
    pos = torch.cat([torch.arange(7, 7 + lead)] + [torch.arange(n) for n in lens])
    got = AT.doc_bounds_from_position_ids(pos.to(DEV))
    ds, de = AT.doc_bounds_from_cu_seqlens(AT.cu_seqlens_from_position_ids(pos), pos.numel())
    assert torch.equal(got[0].cpu(), pos.to(torch.int32))
    assert torch.equal(got[1].cpu(), ds) and torch.equal(got[2].cpu(), de)
