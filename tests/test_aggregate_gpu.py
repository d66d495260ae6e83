"""GPU parity of the segment aggregation kernel (through the C ABI) against the CPU
checker: golden vectors, seeded random graphs, hubs, odd widths, empty inputs."""
import hashlib
import os

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
G = os.path.join(os.path.dirname(__file__), "golden")


def load(name):
    return dict(np.load(os.path.join(G, name + ".npz")))


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def run(jg, x, idx, off, w, chunk=None, n_out=None):
    off_t = dev(off)
    plan = jg.ops.SpmmPlan(off_t, len(idx), chunk) if chunk else None
    y = jg.ops.segment_aggregate(dev(x), dev(idx), off_t, dev(w), n_out=n_out, plan=plan)
    torch.cuda.synchronize()
    return y.cpu().numpy()


def rel_err(y, truth, scale):
    """max |y - truth| / sum_j |w_j x_j| : the error scale of an fp32 sum of those terms."""
    return float((np.abs(y - truth) / (scale + 1e-30)).max()) if y.size else 0.0


def test_reference_smoke_inputs(cuda, oracle):
    d = load("ref_test_mp_spmm")
    assert np.array_equal(run(cuda, d["x"], d["row_indices"], d["column_offset"], d["csc_weight"]), d["out_csc"])
    assert np.array_equal(run(cuda, d["x"], d["column_indices"], d["row_offset"], d["csr_weight"]), d["out_csr"])
    d = load("ref_test_aggregate")
    assert np.array_equal(run(cuda, d["x"], d["row_indices"], d["column_offset"], d["csc_weight"]), d["out_fwd"])
    assert np.array_equal(run(cuda, d["x"], d["column_indices"], d["row_offset"], d["csr_weight"]), d["out_bwd"])


def test_citation_graph_bit_exact(cuda, oracle):
    d = load("citation_2708")
    y7 = run(cuda, d["x7"], d["row_indices"], d["column_offset"], d["csc_weight"])
    assert np.array_equal(y7, d["y7"])
    x256 = np.random.default_rng(int(d["x256_seed"]))
    _ = x256.standard_normal((2708, 7))
    x = x256.standard_normal((2708, 256)).astype(np.float32)
    y = run(cuda, x, d["row_indices"], d["column_offset"], d["csc_weight"], chunk=1024)
    assert np.array_equal(y[::97], d["y256_rows"])
    assert hashlib.sha256(y.tobytes()).digest() == d["y256_sha256"].tobytes()


def random_graph(rng, n_out, n_in, E, hubs=0, hub_deg=0):
    dst = rng.integers(0, n_out, size=E)
    if hubs:
        dst = np.concatenate([dst, np.repeat(rng.integers(0, n_out, size=hubs), hub_deg)])
    src = rng.integers(0, n_in, size=len(dst))
    order = np.argsort(dst, kind="stable")
    off = np.zeros(n_out + 1, np.int32)
    np.add.at(off, dst + 1, 1)
    off = np.cumsum(off).astype(np.int32)
    w = rng.standard_normal(len(dst)).astype(np.float32)
    return src[order].astype(np.int32), off, w


@pytest.mark.parametrize("f", [1, 3, 4, 7, 10, 16, 17, 31, 32, 33, 40, 47, 64, 65, 100, 128, 200, 256, 260, 512, 516])
def test_widths_against_oracle(cuda, oracle, f):
    rng = np.random.default_rng(100 + f)
    idx, off, w = random_graph(rng, 700, 500, 9000, hubs=2, hub_deg=300)
    x = rng.standard_normal((500, f)).astype(np.float32)
    want = oracle.aggregate(x, idx, off, w, n_out=700)
    truth, scale = oracle.aggregate_f64(x, idx, off, w, n_out=700)
    for chunk in (None, 64):
        y = run(cuda, x, idx, off, w, chunk=chunk, n_out=700)
        assert rel_err(y, truth, scale) <= 1e-5
        assert rel_err(y, want, scale) <= 1e-5
        if f < 32 or f > 64:    # one lane group walks the row alone: the reference's summation order
            deg = np.diff(off)
            rows = deg <= (chunk or 1 << 30)
            assert np.array_equal(y[rows], want[rows])


@pytest.mark.parametrize("chunk", [1, 5, 32, 1000])
def test_hub_rows_split_into_pieces(cuda, oracle, chunk):
    rng = np.random.default_rng(chunk)
    idx, off, w = random_graph(rng, 50, 400, 300, hubs=3, hub_deg=5000)
    x = rng.standard_normal((400, 128)).astype(np.float32)
    truth, scale = oracle.aggregate_f64(x, idx, off, w, n_out=50)
    y1 = run(cuda, x, idx, off, w, chunk=chunk, n_out=50)
    y2 = run(cuda, x, idx, off, w, chunk=chunk, n_out=50)
    assert rel_err(y1, truth, scale) <= 1e-5
    assert np.array_equal(y1, y2)  # no atomics on data: run-to-run identical


def test_empty_rows_and_empty_graph(cuda, oracle):
    x = np.ones((4, 128), np.float32)
    off = np.zeros(6, np.int32)
    y = run(cuda, x, np.zeros(0, np.int32), off, np.zeros(0, np.float32), n_out=5)
    assert y.shape == (5, 128) and not y.any()
    off = np.array([0, 0, 2, 2, 2, 3], np.int32)
    idx = np.array([3, 0, 1], np.int32)
    w = np.array([2, 3, 4], np.float32)
    for chunk in (None, 1):
        y = run(cuda, x, idx, off, w, chunk=chunk, n_out=5)
        assert y[:, 0].tolist() == [0, 5, 0, 0, 4]
    y = cuda.ops.segment_aggregate(torch.zeros((3, 0), device="cuda"), dev(idx), dev(off), dev(w), n_out=5)
    assert tuple(y.shape) == (5, 0)


def test_int64_indices_are_narrowed(cuda, oracle):
    d = load("ref_test_spmm")
    # transposed structure of the reference's int64 CSR smoke input (tests/test_spmmcsr.py:13-17)
    src = np.repeat(np.arange(3), np.diff(d["row_offset"]))
    order = np.argsort(d["column_indices"], kind="stable")
    toff = np.concatenate([[0], np.cumsum(np.bincount(d["column_indices"], minlength=3))])
    y = cuda.ops.segment_aggregate(dev(d["csr_x"]), dev(src[order].astype(np.int64)), dev(toff.astype(np.int64)),
                                   dev(d["csr_weight"][order]))
    assert np.array_equal(y.cpu().numpy(), d["csr_out"])


def test_bad_arguments_raise(cuda):
    x = torch.zeros((4, 8), device="cuda")
    off = torch.tensor([0, 1, 2], dtype=torch.int32, device="cuda")
    with pytest.raises(RuntimeError):
        cuda.ops.segment_aggregate(x, torch.zeros(2, dtype=torch.int32, device="cuda"), off, torch.zeros(3, device="cuda"))
    with pytest.raises(RuntimeError):
        cuda.ops.segment_aggregate(x.double(), torch.zeros(2, dtype=torch.int32, device="cuda"), off, torch.zeros(2, device="cuda"))
    from jittorgeometric_b200 import _lib
    L = _lib.lib()
    st = L.jg_aggregate_f32(_lib.ptr(x), _lib.ptr(x), _lib.ptr(off), _lib.ptr(off), _lib.ptr(x), 2, 4, 8, 2, None, 0, None, 0, None)
    assert st == -3 and b"workspace" in L.jg_last_error()
    st = L.jg_aggregate_f32(None, _lib.ptr(x), _lib.ptr(off), _lib.ptr(off), _lib.ptr(x), 2, 4, 8, 2, None, 0, None, 0, None)
    assert st == -1


def test_autograd_pairing(cuda, oracle):
    d = load("citation_2708")
    csc = cuda.CSC(dev(d["row_indices"]), dev(d["column_offset"]), dev(d["csc_weight"]))
    csr = cuda.CSR(dev(d["column_indices"]), dev(d["row_offset"]), dev(d["csr_weight"]))
    x = dev(d["x7"]).requires_grad_(True)
    y = cuda.aggregateWithWeight(x, csc, csr)
    g = torch.from_numpy(np.random.default_rng(5).standard_normal((2708, 7)).astype(np.float32)).cuda()
    y.backward(g)
    want = oracle.aggregate(g.cpu().numpy(), d["column_indices"], d["row_offset"], d["csr_weight"])
    got = x.grad.cpu().numpy()
    # rows no longer than a hub piece are summed in the reference's order: bit-identical; the few
    # longer rows of this small graph are cut into pieces (short ones, so that no warp walks a long
    # row alone) and agree to rounding
    whole = np.diff(d["row_offset"]) <= cuda.ops.default_chunk(len(d["column_indices"]))
    assert whole.sum() > 2600 and not whole.all()
    assert np.array_equal(got[whole], want[whole])
    _, scale = oracle.aggregate_f64(g.cpu().numpy(), d["column_indices"], d["row_offset"], d["csr_weight"])
    assert rel_err(got, want, scale) <= 1e-5


def test_structure_validation(cuda):
    t = lambda a, dt: torch.tensor(a, dtype=dt, device="cuda")
    good_idx, good_off = t([0, 2, 1], torch.int32), t([0, 1, 1, 3], torch.int32)
    cuda.ops.validate_structure(good_idx, good_off, 3)
    for idx, off in (([0, 3, 1], [0, 1, 1, 3]),        # index out of range
                     ([0, -1, 1], [0, 1, 1, 3]),       # negative index
                     ([0, 2, 1], [0, 2, 1, 3]),        # decreasing offsets
                     ([0, 2, 1], [1, 1, 1, 3]),        # does not start at 0
                     ([0, 2, 1], [0, 1, 1, 2])):       # does not end at the entry count
        with pytest.raises(RuntimeError, match="bad structure"):
            cuda.ops.validate_structure(t(idx, torch.int32), t(off, torch.int32), 3)
    cuda.ops.validate_structure(t([], torch.int32), t([0, 0], torch.int32), 5)   # empty graph is fine


def test_cuda_graph_replay(cuda, oracle):
    """The aggregation is a fixed launch sequence with caller-owned buffers: captured once in a CUDA
    graph it can be replayed on new feature values (launch-bound small graphs)."""
    d = load("citation_2708")
    idx, off, w = dev(d["row_indices"]), dev(d["column_offset"]), dev(d["csc_weight"])
    plan = cuda.ops.SpmmPlan(off, idx.numel())
    x = torch.zeros((2708, 64), device="cuda")
    y = torch.empty_like(x)
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        cuda.ops.segment_aggregate(x, idx, off, w, plan=plan, out=y)      # warm-up outside capture
    torch.cuda.current_stream().wait_stream(s)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        cuda.ops.segment_aggregate(x, idx, off, w, plan=plan, out=y)
    rng = np.random.default_rng(3)
    for _ in range(2):
        xv = rng.standard_normal((2708, 64)).astype(np.float32)
        x.copy_(torch.from_numpy(xv))
        g.replay()
        torch.cuda.synchronize()
        got = y.cpu().numpy()
        eager = cuda.ops.segment_aggregate(x, idx, off, w, plan=plan).cpu().numpy()
        assert np.array_equal(got, eager)
        want = oracle.aggregate(xv, d["row_indices"], d["column_offset"], d["csc_weight"])
        truth, scale = oracle.aggregate_f64(xv, d["row_indices"], d["column_offset"], d["csc_weight"])
        assert rel_err(got, want, scale) <= 1e-5


@pytest.mark.parametrize("f", [7, 32, 64, 100, 128, 256, 512])
def test_fused_bias_and_relu_epilogue(cuda, f):
    """act(sum + bias) written by the aggregation kernel equals the aggregation followed by the two
    elementwise passes, bit for bit; rows split into pieces (hubs) and empty rows included."""
    rng = np.random.default_rng(40 + f)
    n = 900
    idx, off, w = random_graph(rng, n, n, 12000, hubs=2, hub_deg=3000)
    off[-1] = off[-2]                                            # make sure the last row is empty
    idx, w = idx[: off[-1]], w[: off[-1]]
    x = rng.standard_normal((n, f)).astype(np.float32)
    bias = rng.standard_normal(f).astype(np.float32)
    off_t = dev(off)
    plan = cuda.ops.SpmmPlan(off_t, len(idx), 1024)
    for pl in (plan, None):
        plain = cuda.ops.segment_aggregate(dev(x), dev(idx), off_t, dev(w), plan=pl)
        for b, relu in ((dev(bias), True), (dev(bias), False), (None, True)):
            got = cuda.ops.segment_aggregate(dev(x), dev(idx), off_t, dev(w), plan=pl, bias=b, relu=relu)
            want = plain if b is None else plain + b
            want = torch.relu(want) if relu else want
            assert torch.equal(got, want)
    assert torch.equal(got[-1], torch.zeros(f, device="cuda"))   # empty row: relu(0) with no bias
    with pytest.raises(RuntimeError):
        cuda.ops.segment_aggregate(dev(x), dev(idx), off_t, dev(w), out=plain, accumulate=True, relu=True)


def test_fused_epilogue_autograd(cuda):
    """aggregate_bias_act against the unfused composition: outputs equal, gradients of x and bias
    equal (the backward masks with the saved output and aggregates over the CSR)."""
    rng = np.random.default_rng(50)
    n, f = 600, 64
    ei = np.unique(rng.integers(0, n, size=(7000, 2)), axis=0).T.astype(np.int32)
    w = rng.random(ei.shape[1]).astype(np.float32)
    csc, csr = cuda.cootocsc(dev(ei), dev(w), n), cuda.cootocsr(dev(ei), dev(w), n)
    x0 = rng.standard_normal((n, f)).astype(np.float32)
    b0 = rng.standard_normal(f).astype(np.float32)
    g0 = dev(rng.standard_normal((n, f)).astype(np.float32))
    res = []
    for fused in (True, False):
        x, b = dev(x0).requires_grad_(True), dev(b0).requires_grad_(True)
        y = cuda.ops.aggregate_bias_act(x, csc, csr, b, relu=True) if fused else torch.relu(cuda.aggregateWithWeight(x, csc, csr) + b)
        y.backward(g0)
        res.append((y.detach(), x.grad, b.grad))
    assert torch.equal(res[0][0], res[1][0]) and torch.equal(res[0][1], res[1][1])
    assert (res[0][2] - res[1][2]).abs().max().item() <= 1e-4 * res[1][2].abs().max().item()


@pytest.mark.parametrize("mode", ["plain", "epilogue", "accumulate", "combine"])
@pytest.mark.parametrize("f", [5, 32, 36, 40, 44, 48, 64, 72, 130])
def test_row_lengths_and_epilogues(cuda, oracle, f, mode):
    """Rows of 0 to 34 entries in every order, runs of empty rows, rows one entry above and below the piece length, an
    infinite value in a row that no entry names; so few rows are walked one by one (several a ticket: further down).
    A sum of k terms is off by at most k + 4 roundings (its epilogue's included) of the sum of magnitudes."""
    rng = np.random.default_rng(f)
    n_in = 500
    lens = np.concatenate([np.arange(35), np.zeros(40, int), rng.integers(0, 35, 3000), [63, 64, 65, 200, 127, 128, 129]])
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    idx = rng.integers(1, n_in, off[-1]).astype(np.int32)
    w = rng.standard_normal(off[-1]).astype(np.float32)
    x = rng.standard_normal((n_in, f)).astype(np.float32)
    x[0] = np.inf
    n = len(lens)
    other = rng.standard_normal((n, f)).astype(np.float32)
    bias = rng.standard_normal(f).astype(np.float32)
    off_t = dev(off)
    plan = cuda.ops.SpmmPlan(off_t, len(idx), 64)
    call = lambda **kw: cuda.ops.segment_aggregate(dev(x), dev(idx), off_t, dev(w), plan=plan, **kw)
    x64 = np.where(np.isfinite(x), x, 0.0)
    truth, scale = oracle.aggregate_f64(x64.astype(np.float32), idx, off, w)
    if mode == "plain":
        got = call()
    elif mode == "epilogue":
        got = call(bias=dev(bias), relu=True)
        truth, scale = np.maximum(truth + bias, 0), scale + np.abs(bias)
    elif mode == "accumulate":
        got = call(out=dev(other), accumulate=True)
        truth, scale = truth + other, scale + np.abs(other)
    else:
        got = call(addend=dev(other), scale=0.9, add_scale=0.1)
        a, b = float(np.float32(0.9)), float(np.float32(0.1))
        truth, scale = a * truth + b * other, a * scale + b * np.abs(other)
    assert np.all(np.abs(got.cpu().numpy() - truth) <= (lens[:, None] + 4) * 2.0**-24 * scale + 1e-30)


@pytest.mark.parametrize("f", [7, 40, 46])
def test_propagation_gradient(cuda, f):
    """The gradient of the hops is the transposed recursion: against float64 autograd, and twice differentiable."""
    from jittorgeometric_b200 import nn
    torch.manual_seed(f)
    n, hops = 300, 4
    ei = torch.randint(0, n, (2, 4000), device="cuda", dtype=torch.int32)
    csc, csr = cuda.gcn_norm_csc_csr(ei, None, n)
    A = torch.zeros((n, n), dtype=torch.float64, device="cuda")
    dst = torch.repeat_interleave(torch.arange(n, device="cuda"), (csc.column_offset[1:] - csc.column_offset[:-1]).long())
    A.index_put_((dst, csc.row_indices.long()), csc.edge_weight.double(), accumulate=True)
    P = torch.eye(n, dtype=torch.float64, device="cuda")
    for _ in range(hops):
        P = 0.9 * (A @ P) + 0.1 * torch.eye(n, dtype=torch.float64, device="cuda")
    x = torch.randn((n, f), device="cuda", requires_grad=True)
    g = torch.randn((n, f), device="cuda", requires_grad=True)
    y = nn.APPNP(hops, 0.1)(x, csc, csr)
    assert y.is_contiguous()
    gx, = torch.autograd.grad(y, x, g, create_graph=True)
    gg, = torch.autograd.grad(gx, g, x)          # the product is linear in g: its derivative along x is P x
    for have, want in ((y, P @ x.double()), (gx, P.t() @ g.double()), (gg, P @ x.double())):
        assert (have.double() - want).abs().max().item() <= 1e-5 * want.abs().max().item()


@pytest.mark.parametrize("f", [4, 36, 64, 128])
def test_workspace_on_an_8_byte_border(cuda, oracle, f):
    """The C ABI asks no more of a workspace than its counter's eight bytes: hubs of few and of many pieces whose
    partial rows start beside a 16-byte border."""
    from jittorgeometric_b200 import _lib
    rng = np.random.default_rng(f)
    lens = np.concatenate([rng.integers(0, 30, 300), [16 * 8, 16 * 8 + 1, 16 * 9, 1000], rng.integers(0, 30, 300)])
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    n_in, nnz, n = 400, int(off[-1]), len(lens)
    idx = rng.integers(0, n_in, nnz).astype(np.int32)
    w = rng.standard_normal(nnz).astype(np.float32)
    x = rng.standard_normal((n_in, f)).astype(np.float32)
    off_t, idx_t, w_t, x_t = dev(off), dev(idx), dev(w), dev(x)
    plan = cuda.ops.SpmmPlan(off_t, nnz, 16)
    L = _lib.lib()
    need = L.jg_aggregate_workspace_bytes(n, nnz, f, 16)
    ws = torch.empty(need + 16, dtype=torch.uint8, device="cuda")
    out = torch.empty((n, f), dtype=torch.float32, device="cuda")
    assert ws.data_ptr() % 16 == 0
    _lib.check(L.jg_aggregate_f32(out.data_ptr(), x_t.data_ptr(), idx_t.data_ptr(), off_t.data_ptr(), w_t.data_ptr(), n, n_in, f, nnz,
                                  plan.buf.data_ptr(), 16, ws.data_ptr() + 8, need, _lib.stream_for(out)), "jg_aggregate_f32")
    truth, scale = oracle.aggregate_f64(x, idx, off, w)
    assert np.all(np.abs(out.cpu().numpy() - truth) <= (lens[:, None] + 4) * 2.0**-24 * scale + 1e-30)


@pytest.mark.parametrize("mode", ["plain", "epilogue", "accumulate", "combine"])
@pytest.mark.parametrize("n,f", [(n, f) for n in (60001, 130003) for f in (32, 36, 40, 44, 48, 52, 56, 60, 64)] +
                         [(930001, f) for f in (32, 40, 64)])
def test_several_rows_a_ticket(cuda, n, f, mode):
    """2, 4 and 8 rows a ticket (the last ticket cut short): rows of 0 to 34 entries in every order, runs of empty rows, hub
    rows between rows of the same ticket.  The same rows in calls too small for that are walked row by row, the sums in
    the same order: equal bit for bit.  Those are checked against float64 above."""
    rng = np.random.default_rng(n + f)
    lens = rng.integers(0, 7, n)
    for at in range(0, n - 200, n // 9):
        lens[at:at + 35], lens[at + 35:at + 75], lens[at + 75:at + 82] = np.arange(35), 0, [63, 64, 65, 200, 0, 129, 7]
    lens[rng.integers(0, n, 200)] = 300
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    n_in, nnz = 5000, int(off[-1])
    gen = torch.Generator(device="cuda").manual_seed(f)
    idx = torch.randint(1, n_in, (nnz,), device="cuda", generator=gen, dtype=torch.int32)
    w = torch.randn(nnz, device="cuda", generator=gen)
    x = torch.randn((n_in, f), device="cuda", generator=gen)
    x[0] = float("inf")          # no entry names it
    other, bias = torch.randn((n, f), device="cuda", generator=gen), torch.randn(f, device="cuda", generator=gen)

    def call(a, b):
        o = dev(off[a:b + 1])
        kw = {"plain": {}, "epilogue": dict(bias=bias, relu=True), "accumulate": dict(out=other[a:b].clone(), accumulate=True),
              "combine": dict(addend=other[a:b], scale=0.9, add_scale=0.1)}[mode]
        return cuda.ops.segment_aggregate(x, idx, o, w, plan=cuda.ops.SpmmPlan(o, nnz, 64), **kw)

    got = call(0, n)
    for a in range(0, n, 30000):
        b = min(a + 30000, n)
        assert torch.equal(got[a:b], call(a, b))
    assert torch.isfinite(got).all()


@pytest.mark.parametrize("f", [36, 48, 60, 64])
def test_long_rows_on_either_kernel(cuda, f):
    """Rows of some 40 to 80 entries are walked row by row while x fits L2 and streamed beyond that: the same rows of a
    short and of a long x take the two kernels.  Equal bit for bit."""
    n, n_in = 40009, 3000
    rng = np.random.default_rng(f)
    lens = rng.integers(40, 56, n) if f < 64 else rng.integers(56, 80, n)
    lens[rng.integers(0, n, 50)] = 700
    off = dev(np.concatenate([[0], np.cumsum(lens)]).astype(np.int32))
    nnz = int(off[-1])
    gen = torch.Generator(device="cuda").manual_seed(f)
    idx = torch.randint(0, n_in, (nnz,), device="cuda", generator=gen, dtype=torch.int32)
    w, x = torch.randn(nnz, device="cuda", generator=gen), torch.randn((n_in, f), device="cuda", generator=gen)
    far = torch.zeros((1_000_000, f), device="cuda")
    far[:n_in] = x
    plan = cuda.ops.SpmmPlan(off, nnz, 256)
    assert torch.equal(cuda.ops.segment_aggregate(x, idx, off, w, plan=plan), cuda.ops.segment_aggregate(far, idx, off, w, plan=plan))


def test_propagation_takes_what_it_took(cuda):
    """Any object with the containers' fields is a container, and a number of hops is a whole number."""
    from types import SimpleNamespace
    from jittorgeometric_b200 import nn
    n = 60
    ei = torch.randint(0, n, (2, 300), device="cuda", dtype=torch.int32)
    csc, csr = cuda.gcn_norm_csc_csr(ei, None, n)
    x = torch.randn((n, 12), device="cuda", requires_grad=True)
    y = nn.APPNP(3, 0.1)(x, csc, csr)
    g, = torch.autograd.grad(y, x, torch.ones_like(y))
    like = nn.APPNP(np.int64(3), 0.1)(x, SimpleNamespace(**vars(csc)), SimpleNamespace(**vars(csr)))
    assert torch.equal(like, y) and torch.equal(torch.autograd.grad(like, x, torch.ones_like(y))[0], g)
    with pytest.raises(TypeError):
        nn.APPNP(2.5, 0.1)(x, csc, csr)
    assert nn.APPNP(0, 0.1)(x, csc, csr) is x
