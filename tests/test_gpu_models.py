"""Model blocks on one GPU (a team of one PE): the whole kernel chain of each layer runs, only the
NVLink hops are local. Compared against plain PyTorch fp32 evaluations of the same layers."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def shm():
    import rocshmem_b200 as s
    if s.is_initialized():
        s.finalize()
    s.init(n_local=1, heap_size="2G", ROCSHMEM_WAIT_TIMEOUT_MS=5000)
    yield s
    torch.cuda.synchronize()
    s.finalize()


def clean(shm):
    torch.cuda.synchronize()
    err = shm.get_error(0)
    assert err["count"] == 0, err


@pytest.mark.parametrize("quantize", [True, False])
@pytest.mark.parametrize("E,K,H,I,T", [(8, 2, 1024, 512, 200), (16, 8, 2048, 256, 333)])
def test_moe_feed_forward(shm, quantize, E, K, H, I, T):
    """bf16 experts: behind a quantised dispatch (rows de-quantised into expert order by one kernel) and behind a bf16
    dispatch (rows gathered inside the GEMM)."""
    from rocshmem_b200.models import moe_ffn
    from rocshmem_b200.ops import gemm, moe
    layer = moe_ffn.MoEFeedForward(E, K, H, I, max_tokens=T + 5, quantize=quantize, seed=2, fp8_experts=False)
    for rep in range(2):
        x = torch.randn(T, H, generator=torch.Generator().manual_seed(rep + 1)).to(torch.bfloat16)
        idx, w = moe.make_routing(T, E, K, seed=50 + rep)
        if rep:
            idx[::6, -1] = -1
        before = gemm.gemm_error_count()
        out = layer(x.cuda(), idx.cuda(), w.cuda())
        clean(shm)
        assert gemm.gemm_error_count() == before
        want = moe_ffn.reference_forward(x, idx, w, H, I, seed=2, quantize=quantize)
        err = (out.float().cpu() - want).abs().max().item()
        assert err <= 3e-2 * want.abs().max().item() + 0.02, (rep, err, want.abs().max().item())
    layer.destroy()


@pytest.mark.parametrize("d_model,d_ff,m", [(1024, 512, 256), (2048, 1280, 384)])
def test_tp_mlp_single_rank(shm, d_model, d_ff, m):
    from rocshmem_b200.models import tp_mlp
    from rocshmem_b200.ops import gemm
    mlp = tp_mlp.TensorParallelMLP(d_model, d_ff, m, seed=4)
    x = (torch.randn(m, d_model, generator=torch.Generator().manual_seed(9)) * 0.5).to(torch.bfloat16)
    want = tp_mlp.reference_forward(x, 1, d_model, d_ff, seed=4)
    for rep in range(2):
        before = gemm.gemm_error_count()
        out = mlp(x.cuda())
        clean(shm)
        assert gemm.gemm_error_count() == before
        err = (out.float().cpu() - want).abs().max().item()
        assert err <= 2e-2 * want.abs().max().item() + 0.05, (rep, err)


def test_moe_feed_forward_fp8_experts(shm):
    """e4m3 rows from the dispatch feed block-scaled fp8 grouped GEMMs directly (the default where shapes allow)."""
    from rocshmem_b200.models import moe_ffn
    from rocshmem_b200.ops import gemm, moe
    E, K, H, I, T = 8, 2, 1024, 512, 300
    layer = moe_ffn.MoEFeedForward(E, K, H, I, max_tokens=T, seed=6)
    assert layer.fp8_experts
    for rep in range(2):
        x = torch.randn(T, H, generator=torch.Generator().manual_seed(rep + 20)).to(torch.bfloat16)
        idx, w = moe.make_routing(T, E, K, seed=70 + rep)
        before = gemm.gemm_error_count()
        out = layer(x.cuda(), idx.cuda(), w.cuda())
        clean(shm)
        assert gemm.gemm_error_count() == before
        want = moe_ffn.reference_forward(x, idx, w, H, I, seed=6, fp8_experts=True)
        err = (out.float().cpu() - want).abs().max().item()
        # the hidden activation is re-quantised from slightly different bf16 values than the reference's
        assert err <= 5e-2 * want.abs().max().item() + 0.03, (rep, err, want.abs().max().item())


@pytest.mark.parametrize("d_model,d_ff,m", [(1024, 512, 256), (2048, 1536, 384)])
def test_tp_mlp_fp8_single_rank(shm, d_model, d_ff, m):
    from rocshmem_b200.models import tp_mlp
    from rocshmem_b200.ops import gemm
    mlp = tp_mlp.TensorParallelMLPFp8(d_model, d_ff, m, seed=4)
    x = (torch.randn(m, d_model, generator=torch.Generator().manual_seed(9)) * 0.5).to(torch.bfloat16)
    want = tp_mlp.reference_forward_fp8(x, 1, d_model, d_ff, seed=4)
    for rep in range(2):
        before = gemm.gemm_error_count()
        out = mlp(x.cuda())
        clean(shm)
        assert gemm.gemm_error_count() == before
        err = (out.float().cpu() - want).abs().max().item()
        assert err <= 5e-2 * want.abs().max().item() + 0.05, (rep, err)


@pytest.mark.parametrize("m", [256, 384])
def test_tp_mlp_alone_reads_the_rows_where_they_are(shm, m):
    """A team of one: rows in ordinary memory, strided rows and results that share memory with an operand give what the
    input buffer gives, and the rows are the input buffer's content afterwards."""
    from rocshmem_b200.models import tp_mlp
    from rocshmem_b200.ops import gemm
    d = 512
    mlp = tp_mlp.TensorParallelMLP(d, d, m, seed=4)
    x = (torch.randn(m, d, generator=torch.Generator().manual_seed(m)) * 0.5).to(torch.bfloat16).cuda()
    mlp.input_buffer().copy_(x)
    want = mlp().clone()
    mlp.input_buffer().zero_()
    assert torch.equal(mlp(x), want)
    assert torch.equal(mlp.input_buffer(), x)
    assert torch.equal(mlp(x.t().contiguous().t()), want)          # strided: copied first
    assert torch.equal(mlp(x.float()), want)                       # another type: converted first
    y = x.clone()
    assert mlp(y, out=y) is y and torch.equal(y, want)
    # The two kernels with their result over an operand.
    h = mlp.tp.ag_gemm(mlp.w_gate_up, swiglu=True).clone()
    mlp.tp.ag_gemm(mlp.w_gate_up, out=mlp.input_buffer(), swiglu=True)
    assert torch.equal(mlp.input_buffer(), h)
    assert torch.equal(mlp.tp.gemm_rs(h, mlp.w_down, out=h), want)
    # The rows given, and the result over the input buffer, or rows and input buffer sharing some of their memory: the
    # rows become the buffer's content first, then the result is written.
    hidden = mlp.tp.ag_gemm(mlp.w_gate_up, swiglu=True, x=x)
    for rep in range(3):
        mlp.tp.ag_gemm(mlp.w_gate_up, out=mlp.input_buffer(), swiglu=True, x=x)
        assert torch.equal(mlp.input_buffer(), hidden)
    both = shm.zeros((m + 8, d), torch.bfloat16)
    tp = gemm.TensorParallelLinear(m)
    own = tp._ag_buffers(d)[0]
    tp._ag_buffers(d)[0] = both[:m]
    for first in (0, 8):
        both[8:].copy_(x)
        got = tp.ag_gemm(mlp.w_gate_up, out=both[first:first + m], swiglu=True, x=both[8:])
        assert torch.equal(got, hidden)
        assert first == 0 or torch.equal(both[:8], x[:8])
    clean(shm)
    tp._ag_buffers(d)[0] = own
    tp.destroy()
    shm.free(both)
    # A call on another stream than the current one: in place where that stream is made current, else copied on it.
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        out = mlp(x)
    torch.cuda.synchronize()
    assert torch.equal(out, want)
    # The call's stream is busy with a call that still has to read the input buffer, and the rows are late.
    other = (x.float() * 0.5).to(torch.bfloat16)
    mlp.input_buffer().copy_(other)
    want_other = mlp().clone()
    late, first, out = (torch.empty_like(x) for _ in range(3))
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        torch.cuda._sleep(20_000_000)          # about 10 ms
    mlp(out=first, stream=side)                # the buffer holds `other`
    torch.cuda._sleep(60_000_000)
    late.copy_(x)
    mlp(late, out=out, stream=side)
    assert not side.query()
    torch.cuda.synchronize()
    assert torch.equal(first, want_other)
    assert torch.equal(mlp.input_buffer(), x)
    clean(shm)
    assert torch.equal(out, want)
    mlp.destroy()


@pytest.mark.parametrize("T", [1, 149, 700])
@pytest.mark.parametrize("H,K,quantize", [(512, 3, True), (4096, 8, True), (4608, 1, True), (7168, 8, True),
                                          (512, 8, False), (4096, 6, False), (8192, 2, False)])
def test_dispatch_and_combine_of_a_rank_on_its_own(shm, T, H, K, quantize):
    """A team of one streams its rows: sizes around the stream's batches (16 vectors a lane: 4096 elements), fewer and
    more tokens than blocks, tokens without an expert. Rows, scales and records come out exactly; the combined rows are
    one fp32 product rounded to bf16."""
    from rocshmem_b200.ops import moe
    E = 16
    g = torch.Generator().manual_seed(T * 7 + H)
    x = torch.randn(T, H, generator=g).to(torch.bfloat16).cuda()
    idx, w = moe.make_routing(T, E, K, T + H)
    idx[::5, -1] = -1
    if T > 3:
        idx[3] = -1
    idx, w = idx.cuda(), w.cuda()
    d = moe.EpDispatcher(E, K, H, max(T, 200), quantize=quantize)
    used = (idx >= 0).any(dim=1)
    n = int(used.sum())
    for rep in range(2):
        r = d.dispatch(x, idx, w)
        clean(shm)
        assert r.num_rows() == n and r.row_ranges() == [(0, n)]
        assert torch.equal(r.src_token()[:n].long(), used.nonzero().flatten())
        assert torch.equal(r.local_expert_idx()[:n], idx[used])
        assert torch.equal(r.gate_weights()[:n], w[used])
        assert torch.equal(r.rows_per_expert()[:E].long(), torch.bincount(idx[idx >= 0].long(), minlength=E))
        if quantize:
            q, s = moe.fp8_quantize_1x128(x[used])
            assert torch.equal(r.recv_x[:n].view(torch.uint8), q.view(torch.uint8))
            assert torch.equal(r.recv_scales[:n], s)
        else:
            assert torch.equal(r.recv_x[:n], x[used])
        y = d.result_buffer()
        y[:n].copy_(torch.randn(n, H, generator=g).to(torch.bfloat16))
        gate = torch.where(idx >= 0, w, torch.zeros_like(w)).sum(dim=1)
        for weighted in (True, False):
            out = d.combine(y, idx, w, T, weighted=weighted)
            want = torch.zeros(T, H, device="cuda")
            want[used] = y[:n].float() * (gate[used, None] if weighted else 1.0)
            clean(shm)
            assert (out.float() - want).abs().max().item() <= 2 ** -8 * want.abs().max().item()   # one bf16 rounding
    d.destroy()


@pytest.mark.parametrize("quantize", [True, False])
@pytest.mark.parametrize("T", [1, 37, 128])
def test_moe_feed_forward_low_latency_alone(shm, quantize, T):
    """Low-latency mode of a rank on its own: the dispatch kernel clears the result rows that the down projection adds
    into, so a second call on the same layer is not added to the first."""
    from rocshmem_b200.models import moe_ffn
    from rocshmem_b200.ops import gemm, moe
    E, K, H, I = 8, 3, 1024, 512
    layer = moe_ffn.MoEFeedForward(E, K, H, I, max_tokens=128, seed=2, quantize=quantize, low_latency=True)
    for rep in range(3):
        x = torch.randn(T, H, generator=torch.Generator().manual_seed(T + rep)).to(torch.bfloat16)
        idx, w = moe.make_routing(T, E, K, seed=T + rep)
        if T > 1:
            idx[rep, :] = -1                     # a token without an expert: its row is zero
        want = moe_ffn.reference_forward(x, idx, w, H, I, seed=2, quantize=quantize, fp8_experts=quantize)
        before = gemm.gemm_error_count()
        out = layer(x.cuda(), idx.cuda(), w.cuda()).float().cpu()
        clean(shm)
        assert gemm.gemm_error_count() == before
        assert (out - want).abs().max().item() <= 5e-2 * want.abs().max().item() + 0.05
    layer.destroy()


@pytest.mark.parametrize("dynamic", [False, True])
def test_refused_zero_result_leaves_the_dispatcher_usable(shm, dynamic):
    """zero_result belongs to low-latency mode: elsewhere it is refused, and the calls after it work."""
    from rocshmem_b200.ops import moe
    T, E, K, H = 40, 8, 2, 512
    x = torch.randn(T, H, generator=torch.Generator().manual_seed(1)).to(torch.bfloat16).cuda()
    idx, w = (t.cuda() for t in moe.make_routing(T, E, K, 3))
    d = moe.EpDispatcher(E, K, H, T, quantize=False, dynamic=dynamic)
    assert not d.dynamic and not hasattr(d, "stage_meta")      # nothing to hand out on a team of one
    for rep in range(3):
        with pytest.raises(ValueError):
            d.dispatch(x, idx, w, zero_result=True)
        r = d.dispatch(x, idx, w)
        clean(shm)
        assert r.num_rows() == T and torch.equal(r.recv_x[:T], x)
        assert torch.equal(r.rows_per_expert()[:E].long(), torch.bincount(idx.flatten().long(), minlength=E))
    d.destroy()
