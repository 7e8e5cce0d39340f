"""The library's allreduce and push kernels by team size and payload: teams of up to four and of more members
take different reduction loops, payloads that are whole 16-byte vectors another copy than others, and a process with one
PE another order of the destinations than one with several."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[1, 2, 3, 4, 6, 8])
def shm(request):
    import rocshmem_b200 as s
    if s.is_initialized():
        s.finalize()
    s.init(n_local=request.param, heap_size="64M", ROCSHMEM_WAIT_TIMEOUT_MS=5000)
    yield s
    torch.cuda.synchronize()
    s.finalize()


def clean(shm, n):
    torch.cuda.synchronize()
    for l in range(n):
        assert shm.get_error(l)["count"] == 0


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.int32])
@pytest.mark.parametrize("elems", [3, 1024, 1027, 40000, 300001])
def test_allreduce_and_pushes(shm, dtype, elems):
    from rocshmem_b200.ops import collectives as coll
    n = shm.n_local_pes()
    g = torch.Generator().manual_seed(elems + n)
    draw = (lambda k: torch.randn(k, generator=g).to(dtype)) if dtype.is_floating_point else (
        lambda k: torch.randint(-1000, 1000, (k,), generator=g).to(dtype))
    src, dst, wide, wide_src = (shm.zeros(k, dtype) for k in (elems, elems, n * elems, n * elems))
    host = [draw(n * elems) for _ in range(n)]
    for l in range(n):
        shm.local_view(src, l).copy_(host[l][:elems])
        shm.local_view(wide_src, l).copy_(host[l])
    torch.cuda.synchronize()
    want = sum(h[:elems].double() for h in host)
    size = sum(h[:elems].double().abs() for h in host)
    # n - 1 additions in fp32, then one rounding to bf16
    tol = {torch.float32: n * 2.0 ** -24, torch.bfloat16: 2.0 ** -8, torch.int32: 0.0}[dtype] * size
    for algo in (shm.ALLREDUCE_AUTO, shm.ALLREDUCE_ONE_SHOT, shm.ALLREDUCE_TWO_SHOT):
        coll.allreduce_async(dst, src, algo=algo)
        clean(shm, n)
        for l in range(n):
            got = shm.local_view(dst, l).double().cpu()
            assert ((got - want).abs() <= tol).all(), (algo, l)
    coll.fcollect_async(wide, src)
    clean(shm, n)
    for l in range(n):
        assert torch.equal(shm.local_view(wide, l).cpu(), torch.cat([h[:elems] for h in host]))
    coll.alltoall_async(wide, wide_src)
    clean(shm, n)
    for l in range(n):
        assert torch.equal(shm.local_view(wide, l).cpu(), torch.cat([h[l * elems:(l + 1) * elems] for h in host]))
    root = n - 1
    for l in range(n):
        shm.local_view(dst, l).fill_(5)
    torch.cuda.synchronize()
    coll.broadcast_async(dst, src, root)
    clean(shm, n)
    for l in range(n):
        assert torch.equal(shm.local_view(dst, l).cpu(), host[root][:elems] if l != root else torch.full((elems,), 5, dtype=dtype))
    shm.free_all([src, dst, wide, wide_src])
