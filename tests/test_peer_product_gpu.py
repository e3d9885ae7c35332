"""Products over several GPUs' shards with every "peer" a buffer of this GPU: the gathered operand, the scattered outputs, and what a
late shard holds up. fp32 sums of bf16 products, outputs rounded to bf16 (2^-9) or kept in fp32 (another order: 1e-5 of the norm)."""
import time

import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return ((a.double() - b).norm() / b.norm()).item()


def _data(rows, K, N, world, seed=0):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    shards = [torch.randn(rows, K, generator=gen, device="cuda").to(torch.bfloat16) for _ in range(world)]
    return shards, (torch.randn(N, K, generator=gen, device="cuda") * K ** -0.5).to(torch.bfloat16)


@pytest.mark.parametrize("rows,K,N,bn", [(128, 64, 64, 64), (200, 136, 200, 128), (328, 384, 576, 192), (1000, 512, 320, 256)])
@pytest.mark.parametrize("world,rank,interleave,chunks", [(2, 0, True, 1), (2, 1, False, 1), (4, 2, False, 3)])
def test_gathered_operand(rows, K, N, bn, world, rank, interleave, chunks):
    from terra_b200.ops.gemm import check_status, gemm

    shards, w = _data(rows, K, N, world)
    flags = torch.full((8 * chunks,), 7, device="cuda", dtype=torch.int32)      # every shard is there
    y = gemm(shards[rank], w, bn=bn, a_peers=[s.data_ptr() for s in shards], rank=rank, a_flags=flags.data_ptr(), a_epoch=7,
             a_interleave=interleave, a_chunks=chunks, a_budget_ns=int(1e9))
    check_status("cuda")
    assert _rel(y, torch.cat(shards).double() @ w.double().t()) < 4e-3


@pytest.mark.parametrize("rows,K,N,world", [(128, 64, 64, 2), (72, 200, 200, 4), (500, 384, 384, 2)])
@pytest.mark.parametrize("f32", [True, False])
def test_scattered_output(rows, K, N, world, f32):
    from terra_b200.ops.gemm import check_status, gemm

    parts, w = _data(rows * world, K, N, 2)
    want = [p.double() @ w.double().t() for p in parts]
    shape = (rows, N) if f32 else (world, rows, N)
    owners = [torch.zeros(shape, device="cuda", dtype=torch.float32 if f32 else torch.bfloat16) for _ in range(world)]
    for rank, p in enumerate(parts):      # two ranks' partial products, one after the other
        gemm(p, w, out=owners[rank], out_peers=[o.data_ptr() for o in owners], rank=rank)
    check_status("cuda")
    for j, o in enumerate(owners):
        block = slice(j * rows, (j + 1) * rows)
        if f32:
            assert _rel(o, want[0][block] + want[1][block]) < 1e-5
        else:
            for rank in range(2):
                assert _rel(o[rank], want[rank][block]) < 4e-3
            assert not o[2:].any()


def test_a_late_shard_holds_up_its_own_stream_only():
    """The kernel waits (for at most a second) for a shard that the host publishes once another stream's product is done: its successor
    on the stream must not have taken the SMs that the wait leaves free."""
    from terra_b200 import _ext
    from terra_b200.ops.gemm import check_status, gemm

    ext = _ext.load()
    shards, w = _data(128, 64, 128, 2)
    (wide,), w2 = _data(148 * 256, 128, 256, 1, seed=1)
    flags = torch.zeros(8, device="cuda", dtype=torch.int32)
    first, late, beside = (torch.empty(*s, device="cuda", dtype=torch.bfloat16) for s in ((256, 128), (148 * 256, 256), (64 * 128, 256)))
    main, other, third = (torch.cuda.Stream() for _ in range(3))

    def run(published):
        flags.fill_(1 if published else 0)
        torch.cuda.synchronize()
        with torch.cuda.stream(main):
            gemm(shards[0], w, bn=128, out=first, a_peers=[s.data_ptr() for s in shards], a_flags=flags.data_ptr(), a_epoch=1,
                 a_budget_ns=int(1e9))
            gemm(wide, w2, bn=256, out=late)
        with torch.cuda.stream(other):
            gemm(wide[:64 * 128], w2, bn=256, out=beside)
        t0 = time.perf_counter()
        other.synchronize()
        took, waiting = time.perf_counter() - t0, not main.query()
        ext.stream_write_value(third.cuda_stream, flags.data_ptr() + 4, 1)
        torch.cuda.synchronize()
        return took, waiting

    run(True)      # every kernel is loaded
    took, waiting = run(False)
    check_status("cuda")
    assert waiting and took < 0.3
    assert _rel(first, torch.cat(shards).double() @ w.double().t()) < 4e-3
    want = wide.double() @ w2.double().t()
    assert _rel(late, want) < 4e-3 and _rel(beside, want[:64 * 128]) < 4e-3
