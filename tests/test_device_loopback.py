"""Device kernels on ONE GPU: all ranks are emulated as rows of one cooperative
launch (a loopback world), results are compared bit for bit with the native
host reducer (rank-ascending order, one rounding for 16-bit floats)."""
import os
import subprocess

import pytest
import torch

pytestmark = pytest.mark.gpu

from stdml_collective_experimental_b200 import DeviceSession, DeviceTimeoutError, _native  # noqa: E402
from stdml_collective_experimental_b200.ops.device import (ALGO_ONESHOT,  # noqa: E402
                                                           ALGO_TWOSHOT, ALGO_TWOSHOT_TMA)
from stdml_collective_experimental_b200.utils.oracle import reduce_many  # noqa: E402

FLOATS = [torch.float32, torch.float64, torch.bfloat16, torch.float16]
INTS = [torch.int8, torch.int16, torch.int32, torch.int64, torch.uint8]


def make_inputs(world, n, dtype, seed, small=False):
    g = torch.Generator().manual_seed(seed)
    outs = []
    for r in range(world):
        if dtype.is_floating_point:
            x = torch.rand(n, generator=g) * 2 - 1
            if small:
                x = x * 0.5 + 1.0  # keeps products away from 0 and inf
            outs.append(x.to(dtype))
        else:
            info = torch.iinfo(dtype)
            lo, hi = max(info.min, -100), min(info.max, 100)
            outs.append(torch.randint(lo, hi + 1, (n,), generator=g).to(dtype))
    return outs


@pytest.fixture(scope="module", params=[1, 2, 4, 8])
def sess(request):
    s = DeviceSession.loopback(request.param, heap_bytes=32 << 20, staging_bytes=1 << 20)
    yield s
    s.close()


@pytest.fixture
def tuned(sess):
    """The same kind of session for one test alone: it may turn any knob."""
    with DeviceSession.loopback(sess.world, heap_bytes=32 << 20, staging_bytes=1 << 20) as s:
        yield s


@pytest.fixture(params=[2, 3, 4, 8])
def job(request):
    """The staging slots of a job (64 MB): tiles of several steps, rings of the full grid."""
    with DeviceSession.loopback(request.param, heap_bytes=20 << 20, staging_bytes=64 << 20) as s:
        yield s


def same(a, b):
    if a.dtype.is_floating_point:
        return torch.equal(a.view(torch.uint8), b.view(torch.uint8)) or torch.equal(a, b)
    return torch.equal(a, b)


@pytest.mark.parametrize("dtype", FLOATS + INTS)
@pytest.mark.parametrize("op", ["sum", "min", "max", "prod", "bit_xor"])
def test_all_reduce_matrix(sess, dtype, op):
    if op == "bit_xor" and dtype.is_floating_point:
        with pytest.raises(ValueError):
            x = [torch.zeros(4, dtype=dtype, device="cuda") for _ in range(sess.world)]
            sess.all_reduce(x if sess.vranks > 1 else x[0], op=op)
        return
    for n in [1, 2, 3, 5, 7, 8, 9, 15, 16, 17, 31, 33, 100, 1024, 4099]:
        host = make_inputs(sess.world, n, dtype, seed=n, small=(op == "prod"))
        want = reduce_many(host, op)
        dev = [h.cuda() for h in host]
        out = [torch.empty_like(d) for d in dev]
        arg = (dev, out) if sess.vranks > 1 else (dev[0], out[0])
        sess.all_reduce(arg[0], out=arg[1], op=op)
        torch.cuda.synchronize()
        sess.check()
        for r in range(sess.world):
            assert same(out[r].cpu(), want), (dtype, op, n, r)
            assert same(dev[r].cpu(), host[r]), "input was modified"
        # in place
        sess.all_reduce(arg[0], op=op)
        torch.cuda.synchronize()
        for r in range(sess.world):
            assert same(dev[r].cpu(), want), (dtype, op, n, r, "in place")


@pytest.mark.parametrize("algo", ["oneshot", "twoshot"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_all_reduce_large_chunked_and_scaled(sess, algo, dtype):
    # 3 MiB+ of data through 1 MiB staging slots: several launches, alternating slots
    n = (3 << 20) // torch.empty((), dtype=dtype).element_size() + 13
    host = make_inputs(sess.world, n, dtype, seed=3)
    scale = 1.0 / sess.world
    want = reduce_many(host, "sum", scale)
    dev = [h.cuda() for h in host]
    arg = dev if sess.vranks > 1 else dev[0]
    sess.all_reduce(arg, op="sum", scale=scale, algo=algo)
    torch.cuda.synchronize()
    sess.check()
    for r in range(sess.world):
        assert same(dev[r].cpu(), want)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.int32])
def test_symmetric_zero_copy_in_place(sess, dtype):
    n = 70001
    host = make_inputs(sess.world, n, dtype, seed=11)
    want = reduce_many(host, "sum")
    sym = sess.symm_empty(n, dtype)
    syms = sym if sess.vranks > 1 else [sym]
    for r in range(sess.world):
        syms[r].copy_(host[r])
    before = sess.launches
    sess.all_reduce(sym)
    torch.cuda.synchronize()
    sess.check()
    assert sess.launches == before + 1
    for r in range(sess.world):
        assert same(syms[r].cpu(), want)
    sess.symm_free(sym)


def test_raw_algorithms_agree(sess):
    n = 50000
    host = make_inputs(sess.world, n, torch.float32, seed=5)
    want = reduce_many(host, "sum", 0.5)
    sym = sess.symm_empty(n, torch.float32)
    syms = sym if sess.vranks > 1 else [sym]
    for blocks in (1, 3, 16):
        src = [h.cuda() for h in host]
        dst = [torch.empty(n, device="cuda") for _ in host]
        a = (src, dst) if sess.vranks > 1 else (src[0], dst[0])
        sess.raw_all_reduce(sym, src=a[0], dst=a[1], algo=ALGO_ONESHOT, blocks=blocks, scale=0.5)
        torch.cuda.synchronize()
        for r in range(sess.world):
            assert same(dst[r].cpu(), want), ("oneshot", blocks)
        dst2 = [torch.empty(n, device="cuda") for _ in host]
        a = (src, dst2) if sess.vranks > 1 else (src[0], dst2[0])
        sess.raw_all_reduce(sym, src=a[0], dst=a[1], algo=ALGO_TWOSHOT, blocks=blocks, scale=0.5)
        torch.cuda.synchronize()
        for r in range(sess.world):
            assert same(dst2[r].cpu(), want), ("twoshot", blocks)
            if sess.world > 1:  # a single GPU copies straight from src to dst
                assert same(syms[r].cpu(), want), ("twoshot leaves the result in the arena",
                                                   blocks)
    sess.check()
    sess.symm_free(sym)


@pytest.mark.parametrize("dtype,op", [(torch.float32, "sum"), (torch.bfloat16, "sum"),
                                      (torch.float64, "prod"), (torch.int32, "max"),
                                      (torch.uint8, "bit_xor"), (torch.float16, "min")])
def test_bulk_copy_two_shot_matches_the_oracle(sess, dtype, op):
    """The two-shot whose owner pulls tiles with bulk async copies into a shared
    memory ring: every dtype path, grids of 1..16 CTAs per rank, tiles small enough
    that each ring slot is reused many times (both mbarrier parities), ragged
    sizes (partial last tile, partial last vector)."""
    if sess.world == 1:
        pytest.skip("a world of one has no peers to pull from")
    for tile_vec, n, blocks in [(0, 1, 1), (0, 33, 3), (64, 4099, 1), (32, 70_001, 2),
                                (128, 1_000_003, 1), (0, 1_000_003, 16), (64, 262_144, 16)]:
        sess.set_knob("tma_tile_vec", tile_vec)
        host = make_inputs(sess.world, n, dtype, seed=n + blocks, small=(op == "prod"))
        scale = 0.5 if dtype.is_floating_point else None
        want = reduce_many(host, op, 1.0 if scale is None else scale)
        sym = sess.symm_empty(n, dtype)
        src = [h.cuda() for h in host]
        dst = [torch.empty_like(x) for x in src]
        sess.raw_all_reduce(sym, src=src, dst=dst, op=op, algo=ALGO_TWOSHOT_TMA, blocks=blocks,
                            scale=scale)
        torch.cuda.synchronize()
        sess.check()
        for r in range(sess.world):
            assert same(dst[r].cpu(), want), (dtype, op, n, blocks, tile_vec, r)
            assert same(sym[r][:n].cpu(), want), "the result also stays in the symmetric buffer"
        sess.symm_free(sym)
    sess.set_knob("tma_tile_vec", 0)


def test_bulk_copy_two_shot_through_the_public_calls(sess):
    """Staged (several 1 MiB slots, pack and unpack fused) and zero-copy in place."""
    n = (3 << 20) // 4 + 13
    host = make_inputs(sess.world, n, torch.float32, seed=21)
    want = reduce_many(host, "sum", 1.0 / sess.world)
    dev = [h.cuda() for h in host]
    sess.all_reduce(dev if sess.vranks > 1 else dev[0], scale=1.0 / sess.world, algo="twoshot_tma")
    sym = sess.symm_empty(n, torch.float32)
    syms = sym if sess.vranks > 1 else [sym]
    for r in range(sess.world):
        syms[r].copy_(host[r])
    sess.all_reduce(sym, scale=1.0 / sess.world, algo="twoshot_tma")
    torch.cuda.synchronize()
    sess.check()
    for r in range(sess.world):
        assert same(dev[r].cpu(), want) and same(syms[r].cpu(), want)
    sess.symm_free(sym)


def test_f64_scale_keeps_all_its_bits(sess):
    """1/3 is not a float: f64 buffers must be scaled in double, like the host reducer."""
    n = 10_007
    host = make_inputs(sess.world, n, torch.float64, seed=9)
    want = reduce_many(host, "sum", 1.0 / 3.0)
    assert torch.allclose(want, torch.stack(host).sum(0) / 3.0, rtol=1e-15, atol=0)
    for algo in ("oneshot", "twoshot", "twoshot_tma"):
        if sess.world == 1 and algo == "twoshot_tma":
            continue
        dev = [h.cuda() for h in host]
        sess.all_reduce(dev if sess.vranks > 1 else dev[0], scale=1.0 / 3.0, algo=algo)
        torch.cuda.synchronize()
        sess.check()
        for r in range(sess.world):
            assert same(dev[r].cpu(), want), algo


def test_kernel_refuses_arguments_that_fail_its_own_checks():
    """With debug checks on, a kernel handed a misaligned offset (or one inside the
    signal pad) reports kStatusBadArgs and touches nothing; recover() clears it."""
    with DeviceSession.loopback(2, heap_bytes=8 << 20, staging_bytes=1 << 20) as s:
        for inject, algo in [(1, ALGO_TWOSHOT), (2, ALGO_TWOSHOT_TMA), (1, ALGO_ONESHOT)]:
            sym = s.symm_empty(4096, torch.float32)
            src = [torch.ones(4096, device="cuda") for _ in range(2)]
            dst = [torch.full((4096,), -7.0, device="cuda") for _ in range(2)]
            for t in sym:
                t.fill_(3.0)
            s.set_knob("debug_inject", inject)
            s.raw_all_reduce(sym, src=src, dst=dst, algo=algo, blocks=2)
            torch.cuda.synchronize()
            assert s.status()[0] == 2  # kStatusBadArgs
            with pytest.raises(ValueError):
                s.check()
            assert all(bool((d == -7.0).all()) for d in dst) and all(bool((t == 3.0).all()) for t in sym)
            s.recover()
            assert s.status()[0] == 0
            # and the same call runs normally afterwards, with the checks on
            s.set_knob("debug_checks", 1)
            s.raw_all_reduce(sym, src=src, dst=dst, algo=algo, blocks=2)
            torch.cuda.synchronize()
            s.check()
            assert bool((dst[0] == 2.0).all()) and bool((dst[1] == 2.0).all())
            s.set_knob("debug_checks", 0)
            s.symm_free(sym)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_group_all_reduce_fused(sess, dtype):
    sizes = [1, 7, 768, 3, 2304, 590_000, 5, 64, 1000, 123_457, 2, 768]
    g = torch.Generator().manual_seed(1)
    host = [[(torch.rand(n, generator=g) * 2 - 1).to(dtype) for n in sizes]
            for _ in range(sess.world)]
    scale = 1.0 / sess.world
    want = [reduce_many([host[r][i] for r in range(sess.world)], "sum", scale)
            for i in range(len(sizes))]
    dev = [[t.cuda() for t in host[r]] for r in range(sess.world)]
    before = sess.launches
    sess.group_all_reduce(dev if sess.vranks > 1 else dev[0], scale=scale)
    torch.cuda.synchronize()
    sess.check()
    launches = sess.launches - before
    total_bytes = sum((n * host[0][0].element_size() + 15) // 16 * 16 for n in sizes)
    assert launches == -(-total_bytes // sess.staging_bytes), "one launch per staging slot"
    for r in range(sess.world):
        for i in range(len(sizes)):
            assert same(dev[r][i].cpu(), want[i]), (r, i)
    # second call hits the cached descriptor table
    sess.group_all_reduce(dev if sess.vranks > 1 else dev[0])
    torch.cuda.synchronize()
    sess.check()


@pytest.mark.parametrize("bulk", [False, True, "short tiles"])
@pytest.mark.parametrize("dtype,op,scale", [
    (torch.float32, "sum", 0.125), (torch.bfloat16, "sum", None), (torch.int32, "max", None),
    (torch.float64, "prod", 1.0 / 3.0), (torch.int8, "bit_xor", None), (torch.float16, "min", None),
])
def test_group_all_reduce_on_registered_loose_tensors(tuned, dtype, op, scale, bulk):
    """Separately allocated tensors, reduced where they lie: one launch, no staging.
    `bulk`: operands come in by bulk asynchronous copies into a shared-memory ring
    (the default from 4 MB up), else by 16-byte peer loads."""
    if tuned.world == 1:
        pytest.skip("needs peers")
    tuned.set_knob("group_bulk_min_bytes", 0 if bulk else -1)
    if bulk == "short tiles":  # more chunks of tiles than blocks: most are drawn by ticket
        tuned.set_knob("tma_tile_vec", 32)
    sizes = [1, 7, 768, 3, 2304, 590_000, 5, 64, 1000, 123_457, 2, 768]
    host = [[make_inputs(1, n, dtype, seed=31 * r + i, small=op == "prod")[0]
             for i, n in enumerate(sizes)] for r in range(tuned.world)]
    want = [reduce_many([host[r][i] for r in range(tuned.world)], op, scale)
            for i in range(len(sizes))]
    tuned.set_knob("register_min_bytes", 0)
    # in place, twice (the second call reuses the table of peer pointers)
    for _ in range(2):
        dev = [[t.cuda() for t in host[r]] for r in range(tuned.world)]
        before = tuned.launches
        tuned.group_all_reduce(dev if tuned.vranks > 1 else dev[0], op=op, scale=scale)
        torch.cuda.synchronize()
        tuned.check()
        assert tuned.launches == before + 1
        for r in range(tuned.world):
            for i in range(len(sizes)):
                assert same(dev[r][i].cpu(), want[i]), (r, i)
    # out of place: inputs stay, outputs carry the result and nothing beyond their end
    dev = [[t.cuda() for t in host[r]] for r in range(tuned.world)]
    pad = 16
    outs = [[torch.full((n + pad,), 3, dtype=dtype, device="cuda") for n in sizes]
            for _ in range(tuned.world)]
    views = [[o[:n] for o, n in zip(outs[r], sizes)] for r in range(tuned.world)]
    before = tuned.launches
    tuned.group_all_reduce(dev if tuned.vranks > 1 else dev[0],
                          outs=views if tuned.vranks > 1 else views[0], op=op, scale=scale)
    torch.cuda.synchronize()
    tuned.check()
    assert tuned.launches == before + 1
    for r in range(tuned.world):
        for i, n in enumerate(sizes):
            assert same(views[r][i].cpu(), want[i]), (r, i)
            assert bool((outs[r][i][n:] == 3).all()), "wrote past the end of a tensor"
            assert torch.equal(dev[r][i].cpu(), host[r][i]), "inputs must stay untouched"
    # a tensor that does not start on a 16-byte boundary sends the set the staged way
    dev = [[t.cuda() for t in host[r]] for r in range(tuned.world)]
    for r in range(tuned.world):
        odd = torch.empty(sizes[5] + 1, dtype=dtype, device="cuda")[1:]
        if odd.data_ptr() % 16 != 0:
            odd.copy_(host[r][5])
            dev[r][5] = odd
    before = tuned.launches
    tuned.group_all_reduce(dev if tuned.vranks > 1 else dev[0], op=op, scale=scale)
    torch.cuda.synchronize()
    tuned.check()
    assert tuned.launches > before
    for r in range(tuned.world):
        for i in range(len(sizes)):
            assert same(dev[r][i].cpu(), want[i]), (r, i)


def test_group_all_reduce_bf16_wire_for_f32_grads(sess):
    sizes = [5, 4096, 33, 100_000]
    g = torch.Generator().manual_seed(2)
    host = [[torch.rand(n, generator=g) * 2 - 1 for n in sizes] for _ in range(sess.world)]
    scale = 1.0 / sess.world
    dev = [[t.cuda() for t in host[r]] for r in range(sess.world)]
    sess.group_all_reduce(dev if sess.vranks > 1 else dev[0], scale=scale,
                          wire_dtype=torch.bfloat16)
    torch.cuda.synchronize()
    sess.check()
    for i in range(len(sizes)):
        want = reduce_many([host[r][i].to(torch.bfloat16) for r in range(sess.world)], "sum",
                           scale).float()
        for r in range(sess.world):
            assert torch.equal(dev[r][i].cpu(), want), (r, i)


def test_group_zero_copy_flat(sess):
    sizes = [8, 100, 4, 50_000]  # every tensor a multiple of 16 bytes: back to back
    flat = sess.symm_empty(sum(sizes), torch.float32)
    flats = flat if sess.vranks > 1 else [flat]
    g = torch.Generator().manual_seed(7)
    host = [torch.rand(sum(sizes), generator=g) for _ in range(sess.world)]
    for r in range(sess.world):
        flats[r].copy_(host[r])
    views = [list(torch.split(f, sizes)) for f in flats]
    before = sess.launches
    sess.group_all_reduce(views if sess.vranks > 1 else views[0], scale=0.25)
    torch.cuda.synchronize()
    sess.check()
    assert sess.launches == before + 1
    want = reduce_many(host, "sum", 0.25)
    for r in range(sess.world):
        assert same(flats[r].cpu(), want)
    sess.symm_free(flat)


@pytest.mark.parametrize("n", [1, 2, 10, 1000, 300_001])
def test_all_gather(sess, n):
    host = make_inputs(sess.world, n, torch.int32, seed=n)
    dev = [h.cuda() for h in host]
    out = [torch.empty(n * sess.world, dtype=torch.int32, device="cuda") for _ in dev]
    a = (dev, out) if sess.vranks > 1 else (dev[0], out[0])
    sess.all_gather(a[0], a[1])
    torch.cuda.synchronize()
    sess.check()
    want = torch.cat(host)
    for r in range(sess.world):
        assert torch.equal(out[r].cpu(), want)


def test_all_gather_odd_bytes(sess):
    n = 37  # 37 bytes per rank: unaligned destinations
    host = make_inputs(sess.world, n, torch.uint8, seed=9)
    dev = [h.cuda() for h in host]
    out = [torch.empty(n * sess.world, dtype=torch.uint8, device="cuda") for _ in dev]
    a = (dev, out) if sess.vranks > 1 else (dev[0], out[0])
    sess.all_gather(a[0], a[1])
    torch.cuda.synchronize()
    want = torch.cat(host)
    for r in range(sess.world):
        assert torch.equal(out[r].cpu(), want)


@pytest.mark.parametrize("n", [1, 17, 300_001])
def test_broadcast_and_reduce(sess, n):
    host = make_inputs(sess.world, n, torch.float32, seed=n)
    for root in sorted({0, sess.world - 1}):
        dev = [h.cuda() for h in host]
        out = [torch.empty_like(d) for d in dev]
        a = (dev, out) if sess.vranks > 1 else (dev[0], out[0])
        sess.broadcast(a[0], out=a[1], root=root)
        torch.cuda.synchronize()
        for r in range(sess.world):
            assert torch.equal(out[r].cpu(), host[root])
        red = [torch.full_like(d, -7.0) for d in dev]
        a = (dev, red) if sess.vranks > 1 else (dev[0], red[0])
        sess.reduce(a[0], out=a[1], op="sum", root=root)
        torch.cuda.synchronize()
        want = reduce_many(host, "sum")
        for r in range(sess.world):
            if r == root:
                assert same(red[r].cpu(), want)
            else:
                assert torch.all(red[r] == -7.0)
    sess.check()


@pytest.mark.parametrize("n", [4, 1000, 300_004])
def test_zero_copy_all_gather_broadcast_reduce_on_symmetric_buffers(sess, n):
    """Output (all_gather, broadcast) or input (reduce) in the symmetric heap: one
    launch, no staging; blocks are pushed straight into every rank's buffer."""
    w = sess.world
    host = make_inputs(w, n, torch.int32, seed=n + 3)
    out = sess.symm_empty(n * w, torch.int32)
    outs = out if sess.vranks > 1 else [out]
    for o in outs:
        o.fill_(-1)
    ins = [h.cuda() for h in host]
    before = sess.launches
    sess.all_gather(ins if sess.vranks > 1 else ins[0], out)
    torch.cuda.synchronize()
    sess.check()
    assert sess.launches == before + 1 or w == 1  # alone: a plain copy through the slots
    for r in range(w):
        assert torch.equal(outs[r].cpu(), torch.cat(host)), r
    # in place: every rank's block already sits in its own output
    for r in range(w):
        outs[r].fill_(-1)
        outs[r][r * n:(r + 1) * n].copy_(host[r])
    views = [outs[r][r * n:(r + 1) * n] for r in range(w)]
    sess.all_gather(views if sess.vranks > 1 else views[0], out)
    torch.cuda.synchronize()
    for r in range(w):
        assert torch.equal(outs[r].cpu(), torch.cat(host)), (r, "in place")
    sess.symm_free(out)

    for root in sorted({0, w - 1}):
        sym = sess.symm_empty(n, torch.int32)
        syms = sym if sess.vranks > 1 else [sym]
        for r in range(w):
            syms[r].copy_(host[r])
        sess.broadcast(sym, root=root)  # in place on a symmetric buffer
        torch.cuda.synchronize()
        sess.check()
        for r in range(w):
            assert torch.equal(syms[r].cpu(), host[root]), (root, r)
        # from an ordinary tensor on root into symmetric buffers everywhere
        for t in syms:
            t.fill_(-5)
        sess.broadcast(ins if sess.vranks > 1 else ins[0], out=sym, root=root)
        torch.cuda.synchronize()
        for r in range(w):
            assert torch.equal(syms[r].cpu(), host[root]), (root, r, "out of place")
        # reduce: symmetric inputs, ordinary output on root only
        for r in range(w):
            syms[r].copy_(host[r])
        res = [torch.full((n,), -7, dtype=torch.int32, device="cuda") for _ in range(w)]
        sess.reduce(sym, out=res if sess.vranks > 1 else res[0], root=root)
        torch.cuda.synchronize()
        sess.check()
        for r in range(w):
            if r == root:
                assert torch.equal(res[r].cpu(), reduce_many(host, "sum"))
            else:
                assert bool((res[r] == -7).all())
            assert torch.equal(syms[r].cpu(), host[r]), "reduce must leave its inputs alone"
        sess.symm_free(sym)


def test_broadcast_in_rounds(tuned):
    """The pipelined broadcast (root sends in rounds and signals, holders forward
    while root goes on) at sizes from one vector to many rounds, staged and on
    symmetric buffers, from both ends of the rank range."""
    if tuned.world < 3:
        pytest.skip("used from three ranks up")
    tuned.set_knob("bcast_pipelined_min_bytes", 0)
    for n in (1, 17, 5000, 300_001, 2_000_003):
        host = make_inputs(tuned.world, n, torch.float32, seed=n + 1)
        for root in sorted({0, tuned.world - 1}):
            dev = [h.cuda() for h in host]
            tuned.broadcast(dev, root=root)
            if n * 4 <= (4 << 20):
                sym = tuned.symm_empty(n, torch.float32)
                for r in range(tuned.world):
                    sym[r].copy_(host[r])
                tuned.broadcast(sym, root=root)
            torch.cuda.synchronize()
            tuned.check()
            for r in range(tuned.world):
                assert torch.equal(dev[r].cpu(), host[root]), (n, root, r)
                if n * 4 <= (4 << 20):
                    assert torch.equal(sym[r].cpu(), host[root]), (n, root, r, "symmetric")
            if n * 4 <= (4 << 20):
                tuned.symm_free(sym)


@pytest.mark.parametrize("algo_knob", [0, 1 << 40])
def test_all_gather_push_and_pull_agree(tuned, algo_knob):
    tuned.set_knob("gather_push_min_bytes", algo_knob)  # 0: always push; huge: always pull
    for n in (3, 1000, 70_001):
        host = make_inputs(tuned.world, n, torch.int16, seed=n)
        outs = [torch.empty(n * tuned.world, dtype=torch.int16, device="cuda")
                for _ in range(tuned.world)]
        ins = [h.cuda() for h in host]
        tuned.all_gather(ins if tuned.vranks > 1 else ins[0],
                        outs if tuned.vranks > 1 else outs[0])
        torch.cuda.synchronize()
        tuned.check()
        for r in range(tuned.world):
            assert torch.equal(outs[r].cpu(), torch.cat(host)), (n, r)


@pytest.mark.parametrize("dtype,op", [(torch.float32, "sum"), (torch.bfloat16, "sum"),
                                      (torch.int8, "bit_xor"), (torch.float64, "max")])
def test_small_all_reduce_in_one_exchange(sess, dtype, op):
    """Messages that go through the mailboxes: one vector, around a block of threads, the
    largest that fits and one more; twice and more in a row (both mailboxes), between
    other collectives, in the heap, off vector boundaries."""
    if sess.world == 1:
        pytest.skip("needs peers")
    es = torch.empty((), dtype=dtype).element_size()
    lanes = 16 // es
    most = min(32768, 2 * 148 // sess.world * 512) * lanes
    for n in (1, lanes - 1 or 1, 511 * lanes + 1, 512 * lanes, 513 * lanes - 1, most - 1, most, most + 1):
        host = make_inputs(sess.world, n, dtype, seed=n)
        want = reduce_many(host, op, 1.0)
        dev = [h.cuda() for h in host]
        odd = [torch.zeros(n + 1, dtype=dtype, device="cuda")[1:] for _ in host]
        sym = sess.symm_empty(n, dtype)
        for r, h in enumerate(host):
            odd[r].copy_(h)
            sym[r].copy_(h)
        outs = [[torch.empty_like(d) for d in dev] for _ in range(3)]
        sess.all_reduce(dev, out=outs[0], op=op)
        sess.all_reduce(odd, out=outs[1], op=op)
        sess.barrier()
        sess.all_reduce(sym, op=op)
        sess.all_reduce(dev, out=outs[2], op=op)
        sess.all_reduce(odd, op=op)
        torch.cuda.synchronize()
        sess.check()
        for r in range(sess.world):
            for got in [o[r] for o in outs] + [sym[r], odd[r]]:
                assert same(got.cpu(), want), (n, r)
            assert same(dev[r].cpu(), host[r])
        sess.symm_free(sym)


@pytest.mark.parametrize("shift", [0, 4, 5])
@pytest.mark.parametrize("n", [1, 15, 16, 17, 4097, 70_001, 3_000_001])
def test_pull_ring_at_every_alignment(tuned, n, shift):
    """Staged all_gather and broadcast by pull: sizes around a vector, a tile and many
    rounds, sources and destinations that start `shift` bytes off a vector boundary;
    nothing beyond a destination's own bytes may change."""
    if tuned.world == 1:
        pytest.skip("needs peers")
    w = tuned.world
    tuned.set_knob("gather_push_min_bytes", -1)
    tuned.set_knob("bcast_pipelined_min_bytes", -1)
    tuned.set_knob("bcast_push_min_bytes", -1)
    host = make_inputs(w, n, torch.uint8, seed=n)
    ins = [torch.zeros(n + 16, dtype=torch.uint8, device="cuda")[shift:shift + n] for _ in range(w)]
    for t, h in zip(ins, host):
        t.copy_(h)
    pads = [torch.full((n * w + 48,), 7, dtype=torch.uint8, device="cuda") for _ in range(w)]
    outs = [p[16 + shift:16 + shift + n * w] for p in pads]
    tuned.all_gather(ins, outs)
    bpads = [torch.full((n + 48,), 7, dtype=torch.uint8, device="cuda") for _ in range(w)]
    bouts = [p[16 + shift:16 + shift + n] for p in bpads]
    tuned.broadcast(ins, out=bouts, root=w - 1)
    tuned.broadcast(ins, root=0)  # in place
    torch.cuda.synchronize()
    tuned.check()
    for r in range(w):
        assert torch.equal(outs[r].cpu(), torch.cat(host)), r
        assert bool((pads[r][:16 + shift] == 7).all() and (pads[r][16 + shift + n * w:] == 7).all())
        assert torch.equal(bouts[r].cpu(), host[w - 1]), r
        assert bool((bpads[r][:16 + shift] == 7).all() and (bpads[r][16 + shift + n:] == 7).all())
        assert torch.equal(ins[r].cpu(), host[0]), r


@pytest.mark.parametrize("world,root", [(2, None), (3, 1), (8, None), (8, 7), (9, None)])
def test_long_pull_at_the_edges_of_its_rounds(world, root):
    """Messages from the smallest of the long kernel's on, one vector around whole rounds, destinations at
    odd bytes; a ninth rank, whose messages are none of them."""
    per_rank = 2 * 148 // world
    with DeviceSession.loopback(world, heap_bytes=1 << 20, staging_bytes=64 << 20) as s:
        for n in (512 * per_rank * 16 - 33, 512 * per_rank * 16, 1600 * per_rank * 16 + 17, 5_000_003):
            for shift in (0, 3, 16):
                ins = [torch.randint(0, 255, (n + 32,), dtype=torch.uint8, device="cuda")[shift:n + shift]
                       for _ in range(world)]
                total = n if root is not None else n * world
                out = [torch.full((total + 64,), 7, dtype=torch.uint8, device="cuda") for _ in range(world)]
                views = [o[shift:total + shift] for o in out]
                if root is None:
                    s.all_gather(ins, views)
                else:
                    s.broadcast(ins, out=views, root=root)
                torch.cuda.synchronize()
                s.check()
                want = torch.cat(ins) if root is None else ins[root]
                for o, v in zip(out, views):
                    assert torch.equal(v, want), (n, shift)
                    assert bool((o[:shift] == 7).all()) and bool((o[total + shift:] == 7).all())


@pytest.mark.parametrize("push", [False, True])
@pytest.mark.parametrize("n", [17, 70_001, 3_000_001])
def test_ranks_without_a_destination_take_part(sess, n, push):
    """all_gather, broadcast and all_reduce where some ranks pass no output: the others get
    theirs, at sizes from one vector to several slots, and nothing beside the staging slot in
    use changes (a heap tensor between its guard bands, the mailboxes)."""
    if sess.world == 1:
        pytest.skip("needs peers")
    w = sess.world
    with DeviceSession.loopback(w, heap_bytes=1 << 20, staging_bytes=1 << 20) as s:
        for knob in ("gather_push_min_bytes", "bcast_push_min_bytes") if push else ():
            s.set_knob(knob, 0)
        sym = s.symm_empty(70_000, torch.uint8)
        for t in sym:
            t.fill_(9)
        host = make_inputs(w, n, torch.uint8, seed=n)
        ins = [h.cuda() for h in host]
        for absent in ({w - 1}, set(range(1, w))):
            outs = [None if r in absent else torch.zeros(n * w, dtype=torch.uint8, device="cuda")
                    for r in range(w)]
            bouts = [None if r in absent else torch.zeros(n, dtype=torch.uint8, device="cuda")
                     for r in range(w)]
            s.all_gather(ins, outs)
            s.broadcast(ins, out=bouts, root=w - 1)
            routs = [None if r in absent else torch.zeros(n, dtype=torch.uint8, device="cuda")
                     for r in range(w)]
            s.all_reduce(ins, out=routs, op="bit_xor")
            small = [torch.ones(3, device="cuda") for _ in range(w)]
            s.all_reduce(small)
            torch.cuda.synchronize()
            s.check()
            for r in set(range(w)) - absent:
                assert torch.equal(outs[r].cpu(), torch.cat(host)), r
                assert torch.equal(bouts[r].cpu(), host[w - 1]), r
                assert torch.equal(routs[r].cpu(), reduce_many(host, "bit_xor")), r
            for r in range(w):
                assert torch.equal(ins[r].cpu(), host[r])
                assert bool((small[r] == w).all()) and bool((sym[r] == 9).all())
        s.symm_free(sym)  # reads the guard bands


def scattered(world, dtype, aligned, seed):
    """A set of 1100 small tensors among three large ones, 5.3 M elements in all: more entries
    than the kernels search in shared memory, several steps per tile with 64 MB slots; unless
    `aligned`, some tensors start off a vector boundary.  Host copies and device tensors."""
    sizes = [1 + 37 * i % 900 for i in range(1100)]
    sizes[0:0], sizes[500:500], sizes[1100:1100] = [1_500_001], [1_600_000], [1_700_003]
    host = [make_inputs(1, sum(sizes), dtype, seed=seed + r)[0] for r in range(world)]
    dev = []
    for h in host:
        flat = torch.empty(sum(sizes) + 16 * len(sizes), dtype=dtype, device="cuda")
        lanes, at, row = 16 // flat.element_size(), 0, []
        for i, part in enumerate(torch.split(h, sizes)):
            at = -(-at // lanes) * lanes + (0 if aligned or i % 7 else 1)
            row.append(flat[at:at + part.numel()])
            at += part.numel()
            row[-1].copy_(part)
        dev.append(row)
    return host, dev


@pytest.mark.parametrize("dtype,wire", [(torch.float32, None), (torch.float32, torch.bfloat16),
                                        (torch.bfloat16, None)])
def test_staged_group_at_the_slots_of_a_job(job, dtype, wire):
    host, dev = scattered(job.world, dtype, aligned=False, seed=5)
    job.group_all_reduce(dev, scale=0.5, wire_dtype=wire)
    torch.cuda.synchronize()
    job.check()
    want = reduce_many([h.to(wire or dtype) for h in host], "sum", 0.5).to(dtype)
    for r in range(job.world):
        assert same(torch.cat(dev[r]).cpu(), want), r


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.int64])
@pytest.mark.parametrize("world", [3, 4, 8, 16])
def test_longest_one_shot_of_ordinary_tensors(world, dtype):
    """Around the size from which single messages go by rounds instead: the same bits on both sides,
    in and out of place, also off a vector boundary, and from the staged kernel when it is asked for."""
    most = int(((44 if dtype.itemsize >= 4 else 26) << 20) / world ** 1.5) // dtype.itemsize
    with DeviceSession.loopback(world, heap_bytes=1 << 20, staging_bytes=64 << 20) as s:
        for n in (most - 1, most, most + 1):
            host = make_inputs(world, n, dtype, seed=n % 1000)
            want = reduce_many(host, "sum")
            for shift in (0, 1):
                ins = [torch.empty(n + 1, dtype=dtype, device="cuda")[shift:n + shift] for _ in host]
                for t, h in zip(ins, host):
                    t.copy_(h)
                outs = [[torch.zeros(n + 2, dtype=dtype, device="cuda") for _ in host] for _ in range(2)]
                views = [[t[shift:n + shift] for t in side] for side in outs]
                s.all_reduce(ins, out=views[0])
                s.all_reduce(ins, out=views[1], algo="twoshot")
                s.all_reduce(ins)
                torch.cuda.synchronize()
                s.check()
                for r in range(world):
                    for got in (views[0][r], views[1][r], ins[r]):
                        assert same(got.cpu(), want), (n, shift, r)
                    for side in outs:
                        assert not side[r][:shift].any() and not side[r][n + shift:].any(), (n, shift, r)


@pytest.mark.parametrize("world,dtype,wire,slot,n", [
    (3, torch.float32, None, 32, 9_500_003), (8, torch.bfloat16, None, 16, 9_000_001),
    (2, torch.float32, torch.bfloat16, 32, 17_000_005), (16, torch.int32, None, 16, 4_400_001)])
def test_staged_message_of_several_slots_is_one_launch(world, dtype, wire, slot, n):
    """The ring of a full grid fits the slot, so the message may be longer than it."""
    host = make_inputs(world, n, dtype, seed=12)
    sizes = [n // 2, 5, n // 3 + 1, n - n // 2 - n // 3 - 6]
    want = reduce_many([h.to(wire or dtype) for h in host], "sum").to(dtype)
    with DeviceSession.loopback(world, heap_bytes=1 << 20, staging_bytes=slot << 20) as s:
        for shift in (0, 1):
            flat = [torch.empty(n + 1, dtype=dtype, device="cuda")[shift:n + shift] for _ in host]
            for f, h in zip(flat, host):
                f.copy_(h)
            dev = [list(torch.split(f, sizes)) for f in flat]
            before = s.launches
            s.group_all_reduce(dev, wire_dtype=wire)
            assert s.launches == before + 1
            torch.cuda.synchronize()
            s.check()
            for r in range(world):
                assert same(flat[r].cpu(), want), (shift, r)
            if shift == 0 and wire is None:
                for f, h in zip(flat, host):
                    f.copy_(h)
                s.all_reduce(flat)
                torch.cuda.synchronize()
                s.check()
                assert s.launches == before + 2
                assert all(same(f.cpu(), want) for f in flat)


def test_staged_buffer_at_the_slots_of_a_job(job):
    n = 5_300_003
    host = make_inputs(job.world, n, torch.int32, seed=8)
    for odd in (0, 1):
        dev = [torch.empty(n + 1, dtype=torch.int32, device="cuda")[odd:n + odd] for _ in host]
        out = [torch.full((n + 2,), 7, dtype=torch.int32, device="cuda") for _ in host]
        for d, h in zip(dev, host):
            d.copy_(h)
        job.all_reduce(dev, out=[o[odd:n + odd] for o in out], op="max")
        torch.cuda.synchronize()
        job.check()
        for r in range(job.world):
            assert torch.equal(out[r][odd:n + odd].cpu(), reduce_many(host, "max")), (odd, r)
            assert bool((out[r][:odd] == 7).all()) and bool((out[r][n + odd:] == 7).all())


@pytest.mark.parametrize("bulk", [False, True])
def test_registered_set_of_many_tensors(job, bulk):
    """More entries than are searched in shared memory; by bulk copies, most chunks by ticket."""
    job.set_knob("register_min_bytes", 0)
    job.set_knob("group_bulk_min_bytes", 0 if bulk else -1)
    job.set_knob("tma_tile_vec", 64)
    host, dev = scattered(job.world, torch.bfloat16, aligned=True, seed=6)
    before = job.launches
    job.group_all_reduce(dev, scale=0.5)
    torch.cuda.synchronize()
    job.check()
    assert job.launches == before + 1
    want = reduce_many(host, "sum", 0.5)
    for r in range(job.world):
        assert same(torch.cat(dev[r]).cpu(), want), r


@pytest.mark.parametrize("algo", [None, "twoshot", "twoshot_tma"])
def test_tiles_drawn_by_ticket(job, algo):
    """In place, 16 MB per rank: past the size from which blocks draw their tiles; three
    calls in a row, whose counters each call has to leave at zero."""
    n = 4_000_003
    host = make_inputs(job.world, n, torch.float32, seed=12)
    sym = job.symm_empty(n, torch.float32)
    for t, h in zip(sym, host):
        t.copy_(h)
    for _ in range(3):
        job.all_reduce(sym, op="max", algo=algo)
    torch.cuda.synchronize()
    job.check()
    for t in sym:
        assert same(t.cpu(), reduce_many(host, "max"))
    for t, h in zip(sym, host):
        t.copy_(h)
    job.all_reduce(sym, scale=0.5, algo=algo)
    torch.cuda.synchronize()
    job.check()
    for t in sym:
        assert same(t.cpu(), reduce_many(host, "sum", 0.5))
    job.symm_free(sym)


@pytest.mark.parametrize("shift", [0, 5])
def test_pull_at_the_slots_of_a_job(job, shift):
    """all_gather and broadcast of several rounds, by the kernel of long messages, from and to addresses
    `shift` bytes off a vector boundary."""
    w = job.world
    for op, n in (("all_gather", {2: 20_000_003, 3: 14_000_001, 4: 7_000_001, 8: 2_000_003}[w]),
                  ("broadcast", {2: 20_000_003, 3: 27_000_005, 4: 20_000_003, 8: 11_000_001}[w])):
        host = make_inputs(w, n, torch.uint8, seed=n)
        ins = [torch.zeros(n + 16, dtype=torch.uint8, device="cuda")[shift:shift + n] for _ in range(w)]
        for t, h in zip(ins, host):
            t.copy_(h)
        want = (torch.cat(host) if op == "all_gather" else host[w - 1]).cuda()
        pads = [torch.full((want.numel() + 48,), 7, dtype=torch.uint8, device="cuda") for _ in range(w)]
        outs = [p[16 + shift:16 + shift + want.numel()] for p in pads]
        if op == "all_gather":
            job.all_gather(ins, outs)
        else:
            job.broadcast(ins, out=outs, root=w - 1)
        torch.cuda.synchronize()
        job.check()
        for r in range(w):
            assert torch.equal(outs[r], want), (op, r)
            assert bool((pads[r][:16 + shift] == 7).all()), (op, r)
            assert bool((pads[r][16 + shift + want.numel():] == 7).all()), (op, r)
            assert torch.equal(ins[r].cpu(), host[r]), (op, r)


def test_kernels_against_plain_pytorch_arithmetic(sess):
    """An oracle that shares nothing with the library: the same reductions done by
    PyTorch in float32 / float64 on the host.  all_reduce (every algorithm), the
    fused group with the 1/world scale, and the bf16 wire format for f32 tensors."""
    w = sess.world
    g = torch.Generator().manual_seed(42)
    n = 100_003
    host = [torch.rand(n, generator=g) * 2 - 1 for _ in range(w)]
    exact = torch.stack([h.double() for h in host]).sum(0)
    f32 = host[0].clone()
    for h in host[1:]:
        f32 += h  # rank-ascending float32 adds: what the peer-load kernels do
    for algo in ("oneshot", "twoshot") + (("twoshot_tma",) if w > 1 else ()):
        dev = [h.cuda() for h in host]
        sess.all_reduce(dev if sess.vranks > 1 else dev[0], algo=algo)
        torch.cuda.synchronize()
        sess.check()
        for r in range(w):
            assert torch.equal(dev[r].cpu(), f32), algo
            assert torch.allclose(dev[r].cpu().double(), exact, rtol=0, atol=w * 2.0 ** -23)
    sizes = [3, 1000, 70_001, 17]
    hosts = [[torch.rand(m, generator=g) * 2 - 1 for m in sizes] for _ in range(w)]
    dev = [[t.cuda() for t in hosts[r]] for r in range(w)]
    sess.group_all_reduce(dev if sess.vranks > 1 else dev[0], scale=1.0 / w)
    dev16 = [[t.cuda() for t in hosts[r]] for r in range(w)]
    sess.group_all_reduce(dev16 if sess.vranks > 1 else dev16[0], scale=1.0 / w,
                          wire_dtype=torch.bfloat16)
    torch.cuda.synchronize()
    sess.check()
    for i in range(len(sizes)):
        mean = torch.stack([hosts[r][i].double() for r in range(w)]).mean(0)
        for r in range(w):
            assert torch.allclose(dev[r][i].cpu().double(), mean, rtol=0, atol=2.0 ** -22)
            # bf16 wire: every operand rounded to 8 bits of mantissa, then the mean rounded
            assert torch.allclose(dev16[r][i].cpu().double(), mean, rtol=0, atol=3 * 2.0 ** -8)


def test_barrier_and_launch_count(sess):
    before = sess.launches
    for _ in range(5):
        sess.barrier()
    torch.cuda.synchronize()
    sess.check()
    assert sess.launches == before + 5


def test_bounded_wait_reports_and_recovers():
    """A rank that never arrives: the wait runs out, the host reads a status, the
    context stays usable, and after recover() collectives work again."""
    s = DeviceSession.loopback(2, heap_bytes=1 << 20, staging_bytes=1 << 20, wait_timeout_ms=200)
    try:
        s.barrier_rows(1)  # rank 1 is not launched: nothing sets its flag
        torch.cuda.synchronize()
        code, rank, block, peer, phase, want, have = s.status()
        assert code == 1 and rank == 0 and peer == 1 and want == have + 1
        with pytest.raises(DeviceTimeoutError):
            s.all_reduce([torch.ones(4, device="cuda"), torch.ones(4, device="cuda")])
        s.recover()
        assert s.status()[0] == 0
        x = [torch.full((9,), 1.0, device="cuda"), torch.full((9,), 2.0, device="cuda")]
        s.all_reduce(x)
        torch.cuda.synchronize()
        s.check()
        assert torch.all(x[0] == 3.0) and torch.all(x[1] == 3.0)
    finally:
        s.close()


@pytest.mark.parametrize("call", ["all_reduce", "all_gather", "broadcast"])
def test_ring_kernels_give_up(call):
    """The last rank takes no part in a call of many rounds: the waits for its flag run out, every warp
    leaves, the host reads which rank was missing, and after recover() the same call gets through."""
    w, n = 3, 3_000_001
    with DeviceSession.loopback(w, heap_bytes=1 << 20, staging_bytes=32 << 20, wait_timeout_ms=200) as s:
        host = make_inputs(w, n, torch.float32, seed=9)
        ins = [h.cuda() for h in host]
        out = [torch.zeros(n * w if call == "all_gather" else n, device="cuda") for _ in range(w)]

        def run():
            if call == "all_reduce":
                s.all_reduce(ins, out=out)
            elif call == "all_gather":
                s.all_gather(ins, out)
            else:
                s.broadcast(ins, out=out, root=0)

        run()
        torch.cuda.synchronize()
        s.check()
        s.set_knob("debug_absent", 1)
        ends = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        ends[0].record()
        run()
        ends[1].record()
        torch.cuda.synchronize()
        code, rank, block, peer, phase, want, have = s.status()
        assert code == 1 and rank in (0, 1) and peer == 2 and phase == 0 and want == have + 1
        # (a warp that waited for copies that it never asked for would add a quarter of the timeout)
        assert 200 < ends[0].elapsed_time(ends[1]) < 235
        with pytest.raises(DeviceTimeoutError):
            run()
        s.recover()
        for o in out:
            o.zero_()
        run()
        torch.cuda.synchronize()
        s.check()
        want = {"all_reduce": reduce_many(host, "sum"), "all_gather": torch.cat(host), "broadcast": host[0]}[call]
        for r in range(w):
            assert same(out[r].cpu(), want) and same(ins[r].cpu(), host[r]), r


def test_waits_between_the_warps_of_a_block():
    prog = os.path.join(_native.CSRC, "build", "bin", "test_ring_sync_cuda")
    if not os.path.exists(prog):
        pytest.skip("needs the C++ programs (make -C csrc)")
    res = subprocess.run([prog], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=120)
    assert res.returncode == 0 and "test-ring-sync: OK" in res.stdout, res.stdout


def test_profile_summary_counts_device_time(sess):
    sess.enable_profile()
    x = [torch.ones(100_000, device="cuda") for _ in range(sess.world)]
    arg = x if sess.vranks > 1 else x[0]
    for _ in range(3):
        sess.all_reduce(arg)
    out = [torch.empty(100_000 * sess.world, device="cuda") for _ in range(sess.world)]
    sess.all_gather(arg, out if sess.vranks > 1 else out[0])
    summary = sess.profile_summary()
    sess.enable_profile(False)
    assert summary["all_reduce"]["calls"] == 3 and summary["all_reduce"]["bytes"] == 3 * 400_000
    assert summary["all_reduce"]["ms"] > 0 and summary["all_gather"]["calls"] == 1
    assert sess.profile_summary() == {}


def test_cuda_graph_capture_and_replay():
    """Collectives are plain kernel launches with device-side epochs: a captured
    graph replays them (world 1: no cooperative launch inside the capture)."""
    with DeviceSession.loopback(1, heap_bytes=1 << 20, staging_bytes=1 << 20) as s:
        sym = s.symm_empty(1000, torch.float32)
        user = torch.empty(1000, device="cuda")
        s.all_reduce(sym, scale=0.5)
        s.all_reduce(user, scale=2.0)
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        cap = torch.cuda.Stream()
        with torch.cuda.stream(cap):
            with torch.cuda.graph(g, stream=cap):
                s.all_reduce(sym, scale=0.5, stream=cap)
                s.all_reduce(user, scale=2.0, stream=cap)
        for it in range(3):
            sym.fill_(4.0 + it)
            user.fill_(1.0 + it)
            torch.cuda.synchronize()
            g.replay()
            torch.cuda.synchronize()
            s.check()
            assert torch.all(sym == (4.0 + it) / 2) and torch.all(user == 2.0 * (1.0 + it))


@pytest.mark.parametrize("staging", [4096, 20_000, 300_000])
@pytest.mark.parametrize("world", [3, 8, 16])
def test_slots_too_small_for_a_ring(world, staging):
    """Every staged collective with slots of a few KB: too small for any ring, for the ring of
    several blocks, for a whole message."""
    with DeviceSession.loopback(world, heap_bytes=1 << 20, staging_bytes=staging) as s:
        for n in (1, 1000, 300_007):
            host = make_inputs(world, n, torch.int32, seed=n)
            want = reduce_many(host, "sum")
            ins = [h.cuda() for h in host]
            out, bc, red = ([torch.zeros_like(t) for t in ins] for _ in range(3))
            ag = [torch.zeros(n * world, dtype=torch.int32, device="cuda") for _ in ins]
            group = [list(torch.split(t.clone(), n // 7 + 1)) for t in ins]
            s.all_reduce(ins, out=out)
            s.all_gather(ins, ag)
            s.broadcast(ins, out=bc, root=world - 1)
            s.reduce(ins, out=red, root=1)
            s.group_all_reduce(group)
            torch.cuda.synchronize()
            s.check()
            assert torch.equal(red[1].cpu(), want), n
            for r in range(world):
                assert torch.equal(out[r].cpu(), want), (n, r)
                assert torch.equal(ag[r].cpu(), torch.cat(host)), (n, r)
                assert torch.equal(bc[r].cpu(), host[world - 1]), (n, r)
                assert torch.equal(torch.cat(group[r]).cpu(), want), (n, r)


@pytest.mark.parametrize("n", [3, 70_001, 2_000_003])
def test_staged_collectives_of_several_ranks_in_a_graph(n):
    """Mailboxes, staged rounds and the pull rings replayed from a graph, between ordinary
    calls that use the same slots and mailboxes."""
    w = 4
    with DeviceSession.loopback(w, heap_bytes=1 << 20, staging_bytes=1 << 20) as s:
        ins, out, bc = ([torch.zeros(n, device="cuda") for _ in range(w)] for _ in range(3))
        ag = [torch.zeros(n * w, device="cuda") for _ in range(w)]
        group = [list(torch.split(torch.zeros(n, device="cuda"), n // 3 + 1)) for _ in range(w)]

        def calls(stream=None):
            s.all_reduce(ins, out=out, stream=stream)
            s.all_gather(ins, ag, stream=stream)
            s.broadcast(ins, out=bc, root=2, stream=stream)
            s.group_all_reduce(group, stream=stream)

        calls()  # the group's table is made outside the capture
        torch.cuda.synchronize()
        g, cap = torch.cuda.CUDAGraph(), torch.cuda.Stream()
        with torch.cuda.graph(g, stream=cap):
            calls(cap)
        for it in range(3):
            for r in range(w):
                ins[r].fill_(r + it)
                for t in group[r]:
                    t.fill_(r + it)
            g.replay()
            torch.cuda.synchronize()
            s.check()
            total = float(sum(r + it for r in range(w)))
            for r in range(w):
                assert bool((out[r] == total).all()) and bool((bc[r] == 2.0 + it).all()), (it, r)
                assert torch.equal(ag[r], torch.cat(ins)), (it, r)
                assert all(bool((t == total).all()) for t in group[r]), (it, r)
            s.all_reduce(ins, out=out)
            s.broadcast(ins, out=bc)
        torch.cuda.synchronize()
        s.check()


@pytest.mark.parametrize("world,n", [(2, 7_000_001), (3, 3_000_001), (8, 2_500_003)])
def test_ring_kernels_of_many_rounds_in_a_graph(world, n):
    """Messages of more than a slot, each in one launch, out of place, with a rank without a destination:
    replayed back to back from a graph, between ordinary calls that use the same slots.  At these sizes
    and slots all_gather and broadcast go by the kernel of long messages."""
    with DeviceSession.loopback(world, heap_bytes=1 << 20, staging_bytes=8 << 20) as s:
        base = (torch.arange(n, device="cuda") % 1009).float()
        ins = [torch.empty(n, device="cuda") for _ in range(world)]
        blank = [None if r == world - 1 else r for r in range(world)]
        out, bc, ag = ([None if r is None else torch.empty(m, device="cuda") for r in blank] for m in (n, n, n * world))
        cuts = [n // 3 + 1, 5, n - n // 3 - 6]
        group_out = [torch.empty(n, device="cuda") for _ in range(world)]
        lists = [[list(torch.split(t, cuts)) for t in side] for side in (ins, group_out)]

        def calls(stream=None):
            s.all_reduce(ins, out=out, stream=stream)
            s.all_gather(ins, ag, stream=stream)
            s.broadcast(ins, out=bc, root=0, stream=stream)
            s.group_all_reduce(lists[0], outs=lists[1], stream=stream)

        for t in ins:
            t.zero_()
        calls()  # the group's table is made outside the capture
        torch.cuda.synchronize()
        g, cap = torch.cuda.CUDAGraph(), torch.cuda.Stream()
        before = s.launches
        with torch.cuda.graph(g, stream=cap):
            calls(cap)
        assert s.launches == before + 4
        for it in range(3):
            for r in range(world):
                ins[r].copy_(base * (r + 1) + it)  # (sums of whole numbers below 2^24)
            for t in out + bc + ag + group_out:
                if t is not None:
                    t.fill_(-1)
            g.replay()
            g.replay()
            torch.cuda.synchronize()
            s.check()
            total = sum(t.double() for t in ins).float()
            for r in range(world):
                assert torch.equal(group_out[r], total), (it, r)
                if r < world - 1:
                    assert torch.equal(out[r], total) and torch.equal(bc[r], ins[0]), (it, r)
                    assert torch.equal(ag[r], torch.cat(ins)), (it, r)
            calls()
            s.broadcast(ins, out=bc, root=0)
        torch.cuda.synchronize()
        s.check()


def test_captured_group_outlives_the_plans_of_other_sets():
    """A graph reads its set's descriptor table at every replay; however many other sets
    follow, the bounded cache of plans must not free it."""
    with DeviceSession.loopback(1, heap_bytes=1 << 20, staging_bytes=1 << 20) as s:
        tensors = [torch.zeros(k, device="cuda") for k in (1000, 3, 70_001)]
        s.group_all_reduce(tensors, scale=2.0)  # its table is made outside the capture
        torch.cuda.synchronize()
        g, cap = torch.cuda.CUDAGraph(), torch.cuda.Stream()
        with torch.cuda.graph(g, stream=cap):
            s.group_all_reduce(tensors, scale=2.0, stream=cap)
        others = [[torch.ones(17 + k, device="cuda"), torch.ones(5, device="cuda")] for k in range(200)]
        for o in others:
            s.group_all_reduce(o, scale=3.0)
        for t in tensors:
            t.fill_(1.5)
        g.replay()
        torch.cuda.synchronize()
        s.check()
        assert all(bool((t == 3.0).all()) for o in others for t in o)
        assert all(bool((t == 3.0).all()) for t in tensors)


@pytest.mark.parametrize("world", [2, 4])
def test_large_staged_messages_are_pipelined_on_three_streams(world, monkeypatch):
    """Above a size threshold staged calls run pack / reduce / unpack of successive
    chunks on three streams; the result must not change."""
    monkeypatch.setenv("STDML_COLLECTIVE_PIPELINE_MIN_BYTES", str(1 << 20))
    with DeviceSession.loopback(world, heap_bytes=1 << 20, staging_bytes=1 << 20) as s:
        n = (5 << 20) // 4 + 13
        host = make_inputs(world, n, torch.float32, seed=21)
        want = reduce_many(host, "sum", 0.5)
        dev = [h.cuda() for h in host]
        out = [torch.empty_like(d) for d in dev]
        before = s.launches
        s.all_reduce(dev, out=out, scale=0.5)
        torch.cuda.synchronize()
        s.check()
        assert s.launches - before == 3 * 6 + 1, \
                "6 slot-sized chunks, three launches each, and the barrier that ends a pipeline"
        for r in range(world):
            assert same(out[r].cpu(), want) and same(dev[r].cpu(), host[r])
        # a fused group above the threshold takes the same route
        sizes = [300_000, 7, 500_000, 64, 400_000]
        g = torch.Generator().manual_seed(3)
        hosts = [[torch.rand(k, generator=g) for k in sizes] for _ in range(world)]
        devs = [[t.cuda() for t in hosts[r]] for r in range(world)]
        s.group_all_reduce(devs, scale=1.0 / world)
        s.all_reduce(dev)  # ordinary call right behind the pipeline
        torch.cuda.synchronize()
        s.check()
        for i in range(len(sizes)):
            w = reduce_many([hosts[r][i] for r in range(world)], "sum", 1.0 / world)
            for r in range(world):
                assert same(devs[r][i].cpu(), w), (r, i)
        assert same(dev[0].cpu(), reduce_many(host, "sum"))


def test_group_with_mixed_dtypes_splits_per_dtype(sess):
    g = torch.Generator().manual_seed(4)
    kinds = [torch.float32, torch.bfloat16, torch.float32, torch.int32, torch.bfloat16]
    sizes = [100, 33, 7, 64, 4096]
    host = [[(torch.rand(n, generator=g) * 8).to(dt) for n, dt in zip(sizes, kinds)]
            for _ in range(sess.world)]
    dev = [[t.cuda() for t in host[r]] for r in range(sess.world)]
    sess.group_all_reduce(dev if sess.vranks > 1 else dev[0])
    torch.cuda.synchronize()
    sess.check()
    for i in range(len(sizes)):
        want = reduce_many([host[r][i] for r in range(sess.world)], "sum")
        for r in range(sess.world):
            assert same(dev[r][i].cpu(), want), (r, i)


def test_session_async_interface_on_cuda_tensors():
    """Peer/Session (the C++ session) with device pointers: a single-rank world,
    the returned task polls a CUDA event."""
    from stdml_collective_experimental_b200.parallel import Peer
    peer = Peer.from_list(0, ["127.0.0.1:10990"])
    sess = peer.join()
    x = torch.arange(100_000, dtype=torch.float32, device="cuda")
    y = torch.empty_like(x)
    task = sess.all_reduce_async(x, out=y, name="dev")
    task.wait()
    assert torch.equal(x, y)
    sess.all_reduce(x, op="max")
    gathered = torch.empty(100_000, device="cuda")
    sess.all_gather(x, gathered)
    torch.cuda.synchronize()
    assert torch.equal(gathered, x)
    sess.close()
    peer.close()
