"""The CUDA table executor with all ranks emulated on one device (a single
cooperative launch), against a plain PyTorch fp32/fp64 reference.  Both data
paths (simt loads/stores and the bulk-copy pipeline) run the same tables."""
import os
import threading

import pytest
import torch

from stragglar_b200 import compiler as sc

pytestmark = pytest.mark.gpu

# simt: every thread moves vectors; tma: the bulk-copy pipeline; simta: the simt data path with control and
# signalling in threads of their own
PATHS = ["simt", "tma", "simta"]


def _inputs(n, count, dtype, dev="cuda:0"):
    from stragglar_b200 import ops
    xs = [torch.empty(count, dtype=dtype, device=dev) for _ in range(n)]
    for r, x in enumerate(xs):
        ops.fill_uniform(x, seed=r)
    torch.cuda.synchronize()
    return xs


def _prephase(xs, alg, straggler):
    n = len(xs)
    non = [r for r in range(n) if r != straggler]
    part = torch.stack([xs[r].float() for r in non]).sum(0).to(xs[0].dtype)
    if alg == "direct":
        for r in non:
            xs[r].copy_(part)
        return
    from helpers import chunk_bounds
    l2p = list(range(n))
    l2p[n - 1], l2p[straggler] = straggler, n - 1
    for i, (b, e) in enumerate(chunk_bounds(xs[0].numel(), xs[0].element_size(), n - 1)):
        xs[l2p[i]][b:e] = part[b:e]


def _run(alg, n, count, dtype=torch.float32, path="simt", prephase=True, straggler=None, scale=1.0, blocks=2,
         tile_bytes=4096, delay_ms=None):
    from stragglar_b200 import ops
    comm = ops.LocalComm(n, emulate=True)
    prog = sc.compile_program(alg, n, prephase, straggler)
    xs = _inputs(n, count, dtype)
    want = torch.stack([x.double() for x in xs]).sum(0) * scale
    if not prephase:
        _prephase(xs, alg, n - 1 if straggler is None else straggler)
    comm.run(prog, xs, path=path, blocks=blocks, tile_bytes=tile_bytes, scale=scale, delay_ms=delay_ms, timeout_s=5.0)
    comm.sync()
    comm.close()
    return xs, want


TOL = {torch.float32: dict(atol=1e-5, rtol=1e-6), torch.bfloat16: dict(atol=6e-2, rtol=2e-2),
       torch.float16: dict(atol=8e-3, rtol=4e-3)}


@pytest.mark.parametrize("path", PATHS)
@pytest.mark.parametrize("alg", ["stragglar", "stragglar_a2a", "ring", "rhd", "direct", "rsag"])
def test_algorithms_n8(alg, path):
    xs, want = _run(alg, 8, 40_003, path=path)
    for x in xs:
        torch.testing.assert_close(x.double(), want, **TOL[torch.float32])


@pytest.mark.parametrize("path", PATHS)
@pytest.mark.parametrize("n", [1, 2, 4, 6])
def test_stragglar_other_sizes(n, path):
    xs, want = _run("stragglar", n, 20_001, path=path, scale=0.5)
    for x in xs:
        torch.testing.assert_close(x.double(), want, **TOL[torch.float32])


@pytest.mark.parametrize("path", PATHS)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_half_precisions(dtype, path):
    xs, want = _run("stragglar", 8, 30_005, dtype=dtype, path=path)
    for x in xs:
        torch.testing.assert_close(x.double(), want, **TOL[dtype])
    # one rounding per reduction, the same on both sides of a matching: all ranks agree bit for bit
    for x in xs[1:]:
        assert torch.equal(x, xs[0])


@pytest.mark.parametrize("path", PATHS)
@pytest.mark.parametrize("alg", ["stragglar", "stragglar_a2a", "direct"])
def test_prephase_done_mode(alg, path):
    xs, want = _run(alg, 8, 25_000, path=path, prephase=False)
    for x in xs:
        torch.testing.assert_close(x.double(), want, atol=2e-5, rtol=1e-6)


@pytest.mark.parametrize("path", PATHS)
def test_late_straggler_swapped_to_last_rank(path):
    # physical rank 2 is 3 ms late and plays logical rank n-1
    delay = [0.0] * 8
    delay[2] = 3.0
    xs, want = _run("stragglar", 8, 50_000, path=path, straggler=2, delay_ms=delay)
    for x in xs:
        torch.testing.assert_close(x.double(), want, **TOL[torch.float32])


@pytest.mark.parametrize("path", PATHS)
@pytest.mark.parametrize("count", [1, 5, 17, 4099])
def test_small_and_ragged(count, path):
    xs, want = _run("stragglar", 4, count, path=path, tile_bytes=2048)
    for x in xs:
        torch.testing.assert_close(x.double(), want, **TOL[torch.float32])


@pytest.mark.parametrize("path", PATHS)
def test_back_to_back_collectives_reuse_flags(path):
    from stragglar_b200 import ops
    n, count = 4, 100_000
    comm = ops.LocalComm(n, emulate=True)
    prog = sc.compile_program("ring", n)
    xs = [torch.full((count,), float(r + 1), device="cuda:0") for r in range(n)]
    for _ in range(3):
        comm.run(prog, xs, path=path, blocks=3, tile_bytes=8192)
    comm.sync()
    for x in xs:
        torch.testing.assert_close(x, torch.full_like(x, 10.0 * n * n))
    comm.close()


@pytest.mark.parametrize("path", PATHS)
def test_larger_than_l2(path):
    # 8 ranks x 64 MiB: every tile crosses HBM
    from stragglar_b200 import ops
    n, count = 8, 16 * 1024 * 1024
    comm = ops.LocalComm(n, emulate=True)
    prog = sc.compile_program("stragglar", n)
    xs = _inputs(n, count, torch.float32)
    comm.run(prog, xs, path=path, blocks=16, timed=True)
    ms = comm.sync()
    for x in xs:
        bad, worst = ops.verify_uniform_sum(x, list(range(n)), atol=1e-5)
        assert bad == 0, (bad, worst)
    assert ms[0] > 0
    comm.close()


def test_wait_runs_out_without_hanging():
    """A rank that arrives after the deadline: every block gives up, the status
    says so, the context stays usable and the next collective works."""
    from stragglar_b200 import ops
    n, count = 4, 10_000
    comm = ops.LocalComm(n, emulate=True)
    prog = sc.compile_program("stragglar", n)
    xs = _inputs(n, count, torch.float32)
    comm.run(prog, xs, blocks=2, tile_bytes=4096, delay_ms=[0, 0, 0, 400.0], timeout_s=0.05)
    comm.sync(check=False)
    assert comm.last_status != 0 and comm.last_status < 0x1000
    assert "timeout" in sc.status_string(comm.last_status) or "aborted" in sc.status_string(comm.last_status)
    torch.cuda.synchronize()
    # after the failure is cleared the communicator works again (fresh inputs, later epoch)
    ys = _inputs(n, count, torch.float32)
    want = torch.stack([y.double() for y in ys]).sum(0)
    comm.run(prog, ys, blocks=2, tile_bytes=4096)
    comm.sync()
    for y in ys:
        torch.testing.assert_close(y.double(), want, **TOL[torch.float32])
    comm.close()


def test_helper_kernels():
    from stragglar_b200 import ops
    x = torch.empty(1000, device="cuda:0")
    ops.fill_uniform(x, seed=7)
    torch.cuda.synchronize()
    assert -1.0 <= x.min().item() and x.max().item() < 1.0 and abs(x.mean().item()) < 0.1
    assert x[5].item() == pytest.approx(ops.host_uniform(7, 5))
    y = torch.empty(1000, device="cuda:0", dtype=torch.bfloat16)
    ops.scale_cast(y, x, 0.5)
    torch.cuda.synchronize()
    torch.testing.assert_close(y, (x * 0.5).bfloat16())
    ops.scale_cast(x, x, 2.0)
    t0 = torch.cuda.Event(enable_timing=True); t1 = torch.cuda.Event(enable_timing=True)
    t0.record(); ops.delay(5.0); t1.record(); torch.cuda.synchronize()
    assert 4.9 <= t0.elapsed_time(t1) < 7.0


@pytest.mark.parametrize("path", PATHS)
def test_round_trace(path):
    """Per-round statistics: every round of a rank's table shows up, starts before it ends, rounds end in order
    on the straggler (its matchings are serial), and a run without tracing leaves the record untouched."""
    from stragglar_b200 import ops
    n, count = 4, 60_000
    comm = ops.LocalComm(n, emulate=True)
    prog = sc.compile_program("stragglar", n)
    xs = _inputs(n, count, torch.float32)
    want = torch.stack([x.double() for x in xs]).sum(0)
    comm.run(prog, xs, path=path, blocks=2, tile_bytes=4096, timeout_s=5.0, trace_rounds=True)
    comm.sync()
    for x in xs:
        torch.testing.assert_close(x.double(), want, **TOL[torch.float32])
    tr = comm.round_trace()
    assert len(tr) == n
    for r in range(n):
        want_rounds = set()
        for t in prog.phases:
            want_rounds |= {int(k) for k in t.ranks[r].ops["round"]}
        assert set(tr[r]) == want_rounds, (r, sorted(tr[r]), sorted(want_rounds))
        for k, (start, end, wait) in tr[r].items():
            assert 0 < start <= end and wait < 5_000_000_000
    ends = [tr[n - 1][k][1] for k in sorted(tr[n - 1])]
    assert ends == sorted(ends)
    before = comm.round_trace()
    comm.run(prog, xs, path=path, blocks=2, tile_bytes=4096, timeout_s=5.0)
    comm.sync()
    assert comm.round_trace() == before
    comm.close()


@pytest.mark.parametrize("path", PATHS)
@pytest.mark.parametrize("alg,n,slack", [("stragglar", 8, 0), ("stragglar", 8, 3), ("stragglar", 6, 0), ("ring", 4, 0),
                                         ("stragglar_a2a", 4, 0)])
def test_round_gating(alg, n, slack, path, monkeypatch):
    """Rounds one after the other (STRAGGLAR_GATE): same sums, twice in a row on the same control words, and with
    the full barrier (slack 0) the traced rounds do not overlap on any rank."""
    monkeypatch.setenv("STRAGGLAR_GATE_SLACK", str(slack))
    from stragglar_b200 import ops
    monkeypatch.setenv("STRAGGLAR_GATE", "all")
    monkeypatch.setenv("STRAGGLAR_GATE_MIN_BYTES", "0")      # gate the small test buffers too
    prog = sc.compile_program(alg, n)
    assert prog.main.gate_rounds
    comm = ops.LocalComm(n, emulate=True)
    for rep in range(2):
        xs = _inputs(n, 50_003, torch.float32)
        want = torch.stack([x.double() for x in xs]).sum(0)
        comm.run(prog, xs, path=path, blocks=2, tile_bytes=4096, timeout_s=5.0, trace_rounds=True)
        comm.sync()
        for x in xs:
            torch.testing.assert_close(x.double(), want, **TOL[torch.float32])
    tr = comm.round_trace()
    starts = {}
    ends = {}
    for r in range(n):
        for k, (s, e, _) in tr[r].items():
            starts[k] = min(starts.get(k, s), s)
            ends[k] = max(ends.get(k, e), e)
    rounds = sorted(starts)
    # GPUs' %globaltimer values agree here: all ranks are emulated on one device
    if slack == 0:
        assert all(ends[a] <= starts[b] for a, b in zip(rounds, rounds[1:])), (starts, ends)
    comm.close()


@pytest.mark.parametrize("path", PATHS)
@pytest.mark.parametrize("alg,n", [("stragglar", 8), ("ring", 4), ("rsag", 4), ("stragglar_a2a", 6), ("stragglar", 1)])
@pytest.mark.parametrize("wire,user", [(torch.float32, torch.float32), (torch.bfloat16, torch.float32),
                                       (torch.float32, torch.bfloat16)])
def test_staged_mode_reads_and_writes_the_callers_tensors(alg, n, wire, user, path):
    """Staged mode: the kernel itself copies the caller's tensor into the buffer peers reach (converting to the wire
    dtype), runs the table and copies every finished tile back; no separate copy or cast kernels."""
    from stragglar_b200 import ops
    count = 70_001
    comm = ops.LocalComm(n, emulate=True)
    prog = sc.compile_program(alg, n)
    if len(prog.phases) != 1:
        pytest.skip("staged mode serves single-phase programs")
    users = _inputs(n, count, user)
    # what the wire carries: the inputs rounded to the wire dtype, summed in fp32
    want = torch.stack([u.to(wire).double() for u in users]).sum(0) * 0.5
    arena = [torch.full((count,), float("nan"), dtype=wire, device="cuda:0") for _ in range(n)]
    torch.cuda.synchronize()
    for rep in range(2):   # twice: the second run finds the flags of the first
        if rep:
            for u, v in zip(users, _inputs(n, count, user)):
                u.copy_(v)
            torch.cuda.synchronize()
        comm.run(prog, arena, path=path, blocks=3, tile_bytes=4096, scale=0.5, timeout_s=5.0, user_tensors=users)
        comm.sync()
        lo = torch.bfloat16 in (wire, user)
        tol = dict(atol=6e-2, rtol=2e-2) if lo else dict(atol=1e-5, rtol=1e-6)
        for u in users:
            torch.testing.assert_close(u.double(), want, **tol)
    comm.close()


@pytest.mark.parametrize("path", PATHS)
@pytest.mark.parametrize("n,count", [(8, 1), (8, 8 * 4096 + 3), (6, 16 * 4096 - 1), (16, 300_007), (2, 2_000_003)])
@pytest.mark.parametrize("staged", [False, True])
def test_default_launch_shape(n, count, staged, path):
    """The launch shape chosen for emulated ranks (from one item of work to more than the device holds at once)
    against two blocks per rank: the split of the work never touches the order of a sum, so the bits are equal."""
    from stragglar_b200 import ops
    comm = ops.LocalComm(n, emulate=True)
    prog = sc.compile_program("stragglar", n)
    outs = []
    for kw in ({}, {"blocks": 2}):
        xs = _inputs(n, count, torch.float32)
        arena = [torch.zeros_like(x) for x in xs] if staged else xs
        comm.run(prog, arena, path=path, scale=1.0 / n, timeout_s=5.0, user_tensors=xs if staged else None, **kw)
        comm.sync()
        outs.append(xs)
    want = torch.stack([x.double() for x in _inputs(n, count, torch.float32)]).mean(0)
    for a, b in zip(*outs):
        assert torch.equal(a, b)
        torch.testing.assert_close(a.double(), want, **TOL[torch.float32])
    comm.close()


@pytest.mark.parametrize("count", [1, 3, 4, 8, 2047, 2048, 2049, 4096 + 7, 1_000_003])
@pytest.mark.parametrize("offset", [0, 8, 1])   # elements: the vector path, 16-byte aligned again, and the scalar path
def test_scale_cast_edges(count, offset):
    """One product in fp32 and one rounding an element: equal bits, whatever the types, the ragged end or the alignment."""
    from stragglar_b200 import ops
    for a in (torch.float32, torch.bfloat16, torch.float16):
        for b in (torch.float32, torch.bfloat16, torch.float16):
            src = torch.randn(count + offset, device="cuda:0").to(a)[offset:]
            guard = torch.full((count + offset + 16,), 7.0, device="cuda:0", dtype=b)
            dst = guard[offset:offset + count]
            ops.scale_cast(dst, src, 0.3)
            torch.cuda.synchronize()
            want = (src.float() * torch.tensor(0.3, dtype=torch.float32)).to(b)
            assert torch.equal(dst, want), (a, b)
            assert (guard[:offset] == 7.0).all() and (guard[offset + count:] == 7.0).all()
            if a == b:
                ops.scale_cast(src, src, 0.3)
                torch.cuda.synchronize()
                assert torch.equal(src, want)


@pytest.mark.parametrize("stages", [2, 3, 6])
@pytest.mark.parametrize("alg,blocks,tile_bytes", [("stragglar", 1, 2048), ("rsag", 2, 2048), ("stragglar_a2a", 3, 98304),
                                                   ("ring", 1, 33280)])
@pytest.mark.parametrize("staged", [False, True])
def test_bulk_copy_ring(alg, blocks, tile_bytes, stages, staged):
    """The hand-over between the roles of a block: rings from two stages up, many items a block (more than a storer's
    queue holds), items of one piece, of several and with a ragged last one, copies that skip the adders, conversions."""
    from stragglar_b200 import ops
    n, count = 8, 150_003
    comm = ops.LocalComm(n, emulate=True)
    prog = sc.compile_program(alg, n)
    xs = _inputs(n, count, torch.float32)
    wire = torch.bfloat16 if staged else torch.float32
    want = torch.stack([x.to(wire).double() for x in xs]).sum(0)
    arena = [torch.zeros(count, dtype=wire, device="cuda:0") for _ in range(n)] if staged else xs
    comm.run(prog, arena, path="tma", blocks=blocks, tile_bytes=tile_bytes, stages=stages, timeout_s=5.0,
             user_tensors=xs if staged else None)
    comm.sync()
    for x in xs:
        torch.testing.assert_close(x.double(), want, **TOL[wire])
    comm.close()


def test_wait_runs_out_on_the_bulk_copy_path():
    """As above with the roles of the bulk-copy path: all of them leave, and the communicator works again."""
    from stragglar_b200 import ops
    n, count = 4, 100_000
    comm = ops.LocalComm(n, emulate=True)
    prog = sc.compile_program("stragglar", n)
    comm.run(prog, _inputs(n, count, torch.float32), path="tma", blocks=2, tile_bytes=4096, delay_ms=[0, 0, 0, 400.0], timeout_s=0.05)
    comm.sync(check=False)
    assert 0 < comm.last_status < 0x1000
    ys = _inputs(n, count, torch.float32)
    want = torch.stack([y.double() for y in ys]).sum(0)
    comm.run(prog, ys, path="tma", blocks=2, tile_bytes=4096)
    comm.sync()
    for y in ys:
        torch.testing.assert_close(y.double(), want, **TOL[torch.float32])
    comm.close()


@pytest.mark.parametrize("path", PATHS)
@pytest.mark.parametrize("wire,user", [(torch.bfloat16, torch.float16), (torch.float16, torch.bfloat16)])
@pytest.mark.parametrize("offset", [0, 1])   # elements: bulk copies or vectors, and element by element
@pytest.mark.parametrize("shape", [{}, {"blocks": 3, "tile_bytes": 4096}])
def test_staged_mode_between_the_two_byte_types(wire, user, path, offset, shape):
    """fp16 and bf16 have the same size and are not the same: both ways of a staged collective convert."""
    from stragglar_b200 import ops
    n, count = 4, 70_005
    comm = ops.LocalComm(n, emulate=True)
    prog = sc.compile_program("rsag", n)
    users = []
    for x in _inputs(n, count, torch.float32):
        u = torch.empty(count + offset, dtype=user, device="cuda:0")[offset:]
        u.copy_(x)
        users.append(u)
    want = torch.stack([u.to(wire).double() for u in users]).sum(0) * 0.5
    arena = [torch.full((count,), float("nan"), dtype=wire, device="cuda:0") for _ in range(n)]
    comm.run(prog, arena, path=path, scale=0.5, timeout_s=5.0, user_tensors=users, **shape)
    comm.sync()
    # one rounding to each type, half an ulp each (2^-8 for 8 significant bits in bf16, 2^-11 for 11 in fp16), after a sum
    # of four values below 1 in fp32
    for u in users:
        torch.testing.assert_close(u.double(), want, rtol=2 ** -8 + 2 ** -11 + 2 ** -18, atol=1e-6)
    comm.close()


def test_launches_beside_another_threads_smaller_ring():
    """The shared-memory limit of a kernel belongs to the device, not to a call: a thread that asks for a launch with few
    ring stages leaves the launches of another thread, with the whole ring, alone."""
    from stragglar_b200 import ops
    n, count = 2, 1000
    comm = ops.LocalComm(n, emulate=True)
    prog = sc.compile_program("rsag", n)
    xs = _inputs(n, count, torch.float32)
    want = torch.stack([x.double() for x in xs]).mean(0)
    stop = threading.Event()

    def ask():
        while not stop.is_set():
            ops.cuda_lib().sar_cuda_emulated_fit(0, ops.local.PATHS["tma"], 0, 2, 1)

    other = threading.Thread(target=ask)
    other.start()
    try:
        for _ in range(50):
            for _ in range(40):
                comm.run(prog, xs, path="tma", blocks=1, stages=6, scale=0.5, timeout_s=5.0)
            comm.sync()
    finally:
        stop.set()
        other.join()
    for x in xs:
        torch.testing.assert_close(x.double(), want, **TOL[torch.float32])
    comm.close()


def test_gating_is_decided_when_the_program_is_compiled(monkeypatch):
    """A program that was compiled with STRAGGLAR_GATE keeps its rounds apart when the variable is gone at run time."""
    from stragglar_b200 import ops
    n = 8
    monkeypatch.setenv("STRAGGLAR_GATE_SLACK", "0")
    monkeypatch.setenv("STRAGGLAR_GATE_MIN_BYTES", "0")
    monkeypatch.setenv("STRAGGLAR_GATE", "1")
    prog = sc.compile_program("stragglar", n)
    monkeypatch.delenv("STRAGGLAR_GATE")
    comm = ops.LocalComm(n, emulate=True)
    xs = _inputs(n, 50_003, torch.float32)
    want = torch.stack([x.double() for x in xs]).sum(0)
    comm.run(prog, xs, path="tma", blocks=2, tile_bytes=4096, timeout_s=5.0, trace_rounds=True)
    comm.sync()
    for x in xs:
        torch.testing.assert_close(x.double(), want, **TOL[torch.float32])
    tr = comm.round_trace()
    rounds = sorted({k for t in tr for k in t})
    for a, b in zip(rounds, rounds[1:]):
        assert max(t[a][1] for t in tr if a in t) <= min(t[b][0] for t in tr if b in t)
    comm.close()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_sixteen_small_simt_blocks_per_sm(dtype):
    """An explicit launch of sixteen 32-thread blocks per SM (what their registers allow) is not refused for the table's
    shared memory."""
    from stragglar_b200 import ops
    n, count = 4, 600_000
    comm = ops.LocalComm(n, emulate=True)
    blocks = torch.cuda.get_device_properties(0).multi_processor_count * 16 // n
    xs = _inputs(n, count, dtype)
    want = torch.stack([x.double() for x in xs]).sum(0)
    comm.run(sc.compile_program("ring", n), xs, path="simt", blocks=blocks, threads=32, timeout_s=5.0)
    comm.sync()
    for x in xs:
        torch.testing.assert_close(x.double(), want, **TOL[dtype])
    comm.close()


@pytest.mark.parametrize("store_window", [3, 16])
def test_store_window_says_that_it_has_no_effect(store_window):
    """A sweep over it would compare identical runs: the call goes on, with a warning."""
    from stragglar_b200 import ops
    comm = ops.LocalComm(2, emulate=True)
    prog = sc.compile_program("rsag", 2)
    xs = _inputs(2, 10_001, torch.float32)
    want = torch.stack([x.double() for x in xs]).sum(0)
    with pytest.warns(UserWarning, match="store_window .* no effect"):
        comm.run(prog, xs, path="tma", timeout_s=5.0, store_window=store_window)
    comm.sync()
    for x in xs:
        torch.testing.assert_close(x.double(), want, **TOL[torch.float32])
    comm.close()


UNIT = {torch.float32: 2.0 ** -24, torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}   # half an ulp, relative


@pytest.mark.parametrize("path", PATHS)
@pytest.mark.parametrize("wire", list(UNIT))
@pytest.mark.parametrize("user", list(UNIT))
@pytest.mark.parametrize("offset", [0, 1])   # elements: an aligned tensor of the caller's, and one that no vector fits
def test_staging_of_every_type_pair(user, wire, offset, path):
    """Tiles of far more vectors than a block has threads, so that the unrolled conversions run and end raggedly: with the
    launch shape chosen for emulated ranks and with large tiles on few blocks."""
    from stragglar_b200 import ops
    n, count, guard = 2, 1_000_003, 16
    comm = ops.LocalComm(n, emulate=True)
    prog = sc.compile_program("rsag", n)
    for shape in ({}, {"blocks": 3, "tile_bytes": 98304}):
        whole = [torch.full((guard + offset + count + guard,), 7.0, dtype=user, device="cuda:0") for _ in range(n)]
        users = [w[guard + offset:guard + offset + count] for w in whole]
        for u, x in zip(users, _inputs(n, count, torch.float32)):
            u.copy_(x)
        want = torch.stack([u.to(wire).double() for u in users]).sum(0) * 0.5
        arena = [torch.full((count,), float("nan"), dtype=wire, device="cuda:0") for _ in range(n)]
        comm.run(prog, arena, path=path, scale=0.5, timeout_s=5.0, user_tensors=users, **shape)
        comm.sync()
        for w, u in zip(whole, users):
            # the sum of two values in fp32, one rounding to the wire and one to the caller's type; atol: subnormal fp16
            torch.testing.assert_close(u.double(), want, rtol=2.0 ** -24 + UNIT[wire] + UNIT[user] + 2.0 ** -18, atol=2.0 ** -23)
            assert (w[:guard + offset] == 7.0).all() and (w[guard + offset + count:] == 7.0).all()
    comm.close()


@pytest.mark.parametrize("path", PATHS)
def test_lone_rank_scales_every_element(path):
    """A communicator of one rank (the launch shape of a c10d group of one) halves its buffer: one product and one rounding
    an element, so equal bits, at one block's worth, around a block per ring stage and beyond a block per SM; with nothing
    written beside it.  Staged: rounded to the wire, halved, rounded to the wire and to the caller's type."""
    from stragglar_b200 import ops
    comm = ops.LocalComm(1)
    prog = sc.compile_program("stragglar", 1)
    guard = 64
    for count in (1, 5, 8 * 1024 + 1, 1 << 20, 9 * (1 << 20) + 3, 34 * (1 << 20) + 1):
        for dtype, wire in ((torch.float32, None), (torch.bfloat16, None), (torch.float16, None), (torch.float32, torch.float32),
                            (torch.float32, torch.bfloat16), (torch.bfloat16, torch.float32), (torch.float16, torch.bfloat16)):
            whole = torch.full((count + 2 * guard,), 7.0, dtype=dtype, device="cuda:0")
            t = whole[guard:guard + count]
            t.normal_(generator=torch.Generator(device="cuda:0").manual_seed(count))
            on_wire = t if wire is None else t.to(wire)
            want = (on_wire.float() * 0.5).to(on_wire.dtype).to(dtype)
            if wire is None:
                comm.run(prog, [t], path=path, scale=0.5, timeout_s=5.0)
            else:
                arena = torch.full((count,), float("nan"), dtype=wire, device="cuda:0")
                comm.run(prog, [arena], path=path, scale=0.5, timeout_s=5.0, user_tensors=[t])
            comm.sync()
            assert torch.equal(t, want), (count, dtype, wire)
            assert (whole[:guard] == 7.0).all() and (whole[guard + count:] == 7.0).all(), (count, dtype, wire)
    comm.close()


@pytest.mark.parametrize("path", PATHS)
@pytest.mark.parametrize("alg", ["stragglar", "stragglar_a2a", "direct"])
@pytest.mark.parametrize("shape", [{"blocks": 2, "tile_bytes": 2048}, {"blocks": 8, "tile_bytes": 4096}, {}])
def test_staged_mode_without_the_prephase(alg, path, shape, monkeypatch):
    """The non-stragglers' sum is in place, so most slots are pushed to without their input having been read: the pushed
    tiles, and their flags, survive the copy-in of that input."""
    from stragglar_b200 import ops
    monkeypatch.setenv("STRAGGLAR_COPY", "push")
    n, count = 8, 190_003
    comm = ops.LocalComm(n, emulate=True)
    prog = sc.compile_program(alg, n, False)
    for rep in range(3):
        users = _inputs(n, count, torch.float32)
        want = torch.stack([u.double() for u in users]).sum(0)
        _prephase(users, alg, n - 1)
        arena = [torch.full((count,), float("nan"), device="cuda:0") for _ in range(n)]
        comm.run(prog, arena, path=path, timeout_s=2.0, user_tensors=users, **shape)
        comm.sync()
        for u in users:
            torch.testing.assert_close(u.double(), want, atol=2e-5, rtol=1e-6)
    comm.close()


@pytest.mark.parametrize("path", PATHS)
def test_gated_runs_one_after_another_on_the_whole_device(path, monkeypatch):
    """The last block of a launch resets the counters of the gate for the next one: back to back, with every block that
    fits, no announcement is lost."""
    from stragglar_b200 import ops
    monkeypatch.setenv("STRAGGLAR_GATE", "all")
    monkeypatch.setenv("STRAGGLAR_GATE_MIN_BYTES", "0")
    monkeypatch.setenv("STRAGGLAR_GATE_SLACK", "3")
    n, count = 8, 200_003
    comm = ops.LocalComm(n, emulate=True)
    prog = sc.compile_program("stragglar", n)
    xs = _inputs(n, count, torch.float32)
    want = torch.stack([x.double() for x in xs]).mean(0)
    for _ in range(100):
        comm.run(prog, xs, path=path, scale=1.0 / n, timeout_s=2.0)
    comm.sync()
    # each run after the first averages n equal values: a sum of eight, one rounding or less a run
    for x in xs:
        torch.testing.assert_close(x.double(), want, rtol=100 * 8 * 2.0 ** -24, atol=1e-5)
    comm.close()
