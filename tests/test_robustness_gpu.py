"""Error paths and device-side ordering of the decode-shape kernels, on one GPU and without ever hanging or
faulting it: every wait in the kernels is bounded, so the tests make a wait run out (a flag that nothing sets,
a copy whose completion is never reported) and check that the kernel returns, that the failure is reported
through every channel, and that the next normal call is correct."""

import threading
import time

import numpy as np
import pytest

from conftest import have_cuda, load_pkg

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

DEV = "cuda:0"
TIMEOUT = -7


@pytest.fixture(scope="module")
def P():
    if not have_cuda():
        pytest.skip("no CUDA device")
    pkg = load_pkg()
    pkg._cabi.lib()
    return pkg


def _problem(P, n, k, m, seed):
    dev = torch.device(DEV)
    w = P.ops.generate(n * k, seed, 0.02, torch.float16, dev).view(n, k)
    pk, sc = P.ops.encode(w, 32)
    x = P.ops.generate(m * k, seed + 1, 1.0, torch.bfloat16, dev).view(m, k)
    return pk, sc, x


def test_chain_orders_itself_on_the_device(P):
    """Dependent grouped launches - the second reads what the first wrote - ordered by the peer-sync block alone (one
    rank, so 'every rank' is this one): results equal the unsynchronised path and the epoch counts the signalled
    launches.  The third splits K over a cluster; the fourth, over two matrices with K > 4096, signals from the reduce
    kernel, and the fifth, over two matrices, from its main kernel."""
    dev = torch.device(DEV)
    m = 4
    pk1, sc1, x = _problem(P, 512, 4096, m, 10)
    pk2, sc2, _ = _problem(P, 256, 512, m, 20)
    pk3, sc3, x3 = _problem(P, 128, 14336, m, 30)
    mid = torch.zeros((m, 512), dtype=torch.bfloat16, device=dev)
    out = torch.zeros((m, 256), dtype=torch.bfloat16, device=dev)
    out3 = torch.zeros((m, 128), dtype=torch.bfloat16, device=dev)
    sync = torch.zeros(64, dtype=torch.int32, device=dev)
    first = P.ops.GroupedGemv([(x, pk1, sc1, None, mid)], [(512, 4096)], peer_delta=[0], peer_sync=sync.data_ptr(),
                              signal_peers=True, static_weights=True)
    second = P.ops.GroupedGemv([(mid, pk2, sc2, None, out)], [(256, 512)], peer_delta=[0], peer_sync=sync.data_ptr(),
                               wait_peers=True, signal_peers=True, static_weights=True)
    third = P.ops.GroupedGemv([(x3, pk3, sc3, None, out3)], [(128, 14336)], peer_delta=[0], peer_sync=sync.data_ptr(),
                              wait_peers=True, signal_peers=True, static_weights=True)
    sync4 = dict(peer_delta=[0], peer_sync=sync.data_ptr(), wait_peers=True, signal_peers=True, static_weights=True)
    out4 = [torch.zeros((m, 128), dtype=torch.bfloat16, device=dev) for _ in range(2)]
    out5 = [torch.zeros((m, 256), dtype=torch.bfloat16, device=dev) for _ in range(2)]
    fourth = P.ops.GroupedGemv([(x3, pk3, sc3, None, y) for y in out4], [(128, 14336)] * 2, **sync4)
    fifth = P.ops.GroupedGemv([(mid, pk2, sc2, None, y) for y in out5], [(256, 512)] * 2, **sync4)
    for _ in range(3):
        first(); second(); third(); fourth(); fifth()
    torch.cuda.synchronize()
    ref_mid = P.ops.linear(x, pk1, sc1, None, 512, 4096, 32)
    ref_out = P.ops.linear(ref_mid, pk2, sc2, None, 256, 512, 32)
    ref3 = P.ops.linear(x3, pk3, sc3, None, 128, 14336, 32)
    assert torch.equal(mid, ref_mid) and torch.equal(out, ref_out) and torch.equal(out3, ref3)
    words = sync.cpu().numpy()
    assert words[0] == 15 and words[1] == 0 and words[2] == 0 and words[4] == 15    # epoch, arrived, status, flag[0]
    for got, want in [(y, ref3) for y in out4] + [(y, ref_out) for y in out5]:              # another kernel: sums in another order
        assert float((got.float() - want.float()).norm() / want.float().norm()) <= 4e-3
    assert P._cabi.lib().ojx_e8t_device_status() == 0


@pytest.mark.parametrize("static", [False, True])
@pytest.mark.parametrize("m,k", [(1, 2048), (2, 2048), (2, 8192), (4, 2048)])
def test_x_is_read_after_the_peers_have_published_it(P, m, k, static):
    """A launch over one matrix that waits for its peers: x, in memory the host can write, changes after the kernel has started
    and before the awaited flag is set (as another rank's stores would), and the result has to be the new x's.  The wait is bounded."""
    dev, n = torch.device(DEV), 96
    pk, sc, x = _problem(P, n, k, m, 60)
    want = P.ops.linear(x, pk, sc, None, n, k, 32)
    host_x = torch.zeros((m, k), dtype=torch.bfloat16).pin_memory()
    sync = torch.zeros(16, dtype=torch.int32).pin_memory()
    sync[0], sync[3] = 1, 1 << 20                               # one launch is awaited; polls before giving up
    y, lib = torch.zeros((m, n), dtype=torch.bfloat16, device=dev), P._cabi.lib()
    prob = P._cabi.GemvProblem(x=host_x.data_ptr(), packed=pk.data_ptr(), scales=sc.data_ptr(), y=y.data_ptr(), N=n, K=k)
    table = torch.frombuffer(bytearray(bytes(prob)), dtype=torch.uint8).to(dev)
    new_x = x.cpu()
    torch.cuda.synchronize()
    flags = P._cabi.OJX_GEMV_WAIT_PEERS | (P._cabi.OJX_GEMV_STATIC_WEIGHTS if static else 0)
    st = lib.ojx_e8t_gemv_grouped_ex(table.data_ptr(), 1, lib.ojx_e8t_gemv_tiles(n, k), m, P._cabi.OJX_BF16, P._cabi.OJX_BF16,
                                     int(lib.ojx_e8t_gemv_kchunks(k) > 1), None, 1, sync.data_ptr(), flags,
                                     torch.cuda.current_stream().cuda_stream)
    time.sleep(0.02)                                            # the kernel is at its wait
    host_x.copy_(new_x)
    sync[4] = 1                                                 # flag[0]
    torch.cuda.synchronize()
    assert st == 0 and int(sync[2]) == 0 and lib.ojx_e8t_device_status() == 0
    assert float((y.float() - want.float()).norm() / want.float().norm()) <= 4e-3       # K split or not: a bf16 rounding each


def test_wait_on_a_rank_that_never_signals_gives_up(P):
    dev = torch.device(DEV)
    lib = P._cabi.lib()
    pk, sc, x = _problem(P, 256, 1024, 2, 40)
    y = torch.zeros((2, 256), dtype=torch.bfloat16, device=dev)
    sync = torch.zeros(64, dtype=torch.int32, device=dev)
    sync[0] = 5          # this rank believes five launches are done; nobody has published them into flag[0]
    sync[3] = 2000       # polls before giving up (about a millisecond)
    grp = P.ops.GroupedGemv([(x, pk, sc, None, y)], [(256, 1024)], peer_delta=[0], peer_sync=sync.data_ptr(), wait_peers=True)
    grp()
    torch.cuda.synchronize()                                  # the kernel returned
    assert int(sync[2].item()) == TIMEOUT
    with pytest.raises(P._cabi.OjxError):                     # the next call through a wrapper raises, no sync needed
        P.ops.linear(x, pk, sc, None, 256, 1024, 32)
    assert lib.ojx_e8t_poll_status() == 0                     # reported once
    assert lib.ojx_e8t_device_status() == TIMEOUT and lib.ojx_e8t_device_status() == 0
    sync.zero_()
    grp()                                                     # epoch 0, flag 0: nothing to wait for
    torch.cuda.synchronize()
    assert torch.equal(y, P.ops.linear(x, pk, sc, None, 256, 1024, 32))
    assert lib.ojx_e8t_device_status() == 0


@pytest.mark.parametrize("count", [1, 2])
def test_copy_that_never_completes_gives_up(P, count):
    """A wait inside the kernel that nothing ends (several matrices: the loader withholds one arrival on the first work
    item's 'copies landed' barrier; one matrix: a barrier made for this) runs into the (shortened) limit, the CTAs stop
    touching their inputs, keep their barriers matched, wait for the copies that are in flight, and return."""
    dev = torch.device(DEV)
    lib = P._cabi.lib()
    pk, sc, x = _problem(P, 4096, 4096, 16, 50)
    y = torch.zeros((16, 4096), dtype=torch.bfloat16, device=dev)
    entries = [(x, pk, sc, None, y)] + [(x, pk, sc, None, torch.zeros_like(y))] * (count - 1)
    good = P.ops.GroupedGemv(entries, [(4096, 4096)] * count)
    bad = P.ops.GroupedGemv(entries, [(4096, 4096)] * count, extra_flags=P._cabi.OJX_GEMV_TEST_LOSE_COPY)
    lib.ojx_e8t_set_wait_limit(3000)
    try:
        bad()
        torch.cuda.synchronize()
    finally:
        lib.ojx_e8t_set_wait_limit(0)
    with pytest.raises(P._cabi.OjxError):
        good()
    assert lib.ojx_e8t_device_status() == TIMEOUT
    good()
    torch.cuda.synchronize()
    wd = P.ops.decode(pk, sc, (4096, 4096), torch.float32)
    ref = x.float() @ wd.t()
    assert float((y.float() - ref).norm() / ref.norm()) <= 2e-3
    assert lib.ojx_e8t_device_status() == 0 and lib.ojx_e8t_poll_status() == 0


def test_two_devices_in_one_process(P):
    """Kernel attributes and the SM count are kept per device: the same process drives cuda:0 and cuda:1."""
    if torch.cuda.device_count() < 2:
        pytest.skip("needs two GPUs")
    outs = []
    for d in (0, 1):
        dev = torch.device("cuda", d)
        w = P.ops.generate(512 * 4096, 3, 0.02, torch.float16, dev).view(512, 4096)
        pk, sc = P.ops.encode(w, 32)
        x = P.ops.generate(16 * 4096, 4, 1.0, torch.bfloat16, dev).view(16, 4096)
        outs.append(P.ops.linear(x, pk, sc, None, 512, 4096, 32).cpu())
        outs.append(P.ops.linear(x.repeat(8, 1), pk, sc, None, 512, 4096, 32, force="gemm")[:16].cpu())
    assert torch.equal(outs[0], outs[2]) and torch.equal(outs[1], outs[3])


def test_independent_launches_overlap_without_changing_results(P):
    """OJX_GEMV_INDEPENDENT: launches over different matrices with their own activations and outputs never wait for
    the launch queued ahead of them; their results equal the ordered launches' bit for bit, a dependent reader queued
    after them sees complete outputs, and the flag is refused together with the cross-GPU ordering flags."""
    dev = torch.device(DEV)
    groups, ordered = [], []
    for i, (n, k, m) in enumerate([(512, 4096, 1), (1024, 14336, 4), (384, 4096, 16), (2048, 4096, 1)]):
        mats = [_problem(P, n, k, m, 40 + 10 * i + j) for j in range(6)]
        y_a = torch.zeros((6, m, n), dtype=torch.bfloat16, device=dev)
        y_b = torch.zeros((6, m, n), dtype=torch.bfloat16, device=dev)
        groups.append((P.ops.GroupedGemv([(x, pk, sc, None, y_a[j]) for j, (pk, sc, x) in enumerate(mats)], [(n, k)] * 6,
                                         static_weights=True, independent=True), y_a))
        ordered.append((P.ops.GroupedGemv([(x, pk, sc, None, y_b[j]) for j, (pk, sc, x) in enumerate(mats)], [(n, k)] * 6), y_b))
    for grp, _ in ordered:
        grp()
    for _ in range(3):                                      # back to back: the tail of one launch is filled by the next
        for grp, _ in groups:
            grp()
    total = sum(y.float().sum() for _, y in groups)         # a dependent reader, queued after the launches
    torch.cuda.synchronize()
    for (_, ya), (_, yb) in zip(groups, ordered):
        assert torch.equal(ya, yb)
    assert torch.isfinite(total)
    groups[0][0](independent=False)                         # per-call override back to an ordered launch
    torch.cuda.synchronize()
    assert torch.equal(groups[0][1], ordered[0][1])
    lib = P._cabi.lib()
    g0 = groups[0][0]
    sync = torch.zeros(16, dtype=torch.int32, device=dev)
    st = lib.ojx_e8t_gemv_grouped_ex(g0.table.data_ptr(), g0.count, g0.total_tiles, g0.M, 2, 2, g0.needs_reduce, None, 1,
                                     sync.data_ptr(), P._cabi.OJX_GEMV_INDEPENDENT | P._cabi.OJX_GEMV_WAIT_PEERS, None)
    assert st == -9


@pytest.mark.parametrize("m", [1, 4, 16])
@pytest.mark.parametrize("n,k", [(40, 256), (1000, 4096), (72, 4352)])
def test_split_flags_do_not_change_results(P, m, n, k):
    """OJX_GEMV_SPLIT_K2 / K4 are hints: K of one chunk, or of fewer than the cluster has CTAs, gives the unsplit launch's result."""
    pk, sc, x = _problem(P, n, k, m, 70)
    outs = []
    for flag in (0, P._cabi.OJX_GEMV_SPLIT_K2, P._cabi.OJX_GEMV_SPLIT_K4):
        y = torch.zeros((m, n), dtype=torch.float32, device=DEV)
        g = P.ops.GroupedGemv([(x, pk, sc, None, y)], [(n, k)], extra_flags=flag)
        g.flags = flag                                          # none that the constructor would choose itself
        g()
        outs.append(y)
    torch.cuda.synchronize()
    wd = P.ops.decode(pk, sc, (n, k), torch.float32).double()
    bound = x.double().abs() @ wd.abs().t()
    for y in outs:
        assert float(((y.double() - x.double() @ wd.t()).abs() / bound).max()) <= 5e-6


@pytest.mark.parametrize("count", [1, 2])
def test_reader_behind_an_independent_launch_sees_what_came_before_it(P, count):
    """linear -> independent launch -> linear that reads the first one's output: the reader may start early, but not before the
    first has ended, although the launch between them waits for nobody.  (Both kernels of grouped launches.)"""
    dev = torch.device(DEV)
    pk, sc, _ = _problem(P, 14336, 4096, 1, 80)
    pk2, sc2, _ = _problem(P, 64, 14336, 1, 82)
    small = [_problem(P, 16, 256, 1, 84 + i) for i in range(count)]
    outs = [torch.zeros((1, 16), dtype=torch.bfloat16, device=dev) for _ in range(count)]
    between = P.ops.GroupedGemv([(x, p, s, None, y) for (p, s, x), y in zip(small, outs)], [(16, 256)] * count, independent=True)
    xs = [P.ops.generate(16 * 4096, 90 + i, 1.0, torch.bfloat16, dev).view(16, 4096) for i in range(2)]
    want = []
    for x in xs:
        y = P.ops.linear(x, pk, sc, None, 14336, 4096, 32)
        torch.cuda.synchronize()
        want.append(P.ops.linear(y, pk2, sc2, None, 64, 14336, 32))
        del y
    for i in range(40):                                     # the first output's memory is used again: a stale read is the other x's
        y = P.ops.linear(xs[i % 2], pk, sc, None, 14336, 4096, 32)
        between()
        z = P.ops.linear(y, pk2, sc2, None, 64, 14336, 32)
        assert torch.equal(z, want[i % 2]), i
        del y


@pytest.mark.parametrize("m", [1, 2, 5, 16])
@pytest.mark.parametrize("n,k,ld,shift,dt", [(256, 1024, 256, 0, "bfloat16"), (100, 512, 104, 0, "float16"), (33, 14336, 40, 0, "bfloat16"),
                                             (520, 8192, 1040, 0, "bfloat16"), (64, 512, 67, 0, "bfloat16"), (96, 4352, 96, 1, "float16"),
                                             (72, 256, 72, 0, "float32")])
def test_outputs_of_one_matrix_reach_every_window(P, m, n, k, ld, shift, dt):
    """Stores into the other ranks' windows (here: buffers of the same GPU) of a launch over one matrix: whole and cut groups of eight
    rows, K of several chunks and split over a cluster, rows of any pitch, windows at odd distances, fp32; nothing beside them."""
    dev, dtype = torch.device(DEV), getattr(torch, dt)
    pk, sc, x = _problem(P, n, k, m, 110)
    step = -(-(m * ld + 8) // 8) * 8
    for world in (2, 8):
        flat = torch.full((world * step + 8,), 7.0, dtype=dtype, device=dev)
        starts = [r * step + (shift if r else 0) for r in range(world)]
        views = [torch.as_strided(flat, (m, n), (ld, 1), s) for s in starts]
        P.ops.GroupedGemv([(x, pk, sc, None, views[0])], [(n, k)], peer_delta=[s * flat.element_size() for s in starts])()
        alone = torch.empty((m, n), dtype=dtype, device=dev)
        P.ops.GroupedGemv([(x, pk, sc, None, alone)], [(n, k)])()
        for v in views:
            assert torch.equal(v, alone)
            v.fill_(7.0)
        assert bool((flat == 7.0).all())


@pytest.mark.parametrize("m", [1, 4, 16])
@pytest.mark.parametrize("n,k,shift", [(64, 512, 0), (64, 512, 1), (72, 14336, 0), (72, 14336, 1), (40, 4352, 3)])
def test_outputs_of_several_matrices_reach_windows_at_any_distance(P, m, n, k, shift):
    """The same of launches over several matrices and of their reduce launch: windows that are no multiple of 16 bytes apart take
    stores of single outputs."""
    dev = torch.device(DEV)
    probs = [_problem(P, n, k, m, 120 + 10 * i) for i in range(2)]
    step = m * n + 8
    flat = torch.full((2 * 2 * step + 8,), 7.0, dtype=torch.bfloat16, device=dev)
    ys = [torch.as_strided(flat, (m, n), (n, 1), i * step) for i in range(2)]
    far = [torch.as_strided(flat, (m, n), (n, 1), 2 * step + shift + i * step) for i in range(2)]
    P.ops.GroupedGemv([(x, pk, sc, None, y) for (pk, sc, x), y in zip(probs, ys)], [(n, k)] * 2, peer_delta=[0, (2 * step + shift) * 2])()
    alone = [torch.empty((m, n), dtype=torch.bfloat16, device=dev) for _ in range(2)]
    P.ops.GroupedGemv([(x, pk, sc, None, y) for (pk, sc, x), y in zip(probs, alone)], [(n, k)] * 2)()
    for got, y, want in zip(far, ys, alone):
        assert torch.equal(got, want) and torch.equal(y, want)
        got.fill_(7.0)
        y.fill_(7.0)
    assert bool((flat == 7.0).all())


def test_a_full_launch_queue_does_not_stop_other_threads(P):
    """Launches wait while the GPU's queue is full (here behind a kernel of about half a second); other Python threads go on."""
    dev = torch.device(DEV)
    pk, sc, x = _problem(P, 256, 512, 1, 130)
    y = torch.zeros((1, 256), dtype=torch.bfloat16, device=dev)
    grp = P.ops.GroupedGemv([(x, pk, sc, None, y)], [(256, 512)])
    for launch in (grp, lambda: P.ops.linear(x, pk, sc, None, 256, 512, 32), lambda: P.ops.decode(pk, sc, (256, 512))):
        launch()
        torch.cuda.synchronize()
        torch.cuda._sleep(1_000_000_000)
        worker = threading.Thread(target=lambda: [launch() for _ in range(3000)])
        longest, last = 0.0, time.perf_counter()
        worker.start()
        while worker.is_alive():
            time.sleep(0.002)
            now = time.perf_counter()
            longest, last = max(longest, now - last), now
        worker.join()
        torch.cuda.synchronize()
        assert longest < 0.15, longest


def test_one_matrix_of_more_than_4_gb(P):
    """Rows whose codes lie beyond 4 GB: a weight of 256 rows over and over, so every 256 outputs are the same."""
    n, k, m, dev = 256 * 5469, 16384, 2, torch.device(DEV)              # 4.3 GB of codes
    if torch.cuda.mem_get_info(dev)[0] < 16 << 30:
        pytest.skip("needs 16 GB")
    pk, sc, x = _problem(P, 256, k, m, 140)
    want = P.ops.linear(x, pk, sc, None, 256, k, 32)
    y = torch.empty((m, n), dtype=torch.bfloat16, device=dev)
    P.ops.GroupedGemv([(x, pk.repeat(n // 256), sc.repeat(n // 256), None, y)], [(n, k)])()
    got = y.view(m, n // 256, 256)
    assert bool((got == got[:, :1]).all())
    assert float((got[:, 0].float() - want.float()).norm() / want.float().norm()) <= 4e-3
