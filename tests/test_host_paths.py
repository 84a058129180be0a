"""Host code of the library where a call fails or a buffer is not what it seems, on a CUDA runtime without
a device (fake_runtime.py): which calls are made, in which order, and what a failed call leaves behind."""
import ctypes

import numpy as np
import pytest

import fake_runtime

PAGE = 4096
_open = []


@pytest.fixture
def fake():
    gpu, f = fake_runtime.load()
    f.reset()
    f.unpin_all()
    yield gpu, f
    f.reset()
    f.unpin_all()
    while _open:
        _open.pop().close()
    gpu.finalize()


def _batch(gpu, shapes, nt=40, ntau=16, k=5):
    """A batch with one group per (size1, problems)."""
    b = gpu.Batch([dict(nt=nt, ntau=ntau, size1=s, sig=-1, solve_order=k, sigma_group=g, beta=2.0, h=0.1)
                   for g, (s, cnt) in enumerate(shapes) for _ in range(cnt)])
    _open.append(b)
    return b


def _pages(n):
    """A page-aligned host buffer of n pages: (owner, address)."""
    a = np.zeros((n + 1) * PAGE, np.uint8)
    return a, (a.ctypes.data + PAGE - 1) // PAGE * PAGE


def _launched(f, kernel):
    return [x for x in f.calls("launch") if kernel in x]


# ---- slices in host memory of different kinds -------------------------------------------------------
NT, NTAU = 400, 100  # a slice of step 400: 14.4 kB, four pages


@pytest.mark.parametrize("pins,write,direct", [
    ([(0, 4)], True, True),                     # one range over all of it
    ([(0, 4)], False, True),
    ([(0, 1), (3, 1)], True, False),            # first and last byte pinned, a gap between
    ([(0, 1), (3, 1)], False, False),
    ([(0, 2), (2, 2)], True, False),            # two ranges side by side are two mappings
    ([(0, 3)], True, False),                    # the end is pageable
    ([(1, 3)], True, False),                    # the start is
    ([(0, 4, "read")], False, True),            # a range the device may only read
    ([(0, 4, "read")], True, False),
])
def test_only_memory_in_one_range_is_used_in_place(fake, pins, write, direct):
    gpu, f = fake
    b = _batch(gpu, [(1, 1)], NT, NTAU)
    owner, base = _pages(4)
    for p in pins:
        f.pin(base + p[0] * PAGE, p[1] * PAGE, read_only=len(p) > 2)
    L = gpu.load_library()
    f.reset()
    call = L.nessi_gpu_get_timestep if write else L.nessi_gpu_set_timestep
    assert call(b._h, 0, NT, ctypes.c_void_p(base)) == 0
    assert len(_launched(f, "k_slice")) == (1 if direct else 0)
    assert len(f.calls("cudaMemcpyAsync")) == (0 if direct else 3)
    assert not f.calls("cudaHostAlloc")


def test_pageable_slices_go_through_a_slot(fake):
    gpu, f = fake
    b = _batch(gpu, [(1, 1)], NT, NTAU)
    owner, base = _pages(4)
    f.reset()
    assert gpu.load_library().nessi_gpu_set_timestep(b._h, 0, NT, ctypes.c_void_p(base)) == 0
    assert len(_launched(f, "k_slice")) == 1 and not f.calls("cudaStreamSynchronize")


# ---- order of a step's launches -----------------------------------------------------------------------
def _order(log):
    """(launches, what each stream's next operation is ordered after), from a log: launches by number,
    streams and events as sets of the launches they wait for."""
    seen, events, launches = {}, {}, []
    for line in log:
        w = line.split()
        if w[0] == "launch":
            launches.append(line)
            seen.setdefault(w[1], set()).add(len(launches) - 1)
        elif w[0] == "cudaEventRecord":
            events[w[1]] = set(seen.get(w[2], ()))
        elif w[0] == "cudaStreamWaitEvent":
            seen.setdefault(w[1], set()).update(events.get(w[2], ()))
    return launches, seen


def _batch_stream(f, b, gpu):
    """The number of the batch stream: it is the one that synchronize waits for."""
    f.reset()
    b.synchronize()
    return f.calls("cudaStreamSynchronize")[0].split()[1]


@pytest.mark.parametrize("shapes", [[(1, 3)], [(1, 2), (3, 2), (8, 1)]])
def test_every_launch_of_a_step_is_joined_whatever_fails(fake, shapes):
    gpu, f = fake
    b = _batch(gpu, shapes)
    main = _batch_stream(f, b, gpu)
    b.dyson_timestep(20)
    for call in ("launch", "cudaEventRecord", "cudaStreamWaitEvent"):
        f.reset()
        b.dyson_timestep(20)
        count = len(f.calls(call))
        launches, seen = _order(f.log())
        assert len(launches) > 10 * len(shapes) and seen[main] == set(range(len(launches)))
        for nth in range(1, count + 1):
            f.reset()
            f.fail(call, nth, 1)
            with pytest.raises(gpu.NessiGpuError):
                b.dyson_timestep(20)
            launches, seen = _order(f.log())
            if call == "launch" or nth <= count - 2 * (len(shapes) - 1):  # a last join that fails can only be reported
                assert seen.get(main, set()) == set(range(len(launches))), (call, nth)


# ---- arrays that are allocated at their first use --------------------------------------------------------
def _hm(gpu, nt=40, ntau=16, s=2):
    from nessi_b200 import herm_matrix
    return herm_matrix(nt, ntau, s, -1)


def _table_uploads(f):
    """The copies of sync_groups: the ones that are waited for right after."""
    log = f.log()
    return [a for a, z in zip(log, log[1:]) if a.startswith("cudaMemcpyAsync") and z.startswith("cudaStreamSynchronize")]


@pytest.mark.parametrize("call,nth", [("cudaMalloc", 1), ("cudaMalloc", 2), ("cudaMemcpyAsync", 1), ("cudaStreamSynchronize", 1)])
def test_a_group_becomes_vie2_as_a_whole(fake, call, nth):
    gpu, f = fake
    f.reset()
    b = _batch(gpu, [(2, 2)])
    table = _table_uploads(f)[-1]  # the last one of the creation
    F = _hm(gpu)
    b.dyson_timestep(20)
    f.reset()
    f.fail(call, nth)
    with pytest.raises(gpu.NessiGpuError):
        b.set_F(0, F, F)
    f.reset()
    with pytest.raises(gpu.NessiGpuError) as e:  # not yet: no launch on half of its arrays
        b.vie2_timestep(20)
    assert "has no VIE2" in str(e.value) and not f.calls("launch")
    b.set_F(0, F, F)
    assert table in _table_uploads(f) and len(f.calls("cudaMalloc")) <= 3  # the rest of F, and Fcc^mat
    for p in (0, 1):
        b.set_Q(p, F)
    b.vie2_timestep(20)


@pytest.mark.parametrize("nth", [1, 2, 3, 4])
def test_a_source_term_is_set_as_a_whole(fake, nth):
    gpu, f = fake
    b = _batch(gpu, [(2, 1)])
    F = _hm(gpu)
    b.set_F(0, F, F)
    f.reset()
    f.fail("cudaMalloc", nth)
    with pytest.raises(gpu.NessiGpuError):
        b.set_Q(0, F)
    f.reset()
    with pytest.raises(gpu.NessiGpuError) as e:
        b.vie2_timestep(20)
    assert "not set" in str(e.value) and not f.calls("launch")
    b.set_Q(0, F)
    assert len(f.calls("cudaMalloc")) == 5 - nth  # what the failed call had got is kept
    b.vie2_timestep(20)


@pytest.mark.parametrize("nth", [1, 2, 3, 4, 5])
def test_the_average_is_allocated_as_a_whole(fake, nth):
    gpu, f = fake
    b = _batch(gpu, [(2, 3)])
    f.reset()
    f.fail("cudaMalloc", nth)
    with pytest.raises(gpu.NessiGpuError):
        b.gloc_timestep(0, 20)
    f.reset()
    b.gloc_timestep(0, 20)
    assert len(f.calls("cudaMalloc")) == 6 - nth and _launched(f, "k_gloc_final")


# ---- chained launches ---------------------------------------------------------------------------------------
def _chained_after_a_wait(log):
    """The chained launches whose stream was last told to wait for another stream."""
    last, bad = {}, []
    for line in log:
        w = line.split()
        if w[0] == "cudaStreamWaitEvent":
            last[w[1]] = line
        elif w[0] == "launch":
            if w[2] == "chained" and last.get(w[1], "").startswith("cudaStreamWaitEvent"):
                bad.append(line)
            last[w[1]] = line
    return bad


@pytest.mark.parametrize("shapes", [[(1, 3)], [(2, 70)], [(1, 2), (3, 2), (8, 1)], [(1, 1)] * 70 + [(2, 1)]])
def test_the_first_launch_after_a_wait_is_plain(fake, shapes):
    gpu, f = fake
    b = _batch(gpu, shapes)
    U = np.ones((42, shapes[0][0]), np.complex128)
    b.set_U(0, U)
    f.reset()
    for n in (20, 21):
        b.dyson_timestep(n)
    for n in (22, 23):
        b.lattice_2b_timestep(n, 2)
    b.dyson_timestep(24)
    b.sigma_2b_timestep(0, 24)
    log = f.log()
    assert not _chained_after_a_wait(log)
    # and most launches are chained: the rule costs no more than the waits of a step
    kinds = [x.split()[2] for x in log if x.startswith("launch")]
    waits = sum(x.startswith("cudaStreamWaitEvent") for x in log)
    assert kinds.count("chained") > 0.5 * len(kinds) and waits < len(kinds)


# ---- staging blocks of the process ---------------------------------------------------------------------------
def _slices(gpu, b, nt=40, ntau=16, s=2, count=6):
    data = np.zeros((2 * (nt + 1) + ntau + 1, s, s), np.complex128)
    for _ in range(count):
        b.set_timestep(0, nt, data)
        b.get_timestep(0, nt, data)


def test_batches_in_a_row_share_a_staging_block(fake):
    gpu, f = fake
    f.reset()
    for _ in range(5):
        b = _batch(gpu, [(2, 1)])
        _slices(gpu, b)
        b.close()
    assert len(f.calls("cudaHostAlloc")) == 1 and not f.calls("cudaFreeHost")
    log = f.log()  # before it is handed on, a batch waits for the uploads that read it
    last = max(i for i, x in enumerate(log) if x.startswith("cudaEventSynchronize"))
    assert last > max(i for i, x in enumerate(log) if x.startswith("launch"))
    gpu.finalize()
    assert len(f.calls("cudaFreeHost")) == 1
    f.reset()
    b = _batch(gpu, [(2, 1)])
    _slices(gpu, b)
    assert len(f.calls("cudaHostAlloc")) == 1  # nothing is kept past finalize


def test_batches_beside_each_other_have_blocks_of_their_own(fake):
    gpu, f = fake
    f.reset()
    bs = [_batch(gpu, [(2, 1)]) for _ in range(20)]
    for b in bs:
        _slices(gpu, b)
    assert len(f.calls("cudaHostAlloc")) == 20
    for b in bs:
        b.close()
    assert len(f.calls("cudaFreeHost")) == 4  # 16 are kept
    gpu.finalize()
    assert len(f.calls("cudaFreeHost")) == 20


def test_the_kept_blocks_are_bounded_in_bytes(fake):
    gpu, f = fake
    f.reset()
    nt, ntau, s = 300, 20, 8  # a slice of 638 kB
    bs = [_batch(gpu, [(s, 1)], nt, ntau) for _ in range(15)]
    for b in bs:
        _slices(gpu, b, nt, ntau, s, 1)
    sizes = [int(x.split()[1]) for x in f.calls("cudaHostAlloc")]
    assert len(sizes) == 15 and sizes[0] >= 4 * 16 * s * s * (2 * (nt + 1) + ntau + 1)
    for b in bs:
        b.close()
    assert 15 - len(f.calls("cudaFreeHost")) == (32 << 20) // sizes[0]
    f.reset()
    b = _batch(gpu, [(2, 1)])  # a block that is larger than needed serves too
    _slices(gpu, b)
    assert not f.calls("cudaHostAlloc")


def test_a_failed_wait_keeps_a_block_from_the_next_batch(fake):
    gpu, f = fake
    b = _batch(gpu, [(2, 1)])
    _slices(gpu, b, count=1)
    f.reset()
    f.fail("cudaEventSynchronize", 1, 1)
    b.close()
    assert len(f.calls("cudaFreeHost")) == 1


def test_creation_makes_no_more_calls_than_it_needs(fake):
    """A batch of one size has no second pair of streams, and its error word, descriptor table and their
    upload are one allocation and one wait."""
    gpu, f = fake
    _batch(gpu, [(2, 1)])
    f.reset()
    _batch(gpu, [(2, 1)])
    assert len(f.calls("cudaStreamSynchronize")) == 1 and not f.calls("cudaMemset")
    assert len(f.calls("cudaEventCreate")) == 2 and len(f.calls("cudaStreamCreate")) == 2
    assert len(f.calls("cudaMalloc")) == 7 + 1 + 16 + 1 + 1  # problem, scratch, group, problems' and groups' tables


# ---- kernel attributes ----------------------------------------------------------------------------------------
def test_kernel_attributes_are_set_again_after_finalize(fake):
    gpu, f = fake

    def step():
        b = _batch(gpu, [(4, 2)])
        f.reset()
        b.dyson_timestep(30)
        sets = f.calls("cudaFuncSetAttribute")
        b.close()
        return sets
    first = step()
    assert not step()  # once per kernel and size
    gpu.finalize()     # a context that is made after it starts without them
    again = step()
    assert again and (not first or again == first)


# ---- which form of a product a step takes -------------------------------------------------------------------
@pytest.mark.parametrize("s,cnt,tiled", [(2, 896, True), (2, 880, False),  # 16 x 56 tiles of 32 x 32, 16 x 55; the line is 6 x 148
                                         (3, 400, False), (4, 224, False), (8, 112, False)])
def test_les_adv_is_tiled_for_small_blocks_only(fake, s, cnt, tiled):
    gpu, f = fake
    n = 255
    b = _batch(gpu, [(s, cnt)], nt=n, ntau=8)
    f.reset()
    b.dyson_timestep(n)
    products = [x for x in f.calls("launch") if "k_zgemm" in x]
    assert len(products) == 3
    assert [("k_zgemm<1>" in x) for x in products].count(True) == int(tiled)  # <1>: Sigma^< G^A, tiled


@pytest.mark.parametrize("s,ntau,cnt,mixed,ret,les", [
    (1, 75, 1200, False, 150, 150),                  # 8 columns a CTA: 219 KB with the tv ring on an SM
    (2, 150, 290, False, 145, 145), (2, 150, 300, False, 150, 75),  # 4 at most for ret, 8 for les
    (2, 149, 300, False, 75, 75),                    # a short stream
    (2, 150, 300, True, 75, 75),                     # no ring in a mixed step
    (3, 225, 52, False, 78, 78),                     # 2
    (4, 300, 37, False, 148, 148), (4, 300, 40, False, 160, 80), (4, 299, 40, False, 80, 80),  # 1 and 2
    (5, 375, 61, False, 77, 77), (8, 600, 38, False, 76, 76)])      # 4: the ring has the SM to itself
def test_the_retarded_recursion_leaves_room_for_the_tv_ring(fake, s, ntau, cnt, mixed, ret, les):
    gpu, f = fake
    b = gpu.Batch([dict(nt=30, ntau=ntau, size1=s, sig=-1, solve_order=5, beta=2.0, h=0.1)] * cnt,
                  gpu.PREC_MIXED if mixed else gpu.PREC_FP64)
    _open.append(b)
    f.reset()
    b.dyson_timestep(30)
    grids = {kind: {int(x.split(" grid ")[1].split()[0]) for x in f.calls("launch")
                    if "k_vol_block<%d, false, %s>" % (s, kind) in x} for kind in ("true", "false")}
    assert grids == {"true": {ret}, "false": {les}}
