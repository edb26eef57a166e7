"""GPU tests at the sizes where a kernel's range ends: window sizes at which the format builder changes
method, column counts around the warp-level kernel's groups, odd row lengths, neighbour lists and traversals
of unusual shape in the row reorders.  Everything against the CPU oracle."""
import numpy as np
import pytest

from mask_b200 import generators as G
from tests.test_gpu_pack import _check_mco, _check_metcf, _check_srbcrs, _dev
from tests.test_gpu_spmm import _assert_close

pytestmark = pytest.mark.gpu


def _rows_to_csr(rows, K, seed):
    rowptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    colind = np.concatenate(rows).astype(np.int32) if rowptr[-1] else np.zeros(0, np.int32)
    values = np.random.Generator(np.random.PCG64(seed)).uniform(-1, 1, colind.size).astype(np.float32)
    return G.CSR(len(rows), K, rowptr, colind, values)


def _window(n, K, hub, seed):
    """16 rows with n entries in all, most of them in one row if `hub`."""
    rng = np.random.Generator(np.random.PCG64(seed))
    share = np.full(16, n // 16) if not hub else np.full(16, n // 64)
    share[3] += n - share.sum()
    return [np.sort(rng.choice(K, int(c), replace=False)) for c in share]


# sizes at which a window is sorted with more registers, ranked in one block's bitmap, shared by a cluster; key
# width changes at 2^22 columns, a block's bitmap covers 2^19 columns at a time (in a cluster 2^20 from 2^22 to 2^23 columns)
@pytest.mark.parametrize("K", [3000, 600_000, 2_200_000, 4_300_000])
@pytest.mark.parametrize("hub", [False, True])
def test_pack_window_sizes(oracle_mod, K, hub):
    from mask_b200 import engine
    sizes = [0, 1, 32, 33, 64, 65, 128, 129, 256, 257, 512, 513, 1023, 1024, 1025, 8191, 8192, 8193, 20000]
    sizes = [n for n in sizes if n < 0.7 * K]
    rows = []
    for i, n in enumerate(sizes):
        rows += _window(n, K, hub, 100 + i)
    m = _rows_to_csr(rows[:-5], K, 7)   # the last window is ragged
    rp, ci, va = _dev(m)
    _check_srbcrs(engine.pack_srbcrs(rp, ci, va, m.M, m.K), oracle_mod.pack_srbcrs(m.M, m.rowptr, m.colind, m.values))
    _check_metcf(engine.pack_metcf(rp, ci, va, m.M, m.K), oracle_mod.pack_metcf(m.M, m.rowptr, m.colind, m.values))
    _check_mco(engine.pack_mco(rp, ci, va, m.M, m.K), oracle_mod.pack_mco(m.M, m.rowptr, m.colind, m.values))


# Windows shared by a cluster: up to 4096 entries a block are kept in registers, more are read again, and a block's range of
# columns is taken in parts where eight bitmaps do not cover K (beyond 2^23); `skew`: most entries among the first columns, so that
# the ranges differ in width
@pytest.mark.parametrize("K", [1 << 18, 1 << 20, 1 << 21, 1 << 22, (1 << 22) + 1, 1 << 23, (1 << 23) + 1, 1 << 24])
@pytest.mark.parametrize("skew", [False, True])
def test_pack_hub_windows(oracle_mod, K, skew):
    from mask_b200 import engine
    rng = np.random.Generator(np.random.PCG64(K + skew))
    rows = []
    for n, longest in ((30_000, 1 / 16), (32_768, 0.6), (70_000, 1 / 16), (200_000, 1 / 16), (200_000, 0.6)):
        for r in range(16):
            u = rng.random(int(n * (longest if r == 5 else (1 - longest) / 15)))
            rows.append(np.unique((K * (u ** 4 if skew else u)).astype(np.int32)))
    m = _rows_to_csr(rows[:-2], K, 7)
    rp, ci, va = _dev(m)
    _check_srbcrs(engine.pack_srbcrs(rp, ci, va, m.M, m.K), oracle_mod.pack_srbcrs(m.M, m.rowptr, m.colind, m.values))
    _check_metcf(engine.pack_metcf(rp, ci, va, m.M, m.K), oracle_mod.pack_metcf(m.M, m.rowptr, m.colind, m.values))


def test_pack_time_of_hub_windows_does_not_jump_with_the_columns():
    """200 windows of 100 000 entries spread over 2^22 columns cost about what they cost over 2^20.  With ranges taken in parts
    they took 1.2 ms against 0.5; 1.6 times leaves room for noise."""
    import torch
    from mask_b200 import engine
    windows, per = 200, 6250
    gen = torch.Generator(device="cuda").manual_seed(3)
    rowptr = torch.arange(16 * windows + 1, dtype=torch.int32, device="cuda") * per
    ms = {}
    for K in (1 << 20, 1 << 22):
        step = K // per
        colind = torch.arange(per, device="cuda") * step + torch.randint(0, step, (16 * windows, per), generator=gen, device="cuda")
        colind = colind.to(torch.int32).reshape(-1)
        times = []
        for _ in range(7):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize()
            a.record()
            engine._analyze(rowptr, colind, 16 * windows, K)
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        ms[K] = sorted(times)[3]
    assert ms[1 << 22] < 1.6 * ms[1 << 20], ms


@pytest.mark.parametrize("n", [40, 1030, 9000])
@pytest.mark.parametrize("fault", ["order", "range"])
def test_pack_finds_faults_in_every_kind_of_window(n, fault):
    from mask_b200 import _lib, engine
    K = 40_000
    m = _rows_to_csr(_window(n, K, True, 3), K, 7)
    e = int(m.rowptr[4]) - 2            # near the end of the longest row
    if fault == "order":
        m.colind[e], m.colind[e + 1] = m.colind[e + 1], m.colind[e]
    else:
        m.colind[e + 1] = K
    with pytest.raises(_lib.MaskError) as err:
        engine.pack_srbcrs(*_dev(m), m.M, m.K)
    assert err.value.status == (3 if fault == "order" else 6)


def _mixed_matrix():
    """Power-law rows, an empty window, a window long enough to be split, a ragged end."""
    a = G.rmat_gcn_normalised(scale=10, samples_per_node=8, seed=5)
    rows = [a.colind[a.rowptr[i]:a.rowptr[i + 1]] for i in range(700)]
    rows[64:80] = [np.zeros(0, np.int32)] * 16
    rng = np.random.Generator(np.random.PCG64(2))
    rows[100] = np.sort(rng.choice(a.K, 900, replace=False)).astype(np.int32)
    return _rows_to_csr(rows[:-3], a.K, 9)


@pytest.mark.parametrize("fmt", ["srbcrs", "metcf", "mco"])
@pytest.mark.parametrize("N", [4, 28, 32, 36, 64, 68, 96, 100, 128, 132, 192, 260])
def test_warp_kernel_column_counts(oracle_mod, fmt, N):
    import torch
    from mask_b200 import engine
    m = _mixed_matrix()
    p = {"srbcrs": engine.pack_srbcrs, "metcf": engine.pack_metcf, "mco": engine.pack_mco}[fmt](*_dev(m), m.M, m.K)
    B = np.random.Generator(np.random.PCG64(N)).standard_normal((m.K, N), dtype=np.float32)
    Bd = torch.from_numpy(B).cuda()
    engine.tune("sweep", 0)
    try:
        plan = p.new_plan("auto")
        assert engine.kernel_signature(p, N, plan)[0] == f"spmm_warp_kernel<{fmt}>"
        for gt in (0, 5):               # whole windows and split ones
            out = torch.full((m.M, N), float("nan"), device="cuda")
            engine.spmm(p, Bd, out=out, plan=p.new_plan("auto", gt), relu=gt == 5)
            _assert_close(oracle_mod, m, B, out.cpu().numpy(), relu=gt == 5)
        if fmt == "srbcrs":
            out = engine.spmm(p, Bd, plan=plan, tf32x3=True).cpu().numpy()
            ref = oracle_mod.spmm_f32(m.M, m.rowptr, m.colind, m.values, B)
            absp = oracle_mod.spmm_abs_f64(m.M, m.rowptr, m.colind, m.values, B)
            bad, worst = oracle_mod.check_tolerance(out, ref, absp, 2e-5, 1e-6)
            assert bad == 0, worst
    finally:
        engine.tune("sweep", 1)


# numbers of windows at which the warp kernel takes more or fewer tiles a step and columns a block
@pytest.mark.parametrize("fmt", ["srbcrs", "metcf", "mco"])
@pytest.mark.parametrize("N", [32, 64, 96, 124, 256])
@pytest.mark.parametrize("windows", [37, 440, 1000, 1700, 4100])
def test_warp_kernel_step_lengths(oracle_mod, fmt, N, windows):
    import torch
    from mask_b200 import engine
    rng = np.random.Generator(np.random.PCG64(windows))
    K, length = 1900, rng.integers(0, 25, 16 * windows - 3)
    rows = [np.sort(rng.choice(K, n, replace=False)) for n in length]
    m = _rows_to_csr(rows, K, 3)
    p = {"srbcrs": engine.pack_srbcrs, "metcf": engine.pack_metcf, "mco": engine.pack_mco}[fmt](*_dev(m), m.M, m.K)
    B = rng.standard_normal((K, N), dtype=np.float32)
    Bd = torch.from_numpy(B).cuda()
    engine.tune("sweep", 0)
    try:
        _assert_close(oracle_mod, m, B, engine.spmm(p, Bd).cpu().numpy())
        if fmt == "srbcrs":
            out = engine.spmm(p, Bd, tf32x3=True).cpu().numpy()
            bad, worst = oracle_mod.check_tolerance(out, oracle_mod.spmm_f32(m.M, m.rowptr, m.colind, m.values, B),
                                                    oracle_mod.spmm_abs_f64(m.M, m.rowptr, m.colind, m.values, B), 2e-5, 1e-6)
            assert bad == 0, worst
    finally:
        engine.tune("sweep", 1)


# tiles with all 128 entries beside tiles with one, windows of 0, 1, 4, 5 and 9 tiles (batches of ids are 4 or 8 tiles), every step
# length; gt: groups of single tiles, of a few, and as the plan has them
@pytest.mark.parametrize("fmt", ["srbcrs", "metcf", "mco"])
@pytest.mark.parametrize("N", [32, 64, 96, 260])
@pytest.mark.parametrize("windows", [9, 900, 5000])
@pytest.mark.parametrize("gt", [0, 1, 6])
def test_warp_kernel_full_tiles_beside_single_entries(oracle_mod, fmt, N, windows, gt):
    import torch
    from mask_b200 import engine
    rng = np.random.Generator(np.random.PCG64(windows + gt))
    K, rows = 300, []
    for w in range(windows):
        tiles = (0, 1, 4, 5, 9)[w % 5]
        full = np.sort(rng.choice(K, 8 * tiles, replace=False))
        rows += [full if w % 3 else full[r::16] for r in range(16)]
    m = _rows_to_csr(rows[:-3], K, 5)
    p = {"srbcrs": engine.pack_srbcrs, "metcf": engine.pack_metcf, "mco": engine.pack_mco}[fmt](*_dev(m), m.M, m.K)
    B = rng.standard_normal((K, N), dtype=np.float32)
    out = torch.full((m.M, N), float("nan"), device="cuda")
    engine.tune("sweep", 0)
    try:
        engine.spmm(p, torch.from_numpy(B).cuda(), out=out, plan=p.new_plan("auto", gt))
    finally:
        engine.tune("sweep", 1)
    _assert_close(oracle_mod, m, B, out.cpu().numpy())


# the groups of the warp kernel are found in chunks of 2048 fragments; the last chunk may be shorter than a group and have none of its own
@pytest.mark.parametrize("windows", [2047, 2048, 2049, 2050, 2052, 4096, 4097, 4099])
def test_plan_groups_at_the_edges_of_chunks(oracle_mod, windows):
    import torch
    from mask_b200 import engine
    rng = np.random.Generator(np.random.PCG64(windows))
    K = 2500
    rows = [np.sort(rng.choice(K, n, replace=False)) for n in rng.integers(0, 3, 16 * windows - 5)]
    m = _rows_to_csr(rows, K, 7)
    p = engine.pack_srbcrs(*_dev(m), m.M, m.K)
    B = rng.standard_normal((K, 64), dtype=np.float32)
    out = torch.full((m.M, 64), float("nan"), device="cuda")
    engine.tune("sweep", 0)
    try:
        engine.spmm(p, torch.from_numpy(B).cuda(), out=out)
    finally:
        engine.tune("sweep", 1)
    _assert_close(oracle_mod, m, B, out.cpu().numpy())


# windows that are far longer than the groups around them are taken first: none, at the end, over the chunks of 2048 fragments in
# which the groups are written; 26 tiles are too few, 27 enough, more than 5/4 of a piece are split
@pytest.mark.parametrize("windows", [60, 2047, 2049, 6200])
@pytest.mark.parametrize("long_tiles", [0, 26, 27, 100, 300])
def test_long_windows_among_short_ones(oracle_mod, windows, long_tiles):
    import torch
    from mask_b200 import engine
    rng = np.random.Generator(np.random.PCG64(windows + long_tiles))
    K, rows = 2500, []
    for w in range(windows):
        long = long_tiles and (w % 97 == 50 or w >= windows - 3)
        cols = np.sort(rng.choice(K, min(8 * long_tiles, K) if long else int(rng.integers(0, 20)), replace=False))
        rows += [cols[r::16] for r in range(16)]
    m = _rows_to_csr(rows[:-5], K, 7)
    p = engine.pack_srbcrs(*_dev(m), m.M, m.K)
    B = rng.standard_normal((K, 64), dtype=np.float32)
    out = torch.full((m.M, 64), float("nan"), device="cuda")
    engine.tune("sweep", 0)
    try:
        engine.spmm(p, torch.from_numpy(B).cuda(), out=out)
    finally:
        engine.tune("sweep", 1)
    _assert_close(oracle_mod, m, B, out.cpu().numpy())


def _windows_of(tiles, K, seed):
    """Windows of exactly tiles[w] tiles, columns spread over all K."""
    rng = np.random.Generator(np.random.PCG64(seed))
    rows = []
    for t in tiles:
        step = K // max(8 * t, 1)
        cols = np.arange(8 * t) * step + rng.integers(0, step, 8 * t)
        rows += [cols[r::16].astype(np.int32) for r in range(16)]
    return _rows_to_csr(rows, K, seed)


def _warp_groups(plan):
    """The groups of the warp kernel: those taken first, the others; (first fragment, end, first tile, tiles) each."""
    import ctypes as C
    from mask_b200 import _lib
    first, rest = C.c_int64(), C.c_int64()
    _lib.check(_lib.lib().mask_plan_warp_groups(plan._h, C.byref(first), C.byref(rest), None), "mask_plan_warp_groups")
    groups = np.full((first.value + rest.value, 4), -1, np.int32)
    _lib.check(_lib.lib().mask_plan_warp_groups(plan._h, None, None, groups.ctypes.data), "mask_plan_warp_groups")
    return groups[:first.value], groups[first.value:]


# Windows long enough to be groups of their own, none of them cut (a piece is as long as the mean window): which are listed, by
# their tiles and their place; 26 tiles are too few wherever they are, 27 enough where what is left is 16 tiles a resident warp
@pytest.mark.parametrize("windows", [60, 2047, 2049, 6200])
@pytest.mark.parametrize("long,short", [(26, 18), (27, 18), (100, 64)])
def test_which_windows_are_taken_first(oracle_mod, windows, long, short):
    import torch
    from mask_b200 import engine
    tiles = np.where(np.arange(windows) % 2 == 1, long, short)
    K = 200_000
    m = _windows_of(tiles, K, windows + long)
    p = engine.pack_srbcrs(*_dev(m), m.M, m.K)
    plan = p.new_plan()
    first, rest = _warp_groups(plan)
    assert p.T == tiles.sum() and plan.info()["partial"] == 0 and plan.column_features()["local_share"] < 0.9
    before = np.cumsum(tiles) - tiles
    takers = 15 * torch.cuda.get_device_properties(0).multi_processor_count
    left = (tiles.sum() + 4 * windows - before - 4 * np.arange(windows)) // takers
    target = np.clip(left, 16, 128)
    listed = 2 * (tiles + 4) > 3 * (target * 5 // 4)
    assert sorted(first[:, 0]) == list(np.flatnonzero(listed))
    # every fragment in exactly one group, every group with the tiles of its fragments
    groups = np.concatenate([first, rest[rest[:, 1] > rest[:, 0]]])
    groups = groups[np.argsort(groups[:, 0])]
    assert groups[0, 0] == 0 and groups[-1, 1] == windows and np.array_equal(groups[1:, 0], groups[:-1, 1])
    assert np.array_equal(groups[:, 2], before[groups[:, 0]]) and np.array_equal(groups[:, 3], np.add.reduceat(tiles, groups[:, 0]))
    B = np.random.Generator(np.random.PCG64(1)).standard_normal((K, 64), dtype=np.float32)
    engine.tune("sweep", 0)
    try:
        out = engine.spmm(p, torch.from_numpy(B).cuda(), plan=plan)
    finally:
        engine.tune("sweep", 1)
    _assert_close(oracle_mod, m, B, out.cpu().numpy())


# Columns of a block and tiles a step by the number of groups (one a window up to 1700), on both sides of what an SM holds; bitmaps take
# more room.  At 64 columns and more blocks than are resident, two tiles a step.
@pytest.mark.parametrize("fmt,N,windows,shape", [
    ("srbcrs", 32, 800, (32, 8)), ("metcf", 32, 800, (32, 8)), ("mco", 32, 740, (32, 8)), ("mco", 32, 800, (32, 4)),
    ("srbcrs", 32, 1700, (32, 4)), ("mco", 32, 1480, (32, 4)), ("mco", 32, 1700, (32, 2)),
    ("srbcrs", 64, 1000, (64, 4)), ("mco", 64, 880, (64, 4)), ("mco", 64, 1000, (64, 2)),
    ("srbcrs", 128, 560, (128, 4)), ("mco", 128, 440, (64, 4)), ("mco", 128, 560, (64, 2)), ("mco", 128, 1180, (128, 2)), ("mco", 128, 1190, (64, 1)),
    ("srbcrs", 96, 1400, (96, 2)), ("mco", 96, 1330, (96, 2)), ("mco", 96, 1400, (96, 1)), ("mco", 96, 1440, (96, 2)), ("mco", 96, 1490, (96, 1)),
    ("srbcrs", 64, 12_000, (64, 2)), ("metcf", 64, 12_000, (64, 2)), ("mco", 64, 12_000, (64, 2)), ("srbcrs", 96, 12_000, (96, 1)),
    ("srbcrs", 64, 16_000, (64, 1)), ("mco", 64, 16_000, (64, 2))])
def test_warp_kernel_shape(oracle_mod, fmt, N, windows, shape):
    import ctypes as C
    import torch
    from mask_b200 import _lib, engine
    K = 200_000
    m = _windows_of(np.full(windows, 26), K, windows)
    p = {"srbcrs": engine.pack_srbcrs, "metcf": engine.pack_metcf, "mco": engine.pack_mco}[fmt](*_dev(m), m.M, m.K)
    plan = p.new_plan()
    columns, step = C.c_int32(), C.c_int32()
    code = {"srbcrs": 0, "metcf": 1, "mco": 2}[fmt]
    _lib.check(_lib.lib().mask_spmm_warp_shape(plan._h, code, N, 0, C.byref(columns), C.byref(step)), "mask_spmm_warp_shape")
    assert (columns.value, step.value) == shape, len(_warp_groups(plan)[1])
    B = np.random.Generator(np.random.PCG64(N)).standard_normal((K, N), dtype=np.float32)
    engine.tune("sweep", 0)
    try:
        out = engine.spmm(p, torch.from_numpy(B).cuda(), plan=plan)
    finally:
        engine.tune("sweep", 1)
    _assert_close(oracle_mod, m, B, out.cpu().numpy())


# The kernel that measured faster, on both sides of the lines of the choice: compact tiles by groups an SM (20 000 rows: 8.4, 4096:
# 1.7) and columns, full-width SR-BCRS of power-law graphs whose B is 4 to 8 times the L2, short groups of 24 tiles
@pytest.mark.parametrize("rows,cols,fmt,N,kernel", [
    (20_000, 10, "metcf", 32, "warp"), (20_000, 10, "mco", 64, "warp"), (20_000, 10, "metcf", 96, "warp"), (20_000, 10, "mco", 108, "sweep"),
    (20_000, 10, "metcf", 192, "sweep"), (40_000, 10, "metcf", 192, "warp"), (20_000, 10, "metcf", 320, "warp"), (20_000, 10, "mco", 512, "sweep"),
    (4096, 21, "metcf", 64, "sweep"), (4096, 21, "srbcrs", 64, "warp"), (6000, 12, "srbcrs", 320, "warp"), (700, 4, "mco", 512, "warp"),
    (1 << 18, 0, "srbcrs", 512, "warp"), (1 << 18, 0, "metcf", 512, "warp"), (60_000, 0, "srbcrs", 512, "sweep"), (60_000, 0, "metcf", 448, "sweep")])
def test_kernel_choice(oracle_mod, rows, cols, fmt, N, kernel):
    import torch
    from mask_b200 import engine
    rng = np.random.Generator(np.random.PCG64(rows + N))
    if cols:
        m = _rows_to_csr([np.unique(rng.integers(0, rows, c)) for c in rng.poisson(cols, rows)], rows, 5)
    else:   # power-law, the first `rows` nodes
        a = G.rmat_gcn_normalised(scale=18 if rows > 65_536 else 16, samples_per_node=16, seed=5)
        keep = np.repeat(np.arange(a.M), np.diff(a.rowptr)) < rows
        keep &= a.colind < rows
        counts = np.add.reduceat(np.append(keep, False), np.minimum(a.rowptr[:rows], len(keep))) * (np.diff(a.rowptr[:rows + 1]) > 0)
        m = G.CSR(rows, rows, np.concatenate([[0], np.cumsum(counts)]).astype(np.int32), a.colind[keep], a.values[keep])
    p = {"srbcrs": engine.pack_srbcrs, "metcf": engine.pack_metcf, "mco": engine.pack_mco}[fmt](*_dev(m), m.M, m.K)
    assert engine.kernel_signature(p, N, p.plan())[0].startswith(f"spmm_{kernel}_kernel")
    B = rng.standard_normal((m.K, N), dtype=np.float32)
    _assert_close(oracle_mod, m, B, engine.spmm(p, torch.from_numpy(B).cuda()).cpu().numpy())


@pytest.mark.parametrize("fmt", ["srbcrs", "metcf", "mco"])
@pytest.mark.parametrize("N,offset,sweep", [(1, 0, 1), (3, 0, 1), (47, 0, 1), (47, 1, 2), (64, 3, 1), (129, 2, 1), (515, 0, 2)])
def test_rows_that_are_not_whole_vectors(oracle_mod, fmt, N, offset, sweep):
    """Any column count, B and C at any multiple of 4 bytes, whole and split windows, both kernels, and a row map."""
    import torch
    from mask_b200 import engine
    m = _mixed_matrix()
    dev = _dev(m)
    p = {"srbcrs": engine.pack_srbcrs, "metcf": engine.pack_metcf, "mco": engine.pack_mco}[fmt](*dev, m.M, m.K)
    packed = [(p, None), (p, 5)]
    if fmt == "srbcrs":
        packed.append((engine.pack_srbcrs(*dev, m.M, m.K, reorder="first_col_sort"), None))
    B = np.random.Generator(np.random.PCG64(N)).standard_normal((m.K, N), dtype=np.float32)
    Bd = torch.empty(m.K * N + offset, device="cuda")[offset:].view(m.K, N)
    Bd.copy_(torch.from_numpy(B))
    engine.tune("sweep", sweep)
    try:
        for q, gt in packed:
            whole = torch.full((m.M * N + offset + 64,), 7.0, device="cuda")
            out = whole[offset:offset + m.M * N].view(m.M, N)
            engine.spmm_any_width(q, Bd, out=out, plan=q.new_plan("auto", gt or 0))
            _assert_close(oracle_mod, m, B, out.cpu().numpy())
            assert bool((whole[:offset] == 7).all()) and bool((whole[offset + m.M * N:] == 7).all())   # nothing beside C was written
    finally:
        engine.tune("sweep", 1)


@pytest.mark.parametrize("fmt", ["srbcrs", "metcf", "mco"])
@pytest.mark.parametrize("N", [47, 130])
def test_rows_that_are_not_whole_vectors_under_the_comparison_knobs(oracle_mod, fmt, N):
    """The register-pipelined kernel, which only the knobs select, writes C 16 bytes at a time."""
    import torch
    from mask_b200 import engine
    m = _mixed_matrix()
    p = {"srbcrs": engine.pack_srbcrs, "metcf": engine.pack_metcf, "mco": engine.pack_mco}[fmt](*_dev(m), m.M, m.K)
    B = np.random.Generator(np.random.PCG64(N)).standard_normal((m.K, N), dtype=np.float32)
    engine.tune("sweep", 0)
    engine.tune("async", 0)
    try:
        for gt in (0, 5):
            out = engine.spmm_any_width(p, torch.from_numpy(B).cuda(), plan=p.new_plan("auto", gt))
            _assert_close(oracle_mod, m, B, out.cpu().numpy())
    finally:
        engine.tune("sweep", 1)
        engine.tune("async", 1)


def _graph(edges, n, extra=()):
    e = np.array(sorted(set(edges) | set(extra)), dtype=np.int64)
    order = np.lexsort((e[:, 1], e[:, 0])) if len(e) else np.zeros(0, np.int64)
    rows = np.split(e[order, 1], np.cumsum(np.bincount(e[:, 0], minlength=n))[:-1]) if len(e) else [np.zeros(0)] * n
    return _rows_to_csr([r.astype(np.int32) for r in rows], n, 1)


def _both(pairs):
    return {(a, b) for a, b in pairs} | {(b, a) for a, b in pairs}


GRAPHS = {
    # one node a level: the part of the traversal that one block does alone, thousands of levels
    "path": lambda: _graph(_both((i, i + 1) for i in range(2999)), 3000),
    # lists longer than a warp sorts (1024) and longer than a block walks at once, and a level of 5000 nodes
    "stars": lambda: _graph(_both([(0, i) for i in range(1, 5001)] + [(7000, i) for i in range(5001, 6100)]), 7001),
    # not symmetric: a one-way ring with chords, and entries on the diagonal
    "one_way": lambda: _graph({(i, (i + 1) % 500) for i in range(500)} | {(i, (7 * i) % 500) for i in range(500)} | {(i, i) for i in range(0, 500, 3)}, 500),
    # hundreds of components of different sizes, isolated nodes between them
    "components": lambda: _graph(_both((10 * c + i, 10 * c + i + 1) for c in range(300) for i in range(c % 8)), 3000),
    # more edges than are united at once: two grids, long lists that join some of their nodes, lone paths
    "many_edges": lambda: _graph(_both([(i, i + d) for i in range(18_000) for d in (1, 150) if (i + d) // 9_000 == i // 9_000]
                                       + [(18_200, i) for i in range(0, 9_000, 4)] + [(18_201, i) for i in range(9_000, 18_000, 5)]
                                       + [(18_300 + 3 * i, 18_301 + 3 * i) for i in range(50)]
                                       + [(i, (i * 7919) % 8_000) for i in range(8_000) if i != (i * 7919) % 8_000]
                                       + [(9_000 + i, 9_000 + (i * 5171) % 8_000) for i in range(8_000) if i != (i * 5171) % 8_000]
                                       + [(i, (i * 6007 + 5) % 8_000) for i in range(8_000) if i != (i * 6007 + 5) % 8_000]
                                       + [(i, (i * 3001 + 9) % 8_000) for i in range(8_000) if i != (i * 3001 + 9) % 8_000]), 18_500),
    "no_edges": lambda: _graph({(3, 3)}, 50),
    "single": lambda: _graph({(0, 0)}, 1),
}


@pytest.mark.parametrize("name", sorted(GRAPHS))
@pytest.mark.parametrize("kind", ["row_rcm", "first_col_sort", "jaccard_greedy"])
def test_reorders_of_unusual_graphs(oracle_mod, name, kind):
    from mask_b200 import engine
    m = GRAPHS[name]()
    rp, ci, va = _dev(m)
    order = engine.reorder_rows(rp, ci, m.M, m.K, kind)
    want = oracle_mod.reorder_rows(kind, m.M, m.K, m.rowptr, m.colind)
    assert np.array_equal(order.cpu().numpy(), want)
    got = engine.permute_rows(rp, ci, va, m.M, order)
    for a, b in zip(got, oracle_mod.permute_csr(m.M, m.rowptr, m.colind, m.values, want)):
        assert np.array_equal(a.cpu().numpy(), b)


def test_column_features_with_very_hot_columns():
    """More than 8192 gathers of a column: the counts that are listed instead of binned."""
    import ctypes as C
    import torch
    from mask_b200 import _lib, engine
    M, K = 16 * 9000, 70_000
    rows = [np.array([0, 5, 100 + (i * 37) % 60_000], dtype=np.int32) if i % 16 == 0 else np.zeros(0, np.int32) for i in range(M)]
    m = _rows_to_csr(rows, K, 3)
    rp, ci, va = _dev(m)
    p = engine.pack_srbcrs(rp, ci, va, m.M, m.K)
    f = _lib.ColumnFeatures()
    _lib.check(_lib.lib().mask_features_columns(p.val_soff.data_ptr(), p.val_sidx.data_ptr(), m.M, m.K, p.T, 512, C.byref(f),
                                                C.c_void_p(torch.cuda.current_stream().cuda_stream)), "mask_features_columns")
    counts = np.bincount(p.val_sidx.cpu().numpy(), minlength=K)
    top = np.sort(counts)[::-1].cumsum()
    assert (counts >= 8192).sum() >= 2 and f.distinct_columns == int((counts > 0).sum())
    for i in range(3):
        assert abs(f.hub_share[i] - top[f.hub_columns[i] - 1] / counts.sum()) < 1e-12
    tuned, plain = p.new_plan(), p.new_plan(autotune=False)
    assert tuned.column_features()["distinct_columns"] == f.distinct_columns and plain.column_features() is None


@pytest.mark.parametrize("rows,N", [(17, 64), (9000, 96), (20_000, 160), (20_000, 100), (5000, 512)])
def test_session_column_chunks(oracle_mod, rows, N):
    """Host-buffer products that are cut into chunks (also with a narrower last one) and that are not."""
    import ctypes as C
    from mask_b200 import _lib
    L = _lib.lib()
    m = _rows_to_csr([np.array([i % 300, 300 + i % 41], dtype=np.int32) for i in range(rows)], max(rows, 400), 5)
    h, ms = C.c_void_p(), C.c_float()
    _lib.check(L.mask_session_create_csr(m.M, m.K, m.nnz, m.rowptr.ctypes.data, m.colind.ctypes.data, m.values.ctypes.data, 0, C.byref(h)), "create")
    B = np.random.Generator(np.random.PCG64(N)).standard_normal((m.K, N), dtype=np.float32)
    try:
        for _ in range(2):
            out = np.full((m.M, N), np.nan, dtype=np.float32)
            _lib.check(L.mask_session_spmm_host(h, B.ctypes.data, out.ctypes.data, N, C.byref(ms)), "spmm_host")
            assert ms.value > 0
            _assert_close(oracle_mod, m, B, out)
    finally:
        L.mask_session_destroy(h)


# tiles a warp of the fill takes (16, 32, 64: more of them than 48 warps an SM take in shorter runs), and scans by
# one block, by chunks, and by chunks whose sums are scanned in turn (more than 2^22 tiles)
@pytest.mark.parametrize("rows", [3_000, 9_001, 250_000, 520_000, 4_300_000])
def test_pack_tile_counts(oracle_mod, rows):
    from mask_b200 import engine
    K = 4000
    rng = np.random.Generator(np.random.PCG64(rows))
    length = np.where(np.arange(rows) % 4096 == 5, 1500, 8)
    step = np.where(length == 8, rng.integers(1, 400, rows), 2)
    start = (rng.random(rows) * (K - length * step)).astype(np.int64)
    rowptr = np.concatenate([[0], np.cumsum(length)])
    at = np.arange(rowptr[-1]) - np.repeat(rowptr[:-1], length)
    colind = (np.repeat(start, length) + at * np.repeat(step, length)).astype(np.int32)
    m = G.CSR(rows, K, rowptr.astype(np.int32), colind, rng.random(colind.size, dtype=np.float32))
    rp, ci, va = _dev(m)
    _check_metcf(engine.pack_metcf(rp, ci, va, m.M, m.K), oracle_mod.pack_metcf(m.M, m.rowptr, m.colind, m.values))
    if rows > 1_000_000:
        return
    _check_srbcrs(engine.pack_srbcrs(rp, ci, va, m.M, m.K), oracle_mod.pack_srbcrs(m.M, m.rowptr, m.colind, m.values))
    _check_mco(engine.pack_mco(rp, ci, va, m.M, m.K), oracle_mod.pack_mco(m.M, m.rowptr, m.colind, m.values))


@pytest.mark.parametrize("n", [1100, 5000, 9000, 20_000])
def test_pack_columns_up_to_the_end_of_int32(oracle_mod, n):
    """Windows that one block and that a cluster ranks, columns spread over 2^31 - 1 (hundreds to thousands of the
    ranges that a block marks at a time) or all in the last range, which is narrower than a step."""
    from mask_b200 import engine
    K = 2**31 - 1
    rng = np.random.Generator(np.random.PCG64(n))
    rows = []
    for span in (K, 300_000, K):
        for i in range(16):
            c = np.unique(np.concatenate([K - 1 - rng.integers(0, span, n // 40 if i else n - 15 * (n // 40)), [K - 1 - i, K - span + i]]))
            rows.append(c.astype(np.int32))
    m = _rows_to_csr(rows[:-3], K, 7)
    rp, ci, va = _dev(m)
    _check_srbcrs(engine.pack_srbcrs(rp, ci, va, m.M, m.K), oracle_mod.pack_srbcrs(m.M, m.rowptr, m.colind, m.values))
    _check_metcf(engine.pack_metcf(rp, ci, va, m.M, m.K), oracle_mod.pack_metcf(m.M, m.rowptr, m.colind, m.values))


def test_rcm_long_lists_over_many_ranks(oracle_mod):
    """Neighbour lists longer than a warp sorts whose ranks lie in several of the ranges that a block marks at a time,
    some of which hold none of them."""
    from mask_b200 import engine
    n = 2_300_000
    rng = np.random.Generator(np.random.PCG64(4))
    a = np.arange(2, n - n % 2, 2)                 # pairs of neighbours, but for the nodes next to one of the hubs 0 and 1
    near = [np.sort(rng.choice(np.arange(1000, 400_000), 1500, replace=False)), np.sort(rng.choice(np.arange(1_700_000, n - 2), 2500, replace=False))]
    taken = np.zeros(n, bool)
    for x in near:
        taken[x] = True
    a = a[~(taken[a] | taken[a + 1])]
    src = np.concatenate([a, a + 1] + [np.full(len(x), h) for h, x in enumerate(near)] + near)
    dst = np.concatenate([a + 1, a] + near + [np.full(len(x), h) for h, x in enumerate(near)])
    order = np.lexsort((dst, src))
    rowptr = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))]).astype(np.int32)
    m = G.CSR(n, n, rowptr, dst[order].astype(np.int32), np.ones(len(src), np.float32))
    rp, ci, _ = _dev(m)
    got = engine.reorder_rows(rp, ci, n, n, "row_rcm").cpu().numpy()
    assert np.array_equal(got, oracle_mod.reorder_rows("row_rcm", n, n, m.rowptr, m.colind))


def _scattered(small_rows, at, M):
    """rowptr of M rows on the GPU: row at[i] is as long as small_rows[i], the others are empty."""
    import torch
    rowptr = torch.zeros(M + 1, dtype=torch.int32, device="cuda")
    for r, row in zip(at, small_rows):
        rowptr[int(r) + 1:] += len(row)
    return rowptr


@pytest.mark.parametrize("kind", ["row_rcm", "first_col_sort", "jaccard_greedy"])
def test_reorders_past_2_27_rows(oracle_mod, kind):
    """A warp per row is more than 2^32 threads.  All but a few hundred rows are empty, so the order follows from those."""
    import torch
    from mask_b200 import engine
    M = 2**27 + 1000
    rng = np.random.Generator(np.random.PCG64(6))
    at = np.unique(np.concatenate([rng.integers(0, M, 150), np.arange(2**27 - 40, 2**27 + 40), np.arange(M - 30, M)]))
    n = len(at)
    pairs = _both((int(a), int(b)) for a, b in rng.integers(0, n, (2 * n, 2)) if a != b) | _both((i, (i + 1) % n) for i in range(n))
    small = _graph(pairs, n)
    rows = [at[small.colind[small.rowptr[i]:small.rowptr[i + 1]]].astype(np.int32) for i in range(n)]
    rp, ci = _scattered(rows, at, M), torch.from_numpy(np.concatenate(rows)).cuda()
    order = engine.reorder_rows(rp, ci, M, M, kind)
    full = torch.zeros(M, dtype=torch.bool, device="cuda")
    full[torch.from_numpy(at).cuda()] = True
    empty = torch.nonzero(~full).squeeze(1).to(torch.int32)
    if kind == "row_rcm":               # isolated nodes are components of their own and come first
        want = np.concatenate([at[oracle_mod.reorder_rows(kind, n, n, small.rowptr, small.colind)]])
        assert torch.equal(order[:M - n], empty)
        assert np.array_equal(order[M - n:].cpu().numpy(), want)
    else:                               # empty rows come last; the first of them share a bucket of 64 with the others
        more = -n % 64
        ids = np.sort(np.concatenate([at, empty[:more].cpu().numpy()]))
        some = _rows_to_csr([rows[np.searchsorted(at, r)] if r in at else np.zeros(0, np.int32) for r in ids], M, 1)
        want = ids[oracle_mod.reorder_rows(kind, len(ids), M, some.rowptr, some.colind)]
        assert np.array_equal(order[:len(ids)].cpu().numpy(), want)
        assert torch.equal(order[len(ids):], empty[more:])
    va = torch.arange(ci.numel(), dtype=torch.float32, device="cuda")
    rp2, ci2, va2 = engine.permute_rows(rp, ci, va, M, order)
    place = torch.nonzero(full[order.long()]).squeeze(1)
    taken = [int(np.searchsorted(at, r)) for r in order[place].cpu().numpy()]
    assert np.array_equal(ci2.cpu().numpy(), np.concatenate([rows[i] for i in taken]))
    assert np.array_equal(va2.cpu().numpy(), np.concatenate([np.arange(small.rowptr[i], small.rowptr[i + 1], dtype=np.float32) for i in taken]))
    assert torch.equal(rp2[1:] - rp2[:-1], (rp[1:] - rp[:-1])[order.long()])


def test_pack_and_product_rows_up_to_the_end_of_int32(oracle_mod):
    """M = 2^31 - 1: 16 times the number of windows, and the index of the row behind the last window, do not fit int32."""
    import torch
    from mask_b200 import engine
    M, K, N = 2**31 - 1, 3000, 4
    rng = np.random.Generator(np.random.PCG64(8))
    at = np.concatenate([np.arange(3, 20), np.arange(2**30 - 5, 2**30 + 9), [2**31 - 100], np.arange(M - 20, M)])
    rows = [np.sort(rng.choice(K, int(c), replace=False)).astype(np.int32) for c in rng.integers(1, 60, len(at))]
    rows[20] = np.sort(rng.choice(K, 1500, replace=False)).astype(np.int32)   # a window that a block ranks
    windows = np.unique(at // 16)
    by_row = dict(zip(at.tolist(), rows))
    small = _rows_to_csr([by_row.get(int(r), np.zeros(0, np.int32)) for w in windows for r in range(16 * w, min(16 * w + 16, M))], K, 5)
    rp, ci, va = _scattered(rows, at, M), torch.from_numpy(small.colind).cuda(), torch.from_numpy(small.values).cuda()
    p = engine.pack_srbcrs(rp, ci, va, M, K)
    del rp
    want = oracle_mod.pack_srbcrs(small.M, small.rowptr, small.colind, small.values)
    for k in ("val_sidx", "val_block_val"):
        assert np.array_equal(getattr(p, k).cpu().numpy().view(np.int32), want[k].view(np.int32)), k
    tiles = torch.diff(p.val_soff)
    assert np.array_equal(tiles[torch.from_numpy(windows).cuda()].cpu().numpy(), np.diff(want["val_soff"]))
    assert int(p.val_soff[0]) == 0 and int(p.val_soff[-1]) == p.T == int(tiles.sum())
    B = rng.standard_normal((K, N), dtype=np.float32)
    out = engine.spmm(p, torch.from_numpy(B).cuda())
    assert p.plan().status() == 0
    ids = torch.from_numpy(np.concatenate([np.arange(16 * w, min(16 * w + 16, M)) for w in windows])).cuda()
    _assert_close(oracle_mod, small, B, out[ids].cpu().numpy())
    out[ids] = 0
    assert not bool(out.any())


# windows without tiles between others: as many as are looked at in a step, in a step of steps, and one more or less
@pytest.mark.parametrize("gap", [1, 31, 32, 33, 1023, 1024, 1055, 1056, 32_768, 40_000])
def test_pack_runs_of_empty_windows(oracle_mod, gap):
    from mask_b200 import engine
    rng = np.random.Generator(np.random.PCG64(gap))
    K, none = 5000, [np.zeros(0, np.int32)]
    some = lambda n: [np.sort(rng.choice(K, int(c), replace=False)) for c in rng.integers(1, 40, n)]
    rows = none * (16 * gap) + some(37) + none * (16 * gap + 11) + some(900) + none * (16 * gap) + some(16) + none * (16 * gap)
    m = _rows_to_csr(rows, K, 7)
    rp, ci, va = _dev(m)
    _check_srbcrs(engine.pack_srbcrs(rp, ci, va, m.M, m.K), oracle_mod.pack_srbcrs(m.M, m.rowptr, m.colind, m.values))
    _check_metcf(engine.pack_metcf(rp, ci, va, m.M, m.K), oracle_mod.pack_metcf(m.M, m.rowptr, m.colind, m.values))
    _check_mco(engine.pack_mco(rp, ci, va, m.M, m.K), oracle_mod.pack_mco(m.M, m.rowptr, m.colind, m.values))


def test_pack_time_does_not_depend_on_where_the_empty_rows_are():
    """2^21 empty rows in the middle of a matrix cost what they cost at its end.  Walking them window by window took
    one warp 7.8 ms, against 0.1 in all; three times the other placing leaves room for noise."""
    import torch
    from mask_b200 import engine
    rows, empty, K = 32_000, 1 << 21, 8
    colind = torch.arange(8, dtype=torch.int32, device="cuda").repeat(rows)   # one tile a window
    values = torch.rand(8 * rows, device="cuda")
    length = torch.full((rows,), 8, dtype=torch.int64, device="cuda")
    gap = torch.zeros(empty, dtype=torch.int64, device="cuda")
    ms = {}
    for where, parts in (("middle", (length[:16 * 1003], gap, length[16 * 1003:])), ("end", (length, gap))):
        rowptr = torch.zeros(rows + empty + 1, dtype=torch.int32, device="cuda")
        rowptr[1:] = torch.cumsum(torch.cat(parts), 0)
        times = []
        for _ in range(7):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            engine.pack_srbcrs(rowptr, colind, values, rows + empty, K)
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        ms[where] = sorted(times)[3]
    assert ms["middle"] < 3 * ms["end"], ms


def _chain(engine, p, plan, x, y, steps, widths):
    """x -> A x -> A A x ..., alternating between two buffers, nothing waited for."""
    for _ in range(steps):
        (engine.spmm if widths else engine.spmm_any_width)(p, x, out=y, plan=plan)
        x, y = y, x
    return x


# kernels start while the one before them drains: both main kernels, with whole and split windows (fix-up pass), rows that
# are padded first, products that fill the GPU and that do not
@pytest.mark.parametrize("sweep", [0, 2])
@pytest.mark.parametrize("N,gt", [(64, 0), (64, 5), (512, 5), (47, 5)])
@pytest.mark.parametrize("scale", [9, 14])
def test_overlapped_launches_keep_their_order(sweep, N, gt, scale):
    import torch
    from mask_b200 import engine
    m = G.rmat_gcn_normalised(scale=scale, samples_per_node=8, seed=5)
    p = engine.pack_srbcrs(*_dev(m), m.M, m.K)
    whole = N % 4 == 0
    gen = torch.Generator(device="cuda").manual_seed(N)
    first = [torch.randn(m.K, N, generator=gen, device="cuda") for _ in range(3)]
    engine.tune("sweep", sweep)
    try:
        plan = p.new_plan("auto", gt)
        nan = lambda: torch.full((m.M, N), float("nan"), device="cuda")
        want = []
        for f in first:                              # one product at a time
            x, y = f.clone(), nan()
            for _ in range(6):
                torch.cuda.synchronize()
                (engine.spmm if whole else engine.spmm_any_width)(p, x, out=y, plan=plan)
                torch.cuda.synchronize()
                x, y = y, x
            want.append(x.clone())
        # back to back: each product reads what the last one wrote and overwrites what it read
        assert torch.equal(_chain(engine, p, plan, first[0].clone(), nan(), 6, whole), want[0])
        # on three streams at once, with a copy into the operand between the chains
        streams, got = [torch.cuda.Stream() for _ in first], []
        x, y = [nan() for _ in first], [nan() for _ in first]
        torch.cuda.synchronize()
        for turn in range(3):
            for s, f, a, b in zip(streams, first, x, y):
                with torch.cuda.stream(s):
                    a.copy_(f)
                    got.append(_chain(engine, p, plan, a, b, 6, whole))
        torch.cuda.synchronize()
        for g, w in zip(got, want * 3):
            assert torch.equal(g, w)
        # captured, and replayed with other operands
        x, y = nan(), nan()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            last = _chain(engine, p, plan, x, y, 6, whole)
        for f, w in list(zip(first, want)) * 2:
            x.copy_(f)
            graph.replay()
            assert torch.equal(last, w)
    finally:
        engine.tune("sweep", 1)


@pytest.mark.parametrize("name", ["path", "stars", "components", "many_edges"])
@pytest.mark.parametrize("how", ["twice", "some_twice", "unsorted"])
def test_rcm_of_rows_that_are_not_strictly_ascending(oracle_mod, name, how):
    """Symmetric patterns with entries listed more than once, or out of order: the order is that of the pattern."""
    from mask_b200 import engine
    m = GRAPHS[name]()
    rng = np.random.Generator(np.random.PCG64(3))
    rows = [m.colind[m.rowptr[i]:m.rowptr[i + 1]] for i in range(m.M)]
    if how == "unsorted":
        rows = [rng.permutation(r) for r in rows]
    else:
        rows = [np.sort(np.concatenate([r, r if how == "twice" else r[rng.random(len(r)) < 0.1]])) for r in rows]
    again = _rows_to_csr(rows, m.K, 1)
    rp, ci, _ = _dev(again)
    got = engine.reorder_rows(rp, ci, m.M, m.K, "row_rcm").cpu().numpy()
    assert np.array_equal(got, oracle_mod.reorder_rows("row_rcm", m.M, m.K, m.rowptr, m.colind))


@pytest.mark.parametrize("by", [4, 8, 12])
def test_pack_writes_tile_values_at_any_alignment(oracle_mod, by):
    import torch
    from mask_b200 import _lib, engine
    from mask_b200.engine import _analyze, _ptr, _stream
    m = _mixed_matrix()
    rp, ci, va = _dev(m)
    ws, soff, T, nnz = _analyze(rp, ci, m.M, m.K)
    sidx = torch.empty(8 * T, dtype=torch.int32, device="cuda")
    room = torch.full((128 * T + 8,), 7.0, device="cuda")
    val = room[by // 4:by // 4 + 128 * T]
    _lib.check(_lib.lib().mask_srbcrs_fill(_ptr(rp), _ptr(ci), _ptr(va), m.M, nnz, _ptr(ws), _ptr(soff), T, _ptr(sidx), _ptr(val), None, None, None,
                                           _stream()), "mask_srbcrs_fill")
    want = oracle_mod.pack_srbcrs(m.M, m.rowptr, m.colind, m.values)
    assert np.array_equal(val.cpu().numpy().view(np.int32), want["val_block_val"].view(np.int32))
    assert np.array_equal(sidx.cpu().numpy(), want["val_sidx"])
    assert bool((room[:by // 4] == 7).all()) and bool((room[by // 4 + 128 * T:] == 7).all())
