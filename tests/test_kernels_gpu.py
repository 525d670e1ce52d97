"""Kernel-level parity: every CUDA entry point of the C ABI against the CPU oracle
on the same seeded inputs.  Integer and index results must be identical; fp16
tensor-core results are within 1e-2 relative (stated per test)."""
import json
import os

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from lidar_ai_solution_b200 import scenes  # noqa: E402
from oracle import oracle as orc  # noqa: E402
from tests.helpers import int8_problem, kaiming  # noqa: E402

pytestmark = pytest.mark.gpu

STAGES = [((3, 3, 3), (2, 2, 2), (1, 1, 1)), ((3, 3, 3), (2, 2, 2), (1, 1, 1)),
          ((3, 3, 3), (2, 2, 2), (0, 1, 1)), ((3, 1, 1), (2, 1, 1), (0, 0, 0))]


def _ops():
    from lidar_ai_solution_b200 import ops
    return ops


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _status_ok(status):
    s = status.cpu().numpy()
    assert s[0] == 0, "device status %s" % s


def test_calls_go_to_the_current_stream(monkeypatch):
    """By torch's own shortcut to its handle, and without it."""
    ops = _ops()
    side = torch.cuda.Stream()
    for shortcut in (ops._raw_stream, None):
        monkeypatch.setattr(ops, "_raw_stream", shortcut)
        assert ops._stream() == torch.cuda.current_stream().cuda_stream != side.cuda_stream
        with torch.cuda.stream(side):
            assert ops._stream() == side.cuda_stream


# ------------------------------------------------------------------ rulebooks
@pytest.mark.parametrize("n,grid,seed", [(20000, (41, 180, 180), 0), (20000, (41, 180, 180), 3),
                                         (120000, (41, 1440, 1440), 1), (1, (41, 180, 180), 0),
                                         (129, (5, 7, 9), 2)])
def test_subm_map_bit_exact(n, grid, seed):
    ops = _ops()
    coords = scenes.make_coords(n, grid, seed)
    ref, pairs = orc.subm_map(coords, grid)
    dc, n_ptr, st = _dev(coords), ops.device_count(n), ops.new_status()
    table = ops.hash_build(dc, n_ptr, grid, status=st)
    m = ops.subm_map(dc, n_ptr, grid, table, status=st)
    torch.cuda.synchronize()
    _status_ok(st)
    got = m.cpu().numpy()
    assert np.array_equal(got, ref)
    assert int((got >= 0).sum()) == pairs


def test_subm_map_capacity_larger_than_rows():
    """Buffers sized for a bound, row count on the device (the DDS calling pattern)."""
    ops = _ops()
    grid, n, cap = (41, 180, 180), 5000, 8192
    coords = scenes.make_coords(n, grid, 5)
    padded = np.full((cap, 4), 7, np.int32)
    padded[:n] = coords
    ref, _ = orc.subm_map(coords, grid, cap=cap)
    dc, n_ptr, st = _dev(padded), ops.device_count(n), ops.new_status()
    table = ops.hash_build(dc, n_ptr, grid, status=st)
    m = torch.full((27, cap), -1, dtype=torch.int32, device="cuda")
    from lidar_ai_solution_b200 import cabi
    cabi.check(cabi.lib().spconvb_subm_map(dc.data_ptr(), n_ptr.data_ptr(), cap, 2048,
                                           cabi.i3(grid), 1, cabi.i3((3, 3, 3)),
                                           cabi.i3((1, 1, 1)), table.data_ptr(), table.numel(),
                                           m.data_ptr(), st.data_ptr(),
                                           torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    _status_ok(st)
    assert np.array_equal(m.cpu().numpy(), ref)


@pytest.mark.parametrize("x_step", [0, 8])
@pytest.mark.parametrize("n,slots", [(4, 8), (8, 16), (128, 256), (4000, 8192), (14000, 32768)])
def test_subm_map_of_rows_that_share_a_place_in_their_runs(n, slots, x_step):
    """Cells in one x plane, or every eighth: all have the same position in their aligned runs of eight
    along x.  They are found like any others, in the smallest table the rows may have."""
    ops = _ops()
    from lidar_ai_solution_b200 import cabi
    grid = (41, 360, 360)
    rng = np.random.default_rng(n)
    cells = rng.choice(41 * 360 * (45 if x_step else 1), n, replace=False)
    coords = np.zeros((n, 4), np.int32)
    coords[:, 1], coords[:, 2] = cells % 41, cells // 41 % 360
    coords[:, 3] = 5 + x_step * (cells // (41 * 360)) if x_step else 203
    ref, _ = orc.subm_map(coords, grid)
    dc, n_ptr, st = _dev(coords), ops.device_count(n), ops.new_status()
    table = torch.empty(slots, dtype=torch.int64, device="cuda")
    cabi.check(cabi.lib().spconvb_hash_build(dc.data_ptr(), n_ptr.data_ptr(), n, 0, cabi.i3(grid), 1,
                                             table.data_ptr(), slots, 0, st.data_ptr(), ops._stream()))
    m = ops.subm_map(dc, n_ptr, grid, table, status=st)
    torch.cuda.synchronize()
    _status_ok(st)
    assert np.array_equal(m.cpu().numpy(), ref)


def test_hash_reports_duplicates_and_range():
    ops = _ops()
    grid = (8, 8, 8)
    coords = np.array([[0, 1, 1, 1], [0, 1, 1, 1], [0, 9, 0, 0]], np.int32)
    st = ops.new_status()
    ops.hash_build(_dev(coords), ops.device_count(3), grid, status=st)
    torch.cuda.synchronize()
    from lidar_ai_solution_b200 import cabi
    bits = int(st.cpu().numpy()[0])
    assert bits & cabi.ST_DUPLICATE and bits & cabi.ST_COORD_RANGE


@pytest.mark.parametrize("n", [6, 160000])
def test_subm_centre_tap_is_the_row_itself(n):
    """Also for rows the table does not hold: repeated cells (it keeps one of them) and cells outside
    the grid; with a thread per plane of a row and with a thread per row."""
    ops = _ops()
    grid = (8, 64, 640)
    coords = scenes.make_coords(min(n, 100000), grid, 3)
    coords = np.concatenate([coords, coords, coords[:1]])[:n]
    coords[n // 2] = (0, 9, 0, 0)
    coords[n // 3] = (0, 0, -1, 0)
    dc, n_ptr = _dev(coords), ops.device_count(n)
    m = ops.subm_map(dc, n_ptr, grid, ops.hash_build(dc, n_ptr, grid))
    assert np.array_equal(m[13].cpu().numpy(), np.arange(n))


def _chain(coords, grid):
    """Stage 0 looks neighbours up in the hash table of the caller's rows; later stages rank
    them in the bitmap the strided rulebook left behind (no hash table)."""
    ops = _ops()
    dc, n_ptr, st = _dev(coords), ops.device_count(len(coords)), ops.new_status()
    table = ops.hash_build(dc, n_ptr, grid, status=st)
    ws = None
    out = []
    for k, s, p in STAGES:
        if ws is None:
            m = ops.subm_map(dc, n_ptr, grid, table, status=st)
        else:
            m = ops.subm_map_ranked(dc, n_ptr, grid, ws, status=st)
            by_hash = ops.subm_map(dc, n_ptr, grid, table, status=st)
            assert torch.equal(m[:, : int(n_ptr.item())], by_hash[:, : int(n_ptr.item())])
        in_ws = ws
        oc, n_out, dm, otab, og, ws = ops.down_map(dc, n_ptr, grid, None, k, s, p, status=st,
                                                   return_ws=True)
        if in_ws is not None:
            # rows made by a strided rulebook: the output-side lookup by rank gives the same
            # coordinates, count and map as the input-side scatter
            oc2, n2, dm2, _, _ = ops.down_map(dc, n_ptr, grid, None, k, s, p, status=st,
                                              in_ws=in_ws)
            kk = int(n_out.item())
            assert int(n2.item()) == kk and torch.equal(oc2[:kk], oc[:kk])
            assert torch.equal(dm2[:, :kk], dm[:, :kk])
        torch.cuda.synchronize()
        _status_ok(st)
        out.append((dc, n_ptr, list(grid), m, oc, n_out, dm, og))
        dc, n_ptr, table, grid = oc, n_out, otab, og
    return out


def test_stage_chain_matches_oracle_and_fixture_counts(golden_dir):
    """The reference's 79 745-voxel CenterPoint frame through the backbone's four
    resolutions: maps and output coordinates identical to the oracle, counts equal
    to the committed golden counts."""
    z = np.load(os.path.join(golden_dir, "fixture_coords.npz"))
    counts = json.load(open(os.path.join(golden_dir, "fixture_counts.json")))
    for name, key in (("centerpoint", "centerpoint_zyx"), ("bevfusion", "bevfusion_zyx")):
        zyx = z[key].astype(np.int32)
        coords = np.concatenate([np.zeros((len(zyx), 1), np.int32), zyx], 1)
        grid = [41, 1440, 1440]
        c_ref = coords
        for stage, (dc, n_ptr, g, m, oc, n_out, dm, og) in enumerate(_chain(coords, grid)):
            n = int(n_ptr.item())
            ref_m, pairs = orc.subm_map(c_ref, g)
            assert np.array_equal(m.cpu().numpy()[:, :n], ref_m)
            k, s, p = STAGES[stage]
            roc, rdm, dpairs, rog, rn = orc.down_map(c_ref, g, k, s, p, cap=oc.shape[0])
            assert int(n_out.item()) == rn and og == rog
            assert np.array_equal(oc.cpu().numpy()[:rn], roc)
            assert np.array_equal(dm.cpu().numpy()[:, :rn], rdm[:, :rn])
            gold = counts[name][stage]
            assert (n, pairs, rn, dpairs) == (gold["n"], gold["subm_pairs"], gold["down_n"],
                                              gold["down_pairs"])
            c_ref = roc


@pytest.mark.parametrize("k,s,p,d", [
    ((3, 3, 3), (2, 2, 2), (1, 1, 1), (1, 1, 1)),   # every strided layer of the backbones
    ((3, 3, 3), (3, 3, 3), (0, 0, 0), (1, 1, 1)),   # stride that is not a power of two
    ((5, 3, 1), (2, 1, 3), (2, 0, 1), (1, 1, 1)),   # mixed extents, stride 1 on an axis
    ((2, 2, 2), (2, 2, 2), (0, 0, 0), (1, 1, 1)),   # even kernel
    ((1, 1, 1), (2, 2, 2), (0, 0, 0), (1, 1, 1)),   # pure subsampling
    ((3, 3, 7), (1, 2, 1), (1, 1, 3), (1, 1, 1)),   # runs of up to 7 adjacent output cells
    ((3, 3, 3), (2, 2, 2), (2, 1, 2), (2, 1, 2)),   # dilated: the tap-pruning path
])
def test_down_map_geometries_match_the_oracle(k, s, p, d):
    """Output coordinates, their order, the count and the whole map of a strided rulebook for
    kernel / stride / padding / dilation combinations beyond the backbones', from the caller's
    rows (input-side scatter) and again from rulebook-made rows (output-side lookup)."""
    ops = _ops()
    grid = (9, 70, 83)
    coords = scenes.make_coords(6000, grid, 5)
    st = ops.new_status()
    dc = _dev(coords)
    oc, n_out, dm, _, og, ws = ops.down_map(dc, ops.device_count(len(coords)), grid, None, k, s, p,
                                            dilation=d, status=st, want_table=False,
                                            return_ws=True)
    roc, rdm, pairs, rog, rn = orc.down_map(coords, grid, k, s, p, d, cap=oc.shape[0])
    _status_ok(st)
    assert int(n_out.item()) == rn and list(og) == list(rog) and pairs > 0
    assert np.array_equal(oc.cpu().numpy()[:rn], roc)
    assert np.array_equal(dm.cpu().numpy()[:, :rn], rdm[:, :rn])
    # second level: the rows just made are the input, looked up by rank from the output side
    k2, s2, p2 = (3, 3, 3), (2, 2, 2), (1, 1, 1)
    oc2, n2, dm2, _, og2 = ops.down_map(oc, n_out, og, None, k2, s2, p2, status=st,
                                        want_table=False, in_ws=ws)
    roc2, rdm2, _, rog2, rn2 = orc.down_map(roc, rog, k2, s2, p2, cap=oc2.shape[0])
    _status_ok(st)
    assert int(n2.item()) == rn2 and list(og2) == list(rog2)
    assert np.array_equal(oc2.cpu().numpy()[:rn2], roc2)
    assert np.array_equal(dm2.cpu().numpy()[:, :rn2], rdm2[:, :rn2])
    # and the geometry under test on rulebook-made rows (the outputs' bitmap then comes from
    # the inputs' bitmap): first a 3x3x3 stride-1 rulebook over the caller's rows, whose
    # outputs are ranked, then the geometry on those
    fo, fn, _, _, fg, fws = ops.down_map(dc, ops.device_count(len(coords)), grid, None, (3, 3, 3),
                                         (1, 1, 1), (1, 1, 1), status=st, want_table=False,
                                         return_ws=True)
    rfo, _, _, rfg, rfn = orc.down_map(coords, grid, (3, 3, 3), (1, 1, 1), (1, 1, 1),
                                       cap=fo.shape[0])
    assert int(fn.item()) == rfn
    oc3, n3, dm3, _, og3 = ops.down_map(fo, fn, fg, None, k, s, p, dilation=d, status=st,
                                        want_table=False, in_ws=fws)
    roc3, rdm3, _, rog3, rn3 = orc.down_map(rfo, rfg, k, s, p, d, cap=oc3.shape[0])
    _status_ok(st)
    assert int(n3.item()) == rn3 and list(og3) == list(rog3)
    assert np.array_equal(oc3.cpu().numpy()[:rn3], roc3)
    assert np.array_equal(dm3.cpu().numpy()[:, :rn3], rdm3[:, :rn3])


@pytest.mark.parametrize("grid,n", [
    ((1, 1, 5), 3),             # one bitmap word, partly outside the grid
    ((4, 32, 32), 3900),        # one scan block, nearly every cell set
    ((4, 32, 33), 4224),        # a scan block and 4 words, every cell set
    ((16, 64, 64), 30000),      # exactly one group of 16 scan blocks
    ((16, 64, 65), 66000),      # a group and a bit
    ((32, 64, 64), 40000),      # exactly two groups
    ((32, 64, 65), 130000),     # two groups and a bit
    ((33, 257, 311), 2000),     # many blocks, most of them empty
])
def test_strided_rows_at_the_edges_of_scan_blocks(grid, n):
    """Output rows, order, count and map where the scan's blocks (128 words of 32 cells) and groups
    of blocks (16) begin and end; a 1x1x1 kernel of stride 1, so the outputs are the inputs."""
    ops = _ops()
    cells = np.sort(np.random.default_rng(n).permutation(int(np.prod(grid)))[:n])
    coords = np.zeros((n, 4), np.int32)
    coords[:, 1:] = np.stack(np.unravel_index(cells, grid), 1)
    order = np.random.default_rng(n + 1).permutation(n)
    st = ops.new_status()
    one = (1, 1, 1)
    oc, n_out, m, _, og, ws = ops.down_map(_dev(coords[order]), ops.device_count(n), grid, None, one,
                                           one, (0, 0, 0), status=st, want_table=False,
                                           return_ws=True)
    _status_ok(st)
    assert int(n_out.item()) == n and list(og) == list(grid)
    assert np.array_equal(oc.cpu().numpy()[:n], coords)
    assert np.array_equal(m.cpu().numpy()[0, :n], np.argsort(order))
    sub = ops.subm_map_ranked(oc, n_out, grid, ws, status=st)
    ref, _ = orc.subm_map(coords, grid)
    _status_ok(st)
    assert np.array_equal(sub.cpu().numpy()[:, :n], ref)


@pytest.mark.parametrize("n", [1, 43, 128, 75776, 75777, 151552, 151553])
def test_maps_where_threads_go_from_planes_to_rows(n):
    """3x3x3 maps by hash and by rank, from one row up and on both sides of the row counts up to
    which a thread takes one plane of a row (227 328 threads: a third of them by rank, two by hash);
    then the strided map of those rows, gathered by rank."""
    ops = _ops()
    grid = (33, 96, 128)
    cells = np.sort(np.random.default_rng(n).permutation(int(np.prod(grid)))[:n])
    coords = np.zeros((n, 4), np.int32)
    coords[:, 1:] = np.stack(np.unravel_index(cells, grid), 1)
    shuffled = coords[np.random.default_rng(n + 1).permutation(n)]
    dc, n_ptr, st = _dev(shuffled), ops.device_count(n), ops.new_status()
    by_hash = ops.subm_map(dc, n_ptr, grid, ops.hash_build(dc, n_ptr, grid, status=st), status=st)
    _status_ok(st)
    assert np.array_equal(by_hash.cpu().numpy()[:, :n], orc.subm_map(shuffled, grid)[0])
    one = (1, 1, 1)
    oc, n_out, _, _, _, ws = ops.down_map(dc, n_ptr, grid, None, one, one, (0, 0, 0), status=st,
                                          want_table=False, return_ws=True)
    by_rank = ops.subm_map_ranked(oc, n_out, grid, ws, status=st)
    _status_ok(st)
    assert np.array_equal(by_rank.cpu().numpy()[:, :n], orc.subm_map(coords, grid)[0])
    args = ((3, 3, 3), (2, 2, 2), one)
    roc, rdm, _, _, rn = orc.down_map(coords, grid, *args)
    goc, gn, gdm = ops.down_map(oc, n_out, grid, None, *args, cap_out=max(rn, 1), status=st,
                                want_table=False, in_ws=ws)[:3]
    _status_ok(st)
    assert int(gn.item()) == rn and np.array_equal(goc.cpu().numpy()[:rn], roc[:rn])
    assert np.array_equal(gdm.cpu().numpy()[:, :rn], rdm[:, :rn])


@pytest.mark.parametrize("s", [(3, 3, 3), (2, 2, 2), (5, 1, 3), (1, 1, 1)])
@pytest.mark.parametrize("k,p", [((3, 3, 3), (1, 0, 1)), ((2, 1, 4), (0, 0, 2)), ((1, 1, 1), (0, 0, 0))])
def test_strided_rows_outside_the_grid(k, s, p):
    """Nothing checks a coordinate before the strided rulebook: rows outside the grid, up to the ends of
    an int, reach the cells that tap = c + pad - cell * stride in [0, K) gives, and no others."""
    ops = _ops()
    grid = (7, 12, 15)
    rng = np.random.default_rng(3)
    coords = np.zeros((3000, 4), np.int32)
    coords[:, 1:] = rng.integers(-6, 20, (3000, 3))
    ends = np.iinfo(np.int32)
    coords[:12, 1:][np.arange(12), np.arange(12) % 3] = [ends.min, ends.max, ends.min + 1, ends.max - 1] * 3
    coords = coords[np.sort(np.unique(coords, axis=0, return_index=True)[1])]  # each cell once
    og = ops.out_grid(grid, k, s, p)
    reached = {}
    for row, c in enumerate(coords[:, 1:].astype(np.int64)):
        axes = [[(o, c[a] + p[a] - o * s[a]) for o in range(og[a]) if 0 <= c[a] + p[a] - o * s[a] < k[a]]
                for a in range(3)]
        for o0, k0 in axes[0]:
            for o1, k1 in axes[1]:
                for o2, k2 in axes[2]:
                    reached.setdefault((o0, o1, o2), {})[(k0 * k[1] + k1) * k[2] + k2] = row
    cells = sorted(reached)
    want = np.full((int(np.prod(k)), len(cells)), -1, np.int32)
    for o, cell in enumerate(cells):
        for tap, row in reached[cell].items():
            want[tap, o] = row
    st = ops.new_status()
    oc, n_out, m, _, _ = ops.down_map(_dev(coords), ops.device_count(len(coords)), grid, None, k, s, p,
                                      cap_out=len(cells) + 50, status=st, want_table=False)
    _status_ok(st)
    assert int(n_out.item()) == len(cells) > 0
    assert np.array_equal(oc.cpu().numpy()[:len(cells), 1:], np.array(cells))
    assert np.array_equal(m.cpu().numpy()[:, :len(cells)], want)


def _carved_down_map(coords, grid, args, shift, cap_out, flags=0, zero="all", runs=1):
    """spconvb_down_map on a workspace `shift` bytes into a buffer; what lies behind it stays as it is.
    With a `zero` other than "none" the bitmap, or all of the workspace, is cleared before each run."""
    ops = _ops()
    from lidar_ai_solution_b200 import cabi
    lib, n = cabi.lib(), len(coords)
    og = ops.out_grid(grid, *args)
    need = lib.spconvb_down_workspace_bytes(cabi.i3(og), 1)
    words = (int(np.prod(og)) + 31) // 32
    kvol = int(np.prod(args[0]))
    buf = torch.full((shift + need + 64,), 0xA5, dtype=torch.uint8, device="cuda")
    dc, n_ptr, st = _dev(coords), ops.device_count(n), ops.new_status()
    for _ in range(runs):
        if zero != "none":
            buf[shift:shift + (need if zero == "all" else 4 * words)].zero_()
        oc = torch.zeros((cap_out, 4), dtype=torch.int32, device="cuda")
        n_out = torch.zeros(1, dtype=torch.int32, device="cuda")
        m = torch.full((kvol, cap_out), -1, dtype=torch.int32, device="cuda")
        cabi.check(lib.spconvb_down_map(
            dc.data_ptr(), n_ptr.data_ptr(), n, 0, cabi.i3(grid), 1, *[cabi.i3(a) for a in args],
            cabi.i3((1, 1, 1)), None, 0, buf.data_ptr() + shift, oc.data_ptr(), n_out.data_ptr(),
            cap_out, m.data_ptr(), None, 0, flags, st.data_ptr(),
            torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()
    _status_ok(st)
    assert int((buf[:shift] != 0xA5).sum()) == 0 and int((buf[shift + need:] != 0xA5).sum()) == 0
    k = int(n_out.item())
    return oc.cpu().numpy()[:k], m.cpu().numpy()[:, :k]


@pytest.mark.parametrize("shift", [0, 4, 8, 12])
@pytest.mark.parametrize("grid", [(9, 70, 83), (41, 180, 180)])
def test_down_map_workspace_may_start_at_any_word(grid, shift):
    """A workspace carved out of a larger buffer at any multiple of 4 bytes gives the oracle's rows and
    map, and nothing beside it is written."""
    coords = scenes.make_coords(6000, grid, 5)
    args = ((3, 3, 3), (2, 2, 2), (1, 1, 1))
    roc, rdm, _, _, rn = orc.down_map(coords, grid, *args)
    oc, m = _carved_down_map(coords, grid, args, shift, rn)
    assert np.array_equal(oc, roc) and np.array_equal(m, rdm[:, :rn])


@pytest.mark.parametrize("zero,flags", [("all", 1), ("bitmap", 1), ("none", 0)])
def test_down_map_on_a_used_workspace(zero, flags):
    """What a call must find zero: with PREZEROED the bitmap, without it nothing; the rest of the
    workspace, the scan's state among it, may be as another use or the call before has left it."""
    grid = (41, 180, 180)
    coords = scenes.make_coords(6000, grid, 6)
    args = ((3, 3, 3), (2, 2, 2), (1, 1, 1))
    roc, rdm, _, _, rn = orc.down_map(coords, grid, *args)
    oc, m = _carved_down_map(coords, grid, args, 0, rn, flags, zero, runs=2)
    assert np.array_equal(oc, roc) and np.array_equal(m, rdm[:, :rn])


def test_down_map_overflow_sets_status():
    ops = _ops()
    from lidar_ai_solution_b200 import cabi
    grid = (9, 33, 33)
    coords = scenes.make_coords(600, grid, 4)
    dc, n_ptr, st = _dev(coords), ops.device_count(600), ops.new_status()
    table = ops.hash_build(dc, n_ptr, grid, status=st)
    oc, n_out, dm, _, _ = ops.down_map(dc, n_ptr, grid, table, (3, 3, 3), (2, 2, 2), (1, 1, 1),
                                       cap_out=64, status=st)
    torch.cuda.synchronize()
    assert int(n_out.item()) == 64
    assert int(st.cpu().numpy()[0]) & cabi.ST_OVERFLOW
    roc, rdm, _, _, rn = orc.down_map(coords, grid, (3, 3, 3), (2, 2, 2), (1, 1, 1), cap=64)
    assert rn > 64 and np.array_equal(oc.cpu().numpy(), roc)
    assert np.array_equal(dm.cpu().numpy(), rdm)


# --------------------------------------------------------------- convolutions
def _int8_layer(n, c_in, c_out, seed, simt, out_kind, grid=(41, 180, 180), hint=False):
    ops = _ops()
    pb = int8_problem(n, c_in, c_out, grid, seed)
    m_ref, _ = orc.subm_map(pb["coords"], grid)
    y32 = orc.conv_i8(pb["xq"], m_ref, n, pb["wq"], pb["scale"], pb["bias"], orc.ACT_RELU,
                      orc.KIND_F32)
    inv_out = np.float32(127.0) / np.float32(max(float(np.abs(y32).max()), 1e-6))
    ref = orc.conv_i8(pb["xq"], m_ref, n, pb["wq"], pb["scale"], pb["bias"], orc.ACT_RELU,
                      out_kind, float(inv_out))
    n_ptr, st = ops.device_count(n), ops.new_status()
    wts = ops.ConvWeights(pb["wq"], ops.I8, pb["scale"], pb["bias"])
    out = ops.conv_forward(_dev(pb["xq"]), _dev(m_ref), n_ptr, wts, act=ops.ACT_RELU,
                           out_kind=out_kind, inv_out_scale=float(inv_out), force_simt=simt,
                           status=st, n_in_ptr=n_ptr if hint else None)
    torch.cuda.synchronize()
    _status_ok(st)
    return out.cpu().numpy(), ref


@pytest.mark.parametrize("c", [16, 32, 64, 128])
@pytest.mark.parametrize("simt", [False, True])
def test_conv_int8_bit_exact(c, simt):
    """int8 x int8 -> int32 is exact, the epilogue is defined operation by operation,
    so the requantised int8 output must be identical (tolerance 0 LSB)."""
    got, ref = _int8_layer(3000 if simt else 10000, c, c, seed=c, simt=simt, out_kind=orc.KIND_I8)
    assert got.dtype == np.int8 and np.array_equal(got, ref)


@pytest.mark.parametrize("c", [16, 32, 64, 128])
@pytest.mark.parametrize("n", [120000, 200000])
def test_conv_int8_bit_exact_at_benchmark_sizes(c, n):
    """The layer sweep of the benchmark configurations: SubM 3x3x3, Cin = Cout = c, on the
    41x1440x1440 grid with 120 k and 200 k voxels (many tiles per CTA, balanced tile heights):
    identical to the oracle, with the input's row count given as a hint."""
    got, ref = _int8_layer(n, c, c, seed=c + n, simt=False, out_kind=orc.KIND_I8,
                           grid=(41, 1440, 1440), hint=True)
    assert got.dtype == np.int8 and np.array_equal(got, ref)


@pytest.mark.parametrize("cin,cout", [(16, 32), (32, 64), (64, 128), (128, 16)])
def test_conv_int8_mixed_channels_fp16_out(cin, cout):
    got, ref = _int8_layer(4097, cin, cout, seed=cin + cout, simt=False, out_kind=orc.KIND_F16)
    assert np.array_equal(got.view(np.uint16), ref.view(np.uint16))


@pytest.mark.parametrize("n", [0, 1, 127, 128, 129, 257])
def test_conv_int8_ragged_row_counts(n):
    if n == 0:
        ops = _ops()
        wts = ops.ConvWeights(np.zeros((16, 27, 16), np.int8), ops.I8, np.ones(16, np.float32),
                              np.zeros(16, np.float32))
        st = ops.new_status()
        out = ops.conv_forward(torch.zeros((1, 16), dtype=torch.int8, device="cuda"),
                               torch.full((27, 1), -1, dtype=torch.int32, device="cuda"),
                               ops.device_count(0), wts, out_kind=ops.I8, status=st)
        torch.cuda.synchronize()
        _status_ok(st)
        assert out.shape == (1, 16)
        return
    got, ref = _int8_layer(n, 32, 32, seed=n, simt=False, out_kind=orc.KIND_I8, grid=(5, 9, 11))
    assert np.array_equal(got, ref)


@pytest.mark.parametrize("n", [1, 3, 255, 256, 257, 511, 513])
@pytest.mark.parametrize("out_kind", ["i8", "f16"])
def test_conv_int8_ragged_row_counts_wide_outputs(n, out_kind):
    """The epilogue takes 16 rows at a time, an element a lane: partial tiles, partial groups,
    single-row inputs, with 2 copies of the weights on the accumulator lanes."""
    kind = orc.KIND_I8 if out_kind == "i8" else orc.KIND_F16
    got, ref = _int8_layer(n, 32, 64, seed=100 + n, simt=False, out_kind=kind, grid=(7, 11, 13))
    assert np.array_equal(got.view(np.uint8), ref.view(np.uint8))


def _f16_problem(n, cin, cout, seed, grid=(41, 180, 180), kvol=27):
    rng = np.random.default_rng(seed)
    coords = scenes.make_coords(n, grid, seed)
    x = rng.standard_normal((n, cin)).astype(np.float16)
    w = kaiming(rng, cout, kvol, cin).astype(np.float16)
    bias = (rng.standard_normal(cout) * 0.1).astype(np.float32)
    return coords, x, w, bias


@pytest.mark.parametrize("n", [1, 31, 148 * 32, 148 * 32 + 1, 148 * 224 - 5, 148 * 256, 148 * 256 + 1,
                               148 * 512 + 33])
@pytest.mark.parametrize("cin,cout,kvol", [(16, 16, 27), (64, 64, 27), (128, 128, 27), (32, 128, 1),
                                           (128, 32, 3)])
def test_conv_int8_tile_heights_and_shared_tail(n, cin, cout, kvol):
    """Row counts around the edges of the tile height the kernel picks (rows dealt to 148 CTAs in
    multiples of 32, at most 256), for layers with fewer and with more K chunks than the stage
    ring (in the latter the producers help to drain the last tile), with a residual; against the
    CUDA-core kernel, bit for bit."""
    ops = _ops()
    rng = np.random.default_rng(n + cin)
    nin = max(n // 2, 1)
    m = _dev(np.where(rng.random((kvol, n)) < 0.5, rng.integers(0, nin, (kvol, n)), -1).astype(np.int32))
    x = _dev(rng.integers(-128, 128, (nin, cin)).astype(np.int8))
    res = _dev(rng.integers(-128, 128, (n, cout)).astype(np.int8))
    wts = ops.ConvWeights(rng.integers(-127, 128, (cout, kvol, cin)).astype(np.int8), ops.I8,
                          np.full(cout, 2e-4, np.float32), rng.standard_normal(cout))
    n_ptr, st = ops.device_count(n), ops.new_status()
    out = [ops.conv_forward(x, m, n_ptr, wts, out_kind=ops.I8, inv_out_scale=9.0, res=res,
                            res_scale=0.1, mid_kind=ops.I8, mid_inv_scale=8.0, mid_scale=0.125,
                            res_relu=True, force_simt=simt, status=st) for simt in (False, True)]
    torch.cuda.synchronize()
    _status_ok(st)
    assert torch.equal(out[0], out[1])


@pytest.mark.parametrize("n", [148 * 32 * h - 5 for h in range(1, 9)] + [148 * 64 * h - 5 for h in range(5, 8)])
@pytest.mark.parametrize("cin,cout", [(16, 16), (64, 32)])
def test_conv_int8_every_tile_height(n, cin, cout):
    """Every height a tile can have, as a CTA's only tile and (from 160 rows on) with a second one: each
    height has barriers of its own.  One layer keeps its weights in shared memory, the other streams them."""
    ops = _ops()
    rng = np.random.default_rng(n + cin)
    m = torch.randint(-n, n, (27, n), dtype=torch.int32, device="cuda").clamp_(min=-1)
    x = _dev(rng.integers(-128, 128, (n, cin)).astype(np.int8))
    wts = ops.ConvWeights(rng.integers(-127, 128, (cout, 27, cin)).astype(np.int8), ops.I8,
                          np.full(cout, 2e-4, np.float32), rng.standard_normal(cout))
    n_ptr, st = ops.device_count(n), ops.new_status()
    out = [ops.conv_forward(x, m, n_ptr, wts, out_kind=ops.I8, inv_out_scale=9.0, force_simt=simt,
                            status=st) for simt in (False, True)]
    torch.cuda.synchronize()
    _status_ok(st)
    assert torch.equal(out[0], out[1])


@pytest.mark.parametrize("n", [1, 33, 148 * 32, 148 * 96 + 1, 148 * 224 - 5, 148 * 256 + 1])
@pytest.mark.parametrize("cin,cout,kvol", [(8, 16, 27), (16, 16, 27), (64, 64, 27), (128, 128, 27),
                                           (128, 32, 3), (32, 128, 1)])
def test_conv_fp16_tile_heights_and_shared_tail(n, cin, cout, kvol):
    """The same row counts in fp16, up to the 256-byte rows and 54 chunks a tile of the widest layer,
    against the CUDA-core kernel.  Operands are small whole numbers: every sum stays below 2^24, so fp32
    holds it whatever the order, and the two kernels agree bit for bit."""
    ops = _ops()
    rng = np.random.default_rng(n + cin)
    nin = max(n // 2, 1)
    m = _dev(np.where(rng.random((kvol, n)) < 0.5, rng.integers(0, nin, (kvol, n)), -1).astype(np.int32))
    x = _dev(rng.integers(-4, 5, (nin, cin)).astype(np.float16))
    res = _dev(rng.integers(-40, 41, (n, cout)).astype(np.float16))
    wts = ops.ConvWeights(rng.integers(-3, 4, (cout, kvol, cin)).astype(np.float16), ops.F16, None,
                          rng.integers(-9, 10, cout).astype(np.float32))
    n_ptr, st = ops.device_count(n), ops.new_status()
    out = [ops.conv_forward(x, m, n_ptr, wts, out_kind=ops.F16, res=res, mid_kind=ops.F16,
                            res_relu=True, force_simt=simt, status=st) for simt in (False, True)]
    torch.cuda.synchronize()
    _status_ok(st)
    assert bool(out[0].any()) and torch.equal(out[0], out[1])


@pytest.mark.parametrize("c", [16, 32, 64, 128])
def test_conv_fp16_tensor_core(c):
    """fp16 operands, fp32 accumulation in a different order than the oracle:
    tolerance 1e-2 relative to the layer's output magnitude."""
    ops = _ops()
    grid, n = (41, 180, 180), 8000
    coords, x, w, bias = _f16_problem(n, c, c, seed=c + 1)
    m_ref, _ = orc.subm_map(coords, grid)
    ref = orc.conv_f16(x, m_ref, n, w, bias, orc.ACT_RELU, orc.KIND_F16).astype(np.float32)
    wts = ops.ConvWeights(w, ops.F16, None, bias)
    st = ops.new_status()
    out = ops.conv_forward(_dev(x), _dev(m_ref), ops.device_count(n), wts, act=ops.ACT_RELU,
                           out_kind=ops.F16, status=st)
    torch.cuda.synchronize()
    _status_ok(st)
    got = out.cpu().numpy().astype(np.float32)
    tol = 1e-2 * max(float(np.abs(ref).max()), 1e-6)
    assert float(np.abs(got - ref).max()) <= tol


def test_conv_fp16_cuda_core_bit_exact_and_first_layer_padding():
    """Cin = 5 padded to 8 (the backbone's first layer) on the tensor-core kernel vs the
    CUDA-core kernel on the unpadded data; the CUDA-core kernel equals the oracle bit for bit."""
    ops = _ops()
    grid, n = (41, 180, 180), 6000
    coords, x, w, bias = _f16_problem(n, 5, 16, seed=11)
    m_ref, _ = orc.subm_map(coords, grid)
    ref = orc.conv_f16(x, m_ref, n, w, bias, orc.ACT_RELU, orc.KIND_F16)
    n_ptr, md = ops.device_count(n), _dev(m_ref)
    simt = ops.conv_forward(_dev(x), md, n_ptr, ops.ConvWeights(w, ops.F16, None, bias),
                            act=ops.ACT_RELU, out_kind=ops.F16, force_simt=True)
    assert np.array_equal(simt.cpu().numpy().view(np.uint16), ref.view(np.uint16))
    wp = np.zeros((16, 27, 8), np.float16)
    wp[:, :, :5] = w
    xp = ops.convert(_dev(x), ops.F16, 8, 1.0, n_ptr)
    st = ops.new_status()
    tc = ops.conv_forward(xp, md, n_ptr, ops.ConvWeights(wp, ops.F16, None, bias),
                          act=ops.ACT_RELU, out_kind=ops.F16, status=st)
    torch.cuda.synchronize()
    _status_ok(st)
    r32 = ref.astype(np.float32)
    assert float(np.abs(tc.cpu().numpy().astype(np.float32) - r32).max()) <= 1e-2 * np.abs(r32).max()


@pytest.mark.parametrize("c,n", [(16, 5000), (32, 5001), (64, 5000), (64, 4999), (128, 2050)])
@pytest.mark.parametrize("res_kind", ["i8", "f16"])
def test_conv_int8_fused_residual_all_widths(c, n, res_kind):
    """Fused conv + Add&ReLU == oracle conv (stored int8) followed by oracle add, for every
    output width (8, 4, 2 or 1 copies of the weights on the accumulator lanes), int8 and
    fp16 residual operands, row counts that leave partial tiles."""
    ops = _ops()
    grid = (41, 180, 180)
    pb = int8_problem(n, c, c, grid, seed=40 + c)
    m_ref, _ = orc.subm_map(pb["coords"], grid)
    rng = np.random.default_rng(6)
    if res_kind == "i8":
        res, res_scale = rng.integers(-128, 128, (n, c)).astype(np.int8), 0.031
    else:
        res, res_scale = (rng.standard_normal((n, c)) * 2).astype(np.float16), 1.0
    mid_dr, out_dr = 3.0, 4.5
    mid = orc.conv_i8(pb["xq"], m_ref, n, pb["wq"], pb["scale"], pb["bias"], orc.ACT_NONE,
                      orc.KIND_I8, float(np.float32(127.0) / np.float32(mid_dr)))
    ref = orc.add(mid, float(np.float32(mid_dr) / np.float32(127.0)), res, res_scale, True,
                  orc.KIND_I8, float(np.float32(127.0) / np.float32(out_dr)))
    wts = ops.ConvWeights(pb["wq"], ops.I8, pb["scale"], pb["bias"])
    st = ops.new_status()
    out = ops.conv_forward(_dev(pb["xq"]), _dev(m_ref), ops.device_count(n), wts,
                           act=ops.ACT_NONE, out_kind=ops.I8,
                           inv_out_scale=float(np.float32(127.0) / np.float32(out_dr)),
                           res=_dev(res), res_scale=res_scale, mid_kind=ops.I8,
                           mid_inv_scale=float(np.float32(127.0) / np.float32(mid_dr)),
                           mid_scale=float(np.float32(mid_dr) / np.float32(127.0)),
                           res_relu=True, status=st)
    torch.cuda.synchronize()
    _status_ok(st)
    assert np.array_equal(out.cpu().numpy(), ref)


@pytest.mark.parametrize("simt", [False, True])
def test_conv_int8_fused_residual_equals_conv_then_add(simt):
    """Fused conv + Add&ReLU epilogue == oracle conv (stored int8) followed by oracle add."""
    ops = _ops()
    grid, n, c = (41, 180, 180), 5000, 64
    pb = int8_problem(n, c, c, grid, seed=21)
    m_ref, _ = orc.subm_map(pb["coords"], grid)
    rng = np.random.default_rng(5)
    res = rng.integers(-128, 128, (n, c)).astype(np.int8)
    res_scale, mid_dr, out_dr = 0.031, 3.0, 4.5
    mid = orc.conv_i8(pb["xq"], m_ref, n, pb["wq"], pb["scale"], pb["bias"], orc.ACT_NONE,
                      orc.KIND_I8, float(np.float32(127.0) / np.float32(mid_dr)))
    ref = orc.add(mid, float(np.float32(mid_dr) / np.float32(127.0)), res, res_scale, True,
                  orc.KIND_I8, float(np.float32(127.0) / np.float32(out_dr)))
    wts = ops.ConvWeights(pb["wq"], ops.I8, pb["scale"], pb["bias"])
    st = ops.new_status()
    out = ops.conv_forward(_dev(pb["xq"]), _dev(m_ref), ops.device_count(n), wts,
                           act=ops.ACT_NONE, out_kind=ops.I8,
                           inv_out_scale=float(np.float32(127.0) / np.float32(out_dr)),
                           res=_dev(res), res_scale=res_scale, mid_kind=ops.I8,
                           mid_inv_scale=float(np.float32(127.0) / np.float32(mid_dr)),
                           mid_scale=float(np.float32(mid_dr) / np.float32(127.0)),
                           res_relu=True, force_simt=simt, status=st)
    torch.cuda.synchronize()
    _status_ok(st)
    assert np.array_equal(out.cpu().numpy(), ref)


def test_strided_conv_int8_through_down_map():
    ops = _ops()
    grid, n = (41, 180, 180), 20000
    pb = int8_problem(n, 16, 32, grid, seed=8)
    roc, rdm, _, og, rn = orc.down_map(pb["coords"], grid, (3, 3, 3), (2, 2, 2), (1, 1, 1))
    ref = orc.conv_i8(pb["xq"], rdm, rn, pb["wq"], pb["scale"], pb["bias"], orc.ACT_RELU,
                      orc.KIND_I8, 20.0)
    dc, n_ptr, st = _dev(pb["coords"]), ops.device_count(n), ops.new_status()
    table = ops.hash_build(dc, n_ptr, grid, status=st)
    oc, n_out, dm, _, _ = ops.down_map(dc, n_ptr, grid, table, (3, 3, 3), (2, 2, 2), (1, 1, 1),
                                       status=st)
    wts = ops.ConvWeights(pb["wq"], ops.I8, pb["scale"], pb["bias"])
    out = ops.conv_forward(_dev(pb["xq"]), dm, n_out, wts, act=ops.ACT_RELU, out_kind=ops.I8,
                           inv_out_scale=20.0, status=st)
    torch.cuda.synchronize()
    _status_ok(st)
    assert int(n_out.item()) == rn
    assert np.array_equal(out.cpu().numpy()[:rn], ref)


# ---------------------------------------------------------------- elementwise
@pytest.mark.parametrize("ak,bk,ok", [(1, 1, 1), (0, 0, 1), (0, 0, 0), (1, 0, 0)])
@pytest.mark.parametrize("ch", [16, 24])
def test_add_relu(ak, bk, ok, ch):
    ops = _ops()
    rng = np.random.default_rng(ak * 4 + bk * 2 + ok)
    n = 3001

    def mk(kind):
        return (rng.integers(-128, 128, (n, ch)).astype(np.int8) if kind
                else rng.standard_normal((n, ch)).astype(np.float16))
    a, b = mk(ak), mk(bk)
    ref = orc.add(a, 0.05, b, 0.021, True, ok, 9.3)
    out = ops.add(_dev(a), 0.05, _dev(b), 0.021, ops.device_count(n), True, ok, 9.3)
    assert np.array_equal(out.cpu().numpy().view(np.uint8), ref.view(np.uint8))


def test_relu_and_convert():
    ops = _ops()
    rng = np.random.default_rng(0)
    n = 1000
    x8 = rng.integers(-128, 128, (n, 16)).astype(np.int8)
    xh = rng.standard_normal((n, 16)).astype(np.float16)
    n_ptr = ops.device_count(n)
    assert np.array_equal(ops.relu(_dev(x8), n_ptr).cpu().numpy(), orc.relu(x8))
    assert np.array_equal(ops.relu(_dev(xh), n_ptr).cpu().numpy().view(np.uint16),
                          orc.relu(xh).view(np.uint16))
    q = ops.convert(_dev(xh), ops.I8, 16, float(np.float32(127.0) / np.float32(3.0)), n_ptr)
    assert np.array_equal(q.cpu().numpy(), orc.quantize_f16(xh, 3.0))


@pytest.mark.parametrize("perm", [None, (0, 2, 1)])
@pytest.mark.parametrize("kind", [0, 1])
def test_scatter_dense(perm, kind):
    ops = _ops()
    grid, n, ch = (2, 180, 180), 7000, 128
    coords = scenes.make_coords(n, grid, 2)
    rng = np.random.default_rng(1)
    feat = (rng.integers(-128, 128, (n, ch)).astype(np.int8) if kind
            else rng.standard_normal((n, ch)).astype(np.float16))
    ref = orc.scatter_dense(feat, coords, grid, 1, 0.02, perm)
    out = ops.scatter_dense(_dev(feat), _dev(coords), ops.device_count(n), grid, 1, 0.02, perm)
    assert np.array_equal(out.cpu().numpy().view(np.uint16), ref.view(np.uint16))


@pytest.mark.parametrize("perm", [None, (2, 0, 1)])
@pytest.mark.parametrize("in_kind,dynamic_range", [(0, 0.0), (0, 2.5), (1, 0.0), (1, 2.54), (1, 3.0)])
@pytest.mark.parametrize("layout,ch", [("NCHW", 128), ("NCHW32", 128), ("NCHW32", 24), ("NHWzC", 128),
                                       ("NHWzC", 24)])
def test_scatter_dense_layouts(layout, ch, in_kind, dynamic_range, perm):
    """Dense outputs in the engine's three layouts, fp16 or int8 (input_dynamic_range > 0):
    bit-exact against the restatement, padding channels and empty cells zero.  The int8 rows
    carry the scale 0.02 = 2.54 / 127, so the range 2.54 is the byte-copy case and 3.0 the
    rescaling one."""
    ops = _ops()
    grid, n = (2, 90, 100), 5000
    coords = scenes.make_coords(n, grid, 2)
    rng = np.random.default_rng(1)
    feat = (rng.integers(-128, 128, (n, ch)).astype(np.int8) if in_kind
            else rng.standard_normal((n, ch)).astype(np.float16))
    in_scale = float(np.float32(2.54) / np.float32(127.0)) if in_kind else 1.0
    if dynamic_range > 0:
        if in_kind and dynamic_range == 2.54:
            q = feat
        elif in_kind:
            inv = np.float32(127.0) / np.float32(dynamic_range)
            q = np.clip(np.rint((feat.astype(np.float32) * np.float32(in_scale)) * inv),
                        -128, 127).astype(np.int8)
        else:
            q = orc.quantize_f16(feat, dynamic_range)
        ref = orc.scatter_dense_i8(q, coords, grid, 1, perm)
    else:
        ref = orc.scatter_dense(feat, coords, grid, 1, in_scale, perm)
    ref = orc.dense_layout(ref, layout, ch)
    out = ops.scatter_dense_layout(_dev(feat), _dev(coords), ops.device_count(n), grid, layout,
                                   dynamic_range, 1, in_scale, perm).cpu().numpy()
    assert out.shape == ref.shape and out.dtype == ref.dtype
    assert np.array_equal(out.view(np.uint8), ref.view(np.uint8))


# ------------------------------------------------------------------ voxelizer
@pytest.mark.parametrize("kind", ["f32", "f16"])
def test_voxelizer_matches_sequential_reference(kind, golden_dir):
    ops = _ops()
    if kind == "f32":
        pts = scenes.make_points(120000, seed=3)
    else:
        pts = np.load(os.path.join(golden_dir, "sweep_points.npz"))["points"]
    prange, vs = scenes.CENTERPOINT_RANGE, scenes.CENTERPOINT_VOXEL
    gxyz = (1440, 1440, 40)
    rf, rc, rn = orc.voxelize(pts, prange, vs, gxyz, 160000, 10, 0)
    params = ops.voxel_params(prange, vs, gxyz, 5, 0 if kind == "f32" else 1, 10, 160000, 0)
    st = ops.new_status()
    feat, idx, n_ptr = ops.voxelize(_dev(pts), params, status=st)
    torch.cuda.synchronize()
    _status_ok(st)
    n = int(n_ptr.item())
    assert n == rn
    assert np.array_equal(idx.cpu().numpy()[:n], rc)
    assert np.array_equal(feat.cpu().numpy()[:n].view(np.uint16), rf.view(np.uint16))


def test_voxelizer_max_voxels_clips():
    ops = _ops()
    from lidar_ai_solution_b200 import cabi
    pts = scenes.make_points(20000, seed=9)
    prange, vs, gxyz = scenes.CENTERPOINT_RANGE, scenes.CENTERPOINT_VOXEL, (1440, 1440, 40)
    rf, rc, rn = orc.voxelize(pts, prange, vs, gxyz, 1000, 10, 1)
    params = ops.voxel_params(prange, vs, gxyz, 5, 0, 10, 1000, 1)
    st = ops.new_status()
    feat, idx, n_ptr = ops.voxelize(_dev(pts), params, status=st)
    torch.cuda.synchronize()
    assert rn > 1000 and int(n_ptr.item()) == 1000
    assert int(st.cpu().numpy()[0]) & cabi.ST_OVERFLOW
    assert np.array_equal(idx.cpu().numpy(), rc)
    assert np.array_equal(feat.cpu().numpy().view(np.uint16), rf.view(np.uint16))


def test_inverse_map_is_the_strided_map_with_rows_swapped():
    """spconvb_inverse_map: map[k][i] = o exactly for the pairs (k, i, o) of the strided
    rulebook (oracle down_map), -1 elsewhere."""
    ops = _ops()
    grid, n = (21, 180, 180), 15000
    coords = scenes.make_coords(n, grid, 31)
    ks, st_, pd = (3, 3, 3), (2, 2, 2), (1, 1, 1)
    roc, rdm, _, og, rn = orc.down_map(coords, grid, ks, st_, pd)
    ref = np.full((27, n), -1, np.int32)
    for k in range(27):
        o = np.nonzero(rdm[k, :rn] >= 0)[0]
        ref[k, rdm[k, o]] = o
    dc, n_ptr, st = _dev(coords), ops.device_count(n), ops.new_status()
    oc, n_out, dm, _, _, ws = ops.down_map(dc, n_ptr, grid, None, ks, st_, pd, status=st,
                                           want_table=False, return_ws=True)
    inv = ops.inverse_map(dc, n_ptr, grid, ws, oc.shape[0], ks, st_, pd, status=st)
    torch.cuda.synchronize()
    _status_ok(st)
    assert int(n_out.item()) == rn
    assert np.array_equal(inv.cpu().numpy(), ref)
    # asymmetric geometry: kernel (3,1,1), stride (2,1,1), no padding
    ks, st_, pd = (3, 1, 1), (2, 1, 1), (0, 0, 0)
    roc, rdm, _, og, rn = orc.down_map(coords, grid, ks, st_, pd)
    ref = np.full((3, n), -1, np.int32)
    for k in range(3):
        o = np.nonzero(rdm[k, :rn] >= 0)[0]
        ref[k, rdm[k, o]] = o
    oc, n_out, dm, _, _, ws = ops.down_map(dc, n_ptr, grid, None, ks, st_, pd, status=st,
                                           want_table=False, return_ws=True)
    inv = ops.inverse_map(dc, n_ptr, grid, ws, oc.shape[0], ks, st_, pd, status=st)
    torch.cuda.synchronize()
    assert np.array_equal(inv.cpu().numpy(), ref)


def test_conv_bounded_wait_runs_out_and_the_context_survives():
    """Failure detection without a GPU fault: with `wait_test` the producers of the
    tensor-core kernel never signal a stage, so the MMA role's wait on it must run out
    (250 ms), raise the CTA-wide abort flag, let every role leave its loop, free TMEM and
    return with SPCONVB_ST_TIMEOUT in the status block.  The next launch on the same
    context is then bit-exact again."""
    ops = _ops()
    from lidar_ai_solution_b200 import cabi
    grid, n, c = (41, 180, 180), 2000, 32
    pb = int8_problem(n, c, c, grid, seed=77)
    m_ref, _ = orc.subm_map(pb["coords"], grid)
    ref = orc.conv_i8(pb["xq"], m_ref, n, pb["wq"], pb["scale"], pb["bias"], orc.ACT_RELU,
                      orc.KIND_I8, 9.0)
    wts = ops.ConvWeights(pb["wq"], ops.I8, pb["scale"], pb["bias"])
    x, m, n_ptr = _dev(pb["xq"]), _dev(m_ref), ops.device_count(n)
    st = ops.new_status()
    ops.conv_forward(x, m, n_ptr, wts, act=ops.ACT_RELU, out_kind=ops.I8, inv_out_scale=9.0,
                     status=st, wait_test=1)
    torch.cuda.synchronize()
    assert int(st.cpu().numpy()[0]) & cabi.ST_TIMEOUT
    st.zero_()
    out = ops.conv_forward(x, m, n_ptr, wts, act=ops.ACT_RELU, out_kind=ops.I8,
                           inv_out_scale=9.0, status=st)
    torch.cuda.synchronize()
    _status_ok(st)
    assert np.array_equal(out.cpu().numpy(), ref)


def _shape_sweep_cases():
    rng = np.random.default_rng(2024)
    chans = [16, 32, 64, 128]
    cases = []
    for i in range(28):
        cin, cout = int(rng.choice(chans)), int(rng.choice(chans))
        n = int(rng.choice([1, 31, 33, 255, 257, 1000, 4736, 4737, 9473, 20000, 37889]))
        kind = ["subm", "down", "k311"][i % 3]
        cases.append((cin, cout, n, kind, i % 2 == 0, 100 + i))
    return cases


@pytest.mark.parametrize("cin,cout,n,kind,i8_out,seed", _shape_sweep_cases())
def test_conv_int8_shape_sweep_bit_exact(cin, cout, n, kind, i8_out, seed):
    """Channel pairs select how many copies of the weights sit on the accumulator lanes; row counts
    select the tile height (32..256), and with it the depth of the rings, and leave partial tiles; the three rulebook kinds give 27 or 3 taps.  Everything int8, so the
    tensor-core kernel must match the oracle bit for bit."""
    ops = _ops()
    grid = (41, 180, 180)
    kvol = 3 if kind == "k311" else 27
    pb = int8_problem(n, cin, cout, grid, seed=seed, kvol=kvol)
    if kind == "subm":
        m_ref, _ = orc.subm_map(pb["coords"], grid)
        n_out = n
    elif kind == "down":
        _, m_ref, _, _, n_out = orc.down_map(pb["coords"], grid, (3, 3, 3), (2, 2, 2), (1, 1, 1))
    else:
        _, m_ref, _, _, n_out = orc.down_map(pb["coords"], grid, (3, 1, 1), (2, 1, 1), (0, 0, 0))
    okind = orc.KIND_I8 if i8_out else orc.KIND_F16
    inv = 11.0 if i8_out else 1.0
    ref = orc.conv_i8(pb["xq"], m_ref, n_out, pb["wq"], pb["scale"], pb["bias"], orc.ACT_RELU,
                      okind, inv)
    wts = ops.ConvWeights(pb["wq"], ops.I8, pb["scale"], pb["bias"])
    assert wts.packed is not None
    st = ops.new_status()
    md = _dev(np.ascontiguousarray(m_ref))
    out = ops.conv_forward(_dev(pb["xq"]), md, ops.device_count(n_out), wts, act=ops.ACT_RELU,
                           out_kind=ops.I8 if i8_out else ops.F16, inv_out_scale=inv, status=st)
    torch.cuda.synchronize()
    _status_ok(st)
    assert np.array_equal(out.cpu().numpy()[:n_out].view(np.uint8), ref[:n_out].view(np.uint8))


@pytest.mark.parametrize("n", [1, 31, 511, 512, 513, 5000])
@pytest.mark.parametrize("max_pts", [1, 2, 10, 16])
def test_voxelizer_crowded_voxels_and_cleared_tail(n, max_pts):
    """Few voxels with many points (every kept-slot cascade full), point counts around the scan
    blocks, and the rows after the last voxel zero in buffers that were not."""
    ops = _ops()
    pts = np.random.default_rng(n).uniform(0, 3, (n, 4)).astype(np.float32)
    params = ops.voxel_params((0, 0, 0, 3, 3, 3), (1, 1, 1), (3, 3, 3), 4, 0, max_pts, 40, 0)
    st = ops.new_status()
    torch.full((40 * 4 * 4 * 8,), 77, dtype=torch.int32, device="cuda")  # dirt for the allocator
    feat, idx, n_ptr = ops.voxelize(_dev(pts), params, status=st)
    _status_ok(st)
    ref_f, ref_i, _ = orc.voxelize(pts, (0, 0, 0, 3, 3, 3), (1, 1, 1), (3, 3, 3), 40, max_pts)
    k = int(n_ptr.item())
    assert k == len(ref_f)
    assert np.array_equal(idx[:k].cpu().numpy(), ref_i)
    assert np.array_equal(feat[:k].cpu().numpy().view(np.uint16), ref_f.view(np.uint16))
    assert int(feat[k:].abs().sum().item()) == 0 and int(idx[k:].abs().sum().item()) == 0


def test_voxelizer_sums_start_at_zero():
    """The mean of a voxel is 0 + x0 + x1 + ... in fp32: a negative zero comes out positive, whether
    it is its voxel's only point or not."""
    ops = _ops()
    pts = np.full((3, 5), -0.0, np.float32)
    pts[:, :3] = [[0.5, 0.5, 0.5], [1.5, 0.5, 0.5], [1.5, 0.5, 0.5]]
    box = ((0, 0, 0, 3, 3, 3), (1, 1, 1), (3, 3, 3))
    feat, _, n_ptr = ops.voxelize(_dev(pts), ops.voxel_params(*box, 5, 0, 10, 40, 0))
    ref, _, n = orc.voxelize(pts, *box, 40, 10)
    assert int(n_ptr.item()) == n == 2
    assert np.array_equal(feat[:n].cpu().numpy().view(np.uint16), ref.view(np.uint16))
    assert not np.signbit(ref).any()


@pytest.mark.parametrize("shift", [0, 4, 8, 12])
def test_voxelizer_workspace_may_start_at_any_word(shift):
    """A workspace carved out of a larger buffer at any multiple of 4 bytes gives the same voxels, and
    nothing beside it is written."""
    ops = _ops()
    from lidar_ai_solution_b200 import cabi
    lib, n = cabi.lib(), 3000
    pts = np.random.default_rng(shift).uniform(0, 20, (n, 5)).astype(np.float32)
    box = ((0, 0, 0, 20, 20, 20), (1, 1, 1), (20, 20, 20))
    params = ops.voxel_params(*box, 5, 0, 4, 4000, 0)
    need = lib.spconvb_voxelize_workspace_bytes(cabi.C.byref(params), n)
    buf = torch.full((shift + need + 64,), 0xA5, dtype=torch.uint8, device="cuda")
    feat = torch.empty((4000, 5), dtype=torch.float16, device="cuda")
    idx = torch.empty((4000, 4), dtype=torch.int32, device="cuda")
    n_ptr, st, d = ops.device_count(0), ops.new_status(), _dev(pts)
    cabi.check(lib.spconvb_voxelize(cabi.C.byref(params), d.data_ptr(), n, buf.data_ptr() + shift,
                                    feat.data_ptr(), idx.data_ptr(), n_ptr.data_ptr(), st.data_ptr(),
                                    torch.cuda.current_stream().cuda_stream))
    _status_ok(st)
    ref_f, ref_i, k = orc.voxelize(pts, *box, 4000, 4)
    assert int(n_ptr.item()) == k
    assert np.array_equal(idx[:k].cpu().numpy(), ref_i)
    assert np.array_equal(feat[:k].cpu().numpy().view(np.uint16), ref_f.view(np.uint16))
    assert int((buf[:shift] != 0xA5).sum()) == 0 and int((buf[shift + need:] != 0xA5).sum()) == 0
