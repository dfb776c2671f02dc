"""What the host side of a call launches, without a GPU (tests/fake_cuda)."""
import ctypes

import pytest

from ncarray_gb300 import _lib
from tests import fake_cuda


def test_short_vectors(built_lib, tmp_path):
    """1-D and 0-d expressions of fewer elements than a 16-byte vector: one launch each, no division by the zero whole
    groups (a process on an x86-64 host dies of one)."""
    code = """
result = []
for dt in (DType.float32, DType.int8, DType.float64, DType.bfloat16):
    for shape in ((), (1,), (2,), (3,), (5,), (15,), (16,), (17,)):
        x = array(shape, dt)
        e = nca.DevExpr.leaf(x) + nca.DevExpr.leaf(x)
        e.evaluate(out=array(shape, e.dtype))
        ls = launches()
        result.append([str(dt), shape, len(ls), ls[0]["grid"], ls[0]["consts"]["NCA_VEC"]])
"""
    for dt, shape, n, grid, _ in fake_cuda.run(code, tmp_path):
        assert n == 1 and grid == [1, 1, 1], (dt, shape)


def test_scatter_shared_memory_limit_never_falls(built_lib, tmp_path):
    """The shared-memory limit of a kernel belongs to the device: a call that lowered it to its own need would fail a
    launch that another thread is about to make with more."""
    code = """
result = []
for dt in (DType.float32, DType.int64):
    n = 1 << 24
    for bytes_ in (200 * 1024, 52 * 1024, 120 * 1024, 48 * 1024 + 8):
        m = bytes_ // nca.dtype.ITEMSIZE[dt]
        dest, idx, src = array((m,), dt), array((n,), DType.int32), array((n,), dt)
        for s in (src, array((2 * n,), dt)[::2]):
            dest.scatter_add(idx, s)
        result += calls()
"""
    calls = fake_cuda.run(code, tmp_path)
    limits = {}
    for c in calls:
        if "smem_limit" in c:
            assert c["smem_limit"] >= limits.get(c["kernel"], 0), c
            limits[c["kernel"]] = c["smem_limit"]
        elif c.get("smem", 0) > 48 * 1024:
            assert c["smem"] <= limits[c["launch"]], c
    assert len(limits) == 2   # both types took private copies above 48 KB


def test_three_step_stencil_only_where_it_pays(built_lib, tmp_path):
    """Flat and narrow grids keep single steps; (steps - 1) // 3 passes elsewhere."""
    code = """
from ncarray_gb300.stencil import Stencil3D, laplacian7, laplacian27
result = []
for points, w in ((7, laplacian7()), (27, laplacian27())):
    for shape in ((1, 2048, 2048), (2, 2048, 2048), (4, 2048, 2048), (1, 300000, 4), (8, 8, 100000), (64, 4096, 8), (1, 8192, 8192),
                  (512, 512, 512), (64, 64, 64), (200, 300, 400), (256, 36, 120)):
        a, b = array(shape, DType.float32), array(shape, DType.float32)
        Stencil3D(w, 0.1).iterate(a, b, 11)
        result.append([points, shape, ["tma3" in c["launch"] for c in launches()]])
"""
    flat = {(1, 2048, 2048), (2, 2048, 2048), (4, 2048, 2048), (1, 300000, 4), (8, 8, 100000), (64, 4096, 8), (1, 8192, 8192)}
    for points, shape, three in fake_cuda.run(code, tmp_path):
        want = [False] * 11 if tuple(shape) in flat else [True] * 3 + [False] * 2
        assert three == want, (points, shape)


def test_three_step_stencil_on_grids_of_one_round(built_lib, tmp_path):
    """Grids whose CTAs all run at once, where a single step's start and march are most of its time: a pass took 0.67 to
    0.95 of three single steps; thin ones, where it takes longer, keep single steps."""
    code = """
from ncarray_gb300.stencil import Stencil3D, laplacian7, laplacian27
result = []
for points, w in ((7, laplacian7()), (27, laplacian27())):
    for shape in ((29, 437, 340), (43, 408, 168), (57, 445, 136), (100, 208, 272), (34, 304, 136), (192, 193, 296), (512, 512, 132),
                  (1, 290, 1452), (2, 1024, 1024)):
        a, b = array(shape, DType.float32), array(shape, DType.float32)
        Stencil3D(w, 0.1).iterate(a, b, 4)
        result.append([points, shape, ["tma3" in c["launch"] for c in launches()]])
"""
    for points, shape, three in fake_cuda.run(code, tmp_path):
        assert three == ([True, False] if shape[0] > 3 else [False] * 4), (points, shape)


def test_weighted_histogram_uses_every_cta(built_lib, tmp_path):
    """2^20 weighted points accumulate on one CTA per resident slot even where the bins outnumber a CTA's records: points
    that crowd into one bin are as many serial adds as a CTA has."""
    code = """
from ncarray_gb300.hist import hist2d_into
fake.fake_resident(1)
n = 1 << 20
x, y, w = (array((n,), DType.float32) for _ in range(3))
result = []
for nb in (8, 128, 1024):
    c, s = array((nb, nb), DType.uint64), array((nb, nb), DType.float32)
    hist2d_into(x, y, c, (0.0, 1.0), (0.0, 1.0), w, s)
    result.append([k["grid"][0] for k in launches() if "accumulate" in k["launch"]])
"""
    assert fake_cuda.run(code, tmp_path) == [[152]] * 3


def test_row_segments_bound_their_registers(built_lib, tmp_path):
    """Groups per thread of odd rows: 8 up to three operands, fewer with more."""
    code = """
result = {}
for n in (2, 3, 4, 6, 12, 24, 48):
    xs = [array((256, 256, 259), DType.float32)[:, :, 1:252] for _ in range(n)]
    e = nca.DevExpr.leaf(xs[0])
    for x in xs[1:]:
        e = e + x
    e.evaluate(out=array((256, 256, 251), DType.float32))
    (c,) = launches()
    result[n] = c["consts"]["NCA_ROWU"]
"""
    got = {int(n): u for n, u in fake_cuda.run(code, tmp_path).items()}
    assert all(max(u, 1) * n <= 24 or u <= 1 for n, u in got.items()), got
    assert got[2] == got[3] == 8 and got[4] == got[6] == 4, got


OUTER = """
def outer(shape, axis, dtype, nops=1, ops=(RedOp.SUM,), stored=False, step=1):
    xs = [array((*shape[:-1], shape[-1] * step), dtype)[..., ::step] for _ in range(nops)]
    e = nca.DevExpr.leaf(xs[0])
    for x in xs[1:]:
        e = e + x
    kept = [n for d, n in enumerate(shape) if d != axis]
    out = array(shape, e.expr_dtype) if stored else None
    from ncarray_gb300.array import _red_out_dtype
    e.evaluate(out=out, reductions=[(op, axis) for op in ops], red_out=[array(kept, _red_out_dtype(op, e.expr_dtype)) for op in ops])
    (c,) = [c for c in launches() if "outer" in c["launch"]]
    return c["consts"]["NCA_K4G"] * c["consts"]["NCA_UNROLL"]   # rows loaded together, 0: one by one


"""


def test_outer_rows_together_only_where_it_pays(built_lib, tmp_path):
    """Rows loaded together: not with more operands than the registers hold, nor with rows that leave the last batch
    nearly empty, nor where fewer resident CTAs cost a second round."""
    code = OUTER + """
F, D = DType.float32, DType.float64
big = (256, 256, 256)
result = {
    "stored": [outer(big, 0, F, n, stored=True) for n in (1, 3, 12, 13, 24, 48)],
    "reduced": [outer((1024, 4096), 0, F, n) for n in (1, 3, 12, 13, 24, 48)],
    "stored64": [outer(big, 0, D, n, stored=True) for n in (1, 6, 7, 24)],
    "rows": [outer((n, 1000000), 0, F) for n in (5, 16, 20, 32, 33, 64, 100)],
    "stored_rows": [outer((n, 100000), 0, F, stored=True) for n in (5, 16, 20, 33)],
    "two": [outer((n, 5000), 0, F, ops=(RedOp.SUM, RedOp.MAX)) for n in (5, 33)],
    "strided": [outer((256, w), 0, F, stored=st, step=2) for w in (1000, 1001) for st in (False, True)],
    "sum64": [outer(s, 0, D, n) for s, n in (((2000, 5000), 1), ((2000, 5000), 2), ((100, 60000), 1), ((33, 1000000), 1))],
}
"""
    got = fake_cuda.run(code, tmp_path)
    # 3 CTAs an SM of the form with the loads together: 456 sets of columns at once
    got["round"] = fake_cuda.run(OUTER + """
fake.fake_resident(3)
result = [outer((1200, 4 * 64 * n), 0, DType.float32) for n in (400, 456, 457, 500)]
""", tmp_path)
    assert got == {"stored": [8, 8, 8, 0, 0, 0], "reduced": [8, 8, 8, 0, 0, 0], "stored64": [2, 2, 0, 0],
                   "rows": [0, 0, 8, 8, 0, 8, 8], "stored_rows": [0, 0, 8, 8], "two": [8, 8], "strided": [0, 0, 8, 8], "sum64": [8, 0, 0, 0],
                   "round": [8, 8, 0, 0]}


def test_odd_vectors_and_rows_of_8_byte_arithmetic(built_lib, tmp_path):
    """Odd 1-D extents keep 16-byte vectors, except float64 and short 8-byte integer arithmetic; float64 rows of three
    operands take no segments."""
    code = """
def flat(n, dtype):
    x, y = array((n,), dtype), array((n,), dtype)
    e = nca.DevExpr.leaf(x) + nca.DevExpr.leaf(y)
    e.evaluate(out=array((n,), e.expr_dtype))
    (c,) = launches()
    return c["consts"]["NCA_VEC"]

def rows(nops, dtype):
    xs = [array((96, 509, 250), dtype)[:, :, 1:250] for _ in range(nops)]
    e = nca.DevExpr.leaf(xs[0])
    for x in xs[1:]:
        e = e + x
    e.evaluate(out=array((96, 509, 249), e.expr_dtype))
    (c,) = launches()
    return c["consts"]["NCA_ROWU"]

F, D, I8 = DType.float32, DType.float64, DType.int8
result = [[flat(n, t) for n in (1003, (1 << 23) + 1, 1 << 23)] for t in (F, D, I8)] + [[rows(n, t) for n in (2, 3)] for t in (F, D)]
"""
    assert fake_cuda.run(code, tmp_path) == [[4, 4, 4], [1, 1, 2], [1, 2, 2], [8, 8], [8, 0]]


REDUCE = """
x = array((4096, 16384), DType.float32)
out = array((16384,), DType.float32)

def launch():
    nca.DevExpr.leaf(x).evaluate(reductions=[(RedOp.SUM, 0)], red_out=[out])
    return [{k: v for k, v in c.items() if k != "aux"} for c in launches()]

"""


def test_tuner_knows_the_untuned_outer_reduction(built_lib, tmp_path):
    """A search includes the form that runs untuned and its stored choice is read back; choices of the former key, made
    without it, are not."""
    plain = fake_cuda.run(REDUCE + "result = launch()", tmp_path / "a")
    # every candidate takes the same (fake) time: the first one, the untuned form, is stored
    found = fake_cuda.run(REDUCE + "tune.set_mode(2)\nls = launch()\nresult = [ls, tune.entries(sys.argv[2])]", tmp_path / "b",
                          args=[tmp_path / "b"])
    assert plain[0] in found[0] and found[0][-1] == plain[0]
    (key, value), = found[1].items()
    assert value == [108, -1, 1]
    assert fake_cuda.run(REDUCE + "result = launch()", tmp_path / "b") == plain
    old = tmp_path / "c"
    old.mkdir()
    (old / "tune.txt").write_text(key.replace("red|k4b|", "red|k4|") + " 8 512 0\n")
    assert fake_cuda.run(REDUCE + "result = launch()", old) == plain
    (old / "tune.txt").write_text(key + " 8 512 0\n")
    assert fake_cuda.run(REDUCE + "result = launch()", old) != plain


BATCH = """
lengths = [1000 + 2000 * k for k in range(160)]
items = (_lib.BatchItem * len(lengths))()
for it, n in zip(items, lengths):
    it.data, it.length, it.dtype = 1 << 40, n, int(DType.float32)

def create():
    h = ctypes.c_void_p()
    _lib.call("nca_batch_create", items, len(lengths), ctypes.byref(h), None)
    return h

def schedule(h):
    c, t, u, n = ctypes.c_int64(), ctypes.c_int32(), ctypes.c_int32(), ctypes.c_int32()
    _lib.call("nca_batch_schedule", h, ctypes.byref(c), ctypes.byref(t), ctypes.byref(u), ctypes.byref(n))
    return [c.value, t.value, u.value, n.value]

"""


def test_batch_tuner_knows_the_untuned_schedule(built_lib, tmp_path):
    """autotune() times the untuned schedule too (the first of equal candidates is kept); schedules stored before the
    chunks were ordered are not read back."""
    plain = fake_cuda.run(BATCH + "result = schedule(create())", tmp_path / "a")
    assert plain[0] % 16384 == 0 and 128 * 1024 <= plain[0] <= 512 * 1024 and plain[0] not in (256 << 10, 512 << 10)
    code = """
h = create()
_lib.call("nca_batch_autotune", h, ctypes.c_void_p(1 << 41), None)
result = [schedule(h), open(sys.argv[2] + "/batch_tune_ws.txt").read()]
"""
    got, text = fake_cuda.run(BATCH + code, tmp_path / "b", args=[tmp_path / "b"])
    assert got == plain
    key, *value = text.split()
    assert fake_cuda.run(BATCH + "result = schedule(create())", tmp_path / "b") == plain
    old = tmp_path / "c"
    old.mkdir()
    (old / "batch_tune_ws.txt").write_text(f"{key.replace('batch2_', 'batch_')} {1 << 20} 256 8192 2\n")
    assert fake_cuda.run(BATCH + "result = schedule(create())", old) == plain
    (old / "batch_tune_ws.txt").write_text(f"{key} {1 << 20} 256 8192 2\n")
    assert fake_cuda.run(BATCH + "result = schedule(create())", old) != plain


def test_staged_launches_take_counters_that_are_still_zero(built_lib, tmp_path):
    """Every launch counts in words that none before it has used since they were zeroed; no compare and swap, no memset of
    its own. The block's memset comes when the next launch would not fit."""
    code = """
t = array((64, 256, 128, 8), DType.int32).transpose(3, 1, 2, 0)
e = nca.DevExpr.leaf(t) * np.int32(3)
kept = [t.shape[d] for d in (0, 1, 3)]
out, red = array(t.shape, e.expr_dtype), array(kept, e.expr_dtype)
result = []
for _ in range(120):
    e.evaluate(out, [(RedOp.MAX, 2)], [red])
    result += [["zero", c["at"], c["memset"]] if "memset" in c else ["count", c["aux"], c["consts"]["NCA_KIND"]]
               for c in calls() if "launch" in c or "memset" in c]
"""
    events = fake_cuda.run(code, tmp_path)
    first = events[0][1]
    units = events[1][1] - first   # bytes that a launch takes
    used, zeroed = set(), 0
    for what, at, n in events:
        if what == "zero":
            assert (at, n) == (first, 4 * 16384)
            used.clear()
            zeroed += 1
        else:
            assert n == 7 and first <= at and at + units <= first + 4 * 16384 and at not in used
            used.add(at)
    assert units >= 4 * 256 and zeroed == 120 * units // (4 * 16384) - (120 * units % (4 * 16384) == 0)


@pytest.mark.parametrize("name", ["nca_jit_selftest", "nca_jit_selftest_forms"])
def test_selftests_report_what_they_compile(built_lib, tmp_path, name):
    code = f"""
n = ctypes.c_int32()
_lib.call("{name}", b"sm_103a", ctypes.byref(n))
result = [n.value, sum("compile" in c for c in calls())]
"""
    reported, compiled = fake_cuda.run(code, tmp_path)
    assert reported == compiled > 0


def test_nvrtc_compiles_every_form(built_lib):
    n = ctypes.c_int32(0)
    _lib.call("nca_jit_selftest_forms", b"sm_103a", ctypes.byref(n))
    assert n.value == 10


def test_general_scatter_privatises_on_four_ctas(built_lib, tmp_path):
    """Strided and converted sources keep private copies to 48 KB and four CTAs an SM; the 1-D form goes to 200 KB."""
    code = """
result = []
for dt in (DType.float32, DType.float64):
    for shape, m in (((4000, 4000), 500), ((4000, 4000), 6000), ((4000, 4000), 50000), ((100, 100), 10)):
        dest, idx, src = array((m,), dt), array(shape, DType.int32), array(shape, dt)
        row = []
        for view in (lambda a: a[:, 1:], lambda a: a.reshape(shape[0] * shape[1])):
            dest.scatter_add(view(idx), view(src))
            (c,) = launches()
            row.append(c["smem"])
        result.append(row)
"""
    got = fake_cuda.run(code, tmp_path)
    assert got == [[2000, 2000], [24000, 24000], [0, 200000], [0, 40], [4000, 4000], [48000, 48000], [0, 0], [0, 80]]
