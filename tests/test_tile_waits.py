"""How the tile kernels end a bounded wait for a bulk copy, read off their source.

A wait that gives up is counted by each thread for itself, so threads of one block can
disagree about it.  A thread that left a tile by its own count would miss the block's later
barriers (and, in the persistent kernels, run a barrier ahead of the others into the next
tile's buffers).  So no tile function returns between its wait and its end, each reports
whether its copy arrived, and the persistent kernels vote on that before the next tile.  What
would happen otherwise is not run on a GPU; this reads the code instead."""
import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "2d-turbulent-navier-stokes_b200", "csrc")
TILES = (("tns_kernels.cu", r"bool stage_tile\("), ("tns_kernels_mx.cu", r"bool stage_mx_tile\("),
         ("tns_visc.cuh", r"bool viscous_tile\("))


def _code(path):
    """The source without comments."""
    with open(path) as f:
        s = f.read()
    return re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", s, flags=re.S))


SOURCES = {os.path.basename(p): _code(p) for p in glob.glob(os.path.join(CSRC, "*.cu*"))}


def _body(code, head):
    """The braces that follow the first match of `head`."""
    at = code.index("{", re.search(head, code).end())
    depth, end = 0, at
    for end in range(at, len(code)):
        depth += {"{": 1, "}": -1}.get(code[end], 0)
        if depth == 0:
            break
    return code[at:end + 1]


def test_no_thread_leaves_a_tile_by_its_own_count():
    assert any("bulk_wait(" in c for c in SOURCES.values())
    for name, code in SOURCES.items():
        assert not re.search(r"(if|while)\s*\(\s*!?\s*bulk_wait\(", code), name
    wait = _body(SOURCES["tns_tile.cuh"], r"bool tile_copy_wait\(")
    assert wait.count("bulk_wait(bar)") == 2 and wait.count("return") == 1 and "__syncthreads();" in wait
    for name, head in TILES:
        body = _body(SOURCES[name], head)
        assert body.count("tile_copy_wait(&S.bar") == 1, name
        after = body[body.index("tile_copy_wait(&S.bar"):]
        # every way out after the wait reports it, and none depends on it
        assert all(r == "return arrived;" for r in re.findall(r"return[^;]*;", re.sub(r"\[&\]\([^)]*\)\s*\{[^}]*\}", "", after))
                   if r != "return;"), name
        assert not re.search(r"if\s*\([^)]*arrived", after), name


def test_persistent_kernels_vote_before_the_next_tile():
    for name, head in (("tns_kernels.cu", r"k_batch_persistent\("), ("tns_kernels_mx.cu", r"k_batch_persistent_mx\(")):
        body = _body(SOURCES[name], head)
        assert body.count("ok = ") == 3 and "if (!__syncthreads_and(ok)) return;" in body, name


def test_a_tile_takes_its_barrier_down_before_the_next_sets_one_up():
    """A loop over tiles puts other data where a tile's barrier was and initialises one there
    again; PTX defines neither while the barrier is live."""
    wait = _body(SOURCES["tns_tile.cuh"], r"bool tile_copy_wait\(")
    assert re.search(r"__syncthreads\(\);\s*if \(arrived && [^)]*\) bulk_barrier_end\(bar\);", wait)
    assert "mbarrier.inval" in _body(SOURCES["tns_tile.cuh"], r"void bulk_barrier_end\(")
    # every barrier a tile function sets up is the one it waits for there
    for name, head in TILES:
        body = _body(SOURCES[name], head)
        assert body.count("bulk_barrier_init(&S.bar)") == 1 == body.count("tile_copy_wait(&S.bar"), name
