"""Kernels that start before their predecessor has ended read its output while it
may still be written, so they may use no load that is defined for read-only memory:
the source of every load that such a kernel makes of a caller's tensor."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "librett_gb300" / "csrc"


def _code(path):
    """The file without its comments."""
    text = re.sub(r"/\*.*?\*/", "", path.read_text(), flags=re.S)
    return re.sub(r"//[^\n]*", "", text)


def test_no_read_only_loads():
    """Inline assembly never asks for the non-coherent path."""
    for path in sorted(CSRC.iterdir()):
        if path.suffix in (".cu", ".cuh", ".inc", ".h"):
            assert not re.search(r"ld\.(volatile\.)?global[\w.:]*\.nc\b", _code(path)), path.name


def test_ldg_reads_tables_only():
    """__ldg is left for tables and lists that the host finished before the launch."""
    tables = ("stSm", "stOff", "ldOff", "offsetBytes(ldRow", "tiles")
    for path in sorted(CSRC.iterdir()):
        if path.suffix not in (".cu", ".cuh", ".inc", ".h"):
            continue
        for arg in re.findall(r"__ldg\((.*)", _code(path)):
            arg = re.sub(r"reinterpret_cast<[^()]*>\(", "", arg)
            assert arg.startswith(tables), (path.name, arg)


def test_dependent_kernels_wait():
    """Every kernel that releases its successors early also waits."""
    for path in sorted(CSRC.iterdir()):
        if path.suffix not in (".cu", ".cuh"):
            continue
        for body in _code(path).split("__global__")[1:]:
            if "dependencyRelease()" in body:
                assert re.search(r"dependencyWait\(\)|bulkIssue<|groupTileBody<", body), path.name


def test_copies_are_waited_for():
    """mlpWeightGrads: a CTA may have no rows (batches of 896 or fewer), so the wait
    for the copies it starts before its loop over rows stands behind the loop."""
    body = _code(CSRC / "mlp.cu").split("mlpWeightGrads(", 1)[1].split("__global__", 1)[0]
    start = body.index("copyRows(s.W4")
    loop = body.index("for (int b0 = first; b0 < batch; b0 += stride")
    end = body.index("float* partial = ")
    assert start < loop < body.index("cpAsyncWaitAll()") < end
