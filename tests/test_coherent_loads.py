"""The step's kernels may be launched while their predecessor still runs
(pq_tuning.pdl), so what an earlier kernel of the step writes is not read-only
for their lifetime and must not be read through the read-only path (__ldg):
only the tables that a context uploads once may be.  Read from the sources."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pequod_b200", "csrc")

# Twiddles, split weights, 2 sin(k pi / N), pivots, mean and wall weights, the
# closure vectors of a channel's periodic columns.
TABLES = ("tw", "wsp", "was", "Mb.piv_off", "Mb.piv_len", "Mb.piv_fix", "piv", "pb", "pc",
          "Mb.wwall", "Mb.wmean")


def arguments(text):
    for m in re.finditer(r"__ldg\(", text):
        depth, k = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[k], 0)
            k += 1
        yield text[m.end():k - 1]


def base(arg):
    """The array an argument addresses: &a[i], a + i, (c ? a : b) + i."""
    names = re.findall(r"[A-Za-z_][\w.]*", re.split(r"\[|\+|\)", arg.replace("Mb.periodic ?", ""))[0])
    return names


def test_read_only_loads_are_of_tables():
    seen, wrong = 0, []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        name = os.path.basename(path)
        if name == "pq_dst_mma.cu":  # launched after its predecessor has ended, never beside it
            continue
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for arg in arguments(text):
            seen += 1
            if not base(arg) or any(b not in TABLES for b in base(arg)):
                wrong.append((name, arg))
    assert seen > 0
    assert wrong == []


def test_tensor_core_dst_is_launched_alone():
    text = open(os.path.join(CSRC, "pq_dst_mma.cu")).read()
    assert "launch_step_kernel" not in text and "ProgrammaticStreamSerialization" not in text
