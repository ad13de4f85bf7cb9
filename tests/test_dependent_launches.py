"""Kernels launched while their predecessor still runs must not read its output by read-only
loads (`const __restrict__` parameters or __ldg): these are defined only for data that nobody
writes while the kernel lives, and may move above the wait.  Plan tables, written at set-up
only, may be read that way.  Checked on the sources."""
import glob
import os
import re

from conftest import ROOT

CSRC = os.path.join(ROOT, "pytomography_gb300", "csrc")
PLAN_TABLES = {"alist", "items", "ioff"}


def _sources():
    return {os.path.basename(p): open(p).read()
            for p in glob.glob(os.path.join(CSRC, "spect_*.cu*"))}


def test_dependent_kernels_take_no_read_only_data():
    src = _sources()
    text = "\n".join(src.values())
    names = set()
    for m in re.finditer(r"launch_dependent\(([^;]*?)\bgrid\b|launch_dependent\(([^;]*?),", text):
        names |= set(re.findall(r"\bk_\w+", m.group(1) or m.group(2)))
    assert {"k_reduce", "k_fwd_strip", "k_fwd_ysum", "k_b1_strip", "k_b2_gather4", "k_b2_nopsf4",
            "k_b2_adjoint", "k_fwd_nopsf", "k_b1_nopsf"} <= names, names
    for n in names:
        m = re.search(r"__global__[^;{]*?\b%s\(([^)]*)\)\s*{" % n, text)
        assert m, n
        for par in m.group(1).split(","):
            if "__restrict__" in par and "const" in par:
                assert par.split()[-1].lstrip("*") in PLAN_TABLES, (n, par.strip())
        body = text[m.end():text.index("\n}\n", m.end())]
        assert "grid_wait()" in body or n in ("k_fwd_strip", "k_fwd_ysum", "k_b1_strip"), n


def test_shared_sampling_code_loads_coherently():
    """The helpers the dependent kernels sample with: __ldg only on plan tables."""
    src = _sources()
    kern = src["spect_kernels.cuh"]
    assert "__ldg(" not in kern[kern.index("float sample("):kern.index("bool plane_rows(")]
    strip = src["spect_strip.cu"]
    for m in re.finditer(r"__ldg\([^;]*;", strip):
        assert re.match(r"__ldg\(reinterpret_cast<const float4 \*>\(Ap\b", m.group(0)), m.group(0)
    fwd = src["spect_fwd.cu"]
    for m in re.finditer(r"__ldg\([^;]*;", fwd):
        assert re.match(r"__ldg\((reinterpret_cast<const float4 \*>\()?A\b", m.group(0)), m.group(0)
    bwd = src["spect_bwd.cu"]
    part = bwd[bwd.index("rdp_sum("):bwd.index("__global__ void k_rdp(")]
    assert "__ldg(" not in part
    part = bwd[bwd.index("b2_gather_sum4("):bwd.index("k_b2_scatter(SpectDev")]
    # the fused form reads the attenuation table (p = As + ...) that way, nothing else
    ldgs = re.findall(r"__ldg\([^;]*;", part)
    assert len(ldgs) == 4 and all("mul4" in ln for ln in part.splitlines() if "__ldg(" in ln)


def test_only_plain_launches_sample_read_only():
    """READ_ONLY samples: in no kernel that is launched while its predecessor runs."""
    text = "\n".join(_sources().values())
    for n in ("k_fwd_nopsf", "k_b2_gather4", "k_b2_nopsf4", "k_b2_adjoint", "k_fwd_strip",
              "k_b1_strip", "k_fwd_ysum", "k_reduce", "k_b1_nopsf"):
        m = re.search(r"__global__[^;{]*?\b%s\(([^)]*)\)\s*{" % n, text)
        assert "READ_ONLY" not in text[m.end():text.index("\n}\n", m.end())], n
    bwd = _sources()["spect_bwd.cu"]
    part = bwd[bwd.index("b2_gather_sum4("):bwd.index("k_b2_gather(SpectDev")]
    assert "READ_ONLY" not in part
    for n in ("k_fwd_psf", "k_b2_gather"):  # plain launches take them
        assert not re.search(r"launch_dependent\(\s*%s\b" % n, text)


def test_movable_loads_depend_on_the_wait():
    """The predicated loads may move, so every dependent kernel that uses them takes its data
    pointer from after_wait(), below its wait."""
    src = _sources()
    for f, names in (("spect_fwd.cu", ["k_fwd_nopsf"]),
                     ("spect_strip.cu", ["b1_strip_item", "fwd_strip_item"]),
                     ("spect_bwd.cu", ["k_b2_nopsf4", "k_b2_gather4"])):
        for n in names:
            m = re.search(r"\b%s\([^;{]*\)\s*{" % n, src[f])
            body = src[f][m.end():src[f].index("\n}\n", m.end())]
            assert body.rindex("grid_wait()") < body.index("after_wait("), n
