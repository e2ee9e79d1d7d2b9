"""The library's compilation units: every kernel the engine may pick is compiled
in exactly one of them, and none by a compiler mode whose output changes from
run to run."""
from mpm_3d_b200 import build


def test_kernels_do_not_depend_on_the_run_of_the_compiler():
    flags = build.NVCC_FLAGS + [f for _, _, more in build.UNITS for f in more]
    assert not any("split-compile" in f for f in flags)


def test_each_kernel_group_is_one_unit():
    groups = [(d.get("MPM_LEAN_CAP"), d.get("MPM_STAGED_DET"), d.get("MPM_POINT")) for _, d, _ in build.UNITS]
    want = [(cap, None, pt) for cap in ("128", "256", "512") for pt in ("double", "float")]
    want += [(None, "0", "double"), (None, "0", "float"), (None, "1", "double"), (None, None, None)]
    assert sorted(groups, key=str) == sorted(want, key=str)
