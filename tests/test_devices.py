"""Handles on two devices of one process, on the stand-in runtime: each device's handle takes every
velocity kernel, those with more dynamic shared memory than a launch gets unasked among them (the
limit belongs to the device)."""
from standin_runtime import run

PROGRAM = r"""
from helpers import config0_params, config1_params, tangle
from nuvort_b200.api import Handle, NuvortError
st = tangle(3, 0.002, n_points=200)
for device in (0, 1):
    for precision in ("fp64", "mixed"):
        with Handle(config0_params(precision=precision), [300], device=device, states=[st]) as h:
            for split in (1, 2, 4, 8):
                h.set_direct_split(split)
                h.calc_velocity()
                h.calc_velocity_direct_at(0, [1, 2, 3])
        with Handle(config1_params("Tree", precision=precision), [300], device=device, states=[st]) as h:
            for parts in (1, 2) if precision == "fp64" else (1, 2, 4, 8):
                h.set_walk_parts(parts)
                h.calc_velocity()
runtime.test_refuse_limits(1)
try:
    Handle(config0_params(), [300])
except NuvortError as e:
    assert "shared-memory limit" in str(e), e
else:
    raise AssertionError("a refused limit went unnoticed")
print("both devices")
"""


def test_every_velocity_kernel_on_a_second_device(tmp_path):
    assert "both devices" in run(tmp_path, PROGRAM)
