"""Registers of the tracking kernels, from the compiler's own account of the build.

The unsliced trackers run at the registers that their blocks per SM leave them;
spilled registers cost the tensor trackers inside a surface 1.5 to 2 % of their time.
"""

import re

import pytest

from tractography_b200._lib import LIB_PATH

LOG = LIB_PATH.parent / "obj" / "tg_track.o.log"
KERNEL = re.compile(r"Compiling entry function '_ZN2tg23track_persistent_kernelI((?:L[ib]\d+E)+)E\S*'.*?"
                    r"(\d+) bytes spill stores, (\d+) bytes spill loads", re.S)


@pytest.mark.skipif(not LOG.exists(), reason="the library was not built here")
def test_unsliced_trackers_do_not_spill():
    kernels = {tuple(int(v) for v in re.findall(r"L[ib](\d+)E", args)): (int(stores), int(loads))
               for args, stores, loads in KERNEL.findall(LOG.read_text())}
    unsliced = {k: v for k, v in kernels.items() if k[-1] == 0}
    assert len(unsliced) == 36                  # six models, two algorithms, three domain forms
    assert {k: v for k, v in unsliced.items() if v != (0, 0)} == {}
