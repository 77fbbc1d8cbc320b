"""Rules of the kernel sources that a run cannot show to be broken."""
import glob
import os

CSRC = os.path.join(os.path.dirname(__file__), "..", "gomc_gb300", "csrc")


def test_shuffle_masks_are_stated():
    """__activemask() names the lanes that happen to be converged; as the mask
    of a shuffle or a vote it may lack one that takes part.  The kernels state
    the lanes instead."""
    files = sorted(glob.glob(os.path.join(CSRC, "*.cu*")))
    assert files
    for f in files:
        assert "__activemask" not in open(f).read(), os.path.basename(f)
