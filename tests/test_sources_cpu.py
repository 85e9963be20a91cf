"""What the CUDA sources may not hold.

The library is loaded by one process per GPU of a node as well as by single-GPU programs, so none of its kernels loads by
TMA with cluster multicast (nor commits MMAs to several CTAs of a cluster, which only such loads need).
"""
import glob
import os

from conftest import ROOT


def test_no_cluster_multicast():
    sources = sorted(glob.glob(os.path.join(ROOT, 'hcipy_gb300', 'csrc', '*.cu*')))
    assert len(sources) > 10
    for path in sources:
        with open(path) as f:
            assert 'multicast' not in f.read(), path
