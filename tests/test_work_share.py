"""Dynamic scheduling: the packet queue and the merging of a block's last
packets (csrc/work_share.cuh) leave every packet's path as it is."""
import numpy as np
import pytest

import scenarios


@pytest.mark.gpu
@pytest.mark.parametrize('name', ['c1_line_hg_radial', 'c2_gk_fluence', 'c3_vox_cylinder'])
@pytest.mark.parametrize('n', [1, 31, 33, 513, 40_000])
def test_last_packets_bit_identical_to_oracle(cuda, lib, oracle, name, n):
    """From a single packet to several warps' worth in every block; the
    EXACT tallies and step counts equal the oracle's."""
    mc = scenarios.build_mc(name, scheduling='dynamic')
    ref = oracle.run(mc, n, 0, oracle.PORTABLE, nthreads=8)
    mc.run(n)
    accu = mc._dev['accu'].cpu().numpy().view(np.uint64)
    got = oracle.tallies(mc, accu)
    for k in got:
        assert np.array_equal(got[k], ref[k]), k
    assert mc.run_report['steps'] == ref['steps']
    assert mc.run_report['packets_done'] == n
