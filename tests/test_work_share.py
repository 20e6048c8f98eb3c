"""Dynamic scheduling and the batched engine: the packet queue, its order and
the merging of a block's last packets (csrc/work_share.cuh) leave every
packet's path as it is."""
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


@pytest.mark.gpu
@pytest.mark.parametrize('num', [1, 33, 1025])
def test_batched_order_bit_identical_to_oracle(cuda, lib, oracle, num):
    """Simulations are queued by the life of their packets: across a tile of
    the ordering block, with empty, unabsorbing and opaque ones among them."""
    from pyxopto_gb300.batched import BatchedMc
    sims = BatchedMc.sample_sims(num, seed=9, packets=(5, 60))
    sims['thickness'][::2] = 5e-4
    sims['num_packets'][1::7] = 0
    sims['mua'][2::8] = 0.0
    sims['thickness'][2::8] = 5e-4
    sims['mua'][3::8] = 1e7
    b = BatchedMc(sims, fast=False, seed=4)
    ref, steps = oracle.batched_run(b, nthreads=8)
    assert np.array_equal(b.run_raw(), ref)
    assert b.last_report['steps'] == steps
    assert b.last_report['packets'] == int(b.packets.sum())
