"""GPU tests of the FP32 drop-in's block forms and layer shapes against the FP32 oracle.

The launcher picks the pixels per block from the frame's size and the network's, and a layer's
tile from its width; every form accumulates each dot product in the oracle's order, so the bits
have to be the oracle's."""
import copy

import numpy as np
import pytest

from neural_wavelet_prt_demo_b200 import netconfig
from oracle import oracle as O
from tests.helpers import make_case

pytestmark = pytest.mark.gpu


def _net(levels=8, features=2, aux=16, op=(64, 0, 26), cn=(64, 2)):
    cfg = copy.deepcopy(netconfig.CONFIG_SMALL)
    cfg["vtx_enc"].update(n_levels=levels, n_features_per_level=features, log2_hashmap_size=12)
    cfg["cmp_enc"]["n_padded_dims"] = aux
    cfg["out_prd"].update(n_neurons=op[0], n_hidden_layers=op[1], n_output_dims=op[2])
    cfg["cmp_net"].update(n_neurons=cn[0], n_hidden_layers=cn[1])
    return cfg


def _check(cfg, w, h, K, flags=0.9, clamp=True, kahan=True):
    from neural_wavelet_prt_demo_b200 import engine as eng
    case = make_case(cfg, w, h, K, seed=w + K, hash_scale=0.5, flag_prob=flags)
    e = eng.RenderEngine(case.cfg)
    e.loadWeights(case.weights)
    env = e.addEnvironmentMap(eng.EnvironmentMap(top_coefficients=case.idx, top_strength=case.strength))
    fr = eng.FullFrame.from_gbuffer(case.gbuf)
    e.setFrame(0, fr)
    e.TCNNPass_p1(0)
    e.TCNNPass_p2(env, 0, eng.RenderConfig(precision="fp32", clamp_terms=clamp, kahan=kahan))
    e.TCNNSync()
    ind, wd = O.relight_f32(case.bound, case.idx, case.strength, clamp=clamp, kahan=kahan)
    assert np.array_equal(fr.fbPredictedIndirect.cpu().numpy().view(np.uint32), ind.view(np.uint32))
    assert np.array_equal(fr.fbPredictedIndirectWithDirect.cpu().numpy().view(np.uint32), wd.view(np.uint32))
    e.close()


@pytest.mark.parametrize("n", [1, 33, 64 * 148, 64 * 148 + 1, 128 * 148 + 1, 256 * 148 + 1, 384 * 148 + 1,
                               512 * 148 + 1])
def test_every_block_size_gives_the_oracles_bits(cuda, n):
    _check(_net(), n, 1, 3)


@pytest.mark.parametrize("net", [dict(op=(20, 1, 3), cn=(33, 1)), dict(op=(33, 2, 48), cn=(48, 3), aux=13),
                                 dict(op=(64, 0, 1), cn=(4, 1)), dict(levels=5, features=4, op=(32, 1, 32), cn=(31, 2)),
                                 dict(levels=16, features=8, op=(64, 1, 64), cn=(64, 0)),
                                 dict(levels=16, op=(53, 7, 53), cn=(53, 7))])
def test_odd_layer_shapes_give_the_oracles_bits(cuda, net):
    _check(_net(**net), 67, 5, 19, clamp=False, kahan=False)
    _check(_net(**net), 419, 53, 2)


@pytest.mark.parametrize("net", [dict(levels=24, features=8, aux=13, op=(33, 7, 33), cn=(33, 7)),
                                 dict(levels=20, features=8, op=(36, 7, 53), cn=(36, 7)),
                                 dict(levels=27, features=6, aux=19, op=(36, 7, 40), cn=(40, 7))])
def test_largest_networks_run_with_fewer_wavelets_at_a_time(cuda, net):
    # accepted by the unpadded limit; their padded weight rows leave room for 8, 8 and 2 wavelets'
    # embedding rows beside 32 pixels
    cfg = _net(**net)
    cfg["vtx_enc"]["per_level_scale"] = 1.2
    _check(cfg, 67, 5, 19)
