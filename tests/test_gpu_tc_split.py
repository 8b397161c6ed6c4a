"""GPU tests of how a tensor-core launch splits its work: whole tiles (one warpgroup each) and
tiles shared by a CTA's five warpgroups (a chunk of the wavelets each).

The launcher picks the split from the number of 128-pixel tiles, so the same pixels take
different paths alone, in a small launch and in a large one.  Every path forms the sum over the
wavelets from the same chunks in the same order: the bits have to be equal."""
import numpy as np
import pytest

from neural_wavelet_prt_demo_b200 import netconfig
from oracle import oracle as O
from tests.helpers import make_case, psnr

pytestmark = pytest.mark.gpu

PSNR_MIN = 45.0


@pytest.mark.parametrize("cfg,K,kahan", [("small", 1, True), ("small", 4, True), ("small", 5, False),
                                         ("small", 6, True), ("small", 40, True), ("large", 13, True),
                                         ("large", 40, False)])
def test_shared_and_whole_tiles_give_the_same_bits(cuda, cfg, K, kahan):
    from neural_wavelet_prt_demo_b200 import engine as eng
    # 774 tiles: on 148 SMs, 740 whole ones and a shared rest
    case = make_case(netconfig.CONFIG_SMALL if cfg == "small" else netconfig.CONFIG_LARGE, 1021, 97, K, seed=K,
                     hash_scale=0.5, flag_prob=0.9)
    n = 1021 * 97
    e = eng.RenderEngine(case.cfg)
    e.loadWeights(case.weights)
    env = e.addEnvironmentMap(eng.EnvironmentMap(top_coefficients=case.idx, top_strength=case.strength))
    fr = eng.FullFrame.from_gbuffer(case.gbuf)
    e.setFrame(0, fr)
    e.TCNNPass_p1(0)
    rc = eng.RenderConfig(precision="bf16", kahan=kahan)
    e.TCNNPass_p2(env, 0, rc)
    e.TCNNSync()
    whole = fr.fbPredictedIndirect.cpu().numpy(), fr.fbPredictedIndirectWithDirect.cpu().numpy()
    r64 = O.relight_f64(case.bound, case.idx, case.strength)
    assert psnr(whole[0][:, :3], r64) >= PSNR_MIN
    # pieces of 1 px to several tiles per SM: shared tiles only (or, at small K, whole ones);
    # every piece starts its tiles at its own first pixel, so rows change lanes and warps too
    cuts = [0, 1, 130, 130 + 148 * 128, 130 + 148 * 128 + 149 * 128, n - 127, n]
    fr.fbPredictedIndirect.fill_(float("nan"))
    fr.fbPredictedIndirectWithDirect.fill_(float("nan"))
    for b, end in zip(cuts[:-1], cuts[1:]):
        e.relightRanges([(env, 0, fr.fbPredictedIndirect, fr.fbPredictedIndirectWithDirect, b, end)], rc)
    e.TCNNSync()
    for got, ref in zip((fr.fbPredictedIndirect, fr.fbPredictedIndirectWithDirect), whole):
        assert np.array_equal(got.cpu().numpy().view(np.uint32), ref.view(np.uint32))
    e.close()


@pytest.mark.parametrize("net,precision,K", [("six", "fp8", 13), ("two", "fp8", 40), ("plan", "fp8", 13),
                                             ("plan", "bf16", 11)])
def test_split_without_the_tensor_core_output_layer(cuda, net, precision, K):
    # the forms that sum T_k in the last layer's epilogue: a frame of 740 whole tiles and 34 shared
    # ones against its first rows alone, whose tiles are all shared (1 per SM, then 2)
    import copy
    import dataclasses

    from neural_wavelet_prt_demo_b200 import engine as eng
    cfg = copy.deepcopy(netconfig.CONFIG_SMALL if net == "two" else netconfig.CONFIG_LARGE)
    if net == "plan":  # five layers: read from the plan at run time
        cfg["out_prd"]["n_hidden_layers"] = cfg["cmp_net"]["n_hidden_layers"] = 2
    case = make_case(cfg, 1021, 97, K, seed=K, hash_scale=0.5, flag_prob=0.9)
    e = eng.RenderEngine(case.cfg)
    e.loadWeights(case.weights)
    env = e.addEnvironmentMap(eng.EnvironmentMap(top_coefficients=case.idx, top_strength=case.strength))
    rc = eng.RenderConfig(precision=precision)
    out = []
    for rows in (97, 18, 30):
        n = 1021 * rows
        gb = dataclasses.replace(case.gbuf, height=rows, **{
            f: getattr(case.gbuf, f)[:n] for f in ("pos", "normal", "reflect", "roughness", "kd", "ks", "direct", "flag")})
        fr = eng.FullFrame.from_gbuffer(gb)
        e.setFrame(0, fr)
        e.TCNNPass_p1(0)
        if precision == "fp8" and not out:
            e.calibrateFP8(env, 0)
        e.TCNNPass_p2(env, 0, rc)
        e.TCNNSync()
        out.append(fr.fbPredictedIndirect.cpu().numpy())
    assert psnr(out[0][:, :3], O.relight_f64(case.bound, case.idx, case.strength)) >= (30.0 if precision == "fp8"
                                                                                       else PSNR_MIN)
    for part in out[1:]:
        assert np.array_equal(part.view(np.uint32), out[0][:len(part)].view(np.uint32))
    e.close()


@pytest.mark.parametrize("w,h", [(67, 5), (1021, 97)])
@pytest.mark.parametrize("K", [1, 5, 13])
def test_infinite_last_term_gives_infinity(cuda, w, h, K):
    # the compensation of a chunk that ends in an infinite term is not a number and must stay out of
    # the sum: infinity (or, where T_k < 0 is clamped, the finite rest), as without compensation
    from neural_wavelet_prt_demo_b200 import engine as eng
    case = make_case(netconfig.CONFIG_SMALL, w, h, K, seed=K, hash_scale=0.5)
    strength = case.strength.copy()
    strength[-1] = np.inf
    e = eng.RenderEngine(case.cfg)
    e.loadWeights(case.weights)
    env = e.addEnvironmentMap(eng.EnvironmentMap(top_coefficients=case.idx, top_strength=strength))
    fr = eng.FullFrame.from_gbuffer(case.gbuf)
    e.setFrame(0, fr)
    e.TCNNPass_p1(0)
    out = []
    for kahan in (True, False):
        e.TCNNPass_p2(env, 0, eng.RenderConfig(precision="bf16", kahan=kahan))
        e.TCNNSync()
        out.append(fr.fbPredictedIndirect.cpu().numpy()[:, :3])
    assert not np.isnan(out[0]).any()
    assert np.isinf(out[0]).any() and np.array_equal(np.isinf(out[0]), np.isinf(out[1]))
    e.close()


def _pixels(sms, rounds, rest):
    """Pixels of `rounds` whole rounds of tiles (five a CTA) and `rest` more tiles, the last one ragged."""
    return (rounds * 5 * sms + rest) * 128 - 37


def _part(gb, begin, end):
    import dataclasses
    return dataclasses.replace(gb, width=end - begin, height=1, **{
        f: getattr(gb, f)[begin:end] for f in ("pos", "normal", "reflect", "roughness", "kd", "ks", "direct", "flag")})


@pytest.mark.parametrize("cfg,precision,rounds,rest,K", [
    ("small", "bf16", 2, 1, 6),     # tiles from the counter, then one shared
    ("small", "bf16", 2, 290, 13),  # then two per SM
    ("small", "bf16", 3, 300, 6),   # first encodings staggered, counter, a partial round of whole tiles (small K)
    ("large", "bf16", 3, 290, 13),  # staggered, counter, shared
    ("large", "bf16", 21, 660, 13),  # a 1080p frame: staggered, counter, nothing shared
    ("large", "fp8", 3, 140, 6),
])
def test_launches_of_several_rounds(cuda, cfg, precision, rounds, rest, K):
    import torch
    from neural_wavelet_prt_demo_b200 import engine as eng, synth
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    case = make_case(netconfig.CONFIG_SMALL if cfg == "small" else netconfig.CONFIG_LARGE, 64, 4, K, seed=K,
                     hash_scale=0.5)
    n = _pixels(sms, rounds, rest)
    gb = synth.make_gbuffer(n, 1, seed=rounds, flag_prob=0.9)
    e = eng.RenderEngine(case.cfg)
    e.loadWeights(case.weights)
    env = e.addEnvironmentMap(eng.EnvironmentMap(top_coefficients=case.idx, top_strength=case.strength))
    fr = eng.FullFrame.from_gbuffer(gb)
    e.setFrame(0, fr)
    e.TCNNPass_p1(0)
    if precision == "fp8":
        e.calibrateFP8(env, 0, 0, 4096)
    rc = eng.RenderConfig(precision=precision)
    fr.fbPredictedIndirect.fill_(float("nan"))
    e.TCNNPass_p2(env, 0, rc)
    e.TCNNSync()
    whole = fr.fbPredictedIndirect.clone(), fr.fbPredictedIndirectWithDirect.clone()
    # alone: pieces of at most a round, whose tiles are a warpgroup's or shared
    for t in (fr.fbPredictedIndirect, fr.fbPredictedIndirectWithDirect):
        t.fill_(float("nan"))
    for b in range(0, n, 700 * 128):
        e.relightRanges([(env, 0, fr.fbPredictedIndirect, fr.fbPredictedIndirectWithDirect, b, min(n, b + 700 * 128))], rc)
    e.TCNNSync()
    for got, ref in zip(whole, (fr.fbPredictedIndirect, fr.fbPredictedIndirectWithDirect)):
        assert torch.equal(got.view(torch.int32), ref.view(torch.int32))
    # pixels of the first, a later and the last tiles against 64 bits
    for b in (0, n // 2, n - 500):
        part = _part(gb, b, b + 500)
        r64 = O.relight_f64(O.Bound(case.desc, case.weights, part), case.idx, case.strength)
        assert psnr(whole[0][b:b + 500, :3].cpu().numpy(), r64) >= (30.0 if precision == "fp8" else PSNR_MIN)
    e.close()


def test_jobs_of_different_wavelet_counts_in_several_rounds(cuda):
    # tiles of different cost: all from the counter, none shared
    import torch
    from neural_wavelet_prt_demo_b200 import engine as eng, synth
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    cases = [make_case(netconfig.CONFIG_SMALL, 64, 4, K, seed=3, hash_scale=0.5) for K in (6, 40)]
    e = eng.RenderEngine(cases[0].cfg)
    e.loadWeights(cases[0].weights)
    rc = eng.RenderConfig(precision="bf16")
    jobs, frames = [], []
    for i, (case, tiles) in enumerate(zip(cases, (6 * sms, 5 * sms + 11))):
        env = e.addEnvironmentMap(eng.EnvironmentMap(top_coefficients=case.idx, top_strength=case.strength))
        fr = eng.FullFrame.from_gbuffer(synth.make_gbuffer(tiles * 128 - 19, 1, seed=i, flag_prob=0.9))
        e.setFrame(i, fr)
        e.TCNNPass_p1(i)
        frames.append(fr)
        jobs.append((env, i, fr.fbPredictedIndirect, fr.fbPredictedIndirectWithDirect, 0, 0))
    e.relightRanges(jobs, rc)
    e.TCNNSync()
    together = [fr.fbPredictedIndirect.clone() for fr in frames]
    for job in jobs:
        e.relightRanges([job], rc)
    e.TCNNSync()
    for fr, t in zip(frames, together):
        assert torch.equal(t.view(torch.int32), fr.fbPredictedIndirect.view(torch.int32))
    e.close()
