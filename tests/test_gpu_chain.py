"""GPU test of calls that follow one another without a synchronisation: kernels may start before the
one ahead of them ends, so every call must still see its inputs complete and leave its outputs to
earlier readers.  The same chain with a synchronisation after each call gives the expected bits."""
import numpy as np
import pytest

from neural_wavelet_prt_demo_b200 import netconfig, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [16, 64])
def test_chain_matches_synchronised_calls(cuda, K):
    import torch
    from neural_wavelet_prt_demo_b200 import engine as eng
    cfg = netconfig.CONFIG_SMALL
    desc = netconfig.parse(cfg)
    S = desc.face_size
    e = eng.RenderEngine(cfg)
    e.loadWeights(synth.make_weights(desc, seed=3, hash_scale=0.5))
    frames = [eng.FullFrame.from_gbuffer(synth.make_gbuffer(w, h, seed=w), cuda) for w, h in ((37, 29), (200, 111))]
    for i, fr in enumerate(frames):
        e.setFrame(i, fr)
    faces = [torch.from_numpy(synth.make_env_faces(S, seed=i)).to(cuda) for i in range(2)]
    flip = np.diag([-1.0, 1.0, -1.0]).astype(np.float32)
    turned = torch.empty_like(faces[0])  # reused by every pass, as the frames' outputs are
    pixels = [torch.empty(fr.width * fr.height, dtype=torch.int32, device=cuda) for fr in frames]
    conf = eng.RenderConfig(precision="bf16")

    def chain(sync):
        step = torch.cuda.synchronize if sync else (lambda: None)
        got = []
        for n in range(12):
            i = n % 2
            fr = frames[i]
            eng.env_rotate(faces[n // 2 % 2], flip, out=turned)
            step()
            env = e.addEnvironmentFaces(turned, K)
            step()
            idx, strength = eng.haar_topk(turned, K)
            step()
            L = eng.sh_project(turned)
            step()
            e.TCNNPass_p1(i)
            step()
            e.relightRanges([(env, i, fr.fbPredictedIndirect, fr.fbPredictedIndirectWithDirect, 0, 0)], conf)
            step()
            eng.tonemap_srgb(fr.fbPredictedIndirectWithDirect, out=pixels[i])
            step()
            got += [idx, strength, L, fr.fbPredictedIndirect.clone(), pixels[i].clone()]
            e.releaseEnvironmentMap(env)
        torch.cuda.synchronize()
        return got

    want = chain(True)
    for _ in range(5):
        for a, b in zip(chain(False), want):
            assert torch.equal(a, b)
