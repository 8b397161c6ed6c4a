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


# Rotations of different maps into one reused buffer, each followed by a reader of it that may start
# before the kernel ahead of it ends: three kernels of such a chain can be under way at once.
READERS = {
    "wavelets": lambda eng, e, t: list(eng.haar_topk(t, 64)),
    "all wavelets": lambda eng, e, t: list(eng.haar_topk(t, 1024)),
    "project": lambda eng, e, t: [eng.sh_project(t)],
    "rotate": lambda eng, e, t: [eng.env_rotate(t, np.eye(3, dtype=np.float32))],
}


def _maps(S, n, device):
    import torch
    return [torch.from_numpy(synth.make_env_faces(S, seed=50 + i)).to(device) for i in range(n)]


@pytest.mark.parametrize("S", [16, 32, 64])
@pytest.mark.parametrize("reader", list(READERS))
def test_back_to_back_rotations_into_one_buffer(cuda, S, reader):
    import torch
    from neural_wavelet_prt_demo_b200 import engine as eng
    faces, turned = _maps(S, 5, cuda), torch.empty((6, S, S, 3), device=cuda)
    turns = [np.diag(d).astype(np.float32) for d in ([-1.0, 1.0, -1.0], [1.0, -1.0, -1.0], [-1.0, -1.0, 1.0])]

    def chain(sync):
        got = []
        for n in range(40):
            eng.env_rotate(faces[n % 5], turns[n % 3], out=turned)
            if sync:
                torch.cuda.synchronize()
            got += READERS[reader](eng, None, turned)
            if sync:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        return got

    want = chain(True)
    for _ in range(5):
        for a, b in zip(chain(False), want):
            assert torch.equal(a, b)


@pytest.mark.parametrize("reader", ["wavelets", "project"])
def test_passes_in_one_graph_and_over_two_streams(cuda, reader):
    # two passes over the same buffer captured into one graph, on one stream and forked over two:
    # the reader waits for an event of the writer's stream, and the next writer for the reader's
    import torch
    from neural_wavelet_prt_demo_b200 import engine as eng
    S = 64
    faces, turned = _maps(S, 4, cuda), torch.empty((6, S, S, 3), device=cuda)
    src = [torch.empty_like(faces[0]) for _ in range(2)]
    flip = np.diag([-1.0, 1.0, -1.0]).astype(np.float32)

    def passes(other):
        got = []
        main = torch.cuda.current_stream()
        for s in src:
            eng.env_rotate(s, flip, out=turned)
            if other is None:
                got += READERS[reader](eng, None, turned)
            else:
                other.wait_stream(main)
                with torch.cuda.stream(other):
                    got += READERS[reader](eng, None, turned)
                main.wait_stream(other)
        return got

    def load(i):
        for j, s in enumerate(src):
            s.copy_(faces[(i + j) % 4])

    side = torch.cuda.Stream()
    for other in (None, side):
        load(0)
        passes(other)  # the readers' set-up happens outside the capture
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            captured = passes(other)
        for i in range(8):
            load(i)
            torch.cuda.synchronize()
            want = [t.clone() for t in passes(None)]
            torch.cuda.synchronize()
            eager = passes(other)
            torch.cuda.synchronize()
            g.replay()
            torch.cuda.synchronize()
            for a, b, c in zip(want, eager, captured):
                assert torch.equal(a, b) and torch.equal(a, c)
