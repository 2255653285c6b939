"""The staged batch over every kind of column sweep it groups: FFT sweeps of
windows beyond the tensor-core sweep's (half-sizes 49 to 60) with two transform
lengths, several windows on the tensor cores, the direct kernel, and more
sequences of one window than a launch takes (64).  Outputs equal the handles' own
frames bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _frames(synth, specs):
    out = []
    for k, ((h, w), _, _, nf, _, _) in enumerate(specs):
        frames, phi0, _ = synth.sequence(h, w, nf, seed=300 + k)
        out.append((frames.astype(np.float32), phi0.astype(np.float32)))
    return out


def _handle(glsu, spec, phi0):
    (_, _), r, rr, _, wp, method = spec
    d = glsu.DPRA(phi0, rr, r, "f32", wp)
    if method is not None:
        d.set_method(method)
    return d


def _check(glsu, synth, specs, graph, steps=None):
    import torch
    data = _frames(synth, specs)
    ref, handles, seqs = [], [], []
    for spec, (fr, phi0) in zip(specs, data):
        d = _handle(glsu, spec, phi0)
        out, _ = d.sequence(fr)
        ref.append((out, d.get(glsu.PHI_REF).copy()))
        d.close()
        handles.append(_handle(glsu, spec, phi0))
        seqs.append(torch.from_numpy(fr).cuda())
    tunings = [d.tuning() for d in handles]
    b = glsu.DpraBatch(handles, graph=graph)
    dphi = [[] for _ in specs]
    for step in range(max(s[3] for s in specs)):
        b.run([seqs[k][step].data_ptr() if step < specs[k][3] else None for k in range(len(specs))], glsu.F32)
        b.sync()
        for k, s in enumerate(specs):
            if step < s[3]:
                dphi[k].append(handles[k].get(glsu.DPHI).copy())
    b.close()
    for k, d in enumerate(handles):
        assert np.array_equal(np.stack(dphi[k]), ref[k][0]), k
        assert np.array_equal(d.get(glsu.PHI_REF), ref[k][1]), k
        d.close()
    return tunings


def _wff(glsu, sigma, step=0.25):
    return glsu.WffParams(sigma, -0.75, 0.75, step, sigma, -0.75, 0.75, step, 0.2)


@pytest.mark.parametrize("graph", [False, True])
def test_classes_of_every_sweep_side_by_side(glsu, synth, graph):
    """Seven frames of most sequences, so that each step (two parities of the phase
    buffers) is run eagerly, captured and replayed in graph mode."""
    fft = glsu.METHOD_FFT
    specs = [((96, 80), 2, 1, 7, _wff(glsu, 17.0), fft),      # half-size 51, length 256
             ((128, 100), 3, 1, 7, _wff(glsu, 20.0), fft),    # half-size 60, length 256
             ((300, 64), 2, 1, 7, _wff(glsu, 17.0), fft),     # length 512
             ((310, 130), 2, 1, 7, _wff(glsu, 20.0), fft),    # length 512
             ((130, 90), 2, 1, 7, _wff(glsu, 10.0), fft),     # tensor cores, half-size 30
             ((333, 70), 3, 1, 7, _wff(glsu, 10.0), fft),
             ((161, 65), 2, 1, 7, _wff(glsu, 4.0), fft),      # tensor cores, half-size 12
             ((64, 200), 2, 1, 7, _wff(glsu, 4.0), fft),
             ((60, 70), 2, 1, 6, _wff(glsu, 4.0), glsu.METHOD_DIRECT)]
    t = _check(glsu, synth, specs, graph)
    assert {v["method"] for v in t[:8]} == {fft} and t[8]["method"] == glsu.METHOD_DIRECT
    assert len({v["fft_length"] for v in t[:4]}) == 2


def test_more_sequences_of_one_window_than_a_launch_takes(glsu, synth):
    specs = [((24 + k % 5, 32 + k % 7), 2, 1, 2, _wff(glsu, 2.0, 0.5), glsu.METHOD_FFT) for k in range(70)]
    _check(glsu, synth, specs, False)
