"""The k-vector tables of a changed setting cannot be sent while the stream
captures: the evaluation is refused then, and the next plain one has to send
them.  Compared with a context that never saw the refusal; both evaluations
are the same launches over the same tables, so the tolerance (1e-12 FP64,
1e-6 mixed, of the largest force) only leaves room for rounding."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def evaluate(ff, sysm, stream):
    import torch
    with torch.cuda.stream(stream):
        x = torch.from_numpy(np.ascontiguousarray(sysm.site)).cuda()
        f = torch.zeros_like(x)
        r = torch.zeros(11, dtype=torch.float64, device="cuda")
        stream.synchronize()

        def go():
            ff.forces_device(x.data_ptr(), f.data_ptr(), r.data_ptr(), r.data_ptr() + 16)
        return go, f, r


@pytest.mark.parametrize("form,tol", [("fp64", 1e-12), ("mixed", 1e-6)])
@pytest.mark.parametrize("change", ["k_cutoff", "alpha", "precision"])
def test_refused_upload_is_made_good(form, tol, change):
    import torch
    from moldy_gb300 import ForceField, system
    from moldy_gb300._lib import MdgpuError
    sysm = system.water(nside=6, seed=2)
    ctl = sysm.control
    if change == "k_cutoff":
        ctl = dataclasses.replace(ctl, k_cutoff=0.8 * ctl.k_cutoff)
    elif change == "alpha":
        ctl = dataclasses.replace(ctl, alpha=0.9 * ctl.alpha)
    stream = torch.cuda.Stream()

    fresh = ForceField(dataclasses.replace(sysm, control=ctl), precision=form)
    fresh.set_stream(stream.cuda_stream)
    go, f0, r0 = evaluate(fresh, sysm, stream)
    go()
    fresh.synchronize()

    other = {"fp64": "mixed", "mixed": "fp64"}[form] if change == "precision" else form
    ff = ForceField(sysm, precision=other)
    ff.set_stream(stream.cuda_stream)
    go, f, r = evaluate(ff, sysm, stream)
    for prec in (form, other):      # every buffer of both forms allocated
        ff.set_precision(prec)
        go()
    ff.synchronize()
    ff.set_control(ctl)
    ff.set_precision(form)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        graph.capture_begin(capture_error_mode="thread_local")
        with pytest.raises(MdgpuError):
            go()
        try:
            graph.capture_end()
        except RuntimeError:
            pass
    f.zero_()
    torch.cuda.synchronize()
    go()
    ff.synchronize()
    for a, b in ((f0, f), (r0, r)):
        assert float((a - b).abs().max()) <= tol * float(a.abs().max())
    ff.close()
    fresh.close()
