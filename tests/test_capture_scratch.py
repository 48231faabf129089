"""An FP64 evaluation that the caller captured keeps its buffers: smaller
batches, other slot counts and other calls on the same model in between leave
the replay's results the same bit for bit."""
import numpy as np
import pytest

from helpers import synth_model_file, three_species_cell

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_replay_after_smaller_batches(precision, tmp_path, gapgb_mod, oracle_mod):
    import torch
    import gapgb.synth as S
    path = synth_model_file(str(tmp_path / "gap_parameters"), oracle_mod, [three_species_cell(0)],
                            M=300, coeff_std=0.1)
    m = gapgb_mod.GapModel.load(path)
    m.set_precision(precision)
    m.set_neighbour_cap(96)
    dev = torch.device("cuda:0")

    def batch(n):
        off, sp, lat, pos = S.pack([three_species_cell(s) for s in range(n)])
        N = int(off[-1])
        return dict(S=n, N=N, off=torch.from_numpy(off).to(dev), sp=torch.from_numpy(sp).to(dev),
                    lat=torch.from_numpy(lat).to(dev), pos=torch.from_numpy(pos).to(dev),
                    E=torch.zeros(n, dtype=torch.float64, device=dev),
                    F=torch.zeros((N, 3), dtype=torch.float64, device=dev),
                    St=torch.zeros((n, 6), dtype=torch.float64, device=dev))

    def call(b):
        m.eval_batch_ptrs(b["S"], b["N"], 32, b["off"].data_ptr(), b["sp"].data_ptr(),
                          b["lat"].data_ptr(), b["pos"].data_ptr(), 1, b["E"].data_ptr(),
                          b["F"].data_ptr(), b["St"].data_ptr(),
                          stream=torch.cuda.current_stream().cuda_stream)

    # 1344 atoms: one block per atom; 1184, 576 and 32: atoms split over blocks
    big, rest = batch(42), [batch(37), batch(18), batch(1)]
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        call(big)
    torch.cuda.synchronize()
    m.check_device_status()
    want = [big[k].clone() for k in ("E", "F", "St")]
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        call(big)
    small = []
    for b in rest:
        call(b)
        torch.cuda.synchronize()
        m.check_device_status()
        small.append(b["F"].clone())
    off, sp, lat, pos = S.pack([three_species_cell(s) for s in range(5)])
    m.descriptors(off, sp, lat, pos)
    for _ in range(2):
        for k in ("E", "F", "St"):
            big[k].zero_()
        g.replay()
        torch.cuda.synchronize()
        m.check_device_status()
        for k, w in zip(("E", "F", "St"), want):
            assert torch.equal(big[k], w)
        for b, f in zip(rest, small):
            call(b)
            torch.cuda.synchronize()
            assert torch.equal(b["F"], f)
    # the library's own graph: a smaller batch on the same model beside it
    args = [big[k].data_ptr() for k in ("off", "sp", "lat", "pos")]
    gr = m.graph(big["S"], big["N"], 32, *args, 1, *[big[k].data_ptr() for k in ("E", "F", "St")])
    for b, f in zip(rest, small):
        call(b)
        torch.cuda.synchronize()
        assert torch.equal(b["F"], f)
        gr.launch()
        torch.cuda.synchronize()
        for k, w in zip(("E", "F", "St"), want):
            assert torch.equal(big[k], w)
    gr.close()
    m.close()
