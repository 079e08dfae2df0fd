"""What the autotuner chooses from: the automatic launch shape is among its
candidates, so that tuning never ends at something slower than not tuning; and a
cached choice belongs to one build of the library."""
import types

import numpy as np
import pytest

from brkga_fft2_b200 import autotune as at


def test_automatic_shape_is_a_candidate(monkeypatch):
    """Timed on the CPU with a stand-in decoder for which the automatic shape is the fastest."""
    class Decoder:
        packed, device = "p", types.SimpleNamespace(index=0)
        calls = []

        def set_launch_config(self, *cfg):
            self.calls.append(cfg)

        def decode(self, chrom, out=None, kernel_events=None):
            return out.zero_()

        def launch_config(self):
            return self.calls[-1] if self.calls[-1][3] >= 0 else self.calls[-1][:3] + (0, 8192)

    dec = Decoder()
    monkeypatch.setattr(at, "_time_decode", lambda d, run, repeats: 1.0 if d.calls[-1][0] == 0 else 2.0)
    import torch
    chrom = torch.zeros(3, 4)
    res = at.autotune(dec, chrom, task_max_values=(), key="k")
    assert res["config"][:3] == (0, 0, -1) and res["ms"] == 1.0
    assert dec.calls[-1][:3] == (0, 0, -1)


def test_key_belongs_to_a_build(monkeypatch):
    import torch
    monkeypatch.setattr(torch.cuda, "get_device_properties",
                        lambda i: types.SimpleNamespace(name="dev", multi_processor_count=148))
    pack = types.SimpleNamespace(arrays={"bin_length": np.array([300, 250]), "bin_width": np.array([300, 250])},
                                 n_genes=100, n_machines=2)
    keys = []
    for build in ("a1", "b2"):
        monkeypatch.setattr(at.abi, "library_build_id", lambda: build)
        keys.append(at.grid_key([pack]))
    assert keys[0] != keys[1] and all("grid300x300" in k for k in keys)


@pytest.mark.gpu
def test_tuning_a_small_population_keeps_the_automatic_speed():
    import torch
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for -m gpu tests")
    from brkga_fft2_b200 import instances, pack_problem
    from brkga_fft2_b200.evaluator import DeviceDecoder
    inst = instances.p100m4(0)
    pk = pack_problem(inst.problem_data, inst.nb_parts, inst.nb_machines, inst.thresholds, inst.instance_parts)
    dec = DeviceDecoder(pk, max_pop=20)
    chrom = torch.from_numpy(instances.chromosomes(20, pk.n_genes, 3)).cuda()

    def ms():
        times = []
        for _ in range(9):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            dec.decode(chrom, kernel_events=e)
            torch.cuda.synchronize()
            times.append(e[0].elapsed_time(e[1]))
        return float(np.median(times))

    dec.decode(chrom)
    automatic = ms()
    at.autotune(dec, chrom)
    assert ms() < 1.08 * automatic  # eight warps against four: 1.19
