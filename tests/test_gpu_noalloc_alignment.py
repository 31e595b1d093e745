"""bafqmc_sweep_noalloc on fields that start at an odd double of a larger buffer (aligned to 8 bytes, not to
16): the bits of the same call on a buffer of its own, in each size class and both sectors."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lx,ly,delta", [(3, 3, None), (5, 5, None), (6, 8, None), (8, 10, None), (2, 3, 0.25), (3, 5, 0.25),
                                         (5, 5, 0.25)])
def test_fields_at_an_odd_double(lx, ly, delta):
    import torch
    from bafqmc_b200 import _lib, build
    from bafqmc_b200.params import SolverParams
    from bafqmc_b200.solver import point_struct
    lib = _lib.load(build.build())
    kw = dict(U1=1.0, U2=-0.5, mu=-7.0, Nlx=lx, Nly=ly, Ltrot=10, Beta=0.5, NlxTherm=lx, NlyTherm=ly, LtrotTherm=10,
              Nwrap=5, Nbin=1, Nsweep=1, shiftLoc=1.0, iniType=2, iniAmpl=1.0)
    p = SolverParams(**kw) if delta is None else SolverParams(**kw, delta=delta, sector=1)
    n = 3
    nf, stride = n * 10 * p.Lq * 2, _lib.OBS_SCALARS + p.Lq
    phi = np.random.default_rng(lx * ly).standard_normal(nf)
    out = []
    for offset in (0, 1):
        buf = torch.zeros(nf + 2, dtype=torch.float64, device="cuda")
        f = buf[offset:offset + nf]
        assert f.data_ptr() % 16 == 8 * offset
        f.copy_(torch.from_numpy(phi))
        seeds = torch.tensor([11, 13, 15], dtype=torch.int32, device="cuda")
        obs = torch.zeros(n * stride, dtype=torch.float64, device="cuda")
        rc = lib.bafqmc_sweep_noalloc(C.byref(point_struct(p)), n, seeds.data_ptr(), f.data_ptr(), 2, obs.data_ptr(),
                                      torch.cuda.current_stream().cuda_stream)
        assert rc == 0, lib.bafqmc_last_error()
        out.append([t.cpu().numpy() for t in (seeds, f, obs)])
        assert buf[offset + nf:].abs().max() == 0 and (offset == 0 or buf[0] == 0)
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
    assert not np.array_equal(out[0][1], phi)
