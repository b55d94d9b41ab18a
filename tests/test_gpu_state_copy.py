"""States in and out between device arrays: every byte arrives and none beside
it, for whole 16-byte words, 4-byte words and addresses that the copy kernel
leaves to the runtime, for odd sizes and for arrays left out."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from aquagpusph_gb300 import case as cases


@pytest.mark.parametrize("dims", [2, 3])
@pytest.mark.parametrize("n", [1, 5, 1023, 4099])
@pytest.mark.parametrize("offset", [0, 4, 2])
def test_state_round_trip_between_device_arrays(dims, n, offset):
    torch = pytest.importorskip("torch")
    from aquagpusph_gb300.solver import Solver
    p = (cases.dam_break_2d(dx=0.02, tank=(1.0, 0.8), column=(0.2, 0.2)) if dims == 2 else
         cases.dam_break_3d(dx=0.05, tank=(1.0, 0.6, 0.6), block=(0.2, 0.2, 0.2),
                            probes_z=(0.1,))).params
    rng = np.random.default_rng(n + dims + offset)
    c = cases.Case(p, n)
    host = {k: np.ascontiguousarray(v) for k, v in c.state_arrays().items()}
    for v in host.values():
        v[...] = (rng.integers(0, n, v.shape) if v.dtype.kind in "iu" else
                  rng.normal(size=v.shape)).astype(v.dtype)
    pad = 64

    def buffers(fill):
        out = {}
        for k, v in host.items():
            b = torch.full((v.nbytes + 2 * pad,), 0xA5, dtype=torch.uint8, device="cuda")
            if fill:
                b[pad + offset:pad + offset + v.nbytes] = torch.from_numpy(
                    v.reshape(-1).view(np.uint8).copy()).cuda()
            out[k] = b
        return out

    src, dst = buffers(True), buffers(False)
    ptr = lambda b: {k: v.data_ptr() + pad + offset for k, v in b.items()}  # noqa: E731
    torch.cuda.synchronize()
    sv = Solver(p, capacity=n)
    sv.set_state_raw(n, ptr(src), False, 0.0, p.dt_fixed, 0)
    out = ptr(dst)
    out.pop("p")  # left out
    sv.get_state_raw(out, False)
    torch.cuda.synchronize()
    for k, v in host.items():
        b = dst[k].cpu().numpy()
        got = b[pad + offset:pad + offset + v.nbytes]
        if k == "p":
            assert np.all(b == 0xA5)
            continue
        assert np.array_equal(got, v.reshape(-1).view(np.uint8)), k
        assert np.all(b[:pad + offset] == 0xA5) and np.all(b[pad + offset + v.nbytes:] == 0xA5), k
    sv.close()
