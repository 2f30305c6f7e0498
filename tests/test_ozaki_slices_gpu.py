"""The FP32 slice kernel against the FP64 chain: a rotation of FP32 columns must
equal, bit for bit, the rotation of the same columns held in FP64 (same slices,
exact integer sums), for column scales from the smallest to the largest FP32
numbers, zero columns, halfway values, lengths around the 128-element padding,
and column counts around the 64 / 128 tiles of the rotation kernel."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rotate(qsb, U, C):
    import torch
    K, N = U.shape
    q = C.shape[0]
    need = ctypes.c_size_t()
    assert qsb.lib.qsb_rotate_ozaki_int8_workspace(ctypes.c_int64(N), K, q, ctypes.byref(need)) == 0
    ws = torch.empty(need.value, dtype=torch.uint8, device="cuda")
    out = torch.empty(q, N, dtype=torch.float32, device="cuda")
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())
    dt = 0 if U.dtype == torch.float64 else 1
    assert qsb.lib.qsb_rotate_ozaki_int8(dt, ctypes.c_int64(N), K, q, ptr(U), ptr(C), ptr(out), ptr(ws),
                                         ctypes.c_size_t(need.value), None) == 0
    torch.cuda.synchronize()
    return out


@pytest.mark.parametrize("N,K,q", [(128, 1, 1), (1000, 63, 64), (4099, 65, 127), (777, 128, 129), (5000, 193, 256),
                                   (20000, 40, 300)])
def test_f32_slices_equal_the_f64_chain(qsb, N, K, q):
    import torch
    rng = np.random.default_rng(N + K)
    U = (rng.uniform(-1, 1, (K, N)) * np.exp2(rng.integers(-40, 1, (K, N)))).astype(np.float32)
    for k in range(K):
        U[k] *= np.float32(2.0) ** rng.integers(-60, 60)
    if K > 8:
        U[1] = 0.0
        U[2] = np.float32(1e-42)                       # subnormal
        U[3] = rng.uniform(-3e38, 3e38, N).astype(np.float32)
        U[4] = (rng.integers(-64, 64, N) + 0.5).astype(np.float32)     # halfway between slices
        U[5] = np.float32(2.0 ** -126)
    C = rng.uniform(-1, 1, (q, K)) * np.exp2(rng.integers(-20, 20, (q, K)).astype(np.float64))
    C[:, 3 % K] *= 1e-30
    a = torch.from_numpy(U).cuda()
    c = torch.from_numpy(C).cuda()
    f32, f64 = _rotate(qsb, a, c), _rotate(qsb, a.double(), c)
    assert torch.equal(f32.view(torch.int32), f64.view(torch.int32))
    # and the rotation itself: the fourth slice leaves 2^-27 of max|u| max|c| per term
    ref = C @ U.astype(np.float64)
    bound = (np.abs(U.astype(np.float64)).max(1)[None, :] * np.abs(C)).sum(1)[:, None]
    err = np.abs(f32.double().cpu().numpy() - ref)
    cmax = (np.abs(C) * np.exp2(np.ceil(np.log2(np.maximum(np.abs(U.astype(np.float64)).max(1), 1e-300))))).max(1)
    assert np.all(err <= 2.0 ** -22 * np.abs(ref) + 2.0 ** -24 * (bound + K * cmax[:, None]) + 1e-44)
    assert qsb.device_status() == 0
