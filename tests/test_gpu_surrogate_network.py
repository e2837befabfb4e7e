"""The surrogate network's inference in one kernel (gdtk_gb300/csrc/mlp_tcgen05.cu, mlp_fused_kernel), bit for bit
against the same network layer by layer through the tcgen05 GEMM (which test_gpu_tcgen05.py holds to FP64 products):
both sum the same BF16 products in the same order and share the activation.  For the layer kernel, sizes are padded with
zeros to multiples of 16, as the fused kernel pads in its tiles.

And in norm against FP64 products of the same BF16 weights and activations: an activation may round to the other BF16
neighbour where the FP32 sum (2^-22 or so off) lies that close to the middle, about one in 2^12 by 2^-8, so 2^-14 of the
norm per layer; 2^-10 is allowed.

Sizes: one row, the edges of a tile, one more tile than there are SMs, several tiles in each of a CTA's two slots; layers
of 8 to 256, sizes that are no multiple of 16, the deepest network; and one too wide, which goes layer by layer."""
import ctypes

import numpy as np
import pytest

from conftest import mech

pytestmark = pytest.mark.gpu

CASES = [("park5", 8, 1, 300), ("j92", 16, 2, 1), ("j92", 256, 4, 127), ("j92", 256, 4, 129), ("drm19", 72, 16, 1000),
         ("j92", 256, 4, 152 * 128 + 1), ("j92", 200, 3, 3 * 152 * 128 + 5), ("j92", 256, 4, 262147), ("j92", 264, 2, 700)]


@pytest.mark.parametrize("name,width,depth,n", CASES)
def test_network_in_one_kernel_matches_fp64_products(name, width, depth, n):
    import torch
    from gdtk_gb300 import check, lib
    from gdtk_gb300.cells import ReactorCells
    from gdtk_gb300.surrogate import ChemSurrogate
    sg = ChemSurrogate(ReactorCells(mech(name + "-gas.lua"), mech(name + "-chem.lua")), width=width, depth=depth)
    rng = np.random.Generator(np.random.PCG64(width * 1000 + n))
    dims = sg.layer_dims()
    W = [rng.normal(0.0, np.sqrt(2.0 / dims[l]), (dims[l + 1], dims[l])) for l in range(depth + 1)]
    b = [rng.normal(0.0, 0.1, dims[l + 1]) for l in range(depth + 1)]
    sg.set_params(np.concatenate([w.ravel() for w in W] + b).astype(np.float32))
    xs, ys = rng.normal(0.0, 1.0, dims[0]), rng.normal(0.0, 1.0, dims[-1])
    xd, yd = rng.uniform(0.5, 2.0, dims[0]), rng.uniform(0.5, 2.0, dims[-1])
    sg.set_normalisation(xs, xd, ys, yd, np.full(dims[0], -1e300), np.full(dims[0], 1e300))
    X = torch.tensor(rng.normal(0.0, 1.0, (n, dims[0])), dtype=torch.float32, device="cuda")
    launches, err = ctypes.c_ulonglong(), ctypes.c_int()
    lib().gdtk_mlp_tcgen05(-1, ctypes.byref(launches), None)
    before = launches.value
    out = sg.predict(X)
    torch.cuda.synchronize()
    lib().gdtk_mlp_tcgen05(-1, ctypes.byref(launches), ctypes.byref(err))
    assert err.value == 0, "a tcgen05 wait gave up (%d)" % err.value
    assert launches.value - before == (1 if width <= 256 else 0)

    f32 = lambda a: torch.tensor(np.asarray(a, np.float32), device="cuda")
    h = ((X - f32(xs)) / f32(xd)).to(torch.bfloat16).double()
    for l in range(depth + 1):
        z = h @ f32(W[l]).to(torch.bfloat16).double().t() + f32(b[l]).double()
        if l < depth:
            z = 0.5 * z * (1.0 + torch.tanh(0.7978845608028654 * (z + 0.044715 * z ** 3)))
            h = z.to(torch.bfloat16).double()
    got = (out.double() - f32(ys).double()) / f32(yd).double()
    assert ((got - z).norm() / z.norm()).item() < 2.0 ** -10

    if width > 256:
        return
    up = lambda k: (k + 15) // 16 * 16
    vp = lambda t: ctypes.c_void_p(t.data_ptr())
    h = torch.zeros((n, up(dims[0])), dtype=torch.bfloat16, device="cuda")
    h[:, :dims[0]] = ((X - f32(xs)) / f32(xd)).to(torch.bfloat16)
    for l in range(depth + 1):
        K, N = up(dims[l]), up(dims[l + 1])
        w = torch.zeros((N, K), dtype=torch.bfloat16, device="cuda")
        w[:dims[l + 1], :dims[l]] = f32(W[l]).to(torch.bfloat16)
        c = torch.zeros(N, device="cuda")
        c[:dims[l + 1]] = f32(b[l])
        D = torch.empty((n, N), device="cuda")
        Dh = torch.empty((n, N), dtype=torch.bfloat16, device="cuda")
        check(lib().gdtk_mlp_gemm(n, N, K, vp(h), K, 0, vp(w), K, 1, vp(c), 1 if l < depth else 0, None, vp(D), vp(Dh), N, 1,
                                  ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "gdtk_mlp_gemm")
        h = Dh
    sg.set_normalisation(xs, xd, np.zeros(dims[-1]), np.ones(dims[-1]), np.full(dims[0], -1e300), np.full(dims[0], 1e300))
    assert torch.equal(sg.predict(X), D[:, :dims[-1]])   # times 1 plus 0
