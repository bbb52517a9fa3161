"""Page-locked arrays are read in place only when one page-locked range holds them."""
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHECK = r"""
#include "tbr_host.h"
#include <cstdio>
int main() {
    const unsigned long long top = ~0ull;
    unsigned long long a, b, c, d;
    while (std::scanf("%llu %llu %llu %llu", &a, &b, &c, &d) == 4) std::printf("%d\n", (int)tbr::range_holds(a, b, c, d));
    return tbr::range_holds(top - 9, 10, top - 9, 10) && !tbr::range_holds(top - 9, 10, top - 8, 10) ? 0 : 1;
}
"""


def test_range_rule(tmp_path):
    src, exe = tmp_path / "check.cpp", tmp_path / "check"
    src.write_text(CHECK)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "turboransac_b200", "csrc"), "-o", exe, src], check=True)
    rows = [(s, z, p, b) for s in (64, 4096) for z in (0, 1, 8, 4096) for p in (56, 64, 72, 4088, 4096, 4104, 8184, 8192)
            for b in (1, 8, 16, 4096, 4097, 2 ** 63)]
    out = subprocess.run([exe], input="\n".join(" ".join(map(str, r)) for r in rows), text=True, capture_output=True, check=True)
    want = [int(s <= p and p + b <= s + z) for s, z, p, b in rows]
    assert [int(x) for x in out.stdout.split()] == want and sum(want) > 10


@pytest.mark.gpu
def test_arrays_across_two_registrations_are_staged(ctx, oracle):
    """A buffer whose first and last pages are registered, each for itself, and whose middle
    is not: its arrays are copied, not read where they are."""
    import mmap

    import torch

    from turboransac_b200 import (BundleOptions_cuda, Camera_cuda, CameraPose_cuda, RansacOptions_cuda, estimate_batch,
                                  scenes)
    f = scenes.make_frame(60000, 0.6, 0.5, 33)
    rt, keep = torch.cuda.cudart(), []

    def split(a):
        buf = mmap.mmap(-1, -(-a.nbytes // 4096) * 4096)
        raw = np.frombuffer(buf, np.uint8)
        out = raw[:a.nbytes].view(np.float64).reshape(a.shape)
        out[:] = a
        at = raw.ctypes.data
        for p in (at, at + raw.size - 4096):
            assert int(rt.cudaHostRegister(p, 4096, 0)) == 0
            keep.append(p)
        return out

    xn = np.ascontiguousarray((f.uv - [f.K[2], f.K[3]]) / [f.K[0], f.K[1]])
    uv, xyz, x = split(f.uv), split(f.xyz), split(xn)
    cam = Camera_cuda(1, 640, 480, [float(k) for k in f.K])
    ro, bo = RansacOptions_cuda(max_iterations=64, max_reproj_error=4.0), BundleOptions_cuda()
    st, pose, m = ctx.estimate_absolute_pose(uv, xyz, cam, ro, bo, seed=f.seed)
    st0, pose0, m0 = ctx.estimate_absolute_pose(f.uv, f.xyz, cam, ro, bo, seed=f.seed)
    np.testing.assert_array_equal(pose.q, pose0.q)
    np.testing.assert_array_equal(m, m0)
    thr = 16.0 / (0.5 * (f.K[0] + f.K[1])) ** 2
    p = CameraPose_cuda(oracle.rotmat_to_quat(f.R_gt), f.t_gt)
    np.testing.assert_array_equal(ctx.get_inliers(p, x, xyz, thr), ctx.get_inliers(p, xn, f.xyz, thr))
    b, _ = ctx.bundle_adjust(uv, xyz, cam, p, bo)
    b0, _ = ctx.bundle_adjust(f.uv, f.xyz, cam, p, bo)
    np.testing.assert_array_equal(b.q, b0.q)
    g = scenes.make_frame(60000, 0.6, 0.5, 33)
    g.uv, g.xyz = uv, xyz
    for r in estimate_batch(ctx, [g, f, g], ro):  # 7 MB: ingested
        np.testing.assert_array_equal(r["q"], pose0.q)
    for q in keep:
        rt.cudaHostUnregister(q)
