"""The sizes of latent attention that the sources accept are sizes that the streaming kernel can be built for: its share of an SM's
shared memory (csrc/latent_decode_ring.h) over every latent and rotated part, compiled and run on the host."""
import os
import shutil
import subprocess

import pytest
import torch

PROGRAM = r"""
#include "latent_decode_ring.h"
#include <cstdio>
int main() {
  for (int rank = 16; rank <= 512; rank += 16)
    for (int rot = 0; rot <= 1024; rot += 16)
      for (int groups = 1; groups <= 2; ++groups) {
        const latent_ring::Ring r = latent_ring::ring(rank, rot, groups);
        std::printf("%d %d %d %d %d %d %d %zu %zu\n", rank, rot, groups, r.teams, r.stages, r.share, r.floats, r.stage_bytes, r.smem);
      }
}
"""


@pytest.fixture(scope="module")
def rings(tmp_path_factory):
    from gemmars_b200.csrc import build
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no C++ compiler")
    folder = tmp_path_factory.mktemp("ring")
    (folder / "ring.cc").write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-I", build.HERE, str(folder / "ring.cc"), "-o", str(folder / "ring")], check=True)
    out = subprocess.run([str(folder / "ring")], check=True, capture_output=True, text=True).stdout
    return {tuple(map(int, line.split()[:3])): tuple(map(int, line.split()[3:])) for line in out.splitlines()}


def test_every_accepted_size_has_a_ring(rings):
    from gemmars_b200 import kernels
    seen = 0
    for (rank, rot, groups), (teams, stages, share, floats, stage_bytes, smem) in rings.items():
        if not kernels.latent_attention_mma_usable(torch.bfloat16, rank, rot, 64):
            continue
        seen += 1
        split = 1 if rank <= 128 else 2 if rank <= 256 else 4
        if rank + rot <= 1024:             # wider rows than the prompts' kernel has room for
            assert stages
        if not stages:
            continue
        assert smem <= 227 * 1024 and stages >= 2 * teams and stages % teams == 0 and teams * split * groups <= 8
        assert stage_bytes >= (rank + rot) * 2 * 32
        # what the kernel lays out: two tiles or more a team, the teams' shares or their results, two barriers a tile
        assert floats >= teams * groups * share and floats >= (teams - 1) * split * groups * (rank // split // 2 + 4) * 32
        assert 1024 + stages * stage_bytes + 4 * floats + 16 * stages + 16 + 4 * 1025 <= smem
    assert seen > 500


@pytest.mark.parametrize("rank,rot,teams", [(512, 64, 2), (256, 64, 4), (256, 32, 4), (64, 32, 4), (256, 96, 2), (128, 256, 4), (256, 256, 2)])
def test_teams_of_a_few_sizes(rings, rank, rot, teams):
    assert rings[rank, rot, 1][0] == teams


def test_expanded_heads_ask_for_a_size_that_fits(rings):
    """Units of prompts over expanded heads have the value's width in the latent's place."""
    from gemmars_b200 import kernels
    for dim, rd, vd in ((192, 64, 128), (192, 64, 256), (192, 128, 128)):
        units = kernels.latent_attention_units("bfloat16", 512, rd, dim, vd)
        sizes = [(dict(d)["GB_LATENT_RANK"], dict(d)["GB_LATENT_ROT"]) for u, d in units if u == "latent_attention_mma"]
        assert (vd, dim + rd) in sizes
        assert all(rings[r, t, g][1] for r, t in sizes for g in (1, 2))


@pytest.mark.parametrize("heads,vdim", [(4, 16), (1, 32), (3, 32)])
def test_latents_of_the_step_go_to_no_product_that_asks_for_its_weights_early(heads, vdim, monkeypatch):
    """The values' product over a prompt's latents has the latents in the weights' place.  The kernel for up to 64 rows reads
    weights before the kernel ahead of it has ended, so latents that this step made must not go there."""
    from gemmars_b200 import kernels
    from gemmars_b200.parts.base import build_part
    from gemmars_b200.parts.plan import PartSpec
    dim, rot, rank, hidden, t = 64, 8, 64, 32, 300
    part = build_part("mixer", PartSpec("latent_attention", {
        "hidden_size": hidden, "num_heads": heads, "dim": dim, "rot_dim": rot, "vdim": vdim, "rank": rank, "scale": 0.1, "norm_eps": 1e-6,
        "gate": False, "window": None}), "bfloat16")
    made = {n: torch.randn(w.shape).to(torch.bfloat16 if w.role == "matrix" else torch.float32) for n, w in part.wants().items()}
    part.load(made)
    latents, shared = torch.randn(kernels.latent_expand_rows(t, 1), rank).bfloat16(), torch.randn(kernels.latent_expand_rows(t, 1), rot).bfloat16()
    early, results = [], {}

    def product(x, w, out, *args, **kwargs):
        out.copy_(x.float() @ w.float().T)

    def few(x, w, out, *args, **kwargs):
        early.append(w.data_ptr())
        product(x, w, out)

    monkeypatch.setattr(kernels, "gemm_tc", few)
    monkeypatch.setattr(kernels, "gemm_tc_persistent", product)
    monkeypatch.setattr(kernels, "attention_prefill_latent", lambda q, o, nh, keys, shared, values, *a: results.update(keys=keys, values=values))
    part.o = type("O", (), {"add_into": lambda self, *a: None})()
    q = torch.zeros(t, heads * (dim + rot), dtype=torch.bfloat16)
    ctx = type("Ctx", (), {"seq_start": torch.zeros(1, dtype=torch.int32)})()
    part._expanded_tc(ctx, q, None, None, (latents, shared, torch.tensor([0, t], dtype=torch.int32)), torch.zeros(t, hidden))
    assert latents.data_ptr() not in early
    assert torch.equal(results["values"], (made["uv"].float() @ latents.float().T).bfloat16())
    assert torch.equal(results["keys"], (latents.float() @ made["uk"].float().T).bfloat16())
