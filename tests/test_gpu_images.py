"""The image sums over a length-ordered prefix of the image cells: image counts at the edges of the
pair numbering (one image, two, a ragged ball of cells, the most a handle takes), cells smaller than
the truncation range, and segments small enough to be cut into one-primitive chunks, against the
oracle (the element-wise bound and equal decision counters of test_gpu_parity)."""
import pytest

from libgint_b200.workload import Workload
from test_gpu_parity import _compare

CASES = [dict(name="periodic_l2", n_mol=2, box_ang=5.5, n_occ=12, n_img_1d=3, max_images=2),
         dict(name="periodic_l2", n_mol=2, box_ang=5.5, n_occ=12, n_img_1d=7, max_images=33),
         dict(name="periodic_l2", n_mol=2, box_ang=5.5, n_occ=12, n_img_1d=7, max_images=256, setq_stride=3),
         dict(name="periodic_l3", n_mol=2, box_ang=6.0, n_occ=12, n_img_1d=5, max_prm=3, max_ncontr=2,
              setq_stride=61),
         dict(name="periodic_l3", n_mol=2, box_ang=6.0, n_occ=12, n_img_1d=3, max_images=1, max_prm=5,
              setq_stride=7)]


@pytest.mark.gpu
@pytest.mark.parametrize("spec", CASES, ids=lambda s: f"{s['name']}-{s.get('max_images', 0)}")
def test_image_prefix_vs_oracle(engine_so, oracle_path, spec):
    _compare(engine_so, oracle_path, Workload(**spec))
