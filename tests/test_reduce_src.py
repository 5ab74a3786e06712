"""ReduceFunction.get_src names the kernels and the CTA sizes that run."""

import vkdispatch_gb300 as vd
import vkdispatch_gb300.codegen as vc


def test_stages_of_fixed_and_compiled_maps():
    @vd.reduce.map_reduce(vd.reduce.SubgroupAdd)
    def fixed(buffer: vc.Buff[vd.float32]) -> vd.float32:
        return buffer[vd.reduce.mapped_io_index()]

    @vd.reduce.map_reduce(vd.reduce.SubgroupAdd)
    def compiled(buffer: vc.Buff[vd.float32], s: vc.Var[vc.f32]) -> vd.float32:
        return buffer[vd.reduce.mapped_io_index()] * s

    s1, s2 = fixed.get_src()
    assert s1.local_size == (256, 1, 1) and "eight warps" in s1.code
    assert s2.local_size == (512, 1, 1) and "one warp per row" in s2.code
    c1, c2 = compiled.get_src()
    assert c1.local_size == (512, 1, 1) and c2.local_size == (512, 1, 1)
