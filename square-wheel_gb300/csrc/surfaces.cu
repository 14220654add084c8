// Surface builder for the GB300 path: every visible polygon surface of a frame in one persistent
// launch.
//
// Replaces build_polygons_surfaces' per-polygon work (src/square_wheel/partial_renderer.rs:1682-1831):
// build_surface_impl_6_static_params (src/square_wheel/surfaces.rs:433-852) followed by the emissive
// layer mix_surface_with_texture (src/square_wheel/surfaces.rs:903-971), fused in one pass.
//
// Work decomposition: the frame's surfaces form one flat texel index space (prefix sums of surface
// areas, in descriptor order). A grid of (#SMs x resident blocks) threads strides over it, so surfaces
// from 4x4 to 512x512 texels share one launch without tail effects. A warp takes `runs` runs of 32 consecutive
// texels: it finds the first texel's surface by a 32-way search of the prefix array, and every lane then steps
// forward to its own surface (at most a few steps, only across tiny surfaces). Neighbouring lanes read
// neighbouring TextureElements, so texture reads and surface writes are coalesced.
// A directional lightmap goes through the reference's row buffer (surfaces.rs:477-502): where the 32 texels lie in one or two
// surface rows (all but surfaces narrower than 17), the warp builds the line entries they touch together, one
// component per lane from neighbouring floats, in shared memory, and each texel only mixes its two entries;
// elsewhere, and for the three floats of a simple lightmap's element, every thread builds its two entries alone. Operations and their order are the reference's either way.
#include "launch_rules.h"
#include "sw_kernels.cuh"

#include <cmath>

namespace swgpu
{

namespace
{

const float NORMAL_UNPACK_SCALE = 1.0f / 127.0f;
constexpr float PI_F = 3.14159265358979323846f;
// Specular lobe constants, src/square_wheel/surfaces.rs:1108-1110 (f32 constant arithmetic).
constexpr float SPEC_A = 2.0f * PI_F / 2.645751311f;
constexpr float SPEC_B = PI_F * 2.645751311f / 2.0f;
constexpr float DIELECTRIC_ZERO_REFLECTIVITY = 0.04f;
constexpr float DIELECTRIC_AVERAGE_REFLECTIVITY = DIELECTRIC_ZERO_REFLECTIVITY * 3.0f;
constexpr float METAL_AVERAGE_SCHLICK_FACTOR = 0.5f;

__device__ __forceinline__ float specular_intensity(float angle_cos, float inv_roughness)
{
	float x = fmul(fsub(angle_cos, 1.0f), inv_roughness);
	return fmul(inv_fast(mad2(fmul(x, x), SPEC_B, SPEC_A)), inv_roughness);
}
__device__ __forceinline__ float fresnel_factor_base(float c)
{
	float omc = fmaxf(fsub(1.0f, c), 0.0f);
	float omc2 = fmul(omc, omc);
	return fmul(fmul(omc2, omc2), omc);
}
__device__ __forceinline__ float specular_k(int spec, float f, float roughness)
{
	if (spec == 1)
	{
		float fresnel = mad2(f, 1.0f - DIELECTRIC_ZERO_REFLECTIVITY, DIELECTRIC_ZERO_REFLECTIVITY);
		return mad2(fresnel, fsub(1.0f, roughness), fmul(DIELECTRIC_AVERAGE_REFLECTIVITY, roughness));
	}
	return mad2(f, fsub(1.0f, roughness), fmul(METAL_AVERAGE_SCHLICK_FACTOR, roughness));
}

struct Lm
{
	float amb[3];
	V3 dir;
	float dev;
	float col[3];
};
// Floats of a lightmap element: ambient, direction, deviation, colour; or the colour alone.
template <bool DIRECTIONAL>
constexpr uint32_t LM_FLOATS = DIRECTIONAL ? 10 : 3;
static_assert(sizeof(SwDirectionalLightmapElement) == LM_FLOATS<true> * sizeof(float), "lightmap element");

template <bool DIRECTIONAL>
__device__ __forceinline__ const float* lm_floats(const SurfaceKernelArgs& a)
{
	return DIRECTIONAL ? reinterpret_cast<const float*>(a.directional_lightmaps) : a.lightmaps;
}

template <bool DIRECTIONAL>
__device__ __forceinline__ Lm lm_load(const float* p)
{
	Lm e;
	if (DIRECTIONAL)
	{
		// 40-byte elements, 8-byte aligned in global and shared memory
		const float2* q = reinterpret_cast<const float2*>(p);
		const float2 q0 = q[0], q1 = q[1], q2 = q[2], q3 = q[3], q4 = q[4];
		e.amb[0] = q0.x;
		e.amb[1] = q0.y;
		e.amb[2] = q1.x;
		e.dir = mkv3(q1.y, q2.x, q2.y);
		e.dev = q3.x;
		e.col[0] = q3.y;
		e.col[1] = q4.x;
		e.col[2] = q4.y;
	}
	else
	{
		e.amb[0] = p[0];
		e.amb[1] = p[1];
		e.amb[2] = p[2];
	}
	return e;
}

// LightmapElementOps::mix(a, b, ratio) = a*ratio + b*(1-ratio), surfaces.rs:996-1071
template <bool DIRECTIONAL>
__device__ __forceinline__ Lm lm_mix(const Lm& a, const Lm& b, float ratio)
{
	const float omr = fsub(1.0f, ratio);
	Lm r;
#pragma unroll
	for (int i = 0; i < 3; ++i) r.amb[i] = mad2(a.amb[i], ratio, fmul(b.amb[i], omr));
	if (DIRECTIONAL)
	{
		r.dir = mkv3(mad2(a.dir.x, ratio, fmul(b.dir.x, omr)), mad2(a.dir.y, ratio, fmul(b.dir.y, omr)),
			mad2(a.dir.z, ratio, fmul(b.dir.z, omr)));
		r.dev = mad2(a.dev, ratio, fmul(b.dev, omr));
#pragma unroll
		for (int i = 0; i < 3; ++i) r.col[i] = mad2(a.col[i], ratio, fmul(b.col[i], omr));
	}
	return r;
}

__device__ __forceinline__ uint32_t wrap(int32_t a, uint32_t b)
{
	int32_t r = a % int32_t(b);
	return uint32_t(r < 0 ? r + int32_t(b) : r);
}
// rem_euclid by a texture side: a mask for powers of two (mask != ~0u), else the remainder
__device__ __forceinline__ uint32_t wrap_side(int32_t a, uint32_t b, uint32_t mask)
{
	return mask != ~0u ? uint32_t(a) & mask : wrap(a, b);
}
// n / d and n % d: the float estimate of the quotient (truncated product with the rounded reciprocal) is
// within one of it while the quotient stays below 2^22 (a surface's row), then corrected exactly
__device__ __forceinline__ void div_row(uint32_t n, uint32_t d, float inv_d, uint32_t& q, uint32_t& r)
{
	int32_t qi = int32_t(__fmul_rz(float(n), inv_d));
	int32_t ri = int32_t(n) - qi * int32_t(d);
	if (ri < 0)
	{
		--qi;
		ri += int32_t(d);
	}
	else if (ri >= int32_t(d))
	{
		++qi;
		ri -= int32_t(d);
	}
	q = uint32_t(qi);
	r = uint32_t(ri);
}

// cube_shadow_map_side_fetch (light.rs:235-258): 1 in light, 0 in shadow.
__device__ __forceinline__ float cube_side_fetch(const unsigned long long* side, uint32_t size, float x, float y, float z)
{
	const float ONE_MINUS_EPS = 1.0f - 1.0f / 65536.0f;
	const float size_f = float(size);
	const float depth = inv_fast(fmaxf(z, MIN_POSITIVE_VALUE));
	const float half_depth = fmul(0.5f, depth);
	const float u_f = fmul(fminf(fmaxf(fadd(fmul(x, half_depth), 0.5f), 0.0f), ONE_MINUS_EPS), size_f);
	const float v_f = fmul(fminf(fmaxf(fadd(fmul(y, half_depth), 0.5f), 0.0f), ONE_MINUS_EPS), size_f);
	const uint32_t u = __float2uint_rz(u_f), v = __float2uint_rz(v_f); // in [0, size)
	return depth >= __uint_as_float(uint32_t(__ldg(side + u + v * size))) ? 1.0f : 0.0f; // the texel's f32 bits
}

// projector_shadow_map_fetch (light.rs:261-294): 0 behind the projector or outside its map.
__device__ __forceinline__ float projector_fetch(const SurfaceKernelArgs& a, const SwLightShadow& m, V3 vec)
{
	const float z = v3dot(mkv3(m.basis_z[0], m.basis_z[1], m.basis_z[2]), vec);
	if (z <= 0.0f) return 0.0f;
	const float depth = inv_fast(z);
	const float half_depth = fmul(0.5f, depth);
	const float size_f = float(m.size);
	const float u_f = fmul(mad2(v3dot(mkv3(m.basis_x[0], m.basis_x[1], m.basis_x[2]), vec), half_depth, 0.5f), size_f);
	const float v_f = fmul(mad2(v3dot(mkv3(m.basis_y[0], m.basis_y[1], m.basis_y[2]), vec), half_depth, 0.5f), size_f);
	if (u_f < 0.0f || v_f < 0.0f || u_f >= size_f || v_f >= size_f) return 0.0f;
	const uint32_t u = __float2uint_rz(u_f), v = __float2uint_rz(v_f); // in [0, size)
	return depth >= __uint_as_float(uint32_t(__ldg(a.shadow_texels + m.offset + u + v * m.size))) ? 1.0f : 0.0f;
}

// get_light_shadow_factor / cube_shadow_map_fetch (light.rs:185-233) for `to_light` = light - point.
__device__ __forceinline__ float light_shadow_factor(const SurfaceKernelArgs& a, uint32_t light, V3 to_light)
{
	if (!a.shadows || light >= a.num_shadows) return 1.0f;
	const SwLightShadow m = a.shadows[light];
	if (m.kind == SW_SHADOW_PROJECTOR) return projector_fetch(a, m, to_light);
	if (m.kind != SW_SHADOW_CUBE) return 1.0f;
	const uint64_t side_texels = uint64_t(m.size) * m.size;
	const unsigned long long* maps = a.shadow_texels + m.offset;
	const float ax = fabsf(to_light.x), ay = fabsf(to_light.y), az = fabsf(to_light.z);
	if (ax >= ay && ax >= az)
		return to_light.x >= 0.0f ? cube_side_fetch(maps + 1 * side_texels, m.size, -to_light.y, to_light.z, ax)
								  : cube_side_fetch(maps + 0 * side_texels, m.size, to_light.y, to_light.z, ax);
	if (ay >= ax && ay >= az)
		return to_light.y >= 0.0f ? cube_side_fetch(maps + 3 * side_texels, m.size, to_light.x, to_light.z, ay)
								  : cube_side_fetch(maps + 2 * side_texels, m.size, -to_light.x, to_light.z, ay);
	return to_light.z >= 0.0f ? cube_side_fetch(maps + 5 * side_texels, m.size, -to_light.x, to_light.y, az)
							  : cube_side_fetch(maps + 4 * side_texels, m.size, -to_light.x, -to_light.y, az);
}

// The fields of a SurfaceGpu that a texel's shading reads, loaded as 16-byte words. (The lightmap's are read where
// they are needed: together they do not fit the registers.)
struct Surf
{
	V3 start_pos, u, v, normal, u_norm, v_norm;
	uint64_t tex_offset;
	uint32_t tex_w, tex_h, flags;
	int32_t tc0, tc1;
	uint32_t num_lights;
	const SurfaceGpu* g;
};
__device__ __forceinline__ Surf load_surf(const SurfaceGpu* g)
{
	static_assert(offsetof(SurfaceGpu, tex_offset) == 80 && offsetof(SurfaceGpu, tex_h) == 96 && offsetof(SurfaceGpu, lm_offset) == 112 &&
			offsetof(SurfaceGpu, inv_scale) == 72,
		"SurfaceGpu layout");
	const float4* f = reinterpret_cast<const float4*>(g);
	const float4 a = f[0], b = f[1], c = f[2], d = f[3], e = f[4];
	const uint4* w = reinterpret_cast<const uint4*>(g);
	const uint4 t = w[5], q = w[6];
	Surf s;
	s.start_pos = mkv3(a.x, a.y, a.z);
	s.u = mkv3(a.w, b.x, b.y);
	s.v = mkv3(b.z, b.w, c.x);
	s.normal = mkv3(c.y, c.z, c.w);
	s.u_norm = mkv3(d.x, d.y, d.z);
	s.v_norm = mkv3(d.w, e.x, e.y);
	s.tex_offset = uint64_t(t.x) | (uint64_t(t.y) << 32);
	s.tex_w = t.w;
	s.tex_h = q.x;
	s.flags = q.y;
	s.tc0 = int32_t(q.z);
	s.tc1 = int32_t(q.w);
	s.num_lights = g->num_lights;
	s.g = g;
	return s;
}

// Line entries of one surface row, by the warp (`s` the same in every lane): the vertical mixes of lightmap rows lv
// and lv + 1 at ratio kv for the columns [lu0, lu1 + 1] that texels [u0, u1] of row v read, as consecutive floats
// at `line`. Returns their number.
__device__ __forceinline__ uint32_t build_line(const SurfaceKernelArgs& a, const SurfaceGpu& s, uint32_t v, uint32_t u0, uint32_t u1, float* line,
	uint32_t lane)
{
	constexpr uint32_t F = LM_FLOATS<true>;
	const uint32_t base_v = v + s.lm_shift1;
	const uint32_t lu0 = (u0 + s.lm_shift0) >> s.lm_log2, lu1 = (u1 + s.lm_shift0) >> s.lm_log2;
	const float kv = mad2(float(base_v & ((1u << s.lm_log2) - 1u)), s.inv_scale, s.k_shift);
	const float omr = fsub(1.0f, kv);
	const float* row0 = lm_floats<true>(a) + (uint64_t(s.lm_offset) + uint64_t(base_v >> s.lm_log2) * s.lm_width + lu0) * F;
	const float* row1 = row0 + uint64_t(s.lm_width) * F;
	const uint32_t n = (lu1 - lu0 + 2) * F;
	for (uint32_t i = lane; i < n; i += 32) line[i] = mad2(__ldg(row1 + i), kv, fmul(__ldg(row0 + i), omr));
	return n;
}

// The texel's lightmap element (surfaces.rs:504-513): the horizontal mix of its two line entries.
__device__ __forceinline__ Lm mix_line(const SurfaceGpu& s, const float* line, uint32_t u, uint32_t u0)
{
	constexpr uint32_t F = LM_FLOATS<true>;
	const uint32_t base_u = u + s.lm_shift0;
	const float ku = mad2(float(base_u & ((1u << s.lm_log2) - 1u)), s.inv_scale, s.k_shift);
	const float* e = line + ((base_u >> s.lm_log2) - ((u0 + s.lm_shift0) >> s.lm_log2)) * F;
	return lm_mix<true>(lm_load<true>(e + F), lm_load<true>(e), ku);
}

// The same element for a single texel: both line entries built for it alone.
template <bool DIRECTIONAL>
__device__ __forceinline__ Lm lightmap_sample_once(const SurfaceKernelArgs& a, const SurfaceGpu& s, uint32_t u, uint32_t v)
{
	constexpr uint32_t F = LM_FLOATS<DIRECTIONAL>;
	const uint32_t log2 = s.lm_log2;
	const uint32_t mask = (1u << log2) - 1u;
	const uint32_t base_v = v + s.lm_shift1;
	const float kv = mad2(float(base_v & mask), s.inv_scale, s.k_shift);
	const uint32_t base_u = u + s.lm_shift0;
	const float ku = mad2(float(base_u & mask), s.inv_scale, s.k_shift);
	const float* row0 = lm_floats<DIRECTIONAL>(a) + (uint64_t(s.lm_offset) + uint64_t(base_v >> log2) * s.lm_width + (base_u >> log2)) * F;
	const float* row1 = row0 + uint64_t(s.lm_width) * F;
	const Lm line0 = lm_mix<DIRECTIONAL>(lm_load<DIRECTIONAL>(row1), lm_load<DIRECTIONAL>(row0), kv);
	const Lm line1 = lm_mix<DIRECTIONAL>(lm_load<DIRECTIONAL>(row1 + F), lm_load<DIRECTIONAL>(row0 + F), kv);
	return lm_mix<DIRECTIONAL>(line1, line0, ku);
}

// Lighting of one texel (surfaces.rs:515-842) with its lightmap element `l` (when the surface has a
// lightmap); returns the ColorVec before conversion.
template <bool DIRECTIONAL>
__device__ __forceinline__ CV shade_texel(const SurfaceKernelArgs& a, const Surf& s, uint64_t texel, uint32_t u,
	uint32_t v, V3 cam, const Lm& l)
{
	const uint32_t tex_flags = s.flags & 7u;
	const bool use_normal_map = (tex_flags & SW_TEX_HAS_NORMAL_MAP) != 0;
	const int spec = (tex_flags & SW_TEX_HAS_NON_ONE_ROUGHNESS) ? ((tex_flags & SW_TEX_IS_METAL) ? 2 : 1) : 0;

	const V3 bnormal = s.normal;
	const V3 pos = v3sma(s.u, float(u), v3sma(s.v, float(v), s.start_pos));

	V3 tn = mkv3(0.0f, 0.0f, 1.0f);
	float rough = 0.0f;
	const int32_t packed = int32_t(uint32_t(texel >> 32));
	if (use_normal_map)
	{
		tn = mkv3(fmul(float(int32_t(uint32_t(packed) << 24) >> 24), NORMAL_UNPACK_SCALE),
			fmul(float(int32_t(uint32_t(packed) << 16) >> 24), NORMAL_UNPACK_SCALE),
			fmul(float(int32_t(uint32_t(packed) << 8) >> 24), NORMAL_UNPACK_SCALE));
		rough = fmul(float(packed >> 24), NORMAL_UNPACK_SCALE);
	}
	else if (spec != 0)
		rough = fmul(float(packed >> 24), NORMAL_UNPACK_SCALE);

	CV albedo = cv_zero(); // total_light_albedo_modulated
	CV direct = cv_zero(); // total_light_direct
	if (s.flags & SW_SG_LIGHTMAP)
	{
		if (spec == 0)
		{
			albedo = cv_rgb(l.amb, 1.0f);
			if (DIRECTIONAL)
			{
				float dot = use_normal_map ? fmaxf(v3dot(l.dir, tn), 0.0f) : l.dir.z;
				albedo = cv_sma(cv_rgb(l.col, 0.0f), dot, albedo);
			}
		}
		else
		{
			const V3 u_norm = s.u_norm, v_norm = s.v_norm;
			const V3 normal = use_normal_map ? tn : mkv3(0.0f, 0.0f, 1.0f);
			const V3 to_cam = v3sub(cam, pos);
			const V3 to_cam_ts = mkv3(v3dot(to_cam, u_norm), v3dot(to_cam, v_norm), v3dot(to_cam, bnormal));
			const float ndot = v3dot(to_cam_ts, normal);
			const V3 refl = v3sub(v3scale(normal, fmul(2.0f, ndot)), to_cam_ts);
			const float refl_len2 = fmaxf(v3dot(refl, refl), MIN_POSITIVE_VALUE);
			const float angle_cos = fmaxf(fmul(ndot, inv_sqrt_fast(refl_len2)), 0.0f);
			const float sk = specular_k(spec, fresnel_factor_base(angle_cos), rough);
			const float omsk = fsub(1.0f, sk);
			const CV constant = cv_rgb(l.amb, 0.0f);
			albedo = cv_scale(constant, omsk);
			direct = cv_scale(constant, sk);
			albedo.a = 1.0f;
			if (DIRECTIONAL)
			{
				const float dir_len2 = v3dot(l.dir, l.dir);
				const float dir_len = fmul(dir_len2, inv_sqrt_fast(dir_len2));
				const float rl_cos = fmul(v3dot(refl, l.dir), inv_sqrt_fast(fmul(refl_len2, dir_len2)));
				const float inv_rc = fmaxf(inv_fast(fadd(rough, l.dev)), 0.75f);
				const float si = specular_intensity(rl_cos, inv_rc);
				const CV dcol = cv_rgb(l.col, 0.0f);
				if (spec == 1)
				{
					const float di = fmaxf(v3dot(l.dir, tn), 0.0f);
					albedo = cv_sma(dcol, fmul(di, omsk), albedo);
					direct = cv_sma(dcol, fmul(fmul(si, sk), dir_len), direct);
				}
				else
				{
					const float sf = fmul(si, dir_len);
					albedo = cv_sma(dcol, fmul(omsk, sf), albedo);
					direct = cv_sma(dcol, fmul(sk, sf), direct);
				}
			}
		}
	}

	if (s.num_lights > 0)
	{
		V3 normal = bnormal;
		if (use_normal_map)
		{
			const V3 u_norm = s.u_norm, v_norm = s.v_norm;
			normal = mkv3(mad2(tn.x, u_norm.x, mad2(tn.y, v_norm.x, fmul(tn.z, bnormal.x))),
				mad2(tn.x, u_norm.y, mad2(tn.y, v_norm.y, fmul(tn.z, bnormal.y))),
				mad2(tn.x, u_norm.z, mad2(tn.y, v_norm.z, fmul(tn.z, bnormal.z))));
		}
		V3 refl = mkv3(0.0f, 0.0f, 0.0f);
		float refl_len2 = 1.0f;
		float sk = 0.0f, inv_rough = 0.0f;
		if (spec != 0)
		{
			const V3 to_cam = v3sub(cam, pos);
			const float ndot = v3dot(to_cam, normal);
			refl = v3sub(v3scale(normal, fmul(2.0f, ndot)), to_cam);
			refl_len2 = fmaxf(v3dot(refl, refl), MIN_POSITIVE_VALUE);
			const float angle_cos = fmaxf(fmul(ndot, inv_sqrt_fast(refl_len2)), 0.0f);
			sk = specular_k(spec, fresnel_factor_base(angle_cos), rough);
			inv_rough = inv_fast(rough);
		}
		for (uint32_t li = 0; li < s.num_lights; ++li)
		{
			const SwLight& L = a.lights[s.g->lights[li]];
			const V3 to_light = v3sub(mkv3(L.position[0], L.position[1], L.position[2]), pos);
			const float tl_len2 = fmaxf(v3dot(to_light, to_light), MIN_POSITIVE_VALUE);
			const float sdf = fmul(light_shadow_factor(a, s.g->lights[li], to_light), fmaxf(fsub(inv_fast(tl_len2), L.inv_square_radius), 0.0f));
			// A factor of 0 (the texel lies outside the light's radius or in its shadow) adds zeros, unless a factor beside
			// it is infinite or NaN. Within these bounds none is: the diffuse cosine is below 1e27, the specular one below
			// 1e36, its intensity at most the roughness' reciprocal (127 or infinite); the light's colour is finite. Such a
			// light is left here: 512 colour32 surfaces with six lights each, most of them out of reach, take 62 us without
			// this, 23 of them for lights, and 55 with it. (A bound on the texel's values alone would be hoisted out of the loop into a register
			// too many, and so would the test before the shadow's: 1.5% of the time of batches without lights.)
			if (sdf == 0.0f && tl_len2 > 1e-18f && tl_len2 < 1e18f && fabsf(v3dot(normal, to_light)) < 1e18f)
			{
				const float len2 = fmul(refl_len2, tl_len2);
				if (fabsf(v3dot(refl, to_light)) < 1e18f && len2 > 1e-36f && len2 < 1e36f && fabsf(fmul(inv_rough, tl_len2)) < 1e36f) continue;
			}
			float di = 0.0f;
			if (spec != 2) di = fmaxf(fmul(v3dot(normal, to_light), inv_sqrt_fast(tl_len2)), 0.0f);
			float si = 0.0f;
			if (spec != 0)
				si = specular_intensity(fmul(v3dot(refl, to_light), inv_sqrt_fast(fmul(refl_len2, tl_len2))), inv_rough);
			const CV lc = cv_rgb(L.color, 0.0f);
			if (spec == 0)
				albedo = cv_sma(lc, fmul(di, sdf), albedo);
			else if (spec == 1)
			{
				albedo = cv_sma(lc, fmul(fmul(di, fsub(1.0f, sk)), sdf), albedo);
				direct = cv_sma(lc, fmul(fmul(si, sk), sdf), direct);
			}
			else
			{
				const float sisdf = fmul(si, sdf);
				albedo = cv_sma(lc, fmul(fsub(1.0f, sk), sisdf), albedo);
				direct = cv_sma(lc, fmul(sk, sisdf), direct);
			}
		}
	}

	CV result = cv_mul(cv_from_c32(uint32_t(texel)), albedo);
	if (spec != 0) result = cv_sma(direct, 255.0f, result);
	return result;
}

template <class P>
__device__ __forceinline__ typename P::T emissive_mix(const SurfaceKernelArgs& a, const SurfaceGpu& s, uint32_t u,
	uint32_t v, typename P::T dst, bool additive)
{
	const uint32_t sv = wrap_side(s.tc1 + int32_t(v), s.em_h, s.em_mask[1]);
	const uint32_t su = wrap_side(s.tc0 + int32_t(u), s.em_w, s.em_mask[0]);
	const uint32_t texel = __ldg(a.emissive_pixels + s.em_offset + uint64_t(sv) * s.em_w + su);
	const CI t = ci_from_c32(texel);
	CI m{{wmul(t.v[0], s.em_light[0]) >> 8, wmul(t.v[1], s.em_light[1]) >> 8, wmul(t.v[2], s.em_light[2]) >> 8, 0}};
	if (!additive) return P::from_ci(m);
	const CI d = P::to_ci(dst);
#pragma unroll
	for (int i = 0; i < 4; ++i) m.v[i] = wadd(m.v[i], d.v[i]);
	return P::from_ci(m);
}

// Surface of texel t: the largest i with prefix[i] <= t, by the whole warp (32 probes a round).
__device__ __forceinline__ uint32_t find_surface(const uint64_t* prefix, uint32_t n, uint64_t t, uint32_t lane)
{
	uint32_t lo = 0; // prefix[lo] <= t < prefix[lo + n]
	while (n > 1)
	{
		const uint32_t step = (n + 31) >> 5;
		const uint32_t i = lane * step;
		const uint32_t below = __popc(__ballot_sync(0xFFFFFFFFu, i < n && __ldg(prefix + lo + i) <= t)); // >= 1: lane 0
		const uint32_t k = (below - 1) * step;
		lo += k;
		n = min(step, n - k);
	}
	return lo;
}

// Bound by issue (78% of the slots): exact, unfused f32 shading and integer indexing, 534 instructions per 32 texels.
// One launch over 4,096 surfaces of 4x4 to 512x512 texels (43.9 M texels, directional lightmaps, half of the
// materials specular, colour64): 764 us, 57 Gtexel/s; 1,119 us and 628 instructions with two lightmap entries per
// texel from global memory and a serial search per 32 texels. Four blocks per SM (64 registers, 44 bytes spilled):
// three are 8% slower, five 24% (spills).
template <class P, bool DIRECTIONAL>
__global__ void __launch_bounds__(256, 4) surf_build_kernel(SurfaceKernelArgs a, uint32_t runs)
{
	typedef typename P::T T;
	// two rows' entries of 32 texels, at least one texel apart
	__shared__ __align__(16) float s_line[8][DIRECTIONAL ? 34 * LM_FLOATS<true> : 1];
	T* arena = static_cast<T*>(a.arena);
	const uint64_t total = a.counts ? a.counts->total_texels : a.total_work;
	const V3 cam = a.cam_pos_dev ? mkv3(a.cam_pos_dev[0], a.cam_pos_dev[1], a.cam_pos_dev[2])
								 : mkv3(a.cam_pos[0], a.cam_pos[1], a.cam_pos[2]);
	const uint32_t num_surfaces = a.counts ? a.counts->num_surfaces : a.num_surfaces;
	const uint64_t stride = uint64_t(gridDim.x) * blockDim.x * runs;
	const uint32_t lane = threadIdx.x & 31u;
	float* line = s_line[threadIdx.x >> 5];
	for (uint64_t first = a.work_begin + (uint64_t(blockIdx.x) * blockDim.x + (threadIdx.x & ~31u)) * runs; first < total; first += stride)
	{
		uint32_t si = find_surface(a.work_prefix, num_surfaces, first, lane);
		uint64_t begin = __ldg(a.work_prefix + si), next = __ldg(a.work_prefix + si + 1);
#pragma unroll 1
		for (uint32_t run = 0; run < runs; ++run)
		{
			const uint64_t t = first + run * 32 + lane;
			const bool active = t < total;
			const uint32_t mask = __ballot_sync(0xFFFFFFFFu, active);
			if (!mask) break;
			if (active && next <= t)
			{
				do
				{
					++si;
					begin = next;
					next = __ldg(a.work_prefix + si + 1);
				} while (next <= t);
			}
			const SurfaceGpu* g = a.surfaces + si;
			const uint32_t local = uint32_t(t - begin);
			uint32_t u = 0, v = 0;
			if (active) div_row(local, g->width, g->inv_width, v, u);
			// the run's surface rows: row 0 is the first lane's, row 1 the first other one (a row's lanes are
			// neighbours: its last texel is its first plus its lanes)
			bool together = false;
			uint32_t row1 = 0, u0 = 0, u1 = 0, line1 = 0;
			if constexpr (DIRECTIONAL)
			{
				const uint32_t si0 = __shfl_sync(0xFFFFFFFFu, si, 0), v0 = __shfl_sync(0xFFFFFFFFu, v, 0);
				const uint32_t row0 = __ballot_sync(0xFFFFFFFFu, active && si == si0 && v == v0);
				const uint32_t rest = mask & ~row0;
				const uint32_t lane1 = rest ? uint32_t(__ffs(int(rest))) - 1u : 0u;
				const uint32_t si1 = __shfl_sync(0xFFFFFFFFu, si, lane1), v1 = __shfl_sync(0xFFFFFFFFu, v, lane1);
				row1 = __ballot_sync(0xFFFFFFFFu, ((rest >> lane) & 1u) && si == si1 && v == v1);
				together = rest == row1;
				u0 = __shfl_sync(0xFFFFFFFFu, u, 0);
				u1 = __shfl_sync(0xFFFFFFFFu, u, lane1);
				if (together)
				{
					const SurfaceGpu& s0 = a.surfaces[si0];
					__syncwarp(); // the last run's entries have been read
					if (s0.flags & SW_SG_LIGHTMAP) line1 = build_line(a, s0, v0, u0, u0 + __popc(row0) - 1, line, lane);
					if (row1)
					{
						const SurfaceGpu& s1 = a.surfaces[si1];
						if (s1.flags & SW_SG_LIGHTMAP) build_line(a, s1, v1, u1, u1 + __popc(row1) - 1, line + line1, lane);
					}
					__syncwarp();
				}
			}
			if (!active) continue;
			const Surf s = load_surf(g);
			const uint32_t flags = s.flags;
			T out = T(0);
			const bool diffuse_layer = (flags & SW_SG_DIFFUSE) != 0;
			if (diffuse_layer)
			{
				const uint2 masks = *reinterpret_cast<const uint2*>(g->tex_mask);
				const uint32_t sv = wrap_side(s.tc1 + int32_t(v), s.tex_h, masks.y);
				const uint32_t su = wrap_side(s.tc0 + int32_t(u), s.tex_w, masks.x);
				const uint64_t texel =
					__ldg(reinterpret_cast<const unsigned long long*>(a.texels) + s.tex_offset + uint64_t(sv) * s.tex_w + su);
				Lm l;
				if (flags & SW_SG_LIGHTMAP)
				{
					const bool second = (row1 >> lane) & 1u;
					if (DIRECTIONAL && together)
						l = mix_line(*g, second ? line + line1 : line, u, second ? u1 : u0);
					else
						l = lightmap_sample_once<DIRECTIONAL>(a, *g, u, v);
				}
				out = P::from_cv(shade_texel<DIRECTIONAL>(a, s, texel, u, v, cam, l));
			}
			if (flags & SW_SG_EMISSIVE) out = emissive_mix<P>(a, *g, u, v, out, diffuse_layer);
			arena[g->out_offset + local] = out;
		}
	}
	pdl_trigger(); // the tile pass may be scheduled (it waits for this grid before reading the arena)
}

template <class P, bool DIRECTIONAL>
void launch_build(const SurfaceKernelArgs& args, unsigned blocks, uint32_t runs, cudaStream_t stream)
{
	surf_build_kernel<P, DIRECTIONAL><<<blocks, 256, 0, stream>>>(args, runs);
}

} // namespace

int launch_surface_build(const SurfaceKernelArgs& args, uint32_t pixel_format, int num_sms, int blocks_per_sm, cudaStream_t stream,
	uint64_t work_hint, uint32_t texels_per_thread)
{
	const uint64_t work = args.counts ? work_hint : args.total_work - args.work_begin;
	if (work == 0 && !args.counts) return 0;
	const uint64_t runs = surface_runs(texels_per_thread, work, num_sms);
	uint64_t blocks_needed = (work + 256 * runs - 1) / (256 * runs);
	if (args.counts && blocks_needed < uint64_t(num_sms)) blocks_needed = uint64_t(num_sms);
	// At most blocks_per_sm blocks per SM (several waves of resident blocks); large batches stride.
	const uint64_t blocks_max = uint64_t(num_sms) * uint64_t(blocks_per_sm);
	const unsigned blocks = unsigned(std::min(blocks_needed, blocks_max));
	const uint32_t r = uint32_t(runs);
	if (pixel_format == SW_PIXEL_C64)
		args.directional ? launch_build<PixC64, true>(args, blocks, r, stream) : launch_build<PixC64, false>(args, blocks, r, stream);
	else
		args.directional ? launch_build<PixC32, true>(args, blocks, r, stream) : launch_build<PixC32, false>(args, blocks, r, stream);
	return int(cudaGetLastError());
}

} // namespace swgpu
