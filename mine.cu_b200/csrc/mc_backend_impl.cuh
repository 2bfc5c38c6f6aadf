// mc_backend_impl.cuh - the environment step for one numerics mode.
//
// Included by exactly two translation units:
//   mc_fast.cu  (MC_NUMERICS_FAST=1, nvcc --use_fast_math): calls the same
//               CUDA math functions as the reference build, in the same op
//               order, so results match the reference bit for bit;
//   mc_ieee.cu  (MC_NUMERICS_FAST=0, -fmad=false): IEEE-754 ops and the trig
//               of mc_ieee_math.h, so results match the CPU checker bit for bit.
// MC_NS names the namespace so both back ends link into one library.
//
// Semantics follow the reference's src/kernels.cu; every device function
// cites the lines it restates.  Two launch forms share these functions:
//   plain : one kernel per reference kernel, in the reference's order;
//   fused : two kernels per step, the agents (a thread per env) and the
//           images (a persistent grid; a warp or a team of warps per env).
#pragma once
#include <cuda_runtime.h>
#include <cuda_fp16.h>
#include <stdint.h>
#include <algorithm>
#include <type_traits>
#include <utility>
#include "mc_internal.h"
#include "mc_ieee_math.h"
#include "mc_philox.h"

#ifndef MC_NS
#error "define MC_NS before including mc_backend_impl.cuh"
#endif

namespace MC_NS {

constexpr int8_t AIR = -1, GRASS = 0, DIRT = 1, OAKLOG = 3, LEAVES = 4, BRICK = 8,
                 COBBLESTONE = 9, PLANKS = 10, BEDROCK = 12;

// Colour tables: the reference's BLOCK_COLORS / SKY_COLOR (kernels.cu:27-44)
// and the pre-rounded BLOCK_COLORS_U8 / SKY_COLOR_U8 (kernels.cu:479-495).
__constant__ float c_rgb[13][3] = {
    {0.30f, 0.65f, 0.20f}, {0.55f, 0.35f, 0.20f}, {0.50f, 0.50f, 0.50f}, {0.55f, 0.40f, 0.25f},
    {0.20f, 0.55f, 0.15f}, {0.90f, 0.85f, 0.60f}, {0.20f, 0.40f, 0.80f}, {0.85f, 0.90f, 0.95f},
    {0.70f, 0.35f, 0.30f}, {0.40f, 0.40f, 0.40f}, {0.75f, 0.60f, 0.40f}, {0.95f, 0.95f, 0.98f},
    {0.15f, 0.15f, 0.15f}};
__constant__ float c_sky[3] = {0.53f, 0.81f, 0.92f};
__constant__ uint8_t c_rgb8[13][3] = {
    {76, 166, 51}, {140, 89, 51}, {127, 127, 127}, {140, 102, 64}, {51, 140, 38},
    {229, 217, 153}, {51, 102, 204}, {217, 229, 242}, {178, 89, 76}, {102, 102, 102},
    {191, 153, 102}, {242, 242, 250}, {38, 38, 38}};
__constant__ uint8_t c_sky8[3] = {135, 206, 235};

// ---------------------------------------------------------------------------
// Numerics policy
// ---------------------------------------------------------------------------
// Arithmetic is written with explicit single-rounding ops so that the
// compiler cannot contract or reorder it differently in different contexts
// (kernel shape, basic blocks, hoisting):
//   mul/add/sub  one IEEE rounding each (never fused);
//   mad(a,b,c)   ref_fast: one fused multiply-add, exactly where the
//                reference build's compiler fuses (determined by comparing
//                outputs with the reference's kernels on millions of inputs);
//                ieee: a*b rounded, then + c rounded (the CPU checker's order).
#if MC_NUMERICS_FAST
struct N {
    static __device__ __forceinline__ float mad(float a, float b, float c) { return __fmaf_rn(a, b, c); }
    // a/b - 1 and 1 - a/b: the build turns the division into a*(1/b) with an
    // approximate reciprocal and fuses it with the +-1
    static __device__ __forceinline__ float div_sub1(float a, float b) { return __fmaf_rn(a, __fdividef(1.0f, b), -1.0f); }
    static __device__ __forceinline__ float one_sub_div(float a, float b) { return __fmaf_rn(-a, __fdividef(1.0f, b), 1.0f); }
    static __device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
    static __device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
    static __device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }
    // a / b as the build computes it (a times the approximate reciprocal of
    // b), with the reciprocal passed in so repeated divisors share it
    static __device__ __forceinline__ float rcp_of(float b) { return __fdividef(1.0f, b); }
    static __device__ __forceinline__ float div_r(float a, float b, float rcp_b) { (void)b; return __fmul_rn(a, rcp_b); }
    static __device__ __forceinline__ float sin(float x) { return sinf(x); }
    static __device__ __forceinline__ float cos(float x) { return cosf(x); }
    static __device__ __forceinline__ float tan(float x) { return tanf(x); }
    static __device__ __forceinline__ void sincos_i(float x, float* s, float* c) { __sincosf(x, s, c); }
    static __device__ __forceinline__ float div(float a, float b) { return a / b; }
    static __device__ __forceinline__ float sqrt(float x) { return sqrtf(x); }
    static __device__ __forceinline__ float rsqrt(float x) { return rsqrtf(x); }
};
#else
struct N {
    static __device__ __forceinline__ float mad(float a, float b, float c) { return __fadd_rn(__fmul_rn(a, b), c); }
    static __device__ __forceinline__ float div_sub1(float a, float b) { return __fsub_rn(__fdiv_rn(a, b), 1.0f); }
    static __device__ __forceinline__ float one_sub_div(float a, float b) { return __fsub_rn(1.0f, __fdiv_rn(a, b)); }
    static __device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
    static __device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
    static __device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }
    static __device__ __forceinline__ float rcp_of(float b) { (void)b; return 0.0f; }
    static __device__ __forceinline__ float div_r(float a, float b, float rcp_b) { (void)rcp_b; return __fdiv_rn(a, b); }
    static __device__ __forceinline__ float sin(float x) { return mc_ieee_sinf(x); }
    static __device__ __forceinline__ float cos(float x) { return mc_ieee_cosf(x); }
    static __device__ __forceinline__ float tan(float x) { return mc_ieee_tanf(x); }
    static __device__ __forceinline__ void sincos_i(float x, float* s, float* c) { mc_ieee_sincosf(x, s, c); }
    static __device__ __forceinline__ float div(float a, float b) { return __fdiv_rn(a, b); }
    static __device__ __forceinline__ float sqrt(float x) { return __fsqrt_rn(x); }
    static __device__ __forceinline__ float rsqrt(float x) { return __fdiv_rn(1.0f, __fsqrt_rn(x)); }
};
#endif

// ---------------------------------------------------------------------------
// Bounds checks of the debug build (MC_CHECK_BOUNDS=1)
// ---------------------------------------------------------------------------
// In the debug build every voxel, shared-memory world, table and observation
// index is checked against its buffer before the access.  A failed check
// skips the access (a voxel read returns air) and records the first
// violation (site, index, limit) and a count in g_bounds, which
// bounds_report() reads and clears; the step kernels also set
// MC_KERR_BOUNDS in their env's error word.  Nothing traps.  The normal
// build compiles every check to nothing.
#ifndef MC_CHECK_BOUNDS
#define MC_CHECK_BOUNDS 0
#endif
#if MC_CHECK_BOUNDS
__device__ int32_t g_bounds[4];  // violations, first site (MC_SITE_*), first index, its limit
__device__ __noinline__ void bounds_fail(long long i, long long n, int site) {
    if (atomicAdd(&g_bounds[0], 1) == 0) {
        g_bounds[1] = site;
        g_bounds[2] = (int32_t)i;
        g_bounds[3] = (int32_t)n;
    }
}
__device__ __forceinline__ bool in_bounds(long long i, long long n, int site) {
    if (i >= 0 && i < n) return true;
    bounds_fail(i, n, site);
    return false;
}
// A step kernel's exit: a violation anywhere is also reported in the env's error word.
__device__ __forceinline__ void bounds_to_flags(int32_t* flags) {
    if (*(volatile int32_t*)&g_bounds[0]) atomicCAS(&flags[MC_FLAG_ERROR], MC_KERR_NONE, MC_KERR_BOUNDS);
}
#else
__device__ __forceinline__ constexpr bool in_bounds(long long, long long, int) { return true; }
__device__ __forceinline__ void bounds_to_flags(int32_t*) {}
#endif

// ---------------------------------------------------------------------------
// Agent step
// ---------------------------------------------------------------------------
struct Dec {
    float fwd, strafe, dyaw, dpitch, speed;
    bool jump, brk, place;
};

// decode_actions_kernel (kernels.cu:1459-1504)
__device__ __forceinline__ Dec decode_buttons(const int8_t b[8], float l0, float l1, float sprint_mult) {
    Dec d;
    d.fwd = N::sub((float)b[0], (float)b[1]);
    d.strafe = N::sub((float)b[3], (float)b[2]);
    d.dyaw = l0;
    d.dpitch = l1;
    d.jump = (b[4] != 0);
    d.brk = (b[5] != 0);
    d.place = (b[6] != 0);
    d.speed = (b[0] && b[7]) ? sprint_mult : 1.0f;
    return d;
}

// Actions of one env group: discrete actions, or buttons + look.
struct ActionSrc {
    const uint8_t* actions;
    const int8_t* buttons;
    const float* look;
};
__device__ __forceinline__ void load_action_from(const ActionSrc& a, float look_delta, long long i, int8_t b[8],
                                                 float& l0, float& l1) {
    if (a.actions) {
        float lk[2];
        mc_discrete_to_buttons(a.actions[i], look_delta, b, lk);
        l0 = lk[0];
        l1 = lk[1];
    } else {
#pragma unroll
        for (int k = 0; k < 8; ++k) b[k] = a.buttons[i * 8 + k];
        l0 = a.look[i * 2 + 0];
        l1 = a.look[i * 2 + 1];
    }
}


struct Agent {
    float x, y, z, vx, vy, vz, yaw, pitch;
    bool og;
};

__device__ __forceinline__ Agent load_agent(const mc_kp& p, long long i) {
    Agent a;
    a.x = p.positions[i * 3 + 0];
    a.y = p.positions[i * 3 + 1];
    a.z = p.positions[i * 3 + 2];
    a.vx = p.velocities[i * 3 + 0];
    a.vy = p.velocities[i * 3 + 1];
    a.vz = p.velocities[i * 3 + 2];
    a.yaw = p.yaws[i];
    a.pitch = p.pitches[i];
    a.og = p.on_ground[i] != 0;
    return a;
}

__device__ __forceinline__ void store_agent(const mc_kp& p, long long i, const Agent& a) {
    p.positions[i * 3 + 0] = a.x;
    p.positions[i * 3 + 1] = a.y;
    p.positions[i * 3 + 2] = a.z;
    p.velocities[i * 3 + 0] = a.vx;
    p.velocities[i * 3 + 1] = a.vy;
    p.velocities[i * 3 + 2] = a.vz;
    p.yaws[i] = a.yaw;
    p.pitches[i] = a.pitch;
    p.on_ground[i] = a.og ? 1 : 0;
}

// physics_kernel (kernels.cu:1511-1584): rotate, walk, gravity, clamp to the
// flat ground at world_y/4 and to [1, W-1] in x and z.  No voxel collision.
//   move_x = ((sin*fwd)*speed)*dt + ((cos*str)*walk)*dt   (the build fuses the strafe product)
//   move_z = ((cos*fwd)*speed)*dt - ((sin*str)*walk)*dt   (the build fuses the forward product)
//   vel_y += gravity*dt;  y += vel_y*dt                   (both fused)
__device__ __forceinline__ void physics(Agent& a, const Dec& d, const mc_kp& p, float& sin_yaw, float& cos_yaw) {
    a.yaw = N::add(a.yaw, d.dyaw);
    float new_pitch = N::add(a.pitch, d.dpitch);
    a.pitch = fminf(fmaxf(new_pitch, -1.56f), 1.56f);
    cos_yaw = N::cos(a.yaw);  // of the new yaw: the interaction's and the camera's too
    sin_yaw = N::sin(a.yaw);
    float fwd = d.fwd, str = d.strafe;
    float speed = N::mul(p.walk_speed, d.speed);
    float fx_ = N::mul(N::mul(N::mul(sin_yaw, fwd), speed), p.dt);
    float move_x = N::mad(N::mul(N::mul(cos_yaw, str), p.walk_speed), p.dt, fx_);
    float sz_ = N::mul(N::mul(N::mul(sin_yaw, str), p.walk_speed), p.dt);
    float move_z = N::mad(N::mul(N::mul(cos_yaw, fwd), speed), p.dt, -sz_);
    float vel_y = a.vy;
    if (d.jump && a.og) vel_y = p.jump_vel;
    vel_y = N::mad(p.gravity, p.dt, vel_y);
    float new_x = N::add(a.x, move_x);
    float new_y = N::mad(vel_y, p.dt, a.y);
    float new_z = N::add(a.z, move_z);
    float ground_y = (float)(p.wy / 4);
    if (new_y <= ground_y) {
        new_y = ground_y;
        vel_y = 0.0f;
        a.og = true;
    } else {
        a.og = false;
    }
    float margin = 1.0f;
    new_x = fminf(fmaxf(new_x, margin), N::sub((float)p.wx, margin));
    new_z = fminf(fmaxf(new_z, margin), N::sub((float)p.wz, margin));
    a.x = new_x;
    a.y = new_y;
    a.z = new_z;
    a.vy = vel_y;
}

// reset_kernel (kernels.cu:1760-1786)
__device__ __forceinline__ void reset_agent(Agent& a, const mc_kp& p) {
    a.x = p.spawn_x;
    a.y = p.spawn_y;
    a.z = p.spawn_z;
    a.vx = 0.0f;
    a.vy = 0.0f;
    a.vz = 0.0f;
    a.yaw = 0.0f;
    a.pitch = 0.0f;
    a.og = false;
}

// episode_check_kernel (kernels.cu:1954-1968) and the Python rule of
// minecu/__init__.py:363-366.
__device__ __forceinline__ bool episode_done(const mc_kp& p, int32_t cnt) {
    if (p.episode_rule == 0) return p.has_limit && cnt >= p.episode_length;
    return p.episode_length > 0 && cnt >= p.episode_length;
}

// One interact sample k of raycast_interact_kernel (kernels.cu:1621-1653):
// the point at t = 0.1 + k * 4/32 along the view direction from the eye.
struct Sample {
    int idx;  // flat in-env voxel index, valid if inb
    bool inb;
};
__device__ __forceinline__ Sample interact_sample(int k, float eye_x, float eye_y, float eye_z,
                                                  float dir_x, float dir_y, float dir_z,
                                                  int wx, int wy, int wz) {
    float reach = 4.0f;
    float t = N::mad((float)k, reach / 32.0f, 0.1f);  // k/8 is exact: same value fused or not
    float px = N::mad(dir_x, t, eye_x);
    float py = N::mad(dir_y, t, eye_y);
    float pz = N::mad(dir_z, t, eye_z);
    int vx = (int)floorf(px);
    int vy = (int)floorf(py);
    int vz = (int)floorf(pz);
    Sample s;
    s.inb = (vx >= 0 && vx < wx && vy >= 0 && vy < wy && vz >= 0 && vz < wz);
    s.idx = vy * (wx * wz) + vx * wz + vz;
    return s;
}

__device__ __forceinline__ void interact_dir(const Agent& a, float& dx, float& dy, float& dz) {
    float cos_yaw = N::cos(a.yaw);
    float sin_yaw = N::sin(a.yaw);
    float cos_pitch = N::cos(a.pitch);
    float sin_pitch = N::sin(a.pitch);
    dx = N::mul(sin_yaw, cos_pitch);
    dy = sin_pitch;
    dz = N::mul(cos_yaw, cos_pitch);
}

__device__ __forceinline__ bool reward_hit(const mc_kp& p, int8_t blk) {
    int8_t target = (int8_t)p.target_block;
    return target < 0 || blk == target;
}

// raycast_interact_kernel (kernels.cu:1591-1680), one thread per env.
// Returns the in-env index written (-1 if none); *reward as the reference.
__device__ __forceinline__ int interact_seq(int8_t* w, const Agent& a, bool brk, bool place,
                                            const mc_kp& p, float* reward) {
    *reward = 0.0f;
    if (!brk && !place) return -1;
    float dx, dy, dz;
    interact_dir(a, dx, dy, dz);
    float eye_x = a.x, eye_y = N::add(a.y, 1.6f), eye_z = a.z;
    int prev = -1;
    for (int k = 0; k < 32; ++k) {
        Sample s = interact_sample(k, eye_x, eye_y, eye_z, dx, dy, dz, p.wx, p.wy, p.wz);
        if (s.inb && in_bounds(s.idx, (long long)p.wx * p.wy * p.wz, MC_SITE_INTERACT)) {
            int8_t blk = w[s.idx];
            if (blk >= 0) {
                if (brk) {
                    if (reward_hit(p, blk)) *reward = p.reward_value;
                    w[s.idx] = AIR;
                    return s.idx;
                } else if (place && prev >= 0) {
                    w[prev] = DIRT;
                    return prev;
                }
                return -1;
            }
            prev = s.idx;
        }
    }
    return -1;
}

// The same interaction for the agent kernel, one thread per env, in two parts:
// all 32 samples are loaded at once (independent loads: one memory latency
// instead of one per sample the sequential loop looks at), then judged.  The
// first in-bounds solid sample is the lowest set bit of `solid` and the
// placement voxel the highest in-bounds sample below it, which is what the
// sequential loop selects.
struct Look {
    float ex, ey, ez, dx, dy, dz;
    unsigned inb, solid;
};
__device__ __forceinline__ void look_samples(Look& l, const int8_t* w, const mc_kp& p) {
    int8_t blk[32];
    l.inb = 0;
    l.solid = 0;
#pragma unroll
    for (int k = 0; k < 32; ++k) {
        const Sample s = interact_sample(k, l.ex, l.ey, l.ez, l.dx, l.dy, l.dz, p.wx, p.wy, p.wz);
        const bool in = s.inb && in_bounds(s.idx, (long long)p.wx * p.wy * p.wz, MC_SITE_INTERACT);
        l.inb |= in ? 1u << k : 0u;
        blk[k] = in ? w[s.idx] : AIR;
    }
#pragma unroll
    for (int k = 0; k < 32; ++k) l.solid |= blk[k] >= 0 ? 1u << k : 0u;
}
// The samples of the envs `who` of a warp's 32, one lane per sample and four
// envs' loads in flight; lane i gets env i's.  Called by the whole warp.
__device__ __forceinline__ void look_together(Look& l, const int8_t* w, const mc_kp& p, unsigned who, int lane) {
    const long long wxyz = (long long)p.wx * p.wy * p.wz;
    while (who) {
        int src[4], blk[4];
        bool in[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            src[j] = __ffs(who) - 1;  // -1: none left
            who &= who - 1u;
            const int i = src[j] < 0 ? 0 : src[j];
            const Sample s = interact_sample(lane, __shfl_sync(0xffffffffu, l.ex, i), __shfl_sync(0xffffffffu, l.ey, i),
                                             __shfl_sync(0xffffffffu, l.ez, i), __shfl_sync(0xffffffffu, l.dx, i),
                                             __shfl_sync(0xffffffffu, l.dy, i), __shfl_sync(0xffffffffu, l.dz, i),
                                             p.wx, p.wy, p.wz);
            const int8_t* wi = (const int8_t*)__shfl_sync(0xffffffffu, (unsigned long long)w, i);
            in[j] = src[j] >= 0 && s.inb && in_bounds(s.idx, wxyz, MC_SITE_INTERACT);
            blk[j] = in[j] ? wi[s.idx] : (int)AIR;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const unsigned inb = __ballot_sync(0xffffffffu, in[j]), solid = __ballot_sync(0xffffffffu, blk[j] >= 0);
            if (lane == src[j]) {
                l.inb = inb;
                l.solid = solid;
            }
        }
    }
}
// Returns the in-env index written (-1 if none), *val the value written there.
__device__ __forceinline__ int interact_judge(const Look& l, int8_t* w, bool brk, const mc_kp& p, float* reward,
                                              int* val) {
    if (l.solid == 0u) return -1;
    const int first = __ffs(l.solid) - 1;
    const unsigned before = l.inb & ((1u << first) - 1u);
    if (!brk && before == 0u) return -1;
    const int k = brk ? first : 31 - __clz(before);
    const int idx = interact_sample(k, l.ex, l.ey, l.ez, l.dx, l.dy, l.dz, p.wx, p.wy, p.wz).idx;
    if (brk && reward_hit(p, w[idx])) *reward = p.reward_value;
    *val = brk ? AIR : DIRT;
    w[idx] = (int8_t)*val;
    return idx;
}

// ---------------------------------------------------------------------------
// Render: per-env camera constants
// ---------------------------------------------------------------------------
struct Cam {
    float eye_x, eye_y, eye_z;
    float fx, fy, fz, rx, rz, ux, uy, uz;  // forward, right (x, z), up
    float sy, cy, cp;                      // sin/cos yaw, cos pitch (TRIG ray pattern)
};

// Per-env constants of the DDA set-up: the eye's voxel and, per axis, the
// distance numerators to its upper and lower faces, (v+1) - eye and v - eye.
struct Dda0 {
    int vx, vy, vz;
    float nxp, nxm, nyp, nym, nzp, nzm;
};
__device__ __forceinline__ Dda0 dda0(const Cam& c) {
    Dda0 d;
    d.vx = (int)floorf(c.eye_x);
    d.vy = (int)floorf(c.eye_y);
    d.vz = (int)floorf(c.eye_z);
    d.nxp = N::sub((float)(d.vx + 1), c.eye_x);
    d.nxm = N::sub((float)d.vx, c.eye_x);
    d.nyp = N::sub((float)(d.vy + 1), c.eye_y);
    d.nym = N::sub((float)d.vy, c.eye_y);
    d.nzp = N::sub((float)(d.vz + 1), c.eye_z);
    d.nzm = N::sub((float)d.vz, c.eye_z);
    return d;
}

// Camera basis as the per-pixel code of render_kernel / _uint8 / _minimal /
// _fp16 / _fast computes it (kernels.cu:113-136): cosf/sinf of yaw/pitch.
// Pure function of the camera, so computing it once per env gives the bits
// every pixel of the reference computes.
__device__ __forceinline__ Cam cam_trig(float cx, float cy, float cz, float yaw, float pitch) {
    Cam c;
    c.eye_x = cx;
    c.eye_y = N::add(cy, 1.6f);
    c.eye_z = cz;
    float cos_yaw = N::cos(yaw);
    float sin_yaw = N::sin(yaw);
    float cos_pitch = N::cos(pitch);
    float sin_pitch = N::sin(pitch);
    c.fx = N::mul(sin_yaw, cos_pitch);
    c.fy = sin_pitch;
    c.fz = N::mul(cos_yaw, cos_pitch);
    c.rx = cos_yaw;
    c.rz = -sin_yaw;
    c.ux = N::mul(-sin_yaw, sin_pitch);
    c.uy = cos_pitch;
    c.uz = N::mul(-cos_yaw, sin_pitch);
    c.sy = sin_yaw;
    c.cy = cos_yaw;
    c.cp = cos_pitch;
    return c;
}

// Ray direction before normalisation, forward + u*right + v*up.  Where the
// reference computes the basis in the same kernel (TRIG: shaded, minimal,
// fp16) its compiler fuses the forward product: fma(v, up, fma(sin, cos,
// u*right)); where the basis is loaded (prebasis) it fuses u*right:
// fma(v, up, fma(u, right, forward)).
template <bool TRIG>
__device__ __forceinline__ void ray_dir(const Cam& c, float u, float v, float& x, float& y, float& z) {
    if (TRIG) {
        x = N::mad(v, c.ux, N::mad(c.sy, c.cp, N::mul(u, c.rx)));
        z = N::mad(v, c.uz, N::mad(c.cy, c.cp, N::mul(u, c.rz)));
    } else {
        x = N::mad(v, c.ux, N::mad(u, c.rx, c.fx));
        z = N::mad(v, c.uz, N::mad(u, c.rz, c.fz));
    }
    y = N::mad(v, c.uy, c.fy);
}

// |ray|^2 = fma(z, z, fma(y, y, x*x))
__device__ __forceinline__ float len2(float x, float y, float z) { return N::mad(z, z, N::mad(y, y, N::mul(x, x))); }

// precompute_camera_basis_kernel (kernels.cu:511-561), all 13 written words.
__device__ __forceinline__ void basis_compute(float cx, float cy, float cz, float yaw, float pitch,
                                              int width, int height, float fov, float out[13]) {
    float sin_yaw, cos_yaw, sin_pitch, cos_pitch;
    N::sincos_i(yaw, &sin_yaw, &cos_yaw);
    N::sincos_i(pitch, &sin_pitch, &cos_pitch);
    float fov_rad = N::mul(fov, 0.01745329f);
    float half_fov = N::tan(N::mul(fov_rad, 0.5f));
    float aspect = N::div((float)width, (float)height);
    out[0] = cx;
    out[1] = N::add(cy, 1.6f);
    out[2] = cz;
    out[3] = N::mul(sin_yaw, cos_pitch);
    out[4] = sin_pitch;
    out[5] = N::mul(cos_yaw, cos_pitch);
    out[6] = cos_yaw;
    out[7] = -sin_yaw;
    out[8] = N::mul(-sin_yaw, sin_pitch);
    out[9] = cos_pitch;
    out[10] = N::mul(-cos_yaw, sin_pitch);
    out[11] = N::mul(half_fov, aspect);
    out[12] = half_fov;
}

// scale_u / scale_v of precompute_camera_basis_kernel (kernels.cu:541-559);
// they do not depend on the camera.
__device__ __forceinline__ void prebasis_scales(int width, int height, float fov, float* su, float* sv) {
    float fov_rad = N::mul(fov, 0.01745329f);
    float half_fov = N::tan(N::mul(fov_rad, 0.5f));
    float aspect = N::div((float)width, (float)height);
    *su = N::mul(half_fov, aspect);
    *sv = half_fov;
}

__device__ __forceinline__ Cam cam_from_basis(const float* b) {
    Cam c;
    c.eye_x = b[0]; c.eye_y = b[1]; c.eye_z = b[2];
    c.fx = b[3]; c.fy = b[4]; c.fz = b[5];
    c.rx = b[6]; c.rz = b[7];
    c.ux = b[8]; c.uy = b[9]; c.uz = b[10];
    c.sy = 0.0f; c.cy = 0.0f; c.cp = 0.0f;  // unused by the prebasis ray pattern
    return c;
}

// Per-column u and per-row v of each family.  They depend only on the pixel
// coordinate and launch constants, so the fused kernel tabulates them.
// Shaded family: kernels.cu:129-134 (fov_rad = fov * 3.14159265 / 180).
__device__ __forceinline__ float u_shaded(int px, int width, int height, float fov) {
    float fov_rad = N::div(N::mul(fov, 3.14159265f), 180.0f);
    float aspect = N::div((float)width, (float)height);
    float half_fov = N::tan(N::mul(fov_rad, 0.5f));
    float a = N::div_sub1(N::mul(2.0f, N::add((float)px, 0.5f)), (float)width);
    return N::mul(N::mul(a, half_fov), aspect);
}
__device__ __forceinline__ float v_shaded(int py, int height, float fov) {
    float fov_rad = N::div(N::mul(fov, 3.14159265f), 180.0f);
    float half_fov = N::tan(N::mul(fov_rad, 0.5f));
    return N::mul(N::one_sub_div(N::mul(2.0f, N::add((float)py, 0.5f)), (float)height), half_fov);
}
// Minimal/fp16 family: kernels.cu:1029-1034 (fov_rad = fov * 0.01745329).
__device__ __forceinline__ float u_minimal(int px, int width, int height, float fov) {
    float fov_rad = N::mul(fov, 0.01745329f);
    float aspect = N::div((float)width, (float)height);
    float half_fov = N::tan(N::mul(fov_rad, 0.5f));
    float a = N::div_sub1(N::mul(2.0f, N::add((float)px, 0.5f)), (float)width);
    return N::mul(N::mul(a, half_fov), aspect);
}
__device__ __forceinline__ float v_minimal(int py, int height, float fov) {
    float fov_rad = N::mul(fov, 0.01745329f);
    float half_fov = N::tan(N::mul(fov_rad, 0.5f));
    return N::mul(N::one_sub_div(N::mul(2.0f, N::add((float)py, 0.5f)), (float)height), half_fov);
}
// Prebasis family: kernels.cu:616-617 (scales from the basis).
__device__ __forceinline__ float u_prebasis(int px, int width, float scale_u) {
    return N::mul(N::div_sub1(N::mul(2.0f, N::add((float)px, 0.5f)), (float)width), scale_u);
}
__device__ __forceinline__ float v_prebasis(int py, int height, float scale_v) {
    return N::mul(N::one_sub_div(N::mul(2.0f, N::add((float)py, 0.5f)), (float)height), scale_v);
}

// Voxel sources for the ray march.  at(idx, n): the voxel at idx of a world
// of n voxels (bounds-checked in the debug build).
struct VoxGlobal {
    const int8_t* w;
    __device__ __forceinline__ int8_t operator()(int idx) const { return w[idx]; }
    __device__ __forceinline__ int8_t at(int idx, int n) const {
        return in_bounds(idx, n, MC_SITE_MARCH_GLOBAL) ? w[idx] : (int8_t)-1;
    }
};
struct VoxLdg {  // read-only world (plain render kernels): the reference's __ldg path
    const int8_t* w;
    __device__ __forceinline__ int8_t operator()(int idx) const { return __ldg(w + idx); }
    __device__ __forceinline__ int8_t at(int idx, int n) const {
        return in_bounds(idx, n, MC_SITE_MARCH_GLOBAL) ? __ldg(w + idx) : (int8_t)-1;
    }
};
struct VoxShared {
    const int8_t* w;
    __device__ __forceinline__ int8_t operator()(int idx) const { return w[idx]; }
    __device__ __forceinline__ int8_t at(int idx, int n) const {
        return in_bounds(idx, n, MC_SITE_MARCH_SHARED) ? w[idx] : (int8_t)-1;
    }
};
struct Hit {
    int blk;    // block id, -1 for sky
    int face;   // -1 none, 0 x, 1 y, 2 z
    float t;    // entry distance of the hit voxel (shaded family only)
    int step_y; // sign of the ray's y (shaded shade rule)
};

#if MC_NUMERICS_FAST
#define MC_PTX_FTZ ".ftz"
#else
#define MC_PTX_FTZ ""
#endif

// Packed march over a world staged in shared memory (the packed form of
// shade_ray's branch-free march).  `packed` holds the voxel index in bits
// 18.. and three 6-bit in-box step counts that set bit 5 of their field when
// the ray leaves the box; p{x,y,z} move index and count of one axis.  Per
// iteration the axis of the reference's if / else-if / else choice
// (kernels.cu:239-255) is three compares whose predicates guard the index
// and distance updates directly (no selects), and the distance update comes
// after the voxel test, so at a hit tm still holds the entry distances the
// choice was made from: the caller recovers the axis and the distance t
// from them once per ray instead of carrying them through the loop.  The
// voxel is loaded before the exit test, so that one test covers both exits;
// the load of the step that leaves the box reads up to wx*wz bytes before or
// after the staged world, which the shared-memory layouts keep allocated
// (the value read there is not used).
// Returns the block hit (>= 0), or -1 when the ray left the box.
// The debug build's marches (below) also check every load address against
// `chk` (the staged world and one layer on either side: the march's own
// claim) and against the CTA's dynamic shared memory.
struct SmemRange {
    uint32_t lo, span;  // shared-memory addresses [lo, lo + span)
};
__device__ __forceinline__ SmemRange staged_range(uint32_t base, int wxz, int nvox) {
    return SmemRange{base - (uint32_t)wxz, (uint32_t)(nvox + 2 * wxz)};
}
#if MC_CHECK_BOUNDS
extern __shared__ __align__(16) uint8_t mc_dyn_smem[];
__device__ __forceinline__ SmemRange dyn_smem_range() {
    uint32_t n;
    asm volatile("mov.u32 %0, %%dynamic_smem_size;" : "=r"(n));
    return SmemRange{(uint32_t)__cvta_generic_to_shared(mc_dyn_smem), n};
}
// A failed check of a PTX march's load address a: which range it left.
__device__ __noinline__ void march_bounds_fail(uint32_t a, SmemRange chk, int site) {
    const SmemRange d = dyn_smem_range();
    if (a - d.lo >= d.span) bounds_fail((long long)a - d.lo, d.span, MC_SITE_MARCH_SMEM);
    else bounds_fail((long long)a - chk.lo, chk.span, site);
}
#endif

// The marches' number type: float, or binary16 for the fp16 family (held in 16
// bits; its adds and compares keep denormals, as the half intrinsics do).
// The axis of a step: x if tmx < tmy and tmx < tmz, else y if tmy < tmz, else
// z (binary16 compares have no second predicate output).
#define MC_F32_T MC_PTX_FTZ ".f32"
#define MC_F16_T ".f16"
#define MC_F32_AXIS                                          \
    "setp.lt" MC_F32_T " pa|pna, %1, %2;\n\t"              \
    "setp.lt.and" MC_F32_T " pbx|pzx, %1, %3, pa;\n\t"     \
    "setp.lt.and" MC_F32_T " pby|pzy, %2, %3, pna;\n\t"    \
    "or.pred pz, pzx, pzy;\n\t"
#define MC_F16_AXIS                                          \
    "setp.lt" MC_F16_T " pa, %1, %2;\n\t"                  \
    "not.pred pna, pa;\n\t"                               \
    "setp.lt.and" MC_F16_T " pbx, %1, %3, pa;\n\t"         \
    "setp.lt.and" MC_F16_T " pby, %2, %3, pna;\n\t"        \
    "or.pred pz, pbx, pby;\n\t"                           \
    "not.pred pz, pz;\n\t"
#if MC_CHECK_BOUNDS
#define MC_MARCH_PACKED(FT, CMP, C) \
    asm volatile( \
        "{\n\t" \
        ".reg .pred pa, pna, pbx, pzx, pby, pzy, pz, pq, pb1, pb2;\n\t" \
        ".reg .b32 ra, rc;\n\t" \
        "MC_CMARCH_LOOP:\n\t" \
        CMP \
        "@pbx add.s32 %4, %4, %6;\n\t" \
        "@pby add.s32 %4, %4, %7;\n\t" \
        "@pz add.s32 %4, %4, %8;\n\t" \
        "shr.s32 ra, %4, 18;\n\t" \
        "add.s32 ra, ra, %10;\n\t" \
        "sub.u32 rc, ra, %15;\n\t" \
        "setp.ge.u32 pb1, rc, %16;\n\t" \
        "sub.u32 rc, ra, %17;\n\t" \
        "setp.ge.u32 pb2, rc, %18;\n\t" \
        "or.pred pb1, pb1, pb2;\n\t" \
        "@pb1 mov.u32 %5, ra;\n\t" \
        "@pb1 bra MC_CMARCH_END;\n\t" \
        "ld.shared.s8 %0, [ra];\n\t" \
        "lop3.b32 ra, %4, %0, %9, 0xA2;\n\t" \
        "setp.ne.b32 pq, ra, 0;\n\t" \
        "@pq bra MC_CMARCH_END;\n\t" \
        "@pbx add.rn" FT " %1, %1, %11;\n\t" \
        "@pby add.rn" FT " %2, %2, %12;\n\t" \
        "@pz add.rn" FT " %3, %3, %13;\n\t" \
        "bra MC_CMARCH_LOOP;\n\t" \
        "MC_CMARCH_END:\n\t" \
        "}" \
        : "+r"(b), "+" C(tmx), "+" C(tmy), "+" C(tmz), "+r"(packed), "+r"(bad) \
        : "r"(px), "r"(py), "r"(pz), "n"(kGuard | (int)0x80000000u), "r"(world), C(tdx), C(tdy), C(tdz), \
          "n"(kGuard), "r"(chk.lo), "r"(chk.span), "r"(dyn.lo), "r"(dyn.span) \
        : "memory");
#else
// one test for both exits: a guard bit of the counts, or the sign bit clear in
// the voxel (a block); c & (a | ~b) = lut 0xA2
#define MC_MARCH_PACKED(FT, CMP, C) \
    asm volatile( \
        "{\n\t" \
        ".reg .pred pa, pna, pbx, pzx, pby, pzy, pz, pq;\n\t" \
        ".reg .b32 ra;\n\t" \
        "MC_MARCH_LOOP:\n\t" \
        CMP \
        "@pbx add.s32 %4, %4, %5;\n\t" \
        "@pby add.s32 %4, %4, %6;\n\t" \
        "@pz add.s32 %4, %4, %7;\n\t" \
        "shr.s32 ra, %4, 18;\n\t" \
        "add.s32 ra, ra, %9;\n\t" \
        "ld.shared.s8 %0, [ra];\n\t" \
        "lop3.b32 ra, %4, %0, %8, 0xA2;\n\t" \
        "setp.ne.b32 pq, ra, 0;\n\t" \
        "@pq bra MC_MARCH_DONE;\n\t" \
        "@pbx add.rn" FT " %1, %1, %10;\n\t" \
        "@pby add.rn" FT " %2, %2, %11;\n\t" \
        "@pz add.rn" FT " %3, %3, %12;\n\t" \
        "bra MC_MARCH_LOOP;\n\t" \
        "MC_MARCH_DONE:\n\t" \
        "}" \
        : "+r"(b), "+" C(tmx), "+" C(tmy), "+" C(tmz), "+r"(packed) \
        : "r"(px), "r"(py), "r"(pz), "n"(kGuard | (int)0x80000000u), "r"(world), C(tdx), C(tdy), C(tdz), \
          "n"(kGuard) \
        : "memory");
#endif

template <class T>
__device__ __forceinline__ int march_packed_shared(uint32_t world, int& packed, int px, int py, int pz, T& tmx, T& tmy,
                                                   T& tmz, T tdx, T tdy, T tdz, SmemRange chk = SmemRange{0u, 0u}) {
    constexpr int kGuard = (32 << 12) | (32 << 6) | 32;
    int b = -1;
#if MC_CHECK_BOUNDS
    const SmemRange dyn = dyn_smem_range();
    uint32_t bad = ~0u;
#else
    (void)chk;
#endif
    if constexpr (sizeof(T) == 4) {
        MC_MARCH_PACKED(MC_F32_T, MC_F32_AXIS, "f")
    } else {
        MC_MARCH_PACKED(MC_F16_T, MC_F16_AXIS, "h")
    }
#if MC_CHECK_BOUNDS
    if (bad != ~0u) {  // a load address outside its range: the load was skipped, the ray ends as sky
        march_bounds_fail(bad, chk, MC_SITE_MARCH_PACKED);
        return -1;
    }
#endif
    return (packed & kGuard) ? -1 : b;
}

// Where a ray going up from the eye's voxel (vx, vy, vz) can still meet a
// solid voxel, per quadrant q of the eye's column (bit 0: the x >= vx side,
// bit 1: the z >= vz side; each side includes the eye's own row): such a
// ray only visits voxels with y >= vy on its quadrant's sides, so once it
// is past the extreme x, the extreme z or the highest layer of the solid
// voxels there it meets none again and ends as sky, as the full march
// would.  One byte per quadrant: x = the largest x (x >= vx side) or the
// smallest (x <= vx side), z likewise, y = the highest layer + 1 (0: none).
struct UpBounds {
    uint32_t x, z, y;
};

// Bounds that cut nothing but the layers above ytop (every quadrant's x and
// z extremes at the box's faces).
__device__ __forceinline__ UpBounds up_none(int ytop) {
    return UpBounds{0xFF00FF00u, 0xFFFF0000u, (uint32_t)(min(max(ytop, -1), 254) + 1) * 0x01010101u};
}

// The highest solid layer at or above vy (-1: none), from the bounds: every
// solid voxel at or above the eye's layer lies in some quadrant.
__device__ __forceinline__ int up_top(const UpBounds& b) {
    return (int)max(max(b.y & 255u, (b.y >> 8) & 255u), max((b.y >> 16) & 255u, b.y >> 24)) - 1;
}

// In-box step counts of a march from the eye's voxel for ray sign
// combination k (bit 0: x >= 0, bit 1: y >= 0, bit 2: z >= 0): the steps
// left to each face of the box, cut for a ray going up by its quadrant's
// bounds; a count of -1 ends the ray (as sky) at its first step.  ylow: the
// lowest layer a ray may enter (0, or the ground-shortcut family's ground).
__device__ __forceinline__ void start_counts(int k, int vx, int vy, int vz, int wx, int wy, int wz, int ylow,
                                             const UpBounds& ub, int& cx, int& cy, int& cz) {
    const bool px = k & 1, py = k & 2, pz = k & 4;
    cx = px ? wx - 1 - vx : vx;
    cy = py ? wy - 1 - vy : vy - ylow;
    cz = pz ? wz - 1 - vz : vz;
    if (py) {
        const int sh = 8 * ((px ? 1 : 0) | (pz ? 2 : 0));
        const int xe = (ub.x >> sh) & 255, ze = (ub.z >> sh) & 255, yt = (int)((ub.y >> sh) & 255) - 1;
        cx = max(min(cx, px ? xe - vx : vx - xe), -1);
        cz = max(min(cz, pz ? ze - vz : vz - ze), -1);
        cy = max(min(cy, yt - vy), -1);
    }
}

// Start values of march_packed_shared for an env whose eye is in voxel
// (vx, vy, vz), one per sign combination k of the ray (bit 0: x >= 0, bit 1:
// y >= 0, bit 2: z >= 0): {packed index and counts, x, y and z increments}.
// Counts from start_counts (at least -1, at most 31).
__device__ __forceinline__ int4 packed_start(int k, int vx, int vy, int vz, int wx, int wy, int wz,
                                             int ylow, const UpBounds& ub) {
    const int sx = (k & 1) ? 1 : -1, sy = (k & 2) ? 1 : -1, sz = (k & 4) ? 1 : -1;
    const int wxz = wx * wz, idx = vy * wxz + vx * wz + vz;
    int cx, cy, cz;
    start_counts(k, vx, vy, vz, wx, wy, wz, ylow, ub, cx, cy, cz);
    return make_int4((idx << 18) | ((31 - cx) << 12) | ((31 - cy) << 6) | (31 - cz),
                     ((sx * wz) << 18) + (1 << 12), ((sy * wxz) << 18) + (1 << 6), (sz << 18) + 1);
}

// Counts of the split march: three 7-bit in-box step counts (z bits 0-6,
// x 7-13, y 14-20) that count up from 63 - (steps left) and set bit 6 of
// their field on leaving the box, and a 9-bit step count (bits 21-29) that
// sets its bit 8 when max_steps voxels have been stepped.  A count that
// starts at or above 64 (y of a ray going up from above `ytop`) ends the ray at
// its first step; clamping it to 126 keeps the carry out of the field.
constexpr int kSplitGuard = (1 << 6) | (1 << 13) | (1 << 20) | (1 << 29);
__device__ __forceinline__ int split_counts(int cx, int cy, int cz, int max_steps, int wx, int wy, int wz) {
    const int s0 = (max_steps > wx + wy + wz) ? 0 : 256 - max_steps;  // no ray takes more than wx+wy+wz steps
    return (63 - cz) | ((63 - cx) << 7) | ((63 - max(cy, -63)) << 14) | (s0 << 21);
}

// The march over a staged world of up to 64 voxels a side, any max_steps:
// the voxel's shared-memory address moves in one register and the counts
// (split_counts) in another, so a single mask tests every exit and the load
// needs no index arithmetic.  Axis choice, predicated updates and the
// distances left at a hit as in march_packed_shared.  Returns the block hit
// (>= 0), or -1 when the ray left the box or ran out of steps.
#if MC_CHECK_BOUNDS
#define MC_MARCH_SPLIT(FT, CMP, C) \
    asm volatile( \
        "{\n\t" \
        ".reg .pred pa, pna, pbx, pzx, pby, pzy, pz, pq, pb1, pb2;\n\t" \
        ".reg .b32 ra, rc;\n\t" \
        "MC_CSPLIT_LOOP:\n\t" \
        CMP \
        "@pbx add.s32 %4, %4, %7;\n\t" \
        "@pby add.s32 %4, %4, %8;\n\t" \
        "@pz add.s32 %4, %4, %9;\n\t" \
        "@pbx add.s32 %5, %5, %10;\n\t" \
        "@pby add.s32 %5, %5, %11;\n\t" \
        "@pz add.s32 %5, %5, %12;\n\t" \
        "sub.u32 rc, %4, %18;\n\t" \
        "setp.ge.u32 pb1, rc, %19;\n\t" \
        "sub.u32 rc, %4, %20;\n\t" \
        "setp.ge.u32 pb2, rc, %21;\n\t" \
        "or.pred pb1, pb1, pb2;\n\t" \
        "@pb1 mov.u32 %6, %4;\n\t" \
        "@pb1 bra MC_CSPLIT_END;\n\t" \
        "ld.shared.s8 %0, [%4];\n\t" \
        "lop3.b32 ra, %5, %0, %13, 0xA2;\n\t" \
        "setp.ne.b32 pq, ra, 0;\n\t" \
        "@pq bra MC_CSPLIT_END;\n\t" \
        "@pbx add.rn" FT " %1, %1, %14;\n\t" \
        "@pby add.rn" FT " %2, %2, %15;\n\t" \
        "@pz add.rn" FT " %3, %3, %16;\n\t" \
        "bra MC_CSPLIT_LOOP;\n\t" \
        "MC_CSPLIT_END:\n\t" \
        "}" \
        : "+r"(b), "+" C(tmx), "+" C(tmy), "+" C(tmz), "+r"(addr), "+r"(cnt), "+r"(bad) \
        : "r"(dax), "r"(day), "r"(daz), "n"((1 << 7) | (1 << 21)), "n"((1 << 14) | (1 << 21)), "n"(1 | (1 << 21)), \
          "n"(kSplitGuard | (int)0x80000000u), C(tdx), C(tdy), C(tdz), "n"(kSplitGuard), "r"(chk.lo), \
          "r"(chk.span), "r"(dyn.lo), "r"(dyn.span) \
        : "memory");
#else
#define MC_MARCH_SPLIT(FT, CMP, C) \
    asm volatile( \
        "{\n\t" \
        ".reg .pred pa, pna, pbx, pzx, pby, pzy, pz, pq;\n\t" \
        ".reg .b32 ra;\n\t" \
        "MC_SPLIT_LOOP:\n\t" \
        CMP \
        "@pbx add.s32 %4, %4, %6;\n\t" \
        "@pby add.s32 %4, %4, %7;\n\t" \
        "@pz add.s32 %4, %4, %8;\n\t" \
        "@pbx add.s32 %5, %5, %9;\n\t" \
        "@pby add.s32 %5, %5, %10;\n\t" \
        "@pz add.s32 %5, %5, %11;\n\t" \
        "ld.shared.s8 %0, [%4];\n\t" \
        "lop3.b32 ra, %5, %0, %12, 0xA2;\n\t" \
        "setp.ne.b32 pq, ra, 0;\n\t" \
        "@pq bra MC_SPLIT_DONE;\n\t" \
        "@pbx add.rn" FT " %1, %1, %13;\n\t" \
        "@pby add.rn" FT " %2, %2, %14;\n\t" \
        "@pz add.rn" FT " %3, %3, %15;\n\t" \
        "bra MC_SPLIT_LOOP;\n\t" \
        "MC_SPLIT_DONE:\n\t" \
        "}" \
        : "+r"(b), "+" C(tmx), "+" C(tmy), "+" C(tmz), "+r"(addr), "+r"(cnt) \
        : "r"(dax), "r"(day), "r"(daz), "n"((1 << 7) | (1 << 21)), "n"((1 << 14) | (1 << 21)), "n"(1 | (1 << 21)), \
          "n"(kSplitGuard | (int)0x80000000u), C(tdx), C(tdy), C(tdz), "n"(kSplitGuard) \
        : "memory");
#endif

template <class T>
__device__ __forceinline__ int march_split_shared(uint32_t addr, int& cnt, int dax, int day, int daz, T& tmx, T& tmy,
                                                  T& tmz, T tdx, T tdy, T tdz, SmemRange chk = SmemRange{0u, 0u}) {
    int b = -1;
#if MC_CHECK_BOUNDS
    const SmemRange dyn = dyn_smem_range();
    uint32_t bad = ~0u;
#else
    (void)chk;
#endif
    if constexpr (sizeof(T) == 4) {
        MC_MARCH_SPLIT(MC_F32_T, MC_F32_AXIS, "f")
    } else {
        MC_MARCH_SPLIT(MC_F16_T, MC_F16_AXIS, "h")
    }
#if MC_CHECK_BOUNDS
    if (bad != ~0u) {
        march_bounds_fail(bad, chk, MC_SITE_MARCH_SPLIT);
        return -1;
    }
#endif
    return (cnt & kSplitGuard) ? -1 : b;
}

// March from the eye's voxel (index idx, in-box steps left cx, cy, cz) through
// a world staged at shared address `base`: the packed form where the world
// is small and every ray leaves the box before max_steps, else the split form.
__device__ __forceinline__ int march_staged(uint32_t base, int idx, int cx, int cy, int cz, int dix, int diy, int diz,
                                           int wx, int wy, int wz, int max_steps, float& tmx, float& tmy, float& tmz,
                                           float tdx, float tdy, float tdz) {
    const SmemRange chk = staged_range(base, wx * wz, wx * wy * wz);
    if (max_steps > wx + wy + wz && mc_packed_world(wx, wy, wz)) {
        int packed = (idx << 18) | ((31 - cx) << 12) | ((31 - max(cy, -32)) << 6) | (31 - cz);
        return march_packed_shared(base, packed, (dix << 18) + (1 << 12), (diy << 18) + (1 << 6), (diz << 18) + 1,
                                   tmx, tmy, tmz, tdx, tdy, tdz, chk);
    }
    int cnt = split_counts(cx, cy, cz, max_steps, wx, wy, wz);
    return march_split_shared(base + idx, cnt, dix, diy, diz, tmx, tmy, tmz, tdx, tdy, tdz, chk);
}

// Whether a march can run on the staged copy: V is a shared-memory source
// (or one flagged as such) and the world fits the counts' 64-voxel range.
template <class V>
__device__ __forceinline__ bool staged_source(const V& vox, int wx, int wy, int wz) {
    if constexpr (std::is_same<V, VoxShared>::value) {
        return wx <= 64 && wy <= 64 && wz <= 64;
    } else {
        (void)vox; (void)wx; (void)wy; (void)wz;
        return false;
    }
}
// The shared-memory address of a staged source (0 for the others, which
// staged_source turns away).
template <class V>
__device__ __forceinline__ uint32_t staged_base(const V& vox) {
    if constexpr (std::is_same<V, VoxShared>::value) {
        return (uint32_t)__cvta_generic_to_shared(vox.w);
    } else {
        (void)vox;
        return 0u;
    }
}

// ray_intersects_aabb (kernels.cu:51-79) exit distance for a box [0, ws]^3
// given the precomputed numerators (0 - eye) and (ws - eye).
__device__ __forceinline__ float aabb_exit(float ix, float iy, float iz, float lo_x, float hi_x,
                                           float lo_y, float hi_y, float lo_z, float hi_z, float* t_entry) {
    float t1 = N::mul(lo_x, ix), t2 = N::mul(hi_x, ix);
    float t3 = N::mul(lo_y, iy), t4 = N::mul(hi_y, iy);
    float t5 = N::mul(lo_z, iz), t6 = N::mul(hi_z, iz);
    *t_entry = fmaxf(fmaxf(fminf(t1, t2), fminf(t3, t4)), fminf(t5, t6));
    return fminf(fminf(fmaxf(t1, t2), fmaxf(t3, t4)), fmaxf(t5, t6));
}

// Shaded ray: ray setup, AABB early-out and DDA of render_kernel /
// render_kernel_uint8 (kernels.cu:137-269) and, with FASTG, the ground
// shortcut of render_kernel_uint8_fast (kernels.cu:1378-1405).  The
// reference's cubic box [0, ws]^3 becomes [0,wx]x[0,wy]x[0,wz], which is the
// same arithmetic when the world is cubic.  `inside` is a per-env flag: eye
// strictly inside the box and view_distance >= 0;
// then the AABB test always passes (t_entry < 0 <= view_distance) and its
// exit distance is only computed if the march leaves the world.
// With `skip_first` (a per-env fact: the eye is inside the world, its voxel
// holds air, view_distance > 0 and max_steps >= 1, and for FASTG the eye is
// at or above the ground) the first loop iteration is known to advance
// without a hit, so its tests are skipped.
//
// With `sky_exit` (per env: `inside`, no ground shortcut, and the caller does
// not need the face and distance of sky pixels, only their colour) the march stops as soon as
// the ray leaves the box: voxel coordinates move monotonically, so a ray that
// left never re-enters, and the reference, which keeps stepping until it is
// past the exit distance, also ends it as sky.  The axis is then chosen with
// selects instead of branches, and the box is tracked with per-axis counts of
// the in-box steps left.  With `vd_safe` (per env: every in-box voxel is
// entered closer than view_distance) the march has no distance test.  In
// both, `ytop` (per env: no solid voxel above this layer) ends rays going up
// once they pass it, as sky.
template <bool FASTG, class V>
__device__ __forceinline__ Hit shade_ray(const Cam& c, const Dda0& d0, float u, float v, const V& vox, int wx, int wy,
                                         int wz, int max_steps, float vd, int gh, bool inside,
                                         bool skip_first = false, bool sky_exit = false, bool vd_safe = false,
                                         int ytop = 1 << 20) {
    float ray_x, ray_y, ray_z;
    ray_dir<true>(c, u, v, ray_x, ray_y, ray_z);
    float ray_len = N::sqrt(len2(ray_x, ray_y, ray_z));
    const float rl = N::rcp_of(ray_len);
    ray_x = N::div_r(ray_x, ray_len, rl);
    ray_y = N::div_r(ray_y, ray_len, rl);
    ray_z = N::div_r(ray_z, ray_len, rl);

    float ix = (ray_x != 0.0f) ? N::div(1.0f, ray_x) : 1e30f;
    float iy = (ray_y != 0.0f) ? N::div(1.0f, ray_y) : 1e30f;
    float iz = (ray_z != 0.0f) ? N::div(1.0f, ray_z) : 1e30f;
    float lo_x = N::sub(0.0f, c.eye_x), hi_x = N::sub((float)wx, c.eye_x);
    float lo_y = N::sub(0.0f, c.eye_y), hi_y = N::sub((float)wy, c.eye_y);
    float lo_z = N::sub(0.0f, c.eye_z), hi_z = N::sub((float)wz, c.eye_z);

    Hit h;
    h.step_y = (ray_y >= 0) ? 1 : -1;
    h.blk = AIR;
    h.face = -1;
    h.t = 0.0f;
    float t_exit = 0.0f;
    bool have_exit = false;
    if (!inside) {
        float t_entry;
        t_exit = aabb_exit(ix, iy, iz, lo_x, hi_x, lo_y, hi_y, lo_z, hi_z, &t_entry);
        have_exit = true;
        if (t_exit < 0 || t_entry > t_exit || t_entry > vd) return h;  // sky
    }
    int vx = d0.vx, vy = d0.vy, vz = d0.vz;
    int sx = (ray_x >= 0) ? 1 : -1;
    int sy = h.step_y;
    int sz = (ray_z >= 0) ? 1 : -1;
    float tdx = fabsf(ix), tdy = fabsf(iy), tdz = fabsf(iz);
    float tmx = N::mul((ray_x >= 0) ? d0.nxp : d0.nxm, ix);
    float tmy = N::mul((ray_y >= 0) ? d0.nyp : d0.nym, iy);
    float tmz = N::mul((ray_z >= 0) ? d0.nzp : d0.nzm, iz);
    float t = 0.0f;
    int face = -1;
    const int wxz = wx * wz;
    const int nvox = wxz * wy;  // for the debug build's checks
    // linear voxel index kept in step with (vx, vy, vz)
    int idx = vy * wxz + vx * wz + vz;
    const int dix = sx * wz, diy = sy * wxz, diz = sz;
    int step = 0;
    if constexpr (std::is_same<V, VoxShared>::value) {
        if (!FASTG && sky_exit && max_steps > 0 && wx <= 64 && wy <= 64 && wz <= 64) {
            // A staged world and the eye inside the box: the PTX marches.
            // They test view_distance once, at the hit: t never decreases
            // along the ray, so a first hit closer than view_distance is the
            // reference's hit, and a first hit at or beyond it means the
            // reference had already ended the ray as sky (its `t >= vd`
            // break); a ray that leaves the box or runs out of steps is sky
            // in both.
            int b = skip_first ? (int)AIR : (int)vox.at(idx, nvox);
            // a ray going up stops above ytop (no solid voxel lies higher): it ends as sky
            const int cx = (sx > 0) ? wx - 1 - vx : vx, cy = (sy > 0) ? min(wy - 1, ytop) - vy : vy,
                      cz = (sz > 0) ? wz - 1 - vz : vz;
            if (b < 0) {
                const uint32_t base = (uint32_t)__cvta_generic_to_shared(vox.w);
                if (vd_safe && max_steps > wx + wy + wz && mc_packed_world(wx, wy, wz)) {
                    // index and in-box counts in one register (march_packed_shared)
                    int packed = (idx << 18) | ((31 - cx) << 12) | ((31 - max(cy, -32)) << 6) | (31 - cz);
                    b = march_packed_shared(base, packed, (dix << 18) + (1 << 12), (diy << 18) + (1 << 6),
                                            (diz << 18) + 1, tmx, tmy, tmz, tdx, tdy, tdz,
                                            staged_range(base, wxz, nvox));
                } else {
                    int cnt = split_counts(cx, cy, cz, max_steps, wx, wy, wz);
                    b = march_split_shared(base + idx, cnt, dix, diy, diz, tmx, tmy, tmz, tdx, tdy, tdz, staged_range(base, wxz, nvox));
                }
                if (b >= 0) {
                    // the axis of the last step, chosen again from the same distances
                    const bool bx = tmx < tmy && tmx < tmz;
                    const bool by = !bx && tmy < tmz;
                    t = bx ? tmx : (by ? tmy : tmz);
                    face = bx ? 0 : (by ? 1 : 2);
                    if (t >= vd) b = AIR;
                }
            }
            h.blk = (b >= 0) ? b : AIR;
            h.face = face;
            h.t = t;
            return h;
        }
    }
    if (!FASTG && sky_exit && vd_safe && max_steps > 0) {
        // The same march with no distance test and no branch per axis: the
        // reference's if / else-if / else choice of axis (kernels.cu:239-255)
        // is made with selects, so lanes stepping different axes do not take
        // turns; one test per iteration ends the loop (hit, left the box, or
        // max_steps).  The eye's voxel is inside the box.
        int8_t b = AIR;
        if (!skip_first && max_steps > 0) b = vox.at(idx, nvox);
        bool lbx = false, lby = false, adv = false;
        // a ray going up stops above ytop (no solid voxel lies higher): it ends as sky
        int cx = (sx > 0) ? wx - 1 - vx : vx, cy = (sy > 0) ? min(wy - 1, ytop) - vy : vy,
            cz = (sz > 0) ? wz - 1 - vz : vz;
        if (max_steps > wx + wy + wz && wx <= 31 && wy <= 31 && wz <= 31 && wx * wy * wz < 8192) {
            // every ray leaves the box before max_steps: no step count.  (The exit
            // test comes before the load, so the layer beyond the box need not fit.)  The
            // voxel index and the three in-box counts share one register:
            // bits 18.. the index, three 6-bit fields below it counting up
            // from 31 - (steps left) to 32, whose bit 5 marks leaving the
            // box; one add moves both, one mask tests the exit.
            const int fx = 31 - cx, fy = 31 - max(cy, -32), fz = 31 - cz;
            int packed = (idx << 18) | (fx << 12) | (fy << 6) | fz;
            const int px = (dix << 18) + (1 << 12), py = (diy << 18) + (1 << 6), pz = (diz << 18) + 1;
            constexpr int kGuard = (32 << 12) | (32 << 6) | 32;
            while (b < 0) {
                const bool bx = tmx < tmy && tmx < tmz;
                const bool by = !bx && tmy < tmz;
                const bool bz = !bx && !by;
                t = bx ? tmx : (by ? tmy : tmz);
                // three adds (FMA pipe) instead of selecting the delta (ALU pipe,
                // the busier one); only the chosen axis keeps its sum
                const float nx = N::add(tmx, tdx), ny = N::add(tmy, tdy), nz = N::add(tmz, tdz);
                tmx = bx ? nx : tmx;
                tmy = by ? ny : tmy;
                tmz = bz ? nz : tmz;
                packed += bx ? px : (by ? py : pz);
                lbx = bx;
                lby = by;
                adv = true;
                if (packed & kGuard) break;
                b = vox.at(packed >> 18, nvox);
            }
        } else {
            while (b < 0 && max_steps > 0) {
                const bool bx = tmx < tmy && tmx < tmz;
                const bool by = !bx && tmy < tmz;
                const bool bz = !bx && !by;
                t = bx ? tmx : (by ? tmy : tmz);
                const float nx = N::add(tmx, tdx), ny = N::add(tmy, tdy), nz = N::add(tmz, tdz);
                tmx = bx ? nx : tmx;
                tmy = by ? ny : tmy;
                tmz = bz ? nz : tmz;
                cx -= bx ? 1 : 0;
                cy -= by ? 1 : 0;
                cz -= bz ? 1 : 0;
                idx += bx ? dix : (by ? diy : diz);
                lbx = bx;
                lby = by;
                adv = true;
                if ((cx | cy | cz) < 0 || ++step >= max_steps) break;
                b = vox.at(idx, nvox);
            }
        }
        if (adv) face = lbx ? 0 : (lby ? 1 : 2);
        h.blk = (b >= 0) ? (int)b : AIR;
        h.face = face;
        h.t = t;
        return h;
    }
    if (!FASTG && sky_exit && max_steps > 0) {
        // the same branch-free march with the distance test and the step
        // count in its single exit test (worlds whose far corners lie beyond
        // view_distance)
        int8_t b = AIR;
        if (!skip_first) b = vox.at(idx, nvox);
        bool lbx = false, lby = false, adv = false;
        // a ray going up stops above ytop (no solid voxel lies higher): it ends as sky
        int cx = (sx > 0) ? wx - 1 - vx : vx, cy = (sy > 0) ? min(wy - 1, ytop) - vy : vy,
            cz = (sz > 0) ? wz - 1 - vz : vz;
        while (b < 0) {
            const bool bx = tmx < tmy && tmx < tmz;
            const bool by = !bx && tmy < tmz;
            const bool bz = !bx && !by;
            t = bx ? tmx : (by ? tmy : tmz);
            const float nx = N::add(tmx, tdx), ny = N::add(tmy, tdy), nz = N::add(tmz, tdz);
            tmx = bx ? nx : tmx;
            tmy = by ? ny : tmy;
            tmz = bz ? nz : tmz;
            cx -= bx ? 1 : 0;
            cy -= by ? 1 : 0;
            cz -= bz ? 1 : 0;
            idx += bx ? dix : (by ? diy : diz);
            lbx = bx;
            lby = by;
            adv = true;
            if ((cx | cy | cz) < 0 || ++step >= max_steps || t >= vd) break;
            b = vox.at(idx, nvox);
        }
        if (adv) face = lbx ? 0 : (lby ? 1 : 2);
        h.blk = (b >= 0) ? (int)b : AIR;
        h.face = face;
        h.t = t;
        return h;
    }
    if (skip_first) {
        if (tmx < tmy && tmx < tmz) {
            t = tmx; tmx = N::add(tmx, tdx); vx += sx; idx += dix; face = 0;
        } else if (tmy < tmz) {
            t = tmy; tmy = N::add(tmy, tdy); vy += sy; idx += diy; face = 1;
        } else {
            t = tmz; tmz = N::add(tmz, tdz); vz += sz; idx += diz; face = 2;
        }
        step = 1;
    }
    for (; step < max_steps; ++step) {
        if (t >= vd) break;
        if (FASTG && vy < gh) {
            h.blk = (vy == gh - 1) ? GRASS : DIRT;
            break;
        }
        if ((unsigned)vx < (unsigned)wx && (unsigned)vy < (unsigned)wy && (unsigned)vz < (unsigned)wz) {
            int8_t b = vox.at(idx, nvox);
            if (b >= 0) {
                h.blk = b;
                break;
            }
        } else {
            if (!have_exit) {
                float t_entry;
                t_exit = aabb_exit(ix, iy, iz, lo_x, hi_x, lo_y, hi_y, lo_z, hi_z, &t_entry);
                have_exit = true;
            }
            if (t > t_exit) break;
        }
        if (tmx < tmy && tmx < tmz) {
            t = tmx; tmx = N::add(tmx, tdx); vx += sx; idx += dix; face = 0;
        } else if (tmy < tmz) {
            t = tmy; tmy = N::add(tmy, tdy); vy += sy; idx += diy; face = 1;
        } else {
            t = tmz; tmz = N::add(tmz, tdz); vz += sz; idx += diz; face = 2;
        }
    }
    h.face = face;
    h.t = t;
    return h;
}

// Every voxel of the box is entered closer than view_distance (with a margin
// far above the rounding of the DDA's accumulated distances), so the march's
// distance test cannot end a ray inside the box.
__device__ __forceinline__ bool box_within_view(const Cam& c, int wx, int wy, int wz, float vd) {
    const float dx = fmaxf(c.eye_x, (float)wx - c.eye_x);
    const float dy = fmaxf(c.eye_y, (float)wy - c.eye_y);
    const float dz = fmaxf(c.eye_z, (float)wz - c.eye_z);
    const float m = vd - 1.0f;
    return m > 0.0f && dx * dx + dy * dy + dz * dz < m * m;
}

__device__ __forceinline__ bool eye_inside(const Cam& c, int wx, int wy, int wz, float vd) {
    return c.eye_x > 0.0f && c.eye_x < (float)wx && c.eye_y > 0.0f && c.eye_y < (float)wy &&
           c.eye_z > 0.0f && c.eye_z < (float)wz && vd >= 0.0f;
}

// Which product each channel's c*shade*(1-fog) + sky*fog fuses in the
// reference build (measured against its kernels): float32 render_kernel
// fuses sky*fog for red only; render_kernel_uint8 for red and green;
// render_kernel_uint8_fast for red only (MC_FASTG_SKY).  Bit k = channel k.
enum { MC_COL_F32 = 0, MC_COL_U8 = 1, MC_COL_U8FAST = 2 };
#ifndef MC_FASTG_SKY
#define MC_FASTG_SKY 0x1
#endif
__device__ __forceinline__ int sky_fused_mask(int kind) {
    return kind == MC_COL_F32 ? 0x1 : (kind == MC_COL_U8 ? 0x3 : MC_FASTG_SKY);
}

// Shading and fog of the shaded family (kernels.cu:271-292, 446-469).
template <int KIND>
__device__ __forceinline__ void shade_rgb(const Hit& h, float vd, float rcp_vd, const float (*rgb)[3], const float* sky,
                                          float out[3]) {
    if (h.blk >= 0 && in_bounds(h.blk, 13, MC_SITE_TABLE)) {
        float r = rgb[h.blk][0], g = rgb[h.blk][1], b_col = rgb[h.blk][2];
        float shade = 1.0f;
        if (h.face == 0) shade = 0.8f;
        else if (h.face == 2) shade = 0.9f;
        else if (h.face == 1 && h.step_y < 0) shade = 0.6f;
        float fog = fminf(N::div_r(h.t, vd, rcp_vd), 1.0f);
        fog = N::mul(fog, fog);
        float omf = N::sub(1.0f, fog);
        const int m = sky_fused_mask(KIND);
        const float c3[3] = {r, g, b_col};
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            float cs = N::mul(c3[k], shade);
            out[k] = ((m >> k) & 1) ? N::mad(sky[k], fog, N::mul(cs, omf)) : N::mad(cs, omf, N::mul(sky[k], fog));
        }
    } else {
        out[0] = sky[0];
        out[1] = sky[1];
        out[2] = sky[2];
    }
}

// (uint8_t)(x * 255) for x*255 in [0, 256): adding 2^23 with round-toward-
// zero leaves trunc(x*255) in the low mantissa bits, which is the C++
// float-to-integer conversion without using the conversion unit.
__device__ __forceinline__ uint32_t to_u8(float x) {
    return __float_as_uint(__fadd_rz(N::mul(x, 255.0f), 8388608.0f)) & 0xffu;
}

// Flat ray of render_kernel_uint8_minimal / _prebasis / _smem
// (kernels.cu:1036-1097, 619-679): rsqrtf normalisation, no AABB, no fog,
// unsigned bounds test, non-cubic world.
// With `sky_exit` (per env: the eye's voxel is inside the world, and the
// caller needs only the colour of sky pixels) the march stops when the ray
// leaves the box, where the reference keeps stepping out-of-box voxels until
// max_steps: a ray that left never re-enters, so both end as sky.
template <bool TRIG, class V>
__device__ __forceinline__ Hit flat_ray(const Cam& c, const Dda0& d0, float u, float v, const V& vox, int wx, int wy,
                                        int wz, int max_steps, bool skip_first = false, bool sky_exit = false,
                                        int ytop = 1 << 20) {
    float ray_x, ray_y, ray_z;
    ray_dir<TRIG>(c, u, v, ray_x, ray_y, ray_z);
    float ray_len = N::rsqrt(len2(ray_x, ray_y, ray_z));
    ray_x = N::mul(ray_x, ray_len);
    ray_y = N::mul(ray_y, ray_len);
    ray_z = N::mul(ray_z, ray_len);
    int wxz = wx * wz;
    const int nvox = wxz * wy;  // for the debug build's checks
    int vx = d0.vx, vy = d0.vy, vz = d0.vz;
    int sx = (ray_x >= 0) ? 1 : -1;
    int sy = (ray_y >= 0) ? 1 : -1;
    int sz = (ray_z >= 0) ? 1 : -1;
    float ix = (ray_x != 0.0f) ? N::div(1.0f, ray_x) : 1e30f;
    float iy = (ray_y != 0.0f) ? N::div(1.0f, ray_y) : 1e30f;
    float iz = (ray_z != 0.0f) ? N::div(1.0f, ray_z) : 1e30f;
    float tdx = fabsf(ix), tdy = fabsf(iy), tdz = fabsf(iz);
    float tmx = N::mul((ray_x >= 0) ? d0.nxp : d0.nxm, ix);
    float tmy = N::mul((ray_y >= 0) ? d0.nyp : d0.nym, iy);
    float tmz = N::mul((ray_z >= 0) ? d0.nzp : d0.nzm, iz);
    Hit h;
    h.blk = AIR;
    h.face = -1;
    h.t = 0.0f;
    h.step_y = sy;
    int face = -1;
    int idx = vy * wxz + vx * wz + vz;
    const int dix = sx * wz, diy = sy * wxz, diz = sz;
    if (sky_exit && max_steps > 0 && staged_source(vox, wx, wy, wz)) {
        // the PTX marches over the staged world (as in shade_ray, no view distance)
        int b = skip_first ? (int)AIR : (int)vox.at(idx, nvox);
        if (b < 0) {
            // a ray going up stops above ytop (no solid voxel lies higher): it ends as sky
            const int cx = (sx > 0) ? wx - 1 - vx : vx, cy = (sy > 0) ? min(wy - 1, ytop) - vy : vy,
                      cz = (sz > 0) ? wz - 1 - vz : vz;
            b = march_staged(staged_base(vox), idx, cx, cy, cz, dix, diy, diz, wx, wy, wz, max_steps, tmx, tmy,
                                 tmz, tdx, tdy, tdz);
            if (b >= 0) {
                const bool bx = tmx < tmy && tmx < tmz;
                face = bx ? 0 : ((tmy < tmz) ? 1 : 2);
            }
        }
        h.blk = (b >= 0) ? b : AIR;
        h.face = face;
        return h;
    }
    if (sky_exit) {
        // branch-free axis choice as in shade_ray; one exit test per iteration
        int8_t b = AIR;
        int step = 0;
        if (!skip_first && max_steps > 0) b = vox.at(idx, nvox);
        while (b < 0 && max_steps > 0) {
            const bool bx = tmx < tmy && tmx < tmz;
            const bool by = !bx && tmy < tmz;
            const bool bz = !bx && !by;
            const float nx = N::add(tmx, tdx), ny = N::add(tmy, tdy), nz = N::add(tmz, tdz);
            tmx = bx ? nx : tmx;
            tmy = by ? ny : tmy;
            tmz = bz ? nz : tmz;
            vx += bx ? sx : 0;
            vy += by ? sy : 0;
            vz += bz ? sz : 0;
            idx += bx ? dix : (by ? diy : diz);
            face = bx ? 0 : (by ? 1 : 2);
            const bool out = (unsigned)vx >= (unsigned)wx || (unsigned)vy >= (unsigned)wy || (unsigned)vz >= (unsigned)wz;
            if (out || ++step >= max_steps) break;
            b = vox.at(idx, nvox);
        }
        h.blk = (b >= 0) ? (int)b : AIR;
        h.face = face;
        return h;
    }
    for (int step = 0; step < max_steps; ++step) {
        // skip_first: the eye's voxel is known to be air or outside the world
        if ((step > 0 || !skip_first) &&
            (unsigned)vx < (unsigned)wx && (unsigned)vy < (unsigned)wy && (unsigned)vz < (unsigned)wz) {
            int8_t b = vox.at(idx, nvox);
            if (b >= 0) {
                h.blk = b;
                break;
            }
        }
        if (tmx < tmy && tmx < tmz) {
            tmx = N::add(tmx, tdx); vx += sx; idx += dix; face = 0;
        } else if (tmy < tmz) {
            tmy = N::add(tmy, tdy); vy += sy; idx += diy; face = 1;
        } else {
            tmz = N::add(tmz, tdz); vz += sz; idx += diz; face = 2;
        }
    }
    h.face = face;
    return h;
}

// render_kernel_uint8_fp16 (kernels.cu:1176-1248): the DDA's t_max/t_delta
// in binary16 (inverse 65504 for a zero component).
template <class V>
__device__ __forceinline__ Hit fp16_ray(const Cam& c, const Dda0& d0, float u, float v, const V& vox, int wx, int wy,
                                        int wz, int max_steps) {
    float ray_x, ray_y, ray_z;
    ray_dir<true>(c, u, v, ray_x, ray_y, ray_z);
    float ray_len = N::rsqrt(len2(ray_x, ray_y, ray_z));
    ray_x = N::mul(ray_x, ray_len);
    ray_y = N::mul(ray_y, ray_len);
    ray_z = N::mul(ray_z, ray_len);
    int wxz = wx * wz;
    const int nvox = wxz * wy;  // for the debug build's checks
    int vx = d0.vx, vy = d0.vy, vz = d0.vz;
    int sx = (ray_x >= 0) ? 1 : -1;
    int sy = (ray_y >= 0) ? 1 : -1;
    int sz = (ray_z >= 0) ? 1 : -1;
    float ixf = (ray_x != 0.0f) ? N::div(1.0f, ray_x) : 65504.0f;
    float iyf = (ray_y != 0.0f) ? N::div(1.0f, ray_y) : 65504.0f;
    float izf = (ray_z != 0.0f) ? N::div(1.0f, ray_z) : 65504.0f;
    __half tdx = __float2half(fabsf(ixf));
    __half tdy = __float2half(fabsf(iyf));
    __half tdz = __float2half(fabsf(izf));
    __half tmx = __float2half(N::mul((ray_x >= 0) ? d0.nxp : d0.nxm, ixf));
    __half tmy = __float2half(N::mul((ray_y >= 0) ? d0.nyp : d0.nym, iyf));
    __half tmz = __float2half(N::mul((ray_z >= 0) ? d0.nzp : d0.nzm, izf));
    Hit h;
    h.blk = AIR;
    h.face = -1;
    h.t = 0.0f;
    h.step_y = sy;
    int face = -1;
    for (int step = 0; step < max_steps; ++step) {
        if ((unsigned)vx < (unsigned)wx && (unsigned)vy < (unsigned)wy && (unsigned)vz < (unsigned)wz) {
            int8_t b = vox.at(vy * wxz + vx * wz + vz, nvox);
            if (b >= 0) {
                h.blk = b;
                break;
            }
        }
        if (__hlt(tmx, tmy) && __hlt(tmx, tmz)) {
            tmx = __hadd(tmx, tdx); vx += sx; face = 0;
        } else if (__hlt(tmy, tmz)) {
            tmy = __hadd(tmy, tdy); vy += sy; face = 1;
        } else {
            tmz = __hadd(tmz, tdz); vz += sz; face = 2;
        }
    }
    h.face = face;
    return h;
}

__device__ __forceinline__ int16_t dbg_code(const Hit& h) { return (int16_t)((h.blk + 1) | ((h.face + 1) << 8)); }

// ---------------------------------------------------------------------------
// Plain form: one kernel per reference kernel
// ---------------------------------------------------------------------------
__device__ __forceinline__ void flag_any(int32_t* flags, bool v) {
    unsigned m = __ballot_sync(__activemask(), v);
    if (m && (threadIdx.x & 31) == (__ffs(m) - 1)) atomicOr(&flags[MC_FLAG_ANY_DONE], 1);
}

__global__ void k_episode_check(mc_kp p) {
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.B) return;
    bool done = p.ext_done ? (p.do_reset[i] != 0) : episode_done(p, p.step_count[i]);
    if (!p.ext_done) p.do_reset[i] = done ? 1 : 0;
    flag_any(p.flags, done);
}

__global__ void k_decode(mc_kp p) {
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.B) return;
    int8_t b[8];
    float l0, l1;
    load_action_from(ActionSrc{p.actions, p.buttons, p.look}, p.look_delta, i, b, l0, l1);
    Dec d = decode_buttons(b, l0, l1, p.sprint_mult);
    p.s_fwd[i] = d.fwd;
    p.s_strafe[i] = d.strafe;
    p.s_dyaw[i] = d.dyaw;
    p.s_dpitch[i] = d.dpitch;
    p.s_jump[i] = d.jump;
    p.s_brk[i] = d.brk;
    p.s_place[i] = d.place;
    p.s_speed[i] = d.speed;
}

__device__ __forceinline__ Dec load_dec(const mc_kp& p, long long i) {
    Dec d;
    d.fwd = p.s_fwd[i];
    d.strafe = p.s_strafe[i];
    d.dyaw = p.s_dyaw[i];
    d.dpitch = p.s_dpitch[i];
    d.jump = p.s_jump[i] != 0;
    d.brk = p.s_brk[i] != 0;
    d.place = p.s_place[i] != 0;
    d.speed = p.s_speed[i];
    return d;
}

__global__ void k_physics(mc_kp p) {
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.B) return;
    Agent a = load_agent(p, i);
    float sy, cy;
    physics(a, load_dec(p, i), p, sy, cy);
    p.positions[i * 3 + 0] = a.x;
    p.positions[i * 3 + 1] = a.y;
    p.positions[i * 3 + 2] = a.z;
    p.velocities[i * 3 + 1] = a.vy;
    p.yaws[i] = a.yaw;
    p.pitches[i] = a.pitch;
    p.on_ground[i] = a.og ? 1 : 0;
}

// break_only: raycast_break_kernel (kernels.cu:1687-1753), no placement.
__global__ void k_interact(mc_kp p, int break_only) {
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.B) return;
    Agent a = load_agent(p, i);
    bool brk = p.s_brk[i] != 0;
    bool place = break_only ? false : (p.s_place[i] != 0);
    float reward;
    long long wxyz = (long long)p.wx * p.wy * p.wz;
    int idx = interact_seq(p.voxels + i * wxyz, a, brk, place, p, &reward);
    p.rewards[i] = reward;
    if (p.dbg_interact) p.dbg_interact[i] = idx;
}

__global__ void k_reset(mc_kp p) {
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.B) return;
    if (p.do_reset[i]) {
        Agent a;
        reset_agent(a, p);
        store_agent(p, i, a);
    }
}

// episode_update_kernel (kernels.cu:1971-1986) == the Python counter update
// of minecu/__init__.py:435-436.
__global__ void k_episode_update(mc_kp p) {
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.B || p.ext_done) return;
    p.step_count[i] = p.do_reset[i] ? 1 : p.step_count[i] + 1;
}

// update_cameras_kernel (kernels.cu:2320-2335)
__global__ void k_cameras(mc_kp p) {
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.B) return;
    p.cameras[i * 5 + 0] = p.positions[i * 3 + 0];
    p.cameras[i * 5 + 1] = p.positions[i * 3 + 1];
    p.cameras[i * 5 + 2] = p.positions[i * 3 + 2];
    p.cameras[i * 5 + 3] = p.yaws[i];
    p.cameras[i * 5 + 4] = p.pitches[i];
}

__global__ void k_basis(mc_kp p) {
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.B) return;
    const float* cam = p.cameras + i * 5;
    float out[13];
    basis_compute(cam[0], cam[1], cam[2], cam[3], cam[4], p.W, p.H, p.fov, out);
#pragma unroll
    for (int k = 0; k < 13; ++k) p.basis[i * 14 + k] = out[k];
}

// Shaded render, one thread per pixel over B*H*W, as render_kernel /
// render_kernel_uint8 / render_kernel_uint8_fast (1-D grid, 128 threads).
template <bool FASTG, bool F32>
__global__ void __launch_bounds__(128) k_render_shaded(mc_kp p) {
    long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    long long hw = (long long)p.H * p.W;
    if (idx >= (long long)p.B * hw) return;
    long long b = idx / hw;
    int pix = (int)(idx - b * hw);
    int py = pix / p.W, px = pix - py * p.W;
    const float* cam = p.cameras + b * 5;
    Cam c = cam_trig(__ldg(cam + 0), __ldg(cam + 1), __ldg(cam + 2), __ldg(cam + 3), __ldg(cam + 4));
    bool inside = eye_inside(c, p.wx, p.wy, p.wz, p.vd);
    float u = u_shaded(px, p.W, p.H, p.fov);
    float v = v_shaded(py, p.H, p.fov);
    VoxLdg vox{p.voxels + b * (long long)p.wx * p.wy * p.wz};
    Hit h = shade_ray<FASTG>(c, dda0(c), u, v, vox, p.wx, p.wy, p.wz, p.max_steps, p.vd, p.gh, inside);
    float rgb[3];
    shade_rgb<F32 ? MC_COL_F32 : (FASTG ? MC_COL_U8FAST : MC_COL_U8)>(h, p.vd, N::rcp_of(p.vd), c_rgb, c_sky, rgb);
    if (F32) {
        float* o = (float*)p.obs + idx * 3;
        o[0] = rgb[0]; o[1] = rgb[1]; o[2] = rgb[2];
    } else {
        uint8_t* o = (uint8_t*)p.obs + idx * 3;
        o[0] = (uint8_t)to_u8(rgb[0]); o[1] = (uint8_t)to_u8(rgb[1]); o[2] = (uint8_t)to_u8(rgb[2]);
    }
    if (p.dbg_pixel) p.dbg_pixel[idx] = dbg_code(h);
}

// Flat render, one thread per pixel over B*H*W (minimal / fp16: per-pixel
// trig; prebasis: reads the [B,14] basis).  The reference launches the
// prebasis kernel on a 2-D grid (pixel blocks, env), which caps B at 65535;
// the per-pixel work is the same.
template <int FAM>
__global__ void __launch_bounds__(128) k_render_flat(mc_kp p) {
    long long hw = (long long)p.H * p.W;
    long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)p.B * hw) return;
    long long b = idx / hw;
    int pix = (int)(idx - b * hw);
    int py = pix / p.W, px = pix - py * p.W;
    Cam c;
    float u, v;
    if (FAM == MC_FAM_PREBASIS) {
        const float* bs = p.basis + b * 14;
        float bb[13];
#pragma unroll
        for (int k = 0; k < 13; ++k) bb[k] = __ldg(bs + k);
        c = cam_from_basis(bb);
        u = u_prebasis(px, p.W, bb[11]);
        v = v_prebasis(py, p.H, bb[12]);
    } else {
        const float* cam = p.cameras + b * 5;
        c = cam_trig(__ldg(cam + 0), __ldg(cam + 1), __ldg(cam + 2), __ldg(cam + 3), __ldg(cam + 4));
        u = u_minimal(px, p.W, p.H, p.fov);
        v = v_minimal(py, p.H, p.fov);
    }
    long long wxyz = (long long)p.wx * p.wy * p.wz;
    VoxLdg vox{p.voxels + b * wxyz};
    Hit h;
    const Dda0 d0 = dda0(c);
    if (FAM == MC_FAM_FP16) h = fp16_ray(c, d0, u, v, vox, p.wx, p.wy, p.wz, p.max_steps);
    else if (FAM == MC_FAM_PREBASIS) h = flat_ray<false>(c, d0, u, v, vox, p.wx, p.wy, p.wz, p.max_steps);
    else h = flat_ray<true>(c, d0, u, v, vox, p.wx, p.wy, p.wz, p.max_steps);
    long long o = (b * hw + pix);
    uint8_t* out = (uint8_t*)p.obs + o * 3;
    const uint8_t* col = (h.blk >= 0 && in_bounds(h.blk, 13, MC_SITE_TABLE)) ? c_rgb8[h.blk] : c_sky8;
    out[0] = col[0]; out[1] = col[1]; out[2] = col[2];
    if (p.dbg_pixel) p.dbg_pixel[o] = dbg_code(h);
}

// render_kernel_uint8_coalesced (kernels.cu:709-826): prebasis semantics over
// a [Y, X, Z, B] voxel layout, a warp = one pixel across 32 envs.
__global__ void __launch_bounds__(128) k_render_coalesced(const int8_t* vox, const float* basis, uint8_t* out,
                                                          int B, int ws, int W, int H, int max_steps) {
    int pix = blockIdx.x;
    int b = blockIdx.y * blockDim.x + threadIdx.x;
    if (pix >= H * W || b >= B) return;
    int py = pix / W, px = pix - py * W;
    float bb[13];
#pragma unroll
    for (int k = 0; k < 13; ++k) bb[k] = __ldg(basis + (long long)b * 14 + k);
    Cam c = cam_from_basis(bb);
    float u = u_prebasis(px, W, bb[11]);
    float v = v_prebasis(py, H, bb[12]);
    struct VoxYXZB {
        const int8_t* v;
        int B, b, ws;
        __device__ __forceinline__ int8_t operator()(int idx) const {
            // idx = y*ws*ws + x*ws + z  ->  [y][x][z][b]
            return __ldg(v + (long long)idx * B + b);
        }
        __device__ __forceinline__ int8_t at(int idx, int n) const {
            return in_bounds(idx, n, MC_SITE_MARCH_GLOBAL) ? (*this)(idx) : (int8_t)-1;
        }
    } acc{vox, B, b, ws};
    Hit h = flat_ray<false>(c, dda0(c), u, v, acc, ws, ws, ws, max_steps);
    const uint8_t* col = (h.blk >= 0 && in_bounds(h.blk, 13, MC_SITE_TABLE)) ? c_rgb8[h.blk] : c_sky8;
    uint8_t* o = out + ((long long)b * H * W + pix) * 3;
    o[0] = col[0]; o[1] = col[1]; o[2] = col[2];
}

// ---------------------------------------------------------------------------
// Fused form: shared-memory layout and helpers of the image kernels
// ---------------------------------------------------------------------------
// Shared memory layout (per CTA): u/v tables, colour tables, then per warp a
// pixel staging buffer, an mbarrier and (stage=1) one world.  A warp marches
// one tile of tile_w x (32/tile_w) pixels per iteration (nearby rays have
// similar lengths, which keeps the lanes of the DDA loop together) and
// stages a band of 32/tile_w full image rows, written out contiguously.
struct FusedLayout {
    int W, H;
    int tile_w, tile_h;
    int stage_bytes;   // staging bytes per warp (one band of rows)
    int world_bytes;   // world bytes per warp (mc_world_slot; 0 when not staged)
    int warp_bytes;    // total per warp (16-aligned)
    int head_bytes;    // tables (16-aligned)
    int pad_bytes;     // allocated after the last warp's world
};

__host__ __device__ inline int mc_align16(int x) { return (x + 15) & ~15; }

// Tables of the per-warp kernel's common-case render loop, at the start of
// its shared memory: per block and shade code the colour times the shade
// (13 x 4 float4), then per block the flat colour packed as r | g << 8 | b << 16.
constexpr int kShadeTableBytes = 13 * 4 * 16;
constexpr int kFastTableBytes = MC_FAST_TABLE_BYTES;
static_assert(kFastTableBytes == kShadeTableBytes + 64, "fast tables");

__host__ __device__ inline FusedLayout fused_layout(int W, int H, int slot, int wxz, int obs_f32, int stage,
                                                   int tile_w, int fast) {
    FusedLayout L;
    L.W = W;
    L.H = H;
    L.tile_w = tile_w;
    L.tile_h = 32 / tile_w;
    L.stage_bytes = mc_band_bytes(W, obs_f32, tile_w, 0, fast);
    L.world_bytes = stage ? slot : 0;
    L.warp_bytes = 16 + 128 + L.stage_bytes + L.world_bytes;  // 16: mbarrier, 128: packed_start table
    L.head_bytes = kFastTableBytes + mc_align16((W + H) * 4 + 13 * 3 * 4 + 16 + 13 * 3 + 3);
    // the march reads up to wx*wz bytes on either side of a staged world:
    // keep that much allocated before the first world and after the last
    L.pad_bytes = stage ? mc_align16(wxz) : 0;
    const int before = L.head_bytes + 16 + 128 + L.stage_bytes;
    if (before < L.pad_bytes) L.head_bytes += mc_align16(L.pad_bytes - before);
    return L;
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

// Bounded wait on an mbarrier phase; returns false on timeout.  polls: 0 =
// MC_WAIT_POLLS_DEFAULT, n > 0 = n polls, < 0 = none (the timeout path's test).
__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t phase, int polls = 0) {
    const int limit = polls == 0 ? MC_WAIT_POLLS_DEFAULT : (polls < 0 ? 0 : polls);
    for (int it = 0; it < limit; ++it) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(mbar), "r"(phase)
            : "memory");
        if (done) return true;
    }
    return false;
}

// Next unit of this warp: claimed from a device counter (flag word `counter`; dynamic schedule,
// balances the uneven per-env work) or by static striding.
__device__ __forceinline__ int next_unit(const mc_kp& p, int counter, int cur, int total_warps, int lane) {
    if (!p.sched_dynamic) return cur + total_warps;
    unsigned v = 0;
    if (lane == 0) v = atomicAdd(reinterpret_cast<unsigned*>(&p.flags[counter]), 1u);
    return (int)__shfl_sync(0xffffffffu, v, 0);
}

// Per-warp view of the shared-memory tables and buffers used by one env.
struct FusedCtx {
    const float* s_u;            // per-column u of the env's image
    const float* s_v;            // per-row v
    const float (*s_rgb)[3];
    const float* s_sky;
    const uint8_t (*s_rgb8)[3];
    const uint8_t* s_sky8;
    uint8_t* stage;              // staging band of this warp
    uint8_t* colours;            // the colour tables' start
    uint32_t mbar_a;             // mbarrier of this warp
    float rcp_vd;                // reciprocal of the env's view distance
    const float4* s_cs;          // colour x shade table of the common-case loop (fast_band)
    const uint32_t* s_rgbp;      // packed flat colours
    int4* sstart;                // this warp's table of march start values (8 entries)
};

// The common-case loop's tables: colour x shade per block and shade code
// (0 x face, 1 z face, 2 y face stepping down, 3 y face stepping up, as in
// shade_rgb) and the flat colours packed r | g << 8 | b << 16.
__device__ __forceinline__ void build_fast_tables(float4* s_cs, uint32_t* s_rgbp) {
    for (int k = threadIdx.x; k < 13 * 4; k += blockDim.x) {
        const int blk = k >> 2, code = k & 3;
        const float shade = code == 0 ? 0.8f : (code == 1 ? 0.9f : (code == 2 ? 0.6f : 1.0f));
        s_cs[k] = make_float4(N::mul(c_rgb[blk][0], shade), N::mul(c_rgb[blk][1], shade),
                              N::mul(c_rgb[blk][2], shade), 0.0f);
    }
    for (int k = threadIdx.x; k < 13; k += blockDim.x)
        s_rgbp[k] = (uint32_t)c_rgb8[k][0] | ((uint32_t)c_rgb8[k][1] << 8) | ((uint32_t)c_rgb8[k][2] << 16);
}

// Shared colour tables: 13*3 + 4 floats, 13*3 + 3 bytes.
constexpr int kColourTableBytes = 13 * 3 * 4 + 16 + 13 * 3 + 3;
static_assert(kColourTableBytes <= MC_COLOUR_TABLE_BYTES, "colour tables");

__device__ __forceinline__ void colour_tables(uint8_t* base, FusedCtx& cx) {
    cx.colours = base;
    cx.s_rgb = reinterpret_cast<const float (*)[3]>(base);
    cx.s_sky = reinterpret_cast<const float*>(base + 13 * 3 * 4);
    cx.s_rgb8 = reinterpret_cast<const uint8_t (*)[3]>(base + 13 * 3 * 4 + 16);
    cx.s_sky8 = base + 13 * 3 * 4 + 16 + 13 * 3;
}

__device__ __forceinline__ void load_colour_tables(uint8_t* base, FusedCtx& cx) {
    colour_tables(base, cx);
    float* rgb = reinterpret_cast<float*>(base);
    uint8_t* rgb8 = base + 13 * 3 * 4 + 16;
    for (int k = threadIdx.x; k < 39; k += blockDim.x) {
        rgb[k] = c_rgb[k / 3][k % 3];
        rgb8[k] = c_rgb8[k / 3][k % 3];
    }
    if (threadIdx.x < 3) {
        rgb[39 + threadIdx.x] = c_sky[threadIdx.x];
        rgb8[39 + threadIdx.x] = c_sky8[threadIdx.x];
    }
}

// u/v tables of one image size (threads of the CTA cooperate).
template <int FAM>
__device__ __forceinline__ void build_uv_tables(const mc_kp& p, float* s_u, float* s_v) {
    const int W = p.W, H = p.H;
    float pb_su = 0.0f, pb_sv = 0.0f;
    if (FAM == MC_FAM_PREBASIS) prebasis_scales(W, H, p.fov, &pb_su, &pb_sv);
    for (int k = threadIdx.x; k < W; k += blockDim.x) {
        if (FAM == MC_FAM_SHADED || FAM == MC_FAM_SHADED_FAST) s_u[k] = u_shaded(k, W, H, p.fov);
        else if (FAM == MC_FAM_MINIMAL || FAM == MC_FAM_FP16) s_u[k] = u_minimal(k, W, H, p.fov);
        else s_u[k] = u_prebasis(k, W, pb_su);
    }
    for (int k = threadIdx.x; k < H; k += blockDim.x) {
        if (FAM == MC_FAM_SHADED || FAM == MC_FAM_SHADED_FAST) s_v[k] = v_shaded(k, H, p.fov);
        else if (FAM == MC_FAM_MINIMAL || FAM == MC_FAM_FP16) s_v[k] = v_minimal(k, H, p.fov);
        else s_v[k] = v_prebasis(k, H, pb_sv);
    }
}

// The parameters a ray needs.
struct RayPar {
    int wx, wy, wz, max_steps, gh;
    float vd;
};
__device__ __forceinline__ RayPar ray_par(const mc_kp& p) {
    RayPar r;
    r.wx = p.wx;
    r.wy = p.wy;
    r.wz = p.wz;
    r.max_steps = p.max_steps;
    r.gh = p.gh;
    r.vd = p.vd;
    return r;
}

// One pixel's ray through one of the two voxel sources.
template <int FAM, class V>
__device__ __forceinline__ Hit march_pixel(const RayPar& p, const Cam& c, const Dda0& d0, float u, float v,
                                           const V& vox, bool inside, bool skip_first, bool sky_exit = false,
                                           bool vd_safe = false, int ytop = 1 << 20) {
    if (FAM == MC_FAM_SHADED || FAM == MC_FAM_SHADED_FAST)
        return shade_ray<FAM == MC_FAM_SHADED_FAST, V>(c, d0, u, v, vox, p.wx, p.wy, p.wz, p.max_steps, p.vd,
                                                              p.gh, inside, skip_first, sky_exit, vd_safe, ytop);
    if (FAM == MC_FAM_FP16) return fp16_ray(c, d0, u, v, vox, p.wx, p.wy, p.wz, p.max_steps);
    return flat_ray<FAM != MC_FAM_PREBASIS>(c, d0, u, v, vox, p.wx, p.wy, p.wz, p.max_steps, skip_first, sky_exit,
                                              ytop);
}

__device__ __forceinline__ void mbar_init_warp(uint32_t mbar_a, int lane) {
    if (lane == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mbar_a) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
}

// The last warp (or team) of a dynamically scheduled launch resets the work
// counters and, for each of the groups, the any-done flag that the launch's
// regeneration has answered.  Every other one has read what it needs by then.
template <class Groups>
__device__ __forceinline__ void finish_dynamic(int32_t* flags, long long total, Groups clear_done) {
    __threadfence();
    unsigned prev = atomicAdd(reinterpret_cast<unsigned*>(&flags[MC_FLAG_WARPS_DONE]), 1u);
    if (prev == (unsigned)(total - 1)) {
        flags[MC_FLAG_WORK] = 0;
        flags[MC_FLAG_SLOW_WORK] = 0;
        flags[MC_FLAG_WARPS_DONE] = 0;
        flags[MC_FLAG_ANY_SLOW] = 0;
        clear_done();
        __threadfence();
    }
}

// Highest layer of a staged world holding a solid voxel (solid = byte >= 0,
// sign bit clear), found by one warp; -1 for an empty world; wy - 1 when its
// layers are no whole aligned 16-byte chunks (not measured).
__device__ __forceinline__ int staged_top_layer(const int8_t* world, int wx, int wy, int wz, int lane) {
    const int layer = wx * wz;
    if ((layer | (int)smem_u32(world)) & 15) return wy - 1;
    const uint4* w4 = reinterpret_cast<const uint4*>(world);
    const int n16 = (layer * wy) >> 4, per_layer = layer >> 4;
    int top = -1;
    for (int k = n16 - 1 - lane; k >= 0; k -= 32) {
        const uint4 q = w4[k];
        if ((~q.x | ~q.y | ~q.z | ~q.w) & 0x80808080u) {
            top = k / per_layer;
            break;  // this lane's remaining chunks lie in lower layers
        }
    }
    return __reduce_max_sync(0xffffffffu, top);
}

// Solid voxels (byte >= 0) of 16 consecutive bytes as a 16-bit mask: per
// 32-bit word the four sign bits (7, 15, 23, 31) of ~w, multiplied by
// 1 + 2^7 + 2^14 + 2^21, land on bits 28..31 with no carries.
__device__ __forceinline__ uint32_t solid_mask16(uint4 q) {
    auto four = [](uint32_t w) { return ((~w & 0x80808080u) * 0x00204081u) >> 28; };
    return four(q.x) | (four(q.y) << 4) | (four(q.z) << 8) | (four(q.w) << 12);
}

// Whether staged_up_bounds can scan a world of this shape: at most 64 voxels a side.
__host__ __device__ __forceinline__ bool up_scan_shape(int wx, int wy, int wz) {
    return wz <= 64 && wx <= 64 && wy <= 64;
}

// Solid voxels of one row of wz bytes as a mask: 16 bytes a load when rows are
// whole 16-byte chunks (`chunks`, uniform), else word by word, each funnelled
// from the two aligned words it lies in (the last one reads up to 7 bytes past
// the row; a staged world has at least one layer allocated after it).
template <typename M>
__device__ __forceinline__ M row_mask(const int8_t* row, int wz, bool chunks) {
    M m = 0;
    if (chunks) {
        const uint4* q = reinterpret_cast<const uint4*>(row);
        for (int k = 0; k < (wz >> 4); ++k) m |= M(solid_mask16(q[k])) << (16 * k);
        return m;
    }
    const uint32_t off = smem_u32(row) & 3u;
    const uint32_t* w = reinterpret_cast<const uint32_t*>(row - off);
    uint32_t lo = w[0];
    for (int k = 0; 4 * k < wz; ++k) {
        const uint32_t hi = w[k + 1], q = __funnelshift_r(lo, hi, 8 * off);
        m |= M(((~q & 0x80808080u) * 0x00204081u) >> 28) << (4 * k);
        lo = hi;
    }
    return wz < (int)(8 * sizeof(M)) ? m & ((M(1) << wz) - 1) : m;
}

// One warp scans the rows (y >= vy, x) of a staged world (up_scan_shape;
// the eye's voxel inside the box) for the bounds of every quadrant.  Each
// lane keeps one x (two in worlds wider than 32): G = 32 / wx groups of wx
// lanes sweep every G-th layer, so per row a lane only ORs the row's solid
// z mask into its column's union and notes the highest layers with a solid
// voxel at z >= vz and at z <= vz; the column's x side and the z extremes
// are settled once, after the sweep.  With nw > 1 warps sharing the scan,
// warp w of them sweeps the layers of groups w*G .. w*G+G-1 of nw*G, and
// the result is the warp's part of the bounds (combined by team_up_bounds).
template <typename M>
struct UpPart {
    int xa0, xa1, xa2, xa3;  // x extremes of q0 (x-, z-), q1 (x+, z-), q2 (x-, z+), q3 (x+, z+)
    int ya0, ya1, ya2, ya3;  // highest layer + 1
    M mp, mm;                // solid z masks of the x >= vx / x <= vx columns
};

template <typename M>
__device__ __forceinline__ UpPart<M> staged_up_part(const int8_t* world, int wx, int wy, int wz, int vx, int vy,
                                                    int vz, int lane, int w = 0, int nw = 1) {
    const bool chunks = ((wz | (int)smem_u32(world)) & 15) == 0;
    constexpr int kBits = 8 * sizeof(M);
    const M zpm = ~M(0) << vz;                            // z >= vz
    const M zmm = (vz + 1 < kBits) ? ((M(1) << (vz + 1)) - 1) : ~M(0);  // z <= vz
    const int G = wx <= 32 ? 32 / wx : 1, g = wx <= 32 ? lane / wx : 0;
    int xa0 = 255, xa1 = 0, xa2 = 255, xa3 = 0;
    int ya0 = 0, ya1 = 0, ya2 = 0, ya3 = 0;
    M mp = 0, mm = 0;
    for (int x = wx <= 32 ? lane - g * wx : lane; g < G && x < wx; x += 32) {
        M mu = 0;
        int yp = 0, ym = 0;  // highest layer + 1 with a solid voxel at z >= vz / z <= vz
        for (int y = vy + w * G + g; y < wy; y += G * nw) {
            const int r = y * wx + x;
            const M m = in_bounds(r, (long long)wx * wy, MC_SITE_SCAN) ? row_mask<M>(world + r * wz, wz, chunks) : M(0);
            mu |= m;
            yp = (m & zpm) ? y + 1 : yp;
            ym = (m & zmm) ? y + 1 : ym;
        }
        if (x >= vx) {
            mp |= mu;
            if (yp) { xa3 = max(xa3, x); ya3 = max(ya3, yp); }
            if (ym) { xa1 = max(xa1, x); ya1 = max(ya1, ym); }
        }
        if (x <= vx) {
            mm |= mu;
            if (yp) { xa2 = min(xa2, x); ya2 = max(ya2, yp); }
            if (ym) { xa0 = min(xa0, x); ya0 = max(ya0, ym); }
        }
    }
    constexpr unsigned F = 0xffffffffu;
    auto or_all = [](M v) -> M {
        if (sizeof(M) == 8)
            return M(__reduce_or_sync(F, (unsigned)v)) | (M(__reduce_or_sync(F, (unsigned)(v >> 16 >> 16))) << 16 << 16);
        return M(__reduce_or_sync(F, (unsigned)v));
    };
    UpPart<M> r;
    r.mp = or_all(mp);
    r.mm = or_all(mm);
    r.xa0 = __reduce_min_sync(F, xa0);
    r.xa1 = __reduce_max_sync(F, xa1);
    r.xa2 = __reduce_min_sync(F, xa2);
    r.xa3 = __reduce_max_sync(F, xa3);
    r.ya0 = __reduce_max_sync(F, ya0);
    r.ya1 = __reduce_max_sync(F, ya1);
    r.ya2 = __reduce_max_sync(F, ya2);
    r.ya3 = __reduce_max_sync(F, ya3);
    return r;
}

// The bounds from the (combined) parts.  z extremes: over a side's solid
// voxels the largest z is the z >= vz quadrant's extreme whenever that
// quadrant holds any (else its y byte is 0 and the value is not used), the
// smallest z likewise.
template <typename M>
__device__ __forceinline__ UpBounds up_bounds_of(const UpPart<M>& r) {
    constexpr int kBits = 8 * sizeof(M);
    auto hi = [](M v) { return kBits - 1 - (sizeof(M) == 8 ? __clzll((long long)v) : __clz((int)v)); };
    auto lo = [](M v) { return (sizeof(M) == 8 ? __ffsll((long long)v) : __ffs((int)v)) - 1; };
    UpBounds b;
    b.x = (unsigned)r.xa0 | ((unsigned)r.xa1 << 8) | ((unsigned)r.xa2 << 16) | ((unsigned)r.xa3 << 24);
    b.z = ((unsigned)lo(r.mm) & 255u) | (((unsigned)lo(r.mp) & 255u) << 8) | (((unsigned)hi(r.mm) & 255u) << 16) |
          (((unsigned)hi(r.mp) & 255u) << 24);
    b.y = (unsigned)r.ya0 | ((unsigned)r.ya1 << 8) | ((unsigned)r.ya2 << 16) | ((unsigned)r.ya3 << 24);
    return b;
}

__device__ __forceinline__ UpBounds staged_up_bounds(const int8_t* world, int wx, int wy, int wz, int vx, int vy,
                                                     int vz, int lane) {
    return wz > 32 ? up_bounds_of(staged_up_part<unsigned long long>(world, wx, wy, wz, vx, vy, vz, lane))
                   : up_bounds_of(staged_up_part<uint32_t>(world, wx, wy, wz, vx, vy, vz, lane));
}

// ---------------------------------------------------------------------------
// Rendering one env
// ---------------------------------------------------------------------------
// The common-case render of one band of an env's image (both step
// kernels): the world is staged, the eye is inside the box with air in its
// voxel (every ray starts one DDA step in, and ends as sky when it leaves
// the box) and no debug output is asked for.  Every ray's march start values
// come from a per-env table of the eight ray sign combinations (packed_start for the
// packed march, split_start for the split march).  Every per-env fact is
// settled before the loop, so the per-ray code has no branch but the
// march's: the same operations in the same order as shade_ray / flat_ray
// and shade_rgb (the bits are identical), with the shading done for every
// lane and the sky colour selected afterwards, the colour times the face's
// shade read from s_cs (built with the same N::mul), and the band address
// stepped incrementally.  The band goes to `stage`, then to `dst` with
// 16-byte stores.
// ODD: the image is no whole number of tile_w x (32/tile_w) tiles, or its
// bands no whole 16-byte pieces: lanes beyond the image march the nearest
// pixel's ray again and store nothing, and the band is staged at dst's offset
// from a 16-byte boundary, so that all but its first and last bytes still go
// out in 16-byte stores (`stage` has 16 bytes to spare).
// TEAM: the team kernel stages float32 pixels two tiles at a time instead (64
// pixels, 768 bytes, whose row pieces are whole 16-byte chunks; with ODD they go
// straight to dst): beside 32 KB worlds, whole bands of 128-pixel rows (6 KB a
// warp) left one CTA on an SM (4096 envs 32^3 128x128: 1151 -> 710 us a step).
// The per-warp kernel keeps whole bands (32x32: 174 us a step, two tiles 186).
struct FastEnv {
    const int4* start;  // per sign combination: packed (index|counts, dx, dy, dz) or split (counts, dax, day, daz)
    uint32_t base;      // staged world (packed) / the eye voxel's address in it (split)
    SmemRange chk;      // the staged world +- one layer (debug build)
    float vd, rcp_vd;
    int wx, wy, wz, max_steps;  // ground-shortcut family only
};

// The ground-shortcut family's rays that leave the box sideways on their way
// down: the reference goes on stepping while t <= the box's exit distance
// (rounding puts the accumulated t on either side of it) and still paints the
// ground if such a step enters it.  bx, by: the axis of the step that left the
// box (tm not advanced for it yet); yleft: layers left above the ground; step:
// voxels stepped.  Returns whether the ray ends in the ground, *t its distance.
__device__ __forceinline__ bool ground_tail(const Cam& c, const FastEnv& fe, float ix, float iy, float iz, float tmx,
                                            float tmy, float tmz, bool bx, bool by, int yleft, int step, float* t) {
    const float lo_x = N::sub(0.0f, c.eye_x), hi_x = N::sub((float)fe.wx, c.eye_x);
    const float lo_y = N::sub(0.0f, c.eye_y), hi_y = N::sub((float)fe.wy, c.eye_y);
    const float lo_z = N::sub(0.0f, c.eye_z), hi_z = N::sub((float)fe.wz, c.eye_z);
    float entry;
    const float t_exit = aabb_exit(ix, iy, iz, lo_x, hi_x, lo_y, hi_y, lo_z, hi_z, &entry);
    while (!(*t >= fe.vd) && !(*t > t_exit) && step < fe.max_steps) {
        if (bx) tmx = N::add(tmx, fabsf(ix));
        else if (by) tmy = N::add(tmy, fabsf(iy));
        else tmz = N::add(tmz, fabsf(iz));
        bx = tmx < tmy && tmx < tmz;
        by = !bx && tmy < tmz;
        *t = bx ? tmx : (by ? tmy : tmz);
        ++step;
        if (by && --yleft < 0) return step < fe.max_steps && !(*t >= fe.vd);
    }
    return false;
}

template <int FAM, bool F32, bool SPLIT, bool ODD, bool TEAM>
__device__ __forceinline__ void fast_band(const Cam& c, const Dda0& d0, const FastEnv& fe, int W, int H, int sh,
                                          int row0, int lane, const float* s_u, const float* s_v, const float4* s_cs,
                                          const uint32_t* s_rgbp, uint8_t* stage, uint8_t* dst) {
    constexpr bool PAIRS = F32 && TEAM && !ODD, DIRECT = F32 && TEAM && ODD;  // how float32 pixels leave
    constexpr bool GROUND = FAM == MC_FAM_SHADED_FAST;
    constexpr bool SHADED = FAM == MC_FAM_SHADED || GROUND;
    constexpr bool HALF = FAM == MC_FAM_FP16;
    constexpr bool TRIG = FAM != MC_FAM_PREBASIS;
    constexpr int bpp = 3 * (F32 ? 4 : 1);
    constexpr int m = F32 ? 0x1 : (GROUND ? MC_FASTG_SKY : 0x3);  // sky_fused_mask of the family's kernel
    const float sky0 = 0.53f, sky1 = 0.81f, sky2 = 0.92f;  // SKY_COLOR (c_sky)
    const int TW = 1 << sh, TH = 32 >> sh;  // sh: log2 of the tile's width
    const int lx = lane & (TW - 1), ly = lane >> sh;
    const bool in_y = !ODD || row0 + ly < H;
    const float v = s_v[ODD ? min(row0 + ly, H - 1) : row0 + ly];
    const float yraw = N::mad(v, c.uy, c.fy);
    if (ODD && !DIRECT) stage += (uint32_t)(uintptr_t)dst & 15u;
    uint8_t* sp = DIRECT ? dst + (ly * W + lx) * bpp : stage + (ly * (PAIRS ? 2 * TW : W) + lx) * bpp;
    for (int tx0 = 0; tx0 < W; tx0 += TW, sp += TW * bpp) {
        const bool in = !ODD || (in_y && tx0 + lx < W);
        const float u = s_u[ODD ? min(tx0 + lx, W - 1) : tx0 + lx];
        float x, y = yraw, z;
        if (TRIG) {
            x = N::mad(v, c.ux, N::mad(c.sy, c.cp, N::mul(u, c.rx)));
            z = N::mad(v, c.uz, N::mad(c.cy, c.cp, N::mul(u, c.rz)));
        } else {
            x = N::mad(v, c.ux, N::mad(u, c.rx, c.fx));
            z = N::mad(v, c.uz, N::mad(u, c.rz, c.fz));
        }
        if (SHADED) {
            const float len = N::sqrt(len2(x, y, z));
            const float rl = N::rcp_of(len);
            x = N::div_r(x, len, rl);
            y = N::div_r(y, len, rl);
            z = N::div_r(z, len, rl);
        } else {
            const float rs = N::rsqrt(len2(x, y, z));
            x = N::mul(x, rs);
            y = N::mul(y, rs);
            z = N::mul(z, rs);
        }
        constexpr float kNone = HALF ? 65504.0f : 1e30f;
        const float ix = (x != 0.0f) ? N::div(1.0f, x) : kNone;
        const float iy = (y != 0.0f) ? N::div(1.0f, y) : kNone;
        const float iz = (z != 0.0f) ? N::div(1.0f, z) : kNone;
        const bool xp = x >= 0.0f, yp = y >= 0.0f, zp = z >= 0.0f;
        float tmx = N::mul(xp ? d0.nxp : d0.nxm, ix);
        float tmy = N::mul(yp ? d0.nyp : d0.nym, iy);
        float tmz = N::mul(zp ? d0.nzp : d0.nzm, iz);
        int4 e = fe.start[(xp ? 1 : 0) | (yp ? 2 : 0) | (zp ? 4 : 0)];
        int b;
        if constexpr (HALF) {
            auto h = [](float f) { return __half_as_ushort(__float2half(f)); };
            unsigned short hx = h(tmx), hy = h(tmy), hz = h(tmz);
            b = SPLIT ? march_split_shared(fe.base, e.x, e.y, e.z, e.w, hx, hy, hz, h(fabsf(ix)), h(fabsf(iy)),
                                           h(fabsf(iz)), fe.chk)
                      : march_packed_shared(fe.base, e.x, e.y, e.z, e.w, hx, hy, hz, h(fabsf(ix)), h(fabsf(iy)),
                                            h(fabsf(iz)), fe.chk);
        } else {
            b = SPLIT ? march_split_shared(fe.base, e.x, e.y, e.z, e.w, tmx, tmy, tmz, fabsf(ix), fabsf(iy), fabsf(iz),
                                           fe.chk)
                      : march_packed_shared(fe.base, e.x, e.y, e.z, e.w, tmx, tmy, tmz, fabsf(ix), fabsf(iy),
                                            fabsf(iz), fe.chk);
        }
        if (SHADED) {
            // the axis of the last step, chosen again from the same distances
            const bool bx = tmx < tmy && tmx < tmz;
            const bool by = !bx && tmy < tmz;
            float t = bx ? tmx : (by ? tmy : tmz);
            int code = bx ? 0 : (by ? (yp ? 3 : 2) : 1);
            if (GROUND && b < 0 && !yp) {
                // a ray going down that left the box: into the ground (grass,
                // from above), sideways, or out of steps (split march)
                constexpr int kOutX = SPLIT ? 1 << 13 : 32 << 12, kOutY = SPLIT ? 1 << 20 : 32 << 6,
                              kOutZ = SPLIT ? 1 << 6 : 32, kSpent = SPLIT ? 1 << 29 : 0;
                if (!(e.x & kSpent)) {
                    if (e.x & kOutY) {
                        b = GRASS;
                    } else if (e.x & (kOutX | kOutZ)) {
                        const int yleft = SPLIT ? 63 - ((e.x >> 14) & 127) : 31 - ((e.x >> 6) & 63);
                        const int s0 = fe.max_steps > fe.wx + fe.wy + fe.wz ? 0 : 256 - fe.max_steps;
                        const int step = SPLIT ? ((e.x >> 21) & 511) - s0 : 0;
                        if (ground_tail(c, fe, ix, iy, iz, tmx, tmy, tmz, bx, by, yleft, step, &t)) {
                            b = GRASS;
                            code = 2;
                        }
                    }
                }
            }
            const bool hit = b >= 0 && !(t >= fe.vd);
            const float4 cs = s_cs[(b >= 0 ? b : 0) * 4 + code];
            float fog = fminf(N::div_r(t, fe.vd, fe.rcp_vd), 1.0f);
            fog = N::mul(fog, fog);
            const float omf = N::sub(1.0f, fog);
            const float c0 = (m & 1) ? N::mad(sky0, fog, N::mul(cs.x, omf)) : N::mad(cs.x, omf, N::mul(sky0, fog));
            const float c1 = (m & 2) ? N::mad(sky1, fog, N::mul(cs.y, omf)) : N::mad(cs.y, omf, N::mul(sky1, fog));
            const float c2 = (m & 4) ? N::mad(sky2, fog, N::mul(cs.z, omf)) : N::mad(cs.z, omf, N::mul(sky2, fog));
            const float o0 = hit ? c0 : sky0, o1 = hit ? c1 : sky1, o2 = hit ? c2 : sky2;
            if (ODD && !in) {
            } else if (F32) {
                float* sf = reinterpret_cast<float*>(sp);
                sf[0] = o0;
                sf[1] = o1;
                sf[2] = o2;
            } else {
                sp[0] = (uint8_t)to_u8(o0);
                sp[1] = (uint8_t)to_u8(o1);
                sp[2] = (uint8_t)to_u8(o2);
            }
        } else {
            // SKY_COLOR_U8 (135, 206, 235) packed
            const uint32_t col = b >= 0 ? s_rgbp[b] : (135u | (206u << 8) | (235u << 16));
            if (in) {
                sp[0] = (uint8_t)col;
                sp[1] = (uint8_t)(col >> 8);
                sp[2] = (uint8_t)(col >> 16);
            }
        }
        if (PAIRS && ((tx0 & TW) || tx0 + TW == W)) {
            // these one or two tiles' rows, 16 bytes a lane
            const int first = tx0 & ~(2 * TW - 1), cols = tx0 + TW - first, cpr = cols * 3 >> 2, n = TH * cpr;
            const int mul = (cols >> sh) == 2 ? 43691 : 87382;  // k / cpr = (k * 4 / (3 cols)), k < 48
            __syncwarp();
            for (int k = lane; k < n; k += 32) {
                const int row = k * mul >> (16 + sh), piece = k - row * cpr;
                *reinterpret_cast<uint4*>(dst + (row * W + first) * bpp + piece * 16) =
                    *reinterpret_cast<const uint4*>(stage + row * 2 * TW * bpp + piece * 16);
            }
            __syncwarp();
            sp = stage + (ly * 2 * TW + lx) * bpp - TW * bpp;
        }
    }
    if (PAIRS || DIRECT) return;
    __syncwarp();
    // copy the band (rows row0 .. row0+TH-1) out with 16-byte stores
    int bytes = W * TH * bpp;
    if (ODD) {
        bytes = W * min(TH, H - row0) * bpp;
        const int head = min((int)(-(uint32_t)(uintptr_t)dst & 15u), bytes);
        const int tail = (bytes - head) & 15;
        if (lane < head) dst[lane] = stage[lane];
        if (lane < tail) dst[bytes - tail + lane] = stage[bytes - tail + lane];
        stage += head;
        dst += head;
        bytes -= head + tail;
    }
    const uint4* s4 = reinterpret_cast<const uint4*>(stage);
    uint4* d4 = reinterpret_cast<uint4*>(dst);
    for (int k = lane; k < (bytes >> 4); k += 32) d4[k] = s4[k];
    __syncwarp();
}

// Start values of march_split_shared for an env whose eye is in voxel (vx,
// vy, vz), one per sign combination k of the ray (as packed_start): {counts,
// x, y and z address steps}; the start address is the eye voxel's.
__device__ __forceinline__ int4 split_start(int k, int vx, int vy, int vz, int wx, int wy, int wz, int ylow,
                                            const UpBounds& ub, int max_steps) {
    const int sx = (k & 1) ? 1 : -1, sy = (k & 2) ? 1 : -1, sz = (k & 4) ? 1 : -1;
    int cx, cy, cz;
    start_counts(k, vx, vy, vz, wx, wy, wz, ylow, ub, cx, cy, cz);
    return make_int4(split_counts(cx, cy, cz, max_steps, wx, wy, wz), sx * wz, sy * wx * wz, sz);
}

// Which march an env on the common path takes: 1 packed (small worlds where
// every ray leaves the box before max_steps; for the shaded family the whole
// box within view distance), 2 split.
template <int FAM>
__device__ __forceinline__ int fast_kind(bool vd_safe, int max_steps, int wx, int wy, int wz) {
    constexpr bool G = FAM == MC_FAM_SHADED_FAST;  // its rays may step on outside the box (ground_tail)
    const bool packed = (FAM == MC_FAM_SHADED || G ? vd_safe : true) && max_steps > wx + wy + wz + (G ? 8 : 0) &&
                        mc_packed_world(wx, wy, wz);
    return packed ? 1 : 2;
}

// The per-env start table (8 lanes write, the warp reads).
__device__ __forceinline__ void build_fast_start(int4* sstart, int kind, const Dda0& d0, int wx, int wy, int wz,
                                                 int ylow, const UpBounds& ub, int max_steps, int lane) {
    if (lane < 8)
        sstart[lane] = kind == 1 ? packed_start(lane, d0.vx, d0.vy, d0.vz, wx, wy, wz, ylow, ub)
                                 : split_start(lane, d0.vx, d0.vy, d0.vz, wx, wy, wz, ylow, ub, max_steps);
    __syncwarp();
}

// Per-env facts of a render (EnvRec::bits, EnvRender::bits).
// MC_ER_SLOW: a marching env that needs the general path (render_slow_from).
enum { MC_ER_DONE = 1, MC_ER_BURIED = 2, MC_ER_INSIDE = 4, MC_ER_SKIP = 8, MC_ER_SLOW = 16 };

// ---------------------------------------------------------------------------
// The agents: one thread per env
// ---------------------------------------------------------------------------
// What the image of one env needs from its agent step: the eye, sin and cos of
// yaw and pitch (the same calls the reference makes per pixel), and the facts
// settled by the eye's voxel.  48 bytes, read as three 16-byte loads.
struct __align__(16) EnvRec {
    float ex, ey, ez;
    int env;             // the env's index in its group
    float sy, cy, sp, cp;
    int bits;            // MC_ER_*
    int fill_blk;        // block of the uniform fill of a buried camera
    int arrived;         // slices of the image that are done (last_slice)
    int pad;
};
static_assert(sizeof(EnvRec) == MC_REC_BYTES, "env record");

__device__ __forceinline__ EnvRec load_rec(const void* rec, long long i) {
    const float4* q = reinterpret_cast<const float4*>(rec) + i * 3;
    const float4 a = q[0], b = q[1];
    const int4 c = reinterpret_cast<const int4*>(q)[2];
    EnvRec r;
    r.ex = a.x; r.ey = a.y; r.ez = a.z;
    r.env = __float_as_int(a.w);
    r.sy = b.x; r.cy = b.y; r.sp = b.z; r.cp = b.w;
    r.bits = c.x;
    r.fill_blk = c.y;
    return r;
}
__device__ __forceinline__ void store_rec(void* rec, long long i, const EnvRec& r) {
    float4* q = reinterpret_cast<float4*>(rec) + i * 3;
    q[0] = make_float4(r.ex, r.ey, r.ez, __int_as_float(r.env));
    q[1] = make_float4(r.sy, r.cy, r.sp, r.cp);
    reinterpret_cast<int4*>(q)[2] = make_int4(r.bits, r.fill_blk, 0, 0);
}

// The camera of a record: the products of cam_trig / basis_compute.
__device__ __forceinline__ Cam cam_of_rec(const EnvRec& r) {
    Cam c;
    c.eye_x = r.ex; c.eye_y = r.ey; c.eye_z = r.ez;
    c.fx = N::mul(r.sy, r.cp);
    c.fy = r.sp;
    c.fz = N::mul(r.cy, r.cp);
    c.rx = r.cy;
    c.rz = -r.sy;
    c.ux = N::mul(-r.sy, r.sp);
    c.uy = r.cp;
    c.uz = N::mul(-r.cy, r.sp);
    c.sy = r.sy;
    c.cy = r.cy;
    c.cp = r.cp;
    return c;
}

// The eye's voxel: its index in the world, -1 outside the box.
__device__ __forceinline__ int eye_index(const EnvRec& r, const mc_kp& p) {
    const int ex = (int)floorf(r.ex), ey = (int)floorf(r.ey), ez = (int)floorf(r.ez);
    const bool inb = (unsigned)ex < (unsigned)p.wx && (unsigned)ey < (unsigned)p.wy && (unsigned)ez < (unsigned)p.wz;
    return inb ? ey * (p.wx * p.wz) + ex * p.wz + ez : -1;
}

// sin and cos of the camera's angles, as the family's render computes them.
template <int FAM>
__device__ __forceinline__ void rec_trig(EnvRec& r, float yaw, float pitch) {
    if (FAM == MC_FAM_PREBASIS) {
        N::sincos_i(yaw, &r.sy, &r.cy);
        N::sincos_i(pitch, &r.sp, &r.cp);
    } else {
        r.cy = N::cos(yaw);
        r.sy = N::sin(yaw);
        r.cp = N::cos(pitch);
        r.sp = N::sin(pitch);
    }
}

// The facts of a record whose eye is set; eye_blk: the block there (AIR outside
// the box).  Every ray starts in the eye's voxel: if the first DDA step
// already hits (the eye is inside a solid voxel, or below ground for the
// ground-shortcut family), every pixel of the env gets the same colour
// (MC_ER_BURIED); if that test is known to fail, rays start advanced by one
// step (MC_ER_SKIP).
template <int FAM>
__device__ __forceinline__ void rec_facts(EnvRec& r, const mc_kp& p, bool eye_inb, int eye_blk, bool done) {
    bool inside = false, buried, skip_first;
    r.fill_blk = eye_blk;
    if (FAM == MC_FAM_SHADED || FAM == MC_FAM_SHADED_FAST) {
        Cam c;
        c.eye_x = r.ex; c.eye_y = r.ey; c.eye_z = r.ez;
        inside = eye_inside(c, p.wx, p.wy, p.wz, p.vd);
        const int ey = (int)floorf(r.ey);
        const bool below = FAM == MC_FAM_SHADED_FAST && ey < p.gh;
        if (below) r.fill_blk = (ey == p.gh - 1) ? GRASS : DIRT;
        const bool can = inside && p.vd > 0.0f && p.max_steps > 0;
        buried = can && (eye_blk >= 0 || below);
        skip_first = can && eye_blk < 0 && !below;
    } else {
        buried = p.max_steps > 0 && eye_inb && eye_blk >= 0;
        skip_first = p.max_steps > 0 && !(eye_inb && eye_blk >= 0);
    }
    // the common case: the launch allows it, and the eye is inside the box with air in its voxel
    const bool fast = p.fast_ok && skip_first && (FAM == MC_FAM_SHADED || FAM == MC_FAM_SHADED_FAST || eye_inb);
    r.bits = (done ? MC_ER_DONE : 0) | (buried ? MC_ER_BURIED : 0) | (inside ? MC_ER_INSIDE : 0) |
             (skip_first ? MC_ER_SKIP : 0) | (!buried && !fast ? MC_ER_SLOW : 0);
}

// Up to this many envs of a warp that interact share its lanes (look_together,
// about 40 instructions an env); more take a thread each (look_samples, about
// 750 for the warp, however few envs).  Uniform discrete actions break in 3
// envs of 32: us a step, a thread per env -> shared lanes, 64 envs 16^3, 32x32
// 14.8 -> 13.2, 4096 envs with host buffers 47.4 -> 45.7, 1024 envs 64x64 with
// buttons (8 of 32) 37.9 -> 37.1; with half the actions breaking 195.0 and 195.1.
constexpr int kLookTogether = 12;

// Decode, episode rule, physics, interaction, reset, counters, camera (and
// basis) of env e, by one thread.  Its loads come in two waves: the action and
// state, then the eye's voxel and the interaction's samples.  The whole warp
// calls it: the lanes without an env (`valid` false) bring the e of another,
// help with the samples and write nothing.
template <int FAM>
__device__ __forceinline__ EnvRec agent_step(const mc_kp& p, const ActionSrc& act, long long e, bool valid,
                                             float* res_rewards, uint8_t* res_dones) {
    const long long wxyz = (long long)p.wx * p.wy * p.wz;
    int8_t btn[8];
    float l0, l1;
    load_action_from(act, p.look_delta, e, btn, l0, l1);
    const Dec d = decode_buttons(btn, l0, l1, p.sprint_mult);
    const int32_t cnt = p.ext_done ? 0 : p.step_count[e];
    const bool done = p.ext_done ? (p.do_reset[e] != 0) : episode_done(p, cnt);
    Agent a = load_agent(p, e);
    float sy, cy;
    physics(a, d, p, sy, cy);
    int8_t* w = p.voxels + e * wxyz;
    Look l;
    l.ex = a.x;
    l.ey = N::add(a.y, 1.6f);
    l.ez = a.z;
    const float cp = N::cos(a.pitch), sp = N::sin(a.pitch);
    l.dx = N::mul(sy, cp);
    l.dy = sp;
    l.dz = N::mul(cy, cp);
    if (done) reset_agent(a, p);
    EnvRec r;
    r.env = (int)e;
    r.ex = a.x;
    r.ey = N::add(a.y, 1.6f);
    r.ez = a.z;
    r.sy = sy; r.cy = cy; r.sp = sp; r.cp = cp;
    if (FAM == MC_FAM_PREBASIS || done) rec_trig<FAM>(r, a.yaw, a.pitch);
    const int eye = eye_index(r, p);
    int eye_blk = AIR;
    if (eye >= 0 && in_bounds(eye, wxyz, MC_SITE_EYE)) eye_blk = w[eye];
    float reward = 0.0f;
    int mod_idx = -1, mod_val = 0;
    const bool want = valid && (d.brk || d.place);
    const unsigned who = __ballot_sync(0xffffffffu, want);
    if (__popc(who) <= kLookTogether)
        look_together(l, w, p, who, threadIdx.x & 31);
    else if (want)
        look_samples(l, w, p);
    if (want) {
        mod_idx = interact_judge(l, w, d.brk, p, &reward, &mod_val);
        if (mod_idx >= 0 && mod_idx == eye) eye_blk = mod_val;
    }
    rec_facts<FAM>(r, p, eye >= 0, eye_blk, done);
    if (!valid) return r;
    store_agent(p, e, a);
    if (!p.ext_done) {
        p.step_count[e] = done ? 1 : cnt + 1;
        p.do_reset[e] = done ? 1 : 0;
    }
    p.rewards[e] = reward;
    if (res_rewards) res_rewards[e] = reward;
    if (res_dones) res_dones[e] = done ? 1 : 0;
    p.cameras[e * 5 + 0] = a.x;
    p.cameras[e * 5 + 1] = a.y;
    p.cameras[e * 5 + 2] = a.z;
    p.cameras[e * 5 + 3] = a.yaw;
    p.cameras[e * 5 + 4] = a.pitch;
    if (p.dbg_interact) p.dbg_interact[e] = mod_idx;
    if (FAM == MC_FAM_PREBASIS && p.basis) {
        float bas[13];
        basis_compute(a.x, a.y, a.z, a.yaw, a.pitch, p.W, p.H, p.fov, bas);
#pragma unroll
        for (int k = 0; k < 13; ++k) p.basis[e * 14 + k] = bas[k];
    }
    return r;
}

// ---- regeneration -----------------------------------------------------------
// The step's regeneration is done by whoever rendered the env last: its world
// is not read again in this step, so the template's bytes go over it right
// after its image, with no pass over all worlds and no kernel of its own.
// Which worlds (p.regen): none, all of them when any env of the group is done
// (MC_KREGEN_ALL; the agent kernel has settled that), or the done envs' own.
// Launches without the common path leave it to a kernel after them (their
// worlds are big beside their images: 1024 envs 80^3 8x8 of which one in 30 is
// done, 170 us a step, 116 with a kernel of its own), and so do team launches
// over worlds of no whole 16 bytes (6153 envs 25x22x39 119.9 -> 81.9).
__device__ __forceinline__ int regen_any(const mc_kp& p) {
    return p.regen == MC_KREGEN_ALL
               ? __shfl_sync(0xffffffffu, *(volatile int32_t*)&p.flags[MC_FLAG_ANY_DONE], 0) : 0;
}
__device__ __forceinline__ bool regen_env(const mc_kp& p, int bits, int any_done) {
    return any_done || (p.regen == MC_KREGEN_PER_ENV && (bits & MC_ER_DONE));
}
// The world an env's image shows: its own, or the template where a reset (not
// a step: `fresh`) regenerates it in this launch.
__device__ __forceinline__ const int8_t* world_of(const mc_kp& p, int e, int bits, int any_done) {
    return p.fresh && regen_env(p, bits, any_done) ? p.world_template
                                                   : p.voxels + e * (long long)p.wx * p.wy * p.wz;
}

// The record of env e, its agent at x, y, z, from its state alone (no step's):
// reset and get_obs, and the images of a launch that has no records (p.rec NULL:
// the stateless step).
template <int FAM>
__device__ __forceinline__ EnvRec look_rec(const mc_kp& p, long long e, float x, float y, float z, float yaw, float pitch,
                                           bool done, int any_done) {
    EnvRec r;
    r.env = (int)e;
    r.ex = x;
    r.ey = N::add(y, 1.6f);
    r.ez = z;
    rec_trig<FAM>(r, yaw, pitch);
    const long long wxyz = (long long)p.wx * p.wy * p.wz;
    const int eye = eye_index(r, p);
    int eye_blk = AIR;
    if (eye >= 0 && in_bounds(eye, wxyz, MC_SITE_EYE)) eye_blk = world_of(p, (int)e, done ? MC_ER_DONE : 0, any_done)[eye];
    rec_facts<FAM>(r, p, eye >= 0, eye_blk, done);
    return r;
}
template <int FAM>
__device__ __noinline__ void look_rec_out(const mc_kp& p, int i, EnvRec& r) {
    const long long e = i;
    r = look_rec<FAM>(p, e, p.positions[e * 3 + 0], p.positions[e * 3 + 1], p.positions[e * 3 + 2], p.yaws[e],
                      p.pitches[e], false, 0);
}
// The record of the launch's i-th unit.
template <int FAM>
__device__ __forceinline__ EnvRec rec_of(const mc_kp& p, int i) {
    if (p.rec) return load_rec(p.rec, i);
    EnvRec r;
    look_rec_out<FAM>(p, i, r);
    return r;
}

constexpr int kAgentThreads = MC_AGENT_THREADS;

// File the block's records (called by all its threads): record e at e, or,
// with more envs than the image kernel has warps (`compact`), the records of the envs on the common path fill the group's record
// array from the front and those of the others (buried, or left to the
// general pass) from the back, so the image kernel's warps claim the costly
// envs first and the cheap uniform fills even out the end of the launch.  One 64-bit counter holds both fill counts;
// the block that brings their sum to the group's size clears it for the next
// launch (every env is filed exactly once, so no other block adds after it).
__device__ __forceinline__ void file_recs(void* rec, int32_t* flags, int32_t* any_slow, long long B, bool compact,
                                          const EnvRec& r, long long e, bool valid, bool step = true) {
    __shared__ unsigned s_m[kAgentThreads / 32], s_b[kAgentThreads / 32];
    __shared__ unsigned long long s_base;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool march = valid && !(r.bits & (MC_ER_BURIED | MC_ER_SLOW)), fill = valid && !march;
    if (valid && (r.bits & MC_ER_SLOW)) *any_slow = 1;
    const unsigned done = __ballot_sync(0xffffffffu, step && valid && (r.bits & MC_ER_DONE));
    if (done && lane == 0) atomicOr(&flags[MC_FLAG_ANY_DONE], 1);
    if (!compact) {
        if (valid && rec) store_rec(rec, e, r);
        return;
    }
    const unsigned mm = __ballot_sync(0xffffffffu, march), mb = __ballot_sync(0xffffffffu, fill);
    if (lane == 0) {
        s_m[warp] = __popc(mm);
        s_b[warp] = __popc(mb);
    }
    __syncthreads();
    unsigned pm = 0, pb = 0, tm = 0, tb = 0;
#pragma unroll
    for (int w = 0; w < kAgentThreads / 32; ++w) {
        if (w == warp) { pm = tm; pb = tb; }
        tm += s_m[w];
        tb += s_b[w];
    }
    if (threadIdx.x == 0) {
        unsigned long long* ctr = reinterpret_cast<unsigned long long*>(&flags[MC_FLAG_FILED]);
        const unsigned long long old = atomicAdd(ctr, ((unsigned long long)tb << 32) | tm);
        s_base = old;
        if ((long long)((old & 0xffffffffu) + tm) + (long long)((old >> 32) + tb) == B) *ctr = 0ull;
    }
    __syncthreads();
    const unsigned below = (1u << lane) - 1u;
    if (march) store_rec(rec, (long long)(unsigned)s_base + pm + __popc(mm & below), r);
    if (fill) store_rec(rec, B - 1 - ((long long)(s_base >> 32) + pb + __popc(mb & below)), r);
}

// Programmatic dependent launch: a kernel of the step may be scheduled while
// its predecessor in the stream still runs; it waits here before it touches
// anything the predecessor writes.  pdl_trigger lets the successor be scheduled.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// What bounds it: the latency of its dependent loads (action and state, then
// interaction samples and eye voxel), overlapped over 32 envs per warp, where a
// warp per env repeated every instruction 32 times.  Cold caches, with a thread
// per interaction (look_samples) throughout, 32768 envs took 11.7 us and 4096
// 11.6, at 17% and 10% of the issue slots.
template <int FAM>
__global__ void __launch_bounds__(kAgentThreads) k_agent(const __grid_constant__ mc_kp p) {
    pdl_trigger();
    pdl_wait();
    const long long e = (long long)blockIdx.x * kAgentThreads + threadIdx.x;
    const bool valid = e < p.B;
    const EnvRec r = agent_step<FAM>(p, ActionSrc{p.actions, p.buttons, p.look}, valid ? e : p.B - 1, valid,
                                     p.res_rewards, p.res_dones);
    file_recs(p.rec, p.flags, &p.flags[MC_FLAG_ANY_SLOW], p.B, p.compact, r, e, valid);
    if (threadIdx.x == 0) bounds_to_flags(p.flags);
}

// Cameras and records without a step (reset, get_obs: always the shaded
// family), one thread per env.  An env whose world this launch regenerates
// (fresh) looks into the template.
__global__ void __launch_bounds__(kAgentThreads) k_look(const __grid_constant__ mc_kp p) {
    pdl_trigger();
    pdl_wait();
    const long long e = (long long)blockIdx.x * kAgentThreads + threadIdx.x;
    const bool valid = e < p.B;
    const int any_done = regen_any(p);
    EnvRec r{};
    if (valid) {
        const float x = p.positions[e * 3 + 0], y = p.positions[e * 3 + 1], z = p.positions[e * 3 + 2];
        const float yaw = p.yaws[e], pitch = p.pitches[e];
        const bool done = p.regen != MC_KREGEN_NONE && p.do_reset[e] != 0;
        p.cameras[e * 5 + 0] = x;
        p.cameras[e * 5 + 1] = y;
        p.cameras[e * 5 + 2] = z;
        p.cameras[e * 5 + 3] = yaw;
        p.cameras[e * 5 + 4] = pitch;
        r = look_rec<MC_FAM_SHADED>(p, e, x, y, z, yaw, pitch, done, any_done);
    }
    file_recs(p.rec, p.flags, &p.flags[MC_FLAG_ANY_SLOW], p.B, p.compact, r, e, valid, false);
    if (threadIdx.x == 0) bounds_to_flags(p.flags);
}

// The same as k_agent for the groups of a ragged launch: blocks ablock[g] .. ablock[g+1]-1 hold group g's envs.
template <int FAM>
__global__ void __launch_bounds__(kAgentThreads) k_agent_groups(const __grid_constant__ mc_ragged_kp rk) {
    pdl_trigger();
    pdl_wait();
    int g = 0;
    while (g + 1 < rk.ngroups && (int)blockIdx.x >= rk.ablock[g + 1]) ++g;
    const mc_kp& p = rk.groups[g];
    const long long e = (long long)((int)blockIdx.x - rk.ablock[g]) * kAgentThreads + threadIdx.x, s0 = rk.start[g];
    const bool valid = e < p.B;
    const ActionSrc act{rk.actions ? rk.actions + s0 : nullptr, rk.actions ? nullptr : rk.buttons + 8 * s0,
                        rk.actions ? nullptr : rk.look + 2 * s0};
    const EnvRec r = agent_step<FAM>(p, act, valid ? e : p.B - 1, valid, rk.rewards_cat ? rk.rewards_cat + s0 : nullptr,
                                     rk.dones_cat ? rk.dones_cat + s0 : nullptr);
    file_recs(reinterpret_cast<EnvRec*>(rk.rec) + s0, p.flags, &rk.flags[MC_FLAG_ANY_SLOW], p.B, p.compact, r, e, valid);
    if (threadIdx.x == 0) bounds_to_flags(p.flags);
}

// ---------------------------------------------------------------------------
// The images
// ---------------------------------------------------------------------------
// What the render of one env needs.
struct EnvRender {
    Cam c;
    int bits;      // MC_ER_*
    int fill_blk;  // block of the uniform fill of a buried camera
    int ytop;      // no solid voxel above this layer (wy - 1 unless measured)
    UpBounds ub;   // bounds of the rays going up (up_none(ytop) unless measured)
};

__device__ __forceinline__ EnvRender render_of_rec(const EnvRec& q, int wy) {
    EnvRender r;
    r.c = cam_of_rec(q);
    r.bits = q.bits;
    r.fill_blk = q.fill_blk;
    r.ytop = wy - 1;
    r.ub = up_none(r.ytop);
    return r;
}

// Whether the eye's voxel lies in the box.
__device__ __forceinline__ bool eye_in_box(const Cam& c, int wx, int wy, int wz) {
    const int ex = (int)floorf(c.eye_x), ey = (int)floorf(c.eye_y), ez = (int)floorf(c.eye_z);
    return (unsigned)ex < (unsigned)wx && (unsigned)ey < (unsigned)wy && (unsigned)ez < (unsigned)wz;
}

// Measure a staged world for the rays going up: per quadrant of the eye's
// column when the eye's voxel lies in the box, else the top layer only.
__device__ __forceinline__ void measure_staged(EnvRender& r, const int8_t* world, int wx, int wy, int wz, int lane) {
    const int ex = (int)floorf(r.c.eye_x), ey = (int)floorf(r.c.eye_y), ez = (int)floorf(r.c.eye_z);
    if (eye_in_box(r.c, wx, wy, wz) && up_scan_shape(wx, wy, wz)) {
        r.ub = staged_up_bounds(world, wx, wy, wz, ex, ey, ez, lane);
        r.ytop = up_top(r.ub);
    } else {
        r.ytop = staged_top_layer(world, wx, wy, wz, lane);
        r.ub = up_none(r.ytop);
    }
}



// Barrier of one team (named barrier `bar`, nthreads threads).
__device__ __forceinline__ void team_sync(int bar, int nthreads) {
    if (nthreads == 32)
        __syncwarp();
    else
        asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(nthreads) : "memory");
}


// Where the staged copy of the world at src lies in its slot: at src's offset
// from a 16-byte boundary, so that a bulk copy can move its whole chunks.
__device__ __forceinline__ int8_t* staged_at(int8_t* slot, const int8_t* src) { return slot + ((uintptr_t)src & 15u); }

// Start the copy of one world into its slot (by one warp): the whole 16-byte
// chunks by a bulk copy, the bytes before and after them (worlds that start or
// end at any byte) by plain loads.  The stores precede lane 0's arrival, so
// whoever waits on the mbarrier sees them too.  All lanes are done with the
// world that was in the slot before any of it is overwritten.
__device__ __forceinline__ void issue_world_copy(uint32_t mbar_a, int8_t* slot, const int8_t* src, int bytes, int lane) {
    const int off = (int)((uintptr_t)src & 15u);
    int8_t* dst = slot + off;
    int head = 0, body = bytes;
    __syncwarp();
    if (off | (bytes & 15)) {  // uniform
        head = min((16 - off) & 15, bytes);
        const int tail = (bytes - head) & 15;
        body = bytes - head - tail;
        if (lane < head) dst[lane] = src[lane];
        if (lane < tail) dst[head + body + lane] = src[head + body + lane];
        __syncwarp();
    }
    if (lane == 0) {
        // generic-proxy reads of the previous world must precede the copy
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mbar_a), "r"(body) : "memory");
        if (body)
            asm volatile(
                "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                    smem_u32(dst + head)),
                "l"(src + head), "r"(body), "r"(mbar_a)
                : "memory");
    }
}

// Debug build: whether a staged world of `bytes` at dst lies in the CTA's
// dynamic shared memory (the same answer for every warp of a team).
__device__ __forceinline__ bool stage_fits(const int8_t* dst, int bytes) {
#if MC_CHECK_BOUNDS
    const SmemRange dyn = dyn_smem_range();
    const long long off = (long long)smem_u32(dst) - dyn.lo;
    return in_bounds(off, dyn.span, MC_SITE_STAGE) && in_bounds(off + bytes - 1, dyn.span, MC_SITE_STAGE);
#else
    (void)dst; (void)bytes;
    return true;
#endif
}

// Repeating 48-byte pattern written with 16-byte stores by nt threads.
__device__ __forceinline__ void fill_pattern16_n(uint8_t* dst, int bytes, uint4 p0, uint4 p1, uint4 p2, int t,
                                                 int nt) {
    uint4* d = reinterpret_cast<uint4*>(dst);
    const int n = bytes >> 4, adv = nt % 3;
    int m = t % 3;
    for (int k = t; k < n; k += nt) {
        d[k] = (m == 0) ? p0 : ((m == 1) ? p1 : p2);
        m += adv;
        if (m >= 3) m -= 3;
    }
}

// The uniform observation of a buried camera, written by nt threads.
template <int FAM, bool F32>
__device__ __forceinline__ void fill_env(const mc_kp& p, int e, int fill_blk, const FusedCtx& cx, int t, int nt) {
    const int HW = p.W * p.H;
    const long long obs_env_bytes = (long long)HW * 3 * (F32 ? 4 : 1);
    uint8_t* oenv = (uint8_t*)p.obs + e * obs_env_bytes;
    const bool vec_ok = ((obs_env_bytes & 15) == 0) && ((((uintptr_t)oenv) & 15) == 0);
    Hit h;
    h.blk = fill_blk;
    h.face = -1;
    h.t = 0.0f;
    h.step_y = 1;
    uint8_t bytes[12];
    if (F32 || FAM == MC_FAM_SHADED || FAM == MC_FAM_SHADED_FAST) {
        float rgb[3];
        shade_rgb<F32 ? MC_COL_F32 : (FAM == MC_FAM_SHADED_FAST ? MC_COL_U8FAST : MC_COL_U8)>(h, p.vd, cx.rcp_vd,
                                                                                              cx.s_rgb, cx.s_sky, rgb);
        if (F32) {
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                uint32_t w32 = __float_as_uint(rgb[k]);
                bytes[4 * k + 0] = (uint8_t)(w32);
                bytes[4 * k + 1] = (uint8_t)(w32 >> 8);
                bytes[4 * k + 2] = (uint8_t)(w32 >> 16);
                bytes[4 * k + 3] = (uint8_t)(w32 >> 24);
            }
        } else {
            bytes[0] = (uint8_t)to_u8(rgb[0]);
            bytes[1] = (uint8_t)to_u8(rgb[1]);
            bytes[2] = (uint8_t)to_u8(rgb[2]);
        }
    } else {
        bytes[0] = cx.s_rgb8[fill_blk][0];
        bytes[1] = cx.s_rgb8[fill_blk][1];
        bytes[2] = cx.s_rgb8[fill_blk][2];
    }
    const int period = F32 ? 12 : 3;
    if (vec_ok) {
        uint32_t w[12];
#pragma unroll
        for (int k = 0; k < 12; ++k) {
            w[k] = (uint32_t)bytes[(4 * k + 0) % period] | ((uint32_t)bytes[(4 * k + 1) % period] << 8) |
                   ((uint32_t)bytes[(4 * k + 2) % period] << 16) | ((uint32_t)bytes[(4 * k + 3) % period] << 24);
        }
        fill_pattern16_n(oenv, (int)obs_env_bytes, make_uint4(w[0], w[1], w[2], w[3]),
                         make_uint4(w[4], w[5], w[6], w[7]), make_uint4(w[8], w[9], w[10], w[11]), t, nt);
    } else {
        for (long long k = t; k < obs_env_bytes; k += nt) oenv[k] = bytes[k % period];
    }
    if (p.dbg_pixel) {
        int16_t code = dbg_code(h);
        for (int k = t; k < HW; k += nt) p.dbg_pixel[(long long)e * HW + k] = code;
    }
}

// Per-env facts that let the march stop early (see shade_ray / flat_ray).
struct MarchFacts {
    bool sky_exit, vd_safe;
};
template <int FAM>
__device__ __forceinline__ MarchFacts march_facts(const mc_kp& p, const EnvRender& r) {
    MarchFacts m;
    m.sky_exit = (FAM == MC_FAM_SHADED) ? ((r.bits & MC_ER_INSIDE) != 0 && p.vd > 0.0f && !p.dbg_pixel)
                                        : (eye_in_box(r.c, p.wx, p.wy, p.wz) && !p.dbg_pixel);
    m.vd_safe = m.sky_exit && box_within_view(r.c, p.wx, p.wy, p.wz, p.vd);
    return m;
}

// The next row band of this warp: the bands in turn when band_ctr is null,
// else those it claims from the team's shared counter.
__device__ __forceinline__ int next_band(int* band_ctr, int prev, int lane) {
    if (!band_ctr) return prev + 1;
    int v = 0;
    if (lane == 0) v = atomicAdd(band_ctr, 1);
    return __shfl_sync(0xffffffffu, v, 0);
}

// The general path, a pixel's ray at a time as in the reference's kernels:
// worlds that are not staged, debug outputs, eyes outside the box or out of
// view, families without a fast march.
template <int FAM, bool F32, class V>
__device__ __forceinline__ void render_slow_from(const mc_kp& p, int e, const EnvRender& r, const FusedCtx& cx,
                                                 const V& vox, int tile_w, int lane, int* band_ctr) {
    const int W = p.W, H = p.H;
    const RayPar rp = ray_par(p);
    int16_t* const dbg_pixel = p.dbg_pixel;
    const float vd = p.vd;
    const long long obs_env_bytes = (long long)W * H * 3 * (F32 ? 4 : 1);
    uint8_t* oenv = (uint8_t*)p.obs + e * obs_env_bytes;
    const bool inside = (r.bits & MC_ER_INSIDE) != 0, skip_first = (r.bits & MC_ER_SKIP) != 0;
    const MarchFacts mf = march_facts<FAM>(p, r);
    const Dda0 d0 = dda0(r.c);
    const int TW = tile_w, TH = 32 / tile_w;
    const int lx = lane % TW, ly = lane / TW;
    const int bpp = 3 * (F32 ? 4 : 1);
    const int nbands = (H + TH - 1) / TH;
    for (int b = next_band(band_ctr, -1, lane); b < nbands; b = next_band(band_ctr, b, lane)) {
        const int row0 = b * TH;
        const int py = row0 + ly;
        const float v = (py < H && in_bounds(py, H, MC_SITE_TABLE)) ? cx.s_v[py] : 0.0f;
        for (int tx0 = 0; tx0 < W; tx0 += TW) {
            const int px = tx0 + lx;
            if (px < W && py < H && in_bounds(px, W, MC_SITE_TABLE)) {
                const float u = cx.s_u[px];
                Hit h = march_pixel<FAM, V>(rp, r.c, d0, u, v, vox, inside, skip_first, mf.sky_exit, mf.vd_safe, r.ytop);
                if (!in_bounds(((long long)py * W + px + 1) * bpp - 1, obs_env_bytes, MC_SITE_COPY_OUT)) continue;
                uint8_t* o = oenv + ((long long)py * W + px) * bpp;
                if (FAM == MC_FAM_SHADED || FAM == MC_FAM_SHADED_FAST) {
                    float rgb[3];
                    shade_rgb<F32 ? MC_COL_F32 : (FAM == MC_FAM_SHADED_FAST ? MC_COL_U8FAST : MC_COL_U8)>(
                        h, vd, cx.rcp_vd, cx.s_rgb, cx.s_sky, rgb);
                    if (F32) {
#pragma unroll
                        for (int k = 0; k < 12; ++k) o[k] = (uint8_t)(__float_as_uint(rgb[k >> 2]) >> (8 * (k & 3)));
                    } else {
                        o[0] = (uint8_t)to_u8(rgb[0]);
                        o[1] = (uint8_t)to_u8(rgb[1]);
                        o[2] = (uint8_t)to_u8(rgb[2]);
                    }
                } else {
                    const uint8_t* col = (h.blk >= 0 && in_bounds(h.blk, 13, MC_SITE_TABLE)) ? cx.s_rgb8[h.blk] : cx.s_sky8;
                    o[0] = col[0];
                    o[1] = col[1];
                    o[2] = col[2];
                }
                if (dbg_pixel && in_bounds(py * W + px, W * H, MC_SITE_DEBUG))
                    dbg_pixel[(long long)e * W * H + py * W + px] = dbg_code(h);
            }
        }
    }
    // the lanes' rays end at different times, and the caller may now overwrite the world (regen_world)
    __syncwarp();
}

template <int FAM, bool F32>
__device__ __forceinline__ void render_slow(const mc_kp& p, const EnvRec& q, int ytop, const FusedCtx& cx,
                                            const int8_t* staged, const int8_t* world, int tile_w, int lane,
                                            int* band_ctr) {
    EnvRender r = render_of_rec(q, p.wy);
    r.ytop = ytop;
    if (staged)
        render_slow_from<FAM, F32>(p, q.env, r, cx, VoxShared{staged}, tile_w, lane, band_ctr);
    else
        render_slow_from<FAM, F32>(p, q.env, r, cx, VoxGlobal{world}, tile_w, lane, band_ctr);
}

// Row bands of slice `part` of `slices` of env e's image by one warp
// (next_band) in the common case: the launch allows it (mc_fast_launch), the
// world is staged, the eye is inside the box with air in its voxel.
template <int FAM, bool F32, bool TEAM>
__device__ __forceinline__ void render_fast(const mc_kp& p, int e, const EnvRender& r, const FusedCtx& cx,
                                            const int8_t* staged, int tile_w, int lane, int* band_ctr, int part,
                                            int slices) {
    const int sh = __ffs(tile_w) - 1, W = p.W, TH = 32 >> sh;
    constexpr int bpp = 3 * (F32 ? 4 : 1);
    uint8_t* oenv = (uint8_t*)p.obs + e * ((long long)W * p.H * bpp);
    const bool vd_safe = box_within_view(r.c, p.wx, p.wy, p.wz, p.vd);
    const int fk = fast_kind<FAM>(vd_safe, p.max_steps, p.wx, p.wy, p.wz);
    const Dda0 d0 = dda0(r.c);
    build_fast_start(cx.sstart, fk, d0, p.wx, p.wy, p.wz, FAM == MC_FAM_SHADED_FAST ? p.gh : 0, r.ub, p.max_steps,
                     lane);
    const uint32_t wb = smem_u32(staged);
    const int wxz = p.wx * p.wz;
    FastEnv fe;
    fe.start = cx.sstart;
    fe.base = fk == 1 ? wb : wb + (uint32_t)(d0.vy * wxz + d0.vx * p.wz + d0.vz);
    fe.chk = staged_range(wb, wxz, wxz * p.wy);
    fe.vd = p.vd;
    fe.rcp_vd = N::rcp_of(p.vd);
    fe.wx = p.wx;
    fe.wy = p.wy;
    fe.wz = p.wz;
    fe.max_steps = p.max_steps;
    const int H = p.H, nb = (H + TH - 1) >> (5 - sh), b0 = part * nb / slices, nbands = (part + 1) * nb / slices - b0;
    const bool odd = p.fast_ok == 2;
    for (int b = next_band(band_ctr, -1, lane); b < nbands; b = next_band(band_ctr, b, lane)) {
        const int row0 = (b0 + b) * TH;
        uint8_t* dst = oenv + row0 * W * bpp;
        if (odd) {
            if (fk == 1)
                fast_band<FAM, F32, false, true, TEAM>(r.c, d0, fe, W, H, sh, row0, lane, cx.s_u, cx.s_v, cx.s_cs,
                                                 cx.s_rgbp, cx.stage, dst);
            else
                fast_band<FAM, F32, true, true, TEAM>(r.c, d0, fe, W, H, sh, row0, lane, cx.s_u, cx.s_v, cx.s_cs,
                                                cx.s_rgbp, cx.stage, dst);
        } else if (fk == 1) {
            fast_band<FAM, F32, false, false, TEAM>(r.c, d0, fe, W, H, sh, row0, lane, cx.s_u, cx.s_v, cx.s_cs, cx.s_rgbp,
                                              cx.stage, dst);
        } else {
            fast_band<FAM, F32, true, false, TEAM>(r.c, d0, fe, W, H, sh, row0, lane, cx.s_u, cx.s_v, cx.s_cs, cx.s_rgbp,
                                             cx.stage, dst);
        }
    }
}

// n bytes of the template t (4-byte aligned, allocated to a multiple of 16) to a
// world d that starts at any byte, by nt threads: the world's aligned words,
// each funnelled from the two of the template it lies across, and the bytes
// before and after them.  (A byte a thread left a warp's 4680-byte world at 147
// rounds of a load and a store: a reset of 64 envs 9x40x13 took 42 us.)
__device__ __forceinline__ void regen_odd(int8_t* d, const int8_t* t, int n, int t0, int nt) {
    const int head = min((int)(-(uint32_t)(uintptr_t)d & 3u), n), words = (n - head) >> 2, tail = (n - head) & 3;
    if (t0 < head) d[t0] = t[t0];
    if (t0 < tail) d[n - tail + t0] = t[n - tail + t0];
    const uint32_t* s4 = reinterpret_cast<const uint32_t*>(t);
    uint32_t* d4 = reinterpret_cast<uint32_t*>(d + head);
#pragma unroll 1
    for (int k = t0; k < words; k += nt)
        d4[k] = __funnelshift_r(__ldg(s4 + k), head ? __ldg(s4 + k + 1) : 0u, 8 * head);
}

// The template's bytes over env e's world, by nt threads.  WORDS: worlds of no whole
// 16 bytes by regen_odd (the per-warp kernel); the team kernel, which has them in
// resets only (a kernel after its steps regenerates them), takes a byte a thread,
// since the words' code cost its other launches 1% (six ragged groups 240.7 -> 242.9
// us a step).
template <bool WORDS>
__device__ __forceinline__ void regen_world(const mc_kp& p, int e, int t, int nt) {
    const int wxyz = p.wx * p.wy * p.wz;
    int8_t* d = p.voxels + e * (long long)wxyz;
    // 16-byte stores only when every world starts on a 16-byte boundary
    // (a voxels view may start at any byte offset)
    if ((wxyz & 15) == 0 && ((((uintptr_t)p.voxels) | ((uintptr_t)p.world_template)) & 15) == 0) {
        uint4* d4 = reinterpret_cast<uint4*>(d);
        const uint4* t4 = reinterpret_cast<const uint4*>(p.world_template);
        for (int k = t; k < (wxyz >> 4); k += nt) d4[k] = __ldg(t4 + k);
    } else {
        if (WORDS)
            regen_odd(d, p.world_template, wxyz, t, nt);
        else
            for (int k = t; k < wxyz; k += nt) d[k] = p.world_template[k];
    }
}
// Whether this warp is the last of its env's slices to get here (all of them
// are then done reading the env's world).
__device__ __forceinline__ bool last_slice(const EnvRec* recs, int i, int slices, int lane) {
    if (slices == 1) return true;
    int prev = 0;
    __syncwarp();
    if (lane == 0) {
        __threadfence();
        prev = atomicAdd(const_cast<int*>(&recs[i].arrived), 1);
    }
    return __shfl_sync(0xffffffffu, prev, 0) == slices - 1;
}

#ifndef MC_FUSED_MIN_BLOCKS
#define MC_FUSED_MIN_BLOCKS 4
#endif
// The per-warp kernel's shared memory as one warp sees it; returns its world slot.
__device__ __forceinline__ int8_t* warp_ctx(const mc_kp& p, const FusedLayout& L, uint8_t* smem, int warp,
                                            FusedCtx& cx) {
    cx.s_cs = reinterpret_cast<const float4*>(smem);
    cx.s_rgbp = reinterpret_cast<const uint32_t*>(smem + kShadeTableBytes);
    float* s_u = reinterpret_cast<float*>(smem + kFastTableBytes);
    cx.s_u = s_u;
    cx.s_v = s_u + L.W;
    colour_tables(reinterpret_cast<uint8_t*>(s_u + L.W + L.H), cx);
    uint8_t* wbase = smem + L.head_bytes + warp * L.warp_bytes;
    cx.mbar_a = smem_u32(wbase);
    cx.sstart = reinterpret_cast<int4*>(wbase + 16);
    cx.stage = wbase + 16 + 128;
    cx.rcp_vd = N::rcp_of(p.vd);
    return reinterpret_cast<int8_t*>(wbase + 16 + 128 + L.stage_bytes);
}

// What a warp does besides the common path, out of line after its loop (so
// that the loop keeps its registers): from unit u on, the units of a warp
// whose copy timed out (no_stage), then its share of the general pass.
// state: bit 0 the mbarrier's phase, bit 1 no_stage, bit 2 that copy may still
// land, bit 3 a unit was left to the general pass.
template <int FAM, bool F32, bool STAGE>
__device__ __noinline__ void warp_rest(const mc_kp& p, int tile_w, int slices, int u, int state) {
    extern __shared__ __align__(16) uint8_t smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const int wxyz = p.wx * p.wy * p.wz;
    const FusedLayout L = fused_layout(p.W, p.H, mc_world_slot(p), p.wx * p.wz, F32, STAGE, tile_w, p.fast_ok);
    FusedCtx cx;
    int8_t* sworld = warp_ctx(p, L, smem, warp, cx);
    uint32_t phase = state & 1;
    bool no_stage = state & 2, pending = state & 4, slow = state & 8;
    const int total_warps = gridDim.x * nwarps, first = blockIdx.x * nwarps + warp;
    const EnvRec* recs = reinterpret_cast<const EnvRec*>(p.rec);
    const int any_done = regen_any(p);
    if (STAGE) {
        const int units = p.B * slices;
        // a copy that timed out: this unit and the rest of the warp's, from
        // global memory (a slice's warp renders the whole image: the others'
        // pixels come out the same)
        for (; no_stage && u < units; u = next_unit(p, MC_FLAG_WORK, u, total_warps, lane)) {
            const int i = u / slices, part = u - i * slices;
            const EnvRec q = rec_of<FAM>(p, i);
            if (q.bits & MC_ER_SLOW) {
                slow = true;
                continue;
            }
            if (!(q.bits & MC_ER_BURIED))
                render_slow<FAM, F32>(p, q, p.wy - 1, cx, nullptr, world_of(p, q.env, q.bits, any_done), tile_w, lane,
                                      nullptr);
            else if (part == 0)
                fill_env<FAM, F32>(p, q.env, q.fill_blk, cx, lane, 32);
            if (regen_env(p, q.bits, any_done) && last_slice(recs, i, slices, lane)) regen_world<true>(p, q.env, lane, 32);
        }
    }
    // the general pass: the envs that the common path left (every env of a
    // launch that has no common path)
    constexpr bool all = !STAGE;
    const int any_slow = __shfl_sync(0xffffffffu, *(volatile int32_t*)&p.flags[MC_FLAG_ANY_SLOW], 0);
    if (all || (p.sched_dynamic ? any_slow != 0 : slow)) {
        // (claimed: the envs; in turn: this warp's units again, whose first slices draw the whole image)
        const int per = p.sched_dynamic ? 1 : slices, units = p.B * per;
        u = p.sched_dynamic ? next_unit(p, MC_FLAG_SLOW_WORK, 0, total_warps, lane) : first;
        for (; u < units; u = next_unit(p, MC_FLAG_SLOW_WORK, u, total_warps, lane)) {
            if (u % per) continue;
            const EnvRec q = rec_of<FAM>(p, u / per);
            if (!all && !(q.bits & MC_ER_SLOW)) continue;
            if (q.bits & MC_ER_BURIED) {
                fill_env<FAM, F32>(p, q.env, q.fill_blk, cx, lane, 32);
            } else {
                const int8_t* world = world_of(p, q.env, q.bits, any_done);
                bool staged = STAGE && !no_stage && stage_fits(sworld, mc_world_slot(p));
                int ytop = p.wy - 1;
                if (staged) {
                    issue_world_copy(cx.mbar_a, sworld, world, wxyz, lane);
                    if (mbar_wait(cx.mbar_a, phase, p.wait_polls)) {
                        phase ^= 1u;
                        EnvRender r = render_of_rec(q, p.wy);
                        measure_staged(r, staged_at(sworld, world), p.wx, p.wy, p.wz, lane);
                        ytop = r.ytop;
                    } else {
                        if (lane == 0) atomicExch(&p.flags[MC_FLAG_ERROR], MC_KERR_TMA_TIMEOUT);
                        no_stage = pending = true;
                        staged = false;
                    }
                }
                render_slow<FAM, F32>(p, q, ytop, cx, staged ? staged_at(sworld, world) : nullptr, world, tile_w, lane, nullptr);
            }
            if (regen_env(p, q.bits, any_done)) regen_world<true>(p, q.env, lane, 32);
        }
    }
    // a timed-out copy may still be in flight: let it land (bounded, with the
    // default budget) before this warp's part of shared memory can be released
    if (STAGE && pending) mbar_wait(cx.mbar_a, phase);
}

// One warp per env: a persistent grid whose warps claim records, fill the
// buried envs and march the others over their world, staged in shared memory
// (STAGE) or in global memory.  Bound by instruction issue in the march; at
// its 64-register budget 4 CTAs of 8 warps share an SM.
//
// A small batch would leave most of the GPU's warps without an env: its images
// are cut into `slices` row ranges (slice_rows), each a unit of its own that stages
// the env's world again (a few KB from L2).
template <int FAM, bool F32, bool STAGE>
__global__ void __launch_bounds__(256, MC_FUSED_MIN_BLOCKS)
    k_render_warp(const __grid_constant__ mc_kp p, int tile_w, int slices) {
    extern __shared__ __align__(16) uint8_t smem[];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int nwarps = blockDim.x >> 5;
    const int total_warps = gridDim.x * nwarps;
    {
        const FusedLayout L = fused_layout(p.W, p.H, mc_world_slot(p), p.wx * p.wz, F32, STAGE, tile_w, p.fast_ok);
        build_fast_tables(reinterpret_cast<float4*>(smem), reinterpret_cast<uint32_t*>(smem + kShadeTableBytes));
        float* s_u = reinterpret_cast<float*>(smem + kFastTableBytes);
        build_uv_tables<FAM>(p, s_u, s_u + L.W);
        FusedCtx cx;
        load_colour_tables(reinterpret_cast<uint8_t*>(s_u + L.W + L.H), cx);
        if (STAGE) mbar_init_warp(smem_u32(smem + L.head_bytes + warp * L.warp_bytes), lane);
    }
    __syncthreads();
    pdl_trigger();
    pdl_wait();

    int u = 0, state = 0;
    if constexpr (STAGE) {
        const int wxyz = p.wx * p.wy * p.wz;
        const FusedLayout L = fused_layout(p.W, p.H, mc_world_slot(p), p.wx * p.wz, F32, STAGE, tile_w, p.fast_ok);
        FusedCtx cx;
        int8_t* sworld = warp_ctx(p, L, smem, warp, cx);
        const EnvRec* recs = reinterpret_cast<const EnvRec*>(p.rec);
        const int any_done = regen_any(p);
        const int units = p.B * slices;
        uint32_t phase = 0;
        u = p.sched_dynamic ? next_unit(p, MC_FLAG_WORK, 0, total_warps, lane) : blockIdx.x * nwarps + warp;
        for (; u < units; u = next_unit(p, MC_FLAG_WORK, u, total_warps, lane)) {
            const int i = u / slices, part = u - i * slices;
            const EnvRec q = rec_of<FAM>(p, i);
            if (q.bits & MC_ER_SLOW) {
                phase |= 2u;
                continue;
            }
            if (q.bits & MC_ER_BURIED) {
                if (part == 0) fill_env<FAM, F32>(p, q.env, q.fill_blk, cx, lane, 32);
            } else {
                if (!stage_fits(sworld, mc_world_slot(p))) {
                    state = 2;
                    break;
                }
                const int8_t* src = world_of(p, q.env, q.bits, any_done);
                issue_world_copy(cx.mbar_a, sworld, src, wxyz, lane);
                const int8_t* world = staged_at(sworld, src);
                EnvRender r = render_of_rec(q, p.wy);
                if (!mbar_wait(cx.mbar_a, phase & 1u, p.wait_polls)) {
                    if (lane == 0) atomicExch(&p.flags[MC_FLAG_ERROR], MC_KERR_TMA_TIMEOUT);
                    state = 2 | 4;
                    break;
                }
                phase ^= 1u;
                measure_staged(r, world, p.wx, p.wy, p.wz, lane);
                render_fast<FAM, F32, false>(p, q.env, r, cx, world, tile_w, lane, nullptr, part, slices);
            }
            if (regen_env(p, q.bits, any_done) && last_slice(recs, i, slices, lane)) regen_world<true>(p, q.env, lane, 32);
        }
        state |= (phase & 1u) | (phase & 2u) << 2;
    }
    // (a launch whose worlds are not staged has no common path)
    const int any_slow = __shfl_sync(0xffffffffu, *(volatile int32_t*)&p.flags[MC_FLAG_ANY_SLOW], 0);
    if (!STAGE || (p.sched_dynamic ? any_slow != 0 : (state & 8) != 0) || (state & 2)) warp_rest<FAM, F32, STAGE>(p, tile_w, slices, u, state);
    // No CTA barrier here: warps leave as soon as their last env is done.
    if (lane == 0) {
        bounds_to_flags(p.flags);
        // every claim of this warp has returned (the last one >= B)
        if (p.sched_dynamic)
            finish_dynamic(p.flags, total_warps, [&] {
                if (p.regen != MC_KREGEN_NONE) p.flags[MC_FLAG_ANY_DONE] = 0;
            });
    }
}

// ---------------------------------------------------------------------------
// Team kernel: the images of env groups of any size, by teams of warps
// ---------------------------------------------------------------------------
// A CTA of warps_per_cta warps is split into teams of team_warps warps.  A
// team claims one work unit at a time from a device counter:
//  * a cooperative group's unit is ONE env: all warps of the team march row
//    bands of its image (bands claimed from a shared counter), reading the
//    world from one shared-memory copy per team when staged.  Big images over
//    big worlds then keep an SM's L1 and shared memory on few worlds, like a
//    per-pixel kernel;
//  * a per-warp group's unit is team_warps envs, one per warp, each rendered
//    by its warp alone.
// Units are ordered by decreasing per-env cost across groups, so the most
// expensive envs are claimed first and do not straggle at the end.
//
// DEPTH 0: a launch without the images' common path (no group has it): the
// general pass alone, buried envs too.  (Passing every unit over in the common
// path's loop first cost 8192 envs 48^3 8x8 627 us a step instead of 375.)
// DEPTH 1: one world buffer per team (or warp); the unit's copy starts when
// its record is read.  DEPTH 2: two buffers; unit k+1's record is read and its
// copy started before unit k is rendered, so it overlaps that render (one
// claim further ahead, twice the shared memory).
//
// A warp whose wait for a copy runs out records the timeout; in the shared scan
// it stands in for its share of the layers with bounds that cut nothing, so
// the others' results stay exact.  After the unit's barrier its whole team draws
// that unit again and the rest of its units from global memory.
struct TeamShared {
    unsigned unit[4];      // claimed units, unit k's number at k & 3
    int band_ctr[2];       // next row band of the cooperative env of unit k & 1
    unsigned long long mbar[2];
    unsigned sunit[2];     // general pass: claimed units, alternating slots
    int lost;              // the unit (the team's k-th; kGeneralUnit + k in the general pass) whose wait for a copy
                           // ran out: no further copies, render from global memory.  A warp compares it with
                           // its own unit, so what warps ahead of it write there does not count yet.
    int any_done;          // bit g: every world of group g is to be regenerated
    int last;              // the team rendered its env's last slice
    int pad;
    // up bounds of the cooperative env of unit k & 1, combined over the team's warps (UpPart)
    int uxa[2][4], uya[2][4];
    unsigned long long ump[2], umm[2];
};
static_assert(sizeof(TeamShared) <= MC_TEAM_HEAD_BYTES, "team head");
constexpr int kGeneralUnit = 1 << 30;

__device__ __forceinline__ void team_unit_reset(TeamShared* ts, int d) {
    ts->band_ctr[d] = 0;
    ts->uxa[d][0] = 255; ts->uxa[d][1] = 0; ts->uxa[d][2] = 255; ts->uxa[d][3] = 0;
    ts->uya[d][0] = ts->uya[d][1] = ts->uya[d][2] = ts->uya[d][3] = 0;
    ts->ump[d] = ts->umm[d] = 0ull;
}

// The up bounds of a cooperative env, scanned by all nw warps of its team
// (warp w sweeps its share of the layers, staged_up_part) and combined in
// the team's shared words with shared-memory atomics, so every warp holds
// the same bounds after the team barrier.  Called by every warp of the team;
// `have` false: this warp may not read the world and adds bounds that cut nothing.
template <typename M>
__device__ __forceinline__ UpBounds team_up_bounds_t(bool have, const int8_t* world, int wx, int wy, int wz, int vx,
                                                     int vy, int vz, int lane, int w, int nw, TeamShared* ts, int d,
                                                     int bar) {
    UpPart<M> r;
    if (have) {
        r = staged_up_part<M>(world, wx, wy, wz, vx, vy, vz, lane, w, nw);
    } else {
        r.xa0 = 0; r.xa1 = wx - 1; r.xa2 = 0; r.xa3 = wx - 1;
        r.ya0 = r.ya1 = r.ya2 = r.ya3 = wy;
        r.mp = r.mm = (M(1) << (wz - 1)) | M(1);
    }
    if (lane == 0) {
        atomicMin(&ts->uxa[d][0], r.xa0);
        atomicMax(&ts->uxa[d][1], r.xa1);
        atomicMin(&ts->uxa[d][2], r.xa2);
        atomicMax(&ts->uxa[d][3], r.xa3);
        atomicMax(&ts->uya[d][0], r.ya0);
        atomicMax(&ts->uya[d][1], r.ya1);
        atomicMax(&ts->uya[d][2], r.ya2);
        atomicMax(&ts->uya[d][3], r.ya3);
        atomicOr(&ts->ump[d], (unsigned long long)r.mp);
        atomicOr(&ts->umm[d], (unsigned long long)r.mm);
    }
    team_sync(bar, nw * 32);
    UpPart<M> t;
    t.xa0 = ts->uxa[d][0];
    t.xa1 = ts->uxa[d][1];
    t.xa2 = ts->uxa[d][2];
    t.xa3 = ts->uxa[d][3];
    t.ya0 = ts->uya[d][0];
    t.ya1 = ts->uya[d][1];
    t.ya2 = ts->uya[d][2];
    t.ya3 = ts->uya[d][3];
    t.mp = (M)ts->ump[d];
    t.mm = (M)ts->umm[d];
    return up_bounds_of(t);
}
__device__ __forceinline__ UpBounds team_up_bounds(bool have, const int8_t* world, int wx, int wy, int wz, int vx,
                                                   int vy, int vz, int lane, int w, int nw, TeamShared* ts, int d,
                                                   int bar) {
    return wz > 32
               ? team_up_bounds_t<unsigned long long>(have, world, wx, wy, wz, vx, vy, vz, lane, w, nw, ts, d, bar)
               : team_up_bounds_t<uint32_t>(have, world, wx, wy, wz, vx, vy, vz, lane, w, nw, ts, d, bar);
}

#ifndef MC_TEAM_MIN_BLOCKS
#define MC_TEAM_MIN_BLOCKS 3  // 80 registers: the render path without spills
#endif
template <int FAM, bool F32, int DEPTH>
__global__ void __launch_bounds__(256, MC_TEAM_MIN_BLOCKS) k_render_team(const __grid_constant__ mc_ragged_kp rk) {
    constexpr bool COMMON = DEPTH > 0;
    constexpr int SLOTS = DEPTH > 1 ? DEPTH : 1;
    extern __shared__ __align__(16) uint8_t smem[];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int nwarps = blockDim.x >> 5;
    const int TWN = rk.team_warps;
    const int team = warp / TWN, wt = warp % TWN;
    const int teams_per_cta = nwarps / TWN;
    const int G = rk.ngroups;
    // layout: colour tables | u/v tables | teams | warps; the groups'
    // parameter blocks stay in the kernel's parameter space
    FusedCtx cx;
    load_colour_tables(smem, cx);
    build_fast_tables(reinterpret_cast<float4*>(smem + MC_COLOUR_TABLE_BYTES),
                      reinterpret_cast<uint32_t*>(smem + MC_COLOUR_TABLE_BYTES + kShadeTableBytes));
    cx.s_cs = reinterpret_cast<const float4*>(smem + MC_COLOUR_TABLE_BYTES);
    cx.s_rgbp = reinterpret_cast<const uint32_t*>(smem + MC_COLOUR_TABLE_BYTES + kShadeTableBytes);
    float* tables = reinterpret_cast<float*>(smem + rk.tables_off);
    for (int g = 0; g < G; ++g)
        build_uv_tables<FAM>(rk.groups[g], tables + rk.uv_off[g], tables + rk.uv_off[g] + rk.groups[g].W);
    TeamShared* ts = reinterpret_cast<TeamShared*>(smem + rk.teams_off + team * rk.team_bytes);
    int8_t* tworld = reinterpret_cast<int8_t*>(ts) + MC_TEAM_HEAD_BYTES;
    uint8_t* wbase = smem + rk.warps_off + warp * rk.warp_bytes;
    cx.mbar_a = smem_u32(wbase);  // this warp's mbarriers (per-warp groups), depth slot d's at + 8 d
    const uint32_t tmbar = smem_u32(ts->mbar);
    cx.sstart = reinterpret_cast<int4*>(wbase + 16);
    cx.stage = wbase + 16 + 128;
    const bool claimer = (wt == 0 && lane == 0);
    if (lane == 0) {
        for (int d = 0; d < SLOTS; ++d) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(cx.mbar_a + 8 * d) : "memory");
            if (wt == 0) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(tmbar + 8 * d) : "memory");
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const long long total_teams = (long long)gridDim.x * teams_per_cta;
    const unsigned total_units = (unsigned)rk.ustart[G];
    auto claim = [&](int counter) -> unsigned {
        return atomicAdd(reinterpret_cast<unsigned*>(&rk.flags[counter]), 1u);
    };
    pdl_trigger();
    pdl_wait();
    if (claimer) {
        ts->lost = 0x7fffffff;
        for (int k = 0; k < DEPTH; ++k) ts->unit[k] = claim(MC_FLAG_WORK);
        int any = 0;
        for (int g = 0; g < G; ++g)
            if (rk.groups[g].regen == MC_KREGEN_ALL && *(volatile int32_t*)&rk.groups[g].flags[MC_FLAG_ANY_DONE])
                any |= 1 << g;
        ts->any_done = any;
        team_unit_reset(ts, 0);
    }
    __syncthreads();
    const int bar = 1 + team, nthr = TWN * 32;
    uint32_t tphase = 0;     // bit d: parity of the team's next wait on depth slot d
    uint32_t wphase = 0;     // ... of this warp's own
    uint32_t tlive = 0, wlive = 0;  // bit d: a copy this warp issued into slot d that it has not seen land

    // Where unit u lies: its group and record, and whether this warp renders it.
    struct Unit {
        int g, i, part;
        bool coop, mine;
    };
    auto locate = [&](unsigned u) -> Unit {
        int vg = 0;
        while (vg + 1 < G && (long long)u >= rk.ustart[vg + 1]) ++vg;
        Unit t;
        t.g = rk.order[vg];
        const int local = (int)((long long)u - rk.ustart[vg]);
        t.coop = (rk.coop_mask >> t.g) & 1;
        t.i = t.coop ? local / rk.slices[t.g] : local * TWN + wt;
        t.part = t.coop ? local - t.i * rk.slices[t.g] : 0;
        t.mine = t.coop || t.i < rk.groups[t.g].B;
        return t;
    };
    auto slot_world = [&](int d, bool coop) -> int8_t* {
        return tworld + (DEPTH > 1 ? d * rk.world_stride : 0) + (coop ? 0 : wt * rk.slot_bytes);
    };
    auto recs_of = [&](int g) { return reinterpret_cast<const EnvRec*>(rk.rec) + rk.start[g]; };
    auto use_group = [&](int g) {
        cx.s_u = tables + rk.uv_off[g];
        cx.s_v = cx.s_u + rk.groups[g].W;
        cx.rcp_vd = N::rcp_of(rk.groups[g].vd);
    };
    // Start the copy of unit t's world into depth slot d when its env is one
    // of `kind` (its MC_ER_BURIED | MC_ER_SLOW bits): the team's first warp
    // for a cooperative env, every warp for its own env otherwise.
    auto issue = [&](const Unit& t, int d, int kind) {
        if (!((rk.stage_mask >> t.g) & 1) || (t.coop && wt != 0) || !t.mine) return;
        const EnvRec q = load_rec(recs_of(t.g), t.i);
        if ((q.bits & (MC_ER_BURIED | MC_ER_SLOW)) != kind) return;
        const mc_kp& p = rk.groups[t.g];
        const int wxyz = p.wx * p.wy * p.wz;
        int8_t* world = slot_world(d, t.coop);
        if (!stage_fits(world, mc_world_slot(p))) return;
        issue_world_copy((t.coop ? tmbar : cx.mbar_a) + 8 * d, world,
                         world_of(p, q.env, q.bits, (ts->any_done >> t.g) & 1), wxyz, lane);
        if (t.coop) tlive |= 1u << d;
        else wlive |= 1u << d;
    };
    // Where the staged copy of unit t's world lies (its record q).
    auto staged_world = [&](const Unit& t, const EnvRec& q, int d) -> const int8_t* {
        return staged_at(slot_world(d, t.coop), world_of(rk.groups[t.g], q.env, q.bits, (ts->any_done >> t.g) & 1));
    };
    // Wait for the copy of unit t, the team's number n, into depth slot d.
    auto landed = [&](const Unit& t, int d, int n) -> bool {
        const mc_kp& p = rk.groups[t.g];
        if (!stage_fits(slot_world(d, t.coop), mc_world_slot(p))) {
            *(volatile int*)&ts->lost = n;
            return false;
        }
        uint32_t& ph = t.coop ? tphase : wphase;
        if (!mbar_wait((t.coop ? tmbar : cx.mbar_a) + 8 * d, (ph >> d) & 1u, p.wait_polls)) {
            if (lane == 0) atomicExch(&p.flags[MC_FLAG_ERROR], MC_KERR_TMA_TIMEOUT);
            *(volatile int*)&ts->lost = n;
            return false;
        }
        ph ^= 1u << d;
        if (t.coop) tlive &= ~(1u << d);
        else wlive &= ~(1u << d);
        return true;
    };
    // After the unit's barrier: regenerate its env's world (see regen_world).
    auto regen = [&](const Unit& t, int bits, int e, bool sliced) {
        if (!t.mine || !regen_env(rk.groups[t.g], bits, (ts->any_done >> t.g) & 1)) return;
        const mc_kp& p = rk.groups[t.g];
        if (!t.coop) {
            regen_world<false>(p, e, lane, 32);
            return;
        }
        if (sliced && rk.slices[t.g] > 1) {  // team-uniform
            if (wt == 0) {
                const bool last = last_slice(recs_of(t.g), t.i, rk.slices[t.g], lane);
                if (lane == 0) ts->last = last;
            }
            team_sync(bar, nthr);
            if (!ts->last) return;
        }
        regen_world<false>(p, e, wt * 32 + lane, nthr);
    };

    if constexpr (COMMON) {
        int k = 0;
        bool redo = false;
        if (DEPTH > 1 && ts->unit[0] < total_units) issue(locate(ts->unit[0]), 0, 0);
        for (;; ++k) {
            const int d = DEPTH > 1 ? (k & 1) : 0;  // world slot and mbarrier of this unit
            const unsigned u = ts->unit[k & 3];
            if (u >= total_units) break;
            const Unit t = locate(u);
            if (DEPTH > 1) {
                const unsigned u1 = ts->unit[(k + 1) & 3];
                if (u1 < total_units) issue(locate(u1), d ^ 1, 0);
            } else {
                issue(t, d, 0);
            }
            if (claimer) team_unit_reset(ts, (k + 1) & 1);
            const mc_kp& p = rk.groups[t.g];
            int bits = MC_ER_SLOW, env = 0;
            if (t.mine) {
                const EnvRec q = load_rec(recs_of(t.g), t.i);
                bits = q.bits;
                env = q.env;
                use_group(t.g);
                if (q.bits & MC_ER_BURIED) {
                    if (t.part == 0)
                        fill_env<FAM, F32>(p, q.env, q.fill_blk, cx, t.coop ? wt * 32 + lane : lane,
                                           t.coop ? nthr : 32);
                } else if (!(q.bits & MC_ER_SLOW)) {
                    const bool ok = landed(t, d, k);
                    const int8_t* world = staged_world(t, q, d);
                    EnvRender r = render_of_rec(q, p.wy);
                    if (t.coop && TWN > 1 && up_scan_shape(p.wx, p.wy, p.wz))  // team-uniform; the eye is in the box
                        r.ub = team_up_bounds(ok, world, p.wx, p.wy, p.wz, (int)floorf(r.c.eye_x),
                                              (int)floorf(r.c.eye_y), (int)floorf(r.c.eye_z), lane, wt, TWN, ts, k & 1,
                                              bar);
                    else if (ok)
                        measure_staged(r, world, p.wx, p.wy, p.wz, lane);
                    if (ok)
                        render_fast<FAM, F32, true>(p, q.env, r, cx, world, rk.tile_w[t.g], lane,
                                                    t.coop ? &ts->band_ctr[k & 1] : nullptr, t.part, rk.slices[t.g]);
                }
            }
            if (claimer) ts->unit[(k + DEPTH) & 3] = claim(MC_FLAG_WORK);
            team_sync(bar, nthr);
            if (*(volatile int*)&ts->lost <= k) {  // the same for the whole team
                redo = true;
                break;
            }
            if (!(bits & MC_ER_SLOW)) regen(t, bits, env, true);
        }
        // a copy timed out: this unit again and the rest of the team's, from global memory
        if (redo) {
            const int k0 = k;
            if (claimer) team_unit_reset(ts, k & 1);
            team_sync(bar, nthr);
            for (;; ++k) {
                const unsigned u = ts->unit[k & 3];
                if (u >= total_units) break;
                const Unit t = locate(u);
                if (claimer) team_unit_reset(ts, (k + 1) & 1);
                const mc_kp& p = rk.groups[t.g];
                int bits = MC_ER_SLOW, env = 0;
                if (t.mine) {
                    const EnvRec q = load_rec(recs_of(t.g), t.i);
                    bits = q.bits;
                    env = q.env;
                    use_group(t.g);
                    if (q.bits & MC_ER_BURIED)
                        fill_env<FAM, F32>(p, q.env, q.fill_blk, cx, t.coop ? wt * 32 + lane : lane, t.coop ? nthr : 32);
                    else if (!(q.bits & MC_ER_SLOW))
                        render_slow<FAM, F32>(p, q, p.wy - 1, cx, nullptr,
                                              world_of(p, q.env, q.bits, (ts->any_done >> t.g) & 1), rk.tile_w[t.g],
                                              lane, t.coop ? &ts->band_ctr[k & 1] : nullptr);
                }
                if (claimer && k > k0) ts->unit[(k + DEPTH) & 3] = claim(MC_FLAG_WORK);
                team_sync(bar, nthr);
                if (!(bits & MC_ER_SLOW)) regen(t, bits, env, true);
            }
        }
    }
    // the general pass: the envs that the common path left
    constexpr int kGeneral = COMMON ? MC_ER_SLOW : MC_ER_SLOW | MC_ER_BURIED;
    if (claimer) {
        ts->sunit[0] = !COMMON || *(volatile int32_t*)&rk.flags[MC_FLAG_ANY_SLOW] ? claim(MC_FLAG_SLOW_WORK) : total_units;
        team_unit_reset(ts, 0);
    }
    team_sync(bar, nthr);
    for (int k = 0;; ++k) {
        const unsigned u = ts->sunit[k & 1];
        if (u >= total_units) break;
        const Unit t = locate(u);
        const mc_kp& p = rk.groups[t.g];
        const bool may_stage = ((rk.stage_mask >> t.g) & 1) && *(volatile int*)&ts->lost >= kGeneralUnit + k;
        if (may_stage && t.part == 0) issue(t, 0, MC_ER_SLOW);
        if (claimer) team_unit_reset(ts, (k + 1) & 1);
        int bits = 0, env = 0;
        bool here = false;  // this unit's env is rendered in this pass (the first slice's unit renders all of it)
        if (t.mine) {
            const EnvRec q = load_rec(recs_of(t.g), t.i);
            bits = q.bits;
            env = q.env;
            here = t.part == 0 && (q.bits & kGeneral);
            use_group(t.g);
            if (!COMMON && (q.bits & MC_ER_BURIED)) {
                fill_env<FAM, F32>(p, q.env, q.fill_blk, cx, t.coop ? wt * 32 + lane : lane, t.coop ? nthr : 32);
            } else if (here) {
                const int8_t* world = staged_world(t, q, 0);
                const bool staged = may_stage && landed(t, 0, kGeneralUnit + k);
                const int ytop = staged ? staged_top_layer(world, p.wx, p.wy, p.wz, lane) : p.wy - 1;
                render_slow<FAM, F32>(p, q, ytop, cx, staged ? world : nullptr,
                                      world_of(p, q.env, q.bits, (ts->any_done >> t.g) & 1), rk.tile_w[t.g], lane,
                                      t.coop ? &ts->band_ctr[k & 1] : nullptr);
            }
        }
        if (claimer) ts->sunit[(k + 1) & 1] = claim(MC_FLAG_SLOW_WORK);
        team_sync(bar, nthr);
        if (here) regen(t, bits, env, false);
    }
    // timed-out copies may still be in flight: let them land (bounded) before
    // this warp's part of shared memory can be released
    for (int d = 0; d < SLOTS; ++d) {
        if ((tlive >> d) & 1u) mbar_wait(tmbar + 8 * d, (tphase >> d) & 1u);
        if ((wlive >> d) & 1u) mbar_wait(cx.mbar_a + 8 * d, (wphase >> d) & 1u);
    }
    if (lane == 0) {
        for (int g = 0; g < G; ++g) bounds_to_flags(rk.groups[g].flags);
    }
    if (claimer)
        finish_dynamic(rk.flags, total_teams, [&] {
            for (int g = 0; g < G; ++g)
                if (rk.groups[g].regen != MC_KREGEN_NONE) rk.groups[g].flags[MC_FLAG_ANY_DONE] = 0;
        });
}

// ---------------------------------------------------------------------------
// Host launchers
// ---------------------------------------------------------------------------
static inline int grid_1d(long long n, int bs) { return (int)((n + bs - 1) / bs); }

static int render_launch(const mc_kp* p, int family, cudaStream_t s) {
    long long total = (long long)p->B * p->H * p->W;
    if (total == 0) return 0;
    switch (family) {
        case MC_FAM_SHADED:
            if (p->obs_f32) k_render_shaded<false, true><<<grid_1d(total, 128), 128, 0, s>>>(*p);
            else k_render_shaded<false, false><<<grid_1d(total, 128), 128, 0, s>>>(*p);
            break;
        case MC_FAM_SHADED_FAST:
            k_render_shaded<true, false><<<grid_1d(total, 128), 128, 0, s>>>(*p);
            break;
        case MC_FAM_MINIMAL:
            k_render_flat<MC_FAM_MINIMAL><<<grid_1d(total, 128), 128, 0, s>>>(*p);
            break;
        case MC_FAM_FP16:
            k_render_flat<MC_FAM_FP16><<<grid_1d(total, 128), 128, 0, s>>>(*p);
            break;
        case MC_FAM_PREBASIS:
            k_render_flat<MC_FAM_PREBASIS><<<grid_1d(total, 128), 128, 0, s>>>(*p);
            break;
        default:
            return (int)cudaErrorInvalidValue;
    }
    return (int)cudaGetLastError();
}

// The reference's step kernel sequence (kernels.cu:2457-2494, 2909-2991):
// episode check, decode, physics, interact, reset, counter, cameras,
// (basis), render.  World regeneration is launched by the caller.
static int step_plain(const mc_kp* p, cudaStream_t s) {
    if (p->B == 0) return 0;
    int gb = grid_1d(p->B, 256);
    k_episode_check<<<gb, 256, 0, s>>>(*p);
    k_decode<<<gb, 256, 0, s>>>(*p);
    k_physics<<<gb, 256, 0, s>>>(*p);
    k_interact<<<gb, 256, 0, s>>>(*p, 0);
    k_reset<<<gb, 256, 0, s>>>(*p);
    k_episode_update<<<gb, 256, 0, s>>>(*p);
    k_cameras<<<gb, 256, 0, s>>>(*p);
    if (p->family == MC_FAM_PREBASIS) k_basis<<<gb, 256, 0, s>>>(*p);
    int rc = (int)cudaGetLastError();
    if (rc) return rc;
    return render_launch(p, p->family, s);
}

static size_t warp_smem(const mc_kp& p, const mc_fused_cfg& cfg, int fast) {
    FusedLayout L = fused_layout(p.W, p.H, mc_world_slot(p), p.wx * p.wz, p.obs_f32, cfg.stage, cfg.tile_w, fast);
    return (size_t)L.head_bytes + (size_t)cfg.warps_per_cta * L.warp_bytes + (size_t)L.pad_bytes;
}

// The per-warp kernel's common path in this shape (mc_fast_launch, 0 where it does not fit).
static int warp_fast(const mc_kp& p, const mc_fused_cfg& cfg) {
    const int fast = mc_fast_launch(p, cfg.stage, cfg.tile_w);
    return warp_smem(p, cfg, fast) > 227 * 1024 ? 0 : fast;
}

// The shape as it is launched: small worlds that no shape can ask to stage are staged where they fit.
static mc_fused_cfg warp_stage(const mc_kp& p, const mc_fused_cfg& cfg) {
    mc_fused_cfg f = cfg;
    if (!f.stage && mc_odd_world(p) && mc_world_slot(p) <= 8192 + 16) {  // as default_launch stages the others
        f.stage = 1;
        if (warp_smem(p, f, warp_fast(p, f)) > 227 * 1024) f.stage = 0;
    }
    return f;
}

static size_t fused_smem(const mc_kp* p, const mc_fused_cfg* cfg) { return warp_smem(*p, *cfg, warp_fast(*p, *cfg)); }

// A launch whose kernel waits for its predecessor itself (pdl_wait), so that
// its own set-up overlaps the predecessor's end.
template <class... P, class... A>
static int launch_pdl(void (*kern)(P...), long long grid, int threads, size_t smem, cudaStream_t s, A&&... args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t lc{};
    lc.gridDim = dim3((unsigned)grid);
    lc.blockDim = dim3((unsigned)threads);
    lc.dynamicSmemBytes = smem;
    lc.stream = s;
    lc.attrs = &at;
    lc.numAttrs = 1;
    return (int)cudaLaunchKernelEx(&lc, kern, std::forward<A>(args)...);
}

// A kernel's dynamic shared memory above 48 KB has to be allowed on each device.
template <class K>
static int allow_smem(mc_once_per_device& limit, K kern, size_t smem) {
    if (smem <= 48 * 1024) return 0;
    int dev = -1;
    const cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    return limit(dev, [&] {
        return (int)cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    });
}

// Row ranges each image of the per-warp kernel is cut into: up to two units
// per warp of the grid.  Measured at 16^3, 32x32 images, in units per warp
// (4736 warps): 4096 envs 64.6 us a step at 0.9, 54.9 at 1.7, 61.8 at 3.5 (a
// slice stages and scans its world again); 32768 envs 163.9 at 6.9, 183.7 at 13.8;
// 64 envs 34.6 whole, 20.8 in 4 slices.
static int slices_of(long long B, int bands, long long warps) {
    int n = 1;
    while (n * 2 <= bands && B * n * 2 <= 2 * warps) n *= 2;
    return n;
}

static int warp_slices(const mc_kp& p, const mc_fused_cfg& f, int num_sms) {
    return slices_of(p.B, (p.H * f.tile_w + 31) / 32, (long long)num_sms * std::max(f.ctas_per_sm, 1) * f.warps_per_cta);
}

template <int FAM, bool F32, bool STAGE>
static int launch_warp_t(const mc_kp* p, const mc_fused_cfg* cfg, int slices, long long grid, cudaStream_t s) {
    auto kern = k_render_warp<FAM, F32, STAGE>;
    const size_t smem = warp_smem(*p, *cfg, p->fast_ok);
    static mc_once_per_device limit;  // per instantiation
    const int rc = allow_smem(limit, kern, smem);
    if (rc) return rc;
    return launch_pdl(kern, grid, 32 * cfg->warps_per_cta, smem, s, *p, cfg->tile_w, slices);
}

// The agents, then the images: one warp per env, or per slice of its image.
template <int FAM, bool F32>
static int launch_fused_f(const mc_kp* kp, const mc_fused_cfg* cfg, int num_sms, cudaStream_t s) {
    mc_kp p = *kp;
    mc_fused_cfg f = warp_stage(p, *cfg);
    cfg = &f;
    p.fast_ok = warp_fast(p, f);
    const int wpc = cfg->warps_per_cta;
    long long grid = (long long)num_sms * (cfg->ctas_per_sm > 0 ? cfg->ctas_per_sm : 1);
    const int slices = p.fast_ok ? warp_slices(p, f, num_sms) : 1;
    const long long units = (long long)p.B * slices;
    p.compact = p.sched_dynamic && units > grid * wpc;
    // static striding: four waves of CTAs, so that warps whose envs are cheap make
    // room (the stateless step, us: 32768 envs 16^3, 32x32 203 in one wave, 194 in
    // two, 190 in four, 204 in six; 4096 envs 45 in each)
    if (!p.sched_dynamic) grid *= 4;
    grid = std::max(1LL, std::min(grid, (units + wpc - 1) / wpc));
    int rc;
    if (FAM == MC_FAM_SHADED && p.look_only)
        rc = launch_pdl(k_look, grid_1d(p.B, kAgentThreads), kAgentThreads, 0, s, p);
    else
        rc = launch_pdl(k_agent<FAM>, grid_1d(p.B, kAgentThreads), kAgentThreads, 0, s, p);
    if (rc) return rc;
    return cfg->stage ? launch_warp_t<FAM, F32, true>(&p, cfg, slices, grid, s)
                      : launch_warp_t<FAM, F32, false>(&p, cfg, slices, grid, s);
}

template <int FAM, bool F32>
static int launch_team_t(const mc_ragged_kp* rk, int warps_per_cta, int ctas_per_sm, int num_sms, cudaStream_t s) {
    const int G = rk->ngroups;
    int rc;
    if (FAM == MC_FAM_SHADED && rk->groups[0].look_only)  // one group
        rc = launch_pdl(k_look, rk->ablock[G], kAgentThreads, 0, s, rk->groups[0]);
    else if (G == 1 && rk->flags == rk->groups[0].flags) {
        // one env's own launch: a parameter block instead of sixteen
        mc_kp p = rk->groups[0];
        p.rec = rk->rec;
        p.actions = rk->actions;
        p.buttons = rk->buttons;
        p.look = rk->look;
        p.res_rewards = rk->rewards_cat;
        p.res_dones = rk->dones_cat;
        rc = launch_pdl(k_agent<FAM>, rk->ablock[G], kAgentThreads, 0, s, p);
    } else {
        rc = launch_pdl(k_agent_groups<FAM>, rk->ablock[G], kAgentThreads, 0, s, *rk);
    }
    if (rc) return rc;
    bool common = false;
    for (int g = 0; g < G; ++g) common |= rk->groups[g].fast_ok != 0;
    const int which = !common ? 0 : (rk->depth == 2 ? 2 : 1);
    auto kern = which == 0 ? k_render_team<FAM, F32, 0> : (which == 2 ? k_render_team<FAM, F32, 2> : k_render_team<FAM, F32, 1>);
    size_t smem = (size_t)rk->warps_off + (size_t)warps_per_cta * rk->warp_bytes + (size_t)rk->tail_bytes;
    static mc_once_per_device limit[3];  // per kernel of this instantiation
    rc = allow_smem(limit[which], kern, smem);
    if (rc) return rc;
    const int teams_per_cta = warps_per_cta / rk->team_warps;
    long long ctas_needed = (rk->ustart[rk->ngroups] + teams_per_cta - 1) / teams_per_cta;
    long long grid = (long long)num_sms * (ctas_per_sm > 0 ? ctas_per_sm : 1);
    if (grid > ctas_needed) grid = ctas_needed;
    if (grid < 1) grid = 1;
    return launch_pdl(kern, grid, 32 * warps_per_cta, smem, s, *rk);
}

static int step_team(const mc_ragged_kp* rk, int family, int obs_f32, int warps_per_cta, int ctas_per_sm,
                     int num_sms, cudaStream_t s) {
    if (rk->ustart[rk->ngroups] == 0) return 0;
    switch (family) {
        case MC_FAM_SHADED:
            return obs_f32 ? launch_team_t<MC_FAM_SHADED, true>(rk, warps_per_cta, ctas_per_sm, num_sms, s)
                           : launch_team_t<MC_FAM_SHADED, false>(rk, warps_per_cta, ctas_per_sm, num_sms, s);
        case MC_FAM_SHADED_FAST: return launch_team_t<MC_FAM_SHADED_FAST, false>(rk, warps_per_cta, ctas_per_sm, num_sms, s);
        case MC_FAM_MINIMAL: return launch_team_t<MC_FAM_MINIMAL, false>(rk, warps_per_cta, ctas_per_sm, num_sms, s);
        case MC_FAM_FP16: return launch_team_t<MC_FAM_FP16, false>(rk, warps_per_cta, ctas_per_sm, num_sms, s);
        case MC_FAM_PREBASIS: return launch_team_t<MC_FAM_PREBASIS, false>(rk, warps_per_cta, ctas_per_sm, num_sms, s);
        default: return (int)cudaErrorInvalidValue;
    }
}

static int fused_common(const mc_kp* p, const mc_fused_cfg* cfg, int num_sms) {
    const mc_fused_cfg f = warp_stage(*p, *cfg);
    return warp_fast(*p, f) ? warp_slices(*p, f, num_sms) : 0;
}

static int step_fused(const mc_kp* p, const mc_fused_cfg* cfg, int num_sms, cudaStream_t s) {
    if (p->B == 0) return 0;
    switch (p->family) {
        case MC_FAM_SHADED:
            return p->obs_f32 ? launch_fused_f<MC_FAM_SHADED, true>(p, cfg, num_sms, s)
                              : launch_fused_f<MC_FAM_SHADED, false>(p, cfg, num_sms, s);
        case MC_FAM_SHADED_FAST: return launch_fused_f<MC_FAM_SHADED_FAST, false>(p, cfg, num_sms, s);
        case MC_FAM_MINIMAL: return launch_fused_f<MC_FAM_MINIMAL, false>(p, cfg, num_sms, s);
        case MC_FAM_FP16: return launch_fused_f<MC_FAM_FP16, false>(p, cfg, num_sms, s);
        case MC_FAM_PREBASIS: return launch_fused_f<MC_FAM_PREBASIS, false>(p, cfg, num_sms, s);
        default: return (int)cudaErrorInvalidValue;
    }
}

#if MC_CHECK_BOUNDS
// One failed check with no memory access behind it: shows that a violation
// reaches the record (the checks themselves cannot be made to fail on
// purpose without an out-of-range access to skip).
__global__ void k_bounds_selftest() {
    if (threadIdx.x == 0) (void)in_bounds(-1, 1, 0);
}
#endif
static int bounds_selftest(cudaStream_t s) {
#if MC_CHECK_BOUNDS
    k_bounds_selftest<<<1, 32, 0, s>>>();
    return (int)cudaGetLastError();
#else
    (void)s;
    return -1;
#endif
}

// The debug build's bounds-check record: out = {violations, first site,
// first index, its limit}, then cleared.  -1 (and out untouched) in the
// normal build, which checks nothing.
static int bounds_report(int32_t out[4], cudaStream_t s) {
#if MC_CHECK_BOUNDS
    int32_t h[4];
    cudaError_t e = cudaMemcpyFromSymbolAsync(h, g_bounds, sizeof(h), 0, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return (int)e;
    const int32_t zero[4] = {0, 0, 0, 0};
    e = cudaMemcpyToSymbolAsync(g_bounds, zero, sizeof(zero), 0, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return (int)e;
    for (int i = 0; i < 4; ++i) out[i] = h[i];
    return 0;
#else
    (void)out;
    (void)s;
    return -1;
#endif
}

static int basis_launch(const mc_kp* p, cudaStream_t s) {
    if (p->B == 0) return 0;
    k_basis<<<grid_1d(p->B, 256), 256, 0, s>>>(*p);
    return (int)cudaGetLastError();
}
static int decode_launch(const mc_kp* p, cudaStream_t s) {
    if (p->B == 0) return 0;
    k_decode<<<grid_1d(p->B, 256), 256, 0, s>>>(*p);
    return (int)cudaGetLastError();
}
static int physics_launch(const mc_kp* p, cudaStream_t s) {
    if (p->B == 0) return 0;
    k_physics<<<grid_1d(p->B, 256), 256, 0, s>>>(*p);
    return (int)cudaGetLastError();
}
static int interact_launch(const mc_kp* p, int break_only, cudaStream_t s) {
    if (p->B == 0) return 0;
    k_interact<<<grid_1d(p->B, 256), 256, 0, s>>>(*p, break_only);
    return (int)cudaGetLastError();
}
static int coalesced_launch(const int8_t* vox, const float* basis, uint8_t* out, int B, int ws, int W, int H,
                            int max_steps, cudaStream_t s) {
    if (B == 0 || W * H == 0) return 0;
    dim3 g(W * H, (B + 127) / 128);
    k_render_coalesced<<<g, 128, 0, s>>>(vox, basis, out, B, ws, W, H, max_steps);
    return (int)cudaGetLastError();
}

}  // namespace MC_NS
